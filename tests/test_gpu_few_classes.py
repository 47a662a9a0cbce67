"""Row-wise top-k and argmax of class scores for few classes (a warp or two a row, a thread a row), against a plain
loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(scores):
    """A one-component model whose scores of row x are x[0] * scores."""
    m = scores.size
    return dict(R=np.array([[1.0], [0.0]]), W_latent=scores.reshape(1, m, 1).copy(order="F"),
                mX=np.zeros((1, 2)), vX=np.ones((1, 2)), mY=np.zeros((1, m)), m=m, p=2, ncomp=np.array([1]),
                pls_method="plssvd")


def _want(row, k):
    order = sorted((c for c in range(row.size) if row[c] > -np.inf), key=lambda c: (-row[c], c))[:k]
    idx = [c + 1 for c in order] + [0] * (k - len(order))
    val = [row[c] for c in order] + [-np.inf] * (k - len(order))
    return idx, val


# warps that share a row: as many as classes, or one for 8 of them where the rows fill the GPU; the argmax by a thread a row up to 4 classes, 48 from 16384 rows on and 128 from 65536 on
@pytest.mark.parametrize("m", [2, 5, 15, 31, 32, 48, 49, 63, 64, 128, 129])
@pytest.mark.parametrize("w", [33, 16383, 16384, 65535, 75777])
def test_few_classes(lib, m, w):
    rng = np.random.default_rng(m)
    base = rng.integers(-3, 4, size=m).astype(np.float64)
    x = np.zeros((w, 2))
    x[:, 0] = rng.choice([1.0, -1.0], size=w)
    k = min(3, m)
    got = lib.predict_classes(_model(base), x, top_k=k, return_scores=True)
    lab = lib.predict_classes(_model(base), x)["top_index"][:, 0, 0]
    for sign in (1.0, -1.0):
        rows = x[:, 0] == sign
        idx, val = _want(sign * base, k)
        assert (got["top_index"][rows, :, 0] == idx).all() and (got["top_score"][rows, :, 0] == val).all()
        assert (lab[rows] == idx[0]).all()
