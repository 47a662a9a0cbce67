"""Row-wise top-k and argmax of class scores: list lengths, class counts around
the warps' strides, ties, NaN and infinities, against a plain loop."""
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


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 8, 9, 13, 17, 21, 32])
@pytest.mark.parametrize("m,w", [(32, 1), (33, 31), (127, 33), (1000, 70), (64, 20000)])
def test_topk_lists(lib, k, m, w):
    rng = np.random.default_rng(k * 1000 + m)
    base = rng.integers(-6, 7, size=m).astype(np.float64)       # many ties
    x = np.zeros((w, 2))
    x[:, 0] = rng.choice([1.0, -1.0, 2.0], size=w)
    bias = rng.integers(-2, 3, size=m) * 0.5
    got = lib.predict_classes(_model(base), x, class_bias=bias, top_k=k, return_scores=True)
    for i in list(range(min(w, 40))) + [w - 1]:
        idx, val = _want(x[i, 0] * base + bias, k)
        assert got["top_index"][i, :, 0].tolist() == idx
        assert got["top_score"][i, :, 0].tolist() == val
    lab = lib.predict_classes(_model(base), x, class_bias=bias, top_k=1)["top_index"][:, 0, 0]
    assert lab.tolist() == (np.argmax(x[:, :1] * base + bias, axis=1) + 1).tolist()


def test_special_values(lib):
    m = 40
    bias = np.zeros(m)
    x = np.array([[1.0, 0.0], [-1.0, 0.0]])
    bias[5], bias[7] = -np.inf, np.nan
    got = lib.predict_classes(_model(np.arange(m, dtype=float)), x, class_bias=bias, top_k=m - 8, return_scores=True)
    assert got["top_index"][0, :3, 0].tolist() == [40, 39, 38] and 8 not in got["top_index"][:, :, 0]
    assert got["top_index"][1, :7, 0].tolist() == [1, 2, 3, 4, 5, 7, 9]
    low = np.full(m, -np.inf)                                   # no finite score at all
    got = lib.predict_classes(_model(np.ones(m)), x, class_bias=low, top_k=4, return_scores=True)
    assert not got["top_index"].any() and np.all(np.isneginf(got["top_score"]))
    assert lib.predict_classes(_model(np.ones(m)), x, class_bias=low)["top_index"].ravel().tolist() == [1, 1]
    first = np.zeros(m)
    first[0] = np.nan                                           # nothing exceeds a NaN first score
    assert lib.predict_classes(_model(np.ones(m)), x, class_bias=first)["top_index"].ravel().tolist() == [1, 1]
