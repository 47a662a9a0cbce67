"""The tensor-core filter of candidate-kNN: FP16 products, split BF16 products, FP64 tiles."""
import numpy as np
import pytest

from oracle import cknn as ok

pytestmark = pytest.mark.gpu


def _case(seed, n_train, n_test, classes, k, spread):
    rng = np.random.default_rng(seed)
    protos = ok.row_l2(rng.standard_normal((classes, k)))
    y = (rng.integers(0, classes, n_train) + 1).astype(np.int32)
    Tr = protos[y - 1] + spread * rng.standard_normal((n_train, k))
    Tt = protos[rng.integers(0, classes, n_test)] + 0.3 * rng.standard_normal((n_test, k))
    return rng, Tr, y, Tt


# k: one column, ends of a 16-wide step and of a 64-wide box, the widest row;
# classes of a few rows, of several 128-row tiles and of two row chunks
@pytest.mark.parametrize("k,knn_k,n_train,classes", [
    (1, 1, 300, 3), (15, 16, 2000, 5), (16, 10, 900, 90), (63, 7, 3000, 6), (64, 16, 9000, 3),
    (65, 10, 3000, 6), (100, 10, 9000, 3), (128, 16, 2600, 20)])
@pytest.mark.parametrize("scaled", [False, True])
def test_filter_matches_oracle(lib, k, knn_k, n_train, classes, scaled):
    rng, Tr, y, Tt = _case(100 + k, n_train, 150, classes, k, 0.3)
    if scaled:   # rows of very different norms: one power of two serves all training rows
        Tr = Tr * 10.0 ** rng.uniform(-4, 4, (n_train, 1))
        Tt = Tt * 10.0 ** rng.uniform(-30, 2, (150, 1))
    cents = ok.centroids(ok.row_l2(Tr), y, classes)
    kw = dict(top_k=2, top_m=3, knn_k=knn_k, tau=0.2, alpha=0.75)
    got = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    ref = ok.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    assert np.array_equal(got["top_index"], ref["top_index"])
    # FP64 dots of at most 128 terms in another order: 128 2^-53 |x||y| each,
    # twice (the similarity and the base score), and a few roundings of the smoothing
    bound = 1e-13 * (1.0 + np.linalg.norm(Tt, axis=1) * np.linalg.norm(Tr, axis=1).max())
    assert np.all(np.abs(got["top_score"] - ref["top_score"]) <= bound[:, None])


# similarities of a class that crowd within 2^-9 of one another but not within
# 2^-13 (1e-3): the split BF16 products decide; within 2^-13 (1e-6): the FP64 tiles
@pytest.mark.parametrize("spread", [1e-3, 1e-6])
def test_crowded_similarities(lib, spread):
    _, Tr, y, Tt = _case(7, 3000, 140, 5, 40, spread)
    cents = ok.centroids(Tr, y, 5)
    kw = dict(top_k=2, top_m=3, knn_k=12, tau=0.2, alpha=0.75)
    got = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    ref = ok.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    assert np.array_equal(got["top_index"], ref["top_index"])
    assert np.max(np.abs(got["top_score"] - ref["top_score"])) <= 1e-13 * (
        1.0 + np.linalg.norm(Tt, axis=1).max() * np.linalg.norm(Tr, axis=1).max())


# rows that are not finite get the FP64 tiles' answer
@pytest.mark.parametrize("where,value", [("train", np.nan), ("train", np.inf), ("test", np.nan), ("test", np.inf),
                                         ("train", 1e200), ("test", 1e200)])
def test_rows_without_a_norm(lib, monkeypatch, where, value):
    _, Tr, y, Tt = _case(9, 1500, 140, 4, 20, 0.3)
    cents = ok.centroids(Tr, y, 4)
    (Tr if where == "train" else Tt)[17, 3] = value
    kw = dict(top_k=2, top_m=3, knn_k=8, tau=0.2, alpha=0.75)
    got = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    monkeypatch.setenv("FASTPLS_CKNN_TILES", "3")
    ref = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    assert np.array_equal(got["top_index"], ref["top_index"])
    fin = np.isfinite(ref["top_score"])
    assert np.array_equal(np.isfinite(got["top_score"]), fin)
    assert np.max(np.abs(got["top_score"][fin] - ref["top_score"][fin]) / (1.0 + np.abs(ref["top_score"][fin]))) <= 1e-13
