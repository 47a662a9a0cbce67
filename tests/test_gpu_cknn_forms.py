"""The forms of candidate-kNN's filter products, and what a call in which one form does not suffice costs."""
import numpy as np
import pytest

from oracle import cknn as ok

pytestmark = pytest.mark.gpu
KW = dict(top_k=2, top_m=3, tau=0.2, alpha=0.75)


def _case(seed, n_train, n_test, classes, k, spread):
    rng = np.random.default_rng(seed)
    protos = ok.row_l2(rng.standard_normal((classes, k)))
    y = (rng.integers(0, classes, n_train) + 1).astype(np.int32)
    Tr = protos[y - 1] + spread * rng.standard_normal((n_train, k))
    Tt = protos[rng.integers(0, classes, n_test)] + 0.3 * rng.standard_normal((n_test, k))
    return Tr, y, Tt, ok.centroids(Tr, y, classes)


def _same_as_tiles(lib, monkeypatch, form, args, knn_k):
    monkeypatch.setenv("FASTPLS_CKNN_TILES", form)
    got = lib.candidate_knn_predict(*args, knn_k=knn_k, **KW)
    monkeypatch.setenv("FASTPLS_CKNN_TILES", "3")
    ref = lib.candidate_knn_predict(*args, knn_k=knn_k, **KW)
    assert np.array_equal(got["top_index"], ref["top_index"])
    fin = np.isfinite(ref["top_score"])
    assert np.array_equal(np.isfinite(got["top_score"]), fin)
    return got["top_score"][fin], ref["top_score"][fin]


# classes below, at and above the 32 candidates of one register and the 128 slots of a pair; spreads with a few,
# all and too many rows of a class within the bar of the FP16 products (0.3, 3e-3) and of the split ones (1e-5)
@pytest.mark.parametrize("form", ["4", "5", "6"])
@pytest.mark.parametrize("n_train,classes", [(60, 3), (99, 3), (380, 3), (640, 5), (6000, 3)])
@pytest.mark.parametrize("spread", [0.3, 3e-3, 1e-5])
@pytest.mark.parametrize("k,knn_k", [(5, 1), (97, 16)])
def test_forms_agree_with_the_tiles(lib, monkeypatch, form, n_train, classes, spread, k, knn_k):
    Tr, y, Tt, cents = _case(31, n_train, 131, classes, k, spread)
    got, ref = _same_as_tiles(lib, monkeypatch, form, (Tt, Tr, y, cents), knn_k)
    # FP64 dots of at most 97 terms in another order (97 2^-53 |x||y|, twice), and the roundings of the smoothing
    assert np.max(np.abs(got - ref)) <= 1e-13 * (
        1.0 + np.linalg.norm(Tt, axis=1).max() * np.linalg.norm(Tr, axis=1).max())


# rows whose products, or themselves, fall below the range that the split products cover, and rows without a norm
@pytest.mark.parametrize("form", ["5", "6"])
@pytest.mark.parametrize("train,test", [(1e-40, 1e20), (1e20, 1e-40), (1e-25, 1e-16), (0.0, 1.0), (1.0, 0.0)])
def test_small_norms(lib, monkeypatch, form, train, test):
    Tr, y, Tt, cents = _case(33, 900, 141, 3, 40, 0.3)
    got, ref = _same_as_tiles(lib, monkeypatch, form, (test * Tt, train * Tr, y, cents), 7)
    scale = 1e-13 * (test * np.linalg.norm(Tt, axis=1).max()) * max(1.0, train * np.linalg.norm(Tr, axis=1).max())
    assert np.max(np.abs(got - ref), initial=0.0) <= scale


@pytest.mark.parametrize("form", ["5", "6"])
@pytest.mark.parametrize("where", ["train", "test"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e200])
def test_rows_without_a_norm(lib, monkeypatch, form, where, value):
    Tr, y, Tt, cents = _case(34, 1500, 140, 4, 20, 0.3)
    (Tr if where == "train" else Tt)[17, 3] = value
    got, ref = _same_as_tiles(lib, monkeypatch, form, (Tt, Tr, y, cents), 8)
    assert np.max(np.abs(got - ref) / (1.0 + np.abs(ref))) <= 1e-13


# a call of this size does not run its products twice where similarities crowd
@pytest.mark.parametrize("k", [20, 128])
def test_crowded_call_launches(lib, k):
    def launches(spread):
        Tr, y, Tt, cents = _case(35, 6000, 300, 20, k, spread)
        n0 = lib.launch_count()
        lib.candidate_knn_predict(Tt, Tr, y, cents, knn_k=5, **KW)
        return lib.launch_count() - n0
    assert launches(3e-3) == launches(0.3)
