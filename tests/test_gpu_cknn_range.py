"""Candidate-kNN on score rows whose dot products leave the range of FP32: the scaled FP16 filter, and, where the
similarities crowd, the FP64 tiles in place of the unscaled split products."""
import numpy as np
import pytest

from oracle import cknn as ok

pytestmark = pytest.mark.gpu


# 141 test rows: the last tile of pairs of every class is ragged
@pytest.mark.parametrize("spread", [0.3, 1e-3])
def test_large_norms(lib, monkeypatch, spread):
    rng = np.random.default_rng(5)
    protos = ok.row_l2(rng.standard_normal((5, 40)))
    y = (rng.integers(0, 5, 3000) + 1).astype(np.int32)
    Tr = 1e25 * (protos[y - 1] + spread * rng.standard_normal((3000, 40)))
    Tt = 1e25 * (protos[rng.integers(0, 5, 141)] + 0.3 * rng.standard_normal((141, 40)))
    cents = ok.centroids(Tr, y, 5)
    kw = dict(top_k=2, top_m=3, knn_k=12, tau=0.2, alpha=0.75)
    got = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    monkeypatch.setenv("FASTPLS_CKNN_TILES", "3")
    ref = lib.candidate_knn_predict(Tt, Tr, y, cents, **kw)
    assert np.array_equal(got["top_index"], ref["top_index"])
    # the same FP64 dots of 40 terms in another order
    assert np.max(np.abs(got["top_score"] / ref["top_score"] - 1.0)) < 1e-13
