"""Matrices that a call reads where they lie in device memory: aligned to a double only, with every scaling, next to
or inside the output's memory, and unchanged afterwards."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _at(a, offset, pad=0):
    """A column-major device matrix that starts `offset` doubles into its allocation; the allocation."""
    a = np.asarray(a, dtype=np.float64)
    mem = torch.full((a.size + offset + pad,), 7.25, dtype=torch.float64, device="cuda")
    mem[offset:offset + a.size] = torch.from_numpy(np.ascontiguousarray(a.T).ravel())
    return mem[offset:offset + a.size].reshape(a.shape[1], a.shape[0]).T, mem


def _host(t):
    return t.cpu().numpy()


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(2)
    L = rng.standard_normal((301, 5))
    X = L @ rng.standard_normal((5, 97)) + 0.3 * rng.standard_normal((301, 97))
    return X, L @ rng.standard_normal((5, 9)) + 0.1 * rng.standard_normal((301, 9)), rng.standard_normal((13, 97))


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("scaling", [1, 2, 3])
def test_fits_read_device_matrices(lib, data, scaling, offset):
    X, Y, Xt = data
    (Xd, xm), (Yd, ym), (Td, tm) = _at(X, offset), _at(Y, offset), _at(Xt, offset)
    before = [_host(m) for m in (xm, ym, tm)]
    y = (1 + np.arange(301) % 9).astype(np.int32)
    calls = {"fast": lambda X, Y, T: lib.pls_model2_fast(X, Y, [2, 4], scaling=scaling, fit=True),
             "classic": lambda X, Y, T: lib.pls_model2(X, Y, [2, 4], scaling=scaling, fit=True, svd_method=4),
             "plssvd": lambda X, Y, T: lib.pls_model1(X, Y, [2, 4], scaling=scaling, fit=True),
             "xprod": lambda X, Y, T: lib.pls_model1(X, Y, [2, 4], scaling=scaling, svd_method=4, xprod=True),
             "opls": lambda X, Y, T: lib.opls_filter(X, Y, 2, scaling=scaling),
             "lda": lambda X, Y, T: lib.pls_lda(X, Y, y, T, [2, 4], 9, scaling=scaling),
             "encode": lambda X, Y, T: lib.gaussian_y_encode(Y, np.linspace(-1, 1, 27).reshape(9, 3))}
    for name, call in calls.items():
        want, got = call(X, Y, Xt), call(Xd, Yd, Td)
        for key, w in want.items():
            if isinstance(w, np.ndarray):
                assert np.array_equal(got[key], w, equal_nan=True), (name, key)
    model = lib.pls_model2_fast(X, Y, [2, 4], scaling=scaling)
    assert np.array_equal(lib.predict_lowrank(model, Td)["Ypred"], lib.predict_lowrank(model, Xt)["Ypred"])
    assert np.array_equal(lib.predict_classes(model, Td)["top_index"], lib.predict_classes(model, Xt)["top_index"])
    for m, b in zip((xm, ym, tm), before):
        assert np.array_equal(_host(m), b)


@pytest.mark.parametrize("shift", [0, 5, 301 * 97])   # the output on the input, over part of it, behind it
def test_filter_output_over_its_input(lib, data, shift):
    X, Y, _ = data
    want = lib.opls_filter(X, Y, 2, scaling=2)
    Xd, mem = _at(X, 0, pad=shift)
    out = mem[shift:shift + X.size].reshape(97, 301).T
    got = lib.opls_filter(Xd, Y, 2, scaling=2, out=out)
    assert np.array_equal(_host(out), want["X"]) and np.array_equal(got["W_orth"], want["W_orth"])
    # and of the application, on its matrix
    again, mem = _at(X, 0, pad=shift)
    out = mem[shift:shift + X.size].reshape(97, 301).T
    args = (want["mX"], want["vX"], want["W_orth"], want["P_orth"])
    lib.opls_apply_filter(again, *args, out=out)
    assert np.array_equal(_host(out), lib.opls_apply_filter(X, *args))


def test_application_over_its_weights(lib, data):
    X, Y, _ = data
    f = lib.opls_filter(X, Y, 2)
    args = (f["mX"], f["vX"], f["W_orth"], f["P_orth"])
    want = lib.opls_apply_filter(X, *args)
    Xd, _ = _at(X, 0)
    out, mem = _at(np.zeros_like(X), 0)
    W, P = mem[:194], mem[194:388]   # the weights lie where the result goes
    W.copy_(torch.from_numpy(np.ascontiguousarray(f["W_orth"].T).ravel()))
    P.copy_(torch.from_numpy(np.ascontiguousarray(f["P_orth"].T).ravel()))
    torch.cuda.synchronize()
    lib.opls_apply_filter(Xd, f["mX"], f["vX"], W.reshape(2, 97).T, P.reshape(2, 97).T, out=out)
    assert np.array_equal(_host(out), want)
