"""GPU tests of the float4 column-marching operator kernels at the extents where
their groups of four columns, strips and level chunks end: the operator, the
set-up residual and the true residual against numpy."""
import ctypes as C

import numpy as np
import pytest

from hicar_b200 import _capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

OFF = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 1), (1, 0, -1),
       (-1, 0, 1), (-1, 0, -1), (1, 1, 0), (1, -1, 0), (-1, 1, 0), (-1, -1, 0)]


@pytest.fixture(autouse=True)
def _fresh(lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hicar_b200 import wind, wind_iterative
    wind_iterative.finalize_iter_winds()
    wind.reset()
    yield
    wind_iterative.finalize_iter_winds()
    wind.reset()


def _apply(coefs, x):
    """All rows: 15 points inside, identity on the ghost cells."""
    y = x.copy()
    n = [s - 2 for s in x.shape]
    acc = np.zeros(n)
    for c, (dk, dj, di) in zip(coefs.astype(np.float64), OFF):
        acc += c * x[1 + dj:1 + dj + n[0], 1 + dk:1 + dk + n[1], 1 + di:1 + di + n[2]]
    y[1:-1, 1:-1, 1:-1] = acc
    return y


@pytest.mark.parametrize("nx", [3, 4, 5, 6, 7, 127, 128, 129, 130, 131, 257])
@pytest.mark.parametrize("ny,nz", [(3, 2), (5, 17)])
def test_operator_and_residuals(nx, ny, nz):
    """Tolerance 1e-13: 15 FP64 products of FP32 coefficients summed in FP64; the
    norms are FP64 sums in another order."""
    from hicar_b200 import wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    dom = DeviceDomain.from_case(cases.build_case(nx, ny, nz, seed=1, n_hills=2), "cuda")
    opt = wi.WindOptions(tol_rel=1e-30, tol_abs=0.0, wind_solver_iterations=2)
    wi.init_iter_winds(dom, opt)
    h, lib = wi.handle(dom.nest_indx), _capi.load()
    rng = np.random.default_rng(nx + ny)
    coefs = rng.standard_normal((15, ny, nz, nx)).astype(np.float32)
    coefs[0] += 30.0  # diagonally dominant: the iterations below stay finite
    _capi.check(lib.hicarw_set_coefs(h, coefs.ctypes.data, 1, _capi.MEM_HOST, None), h)
    x = rng.standard_normal((ny + 2, nz + 2, nx + 2))
    y = np.empty_like(x)
    _capi.check(lib.hicarw_apply_operator(h, x.ctypes.data, y.ctypes.data, _capi.MEM_HOST, None), h)
    ref = _apply(coefs, x)
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)
    b = np.zeros_like(x)
    b[1:-1, 1:-1, 1:-1] = x[1:-1, 1:-1, 1:-1]
    st = _capi.Stats()
    lam = np.empty_like(x)
    for k in range(2):  # a cold start, then one from the solution so far
        res0 = np.linalg.norm(b) if k == 0 else np.linalg.norm(b - _apply(coefs, lam))
        _capi.check(lib.hicarw_solve_rhs(h, b.ctypes.data, _capi.MEM_HOST, None, C.byref(st)), h)
        _capi.check(lib.hicarw_get_lambda(h, lam.ctypes.data, _capi.MEM_HOST, None), h)
        assert st.iterations == 2  # (a breakdown at such a residual is no fault)
        bar = 1e-13 * np.linalg.norm(b)
        assert abs(st.res0 - res0) <= bar
        assert abs(st.true_res - np.linalg.norm(b - _apply(coefs, lam))) <= bar
