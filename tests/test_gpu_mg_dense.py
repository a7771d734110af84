"""GPU tests of the dense coarse cycle: the V-cycle whose coarse levels are one
tabulated matrix against the numpy restatement, at the sizes where the choice of
the dense level changes, and after a change of the cycle's parameters."""
import ctypes as C

import numpy as np
import pytest

from hicar_b200 import _capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _fresh(lib, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hicar_b200 import wind, wind_iterative
    monkeypatch.delenv("HICARW_MG_FUSE", raising=False)
    wind_iterative.finalize_iter_winds()
    wind.reset()
    yield
    wind_iterative.finalize_iter_winds()
    wind.reset()


def _direction(h, x, **cycle):
    """M x up to a factor: one FGMRES step from zero for the right-hand side x moves
    along M x (hicarw_apply_precond itself runs the cycle step by step)."""
    from hicar_b200 import wind_iterative as wi
    wi.set_options(wi.WindOptions(tol_rel=1e-30, tol_abs=0.0, wind_solver_iterations=1, fgmres_restart=1,
                                  solver=_capi.SOLVER_FGMRES, precond=_capi.PRECOND_MG, **cycle))
    lib, y, st = _capi.load(), np.empty_like(x), _capi.Stats()
    _capi.check(lib.hicarw_reset_solution(h, None), h)
    _capi.check(lib.hicarw_solve_rhs(h, x.ctypes.data, _capi.MEM_HOST, None, C.byref(st)), h)
    _capi.check(lib.hicarw_get_lambda(h, y.ctypes.data, _capi.MEM_HOST, None), h)
    return y / np.linalg.norm(y)


def _dense_level(h):
    """The level that the profile's dense products name."""
    cap = 64
    names, ms, by, cnt = C.create_string_buffer(32 * cap), (C.c_double * cap)(), (C.c_double * cap)(), (C.c_int * cap)()
    n = _capi.load().hicarw_profile_iteration(h, 1, names, ms, by, cnt, cap, None)
    levels = [s for s in (names.raw[32 * q:32 * q + 32].split(b"\0")[0].decode() for q in range(n)) if "dense" in s]
    assert len(levels) == 1, levels
    return int(levels[0].replace("mg_dense_l", ""))


# dense level 1 with few, with an odd number of and with many unknowns; a lower level; rows of one aggregate;
# level 1 with 4096, 4092 and 3300 unknowns (dense with repeats only), with 3072 (the limit without) and 4224
# (over both limits)
@pytest.mark.parametrize("shape", [(6, 4, 3), (9, 7, 5), (32, 32, 8), (63, 65, 4), (33, 31, 9), (3, 40, 24), (70, 50, 33),
                                   (64, 64, 4), (66, 62, 4), (66, 50, 4), (64, 48, 4)])
def test_dense_coarse_cycle_against_the_restatement(shape):
    """Tolerance: the restatement runs the levels in FP32 as the per-level kernels
    do; 1e-5 is the bar of those kernels' own tests."""
    import mg_ref
    from hicar_b200 import wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    nx, ny, nz = shape
    case = cases.build_case(nx, ny, nz, seed=31, adv_den=True, n_hills=6)
    dom = DeviceDomain.from_case(case, "cuda")
    wi.init_iter_winds(dom, wi.WindOptions())
    wind.calibrate_projection_operator(dom, wi.WindOptions())
    h = wi.handle(dom.nest_indx)
    coefs = np.empty((15, ny, nz, nx), np.float32)
    _capi.check(_capi.load().hicarw_get_coefs(h, coefs.ctypes.data, _capi.MEM_HOST, None), h)
    rng = np.random.default_rng(41)
    x = np.zeros((ny + 2, nz + 2, nx + 2))
    x[1:-1, 1:-1, 1:-1] = rng.standard_normal((ny, nz, nx))
    first = None
    # the matrix belongs to the parameters of the call: change them and change them back
    for omega, wlev, scale, skip in ((0.8, (), 1.35, False), (1.0, (2, 3, 4), 1.35, True), (1.0, (1, 2), 1.1, True),
                                     (0.8, (), 1.35, False)):
        y = _direction(h, x, mg_omega=omega, mg_w_levels=wlev, mg_coarse_scale=scale, mg_skip_fine_presmooth=skip)
        ref = mg_ref.VCycle(coefs, omega, scale, fine_presmooth=not skip, wlevels=wlev)(x[1:-1, 1:-1, 1:-1])
        ref = ref / np.linalg.norm(ref)
        got = y[1:-1, 1:-1, 1:-1]
        sizes, level = (nx, ny), 0
        while not level or sizes[0] * sizes[1] * nz > (4096 if level in wlev else 3072):
            sizes, level = ((sizes[0] + 1) // 2, (sizes[1] + 1) // 2), level + 1
        assert _dense_level(h) == level
        assert np.linalg.norm(got - np.sign((got * ref).sum()) * ref) < 1e-5, (omega, wlev)
        assert not y[0].any() and not y[-1].any() and not y[:, 0].any() and not y[:, :, -1].any()
        first = y if first is None else first
    np.testing.assert_array_equal(y, first)
