"""GPU tests of the one-pass calibration (calibrate_kernel) against the
reference's probe hooks run one colour at a time, and of the coefficient copies
between the padded and the caller's layout."""
import ctypes as C

import numpy as np
import pytest

from hicar_b200 import _capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


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


def _coefs(dom, host):
    from hicar_b200 import wind_iterative as wi
    h, shape = wi.handle(dom.nest_indx), (15, dom.ny, dom.nz, dom.nx)
    if host:
        out = np.empty(shape, np.float32)
        _capi.check(_capi.load().hicarw_get_coefs(h, out.ctypes.data, _capi.MEM_HOST, None), h)
        return out
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    _capi.check(_capi.load().hicarw_get_coefs(h, C.c_void_p(out.data_ptr()), _capi.MEM_DEVICE, None), h)
    return out.cpu().numpy()


# smallest extents (every face an outer one, nz = 2: no inner level), block edges, odd sizes
@pytest.mark.parametrize("shape", [(3, 3, 2), (4, 5, 3), (129, 4, 2), (128, 7, 5), (37, 41, 9)])
@pytest.mark.parametrize("adv", [True, False])
def test_one_pass_calibration_equals_the_probe_hooks(shape, adv, capfd):
    from hicar_b200 import wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    case = cases.build_case(*shape, seed=11, adv_den=adv, n_hills=3, alpha="smooth")
    dom = DeviceDomain.from_case(case, "cuda")
    opt = wi.WindOptions(advect_density=adv)
    wi.init_iter_winds(dom, opt)
    leak = wind.calibrate_projection_operator(dom, opt)
    assert "leakage" not in capfd.readouterr().err  # none is measured
    one = _coefs(dom, host=False)
    np.testing.assert_array_equal(one, _coefs(dom, host=True))
    winds = [a.clone() for a in (dom.u_dqdt, dom.v_dqdt, dom.w_dqdt)]
    div = torch.empty((dom.ny, dom.nz, dom.nx), dtype=torch.float32, device="cuda")
    leak_hooks = wind.calibrate_projection_operator(dom, opt, div, on_device=False)
    assert "leakage max |T| = 0" in capfd.readouterr().err
    np.testing.assert_array_equal(one, _coefs(dom, host=False))
    assert leak == leak_hooks
    for a, b in zip(winds, (dom.u_dqdt, dom.v_dqdt, dom.w_dqdt)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("field", ["density", "alpha", "jacobian_u", "jacobian_v", "jacobian_w", "jacobian", "dzdx_u",
                                   "dzdy_v", "advection_dz", "mapfac_mx_u", "mapfac_my_u", "mapfac_mx_v", "mapfac_mxy"])
@pytest.mark.parametrize("adv", [True, False])
def test_undefined_geometry_reaches_the_same_coefficients(field, adv):
    """Zeros, infinities and NaN at a few places of one input field: the same finite, infinite and undefined
    coefficients as the probe hooks record."""
    from hicar_b200 import wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    case = cases.build_case(13, 11, 7, seed=12, adv_den=adv, n_hills=3, alpha="smooth")
    dom = DeviceDomain.from_case(case, "cuda")
    a = dom.density if field == "density" else dom.wind_alpha if field == "alpha" else dom.metrics[field]
    flat, rng = a.view(-1), np.random.default_rng(len(field))
    for value in (0.0, float("inf"), float("-inf"), float("nan")):
        flat[torch.from_numpy(rng.integers(0, flat.numel(), 2)).cuda()] = value
    if a.dim() == 3:  # the lowest and the highest level too
        a[3, 0, 5], a[7, -1, 4] = 0.0, float("nan")
    opt = wi.WindOptions(advect_density=adv)
    wi.init_iter_winds(dom, opt)
    leak = wind.calibrate_projection_operator(dom, opt)
    one = _coefs(dom, host=False)
    div = torch.empty((dom.ny, dom.nz, dom.nx), dtype=torch.float32, device="cuda")
    leak_hooks = wind.calibrate_projection_operator(dom, opt, div, on_device=False)
    np.testing.assert_array_equal(one, _coefs(dom, host=False))
    assert leak == leak_hooks


@pytest.mark.parametrize("shape", [(3, 3, 2), (130, 5, 3)])
@pytest.mark.parametrize("host", [True, False])
def test_coefficients_round_trip(shape, host):
    from hicar_b200 import wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    case = cases.build_case(*shape, seed=3, adv_den=True, n_hills=3)
    dom = DeviceDomain.from_case(case, "cuda")
    wi.init_iter_winds(dom, wi.WindOptions())
    h, lib = wi.handle(dom.nest_indx), _capi.load()
    rng = np.random.default_rng(1)
    a = rng.standard_normal((15, dom.ny, dom.nz, dom.nx)).astype(np.float32)
    t = torch.from_numpy(a).cuda()
    src = a.ctypes.data if host else t.data_ptr()
    _capi.check(lib.hicarw_set_coefs(h, C.c_void_p(src), 1, _capi.MEM_HOST if host else _capi.MEM_DEVICE, None), h)
    np.testing.assert_array_equal(_coefs(dom, host=True), a)
    np.testing.assert_array_equal(_coefs(dom, host=False), a)


@pytest.mark.parametrize("shift", [1, 4])
def test_copies_take_device_arrays_of_any_alignment(shift):
    """Coefficients, vectors and lambda in device arrays that start `shift` bytes past an aligned address: as from
    aligned ones."""
    from hicar_b200 import wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    case = cases.build_case(13, 9, 5, seed=4, adv_den=True, n_hills=3)
    dom = DeviceDomain.from_case(case, "cuda")
    wi.init_iter_winds(dom, wi.WindOptions(tol_rel=1e-8))
    wind.calibrate_projection_operator(dom, wi.WindOptions())
    h, lib = wi.handle(dom.nest_indx), _capi.load()

    def shifted(like, fill):
        raw = torch.zeros(like.numel() * like.element_size() + 16, dtype=torch.uint8, device="cuda")
        part = raw[shift:shift + like.numel() * like.element_size()]
        if fill:
            part.copy_(like.reshape(-1).view(torch.uint8))
        return part, C.c_void_p(part.data_ptr())

    def call(name, *a):
        rc = getattr(lib, name)(h, *a)
        assert rc >= 0, lib.hicarw_last_error(h)

    dev, rng = _capi.MEM_DEVICE, np.random.default_rng(9)
    x = torch.from_numpy(rng.standard_normal((dom.ny + 2, dom.nz + 2, dom.nx + 2))).cuda()
    xs, xp = shifted(x, True)
    for sweeps in (None, 0, 2):
        y = torch.empty_like(x)
        ys, yp = shifted(y, False)
        for src, dst in ((C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), (xp, yp)):
            if sweeps is None:
                call("hicarw_apply_operator", src, dst, dev, None)
            else:
                call("hicarw_apply_precond", src, dst, sweeps, dev, None)
        assert torch.equal(ys, y.reshape(-1).view(torch.uint8))
    lam, st = [], _capi.Stats()
    for src, out in ((C.c_void_p(x.data_ptr()), torch.empty_like(x)), (xp, None)):
        call("hicarw_reset_solution", None)
        call("hicarw_solve_rhs", src, dev, None, C.byref(st))
        if out is None:
            part, op = shifted(x, False)
            call("hicarw_get_lambda", op, dev, None)
            lam.append(part)
        else:
            call("hicarw_get_lambda", C.c_void_p(out.data_ptr()), dev, None)
            lam.append(out.reshape(-1).view(torch.uint8))
    assert torch.equal(*lam)
    coefs = torch.from_numpy(_coefs(dom, host=True)).cuda()
    part, p = shifted(coefs, False)
    call("hicarw_get_coefs", p, dev, None)
    assert torch.equal(part, coefs.reshape(-1).view(torch.uint8))
    other = coefs * 2
    part, p = shifted(other, True)
    call("hicarw_set_coefs", p, 1, dev, None)
    np.testing.assert_array_equal(_coefs(dom, host=True), other.cpu().numpy())


@pytest.mark.parametrize("ny", [65533, 65535])
def test_copies_of_as_many_lines_as_a_grid_has(ny):
    """Lambda, vectors and coefficients of the longest domain that a handle can be made for: with its two ghost lines
    it has more than 65535."""
    from hicar_b200 import wind_iterative as wi
    nx, nz, lib, dev = 3, 2, _capi.load(), _capi.MEM_DEVICE
    ones = lambda *s: torch.ones(s, device="cuda")  # noqa: E731
    shape = {"jacobian_u": (ny, nz, nx + 1), "dzdx_u": (ny, nz, nx + 1), "jacobian_v": (ny + 1, nz, nx),
             "dzdy_v": (ny + 1, nz, nx), "neighbor_terrain": (ny, nx), "mapfac_mx_u": (ny, nx + 1),
             "mapfac_my_v": (ny + 1, nx), "mapfac_my_u": (ny, nx + 1), "mapfac_mx_v": (ny + 1, nx), "mapfac_mxy": (ny, nx)}
    metrics = [ones(*shape.get(n, (ny, nz, nx))) for n in _capi.METRIC_FIELDS]
    h, g = C.c_void_p(), _capi.Grid(nx, ny, nz, 250.0, 1)
    m = _capi.Metrics(*[C.c_void_p(a.data_ptr()) for a in metrics])
    _capi.check(lib.hicarw_init_iter_winds(C.byref(g), C.byref(wi.WindOptions().to_c()), C.byref(m), dev, None, C.byref(h)))
    try:
        coefs = torch.zeros((15, ny, nz, nx), device="cuda")
        coefs[0] = torch.rand((ny, nz, nx), device="cuda") + 1
        _capi.check(lib.hicarw_set_coefs(h, C.c_void_p(coefs.data_ptr()), 1, dev, None), h)
        back = torch.empty_like(coefs)
        _capi.check(lib.hicarw_get_coefs(h, C.c_void_p(back.data_ptr()), dev, None), h)
        assert torch.equal(back, coefs)
        x = torch.rand((ny + 2, nz + 2, nx + 2), dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        _capi.check(lib.hicarw_apply_operator(h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), dev, None), h)
        assert torch.equal(y[1:-1, 1:-1, 1:-1], coefs[0].double() * x[1:-1, 1:-1, 1:-1])
        _capi.check(lib.hicarw_get_lambda(h, C.c_void_p(y.data_ptr()), dev, None), h)
        assert not bool(y.any())
    finally:
        lib.hicarw_finalize_iter_winds(h)
