"""GPU tests of the per-step kernels where their tiles end: update_stability in
columns of 32 and levels of 8, the w predictor in levels of 8, calc_alpha's edge
cells (each also over its own input), against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from hicar_b200 import _capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx,ny,nz", [(5, 6, 5), (31, 5, 8), (32, 5, 9), (33, 17, 17), (129, 16, 16)])
@pytest.mark.parametrize("halo", [0, 1, 2])
def test_per_step_kernels(lib, oracle_mod, nx, ny, nz, halo):
    from hicar_b200 import wind, wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    wi.finalize_iter_winds()
    case = cases.build_case(nx, ny, nz, seed=nx + halo, n_hills=3)
    dom = DeviceDomain.from_case(case, "cuda")
    wi.init_iter_winds(dom, wi.WindOptions())
    s = oracle_mod.OracleSolver(case.domain)
    rng = np.random.default_rng(nz)
    new = lambda: torch.empty((ny, nz, nx), device="cuda")  # noqa: E731
    # the w predictor
    w_real = rng.standard_normal((ny, nz, nx)).astype(np.float32)
    wind.calc_idealized_wgrid(dom, torch.from_numpy(w_real).cuda())
    want = s.idealized_wgrid(case.u, case.v, w_real)
    np.testing.assert_array_equal(dom.w_dqdt.cpu().numpy(), want)
    dom.w_dqdt.copy_(torch.from_numpy(w_real))
    wind.calc_idealized_wgrid(dom, dom.w_dqdt)
    np.testing.assert_array_equal(dom.w_dqdt.cpu().numpy(), want)
    # the bulk Richardson number (the Froude number's sector may differ within an ulp: its other test)
    theta, ft = cases.stability_inputs(case, seed=1, nsect=4)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (case.domain.z, theta, ft)]
    froude, ri = new(), new()
    wind.update_stability(dom, dev[0], dev[1], froude, ri, dev[2])
    fr_ref, ri_ref = s.update_stability(case.u, case.v, case.domain.z, theta, ft)
    np.testing.assert_array_equal(ri.cpu().numpy(), ri_ref)
    assert np.mean(froude.cpu().numpy() != fr_ref) < 0.01
    # the same over its inputs: each output in the place of theta or of the heights
    for f_at, r_at in ((0, None), (1, None), (None, 0), (None, 1), (0, 1), (1, 0)):
        ins, outs = [dev[0].clone(), dev[1].clone()], [new(), new()]
        for q, at in enumerate((f_at, r_at)):
            if at is not None:
                outs[q] = ins[at]
        wind.update_stability(dom, ins[0], ins[1], outs[0], outs[1], dev[2])
        assert torch.equal(outs[0], froude) and torch.equal(outs[1], ri)
    # alpha, into another array and over its input
    lib_ = _capi.load()
    fr = torch.from_numpy(fr_ref).cuda()
    out = new()
    h = wi.handle(dom.nest_indx)
    want = s.calc_alpha(fr_ref, halo)
    for dst in (out, fr):
        _capi.check(lib_.hicarw_calc_alpha(h, C.c_void_p(fr.data_ptr()), C.c_void_p(dst.data_ptr()), halo, 0, None), h)
        np.testing.assert_array_equal(dst.cpu().numpy(), want)
    # smoothing passes of every window kernel (marching rows in 16s, and the general one)
    for window, passes in ((1, 1), (1, 2), (2, 3), (3, 1)):
        a = torch.from_numpy(want).cuda()
        _capi.check(lib_.hicarw_smooth_alpha(h, C.c_void_p(a.data_ptr()), window, passes, 0, None), h)
        np.testing.assert_array_equal(a.cpu().numpy(), s.smooth_array(want, window, passes))
    wi.finalize_iter_winds()


def test_alpha_over_its_input_can_be_captured(lib, oracle_mod):
    """calc_alpha written over its Froude numbers, as the first call on a handle inside a stream capture: nothing is allocated."""
    from hicar_b200 import wind_iterative as wi
    from hicar_b200.domain import DeviceDomain
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    wi.finalize_iter_winds()
    case = cases.build_case(33, 17, 9, seed=5, n_hills=3)
    dom = DeviceDomain.from_case(case, "cuda")
    wi.init_iter_winds(dom, wi.WindOptions())
    fr = np.exp(np.random.default_rng(5).uniform(-3.0, 3.0, case.w.shape)).astype(np.float32)
    a = torch.from_numpy(fr).cuda()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = _capi.load().hicarw_calc_alpha(wi.handle(dom.nest_indx), C.c_void_p(a.data_ptr()), C.c_void_p(a.data_ptr()), 2,
                                            _capi.MEM_DEVICE, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _capi.HICARW_OK
    graph.replay()
    np.testing.assert_array_equal(a.cpu().numpy(), oracle_mod.OracleSolver(case.domain).calc_alpha(fr, 2))
    wi.finalize_iter_winds()
