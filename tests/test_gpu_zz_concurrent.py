"""GPU test of solves that run at the same time: handles of their own, each on its
own stream and host thread, must give the residual history that they give alone.
The grids have enough columns (32 x 2 x 148) for the post-smoother fed by tensor
copies, whose stages were once overwritten while other kernels shared an SM."""
import ctypes as C
import threading

import numpy as np
import pytest

from hicar_b200 import _capi, cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [(192, 193, 20), (224, 161, 32), (256, 160, 28), (160, 224, 24)]


@pytest.mark.parametrize("skip", [True, False])
def test_solves_on_several_streams_equal_the_solves_alone(lib, skip):
    from hicar_b200.domain import DeviceDomain, ptr
    from hicar_b200.wind_iterative import WindOptions
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = _capi.load()
    opt = WindOptions(windtype=0, tol_rel=1e-9, wind_solver_iterations=3000, precond=_capi.PRECOND_MG, stall_iters=50,
                      mg_omega=1.0 if skip else 0.8, mg_skip_fine_presmooth=skip, mg_w_levels=(2, 3, 4)).to_c()
    subs, failed = [], []
    try:
        for q, (nx, ny, nz) in enumerate(2 * SHAPES):
            dom = DeviceDomain.from_case(cases.build_case(nx, ny, nz, seed=70 + q, adv_den=True, n_hills=6), "cuda")
            h, stream, leak = C.c_void_p(), torch.cuda.Stream(), C.c_float()
            g = _capi.Grid(nx, ny, nz, dom.dx, 1)
            m = _capi.Metrics(*[ptr(dom.metrics[n]) for n in _capi.METRIC_FIELDS])
            torch.cuda.synchronize()
            _capi.check(lib.hicarw_init_iter_winds(C.byref(g), C.byref(opt), C.byref(m), _capi.MEM_DEVICE,
                                                   stream.cuda_stream, C.byref(h)))
            x = torch.zeros((ny + 2, nz + 2, nx + 2), dtype=torch.float64, device="cuda")
            x[1:-1, 1:-1, 1:-1] = torch.from_numpy(np.random.default_rng(q).standard_normal((ny, nz, nx)))
            subs.append((h, dom, stream, x))
            torch.cuda.synchronize()
            _capi.check(lib.hicarw_calibrate_projection_operator(
                h, ptr(dom.wind_alpha), ptr(dom.density), 1, ptr(dom.u_dqdt), ptr(dom.v_dqdt), ptr(dom.w_dqdt),
                C.byref(leak), _capi.MEM_DEVICE, stream.cuda_stream), h)

        def history(q):
            h, _, stream, x = subs[q]
            st, out = _capi.Stats(), (C.c_double * 200)()
            _capi.check(lib.hicarw_reset_solution(h, stream.cuda_stream), h)
            _capi.check(lib.hicarw_solve_rhs(h, ptr(x), _capi.MEM_DEVICE, stream.cuda_stream, C.byref(st)), h)
            assert st.status == 0
            return out[:lib.hicarw_get_history(h, out, 200)]

        def run(q):
            for _ in range(60):
                if history(q) != alone[q]:
                    failed.append(q)

        alone = [history(q) for q in range(len(subs))]
        threads = [threading.Thread(target=run, args=(q,)) for q in range(len(subs))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed, failed
    finally:
        for h, *_ in subs:
            lib.hicarw_finalize_iter_winds(h)
