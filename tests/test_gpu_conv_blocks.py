"""GPU tests of the blocked tensor-core convolution where its blocks end: output
lines in fours, levels per block, 128-cell x-tiles, grids with fewer and with more
blocks than CTAs."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = torch.nn.functional


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (128, 4, 2), (129, 5, 1), (40, 3, 9), (127, 8, 33), (257, 6, 5),
                                      (20, 330, 7), (130, 61, 40)])
def test_blocks_against_fp64(lib, cin, cout, nx, ny, nz):
    """Channel 0 in FP32 against FP64 conv3d of the same BF16 values: 27 cin products
    summed in FP32, 1e-4 of the largest value as in the kernel's other tests; the
    BF16 outputs within BF16 rounding plus that; the halo stays zero."""
    from hicar_b200 import learned as L
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(nx + 7 * ny + nz)
    bf = lambda t: t.to(torch.bfloat16).double()  # noqa: E731
    x = bf(torch.randn((cin, ny, nz, nx), generator=g))
    w = bf(torch.randn((27, cin, cout), generator=g) * 0.1)
    b = torch.randn((cout,), generator=g)
    wt = w.reshape(3, 3, 3, cin, cout).permute(4, 3, 0, 1, 2)
    ref = F.conv3d(x[None], wt, b.double(), padding=1)[0]
    out, out0 = L.conv3(L.to_act(x), w.float().cuda(), b.cuda(), nx, ny, nz, cin, cout, want_out0=True)
    top = float(ref.abs().max())
    assert float((out0.double().cpu() - ref[0]).abs().max()) <= 1e-4 * top
    got = L.from_act(out, nx).double().cpu()
    assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3 * top).all())
    o = out.float()
    o[1:-1, 1:-1, :, 1:nx + 1] = 0
    assert not bool(o.any())


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (128, 2, 1), (129, 3, 2), (40, 4, 5), (20, 331, 3)])
@pytest.mark.parametrize("shift", [0, 1])
def test_weight_gradient_blocks_against_fp64(lib, cin, cout, nx, ny, nz, shift):
    """dY lines in ones, twos or threes with a remainder, added to what the gradient
    holds, also where it is not 16-byte aligned (shift); 1e-4 of the largest
    value, as in the kernel's other test."""
    import ctypes as C
    from hicar_b200 import _capi, learned as L
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(3 * nx + ny + nz)
    bf = lambda t: t.to(torch.bfloat16).double()  # noqa: E731
    x, dy = bf(torch.randn((cin, ny, nz, nx), generator=g)), bf(torch.randn((cout, ny, nz, nx), generator=g))
    wt = torch.zeros((cout, cin, 3, 3, 3), dtype=torch.float64, requires_grad=True)
    (F.conv3d(x[None], wt, padding=1)[0] * dy).sum().backward()
    ref = wt.grad.permute(2, 3, 4, 1, 0).reshape(27, cin, cout)
    buf = torch.ones(27 * cin * cout + 4, device="cuda")
    dw, db = buf[shift:shift + 27 * cin * cout], torch.zeros(cout, device="cuda")
    xa, ya = L.to_act(x), L.to_act(dy)
    rc = _capi.load().hicarw_nn_conv3_wgrad(cin, cout, nx, ny, nz, C.c_void_p(xa.data_ptr()), C.c_void_p(ya.data_ptr()),
                                            C.c_void_p(dw.data_ptr()), C.c_void_p(db.data_ptr()), None)
    assert rc == 0
    got = dw.double().cpu().reshape(27, cin, cout) - 1.0
    assert float((got - ref).abs().max()) <= 1e-4 * max(float(ref.abs().max()), 1.0)
    rb = dy.sum((1, 2, 3))
    assert float((db.double().cpu() - rb).abs().max()) <= 1e-4 * float(rb.abs().max().clamp(min=1.0))


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("ny", [1, 2, 4, 5, 331])
def test_weight_gradient_keeps_an_infinite_input_to_its_taps(lib, cin, cout, ny):
    """An infinite input in the last line, where the blocks of dY lines have a
    remainder: it enters no product of the taps dj = -1, whose dY line would be the one
    after the last; those gradients are as without it (1e-4 of the largest value)."""
    import ctypes as C
    from hicar_b200 import _capi, learned as L
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nx, nz = 40, 3
    g = torch.Generator().manual_seed(ny)
    bf = lambda t: t.to(torch.bfloat16).double()  # noqa: E731
    x, dy = bf(torch.randn((cin, ny, nz, nx), generator=g)), bf(torch.randn((cout, ny, nz, nx), generator=g))
    wt = torch.zeros((cout, cin, 3, 3, 3), dtype=torch.float64, requires_grad=True)
    (F.conv3d(x[None], wt, padding=1)[0] * dy).sum().backward()
    ref = wt.grad.permute(2, 3, 4, 1, 0).reshape(27, cin, cout)[:9]
    x[3, ny - 1, 1, 7] = float("inf")
    dw, db = torch.zeros(27 * cin * cout, device="cuda"), torch.zeros(cout, device="cuda")
    xa, ya = L.to_act(x), L.to_act(dy)
    rc = _capi.load().hicarw_nn_conv3_wgrad(cin, cout, nx, ny, nz, C.c_void_p(xa.data_ptr()), C.c_void_p(ya.data_ptr()),
                                            C.c_void_p(dw.data_ptr()), C.c_void_p(db.data_ptr()), None)
    assert rc == 0
    got = dw.double().cpu().reshape(27, cin, cout)
    assert float((got[:9] - ref).abs().max()) <= 1e-4 * max(float(ref.abs().max()), 1.0)
    assert not bool(torch.isfinite(got[13, 3]).any())
