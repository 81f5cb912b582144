"""The proposer's convolution and weight gradient cut into several launches (a batch beyond 400,000 samples is; here a few samples a
launch, by the test hooks): the outputs are the single launch's bit for bit, the sums' order aside for the weight gradient."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

R = 50


@pytest.mark.parametrize("cin", [16, 32])
@pytest.mark.parametrize("n,per", [(7, 1), (7, 2), (7, 3), (33, 32)])
def test_cut_batches(cuda_lib, n, per, cin):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n * per + cin)

    def planes(c):
        x = torch.randn((n, c, 48, 48), generator=g, device="cuda").to(torch.bfloat16)
        r = torch.zeros((n, R, R, c), dtype=x.dtype, device="cuda")
        r[:, 1:-1, 1:-1, :] = x.permute(0, 2, 3, 1)
        return r.reshape(n * R * R, c // 8, 8).permute(1, 0, 2).contiguous()

    x, dz, mask = planes(cin), planes(32), planes(32)
    w = (torch.randn((9, 32, cin), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    b = torch.randn(32, generator=g, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    ys, dws, dbs = [], [], []
    for limit in (None, per):
        y = torch.full((4, n * R * R, 8), 7.0, dtype=torch.bfloat16, device="cuda")
        dw, db = torch.zeros((9, 32, cin), device="cuda"), torch.zeros(32, device="cuda")
        conv = (x.data_ptr(), cin, n, w.data_ptr(), b.data_ptr(), 1, mask.data_ptr(), y.data_ptr(), err.data_ptr(), s)
        grad = (x.data_ptr(), cin, dz.data_ptr(), n, dw.data_ptr(), db.data_ptr(), err.data_ptr(), s)
        if limit is None:
            assert cuda_lib.ironav_prop_conv3x3(*conv) == 0 and cuda_lib.ironav_prop_wgrad3x3(*grad) == 0
        else:
            V, I, L = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
            cuda_lib.ironav_debug_prop_conv3x3.argtypes = [V, I, L, V, V, I, V, V, V, V, L]
            cuda_lib.ironav_debug_prop_wgrad3x3.argtypes = [V, I, V, L, V, V, V, V, L]
            assert cuda_lib.ironav_debug_prop_conv3x3(*conv, limit) == 0 and cuda_lib.ironav_debug_prop_wgrad3x3(*grad, limit) == 0
            assert cuda_lib.ironav_debug_prop_conv3x3(*conv, 0) == 3 and cuda_lib.ironav_debug_prop_wgrad3x3(*grad, 400001) == 3
        ys.append(y)
        dws.append(dw.double())
        dbs.append(db.double())
    assert int(err.item()) == 0
    assert torch.equal(ys[0], ys[1])
    # each a sum of n * 2304 products in FP32, aligned to a step's largest term by the tensor cores (2^-22 of the magnitudes a
    # step of 16 pixels, as the edge tests take it), whatever the order
    f = x.float().permute(1, 0, 2).reshape(n, R, R, cin)
    d = dz.float().permute(1, 0, 2).reshape(n, R, R, 32)[:, 1:-1, 1:-1].abs().double()
    mags = torch.stack([torch.einsum("nyxo,nyxi->oi", d, f[:, t // 3:t // 3 + 48, t % 3:t % 3 + 48].abs().double()) for t in range(9)])
    assert torch.all((dws[0] - dws[1]).abs() <= 2 * n * 160 * 2.0 ** -22 * mags + 2.0 ** -20)
    assert torch.all((dbs[0] - dbs[1]).abs() <= 2 * n * 2500 * 2.0 ** -24 * d.sum((0, 1, 2)) + 2.0 ** -20)
