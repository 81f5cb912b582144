"""The proposer's kernels at the edges of their tiles: batches around a CTA's samples and slices, against torch in 64 bits, with
tolerances from the operands' precision (BF16 products are exact in FP32; an FP32 sum of n terms is off by at most n * 2^-24 of the
sum of their magnitudes, and a BF16 result by 2^-9 of itself)."""
import pytest

pytestmark = pytest.mark.gpu

R, NFEAT, NOUT = 50, 32 * 48 * 48, 13


def _planes(x):
    import torch

    n, c = x.shape[:2]
    r = torch.zeros((n, R, R, c), dtype=x.dtype, device=x.device)
    r[:, 1:-1, 1:-1, :] = x.permute(0, 2, 3, 1)
    return r.reshape(n * R * R, c // 8, 8).permute(1, 0, 2).contiguous()


@pytest.mark.parametrize("n,shift", [(1, 0), (7, 0), (33, 0), (64, 0), (65, 1), (129, 0), (513, 0)])
def test_head_forward_and_backward(cuda_lib, n, shift):
    """shift: the backward pass's features and weights that many elements past a 16-byte boundary."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    feat = torch.relu(torch.randn((n, 32, 48, 48), generator=g, device="cuda")).to(torch.bfloat16)
    hw = torch.randn((NOUT, NFEAT), generator=g, device="cuda") * 1e-3
    hb = torch.randn(NOUT, generator=g, device="cuda")
    dout = torch.randn((n, NOUT), generator=g, device="cuda") / n
    s = torch.cuda.current_stream().cuda_stream
    fp = _planes(feat)
    hwt = torch.zeros((NFEAT, 16), device="cuda")
    out = torch.full((n, NOUT), 7.0, device="cuda")
    assert cuda_lib.ironav_prop_head_pack(hw.data_ptr(), hwt.data_ptr(), s) == 0
    assert cuda_lib.ironav_prop_head_fwd_packed(fp.data_ptr(), n, hwt.data_ptr(), hb.data_ptr(), out.data_ptr(), s) == 0
    f = feat.double().permute(0, 2, 3, 1).reshape(n, NFEAT)
    eps = 2.0 ** -24
    lim = NFEAT * eps * (f @ hw.double().abs().T + hb.double().abs())
    assert torch.all((out.double() - (f @ hw.double().T + hb.double())).abs() <= lim)
    fs, hs = torch.empty(fp.numel() + 8, dtype=fp.dtype, device="cuda"), torch.empty(hw.numel() + 4, device="cuda")
    fs[shift:shift + fp.numel()] = fp.reshape(-1)
    hs[shift:shift + hw.numel()] = hw.reshape(-1)
    ghw, ghb = torch.full_like(hw, 0.5), torch.full_like(hb, 0.25)  # accumulated into
    dz = torch.full((4, n * R * R, 8), 3.0, dtype=torch.bfloat16, device="cuda")
    assert cuda_lib.ironav_prop_head_bwd(fs.data_ptr() + 2 * shift, n, dout.data_ptr(), hs.data_ptr() + 4 * shift, ghw.data_ptr(), ghb.data_ptr(),
                                         dz.data_ptr(), s) == 0
    d = dout.double()
    assert torch.all((ghw.double() - 0.5 - d.T @ f).abs() <= (n + 2) * eps * (d.abs().T @ f + 0.5))
    assert torch.all((ghb.double() - 0.25 - d.sum(0)).abs() <= (n + 2) * eps * (d.abs().sum(0) + 0.25))
    want = _planes(((d @ hw.double()) * (f > 0)).reshape(n, 48, 48, 32).permute(0, 3, 1, 2))
    mags = _planes((d.abs() @ hw.double().abs()).reshape(n, 48, 48, 32).permute(0, 3, 1, 2))
    assert torch.all((dz.double() - want).abs() <= 2.0 ** -8 * want.abs() + (NOUT + 1) * eps * mags)


@pytest.mark.parametrize("cin", [16, 32])
@pytest.mark.parametrize("n", [1, 2, 31])
def test_convolution_and_weight_gradient(cuda_lib, n, cin):
    """One sample (9.8 tiles of 256 pixels, 19.5 of 128), a few, and enough that a CTA takes several tiles."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n + cin)
    x = torch.randn((n, cin, 48, 48), generator=g, device="cuda").to(torch.bfloat16)
    dz = torch.randn((n, 32, 48, 48), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((9, 32, cin), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    b = torch.randn(32, generator=g, device="cuda")
    xp, zp = _planes(x), _planes(dz)
    y = torch.full((4, n * R * R, 8), 7.0, dtype=torch.bfloat16, device="cuda")
    dw, db = torch.full((9, 32, cin), 0.5, device="cuda"), torch.full((32,), 0.25, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert cuda_lib.ironav_prop_conv3x3(xp.data_ptr(), cin, n, w.data_ptr(), b.data_ptr(), 0, None, y.data_ptr(), err.data_ptr(), s) == 0
    assert cuda_lib.ironav_prop_wgrad3x3(xp.data_ptr(), cin, zp.data_ptr(), n, dw.data_ptr(), db.data_ptr(), err.data_ptr(), s) == 0
    assert int(err.item()) == 0
    pad = torch.nn.functional.pad(x.double(), (1, 1, 1, 1))
    views = torch.stack([pad[:, :, t // 3:t // 3 + 48, t % 3:t % 3 + 48] for t in range(9)])  # [tap, n, in, 48, 48]
    want = _planes(torch.einsum("toi,tnihw->nohw", w.double(), views) + b.double()[:, None, None])
    ring = _planes(torch.ones((n, 32, 48, 48), device="cuda"))
    want = want * (ring > 0)
    mags = _planes(torch.einsum("toi,tnihw->nohw", w.double().abs(), views.abs()) + b.double().abs()[:, None, None])
    # tensor-core sums may be aligned to the largest term of a step: 2^-22 of the magnitudes covers 9 * cin / 16 steps
    assert torch.all((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 9 * cin * 2.0 ** -22 * mags)
    gw = torch.einsum("nohw,tnihw->toi", dz.double(), views)
    gm = torch.einsum("nohw,tnihw->toi", dz.double().abs(), views.abs())
    assert torch.all((dw.double() - 0.5 - gw).abs() <= n * 160 * 2.0 ** -22 * gm + 2.0 ** -20)
    assert torch.all((db.double() - 0.25 - dz.double().sum((0, 2, 3))).abs() <= n * 2500 * 2.0 ** -24 * dz.double().abs().sum((0, 2, 3)) + 2.0 ** -20)
