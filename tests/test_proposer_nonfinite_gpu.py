"""The head's weight gradient with an output gradient that is not finite: the weights of the features that are zero in that sample
keep the other samples' gradient; the others take what IEEE arithmetic gives."""
import pytest

pytestmark = pytest.mark.gpu

R, NFEAT, NOUT = 50, 32 * 48 * 48, 13


@pytest.mark.parametrize("n,at", [(1, 0), (40, 5), (300, 299)])
def test_head_weight_gradient(cuda_lib, n, at):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    feat = torch.relu(torch.randn((n, 32, 48, 48), generator=g, device="cuda")).to(torch.bfloat16)
    r = torch.zeros((n, R, R, 32), dtype=feat.dtype, device="cuda")
    r[:, 1:-1, 1:-1, :] = feat.permute(0, 2, 3, 1)
    planes = r.reshape(n * R * R, 4, 8).permute(1, 0, 2).contiguous()
    hw = torch.randn((NOUT, NFEAT), generator=g, device="cuda") * 1e-3
    dout = torch.randn((n, NOUT), generator=g, device="cuda") / n
    dout[at, 0], dout[at, 3], dout[at, 12] = float("inf"), float("-inf"), float("nan")
    ghw, dz = torch.zeros_like(hw), torch.empty((4, n * R * R, 8), dtype=torch.bfloat16, device="cuda")
    assert cuda_lib.ironav_prop_head_bwd(planes.data_ptr(), n, dout.data_ptr(), hw.data_ptr(), ghw.data_ptr(), None, dz.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream) == 0
    f = feat.double().permute(0, 2, 3, 1).reshape(n, NFEAT)
    zero = f[at] == 0
    d = dout.double().clone()
    fin = torch.isfinite(d)
    d[~fin] = 0
    want = d.T @ f
    lim = (n + 2) * 2.0 ** -24 * (d.abs().T @ f)
    for j in range(NOUT):
        m = zero if not fin[at, j] else torch.ones_like(zero)
        assert torch.all((ghw[j, m].double() - want[j, m]).abs() <= lim[j, m]), j
    assert torch.all(ghw[0, ~zero] == float("inf")) and torch.all(ghw[3, ~zero] == float("-inf"))
    assert torch.all(torch.isnan(ghw[12, ~zero]))
