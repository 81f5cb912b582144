"""Reconstruction planes of other bases and strides through the coding kernel, which stores words of four samples: against the oracle
sample for sample and byte for byte outside the picture where the entry point takes them (16-byte bases, luma strides of 16 bytes,
chroma strides of 8 samples), refused with nothing written where it does not."""
import numpy as np
import pytest

from ironav_b200.inter import INTERCODE_DTYPE
from test_residual import _check_same, _random_decisions, blank_rec, p_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("off,pad", [(0, 0), (16, 16), (32, 48), (1, 0), (0, 1), (2, 2), (3, 5), (0, 4)])
def test_planes_of_other_bases_and_strides(oracle_lib, cuda_lib, off, pad, bd):
    import torch

    o, _, _, _, _ = p_case(oracle_lib, refs=2, bd=bd)
    c, _, _, _, _ = p_case(cuda_lib, refs=2, bd=bd, threads=False)
    decs = _random_decisions(np.random.default_rng(off * 10 + pad + bd), o.nmb, 2)
    decs["mode"][decs["mode"] == 0] = 2  # every sample is written
    want = o.code_inter(24, decs, blank_rec(o, bd))
    dt = np.uint8 if bd == 8 else np.uint16
    size, mark = np.dtype(dt).itemsize, 0x7A
    planes, shapes = [], [p.shape for p in want[1]]
    for h, w in shapes:  # `off` and `pad` in samples
        planes.append(torch.full((off * size + h * (w + pad) * size,), mark, dtype=torch.uint8, device="cuda"))
    c.set_stream(torch.cuda.current_stream().cuda_stream)
    td = torch.from_numpy(decs.view(np.uint8)).cuda()
    tc = torch.zeros(c.nmb * INTERCODE_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    ptr = [p.data_ptr() + off * size for p in planes]
    status = c.lib.ironav_code_inter_picture_device(c.ctx, 24, td.data_ptr(), tc.data_ptr(), ptr[0], shapes[0][1] + pad, ptr[1], ptr[2],
                                                    shapes[1][1] + pad)
    c.sync()
    if off % 16 or pad % 16:
        assert status == 3 and all((p.cpu().numpy() == mark).all() for p in planes)
        return
    assert status == 0
    got = []
    for (h, w), p in zip(shapes, planes):
        flat = p.cpu().numpy()
        rows = flat[off * size:].view(dt).reshape(h, w + pad)
        assert (flat[:off * size] == mark).all() and (rows[:, w:].copy().view(np.uint8) == mark).all()
        got.append(rows[:, :w])
    _check_same((tc.cpu().numpy().view(INTERCODE_DTYPE), got), want, f"off {off} pad {pad}")
