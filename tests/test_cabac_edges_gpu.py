"""CABAC at the edges of its pieces, bit for bit against the oracle: pictures about a group of five macroblocks wide (the P_Skip tests
of a group, and the ones that end a row), levels dense and large enough that a macroblock's bins take several turns of a list
(QP 0, escape-coded levels), both transforms, both bit depths; and a launch of more chains than the chip has SMs."""
from __future__ import annotations

import numpy as np
import pytest

from ironav_b200.encoder import Encoder
from tests.test_chain_gpu import _run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mb_w", [1, 2, 4, 5, 6, 11])
@pytest.mark.parametrize("bd", [8, 10])
def test_widths_about_a_group(oracle_lib, mb_w, bd):
    _run_pair(oracle_lib, "cif", 4, size=(mb_w * 16, 64), qp=30, keyint=30, refs=1, nslices=2, bd=bd, cabac=True)


@pytest.mark.parametrize("transform8", [False, True])
@pytest.mark.parametrize("bd,qp", [(8, 0), (8, 6), (10, 0), (10, 4)])
def test_long_lists(oracle_lib, cuda_lib, bd, qp, transform8):
    """Noise: every level non-zero, most beyond the unary prefix."""
    rng = np.random.default_rng(qp + 50)
    a, b = (Encoder(80, 48, qp=qp, keyint=30, nslices=2, refs=1, bd=bd, scene_cut=False, lib=lib, cabac=True, transform8=transform8)
            for lib in (oracle_lib, cuda_lib))
    dt = np.uint8 if bd == 8 else np.uint16
    for t in range(3):
        f = tuple(rng.integers(0, 1 << bd, s).astype(dt) for s in ((48, 80), (24, 40), (24, 40)))
        assert a.encode(*f) == b.encode(*f), f"picture {t}"
    a.close()
    b.close()


def test_more_chains_than_sms(oracle_lib, cuda_lib):
    """40 streams of four to six bands: the first chains in the wide form, the others a warp each; every stream as on its own."""
    import torch

    from ironav_b200.inter import MBCODE_DTYPE, MBSTATE_DTYPE, InterBatch
    from tests.test_decide import _same_decisions, decide_case

    cases = [dict(size=(96, 96), nslices=4 + i % 3, qp=22 + i % 9, new_content=i % 5 == 0) for i in range(40)]
    stages, want = [], []
    for kw in cases:
        st = decide_case(cuda_lib, threads=False, **kw)[0]
        st.set_entropy(True, True)
        stages.append(st)
        o = decide_case(oracle_lib, **kw)[0]
        o.set_entropy(True, True)
        want.append(o.decide_p_picture())
        o.close()
    stream = torch.cuda.Stream()
    for st in stages:
        st.set_stream(stream.cuda_stream)
    u8 = dict(dtype=torch.uint8, device="cuda")
    bufs = [(torch.zeros(st.nmb * 72, **u8), torch.zeros(st.nmb * 1516, **u8), torch.zeros((st.mb_h * 16, st.mb_w * 16), **u8),
             torch.zeros((2, st.mb_h * 8, st.mb_w * 8), **u8)) for st in stages]
    batch = InterBatch(stages)
    batch.decide([b[0].data_ptr() for b in bufs], [b[1].data_ptr() for b in bufs], [b[2].data_ptr() for b in bufs],
                 [b[2].shape[1] for b in bufs], [b[3][0].data_ptr() for b in bufs], [b[3][1].data_ptr() for b in bufs],
                 [b[3].shape[2] for b in bufs])
    batch.sync()
    for k, (st, b) in enumerate(zip(stages, bufs)):
        got = (b[0].cpu().numpy().view(MBSTATE_DTYPE), b[1].cpu().numpy().view(MBCODE_DTYPE),
               (b[2].cpu().numpy(), b[3][0].cpu().numpy(), b[3][1].cpu().numpy()))
        _same_decisions(got, want[k], f"stream {k} {cases[k]}")
    batch.close()
    for st in stages:
        st.close()
