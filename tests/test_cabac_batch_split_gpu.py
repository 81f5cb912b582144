"""The batched CABAC decision about as many slice bands as the chip has SMs: up to there a band has an SM to itself, beyond it two
bands share one. Every stream is decided as the oracle decides it on its own, on both sides and when bands wait for an SM, and one
band more than SMs does not cost the step a second wave."""
from __future__ import annotations

import numpy as np
import pytest

from ironav_b200.inter import MBCODE_DTYPE, MBSTATE_DTYPE, InterBatch, InterStage
from ironav_b200.synth import Sequence
from tests.test_decide import _same_decisions, decide_case

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


class _Step:
    """The streams' batch, their device buffers and one decision of all of them."""

    def __init__(self, stages):
        import torch

        self.stages = stages
        for st in stages:
            st.set_entropy(True, True)
            st.set_stream(torch.cuda.current_stream().cuda_stream)
        u8 = dict(dtype=torch.uint8, device="cuda")
        self.bufs = []
        for st in stages:
            px = dict(dtype=torch.int16 if st.bd > 8 else torch.uint8, device="cuda")
            self.bufs.append((torch.zeros(st.nmb * 72, **u8), torch.zeros(st.nmb * 1516, **u8), torch.zeros((st.mb_h * 16, st.mb_w * 16), **px),
                              torch.zeros((2, st.mb_h * 8, st.mb_w * 8), **px)))
        self.batch = InterBatch(stages)

    def decide(self):
        b = self.bufs
        self.batch.decide([x[0].data_ptr() for x in b], [x[1].data_ptr() for x in b], [x[2].data_ptr() for x in b], [x[2].shape[1] for x in b],
                          [x[3][0].data_ptr() for x in b], [x[3][1].data_ptr() for x in b], [x[3].shape[2] for x in b])

    def close(self):
        self.batch.close()
        for st in self.stages:
            st.close()


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("chains", ["sms", "sms + 1", "2 * sms + 1"])
def test_chains_about_the_sms(oracle_lib, cuda_lib, bd, chains):
    left = eval(chains, {"sms": _sms()})
    cases = []
    while left:
        n = min(10, left)  # 48 x 160: a stream of up to ten bands of one row
        cases.append(dict(size=(48, 160), nslices=n, qp=24 + len(cases) % 3, bd=bd, new_content=len(cases) % 3 == 2))
        left -= n
    step = _Step([decide_case(cuda_lib, threads=False, **kw)[0] for kw in cases])
    step.decide()
    step.batch.sync()
    want = {}
    for kw, st, b in zip(cases, step.stages, step.bufs):
        key = tuple(sorted((k, v) for k, v in kw.items()))
        if key not in want:
            o = decide_case(oracle_lib, **kw)[0]
            o.set_entropy(True, True)
            want[key] = o.decide_p_picture()
            o.close()
        px = MBSTATE_DTYPE, MBCODE_DTYPE, np.uint16 if bd > 8 else np.uint8
        got = (b[0].cpu().numpy().view(px[0]), b[1].cpu().numpy().view(px[1]),
               tuple(p.cpu().numpy().view(px[2]) for p in (b[2], b[3][0], b[3][1])))
        _same_decisions(got, want[key], str(kw))
    step.close()


def test_one_chain_more_than_sms_takes_no_second_wave(cuda_lib):
    """A second wave, or a slower form for the chains beyond the SMs, takes a step of equal bands half as long again; two bands on
    one SM slow each other down by less than a quarter."""
    import torch

    seq = Sequence.config("cif", 2, size=(320, 176))
    times = []
    for n in (_sms(), _sms() + 1):
        stages = []
        for _ in range(n):
            st = InterStage(320, 176, nslices=1, lib=cuda_lib)
            st.push_reference(seq.frame(0))
            st.push_reference_chroma(*seq.chroma(0))
            st.set_source(seq.frame(1))
            st.set_source_chroma(*seq.chroma(1))
            st.begin_p_picture(26)
            stages.append(st)
        step = _Step(stages)
        ms = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            step.decide()
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        times.append(sorted(ms[2:])[2])
        step.close()
    assert times[1] < 1.4 * times[0], times
