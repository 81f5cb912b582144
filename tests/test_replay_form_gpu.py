"""Replay mode's kernel as the library chooses it, by the picture's size, depth and search: below and above each line of the
choice, the results are those of the 8-lane groups (which tests/test_parity_gpu.py compares with the oracle)."""
import numpy as np
import pytest

from ironav_b200.inter import InterStage
from ironav_b200.synth import Sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("size", [(64, 48), (848, 480), (1280, 720), (1920, 1088), (2560, 1440), (3840, 2160)])
def test_chosen_form(cuda_lib, size, bd):
    w, h = size
    seq = Sequence.config("1080p", 2, size=size)
    frame = seq.frame if bd == 8 else seq.frame10
    results = []
    for form in (None, 0):
        st = InterStage(w, h, nslices=2, lib=cuda_lib, bd=bd)
        if form is not None:
            assert cuda_lib.ironav_set_replay_form(st.ctx, form) == 0
        st.push_reference(frame(0))
        st.set_source(frame(1))
        got = []
        for mode in ({}, {"fast": True}, {"sub8": True}):
            st.begin_p_picture(27 + 6 * (bd - 8), **mode)
            states, _ = st.analyse_auto()
            got.append(st.analyse_replay(states))
        results.append(got)
        st.close()
    for chosen, groups in zip(*results):
        assert np.array_equal(chosen, groups)
