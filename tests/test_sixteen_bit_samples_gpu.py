"""10-bit pictures come in 16-bit samples that are taken as they are given: costs are sums in 32 bits and squared errors in 64, so a
picture with larger samples than 1023 is analysed and decided as the oracle does it, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from ironav_b200.encoder import Encoder
from ironav_b200.inter import InterStage

pytestmark = pytest.mark.gpu

W, H = 96, 64


def _frames(top, n):
    """Noise over a moving texture, samples up to `top`."""
    rng = np.random.default_rng(top)
    base = rng.integers(0, top + 1, (H + 32, W + 32)).astype(np.int64)
    base = (base + np.roll(base, 1, 0) + np.roll(base, 1, 1) + np.roll(base, 2, 1)) // 4
    out = []
    for t in range(n):
        f = base[2 * t:2 * t + H, 3 * t:3 * t + W] + rng.integers(-top // 64 - 1, top // 64 + 2, (H, W))
        out.append(np.clip(f, 0, top).astype(np.uint16))
    return out


@pytest.mark.parametrize("top", [1023, 2047, 4095, 65535])
def test_analysis(oracle_lib, cuda_lib, top):
    frames = _frames(top, 3)
    got = []
    for lib in (oracle_lib, cuda_lib):
        st = InterStage(W, H, max_refs=2, nslices=2, lib=lib, bd=10)
        st.push_reference(frames[0])
        st.push_reference(frames[1])
        st.set_source(frames[2])
        st.begin_p_picture(30, nrefs_active=2, sub8=True)
        states, res = st.analyse_auto()
        out = [states, res]
        for form in range(4):
            assert lib.ironav_set_replay_form(st.ctx, form) == 0
            out.append(st.analyse_replay(got[0][0] if got else states))
        got.append(out)
        st.close()
    for what, a, b in zip(("states", "results", "form 0", "form 1", "form 2", "form 3"), *got):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("top", [1023, 65535])
def test_cabac_decision(oracle_lib, cuda_lib, top):
    y = _frames(top, 3)
    rng = np.random.default_rng(1)
    a, b = (Encoder(W, H, qp=30, keyint=30, nslices=2, refs=1, bd=10, scene_cut=False, lib=lib, cabac=True) for lib in (oracle_lib, cuda_lib))
    for t in range(3):
        c = [rng.integers(0, top + 1, (H // 2, W // 2)).astype(np.uint16) for _ in range(2)]
        assert a.encode(y[t], *c) == b.encode(y[t], *c), f"picture {t}"
        assert np.array_equal(a.codes, b.codes) and np.array_equal(a.states, b.states)
    a.close()
    b.close()
