"""The deblocking filter's and the CABAC writer's waits are bounded: with a poll limit that their first real waits run out of (a
host-side test hook), the call returns an error status, and the next one, with the default limit, is the oracle's."""
import numpy as np
import pytest

from ironav_b200.encoder import Encoder
from ironav_b200.inter import IronavError, InterStage
from ironav_b200.synth import Sequence, dbk_planes, dbk_records

pytestmark = pytest.mark.gpu

DEFAULT = 1 << 22


@pytest.mark.parametrize("mb_w,mb_h", [(120, 4), (120, 68)])
def test_deblocking(oracle_lib, cuda_lib, mb_w, mb_h):
    """One group of rows, which wait on shared memory alone, and many, which wait on one another. Every edge is filtered."""
    rng = np.random.default_rng(mb_h)
    planes = dbk_planes(rng, mb_w, mb_h, 8)
    mbs, slices = dbk_records(rng, mb_w, mb_h, 1, 8)
    mbs["slice"], mbs["inter"], mbs["keep"], mbs["t8x8"], mbs["qp"] = 1, 0, 0, 0, 35
    slices[:] = 0
    st = InterStage(mb_w * 16, mb_h * 16, lib=cuda_lib)
    assert cuda_lib.ironav_debug_wait_limit(st.ctx, 1) == 0
    try:
        with pytest.raises(IronavError) as e:
            for _ in range(20):  # a row that is ahead by luck does not wait
                st.deblock(*planes, mbs, slices)
        assert e.value.status == 100
    finally:
        assert cuda_lib.ironav_debug_wait_limit(st.ctx, DEFAULT) == 0
    want = InterStage(mb_w * 16, mb_h * 16, lib=oracle_lib).deblock(*planes, mbs, slices)
    for g, w in zip(st.deblock(*planes, mbs, slices), want):
        assert np.array_equal(g, w)


def test_cabac_writer(oracle_lib, cuda_lib):
    seq = Sequence.config("cif", 2)
    a, b = (Encoder(352, 288, qp=26, keyint=30, nslices=2, lib=lib, cabac=True) for lib in (oracle_lib, cuda_lib))
    f = [(seq.frame(t), *seq.chroma(t)) for t in range(2)]
    assert a.encode(*f[0]) == b.encode(*f[0])
    assert cuda_lib.ironav_debug_wait_limit(b.st.ctx, 1) == 0
    try:
        with pytest.raises(IronavError) as e:
            b.st.write_slices(True, 0, 0, b.codes)
        assert e.value.status == 13
    finally:
        assert cuda_lib.ironav_debug_wait_limit(b.st.ctx, DEFAULT) == 0
    assert a.encode(*f[1]) == b.encode(*f[1])
