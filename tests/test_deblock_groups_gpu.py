"""The deblocking filter's row groups (4 macroblock rows a CTA, rings of 4 or 8 macroblocks between rows): pictures at the
edges of a group and of a ring, against the oracle, sample for sample."""
import numpy as np
import pytest

from ironav_b200.inter import InterStage
from ironav_b200.synth import dbk_planes, dbk_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("mb_w,mb_h", [(1, 4), (2, 5), (3, 8), (4, 9), (5, 3), (8, 12), (9, 13), (17, 6), (33, 17)])
def test_group_and_ring_edges(oracle_lib, cuda_lib, mb_w, mb_h, bd):
    rng = np.random.default_rng(mb_w * 100 + mb_h + bd)
    y, cb, cr = dbk_planes(rng, mb_w, mb_h, bd)
    mbs, slices = dbk_records(rng, mb_w, mb_h, 2, bd)
    if mb_w % 2:  # every edge filtered: no macroblock skips its pass or its wait
        mbs["slice"], mbs["inter"], mbs["keep"], mbs["t8x8"], mbs["qp"] = 1, 0, 0, 0, 35
        slices[:] = 0
    want, got = (InterStage(mb_w * 16, mb_h * 16, lib=lib, bd=bd).deblock(y, cb, cr, mbs, slices) for lib in (oracle_lib, cuda_lib))
    for g, w, name in zip(got, want, ("Y", "Cb", "Cr")):
        assert np.array_equal(g, w), f"{name} differs at {np.argwhere(g != w)[:4].tolist()}"
