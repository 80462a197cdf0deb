"""The autotuner sweeps the bit of several lanes per particle for every launch that
takes it: crowded ones take it up to a higher limit."""
import dataclasses

import pytest

from libfluid_gb300 import autotune, workloads as W
from test_autotune_cpu import _define

TYPES = "libfluid_gb300/csrc/sph_types.h"


def test_limits_match_the_library():
    assert autotune.CROWDED_MAX == _define(TYPES, "SPH_CROWDED8_MAX")
    assert autotune.CROWDED_NEIGHBOURS == _define(TYPES, "SPH_CROWDED_NBRS")


def test_lanes_bit_swept_for_crowded_launches():
    assert autotune.variants_for(autotune.CROWDED_MAX, 0, True) == tuple(range(64))
    assert autotune.variants_for(autotune.CROWDED_MAX + 1, 0, True) == tuple(range(32))
    assert autotune.variants_for(autotune.CROWDED_MAX, 2, True) == tuple(range(32))
    assert autotune.variants_for(autotune.CROWDED_MAX, 0) == tuple(range(32))


# a mass of 1/79 or 1/81 of the fluid within h
@pytest.mark.parametrize("cube", [0, 25])
@pytest.mark.parametrize("neighbours, want", [(79, False), (81, True)])
def test_crowded_scenes(cube, neighbours, want):
    s = W.small_dam_break()
    h = 1.0 / cube if cube else s.h
    s = dataclasses.replace(s, unit_cube_res=cube, mass=4.18879 * h ** 3 * s.rest_density / neighbours)
    assert autotune.crowded([s, s]) is want
