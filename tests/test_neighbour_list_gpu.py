"""The neighbour list around its limits: particles with about as many
neighbours as it holds (68), more, and cell rows longer than its offsets reach
(128 candidates), against the CPU oracle and over its two builders.

Tolerances are those of the crowded-cell tests: integer fields bit-exact,
density within 1e-5, forces and normals within 1e-4 of the magnitude of their
pair terms and no further from FP64 than twice the FP32 oracle.
"""
import dataclasses

import numpy as np
import pytest

import oracle
from helpers import check_vector_field, configure_gpu, configure_oracle, pair_scale, rel_err
from libfluid_gb300 import FluidSystem
from test_parity_crowded_gpu import crowded

pytestmark = pytest.mark.gpu

# spacing -> neighbours of an inner particle: 58, 68, 160, 268 (rows of 192 candidates)
SPACINGS = [0.00833, 0.0079, 0.006, 0.005]


def _scene(spacing):
    return dataclasses.replace(crowded(spacing, 20, seed=9), surface_tension=0.05)


@pytest.mark.parametrize("spacing", SPACINGS)
def test_list_limits_match_oracle(spacing):
    spec = _scene(spacing)
    fs = FluidSystem(0)
    fs.debugEnable(True)
    configure_gpu(fs, spec)
    o32, o64 = (configure_oracle(oracle.Oracle(p), spec) for p in (32, 64))
    for o in (o32, o64):
        o.track_scales(True)
        o.advance(spec.dt, 1)
    assert fs.advance(spec.dt, 1) == 1
    for f in ("hash", "perm", "nbrcount"):
        assert np.array_equal(fs.debug(f), o32.get(f)), f
    print(f"{spacing}: up to {fs.debug('nbrcount').max()} neighbours")
    assert rel_err(fs.debug("density"), o32.get("density"), 1.0) < 1e-5
    for f in ("fpressure", "fviscosity", "ftension", "normal"):
        check_vector_field(f"{spacing} {f}", fs.debug(f), o32.get(f), o64.get(f), pair_scale(o32, o64, f), 1e-4)
    fs.close()


@pytest.mark.parametrize("spacing", SPACINGS)
@pytest.mark.parametrize("tile", [64, 256])
def test_split_builds_the_same_list(spacing, tile):
    """Three threads' lists appended against one thread's: bit-identical."""
    spec = _scene(spacing)
    out = []
    for variant in (31, 63):
        fs = FluidSystem(0)
        configure_gpu(fs, spec)
        fs.setExec(tile=tile, variant=variant)
        for _ in range(3):
            fs.advance(spec.dt, 1)
        out.append(fs.exportToData())
        fs.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
