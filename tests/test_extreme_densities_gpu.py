"""Values that the pair loop's short forms do not hold for: densities whose square
or its reciprocal leaves the normal numbers, and infinite sound speeds of pairs that
do not approach.  One thread and several lanes per particle against the FP32 oracle.

Tolerance: 1e-4 of the pair terms' magnitude, the bar of every force test."""
import numpy as np
import pytest

import oracle
from helpers import SCALE_FIELD, configure_gpu, configure_oracle, scaled_err
from libfluid_gb300 import workloads as W


def _check(spec, variant):
    from libfluid_gb300 import FluidSystem
    fs = FluidSystem(0)
    fs.setExec(tile=128, variant=variant)
    fs.debugEnable(True)
    configure_gpu(fs, spec)
    o = configure_oracle(oracle.Oracle(32), spec)
    o.track_scales(True)
    o.advance(spec.dt, 1)
    assert fs.advance(spec.dt, 1) == 1
    assert np.array_equal(fs.debug("nbrcount"), o.get("nbrcount"))
    for f in ("fpressure", "fviscosity"):
        r, g = o.get(f), fs.debug(f)
        assert np.isfinite(r).all() and np.isfinite(g).all()
        assert scaled_err(g, r, o.get(SCALE_FIELD[f])) < 1e-4, f
    fs.close()


# rho^2 subnormal, its reciprocal subnormal, rho^2 infinite; and an ordinary one
@pytest.mark.gpu
@pytest.mark.parametrize("variant", [31, 63])
@pytest.mark.parametrize("rest", [8e-20, 1.2e19, 1e20, 1000.0])
def test_densities_of_any_size(rest, variant):
    lat = W.Lattice(lo=(0.1, 0.1, 0.1), spacing=0.01, nx=9, ny=10, nz=11, jitter=2e-3, seed=5)
    vel = np.random.default_rng(5).uniform(-0.5, 0.5, (lat.n, 3)).astype(np.float32)
    _check(W.SceneSpec(box=(0.4, 0.4, 0.4), h=0.02, blocks=[], rest_density=rest, mass=rest * 1e-6,
                       extra_pos=lat.positions(), extra_vel=vel), variant)


# pairs exactly one h apart, so that their densities vanish and with gamma < 1 their sound speeds are infinite
@pytest.mark.gpu
@pytest.mark.parametrize("variant", [31, 63])
def test_infinite_sound_speeds(variant):
    h = 2.0 ** -5
    sites = (np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) * 4 + 2) * h
    d = np.zeros_like(sites)
    d[np.arange(len(d)), np.arange(len(d)) % 3] = h
    pos = np.concatenate([sites, sites + d]).astype(np.float32)
    vel = np.concatenate([-d, d]).astype(np.float32)   # apart
    _check(W.SceneSpec(box=(36 * h,) * 3, h=h, blocks=[], gamma=0.5, extra_pos=pos, extra_vel=vel), variant)
