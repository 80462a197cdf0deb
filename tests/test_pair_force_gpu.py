"""Forces of isolated particle pairs at every distance up to h, GPU against the
FP32 oracle.

One pair per site, sites 4 h apart, so that each force is a single pair's
term and nothing averages its error.  The distances cover both branches of the
cohesion kernel, pairs near r = h, where h - r is a few ulp of r, and pairs
beyond it.

Tolerance: 1e-4 of the pair's own magnitude, the bar of every force test; half
an ulp of r would be 3e-5 of h - r at r = h (1 - 2^-9).
"""
import numpy as np
import pytest

import oracle
from helpers import configure_gpu, configure_oracle, pair_scale, scaled_err
from libfluid_gb300 import workloads as W

H = 0.02


def _pairs(near, tension):
    rng = np.random.default_rng(11)
    sites = (np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) * 4 + 2) * H
    n = sites.shape[0]
    if near:    # 1 - (r/h)^2 from 2^-5 down to 2^-20, and just past h
        r = np.sqrt(1.0 - np.concatenate([2.0 ** -rng.uniform(5, 20, n - 32), -2.0 ** -rng.uniform(12, 22, 32)]))
    else:
        r = np.concatenate([rng.uniform(0.05, 1.0, n - 64), 0.5 + rng.uniform(-1e-3, 1e-3, 64)])
    d = rng.normal(size=(n, 3))
    d *= (r * H / np.linalg.norm(d, axis=1))[:, None]
    pos = np.concatenate([sites, sites + d]).astype(np.float32)
    vel = rng.uniform(-0.5, 0.5, pos.shape).astype(np.float32)
    return W.SceneSpec(box=(0.72, 0.72, 0.72), h=H, blocks=[], surface_tension=tension, extra_pos=pos, extra_vel=vel)


@pytest.mark.gpu
@pytest.mark.parametrize("tension", [0.0, 0.05])
@pytest.mark.parametrize("near", [False, True])
def test_isolated_pairs(near, tension):
    from libfluid_gb300 import FluidSystem
    spec = _pairs(near, tension)
    fs = FluidSystem(0)
    fs.debugEnable(True)
    configure_gpu(fs, spec)
    assert fs.advance(spec.dt, 1) == 1
    o32, o64 = (configure_oracle(oracle.Oracle(p), spec) for p in (32, 64))
    for o in (o32, o64):
        o.track_scales(True)
        o.advance(spec.dt, 1)
    assert np.array_equal(fs.debug("nbrcount"), o32.get("nbrcount"))
    for f in ("fpressure", "fviscosity") + (("ftension", "normal") if tension else ()):
        S = pair_scale(o32, o64, f)
        g, r = fs.debug(f), o32.get(f)
        # two pairs are so near r = h that p / rho^2 overflows, on both sides
        ok = np.isfinite(r).all(1)
        assert np.array_equal(np.isfinite(g).all(1), ok) and np.count_nonzero(~ok) <= 4
        e = scaled_err(g[ok], r[ok], S[ok])
        print(f"near={near} tension={tension} {f}: {e:.2e} of the pair")
        assert e < 1e-4, (f, e)
