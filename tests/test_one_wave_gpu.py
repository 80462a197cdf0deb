"""The builds of launches that the GPU holds at once (116,736 threads) against the
others', which a persistent launch runs at any size: bit-identical states, with
and without surface tension, with short, full and overflowing neighbour lists."""
import numpy as np
import pytest

from libfluid_gb300 import workloads as W
from libfluid_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _run(spec, tile, persistent, steps):
    b = Batch(0)
    b.set_exec(tile=tile, variant=31, persistent=persistent)
    sid = b.add_scene(spec)
    b.step(steps)
    out = b.get_state(sid)
    b.close()
    return out


# particles: 1, 77, 2,730, 116,736 (all of the limit), 116,850
@pytest.mark.parametrize("tension", [0.0, 0.05])
@pytest.mark.parametrize("dims, spacing", [((1, 1, 1), 0.01), ((7, 11, 1), 0.01), ((13, 14, 15), 0.01),
                                           ((13, 14, 15), 0.0078), ((13, 14, 15), 0.005), ((48, 38, 64), 0.01),
                                           ((50, 41, 57), 0.01)])
def test_builds_bit_identical(dims, spacing, tension):
    nx, ny, nz = dims
    lat = W.Lattice(lo=(0.0, 0.0, 0.0), spacing=spacing, nx=nx, ny=ny, nz=nz, jitter=0.2 * spacing, seed=4,
                    vel=(0.1, -0.2, 0.05))
    spec = W.SceneSpec(box=tuple(max(1.3 * k * spacing, 0.04) for k in dims), h=0.02, blocks=[lat],
                       mass=1000.0 * spacing ** 3, particle_size=0.5 * spacing, surface_tension=tension, dt=2e-4)
    for tile in (128,) if nx > 40 else (64, 128, 256):
        for x, y in zip(_run(spec, tile, 0, 2), _run(spec, tile, 4, 2)):
            assert np.array_equal(x, y)
