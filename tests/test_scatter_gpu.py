"""The sort's scatter, which takes four tiles to a block: cell order against the
CPU oracle for tile counts around a multiple of four, one scene or several (whose
last tiles are part full).  Integer fields, bit-exact."""
import numpy as np
import pytest

import oracle
from helpers import configure_gpu, configure_oracle
from libfluid_gb300 import FluidSystem
from libfluid_gb300 import workloads as W
from libfluid_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _spec(nx, ny, nz, seed=3):
    lat = W.Lattice(lo=(0.0, 0.0, 0.0), spacing=0.01, nx=nx, ny=ny, nz=nz, jitter=0.002, seed=seed,
                    vel=(0.3, -0.2, 0.1))
    box = tuple(max(0.013 * k, 0.04) for k in (nx, ny, nz))
    return W.SceneSpec(box=box, h=0.02, blocks=[lat], mass=1e-3, particle_size=0.005, dt=2e-4)


# tiles of 64 particles: 1, 3 (the last of one), 4, 5 (one), 7, 8, 9
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 43, 1), (4, 8, 8), (257, 1, 1), (7, 8, 8), (8, 8, 8), (19, 3, 10)])
def test_cell_order_matches_oracle(dims):
    spec = _spec(*dims)
    fs = FluidSystem(0)
    fs.debugEnable(True)
    configure_gpu(fs, spec)
    fs.setExec(tile=64)
    o = configure_oracle(oracle.Oracle(32), spec)
    for _ in range(2):
        fs.advance(spec.dt, 1)
        o.advance(spec.dt, 1)
        for f in ("hash", "perm"):
            assert np.array_equal(fs.debug(f), o.get(f)), f
    fs.close()


@pytest.mark.parametrize("count", [2, 3, 5])
def test_scenes_share_a_block(count):
    """Scenes of one launch against the same scenes alone."""
    specs = [_spec(3 + 2 * k, 5, 7, seed=k) for k in range(count)]
    b = Batch(0)
    b.set_exec(tile=64, variant=31)
    ids = [b.add_scene(s) for s in specs]
    b.step(3)
    for s, i in zip(specs, ids):
        one = Batch(0)
        one.set_exec(tile=64, variant=31)
        k = one.add_scene(s)
        one.step(3)
        for x, y in zip(b.get_state(i), one.get_state(k)):
            assert np.array_equal(x, y)
        one.close()
    b.close()
