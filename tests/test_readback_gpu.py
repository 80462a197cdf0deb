"""Reading states: exports just below and above the size that goes through pinned
memory, against the exact snapshot; and scenes of a batch read one after the
other (one scene's prefix, then one over all scenes that the next step starts
from), against the same batch read only at the end."""
import numpy as np
import pytest

from helpers import configure_gpu, snapshot_state
from libfluid_gb300 import FluidSystem
from libfluid_gb300 import workloads as W
from libfluid_gb300.batch import Batch

pytestmark = pytest.mark.gpu


# 36 bytes a particle, 384 KiB: 10,922 particles go through pinned memory, 10,923 do not
@pytest.mark.parametrize("n", [1, 1000, 10922, 10923])
@pytest.mark.parametrize("sync", [True, False])
def test_export_sizes(n, sync):
    lat = W.Lattice(lo=(0.0, 0.0, 0.0), spacing=0.01, nx=1, ny=1, nz=1, jitter=0.0)
    spec = W.SceneSpec(box=(0.5, 0.5, 0.5), h=0.02, blocks=[lat])
    rng = np.random.default_rng(3)
    pos = rng.uniform(0.01, 0.49, (n, 3)).astype(np.float32)
    fs = FluidSystem(0)
    configure_gpu(fs, spec, pos=pos, vel=np.zeros_like(pos))
    for _ in range(3):
        fs.advance(spec.dt, 1) if sync else fs.advanceAsync(spec.dt, 1)
    p, c, v = fs.exportToData()
    sp, sv, _ = snapshot_state(fs)
    assert np.array_equal(p, sp) and np.array_equal(v, sv)
    assert np.all(np.isfinite(c)) and (c.sum(1) > 0.99).all()
    fs.close()


def _batch():
    b = Batch(0)
    return b, [b.add_scene(s) for s in W.batch_manifest(num_scenes=6, seed=71, nmin=300, nmax=30000)]


def test_batch_reads_between_steps():
    b, ids = _batch()
    b.step(3)
    mid = [b.get_state(i) for i in ids]
    again = [b.get_state(i) for i in reversed(ids)][::-1]
    b.step(2)
    b.get_state(ids[2])
    extra = b.add_scene(W.small_dam_break(seed=2))   # the layout changes between two reads
    late = [b.get_state(i) for i in ids]
    b.step(1)
    end = [b.get_state(i) for i in ids + [extra]]
    b.close()
    c, ids = _batch()
    c.step(3)
    lone = c.get_state(ids[4])
    c.step(2)
    want = c.get_state(ids[3])
    c.add_scene(W.small_dam_break(seed=2))
    c.step(1)
    last = [c.get_state(i) for i in c.scenes]
    c.close()
    for x, y in [(mid, again), ([mid[4]], [lone]), ([late[3]], [want]), (end, last)]:
        for s, t in zip(x, y):
            for p, q in zip(s, t):
                assert np.array_equal(p, q)
