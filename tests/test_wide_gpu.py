"""Several lanes per particle in the neighbour passes (small launches) against
one thread per particle (variant without bit 0x20): bit-identical states, from
one particle to the limits of eight and of four lanes, crowded or not, with and
without surface tension, and for a batch of scenes that share a launch."""
import numpy as np
import pytest

from helpers import configure_gpu
from libfluid_gb300 import FluidSystem
from libfluid_gb300 import workloads as W
from libfluid_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _run(specs, variant, tile, steps=3):
    b = Batch(0)
    b.set_exec(tile=tile, variant=variant)
    ids = [b.add_scene(s) for s in specs]
    b.step(steps)
    out = [b.get_state(i) for i in ids]
    b.close()
    return out


def _block(nx, ny, nz, tension, spacing=0.01, h=0.02, seed=5):
    lat = W.Lattice(lo=(0.0, 0.0, 0.0), spacing=spacing, nx=nx, ny=ny, nz=nz, jitter=0.2 * spacing, seed=seed,
                    vel=(0.1, -0.2, 0.05))
    box = tuple(max(1.3 * k * spacing, 2 * h) for k in (nx, ny, nz))
    return W.SceneSpec(box=box, h=h, blocks=[lat], mass=1000.0 * spacing ** 3, particle_size=0.5 * spacing,
                       surface_tension=tension, dt=2e-4)


def _same(specs, tile=128):
    for x, y in zip(_run(specs, 31, tile), _run(specs, 63, tile)):
        for a, b in zip(x, y):
            assert np.array_equal(a, b)


# particles: 1, 15, 17, 1001, 14,336 and 14,382 (eight lanes, then four), 34,816 and 34,848 (four, then one)
@pytest.mark.parametrize("tension", [0.0, 0.05])
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 3, 5), (1, 1, 17), (7, 11, 13), (28, 32, 16), (17, 18, 47),
                                  (32, 34, 32), (32, 33, 33)])
def test_lanes_bit_identical(dims, tension):
    _same([_block(*dims, tension)])


@pytest.mark.parametrize("tile", [64, 256])
def test_lanes_at_other_tiles(tile):
    _same([_block(9, 10, 11, 0.03), _block(26, 27, 25, 0.0, seed=6)], tile)


# about 113 neighbours: eight lanes to 61,440 particles
@pytest.mark.parametrize("dims", [(20, 20, 20), (35, 36, 34)])
def test_crowded_lanes(dims):
    _same([_block(*dims, 0.04, spacing=0.00667)])


def test_batch_of_small_scenes():
    _same([_block(3 + k, 4, 5, 0.01 * (k % 2), seed=k) for k in range(40)])


# neighbours of an inner particle around the 92 that a list built by several lanes
# holds, far above, and with cell rows past its offsets (of 128): the rest is found
# by testing candidates again, in the same order
@pytest.mark.parametrize("spacing", [0.0078, 0.00714, 0.0066, 0.006, 0.005, 0.0042])
def test_past_the_list(spacing):
    _same([_block(13, 14, 15, 0.04, spacing=spacing)])


def test_past_the_list_at_the_limit():
    _same([_block(39, 39, 40, 0.03, spacing=0.0064)])      # 60,840 particles
    _same([_block(40, 40, 39, 0.03, spacing=0.0064)])      # 62,400: one thread each


def test_past_the_list_for_some():
    """Particles of one warp whose lists end early and not."""
    _same([_block(2 + k, 3, 5, 0.02, spacing=0.005 if k % 2 else 0.01, seed=k) for k in range(20)]
          + [_block(20, 20, 20, 0.0, spacing=0.005)])


@pytest.mark.parametrize("spacing", [0.00714, 0.005])
def test_past_the_list_with_a_pass_per_substep(spacing):
    """XSPH by its own pass: a shorter list, the axis copies in other rows."""
    out = []
    for variant in (31, 63):
        b = Batch(0)
        b.set_exec(tile=128, variant=variant)
        b.set_deferred_xsph(False)
        sid = b.add_scene(_block(13, 14, 15, 0.04, spacing=spacing))
        b.step(3)
        out.append(b.get_state(sid))
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dims", [(9, 10, 11), (33, 34, 33)])
def test_lanes_switched_between_steps(dims):
    """A blocking step leaves the next substep's density pass done; one that follows
    with other lanes does not read what that pass stored for its own."""
    spec = _block(*dims, 0.05)
    out = []
    for variants in ((31, 31, 31), (63, 31, 63), (31, 63, 31)):
        fs = FluidSystem(0)
        configure_gpu(fs, spec)
        for v in variants:
            fs.setExec(tile=128, variant=v)
            fs.advance(spec.dt, 1)
        n = spec.n
        got = [np.zeros((n, 3), np.float32) for _ in range(3)]
        fs.exportToData(*got)
        out.append(got)
        fs.close()
    for got in out[1:]:
        for x, y in zip(out[0], got):
            assert np.array_equal(x, y)
