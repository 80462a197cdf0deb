"""The candidate test in half precision (one thread per particle): it must find
every pair within h.  On the CPU its arithmetic, restated with numpy's halves, over
pairs just inside h at every place in the cell; on the GPU its passes against
those of several lanes per particle, whose test is exact, to the bit."""
import math

import numpy as np
import pytest


def near2(hc, cells):
    """DevParams::near2: the threshold in cells squared."""
    e = 2.0 ** -11 + 2.0 ** -12 + (2.0 * hc if hc > 1.001 else 1.0) * 2.0 ** -12 + (cells + 4) * 2.0 ** -22
    t = hc * hc * (1 + 0.0011) + 3.4642 * hc * e + 3 * e * e + 1e-5
    return min(t, 16.0)


def half_down(x):
    h = np.float16(x)
    return h if float(h) <= x else np.nextafter(h, np.float16(-np.inf))


def hits(pi, pj, inv_cell, t):
    """HalfScan on positions pi, pj (float32, n x 3) whose cells differ by at most one."""
    f32, f16 = np.float32, np.float16
    ui, uj = pi * f32(inv_cell), pj * f32(inv_cell)
    ci, cj = np.floor(ui), np.floor(uj)
    fi, fj = ui - ci, uj - cj
    gx, hx = ci[:, 0].astype(np.int64), cj[:, 0].astype(np.int64)
    second = ((gx - 1) & 2) != 0
    xj = np.where(second, fj[:, 0] + (((hx + 2) & 3) - 2).astype(f32), fj[:, 0] + ((hx & 3) - 2).astype(f32)).astype(f16)
    nx = (-(fi[:, 0] + (((gx + np.where(second, 2, 0)) & 3) - 2).astype(f32))).astype(f16)
    s = f32(0) * fi[:, 0] + np.float64(half_down(-t))
    d = [(xj.astype(np.float64) + nx).astype(f16)]
    for a in (1, 2):
        row = (cj[:, a] - ci[:, a]).astype(f32)      # -1, 0, 1: r % 3 - 1 and r / 3 - 1
        n = (row + f32(0.5) - fi[:, a]).astype(f16)
        d.append(((fj[:, a] - f32(0.5)).astype(f16).astype(np.float64) + n).astype(f16))
    for x in d:
        s = (x.astype(np.float64) ** 2 + s).astype(f16).astype(np.float64)   # one rounding, as the fused operation
    return s < 0


# h in cells, cells along the longest side
@pytest.mark.parametrize("hc", [1.0, 0.37, 0.05, 1.7])
@pytest.mark.parametrize("cells", [8, 100, 1000, 40000])
def test_finds_every_pair_within_h(hc, cells):
    rng = np.random.default_rng([int(100 * hc), cells])
    cell = np.float32(0.0173)
    inv = np.float32(1.0) / cell
    h = np.float32(hc) * cell
    n = 100_000
    # first particles anywhere, some on cell boundaries; the second at h (1 - up to 1e-2, mostly far less) from them,
    # directions of any kind, some along the axes
    pi = (rng.random((n, 3)) * (cells - 4) + 2) * float(cell)
    edge = rng.random((n, 3)) < 0.1
    pi = np.where(edge, np.round(pi / float(cell)) * float(cell) + rng.choice([-1e-6, 0.0, 1e-6], (n, 3)) * float(cell), pi)
    v = rng.normal(size=(n, 3)) * np.where(rng.random((n, 3)) < 0.2, 1e-3, 1.0)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    r = float(h) * (1 - 10.0 ** rng.uniform(-8, -2, (n, 1)))
    pi, pj = pi.astype(np.float32), (pi + v * r).astype(np.float32)
    d = pi - pj
    rr = (d * d).sum(1, dtype=np.float32)
    near = np.abs(np.floor(pi * inv) - np.floor(pj * inv)).max(1) <= 1
    pick = (rr <= h * h) & near & (pj > 0).all(1)
    assert pick.sum() > n // 10
    assert hits(pi[pick], pj[pick], inv, near2(float(h) * float(inv), cells)).all()


def test_few_pairs_beyond_h():
    """What lists grow by: below 1% of the volume at 100 cells."""
    assert math.sqrt(-float(half_down(-near2(1.0, 100)))) ** 3 < 1.01


def _run(box, h, pos, variant, steps=3):
    from libfluid_gb300 import workloads as W
    from libfluid_gb300.batch import Batch
    spec = W.SceneSpec(box=box, h=h, blocks=[], mass=1000.0 * (0.5 * h) ** 3, particle_size=0.25 * h,
                       surface_tension=0.05, dt=1e-5, extra_pos=pos, extra_vel=np.zeros_like(pos))
    b = Batch(0)
    b.set_exec(tile=128, variant=variant)
    sid = b.add_scene(spec)
    out = []
    for _ in range(steps):
        b.step(1)
        out += b.get_state(sid)
    b.close()
    return out


# boxes of few and of many cells along each axis, in any place modulo four
@pytest.mark.gpu
@pytest.mark.parametrize("box", [(5, 7, 6), (61, 3, 3), (3, 64, 4), (4, 3, 67), (900, 2, 2)])
def test_same_pairs_as_the_exact_scan(box):
    h = 0.02
    rng = np.random.default_rng(int(sum(box)))
    m = 700
    a = rng.random((m, 3)) * (np.asarray(box) - 0.02) * h + 0.01 * h
    v = rng.normal(size=(4, m, 3))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    r = h * (1 + rng.choice([-1e-3, -1e-6, -1e-7, 0.0, 1e-7, 1e-6, 1e-3], (4, m, 1)))
    pos = np.concatenate([a, (a + v * r).reshape(-1, 3)])
    pos = np.clip(pos, 0.01 * h, (np.asarray(box) - 0.01) * h).astype(np.float32)
    box = tuple(float(b * h) for b in box)
    one, lanes = _run(box, h, pos, 31), _run(box, h, pos, 63)
    assert all(np.isfinite(x).all() for x in lanes)
    for x, y in zip(one, lanes):
        assert np.array_equal(x, y)
