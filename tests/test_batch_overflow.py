"""One scene of a batch whose cell holds too many particles: it alone cannot be
read; the other scenes' states come back, in whatever order they are read.  On the
CPU with the engine on a stand-in of the CUDA runtime, on the GPU against the same
scenes without the bad one."""
import dataclasses

import numpy as np
import pytest

from host_engine import run_driver

DRIVER = r"""
#include "fake_cuda.h"
#include <cstdio>
using namespace sph;
int main() {
    SceneConfig c;
    c.box_mode = 1;
    c.h = 0.1f;
    Engine e(0);
    const uint32_t n = 300;
    int id[4];
    for (int& i : id) e.add_scene(c, n, &i);
    std::vector<float> p(3 * n), v(3 * n);
    std::printf("%d", e.step(2));
    fake::st.crowded = {e.scene(id[2])->part_base};   // full by the next prefix
    for (int round = 0; round < 2; ++round) {
        fake::st.sorts.clear();
        for (int i : {0, 1, 2, 3, 2, 1, 0}) std::printf(" %d", e.get_state(id[i], p.data(), nullptr, v.data(), n, false, true));
        int shared = 0;
        for (uint32_t t : fake::st.sorts) shared += t > 3u;   // three tiles to a scene
        std::printf(" %d", shared);
        if (round == 0) std::printf(" %d", e.step(1));
    }
    e.set_state(id[2], p.data(), nullptr, n);   // spread out again
    fake::st.crowded.clear();
    std::printf(" %d", e.step(1));
    for (int i : {0, 2}) std::printf(" %d", e.get_state(id[i], p.data(), nullptr, v.data(), n, false, true));
}
"""
OK, ECELL = 0, 7


def test_only_the_crowded_scene_fails():
    got = list(map(int, run_driver(DRIVER).split()))
    reads = [OK, OK, ECELL, OK, ECELL, OK, OK]
    shared = 1   # tried once, not with every read
    assert got == [OK] + reads + [shared] + [ECELL] + reads + [shared] + [OK, OK, OK]


@pytest.mark.gpu
def test_healthy_scenes_are_read_as_without_it():
    from libfluid_gb300 import _capi, workloads as W
    from libfluid_gb300.batch import Batch
    specs = [W.small_dam_break(seed=s) for s in (3, 4)]
    # half of 8,400 particles enter the others' cell in the first substep
    rng = np.random.default_rng(5)
    pos = rng.uniform(0.505, 0.545, (8400, 3)).astype(np.float32)
    pos[4200:, 0] = rng.uniform(0.5502, 0.5508, 4200)
    vel = np.zeros_like(pos)
    vel[4200:, 0] = -2.0
    bad = dataclasses.replace(specs[0], box=(1.0, 1.0, 1.0), h=0.05, blocks=[], extra_pos=pos, extra_vel=vel, dt=1e-3)

    b = Batch(0)
    ids = [b.add_scene(s) for s in (specs[0], bad, specs[1])]
    b.step(1)
    got = []
    for i in (0, 2, 1, 2, 0):
        if i == 1:
            with pytest.raises(_capi.SphError) as err:
                b.get_state(ids[i])
            assert err.value.code == _capi.SPH_ECELL
        else:
            got.append(b.get_state(ids[i]))
    with pytest.raises(_capi.SphError):
        b.step(1)
    got += [b.get_state(ids[i]) for i in (2, 0)]
    b.close()

    c = Batch(0)
    ids = [c.add_scene(s) for s in specs]
    c.step(1)
    want = [c.get_state(i) for i in ids]
    c.close()
    for g, w in zip(got, (0, 1, 1, 0, 1, 0)):
        for x, y in zip(g, want[w]):
            assert np.array_equal(x, y)
