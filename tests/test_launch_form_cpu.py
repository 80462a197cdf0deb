"""The form in which the engine launches its passes (csrc/launch_form.h): the
passes of one substep, from captured graphs or not, always share one.  The engine
runs on a stand-in of the CUDA runtime, so nothing here touches a GPU.

A parameter change (mass, rest density) moves a scene of some ten thousand
particles across the line between one and eight lanes per particle, which store
positions, lists and copies differently; an export's passes run ahead are launched
outside the graphs."""
import pytest

from host_engine import run_driver

DRIVER = r"""
#include "fake_cuda.h"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace sph;

static SceneConfig config(bool crowded, bool tension) {
    SceneConfig c;
    c.box_mode = 1;
    c.lx = c.ly = c.lz = 1.f;
    c.h = 0.1f;
    c.rest_density = 1000.f;
    c.mass = 1000.f * 4.19e-3f / (crowded ? 200.f : 33.f);   // neighbours at rest density
    c.surface_tension = tension ? 0.05f : 0.f;
    return c;
}
static void frame(Engine& e, int id, uint32_t n) {
    std::vector<float> pos(3 * n), vel(3 * n);
    e.step(1);
    e.get_state(id, pos.data(), nullptr, vel.data(), n);
}
// Frames with the mass changed between them; the passes run ahead are taken.
static void frames(uint32_t n, bool tension) {
    Engine e(0);
    int id = 0;
    e.add_scene(config(true, tension), n, &id);
    for (int i = 0; i < 12; ++i) {
        frame(e, id, n);
        if (i % 3 == 2) e.set_config(id, config((i / 3) % 2 != 0, tension));
    }
}
// Any calls in any order.
static void calls(uint32_t n, uint32_t seed) {
    std::mt19937 rng(seed);
    Engine e(0);
    std::vector<int> ids(1);
    bool crowded = false, tension = false;
    e.add_scene(config(false, false), n, &ids[0]);
    std::vector<float> a(3 * n), b(3 * n);
    std::vector<float4> state(3 * n);
    for (int i = 0; i < 300; ++i) {
        const int id = ids[rng() % ids.size()];
        const uint32_t m = e.scene(id)->n;
        switch (rng() % 13) {
            case 0: case 1: e.step(1); break;
            case 2: e.step(3); break;
            case 3: case 4: case 5: e.get_state(id, a.data(), nullptr, b.data(), m, false, rng() % 2 == 0); break;
            case 6: crowded = !crowded; e.set_config(id, config(crowded, tension)); break;
            case 7: tension = rng() % 2; e.set_config(id, config(crowded, tension)); break;
            case 8: {
                ExecConfig x = e.exec();
                x.variant = rng() % 4 ? SPH_VARIANT_DEFAULT : 31u;
                x.tile = 64u << (rng() % 3);
                x.persistent = rng() % 4 ? 0u : 2u;
                e.set_exec(x);
                break;
            }
            case 9: e.set_use_graph(rng() % 4 != 0); break;
            case 10: e.set_profiling(rng() % 4 == 0); break;
            case 11: e.set_deferred_xsph(rng() % 4 != 0); break;
            case 12:
                if (ids.size() > 1 && rng() % 2) {
                    e.remove_scene(ids.back());
                    ids.pop_back();
                } else if (ids.size() < 4) {
                    ids.push_back(0);
                    e.add_scene(config(crowded, tension), 1u + rng() % n, &ids.back());
                } else {
                    e.save_state(id, state.data(), m);
                }
        }
    }
}
int main(int, char** argv) {
    const uint32_t n = (uint32_t)std::atoi(argv[1]);
    frames(n, false);
    frames(n, true);
    for (uint32_t s = 0; s < 20; ++s) calls(n, s);
    std::printf("%llu %llu %zu %llu\n", (unsigned long long)fake::st.substeps, (unsigned long long)fake::st.mixed,
                fake::st.lanes.size(), (unsigned long long)fake::st.null_writes);
}
"""


# particles that the change takes from one to eight lanes and back; from four to eight; always eight
@pytest.mark.parametrize("n, forms", [(40_000, 2), (20_000, 2), (2_000, 2)])
def test_passes_of_a_substep_share_one_form(n, forms):
    substeps, mixed, lanes, bad = map(int, run_driver(DRIVER, n).split())
    assert substeps > 1000 and lanes >= forms
    assert mixed == 0 and bad == 0


ONE_WAVE = r"""
#include "launch_form.h"
#include <cstdio>
#include <initializer_list>
int main() {
    for (uint32_t sms : {152u, 148u, 1u})
        for (uint32_t tiles : {sms * 6u, sms * 6u + 1u})
            for (bool persistent : {false, true})
                std::printf("%d ", sph::launch_form(tiles, 128u, persistent, 31u, false, false, false, sms).one_wave);
}
"""


def test_one_wave_follows_the_gpu():
    """Six blocks of 128 threads to an SM, and one block more; not when persistent."""
    assert run_driver(ONE_WAVE).split() == ["1", "0", "0", "0"] * 3


LANES = r"""
#include "engine.h"
#include <cstdio>
#include <initializer_list>
int main() {
    using namespace sph;
    auto lanes = [](uint32_t scenes, uint32_t n, uint32_t tile, bool crowded, uint32_t variant = SPH_VARIANT_DEFAULT) {
        const uint32_t tiles = scenes * ((n + tile - 1u) / tile);
        std::printf("%u ", launch_form(tiles, tile, false, variant, crowded, false, false, 152u).lanes);
    };
    for (uint32_t tile : {64u, 128u, 256u})   // one scene at the limits
        for (uint32_t n : {1u, 14336u, 14337u, 34816u, 34817u}) lanes(1, n, tile, false);
    for (uint32_t n : {34817u, 61440u, 61441u}) lanes(1, n, 128, true);
    lanes(1, 100, 128, false, 31);
    for (uint32_t scenes : {112u, 113u, 272u, 273u, 14000u, 100000u}) lanes(scenes, 1, 128, false);
}
"""


def test_lanes_go_by_the_tiles():
    """A scene alone by its particles; many tiny scenes by the threads launched for
    them (one lane where most blocks would have no particle)."""
    assert run_driver(LANES).split() == ["8", "8", "4", "4", "1"] * 3 + ["8", "8", "1"] + ["1"] + [
        "8", "4", "4", "1", "1", "1"]
