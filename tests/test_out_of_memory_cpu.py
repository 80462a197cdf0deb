"""Device allocations that fail while the engine grows: the call reports it, what was
there goes on, and no launch is given an array that was freed on the way.  The engine
runs on a stand-in of the CUDA runtime whose allocations fail at a chosen point."""
import pytest

from host_engine import run_driver

DRIVER = r"""
#include "fake_cuda.h"
#include <cstdio>
#include <cstdlib>
using namespace sph;
static SceneConfig config(float size) {
    SceneConfig c;
    c.box_mode = 1;
    c.lx = c.ly = c.lz = size;
    c.h = 0.1f;
    return c;
}
// A growth of `kind` with `count` failing allocations from the at-th on.
static bool grow(int kind, int at, int count, bool graph, bool debug) {
    Engine e(0);
    e.set_use_graph(graph);
    int a = 0, b = 0;
    if (e.add_scene(config(1.f), 1000, &a)) return false;
    if (debug) e.debug_enable(true);
    std::vector<float> p(3 * 9000), v(3 * 9000);
    if (e.step(2) || e.get_state(a, p.data(), nullptr, v.data(), 1000)) return false;
    fake::st.mallocs = 0;
    fake::st.fail_from = at;
    fake::st.fail_count = count;
    int rc = 0;
    switch (kind) {
        case 0: rc = e.add_scene(config(1.f), 9000, &b); break;     // slots
        case 1: rc = e.set_config(a, config(9.f)); break;           // cells
        case 2: rc = e.reserve(20000, 100000); break;
        case 3:                                                     // tables
            for (int i = 0; i < 40 && rc == 0; ++i) rc = e.add_scene(config(0.3f), 5, &b);
            break;
    }
    const int stepped = e.step(1), read = e.get_state(a, p.data(), nullptr, v.data(), 1000);
    const bool hit = fake::st.mallocs > (uint64_t)at;
    fake::st.fail_from = -1;
    // an error or the step, nothing else; and with memory again everything works
    for (int r : {rc, stepped, read})
        if (r != ENG_OK && r != ENG_ENOMEM) { std::printf("kind %d at %d: %d %d %d %s\n", kind, at, rc, stepped, read, e.last_error().c_str()); std::exit(1); }
    if (rc && kind == 0) rc = e.add_scene(config(1.f), 9000, &b);
    if (e.step(2) || e.get_state(a, p.data(), nullptr, v.data(), 1000) ||
        (kind == 0 && e.get_state(b, p.data(), nullptr, v.data(), 9000, false, true))) {
        std::printf("kind %d at %d: %s\n", kind, at, e.last_error().c_str());
        std::exit(1);
    }
    return hit;
}
int main(int, char** argv) {
    const int kind = std::atoi(argv[1]), count = std::atoi(argv[2]);
    int points = 0;
    for (bool graph : {true, false})
        for (bool debug : {false, true})
            for (int at = 0; grow(kind, at, count, graph, debug); ++at) ++points;
    std::printf("%d %llu %llu %llu", points, (unsigned long long)fake::st.bad_arrays,
                (unsigned long long)fake::st.null_writes, (unsigned long long)fake::st.mixed);
}
"""


# slots, cells, both reserved, scene tables; one allocation that fails, or all from there on
@pytest.mark.parametrize("kind, least", [(0, 40), (1, 12), (2, 40), (3, 20)])
@pytest.mark.parametrize("count", [1, 1000])
def test_growth_without_memory(kind, least, count):
    out = run_driver(DRIVER, kind, count).split()
    assert out[1:] == ["0", "0", "0"]
    assert int(out[0]) >= least
