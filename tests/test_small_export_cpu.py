"""Exports small enough for the kernels to write into pinned host memory, with the
engine on a stand-in of the CUDA runtime."""
import pytest

from host_engine import run_driver

DRIVER = r"""
#include "fake_cuda.h"
#include <cstdio>
#include <cstdlib>
using namespace sph;
int main(int, char** argv) {
    const uint32_t n = (uint32_t)std::atoi(argv[1]);
    fake::st.pinned_limit = std::atoi(argv[2]) ? 4096u : ~(size_t)0;
    SceneConfig c;
    c.box_mode = 1;
    c.h = 0.1f;
    Engine e(0);
    int id;
    int rc = e.add_scene(c, n, &id);
    std::vector<float> p(3 * n), q(3 * n), v(3 * n);
    int wrong = 0;
    for (int i = 0; i < 6; ++i) {
        rc |= e.step(1, i % 3 != 2);   // blocking: the prefix runs behind it
        p.assign(3 * n, -1.f); q.assign(3 * n, -1.f); v.assign(3 * n, -1.f);
        rc |= e.get_state(id, p.data(), q.data(), v.data(), n);
        for (uint32_t k = 0; k < 3 * n; ++k)
            wrong += p[k] != fake::kPosition || q[k] != fake::kPosition || v[k] != fake::kVelocity;
    }
    std::printf("%d %d %llu\n", rc, wrong, (unsigned long long)fake::st.null_writes);
}
"""


@pytest.mark.parametrize("n", [1, 300, 10922, 10923])
@pytest.mark.parametrize("refused", [False, True])
def test_exports_with_pinned_memory_refused(n, refused):
    assert run_driver(DRIVER, n, int(refused)).split() == ["0", "0", "0"]


FAILED = r"""
#include "fake_cuda.h"
#include <cstdio>
#include <cstdlib>
using namespace sph;
int main(int, char** argv) {
    const uint32_t n = 300;
    SceneConfig c;
    c.box_mode = 1;
    c.h = 0.1f;
    Engine e(0);
    int id, other;
    e.add_scene(c, n, &id);
    if (std::atoi(argv[2])) e.add_scene(c, n, &other);   // a batch: the read runs its scene's prefix
    e.set_export_ahead(false);
    std::vector<float> p(3 * n), q(3 * n), v(3 * n, 0.f);
    int rc = e.step(1);
    rc |= e.get_state(id, p.data(), q.data(), v.data(), n);   // leaves velocities in the landing place
    fake::st.after_force = [&] { fake::st.crowded = {e.scene(id)->part_base}; };
    rc |= e.set_export_ahead(std::atoi(argv[3]) != 0);
    rc |= e.step(1, std::atoi(argv[1]) != 0);   // the next substep's prefix fails
    for (int i = 0; i < 2; ++i) {
        p.assign(3 * n, -1.f); q.assign(3 * n, -1.f); v.assign(3 * n, -1.f);
        const int err = e.get_state(id, p.data(), q.data(), v.data(), n);
        int wrong = 0;
        for (uint32_t k = 0; k < 3 * n; ++k)
            wrong += p[k] != fake::kPosition || q[k] != fake::kPosition || v[k] != -1.f;
        std::printf("%d %d %d ", rc, err, wrong);
    }
}
"""


@pytest.mark.parametrize("blocking", [1, 0])
@pytest.mark.parametrize("many", [0, 1])
@pytest.mark.parametrize("ahead", [0, 1])
def test_export_after_a_failed_prefix(blocking, many, ahead):
    """The error comes with the state's positions and colours, and the caller's
    velocities are left alone: none were computed."""
    assert run_driver(FAILED, blocking, many, ahead).split() == ["0", "7", "0"] * 2


PINNED = r"""
#include "fake_cuda.h"
#include <cstdio>
using namespace sph;
int main() {
    SceneConfig c;
    c.box_mode = 1;
    c.h = 0.1f;
    {
        Engine e(0);
        int id[4];
        const uint32_t n[] = {300, 1000, 10922, 10923};
        for (int i = 0; i < 4; ++i) e.add_scene(c, n[i], &id[i]);
        std::vector<float> p(3 * 10923), v(3 * 10923);
        e.step(1);
        const size_t before = fake::st.pinned;
        for (int i : {3, 0, 1, 2, 0}) {
            e.get_state(id[i], p.data(), nullptr, v.data(), n[i]);
            std::printf("%zu ", fake::st.pinned - before);
        }
        std::printf("%d ", before < 4096u);
    }
    std::printf("%zu", fake::st.pinned);
}
"""


def test_pinned_memory_as_needed():
    """Nothing for a system that exports nothing small; then as much as the largest
    needs, given back with the system."""
    assert run_driver(PINNED).split() == ["0", "32768", "65536", "393216", "393216", "1", "0"]
