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
