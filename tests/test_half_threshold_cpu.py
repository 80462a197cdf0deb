"""The threshold of the half-precision candidate test that derive_params hands to the
kernels is the one that tests/test_half_scan.py shows to accept every pair within h."""
import numpy as np

from host_engine import run_driver
from test_half_scan import near2

DRIVER = r"""
#include "engine.h"
#include <cstdio>
int main() {
    using namespace sph;
    auto show = [](const SceneConfig& c) {
        DevParams d;
        if (!derive_params(c, d, nullptr)) return;
        const uint32_t cells = d.gx > d.gy ? (d.gx > d.gz ? d.gx : d.gz) : (d.gy > d.gz ? d.gy : d.gz);
        std::printf("%.17g %u %.9g\n", (double)d.h * d.inv_cell, cells, d.near2);
    };
    SceneConfig c;
    for (c.res = 1; c.res < 1200; c.res += c.res < 40 ? 1 : 97) show(c);
    c.box_mode = 1;
    for (float h : {0.02f, 0.0173f, 0.1f, 3.0f, 1e-3f, 7e-5f})
        for (float x : {1.f, 10.f, 333.f, 40000.f}) {
            c.h = h;
            c.lx = x * h;
            c.ly = 3 * h;
            c.lz = 0.5f * h;
            show(c);
        }
}
"""


def test_threshold_is_the_tested_one():
    rows = [line.split() for line in run_driver(DRIVER).splitlines()]
    assert len(rows) > 70
    for hc, cells, got in rows:
        assert abs(float(hc) - 1.0) < 2e-7   # h is a cell up to rounding
        assert np.isclose(float(got), near2(float(hc), int(cells)), rtol=1e-6, atol=0)
