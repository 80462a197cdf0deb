"""A mass that crosses, between frames, the line between one and eight lanes per
particle: the passes that an export runs ahead, outside the graphs, are launched
in the form of the passes before them.  Lists end early here, so a pass that read
the other form's copies of the positions would miss neighbours."""
import numpy as np
import pytest

from helpers import configure_gpu
from libfluid_gb300 import FluidSystem, workloads as W

pytestmark = pytest.mark.gpu


def _mass(h, neighbours):
    return 1000.0 * 4.0 / 3.0 * np.pi * h ** 3 / neighbours


# 49,600 particles: one lane or eight; 19,840: four or eight
@pytest.mark.parametrize("tension", [0.0, 0.05])
@pytest.mark.parametrize("nx", [40, 16])
def test_mass_across_the_line_between_frames(nx, tension):
    h, spacing = 0.02, 0.0064
    lat = W.Lattice(lo=(0.0, 0.0, 0.0), spacing=spacing, nx=nx, ny=40, nz=31, jitter=0.2 * spacing, seed=9,
                    vel=(0.1, -0.2, 0.05))
    spec = W.SceneSpec(box=tuple(1.3 * k * spacing for k in (nx, 40, 31)), h=h, blocks=[lat], mass=_mass(h, 100),
                       gas_constant=1.0, particle_size=0.5 * spacing, surface_tension=tension, dt=5e-5)
    runs = []
    for ahead, graph in ((True, True), (False, True), (False, False)):
        fs = configure_gpu(FluidSystem(0), spec)
        fs.setExportAhead(ahead)
        fs.setUseGraph(graph)
        out = []
        for frame in range(9):
            if frame in (3, 6):
                fs.setMass(_mass(h, 60 if frame == 3 else 100))
            fs.advance(spec.dt, 1)
            out += [a.copy() for a in fs.exportToData()]
        if ahead:
            assert fs.exportAheadStats()["taken"] >= 4
        runs.append(out)
        fs.close()
    assert all(np.isfinite(x).all() for x in runs[0])
    for other in runs[1:]:
        for x, y in zip(runs[0], other):
            assert np.array_equal(x, y)
