"""Plans check the material ids on the device: an id outside the materials anywhere in the
grid refuses the plan, and the next plan is none the worse for it."""

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig
from proton_dose_m1_b200.enums import Material
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import FieldPlan, M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

# below a warp, off every multiple, more cells than the kernel's grid has threads (8 x 148 x 256)
SHAPES = [(2, 3, 4), (7, 5, 37), (81, 80, 79)]


def problem(shape, moving=False):
    size = tuple(n * 1e-3 for n in shape)
    cfg = SolverConfig(geometry=Geometry(size=size, resolution=shape),
                       beam=Beam(n_protons=1e6, energy=40.0, sigma=(0.002, 0.002)), physics=Physics(),
                       numerics=Numerics(max_energy_step=0.5, moving_active_domain=moving))
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    ids = np.zeros(shape, dtype=np.int32)
    ids.reshape(-1)[::3] = 1
    mm = replace(mm, ids=ids, materials=(Material.WATER, Material.BONE_COMPACT))
    return cfg, mm, grid


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bad", [2, 16, -1, 2**31 - 1, -2**31])
def test_id_outside_the_materials_is_refused(shape, bad):
    cfg, mm, grid = problem(shape)
    inflow = BeamInflow.from_beam(cfg.beam, grid)
    for where in (0, mm.ids.size // 2, mm.ids.size - 1):
        ids = mm.ids.copy()
        ids.reshape(-1)[where] = bad
        with pytest.raises(ValueError, match="material id out of range"):
            M1Plan(cfg, replace(mm, ids=ids), grid, inflow)
    plan = M1Plan(cfg, mm, grid, inflow)
    _, _, E = plan.march_steps(2)
    assert len(E) == 3
    plan.close()


def test_field_refuses_too():
    cfg, mm, grid = problem((20, 20, 40), moving=True)
    ids = mm.ids.copy()
    ids[-1, -1, -1] = 2
    with pytest.raises(ValueError, match="material id out of range"):
        FieldPlan(cfg, replace(mm, ids=ids), grid, [cfg.beam, cfg.beam])
