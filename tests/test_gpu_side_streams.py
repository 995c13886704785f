"""Plans that are made, set and marched at once on streams that do not wait for the legacy
default stream: the uploads of the plan, its tile, its box model and its schedule are on the
device before the march starts."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from proton_dose_m1_b200 import Accel, Beam, Box, Geometry, Numerics, Physics, SolverConfig, learned_box
from proton_dose_m1_b200.enums import EnergyScheme, Material, Precision, Scattering
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import FieldPlan, M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu


def problem(precision, tile=None, model=None):
    shape = (24, 26, 60)
    geo = Geometry(size=(0.024, 0.026, 0.06), resolution=shape,
                   objects=[Box(0.0, 0.012, -0.013, 0.013, 0.02, 0.03, Material.BONE_COMPACT)])
    cfg = SolverConfig(geometry=geo, beam=Beam(n_protons=1e6, energy=50.0, energy_spread=1.0, sigma=(0.002, 0.0025)),
                       physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                       numerics=Numerics(energy_scheme=EnergyScheme.IF_SSPRK3, cfl=0.9, max_energy_step=0.5,
                                         moving_active_domain=True),
                       accel=Accel(precision=precision, tile=tile, box_model=model))
    grid = Grid.from_geometry(geo)
    return cfg, MaterialMap.from_geometry(geo, grid), grid


def march(cfg, mm, grid, schedule=None):
    plan = M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid))
    if schedule is not None:
        plan.set_schedule(schedule)
    _, dose, E, _ = plan.march(None)
    out = dose.cpu().numpy(), E
    plan.close()
    return out


def field(cfg, mm, grid):
    fp = FieldPlan(cfg, mm, grid, [cfg.beam] * 3, box_capacity_cells=int(np.prod(grid.shape)))
    dose, steps = fp.march()
    out = dose.cpu().numpy(), np.array(steps)
    fp.close()
    return out


@pytest.mark.parametrize("precision", list(Precision))
@pytest.mark.parametrize("settings", [{}, {"tile": (8, 8, 4)}, {"model": True}], ids=["plain", "tile", "learned"])
def test_side_stream_marches_equal_the_default_stream(precision, settings):
    settings = {**settings, **({"model": learned_box.default_model()} if "model" in settings else {})}
    cfg, mm, grid = problem(precision, **settings)
    plain = march(cfg, mm, grid)
    scheduled = march(cfg, mm, grid, schedule=plain[1])
    ref_field, ref_steps = field(cfg, mm, grid)
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(3):
            for schedule, (ref, ref_E) in ((None, plain), (plain[1], scheduled)):
                d, E = march(cfg, mm, grid, schedule)
                np.testing.assert_array_equal(E, ref_E)
                np.testing.assert_array_equal(d, ref)
            d, steps = field(cfg, mm, grid)
            np.testing.assert_array_equal(steps, ref_steps)
            # the beams' atomic sums in another order: a few hundred 64-bit terms a voxel
            assert np.abs(d - ref_field).max() <= 1e-12 * ref_field.max()
