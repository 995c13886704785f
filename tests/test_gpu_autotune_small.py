"""The autotuner on plans that run on 4x4x4 tiles under every setting: there is nothing to
measure, and nothing is kept for larger plans on the same grid."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from proton_dose_m1_b200 import Accel, Beam, Geometry, Numerics, Physics, SolverConfig, _native
from proton_dose_m1_b200.enums import EnergyScheme, Precision, Scattering
from proton_dose_m1_b200.numerics import energy as en
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import FieldPlan, M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

SHAPE = (12, 11, 41)   # 99 tiles of 4x4x4: a B200 holds 296 FP64 CTAs, 592 of the FP32 form


def problem(precision, moving, tile="auto"):
    size = tuple(n * 1e-3 for n in SHAPE)
    cfg = SolverConfig(geometry=Geometry(size=size, resolution=SHAPE),
                       beam=Beam(n_protons=1e6, energy=45.0, energy_spread=1.0, sigma=(0.002, 0.002)),
                       physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                       numerics=Numerics(energy_scheme=EnergyScheme.IF_SSPRK3, cfl=0.9, max_energy_step=0.5,
                                         moving_active_domain=moving),
                       accel=Accel(precision=precision, tile=tile))
    grid = Grid.from_geometry(cfg.geometry)
    return cfg, MaterialMap.from_geometry(cfg.geometry, grid), grid


@pytest.mark.parametrize("precision", list(Precision))
@pytest.mark.parametrize("moving", [False, True])
def test_one_beam_measures_and_keeps_nothing(precision, moving):
    cfg, mm, grid = problem(precision, moving)
    plan = M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid))   # tunes
    best = C.c_int(-1)
    ns = (C.c_double * _native.NUM_TILES)(*[7.0] * _native.NUM_TILES)
    _native.check(_native.lib().pdm1_plan_autotune(plan._h, 8, C.byref(best), ns, plan._stream()))
    assert best.value == 0 and list(ns) == [0.0] * _native.NUM_TILES
    assert (precision.name, grid.shape, 1, moving) not in en.autotuned_tiles()
    _, dose, E, _ = plan.march(None)
    plan.close()
    cfg, mm, grid = problem(precision, moving, tile=None)
    plan = M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid))
    _, ref, ref_E, _ = plan.march(None)
    plan.close()
    np.testing.assert_array_equal(E, ref_E)
    assert torch.equal(dose, ref)


def test_small_field_leaves_the_choice_to_larger_ones():
    cfg, mm, grid = problem(Precision.FP64, True)
    key = (Precision.FP64.name, tuple(grid.shape), "field", True)
    for beams, measured in ((2, False), (3, True), (2, True)):   # 198 tiles, 297, 198 again
        fp = FieldPlan(cfg, mm, grid, [cfg.beam] * beams, box_capacity_cells=int(np.prod(SHAPE)))
        fp.march()
        fp.close()
        assert (key in en.autotuned_tiles()) == measured
    assert all(t > 0.0 for t in en.autotuned_tiles()[key][1])
