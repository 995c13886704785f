"""Domains that fit one wave of 4x4x4 tiles (csrc/pdm1_device.cuh, SmallTile).

The tile a cell sits in changes no result: grids on either side of the limit, with
ragged edges and at the smallest size, give the oracle's doubles.
"""

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle.oracle import OracleProblem
from proton_dose_m1_b200 import Accel, Beam, Box, Geometry, Numerics, Physics, SolverConfig
from proton_dose_m1_b200.enums import EnergyScheme, Material, Precision, Scattering
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

# 4x4x4 tiles: 1; 3 x 2 x 10; 4 x 4 x 18 = 288; 4 x 5 x 15 = 300 (a B200 holds 296 FP64 CTAs)
SHAPES = [(4, 4, 4), (9, 5, 37), (16, 13, 72), (16, 17, 60)]


def config(shape, **numerics):
    size = tuple(n * 1e-3 for n in shape)
    geo = Geometry(size=size, resolution=shape,
                   objects=[Box(-size[0] / 2, size[0] / 2, -size[1] / 2, size[1] / 2, 0.4 * size[2], 0.5 * size[2],
                                Material.BONE_COMPACT)])
    return SolverConfig(geometry=geo, beam=Beam(n_protons=1e6, energy=60.0, sigma=(0.002, 0.002)),
                        physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                        numerics=Numerics(energy_scheme=EnergyScheme.IF_SSPRK3, cfl=0.9, max_energy_step=0.5, **numerics))


def plan_of(cfg):
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    return M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid)), OracleProblem(cfg, mm), grid.shape


@pytest.mark.parametrize("shape", SHAPES)
def test_march_equals_oracle(shape):
    plan, oracle, _ = plan_of(config(shape))
    U, dose, E = plan.march_steps(25)
    Uo, doseo, steps = oracle.march_steps(25)
    assert len(E) - 1 == steps
    np.testing.assert_array_equal(U.cpu().numpy(), Uo)
    np.testing.assert_array_equal(dose.cpu().numpy(), doseo)


def test_moving_box_across_the_limit_equals_oracle():
    # the box grows from 4 x 4 x 3 tiles to the 10-cell-wide beam's whole depth window
    plan, oracle, shape = plan_of(config((20, 20, 60), moving_active_domain=True))
    U, dose, E, _ = plan.march(None)
    Uo, doseo, Eo, _ = oracle.march(np.zeros((4, *shape)))
    np.testing.assert_array_equal(E, Eo)
    np.testing.assert_array_equal(dose.cpu().numpy(), doseo)


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_operator_near_oracle(shape):
    cfg = config(shape)
    plan, oracle, _ = plan_of(replace(cfg, accel=Accel(precision=Precision.FP32_FP64)))
    U, _, _ = oracle.march_steps(12)
    got, want = plan.spatial_operator(U, 55.0).cpu().numpy(), oracle.spatial_operator(U, 55.0)
    # the float face flux is within 3.8e-4 of phi of the double one (six faces per cell), and
    # its own reading of the state rounds phi by 6e-8
    top = max(np.abs(U[0]).max(), 1.1 * np.abs(oracle.inflow_state(55.0)).max())
    assert np.abs(got - want).max() <= 6 * 3.8e-4 * top / 1e-3
