"""The FP64 stage kernels' face path over the range of a double.

Inside a range of exponents the kernels take quotients and square roots without
the compiler's IEEE routines (csrc/pdm1_fp64.cuh); a tile or a face that leaves it
takes the IEEE path.  Both give the oracle's doubles: states whose magnitudes lie
on either side of each limit, mixed with zeros, reproduce it bit for bit.
"""

from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle.oracle import OracleProblem
from proton_dose_m1_b200.enums import SpatialScheme, WaveSpeeds
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap
from tests import cases

pytestmark = pytest.mark.gpu


def plan_and_oracle(**numerics):
    cfg = cases.operator_config("if_full")
    cfg = replace(cfg, numerics=replace(cfg.numerics, **numerics))
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    return M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid)), OracleProblem(cfg, mm), grid.shape


def state(shape, low, high, seed):
    """phi = 2^e with e uniform in [low, high], |J|/phi from at rest to not realizable, a tenth of the cells empty."""
    r = np.random.default_rng(seed)
    phi = np.ldexp(1.0 + r.random(shape), r.integers(low, high + 1, shape))
    J = r.standard_normal((3, *shape))
    J *= phi * r.choice([0.0, 1e-9, 0.3, 0.9999, 1.2], shape) / np.sqrt((J * J).sum(0))
    J[r.random((3, *shape)) < 0.1] = 0.0
    U = np.concatenate([phi[None], J])
    U[:, r.random(shape) < 0.1] = 0.0
    return U


# about the ordinary magnitudes of a march; across |J|^2 >= 2^-900 and phi >= 2^-450;
# across the state's 2^-940 into the subnormal range; across its upper limit 2^200; all of it
RANGES = [(-20, 34), (-470, -440), (-1074, -930), (190, 206), (-1074, 205)]


@pytest.mark.parametrize("low,high", RANGES)
@pytest.mark.parametrize("numerics", [{}, {"spatial_scheme": SpatialScheme.WENO3}, {"spatial_scheme": SpatialScheme.MUSCL},
                                      {"wave_speeds": WaveSpeeds.UNIT}], ids=["wenoz", "weno3", "muscl", "unit"])
def test_operator_and_step_equal_oracle(low, high, numerics):
    plan, oracle, shape = plan_and_oracle(**numerics)
    U = state(shape, low, high, seed=high - low)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(plan.spatial_operator(U, 99.0).cpu().numpy(), oracle.spatial_operator(U, 99.0))
        Un, dep = plan.advance(U, 99.0, 0.05)
        Uo, depo = oracle.advance(U, 99.0, 0.05)
    np.testing.assert_array_equal(Un.cpu().numpy(), Uo)
    np.testing.assert_array_equal(dep.cpu().numpy(), depo)
    assert plan.energy_step(U, 99.0) == oracle.energy_step(U, 99.0)
