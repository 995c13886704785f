"""A single step works on the full grid: a field plan of one beam whose buffers hold a smaller
box refuses it, one whose buffers hold the grid takes it."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle.oracle import OracleProblem
from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig, _native
from proton_dose_m1_b200.enums import EnergyScheme, Scattering
from proton_dose_m1_b200.numerics.energy import FieldPlan, M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

SHAPE = (24, 24, 40)


@pytest.mark.parametrize("short", [0, 1, 9000])
def test_advance_needs_buffers_of_the_grid(short):
    size = tuple(n * 1e-3 for n in SHAPE)
    cfg = SolverConfig(geometry=Geometry(size=size, resolution=SHAPE),
                       beam=Beam(n_protons=1e6, energy=50.0, energy_spread=1.0, sigma=(0.001, 0.001)),
                       physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                       numerics=Numerics(energy_scheme=EnergyScheme.IF_SSPRK3, max_energy_step=0.5,
                                         moving_active_domain=True))
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    fp = FieldPlan(cfg, mm, grid, [cfg.beam], box_capacity_cells=int(np.prod(SHAPE)) - short)
    r = np.random.default_rng(4)
    U0 = r.random((4, *SHAPE))
    U0[1:] *= 0.2
    U = torch.as_tensor(U0, device="cuda")
    edep = torch.zeros(SHAPE, dtype=torch.float64, device="cuda")
    rc = _native.lib().pdm1_advance(fp._plans[0], C.c_void_p(U.data_ptr()), 45.0, 0.1, C.c_void_p(edep.data_ptr()),
                                    M1Plan._stream())
    if short:
        with pytest.raises(ValueError, match="moving box"):
            _native.check(rc)
        np.testing.assert_array_equal(U.cpu().numpy(), U0)
    else:
        _native.check(rc)
        Uo, depo = OracleProblem(cfg, mm).advance(U0, 45.0, 0.1)
        np.testing.assert_array_equal(U.cpu().numpy(), Uo)
        np.testing.assert_array_equal(edep.cpu().numpy(), depo)
    fp.close()
