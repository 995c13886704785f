"""The entrance tiles' choice between the branch-free and the IEEE reconstructions.

It follows from the cells and ghosts of the tile alone.  The narrower stencils write fewer
ghost cells than the tile's shared memory has room for; what an earlier kernel left in
the others decides nothing, so a WENO3 operator takes the same time (with its IEEE path
the call took 0.93 ms instead of 0.64) and gives the same doubles whatever ran before it.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig
from proton_dose_m1_b200.enums import SpatialScheme
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

SHAPE = (512, 512, 8)   # every tile is an entrance tile


def plan_of(scheme):
    size = tuple(n * 1e-3 for n in SHAPE)
    cfg = SolverConfig(geometry=Geometry(size=size, resolution=SHAPE),
                       beam=Beam(n_protons=1e6, energy=60.0, sigma=(0.05, 0.05)), physics=Physics(),
                       numerics=Numerics(spatial_scheme=scheme))
    grid = Grid.from_geometry(cfg.geometry)
    return M1Plan(cfg, MaterialMap.from_geometry(cfg.geometry, grid), grid, BeamInflow.from_beam(cfg.beam, grid))


def test_stale_ghosts_decide_nothing():
    wide, narrow = plan_of(SpatialScheme.WENO_Z), plan_of(SpatialScheme.WENO3)
    r = torch.Generator(device="cuda").manual_seed(5)
    U = torch.rand((4, *SHAPE), dtype=torch.float64, device="cuda", generator=r)
    U[1:] *= 0.3
    # the wide stencil's ghosts of these are 0, and beyond the branch-free range
    before = {"in range": torch.zeros_like(U), "out of range": torch.full_like(U, 1e80)}
    times = {k: [] for k in before}
    out = {}
    for rep in range(12):
        for k, state in before.items():
            wide.spatial_operator(state, 60.0)
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            out[k] = narrow.spatial_operator(U, 60.0)
            end.record()
            end.synchronize()
            if rep >= 2:
                times[k].append(begin.elapsed_time(end))
    assert torch.equal(out["in range"], out["out of range"])
    fast, after = (float(np.median(times[k])) for k in before)
    # the same instructions on the same data; a fifth is far above the timer's noise
    assert after <= 1.2 * fast, (fast, after)
    wide.close()
    narrow.close()
