"""What scoring and the analytical dose keep between calls is bounded by their largest call,
not by the number of different sizes they were called with."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig, _native, metrics
from proton_dose_m1_b200.analytical import analytical_csda_dose
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu


def cached_by(call, sizes):
    """Bytes the pool holds after the first, largest size and after all of them."""
    L = _native.lib()
    _native.check(L.pdm1_pool_release())
    call(sizes[0])
    first = L.pdm1_pool_cached_bytes()
    for s in sizes[1:]:
        call(s)
    last = L.pdm1_pool_cached_bytes()
    _native.check(L.pdm1_pool_release())
    assert 0 < first
    return first, last


def analytical(nz):
    shape = (160, 160, nz)
    cfg = SolverConfig(geometry=Geometry(size=tuple(n * 5e-4 for n in shape), resolution=shape),
                       beam=Beam(n_protons=1e6, energy=60.0, energy_spread=1.0, sigma=(0.003, 0.003)),
                       physics=Physics(), numerics=Numerics())
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    dose = analytical_csda_dose(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid), num_energy_points=4000)
    assert dose.max() > 0.0


def gamma(fraction):
    ref = 1.0 + np.random.default_rng(1).random((6, 5, 7))
    metrics.gamma(1.001 * ref, ref, (1.0, 1.0, 1.0), interp_fraction=fraction)


# a block of a power of two bytes per call: all the smaller ones together are smaller than the largest
@pytest.mark.parametrize("call,sizes", [(analytical, range(400, 150, -25)), (gamma, range(14, 3, -1))],
                         ids=["analytical", "gamma"])
def test_kept_memory_is_bounded_by_the_largest_call(call, sizes):
    first, last = cached_by(call, list(sizes))
    assert last < 2 * first, (first, last)
