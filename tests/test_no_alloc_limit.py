"""The largest problems of the allocation-free march: its scratch is 16 MiB, and a problem that
needs no more of it is taken."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

LIMIT = 16 << 20
HEAD = 7936          # the march's own records
TABLE_NODES = 6000   # of each coefficient table
# one material each; the third number of cells along z is the last that fits
FIT = [(9, 62, 271), (16, 54, 175), (18, 31, 271)]


def scratch_bytes(shape, materials=1):
    """ids, inflow profile, three states of four components, the dose quadrature, each padded to 256 bytes."""
    n = int(np.prod(shape))
    sizes = [3 * 8 * TABLE_NODES] * (3 * materials) + [4 * n, 8 * shape[0] * shape[1]] + 3 * [32 * n] + [8 * n]
    return HEAD + sum((s + 255) & ~255 for s in sizes)


CALL = """
import ctypes as C, sys
import numpy as np
from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig, _native
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import _problem_struct
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap
shape = tuple(int(v) for v in sys.argv[1:4])
cfg = SolverConfig(geometry=Geometry(size=tuple(n * 1e-3 for n in shape), resolution=shape),
                   beam=Beam(n_protons=1e6, energy=20.0, sigma=(0.002, 0.002)), physics=Physics(), numerics=Numerics())
grid = Grid.from_geometry(cfg.geometry)
p, keep, _ = _problem_struct(cfg, MaterialMap.from_geometry(cfg.geometry, grid), grid,
                             BeamInflow.from_beam(cfg.beam, grid).spatial)
L = _native.lib()
L.pdm1_march_noalloc.argtypes = [C.c_void_p] * 4 + [C.c_int] + [C.c_void_p] * 2
rc = L.pdm1_march_noalloc(C.byref(p), 256, 512, 768, 10, None, None)
print(rc, L.pdm1_last_error().decode())
"""


def without_a_gpu(shape):
    """The call's answer in a process that sees no GPU: past its checks it finds no device."""
    r = subprocess.run([sys.executable, "-c", CALL, *map(str, shape)], env={**os.environ, "CUDA_VISIBLE_DEVICES": ""},
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
    return r.stdout


@pytest.mark.parametrize("shape", FIT)
def test_limit_is_the_scratch(shape):
    longer = (*shape[:2], shape[2] + 1)
    assert scratch_bytes(shape) <= LIMIT < scratch_bytes(longer)
    assert "scratch" not in without_a_gpu(shape)
    assert f"needs {scratch_bytes(longer)} bytes of scratch" in without_a_gpu(longer)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", FIT)
def test_largest_problems_equal_the_planned_march(shape):
    torch = pytest.importorskip("torch")
    from proton_dose_m1_b200 import Beam, Geometry, Numerics, Physics, SolverConfig, _native
    from proton_dose_m1_b200.enums import Scattering
    from proton_dose_m1_b200.numerics.boundary import BeamInflow
    from proton_dose_m1_b200.numerics.energy import M1Plan, _problem_struct
    from proton_dose_m1_b200.numerics.grid import Grid
    from proton_dose_m1_b200.physics.materials import MaterialMap
    cfg = SolverConfig(geometry=Geometry(size=tuple(n * 1e-3 for n in shape), resolution=shape),
                       beam=Beam(n_protons=1e6, energy=20.0, energy_spread=0.5, sigma=(0.002, 0.002)),
                       physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                       numerics=Numerics(max_energy_step=0.5))
    grid = Grid.from_geometry(cfg.geometry)
    mm = MaterialMap.from_geometry(cfg.geometry, grid)
    inflow = BeamInflow.from_beam(cfg.beam, grid)
    plan = M1Plan(cfg, mm, grid, inflow)
    U0, dose0, E0, _ = plan.march(None)
    plan.close()
    p, keep, _ = _problem_struct(cfg, mm, grid, inflow.spatial)
    L = _native.lib()
    L.pdm1_march_noalloc.argtypes = [C.POINTER(_native.Problem), C.c_void_p, C.c_void_p, C.c_void_p, C.c_int,
                                     C.POINTER(_native.MarchInfo), C.c_void_p]
    U = torch.zeros((4, *shape), dtype=torch.float64, device="cuda")
    dose, energies = torch.empty_like(U[0]), torch.empty(10001, dtype=torch.float64, device="cuda")
    info = _native.MarchInfo()
    _native.check(L.pdm1_march_noalloc(C.byref(p), C.c_void_p(U.data_ptr()), C.c_void_p(dose.data_ptr()),
                                       C.c_void_p(energies.data_ptr()), 10000, C.byref(info), M1Plan._stream()))
    np.testing.assert_array_equal(energies[: info.n_steps + 1].cpu().numpy(), E0)
    assert torch.equal(dose, dose0) and torch.equal(U, U0)
