"""Moving boxes, learned boxes and fields on 4x4x4 tiles (csrc/pdm1_device.cuh, SmallTile).

A plan runs on them where the 4x4x4 tiles of its grids, all beams together, fit one wave of
CTAs: 296 in double, 592 in the FP32 form on a B200.  Each case states which side of that
line it lies on, and the plan is asked: the autotuner measures nothing on such a plan.
"""

import ctypes as C
from dataclasses import replace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import mlp as omlp
from oracle.oracle import OracleProblem
from proton_dose_m1_b200 import (Accel, Beam, Box, Geometry, Numerics, Physics, SolverConfig, _native, learned_box,
                                 metrics)
from proton_dose_m1_b200.enums import EnergyScheme, Material, Precision, Scattering
from proton_dose_m1_b200.numerics.boundary import BeamInflow
from proton_dose_m1_b200.numerics.energy import FieldPlan, M1Plan
from proton_dose_m1_b200.numerics.grid import Grid
from proton_dose_m1_b200.physics.materials import MaterialMap

pytestmark = pytest.mark.gpu

FP64, FP32 = Precision.FP64, Precision.FP32_FP64
# every margin the guard, the flux check silent: the heuristic boxes
GUARD = learned_box.BoxModel(params=np.zeros(omlp.N_PARAMS, np.float32), x_mean=np.zeros(16, np.float32),
                             x_inv_std=np.ones(16, np.float32), y_scale=np.zeros(6, np.float32),
                             y_offset=np.full(6, 9.0, np.float32), margin_min=0, margin_max=64, leak_tolerance=1e30)
# margins of zero: the flux check grows the faces
TINY = replace(GUARD, y_offset=np.zeros(6, np.float32), grow_cells=2, extra_max=40, leak_tolerance=1e-6)


def config(shape, precision=FP64, moving=True, model=None):
    size = tuple(n * 1e-3 for n in shape)
    geo = Geometry(size=size, resolution=shape,
                   objects=[Box(0.0, size[0] / 2, -size[1] / 2, size[1] / 2, 0.010, 0.018, Material.BONE_COMPACT)])
    return SolverConfig(geometry=geo, beam=Beam(n_protons=1e6, energy=55.0, energy_spread=1.0, sigma=(0.0015, 0.0015)),
                        physics=Physics(scattering=Scattering.WENTZEL, nuclear=True),
                        numerics=Numerics(energy_scheme=EnergyScheme.IF_SSPRK3, cfl=0.9, max_energy_step=0.5,
                                          moving_active_domain=moving),
                        accel=Accel(precision=precision, box_model=model))


def on_small_tiles(handle) -> bool:
    ns = (C.c_double * _native.NUM_TILES)()
    _native.check(_native.lib().pdm1_plan_autotune(handle, 4, C.byref(C.c_int()), ns, M1Plan._stream()))
    return not any(ns)


def problem(cfg):
    grid = Grid.from_geometry(cfg.geometry)
    return MaterialMap.from_geometry(cfg.geometry, grid), grid


def march(cfg, small, staging=None):
    mm, grid = problem(cfg)
    plan = M1Plan(cfg, mm, grid, BeamInflow.from_beam(cfg.beam, grid))
    assert on_small_tiles(plan._h) == small
    if staging is not None:
        _native.check(_native.lib().pdm1_plan_set_staging(plan._h, staging))
    U, dose, E, _ = plan.march(None)
    info = plan.last_info
    plan.close()
    return U.cpu().numpy(), dose.cpu().numpy(), E, info, grid


# 4 x 4 x 18 = 288 tiles; 4 x 5 x 15 = 300
@pytest.mark.parametrize("shape,small", [((16, 16, 72), True), ((16, 17, 60), False)])
@pytest.mark.parametrize("model", [None, GUARD], ids=["heuristic", "learned"])
def test_moving_box_equals_oracle(shape, small, model):
    cfg = config(shape, model=model)
    _, dose, E, _, _ = march(cfg, small)
    _, doseo, Eo, _ = OracleProblem(cfg, problem(cfg)[0]).march(np.zeros((4, *shape)))
    np.testing.assert_array_equal(E, Eo)
    np.testing.assert_array_equal(dose, doseo)


# 4 x 5 x 29 = 580 tiles; 4 x 5 x 30 = 600; ragged along every axis
@pytest.mark.parametrize("shape,small", [((16, 20, 116), True), ((16, 20, 120), False), ((15, 18, 61), True)])
@pytest.mark.parametrize("moving,model", [(False, None), (True, None), (True, GUARD), (True, TINY)],
                         ids=["full", "heuristic", "learned", "learned_grows"])
def test_fp32_march(shape, small, moving, model):
    """Bulk row copies and cell loads give the same bits, and the dose holds the gate of the
    FP32 form (gamma 1 %/1 mm on 99.5 %, maximum within 0.5 %) against the full-domain FP64
    march; with margins of zero, whose boxes cut 0.55 % off the maximum in FP64 too, against
    the FP64 march on those boxes."""
    cfg = config(shape, FP32, moving, model)
    U1, d1, E1, info, grid = march(cfg, small, staging=1)
    U0, d0, E0, _, _ = march(cfg, small, staging=0)
    np.testing.assert_array_equal(E1, E0)
    np.testing.assert_array_equal(U1, U0)
    np.testing.assert_array_equal(d1, d0)
    if model is TINY:
        assert info.box_grow_events > 0
    plain = config(shape, FP64, True, TINY) if model is TINY else config(shape, FP64, False)
    mm, _ = problem(plain)
    plan = M1Plan(plain, mm, grid, BeamInflow.from_beam(plain.beam, grid))
    _, ref, _, _ = plan.march(None)
    plan.close()
    score = metrics.compare(d1, ref, grid)
    assert score["gamma_1pct_1mm_pass_percent"] >= 99.5, score
    assert abs(score["maximum_dose_relative_difference"]) <= 0.005, score


@pytest.mark.parametrize("precision,shape", [(FP64, (16, 16, 72)), (FP32, (16, 20, 116))])
def test_guard_model_is_the_heuristic_box(precision, shape):
    _, d, E, info, _ = march(config(shape, precision), True)
    _, dl, El, infol, _ = march(config(shape, precision, model=GUARD), True)
    np.testing.assert_array_equal(El, E)
    np.testing.assert_array_equal(dl, d)
    assert infol.cell_steps == info.cell_steps and infol.box_grow_events == 0


BEAMS = [Beam(n_protons=1e6, energy=50.0, energy_spread=1.0, sigma=(0.0012, 0.0015), center=(-0.002, 0.001)),
         Beam(n_protons=2e6, energy=57.0, energy_spread=0.8, sigma=(0.0015, 0.0012), center=(0.002, -0.001)),
         Beam(n_protons=1e6, energy=43.0, energy_spread=1.2, sigma=(0.001, 0.002), center=(0.0, 0.002))]


# 3 x 4 x 12 = 144 tiles a beam: two FP64 beams and four FP32 ones fit, one more does not
@pytest.mark.parametrize("precision,n,small", [(FP64, 2, True), (FP64, 3, False), (FP32, 4, True), (FP32, 5, False)])
@pytest.mark.parametrize("model", [None, GUARD], ids=["heuristic", "learned"])
def test_field_is_the_sum_of_its_beams(precision, n, small, model):
    shape = (12, 13, 48)
    cfg = config(shape, precision, model=model)
    beams = [BEAMS[k % 3] for k in range(n)]
    mm, grid = problem(cfg)
    fp = FieldPlan(cfg, mm, grid, beams, box_capacity_cells=int(np.prod(shape)))
    assert on_small_tiles(fp._plans[0]) == small
    dose, steps = fp.march()
    dose = dose.cpu().numpy()
    fp.close()
    total = np.zeros(shape)
    for b, n_steps in zip(beams, steps):
        _, d, E, _, _ = march(replace(cfg, beam=b), True)
        assert n_steps == len(E) - 1
        if precision is FP64:
            _, doseo, Eo, _ = OracleProblem(replace(cfg, beam=b), mm).march(np.zeros((4, *shape)))
            np.testing.assert_array_equal(E, Eo)
            np.testing.assert_array_equal(d, doseo)
        total += d
    # the order of the atomic sums: at most a few thousand additions of 64-bit terms of one
    # sign; beside tiles of another shape the FP32 stencil may round a face differently
    bound = 1e-12 if precision is FP64 or small else 1e-4
    assert np.abs(dose - total).max() <= bound * total.max()
