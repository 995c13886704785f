"""Edges of the gamma index's entry: search radii that the candidate lattice cannot count,
doses with an axis of one cell."""

import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import gamma as gamma_oracle
from proton_dose_m1_b200 import metrics

# distance, candidates per distance, max gamma: an infinite radius, an infinite distance, a
# radius past every integer
UNBOUNDED = [(1.0, 10, float("inf")), (float("inf"), 10, 1.1), (1.0, 10, 1e300), (1.0, 10, 3e8)]

CALL = """
import sys
from proton_dose_m1_b200 import _native
d, n, g = float(sys.argv[1]), int(sys.argv[2]), float(sys.argv[3])
print(_native.lib().pdm1_gamma(256, 512, 2, 3, 4, 1.0, 1.0, 1.0, 1.0, d, 10.0, n, g, 1.0, 768, None, None))
"""


@pytest.mark.parametrize("distance,fraction,max_gamma", UNBOUNDED)
def test_unbounded_search_returns_a_status(distance, fraction, max_gamma):
    # a process without a GPU: the candidates are listed, then the allocation is refused
    r = subprocess.run([sys.executable, "-c", CALL, str(distance), str(fraction), str(max_gamma)],
                       env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
    assert int(r.stdout) != 0


@pytest.mark.gpu
@pytest.mark.parametrize("distance,fraction,max_gamma", UNBOUNDED)
def test_unbounded_search_has_no_candidates(distance, fraction, max_gamma):
    ref = np.random.default_rng(2).random((3, 4, 5))
    rate, g = metrics.gamma(ref, ref, (1.0, 1.0, 1.0), 1.0, distance, interp_fraction=fraction, max_gamma=max_gamma)
    g = g.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(g), ref < 0.1 * ref.max())
    assert rate == 0.0 and np.isinf(g[~np.isnan(g)]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 9, 8), (7, 1, 8), (7, 9, 1), (1, 1, 12), (1, 12, 1), (12, 1, 1), (1, 1, 1), (2, 1, 2)])
def test_axis_of_one_cell_equals_oracle(shape):
    """Doses of one layer or one line: the interpolation stays on their only layer."""
    r = np.random.default_rng(sum(shape))
    ref = 1.0 + 0.02 * r.random(shape)
    ev = ref * (1.0 + 0.03 * r.standard_normal(shape))
    spacing = (1.0, 0.8, 1.2)
    rate, g = metrics.gamma(ev, ref, spacing)
    rate_o, g_o = gamma_oracle.gamma(ev, ref, spacing)
    g = g.cpu().numpy()
    assert rate == pytest.approx(rate_o, abs=1e-12)
    np.testing.assert_array_equal(g <= 1.0, g_o <= 1.0)
    # the kernel stops at the first candidate that passes; a voxel where none does takes the
    # smallest of them: a handful of operations of 64-bit numbers of order one
    failing = np.isfinite(g_o) & (g_o > 1.0)
    np.testing.assert_allclose(g[failing], g_o[failing], rtol=1e-12, atol=1e-14)
    np.testing.assert_array_equal(np.isinf(g), np.isinf(g_o))
