"""Edges of the gamma index's entry: search radii that the candidate lattice cannot count."""

import os
import subprocess
import sys

import numpy as np
import pytest

from proton_dose_m1_b200 import _native, metrics

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
