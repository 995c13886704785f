"""The gamma index where nearly every voxel passes at once: two close doses without a cutoff.

Such a voxel needs one candidate, its own position; the call then takes a few times as long
as one that searches no voxel at all, and the voxels' gammas are those of the plain search."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import gamma as gamma_oracle
from proton_dose_m1_b200 import metrics

pytestmark = pytest.mark.gpu


def median_ms(call, n=9):
    times = []
    for _ in range(n + 2):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        call()
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    return float(np.median(times[2:]))


def test_passing_voxels_cost_one_candidate():
    g = torch.Generator(device="cuda").manual_seed(3)
    ref = 1.0 + torch.rand((256, 256, 320), dtype=torch.float64, device="cuda", generator=g)
    close = 1.002 * ref
    rate, _ = metrics.gamma(close, ref, (1.0, 1.0, 1.0), lower_percent_dose_cutoff=0.0)
    assert rate == 100.0
    searched = median_ms(lambda: metrics.gamma(close, ref, (1.0, 1.0, 1.0), lower_percent_dose_cutoff=0.0))
    none = median_ms(lambda: metrics.gamma(close, ref, (1.0, 1.0, 1.0), lower_percent_dose_cutoff=101.0))
    # one candidate reads nine doses a voxel where none reads one (a warp per voxel: 32
    # candidates and some 30 times as long)
    assert searched <= 10.0 * none, (searched, none)


@pytest.mark.parametrize("share", [0.0, 0.03, 0.5, 1.0])
def test_voxels_that_fail_among_those_that_pass(share):
    """From no voxel to every voxel of a CTA goes on to the search, grid of 2.3 CTAs."""
    r = np.random.default_rng(8)
    shape = (9, 8, 8)
    ref = 1.0 + 0.1 * r.random(shape)
    ev = ref * np.where(r.random(shape) < share, 1.08, 1.001)
    rate, g = metrics.gamma(ev, ref, (1.0, 1.0, 1.0), lower_percent_dose_cutoff=92.0)
    rate_o, g_o = gamma_oracle.gamma(ev, ref, (1.0, 1.0, 1.0), cutoff_percent=92.0)
    g = g.cpu().numpy()
    assert rate == pytest.approx(rate_o, abs=1e-12)
    np.testing.assert_array_equal(np.isnan(g), np.isnan(g_o))
    np.testing.assert_array_equal(np.isinf(g), np.isinf(g_o))
    np.testing.assert_array_equal(g <= 1.0, g_o <= 1.0)
    failing = np.isfinite(g_o) & (g_o > 1.0)
    # the kernel stops at the first candidate that passes; a failing voxel takes the smallest of
    # all: a handful of operations of 64-bit numbers of order one
    np.testing.assert_allclose(g[failing], g_o[failing], rtol=1e-12, atol=1e-14)
