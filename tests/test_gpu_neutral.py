"""Neutral fractions summed on the GPU: against the correctly rounded sum of
the box that the same call returned, with one to three sets (the boxes leave
by two staging buffers in turn).  A block adds n3 / 622592 terms per column and
ten levels, the host 608 blocks: within 640 2^-53 of the sum at these sides."""
import math

import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 64, 96])
@pytest.mark.parametrize("nsets", [1, 2, 3])
def test_neutral_is_the_boxes_sum(hii, N, nsets):
    w = synth.Workload(N=N, L=float(N), zs=[8.0], zeta=30.0, Rmax=12.0, factor=1.1, seed=N)
    delta, src = synth.make_boxes(w, 8.0)
    fb = hii.FilterBank(N, float(N), 0.7, [(20.0 + 10.0 * s, 12.0, 8) for s in range(nsets)])
    x, neutral = fb.run_z(8.0, delta, src)
    fb.close()
    for s in range(nsets):
        want = math.fsum((1.0 - x[s].astype(np.float64)).ravel()) / N ** 3
        assert abs(neutral[s] - want) <= 640 * 2.0 ** -53 * abs(want)
