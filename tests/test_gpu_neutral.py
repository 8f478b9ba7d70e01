"""Neutral fractions summed in chunks on the GPU: the serial double sum of the
box that the same call returned, bit for bit, with one to three sets (the boxes
leave by two staging buffers in turn)."""
import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 64, 96, 160])
@pytest.mark.parametrize("nsets", [1, 2, 3])
def test_neutral_is_the_boxes_sum(hii, N, nsets):
    w = synth.Workload(N=N, L=float(N), zs=[8.0], zeta=30.0, Rmax=12.0, factor=1.1, seed=N)
    delta, src = synth.make_boxes(w, 8.0)
    fb = hii.FilterBank(N, float(N), 0.7, [(20.0 + 10.0 * s, 12.0, 8) for s in range(nsets)])
    x, neutral = fb.run_z(8.0, delta, src)
    fb.close()
    for s in range(nsets):
        want = np.add.accumulate(1.0 - x[s].astype(np.float64).ravel())[-1] / N ** 3  # one addition after the other
        assert neutral[s] == want
