"""Neutral fractions of boxes with one or two values of xHII (cells partly
ionised by their own source), whose terms all round the same way, against the
serial double sum of the box that the same call returned: from one chunk of
the sum to many, a last chunk that is not full, and more chunks than one pass
of their scan takes."""
import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 32, 40, 128, 256, 320])
def test_neutral_of_uniform_boxes(hii, N):
    z, zeta, L = 7.0, 30.0, 0.5 * N
    fb = hii.FilterBank(N, L, 0.7, [(zeta, 4.0, 4)])
    for low, high in ((0.2, 0.2), (0.0, 0.0), (1e-9, 0.4), (0.18, 0.001)):  # xHII of each half, about
        delta = np.zeros((N, N, N), np.float32)
        rec0, _, _ = fb.prologue(z, delta, delta)
        ratio = np.full((N, N, N), low, np.float32)
        ratio[N // 2:] = high
        src = (ratio * rec0 / ((L / N) ** 3 * synth.qion(z) * zeta)).astype(np.float32)
        x, neutral = fb.run_z(z, delta, src)
        assert len(np.unique(x)) == 1 + (low != high) and abs(x[0, 0, 0, 0] - low) <= 1e-3 * low
        want = np.add.accumulate(1.0 - x[0].astype(np.float64).ravel())[-1] / N ** 3  # one addition after the other
        assert neutral[0] == want
    fb.close()
