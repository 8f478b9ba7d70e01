"""Power spectra of boxes of any size of value: P(k) of a box times 2^k is the
P(k) of the box times 2^2k, also where a bin's sum over the box is beyond the
largest float, and a bin with an infinite mode is infinite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 120])
def test_scaled_boxes(hii, N):
    fb = hii.FilterBank(N, float(N), 0.7, [(1.0, N / 4, 1)], kmax=1, path=1)
    box = np.random.default_rng(N).standard_normal((N, N, N)).astype(np.float32)
    _, P = fb.power_spectrum(box, 1.0)
    # white noise: |F|^2 is N^3 a mode, up to 15 times that; the largest one near 2^122,
    # so that a CTA's float sum (some tens of modes of a bin) is finite
    top = 122 - int(np.ceil(np.log2(16.0 * N ** 3)))
    modes = 1.8 * N * N  # of the half-spectrum in the largest bins, about
    assert N ** 3 * 2.0 ** (top // 2 * 2) * modes > 2.0 ** 128  # the bins' sums are no floats
    for k in (top // 2, -30):
        _, Q = fb.power_spectrum(box * np.float32(2.0 ** k), 1.0)
        # the CTAs' float sums are in no fixed order: 32 rows' N/2 + 1 modes at most, 2^-24 each, in both
        np.testing.assert_allclose(Q, P * 4.0 ** k, rtol=32 * (N / 2 + 1) * 2.0 ** -23)
    _, Q = fb.power_spectrum(box * np.float32(2.0 ** (top // 2 + 16)), 1.0)
    assert np.isinf(Q[N // 4: N // 2]).all()
    box[0, 0, 0] = np.nan
    _, Q = fb.power_spectrum(box, 1.0)
    assert np.isnan(Q).all()
    fb.close()
