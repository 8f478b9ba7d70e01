"""The pair lines on one natural-layout box (forward passes, the power
spectrum's half box, the 21-cm stage's inverse) against the restatements, at
sides whose last column block is cut (N mod 16 = 8), at the smallest ones and
at a few of each kind of plan.  Tolerances as for the stages' other tests:
1e-5 of the value for P(k), 1e-5 of the box's largest |T_b|."""
import numpy as np
import pytest

from oracle import pk_oracle as PK
from oracle import t21_oracle as T
from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 32, 40, 48, 72, 96, 160, 200, 216, 240, 256, 360])
def test_power_spectrum_and_velocity_gradient(hii, N):
    L = 0.7 * N
    box = synth.lognormal_delta(synth.gaussian_field(N, 31 + N), 0.8)
    fb = hii.FilterBank(N, L, 0.71, [(1.0, L / 4, 1)], kmax=1, path=1)
    k, P = fb.power_spectrum(box, 0.7, 1)
    kr, Pr, _ = PK.power_spectrum(box, 0.7, 1)
    assert len(k) == len(kr)
    np.testing.assert_allclose(k, kr, rtol=1e-12)
    np.testing.assert_allclose(P, Pr, rtol=1e-5, atol=1e-5 * np.abs(Pr).max() * 1e-3)
    x = np.clip(np.random.default_rng(N).random(box.shape) * 1.6 - 0.3, 0, 1).astype(np.float32)
    for axis in (1, 3):
        tb, m, _ = fb.t21(8.0, box, x, vel_comp=axis, omega_m=0.27, omega_b=0.046, omega_lambda=0.73)
        ref, mref, _ = T.t21_box(8.0, box, x, L, T.Cosmo(0.27, 0.046, 0.73, 0.71), axis)
        assert np.abs(tb - ref).max() <= 1e-5 * np.abs(ref).max()
        assert abs(m - mref) <= 1e-5 * abs(mref)
    fb.close()
