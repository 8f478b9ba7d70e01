"""The passes over pairs of radii (kernels_pair.cuh) against the passes that
take one radius at a time: the same bits, at every box side that has them
(each side has line plans of its own), with an even and an odd number of radii
per batch (an odd batch carries its last radius twice)."""
import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu

POW2 = [16, 32, 64, 128, 256]
RAGGED = [24, 40, 48, 72, 80, 96, 120, 144, 160, 192, 200, 216, 240, 288, 320, 360, 384, 400, 432, 480, 576, 600]


@pytest.mark.parametrize("N", POW2 + RAGGED)
def test_pairs_give_the_bits_of_single_radii(hii, N):
    import torch
    L, z = 0.6 * N, 8.0
    delta, src = synth.make_boxes_torch(N, L, z, 100 + N)
    sets = [(30.0, L / 6, 11), (60.0, L / 4, 12)]
    one = dict(path=1) if N in POW2 else dict(kmax=1)  # one radius at a time
    pairs = [dict(path=5, kmax=8), dict(path=5, kmax=5)] if N in POW2 else [dict(kmax=8), dict(kmax=5)]
    ref = None
    for kw in [one] + pairs:
        fb = hii.FilterBank(N, L, 0.71, sets, **kw)
        x = torch.empty((2, N, N, N), device="cuda")
        torch.cuda.synchronize()
        fb.run_z_device(z, delta.data_ptr(), src.data_ptr(), x.data_ptr(),
                        stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        # the first-hit radius shows each centre decision, also inside larger bubbles
        rc = fb.first_hit(z, delta.cpu().numpy(), src.cpu().numpy(), s=1)
        fb.close()
        if ref is None:
            ref = (x, rc)
            assert (rc != 255).any() and (rc == 255).any()
        else:
            assert torch.equal(x, ref[0])
            np.testing.assert_array_equal(rc, ref[1])


@pytest.mark.parametrize("N", [16, 24, 32, 48, 64, 96, 120, 128, 160, 192, 216, 240, 256, 360])
def test_criterion_and_vjp_in_pairs(hii, N):
    """The criterion, its argmax and the VJP against the one-radius kernels:
    C and the argmax bit for bit; the gradients are sums over the radii in
    the same order, but their real-space passes may round differently at the
    2-3-5 sides, so they are held to float32's 2e-5 of their norm."""
    import torch
    L, z = 0.6 * N, 8.0
    delta, src = synth.make_boxes_torch(N, L, z, 200 + N)
    d, s = delta.cpu().numpy(), src.cpu().numpy()
    g = np.random.default_rng(N).random((N, N, N)).astype(np.float32)
    sets = [(30.0, L / 3, 9)]
    one = dict(path=1) if N in POW2 else dict(kmax=1)
    ref = None
    for kw in [one, dict(kmax=8, path=5 if N in POW2 else 0), dict(kmax=3, path=5 if N in POW2 else 0)]:
        fb = hii.FilterBank(N, L, 0.71, sets, **kw)
        C, A = fb.criterion(z, d, s)
        out = fb.vjp(z, d, s, g)
        fb.close()
        torch.cuda.synchronize()
        if ref is None:
            ref = (C, A, out)
            assert (C > 0).any()
            continue
        np.testing.assert_array_equal(C, ref[0])
        np.testing.assert_array_equal(A, ref[1])
        for got, want in zip(out[:2], ref[2][:2]):
            got, want = got.astype(np.float64), want.astype(np.float64)
            assert np.linalg.norm(got - want) <= 2e-5 * np.linalg.norm(want)
        assert abs(out[2] - ref[2][2]) <= 2e-5 * abs(ref[2][2])
