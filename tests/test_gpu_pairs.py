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
