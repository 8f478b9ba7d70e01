"""Sides whose radii go several batches to a launch: the grid rows' first hits
meet in one box.  One call with all radii in a launch and one that takes three
radii at a time give the same first hits and the same boxes, for odd and even
numbers of radii, below and above one batch, with several sets."""
import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 32, 48, 64, 72, 80])
@pytest.mark.parametrize("nbins", [5, 16, 35, 70])
def test_grouped_radii(hii, N, nbins):
    L = 0.5 * N
    w = synth.Workload(N=N, L=L, zs=[8.0], zeta=30.0, Rmax=L / 3, factor=1.1, seed=N)
    delta, src = synth.make_boxes(w, 8.0)
    sets = [(30.0, L / 3, nbins), (12.0, L / 5, max(nbins // 2, 1))]
    out = []
    for kmax in (0, 3):
        fb = hii.FilterBank(N, L, 0.7, sets, kmax=kmax)
        for again in range(2):
            x, neutral = fb.run_z(8.0, delta, src)
        out.append((x, neutral, [fb.first_hit(8.0, delta, src, s) for s in range(2)]))
        fb.close()
    assert np.array_equal(out[0][0].view(np.uint32), out[1][0].view(np.uint32))
    assert np.array_equal(out[0][1], out[1][1])
    for s in range(2):
        assert np.array_equal(out[0][2][s], out[1][2][s])
    assert (out[0][2][0] != 255).any()
