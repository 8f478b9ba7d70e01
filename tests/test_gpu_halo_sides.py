"""The halo deposit at every block side that has tiles of its own and the first
that has not, with few and many tiles and with catalogues on both sides of the
line between the tiles and the fine grid, against the CPU restatement, bit for
bit; and a context that meets a small catalogue, a large one and the small one
again."""
import numpy as np
import pytest

from test_gpu_sfr import _random_catalogue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N_halo", [25, 61, 132])
def test_block_sides(hii, oracle_lib, side, N_halo):
    from simfast21_gb300 import sfr
    L, z, N = 20.0, 8.0, N_halo // side
    assert round(N_halo / N) == side
    p = oracle_lib.params(N, L, 0.71, L / 2, 10, 30.0, N_halo=N_halo)
    s = sfr.SFRBox(N_halo, N, L)
    for n in (40, N_halo ** 3 // 3, 1500, 40):
        cat = _random_catalogue(n, N_halo, seed=n + side, edges=n == 1500, discrete=n != 40)
        want, _ = oracle_lib.sfrd_box(p, z, cat)
        got, _ = s.box(z, cat)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), n
    s.close()
