"""The halo deposit by tiles against the CPU restatement, bit for bit: one,
two and many tiles per axis, block sides up to the largest that has tiles and
the first that keeps the fine grid, grids that the blocks do not cover, tiles
with more halos than threads (spread over the runs, in one run, in one cell)
and coordinates outside the grid."""
import numpy as np
import pytest

from test_gpu_sfr import _random_catalogue

pytestmark = pytest.mark.gpu


def _crowd(cat, N_halo, kind):
    n = len(cat)
    rng = np.random.default_rng(n)
    lo, side = {"tile": (2.0, 12.0), "edges": (7.5, 1.0), "cell": (9.25, 0.5), "outside": (-1.5, N_halo + 3.0)}[kind]
    for ax in ("x", "y", "z"):
        cat[ax][: n // 2] = (lo + side * rng.random(n // 2)).astype(np.float32)
    return cat


@pytest.mark.parametrize("N_halo,N", [(8, 8), (16, 8), (33, 11), (40, 16), (55, 5), (64, 4), (68, 4), (90, 45)])
@pytest.mark.parametrize("kind", ["tile", "edges", "cell", "outside"])
def test_tiles(hii, oracle_lib, N_halo, N, kind):
    from simfast21_gb300 import sfr
    L, z = 20.0, 8.0
    cat = _crowd(_random_catalogue(3000, N_halo, seed=N_halo, edges=False, discrete=N_halo % 2 == 0), N_halo, kind)
    want, _ = oracle_lib.sfrd_box(oracle_lib.params(N, L, 0.71, L / 2, 10, 30.0, N_halo=N_halo), z, cat)
    s = sfr.SFRBox(N_halo, N, L)
    got, _ = s.box(z, cat)
    again, _ = s.box(z, cat[::-1].copy())  # another order is another chain, on the same scratch
    back, _ = s.box(z, cat)
    s.close()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(back.view(np.uint32), want.view(np.uint32))
    np.testing.assert_allclose(again, want, rtol=1e-3)
