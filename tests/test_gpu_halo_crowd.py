"""The halo deposit of catalogues with many halos in a cell, on grids that go by
tiles: the bits of the CPU restatement, whatever the crowd's place in its tile,
beside other crowds and among other halos; and no longer a time than a halo of
the chain takes by the fine grid (0.44 us), with some room."""
import numpy as np
import pytest

from test_gpu_sfr import _random_catalogue

pytestmark = pytest.mark.gpu


def _crowded(n, N_halo, kind, seed):
    cat = _random_catalogue(n, N_halo, seed=seed, edges=False, discrete=seed % 2 == 0)
    rng = np.random.default_rng(seed)
    for ax in ("x", "y", "z"):
        p = {"cell": 9.0 + rng.random(n), "edge": 7.5 + rng.random(n), "corner": N_halo - 0.5 + rng.random(n),
             "faces": 11.0 + 0.0 * rng.random(n), "two": 20.0 + rng.random(n) + 3.0 * rng.integers(0, 2, n)}[kind]
        crowd = np.arange(n) % 7 != 0
        cat[ax] = np.where(crowd, (p % N_halo).astype(np.float32), cat[ax])
    cat["Mass"][::50] = 0.0
    return cat


@pytest.mark.parametrize("kind", ["cell", "edge", "corner", "faces", "two"])
@pytest.mark.parametrize("side", [1, 2, 3, 4])
def test_bits(hii, oracle_lib, kind, side):
    from simfast21_gb300 import sfr
    N_halo, L, z = 132, 20.0, 8.0
    N = N_halo // side
    p = oracle_lib.params(N, L, 0.71, L / 2, 10, 30.0, N_halo=N_halo)
    s = sfr.SFRBox(N_halo, N, L)
    for n in (3000, 97, 25):
        cat = _crowded(n, N_halo, kind, n + side)
        want, _ = oracle_lib.sfrd_box(p, z, cat)
        got, _ = s.box(z, cat)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), n
    s.close()


def test_time(hii):
    import torch
    from simfast21_gb300 import sfr
    N_halo, n = 480, 40000
    cat = torch.rand((n, 4), generator=torch.Generator("cuda").manual_seed(1), device="cuda") + 9.0
    cat[:, 0] = 1e9
    out = torch.empty((240,) * 3, device="cuda")
    s, st, best = sfr.SFRBox(N_halo, 240, 100.0), torch.cuda.Stream(), 1e9
    torch.cuda.synchronize()
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        s.box_device(8.0, n, cat.data_ptr(), out.data_ptr(), st.cuda_stream)
        b.record(st)
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    s.close()
    assert best < 0.6e-3 * n
