"""Halo finder at box sides with every way the a-axis pass stores its bits
(runs of one, two and four tiles of eight columns, several tiles per CTA,
outputs per thread that are no multiple of eight) and a subgrid cycle whose
draws take one uniform, a few, and more than a lane's segment of positions:
the oracle's serial loop on the GPU's candidates gives the same bytes."""
import numpy as np
import pytest

from simfast21_gb300 import synth
from test_gpu_halos import H, _check_case  # noqa: F401  (H: the fixture)

pytestmark = pytest.mark.gpu


def _case(N, cell, zs, **kw):
    w = synth.HaloWorkload(N=N, L_mpc=N * cell, seed=N, **kw)
    return {"ini": synth.halo_ini_text(w, min(zs), max(zs), 1.0), "delta": w.density().reshape((N,) * 3),
            "zs": np.array(zs)}


@pytest.mark.parametrize("N", [32, 40, 48, 72, 80, 144])
def test_bit_sets(H, N):  # noqa: F811
    rep = _check_case(H, f"n{N}", g=_case(N, 0.2, [7.0], sigma=3.7))
    assert rep[0][1] > 0


@pytest.mark.parametrize("cell, Mmin", [(0.3, 1e8), (0.6, 1e8), (1.2, 1e8)])
def test_subgrid_means(H, cell, Mmin):  # noqa: F811
    """Means per cell from well under one up to several (the cycle refuses more than 10)."""
    rep = _check_case(H, f"cell {cell}", g=_case(40, cell, [6.0, 8.0], sigma=1.5, subgrid=True, Mmin=Mmin))
    assert rep[0][1] > 0
