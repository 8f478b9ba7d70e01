"""The pair lines at the larger sides, each with a line plan, a thread count and
shared memory of its own: the radius passes and the criterion against the
single-radius kernels (the same bits), the VJP (2e-5 of its norm: another order
of the sums), the power spectrum and the 21-cm stage against float64 (1e-5 of
the value, 1e-5 of the largest |T_b|, as at the smaller sides), and the halo
finder's bits against its fields from the single transforms (equal but within
2e-6 of the largest field value of the threshold)."""
import numpy as np
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [512, 640, 648, 768, 800, 864, 960, 1024])
def test_radius_passes(hii, N):
    import torch
    L, z, pow2 = 0.6 * N, 8.0, N & (N - 1) == 0
    delta, src = synth.make_boxes_torch(N, L, z, 300 + N)
    g = torch.rand(delta.shape, generator=torch.Generator("cuda").manual_seed(N), device="cuda")
    torch.cuda.synchronize()
    ref = None
    for kw in [dict(path=1 if pow2 else 0, kmax=1), dict(path=5 if pow2 else 0, kmax=4)]:
        fb = None
        for div in (16, 15, 14, 13):  # an odd number of radii (the last one is a cell, or just missed): a last batch of one
            if fb:
                fb.close()
            fb = hii.FilterBank(N, L, 0.71, [(30.0, L / div, 4)], **kw)
            if len(fb.radii()[0]) == 5:
                break
        assert len(fb.radii()[0]) == 5
        x, C, gd, gs = (torch.empty_like(delta) for _ in range(4))
        A = torch.empty(delta.shape, dtype=torch.uint8, device="cuda")
        p, s = (delta.data_ptr(), src.data_ptr()), torch.cuda.Stream().cuda_stream
        fb.run_z_device(z, *p, x.data_ptr(), stream=s)
        fb.criterion_device(z, *p, C.data_ptr(), A.data_ptr(), stream=s)
        gz = fb.vjp_device(z, *p, g.data_ptr(), gd.data_ptr(), gs.data_ptr(), stream=s)
        torch.cuda.synchronize()
        fb.close()
        if ref is None:
            assert (C >= 1).any() and (x < 1).any()
            ref = (x, C, A, gd, gs, gz)
            continue
        for got, want in zip((x, C, A), ref):
            assert torch.equal(got, want)
        for got, want in ((gd, ref[3]), (gs, ref[4])):
            assert (got - want).double().norm() <= 2e-5 * want.double().norm()
        assert abs(gz - ref[5]) <= 2e-5 * abs(ref[5])


@pytest.mark.parametrize("N", [640, 648, 768, 800, 864, 960])
def test_power_spectrum(hii, N):
    import torch
    from perf import cases
    case = dict(kind="pk", N=N, dl=0.3, window=1)
    k, P = cases.run(cases.prepare(case, N))
    Pr = cases.exact(case, N)[1].cpu().numpy()
    torch.cuda.empty_cache()
    np.testing.assert_allclose(k, np.arange(len(Pr)) * (2.0 * np.pi / (N * case["dl"])), rtol=1e-12)
    np.testing.assert_allclose(P, Pr, rtol=1e-5, atol=1e-8 * np.abs(Pr).max())


@pytest.mark.parametrize("N", [640, 648, 800, 864])
def test_brightness_temperature(hii, N):
    import torch
    from perf import cases
    case = dict(kind="t21", N=N, L=0.5 * N, z=9.0, axis=1 + N % 3, spin=False)
    tb, mean = cases.run(cases.prepare(case, N))
    ref, mref = cases.exact(case, N)
    assert float((torch.from_numpy(tb).cuda().double() - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert abs(mean - float(mref)) <= 1e-5 * abs(float(mref))
    del ref
    torch.cuda.empty_cache()


@pytest.mark.parametrize("N", [512, 640, 648, 800])
def test_halo_bits(hii, N):
    import torch
    from simfast21_gb300 import halos
    z = 7.0
    w = synth.HaloWorkload(N=N, L_mpc=0.2 * N, seed=N)
    cfg = halos.config_from_ini(halos.parse_ini(synth.halo_ini_text(w, z, z, 1.0)))
    gen = torch.Generator("cuda").manual_seed(N)
    d = 3.7 * torch.randn((N, N, N), generator=gen, device="cuda")
    hf = halos.HaloFinder(cfg)
    hf.set_density(d.cpu().numpy())
    del d
    assert len(hf.find_z(z)) > 0
    sch = halos.schedule(cfg, z)
    active = [m for m, s in enumerate(sch) if s["active"]]
    some = 0
    for m in active[-1:] + active[1:-1:5]:
        bits = np.unpackbits(hf.candidates(m).view(np.uint8), bitorder="little").astype(bool)
        field = hf.field(z, m).ravel()
        near = np.abs(field.astype(np.float64) - sch[m]["dcmz"]) <= 2e-6 * np.abs(field).max()
        assert not ((bits != (field > sch[m]["dcmz"])) & ~near).any()
        some += int(bits.sum())
    hf.close()
    assert some > 0
