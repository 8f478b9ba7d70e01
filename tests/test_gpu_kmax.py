"""Contexts with a given number of radii per batch hold that many work boxes,
and pipeline 5 gives the same boxes whatever the number: pairs of radii for an
even one, pairs of one less for an odd one, single radii for one."""
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, path", [(128, 5), (128, 0), (120, 0)])
def test_work_boxes(hii, N, path):
    import torch
    torch.cuda.synchronize()
    hii.FilterBank(N, 60.0, 0.7, [(30.0, 15.0, 9)], kmax=8, path=path).close()  # the kernels' own memory
    used = []
    for k in range(1, 9):
        free = torch.cuda.mem_get_info()[0]
        fb = hii.FilterBank(N, 60.0, 0.7, [(30.0, 15.0, 9)], kmax=k, path=path)
        used.append(free - torch.cuda.mem_get_info()[0])
        assert fb.batch_radii() == k
        fb.close()
    box, grain = 8 * N ** 3, 4 << 20  # allocations come in pages of 2 MB
    for k in range(1, 8):
        assert abs(used[k] - used[k - 1] - box) <= grain, used


@pytest.mark.parametrize("N", [16, 32, 64, 128, 256])
def test_pipeline_5_whatever_the_batch(hii, N):
    import torch
    L, z = 0.6 * N, 8.0
    delta, src = synth.make_boxes_torch(N, L, z, N)
    d, s = delta.cpu().numpy(), src.cpu().numpy()
    ref = None
    for kw in [dict(path=1), dict(path=5, kmax=1), dict(path=5, kmax=2), dict(path=5, kmax=3), dict(path=5, kmax=7)]:
        fb = hii.FilterBank(N, L, 0.71, [(30.0, L / 4, 12)], **kw)
        x = torch.empty((N, N, N), device="cuda")
        torch.cuda.synchronize()
        fb.run_z_device(z, delta.data_ptr(), src.data_ptr(), x.data_ptr())
        fb.check()
        got = (x, *(torch.from_numpy(a) for a in fb.criterion(z, d, s)))
        fb.close()
        ref = ref or got
        assert all(torch.equal(a, b) for a, b in zip(got, ref)), kw
