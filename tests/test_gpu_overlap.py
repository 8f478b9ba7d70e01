"""run_z_device with the inputs inside the output range (a caller that keeps
one buffer): the same boxes as with buffers apart, with and without the captured
schedule, at a box of the output, across two of them and past its end."""
import pytest

from simfast21_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("at", [0.0, 0.5, 1.0, 2.0, 2.25])
def test_source_inside_the_outputs(hii, graph, at):
    import torch
    N, L, z = 64, 40.0, 8.0
    n3 = N ** 3
    delta, src = synth.make_boxes_torch(N, L, z, 5)
    fb = hii.FilterBank(N, L, 0.7, [(20.0, 12.0, 8), (35.0, 10.0, 8), (50.0, 8.0, 8)], graph=graph)
    st = torch.cuda.Stream()
    want = torch.empty(3 * n3, device="cuda")
    buf = torch.empty(4 * n3, device="cuda")
    part = buf[int(at * n3):][:n3]
    torch.cuda.synchronize()
    fb.run_z_device(z, delta.data_ptr(), src.data_ptr(), want.data_ptr(), stream=st.cuda_stream)
    st.synchronize()
    for what in ("src", "src", "delta"):  # the second pass replays the first one's schedule
        part.copy_((src if what == "src" else delta).ravel())
        torch.cuda.synchronize()
        d, s = (delta, part) if what == "src" else (part, src)
        fb.run_z_device(z, d.data_ptr(), s.data_ptr(), buf.data_ptr(), stream=st.cuda_stream)
        st.synchronize()
        assert torch.equal(buf[:3 * n3], want), what
    fb.close()
