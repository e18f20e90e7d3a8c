"""Caller memory aligned to its element size only (8 bytes), in paths that load
16 bytes at a time: the same values as from memory of the allocator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("nch", [1, 8])
@pytest.mark.parametrize("B", [3, 32])  # block partials that fill their section to the last byte (32 x 8), or not
def test_fd_scratch(torch_cuda, nch, B):
    torch = torch_cuda
    from eobgpu_gb300 import _lib, fd
    N, n = 4096, 2049
    rng = np.random.default_rng(B)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    H = d(rng.normal(size=(B, N, 2)))
    data = d(rng.normal(size=(nch, n)) + 1j * rng.normal(size=(nch, n)))
    psd = d(rng.uniform(0.5, 2.0, (nch, n)))
    net = [d(rng.uniform(-0.02, 0.02, (nch, B))) for _ in range(3)]
    need = int(_lib.load().eob_fd_lnl_scratch_bytes(B, N))
    out = []
    for shift in (0, 8):
        scratch = torch.zeros(need + 16, dtype=torch.uint8, device="cuda")[shift:shift + need]
        assert scratch.data_ptr() % 16 == shift
        out.append(fd.fd_lnl_from_fft(H, data, psd, *net, 0.25, 0, scratch).cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])


def test_workspace_mixed_precision(torch_cuda):
    """The FP32 copies of the splines, written and read as vectors where the workspace allows it."""
    torch = torch_cuda
    from eobgpu_gb300 import _lib, workload
    from eobgpu_gb300.pipeline import WaveformLikelihood
    P = torch.tensor(workload.draw_params(workload.CONFIGS[1], 5, stream=3), device="cuda")
    data = torch.tensor(np.random.default_rng(1).normal(size=4096), device="cuda")
    opt = _lib.default_options()
    opt.precision = 1
    out = []
    for shift in (0, 8):
        wl = WaveformLikelihood(5, 4000, [(2, 2), (3, 3)], 4096, options=opt)
        buf = torch.zeros(wl.ws_bytes + 16, dtype=torch.uint8, device="cuda")
        wl.ws = buf[shift:shift + wl.ws_bytes]
        assert wl.ws.data_ptr() % 16 == shift
        lnl, status = wl.run(P, data, 1.0 / 1024, 20.0)
        h, _ = wl.strain(P, 1.0 / 1024, 4096)
        assert int(status.abs().max()) == 0
        out.append((lnl.cpu().numpy(), h.cpu().numpy()))
        # the last bytes of the workspace's neighbours are untouched
        assert int(buf[:shift].sum()) == 0 and int(buf[shift + wl.ws_bytes:].sum()) == 0
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
