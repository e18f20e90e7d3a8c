"""A ringdown amplitude that is no number reaches the strain: with the
argument of its tanh broken in one binary's attachment record, that binary's
ringdown samples are NaN (the inspiral and the other binary as before).

The records lie behind the workspace's part without the merger-ringdown:
five pairs of spline planes (rows doubles each, 256-byte aligned), then 15
doubles per binary and mode (a1 a2 a3 b1 b2 c1c c2c c1f c2f d1c d1f d2f
phi_match om_re om_im), and eta."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_broken_amplitude():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300 import _lib, workload
    from eobgpu_gb300.pipeline import WaveformLikelihood
    opt = _lib.default_options()
    opt.imr = 1
    B, rows, N, dt = 2, 4000, 16384, 1.0 / 4096
    params = workload.draw_params(workload.CONFIGS[1], B, stream=13)
    wl = WaveformLikelihood(B, rows, [(2, 2)], N, options=opt)
    wl.prepare(torch.tensor(params, device="cuda"), dt)
    h, status = wl.synth_strain(B, dt, N, per_mode=True)
    assert int(status.abs().max()) == 0
    h = h.cpu().numpy()[:, 0]
    plane = (16 * B * rows + 255) // 256 * 256
    at = int(wl.lib.eob_workspace_bytes(B, rows, 1, N)) + 5 * plane
    rec = wl.ws[at:at + 128 * B].view(torch.float64).view(B, 16)
    eta = params[:, 0] * params[:, 1] / (params[:, 0] + params[:, 1]) ** 2
    np.testing.assert_allclose(rec[:, 15].cpu().numpy(), eta, rtol=1e-12)
    rec[1, 8] = float("nan")  # c2f
    g = wl.synth_strain(B, dt, N, per_mode=True)[0].cpu().numpy()[:, 0]
    np.testing.assert_array_equal(g[0], h[0])
    bad = np.isnan(g[1])
    assert bad.any()
    first = int(np.argmax(bad))
    np.testing.assert_array_equal(g[1][:first], h[1][:first])  # the inspiral
    last = int(np.argmax(np.abs(h[1]) > 0) + np.count_nonzero(h[1]) - 1)
    assert bad[first:last + 1].all() and last - first > 10
