"""The mixed-precision likelihood beyond the ordinary phases and modes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prepared():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300 import _lib, workload
    from eobgpu_gb300.pipeline import WaveformLikelihood
    opt = _lib.default_options()
    opt.precision = 1
    P = torch.tensor(workload.draw_params(workload.CONFIGS[1], 3, stream=21), device="cuda")
    wl = WaveformLikelihood(3, 4000, [(2, 2)], 8192, options=opt)
    wl.prepare(P, 1.0 / 1024)
    data = torch.tensor(np.random.default_rng(2).normal(size=8192), device="cuda")
    return torch, _lib, wl, data


def _lnl(wl, data, precision=1):
    wl.options.precision = precision
    lnl, status = wl.synth_lnl(3, data, 1.0 / 1024, 20.0)
    wl.options.precision = 1
    assert int(status.abs().max()) == 0
    return lnl.cpu().numpy()


def test_negative_m(prepared):
    """The synthesis takes any m.  FP32 amplitudes, sines and residuals: 1e-5 of the likelihood."""
    torch, _lib, wl, data = prepared
    wl.mms[0] = -2
    try:
        mixed, full = _lnl(wl, data), _lnl(wl, data, 0)
    finally:
        wl.mms[0] = 2
    np.testing.assert_allclose(mixed, full, rtol=1e-5)
