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


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_phases_that_are_no_numbers(prepared, value):
    """A phase that is no number makes that binary's likelihood NaN, as in FP64, and no other's."""
    torch, _lib, wl, data = prepared
    v = wl.views()
    off = wl._dev_array(v.row_off, 4, torch.int64).cpu().numpy()
    phase = wl._dev_array(v.spline_y, int(v.rows_capacity), torch.float64)
    before = _lnl(wl, data)
    at = int(off[1]) + 5
    keep = phase[at].item()
    phase[at] = value
    try:
        mixed, full = _lnl(wl, data), _lnl(wl, data, 0)
    finally:
        phase[at] = keep
    assert np.isnan(mixed).tolist() == np.isnan(full).tolist() == [False, True, False]
    np.testing.assert_array_equal(mixed[[0, 2]], before[[0, 2]])
