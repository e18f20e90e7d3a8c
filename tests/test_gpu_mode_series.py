"""Every (l, m) of the drop-in waveform entry point on the GPU against the
oracle, with both coefficient settings of update_information
(mode_cases.py: points and bound)."""
import numpy as np
import pytest

from mode_cases import BINARIES, LM, oracle_modes, params, rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_hm", [0, 1])
@pytest.mark.parametrize("binary", BINARIES)
def test_every_mode(oracle, binary, use_hm):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pyEOB
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    par, q = params(*binary), rows()
    n = len(q)
    cls = pyEOB.SEOBNRv5Class()
    cls.update_information(*(d([v]) for v in par), use_hm, 1, None)
    r, phi, pphi, v, H, vphi = (d(q[:, k]) for k in range(6))
    out = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    ref = oracle_modes(oracle, *binary, use_hm)
    for k, (l, m) in enumerate(LM):
        cls.EOBGetSpinFactorizedWaveform(out, r, phi, torch.zeros_like(r), pphi, v, H, d([par[2]]), vphi, l, m,
                                         d([1.0, 0.0]), 0.3, 1, n, torch.zeros(1, dtype=torch.int32, device="cuda"))
        got = out.cpu().numpy().view(np.complex128)
        assert np.max(np.abs(got - ref[k])) <= 1e-12 * np.max(np.abs(ref[k])), (l, m)
