"""`order` is the integrator's queue order alone: the multipoles and splines
(stages = 4) build every binary's tables whatever it holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tables_do_not_read_the_order():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300 import workload
    from eobgpu_gb300.pipeline import WaveformLikelihood
    B = 6
    P = torch.tensor(workload.draw_params(workload.CONFIGS[1], B, stream=9), device="cuda")
    wl = WaveformLikelihood(B, 4000, [(2, 2)], 1024)
    wl.prepare(P, 1.0 / 1024)
    rows = wl.counters()["rows"]
    v = wl.views()
    rc = int(v.rows_capacity)
    planes = [wl._dev_array(a, 3 * rc, torch.float64).view(3, rc)[:, :rows] for a in
              (v.spline_c1, v.spline_c2, v.spline_c3)]
    ref = [p.clone() for p in planes]
    for p in planes:
        p.zero_()
    wl.prepare(P, 1.0 / 1024, order=torch.zeros(B, dtype=torch.int32, device="cuda"), stages=4)
    for p, r in zip(planes, ref):
        np.testing.assert_array_equal(p.cpu().numpy(), r.cpu().numpy())
