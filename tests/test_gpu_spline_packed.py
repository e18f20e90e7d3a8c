"""The fused path's splines against the oracle's serial sweep on trajectories of
every launch's range: one tile of the short blocks (up to 576 rows), one tile of
the long ones, and several tiles (above 2304 rows).

Each coefficient's contribution over its interval is held to 1e-12 of the
series' scale, as for the drop-in builder (test_gpu_spline.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes", [[(2, 2)], [(2, 2), (3, 3), (4, 4)]])
def test_tables_of_every_length(oracle, modes):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.pipeline import WaveformLikelihood
    P = np.array([[50.0, 40.0, 0.1, -0.2, 20.0], [8.0, 2.0, 0.3, 0.2, 8.0], [25.0, 15.0, 0.0, 0.1, 15.0],
                  [80.0, 60.0, -0.1, 0.2, 20.0], [16.0, 4.0, 0.5, -0.5, 10.0]])
    B, K = len(P), len(modes)
    wl = WaveformLikelihood(B, 16000, modes, 1024)
    wl.prepare(torch.tensor(P, device="cuda"), 1.0 / 2048)
    nsteps, _, status, _ = wl.trajectories()
    assert np.all(status == 0)
    assert np.any(nsteps <= 576) and np.any((nsteps > 576) & (nsteps <= 2304)) and np.any(nsteps > 2304)
    v = wl.views()
    rc = int(v.rows_capacity)
    off = wl._dev_array(v.row_off, B + 1, torch.int64).cpu().numpy()
    plane = lambda a: wl._dev_array(a, (1 + 2 * K) * rc, torch.float64).view(-1, rc)[:, :off[-1]].cpu().numpy()
    y, c = plane(v.spline_y), [plane(a) for a in (v.spline_c1, v.spline_c2, v.spline_c3)]
    x = wl._dev_array(v.tin, rc, torch.float64)[:off[-1]].cpu().numpy()
    for b, n in enumerate(nsteps):
        t = x[off[b]:off[b + 1]]
        dx = np.diff(t)
        for s in range(1 + 2 * K):
            yb = y[s, off[b]:off[b + 1]].copy()
            ref = oracle.interpolate_td(t.copy(), yb, [n], 1, 1)
            scale = np.max(np.abs(yb))
            for p, (g, r) in enumerate(zip(c, ref), 1):
                assert np.max(np.abs(g[s, off[b]:off[b] + n - 1] - r[:n - 1]) * dx ** p) <= 1e-12 * scale, (b, s, p)
