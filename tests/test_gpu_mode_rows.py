"""The fused path's multipoles on every trajectory row -- the closed form on
ordinary rows, the log-Gamma sums on the fine pass's -- against the
reference-shaped compute_hlms on the same rows, rotated by e^{i m phi}: one
function, within 1e-12 of each mode's peak (its evaluations round at 2e-14, the
rotation at eps of phases up to 1e3 rad, 2e-13)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = [(2, 2), (2, 1), (3, 3), (4, 4), (5, 5)]


@pytest.mark.parametrize("modes", [MODES[:1], MODES, [(8, 8), (7, 6), (3, 1)]])
@pytest.mark.parametrize("batch", [1, 7])
def test_tables_match_compute_hlms(modes, batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300 import workload
    from eobgpu_gb300.eob.seobnrv4phm import SEOBNRv4PHM
    from eobgpu_gb300.pipeline import WaveformLikelihood
    params = workload.draw_params(workload.CONFIGS[2], batch, stream=31)
    P = torch.tensor(params, device="cuda")
    wl = WaveformLikelihood(batch, 6000, modes, 1024)
    wl.prepare(P, 1.0 / 2048)
    nsteps, _, status, trajs = wl.trajectories()
    assert np.all(status == 0)
    v = wl.views()
    rc = int(v.rows_capacity)
    off = wl._dev_array(v.row_off, batch + 1, torch.int64).cpu().numpy()
    tab = wl._dev_array(v.spline_y, (1 + 2 * len(modes)) * rc, torch.float64).view(-1, rc)[:, :off[-1]].cpu().numpy()
    m1, m2 = P[:, 0] / (P[:, 0] + P[:, 1]), P[:, 1] / (P[:, 0] + P[:, 1])
    gen = SEOBNRv4PHM()
    gen.setup_class(m1, m2, P[:, 2], P[:, 3], torch.ones_like(m1))
    cls, lm = gen.eob_c_class, list(zip(gen.l_vals, gen.m_vals))
    pre = gen.prefixes[[lm.index(x) for x in modes]]  # [K][B]
    cls.newtonian_prefixes = torch.view_as_real(pre.contiguous()).contiguous().reshape(-1)
    K, L = len(modes), int(nsteps.max())
    y = np.zeros((4, batch, L))
    for b, (t, yy) in enumerate(trajs):
        y[:, b, :len(t)] = yy.T
    cols = [torch.tensor(np.ascontiguousarray(a).reshape(-1), device="cuda") for a in y]
    i32 = lambda a: torch.tensor(np.asarray(a, dtype=np.int32), device="cuda")
    out = torch.zeros(2 * batch * K * L, dtype=torch.float64, device="cuda")
    cls.compute_hlms(out, *cols, m1.contiguous(), m2.contiguous(), P[:, 2].contiguous(), P[:, 3].contiguous(),
                     i32(nsteps), L, i32([l for l, _ in modes]), i32([m for _, m in modes]), K, batch,
                     gen.additionalArgs.contiguous(), gen.num_add_args_total)
    ref = out.cpu().numpy().view(np.complex128).reshape(batch, K, L)
    kinds = set()
    for b, (t, yy) in enumerate(trajs):
        n = int(nsteps[b])
        kinds.update((np.diff(t) < 0.04).tolist())
        for k, (l, m) in enumerate(modes):
            got = tab[1 + 2 * k, off[b]:off[b + 1]] + 1j * tab[2 + 2 * k, off[b]:off[b + 1]]
            want = ref[b, k, :n] * np.exp(1j * m * yy[:, 1])
            assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want)), (b, l, m)
    assert kinds == {True, False}
