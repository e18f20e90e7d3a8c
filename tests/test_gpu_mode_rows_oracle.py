"""The fused path's multipoles, every (l, m), l <= 8, on every trajectory row
against the oracle's evaluation (which shares no code with theirs but the
coefficient builder), on ordinary rows (closed form) and on rows within 0.2 M of a
neighbour (log-Gamma sums), equal masses among the binaries.  The oracle takes v,
H_real and the v_phi input from the drop-in Hamiltonian at the row's state.

Bound: 1e-12 of each mode's peak for the evaluation (mode_cases.py), and the
rounding of phases m phi in the oracle's e^{-i m phi} and in the rotation here, 2^-52 m
max|phi|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LM = [(l, m) for l in range(2, 9) for m in range(1, l + 1)]
P = np.array([[30.0, 30.0, 0.3, -0.2, 20.0], [45.0, 15.0, 0.5, 0.4, 20.0], [20.0, 18.0, -0.6, 0.1, 25.0]])


@pytest.mark.parametrize("group", range(7))
def test_tables_match_the_oracle(oracle, group):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pyEOB
    from eobgpu_gb300.eob.seobnrv4phm import SEOBNRv4PHM
    from eobgpu_gb300.pipeline import WaveformLikelihood
    modes = LM[5 * group:5 * group + 5]
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    B = len(P)
    wl = WaveformLikelihood(B, 4000, modes, 1024)
    wl.prepare(d(P), 1.0 / 2048)
    nsteps, _, status, trajs = wl.trajectories()
    assert np.all(status == 0)
    v = wl.views()
    rc = int(v.rows_capacity)
    off = wl._dev_array(v.row_off, B + 1, torch.int64).cpu().numpy()
    tab = wl._dev_array(v.spline_y, 11 * rc, torch.float64).view(-1, rc)[:, :off[-1]].cpu().numpy()
    for b, (t, y) in enumerate(trajs):
        n = len(t)
        m1, m2 = P[b, 0] / (P[b, 0] + P[b, 1]), P[b, 1] / (P[b, 0] + P[b, 1])
        one = lambda x: d(np.full(n, x))
        gen = SEOBNRv4PHM()
        gen.setup_class(one(m1), one(m2), one(P[b, 2]), one(P[b, 3]), one(1.0))
        add = gen.additionalArgs.contiguous()

        def grad(pr):
            g = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
            pyEOB.grad_Ham_align_AD(d(np.concatenate([y[:, 0], y[:, 1], pr, y[:, 3]])), g, add, n)
            return g.cpu().numpy().reshape(4, n)

        H = torch.zeros(n, dtype=torch.float64, device="cuda")
        a = add.view(-1, n)
        K, d5, dSO, dSS = (float(a[5 + q, 0]) for q in range(4))
        pyEOB.evaluate_Ham_align_AD(H, *(d(y[:, q]) for q in range(4)), a[0].contiguous(), a[1].contiguous(),
                                    a[2].contiguous(), a[3].contiguous(), K, d5, dSO, dSS, n)
        nu = m1 * m2
        omega, omega_c = grad(y[:, 2])[3], grad(0.0 * y[:, 2])[3]
        r = y[:, 0]
        ctx = oracle.context(np.array([m1]), np.array([m2]), P[b, 2:3], P[b, 3:4])
        lm = list(zip(gen.l_vals, gen.m_vals))
        pre = gen.prefixes.cpu().numpy()[:, 0]
        dt = np.diff(t)
        close = np.zeros(n, dtype=bool)
        close[1:] |= dt < 0.2
        close[:-1] |= dt < 0.2
        assert close.any() and not close.all()
        for k, (l, m) in enumerate(modes):
            h = ctx.waveform(r, y[:, 1], y[:, 2], y[:, 3], np.cbrt(omega), nu * H.cpu().numpy(), nu,
                             1.0 / (omega_c ** 2 * r ** 3), l, m, pre[lm.index((l, m))])
            want = h * np.exp(1j * m * y[:, 1])
            got = tab[1 + 2 * k, off[b]:off[b + 1]] + 1j * tab[2 + 2 * k, off[b]:off[b + 1]]
            bound = (1e-12 + 2.0 ** -52 * m * np.max(np.abs(y[:, 1]))) * np.max(np.abs(want))
            for rows in (close, ~close):
                assert np.max(np.abs(got - want)[rows]) <= bound, (b, l, m)
