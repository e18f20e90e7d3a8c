"""The work that users of this framework have it do, as measurable cases.

Each case is one call (or one stage of the batched path) through the public
entry points: the fused likelihood of a batch, its stages on a prepared
workspace (multipoles and splines, synthesis + likelihood, strain), the
frequency-domain likelihood, and the drop-in `eob` functions.

  listed()            the cases that are timed
  draw(rng)           another case from the same ranges
  prepare(case, seed) what a program holds before the call, on the GPU
  run(state)          one pass; returns its outputs
  work(case)          bytes and floating-point operations a pass cannot do without
  exact(case, seed)   what run returns, by plain torch in 64 bits (None where the
                      outputs have no such closed evaluation)
"""
from __future__ import annotations

import math

import numpy as np
import torch

MTSUN = 4.925491025543576e-06
MODES5 = ((2, 2), (2, 1), (3, 3), (4, 4), (5, 5))
# trajectory rows a workspace holds per binary, and right-hand sides an
# average binary needs, by population (the workload module's configurations)
ROWS = {1: 4000, 2: 6000}
MEAN_ROWS = {1: 520, 2: 680}
MEAN_RHS = {1: 6500.0, 2: 7600.0}
RHS_FLOPS = 1533.0  # one right-hand side of the equations of motion


def listed():
    return [
        # one likelihood call of a small sampler: 8 binaries, (2,2), 8 s of data
        dict(name="lnl_small", kind="lnl", pop=1, batch=8, modes=1, samples=8192, rate=1024, mixed=False),
        # the flagship: 1024 binaries whose lengths differ by about 100x
        dict(name="lnl_ragged", kind="lnl", pop=2, batch=1024, modes=1, samples=131072, rate=2048, mixed=False),
        # multipoles on the trajectories and their splines: the ragged batch, (2,2)
        dict(name="tables_ragged", kind="tables", pop=2, batch=1024, modes=1, samples=131072, rate=2048, mixed=False),
        # the same for a large batch with every higher mode, mixed precision
        dict(name="tables_modes", kind="tables", pop=1, batch=4096, modes=5, samples=131072, rate=2048, mixed=True),
        # synthesis + likelihood of the ragged batch in FP64 (new data on the same templates)
        dict(name="synth_ragged", kind="synth", pop=2, batch=1024, modes=1, samples=131072, rate=2048, mixed=False),
        # synthesis + likelihood of the large five-mode batch, mixed precision
        dict(name="synth_modes", kind="synth", pop=1, batch=4096, modes=5, samples=131072, rate=2048, mixed=True),
        # the waveform generator's per-mode output with the merger-ringdown attached
        dict(name="strain_modes", kind="strain", pop=1, batch=64, modes=5, samples=24576, rate=4096, imr=True),
        # the drop-in spline builder on a batch of trajectories, five modes
        dict(name="spline_td", kind="spline", batch=512, modes=5, rows=700),
        # the drop-in mode synthesis on a uniform time grid
        dict(name="tdinterp", kind="tdinterp", batch=128, modes=2, rows=700, samples=32768),
        # the detector-network likelihood of a batch from the templates' FFTs
        dict(name="fd_network", kind="fd", batch=512, samples=65536, channels=3),
        # the drop-in frequency-domain residual (two polarisations given)
        dict(name="fd_dropin", kind="allinone", batch=96, bins=30721, channels=2),
        # the drop-in equations of motion for a batch of walkers
        dict(name="ode", kind="ode", batch=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lnl", "tables", "synth", "strain", "spline", "tdinterp", "fd", "allinone", "ode"])
    if kind in ("lnl", "tables", "synth"):
        pop = rng.choice([1, 2])
        return dict(kind=kind, pop=pop, batch=_log_int(rng, 1, 1024 if pop == 1 else 384),
                    modes=rng.choice([1, 2, 3, 5]), samples=_log_int(rng, 4096, 131072),
                    rate=rng.choice([1024, 2048, 4096]), mixed=rng.choice([False, True]))
    if kind == "strain":
        return dict(kind=kind, pop=1, batch=_log_int(rng, 1, 128), modes=rng.choice([1, 2, 5]),
                    samples=_log_int(rng, 4096, 32768), rate=rng.choice([1024, 2048, 4096]),
                    imr=rng.choice([False, True]))
    if kind == "spline":
        return dict(kind=kind, batch=_log_int(rng, 1, 1024), modes=rng.choice([1, 2, 5]), rows=_log_int(rng, 40, 3000))
    if kind == "tdinterp":
        return dict(kind=kind, batch=_log_int(rng, 1, 256), modes=rng.choice([1, 2, 3, 5]),
                    rows=_log_int(rng, 100, 1500), samples=_log_int(rng, 2048, 65536))
    if kind == "fd":
        return dict(kind=kind, batch=_log_int(rng, 1, 512), samples=2 * _log_int(rng, 2048, 65536),
                    channels=rng.randint(1, 4))
    if kind == "allinone":
        return dict(kind=kind, batch=_log_int(rng, 1, 128), bins=_log_int(rng, 1025, 65537),
                    channels=rng.randint(1, 4))
    return dict(kind="ode", batch=_log_int(rng, 1, 16384))


# ---------------------------------------------------------------- inputs


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _params(case, seed):
    """(m1, m2, chi1, chi2, f0) of the batch, drawn from the population's prior."""
    from eobgpu_gb300 import workload
    cfg = workload.CONFIGS[case["pop"]]
    return torch.tensor(workload.draw_params(cfg, case["batch"], stream=100000 + int(seed)), device="cuda")


def _engine(case, batch=None):
    from eobgpu_gb300 import _lib
    from eobgpu_gb300.pipeline import WaveformLikelihood
    opt = _lib.default_options()
    opt.precision = 1 if case.get("mixed") else 0
    opt.imr = 1 if case.get("imr") else 0
    return WaveformLikelihood(case["batch"] if batch is None else batch, ROWS[case["pop"]],
                              MODES5[:case["modes"]], case["samples"], options=opt)


def _data(case, seed, params):
    """White noise with the batch's first binary injected at SNR 30: (data, amplitude)."""
    h, _ = _engine(case, 1).strain(params[:1].contiguous(), 1.0 / case["rate"], case["samples"])
    h = h[0].real
    amp = 30.0 / float(torch.sqrt((h * h).sum()))
    return amp * h + _normal(_generator(seed, 7), case["samples"]), amp


def _prepared(case, seed):
    from eobgpu_gb300.pipeline import longest_first
    params = _params(case, seed)
    wl = _engine(case)
    order = longest_first(params)
    wl.prepare(params, 1.0 / case["rate"], order=order)
    return wl, params, order


def _table_rows(case):
    """Rows the packed tables of a batch may take: the average and a margin."""
    B, pop = case["batch"], case["pop"]
    margin = {1: 500, 2: 2500}[pop] * math.sqrt(B)
    return min(B * ROWS[pop], int(1.3 * B * MEAN_ROWS[pop] + margin))


def _tables(wl, batch, modes, rows):
    """The last prepare's knot times, spline tables and sample counts, as views
    of the workspace (`rows` packed rows of each series)."""
    v = wl.views()
    base, rc = wl.ws.data_ptr(), int(v.rows_capacity)

    def at(addr, count, dtype):
        off = int(addr) - base
        return wl.ws[off:off + count * torch.empty(0, dtype=dtype).element_size()].view(dtype)

    ns = 1 + 2 * modes
    out = dict(t=at(v.tin, rows, torch.float64), samples=at(v.npts, batch, torch.int32))
    for name, addr in (("y", v.spline_y), ("c1", v.spline_c1), ("c2", v.spline_c2), ("c3", v.spline_c3)):
        out[name] = at(addr, ns * rc, torch.float64).view(ns, rc)[:, :rows]
    return out, at(v.row_off, batch + 1, torch.int64)


def _chirp(case, seed):
    """Knot times [B, L] (ragged: L_b of them), and the real and imaginary mode
    amplitudes and the orbital phase as functions of the time to coalescence,
    with three derivatives: arrays [4][B, 2 K + 1, L] (value and Taylor
    coefficients), series in the order Re h_k, Im h_k, phase."""
    B, K, L = case["batch"], case["modes"], case["rows"]
    g = _generator(seed, 11)
    lens = (L * _uniform(g, B, 0.6, 1.0)).long().clamp(min=8)
    lens[int(torch.randint(B, (1,), generator=g, device="cuda"))] = L
    span = _uniform(g, B, 0.5, 1.0) * 4.0 * case.get("samples", 16 * L)
    j = torch.arange(L, device="cuda", dtype=torch.float64)[None, :]
    left = ((lens[:, None] - j) / lens[:, None].double()).clamp(min=0.0)
    step = 1.0 + 0.05 * torch.rand(B, L, generator=g, device="cuda", dtype=torch.float64)
    t = span[:, None] * (1.0 - left ** 3) + 0.2 * torch.cumsum(step, 1)
    t = t - t[:, :1]
    ahead = (span + 0.22 * L + 30.0)[:, None] - t  # time to coalescence
    eta = _uniform(g, B, 0.15, 0.25)[:, None]

    def power(c, p):
        return [c * ahead ** p, -c * p * ahead ** (p - 1), c * p * (p - 1) / 2 * ahead ** (p - 2),
                -c * p * (p - 1) * (p - 2) / 6 * ahead ** (p - 3)]

    parts = [[], [], [], []]
    for k in range(2 * K):
        f = power(_uniform(g, B, -1.0, 1.0)[:, None] / (1 + k // 2), -0.25 * (1 + k // 2))
        for a, b in zip(parts, f):
            a.append(b)
    f = power(-(eta / 5.0) ** 0.625 / eta, 0.625)
    for a, b in zip(parts, f):
        a.append(b)
    return t, lens, [torch.stack(p, 1) for p in parts]


def _psd(n, df, channels, g):
    f = torch.arange(n, device="cuda", dtype=torch.float64) * df
    s = 1e-46 * ((f.clamp(min=10.0) / 30.0) ** -4.2 + 0.5 + 0.5 * (f / 200.0) ** 2)
    s = s[None, :] * _uniform(g, channels, 0.7, 1.5)[:, None]
    s[:, f < 20.0] = 1e300  # as infinite entries are stored
    return s.contiguous()


def _chirp_fft(B, N, rate, g):
    """Complex FFT of h_+ + i h_x of B chirps of strain about 1e-22 in N samples."""
    t = torch.arange(N, device="cuda", dtype=torch.float64)[None, :] / rate
    end = _uniform(g, B, 0.5, 0.98)[:, None] * (N / rate)
    chirp = _uniform(g, B, 300.0, 900.0)[:, None]
    a = 1e-22 * _uniform(g, B, 0.3, 1.0)[:, None]
    out = torch.empty(B, N, dtype=torch.complex128, device="cuda")
    for lo in range(0, B, 64):
        s = slice(lo, min(B, lo + 64))
        left = (end[s] - t).clamp(min=2e-3)
        h = torch.polar(a[s] * left ** -0.25, chirp[s] * left ** 0.625)
        h[t.expand_as(h) > end[s]] = 0.0
        out[s] = torch.fft.fft(h, dim=-1) / rate
    return out


def _noise_fd(psd, df, g):
    sd = torch.where(psd > 1e200, torch.zeros_like(psd), torch.sqrt(psd / (4.0 * df)))
    return torch.complex(sd * _normal(g, *psd.shape), sd * _normal(g, *psd.shape))


def _network(B, channels, g):
    return (_uniform(g, channels * B, -1.0, 1.0), _uniform(g, channels * B, -1.0, 1.0),
            _uniform(g, channels * B, -0.021, 0.021))


def _split(H):
    N = H.shape[-1]
    n = N // 2 + 1
    z = torch.conj(H[..., (N - torch.arange(n, device=H.device)) % N])
    a = H[..., :n]
    return 0.5 * (a + z), (a - z) / 2j


# ---------------------------------------------------------------- prepare


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "lnl":
        s["params"] = _params(case, seed)
        s["wl"] = _engine(case)
        s["data"], s["amp"] = _data(case, seed, s["params"])
    elif kind == "tables":
        s["wl"], s["params"], s["order"] = _prepared(case, seed)
        s["out"], _ = _tables(s["wl"], case["batch"], case["modes"], _table_rows(case))
        used = s["wl"].counters()["rows"]
        for name in ("t", "y", "c1", "c2", "c3"):  # packed rows past the batch's own hold nothing
            s["out"][name][..., used:] = 0.0
    elif kind == "synth":
        s["wl"], s["params"], _ = _prepared(case, seed)
        s["data"], s["amp"] = _data(case, seed, s["params"])
    elif kind == "strain":
        s["wl"], s["params"], _ = _prepared(case, seed)
    elif kind == "spline":
        t, lens, parts = _chirp(case, seed)
        s["t"] = t.T.contiguous().reshape(-1)  # [L][B]
        s["y"] = parts[0].permute(2, 1, 0).contiguous().reshape(-1)  # [L][series][B]
        s["lens"] = lens.to(torch.int32)
        s["slope"], s["c1"], s["c2"], s["c3"] = (torch.zeros_like(s["y"]) for _ in range(4))
    elif kind == "tdinterp":
        B, K, L, N = case["batch"], case["modes"], case["rows"], case["samples"]
        t, lens, parts = _chirp(case, seed)
        grid = 4.0 * torch.arange(N, device="cuda", dtype=torch.float64)
        rows = torch.arange(L, device="cuda")[None, :]
        pad = torch.where(rows < lens[:, None], t, torch.full_like(t, 1e30))
        ends = torch.gather(t, 1, lens[:, None] - 1)[:, 0]
        s["lengths"] = torch.searchsorted(grid, ends.contiguous()).to(torch.int32)
        s["max_length"] = m = int(s["lengths"].max())
        s["inds"] = (torch.searchsorted(pad, grid[None, :m].expand(B, m).contiguous(), right=True) - 1).to(
            torch.int32).reshape(-1)
        # series s of binary b at row (b (2 K + 1) L + s L_b + j)
        src = (rows < lens[:, None])[:, None, :].expand(B, 2 * K + 1, L)
        dst = (torch.arange(B, device="cuda")[:, None, None] * (2 * K + 1) * L
               + torch.arange(2 * K + 1, device="cuda")[None, :, None] * lens[:, None, None] + rows[:, None, :])
        s["tables"] = []
        for p in parts:
            a = torch.zeros(B * (2 * K + 1) * L, dtype=torch.float64, device="cuda")
            a[dst[src]] = p[src]
            s["tables"].append(a)
        s["t"] = torch.where(rows < lens[:, None], t, torch.zeros_like(t)).reshape(-1)
        s["grid"], s["lens"] = grid, lens.to(torch.int32)
        s["ls"] = torch.tensor([l for l, _ in MODES5[:K]], dtype=torch.int32, device="cuda")
        s["ms"] = torch.tensor([m for _, m in MODES5[:K]], dtype=torch.int32, device="cuda")
        s["out"] = torch.zeros(B * N, dtype=torch.complex128, device="cuda")
    elif kind == "fd":
        from eobgpu_gb300 import _lib
        B, N, nch, rate = case["batch"], case["samples"], case["channels"], 2048.0
        g = _generator(seed, 13)
        n, df = N // 2 + 1, rate / N
        s["H"] = torch.view_as_real(_chirp_fft(B, N, rate, g)).contiguous()
        s["psd"] = _psd(n, df, nch, g)
        s["Fp"], s["Fx"], s["tau"] = (x.view(nch, B) for x in _network(B, nch, g))
        hp, hx = _split(torch.view_as_complex(s["H"][:1]))
        s["data"] = _noise_fd(s["psd"], df, g) + s["Fp"][:, :1] * hp + s["Fx"][:, :1] * hx
        s["df"], s["start"] = df, int(20.0 / df)
        s["scratch"] = torch.empty(int(_lib.load().eob_fd_lnl_scratch_bytes(B, N)), dtype=torch.uint8, device="cuda")
    elif kind == "allinone":
        B, n, nch = case["batch"], case["bins"], case["channels"]
        g = _generator(seed, 17)
        N = 2 * (n - 1)
        s["df"] = 2048.0 / N
        hp, hx = _split(_chirp_fft(B, N, 2048.0, g))
        psd = _psd(n, s["df"], nch, g)
        s["Fp"], s["Fx"], s["tau"] = _network(B, nch, g)
        data = (_noise_fd(psd, s["df"], g) + s["Fp"].view(nch, B)[:, :1] * hp[:1]
                + s["Fx"].view(nch, B)[:, :1] * hx[:1])
        s["hp"], s["hx"], s["data"], s["psd"] = (x.contiguous().reshape(-1) for x in (hp, hx, data, psd))
        s["out"] = torch.zeros(-(-n // 1024) * B * nch, dtype=torch.complex128, device="cuda")
    elif kind == "ode":
        from eobgpu_gb300.eob.seobnrv4phm import SEOBNRv4PHM
        n = case["batch"]
        g = _generator(seed, 19)
        q, chi1, chi2 = _uniform(g, n, 1.0, 6.0), _uniform(g, n, -0.8, 0.8), _uniform(g, n, -0.8, 0.8)
        r = torch.exp(_uniform(g, n, math.log(5.0), math.log(25.0)))
        gen = SEOBNRv4PHM()
        gen.setup_class(q / (1 + q), 1 / (1 + q), chi1, chi2, r ** -1.5)
        s["cls"], s["add"] = gen.eob_c_class, gen.additionalArgs.contiguous()
        circular = torch.sqrt(r) * (1.0 + 1.5 / r + 27.0 / (8.0 * r * r))
        s["state"] = torch.stack([r, _uniform(g, n, 0.0, 300.0), -_uniform(g, n, 1e-5, 2e-3),
                                  circular * _uniform(g, n, 0.99, 1.01)]).contiguous().reshape(-1)
        s["x"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["index"] = torch.arange(n, dtype=torch.int32, device="cuda")
        s["k"] = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
    else:
        raise ValueError(kind)
    return s


# ---------------------------------------------------------------- run


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "lnl":
        lnl, status = s["wl"].run(s["params"], s["data"], 1.0 / case["rate"], s["amp"])
        return dict(lnl=lnl, status=status)
    if kind == "tables":
        s["wl"].prepare(s["params"], 1.0 / case["rate"], order=s["order"], stages=4)
        return s["out"]
    if kind == "synth":
        lnl, status = s["wl"].synth_lnl(case["batch"], s["data"], 1.0 / case["rate"], s["amp"])
        return dict(lnl=lnl, status=status)
    if kind == "strain":
        h, status = s["wl"].synth_strain(case["batch"], 1.0 / case["rate"], case["samples"], per_mode=True)
        return dict(strain=h, status=status)
    if kind == "spline":
        from eobgpu_gb300.eob import pytdinterp
        pytdinterp.interpolate_TD_wrap(s["t"], s["y"], s["slope"], s["c1"], s["c2"], s["c3"], s["lens"],
                                       case["batch"], 2 * case["modes"] + 1)
        return dict(c1=s["c1"], c2=s["c2"], c3=s["c3"])
    if kind == "tdinterp":
        from eobgpu_gb300.eob import pytdinterp
        pytdinterp.TDInterp_wrap2(s["out"], s["grid"], s["t"], *s["tables"], case["rows"], s["lens"], case["samples"],
                                  case["batch"], case["modes"], s["ls"], s["ms"], s["inds"], s["lengths"],
                                  s["max_length"])
        return s["out"]
    if kind == "fd":
        from eobgpu_gb300 import fd
        return fd.fd_lnl_from_fft(s["H"], s["data"], s["psd"], s["Fp"], s["Fx"], s["tau"], s["df"], s["start"],
                                  s["scratch"])
    if kind == "allinone":
        from eobgpu_gb300.eob import pytdinterp
        pytdinterp.all_in_one_likelihood(s["out"], s["hp"], s["hx"], s["data"], s["psd"], s["Fp"], s["Fx"], s["tau"],
                                         s["df"], case["batch"], case["channels"], case["bins"])
        return s["out"]
    s["cls"].ODE_Ham_align_AD(s["x"], s["state"], s["k"], s["add"], case["batch"], s["index"])
    return s["k"]


# ---------------------------------------------------------------- work


def _mean_samples(case):
    """Samples of an average binary's template, from the Newtonian chirp time of the population."""
    from eobgpu_gb300 import workload
    p = workload.draw_params(workload.CONFIGS[case["pop"]], 512, stream=5)
    M = (p[:, 0] + p[:, 1]) * MTSUN
    eta = p[:, 0] * p[:, 1] / (p[:, 0] + p[:, 1]) ** 2
    t = 5.0 / 256.0 / eta * M * (math.pi * M * p[:, 4]) ** (-8.0 / 3.0)
    return float(np.minimum(t * case["rate"], case["samples"]).mean())


def work(case):
    kind, B = case["kind"], case["batch"]
    K = case.get("modes", 1)
    series = 2 * K + 1
    if kind in ("lnl", "tables", "synth", "strain"):
        n = B * _mean_samples(case)
        rows = B * MEAN_ROWS[case["pop"]]
        synth = n * (12.0 + 26.0 * K)  # phase, sine and cosine, two amplitude splines a mode, the residual
        table = rows * (150.0 + 250.0 * K + 25.0 * series)  # Hamiltonian, multipoles, splines
        if kind == "lnl":
            return {"bytes": 40.0 * B + 8.0 * case["samples"] + 12.0 * B,
                    "flops": B * MEAN_RHS[case["pop"]] * RHS_FLOPS + table + synth}
        if kind == "tables":
            return {"bytes": 8.0 * rows * (5 + 1 + 4 * series), "flops": table}
        if kind == "synth":
            return {"bytes": 8.0 * rows * (1 + 4 * series) + 8.0 * case["samples"] + 12.0 * B, "flops": synth}
        return {"bytes": 8.0 * rows * (1 + 4 * series) + 16.0 * B * K * case["samples"], "flops": synth}
    if kind == "spline":
        n = B * case["rows"] * 0.8
        return {"bytes": 8.0 * n * (1 + 4 * series), "flops": n * 25.0 * series}
    if kind == "tdinterp":
        n = 0.7 * B * case["samples"]
        return {"bytes": n * (16.0 + 4.0) + 8.0 * case["rows"] * B * (1 + 4 * series), "flops": n * (12.0 + 30.0 * K)}
    if kind == "fd":
        n = B * (case["samples"] // 2 + 1)
        return {"bytes": 16.0 * B * case["samples"] + 24.0 * case["channels"] * (case["samples"] // 2 + 1),
                "flops": n * (4.0 + 30.0 * case["channels"])}
    if kind == "allinone":
        return {"bytes": 32.0 * B * case["bins"] + 24.0 * case["channels"] * case["bins"],
                "flops": 30.0 * B * case["bins"] * case["channels"]}
    return {"bytes": 8.0 * B * (80 + 8), "flops": RHS_FLOPS * B}


# ---------------------------------------------------------------- exact


def _exact_series(s, case):
    """Per binary: its modes h_lm(t_k) [K, n] on the uniform grid (t clamped to the last knot), and its samples."""
    wl, K = s["wl"], case["modes"]
    tab, off = _tables(wl, case["batch"], K, wl.counters()["rows"])
    ms = torch.tensor([m for _, m in MODES5[:K]], dtype=torch.float64, device="cuda")
    npts, off = tab["samples"].cpu().tolist(), off.cpu().tolist()
    mass = (s["params"][:, 0] + s["params"][:, 1]).cpu().tolist()
    for b in range(case["batch"]):
        np_b, lo, hi = npts[b], off[b], off[b + 1]
        n = case["samples"] if case["kind"] == "strain" else min(np_b, case["samples"])
        if np_b <= 0:
            yield None, 0
            continue
        x = tab["t"][lo:hi]
        t = torch.arange(n, device="cuda", dtype=torch.float64) * (1.0 / case["rate"] / (mass[b] * MTSUN)) + x[0]
        t = torch.minimum(t, x[-1])
        i = (torch.searchsorted(x, t, right=True) - 1).clamp(0, hi - lo - 1)
        d = t - x[i]
        v = tab["c3"][:, lo:hi][:, i]
        for c in ("c2", "c1", "y"):
            v = v * d + tab[c][:, lo:hi][:, i]
        ph = ms[:, None] * v[0]
        yield torch.complex(v[1::2], v[2::2]) * torch.polar(torch.ones_like(ph), -ph), np_b


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lnl", "tables", "ode") or case.get("imr"):
        return None  # adaptive integration and the model's own series: no closed evaluation
    s = prepare(case, seed)
    if kind == "synth":
        base = (s["data"] ** 2).sum()
        out = []
        for h, np_b in _exact_series(s, case):
            if h is None:
                out.append(torch.tensor(math.nan, dtype=torch.float64, device="cuda"))
                continue
            hk = s["amp"] * h.real.sum(0)
            out.append(-0.5 * (base + (hk * hk - 2.0 * s["data"][:hk.numel()] * hk).sum()))
        return dict(lnl=torch.stack(out), status=None)
    if kind == "strain":
        out = torch.zeros(case["batch"], case["modes"], case["samples"], dtype=torch.complex128, device="cuda")
        for b, (h, np_b) in enumerate(_exact_series(s, case)):
            if h is not None:
                out[b] = h
        return dict(strain=out, status=None)
    if kind == "spline":
        return _exact_spline(s, case)
    if kind == "tdinterp":
        B, K, L, N = case["batch"], case["modes"], case["rows"], case["samples"]
        out = torch.zeros(B * N, dtype=torch.complex128, device="cuda")
        lens, lengths = s["lens"].cpu().tolist(), s["lengths"].cpu().tolist()
        ms = torch.tensor([m for _, m in MODES5[:K]], dtype=torch.float64, device="cuda")
        for b in range(B):
            n, m = lengths[b], s["max_length"]
            j = s["inds"][b * m:b * m + n].long()
            d = s["grid"][:n] - s["t"][b * L + j]
            at = b * (2 * K + 1) * L + torch.arange(2 * K + 1, device="cuda")[:, None] * lens[b] + j[None, :]
            v = s["tables"][3][at]
            for c in (2, 1, 0):
                v = v * d + s["tables"][c][at]
            ph = ms[:, None] * v[2 * K]
            out[b * N:b * N + n] = (torch.complex(v[:K], v[K:2 * K]) * torch.polar(torch.ones_like(ph), -ph)).sum(0)
        return out
    if kind == "fd":
        B, nch = case["batch"], case["channels"]
        n = case["samples"] // 2 + 1
        f = s["df"] * torch.arange(n, device="cuda", dtype=torch.float64)
        out = torch.zeros(B, dtype=torch.float64, device="cuda")
        for b in range(B):
            hp, hx = _split(torch.view_as_complex(s["H"][b]))
            hp[:s["start"]] = 0.0
            hx[:s["start"]] = 0.0
            ph = -2.0 * math.pi * f[None, :] * s["tau"][:, b:b + 1]
            d = s["data"] - (s["Fp"][:, b:b + 1] * hp + s["Fx"][:, b:b + 1] * hx) * torch.polar(torch.ones_like(ph), ph)
            out[b] = -2.0 * s["df"] * ((d.real ** 2 + d.imag ** 2) / s["psd"]).sum()
        return out
    B, n, nch = case["batch"], case["bins"], case["channels"]
    nblk = -(-n // 1024)
    out = torch.zeros(nblk, B, nch, dtype=torch.complex128, device="cuda")
    f = s["df"] * torch.arange(n, device="cuda", dtype=torch.float64)
    data, psd = s["data"].view(nch, n), s["psd"].view(nch, n)
    for b in range(B):
        hp, hx = s["hp"].view(B, n)[b], s["hx"].view(B, n)[b]
        for c in range(nch):
            i = c * B + b
            ph = -2.0 * math.pi * f * s["tau"][i]
            d = data[c] - (s["Fp"][i] * hp + s["Fx"][i] * hx) * torch.polar(torch.ones_like(ph), ph)
            e = torch.zeros(nblk * 1024, dtype=torch.float64, device="cuda")
            e[:n] = (d.real ** 2 + d.imag ** 2) / psd[c]
            out[:, b, c] = e.view(nblk, 1024).sum(1)
    return out.reshape(-1)


def _exact_spline(s, case):
    """Not-a-knot cubic splines by one elimination sweep over the rows, every
    series at once.  Each series' last row holds no interval: the slope
    system's own entries there (0, the eliminated diagonal, the outer span)."""
    B, S, L = case["batch"], 2 * case["modes"] + 1, case["rows"]
    t = s["t"].view(L, 1, B).expand(L, S, B)
    y = s["y"].view(L, S, B)
    n = s["lens"].long().view(1, B).expand(S, B)
    h = t[1:] - t[:-1]
    slope = (y[1:] - y[:-1]) / h
    diag, rhs = torch.zeros_like(y), torch.zeros_like(y)
    up, low = torch.zeros_like(y), torch.zeros_like(y)
    d = t[2] - t[0]
    diag[0], up[0] = h[1], d
    rhs[0] = ((h[0] + 2 * d) * h[1] * slope[0] + h[0] ** 2 * slope[1]) / d
    for i in range(1, L):
        last, inner = n == i + 1, n > i + 1
        d = t[i] - t[i - 2] if i >= 2 else torch.ones_like(t[0])
        low_l = d
        rhs_l = (h[i - 1] ** 2 * slope[i - 2] + (2 * d + h[i - 1]) * h[i - 2] * slope[i - 1]) / d if i >= 2 else d
        dia_l = h[i - 2] if i >= 2 else d
        if i < L - 1:
            low_i, up_i, dia_i = h[i], h[i - 1], 2 * (h[i - 1] + h[i])
            rhs_i = 3.0 * (h[i] * slope[i - 1] + h[i - 1] * slope[i])
        else:
            low_i, up_i, dia_i, rhs_i = low_l, torch.zeros_like(d), dia_l, rhs_l
        low[i] = torch.where(last, low_l, low_i)
        w = low[i] / diag[i - 1]
        up[i] = torch.where(inner, up_i, torch.zeros_like(d))
        diag[i] = torch.where(last, dia_l, dia_i) - w * up[i - 1]
        rhs[i] = torch.where(last, rhs_l, rhs_i) - w * rhs[i - 1]
        gone = i >= n
        diag[i] = torch.where(gone, torch.ones_like(d), diag[i])
        rhs[i] = torch.where(gone, torch.zeros_like(d), rhs[i])
    m = torch.zeros_like(y)
    m[L - 1] = rhs[L - 1] / diag[L - 1]
    for i in range(L - 2, -1, -1):
        m[i] = torch.where(i + 1 < n, (rhs[i] - up[i] * m[i + 1]) / diag[i], rhs[i] / diag[i])
    rows = torch.arange(L, device="cuda").view(L, 1, 1)
    c1, c2, c3 = torch.zeros_like(y), torch.zeros_like(y), torch.zeros_like(y)
    k = (m[:-1] + m[1:] - 2 * slope) / h
    c1[:-1], c2[:-1], c3[:-1] = m[:-1], (slope - m[:-1]) / h - k, k / h
    inside, last = rows < n - 1, rows == n - 1
    zero = torch.zeros_like(y)
    c1 = torch.where(inside, c1, zero)
    c2 = torch.where(inside, c2, torch.where(last, diag, zero))
    c3 = torch.where(inside, c3, torch.where(last, low, zero))
    return dict(c1=c1.reshape(-1), c2=c2.reshape(-1), c3=c3.reshape(-1))
