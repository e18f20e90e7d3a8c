"""The block-wide spline build (drop-in interpolate_TD) against the oracle's
serial sweep, at lengths around its chunk and tile edges: the shortest, one row
per chunk, odd and even chunks, one tile full, one row into the next, several
tiles; and binaries of different lengths sharing a block.

Each coefficient's contribution over its interval is held to 1e-12 of the
series' scale: both sides round at eps of the slopes, which the solve (diagonal
dominance: inverse below 1 / (b/2)) passes on with a factor of order one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 64 * 13


@pytest.mark.parametrize("lengths", [[4, 5, 6, 7], [63, 64, 65], [129, 192, 2, 700, 701], [TILE - 1, TILE, TILE + 1],
                                     [2 * TILE + 5, 17, TILE + 40, 300, 3 * TILE]])
@pytest.mark.parametrize("nsubs", [1, 3])
def test_interpolate_td_edges(oracle, lengths, nsubs):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pytdinterp
    rng = np.random.default_rng(len(lengths) * 10 + nsubs)
    B, L = len(lengths), max(lengths)
    # steps that grow and shrink by up to 6 and 1/3, as the step controller's
    t = np.cumsum(np.exp(np.clip(np.cumsum(rng.uniform(-1.0, 1.0, (L, B)), axis=0), -3.0, 3.0)), axis=0)
    y = rng.normal(size=(L, nsubs, B)) * 0.1 + np.sin(0.1 * t)[:, None, :]
    d = lambda a: torch.tensor(np.ascontiguousarray(a).reshape(-1), device="cuda")
    Bv, ud, dg, ld = (torch.zeros(L * nsubs * B, dtype=torch.float64, device="cuda") for _ in range(4))
    pytdinterp.interpolate_TD_wrap(d(t), d(y), Bv, ud, dg, ld,
                                   torch.tensor(lengths, dtype=torch.int32, device="cuda"), B, nsubs)
    got = [a.cpu().numpy().reshape(L, nsubs, B) for a in (ud, dg, ld)]
    slopes = Bv.cpu().numpy().reshape(L, nsubs, B)
    for b, n in enumerate(lengths):
        for g in got:
            assert np.all(g[n:, :, b] == 0)  # rows past the binary's own are not touched
        if n < 3:
            assert all(np.all(g[:, :, b] == 0) for g in got)
            continue
        x = t[:n, b].copy()
        dx = np.diff(x)
        for s in range(nsubs):
            ref = oracle.interpolate_td(x, y[:n, s, b].copy(), [n], 1, 1)
            scale = np.max(np.abs(y[:n, s, b]))
            for p, (g, r) in enumerate(zip(got, ref), 1):
                assert np.max(np.abs(g[:n - 1, s, b] - r[:n - 1]) * dx ** p) <= 1e-12 * scale, (b, s, p)
            # the slope system's last row, as the reference's sweep leaves it
            assert got[0][n - 1, s, b] == 0
            assert abs(got[2][n - 1, s, b] / (x[-1] - x[-3]) - 1) < 1e-15
            np.testing.assert_array_equal(slopes[:n - 1, s, b], got[0][:n - 1, s, b])
