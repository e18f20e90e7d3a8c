"""The drop-in right-hand side at sizes on both sides of its switch between
clusters and one thread per system, and around a cluster's 32 systems, against the
oracle on a sample of the systems: 1e-11 of each system's largest component, as the
reference-shaped entry points on states with r >= 4; and the same system gives
the same values (1e-13) whatever the batch around it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 700, 4864, 4865, 9001])
def test_ode_sizes(oracle, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob.seobnrv4phm import SEOBNRv4PHM
    rng = np.random.default_rng(4)  # the same systems at every n
    big = 9001
    q, c1, c2 = rng.uniform(1, 6, big), rng.uniform(-.8, .8, big), rng.uniform(-.8, .8, big)
    r = rng.uniform(4.5, 25, big)
    y = np.stack([r, rng.uniform(0, 100, big), -rng.uniform(1e-5, 5e-3, big), np.sqrt(r) * (1 + 1.6 / r)])

    def run(sel):
        gen = SEOBNRv4PHM()
        d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
        qs = q[sel]
        gen.setup_class(d(qs / (1 + qs)), d(1 / (1 + qs)), d(c1[sel]), d(c2[sel]), torch.ones(len(qs), device="cuda",
                                                                                             dtype=torch.float64))
        k = torch.zeros(4 * len(qs), dtype=torch.float64, device="cuda")
        add = gen.additionalArgs.contiguous()
        gen.eob_c_class.ODE_Ham_align_AD(torch.zeros(1, device="cuda", dtype=torch.float64), d(y[:, sel].reshape(-1)), k,
                                         add, len(qs), torch.arange(len(qs), dtype=torch.int32, device="cuda"))
        return k.cpu().numpy().reshape(4, -1), add.cpu().numpy()

    sel = np.arange(n)
    k, add = run(sel)
    few = np.unique(np.linspace(0, n - 1, 12).astype(int))
    again, _ = run(few)
    scale = np.abs(k[:, few]).max(axis=0)
    assert np.max(np.abs(again - k[:, few]) / scale) < 1e-13
    for j in few:
        ctx = oracle.context(np.array([q[j] / (1 + q[j])]), np.array([1 / (1 + q[j])]), np.array([c1[j]]),
                             np.array([c2[j]]))
        ref = ctx.ode(y[:, j:j + 1], add[:, j:j + 1])[:, 0]
        assert np.max(np.abs(k[:, j] - ref)) < 1e-11 * np.abs(ref).max()
