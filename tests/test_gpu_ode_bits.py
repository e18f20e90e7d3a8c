"""The drop-in right-hand side of a system has the same bits in a batch of any
size: on both sides of the switch between its two kernels, with every
calibration coefficient in use (a zero would hide a term), equal masses among
the systems, and either coefficient setting."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_hm", [0, 1])
def test_bits_do_not_depend_on_the_batch(use_hm):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pyEOB
    from eobgpu_gb300.eob.seobnrv4phm import SEOBNRv4PHM
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    limit, big = 48 * sms, 64 * sms
    rng = np.random.default_rng(12)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    q, c1, c2 = rng.uniform(1, 10, big), rng.uniform(-.9, .9, big), rng.uniform(-.9, .9, big)
    q[::20] = 1.0
    r = rng.uniform(3.0, 30.0, big)
    y = np.stack([r, rng.uniform(0, 100, big), -rng.uniform(1e-5, 5e-3, big), np.sqrt(r) * (1 + 1.6 / r)])
    m1, m2 = q / (1 + q), 1 / (1 + q)
    gen = SEOBNRv4PHM()
    gen.setup_class(d(m1), d(m2), d(c1), d(c2), torch.ones(big, device="cuda", dtype=torch.float64))
    add = gen.additionalArgs.cpu().numpy().reshape(-1, big).copy()
    add[5:10] = rng.uniform([[0.5], [-50.0], [-30.0], [-10.0], [-5.0]], [[2.0], [50.0], [30.0], [10.0], [5.0]], (5, big))
    eta, chiS, chiA = m1 * m2, (c1 + c2) / 2, (c1 - c2) / 2

    def run(n):
        cls = pyEOB.SEOBNRv5Class()
        cls.update_information(d(m1[:n]), d(m2[:n]), d(eta[:n]), d(((1 - 2 * eta) * chiS + (m1 - m2) * chiA)[:n]),
                               d(chiS[:n]), d(chiA[:n]), use_hm, n, None)
        k = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
        cls.ODE_Ham_align_AD(torch.zeros(1, device="cuda", dtype=torch.float64), d(y[:, :n].reshape(-1)), k,
                             d(add[:, :n].reshape(-1)), n, torch.arange(n, dtype=torch.int32, device="cuda"))
        return k.cpu().numpy().reshape(4, n)

    ref = run(big)
    assert np.isfinite(ref).mean() > 0.9
    for n in (1, 33, 700, 32 * sms + 1, limit, limit + 1):
        np.testing.assert_array_equal(run(n), ref[:, :n])
