"""S^-1 of small batches on vectors longer than the block substitution's shared memory (k_ar_sinv_sys, P lanes per recurrence)
against one lane per recurrence (QPC_AR_SINV=1), through whole Arnoldi steps just past the length for two degrees: the
same sums in another order, 1e-12 as in test_gpu_arnoldi_blocks, and not the same kernel."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,p,n_l,B", [(5125, 6, 2, 1), (2565, 3, 3, 3)])
def test_long_vectors(q, monkeypatch, n_r, p, n_l, B):
    rng = np.random.default_rng(n_r)
    S, R, _, _, H = q.radial_setup(n_r, p, n_l, q.linear_knots(n_r, p, 0.0, 0.5 * n_r))
    r = 0.5 * np.arange(1, n_r + 1)
    l = np.arange(n_l)[:, None]
    c0 = np.exp(-((r - 6.0) / 5.0) ** 2) * (r / (1 + r)) ** (l + 2) * 0.7 ** l * np.exp(1j * rng.uniform(0, 6, (B, 1, n_l, 1)))
    ez = 0.05 * rng.standard_normal((B, 2))
    out = []
    for mode in ("1", "2"):
        monkeypatch.setenv("QPC_AR_SINV", mode)
        prop = q.propagator_hc_lgwz(5, 1e-14, 1e-8).initialize(n_r, p, n_l, S, R, H, q.y10_coupling(n_l), 0.01, n_inst=B)
        prop.put(c0)
        prop.run(ez)
        out.append(prop.get())
        prop.close()
    assert rel_l2(out[1], out[0]) < 1e-12
    assert not np.array_equal(out[1], out[0])
