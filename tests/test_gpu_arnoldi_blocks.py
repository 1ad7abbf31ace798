"""S^-1 by block substitution (k_ar_sinv_blk) against one lane per recurrence (QPC_AR_SINV=1), through whole Arnoldi
steps: grids that end inside a block of p rows, every degree, channel counts that leave lanes of a warp idle, and the
batch sizes on both sides of the one-element-per-thread kernels.  Well-conditioned steps (dt = 0.01): same sums in
another order, 1e-12."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,p,n_l,n_m,B,kmax", [(40, 2, 1, 1, 1, 4), (41, 3, 2, 1, 3, 6), (43, 4, 5, 1, 2, 12), (64, 5, 3, 2, 2, 9),
                                                  (65, 6, 4, 1, 5, 12), (90, 7, 6, 1, 1, 32), (81, 8, 3, 3, 2, 8), (300, 6, 21, 1, 60, 6)])
def test_sinv_kernels_agree(q, monkeypatch, n_r, p, n_l, n_m, B, kmax):
    m0 = -(n_m // 2)
    rng = np.random.default_rng(n_r + p)
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    S, R, _, _, H = q.radial_setup(n_r, p, nlh, q.linear_knots(n_r, p, 0.0, 0.5 * n_r))
    y10 = np.stack([q.y10_coupling(n_l, m0 + i) for i in range(n_m)])
    r = 0.5 * np.arange(1, n_r + 1)
    l = np.arange(n_l)[:, None]
    c0 = np.exp(-((r - 6.0) / 5.0) ** 2) * (r / (1 + r)) ** (l + 2) * 0.7 ** l * np.exp(1j * rng.uniform(0, 6, (B, n_m, n_l, 1)))
    ez = 0.05 * rng.standard_normal((B, 3))
    out = []
    for mode in ("1", "2"):
        monkeypatch.setenv("QPC_AR_SINV", mode)
        prop = q.propagator_hc_lgwz(kmax, 1e-14, 1e-8).initialize(n_r, p, n_l, S, R, H, y10, 0.01, n_m=n_m, m0=m0, n_inst=B)
        prop.put(c0)
        crit = prop.run(ez, np.minimum(3, np.arange(B) % 4 + 1))
        out.append((prop.get(), crit))
        prop.close()
    assert rel_l2(out[1][0], out[0][0]) < 1e-12
    assert np.array_equal(out[0][1] < 0, out[1][1] < 0)
