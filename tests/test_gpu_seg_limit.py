"""Runs of the segmented chain solver (few wavefunctions, banded solves) at sizes whose dynamic shared memory stays below 48 KB
while the kernel's static arrays take it beyond, against the CPU oracle: 1e-12, the bar of the single-step parity
tests."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,p,n_l,n_m,m0,B", [(551, 3, 64, 2, -1, 2), (151, 7, 3, 2, 3, 8)])
def test_sizes_beside_the_default_limit(q, oracle, monkeypatch, n_r, p, n_l, n_m, m0, B):
    monkeypatch.setenv("QPC_POS", "0")
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    S, R, _, _, H = q.radial_setup(n_r, p, nlh, q.linear_knots(n_r, p, 0.0, 0.5 * n_r))
    rng = np.random.default_rng(n_r)
    c0 = (rng.standard_normal((B, n_m, n_l, n_r)) + 1j * rng.standard_normal((B, n_m, n_l, n_r))) * np.exp(-0.02 * np.arange(n_r))
    f = 0.05 * rng.standard_normal((B, 3))
    prop = q.propagator_cn_hc_lgwz().initialize(n_r, p, n_l, S, R, H, 0.05, n_m=n_m, m0=m0, n_inst=B)
    prop.put(c0)
    prop.run(f, np.full(B, 2), np.full(B, 3))
    got = prop.get()
    prop.close()
    g = oracle.grid(S, R, H, 0.05, n_l, n_m=n_m, m0=m0, n_inst=B)
    want = oracle.run(g, c0.reshape(B, -1), f, np.full(B, 2), np.full(B, 3))
    assert rel_l2(got.reshape(B, -1), np.asarray(want).reshape(B, -1)) < 1e-12
