"""Velocity-gauge steps with diagonal radial couplings (csrc/qpc_vpos.cu) against the banded solves (QPC_POS=0):
odd and even grids (the momentum basis has a null vector for odd N_r), parity blocks of unequal m-parity sets, one
m or one l, several wavefunctions with their own pulses and tails, and the recorded dipoles.  Same operators, other
rounding: 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(q, n_r, p, n_l, n_m, m0, B, dipole=False, steps=6, even=False):
    rng = np.random.default_rng(n_r + 31 * n_l + n_m)
    t = q.linear_knots(n_r, p, 0.0, 0.5 * n_r)
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    S, R, Ri, D, H = q.radial_setup(n_r, p, nlh, t)
    r = np.arange(1, n_r + 1)
    c0 = (rng.standard_normal((B, n_m, n_l, n_r)) + 1j * rng.standard_normal((B, n_m, n_l, n_r))) * np.exp(-0.03 * r)
    nf = np.full(B, steps) if even else rng.integers(0, steps + 1, B)
    nt = nf + (0 if even else rng.integers(0, 4, B))
    A = 1.5 * rng.standard_normal((B, steps + 1, 2))
    prop = q.propagator_cn_hc_vgwr().initialize(n_r, p, n_l, n_m, m0, S, Ri, D, H, 0.05, n_inst=B)
    prop.put(c0)
    xy = prop.run_dipole(A, nf, nt, R) if dipole else prop.run(A, nf, nt)
    c = prop.get()
    prop.close()
    return c, xy


def _both(q, monkeypatch, *a, **k):
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        out.append(_run(q, *a, **k))
    return out


@pytest.mark.parametrize("n_r,p,n_l,n_m,m0,B,even", [
    (64, 6, 4, 5, -2, 1, True), (65, 5, 3, 6, -3, 2, True), (97, 7, 5, 3, -1, 5, False), (130, 3, 2, 2, 1, 3, False),
    (33, 4, 1, 5, -2, 2, False), (96, 8, 6, 1, 0, 2, False), (75, 6, 9, 9, -4, 17, False), (40, 6, 21, 41, -20, 1, True)])
def test_runs_agree(q, monkeypatch, n_r, p, n_l, n_m, m0, B, even):
    (a, _), (b, _) = _both(q, monkeypatch, n_r, p, n_l, n_m, m0, B, even=even)
    for k in range(B):
        assert rel_l2(b[k], a[k]) < 1e-12, k


@pytest.mark.parametrize("n_r,B", [(70, 1), (81, 4)])
def test_dipoles_agree(q, monkeypatch, n_r, B):
    (a, za), (b, zb) = _both(q, monkeypatch, n_r, 6, 4, 5, -2, B, dipole=True)
    assert rel_l2(b, a) < 1e-12
    for x, y in zip(za, zb):
        assert np.abs(x - y).max() < 1e-12 * max(1.0, np.abs(x).max())
