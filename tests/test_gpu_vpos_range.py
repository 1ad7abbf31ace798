"""The velocity gauge's dense radial transforms on a long grid: a state that is an eigenfunction of d/dr is a row of the
transform, so its product adds up to 38 at 4400 splines in units of its largest element.  The unit is rounded up to a power of
two and the row has a phase of its own, so 32 wavefunctions go through eight scales of a factor of two and four phases
of a quarter turn: the nearest comes to 34.  Against the banded solves (QPC_POS=0), each wavefunction by itself; two
steps, 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def test_sums_of_momentum_eigenstates(q, monkeypatch):
    sp = pytest.importorskip("scipy.sparse")
    sl = pytest.importorskip("scipy.sparse.linalg")
    n_r, p, n_l, n_m, m0, B = 4400, 6, 2, 3, -1, 32
    S, R, Ri, D, H = q.radial_setup(n_r, p, n_l + 1, q.linear_knots(n_r, p, 0.0, 0.5 * n_r))

    def full(b, sign):
        k = range(1, p + 1)
        return sp.diags([b[:, 0]] + [b[:n_r - i, i] for i in k] + [sign * b[:n_r - i, i] for i in k], [0] + list(k) + [-i for i in k], format="csc")

    _, u = sl.eigsh(1j * full(D, -1.0), k=1, M=full(S, 1.0).astype(complex), sigma=0.4, v0=np.ones(n_r, complex))
    k = np.arange(B)[:, None, None, None]
    c0 = u[:, 0] * (2.0 ** (k % 8 / 8.0) * np.exp(0.125j * np.pi * (k // 8))) * np.array([1.0, 0.7, 0.4, 0.9, 0.3, 0.8]).reshape(n_m, n_l, 1)
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        prop = q.propagator_cn_hc_vgwr().initialize(n_r, p, n_l, n_m, m0, S, Ri, D, H, 0.05, n_inst=B)
        assert prop.path()["position"] == (mode == "1")
        prop.put(c0)
        prop.run(np.full((B, 3, 2), 1e-3), np.full(B, 2), np.full(B, 2))
        out.append(prop.get())
        prop.close()
    for k in range(B):
        assert rel_l2(out[1][k], out[0][k]) < 1e-12, k
