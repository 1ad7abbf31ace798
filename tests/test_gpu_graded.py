"""Runs in the position basis on graded grids: breakpoints a i^k near the nucleus, then uniform ones, with spacings 81, 14 000 and
1.9 million apart.  The rows of the operators that lead into the basis and back differ by the root of that.  Against the
banded solves (QPC_POS=0), 20 steps; 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _knots(n_r, p, r1, rmax, power):
    """a i^power out to about r1, then equal steps of the last spacing to about rmax"""
    nb = n_r - p + 3
    i = np.arange(nb)

    def grid(n):
        b = np.where(i <= n, r1 * (i / n) ** power, 0.0)
        h = b[n] - b[n - 1]
        return np.where(i <= n, b, r1 + h * (i - n))

    b = min((grid(n) for n in range(4, nb - 1)), key=lambda b: abs(b[-1] - rmax))
    return np.concatenate([np.zeros(p), b, np.full(p, b[-1])])


GRIDS = [(400, 6, 10.0, 180.0, 2), (400, 6, 10.0, 150.0, 3), (300, 6, 5.0, 60.0, 4), (300, 4, 5.0, 60.0, 4)]


@pytest.mark.parametrize("B", [1, 4, 8])
@pytest.mark.parametrize("n_r,p,r1,rmax,power", GRIDS)
def test_length_gauge(q, monkeypatch, n_r, p, r1, rmax, power, B):
    n_l, steps = 6, 20
    S, R, _, _, H = q.radial_setup(n_r, p, n_l, _knots(n_r, p, r1, rmax, power))
    rng = np.random.default_rng(power)
    i = np.arange(n_r)
    c0 = 0.0	# packets, most of their size on the fine end of the grid
    for weight, x0 in ((1.0, 0.02), (0.2, 0.15), (0.05, 0.5)):
        at, w, k, a = (rng.uniform(lo, hi, (B, 1, n_l, 1)) for lo, hi in ((0, x0 * n_r), (2, 12), (-0.6, 0.6), (0, 6.28)))
        c0 = c0 + weight * np.exp(-((i - at) / w) ** 2 + 1j * (k * i + a)) * 0.8 ** np.arange(n_l)[:, None]
    c0 *= (i / (1.0 + i)) ** (np.arange(n_l)[:, None] + 1)
    f = 0.05 * rng.standard_normal((B, steps + 1))
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        monkeypatch.setenv("QPC_POS_TC", "1" if B == 8 else "0")
        prop = q.propagator_cn_hc_lgwz().initialize(n_r, p, n_l, S, R, H, 0.05, n_inst=B)
        prop.put(c0)
        z = prop.run_dipole(f, np.full(B, steps), np.full(B, steps + 2), R)
        out.append((prop.get(), z))
        path = prop.path()
        assert path["last_run"] == ("position" if mode == "1" else "banded") and path["digits"][1:] == ((B == 8 and mode == "1"),) * 2
        prop.close()
    assert rel_l2(out[1][0], out[0][0]) < 1e-12
    assert np.abs(out[1][1] - out[0][1]).max() < 1e-12 * np.abs(out[0][1]).max()


# (not the finest: d/dr turns its shortest waves by 10^4 and more, known to 10^-12 in FP64 on either path)
@pytest.mark.parametrize("n_r,p,r1,rmax,power", GRIDS[:2])
def test_velocity_gauge(q, monkeypatch, n_r, p, r1, rmax, power):
    n_l, n_m, m0, steps, B = 3, 3, -1, 10, 2
    S, _, Ri, D, H = q.radial_setup(n_r, p, n_l + 1, _knots(n_r, p, r1, rmax, power))
    rng = np.random.default_rng(power)
    r = np.arange(n_r)
    l = np.arange(n_l)[:, None] + np.abs(np.arange(n_m) + m0)[:, None, None]
    # channels that vanish at the origin, as the velocity gauge's 1 / r couplings presume
    c0 = (rng.standard_normal((B, n_m, n_l, n_r)) + 1j * rng.standard_normal((B, n_m, n_l, n_r))) * np.exp(-0.02 * r) * (r / (20.0 + r)) ** (l + 1)
    A = 0.5 * rng.standard_normal((B, steps + 1, 2))
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        prop = q.propagator_cn_hc_vgwr().initialize(n_r, p, n_l, n_m, m0, S, Ri, D, H, 0.05, n_inst=B)
        path = prop.path()["position"]
        prop.put(c0)
        prop.run(A, np.full(B, steps), np.full(B, steps + 2))
        out.append((prop.get(), path))
        prop.close()
    assert not out[0][1] and out[1][1]
    assert rel_l2(out[1][0], out[0][0]) < 1e-12
