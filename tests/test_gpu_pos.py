"""Runs in the position basis (csrc/qpc_pos.cu) against the banded solves (QPC_POS=0) at the sizes where its
kernels change shape: the edges of the 32-row tiles, every split of columns over warps, grids narrower than the
band, even and odd n_l, every spline degree, several m, own potentials, uneven pulses, the mask and the dipole.
Both evaluate the same operators in FP64 with their own rounding; 1e-12 is the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _grid(q, n_r, p, n_l, pot=None):
    t = q.linear_knots(n_r, p, 0.0, 0.5 * n_r)
    S, R, _, _, H = q.radial_setup(n_r, p, n_l, t, *(() if pot is None else (pot,)))
    return t, S, R, H


def _both(q, monkeypatch, run):
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        out.append(run())
    return out


def _run(q, n_r, p, n_l, B, n_m=1, m0=0, own=False, kind="run", steps=9, seed=0):
    rng = np.random.default_rng(seed + 7 * n_r + n_l + B)
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    t, S, R, H = _grid(q, n_r, p, nlh)
    if own:
        H = np.stack([_grid(q, n_r, p, nlh, (q.POTENTIAL_YUKAWA, 1.0, rng.uniform(0, 9), rng.uniform(1, 3)))[3] for _ in range(B)])
    r = np.arange(1, n_r + 1)
    c0 = (rng.standard_normal((B, n_m, n_l, n_r)) + 1j * rng.standard_normal((B, n_m, n_l, n_r))) * np.exp(-0.02 * r) * 0.7 ** np.arange(n_l)[:, None]
    nf = rng.integers(0, steps + 1, B)
    nt = nf + rng.integers(0, 4, B)
    f = 0.08 * rng.standard_normal((B, steps + 1))
    prop = q.propagator_cn_hc_lgwz().initialize(n_r, p, n_l, S, R, H, 0.05, n_m=n_m, m0=m0, n_inst=B)
    prop.put(c0)
    z = None
    if kind == "dipole":
        z = prop.run_dipole(f, nf, nt, R)
    elif kind == "mask":
        prop.run_ex(f, nf, nt, mask=q.mask_band(n_r, p, t, 0.3 * n_r, 0.5 * n_r))
    else:
        prop.run(f, nf, nt)
    c = prop.get()
    prop.close()
    return c, z


@pytest.mark.parametrize("n_r,p,n_l,B", [
    (32, 6, 2, 1), (33, 5, 3, 2), (63, 3, 9, 3), (64, 4, 8, 5), (65, 7, 16, 9), (96, 8, 17, 17), (97, 6, 33, 33), (289, 6, 5, 1),
    (300, 5, 6, 65), (321, 7, 4, 97), (256, 6, 41, 2), (160, 4, 64, 4), (40, 6, 128, 2), (161, 6, 7, 90), (64, 4, 41, 229), (33, 5, 2, 228)])
def test_runs_agree(q, monkeypatch, n_r, p, n_l, B):
    a, b = _both(q, monkeypatch, lambda: _run(q, n_r, p, n_l, B)[0])
    for k in range(B):
        assert rel_l2(b[k], a[k]) < 1e-12, k


@pytest.mark.parametrize("n_m,m0", [(3, -1), (2, 1)])
@pytest.mark.parametrize("kind", ["run", "dipole", "mask"])
def test_several_m(q, monkeypatch, n_m, m0, kind):
    (a, za), (b, zb) = _both(q, monkeypatch, lambda: _run(q, 75, 6, 7, 4, n_m, m0, kind=kind))
    assert rel_l2(b, a) < 1e-12
    if kind == "dipole":
        assert np.abs(zb - za).max() < 1e-12 * np.abs(za).max()


@pytest.mark.parametrize("kind,B", [("run", 1), ("run", 5), ("dipole", 3), ("mask", 3)])
def test_own_potentials(q, monkeypatch, kind, B):
    (a, za), (b, zb) = _both(q, monkeypatch, lambda: _run(q, 130, 6, 9, B, own=True, kind=kind, steps=40))
    assert rel_l2(b, a) < 1e-12
    if kind == "dipole":
        assert np.abs(zb - za).max() < 1e-12 * np.abs(za).max()


def test_not_finite(q):
    """a value that is not finite is reported, whatever it is"""
    t, S, R, H = _grid(q, 80, 6, 5)
    for bad in (np.nan, np.inf):
        c0 = np.ones((2, 1, 5, 80), complex)
        c0[1, 0, 3, 41] = bad
        prop = q.propagator_cn_hc_lgwz().initialize(80, 6, 5, S, R, H, 0.05, n_inst=2)
        prop.put(c0)
        with pytest.raises(q.QpcError) as e:
            prop.run(np.full((2, 4), 0.01), [3, 3])
        assert e.value.code == 5


def test_zero_and_tiny_states(q, monkeypatch):
    """a zero wavefunction stays zero; scaling by a power of two scales the result exactly"""
    t, S, R, H = _grid(q, 80, 6, 5)
    rng = np.random.default_rng(5)
    c = rng.standard_normal((1, 5, 80)) + 1j * rng.standard_normal((1, 5, 80))
    prop = q.propagator_cn_hc_lgwz().initialize(80, 6, 5, S, R, H, 0.05, n_inst=4)
    prop.put(np.stack([c, 0 * c, c * 2.0 ** -300, c * 2.0 ** 300]))
    prop.run(np.full((4, 6), 0.02), [5] * 4)
    o = prop.get()
    assert np.all(o[1] == 0)
    assert np.array_equal(o[2] * 2.0 ** 300, o[0]) and np.array_equal(o[3] * 2.0 ** -300, o[0])
