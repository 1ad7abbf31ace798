"""The digit products on the tensor cores (csrc/qpc_tcband.cu) against the multiply-adds (QPC_POS_TC=0) where the kernel
changes shape: the edges of its 128 rows, 16, 24 or 32 columns and 32-deep stages, grids below a stage, every spline degree, several
m, uneven runs, the mask, zero states.  A product drops less than 2^-49 of a column's largest element per output, so
sqrt(N) 2^-49 of the norm: 14 products of up to 400 rows stay below 5e-13."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_pos import _grid, _run

pytestmark = pytest.mark.gpu


def _both(monkeypatch, run):
    monkeypatch.setenv("QPC_POS", "1")
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS_TC", mode)
        out.append(run())
    return out


@pytest.mark.parametrize("n_r,p,n_l,B", [
    (31, 6, 2, 1), (33, 5, 3, 2), (97, 3, 9, 3), (127, 4, 8, 31), (128, 7, 16, 32), (129, 8, 5, 33), (160, 6, 3, 63), (161, 6, 4, 64),
    (255, 5, 6, 65), (257, 7, 4, 12), (385, 6, 3, 17), (400, 6, 5, 97),
    (257, 6, 20, 48), (270, 6, 20, 41), (257, 6, 30, 96), (300, 5, 30, 85)])	# blocks of 24 and of 32 columns, full and ragged; 16 above
def test_runs_agree(q, monkeypatch, n_r, p, n_l, B):
    a, b = _both(monkeypatch, lambda: _run(q, n_r, p, n_l, B)[0])
    for k in range(B):
        assert rel_l2(b[k], a[k]) < 5e-13, k


@pytest.mark.parametrize("kind", ["run", "dipole", "mask"])
def test_several_m(q, monkeypatch, kind):
    (a, za), (b, zb) = _both(monkeypatch, lambda: _run(q, 150, 6, 7, 20, 3, -1, kind=kind))
    assert rel_l2(b, a) < 5e-13
    if kind == "dipole":
        assert np.abs(zb - za).max() < 5e-13 * np.abs(za).max()


def test_zero_and_not_finite(q, monkeypatch):
    """a zero wavefunction stays zero beside the others; a value that is not finite is reported"""
    monkeypatch.setenv("QPC_POS", "1")
    monkeypatch.setenv("QPC_POS_TC", "1")
    t, S, R, H = _grid(q, 140, 6, 3)
    rng = np.random.default_rng(3)
    c0 = rng.standard_normal((14, 1, 3, 140)) * np.exp(-0.05 * np.arange(140)) + 0j
    c0[5] = 0.0
    prop = q.propagator_cn_hc_lgwz().initialize(140, 6, 3, S, R, H, 0.05, n_inst=14)
    prop.put(c0)
    prop.run(0.05 * np.ones((14, 5)), np.full(14, 4), np.full(14, 4))
    c = prop.get()
    assert np.all(c[5] == 0.0) and np.all(np.isfinite(c)) and np.all(np.abs(c[4]).max(-1) > 0)
    c0[7, 0, 1, 60] = np.inf
    with pytest.raises(Exception):
        prop.put(c0)
        prop.run(0.05 * np.ones((14, 5)), np.full(14, 4), np.full(14, 4))
    prop.close()


@pytest.mark.parametrize("n_r,p,n_l,n_m,m0,B", [(64, 6, 4, 5, -2, 1), (129, 5, 3, 6, -3, 2), (160, 7, 5, 3, -1, 5), (97, 4, 2, 3, 1, 1)])
def test_dense_transforms_agree(q, monkeypatch, n_r, p, n_l, n_m, m0, B):
    """the velocity gauge's dense radial transforms: about 9 of them in each of 6 steps, so 1.2e-12"""
    from test_gpu_vpos import _run as vrun
    (a, _), (b, _) = _both(monkeypatch, lambda: vrun(q, n_r, p, n_l, n_m, m0, B))
    for k in range(B):
        assert rel_l2(b[k], a[k]) < 1.2e-12, k
