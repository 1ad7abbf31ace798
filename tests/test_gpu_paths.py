"""The comparisons of test_gpu_pos, test_gpu_tcband, test_gpu_vpos and test_gpu_pcs_tc run one kernel against another.  Here the
handles of the same cases say that they hold the kernels under test, so that those comparisons are not of one
path with itself; own potentials are compared on a grid wider than the band, where their bands are checked against the
first one's."""
import numpy as np
import pytest

import test_gpu_pcs_tc as tpcs
import test_gpu_pos as tpos
import test_gpu_tcband as ttc
import test_gpu_vpos as tvg
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _cases(f):
    return [m for m in f.pytestmark if m.name == "parametrize"][0].args[1]


def _lgwz(q, n_r, p, n_l, B, n_m=1, m0=0):
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    _, S, R, H = tpos._grid(q, n_r, p, nlh)
    return q.propagator_cn_hc_lgwz().initialize(n_r, p, n_l, S, R, H, 0.05, n_m=n_m, m0=m0, n_inst=B)


def _vgwr(q, n_r, p, n_l, n_m, m0, B):
    nlh = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    S, R, Ri, D, H = q.radial_setup(n_r, p, nlh, q.linear_knots(n_r, p, 0.0, 0.5 * n_r))
    return q.propagator_cn_hc_vgwr().initialize(n_r, p, n_l, n_m, m0, S, Ri, D, H, 0.05, n_inst=B)


def _path(h):
    out = h.path()
    h.close()
    return out


@pytest.mark.parametrize("n_r,p,n_l,B", _cases(tpos.test_runs_agree))
def test_position_basis(q, monkeypatch, n_r, p, n_l, B):
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        assert _path(_lgwz(q, n_r, p, n_l, B))["position"] == (mode == "1")


@pytest.mark.parametrize("n_r,p,n_l,B", _cases(ttc.test_runs_agree))
def test_digit_planes(q, monkeypatch, n_r, p, n_l, B):
    monkeypatch.setenv("QPC_POS", "1")
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS_TC", mode)
        assert _path(_lgwz(q, n_r, p, n_l, B))["digits"] == (mode == "1",) * 3


@pytest.mark.parametrize("n_r,p,n_l,n_m,m0,B", [c[:6] for c in _cases(tvg.test_runs_agree)] + [(70, 6, 4, 5, -2, 1), (81, 6, 4, 5, -2, 4)])
def test_diagonal_couplings(q, monkeypatch, n_r, p, n_l, n_m, m0, B):
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        assert _path(_vgwr(q, n_r, p, n_l, n_m, m0, B))["position"] == (mode == "1")


@pytest.mark.parametrize("n_r,p,n_l,n_m,m0,B", _cases(ttc.test_dense_transforms_agree))
def test_dense_digit_planes(q, monkeypatch, n_r, p, n_l, n_m, m0, B):
    monkeypatch.setenv("QPC_POS", "1")
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS_TC", mode)
        assert _path(_vgwr(q, n_r, p, n_l, n_m, m0, B)) == {"position": True, "digits": (mode == "1",) * 2}


@pytest.mark.parametrize("n_r,nkr,n_inst,n_l,n_m,m0", _cases(tpcs.test_projections))
def test_projection_segments(q, n_r, nkr, n_inst, n_l, n_m, m0):
    nl = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    for bad in (False, True):
        t = tpcs._tables(np.random.default_rng(1), nkr, nl, n_r, n_m * n_l)
        t["plm"] = t["plm"].reshape(1, n_m, n_l)
        t["exm"] = np.ones((1, n_m), complex)
        if bad:
            t["ijl"][0, -1, -1] = np.inf
        pcs = q.spectrum_c_pcs(nkr, 1, 1).initialize(n_r, 6, n_l, q.linear_knots(n_r, 6, 0.0, 0.5 * n_r), 0.05, 2.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0, n_m,
                                                     m0, tables=t)
        assert _path(pcs)["segments"] == (0 if bad else -(-n_r // 896))


@pytest.mark.parametrize("n_r,B", [(130, 5), (350, 1), (350, 5), (401, 2)])
def test_own_potentials(q, monkeypatch, n_r, B):
    seen = []
    init = q.propagator_cn_hc_lgwz.close

    def close(self):
        if self._h is not None:
            seen.append(self.path())
        init(self)

    monkeypatch.setattr(q.propagator_cn_hc_lgwz, "close", close)
    (a, _), (b, _) = tpos._both(q, monkeypatch, lambda: tpos._run(q, n_r, 6, 9, B, own=True, steps=12))
    assert [s["last_run"] for s in seen if s["last_run"]] == ["banded", "position"]
    assert rel_l2(b, a) < 1e-12


def test_product_kernels(q, monkeypatch):
    """one column, few, many: the kernels the header of csrc/qpc_radial.cu describes"""
    monkeypatch.setenv("QPC_POS", "1")
    for B, want in ((1, "k_band_one"), (3, "k_band_apply"), (64, "k_tc_apply")):
        prop = _lgwz(q, 400, 6, 21, B)
        assert prop.path() == {"position": True, "last_run": None, "digits": (B == 64,) * 3, "product": None}
        prop.put(np.ones((B, 1, 21, 400), complex))
        prop.run(np.zeros((B, 3)), np.full(B, 2), np.full(B, 2))
        assert prop.path() == {"position": True, "last_run": "position", "digits": (B == 64,) * 3, "product": want}
        prop.close()
