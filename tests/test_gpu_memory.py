"""Handles on a card without room for the operators of the position basis and for digit planes (QPC_ALLOC_MAX: larger
allocations fail): they are made all the same and run on what needs less.  Against handles made with room for
everything on the other path; 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_pos import _grid

pytestmark = pytest.mark.gpu


def _lgwz(q, n_r, n_l, B):
    _, S, R, H = _grid(q, n_r, 6, n_l)
    rng = np.random.default_rng(n_r)
    prop = q.propagator_cn_hc_lgwz().initialize(n_r, 6, n_l, S, R, H, 0.05, n_inst=B)
    prop.put((rng.standard_normal((B, 1, n_l, n_r)) + 1j * rng.standard_normal((B, 1, n_l, n_r))) * np.exp(-0.02 * np.arange(n_r)))
    prop.run(0.05 * rng.standard_normal((B, 5)), np.full(B, 4), np.full(B, 5))
    out = prop.get(), prop.path()
    prop.close()
    return out


# 1.3 MB: one matrix of 400 x 400; 23 and 20 MB: the set-up's columns and bands
@pytest.mark.parametrize("limit", [1000000, 2000000, 21000000])
def test_length_gauge(q, monkeypatch, limit):
    monkeypatch.setenv("QPC_FAC_BYTES", "1")
    a, pa = _lgwz(q, 400, 9, 1)
    monkeypatch.setenv("QPC_ALLOC_MAX", str(limit))
    b, pb = _lgwz(q, 400, 9, 1)
    assert (pa["position"], pa["last_run"]) == (True, "position") and (pb["position"], pb["last_run"]) == (False, "banded")
    assert rel_l2(b, a) < 1e-12


def test_digit_planes(q, monkeypatch):
    """room for the bands (20 MB) and not for the planes of F~ (29 MB)"""
    monkeypatch.setenv("QPC_FAC_BYTES", "1")
    a, pa = _lgwz(q, 400, 9, 8)
    monkeypatch.setenv("QPC_ALLOC_MAX", "24000000")
    b, pb = _lgwz(q, 400, 9, 8)
    assert pa["digits"] == (True,) * 3 and pb["digits"] == (False, True, True) and pb["last_run"] == "position"
    assert rel_l2(b, a) < 1e-12


def test_velocity_gauge(q, monkeypatch):
    n_r, n_l, n_m, m0 = 600, 3, 3, -1
    S, R, Ri, D, H = q.radial_setup(n_r, 6, n_l + 1, q.linear_knots(n_r, 6, 0.0, 0.5 * n_r))
    rng = np.random.default_rng(2)
    c0 = (rng.standard_normal((1, n_m, n_l, n_r)) + 1j * rng.standard_normal((1, n_m, n_l, n_r))) * np.exp(-0.02 * np.arange(n_r))
    out = []
    for limit in (None, "7000000"):	# the digit slices both paths hold: 6.6 MB; the set-up's columns: 23 MB
        if limit:
            monkeypatch.setenv("QPC_ALLOC_MAX", limit)
        prop = q.propagator_cn_hc_vgwr().initialize(n_r, 6, n_l, n_m, m0, S, Ri, D, H, 0.05)
        assert prop.path()["position"] == (limit is None)
        prop.put(c0)
        prop.run(np.full((1, 4, 2), 0.3), [3], [4])
        out.append(prop.get())
        prop.close()
    assert rel_l2(out[1], out[0]) < 1e-12


def test_projections(q, monkeypatch):
    from test_gpu_pcs_tc import _tables
    n_r, nkr, n_l = 800, 40, 4
    t = _tables(np.random.default_rng(3), nkr, n_l, n_r, n_l)
    t["plm"] = t["plm"].reshape(1, 1, n_l)
    rng = np.random.default_rng(5)
    c = rng.standard_normal((3, 1, n_l, n_r)) + 1j * rng.standard_normal((3, 1, n_l, n_r))
    monkeypatch.setenv("QPC_ALLOC_MAX", "2000000")	# the table: 1 MB, its planes: 13 MB
    pcs = q.spectrum_c_pcs(nkr, 1, 1).initialize(n_r, 6, n_l, q.linear_knots(n_r, 6, 0.0, 400.0), 0.05, 2.0, 0.0, 0.0, 0.0, 0.0, 1.0, tables=t)
    assert pcs.path()["segments"] == 0
    got = pcs.measure_lmd(c)[:, :, 0]
    pcs.close()
    scale = 0.797884560802865 * t["cps"]
    want = np.einsum("klr,ilr->ikl", t["ijl"].astype(np.longdouble), c[:, 0].astype(np.clongdouble)) * scale
    # a sum of n terms in FP64, whatever its order: n roundings of the magnitudes' sum; the factors' few on top
    bound = (n_r + 8) * 2.0 ** -53 * np.einsum("klr,ilr->ikl", np.abs(t["ijl"]), np.abs(c[:, 0].real) + np.abs(c[:, 0].imag)) * np.abs(scale)
    assert np.all(np.abs(got - want) <= bound)


def test_both_paths_share_buffers(q, monkeypatch):
    """the banded solves' work vectors are the position basis' buffers: one state more, beside the factors"""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("QPC_FAC_BYTES", "1")
    n_r, n_l, B = 400, 21, 256
    _, S, R, H = _grid(q, n_r, 6, n_l)
    state, factors = 16 * n_r * n_l * B, 16 * n_r * 7 * (n_l // 2) * B
    f = np.zeros((B, 2))
    used = []
    for _ in range(3):	# free memory is a whole-device figure that other processes move too
        prop = q.propagator_cn_hc_lgwz().initialize(n_r, 6, n_l, S, R, H, 0.05, n_inst=B)
        prop.put(np.ones((B, 1, n_l, n_r), complex))
        prop.run_dipole(f, np.ones(B), np.ones(B), R)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        prop.run_dipole(f, np.ones(B), np.ones(B), 0.5 * R)
        assert prop.path()["last_run"] == "banded"
        torch.cuda.synchronize()
        used.append(before - torch.cuda.mem_get_info()[0])
        prop.close()
        if used[-1] < factors + 1.6 * state:
            return
    pytest.fail("%s states beside the factors" % [(u - factors) / state for u in used])
