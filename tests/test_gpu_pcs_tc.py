"""The projections of spectrum_c_pcs as digit sums on the tensor cores (csrc/qpc_tcband.cu) against a sum in extended precision, where the
kernel changes shape: the edges of its 128 momenta, 32 wavefunctions and 32-deep stages, one to three segments of columns,
several m, rows of very different size.  An output drops less than 2^-50 of the row's largest entry times the channel's
largest coefficient per 250 terms, and is rounded a few times."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(rng, nkr, nl, n_r, n_ch):
    k = np.linspace(0.05, 2.0, nkr)
    size = 10.0 ** rng.uniform(-200, 3, (nkr, nl, 1))
    size[0] = 0.0
    ijl = size * np.sin(k[:, None, None] * 0.3 * np.arange(n_r) + rng.uniform(0, 6, (nkr, nl, 1)))
    return dict(kr=k, kt=np.zeros(1), kp=np.zeros(1), ijl=ijl, plm=np.ones((1, n_ch)), exm=np.ones((1, 1), complex),
                cps=np.exp(1j * rng.uniform(0, 6, (nkr, nl))))


@pytest.mark.parametrize("n_r,nkr,n_inst,n_l,n_m,m0", [
    (33, 1, 1, 3, 1, 0), (32, 127, 31, 2, 1, 0), (95, 128, 32, 4, 3, -1), (160, 129, 33, 3, 2, 1), (400, 257, 65, 2, 1, 0), (896, 40, 5, 3, 1, 0),
    (897, 40, 5, 3, 1, 0), (1000, 30, 2, 33, 1, 0), (1900, 130, 7, 2, 1, 0)])
def test_projections(q, n_r, nkr, n_inst, n_l, n_m, m0):
    rng = np.random.default_rng(n_r + nkr)
    nl = max(abs(m0), abs(m0 + n_m - 1)) + n_l
    t = _tables(rng, nkr, nl, n_r, n_m * n_l)
    t["plm"] = t["plm"].reshape(1, n_m, n_l)
    t["exm"] = np.ones((1, n_m), complex)
    pcs = q.spectrum_c_pcs(nkr, 1, 1).initialize(n_r, 6, n_l, q.linear_knots(n_r, 6, 0.0, 0.5 * n_r), 0.05, 2.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0, n_m, m0,
                                                 tables=t)
    c = (rng.standard_normal((n_inst, n_m, n_l, n_r)) + 1j * rng.standard_normal((n_inst, n_m, n_l, n_r))) * 10.0 ** rng.uniform(-9, 9, (n_inst, n_m, n_l, 1))
    c[0, 0, 0] = 0.0
    got = pcs.measure_lmd(c)
    pcs.close()
    for im in range(n_m):
        for il in range(n_l):
            l = abs(m0 + im) + il
            want = 0.797884560802865 * np.einsum("kr,ir->ik", t["ijl"][:, l].astype(np.longdouble), c[:, im, il].astype(np.clongdouble)) * t["cps"][:, l]
            bound = np.abs(t["ijl"][:, l]).max(-1) * np.abs(c[:, im, il]).max(-1)[:, None]
            assert np.all(np.abs(got[:, :, im, il] - want) <= 2.0 ** -50 * max(1.0, n_r / 250) * 4 * bound)


def test_not_finite_table(q):
    """a table with a value that is not finite takes the plain sums: only its own momentum and channel are touched"""
    rng = np.random.default_rng(1)
    t = _tables(rng, 20, 2, 64, 2)
    t["plm"] = t["plm"].reshape(1, 1, 2)
    t["ijl"][3, 1, 5] = np.nan
    pcs = q.spectrum_c_pcs(20, 1, 1).initialize(64, 6, 2, q.linear_knots(64, 6, 0.0, 32.0), 0.05, 2.0, 0.0, 0.0, 0.0, 0.0, 1.0, tables=t)
    got = pcs.measure_lmd(rng.standard_normal((9, 1, 2, 64)) + 0j)
    bad = np.zeros(got.shape[1:], bool)
    bad[3, 0, 1] = True
    assert np.all(np.isnan(got[:, bad])) and np.all(np.isfinite(got[:, ~bad]))
