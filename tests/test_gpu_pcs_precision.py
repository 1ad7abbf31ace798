"""The projections of spectrum_c_pcs as digit sums are no further from a sum in extended precision than the plain FP64 sums of
the same handle without room for digit planes (QPC_ALLOC_MAX): outgoing waves against wave packets most of whose size is
near the nucleus, over one segment of columns, two and three, 8- and 7-bit digits (short and long rows), blocks of 16 to
32 wavefunctions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,nkr,n_inst", [(95, 87, 28), (167, 48, 13), (253, 42, 51), (400, 130, 5), (800, 250, 16), (1000, 40, 33), (1900, 64, 9)])
def test_digit_sums_are_no_worse(q, monkeypatch, n_r, nkr, n_inst):
    rng = np.random.default_rng(n_r)
    n_l = 3
    k = np.linspace(0.02, 2.5, nkr)
    r = 0.5 * np.arange(1, n_r + 1)
    l = np.arange(n_l)
    arg = k[:, None, None] * r - l[:, None] * np.pi / 2 + np.log(2 * k[:, None, None] * r) / k[:, None, None] + rng.uniform(-1, 1, (nkr, n_l, 1))
    t = dict(kr=k, kt=np.zeros(1), kp=np.zeros(1), ijl=np.sin(arg) * (0.5 / k)[:, None, None], plm=np.ones((1, 1, n_l)), exm=np.ones((1, 1), complex),
             cps=np.ones((nkr, n_l), complex))
    c = np.zeros((n_inst, n_l, n_r), complex)
    for weight, lo, hi in ((1.0, 0.0, 0.05), (0.2, 0.05, 0.3), (0.05, 0.2, 0.7)):
        x0, w, p, a = (rng.uniform(u, v, (n_inst, n_l, 1)) for u, v in ((lo * r[-1], hi * r[-1]), (2, 12), (-1.2, 1.2), (0, 6.28)))
        c += weight * np.exp(-((r - x0) / w) ** 2 + 1j * (p * r + a))
    want = 0.797884560802865405727 * np.einsum("klr,ilr->ikl", t["ijl"].astype(np.longdouble), c.astype(np.clongdouble))
    err = []
    for limit in (None, 8 * nkr * n_l * n_r + 65536):
        if limit:
            monkeypatch.setenv("QPC_ALLOC_MAX", str(limit))
        pcs = q.spectrum_c_pcs(nkr, 1, 1).initialize(n_r, 6, n_l, q.linear_knots(n_r, 6, 0.0, 0.5 * n_r), 0.02, 2.5, 0.0, 0.0, 0.0, 0.0, 1.0, tables=t)
        assert pcs.path()["segments"] == (0 if limit else -(-n_r // 896))
        monkeypatch.delenv("QPC_ALLOC_MAX", raising=False)
        got = pcs.measure_lmd(c[:, None])[:, :, 0]
        pcs.close()
        err.append(float(np.linalg.norm(got - want) / np.linalg.norm(want)))
    assert err[0] <= err[1], err
