"""Sizes the position basis does not serve keep the banded solves: more channels (n_m x n_l) than a launch's second grid
dimension holds, on both sides of that limit.  Against QPC_POS=0; 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_m", [32767, 32768])
def test_many_channels(q, monkeypatch, n_m):
    n_r, p, n_l = 20, 3, 2
    m0 = -(n_m // 2)
    S, R, _, _, H = q.radial_setup(n_r, p, n_l + n_m // 2, q.linear_knots(n_r, p, 0.0, 10.0))
    c0 = np.random.default_rng(0).standard_normal((1, n_m, n_l, n_r)) + 0j
    out, paths = [], []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        prop = q.propagator_cn_hc_lgwz().initialize(n_r, p, n_l, S, R, H, 0.05, n_m=n_m, m0=m0, n_inst=1)
        prop.put(c0)
        prop.run(np.full((1, 4), 0.02), [3], [3])
        out.append(prop.get())
        paths.append(prop.path()["last_run"])
        prop.close()
    assert paths == ["banded", "position" if n_m * n_l <= 65535 else "banded"]
    assert rel_l2(out[1], out[0]) < 1e-12
