"""Masks in runs on a handle of the position basis (csrc/qpc_pos.cu): zeros, a size the fixed-point operators decline (the
banded solves then serve the run), and a handle that goes from one path to the other and back with its state.  Against a
handle of the banded solves (QPC_POS=0); 1e-12, the bar of the short runs."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_pos import _grid

pytestmark = pytest.mark.gpu

N, P, L, B = 130, 6, 5, 3


def _both(q, monkeypatch, calls):
    t, S, R, H = _grid(q, N, P, L)
    rng = np.random.default_rng(4)
    c0 = (rng.standard_normal((B, 1, L, N)) + 1j * rng.standard_normal((B, 1, L, N))) * np.exp(-0.03 * np.arange(N))
    mask = q.mask_band(N, P, t, 0.3 * N, 0.5 * N)
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QPC_POS", mode)
        prop = q.propagator_cn_hc_lgwz().initialize(N, P, L, S, R, H, 0.05, n_inst=B)
        prop.put(c0)
        out.append(calls(prop, R, mask))
        prop.close()
    return out


def _f(seed, steps):
    return 0.05 * np.random.default_rng(seed).standard_normal((B, steps + 1))


def test_zero_mask(q, monkeypatch):
    def calls(prop, R, mask):
        prop.run_ex(_f(1, 4), [4, 2, 0], [4, 3, 0], mask=np.zeros_like(mask))
        return prop.get(), prop.path()["last_run"]

    (a, pa), (b, pb) = _both(q, monkeypatch, calls)
    assert (pa, pb) == ("banded", "position")
    assert np.all(a[:2] == 0) and np.all(b[:2] == 0) and np.array_equal(a[2], b[2]) and np.any(b[2] != 0)


def test_declined_mask(q, monkeypatch):
    """entries of 1e210: beyond what an operator's exponent may be, finite all the same"""
    def calls(prop, R, mask):
        prop.run_ex(_f(2, 1), [1, 1, 0], [1, 1, 0], mask=1e210 * mask)
        return prop.get(), prop.path()["last_run"]

    (a, _), (b, path) = _both(q, monkeypatch, calls)
    assert path == "banded"
    for k in range(B):
        scale = 1e210 if k < 2 else 1.0
        assert rel_l2(b[k] / scale, a[k] / scale) < 1e-12, k


def test_paths_in_turn(q, monkeypatch):
    def calls(prop, R, mask):
        paths, out = [], []

        def note():
            paths.append(prop.path()["last_run"])

        nf, nt = np.array([3, 1, 2]), np.array([3, 4, 2])
        prop.run(_f(3, 3), nf, nt), note()
        out.append(prop.norm())
        out.append(prop.run_dipole(_f(4, 3), nf, nt, 0.5 * R)), note()	# another operator than R
        prop.run_ex(_f(5, 3), nf, nt, mask=mask), note()
        prop.mask(mask)
        out.append(prop.dipole(R))
        out.append(prop.run_dipole(_f(6, 3), nf, nt, R)), note()
        prop.run_ex(_f(7, 1), np.ones(B), np.ones(B), mask=1e210 * mask), note()
        prop.run_ex(_f(8, 1), np.ones(B), np.ones(B), mask=1e-150 * mask), note()
        prop.run_ex(_f(9, 1), np.ones(B), np.ones(B), mask=1e-60 * mask), note()
        out.append(prop.norm())
        out.append(prop.get())
        return out, paths

    (a, pa), (b, pb) = _both(q, monkeypatch, calls)
    assert pa == ["banded"] * 7 and pb == ["position", "banded", "position", "position", "banded", "position", "position"]
    for k, (x, y) in enumerate(zip(a, b)):
        assert rel_l2(y / np.abs(x).max(), x / np.abs(x).max()) < 1e-12, k


@pytest.mark.parametrize("state,scale", [(1e200, 1e150), (1e150, 1e190)])
def test_overflow_is_reported(q, monkeypatch, state, scale):
    """a mask that grows the state past the largest double"""
    def calls(prop, R, mask):
        prop.put(state * prop.get())
        with pytest.raises(q.QpcError) as e:
            prop.run_ex(_f(3, 1), np.ones(B), np.ones(B), mask=scale * mask)
        return e.value.code

    assert _both(q, monkeypatch, calls) == [5, 5]
