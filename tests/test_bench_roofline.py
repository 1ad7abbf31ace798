"""The bench's roofline names the kernel that ran: digit products on the tensor cores only where the handle reports
k_tc_apply, the operators' bytes for the multiply-add kernels of small batches and of QPC_POS_TC=0."""
import importlib.util
import os

import pytest

from conftest import ROOT

spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)


@pytest.mark.parametrize("product,bound", [("k_tc_apply", "tensor"), ("k_band_apply", "integer multiply-adds"), ("k_band_one", "hbm")])
def test_roofline_of_the_kernel_that_ran(product, bound):
    r = bench.pos_roofline({"fieldfree": (1.2, 12)}, 800, 41, 4, product)
    assert r["kernel"].startswith(product) and r["bound"] == bound and r["launch_ms"] == pytest.approx(0.1) and r["achieved"] > 0


def test_operator_entries():
    """n rows of 2 w + 1 entries less the corners"""
    assert bench.band_entries(1000, 1, 3, 1) == (3 * 1000 - 2, 7 * 1000 - 12 - (3 * 1000 - 2))
