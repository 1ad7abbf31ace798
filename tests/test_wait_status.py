"""A wait that runs out in k_tc_apply skips its outputs and reports it in a status word.  No test can make such a wait run out,
so this reads the sources: every caller hands the kernel a word, and the velocity gauge clears and reads its word when
either of its two dense transforms has digit planes (they pass the exact-sum bound independently)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qpc-tdse-cpc_gb300", "csrc")


def _body(text, name):
    m = re.search(r"^(?:int|void|bool) %s\(.*?^}" % name, text, re.S | re.M)
    return m.group(0)


def test_velocity_gauge_reads_the_word_of_both_transforms():
    text = open(os.path.join(CSRC, "qpc_vpos.cu")).read()
    guard = re.search(r"bool on_tensor_cores\(\) const { return (.*?); }", text)
    assert guard and set(re.findall(r"\b(TD|TI)\.has_tc", guard.group(1))) == {"TD", "TI"} and "||" in guard.group(1)
    assert re.search(r"if \(p->on_tensor_cores\(\)\) QPC_CUDA\(cudaMemsetAsync\(p->status", _body(text, "vpos_begin"))
    assert re.search(r"if \(p->on_tensor_cores\(\)\) QPC_CUDA\(cudaMemcpyAsync\(p->hstatus, p->status", _body(text, "vpos_end"))
    assert "cudaMemsetAsync(p->status" in _body(text, "build")


def test_products_with_planes_get_a_status_word():
    for name in ("qpc_pos.cu", "qpc_vpos.cu"):
        for call in re.findall(r"band_apply\((.*?)\);", open(os.path.join(CSRC, name)).read()):
            args = [a.strip() for a in call.split(",")]
            assert len(args) == 4 or (len(args) == 7 and args[5] not in ("nullptr", "0")), call
