"""Every copy and fill of the library is ordered on the stream of the work that uses it.  The handles' streams do not
block on the legacy stream, to which a plain cudaMemcpy or cudaMemset belongs: one that has returned may still be on its
way when a kernel on the handle's stream reads its target.  Which of the two comes first is not repeatable, so the
sources are checked."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qpc-tdse-cpc_gb300", "csrc")


def test_no_copy_or_fill_on_the_legacy_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        code = re.sub(r"//[^\n]*", "", open(path).read())
        found += ["%s: %s" % (os.path.basename(path), m) for m in re.findall(r"\b(cudaMemcpy(?:2D|ToSymbol)?|cudaMemset)\s*\(", code)]
    assert not found, found
