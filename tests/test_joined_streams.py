"""The first kernel behind a wait for another stream's event is launched without
overlap: wherever a context's stream waits, the context notes it, and the
launches ask (the sources are read; no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "flecsph_gb300", "csrc")


def test_every_wait_is_noted():
    src = "".join(open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    src = re.sub(r"//[^\n]*", "", src)
    waits = [m.end() for m in re.finditer(r"cudaStreamWaitEvent\((mb\.)?c->stream,[^;]*;", src)]
    assert len(waits) >= 4
    for w in waits:
        assert re.match(r"\s*(mb\.)?c->joined = true;", src[w:]), src[w - 90:w + 60]
    # no launch takes the attribute without asking
    assert len(re.findall(r"numAttrs = L\.overlap\(\)", src)) == 2
    assert not re.search(r"numAttrs = L\.chained", src)
