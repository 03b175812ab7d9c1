"""Every read-out waits through ctx_sync, which reads the error flags of the kernels'
bounded waits: an expired wait leaves W, h2 or a Krylov step incomplete, and the entry
point has to fail.  The flags are set by a kernel that gave up, which no test provokes, so
the waits are counted in the sources."""
import os
import re

from codyfortran_gb300 import build

# waits of the set-up, before any kernel with a bounded wait has run
SET_UP = {"k_ci.cu": 3, "k_mixed.cu": 1}


def test_every_wait_reads_the_error_flags():
    found = {}
    for f in sorted(os.listdir(build.CSRC)):
        with open(os.path.join(build.CSRC, f)) as h:
            text = h.read()
        n = len(re.findall(r"cudaStreamSynchronize\(", text))
        if f == "ctx.cu":
            body = re.search(r"\nvoid ctx_sync\(cgpu_ctx\* c\) \{(.*?)\n\}", text, re.S).group(1)
            assert "sil_check(c)" in body and "mixed_error(c)" in body
            n -= len(re.findall(r"cudaStreamSynchronize\(", body))
        if n:
            found[f] = n
    assert found == SET_UP


def test_event_waits_are_followed_by_a_check():
    """An elapsed time is a read-out too: each wait for an event comes before a check of the flags."""
    for f in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, f)) as h:
            text = h.read()
        for m in re.finditer(r"cudaEventSynchronize\(", text):
            rest = text[m.end():text.index("\n}", m.end())]
            assert re.search(r"\b(ctx_)?sync\(c\)|mixed_error\(c\)", rest), f
