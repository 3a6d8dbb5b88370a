"""Properties of the kernels that no run shows reliably, read from their sources."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "numfast_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _body(text, kernel):
    """Text of a __global__ function from its name to the next one."""
    at = re.search(r"__global__[^;{]*\b%s\(" % kernel, text).end()
    end = text.find("__global__", at)
    return text[at:end if end >= 0 else len(text)]


def test_sample_state_is_read_before_it_is_moved_on():
    """k_tk_sample: every thread of the last CTA reads the target rank, one thread writes the next
    one after the scan; only the scan's barriers are between them."""
    body = _body(_source("topk.cu"), "k_tk_sample")
    last_read = max(m.end() for f in ("target", "below") for m in re.finditer(r"st->%s\b(?!\s*=[^=])" % f, body))
    first_write = min(m.start() for f in ("target", "below") for m in re.finditer(r"st->%s\s*=[^=]" % f, body))
    assert "block_excl_scan" in body[last_read:first_write]


def test_shared_arrays_read_as_vectors_are_aligned():
    """A __shared__ array that is accessed by 16-byte vectors declares that alignment."""
    loose = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = _source(os.path.basename(path))
        for name in set(re.findall(r"reinterpret_cast<(?:const )?(?:u?int4|ulonglong2|double2)\*>\(&?(\w+)\b", text)):
            for decl in re.findall(r"[^;{}]*__shared__[^;{}]*\b%s\s*\[[^;{}]*;" % name, text):
                if "__align__(16)" not in decl and "__align__(128)" not in decl:
                    loose.append((os.path.basename(path), " ".join(decl.split())))
    assert not loose, loose
