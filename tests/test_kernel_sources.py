"""Rules of the CUDA sources whose breach shows on the GPU only by a race or a fault,
if at all: checked on the text of every kernel."""
import glob
import os
import re

import pytest

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "pyfwix_b200", "csrc")


def _match(s, i, open_, close):
    """Index behind the bracket that closes the one at i."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == open_) - (s[k] == close)
        if depth == 0:
            return k + 1
    raise ValueError("unbalanced brackets")


def kernels():
    """(name, parameters, body) of every kernel, comments removed."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", s):
            k = s.index("k_", m.end())
            name = re.match(r"\w+", s[k:]).group()
            p0 = s.index("(", k)
            p1 = _match(s, p0, "(", ")")
            b0 = s.index("{", p1)
            out.append((os.path.basename(path) + ":" + name, s[p0:p1], s[b0:_match(s, b0, "{", "}")]))
    return out


KERNELS = kernels()
CHAINED = [k for k in KERNELS if "chain_wait()" in k[2]]


def test_kernels_are_found():
    names = {k[0] for k in CHAINED}
    for n in ("pointwise.cu:k_record", "spectral.cu:k_weight", "fast.cuh:k_col_b_tma", "flex.cuh:k_row_inv"):
        assert n in names


@pytest.mark.parametrize("name,params,body", CHAINED, ids=[k[0] for k in CHAINED])
def test_chained_kernels_read_through_plain_pointers(name, params, body):
    """A chained kernel runs while the kernel before it still writes: const
    __restrict__ would promise that nobody does."""
    for p in params.split(","):
        assert not ("const" in p and "__restrict__" in p), p
    assert body.index("chain_wait()") < min([body.find(t) for t in ("return", "a.in[") if t in body] or [len(body)])


TMA = [k for k in KERNELS if "mbar_wait(" in k[2]]


@pytest.mark.parametrize("name,params,body", TMA, ids=[k[0] for k in TMA])
def test_tma_kernels_leave_with_no_load_in_flight(name, params, body):
    """A CTA that gives up on a wait lets its own loads land first (bail), and no
    barrier is armed again before the wait on it was checked by the whole CTA."""
    exits = [m.start() for m in re.finditer(r"__syncthreads_and\(", body)]
    assert exits
    for i in exits:
        block = body[body.index("{", i):]
        block = block[:_match(block, 0, "{", "}")]
        assert "bail(" in block and "return" in block, block
    armed = [m.start() for m in re.finditer(r"issue_q\(term \+", body)]
    for i in armed:
        wait = max(body.rfind(w, 0, i) for w in ("= tma::mbar_wait(&bar[2]", "= wait_q("))
        assert wait >= 0 and "__syncthreads_and(" in body[wait:i], body[wait:i]


def test_phase_slots_are_fenced_before_their_next_load():
    """A phase tile is read by plain loads and overwritten by TMA: the reading lanes pass
    a proxy fence and a CTA barrier in between."""
    body = {k[0]: k[2] for k in KERNELS}
    a = body["fast.cuh:k_col_a_tma"]
    free = a[a.index("auto stage_free"):]
    free = free[:free.index("};")]
    assert 0 <= free.find("fence_proxy_async()") < free.find("__syncthreads()")
    read, issue = a.index("qr[T::qat("), a.index("issue_q(term + C::SLOTS)")
    assert "stage_free()" in a[read:issue]
    late = a.index("issue_q(term + C::SLOTS)", issue + 1)  # the other place: behind the store's fence and barrier
    put = a[a.index("auto store ="):]
    put = put[:put.index("};")]
    assert 0 <= put.find("fence_proxy_async()") < put.find("__syncthreads()") and "store(term);" in a[issue:late]
    b = body["fast.cuh:k_col_b_tma"]
    read, issue = b.index("qr[C::qat("), b.index("issue_q(term + 1)")
    fence = b.find("fence_proxy_async()", read)
    assert read < fence < b.index("__syncthreads_and(good)", read) < issue
