"""Shared memory that copies refill (TMA): a thread's ordinary loads are ordered before a copy
that another thread issues behind a barrier only by a proxy fence of the loading thread in
front of that barrier.  A missing fence shows in results only under load and seldom, so the
sources are read: in every kernel that issues copies again after its first ones, each refill is
behind a barrier that every thread reaches through a fence."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "kfvm-kokkos_b200", "csrc")
FENCE = r"smem_release_to_copies\(\);|fence\.proxy\.async\.shared::cta;"

# the source, the end of the kernel's first copies, and what refills a slot
KERNELS = [
    ("recon_sym.cu", "wait_start|bool ok = wait", r"\bissue\(k|planes\.refill"),
    ("recon_tc.cu", r"bool ok = mbar_wait", r"\bissue_tile\("),
    ("mlp.cu", r"int it = 0;", r"\btile_load\("),
]


@pytest.mark.parametrize("src,start,refill", KERNELS)
def test_refills_follow_a_fence_and_a_barrier(src, start, refill):
    with open(os.path.join(CSRC, src)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[re.search(start, text).end():]
    events = [(m.start(), m.group(0)) for m in re.finditer(FENCE + r"|__syncthreads\w*\(|" + refill, body)]
    found = 0
    for n, (_, e) in enumerate(events):
        if not re.match(refill, e):
            continue
        found += 1
        # walking back: a barrier, and a fence before it since the previous refill (a loop's first
        # refill: in the loop's body, which comes behind it in the text)
        back = [x for _, x in events[:n]]
        cut = max([k for k, x in enumerate(back) if re.match(refill, x)], default=-1)
        span = back[cut + 1:] if src != "mlp.cu" else [x for _, x in events[n + 1:]]
        bars = [k for k, x in enumerate(span) if x.startswith("__syncthreads")]
        fences = [k for k, x in enumerate(span) if re.match(FENCE, x)]
        assert bars and fences and min(fences) < max(bars), (src, span)
    assert found


@pytest.mark.parametrize("src", ["kernels.cu", "recon_sym.cu", "recon_tc.cu", "mlp.cu"])
def test_whoever_gives_up_records_it(src):
    """A thread that leaves because its own wait gave up sets the fault itself: another thread's
    wait on the same barrier may just have succeeded, and the step would then go on with the
    cells that were not written.  (Where the block decides together, one thread is enough.)"""
    with open(os.path.join(CSRC, src)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"if \(!mbar_wait\([^;{]*\{", text):
        assert re.match(r"\s*atomicExch\(&sc->fault, 1u\);", text[m.end():]), text[m.start():m.end() + 80]
