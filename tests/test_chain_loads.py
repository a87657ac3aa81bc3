"""Kernels of an evaluation's chain are launched before their predecessor has finished
(launch_chain) and wait for it in pdl_begin().  A read of a predecessor's array therefore has
to be an ordinary load behind the wait: not the non-coherent path (__ldg, or a pointer that is
const and __restrict__), and not through a __restrict__ pointer, whose loads the compiler may
move above the wait.  Which loads are emitted is not visible in results, so the sources are
read: every kernel with pdl_begin() may have __restrict__ only on the stencil tables and on
arrays that it only writes, listed here."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "kfvm-kokkos_b200", "csrc")

RECON_OUT = {"F0", "F1", "F2", "W0", "W1", "W2", "src", "status", "lamvel", "bnd"}
# the arrays that a kernel of the chain writes and never reads
WRITTEN_ONLY = {
    "bc_fill_kernel": set(),
    "recon_tma_kernel": RECON_OUT,
    "recon_sym3_kernel": RECON_OUT,
    "recon_sym2_kernel": RECON_OUT,
    "flag_kernel": {"flag"},
    "compact_kernel": {"applied", "theta", "heavy"},
    "heavy_var_kernel": {"theta"},
    "riemann_kernel": set(),
    "riemann_dir": {"G"},
    "glm_sources": set(),
    "stage_kernel": {"Unext", "K", "part"},
    "finalize_kernel": set(),
    "stage_pre_kernel": {"U1", "Uhat", "Utmp"},
}
# device functions of those kernels that take their arrays
HELPERS = {"riemann_dir", "glm_sources"}


def _source():
    text = ""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            with open(os.path.join(CSRC, f)) as h:
                text += re.sub(r"//[^\n]*", "", h.read())
    return text


def _bracketed(s, i, a, b):
    """s[i] is `a`: the text up to the matching `b`, and the position after it."""
    n, k = 0, i
    while True:
        n += (s[k] == a) - (s[k] == b)
        k += 1
        if n == 0:
            return s[i + 1:k - 1], k


def _functions():
    """name -> (parameters, body) of the kernels that call pdl_begin(), and the helpers"""
    s, out = _source(), {}
    for m in re.finditer(r"\b(\w+)\(", s):
        if not (m.group(1).endswith("_kernel") or m.group(1) in HELPERS):
            continue
        params, k = _bracketed(s, m.end() - 1, "(", ")")
        if not re.match(r"\s*\{", s[k:]):
            continue
        body, _ = _bracketed(s, s.index("{", k), "{", "}")
        if "pdl_begin()" in body or m.group(1) in HELPERS:
            out[m.group(1)] = (params, body)
    return out


def test_every_chain_kernel_is_covered():
    s = _source()
    launched = set(re.findall(r"launch_chain\(\s*g\.chain,\s*(\w+)", s))
    assert launched and launched == {n for n in WRITTEN_ONLY if n not in HELPERS}
    assert set(_functions()) == set(WRITTEN_ONLY)


@pytest.mark.parametrize("name", sorted(WRITTEN_ONLY))
def test_reads_are_ordinary_loads_behind_the_wait(name):
    params, body = _functions()[name]
    assert "__ldg" not in body and "ld.global.nc" not in body
    if name not in HELPERS:
        # the wait comes before any use of a parameter: only type aliases may precede it
        head = body[:body.index("pdl_begin()")]
        assert all(re.match(r"\s*(using\b.*)?$", t, re.S) for t in head.split(";")), head
    restricted = {}
    for p in params.split(","):
        if "__restrict__" in p:
            restricted[p.split()[-1].lstrip("*")] = p
    for n, p in restricted.items():
        if "DevStencil" in p:
            continue
        assert "const" not in p, p
        assert n in WRITTEN_ONLY[name], p


def test_copies_are_ordered_behind_the_wait():
    """What pdl_begin's wait makes visible, it makes visible to ordinary loads: the thread that
    issues TMA copies of the predecessors' arrays passes a proxy fence first."""
    found = 0
    for name, (_, body) in _functions().items():
        if "tma_load_4d(" not in body:
            continue
        found += 1
        # (in recon_sym3_kernel the load stands in a function that the first loop calls)
        first = body.index("issue(p);" if "auto issue" in body else "tma_load_4d(")
        assert body.index("pdl_begin()") < body.index("global_acquire_for_copies();") < first, name
    assert found == 3
