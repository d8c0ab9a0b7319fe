"""Kernels launched with launch_chained() are resident while earlier kernels of the chain still write
what they read, so they must not promise the compiler that this memory is read-only or unshared:
no __restrict__ parameters and no __ldg, in them or in the device functions that they call."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "treecode-accelerated-green-iteration_gb300", "csrc")


def _code(path):
    s = open(path).read()
    s = re.sub(r"//[^\n]*", "", s)
    return re.sub(r"/\*.*?\*/", "", s, flags=re.S)


def _functions(s):
    """name -> list of (signature, body) of the file's device functions and kernels."""
    out = {}
    for m in re.finditer(r"(?:__global__|__device__)[^;{}]*?\(", s):
        j = s.find("{", m.start())
        sig = s[m.start():j]
        if ";" in sig:
            continue
        depth, k = 0, j
        while True:
            depth += {"{": 1, "}": -1}.get(s[k], 0)
            if depth == 0:
                break
            k += 1
        plain = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", sig)
        name = re.search(r"(\w+)\s*(?:<[^<>]*>)?\s*\(", plain).group(1)
        out.setdefault(name, []).append((plain, s[j:k + 1]))
    return out


def _chained(s, fns):
    """Kernels that launch_chained() starts or that wait for earlier ones before they read."""
    waits = {n for n, v in fns.items() for sig, body in v if "chain_begin()" in body or "griddepcontrol.wait" in body}
    waits -= {"pass_end"}   # the field passes wait at their end: they read nothing that the chain writes
    names = {n for call in re.findall(r"launch_chained\(([^;]*?)\)", s, re.S) for n in re.findall(r"\w+", call)}
    # a kernel that calls a device function which waits is one too
    kernels = {n for n, v in fns.items() for sig, body in v if "__global__" in sig
               and (n in names or n in waits or any(re.search(rf"\b{w}\s*[(<]", body) for w in waits))}
    return kernels


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_chained_kernels_make_no_read_only_promise(path):
    s = _code(path)
    fns = _functions(s)
    todo, seen, bad = sorted(_chained(s, fns)), set(), []
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for sig, body in fns[n]:
            if "__restrict__" in sig or "__restrict__" in body or "__ldg(" in body:
                bad.append(n)
            todo += [c for c in fns if c not in seen and re.search(rf"\b{c}\s*(<[^;{{}}]*?>)?\s*\(", body)]
    assert not bad, f"{os.path.basename(path)}: {sorted(set(bad))}"


def test_chained_kernels_are_found():
    """The scan sees the kernels that it is about."""
    found = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        s = _code(path)
        found |= _chained(s, _functions(s))
    assert {"rs_histogram", "rs_scatter", "place_sorted", "bbox_final", "node_boxes", "preorder", "p2m_mixed", "p2m_reduce",
            "mesh_level", "mgs_dots", "mgs_subtract", "gemm_tc", "colsum_partial", "splitk_reduce", "prep_sources",
            "orbital_constants"} <= found
