"""
Kernels that start before their predecessor has ended (programmatic dependent launch) and what they read of it: through
load_fresh, from a pointer that is no __restrict__ parameter and not through the read-only path, or the load may move
above the wait.  Read from the CUDA sources.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "differentiable-fea_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _closing(s, i, pair):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j


def _functions(text):
    """(name, parameters, body) of the functions defined in a source, comments removed."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        if m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__", "sizeof"):
            continue
        j = _closing(text, m.end() - 1, "()")
        rest = text[j + 1:j + 40].lstrip() if j else ""
        if rest.startswith("{"):
            k = text.index("{", j)
            yield m.group(1), text[m.end():j], text[k:_closing(text, k, "{}")]


def _fresh_and_restricted(params, body):
    """(names that load_fresh reads, with locals resolved to the pointers they were made from; restricted parameters)"""
    alias = dict(re.findall(r"(\w+)\s*=\s*reinterpret_cast<[^(]*>\((\w+)\)", body))
    fresh = set(re.findall(r"load_fresh\(\s*(?:reinterpret_cast<[^(]*>\()?(\w+)", body))
    return {alias.get(n, n) for n in fresh} | fresh, set(re.findall(r"__restrict__\s+(\w+)", params))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_what_a_predecessor_wrote_is_read_unrestricted(path):
    for name, params, body in _functions(open(path).read()):
        fresh, restricted = _fresh_and_restricted(params, body)
        assert not fresh & restricted, (name, sorted(fresh & restricted))


def test_the_sources_are_understood():
    """The functions whose reads are the rule's point are found, with what they read."""
    found = {}
    for path in SOURCES:
        for name, params, body in _functions(open(path).read()):
            found.setdefault(name, set()).update(_fresh_and_restricted(params, body)[0])
    for name, reads in {"node_sum": "fe2", "k_apply": "y", "k_apply_ref_elem": "done", "k_frame_node_residual": "part",
                        "k_pcg_elem_fused_ref": "r", "k_mg_cg_elem": "z", "k_mg_cheb_apply_step": "d_in",
                        "k_frame_node_diag": "fb", "k_frame_node_fields": "elem"}.items():
        assert reads in found[name], (name, found.get(name))
