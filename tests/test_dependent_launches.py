"""Kernels that are launched before their predecessor has ended (they call wait_predecessor) must not read through the
non-coherent path: what they read is written while they are already resident, and ld.global.nc is defined for memory that
stays read-only for the kernel's whole life. So neither they nor the device functions they call use __ldg, or pointers
that promise the compiler as much (__restrict__)."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "grasph2_b200", "csrc")


def span(text, at, opening, closing):
    """The end of the bracketed text that starts at text[at]."""
    depth = 0
    for k in range(at, len(text)):
        depth += (text[k] == opening) - (text[k] == closing)
        if depth == 0:
            return k + 1
    raise ValueError("unbalanced %s" % opening)


def functions():
    """[(file, name, kernel?, text)] of every __global__ and __device__ function definition."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"(__global__|__device__)\b(?:[^;{}()]|__launch_bounds__\([^;{}]*?\)(?=\s+\w))*?\b(\w+)\s*(?=\()", text):
            at = m.end()
            if m.group(2) == "__launch_bounds__":
                at = span(text, at, "(", ")")
                n = re.match(r"\s*(\w+)\s*", text[at:])
                if not n:
                    continue
                name, at = n.group(1), at + n.end()
            else:
                name = m.group(2)
            end = span(text, at, "(", ")")
            b = re.match(r"\s*(const)?\s*\{", text[end:])
            if not b:
                continue  # a declaration
            out.append((f, name, m.group(1) == "__global__", text[at:span(text, end + b.end() - 1, "{", "}")]))
    return out


def test_no_non_coherent_reads_behind_an_early_launch():
    fs = functions()
    by_name = {}
    for f in fs:
        by_name.setdefault(f[1], []).append(f)
    todo = [f for f in fs if f[2] and "wait_predecessor()" in f[3]]
    assert {"k_near", "k_gravity_fold", "k_gravity_finish", "k_pairs_near", "k_pairs_finish", "k_chunk_lists",
            "k_leapfrog_fixed"} <= {f[1] for f in todo}
    seen, bad = set(), []
    while todo:
        f = todo.pop()
        if f[:2] in seen:
            continue
        seen.add(f[:2])
        if "__ldg(" in f[3] or "__restrict__" in f[3]:
            bad.append("%s: %s" % f[:2])
        for word in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", f[3])):
            todo += [g for g in by_name.get(word, []) if not g[2]]
    assert {"fold_slots", "pairs_near", "near_scan"} <= {name for _, name in seen}
    assert not bad, bad
