"""Kernels that start before the kernel ahead of them has ended promise nothing about its data.

`const __restrict__` and __ldg say that the memory is constant from the kernel's start; a kernel
that calls overlap_launch() starts while its predecessor still writes the LSQR vectors and
scalars.  No result shows it (the compiler keeps the loads behind the wait today), so the
sources are read.
"""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "crowdphot.jl_b200", "csrc", "cpb_sim.cu")
# parameters through which the kernels of an inner iteration hand their results on
CHAINED = {"k_gather": {"vt", "u_src", "outu", "sc"}, "k_JT": {"u", "z", "sc"},
           "k_lsqr_update": {"vt", "x", "wl", "sc"}}


def kernels():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    out = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*\)\s*)?(\w+)\(([^)]*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1)] = (m.group(2), text[m.end():i])
    return text, out


def test_chained_vectors_are_not_declared_constant():
    text, ks = kernels()
    found = {k for k, (_, body) in ks.items() if "overlap_launch()" in body}
    assert found == set(CHAINED)
    for k in found:
        params, body = ks[k]
        names = {re.search(r"(\w+)$", p.strip()).group(1): p for p in params.split(",")}
        assert CHAINED[k] <= set(names), k
        for n in CHAINED[k]:
            assert "__restrict__" not in names[n], (k, n)
            assert not re.search(r"__ldg\(\s*&?\(?%s\b" % n, body), (k, n)


def test_their_vector_loads_are_plain():
    text, _ = kernels()
    bodies = re.findall(r"void ld_px16\([^{]*\{([^}]*)\}", text)
    assert len(bodies) == 2 and not any("__ldg" in b for b in bodies)
