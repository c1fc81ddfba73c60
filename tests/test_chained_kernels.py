"""Kernels launched while their predecessor ends (griddepcontrol) read what it writes by ordered, coherent loads only.

A non-coherent load (__ldg, or a load that the compiler makes one through const __restrict__) is defined for memory
that nobody writes while the kernel lives, and a __restrict__ pointer lets the compiler move accesses across the
wait.  Shown on the sources: a wrong value needs a race that no run has to show.
"""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "alps_b200", "csrc")
# what the kernels of the chain write for one another: vectors, partial sums, scalars
CHAIN = ("x", "xr", "y", "vprev", "alpha_part", "beta_part", "part", "partB", "beta_prev", "alpha_out", "beta_out")


def _functions():
    """(name, parameter text, body, chained kernel) of every function in the CUDA sources."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"(\w+)\s*\(([^;{}]*)\)\s*\{", text):
            if m.group(1) in ("if", "for", "while", "switch"):
                continue
            depth, i = 1, m.end()
            while depth and i < len(text):
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            head = text[max(0, m.start() - 160):m.start()]
            head = head[max(head.rfind("}"), head.rfind(";")) + 1:]
            body = text[m.end():i]
            out.append((m.group(1), m.group(2), body, "__global__" in head and "chain_wait()" in body))
    return out


FUNCTIONS = _functions()


def _reached(name):
    """The functions that a body reaches, by name."""
    todo, seen = [name], set()
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for fn, _, body, _ in FUNCTIONS:
            if fn == n:
                todo += [w for w in set(re.findall(r"\b(\w+)\s*[<(]", body)) if w in NAMES and w not in seen]
    return seen


NAMES = {f[0] for f in FUNCTIONS}
KERNELS = sorted({f[0] for f in FUNCTIONS if f[3]})


def test_the_chained_kernels_are_found():
    assert {"hvr_kernel", "spin_rows_kernel", "mom_rows_kernel", "lanczos_update_fin_kernel",
            "lanczos_normalize_fin_kernel", "axpy_kernel"} <= set(KERNELS)


@pytest.mark.parametrize("kernel", KERNELS)
def test_chained_kernel_reads_its_predecessors_results_coherently(kernel):
    reached = _reached(kernel)
    for name, params, body, _ in FUNCTIONS:
        if name not in reached:
            continue
        for p in CHAIN:
            assert not re.search(r"__restrict__\s+%s\s*(,|$)" % p, params), (name, p)
            if re.search(r"\*\s*(const\s+)?%s\s*(,|$)" % p, params):
                assert not re.search(r"__ldg\(\s*%s\b" % p, body), (name, p)
                assert not re.search(r"__ldg\(\s*reinterpret_cast[^;]*\b%s\b" % p, body), (name, p)
    # the names above are all pointers that a chained kernel takes
    for name, params, _, chained in FUNCTIONS:
        if name == kernel and chained:
            assert not re.search(r"__ldg\(\s*rw\.(ent|diag)\b", body)  # formed by the kernel before a handle's first product
            pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*(?:,|$)", params)
            assert set(pointers) <= set(CHAIN) | {"alpha_host", "beta_host"}, pointers
