"""Kernels launched before the end of the launch they depend on (launch_pdl) read what that launch writes
with ordinary loads: a read-only load, or a const pointer declared __restrict__ in a helper, lets the
compiler move the load above the wait.  Read from the sources: every function that such a kernel
reaches."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "emerge_gb300", "csrc")


def _functions():
    """name -> (parameters, body) of the device functions and kernels of all sources."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|__(?:launch_bounds|maxnreg|align)__\s*\([^)]*\)", "", open(path).read())
        for m in re.finditer(r"__(?:global|device)__[^;{}()]*?\b(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params, j = text[m.end():i], i
            while text[j] in " \n":
                j += 1
            if text[j] != "{":
                continue
            depth, k = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[k], 0)
                k += 1
            out.setdefault(m.group(1), []).append((params, text[j:k]))
    return out


def _chained():
    names = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        names |= set(re.findall(r"launch_pdl\(\s*(?:\w+::)*(k_\w+)", text))
        # kernels chosen first: auto name = cond ? k_a<1> : k_b<2>; ... launch_pdl(name, ...)
        for m in re.finditer(r"launch_pdl\(\s*(?!k_)([a-z]\w*)\s*,", text):
            names |= set(re.findall(r"\b(k_\w+)<", re.findall(r"auto " + m.group(1) + r" = ([^;]*);", text[:m.start()])[-1]))
    return names


def test_loads_after_the_wait():
    funcs, kernels = _functions(), _chained()
    assert {"k_scales", "k_fill_small", "k_series64", "k_gj_row", "k_couple", "k_rowmv", "k_rows8", "k_slab_split",
            "k_gj_update_tc"} <= kernels <= set(funcs)
    bad = []
    for kernel in sorted(kernels):
        todo, seen = [kernel], set()
        while todo:
            f = todo.pop()
            if f in seen:
                continue
            seen.add(f)
            for params, body in funcs[f]:
                if re.search(r"__ld(g|cg|ca|cs|lu|cv)\b|ld\.global\.nc|\bReadOnly\b", body):
                    bad.append(f"{kernel}: {f} has a read-only or unordered load")
                if f != kernel and re.search(r"const\s+\w+\s*\*\s*__restrict__", params):
                    bad.append(f"{kernel}: {f} takes a const __restrict__ pointer")
                todo += [g for g in set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\s*\(", body)) | set(re.findall(r"\b(\w+)::", body))
                         if g in funcs]
    assert not bad, "\n".join(bad)
