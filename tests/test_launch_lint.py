"""Lint of the kernels that are launched with programmatic serialization (CPU
only).  Such a kernel may be placed before the one in front of it has ended.  Its
first statement has to be dep_wait(), and it may declare only what no launch of
the solve writes to be unchanging for its whole life: by __ldg (or another
read-only load), or by a const __restrict__ parameter."""
import glob
import os
import re

from conftest import ROOT
from test_race_lint import code_lines

CSRC = os.path.join(ROOT, "ecl-suite_b200", "csrc")

# the solves' inputs
INPUTS = {"nindex", "nlist", "eweight", "vbase", "ebase", "avgs"}
# functions of cooperative launches, which start after everything before them,
# and the measurement probes
PLAIN = {"gc_pull", "gc_long_row", "gc_short_row", "mst_boruvka", "scc_giant", "scc_solve", "rs_sort", "gather_kernel"}

HEAD = re.compile(r"(?:__global__|__device__)[^;{}=]*?\b(\w+)\s*\(")


def functions(text):
    """(name, parameters, body) of every device function with a body."""
    text = "\n".join(code_lines(text))
    text = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in HEAD.finditer(text):
        at, depth = m.end(), 1
        while depth and at < len(text):  # the parameter list
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params = text[m.end():at - 1]
        rest = re.match(r"\s*(?:const)?\s*\{", text[at:])
        if not rest:
            continue
        beg = at = at + rest.end()
        depth = 1
        while depth and at < len(text):
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), params, text[beg:at - 1]


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        yield os.path.basename(path), open(path).read()


def early_loads(text):
    """Unchanging loads of something other than an input."""
    found = []
    for name, params, body in functions(text):
        if name in PLAIN:
            continue
        for arr in re.findall(r"const\s+[\w\s]+\*\s*__restrict__\s+(\w+)", params):
            if arr not in INPUTS:
                found.append(f"{name}: const __restrict__ {arr}")
        for arr in re.findall(r"__ld(?:g|cs)\(\s*(?:reinterpret_cast<[^>]*>\()?&?(?:\w+\.)?(\w+)", body):
            if arr not in INPUTS and not (name == "ldg" and arr == "p"):
                found.append(f"{name}: __ldg of {arr}")
    return found


def test_only_inputs_are_declared_unchanging():
    bad = [f"{f}: {x}" for f, text in sources() for x in early_loads(text)]
    assert not bad, "\n".join(bad)


def test_every_kernel_placed_early_waits_first():
    bodies, launched = {}, set()
    for f, text in sources():
        bodies.update({n: b for n, _, b in functions(text)})
        code = "\n".join(code_lines(text))
        for call in re.findall(r"(?:ECL_LAUNCH_NEXT|launch_cluster)\(([^;]*?),", code):
            launched |= {x for x in re.findall(r"\b(\w+)(?:<\w+>)?", call) if x in bodies}
    assert len(launched) > 25
    late = [k for k in sorted(launched) if not re.match(r"\s*(?:dev::)?dep_wait\(\);", bodies[k])]
    assert not late, late


def test_the_lint_catches_an_early_load(tmp_path):
    text = ("__device__ int help(const int* a, int v) { return __ldg(&a[v]); }\n"
            "__global__ void k(const int* __restrict__ nindex, const int* __restrict__ parent, int* out) {\n"
            "  dep_wait();\n"
            "  out[0] = parent[__ldg(&nindex[0])] + __ldg(&out[1]);\n"
            "}\n")
    assert early_loads(text) == ["help: __ldg of a", "k: const __restrict__ parent", "k: __ldg of out"]
