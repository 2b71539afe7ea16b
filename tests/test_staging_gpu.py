"""Copies of pageable host memory through the library's page-locked blocks:
what the pool keeps between calls, and every way in which a copy goes without
a block.  Each test runs in a process of its own, because the pool, the OpenMP
settings and the CUDA context belong to the process."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# A path of n vertices without every tenth link: labels, forest and weight are
# known without a solver.  The CSR and the outputs are above the size from
# which a copy goes through a block (256 kB).
PRELUDE = """
import sys
import numpy as np

sys.path.insert(0, sys.argv[1])
import ecl_b200 as ecl


def graph(n):
    link = np.arange(n - 1) % 10 != 9
    u = np.flatnonzero(link)
    row, col = np.concatenate([u, u + 1]), np.concatenate([u + 1, u])
    order = np.lexsort((col, row))
    row, col = row[order], col[order]
    nindex = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    w = 1 + np.minimum(row, col) % 1000
    g = ecl.Graph(nindex, col, w, True)
    want = np.arange(n) // 10 * 10
    return g, want, int((1 + u % 1000).sum())


def check(g, want, total):
    out = np.full(g.nodes, -1, np.int32)
    ecl.cc(g, out=out)
    assert np.array_equal(out, want)
    flags, weight = ecl.mst(g)
    assert weight == total and int(flags.sum()) == g.edges // 2
    return 1
"""


def run(body, **env):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body, os.path.join(ROOT, "ecl-suite_b200")],
                       env={**os.environ, **env}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split()[-1] == "done"


def test_blocks_do_not_outlive_their_context():
    """cudaDeviceReset ends the context and with it the blocks and their events:
    the solves after it make new ones, more often than there are blocks."""
    run("""
g = graph(300000)
for _ in range(6):
    check(*g)
    assert ecl.lib.cudaDeviceReset() == 0
check(*g)
print("done")
""", OMP_NUM_THREADS="4")


def test_allocation_free_cc_after_its_context_was_replaced():
    """ecl_cc_noalloc's scratch array has another address, or none yet, in the
    context that follows a reset, whose handle may well be the old one."""
    run("""
import ctypes as C

f = ecl.lib.ecl_cc_noalloc
f.restype, f.argtypes = C.c_int, [C.c_int32, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
rt = ecl.lib
rt.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
g, want, _ = graph(20000)
for k in range(3):
    pad, d = C.c_void_p(), [C.c_void_p() for _ in range(3)]
    assert rt.cudaMalloc(C.byref(pad), (k + 1) << 20) == 0  # another start for what the context loads
    for p, a in zip(d, (g.nindex, g.nlist, want.astype(np.int32))):
        assert rt.cudaMalloc(C.byref(p), a.nbytes) == 0
        assert rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, 1) == 0
    for _ in range(2):
        assert f(g.nodes, g.edges, d[0], d[1], d[2], None) == ecl.OK
    out = np.empty(g.nodes, np.int32)
    assert rt.cudaMemcpy(out.ctypes.data, d[2], out.nbytes, 2) == 0
    assert np.array_equal(out, want)
    assert rt.cudaDeviceReset() == 0
print("done")
""")


@pytest.mark.parametrize("threads", ["1", "3", "4", "8"])
def test_copies_with_any_number_of_host_threads(threads):
    """Below four host threads every copy is plain, from four on they fill the
    blocks; the results are the same."""
    run("""
for n in (65537, 262145, 1350001):
    check(*graph(n))
print("done")
""", OMP_NUM_THREADS=threads)


@pytest.mark.parametrize("users", [1, 4, 5, 9])  # as many as there are blocks, and more
def test_blocks_shared_by_threads(users):
    """Every call of every thread goes through and is right; an exception in a
    thread ends the test."""
    run(f"""
from concurrent.futures import ThreadPoolExecutor

graphs = [graph(n) for n in (65537, 262145, 300001, 1048577)]
with ThreadPoolExecutor({users}) as pool:
    jobs = [pool.submit(check, *graphs[(k + i) % len(graphs)]) for k in range({users}) for i in range(2 * len(graphs))]
    assert sum(j.result() for j in jobs) == {users} * 2 * len(graphs)
print("done")
""", OMP_NUM_THREADS="4")


def test_page_locked_arrays_are_copied_as_they_are():
    run("""
import torch

g, want, total = graph(300001)
pin = lambda a: torch.from_numpy(a).pin_memory().numpy()
locked = ecl.Graph(pin(g.nindex), pin(g.nlist), pin(g.eweight), True)
out = torch.empty(g.nodes, dtype=torch.int32).pin_memory().numpy()
ecl.cc(locked, out=out)
assert np.array_equal(out, want)
for _ in range(2):
    check(locked, want, total)
    check(g, want, total)
print("done")
""", OMP_NUM_THREADS="4")
