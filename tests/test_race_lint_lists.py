"""The race-freedom lint over the solvers' lists and bit sets (CPU only): what one
launch builds and another thread of it, or a later phase behind a grid barrier,
reads -- besides the per-vertex state that test_race_lint looks at."""
import os

import pytest

from test_race_lint import CSRC, SHARED, plain_accesses

# shared arrays per source file, by the names under which the kernels know them
LISTS = {
    "apsp.cu": ["A"],
    "cc.cu": ["ing", "chunks"],
    "flat_scan.cuh": ["tilerow"],
    "gc.cu": ["rank", "order", "keys", "skeys", "svals", "vhash", "nl2", "rowinfo"],
    "mis.cu": ["items"],
    "mst.cu": ["list", "rin"],
    "radix_sort.cu": ["kin", "vin", "kout", "vout", "order", "counts"],
    "scc.cu": ["fwd", "bwd", "next", "queue", "chunks", "bits", "comp", "top", "cur", "nxt", "wl", "in"],
}


@pytest.mark.parametrize("fname", sorted(LISTS))
def test_every_access_to_a_shared_list_is_atomic_or_justified(fname):
    bad = plain_accesses(os.path.join(CSRC, fname), LISTS[fname])
    assert not bad, "plain accesses to shared lists:\n" + "\n".join(bad)


def test_the_table_names_what_is_there():
    """Every name of the table is indexed somewhere in its file."""
    for fname, names in LISTS.items():
        text = open(os.path.join(CSRC, fname)).read()
        missing = [n for n in names if n + "[" not in text]
        assert not missing, (fname, missing)
        assert not set(names) & set(SHARED.get(fname, []))
