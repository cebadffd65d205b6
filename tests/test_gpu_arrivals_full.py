"""Arrivals where the ordering and the replay work hardest, against the oracle, which
applies them one after another: cells that fill and evict with more than 32 slots (the
lanes of a warp look at two or three slots each for the weakest), and more than
1,048,576 candidates (the radix sort's scan of a digit takes more than one pass of 1024
tiles).

Candidates are the same FP64 contributions; their amplitudes differ from the oracle's in
the last bits, so of two nearly equal weakest arrivals either may be evicted. Counts are
equal, and so are the sorted amplitudes of a cell within 1e-4, as far as single
amplitudes are equal elsewhere. Without eviction the order is the oracle's too."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200 import workloads as W
from bellhopcuda_b200.envfile import write_env
import oracle_ctypes

pytestmark = pytest.mark.gpu


def both(spec, max_narr, merging, root):
    o = oracle_ctypes.run(spec, max_narr=max_narr, allow_merging=int(merging))
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.set_arrival_options(max_narr, merging)
        narr, arr = t.setup(write_env(spec, root)).run().arrivals()
        assert t.stats()["evals"] == o["nevals"]
    np.testing.assert_array_equal(narr, o["narr"])
    return narr, arr, o["arr"]


@pytest.mark.parametrize("merging", [True, False], ids=["merge", "append"])
@pytest.mark.parametrize("max_narr", [33, 64, 70])
def test_full_cells(max_narr, merging, tmp_path):
    s = W.munk_tl(nalpha=1601, nrz=5, nrr=7, beam="B")
    s.run_type = "aB RR "
    narr, arr, ref = both(s, max_narr, merging, os.path.join(str(tmp_path), "e"))
    assert (narr == max_narr).mean() > 0.4
    for cell in np.argwhere(narr > 0):
        k = narr[tuple(cell)]
        a, b = arr[tuple(cell)][:k]["a"], ref[tuple(cell)][:k]["a"]
        np.testing.assert_allclose(a if not merging else np.sort(a), b if not merging else np.sort(b), rtol=1e-4)


def test_more_candidates_than_a_scan_pass(tmp_path):
    s = W.munk_tl(nalpha=4001, nrz=41, nrr=101, beam="B")
    s.run_type = "aB RR "
    narr, arr, ref = both(s, 1500, False, os.path.join(str(tmp_path), "e"))
    assert narr.sum() > 1 << 20   # (full cells keep their first 1500)
    n = narr[..., None] > np.arange(1500)
    g, r = arr[n], ref[n]
    np.testing.assert_array_equal(g["NTopBnc"], r["NTopBnc"])
    np.testing.assert_array_equal(g["NBotBnc"], r["NBotBnc"])
    np.testing.assert_allclose(g["SrcDeclAngle"], r["SrcDeclAngle"], rtol=1e-5, atol=1e-5)
    np.testing.assert_allclose(g["delay_re"], r["delay_re"], rtol=1e-6)
    np.testing.assert_allclose(g["a"], r["a"], rtol=1e-4)
