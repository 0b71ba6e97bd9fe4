"""k_ilu_narrow (lywell_gb300/csrc/mlf_solver.cu): warps poll values of x in shared
memory that others store, and take a value as there once its high word is not
that of the absent one.  A vector access is one access per element in no stated
order, so the elements that are read have to be the 64-bit values that are
stored: with 32-bit elements a new high word could come with an old low word.
Such a race shows on no run that can be counted on; this looks at the source."""
import os
import re

from conftest import ROOT


def test_elements_read_are_the_elements_stored():
    src = open(os.path.join(ROOT, "lywell_gb300", "csrc", "mlf_solver.cu")).read()
    body = src[src.index("__device__ void ilu_narrow_sweep"):src.index("k_ilu_narrow(int N")]
    found = re.findall(r'"(ld|st)\.volatile\.shared(?:\.v\d)?\.([a-z]\d+)', body)
    assert {op for op, _ in found} == {"ld", "st"}
    assert {t[1:] for _, t in found} == {"64"}, found
