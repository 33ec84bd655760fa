"""The cluster form of k_tridiag (CL > 1) needs a cluster barrier between the loads of column 0, which every CTA
of the cluster reads, and the column loop, in which rank 0 overwrites that column and to_all writes into the other
CTAs' shared memory. Results show its absence only when a CTA starts late, so it is looked for in the source."""
import os
import re

from ultimateepm_gb300 import build


def test_a_cluster_barrier_stands_between_the_first_loads_and_the_column_loop():
    with open(os.path.join(build.CSRC, "tridiag_kernel.cuh")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    body = src[src.index("k_tridiag(S* __restrict__ H"):]
    load = body.index("ldc(A + r)")
    loop = body.index("for (int i = 0; i < n - 1; ++i)")
    first_store = body.index("stc(col,")
    assert load < loop < first_store < body.index("to_all(pacc")
    assert re.search(r"if constexpr \(CL > 1\) sync_cluster\(\);", body[load:loop])
