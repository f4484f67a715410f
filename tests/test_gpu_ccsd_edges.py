"""CCSD T1-dressing terms where the O1 kernels change shape: one to four column
fragments, no = 32 and past it (the W-build tile on gathered rows), nu at the
edges of the 16-wide chunks, and more rows than a pass of ten warps holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nu", [(1, 3), (2, 337), (9, 16), (16, 47), (17, 33), (25, 18), (32, 20), (33, 17)])
def test_terms_match_oracle_at_kernel_edges(no, nu):
    from libcc_b200 import api as A
    from oracle import oracle as O
    rng = np.random.default_rng(no * 1000 + nu)
    n4, nvv = no * nu * nu * no, nu * (nu + 1) // 2 * nu * no
    o1, vvvo = rng.normal(0, 0.1, no * nu), rng.normal(size=nvv)
    t2, vl, vr, o2, vm = (rng.normal(size=n) for n in (n4, n4, n4, n4, no ** 3 * nu))
    got = A.ccsd_terms_29_31(no, nu, o1, t2, vl, vr, vvvo)
    ref = O.literal_terms_29_30_31(no, nu, o1, t2.copy(), vl, vr, vvvo)
    # sums of up to nu + no products of FP64 values: a few hundred rounding errors of the largest term
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    got = A.ccsd_terms_32_35(no, nu, o1, o2, t2, vm, vvvo)
    ref = O.literal_terms_32_35(no, nu, o1, o2.copy(), t2.copy(), vm.copy(), vvvo)
    for name, g, r in zip(("t2", "o2", "vm", "rl"), got, ref):
        assert np.abs(g - r).max() <= 1e-12 * max(np.abs(r).max(), 1e-300), name
