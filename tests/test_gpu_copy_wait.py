"""The reductions' bounded wait for their bulk copies, made to run out by its
poll limit: the copies still land, every block leaves, the call returns
CCT_ERR_TIMEOUT, and with the limit restored the same object gives its bits again."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu
TIMEOUT = 7


@pytest.mark.parametrize("no,nu,form", [(4, 17, "fp64"), (3, 24, "int8:5"), (8, 72, "fp64"), (6, 96, "int8:3")])
def test_plan_wait_runs_out_and_recovers(no, nu, form):
    from libcc_b200 import _native as N
    from libcc_b200 import api as A
    with A.TriplesPlan.for_form(no, nu, form) as p:
        p.set_system(S.generate(no, nu, 5))
        good = p.forward()
        N.check(N.load().ccT_debug_wait_limit(p._h, 0), "limit")
        with pytest.raises(N.CctError) as e:
            p.forward()
        assert e.value.status == TIMEOUT
        N.check(N.load().ccT_debug_wait_limit(p._h, -1), "limit")
        again = p.forward()
        assert again[:2] == good[:2] and np.array_equal(again[2], good[2])


@pytest.mark.parametrize("form,mode,bn", [("fp64", 0, 64), ("fp64", 1, 0), ("int8", 2, 0)])
def test_batch_wait_runs_out_and_recovers(form, mode, bn):
    from libcc_b200 import _native as N
    from libcc_b200 import batch as B
    shapes = [(3, 24), (5, 40), (2, 9)]
    with B.TriplesBatch(shapes, form=form) as b:
        for k, (no, nu) in enumerate(shapes):
            b.set_system(k, S.generate(no, nu, k))
        b.configure(mode, bn, 0, 1 << 20)
        good = b.forward()
        N.check(N.load().ccT_batch_debug_wait_limit(b._h, 0), "limit")
        with pytest.raises(N.CctError) as e:
            b.forward()
        assert e.value.status == TIMEOUT
        N.check(N.load().ccT_batch_debug_wait_limit(b._h, -1), "limit")
        again = b.forward()
        assert all(np.array_equal(x, y) for x, y in zip(good, again))


def test_wait_limit_without_a_plan_is_a_state_error():
    from libcc_b200 import _native as N
    assert N.load().ccT_debug_wait_limit(None, 0) == 6
