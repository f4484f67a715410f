"""The backward's recompute against W kept by the forward: the same kernels on the
same X, so every gradient has the same bits, whatever the place of the range in
the X ring (one group, a start inside a group, several groups with the ring in
use again, a short last group)."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nu,begin,end", [(2, 9, 0, 2), (4, 20, 3, 4), (8, 72, 5, 70), (8, 120, 0, 112),
                                             (8, 120, 9, 101), (6, 33, 30, 50)])
def test_recompute_equals_kept_w(no, nu, begin, end):
    from libcc_b200 import api as A
    inp = S.generate(no, nu, 21)
    grads = []
    for keep in (False, True):
        with A.TriplesPlan(no, nu, keep_w=keep) as p:
            p.set_system(inp)
            p.forward(begin, end)
            assert (p.kept_tuples == end - begin) == keep
            grads.append(p.backward(begin, end))
            again = p.backward(begin, end)
            assert all(np.array_equal(again[k], grads[-1][k]) for k in again)
    for k in grads[0]:
        assert np.array_equal(grads[0][k], grads[1][k]), k


@pytest.mark.parametrize("no,nu,begin,end", [(2, 9, 0, 2), (4, 36, 0, 16), (4, 20, 3, 4), (8, 72, 5, 70),
                                             (8, 120, 9, 101), (6, 33, 30, 50)])
def test_emulated_plan_t1_gradient_is_twice_v1(no, nu, begin, end):
    """dE/dT1 = 2 v1, summed by an emulated plan's backward from the W it rebuilds in
    FP64, several tuples a launch where they are small: the FP64 plan's v1 to 1e-12."""
    from libcc_b200 import api as A
    inp = S.generate(no, nu, 22)
    with A.TriplesPlan(no, nu) as p:
        p.set_system(inp)
        v1 = p.forward(begin, end)[2]
    with A.TriplesPlan.for_form(no, nu, "int8:5") as p:
        p.set_system(inp)
        p.forward(begin, end)
        g = p.backward(begin, end)["t1"]
        assert np.array_equal(p.backward(begin, end)["t1"], g)
    want = 2.0 * v1.reshape(no, nu).T.reshape(-1)  # v1(a,i), a fastest -> T1(i,a), i fastest
    assert np.abs(g - want).max() <= 1e-12 * np.abs(want).max()
