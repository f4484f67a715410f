"""Groups of more X than the ring of three holds take two ring slots: with three
and more groups in flight each slot is written again while the other is read."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# three groups and a short last one; a range that begins and ends inside groups
@pytest.mark.parametrize("no,nu,form,begin,end", [(8, 120, "fp64", 0, 112), (8, 128, "int8:3", 0, 112),
                                                  (8, 121, "int8:4", 9, 101)])
def test_two_slot_ring_is_bitwise_the_per_tuple_forward(no, nu, form, begin, end):
    from libcc_b200 import api
    inp = S.generate(no, nu, 11, "normal")
    with api.TriplesPlan.for_form(no, nu, form) as plan:
        plan.set_system(inp)
        grouped = plan.forward(begin, end)
        again = plan.forward(begin, end)
        plan.set_profiling(True)
        single = plan.forward(begin, end)
    for other in (again, single):
        assert grouped[0] == other[0] and grouped[1] == other[1] and np.array_equal(grouped[2], other[2])
