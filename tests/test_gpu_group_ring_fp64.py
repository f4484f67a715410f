"""The two-slot X ring of FP64 plans, whose W builds alternate between two streams
beside a reduction stream: no8-nu120 and no9-nu120 run in groups of 28 tuples."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# a range that begins and ends inside groups, one that begins on a group and ends
# inside the fourth, five groups and a short last one
@pytest.mark.parametrize("no,begin,end", [(8, 9, 101), (8, 28, 110), (9, 0, 156)])
def test_fp64_ring_is_bitwise_the_per_tuple_forward(no, begin, end):
    from libcc_b200 import api
    inp = S.generate(no, 120, 11, "normal")
    with api.TriplesPlan(no, 120) as plan:
        plan.set_system(inp)
        grouped = plan.forward(begin, end)
        again = plan.forward(begin, end)
        plan.set_profiling(True)
        single = plan.forward(begin, end)
    for other in (again, single):
        assert grouped[0] == other[0] and grouped[1] == other[1] and np.array_equal(grouped[2], other[2])
