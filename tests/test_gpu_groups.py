"""Tuple groups of the forward: a profiled forward launches one tuple at a time,
an ordinary one a group of tuples per launch, in the same order of sums."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# one group of every tuple, groups that end inside a range, a last group of one, both tuple kinds in a group
@pytest.mark.parametrize("no,nu,form,begin,end", [(2, 5, "fp64", 0, 2), (4, 36, "fp64", 0, 16), (4, 36, "fp64", 3, 4),
                                                  (7, 24, "fp64", 5, 70), (8, 24, "fp64", 31, 97),
                                                  (9, 83, "int8:4", 7, 92), (5, 17, "int8:3", 0, 30),
                                                  (3, 130, "fp64", 1, 7)])
def test_grouped_forward_is_bitwise_the_per_tuple_forward(no, nu, form, begin, end):
    from libcc_b200 import api
    inp = S.generate(no, nu, 11, "normal")
    with api.TriplesPlan.for_form(no, nu, form) as plan:
        plan.set_system(inp)
        grouped = plan.forward(begin, end)
        plan.set_profiling(True)
        single = plan.forward(begin, end)
        assert plan.kernel_profile()["reduce"][1] == end - begin
    assert grouped[0] == single[0] and grouped[1] == single[1] and np.array_equal(grouped[2], single[2])
