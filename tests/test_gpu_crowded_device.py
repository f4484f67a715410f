"""Plans on a device that is almost full: the X ring of tuple groups takes a small
part of what is left, so that the backward's buffers and other plans still find
the room they had without groups, with the same results."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture
def crowd():
    """Takes device memory until `left` bytes are free."""
    torch = pytest.importorskip("torch")
    held = []

    def take(left):
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        if free > left:
            held.append(torch.empty(free - left, dtype=torch.uint8, device="cuda"))
        return torch.cuda.mem_get_info()[0]

    yield take
    held.clear()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("form", ["fp64", "int8:5"])
def test_forward_and_backward_fit_where_single_tuples_do(crowd, form):
    """no12-nu120: some 0.5 GB a plan with single-tuple X buffers (0.7 emulated) and
    0.7 GB of backward buffers; a ring of whole groups alone is 2.3 GB."""
    from libcc_b200 import api as A
    no, nu = 12, 120
    inp = S.generate(no, nu, 4)
    with A.TriplesPlan.for_form(no, nu, form) as p:
        p.set_system(inp)
        want = p.forward()
        grads = p.backward()
    free = crowd(1900 << 20)
    assert free < 2000 << 20
    with A.TriplesPlan.for_form(no, nu, form) as p:
        p.set_system(inp)
        got = p.forward()
        assert got[:2] == want[:2] and np.array_equal(got[2], want[2])
        again = p.backward()
        for k in grads:
            assert np.array_equal(again[k], grads[k]), k


def test_groups_leave_room_for_other_plans(crowd):
    import torch
    from libcc_b200 import api as A
    free = crowd(4 << 30)
    plans = []
    for _ in range(4):
        plans.append(A.TriplesPlan(12, 120, vvvo="expanded"))
    used = free - torch.cuda.mem_get_info()[0]
    for p in plans:
        p.close()
    # four plans with three single-tuple X sets (0.5 GB each), and at most 1/32 of what is free each
    assert used <= 4 * ((500 << 20) + free // 32)
