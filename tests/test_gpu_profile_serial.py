"""Profiled launches run one after the other: their times are disjoint intervals of
the forward, so they add up to no more than its time."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,no,nu,end", [("fp64", 4, 320, 8), ("fp64", 6, 96, 40), ("int8:3", 6, 96, 40)])
def test_profiled_launches_do_not_overlap(form, no, nu, end):
    torch = pytest.importorskip("torch")
    from libcc_b200 import api as A
    gen = torch.Generator(device="cuda").manual_seed(1)
    arrays = {k: torch.empty(n, dtype=torch.float64, device="cuda").normal_(0.0, 0.05, generator=gen)
              for k, n in A.input_sizes(no, nu).items()}
    arrays["eh"] = torch.linspace(-1.4, -0.4, no, dtype=torch.float64, device="cuda")
    arrays["ep"] = torch.linspace(0.1, 4.0, nu, dtype=torch.float64, device="cuda")
    with A.TriplesPlan.for_form(no, nu, form) as p:
        p.set_inputs(**arrays)
        want = p.forward(0, end)
        p.set_profiling(True)
        for _ in range(3):
            got = p.forward(0, end)
            prof = p.kernel_profile()
            assert prof["wbuild"][1] == prof["reduce"][1] == end
            assert prof["wbuild"][0] + prof["reduce"][0] <= p.last_forward_ms
        p.set_profiling(False)
        again = p.forward(0, end)
        assert got[:2] == want[:2] == again[:2]
