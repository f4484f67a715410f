"""The emulated W build at the ends of the exponent range.  Its digits depend on
the inputs' mantissas alone, so inputs scaled by 2^s give W scaled by 2^2s: every
bit while the X values are normal.  Below that each of the (at most four) X
values a W sums is rounded to the subnormal grid of 2^-1074, and a sum that meets
such a value may round differently by an ulp: a tolerance of 16 (2^-1074 + 2^-53
max |W|) covers four X values and three additions on either side."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("digits", [3, 5, 6, 7])
@pytest.mark.parametrize("no,nu", [(3, 9), (3, 20), (4, 72)])
def test_w_scales_with_the_inputs(no, nu, digits):
    from libcc_b200 import api as A
    inp = S.generate(no, nu, 11)

    def w_of(scale, tuple_index):
        with A.TriplesPlan.for_form(no, nu, f"int8:{digits}") as p:
            p.set_inputs(inp.eh, inp.ep, inp.t1, np.ldexp(inp.t2, scale), np.ldexp(inp.vm, scale), inp.voe,
                         np.ldexp(inp.vvvo, scale))
            return p.tuple_w(tuple_index)

    for t in (0, no * (no - 1) * (no - 2) // 6):  # an (i,j,k) and an (i,j,j) tuple
        base = w_of(0, t)
        assert np.abs(base).max() > 0.0
        for scale in (-450, 400):
            assert np.array_equal(w_of(scale, t), np.ldexp(base, 2 * scale)), scale
        for scale in (-500, -508, -511, -514):
            got, want = w_of(scale, t), np.ldexp(base, 2 * scale)
            assert np.abs(got - want).max() <= 16 * (2.0 ** -1074 + 2.0 ** -53 * np.abs(want).max()), scale
