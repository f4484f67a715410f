"""An emulated batch with inputs that its plans refuse."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["nan", "denominator"])
def test_rejected_inputs_are_rejected_again_and_can_be_replaced(bad):
    """A system whose inputs an emulated plan refuses has no digit operands: every
    forward answers with the plan's own error (the second one must not run
    the system on operands that were never built), and new inputs for that
    system alone make the batch whole again."""
    from libcc_b200 import _native as N
    from libcc_b200 import api as A
    from libcc_b200 import batch as B
    shapes = [(3, 24), (4, 17), (3, 9)]
    good = [S.generate(no, nu, 40 + k) for k, (no, nu) in enumerate(shapes)]
    arrays = [np.array(a) for a in good[1].arrays()]
    if bad == "nan":
        arrays[3][5] = np.nan
    else:
        arrays[1][0] = -10.0  # a virtual energy below every occupied one
    with A.TriplesPlan.for_form(4, 17, "int8") as p, pytest.raises(N.CctError) as refused:
        p.set_inputs(*arrays)
    with B.TriplesBatch(shapes, form="int8") as b:
        for k in (0, 2):
            b.set_system(k, good[k])
        b.set_inputs(1, *arrays)
        for _ in range(2):
            with pytest.raises(N.CctError) as e:
                b.forward()
            assert e.value.status == refused.value.status
            with pytest.raises(N.CctError):
                b.emu_digits(1)
        b.set_system(1, good[1])
        ets, etd = b.forward()
        for k, inp in enumerate(good):
            with A.TriplesPlan.for_form(inp.no, inp.nu, "int8") as p:
                p.set_system(inp)
                assert (ets[k], etd[k]) == p.forward()[:2], k
