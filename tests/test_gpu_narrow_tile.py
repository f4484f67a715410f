"""The emulated W build where the last column tile is narrow (16 or 32 columns
of what is left of nu), just not narrow, or the only one: against the oracle,
at the bars of test_gpu_emulated.py."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nu", [(2, 9), (2, 17), (2, 33), (3, 65), (3, 80), (3, 96), (2, 97), (2, 129)])
def test_last_column_tile_matches_oracle(no, nu):
    from libcc_b200 import api
    from oracle import oracle as O
    inp = S.generate(no, nu, 21, "normal")
    with api.TriplesPlan.for_form(no, nu, "int8:7") as plan:
        plan.set_system(inp)
        w = plan.tuple_w(0)
        ets, etd, v1 = plan.forward()
    kind, i, j, k = O.all_tuples(no)[0]
    ref = O.c_tuple_w(inp, kind, i, j, k).ravel(order="F")
    assert np.abs(w - ref).max() <= 1e-12 * np.abs(ref).max()
    ets_o, etd_o, v1_o = O.c_cc_triples(inp)
    assert abs(etd - etd_o) <= 1e-11 * abs(etd_o)
    assert np.abs(v1 - v1_o.ravel(order="F")).max() <= 1e-9 * np.abs(v1_o).max()


def test_rebuilt_operands_of_a_wider_tile():
    """An automatic plan padded to 64s that runs few digits on 80-column tiles."""
    from libcc_b200 import api
    inp = S.generate(2, 260, 22, "normal")
    with api.TriplesPlan(2, 260) as ref, api.TriplesPlan.for_form(2, 260, "int8@2.1e-7") as emu:
        ref.set_system(inp)
        emu.set_system(inp)
        d = emu.emu_digits()
        a, b = ref.forward(), emu.forward()
    assert d["digits"] <= 6
    assert abs((a[0] + a[1]) - (b[0] + b[1])) <= d["target"]
