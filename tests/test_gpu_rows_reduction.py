"""The reduction on X kept in rows (a forward that keeps W) against the one on X in
blocks: the same X and the same arithmetic in the same order, so the same bits,
at nu around the 8-wide blocks and the W build's column tiles, several
block triples a CTA and one."""
import numpy as np
import pytest

from libcc_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nu", [(2, 1), (2, 7), (3, 8), (3, 9), (3, 33), (2, 64), (4, 65), (3, 121), (2, 200)])
def test_rows_and_blocks_give_the_same_bits(no, nu):
    from libcc_b200 import api as A
    inp = S.generate(no, nu, 31)
    out = []
    for keep in (False, True):
        with A.TriplesPlan(no, nu, keep_w=keep) as p:
            p.set_system(inp)
            out.append(p.forward())
            assert (p.kept_tuples == p.num_tuples) == keep
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
