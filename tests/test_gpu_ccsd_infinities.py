"""CCSD terms 29-31 with an infinite T1 amplitude: only the elements that meet it
are infinite, with the sign that every term of them has, and none is NaN.  Inputs of
one sign make it so: X < 0 and P, Q > 0 as soon as O1 > 0, all three entering as
negative terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nu", [(1, 8), (3, 17), (5, 24), (9, 33), (17, 20), (30, 24), (33, 12)])
def test_infinite_amplitude_stays_where_it_belongs(no, nu):
    from libcc_b200 import api as A
    rng = np.random.default_rng(no)
    i0, x0 = no // 2, nu // 3
    o1 = rng.uniform(0.1, 1.0, (nu, no))  # [x][i]
    o1[x0, i0] = np.inf
    n4 = no * nu * nu * no
    t2, vl, vr = rng.uniform(0.1, 1.0, n4), rng.uniform(0.1, 1.0, n4), rng.uniform(0.1, 1.0, n4)
    vvvo = -rng.uniform(0.1, 1.0, nu * (nu + 1) // 2 * nu * no)
    got = A.ccsd_terms_29_31(no, nu, o1.ravel(), t2, vl, vr, vvvo).reshape(no, nu, nu, no)  # [j][z][y][i]
    want = np.zeros(got.shape, dtype=bool)
    want[:, :, :, i0] = True  # O1(i0, .) in X, P and Q
    want[:, x0, :, :] = True  # O1(k = i0, z = x0) P
    want[:, :, x0, :] = True  # O1(k = i0, y = x0) Q
    assert np.array_equal(got == -np.inf, want)
    assert np.isfinite(got[~want]).all()
