'''The two-site matvec's one launch at the sizes where its tiles change (8 x 8 to 32 x 32, a tile's K whole
or cut), against the oracle.

Bound: an entry is a sum of k1 products of sums of k2, each of at most 6 chi terms (5 operator states and a
physical one); n additions of independent terms of size s err by at most n 2^-53 of their absolute sum, which
is at most sqrt(n) times the largest entry s sqrt(n): (6 chi)^1.5 2^-53 of the largest entry.'''
import pytest

import tentorch_gb300 as tg
from tentorch_gb300 import linalg as la
from convert import max_relative, to_product
from oracle import engine as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('chi', [17, 32, 47, 64, 97, 129, 190, 215, 250])
def test_matvec_tiles_match_the_oracle(chi):
    head, tail, theta = orc.matvec_inputs(chi, seed = chi)
    want = orc.einsum(orc.MATVEC, head, tail, theta).blocks
    h, t, v = (to_product(x, tg.u1) for x in (head, tail, theta))
    assert la.plan_of(orc.MATVEC, h, t, v).describe().startswith('chain ops')
    for _ in range(2):
        assert max_relative(tg.einsum(orc.MATVEC, h, t, v), want) < (6 * chi) ** 1.5 * 2.0 ** -53
