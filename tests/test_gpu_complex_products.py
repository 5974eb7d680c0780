'''complex128 block products on both sizes of tile: few and many tiles, ragged at the edges of 16 and 32, K of one step,
of one and of several, one block and several pairs.

A complex dot product of length K is off by at most 2 (K + 2) eps of the sum of its terms' magnitudes.'''
import numpy as np
import pytest
import torch

import tentorch_gb300 as tg

pytestmark = pytest.mark.gpu


def _tensor(blocks, cat, charges):
    rows, cols = ([b.shape[at] for b in blocks] for at in (0, 1))
    t = tg.Tensor(cat, [tg.Leg(cat, charges, rows)], [tg.Leg(cat, charges, cols)], cat.trivial(), dtype = torch.complex128, device = 'cuda')
    for q, b in zip(charges, blocks):
        t.block(q, q).copy_(torch.from_numpy(b))
    return t


@pytest.mark.parametrize('sizes', [[(5, 7, 3)], [(100, 130, 40)], [(801, 799, 17)], [(9801, 33, 1)], [(33, 9801, 12)], [(1100, 1090, 33)],
                                   [(600, 610, 9), (17, 31, 2), (400, 33, 12)]])
def test_products_within_their_bound(sizes):
    rng = np.random.default_rng(sizes[0][0])
    charges = [(2 * q,) for q in range(len(sizes))]
    draw = lambda m, n: rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    a, b = [draw(m, k) for m, _, k in sizes], [draw(k, n) for _, n, k in sizes]
    got = tg.contract(_tensor(a, tg.u1, charges), _tensor(b, tg.u1, charges), [1], [0])
    for q, x, y, (_, _, k) in zip(charges, a, b, sizes):
        bound = 2 * (k + 2) * 2.0 ** -52 * (np.abs(x) @ np.abs(y))
        assert (np.abs(got.block(q, q).cpu().numpy() - x @ y) <= bound).all()
