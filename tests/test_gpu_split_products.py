'''Split-precision block products at the sizes where their kernels can go wrong: one block of m x k times
k x n around the tiles (128 rows, 32 and 64 columns), the groups of eight lines, the steps of 32 and the
exact chunks of 512 of K, with K shared by several CTAs; rows and columns scaled far apart, a zero row,
and results below the normal range.

The bound, per entry, with e the exponents above the row's and the column's largest entries and
u = 2^(e_row + e_col): each operand's S digits leave at most 2^(-7S-1) (1 + 2^-6) of its scale, the
products of digits past level S - 1 sum to at most (S - 1) 2^(-7S-2) (1 + 2^-6) a K, and the levels from 4
on (below 2^-25 K u together) are added in fp32: below 2^-48 K u.  The result is rounded to FP64 once.'''
import numpy as np
import pytest
import torch

import tentorch_gb300 as tg
from tentorch_gb300 import linalg as la

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (7, 9, 31), (8, 32, 32), (129, 65, 33), (128, 64, 512), (130, 33, 545), (40, 31, 1100)]


def _tensor(matrix):
    m, n = matrix.shape
    cat = tg.no_symmetry
    legs = [tg.Leg(cat, [(0,)], [x]) for x in (m, n)]
    out = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = torch.float64, device = 'cuda')
    out.block((0,), (0,)).copy_(torch.from_numpy(matrix))
    return out


def _exponents(largest):
    return np.where(largest > 0, np.frexp(largest)[1], 0)


@pytest.mark.parametrize('slices', [1, 3, 6, 8])
@pytest.mark.parametrize('size', SIZES)
def test_one_block_within_its_bound(size, slices):
    m, n, k = size
    rng = np.random.default_rng(m * 1000 + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a *= 2.0 ** rng.integers(-40, 40, m)[:, None]
    b *= 2.0 ** rng.integers(-40, 40, n)[None, :]
    if m > 2:
        a[1] = 0.0
        a[2] *= 2.0 ** -990  # its products with the smaller columns lie below the normal range
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    scale = np.ldexp(np.longdouble(1), _exponents(np.abs(a).max(1))[:, None] + _exponents(np.abs(b).max(0))[None, :])
    bound = k * scale * (2.0 ** (-7 * slices) * (1.02 + 0.26 * (slices - 1)) + 2.0 ** -48) + 2.0 ** -52 * np.abs(want) + 2.0 ** -1074
    ta, tb = _tensor(a), _tensor(b)
    with tg.precision(slices):
        plan = la.contract_plan(ta._space, tb._space, [1], [0])
        try:
            for forms in (0, la.FORM_NO_TENSOR_CORES):
                la.store_forms(plan, forms)
                for _ in range(2):
                    got = tg.contract(ta, tb, [1], [0]).block((0,), (0,)).cpu().numpy()
                    worst = np.abs(got.astype(np.longdouble) - want) / bound
                    assert worst.max() <= 1, (forms, float(worst.max()))
        finally:
            la.clear_tuning()


def _digits(x, axis, slices):
    '''The first digits of x over the power of two above its lines' largest entries: each prefix is x at that place
    rounded to nearest, halves up (the rest after it is exact in FP64).'''
    e = _exponents(np.abs(x).max(axis, keepdims = True))
    rest, digits = np.ldexp(x, -e), []
    for t in range(slices):
        digits.append(np.floor(np.ldexp(rest, 7 * (t + 1)) + 0.5))
        rest = rest - np.ldexp(digits[-1], -7 * (t + 1))
    return digits, e


@pytest.mark.parametrize('slices', [1, 2, 3, 4])
@pytest.mark.parametrize('size', [(9, 10, 33), (130, 70, 600)])
def test_the_digits_are_the_nearest_at_every_place(size, slices):
    '''Up to four slices every sum is an integer below 2^53, so the product is that of the digits to the last bit;
    half the entries have 30 bits, so that many lie half way between two digits.'''
    m, n, k = size
    rng = np.random.default_rng(slices)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[:, ::2], b[::2] = (np.ldexp(np.rint(np.ldexp(x, 27)), -27) for x in (a[:, ::2], b[::2]))
    (da, ea), (db, eb) = _digits(a, 1, slices), _digits(b, 0, slices)
    want = np.ldexp(sum(np.ldexp(da[t] @ db[u], -7 * (t + u + 2)) for t in range(slices) for u in range(slices - t)), ea + eb)
    with tg.precision(slices):
        got = tg.contract(_tensor(a), _tensor(b), [1], [0]).block((0,), (0,)).cpu().numpy()
    assert np.array_equal(got, want)


@pytest.mark.parametrize('slices', [1, 3, 6, 8])
def test_lines_below_the_normal_range(slices):
    '''Rows (and columns) whose largest entry is subnormal or just above, against factors that bring the products
    back: the bound of one block.'''
    rng = np.random.default_rng(slices)
    m, n, k = 12, 10, 33
    small, large = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    small *= 2.0 ** -np.arange(1012, 1060, 4)[:, None]
    small[:, 5] = 0.0
    large *= 2.0 ** 600
    for a, b in ((small, large), (large.T.copy(), small.T.copy())):
        want = a.astype(np.longdouble) @ b.astype(np.longdouble)
        scale = np.ldexp(np.longdouble(1), _exponents(np.abs(a).max(1))[:, None] + _exponents(np.abs(b).max(0))[None, :])
        bound = k * scale * (2.0 ** (-7 * slices) * (1.02 + 0.26 * (slices - 1)) + 2.0 ** -48) + 2.0 ** -52 * np.abs(want)
        with tg.precision(slices):
            got = tg.contract(_tensor(a), _tensor(b), [1], [0]).block((0,), (0,)).cpu().numpy()
        assert (np.abs(got.astype(np.longdouble) - want) / bound).max() <= 1


def test_a_lost_part_of_a_tile_shows_and_leaves_no_trace():
    '''A part of K whose wait gave up marks its tile's ticket.  The mark is set here by hand, as one of several parts'
    would be: that tile's entries become NaN and no others, the tickets are zero afterwards, and the next product
    is right.'''
    rng = np.random.default_rng(6)
    ta, tb = _tensor(rng.standard_normal((100, 4000))), _tensor(rng.standard_normal((4000, 70)))
    with tg.precision(6):
        want = tg.contract(ta, tb, [1], [0]).block((0,), (0,)).clone()
        (pool,) = (p for key, p in la._pools.items() if key[1] == torch.cuda.current_stream().cuda_stream and key[2] == torch.float64)
        tickets = pool.view(torch.int32)[:16384]
        assert int(tickets.count_nonzero()) == 0
        tickets[1] = 1 << 16  # the second of the three tiles of 32 columns
        lost = tg.contract(ta, tb, [1], [0]).block((0,), (0,))
        assert int(tickets.count_nonzero()) == 0
        assert torch.isnan(lost[:, 32:64]).all()
        assert torch.equal(lost[:, :32], want[:, :32]) and torch.equal(lost[:, 64:], want[:, 64:])
        assert torch.equal(tg.contract(ta, tb, [1], [0]).block((0,), (0,)), want)


@pytest.mark.parametrize('slices', [1, 6, 7, 8])
@pytest.mark.parametrize('size', [(8, 20001, 3), (20001, 8, 3), (33, 11000, 32), (2100, 2100, 5), (8, 20001, 33)])
def test_products_of_one_step_of_K(size, slices):
    '''Many tiles of one step of K, on either kernel by their shape: the bound of one block.'''
    test_one_block_within_its_bound(size, slices)
