'''The batched QR and RQ where its kernel changes: one row or column, tall and wide blocks, the cluster's
thresholds (16 and 96 columns), odd sizes (blocks followed by a pad), several blocks in one launch, and
columns that are already zero below the diagonal, in float64 and complex128, scaled far from one.

Against LAPACK (numpy) with its signs: Householder QR is columnwise backward stable, so Q R reproduces the
block, Q^H Q the identity, to 8 max(m, n) eps, and R lies within 8 max(m, n) eps times the condition of the
leading columns (below 100 n for these random blocks) of LAPACK's.'''
import numpy as np
import pytest
import torch

import tentorch_gb300 as tg

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize('scale', [0, -600, 500])
@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('side', ['qr', 'rq'])
@pytest.mark.parametrize('sizes', [[(1, 1), (1, 7), (7, 1), (2, 2)], [(15, 15), (9, 20), (20, 9)], [(16, 16), (17, 40), (33, 17)],
                                   [(95, 96), (130, 97), (60, 200)]])
def test_factors_match_lapack(sizes, side, dtype, scale):
    rng = np.random.default_rng(len(sizes) * 1000 + sizes[0][0])
    blocks = []
    for m, n in sizes:
        b = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if dtype.is_complex else 0)
        if m > 3 and n > 3:
            b[1:, 0] = 0  # nothing to reflect
        blocks.append(b * 2.0 ** scale)
    cat = tg.su2
    legs = [tg.Leg(cat, [(i,) for i in range(len(sizes))], [s[at] for s in sizes]) for at in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = dtype, device = 'cuda')
    for i, b in enumerate(blocks):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    first, second = getattr(tg, side)(t)
    for i, b in enumerate(blocks):
        one, two = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
        q, r, want = (one, two, b) if side == 'qr' else (two.T, one.T, b.T)
        wq, wr = np.linalg.qr(want)
        n = max(b.shape)
        tol = 8 * n * EPS
        norm = np.abs(want / 2.0 ** scale).sum(0).max()
        assert np.abs(q.conj().T @ q - np.eye(q.shape[1])).max() <= tol
        assert np.abs((q @ (r / 2.0 ** scale)) - want / 2.0 ** scale).max() <= tol * norm
        assert np.abs((r - wr) / 2.0 ** scale).max() <= tol * 100 * n * norm
        assert np.abs(np.tril(r, -1)).max(initial = 0) == 0


@pytest.mark.parametrize('small', [1e-140, 1e-155, 1e-158, 1e-160, 1e-161, 1e-170, 1e-300])
@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('side', ['qr', 'rq'])
@pytest.mark.parametrize('columns', [[0], [1], [1, 2]])
def test_columns_far_below_the_largest(columns, side, dtype, small):
    '''Columns whose squares vanish: Q is orthonormal, and Q R reproduces each column to 8 max(m, n) eps of its own
    entries (columnwise backward stability), the block's largest entry near 1 and near 2^1000.'''
    rng = np.random.default_rng(columns[0] + 7)
    blocks = []
    for m, n in [(5, 3), (40, 33), (20, 50)]:
        b = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if dtype.is_complex else 0)
        b[:, columns] *= small
        blocks.append(b)
    blocks.append(blocks[1] * 2.0 ** 1000)
    given = [b if side == 'qr' else b.T.copy() for b in blocks]
    cat = tg.su2
    legs = [tg.Leg(cat, [(i,) for i in range(len(given))], [b.shape[at] for b in given]) for at in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = dtype, device = 'cuda')
    for i, b in enumerate(given):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    first, second = getattr(tg, side)(t)
    for i, b in enumerate(blocks):
        one, two = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
        q, r = (one, two) if side == 'qr' else (two.T, one.T)
        tol = 8 * max(b.shape) * EPS
        assert np.abs(q.conj().T @ q - np.eye(q.shape[1])).max() <= tol
        norms = np.abs(b).sum(0)  # each column over its norm: no product leaves the normal range
        assert (np.abs(q @ (r / norms) - b / norms).max(0) <= tol).all()


@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('side', ['qr', 'rq'])
@pytest.mark.parametrize('sizes,batched', [([(1300, 80)], False), ([(1000, 20)], False), ([(5, 20000)], None), ([(20, 5000)], True),
                                           ([(3, 1000), (15, 17), (1, 96)], True), ([(500, 60)] * 6, True)])
def test_long_and_wide_blocks(sizes, batched, side, dtype):
    '''Blocks that are faster in cuSOLVER go there, several side by side and wide ones (a cluster by their columns) do
    not; by either way the bounds of the other sizes, and R within them of LAPACK's.'''
    la = tg.linalg
    la.clear_plans()
    test_factors_match_lapack(sizes, side, dtype, 0)
    if batched is not None and side == 'qr':
        (plan,) = la._qr_plans.values()
        assert (plan is not None) == batched
