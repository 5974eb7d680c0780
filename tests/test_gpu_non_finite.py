'''Blocks with a NaN: no factorisation drops it and none reads past its block.  A split raises, as
at::linalg_svd does on the host (the reference's own call).'''
import numpy as np
import pytest
import torch

import tentorch_gb300 as tg

pytestmark = pytest.mark.gpu


def _tensor(blocks, dtype):
    cat = tg.su2
    legs = [tg.Leg(cat, [(i,) for i in range(len(blocks))], [b.shape[at] for b in blocks]) for at in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = dtype, device = 'cuda')
    for i, b in enumerate(blocks):
        t.block((i,), (i,)).copy_(torch.from_numpy(b).to(dtype))
    return t


@pytest.mark.parametrize('columns', [1, 2, 31, 40])
@pytest.mark.parametrize('wide', [False, True])
@pytest.mark.parametrize('where', [[(0, 0)], [(-1, -1)], [(1, 0), (0, -1)]])
def test_a_split_of_a_nan_raises(where, wide, columns):
    rng = np.random.default_rng(columns)
    clean = [rng.standard_normal((columns + 3, columns)), rng.standard_normal((5, 4))]
    bad = clean[0].copy()
    for at in where:
        bad[at] = np.nan
    if wide:
        clean[0], bad = clean[0].T.copy(), bad.T.copy()
    with pytest.raises(torch.linalg.LinAlgError):
        tg.svd(_tensor([bad, clean[1]], torch.float64), None, 0.0)
    # the next split of the same space is sound (16 n eps a value, n the longer side)
    _, values, _ = tg.svd(_tensor(clean, torch.float64), None, 0.0)
    want = np.concatenate([np.linalg.svd(b, compute_uv = False) for b in clean])
    assert np.abs(values.cpu().numpy() - want).max() <= 16 * (columns + 3) * 2.0 ** -52 * want.max()


@pytest.mark.parametrize('columns', [2, 3, 24])
@pytest.mark.parametrize('where', [[(0, 0)], [(1, 0)], [(-1, -1)], [(1, 0), (0, -1)]])
def test_a_complex_split_of_a_nan_raises(where, columns):
    '''Real numbers, so that a column's head has no imaginary part to reflect.'''
    bad = np.random.default_rng(columns).standard_normal((columns + 3, columns)) + 0j
    for at in where:
        bad[at] = np.nan
    for block in (bad, bad.T.copy()):
        with pytest.raises(torch.linalg.LinAlgError):
            tg.svd(_tensor([block], torch.complex128), None, 0.0)


@pytest.mark.parametrize('bad', [np.nan, np.inf])
@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('side', ['qr', 'rq'])
@pytest.mark.parametrize('shape', [(4, 3), (6, 9), (40, 33)])
def test_qr_keeps_what_is_not_finite(shape, side, dtype, bad):
    '''At any place of the block the factors are not finite, as LAPACK's are not; with nothing to reflect before it
    too (the columns of an identity).  The block beside it is factored as ever (8 n eps of its columns' sums).'''
    rng = np.random.default_rng(shape[0])
    beside = rng.standard_normal(shape)
    for start in (rng.standard_normal(shape), np.eye(*shape)):
        for at in [(0, 0), (1, 0), (shape[0] - 1, 0), (2, 2), (0, 1), (shape[0] - 1, shape[1] - 1)]:
            block = start.copy()
            block[at] = bad
            blocks = [block, beside] if side == 'qr' else [block.T.copy(), beside.T.copy()]
            first, second = getattr(tg, side)(_tensor(blocks, dtype))
            one, two = first.block((0,), (0,)), second.block((0,), (0,))
            assert not (torch.isfinite(one.abs()).all() and torch.isfinite(two.abs()).all()), at
            got = (first.block((1,), (1,)) @ second.block((1,), (1,))).cpu().numpy()
            assert np.abs(got - blocks[1]).max() <= 8 * max(shape) * 2.0 ** -52 * np.abs(beside).sum(0).max()
