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
