'''The engine's batched SVD where its phases change: one column, the smallest preconditioned blocks, the
padding of the column blocks (8), the cluster's thresholds (16, 128 columns), the longest columns of the
blocked FP32 sweeps (320), tall and wide; spectra over twelve decades, without structure, and rank
deficient, several blocks in one launch.

Bounds, with n the longer side and eps = 2^-52: Jacobi's method and the products around it are backward
stable with errors of a few eps sqrt(n) a column; 8 n eps, relative to the largest singular value, for
the values and the product of the factors, and for the orthonormality of the vectors of nonzero values.'''
import numpy as np
import pytest
import torch

import tentorch_gb300 as tg

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _graded(rng, m, n):
    k = min(m, n)
    u, v = (np.linalg.qr(rng.standard_normal((x, k)))[0] for x in (m, n))
    return (u * 10.0 ** (-12 * np.arange(k) / k)) @ v.T


def _deficient(rng, m, n):
    r = max(1, min(m, n) // 3)
    return rng.standard_normal((m, r)) @ rng.standard_normal((r, n))


SPECTRA = {'graded': _graded, 'unstructured': lambda rng, m, n: rng.standard_normal((m, n)), 'deficient': _deficient}


@pytest.mark.parametrize('spectrum', SPECTRA)
@pytest.mark.parametrize('sizes', [[(1, 1), (1, 5), (2, 2), (9, 2)], [(15, 15), (16, 40), (7, 7)], [(17, 16), (31, 33), (8, 9)],
                                   [(127, 70), (97, 96)], [(128, 128), (33, 200), (16, 16)], [(321, 40), (161, 161)], [(330, 325)]])
def test_factors_within_their_bounds(sizes, spectrum):
    rng = np.random.default_rng(len(sizes) * 1000 + sizes[0][0])
    blocks = [SPECTRA[spectrum](rng, m, n) for m, n in sizes]
    cat = tg.su2  # its sectors are their own duals: the split keeps each block's values
    legs = [tg.Leg(cat, [(i,) for i in range(len(sizes))], [s[side] for s in sizes]) for side in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = torch.float64, device = 'cuda')
    for i, b in enumerate(blocks):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    first, values, second = tg.svd(t, None, 1e-13)
    bond = first.domain[0]
    at = 0
    kept = dict(zip(bond.sectors, bond.multiplicities))
    for i, b in enumerate(blocks):
        n = max(b.shape)
        count = kept.get((i,), 0)
        u, v = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
        s = values[at:at + count].cpu().numpy()
        at += count
        want = np.linalg.svd(b, compute_uv = False)
        scale, tol = want[0], 8 * n * EPS
        assert np.abs(s - want[:count]).max() <= tol * scale
        assert want[count:].max(initial = 0.0) <= 1e-13 + tol * scale
        for q in (u.T @ u, v @ v.T):
            assert np.abs(q - np.eye(count)).max() <= tol
        assert np.abs((u * s) @ v - b).max() <= tol * scale + 1e-13 * n


def test_the_pads_after_odd_blocks_are_zero():
    '''The factors are written into uninitialised memory when they cover their arenas: the alignment pads after
    blocks of odd size, which arena-wide sums read, have to be written too.'''
    rng = np.random.default_rng(3)
    cat = tg.su2
    sizes = [(3, 5), (7, 7), (5, 9)]
    legs = [tg.Leg(cat, [(i,) for i in range(3)], [s[side] for s in sizes]) for side in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = torch.float64, device = 'cuda')
    for i, (m, n) in enumerate(sizes):
        t.block((i,), (i,)).copy_(torch.from_numpy(rng.standard_normal((m, n))))
    for n in (64, 128, 256, 512, 1024):  # freed memory of the sizes the factors take, full of NaN
        filled = [torch.full((n,), float('nan'), dtype = torch.float64, device = 'cuda') for _ in range(8)]
        del filled
    for factor in (tg.svd(t, None, 0.0)[0], tg.svd(t, None, 0.0)[2]):
        blocks = sum(float(b.square().sum()) for b in factor.to_tuple()[3].values())
        assert abs(float(factor.data.square().sum()) - blocks) <= 1e-12 * blocks


def _complex(make):
    def block(rng, m, n):
        re, im = (make(rng, m, n) for _ in range(2))
        return re + 1j * im
    return block


def _complex_graded(rng, m, n):
    k = min(m, n)
    u, v = (np.linalg.qr(rng.standard_normal((x, k)) + 1j * rng.standard_normal((x, k)))[0] for x in (m, n))
    return (u * 10.0 ** (-12 * np.arange(k) / k)) @ v.conj().T


COMPLEX_SPECTRA = {'graded': _complex_graded, 'unstructured': _complex(SPECTRA['unstructured']),
                   'deficient': lambda rng, m, n: _complex_graded(rng, m, max(1, min(m, n) // 3)) @ _complex_graded(rng, max(1, min(m, n) // 3), n),
                   'equal': lambda rng, m, n: 1e-40 * np.linalg.qr(rng.standard_normal((max(m, n),) * 2) + 1j)[0][:m, :n]}


@pytest.mark.parametrize('spectrum', COMPLEX_SPECTRA)
@pytest.mark.parametrize('sizes', [[(1, 1), (1, 5), (2, 2), (9, 2)], [(15, 15), (16, 40), (24, 24)], [(32, 33), (31, 7)], [(33, 64), (8, 9), (64, 65)],
                                   [(97, 96), (65, 70)], [(128, 129)], [(300, 20), (20, 160), (160, 161)]])
def test_complex_factors_within_their_bounds(sizes, spectrum):
    '''The complex128 kernels: one CTA up to 32 columns, clusters of 8 and (from 96) of 16, one to five registers a
    lane and column, the most columns (160); 'equal' a spectrum of ones at a scale whose squares vanish in FP32.
    A complex multiply-add's error is at most sqrt(8) times a real one's: 24 n eps.'''
    rng = np.random.default_rng(len(sizes) * 1000 + sizes[0][0])
    blocks = [COMPLEX_SPECTRA[spectrum](rng, m, n) for m, n in sizes]
    cat = tg.su2
    legs = [tg.Leg(cat, [(i,) for i in range(len(sizes))], [s[side] for s in sizes]) for side in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = torch.complex128, device = 'cuda')
    for i, b in enumerate(blocks):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    cut = 1e-13 * max(np.abs(b).max() for b in blocks)
    first, values, second = tg.svd(t, None, cut)
    bond = first.domain[0]
    at = 0
    kept = dict(zip(bond.sectors, bond.multiplicities))
    for i, b in enumerate(blocks):
        n = max(b.shape)
        count = kept.get((i,), 0)
        u, v = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
        s = values[at:at + count].cpu().numpy()
        at += count
        want = np.linalg.svd(b, compute_uv = False)
        scale, tol = want[0], 24 * n * EPS
        assert np.abs(s - want[:count]).max(initial = 0.0) <= tol * scale
        assert want[count:].max(initial = 0.0) <= cut + tol * scale
        for q in (u.conj().T @ u, v @ v.conj().T):
            assert np.abs(q - np.eye(count)).max(initial = 0.0) <= tol
        assert np.abs((u * s) @ v - b).max() <= tol * scale + cut * n


@pytest.mark.parametrize('scale', [-1020, -700, -200, 200, 500, 1000])
@pytest.mark.parametrize('spectrum', SPECTRA)
def test_blocks_far_from_one(spectrum, scale):
    '''Blocks whose squares under- or overflow, with 2, 9, 31, 40 and 1 columns, tall and wide: the same bounds (a
    power of two takes them to the scale of the other tests; below the normal range half a unit, 2^-1075, more).'''
    rng = np.random.default_rng(abs(scale))
    blocks = [SPECTRA[spectrum](rng, m, n) for m, n in [(5, 2), (9, 12), (31, 33), (50, 40), (6, 1)]]
    scaled = [np.ldexp(b, scale - int(np.frexp(np.abs(b).max())[1])) for b in blocks]
    blocks = [np.ldexp(b, -scale) for b in scaled]  # what the kernel is given, near one
    cat = tg.su2
    legs = [tg.Leg(cat, [(i,) for i in range(len(blocks))], [b.shape[at] for b in blocks]) for at in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = torch.float64, device = 'cuda')
    for i, b in enumerate(scaled):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    first, values, second = tg.svd(t, None, float(np.ldexp(1e-13, scale)))
    bond = first.domain[0]
    kept, at = dict(zip(bond.sectors, bond.multiplicities)), 0
    for i, b in enumerate(blocks):
        n = max(b.shape)
        count = kept.get((i,), 0)
        u, v = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
        s = np.ldexp(values[at:at + count].cpu().numpy(), -scale)
        at += count
        want = np.linalg.svd(b, compute_uv = False)
        tol, flat = 8 * n * EPS * want[0], float(np.ldexp(1.0, -1075 - scale)) if scale < 0 else 0.0
        assert np.abs(s - want[:count]).max() <= tol + flat
        assert want[count:].max(initial = 0.0) <= 1e-13 + tol + flat
        for q in (u.T @ u, v @ v.T):
            assert np.abs(q - np.eye(count)).max() <= 8 * n * EPS
        assert np.abs((u * s) @ v - b).max() <= tol + 1e-13 * n + flat * n


@pytest.mark.parametrize('small', [1e-30, 1e-76, 1e-80, 1e-90, 1e-120, 1e-127, 1e-150, 1e-200])
@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('sizes', [(3, 2), (10, 12), (20, 30)])
def test_values_far_below_the_largest(sizes, dtype, small):
    '''Two blocks on a diagonal, the second `small` times the first: the squares of its columns' products vanish, and
    its vectors are orthonormal to the same bounds (below 1e-128 the block is at::linalg_svd's).'''
    rng = np.random.default_rng(sizes[0])
    p, q = sizes
    b = np.zeros((p + q, p + q), dtype = np.complex128 if dtype.is_complex else np.float64)
    for part, n, scale in ((slice(0, p), p, 1.0), (slice(p, p + q), q, small)):
        b[part, part] = scale * (rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if dtype.is_complex else 0))
    cat = tg.no_symmetry
    leg = tg.Leg(cat, [(0,)], [p + q])
    t = tg.Tensor(cat, [leg], [leg], (0,), dtype = dtype, device = 'cuda')
    t.block((0,), (0,)).copy_(torch.from_numpy(b))
    first, values, second = tg.svd(t, None, 0.0)
    u, v = (f.block((0,), (0,)).cpu().numpy() for f in (first, second))
    s = values.cpu().numpy().real
    count, tol = len(s), (24 if dtype.is_complex else 8) * (p + q) * EPS
    assert count == p + q
    for x in (u.conj().T @ u, v @ v.conj().T):
        assert np.abs(x - np.eye(count)).max() <= tol
    want = np.linalg.svd(b[:p, :p], compute_uv = False)
    assert np.abs(s[:p] - want).max() <= tol * want[0]
    assert np.abs((u * s) @ v - b).max() <= tol * want[0]
    # Jacobi's method on the sorted, factored columns keeps the second block's values to its own scale
    if small >= 1e-120:
        want = np.linalg.svd(b[p:, p:] / small, compute_uv = False)
        assert np.abs(s[p:] / small - want).max() <= tol * want[0]


@pytest.mark.parametrize('spectrum', SPECTRA)
@pytest.mark.parametrize('sizes', [[(600, 20), (601, 20)], [(9, 700), (1300, 33)], [(3200, 64), (26500, 5)]])
def test_long_columns(sizes, spectrum):
    '''Columns whose reflectors one warp makes ahead (to 600 entries) and whose CTA makes them, in shared memory or (3200
    x 64) in global memory, and one too long to be staged there (26500): the bounds of the other sizes.'''
    test_factors_within_their_bounds(sizes, spectrum)


@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
@pytest.mark.parametrize('sizes', [[(2, 2), (1, 3)], [(16, 31), (24, 24)], [(64, 65), (100, 90)]])
def test_zero_values_need_no_second_factorisation(sizes, dtype):
    '''Blocks of zeros but for a corner, and zero blocks: the kernels' own factors, none handed on, with the bounds of
    the other sizes; a tolerance below zero keeps the zeros, with orthonormal vectors in complex128 as at::linalg_svd
    gives them.'''
    rng = np.random.default_rng(sizes[0][0])
    blocks, cat = [], tg.su2
    for m, n in sizes:
        b = np.zeros((m, n), dtype = np.complex128 if dtype.is_complex else np.float64)
        h = min(m, n) // 2
        b[:h, :h] = rng.standard_normal((h, h)) + (1j * rng.standard_normal((h, h)) if dtype.is_complex else 0)
        blocks.append(b)
    legs = [tg.Leg(cat, [(i,) for i in range(len(sizes))], [s[side] for s in sizes]) for side in (0, 1)]
    t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = dtype, device = 'cuda')
    for i, b in enumerate(blocks):
        t.block((i,), (i,)).copy_(torch.from_numpy(b))
    before = tg.linalg.svd_fallbacks
    for tol in (0.0, -1.0) if dtype.is_complex else (0.0,):
        first, values, second = tg.svd(t, None, tol)
        kept = dict(zip(first.domain[0].sectors, first.domain[0].multiplicities))
        at = 0
        for i, b in enumerate(blocks):
            count, bound = kept.get((i,), 0), (24 if dtype.is_complex else 8) * max(b.shape) * EPS
            want = np.linalg.svd(b, compute_uv = False)
            assert count == (min(b.shape) if tol < 0 else min(b.shape) // 2)
            if count == 0:
                continue
            u, v = first.block((i,), (i,)).cpu().numpy(), second.block((i,), (i,)).cpu().numpy()
            s = values[at:at + count].cpu().numpy().real
            at += count
            scale = max(want[0], 1e-300)
            assert np.abs(s - want[:count]).max() <= bound * scale
            for q in (u.conj().T @ u, v @ v.conj().T):
                assert np.abs(q - np.eye(count)).max() <= bound
            assert np.abs((u * s) @ v - b).max() <= bound * scale
        if tol >= 0:
            assert tg.linalg.svd_fallbacks == before
