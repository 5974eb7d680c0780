'''
The work that a user of this framework has it do, as measured cases.

A two-site DMRG program contracts the effective Hamiltonian with a vector (`matvec`), runs the Krylov
loop of a window (`window`), splits the two-site tensor (`split`), moves the orthogonality centre
(`canonical`), advances an environment over a site (`environment`), and repeats all of it along the
chain (`sweep`); a program with many independent windows batches their matvecs (`batch`); one over
non-abelian charges contracts tensors whose legs have to be braided first (`recouple`).  Bonds run from
32 to about a thousand multiplets over 5 to 17 U(1) charges, the scalar type is float64 or the
package's default complex128, and block products are FP64 or split into bf16 slices, as the caller asks.

`exact` gives the same results from dense tensors (or, for the braided contraction, block by block) in
plain torch, with no code of this package: block sparsity is a gather from the dense result.
'''
import functools
import math
import random

import numpy as np
import torch
from torch.autograd.graph import increment_version

DEVICE = 'cuda'
MATVEC = 'EPaqj,JRSFb,AQsb->EPrf'
BRAIDED = 'ABcd,DCef->ABef'
ADVANCE_LEFT = 'EIa,Feq,aPb,IqPj->FJb'
ADVANCE_RIGHT = 'Gfq,aPb,IqPk,Gkb->FIa'
DTYPES = {'f64': torch.float64, 'c128': torch.complex128}
CUTOFF = 1e-14  # the singular values a DMRG run drops (its default svd_tol)


def listed():
    return [
        # one application of a small chain's effective Hamiltonian: launches and host work
        {'name': 'matvec_chi32', 'kind': 'matvec', 'chi': 32, 'charges': 9, 'dtype': 'f64', 'slices': 0},
        # the bond most runs settle at, with FP64 block products
        {'name': 'matvec_chi256', 'kind': 'matvec', 'chi': 256, 'charges': 17, 'dtype': 'f64', 'slices': 0},
        # the same in the split precision a DMRG run uses (six slices)
        {'name': 'matvec_chi256_s6', 'kind': 'matvec', 'chi': 256, 'charges': 17, 'dtype': 'f64', 'slices': 6},
        # the largest bonds, an odd size
        {'name': 'matvec_chi1001_s6', 'kind': 'matvec', 'chi': 1001, 'charges': 17, 'dtype': 'f64', 'slices': 6},
        # a window's whole Krylov loop
        {'name': 'window_chi256_s6', 'kind': 'window', 'chi': 256, 'charges': 17, 'dtype': 'f64', 'slices': 6, 'steps': 10},
        # an environment over one more site, in the default scalar type
        {'name': 'environment_chi203_c128', 'kind': 'environment', 'chi': 203, 'charges': 13, 'dtype': 'c128', 'slices': 0, 'side': 'left'},
        # the truncating split of the two-site tensor, once a window
        {'name': 'split_chi256', 'kind': 'split', 'chi': 256, 'charges': 17, 'dtype': 'f64', 'decades': 12},
        # the same in the default scalar type, at a small run's bond
        {'name': 'split_chi64_c128', 'kind': 'split', 'chi': 64, 'charges': 9, 'dtype': 'c128', 'decades': 8},
        # one step of the orthogonality centre (canonical form of a state)
        {'name': 'canonical_chi256', 'kind': 'canonical', 'chi': 256, 'charges': 17, 'dtype': 'f64', 'side': 'left'},
        # SU(2) tensors, spins 0 .. 4 with 8 multiplets each, braided and contracted in split precision
        {'name': 'recouple_su2_s6', 'kind': 'recouple', 'category': 'su2', 'top': 8, 'mult': 8, 'slices': 6},
        # independent windows of drawn bonds, applied in one call
        {'name': 'batch_64', 'kind': 'batch', 'windows': 64, 'pick': 0, 'slices': 0},
        # a sweep from a random state, every call of the driver in it
        {'name': 'sweep_L64_chi64', 'kind': 'sweep', 'length': 64, 'chi': 64, 'steps': 5, 'dtype': 'f64', 'slices': 0},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(('matvec', 'matvec', 'window', 'environment', 'split', 'canonical', 'recouple', 'batch', 'sweep'))
    dtype = rng.choice(('f64', 'f64', 'c128'))
    slices = rng.choice((0, 6, 6, 4, 8)) if dtype == 'f64' else 0  # slices apply to float64 products
    charges = rng.choice((5, 9, 13, 17))
    if kind in ('matvec', 'window'):
        chi = _spread(rng, 24, 1024 if slices else 512 if dtype == 'f64' else 256)
        case = {'kind': kind, 'chi': chi, 'charges': charges, 'dtype': dtype, 'slices': slices}
        return dict(case, steps = rng.choice((5, 8, 10))) if kind == 'window' else case
    if kind == 'environment':
        return {'kind': kind, 'chi': _spread(rng, 24, 512 if dtype == 'f64' else 256), 'charges': charges, 'dtype': dtype,
                'slices': slices, 'side': rng.choice(('left', 'right'))}
    if kind == 'split':
        return {'kind': kind, 'chi': _spread(rng, 24, 400 if dtype == 'f64' else 80), 'charges': charges, 'dtype': dtype,
                'decades': rng.choice((3, 8, 12))}
    if kind == 'canonical':
        return {'kind': kind, 'chi': _spread(rng, 24, 512 if dtype == 'f64' else 256), 'charges': charges, 'dtype': dtype,
                'side': rng.choice(('left', 'right'))}
    if kind == 'recouple':
        if dtype == 'c128':
            return {'kind': kind, 'category': 'fibonacci', 'top': 1, 'mult': _spread(rng, 4, 24), 'slices': 0}
        return {'kind': kind, 'category': 'su2', 'top': rng.randint(3, 8), 'mult': rng.randint(3, 8), 'slices': slices}
    if kind == 'batch':
        return {'kind': kind, 'windows': _spread(rng, 4, 64), 'pick': rng.randrange(1000), 'slices': slices}
    return {'kind': kind, 'length': rng.randint(6, 16), 'chi': _spread(rng, 8, 32), 'steps': rng.choice((3, 5)), 'dtype': dtype,
            'slices': slices}


# ---------------------------------------------------------------------------------------------
# legs and blocks in plain numbers: a leg is ((charge, multiplets), ...), charges ascending and the
# same multiplets at +q and -q; a block (r, r) has one row per codomain state of charge r, ordered by
# the legs' charges and then by their copies, the last leg fastest, and columns over the domain alike
# ---------------------------------------------------------------------------------------------

PHYSICAL = ((-1, 1), (1, 1))
OPERATOR = ((-2, 1), (0, 3), (2, 1))  # the Heisenberg automaton's bond


@functools.lru_cache(maxsize = None)
def bond(chi, charges, odd = False):
    '''chi multiplets (at least one a charge) over `charges` charges (one more when odd), Gaussian in the charge.'''
    top = charges // 2
    qs = [2 * q + 1 for q in range(-top - 1, top + 1)] if odd else [2 * q for q in range(-top, top + 1)]
    weight = [math.exp(-q * q / 32) for q in qs]
    count = [1 + int((max(chi, len(qs)) - len(qs)) * w / sum(weight)) for w in weight]
    left = max(chi, len(qs)) - sum(count)
    for at in range(len(qs) // 2 - 1, -1, -1):
        if left >= 2:
            count[at], count[-1 - at], left = count[at] + 1, count[-1 - at] + 1, left - 2
    if not odd:
        count[top] += left
    return tuple(zip(qs, count))


@functools.lru_cache(maxsize = 512)
def states(legs):
    '''{charge: the flat dense indices of the states of that charge, in row order}'''
    charge, code = np.zeros(1, np.int64), np.zeros(1, np.int64)
    for leg in legs:
        q = np.repeat([c for c, _ in leg], [m for _, m in leg])
        at = np.repeat(np.arange(len(leg)), [m for _, m in leg])
        charge = (charge[:, None] + q[None, :]).ravel()
        code = (code[:, None] * len(leg) + at[None, :]).ravel()
    order = np.argsort(code, kind = 'stable')
    return {int(q): order[charge[order] == q] for q in np.unique(charge)}


def shapes(cod, dom):
    '''{charge: (rows, cols)} of a neutral tensor's blocks, ascending.'''
    rows, cols = states(cod), states(dom)
    return {q: (len(rows[q]), len(cols[q])) for q in sorted(set(rows) & set(cols))}


def size(leg):
    return sum(m for _, m in leg)


def to_dense(blocks, cod, dom):
    rows, cols, dtype = states(cod), states(dom), next(iter(blocks.values())).dtype
    dims = [size(l) for l in cod + dom]
    out = torch.zeros((math.prod(dims[:len(cod)]), math.prod(dims[len(cod):])), dtype = dtype, device = DEVICE)
    for q, block in blocks.items():
        at = torch.from_numpy(rows[q]).to(DEVICE)[:, None], torch.from_numpy(cols[q]).to(DEVICE)[None, :]
        out[at] = block
    return out.view(dims)


def to_arena(dense, cod, dom):
    '''A dense tensor's blocks back to back, an odd block followed by one zero: the layout of `Tensor.data`.'''
    rows, cols = states(cod), states(dom)
    flat = dense.reshape(math.prod(size(l) for l in cod), -1)
    parts = [flat[torch.from_numpy(rows[q]).to(DEVICE)][:, torch.from_numpy(cols[q]).to(DEVICE)] for q in shapes(cod, dom)]
    return arena(parts)


def arena(blocks):
    parts = [b.reshape(-1) for b in blocks]
    return torch.cat([torch.nn.functional.pad(p, (0, p.numel() % 2)) for p in parts])


def flipped(t, axis, leg):
    '''Charge q of an axis read as -q (a leg on the other side of the tensor).'''
    start = dict(zip((q for q, _ in leg), np.cumsum([0] + [m for _, m in leg])))
    order = np.concatenate([np.arange(m) + start[-q] for q, m in leg])
    return t.index_select(axis, torch.from_numpy(order).to(t.device))


# ---------------------------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------------------------


def generator(seed):
    return torch.Generator(device = DEVICE).manual_seed(int(seed))


def normal(shape, dtype, gen):
    return torch.randn(shape, dtype = dtype, device = DEVICE, generator = gen)


def drawn(cod, dom, dtype, gen):
    return {q: normal(s, dtype, gen) for q, s in shapes(cod, dom).items()}


def hermitian_environment(leg, dtype, gen):
    '''(bond, operator | bond): Hermitian at the neutral operator states, adjoint to one another at charges
    2 and -2, as the environments of a Hermitian chain are; entries of a block scaled to a norm of order one.'''
    dense = torch.zeros((size(leg), 5, size(leg)), dtype = dtype, device = DEVICE)
    for copy in range(3):
        m = to_dense(drawn((leg,), (leg,), dtype, gen), (leg,), (leg,))
        dense[:, 1 + copy] = (m + m.mH) / 2
    raised = to_dense(drawn((leg, ((2, 1),)), (leg,), dtype, gen), (leg, ((2, 1),)), (leg,))[:, 0]
    dense[:, 4], dense[:, 0] = raised, raised.mH
    return dense / math.sqrt(size(leg))


def site_tensor(dtype):
    '''The Heisenberg automaton's bulk site (operator, out | in, operator), dense.'''
    up, down = 1, 0  # positions of the charges 1 and -1
    site = torch.zeros((5, 2, 2, 5), dtype = dtype, device = DEVICE)
    begin, z, done, plus, minus = 1, 2, 3, 4, 0
    for s, sign in ((up, 0.5), (down, -0.5)):
        site[begin, s, s, begin] = site[done, s, s, done] = 1
        site[begin, s, s, z] = site[z, s, s, done] = sign
    site[begin, up, down, plus] = site[begin, down, up, minus] = 1
    site[plus, down, up, done] = site[minus, up, down, done] = 0.5
    return site


def window_dense(case, seed):
    '''The two environments and the vector of one window.'''
    leg, dtype, gen = bond(case['chi'], case['charges']), DTYPES[case['dtype']], generator(seed)
    left, right = (hermitian_environment(leg, dtype, gen) for _ in range(2))
    theta = drawn((leg, PHYSICAL), (PHYSICAL, leg), dtype, gen)
    return leg, left, right, theta


def graded_blocks(case, seed):
    '''A two-site tensor of norm one whose blocks' singular values fall over the case's decades: the Schmidt
    values of each charge evenly spread in their logarithm, the blocks' ladders offset from one another.'''
    leg, dtype, gen = bond(case['chi'], case['charges']), DTYPES[case['dtype']], generator(seed)
    blocks = {}
    sides = shapes((leg, PHYSICAL), (PHYSICAL, leg))
    for at, (q, (m, n)) in enumerate(sides.items()):
        k = min(m, n)
        ladder = (torch.arange(k, dtype = torch.float64, device = DEVICE) + (at + 1) / (len(sides) + 2)) / k
        fall = math.exp(-q * q / 32) * 10 ** (-case['decades'] * ladder)
        u, v = (torch.linalg.qr(normal((x, k), dtype, gen))[0] for x in (m, n))
        blocks[q] = (u * fall) @ v.mT
    norm = math.sqrt(sum(float(torch.linalg.vector_norm(b)) ** 2 for b in blocks.values()))
    return leg, {q: b / norm for q, b in blocks.items()}


def site_legs(case):
    '''(bond, physical | bond) of one site, the bond to its right of odd charges.'''
    leg = bond(case['chi'], case['charges'])
    return leg, bond(case['chi'], case['charges'], True)


def braided_rows(case):
    '''{root: [(first, second), ...]} of the two-leg trees of the category's charges, in row order.'''
    out = {}
    for a in range(case['top'] + 1):
        for b in range(case['top'] + 1):
            if case['category'] == 'su2':
                roots = range(abs(a - b), a + b + 1, 2)
            else:
                roots = (0, 1) if a == b == 1 else (a + b,)
            for r in roots:
                out.setdefault(r, []).append((a, b))
    return dict(sorted(out.items()))


def braided_blocks(case, seed):
    gen, dtype = generator(seed), torch.complex128 if case['category'] == 'fibonacci' else torch.float64
    sides = {r: len(t) * case['mult'] ** 2 for r, t in braided_rows(case).items()}
    return [{r: normal((n, n), dtype, gen) for r, n in sides.items()} for _ in range(2)]


def batch_windows(case):
    rng = random.Random(case['pick'])
    return [{'chi': rng.choice((32, 64, 128, 256, 512)), 'charges': 17, 'dtype': 'f64'} for _ in range(case['windows'])]


# ---------------------------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------------------------


def tensor(cod, dom, blocks):
    import tentorch_gb300 as tg
    legs = [tg.Leg(tg.u1, [(q,) for q, _ in l], [m for _, m in l]) for l in cod + dom]
    out = tg.Tensor(tg.u1, legs[:len(cod)], legs[len(cod):], (0,), dtype = next(iter(blocks.values())).dtype, device = DEVICE)
    for q, block in blocks.items():
        out.block((q,), (q,)).copy_(block)
    return out


def from_dense(dense, cod, dom):
    rows, cols = states(cod), states(dom)
    flat = dense.reshape(math.prod(size(l) for l in cod), -1)
    return tensor(cod, dom, {q: flat[torch.from_numpy(rows[q]).to(DEVICE)][:, torch.from_numpy(cols[q]).to(DEVICE)]
                             for q in shapes(cod, dom)})


def window_tensors(case, seed):
    import tentorch_gb300 as tg
    leg, left, right, theta = window_dense(case, seed)
    site = from_dense(site_tensor(DTYPES[case['dtype']]), (OPERATOR, PHYSICAL), (PHYSICAL, OPERATOR))
    head = tg.einsum('EIa,IPqj->EPaqj', from_dense(left, (leg, OPERATOR), (leg,)), site)
    tail = tg.einsum('JRsk,Fkb->JRSFb', site, from_dense(right, (leg, OPERATOR), (leg,)))
    return head, tail, tensor((leg, PHYSICAL), (PHYSICAL, leg), theta)


def prepare(case, seed):
    import tentorch_gb300 as tg
    kind = case['kind']
    state = {'case': case}
    if kind in ('matvec', 'window'):
        state['head'], state['tail'], state['theta'] = window_tensors(case, seed)
    elif kind == 'batch':
        state['windows'] = [window_tensors(w, seed * 64 + i) for i, w in enumerate(batch_windows(case))]
    elif kind == 'environment':
        dtype, gen = DTYPES[case['dtype']], generator(seed)
        even, odd = site_legs(case)
        edge = even if case['side'] == 'left' else odd
        state['environment'] = from_dense(hermitian_environment(edge, dtype, gen), (edge, OPERATOR), (edge,))
        state['tensor'] = tensor((even, PHYSICAL), (odd,), drawn((even, PHYSICAL), (odd,), dtype, gen))
        state['site'] = from_dense(site_tensor(dtype), (OPERATOR, PHYSICAL), (PHYSICAL, OPERATOR))
    elif kind == 'split':
        leg, blocks = graded_blocks(case, seed)
        state['theta'] = tensor((leg, PHYSICAL), (PHYSICAL, leg), blocks)
    elif kind == 'canonical':
        even, odd = site_legs(case)
        blocks = drawn((even, PHYSICAL), (odd,), DTYPES[case['dtype']], generator(seed))
        state['tensor'] = tensor((even, PHYSICAL), (odd,), blocks)
    elif kind == 'recouple':
        cat = getattr(tg, case['category'])
        leg = tg.Leg(cat, [(q,) for q in range(case['top'] + 1)], [case['mult']] * (case['top'] + 1))
        state['operands'] = []
        for blocks in braided_blocks(case, seed):
            t = tg.Tensor(cat, [leg, leg], [leg, leg], (0,), dtype = blocks[0].dtype, device = DEVICE)
            for r, block in blocks.items():
                t.block((r,), (r,)).copy_(block)
            state['operands'].append(t)
    else:
        from tentorch_gb300.networks import DMRG, Model
        # as bench.py starts its runs: every block of the state from one seeded generator
        state['driver'] = DMRG(Model(case['length'] // 2 * 2, cat = tg.u1), max_bond_dim = case['chi'], n_iter = case['steps'],
                               dtype = DTYPES[case['dtype']], device = DEVICE,
                               generator = torch.Generator().manual_seed(seed), precision = case['slices'])
        state['start'] = [t.clone() for t in state['driver'].state.tensors]
    return state


def run(state):
    import tentorch_gb300 as tg
    case = state['case']
    kind = case['kind']
    if kind == 'matvec':
        # a Krylov step's vector is one that was just written
        increment_version(state['theta'].data)
        with tg.precision(case['slices']):
            return tg.einsum(MATVEC, state['head'], state['tail'], state['theta']).data
    if kind == 'window':
        from tentorch_gb300.lanczos import lanczos_einsum
        with tg.precision(case['slices']):
            energy, vector = lanczos_einsum(MATVEC, [state['head'], state['tail'], None], 2, state['theta'], case['steps'],
                                            wait = False)
        return {'energy': energy, 'vector': vector.data}
    if kind == 'batch':
        from tentorch_gb300.linalg import einsum_batch
        for _, _, theta in state['windows']:
            increment_version(theta.data)
        with tg.precision(case['slices']):
            return [t.data for t in einsum_batch(MATVEC, state['windows'])]
    if kind == 'environment':
        t, site, environment = state['tensor'], state['site'], state['environment']
        increment_version(t.data)  # the site a window just wrote, the environment it just advanced
        increment_version(environment.data)
        with tg.precision(case['slices']):
            if case['side'] == 'left':
                return tg.einsum(ADVANCE_LEFT, environment, t.conj(), t, site).data
            return tg.einsum(ADVANCE_RIGHT, t.conj(), t, site, environment).data
    if kind == 'split':
        # the values and the truncated two-site tensor: what the two factors are apart from their bond's basis
        first, values, second = tg.svd(state['theta'], case['chi'], CUTOFF, 2)
        return {'values': values, 'joined': tg.contract(first, second, tg.domain_legs(first), [0]).data}
    if kind == 'canonical':
        first, second = tg.qr(state['tensor'], [0, 1]) if case['side'] == 'left' else tg.rq(state['tensor'], [0])
        return {'first': first.data, 'second': second.data}
    if kind == 'recouple':
        for t in state['operands']:
            increment_version(t.data)
        with tg.precision(case['slices']):
            return tg.einsum(BRAIDED, *state['operands']).data
    driver = state['driver']
    driver.state.tensors, driver.state.center = [t.clone() for t in state['start']], 0
    energy, _ = driver.sweep()
    # the last window's Ritz value, and the energy of the state the sweep left
    return {'energy': energy, 'state': driver.energy().real}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits without the framework
# ---------------------------------------------------------------------------------------------


def dense_matvec(leg, left, right, site):
    '''theta (A, Q, s, b) -> image (E, P, r, f): two codomain legs of one letter pair charge q with -q, and so
    do two domain legs; a leg that changes sides reads q as -q.'''
    head = torch.einsum('eia,ipqj->epaqj', flipped(left, 1, OPERATOR), site)
    tail = torch.einsum('jrsk,fkb->jrsfb', site, right)
    tail = flipped(flipped(flipped(flipped(tail, 1, PHYSICAL), 2, PHYSICAL), 3, leg), 4, leg)

    def apply(theta):
        moved = torch.einsum('epaqj,aqsb->epjsb', head, theta)
        return torch.einsum('epjsb,jrsfb->eprf', moved, tail)
    return apply


def exact_window(case, seed):
    leg, left, right, theta = window_dense(case, seed)
    apply = dense_matvec(leg, left, right, site_tensor(DTYPES[case['dtype']]))
    sides = (leg, PHYSICAL), (PHYSICAL, leg)
    return apply, to_dense(theta, *sides), sides


def lowest(apply, start, steps):
    '''The lowest Ritz pair of a Krylov space, the tridiagonal vector's largest component positive.'''
    basis, alpha, beta = [start / torch.linalg.vector_norm(start)], [], []
    for _ in range(steps):
        image = apply(basis[-1])
        alpha.append(torch.vdot(basis[-1].reshape(-1), image.reshape(-1)).real)
        for _ in range(3):
            for v in basis:
                image = image - torch.vdot(v.reshape(-1), image.reshape(-1)) * v
        beta.append(torch.linalg.vector_norm(image))
        basis.append(image / beta[-1])
    t = torch.diag(torch.stack(alpha))
    for i, b in enumerate(beta[:-1]):
        t[i, i + 1] = t[i + 1, i] = b
    values, vectors = torch.linalg.eigh(t.cpu())
    v = vectors[:, 0]
    v = (v * torch.sign(v[v.abs().argmax()])).tolist()
    out = sum(c * b for c, b in zip(v, basis))
    return values[0], out / torch.linalg.vector_norm(out)


def exact_split(case, seed):
    leg, blocks = graded_blocks(case, seed)
    parts = {q: torch.linalg.svd(b.cpu(), full_matrices = False) for q, b in blocks.items()}
    ranked = sorted(((-float(s), q, i) for q, (_, sv, _) in parts.items() for i, s in enumerate(sv)), key = lambda c: c[0])
    ranked = [c for c in ranked if -c[0] > CUTOFF][:case['chi']]
    count = {q: sum(c[1] == q for c in ranked) for q in parts}
    # the bond keeps as many multiplets at q as at -q
    if any(count[q] and count.get(-q, 0) for q in count):
        count = {q: min(n, count.get(-q, 0)) for q, n in count.items()}
    values, joined = [], []
    for q, (u, s, vh) in parts.items():
        n = count[q]
        values.append(s[:n])
        joined.append((u[:, :n] * s[:n]) @ vh[:n])
    return {'values': torch.cat(values).to(DTYPES[case['dtype']]), 'joined': arena(joined)}


def exact_canonical(case, seed):
    even, odd = site_legs(case)
    blocks = drawn((even, PHYSICAL), (odd,), DTYPES[case['dtype']], generator(seed))
    if case['side'] == 'left':
        pairs = [torch.linalg.qr(b.cpu()) for b in blocks.values()]
        return {'first': arena([q for q, _ in pairs]), 'second': arena([r for _, r in pairs])}
    # (bond | physical, bond): the physical leg reads -q in the domain, ahead of the bond
    dense = flipped(to_dense(blocks, (even, PHYSICAL), (odd,)), 1, PHYSICAL)
    rows, cols = states((even,)), states((PHYSICAL, odd))
    flat = dense.reshape(size(even), -1)
    pairs = []
    for q in shapes((even,), (PHYSICAL, odd)):
        m = flat[torch.from_numpy(rows[q]).to(DEVICE)][:, torch.from_numpy(cols[q]).to(DEVICE)]
        pairs.append([f.transpose(0, 1) for f in torch.linalg.qr(m.cpu().transpose(0, 1))])
    return {'first': arena([r for _, r in pairs]), 'second': arena([q for q, _ in pairs])}


def braid(case, a, b, root):
    '''The phase of exchanging two charges under a root.'''
    if case['category'] == 'su2':
        return -1.0 if (a + b - root) // 2 % 2 else 1.0
    angle = (-4 if root == 0 else 3) * math.pi / 5 if a == b == 1 else 0.0
    return complex(math.cos(angle), math.sin(angle))


def exact_braided(case, seed):
    left, right = braided_blocks(case, seed)
    m, out = case['mult'], []
    for root, trees in braided_rows(case).items():
        n = len(trees)
        block = right[root].view(n, m, m, -1)
        moved = torch.empty_like(block)
        for i, (c, d) in enumerate(trees):
            moved[i] = block[trees.index((d, c))].transpose(0, 1) * braid(case, c, d, root)
        out.append(left[root] @ moved.reshape(n * m * m, -1))
    return arena(out)


def exact_environment(case, seed):
    dtype, gen = DTYPES[case['dtype']], generator(seed)
    even, odd = site_legs(case)
    edge = even if case['side'] == 'left' else odd
    environment = hermitian_environment(edge, dtype, gen)
    t = to_dense(drawn((even, PHYSICAL), (odd,), dtype, gen), (even, PHYSICAL), (odd,))
    site = site_tensor(dtype)
    if case['side'] == 'left':
        out = torch.einsum('eia,eqf->iaqf', flipped(environment, 1, OPERATOR), t.conj())
        out = torch.einsum('iaqf,apb->ifqpb', out, t)
        out = torch.einsum('ifqpb,iqpj->fjb', out, site)
        return to_arena(flipped(out, 1, OPERATOR), (odd, OPERATOR), (odd,))
    environment = flipped(flipped(environment, 0, edge), 2, edge)
    out = torch.einsum('fqg,gkb->fqkb', t.conj(), environment)
    out = torch.einsum('fqkb,apb->fqkap', out, t)
    out = torch.einsum('fqkap,iqpk->fia', out, site)
    return to_arena(flipped(flipped(out, 0, even), 2, even), (even, OPERATOR), (even,))


def exact(case, seed):
    kind = case['kind']
    if kind in ('matvec', 'batch'):
        out = []
        for i, w in enumerate([case] if kind == 'matvec' else batch_windows(case)):
            apply, theta, sides = exact_window(w, seed if kind == 'matvec' else seed * 64 + i)
            out.append(to_arena(apply(theta), *sides))
        return out[0] if kind == 'matvec' else out
    if kind == 'window':
        apply, theta, sides = exact_window(case, seed)
        energy, vector = lowest(apply, theta, case['steps'])
        return {'energy': energy, 'vector': to_arena(vector, *sides)}
    if kind == 'sweep':
        return None  # the whole algorithm over again, many seconds of it in plain torch
    return {'environment': exact_environment, 'split': exact_split, 'canonical': exact_canonical,
            'recouple': exact_braided}[kind](case, seed)


# ---------------------------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------------------------


def entries(cod, dom):
    return sum(m * n for m, n in shapes(cod, dom).values())


def product_flops(rows, mid, cols):
    a, b, c = states(rows), states(mid), states(cols)
    return 2 * sum(len(a[q]) * len(b[q]) * len(c[q]) for q in set(a) & set(b) & set(c))


def matvec_work(case):
    leg = bond(case['chi'], case['charges'])
    width, factor = (16, 4) if case['dtype'] == 'c128' else (8, 1)
    head = entries((leg, PHYSICAL), (leg, PHYSICAL, OPERATOR))
    moved = product_flops((leg, PHYSICAL, OPERATOR), (leg, PHYSICAL), (PHYSICAL, leg))
    image = product_flops((leg, PHYSICAL), (OPERATOR, PHYSICAL, leg), (PHYSICAL, leg))
    return {'bytes': width * (2 * head + 2 * entries((leg, PHYSICAL), (PHYSICAL, leg))), 'flops': factor * (moved + image)}


def work(case):
    kind = case['kind']
    width, factor = (16, 4) if case.get('dtype') == 'c128' or case.get('category') == 'fibonacci' else (8, 1)
    if kind == 'matvec':
        return matvec_work(case)
    if kind == 'window':
        one = matvec_work(case)
        leg = bond(case['chi'], case['charges'])
        vector = entries((leg, PHYSICAL), (PHYSICAL, leg))
        # every Krylov vector written once and read for the projections of the later steps
        return {'bytes': one['bytes'] + width * vector * case['steps'], 'flops': case['steps'] * one['flops'] +
                factor * 12 * vector * case['steps'] * (case['steps'] + 1) / 2}
    if kind == 'batch':
        parts = [matvec_work(w) for w in batch_windows(case)]
        return {k: sum(p[k] for p in parts) for k in ('bytes', 'flops')}
    if kind == 'environment':
        even, odd = site_legs(case)
        edge, other = (even, odd) if case['side'] == 'left' else (odd, even)
        size_in, size_out, site = entries((edge, OPERATOR), (edge,)), entries((other, OPERATOR), (other,)), entries((even, PHYSICAL), (odd,))
        first = product_flops((edge, OPERATOR), (edge,), (PHYSICAL, other))
        second = product_flops((other,), (PHYSICAL, edge), (OPERATOR, other))
        return {'bytes': width * (size_in + size_out + site), 'flops': factor * (first + second)}
    if kind == 'split':
        leg = bond(case['chi'], case['charges'])
        blocks = shapes((leg, PHYSICAL), (PHYSICAL, leg)).values()
        flops = sum(6 * max(s) * min(s) ** 2 + 20 * min(s) ** 3 for s in blocks)
        return {'bytes': width * 2 * sum(m * n for m, n in blocks), 'flops': factor * flops}
    if kind == 'canonical':
        even, odd = site_legs(case)
        sides = ((even, PHYSICAL), (odd,)) if case['side'] == 'left' else ((even,), (PHYSICAL, odd))
        blocks = shapes(*sides).values()
        flops = sum(4 * max(s) * min(s) ** 2 - 4 * min(s) ** 3 / 3 for s in blocks)
        return {'bytes': width * sum(m * n + min(m, n) * (m + n) for m, n in blocks), 'flops': factor * flops}
    if kind == 'recouple':
        sides = [len(t) * case['mult'] ** 2 for t in braided_rows(case).values()]
        return {'bytes': 3 * width * sum(n * n for n in sides), 'flops': factor * sum(2 * n ** 3 for n in sides)}
    # a sweep: two windows a bond, each its Krylov steps, at the bonds a chain of this length reaches
    total = {'bytes': 0, 'flops': 0}
    length = case['length'] // 2 * 2
    for at in range(1, length):
        chi = min(case['chi'], 2 ** min(at, length - at))
        one = matvec_work(dict(case, chi = chi, charges = 5))
        total['bytes'] += 2 * one['bytes']
        total['flops'] += 2 * case['steps'] * one['flops']
    return total
