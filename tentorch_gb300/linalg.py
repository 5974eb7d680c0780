'''
The contraction path and the linear algebra over block-sparse tensors, with the Python surface of
the reference: `einsum(spec, *tensors, outcharge=None)`, `contract(left, right, left_legs,
right_legs, charge=None)`, `Tensor.place`, `inner`, `norm`, `is_close`, `svd`, `svdvals`, `qr`,
`rq` (tentorch/_ext/bindings.cpp:330-431).

`einsum`, `contract` and `place` compile a plan once per combination of operand spaces (the
engine caches it) and run it on the tensors' CUDA device, on the current torch stream, with no
host synchronisation.  An operand's "prepare" work (the leg moves that depend on it alone) is
cached against the operand's arena and its version counter, so a loop that applies the same
operator to changing vectors (the Lanczos matvec) recouples the operator once.

Block products run in FP64 by default; `precision(k)` switches them to split products on the
tensor cores with k bf16 slices per operand (see gemm.h).
'''
from __future__ import annotations

import contextlib
import ctypes
import math
import weakref
from typing import Optional

import torch

from tentorch_gb300._lib import check, f64, i32, i64, ints32, ints64, lib, pointers, vp
from tentorch_gb300.symmetry import Leg, _label
from tentorch_gb300.tensor import BlockKey, Space, Tensor

_DTYPE = {torch.float64: 0, torch.complex128: 1}
_precision = 0
PER_BLOCK = -1  # the plain per-block FP64 form: one cuBLAS call per block pair


def set_precision(slices: int) -> None:
    '''0: FP64 block products in the grouped kernels; k in 1..8: split products with k bf16 slices
    per operand; PER_BLOCK (-1): the plain per-block FP64 form, one cuBLAS call per block pair, as
    the reference issues its block products on a CUDA device (tentorch/linalg/graded/contract.cpp:148-163).'''
    global _precision
    if not PER_BLOCK <= int(slices) <= 8:
        raise ValueError(f'precision is 0 (FP64), 1..8 slices or -1 (per-block FP64), not {slices}')
    _precision = int(slices)


def get_precision() -> int:
    return _precision


@contextlib.contextmanager
def precision(slices: int):
    '''Run the block products inside the block with `slices` bf16 slices (0: FP64).'''
    old = _precision
    set_precision(slices)
    try:
        yield
    finally:
        set_precision(old)


def _raw_stream(index: int) -> int:
    '''The current stream of a CUDA device as a raw handle (without building a torch.cuda.Stream).'''
    return torch._C._cuda_getCurrentRawStream(index)


def _capturing() -> bool:
    return torch._C._cuda_isCurrentStreamCapturing()


# ctypes array types by length
_vector_types = {}


def _addresses(values):
    '''A ctypes array of the addresses (None: null).'''
    kind = _vector_types.get(len(values))
    if kind is None:
        kind = _vector_types[len(values)] = vp * len(values)
    return kind(*values)


class Plan:
    '''A compiled program: its output space, workspace and the size of each operand's prepared
    arena.  The engine owns the program; a wholesale clear of the plan caches frees it, and a Plan
    held across that clear compiles its program again on its next use (same key, same result).'''
    __slots__ = ('_handle', 'generation', 'key', 'build', 'cat', 'out_space', 'workspace', 'flops', 'moved', 'n_ops',
                 'sizes', '__weakref__')

    def __init__(self, handle, cat, key = None, build = None):
        self._handle, self.cat, self.key, self.build = handle, cat, key, build
        self.generation = _generation
        space, ws, flops, moved, ops = i32(), i64(), f64(), i64(), i32()
        check(lib.tt_plan_info(handle, ctypes.byref(space), ctypes.byref(ws), ctypes.byref(flops), ctypes.byref(moved),
                               ctypes.byref(ops)))
        self.out_space = Space._load(cat, space.value)
        self.workspace, self.flops, self.moved, self.n_ops = ws.value, flops.value, moved.value, ops.value
        self.sizes = {}

    @property
    def handle(self):
        if self.generation != _generation:
            if self.build is None:
                raise RuntimeError('this plan was freed by clear_plans()')
            fresh = _plan(self.key, self.build, self.cat)
            self._handle, self.generation = fresh._handle, fresh.generation
        return self._handle

    def describe(self) -> str:
        '''The plan's operations and GEMM block shapes, as text.'''
        n = i64()
        check(lib.tt_plan_describe(self.handle, 0, None, ctypes.byref(n)))
        buf = ctypes.create_string_buffer(n.value + 1)
        check(lib.tt_plan_describe(self.handle, n.value + 1, buf, ctypes.byref(n)))
        return buf.value.decode()

    def prepared_size(self, operand: int) -> int:
        size = self.sizes.get(operand)
        if size is None:
            n = i64()
            check(lib.tt_plan_prepared_size(self.handle, operand, ctypes.byref(n)))
            size = self.sizes[operand] = n.value
        return size


_plans = {}
# compiled plans kept before a wholesale clear (the reference clears its plan caches wholesale at a
# budget, tentorch/tensors/cache.cpp:203-217): DMRG compiles new shapes at every window, so without
# a bound the caches would grow with the length of the run
_PLAN_BUDGET = 4096
_generation = 0
# (plan handle, operand) -> (weakref to the operand arena, its version, the prepared arena or None
# when the operand has been seen once and not prepared yet)
_prepared = {}
# (device index, stream, dtype) -> a workspace arena that grows to the largest plan run on it; the
# ops of one stream run in order, so consecutive plans share it
_pools = {}
# workspaces replaced by larger ones after a capture (a captured graph may still address them)
_superseded = []
# set once a plan has run inside a CUDA graph capture: the graph holds the device addresses of its
# tables and workspace, so the automatic clear at the budget no longer runs
_captured = False


def clear_plans() -> None:
    '''Forget every compiled plan, here and in the engine (their device tables are freed): the next
    contraction of each shape compiles again.  Runs by itself when the cache reaches its budget
    (unless a CUDA graph captured plans of this process); by hand, for timing compilation.  A CUDA
    graph captured before a clear launches freed tables: capture it again after one.'''
    global _generation, _captured
    _generation += 1
    _captured = False
    _plans.clear()
    _prepared.clear()
    _pools.clear()
    _batch_pools.clear()
    _superseded.clear()
    _qr_plans.clear()
    _split_layouts.clear()
    _split_writes.clear()
    check(lib.tt_plan_cache_clear())


def cached_plans() -> int:
    '''How many compiled plans the cache holds.'''
    return len(_plans)


def _note_capture() -> None:
    global _captured
    _captured = True


def _plan(key, build, cat) -> Plan:
    plan = _plans.get(key)
    if plan is None:
        if len(_plans) >= _PLAN_BUDGET and not _captured:
            clear_plans()
        handle = vp()
        check(build(ctypes.byref(handle)))
        plan = Plan(handle, cat, key, build)
        _plans[key] = plan
    return plan


def _uploaded(values, dtype, device) -> torch.Tensor:
    '''A small host table on the device without waiting for the stream's queued work: staged
    through page-locked memory (torch's host cache keeps the staging block until the copy is done),
    so the copy is queued like a kernel and the host returns at once.'''
    if not values:
        return torch.empty(0, dtype = dtype, device = device)
    return torch.tensor(values, dtype = dtype).pin_memory().to(device, non_blocking = True)


class _KeptTable:
    '''A device table that later calls use too, on whichever stream they run: one of another stream than the upload's
    waits for the upload and is recorded with the table's memory.  (Under capture neither is needed or possible: a
    capture begins with the device idle, and what it uses is not dropped.)'''
    __slots__ = ('table', 'stream', 'uploaded')

    def __init__(self, values, dtype, device):
        self.table = _uploaded(values, dtype, device)
        self.stream = _raw_stream(self.table.get_device())
        self.uploaded = torch.cuda.Event()
        self.uploaded.record(torch.cuda.current_stream(device))

    def address(self, stream: int) -> int:
        if stream != self.stream and not _capturing():
            current = torch.cuda.current_stream(self.table.device)
            current.wait_event(self.uploaded)
            self.table.record_stream(current)
        return self.table.data_ptr()


def _check_device(tensors) -> None:
    dtype, device = tensors[0].dtype, tensors[0].device
    for t in tensors:
        if t.dtype != dtype:
            raise ValueError('a contraction needs both tensors of one scalar type')
        if t.device != device:
            raise ValueError('a contraction needs every tensor on one device')
    if device.type != 'cuda':
        raise RuntimeError('tentorch_gb300 computes on a CUDA device; these tensors live on the host '
                           '(move them with .to("cuda"))')


def _workspace(plan: Plan, device, dtype, stream) -> Optional[torch.Tensor]:
    if plan.workspace <= 0:
        return None
    key = (device.index, stream, dtype)
    pool = _pools.get(key)
    if pool is None or pool.numel() < plan.workspace:
        if pool is not None and _captured:
            # a CUDA graph captured earlier may hold this pool's address: keep it allocated, so that
            # a replay never writes into memory the caching allocator has handed to another tensor
            _superseded.append(pool)
        # zero: the head of a workspace holds the GEMM tickets, which every execution leaves zero
        pool = _pools[key] = torch.zeros(max(plan.workspace, 1 << 16), dtype = dtype, device = device)
    return pool


def _prepared_arena(plan: Plan, operand: int, tensor: Tensor, ws, stream, force: bool = False) -> Optional[torch.Tensor]:
    """The operand's prepared arena when the same arena (same version) comes back to this plan: the
    first sighting runs the operand's phase inside the plan and only remembers the arena; the
    second prepares it once for every call after (the head and tail of a Lanczos window).  Entries
    are per arena, so windows that share a plan each keep theirs; an entry goes with its arena."""
    size = plan.prepared_size(operand)
    if size <= 0:
        return None
    data = tensor._data
    key = (plan.handle.value, operand, data.data_ptr())
    held = _prepared.get(key)
    mine = held is not None and held[0]() is data
    seen = mine and held[1] == data._version
    if seen and held[2] is not None:
        return held[2]
    arena = None
    if force or seen:
        arena = torch.empty(size, dtype = data.dtype, device = data.device)
        check(lib.tt_plan_prepare(plan.handle, _DTYPE[data.dtype], operand, data.data_ptr(), arena.data_ptr(),
                                  ws.data_ptr() if ws is not None else None, stream))
    if not mine:
        def forget(ref, key = key):
            entry = _prepared.get(key)
            if entry is not None and entry[0] is ref:
                del _prepared[key]
        ref = weakref.ref(data, forget)
    else:
        ref = held[0]
    _prepared[key] = (ref, data._version, arena)
    return arena


def _prepare_now(plan: Plan, operand: int, tensor: Tensor, ws, stream) -> Optional[torch.Tensor]:
    '''The operand prepared into a new arena, not cached (the form a CUDA graph captures).'''
    size = plan.prepared_size(operand)
    if size <= 0:
        return None
    data = tensor._data
    arena = torch.empty(size, dtype = data.dtype, device = data.device)
    check(lib.tt_plan_prepare(plan.handle, _DTYPE[data.dtype], operand, data.data_ptr(), arena.data_ptr(),
                              ws.data_ptr() if ws is not None else None, stream))
    return arena


def run(plan: Plan, tensors, out: Optional[Tensor] = None, reuse_prepared: bool = True) -> Tensor:
    """Execute a plan on the operands' device and return the output tensor."""
    data0 = tensors[0]._data
    dtype, index = data0.dtype, data0.get_device()
    for t in tensors:
        if t._data.dtype != dtype or t._data.get_device() != index:
            _check_device(tensors)
    if index < 0:
        _check_device(tensors)
    device = data0.device
    if out is None:
        out = Tensor._wrap(plan.out_space, torch.empty(plan.out_space.size, dtype = dtype, device = device))
    stream = _raw_stream(index)
    # a captured CUDA graph reads every operand from its own buffer at each replay, never a prepared copy
    if _capturing():
        _note_capture()
        reuse_prepared = False
    handle = plan.handle
    ws = _workspace(plan, device, dtype, stream)
    ws_at = ws.data_ptr() if ws is not None else None
    if reuse_prepared:
        prep = []
        for i, t in enumerate(tensors):
            arena = _prepared_arena(plan, i, t, ws, stream)
            prep.append(arena.data_ptr() if arena is not None else None)
        prep = _addresses(prep)
    else:
        prep = None
    status = lib.tt_plan_execute(handle, _DTYPE[dtype], _precision, _addresses([t._data.data_ptr() for t in tensors]), prep,
                                 out._data.data_ptr(), ws_at, stream)
    if status:
        check(status)
    return out


def place(tensor: Tensor, above, below = None) -> Tensor:
    '''tentorch/tensors/place.cpp:183-247'''
    total = tensor.nlegs()
    above = [int(a) for a in above]
    if below is None:
        named = set(a for a in above if 0 <= a < total)
        below = [leg for leg in range(total) if leg not in named]
    below = [int(b) for b in below]
    plan = place_plan(tensor._space, above, below)
    if plan.n_ops == 0:
        return tensor
    return run(plan, [tensor], reuse_prepared = False)


def place_plan(space: Space, above, below) -> Plan:
    '''The compiled plan of `place` on a tensor of this space (legs already resolved).'''
    above, below = tuple([int(x) for x in above]), tuple([int(x) for x in below])
    key = ('place', space.id, above, below)
    plan = _plans.get(key)
    if plan is not None:
        return plan
    a, na = ints32(above)
    b, nb = ints32(below)
    return _plan(key, lambda out: lib.tt_plan_place(space.id, na, a, nb, b, out), space.cat)


def conj(tensor: Tensor) -> Tensor:
    '''tentorch/tensors/tensor.cpp:99-107: the bra of a tensor, one compiled pass.'''
    return run(conj_plan(tensor._space), [tensor], reuse_prepared = False)


def conj_plan(space: Space) -> Plan:
    '''The compiled plan of `conj` on a tensor of this space.'''
    return _plan(('conj', space.id), lambda out: lib.tt_plan_conj(space.id, out), space.cat)


def contract(left: Tensor, right: Tensor, left_legs, right_legs, charge = None) -> Tensor:
    '''tentorch/linalg/graded/contract.cpp:117-175'''
    if left.cat is not right.cat:
        raise ValueError('a contraction needs both tensors over one category')
    if left.dtype != right.dtype:
        raise ValueError('a contraction needs both tensors of one scalar type')
    return run(contract_plan(left._space, right._space, left_legs, right_legs, charge), [left, right])


def contract_plan(left: Space, right: Space, left_legs, right_legs, charge = None) -> Plan:
    '''The compiled plan of `contract` on tensors of these spaces.'''
    left_legs, right_legs = tuple([int(x) for x in left_legs]), tuple([int(x) for x in right_legs])
    has = charge is not None
    q = _label(charge) if has else 0
    key = ('contract', left.id, right.id, left_legs, right_legs, has, q)
    plan = _plans.get(key)
    if plan is not None:
        return plan
    la, n = ints32(left_legs)
    ra, m = ints32(right_legs)
    if n != m:
        raise ValueError(f'the two legs of a contraction must be given in pairs, got {n} and {m}')
    return _plan(key, lambda out: lib.tt_plan_contract(left.id, right.id, n, la, ra, int(has), q, out), left.cat)


def einsum(spec: str, *tensors: Tensor, **options) -> Tensor:
    '''tentorch/linalg/graded/einsum.cpp:444-605 with the binding's keyword handling
    (tentorch/_ext/bindings.cpp:347-361): only `outcharge` is accepted.'''
    for name in options:
        if name != 'outcharge':
            raise ValueError(f"einsum does not take the keyword '{name}'")
    outcharge = options.get('outcharge')
    if not tensors:
        raise ValueError('an einsum needs at least one operand')
    cat = tensors[0]._space.cat
    for t in tensors:
        if t._space.cat is not cat:
            raise ValueError('an einsum needs every operand over one category')
    return run(einsum_plan(spec, [t._space for t in tensors], outcharge), tensors)


# per (device, stream, dtype, window): the workspace of one window of a batch (a batch's windows run
# together, so each needs its own)
_batch_pools = {}
# launches of block products the last einsum_batch made (1 when its windows ran as one launch)
last_batch_launches = 0


def einsum_batch(spec: str, operand_lists, outcharge = None) -> list:
    '''`[einsum(spec, *ops) for ops in operand_lists]` as one call (tt_plan_execute_batch): in FP64
    the two-site matvecs of many windows (different bond dimensions allowed) run as ONE persistent
    launch with their work items dealt together over the SMs; in split precision, or for equations
    that are not a product chain, one window after another.  At most 64 windows per launch (longer
    lists are cut into launches of 64).  Operands are prepared per window as `einsum` prepares them;
    under a CUDA graph capture every operand is read from its buffer (a warm-up call outside the
    capture compiles the plans and deals the batch first).'''
    global last_batch_launches
    operand_lists = [list(ops) for ops in operand_lists]
    if len(operand_lists) > 64:
        return einsum_batch(spec, operand_lists[:64], outcharge) + einsum_batch(spec, operand_lists[64:], outcharge)
    if not operand_lists:
        return []
    first = operand_lists[0][0]
    device, dtype = first._data.device, first._data.dtype
    stream = _raw_stream(first._data.get_device())
    # a captured CUDA graph reads every operand from its own buffer at each replay
    capturing = _capturing()
    if capturing:
        _note_capture()
    handles, outs, keep, inputs, prepared, workspaces = [], [], [], [], [], []
    for w, ops in enumerate(operand_lists):
        _check_device(ops)
        plan = plan_of(spec, *ops, outcharge = outcharge)
        key = (device.index, stream, dtype, w)
        pool = _batch_pools.get(key)
        if pool is None or pool.numel() < plan.workspace:
            if pool is not None and _captured:
                _superseded.append(pool)
            pool = _batch_pools[key] = torch.zeros(max(plan.workspace, 1 << 16), dtype = dtype, device = device)
        prep = [None if capturing else _prepared_arena(plan, i, t, pool, stream) for i, t in enumerate(ops)]
        out = Tensor._wrap(plan.out_space, torch.empty(plan.out_space.size, dtype = dtype, device = device))
        handles.append(plan.handle.value)
        outs.append(out)
        ins = pointers(t._data.data_ptr() for t in ops)
        pre = pointers((p.data_ptr() if p is not None else None) for p in prep)
        keep += [ins, pre, prep]
        inputs.append(ctypes.cast(ins, vp).value)
        prepared.append(ctypes.cast(pre, vp).value)
        workspaces.append(pool.data_ptr())
    launched = i32()
    check(lib.tt_plan_execute_batch(len(handles), pointers(handles), _DTYPE[dtype], _precision, pointers(inputs),
                                    pointers(prepared), pointers(o._data.data_ptr() for o in outs),
                                    pointers(workspaces), stream, ctypes.byref(launched)))
    last_batch_launches = launched.value
    return outs


# the forms a plan's block products run in (tt_autotune): bits of the integer autotune returns
FORM_SEPARATE = 1          # a product chain (the two-site matvec) as separate launches
FORM_NO_TENSOR_CORES = 2   # split products on mma.sync instead of tcgen05


def histogram_key(plan: Plan) -> int:
    '''The 64-bit key of a plan's block-size histogram (the autotuner's cache key).'''
    key = ctypes.c_uint64()
    check(lib.tt_plan_histogram(plan.handle, ctypes.byref(key)))
    return key.value


def autotune(spec: str, *operands: Tensor, outcharge = None) -> tuple:
    '''Time every form the einsum's block products can run in on these operands, in the current
    precision, and cache the fastest under the plan's block-size histogram: every later execution
    of a plan with the same histogram (any operands of these shapes, or of others that bin alike)
    runs it.  Returns (forms, milliseconds).  Synchronous; call it outside CUDA graph captures.'''
    _check_device(operands)
    plan = plan_of(spec, *operands, outcharge = outcharge)
    data0 = operands[0]._data
    device = data0.device
    stream = torch.cuda.current_stream(device).cuda_stream
    ws = _workspace(plan, device, data0.dtype, stream)
    prepared = [_prepared_arena(plan, i, t, ws, stream, force = True) for i, t in enumerate(operands)]
    out = torch.empty(plan.out_space.size, dtype = data0.dtype, device = device)
    forms, ms = i32(), ctypes.c_float()
    check(lib.tt_autotune(plan.handle, _DTYPE[data0.dtype], _precision, pointers(t._data.data_ptr() for t in operands),
                          pointers((p.data_ptr() if p is not None else None) for p in prepared), out.data_ptr(),
                          ws.data_ptr() if ws is not None else None, stream, ctypes.byref(forms), ctypes.byref(ms)))
    return forms.value, ms.value


def tuned_forms(plan: Plan, dtype = torch.float64, precision: Optional[int] = None) -> Optional[int]:
    '''The forms cached for the plan's histogram (tt_autotune_lookup), or None.'''
    forms, found = i32(), i32()
    check(lib.tt_autotune_lookup(histogram_key(plan), _DTYPE[dtype], _precision if precision is None else precision,
                                 ctypes.byref(forms), ctypes.byref(found)))
    return forms.value if found.value else None


def store_forms(plan: Plan, forms: int, dtype = torch.float64, precision: Optional[int] = None) -> None:
    '''Cache forms for the plan's histogram by hand (tt_autotune_store): a saved tuning restored.'''
    check(lib.tt_autotune_store(histogram_key(plan), _DTYPE[dtype], _precision if precision is None else precision,
                                int(forms)))


def clear_tuning() -> None:
    '''Forget every cached form choice (tt_autotune_clear).'''
    check(lib.tt_autotune_clear())


def link_copy(dst: torch.Tensor, src: torch.Tensor) -> torch.Tensor:
    '''dst.copy_(src) between a page-locked host tensor and a CUDA tensor (either way round) by a
    kernel that reads or writes the host end over the coherent CPU-GPU link (tt_link_copy), on the
    current stream, without a copy-engine call.  Both contiguous, of one dtype and size; the host
    tensor pinned (`pin_memory=True`), else ValueError.'''
    if dst.dtype != src.dtype or dst.numel() != src.numel() or not dst.is_contiguous() or not src.is_contiguous():
        raise ValueError('link_copy needs two contiguous tensors of one dtype and size')
    if dst.device.type == 'cuda' and src.device.type == 'cpu':
        direction, device = 0, dst.device
    elif dst.device.type == 'cpu' and src.device.type == 'cuda':
        direction, device = 1, src.device
    else:
        raise ValueError('link_copy copies between a host tensor and a CUDA tensor')
    stream = torch.cuda.current_stream(device).cuda_stream
    check(lib.tt_link_copy(dst.data_ptr(), src.data_ptr(), dst.numel() * dst.element_size(), direction, stream))
    # the kernel wrote dst behind torch's back: mark it written, so that no prepared copy of its
    # old contents is reused
    from torch.autograd.graph import increment_version
    increment_version(dst)
    return dst


def plan_of(spec: str, *tensors: Tensor, outcharge = None) -> Plan:
    '''The compiled plan an einsum of these operands runs (for timing and the roofline).'''
    return einsum_plan(spec, [t._space for t in tensors], outcharge)


def einsum_plan(spec: str, spaces, outcharge = None) -> Plan:
    '''The compiled plan of an einsum over operands of these spaces: compiling ahead of the call
    (from spaces a caller expects) fills the cache the call reads.'''
    has = outcharge is not None
    q = _label(outcharge) if has else 0
    key = ('einsum', spec, tuple([s.id for s in spaces]), has, q)
    plan = _plans.get(key)
    if plan is not None:
        return plan
    ids, n = ints32(s.id for s in spaces)
    return _plan(key,
                 lambda out: lib.tt_plan_einsum(spec.encode(), n, ids, int(has), q, out), spaces[0].cat)


# ---------------------------------------------------------------------------------------------
# scalar products (tentorch/linalg/graded/compare.cpp)
# ---------------------------------------------------------------------------------------------


def _same_legs(a: Tensor, b: Tensor) -> None:
    if a.cat is not b.cat:
        raise ValueError('a scalar product needs both tensors over one category')
    if a._space.codomain != b._space.codomain or a._space.domain != b._space.domain:
        raise ValueError('a scalar product needs both tensors with the same legs')


def inner_device(a: Tensor, b: Tensor) -> torch.Tensor:
    '''<a, b> as a 0-d device tensor, with no host synchronisation (the arena padding is zero).'''
    _same_legs(a, b)
    if a.qtotal != b.qtotal:
        return torch.zeros((), dtype = a.dtype, device = a.device)
    return torch.vdot(a._data, b._data)


def inner(a: Tensor, b: Tensor) -> complex:
    '''tentorch/linalg/graded/compare.cpp:31-43'''
    return complex(inner_device(a, b).item())


def norm(t: Tensor) -> float:
    '''tentorch/linalg/graded/compare.cpp:45'''
    return math.sqrt(abs(inner(t, t)))


def is_close(first: Tensor, second: Tensor, rtol: float = 1e-10, atol: float = 1e-12) -> bool:
    '''tentorch/linalg/graded/compare.cpp:12-29'''
    if first.cat is not second.cat or first.qtotal != second.qtotal:
        return False
    if first._space is not second._space:
        return False
    return bool(torch.allclose(first._data, second._data.to(first.device), rtol = rtol, atol = atol))


# ---------------------------------------------------------------------------------------------
# splittings (tentorch/linalg/graded/svd.cpp)
# ---------------------------------------------------------------------------------------------


# The cuSOLVER method of the per-block SVDs on a CUDA device.  'gesvd' (QR iteration) leaves the
# factors orthonormal to ~4e-15; torch's default for these block sizes (Jacobi, gesvdj) only to
# ~1e-13, which moves a DMRG sweep energy at L = 64, bond 256 by ~1.4e-10.  None picks torch's
# default, which is what the reference's at::linalg_svd (tentorch/linalg/graded/svd.cpp:59) runs
# on a CUDA device.
PER_BLOCK_SVD_DRIVER: Optional[str] = 'gesvd'


# splits whose Jacobi SVD left a block unsettled and were redone per block with cuSOLVER
svd_fallbacks = 0


def _factor_blocks_per_block(arranged: Tensor, present, while_waiting = None):
    '''The thin SVD of each present block by at::linalg_svd, one block at a time (svd.cpp:57-62).'''
    factors = []
    driver = PER_BLOCK_SVD_DRIVER if arranged.device.type == 'cuda' else None
    for i, key in present:
        u, sv, vh = torch.linalg.svd(arranged._view(i), full_matrices = False, driver = driver)
        factors.append([key, u, sv, vh, 0, 0])
    if while_waiting is not None:
        while_waiting()
    host = torch.cat([f[2] for f in factors]).to('cpu', torch.float64).tolist() if factors else []
    return factors, host


class _SplitLayout:
    '''What the batched SVD of the tensors of one space needs on a device, laid out once: the device table of its blocks
    and of the ranking, the places of the packed factors and the workspace in one buffer.'''
    __slots__ = ('present', 'count', 'largest', 'blocks', 'table', 'order', 'qr_ranks', 'ranking', 'n_blocks', 'n_sectors', 'sv_at',
                 'vh_at', 'ws_at', 'values', 'size')

    def __init__(self, space: Space, device, present, places, total: int, width: int, qr = None):
        '''`places` and `total`: each block's workspace and all of it in elements, of `width` doubles; `qr` (complex128): the
        blocks' QR table (a row a block) and the cluster size.'''
        cat = space.cat
        self.present = present
        entries, self.blocks, ids = [], [], {}
        u_at = s_at = vh_at = 0
        for at, (i, key) in enumerate(self.present):
            rows, cols = space.shapes[i]
            k = min(rows, cols)
            entries.append([space.offsets[i], rows, cols, u_at, s_at, vh_at, places[at]])
            self.blocks.append((key, rows, cols, k, u_at, s_at, vh_at))
            u_at, s_at, vh_at = u_at + rows * k, s_at + k, vh_at + k * cols
            for sector in (key.domain, cat.dual(key.domain)):
                ids.setdefault(sector, len(ids))
        # the largest blocks first: the launch's clusters then finish together, small blocks last
        self.order = sorted(range(len(entries)), key = lambda at: -min(entries[at][1:3]) ** 2 * max(entries[at][1:3]))
        rows = [x for at in self.order for x in entries[at]]
        self.qr_ranks = 0
        if qr is not None:
            rows += [x for at in self.order for x in qr[0][8 * at:8 * at + 8]]
            self.qr_ranks = qr[1]
        self.count = self.n_blocks = len(self.present)
        self.largest = max((b[3] for b in self.blocks), default = 0)
        self.n_sectors = len(ids)
        self.values = s_at
        # one buffer: U, the values, Vh, then the workspace, each from a multiple of 32 doubles
        up = lambda n: (n + 31) // 32 * 32
        self.sv_at = up(width * u_at)
        self.vh_at = self.sv_at + up(s_at)
        self.ws_at = self.vh_at + up(width * vh_at)
        self.size = max(self.ws_at + width * total, 1)
        # no wait for the stream's queued work (the window's Lanczos): the SVD is queued behind it
        self.table = _KeptTable(rows, torch.int64, device)
        self.ranking = _KeptTable([b[3] for b in self.blocks] + [ids[b[0].domain] for b in self.blocks] +
                                  [ids[cat.dual(sector)] for sector in sorted(ids, key = ids.get)], torch.int32, device)


def _split_layout(space: Space, device, dtype):
    '''The layout of the batched SVD, None when some block is too large for it.'''
    present = [(i, key) for i, key in enumerate(space.keys) if space.shapes[i][0] * space.shapes[i][1] > 0]
    count = len(present)
    if any(min(space.shapes[i]) > 1024 for i, _ in present):
        return None
    dims, _ = ints64(x for i, _ in present for x in space.shapes[i])
    places, total = (i64 * max(count, 1))(), i64()
    if dtype == torch.float64:
        check(lib.tt_svd_workspace(count, dims, places, ctypes.byref(total)))
        return _SplitLayout(space, device, present, places, total.value, 1)
    table, ranks = (i64 * max(8 * count, 1))(), i32()
    check(lib.tt_svd_complex_plan(count, dims, places, ctypes.byref(total), table, ctypes.byref(ranks)))
    if count and not ranks.value:
        return None
    return _SplitLayout(space, device, present, places, total.value, 2, (table, ranks.value))


class _SplitWrite:
    '''Where the kept factors of one space's split go: the two output spaces, the bond's multiplets and the device table of
    the kept blocks; `covered` when every entry of the outputs is written.'''
    __slots__ = ('first', 'second', 'multiplets', 'table', 'count', 'covered')

    def __init__(self, space: Space, layout: _SplitLayout, kept, absorb: int, device):
        cat = space.cat
        multiplicities, offsets = {}, []
        for (key, *_), n in zip(layout.blocks, kept):
            offsets.append(multiplicities.get(key.domain, 0))
            if n:
                multiplicities[key.domain] = offsets[-1] + n
        placed, at = {}, 0
        for sector in sorted(multiplicities):
            placed[sector] = at
            at += multiplicities[sector]
        bond = Leg.from_blocks(cat, sorted((multiplicities or {cat.trivial(): 1}).items()))[0]
        self.first = Space.of(cat, space.codomain, [bond], space.qtotal)
        self.second = Space.of(cat, [bond], space.domain, cat.trivial())
        self.multiplets = bond.multiplets()
        table, written = [], [0, 0]
        self.count = 0
        for (key, rows, cols, k, u_at, s_at, vh_at), n, offset in zip(layout.blocks, kept, offsets):
            if n == 0:
                continue
            fi = self.first.index[BlockKey(key.codomain, key.domain, key.copy)]
            si = self.second.index[BlockKey(key.domain, key.domain, 0)]
            table += [u_at, s_at, vh_at, self.first.offsets[fi], self.second.offsets[si], placed[key.domain] + offset,
                      rows | cols << 32, k | n << 32, self.first.shapes[fi][1] | offset << 32, offset | absorb << 32]
            written[0] += rows * n
            written[1] += n * cols
            self.count += 1
        self.covered = (self.count > 0 and written[0] == sum(m * n for m, n in self.first.shapes) and
                        written[1] == sum(m * n for m, n in self.second.shapes))
        self.table = _KeptTable(table, torch.int64, device)


# (space, device, dtype) -> its split's layout (None: not for the batched SVD); (space, kept counts, absorb, device)
# -> where its factors go
_split_layouts = {}
_split_writes = {}


def _remembered(cache: dict, key, make):
    found = cache.get(key, cache)
    if found is cache:
        found = make()
        if _capturing():  # its uploads are part of the graph: not for other calls
            return found
        if len(cache) >= _PLAN_BUDGET:
            cache.clear()
        cache[key] = found
    return found


def _split_batched(arranged: Tensor, max_bond, tol, absorb, while_waiting = None):
    """The split on the GPU: the engine's Jacobi SVD for all blocks (tt_svd_blocks; complex128 tt_svd_complex_blocks),
    the ranking of the values on the device (tt_svd_rank), one read of each block's kept count with the
    SVD's sweep counts, and one launch that writes the kept factors (tt_svd_keep).  Blocks that did not settle
    go through at::linalg_svd before the values are ranked again.  None when the blocks are not for it."""
    global svd_fallbacks
    space, data, dtype = arranged._space, arranged._data, arranged._data.dtype
    if not (data.is_cuda and _precision != PER_BLOCK and dtype in (torch.float64, torch.complex128)):
        return None
    device, index = data.device, data.get_device()
    layout = _remembered(_split_layouts, (space.id, index, dtype), lambda: _split_layout(space, device, dtype))
    if layout is None:
        return None
    buffer = torch.empty(layout.size, dtype = torch.float64, device = device)
    counts = torch.empty(max(layout.count + layout.n_blocks, 1), dtype = torch.int32, device = device)
    u = buffer.data_ptr()
    sv, vh, ws = u + 8 * layout.sv_at, u + 8 * layout.vh_at, u + 8 * layout.ws_at
    info, kept_at = counts.data_ptr(), counts.data_ptr() + 4 * layout.count
    stream = _raw_stream(index)
    table = layout.table.address(stream)
    if dtype == torch.float64:
        check(lib.tt_svd_blocks(layout.count, layout.largest, table, data.data_ptr(), u, sv, vh, ws, info, stream))
    elif layout.count:
        check(lib.tt_svd_complex_blocks(layout.count, layout.largest, layout.qr_ranks, table, table + 56 * layout.count, data.data_ptr(),
                                        u, sv, vh, ws, info, stream))
    ranking = layout.ranking.address(stream)

    def rank():
        # the host's ranking for splits too large for the kernel
        status = lib.tt_svd_rank(sv, layout.values, ranking, ranking + 4 * layout.n_blocks, layout.n_blocks,
                                 ranking + 8 * layout.n_blocks, layout.n_sectors, float(tol), -1 if max_bond is None else int(max_bond),
                                 kept_at, stream)
        if status not in (0, 1):
            check(status)
        return status

    status = rank()
    if while_waiting is not None:
        while_waiting()
    host = counts.tolist() if layout.count else []
    # (-2: complete but for the vectors of zero values, which a tolerance below zero alone keeps)
    unsettled = [layout.order[at] for at in range(layout.count) if host[at] < 0 and not (host[at] == -2 and tol >= 0)]
    if unsettled:
        svd_fallbacks += 1
        _factor_into(arranged, layout, buffer, unsettled)
        rank()
        host = counts.tolist()
    if status == 0:
        kept = tuple(host[layout.count:])
    else:
        kept = _ranked_on_host(arranged, layout, buffer[layout.sv_at:layout.sv_at + layout.values].tolist(), max_bond, tol)
    write = _remembered(_split_writes, (space.id, kept, absorb, index), lambda: _SplitWrite(space, layout, kept, absorb, device))
    # (the kernel writes the pads after odd blocks)
    make = torch.empty if write.covered else torch.zeros
    first, second, values = (make(n, dtype = dtype, device = device)
                             for n in (write.first.size, write.second.size, write.multiplets))
    if write.count:
        keep = lib.tt_svd_keep if dtype == torch.float64 else lib.tt_svd_complex_keep
        check(keep(write.count, write.table.address(stream), u, sv, vh, first.data_ptr(), second.data_ptr(), values.data_ptr(), stream))
    return Tensor._wrap(write.first, first), values, Tensor._wrap(write.second, second)


def _factor_into(arranged: Tensor, layout: _SplitLayout, buffer, blocks):
    '''at::linalg_svd of these blocks of the layout, into the packed factors.'''
    parts = [buffer[:layout.sv_at], buffer[layout.vh_at:layout.ws_at]]
    if arranged.dtype == torch.complex128:
        parts = [torch.view_as_complex(p.view(-1, 2)) for p in parts]
    for at in blocks:
        _, rows, cols, k, u_at, s_at, vh_at = layout.blocks[at]
        block = arranged._view(layout.present[at][0])
        # (LAPACK refuses such a block, cuSOLVER from three columns on; below it hands NaN values to the ranking)
        if not bool(torch.isfinite(block).all()):
            raise torch.linalg.LinAlgError('linalg.svd: the input matrix contained non-finite values')
        u, sv, vh = torch.linalg.svd(block, full_matrices = False, driver = PER_BLOCK_SVD_DRIVER)
        parts[0][u_at:u_at + rows * k].view(rows, k).copy_(u)
        buffer[layout.sv_at + s_at:layout.sv_at + s_at + k].copy_(sv)
        parts[1][vh_at:vh_at + k * cols].view(k, cols).copy_(vh)


def _ranked_on_host(arranged: Tensor, layout: _SplitLayout, values, max_bond, tol):
    '''The device ranking's kept counts, from the values on the host.'''
    factors = [[b[0], None, None, None, 0, 0] for b in layout.blocks]
    candidates, at = [], 0
    for fi, b in enumerate(layout.blocks):
        for i in range(b[3]):
            candidates.append((values[at], fi, i))
            at += 1
    _rank_candidates(factors, candidates, max_bond, tol, arranged.cat)
    return tuple(f[4] for f in factors)


def _split_over(tensor: Tensor, left, max_bond, tol, absorb, while_waiting = None):
    '''tentorch/linalg/graded/svd.cpp:41-177: the SVD of every block, the global ranking of the
    singular values, truncation and the +-q pairing of the bond (on the device for the engine's
    batched SVD: one read of each block's kept count), then the two factors.  `while_waiting`, when
    given, runs on the host once the split's device work is queued and before the split reads its
    results (host work of the caller's that needs no device result: it overlaps the SVD).'''
    if absorb not in (0, 1, 2, 3):
        raise ValueError(f'absorb has to be 0, 1, 2 or 3, got {absorb}')
    if max_bond is not None and max_bond < 1:
        raise ValueError(f'a bond needs at least one multiplet, got {max_bond}')
    arranged = tensor.place(left) if left is not None else tensor
    batched = _split_batched(arranged, max_bond, tol, absorb, while_waiting)
    if batched is not None:
        return batched
    present = [(i, key) for i, key in enumerate(arranged.keys()) if arranged._space.shapes[i][0] * arranged._space.shapes[i][1] > 0]
    factors, host = _factor_blocks_per_block(arranged, present, while_waiting)
    candidates, at = [], 0
    for fi, f in enumerate(factors):
        for index in range(f[2].numel()):
            candidates.append((host[at], fi, index))
            at += 1
    multiplicities = _rank_candidates(factors, candidates, max_bond, tol, arranged.cat)
    return _split_finish(arranged, factors, multiplicities, absorb)


def _rank_candidates(factors, candidates, max_bond, tol, cat):
    '''tentorch/linalg/graded/svd.cpp:68-118: the global ranking, truncation and +-q pairing of the
    bond over (value, block, index) candidates; sets each block's kept count f[4] and returns the
    bond's multiplets per domain sector.'''
    candidates.sort(key = lambda c: -c[0])
    cut = next((i for i, c in enumerate(candidates) if c[0] <= tol), len(candidates))
    candidates = candidates[:cut]
    if max_bond is not None and len(candidates) > max_bond:
        candidates = candidates[:max_bond]
    for _, fi, index in candidates:
        factors[fi][4] = max(factors[fi][4], index + 1)
    multiplicities = {}
    for f in factors:
        if f[4]:
            multiplicities[f[0].domain] = multiplicities.get(f[0].domain, 0) + f[4]
    paired = {}
    for sector, count in multiplicities.items():
        other = multiplicities.get(cat.dual(sector))
        if other is not None:
            paired[sector] = min(count, other)
    if paired and paired != multiplicities:
        for f in factors:
            f[4] = 0
        used = {}
        for _, fi, index in candidates:
            f = factors[fi]
            room = paired.get(f[0].domain)
            if room is None or used.get(f[0].domain, 0) >= room:
                continue
            used[f[0].domain] = used.get(f[0].domain, 0) + 1
            f[4] = max(f[4], index + 1)
        multiplicities = paired
    return multiplicities


def _split_finish(arranged: Tensor, factors, multiplicities, absorb):
    '''The bond of the split from its multiplets per domain sector, and the two factors and the
    values written block by block.'''
    cat = arranged.cat
    nxt = {}
    for f in factors:
        f[5] = nxt.get(f[0].domain, 0)
        nxt[f[0].domain] = f[5] + f[4]
    placed, run_at = {}, 0
    for sector in sorted(multiplicities):
        placed[sector] = run_at
        run_at += multiplicities[sector]
    if not multiplicities:
        multiplicities = {cat.trivial(): 1}
    bond = Leg.from_blocks(cat, sorted(multiplicities.items()))[0]
    first = Tensor(cat, arranged.codomain, [bond], arranged.qtotal, arranged.dtype, arranged.device)
    values = torch.zeros(bond.multiplets(), dtype = arranged.dtype, device = arranged.device)
    second = Tensor(cat, [bond], arranged.domain, cat.trivial(), arranged.dtype, arranged.device)
    for key, u, s, vh, kept, offset in factors:
        if kept == 0:
            continue
        u, vh, s = u[:, :kept], vh[:kept], s[:kept]
        if absorb == 3:
            u = u * s.sqrt()
            vh = s.sqrt().unsqueeze(1) * vh
        elif absorb == 1:
            u = u * s
        elif absorb == 2:
            vh = s.unsqueeze(1) * vh
        first.block(key.codomain, key.domain, key.copy)[:, offset:offset + kept].copy_(u)
        second.block(key.domain, key.domain)[offset:offset + kept, :].copy_(vh)
        values[placed[key.domain] + offset:placed[key.domain] + offset + kept].copy_(s.to(arranged.dtype))
    return first, values, second


def svd(tensor: Tensor, *args, **kwargs):
    '''svd(tensor, max_bond=None, tol=0.0, absorb=0) or svd(tensor, left, max_bond=None, tol=0.0,
    absorb=0) -> (first, values, second): the two overloads of tentorch/_ext/bindings.cpp:365-382.'''
    left = None
    if args and isinstance(args[0], (list, tuple)):
        left, args = list(args[0]), args[1:]
    elif 'left' in kwargs:
        left = kwargs.pop('left')
    params = {'max_bond': None, 'tol': 0.0, 'absorb': 0}
    for name, value in zip(('max_bond', 'tol', 'absorb'), args):
        params[name] = value
    for name, value in kwargs.items():
        if name not in params:
            raise TypeError(f'svd() got an unexpected keyword argument {name!r}')
        params[name] = value
    return _split_over(tensor, left, params['max_bond'], params['tol'], params['absorb'])


def svdvals(tensor: Tensor, left = None) -> torch.Tensor:
    return _split_over(tensor, left, None, 0.0, 0)[1]


def _split_blocks(tensor: Tensor, pieces):
    '''tentorch/linalg/graded/svd.cpp:203-229'''
    cat = tensor.cat
    multiplicities, nxt, placed = {}, {}, []
    for key, left, right, kept in pieces:
        if kept == 0:
            continue
        offset = nxt.get(key.domain, 0)
        nxt[key.domain] = offset + kept
        multiplicities[key.domain] = multiplicities.get(key.domain, 0) + kept
        placed.append((key, left, right, kept, offset))
    if not multiplicities:
        multiplicities = {cat.trivial(): 1}
    bond = Leg.from_blocks(cat, sorted(multiplicities.items()))[0]
    first = Tensor(cat, tensor.codomain, [bond], tensor.qtotal, tensor.dtype, tensor.device)
    second = Tensor(cat, [bond], tensor.domain, cat.trivial(), tensor.dtype, tensor.device)
    for key, left, right, kept, offset in placed:
        first.block(key.codomain, key.domain, key.copy)[:, offset:offset + kept].copy_(left)
        second.block(key.domain, key.domain)[offset:offset + kept, :].copy_(right)
    return first, second


# (space, rows or columns first, dtype, device) -> the batched QR of a tensor of that space: its two
# output spaces, the device table, workspace elements and cluster size; None where a block
# does not fit or cuSOLVER, block by block, is faster (csrc/qr.cu qr_pays)
_qr_plans = {}


def _qr_plan(arranged: Tensor, transposed: bool):
    space, device = arranged._space, arranged.device
    key = (space.id, transposed, arranged.dtype, device.index)
    if key in _qr_plans:
        return _qr_plans[key]
    if _capturing():  # a table uploaded now would be the graph's: the blocks go one by one
        return None
    cat = space.cat
    present = [(i, k) for i, k in enumerate(space.keys) if space.shapes[i][0] * space.shapes[i][1] > 0]
    multiplicities, offsets = {}, []
    for i, k in present:
        offsets.append(multiplicities.get(k.domain, 0))
        multiplicities[k.domain] = offsets[-1] + min(space.shapes[i])
    bond = Leg.from_blocks(cat, sorted((multiplicities or {cat.trivial(): 1}).items()))[0]
    first = Space.of(cat, space.codomain, [bond], space.qtotal)
    second = Space.of(cat, [bond], space.domain, cat.trivial())
    # the matrix factored is the block, or its transpose
    shapes, count = ints64(x for i, _ in present for x in (reversed(space.shapes[i]) if transposed else space.shapes[i]))
    places, total, ranks = (i64 * max(len(present), 1))(), i64(), i32()
    check(lib.tt_qr_plan(_DTYPE[arranged.dtype], len(present), shapes, places, ctypes.byref(total), ctypes.byref(ranks)))
    plan = None
    if ranks.value and max([s for i, _ in present for s in space.shapes[i]] + list(multiplicities.values()), default = 0) < 2 ** 31:
        table = []
        for at, ((i, k), offset) in enumerate(zip(present, offsets)):
            rows, cols = space.shapes[i]
            fi, si = first.index[BlockKey(k.codomain, k.domain, k.copy)], second.index[BlockKey(k.domain, k.domain, 0)]
            ld = first.shapes[fi][1]
            head, tail = first.offsets[fi] + offset, second.offsets[si] + offset * cols
            if transposed:  # Q^T goes to the second factor, R^T to the first
                entry, strides = (space.offsets[i], tail, head), (cols, rows, 1, cols, 1, cols, 1, ld)
            else:
                entry, strides = (space.offsets[i], head, tail), (rows, cols, cols, 1, ld, 1, cols, 1)
            table += [*entry, places[at], *(strides[s] | strides[s + 1] << 32 for s in range(0, 8, 2))]
        plan = (len(present), first, second, _KeptTable(table, torch.int64, device), total.value, ranks.value)
    if len(_qr_plans) >= _PLAN_BUDGET and not _captured:
        _qr_plans.clear()
    _qr_plans[key] = plan
    return plan


def _qr_blocks(arranged: Tensor, transposed: bool):
    '''Every block factored in one launch straight into the two output arenas, or None when the tensor is not on
    a CUDA device or the plan is not to (then the blocks are factored one by one).'''
    if arranged.device.type != 'cuda' or _precision == PER_BLOCK:
        return None
    plan = _qr_plan(arranged, transposed)
    if plan is None:
        return None
    count, first, second, table, total, ranks = plan
    data = arranged._data
    stream = _raw_stream(data.get_device())
    if _capturing():
        _note_capture()
    # zeros: what no block covers (and the pads after odd blocks) is part of the factors
    out = [torch.zeros(s.size, dtype = data.dtype, device = data.device) for s in (first, second)]
    if count:
        ws = torch.empty(total, dtype = data.dtype, device = data.device)
        q, r = (out[1], out[0]) if transposed else (out[0], out[1])
        check(lib.tt_qr_blocks(_DTYPE[data.dtype], count, ranks, table.address(stream), data.data_ptr(), q.data_ptr(), r.data_ptr(),
                               ws.data_ptr(), stream))
    return Tensor._wrap(first, out[0]), Tensor._wrap(second, out[1])


def qr(tensor: Tensor, left = None):
    '''tentorch/linalg/graded/svd.cpp:233-244'''
    arranged = tensor.place(left) if left is not None else tensor
    factors = _qr_blocks(arranged, False)
    if factors is not None:
        return factors
    pieces = []
    for i, key in enumerate(arranged.keys()):
        matrix = arranged._view(i)
        if matrix.numel() == 0:
            continue
        q, r = torch.linalg.qr(matrix, mode = 'reduced')
        pieces.append((key, q, r, q.shape[1]))
    return _split_blocks(arranged, pieces)


def rq(tensor: Tensor, left = None):
    '''tentorch/linalg/graded/svd.cpp:246-257'''
    arranged = tensor.place(left) if left is not None else tensor
    factors = _qr_blocks(arranged, True)
    if factors is not None:
        return factors
    pieces = []
    for i, key in enumerate(arranged.keys()):
        matrix = arranged._view(i)
        if matrix.numel() == 0:
            continue
        q, r = torch.linalg.qr(matrix.transpose(0, 1), mode = 'reduced')
        pieces.append((key, r.transpose(0, 1), q.transpose(0, 1), q.shape[1]))
    return _split_blocks(arranged, pieces)
