'''The forms the autotuner stores reach every product of a plan: with FORM_NO_TENSOR_CORES both products of the
two-site matvec run on mma.sync, the first one, which stores through the leg move, too.'''
import os
import subprocess
import sys

import pytest
import torch

import tentorch_gb300 as tg
from tentorch_gb300 import linalg as la
from oracle import engine as orc

pytestmark = pytest.mark.gpu


def operands():
    '''Head, tail and theta of a window of bond 288 without symmetry: one block each, K = 576 in both products, more
    than one chunk of exact sums in either kernel, whose chunks differ.'''
    cat = tg.no_symmetry
    bond, phys, w = (tg.Leg(cat, [(0,)], [n]) for n in (288, 2, 5))
    gen = torch.Generator().manual_seed(5)
    tensors = []
    for codomain, domain in (([bond, phys], [bond, phys, w]), ([w, phys, phys, bond], [bond]), ([bond, phys], [phys, bond])):
        t = tg.Tensor(cat, codomain, domain, (0,), dtype = torch.float64, device = 'cuda')
        t.data.copy_(torch.randn(t.data.numel(), dtype = torch.float64, generator = gen))
        tensors.append(t)
    return tensors


def product():
    with tg.precision(8):
        return tg.einsum(orc.MATVEC, *operands()).data.cpu()


def test_without_tensor_cores_is_mma_sync_throughout(tmp_path):
    '''The kernels fold their level sums after different chunks of K, so their results differ in the last bits: the
    stored form gives those of a process with the tensor cores switched off.'''
    here = os.path.dirname(os.path.abspath(__file__))
    path = str(tmp_path / 'product.pt')
    code = f'import sys; sys.path[:0] = [{os.path.dirname(here)!r}, {here!r}]; import torch, test_gpu_forms as f; torch.save(f.product(), {path!r})'
    subprocess.run([sys.executable, '-c', code], check = True, env = {**os.environ, 'TENTORCH_GB300_TCGEN05': '0'})
    off = torch.load(path)
    with tg.precision(8):
        plan = la.plan_of(orc.MATVEC, *operands())
    assert plan.describe().startswith('chain ops')
    la.clear_tuning()
    try:
        on = product()
        with tg.precision(8):
            la.store_forms(plan, la.FORM_NO_TENSOR_CORES)
        stored = product()
    finally:
        la.clear_tuning()
    assert not torch.equal(on, off)
    assert torch.equal(stored, off)
