'''Splits and QR of one space on several streams: the tables of the first call are kept, and a call on another stream
may come before their upload has run (here the first stream is held up).'''
import threading
import time

import pytest
import torch

import tentorch_gb300 as tg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [torch.float64, torch.complex128])
def test_a_second_stream_waits_for_the_kept_tables(dtype):
    cat, sizes = tg.su2, [(5, 7), (9, 4), (12, 12)]
    legs = [tg.Leg(cat, [(i,) for i in range(3)], [s[side] for s in sizes]) for side in (0, 1)]
    gen = torch.Generator().manual_seed(11)
    tensors = []
    for _ in range(2):
        t = tg.Tensor(cat, [legs[0]], [legs[1]], (0,), dtype = dtype, device = 'cuda')
        for i, (m, n) in enumerate(sizes):
            t.block((i,), (i,)).copy_(torch.randn(m, n, dtype = dtype, generator = gen))
        tensors.append(t)
    tg.linalg.clear_plans()
    torch.cuda.synchronize()
    results = [None, None]

    def factor(at, held_up):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            if held_up:
                torch.cuda._sleep(200_000_000)  # some 100 ms
            results[at] = (tg.qr(tensors[at]), tg.svd(tensors[at], None, 0.0))
        stream.synchronize()

    first = threading.Thread(target = factor, args = (0, True))
    first.start()
    time.sleep(0.03)  # its tables are made, their uploads wait behind the held stream
    factor(1, False)
    first.join()
    for t, ((q_of, r_of), (_, values, _)) in zip(tensors, results):
        for i, (m, n) in enumerate(sizes):
            b, q, r = (f.block((i,), (i,)) for f in (t, q_of, r_of))
            # 8 n eps of the block's norm (below 25)
            assert (q @ r - b).abs().max() < 8 * 12 * 2.0 ** -52 * 25
        total = sum(float(t.block((i,), (i,)).abs().square().sum()) for i in range(3))
        assert abs(float(values.abs().square().sum()) - total) < 8 * 12 * 2.0 ** -52 * total * 12
