"""Products enqueued back to back on one stream without a synchronisation: every
kernel may be scheduled before the one ahead of it has finished, so each product of a
chain reads the product before it, overwrites its operands' buffers, and shares its
scratch. The same chain runs from a CUDA graph."""
import numpy as np
import pytest

import oracle
from nttanafis_gb300.operands import operand

pytestmark = pytest.mark.gpu


def chain(gpu, torch, ws, x, sizes, stream):
    """x -> x * x cut to the next size, through the sizes; every buffer it made."""
    made = [x]
    for n in sizes:
        a = made[-1]
        dst = torch.empty(2 * a.numel(), dtype=torch.int64, device="cuda")
        b = a.flip(0)  # a copy by another kernel, in front of the product
        assert ws.mul_device(dst, a, b, stream), gpu.last_error()
        made.append(dst[:n].clone())
    return made


def expected(x, sizes):
    for n in sizes:
        x = oracle.mul(x, np.ascontiguousarray(x[::-1]), 4)[:n]
    return x


# the basecase (1 CTA and clusters), the fused one-CTA transforms, the four-step
# sequence with and without unneeded octants, in both directions of size
SIZES = [40, 80, 150, 290, 570, 1100, 2200, 4300, 8600, 17000, 33000, 65536, 65536, 30000, 5000, 900, 90, 30]


def test_dependent_products_on_one_stream(gpu):
    import torch

    ws = gpu.GpuMulWorkspace()
    x = operand(20, 3)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        dev = torch.from_numpy(x.view(np.int64)).cuda()
        ws.mul_device(torch.empty(2 * 65536, dtype=torch.int64, device="cuda"),
                      *[torch.zeros(65536, dtype=torch.int64, device="cuda")] * 2, stream)  # the largest arena
        results = [chain(gpu, torch, ws, dev, SIZES, stream)[-1] for _ in range(3)]
    stream.synchronize()
    want = expected(x, SIZES)
    for got in results:
        assert np.array_equal(got.cpu().numpy().view(np.uint64), want)
    assert ws.status() == 0
    ws.close()


def test_dependent_products_captured_in_a_graph(gpu):
    import torch

    ws, cws = gpu.GpuMulWorkspace(), gpu.GpuConvWorkspace()
    x = operand(20, 5)
    la, lb = 3000, 2000
    u = torch.from_numpy((operand(la, 6) & np.uint64(0xFFFF)).view(np.int64)).cuda()
    v = torch.from_numpy((operand(lb, 7) & np.uint64(0xFFFF)).view(np.int64)).cuda()
    plan = gpu.ConvPlan.new(la, lb, 0xFFFF, 0xFFFF)
    assert cws.prepare(plan)
    conv = torch.empty(plan.output_len(), dtype=torch.int64, device="cuda")
    dev = torch.from_numpy(x.view(np.int64)).cuda()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):  # arenas and tables before the capture
        ws.mul_device(torch.empty(2 * 65536, dtype=torch.int64, device="cuda"),
                      *[torch.zeros(65536, dtype=torch.int64, device="cuda")] * 2, stream)
        chain(gpu, torch, ws, dev, SIZES, stream)
        assert cws.convolve_device(conv, u, v, stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        made = chain(gpu, torch, ws, dev, SIZES, torch.cuda.current_stream())
        assert cws.convolve_device(conv, u, v, torch.cuda.current_stream())
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(made[-1].cpu().numpy().view(np.uint64), expected(x, SIZES))
    assert np.array_equal(conv.cpu().numpy().view(np.uint64),
                          oracle.conv(u.cpu().numpy().view(np.uint64), v.cpu().numpy().view(np.uint64), 0xFFFF, 0xFFFF))
    del graph
    ws.close()
    cws.close()


# block splits on one-CTA blocks (2^11..2^13 points), on four-step ones and in more than
# one chunk of blocks, either operand the longer one, beside unsplit products
LONGEST = (30_000_000, 3000)
SPLITS = [(1 << 20, 1000), (4096, 4096), (3001, 1 << 20), (600000, 20000), (200000, 1000), (1 << 20, 100003),
          (65536, 65536), LONGEST, (1 << 20, 1000), (100003, 600000), (700, 600), (1 << 18, 300)]


def test_dependent_block_splits_on_one_stream(gpu):
    import torch

    plans = [gpu.MulPlan.new(la, lb) for la, lb in SPLITS]
    split = {p.log_transform for p in plans if p.blocks}
    assert min(split) < 13 < max(split)
    longest = gpu.MulPlan.new(*LONGEST)
    assert longest.blocks * (20 << longest.log_transform) > 512 << 20  # above one chunk's arena
    pool = torch.from_numpy(operand(LONGEST[0], 17).view(np.int64)).cuda()
    pairs = [(pool[:la], pool[-lb:]) for la, lb in SPLITS]
    outs = [[torch.full((la + lb,), -1, dtype=torch.int64, device="cuda") for la, lb in SPLITS] for _ in range(4)]
    scratch = torch.full((max(p.scratch_len() for p in plans),), 0x5A5A5A5A5A5A5A5A, dtype=torch.int64, device="cuda")
    ws = gpu.GpuMulWorkspace()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for dsts in outs[:2]:  # the workspace's scratch, which every product overwrites
        for dst, (a, b) in zip(dsts, pairs):
            assert ws.mul_device(dst, a, b, stream), gpu.last_error()
    for dsts in outs[2:]:  # a caller's scratch
        for dst, (a, b), plan in zip(dsts, pairs, plans):
            assert plan.mul_device(dst, a, b, scratch, stream), gpu.last_error()
    stream.synchronize()
    assert ws.status() == 0
    for k, (a, b) in enumerate(pairs):
        x, y = (v.cpu().numpy().view(np.uint64) for v in (a, b))
        want = torch.from_numpy(oracle.mul(x, y, 16).view(np.int64)).cuda()
        for dsts in outs:
            assert torch.equal(dsts[k], want), SPLITS[k]
    ws.close()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("la,lb", [(40, 40), (1000, 731), (4000, 4000), (20000, 6007), (300000, 200000), (1 << 20, 1000)])
def test_an_operand_that_arrives_by_an_event(gpu, la, lb, captured):
    # the product's first kernel is launched dependently on the product before it in its
    # stream, and must still wait for the other stream's event
    import torch

    ws = gpu.GpuMulWorkspace()
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    x, y = operand(la, 3), operand(lb, 4)
    src, b = (torch.from_numpy(v.view(np.int64)).cuda() for v in (x, y))
    a = torch.zeros_like(src)
    before, dst = (torch.empty(n, dtype=torch.int64, device="cuda") for n in (la + 2 * lb, la + lb))

    def work():
        assert ws.mul_device(before, a, b, main), gpu.last_error()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            torch.cuda._sleep(400_000)  # a fifth of a millisecond
            a.copy_(src)
        assert ws.mul_device(before, b, b, main), gpu.last_error()
        main.wait_stream(side)
        assert ws.mul_device(dst, a, b, main), gpu.last_error()
        with torch.cuda.stream(main):
            a.zero_()

    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        work()
    main.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            work()
    want = torch.from_numpy(oracle.mul(x, y, 4).view(np.int64)).cuda()
    for _ in range(5):
        dst.fill_(-1)
        torch.cuda.synchronize()
        if captured:
            graph.replay()
        else:
            work()
        torch.cuda.synchronize()
        assert torch.equal(dst, want)
    if captured:
        del graph
    ws.close()
