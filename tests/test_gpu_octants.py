"""Products shorter than their transform: the passes leave out the octants that the
coefficients do not need, and the inverse column pass solves for the rest. Every
octant count (5 to 8 eighths of the transform), one coefficient below, at and above
each edge, in every column kernel, against the oracle; residues that the largest
limbs make (all ones) against their closed form."""
import os

import numpy as np
import pytest

import oracle
from nttanafis_gb300.operands import operand

pytestmark = pytest.mark.gpu
MASK = (1 << 64) - 1
THREADS = os.cpu_count() or 1


def all_ones_product(la: int, lb: int) -> np.ndarray:
    """Limbs of (B^la - 1)(B^lb - 1)."""
    left, right = max(la, lb), min(la, lb)
    out = np.zeros(la + lb, dtype=np.uint64)
    out[0] = 1
    out[right:] = MASK
    out[left] = MASK - 1
    return out


def lengths(log_t: int):
    """(la, lb) whose coefficient counts sit at the octant edges of 2^log_t points."""
    t = 1 << log_t
    for l in (5, 6, 7, 8):
        for n in (l * t // 8 - 1, l * t // 8, l * t // 8 + 1 if l < 8 else l * t // 8 - t // 16):
            lb = n // 2 - n // 11  # 41% of the coefficients: no block split
            yield n + 1 - lb, lb


@pytest.fixture(scope="module")
def ws(gpu):
    w = gpu.GpuMulWorkspace()
    yield w
    w.close()


def product(gpu, ws, a, b):
    dst = np.full(a.size + b.size + 1, MASK, dtype=np.uint64)
    ok = ws.sqr(dst, a) if b is a else ws.mul(dst, a, b)
    assert ok, gpu.last_error()
    assert dst[-1] == MASK, "suffix was overwritten"
    return dst[:-1]


@pytest.mark.parametrize("log_t,log_r", [(13, 0), (14, 6), (14, 7), (15, 8), (16, 9), (17, 10), (18, 11), (20, 10)])
def test_octant_edges_in_every_lazy_column_kernel(gpu, ws, log_t, log_r):
    previous = gpu.set_split(log_t, log_r) if log_r else None
    try:
        for i, (la, lb) in enumerate(lengths(log_t)):
            assert gpu.MulPlan.new(la, lb).log_transform == log_t
            a, b = operand(la, 11 + i), operand(lb, 31 + i)
            assert np.array_equal(product(gpu, ws, a, b), oracle.mul(a, b, THREADS)), (la, lb)
            a, b = np.full(la, MASK, np.uint64), np.full(lb, MASK, np.uint64)
            assert np.array_equal(product(gpu, ws, a, b), all_ones_product(la, lb)), (la, lb)
    finally:
        if log_r:
            gpu.set_split(log_t, previous)


# the splits that lone products run while none is set, and the 2^10-point columns of
# lengths whose default is another
@pytest.mark.parametrize("log_t,log_r", [(14, 6), (15, 6), (16, 6), (17, 7), (18, 8), (19, 9), (20, 8), (21, 9),
                                         (18, 10), (19, 10)])
def test_octant_edges_of_the_lone_defaults(gpu, ws, log_t, log_r):
    if gpu.lone_split(log_t) != log_r:
        gpu.set_split(log_t, log_r)
    try:
        assert gpu.lone_split(log_t) == log_r
        test_octant_edges_in_every_lazy_column_kernel(gpu, ws, log_t, 0)
    finally:
        gpu.set_split(log_t, 0)


@pytest.mark.parametrize("log_t,octants", [(22, 5), (22, 7), (23, 6), (24, 5), (24, 6), (24, 7), (25, 5)])
def test_octants_of_the_wide_lengths(gpu, ws, log_t, octants):
    n = octants * (1 << log_t) // 8
    lb = n // 2 - 3
    la = n + 1 - lb
    assert gpu.MulPlan.new(la, lb).log_transform == log_t
    a, b = np.full(la, MASK, np.uint64), np.full(lb, MASK, np.uint64)
    assert np.array_equal(product(gpu, ws, a, b), all_ones_product(la, lb))
    if log_t <= 24:
        a, b = operand(la, 5), operand(lb, 6)
        assert np.array_equal(product(gpu, ws, a, b), oracle.mul(a, b, THREADS))


@pytest.mark.parametrize("log_t", [15, 19])
def test_octants_of_squares_and_convolutions(gpu, ws, log_t):
    cws = gpu.GpuConvWorkspace()
    for octants in (5, 6, 7):
        n = octants * (1 << log_t) // 8
        a = operand(n // 2, 7)
        assert np.array_equal(product(gpu, ws, a, a), oracle.sqr(a, THREADS))
        la, lb = n - 999, 1000
        a, b = operand(la, 8) & np.uint64(0xFFFF), operand(lb, 9) & np.uint64(0xFFFF)
        plan = gpu.ConvPlan.new(la, lb, 0xFFFF, 0xFFFF)
        assert cws.prepare(plan)
        dst = np.zeros(plan.output_len(), dtype=np.uint64)
        assert cws.convolve(dst, a, b)
        assert np.array_equal(dst, oracle.conv(a, b, 0xFFFF, 0xFFFF, False, THREADS)), octants
    cws.close()


def test_batch_members_of_every_octant_count_in_one_class(gpu):
    import torch

    rows = list(lengths(15)) + [(1 << 14, 1 << 14)]
    host = [(operand(la, 60 + i), operand(lb, 90 + i)) for i, (la, lb) in enumerate(rows)]
    dev = [[torch.from_numpy(x.view(np.int64)).cuda() for x in pair] for pair in host]
    dst = [torch.full((la + lb,), -1, dtype=torch.int64, device="cuda") for la, lb in rows]
    batch = gpu.GpuBatch()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(9):  # direct runs, tuning runs, and the captured graph
        assert batch.run([gpu.Request(d, a, b) for d, (a, b) in zip(dst, dev)], stream), gpu.last_error()
    stream.synchronize()
    assert batch.status() == 0
    for d, (a, b) in zip(dst, host):
        assert np.array_equal(d.cpu().numpy().view(np.uint64), oracle.mul(a, b, THREADS)), (a.size, b.size)
    batch.close()


def test_wide_plan_call_with_scratch_off_the_16_byte_boundary(gpu):
    # the persistent inverse column pass copies 16 bytes at a time; such a scratch
    # takes the kernel that reads word by word
    import torch

    la, lb = 5 << 20, (5 << 20) - 7  # 2^24 points, five octants
    plan = gpu.MulPlan.new(la, lb)
    assert plan.log_transform == 24
    scratch = torch.zeros(plan.scratch_len() + 1, dtype=torch.int64, device="cuda")[1:]
    a, b = (torch.full((n,), -1, dtype=torch.int64, device="cuda") for n in (la, lb))
    want = torch.from_numpy(all_ones_product(la, lb).view(np.int64)).cuda()
    for _ in range(16):  # a race between a CTA's warps shows in some runs only
        dst = torch.zeros(la + lb, dtype=torch.int64, device="cuda")
        assert plan.mul_device(dst, a, b, scratch, torch.cuda.current_stream()), gpu.last_error()
        torch.cuda.synchronize()
        assert torch.equal(dst, want)


def test_wide_block_split_with_scratch_off_the_16_byte_boundary(gpu):
    # blocks of 2^24 points, whose residues lie in the caller's scratch
    import torch

    la, lb = 40_000_000, 2_000_000
    plan = gpu.MulPlan.new(la, lb)
    assert plan.blocks > 1 and plan.log_transform == 24
    scratch = torch.zeros(plan.scratch_len() + 1, dtype=torch.int64, device="cuda")[1:]
    assert scratch.data_ptr() % 16 == 8
    a, b = (torch.full((n,), -1, dtype=torch.int64, device="cuda") for n in (la, lb))
    dst = torch.zeros(la + lb, dtype=torch.int64, device="cuda")
    for x, y in ((a, b), (b, a)):
        dst.zero_()
        plan = gpu.MulPlan.new(x.numel(), y.numel())
        assert plan.mul_device(dst, x, y, scratch, torch.cuda.current_stream()), gpu.last_error()
        torch.cuda.synchronize()
        assert torch.equal(dst, torch.from_numpy(all_ones_product(la, lb).view(np.int64)).cuda())
