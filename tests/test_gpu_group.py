"""Grouped queries on the tensor-core kernel (compute_group.cuh) against the CPU oracle (a few
heads) and the general kernel (all heads), at the edges of its tiles, chunks and work split.
Tolerances: helpers.RTOL / helpers.ATOL for both, as for every other attention kernel."""
import numpy as np
import pytest

from helpers import CpuHeads, assert_close

pytestmark = pytest.mark.gpu

SMS = 148
CHUNK = {1: 2048, 2: 1536}  # tokens between softmaxes, by column tiles (two queries each)


def plan(heads, n, nq):
    """launch_group's split: (column tiles, tokens of the longest piece of a head that one group walks)."""
    nt = 1 if nq <= 2 else 2
    items = heads * -(-nq // (2 * nt))
    if heads * nq > 16384:  # more queries than arrival counters: whole heads
        return nt, n
    units = -(-n // 64)
    total = items * units
    runs = 2 * max(1, min(SMS, total // (2 * max(4, units // 16))))
    longest = 0
    for r in range(runs):
        u, end = r * total // runs, (r + 1) * total // runs
        while u < end:
            cnt = min(units - u % units, end - u)
            longest = max(longest, min(n, (u % units + cnt) * 64) - u % units * 64)
            u += cnt
    return nt, longest


# dim, k_bits, v_bits, tokens, queries per head, capacity (0: tokens), heads (0: just above the size where the
# kernel is considered), several chunks in one piece of a head
CASES = [
    (128, 4, 2, 2, 4, 0, 0, False),        # two tokens; more queries than arrival counters, so heads stay whole
    (128, 4, 4, 17, 3, 0, 0, False),       # one row past a tile of 16
    (64, 2, 3, 33, 5, 0, 0, False),        # one past the V stream's 32; two query groups, 3 + 2
    (128, 3, 3, 64, 2, 0, 0, False),       # exactly one unit of the split
    (64, 4, 4, 65, 8, 0, 0, False),
    (128, 2, 4, 127, 7, 0, 0, False),
    (64, 3, 2, 129, 4, 0, 0, False),       # one past a stage
    (128, 4, 3, 1536, 4, 0, 400, False),   # exactly one chunk of three and four queries
    (64, 4, 2, 1537, 6, 0, 200, True),     # one past it
    (128, 2, 2, 2049, 2, 0, 400, True),    # one past the chunk of two
    (64, 2, 2, 3001, 4, 0, 0, False),      # 2-bit keys at 64: not a shape of the streaming kernel
    (128, 3, 2, 40000, 3, 0, 20, True),    # few heads, many pieces each
    (64, 3, 4, 1100, 2, 1024, 1300, False),  # wrapped ring
    (96, 4, 2, 700, 4, 0, 300, False),       # padded dimension
    (64, 4, 2, 2100, 8, 0, 2100, True),    # whole heads longer than a chunk
]


def fill(torch, gen, ctx, n, heads, dim):
    """n tokens of normal values, 0.2 % of the keys ten times larger; returns the rows of heads 0, middle and last."""
    pick, rows, step = [0, heads // 2, heads - 1], [], max(1, 2**27 // (heads * dim))
    for t in range(0, n, step):
        k, v = (torch.randn((min(step, n - t), heads, dim), device="cuda", generator=gen) for _ in range(2))
        k[torch.rand(k.shape, device="cuda", generator=gen) < 0.002] *= 10
        ctx.append_all(k, v)
        rows.append((k[:, pick].cpu().numpy(), v[:, pick].cpu().numpy()))
    return pick, [np.concatenate(r) for r in zip(*rows)]


def general(gpu_lib, ctx, q):
    try:
        gpu_lib.adaptq_set_kernel_policy(1)
        return ctx.compute_all(q)
    finally:
        gpu_lib.adaptq_set_kernel_policy(0)


@pytest.mark.parametrize("dim,kb,vb,n,nq,cap,heads,chunks", CASES)
def test_grouped_queries(gpu_lib, orc, dim, kb, vb, n, nq, cap, heads, chunks):
    import torch
    from adaptq_b200 import MHAContext
    padded = 64 if dim == 64 else 128
    live = min(n, cap or n)
    row = padded * (kb + vb) // 8 + 8
    heads = heads or max(3, int((80e6 if nq == 2 else 40e6) / (nq * live * row)) + 1)
    if torch.cuda.get_device_properties(0).multi_processor_count == SMS:
        nt, longest = plan(heads, live, nq)
        assert (longest > CHUNK[nt]) == chunks
    gen = torch.Generator(device="cuda").manual_seed(dim + 7 * kb + 11 * vb + n)
    seeds = [(42 ^ (i % 5)) for i in range(heads)]
    ctx = MHAContext(heads, dim, kb, vb, cap or n, v_mass=0.0, hybrid_thresh=0, seeds=seeds)
    pick, (k, v) = fill(torch, gen, ctx, n, heads, dim)
    q = torch.randn((heads, nq, dim), device="cuda", generator=gen)
    before = gpu_lib.adaptq_kernel_launches()
    out = ctx.compute_all(q)
    assert gpu_lib.adaptq_last_attention_kernel() == b"group"
    assert gpu_lib.adaptq_kernel_launches() - before == 1, "one launch for all queries"
    assert torch.equal(out, ctx.compute_all(q)), "integer sums: the same bits every time"
    ctx.synchronize()
    cpu = CpuHeads(orc, 3, dim, kb, vb, cap or n, 0, seeds=[seeds[i] for i in pick])
    cpu.append_many(k, v)
    assert_close(out[pick].cpu().numpy(), cpu.compute_batch(q[pick].cpu().numpy()), "against the oracle")
    assert_close(out.cpu().numpy(), general(gpu_lib, ctx, q).cpu().numpy(), "against the general kernel")


@pytest.mark.parametrize("nq", [2, 3])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("vb", [2, 3, 4])
@pytest.mark.parametrize("kb", [2, 3, 4])
def test_every_instantiation_over_several_chunks(gpu_lib, kb, vb, dim, nq):
    """Pieces longer than a chunk: the running maximum, the rescaled accumulator and stages carried over."""
    import torch
    from adaptq_b200 import MHAContext
    heads, n = 360, 3001
    if torch.cuda.get_device_properties(0).multi_processor_count == SMS:
        nt, longest = plan(heads, n, nq)
        assert longest > CHUNK[nt]
    gen = torch.Generator(device="cuda").manual_seed(dim + 7 * kb + 11 * vb)
    ctx = MHAContext(heads, dim, kb, vb, n, seed=5, v_mass=0.0, hybrid_thresh=0)
    fill(torch, gen, ctx, n, heads, dim)
    q = torch.randn((heads, nq, dim), device="cuda", generator=gen)
    out = ctx.compute_all(q)
    assert gpu_lib.adaptq_last_attention_kernel() == b"group"
    ctx.synchronize()
    assert_close(out.cpu().numpy(), general(gpu_lib, ctx, q).cpu().numpy(), "against the general kernel")


def test_without_room_for_pieces_heads_stay_whole(gpu_lib):
    """No memory for the pieces' partials, or a stream capture under way that forbids allocating them."""
    import torch
    from adaptq_b200 import MHAContext
    heads, dim, n, nq = 100, 128, 1700, 4
    gen = torch.Generator(device="cuda").manual_seed(8)
    made = lambda: MHAContext(heads, dim, 4, 2, n, seed=5, v_mass=0.0, hybrid_thresh=0)  # noqa: E731
    k, v = (torch.randn((n, heads, dim), device="cuda", generator=gen) for _ in range(2))
    q = torch.randn((heads, nq, dim), device="cuda", generator=gen)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ctx, refused, captured = made(), made(), made()
        for c in (ctx, refused, captured):
            c.append_all(k, v)
        want = ctx.compute_all(q)
        assert gpu_lib.adaptq_last_attention_kernel() == b"group"
        ref = general(gpu_lib, ctx, q)
        gpu_lib.adaptq_inject_failure(1, 1)
        try:
            got = refused.compute_all(q)
        finally:
            gpu_lib.adaptq_inject_failure(1, 0)
        assert gpu_lib.adaptq_last_attention_kernel() == b"group" and gpu_lib.adaptq_last_error() == b""
        again = refused.compute_all(q)  # now there is room
        refused.synchronize()
        out = torch.empty_like(q)
        graph = torch.cuda.CUDAGraph()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            captured.compute_all(q, out=out)
        assert gpu_lib.adaptq_last_attention_kernel() == b"group"
        graph.replay()
        first = out.clone()
        out.zero_()
        graph.replay()
    torch.cuda.synchronize()
    captured.synchronize()
    assert torch.equal(again, want) and torch.equal(first, got) and torch.equal(out, got)
    for o in (want, got):
        assert_close(o.cpu().numpy(), ref.cpu().numpy(), "against the general kernel")


def test_grouped_queries_non_finite(gpu_lib):
    """A NaN query gives NaN outputs for itself alone; an infinite value row for its head alone; a
    zero query averages."""
    import torch
    from adaptq_b200 import MHAContext
    heads, dim, n, nq = 300, 128, 400, 4
    gen = torch.Generator(device="cuda").manual_seed(3)
    k, v, q = (torch.randn(s, device="cuda", generator=gen) for s in ((n, heads, dim), (n, heads, dim), (heads, nq, dim)))
    v[7, 1] = float("inf")
    q[0, 2] = 0.0
    ctx = MHAContext(heads, dim, 4, 2, n, seed=1, v_mass=0.0, hybrid_thresh=0)
    ctx.append_all(k, v)
    want = ctx.compute_all(q)
    q[0, 1, 5] = float("nan")
    got = ctx.compute_all(q)
    try:
        gpu_lib.adaptq_set_kernel_policy(1)
        ref = ctx.compute_all(q)
    finally:
        gpu_lib.adaptq_set_kernel_policy(0)
    assert torch.isnan(got[0, 1]).all() and torch.isnan(got[1]).all()
    rest = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(got), rest)
    assert_close(got[rest].cpu().numpy(), ref[rest].cpu().numpy(), "against the general kernel")
    same = torch.ones_like(rest)
    same[0, 1] = same[1] = False
    assert torch.equal(got[same], want[same])


@pytest.mark.parametrize("heads,n,nq,dim,kb,hyb,usual", [(1, 90000, 8, 128, 4, 0, b"stream"), (1, 240000, 8, 64, 2, 0, b"general"),
                                                         (1, 65536, 1, 128, 4, 65536, b"general")])
def test_calls_whose_faster_kernel_needs_scratch_run_without_it(gpu_lib, heads, n, nq, dim, kb, hyb, usual):
    """The first call of a handle inside a stream capture, or with no memory to be had: the spans' partials of
    the streaming and general kernels cannot be allocated, so the grouped or the window kernel takes the call."""
    import torch
    from adaptq_b200 import MHAContext
    gen = torch.Generator(device="cuda").manual_seed(n)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        handles = [MHAContext(heads, dim, kb, 2, n, seed=5, v_mass=0.0, hybrid_thresh=hyb) for _ in range(3)]
        for t in range(0, n, 32768):
            k, v = (torch.randn((min(32768, n - t), heads, dim), device="cuda", generator=gen) for _ in range(2))
            for c in handles:
                c.append_all(k, v)
        q = torch.randn((heads, nq, dim), device="cuda", generator=gen)
        want = handles[0].compute_all(q)
        assert gpu_lib.adaptq_last_attention_kernel() == usual
        gpu_lib.adaptq_inject_failure(1, 1)
        try:
            refused = handles[1].compute_all(q)
        finally:
            gpu_lib.adaptq_inject_failure(1, 0)
        without = b"window" if hyb else b"group"
        assert gpu_lib.adaptq_last_attention_kernel() == without
        captured = torch.empty_like(q)
        graph = torch.cuda.CUDAGraph()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            handles[2].compute_all(q, out=captured)
        assert gpu_lib.adaptq_last_attention_kernel() == without
        graph.replay()
    torch.cuda.synchronize()
    for o in (refused, captured):
        assert_close(o.cpu().numpy(), want.cpu().numpy(), "without scratch")
    for c in handles:
        c.synchronize()


def _us(torch, fn, calls=20, batches=5):
    """Best time of a call, back to back on the device."""
    fn(), fn(), torch.cuda.synchronize()
    best = float("inf")
    for _ in range(batches):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(calls):
            fn()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) / calls * 1e3)
    return best


@pytest.mark.parametrize("heads,n,nq,dim,kb,vb", [(1, 131072, 4, 128, 4, 2), (4, 131072, 2, 128, 2, 2), (8, 131072, 2, 128, 3, 3),
                                                  (16, 4096, 8, 128, 4, 2), (32, 4096, 7, 128, 2, 4)])
def test_calls_that_the_streaming_kernel_does_faster_stay_there(gpu_lib, heads, n, nq, dim, kb, vb):
    """Few heads give compute_group_kernel too few runs to fill the chip, and small calls do not pay for its
    launch.  compute_partial always walks the streaming kernel over the same rows; the grouped kernel takes
    1.35 to 4 times as long here, and 25 % is far above what two runs of one kernel differ by."""
    import torch
    from adaptq_b200 import MHAContext
    gen = torch.Generator(device="cuda").manual_seed(n)
    ctx = MHAContext(heads, dim, kb, vb, n, seed=1, v_mass=0.0, hybrid_thresh=0)
    for t in range(0, n, 32768):
        k, v = (torch.randn((min(32768, n - t), heads, dim), device="cuda", generator=gen) for _ in range(2))
        ctx.append_all(k, v)
    q = torch.randn((heads, nq, dim), device="cuda", generator=gen)
    out, part = torch.empty_like(q), ctx.compute_partial(q)
    chosen, stream = _us(torch, lambda: ctx.compute_all(q, out=out)), _us(torch, lambda: ctx.compute_partial(q, out=part))
    assert chosen < 1.25 * stream, (chosen, stream)
