"""BatchedAdaptQAttention against a loop over per-sequence AdaptQAttention
modules (upstream's prescription for batch_size > 1,
adaptq/torch_adapter.py:78-85): same outputs, tensors stay on the GPU."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [dict(k_bits=4, v_bits=2, v_mass=0.0, hybrid_thresh=0),
                                 dict(k_bits=4, v_bits=4, v_mass=0.95, hybrid_thresh=8),
                                 dict(k_bits=16, v_bits=2, v_mass=0.0, hybrid_thresh=0)])
def test_batched_equals_loop_of_single_sequence_modules(gpu_lib, orc, cfg):
    import torch
    from adaptq_b200 import BatchedAdaptQAttention, Engine
    from helpers import CpuHeads, assert_close, assert_sparse_close
    batch, heads, dim, cap = 3, 4, 64, 24
    # CPU oracle for the first and the last sequence (every sequence is seeded alike)
    cpus = {b: CpuHeads(orc, heads, dim, cfg["k_bits"], cfg["v_bits"], cap, 42, cfg["v_mass"], cfg["hybrid_thresh"])
            for b in (0, batch - 1)}
    g = torch.Generator(device="cuda").manual_seed(2)
    bat = BatchedAdaptQAttention(dim, heads, batch, capacity=cap, seed=42, **cfg)
    singles = [Engine(dim=dim, heads=heads, capacity=cap, seed=42, **cfg) for _ in range(batch)]
    pk = torch.randn((batch, 10, heads, dim), device="cuda", generator=g)
    pv = torch.randn((batch, 10, heads, dim), device="cuda", generator=g)
    bat.prefill(pk, pv)
    for b, e in enumerate(singles):
        e.append_many(pk[b].contiguous(), pv[b].contiguous())
    for b, c in cpus.items():
        c.append_many(pk[b].cpu().numpy(), pv[b].cpu().numpy())
    for step in range(20):  # wraps the ring
        q = torch.randn((batch, heads, dim), device="cuda", generator=g)
        k = torch.randn((batch, heads, dim), device="cuda", generator=g)
        v = torch.randn((batch, heads, dim), device="cuda", generator=g)
        out = bat(q, k, v)
        assert out.shape == q.shape and out.device == q.device
        for b, e in enumerate(singles):
            want = e.step(k[b].contiguous(), v[b].contiguous(), q[b].contiguous())
            # 1e-5 relative / 1e-4 absolute; identical kernels, so in practice bit-equal
            torch.testing.assert_close(out[b], want, rtol=1e-5, atol=1e-4, msg=f"step {step} sequence {b}")
        for b, c in cpus.items():
            c.append_many(k[b].cpu().numpy()[None], v[b].cpu().numpy()[None])
            qb, ob = q[b].cpu().numpy(), out[b].cpu().numpy()
            sparse = cfg["v_mass"] > 0 and cfg["k_bits"] != 16 and c.heads[0].mirror_tokens != c.heads[0].size
            for h in range(heads):
                if sparse:
                    assert_sparse_close(ob[h], c.heads[h], qb[h], cfg["v_mass"], f"step {step} sequence {b} head {h} vs oracle")
                else:
                    assert_close(ob[h], c.heads[h].compute(qb[h])[0], f"step {step} sequence {b} head {h} vs oracle")
    bat.reset_cache()
    assert bat.pos == 0


def test_grouped_queries(gpu_lib, orc):
    import torch
    from adaptq_b200 import BatchedAdaptQAttention, MHAContext
    from helpers import CpuHeads, assert_close
    batch, heads, dim, G = 2, 3, 128, 4
    cpu = CpuHeads(orc, heads, dim, 4, 2, 64, 7)   # sequence 0 on the CPU oracle
    g = torch.Generator(device="cuda").manual_seed(3)
    bat = BatchedAdaptQAttention(dim, heads, batch, k_bits=4, v_bits=2, capacity=64, seed=7, q_per_kv=G,
                                 v_mass=0.0, hybrid_thresh=0)
    ref = [MHAContext(heads, dim, 4, 2, 64, seed=7, v_mass=0.0, hybrid_thresh=0) for _ in range(batch)]
    for step in range(12):
        q = torch.randn((batch, heads * G, dim), device="cuda", generator=g)
        k = torch.randn((batch, heads, dim), device="cuda", generator=g)
        v = torch.randn((batch, heads, dim), device="cuda", generator=g)
        out = bat(q, k, v)
        for b in range(batch):
            ref[b].append_all(k[b].contiguous(), v[b].contiguous())
            for h in range(heads):
                want = ref[b].compute_batch(h, q[b, h * G:(h + 1) * G].contiguous().cpu().numpy())
                torch.testing.assert_close(out[b, h * G:(h + 1) * G].cpu(), torch.from_numpy(want), rtol=1e-5, atol=1e-4)
        cpu.append_many(k[0].cpu().numpy()[None], v[0].cpu().numpy()[None])
        want0 = cpu.compute_batch(q[0].cpu().numpy().reshape(heads, G, dim))
        assert_close(out[0].cpu().numpy().reshape(heads, G, dim), want0, f"step {step} against the oracle")


def test_shape_errors(gpu_lib):
    import torch
    from adaptq_b200 import BatchedAdaptQAttention
    m = BatchedAdaptQAttention(64, 2, 2, capacity=8)
    x = torch.zeros((2, 2, 64), device="cuda")
    with pytest.raises(ValueError):
        m(x, x[:1], x)
    with pytest.raises(ValueError):
        m(torch.zeros((2, 4, 64), device="cuda"), x, x)
    with pytest.raises(ValueError):
        m.prefill(torch.zeros((2, 3, 2, 32), device="cuda"), torch.zeros((2, 3, 2, 32), device="cuda"))


def test_grouped_workspace_comes_with_handles_made_for_several_queries(gpu_lib):
    """Room for the pieces of grouped queries: not in a plain handle, from the start (and once) in a module
    with several queries per KV head, with the first call elsewhere."""
    import ctypes as C
    import torch
    from adaptq_b200 import BatchedAdaptQAttention, MHAContext, _lib
    batch, heads, dim, cap = 64, 8, 128, 1024
    kw = dict(v_mass=0.0, hybrid_thresh=0)

    def device_bytes(ctx):
        info = _lib.MhaInfo()
        assert gpu_lib.adaptq_mha_info(ctx._h, C.byref(info)) == 0
        return info.device_bytes

    rows = batch * heads * (cap * (64 + 32) + 2 * 128 + 2 * 4 * (cap + 32) + 16) + 16  # rows, slack, scales, signs; status word
    plain = MHAContext(batch * heads, dim, 4, 2, cap, seed=1, **kw)
    single = BatchedAdaptQAttention(dim, heads, batch, 4, 2, cap, **kw)
    grouped = BatchedAdaptQAttention(dim, heads, batch, 4, 2, cap, q_per_kv=4, **kw)
    assert device_bytes(plain) == device_bytes(single._ctx) == rows
    reserved = device_bytes(grouped._ctx)
    assert rows < reserved < rows + 2 * 2**20
    x = lambda *s: torch.randn(s, device="cuda")  # noqa: E731
    k, v = x(cap - 1, batch * heads, dim), x(cap - 1, batch * heads, dim)
    plain.append_all(k, v)
    grouped._ctx.append_all(k, v)
    grouped(x(batch, heads * 4, dim), x(batch, heads, dim), x(batch, heads, dim))
    assert device_bytes(grouped._ctx) == reserved
    q = x(batch * heads, 4, dim)
    plain.compute_all(q)
    assert rows < device_bytes(plain) < rows + 2 * 2**20
    plain.reserve_queries(8)
    with pytest.raises(RuntimeError):
        plain.reserve_queries(-1)
    # one long sequence: spans of one query come with the handle, those of more queries when asked for
    n = 100000
    for d, bits in ((dim, 4), (64, 2)):  # 2-bit keys at 64: the general kernel
        long = MHAContext(4, d, bits, 2, n, seed=1, **kw)
        long.append_all(x(n, 4, d), x(n, 4, d))
        q = x(4, 4, d)
        start = device_bytes(long)
        long.compute_all(q[:, 0].contiguous())
        assert device_bytes(long) == start
        long.reserve_queries(4)
        start = device_bytes(long)
        long.compute_all(q)
        assert device_bytes(long) == start
