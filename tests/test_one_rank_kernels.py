"""Kernels that only a one-rank communicator takes (nothing to exchange, so nothing is staged), and the prompt-side
kernel, against plain PyTorch, at the edges of their grids."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    import torch_ccl_b200._C as C

    return C.CudaComm.create(None, 0, 1, 8 << 20, 1000, "ccl/one-rank-test")


# one row / the last row count of the wide form and the first of the narrow one / hidden from one vector to the largest
@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 4096), (592, 952), (593, 952), (700, 4096), (5, 5120), (600, 16384)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_residual_rmsnorm(comm, rows, hidden, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows * hidden)
    x, res, w = (torch.randn(*s, generator=g, device="cuda").to(dtype) for s in ((rows, hidden), (rows, hidden), (hidden,)))
    h = (x.float() + res.float()).to(dtype)
    n = (h.float() * torch.rsqrt(h.float().pow(2).mean(-1, keepdim=True) + 1e-5)).to(dtype)
    out = torch.empty_like(x)
    comm.allreduce_residual_rmsnorm([x], [res], [w], [out], 1e-5)
    assert torch.equal(res, h)
    # half a unit in the last place is at most 2^-8 (bf16: 8 significant bits) or 2^-11 (f16: 11 bits) of a value. The mean
    # in another order may move the normalised value by one unit in the last place (two halves), and the product with the
    # weight is rounded (one half): three halves in all.
    half = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    torch.testing.assert_close(out.float(), n.float() * w.float(), rtol=3 * half, atol=1e-6)


@pytest.mark.parametrize("rows,hidden", [(2, 4096), (593, 952), (700, 1024), (700, 1032), (700, 2048), (700, 2056),
                                         (700, 4096), (5, 4104), (600, 5120), (600, 5128), (600, 6152), (600, 8192), (600, 8200), (600, 16384)])
def test_residual_rmsnorm_sums_in_the_order_of_the_staged_kernel(comm, rows, hidden):
    """Bit for bit what the kernel for several ranks gives for one (the emulation takes that one)."""
    import torch_ccl_b200._C as C

    g = torch.Generator(device="cuda").manual_seed(rows * hidden)
    x, res, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((rows, hidden), (rows, hidden), (hidden,)))
    # one element carries most of a row's sum, so that the order of the small ones shows in its last bits
    x[:, 0] = 64.0
    got = []
    for c in (comm, C.CudaComm.emulated(1, 1 << 20, 1000, 8)):
        r, out = res.clone(), torch.empty_like(x)
        c.allreduce_residual_rmsnorm([x], [r], [w], [out], 1e-5)
        got.append((r, out))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_residual_rmsnorm_embedding(comm):
    """Token ids outside this rank's part of the table contribute zeros; the residual is not read."""
    table = torch.randn(50, 256, device="cuda").bfloat16()
    tok = torch.tensor([0, 99, 100, 149, 150, 7], device="cuda")
    res = torch.full((6, 256), float("nan"), device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(res)
    comm.allreduce_residual_rmsnorm([table], [res], [torch.ones(256, device="cuda").bfloat16()], [out], 1e-5, [tok], [100], True)
    want = torch.zeros_like(res)
    want[2], want[3] = table[0], table[49]
    assert torch.equal(res, want) and not torch.isnan(out.float()).any()


@pytest.mark.parametrize("n,seq,heads,kv,room", [(1, 1, 4, 4, 8), (3, 77, 8, 2, 80), (2, 130, 0, 3, 130)])
def test_rope_append(n, seq, heads, kv, room):
    import torch_ccl_b200._C as C

    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv = torch.randn(n * seq, (heads + 2 * kv) * 128, generator=g, device="cuda").bfloat16()
    inv = 1.0 / (10000.0 ** (torch.arange(0, 128, 2, device="cuda").float() / 128))
    ang = torch.arange(room, device="cuda").float()[:, None] * inv[None]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    c, s = (t[:seq].bfloat16()[None, :, None] for t in (cos, sin))
    x = qkv.view(n, seq, -1, 128).clone()
    t1, t2 = x[:, :, : heads + kv, :64], x[:, :, : heads + kv, 64:]
    rot = torch.cat([t1 * c - t2 * s, t2 * c + t1 * s], -1)
    kc = torch.full((n, kv, room, 128), 7.0, device="cuda", dtype=torch.bfloat16)
    vc = kc.clone()
    C.rope_append(qkv, kc, vc, cos, sin, heads, seq)
    got = qkv.view(n, seq, -1, 128)
    assert torch.equal(got[:, :, :heads], rot[:, :, :heads]) and torch.equal(got[:, :, heads:], x[:, :, heads:])
    assert torch.equal(kc[:, :, :seq], rot[:, :, heads:].transpose(1, 2)) and torch.equal(vc[:, :, :seq], x[:, :, heads + kv:].transpose(1, 2))
    assert (kc[:, :, seq:] == 7.0).all() and (vc[:, :, seq:] == 7.0).all()


@pytest.mark.parametrize("tokens,hidden,experts,topk", [(0, 64, 2, 1), (1, 8, 4, 1), (33, 256, 8, 2), (100, 4104, 16, 5), (7, 8192, 8, 9)])
def test_moe(comm, tokens, hidden, experts, topk):
    """Dispatch in slot order; combine from any order of rows and records; a slot whose row is missing counts as zero."""
    g = torch.Generator(device="cuda").manual_seed(hidden)
    x = torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16()
    idx = torch.randint(0, experts, (tokens, topk), generator=g, device="cuda", dtype=torch.int32)
    gate = torch.rand(tokens, topk, generator=g, device="cuda")
    n = tokens * topk
    rows = torch.empty(n, hidden, device="cuda", dtype=torch.bfloat16)
    meta = torch.empty(n, 3, device="cuda", dtype=torch.int32)
    count = torch.full((16,), -1, device="cuda", dtype=torch.int32)
    comm.moe_dispatch([x], [idx], [rows], [meta], [count], experts)
    assert count[:2].tolist() == [n, n] and (count[2:] == -1).all()
    assert torch.equal(rows, x.repeat_interleave(topk, 0)) and torch.equal(meta[:, 2], idx.view(-1)) and comm.status()[0] == 0
    y = (rows.float() * (1 + meta[:, 2:3])).bfloat16()
    p = torch.randperm(n, device="cuda")
    out = torch.empty(tokens, hidden, device="cuda", dtype=torch.bfloat16)
    comm.moe_combine([y[p].contiguous()], [meta[p].contiguous()], [count], [gate], [out])
    ref = (y.double().view(tokens, topk, hidden) * gate.double()[:, :, None]).sum(1)
    # fp32 sum of topk products (2^-24 each of their magnitude), then one rounding to bf16
    bound = ref.abs() * 2.0**-8 + (y.double().view(tokens, topk, hidden).abs() * gate.double()[:, :, None]).sum(1) * topk * 2.0**-23
    assert ((out.double() - ref).abs() <= bound).all()
    if n:  # the last row does not come back
        count[0] = n - 1
        comm.moe_combine([y[p].contiguous()], [meta[p].contiguous()], [count], [gate], [out])
        left = y.clone()
        left[int(meta[p[-1], 1])] = 0
        ref = (left.double().view(tokens, topk, hidden) * gate.double()[:, :, None]).sum(1)
        assert ((out.double() - ref).abs() <= bound + ref.abs() * 2.0**-8).all()


@pytest.mark.parametrize("tokens,hidden,topk", [(5, 64, 0), (0, 64, 2), (5, 0, 2)])
def test_moe_of_nothing(comm, tokens, hidden, topk):
    """No experts a token (the sums are zero), no tokens, rows without elements."""
    x = torch.ones(tokens, hidden, device="cuda").bfloat16()
    n = tokens * topk
    rows, meta = torch.empty(n + 1, hidden, device="cuda", dtype=torch.bfloat16), torch.zeros(n + 1, 3, device="cuda", dtype=torch.int32)
    count = torch.full((16,), -1, device="cuda", dtype=torch.int32)
    comm.moe_dispatch([x], [torch.zeros(tokens, topk, device="cuda", dtype=torch.int32)], [rows], [meta], [count], 1)
    out = torch.full((tokens, hidden), 7.0, device="cuda").bfloat16()
    comm.moe_combine([rows], [meta], [count], [torch.zeros(tokens, topk, device="cuda")], [out])
    assert int(count[0]) == n and (out == 0).all() and comm.status()[0] == 0


@pytest.mark.parametrize("shift", [0, 5])
def test_moe_results_over_inputs(comm, shift):
    """out= of combine may share memory with the rows that it sums (one expert a token), and dispatch's rows with x."""
    T, H = 300, 512
    g = torch.Generator(device="cuda").manual_seed(shift)
    store = torch.zeros(T + shift, H, device="cuda", dtype=torch.bfloat16)
    y, out = store[shift:], store[:T]
    y.copy_(torch.randn(T, H, generator=g, device="cuda"))
    src = y.clone()
    gate = torch.rand(T, 1, generator=g, device="cuda")
    slot = torch.randperm(T, generator=g, device="cuda").int()
    meta = torch.stack([torch.zeros_like(slot), slot, torch.zeros_like(slot)], 1).contiguous()
    count = torch.zeros(16, device="cuda", dtype=torch.int32)
    count[:2] = T
    comm.moe_combine([y], [meta], [count], [gate], [out])
    want = torch.empty_like(src)
    want[slot.long()] = src
    assert torch.equal(out, (want.float() * gate).bfloat16())

    y.copy_(src)
    idx = torch.zeros(T, 1, device="cuda", dtype=torch.int32)
    comm.moe_dispatch([y], [idx], [out], [meta], [count], 1)
    assert torch.equal(out, src[meta[:, 1].long()]) and sorted(meta[:, 1].tolist()) == list(range(T)) and int(count[0]) == T
    with pytest.raises(RuntimeError, match="moe_dispatch"):
        comm.moe_dispatch([y], [idx], [out[: T - 1]], [meta], [count], 1)


def _combine_case(T, seed):
    """y, meta, gate of a combine with two experts a token whose rows come back in another order, and the result."""
    H, g = 1024, torch.Generator(device="cuda").manual_seed(seed)
    y = torch.randn(2 * T, H, generator=g, device="cuda").bfloat16()
    slot = torch.randperm(2 * T, generator=g, device="cuda").int()
    meta = torch.stack([torch.zeros_like(slot), slot, torch.zeros_like(slot)], 1).contiguous()
    back = torch.empty_like(y)
    back[slot.long()] = y
    back = back.float().view(T, 2, H)
    gate = torch.full((T, 2), 0.5, device="cuda")  # exact products
    return y, meta, torch.full((16,), 2 * T, device="cuda", dtype=torch.int32), gate, ((back[:, 0] + back[:, 1]) * 0.5).bfloat16()


@pytest.mark.parametrize("captured", [False, True])
def test_launches_on_two_streams_are_ordered(comm, captured):
    """Combines share the communicator's arena (the inverse of the records): from two streams, eager or within one capture,
    one runs after the other."""
    cases = [_combine_case(1000, i) for i in range(4)]
    outs = [torch.empty_like(c[4]) for c in cases]

    def work(s1, s2):
        start, ends = torch.cuda.Event(), [torch.cuda.Event() for _ in range(2)]
        start.record(s1)
        s2.wait_event(start)
        for i, (y, meta, count, gate, _) in enumerate(cases):
            with torch.cuda.stream((s1, s2)[i % 2]):
                comm.moe_combine([y], [meta], [count], [gate], [outs[i]])
        ends[1].record(s2)
        s1.wait_event(ends[1])

    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    work(s1, s2)
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s1):
            work(s1, s2)
        for out in outs:
            out.zero_()
        for _ in range(20):
            graph.replay()
        torch.cuda.synchronize()
    for out, c in zip(outs, cases):
        assert torch.equal(out, c[4])


def test_stream_destroyed_after_a_launch(comm):
    """A launch on another stream still waits for the one before it when that one's stream is gone."""
    import ctypes

    cudart = torch.cuda.cudart()
    cases = [_combine_case(1000, i) for i in range(2)]
    outs = [torch.empty_like(c[4]) for c in cases]
    handle = ctypes.c_ulonglong(0)
    assert int(cudart.cudaStreamCreate(ctypes.cast(ctypes.pointer(handle), ctypes.c_void_p).value)) == 0
    torch.cuda.synchronize()
    (y, meta, count, gate, _), own = cases[0], torch.cuda.ExternalStream(handle.value)
    with torch.cuda.stream(own):
        torch.cuda._sleep(20_000_000)
        comm.moe_combine([y], [meta], [count], [gate], [outs[0]])
        comm.launched()
    assert int(cudart.cudaStreamDestroy(handle.value)) == 0
    y, meta, count, gate, _ = cases[1]
    comm.moe_combine([y], [meta], [count], [gate], [outs[1]])
    torch.cuda.synchronize()
    for out, c in zip(outs, cases):
        assert torch.equal(out, c[4])


def test_moe_over_capacity(comm):
    """Rows that out_x has no room for are dropped and reported."""
    x, idx = torch.ones(4, 64, device="cuda").bfloat16(), torch.zeros(4, 2, device="cuda", dtype=torch.int32)
    store = torch.full((8, 64), 5.0, device="cuda").bfloat16()
    meta, count = torch.zeros(8, 3, device="cuda", dtype=torch.int32), torch.zeros(16, device="cuda", dtype=torch.int32)
    comm.moe_dispatch([x], [idx], [store[:6]], [meta], [count], 1)
    torch.cuda.synchronize()
    assert comm.status()[0] == 2 and int(count[0]) == 6 and (store[6:] == 5.0).all()
    comm.clear_status()


@pytest.mark.parametrize("sizes", [[1], [7, 8, 9], [4096, 3, 100001], [5] * 60])
@pytest.mark.parametrize("src,dst", [(torch.bfloat16, torch.float32), (torch.float16, torch.float32), (torch.float32, torch.float32),
                                     (torch.bfloat16, torch.bfloat16)])
def test_accumulate_cast(sizes, src, dst):
    """Any offsets (so any alignment of the destination), more tensors than one launch takes."""
    import torch_ccl_b200._C as C

    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    xs = [torch.randn(n, generator=g, device="cuda").to(src) for n in sizes]
    offs = [sum(sizes[:i]) + 3 for i in range(len(sizes))]
    acc = torch.randn(sum(sizes) + 8, generator=g, device="cuda").to(dst)
    want = acc.clone()
    for x, o in zip(xs, offs):
        want[o:o + x.numel()] = (want[o:o + x.numel()].float() + x.float() * 0.5).to(dst)
    C.accumulate_cast(xs, acc, offs, 0.5)
    assert torch.equal(acc, want)  # the product with 0.5 is exact, so a fused multiply-add rounds the same


@pytest.mark.parametrize("M,N,K", [(128, 16, 64), (384, 1024, 520)])
def test_gemm_collective_ops_alone(comm, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = torch.randn(M, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    for op in (comm.gemm_rs, comm.ag_gemm):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        op([a], [b], [out])
        assert ((out.float() - ref).norm() / ref.norm()).item() <= 2.0**-9 + K * 2.0**-24


def test_gemm_collective_ops_keep_their_limit():
    """What a larger group could not stage is refused with one rank too (callers ask for the capacity first)."""
    import torch_ccl_b200._C as C

    small = C.CudaComm.create(None, 0, 1, 1 << 20, 1000, "ccl/one-rank-limit")
    for op, shape in ((small.gemm_rs, (1024, 528, 64)), (small.ag_gemm, (1024, 64, 520))):  # (M, N, K): a little above 1 MB
        for m in (1024, 896):
            _, N, K = shape
            a, b = torch.ones(m, K, device="cuda").bfloat16(), torch.ones(N, K, device="cuda").bfloat16()
            out = torch.empty(m, N, device="cuda", dtype=torch.bfloat16)
            if m == 1024:
                with pytest.raises(RuntimeError, match="invalid argument"):
                    op([a], [b], [out])
            else:
                op([a], [b], [out])
                assert (out == K).all()


@pytest.mark.parametrize("M,K", [(256, 1024), (1024, 256)])
def test_gemm_rs_result_over_an_operand(comm, M, K):
    """out= may share memory with either operand (N = K, or N = K = M)."""
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = torch.randn(M, K, generator=g, device="cuda").bfloat16(), torch.randn(K, K, generator=g, device="cuda").bfloat16()
    want = torch.empty(M, K, device="cuda", dtype=torch.bfloat16)
    comm.gemm_rs([a], [b], [want])
    for shift in (0, 3):  # the same rows, and rows further on in one allocation
        both = torch.zeros(M + shift, K, device="cuda", dtype=torch.bfloat16)
        both[shift:] = a
        comm.gemm_rs([both[shift:]], [b], [both[:M]])
        assert torch.equal(both[:M], want)
    if M >= K:
        over = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
        over[:K] = b
        comm.gemm_rs([a], [over[:K]], [over])
        assert torch.equal(over, want)


@pytest.fixture()
def group():
    import torch.distributed as dist

    import oneccl_bindings_for_pytorch  # noqa: F401

    dist.init_process_group("ccl", store=dist.HashStore(), rank=0, world_size=1)
    yield dist.group.WORLD
    dist.destroy_process_group()


@pytest.mark.parametrize("async_op", [False, True])
def test_tensor_of_another_stream_outlives_the_collective(group, async_op):
    """A tensor allocated on one stream, used by a collective issued from another and freed at once: its memory is not
    handed out on the first stream while the collective is pending."""
    import torch.distributed as dist

    n = 1 << 20
    home = torch.cuda.Stream()
    with torch.cuda.stream(home):
        t = torch.ones(n, device="cuda")
    torch.cuda.current_stream().wait_stream(home)
    out = torch.empty(n, device="cuda")
    # set-up of the communicator, and everything loaded: loading a kernel may wait for the device
    dist.all_gather_into_tensor(out, torch.zeros(n, device="cuda"), group=group, async_op=async_op)
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s of device time before the collective may run
    work = dist.all_gather_into_tensor(out, t, group=group, async_op=async_op)
    if async_op:
        work.wait()
        del work
    was = t.data_ptr()
    del t
    with torch.cuda.stream(home):
        other = torch.zeros(n, device="cuda")
    assert other.data_ptr() != was
    torch.cuda.synchronize()
    assert (out == 1).all()


def test_full_shard_unit_with_a_sparse_gradient(group):
    from torch_ccl_b200.parallel.fsdp import FullyShardedSequential

    torch.manual_seed(0)
    emb = torch.nn.Embedding(40, 16, sparse=True, device="cuda")
    engine = FullyShardedSequential([emb], group=group)
    ids = torch.tensor([[3, 5, 3]], device="cuda")
    engine(ids).backward(torch.ones(1, 3, 16, device="cuda", dtype=torch.bfloat16))
    grad = engine.master_params()[0].grad[: 40 * 16].view(40, 16)
    want = torch.zeros(40, 16, device="cuda")
    want[3], want[5] = 2.0, 1.0
    assert torch.equal(grad, want)


def test_norm_weight_written_by_the_kernel_before(group):
    """The norm reads its weight after the kernels before it on the stream, which start their successor early."""
    from torch_ccl_b200 import ops

    rows, hidden, steps = 4, 4096, 50
    x = torch.randn(rows, hidden, device="cuda").bfloat16()
    n = (x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5)).bfloat16()
    # the cast is long (its tail is the weight), so that an early read would find the weight of the step before
    long_in = [torch.full((1 << 24,), float(i), device="cuda").bfloat16() for i in (1, 2)]
    long_out = torch.zeros(1 << 24, device="cuda").bfloat16()
    w = long_out[-hidden:]
    res = torch.zeros(steps, rows, hidden, device="cuda").bfloat16()
    got = []
    for i in range(steps):  # (nothing of torch's between the two, which would wait for the first)
        ops.reduce_scatter_cast(long_in[i % 2], long_out)
        got.append(ops.allreduce_residual_rmsnorm(x, res[i], w))
    for i, y in enumerate(got):
        torch.testing.assert_close(y.float(), n.float() * (1 + i % 2), rtol=2.0**-7, atol=1e-6)


def test_reduce_scatter_cast_types_and_overlap(group):
    """With one rank: every type that torch copies, in place, and no partial overlap."""
    from torch_ccl_b200 import ops

    x = torch.randn(1000, device="cuda")
    for dt in (torch.float32, torch.float16, torch.bfloat16, torch.float64, torch.float8_e4m3fn, torch.int32):
        a = (x * 10).to(dt)
        for out_dt in {dt, torch.float32}:
            out = torch.empty(1000, device="cuda", dtype=out_dt)
            assert torch.equal(ops.reduce_scatter_cast(a, out).float(), a.float())
    own = x.clone()
    assert torch.equal(ops.reduce_scatter_cast(own, own, 0.5), x * 0.5)
    for a, out in ((own[:500], own[100:600]), (own.view(torch.bfloat16)[:500], own[:500])):
        with pytest.raises(RuntimeError, match="memory location"):
            ops.reduce_scatter_cast(a, out)


@pytest.mark.parametrize("pending", [False, True])
def test_future_of_a_dropped_work(group, pending):
    """A future without tensors is completed, and its callbacks run, also when its holder has let the Work go."""
    import time

    import torch.distributed as dist

    dist.barrier(device_ids=[0])  # set-up of the communicator
    if pending:
        torch.cuda._sleep(100_000_000)
    fut = dist.barrier(async_op=True, device_ids=[0]).get_future()
    called = []
    fut.add_done_callback(lambda f: called.append(1))
    limit = time.time() + 10
    while not (fut.done() and called) and time.time() < limit:
        time.sleep(0.001)
    assert fut.done() and called == [1]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_full_shard_step_on_two_streams(group, dtype):
    """Forward and backward on streams of their own, the optimizer on another, each late: every one sees what the one before
    it left, without a word from the caller."""
    from torch_ccl_b200.parallel.fsdp import FullyShardedSequential

    def train(compute, late):
        torch.manual_seed(0)
        engine = FullyShardedSequential([torch.nn.Linear(64, 64, device="cuda") for _ in range(3)], group=group, param_dtype=dtype)
        g = torch.Generator(device="cuda").manual_seed(1)
        x, dy = (torch.randn(6, 32, 64, generator=g, device="cuda").to(dtype) for _ in range(2))
        third = torch.cuda.Stream() if late else torch.cuda.current_stream()
        torch.cuda.synchronize()
        seen, evals = [], []
        for i in range(3):
            for s, j in zip(compute, (2 * i, 2 * i + 1)):  # two micro-batches a step
                with torch.cuda.stream(s):
                    torch.cuda._sleep(late)
                    engine(x[j]).backward(dy[j])
            with torch.cuda.stream(third), torch.no_grad():  # a forward pass alone, of the weights before the step
                torch.cuda._sleep(late)
                evals.append(engine(x[0]))
            masters = engine.master_params()
            seen.append([m.grad.clone() for m in masters])
            torch.cuda._sleep(late)
            for m in masters:
                m -= 0.1 * m.grad
            engine.after_step()
        torch.cuda.synchronize()
        return [t for grads in seen for t in grads] + evals + [u.master for u in engine.units] + [u.shard for u in engine.units]

    here = torch.cuda.current_stream()
    want = train([here, here], 0)
    got = train([torch.cuda.Stream(), torch.cuda.Stream()], 20_000_000)
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_packed_weight_cast_just_before_its_product(group):
    """A GEMM fetches its packed weight before the kernel in front of it has ended; a cast that writes that weight comes first."""
    import torch_ccl_b200._C as C

    from torch_ccl_b200 import ops

    rows, K = 256, 4096
    x = torch.randn(16, K, device="cuda").bfloat16()
    w = [torch.randn(rows, K, device="cuda").bfloat16() for _ in range(2)]
    # the cast is long, with the weight at its end
    n = 1 << 24
    src = [torch.cat([torch.zeros(n - rows * K, device="cuda").bfloat16(), ops.pack_weight(t).view(-1)]) for t in w]
    dst = torch.zeros(n, device="cuda").bfloat16()
    packed = dst[n - rows * K:].view(-1, 64)
    out = torch.empty(40, 16, rows, device="cuda")
    for i in range(40):
        ops.reduce_scatter_cast(src[i % 2], dst)
        C.gemm_bf16_tn(packed, x, out[i], True, 0, 0, 0, rows)
    want = [torch.empty(16, rows, device="cuda") for _ in w]
    for t, o in zip(w, want):
        C.gemm_bf16_tn(ops.pack_weight(t), x, o, True, 0, 0, 0, rows)
    assert all(torch.equal(out[i], want[i % 2]) for i in range(40))


def test_full_shard_pass_in_a_graph(group):
    """Forward and backward captured once, replayed between optimizer steps on another stream."""
    from torch_ccl_b200.parallel.fsdp import FullyShardedSequential

    torch.manual_seed(0)
    engine = FullyShardedSequential([torch.nn.Linear(64, 64, device="cuda") for _ in range(2)], group=group)
    x, dy = torch.randn(32, 64, device="cuda").bfloat16(), torch.randn(32, 64, device="cuda").bfloat16()

    def one():
        engine(x).backward(dy)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        one()
        one()
    torch.cuda.synchronize()
    engine.after_step()
    one()
    want = [m.grad.clone() for m in engine.master_params()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        one()
    for _ in range(3):
        engine.after_step()
        graph.replay()
        assert all(torch.equal(m.grad, w) for m, w in zip(engine.master_params(), want))
