"""One PE on one GPU: VMM heap, symmetric tensors, host RMA to self, collectives of size one, fused ops."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nv():
    import nvshmem_b200.core as nv
    torch.cuda.set_device(0)
    nv.init(device=0, uid=nv.get_unique_id(), rank=0, nranks=1)
    yield nv
    nv.finalize()


def test_world_of_one(nv):
    assert nv.my_pe() == 0 and nv.n_pes() == 1
    info = nv.heap_info()
    assert info["backed"] >= 1 << 30 and info["stride"] >= info["backed"]
    assert "B200" in nv.topology() or "NVIDIA" in nv.topology()


def test_tensor_alloc_put_get_roundtrip(nv):
    a = nv.tensor((1 << 20,), torch.float32)
    b = nv.tensor((1 << 20,), torch.float32)
    src = torch.rand(1 << 20, device="cuda")
    nv.put(a, src, 0)
    nv.get(b, a, 0)
    nv.quiet()
    torch.cuda.synchronize()
    assert torch.equal(b, src)
    nv.free_tensor(a)
    nv.free_tensor(b)


def test_heap_growth_keeps_old_data(nv):
    small = nv.tensor((1024,), torch.int32)
    small.copy_(torch.arange(1024, dtype=torch.int32, device="cuda"))
    before = nv.heap_info()["chunks"]
    big = nv.tensor(((3 << 30) // 4,), torch.float32)  # larger than the initial 1 GiB: forces growth
    assert nv.heap_info()["chunks"] > before
    big[-1] = 7.0
    torch.cuda.synchronize()
    assert torch.equal(small.cpu(), torch.arange(1024, dtype=torch.int32))
    assert float(big[-1]) == 7.0
    nv.free_tensor(big)
    nv.free_tensor(small)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32, torch.int64])
def test_collectives_on_one_pe_are_copies(nv, dtype):
    n = 4096
    src = nv.tensor((n,), dtype)
    dst = nv.tensor((n,), dtype)
    src.copy_((torch.arange(n, device="cuda") % 97).to(dtype))
    for coll in ("reduce", "reducescatter", "fcollect", "alltoall", "broadcast"):
        dst.zero_()
        nv.collective_on_buffer(coll, 0, dst, src, op="sum")
        nv.barrier_all()
        torch.cuda.synchronize()
        assert torch.equal(dst, src), coll
    assert nv.error_bits() == 0
    nv.free_tensor(src)
    nv.free_tensor(dst)


@pytest.mark.parametrize("n,so,do", [(1, 0, 0), (15, 0, 0), (16384, 0, 0), (16401, 0, 0), ((1 << 25) + 3, 16, 16), (40000, 8, 16), (40002, 4, 12), (40001, 2, 6), (70001, 1, 4)])
def test_collectives_of_one_member_copy_every_byte_and_no_more(nv, n, so, do):
    """Tails, all alignments of the two addresses, one and several rounds of the copy kernel; nothing outside is written."""
    src = nv.tensor((n + 64,), torch.uint8)
    dst = nv.tensor((n + 64,), torch.uint8)
    src.copy_(torch.randint(0, 256, (n + 64,), device="cuda", dtype=torch.uint8))
    for coll in ("reduce", "reducescatter", "fcollect", "alltoall", "broadcast"):
        dst.fill_(7)
        nv.collective_on_buffer(coll, 0, dst[do:do + n], src[so:so + n], op="sum")
        torch.cuda.synchronize()
        assert torch.equal(dst[do:do + n], src[so:so + n]), coll
        assert bool((dst[:do] == 7).all()) and bool((dst[do + n:] == 7).all()), coll
        nv.collective_on_buffer(coll, 0, dst[do:do + n], dst[do:do + n], op="sum")  # in place
    torch.cuda.synchronize()
    assert torch.equal(dst[do:do + n], src[so:so + n]) and nv.error_bits() == 0
    nv.free_tensor(src)
    nv.free_tensor(dst)


def _kernels(call):
    """(name, CTAs) of every kernel that `call` launches on the current stream, in order."""
    driver = pytest.importorskip("cuda.bindings.driver")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    nodes = driver.cuGraphGetNodes(raw, driver.cuGraphGetNodes(raw, 0)[2])[1]
    out = []
    for node in nodes:
        if driver.cuGraphNodeGetType(node)[1] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, p = driver.cuGraphKernelNodeGetParams(node)
            assert int(err) == 0
            err, name = driver.cuFuncGetName(p.func) if int(p.func) else driver.cuKernelGetName(p.kern)
            assert int(err) == 0
            out.append((name.decode(), p.gridDimX * p.gridDimY * p.gridDimZ))
    return out


@pytest.mark.parametrize("dtype,n", [(torch.float32, 1), (torch.bfloat16, 4099), (torch.int32, 70001), (torch.float64, 1 << 20)])
def test_a_named_algorithm_runs_its_kernel_on_a_team_of_one(nv, dtype, n):
    """The kernels for several members, which the automatic choice leaves aside for one member: reachable by naming an algorithm
    (the all-to-all through a test hook), same bytes as the copy kernel, nothing written beyond."""
    import ctypes as C
    from nvshmem_b200.bindings import host as H
    src, dst = nv.tensor((n + 8,), dtype), nv.tensor((n + 8,), dtype)
    src.copy_((torch.arange(n + 8, device="cuda") % 113).to(dtype))

    def alltoall_kernel():
        assert H.load().bshmem_test_alltoall_kernel(0, C.c_void_p(dst.data_ptr()), C.c_void_p(src.data_ptr()), C.c_size_t(n * src.element_size()),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0

    calls = [("reduce_kernel", lambda a=a: nv.reduce(0, dst[:n], src[:n], "sum", algo=a)) for a in ("oneshot", "twoshot", "ll", "ll128", "recexch")]
    calls += [("reducescatter_kernel", lambda: nv.reducescatter(0, dst[:n], src[:n], "sum", algo="pull"))]
    calls += [("fcollect_kernel", lambda a=a: nv.fcollect(0, dst[:n], src[:n], algo=a)) for a in ("push", "ll", "ll128")]
    calls += [("broadcast_kernel", lambda a=a: nv.broadcast(0, dst[:n], src[:n], algo=a)) for a in ("push", "pull", "ll")]
    calls += [("alltoall_kernel", alltoall_kernel), ("local_copy_kernel", lambda: nv.reduce(0, dst[:n], src[:n], "sum"))]
    for kernel, call in calls:
        dst.fill_(7)
        call()
        torch.cuda.synchronize()
        assert torch.equal(dst[:n], src[:n]) and bool((dst[n:] == 7).all()), kernel
        names = _kernels(call)
        assert len(names) == 1 and kernel in names[0][0], (kernel, names)
    assert nv.error_bits() == 0
    nv.free_tensor(src)
    nv.free_tensor(dst)


def test_signal_and_wait_on_stream(nv):
    sig = nv.tensor((1,), torch.int64, zero=True)
    nv.signal_op(sig, 5, nv.SignalOp.SIGNAL_SET, 0)
    nv.signal_wait(sig, 5, nv.ComparisonType.CMP_GE)
    nv.signal_op(sig, 3, nv.SignalOp.SIGNAL_ADD, 0)
    torch.cuda.synchronize()
    assert nv.signal_fetch(sig) == 8
    nv.free_tensor(sig)


def test_bounded_wait_reports_timeout_instead_of_hanging(nv):
    """A signal that nobody sets: the wait kernel gives up after the bound and the status says so."""
    sig = nv.tensor((1,), torch.int64, zero=True)
    nv.set_wait_timeout_ms(200)
    nv.clear_errors()
    from nvshmem_b200.bindings import host as H
    # CMP_GT cannot use the stream memory operation, so this runs the device wait loop.
    nv.signal_wait(sig, 1, nv.ComparisonType.CMP_GT)
    torch.cuda.synchronize()
    assert nv.error_bits() & H.ERR_WAIT_TIMEOUT
    nv.clear_errors()
    nv.set_wait_timeout_ms(30000)
    nv.free_tensor(sig)


def test_fused_ops_single_pe(nv):
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(1)
    M, N, K = 512, 512, 256
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ref = x.float() @ w.float().t()
    tol = ref.abs().max().item() * 2 ** -7 + 1e-3
    rs = fg.GemmReduceScatter(M, N, mode="rs")
    assert (rs(x, w).float() - ref).abs().max().item() <= tol
    ar = fg.GemmReduceScatter(M, N, mode="ar")
    assert (ar(x, w).float() - ref).abs().max().item() <= tol
    ag = fg.AllGatherGemm(M, K)
    ag.shard.copy_(x)
    assert (ag(w).float() - ref).abs().max().item() <= tol
    fg.check_errors()


def test_tp_mlp_forward_backward_single_pe(nv):
    from nvshmem_b200.models.tp_mlp import TensorParallelMLP
    torch.manual_seed(2)
    mlp = TensorParallelMLP(hidden=512, ffn=1024, tokens=256)
    x = torch.randn(256, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = mlp(x)
    y.float().pow(2).mean().backward()
    ref = mlp.reference(x.detach())
    assert (y.float() - ref).abs().max().item() <= 0.03 * ref.abs().max().item() + 1e-2
    # gradient check against autograd through the fp32 reference
    x32 = x.detach().float().requires_grad_(True)
    w1 = mlp.up.weight.detach().float().requires_grad_(True)
    w2 = mlp.down.weight.detach().float().requires_grad_(True)
    yr = torch.nn.functional.gelu(x32 @ w1.t(), approximate="tanh") @ w2.t()
    yr.pow(2).mean().backward()
    for got, want in ((x.grad, x32.grad), (mlp.up.weight.grad, w1.grad), (mlp.down.weight.grad, w2.grad)):
        denom = want.abs().max().item() + 1e-12
        assert (got.float() - want).abs().max().item() / denom < 0.06


def test_moe_dispatch_combine_single_pe(nv):
    """All experts local: dispatch is a permutation by expert, combine its weighted inverse."""
    import tests.workers as W
    W._moe_check(nv, "bf16", T=200, H=512, K=4, E=16, seed=11)
    W._moe_check(nv, "fp8", T=128, H=1024, K=8, E=32, seed=12)


@pytest.mark.parametrize("payload", [0, 1])
@pytest.mark.parametrize("T,H,K,E,cap", [(1, 128, 1, 1, 0), (3, 640, 16, 1024, 0), (128, 256, 16, 64, 0), (2049, 128, 1, 7, 0), (683, 2176, 3, 5, 0),
                                         (700, 2304, 8, 256, 0), (9000, 384, 9, 1000, 0), (8193, 128, 8, 33, 0), (100, 256, 4, 8, 77), (1000, 1152, 8, 8, 5000), (5, 16512, 2, 4, 0)])
def test_local_dispatch_agrees_with_the_general_one(T, H, K, E, cap, payload):
    """One PE without `dup_src` takes the kernels that meet nobody (one for up to 2048 pairs, two above); with `dup_src` the
    general kernel runs.  Offsets, counts and the multiset of rows per expert must be the same, and every row must hold what its slot
    says, to the byte; too small a buffer drops the rows beyond it and sets the overflow bit."""
    import ctypes as C
    from nvshmem_b200.ops.moe import _lib, _DispatchArgs
    lib = _lib()
    torch.manual_seed(T + H + K + E)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    x[0, :128] = 0
    idx = torch.randint(-1, E + 1, (T, K), device="cuda", dtype=torch.int32)  # -1 and E are dropped
    cap = cap or T * K
    res = []
    for general in (False, True):
        z = lambda *s, dt=torch.int32, v=0: torch.full(s, v, dtype=dt, device="cuda")
        recv = z(cap + 1, H if payload else 2 * H, dt=torch.uint8, v=9)
        scale, slot, offs, src = z(cap + 1, H // 128, dt=torch.float32, v=9), z(T, K, v=-7), z(E + 1, v=-7), z(E, 1, v=-7)
        counts, flags, scratch, err, dup = z(E, v=-7), z(4, dt=torch.int64), z(lib.bshmem_moe_scratch_bytes(E) // 4 + 64), z(1), z(cap)
        a = _DispatchArgs()
        a.T, a.H, a.K, a.E, a.rank, a.npes, a.payload, a.cap_rows, a.epoch = T, H, K, E, 0, 1, payload, cap, 1
        a.error_flag, a.x, a.topk_idx = err.data_ptr(), x.data_ptr(), idx.data_ptr()
        a.recv_x[0], a.recv_scale[0], a.counts[0], a.flags[0] = recv.data_ptr(), scale.data_ptr(), counts.data_ptr(), flags.data_ptr()
        a.slot_map, a.expert_offsets, a.src_offsets, a.scratch = slot.data_ptr(), offs.data_ptr(), src.data_ptr(), scratch.data_ptr()
        if general:
            a.dup_src[0] = dup.data_ptr()
        assert lib.bshmem_moe_dispatch(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert bool((recv[cap] == 9).all()) and bool((scale[cap] == 9).all()), "written past the buffer"
        res.append((recv, scale, slot, offs, src, counts, int(err)))
    local, general = res
    valid = (idx >= 0) & (idx < E)
    for k in (3, 4, 5):
        assert torch.equal(local[k], general[k])
    total = int(valid.sum())
    assert int(local[3][E]) == total and local[6] == (2 if total > cap else 0) and local[6] == general[6]
    got = local[2].long()
    assert bool((got[~valid] == -1).all()) and int((got >= 0).sum()) == min(total, cap)
    t, k = (got >= 0).nonzero(as_tuple=True)
    rows, e = got[t, k], idx[t, k].long()
    assert torch.equal(rows.sort().values, torch.arange(rows.numel(), device="cuda"))
    assert bool(((rows >= local[3].long()[e]) & (rows < local[3].long()[e + 1])).all())
    if payload:  # the general kernel's bytes for the same token, wherever that one put it
        tg, kg = (general[2] >= 0).nonzero(as_tuple=True)
        q, s = torch.zeros(T, H, dtype=torch.uint8, device="cuda"), torch.zeros(T, H // 128, device="cuda")
        q[tg], s[tg] = general[0][general[2].long()[tg, kg]], general[1][general[2].long()[tg, kg]]
        seen = torch.zeros(T, dtype=torch.bool, device="cuda")
        seen[tg] = True
        keep = seen[t]
        assert torch.equal(local[0][rows][keep], q[t][keep]) and torch.equal(local[1][rows][keep], s[t][keep])
    else:
        assert torch.equal(local[0][rows].view(torch.bfloat16), x[t])


@pytest.mark.parametrize("T,H,K", [(1, 128, 1), (3, 640, 16), (61, 7168, 8), (295, 256, 9), (1500, 384, 4), (5000, 128, 16), (4001, 2176, 1)])
def test_local_combine_over_column_ranges(nv, T, H, K):
    """Few tokens: a token's row is cut into column ranges for several CTAs.  fp32 sums of K products, one rounding to bf16."""
    from nvshmem_b200.ops.moe import MoeDispatchCombine
    torch.manual_seed(T + H + K)
    moe = MoeDispatchCombine(T, H, K, 32)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    w = torch.rand(T, K, device="cuda")
    idx = torch.rand(T, 32, device="cuda").topk(K, dim=-1).indices.to(torch.int32).contiguous()
    idx[T // 2, K - 1] = -1
    recv, _ = moe.dispatch(x, idx)
    moe.expert_out.copy_(recv)
    want = x.double() * (w * (idx >= 0)).double().sum(-1, keepdim=True)
    got = moe.combine(idx, w).double()
    # one rounding to bf16 (8 significant bits: half a unit in the last place is at most 2^-8 of the value) and the rounding
    # of K fp32 products and sums, all of one sign
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -8 + 2 * K * 2.0 ** -24) + 1e-30).all())
    moe.close()


@pytest.mark.parametrize("payload", ["bf16", "fp8"])
@pytest.mark.parametrize("T,H,K,E", [(1, 128, 1, 8), (61, 7168, 8, 32), (300, 256, 16, 64), (700, 2176, 9, 16), (5000, 128, 4, 256)])
def test_exchange_of_several_pes_run_on_one(nv, T, H, K, E, payload):
    """The kernels that several PEs run (cooperative, with barriers), on one PE against the ones without barriers: same
    offsets, same rows per token, and the same bits from combine (builds for up to 8 and up to 16 choices)."""
    from nvshmem_b200.ops import fused_gemm as fg
    from nvshmem_b200.ops.moe import MoeDispatchCombine
    torch.manual_seed(T + H)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    idx = torch.randint(-1, E, (T, K), device="cuda", dtype=torch.int32)
    wt = torch.rand(T, K, device="cuda")
    rows = torch.randn(T, K, H, device="cuda").to(torch.bfloat16)  # an expert's answer for every (token, choice)
    valid = idx >= 0
    res = []
    for several in (False, True):
        moe = MoeDispatchCombine(T, H, K, E, payload=payload)
        moe._use_kernels_for_several_pes(several)
        for _ in range(2):  # the second call finds what the first one left in flags and scratch
            recv, offsets = moe.dispatch(x, idx)
            at = moe.slot_map[valid].long()
            moe.expert_out[at] = rows[valid]
            out = moe.combine(idx, wt)
        names = [n for n, _ in _kernels(lambda: (moe.dispatch(x, idx), moe.combine(idx, wt)))]
        assert ("15dispatch_kernel" in names[0]) == several, names
        fg.check_errors()
        res.append((offsets.clone(), recv.view(torch.uint8)[at].clone(), moe.recv_scale[at].clone() if payload == "fp8" else None, moe.src_offsets.clone(), out.clone()))
        moe.close()
    one, general = res
    for k in (0, 1, 3, 4):
        assert torch.equal(one[k], general[k]), k
    if payload == "fp8":
        assert torch.equal(one[2], general[2])


@pytest.mark.parametrize("M,N,K", [(256, 512, 192), (1152, 2048, 64)])
def test_fused_ops_with_a_transposed_weight(nv, M, N, K):
    """``w_t=True`` of the ops that the backward passes on several PEs use, on one."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    want = fg.gemm(x, w)
    ag = fg.AllGatherGemm(M, K)
    ag.shard.copy_(x)
    for got in (ag(w.t().contiguous(), w_t=True), fg.GemmReduceScatter(M, N, mode="rs")(x, w.t().contiguous(), w_t=True),
                fg.GemmReduceScatter(M, N, mode="ar")(x, w.t().contiguous(), w_t=True)):
        assert torch.equal(got, want)
    fg.check_errors()


@pytest.mark.parametrize("limit", [1, 3, 4, 7, 8, 100])
@pytest.mark.parametrize("T,payload", [(64, "bf16"), (900, "bf16"), (900, "fp8")])
def test_max_ctas_holds_for_every_kernel_of_the_exchange(nv, T, payload, limit):
    """The grids of a captured dispatch and combine keep to `max_ctas` (the routing kernel too), and the rows land as they do
    without a limit."""
    from nvshmem_b200.ops.moe import MoeDispatchCombine
    torch.manual_seed(T + limit)
    H, K, E = 256, 5, 24
    moe = MoeDispatchCombine(T, H, K, E, payload=payload)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    idx = torch.randint(-1, E, (T, K), device="cuda", dtype=torch.int32)
    wt = torch.rand(T, K, device="cuda")
    valid = idx >= 0
    moe.dispatch(x, idx)
    want_rows = moe.recv_raw[moe.slot_map[valid].long()].clone()
    want_offsets, want_out = moe.expert_offsets.clone(), None
    moe.expert_out.copy_(torch.randn(moe.cap_rows, H, device="cuda"))
    by_slot = moe.expert_out[moe.slot_map.clamp(min=0).long()].clone()
    want_out = moe.combine(idx, wt).clone()
    moe._dispatch_args.max_ctas = moe._combine_args.max_ctas = limit
    grids = [ctas for _, ctas in _kernels(lambda: (moe.dispatch(x, idx), moe.combine(idx, wt)))]
    assert len(grids) == (2 if T * K <= 2048 else 3) and max(grids) <= limit, grids
    moe.dispatch(x, idx)
    torch.cuda.synchronize()
    assert torch.equal(moe.expert_offsets, want_offsets) and bool((moe.slot_map[~valid] == -1).all())
    rows = moe.slot_map[valid].long()
    e = idx[valid].long()
    assert torch.equal(rows.sort().values, torch.arange(rows.numel(), device="cuda"))
    assert bool(((rows >= want_offsets[e]) & (rows < want_offsets[e + 1])).all())
    assert torch.equal(moe.recv_raw[rows], want_rows)
    moe.expert_out[rows] = by_slot[valid]
    assert torch.equal(moe.combine(idx, wt), want_out)
    moe.close()


@pytest.mark.parametrize("T", [100, 700])
def test_sizes_of_the_exchange_count_as_they_stand_at_the_call(nv, T):
    """`cap_rows` lowered after the first call: rows beyond it are dropped and reported; `T` lowered: a shorter batch."""
    from nvshmem_b200.ops import fused_gemm as fg
    from nvshmem_b200.ops.moe import MoeDispatchCombine
    torch.manual_seed(T)
    H, K, E = 256, 4, 8
    moe = MoeDispatchCombine(T, H, K, E)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    idx = torch.rand(T, E, device="cuda").topk(K, dim=-1).indices.to(torch.int32).contiguous()
    wt = torch.full((T, K), 0.25, device="cuda")
    moe.dispatch(x, idx)
    assert fg.take_error() == 0 and int(moe.slot_map.max()) == T * K - 1
    moe.cap_rows = cap = T * K // 3
    moe.recv_raw.fill_(9)
    moe.dispatch(x, idx)
    assert fg.take_error() == 2 and int(moe.slot_map.max()) == cap - 1 and bool((moe.recv_raw[cap:] == 9).all())
    moe.cap_rows, moe.T = T * K, T // 2
    recv, offsets = moe.dispatch(x[:T // 2], idx[:T // 2])
    assert fg.take_error() == 0 and int(offsets[-1]) == T // 2 * K
    moe.expert_out.copy_(recv)
    moe.out.fill_(9)
    out = moe.combine(idx[:T // 2], wt[:T // 2])
    torch.cuda.synchronize()
    assert torch.equal(out[:T // 2], x[:T // 2]) and bool((out[T // 2:] == 9).all())
    moe.close()


@pytest.mark.parametrize("T,payload", [(40, "bf16"), (1200, "bf16"), (1200, "fp8")])
def test_captured_calls_replay_on_new_inputs(nv, T, payload):
    """Dispatch (one and two kernels), grouped GEMM, combine, a small GEMM, one with a finer last wave and a collective in one
    CUDA graph, among them launches that overlap the kernel before: replays on new inputs equal eager calls."""
    from nvshmem_b200.ops import fused_gemm as fg
    from nvshmem_b200.ops.moe import MoeDispatchCombine
    torch.manual_seed(T)
    H, K, E = 512, 4, 8
    moe = MoeDispatchCombine(T, H, K, E, payload=payload)
    w = (torch.randn(E, H, H, device="cuda") * 0.05).to(torch.bfloat16)
    big_w = (torch.randn(2304, H, device="cuda") * 0.05).to(torch.bfloat16)
    src, dst = nv.tensor((20011,), torch.float32), nv.tensor((20011,), torch.float32)
    x, big = torch.empty(T, H, dtype=torch.bfloat16, device="cuda"), torch.empty(2176, H, dtype=torch.bfloat16, device="cuda")
    idx, wt = torch.empty(T, K, dtype=torch.int32, device="cuda"), torch.empty(T, K, device="cuda")

    def fill(seed):
        torch.manual_seed(seed)
        x.copy_(torch.randn(T, H, device="cuda"))
        big.copy_(torch.randn(2176, H, device="cuda"))
        idx.copy_(torch.rand(T, E, device="cuda").topk(K).indices)
        wt.copy_(torch.rand(T, K, device="cuda"))
        src.copy_(torch.randn(20011, device="cuda"))

    def calls():
        recv, offs = moe.dispatch(x, idx)
        if payload == "bf16":
            fg.grouped_gemm(recv, w, offs, out=moe.expert_out)
        else:
            moe.expert_out.copy_(moe.dequantized(moe.cap_rows))
        y = fg.gemm(fg.gemm(big, big_w)[:256, :H].contiguous(), big_w[:256])
        nv.reduce(0, dst, src, "sum")
        return moe.combine(idx, wt), y, dst

    fill(1)
    calls()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = calls()
    torch.cuda.synchronize()
    for seed in (2, 3):
        fill(seed)
        want = [t.clone() for t in calls()]
        for t in out:
            t.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        fg.check_errors()
        for got, ref in zip(out, want):
            assert torch.equal(got, ref)
    moe.close()
    nv.free_tensor(src)
    nv.free_tensor(dst)


@pytest.mark.parametrize("payload,tol", [("bf16", 0.03), ("fp8", 0.08)])
def test_moe_block_matches_fp32_reference_single_pe(nv, payload, tol):
    """Router + dispatch + expert MLPs + combine against a plain PyTorch fp32 version of the same block."""
    from nvshmem_b200.models.moe_block import ExpertParallelMoE, reference_forward
    from nvshmem_b200.ops import fused_gemm as fg
    T, H, F, E, K = 192, 256, 384, 8, 2
    block = ExpertParallelMoE(T, H, F, E, K, payload=payload, seed=3, wait_limit_ms=5000)
    torch.manual_seed(17)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    got = block(x)
    torch.cuda.synchronize()
    fg.check_errors()
    want = reference_forward(x, block.router, block.w_in, block.w_out, K)
    err = (got.float() - want).abs().max().item()
    assert err <= tol * want.abs().max().item() + 1e-3, (payload, err, want.abs().max().item())
    block.close()


def test_copy_engine_collectives_on_one_pe(nv):
    """The copy-engine variants of fcollect / alltoall / broadcast (one memcpy per member + barrier)."""
    n = 1 << 16
    src = nv.tensor((n,), torch.float32)
    dst = nv.tensor((n,), torch.float32)
    src.copy_(torch.arange(n, device="cuda", dtype=torch.float32))
    nv.set_ce_collectives(1)
    try:
        for coll in ("fcollect", "alltoall", "broadcast"):
            dst.zero_()
            nv.collective_on_buffer(coll, 0, dst, src, op="sum")
            nv.barrier_all()
            torch.cuda.synchronize()
            assert torch.equal(dst, src), coll
    finally:
        nv.set_ce_collectives(0)
    assert nv.error_bits() == 0
    nv.free_tensor(src)
    nv.free_tensor(dst)


def test_device_code_in_a_separately_loaded_module():
    """A cubin built from tests/data/device_module_kernel.cu is loaded with the driver API, given the library state with
    nvshmemx_cumodule_init and puts to PE 0 (itself).  Runs as a child process with its own initialisation."""
    from tests._mp import run_workers
    run_workers("device_module_via_driver_api", 1, gpu=True, env={"NVSHMEM_DISABLE_NVLS": "1"}, timeout=300)
