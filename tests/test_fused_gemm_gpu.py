"""Numerics of the tcgen05 GEMM kernel against a plain PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(x, w):
    return x.float() @ w.float().t()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 256), (256, 512, 192), (1024, 768, 512), (2048, 256, 3584), (384, 1280, 1088)])
def test_gemm_matches_fp32_reference(M, N, K):
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    out = fg.gemm(x, w)
    torch.cuda.synchronize()
    fg.check_errors()
    ref = _ref(x, w)
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    # bf16 output rounding: half an ulp of the largest magnitude, plus accumulation-order slack
    assert err <= scale * 2 ** -7 + 1e-3, f"max abs err {err} at scale {scale}"


def test_gemm_structured_operands_catch_layout_errors():
    """Operands with distinct values per row and per k make a wrong swizzle or descriptor visible."""
    from nvshmem_b200.ops import fused_gemm as fg
    M, N, K = 256, 256, 128
    x = torch.zeros(M, K, device="cuda")
    w = torch.zeros(N, K, device="cuda")
    x[torch.arange(M), torch.arange(M) % K] = 1.0          # row i picks column i % K of w^T
    w += (torch.arange(N, device="cuda").float()[:, None] % 7 + 1) * (torch.arange(K, device="cuda").float()[None, :] % 5 + 1)
    out = fg.gemm(x.to(torch.bfloat16), w.to(torch.bfloat16))
    torch.cuda.synchronize()
    ref = _ref(x.to(torch.bfloat16), w.to(torch.bfloat16))
    assert torch.equal(out.float(), ref.to(torch.bfloat16).float())


def test_gemm_rejects_bad_shapes():
    from nvshmem_b200.ops import fused_gemm as fg
    x = torch.zeros(100, 64, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(256, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(fg.FusedGemmError):
        fg.gemm(x, w)


def test_gemm_with_few_ctas_walks_all_tiles():
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(5)
    x = torch.randn(1024, 320, device="cuda").to(torch.bfloat16)
    w = torch.randn(1024, 320, device="cuda").to(torch.bfloat16)
    out = fg.gemm(x, w, max_ctas=3)  # 32 tiles on 3 CTAs: exercises the persistent loop and both TMEM buffers
    torch.cuda.synchronize()
    ref = _ref(x, w)
    assert (out.float() - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -7 + 1e-3


@pytest.mark.parametrize("G,N,K,act", [(4, 256, 128, None), (7, 512, 320, None), (5, 512, 256, "swiglu"), (32, 1024, 512, "swiglu")])
def test_grouped_gemm_over_ragged_groups(G, N, K, act):
    """Rows fall into groups of uneven size (some empty, none a multiple of 128); each group has its own weight.
    The group boundaries are read by the kernel from device memory."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(G * 1000 + N + K)
    sizes = torch.randint(0, 400, (G,))
    sizes[G // 2] = 0                      # an empty group in the middle
    sizes[0] = 129                         # one full block and a block of one row
    offs = torch.zeros(G + 1, dtype=torch.int32)
    offs[1:] = sizes.cumsum(0).to(torch.int32)
    rows = int(offs[-1])
    cap = rows + 77                        # the buffers are larger than what the groups use
    x = torch.randn(cap, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N, K, device="cuda") * 0.05).to(torch.bfloat16)
    out_cols = N // 2 if act == "swiglu" else N
    out = torch.full((cap, out_cols), 7.0, dtype=torch.bfloat16, device="cuda")
    w_used = fg.interleave_gate_up(w) if act == "swiglu" else w
    fg.grouped_gemm(x, w_used, offs.cuda(), out=out, act=act)
    torch.cuda.synchronize()
    fg.check_errors()
    assert bool((out[rows:] == 7.0).all()), "rows beyond the last group were written"
    for g in range(G):
        lo, hi = int(offs[g]), int(offs[g + 1])
        if hi == lo:
            continue
        ref = x[lo:hi].float() @ w[g].float().t()
        if act == "swiglu":
            ref = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
        err = (out[lo:hi].float() - ref).abs().max().item()
        assert err <= ref.abs().max().item() * 2 ** -6 + 2e-3, (g, lo, hi, err)


def test_interleave_gate_up_orders_rows_in_blocks_of_32():
    from nvshmem_b200.ops import fused_gemm as fg
    F, K = 64, 4
    w = torch.arange(2 * F, dtype=torch.float32).view(2 * F, 1).expand(2 * F, K).contiguous()
    r = fg.interleave_gate_up(w)[:, 0].tolist()
    assert r[:32] == list(range(0, 32)) and r[32:64] == list(range(F, F + 32)) and r[64:96] == list(range(32, 64)) and r[96:] == list(range(F + 32, 2 * F))


@pytest.mark.parametrize("x_t,w_t", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (384, 512, 192), (256, 256, 64), (512, 1280, 1088)])
def test_gemm_reads_transposed_operands_as_they_lie(M, N, K, x_t, w_t):
    """Operands stored with K outermost, for one CTA per tile (odd number of 128-row blocks) and for CTA pairs: the same
    MMAs on the same values in the same order, so the result equals the one of the K-major operands bit by bit."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    got = fg.gemm(x.t().contiguous() if x_t else x, w.t().contiguous() if w_t else w, x_t=x_t, w_t=w_t)
    want = fg.gemm(x, w)
    torch.cuda.synchronize()
    fg.check_errors()
    assert torch.equal(got, want)
    ref = _ref(x, w)
    assert (got.float() - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -7 + 1e-3


@pytest.mark.parametrize("act", [None, "gelu_tanh"])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 128), (128, 1024, 2048), (256, 512, 8192), (128, 3584, 8128), (384, 1536, 704), (512, 3584, 1984), (1152, 2816, 192),
                                   (128, 8192, 3584), (1280, 2816, 1984)])
def test_products_of_few_tiles(M, N, K, act):
    """Tiles of 64, 128 and 256 columns, the single wave they have to fit and the persistent kernel beyond.  fp32 sums in another order differ by about sqrt(K) 2^-24 of the operands' scale, far below the
    rounding to bf16 (2^-8 of the value at most)."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    room = 1e-4 * want.abs().max()
    if act:
        # the hardware tanh is good to 2^-10.99 relative; its share of x is at most half of that
        room = room + want.abs() * 2 ** -11
        want = torch.nn.functional.gelu(want, approximate="tanh")
    for x_t, w_t in ((False, False), (True, True), (False, True)):
        got = fg.gemm(x.t().contiguous() if x_t else x, w.t().contiguous() if w_t else w, act=act, x_t=x_t, w_t=w_t)
        torch.cuda.synchronize()
        fg.check_errors()
        assert bool(((got.double() - want).abs() <= want.abs() * 2 ** -8 + room).all()), (x_t, w_t)
    assert torch.equal(fg.gemm(x, w, act=act), fg.gemm(x, w, act=act))


@pytest.mark.parametrize("M,N,K,act", [(128, 1024, 2048, None), (256, 512, 8192, "gelu_tanh"), (512, 3584, 1024, None), (1024, 1024, 1024, None), (2048, 2560, 4096, None),
                                       (4096, 3584, 2048, "gelu_tanh")])
def test_bits_of_a_row_do_not_depend_on_the_size_of_the_call(M, N, K, act):
    """One chain of sums over K for every element: a part of the rows or of the weights gives the bits that the whole product
    has, whichever kernel and tile width each of them takes (few tiles, one CTA, pairs, a last wave cut finer)."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    whole = fg.gemm(x, w, act=act)
    assert torch.equal(whole[:128], fg.gemm(x[:128], w, act=act, max_ctas=1))
    for rows in {128, M // 2 // 128 * 128} - {0}:
        assert torch.equal(whole[:rows], fg.gemm(x[:rows], w, act=act)), rows
        assert torch.equal(whole[M - rows:], fg.gemm(x[M - rows:], w, act=act)), rows
    for cols in (256, N // 2 // 256 * 256):
        assert torch.equal(whole[:, N - cols:], fg.gemm(x, w[N - cols:], act=act)), cols
    assert torch.equal(whole, fg.gemm(x.t().contiguous(), w.t().contiguous(), act=act, x_t=True, w_t=True))
    fg.check_errors()


@pytest.mark.parametrize("M,N,K,act", [(2176, 2304, 192, None), (4480, 3584, 128, "gelu_tanh"), (2048, 4864, 1024, None), (3328, 3072, 2048, None), (1152, 8448, 64, None)])
def test_odd_row_blocks_in_pairs_and_a_last_wave_cut_finer(M, N, K, act):
    """More than a wave of tiles: an odd number of row blocks rounded up to pairs (the added block is neither loaded nor
    stored), and the tiles of the last, partial wave on the kernel for few tiles; every element against float64."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    room = 1e-4 * want.abs().max()  # order of the fp32 sums, as above
    if act:
        room = room + want.abs() * 2 ** -11
        want = torch.nn.functional.gelu(want, approximate="tanh")
    guard = torch.full((M + 128, N), 7.0, dtype=torch.bfloat16, device="cuda")
    for x_t, w_t in ((False, False), (True, True)):
        got = fg.gemm(x.t().contiguous() if x_t else x, w.t().contiguous() if w_t else w, out=guard[:M], act=act, x_t=x_t, w_t=w_t)
        torch.cuda.synchronize()
        fg.check_errors()
        assert bool(((got.double() - want).abs() <= want.abs() * 2 ** -8 + room).all()), (x_t, w_t)
        assert bool((guard[M:] == 7.0).all()), "rows past the output were written"


@pytest.mark.parametrize("M,N,K", [(4224, 8192, 64), (4224, 8192, 128), (8320, 8192, 64), (8320, 8192, 128), (4480, 3584, 64)])
def test_added_row_blocks_leave_the_staging_buffers_alone(M, N, K):
    """Short K: the next accumulator is ready at once, so the tile after a stored one finds its last store still in flight.  Every
    element against float64, new inputs every time."""
    from nvshmem_b200.ops import fused_gemm as fg
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    for _ in range(60):
        x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
        w = (torch.randn(N, K, device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
        got = fg.gemm(x, w)
        want = x.double() @ w.double().t()
        # one rounding to bf16 (2^-8 of the value), K products of 2^-24 each of the largest sum
        assert bool(((got.double() - want).abs() <= want.abs() * 2 ** -8 + K * 2.0 ** -24 * want.abs().max()).all())
    fg.check_errors()


def test_gemm_is_a_threads_first_cuda_call():
    """A thread that has not touched the GPU before (as an autograd worker may not have) calls the GEMM first."""
    import threading
    from nvshmem_b200.ops import fused_gemm as fg
    x = torch.randn(128, 64, device="cuda").to(torch.bfloat16)
    w = torch.randn(256, 64, device="cuda").to(torch.bfloat16)
    want = fg.gemm(x, w)
    out = torch.empty_like(want)
    torch.cuda.synchronize()
    failed = []

    def work():
        try:
            fg.gemm(x, w, out=out)
        except Exception as e:  # noqa: BLE001 - handed to the main thread
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not failed and torch.equal(out, want)


@pytest.mark.parametrize("sizes,N,K,act", [([1030, 0, 256, 257], 512, 320, None), ([1, 0, 0, 33], 256, 64, "gelu_tanh"), ([512, 513, 31, 225], 768, 128, "swiglu"),
                                           ([0, 0, 0, 0], 256, 64, None), ([15, 16, 17, 32], 1024, 1088, "swiglu"), ([300] * 40, 256, 128, None)])
def test_grouped_gemm_chunk_edges(sizes, N, K, act):
    """Row counts at the edges of the 32-row steps and 256-row chunks, empty groups at either end, more groups than one
    warp scans at once, every fused activation; rows outside the groups stay as they were."""
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(sum(sizes) + N + K)
    G, first = len(sizes), 5                       # the first group does not start at row 0
    offs = torch.zeros(G + 1, dtype=torch.int32)
    offs[1:] = torch.tensor(sizes).cumsum(0).to(torch.int32)
    offs += first
    cap = int(offs[-1]) + 3
    x = torch.randn(cap, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N, K, device="cuda") * 0.05).to(torch.bfloat16)
    out_cols = N // 2 if act == "swiglu" else N
    out = torch.full((cap, out_cols), 7.0, dtype=torch.bfloat16, device="cuda")
    fg.grouped_gemm(x, fg.interleave_gate_up(w) if act == "swiglu" else w, offs.cuda(), out=out, act=act)
    torch.cuda.synchronize()
    fg.check_errors()
    assert bool((out[:first] == 7.0).all()) and bool((out[int(offs[-1]):] == 7.0).all())
    for g in range(G):
        lo, hi = int(offs[g]), int(offs[g + 1])
        if hi == lo:
            continue
        ref = x[lo:hi].double() @ w[g].double().t()
        room = 1e-4 * ref.abs().max()              # order of the fp32 sums
        if act == "swiglu":
            # silu' is at most 1.1: the room of the gate, times the largest up value, and the other way round
            room = 2.2 * room * ref.abs().max()
            ref = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
        elif act:
            room = room + ref.abs() * 2 ** -11     # the hardware tanh
            ref = torch.nn.functional.gelu(ref, approximate="tanh")
        assert bool(((out[lo:hi].double() - ref).abs() <= ref.abs() * 2 ** -8 + room).all()), (g, lo, hi)


def test_grouped_gemm_on_one_cta_and_an_odd_number():
    """`max_ctas` below two leaves no CTA pair; an odd limit leaves one CTA out.  Same values either way."""
    import ctypes as C
    from nvshmem_b200.ops import fused_gemm as fg
    torch.manual_seed(3)
    x = torch.randn(600, 128, device="cuda").to(torch.bfloat16)
    w = (torch.randn(3, 512, 128, device="cuda") * 0.05).to(torch.bfloat16)
    offs = torch.tensor([0, 290, 291, 600], dtype=torch.int32, device="cuda")
    want = fg.grouped_gemm(x, w, offs)
    for limit in (1, 3):
        out = torch.zeros_like(want)
        a = fg._Args()
        a.A, a.B, a.out = x.data_ptr(), w.data_ptr(), out.data_ptr()
        a.M, a.N, a.K, a.npes, a.mode, a.epoch, a.max_ctas = 600, 512, 128, 1, fg.MODES["grouped"], 1, limit
        a.group_offsets, a.groups, a.error_flag = offs.data_ptr(), 3, fg._error_flag(x.device).data_ptr()
        assert fg.fused_lib().bshmem_fused_gemm(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        fg.check_errors()
        assert torch.equal(out, want)
    big = torch.randn(1152, 64, device="cuda").to(torch.bfloat16)     # nine row blocks, odd limits for the plain product as well
    wb = torch.randn(512, 64, device="cuda").to(torch.bfloat16)
    assert torch.equal(fg.gemm(big, wb, max_ctas=5), fg.gemm(big, wb, max_ctas=1))
