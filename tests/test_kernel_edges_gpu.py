"""Kernels at the sizes where a tile, a ring or a path of the dispatch ends, against plain fp32 (or fp64) torch."""
import pytest
import torch

from prime_b200.ops import attention as A
from prime_b200.ops import kernels as ops

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _attention_case(starts, M, H, KV, hd, seed=0):
    torch.manual_seed(seed)
    qkv = (torch.randn(M, (H + 2 * KV) * hd, device="cuda") * 0.7).bfloat16()
    ss = torch.zeros(M, dtype=torch.int32)
    for s, e in zip(starts, list(starts[1:]) + [M]):
        ss[s:e] = s
    ss = ss.cuda()
    o, lse2 = A.attention_fwd(qkv, ss, H, KV, hd)
    x = qkv.float().requires_grad_(True)
    ref = A.attention_reference(x, ss, H, KV, hd)
    # bf16 P (2^-9) and output (2^-9)
    assert _rel(o, ref.detach()) < 1e-2
    _, lse_ref = A.attention_fwd(qkv.cpu(), ss.cpu(), H, KV, hd)
    assert (lse2.cpu() - lse_ref).abs().max().item() < 1e-2
    dout = (torch.randn(M, H * hd, device="cuda") * 0.5).bfloat16()
    table = ops.rope_table(M, hd, 10000.0, "cuda")
    g = A.attention_bwd(qkv, o, dout, lse2, ss, H, KV, hd, rope_table=table, seq_len=M)
    ops.check_status()
    (gref,) = torch.autograd.grad(ref, x, dout.float())
    gref = ops.rope_(gref.cpu(), table.cpu(), M, H + KV, hd, backward=True).cuda()
    qk, v = qkv[:, : (H + KV) * hd].float().abs().max(), qkv[:, (H + KV) * hd:].float().view(M, KV, hd).repeat_interleave(H // KV, 1)
    dp = (dout.float().view(M, H, hd) * v).sum(-1).abs().max()
    for cols in (slice(0, H * hd), slice(H * hd, (H + KV) * hd), slice((H + KV) * hd, None)):
        # a row that sees only itself has P = 1 and dS = 0: nothing but rounding in dQ and dK, a bf16 unit (2^-8) of P and one of O at most
        if len(starts) < M or cols.stop is None:
            assert _rel(g[:, cols], gref[:, cols]) < 2e-2
        else:
            assert g[:, cols].float().abs().max().item() <= 2 * 2.0 ** -8 * (H // KV) * (dp * qk).item() * hd ** -0.5      # (false for NaN)


# The forward takes two 128-row query tiles at a time: one tile only, an odd number of them, a last tile of one row, documents that
# start in the second tile of a pair (its kv tiles begin later), at tile edges and one row beside them, and one row per document
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("M,starts", [(1, (0,)), (128, (0,)), (129, (0,)), (257, (0, 256)), (640, (0, 128, 384)), (900, (0, 127, 129, 300, 511, 513)),
                                      (512, tuple(range(512)))])
def test_attention_tile_pairs(hd, M, starts):
    _attention_case(starts, M, 4, 2, hd)


# More pairs of query tiles than SMs, so that CTAs take over the work of others, rings wrap and heads change on the way; odd tile count
@pytest.mark.parametrize("hd,H,KV", [(64, 16, 4), (128, 12, 3), (32, 16, 16)])
def test_attention_more_pairs_than_sms(hd, H, KV):
    M = 128 * 33 - 5
    _attention_case((0, 700, 1400, 1401, 3000), M, H, KV, hd, seed=3)


# recorded and replayed on other inputs, behind a kernel that is still running: work is drawn anew in every replay
def test_attention_of_wide_heads_in_a_graph():
    M, H, KV, hd = 128 * 41, 16, 4, 128
    torch.manual_seed(0)
    qkv = (torch.randn(M, (H + 2 * KV) * hd, device="cuda") * 0.7).bfloat16()
    ss = A.seq_start_from_batch(1, M, "cuda")
    o, lse2, g = torch.empty(M, H * hd, device="cuda", dtype=torch.bfloat16), torch.empty(H, M, device="cuda"), torch.empty_like(qkv)
    dout = torch.randn(M, H * hd, device="cuda").bfloat16()

    def step():
        A.attention_fwd(qkv, ss, H, KV, hd, out=o, lse2=lse2)
        A.attention_bwd(qkv, o, dout, lse2, ss, H, KV, hd, dqkv=g)
    step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for seed in (1, 2):
        qkv.copy_((torch.randn(M, qkv.shape[1], device="cuda", generator=torch.Generator("cuda").manual_seed(seed)) * 0.7).bfloat16())
        step()
        want_o, want_l, want_g = o.clone(), lse2.clone(), g.clone()
        o.zero_(), lse2.zero_(), g.zero_()
        graph.replay()
        ops.check_status()
        assert torch.equal(o, want_o) and torch.equal(lse2, want_l) and _rel(g, want_g) < 1e-3      # dQ is summed in the order of arrival


@pytest.mark.parametrize("hd,parts", [(64, 1), (128, 2)])
def test_attention_backward_takes_row_dots_in_parts(hd, parts):
    torch.manual_seed(0)
    M, H, KV = 700, 4, 2
    qkv = (torch.randn(M, (H + 2 * KV) * hd, device="cuda") * 0.7).bfloat16()
    ss = A.seq_start_from_batch(1, M, "cuda")
    o, lse2 = A.attention_fwd(qkv, ss, H, KV, hd)
    dh = torch.randn(M, 512, device="cuda").bfloat16()
    wo = (torch.randn(512, H * hd, device="cuda") * 512 ** -0.5).bfloat16()
    do = torch.empty(M, H * hd, device="cuda", dtype=torch.bfloat16)
    dots = A.row_dots_buffer(do.device, M, H, parts)
    assert ops.gemm_rowdot(dh, wo, do, o, dots, hd, b_mn=True)
    want_dots = (dh.float() @ wo.float() * o.float()).reshape(M, H, parts, 64).sum(-1).permute(1, 2, 0)
    assert _rel(dots.view(H, parts, M), want_dots) < 1e-3
    got = A.attention_bwd(qkv, o, do, lse2, ss, H, KV, hd, row_dots=dots.clone())
    want = A.attention_bwd(qkv, o, do, lse2, ss, H, KV, hd)
    ops.check_status()
    assert _rel(got, want) < 1e-2                            # the sums are over dO before and after its rounding to bf16


# Tile widths of the CTA-pair GEMM: outputs for which each width is chosen, with ragged last rows, a last tile that is cut inside a
# 64-column box, and every epilogue
@pytest.mark.parametrize("M,N,K", [(512, 256, 128), (520, 1024, 1024), (2331, 1024, 320), (2331, 1000, 256), (700, 1416, 512), (8192, 256, 256),
                                   (1300, 3072, 512)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_tile_widths(M, N, K, b_mn):
    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    b = w.t().contiguous() if b_mn else w
    ref = x.float() @ w.float().t()
    r = torch.randn(M, N, device="cuda").bfloat16()
    wide = torch.full((M, N + 8), 7.0, device="cuda").bfloat16()
    ops.gemm(x, b, out=wide[:, :N], b_mn=b_mn)
    assert _rel(wide[:, :N], ref) < 1e-2 and bool((wide[:, N:] == 7).all())
    assert _rel(ops.gemm(x, b, residual=r, b_mn=b_mn), ref + r.float()) < 1e-2
    f = torch.randn(M, N, device="cuda")
    want = f + ref
    assert _rel(ops.gemm(x, b, out=f, residual=f, b_mn=b_mn), want) < 1e-3
    assert _rel(ops.gemm(x, b, out_dtype=torch.float32, b_mn=b_mn), ref) < 1e-3
    if N % 64 == 0 and b_mn:
        o, dots = torch.empty_like(r), torch.empty(N // 64 * M, device="cuda")
        assert ops.gemm_rowdot(x, b, o, r, dots, 64, b_mn=True)
        assert _rel(o, ref) < 1e-2
        assert _rel(dots.view(N // 64, M), (ref * r.float()).view(M, N // 64, 64).sum(-1).t()) < 1e-3
    ops.check_status()


@pytest.mark.parametrize("M", [512, 777, 2331, 8192])
@pytest.mark.parametrize("F", [192, 704, 1536])
def test_swiglu_epilogues_of_narrow_tiles(M, F):
    torch.manual_seed(0)
    K = 256
    x = torch.randn(M, K, device="cuda").bfloat16()
    w13 = (torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16()
    h13, act = torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16), torch.empty(M, F, device="cuda", dtype=torch.bfloat16)
    ops.gemm_swiglu(x, w13, h13, act)
    ref = x.float() @ w13.float().t()
    assert _rel(h13, ref) < 1e-2
    assert _rel(act, torch.nn.functional.silu(ref[:, :F]) * ref[:, F:]) < 1e-2
    w2 = (torch.randn(128, F, device="cuda") * F ** -0.5).bfloat16()
    dout = torch.randn(M, 128, device="cuda").bfloat16()
    gb, ub, d = h13[:, :F].float(), h13[:, F:].float(), dout.float() @ w2.float()
    sg = torch.sigmoid(gb)
    want = torch.cat([d * ub * sg * (1 + gb * (1 - sg)), d * gb * sg], 1)
    ops.gemm_dswiglu(dout, w2, h13)
    ops.check_status()
    assert _rel(h13, want) < 1.5e-2


# heads whose columns divide the epilogue's 128-column rounds and one (192) whose table differs from round to round; rows that wrap
# around the positions inside a tile
@pytest.mark.parametrize("hd", [8, 32, 64, 128, 192])
@pytest.mark.parametrize("M,T", [(600, 200), (2331, 777), (1024, 1024)])
def test_rope_epilogue_heads(hd, M, T):
    torch.manual_seed(0)
    K, H, KV = 192, 768 // hd, 384 // hd
    N = (H + 2 * KV) * hd
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    table = ops.rope_table(T, hd, 10000.0, "cuda")
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_rope(x, w, out, table, T, H + KV, hd)
    ref = ops.rope_((x.float() @ w.float().t()).cpu(), table.cpu(), T, H + KV, hd).cuda()
    ops.check_status()
    assert _rel(out, ref) < 1e-2


# Whole chunks of finite values take a path of their own; a ragged last chunk, one with an infinity or NaN and one whose sum of squares
# overflows take the general one. Zeros, outliers (clamping bins) and tiny values on the first.
@pytest.mark.parametrize("what", ["normal", "outliers", "zeros", "tiny", "constant", "inf", "nan", "huge"])
def test_quantizer_paths(what):
    from prime_b200 import native
    from prime_b200.ops.quant import uniform_8bit_quantize_cuda
    chunk = native.cuda().pb_dl_chunk()
    torch.manual_seed(0)
    x = torch.randn(2 * chunk + 37, device="cuda") * 1e-3
    if what == "outliers":
        x[::97] *= 300
    elif what == "zeros":
        x[:chunk] = 0
    elif what == "tiny":
        x[:chunk] *= 1e-24
    elif what == "constant":
        x[:chunk] = 3.0
    elif what == "inf":
        x[5], x[9] = float("inf"), -float("inf")
    elif what == "nan":
        x[5] = float("nan")
    elif what == "huge":
        x[:chunk] *= 1e30
    q, lut = uniform_8bit_quantize_cuda(x)
    for c in range(3):
        v = x[c * chunk: (c + 1) * chunk]
        n = v.numel()
        ss = (v * v).double().sum()             # squared in fp32: tiny squares vanish, huge ones overflow
        scale = (6 * (ss / max(n - 1, 1)).sqrt() / 256).float().item()
        if not (0 < scale < 3e38):
            scale = 1.0
        t = v.double() / scale
        fin = torch.isfinite(t)
        want = (torch.round(t) + 128).clamp(0, 255)
        got = q[c * chunk: (c + 1) * chunk].double()
        # a value within the fp32 rounding of scale and t of a bin's edge may go either way
        near = ((t - torch.floor(t)) - 0.5).abs() < 1e-5 * t.abs().clamp_min(1)
        assert bool(((got == want) | near | ~fin | (t.abs() > 1e6)).all()), (what, c)
        if not bool(fin.all()) or float(t.abs().max()) > 1e6:
            continue
        for b in (0, 1, 100, 128, 200, 255):
            m = got == b
            if bool(m.any()):
                mean = v[m].double().mean().item()
                # inner bins: offsets in steps of 1/512 of a bin
                assert abs(lut[c, b].item() - mean) <= 2e-3 * scale + 1e-5 * abs(mean), (what, c, b)


# Three outputs of one split product, outputs too large or too short in K to be split (one GEMM each), rows that share 256-row tiles
@pytest.mark.parametrize("K,N,rows", [(8192, 512, (512, 512, 512)), (8192, 512, (1536, 1536)), (4096, 256, (256, 128, 128)), (512, 512, (512, 256)),
                                      (2304, 260, (300, 20, 192, 8))])
def test_gemm_row_parts(K, N, rows):
    torch.manual_seed(0)
    a = torch.randn(K, sum(rows), device="cuda").bfloat16()
    b = torch.randn(K, (N + 7) // 8 * 8, device="cuda").bfloat16()[:, :N]
    outs = ops.gemm_row_parts(a, b, rows)
    ref = a.float().t() @ b.float()
    ops.check_status()
    assert [tuple(o.shape) for o in outs] == [(n, N) for n in rows] and all(o.is_contiguous() and o.dtype == torch.float32 for o in outs)
    assert len({o.untyped_storage().data_ptr() for o in outs}) == len(outs)
    assert _rel(torch.cat(outs), ref) < 1e-3


# dP and the dO . O sums have to come from one and the same dO: rows of V that have a large part in common (here five times their
# spread) leave of dP - D little but what the two terms differ by
@pytest.mark.parametrize("hd", [64, 128])
def test_row_dots_of_the_engine_are_those_of_the_stored_gradient(hd, monkeypatch):
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    T, H = 600, 512 // hd
    eng = FusedLlama(ModelArgs(dim=512, n_layers=1, n_heads=H, ffn_hidden=512, vocab_size=1024, max_seq_len=T, init_mode="normal"),
                     device="cuda", ce_chunk_tokens=512)
    eng.init_weights(seed=3)
    seen = []
    whole = A.attention_bwd

    def check_dots(qkv, o, do, *args, row_dots=None, **kw):
        terms = (do.double() * o.double()).view(T, H, hd // 64, 64)
        want, size = terms.sum(-1).permute(1, 2, 0), terms.abs().sum(-1).permute(1, 2, 0)
        # 64 products of bf16 pairs are exact in fp32, their sum takes 64 roundings
        seen.append(bool(((row_dots.view(H, hd // 64, T).double() - want).abs() <= 64 * 2.0 ** -24 * size).all()))
        return whole(qkv, o, do, *args, row_dots=row_dots, **kw)
    monkeypatch.setattr(A, "attention_bwd", check_dots)
    ids = torch.randint(0, 1024, (1, T + 1), device="cuda")
    eng.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous())
    ops.check_status()
    assert seen == [True]


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_backward_of_values_with_a_common_part(hd):
    torch.manual_seed(0)
    M, H, KV = 1024, 4, 2
    qkv = torch.randn(M, (H + 2 * KV) * hd, device="cuda") * 0.7
    qkv[:, (H + KV) * hd:] += 3.5
    qkv, ss = qkv.bfloat16(), A.seq_start_from_batch(1, M, "cuda")
    o, lse2 = A.attention_fwd(qkv, ss, H, KV, hd)
    dh = torch.randn(M, 512, device="cuda").bfloat16()
    wo = (torch.randn(512, H * hd, device="cuda") * 512 ** -0.5).bfloat16()
    do = torch.empty(M, H * hd, device="cuda", dtype=torch.bfloat16)
    dots = A.row_dots_buffer(do.device, M, H, hd // 64)
    assert ops.gemm_rowdot(dh, wo, do, o, dots, hd, b_mn=True, as_stored=True)
    got = A.attention_bwd(qkv, o, do, lse2, ss, H, KV, hd, row_dots=dots.clone())
    want = A.attention_bwd(qkv, o, do, lse2, ss, H, KV, hd)
    ops.check_status()
    # the two differ in the order of fp32 sums only: now and then a value falls on the other side of a bf16 rounding (2^-8)
    assert _rel(got, want) < 1e-3


# An odd number of 64-feature blocks: one launch where the narrow tiles of the fused kernel pay, GEMM and SwiGLU pass where they do not
@pytest.mark.parametrize("M,F,K,launches", [(1024, 704, 384, 1), (16384, 704, 384, 1), (1024, 704, 1536, 1), (16384, 704, 392, 2), (4096, 320, 1024, 2),
                                            (512, 192, 2048, 3)])
def test_swiglu_of_odd_blocks_is_fused_where_that_is_faster(M, F, K, launches):
    from prime_b200 import native
    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w13 = (torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16()
    h13, act = torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16), torch.empty(M, F, device="cuda", dtype=torch.bfloat16)
    before = native.launch_counter()
    ops.gemm_swiglu(x, w13, h13, act)
    assert native.launch_counter() - before == launches          # (a product that is split over K has a reduce)
    ref = x.float() @ w13.float().t()
    ops.check_status()
    assert _rel(h13, ref) < 1e-2
    assert _rel(act, torch.nn.functional.silu(ref[:, :F]) * ref[:, F:]) < 1e-2


# more heads than SMs, which all come before the second tile of any; a pair and a single tile per head
@pytest.mark.parametrize("M", [128, 300])
def test_attention_of_more_heads_than_sms(M):
    _attention_case((0, 100), M, 160, 80, 72, seed=5)


def _chunks_of_every_kind(n, chunk, grid):
    """Neighbours, and the chunks that one CTA takes one after the other, are of different kinds: clamping bins with members, without
    any (uniform values stay within 1.8 sigma of 3), infinities (general path), zeros, bell-shaped."""
    torch.manual_seed(0)
    x = torch.randn(n, device="cuda") * 1e-3
    for c in range((n + chunk - 1) // chunk):
        v = x[c * chunk: (c + 1) * chunk]
        kind = (c + c // grid) % 5
        if kind == 0:
            v[::97] *= 300
        elif kind == 1:
            v.uniform_(-1e-3, 1e-3)
        elif kind == 2:
            v[1], v[-1] = float("inf"), -float("inf")
        elif kind == 3:
            v.zero_()
    return x


# A CTA carries its table and its clamping bins' sums from chunk to chunk: of three chunks and more per CTA, every one has to come out
# as it does alone
@pytest.mark.parametrize("off", [0, 1])                      # staged through shared memory, and read directly
def test_quantizer_chunks_do_not_depend_on_those_before(off):
    from prime_b200 import native
    from prime_b200.ops.quant import uniform_8bit_quantize_cuda
    chunk = native.cuda().pb_dl_chunk()
    grid = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = (2 * grid + 11) * chunk + 37
    x = torch.empty(n + off, device="cuda")[off:].copy_(_chunks_of_every_kind(n, chunk, grid))
    q, lut = uniform_8bit_quantize_cuda(x)
    for c in range((n + chunk - 1) // chunk):
        s = slice(c * chunk, (c + 1) * chunk)
        q1, lut1 = uniform_8bit_quantize_cuda(x[s])
        assert torch.equal(q[s], q1) and torch.equal(lut[c], lut1[0]), c


# One active rank of a group: it waits for nobody but its own earlier stages. 16 ranks are the most that there may be; their
# codebooks take stage B beyond 48 KB of shared memory.
@pytest.mark.parametrize("world,rank,with_b", [(1, 0, True), (16, 5, False)])
def test_exchange_chunks_do_not_depend_on_those_before(world, rank, with_b):
    import ctypes as C

    from prime_b200 import native
    from prime_b200.parallel import diloco_comm  # noqa: F401  (declares the C signatures)
    lib, ptr = native.cuda(), native.ptr
    chunk = lib.pb_dl_chunk()
    grid = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = (2 * grid + 11) * chunk + 37
    x = _chunks_of_every_kind(n, chunk, grid)
    b = x.flip(0).contiguous().nan_to_num_(0, 0, 0) if with_b else None
    chunks = (n + chunk - 1) // chunk
    epoch = 0

    def exchange(a, b):
        nonlocal epoch
        epoch += 1
        m = a.numel()
        bufs = [torch.zeros(m, dtype=torch.uint8, device="cuda"), torch.zeros((m + chunk - 1) // chunk, 256, device="cuda")]
        bufs += [torch.zeros_like(t) for t in bufs]
        flags, counters, g = torch.zeros(3 * 16, dtype=torch.int32, device="cuda"), torch.zeros(3, dtype=torch.int32, device="cuda"), torch.empty_like(a)
        tables = [(C.c_void_p * world)(*[t.data_ptr()] * world) for t in (*bufs, flags)]
        native.check(lib.pb_dl_allreduce(*tables, world, rank, 1 << rank, epoch, 0, 0, m, ptr(a), ptr(b), 1.0, 0, None, None, None, 0.0, 0.0, ptr(g),
                                         ptr(counters), ptr(ops.status_word(a.device)), 1_000_000_000, native.stream_ptr()), "pb_dl_allreduce")
        return *bufs, g
    q, lut, q2, lut2, g = exchange(x, b)
    ops.check_status()
    for c in range(chunks):
        s = slice(c * chunk, (c + 1) * chunk)
        one = exchange(x[s], b[s] if with_b else None)
        assert all(torch.equal(t, o) for t, o in zip((q[s], lut[c:c + 1], q2[s], lut2[c:c + 1], g[s]), one)), c
    ops.check_status()
