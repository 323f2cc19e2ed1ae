"""Sizes at the edges of the GEMM and attention dispatch: few rows, short K, narrow heads."""
import pytest
import torch

from prime_b200.ops import attention as A
from prime_b200.ops import kernels as ops

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


# 256 rows or columns, K that the slices do not divide, N that is no multiple of the tile
@pytest.mark.parametrize("M,N,K,res", [(256, 256, 8192, True), (256, 704, 4099, False), (1024, 260, 2304, True), (300, 1024, 2048, False)])
def test_split_k_of_narrow_products(M, N, K, res):
    torch.manual_seed(0)
    a = torch.randn(K, (M + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :M]      # row pitch of whole 16-byte units
    b = torch.randn(K, (N + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :N]
    assert ops._splitk_slices(M, N, K, a.device) > 1
    ref = a.float().t() @ b.float()
    for dt in (torch.bfloat16, torch.float32):
        ld = (N + 7) // 8 * 8
        r = torch.randn(M, ld, device="cuda", dtype=dt)[:, :N] if res else None
        out = torch.empty(M, ld, device="cuda", dtype=dt)[:, :N]
        ops.gemm(a, b, out=out, residual=r, a_mn=True, b_mn=True)
        ops.check_status()
        assert _rel(out, ref + (r.float() if res else 0)) < (1e-2 if dt == torch.bfloat16 else 1e-3)


# heads of 8 to 120 columns through the 64- and 128-column kernels; M no multiple of the 128-row tile
@pytest.mark.parametrize("hd", [8, 16, 32, 40, 72, 96, 120])
def test_narrow_heads(hd):
    torch.manual_seed(0)
    B, T, H, KV = 2, 203, 4, 2
    qkv = torch.randn(B * T, (H + 2 * KV) * hd, device="cuda", dtype=torch.bfloat16)
    ss = A.seq_start_from_seqlens([[100, 103], [203]], T, "cuda")
    o, lse2 = A.attention_fwd(qkv, ss, H, KV, hd)
    x = qkv.float().requires_grad_(True)
    ref = A.attention_reference(x, ss, H, KV, hd)
    assert _rel(o, ref.detach()) < 2e-2
    dout = torch.randn(B * T, H * hd, device="cuda", dtype=torch.bfloat16)
    table = ops.rope_table(T, hd, 10000.0, "cuda")
    g = A.attention_bwd(qkv, o, dout, lse2, ss, H, KV, hd, rope_table=table, seq_len=T)
    ops.check_status()
    (gref,) = torch.autograd.grad(ref, x, dout.float())
    gref = ops.rope_(gref.cpu(), table.cpu(), T, H + KV, hd, backward=True).cuda()
    # bf16 P and dS (2^-9 each) against fp32: as for the full-width heads
    assert _rel(g, gref) < 3e-2


# (rows, positions): rows that divide neither tile nor positions, one position, whole tiles; one more rotated head than the epilogue's
# 64-column boxes hold goes to the separate kernel
@pytest.mark.parametrize("M,T", [(777, 200), (512, 1), (1024, 1024)])
@pytest.mark.parametrize("hd,extra", [(8, 0), (16, 0), (32, 0), (8, 1), (16, 1), (32, 1)])
def test_rope_epilogue_narrow_heads(hd, extra, M, T):
    torch.manual_seed(0)
    K, H, KV = 256, 256 // hd, 128 // hd + extra
    N = (H + 2 * KV) * hd
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    table = ops.rope_table(T, hd, 10000.0, "cuda")
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_rope(x, w, out, table, T, H + KV, hd)
    ref = ops.rope_((x.float() @ w.float().t()).cpu(), table.cpu(), T, H + KV, hd).cuda()
    ops.check_status()
    assert _rel(out, ref) < 1e-2


# vocabularies at the edges of the three block widths, with and without a ragged tail, down to a row shorter than one vector
@pytest.mark.parametrize("V", [5, 1024, 4099, 49152, 49160, 98304, 98315, 128256])
@pytest.mark.parametrize("z_mode", [ops.Z_NONE, ops.Z_MAX, ops.Z_LSE])
def test_cross_entropy_widths(V, z_mode):
    torch.manual_seed(0)
    rows, ld = 37, (V + 7) // 8 * 8
    x = (torch.randn(rows, ld, device="cuda") * 3).bfloat16()[:, :V]
    x[3, V - 1] = x[3, 0] = 30.0                       # a tie of the maximum: the first index counts
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[::5], labels[1], labels[2] = -100, 0, V - 1
    inv = ops.count_valid(labels)
    loss, z = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    ref, rloss, rz = x.cpu().clone(), torch.empty(rows), torch.empty(rows)
    ops.cross_entropy_(x, labels, inv, loss, z, grad_scale=0.5, z_mode=z_mode, z_weight=1e-2)
    ops.cross_entropy_(ref, labels.cpu(), inv.cpu(), rloss, rz, grad_scale=0.5, z_mode=z_mode, z_weight=1e-2)
    # fp32 sums of up to 2^17 exponentials, each within a few 2^-23
    assert torch.allclose(loss.cpu(), rloss, rtol=2e-5, atol=2e-5) and torch.allclose(z.cpu(), rz, rtol=2e-5, atol=2e-5)
    assert _rel(x.cpu(), ref) < 4e-3                   # both sides round to bf16 (2^-9)


# fp32 outputs: tiles cut in both directions, a pitch wider than the row, accumulation into C, another addend (direct stores)
@pytest.mark.parametrize("M,N,K", [(512, 256, 64), (513, 260, 520), (600, 1027, 64), (777, 1028, 128), (1000, 4096 + 36, 256)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_fp32_output(M, N, K, a_mn, b_mn):
    torch.manual_seed(0)

    def operand(rows, mn):
        r8, k8 = (rows + 7) // 8 * 8, (K + 7) // 8 * 8
        return torch.randn(K, r8, device="cuda").bfloat16()[:, :rows] if mn else torch.randn(rows, k8, device="cuda").bfloat16()[:, :K]
    a, b = operand(M, a_mn), operand(N, b_mn)
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    wide = torch.full((M + 1, (N + 3) // 4 * 4 + 12), 7.0, device="cuda")
    out = wide[:M, :N]
    ops.gemm(a, b, out=out, a_mn=a_mn, b_mn=b_mn)
    tol = 2.0 ** -22 * K ** 0.5                        # fp32 accumulation of K products
    assert _rel(out.double(), ref) < tol
    assert (wide[M] == 7).all() and (wide[:, N:] == 7).all()
    ops.gemm(a, b, out=out, residual=out, a_mn=a_mn, b_mn=b_mn)
    assert _rel(out.double(), 2 * ref) < tol
    res = torch.randn(M, wide.shape[1], device="cuda")[:, :N]
    ops.gemm(a, b, out=out, residual=res, a_mn=a_mn, b_mn=b_mn)
    ops.check_status()
    assert _rel(out.double(), ref + res.double()) < tol
    assert (wide[M] == 7).all() and (wide[:, N:] == 7).all()


@pytest.mark.parametrize("M,H,KV,hd,Fd", [(96, 4, 2, 64, 512), (700, 4, 4, 32, 704), (1030, 2, 1, 128, 520)])
def test_fused_projections_match_the_separate_ops(M, H, KV, hd, Fd):
    from prime_b200.ops import functional as F_
    torch.manual_seed(0)
    D = 256
    x0 = torch.randn(M, D, device="cuda").bfloat16()
    ws = [(torch.randn(n, D, device="cuda") * D ** -0.5).requires_grad_() for n in (H * hd, KV * hd, KV * hd, Fd, Fd)]
    ws[2].requires_grad_(False)                        # a frozen weight gets no gradient
    table, ss = ops.rope_table(M, hd, 10000.0, "cuda"), A.seq_start_from_batch(1, M, "cuda")
    go, ga = torch.randn(M, H * hd, device="cuda").bfloat16(), torch.randn(M, Fd, device="cuda").bfloat16()

    def grads(attn, act, x):
        for keep in (True, False):                     # a second backward finds the saved tensors as they were
            g = torch.autograd.grad([attn, act], [x, ws[0], ws[1], ws[3], ws[4]], [go, ga], retain_graph=keep)
        return [attn.detach(), act.detach(), *g]
    x = x0.clone().requires_grad_()
    got = grads(F_.self_attention(x, *ws[:3], table, ss, M, H, KV, hd), F_.swiglu_linear(x, *ws[3:]), x)
    x = x0.clone().requires_grad_()
    qkv = F_.rope(torch.cat([F_.linear(x, w) for w in ws[:3]], -1), table, M, H + KV, hd)
    want = grads(F_.attention(qkv, ss, H, KV, hd), F_.swiglu(torch.cat([F_.linear(x, w) for w in ws[3:]], -1)), x)
    ops.check_status()
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and g.shape == w.shape and _rel(g, w) < 2e-2      # a few more bf16 roundings on the separate side


# fewer rows than one CTA iteration, one more than it, and around the number of CTAs, for one, two and four warps per row
@pytest.mark.parametrize("M", [1, 7, 9, 593, 2371])
@pytest.mark.parametrize("N", [256, 1024, 1536, 4096])
def test_rmsnorm_bwd_row_counts(M, N):
    torch.manual_seed(0)
    x, dy = (torch.randn(M, N, device="cuda").bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    _, rstd = ops.rmsnorm_fwd(x, w, 1e-5)
    dw, rdw = torch.full((N,), 3.0, device="cuda"), torch.full((N,), 3.0)
    for acc in (False, True):
        dx = ops.rmsnorm_bwd(x, w, rstd, dy, dw, accumulate_dw=acc)
        rdx = ops.rmsnorm_bwd(x.cpu(), w.cpu(), rstd.cpu(), dy.cpu(), rdw, accumulate_dw=acc)
    assert _rel(dx.cpu(), rdx) < 4e-3                  # bf16 results of the same fp32 math
    assert _rel(dw.cpu(), rdw) < 1e-5                  # fp32 sums of M terms in two orders


# a product that is split over K, into and with a matrix that starts inside a 16-byte unit: refused like by the other kernels
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_split_k_into_an_unaligned_output_is_refused(dt):
    from prime_b200.native import NativeError
    a = torch.randn(2304, 256, device="cuda").bfloat16()
    wide = torch.full((256, 1032), 7.0, device="cuda", dtype=dt)
    b = torch.randn(2304, 1024, device="cuda").bfloat16()
    assert ops._splitk_slices(256, 1024, 2304, a.device) > 1
    with pytest.raises(NativeError):
        ops.gemm(a, b, out=wide[:, 1:1025], a_mn=True, b_mn=True)
    with pytest.raises(NativeError):
        ops.gemm(a, b, out=wide[:, :1024], residual=wide[:, 1:1025], a_mn=True, b_mn=True)
    assert (wide == 7).all()


# bf16 rows that end inside a 16-byte unit, in a wider matrix: what lies behind them stays (plain, added and rotated outputs)
@pytest.mark.parametrize("M,N,K", [(512, 257, 64), (513, 263, 520), (700, 319, 64), (600, 1027, 128), (1000, 4092, 256)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_bf16_output_in_a_wider_matrix(M, N, K, a_mn, b_mn):
    torch.manual_seed(0)

    def operand(rows, mn):
        r8, k8 = (rows + 7) // 8 * 8, (K + 7) // 8 * 8
        return torch.randn(K, r8, device="cuda").bfloat16()[:, :rows] if mn else torch.randn(rows, k8, device="cuda").bfloat16()[:, :K]
    a, b = operand(M, a_mn), operand(N, b_mn)
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    wide = torch.full((M + 1, (N + 7) // 8 * 8 + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    out = wide[:M, :N]
    res = torch.randn(M, wide.shape[1], device="cuda").bfloat16()[:, :N]
    for r in (None, res):
        ops.gemm(a, b, out=out, residual=r, a_mn=a_mn, b_mn=b_mn)
        want = ref if r is None else ref + r.double()
        assert _rel(out, want) < 3e-3                  # one rounding to bf16 (2^-9)
        assert _rel(out[:, N - 8:], want[:, N - 8:]) < 4e-3
        assert (wide[M] == 7).all() and (wide[:, N:] == 7).all()
    before = out.double()
    ops.gemm(a, b, out=out, residual=out, a_mn=a_mn, b_mn=b_mn)
    ops.check_status()
    assert _rel(out, ref + before) < 3e-3
    assert (wide[M] == 7).all() and (wide[:, N:] == 7).all()
    if not a_mn and not b_mn:
        table, hd = ops.rope_table(M, 64, 10000.0, "cuda"), 64
        ops.gemm_rope(a, b, out, table, M, 4, hd)
        want = ops.rope_(ref.float().cpu(), table.cpu(), M, 4, hd).cuda()
        ops.check_status()
        assert _rel(out, want) < 4e-3
        assert (wide[M] == 7).all() and (wide[:, N:] == 7).all()


def test_narrow_heads_in_any_layout():
    """Rows of odd pitch, rows off the 16-byte boundary and fp32 results give what dense tensors give."""
    torch.manual_seed(0)
    M, H, KV, hd = 203, 4, 2, 32
    W, Wo = (H + 2 * KV) * hd, H * hd

    def odd(t, pad=1):                                 # the same values one column into a matrix of odd pitch
        wide = torch.zeros(t.shape[0], t.shape[1] + 2 * pad + 1, device="cuda", dtype=t.dtype)
        wide[:, pad: pad + t.shape[1]] = t
        return wide[:, pad: pad + t.shape[1]]
    qkv, dout = torch.randn(M, W, device="cuda").bfloat16(), torch.randn(M, Wo, device="cuda").bfloat16()
    ss, table = A.seq_start_from_batch(1, M, "cuda"), ops.rope_table(M, hd, 10000.0, "cuda")
    o, lse2 = A.attention_fwd(qkv, ss, H, KV, hd)
    g = A.attention_bwd(qkv, o, dout, lse2, ss, H, KV, hd, rope_table=table, seq_len=M)
    for dt in (torch.bfloat16, torch.float32):
        out, dqkv = odd(torch.zeros(M, Wo, device="cuda", dtype=dt)), odd(torch.zeros(M, W, device="cuda", dtype=dt))
        o2, lse2b = A.attention_fwd(odd(qkv), ss, H, KV, hd, out=out)
        assert o2 is out and torch.equal(out.float(), o.float()) and torch.equal(lse2b, lse2)
        g2 = A.attention_bwd(odd(qkv), odd(o), odd(dout), lse2, ss, H, KV, hd, dqkv=dqkv, rope_table=table, seq_len=M)
        ops.check_status()
        # dQ is summed by atomic adds: their order moves its rounding to bf16 by one unit at most
        assert g2 is dqkv and _rel(dqkv, g) < 2.0 ** -8


# K that ends inside a 16-byte unit: what lies behind an operand's last column is not read (a logits buffer's padding holds anything)
@pytest.mark.parametrize("M,N", [(600, 512), (100, 128)])
@pytest.mark.parametrize("K", [1025, 1031])
@pytest.mark.parametrize("b_mn", [False, True])
def test_operand_padding_is_not_read(M, N, K, b_mn):
    torch.manual_seed(0)

    def padded(rows):
        wide = torch.full((rows, (K + 7) // 8 * 8), float("nan"), device="cuda", dtype=torch.bfloat16)
        wide[:, :K] = torch.randn(rows, K, device="cuda")
        return wide[:, :K]
    a, b = padded(M), torch.randn(K, N, device="cuda").bfloat16() if b_mn else padded(N)
    out = ops.gemm(a, b, b_mn=b_mn, out_dtype=torch.float32)
    ops.check_status()
    ref = a.double() @ (b.double() if b_mn else b.double().t())
    assert _rel(out.double(), ref) < 2.0 ** -22 * K ** 0.5      # fp32 accumulation of K products
