"""Gradient reduction, global norm and AdamW kernels of the sharded update against fp32 torch."""
import ctypes as C

import pytest
import torch

from prime_b200 import native
from prime_b200.engine import fused_llama  # noqa: F401  (declares the C signatures)
from prime_b200.native import check, ptr, stream_ptr
from prime_b200.ops import kernels as K

pytestmark = pytest.mark.gpu

# segment tables: one vector-aligned run, a run with a ragged tail, an unaligned start (scalar path), a run smaller than a vector
SEGS = [[(0, 0, 4096)], [(0, 0, 70001)], [(1, 1, 5000), (6008, 5008, 3)], [(64, 0, 1 << 20), ((1 << 20) + 128, 1 << 20, 999)]]


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def _arrays(segs):
    arr = C.c_longlong * len(segs)
    return arr(*[s[0] for s in segs]), arr(*[s[1] for s in segs]), arr(*[s[2] for s in segs])


@pytest.mark.parametrize("segs", SEGS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_reduce_and_norm(segs, dtype):
    torch.manual_seed(0)
    n_full, n_shard = max(s[0] + s[2] for s in segs) + 8, max(s[1] + s[2] for s in segs) + 8
    g = torch.randn(n_full, device="cuda").to(dtype)
    full, shard, numel = _arrays(segs)
    lib = native.cuda()
    fp32 = int(dtype == torch.float32)
    partial = torch.zeros(4096, device="cuda")
    want = torch.cat([g[a: a + n].float() for a, _, n in segs])
    for ctas in (len(segs), 37, 148):
        out, sq = torch.full((n_shard,), 7.0, device="cuda"), torch.zeros(1, device="cuda")
        check(lib.pb_zero_reduce_grads((C.c_void_p * 1)(g.data_ptr()), 1, 0, fp32, len(segs), full, shard, numel, ptr(out), 0.5,
                                       ptr(partial), ptr(sq), 0, ctas, stream_ptr()), "pb_zero_reduce_grads")
        got = torch.cat([out[b: b + n] for _, b, n in segs])
        assert torch.equal(got, want * 0.5)
        # fp32 sums of n squares in a tree: relative error below sqrt(n) * 2^-24, far under 1e-5 here
        ref = (want * 0.5).double().square().sum().item()
        assert abs(sq.item() - ref) < 1e-5 * ref
        cnt, sq2 = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, device="cuda")
        for _ in range(2):         # twice: the counter has to be back at zero
            check(lib.pb_grad_sumsq(ptr(g), fp32, len(segs), full, numel, ptr(partial), ptr(cnt), ptr(sq2), ctas, stream_ptr()), "pb_grad_sumsq")
            assert abs(sq2.item() - 4 * ref) < 1e-5 * 4 * ref


@pytest.mark.parametrize("segs", SEGS)
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_adamw_reads_shard_or_own_gradients(segs, kind):
    torch.manual_seed(1)
    n_full, n_shard = max(s[0] + s[2] for s in segs) + 8, max(s[1] + s[2] for s in segs) + 8
    full, shard, numel = _arrays(segs)
    gsrc = torch.randn(n_shard if kind == 0 else n_full, device="cuda").to(torch.bfloat16 if kind == 1 else torch.float32)
    p, m, v = (torch.randn(n_shard, device="cuda") for _ in range(3))
    v.abs_()
    ref = [t.clone() for t in (p, m, v)]
    params = torch.zeros(n_full, dtype=torch.bfloat16, device="cuda")
    sq = torch.tensor([16.0], device="cuda")
    check(native.cuda().pb_zero_adamw_gather((C.c_void_p * 1)(params.data_ptr()), 1, 0, len(segs), full, shard, numel, ptr(p), ptr(gsrc), kind,
                                             ptr(m), ptr(v), 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, ptr(sq), 1.0, None, 148, stream_ptr()),
          "pb_zero_adamw_gather")
    for a, b, n in segs:
        g = (gsrc[b: b + n] if kind == 0 else gsrc[a: a + n]).float().cpu()
        rp, rm, rv = (t[b: b + n].cpu() for t in ref)
        K.adamw_(rp, g, rm, rv, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, gnorm=torch.tensor(4.0), max_norm=1.0)
        for got, want in ((p, rp), (m, rm), (v, rv)):
            assert torch.allclose(got[b: b + n].cpu(), want, rtol=2e-5, atol=2e-6)
        assert torch.equal(params[a: a + n], p[b: b + n].bfloat16())


@pytest.mark.parametrize("n", [1, 1000, 65536 + 3])
def test_label_count_and_loss_sums(n):
    torch.manual_seed(2)
    labels = torch.randint(0, 50, (n,), device="cuda")
    labels[::7] = -100
    cnt = torch.zeros(4, dtype=torch.int32, device="cuda")
    rows, z = torch.rand(n, device="cuda"), torch.rand(n, device="cuda")
    partial, acc = torch.zeros(512, device="cuda"), torch.tensor([1.0, 2.0], device="cuda")
    k = int((labels != -100).sum())
    for _ in range(2):             # the counters are zero again after a launch
        inv = K.count_valid(labels, counter=cnt[1:3])
        assert inv.tolist() == pytest.approx([1.0 / max(k, 1), k], rel=1e-6)
        out = torch.zeros(2, device="cuda")
        K.loss_sums(rows, z, inv, 0.5, out, partial, cnt[3:], acc=acc, acc_scale=0.25, acc_first=False)
    want = [rows.double().sum().item() / max(k, 1), 0.5 * z.double().sum().item() / max(k, 1)]
    assert out.tolist() == pytest.approx(want, rel=1e-5)
    assert acc.tolist() == pytest.approx([1.0 + 0.5 * want[0], 2.0 + 0.5 * want[1]], rel=1e-5)
    K.loss_sums(rows, None, inv, 0.5, out, partial, cnt[3:])
    assert out.tolist() == pytest.approx([want[0], 0.0], rel=1e-5)
    assert not cnt.any()


@pytest.mark.parametrize("hd,micro,packed,fp32", [(64, 4, False, True), (64, 2, True, True), (32, 2, True, False)])
def test_graphed_steps_match_steps_launched_one_by_one(monkeypatch, hd, micro, packed, fp32):
    """Same inputs, new ones each step, one shape in between that makes the workspaces grow and drops the recorded graphs."""
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    args = ModelArgs(dim=256, n_layers=2, n_heads=256 // hd, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal")
    dt = torch.float32 if fp32 else torch.bfloat16
    a, b = (FusedLlama(args, device="cuda", ce_chunk_tokens=512, grad_dtype=dt) for _ in range(2))
    for e in (a, b):
        e.init_weights(seed=3)
    monkeypatch.setattr(b, "_graphable", lambda *x: False)
    g = torch.Generator(device="cuda").manual_seed(1)
    replayed = 0
    for i, (B, T) in enumerate([(4, 200)] * 4 + [(8, 256)] + [(4, 200)] * 3):
        ids = torch.randint(0, 1024, (B, T + 1), device="cuda", generator=g)
        ss = None
        if packed:
            cut = 37 + 20 * i
            ss = (torch.arange(B * T, device="cuda", dtype=torch.int32) // T) * T
            ss += torch.where(torch.arange(B * T, device="cuda") % T >= cut, cut, 0).int()
        res = [e.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3 * (i + 1), micro_bs=micro, seq_start=ss) for e in (a, b)]
        replayed += bool(a._graphs)
        # the kernels are the same; the atomic adds of dQ and of the embedding gradient may come in another order (bf16: 2^-8 each).
        # Adam turns such a difference of a tiny gradient into one of the update's full size, so every step starts from one state
        assert res[0] == pytest.approx(res[1], rel=2e-3)
        assert ((a.master - b.master).norm() / b.master.norm()).item() < (1e-4 if fp32 else 5e-3)
        assert ((a.exp_avg - b.exp_avg).norm() / b.exp_avg.norm()).item() < (1e-3 if fp32 else 3e-2)
        for name in ("master", "exp_avg", "exp_avg_sq", "params"):
            getattr(b, name).copy_(getattr(a, name))
    assert replayed >= 5 and not b._graphs
    assert a.opt_step == b.opt_step == 8
    loss, norm = a.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3, micro_bs=micro, seq_start=ss, sync_loss=False)
    keep = loss.item()
    a.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3, micro_bs=micro, seq_start=ss, sync_loss=False)
    assert loss.item() == keep and norm.item() > 0
    K.check_status()


def test_grad_shard_holds_the_gradients_of_a_step_without_peers():
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    eng = FusedLlama(ModelArgs(dim=256, n_layers=2, n_heads=4, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal"),
                     device="cuda", ce_chunk_tokens=512)
    eng.init_weights(seed=3)
    ids = torch.randint(0, 1024, (2, 129), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    for _ in range(3):
        loss, norm = eng.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3)
        # the norm is the root of the shard's sum of squares: fp32 sums, far below 1e-4
        assert eng.grad_shard.double().norm().item() == pytest.approx(norm, rel=1e-4)
    for name, g in eng.g.items():
        assert torch.equal(eng.shard_view(eng.grad_shard, name), g.float())


def test_scratch_is_one_per_stream():
    a = torch.randn(4096, 256, device="cuda").bfloat16()
    K.gemm(a, a, a_mn=True, b_mn=True)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        K.gemm(a, a, a_mn=True, b_mn=True)
    torch.cuda.synchronize()
    ws = [t.data_ptr() for k, t in K._scratch.items() if k[2] == "splitk"]
    assert len(ws) >= 2 and len(set(ws)) == len(ws)
    assert K.take_scratch(side) and not any(k[1] == side.cuda_stream for k in K._scratch)


@pytest.mark.parametrize("overlap", [True, False])
def test_first_reduced_step_keeps_every_gradient(overlap):
    """The reduce path with one rank: the shard holds the gradient buffer after the first step, whichever stream reduced it."""
    from prime_b200.engine.fused_llama import FusedLlama, LocalComm
    from prime_b200.models.llama import ModelArgs

    class OneRank(LocalComm):       # not the plain LocalComm, whose runs update from their own gradients
        pass
    eng = FusedLlama(ModelArgs(dim=256, n_layers=2, n_heads=4, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal"),
                     device="cuda", comm=OneRank(), ce_chunk_tokens=512)
    eng.overlap_reduce = overlap
    eng.init_weights(seed=3)
    ids = torch.randint(0, 1024, (2, 129), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    _, norm = eng.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3)
    for name, g in eng.g.items():
        assert torch.equal(eng.shard_view(eng.grad_shard, name), g.float()), name
    # the norm is the root of the shard's sum of squares: fp32 sums, far below 1e-4
    assert eng.grad_shard.double().norm().item() == pytest.approx(norm, rel=1e-4)


def test_update_sees_the_gradients_of_the_weight_gradient_stream(monkeypatch):
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    args = ModelArgs(dim=1024, n_layers=2, n_heads=16, ffn_hidden=4096, vocab_size=1024, max_seq_len=512, init_mode="normal")
    runs = []
    for on in ("0", "1"):
        monkeypatch.setenv("PRIME_B200_WGRAD_STREAM", on)
        eng = FusedLlama(args, device="cuda", grad_dtype=torch.float32)
        assert (eng.wgrad_stream is not None) == (on == "1")
        eng.init_weights(seed=3)
        ids = torch.randint(0, 1024, (16, 513), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
        loss, norm = eng.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3)
        # first moment of the first step: 0.1 * clipped gradient, in fp32 products
        want = 0.1 * min(1.0, 1.0 / (norm + 1e-6)) * eng.grads
        for p in eng.layout.params:
            s = slice(p.offset, p.offset + p.numel)
            assert _rel(eng.shard_view(eng.exp_avg, p.name).flatten(), want[s]) < 1e-5, p.name
        assert eng.grad_shard.double().norm().item() == pytest.approx(norm, rel=1e-4)
        runs.append((loss, norm, eng))
    (l0, n0, a), (l1, n1, b) = runs
    # The kernels are the same. dQ is summed by atomic adds, whose order moves its rounding to bf16 by one unit (2^-8) at most: that
    # reaches every gradient below the upper block's attention, once per block
    assert l0 == pytest.approx(l1, rel=1e-6) and n0 == pytest.approx(n1, rel=2 * 2.0 ** -8)
    for name, g in a.g.items():
        assert _rel(b.g[name], g) < 2 * 2.0 ** -8, name
    K.check_status()


def test_threads_on_one_stream_do_not_share_partials():
    """Products whose partials one launch writes and the next one sums, from two threads on the default stream."""
    import threading
    torch.manual_seed(4)
    ops_ = [torch.randn(8192, n, device="cuda").bfloat16() for n in (256, 512)]
    want = [x.float().t() @ x.float() for x in ops_]
    torch.cuda.synchronize()
    start, good = threading.Barrier(2), []

    def work(i):
        torch.cuda.set_device(0)
        start.wait()
        outs = [K.gemm(ops_[i], ops_[i], a_mn=True, b_mn=True, out_dtype=torch.float32) for _ in range(200)]
        torch.cuda.synchronize()
        good.extend(1 for o in outs if _rel(o, want[i]) < 1e-3)       # fp32 sums of the same products in another order
    assert all(K._splitk_slices(x.shape[1], x.shape[1], 8192, x.device) > 1 for x in ops_)
    ts = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(good) == 400
    K.check_status()


def test_steps_whose_graphs_give_way_to_each_other(monkeypatch):
    """Three shapes and room for two graphs: recorded, replayed, evicted and recorded again, every step against one launched directly."""
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    monkeypatch.setattr(FusedLlama, "_MAX_GRAPHS", 2)
    monkeypatch.setattr(FusedLlama, "_RUNS_TO_EVICT", 2)
    args = ModelArgs(dim=256, n_layers=2, n_heads=4, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal")
    a, b = (FusedLlama(args, device="cuda", ce_chunk_tokens=512, grad_dtype=torch.float32) for _ in range(2))
    for e in (a, b):
        e.init_weights(seed=3)
    monkeypatch.setattr(b, "_graphable", lambda *x: False)
    g, held = torch.Generator(device="cuda").manual_seed(1), set()
    for i, (B, T) in enumerate([(4, 256), (4, 200), (2, 64)] * 9):
        ids = torch.randint(0, 1024, (B, T + 1), device="cuda", generator=g)
        res = [e.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3) for e in (a, b)]
        held |= {k[:2] for k in a._graphs}
        assert len(a._graphs) <= 2
        # the kernels are the same, atomic adds (dQ, embedding) may come in another order: one unit of bf16 at most
        assert res[0] == pytest.approx(res[1], rel=2e-3)
        assert _rel(a.exp_avg, b.exp_avg) < 2 * 2.0 ** -8
        for name in ("master", "exp_avg", "exp_avg_sq", "params"):
            getattr(b, name).copy_(getattr(a, name))
    assert held == {(4, 256), (4, 200), (2, 64)}      # every shape had a graph at some time
    K.check_status()


def test_a_gradient_shard_in_hand_follows_recorded_steps():
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    eng = FusedLlama(ModelArgs(dim=256, n_layers=2, n_heads=4, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal"),
                     device="cuda", ce_chunk_tokens=512)
    eng.init_weights(seed=3)
    held, g = eng.grad_shard, torch.Generator(device="cuda").manual_seed(1)
    for _ in range(4):             # launched one by one, recorded, replayed
        ids = torch.randint(0, 1024, (2, 129), device="cuda", generator=g)
        eng.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3)
        assert all(torch.equal(eng.shard_view(held, name), v.float()) for name, v in eng.g.items()) and held.any()
    assert eng._graphs


@pytest.mark.parametrize("segs", SEGS)
@pytest.mark.parametrize("world", [2, 5, 9])      # the three widths of the kernel's rank loop
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_reduce_over_several_buffers(segs, world, dtype):
    """One rank's part of the reduce, with every rank's buffer on this GPU: the kernel reads them all and waits for nobody."""
    torch.manual_seed(0)
    n_full, n_shard = max(s[0] + s[2] for s in segs) + 8, max(s[1] + s[2] for s in segs) + 8
    gs = [torch.randn(n_full, device="cuda").to(dtype) for _ in range(world)]
    full, shard, numel = _arrays(segs)
    total = torch.zeros(n_full, device="cuda")
    for g in gs:                                   # in rank order, like the kernel
        total += g.float()
    want = torch.cat([total[a: a + n] for a, _, n in segs]) * 0.25
    out, sq, partial = torch.full((n_shard,), 7.0, device="cuda"), torch.zeros(1, device="cuda"), torch.zeros(4096, device="cuda")
    check(native.cuda().pb_zero_reduce_grads((C.c_void_p * world)(*[g.data_ptr() for g in gs]), world, 1, int(dtype == torch.float32),
                                             len(segs), full, shard, numel, ptr(out), 0.25, ptr(partial), ptr(sq), 0, 148, stream_ptr()),
          "pb_zero_reduce_grads")
    assert torch.equal(torch.cat([out[b: b + n] for _, b, n in segs]), want)
    ref = want.double().square().sum().item()
    assert abs(sq.item() - ref) < 1e-5 * ref       # fp32 sums of n squares in a tree, as above
    keep = torch.ones(n_shard, dtype=torch.bool, device="cuda")
    for _, b, n in segs:
        keep[b: b + n] = False
    assert (out[keep] == 7).all()


def test_norm_weight_gradients_on_another_stream():
    """Call after call into one weight gradient, on a stream that has yet to read the first call's partial sums."""
    M, N, calls = 600, 512, 4
    g = torch.Generator(device="cuda").manual_seed(0)
    w = torch.rand(N, device="cuda", generator=g).bfloat16()
    data = [[torch.randn(M, N, device="cuda", generator=g).bfloat16() for _ in range(2)] for _ in range(calls)]
    rstd = [K.rmsnorm_fwd(x, w, 1e-5)[1] for x, _ in data]
    before = {k[2] for k in K._scratch}
    side = torch.cuda.Stream()
    got, want = torch.zeros(N, device="cuda"), torch.zeros(N, device="cuda")
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                       # some 10 ms
    dxs = [K.rmsnorm_bwd(x, w, r, dy, got, dw_stream=side) for (x, dy), r in zip(data, rstd)]
    torch.empty(4 << 20, device="cuda").fill_(float("nan"))  # what the caller allocates next must not be the partial sums
    assert {k[2] for k in K._scratch} == before              # nothing that a later user of the scratch table could take away
    torch.cuda.current_stream().wait_stream(side)
    for (x, dy), r, dx in zip(data, rstd, dxs):
        assert torch.equal(K.rmsnorm_bwd(x, w, r, dy, want), dx)
    assert torch.equal(got, want)


@pytest.mark.parametrize("layers,ac,micro", [(2, True, 2), (3, 2, 2), (17, False, 4), (17, True, 2)])
def test_recorded_steps_of_checkpointed_and_deep_models(monkeypatch, layers, ac, micro):
    """The branch of the weight gradients reads the workspace that a recomputed block overwrites, and has the norms' gradients of any
    number of blocks on it. Rows of 200 tokens have two kv tiles: dQ is the sum of two numbers, the same in either order."""
    from prime_b200.engine.fused_llama import FusedLlama
    from prime_b200.models.llama import ModelArgs
    args = ModelArgs(dim=256, n_layers=layers, n_heads=4, ffn_hidden=512, vocab_size=1024, max_seq_len=256, init_mode="normal")
    a, b = (FusedLlama(args, device="cuda", ce_chunk_tokens=512, grad_dtype=torch.float32, ac_ckpt=ac) for _ in range(2))
    for e in (a, b):
        e.init_weights(seed=3)
    monkeypatch.setattr(b, "_graphable", lambda *x: False)
    g = torch.Generator(device="cuda").manual_seed(1)
    for _ in range(4):
        ids = torch.randint(0, 1024, (4, 201), device="cuda", generator=g)
        res = [e.train_step(ids[:, :-1], ids[:, 1:], lr=1e-3, micro_bs=micro) for e in (a, b)]
        # only the atomic adds of the embedding's gradient may come in another order
        assert res[0] == pytest.approx(res[1], rel=1e-5)
        for name, grad in b.g.items():
            assert _rel(a.g[name], grad) < 1e-5, name
        for name in ("master", "exp_avg", "exp_avg_sq", "params"):
            getattr(b, name).copy_(getattr(a, name))
    assert len(a._graphs) == 1 and not b._graphs
    K.check_status()
