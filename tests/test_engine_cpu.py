"""The fused engine's hand-written backward and update against autograd on the eager model (CPU, fp32)."""
import copy

import pytest
import torch

from prime_b200.engine.fused_llama import FusedLlama
from prime_b200.models.llama import ModelArgs, Transformer


def _tiny(**kw):
    base = dict(dim=64, n_layers=2, n_heads=4, n_kv_heads=2, ffn_hidden=128, vocab_size=96, max_seq_len=16, init_mode="normal",
                init_std=0.2)
    base.update(kw)
    return ModelArgs(**base)


class _F32Engine(FusedLlama):
    """fp32 replicas / activations so the CPU comparison is tight."""

    def _buf(self, name, shape, dtype=torch.bfloat16):
        return super()._buf(name, shape, torch.float32 if dtype == torch.bfloat16 else dtype)


def _mk(args, ac=False, z=(0, 0.0)):
    torch.manual_seed(0)
    model = Transformer(args)
    eng = _F32Engine(args, device="cpu", grad_dtype=torch.float32, ac_ckpt=ac, ce_chunk_tokens=24, z_mode=z[0], z_weight=z[1])
    eng.params = eng.params.float()
    for p in eng.layout.params:
        eng.w[p.name] = eng.params[p.offset: p.offset + p.numel].view(p.shape)
    H, KV, hd, D, F = args.n_heads, args.kv_heads, args.head_dim, args.dim, args.hidden_dim
    for i in range(args.n_layers):
        q = eng.layout.params[eng.layout.by_name[f"layers.{i}.attention.wq.weight"]]
        eng.wqkv[i] = eng.params[q.offset: q.offset + (H + 2 * KV) * hd * D].view(-1, D)
        w1 = eng.layout.params[eng.layout.by_name[f"layers.{i}.feed_forward.w1.weight"]]
        eng.w13[i] = eng.params[w1.offset: w1.offset + 2 * F * D].view(2 * F, D)
    eng._rope = model.rope_table()
    eng.load_from_module(model)
    for name, v in eng.named_master_shards():   # fp32 publish
        s = eng.layout.segments[0][eng.layout.by_name[name]]
        eng.params[s.full_offset: s.full_offset + s.numel].copy_(v.reshape(-1))
    return model, eng


@pytest.mark.parametrize("ac", [False, True, 2])
@pytest.mark.parametrize("packed", [False, True])
def test_engine_grads_match_autograd(ac, packed):
    args = _tiny()
    model, eng = _mk(args, ac=ac)
    B, T = 3, 16
    tokens = torch.randint(0, args.vocab_size, (B, T))
    labels = torch.randint(0, args.vocab_size, (B, T))
    labels[0, :3] = -100
    seqlens = [[5, 11], [16], [1, 7, 8]] if packed else None
    from prime_b200.ops.attention import seq_start_from_seqlens
    ss = seq_start_from_seqlens(seqlens, T, "cpu") if packed else None
    out = eng.forward_backward(tokens, labels, seq_start=ss)
    logits = model(tokens, seqlens=seqlens)
    ref = torch.nn.functional.cross_entropy(logits.reshape(-1, args.vocab_size), labels.reshape(-1), ignore_index=-100)
    ref.backward()
    assert abs(out["loss"].item() - ref.item()) < 1e-4
    for name, p in model.named_parameters():
        g = eng.g[name]
        err = (g - p.grad).norm() / (p.grad.norm() + 1e-12)
        assert err < 1e-4, (name, err.item())
    assert torch.allclose(eng.forward_logits(tokens, seq_start=ss), logits, atol=1e-4)


def test_engine_grad_accumulation_and_adamw_step():
    args = _tiny()
    model, eng = _mk(args)
    opt = torch.optim.AdamW(model.parameters(), lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1)
    B, T = 2, 16
    for step in range(2):
        for mb in range(2):
            tokens = torch.randint(0, args.vocab_size, (B, T))
            labels = torch.randint(0, args.vocab_size, (B, T))
            eng.forward_backward(tokens, labels, loss_scale=0.5)
            loss = torch.nn.functional.cross_entropy(model(tokens).reshape(-1, args.vocab_size), labels.reshape(-1)) * 0.5
            loss.backward()
        ref_norm = torch.nn.utils.clip_grad_norm_(model.parameters(), 1.0)
        opt.step()
        opt.zero_grad()
        norm = eng.optimizer_step(1e-2, (0.9, 0.95), 1e-8, 0.1, 1.0)
        assert abs(norm.item() - ref_norm.item()) / ref_norm.item() < 1e-4
        for name, v in eng.named_master_shards():   # republish in fp32 for the next comparison
            s = eng.layout.segments[0][eng.layout.by_name[name]]
            eng.params[s.full_offset: s.full_offset + s.numel].copy_(v.reshape(-1))
    sd = dict(model.named_parameters())
    for name, v in eng.named_master_shards():
        # Adam normalises the update, so elements whose gradient is ~0 amplify round-off: compare in norm
        assert (v - sd[name]).norm() / sd[name].norm() < 1e-3, name


def test_z_loss_modes_match_autograd():
    from prime_b200.ops import kernels as K
    args = _tiny()
    for mode in (K.Z_MAX, K.Z_LSE):
        model, eng = _mk(args, z=(mode, 1e-2))
        tokens = torch.randint(0, args.vocab_size, (2, 16))
        labels = torch.randint(0, args.vocab_size, (2, 16))
        out = eng.forward_backward(tokens, labels)
        lg = model(tokens).reshape(-1, args.vocab_size)
        z = (lg.max(-1).values ** 2).mean() if mode == K.Z_MAX else (torch.logsumexp(lg, -1) ** 2).mean()
        ref = torch.nn.functional.cross_entropy(lg, labels.reshape(-1)) + 1e-2 * z
        ref.backward()
        assert abs((out["loss"] + out["z_loss"]).item() - ref.item()) < 1e-4
        for name, p in model.named_parameters():
            assert (eng.g[name] - p.grad).norm() / (p.grad.norm() + 1e-12) < 1e-4, name


def test_segment_tables_merge_contiguous_runs():
    """With one rank neighbouring parameters are contiguous in both the full and the shard buffer and collapse
    into few runs; with two ranks every parameter keeps its own row-shard segment."""
    from prime_b200.engine.fused_llama import _SegArrays
    from prime_b200.engine.layout import llama_layout
    args = ModelArgs(dim=64, n_layers=2, n_heads=4, ffn_hidden=128, vocab_size=96, max_seq_len=32)
    for world in (1, 2):
        lay = llama_layout(args, world)
        segs = [s for g in range(len(lay.groups)) for s in lay.group_segments(0, g)]
        sa = _SegArrays(segs)
        assert sa.total == sum(s.numel for s in segs)
        covered = sorted((sa.full[i], sa.numel[i]) for i in range(sa.n))
        for (o0, n0), (o1, _) in zip(covered, covered[1:]):
            assert o0 + n0 <= o1
        if world == 1:
            assert sa.n < len([s for s in segs if s.numel > 0])
        else:
            assert sa.n <= len(segs)


def test_optimizer_cta_ranges_cover_every_segment():
    """The reduce / AdamW launches give each non-empty segment its own CTA range: a segment without one would
    silently keep stale gradients. Ranges are monotone, end at the grid size and follow the segment sizes."""
    import ctypes as C

    from prime_b200 import native
    try:
        lib = native.cuda()
    except native.NativeError:
        pytest.skip("CUDA library not built")
    gen = torch.Generator().manual_seed(0)
    cases = [[5], [1, 1, 1], [0, 7, 0, 9, 0], [1 << 24, 512, 1 << 21, 0, 3, 1 << 24],
             torch.randint(1, 1 << 22, (111,), generator=gen).tolist(), [1] * 128]
    for numel in cases:
        n = len(numel)
        arr = (C.c_longlong * n)(*numel)
        for ctas in (1, n, 148, 640, 4096):
            out = (C.c_int * (n + 1))()
            grid = lib.pb_zero_cta_ranges(n, arr, ctas, out)
            begins = list(out)
            nonempty = sum(1 for x in numel if x > 0)
            assert grid == begins[-1] and grid >= nonempty
            if nonempty:
                assert grid == max(ctas, n)
            total = sum(numel)
            for i, x in enumerate(numel):
                width = begins[i + 1] - begins[i]
                assert width >= (1 if x > 0 else 0) and (x > 0 or width == 0)
                share = x / total * grid if total else 0.0
                if share >= 4.0:                # large segments get about their share of the grid
                    assert 0.5 * share <= width <= 1.5 * share + 1


def test_soap_runs_as_a_shard_optimizer_of_the_fused_engine(tmp_path):
    """``optim.type = "soap"`` with the fused engine: the engine produces the reduced fp32 gradient shard and the global
    norm, SOAP steps the fp32 master shards in place, the bf16 replica is refreshed. Checked against SOAP applied by hand
    to copies of the same shards with the same clipped gradients, over enough steps to cross a basis refresh; then the
    optimizer state round-trips through the flat state dict a checkpoint uses."""
    from prime_b200.backend import FusedBackend
    from prime_b200.config import SoapConfig
    from prime_b200.lr_scheduler import get_scheduler
    from prime_b200.optimizers import SOAP
    args = ModelArgs(dim=64, n_layers=2, n_heads=4, n_kv_heads=2, ffn_hidden=128, vocab_size=200, max_seq_len=32,
                     init_mode="normal", init_std=0.05)
    cfg = SoapConfig(lr=3e-3, weight_decay=0.01, precondition_frequency=3, max_preconditioner_dim=256)
    eng = FusedLlama(args, device="cpu", grad_dtype=torch.float32, ce_chunk_tokens=64)
    eng.init_weights(seed=2)
    backend = FusedBackend(eng, cfg, lambda o: get_scheduler("cosine", o, 1, 0, 100), max_norm=0.5)
    assert backend.shard_optimizer is not None and eng._shard_opt is backend.shard_optimizer
    # the hand-run twin: copies of the shards, their own SOAP
    twin = [torch.nn.Parameter(t.clone()) for _, t in eng.named_master_shards()]
    opt = SOAP(twin, lr=cfg.lr, betas=(cfg.betas1, cfg.betas2), eps=1e-12, weight_decay=cfg.weight_decay,
               max_preconditioner_dim=cfg.max_preconditioner_dim, precondition_frequency=cfg.precondition_frequency)
    g = torch.Generator().manual_seed(0)
    losses = []
    for step in range(5):
        tok = torch.randint(0, args.vocab_size, (2, 33), generator=g)
        batch = {"input_ids": tok[:, :-1].contiguous(), "labels": tok[:, 1:].contiguous()}
        lr = backend.current_lr()
        out = backend.train_step(batch, micro_bs=2)
        losses.append(out["loss"])
        # grad_shard still holds the clipped gradients the shard optimizer consumed
        for q, (name, _) in zip(twin, eng.named_master_shards()):
            q.grad = eng.shard_view(eng.grad_shard, name).clone()
        for group in opt.param_groups:
            group["lr"] = lr
        opt.step()
        for q, (name, t) in zip(twin, eng.named_master_shards()):
            assert torch.allclose(q.data, t, rtol=1e-5, atol=1e-6), (step, name)
        # the bf16 replica follows the master shard
        name0, t0 = next(iter(eng.named_master_shards()))
        assert torch.allclose(eng.w[name0].float(), t0, atol=2e-2)
    assert out["grad_norm"] > 0 and all(torch.isfinite(torch.tensor(losses)))
    # state dict: every tensor of the shard optimizer's state, keyed by rank and parameter; loading fills them in place
    sd = backend.optimizer_state_dict()
    assert any(k.endswith(".Q_L") for k in sd) and any(k.endswith(".GG_R") for k in sd) and "state.step" in sd
    saved = {k: v.clone() for k, v in sd.items()}
    eng2 = FusedLlama(args, device="cpu", grad_dtype=torch.float32, ce_chunk_tokens=64)
    eng2.init_weights(seed=2)
    backend2 = FusedBackend(eng2, cfg, lambda o: get_scheduler("cosine", o, 1, 0, 100), max_norm=0.5)
    sd2 = backend2.optimizer_state_dict()
    assert set(sd2) == set(sd)
    for k, v in sd2.items():
        v.copy_(saved[k])                     # what the checkpoint loader does
    backend2.load_optimizer_state_dict(sd2)
    assert eng2.opt_step == eng.opt_step
    q0 = eng2._shard_params[0]
    assert backend2.shard_optimizer.state[q0]["step"] == 5


def test_a_run_that_reduces_has_its_gradient_shard_from_the_start():
    """Allocated later, its zero fill would be queued behind the event that lets the communication stream start the reduce."""
    _, eng = _mk(_tiny())
    assert not eng._solo and eng._grad_shard is not None
    assert eng._grad_shard.numel() == eng.layout.shard_numel[0] and not eng._grad_shard.any()


def test_update_without_peers_waits_for_the_weight_gradient_stream(monkeypatch):
    """The host's order of calls, on stand-ins for the streams and the kernel library: the update and a reader of the gradient shard
    join the stream of the weight gradients before they touch a gradient."""
    from prime_b200 import native
    from prime_b200.engine import fused_llama
    _, eng = _mk(_tiny())
    order = []

    class Stream:
        def wait_stream(self, s):
            order.append("join" if s is eng.wgrad_stream else "other")

    class Lib:
        def __getattr__(self, name):
            return lambda *a: order.append(name) or 0
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(native, "cuda", Lib)
    monkeypatch.setattr(fused_llama, "stream_ptr", lambda *a: None)
    eng._solo, eng.wgrad_stream = True, object()
    eng._readers = {1: "event"}
    eng._update_from_own_grads(1e-3, (0.9, 0.95), 1e-8, 0.1, 1.0)
    assert order == ["join", "pb_grad_sumsq", "pb_zero_adamw_gather"]
    order.clear()
    eng._grad_shard, eng._readers = None, {1: "event"}
    assert eng.grad_shard is not None and order == ["join"]


def test_norm_gradients_beside_the_chain_are_waited_for_by_themselves(monkeypatch):
    """No weight-gradient GEMM that could stand for them has left an entry."""
    from prime_b200.engine import fused_llama
    _, eng = _mk(_tiny())
    joined = []

    class Stream:
        def wait_stream(self, s):
            joined.append(s)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(fused_llama.K, "rmsnorm_bwd", lambda *a, dw_stream, **k: None)
    side = object()
    for stream, want in ((side, [side]), (None, [])):
        joined.clear()
        eng.wgrad_stream, eng._norm_dw_stream = side, stream
        eng._norm_bwd(None, "norm.weight", None, None, None)
        for _ in range(2):                     # the second time there is nothing left to wait for
            eng._wait_all_wgrads()
            assert joined == want


@pytest.mark.parametrize("micro", [1, 2, 4])
def test_row_maps_reach_the_kernels_dense(monkeypatch, micro):
    """Every second element of a longer tensor, or one value for all rows: a micro-batch gets its own dense part, the first one too."""
    _, eng = _mk(_tiny())
    B, T = 4, 16
    starts = torch.arange(B).repeat_interleave(T).int() * T
    tokens = torch.zeros(B, T, dtype=torch.int64)
    for given in (torch.stack([starts, starts + 1], 1)[:, 0], torch.zeros(1, dtype=torch.int32).expand(B * T), starts):
        seen = []
        monkeypatch.setattr(eng, "forward_backward", lambda *a, seq_start, **k: seen.append(seq_start))
        eng._accumulate_micro_batches(tokens, tokens, given, micro)
        assert len(seen) == B // micro and all(s.is_contiguous() and s.dtype == torch.int32 for s in seen)
        for mb, s in enumerate(seen):
            assert torch.equal(s, given[mb * micro * T: (mb + 1) * micro * T] - mb * micro * T)


@pytest.fixture()
def graph_engine(monkeypatch):
    """An engine whose steps and graphs are stand-ins that write down what is recorded, replayed and launched."""
    from prime_b200 import native
    from prime_b200.engine import fused_llama
    _, eng = _mk(_tiny())
    log = []

    class Graph:
        launches = 0

        def __init__(self, eng, B, T, *a):
            self.tokens = self.labels = self.hyper = torch.zeros(1)
            self.seq_start, self.graph, self.shape = None, self, (B, T)
            log.append(("record", B, T))

        def replay(self):
            log.append(("replay", *self.shape))
            getattr(eng, "on_replay", lambda: None)()

    def run(tokens, *a):
        log.append(("run", *tokens.shape))
        eng._buf("work", tokens.shape)
    monkeypatch.setattr(fused_llama, "_StepGraph", Graph)
    monkeypatch.setattr(fused_llama, "stream_ptr", lambda *a: None)
    monkeypatch.setattr(native, "cuda", lambda: type("Lib", (), {"pb_stage_step": staticmethod(lambda *a: 0)}))
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(eng, "_accumulate_micro_batches", run)
    monkeypatch.setattr(eng, "_update_from_own_grads", lambda *a, **k: None)
    monkeypatch.setattr(eng, "_report", lambda *a: None)

    def step(B, T):
        n = len(log)
        x = torch.zeros(B, T, dtype=torch.int64)
        eng._graphed_step(x, x, None, B, 1e-3, (0.9, 0.95), 1e-8, 0.1, 1.0)
        return [e[0] for e in log[n:]]
    return eng, step, log


def test_more_shapes_than_graphs_are_not_recorded_over_and_over(graph_engine):
    eng, step, log = graph_engine
    eng._buf("work", (64, 64))
    rounds, shapes = 100, [(2, 8 + i) for i in range(eng._MAX_GRAPHS + 1)]
    for _ in range(rounds):
        for s in shapes:
            step(*s)
    # one recording for each of the first eight, then one per _RUNS_TO_EVICT rounds
    assert sum(e[0] == "record" for e in log) <= eng._MAX_GRAPHS + rounds / eng._RUNS_TO_EVICT
    assert sum(e[0] == "replay" for e in log) >= (rounds - 2) * eng._MAX_GRAPHS - eng._MAX_GRAPHS
    assert len(eng._graphs) == eng._MAX_GRAPHS


def test_the_least_recently_used_graph_gives_way(graph_engine):
    eng, step, log = graph_engine
    eng._buf("work", (64, 64))
    shapes = [(2, 8 + i) for i in range(eng._MAX_GRAPHS)]
    for s in shapes:
        assert step(*s) == ["run"] and step(*s) == ["record", "replay"]
    assert step(*shapes[0]) == ["replay"]               # now shapes[1] was used longest ago
    for _ in range(eng._RUNS_TO_EVICT):
        assert step(3, 8) == ["run"]
    assert step(3, 8) == ["record", "replay"]
    assert step(*shapes[0]) == ["replay"] and step(*shapes[2]) == ["replay"] and step(*shapes[1]) == ["run"]


def test_growing_steps_are_not_recorded_in_between(graph_engine):
    """A short shape that alternates with ever longer ones: each growth of a workspace drops what was recorded before it."""
    eng, step, log = graph_engine
    for i in range(20):
        step(2, 8)
        step(2, 16 + i)
    assert not any(e[0] == "record" for e in log)
    assert step(2, 8) == ["run"] and step(2, 8) == ["record", "replay"]      # once it has stopped


def test_shard_optimizer_reads_the_gradient_shard_once(monkeypatch):
    _, eng = _mk(_tiny())
    reads, shard = [], FusedLlama.grad_shard
    monkeypatch.setattr(FusedLlama, "grad_shard", property(lambda self: reads.append(1) or shard.fget(self)))
    eng.set_shard_optimizer(lambda ps: torch.optim.SGD(ps, lr=0.1))
    assert len(reads) == 1
    for (name, _), q in zip(eng.named_master_shards(), eng._shard_params):
        assert q.grad.data_ptr() == eng.shard_view(eng._grad_shard, name).data_ptr()


@pytest.mark.parametrize("graphed", [False, True])
def test_a_gradient_shard_in_hand_follows_the_steps(graph_engine, monkeypatch, graphed):
    """Without peers the shard is filled for those who ask for it: who keeps the tensor finds each step's gradients in it, and those
    of the last step while the next one's accumulate."""
    eng, _, log = graph_engine
    eng._solo, eng._grad_shard = True, None
    monkeypatch.setattr(eng, "_graphable", lambda *a: graphed)

    def step(value):
        def backward(*a):
            eng.grads.fill_(value)
            eng._accum = True
        monkeypatch.setattr(eng, "_accumulate_micro_batches", backward)
        x = torch.zeros(1, 8, dtype=torch.int64)
        if graphed:
            eng.on_replay = lambda: eng.grads.fill_(value)
            eng.train_step(x, x, lr=1e-3, sync_loss=False)
        else:                    # what train_step does on a GPU; the CPU has an update of its own
            backward()
            monkeypatch.setattr(eng, "device", torch.device("cuda"))
            eng.optimizer_step(1e-3)
            monkeypatch.setattr(eng, "device", torch.device("cpu"))
    step(1.0)
    assert eng._grad_shard is None                       # nobody asked yet
    held = eng.grad_shard
    assert (held == 1).all()
    for v in (2.0, 3.0, 4.0):
        step(v)
        assert (held == v).all() and eng.grad_shard is held
    eng.grads.fill_(9.0)                                 # the next step's backward
    assert (eng.grad_shard == 4).all()
