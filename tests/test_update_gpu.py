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
                                             ptr(m), ptr(v), 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, ptr(sq), 1.0, 148, stream_ptr()),
          "pb_zero_adamw_gather")
    for a, b, n in segs:
        g = (gsrc[b: b + n] if kind == 0 else gsrc[a: a + n]).float().cpu()
        rp, rm, rv = (t[b: b + n].cpu() for t in ref)
        K.adamw_(rp, g, rm, rv, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, gnorm=torch.tensor(4.0), max_norm=1.0)
        for got, want in ((p, rp), (m, rm), (v, rv)):
            assert torch.allclose(got[b: b + n].cpu(), want, rtol=2e-5, atol=2e-6)
        assert torch.equal(params[a: a + n], p[b: b + n].bfloat16())
