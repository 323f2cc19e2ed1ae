"""Which route a call takes, and what the C entries refuse, as far as that needs no GPU."""
import ctypes as C

import pytest
import torch

from prime_b200 import native
from prime_b200.ops import kernels as K


def _lib():
    try:
        return native.cuda()
    except native.NativeError:
        pytest.skip("CUDA library not built")


# a made-up address must not reach a device, even if the check that this tests is lost
no_device = pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up")


@no_device
@pytest.mark.parametrize("fp32", [True, False])
def test_splitk_reduce_refuses_what_its_vectors_do_not_fit(fp32):
    """Outputs and addends off the 16 (fp32) or 8 (bf16) bytes of four elements: refused before any launch (the addresses are made up)."""
    lib, size, base = _lib(), 4 if fp32 else 2, 1 << 40

    def call(ws=base, res=0, out=base, ld_out=1028, ld_res=1028, N=1024):
        return lib.pb_splitk_reduce(C.c_void_p(ws), 2, 256, N, C.c_void_p(res or None), ld_res, C.c_void_p(out), ld_out, int(fp32), None)
    for k in (1, 2, 3):
        assert call(out=base + k * size) == -1
        assert call(res=base + k * size) == -1
        assert call(ws=base + 4 * k) == -1
        assert call(ld_out=1028 + k) == -1
        assert call(res=base, ld_res=1028 + k) == -1
        assert call(N=1024 + k) == -1


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_splitk_is_chosen_for_whole_vectors_only(dtype):
    wide = torch.zeros(256, 1032, dtype=dtype)
    good = wide[:, 4:1028]
    assert K._splitk_fits(good, None) and K._splitk_fits(good, good)
    for bad in (wide[:, 1:1025], wide[:, 2:1026], torch.zeros(256, 1030, dtype=dtype)[:, :1024]):
        assert not K._splitk_fits(bad, None) and not K._splitk_fits(good, bad)


@no_device
def test_attention_backward_refuses_rows_off_16_bytes():
    """o and dqkv are read and written in 16-byte vectors that no tensor map checks."""
    lib = _lib()
    from prime_b200.ops import attention  # noqa: F401  (declares the C signatures)
    base = 1 << 40

    def call(**off):
        a = [C.c_void_p(base + off.get(k, 0)) for k in ("qkv", "o", "dout", "lse2", "ss", "dqkv", "dq", "D")]
        return lib.pb_attn_bwd(*a, None, 1, 256, 4, 2, 64, 512, 256, 256, 512, 0.125, None, None, None)
    for k in ("qkv", "o", "dout", "dqkv"):
        for bytes_off in (2, 4, 8):
            assert call(**{k: bytes_off}) == -2


def test_narrow_heads_are_copied_only_where_the_kernels_cannot_reach_them():
    from prime_b200.ops import attention as A
    wide = torch.zeros(16, 272, dtype=torch.bfloat16)
    fits = wide[:, 8:264]
    for bad in (wide[:, 1:257], torch.zeros(16, 260, dtype=torch.bfloat16)[:, :256], torch.zeros(256, 16, dtype=torch.bfloat16).t()):
        for hd in (8, 32, 96):
            assert A._fitting_input(fits, hd) is fits and A._fitting_output(fits, hd) is fits
            assert A._rows_fit(A._fitting_input(bad, hd)) and A._rows_fit(A._fitting_output(bad, hd))
        for hd in (64, 128):
            assert A._fitting_input(bad, hd) is bad and A._fitting_output(bad, hd) is bad
    assert A._fitting_output(torch.zeros(16, 256), 32).dtype == torch.bfloat16


def test_scratch_belongs_to_one_thread_and_is_bounded(monkeypatch):
    import threading
    monkeypatch.setattr(native, "raw_stream", lambda index=None: 7)
    monkeypatch.setattr(K, "_scratch", {})
    dev = torch.device("cpu")
    mine, theirs = K._scratch_buf(dev, "splitk", 100), []
    t = threading.Thread(target=lambda: theirs.append(K._scratch_buf(dev, "splitk", 100)))
    t.start()
    t.join()
    assert mine.data_ptr() != theirs[0].data_ptr()                    # one stream, one use, two threads
    assert K._scratch_buf(dev, "splitk", 80).data_ptr() == mine.data_ptr()
    for i in range(200):                                              # what stays in use outlives what does not
        K._scratch_buf(dev, f"use{i}", 1)
        assert K._scratch_buf(dev, "splitk", 100).data_ptr() == mine.data_ptr() and len(K._scratch) <= 64
    got = K.take_scratch(type("S", (), {"cuda_stream": 7})())
    assert any(g.data_ptr() == mine.data_ptr() for g in got) and not any(k[3] == threading.get_ident() for k in K._scratch)


def test_odd_swiglu_blocks_are_fused_up_to_the_measured_lines():
    fits = [(512, 192, 1536), (1024, 704, 1536), (65536, 2752, 384)]
    loses = [(1024, 1472, 1024), (65536, 704, 392), (512, 192, 2048), (4736, 320, 512)]
    assert all(K._narrow_swiglu_pays(*s, 74) for s in fits) and not any(K._narrow_swiglu_pays(*s, 74) for s in loses)


class _NoLaunch:
    """Stands in for the CUDA library: every entry only notes that it was reached."""
    def __init__(self):
        self.reached = []

    def __getattr__(self, name):
        return lambda *a: self.reached.append(name) or 0


def test_fused_products_refuse_operands_that_the_plain_product_refuses(monkeypatch):
    lib = _NoLaunch()
    monkeypatch.setattr(native, "cuda", lambda: lib)
    monkeypatch.setattr(native, "stream_ptr", lambda *a: None)
    monkeypatch.setattr(K, "stream_ptr", lambda *a: None)
    monkeypatch.setattr(K, "status_word", lambda d: torch.zeros(1, dtype=torch.int32))
    x, w, h, act = (torch.zeros(*s, dtype=torch.bfloat16) for s in ((512, 128), (384, 128), (512, 384), (512, 192)))

    def call(x, w, h13=h):
        K._gemm_epi(x, w, h13, 512, 384, 128, False, 1, 192, 0, 0, act, "swiglu")
    wide = torch.zeros(512, 256, dtype=torch.bfloat16)
    for bad in ((x.float(), w), (x, w.float()), (x.half(), w), (wide[:, ::2], w), (x, torch.zeros(384, 256, dtype=torch.bfloat16)[:, ::2]),
                (x, torch.zeros(384, 136, dtype=torch.bfloat16)), (x, w, h.float())):
        with pytest.raises(AssertionError):
            call(*bad)
    assert not lib.reached
    call(x, w)
    assert lib.reached


@pytest.mark.parametrize("group", [64, 128])
def test_row_dots_do_not_apply_to_rows_that_tma_cannot_move(group):
    out, dots = torch.zeros(512, 256, dtype=torch.bfloat16), torch.zeros(4 * 512)
    wide = torch.zeros(512, 272, dtype=torch.bfloat16)
    assert K._rowdot_fits(512, 256, out, out, dots, group) and K._rowdot_fits(512, 256, wide[:, 8:264], out, dots, group)
    for bad in (wide[:, 1:257], torch.zeros(512, 260, dtype=torch.bfloat16)[:, :256], torch.zeros(256, 512, dtype=torch.bfloat16).t(), out.float(),
                out[:, :128]):
        assert not K._rowdot_fits(512, 256, bad, out, dots, group) and not K._rowdot_fits(512, 256, out, bad, dots, group)
    assert not K._rowdot_fits(512, 256, out, out, dots[:-1], group) and not K._rowdot_fits(512, 256, out, out, dots.double(), group)


@no_device
def test_attention_backward_refuses_partial_sums_that_its_kernels_do_not_read():
    lib = _lib()
    from prime_b200.ops import attention  # noqa: F401  (declares the C signatures)
    base = C.c_void_p(1 << 40)

    def call(hd, d_parts, o=None):
        n = 4 * hd
        return lib.pb_attn_bwd_parts(base, o, base, base, base, base, base, base, d_parts, None, 1, 256, 4, 2, hd, 2 * n, n, n, 2 * n, 0.125, None, None, None)
    for hd, parts in ((64, 2), (32, 2), (128, 3), (128, 0), (64, 0), (128, -1)):
        assert call(hd, parts) == -4
    # accepted as far as this check goes (without a device the next step fails), and not asked where the kernel takes the sums itself
    assert all(call(hd, parts) != -4 for hd, parts in ((64, 1), (128, 1), (128, 2), (96, 2))) and call(64, 2, base) != -4
