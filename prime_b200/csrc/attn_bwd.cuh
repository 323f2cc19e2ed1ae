// What the two backward attention kernels (heads of up to 64 columns, attn_bwd_sm100.cu, and of up to 128, attn_bwd128_sm100.cu)
// share: parameters, work items, the arithmetic of a score tile and the write-out of a kv tile's gradients.
#pragma once
#include "common.cuh"

namespace pb {

struct AttnBwdParams {
    int M, H, KV, n_tiles;
    int hd;                // columns of a head, <= HD (narrower heads are zero-filled by the tensor maps)
    const int* seq_start;
    const float* lse2;     // [H, M]
    const float* D;        // [H, d_parts, M]: the one or two parts of a row's sum are added up
    int d_parts;
    float* dq_acc;         // [M, H*hd] fp32, zeroed by the span pre-pass of the same call
    __nv_bfloat16* dqkv;   // [M, (H+2KV)*hd]; the backward kernel writes the k and v column blocks
    long long dqkv_stride;
    float scale, scale_log2;
    int* status;
    // query-tile count per kv tile (set by a pre-pass of the launch) and work-item count (= n_tiles * KV)
    int* nq;
    int n_items;
    int* counter;          // the global work counter (next item number)
    const float* rope;     // fp32 [T, hd/2, 2] (cos, sin): dK leaves rotated back; null: as it is
    int T;
};

__device__ __forceinline__ void reg_dealloc_64() { asm volatile("setmaxnreg.dec.sync.aligned.u32 64;"); }
__device__ __forceinline__ void reg_dealloc_88() { asm volatile("setmaxnreg.dec.sync.aligned.u32 88;"); }
__device__ __forceinline__ void reg_alloc_176() { asm volatile("setmaxnreg.inc.sync.aligned.u32 176;"); }

// A work item is one (kv tile, kv head). The grid is one CTA per SM; every CTA draws items from a global counter
// (the producer warp does, and hands the numbers to the other warps through a four-entry ring in shared memory), so
// barriers, tensor memory and the Q/dO ring are set up once per SM and the next item's K/V/Q/dO loads run under the
// current item's dK/dV write-out. Items are numbered head by head, kv tiles in row order, so the CTAs that run at the
// same time share Q, dO and the dQ accumulator rows in L2.
struct BwdItem {
    int kv_tile, g;
};

__device__ __forceinline__ BwdItem bwd_item_of(const AttnBwdParams& p, int idx) {
    BwdItem it;
    it.g = idx / p.n_tiles;
    it.kv_tile = idx - it.g * p.n_tiles;
    return it;
}

// dK (scaled, rotated back) and dV of one kv row, this warp's half of the columns, from tensor memory to the bf16 gradient buffer.
// The inverse RoPE of dK happens here on the fp32 sums: as part of the finish kernel it cost another read and write of dK.
template <int HD>
__device__ __forceinline__ void bwd_write_dkdv(const AttnBwdParams& p, uint32_t tDK, uint32_t tDV, int row, int g, int half) {
    __nv_bfloat16* dk_row = p.dqkv + (long long)row * p.dqkv_stride + (p.H + g) * p.hd;
    __nv_bfloat16* dv_row = p.dqkv + (long long)row * p.dqkv_stride + (p.H + p.KV + g) * p.hd;
    const float* cs_row = p.rope ? p.rope + (long long)(row % p.T) * p.hd : nullptr;
#pragma unroll 1
    for (int cidx = half * (HD / 2); cidx < (half + 1) * (HD / 2); cidx += 32) {
        uint32_t a[32], b[32];
        tmem_ld32(tDK + cidx, a);
        tmem_ld32(tDV + cidx, b);
        tmem_ld_wait();
        if (row < p.M) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
                if (cidx + i >= p.hd) break;
                uint32_t u[4], w[4];
                float cs[8];
                if (p.rope) {
                    *reinterpret_cast<float4*>(cs) = *reinterpret_cast<const float4*>(cs_row + cidx + i);
                    *reinterpret_cast<float4*>(cs + 4) = *reinterpret_cast<const float4*>(cs_row + cidx + i + 4);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    float x = __uint_as_float(a[i + 2 * t]) * p.scale, y = __uint_as_float(a[i + 2 * t + 1]) * p.scale;
                    if (p.rope) {
                        const float xr = x * cs[2 * t] + y * cs[2 * t + 1];
                        y = y * cs[2 * t] - x * cs[2 * t + 1];
                        x = xr;
                    }
                    u[t] = pack_bf16x2(x, y);
                    w[t] = pack_bf16x2(__uint_as_float(b[i + 2 * t]), __uint_as_float(b[i + 2 * t + 1]));
                }
                *reinterpret_cast<uint4*>(dk_row + cidx + i) = make_uint4(u[0], u[1], u[2], u[3]);
                *reinterpret_cast<uint4*>(dv_row + cidx + i) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
}

// Row constants of one (query head, query tile) pair for the thread's query row.
struct BwdRow {
    float lse, Dr;
    int my_start;
    int q0, tile_last_start;
};

template <bool PARTS>      // D may lie in two parts
__device__ __forceinline__ BwdRow bwd_row(const AttnBwdParams& p, int hq, int q_tile, int r) {
    BwdRow x;
    x.q0 = q_tile * 128;
    const int row = x.q0 + r;
    const bool row_ok = row < p.M;
    x.lse = row_ok ? p.lse2[(long long)hq * p.M + row] : 0.f;
    x.Dr = row_ok ? p.D[(long long)hq * (PARTS ? p.d_parts : 1) * p.M + row] : 0.f;
    if (PARTS && row_ok && p.d_parts > 1) x.Dr += p.D[((long long)hq * 2 + 1) * p.M + row];
    x.my_start = row_ok ? p.seq_start[row] : 0x7fffffff;   // a row past M sees no kv position
    x.tile_last_start = p.seq_start[min(x.q0 + 127, p.M - 1)];
    return x;
}

__device__ __forceinline__ bool bwd_needs_mask(const AttnBwdParams& p, const BwdRow& x, int kv0) {
    return (kv0 + 127 > x.q0) || (kv0 < x.tile_last_start) || (x.q0 + 127 >= p.M);
}

// Scores of one query row against 64 kv positions from s0 on -> probabilities as packed bf16 pairs in sv[0..31]. Exponentials are
// taken two at a time on packed bf16 pairs (ex2.approx.bf16x2): the result is P as the MMA will read it, and dS is formed from
// those same rounded values.
template <bool MASK>
__device__ __forceinline__ void bwd_probs(uint32_t (&sv)[64], const BwdRow& x, int row, int s0, float c) {
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
        float x0 = __uint_as_float(sv[i]) * c - x.lse;
        float x1 = __uint_as_float(sv[i + 1]) * c - x.lse;
        if (MASK) {
            if (s0 + i > row || s0 + i < x.my_start) x0 = -INFINITY;
            if (s0 + i + 1 > row || s0 + i + 1 < x.my_start) x1 = -INFINITY;
        }
        asm("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(sv[i >> 1]) : "r"(pack_bf16x2(x0, x1)));
    }
}

// dS = P * (dP - D), packed bf16 pairs in dv[0..31]
__device__ __forceinline__ void bwd_dscores(const uint32_t (&pv)[64], uint32_t (&dv)[64], float D) {
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
        const uint32_t e = pv[i >> 1];
        dv[i >> 1] = pack_bf16x2(__uint_as_float(e << 16) * (__uint_as_float(dv[i]) - D), __uint_as_float(e & 0xffff0000u) * (__uint_as_float(dv[i + 1]) - D));
    }
}

// Both in one pass, for a thread that holds S and dP at the same time: the arithmetic of one pair of values fills the latency of the
// other's exponential (heads of 64, 4 x 8192 tokens: 2.00 ms, one pass after the other 2.13).
template <bool MASK>
__device__ __forceinline__ void bwd_probs_dscores(uint32_t (&sv)[64], uint32_t (&dv)[64], const BwdRow& x, int row, int s0, float c) {
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
        float x0 = __uint_as_float(sv[i]) * c - x.lse;
        float x1 = __uint_as_float(sv[i + 1]) * c - x.lse;
        if (MASK) {
            if (s0 + i > row || s0 + i < x.my_start) x0 = -INFINITY;
            if (s0 + i + 1 > row || s0 + i + 1 < x.my_start) x1 = -INFINITY;
        }
        uint32_t e;
        asm("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(e) : "r"(pack_bf16x2(x0, x1)));
        const float d0 = __uint_as_float(e << 16) * (__uint_as_float(dv[i]) - x.Dr);
        const float d1 = __uint_as_float(e & 0xffff0000u) * (__uint_as_float(dv[i + 1]) - x.Dr);
        sv[i >> 1] = e;
        dv[i >> 1] = pack_bf16x2(d0, d1);
    }
}

// This row's 64 packed values -> column half `half` of a [128 x 128] bf16 tile (two 128-byte-swizzled blocks of 64 columns)
__device__ __forceinline__ void bwd_store_half(uint8_t* tile, const uint32_t (&v)[64], int half, int r) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
        *reinterpret_cast<uint4*>(tile + half * 16384 + r * 128 + ((q ^ (r & 7)) << 4)) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// 64 dQ columns of one row (scaled) -> this warp's two staging boxes of 32 rows x 32 floats, 128-byte-swizzled
__device__ __forceinline__ void bwd_stage_dq(uint8_t* boxes, const uint32_t (&v)[64], int lane, float scale) {
#pragma unroll
    for (int q = 0; q < 16; ++q)
        *reinterpret_cast<float4*>(boxes + (q >> 3) * 4096 + lane * 128 + (((q & 7) ^ (lane & 7)) << 4)) =
            make_float4(__uint_as_float(v[4 * q]) * scale, __uint_as_float(v[4 * q + 1]) * scale, __uint_as_float(v[4 * q + 2]) * scale,
                        __uint_as_float(v[4 * q + 3]) * scale);
}

int launch_attn_bwd128(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tdq, const AttnBwdParams& p, cudaStream_t st);
int sm_count();

}  // namespace pb
