// Attention forward for heads of 65 to 128 columns (zero-filled to 128 by the tensor map): inputs, masks and results of
// attn_fwd_sm100.cu.
//
// One CTA per SM works on two adjacent 128-row query tiles of one head at a time, which share every K and V tile they read
// from L2. 384 threads in three warpgroups: warp 0 TMA producer, warps 1 and 2 MMA issuers of the two query tiles (one thread
// each; warp 1 owns TMEM), warp 3 only fills the warpgroup; warps 4-7 and 8-11 softmax of the first and the second tile (one
// thread per query row: row max / sum are thread-local). The exponentials of one tile run under the MMAs of the other; the first
// warpgroup gives registers up (setmaxnreg) so that a softmax thread can hold its 128-wide score row without spilling.
// The grid has a CTA for every pair of tiles of every head, but a CTA that runs takes over the work of CTAs that have not started
// (clusterlaunchcontrol), so that barriers and tensor memory are set up once per SM and the next pair's Q, K and V arrive under the
// end of this one, while the hardware still deals the pairs out one by one. Every issuer and softmax group moves on to the next
// pair by itself.
//   S = Q K^T            -> TMEM [128 x 128] fp32
//   P = exp2(S*c - m*c)  -> bf16 pairs in TMEM (tcgen05.st), read by the PV MMA as its A operand
//   O  += P V            -> TMEM [128 x 128] fp32, accumulated by the MMA across KV tiles; rows are
//                           rescaled in TMEM only when their running maximum grows by > 2^8
// Outputs: o[M, H*HD] bf16 and lse2[H, M] = log2-sum-exp of the scaled scores (log2 units).
#include "attn_fwd.cuh"

namespace pb {

struct AttnFwd128Cfg {
    static constexpr int TILE_BYTES = 128 * 128 * 2;         // one Q / K / V tile
    static constexpr int RING = 5;                           // K and V tiles in turn: K0 V0 K1 V1 ...
    static constexpr int SMEM_BYTES = TILE_BYTES * (2 + RING) + 1024 + 512;
    // TMEM columns of the two query tiles: S (fp32) 128 each from 0, O (fp32) 128 each from 256. P (bf16 pairs, A operand of the PV
    // MMA) takes the place of S, whose row the softmax thread already holds, and the next S follows PV. Two CTAs per SM with
    // a tile each (the earlier form) had the same overlap, but fetched every K and V tile twice, into one stage:
    // 8 x 2048 tokens, 16 heads 227 -> 190 us; 1 x 8192, 32 / 8 heads 702 -> 606.
};

__device__ __forceinline__ void fwd_reg_dealloc_56() { asm volatile("setmaxnreg.dec.sync.aligned.u32 56;"); }
__device__ __forceinline__ void fwd_reg_alloc_224() { asm volatile("setmaxnreg.inc.sync.aligned.u32 224;"); }

// Cluster launch control: ask for the work of a CTA that has not started yet. The answer (16 bytes) lands in shared memory and
// completes `bar`. Once it was "none left", no further request may be made.
__device__ __forceinline__ void clc_request(uint32_t answer, uint32_t bar) {
    mbar_expect_tx(bar, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer), "r"(bar) : "memory");
}
__device__ __forceinline__ bool clc_answer(uint32_t answer, int& x) {
    uint32_t got;
    asm volatile(
        "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
        "ld.shared.b128 h, [%2];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "mov.b32 %1, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}\n"
        : "=r"(got), "=r"(x)
        : "r"(answer)
        : "memory");
    return got != 0;
}

// What every role needs to know of a pair of query tiles of `head`: the first tile (the other is the next one) and the first kv tile of
// each (the last one is the query tile's own number). head < 0: no more work.
struct FwdItem {
    int tile, head, lo[2];
};

__global__ void __launch_bounds__(384, 1)
attn_fwd128_kernel(const __grid_constant__ CUtensorMap tm, const AttnFwdParams p, const int per_cta, const int n_units) {
    using Cfg = AttnFwd128Cfg;
    constexpr int HD = 128, TILE = Cfg::TILE_BYTES, RING = Cfg::RING;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t sQ = base;                        // [2]
    const uint32_t sKV = sQ + 2 * TILE;              // [RING]
    uint64_t* bars = reinterpret_cast<uint64_t*>(gen + TILE * (2 + RING));
    const uint32_t clc_slot = smem_u32(bars);        // 16 bytes
    const uint32_t bar_clc = clc_slot + 16;
    const uint32_t bar_qfull = bar_clc + 8;          // [2] by query tile
    const uint32_t bar_qempty = bar_qfull + 16;      // [2] the tile's last S has retired
    const uint32_t bar_sfull = bar_qempty + 16;      // [2]
    const uint32_t bar_pfull = bar_sfull + 16;       // [2] (count 4)
    const uint32_t bar_pv = bar_pfull + 16;          // [2] O += P V of a kv tile has retired
    const uint32_t bar_ofree = bar_pv + 16;          // [2] O of a finished query tile has been read (count 4)
    const uint32_t bar_full = bar_ofree + 16;        // [RING]
    const uint32_t bar_empty = bar_full + 8 * RING;  // [RING] both query tiles are done with the K or V tile (count 2)
    const uint32_t bar_ifull = bar_empty + 8 * RING; // [4] item ring
    const uint32_t bar_iempty = bar_ifull + 32;      // [4] (count 10: two MMA threads, eight softmax warps)
    int* ring = reinterpret_cast<int*>(gen + (bar_iempty + 32 - base));                    // [4] FwdItem
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(bar_clc, 1);
        for (int g = 0; g < 2; ++g) {
            mbar_init(bar_qfull + 8 * g, 1);
            mbar_init(bar_qempty + 8 * g, 1);
            mbar_init(bar_sfull + 8 * g, 1);
            mbar_init(bar_pfull + 8 * g, 4);
            mbar_init(bar_pv + 8 * g, 1);
            mbar_init(bar_ofree + 8 * g, 4);
        }
        for (int s = 0; s < RING; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 2);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(bar_ifull + 8 * s, 1);
            mbar_init(bar_iempty + 8 * s, 10);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tm);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_sync();

    const int n_tiles = (p.M + 127) / 128;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) -> bool {      // one thread
        return mbar_wait(bar, parity & 1, abort_flag, p.status, code);
    };
    auto wait_warp = [&](uint32_t bar, uint32_t parity, int code) -> bool {
        const bool good = mbar_wait(bar, parity & 1, abort_flag, p.status, code);
        return __all_sync(0xffffffffu, good);
    };
    // the k-th item, read by a thread whose wait for the entry has succeeded
    auto read_item = [&](int k) {
        const volatile int* e = ring + 4 * (k & 3);
        FwdItem it;
        it.tile = e[0]; it.head = e[1]; it.lo[0] = e[2]; it.lo[1] = e[3];
        return it;
    };

    // 128 x 56 + 256 x 224 registers = those of the launch, 384 x 168
    if (warp < 4) {
        fwd_reg_dealloc_56();
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            bool ok = true;
            int x = blockIdx.x;                  // number of the CTA whose work this is; -1: none left
            uint32_t nq[2] = {0, 0};             // query tiles loaded
            int slot = 0;                        // next K / V slot of the ring
            uint32_t ph = 0;
            auto load_q = [&](int g, int head, int tile) -> bool {
                if (!wait_warp(bar_qempty + 8 * g, nq[g] ^ 1, PB_ERR_TIMEOUT_EMPTY)) return false;
                ++nq[g];
                if (lane == 0) {
                    mbar_expect_tx(bar_qfull + 8 * g, TILE);
#pragma unroll
                    for (int b = 0; b < 2; ++b) tma_load_3d(sQ + g * TILE + b * 16384, &tm, bar_qfull + 8 * g, 64 * b, head, tile * 128);
                }
                __syncwarp();
                return true;
            };
            auto load_kv = [&](int col_head, int tile) -> bool {
                if (!wait_warp(bar_empty + 8 * slot, ph ^ 1, PB_ERR_TIMEOUT_EMPTY)) return false;
                if (lane == 0) {
                    mbar_expect_tx(bar_full + 8 * slot, TILE);
#pragma unroll
                    for (int b = 0; b < 2; ++b) tma_load_3d(sKV + slot * TILE + b * 16384, &tm, bar_full + 8 * slot, 64 * b, col_head, tile * 128);
                }
                __syncwarp();
                if (++slot == RING) { slot = 0; ph ^= 1; }
                return true;
            };
            for (int k = 0;; ++k) {
                const bool have = x >= 0;
                const int head = have ? x % p.H : -1;
                const int tile = have ? (n_units - 1 - x / p.H) * per_cta : 0;     // latest (heaviest) tiles of all heads first
                int lo0 = 0, lo1 = 0;
                const bool two = per_cta == 2 && tile + 1 < n_tiles;
                if (have) {
                    lo0 = p.seq_start[tile * 128] / 128;
                    lo1 = two ? p.seq_start[tile * 128 + 128] / 128 : lo0;
                }
                ok = wait_warp(bar_iempty + 8 * (k & 3), ((k >> 2) & 1) ^ 1, PB_ERR_TIMEOUT_EMPTY);
                if (!ok) break;
                if (lane == 0) {
                    volatile int* e = ring + 4 * (k & 3);
                    e[0] = tile; e[1] = head; e[2] = lo0; e[3] = lo1;
                    mbar_arrive(bar_ifull + 8 * (k & 3));
                }
                __syncwarp();
                if (!have) break;
                const int kvh = head / (p.H / p.KV);
                const int lo = min(lo0, lo1), hi = two ? tile + 1 : tile;
                ok = load_q(0, head, tile);
                for (int j = lo; j <= hi && ok; ++j) {
                    ok = load_kv(p.H + kvh, j);
                    if (ok && j == lo && two) ok = load_q(1, head, tile + 1);
                    if (ok) ok = load_kv(p.H + p.KV + kvh, j);
                }
                if (!ok) break;
                // the next pair is asked for only now, with this one's last loads in flight: a CTA that is still busy leaves the work to others
                if (lane == 0) {
                    fence_proxy_async_smem();                     // the last answer has been read
                    clc_request(clc_slot, bar_clc);
                }
                __syncwarp();
                ok = wait_warp(bar_clc, k, PB_ERR_TIMEOUT_MISC);
                if (!ok) break;
                int nx;
                const bool got = clc_answer(clc_slot, nx);
                __syncwarp();
                x = got ? nx : -1;
            }
            if (!ok) for (int i = 0; i < 64; ++i) __nanosleep(10000);
        } else if (warp < 3) {
            // ------------------------------ MMA issuers ------------------------------
            if (lane == 0) {
                const int g = warp - 1;
                constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
                constexpr uint32_t idesc_o = umma_idesc_bf16(128, HD, 0, 1);
                const uint32_t tS = tmem_base + 128 * g, tO = tmem_base + 256 + HD * g, tP = tS;
                bool ok = true;
                int slot = 0;                    // ring position of the next K or V tile of this query tile
                uint32_t ph = 0, t = 0, nq = 0;  // kv tiles and query tiles done
                auto next = [&] { if (++slot == RING) { slot = 0; ph ^= 1; } };
                auto skip = [&] {                // a K or V tile that only the other query tile sees: release it once it is there
                    if (ok) ok = wait(bar_full + 8 * slot, ph, PB_ERR_TIMEOUT_FULL);
                    if (ok) mbar_arrive(bar_empty + 8 * slot);
                    next();
                };
                // S of a kv tile whose K is at (ks, kph)
                auto issue_s = [&](int ks, uint32_t kph, bool last) {
                    ok = wait(bar_full + 8 * ks, kph, PB_ERR_TIMEOUT_FULL);
                    if (!ok) return;
                    tc_fence_after();
                    const uint32_t q = sQ + g * TILE, kb = sKV + ks * TILE;
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        umma4_f16_ss_peek(tS, umma_smem_desc(q + b * 16384, 16, 1024), umma_smem_desc(kb + b * 16384, 16, 1024), 2, 2, idesc_s,
                                          b ? 1u : 0u, b ? bar_sfull + 8 * g : 0, b ? bar_empty + 8 * ks : 0,
                                          b && last ? bar_qempty + 8 * g : 0, 0, 0, 0, 0);
                };
                for (int k = 0; ok; ++k) {
                    ok = wait(bar_ifull + 8 * (k & 3), k >> 2, PB_ERR_TIMEOUT_FULL);
                    if (!ok) break;
                    const FwdItem it = read_item(k);
                    mbar_arrive(bar_iempty + 8 * (k & 3));
                    if (it.head < 0) break;
                    const bool two = per_cta == 2 && it.tile + 1 < n_tiles;
                    const int hi = two ? it.tile + 1 : it.tile;               // last kv tile that is loaded
                    const bool live = g == 0 || two;
                    const int first = live ? it.lo[g] : hi + 1, last = live ? it.tile + g : hi;
                    for (int j = min(it.lo[0], it.lo[1]); j < first; ++j) { skip(); skip(); }
                    if (live) {
                        ok = ok && wait(bar_qfull + 8 * g, nq, PB_ERR_TIMEOUT_FULL);
                        if (!ok) break;
                        issue_s(slot, ph, first == last);
                        for (int j = first; j <= last && ok; ++j, ++t) {
                            next();
                            const int vs = slot;
                            const uint32_t vph = ph;
                            next();
                            // now at K of the kv tile after this one
                            ok = wait(bar_full + 8 * vs, vph, PB_ERR_TIMEOUT_FULL) && wait(bar_pfull + 8 * g, t, PB_ERR_TIMEOUT_MISC);
                            if (ok && j == first && nq > 0) ok = wait(bar_ofree + 8 * g, nq - 1, PB_ERR_TIMEOUT_TMEM_EMPTY);
                            if (!ok) break;
                            tc_fence_after();
                            const uint32_t vb = sKV + vs * TILE;
#pragma unroll
                            for (int h = 0; h < 2; ++h)     // 128 kv rows, 16 per MMA; A = P straight from tensor memory, 8 columns per MMA
                                umma4_f16_ts_peek(tO, tP + 32 * h, umma_smem_desc(vb + h * 8192, 16384, 1024), 8, 128, idesc_o,
                                                  (j > first || h) ? 1u : 0u, h ? bar_pv + 8 * g : 0, h ? bar_empty + 8 * vs : 0, 0, 0, 0, 0, 0);
                            // tcgen05.mma of one thread run in the order of issue: S may overwrite the P that PV reads
                            if (j < last) issue_s(slot, ph, j + 1 == last);
                        }
                        ++nq;
                    }
                    if (!ok) break;
                    for (int j = last + 1; j <= hi; ++j) { skip(); skip(); }
                }
            }
            __syncwarp();
        }
    } else {
        fwd_reg_alloc_224();
        // ------------------------------ softmax warps ------------------------------
        // One thread per query row. The whole 128-wide score row is pulled from TMEM in one go and
        // stays in registers; O lives in TMEM (the PV MMA accumulates into it) and is rescaled only
        // when a row's running maximum grows by more than 2^8 -- until then exponentials use the
        // older maximum, which is exact after the final division by the row sum.
        const int quad = warp & 3, g = (warp - 4) >> 2;
        const int r = quad * 32 + lane;           // row within the tile == TMEM lane
        const uint32_t lane_off = uint32_t(quad * 32) << 16;
        const uint32_t tS = tmem_base + 128 * g + lane_off, tO = tmem_base + 256 + HD * g + lane_off, tP = tS;
        const float c = p.scale_log2;
        bool ok = true;
        uint32_t t = 0;                           // kv tiles done
        for (int k = 0;; ++k) {
            ok = wait_warp(bar_ifull + 8 * (k & 3), k >> 2, PB_ERR_TIMEOUT_FULL);
            if (!ok) break;
            const FwdItem it = read_item(k);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_iempty + 8 * (k & 3));
            if (it.head < 0) break;
            const int tile = it.tile + g;
            if (g && (per_cta == 1 || tile >= n_tiles)) continue;
            const int q0 = tile * 128, row = q0 + r;
            const int my_start = p.seq_start[min(row, p.M - 1)];
            const int tile_last_start = p.seq_start[min(q0 + 127, p.M - 1)];
            float m_used = -INFINITY, l_run = 0.f;
            const int first = g ? it.lo[1] : it.lo[0];
            for (int j = first; j <= tile; ++j, ++t) {
                const int kv0 = j * 128;
                ok = wait_warp(bar_sfull + 8 * g, t, PB_ERR_TIMEOUT_TMEM_FULL);
                if (!ok) break;
                tc_fence_after();
                uint32_t v[4][32];
#pragma unroll
                for (int q = 0; q < 4; ++q) tmem_ld32(tS + 32 * q, v[q]);
                tmem_ld_wait();
                const bool need_mask = (kv0 + 127 > q0) || (kv0 < tile_last_start);
                if (need_mask) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int s = kv0 + 32 * q + i;
                            if (!(s <= row && s >= my_start)) v[q][i] = 0xff800000u;      // -inf
                        }
                }
                // row maximum: 3-input max over four independent chains
                float mxp[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        mxp[(i >> 1) & 3] = max3(mxp[(i >> 1) & 3], __uint_as_float(v[q][i]), __uint_as_float(v[q][i + 1]));
                const float mx = fmaxf(fmaxf(mxp[0], mxp[1]), fmaxf(mxp[2], mxp[3]));
                const bool grow = (mx != -INFINITY) && (m_used == -INFINITY || (mx - m_used) * c > 8.f);
                if (__any_sync(0xffffffffu, grow)) {
                    const float m_new = grow ? fmaxf(m_used, mx) : m_used;
                    const float alpha = (m_used == -INFINITY) ? 0.f : exp2f((m_used - m_new) * c);
                    if (j > first) {      // O of the previous tiles exists (their PV came before this S): rescale the row
#pragma unroll
                        for (int cidx = 0; cidx < HD; cidx += 32) {
                            uint32_t o[32];
                            tmem_ld32(tO + cidx, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st32(tO + cidx, o);
                        }
                        tmem_st_wait();
                    }
                    l_run *= alpha;
                    m_used = m_new;
                }
                const float m_sub = (m_used == -INFINITY) ? 0.f : m_used * c;
                // P = exp2(S*c - m*c): the scale-and-shift and the row sum run on packed fp32 pairs (one f32x2
                // instruction per two scores), the exponentials on the special-function unit (16 per clock per SM
                // whether packed or not, so they are taken in fp32, one per score)
                const unsigned long long cc = f32x2_pack(c, c), nm = f32x2_pack(-m_sub, -m_sub);
                unsigned long long rs2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pw[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const unsigned long long x2 =
                            f32x2_fma(f32x2_pack(__uint_as_float(v[q][2 * i]), __uint_as_float(v[q][2 * i + 1])), cc, nm);
                        float x0, x1;
                        f32x2_unpack(x2, x0, x1);
                        const float e0 = ex2_approx(x0), e1 = ex2_approx(x1);      // masked entries are -inf -> 0
                        pw[i] = pack_bf16x2(e0, e1);
                        rs2[i & 3] = f32x2_add(rs2[i & 3], f32x2_pack(e0, e1));
                    }
                    tmem_st16(tP + 16 * q, pw);   // 32 kv columns = 16 packed words of this row
                }
                {
                    float a0, a1;
                    f32x2_unpack(f32x2_add(f32x2_add(rs2[0], rs2[1]), f32x2_add(rs2[2], rs2[3])), a0, a1);
                    l_run += a0 + a1;
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_pfull + 8 * g);
            }
            if (ok) ok = wait_warp(bar_pv + 8 * g, t - 1, PB_ERR_TIMEOUT_TMEM_FULL);
            if (!ok) break;
            tc_fence_after();
            const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
            __nv_bfloat16* dst = p.O + (long long)row * p.o_stride + it.head * p.hd;
#pragma unroll
            for (int cidx = 0; cidx < HD; cidx += 64) {
                uint32_t o[64];
                tmem_ld32(tO + cidx, *reinterpret_cast<uint32_t(*)[32]>(o));
                tmem_ld32(tO + cidx + 32, *reinterpret_cast<uint32_t(*)[32]>(o + 32));
                tmem_ld_wait();
                if (cidx + 64 == HD) {            // the next query tile's PV may write O
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_ofree + 8 * g);
                }
                if (row < p.M) {
#pragma unroll
                    for (int i = 0; i < 64; i += 8) {
                        if (cidx + i >= p.hd) break;
                        uint4 u;
                        u.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                        u.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                        u.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                        u.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + cidx + i) = u;
                    }
                }
            }
            if (row < p.M) p.lse2[(long long)it.head * p.M + row] = (l_run > 0.f) ? (m_used * c + log2f(l_run)) : -INFINITY;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// Two tiles per CTA, but one where every tile then has an SM to itself. CTAs are numbered with the head running fastest, so that the
// long rows of all heads start first and the short ones fill the end: with the tiles running fastest the last heads' longest pairs
// started late, and from 150 to 800 tiles of long rows two to a CTA lost 2-8 % against one each. One CTA per tile; tiles fastest; heads
// fastest, us: 1 x 4096 tokens, 16 heads 140, 149, 100; 1 x 8192, 8 heads 246, 268, 187; 32 / 8 heads 703, 666, 606; 64 x 1024, 16 heads
// 503, 441, 429. What still loses to one CTA per tile: up to two tiles per SM of long rows (1 x 4096, 8 heads 94 and 98; one
// tile per CTA takes 72 there, but 45 instead of 35 at 37 x 777, one head, and the launch does not know where rows end), and rows of
// 128 tokens (8 x 128, 8 heads, one launch behind the other, 7.3 and 7.8).
int launch_attn_fwd128(const CUtensorMap& tm, const AttnFwdParams& p, cudaStream_t st) {
    using Cfg = AttnFwd128Cfg;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(attn_fwd128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess) return -20;
        configured = true;
    }
    const int n_tiles = (p.M + 127) / 128, n_sm = sm_count();
    const int per_cta = n_tiles * p.H <= n_sm ? 1 : 2;
    const int n_units = (n_tiles + per_cta - 1) / per_cta;
    launch_pdl(attn_fwd128_kernel, LaunchCfg(n_units * p.H, 384, Cfg::SMEM_BYTES, st), tm, p, per_cta, n_units);
    return cudaGetLastError() == cudaSuccess ? 0 : -30;
}

}  // namespace pb
