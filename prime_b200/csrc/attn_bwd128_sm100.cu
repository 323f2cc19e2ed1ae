// Attention backward for heads of 65 to 128 columns (zero-filled to 128 by the tensor maps): the same work items, masks and
// sums as attn_bwd_sm100.cu, with another pipeline, since neither the shared nor the tensor memory holds what that one keeps.
//
// Shared memory: K, V, two Q tiles, one dO tile, P and dS of 32 KB each. The dQ staging boxes of the drain warps (64 KB a pair)
// have no room of their own: columns 0-63 go through the P tile once the dV MMA has read it, columns 64-127 through the dS tile
// once the dK MMA has. Tensor memory: S | dP | dV | dK of 128 columns; dQ takes the place of dP, whose values the softmax
// warps hold in registers by then.
//
// Per pair i the tensor core runs
//   S(i+1)             as soon as the softmax warps hold S(i): their exponentials of pair i+1 run under the MMAs of pair i
//   dV(i), dQ(i), dK(i) when P(i) and dS(i) are in shared memory; dO's tile is refilled behind dV, Q's behind dK
//   dP(i+1)            when the drain warps have read dQ(i), which they do under dK(i)
// so that between "P and dS are there" of two pairs stand the four MMAs, one read of dP, and dS = P (dP - D). With one Q / dO
// stage, S and dP issued together and dQ in the place of S (the earlier form of this kernel) every step waited for the one before:
// whole backward, 8 x 2048 tokens, 16 heads 771 -> 626 us, 1 x 8192, 32 / 8 heads 2733 -> 2047.
// What bounds it: the chain, no unit is full. A pair takes 7400 cycles (8 x 2048 tokens, 16 heads), of which the five MMAs need 2560
// (tensor pipe 35 %); the way of the dQ sums to L2 is busy for 45 %, the data banks of shared memory and L1 read for 20 % and written
// for 10 %. A softmax warp spends half of its time waiting for tensor memory: dP(i+1) follows the read of dQ(i), which follows dS(i),
// which follows dP(i).
#include "attn_bwd.cuh"

namespace pb {

struct AttnBwd128Cfg {
    static constexpr int TILE = 128 * 128 * 2;
    static constexpr int SMEM_BYTES = 7 * TILE + 1024 + 256;
    static constexpr int T_S = 0, T_DP = 128, T_DV = 256, T_DK = 384;
};

__global__ void __launch_bounds__(512, 1)
attn_bwd128_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmDQ, const AttnBwdParams p) {
    using Cfg = AttnBwd128Cfg;
    constexpr int TILE = Cfg::TILE;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t sK = base, sV = sK + TILE, sQ = sV + TILE /* [2] */, sDO = sQ + 2 * TILE, sP = sDO + TILE, sDS = sP + TILE;
    uint8_t* gP = gen + (sP - base);
    uint8_t* gDS = gen + (sDS - base);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gen + 7 * TILE);
    const uint32_t bar_kv = smem_u32(bars);
    const uint32_t bar_final = bar_kv + 8;       // every MMA of an item has retired
    const uint32_t bar_qfull = bar_final + 8;    // [2]
    const uint32_t bar_qempty = bar_qfull + 16;  // [2] dK of the pair has retired
    const uint32_t bar_dofull = bar_qempty + 16;
    const uint32_t bar_doempty = bar_dofull + 8; // dV of the pair has retired
    const uint32_t bar_sfull = bar_doempty + 8;
    const uint32_t bar_sfree = bar_sfull + 8;    // softmax warps hold S in registers (count 8)
    const uint32_t bar_dpfull = bar_sfree + 8;
    const uint32_t bar_pdsfull = bar_dpfull + 8; // P and dS are in shared memory, dP is out of TMEM (count 8)
    const uint32_t bar_dqfull = bar_pdsfull + 8; // dV and dQ of the pair have retired
    const uint32_t bar_dqempty = bar_dqfull + 8; // drain warps have read dQ out of TMEM (count 4)
    const uint32_t bar_dkdone = bar_dqempty + 8; // dK of the pair has retired
    const uint32_t bar_pfree = bar_dkdone + 8;   // the dQ boxes in the P tile have been sent (count 4)
    const uint32_t bar_dsfree = bar_pfree + 8;   // ... and those in the dS tile (count 4)
    ItemRing items;
    items.bar_full = bar_dsfree + 8;                // [4]
    items.bar_empty = items.bar_full + 32;          // [4]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17 + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    items.ring = reinterpret_cast<volatile int*>(tmem_slot + 2);
    items.abort_flag = abort_flag;
    items.status = p.status;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.H / p.KV;

    if (threadIdx.x == 0) {
        mbar_init(bar_kv, 1);
        mbar_init(bar_final, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar_qfull + 8 * s, 1);
            mbar_init(bar_qempty + 8 * s, 1);
        }
        mbar_init(bar_dofull, 1);
        mbar_init(bar_doempty, 1);
        mbar_init(bar_sfull, 1);
        mbar_init(bar_sfree, 8);
        mbar_init(bar_dpfull, 1);
        mbar_init(bar_pdsfull, 8);
        mbar_init(bar_dqfull, 1);
        mbar_init(bar_dqempty, 4);
        mbar_init(bar_dkdone, 1);
        mbar_init(bar_pfree, 4);
        mbar_init(bar_dsfree, 4);
        for (int s = 0; s < 4; ++s) {
            mbar_init(items.bar_full + 8 * s, 1);
            mbar_init(items.bar_empty + 8 * s, 13);   // MMA thread, eight softmax warps, four drain warps
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQKV);
        tma_prefetch_desc(&tmDO);
        tma_prefetch_desc(&tmDQ);
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
    // a wait of a whole warp
    auto wait = [&](uint32_t bar, uint32_t parity, int code) -> bool {
        const bool good = mbar_wait(bar, parity & 1, abort_flag, p.status, code);
        return __all_sync(0xffffffffu, good);
    };

    if (warp < 4) {
        reg_dealloc_64();
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            bool ok = true;
            uint32_t gi = 0;          // running pair count: ring stages and barrier parities carry over from item to item
            int idx = items.publish(0, p.counter, p.n_items);
            for (int k = 0; ok && idx >= 0; ++k) {
                const BwdItem item = bwd_item_of(p, idx);
                const int kv0 = item.kv_tile * 128;
                const int n_q = p.nq[item.kv_tile];
                if (k > 0) {   // every MMA of the previous item has retired: K and V may be replaced
                    ok = wait(bar_final, k - 1, PB_ERR_TIMEOUT_EMPTY);
                    if (!ok) break;
                }
                if (lane == 0) {
                    mbar_expect_tx(bar_kv, 2 * TILE);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        tma_load_3d(sK + b * 16384, &tmQKV, bar_kv, 64 * b, p.H + item.g, kv0);
                        tma_load_3d(sV + b * 16384, &tmQKV, bar_kv, 64 * b, p.H + p.KV + item.g, kv0);
                    }
                }
                int hq = item.g * G, qi = 0;
                const int n_it = n_q * G;
                for (int it = 0; it < n_it; ++it, ++gi) {
                    const int st = gi & 1;
                    const int q0 = (item.kv_tile + qi) * 128;
                    ok = wait(bar_qempty + 8 * st, (gi >> 1) ^ 1, PB_ERR_TIMEOUT_EMPTY);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(bar_qfull + 8 * st, TILE);
#pragma unroll
                        for (int b = 0; b < 2; ++b) tma_load_3d(sQ + st * TILE + b * 16384, &tmQKV, bar_qfull + 8 * st, 64 * b, hq, q0);
                    }
                    ok = wait(bar_doempty, gi ^ 1, PB_ERR_TIMEOUT_EMPTY);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(bar_dofull, TILE);
#pragma unroll
                        for (int b = 0; b < 2; ++b) tma_load_3d(sDO + b * 16384, &tmDO, bar_dofull, 64 * b, hq, q0);
                    }
                    __syncwarp();
                    if (++qi == n_q) { qi = 0; ++hq; }
                }
                if (!ok) break;
                // drawn only now, with this item's last loads in flight: a CTA busy with a heavy item leaves the counter to the others
                idx = items.publish(k + 1, p.counter, p.n_items);
                if (idx == -2) ok = false;
            }
            if (!ok) for (int i = 0; i < 64; ++i) __nanosleep(10000);
        } else if (warp == 1) {
            // ------------------------------ MMA issuer (one thread) ------------------------------
            if (lane == 0) {
                constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
                constexpr uint32_t idesc_kv = umma_idesc_bf16(128, 128, 1, 1);   // dV, dK: both operands MN-major
                constexpr uint32_t idesc_dq = umma_idesc_bf16(128, 128, 0, 1);
                const uint32_t tS = tmem_base + Cfg::T_S, tDP = tmem_base + Cfg::T_DP, tDV = tmem_base + Cfg::T_DV, tDK = tmem_base + Cfg::T_DK;
                bool ok = true;
                auto await = [&](uint32_t bar, uint32_t parity, int code) {
                    ok = ok && mbar_wait(bar, parity & 1, abort_flag, p.status, code);
                };
                // D = A B^T over 128 columns of both tiles (two 64-column blocks)
                auto rows = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t c0) {
                    umma4_f16_ss_peek(d, umma_smem_desc(a, 16, 1024), umma_smem_desc(b, 16, 1024), 2, 2, idesc_s, 0u, 0, 0, 0, 0, 0, 0, 0);
                    umma4_f16_ss_peek(d, umma_smem_desc(a + 16384, 16, 1024), umma_smem_desc(b + 16384, 16, 1024), 2, 2, idesc_s, 1u, c0, 0, 0, 0, 0, 0, 0);
                };
                // D (+)= A^T B over the 128 rows of both tiles; up to three commits
                auto cols = [&](uint32_t d, uint32_t a, uint32_t b, bool acc, uint32_t c0, uint32_t c1, uint32_t c2) {
                    umma4_f16_ss_peek(d, umma_smem_desc(a, 16384, 1024), umma_smem_desc(b, 16384, 1024), 128, 128, idesc_kv, acc ? 1u : 0u, 0, 0, 0, 0, 0, 0, 0);
                    umma4_f16_ss_peek(d, umma_smem_desc(a + 8192, 16384, 1024), umma_smem_desc(b + 8192, 16384, 1024), 128, 128, idesc_kv, 1u, c0, c1, c2, 0, 0, 0, 0);
                };
                auto issue_s = [&](uint32_t g) {
                    await(bar_qfull + 8 * (g & 1), g >> 1, PB_ERR_TIMEOUT_FULL);
                    if (g > 0) await(bar_sfree, g - 1, PB_ERR_TIMEOUT_TMEM_EMPTY);
                    if (!ok) return;
                    tc_fence_after();
                    rows(tS, sQ + (g & 1) * TILE, sK, bar_sfull);
                };
                auto issue_dp = [&](uint32_t g) {
                    await(bar_dofull, g, PB_ERR_TIMEOUT_FULL);
                    if (g > 0) await(bar_dqempty, g - 1, PB_ERR_TIMEOUT_TMEM_EMPTY);
                    if (!ok) return;
                    tc_fence_after();
                    rows(tDP, sDO, sV, bar_dpfull);
                };
                uint32_t gi = 0;      // running pair count over all items of this CTA
                for (int k = 0; ok; ++k) {
                    const int idx = items.take_thread(k);
                    if (idx < 0) break;
                    const int n_it = p.nq[bwd_item_of(p, idx).kv_tile] * G;
                    await(bar_kv, k, PB_ERR_TIMEOUT_FULL);
                    if (!ok) break;
                    issue_s(gi);
                    issue_dp(gi);
                    for (int it = 0; it < n_it && ok; ++it, ++gi) {
                        const bool more = it + 1 < n_it;
                        if (more) issue_s(gi + 1);
                        await(bar_pdsfull, gi, PB_ERR_TIMEOUT_MISC);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t q = sQ + (gi & 1) * TILE;
                        // the first pair of an item starts new accumulators: the softmax warps wrote the previous item's dK / dV out
                        // before they signalled this pair's P and dS
                        cols(tDV, sP, sDO, it > 0, bar_doempty, 0, 0);
                        umma4_f16_ss_peek(tDP, umma_smem_desc(sDS, 16, 1024), umma_smem_desc(sK, 16384, 1024), 2, 128, idesc_dq, 0u, 0, 0, 0, 0, 0, 0, 0);
                        umma4_f16_ss_peek(tDP, umma_smem_desc(sDS + 16384, 16, 1024), umma_smem_desc(sK + 8192, 16384, 1024), 2, 128, idesc_dq, 1u,
                                          bar_dqfull, 0, 0, 0, 0, 0, 0);
                        cols(tDK, sDS, q, it > 0, bar_dkdone, bar_qempty + 8 * (gi & 1), more ? 0 : bar_final);
                        if (more) issue_dp(gi + 1);
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp >= 12) {
        reg_dealloc_88();
        // ------------------------------ dQ drain warps ------------------------------
        // dQ of one pair -> registers -> staging boxes in the P and dS tiles -> bulk reduce-add into the fp32 accumulator (rows past
        // M are clipped by the tensor map). Warp w moves the 32 query rows of quadrant w & 3.
        const int quad = warp & 3;
        const uint32_t tDQ = tmem_base + Cfg::T_DP + (uint32_t(quad * 32) << 16);
        bool ok = true;
        uint32_t gi = 0;
        for (int k = 0; ok; ++k) {
            const int idx = items.take(k);
            if (idx < 0) break;
            const BwdItem item = bwd_item_of(p, idx);
            const int n_q = p.nq[item.kv_tile];
            const int n_it = n_q * G;
            int hq = item.g * G, qi = 0;
            for (int it = 0; it < n_it; ++it, ++gi) {
                ok = wait(bar_dqfull, gi, PB_ERR_TIMEOUT_TMEM_FULL);
                if (!ok) break;
                tc_fence_after();
                const int dq_y = (item.kv_tile + qi) * 128 + quad * 32;
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    uint32_t v[64];
                    tmem_ld32(tDQ + 64 * part, *reinterpret_cast<uint32_t(*)[32]>(v));
                    tmem_ld32(tDQ + 64 * part + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
                    tmem_ld_wait();
                    if (part) {                              // all of dQ is in registers or on its way
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(bar_dqempty);
                            tma_store_wait_read<0>();
                            mbar_arrive(bar_pfree);
                        }
                        __syncwarp();
                        ok = wait(bar_dkdone, gi, PB_ERR_TIMEOUT_TMEM_FULL);      // the dK MMA has read dS
                        if (!ok) break;
                    }
                    const uint32_t box = (part ? sDS : sP) + quad * 8192;
                    bwd_stage_dq(gen + (box - base), v, lane, p.scale);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (64 * part < p.hd) tma_reduce_add_3d(&tmDQ, box, 64 * part, hq, dq_y);
                        if (64 * part + 32 < p.hd) tma_reduce_add_3d(&tmDQ, box + 4096, 64 * part + 32, hq, dq_y);
                        tma_store_commit();
                    }
                }
                if (!ok) break;
                if (lane == 0) {
                    tma_store_wait_read<0>();
                    mbar_arrive(bar_dsfree);
                }
                __syncwarp();
                if (++qi == n_q) { qi = 0; ++hq; }
            }
        }
        if (lane == 0) tma_store_wait<0>();   // all reduce-adds of this warp have landed
    } else {
        reg_alloc_176();
        // ------------------------------ softmax / dS / write-out warps ------------------------------
        // Eight warps: warp w reads TMEM lane quadrant w & 3 (a hardware rule) and takes column half
        // (w - 4) >> 2 of every 128-wide row, so two warps share each query row of the tile.
        const int quad = warp & 3;
        const int half = (warp - 4) >> 2;
        const int r = quad * 32 + lane;
        const uint32_t lane_off = uint32_t(quad * 32) << 16;
        const uint32_t tS = tmem_base + Cfg::T_S + lane_off + half * 64, tDP = tmem_base + Cfg::T_DP + lane_off + half * 64,
                       tDV = tmem_base + Cfg::T_DV + lane_off, tDK = tmem_base + Cfg::T_DK + lane_off;
        const float c = p.scale_log2;
        bool ok = true;
        uint32_t gi = 0;
        int idx = items.take(0);
        BwdItem item = {};
        int n_q = 0;
        BwdRow cur = {};
        if (idx >= 0) {
            item = bwd_item_of(p, idx);
            n_q = p.nq[item.kv_tile];
            cur = bwd_row<true>(p, item.g * G, item.kv_tile, r);
        }
        for (int k = 0; idx >= 0; ++k) {
            const int kv0 = item.kv_tile * 128, g = item.g, n_it = n_q * G;
            int hq = g * G, qi = 0;
            for (int it = 0; it < n_it; ++it, ++gi) {
                uint32_t sv[64], dv[64];
                ok = wait(bar_sfull, gi, PB_ERR_TIMEOUT_TMEM_FULL);
                if (!ok) break;
                tc_fence_after();
                tmem_ld32(tS, *reinterpret_cast<uint32_t(*)[32]>(sv));
                tmem_ld32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(sv + 32));
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_sfree);
                const BwdRow x = cur;
                if (++qi == n_q) { qi = 0; ++hq; }
                if (it + 1 < n_it) cur = bwd_row<true>(p, hq, item.kv_tile + qi, r);      // lands while this pair is exponentiated
                if (bwd_needs_mask(p, x, kv0)) bwd_probs<true>(sv, x, x.q0 + r, kv0 + half * 64, c);
                else bwd_probs<false>(sv, x, x.q0 + r, kv0 + half * 64, c);
                if (gi > 0) {   // dV of the previous pair has read its P, and the dQ boxes that followed it there have left
                    ok = wait(bar_pfree, gi - 1, PB_ERR_TIMEOUT_MISC);
                    if (!ok) break;
                }
                bwd_store_half(gP, sv, half, r);
                ok = wait(bar_dpfull, gi, PB_ERR_TIMEOUT_TMEM_FULL);
                if (!ok) break;
                tc_fence_after();
                tmem_ld32(tDP, *reinterpret_cast<uint32_t(*)[32]>(dv));
                tmem_ld32(tDP + 32, *reinterpret_cast<uint32_t(*)[32]>(dv + 32));
                tmem_ld_wait();
                bwd_dscores(sv, dv, x.Dr);
                if (gi > 0) {
                    ok = wait(bar_dsfree, gi - 1, PB_ERR_TIMEOUT_MISC);
                    if (!ok) break;
                }
                bwd_store_half(gDS, dv, half, r);
                tc_fence_before();
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_pdsfull);
            }
            if (!ok) break;
            // dK and dV of this kv tile, once every MMA of the item has retired; the next item's first row constants are
            // requested before, so that they arrive under it
            ok = wait(bar_final, k, PB_ERR_TIMEOUT_TMEM_FULL);
            if (!ok) break;
            idx = items.take(k + 1);
            if (idx >= 0) {
                item = bwd_item_of(p, idx);
                n_q = p.nq[item.kv_tile];
                cur = bwd_row<true>(p, item.g * G, item.kv_tile, r);
            }
            tc_fence_after();
            bwd_write_dkdv<128>(p, tDK, tDV, kv0 + r, g, half);
            tc_fence_before();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

int launch_attn_bwd128(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tdq, const AttnBwdParams& p, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(attn_bwd128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnBwd128Cfg::SMEM_BYTES) != cudaSuccess) return -20;
        configured = true;
    }
    const int grid = p.n_items < sm_count() ? p.n_items : sm_count();     // one CTA per SM draws items until none are left
    launch_pdl(attn_bwd128_kernel, LaunchCfg(grid, 512, AttnBwd128Cfg::SMEM_BYTES, st), tq, tdo, tdq, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -30;
}

}  // namespace pb
