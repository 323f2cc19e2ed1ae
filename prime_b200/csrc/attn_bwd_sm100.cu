// Flash attention backward (causal / document mask, GQA) for sm_100a on tcgen05 + TMEM + TMA.
//
// A work item is one 128-row KV tile of one KV head; the CTA that holds it walks every (query head of the
// group, query tile) pair that can see it. Per pair (all MMAs are 128-row tcgen05 instructions):
//   S  = Q K^T,  dP = dO V^T                 -> TMEM
//   P  = exp2(S*c - lse2),  dS = P * (dP - D) -> bf16 in shared memory (softmax warps)
//   dV += P^T dO,  dK += dS^T Q               -> TMEM accumulators kept for the whole item
//   dQ  = dS K                                -> TMEM -> shared memory -> bulk reduce-add (TMA) into dq_acc
// Heads of up to 64 columns (the kernel for wider ones is in attn_bwd128_sm100.cu). The pairs are software-pipelined: the tensor
// core computes S/dP of pair i+1 and dV/dK/dQ of pair i-1 while the softmax warps work on pair i from registers.
// D[h, m] = rowsum(dO * O) comes from a small pre-pass. dK/dV of a KV head are reduced over the
// query heads of its group inside the CTA (no repeat_kv materialisation, no cross-CTA atomics
// for them). The same shared-memory tile is consumed K-major by one MMA and MN-major by another
// (e.g. Q is A of S and B of dK), which the 128-byte-swizzled layout allows without a copy.
// Gradient semantics match autograd through the reference attention
// (models/llama/model.py:282-302) for scores scaled by `scale`.
#include "attn_bwd.cuh"

namespace pb {

struct AttnBwdCfg {
    static constexpr int HD = 64;
    static constexpr int TILE_BYTES = 128 * HD * 2;
    static constexpr int PS_BYTES = 128 * 128 * 2;
    static constexpr int STAGES = 3;
    static constexpr int DQ_STAGE_BYTES = 8 * 4096;   // one 32-row x 32-float box per softmax warp
    static constexpr int SMEM_BYTES = TILE_BYTES * (2 + 2 * STAGES) + 2 * PS_BYTES + DQ_STAGE_BYTES + 1024 + 256;
    static constexpr int T_S = 0, T_DP = 128;
    static constexpr int T_DV = 256, T_DK = 256 + HD, T_DQ = 384;
};

// 512 threads in four warpgroups (register budgets are re-split with setmaxnreg):
//   warps 0-3   : warp 0 = TMA producer, warp 1 = MMA issuer (2 and 3 only hold the warpgroup together)
//   warps 4-11  : softmax warps; warp w reads TMEM lane quadrant w & 3 and column half (w - 4) >> 2
//   warps 12-15 : dQ drain warps; warp w moves the 32 query rows of quadrant w & 3 to dq_acc
__global__ void __launch_bounds__(512, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmDQ, const AttnBwdParams p) {
    using Cfg = AttnBwdCfg;
    constexpr int HD = Cfg::HD, STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t sK = base;
    const uint32_t sV = sK + Cfg::TILE_BYTES;
    const uint32_t sQ = sV + Cfg::TILE_BYTES;                    // [STAGES]
    const uint32_t sDO = sQ + STAGES * Cfg::TILE_BYTES;          // [STAGES]
    const uint32_t sP = sDO + STAGES * Cfg::TILE_BYTES;
    const uint32_t sDS = sP + Cfg::PS_BYTES;
    uint8_t* gP = gen + (sP - base);
    uint8_t* gDS = gen + (sDS - base);
    const uint32_t sDQ = sDS + Cfg::PS_BYTES;                    // [4 drain warps][2 boxes][32 rows][32 floats], 128B-swizzled
    uint64_t* bars = reinterpret_cast<uint64_t*>(gen + (sDQ - base) + Cfg::DQ_STAGE_BYTES);
    const uint32_t bar_kv = smem_u32(bars);
    const uint32_t bar_qfull = bar_kv + 8;           // [3] Q and dO of a pair are in shared memory
    const uint32_t bar_qdoempty = bar_qfull + 24;    // [3]
    const uint32_t bar_sdpfull = bar_qdoempty + 24;  // S and dP of a pair are in TMEM
    const uint32_t bar_sdpfree = bar_sdpfull + 8;    // softmax warps hold S and dP in registers (count 8)
    const uint32_t bar_pdsfull = bar_sdpfree + 8;    // P and dS of a pair are in shared memory (count 8)
    const uint32_t bar_dqfull = bar_pdsfull + 8;     // dV/dK/dQ MMAs of a pair are done: dQ readable, P/dS reusable
    const uint32_t bar_dqempty = bar_dqfull + 8;     // drain warps have read dQ out of TMEM (count 4)
    const uint32_t bar_final = bar_dqempty + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    ItemRing items;
    items.bar_full = bar_final + 8;                 // [4]
    items.bar_empty = items.bar_full + 32;          // [4]
    items.ring = reinterpret_cast<volatile int*>(tmem_slot + 2);
    items.abort_flag = abort_flag;
    items.status = p.status;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.H / p.KV;

    if (threadIdx.x == 0) {
        mbar_init(bar_kv, 1);
        for (int s = 0; s < 3; ++s) {
            mbar_init(bar_qfull + 8 * s, 1);
            mbar_init(bar_qdoempty + 8 * s, 1);
        }
        mbar_init(bar_sdpfull, 1);
        mbar_init(bar_sdpfree, 8);
        mbar_init(bar_pdsfull, 8);
        mbar_init(bar_dqfull, 1);
        mbar_init(bar_dqempty, 4);
        mbar_init(bar_final, 1);
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

    if (warp < 4) {
        reg_dealloc_64();
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            bool ok = true;
            uint32_t gi = 0;          // running pair count: ring stage and barrier parities carry over from item to item
            int idx = items.publish(0, p.counter, p.n_items);
            for (int k = 0; ok && idx >= 0; ++k) {
                const BwdItem item = bwd_item_of(p, idx);
                const int kv0 = item.kv_tile * 128;
                const int n_q = p.nq[item.kv_tile];
                if (k > 0) {   // every MMA of the previous item has retired: K and V may be replaced
                    ok = mbar_wait(bar_final, (k - 1) & 1, abort_flag, p.status, PB_ERR_TIMEOUT_EMPTY);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                if (lane == 0) {
                    mbar_expect_tx(bar_kv, 2 * Cfg::TILE_BYTES);
                    tma_load_3d(sK, &tmQKV, bar_kv, 0, p.H + item.g, kv0);
                    tma_load_3d(sV, &tmQKV, bar_kv, 0, p.H + p.KV + item.g, kv0);
                }
                int hq = item.g * G, qi = 0;
                const int n_it = n_q * G;
                for (int it = 0; it < n_it && ok; ++it, ++gi) {
                    const int st = gi % STAGES;
                    const uint32_t ph = (gi / STAGES) & 1;
                    ok = mbar_wait(bar_qdoempty + 8 * st, ph ^ 1, abort_flag, p.status, PB_ERR_TIMEOUT_EMPTY);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (lane == 0) {
                        const int q0 = (item.kv_tile + qi) * 128;
                        mbar_expect_tx(bar_qfull + 8 * st, 2 * Cfg::TILE_BYTES);   // Q and dO land on one barrier
                        tma_load_3d(sQ + st * Cfg::TILE_BYTES, &tmQKV, bar_qfull + 8 * st, 0, hq, q0);
                        tma_load_3d(sDO + st * Cfg::TILE_BYTES, &tmDO, bar_qfull + 8 * st, 0, hq, q0);
                    }
                    __syncwarp();
                    if (++qi == n_q) { qi = 0; ++hq; }
                }
                if (!ok) break;
                // The next item is drawn only now, when this item's last loads are in flight: a CTA that is still busy
                // with a heavy item leaves the counter to the others. The other warps ask for it after their last pair.
                idx = items.publish(k + 1, p.counter, p.n_items);
                if (idx == -2) ok = false;
            }
            if (!ok) for (int i = 0; i < 64; ++i) __nanosleep(10000);
        } else if (warp == 1) {
            // ------------------------------ MMA issuer ------------------------------
            // One thread runs the whole loop. Barriers that are certain to complete while a batch of
            // MMAs is being issued are polled inside that batch (umma4_f16_ss_peek), so their latency
            // is not paid between batches.
            if (lane == 0) {
                constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
                constexpr uint32_t idesc_kv = umma_idesc_bf16(128, HD, 1, 1);   // dV, dK: both operands MN-major
                constexpr uint32_t idesc_dq = umma_idesc_bf16(128, HD, 0, 1);
                const uint32_t tS = tmem_base + Cfg::T_S, tDP = tmem_base + Cfg::T_DP, tDV = tmem_base + Cfg::T_DV,
                               tDK = tmem_base + Cfg::T_DK, tDQ = tmem_base + Cfg::T_DQ;
                bool ok = true;
                // S = Q K^T and dP = dO V^T of running pair gi (operands in stage gi % STAGES); polls (peek, par) meanwhile
                auto issue_s_dp = [&](uint32_t gi, bool q_ready, uint32_t peek, uint32_t par) -> bool {
                    const int st = gi % STAGES;
                    const uint32_t ph = (gi / STAGES) & 1;
                    if (!q_ready) {
                        ok = mbar_wait(bar_qfull + 8 * st, ph, abort_flag, p.status, PB_ERR_TIMEOUT_FULL);
                        if (!ok) return false;
                    }
                    tc_fence_after();
                    const uint32_t q = sQ + st * Cfg::TILE_BYTES, d = sDO + st * Cfg::TILE_BYTES;
                    umma4_f16_ss_peek(tS, umma_smem_desc(q, 16, 1024), umma_smem_desc(sK, 16, 1024), 2, 2, idesc_s, 0u, 0, 0, 0, 0, 0, 0, 0);
                    const uint32_t got = umma4_f16_ss_peek(tDP, umma_smem_desc(d, 16, 1024), umma_smem_desc(sV, 16, 1024), 2, 2, idesc_s, 0u,
                                                           bar_sdpfull, 0, 0, peek, par, 0, 0);
                    return got & 1;
                };
                uint32_t gi = 0;      // running pair count over all items of this CTA
                for (int k = 0; ok; ++k) {
                    const int idx = items.take_thread(k);
                    if (idx < 0) break;
                    const int n_it = p.nq[bwd_item_of(p, idx).kv_tile] * G;
                    ok = mbar_wait(bar_kv, k & 1, abort_flag, p.status, PB_ERR_TIMEOUT_FULL);
                    if (!ok) break;
                    if (gi > 0) {   // the softmax warps hold the previous item's last pair in registers (long since)
                        ok = mbar_wait(bar_sdpfree, (gi - 1) & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_EMPTY);
                        if (!ok) break;
                    }
                    issue_s_dp(gi, false, 0, 0);
                    bool sdpfree_ready = false, qnext_ready = false;
                    for (int it = 0; it < n_it && ok; ++it, ++gi) {
                        const int st = gi % STAGES;
                        bool pds_ready = false;
                        if (it + 1 < n_it) {
                            if (!sdpfree_ready) {
                                ok = mbar_wait(bar_sdpfree, gi & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_EMPTY);
                                if (!ok) break;
                            }
                            pds_ready = issue_s_dp(gi + 1, qnext_ready, bar_pdsfull, gi & 1);
                            if (!ok) break;
                        }
                        if (!pds_ready) {
                            ok = mbar_wait(bar_pdsfull, gi & 1, abort_flag, p.status, PB_ERR_TIMEOUT_MISC);
                            if (!ok) break;
                        }
                        tc_fence_after();
                        const uint32_t q = sQ + st * Cfg::TILE_BYTES, d = sDO + st * Cfg::TILE_BYTES;
                        const bool wait_dqe = gi > 0;   // the drain warps have read dQ of the previous pair
                        uint32_t got = 0;
                        // dV += P^T dO, dK += dS^T Q: reduction over the 128 query rows, 16 per MMA; the first pair of an
                        // item starts new accumulators (the softmax warps wrote the previous item's dK/dV out before they
                        // signalled this pair's P and dS)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            got |= umma4_f16_ss_peek(tDV, umma_smem_desc(sP + h * 8192, 16384, 1024), umma_smem_desc(d + h * 8192, 16384, 1024),
                                                     128, 128, idesc_kv, (it | h) ? 1u : 0u, 0, 0, 0,
                                                     (h == 0 && wait_dqe) ? bar_dqempty : 0, (gi - 1) & 1, 0, 0);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            umma4_f16_ss_peek(tDK, umma_smem_desc(sDS + h * 8192, 16384, 1024), umma_smem_desc(q + h * 8192, 16384, 1024),
                                              128, 128, idesc_kv, (it | h) ? 1u : 0u, 0, 0, 0, 0, 0, 0, 0);
                        if (wait_dqe && !(got & 1)) {
                            ok = mbar_wait(bar_dqempty, (gi - 1) & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_EMPTY);
                            if (!ok) break;
                        }
                        if (wait_dqe) tc_fence_after();
                        // dQ = dS K: reduction over the 128 kv rows. Meanwhile poll what the next iteration needs first.
                        const uint32_t gnx = gi + 2;                           // pair whose Q/dO stage is needed next
                        const bool more = it + 2 < n_it;                       // ... if it is one of this item
                        got = umma4_f16_ss_peek(tDQ, umma_smem_desc(sDS, 16, 1024), umma_smem_desc(sK, 16384, 1024), 2, 128, idesc_dq, 0u,
                                                0, 0, 0, more ? bar_qfull + 8 * (gnx % STAGES) : 0, (gnx / STAGES) & 1,
                                                more ? bar_sdpfree : 0, (gi + 1) & 1);
                        umma4_f16_ss_peek(tDQ, umma_smem_desc(sDS + 16384, 16, 1024), umma_smem_desc(sK + 8192, 16384, 1024), 2, 128, idesc_dq,
                                          1u, bar_dqfull, bar_qdoempty + 8 * st, it == n_it - 1 ? bar_final : 0, 0, 0, 0, 0);
                        qnext_ready = got & 1;
                        sdpfree_ready = got & 2;
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp >= 12) {
        reg_dealloc_88();
        // ------------------------------ dQ drain warps ------------------------------
        // dQ tile of one pair -> registers -> this warp's two staging boxes in shared memory -> bulk
        // reduce-add into the fp32 accumulator (rows past M are clipped by the tensor map)
        const int quad = warp & 3;
        const uint32_t tDQ = tmem_base + Cfg::T_DQ + (uint32_t(quad * 32) << 16);
        const uint32_t my_dq = sDQ + quad * 8192;
        uint8_t* g_dq = gen + (my_dq - base);
        bool ok = true;
        uint32_t gi = 0;
        for (int k = 0; ok; ++k) {
            const int idx = items.take(k);
            if (idx < 0) break;
            const BwdItem item = bwd_item_of(p, idx);
            const int n_q = p.nq[item.kv_tile];
            const int n_it = n_q * G;
            int hq = item.g * G, qi = 0;
            for (int it = 0; it < n_it && ok; ++it, ++gi) {
                ok = mbar_wait(bar_dqfull, gi & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_FULL);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const int dq_y = (item.kv_tile + qi) * 128 + quad * 32;
                uint32_t v[64];
                tmem_ld32(tDQ, *reinterpret_cast<uint32_t(*)[32]>(v));
                tmem_ld32(tDQ + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
                if (lane == 0) tma_store_wait_read<0>();   // earlier reduce-adds have read the staging boxes
                __syncwarp();
                tmem_ld_wait();
                tc_fence_before();                         // dQ of this pair is out of TMEM
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_dqempty);
                bwd_stage_dq(g_dq, v, lane, p.scale);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_reduce_add_3d(&tmDQ, my_dq, 0, hq, dq_y);
                    if (p.hd > 32) tma_reduce_add_3d(&tmDQ, my_dq + 4096, 32, hq, dq_y);
                    tma_store_commit();
                }
                if (++qi == n_q) { qi = 0; ++hq; }
            }
        }
        if (lane == 0) tma_store_wait<0>();   // all reduce-adds of this warp have landed
    } else {
        reg_alloc_176();
        // ------------------------------ softmax / dS / epilogue warps ------------------------------
        // Eight warps: warp w reads TMEM lane quadrant w & 3 (a hardware rule) and takes column half
        // (w - 4) >> 2 of every 128-wide row, so two warps share each query row of the tile.
        const int quad = warp & 3;
        const int half = (warp - 4) >> 2;
        const int r = quad * 32 + lane;
        const uint32_t lane_off = uint32_t(quad * 32) << 16;
        const uint32_t tS = tmem_base + Cfg::T_S + lane_off, tDP = tmem_base + Cfg::T_DP + lane_off,
                       tDV = tmem_base + Cfg::T_DV + lane_off, tDK = tmem_base + Cfg::T_DK + lane_off;
        const float c = p.scale_log2;
        bool ok = true;
        // Per (head, query tile) pair: this thread's row constants, then its 64 S and 64 dP values in
        // registers. The pair after the one being exponentiated is already in TMEM.
        // (query head, query tile) of the pair whose row constants are loaded next, inside the current item
        int kv_tile = 0, n_q = 0, hq_n = 0, qi_n = 0;
        auto row_ctx = [&]() {
            const BwdRow x = bwd_row<false>(p, hq_n, kv_tile + qi_n, r);
            if (++qi_n == n_q) { qi_n = 0; ++hq_n; }
            return x;
        };
        uint32_t sv[64], dv[64];
        auto load_sdp = [&](uint32_t gi) -> bool {
            bool good = mbar_wait(bar_sdpfull, gi & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_FULL);
            good = __all_sync(0xffffffffu, good);
            if (!good) return false;
            tc_fence_after();
            tmem_ld32(tS + half * 64, *reinterpret_cast<uint32_t(*)[32]>(sv));
            tmem_ld32(tS + half * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(sv + 32));
            tmem_ld32(tDP + half * 64, *reinterpret_cast<uint32_t(*)[32]>(dv));
            tmem_ld32(tDP + half * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(dv + 32));
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sdpfree);
            return true;
        };
        BwdRow cur = {}, nxt = {};
        uint32_t gi = 0;
        BwdItem item = {};
        int idx = items.take(0);
        bool have = idx >= 0;
        if (have) {
            item = bwd_item_of(p, idx);
            kv_tile = item.kv_tile; n_q = p.nq[kv_tile]; hq_n = item.g * G; qi_n = 0;
            cur = row_ctx();
        }
        for (int k = 0; have && ok; ++k) {
            const int kv0 = kv_tile * 128;
            const int g = item.g;
            int left = n_q * G;                 // pairs of this item not yet started
            ok = load_sdp(gi);
            while (ok) {
                --left;
                if (left) nxt = row_ctx();      // global loads land while this pair is exponentiated
                const int row = cur.q0 + r;
                if (bwd_needs_mask(p, cur, kv0)) bwd_probs_dscores<true>(sv, dv, cur, row, kv0 + half * 64, c);
                else bwd_probs_dscores<false>(sv, dv, cur, row, kv0 + half * 64, c);
                if (gi > 0) {
                    // the MMAs of the previous pair have read its P/dS out of shared memory
                    ok = mbar_wait(bar_dqfull, (gi - 1) & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_FULL);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const uint32_t off = half * 16384 + r * 128 + ((q ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(gP + off) = make_uint4(sv[4 * q], sv[4 * q + 1], sv[4 * q + 2], sv[4 * q + 3]);
                    *reinterpret_cast<uint4*>(gDS + off) = make_uint4(dv[4 * q], dv[4 * q + 1], dv[4 * q + 2], dv[4 * q + 3]);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_pdsfull);
                ++gi;
                if (!left) break;
                cur = nxt;
                ok = load_sdp(gi);
            }
            if (!ok) break;
            // dK (scaled) and dV of this kv tile -> bf16 gradient buffer, once every MMA of the item has retired
            ok = mbar_wait(bar_final, k & 1, abort_flag, p.status, PB_ERR_TIMEOUT_TMEM_FULL);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            // the next item's first row constants are requested before the write-out, so they arrive under it
            idx = items.take(k + 1);
            have = idx >= 0;
            if (have) {
                item = bwd_item_of(p, idx);
                kv_tile = item.kv_tile; n_q = p.nq[kv_tile]; hq_n = item.g * G; qi_n = 0;
                cur = row_ctx();
            }
            tc_fence_after();
            bwd_write_dkdv<HD>(p, tDK, tDV, kv0 + r, g, half);
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

// D[h, m] = sum_d dO[m, h*hd + d] * O[m, h*hd + d]. LPR consecutive lanes (hd / 8 rounded up to a power of two) share one
// (m, h) row and load 16 bytes each; every thread keeps four rows in flight.
template <int LPR>
__global__ void __launch_bounds__(256) attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                            float* __restrict__ D, long long M, int H, int hd, long long o_stride,
                                                            long long do_stride) {
    constexpr int ROWS_PER_BLOCK = 256 / LPR;
    pdl_sync();
    const int sub = threadIdx.x % LPR;
    const long long total = M * H;
    const long long stride = (long long)gridDim.x * ROWS_PER_BLOCK;
    for (long long base = (long long)blockIdx.x * ROWS_PER_BLOCK + threadIdx.x / LPR; base < total; base += 4 * stride) {
        uint4 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long it = base + u * stride;
            if (it < total && sub * 8 < hd) {
                const long long m = it / H;
                const int h = int(it - m * H);
                a[u] = *reinterpret_cast<const uint4*>(o + m * o_stride + h * hd + sub * 8);
                b[u] = *reinterpret_cast<const uint4*>(dout + m * do_stride + h * hd + sub * 8);
            } else {
                a[u] = make_uint4(0, 0, 0, 0);
                b[u] = make_uint4(0, 0, 0, 0);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float2 a0 = unpack_bf16x2(a[u].x), a1 = unpack_bf16x2(a[u].y), a2 = unpack_bf16x2(a[u].z), a3 = unpack_bf16x2(a[u].w);
            const float2 b0 = unpack_bf16x2(b[u].x), b1 = unpack_bf16x2(b[u].y), b2 = unpack_bf16x2(b[u].z), b3 = unpack_bf16x2(b[u].w);
            float acc = a0.x * b0.x + a0.y * b0.y + a1.x * b1.x + a1.y * b1.y + a2.x * b2.x + a2.y * b2.y + a3.x * b3.x + a3.y * b3.y;
#pragma unroll
            for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            const long long it = base + u * stride;
            if (sub == 0 && it < total) {
                const long long m = it / H;
                const int h = int(it - m * H);
                D[(long long)h * M + m] = acc;
            }
        }
    }
}

// dq (fp32 accumulator, [M, H*HD]) -> inverse RoPE -> bf16 q columns of dqkv
__global__ void attn_bwd_finish_kernel(const float* __restrict__ dq_acc, __nv_bfloat16* __restrict__ dqkv,
                                       const float* __restrict__ table, long long M, int T, int H, int HD, long long stride) {
    pdl_sync();
    const int vpr = H * HD / 8, vph = HD / 8;
    const long long total = M * vpr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / vpr;
        const int c = int(i - m * vpr);
        const float4* src = reinterpret_cast<const float4*>(dq_acc + 8 * i);
        const float4 a = src[0], b = src[1];
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t u[4];
        if (table) {
            const float4* cs = reinterpret_cast<const float4*>(table + (m % T) * HD + (c % vph) * 8);
            const float4 c0 = cs[0], c1 = cs[1];
            const float co[4] = {c0.x, c0.z, c1.x, c1.z}, si[4] = {c0.y, c0.w, c1.y, c1.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                u[k] = pack_bf16x2(f[2 * k] * co[k] + f[2 * k + 1] * si[k], f[2 * k + 1] * co[k] - f[2 * k] * si[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) u[k] = pack_bf16x2(f[2 * k], f[2 * k + 1]);
        }
        *reinterpret_cast<uint4*>(dqkv + m * stride + c * 8) = make_uint4(u[0], u[1], u[2], u[3]);
    }
}

// nq[kv_tile] = number of query tiles that can see the kv tile: the diagonal tile plus every later tile whose first
// row's sequence starts at or before the tile's last kv row (seq_start is non-decreasing). One warp per kv tile, 32
// candidate tiles per step (one load latency per 32 tiles instead of one per tile). Also zeroes the work counter and
// the dQ accumulator (n16 vectors of 16 bytes): a memset would break the chain of early launches and cost a launch of its own. Against
// the memset, L2 flushed, a whole backward takes 2 us less at 16 x 1024 tokens, 8 heads of 64, 2 us more at 8 x 2048, 16 heads of 128, and
// 3 us more at 64 x 1024, 16 heads of 64 (268 MB to zero), where the memset streams a little better.
__global__ void __launch_bounds__(256) attn_bwd_span_kernel(const int* __restrict__ seq_start, int n_tiles, int* __restrict__ nq, int* counter,
                                                            uint4* __restrict__ dq_acc, long long n16) {
    pdl_sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n16; i += (long long)gridDim.x * 256) dq_acc[i] = make_uint4(0, 0, 0, 0);
    const int kv_tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (kv_tile >= n_tiles) return;
    const int kv_last = kv_tile * 128 + 127;
    int n_q = 1;
    for (int t0 = kv_tile + 1; t0 < n_tiles; t0 += 32) {
        const int t = t0 + lane;
        const bool sees = t < n_tiles && seq_start[t * 128] <= kv_last;
        const uint32_t m = __ballot_sync(0xffffffffu, sees);
        const int run = __ffs(~m) - 1;          // leading run of visible tiles (m == all ones: ffs(0) - 1 = -1)
        if (run >= 0) { n_q += run; break; }
        n_q += 32;
    }
    if (lane == 0) nq[kv_tile] = n_q;
}

int make_tmap_heads(CUtensorMap* out, const void* ptr, int elem_bytes, uint64_t hd, uint64_t n_heads, uint64_t outer, uint64_t ld,
                    uint32_t box_inner, uint32_t box_outer);

static void launch_span(const AttnBwdParams& p, cudaStream_t st) {
    const long long n16 = (long long)p.M * p.H * p.hd / 4;                // a head is a multiple of 8 columns
    long long blocks = (n16 + 1023) / 1024;                               // four stores per thread, at most 8 CTAs per SM ...
    if (blocks > 148 * 8) blocks = 148 * 8;
    if (blocks < (p.n_tiles + 7) / 8) blocks = (p.n_tiles + 7) / 8;       // ... and a warp for every kv tile
    launch_pdl(attn_bwd_span_kernel, LaunchCfg(unsigned(blocks), 256, 0, st).traffic(16.0 * n16), p.seq_start, p.n_tiles, p.nq, p.counter,
               reinterpret_cast<uint4*>(p.dq_acc), n16);
}

static int launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tdq, const AttnBwdParams& p, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnBwdCfg::SMEM_BYTES) != cudaSuccess) return -20;
        configured = true;
    }
    const int grid = p.n_items < sm_count() ? p.n_items : sm_count();     // one CTA per SM draws items until none are left
    launch_pdl(attn_bwd_kernel, LaunchCfg(grid, 512, AttnBwdCfg::SMEM_BYTES, st), tq, tdo, tdq, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -30;
}

}  // namespace pb

// dq_acc: fp32 [M, H*HD] scratch (zeroed here); D: fp32 [H, M] scratch, computed here from o and dout unless o is
// null (then the caller has already filled it with [H, d_parts, M] partial sums: one, or two for heads of more than 64 columns).
// Writes all of dqkv.
// rope_table != null: the inverse rotation is applied to dq and dk on the way out (position = row % T).
// tile_scratch: >= ceil(M / 128) + 1 ints of device scratch (query-tile count of every kv tile and the work counter).
extern "C" int pb_attn_bwd_parts(const void* qkv, const void* o, const void* dout, const float* lse2, const int* seq_start,
                                 void* dqkv, float* dq_acc, float* D, int d_parts, const float* rope_table, int T, int M, int H, int KV, int HD,
                                 long long qkv_stride, long long o_stride, long long do_stride, long long dqkv_stride, float scale,
                                 int* tile_scratch, int* status, void* stream) {
    using namespace pb;
    if (HD <= 0 || HD > 128 || HD % 8) return -1;
    if (H % KV) return -1;
    if (!o && d_parts != 1 && (d_parts != 2 || HD <= 64)) return -4;      // the kernel for heads of up to 64 columns reads whole sums
    if ((qkv_stride % 8) || (o_stride % 8) || (do_stride % 8) || (dqkv_stride % 8) ||
        ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dqkv)) & 15))
        return -2;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    CUtensorMap tq, tdo, tdq;
    int rc = make_tmap_heads(&tq, qkv, 2, HD, uint64_t(H + 2 * KV), M, qkv_stride, 64, 128);
    if (rc) return rc;
    rc = make_tmap_heads(&tdo, dout, 2, HD, H, M, do_stride, 64, 128);
    if (rc) return rc;
    rc = make_tmap_heads(&tdq, dq_acc, 4, HD, H, M, uint64_t(H) * HD, 32, 32);
    if (rc) return rc;
    if (o) {   // o == null: the caller already filled D
        const long long rows = (long long)M * H;
        const int lpr = HD <= 16 ? 2 : HD <= 32 ? 4 : HD <= 64 ? 8 : 16;
        const int rows_per_block = 256 / lpr;
        long long blocks = (rows + 4LL * rows_per_block - 1) / (4LL * rows_per_block);
        if (blocks < 1) blocks = 1;
        auto kern = lpr == 2 ? attn_bwd_prep_kernel<2> : lpr == 4 ? attn_bwd_prep_kernel<4> : lpr == 8 ? attn_bwd_prep_kernel<8>
                                                                                               : attn_bwd_prep_kernel<16>;
        launch_pdl(kern, LaunchCfg(unsigned(blocks), 256, 0, st).traffic(4.0 * rows * HD), (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, D, M, H, HD, o_stride,
                   do_stride);
    }
    AttnBwdParams p;
    p.M = M; p.H = H; p.KV = KV; p.hd = HD; p.n_tiles = (M + 127) / 128; p.seq_start = seq_start; p.lse2 = lse2; p.D = D;
    p.dq_acc = dq_acc; p.dqkv = reinterpret_cast<__nv_bfloat16*>(dqkv); p.dqkv_stride = dqkv_stride;
    p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
    p.d_parts = o ? 1 : d_parts; p.rope = rope_table; p.T = T;
    if (tile_scratch == nullptr) return -3;
    p.nq = tile_scratch; p.counter = tile_scratch + p.n_tiles; p.n_items = p.n_tiles * KV;
    launch_span(p, st);
    rc = HD <= 64 ? launch_attn_bwd(tq, tdo, tdq, p, st) : launch_attn_bwd128(tq, tdo, tdq, p, st);
    if (rc) return rc;
    const long long total = (long long)M * H * (HD / 8);
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    launch_pdl(attn_bwd_finish_kernel, LaunchCfg(unsigned(blocks), 256, 0, st).traffic(6.0 * M * H * HD), dq_acc, (__nv_bfloat16*)dqkv, rope_table, M, T, H, HD,
               dqkv_stride);
    return cudaGetLastError() == cudaSuccess ? 0 : -30;
}

// D whole: [H, M]
extern "C" int pb_attn_bwd(const void* qkv, const void* o, const void* dout, const float* lse2, const int* seq_start,
                           void* dqkv, float* dq_acc, float* D, const float* rope_table, int T, int M, int H, int KV, int HD,
                           long long qkv_stride, long long o_stride, long long do_stride, long long dqkv_stride, float scale,
                           int* tile_scratch, int* status, void* stream) {
    return pb_attn_bwd_parts(qkv, o, dout, lse2, seq_start, dqkv, dq_acc, D, 1, rope_table, T, M, H, KV, HD, qkv_stride, o_stride, do_stride,
                             dqkv_stride, scale, tile_scratch, status, stream);
}
