// Bandwidth-bound kernels of the Llama training step for sm_100a: RMSNorm fwd/bwd,
// RoPE, SwiGLU fwd/bwd, embedding gather / scatter-add, softmax cross-entropy with
// in-place logit gradient, fused AdamW, and small reductions (sum of squares).
// All of them move 16-byte vectors, keep fp32 math in registers and use fixed-order
// reductions so results are bit-reproducible run to run.
//
// Reference behaviour being reproduced (paths inside the reference project):
//   RMSNorm      src/zeroband/models/norms.py:79-106 (eager), :116-221 (Triton fwd/bwd)
//   RoPE         src/zeroband/models/llama/model.py:118-144 (interleaved complex pairs)
//   SwiGLU       src/zeroband/models/llama/model.py:340-341
//   CE / z-loss  src/zeroband/loss.py:70-87 (max-z) and :47-66 (lse^2 z-loss of the fused path)
//   AdamW        src/zeroband/optimizers.py:25-30 (torch.optim.AdamW semantics)
#include "common.cuh"
#include "rmsnorm_bwd.cuh"
#include <algorithm>

namespace pb {

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}

// ----------------------------------------------------------------------------
// RMSNorm forward: one warp per row. y = x * rstd * w ; rstd saved (fp32).
// Memory-bound: 4 bytes per element. NCH = N / 256 > 0: the row stays in registers between its sum of squares and its scaling, and all
// of its loads are issued before the first use; the plain loop (NCH = 0, any multiple of 8) has one load in flight per lane and
// reads the row a second time. Measured: 65536 x 1024
// 55.6 -> 47.6 us (5.6 TB/s), 16384 x 2048 29.1 -> 27.0, 8192 x 2048 21.9 -> 20.7.
// ----------------------------------------------------------------------------
// not hoisted out of the row loop: the weights of a wide row would take twice the registers of the row itself
__device__ __forceinline__ uint4 load16_here(const __nv_bfloat16* p) {
    uint4 u;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(p));
    return u;
}
template <int NCH>
__global__ void __launch_bounds__(256, NCH <= 2 ? 5 : NCH <= 4 ? 4 : NCH <= 6 ? 3 : 2) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                                          int M, int N, float eps) {
    pdl_sync();
    const int warps_per_block = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    for (long long row = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < M;
         row += (long long)gridDim.x * warps_per_block) {
        const __nv_bfloat16* xr = x + row * N;
        __nv_bfloat16* yr = y + row * N;
        float ss = 0.f;
        if constexpr (NCH > 0) {
            uint4 u[NCH];
#pragma unroll
            for (int j = 0; j < NCH; ++j) u[j] = *reinterpret_cast<const uint4*>(xr + lane * 8 + j * 256);
#pragma unroll
            for (int j = 0; j < NCH; ++j) {
                float f[8];
                unpack8(u[j], f);
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
            }
            ss = warp_sum(ss);
            const float r = rsqrtf(ss / N + eps);
            if (lane == 0 && rstd) rstd[row] = r;
#pragma unroll
            for (int j = 0; j < NCH; ++j) {
                float f[8], g[8];
                asm volatile("" : "+r"(u[j].x), "+r"(u[j].y), "+r"(u[j].z), "+r"(u[j].w));    // unpack again: packed words are kept, not floats
                unpack8(u[j], f);
                unpack8(load16_here(w + lane * 8 + j * 256), g);
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = f[i] * r * g[i];
                store8(yr + lane * 8 + j * 256, f);
            }
        } else {
            for (int c = lane * 8; c < N; c += 256) {
                float f[8];
                load8(xr + c, f);
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
            }
            ss = warp_sum(ss);
            const float r = rsqrtf(ss / N + eps);
            if (lane == 0 && rstd) rstd[row] = r;
            for (int c = lane * 8; c < N; c += 256) {
                float f[8], g[8];
                load8(xr + c, f);
                load8(w + c, g);
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = f[i] * r * g[i];
                store8(yr + c, f);
            }
        }
    }
}

// ----------------------------------------------------------------------------
// RoPE on interleaved (re, im) pairs, in place, on the q and k slices of a fused
// qkv activation [M, (H + 2*KV) * hd]. Position of row m is m % T.
// table: [>=T, hd/2, 2] fp32 (cos, sin). sign=+1 forward, -1 backward (conjugate).
// ----------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ table, long long M, int T,
                            int n_rot_heads, int hd, int row_stride, float sign) {
    pdl_sync();
    // one thread handles 8 consecutive elements (4 pairs)
    const int vec_per_head = hd / 8;
    const long long total = M * n_rot_heads * vec_per_head;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int v = int(i % vec_per_head);
        const long long t = i / vec_per_head;
        const int h = int(t % n_rot_heads);
        const long long m = t / n_rot_heads;
        const int pos = int(m % T);
        __nv_bfloat16* p = qkv + m * row_stride + h * hd + v * 8;
        float f[8];
        load8(p, f);
        const float4* cs = reinterpret_cast<const float4*>(table + ((long long)pos * (hd / 2) + v * 4) * 2);
        float4 c0 = cs[0], c1 = cs[1];
        const float co[4] = {c0.x, c0.z, c1.x, c1.z};
        const float si[4] = {c0.y * sign, c0.w * sign, c1.y * sign, c1.w * sign};
        float o[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            o[2 * k] = f[2 * k] * co[k] - f[2 * k + 1] * si[k];
            o[2 * k + 1] = f[2 * k] * si[k] + f[2 * k + 1] * co[k];
        }
        store8(p, o);
    }
}

// ----------------------------------------------------------------------------
// SwiGLU. h13 is [M, 2F]: gate = cols [0,F), up = cols [F,2F). act = silu(gate)*up.
// ----------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ h13, __nv_bfloat16* __restrict__ act,
                                  long long M, int F) {
    pdl_sync();
    const int vpr = F / 8;
    const long long total = M * vpr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / vpr;
        const int c = int(i % vpr) * 8;
        float g[8], u[8], o[8];
        load8(h13 + m * 2 * F + c, g);
        load8(h13 + m * 2 * F + F + c, u);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = g[k] / (1.f + __expf(-g[k])) * u[k];
        store8(act + m * F + c, o);
    }
}
// dgate = dact * up * sig*(1 + g*(1-sig)) ; dup = dact * silu(g). Written into dh13 [M,2F]
// (dh13 may alias h13: each thread reads its inputs before writing the same locations).
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* h13, const __nv_bfloat16* __restrict__ dact,
                                  __nv_bfloat16* dh13, long long M, int F) {
    pdl_sync();
    const int vpr = F / 8;
    const long long total = M * vpr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / vpr;
        const int c = int(i % vpr) * 8;
        float g[8], u[8], d[8], dg[8], du[8];
        load8(h13 + m * 2 * F + c, g);
        load8(h13 + m * 2 * F + F + c, u);
        load8(dact + m * F + c, d);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float s = 1.f / (1.f + __expf(-g[k]));
            du[k] = d[k] * g[k] * s;
            dg[k] = d[k] * u[k] * s * (1.f + g[k] * (1.f - s));
        }
        store8(dh13 + m * 2 * F + c, dg);
        store8(dh13 + m * 2 * F + F + c, du);
    }
}

// ----------------------------------------------------------------------------
// Embedding gather and its backward (scatter-add with atomics; fp32 or bf16 grads)
// ----------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const long long* __restrict__ tok, const __nv_bfloat16* __restrict__ E,
                                     __nv_bfloat16* __restrict__ out, long long M, int D) {
    pdl_sync();
    const int vpr = D / 8;
    const long long total = M * vpr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / vpr;
        const int c = int(i % vpr) * 8;
        *reinterpret_cast<uint4*>(out + m * D + c) = *reinterpret_cast<const uint4*>(E + tok[m] * D + c);
    }
}
__global__ void embedding_bwd_kernel(const long long* __restrict__ tok, const __nv_bfloat16* __restrict__ dout,
                                     void* __restrict__ dE, long long M, int D, int grad_fp32) {
    pdl_sync();
    const int vpr = D / 8;
    const long long total = M * vpr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / vpr;
        const int c = int(i % vpr) * 8;
        const long long t = tok[m];
        if (grad_fp32) {
            float f[8];
            load8(dout + m * D + c, f);
            float* g = reinterpret_cast<float*>(dE) + t * D + c;
#pragma unroll
            for (int k = 0; k < 8; ++k) atomicAdd(g + k, f[k]);
        } else {
            uint4 u = *reinterpret_cast<const uint4*>(dout + m * D + c);
            __nv_bfloat162* g = reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(dE) + t * D + c);
            atomicAdd(g + 0, *reinterpret_cast<__nv_bfloat162*>(&u.x));
            atomicAdd(g + 1, *reinterpret_cast<__nv_bfloat162*>(&u.y));
            atomicAdd(g + 2, *reinterpret_cast<__nv_bfloat162*>(&u.z));
            atomicAdd(g + 3, *reinterpret_cast<__nv_bfloat162*>(&u.w));
        }
    }
}

// ----------------------------------------------------------------------------
// Cross-entropy over bf16 logits [rows, V] (row pitch ld) with in-place gradient.
// One CTA per row; online max/sum in pass 1, gradient written in pass 2 (row is
// L2-resident). Per-row outputs: loss_i (0 for ignored rows) and z_i.
//   z_mode 0: none; 1: max-z  (z_i = max^2);  2: lse^2 (z_i = lse^2)
//   dlogits = scale * [softmax - onehot] + dz, scale = *inv_count * grad_scale
// Bound: 4 bytes of memory traffic and two exponentials per logit (16 a clock and SM). With one compare per logit for the
// maximum, the label and the argmax each, the issue slots were the limit; now a vector of eight has one maximum, subtraction
// and scaling run on packed fp32 pairs, the label is compared once per vector and the argmax exists in the max-z variant only.
// The rows that are resident at once must fit L2 together, or pass 2 reads memory again. Measured: 32768 x 32000
// 993 -> 709 us (5.9 TB/s), 16384 x 32000 504 -> 361, 8192 x 128256 1061 -> 865, 8192 x 1024 37 -> 29.
// ----------------------------------------------------------------------------
// exp(f[i] + shift) of eight values; *coef unless null
__device__ __forceinline__ void exp8(float (&f)[8], float shift, const float* coef) {
    const unsigned long long sh = f32x2_pack(shift, shift), l2e = f32x2_pack(1.4426950408889634f, 1.4426950408889634f);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float x, y;
        f32x2_unpack(f32x2_mul(f32x2_add(f32x2_pack(f[i], f[i + 1]), sh), l2e), x, y);
        f[i] = ex2_approx(x);
        f[i + 1] = ex2_approx(y);
        if (coef) f32x2_unpack(f32x2_mul(f32x2_pack(f[i], f[i + 1]), f32x2_pack(*coef, *coef)), f[i], f[i + 1]);
    }
}

template <int THREADS, bool ARG>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS)
cross_entropy_kernel(__nv_bfloat16* logits, const long long* __restrict__ labels, float* __restrict__ loss_rows,
                     float* __restrict__ z_rows, const float* __restrict__ inv_count, float grad_scale, int V, long long ld,
                     int ignore_index, int z_mode, float z_weight, int write_grad) {
    constexpr int WARPS = THREADS / 32, STEP = THREADS * 8;
    pdl_sync();
    __shared__ float s_m[WARPS], s_s[WARPS];
    __shared__ int s_arg[WARPS];
    const long long row = blockIdx.x;
    __nv_bfloat16* lr = logits + row * ld;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long label = labels[row];
    const bool ignored = (label == ignore_index);
    float mx = -INFINITY;
    unsigned long long sum2[2] = {0ull, 0ull};
    int arg = 0;
    const int V8 = V & ~7;
    auto take = [&](const uint4& u, int c) {
        float f[8];
        unpack8(u, f);
        const float cm = max3(max3(f[0], f[1], f[2]), max3(f[3], f[4], f[5]), fmaxf(f[6], f[7]));
        if (cm > mx) {
            const float a = __expf(mx - cm);
            sum2[0] = f32x2_mul(sum2[0], f32x2_pack(a, a));
            sum2[1] = f32x2_mul(sum2[1], f32x2_pack(a, a));
            mx = cm;
            if (ARG) {
#pragma unroll
                for (int k = 7; k >= 0; --k)
                    if (f[k] == cm) arg = c + k;
            }
        }
        exp8(f, -mx, nullptr);
#pragma unroll
        for (int k = 0; k < 8; k += 2) sum2[(k >> 1) & 1] = f32x2_add(sum2[(k >> 1) & 1], f32x2_pack(f[k], f[k + 1]));
    };
    int c = tid * 8;
    for (; c + STEP < V8; c += 2 * STEP) {        // two loads in flight per thread
        const uint4 u0 = *reinterpret_cast<const uint4*>(lr + c), u1 = *reinterpret_cast<const uint4*>(lr + c + STEP);
        take(u0, c);
        take(u1, c + STEP);
    }
    if (c < V8) take(*reinterpret_cast<const uint4*>(lr + c), c);
    float sm;
    {
        float x, y;
        f32x2_unpack(f32x2_add(sum2[0], sum2[1]), x, y);
        sm = x + y;
    }
    for (int t = V8 + tid; t < V; t += THREADS) {
        const float f = __bfloat162float(lr[t]);
        if (f > mx) { sm *= __expf(mx - f); mx = f; arg = t; }
        sm += __expf(f - mx);
    }
    // warp then CTA reduction of (max, sum, argmax); ties resolve to the lowest index
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, mx, o);
        const float os = __shfl_xor_sync(0xffffffffu, sm, o);
        const float nm = fmaxf(mx, om);
        sm = (mx == -INFINITY ? 0.f : sm * __expf(mx - nm)) + (om == -INFINITY ? 0.f : os * __expf(om - nm));
        if (ARG) {
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (om > mx || (om == mx && oa < arg)) arg = oa;
        }
        mx = nm;
    }
    if (lane == 0) { s_m[warp] = mx; s_s[warp] = sm; if (ARG) s_arg[warp] = arg; }
    __syncthreads();
    mx = s_m[0]; sm = s_s[0];
    if (ARG) arg = s_arg[0];
    for (int w2 = 1; w2 < WARPS; ++w2) {
        const float om = s_m[w2], os = s_s[w2];
        const float nm = fmaxf(mx, om);
        sm = (mx == -INFINITY ? 0.f : sm * __expf(mx - nm)) + (om == -INFINITY ? 0.f : os * __expf(om - nm));
        if (ARG) {
            const int oa = s_arg[w2];
            if (om > mx || (om == mx && oa < arg)) arg = oa;
        }
        mx = nm;
    }
    const float lse = mx + __logf(sm);
    if (tid == 0) {
        float li = 0.f, zi = 0.f;
        if (!ignored) {
            li = lse - __bfloat162float(lr[label]);
            zi = z_mode == 1 ? mx * mx : (z_mode == 2 ? lse * lse : 0.f);
        }
        loss_rows[row] = li;
        if (z_rows) z_rows[row] = zi;
    }
    if (!write_grad) return;
    __syncthreads();  // label logit was read above before anyone overwrites it
    const float scale = ignored ? 0.f : (*inv_count) * grad_scale;
    // d(lse^2 * zw)/dlogit = 2 zw lse softmax ;  d(max^2 * zw)/dlogit = 2 zw max at argmax
    const float soft_coef = scale * (1.f + (z_mode == 2 ? 2.f * z_weight * lse : 0.f));
    const float max_coef = (z_mode == 1) ? scale * 2.f * z_weight * mx : 0.f;
    const int lab = ignored ? -8 : int(label);
    auto give = [&](const uint4& u, int at) {
        float f[8];
        unpack8(u, f);
        exp8(f, -lse, &soft_coef);
        if (unsigned(lab - at) < 8u) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (at + k == lab) f[k] -= scale;
        }
        if (ARG && unsigned(arg - at) < 8u) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (at + k == arg) f[k] += max_coef;
        }
        store8(lr + at, f);
    };
    c = tid * 8;
    for (; c + STEP < V8; c += 2 * STEP) {
        const uint4 u0 = *reinterpret_cast<const uint4*>(lr + c), u1 = *reinterpret_cast<const uint4*>(lr + c + STEP);
        give(u0, c);
        give(u1, c + STEP);
    }
    if (c < V8) give(*reinterpret_cast<const uint4*>(lr + c), c);
    for (int t = V8 + tid; t < V; t += THREADS) {
        float g = soft_coef * __expf(__bfloat162float(lr[t]) - lse);
        if (t == lab) g -= scale;
        if (ARG && t == arg) g += max_coef;
        lr[t] = __float2bfloat16(g);
    }
}

// count of labels != ignore_index -> inv_count[0] = 1 / max(count, 1), inv_count[1] = count. Counts are integers, so the order of the
// CTAs does not matter. With one CTA 65536 labels took 12.8 us (64 dependent rounds of loads); several CTAs need `counter`
// (two zero-initialised words of the caller that are zero again afterwards).
__global__ void __launch_bounds__(1024) count_valid_kernel(const long long* __restrict__ labels, long long n, int ignore_index,
                                                          float* __restrict__ inv_count, unsigned* counter) {
    pdl_sync();
    __shared__ unsigned s[32];
    unsigned c = 0;
    for (long long i = (long long)blockIdx.x * 1024 + threadIdx.x; i < n; i += (long long)gridDim.x * 1024) c += (labels[i] != ignore_index);
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int i = 0; i < 32; ++i) t += s[i];
        if (gridDim.x > 1) {
            atomicAdd(counter + 1, t);
            __threadfence();
            if (atomicAdd(counter, 1u) != gridDim.x - 1) return;
            __threadfence();
            t = atomicExch(counter + 1, 0u);
            *counter = 0u;
        }
        inv_count[0] = 1.f / float(t > 0 ? t : 1);
        inv_count[1] = float(t);
    }
}

// out[0] = inv[0] * sum(loss_rows), out[1] = inv[0] * z_weight * sum(z_rows) (0 without z_rows); acc[0..1] (+)= acc_scale * out[0..1].
// One launch for both means and the accumulation over micro-batches. Per-CTA partials are added by the last CTA in a
// fixed tree, so the sums are bit-reproducible. partial: 2 * gridDim floats; counter: one zeroed word of the caller.
__global__ void __launch_bounds__(256) loss_sums_kernel(const float* __restrict__ loss_rows, const float* __restrict__ z_rows, int n,
                                                        const float* __restrict__ inv, float z_weight, float* out, float* acc,
                                                        float acc_scale, int acc_first, float* partial, unsigned* counter) {
    pdl_sync();
    __shared__ float red[2][8];
    __shared__ bool last;
    const int tid = threadIdx.x;
    auto block_sum = [&](float& a, float& b) {
        a = warp_sum(a);
        b = warp_sum(b);
        if ((tid & 31) == 0) { red[0][tid >> 5] = a; red[1][tid >> 5] = b; }
        __syncthreads();
        a = b = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) { a += red[0][i]; b += red[1][i]; }
        __syncthreads();
    };
    float a = 0.f, b = 0.f;
    for (int i = blockIdx.x * 256 + tid; i < n; i += gridDim.x * 256) {
        a += loss_rows[i];
        if (z_rows) b += z_rows[i];
    }
    block_sum(a, b);
    if (gridDim.x > 1) {
        if (tid == 0) {
            partial[2 * blockIdx.x] = a;
            partial[2 * blockIdx.x + 1] = b;
            __threadfence();
            last = atomicAdd(counter, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        a = b = 0.f;
        for (int i = tid; i < int(gridDim.x); i += 256) {
            a += __ldcg(partial + 2 * i);
            b += __ldcg(partial + 2 * i + 1);
        }
        block_sum(a, b);
        if (tid == 0) *counter = 0u;
    }
    if (tid == 0) {
        const float l = a * inv[0], z = b * inv[0] * z_weight;
        out[0] = l;
        out[1] = z;
        if (acc) {
            acc[0] = (acc_first ? 0.f : acc[0]) + l * acc_scale;
            acc[1] = (acc_first ? 0.f : acc[1]) + z * acc_scale;
        }
    }
}

// Inputs of a graphed step -> the buffers that the graph reads, and the step's scalars: hyper = {lr, 1 - beta1^t, sqrt(1 - beta2^t)}.
__global__ void __launch_bounds__(256) stage_step_kernel(const long long* __restrict__ tok, const long long* __restrict__ lab,
                                                         const int* __restrict__ seq_start, int n, long long* __restrict__ tok_dst,
                                                         long long* __restrict__ lab_dst, int* __restrict__ seq_dst, float lr, float bc1,
                                                         float bc2, float* __restrict__ hyper) {
    pdl_sync();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) {
        tok_dst[i] = tok[i];
        lab_dst[i] = lab[i];
        if (seq_start) seq_dst[i] = seq_start[i];
    }
    if (i == 0) { hyper[0] = lr; hyper[1] = bc1; hyper[2] = bc2; }
}

// what the host reads after a step: {mean loss, z loss, gradient norm, status word}
__global__ void step_report_kernel(const float* __restrict__ total, const float* __restrict__ norm_sq, const int* __restrict__ status,
                                   float* __restrict__ report) {
    pdl_sync();
    report[0] = total[0];
    report[1] = total[1];
    report[2] = sqrtf(*norm_sq);
    report[3] = float(*status);
}

// out[0] (+)= scale * sum(x[0:n]) — two-stage fixed-order sum of fp32 values
__global__ void sum_stage1_kernel(const float* __restrict__ x, long long n, float* __restrict__ partial) {
    pdl_sync();
    __shared__ float s[32];
    float a = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        a += x[i];
    a = warp_sum(a);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < (blockDim.x >> 5); ++i) t += s[i];
        partial[blockIdx.x] = t;
    }
}
__global__ void sum_stage2_kernel(const float* __restrict__ partial, int nb, const float* __restrict__ scale_ptr,
                                  float scale, float* __restrict__ out, int accumulate) {
    pdl_sync();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < nb; ++i) t += partial[i];
        t *= scale * (scale_ptr ? *scale_ptr : 1.f);
        out[0] = accumulate ? out[0] + t : t;
    }
}

// ----------------------------------------------------------------------------
// sum of squares of a bf16 / fp32 buffer -> per-CTA partials (fixed order)
// ----------------------------------------------------------------------------
template <typename T>
__global__ void sumsq_kernel(const T* __restrict__ x, long long n, float* __restrict__ partial) {
    pdl_sync();
    __shared__ float s[32];
    float a = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float f = float(x[i]);
        a += f * f;
    }
    a = warp_sum(a);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < (blockDim.x >> 5); ++i) t += s[i];
        partial[blockIdx.x] = t;
    }
}

// ----------------------------------------------------------------------------
// AdamW on a flat fp32 shard with bf16 or fp32 gradients; refreshes the bf16 compute copy.
//   clip: optional device pointer to the total grad norm; grads are scaled by
//         min(1, max_norm / (norm + 1e-6)) as torch.nn.utils.clip_grad_norm_ does.
// ----------------------------------------------------------------------------
template <typename G>
__global__ void adamw_kernel(float* __restrict__ p, const G* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                             __nv_bfloat16* __restrict__ p_bf16, long long n, float lr, float beta1, float beta2,
                             float eps, float wd, float bc1, float bc2, const float* __restrict__ gnorm,
                             float max_norm, float gscale) {
    pdl_sync();
    float clip = gscale;
    if (gnorm) {
        const float c = max_norm / (*gnorm + 1e-6f);
        clip *= c < 1.f ? c : 1.f;
    }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = float(g[i]) * clip;
        float pi = p[i];
        pi *= (1.f - lr * wd);
        const float mi = beta1 * m[i] + (1.f - beta1) * gi;
        const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float denom = sqrtf(vi) / bc2 + eps;   // bc2 = sqrt(1 - beta2^t)
        pi -= (lr / bc1) * (mi / denom);
        p[i] = pi;
        if (p_bf16) p_bf16[i] = __float2bfloat16(pi);
    }
}

__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    pdl_sync();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16(src[i]);
}

// residual add: out = a + b (bf16)
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ out, long long n8) {
    pdl_sync();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
        float x[8], y[8];
        load8(a + i * 8, x);
        load8(b + i * 8, y);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] += y[k];
        store8(out + i * 8, x);
    }
}

static inline int grid_for(long long work_items, int block, int max_blocks = 148 * 8) {
    long long b = (work_items + block - 1) / block;
    if (b < 1) b = 1;
    return int(b < max_blocks ? b : max_blocks);
}

}  // namespace pb

using namespace pb;
#define ST(s) reinterpret_cast<cudaStream_t>(s)
#define CHECK_LAUNCH() (cudaGetLastError() == cudaSuccess ? 0 : -30)

extern "C" int pb_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int M, int N, float eps, void* stream) {
    if (N % 8) return -1;
    auto launch = [&](auto kern) {
        launch_pdl(kern, LaunchCfg(grid_for(M, 8), 256, 0, ST(stream)).traffic(4.0 * M * N), (const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                   (__nv_bfloat16*)y, rstd, M, N, eps);
    };
    switch (N % 256 ? 0 : N / 256) {       // widths of up to 3072 in whole 256-column chunks (4096 would spill)
        case 1: launch(rmsnorm_fwd_kernel<1>); break;
        case 2: launch(rmsnorm_fwd_kernel<2>); break;
        case 3: launch(rmsnorm_fwd_kernel<3>); break;
        case 4: launch(rmsnorm_fwd_kernel<4>); break;
        case 6: launch(rmsnorm_fwd_kernel<6>); break;
        case 8: launch(rmsnorm_fwd_kernel<8>); break;
        case 12: launch(rmsnorm_fwd_kernel<12>); break;
        default: launch(rmsnorm_fwd_kernel<0>);
    }
    return CHECK_LAUNCH();
}

// number of CTAs (= rows of the fp32 partial buffer [ctas, N]) the backward uses at most
extern "C" int pb_rmsnorm_bwd_ctas() { return 148 * 2; }

static int rmsnorm_bwd_used_ctas(int M, int N) {
    const int rows_per_cta = N <= 1024 ? 8 : N <= 2048 ? 4 : 2;      // of one iteration; a CTA without rows would only add a zero partial
    return std::max(1, std::min(pb_rmsnorm_bwd_ctas(), (M + rows_per_cta - 1) / rows_per_cta));
}

// The second half of pb_rmsnorm_bwd by itself: the weight gradient from the partial sums that pb_rmsnorm_bwd left for M rows of N
// columns when it was given no dw.
extern "C" int pb_rmsnorm_bwd_dw(const float* dw_partial, void* dw, int dw_fp32, int dw_accumulate, int M, int N, void* stream) {
    launch_pdl(colsum_partials_kernel, LaunchCfg((N + 31) / 32, 32 * COLSUM_GROUPS, 0, ST(stream)), dw_partial, dw, rmsnorm_bwd_used_ctas(M, N), N,
               dw_fp32, dw_accumulate);
    return CHECK_LAUNCH();
}

extern "C" int pb_rmsnorm_bwd(const void* x, const void* w, const float* rstd, const void* dy, const void* dres,
                              void* dx, float* dw_partial, void* dw, int dw_fp32, int dw_accumulate, int M, int N,
                              void* stream) {
    if (N % 256 || N > 4096) return -1;
    const int ctas = rmsnorm_bwd_used_ctas(M, N);
    auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w; auto DY = (const __nv_bfloat16*)dy;
    auto DR = (const __nv_bfloat16*)dres; auto DX = (__nv_bfloat16*)dx;
    // rows wider than 1024 are shared by two or four warps (at most four 256-column chunks per warp)
#define RB(NCH, WPR) case NCH: launch_pdl(rmsnorm_bwd_kernel<NCH, WPR>, LaunchCfg(ctas, 256, 0, ST(stream)).traffic(8.0 * M * N), X, W, rstd, DY, DR, DX, dw_partial, M); break;
    switch (N / 256) {
        RB(1, 1) RB(2, 1) RB(3, 1) RB(4, 1) RB(6, 2) RB(8, 2) RB(12, 4) RB(16, 4)
        default: return -1;
    }
#undef RB
    if (cudaGetLastError() != cudaSuccess) return -30;
    return dw ? pb_rmsnorm_bwd_dw(dw_partial, dw, dw_fp32, dw_accumulate, M, N, stream) : 0;
}

extern "C" int pb_rope(void* qkv, const float* table, long long M, int T, int n_rot_heads, int hd, int row_stride,
                       int backward, void* stream) {
    if (hd % 8 || row_stride % 8) return -1;
    launch_pdl(rope_kernel, LaunchCfg(grid_for(M * n_rot_heads * (hd / 8), 256), 256, 0, ST(stream)).traffic(4.0 * M * n_rot_heads * hd), 
        (__nv_bfloat16*)qkv, table, M, T, n_rot_heads, hd, row_stride, backward ? -1.f : 1.f);
    return CHECK_LAUNCH();
}

extern "C" int pb_swiglu_fwd(const void* h13, void* act, long long M, int F, void* stream) {
    if (F % 8) return -1;
    launch_pdl(swiglu_fwd_kernel, LaunchCfg(grid_for(M * (F / 8), 256), 256, 0, ST(stream)).traffic(6.0 * M * F), (const __nv_bfloat16*)h13, (__nv_bfloat16*)act, M, F);
    return CHECK_LAUNCH();
}
extern "C" int pb_swiglu_bwd(const void* h13, const void* dact, void* dh13, long long M, int F, void* stream) {
    if (F % 8) return -1;
    launch_pdl(swiglu_bwd_kernel, LaunchCfg(grid_for(M * (F / 8), 256), 256, 0, ST(stream)).traffic(10.0 * M * F), (const __nv_bfloat16*)h13, (const __nv_bfloat16*)dact,
                                                                          (__nv_bfloat16*)dh13, M, F);
    return CHECK_LAUNCH();
}

extern "C" int pb_embedding_fwd(const long long* tok, const void* E, void* out, long long M, int D, void* stream) {
    if (D % 8) return -1;
    launch_pdl(embedding_fwd_kernel, LaunchCfg(grid_for(M * (D / 8), 256), 256, 0, ST(stream)).traffic(4.0 * M * D), tok, (const __nv_bfloat16*)E, (__nv_bfloat16*)out, M, D);
    return CHECK_LAUNCH();
}
extern "C" int pb_embedding_bwd(const long long* tok, const void* dout, void* dE, long long M, int D, int grad_fp32, void* stream) {
    if (D % 8) return -1;
    launch_pdl(embedding_bwd_kernel, LaunchCfg(grid_for(M * (D / 8), 256), 256, 0, ST(stream)).traffic(6.0 * M * D), tok, (const __nv_bfloat16*)dout, dE, M, D, grad_fp32);
    return CHECK_LAUNCH();
}

// counter: two zeroed words, or null (then one CTA counts)
extern "C" int pb_count_valid(const long long* labels, long long n, int ignore_index, float* inv_count, unsigned* counter, void* stream) {
    const int grid = counter ? grid_for(n, 2048, 148) : 1;
    launch_pdl(count_valid_kernel, LaunchCfg(grid, 1024, 0, ST(stream)), labels, n, ignore_index, inv_count, counter);
    return CHECK_LAUNCH();
}

// partial: 2 * 148 floats; counter: one zeroed word
extern "C" int pb_loss_sums(const float* loss_rows, const float* z_rows, int n, const float* inv, float z_weight, float* out, float* acc,
                            float acc_scale, int acc_first, float* partial, unsigned* counter, void* stream) {
    launch_pdl(loss_sums_kernel, LaunchCfg(grid_for(n, 1024, 148), 256, 0, ST(stream)), loss_rows, z_rows, n, inv, z_weight, out, acc, acc_scale,
               acc_first, partial, counter);
    return CHECK_LAUNCH();
}

extern "C" int pb_stage_step(const long long* tok, const long long* lab, const int* seq_start, int n, long long* tok_dst, long long* lab_dst,
                             int* seq_dst, float lr, float beta1, float beta2, int step, float* hyper, void* stream) {
    if (n <= 0) return -1;
    const float bc1 = 1.f - powf(beta1, float(step));
    const float bc2 = sqrtf(1.f - powf(beta2, float(step)));
    launch_pdl(stage_step_kernel, LaunchCfg((n + 255) / 256, 256, 0, ST(stream)), tok, lab, seq_start, n, tok_dst, lab_dst, seq_dst, lr, bc1,
               bc2, hyper);
    return CHECK_LAUNCH();
}

extern "C" int pb_step_report(const float* total, const float* norm_sq, const int* status, float* report, void* stream) {
    launch_pdl(step_report_kernel, LaunchCfg(1, 1, 0, ST(stream)), total, norm_sq, status, report);
    return CHECK_LAUNCH();
}

extern "C" int pb_cross_entropy(void* logits, const long long* labels, float* loss_rows, float* z_rows,
                                const float* inv_count, float grad_scale, long long rows, int V, long long ld,
                                int ignore_index, int z_mode, float z_weight, int write_grad, void* stream) {
    if (rows <= 0) return 0;
    if (ld % 8) return -1;
    // 1536 threads per SM: six rows of 256 threads, so that one row's exponentials overlap another's loads. 148 x 6 rows of up to 48 K
    // logits stay below 90 MB of the 126 MB L2; longer rows get three and then two wider CTAs per SM.
    auto launch = [&](auto kern, int threads) {
        launch_pdl(kern, LaunchCfg((unsigned)rows, threads, 0, ST(stream)).traffic(4.0 * rows * V), (__nv_bfloat16*)logits, labels, loss_rows,
                   z_rows, inv_count, grad_scale, V, ld, ignore_index, z_mode, z_weight, write_grad);
    };
    if (V <= 49152) z_mode == 1 ? launch(cross_entropy_kernel<256, true>, 256) : launch(cross_entropy_kernel<256, false>, 256);
    else if (V <= 98304) z_mode == 1 ? launch(cross_entropy_kernel<512, true>, 512) : launch(cross_entropy_kernel<512, false>, 512);
    else z_mode == 1 ? launch(cross_entropy_kernel<768, true>, 768) : launch(cross_entropy_kernel<768, false>, 768);
    return CHECK_LAUNCH();
}

// out (+)= scale * (*scale_ptr) * sum(x) ; scratch: >= 1024 floats
extern "C" int pb_sum_f32(const float* x, long long n, float* scratch, const float* scale_ptr, float scale, float* out,
                          int accumulate, void* stream) {
    const int nb = grid_for(n, 256, 1024);
    launch_pdl(sum_stage1_kernel, LaunchCfg(nb, 256, 0, ST(stream)), x, n, scratch);
    launch_pdl(sum_stage2_kernel, LaunchCfg(1, 32, 0, ST(stream)), scratch, nb, scale_ptr, scale, out, accumulate);
    return CHECK_LAUNCH();
}

// out (+)= sum(x^2) ; scratch >= 1024 floats
extern "C" int pb_sumsq(const void* x, long long n, int is_fp32, float* scratch, float* out, int accumulate, void* stream) {
    const int nb = grid_for(n, 256, 1024);
    if (is_fp32) launch_pdl(sumsq_kernel<float>, LaunchCfg(nb, 256, 0, ST(stream)).traffic(4.0 * n), (const float*)x, n, scratch);
    else launch_pdl(sumsq_kernel<__nv_bfloat16>, LaunchCfg(nb, 256, 0, ST(stream)).traffic(2.0 * n), (const __nv_bfloat16*)x, n, scratch);
    launch_pdl(sum_stage2_kernel, LaunchCfg(1, 32, 0, ST(stream)), scratch, nb, nullptr, 1.f, out, accumulate);
    return CHECK_LAUNCH();
}

extern "C" int pb_adamw(float* p, const void* g, int g_fp32, float* m, float* v, void* p_bf16, long long n, float lr,
                        float beta1, float beta2, float eps, float wd, int step, const float* gnorm, float max_norm,
                        float gscale, void* stream) {
    if (n <= 0) return 0;
    const float bc1 = 1.f - powf(beta1, float(step));
    const float bc2 = sqrtf(1.f - powf(beta2, float(step)));
    const int nb = grid_for(n, 256, 148 * 16);
    if (g_fp32)
        launch_pdl(adamw_kernel<float>, LaunchCfg(nb, 256, 0, ST(stream)).traffic(28.0 * n), p, (const float*)g, m, v, (__nv_bfloat16*)p_bf16, n, lr, beta1, beta2, eps,
                                                         wd, bc1, bc2, gnorm, max_norm, gscale);
    else
        launch_pdl(adamw_kernel<__nv_bfloat16>, LaunchCfg(nb, 256, 0, ST(stream)).traffic(28.0 * n), p, (const __nv_bfloat16*)g, m, v, (__nv_bfloat16*)p_bf16, n, lr,
                                                                 beta1, beta2, eps, wd, bc1, bc2, gnorm, max_norm, gscale);
    return CHECK_LAUNCH();
}

extern "C" int pb_cast_f32_bf16(const float* src, void* dst, long long n, void* stream) {
    if (n <= 0) return 0;
    launch_pdl(cast_f32_to_bf16_kernel, LaunchCfg(grid_for(n, 256, 148 * 16), 256, 0, ST(stream)).traffic(6.0 * n), src, (__nv_bfloat16*)dst, n);
    return CHECK_LAUNCH();
}

extern "C" int pb_add_bf16(const void* a, const void* b, void* out, long long n, void* stream) {
    if (n % 8) return -1;
    launch_pdl(add_bf16_kernel, LaunchCfg(grid_for(n / 8, 256), 256, 0, ST(stream)).traffic(6.0 * n), (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, (__nv_bfloat16*)out, n / 8);
    return CHECK_LAUNCH();
}

// out[r, c] = sum_s ws[s][r][c] (+ res[r, c]); ws is fp32 [slices][M][N] (N % 4 == 0), out / res are bf16 or fp32
template <bool OUT_FP32>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ ws, int slices, long long M, int N, const void* res,
                                                            long long ld_res, void* out, long long ld_out) {
    pdl_sync();
    const int vpr = N / 4;
    const long long total = M * vpr;
    const long long slice_stride = M * (long long)N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / vpr;
        const int c = int(i % vpr) * 4;
        float4 acc = *reinterpret_cast<const float4*>(ws + r * N + c);
        for (int s = 1; s < slices; ++s) {
            const float4 v = *reinterpret_cast<const float4*>(ws + s * slice_stride + r * N + c);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        if (OUT_FP32) {
            if (res) {
                const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(res) + r * ld_res + c);
                acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
            }
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + r * ld_out + c) = acc;
        } else {
            if (res) {
                const uint2 v = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(res) + r * ld_res + c);
                const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y);
                acc.x += a.x; acc.y += a.y; acc.z += b.x; acc.w += b.y;
            }
            uint2 o;
            o.x = pack_bf16x2(acc.x, acc.y);
            o.y = pack_bf16x2(acc.z, acc.w);
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + r * ld_out + c) = o;
        }
    }
}

// The same sum of partials whose rows belong to up to four outputs of their own (contiguous fp32, rows[p] rows each, one below the
// other in the partials): the weight gradients of stacked projections out of one GEMM.
struct ReduceParts {
    float* out[4];
    int row0[5];
};
__global__ void __launch_bounds__(256) splitk_reduce_parts_kernel(const float* __restrict__ ws, int slices, long long M, int N, const ReduceParts parts) {
    pdl_sync();
    const int vpr = N / 4;
    const long long total = M * vpr, slice_stride = M * (long long)N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int r = int(i / vpr);
        float4 acc = *reinterpret_cast<const float4*>(ws + 4 * i);
        for (int s = 1; s < slices; ++s) {
            const float4 v = *reinterpret_cast<const float4*>(ws + s * slice_stride + 4 * i);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        int p = 0;
        while (r >= parts.row0[p + 1]) ++p;
        *reinterpret_cast<float4*>(parts.out[p] + 4 * (i - (long long)parts.row0[p] * vpr)) = acc;
    }
}

extern "C" int pb_splitk_reduce_parts(const float* ws, int slices, int N, int n_parts, const int* rows, void* const* outs, void* stream) {
    if (n_parts < 1 || n_parts > 4 || N % 4 || reinterpret_cast<uintptr_t>(ws) % 16) return -1;
    ReduceParts parts{};
    for (int p = 0; p < n_parts; ++p) {
        if (rows[p] <= 0 || reinterpret_cast<uintptr_t>(outs[p]) % 16) return -1;
        parts.out[p] = reinterpret_cast<float*>(outs[p]);
        parts.row0[p + 1] = parts.row0[p] + rows[p];
    }
    const long long M = parts.row0[n_parts];
    launch_pdl(splitk_reduce_parts_kernel, LaunchCfg(grid_for(M * (N / 4), 256), 256, 0, ST(stream)).traffic(4.0 * slices * M * N), ws, slices, M, N, parts);
    return CHECK_LAUNCH();
}

extern "C" int pb_splitk_reduce(const float* ws, int slices, long long M, int N, const void* res, long long ld_res, void* out,
                                long long ld_out, int out_fp32, void* stream) {
    // whole vectors of four elements: 16 bytes of fp32, 8 of bf16
    const uintptr_t vec = out_fp32 ? 16 : 8;
    if (N % 4 || ld_out % 4 || (res && ld_res % 4) || (reinterpret_cast<uintptr_t>(ws) % 16) || (reinterpret_cast<uintptr_t>(out) % vec) ||
        (reinterpret_cast<uintptr_t>(res) % vec))
        return -1;
    const unsigned grid = grid_for(M * (N / 4), 256);
    if (out_fp32) launch_pdl(splitk_reduce_kernel<true>, LaunchCfg(grid, 256, 0, ST(stream)).traffic(4.0 * slices * M * N), ws, slices, M, N, res, ld_res, out, ld_out);
    else launch_pdl(splitk_reduce_kernel<false>, LaunchCfg(grid, 256, 0, ST(stream)).traffic(4.0 * slices * M * N), ws, slices, M, N, res, ld_res, out, ld_out);
    return CHECK_LAUNCH();
}
