// Small MoE-layer kernels around the expert GEMVs: the router (softmax top-k on the device), SwiGLU, the weighted
// combine of the expert outputs, and the routing sort that feeds the batched (prefill) kernel.
#include "decode.cuh"
#include "launch.h"

namespace b16 {
namespace {

using namespace dev;

// ---------------------------------------------------------------- router: softmax + top-k, one warp per token

// The k largest logits of a token (ties: lowest expert index), weights exp(z_i - max) renormalised over the selected
// ones, which equals softmax followed by renormalisation. Lane l holds experts l, l+32, ...; up to 1024 experts.
constexpr int TOPK_MAX_PER_LANE = 32;

template <int PER> // experts per lane: the register array and every scan are this long
__global__ void __launch_bounds__(32) k_topk(const float * __restrict__ logits, int n_experts, int k, int32_t * __restrict__ ids,
                                             float * __restrict__ weights) {
    grid_dependency_wait(); // the logits come from an earlier kernel
    const int t = blockIdx.x, lane = threadIdx.x;
    const float * z = logits + (int64_t) t * n_experts;
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = i * 32 + lane;
        v[i] = ld_act_f32(z + min(e, n_experts - 1)); // all in flight together: no branch around a load
    }
#pragma unroll
    for (int i = 0; i < PER; i++) {
        if (i * 32 + lane >= n_experts) { v[i] = -INFINITY; }
    }
    float zmax = 0.f, denom = 0.f;
    for (int s = 0; s < k; s++) {
        // lane-local best (lowest index on ties: strict > while scanning upward)
        float best = -INFINITY;
        int bi = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            if (v[i] > best) { best = v[i]; bi = i * 32 + lane; }
        }
        // warp arg-max with the same tie rule
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float ob = __shfl_xor_sync(FULL, best, o);
            const int oi = __shfl_xor_sync(FULL, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (s == 0) { zmax = best; }
        const float pw = __expf(best - zmax);
        denom += pw;
        if (lane == 0) {
            ids[(int64_t) t * k + s] = bi;
            weights[(int64_t) t * k + s] = pw;
        }
        if ((bi & 31) == lane) { // retire the winner
#pragma unroll
            for (int i = 0; i < PER; i++) {
                if (i == (bi >> 5)) { v[i] = -INFINITY; }
            }
        }
    }
    __syncwarp();
    if (lane < k) { weights[(int64_t) t * k + lane] = __fdividef(weights[(int64_t) t * k + lane], denom); }
}

// ---------------------------------------------------------------- elementwise

__global__ void k_swiglu(const float * __restrict__ g, const float * __restrict__ u, float * __restrict__ y, int64_t n) {
    grid_dependency_wait();
    for (int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
        y[i] = silu_f(ld_act_f32(g + i)) * ld_act_f32(u + i);
    }
}

// y[t, i] = sum over slots k, in slot order, of w[t, k] * ys[t, k, i]
__global__ void k_combine(const float * __restrict__ ys, const char * __restrict__ w, bool w_bf16, char * __restrict__ y, bool y_bf16,
                          int n_used, int64_t n) {
    const int t = blockIdx.y;
    const OutVec out = {y + (int64_t) t * n * (y_bf16 ? 2 : 4), y_bf16};
    for (int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
        float acc = 0.f;
        for (int k = 0; k < n_used; k++) {
            const int64_t s = (int64_t) t * n_used + k;
            const float wk = w_bf16 ? to_f32(((const __nv_bfloat16 *) w)[s]) : ((const float *) w)[s];
            acc = fmaf(wk, ys[s * n + i], acc);
        }
        out.put(i, acc);
    }
}

// The same for rows of whole 16-byte groups, four columns to a thread, the loads of eight slots in flight together (slots beyond a
// multiple of eight one by one: a step of four for them slowed the loop of eights, 8.2 -> 10.6 us for 512 tokens of 2048 columns
// and 16 slots). HBM bound: FP32 rows of every slot are read once. One column / four columns per thread in us, eight slots: 10.7 / 7.6
// for 512 tokens of 4096 columns, 2.8 / 2.8 for 64 of 4096, 2.1 / 2.5 for 64 of 1024 (its weights in shared memory cost a barrier).
template <int S>
__device__ __forceinline__ void combine4(const float * ys, const float * wk, int64_t n, float4 & acc) {
    float4 v[S];
#pragma unroll
    for (int k = 0; k < S; k++) { v[k] = __ldcs((const float4 *) (ys + k * n)); }
#pragma unroll
    for (int k = 0; k < S; k++) {
        acc.x = fmaf(wk[k], v[k].x, acc.x); acc.y = fmaf(wk[k], v[k].y, acc.y);
        acc.z = fmaf(wk[k], v[k].z, acc.z); acc.w = fmaf(wk[k], v[k].w, acc.w);
    }
}
__global__ void __launch_bounds__(256) k_combine4(const float * __restrict__ ys, const char * __restrict__ w, bool w_bf16, char * __restrict__ y, bool y_bf16,
                                                  int n_used, int64_t n) {
    __shared__ float ws[1024];
    const int t = blockIdx.y;
    for (int k = threadIdx.x; k < n_used; k += 256) {
        const int64_t s = (int64_t) t * n_used + k;
        ws[k] = w_bf16 ? to_f32(((const __nv_bfloat16 *) w)[s]) : ((const float *) w)[s];
    }
    __syncthreads();
    for (int64_t i = (blockIdx.x * 256ll + threadIdx.x) * 4; i < n; i += gridDim.x * 1024ll) {
        const float * p = ys + (int64_t) t * n_used * n + i;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        int k = 0;
        for (; k + 8 <= n_used; k += 8) { combine4<8>(p + k * n, ws + k, n, acc); }
        for (; k < n_used; k++) { combine4<1>(p + k * n, ws + k, n, acc); }
        if (y_bf16) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(acc.x, acc.y), b = __floats2bfloat162_rn(acc.z, acc.w);
            ((uint2 *) y)[(t * n + i) / 4] = make_uint2(*(const uint32_t *) &a, *(const uint32_t *) &b);
        } else { ((float4 *) y)[(t * n + i) / 4] = acc; }
    }
}

// ---------------------------------------------------------------- routing sort (prefill)

// One block per expert. Pass 1 counts the routed pairs of lower-numbered experts (this expert's first output index);
// pass 2 walks the tokens in order, THREADS at a time (latency bound: a step is two block barriers and a trip to L2), and
// compacts the tokens that use this expert with a block-wide exclusive scan, so the expert's pairs come out sorted by token.
// Blocks of 1024 threads take fewer steps where every block has an SM to itself and the tokens are many; otherwise they only
// start later and share SMs. 256 / 1024 threads in us, eight slots per token: 64 experts 2.4 / 3.4 at 64 tokens, 4.1 / 4.1 at
// 1024, 25.1 / 17.0 at 8192; 160 experts 4.7 / 5.8 at 1024, 27.0 / 28.7 at 8192; 512 experts 33.9 / 52.3 at 8192.
template <int THREADS, typename TI>
__global__ void __launch_bounds__(THREADS) k_route(const TI * __restrict__ ids, int64_t row_stride, int32_t * __restrict__ ids_src1,
                                                   int32_t * __restrict__ ids_dst, int32_t * __restrict__ bounds, int n_tok, int n_used,
                                                   int nchannels_y, int sis1) {
    constexpr int WARPS = THREADS / 32;
    const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int warp_tot[WARPS];
    __shared__ int s_base;

    // int32 ids in contiguous rows of a multiple of four: four ids per load (the common case: 8 slots per token)
    const bool vec = sizeof(TI) == 4 && n_used % 4 == 0 && row_stride == n_used && ((uintptr_t) ids & 15) == 0;
    int lower = 0;
    if (vec) {
        const int4 * v = (const int4 *) ids;
        for (int64_t i = tid; i < (int64_t) n_tok * n_used / 4; i += THREADS) {
            const int4 q = __ldg(v + i);
            lower += (q.x < e) + (q.y < e) + (q.z < e) + (q.w < e);
        }
    } else {
        for (int64_t i = tid; i < (int64_t) n_tok * n_used; i += THREADS) {
            const int t = (int) (i / n_used), s = (int) (i - (int64_t) t * n_used);
            lower += (int) ids[t * row_stride + s] < e;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) { lower += __shfl_xor_sync(FULL, lower, o); }
    if (lane == 0) { warp_tot[warp] = lower; }
    __syncthreads();
    if (tid == 0) {
        int b = 0;
        for (int i = 0; i < WARPS; i++) { b += warp_tot[i]; }
        s_base = b;
    }
    __syncthreads();
    const int base = s_base;
    int done = 0;
    for (int t0 = 0; t0 < n_tok; t0 += THREADS) {
        const int t = t0 + tid;
        int slot = -1;
        if (t < n_tok) {
            if (vec) {
                const int4 * v = (const int4 *) ids + (int64_t) t * (n_used / 4);
                for (int s4 = n_used / 4 - 1; s4 >= 0; s4--) { // downwards, so that the lowest matching slot wins
                    const int4 q = __ldg(v + s4);
                    slot = q.w == e ? 4 * s4 + 3 : slot;
                    slot = q.z == e ? 4 * s4 + 2 : slot;
                    slot = q.y == e ? 4 * s4 + 1 : slot;
                    slot = q.x == e ? 4 * s4 : slot;
                }
            } else {
                for (int s = 0; s < n_used; s++) {
                    if ((int) ids[t * row_stride + s] == e) { slot = s; break; }
                }
            }
        }
        const unsigned hit = __ballot_sync(FULL, slot >= 0);
        __syncthreads(); // warp_tot is reused
        if (lane == 0) { warp_tot[warp] = __popc(hit); }
        __syncthreads();
        int before = 0, total = 0;
        for (int i = 0; i < WARPS; i++) {
            before += i < warp ? warp_tot[i] : 0;
            total += warp_tot[i];
        }
        if (slot >= 0) {
            const int j = base + done + before + __popc(hit & ((1u << lane) - 1));
            ids_src1[j] = t * sis1 + slot % nchannels_y;
            ids_dst[j] = t * n_used + slot;
        }
        done += total;
    }
    if (tid == 0) {
        bounds[e] = base;
        if (e == (int) gridDim.x - 1) { bounds[e + 1] = base + done; }
    }
}

} // namespace

void moe_init() {}

void moe_topk(const float * logits, int n_tok, int n_experts, int k, int32_t * ids, float * weights, cudaStream_t st) {
    require(n_tok >= 0 && n_experts > 0 && n_experts <= 32 * TOPK_MAX_PER_LANE, "moe_topk: 1..1024 experts");
    require(k > 0 && k <= 32 && k <= n_experts, "moe_topk: k must be in 1..min(32, n_experts)");
    if (n_tok == 0) { return; }
    if (n_experts <= 256) {
        launch_chained(k_topk<8>, dim3(n_tok), dim3(32), 0, st, logits, n_experts, k, ids, weights);
    } else {
        launch_chained(k_topk<TOPK_MAX_PER_LANE>, dim3(n_tok), dim3(32), 0, st, logits, n_experts, k, ids, weights);
    }
}

void moe_combine(const float * ys, const void * w, bool w_bf16, void * y, bool y_bf16, int n_tok, int n_used, int64_t n,
                 cudaStream_t st) {
    if (n_tok == 0 || n == 0) { return; }
    require(n_tok <= 65535, "moe_combine: too many tokens for one launch");
    if (n_tok * n >= 1 << 18 && n % 4 == 0 && n_used <= 1024 && ((uintptr_t) ys | (uintptr_t) y) % 16 == 0) {
        const dim3 grid4((unsigned) std::min<int64_t>((n + 1023) / 1024, 64), (unsigned) n_tok);
        k_combine4<<<grid4, 256, 0, st>>>(ys, (const char *) w, w_bf16, (char *) y, y_bf16, n_used, n);
        check_launch();
        return;
    }
    const dim3 grid((unsigned) std::min<int64_t>((n + 255) / 256, 64), (unsigned) n_tok);
    k_combine<<<grid, 256, 0, st>>>(ys, (const char *) w, w_bf16, (char *) y, y_bf16, n_used, n);
    check_launch();
}

void moe_swiglu(const float * g, const float * u, float * y, int64_t n, cudaStream_t st) {
    if (n == 0) { return; }
    const unsigned blocks = (unsigned) std::min<int64_t>((n + 255) / 256, (int64_t) device_info().sms * 8);
    launch_chained(k_swiglu, dim3(blocks), dim3(256), 0, st, g, u, y, n);
    check_launch();
}

void moe_route(const void * ids, bool ids_i64, int64_t ids_row_stride, int32_t * ids_src1, int32_t * ids_dst, int32_t * bounds,
               int n_experts, int n_tok, int n_used, int nchannels_y, int sis1, cudaStream_t st) {
    require(n_tok > 0 && n_tok < (1 << 22) && n_used > 0 && n_used < (1 << 10), "routing sizes out of range");
    require(n_experts > 0, "routing needs at least one expert");
    require((int64_t) n_tok * ids_row_stride < INT32_MAX, "routing ids too large for 32-bit indexing");
    const bool wide = n_experts <= device_info().sms && n_tok >= 1024;
    if (ids_i64) {
        const auto kernel = wide ? k_route<1024, int64_t> : k_route<256, int64_t>;
        kernel<<<n_experts, wide ? 1024 : 256, 0, st>>>((const int64_t *) ids, ids_row_stride, ids_src1, ids_dst, bounds, n_tok, n_used, nchannels_y, sis1);
    } else {
        const auto kernel = wide ? k_route<1024, int32_t> : k_route<256, int32_t>;
        kernel<<<n_experts, wide ? 1024 : 256, 0, st>>>((const int32_t *) ids, ids_row_stride, ids_src1, ids_dst, bounds, n_tok, n_used, nchannels_y, sis1);
    }
    check_launch();
}

} // namespace b16
