// Draft-only k-bit copies of an output head (the reference's core/include/bf16n/draft_head.cuh:22-281, declared for its
// op shim at core/torch/torch_bindings.cpp:22-29): a 4-bit or 2-bit copy of a BF16 matrix with one FP32 scale per 128
// weights scores candidates, which the caller re-scores exactly from the lossless rows. The stored formats are the
// reference's, so copies made by either library serve either GEMV:
//   4 bit: q[r][k / 2], column k in the low (k even) or high nibble, value + 8; scale = amax / 7 (1 for a zero group)
//   2 bit: bits 2 (k % 16) of 32-bit word k / 16 of row r hold n in 0..3, value (n - 1.5) s, s = amax / 1.5 correctly
//          rounded; floor(w / s) clamped to [-2, 1], so ties go to the upper level; an all-zero group has s = 0
// The products are approximate by design (FP16 partial sums over one 32-bit word of weights); every column takes the
// same operations in the same order whatever the batch, so a column's scores do not depend on its neighbours.
//
// Built for B200 rather than carried over: quantisation is warp-cooperative (a warp per 128-weight group: coalesced
// 8-byte loads, shuffle reductions, packing by shuffles), and the GEMV is a persistent grid of one-warp-per-row loops
// with the next rows' 16 bytes per lane in flight while the current one is multiplied. A whole draft step (one token, 62080
// rows, 2 bits, 128 candidates) takes 66 us, about a third each for the scores, the selection and the row gather; with torch's topk,
// einsum, fill and scatter around the general row gather it took 270.
#include "decode.cuh"
#include "launch.h"

#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <type_traits>

namespace b16 {
namespace {

using namespace dev;
using bf16 = __nv_bfloat16;
constexpr int G = 128; // weights per scale

// One warp per (row, group): lane l holds columns 4 l .. 4 l + 3 of the group.
template <int BITS>
__global__ void __launch_bounds__(256) k_kbit_quantize(const bf16 * __restrict__ w, int64_t rows, int K, uint8_t * __restrict__ q,
                                                       float * __restrict__ s) {
    const int lane = threadIdx.x & 31;
    const int groups = K / G;
    const int64_t total = rows * groups;
    for (int64_t i = (blockIdx.x * (int64_t) blockDim.x + threadIdx.x) >> 5; i < total; i += ((int64_t) gridDim.x * blockDim.x) >> 5) {
        const int64_t r = i / groups;
        const int g = (int) (i - r * groups);
        const uint2 raw = __ldg((const uint2 *) (w + r * K + g * G) + lane);
        const float v[4] = {bf16lo_f32(raw.x), bf16hi_f32(raw.x), bf16lo_f32(raw.y), bf16hi_f32(raw.y)};
        float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
        for (int o = 16; o; o >>= 1) { amax = fmaxf(amax, __shfl_xor_sync(FULL, amax, o)); }
        if (BITS == 4) {
            const float scale = amax > 0.f ? __fdiv_rn(amax, 7.f) : 1.f;
            uint32_t nib = 0; // four nibbles: columns 4 l .. 4 l + 3 = two bytes
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int a = (int) fminf(fmaxf(rintf(__fdiv_rn(v[c], scale)), -8.f), 7.f) + 8;
                nib |= (uint32_t) a << (4 * c);
            }
            ((uint16_t *) (q + r * (K / 2) + g * (G / 2)))[lane] = (uint16_t) nib;
            if (lane == 0) { s[i] = scale; }
        } else {
            const float scale = __fdiv_rn(amax, 1.5f);
            uint32_t bits = 0; // four 2-bit levels = one byte: columns 4 l .. 4 l + 3 are bits 8 (l % 4) .. of word l / 4
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int n = scale > 0.f ? (int) fminf(fmaxf(floorf(__fdiv_rn(v[c], scale)), -2.f), 1.f) + 2 : 2;
                bits |= (uint32_t) n << (2 * c);
            }
            (q + r * (K / 4) + g * (G / 4))[lane] = (uint8_t) bits;
            if (lane == 0) { s[i] = scale; }
        }
    }
}

__device__ __forceinline__ __half2 magic_half2(uint32_t fields) { // two small integers in bits 0.. and 16.. -> (1024 + a, 1024 + b)
    const uint32_t p = fields | 0x64006400u;
    return *(const __half2 *) &p;
}

// eight consecutive activations; x need only be aligned to its elements
__device__ __forceinline__ void load_x8(const uint16_t * p, uint32_t (&v)[4]) {
    if (((uintptr_t) p & 15) == 0) {
        const uint4 q = __ldg((const uint4 *) p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) { v[i] = (uint32_t) __ldg(p + 2 * i) | (uint32_t) __ldg(p + 2 * i + 1) << 16; }
    }
}

// 4 bit: one warp per row; per 1024 columns a lane owns 16 contiguous bytes (columns 32 l .. 32 l + 31 of the slab: a
// quarter of a scale group). Word w of them holds columns 8 w .. 8 w + 7, nibble m = column 8 w + m; a half2 pairs
// nibbles j and j + 4 (one shift and one mask). x in registers as half2 in that order.
template <int T, int NIT>
__global__ void __launch_bounds__(256) k_int4_gemv(const bf16 * __restrict__ x, const uint8_t * __restrict__ q, const float * __restrict__ s,
                                                   int64_t rows, float * __restrict__ y) {
    constexpr int K = NIT * 1024;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    grid_dependency_wait(); // at once: launched behind everything older
    __half2 xr[T][NIT][16];
#pragma unroll
    for (int t = 0; t < T; t++) {
#pragma unroll
        for (int it = 0; it < NIT; it++) {
            const uint16_t * xp = (const uint16_t *) x + (int64_t) t * K + it * 1024 + lane * 32;
#pragma unroll
            for (int w = 0; w < 4; w++) {
                uint32_t v8[4];
                load_x8(xp + 8 * w, v8);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t a = v8[j >> 1], b = v8[2 + (j >> 1)];
                    xr[t][it][4 * w + j] = __floats2half2_rn((j & 1) ? bf16hi_f32(a) : bf16lo_f32(a), (j & 1) ? bf16hi_f32(b) : bf16lo_f32(b));
                }
            }
        }
    }
    const __half2 bias = __float2half2_rn(1032.f); // 1024 + 8
    const int64_t stride = (int64_t) gridDim.x * 8;
    int64_t r = blockIdx.x * 8 + warp;
    uint4 v[NIT]; float sc[NIT];
    auto load = [&](int64_t row, uint4 (&vv)[NIT], float (&ss)[NIT]) {
#pragma unroll
        for (int it = 0; it < NIT; it++) {
            vv[it] = ld_stream16(q + row * (K / 2) + it * 512 + lane * 16);
            ss[it] = __ldg(s + row * (K / G) + it * 8 + lane / 4);
        }
    };
    if (r < rows) { load(r, v, sc); }
    for (; r < rows; r += stride) {
        uint4 vn[NIT]; float scn[NIT];
#pragma unroll
        for (int it = 0; it < NIT; it++) { vn[it] = make_uint4(0, 0, 0, 0); scn[it] = 0.f; }
        if (r + stride < rows) { load(r + stride, vn, scn); }
        float acc[T];
#pragma unroll
        for (int t = 0; t < T; t++) { acc[t] = 0.f; }
#pragma unroll
        for (int it = 0; it < NIT; it++) {
            const uint32_t words[4] = {v[it].x, v[it].y, v[it].z, v[it].w};
            __half2 h[T];
#pragma unroll
            for (int t = 0; t < T; t++) { h[t] = __float2half2_rn(0.f); }
#pragma unroll
            for (int w = 0; w < 4; w++) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __half2 wv = __hsub2(magic_half2((words[w] >> (4 * j)) & 0x000F000Fu), bias);
#pragma unroll
                    for (int t = 0; t < T; t++) { h[t] = __hfma2(wv, xr[t][it][4 * w + j], h[t]); }
                }
            }
#pragma unroll
            for (int t = 0; t < T; t++) {
                const float2 f = __half22float2(h[t]);
                acc[t] = fmaf(f.x + f.y, sc[it], acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < T; t++) {
            const float val = warp_sum(acc[t]);
            if (lane == 0) { y[(int64_t) t * rows + r] = val; }
        }
#pragma unroll
        for (int it = 0; it < NIT; it++) { v[it] = vn[it]; sc[it] = scn[it]; }
    }
}

// Two 2-bit fields where they lie (bits 2 j, 2 j + 1 of the halves, j <= 4; fields 5..7 are 2..4 of the word moved down by six) under the
// exponent of 1024.0: 1024 + n 4^j, and n by one exact multiply-add. Against fields moved to one place by a multiply each: fewer
// instructions on the pipe that the half-precision products need (98 -> 82 a row).
struct FieldScale { __half2 unit[5], offset[5]; }; // 4^-j, -1024 4^-j
template <int J> __device__ __forceinline__ __half2 field(uint32_t word, uint32_t down6, const FieldScale & k) { // field J of both halves
    constexpr int P = J < 5 ? J : J - 3;
    uint32_t p;
    asm("lop3.b32 %0, %1, %2, 0x64006400, 0xEA;" : "=r"(p) : "r"(J < 5 ? word : down6), "n"(0x00030003 << (2 * P))); // (a & b) | c
    return __hfma2(*(const __half2 *) &p, k.unit[P], k.offset[P]);
}

// warp_sum of four values: lanes 8 i .. 8 i + 7 get the i-th. The same additions in the same order (xor 16, 8, 4, 2, 1), six
// shuffles for four values instead of twenty.
__device__ __forceinline__ float warp_sum4(const float (&v)[4], int lane) {
    const bool up = lane & 16, odd = lane & 8;
    const float a = (up ? v[2] : v[0]) + __shfl_xor_sync(FULL, up ? v[0] : v[2], 16);
    const float b = (up ? v[3] : v[1]) + __shfl_xor_sync(FULL, up ? v[1] : v[3], 16);
    float s = (odd ? b : a) + __shfl_xor_sync(FULL, odd ? a : b, 8);
#pragma unroll
    for (int o = 4; o; o >>= 1) { s += __shfl_xor_sync(FULL, s, o); }
    return s;
}

// 2 bit, K = 2048: a lane owns 16 contiguous bytes = 64 weights (half a scale group); a half2 pairs the fields at bits
// 2 j and 2 j + 16 of a word (columns 16 wd + j and 16 wd + j + 8). sum_k (n_k - 1.5) x_k = sum_k n_k x_k - 1.5 sum_k x_k:
// the second sum is a per-lane constant of the column. 62080 rows, one column: 20.0 us with moved fields and a butterfly to each
// row, 18.0 with fields in place and one butterfly for four rows (two columns 27.4 and 24.2). A row is only 512 bytes, so a warp keeps AHEAD rows in flight.
template <int NC>
__global__ void __launch_bounds__(256, NC == 1 ? 2 : 1) k_int2_gemv(const bf16 * __restrict__ x, const uint8_t * __restrict__ q,
                                                                      const float * __restrict__ s, int64_t rows, float * __restrict__ y, const FieldScale k) {
    constexpr int K = 2048, AHEAD = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    grid_dependency_wait(); // at once: launched behind everything older
    const int64_t stride = (int64_t) gridDim.x * 8;
    int64_t r = blockIdx.x * 8 + warp;
    uint4 v[AHEAD]; float sc[AHEAD];
    auto load = [&](int64_t row, uint4 & vv, float & ss) {
        vv = make_uint4(0, 0, 0, 0);
        ss = 0.f;
        if (row < rows) {
            vv = ld_stream16(q + row * (K / 4) + lane * 16);
            ss = __ldg(s + row * (K / G) + lane / 2);
        }
    };
#pragma unroll
    for (int i = 0; i < AHEAD; i++) { load(r + i * stride, v[i], sc[i]); }
    __half2 xr[NC][32];
    float xsum[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const uint16_t * xp = (const uint16_t *) x + (int64_t) c * K + lane * 64;
        float sum = 0.f;
#pragma unroll
        for (int wd = 0; wd < 4; wd++) {
            uint32_t a8[4], b8[4]; // columns 16 wd .. + 7 and + 8 .. + 15
            load_x8(xp + 16 * wd, a8);
            load_x8(xp + 16 * wd + 8, b8);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float a = (j & 1) ? bf16hi_f32(a8[j >> 1]) : bf16lo_f32(a8[j >> 1]);
                const float b = (j & 1) ? bf16hi_f32(b8[j >> 1]) : bf16lo_f32(b8[j >> 1]);
                xr[c][8 * wd + j] = __floats2half2_rn(a, b);
                sum += a + b;
            }
        }
        xsum[c] = sum;
    }
    for (; r < rows; r += AHEAD * stride) {
        float sums[NC][AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int64_t ri = r + i * stride;
            const uint32_t words[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            const float scale = sc[i];
            load(ri + AHEAD * stride, v[i], sc[i]);
            float nx[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) { nx[c] = 0.f; }
#pragma unroll
            for (int wd = 0; wd < 4; wd++) {
                const uint32_t down6 = words[wd] >> 6;
                __half2 h0[NC], h1[NC]; // two chains of four products: half the dependent latency
#pragma unroll
                for (int c = 0; c < NC; c++) { h0[c] = h1[c] = __float2half2_rn(0.f); }
                auto two = [&](auto jj) {
                    constexpr int j = decltype(jj)::value;
                    const __half2 w0 = field<j>(words[wd], down6, k), w1 = field<j + 1>(words[wd], down6, k);
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        h0[c] = __hfma2(w0, xr[c][8 * wd + j], h0[c]);
                        h1[c] = __hfma2(w1, xr[c][8 * wd + j + 1], h1[c]);
                    }
                };
                two(std::integral_constant<int, 0>{}); two(std::integral_constant<int, 2>{});
                two(std::integral_constant<int, 4>{}); two(std::integral_constant<int, 6>{});
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const float2 f = __half22float2(__hadd2(h0[c], h1[c]));
                    nx[c] += f.x + f.y;
                }
            }
#pragma unroll
            for (int c = 0; c < NC; c++) { sums[c][i] = fmaf(fmaf(-1.5f, xsum[c], nx[c]), scale, 0.f); }
        }
        const int64_t ri = r + (lane >> 3) * stride;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const float val = warp_sum4(sums[c], lane);
            if ((lane & 7) == 0 && ri < rows) { y[(int64_t) c * rows + ri] = val; }
        }
    }
}

unsigned quantize_blocks(int64_t rows, int K) { // 8 warps per block, a warp per group
    return (unsigned) std::max<int64_t>(1, std::min<int64_t>((rows * (K / G) + 7) / 8, (int64_t) device_info().sms * 32));
}

template <int T>
void int4_gemv_t(const bf16 * x, const uint8_t * q, const float * s, int64_t rows, int K, float * y, unsigned blocks, cudaStream_t st) {
    switch (K) {
        case 1024: k_int4_gemv<T, 1><<<blocks, 256, 0, st>>>(x, q, s, rows, y); break;
        case 2048: k_int4_gemv<T, 2><<<blocks, 256, 0, st>>>(x, q, s, rows, y); break;
        default: k_int4_gemv<T, 4><<<blocks, 256, 0, st>>>(x, q, s, rows, y); break;
    }
}

// ---------------------------------------------------------------- candidates of a draft step
//
// The n_cand largest of a token's scores (ties: lowest row; NaN counts as the largest value), in no particular order, and
// -inf in every logit. One cluster of eight blocks per token keeps the order-preserving integer keys of the scores in
// shared memory and finds the n_cand-th largest key digit by digit (11 + 11 + 10 bits): a histogram per block, added up
// over the cluster through distributed shared memory, one cluster barrier per digit. Latency bound: 248 KB of scores for
// 62080 rows.
constexpr int SEL_BLOCKS = 8, SEL_THREADS = 1024, SEL_BINS = 2048;
// Most of that is the barriers and the trips to the other blocks' histograms, and few keys matter: a block whose n_cand-th largest key lies in
// a bin of the first digit has n_cand keys from that bin on, so no key below the largest of the blocks' bins is wanted. Each block
// lists its keys from there on (a hundred or two of 7760 for 62080 rows and 128 candidates), and the first block finds the n_cand largest of the
// lists on its own: a draft step of 62080 rows 43.1 -> 36.0 us, of four tokens 90 -> 70. Where a list does not fit (scores of many rows that are all alike), the
// digits are found by the whole cluster. Scores that are all alike and fit (a hidden state of zeros, up to 8192 rows): a step
// of 8192 rows 47 us by the whole cluster, 2109 with each tie compared with every entry, 29 with the rows found digit by digit too.
constexpr int SEL_LIST = 1024;            // keys of a block's list
constexpr int SEL_KEYS_MAX = 48 * 1024;   // keys of a block that shared memory holds; beyond, every pass reads the scores again

__device__ __forceinline__ uint32_t score_key(float v) {
    const uint32_t b = __float_as_uint(v);
    return v == v ? b ^ ((b & 0x80000000u) ? 0xffffffffu : 0x80000000u) : 0xffffffffu;
}

__global__ void __cluster_dims__(SEL_BLOCKS, 1, 1) __launch_bounds__(SEL_THREADS)
k_select(const float * __restrict__ scores, int rows, int n_cand, int32_t * __restrict__ cand, float * __restrict__ out, int64_t vocab,
         int per, int keys_in_smem, int listed) {
    extern __shared__ __align__(16) uint32_t keys[];
    __shared__ uint32_t hist[3][SEL_BINS];
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t s_bin, s_above, s_equal, s_count, s_run, s_listed;
    __shared__ uint2 list[SEL_LIST]; // key, row
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int) cluster.block_rank(), t = blockIdx.y;
    for (int i = tid; i < 3 * SEL_BINS; i += SEL_THREADS) { hist[0][i] = 0u; }
    if (tid == 0) { s_count = 0u; s_listed = 0u; s_bin = 0u; }
    grid_dependency_wait(); // the scores come from the launch before this one, which may also be reading `out`'s last values
    const float * z = scores + (int64_t) t * rows;
    const int lo = min(rows, rank * per), n = min(rows, lo + per) - lo;
    auto key = [&](int i) -> uint32_t { return keys_in_smem ? keys[i] : score_key(ld_act_f32(z + lo + i)); };
    if (keys_in_smem) {
        int i = tid;
        for (; i + 7 * SEL_THREADS < n; i += 8 * SEL_THREADS) { // eight loads in flight: one trip to L2, not eight
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) { v[j] = ld_act_f32(z + lo + i + j * SEL_THREADS); }
#pragma unroll
            for (int j = 0; j < 8; j++) { keys[i + j * SEL_THREADS] = score_key(v[j]); }
        }
        float v[8];
#pragma unroll
        for (int j = 0; j < 7; j++) { v[j] = i + j * SEL_THREADS < n ? ld_act_f32(z + lo + i + j * SEL_THREADS) : 0.f; }
#pragma unroll
        for (int j = 0; j < 7; j++) {
            if (i + j * SEL_THREADS < n) { keys[i + j * SEL_THREADS] = score_key(v[j]); }
        }
    }
    {   // this block's share of the logits
        const int64_t share = (vocab + SEL_BLOCKS - 1) / SEL_BLOCKS, first = rank * share, last = first + share < vocab ? first + share : vocab;
        for (int64_t i = first + tid; i < last; i += SEL_THREADS) { out[t * vocab + i] = -INFINITY; }
    }
    __syncthreads();

    // Where the need-th largest key lies goes to s_bin, s_above (keys in larger bins) and s_equal (keys in the bin); bins from the
    // largest down: a thread holds b0 with c0 keys and the one below with c1
    auto find = [&](int b0, uint32_t c0, uint32_t c1, uint32_t need) {
        uint32_t run = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, run, o);
            if (lane >= o) { run += up; }
        }
        if (lane == 31) { warp_tot[warp] = run; }
        __syncthreads();
        uint32_t before = 0;
        for (int w = 0; w < warp; w++) { before += warp_tot[w]; }
        before += run - (c0 + c1); // keys in larger bins
        if (before < need && need <= before + c0) { s_bin = (uint32_t) b0; s_above = before; s_equal = c0; }
        else if (before + c0 < need && need <= before + c0 + c1) { s_bin = (uint32_t) b0 - 1u; s_above = before + c0; s_equal = c1; }
        __syncthreads();
    };
    auto digit = [](int pass, int & shift, int & width) { shift = pass == 0 ? 21 : pass == 1 ? 10 : 0; width = pass == 2 ? 10 : 11; };
    int32_t * mine = cand + (int64_t) t * n_cand;
    uint32_t prefix = 0, need = (uint32_t) n_cand, equal = 0;
    if (listed) {
        for (int i = tid; i < n; i += SEL_THREADS) { atomicAdd(&hist[0][key(i) >> 21], 1u); }
        __syncthreads();
        const int top_bin = SEL_BINS - 1 - 2 * tid;
        find(top_bin, hist[0][top_bin], hist[0][top_bin - 1], need); // fewer than n_cand keys: bin 0 stays
        cluster.sync();
        uint32_t low = 0;
        for (int r = 0; r < SEL_BLOCKS; r++) { low = max(low, *cluster.map_shared_rank(&s_bin, r)); }
        low <<= 21;
        for (int i0 = 0; i0 < n; i0 += SEL_THREADS) {
            const uint32_t v = i0 + tid < n ? key(i0 + tid) : 0u;
            const bool hit = i0 + tid < n && v >= low;
            const uint32_t m = __ballot_sync(FULL, hit);
            uint32_t at = 0;
            if (lane == 0 && m) { at = atomicAdd(&s_listed, (uint32_t) __popc(m)); }
            at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (hit && at < SEL_LIST) { list[at] = make_uint2(v, (uint32_t) (lo + i0 + tid)); }
        }
        cluster.sync();
        uint32_t first[SEL_BLOCKS + 1] = {0u};
        bool fits = true;
#pragma unroll
        for (int r = 0; r < SEL_BLOCKS; r++) {
            const uint32_t c = *cluster.map_shared_rank(&s_listed, r);
            fits = fits && c <= SEL_LIST;
            first[r + 1] = first[r] + c;
        }
        if (fits) { // the whole cluster takes this branch
            if (rank != 0) { cluster.sync(); return; } // until the lists are read
            uint2 * all = (uint2 *) keys; // the keys are not read again
            const int total = (int) first[SEL_BLOCKS];
#pragma unroll
            for (int r = 0; r < SEL_BLOCKS; r++) {
                const uint2 * l = cluster.map_shared_rank(&list[0], r);
                for (int i = tid; i < (int) (first[r + 1] - first[r]); i += SEL_THREADS) { all[first[r] + i] = l[i]; }
            }
            cluster.sync();
            // digit by digit the n_cand-th largest key, and where more entries have it than are wanted, the first rows of those: the
            // need-th largest of their rows' complements, in the same three passes
            uint32_t last_row = 0xffffffffu;
#pragma unroll 1
            for (int by_row = 0; by_row < 2; by_row++) {
                for (int i = tid; i < 3 * SEL_BINS; i += SEL_THREADS) { hist[0][i] = 0u; }
                __syncthreads();
                uint32_t found = 0;
#pragma unroll 1
                for (int pass = 0; pass < 3; pass++) {
                    int shift, width;
                    digit(pass, shift, width);
                    for (int i = tid; i < total; i += SEL_THREADS) {
                        const uint2 e = all[i];
                        const uint32_t v = by_row ? ~e.y : e.x;
                        if ((!by_row || e.x == prefix) && (pass == 0 || (v >> (shift + width)) == found)) { atomicAdd(&hist[pass][(v >> shift) & ((1u << width) - 1u)], 1u); }
                    }
                    __syncthreads();
                    const int b = (1 << width) - 1 - 2 * tid;
                    find(b, b >= 0 ? hist[pass][b] : 0u, b >= 0 ? hist[pass][b - 1] : 0u, need);
                    found = found << width | s_bin;
                    need -= s_above;
                    equal = s_equal;
                }
                if (by_row) { last_row = ~found; break; }
                prefix = found;
                if (equal == need) { break; }
            }
            for (int i = tid; i < total; i += SEL_THREADS) {
                const uint2 v = all[i];
                if (v.x > prefix || (v.x == prefix && v.y <= last_row)) { mine[atomicAdd(&s_count, 1u)] = (int32_t) v.y; }
            }
            return;
        }
    }
#pragma unroll 1
    for (int pass = 0; pass < 3; pass++) {
        int shift, width;
        digit(pass, shift, width);
        for (int i = tid; i < n && !(listed && pass == 0); i += SEL_THREADS) { // listed: the first digit is counted
            const uint32_t v = key(i);
            if (pass == 0 || (v >> (shift + width)) == prefix) { atomicAdd(&hist[pass][(v >> shift) & ((1u << width) - 1u)], 1u); }
        }
        cluster.sync();
        const int b0 = (1 << width) - 1 - 2 * tid;
        uint32_t c0 = 0, c1 = 0;
        if (b0 >= 0) {
            for (int r = 0; r < SEL_BLOCKS; r++) {
                const uint32_t * h = cluster.map_shared_rank(&hist[pass][0], r);
                c0 += h[b0];
                c1 += h[b0 - 1];
            }
        }
        find(b0, c0, c1, need);
        prefix = prefix << width | s_bin;
        need -= s_above;
        equal = s_equal;
    }
    // every key above `prefix`, and `need` of the `equal` ones that are the same: the first in row order
    uint32_t * count = cluster.map_shared_rank(&s_count, 0);
    for (int i = tid; i < n; i += SEL_THREADS) {
        const uint32_t v = key(i);
        if (v > prefix || (v == prefix && equal == need)) { mine[atomicAdd(count, 1u)] = lo + i; }
    }
    if (equal != need) { // the whole cluster takes this branch
        uint32_t before = 0;
        for (int r = 0; r < rank; r++) { before += cluster.map_shared_rank(&hist[2][0], r)[prefix & 1023u]; }
        if (tid == 0) { s_run = before; }
        __syncthreads();
        for (int i0 = 0; i0 < n && s_run < need; i0 += SEL_THREADS) {
            const bool hit = i0 + tid < n && key(i0 + tid) == prefix;
            const uint32_t m = __ballot_sync(FULL, hit);
            if (lane == 0) { warp_tot[warp] = __popc(m); }
            const uint32_t start = s_run;
            __syncthreads();
            uint32_t at = start, total = 0;
            for (int w = 0; w < SEL_THREADS / 32; w++) {
                at += w < warp ? warp_tot[w] : 0u;
                total += warp_tot[w];
            }
            at += __popc(m & ((1u << lane) - 1u));
            if (hit && at < need) { mine[atomicAdd(count, 1u)] = lo + i0 + tid; }
            __syncthreads();
            if (tid == 0) { s_run = start + total; }
            __syncthreads();
        }
    }
    cluster.sync(); // no block leaves while another still reads or counts in its shared memory
}

// out[t, cand[t, c]] = row . h_t, one warp per candidate: exact BF16 rows, FP32 sums
__global__ void __launch_bounds__(128) k_rescore(const bf16 * __restrict__ x, const bf16 * __restrict__ row, const int32_t * __restrict__ cand,
                                                 int n, int n_cand, int K, float * __restrict__ out, int64_t vocab) {
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= n) { return; }
    const int t = i / n_cand;
    const bf16 * a = row + (int64_t) i * K, * b = x + (int64_t) t * K;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = lane * 8; k < K; k += 256) {
        const uint4 p = ld_act16(a + k), q = ld_act16(b + k);
        acc[0] = fmaf(bf16lo_f32(p.x), bf16lo_f32(q.x), acc[0]); acc[1] = fmaf(bf16hi_f32(p.x), bf16hi_f32(q.x), acc[1]);
        acc[2] = fmaf(bf16lo_f32(p.y), bf16lo_f32(q.y), acc[2]); acc[3] = fmaf(bf16hi_f32(p.y), bf16hi_f32(q.y), acc[3]);
        acc[0] = fmaf(bf16lo_f32(p.z), bf16lo_f32(q.z), acc[0]); acc[1] = fmaf(bf16hi_f32(p.z), bf16hi_f32(q.z), acc[1]);
        acc[2] = fmaf(bf16lo_f32(p.w), bf16lo_f32(q.w), acc[2]); acc[3] = fmaf(bf16hi_f32(p.w), bf16hi_f32(q.w), acc[3]);
    }
    const float v = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
    const int32_t r = *(const volatile int32_t *) (cand + i);
    if (lane == 0) { out[t * vocab + r] = v; }
}

} // namespace

void draft_quantize(int bits, const void * w_bf16, int64_t rows, int K, uint8_t * q, float * s, cudaStream_t st) {
    require(bits == 2 || bits == 4, "draft head: 2 or 4 bits");
    require(K > 0 && K % G == 0, bits == 4 ? "int4_quantize: K must be a multiple of 128" : "int2_quantize: K must be a multiple of 128");
    require(rows >= 0 && (rows == 0 || (w_bf16 && q && s)), "draft head quantize: null argument");
    require((uintptr_t) w_bf16 % 8 == 0 && (uintptr_t) q % 4 == 0, "draft head quantize: w must be 8-byte and q 4-byte aligned");
    if (rows == 0) { return; }
    if (bits == 4) { k_kbit_quantize<4><<<quantize_blocks(rows, K), 256, 0, st>>>((const bf16 *) w_bf16, rows, K, q, s); }
    else { k_kbit_quantize<2><<<quantize_blocks(rows, K), 256, 0, st>>>((const bf16 *) w_bf16, rows, K, q, s); }
    check_launch();
}

void draft_gemv(int bits, const void * x_bf16, int T, const uint8_t * q, const float * s, int64_t rows, int K, float * y, cudaStream_t st) {
    require(bits == 2 || bits == 4, "draft head: 2 or 4 bits");
    if (bits == 4) { require(K == 1024 || K == 2048 || K == 4096, "int4_gemv: K must be 1024, 2048 or 4096"); }
    else { require(K == 2048, "int2_gemv: K must be 2048"); }
    require(T >= 1 && T <= 4, bits == 4 ? "int4_gemv: 1 to 4 columns" : "int2_gemv: 1 to 4 columns");
    require(rows >= 0 && (rows == 0 || (x_bf16 && q && s && y)), "draft head gemv: null argument");
    require((uintptr_t) q % 16 == 0, "draft head gemv: q must be 16-byte aligned");
    if (rows == 0) { return; }
    const bf16 * x = (const bf16 *) x_bf16;
    const int64_t sms = device_info().sms;
    if (bits == 4) {
        const unsigned blocks = (unsigned) std::min<int64_t>((rows + 7) / 8, sms * 8);
        switch (T) {
            case 1: int4_gemv_t<1>(x, q, s, rows, K, y, blocks, st); break;
            case 2: int4_gemv_t<2>(x, q, s, rows, K, y, blocks, st); break;
            case 3: int4_gemv_t<3>(x, q, s, rows, K, y, blocks, st); break;
            default: int4_gemv_t<4>(x, q, s, rows, K, y, blocks, st); break;
        }
    } else {
        FieldScale fields;
        for (int j = 0; j < 5; j++) {
            const float unit = 1.f / (float) (1 << (2 * j));
            fields.unit[j] = __float2half2_rn(unit);
            fields.offset[j] = __float2half2_rn(-1024.f * unit);
        }
        for (int t = 0; t < T; t += 2) { // two columns per launch, an odd last one alone
            if (T - t >= 2) {
                const unsigned blocks = (unsigned) std::min<int64_t>((rows + 7) / 8, sms);
                k_int2_gemv<2><<<blocks, 256, 0, st>>>(x + (int64_t) t * K, q, s, rows, y + (int64_t) t * rows, fields);
            } else {
                const unsigned blocks = (unsigned) std::min<int64_t>((rows + 7) / 8, sms * 2);
                k_int2_gemv<1><<<blocks, 256, 0, st>>>(x + (int64_t) t * K, q, s, rows, y + (int64_t) t * rows, fields);
            }
        }
    }
    check_launch();
}

void draft_init() {
    allow_dynamic_smem((const void *) k_select, SEL_KEYS_MAX * 4, device_info().smem_optin, "k_select");
}

void draft_select(const float * scores, int T, int64_t rows, int n_cand, int32_t * cand, float * out, int64_t vocab, cudaStream_t st) {
    const int per = (int) ((rows + SEL_BLOCKS - 1) / SEL_BLOCKS);
    const bool in_smem = per <= SEL_KEYS_MAX;
    const bool listed = in_smem && n_cand <= SEL_LIST / 2; // lists of more than twice the candidates are rare: scores that are alike
    const size_t shm = !in_smem ? 0 : std::max((size_t) per * 4, listed ? sizeof(uint2) * SEL_BLOCKS * SEL_LIST : 0);
    launch_chained(k_select, dim3(SEL_BLOCKS, (unsigned) T), dim3(SEL_THREADS), shm, st, scores, (int) rows, n_cand, cand, out, vocab, per, in_smem ? 1 : 0,
                   listed ? 1 : 0);
    check_launch();
}

void draft_rescore(const void * x_bf16, const void * rows_bf16, const int32_t * cand, int T, int n_cand, int K, float * out, int64_t vocab,
                   cudaStream_t st) {
    const int n = T * n_cand;
    launch_chained(k_rescore, dim3((unsigned) ((n + 3) / 4)), dim3(128), 0, st, (const bf16 *) x_bf16, (const bf16 *) rows_bf16, cand, n, n_cand, K,
                   out, vocab);
    check_launch();
}

} // namespace b16
