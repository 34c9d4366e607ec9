// Decode-inside-GEMV kernels for 1..4 activation columns, exact dequantisation / verification and row gather, for the
// three BF16N exponent formats. One warp owns one unit (R rows) of a Huffman-coded matrix or one row of a NIBBLE
// matrix; every lane walks its own bit stream; products are accumulated in FP32 in the order the format's lane layout
// implies (four accumulators per lane by column & 3, chunks in order, then a xor butterfly), which makes the results
// independent of the launch geometry and equal, bit for bit, to the reference kernels' order
// (core/include/bf16n/kernels.cuh:498-535, 958-986, 139-187).
#include "sinks.cuh"
#include "staged.cuh"
#include "launch.h"
#include <cstdlib>

namespace b16 {
namespace {

using namespace dev;

// FP32 products of one row-chunk (this lane's 16 weights, as 8 BF16x2 words) with the matching activations
__device__ __forceinline__ void fma_chunk(const uint32_t (&w)[8], const float4 (&x)[4], float (&a)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        a[0] = fmaf(bf16lo_f32(w[2 * j]), x[j].x, a[0]);
        a[1] = fmaf(bf16hi_f32(w[2 * j]), x[j].y, a[1]);
        a[2] = fmaf(bf16lo_f32(w[2 * j + 1]), x[j].z, a[2]);
        a[3] = fmaf(bf16hi_f32(w[2 * j + 1]), x[j].w, a[3]);
    }
}

template <typename TX>
__device__ __forceinline__ void stage_x(float * xs, const TX * xg, int K) {
    for (int i = threadIdx.x; i < K; i += blockDim.x) { xs[i] = to_f32(xg[i]); }
}
__device__ __forceinline__ void stage_lut(uint32_t * dst, const uint32_t * src, int n) {
    for (int i = threadIdx.x; i < n / 4; i += blockDim.x) { ((uint4 *) dst)[i] = __ldg((const uint4 *) src + i); }
}

// ---------------------------------------------------------------- HUFPAIR, row-major units

// NC dense columns (NC == 1: also routed columns, one per blockIdx.y). XR: the lane's activations live in registers.
template <int C, int NC, typename TX, bool XR, bool PEERS = false>
__global__ void __launch_bounds__(512) k_pair_gemv(const PairView w, int R, Cols p) {
    constexpr int K = C * CHUNK;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem;
    float * xs = (float *) (smem + 4 * HP_MAX_PAIRS);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;

    const TX * xg; OutVec out; int64_t rbase;
    column<TX>(p, NC == 1 ? blockIdx.y : 0, xg, out, rbase);
    stage_lut(lut, w.lut, HP_MAX_PAIRS);
#pragma unroll
    for (int n = 0; n < NC; n++) { stage_x<TX>(xs + n * K, (const TX *) ((const char *) xg + n * p.x_tok), K); }
    __syncthreads();

    float4 xr[XR ? C * 4 : 1];
    if (XR) {
#pragma unroll
        for (int i = 0; i < C * 4; i++) { xr[i] = *(const float4 *) (xs + (i >> 2) * CHUNK + 128 * (i & 3) + 4 * lane); }
    }

    const int64_t units = p.nrows / R;
    for (int64_t u = (int64_t) blockIdx.x * nwarp + warp; u < units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t gu = rbase / R + u;
        PairReader rd;
        rd.open(w, gu, lane);
        const uint8_t * pl = w.plane + gu * R * K + 16 * lane;
        uint4 nxt[C];
#pragma unroll
        for (int c = 0; c < C; c++) { nxt[c] = ld_stream16(pl + c * CHUNK); }
        for (int rr = 0; rr < R; rr++) {
            uint4 cur[C];
#pragma unroll
            for (int c = 0; c < C; c++) { cur[c] = nxt[c]; }
            if (rr + 1 < R) {
#pragma unroll
                for (int c = 0; c < C; c++) { nxt[c] = ld_stream16(pl + (rr + 1) * K + c * CHUNK); }
            }
            float a[NC][4];
#pragma unroll
            for (int n = 0; n < NC; n++) { a[n][0] = a[n][1] = a[n][2] = a[n][3] = 0.f; }
#pragma unroll
            for (int c = 0; c < C; c++) {
                uint32_t e[8], wv[8];
                rd.take8(lut, e);
                assemble8(cur[c], e, wv);
#pragma unroll
                for (int n = 0; n < NC; n++) {
                    float4 xq[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        xq[j] = XR ? xr[c * 4 + j] : *(const float4 *) (xs + n * K + c * CHUNK + 128 * j + 4 * lane);
                    }
                    fma_chunk(wv, xq, a[n]);
                }
            }
#pragma unroll
            for (int n = 0; n < NC; n++) {
                const float s = warp_sum((a[n][0] + a[n][1]) + (a[n][2] + a[n][3]));
                if (lane == 0) {
                    OutVec o = out;
                    o.p += n * p.y_tok;
                    o.put(u * R + rr, s);
                    if (PEERS) { peers_put(p, blockIdx.y, u * R + rr, s); }
                }
            }
        }
    }
    if (PEERS) { peers_done(p); }
}

// y = silu(gate x) * (up x), separate row-major gate / up matrices with the same geometry
template <int C, typename TX>
__global__ void __launch_bounds__(512) k_pair_glu(const PairView g, const PairView v, int R, Cols p) {
    constexpr int K = C * CHUNK;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t * lut_g = (uint32_t *) smem;
    uint32_t * lut_v = lut_g + HP_MAX_PAIRS;
    float * xs = (float *) (lut_v + HP_MAX_PAIRS);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const TX * xg; OutVec out; int64_t rbase;
    column<TX>(p, blockIdx.y, xg, out, rbase);
    stage_lut(lut_g, g.lut, HP_MAX_PAIRS);
    stage_lut(lut_v, v.lut, HP_MAX_PAIRS);
    stage_x<TX>(xs, xg, K);
    __syncthreads();
    const int64_t units = p.nrows / R;
    for (int64_t u = (int64_t) blockIdx.x * nwarp + warp; u < units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t gu = rbase / R + u;
        PairReader rg, rv;
        rg.open(g, gu, lane);
        rv.open(v, gu, lane);
        for (int rr = 0; rr < R; rr++) {
            const int64_t row = gu * R + rr;
            float ag[4] = {0.f, 0.f, 0.f, 0.f}, av[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < C; c++) {
                const uint4 sg = ld_stream16(g.plane + row * K + c * CHUNK + 16 * lane);
                const uint4 sv = ld_stream16(v.plane + row * K + c * CHUNK + 16 * lane);
                float4 xq[4];
#pragma unroll
                for (int j = 0; j < 4; j++) { xq[j] = *(const float4 *) (xs + c * CHUNK + 128 * j + 4 * lane); }
                uint32_t e[8], wv[8];
                rg.take8(lut_g, e);
                assemble8(sg, e, wv);
                fma_chunk(wv, xq, ag);
                rv.take8(lut_v, e);
                assemble8(sv, e, wv);
                fma_chunk(wv, xq, av);
            }
            const float gs = warp_sum((ag[0] + ag[1]) + (ag[2] + ag[3]));
            const float vs = warp_sum((av[0] + av[1]) + (av[2] + av[3]));
            if (lane == 0) { out.put(u * R + rr, vs * silu_f(gs)); }
        }
    }
}

// ---------------------------------------------------------------- HUFPAIR, chunk-major units (expert stacks, K > 512)

// Streams and plane run chunk -> row inside a unit: per chunk the lane's 16 activations are read once and reused for
// the R rows; each row adds its per-chunk lane sum, lanes are reduced once per unit.
template <int C, int R, typename TX>
__global__ void __launch_bounds__(512) k_pair_gemv_cm(const PairView w, Cols p) {
    constexpr int K = C * CHUNK;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem;
    float * xs = (float *) (smem + 4 * HP_MAX_PAIRS);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const TX * xg; OutVec out; int64_t rbase;
    column<TX>(p, blockIdx.y, xg, out, rbase);
    stage_lut(lut, w.lut, HP_MAX_PAIRS);
    stage_x<TX>(xs, xg, K);
    __syncthreads();
    const int64_t units = p.nrows / R;
    for (int64_t u = (int64_t) blockIdx.x * nwarp + warp; u < units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t gu = rbase / R + u;
        PairReader rd;
        rd.open(w, gu, lane);
        const uint8_t * pl = w.plane + gu * R * K + 16 * lane;
        float acc[R];
#pragma unroll
        for (int rr = 0; rr < R; rr++) { acc[rr] = 0.f; }
#pragma unroll 1
        for (int c = 0; c < C; c++) {
            float4 xq[4];
#pragma unroll
            for (int j = 0; j < 4; j++) { xq[j] = *(const float4 *) (xs + c * CHUNK + 128 * j + 4 * lane); }
            uint4 sm[R];
#pragma unroll
            for (int rr = 0; rr < R; rr++) { sm[rr] = ld_stream16(pl + (c * R + rr) * CHUNK); }
#pragma unroll
            for (int rr = 0; rr < R; rr++) {
                uint32_t e[8], wv[8];
                rd.take8(lut, e);
                assemble8(sm[rr], e, wv);
                float a[4] = {0.f, 0.f, 0.f, 0.f};
                fma_chunk(wv, xq, a);
                acc[rr] += (a[0] + a[1]) + (a[2] + a[3]);
            }
        }
#pragma unroll
        for (int rr = 0; rr < R; rr++) {
            const float s = warp_sum(acc[rr]);
            if (lane == 0) { out.put(u * R + rr, s); }
        }
    }
}

// ---------------------------------------------------------------- HUFFMAN (single-exponent fallback), row-major units

template <typename TX, bool GLU>
__global__ void __launch_bounds__(256) k_huf_gemv(const HufView g, const HufView v, int C, int R, Cols p) {
    const int K = C * CHUNK;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t * lut_g = (uint32_t *) smem;
    uint32_t * lut_v = lut_g + (1 << HUF_LMAX);
    float * xs = (float *) (lut_v + (GLU ? (1 << HUF_LMAX) : 0));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const TX * xg; OutVec out; int64_t rbase;
    column<TX>(p, blockIdx.y, xg, out, rbase);
    stage_lut(lut_g, g.lut, 1 << HUF_LMAX);
    if (GLU) { stage_lut(lut_v, v.lut, 1 << HUF_LMAX); }
    stage_x<TX>(xs, xg, K);
    __syncthreads();
    const int64_t units = p.nrows / R;
    for (int64_t u = (int64_t) blockIdx.x * nwarp + warp; u < units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t gu = rbase / R + u;
        HufReader rg, rv;
        rg.open(g, gu, lane);
        if (GLU) { rv.open(v, gu, lane); }
        for (int rr = 0; rr < R; rr++) {
            const int64_t row = gu * R + rr;
            float ag[4] = {0.f, 0.f, 0.f, 0.f}, av[4] = {0.f, 0.f, 0.f, 0.f};
            for (int c = 0; c < C; c++) {
                float4 xq[4];
#pragma unroll
                for (int j = 0; j < 4; j++) { xq[j] = *(const float4 *) (xs + c * CHUNK + 128 * j + 4 * lane); }
                uint32_t e[8], wv[8];
                rg.take8(lut_g, e);
                assemble8(ld_stream16(g.plane + row * K + c * CHUNK + 16 * lane), e, wv);
                fma_chunk(wv, xq, ag);
                if (GLU) {
                    rv.take8(lut_v, e);
                    assemble8(ld_stream16(v.plane + row * K + c * CHUNK + 16 * lane), e, wv);
                    fma_chunk(wv, xq, av);
                }
            }
            const float gs = warp_sum((ag[0] + ag[1]) + (ag[2] + ag[3]));
            if (GLU) {
                const float vs = warp_sum((av[0] + av[1]) + (av[2] + av[3]));
                if (lane == 0) { out.put(u * R + rr, vs * silu_f(gs)); }
            } else if (lane == 0) {
                out.put(u * R + rr, gs);
            }
        }
    }
}

// ---------------------------------------------------------------- NIBBLE: one warp per row

template <int C>
struct NibRow { uint4 sm[C]; uint2 cd[C]; uint4 L; uint32_t e0, e1, rec; }; // rec: this lane's first escape record

template <int C, bool RECORDS>
__device__ __forceinline__ void nib_load(NibRow<C> & d, const NibView & w, int64_t row, int lane) {
    constexpr int K = C * CHUNK;
#pragma unroll
    for (int c = 0; c < C; c++) {
        d.sm[c] = __ldg((const uint4 *) (w.plane + row * K + c * CHUNK) + lane);
        d.cd[c] = __ldg((const uint2 *) (w.codes + row * (K / 2) + c * 256) + lane);
    }
    d.L = __ldg(w.row_lut + row);
    d.e0 = __ldg(w.esc_off + row);
    d.e1 = __ldg(w.esc_off + row + 1);
    if (RECORDS) { d.rec = d.e0 + lane < d.e1 ? __ldg(w.esc + d.e0 + lane) : 0u; }
}

// the row's BF16 pairs (escaped slots decode to +0), ready before the activations are
template <int C>
struct NibWords { uint32_t w[C][8]; uint32_t e0, e1, rec; };

template <int C>
__device__ __forceinline__ void nib_decode(const NibRow<C> & r, NibWords<C> & d) {
#pragma unroll
    for (int c = 0; c < C; c++) {
        nib_assemble8(r.sm[c], r.cd[c], r.L, d.w[c]);
#pragma unroll
        for (int q = 0; q < 8; q++) { asm volatile("" : "+r"(d.w[c][q])); } // decoded here, not where they are used
    }
    d.e0 = r.e0; d.e1 = r.e1; d.rec = r.rec;
}

// four activations as they lie in memory
template <typename TX> struct RawX4;
template <> struct RawX4<float> {
    uint4 v;
    __device__ __forceinline__ void load(const float * x) { v = ld_act16(x); }
    __device__ __forceinline__ float4 f() const { return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
};
template <> struct RawX4<bf16> {
    uint2 v;
    __device__ __forceinline__ void load(const bf16 * x) { v = ld_act8(x); }
    __device__ __forceinline__ float4 f() const { return make_float4(bf16lo_f32(v.x), bf16hi_f32(v.x), bf16lo_f32(v.y), bf16hi_f32(v.y)); }
};

// dots of M decoded rows with x: dense pass, then each row's escapes, then the butterfly. The activations of up to four
// chunks are requested before the first of them is used: one trip to L2, not one per chunk.
template <int C, int M, typename TX>
__device__ __forceinline__ void nib_dots(const NibWords<C> (&d)[M], const NibView * const (&w)[M], const TX * x, int lane, float (&sum)[M]) {
    constexpr int G = C < 4 ? C : 4;
    float a[M][4];
#pragma unroll
    for (int m = 0; m < M; m++) { a[m][0] = a[m][1] = a[m][2] = a[m][3] = 0.f; }
#pragma unroll
    for (int c0 = 0; c0 < C; c0 += G) {
        RawX4<TX> q[G * 4];
#pragma unroll
        for (int i = 0; i < G * 4; i++) { q[i].load(x + (c0 + (i >> 2)) * CHUNK + 128 * (i & 3) + 4 * lane); }
#pragma unroll
        for (int c = 0; c < G; c++) {
            const float4 xq[4] = {q[4 * c].f(), q[4 * c + 1].f(), q[4 * c + 2].f(), q[4 * c + 3].f()};
#pragma unroll
            for (int m = 0; m < M; m++) { fma_chunk(d[m].w[c0 + c], xq, a[m]); }
        }
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        float acc = (a[m][0] + a[m][1]) + (a[m][2] + a[m][3]);
        uint32_t rec = d[m].rec;
        for (uint32_t i = d[m].e0 + lane; i < d[m].e1;) {
            acc = fmaf(__uint_as_float(esc_bits(rec) << 16), ldg_x1(x, rec & 0xFFF), acc);
            i += 32;
            if (i < d[m].e1) { rec = __ldg(w[m]->esc + i); }
        }
        sum[m] = warp_sum(acc);
    }
}

// the same for one row as loaded, decoded chunk by chunk as it is multiplied: the same operations in the same order
template <int C, typename TX>
__device__ __forceinline__ float nib_dot(const NibRow<C> & d, const NibView & w, const TX * x, int lane) {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < C; c++) {
        uint32_t wv[8];
        nib_assemble8(d.sm[c], d.cd[c], d.L, wv);
        float4 xq[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { xq[j] = ldg_x4(x, c * CHUNK + 128 * j + 4 * lane); }
        fma_chunk(wv, xq, a);
    }
    float acc = (a[0] + a[1]) + (a[2] + a[3]);
    for (uint32_t i = d.e0 + lane; i < d.e1; i += 32) {
        const uint32_t rec = __ldg(w.esc + i);
        acc = fmaf(__uint_as_float(esc_bits(rec) << 16), ldg_x1(x, rec & 0xFFF), acc);
    }
    return warp_sum(acc);
}

// sums of M rows, AHEAD or as they come; `waited`: this warp has waited for the kernel before this one
template <int C, bool AHEAD, int M, typename TX>
__device__ __forceinline__ void nib_rows(const NibView * const (&w)[M], int64_t row, const TX * x, int lane, bool & waited, float (&sum)[M]) {
    NibRow<C> raw[M];
#pragma unroll
    for (int m = 0; m < M; m++) { nib_load<C, AHEAD>(raw[m], *w[m], row, lane); }
    if constexpr (AHEAD) {
        NibWords<C> d[M];
#pragma unroll
        for (int m = 0; m < M; m++) { nib_decode<C>(raw[m], d[m]); }
        if (!waited) { grid_dependency_wait(); waited = true; }
        nib_dots<C, M, TX>(d, w, x, lane, sum);
    } else {
        if (!waited) { grid_dependency_wait(); waited = true; }
#pragma unroll
        for (int m = 0; m < M; m++) { sum[m] = nib_dot<C, TX>(raw[m], *w[m], x, lane); }
    }
}

// GLU: g rows are the gate, v rows the up half (separate matrices, or the same matrix shifted by nrows rows)
//
// What bounds it: a decode step is a row of launches that depend on each other, each of a few microseconds. So everything
// that does not need the kernel before it is done before the wait for it (launch_chained): the warp's first row is loaded, its
// escapes with it, and decoded to BF16 pairs; its own dependents may start at once, since what they touch before their
// wait belongs to no kernel (weights) and their wait ends only when this kernel, and with it the one it waits for, is complete.
// Behind the wait are one trip to L2 for the activations (one per chunk, and two for a gate/up pair, before), the products and the
// sums. 48 layers of three launches each: 460 -> 349 us; 20 layers at 2 / 4 tokens: 237 / 337 -> 188 / 256 us. Measured and left:
// activations staged in shared memory once per block, its rows multiplied with up to four columns (359 us; 225 / 360).
// A warp's later rows find the kernel before long complete, and there decoding ahead only puts the trip for the row in front of the
// trip for the activations, in registers that cost resident blocks: launches of more than three rows per resident warp request both
// together and decode as they multiply (AHEAD = false / true, us: 2048 x 512, eight tokens 4.5 / 5.2; 8192 x 512, two tokens
// 4.6 / 5.0; 8192 x 4096, one token 10.4 / 11.1).
constexpr int nib_blocks(int C, bool glu) { return glu ? (C <= 2 ? 3 : C == 4 ? 2 : 1) : C == 8 ? 2 : C == 4 ? 3 : 4; } // AHEAD, per SM: room for the launches behind (otherwise 0: the compiler's own choice)
template <int C, typename TX, bool GLU, bool AHEAD>
__global__ void __launch_bounds__(256, AHEAD ? nib_blocks(C, GLU) : 0) k_nib_gemv(const NibView g, const NibView v, Cols p) {
    constexpr int M = GLU ? 2 : 1;
    bool waited = p.ids != nullptr; // expert ids, when there are any, belong to an earlier kernel too
    if (waited) { grid_dependency_wait(); } else if (AHEAD) { grid_launch_dependents(); }
    const TX * xg; OutVec out; int64_t rbase;
    column<TX>(p, blockIdx.y, xg, out, rbase);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NibView * w[M];
    w[0] = &g;
    if constexpr (GLU) { w[1] = &v; }
    for (int64_t r = (int64_t) blockIdx.x * 8 + warp; r < p.nrows; r += (int64_t) gridDim.x * 8) {
        float s[M];
        nib_rows<C, AHEAD, M, TX>(w, rbase + r, xg, lane, waited, s);
        if (lane == 0) {
            if constexpr (GLU) { out.put(r, s[1] * silu_f(s[0])); } else { out.put(r, s[0]); }
        }
    }
}

// ---------------------------------------------------------------- exact reconstruction (dequant / verify / gather)

template <typename Sink>
__global__ void __launch_bounds__(256) k_pair_expand(const PairView w, int C, int R, bool cm, int64_t row0, int64_t nrows, const Sink sink_in) {
    Sink sink = sink_in;
    __shared__ uint32_t lut[HP_MAX_PAIRS];
    stage_lut(lut, w.lut, HP_MAX_PAIRS);
    __syncthreads();
    const int64_t K = (int64_t) C * CHUNK;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t u = (int64_t) blockIdx.x * 8 + warp; u < nrows / R; u += (int64_t) gridDim.x * 8) {
        const int64_t gu = row0 / R + u;
        PairReader rd;
        rd.open(w, gu, lane);
        const uint8_t * pl = w.plane + gu * R * K + 16 * lane;
        for (int o = 0; o < R * C; o++) {
            const int rr = cm ? o % R : o / C, c = cm ? o / R : o % C;
            const uint4 sm = ld_stream16(pl + (cm ? (int64_t) (c * R + rr) * CHUNK : rr * K + (int64_t) c * CHUNK));
            uint32_t e[8], wv[8];
            rd.take8(lut, e);
            assemble8(sm, e, wv);
            sink.chunk(u * R + rr, c, lane, wv);
        }
    }
    sink.finish(lane);
}

template <typename Sink>
__global__ void __launch_bounds__(256) k_huf_expand(const HufView w, int C, int R, int64_t row0, int64_t nrows, const Sink sink_in) {
    Sink sink = sink_in;
    __shared__ uint32_t lut[1 << HUF_LMAX];
    stage_lut(lut, w.lut, 1 << HUF_LMAX);
    __syncthreads();
    const int64_t K = (int64_t) C * CHUNK;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t u = (int64_t) blockIdx.x * 8 + warp; u < nrows / R; u += (int64_t) gridDim.x * 8) {
        const int64_t gu = row0 / R + u;
        HufReader rd;
        rd.open(w, gu, lane);
        for (int o = 0; o < R * C; o++) {
            const int rr = o / C, c = o % C;
            const uint4 sm = ld_stream16(w.plane + (gu * R + rr) * K + (int64_t) c * CHUNK + 16 * lane);
            uint32_t e[8], wv[8];
            rd.take8(lut, e);
            assemble8(sm, e, wv);
            sink.chunk(u * R + rr, c, lane, wv);
        }
    }
    sink.finish(lane);
}

template <typename Sink>
__global__ void __launch_bounds__(256) k_nib_expand(const NibView w, int C, int64_t row0, int64_t nrows, const Sink sink_in) {
    Sink sink = sink_in;
    const int64_t K = (int64_t) C * CHUNK;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t r = (int64_t) blockIdx.x * 8 + warp; r < nrows; r += (int64_t) gridDim.x * 8) {
        const int64_t gr = row0 + r;
        const uint4 L = __ldg(w.row_lut + gr);
        for (int c = 0; c < C; c++) {
            const uint4 sm = __ldg((const uint4 *) (w.plane + gr * K + (int64_t) c * CHUNK) + lane);
            const uint2 cd = __ldg((const uint2 *) (w.codes + gr * (K / 2) + (int64_t) c * 256) + lane);
            uint32_t wv[8];
            nib_assemble8(sm, cd, L, wv);
            sink.chunk(r, c, lane, wv);
        }
        __syncwarp();
        for (uint32_t i = __ldg(w.esc_off + gr) + lane; i < __ldg(w.esc_off + gr + 1); i += 32) {
            const uint32_t rec = __ldg(w.esc + i);
            sink.one(r, rec & 0xFFF, esc_bits(rec));
        }
    }
    sink.finish(lane);
}

// gather: dst[i] = W[row0 + ids[i]], FP32 or BF16. A Huffman-coded row is reached by decoding its unit from the start.
template <bool BF>
__global__ void __launch_bounds__(256) k_pair_rows(const PairView w, int C, int R, const char * ids, int64_t ids_s0, int64_t n,
                                                    int64_t row0, char * dst, int64_t dst_s1) {
    __shared__ uint32_t lut[HP_MAX_PAIRS];
    stage_lut(lut, w.lut, HP_MAX_PAIRS);
    __syncthreads();
    const int64_t K = (int64_t) C * CHUNK;
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) { return; }
    const int64_t gr = row0 + *(const int32_t *) (ids + i * ids_s0);
    const int64_t gu = gr / R;
    PairReader rd;
    rd.open(w, gu, lane);
    for (int64_t r = gu * R; r <= gr; r++) {
        for (int c = 0; c < C; c++) {
            uint32_t e[8];
            rd.take8(lut, e);
            if (r == gr) {
                uint32_t wv[8];
                assemble8(ld_stream16(w.plane + r * K + (int64_t) c * CHUNK + 16 * lane), e, wv);
                put_row_chunk<BF>(dst + i * dst_s1, c, lane, wv);
            }
        }
    }
}

// The same gather for few rows (a draft step's candidates, the tokens of a decode batch), where the time is one warp's
// chain of table lookups from the start of its unit: up to R - 1 rows only to find where the wanted one begins. The unit's
// streams come into shared memory with one bulk copy, and the rows before the wanted one are passed over with a second
// table that gives, for 12 bits of stream, the codes that end in them (up to three, two for most) and their length: each
// lane passes over its own codes, the lanes need not stay in step before the row is read.
constexpr int ROWS_THREADS = 256;
template <bool BF>
__global__ void __launch_bounds__(ROWS_THREADS) k_pair_rows_staged(const PairView w, const AuxHeader * hdr, int C, int R, const char * ids,
                                                                   int64_t ids_s0, int64_t n, int64_t row0, char * dst, int64_t dst_s1, int rows_per_block,
                                                                   uint32_t cap, const Opaque k) {
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem;                              // code table | codes and bits per 12 bits | one barrier per row | streams
    uint16_t * many = (uint16_t *) (smem + 4 * HP_MAX_PAIRS);
    uint64_t * bars = (uint64_t *) (smem + 6 * HP_MAX_PAIRS);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char * buf = smem + 6 * HP_MAX_PAIRS + 128 + (size_t) warp * cap;
    const uint32_t bar = smem_u32(bars + warp);
    const bool reads = warp < rows_per_block;
    if (reads && lane == 0) { mbar_init(bar, 1); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    stage_lut(lut, w.lut, HP_MAX_PAIRS);
    __syncthreads();
    for (int i = threadIdx.x; i < HP_MAX_PAIRS; i += ROWS_THREADS) { many[i] = (uint16_t) codes_in_window(lut, (uint32_t) i); }
    grid_dependency_wait(); // the row ids may come from the kernel before this one; everything above is the matrix's own
    const int64_t i = (int64_t) blockIdx.x * rows_per_block + warp;
    const bool live = reads && i < n;
    int64_t gr = 0, gu = 0;
    uint32_t first = 0, bytes = 0;
    if (live) {
        gr = row0 + *(const volatile int32_t *) (ids + i * ids_s0);
        gu = gr / R;
        const uint32_t w0 = __ldg(w.ubase + gu), w1 = gu + 1 < (int64_t) hdr->n_a ? __ldg(w.ubase + gu + 1) : (uint32_t) hdr->n_b;
        const uint32_t start = w0 & ~3u;
        bytes = ((w1 - start + 4u + 3u) & ~3u) * 4u;
        if (bytes <= cap && lane == 0) {
            mbar_expect_tx(bar, bytes);
            bulk_g2s(smem_u32(buf), w.stream + start, bytes, bar);
        }
        first = 4u * (w0 - start + __ldg(w.lrel + gu * 32 + lane));
    }
    __syncthreads(); // `many` is complete
    if (!live) { return; }
    const int64_t K = (int64_t) C * CHUNK;
    const uint8_t * pl = w.plane + gr * K + 16 * lane;
    char * o = dst + i * dst_s1;
    auto row = [&](auto & rd, uint32_t lut_arg) {
        for (int c = 0; c < C; c++) {
            uint32_t e[8], wv[8];
            rd.take8(lut_arg, k, e);
            assemble8(ld_stream16(pl + (int64_t) c * CHUNK), e, wv);
            put_row_chunk<BF>(o, c, lane, wv);
        }
    };
    if (bytes <= cap) {
        const uint32_t landed = mbar_wait(bar, 0u);
        if (!landed) { // the copy never arrived: the flag reports it and the row becomes NaN
            if (lane == 0) { atomicOr(&g_wait_expired, 1u); }
            const uint32_t nan[8] = {0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u};
            for (int c = 0; c < C; c++) { put_row_chunk<BF>(o, c, lane, nan); }
            return;
        }
        WindowReader rd;
        rd.open(smem_u32(buf) + first, landed);
        rd.skip((int) (gr - gu * R) * C * 8, smem_u32(many), smem_u32(lut), k);
        row(rd, smem_u32(lut));
    } else { // more than 3 bits per weight: straight from global memory
        GlobalReader rd;
        rd.lut = lut;
        rd.rd.open(w, gu, lane);
        uint32_t e[8];
        for (int c = 0; c < (int) (gr - gu * R) * C; c++) { rd.take8(0u, k, e); }
        row(rd, 0u);
    }
}

template <bool BF>
__global__ void __launch_bounds__(256) k_nib_rows(const NibView w, int C, const char * ids, int64_t ids_s0, int64_t n, int64_t row0,
                                                   char * dst, int64_t dst_s1) {
    const int64_t K = (int64_t) C * CHUNK;
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) { return; }
    const int64_t gr = row0 + *(const int32_t *) (ids + i * ids_s0);
    char * o = dst + i * dst_s1;
    const uint4 L = __ldg(w.row_lut + gr);
    for (int c = 0; c < C; c++) {
        const uint4 sm = __ldg((const uint4 *) (w.plane + gr * K + (int64_t) c * CHUNK) + lane);
        const uint2 cd = __ldg((const uint2 *) (w.codes + gr * (K / 2) + (int64_t) c * 256) + lane);
        uint32_t wv[8];
        nib_assemble8(sm, cd, L, wv);
        put_row_chunk<BF>(o, c, lane, wv);
    }
    __syncwarp();
    for (uint32_t k = __ldg(w.esc_off + gr) + lane; k < __ldg(w.esc_off + gr + 1); k += 32) {
        const uint32_t rec = __ldg(w.esc + k);
        if (BF) { ((uint16_t *) o)[rec & 0xFFF] = (uint16_t) esc_bits(rec); }
        else { ((float *) o)[rec & 0xFFF] = __uint_as_float(esc_bits(rec) << 16); }
    }
}

// ---------------------------------------------------------------- views and geometry

// warps per block and blocks for `units` warp-sized work items per column: spread few units over all SMs with small
// blocks, fill the machine with 16-warp blocks otherwise
void unit_geometry(int64_t units, int ncols, int max_warps, dim3 & grid, int & threads) {
    const int64_t sms = device_info().sms;
    const int64_t per_col = std::max<int64_t>(1, sms / std::max(1, ncols));
    const int64_t wpb = std::min<int64_t>(std::max<int64_t>((units + per_col - 1) / per_col, 2), max_warps);
    threads = (int) wpb * 32;
    grid = dim3((unsigned) std::max<int64_t>(1, std::min<int64_t>((units + wpb - 1) / wpb, per_col)), (unsigned) ncols);
}

dim3 row_geometry(int64_t work, int ncols) { // 8 warps per block, one work item per warp
    const int64_t cap = std::max<int64_t>(1, (int64_t) device_info().sms * 8 / std::min(ncols, 8));
    return dim3((unsigned) std::max<int64_t>(1, std::min<int64_t>((work + 7) / 8, cap)), (unsigned) ncols);
}

template <int C, typename TX, bool GLU>
void launch_nib_c(const NibView & g, const NibView & v, const Cols & p, int ncols, cudaStream_t st) {
    const dim3 grid = row_geometry(p.nrows, ncols);
    const bool few = p.nrows * ncols <= 3 * (int64_t) device_info().sms * nib_blocks(C, GLU) * 8; // rows against resident warps
    // spread evenly (even_smem): chains of products of 1024 x 2048, 2048 x 2048, 1024 x 4096, one column: 2.49 / 2.90 / 3.26 us a launch with blocks
    // crowded where the launch in front had ended, 1.75 / 2.29 / 2.31 so; two tokens through 24 layers of small matrices 227 and 201 us
    launch_chained(few ? k_nib_gemv<C, TX, GLU, true> : k_nib_gemv<C, TX, GLU, false>, grid, dim3(256), even_smem(0, (int64_t) grid.x * grid.y), st, g, v, p);
}
template <typename TX, bool GLU>
void launch_nib(const NibView & g, const NibView & v, const Cols & p, int64_t K, int ncols, cudaStream_t st) {
    switch (K / CHUNK) {
        case 1: launch_nib_c<1, TX, GLU>(g, v, p, ncols, st); break;
        case 2: launch_nib_c<2, TX, GLU>(g, v, p, ncols, st); break;
        case 4: launch_nib_c<4, TX, GLU>(g, v, p, ncols, st); break;
        case 8: launch_nib_c<8, TX, GLU>(g, v, p, ncols, st); break;
        default: fail_invalid("unsupported K");
    }
}

// Mid-size dense HUFPAIR matrices (256 units up to 4 per SM) with several columns: one staged decode per column over all
// SMs instead of the general kernel's shared decode, whose warps read their lane streams straight from global memory
// (4096 x 2048, R = 8: 29 -> 19 us at 4 tokens, 54 -> 33 us at 8; from 1024 units on the two forms are level).
static bool mid_size_by_column(const bf16n_weight & w, const bf16n_mmv_args & a, int64_t units) {
    if (units > (int64_t) device_info().sms * 4) { return false; }
    bf16n_mmv_args one = a;
    one.ncols = 1;
    return gemv_staged_applies(w, one);
}

template <typename TX>
void launch_gemv(const bf16n_weight & w, const bf16n_mmv_args & a, cudaStream_t st, bool multi_col, const bf16n_peer_out * peers, const uint16_t * marks) {
    const Cols p = make_cols(a, peers);
    if (peers && peers->n_peers > 0) {
        require(w.format == FMT_HUFPAIR && !w.cm && !a.ids, "peer outputs need a dense row-major HUFPAIR product");
        multi_col = false; // one column per blockIdx.y: the kernels that fan out
    }
    const int C = (int) (w.K / CHUNK);
    if (w.format == FMT_HUFPAIR) {
        const int64_t units = a.nrows / w.R;
        dim3 grid; int threads;
        if (w.cm) {
            unit_geometry(units, a.ncols, 16, grid, threads);
            const size_t shm = 4 * HP_MAX_PAIRS + w.K * 4;
#define CM(CC, RR) case CC * 100 + RR: k_pair_gemv_cm<CC, RR, TX><<<grid, threads, shm, st>>>(pair_view(w), p); break;
            switch (C * 100 + w.R) {
                CM(2, 4) CM(2, 8) CM(2, 16) CM(4, 4) CM(4, 8) CM(4, 16) CM(8, 4) CM(8, 8) CM(8, 16)
                default: fail_invalid("unsupported chunk-major K/R");
            }
#undef CM
        } else if (gemv_rings_enabled() && gemv_rings_applies(w, a)) {
            gemv_rings(w, a, st, multi_col, peers, marks); // large matrices, BF16 activations: 1, 2 or 4 columns per decode
            return;
        } else if (!a.ids && a.ncols > 1 && multi_col && !mid_size_by_column(w, a, units)) {
            unit_geometry(units, 1, 16, grid, threads);
            for (int c0 = 0; c0 < a.ncols; c0 += 4) {
                const int nc = std::min(4, a.ncols - c0);
                Cols q = p;
                q.x += c0 * p.x_tok;
                q.y += c0 * p.y_tok;
                const size_t shm = 4 * HP_MAX_PAIRS + (size_t) nc * w.K * 4;
#define MC(CC, NN) case CC * 10 + NN: k_pair_gemv<CC, NN, TX, false><<<grid, threads, shm, st>>>(pair_view(w), w.R, q); break;
                switch (C * 10 + nc) {
                    MC(1, 1) MC(1, 2) MC(1, 3) MC(1, 4) MC(2, 1) MC(2, 2) MC(2, 3) MC(2, 4)
                    MC(4, 1) MC(4, 2) MC(4, 3) MC(4, 4) MC(8, 1) MC(8, 2) MC(8, 3) MC(8, 4)
                    default: fail_invalid("unsupported K");
                }
#undef MC
            }
        } else if (gemv_staged_applies(w, a) || (!a.ids && a.ncols > 1 && mid_size_by_column(w, a, units))) {
            gemv_staged(w, a, st, peers);
            return;
        } else {
            unit_geometry(units, a.ncols, 16, grid, threads);
            const size_t shm = 4 * HP_MAX_PAIRS + w.K * 4;
            if (p.peers.n) {
                switch (C) {
                    case 1: k_pair_gemv<1, 1, TX, true, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 2: k_pair_gemv<2, 1, TX, true, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 4: k_pair_gemv<4, 1, TX, true, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 8: k_pair_gemv<8, 1, TX, false, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    default: fail_invalid("unsupported K");
                }
            } else {
                switch (C) {
                    case 1: k_pair_gemv<1, 1, TX, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 2: k_pair_gemv<2, 1, TX, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 4: k_pair_gemv<4, 1, TX, true><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    case 8: k_pair_gemv<8, 1, TX, false><<<grid, threads, shm, st>>>(pair_view(w), w.R, p); break;
                    default: fail_invalid("unsupported K");
                }
            }
        }
    } else if (w.format == FMT_NIBBLE) {
        launch_nib<TX, false>(nib_view(w), nib_view(w), p, w.K, a.ncols, st);
    } else {
        const dim3 grid = row_geometry(a.nrows / w.R, a.ncols);
        const size_t shm = (4u << HUF_LMAX) + w.K * 4;
        k_huf_gemv<TX, false><<<grid, 256, shm, st>>>(huf_view(w), huf_view(w), C, w.R, p);
    }
    check_launch();
}

template <typename TX>
void launch_glu(const bf16n_weight & g, const NibView * up_nib, const bf16n_weight * u, const bf16n_mmv_args & a, cudaStream_t st) {
    const Cols p = make_cols(a);
    const int C = (int) (g.K / CHUNK);
    if (g.format == FMT_NIBBLE) {
        launch_nib<TX, true>(nib_view(g), up_nib ? *up_nib : nib_view(*u), p, g.K, a.ncols, st);
    } else if (g.format == FMT_HUFPAIR) {
        dim3 grid; int threads;
        unit_geometry(a.nrows / g.R, a.ncols, 16, grid, threads);
        const size_t shm = 8 * HP_MAX_PAIRS + g.K * 4;
        switch (C) {
            case 1: k_pair_glu<1, TX><<<grid, threads, shm, st>>>(pair_view(g), pair_view(*u), g.R, p); break;
            case 2: k_pair_glu<2, TX><<<grid, threads, shm, st>>>(pair_view(g), pair_view(*u), g.R, p); break;
            case 4: k_pair_glu<4, TX><<<grid, threads, shm, st>>>(pair_view(g), pair_view(*u), g.R, p); break;
            case 8: k_pair_glu<8, TX><<<grid, threads, shm, st>>>(pair_view(g), pair_view(*u), g.R, p); break;
            default: fail_invalid("unsupported K");
        }
    } else {
        const dim3 grid = row_geometry(a.nrows / g.R, a.ncols);
        const size_t shm = (8u << HUF_LMAX) + g.K * 4;
        k_huf_gemv<TX, true><<<grid, 256, shm, st>>>(huf_view(g), huf_view(*u), C, g.R, p);
    }
    check_launch();
}

template <typename Sink>
void launch_expand(const bf16n_weight & w, int64_t row0, int64_t nrows, const Sink & sink, cudaStream_t st) {
    const int C = (int) (w.K / CHUNK);
    const int64_t work = w.format == FMT_NIBBLE ? nrows : nrows / w.R;
    const unsigned gx = (unsigned) std::max<int64_t>(1, std::min<int64_t>((work + 7) / 8, (int64_t) device_info().sms * 16));
    if (w.format == FMT_NIBBLE) {
        k_nib_expand<Sink><<<gx, 256, 0, st>>>(nib_view(w), C, row0, nrows, sink);
    } else if (expand_rows_applies(w, nrows)) {
        expand_rows(w, row0, nrows, sink, st);
    } else if (w.format == FMT_HUFPAIR) { // short units, or fewer than four steps of 512 weights to one
        k_pair_expand<Sink><<<gx, 256, 0, st>>>(pair_view(w), C, w.R, w.cm != 0, row0, nrows, sink);
    } else {
        k_huf_expand<Sink><<<gx, 256, 0, st>>>(huf_view(w), C, w.R, row0, nrows, sink);
    }
    check_launch();
}

} // namespace

// ---------------------------------------------------------------- entry points used by the C ABI (capi.cu)

BF16N_DEFINE_FAULT_WORD(row_gather_fault_word)

static void gemv_group_init();
void gemv_init() {
    const int optin = device_info().smem_optin;
#define ATTR(KERNEL, BYTES) allow_dynamic_smem((const void *) KERNEL, (int) (BYTES), optin, #KERNEL)
#define MC_ATTR(TX, CC) \
    ATTR((k_pair_gemv<CC, 1, TX, false>), 4 * HP_MAX_PAIRS + 1 * CC * CHUNK * 4); ATTR((k_pair_gemv<CC, 2, TX, false>), 4 * HP_MAX_PAIRS + 2 * CC * CHUNK * 4); \
    ATTR((k_pair_gemv<CC, 3, TX, false>), 4 * HP_MAX_PAIRS + 3 * CC * CHUNK * 4); ATTR((k_pair_gemv<CC, 4, TX, false>), 4 * HP_MAX_PAIRS + 4 * CC * CHUNK * 4);
    MC_ATTR(float, 1) MC_ATTR(float, 2) MC_ATTR(float, 4) MC_ATTR(float, 8)
    MC_ATTR(bf16, 1) MC_ATTR(bf16, 2) MC_ATTR(bf16, 4) MC_ATTR(bf16, 8)
#undef MC_ATTR
    ATTR((k_pair_glu<8, float>), 8 * HP_MAX_PAIRS + 8 * CHUNK * 4);
    ATTR((k_pair_glu<8, bf16>), 8 * HP_MAX_PAIRS + 8 * CHUNK * 4);
    ATTR((k_pair_glu<4, float>), 8 * HP_MAX_PAIRS + 4 * CHUNK * 4);
    ATTR((k_pair_glu<4, bf16>), 8 * HP_MAX_PAIRS + 4 * CHUNK * 4);
    ATTR(k_pair_rows_staged<true>, 6 * HP_MAX_PAIRS + 128 + 2 * (16 * K_MAX * 3 / 8 + 80));
    ATTR(k_pair_rows_staged<false>, 6 * HP_MAX_PAIRS + 128 + 2 * (16 * K_MAX * 3 / 8 + 80));
#undef ATTR
#define NIB_ATTR(C, TX, GLU) allow_dynamic_smem((const void *) k_nib_gemv<C, TX, GLU, true>, optin, optin, "nib"); allow_dynamic_smem((const void *) k_nib_gemv<C, TX, GLU, false>, optin, optin, "nib");
#define NIB_ATTR_C(C) NIB_ATTR(C, float, false) NIB_ATTR(C, bf16, false) NIB_ATTR(C, float, true) NIB_ATTR(C, bf16, true)
    NIB_ATTR_C(1) NIB_ATTR_C(2) NIB_ATTR_C(4) NIB_ATTR_C(8)
#undef NIB_ATTR_C
#undef NIB_ATTR
    gemv_group_init();
    expand_rows_init();
    gemv_staged_init();
    gemv_rings_init();
    gemv_parts_init();
}

void gemv(const bf16n_weight & w, const bf16n_mmv_args & a, cudaStream_t st, bool multi_col, const bf16n_peer_out * peers, const uint16_t * marks) {
    if (!(peers && peers->n_peers > 0) && (multi_col || a.ncols == 1) && gemv_parts_applies(w, marks, a)) { gemv_parts(w, marks, a, st); return; }
    if (a.x_bf16) { launch_gemv<bf16>(w, a, st, multi_col, peers, marks); } else { launch_gemv<float>(w, a, st, multi_col, peers, marks); }
}

// ---------------------------------------------------------------- several independent small products in one launch

namespace {

constexpr int GROUP_MAX = 8;
struct NibItem { // one dense NIBBLE product of a group
    NibView v;
    const char * x; char * y;
    int64_t x_tok, y_tok, row0, nrows;
    int ncols, chunks, first_block, blocks; // `blocks` blocks from first_block on serve each column
    bool x_bf16, y_bf16;
};
struct NibGroup { int n; NibItem item[GROUP_MAX]; };

template <int C, bool AHEAD, typename TX>
__device__ __forceinline__ void nib_item_rows(const NibItem & it, int block, int col) {
    const TX * xg = (const TX *) (it.x + col * it.x_tok);
    const OutVec out = {it.y + col * it.y_tok, it.y_bf16};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NibView * w[1] = {&it.v};
    bool waited = false;
    for (int64_t r = (int64_t) block * 8 + warp; r < it.nrows; r += (int64_t) it.blocks * 8) {
        float s[1];
        nib_rows<C, AHEAD, 1, TX>(w, it.row0 + r, xg, lane, waited, s); // weights first, then the activations an earlier kernel may have written
        if (lane == 0) { out.put(r, s[0]); }
    }
    if (!waited) { grid_dependency_wait(); }
}

// Every block belongs to one item of the group (a prefix table of block ranges); within its item it is a block of the
// single-product kernel: same loads, same order of operations, so the results are the same bits. Three blocks fit an SM, and the
// 352 blocks of a layer's three products are resident at once (two left a second wave). WIDE adds rows of 4096 columns and
// decodes every item as it multiplies: ahead, such a row's registers left one block per SM (three products of 2048 x 4096: 13.2
// against 10.8 us).
template <bool WIDE>
__global__ void __launch_bounds__(256, WIDE ? 0 : 3) k_nib_gemv_group(const NibGroup g) {
    if (!WIDE) { grid_launch_dependents(); } // as in k_nib_gemv
    int m = 0;
    while (m + 1 < g.n && (int) blockIdx.x >= g.item[m + 1].first_block) { m++; }
    const NibItem & it = g.item[m];
    const int local = (int) blockIdx.x - it.first_block, col = local / it.blocks, block = local % it.blocks;
    switch (it.chunks * 2 + (it.x_bf16 ? 1 : 0)) {
        case 2: nib_item_rows<1, !WIDE, float>(it, block, col); break;
        case 3: nib_item_rows<1, !WIDE, bf16>(it, block, col); break;
        case 4: nib_item_rows<2, !WIDE, float>(it, block, col); break;
        case 5: nib_item_rows<2, !WIDE, bf16>(it, block, col); break;
        case 8: nib_item_rows<4, !WIDE, float>(it, block, col); break;
        case 9: nib_item_rows<4, !WIDE, bf16>(it, block, col); break;
        case 16: if constexpr (WIDE) { nib_item_rows<8, false, float>(it, block, col); } break;
        case 17: if constexpr (WIDE) { nib_item_rows<8, false, bf16>(it, block, col); } break;
        default: grid_dependency_wait(); break;
    }
}

} // namespace

static void gemv_group_init() {
    allow_dynamic_smem((const void *) k_nib_gemv_group<false>, device_info().smem_optin, device_info().smem_optin, "nib group");
    allow_dynamic_smem((const void *) k_nib_gemv_group<true>, device_info().smem_optin, device_info().smem_optin, "nib group");
}

// dense NIBBLE products of up to 8 columns can share a grid
bool gemv_groupable(const bf16n_weight & w, const bf16n_mmv_args & a) {
    const int C = (int) (w.K / CHUNK);
    return w.format == FMT_NIBBLE && !a.ids && a.nrows > 0 && a.ncols >= 1 && a.ncols <= 8 && (C == 1 || C == 2 || C == 4 || C == 8);
}

// n independent groupable products (different matrices, activations and outputs) on one stream: one grid per eight.
void gemv_group(const bf16n_weight * w, const bf16n_mmv_args * a, int n, cudaStream_t st) {
    int i = 0;
    while (i < n) {
        NibGroup g = {};
        int blocks = 0;
        bool wide = false, one_chunk = true;
        while (i < n && g.n < GROUP_MAX) {
            NibItem & it = g.item[g.n++];
            it.v = nib_view(w[i]);
            it.x = (const char *) a[i].x; it.y = (char *) a[i].y;
            it.x_tok = a[i].x_tok; it.y_tok = a[i].y_tok; it.row0 = a[i].row0; it.nrows = a[i].nrows;
            it.ncols = a[i].ncols; it.chunks = (int) (w[i].K / CHUNK);
            it.x_bf16 = a[i].x_bf16 != 0; it.y_bf16 = a[i].y_bf16 != 0;
            const dim3 geo = row_geometry(a[i].nrows, a[i].ncols);
            it.first_block = blocks;
            wide = wide || it.chunks > 4;
            one_chunk = one_chunk && it.chunks == 1;
            it.blocks = (int) geo.x;
            blocks += it.blocks * it.ncols;
            i++;
        }
        // Spread evenly (even_smem) unless all rows are of 512 columns, whose blocks are gone before crowding tells: crowded / spread, groups of
        // eight of 64 x 512, two tokens, 1.28 / 1.64 us, of four of 256 x 512, one token, 1.35 / 1.47; of four of 256 x 2048 2.57 / 1.98.
        launch_chained(wide ? k_nib_gemv_group<true> : k_nib_gemv_group<false>, dim3((unsigned) blocks), dim3(256), one_chunk ? 0 : even_smem(0, blocks), st, g);
        check_launch();
    }
}

void gemv_glu_merged(const bf16n_weight & w, const bf16n_mmv_args & a, cudaStream_t st) {
    const NibView up = nib_view(w, a.nrows);
    if (a.x_bf16) { launch_glu<bf16>(w, &up, nullptr, a, st); } else { launch_glu<float>(w, &up, nullptr, a, st); }
}

void gemv_glu(const bf16n_weight & g, const bf16n_weight & u, const bf16n_mmv_args & a, cudaStream_t st) {
    if (a.x_bf16) { launch_glu<bf16>(g, nullptr, &u, a, st); } else { launch_glu<float>(g, nullptr, &u, a, st); }
}

void expand_store(const bf16n_weight & w, int64_t row0, int64_t nrows, uint16_t * out, cudaStream_t st, const uint16_t * marks) {
    if (expand_parts_applies(w, marks, nrows)) { expand_parts(w, marks, row0, nrows, StoreBF16{out, w.K}, st); return; }
    launch_expand(w, row0, nrows, StoreBF16{out, w.K}, st);
}

void expand_compare(const bf16n_weight & w, int64_t row0, int64_t nrows, const uint16_t * src, unsigned long long * total,
                    cudaStream_t st) {
    launch_expand(w, row0, nrows, CompareBF16{src, w.K, total, 0u}, st);
}

void gather_rows(const bf16n_weight & w, const void * ids, int64_t ids_s0, int64_t n, void * dst, bool dst_bf16, int64_t dst_s1,
                 int64_t row0, cudaStream_t st, bool behind_own, const uint16_t * marks) {
    if (rows_parts_applies(w, marks, n)) {
        rows_parts(w, marks, ids, ids_s0, n, dst, dst_bf16, dst_s1, row0, nullptr, st, behind_own);
        return;
    }
    const int C = (int) (w.K / CHUNK);
    const unsigned gx = (unsigned) ((n + 7) / 8);
    const char * ip = (const char *) ids;
    char * dp = (char *) dst;
    if (w.format == FMT_NIBBLE) {
        if (dst_bf16) { k_nib_rows<true><<<gx, 256, 0, st>>>(nib_view(w), C, ip, ids_s0, n, row0, dp, dst_s1); }
        else { k_nib_rows<false><<<gx, 256, 0, st>>>(nib_view(w), C, ip, ids_s0, n, row0, dp, dst_s1); }
    } else if (n <= (int64_t) device_info().sms * 4 && w.R * C >= 32) {
        // Few rows: spread over the SMs, at most two to a block (k_pair_rows: eight). Units of fewer than 32 chunks have little to
        // pass over, and the skip table costs more than it saves. General / staged in us, 64 rows: R * C = 1: 2.9 / 6.0,
        // 4: 4.1 / 6.8, 8: 6.2 / 8.0, 16: 10.3 / 9.5 (256 rows: 10.5 / 11.4), 32: 19.4 / 13.3.
        const int per = n > device_info().sms * 2 ? 2 : 1;
        const uint32_t cap = (uint32_t) ((w.R * w.K * 3 / 8 + 64 + 15) & ~15ll);
        const size_t shm = 6 * HP_MAX_PAIRS + 128 + (size_t) per * cap;
        const Opaque k = {1u, 4u};
        launch_behind(behind_own, dst_bf16 ? k_pair_rows_staged<true> : k_pair_rows_staged<false>, dim3((unsigned) ((n + per - 1) / per)), dim3(ROWS_THREADS),
                      shm, st, pair_view(w), (const AuxHeader *) w.aux, C, w.R, ip, ids_s0, n, row0, dp, dst_s1, per, cap, k);
    } else {
        if (dst_bf16) { k_pair_rows<true><<<gx, 256, 0, st>>>(pair_view(w), C, w.R, ip, ids_s0, n, row0, dp, dst_s1); }
        else { k_pair_rows<false><<<gx, 256, 0, st>>>(pair_view(w), C, w.R, ip, ids_s0, n, row0, dp, dst_s1); }
    }
    check_launch();
}

} // namespace b16
