// Building blocks of the kernels that stage a unit's exponent streams in shared memory with one bulk async copy:
// mbarrier / bulk-copy wrappers with bounded waits, the lane-stream reader over staged words, the lane's activations
// in registers. See gemv_staged.cu for the design notes.
#pragma once

#include "decode.cuh"

namespace b16 {
namespace dev {

using bf16 = __nv_bfloat16;

// Set when a bounded mbarrier wait ran out (one copy per translation unit; bf16n_fault_status reads and clears them).
// The outputs of the work item whose wait expired are written as NaN.
static __device__ unsigned int g_wait_expired;
// defines `unsigned int * NAME()`: the device address of this translation unit's word (device current, outside capture)
#define BF16N_DEFINE_FAULT_WORD(NAME)                                                           \
    unsigned int * NAME() {                                                                     \
        unsigned int * p = nullptr;                                                             \
        cuda_ok(cudaGetSymbolAddress((void **) &p, dev::g_wait_expired), "fault word address"); \
        return p;                                                                               \
    }

constexpr uint32_t WAIT_LIMIT = 1u << 20; // try_wait polls before a warp gives up on its bulk copy

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// returns 1 when the phase completed (the value doubles as the token staged reads depend on), 0 when the wait ran out
__device__ __forceinline__ uint32_t mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) { return done; }
    }
    return 0;
}
// global -> shared bulk copy; dst/src 16-byte aligned, bytes a multiple of 16; completes on the mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void * src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void prefetch_l2(const void * p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void bulk_prefetch_l2(const void * src, uint32_t bytes) { // 16-byte aligned, multiple of 16
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint32_t shl_wrap_hi(uint32_t lo, uint32_t hi, uint32_t n) { // high word of {hi:lo} << (n & 31)
    uint32_t d;
    asm("shf.l.wrap.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(lo), "r"(hi), "r"(n));
    return d;
}

// Integer constants the compiler must not see through: passed as kernel arguments so that "a * k + b" stays an integer
// multiply-add. On sm_100a shifts, logic ops and byte permutes issue at half rate on one pipe and integer multiply-adds
// at half rate on another; the decoder is bound by the first, so every add that can be phrased as a multiply-add by one
// of these constants runs on the second instead.
struct Opaque { uint32_t one, four; };

__device__ __forceinline__ uint32_t imad(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// `token` is produced by the mbarrier wait of the bulk copy whose bytes are read: the data dependency keeps a read of
// staged stream words after that wait (table reads pass 0: the table is complete before the block barrier).
__device__ __forceinline__ uint32_t lds32(uint32_t addr, uint32_t token = 0) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr), "r"(token));
    return v;
}

// The code table without bank conflicts. Codes are canonical, so the long ones are the numerically largest: a view of 12 bits that
// starts with a code of at most 8 bits needs its first 8 bits only, and the entries are q (those views by 8 bits) and 4096 - 16 q (the
// others by all 12); on the weights of the benchmark 466 instead of 4096. So many fit a copy for every lane (or every second one,
// and so on for flatter tables), and lanes that share no copy cannot collide. Entry of a view: max(view >> 8, view - 15 q).
constexpr int SPREAD_BYTES = 64 << 10;
struct SpreadTable {
    uint32_t base, stride; // address of this lane's copy of entry 0, bytes from entry to entry
    int32_t shift;         // -15 q
    __device__ __forceinline__ uint32_t look(uint32_t view) const { // view: the stream from the code on, at the top
        return lds32(imad((uint32_t) __viaddmax_s32((int32_t) (view >> (32 - HP_LMAX)), shift, (int32_t) (view >> 24)), stride, base));
    }
};
// Every thread of the block; the caller's next block barrier completes the table. Whatever the table holds, entries stay below
// SPREAD_BYTES: the largest view is entry 4095 - 15 q of 4096 - 15 q.
__device__ __forceinline__ SpreadTable stage_spread(unsigned char * table, const uint32_t * lut) {
    constexpr int SHORT = HP_MAX_PAIRS / 16;
    __shared__ int first_long;
    if (threadIdx.x == 0) { first_long = SHORT; }
    __syncthreads();
    for (int i = threadIdx.x; i < SHORT; i += blockDim.x) {
        if ((__ldg(lut + 16 * i) & 31u) > 8u) { atomicMin(&first_long, i); }
    }
    __syncthreads();
    int q = first_long, entries = HP_MAX_PAIRS - 15 * q;
    const int log_copies = entries <= SPREAD_BYTES / 128 ? 5 : entries <= SPREAD_BYTES / 64 ? 4 : entries <= SPREAD_BYTES / 32 ? 3 : 2;
    if (log_copies == 2) { q = 0; entries = HP_MAX_PAIRS; }
    for (int i = threadIdx.x; i < entries << (log_copies - 2); i += blockDim.x) {
        const int at = i >> (log_copies - 2);
        const uint32_t e = __ldg(lut + (at < q ? 16 * at : at + 15 * q));
        ((uint4 *) table)[i] = make_uint4(e, e, e, e);
    }
    return {smem_u32(table) + (threadIdx.x & ((1u << log_copies) - 1u)) * 4u, 4u << log_copies, -15 * q};
}

// Lane stream reader over words in shared memory (addresses are 32-bit shared-window addresses). The stream is seen through
// a window of three consecutive words and a bit offset, as in rings.cuh: a view is one funnel shift and nothing is shifted
// per code. Against a 64-bit buffer that is shifted and refilled (its predecessor here) the chain of a code is two
// instructions shorter: 238 -> 222 us for eight one-token steps of 256 routed experts (212 with the slide predicated, below),
// 287 -> 264 us for four four-token steps of 128, 71 -> 62 us for FP32 activations on 62080 x 2048.
struct WindowReader {
    uint32_t next, hi, lo, ahead, o, token;

    __device__ __forceinline__ void open(uint32_t addr, uint32_t wait_token) {
        token = wait_token;
        hi = lds32(addr, token); lo = lds32(addr + 4, token); ahead = lds32(addr + 8, token); next = addr + 12; o = 0;
    }
    // the same at bit `bit` (0..31) of the word at `addr`; position(): bits from the word at `start` to the next code
    __device__ __forceinline__ void open_at(uint32_t addr, uint32_t bit, uint32_t wait_token) { open(addr, wait_token); o = bit; }
    __device__ __forceinline__ uint32_t position(uint32_t start) const { return (next - 12u - start) * 8u + (o & 31u); }
    // at most one word on; predicated, so that lookups and products are scheduled across it (a branch: 223 against 212 us for
    // the eight one-token steps above)
    __device__ __forceinline__ void slide(uint32_t o2, const Opaque & k) {
        asm("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\txor.b32 t, %5, %6;\n\tand.b32 t, t, 32;\n\tsetp.ne.u32 p, t, 0;\n\t"
            "@p mov.u32 %0, %1;\n\t@p mov.u32 %1, %2;\n\t@p ld.shared.u32 %2, [%3];\n\t@p mad.lo.u32 %3, %7, %8, %3;\n\t}"
            : "+r"(hi), "+r"(lo), "+r"(ahead), "+r"(next) : "r"(token), "r"(o), "r"(o2), "r"(k.four), "r"(k.one));
        o = o2;
    }
    __device__ __forceinline__ void take8(uint32_t lut, const Opaque & k, uint32_t (&e)[8]) {
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
            const uint32_t v1 = shl_wrap_hi(lo, hi, o); // 32 bits from the offset on: two codes are at most 24
            e[q] = lds32(imad(v1 >> (32 - HP_LMAX), k.four, lut));
            const uint32_t v2 = shl_wrap_hi(0u, v1, e[q]);
            e[q + 1] = lds32(imad(v2 >> (32 - HP_LMAX), k.four, lut));
            slide(o + e[q] + e[q + 1], k);
        }
    }
    __device__ __forceinline__ void take8(const SpreadTable & t, const Opaque & k, uint32_t (&e)[8]) {
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
            const uint32_t v1 = shl_wrap_hi(lo, hi, o);
            e[q] = t.look(v1);
            e[q + 1] = t.look(shl_wrap_hi(0u, v1, e[q]));
            slide(o + e[q] + e[q + 1], k);
        }
    }
    // passes over `n` codes; many: 16-bit entries of codes_in_window (format.h): each names one to three codes, so this ends
    __device__ __forceinline__ void skip(int n, uint32_t many, uint32_t lut, const Opaque & k) {
        while (n >= 3) {
            uint32_t m;
            asm("ld.shared.u16 %0, [%1];" : "=r"(m) : "r"(many + 2 * (shl_wrap_hi(lo, hi, o) >> (32 - HP_LMAX))));
            n -= (int) (m >> 8);
            slide(o + (m & 31u), k);
        }
        for (; n > 0; n--) { slide(o + lds32(imad(shl_wrap_hi(lo, hi, o) >> (32 - HP_LMAX), k.four, lut)), k); }
    }
};

// the same interface over the general reader (streams in global memory, table through a generic pointer)
struct GlobalReader {
    PairReader rd;
    const uint32_t * lut;
    template <typename Table> __device__ __forceinline__ void take8(const Table &, const Opaque &, uint32_t (&e)[8]) { rd.take8(lut, e); }
};

// this lane's activations of a K-column row, in registers
template <int C, typename TX> struct LaneX;
template <int C> struct LaneX<C, float> {
    float4 q[C * 4];
    __device__ __forceinline__ void load(const float * x, int lane) {
#pragma unroll
        for (int i = 0; i < C * 4; i++) { q[i] = ldg_x4(x, (i >> 2) * CHUNK + 128 * (i & 3) + 4 * lane); }
    }
    __device__ __forceinline__ void fma(int c, const uint32_t (&w)[8], float (&a)[4]) const {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            a[0] = fmaf(bf16lo_f32(w[2 * j]), q[c * 4 + j].x, a[0]);
            a[1] = fmaf(bf16hi_f32(w[2 * j]), q[c * 4 + j].y, a[1]);
            a[2] = fmaf(bf16lo_f32(w[2 * j + 1]), q[c * 4 + j].z, a[2]);
            a[3] = fmaf(bf16hi_f32(w[2 * j + 1]), q[c * 4 + j].w, a[3]);
        }
    }
};
template <int C> struct LaneX<C, bf16> {
    uint2 q[C * 4]; // two BF16 pairs per column quad
    __device__ __forceinline__ void load(const bf16 * x, int lane) {
#pragma unroll
        for (int i = 0; i < C * 4; i++) { q[i] = ld_act8(x + (i >> 2) * CHUNK + 128 * (i & 3) + 4 * lane); }
    }
    // acc += w.lo * x.lo ; acc2 += w.hi * x.hi with BF16 operands and FP32 accumulate
    static __device__ __forceinline__ void fma2(uint32_t w, uint32_t x, float & lo, float & hi) {
        asm("{ .reg .b16 wl, wh, xl, xh;\n\t"
            "mov.b32 {wl, wh}, %2;\n\t"
            "mov.b32 {xl, xh}, %3;\n\t"
            "fma.rn.f32.bf16 %0, wl, xl, %0;\n\t"
            "fma.rn.f32.bf16 %1, wh, xh, %1; }"
            : "+f"(lo), "+f"(hi) : "r"(w), "r"(x));
    }
    __device__ __forceinline__ void fma(int c, const uint32_t (&w)[8], float (&a)[4]) const {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            fma2(w[2 * j], q[c * 4 + j].x, a[0], a[1]);
            fma2(w[2 * j + 1], q[c * 4 + j].y, a[2], a[3]);
        }
    }
};

} // namespace dev
} // namespace b16
