// Units cut into parts: several warps walk one unit's lane streams at once.
//
// A lane's stream is serial by the format: where a code starts is known only when the code before it has been looked up, so
// a matrix of few units (8192 x 2048 at R = 16: 512) leaves the GPU waiting for chains of R K / 64 dependent lookups. Marks
// cut the chains: for every 64 codes of a lane, the bit of its stream at which the next 64 begin, taken down once when the
// matrix is loaded (2 bytes per lane and 64 codes, 1.2 % of the stored bytes).
//
// Marks are hints, never trusted: the warp of a part compares where its last code ended with the mark that the next part
// started from. If they agree in every lane of every part, each part started where the one before it ended, back to the
// unit's own start, so all of them are right; if one differs (a matrix overwritten since, marks that were never written) one
// warp decodes the whole unit again from its start, in global memory. A wrong mark therefore costs time and changes nothing.
// It reads inside the staged bytes too: a start is clamped to them and 64 codes move a reader by 32 words at most
// (WindowReader::slide), which PART_SLACK bytes behind every buffer allow for.
#pragma once

#include "staged.cuh"
#include "launch.h"

namespace b16 {
namespace dev {

constexpr int PART_STEPS = 8;                 // steps of 512 weights to a part: 64 codes of a lane
constexpr int PART_AHEAD = 4;                 // steps of plane bytes in registers
constexpr uint32_t PART_SLACK = 160;          // 32 words that a part can advance and the window's three

struct Parts {                                // the cut units of one matrix
    PairView w;
    const AuxHeader * hdr;
    const uint16_t * marks;                   // [unit][part 1 ..][lane]
    int parts;                                // parts of a unit: R K / 4096
    uint32_t cap;                             // bytes of streams that half of a unit's buffer holds: 3 bits a weight
    uint32_t whole;                           // and all of it: part_whole(cap)
};
// 6 bits a weight, the most that codes of HP_LMAX bits for two take, and what lanes and unit are rounded up by. From the host: worked out in
// the kernels it cost a decode step of one token 0.3 us.
constexpr uint32_t part_whole(uint32_t cap) { return 2 * cap + PART_SLACK; }

// shared memory of a block that walks `units` units at a time with `warps` warps: table | barriers | starts | a buffer of
// streams per unit (two halves in turn, or one of twice the size) | what the caller adds
struct PartSmem { uint32_t bars, starts, streams, end; };
__host__ __device__ inline PartSmem part_smem(int warps, int units, uint32_t cap) {
    PartSmem s;
    s.bars = 4 * HP_MAX_PAIRS;
    s.starts = s.bars + 16 * 8;
    s.streams = s.starts + 2 * warps * 128;
    s.end = s.streams + 2 * units * (cap + PART_SLACK);
    return s;
}
constexpr int PART_UNITS = 8;                 // units of a block at a time, at most

// Where one warp's part of a unit begins.
struct PartStart {
    uint32_t bytes;                           // of the unit's streams from their 16-byte boundary on
    uint32_t first, my, at;                   // stream word of that boundary; words from it to this lane's stream; this lane's mark
    __device__ __forceinline__ void load(const Parts & p, int64_t unit, int part, int lane) {
        const uint32_t w0 = __ldg(p.w.ubase + unit);
        const uint32_t w1 = unit + 1 < (int64_t) p.hdr->n_a ? __ldg(p.w.ubase + unit + 1) : (uint32_t) p.hdr->n_b;
        first = w0 & ~3u;
        bytes = ((w1 - first + 4u + 3u) & ~3u) * 4u;
        my = w0 - first + __ldg(p.w.lrel + unit * 32 + lane);
        at = part ? __ldg(p.marks + (unit * (p.parts - 1) + part - 1) * 32 + lane) : 0u;
    }
};

// The plane bytes of one warp's part, PART_AHEAD steps ahead of the decode and from the end of a part into the warp's next one.
struct PartPlane {
    const uint8_t * cur, * next;              // this lane's bytes of the part's first step, here and in the warp's next unit
    uint4 sm[PART_AHEAD];
    __device__ __forceinline__ void load(const uint8_t * from) {
        cur = from;
#pragma unroll
        for (int i = 0; i < PART_AHEAD; i++) { sm[i] = ld_stream16(cur + i * CHUNK); }
    }
    // step h + i of the part (h a multiple of PART_AHEAD)
    template <bool LOOP> __device__ __forceinline__ uint4 step(int h, int i) {
        const uint4 v = sm[i];
        if (h + PART_AHEAD < PART_STEPS) { sm[i] = ld_stream16(cur + (h + PART_AHEAD + i) * CHUNK); }
        else if (LOOP) { sm[i] = ld_stream16(next + i * CHUNK); }
        return v;
    }
};

__device__ __forceinline__ void stage_table(unsigned char * smem, const uint32_t * lut) {
    for (int i = threadIdx.x; i < HP_MAX_PAIRS / 4; i += blockDim.x) { ((uint4 *) smem)[i] = __ldg((const uint4 *) lut + i); }
}

// the unit, of those that a block takes at a time, that this warp works on
__device__ __forceinline__ int64_t first_unit(const Parts & p) {
    const int per_block = (int) (blockDim.x >> 5) / p.parts;
    return (int64_t) blockIdx.x * per_block + (int) (threadIdx.x >> 5) / p.parts;
}

// Every block takes units in turn, one warp to a part, all parts of a unit at once; the next unit's streams are copied, its plane
// asked for and its start looked up while this one is decoded, and one block barrier a unit carries the check of its marks. Units that
// fit half of the buffer (3 bits a weight; the benchmark's take 2.6) are copied into the halves in turn. A longer one takes the whole
// buffer, so that it and its neighbours are copied when the unit before them is done: 62080 x 2048 of 3.4 bits, eight columns (one
// turn), 159 us without marks, 667 where such units were left to one warp, 129 so; two columns, 16384 x 2048, 30.0, 114 and 22.5. Codes
// that all have the same length put the lanes' words into one bank: 16384 x 2048 of 32 exponents that are equally likely, two columns, 29.8 and 43.8.
//   u, units, unit0             this warp's (first) unit, where units end, and the matrix's unit that is unit 0
//   prologue()                  what else the block needs, and the wait for the kernel in front (unless the kernel waited before): single-turn
//                               kernels let the next one start from here on. The barrier behind it is here. The
//                               code table (stage_table) is at the front of the shared memory before that barrier
//   decode(rd, lut, pl, u, s)   the 64 codes of part s
//   store(u, s, alone)          after the check: results that decode() kept; alone: this warp decodes all parts, s is the last so far
// LOOP = false: a block has one turn (as many blocks as it takes), and nothing of a next one is kept in registers.
template <bool LOOP, typename Prologue, typename Decode, typename Store>
__device__ __forceinline__ void walk_parts(const Parts & p, int64_t u, int64_t units, int64_t unit0, int unit_bytes, unsigned char * smem,
                                           Prologue && prologue, Decode && decode, Store && store) {
    __shared__ int broken[3][PART_UNITS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5, per_block = nwarp / p.parts;
    const int ul = warp / p.parts, part = warp - ul * p.parts;
    const PartSmem lay = part_smem(nwarp, per_block, p.cap);
    const uint32_t base = smem_u32(smem), bar = base + lay.bars + 16 * ul, buf0 = base + lay.streams + 2 * ul * (p.cap + PART_SLACK);
    const uint32_t starts0 = base + lay.starts + warp * 128 + lane * 4;
    const int64_t stride = (int64_t) gridDim.x * per_block;
    const int rounds = !LOOP ? 1 : (int) ((units - (u - ul) + stride - 1) / stride); // the same for every warp of the block
    const uint8_t * plane = p.w.plane + part * (PART_STEPS * CHUNK) + 16 * lane;

    bool dead = false; // a copy never arrived (reported): this warp's units are decoded from global memory from then on
    auto place = [&](const PartStart & t, int b) { return buf0 + (LOOP && b && t.bytes <= p.cap ? p.cap + PART_SLACK : 0u); };
    // the part's start into shared memory for the check, a block barrier before it is read there
    auto announce = [&](const PartStart & t, int b) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(starts0 + b * nwarp * 128), "r"(t.at) : "memory"); };
    // the unit's streams on their way, barrier b to tell of it
    auto copy = [&](const PartStart & t, int b) {
        if (part == 0 && lane == 0 && t.bytes <= p.whole && !dead) {
            mbar_expect_tx(bar + 8 * b, t.bytes);
            bulk_g2s(place(t, b), p.w.stream + t.first, t.bytes, bar + 8 * b);
        }
    };
    if (part == 0 && lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    PartStart cur = {};
    PartPlane pl = {};
    if (u < units) {
        pl.load(plane + (unit0 + u) * unit_bytes); // ahead of the start, whose trip to memory the streams' copy waits for
        cur.load(p, unit0 + u, part, lane);
        announce(cur, 0);
        copy(cur, 0);
        if (lane == 0) { bulk_prefetch_l2(pl.cur - 16 * lane + PART_AHEAD * CHUNK, (PART_STEPS - PART_AHEAD) * CHUNK); }
    }
    if (threadIdx.x < 3 * PART_UNITS) { ((int *) broken)[threadIdx.x] = 0; }
    prologue();
    __syncthreads();
    uint32_t phases = 0;
    for (int r = 0, slot = 0; r < rounds; r++, u += stride, slot = slot == 2 ? 0 : slot + 1) {
        const int b = r & 1;
        const bool active = u < units, staged = cur.bytes <= p.whole, more = LOOP && u + stride < units;
        PartStart nxt = {};
        pl.next = pl.cur;
        bool behind = false; // the next unit's streams have no room beside this one's
        if (more) {
            nxt.load(p, unit0 + u + stride, part, lane);
            announce(nxt, b ^ 1);
            behind = max(cur.bytes, nxt.bytes) > p.cap;
            if (!behind) { copy(nxt, b ^ 1); }
            pl.next = plane + (unit0 + u + stride) * unit_bytes;
            if (lane == 0) { bulk_prefetch_l2(pl.next, PART_STEPS * CHUNK); }
        }
        if (active && staged) {
            const uint32_t landed = dead ? 0u : mbar_wait(bar + 8 * b, (phases >> b) & 1u), words = place(cur, b);
            if (!LOOP) { grid_launch_dependents(); }
            phases ^= 1u << b;
            bool joined = false;
            if (landed) {
                WindowReader rd;
                rd.open_at(words + 4 * min(cur.my + (cur.at >> 5), cur.bytes / 4), cur.at & 31u, landed);
                decode(rd, base, pl, u, part);
                // whether the part ended where the next one (the next warp's) began, in every lane. The start that the next part
                // took is compared, not the mark in memory: that one may be being written.
                joined = __all_sync(FULL, part + 1 == p.parts || rd.position(words + 4 * cur.my) == lds32(starts0 + b * nwarp * 128 + 128, rd.next));
            } else {
                if (lane == 0) { atomicOr(&g_wait_expired, 1u); }
                dead = true;
                if (LOOP) { pl.load(pl.next); }
            }
            if (!joined && lane == 0) { broken[slot][ul] = 1; }
        }
        __syncthreads();
        if (behind) { copy(nxt, b ^ 1); } // no warp reads this unit's streams any more
        if (threadIdx.x < PART_UNITS) { broken[slot == 0 ? 2 : slot - 1][threadIdx.x] = 0; } // read before this barrier, used after the next
        if (active && staged && !broken[slot][ul]) {
            store(u, part, false);
        } else if (active && part == 0) { // marks that are not this matrix's, or streams longer than any code makes them: the unit from its start
            GlobalReader rd;
            rd.lut = (const uint32_t *) smem;
            rd.rd.open(p.w, unit0 + u, lane);
            const uint8_t * next = pl.next;
            for (int s = 0; s < p.parts; s++) {
                pl.load(plane + (unit0 + u) * unit_bytes + s * (PART_STEPS * CHUNK));
                pl.next = pl.cur;
                decode(rd, 0u, pl, u, s);
                store(u, s, true);
            }
            if (LOOP) { pl.load(next); pl.next = next; }
        } else if (LOOP && !staged) {
            pl.load(pl.next);
        }
        pl.cur = pl.next;
        cur = nxt;
    }
}

} // namespace dev

inline dev::Parts make_parts(const bf16n_weight & w, const uint16_t * marks) {
    const uint32_t cap = (uint32_t) ((w.R * w.K * 3 / 8 + 64 + 15) & ~15ll);
    return {dev::pair_view(w), (const AuxHeader *) w.aux, marks, unit_parts(w), cap, dev::part_whole(cap)};
}

} // namespace b16
