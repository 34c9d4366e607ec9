// Matrices of few lane-major pair-Huffman units with marks (parts.cuh): the decode GEMV of 1 to 8 dense columns and the exact
// reconstruction. One warp per part, so that a chain is 64 lookups long whatever the unit's size, and all parts of a unit in
// one block.
//
// What bounds them is latency: the code table, the unit's streams (one bulk copy) and the part's first plane bytes (straight into
// registers, the others into L2) are one trip to memory together, then come 64 dependent lookups. 8192 x 2048, one token: 20.4 us
// with a warp to each of the 512 units, 10.8 with 4096 parts (2.1 TB/s of stored bytes; 0.32 of what HBM gives). Activations lie in
// shared memory as they are given; a quad of a column is read where it is multiplied, off the chain. Four blocks fit an SM at 64
// registers, so 512 units of eight parts are one wave. Two and four columns take units in turn (16384 x 2048, 2 columns: 23.7 us
// with a block to each unit, 20.4 so); one and eight do not, whose registers that overflows (9.1 against 10.1, 42 against 44).
#include "parts.cuh"
#include "sinks.cuh"

namespace b16 {
namespace {

using namespace dev;

constexpr int PART_WARPS = 8;                 // of a block; 16 where a unit has sixteen parts
static_assert(PART_WARPS / 2 <= PART_UNITS, "units of two parts");

// a quad of a column's activations: products in the format's order
template <typename TX> struct Quad;
template <> struct Quad<bf16> {
    uint2 v;
    __device__ __forceinline__ void load(uint32_t xs, int col) { asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(xs + col * 2)); }
    __device__ __forceinline__ void fma(uint32_t w0, uint32_t w1, float (&a)[4]) const {
        LaneX<1, bf16>::fma2(w0, v.x, a[0], a[1]);
        LaneX<1, bf16>::fma2(w1, v.y, a[2], a[3]);
    }
};
template <> struct Quad<float> {
    float4 v;
    __device__ __forceinline__ void load(uint32_t xs, int col) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(xs + col * 4));
    }
    __device__ __forceinline__ void fma(uint32_t w0, uint32_t w1, float (&a)[4]) const {
        a[0] = fmaf(bf16lo_f32(w0), v.x, a[0]);
        a[1] = fmaf(bf16hi_f32(w0), v.y, a[1]);
        a[2] = fmaf(bf16lo_f32(w1), v.z, a[2]);
        a[3] = fmaf(bf16hi_f32(w1), v.w, a[3]);
    }
};

// NC dense columns (those from ncols on are computed and not stored) of row-major units. A part is 8 / C whole rows, so parts
// share nothing but the check of their starts.
__host__ __device__ constexpr int parts_resident(int C, int NC) { return C == 8 ? (NC == 1 ? 2 : 1) : NC == 1 ? 4 : NC <= 4 ? 3 : 2; } // blocks of an SM, by registers
__host__ __device__ constexpr bool parts_loop(int NC) { return NC == 2 || NC == 4; }
template <int C, int NC, typename TX>
__global__ void __launch_bounds__(C == 8 ? 512 : 256, parts_resident(C, NC)) k_gemv_parts(const Parts p, const Cols q, int R, int ncols, const Opaque k) {
    constexpr int K = C * CHUNK, ROWS = PART_STEPS / C;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    unsigned char * xs = smem + part_smem(blockDim.x >> 5, (blockDim.x >> 5) / p.parts, p.cap).end;
    const uint32_t xa = smem_u32(xs);
    float mine[NC]; // lane r: row r of the part
    // Before anything of the matrix: a kernel of the caller's in front may have written it. 8192 x 2048, products one after the other, one /
    // two / eight tokens: 9.0 / 13.5 / 20.9 us with the matrix read above the wait, 10.8 / 13.4 / 21.8 so; with the release of the next kernel
    // here too (walk_parts has it behind the streams' arrival) 10.9 / 15.0 / 22.3, as an ordinary launch 11.2 / 13.8 / 22.4.
    bare_grid_dependency_wait();
    auto prologue = [&] {
        stage_table(smem, p.w.lut);
        constexpr int VEC = 8 / (int) sizeof(TX); // eight bytes a load: what the interface asks of x and its strides
        for (int i = threadIdx.x; i < NC * (K / VEC); i += blockDim.x) {
            const int n = i / (K / VEC), c = i - n * (K / VEC);
            ((uint2 *) xs)[i] = ld_act8(q.x + min(n, ncols - 1) * q.x_tok + c * 8);
        }
    };
    auto rows = [&](auto & rd, uint32_t lut, PartPlane & pl, int64_t, int) {
        float a[NC][4];
#pragma unroll 1
        for (int h = 0; h < PART_STEPS; h += PART_AHEAD) { // four steps as straight code: eight spill
#pragma unroll
            for (int i = 0; i < PART_AHEAD; i++) {
                const int c = C == 8 ? h + i : i % C;
                if (C == 8 ? h + i == 0 : c == 0) {
#pragma unroll
                    for (int n = 0; n < NC; n++) { a[n][0] = a[n][1] = a[n][2] = a[n][3] = 0.f; }
                }
                uint32_t e[8], wv[8];
                rd.take8(lut, k, e);
                assemble8(pl.template step<parts_loop(NC)>(h, i), e, wv);
#pragma unroll
                for (int n = 0; n < NC; n++) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        Quad<TX> x;
                        x.load(xa + n * K * (int) sizeof(TX), c * CHUNK + 128 * j + 4 * lane);
                        x.fma(wv[2 * j], wv[2 * j + 1], a[n]);
                    }
                }
                if (C == 8 ? h + i == C - 1 : c == C - 1) {
#pragma unroll
                    for (int n = 0; n < NC; n++) {
                        const float sum = warp_sum((a[n][0] + a[n][1]) + (a[n][2] + a[n][3]));
                        if (lane == (h + i) / C) { mine[n] = sum; }
                    }
                    if (C < 4) { __syncwarp(); } // keeps the next row's activation loads, and their registers, behind this row
                }
            }
        }
    };
    auto put = [&](int64_t u, int s, bool) {
        if (lane < ROWS) {
#pragma unroll
            for (int n = 0; n < NC; n++) {
                const OutVec out = {q.y + n * q.y_tok, q.y_bf16};
                if (n < ncols) { out.put(u * R + s * ROWS + lane, mine[n]); }
            }
        }
    };
    walk_parts<parts_loop(NC)>(p, first_unit(p), q.nrows / R, q.row0 / R, R * K, smem, prologue, rows, put);
}

// a BF16 row in shared memory times a token's activations: FP32 sums, as k_rescore of draft.cu adds them
template <int K>
__device__ __forceinline__ float row_product(const bf16 * a, const bf16 * b, int lane) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = lane * 8; k < K; k += 256) {
        const uint4 p = *(const uint4 *) (a + k), q = ld_act16(b + k);
        acc[0] = fmaf(bf16lo_f32(p.x), bf16lo_f32(q.x), acc[0]); acc[1] = fmaf(bf16hi_f32(p.x), bf16hi_f32(q.x), acc[1]);
        acc[2] = fmaf(bf16lo_f32(p.y), bf16lo_f32(q.y), acc[2]); acc[3] = fmaf(bf16hi_f32(p.y), bf16hi_f32(q.y), acc[3]);
        acc[0] = fmaf(bf16lo_f32(p.z), bf16lo_f32(q.z), acc[0]); acc[1] = fmaf(bf16hi_f32(p.z), bf16hi_f32(q.z), acc[1]);
        acc[2] = fmaf(bf16lo_f32(p.w), bf16lo_f32(q.w), acc[2]); acc[3] = fmaf(bf16hi_f32(p.w), bf16hi_f32(q.w), acc[3]);
    }
    return warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
}

template <typename Sink, int THREADS> // 512: units of more than eight parts
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_expand_parts(const Parts p, int C, int R, bool cm, int64_t unit0, int64_t units, const Sink sink_in, const Opaque k) {
    Sink sink = sink_in;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    auto chunks = [&](auto & rd, uint32_t lut, PartPlane & pl, int64_t u, int s) {
        int rr = cm ? s * PART_STEPS % R : s * PART_STEPS / C, c = cm ? s * PART_STEPS / R : s * PART_STEPS % C;
#pragma unroll 1
        for (int h = 0; h < PART_STEPS; h += PART_AHEAD) {
#pragma unroll
            for (int i = 0; i < PART_AHEAD; i++) {
                uint32_t e[8], wv[8];
                rd.take8(lut, k, e);
                assemble8(pl.template step<false>(h, i), e, wv);
                sink.chunk(u * R + rr, c, lane, wv);
                if (cm) { if (++rr == R) { rr = 0; c++; } } else { if (++c == C) { c = 0; rr++; } }
            }
        }
    };
    walk_parts<false>(p, first_unit(p), units, unit0, R * C * CHUNK, smem, [&] {
        stage_table(smem, p.w.lut);
        bare_grid_dependency_wait(); // an ordinary launch, to which this is nothing; walk_parts lets the next kernel start
    }, chunks, [](int64_t, int, bool) {});
}

// Few rows (a draft step's candidates, the tokens of a decode batch), one block each: the warp of the part that the row lies in
// passes over the rows before it there and decodes it, the warps of the parts before that only walk their codes, so that the row's
// start is known to be right when the block meets. 128 candidates of 62080 x 2048: 19.7 us by a walk of up to 15 rows from the unit's
// start (with a table of the codes that end in 12 bits of stream), 4.7 so. SCORED: the row is multiplied with its token's activations as well.
__device__ unsigned int g_row_wait_expired; // a copy of a gathered row's unit never arrived: the row gather's word, not the products'
template <int C, bool BF, bool SCORED>
__global__ void __launch_bounds__(512) k_rows_parts(const Parts p, int R, const char * ids, int64_t ids_s0, int64_t row0, char * dst, int64_t dst_s1,
                                                    const RowScores scores, const Opaque k) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int broken;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const PartSmem lay = part_smem(nwarp, 1, p.cap);
    const uint32_t base = smem_u32(smem), bar = base + lay.bars, words = base + lay.streams, starts = base + lay.starts + warp * 128 + lane * 4;
    if (threadIdx.x == 0) {
        broken = 0;
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    stage_table(smem, p.w.lut);
    grid_dependency_wait(); // the row ids may come from the kernel before this one; everything above is the matrix's own
    const int64_t gr = row0 + *(const volatile int32_t *) (ids + blockIdx.x * ids_s0), unit = gr / R;
    const int t0 = (int) (gr - unit * R) * C, part = t0 / PART_STEPS;
    const uint8_t * pl = p.w.plane + gr * (C * CHUNK) + 16 * lane;
    PartStart cur = {};
    uint4 sm[C];
    if (warp <= part) {
        if (warp == part) {
#pragma unroll
            for (int c = 0; c < C; c++) { sm[c] = ld_stream16(pl + c * CHUNK); }
        }
        cur.load(p, unit, warp, lane);
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(starts), "r"(cur.at) : "memory");
        if (threadIdx.x == 0 && cur.bytes <= p.whole) {
            mbar_expect_tx(bar, cur.bytes);
            bulk_g2s(words, p.w.stream + cur.first, cur.bytes, bar);
        }
    }
    __syncthreads();
    char * o = dst + blockIdx.x * dst_s1;
    unsigned char * row_s = smem + lay.end; // SCORED: the row as BF16
    auto row = [&](auto & rd, uint32_t lut, int before) { // `before` steps, then the row
        for (int i = 0; i < before; i++) { uint32_t e[8]; rd.take8(lut, k, e); }
#pragma unroll
        for (int c = 0; c < C; c++) {
            uint32_t e[8], wv[8];
            rd.take8(lut, k, e);
            assemble8(sm[c], e, wv);
            put_row_chunk<BF>(o, c, lane, wv);
            if (SCORED) { put_row_chunk<true>((char *) row_s, c, lane, wv); }
        }
    };
    if (warp <= part) {
        bool good = false;
        if (cur.bytes <= p.whole) {
            const uint32_t landed = mbar_wait(bar, 0u);
            if (landed) {
                WindowReader rd;
                rd.open_at(words + 4 * min(cur.my + (cur.at >> 5), cur.bytes / 4), cur.at & 31u, landed);
                if (warp == part) {
                    row(rd, base, t0 - part * PART_STEPS);
                    good = true;
                } else {
                    for (int i = 0; i < PART_STEPS; i++) { uint32_t e[8]; rd.take8(base, k, e); }
                    good = __all_sync(FULL, rd.position(words + 4 * cur.my) == lds32(starts + 128, rd.next));
                }
            } else if (lane == 0) {
                atomicOr(&g_row_wait_expired, 1u);
            }
        }
        if (!good && lane == 0) { broken = 1; }
    }
    __syncthreads();
    if (warp != part) { return; }
    if (broken) {
        GlobalReader rd;
        rd.lut = (const uint32_t *) smem;
        rd.rd.open(p.w, unit, lane);
        row(rd, 0u, t0);
    }
    if (SCORED) {
        __syncwarp();
        const int t = (int) blockIdx.x / scores.n_cand;
        const bf16 * a = (const bf16 *) row_s, * b = (const bf16 *) scores.x_bf16 + (int64_t) t * (C * CHUNK);
        const float v = row_product<C * CHUNK>(a, b, lane);
        if (lane == 0) { scores.out[t * scores.vocab + (gr - row0)] = v; }
    }
}

// One warp per unit, once per matrix: where every 64 codes of a lane begin. `last`: the last stream word that may be read. A loader may
// upload memory that it fills later, so nothing that the aux buffer holds is taken for right here: words behind `last` are not
// read, and a length counts as at most HP_LMAX bits.
__global__ void __launch_bounds__(256) k_marks(const PairView w, int parts, int64_t units, uint16_t * marks, uint32_t last) {
    __shared__ uint32_t lut[HP_MAX_PAIRS];
    for (int i = threadIdx.x; i < HP_MAX_PAIRS; i += 256) { lut[i] = __ldg(w.lut + i); }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int64_t u = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += (int64_t) gridDim.x * 8) {
        uint32_t next = __ldg(w.ubase + u) + __ldg(w.lrel + u * 32 + lane);
        auto word = [&] { return __ldg(w.stream + min(next++, last)); };
        uint64_t buf = (uint64_t) word() << 32;
        buf |= word();
        uint32_t ahead = word(), bits = 0;
        int have = 64;
        for (int s = 1; s < parts; s++) {
#pragma unroll 1
            for (int i = 0; i < 32 * PART_STEPS / 8; i++) { // two codes
                if (have <= 32) {
                    buf |= (uint64_t) ahead << (32 - have);
                    have += 32;
                    ahead = word();
                }
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int n = min((int) (lut[(uint32_t) (buf >> (64 - HP_LMAX))] & 31u), HP_LMAX);
                    buf <<= n;
                    have -= n;
                    bits += n;
                }
            }
            marks[(u * (parts - 1) + s - 1) * 32 + lane] = (uint16_t) bits;
        }
    }
}

// units of a block: as many as eight warps take
int units_per_block(int parts) { return std::max(1, PART_WARPS / parts); }

template <int C, int NC, typename TX>
void launch_gemv_parts(const bf16n_weight & w, const uint16_t * marks, const Cols & q, int ncols, cudaStream_t st) {
    const Parts p = make_parts(w, marks);
    const int per = units_per_block(p.parts), warps = per * p.parts;
    const int64_t units = q.nrows / w.R, blocks = (units + per - 1) / per;
    // spread evenly (even_smem): 256 blocks of 8192 x 1024 and 4096 x 2048, two / four columns: 8.7 / 10.8 and 8.3 / 10.6 us crowded, 7.3 / 8.9 and
    // 7.0 / 8.4 so; expert parts, gathers and fragment-order products were level
    const size_t shm = even_smem(part_smem(warps, per, p.cap).end + (size_t) NC * w.K * sizeof(TX), blocks);
    const Opaque k = {1u, 4u};
    launch_chained(k_gemv_parts<C, NC, TX>, dim3((unsigned) (parts_loop(NC) ? std::min(blocks, (int64_t) device_info().sms * parts_resident(C, NC)) : blocks)), dim3(warps * 32), shm, st, p, q, w.R, ncols, k);
}
template <int C, typename TX>
void gemv_parts_c(const bf16n_weight & w, const uint16_t * marks, const Cols & q, int ncols, cudaStream_t st) {
    switch (ncols) {
        case 1: launch_gemv_parts<C, 1, TX>(w, marks, q, ncols, st); break;
        case 2: launch_gemv_parts<C, 2, TX>(w, marks, q, ncols, st); break;
        case 3: case 4: launch_gemv_parts<C, 4, TX>(w, marks, q, ncols, st); break;
        default: launch_gemv_parts<C, 8, TX>(w, marks, q, ncols, st); break;
    }
}

} // namespace

BF16N_DEFINE_FAULT_WORD(gemv_parts_fault_word)
unsigned int * rows_parts_fault_word() {
    unsigned int * p = nullptr;
    cuda_ok(cudaGetSymbolAddress((void **) &p, g_row_wait_expired), "fault word address");
    return p;
}

void gemv_parts_init() {
    const int optin = device_info().smem_optin;
#define ATTR(C, N, TX) allow_dynamic_smem((const void *) k_gemv_parts<C, N, TX>, optin, optin, "parts");
#define ATTR_C(C, TX) ATTR(C, 1, TX) ATTR(C, 2, TX) ATTR(C, 4, TX) ATTR(C, 8, TX)
    ATTR_C(1, bf16) ATTR_C(2, bf16) ATTR_C(4, bf16) ATTR_C(8, bf16) ATTR_C(1, float) ATTR_C(2, float) ATTR_C(4, float) ATTR_C(8, float)
#undef ATTR_C
#undef ATTR
#define ATTR(C) allow_dynamic_smem((const void *) k_rows_parts<C, true, true>, optin, optin, "rows"); allow_dynamic_smem((const void *) k_rows_parts<C, true, false>, optin, optin, "rows"); \
                allow_dynamic_smem((const void *) k_rows_parts<C, false, false>, optin, optin, "rows");
    ATTR(1) ATTR(2) ATTR(4) ATTR(8)
#undef ATTR
    allow_dynamic_smem((const void *) k_expand_parts<StoreBF16, 256>, optin, optin, "parts");
    allow_dynamic_smem((const void *) k_expand_parts<StoreBF16, 512>, optin, optin, "parts");
}

int unit_parts(const bf16n_weight & w) {
    const int64_t steps = w.R * (w.K / CHUNK);
    return w.format == FMT_HUFPAIR && !w.fo && steps % PART_STEPS == 0 && steps >= 2 * PART_STEPS && steps <= 16 * PART_STEPS ? (int) (steps / PART_STEPS) : 0;
}

// Walk from the unit's start (a warp to a row) / parts in us: 592 rows of 2048 columns 21.9 / 7.4, 9472 101 / 68; 592 rows of 512 columns (two
// parts) 10.0 / 5.2, 2368 11.1 / 10.3, 4736 15.4 / 17.4.
bool rows_parts_applies(const bf16n_weight & w, const uint16_t * marks, int64_t n) {
    const int64_t C = w.K / CHUNK;
    return marks && unit_parts(w) && !w.cm && n <= (int64_t) device_info().sms * (unit_parts(w) > 2 ? 64 : 16) && (C == 1 || C == 2 || C == 4 || C == 8);
}

void rows_parts(const bf16n_weight & w, const uint16_t * marks, const void * ids, int64_t ids_s0, int64_t n, void * dst, bool dst_bf16, int64_t dst_s1,
                int64_t row0, const RowScores * scores, cudaStream_t st, bool behind_own) {
    const Parts p = make_parts(w, marks);
    const size_t shm = part_smem(p.parts, 1, p.cap).end + (scores ? (size_t) w.K * 2 : 0);
    auto go = [&](auto * kernel) {
        launch_behind(behind_own, kernel, dim3((unsigned) n), dim3(p.parts * 32), shm, st, p, w.R, (const char *) ids, ids_s0, row0, (char *) dst, dst_s1,
                      scores ? *scores : RowScores{}, Opaque{1u, 4u});
        check_launch();
    };
#define GO(C) case C: if (scores) { go(k_rows_parts<C, true, true>); } else if (dst_bf16) { go(k_rows_parts<C, true, false>); } else { go(k_rows_parts<C, false, false>); } break;
    switch (w.K / CHUNK) { GO(1) GO(2) GO(4) GO(8) default: fail_invalid("unsupported K"); }
#undef GO
}

size_t marks_bytes(const bf16n_weight & w) {
    const int parts = unit_parts(w);
    return parts ? (size_t) (w.rows / w.R) * (parts - 1) * 32 * sizeof(uint16_t) : 0;
}

void marks_build(const bf16n_weight & w, uint64_t aux_bytes, uint16_t * marks, cudaStream_t st) {
    const uint64_t units = (uint64_t) (w.rows / w.R);
    auto holds = [&](uint64_t off, uint64_t n, uint64_t align) { return off % align == 0 && off <= aux_bytes && n <= aux_bytes - off; };
    require(holds(w.off_a, 4 * HP_MAX_PAIRS, 4) && holds(w.off_b, units * 4, 4) && holds(w.off_c, units * 64, 2) && holds(w.off_d, 4, 4),
            "marks_build: aux shorter than its offsets");
    const uint64_t words = (aux_bytes - w.off_d) / 4;
    if (units == 0) { return; }
    k_marks<<<(unsigned) std::min<uint64_t>((units + 7) / 8, 1184), 256, 0, st>>>(pair_view(w), unit_parts(w), (int64_t) units, marks,
                                                                                  (uint32_t) std::min<uint64_t>(words - 1, UINT32_MAX));
    check_launch();
}

// Where the parts are the faster form, by units of the product. Time with parts over time without marks, units of 16 x 2048 (20 to 90 us; other K,
// and units of 8 and 4 rows, alike):
//   units            512  1024  1280  1536  2048  2560  3072  3584  4096
//   1 column, BF16  0.55  0.82  0.96  1.09  1.29  1.23  1.30  1.29  1.41
//   2               0.59  0.77  0.77  0.89  1.03  1.09  1.14  0.87  0.97
//   3               0.36  0.48  0.49  0.58  0.68  0.73  0.76  0.66  0.72
//   4               0.63  0.83  0.82  0.96  1.10  1.14  0.88  0.99  1.07
//   5 / 6           0.46  0.61  0.69  0.82  0.92  1.02  0.88  0.98  1.05 / 0.89 (2960 units: 1.11 / 1.08; 4096 units of 4 x 2048 0.86 / 0.78)
//   7 / 8           0.44  0.58  0.63  0.75  0.83  0.91  0.70  0.79  0.85 (of the two the slower)
//   1 column, FP32  0.57  0.94  1.03  1.20  1.40  1.07  1.28  1.28  1.33
//   2               0.68  0.56  0.57  0.67  0.83  0.48  0.56  0.65  0.75 (2048 units of 512 to 1024 columns or 4 rows 1.03 to 1.08)
//   3               0.77  0.83  0.82  0.98  1.17  0.66  0.77  0.91  1.04 (1536 units of 8 and 4 rows 1.5)
//   5 to 8          0.67  0.60  0.69  0.80  0.92  0.56  0.65  0.77  0.87
// The kernels without marks take units in rounds, of 28, 24 and 20 per SM for one, two and four columns of BF16 and of 16 for FP32, and
// are at their best when a round is just full. Differences of up to 8 % either way come with where the buffers lie. 4096 columns of weights have no other form that stages streams: 0.14 to 0.94 up to 4096
// units, but three to six of FP32 up to 1.12 just before their round is full.
// With marks of another matrix (overwritten since, by a program that makes no new ones) every unit is decoded twice, the second time by one warp:
// without marks / with wrong ones, 8192 x 2048, one and eight columns 20 / 48 and 51 / 101, 62080 x 2048, eight columns 161 / 710, reconstructed
// 86 / 410, a decode step of one and eight tokens 24 / 55 and 101 / 333. So the marks are made again behind an update (45 us for 1024 x 2048
// under a profiler), by the Python layer where it sees one. Kernels that wrote the true marks themselves were tried: 1 to 5 % on every call.
bool gemv_parts_applies(const bf16n_weight & w, const uint16_t * marks, const bf16n_mmv_args & a) {
    const int C = (int) (w.K / CHUNK), parts = unit_parts(w);
    if (!marks || !parts || parts > (C == 8 ? 2 : 1) * PART_WARPS || w.cm || a.ids || a.ncols > 8 || !(C == 1 || C == 2 || C == 4 || C == 8)) { return false; }
    const int64_t units = a.nrows / w.R;
    const bool large = w.R * C >= 64; // units of 16 x 2048 weights and more
    auto fills = [&](int64_t from, int per_sm) { return units > from && units <= per_sm * device_info().sms; };
    if (units > 4096) { return false; }
    if (C == 8) { return a.x_bf16 || a.ncols < 3 || a.ncols > 6 || !fills(1536, 16); }
    switch (a.ncols) {
        case 1: case 4: return units <= 1024;
        case 2: return units * C <= 6144;
        case 3: return a.x_bf16 || units <= (large ? 1536 : 1024) || (w.R >= 16 && units <= 3584 && !fills(1024, 16));
        case 5: case 6: return !a.x_bf16 || !large || !fills(2304, 20);
        default: return true;
    }
}

void gemv_parts(const bf16n_weight & w, const uint16_t * marks, const bf16n_mmv_args & a, cudaStream_t st) {
    const Cols q = make_cols(a);
#define GO(C) case C: if (a.x_bf16) { gemv_parts_c<C, bf16>(w, marks, q, a.ncols, st); } else { gemv_parts_c<C, float>(w, marks, q, a.ncols, st); } break;
    switch (w.K / CHUNK) { GO(1) GO(2) GO(4) GO(8) default: fail_invalid("unsupported K"); }
#undef GO
}

// Rings or general kernel / parts in us: 8192 x 2048 24.5 / 10.6, 16384 x 2048 31.0 / 21.1, 62080 x 2048 87.5 / 73.5, 16384 x 4096 64.7 /
// 46.1, 65536 x 1024 43.5 / 43.2; units of two parts: 16384 x 512 9.4 / 6.6, 65536 x 512 20.7 / 22.4.
bool expand_parts_applies(const bf16n_weight & w, const uint16_t * marks, int64_t nrows) {
    const int parts = unit_parts(w);
    return marks && parts && nrows / w.R <= (parts > 2 ? 4096 : 2048);
}

template <typename Sink>
static void expand_parts_to(const bf16n_weight & w, const uint16_t * marks, int64_t row0, int64_t nrows, const Sink & sink, cudaStream_t st) {
    const Parts p = make_parts(w, marks);
    const int per = units_per_block(p.parts), warps = per * p.parts;
    const int64_t units = nrows / w.R;
    if (units == 0) { return; }
    const Opaque k = {1u, 4u};
    auto * kernel = warps > 8 ? k_expand_parts<Sink, 512> : k_expand_parts<Sink, 256>;
    kernel<<<(unsigned) ((units + per - 1) / per), warps * 32, part_smem(warps, per, p.cap).end, st>>>(p, (int) (w.K / CHUNK), w.R, w.cm != 0, row0 / w.R, units,
                                                                                                      sink, k);
    check_launch();
}
void expand_parts(const bf16n_weight & w, const uint16_t * marks, int64_t row0, int64_t nrows, const StoreBF16 & sink, cudaStream_t st) {
    expand_parts_to(w, marks, row0, nrows, sink, st);
}

} // namespace b16
