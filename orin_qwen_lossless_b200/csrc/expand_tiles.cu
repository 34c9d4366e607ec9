// First pass of the two-pass batched (prefill) product: decode whole expert matrices, at full occupancy, into BF16
// operand tiles that the tensor-core pass (k_tile_mm in prefill.cu) copies into shared memory with one bulk copy each.
//
// The fused prefill kernel decodes inside the block that multiplies; its 16 decoder warps per SM are register-bound and
// their dependent table lookups set the pace of the layer. Here one unit per warp and 28 warps per SM decode with the
// ring reader of the large-matrix GEMV (per-lane cp.async rings, window reader, four interleaved table copies), and
// what they write is already the shared-memory image of the B operand:
//
//   image of (expert e, row block nb) = [K / 64 k-tiles][256 rows][128 bytes], K-major, 128-byte swizzled
//   (16-byte piece p of row r is stored at piece p ^ (r & 7)); a k-tile of a row block is 32 KB, contiguous.
//
// Row block of a plain matrix: its rows 256 nb .. 256 nb + 255. Row block of a gate/up pair (SwiGLU): gate rows
// 128 nb .. 128 nb + 127 as image rows 0..127 and the same rows of up as image rows 128..255, so that the thread that
// reads a token's accumulators holds gate and up of the same output.
//
// A lane's 4 consecutive weights (lane-major chunk: column 128 j + 4 l + {0..3} of quad j) are one 8-byte store; the 32
// lanes of a store instruction fill two whole 128-byte lines (k-tiles 2 j and 2 j + 1 of the chunk). Both unit layouts
// are one linear walk over (row, chunk) steps of 512 weights: row-major units step chunks fastest, chunk-major units
// rows fastest; the plane and the streams are in step order either way.
#include "launch.h"
#include "rings.cuh"

namespace b16 {
namespace {

using namespace dev;
using namespace ring;

constexpr int EXPAND_WARPS = 28;              // 72 registers per thread: four steps of plane bytes in flight per lane
constexpr int AHEAD = 4;                     // plane bytes are loaded this many steps (of 512 weights) before they are decoded
constexpr int IMG_ROWS = 256;                 // rows of a row block = N of the tensor-core pass
constexpr int IMG_KTILE_BYTES = IMG_ROWS * 128;

struct ExpandArgs {
    PairView w[2];               // [1]: the up matrix of a gate/up pair (blockIdx.y picks the matrix)
    unsigned char * images;      // row-block images of the experts (see the layout above)
    const int32_t * bounds;      // per expert: first routed pair (n_experts + 1 entries); experts without pairs are skipped; may be null
    int64_t units;               // units of the whole (expert-stacked) matrix
    int rows_per_expert;
    int rows_per_block;          // 256 (plain) or 128 (one half of a gate/up pair; the up half fills image rows 128..255)
    int blocks_per_expert;
};

template <int C, int R, bool CM>
__global__ void __launch_bounds__(EXPAND_WARPS * 32, 1) k_expand_tiles(const ExpandArgs p, const Opaque k) {
    constexpr int K = C * CHUNK, STEPS = R * C, KT = K / 64;
    static_assert(AHEAD == 4 && STEPS % AHEAD == 0, "the rings are topped up every four steps (32 codes), which is also the plane read-ahead");
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem; // four interleaved tables | one 4 KB ring set per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const uint32_t lut_s = smem_u32(lut);
    const uint32_t lut_l = lut_s + (lane & 3) * 4;
    const uint32_t key = (lut_s + LUT_BYTES + (uint32_t) warp * (32 * RING_BYTES) + lane * RING_BYTES) | ((lane & 7) << 4);
    const PairView w = blockIdx.y ? p.w[1] : p.w[0];
    const int row_offset = blockIdx.y ? IMG_ROWS / 2 : 0;
    for (int i = threadIdx.x; i < HP_MAX_PAIRS; i += blockDim.x) { const uint32_t e = __ldg(w.lut + i); ((uint4 *) lut)[i] = make_uint4(e, e, e, e); }
    grid_dependency_wait(); // the routing is an earlier kernel's, and the images may still be read by one
    __syncthreads();

    const uint32_t piece = (uint32_t) (lane & 15) >> 1;
    const uint32_t lane_part = (uint32_t) (lane >> 4) * IMG_KTILE_BYTES + (uint32_t) (lane & 1) * 8;
    for (int64_t u = (int64_t) blockIdx.x * nwarp + warp; u < p.units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t row0 = u * R;
        const int e = (int) (row0 / p.rows_per_expert), ri = (int) (row0 - (int64_t) e * p.rows_per_expert);
        if (p.bounds && ld_act_s32(p.bounds + e + 1) == ld_act_s32(p.bounds + e)) { continue; }
        const int nb = ri / p.rows_per_block, img_row0 = ri - nb * p.rows_per_block + row_offset;
        unsigned char * img = p.images + ((int64_t) e * p.blocks_per_expert + nb) * ((int64_t) KT * IMG_KTILE_BYTES) + lane_part;
        RingReader rd;
        {
            const uint32_t w0 = __ldg(w.ubase + u), l0 = __ldg(w.lrel + u * 32 + lane);
            rd.open((const uint8_t *) (w.stream + (w0 & ~3u)), ((w0 & 3u) + l0) * 4u, key, k);
        }
        cp_async_commit();
        const uint8_t * pl = w.plane + u * R * K + 16 * lane;
        // Plane bytes AHEAD steps ahead of the decode: with every SM writing tiles at the same time a load takes several
        // microseconds, more than one step of decoding hides.
        uint4 nx[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) { nx[i] = ld_stream16(pl + i * CHUNK); }
        rd.token = cp_async_wait_all();
        rd.first_words();
#pragma unroll 1
        for (int t0 = 0; t0 < STEPS; t0 += AHEAD) {
            if (t0) {
                rd.token = cp_async_wait_all(); // copies issued four steps ago
                rd.template top_up<3>(k);
                cp_async_commit();
            }
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int t = t0 + i;
                const int rr = CM ? t % R : t / C, c = CM ? t / R : t % C;
                const uint4 sm = nx[i];
                nx[i] = ld_stream16(pl + (t + AHEAD < STEPS ? t + AHEAD : t) * CHUNK); // the last steps re-read themselves: harmless L2 hits
                const uint32_t pw[4] = {sm.x, sm.y, sm.z, sm.w};
                const uint32_t row = (uint32_t) (img_row0 + rr);
                unsigned char * rp = img + (size_t) c * 8 * IMG_KTILE_BYTES + row * 128 + ((piece ^ (row & 7)) << 4);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    uint32_t en[4];
                    rd.take2(lut_l, k, en[0], en[1]);
                    rd.take2(lut_l, k, en[2], en[3]);
#pragma unroll
                    for (int jj = 0; jj < 2; jj++) { // quad 2 half + jj of the chunk: k-tiles 2 (2 half + jj) and the next one
                        const uint32_t lo = merge_sm_exp(spread_lo(pw[2 * half + jj]), en[2 * jj]);
                        const uint32_t hi = merge_sm_exp(spread_hi(pw[2 * half + jj]), en[2 * jj + 1]);
                        *(uint2 *) (rp + (size_t) (2 * (2 * half + jj)) * IMG_KTILE_BYTES) = make_uint2(lo, hi);
                    }
                }
            }
        }
    }
}

// The same pass for fragment-order experts (the vLLM layout, fo.cu): a unit is one 512-column slab of a 16-row band, and a
// lane's symbols of a 16 x 16 tile are the A fragment of mma.m16n8k16. Four tiles of a band are 16 rows of one k-tile of
// the image, 2048 contiguous bytes, so a warp puts its fragments into a 2 KB shared-memory copy of that piece with one
// stmatrix per tile (the fragment layout is stmatrix's) and sends it with one bulk store: one store request for every
// 1024 weights, whole lines only, no shuffles. What bounds it is HBM, as above (one byte read per weight and 2.6 bits of
// stream, two bytes written). Whole layer (route, gate/up, down, combine) at 8192 tokens and 256 experts: 3227 us with the
// fused kernel (an expert's 256 tokens decode it three times), 1670 us with this pass and k_tile_mm. Experts are taken in ranges, so that the images of a range fit the caller's scratch.
constexpr int FO_BAND = 16, FO_UNIT_W = FO_BAND * CHUNK;   // rows of a band, weights of a unit
constexpr int FO_STEPS = FO_UNIT_W / CHUNK;               // steps of 512 weights = two 16 x 16 tiles
constexpr int FO_STAGE = FO_BAND * 128;                   // a band's piece of one k-tile
constexpr int FO_EXPAND_WARPS = 26;                       // 64 KB of tables + 26 x (4 KB ring + 2 KB piece) of the 227 KB

struct ExpandFoArgs {
    PairView w[2];               // [1]: the up matrix of a gate/up pair (blockIdx.y picks the matrix)
    unsigned char * images;      // images of the range's first expert on
    const int32_t * bounds;      // of the range's first expert on
    int64_t unit0, units;        // units of the range
    int units_per_expert, C;
    int bands_per_block;         // 16 (plain) or 8 (one half of a gate/up pair)
    int blocks_per_expert;
};

__device__ __forceinline__ void stmatrix4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__global__ void __launch_bounds__(FO_EXPAND_WARPS * 32, 1) k_expand_tiles_fo(const ExpandFoArgs p, const Opaque k) {
    static_assert(FO_STEPS % AHEAD == 0 && AHEAD == 4, "the rings are topped up every four steps (32 codes), which is also the plane read-ahead");
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem; // four interleaved tables | per warp: 4 KB ring set | per warp: 2 KB piece
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const uint32_t lut_s = smem_u32(lut);
    const uint32_t lut_l = lut_s + (lane & 3) * 4;
    const uint32_t key = (lut_s + LUT_BYTES + (uint32_t) warp * (32 * RING_BYTES) + lane * RING_BYTES) | ((lane & 7) << 4);
    const uint32_t piece = lut_s + LUT_BYTES + (uint32_t) nwarp * (32 * RING_BYTES) + (uint32_t) warp * FO_STAGE;
    // stmatrix: lanes 8 i .. 8 i + 7 address the rows of matrix i = rows 8 (i & 1) .. of the band, 16-byte column i >> 1 of
    // the tile; tile j of the k-tile starts at 16-byte column 2 j, which under the 128-byte swizzle is one XOR
    const int mrow = (lane & 7) + 8 * ((lane >> 3) & 1);
    const uint32_t st0 = piece + (uint32_t) mrow * 128 + (uint32_t) (((lane >> 4) ^ (lane & 7)) << 4);
    const PairView w = blockIdx.y ? p.w[1] : p.w[0];
    const int row_offset = blockIdx.y ? IMG_ROWS / 2 : 0;
    for (int i = threadIdx.x; i < HP_MAX_PAIRS; i += blockDim.x) { const uint32_t e = __ldg(w.lut + i); ((uint4 *) lut)[i] = make_uint4(e, e, e, e); }
    grid_dependency_wait(); // the routing is an earlier kernel's, and the images may still be read by one
    __syncthreads();

    const int KT = p.C * 8;
    for (int64_t ur = (int64_t) blockIdx.x * nwarp + warp; ur < p.units; ur += (int64_t) gridDim.x * nwarp) {
        const int e = (int) (ur / p.units_per_expert), ue = (int) (ur - (int64_t) e * p.units_per_expert);
        if (ld_act_s32(p.bounds + e + 1) == ld_act_s32(p.bounds + e)) { continue; }
        const int64_t u = p.unit0 + ur;
        const int band = ue / p.C, slab = ue - band * p.C;
        const int nb = band / p.bands_per_block, img_row0 = (band - nb * p.bands_per_block) * FO_BAND + row_offset;
        unsigned char * img = p.images + (((int64_t) e * p.blocks_per_expert + nb) * KT + slab * 8) * (int64_t) IMG_KTILE_BYTES + img_row0 * 128;
        RingReader rd;
        {
            const uint32_t w0 = __ldg(w.ubase + u), l0 = __ldg(w.lrel + u * 32 + lane);
            rd.open((const uint8_t *) (w.stream + (w0 & ~3u)), ((w0 & 3u) + l0) * 4u, key, k);
        }
        cp_async_commit();
        const uint8_t * pl = w.plane + u * FO_UNIT_W + 16 * lane;
        uint4 nx[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) { nx[i] = ld_stream16(pl + i * CHUNK); }
        rd.token = cp_async_wait_all();
        rd.first_words();
#pragma unroll 1
        for (int t0 = 0; t0 < FO_STEPS; t0 += AHEAD) {
            if (t0) {
                rd.token = cp_async_wait_all(); // copies issued four steps ago
                rd.template top_up<3>(k);
                cp_async_commit();
            }
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int t = t0 + i;
                const uint4 sm = nx[i];
                nx[i] = ld_stream16(pl + (t + AHEAD < FO_STEPS ? t + AHEAD : t) * CHUNK); // the last steps re-read themselves: harmless L2 hits
                const uint32_t pw[4] = {sm.x, sm.y, sm.z, sm.w};
#pragma unroll
                for (int half = 0; half < 2; half++) { // tile 2 t + half
                    uint32_t en[4], wv[4];
                    rd.take2(lut_l, k, en[0], en[1]);
                    rd.take2(lut_l, k, en[2], en[3]);
                    wv[0] = merge_sm_exp(spread_lo(pw[2 * half]), en[0]);
                    wv[1] = merge_sm_exp(spread_hi(pw[2 * half]), en[1]);
                    wv[2] = merge_sm_exp(spread_lo(pw[2 * half + 1]), en[2]);
                    wv[3] = merge_sm_exp(spread_hi(pw[2 * half + 1]), en[3]);
                    if ((i & 1) == 0 && half == 0) { // the piece is written again: its last bulk store must have read it
                        if (lane == 0) { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
                        __syncwarp();
                    }
                    stmatrix4(st0 ^ (uint32_t) ((2 * (i & 1) + half) << 5), wv[0], wv[1], wv[2], wv[3]);
                }
                if (i & 1) { // four tiles: the piece of k-tile (t / 2) of the slab is complete
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                     ::"l"(img + (int64_t) (t >> 1) * IMG_KTILE_BYTES), "r"(piece), "n"(FO_STAGE) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            }
        }
    }
    if (lane == 0) { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
}

constexpr size_t FO_EXPAND_SMEM = LUT_BYTES + (size_t) FO_EXPAND_WARPS * (32 * RING_BYTES + FO_STAGE);

constexpr size_t EXPAND_SMEM = LUT_BYTES + (size_t) EXPAND_WARPS * 32 * RING_BYTES;

} // namespace

void expand_tiles_init() {
    const int optin = device_info().smem_optin;
    allow_dynamic_smem((const void *) k_expand_tiles<4, 8, true>, (int) EXPAND_SMEM, optin, "expand tiles");
    allow_dynamic_smem((const void *) k_expand_tiles<1, 16, false>, (int) EXPAND_SMEM, optin, "expand tiles");
    allow_dynamic_smem((const void *) k_expand_tiles_fo, (int) FO_EXPAND_SMEM, optin, "expand fragment-order tiles");
}

bool expand_tiles_supported(const bf16n_weight & w) {
    const int C = (int) (w.K / CHUNK);
    return w.format == FMT_HUFPAIR && !w.fo && w.K % CHUNK == 0 && ((C == 4 && w.R == 8 && w.cm) || (C == 1 && w.R == 16));
}

// Decodes every expert of `w` (and of `up`, the second matrix of a gate/up pair, in the same launch) that has routed
// pairs into its row-block images: 256-row blocks of a plain matrix, 128 + 128 rows of a pair.
void expand_tiles(const bf16n_weight & w, const bf16n_weight * up, int n_experts, const int32_t * bounds, void * images, cudaStream_t st) {
    ExpandArgs a = {};
    a.w[0] = pair_view(w);
    a.w[1] = up ? pair_view(*up) : a.w[0];
    a.images = (unsigned char *) images;
    a.bounds = bounds;
    a.units = w.rows / w.R;
    a.rows_per_expert = (int) (w.rows / n_experts);
    a.rows_per_block = up ? IMG_ROWS / 2 : IMG_ROWS;
    a.blocks_per_expert = a.rows_per_expert / a.rows_per_block;
    require(a.rows_per_expert % a.rows_per_block == 0, "rows per expert must be a multiple of the tensor-core pass's row block");
    const int n_mats = up ? 2 : 1;
    const unsigned gx = (unsigned) std::min<int64_t>(std::max(1, device_info().sms / n_mats), (a.units + EXPAND_WARPS - 1) / EXPAND_WARPS);
    const dim3 grid(gx, (unsigned) n_mats);
    const Opaque k = {1u, 4u, ~0u, 16u};
    // the first kernel of its call: behind whatever the caller launched (launch_behind)
    launch_behind(false, w.K == 4 * CHUNK ? k_expand_tiles<4, 8, true> : k_expand_tiles<1, 16, false>, grid, dim3(EXPAND_WARPS * 32), EXPAND_SMEM, st, a, k);
    check_launch();
}

// The same for experts [e0, e0 + n) of fragment-order matrices; `bounds` and `images` start at expert e0.
void expand_tiles_fo(const bf16n_weight & w, const bf16n_weight * up, int n_experts, int e0, int n, const int32_t * bounds, void * images,
                     cudaStream_t st, bool behind_own) {
    ExpandFoArgs a = {};
    a.w[0] = pair_view(w);
    a.w[1] = up ? pair_view(*up) : a.w[0];
    a.images = (unsigned char *) images;
    a.bounds = bounds;
    const int64_t rows_per_expert = w.rows / n_experts;
    const int rows_per_block = up ? IMG_ROWS / 2 : IMG_ROWS;
    require(rows_per_expert % rows_per_block == 0, "rows per expert must be a multiple of the tensor-core pass's row block");
    a.C = (int) (w.K / CHUNK);
    a.units_per_expert = (int) (rows_per_expert / FO_BAND) * a.C;
    a.unit0 = (int64_t) e0 * a.units_per_expert;
    a.units = (int64_t) n * a.units_per_expert;
    a.bands_per_block = rows_per_block / FO_BAND;
    a.blocks_per_expert = (int) (rows_per_expert / rows_per_block);
    const int n_mats = up ? 2 : 1;
    // units are dealt round robin: of the last few warp counts, the one that leaves the last round fullest (256 experts of 512 x
    // 2048: 17.03 rounds of 26 warps, 17.7 of 25)
    const int64_t blocks = std::max(1, device_info().sms / n_mats);
    int warps = FO_EXPAND_WARPS;
    double best = 0.0;
    for (int nw = FO_EXPAND_WARPS; nw >= FO_EXPAND_WARPS - 4; nw--) {
        const int64_t slots = blocks * nw, rounds = (a.units + slots - 1) / slots;
        const double full = (double) a.units / (double) (rounds * slots) * (1.0 - 0.005 * (FO_EXPAND_WARPS - nw));
        if (full > best + 1e-9) { best = full; warps = nw; }
    }
    const dim3 grid((unsigned) std::min<int64_t>(blocks, (a.units + warps - 1) / warps), (unsigned) n_mats);
    const Opaque k = {1u, 4u, ~0u, 16u};
    launch_behind(behind_own, k_expand_tiles_fo, grid, dim3(warps * 32), LUT_BYTES + (size_t) warps * (32 * RING_BYTES + FO_STAGE), st, a, k);
    check_launch();
}

} // namespace b16
