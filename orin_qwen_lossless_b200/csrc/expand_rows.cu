// Exact reconstruction of lane-major pair-Huffman matrices (dequantise for a prompt's GEMM, verify at load) with the ring
// reader of the large-matrix decode GEMV: one unit per warp, streams through per-lane cp.async rings, plane bytes four
// steps ahead. What bounds it depends on the matrix: one with a few hundred units (8192 x 2048, R = 16: 512) is one chain
// of R K / 64 dependent table lookups per lane, and reading the streams and the plane lane by lane from global memory
// inside that chain (k_pair_expand) more than doubled it (8192 x 2048: 71 us, here 26, warm); a matrix with many units is bound by
// HBM and the table's bank conflicts.
// Units are dealt over the blocks first and the warps of a block second, so that few units reach every SM.
#include "launch.h"
#include "rings.cuh"
#include "sinks.cuh"

namespace b16 {
namespace {

using namespace dev;
using namespace ring;

constexpr int ROW_WARPS = 28, AHEAD = 4;
constexpr size_t ROW_SMEM = LUT_BYTES + (size_t) ROW_WARPS * 32 * RING_BYTES;

template <typename Sink>
__global__ void __launch_bounds__(ROW_WARPS * 32, 1) k_expand_rows(const PairView w, int C, int R, bool cm, int64_t row0, int64_t units, const Sink sink_in,
                                                                   const ring::Opaque k) {
    Sink sink = sink_in;
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t * lut = (uint32_t *) smem; // four interleaved tables | one 4 KB ring set per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const uint32_t lut_s = ring::smem_u32(lut);
    const uint32_t lut_l = lut_s + (lane & 3) * 4;
    const uint32_t key = (lut_s + LUT_BYTES + (uint32_t) warp * (32 * RING_BYTES) + lane * RING_BYTES) | ((lane & 7) << 4);
    for (int i = threadIdx.x; i < HP_MAX_PAIRS; i += blockDim.x) { const uint32_t e = __ldg(w.lut + i); ((uint4 *) lut)[i] = make_uint4(e, e, e, e); }
    __syncthreads();
    const int steps = R * C; // of 512 weights, in stream and plane order; a multiple of AHEAD
    for (int64_t u = (int64_t) warp * gridDim.x + blockIdx.x; u < units; u += (int64_t) gridDim.x * nwarp) {
        const int64_t gu = row0 / R + u;
        RingReader rd;
        {
            const uint32_t w0 = __ldg(w.ubase + gu), l0 = __ldg(w.lrel + gu * 32 + lane);
            rd.open((const uint8_t *) (w.stream + (w0 & ~3u)), ((w0 & 3u) + l0) * 4u, key, k);
        }
        cp_async_commit();
        const uint8_t * pl = w.plane + gu * R * ((int64_t) C * CHUNK) + 16 * lane;
        uint4 nx[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) { nx[i] = ld_stream16(pl + i * CHUNK); }
        rd.token = cp_async_wait_all();
        rd.first_words();
        int rr = 0, c = 0;
#pragma unroll 1
        for (int t0 = 0; t0 < steps; t0 += AHEAD) {
            if (t0) {
                rd.token = cp_async_wait_all(); // copies issued four steps (32 codes) ago
                rd.template top_up<3>(k);
                cp_async_commit();
            }
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int t = t0 + i;
                const uint4 sm = nx[i];
                nx[i] = ld_stream16(pl + (t + AHEAD < steps ? t + AHEAD : t) * CHUNK); // the last steps re-read themselves
                uint32_t e[8], wv[8];
#pragma unroll
                for (int q = 0; q < 8; q += 2) { rd.take2(lut_l, k, e[q], e[q + 1]); }
                assemble8(sm, e, wv);
                sink.chunk(u * R + rr, c, lane, wv);
                if (cm) { if (++rr == R) { rr = 0; c++; } } else { if (++c == C) { c = 0; rr++; } }
            }
        }
    }
    sink.finish(lane);
}

template <typename Sink>
void launch(const bf16n_weight & w, int64_t row0, int64_t nrows, const Sink & sink, cudaStream_t st) {
    const int64_t units = nrows / w.R, sms = device_info().sms;
    if (units == 0) { return; }
    const int warps = (int) std::min<int64_t>(ROW_WARPS, std::max<int64_t>((units + sms - 1) / sms, 8)); // eight stage the tables
    const unsigned blocks = (unsigned) std::min(sms, units);
    const ring::Opaque k = {1u, 4u, ~0u, 16u};
    k_expand_rows<Sink><<<blocks, warps * 32, LUT_BYTES + (size_t) warps * 32 * RING_BYTES, st>>>(pair_view(w), (int) (w.K / CHUNK), w.R, w.cm != 0, row0,
                                                                                                units, sink, k);
    check_launch();
}

} // namespace

void expand_rows_init() {
    const int optin = device_info().smem_optin;
    allow_dynamic_smem((const void *) k_expand_rows<StoreBF16>, (int) ROW_SMEM, optin, "expand rows");
    allow_dynamic_smem((const void *) k_expand_rows<CompareBF16>, (int) ROW_SMEM, optin, "expand rows");
}

// Opening a unit costs the rings a trip to memory that only the unit's own steps hide, and 28 warps per SM hide less of it than
// the general kernel's 64; so short units take the rings only while the call has few of them. General / rings in us by steps
// of 512 weights to a unit and units of the call: 4 steps: 4.8 / 4.5 for 256 units, 5.8 / 5.6 for 1024, 5.9 / 6.9 for 2048,
// 44 / 63 for 32768; 8 steps: 12.4 / 9.1 for 2048, 14.7 / 14.1 for 4096, 23.2 / 24.3 for 8192, 84.5 / 95.7 for 32768; 16 steps: 20.9 / 12.7
// for 2048, 46.3 / 48.0 for 8192, 95.1 / 90.7 for 16384; 32 steps: 27.8 / 16.1 for 1024, 58.5 / 44.6 for 4096, 218 / 177 for 16384.
bool expand_rows_applies(const bf16n_weight & w, int64_t nrows) {
    const int64_t steps = w.R * (w.K / CHUNK);
    if (w.format != FMT_HUFPAIR || w.fo || steps % AHEAD) { return false; }
    const int64_t units = nrows / w.R, round = (int64_t) ROW_WARPS * device_info().sms;
    return steps >= 32 || units <= (steps == 4 ? round / 4 : round) || (steps == 16 && units >= 3 * round);
}

void expand_rows(const bf16n_weight & w, int64_t row0, int64_t nrows, const StoreBF16 & sink, cudaStream_t st) { launch(w, row0, nrows, sink, st); }
void expand_rows(const bf16n_weight & w, int64_t row0, int64_t nrows, const CompareBF16 & sink, cudaStream_t st) { launch(w, row0, nrows, sink, st); }

} // namespace b16
