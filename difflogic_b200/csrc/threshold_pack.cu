// Thermometer encoding and bit packing in one pass, straight from uint8 features.
//
// The reference's image pipeline turns every pixel into T binary features (pixel / 255 > (i+1) / (T+1)),
// concatenated threshold-major (experiments/main.py:56-59), then PackBitsTensor transposes and packs the float
// or bool matrix (difflogic/packbitstensor.py:15-16).  For 2^20 samples that is gigabytes of intermediate bools.
// Here the uint8 matrix t[batch][n] is read once (for up to four thresholds at a time) and the packed rows
// out[i*n + f][word] come out directly: bit s of row i*n + f is  t[s][f] > thresholds[i].
//
// The tiles are those of pack_tile.cuh.
#include "common.cuh"
#include "pack_tile.cuh"

namespace dl {

constexpr int kMaxThresholds = 16;
struct Thresholds {
    unsigned char v[kMaxThresholds];
};

// NT thresholds per pass over the source: the pixels are read once for up to kThresholdsPerPass of them.
constexpr int kThresholdsPerPass = 4;

template <int NT, int KIND, bool ALIGNED>
__global__ void __launch_bounds__(kThreads, 2)
threshold_pack_kernel(const uint8_t *__restrict__ t, Thresholds thr, int first, uint8_t *__restrict__ out, PackShape sh) {
    using Tile = PackTileOf<KIND>;
    __shared__ __align__(16) uint8_t s_bytes[Tile::kShared];
    ByteThreshold above[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) above[i] = byte_threshold(thr.v[first + i]);
    uint8_t *dst = out + (int64_t)first * sh.n * sh.row_bytes;
    for (int64_t sblk = blockIdx.y; sblk * Tile::kRun < sh.row_bytes; sblk += gridDim.y)
        pack_tile<NT, Tile::kFeatures / 8, KIND == 0 ? 1 : 4, ALIGNED>(t, dst, sh.n * sh.row_bytes, sh, blockIdx.x, sblk, s_bytes, above);
}

template <int NT, bool ALIGNED>
static void launch_threshold_pack(const PackGrid &g, const uint8_t *t, const Thresholds &thr, int first, uint8_t *out, const PackShape &sh,
                                  cudaStream_t st) {
    switch (g.kind) {
        case 0: threshold_pack_kernel<NT, 0, ALIGNED><<<g.grid, kThreads, 0, st>>>(t, thr, first, out, sh); break;
        default: threshold_pack_kernel<NT, 1, ALIGNED><<<g.grid, kThreads, 0, st>>>(t, thr, first, out, sh); break;
    }
}
template <bool ALIGNED>
static void launch_thresholds(const PackGrid &g, const uint8_t *t, const Thresholds &thr, int count, uint8_t *out, const PackShape &sh,
                              cudaStream_t st) {
    for (int first = 0; first < count; first += kThresholdsPerPass) {
        switch (count - first < kThresholdsPerPass ? count - first : kThresholdsPerPass) {
            case 1: launch_threshold_pack<1, ALIGNED>(g, t, thr, first, out, sh, st); break;
            case 2: launch_threshold_pack<2, ALIGNED>(g, t, thr, first, out, sh, st); break;
            case 3: launch_threshold_pack<3, ALIGNED>(g, t, thr, first, out, sh, st); break;
            default: launch_threshold_pack<4, ALIGNED>(g, t, thr, first, out, sh, st); break;
        }
    }
}

}  // namespace dl

using namespace dl;

extern "C" DL_API int dl_threshold_packbits_batch_major(const uint8_t *t, const uint8_t *thresholds, int n_thresholds, void *out,
                                                        int64_t n, int64_t batch, int bit_count, void *stream) {
    DL_REQUIRE(bit_count == 8 || bit_count == 16 || bit_count == 32 || bit_count == 64 || bit_count == 128, DL_ERR_BAD_BIT_COUNT,
               "dl_threshold_packbits_batch_major: `bit_count` has to be in { 8, 16, 32, 64, 128 }, got %d", bit_count);
    DL_REQUIRE(n >= 0 && batch >= 0, DL_ERR_INVALID_ARG, "dl_threshold_packbits_batch_major: negative size");
    DL_REQUIRE(thresholds != nullptr && n_thresholds >= 1 && n_thresholds <= kMaxThresholds, DL_ERR_INVALID_ARG,
               "dl_threshold_packbits_batch_major: between 1 and %d thresholds (a host array)", kMaxThresholds);
    if (n == 0 || batch == 0) return DL_OK;
    DL_REQUIRE(t && out, DL_ERR_INVALID_ARG, "dl_threshold_packbits_batch_major: null pointer");
    Thresholds thr;
    for (int i = 0; i < kMaxThresholds; ++i) thr.v[i] = i < n_thresholds ? thresholds[i] : 0;
    const int64_t row_bytes = ceil_div(batch, bit_count) * (bit_count / 8);
    uint8_t *o = reinterpret_cast<uint8_t *>(out);
    const PackShape sh = {n, batch, row_bytes};
    if (n % 8 == 0 && aligned_to(t, 8)) launch_thresholds<true>(pack_grid(sh), t, thr, n_thresholds, o, sh, as_stream(stream));
    else launch_thresholds<false>(pack_grid(sh), t, thr, n_thresholds, o, sh, as_stream(stream));
    return launch_status("dl_threshold_packbits_batch_major");
}
