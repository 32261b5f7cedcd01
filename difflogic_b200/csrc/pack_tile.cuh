// Transpose-and-pack of a batch-major byte matrix t[batch][n] into feature-major bit rows, shared by the bool packer
// (packed.cu) and the thermometer packer (threshold_pack.cu).
//
// A thread owns eight adjacent features and reads eight samples of them at a time, eight bytes each.  No bit is moved on its
// own: every byte is compared with its threshold in place (bytes_above, four at a time), which leaves the answer in its top bit, and
// the answers of successive samples are shifted down the bytes: after eight samples byte f holds the samples' bits of feature f,
// which is the transposed order that is wanted.  Five instructions for four bytes.  (Squeezing a sample's answers together and
// transposing 8 x 8 bits afterwards took three times as many instructions; the packer waited for those and for the loads in turn.)
// Bound by memory: bool 784 x 2^20 226 -> 156 us (5.9 TB/s), uint8 3072 x 10000 with three thresholds 20.2 -> 13.1 us, 1021 x 2^18
// 260 -> 116 us.
//
// A CTA of 256 threads takes 8 * WF features x 8 * K * (256 / WF) samples: WF threads side by side over the features, each going
// through 8 * K samples.  The bytes meet in shared memory, so that a feature's samples leave as one run of K * 256 / WF bytes.
//   WF = 32, K = 1   256 features, 64 samples, one round of loads per thread: thousands of short CTAs
//   WF =  8, K = 4   64 features, 1024 samples, runs of 128 bytes: for matrices too narrow for 256 features, whose lanes would
//                    be idle, and for very long rows
//
// Rows of the source that do not start at 8-byte boundaries (n % 8 != 0) are read as three aligned 4-byte words and shifted
// into place; the words that hold the matrix's first and last byte are the only ones that reach beyond it, by less than 4 bytes.
// Rows of the output need no alignment (ragged ends go byte by byte).
#pragma once

#include "common.cuh"

namespace dl {

// Threshold t for bytes_above: what a byte's low seven bits need to reach bit 7, in every byte, and all ones for t < 128.
struct ByteThreshold {
    uint32_t add, either;
};
__host__ __device__ __forceinline__ ByteThreshold byte_threshold(int t) {
    return {(uint32_t)(127 - (t & 127)) * 0x01010101u, t < 128 ? 0xffffffffu : 0u};
}
// Top bit of every byte of v: whether the byte is above the threshold.  The low seven bits decide alone or, for t < 128, together with
// the top bit, which is enough then; for t >= 128 the top bit is needed as well.  Other bits: undefined.
__device__ __forceinline__ uint32_t bytes_above(uint32_t v, const ByteThreshold &t) {
    const uint32_t low = (v & 0x7f7f7f7fu) + t.add;
    return (low & v) | ((low | v) & t.either);
}

// r[i] byte j  <-  v[j] byte i   for four 32-bit values
__device__ __forceinline__ void transpose_bytes_4x4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t r[4]) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(c, d, 0x5140);  // a0 b0 a1 b1 | c0 d0 c1 d1
    const uint32_t t2 = __byte_perm(a, b, 0x7362), t3 = __byte_perm(c, d, 0x7362);  // a2 b2 a3 b3 | c2 d2 c3 d3
    r[0] = __byte_perm(t0, t1, 0x5410);
    r[1] = __byte_perm(t0, t1, 0x7632);
    r[2] = __byte_perm(t2, t3, 0x5410);
    r[3] = __byte_perm(t2, t3, 0x7632);
}

struct PackShape {
    int64_t n, batch, row_bytes;
};

// The eight bytes of features f .. f + 7 of one sample; features beyond n give any value.
template <bool ALIGNED>
__device__ __forceinline__ uint2 load_features(const uint8_t *__restrict__ p, int features) {
    if (ALIGNED) return __ldg(reinterpret_cast<const uint2 *>(p));
    const uint32_t off = (uint32_t)reinterpret_cast<uintptr_t>(p) & 3u;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(p - off);
    const uint32_t need = off + (uint32_t)features;  // a word is read only when it holds a byte that is wanted
    const uint32_t w0 = __ldg(w), w1 = need > 4 ? __ldg(w + 1) : 0u, w2 = need > 8 ? __ldg(w + 2) : 0u;
    return make_uint2(__funnelshift_r(w0, w1, 8 * off), __funnelshift_r(w1, w2, 8 * off));
}

// Eight samples from src on, `live` of which exist; the others count as zeros, which are above no threshold.
template <bool ALIGNED>
__device__ __forceinline__ void load_eight(const uint8_t *__restrict__ src, int64_t n, int features, int live, uint2 (&v)[8]) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        v[r] = make_uint2(0u, 0u);
        if (r < live) v[r] = load_features<ALIGNED>(src + (int64_t)r * n, features);
    }
}
// out[i] byte f = the eight samples' bits of feature f for threshold i.
template <int NT>
__device__ __forceinline__ void pack_eight(const uint2 (&v)[8], const ByteThreshold (&thr)[NT], unsigned long long (&out)[NT]) {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        uint32_t lo = 0u, hi = 0u;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            lo = lo >> 1 | (bytes_above(v[r].x, thr[i]) & 0x80808080u);
            hi = hi >> 1 | (bytes_above(v[r].y, thr[i]) & 0x80808080u);
        }
        out[i] = (unsigned long long)lo | ((unsigned long long)hi << 32);
    }
}

// Shared memory of a tile: [feature % 8][feature / 8, one more than WF][bytes of the run + 16], so that neither the writes, eight
// features apart, nor the 16-byte reads pile up on banks.
template <int WF, int K>
struct PackTile {
    static constexpr int kFeatures = 8 * WF, kRun = K * (kThreads / WF), kPitch = kRun + (kRun > 8 ? 16 : 0);
    static constexpr int kShared = 8 * (WF + 1) * kPitch;  // bytes
};

// Output i goes to the rows starting at dst + i * out_stride (row_bytes bytes per feature row).  Samples beyond the batch give
// zero bits.  fblk, sblk: which tile.
template <int NT, int WF, int K, bool ALIGNED>
__device__ __forceinline__ void pack_tile(const uint8_t *__restrict__ t, uint8_t *__restrict__ dst, int64_t out_stride, const PackShape &sh,
                                          int64_t fblk, int64_t sblk, uint8_t *s_bytes, const ByteThreshold (&thr)[NT]) {
    using Tile = PackTile<WF, K>;
    static_assert(K == 1 || K == 4, "a thread's bytes are written one or four at a time");
    const int group = threadIdx.x / WF, octet = threadIdx.x % WF;
    const int64_t f0 = fblk * Tile::kFeatures, f = f0 + octet * 8, byte0 = sblk * Tile::kRun, s0 = (byte0 + group * K) * 8;
    const int live = f < sh.n ? (int)max((int64_t)0, min((int64_t)(8 * K), sh.batch - s0)) : 0;
    const int features = (int)min((int64_t)8, sh.n - f);
    unsigned long long bits[K][NT];  // per round of 8 samples and output: byte f = the samples' bits of feature f
    const uint8_t *src = t + s0 * sh.n + f;
    if (live == 8 * K) {  // the next eight samples are on their way while eight are packed
        uint2 v[8];
        load_eight<ALIGNED>(src, sh.n, features, 8, v);
#pragma unroll
        for (int g = 0; g < K; ++g) {
            uint2 next[8];
            if (g + 1 < K) load_eight<ALIGNED>(src + (int64_t)(g + 1) * 8 * sh.n, sh.n, features, 8, next);
            pack_eight<NT>(v, thr, bits[g]);
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (g + 1 < K) v[r] = next[r];
        }
    } else {
#pragma unroll
        for (int g = 0; g < K; ++g) {
            uint2 v[8];
            load_eight<ALIGNED>(src + (int64_t)g * 8 * sh.n, sh.n, features, live - g * 8, v);
            pack_eight<NT>(v, thr, bits[g]);
        }
    }
    constexpr int kPiece = Tile::kRun >= 16 ? 16 : 8, kPieces = Tile::kRun / kPiece;
    const bool wide = sh.row_bytes % kPiece == 0 && (reinterpret_cast<uintptr_t>(dst) % kPiece) == 0 && out_stride % kPiece == 0;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        uint8_t *mine = s_bytes + octet * Tile::kPitch + group * K;
        if constexpr (K == 1) {
#pragma unroll
            for (int q = 0; q < 8; ++q) mine[q * (WF + 1) * Tile::kPitch] = (uint8_t)(bits[0][i] >> (8 * q));
        } else {
            uint32_t lo[4], hi[4];  // a feature's four bytes
            transpose_bytes_4x4((uint32_t)bits[0][i], (uint32_t)bits[1][i], (uint32_t)bits[2][i], (uint32_t)bits[3][i], lo);
            transpose_bytes_4x4((uint32_t)(bits[0][i] >> 32), (uint32_t)(bits[1][i] >> 32), (uint32_t)(bits[2][i] >> 32),
                                (uint32_t)(bits[3][i] >> 32), hi);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                *reinterpret_cast<uint32_t *>(mine + q * (WF + 1) * Tile::kPitch) = lo[q];
                *reinterpret_cast<uint32_t *>(mine + (q + 4) * (WF + 1) * Tile::kPitch) = hi[q];
            }
        }
        __syncthreads();
        uint8_t *rows = dst + (int64_t)i * out_stride;
        for (int idx = threadIdx.x; idx < Tile::kFeatures * kPieces; idx += kThreads) {
            const int fl = idx / kPieces, piece = idx % kPieces;
            if (f0 + fl >= sh.n) continue;
            const uint8_t *from = s_bytes + ((fl % 8) * (WF + 1) + fl / 8) * Tile::kPitch + piece * kPiece;
            uint8_t *to = rows + (f0 + fl) * sh.row_bytes + byte0 + piece * kPiece;
            const int64_t left = sh.row_bytes - (byte0 + piece * kPiece);
            if (left >= kPiece && wide) {
                if constexpr (kPiece == 16) *reinterpret_cast<uint4 *>(to) = *reinterpret_cast<const uint4 *>(from);
                else *reinterpret_cast<uint2 *>(to) = *reinterpret_cast<const uint2 *>(from);
            } else {
                for (int by = 0; by < kPiece && by < left; ++by) to[by] = from[by];
            }
        }
        __syncthreads();
    }
}

// Tile of a packer launch: kind 0 or 1 in the order of the list above.
template <int KIND>
using PackTileOf = PackTile<(KIND == 0 ? 32 : 8), (KIND == 0 ? 1 : 4)>;

struct PackGrid {
    int kind;
    dim3 grid;
};
// The 64 x 1024 tile once there are two of them per SM.  Measured (us, 64 x 1024 / 256 x 64; bool n x batch, in brackets the tiles):
// 784 x 1000 (13): 4.1 / 2.3; 784 x 10000 (130): 4.3 / 4.2; 783 x 10000 (130): 7.8 / 5.3; 256 x 2^17 (512): 6.0 / 8.0; 117 x 2^18 (512): 12.3 /
// 19.5; 1001 x 60000 (944): 18.6 / 18.0; 784 x 100000 (1274): 14.1 / 18.5; 784 x 2^20: 156 / 189; 30 x 2^20 (1024): 19 / 64; three
// thresholds: 1021 x 10000 (160): 11.0 / 9.0; 3072 x 10000 (480): 13.1 / 16.4.
static inline PackGrid pack_grid(const PackShape &sh) {
    auto grid = [&](int64_t features, int64_t bytes) {
        const int64_t sb = ceil_div(sh.row_bytes, bytes);
        return dim3((unsigned)ceil_div(sh.n, features), (unsigned)(sb < 65535 ? sb : 65535));
    };
    const PackGrid small = {0, grid(256, 8)}, large = {1, grid(64, 128)};
    const int64_t tiles = (int64_t)large.grid.x * large.grid.y;
    return tiles >= 2 * current_sms() ? large : small;
}

}  // namespace dl
