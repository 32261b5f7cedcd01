// Packed networks too wide for shared memory, layer by layer over the gates that folding leaves (fold.cu).
//
// Every gate that is left has a row in one POOL, layers one after the other; a gate reads rows of the pool or of the packed
// input, from whichever layer its inputs come, so rows that a layer only hands on are neither moved nor stored.  The kernels are
// those for whole layers (eval_rows), over shorter lists; the last layer keeps all of its neurons, in order, because its rows or
// class counts are wanted, with the gates in terms of pool rows: constants read nothing and copies one row.  Where the counts are
// wanted, a table by class (one per number of classes) leaves the constants out: what the counting kernel takes goes by its
// neurons, whatever they read.
//
// Bound by memory as before, with fewer rows: 256 -> 12 x 64000, 2^17 samples 4340 -> 1190 us (12 x 64000 neurons of which 139000 are
// left as gates); 9216 -> 4 x 128000, 10000 samples, with the packing 289 -> 195 us.
#include "fold.cuh"
#include "gates.cuh"

namespace dl {

int eval_rows(const SplitRows &x, const int64_t *a, const int64_t *b, const uint8_t *gate, void *y, int64_t n_in, int64_t n_out,
              int64_t row_bytes, cudaStream_t st);                                                   // packed.cu
int eval_class_counts(const SplitRows &x, const int64_t *a, const int64_t *b, const uint8_t *gate, int32_t *out, int64_t row_bytes,
                      int64_t batch, int64_t k, const ClassRows &classes, bool in_parts, cudaStream_t st);  // eval_groupbitsum.cu
bool class_counts_in_parts(int64_t m);

// The lists: gates that are left by place, then the last layer's neurons.
struct GateList {
    int64_t *a, *b;
    uint8_t *gate;
};

__global__ void __launch_bounds__(kThreads)
fold_emit_kernel(int n0, int hidden, int tail, const int32_t *__restrict__ ref, const int32_t *__restrict__ in_a, const int32_t *__restrict__ in_b,
                 const int32_t *__restrict__ use, const int32_t *__restrict__ row, GateList list) {
    const int j = blockIdx.x * kThreads + threadIdx.x;  // neuron, counted through all layers
    if (j >= hidden + tail) return;
    const int vb = __ldg(in_b + j);
    int op = vb >> kFoldValueBits;
    auto place = [&](int v) { return (int64_t)(v < n0 ? v : n0 + __ldg(row + v)); };
    int64_t at = j, a = 0, b = 0;
    if (op != 0) {
        if (j < hidden) {
            if (__ldg(use + n0 + j) == 0) return;
            at = __ldg(row + n0 + j);
        } else if (__ldg(ref + j) & 1) {
            op ^= 15;
        }
        a = place(__ldg(in_a + j));
        b = place(vb & ((1 << kFoldValueBits) - 1));
    } else {
        if (j < hidden) return;
        const int r = __ldg(ref + j);
        op = (r & 1) ? 15 : 0;
        if (!ref_is_constant(r)) {
            op ^= 3;
            a = b = place(r >> 1);
        }
    }
    list.a[at] = a;
    list.b[at] = b;
    list.gate[at] = (uint8_t)op;
}

static GateList gate_list(const FoldShape &sh, void *lists) {
    const int64_t neurons = sh.first[sh.layers + 1] - sh.n[0];
    GateList l;
    l.a = reinterpret_cast<int64_t *>(lists);
    l.b = l.a + neurons;
    l.gate = reinterpret_cast<uint8_t *>(l.b + neurons);
    return l;
}

// Neurons of the last layer by class, without constants.
struct TailTable {
    GateList list;
    int32_t *start, *longest, *ones, *count, *rank;  // [k + 1], [1], [k], [k], by neuron
};
static int64_t tail_table(int64_t n, int64_t k, TailTable *t, void *at) {
    t->list.a = reinterpret_cast<int64_t *>(at);
    t->list.b = t->list.a + n;
    t->longest = reinterpret_cast<int32_t *>(t->list.b + n);  // at byte 16 n, as the header says
    t->start = t->longest + 1;
    t->ones = t->start + k + 1;
    t->count = t->ones + k;
    t->rank = t->count + k;
    t->list.gate = reinterpret_cast<uint8_t *>(t->rank + n);
    return 21 * n + 4 * (3 * k + 2);
}

__global__ void __launch_bounds__(kThreads)
tail_count_kernel(TailTable t, int n, int rows_per_class, const uint8_t *__restrict__ gate) {
    grid_dependents_launch();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    const int op = j < n ? gate[j] : 0, c = j < n ? j / rows_per_class : 0;
    // a warp's neurons are mostly of one class: one addition for all
    const bool one = __all_sync(0xffffffffu, c == __shfl_sync(0xffffffffu, c, 0) || j >= n);
    const bool counts = op != 0 && op != 15;
    const unsigned listed = __ballot_sync(0xffffffffu, counts), lane = threadIdx.x % 32;
    if (one) {
        const unsigned always = __ballot_sync(0xffffffffu, op == 15);
        int base = 0;
        if (lane == 0) {
            if (listed) base = atomicAdd(t.count + c, __popc(listed));
            if (always) atomicAdd(t.ones + c, __popc(always));
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        if (counts) t.rank[j] = base + __popc(listed & ((1u << lane) - 1u));
    } else if (counts) {
        t.rank[j] = atomicAdd(t.count + c, 1);
    } else if (op == 15) {
        atomicAdd(t.ones + c, 1);
    }
}

__global__ void __launch_bounds__(1024)
tail_start_kernel(TailTable t, int k) {
    __shared__ int s_sum[1024], s_most;
    grid_dependency_wait();
    grid_dependents_launch();
    const int tid = threadIdx.x, each = (k + 1023) / 1024;
    if (tid == 0) s_most = 0;
    int mine = 0, most = 0;
    for (int c = tid * each; c < min(k, (tid + 1) * each); ++c) {
        mine += __ldcg(t.count + c);
        most = max(most, __ldcg(t.count + c));
    }
    s_sum[tid] = mine;
    __syncthreads();
    atomicMax(&s_most, most);
    for (int d = 1; d < 1024; d <<= 1) {
        const int v = tid >= d ? s_sum[tid - d] : 0;
        __syncthreads();
        s_sum[tid] += v;
        __syncthreads();
    }
    int at = s_sum[tid] - mine;
    for (int c = tid * each; c < min(k, (tid + 1) * each); ++c) {
        t.start[c] = at;
        at += __ldcg(t.count + c);
    }
    if (tid == 1023) {
        t.start[k] = s_sum[tid];
        *t.longest = s_most;
    }
}

__global__ void __launch_bounds__(kThreads)
tail_place_kernel(TailTable t, int n, int rows_per_class, GateList from) {
    grid_dependency_wait();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= n) return;
    const int op = from.gate[j];
    if (op == 0 || op == 15) return;
    const int at = __ldcg(t.start + j / rows_per_class) + t.rank[j];
    t.list.a[at] = from.a[j];
    t.list.b[at] = from.b[j];
    t.list.gate[at] = (uint8_t)op;
}

// ---------------------------------------------------------------------------------------------
// class counts of a folded last layer
// ---------------------------------------------------------------------------------------------
// A CTA takes (512 bytes of the rows, class, part of its neurons), a warp an eighth of those: lane l holds 16 bytes of the columns and
// adds the gates' outputs up bit by bit (carry-save, eight neurons at a time); the sixteen loads of eight neurons are in flight at
// once, straight into registers.  What a warp needs to know of 32 neurons lies in shared memory.  At the end the eight warps' sums meet
// there, as planes, and become integers that are stored, or added where a class has several parts.
//
// eval_groupbitsum_kernel stages rows in shared memory for eight neurons at a time and takes its 1.2 us for them whatever the length of
// the rows, from 512 bytes on; its 2 KB pieces suit long rows.  Whole folded passes, us, that kernel / this one: 9216 -> 4 x 128000, rows of
// 576 bytes 135 / 108, 1264 158 / 138, 4096 364 / 352; 256 -> 12 x 64000, 4096 277 / 273, 16384 1027 / 1028; 784 -> 2 x 20000, 1264 42 / 29, 16384
// 130 / 142; 784 -> 5 x 32000 in 100 classes, 1264 70 / 61, 16384 423 / 453.
constexpr int64_t kTailLongest = 4096;  // bytes of a row
constexpr int kTailWarps = kThreads / 32, kTailPlanes = 10, kTailShare = (1 << kTailPlanes) - 1;  // neurons of a warp at most
constexpr int kTailSum = kTailPlanes + 3;                                                          // planes of a CTA's sums
constexpr uint32_t kTailMore = 1u << 31;  // of an offset: in the second buffer

__global__ void __launch_bounds__(kThreads, 2)
tail_counts_kernel(const SplitRows x, const int64_t *__restrict__ a, const int64_t *__restrict__ b, const uint8_t *__restrict__ gate,
                   const int32_t *__restrict__ start, const int32_t *__restrict__ ones, int32_t *__restrict__ out, int64_t row_bytes,
                   int64_t batch, int k, int parts) {
    __shared__ uint4 s_mask[kTailWarps][32];
    __shared__ uint2 s_row[kTailWarps][32];                 // offsets of both inputs, in 16-byte units
    __shared__ uint32_t s_plane[kTailWarps][kTailPlanes][128];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int c = blockIdx.x % k, part = blockIdx.x / k;
    const int64_t col = (int64_t)blockIdx.y * 512 + lane * 16;
    const bool live = col < row_bytes;
    const int begin = __ldg(start + c), len = __ldg(start + c + 1) - begin;
    const int from = begin + (int)((int64_t)len * part / parts), to = begin + (int)((int64_t)len * (part + 1) / parts);
    const int mine = from + (int)((int64_t)(to - from) * warp / kTailWarps), end = from + (int)((int64_t)(to - from) * (warp + 1) / kTailWarps);
    const int64_t units = row_bytes / 16;
    const uint4 *base = reinterpret_cast<const uint4 *>(x.x + col), *more = reinterpret_cast<const uint4 *>(x.more + col);

    uint32_t p[4][kTailPlanes];
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
        for (int i = 0; i < kTailPlanes; ++i) p[w][i] = 0u;
    for (int j0 = mine; j0 < end; j0 += 32) {
        {
            const int j = j0 + lane;
            uint2 rows = make_uint2(0u, 0u);
            GateMasks m = {0u, 0u, 0u, 0u};
            if (j < end) {
                const int64_t ia = __ldg(a + j), ib = __ldg(b + j);
                rows.x = ia < x.split ? (uint32_t)(ia * units) : (uint32_t)((ia - x.split) * units) | kTailMore;
                rows.y = ib < x.split ? (uint32_t)(ib * units) : (uint32_t)((ib - x.split) * units) | kTailMore;
                m = gate_masks(__ldg(gate + j));
            }
            __syncwarp();
            s_row[warp][lane] = rows;
            s_mask[warp][lane] = make_uint4(m.m0, m.ma, m.mb, m.mab);
            __syncwarp();
        }
        const int here = min(32, end - j0);
        for (int g = 0; g < here; g += 8) {
            uint4 va[8], vb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint2 r = s_row[warp][g + i];
                const uint4 m = s_mask[warp][g + i];
                va[i] = vb[i] = make_uint4(0u, 0u, 0u, 0u);
                if ((m.y | m.w) != 0u && live) va[i] = __ldg((r.x & kTailMore ? more : base) + (r.x & ~kTailMore));
                if ((m.z | m.w) != 0u && live) vb[i] = __ldg((r.y & kTailMore ? more : base) + (r.y & ~kTailMore));
            }
            uint32_t two[4], four[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 m0 = s_mask[warp][g + 2 * q], m1 = s_mask[warp][g + 2 * q + 1];
                const uint32_t a0[4] = {va[2 * q].x, va[2 * q].y, va[2 * q].z, va[2 * q].w}, b0[4] = {vb[2 * q].x, vb[2 * q].y, vb[2 * q].z, vb[2 * q].w};
                const uint32_t a1[4] = {va[2 * q + 1].x, va[2 * q + 1].y, va[2 * q + 1].z, va[2 * q + 1].w},
                               b1[4] = {vb[2 * q + 1].x, vb[2 * q + 1].y, vb[2 * q + 1].z, vb[2 * q + 1].w};
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const uint32_t v0 = gate32(a0[w], b0[w], {m0.x, m0.y, m0.z, m0.w}), v1 = gate32(a1[w], b1[w], {m1.x, m1.y, m1.z, m1.w});
                    uint32_t t, f;
                    DL_CSA32(t, p[w][0], p[w][0], v0, v1);
                    if (q % 2 == 0) {
                        two[w] = t;
                    } else {
                        DL_CSA32(f, p[w][1], p[w][1], two[w], t);
                        if (q == 1) {
                            four[w] = f;
                        } else {
                            uint32_t carry;
                            DL_CSA32(carry, p[w][2], p[w][2], four[w], f);
#pragma unroll
                            for (int i = 3; i < kTailPlanes; ++i) {
                                const uint32_t n = p[w][i] & carry;
                                p[w][i] ^= carry;
                                carry = n;
                            }
                        }
                    }
                }
            }
        }
    }
    // ---- the warps' sums meet; a thread adds up those of one word of 32 samples and takes half of the samples on ----
#pragma unroll
    for (int i = 0; i < kTailPlanes; ++i) *reinterpret_cast<uint4 *>(&s_plane[warp][i][lane * 4]) = make_uint4(p[0][i], p[1][i], p[2][i], p[3][i]);
    __syncthreads();
    const int word = tid % 128, first = tid / 128 * 16;
    const int64_t s0 = ((int64_t)blockIdx.y * 512 + word * 4) * 8 + first;
    if (s0 >= batch) return;
    uint32_t sum[kTailSum];
#pragma unroll
    for (int i = 0; i < kTailSum; ++i) sum[i] = 0u;
#pragma unroll
    for (int r = 0; r < kTailWarps; ++r) {
        uint32_t carry = 0u;
#pragma unroll
        for (int i = 0; i < kTailSum; ++i) {
            uint32_t h, l;
            DL_CSA32(h, l, sum[i], i < kTailPlanes ? s_plane[r][i][word] : 0u, carry);
            sum[i] = l;
            carry = h;
        }
    }
    const int always = part == 0 ? __ldg(ones + c) : 0;
    int32_t *dst = out + s0 * k + c;
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // four samples: a nibble of each plane -> a bit in each of four bytes
        uint32_t low = 0u, high = 0u;
#pragma unroll
        for (int i = 0; i < kTailSum; ++i) {
            const uint32_t bits = (((sum[i] >> (first + 4 * q)) & 15u) * 0x00204081u) & 0x01010101u;
            if (i < 8) low |= bits << i;
            else high |= bits << (i - 8);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int count = (int)((low >> (8 * i)) & 255u) + ((int)((high >> (8 * i)) & 255u) << 8) + always;
            if (s0 + 4 * q + i < batch) {
                if (parts == 1) dst[(int64_t)(4 * q + i) * k] = count;
                else if (count != 0) atomicAdd(dst + (int64_t)(4 * q + i) * k, count);
            }
        }
    }
}

}  // namespace dl

using namespace dl;

extern "C" DL_API int64_t dl_fold_layers_bytes(const int64_t *n, int layers) {
    FoldShape sh;
    if (!fold_shape(n, layers, &sh)) return 0;
    return 17 * ((int64_t)sh.first[layers + 1] - sh.n[0]);
}
extern "C" DL_API int64_t dl_fold_scratch_bytes(const int64_t *n, int layers) {
    FoldShape sh;
    return fold_shape(n, layers, &sh) ? 4 * fold_words(sh) : 0;
}

extern "C" DL_API int dl_fold_layers(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n, int layers,
                                     void *lists, void *scratch, void *stream) {
    FoldShape sh;
    DL_REQUIRE(a && b && gate && n && lists && scratch && aligned_to(lists, 16) && aligned_to(scratch, 16), DL_ERR_INVALID_ARG,
               "dl_fold_layers: null or unaligned pointer");
    DL_REQUIRE(fold_shape(n, layers, &sh), DL_ERR_TOO_LARGE, "dl_fold_layers: 1 .. %d layers of fewer than 2^27 rows in all", kFoldLayers);
    for (int l = 0; l < layers; ++l) DL_REQUIRE(a[l] && b[l] && gate[l], DL_ERR_INVALID_ARG, "dl_fold_layers: null pointer");
    const FoldScratch s = fold_scratch(sh, reinterpret_cast<int32_t *>(scratch));
    if (int e = fold_network(sh, a, b, gate, s, true, as_stream(stream))) return e;
    const int tail = sh.n[layers], hidden = sh.first[layers + 1] - sh.n[0] - tail;
    fold_emit_kernel<<<(unsigned)ceil_div(hidden + tail, kThreads), kThreads, 0, as_stream(stream)>>>(sh.n[0], hidden, tail, s.ref, s.in_a, s.in_b,
                                                                                                      s.use, s.row, gate_list(sh, lists));
    return launch_status("dl_fold_layers");
}

extern "C" DL_API int64_t dl_fold_tail_bytes(const int64_t *n, int layers, int64_t k) {
    FoldShape sh;
    TailTable t;
    if (!fold_shape(n, layers, &sh) || k < 1 || n[layers] % k != 0) return 0;
    return tail_table(n[layers], k, &t, nullptr);
}
extern "C" DL_API int dl_fold_tail(const void *lists, const int64_t *n, int layers, int64_t k, void *table, void *stream) {
    FoldShape sh;
    TailTable t;
    DL_REQUIRE(lists && n && table && aligned_to(lists, 16) && aligned_to(table, 16), DL_ERR_INVALID_ARG, "dl_fold_tail: null or unaligned pointer");
    DL_REQUIRE(fold_shape(n, layers, &sh) && k >= 1 && n[layers] % k == 0, DL_ERR_INVALID_ARG, "dl_fold_tail: bad sizes");
    const int rows = sh.n[layers], rows_per_class = (int)(rows / k);
    tail_table(rows, k, &t, table);
    GateList list = gate_list(sh, const_cast<void *>(lists));
    const int64_t tail = sh.first[layers] - sh.n[0];
    list.a += tail;
    list.b += tail;
    list.gate += tail;
    cudaStream_t st = as_stream(stream);
    if (cudaMemsetAsync(t.ones, 0, (size_t)(2 * k) * sizeof(int32_t), st) != cudaSuccess) return launch_status("dl_fold_tail (clear)");
    const dim3 grid((unsigned)ceil_div(rows, kThreads));
    launch_dependent(false, tail_count_kernel, grid, dim3(kThreads), 0, st, t, rows, rows_per_class, (const uint8_t *)list.gate);
    launch_dependent(true, tail_start_kernel, dim3(1), dim3(1024), 0, st, t, (int)k);
    launch_dependent(true, tail_place_kernel, grid, dim3(kThreads), 0, st, t, rows, rows_per_class, list);
    return launch_status("dl_fold_tail");
}

extern "C" DL_API int dl_eval_folded(const void *x, const void *lists, const int64_t *n, const int32_t *left, int layers, void *pool,
                                     const void *table, int64_t longest, int32_t *out, void *rows_out, int64_t row_bytes, int64_t batch,
                                     int64_t k, void *stream) {
    const char *who = "dl_eval_folded";
    FoldShape sh;
    DL_REQUIRE(x && lists && n && left && (out != nullptr) != (rows_out != nullptr) && aligned_to(lists, 16), DL_ERR_INVALID_ARG, "%s: null pointer", who);
    DL_REQUIRE(fold_shape(n, layers, &sh) && row_bytes > 0 && batch > 0 && batch <= row_bytes * 8 && k > 0 && n[layers] % k == 0,
               DL_ERR_INVALID_ARG, "%s: bad sizes", who);
    int64_t rows = 0;
    for (int l = 1; l < layers; ++l) {
        DL_REQUIRE(left[l] >= 0 && left[l] <= n[l], DL_ERR_INVALID_ARG, "%s: layer %d has more gates left than neurons", who, l);
        rows += left[l];
    }
    DL_REQUIRE(pool != nullptr || rows == 0, DL_ERR_INVALID_ARG, "%s: null pointer", who);
    const int64_t m = n[layers] / k;
    DL_REQUIRE(out == nullptr || (table && aligned_to(table, 16) && longest >= 0 && longest <= m), DL_ERR_INVALID_ARG, "%s: counts need a table", who);
    const bool staged = aligned_to(pool, 16) && (dl_eval_groupbitsum_applicable(x, n[0], n[layers], row_bytes, 8, k) == 1 ||
                                                 dl_eval_groupbitsum_parts_applicable(x, n[0], n[layers], row_bytes, 8, k) == 1);
    const int64_t most_rows = rows > n[0] ? rows : n[0];
    const bool direct = row_bytes % 16 == 0 && aligned_to(x, 16) && aligned_to(pool, 16) && most_rows * (row_bytes / 16) <= INT32_MAX &&
                        ceil_div(row_bytes, 512) <= 65535 && k * (ceil_div(m, 64) + 1) <= INT32_MAX;
    DL_REQUIRE(out == nullptr || staged || direct, DL_ERR_INVALID_ARG, "%s: rows whose classes no kernel counts", who);
    const GateList list = gate_list(sh, const_cast<void *>(lists));
    const SplitRows src = {reinterpret_cast<const uint8_t *>(x), reinterpret_cast<const uint8_t *>(pool), n[0]};
    int64_t at = rows;  // the first layer's gates come last
    for (int l = 1; l < layers; ++l) {
        at -= left[l];
        if (left[l] == 0) continue;
        if (int e = eval_rows(src, list.a + at, list.b + at, list.gate + at, reinterpret_cast<uint8_t *>(pool) + at * row_bytes, n[l - 1], left[l],
                              row_bytes, as_stream(stream)))
            return e;
    }
    const int64_t tail = sh.first[layers] - sh.n[0];
    if (out != nullptr) {
        TailTable t;
        tail_table(n[layers], k, &t, const_cast<void *>(table));
        const ClassRows classes = {t.start, t.ones, longest > 0 ? (int)longest : 1};
        if (direct && (!staged || row_bytes <= kTailLongest)) {
            // parts: as many as leave the busiest of the CTAs that run at a time (two per SM) the fewest neurons; 200: what a part costs besides
            const int64_t blocks = ceil_div(row_bytes, 512), slots = 2 * current_sms(), fewest = ceil_div(classes.m, kTailShare * kTailWarps);
            int64_t parts = fewest, least = 0;
            for (int64_t p = fewest; p <= fewest + 64 && (p == fewest || p <= classes.m / 64); ++p) {
                const int64_t cost = ceil_div(blocks * k * p, slots) * (ceil_div(classes.m, p) + 200);
                if (least == 0 || cost < least) {
                    least = cost;
                    parts = p;
                }
            }
            cudaStream_t st = as_stream(stream);
            if (parts > 1 && cudaMemsetAsync(out, 0, (size_t)batch * k * sizeof(int32_t), st) != cudaSuccess)
                return launch_status("dl_eval_folded (clear)");
            tail_counts_kernel<<<dim3((unsigned)(k * parts), (unsigned)blocks), kThreads, 0, st>>>(
                src, t.list.a, t.list.b, t.list.gate, t.start, t.ones, out, row_bytes, batch, (int)k, (int)parts);
            return launch_status("dl_eval_folded");
        }
        return eval_class_counts(src, t.list.a, t.list.b, t.list.gate, out, row_bytes, batch, k, classes, class_counts_in_parts(classes.m),
                                 as_stream(stream));
    }
    return eval_rows(src, list.a + tail, list.b + tail, list.gate + tail, rows_out, n[layers - 1], n[layers], row_bytes, as_stream(stream));
}
