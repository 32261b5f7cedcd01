// Packed networks too wide for shared memory, layer by layer over the gates that folding leaves (fold.cu).
//
// Every gate that is left has a row in one POOL, layers one after the other; a gate reads rows of the pool or of the packed
// input, from whichever layer its inputs come, so rows that a layer only hands on are neither moved nor stored.  The kernels are
// those for whole layers (eval_rows), over shorter lists; the last layer keeps all of its neurons, in order, because its rows or
// class counts are wanted, with the gates in terms of pool rows: constants read nothing and copies one row.
//
// Bound by memory as before, with fewer rows: 256 -> 12 x 64000, 2^17 samples 4340 -> 1190 us (12 x 64000 neurons of which 139000 are
// left as gates); 9216 -> 4 x 128000, 10000 samples, with the packing 289 -> 195 us.
#include "fold.cuh"
#include "gates.cuh"

namespace dl {

int eval_rows(const SplitRows &x, const int64_t *a, const int64_t *b, const uint8_t *gate, void *y, int64_t n_in, int64_t n_out,
              int64_t row_bytes, cudaStream_t st);                                                   // packed.cu
int eval_class_counts(const SplitRows &x, const int64_t *a, const int64_t *b, const uint8_t *gate, int32_t *out, int64_t row_bytes,
                      int64_t batch, int64_t k, int64_t m, bool in_parts, cudaStream_t st);          // eval_groupbitsum.cu

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

static GateList gate_list(const FoldShape &sh, void *work) {
    const int64_t neurons = sh.first[sh.layers + 1] - sh.n[0];
    GateList l;
    l.a = reinterpret_cast<int64_t *>(reinterpret_cast<int32_t *>(work) + (fold_words(sh) + 3) / 4 * 4);
    l.b = l.a + neurons;
    l.gate = reinterpret_cast<uint8_t *>(l.b + neurons);
    return l;
}

}  // namespace dl

using namespace dl;

extern "C" DL_API int64_t dl_fold_layers_bytes(const int64_t *n, int layers) {
    FoldShape sh;
    if (!fold_shape(n, layers, &sh)) return 0;
    return (fold_words(sh) + 3) / 4 * 16 + 17 * ((int64_t)sh.first[layers + 1] - sh.n[0]);
}

extern "C" DL_API int dl_fold_layers(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n, int layers,
                                     void *work, void *stream) {
    FoldShape sh;
    DL_REQUIRE(a && b && gate && n && work && aligned_to(work, 16), DL_ERR_INVALID_ARG, "dl_fold_layers: null pointer or unaligned scratch");
    DL_REQUIRE(fold_shape(n, layers, &sh), DL_ERR_TOO_LARGE, "dl_fold_layers: 1 .. %d layers of fewer than 2^27 rows in all", kFoldLayers);
    for (int l = 0; l < layers; ++l) DL_REQUIRE(a[l] && b[l] && gate[l], DL_ERR_INVALID_ARG, "dl_fold_layers: null pointer");
    const FoldScratch s = fold_scratch(sh, reinterpret_cast<int32_t *>(work));
    if (int e = fold_network(sh, a, b, gate, s, true, as_stream(stream))) return e;
    const int tail = sh.n[layers], hidden = sh.first[layers + 1] - sh.n[0] - tail;
    fold_emit_kernel<<<(unsigned)ceil_div(hidden + tail, kThreads), kThreads, 0, as_stream(stream)>>>(sh.n[0], hidden, tail, s.ref, s.in_a, s.in_b,
                                                                                                      s.use, s.row, gate_list(sh, work));
    return launch_status("dl_fold_layers");
}

extern "C" DL_API int dl_eval_folded(const void *x, const void *work, const int64_t *n, const int32_t *left, int layers, void *pool,
                                     int32_t *out, void *rows_out, int64_t row_bytes, int64_t batch, int64_t k, void *stream) {
    const char *who = "dl_eval_folded";
    FoldShape sh;
    DL_REQUIRE(x && work && n && left && (out != nullptr) != (rows_out != nullptr) && aligned_to(work, 16), DL_ERR_INVALID_ARG, "%s: null pointer", who);
    DL_REQUIRE(fold_shape(n, layers, &sh) && row_bytes > 0 && batch > 0 && batch <= row_bytes * 8 && k > 0 && n[layers] % k == 0,
               DL_ERR_INVALID_ARG, "%s: bad sizes", who);
    int64_t rows = 0;
    for (int l = 1; l < layers; ++l) {
        DL_REQUIRE(left[l] >= 0 && left[l] <= n[l], DL_ERR_INVALID_ARG, "%s: layer %d has more gates left than neurons", who, l);
        rows += left[l];
    }
    DL_REQUIRE(pool != nullptr || rows == 0, DL_ERR_INVALID_ARG, "%s: null pointer", who);
    const int64_t m = n[layers] / k;
    const bool whole = dl_eval_groupbitsum_applicable(x, n[0], n[layers], row_bytes, 8, k) == 1;
    DL_REQUIRE(out == nullptr || (aligned_to(pool, 16) && (whole || dl_eval_groupbitsum_parts_applicable(x, n[0], n[layers], row_bytes, 8, k) == 1)),
               DL_ERR_INVALID_ARG, "%s: counts outside the range of dl_eval_groupbitsum and dl_eval_groupbitsum_parts", who);
    const GateList list = gate_list(sh, const_cast<void *>(work));
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
    if (out != nullptr)
        return eval_class_counts(src, list.a + tail, list.b + tail, list.gate + tail, out, row_bytes, batch, k, m, !whole, as_stream(stream));
    return eval_rows(src, list.a + tail, list.b + tail, list.gate + tail, rows_out, n[layers - 1], n[layers], row_bytes, as_stream(stream));
}
