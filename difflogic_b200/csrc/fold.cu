// Packed networks with fixed gates, simplified before they are evaluated.
//
// Once every neuron has its arg-max gate the network is a logic circuit, and much of what the layers spell out needs no work:
// a neuron whose gate ignores an input, or has a constant for one, or one row for both, hands on a row that exists already (or
// its inverse), or a constant; and a row that nothing reads any further need not be computed.  Two sweeps find out:
//
//   forward   every neuron's output becomes a reference: a constant, an earlier value or its inverse, or a value of its own.
//             Inversions travel with the references, so a value is the AND of two values or their inverses, or an XOR.
//   backward  from what the last layer hands on: which values are read, by which layer last.  Gates that are left get
//             consecutive places in a list, layer by layer from the last one to the first.
//
// Same counts, same rows, for every input.  Of 64000 x 12 neurons with gates drawn evenly from the sixteen 18 % are left as
// gates (784 -> 4 x 8000: 40 %); of a network whose neurons all need both inputs and are all read, everything is.
//
// Bound by latency: a sweep is a chain of one launch per layer, about 2 us each, with random reads of 4 bytes out of L2.
#include "fold.cuh"
#include "gates.cuh"

namespace dl {

// Truth table (bit 3: f(0,0), 2: f(0,1), 1: f(1,0), 0: f(1,1)) of a gate in terms of the values behind its inputs' references.
// A constant input leaves a gate that ignores it; so does reading one value twice.
__device__ __forceinline__ int gate_of_values(int op, int ra, int rb) {
    if (ref_is_constant(ra)) op = (ra & 1) ? (op & 3) * 5 : (op >> 2) * 5;
    else if (ra & 1) op = op >> 2 | (op & 3) << 2;
    if (ref_is_constant(rb)) {
        const int kept = ((rb & 1) ? op : op >> 1) & 5;
        op = kept | kept << 1;
    } else if (rb & 1) {
        op = ((op >> 1) & 5) | ((op & 5) << 1);
    }
    if (!ref_is_constant(ra) && ra >> 1 == rb >> 1) op = (op & 8 ? 12 : 0) | (op & 1 ? 3 : 0);
    return op;
}

// One layer of the forward sweep.  ref_in: references of its inputs, null where they are the network's.
__global__ void __launch_bounds__(kThreads)
fold_layer_kernel(const int64_t *__restrict__ a, const int64_t *__restrict__ b, const uint8_t *__restrict__ gate, int n_in, int n_out,
                  const int32_t *__restrict__ ref_in, int first, int32_t *__restrict__ ref, int32_t *__restrict__ in_a,
                  int32_t *__restrict__ in_b) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= n_out) return;
    auto input = [&](int64_t i) {
        const int v = i < 0 || i >= n_in ? 0 : (int)i;
        return ref_in != nullptr ? __ldcg(ref_in + v) : v << 1;
    };
    const int ra = input(__ldg(a + j)), rb = input(__ldg(b + j));
    int op = gate_of_values(__ldg(gate + j) & 15, ra, rb);
    const bool needs_a = gate_needs_input(op, 0), needs_b = gate_needs_input(op, 1);
    int out, va = 0, vb = 0;
    if (needs_a && needs_b) {
        const int inverted = __popc(op) == 3 || op == 9;
        if (inverted) op ^= 15;
        out = (first + j) << 1 | inverted;
        va = ra >> 1;
        vb = rb >> 1 | op << kFoldValueBits;
    } else if (needs_a) {
        out = (ra & ~1) | (op >> 3);
    } else if (needs_b) {
        out = (rb & ~1) | (op >> 3);
    } else {
        out = kRefFalse | (op & 1);
    }
    ref[j] = out;
    in_a[j] = va;
    in_b[j] = vb;
}

// The layer that hands its rows on: whatever is not constant is read there.
__global__ void __launch_bounds__(kThreads)
fold_read_kernel(const int32_t *__restrict__ ref, int n, int layer, int32_t *__restrict__ use) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= n) return;
    const int r = __ldcg(ref + j);
    if (!ref_is_constant(r)) use[r >> 1] = layer;
}

// One layer of the backward sweep: gates that are read take their places and read their inputs.  An input is met first by the
// last layer that reads it.  unlisted: the layer's gates take no places; all of them read.
__global__ void __launch_bounds__(kThreads)
fold_mark_kernel(int layer, int layers, int first, int n, bool unlisted, const int32_t *__restrict__ ref, const int32_t *__restrict__ in_a,
                 const int32_t *__restrict__ in_b, int32_t *use, int32_t *__restrict__ row, int32_t *header) {
    __shared__ int s_warp[kThreads / 32], s_base;
    grid_dependency_wait();
    grid_dependents_launch();
    const int tid = threadIdx.x, j = blockIdx.x * kThreads + tid;
    const int vb = j < n ? __ldcg(in_b + j) : 0;
    const bool gate = vb >> kFoldValueBits != 0;
    const bool left = gate && (unlisted || __ldcg(use + first + j) != 0);
    auto read = [&](int v) { return __ldcg(use + v) == 0 && atomicCAS(use + v, 0, layer) == 0 ? 1 : 0; };
    int last = 0;  // values that this layer is the last to read
    if (left) {
        last = read(__ldcg(in_a + j));
        last += read(vb & ((1 << kFoldValueBits) - 1));
    } else if (unlisted && j < n) {
        const int r = __ldcg(ref + j);
        if (!ref_is_constant(r)) read(r >> 1);
    }
    if (unlisted) return;
    last = __reduce_add_sync(0xffffffffu, last);
    if (tid % 32 == 0 && last != 0) atomicAdd(header + kFoldDead + layer, last);
    const unsigned mask = __ballot_sync(0xffffffffu, left);
    if (tid % 32 == 0) s_warp[tid / 32] = __popc(mask);
    __syncthreads();
    if (tid == 0) {
        int total = 0, before = 0;
        for (int w = 0; w < kThreads / 32; ++w) {
            const int c = s_warp[w];
            s_warp[w] = total;
            total += c;
        }
        for (int l = layer + 1; l <= layers; ++l) before += __ldcg(header + l);
        s_base = before + (total ? atomicAdd(header + layer, total) : 0);
    }
    __syncthreads();
    if (left) row[first + j] = s_base + s_warp[tid / 32] + __popc(mask & ((1u << (tid % 32)) - 1u));
}

bool fold_shape(const int64_t *n, int layers, FoldShape *sh) {
    if (n == nullptr || layers < 1 || layers > kFoldLayers) return false;
    sh->layers = layers;
    int64_t first = 0;
    for (int l = 0; l <= layers; ++l) {
        if (n[l] < 1 || n[l] >= ((int64_t)1 << kFoldValueBits)) return false;
        sh->n[l] = (int)n[l];
        sh->first[l] = (int)first;
        first += n[l];
        if (first >= ((int64_t)1 << kFoldValueBits)) return false;
    }
    sh->first[layers + 1] = (int)first;
    return true;
}

int fold_network(const FoldShape &sh, const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const FoldScratch &s,
                 bool tail_rows, cudaStream_t st) {
    const int L = sh.layers;
    if (cudaMemsetAsync(s.header, 0, (kFoldHeader + (size_t)sh.first[L + 1]) * sizeof(int32_t), st) != cudaSuccess)
        return launch_status("fold_network (clear)");
    auto at = [&](int32_t *p, int l) { return p + (sh.first[l] - sh.n[0]); };
    auto grid = [](int n) { return dim3((unsigned)ceil_div(n, kThreads)); };
    for (int l = 1; l <= L; ++l)
        launch_dependent(l > 1, fold_layer_kernel, grid(sh.n[l]), dim3(kThreads), 0, st, a[l - 1], b[l - 1], gate[l - 1], sh.n[l - 1], sh.n[l],
                         l == 1 ? nullptr : at(s.ref, l - 1), sh.first[l], at(s.ref, l), at(s.in_a, l), at(s.in_b, l));
    if (!tail_rows)
        launch_dependent(true, fold_read_kernel, grid(sh.n[L]), dim3(kThreads), 0, st, at(s.ref, L), sh.n[L], L + 1, s.use);
    for (int l = L; l >= 1; --l)
        launch_dependent(true, fold_mark_kernel, grid(sh.n[l]), dim3(kThreads), 0, st, l, L, sh.first[l], sh.n[l], tail_rows && l == L,
                         at(s.ref, l), at(s.in_a, l), at(s.in_b, l), s.use, s.row, s.header);
    return launch_status("fold_network");
}

}  // namespace dl
