// Packed inference of a WHOLE network in one kernel: a CTA takes a narrow block of samples (V = 16, 8 or 4 bytes of every
// row) through all layers with the activations in shared memory, and counts the classes at the end.
//
// Why: layer by layer every activation row is written to memory and gathered again, 8000 gates x 2^20 samples: 1 GB out and
// 1 GB in per layer.  Here only the input bits are read and the counts written; a layer costs two shared-memory row loads and
// one row store per gate.  What bounds it is shared-memory bandwidth, so bank conflicts decide: the rows of a layer are
// gathered at random, and a phase of NC = 128 / V lanes (8 lanes of 16 bytes ...) that hits random banks takes about 2.6
// cycles instead of one.  The PROGRAM of a network (resident_program_kernel, once per set of weights) therefore puts its
// neurons in an order in which the lanes of a phase read distinct bank classes, for both inputs, and gives every neuron the
// row slot of its position, so that stores are free of conflicts as well.
//
// In-place update: a thread keeps the outputs of its R neurons in registers until every thread has read its inputs, then
// all store.  That halves the shared memory a layer needs and with it doubles the samples per block.
//
// Program word of a neuron, 32 bits: slot of the first input (14) | slot of the second (14) | masks m0, ma, mb, mab (4), so
// layers and inputs are limited to 16384 rows.  It is read from L2 by every CTA: 4 bytes per gate against 3 V bytes of shared
// memory traffic.
#include "common.cuh"
#include "gates.cuh"

namespace dl {

constexpr int kResLayers = 32;        // layers per network
constexpr int kResRows = 1 << 14;     // rows per layer or input
constexpr int kResPlanes = 10;        // a counting task has at most ceil(16384 / 32) = 512 rows

struct ResidentSizes {
    int layers;
    int n[kResLayers + 1];  // rows of the input and of every layer
};

// ---------------------------------------------------------------------------------------------
// program: one launch per layer, one CTA
// ---------------------------------------------------------------------------------------------
// A neuron reads bank classes ca and cb = ca + d (mod nc).  Neurons of the same d are dealt out in rounds over ca = 0 .. nc-1:
// nc consecutive ones then read nc distinct classes with either input.  A neuron may be taken with its inputs swapped
// (class cb, difference -d); it joins the emptier of its two buckets, which keeps the rounds full.
__global__ void __launch_bounds__(1024)
resident_program_kernel(const int64_t *__restrict__ a, const int64_t *__restrict__ b, const uint8_t *__restrict__ gate, int n_in,
                        int n_out, int nc, const uint32_t *__restrict__ slot_in, uint32_t *__restrict__ prog,
                        uint32_t *__restrict__ slot_out, uint32_t *__restrict__ order, uint32_t *__restrict__ key) {
    __shared__ int cnt[256], base[16];
    volatile int *vcnt = cnt;
    for (int t = threadIdx.x; t < 256; t += blockDim.x) cnt[t] = 0;
    __syncthreads();
    auto slot = [&](int64_t i) {
        const int v = i < 0 || i >= n_in ? 0 : (int)i;
        return slot_in != nullptr ? slot_in[v] : (uint32_t)v;
    };
    for (int j = threadIdx.x; j < n_out; j += blockDim.x) {
        const int ca = (int)(slot(a[j]) & (nc - 1)), cb = (int)(slot(b[j]) & (nc - 1)), d = (cb - ca) & (nc - 1);
        const int one = d * nc + ca, two = ((nc - d) & (nc - 1)) * nc + cb;
        const int flip = vcnt[two] < vcnt[one];
        const int bucket = flip ? two : one;
        key[j] = (uint32_t)atomicAdd(&cnt[bucket], 1) << 9 | (uint32_t)bucket << 1 | (uint32_t)flip;
    }
    __syncthreads();
    if ((int)threadIdx.x < nc) {
        int s = 0;
        for (int t = 0; t < (int)threadIdx.x * nc; ++t) s += cnt[t];
        base[threadIdx.x] = s;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < n_out; j += blockDim.x) {
        const uint32_t e = key[j];
        const int rank = (int)(e >> 9), bucket = (int)(e >> 1) & 255, flip = (int)(e & 1), d = bucket / nc, c = bucket % nc;
        int pos = base[d];  // neurons of this d in earlier rounds, and earlier in this round
        for (int i = 0; i < nc; ++i) {
            const int have = cnt[d * nc + i];
            pos += min(have, rank) + (i < c && have > rank ? 1 : 0);
        }
        const GateMasks g = gate_masks((int)gate[j]);
        const uint32_t first = slot(flip ? b[j] : a[j]), second = slot(flip ? a[j] : b[j]);
        const uint32_t ma = (flip ? g.mb : g.ma) & 1u, mb = (flip ? g.ma : g.mb) & 1u;
        prog[pos] = first | second << 14 | (g.m0 & 1u) << 28 | ma << 29 | mb << 30 | (g.mab & 1u) << 31;
        if (slot_out != nullptr) slot_out[j] = (uint32_t)pos;
        if (order != nullptr) order[pos] = (uint32_t)j;
    }
}

// ---------------------------------------------------------------------------------------------
// evaluation
// ---------------------------------------------------------------------------------------------
template <int WORDS> struct ResRow;
template <> struct ResRow<1> { using type = uint32_t; };
template <> struct ResRow<2> { using type = uint2; };
template <> struct ResRow<4> { using type = uint4; };

struct ResMasks {
    uint32_t m0, ma, mb, mab;
};
__device__ __forceinline__ uint32_t res_gate(uint32_t a, uint32_t b, const ResMasks &m) {
    const uint32_t u = m.ma ^ (m.mab & b);
    return ((a & u) ^ m.m0) ^ (m.mb & b);
}
__device__ __forceinline__ uint32_t res_apply(uint32_t a, uint32_t b, const ResMasks &m) { return res_gate(a, b, m); }
__device__ __forceinline__ uint2 res_apply(const uint2 &a, const uint2 &b, const ResMasks &m) {
    return make_uint2(res_gate(a.x, b.x, m), res_gate(a.y, b.y, m));
}
__device__ __forceinline__ uint4 res_apply(const uint4 &a, const uint4 &b, const ResMasks &m) {
    return make_uint4(res_gate(a.x, b.x, m), res_gate(a.y, b.y, m), res_gate(a.z, b.z, m), res_gate(a.w, b.w, m));
}

#define DL_CSA32(h, l, a, b, c)        \
    {                                  \
        const uint32_t u_ = (a) ^ (b); \
        const uint32_t c_ = (c);       \
        h = ((a) & (b)) | (u_ & c_);   \
        l = u_ ^ c_;                   \
    }

// adds one word of weight 2^from to a bit-sliced counter
__device__ __forceinline__ void planes_add(uint32_t (&p)[kResPlanes], uint32_t carry, int from) {
#pragma unroll
    for (int i = 0; i < kResPlanes; ++i) {
        if (i >= from) {
            const uint32_t t = p[i] & carry;
            p[i] ^= carry;
            carry = t;
        }
    }
}

// WORDS: 32-bit words per row of a block (V = 4 * WORDS bytes); T threads; R neurons per thread and layer at most.
template <int WORDS, int T, int R>
__global__ void __launch_bounds__(T, 1024 / T)
resident_kernel(const uint8_t *__restrict__ x, int64_t row_bytes, const uint32_t *__restrict__ prog, ResidentSizes sz,
                int32_t *__restrict__ out, uint8_t *__restrict__ rows_out, int64_t batch, int k, int rows_per_class, int row_slots) {
    using Row = typename ResRow<WORDS>::type;
    constexpr int V = 4 * WORDS;
    extern __shared__ __align__(16) uint8_t res_smem[];
    Row *rows = reinterpret_cast<Row *>(res_smem);
    int *counts = reinterpret_cast<int *>(res_smem + (size_t)row_slots * V);  // [8 V samples][k]
    const int tid = threadIdx.x;

    const uint8_t *src = x + (int64_t)blockIdx.x * V;
    for (int i = tid; i < sz.n[0]; i += T) rows[i] = __ldg(reinterpret_cast<const Row *>(src + (int64_t)i * row_bytes));
    for (int t = tid; t < 8 * V * k; t += T) counts[t] = 0;

    uint32_t w[R];
    int n = sz.n[1];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = tid + r * T < n ? __ldg(prog + tid + r * T) : 0u;
    __syncthreads();
    for (int l = 1; l <= sz.layers; ++l) {
        const uint32_t *next = prog + n;  // program of the next layer; after the last one, the rows' order
        const int n_next = l < sz.layers ? sz.n[l + 1] : n;
        Row y[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (tid + r * T < n) {
                const Row va = *reinterpret_cast<const Row *>(res_smem + (w[r] & 0x3fffu) * V);
                const Row vb = *reinterpret_cast<const Row *>(res_smem + ((w[r] >> 14) & 0x3fffu) * V);
                const ResMasks m = {(uint32_t)((int)(w[r] << 3) >> 31), (uint32_t)((int)(w[r] << 2) >> 31),
                                    (uint32_t)((int)(w[r] << 1) >> 31), (uint32_t)((int)w[r] >> 31)};
                y[r] = res_apply(va, vb, m);
            }
        }
        // the next layer's program words are on their way while this layer's rows are exchanged
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = tid + r * T < n_next ? __ldg(next + tid + r * T) : 0u;
        if (l == sz.layers && rows_out != nullptr) {  // the rows themselves are wanted
            uint8_t *dst = rows_out + (int64_t)blockIdx.x * V;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (tid + r * T < n) *reinterpret_cast<Row *>(dst + (int64_t)w[r] * row_bytes) = y[r];
            return;
        }
        __syncthreads();
        if (l < sz.layers) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (tid + r * T < n) rows[tid + r * T] = y[r];
        } else {
            // the last layer's rows go where their classes are
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (tid + r * T < n) rows[w[r]] = y[r];
        }
        __syncthreads();
        prog = next;
        n = n_next;
    }

    // ---- class counts: a warp takes a run of rows of one class; lane = (row, word), 128 bytes of rows per load ----
    constexpr int kSubs = 32 / WORDS;
    const int warp = tid / 32, lane = tid % 32, word = lane % WORDS, sub = lane / WORDS;
    const int parts = (32 + k - 1) / k, tasks = k * parts;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(res_smem) + word;
    for (int task = warp; task < tasks; task += T / 32) {
        const int c = task / parts, q = task % parts;
        const int beg = c * rows_per_class + rows_per_class * q / parts, end = c * rows_per_class + rows_per_class * (q + 1) / parts;
        uint32_t p[kResPlanes];
#pragma unroll
        for (int i = 0; i < kResPlanes; ++i) p[i] = 0u;
        for (int r = beg + sub; r < end; r += 8 * kSubs) {
            uint32_t v[8], t2a, t2b, t4a, t4b, e8;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = r + i * kSubs < end ? words[(r + i * kSubs) * WORDS] : 0u;
            DL_CSA32(t2a, p[0], p[0], v[0], v[1]);
            DL_CSA32(t2b, p[0], p[0], v[2], v[3]);
            DL_CSA32(t4a, p[1], p[1], t2a, t2b);
            DL_CSA32(t2a, p[0], p[0], v[4], v[5]);
            DL_CSA32(t2b, p[0], p[0], v[6], v[7]);
            DL_CSA32(t4b, p[1], p[1], t2a, t2b);
            DL_CSA32(e8, p[2], p[2], t4a, t4b);
            planes_add(p, e8, 3);
        }
#pragma unroll
        for (int off = WORDS; off < 32; off <<= 1) {  // bit-sliced sums over the lanes of a word
            uint32_t carry = 0u;
#pragma unroll
            for (int i = 0; i < kResPlanes; ++i) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, p[i], off);
                uint32_t h, s;
                DL_CSA32(h, s, p[i], o, carry);
                p[i] = s;
                carry = h;
            }
        }
#pragma unroll
        for (int i = 0; i < WORDS; ++i) {  // every lane of a word has its sums; it takes 32 / kSubs of the samples
            const int s = sub * WORDS + i;
            int count = 0;
#pragma unroll
            for (int pl = 0; pl < kResPlanes; ++pl) count |= (int)((p[pl] >> s) & 1u) << pl;
            int *dst = counts + (word * 32 + s) * k + c;
            if (parts == 1) *dst = count;
            else if (count) atomicAdd(dst, count);
        }
    }
    __syncthreads();
    const int64_t s0 = (int64_t)blockIdx.x * (8 * V);
    const int live = (int)min((int64_t)(8 * V), batch - s0) * k;
    for (int t = tid; t < live; t += T) out[s0 * k + t] = counts[t];
}

static int res_sms() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    return n;
}
static size_t res_shared_bytes(int row_slots, int V, int64_t k) { return (size_t)row_slots * V + (size_t)8 * V * k * sizeof(int); }

constexpr size_t kResMaxShared = 227 * 1024;

struct ResPlan {
    int V, T;
};

// V: the width for which the busiest SM has least to do.  A block of V bytes costs V bytes of row traffic per gate plus what
// does not depend on V (program words, instructions; about 4 bytes' worth).
static ResPlan res_plan(const int64_t *n, int layers, int64_t batch, int64_t k) {
    ResPlan best = {0, 0};
    if (layers < 1 || layers > kResLayers || batch < 1 || k < 1) return best;
    int64_t most = 0;
    for (int l = 0; l <= layers; ++l) {
        if (n[l] < 1 || n[l] > kResRows) return best;
        most = n[l] > most ? n[l] : most;
    }
    if (n[layers] % k != 0) return best;
    int64_t widest = 0;
    for (int l = 1; l <= layers; ++l) widest = n[l] > widest ? n[l] : widest;
    const int sms = res_sms();
    int64_t least = 0;
    for (const int V : {16, 8, 4}) {
        const int R = V == 16 ? 10 : 16;
        if (widest > (int64_t)R * 1024 || k > (1 << 14) || res_shared_bytes((int)most, V, k) > kResMaxShared) continue;
        const int64_t blocks = ceil_div(batch, 8 * V);
        if (blocks >= ((int64_t)1 << 31)) continue;
        const int64_t cost = ceil_div(blocks, sms) * (V + 4);
        if (best.V == 0 || cost < least) {
            least = cost;
            // as many threads as there are rows for when an SM has one block at a time anyway, else several smaller CTAs
            int T = 1024;
            if (blocks > sms) while (T > 256 && widest <= (int64_t)R * (T / 2)) T /= 2;
            best = {V, T};
        }
    }
    return best;
}

template <int WORDS, int T, int R>
static int launch_resident(const void *x, int64_t row_bytes, const uint32_t *prog, const ResidentSizes &sz, int32_t *out, uint8_t *rows_out,
                           int64_t batch, int64_t k, int row_slots, cudaStream_t st) {
    constexpr int V = 4 * WORDS;
    const size_t smem = res_shared_bytes(row_slots, V, k);
    if (cudaFuncSetAttribute(resident_kernel<WORDS, T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return launch_status("dl_eval_network (shared memory opt-in)");
    resident_kernel<WORDS, T, R><<<(unsigned)ceil_div(batch, 8 * V), T, smem, st>>>(
        reinterpret_cast<const uint8_t *>(x), row_bytes, prog, sz, out, rows_out, batch, (int)k, (int)(sz.n[sz.layers] / k), row_slots);
    return launch_status("dl_eval_network");
}

// lanes that share a phase of a shared-memory access: the widest rows that the layer sizes allow
static int res_classes(const int64_t *n, int layers) {
    int64_t most = 0;
    for (int l = 0; l <= layers; ++l) most = n[l] > most ? n[l] : most;
    return most > 10 * 1024 ? 16 : 8;
}

}  // namespace dl

using namespace dl;

extern "C" DL_API int dl_eval_network_applicable(const void *x, const int64_t *n, int layers, int64_t row_bytes, int64_t batch, int64_t k) {
    if (x == nullptr || n == nullptr || row_bytes < 16 || row_bytes % 16 != 0 || !aligned_to(x, 16) || batch > row_bytes * 8) return 0;
    return res_plan(n, layers, batch, k).V;
}

// 32-bit words of the program of a network (the layers' words, the last layer's order, and scratch for building it).
extern "C" DL_API int64_t dl_network_program_words(const int64_t *n, int layers) {
    if (n == nullptr || layers < 1 || layers > kResLayers) return 0;
    int64_t words = n[layers], widest = 0;
    for (int l = 1; l <= layers; ++l) {
        words += n[l];
        widest = n[l] > widest ? n[l] : widest;
    }
    return words + 3 * widest;
}

extern "C" DL_API int dl_network_program(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n,
                                         int layers, uint32_t *program, void *stream) {
    DL_REQUIRE(a && b && gate && n && program, DL_ERR_INVALID_ARG, "dl_network_program: null pointer");
    DL_REQUIRE(layers >= 1 && layers <= kResLayers, DL_ERR_INVALID_ARG, "dl_network_program: 1 .. %d layers", kResLayers);
    int64_t total = n[layers], widest = 0;
    for (int l = 0; l <= layers; ++l) {
        DL_REQUIRE(n[l] >= 1 && n[l] <= kResRows, DL_ERR_TOO_LARGE, "dl_network_program: layers of 1 .. %d rows", kResRows);
        if (l > 0) {
            DL_REQUIRE(a[l - 1] && b[l - 1] && gate[l - 1], DL_ERR_INVALID_ARG, "dl_network_program: null pointer");
            total += n[l];
            widest = n[l] > widest ? n[l] : widest;
        }
    }
    uint32_t *at = program, *order = program + (total - n[layers]), *scratch = program + total;
    const int nc = res_classes(n, layers);
    for (int l = 1; l <= layers; ++l) {
        const uint32_t *slot_in = l == 1 ? nullptr : scratch + (int64_t)(l % 2) * widest;
        uint32_t *slot_out = l == layers ? nullptr : scratch + (int64_t)((l + 1) % 2) * widest;
        resident_program_kernel<<<1, 1024, 0, as_stream(stream)>>>(a[l - 1], b[l - 1], gate[l - 1], (int)n[l - 1], (int)n[l], nc, slot_in, at,
                                                                   slot_out, l == layers ? order : nullptr, scratch + 2 * widest);
        at += n[l];
    }
    return launch_status("dl_network_program");
}

extern "C" DL_API int dl_eval_network(const void *x, const uint32_t *program, const int64_t *n, int layers, int32_t *out, void *rows_out,
                                      int64_t row_bytes, int64_t batch, int64_t k, void *stream) {
    DL_REQUIRE(program && (out != nullptr) != (rows_out != nullptr) && aligned_to(rows_out, 16) &&
                   dl_eval_network_applicable(x, n, layers, row_bytes, batch, k) != 0, DL_ERR_INVALID_ARG,
               "dl_eval_network: bad pointer or sizes outside the kernel's range (ask dl_eval_network_applicable first)");
    const ResPlan plan = res_plan(n, layers, batch, k);
    ResidentSizes sz = {};
    sz.layers = layers;
    int row_slots = 0;
    for (int l = 0; l <= layers; ++l) {
        sz.n[l] = (int)n[l];
        row_slots = sz.n[l] > row_slots ? sz.n[l] : row_slots;
    }
    cudaStream_t st = as_stream(stream);
#define DL_RES(WW, TT, RR)          \
    if (plan.V == 4 * WW && plan.T == TT) return launch_resident<WW, TT, RR>(x, row_bytes, program, sz, out, reinterpret_cast<uint8_t *>(rows_out), batch, k, row_slots, st)
    DL_RES(4, 1024, 10);
    DL_RES(4, 512, 10);
    DL_RES(4, 256, 10);
    DL_RES(2, 1024, 16);
    DL_RES(2, 512, 16);
    DL_RES(2, 256, 16);
    DL_RES(1, 1024, 16);
    DL_RES(1, 512, 16);
    DL_RES(1, 256, 16);
#undef DL_RES
    return fail(DL_ERR_INVALID_ARG, "dl_eval_network: no kernel for rows of %d bytes", plan.V);
}
