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
// Measured, whole kernel: 784 -> 4 x 8000, 2^20 samples 827 us (1020 with general gates and a full adder tree per count; 1210 layer
// by layer), of which the busiest unit, the shared-memory pipe, works 65 %; 784 -> 5 x 16000, 10000 samples 43 us (97 layer by layer).
//
// CTAs that stay for several blocks and fetch the next one's input while they count were slower (needs more than 64 registers:
// 16000 wide, 10000 samples 45 -> 51 us, 8000 wide, 2^18 samples 208 -> 212).
//
// In-place update: a thread keeps the outputs of its R neurons in registers until every thread has read its inputs, then
// all store.  That halves the shared memory a layer needs and with it doubles the samples per block.
//
// Instructions come next: a general gate is three operations per word and four masks.  With inversions pushed through to the
// readers every gate is one of four KINDS, and the neurons of a layer are sorted by kind:
//   AND    (a ^ i) & (b ^ j)   the eight gates with one or three ones in their truth table; two operations, two masks
//   XOR    a ^ b               and its inverse
//   COPY   a                   and b, and their inverses; one row load instead of two
//   CONST  0                   and 1; none
// Three ones, XNOR, NOT and 1 are the inverses of what is stored; whoever reads the row folds that into its own i, j or
// inversion, and the last layer inverts what it hands on.
//
// Program word of a neuron, 32 bits: second slot (bits 0 .. 13), j (15), first slot (16 .. 29), i (31), so layers and inputs are
// limited to 16384 rows.  It is read from L2 by every CTA: 4 bytes per gate against up to 3 V bytes of shared-memory traffic.
#include "common.cuh"
#include "gates.cuh"

namespace dl {

constexpr int kResLayers = 32;        // layers per network
constexpr int kResRows = 1 << 14;     // rows per layer or input
constexpr int kResPlanes = 11;        // planes of a counting task: at most 2047 rows
constexpr int kResPad = 1 << 14;      // words behind a program that a CTA may read and not use

struct ResidentSizes {
    int layers;
    int n[kResLayers + 1];  // rows of the input and of every layer
};

constexpr int kResHeader = 4;  // words in front of a layer's program: where AND, XOR and COPY end
enum { kResAnd = 0, kResXor = 1, kResCopy = 2, kResConst = 3 };

// A gate in terms of the STORED rows of its inputs, which are the inverses of the inputs where inv_a / inv_b is set.
struct ResGate {
    int kind, i, j, inv;  // inv: what is stored is the inverse of the gate's output
    bool second;          // COPY: the second input's row
};
__device__ __forceinline__ ResGate res_classify(int op, int inv_a, int inv_b) {
    const int t00 = (op >> 3) & 1, t01 = (op >> 2) & 1, t10 = (op >> 1) & 1, t11 = op & 1;
    const int ones = t00 + t01 + t10 + t11;
    ResGate g = {kResConst, 0, 0, ones == 4, false};
    if (ones == 1 || ones == 3) {
        g.kind = kResAnd;
        g.inv = ones == 3;
        // the input pair whose output differs from the other three
        const int at = (t00 ^ g.inv) ? 0 : (t01 ^ g.inv) ? 1 : (t10 ^ g.inv) ? 2 : 3;
        g.i = (at < 2) ^ inv_a;           // AND of the inputs, inverted where they are 0 there
        g.j = (at % 2 == 0) ^ inv_b;
    } else if (ones == 2) {
        if (t00 == t11) {
            g.kind = kResXor;
            g.inv = t00 ^ inv_a ^ inv_b;
        } else {
            g.kind = kResCopy;
            g.second = t00 != t01;
            g.inv = t00 ^ (g.second ? inv_b : inv_a);
        }
    }
    return g;
}

// ---------------------------------------------------------------------------------------------
// program: one launch per layer, one CTA
// ---------------------------------------------------------------------------------------------
// A neuron reads bank classes ca and cb = ca + d (mod NC).  Neurons of the same kind and d are dealt out in rounds over ca =
// 0 .. NC-1: NC consecutive ones then read NC distinct classes with either input.  A neuron with two inputs may be taken with
// them swapped (class cb, difference -d); it joins the emptier of its two buckets, which keeps the rounds full.
// slot_in / slot_out / order: row slot (neuron, for order) << 1 | inverse stored.
// Between the look-up of its inputs and the writing of its word a neuron waits in shared memory, 8 bytes.
template <int NC>
__global__ void __launch_bounds__(1024)
resident_program_kernel(const int64_t *__restrict__ a, const int64_t *__restrict__ b, const uint8_t *__restrict__ gate, int n_in,
                        int n_out, const uint32_t *__restrict__ slot_in, uint32_t *__restrict__ prog, uint32_t *__restrict__ slot_out,
                        uint32_t *__restrict__ order) {
    constexpr int kGroups = 2 * NC + 2;  // AND by d, XOR by d, COPY, CONST
    __shared__ int cnt[kGroups * NC], size[kGroups], base[kGroups];
    extern __shared__ uint2 s_neuron[];  // slots of both inputs, 15 bits each; gate (4) | swapped (1) | bucket (10) | rank (14)
    volatile int *vcnt = cnt;
    const int tid = threadIdx.x;
    for (int t = tid; t < kGroups * NC; t += 1024) cnt[t] = 0;
    auto slot = [&](int64_t i) {
        const int v = i < 0 || i >= n_in ? 0 : (int)i;
        return slot_in != nullptr ? __ldg(slot_in + v) : (uint32_t)v << 1;
    };
#pragma unroll 4
    for (int j = tid; j < n_out; j += 1024)
        s_neuron[j] = make_uint2(slot(__ldg(a + j)) | slot(__ldg(b + j)) << 15, __ldg(gate + j) & 15u);
    __syncthreads();
#pragma unroll 1
    for (int j = tid; j < n_out; j += 1024) {
        const uint2 e = s_neuron[j];
        const uint32_t sa = e.x & 0x7fffu, sb = e.x >> 15;
        const ResGate g = res_classify((int)e.y, sa & 1, sb & 1);
        const int ca = (int)(sa >> 1) & (NC - 1), cb = (int)(sb >> 1) & (NC - 1), d = (cb - ca) & (NC - 1);
        int bucket, flip = 0;
        if (g.kind == kResConst) {
            bucket = (2 * NC + 1) * NC;
        } else if (g.kind == kResCopy) {
            flip = g.second;
            bucket = 2 * NC * NC + (flip ? cb : ca);
        } else {
            const int from = g.kind == kResXor ? NC * NC : 0;
            const int one = from + d * NC + ca, two = from + ((NC - d) & (NC - 1)) * NC + cb;
            flip = vcnt[two] < vcnt[one];
            bucket = flip ? two : one;
        }
        s_neuron[j].y = e.y | (uint32_t)flip << 4 | (uint32_t)bucket << 5 | (uint32_t)atomicAdd(&cnt[bucket], 1) << 15;
    }
    __syncthreads();
    if (tid < kGroups) {
        int s = 0;
#pragma unroll
        for (int i = 0; i < NC; ++i) s += cnt[tid * NC + i];
        size[tid] = s;
    }
    __syncthreads();
    if (tid < kGroups) {
        int s = 0;
        for (int t = 0; t < tid; ++t) s += size[t];
        base[tid] = s;
        if (tid == NC) prog[0] = (uint32_t)s;
        if (tid == 2 * NC) prog[1] = (uint32_t)s;
        if (tid == 2 * NC + 1) prog[2] = (uint32_t)s;
    }
    __syncthreads();
#pragma unroll 1
    for (int j = tid; j < n_out; j += 1024) {
        const uint2 e = s_neuron[j];
        const uint32_t sa = e.x & 0x7fffu, sb = e.x >> 15;
        const int flip = (int)(e.y >> 4) & 1, bucket = (int)(e.y >> 5) & 1023, rank = (int)(e.y >> 15);
        const int group = bucket / NC, c = bucket % NC;
        int pos = base[group];  // neurons of this group in earlier rounds, and earlier in this round
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int have = cnt[group * NC + i];
            pos += min(have, rank) + (i < c && have > rank ? 1 : 0);
        }
        const ResGate g = res_classify((int)(e.y & 15u), sa & 1, sb & 1);
        const uint32_t first = (flip ? sb : sa) >> 1, second = (flip ? sa : sb) >> 1;
        prog[kResHeader + pos] = second | (uint32_t)(flip ? g.i : g.j) << 15 | first << 16 | (uint32_t)(flip ? g.j : g.i) << 31;
        if (slot_out != nullptr) slot_out[j] = (uint32_t)pos << 1 | (uint32_t)g.inv;
        if (order != nullptr) order[pos] = (uint32_t)j << 1 | (uint32_t)g.inv;
    }
}

// ---------------------------------------------------------------------------------------------
// evaluation
// ---------------------------------------------------------------------------------------------
template <int WORDS> struct ResRow;
template <> struct ResRow<1> { using type = uint32_t; };
template <> struct ResRow<2> { using type = uint2; };
template <> struct ResRow<4> { using type = uint4; };

__device__ __forceinline__ uint32_t res_and(uint32_t a, uint32_t b, uint32_t i, uint32_t j) { return (a ^ i) & (b ^ j); }
__device__ __forceinline__ uint2 res_and(const uint2 &a, const uint2 &b, uint32_t i, uint32_t j) {
    return make_uint2(res_and(a.x, b.x, i, j), res_and(a.y, b.y, i, j));
}
__device__ __forceinline__ uint4 res_and(const uint4 &a, const uint4 &b, uint32_t i, uint32_t j) {
    return make_uint4(res_and(a.x, b.x, i, j), res_and(a.y, b.y, i, j), res_and(a.z, b.z, i, j), res_and(a.w, b.w, i, j));
}
__device__ __forceinline__ uint32_t res_xor(uint32_t a, uint32_t b) { return a ^ b; }
__device__ __forceinline__ uint2 res_xor(const uint2 &a, const uint2 &b) { return make_uint2(a.x ^ b.x, a.y ^ b.y); }
__device__ __forceinline__ uint4 res_xor(const uint4 &a, const uint4 &b) { return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w); }
__device__ __forceinline__ void res_fill(uint32_t &v, uint32_t m) { v = m; }
__device__ __forceinline__ void res_fill(uint2 &v, uint32_t m) { v = make_uint2(m, m); }
__device__ __forceinline__ void res_fill(uint4 &v, uint32_t m) { v = make_uint4(m, m, m, m); }
// all ones where bit 15 of w is set
__device__ __forceinline__ uint32_t res_mask15(uint32_t w) {
    uint32_t m;
    asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(m) : "r"(w));
    return m;
}

#define DL_CSA32(h, l, a, b, c)        \
    {                                  \
        const uint32_t u_ = (a) ^ (b); \
        const uint32_t c_ = (c);       \
        h = ((a) & (b)) | (u_ & c_);   \
        l = u_ ^ c_;                   \
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
    int n = sz.n[1], and_end = (int)__ldg(prog), xor_end = (int)__ldg(prog + 1), copy_end = (int)__ldg(prog + 2);
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = r * T < n ? __ldg(prog + kResHeader + tid + r * T) : 0u;
    __syncthreads();
    for (int l = 1; l <= sz.layers; ++l) {
        const uint32_t *next = prog + kResHeader + n;  // program of the next layer; after the last one, the rows' order
        const bool last = l == sz.layers;
        const int n_next = last ? n : sz.n[l + 1];
        Row y[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r * T >= n) break;
            const int p = tid + r * T;
            const Row *first = reinterpret_cast<const Row *>(res_smem + ((w[r] >> 16) & 0x3fffu) * V);
            const Row *second = reinterpret_cast<const Row *>(res_smem + (w[r] & 0x3fffu) * V);
            if (p < and_end) {
                y[r] = res_and(*first, *second, (uint32_t)((int)w[r] >> 31), res_mask15(w[r]));
            } else if (p < xor_end) {
                y[r] = res_xor(*first, *second);
            } else if (p < copy_end) {
                y[r] = *first;
            } else {
                res_fill(y[r], 0u);
            }
        }
        // the next layer's program is on its way while this layer's rows are exchanged
        if (!last) {
            and_end = (int)__ldg(next);
            xor_end = (int)__ldg(next + 1);
            copy_end = (int)__ldg(next + 2);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = r * T < n_next ? __ldg(next + kResHeader + tid + r * T) : 0u;
        if (last) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                Row m;
                res_fill(m, 0u - (w[r] & 1u));
                y[r] = res_xor(y[r], m);
                w[r] >>= 1;
            }
            if (rows_out != nullptr) {  // the rows themselves are wanted
                uint8_t *dst = rows_out + (int64_t)blockIdx.x * V;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (tid + r * T < n) *reinterpret_cast<Row *>(dst + (int64_t)w[r] * row_bytes) = y[r];
                return;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r)  // the last layer's rows go where their classes are
            if (tid + r * T < n) rows[last ? w[r] : (uint32_t)(tid + r * T)] = y[r];
        __syncthreads();
        prog = next;
        n = n_next;
    }

    // ---- class counts: a warp takes a run of rows of one class; lane = (row, word), 128 bytes of rows per load ----
    constexpr int kSubs = 32 / WORDS, kSteps = WORDS == 4 ? 3 : WORDS == 2 ? 4 : 5;
    constexpr int kLane = kResPlanes - kSteps;  // planes of one lane's count
    const int warp = tid / 32, lane = tid % 32, word = lane % WORDS, sub = lane / WORDS;
    const int parts = max(T / 32 / k, (rows_per_class + 511) / 512), tasks = k * parts;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(res_smem) + word;
    for (int task = warp; task < tasks; task += T / 32) {
        const int c = task / parts, q = task % parts;
        const int beg = c * rows_per_class + rows_per_class * q / parts, end = c * rows_per_class + rows_per_class * (q + 1) / parts;
        uint32_t p[kResPlanes];
#pragma unroll
        for (int i = 0; i < kResPlanes; ++i) p[i] = 0u;
        auto add8 = [&](const uint32_t (&v)[8]) {
            uint32_t t2a, t2b, t4a, t4b, carry;
            DL_CSA32(t2a, p[0], p[0], v[0], v[1]);
            DL_CSA32(t2b, p[0], p[0], v[2], v[3]);
            DL_CSA32(t4a, p[1], p[1], t2a, t2b);
            DL_CSA32(t2a, p[0], p[0], v[4], v[5]);
            DL_CSA32(t2b, p[0], p[0], v[6], v[7]);
            DL_CSA32(t4b, p[1], p[1], t2a, t2b);
            DL_CSA32(carry, p[2], p[2], t4a, t4b);
#pragma unroll
            for (int i = 3; i < kLane; ++i) {
                const uint32_t t = p[i] & carry;
                p[i] ^= carry;
                carry = t;
            }
        };
        int r = beg;
        for (; r + 8 * kSubs <= end; r += 8 * kSubs) {
            uint32_t v[8];
            const uint32_t *at = words + (r + sub) * WORDS;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = at[i * 32];
            add8(v);
        }
        if (r < end) {
            uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = r + sub + i * kSubs < end ? words[(r + sub + i * kSubs) * WORDS] : 0u;
            add8(v);
        }
#pragma unroll
        for (int step = 0; step < kSteps; ++step) {  // bit-sliced sums over the lanes of a word, a plane more each time
            uint32_t carry = 0u;
#pragma unroll
            for (int i = 0; i < kLane + step; ++i) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, p[i], WORDS << step);
                uint32_t h, l;
                DL_CSA32(h, l, p[i], o, carry);
                p[i] = l;
                carry = h;
            }
            p[kLane + step] = carry;
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
    int V, T, R;
};

// V: the width for which the busiest SM has least to do.  A block of V bytes costs V bytes of row traffic per gate plus what does
// not depend on V (program words, instructions; about 8 bytes' worth).  Measured, us with V = 16 / 8 / 4, 784 -> 4 layers: 8000 wide,
// 100 samples: 19.5 / 18.3 / 18.0, 4000: 20.0 / 19.1 / 17.7, 10000: 20.0 / 24.0 / 28.7, 2^18: 207 / 255 / 399; 10000 wide, 19000: 38 / 48 / 63;
// 16000 wide, 5 layers, 10000: - / 46 / 54.
static ResPlan res_plan(const int64_t *n, int layers, int64_t batch, int64_t k) {
    ResPlan best = {0, 0, 0};
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
        const int R = V == 16 ? (widest <= 8 * 1024 ? 8 : 10) : 16;
        if (widest > (int64_t)R * 1024 || k > (1 << 14) || res_shared_bytes((int)most, V, k) > kResMaxShared) continue;
        const int64_t blocks = ceil_div(batch, 8 * V);
        if (blocks >= ((int64_t)1 << 31)) continue;
        const int64_t cost = ceil_div(blocks, sms) * (V + 8);
        if (best.V == 0 || cost < least) {
            least = cost;
            // as many threads as there are rows for when an SM has one block at a time anyway, else several smaller CTAs
            int T = 1024;
            if (blocks > sms) while (T > 256 && widest <= (int64_t)R * (T / 2)) T /= 2;
            best = {V, T, R};
        }
    }
    return best;
}

template <int WORDS, int T, int R>
static int launch_resident(const void *x, int64_t row_bytes, const uint32_t *prog, const ResidentSizes &sz, int32_t *out, uint8_t *rows_out,
                           int64_t batch, int64_t k, int row_slots, cudaStream_t st) {
    constexpr int V = 4 * WORDS;
    const size_t smem = res_shared_bytes(row_slots, V, k);
    // the most there may be, not this launch's bytes: the limit is the kernel's, and other threads launch it for other networks
    if (cudaFuncSetAttribute(resident_kernel<WORDS, T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResMaxShared) != cudaSuccess)
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
    int64_t words = n[layers] + kResHeader, widest = 0;
    for (int l = 1; l <= layers; ++l) {
        words += n[l] + kResHeader;
        widest = n[l] > widest ? n[l] : widest;
    }
    return words + 2 * widest + kResPad;
}

extern "C" DL_API int dl_network_program(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n,
                                         int layers, uint32_t *program, void *stream) {
    DL_REQUIRE(a && b && gate && n && program, DL_ERR_INVALID_ARG, "dl_network_program: null pointer");
    DL_REQUIRE(layers >= 1 && layers <= kResLayers, DL_ERR_INVALID_ARG, "dl_network_program: 1 .. %d layers", kResLayers);
    int64_t total = n[layers] + kResHeader, widest = 0;
    for (int l = 0; l <= layers; ++l) {
        DL_REQUIRE(n[l] >= 1 && n[l] <= kResRows, DL_ERR_TOO_LARGE, "dl_network_program: layers of 1 .. %d rows", kResRows);
        if (l > 0) {
            DL_REQUIRE(a[l - 1] && b[l - 1] && gate[l - 1], DL_ERR_INVALID_ARG, "dl_network_program: null pointer");
            total += n[l] + kResHeader;
            widest = n[l] > widest ? n[l] : widest;
        }
    }
    uint32_t *at = program, *order = program + (total - n[layers]), *scratch = program + total;
    auto kernel = res_classes(n, layers) == 8 ? resident_program_kernel<8> : resident_program_kernel<16>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kResRows * sizeof(uint2))) != cudaSuccess)
        return launch_status("dl_network_program (shared memory opt-in)");
    for (int l = 1; l <= layers; ++l) {
        const uint32_t *slot_in = l == 1 ? nullptr : scratch + (int64_t)(l % 2) * widest;
        uint32_t *slot_out = l == layers ? nullptr : scratch + (int64_t)((l + 1) % 2) * widest;
        kernel<<<1, 1024, n[l] * sizeof(uint2), as_stream(stream)>>>(a[l - 1], b[l - 1], gate[l - 1], (int)n[l - 1], (int)n[l], slot_in, at,
                                                                     slot_out, l == layers ? order : nullptr);
        at += n[l] + kResHeader;
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
    if (plan.V == 4 * WW && plan.T == TT && plan.R == RR) return launch_resident<WW, TT, RR>(x, row_bytes, program, sz, out, reinterpret_cast<uint8_t *>(rows_out), batch, k, row_slots, st)
    DL_RES(4, 1024, 8);
    DL_RES(4, 512, 8);
    DL_RES(4, 256, 8);
    DL_RES(4, 1024, 10);
    DL_RES(2, 1024, 16);
    DL_RES(2, 512, 16);
    DL_RES(2, 256, 16);
    DL_RES(1, 1024, 16);
    DL_RES(1, 512, 16);
    DL_RES(1, 256, 16);
#undef DL_RES
    return fail(DL_ERR_INVALID_ARG, "dl_eval_network: no kernel for rows of %d bytes", plan.V);
}
