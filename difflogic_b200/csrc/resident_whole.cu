// The whole-network kernel for networks that folding leaves nearly as they are, and for small passes (resident.cu has the idea and the
// folded form).
//
// Small passes: the host takes longer than either kernel, and this program is one launch per layer, where the folded one takes 26 launches
// for four layers and a table: second pass of 784 -> 4 x 2000, 10000 samples, 66 us, 203 folded.
//
// Every neuron is evaluated and its row's slot is its position in the layer: no output slots to fetch, no row that waits for a later
// reader, and the last layer's rows are put where their classes are, so that they are counted without a table.  That saves more
// than folding does once three quarters of the neurons are left as gates.  Folded / here, us, with all, 79, 69 and 58 % left:
//   784 -> 4 x 8000, 2^18 samples    237 / 216   225 / 212   208 / 208   202 / 204
//   784 -> 5 x 16000, 2^18           828 / 573   770 / 565   583 / 565   553 / 562
//   784 -> 4 x 4000, 2^19            242 / 205   227 / 200   217 / 199   206 / 195
//   256 -> 12 x 4000, 2^18           245 / 221   225 / 214   207 / 208   192 / 202
//   784 -> 12 x 12000, 2^16          291 / 234   231 / 232   169 / 231   157 / 230
//   784 -> 4 x 10000, 2^18           319 / 253   243 / 247   233 / 245   218 / 241
//
// Neurons are sorted by KIND, inversions pushed through to the readers: AND (a ^ i) & (b ^ j), XOR a ^ b, COPY a, CONST 0.
#include "common.cuh"
#include "resident.cuh"

namespace dl {

constexpr int kWholeLayers = 32;        // layers per network
constexpr int kWholeRows = 1 << 14;     // rows per layer or input
constexpr int kWholePlanes = 11;        // planes of a counting task: at most 2047 rows
constexpr int kWholePad = 1 << 14;      // words behind a program that a CTA may read and not use

struct WholeSizes {
    int layers;
    int n[kWholeLayers + 1];  // rows of the input and of every layer
};

constexpr int kWholeHeader = 4;  // words in front of a layer's program: where AND, XOR and COPY end
enum { kWholeAnd = 0, kWholeXor = 1, kWholeCopy = 2, kWholeConst = 3 };

// A gate in terms of the STORED rows of its inputs, which are the inverses of the inputs where inv_a / inv_b is set.
struct WholeGate {
    int kind, i, j, inv;  // inv: what is stored is the inverse of the gate's output
    bool second;          // COPY: the second input's row
};
__device__ __forceinline__ WholeGate whole_classify(int op, int inv_a, int inv_b) {
    const int t00 = (op >> 3) & 1, t01 = (op >> 2) & 1, t10 = (op >> 1) & 1, t11 = op & 1;
    const int ones = t00 + t01 + t10 + t11;
    WholeGate g = {kWholeConst, 0, 0, ones == 4, false};
    if (ones == 1 || ones == 3) {
        g.kind = kWholeAnd;
        g.inv = ones == 3;
        // the input pair whose output differs from the other three
        const int at = (t00 ^ g.inv) ? 0 : (t01 ^ g.inv) ? 1 : (t10 ^ g.inv) ? 2 : 3;
        g.i = (at < 2) ^ inv_a;           // AND of the inputs, inverted where they are 0 there
        g.j = (at % 2 == 0) ^ inv_b;
    } else if (ones == 2) {
        if (t00 == t11) {
            g.kind = kWholeXor;
            g.inv = t00 ^ inv_a ^ inv_b;
        } else {
            g.kind = kWholeCopy;
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
whole_program_kernel(const int64_t *__restrict__ a, const int64_t *__restrict__ b, const uint8_t *__restrict__ gate, int n_in,
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
        const WholeGate g = whole_classify((int)e.y, sa & 1, sb & 1);
        const int ca = (int)(sa >> 1) & (NC - 1), cb = (int)(sb >> 1) & (NC - 1), d = (cb - ca) & (NC - 1);
        int bucket, flip = 0;
        if (g.kind == kWholeConst) {
            bucket = (2 * NC + 1) * NC;
        } else if (g.kind == kWholeCopy) {
            flip = g.second;
            bucket = 2 * NC * NC + (flip ? cb : ca);
        } else {
            const int from = g.kind == kWholeXor ? NC * NC : 0;
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
        const WholeGate g = whole_classify((int)(e.y & 15u), sa & 1, sb & 1);
        const uint32_t first = (flip ? sb : sa) >> 1, second = (flip ? sa : sb) >> 1;
        prog[kWholeHeader + pos] = second | (uint32_t)(flip ? g.i : g.j) << 15 | first << 16 | (uint32_t)(flip ? g.j : g.i) << 31;
        if (slot_out != nullptr) slot_out[j] = (uint32_t)pos << 1 | (uint32_t)g.inv;
        if (order != nullptr) order[pos] = (uint32_t)j << 1 | (uint32_t)g.inv;
    }
}

// ---------------------------------------------------------------------------------------------
// evaluation
// ---------------------------------------------------------------------------------------------
// WORDS: 32-bit words per row of a block (V = 4 * WORDS bytes); T threads; R neurons per thread and layer at most.
template <int WORDS, int T, int R>
__global__ void __launch_bounds__(T, 1024 / T)
whole_kernel(const uint8_t *__restrict__ x, int64_t row_bytes, const uint32_t *__restrict__ prog, WholeSizes sz,
                int32_t *__restrict__ out, uint8_t *__restrict__ rows_out, int64_t batch, int k, int rows_per_class, int row_slots) {
    using Row = typename ResRow<WORDS>::type;
    constexpr int V = 4 * WORDS;
    extern __shared__ __align__(16) uint8_t whole_smem[];
    Row *rows = reinterpret_cast<Row *>(whole_smem);
    int *counts = reinterpret_cast<int *>(whole_smem + (size_t)row_slots * V);  // [8 V samples][k]
    const int tid = threadIdx.x;

    const uint8_t *src = x + (int64_t)blockIdx.x * V;
    for (int i = tid; i < sz.n[0]; i += T) rows[i] = __ldg(reinterpret_cast<const Row *>(src + (int64_t)i * row_bytes));
    for (int t = tid; t < 8 * V * k; t += T) counts[t] = 0;

    uint32_t w[R];
    int n = sz.n[1], and_end = (int)__ldg(prog), xor_end = (int)__ldg(prog + 1), copy_end = (int)__ldg(prog + 2);
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = r * T < n ? __ldg(prog + kWholeHeader + tid + r * T) : 0u;
    __syncthreads();
    for (int l = 1; l <= sz.layers; ++l) {
        const uint32_t *next = prog + kWholeHeader + n;  // program of the next layer; after the last one, the rows' order
        const bool last = l == sz.layers;
        const int n_next = last ? n : sz.n[l + 1];
        Row y[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r * T >= n) break;
            const int p = tid + r * T;
            const Row *first = reinterpret_cast<const Row *>(whole_smem + ((w[r] >> 16) & 0x3fffu) * V);
            const Row *second = reinterpret_cast<const Row *>(whole_smem + (w[r] & 0x3fffu) * V);
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
        for (int r = 0; r < R; ++r) w[r] = r * T < n_next ? __ldg(next + kWholeHeader + tid + r * T) : 0u;
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
    constexpr int kLane = kWholePlanes - kSteps;  // planes of one lane's count
    const int warp = tid / 32, lane = tid % 32, word = lane % WORDS, sub = lane / WORDS;
    const int parts = max(T / 32 / k, (rows_per_class + 511) / 512), tasks = k * parts;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(whole_smem) + word;
    for (int task = warp; task < tasks; task += T / 32) {
        const int c = task / parts, q = task % parts;
        const int beg = c * rows_per_class + rows_per_class * q / parts, end = c * rows_per_class + rows_per_class * (q + 1) / parts;
        uint32_t p[kWholePlanes];
#pragma unroll
        for (int i = 0; i < kWholePlanes; ++i) p[i] = 0u;
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
            for (int pl = 0; pl < kWholePlanes; ++pl) count |= (int)((p[pl] >> s) & 1u) << pl;
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

static size_t whole_shared_bytes(int row_slots, int V, int64_t k) { return (size_t)row_slots * V + (size_t)8 * V * k * sizeof(int); }

constexpr size_t kWholeMaxShared = 227 * 1024;

struct WholePlan {
    int V, T, R;
};

// V: the width for which the busiest SM has least to do.  A block of V bytes costs V bytes of row traffic per gate plus what does
// not depend on V (program words, instructions; about 8 bytes' worth).  Measured, us with V = 16 / 8 / 4, 784 -> 4 layers: 8000 wide,
// 100 samples: 19.5 / 18.3 / 18.0, 4000: 20.0 / 19.1 / 17.7, 10000: 20.0 / 24.0 / 28.7, 2^18: 207 / 255 / 399; 10000 wide, 19000: 38 / 48 / 63;
// 16000 wide, 5 layers, 10000: - / 46 / 54.
static WholePlan whole_plan(const int64_t *n, int layers, int64_t batch, int64_t k) {
    WholePlan best = {0, 0, 0};
    if (layers < 1 || layers > kWholeLayers || batch < 1 || k < 1) return best;
    int64_t most = 0;
    for (int l = 0; l <= layers; ++l) {
        if (n[l] < 1 || n[l] > kWholeRows) return best;
        most = n[l] > most ? n[l] : most;
    }
    if (n[layers] % k != 0) return best;
    int64_t widest = 0;
    for (int l = 1; l <= layers; ++l) widest = n[l] > widest ? n[l] : widest;
    const int sms = current_sms();
    int64_t least = 0;
    for (const int V : {16, 8, 4}) {
        const int R = V == 16 ? (widest <= 8 * 1024 ? 8 : 10) : 16;
        if (widest > (int64_t)R * 1024 || k > (1 << 14) || whole_shared_bytes((int)most, V, k) > kWholeMaxShared) continue;
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
static int launch_whole(const void *x, int64_t row_bytes, const uint32_t *prog, const WholeSizes &sz, int32_t *out, uint8_t *rows_out,
                           int64_t batch, int64_t k, int row_slots, cudaStream_t st) {
    constexpr int V = 4 * WORDS;
    const size_t smem = whole_shared_bytes(row_slots, V, k);
    // the most there may be, not this launch's bytes: the limit is the kernel's, and other threads launch it for other networks
    if (cudaFuncSetAttribute(whole_kernel<WORDS, T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWholeMaxShared) != cudaSuccess)
        return launch_status("dl_eval_whole (shared memory opt-in)");
    whole_kernel<WORDS, T, R><<<(unsigned)ceil_div(batch, 8 * V), T, smem, st>>>(
        reinterpret_cast<const uint8_t *>(x), row_bytes, prog, sz, out, rows_out, batch, (int)k, (int)(sz.n[sz.layers] / k), row_slots);
    return launch_status("dl_eval_whole");
}

// lanes that share a phase of a shared-memory access: the widest rows that the layer sizes allow
static int whole_classes(const int64_t *n, int layers) {
    int64_t most = 0;
    for (int l = 0; l <= layers; ++l) most = n[l] > most ? n[l] : most;
    return most > 10 * 1024 ? 16 : 8;
}

}  // namespace dl

using namespace dl;

static bool whole_applicable(const void *x, const int64_t *n, int layers, int64_t row_bytes, int64_t batch, int64_t k) {
    return x != nullptr && n != nullptr && row_bytes >= 16 && row_bytes % 16 == 0 && aligned_to(x, 16) && batch <= row_bytes * 8 &&
           whole_plan(n, layers, batch, k).V != 0;
}

// 32-bit words of the program of a network (the layers' words, the last layer's order, and scratch for building it).
extern "C" DL_API int64_t dl_network_whole_words(const int64_t *n, int layers) {
    if (n == nullptr || layers < 1 || layers > kWholeLayers) return 0;
    int64_t words = n[layers] + kWholeHeader, widest = 0;
    for (int l = 1; l <= layers; ++l) {
        words += n[l] + kWholeHeader;
        widest = n[l] > widest ? n[l] : widest;
    }
    return words + 2 * widest + kWholePad;
}

extern "C" DL_API int dl_network_whole(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n,
                                         int layers, uint32_t *program, void *stream) {
    DL_REQUIRE(a && b && gate && n && program, DL_ERR_INVALID_ARG, "dl_network_whole: null pointer");
    DL_REQUIRE(layers >= 1 && layers <= kWholeLayers, DL_ERR_INVALID_ARG, "dl_network_whole: 1 .. %d layers", kWholeLayers);
    int64_t total = n[layers] + kWholeHeader, widest = 0;
    for (int l = 0; l <= layers; ++l) {
        DL_REQUIRE(n[l] >= 1 && n[l] <= kWholeRows, DL_ERR_TOO_LARGE, "dl_network_whole: layers of 1 .. %d rows", kWholeRows);
        if (l > 0) {
            DL_REQUIRE(a[l - 1] && b[l - 1] && gate[l - 1], DL_ERR_INVALID_ARG, "dl_network_whole: null pointer");
            total += n[l] + kWholeHeader;
            widest = n[l] > widest ? n[l] : widest;
        }
    }
    uint32_t *at = program, *order = program + (total - n[layers]), *scratch = program + total;
    auto kernel = whole_classes(n, layers) == 8 ? whole_program_kernel<8> : whole_program_kernel<16>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kWholeRows * sizeof(uint2))) != cudaSuccess)
        return launch_status("dl_network_whole (shared memory opt-in)");
    for (int l = 1; l <= layers; ++l) {
        const uint32_t *slot_in = l == 1 ? nullptr : scratch + (int64_t)(l % 2) * widest;
        uint32_t *slot_out = l == layers ? nullptr : scratch + (int64_t)((l + 1) % 2) * widest;
        kernel<<<1, 1024, n[l] * sizeof(uint2), as_stream(stream)>>>(a[l - 1], b[l - 1], gate[l - 1], (int)n[l - 1], (int)n[l], slot_in, at,
                                                                     slot_out, l == layers ? order : nullptr);
        at += n[l] + kWholeHeader;
    }
    return launch_status("dl_network_whole");
}

extern "C" DL_API int dl_eval_whole(const void *x, const uint32_t *program, const int64_t *n, int layers, int32_t *out, void *rows_out,
                                      int64_t row_bytes, int64_t batch, int64_t k, void *stream) {
    DL_REQUIRE(program && (out != nullptr) != (rows_out != nullptr) && aligned_to(rows_out, 16) &&
                   whole_applicable(x, n, layers, row_bytes, batch, k), DL_ERR_INVALID_ARG,
               "dl_eval_whole: bad pointer or sizes outside the kernel's range (ask dl_eval_network_applicable first)");
    const WholePlan plan = whole_plan(n, layers, batch, k);
    WholeSizes sz = {};
    sz.layers = layers;
    int row_slots = 0;
    for (int l = 0; l <= layers; ++l) {
        sz.n[l] = (int)n[l];
        row_slots = sz.n[l] > row_slots ? sz.n[l] : row_slots;
    }
    cudaStream_t st = as_stream(stream);
#define DL_WHOLE(WW, TT, RR)          \
    if (plan.V == 4 * WW && plan.T == TT && plan.R == RR) return launch_whole<WW, TT, RR>(x, row_bytes, program, sz, out, reinterpret_cast<uint8_t *>(rows_out), batch, k, row_slots, st)
    DL_WHOLE(4, 1024, 8);
    DL_WHOLE(4, 512, 8);
    DL_WHOLE(4, 256, 8);
    DL_WHOLE(4, 1024, 10);
    DL_WHOLE(2, 1024, 16);
    DL_WHOLE(2, 512, 16);
    DL_WHOLE(2, 256, 16);
    DL_WHOLE(1, 1024, 16);
    DL_WHOLE(1, 512, 16);
    DL_WHOLE(1, 256, 16);
#undef DL_WHOLE
    return fail(DL_ERR_INVALID_ARG, "dl_eval_whole: no kernel for rows of %d bytes", plan.V);
}
