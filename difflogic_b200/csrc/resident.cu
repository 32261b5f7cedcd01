// Packed inference of a WHOLE network in one kernel: a CTA takes a narrow block of samples (V = 16, 8 or 4 bytes of every
// row) through all layers with the activations in shared memory, and counts the classes at the end.
//
// Why: layer by layer every activation row is written to memory and gathered again, 8000 gates x 2^20 samples: 1 GB out and
// 1 GB in per layer.  Here only the input bits are read and the counts written; a gate costs two shared-memory row loads and
// one row store.  What bounds it is shared-memory bandwidth, so bank conflicts decide: the rows of a layer are
// gathered at random, and a phase of NC = 128 / V lanes (8 lanes of 16 bytes ...) that hits random banks takes about 2.6
// cycles instead of one.  The PROGRAM of a network (once per set of weights) therefore puts the gates of a layer in an order in
// which the lanes of a phase read distinct bank classes, for both inputs, and gives every gate a row slot of its lane's class,
// so that stores are free of conflicts as well.
//
// The program is that of the FOLDED network (fold.cu): only gates that need both inputs and are read by something, each one
// AND(a ^ i, b ^ j) or XOR(a, b); a row that later layers only hand on stays in its slot until its last reader has read it.
//
// Measured, whole kernel, all neurons in the program and their rows put into class order for the counts -> now, us: 784 -> 4 x 8000, 2^20
// samples 826 -> 492 (1210 layer by layer); 784 -> 5 x 16000, 10000 samples 45 -> 23, 2^18 560 -> 248; 784 -> 12 x 12000, 2^17 451 -> 167;
// 256 -> 12 x 4000, 2^18 201 -> 85; 784 -> 4 x 8000, 100 samples 14.4 -> 15.7 (four CTAs whose loads wait for one another): so few
// run in resident_whole.cu.  What is left as gates: 40 % of the neurons with gates drawn evenly; networks of which three quarters are left
// run there as well.  Shared-memory pipe 59 %, issue 59 % busy: neither is what bounds it alone; a block goes through load, layers and counts one after
// the other and two blocks share an SM.  Loading
// the input four rows per thread at a time, and fetching the next block's into L2, changed nothing.
//
// CTAs that stay for several blocks and fetch the next one's input while they count were slower (needs more than 64 registers:
// 16000 wide, 10000 samples 45 -> 51 us, 8000 wide, 2^18 samples 208 -> 212).
//
// In-place update: a thread keeps the outputs of its R gates in registers until every thread has read its inputs, then
// all store -- into the slots of rows that nothing reads any more, too.  So a network never needs more slots than its widest
// layer has rows, and mostly far fewer, which lets several blocks share an SM.
//
// Program word of a gate, 32 bits: second slot (bits 0 .. 13), j (15), first slot (16 .. 29), i (31), so layers and inputs are
// limited to 16384 rows; 16 more bits say where the output goes.  Both are read from L2 by every CTA: 6 bytes per gate against
// 3 V bytes of shared-memory traffic.
#include "common.cuh"
#include "fold.cuh"
#include "resident.cuh"
#include "gates.cuh"

namespace dl {

constexpr int kResLayers = kFoldLayers;  // layers per network: a lane each
constexpr int kResRows = 1 << 14;        // rows per layer or input
constexpr int kResPad = 1 << 14;         // words behind a program that a CTA may read and not use

struct ResidentSizes {
    int layers;
    int n[kResLayers + 1];  // rows of the input and of every layer
};

// A program, in 32-bit words: a header {slots, most gates of a layer, bank classes, gates in all}; per layer a header {gates that
// are ANDs, gates}, the gates'
// words and their output slots (16 bits each); the last layer's rows (16 bits each: slot, above it whether inverted).  A warp takes
// 64 gates at a time, lane l gates l and l + 32, whose words lie side by side.
constexpr int kResHeader = 4;
constexpr int kResPitch = 33;   // counts of a word's 32 samples
constexpr int kResOutput = 15;  // bit of the last layer's entry: inverted
__host__ __device__ __forceinline__ int res_whole(int n) { return (n + 63) / 64 * 64; }
__host__ __device__ __forceinline__ int64_t res_layer_words(int n) { return kResHeader + res_whole(n) / 2 * 3; }
__device__ __forceinline__ int res_place(int p) { return p / 64 * 64 + p % 32 * 2 + p % 64 / 32; }

// ---------------------------------------------------------------------------------------------
// program: two launches per layer, after those of the folding
// ---------------------------------------------------------------------------------------------
// A gate reads bank classes ca and cb = ca + d (mod NC).  Gates of the same kind and d are dealt out in rounds over ca =
// 0 .. NC-1: NC consecutive ones then read NC distinct classes with either input.  A gate may be taken with its inputs
// swapped (class cb, difference -d): of a bucket and its counterpart the fuller one hands over half of the difference, which
// keeps the rounds full.
//
// Slots of rows without a reader wait on one stack per class.  A gate in position p takes a slot of class p mod NC: from the
// stack, then one that was never used, and where the class has neither, what other classes have left.
constexpr int kResClasses = 16;  // NC is 8 (rows of 16 bytes) or 16
constexpr int kResBuckets = 2 * kResClasses * kResClasses;

struct ResBuild {
    const int32_t *fold_header, *ref, *in_a, *in_b;
    int32_t *use;     // by value; -1 where its slot has been given back
    int32_t *slot;    // by value
    int32_t *rank;    // by neuron of the layer: bucket << 16 | place in it, -1: no gate
    int32_t *bucket;  // [layers][kResBuckets]
    int32_t *state;   // [layers + 1][2 kResClasses]: by class, slots on its stack and slots ever used
    int32_t *stack;   // [class][slots / NC]
    int slots;        // there may be at most
    int layers, n0;
};

// Bank classes: those of rows of 16 bytes if as many rows as are ever needed at a time fit shared memory in that width.
__device__ __forceinline__ int res_classes(const ResBuild &p) {
    int live = p.n0, most = p.n0;
    for (int l = 1; l <= p.layers; ++l) {
        live += __ldcg(p.fold_header + l) - __ldcg(p.fold_header + kFoldDead + l);
        most = max(most, live);
    }
    return most > 10 * 1024 ? 16 : 8;
}
__device__ __forceinline__ int res_stack_room(const ResBuild &p, int nc) { return p.slots / nc + 1; }

__device__ __forceinline__ void res_give_back(const ResBuild &p, int nc, int32_t *state, int slot) {
    const int c = slot & (nc - 1);
    p.stack[(int64_t)c * res_stack_room(p, nc) + atomicAdd(state + c, 1)] = slot;
}

// Gates in all, for those who want to know before the program is made.
__global__ void __launch_bounds__(32)
res_left_kernel(ResBuild p, uint32_t *__restrict__ prog) {
    grid_dependency_wait();
    const int left = __reduce_add_sync(0xffffffffu, (int)threadIdx.x < p.layers ? __ldcg(p.fold_header + 1 + threadIdx.x) : 0);
    if (threadIdx.x == 0) prog[3] = (uint32_t)left;
}

// The input's rows are in slots 0 ..; those that nothing reads are free from the start.
__global__ void __launch_bounds__(kThreads)
res_inputs_kernel(ResBuild p, uint32_t *__restrict__ prog) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int nc = res_classes(p), i = blockIdx.x * kThreads + threadIdx.x;
    if (i < nc) p.state[kResClasses + i] = (p.n0 - i + nc - 1) / nc;
    if (i == 0) {
        prog[0] = (uint32_t)p.n0;
        prog[1] = 0u;
        prog[2] = (uint32_t)nc;
        prog[3] = 0u;
    }
    if (i >= p.n0) return;
    p.slot[i] = i;
    if (__ldcg(p.use + i) == 0) res_give_back(p, nc, p.state, i);
}

__global__ void __launch_bounds__(kThreads)
res_bucket_kernel(ResBuild p, int layer, int first, int n, const uint32_t *__restrict__ prog) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int j = blockIdx.x * kThreads + threadIdx.x, nc = (int)__ldcg(prog + 2);
    if (j >= n) return;
    const int vb = p.in_b[first - p.n0 + j], op = vb >> kFoldValueBits;
    int mark = -1;
    if (op != 0 && __ldcg(p.use + first + j) != 0) {
        const int va = p.in_a[first - p.n0 + j], v2 = vb & ((1 << kFoldValueBits) - 1);
        const int sa = __ldcg(p.slot + va), sb = __ldcg(p.slot + v2);
        const int ca = sa & (nc - 1), d = (sb - sa) & (nc - 1);
        const int bucket = ((op == 6 ? nc : 0) + d) * nc + ca;
        mark = bucket << 16 | atomicAdd(p.bucket + (int64_t)(layer - 1) * kResBuckets + bucket, 1);
        int32_t *state = p.state + (int64_t)(layer - 1) * 2 * kResClasses;
        if (__ldcg(p.use + va) == layer && atomicCAS(p.use + va, layer, -1) == layer) res_give_back(p, nc, state, sa);
        if (__ldcg(p.use + v2) == layer && atomicCAS(p.use + v2, layer, -1) == layer) res_give_back(p, nc, state, sb);
    }
    p.rank[j] = mark;
}

__global__ void __launch_bounds__(kThreads)
res_place_kernel(ResBuild p, int layer, int first, int n, uint32_t *__restrict__ prog, uint32_t *__restrict__ level) {
    __shared__ int s_raw[kResBuckets], s_cnt[kResBuckets], s_base[2 * kResClasses + 1];
    __shared__ int s_have[kResClasses], s_room[kResClasses], s_used[kResClasses], s_lack[kResClasses + 1], s_spare[kResClasses + 1];
    const int tid = threadIdx.x, j = blockIdx.x * kThreads + tid;
    grid_dependency_wait();
    grid_dependents_launch();
    const int nc = (int)__ldcg(prog + 2), buckets = 2 * nc * nc;
    for (int t = tid; t < buckets; t += kThreads) s_raw[t] = __ldcg(p.bucket + (int64_t)(layer - 1) * kResBuckets + t);
    const int32_t *state = p.state + (int64_t)(layer - 1) * 2 * kResClasses;
    if (tid < nc) {
        s_have[tid] = __ldcg(state + tid);
        s_used[tid] = __ldcg(state + kResClasses + tid);
        s_room[tid] = (p.slots - tid + nc - 1) / nc - s_used[tid];
    }
    auto counterpart = [&](int t) {  // (kind, d, ca) -> (kind, -d, ca + d)
        const int ca = t & (nc - 1), d = t / nc & (nc - 1);
        return t - (d * nc + ca) + ((nc - d) & (nc - 1)) * nc + ((ca + d) & (nc - 1));
    };
    __syncthreads();
    for (int t = tid; t < buckets; t += kThreads) {
        const int x = s_raw[t], y = s_raw[counterpart(t)];
        s_cnt[t] = x > y ? (x + y + 1) / 2 : x < y ? (x + y) / 2 : x;
    }
    __syncthreads();
    if (tid < 2 * nc) {
        int size = 0;
        for (int i = 0; i < nc; ++i) size += s_cnt[tid * nc + i];
        s_base[tid + 1] = size;
    }
    __syncthreads();
    if (tid == 0) {
        s_base[0] = 0;
        for (int t = 1; t <= 2 * nc; ++t) s_base[t] += s_base[t - 1];
        const int total = s_base[2 * nc];
        s_lack[0] = s_spare[0] = 0;
        for (int c = 0; c < nc; ++c) {
            const int need = total / nc + (c < total % nc), there = s_have[c] + s_room[c];
            s_lack[c + 1] = s_lack[c] + max(0, need - there);
            s_spare[c + 1] = s_spare[c] + max(0, there - need);
        }
    }
    __syncthreads();
    const int total = s_base[2 * nc];
    // slot r of class c: its stack from the top, then what was never used
    auto slot_of = [&](int c, int r) {
        return r < s_have[c] ? p.stack[(int64_t)c * res_stack_room(p, nc) + s_have[c] - 1 - r] : (s_used[c] + r - s_have[c]) * nc + c;
    };
    if (blockIdx.x == 0 && tid == 0) {
        level[0] = (uint32_t)s_base[nc];
        level[1] = (uint32_t)total;
        int slots = (int)__ldcg(prog), left = s_lack[nc];
        int32_t *next = p.state + (int64_t)layer * 2 * kResClasses;
        for (int c = 0; c < nc; ++c) {
            const int need = total / nc + (c < total % nc), there = s_have[c] + s_room[c];
            int taken = min(need, there);
            const int more = min(left, there - taken);  // for classes that lack slots
            taken += more;
            left -= more;
            next[c] = max(0, s_have[c] - taken);
            const int used = s_used[c] + max(0, taken - s_have[c]);
            next[kResClasses + c] = used;
            if (used > 0) slots = max(slots, (used - 1) * nc + c + 1);
        }
        prog[0] = (uint32_t)slots;
        prog[1] = max(__ldcg(prog + 1), (uint32_t)total);
        prog[3] = __ldcg(prog + 3) + (uint32_t)total;
    }
    if (j >= n) return;
    const int mark = p.rank[j];
    if (mark < 0) return;
    int bucket = mark >> 16, rank = mark & 0xffff;
    const int other = counterpart(bucket), x = s_raw[bucket], y = s_raw[other], half = (x + y + 1) / 2;
    const bool flip = x > y && rank >= half;
    if (flip) {
        bucket = other;
        rank = y + rank - half;
    }
    const int group = bucket / nc, ca = bucket % nc;
    int pos = s_base[group];  // gates of this group in earlier rounds, and earlier in this round
    for (int i = 0; i < nc; ++i) {
        const int have = s_cnt[group * nc + i];
        pos += min(have, rank) + (i < ca && have > rank ? 1 : 0);
    }
    const int vb = p.in_b[first - p.n0 + j], op = vb >> kFoldValueBits;
    const int sa = __ldcg(p.slot + p.in_a[first - p.n0 + j]), sb = __ldcg(p.slot + (vb & ((1 << kFoldValueBits) - 1)));
    uint32_t ia = op & 12 ? 1u : 0u, ib = op & 10 ? 1u : 0u;  // AND: the input pair for which it is true has zeros there
    if (op == 6) ia = ib = 0u;
    const uint32_t one = (uint32_t)sa | ia << 15, two = (uint32_t)sb | ib << 15;
    // out
    int c = pos & (nc - 1), r = pos / nc;
    if (r >= s_have[c] + s_room[c]) {
        const int lack = s_lack[c] + r - s_have[c] - s_room[c];
        for (c = 0; c < nc - 1 && s_spare[c + 1] <= lack; ++c) {
        }
        r = total / nc + (c < total % nc) + lack - s_spare[c];
    }
    const int out = slot_of(c, r), at = res_place(pos);
    level[kResHeader + at] = flip ? one | two << 16 : two | one << 16;
    reinterpret_cast<uint16_t *>(level + kResHeader + res_whole(n))[at] = (uint16_t)out;
    p.slot[first + j] = out;
}

// The last layer's rows: a constant is the row behind all slots, which holds zeros.
__global__ void __launch_bounds__(kThreads)
res_outputs_kernel(ResBuild p, int n, const int32_t *__restrict__ ref, const uint32_t *__restrict__ prog, uint16_t *__restrict__ outputs) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= n) return;
    const int r = __ldcg(ref + j);
    const int slot = ref_is_constant(r) ? (int)__ldcg(prog) : __ldcg(p.slot + (r >> 1));
    outputs[j] = (uint16_t)(slot | (r & 1) << kResOutput);
}

// ---------------------------------------------------------------------------------------------
// class table of a program: what the last layer's rows are when they are counted in k classes
// ---------------------------------------------------------------------------------------------
// By class: constants that are true (they are counted once and for all), and the rows, dealt out over the bank classes as above.
// A class begins with a whole group of 8 NC entries.  A lane of the counting loop loads eight entries at a time, so the entries
// of a group lie lane by lane: entry q at (q mod NC) * 8 + q / NC.  Short classes, of which groups would be mostly empty, take whole
// eights instead, in order.  What a class does not fill reads the row of zeros.
constexpr int kResShort = 256;  // rows of a class
struct ResTable {
    uint32_t *start;    // [k + 1] first entry, by class
    uint32_t *ones;     // [k]
    uint16_t *entries;
    int32_t *count;     // [k][kResClasses]
    int32_t *rank;      // by row of the last layer
    int64_t room;       // entries
};
static int64_t res_table_words(int64_t n, int64_t k, ResTable *t, uint32_t *at) {
    t->room = (n + k * 8 * kResClasses + 7) / 8 * 8;
    t->entries = reinterpret_cast<uint16_t *>(at);  // 16-byte aligned
    t->start = at + t->room / 2;
    t->ones = t->start + k + 1;
    t->count = reinterpret_cast<int32_t *>(t->ones + k);  // cleared with them
    t->rank = t->count + k * kResClasses;
    return t->room / 2 + 2 * k + 1 + k * kResClasses + n;
}

__global__ void __launch_bounds__(kThreads)
res_table_count_kernel(ResTable t, int n, int rows_per_class, const uint32_t *__restrict__ prog, const uint16_t *__restrict__ outputs) {
    grid_dependents_launch();
    const int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const uint32_t zero = __ldg(prog), nc = __ldg(prog + 2);
    if (j < t.room / 2) reinterpret_cast<uint32_t *>(t.entries)[j] = zero << 16 | zero;
    if (j >= n) return;
    const uint32_t e = outputs[j], slot = e & ((1u << kResOutput) - 1u);
    const int64_t c = j / rows_per_class;
    int rank = -1;
    if (slot == zero) {
        if (e >> kResOutput) atomicAdd(t.ones + c, 1u);
    } else {
        rank = atomicAdd(t.count + c * kResClasses + (slot & (nc - 1)), 1);
    }
    t.rank[j] = rank;
}

__global__ void __launch_bounds__(1024)
res_table_start_kernel(ResTable t, int k, int rows_per_class, const uint32_t *__restrict__ prog) {
    __shared__ int s_sum[1024];
    grid_dependency_wait();
    grid_dependents_launch();
    const int tid = threadIdx.x, each = (k + 1023) / 1024, group = rows_per_class < kResShort ? 8 : 8 * (int)__ldg(prog + 2);
    auto entries = [&](int c) {
        int rows = 0;
        for (int i = 0; i < kResClasses; ++i) rows += __ldcg(t.count + (int64_t)c * kResClasses + i);
        return (rows + group - 1) / group * group;
    };
    int mine = 0;
    for (int c = tid * each; c < min(k, (tid + 1) * each); ++c) mine += entries(c);
    s_sum[tid] = mine;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
        const int v = tid >= d ? s_sum[tid - d] : 0;
        __syncthreads();
        s_sum[tid] += v;
        __syncthreads();
    }
    int at = s_sum[tid] - mine;
    for (int c = tid * each; c < min(k, (tid + 1) * each); ++c) {
        t.start[c] = (uint32_t)at;
        at += entries(c);
    }
    if (tid == 1023) t.start[k] = (uint32_t)s_sum[tid];
}

__global__ void __launch_bounds__(kThreads)
res_table_place_kernel(ResTable t, int n, int rows_per_class, const uint32_t *__restrict__ prog, const uint16_t *__restrict__ outputs) {
    grid_dependency_wait();
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= n) return;
    const int rank = t.rank[j], nc = (int)__ldg(prog + 2), c = j / rows_per_class;
    if (rank < 0) return;
    const uint32_t e = outputs[j];
    const int cls = (int)e & (nc - 1);
    int q = 0;
    for (int i = 0; i < nc; ++i) {
        const int have = __ldcg(t.count + (int64_t)c * kResClasses + i);
        q += min(have, rank) + (i < cls && have > rank ? 1 : 0);
    }
    const int group = 8 * nc;
    if (rows_per_class >= kResShort) q = q / group * group + q % nc * 8 + q % group / nc;
    t.entries[__ldcg(t.start + c) + q] = (uint16_t)e;
}

// ---------------------------------------------------------------------------------------------
// evaluation
// ---------------------------------------------------------------------------------------------
// Rows that a group of lanes counts side by side: all that a warp has lanes for, or fewer where there are more classes than warps.
template <int WORDS, int T>
__device__ __forceinline__ int res_side_by_side(int k) {
    constexpr int kParts = WORDS < 2 ? 1 : WORDS / 2;
    int subs = 32 / kParts;
    while (subs > 1 && subs * kParts * k > T) subs /= 2;
    return subs;
}

// The counts of many classes: groups of as few lanes as there are classes for (down to the parts of one row) take a class each, and
// the sums over the lanes, which cost as much as 200 rows, shrink with them.  400 -> 4 x 1000, 100 classes, 2^18 samples: 193 us with a
// warp per class, 120 so; 400 -> 3 x 8000, 1000 classes, 2^14: 308 and 74.  A function of its own: as part of the kernel it takes
// registers away from the layers (784 -> 12 x 12000: 189 -> 206 us).
template <int WORDS, int T>
__device__ __noinline__ void res_count_many(int row_slots, const uint32_t *__restrict__ table, const uint16_t *__restrict__ outputs,
                                               int zero_row, int k) {
    constexpr int V = 4 * WORDS, kPitch = kResPitch * WORDS;
    extern __shared__ __align__(16) uint8_t res_smem[];
    int *counts = reinterpret_cast<int *>(res_smem + (size_t)row_slots * V);
    const int *starts = counts + kPitch * k;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr int kWords = WORDS < 2 ? 1 : 2, kParts = WORDS / kWords;  // words of a lane, lanes of a row
    constexpr int kSubs = 32 / kParts;
    constexpr int kSteps = kSubs == 16 ? 4 : 5;                        // of adding up over the lanes, at most
    constexpr int kLane = 6, kPlanes = kLane + kSteps;                 // planes of a lane's count, and of the sum
    constexpr int kLaneRows = 56;                                      // rows of a lane at a time at most
    using Pair = typename ResRow<kWords>::type;
    const int subs = res_side_by_side<WORDS, T>(k);
    const int part = lane % kParts;
    const uint8_t *mine = res_smem + part * (int)sizeof(Pair);
    auto fetch = [&](int r, int end) {
        const uint32_t none = (uint32_t)zero_row << 16 | (uint32_t)zero_row;
        uint4 e = make_uint4(none, none, none, none);
        if (table != nullptr) {
            if (r < end) e = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(table) + r));
        } else {
            uint32_t *half = &e.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (r + 2 * i < end) half[i] = (half[i] & 0xffff0000u) | __ldg(outputs + r + 2 * i);
                if (r + 2 * i + 1 < end) half[i] = (half[i] & 0xffffu) | (uint32_t)__ldg(outputs + r + 2 * i + 1) << 16;
            }
        }
        return e;
    };
    // rows pos .. end - 1 (at most kLaneRows * subs) of class c, which may be none; all groups of a warp together.
    auto count_rows = [&](int c, int pos, int end) {
        const int sub = lane / kParts % subs, stride = 8 * subs;

        uint32_t p[kWords][kPlanes];
#pragma unroll
        for (int i = 0; i < kPlanes; ++i)
#pragma unroll
            for (int h = 0; h < kWords; ++h) p[h][i] = 0u;
        auto add8 = [&](uint32_t (&q)[kPlanes], const uint32_t (&v)[8]) {
            uint32_t t2a, t2b, t4a, t4b, carry;
            DL_CSA32(t2a, q[0], q[0], v[0], v[1]);
            DL_CSA32(t2b, q[0], q[0], v[2], v[3]);
            DL_CSA32(t4a, q[1], q[1], t2a, t2b);
            DL_CSA32(t2a, q[0], q[0], v[4], v[5]);
            DL_CSA32(t2b, q[0], q[0], v[6], v[7]);
            DL_CSA32(t4b, q[1], q[1], t2a, t2b);
            DL_CSA32(carry, q[2], q[2], t4a, t4b);
#pragma unroll
            for (int i = 3; i < kLane; ++i) {
                const uint32_t t = q[i] & carry;
                q[i] ^= carry;
                carry = t;
            }
        };
        int r = pos + sub * 8;
        uint4 e = fetch(r, end);
        while (__any_sync(0xffffffffu, r < end)) {
            r += stride;
            const uint4 next = fetch(r, end);
            const uint32_t pairs[4] = {e.x, e.y, e.z, e.w};
            uint32_t v[kWords][8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t one = i % 2 ? pairs[i / 2] >> 16 : pairs[i / 2], m = res_mask15(one);
                const Pair row = *reinterpret_cast<const Pair *>(mine + (one & ((1u << kResOutput) - 1u)) * V);
                v[0][i] = *reinterpret_cast<const uint32_t *>(&row) ^ m;
                if (kWords == 2) v[kWords - 1][i] = (reinterpret_cast<const uint32_t *>(&row))[kWords - 1] ^ m;
            }
#pragma unroll
            for (int h = 0; h < kWords; ++h) add8(p[h], v[h]);
            e = next;
        }
        // four samples' counts, from a nibble of each plane a bit in each of four bytes, are added
        auto put = [&](const uint32_t (&planes)[kPlanes], int word, int first, int from, int step) {
            uint32_t low = 0u, high = 0u;
#pragma unroll
            for (int pl = 0; pl < kPlanes; ++pl) {
                const uint32_t bits = (((planes[pl] >> first) & 15u) * 0x00204081u) & 0x01010101u;
                if (pl < 8) low |= bits << pl;
                else high |= bits << (pl - 8);
            }
            int *at = counts + c * kPitch + word * kResPitch + first;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int count = (int)((low >> (8 * i)) & 255u) | (int)((high >> (8 * i)) & 255u) << 8;
                if (i % step == from && count) atomicAdd(at + i, count);
            }
        };
        if (subs == 1) {
#pragma unroll
            for (int h = 0; h < kWords; ++h)
#pragma unroll 1
                for (int nibble = 0; nibble < 8; ++nibble) put(p[h], part * kWords + h, 4 * nibble, 0, 1);
            return;
        }
        // sums over the lanes of a part, a plane more each time; in the first step a lane hands one of its two words over and
        // keeps the other
        const bool upper = kWords == 2 && (sub & 1);
        uint32_t s[kPlanes];
#pragma unroll
        for (int i = 0; i < kPlanes; ++i) s[i] = upper ? p[kWords - 1][i] : p[0][i];
#pragma unroll
        for (int step = 0; step < kSteps; ++step) {
            if (1 << step >= subs) break;
            uint32_t carry = 0u;
#pragma unroll
            for (int i = 0; i < kLane + step; ++i) {
                const uint32_t give = step == 0 && kWords == 2 ? (upper ? p[0][i] : p[kWords - 1][i]) : s[i];
                const uint32_t o = __shfl_xor_sync(0xffffffffu, give, kParts << step);
                uint32_t h, l;
                DL_CSA32(h, l, s[i], o, carry);
                s[i] = l;
                carry = h;
            }
            s[kLane + step] = carry;
        }
        // the lanes that hold one word's sums share its samples, four at a time, or four among two lanes and more
        const int holders = subs / kWords, holder = sub / kWords, word = part * kWords + (upper ? 1 : 0);
        if (holders >= 8) {
            const int share = holders / 8;
            put(s, word, holder / share * 4, holder % share, share);
        } else {
#pragma unroll 1
            for (int nibble = holder; nibble < 8; nibble += holders) put(s, word, 4 * nibble, 0, 1);
        }
    };
    const int lanes = kParts * subs;
    for (int c0 = warp * (32 / lanes); c0 < k; c0 += T / lanes) {
        const int c = min(c0 + lane / lanes, k - 1);
        int pos = starts[c];
        const int stop = c0 + lane / lanes < k ? starts[c + 1] : pos;
        while (__any_sync(0xffffffffu, pos < stop)) {
            const int end = min(stop, pos + kLaneRows * subs);
            count_rows(c, pos, end);
            pos = end;
        }
    }
}

// WORDS: 32-bit words per row of a block (V = 4 * WORDS bytes); T threads; R gates per thread and layer at most.
template <int WORDS, int T, int R>
__global__ void __launch_bounds__(T, 1024 / T)
resident_kernel(const uint8_t *__restrict__ x, int64_t row_bytes, const uint32_t *__restrict__ prog, ResidentSizes sz,
                const uint32_t *__restrict__ table, int32_t *__restrict__ out, uint8_t *__restrict__ rows_out, int64_t batch, int k,
                int rows_per_class, int row_slots) {
    using Row = typename ResRow<WORDS>::type;
    constexpr int V = 4 * WORDS, W = T / 32;
    static_assert(R % 2 == 0, "gates are taken in pairs");
    extern __shared__ __align__(16) uint8_t res_smem[];
    Row *rows = reinterpret_cast<Row *>(res_smem);
    int *counts = reinterpret_cast<int *>(res_smem + (size_t)row_slots * V);  // [k][WORDS][33]: a word's samples, and no two words' in a bank
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;

    const uint8_t *src = x + (int64_t)blockIdx.x * V;
    for (int i = tid; i < sz.n[0]; i += T) rows[i] = __ldg(reinterpret_cast<const Row *>(src + (int64_t)i * row_bytes));
    const int zero_row = (int)__ldg(prog);
    // the rows to be counted, by class: those of a table, or all in their own order
    const uint32_t *start_of = table != nullptr ? table + (sz.n[sz.layers] + (int64_t)k * 8 * kResClasses + 7) / 8 * 4 : nullptr;
    constexpr int kPitch = kResPitch * WORDS;
    int *starts = counts + kPitch * k;  // [k + 1]
    if (rows_out == nullptr) {
        for (int t = tid; t <= k; t += T) starts[t] = start_of != nullptr ? (int)__ldg(start_of + t) : t * rows_per_class;
        for (int t = tid; t < kPitch * k; t += T) counts[t] = start_of != nullptr ? (int)__ldg(start_of + k + 1 + t / kPitch) : 0;
    }

    // layer l: `level`; its output slots are fetched before its gates are evaluated, the gates of the next one before the rows are
    // exchanged (rows of 4 bytes) or behind the last use of the slots (wider ones: held at the same time they do not fit the registers)
    // and, so that this is short, into L1 before
    constexpr bool kEarly = WORDS == 1;
    const uint32_t *level = prog + kResHeader;
    uint2 w[R / 2];
    uint32_t o[R / 2];
    auto fetch_gates = [&](const uint32_t *at, int gates) {
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
            const int chunk = warp + r * W;
            w[r] = chunk * 64 < gates ? __ldg(reinterpret_cast<const uint2 *>(at + kResHeader) + chunk * 32 + lane) : make_uint2(0u, 0u);
        }
    };
    int and_end = (int)__ldg(level), n = (int)__ldg(level + 1);
    fetch_gates(level, n);
    __syncthreads();
    for (int l = 1; l <= sz.layers; ++l) {
        const uint32_t *outs = level + kResHeader + res_whole(sz.n[l]);
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
            const int chunk = warp + r * W;
            o[r] = chunk * 64 < n ? __ldg(outs + chunk * 32 + lane) : 0u;
        }
        int next_and_end = 0, next_n = 0;
        if (l < sz.layers) {
            const uint32_t *ahead = level + res_layer_words(sz.n[l]);
            next_and_end = (int)__ldg(ahead);
            next_n = (int)__ldg(ahead + 1);
            for (int t = tid * 32; t < kResHeader + (int)sz.n[l + 1]; t += T * 32)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead + t));
        }
        Row y[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if ((warp + r / 2 * W) * 64 >= n) break;
            const int p = (warp + r / 2 * W) * 64 + r % 2 * 32 + lane;
            const uint32_t g = r % 2 ? w[r / 2].y : w[r / 2].x;
            const Row *first = reinterpret_cast<const Row *>(res_smem + ((g >> 16) & 0x3fffu) * V);
            const Row *second = reinterpret_cast<const Row *>(res_smem + (g & 0x3fffu) * V);
            if (p < and_end) y[r] = res_and(*first, *second, (uint32_t)((int)g >> 31), res_mask15(g));
            else if (p < n) y[r] = res_xor(*first, *second);
        }
        const int live = n;
        level += res_layer_words(sz.n[l]);
        if (kEarly && l < sz.layers) fetch_gates(level, next_n);
        and_end = next_and_end;
        n = next_n;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            // (checked for every pair of gates, rows of 16 bytes are stored later: 784 -> 5 x 16000 248 -> 261 us; never: 784 -> 12 x 12000 167 -> 182)
            if ((WORDS == 1 || r == R / 2 / 2 * 2) && (warp + r / 2 * W) * 64 >= live) break;
            const int p = (warp + r / 2 * W) * 64 + r % 2 * 32 + lane;
            if (p < live) rows[r % 2 ? o[r / 2] >> 16 : o[r / 2] & 0xffffu] = y[r];
        }
        if (!kEarly && l < sz.layers) fetch_gates(level, n);
        if (l == sz.layers && tid == 0) res_fill(rows[zero_row], 0u);
        __syncthreads();
    }
    const uint16_t *outputs = reinterpret_cast<const uint16_t *>(level);
    if (rows_out != nullptr) {  // the rows themselves are wanted
        uint8_t *dst = rows_out + (int64_t)blockIdx.x * V;
        for (int j = tid; j < sz.n[sz.layers]; j += T) {
            const uint32_t e = __ldg(outputs + j);
            Row m;
            res_fill(m, 0u - (e >> kResOutput));
            *reinterpret_cast<Row *>(dst + (int64_t)j * row_bytes) = res_xor(rows[e & ((1u << kResOutput) - 1u)], m);
        }
        return;
    }

    // ---- class counts.  Many classes: see there.  Else every warp takes its share of the rows, class by class.  A lane adds up eight
    // rows at a time of one row word, or of two (an instruction that finds a row is paid once for both); lane = (row, part of a row) ----
    constexpr int kWords = WORDS < 2 ? 1 : 2, kParts = WORDS / kWords;  // words of a lane, lanes of a row
    constexpr int kSubs = 32 / kParts;
    constexpr int kSteps = kSubs == 16 ? 4 : 5;                        // of adding up over the lanes
    constexpr int kLane = 6, kPlanes = kLane + kSteps;                 // planes of a lane's count, and of the sum
    constexpr int kStride = 8 * kSubs, kRun = kStride * 7;             // rows per step, and at a time at most: 56 of a lane
    using Pair = typename ResRow<kWords>::type;
    const int part = lane % kParts, sub = lane / kParts;
    const uint8_t *mine = res_smem + part * (int)sizeof(Pair);
    const bool many = res_side_by_side<WORDS, T>(k) < kSubs;
    if (many) res_count_many<WORDS, T>(row_slots, table, outputs, zero_row, k);
    const int total = many ? 0 : starts[k], share = (total / 8 + W) / W * 8;
    int pos = min(total, warp * share), c = 0;
    const int stop = min(total, pos + share);
    for (int hi = k; hi - c > 1;) {  // the class of row `pos`
        const int mid = (c + hi) / 2;
        if (starts[mid] <= pos) c = mid;
        else hi = mid;
    }
    auto fetch = [&](int r, int end) {
        const uint32_t none = (uint32_t)zero_row << 16 | (uint32_t)zero_row;
        uint4 e = make_uint4(none, none, none, none);
        if (table != nullptr) {
            if (r < end) e = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(table) + r));
        } else {
            uint32_t *half = &e.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (r + 2 * i < end) half[i] = (half[i] & 0xffff0000u) | __ldg(outputs + r + 2 * i);
                if (r + 2 * i + 1 < end) half[i] = (half[i] & 0xffffu) | (uint32_t)__ldg(outputs + r + 2 * i + 1) << 16;
            }
        }
        return e;
    };
    while (pos < stop) {
        while (starts[c + 1] <= pos) ++c;
        const int end = min(min(stop, starts[c + 1]), pos + kRun);
        uint32_t p[kWords][kPlanes];
#pragma unroll
        for (int i = 0; i < kPlanes; ++i)
#pragma unroll
            for (int h = 0; h < kWords; ++h) p[h][i] = 0u;
        auto add8 = [&](uint32_t (&q)[kPlanes], const uint32_t (&v)[8]) {
            uint32_t t2a, t2b, t4a, t4b, carry;
            DL_CSA32(t2a, q[0], q[0], v[0], v[1]);
            DL_CSA32(t2b, q[0], q[0], v[2], v[3]);
            DL_CSA32(t4a, q[1], q[1], t2a, t2b);
            DL_CSA32(t2a, q[0], q[0], v[4], v[5]);
            DL_CSA32(t2b, q[0], q[0], v[6], v[7]);
            DL_CSA32(t4b, q[1], q[1], t2a, t2b);
            DL_CSA32(carry, q[2], q[2], t4a, t4b);
#pragma unroll
            for (int i = 3; i < kLane; ++i) {
                const uint32_t t = q[i] & carry;
                q[i] ^= carry;
                carry = t;
            }
        };
        uint4 e = fetch(pos + sub * 8, end);
        for (; pos < end; pos += kStride) {
            const uint4 next = fetch(pos + kStride + sub * 8, end);
            const uint32_t pairs[4] = {e.x, e.y, e.z, e.w};
            uint32_t v[kWords][8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t one = i % 2 ? pairs[i / 2] >> 16 : pairs[i / 2], m = res_mask15(one);
                const Pair row = *reinterpret_cast<const Pair *>(mine + (one & ((1u << kResOutput) - 1u)) * V);
                v[0][i] = *reinterpret_cast<const uint32_t *>(&row) ^ m;
                if (kWords == 2) v[kWords - 1][i] = (reinterpret_cast<const uint32_t *>(&row))[kWords - 1] ^ m;
            }
#pragma unroll
            for (int h = 0; h < kWords; ++h) add8(p[h], v[h]);
            e = next;
        }
        pos = end;
        // sums over the lanes of a part, a plane more each time; in the first step a lane hands one of its two words over and
        // keeps the other
        const bool upper = kWords == 2 && (sub & 1);
        uint32_t s[kPlanes];
#pragma unroll
        for (int i = 0; i < kPlanes; ++i) s[i] = upper ? p[kWords - 1][i] : p[0][i];
#pragma unroll
        for (int step = 0; step < kSteps; ++step) {
            uint32_t carry = 0u;
#pragma unroll
            for (int i = 0; i < kLane + step; ++i) {
                const uint32_t give = step == 0 && kWords == 2 ? (upper ? p[0][i] : p[kWords - 1][i]) : s[i];
                const uint32_t o = __shfl_xor_sync(0xffffffffu, give, kParts << step);
                uint32_t h, l;
                DL_CSA32(h, l, s[i], o, carry);
                s[i] = l;
                carry = h;
            }
            s[kLane + step] = carry;
        }
        // the lanes that hold one word's sums take 4 of its samples each (two lanes per eighth where a word has 16 or 32 lanes):
        // a nibble of each plane -> a bit in each of four bytes
        constexpr int kHolders = kSubs / kWords, kShare = kHolders / 8;   // lanes per word; of one nibble
        const int holder = sub / kWords, first = holder / kShare * 4;
        uint32_t low = 0u, high = 0u;
#pragma unroll
        for (int pl = 0; pl < kPlanes; ++pl) {
            const uint32_t bits = (((s[pl] >> first) & 15u) * 0x00204081u) & 0x01010101u;
            if (pl < 8) low |= bits << pl;
            else high |= bits << (pl - 8);
        }
        int *at = counts + c * kPitch + (part * kWords + (upper ? 1 : 0)) * kResPitch + first;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int count = (int)((low >> (8 * i)) & 255u) | (int)((high >> (8 * i)) & 255u) << 8;
            if (holder % kShare == i % kShare && count) atomicAdd(at + i, count);
        }
    }
    __syncthreads();
    const int64_t s0 = (int64_t)blockIdx.x * (8 * V);
    const int live = (int)min((int64_t)(8 * V), batch - s0) * k;
    const float per_sample = 1.f / (float)k;
    for (int t = tid; t < live; t += T) {
        const int sample = (int)(((float)t + 0.5f) * per_sample);  // t / k: t < 2^21, so the error stays below the half
        out[s0 * k + t] = counts[(t - sample * k) * kPitch + sample / 32 * kResPitch + sample % 32];
    }
}

static size_t res_shared_bytes(int64_t row_slots, int V, int64_t k) {
    return (size_t)row_slots * V + ((size_t)kResPitch * (V / 4) * k + k + 1) * sizeof(int);
}

constexpr size_t kResMaxShared = 227 * 1024;

// Kernels: bytes of a row per block, threads, gates per thread and layer; in order of preference.  Registers decide: 64 (T a power of
// two) hold the outputs of 8 gates of 16 bytes, 72 those of 10 (in 64, 68 bytes per thread went through local memory and took 15 % of
// the shared-memory pipe).
struct ResShape {
    int V, T, R;
};
using ResPlan = ResShape;
constexpr ResShape kResShapes[] = {{16, 256, 8}, {16, 224, 10}, {16, 512, 8}, {16, 448, 10}, {16, 1024, 8}, {16, 896, 10}, {16, 1024, 10},
                                   {8, 256, 12}, {8, 512, 12}, {8, 1024, 12}, {8, 1024, 16}, {4, 256, 16}, {4, 512, 16}, {4, 1024, 16}};

// V: the width for which the busiest SM has least to do.  A block of V bytes costs V bytes of row traffic per gate plus what does
// not depend on V (program words, instructions; about 8 bytes' worth).  slots, gates: what the program says that it needs, or as many
// as the widest layer has rows.  Measured (with the whole layers in the program), us with V = 16 / 8 / 4, 784 -> 4 layers: 8000 wide,
// 100 samples: 19.5 / 18.3 / 18.0, 4000: 20.0 / 19.1 / 17.7, 10000: 20.0 / 24.0 / 28.7, 2^18: 207 / 255 / 399; 10000 wide, 19000: 38 / 48 / 63.
static ResPlan res_plan(const int64_t *n, int layers, int64_t batch, int64_t k, int64_t slots, int64_t gates) {
    ResPlan best = {0, 0, 0};
    if (layers < 1 || layers > kResLayers || batch < 1 || k < 1) return best;
    int64_t most = 0, widest = 0;
    for (int l = 0; l <= layers; ++l) {
        if (n[l] < 1 || n[l] > kResRows) return best;
        most = n[l] > most ? n[l] : most;
        if (l > 0) widest = n[l] > widest ? n[l] : widest;
    }
    if (n[layers] % k != 0) return best;
    if (slots <= 0 || slots > most) slots = most;
    if (gates < 0 || gates > widest) gates = widest;
    const int sms = current_sms();
    int64_t least = 0;
    for (const int V : {16, 8, 4}) {
        const size_t smem = res_shared_bytes(slots + 1, V, k);
        const int64_t blocks = ceil_div(batch, 8 * V);
        if (k > (1 << 14) || smem > kResMaxShared || blocks >= ((int64_t)1 << 31)) continue;
        const int64_t cost = ceil_div(blocks, sms) * (V + 8);
        if (best.V != 0 && cost >= least) continue;
        // as many threads as there are gates for when an SM has one block at a time anyway, else several smaller CTAs
        for (const ResShape &s : kResShapes)
            if (s.V == V && gates <= (int64_t)s.T * s.R &&
                (s.T >= 896 || (blocks > sms && (smem + 1024) * (1024 / s.T) <= kResMaxShared + 1024))) {
                best = {V, s.T, s.R};
                least = cost;
                break;
            }
    }
    return best;
}

template <int WORDS, int T, int R>
static int launch_resident(const void *x, int64_t row_bytes, const uint32_t *prog, const ResidentSizes &sz, const uint32_t *table, int32_t *out,
                           uint8_t *rows_out, int64_t batch, int64_t k, int row_slots, cudaStream_t st) {
    constexpr int V = 4 * WORDS;
    const size_t smem = res_shared_bytes(row_slots, V, k);
    // the most there may be, not this launch's bytes: the limit is the kernel's, and other threads launch it for other networks
    if (cudaFuncSetAttribute(resident_kernel<WORDS, T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResMaxShared) != cudaSuccess)
        return launch_status("dl_eval_network (shared memory opt-in)");
    resident_kernel<WORDS, T, R><<<(unsigned)ceil_div(batch, 8 * V), T, smem, st>>>(
        reinterpret_cast<const uint8_t *>(x), row_bytes, prog, sz, table, out, rows_out, batch, (int)k, (int)(sz.n[sz.layers] / k), row_slots);
    return launch_status("dl_eval_network");
}

}  // namespace dl

using namespace dl;

static int network_applicable(const void *x, const int64_t *n, int layers, int64_t row_bytes, int64_t batch) {
    return x != nullptr && n != nullptr && row_bytes >= 16 && row_bytes % 16 == 0 && aligned_to(x, 16) && batch <= row_bytes * 8;
}

extern "C" DL_API int dl_eval_network_applicable(const void *x, const int64_t *n, int layers, int64_t row_bytes, int64_t batch, int64_t k) {
    if (!network_applicable(x, n, layers, row_bytes, batch)) return 0;
    return res_plan(n, layers, batch, k, 0, -1).V;
}

// Words of a program proper, and of the scratch for building it behind it.
static int64_t program_words(const FoldShape &sh) {
    int64_t words = kResHeader;
    for (int l = 1; l <= sh.layers; ++l) words += res_layer_words(sh.n[l]);
    return (words + res_whole(sh.n[sh.layers]) / 2 + 63) / 64 * 64;
}
static int64_t most_rows(const FoldShape &sh) {
    int64_t most = 0;
    for (int l = 0; l <= sh.layers; ++l) most = sh.n[l] > most ? sh.n[l] : most;
    return most;
}
static bool network_shape(const int64_t *n, int layers, FoldShape *sh) { return fold_shape(n, layers, sh) && most_rows(*sh) <= kResRows; }

extern "C" DL_API int64_t dl_network_program_words(const int64_t *n, int layers) {
    FoldShape sh;
    if (!network_shape(n, layers, &sh)) return 0;
    const int64_t most = most_rows(sh);
    return program_words(sh) + fold_words(sh) + sh.first[layers + 1] + most + (int64_t)layers * kResBuckets +
           (int64_t)(layers + 1) * 2 * kResClasses + most + 2 * kResClasses + kResPad;
}

// Where a program's scratch is, behind the program proper.
static FoldScratch program_scratch(const FoldShape &sh, uint32_t *program, ResBuild *p) {
    const int64_t most = most_rows(sh);
    int32_t *work = reinterpret_cast<int32_t *>(program) + program_words(sh);
    const FoldScratch s = fold_scratch(sh, work);
    *p = {s.header, s.ref, s.in_a, s.in_b, s.use};
    p->slot = work + fold_words(sh);
    p->rank = p->slot + sh.first[sh.layers + 1];
    p->bucket = p->rank + most;
    p->state = p->bucket + (int64_t)sh.layers * kResBuckets;
    p->stack = p->state + (int64_t)(sh.layers + 1) * 2 * kResClasses;
    p->slots = (int)most;
    p->layers = sh.layers;
    p->n0 = sh.n[0];
    return s;
}

extern "C" DL_API int dl_network_fold(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n,
                                      int layers, uint32_t *program, void *stream) {
    DL_REQUIRE(a && b && gate && n && program && aligned_to(program, 16), DL_ERR_INVALID_ARG, "dl_network_fold: null or unaligned pointer");
    DL_REQUIRE(layers >= 1 && layers <= kResLayers, DL_ERR_INVALID_ARG, "dl_network_fold: 1 .. %d layers", kResLayers);
    FoldShape sh;
    DL_REQUIRE(network_shape(n, layers, &sh), DL_ERR_TOO_LARGE, "dl_network_fold: layers of 1 .. %d rows", kResRows);
    for (int l = 0; l < layers; ++l) DL_REQUIRE(a[l] && b[l] && gate[l], DL_ERR_INVALID_ARG, "dl_network_fold: null pointer");
    ResBuild p;
    const FoldScratch s = program_scratch(sh, program, &p);
    if (int e = fold_network(sh, a, b, gate, s, false, as_stream(stream))) return e;
    launch_dependent(true, res_left_kernel, dim3(1), dim3(32), 0, as_stream(stream), p, program);
    return launch_status("dl_network_fold");
}

extern "C" DL_API int dl_network_order(const int64_t *n, int layers, uint32_t *program, void *stream) {
    FoldShape sh;
    DL_REQUIRE(program && aligned_to(program, 16), DL_ERR_INVALID_ARG, "dl_network_order: null or unaligned pointer");
    DL_REQUIRE(network_shape(n, layers, &sh), DL_ERR_TOO_LARGE, "dl_network_order: 1 .. %d layers of 1 .. %d rows", kResLayers, kResRows);
    cudaStream_t st = as_stream(stream);
    ResBuild p;
    const FoldScratch s = program_scratch(sh, program, &p);
    if (cudaMemsetAsync(p.bucket, 0, ((size_t)layers * kResBuckets + (size_t)(layers + 1) * 2 * kResClasses) * sizeof(int32_t), st) != cudaSuccess)
        return launch_status("dl_network_order (clear)");
    auto grid = [](int rows) { return dim3((unsigned)ceil_div(rows, kThreads)); };
    launch_dependent(false, res_inputs_kernel, grid(sh.n[0]), dim3(kThreads), 0, st, p, program);
    uint32_t *level = program + kResHeader;
    for (int l = 1; l <= layers; ++l) {
        launch_dependent(true, res_bucket_kernel, grid(sh.n[l]), dim3(kThreads), 0, st, p, l, sh.first[l], sh.n[l], (const uint32_t *)program);
        launch_dependent(true, res_place_kernel, grid(sh.n[l]), dim3(kThreads), 0, st, p, l, sh.first[l], sh.n[l], program, level);
        level += res_layer_words(sh.n[l]);
    }
    launch_dependent(true, res_outputs_kernel, grid(sh.n[layers]), dim3(kThreads), 0, st, p, sh.n[layers],
                     (const int32_t *)(s.ref + (sh.first[layers] - sh.n[0])), (const uint32_t *)program, reinterpret_cast<uint16_t *>(level));
    return launch_status("dl_network_order");
}

extern "C" DL_API int dl_network_program(const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const int64_t *n,
                                         int layers, uint32_t *program, void *stream) {
    if (int e = dl_network_fold(a, b, gate, n, layers, program, stream)) return e;
    return dl_network_order(n, layers, program, stream);
}

extern "C" DL_API int64_t dl_network_table_words(const int64_t *n, int layers, int64_t k) {
    FoldShape sh;
    ResTable t;
    if (!network_shape(n, layers, &sh) || k < 1 || n[layers] % k != 0) return 0;
    return res_table_words(n[layers], k, &t, nullptr);
}

extern "C" DL_API int dl_network_table(const uint32_t *program, const int64_t *n, int layers, int64_t k, uint32_t *table, void *stream) {
    FoldShape sh;
    ResTable t;
    DL_REQUIRE(program && n && table && aligned_to(table, 16), DL_ERR_INVALID_ARG, "dl_network_table: null or unaligned pointer");
    DL_REQUIRE(network_shape(n, layers, &sh) && k >= 1 && n[layers] % k == 0, DL_ERR_INVALID_ARG, "dl_network_table: bad sizes");
    const int rows = sh.n[layers], rows_per_class = rows / (int)k;
    res_table_words(rows, k, &t, table);
    cudaStream_t st = as_stream(stream);
    if (cudaMemsetAsync(t.ones, 0, (size_t)k * (1 + kResClasses) * sizeof(int32_t), st) != cudaSuccess) return launch_status("dl_network_table (clear)");
    const uint32_t *level = program + kResHeader;
    for (int l = 1; l <= layers; ++l) level += res_layer_words(sh.n[l]);
    const uint16_t *outputs = reinterpret_cast<const uint16_t *>(level);
    const int64_t fill = t.room / 2 > rows ? t.room / 2 : rows;
    launch_dependent(false, res_table_count_kernel, dim3((unsigned)ceil_div(fill, kThreads)), dim3(kThreads), 0, st, t, rows, rows_per_class, program, outputs);
    launch_dependent(true, res_table_start_kernel, dim3(1), dim3(1024), 0, st, t, (int)k, rows_per_class, program);
    launch_dependent(true, res_table_place_kernel, dim3((unsigned)ceil_div(rows, kThreads)), dim3(kThreads), 0, st, t, rows, rows_per_class, program, outputs);
    return launch_status("dl_network_table");
}

extern "C" DL_API int dl_eval_network_sized(const void *x, const uint32_t *program, const int64_t *n, int layers, int64_t slots, int64_t gates,
                                            const uint32_t *table, int32_t *out, void *rows_out, int64_t row_bytes, int64_t batch, int64_t k,
                                            void *stream) {
    DL_REQUIRE(program && (out != nullptr) != (rows_out != nullptr) && aligned_to(rows_out, 16) && aligned_to(program, 16) && aligned_to(table, 16) &&
                   network_applicable(x, n, layers, row_bytes, batch), DL_ERR_INVALID_ARG, "dl_eval_network: bad pointer or sizes");
    const ResPlan plan = res_plan(n, layers, batch, k, slots, gates);
    DL_REQUIRE(plan.V != 0, DL_ERR_INVALID_ARG, "dl_eval_network: sizes outside the kernel's range (ask dl_eval_network_applicable first)");
    ResidentSizes sz = {};
    sz.layers = layers;
    int row_slots = 0;
    for (int l = 0; l <= layers; ++l) {
        sz.n[l] = (int)n[l];
        row_slots = sz.n[l] > row_slots ? sz.n[l] : row_slots;
    }
    row_slots = (slots > 0 && slots < row_slots ? (int)slots : row_slots) + 1;  // and a row of zeros
    cudaStream_t st = as_stream(stream);
#define DL_RES(WW, TT, RR)          \
    if (plan.V == 4 * WW && plan.T == TT && plan.R == RR) return launch_resident<WW, TT, RR>(x, row_bytes, program, sz, table, out, reinterpret_cast<uint8_t *>(rows_out), batch, k, row_slots, st)
    DL_RES(4, 256, 8);
    DL_RES(4, 224, 10);
    DL_RES(4, 512, 8);
    DL_RES(4, 448, 10);
    DL_RES(4, 1024, 8);
    DL_RES(4, 896, 10);
    DL_RES(4, 1024, 10);
    DL_RES(2, 256, 12);
    DL_RES(2, 512, 12);
    DL_RES(2, 1024, 12);
    DL_RES(2, 1024, 16);
    DL_RES(1, 256, 16);
    DL_RES(1, 512, 16);
    DL_RES(1, 1024, 16);
#undef DL_RES
    return fail(DL_ERR_INVALID_ARG, "dl_eval_network: no kernel for rows of %d bytes", plan.V);
}

extern "C" DL_API int dl_eval_network(const void *x, const uint32_t *program, const int64_t *n, int layers, int32_t *out, void *rows_out,
                                      int64_t row_bytes, int64_t batch, int64_t k, void *stream) {
    return dl_eval_network_sized(x, program, n, layers, 0, -1, nullptr, out, rows_out, row_bytes, batch, k, stream);
}
