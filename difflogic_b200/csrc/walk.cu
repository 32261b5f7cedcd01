// Training kernels that WALK a layer's connection graph: forward, and backward_w + backward_x in one pass.
//
// Take the layer's inputs as nodes and its neurons as edges (a neuron joins its two input rows).  A walk along edges
// meets the neurons in an order in which each neuron shares an input row with the one before it, so a row that was
// loaded for one neuron is still in registers for the next: one row load per neuron instead of two.  The order in which
// neurons are processed is free -- every neuron writes its own output row -- so the walk is computed once per layer
// (dl_build_walk, on the host) and the kernels follow it.
//
// In a square layer with random connections every input feeds exactly two neurons: the graph is a set of closed
// walks, every node lies on one of them once, and both terms of its input gradient come from two neighbouring steps.
// The backward kernel then carries the first term in a register to the next step and stores the finished row: per neuron
// it reads one row of x and one of grad_y and writes one of grad_x, and the four batch sums of the weight gradient come
// from the same registers.  The two gather kernels of train.cu (backward_w: three rows read; backward_x: four read, one
// written) move eight rows for the same result.
//
// Bound by memory: measured per launch in a captured chain, 64000 x 64000 at batch 1024: forward 118 -> 89 us (81 us for its
// bytes at the measured copy bandwidth), both gradients with Adam 316 (199 + 116 one after the other) -> 147 us (124);
// 128000 x 128000 at batch 256: 66 -> 45 us and 168 -> 79 us (68).
//
// A walk is cut into chunks; a chunk's warps handle up to 128 batch columns each.  What a chunk needs from the step
// before it (the carried gradient term) it recomputes from that step's operands: two extra row loads per chunk.
#include <stdlib.h>

#include <new>
#include <type_traits>
#include <vector>

#include "adam_math.cuh"
#include "common.cuh"
#include "gates.cuh"
#include "tma.cuh"

namespace dl {

constexpr int kWalkSteps = 8;          // steps that a lane group takes between two reductions, all their loads in flight
constexpr int kWalkWarps = kThreads / 32;

// Entry of a walk, two int32:
//   x = node << 1 | store     the input row this step stands on; store: its gradient is complete here and is stored
//   y = neuron << 2 | flip << 1 | emit, or -1 when no neuron leads on (the end of an open walk, a node nobody reads)
//                             flip: the row stood on is the neuron's SECOND input; emit: the neuron's outputs belong to
//                             this entry (an entry in front of a closed walk repeats its last one without store and emit)
// The neuron leads to the node of the next entry.

// Four values of a row per lane.  VEC: four adjacent ones (16-byte loads); else four that lie G lanes apart, so that
// rows of any length and alignment are read in whole sectors.
template <int G, bool VEC>
struct RowIo {
    int64_t col;    // first column of this lane
    int live;       // bit i: component i lies inside the row
    __device__ __forceinline__ RowIo(int64_t col0, int lane, int64_t batch) {
        if (VEC) {
            col = col0 + lane * 4;
            live = col < batch ? 15 : 0;
        } else {
            col = col0 + lane;
            live = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) live |= (col + i * G < batch ? 1 : 0) << i;
        }
    }
    __device__ __forceinline__ float4 load(const float *__restrict__ m, int64_t row, int64_t batch) const {
        const float *p = m + row * batch + col;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (live) v = __ldg(reinterpret_cast<const float4 *>(p));
        } else {
            if (live & 1) v.x = __ldg(p);
            if (live & 2) v.y = __ldg(p + G);
            if (live & 4) v.z = __ldg(p + 2 * G);
            if (live & 8) v.w = __ldg(p + 3 * G);
        }
        return v;
    }
    __device__ __forceinline__ void store(float *__restrict__ m, int64_t row, int64_t batch, const float4 &v) const {
        float *p = m + row * batch + col;
        if (VEC) {
            if (live) *reinterpret_cast<float4 *>(p) = v;
        } else {
            if (live & 1) p[0] = v.x;
            if (live & 2) p[G] = v.y;
            if (live & 4) p[2 * G] = v.z;
            if (live & 8) p[3 * G] = v.w;
        }
    }
};

// Selected value by value: a branch here keeps the steps' loads apart (784 -> 5 x 16000, 1000 samples: 139 us
// against 136; 134 without either, at the price of other bits than the gather kernel's).
__device__ __forceinline__ float4 pick4(bool first, const float4 &a, const float4 &b) {
    float4 r;
    asm("{.reg .pred p; setp.ne.s32 p, %12, 0; selp.f32 %0, %4, %8, p; selp.f32 %1, %5, %9, p; selp.f32 %2, %6, %10, p; selp.f32 %3, %7, %11, p;}"
        : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
        : "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "r"((int)first));
    return r;
}

// ---------------------------------------------------------------------------------------------
// forward along the walk: y[j] = mix(x[a_j], x[b_j]), the coefficients of the CTA's neurons computed by four lanes each
// while the first rows are in flight
// ---------------------------------------------------------------------------------------------
template <int G, bool VEC>
__global__ void __launch_bounds__(kThreads, 4)
walk_forward_kernel(const float *__restrict__ x, const float *__restrict__ w, int w_mode, float *__restrict__ y,
                    float4 *__restrict__ coef_out, const int2 *__restrict__ walk, int entries, int64_t batch, int wc, int ncb) {
    constexpr int N = kWalkWarps * (32 / G) * kWalkSteps;  // entries per CTA
    __shared__ int s_node[N + 1], s_edge[N + 1];
    __shared__ float4 s_coef[N];

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % G;
    const int first = blockIdx.x * N;
    for (int t = tid; t <= N; t += kThreads) {
        const int2 e = first + t < entries ? __ldg(walk + first + t) : make_int2(-1, -1);
        s_node[t] = e.x >> 1;
        s_edge[t] = e.y;
        if (t < N && e.y >= 0) prefetch_l2(w + (int64_t)(e.y >> 2) * 16);
    }
    __syncthreads();
    grid_dependency_wait();
    grid_dependents_launch();

    const int wcol = warp % wc;
    const int p = ((warp / wc) * (32 / G) + (tid % 32) / G) * (kWalkSteps * wc);  // this chunk's first entry
    float4 xin = make_float4(0.f, 0.f, 0.f, 0.f), xn[kWalkSteps];
    auto fetch = [&](const RowIo<G, VEC> &io, int q) {
#pragma unroll
        for (int i = 0; i < kWalkSteps; ++i) {
            xn[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            const int node = s_node[q + i + 1];
            if (node >= 0) xn[i] = io.load(x, node, batch);
        }
    };
    auto begin = [&](const RowIo<G, VEC> &io) {
        const int node = s_node[p];
        xin = node >= 0 ? io.load(x, node, batch) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    int cb = wcol;
    if (cb < ncb) {
        const RowIo<G, VEC> io((int64_t)cb * (4 * G), lane, batch);
        begin(io);
        fetch(io, p);
    }
    for (int t = tid; t < N * 4; t += kThreads) {
        const int nl = t >> 2, q = t & 3, e = s_edge[nl];
        const bool live = e >= 0 && (e & 1);
        const int64_t j = live ? e >> 2 : 0;
        const float4 c = quad_coef(w + j * 16 + q * 4, live, q, w_mode);
        if (q == 0 && live) {
            s_coef[nl] = c;
            if (coef_out != nullptr) coef_out[j] = c;
        }
    }
    __syncthreads();
    bool fetched = true;
    for (; cb < ncb; cb += wc) {
        const RowIo<G, VEC> io((int64_t)cb * (4 * G), lane, batch);
        if (!fetched) begin(io);
        for (int sb = 0; sb < wc; ++sb) {
            const int q = p + sb * kWalkSteps;
            if (!fetched) fetch(io, q);
            fetched = false;
#pragma unroll
            for (int i = 0; i < kWalkSteps; ++i) {
                const int e = s_edge[q + i];
                // the neuron's inputs in their own order: the bits are those of the gather kernel
                if (e >= 0 && (e & 1)) io.store(y, e >> 2, batch, mixv(s_coef[q + i], pick4(e & 2, xn[i], xin), pick4(e & 2, xin, xn[i])));
                xin = xn[i];
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// backward along the walk
// ---------------------------------------------------------------------------------------------
// Four columns as two pairs: the packed instructions round each half as the scalar ones do and take half the issue slots, which is
// what the backward kernels run out of first (64000 x 1024, weight gradients alone: 56 us of issue in 84 us).
struct Quad {
    uint64_t lo, hi;
    __device__ __forceinline__ Quad() {}
    __device__ __forceinline__ Quad(uint64_t l, uint64_t h) : lo(l), hi(h) {}
    __device__ __forceinline__ Quad(const float4 &v) {
        asm("mov.b64 %0, {%1, %2};" : "=l"(lo) : "f"(v.x), "f"(v.y));
        asm("mov.b64 %0, {%1, %2};" : "=l"(hi) : "f"(v.z), "f"(v.w));
    }
    __device__ __forceinline__ float4 values() const {
        float4 v;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(lo));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(hi));
        return v;
    }
};
__device__ __forceinline__ uint64_t both(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float sum_of(uint64_t v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
}
__device__ __forceinline__ Quad mul4(const Quad &a, const Quad &b) { return Quad(mul2(a.lo, b.lo), mul2(a.hi, b.hi)); }
__device__ __forceinline__ float sum4(const Quad &v) { return sum_of(add2(v.lo, v.hi)); }
__device__ __forceinline__ float dot4(const Quad &a, const Quad &b) { return sum_of(fma2(a.hi, b.hi, mul2(a.lo, b.lo))); }
__device__ __forceinline__ Quad scale4(const Quad &a, float s) { return Quad(mul2(a.lo, both(s)), mul2(a.hi, both(s))); }
// (c + cab * p) * g, and the same added to acc
__device__ __forceinline__ Quad term4(float c, float cab, const Quad &p, const Quad &g) {
    return Quad(mul2(fma2(both(cab), p.lo, both(c)), g.lo), mul2(fma2(both(cab), p.hi, both(c)), g.hi));
}
__device__ __forceinline__ Quad term4_add(float c, float cab, const Quad &p, const Quad &g, const Quad &acc) {
    return Quad(fma2(fma2(both(cab), p.lo, both(c)), g.lo, acc.lo), fma2(fma2(both(cab), p.hi, both(c)), g.hi, acc.hi));
}
// The same on plain values, for the register kernel with grad_x: pairs of registers do not fit it.
__device__ __forceinline__ float4 mul4(const float4 &a, const float4 &b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float sum4(const float4 &v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float dot4(const float4 &a, const float4 &b) { return sum4(mul4(a, b)); }
__device__ __forceinline__ float4 scale4(const float4 &a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float4 term4(float c, float cab, const float4 &p, const float4 &g) {
    return make_float4(fmaf(cab, p.x, c) * g.x, fmaf(cab, p.y, c) * g.y, fmaf(cab, p.z, c) * g.z, fmaf(cab, p.w, c) * g.w);
}
__device__ __forceinline__ float4 term4_add(float c, float cab, const float4 &p, const float4 &g, const float4 &acc) {
    return make_float4(fmaf(fmaf(cab, p.x, c), g.x, acc.x), fmaf(fmaf(cab, p.y, c), g.y, acc.y),
                       fmaf(fmaf(cab, p.z, c), g.z, acc.z), fmaf(fmaf(cab, p.w, c), g.w, acc.w));
}
// The four sums of a step: g, a g, b g, a b g.
template <typename Four>
__device__ __forceinline__ void step_sums(const Four &a, const Four &b, const Four &g, float *v) {
    const Four ag = mul4(a, g);
    v[0] = sum4(g);
    v[1] = sum4(ag);
    v[2] = dot4(b, g);
    v[3] = dot4(ag, b);
}

// Sums over the G lanes of a group for 32 values per lane at once: at every step a lane hands half of its values to its
// partner and keeps the other half, so 32 sums cost 31 (G = 32) shuffles instead of 160.  Afterwards v[0 .. 32/G) of lane l
// hold the sums of values l * 32/G ...
template <int G>
__device__ __forceinline__ void transpose_sum(float (&v)[4 * kWalkSteps], int lane) {
    int n = 4 * kWalkSteps;
#pragma unroll
    for (int h = G / 2; h >= 1; h >>= 1) {
        n >>= 1;
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < 2 * kWalkSteps; ++i) {
            if (i < n) {
                const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
            }
        }
    }
}

__device__ __forceinline__ void async_copy16(void *dst_smem, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Optional Adam step in the epilogue, as in train.cu's backward_w: moments of this layer, state = {steps done, ticket}.
struct WalkAdam {
    float *m, *v;
    int *state;
    float lr, beta1, beta2, eps, grad_scale;
};

// A quarter of a neuron's weight gradient (gates 4 q ..) from the four batch sums, softmax backward included; four adjacent lanes.
__device__ __forceinline__ float4 walk_weight_gradient(const float4 &w4, int q, float s0, float sa, float sb, float sab) {
    float pr[4] = {w4.x, w4.y, w4.z, w4.w}, out[4];
    float mx = fmaxf(fmaxf(pr[0], pr[1]), fmaxf(pr[2], pr[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) { pr[i] = expf(pr[i] - mx); s += pr[i]; }
    s = quad_sum(s);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        pr[i] = pr[i] / s;
        out[i] = gate_grad_from_sums(4 * q + i, s0, sa, sb, sab);
        dot += pr[i] * out[i];
    }
    dot = quad_sum(dot);
    return make_float4(pr[0] * (out[0] - dot), pr[1] * (out[1] - dot), pr[2] * (out[2] - dot), pr[3] * (out[3] - dot));
}
// Its Adam step; w4, m4, v4: the weights and moments as they were.
__device__ __forceinline__ void walk_adam(float4 w4, float4 o, float4 m4, float4 v4, float *w, int64_t at, const WalkAdam &adam, float step_size,
                                          float bc2_sqrt) {
    const AdamConsts consts = {1.f - adam.beta1, adam.beta2, 1.f - adam.beta2, step_size, bc2_sqrt, adam.eps};
    o = make_float4(__fmul_rn(o.x, adam.grad_scale), __fmul_rn(o.y, adam.grad_scale), __fmul_rn(o.z, adam.grad_scale),
                    __fmul_rn(o.w, adam.grad_scale));
    adam_update4(w4, o, m4, v4, consts);
    *reinterpret_cast<float4 *>(w) = w4;
    *reinterpret_cast<float4 *>(adam.m + at) = m4;
    *reinterpret_cast<float4 *>(adam.v + at) = v4;
}

// GX: grad_x is wanted and the walk passes every input row once (WalkPlan complete); else only the weight gradients.
template <int G, bool VEC, bool GX>
__global__ void __launch_bounds__(kThreads, 2)
walk_backward_kernel(const float *__restrict__ x, const float *__restrict__ gy, const float4 *__restrict__ coef, const float *w,
                     float *__restrict__ grad_w, float *__restrict__ gx, float scale, const int2 *__restrict__ walk, int entries,
                     int64_t batch, int wc, int ncb, int gy_group, WalkAdam adam) {
    constexpr int N = kWalkWarps * (32 / G) * kWalkSteps;
    constexpr bool kStaged = N * 4 == kThreads;  // one quarter neuron per thread: weights and moments are fetched ahead
    __shared__ int s_node[N + 2], s_edge[N + 2], s_gy[N + 2];  // index t: entry first - 1 + t
    __shared__ float4 s_coef[N + 1];                           // {c of the row stood on, c of the row led to, cab, -}
    __shared__ float s_sum[G == 32 ? kWalkWarps * N * 4 : N * 4];
    __shared__ float4 s_ahead[kStaged ? 3 * kThreads : 1];
    __shared__ float s_step_size, s_bc2_sqrt;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % G;
    const int first = blockIdx.x * N;
    for (int t = tid; t < N + 2; t += kThreads) {
        const int at = first - 1 + t;
        const int2 e = at >= 0 && at < entries ? __ldg(walk + at) : make_int2(-1, -1);
        s_node[t] = e.x;
        s_edge[t] = e.y;
        s_gy[t] = e.y < 0 ? 0 : gy_group == 1 ? e.y >> 2 : (e.y >> 2) / gy_group;
    }
    if (adam.m != nullptr && tid == 0) {
        const float t = (float)(adam.state[0] + 1);
        s_step_size = adam.lr / (1.f - powf(adam.beta1, t));
        s_bc2_sqrt = sqrtf(1.f - powf(adam.beta2, t));
    }
    __syncthreads();
    // the quarter neuron of this thread in the epilogue (kStaged); its moments are touched by this kernel only, one step
    // apart, so they may be fetched before the kernel in front is through
    const int my_edge = kStaged ? s_edge[(tid >> 2) + 1] : -1;
    const bool my_emit = kStaged && my_edge >= 0 && (my_edge & 1);
    const int64_t my_at = (int64_t)(my_edge >> 2) * 16 + (tid & 3) * 4;
    if (my_emit && adam.m != nullptr) {
        async_copy16(s_ahead + kThreads + tid, adam.m + my_at);
        async_copy16(s_ahead + 2 * kThreads + tid, adam.v + my_at);
    }
    grid_dependency_wait();
    grid_dependents_launch();
    if (my_emit) async_copy16(s_ahead + tid, w + my_at);

    const int wcol = warp % wc;
    const int p = ((warp / wc) * (32 / G) + (tid % 32) / G) * (kWalkSteps * wc) + 1;  // this chunk's first entry, as an index t
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xin = zero4, xh = zero4, gh = zero4, dprev = zero4, xn[kWalkSteps], g[kWalkSteps];
    using Four = typename std::conditional<GX, float4, Quad>::type;
    auto begin = [&](const RowIo<G, VEC> &io) {
        xin = s_node[p] >= 0 ? io.load(x, s_node[p] >> 1, batch) : zero4;
        if (GX) {
            xh = gh = zero4;
            if (s_edge[p - 1] >= 0) {
                xh = io.load(x, s_node[p - 1] >> 1, batch);
                gh = io.load(gy, s_gy[p - 1], batch);
            }
        }
    };
    auto fetch = [&](const RowIo<G, VEC> &io, int q) {
#pragma unroll
        for (int i = 0; i < kWalkSteps; ++i) {
            xn[i] = g[i] = zero4;
            if (s_node[q + i + 1] >= 0) xn[i] = io.load(x, s_node[q + i + 1] >> 1, batch);
            if (s_edge[q + i] >= 0) g[i] = io.load(gy, s_gy[q + i], batch);
        }
    };
    float4 my_coef[(N + kThreads) / kThreads];
#pragma unroll
    for (int r = 0; r < (N + kThreads) / kThreads; ++r) {
        const int t = tid + r * kThreads;
        my_coef[r] = zero4;
        if (t <= N && s_edge[t] >= 0) my_coef[r] = __ldg(coef + (s_edge[t] >> 2));
    }
    int cb = wcol;
    if (cb < ncb) {
        const RowIo<G, VEC> io((int64_t)cb * (4 * G), lane, batch);
        begin(io);
        fetch(io, p);
    }
#pragma unroll
    for (int r = 0; r < (N + kThreads) / kThreads; ++r) {
        const int t = tid + r * kThreads;
        if (t <= N) {
            const float4 c = my_coef[r];
            s_coef[t] = (s_edge[t] & 2) ? make_float4(c.z, c.y, c.w, 0.f) : make_float4(c.y, c.z, c.w, 0.f);
        }
    }
    __syncthreads();
    bool fetched = true;
    for (; cb < ncb; cb += wc) {
        const RowIo<G, VEC> io((int64_t)cb * (4 * G), lane, batch);
        if (!fetched) begin(io);
        if (GX) {
            const float4 c = s_coef[p - 1];
            dprev = s_edge[p - 1] >= 0 ? term4(c.y, c.z, xh, gh) : zero4;
        }
        for (int sb = 0; sb < wc; ++sb) {
            const int q = p + sb * kWalkSteps;
            if (!fetched) fetch(io, q);
            fetched = false;
            float v[4 * kWalkSteps];
#pragma unroll
            for (int i = 0; i < kWalkSteps; ++i) {
                const int e = s_edge[q + i];
                if (GX) {
                    const int node = s_node[q + i];
                    float4 acc = dprev;
                    dprev = zero4;
                    if (e >= 0) {
                        const float4 c = s_coef[q + i];
                        acc = term4_add(c.x, c.z, xn[i], g[i], acc);
                        dprev = term4(c.y, c.z, xin, g[i]);
                    }
                    if (node >= 0 && (node & 1)) io.store(gx, node >> 1, batch, scale4(acc, scale));
                }
                step_sums(Four(xin), Four(xn[i]), Four(g[i]), v + 4 * i);
                xin = xn[i];
            }
            transpose_sum<G>(v, lane);
            float *dst = s_sum + (G == 32 ? wcol * N * 4 : 0) + (q - 1) * 4 + lane * (32 / G);
#pragma unroll
            for (int i = 0; i < 32 / G; ++i) dst[i] = cb == wcol ? v[i] : dst[i] + v[i];
        }
    }
    async_copies_wait();
    __syncthreads();

    // ---- epilogue: four lanes per neuron, four gates each: 16 gradients, softmax backward, Adam
    const int parts = wc < ncb ? wc : ncb;
    for (int t = tid; t < N * 4; t += kThreads) {
        const int e = s_edge[(t >> 2) + 1], q = t & 3;
        const bool emit = e >= 0 && (e & 1);
        const int64_t at = (int64_t)(e >> 2) * 16 + q * 4;
        float mine = 0.f;
        for (int r = 0; r < parts; ++r) mine += s_sum[r * N * 4 + t];
        const int base = tid & 28;
        const float s0 = __shfl_sync(0xffffffffu, mine, base), s1 = __shfl_sync(0xffffffffu, mine, base + 1),
                    s2 = __shfl_sync(0xffffffffu, mine, base + 2), sab = __shfl_sync(0xffffffffu, mine, base + 3);
        const float sa = (e & 2) ? s2 : s1, sb = (e & 2) ? s1 : s2;
        float4 w4 = make_float4(0.f, 0.f, 0.f, 0.f), m4 = w4, v4 = w4;
        if (emit) {
            if (kStaged) {
                w4 = s_ahead[tid];
            } else {
                w4 = *reinterpret_cast<const float4 *>(w + at);
            }
            if (adam.m != nullptr) {
                m4 = kStaged ? s_ahead[kThreads + tid] : *reinterpret_cast<const float4 *>(adam.m + at);
                v4 = kStaged ? s_ahead[2 * kThreads + tid] : *reinterpret_cast<const float4 *>(adam.v + at);
            }
        }
        float4 o = walk_weight_gradient(w4, q, s0, sa, sb, sab);
        if (emit) {
            if (grad_w != nullptr) *reinterpret_cast<float4 *>(grad_w + at) = o;
            if (adam.m != nullptr) walk_adam(w4, o, m4, v4, const_cast<float *>(w) + at, at, adam, s_step_size, s_bc2_sqrt);
        }
    }
    if (adam.m != nullptr && tid == 0) {
        // thread 0 of every CTA has read the step count at its start; the last one to get here advances it
        if (atomicAdd(adam.state + 1, 1) == (int)gridDim.x - 1) {
            adam.state[1] = 0;
            adam.state[0] = adam.state[0] + 1;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// backward along the walk, rows staged in shared memory
// ---------------------------------------------------------------------------------------------
// The kernel above holds the rows of eight steps in registers: a warp loads, then computes, then stores, and what is in flight comes
// and goes with it (0.7 of the copy bandwidth at 128000 x 256).  Here a warp follows its part of the walk from end to end and has the
// rows of the next steps copied into shared memory meanwhile: kStagedSlots * 4 steps per warp, 16 warps per SM, 190 KB under way.  Every
// lane copies, with 16-byte asynchronous copies, what it will read itself, so nobody waits for anybody.  (Bulk copies, one per row,
// are issued lane by lane and took half of all instructions: 9216 -> 128000 x 256 58 us.)
// As many warps as there are column blocks share a part.  Each leaves the sums of eight steps in shared memory; after as many turns as
// there are warps (at most eight) they meet, and each takes one turn's eight neurons to the end: softmax backward, Adam.  (One warp
// after each turn, in rotation: the others waited for it at the next turn, 64000 x 1024 159 us.)
// What a part needs from the step before it is loaded once per part, not once per 64 steps.
// Bound by memory where grad_x is wanted (0.84 to 0.86 of the copy bandwidth: 512-byte pieces of rows in random order, read and
// written); for weight gradients alone by instructions as much (40 % of the issue slots, loads in between).
constexpr int kStagedWarps = 16, kStagedThreads = 32 * kStagedWarps;
constexpr int kStagedSteps = 4, kStagedSlots = 3;  // steps per slot, slots per warp
constexpr int kStagedSlot = kStagedSteps * (2 * 512 + 16) + 64;  // a slot: rows of x, rows of grad_y, coefficients; whole 128 bytes
constexpr int kStagedRing = 32;                    // entries of the walk that a warp has at hand, and where their rows are
constexpr int kStagedTurns = 8;                    // at most: reductions that wait for one epilogue
constexpr int kStagedWarpBytes = kStagedSlots * kStagedSlot + kStagedRing * 16 + kStagedTurns * 32 * 4;
static_assert(kStagedSlot % 128 == 0 && kStagedWarpBytes % 16 == 0, "layout of a warp's shared memory");
static_assert(kStagedWarps * kStagedWarpBytes + 1024 <= 227 * 1024, "shared memory of a CTA");

__device__ __forceinline__ void async_row16(void *dst_smem, const void *src, bool there) {  // zeros where there is nothing
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(smem_addr(dst_smem)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// Sums over the lanes for 32 values per lane, by way of 4 KB of shared memory: lane l gets that of value l % 8 * 4 + l / 8 % 2 * 2 + l / 16.
// The 16-byte pieces of a lane's row are swapped about so that neither writes nor reads meet in a bank.  48 instructions, where
// handing halves on from lane to lane (transpose_sum) takes 31 shuffles and 62 selections.
__device__ __forceinline__ float lane_sums(const float (&v)[4 * kWalkSteps], float4 *room, int lane) {
#pragma unroll
    for (int c = 0; c < 8; ++c) room[lane * 8 + (c ^ (lane & 7))] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    __syncwarp();
    const float4 *from = room + lane / 8 * 64;  // eight lanes' rows, of each the piece with values lane % 8 * 4 ..
    Quad sum(from[lane & 7]);
#pragma unroll
    for (int r = 1; r < 8; ++r) {
        const Quad q(from[r * 8 + ((lane & 7) ^ r)]);
        sum = Quad(add2(sum.lo, q.lo), add2(sum.hi, q.hi));
    }
    const float4 s = sum.values();
    const bool up8 = lane & 8, up16 = lane & 16;
    const float a = (up8 ? s.z : s.x) + __shfl_xor_sync(0xffffffffu, up8 ? s.x : s.z, 8);
    const float b = (up8 ? s.w : s.y) + __shfl_xor_sync(0xffffffffu, up8 ? s.y : s.w, 8);
    return (up16 ? b : a) + __shfl_xor_sync(0xffffffffu, up16 ? a : b, 16);
}

template <bool GX>
__global__ void __launch_bounds__(kStagedThreads, 1)
walk_backward_staged_kernel(const float *__restrict__ x, const float *__restrict__ gy, const float4 *__restrict__ coef, const float *w,
                            float *__restrict__ grad_w, float *__restrict__ gx, float scale, const int2 *__restrict__ walk, int entries,
                            int64_t batch, int wc, int part, int gy_group, WalkAdam adam) {
    extern __shared__ __align__(128) uint8_t walk_smem[];
    __shared__ float s_step_size, s_bc2_sqrt;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, group = warp / wc, wcol = warp % wc;
    const int warps = blockDim.x / 32;
    uint8_t *slots = walk_smem + (size_t)warp * kStagedSlots * kStagedSlot;
    uint8_t *rest = walk_smem + (size_t)warps * kStagedSlots * kStagedSlot;
    int2 *ring = reinterpret_cast<int2 *>(rest) + warp * kStagedRing;
    // by step: the row that it leads to and its gradient's, in 16-byte units, -1: none
    int *xrow = reinterpret_cast<int *>(rest + warps * kStagedRing * 8) + warp * kStagedRing;
    int *grow = reinterpret_cast<int *>(rest + warps * kStagedRing * 12) + warp * kStagedRing;
    float *sums = reinterpret_cast<float *>(rest + warps * kStagedRing * 16);  // [warp][kStagedTurns][32]
    const int turns = min(wc, kStagedTurns);
    auto meet = [&] {
        if (wc == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(wc * 32) : "memory");
    };
    const int q0 = (int)((int64_t)(blockIdx.x * (warps / wc) + group) * part);
    const int len = q0 < entries ? part : 0;  // steps of this part; what lies behind the walk's end is neither row nor neuron
    auto entry = [&](int t) { return q0 + t < entries ? __ldg(walk + q0 + t) : make_int2(-1, -1); };
    const int row_units = (int)(batch / 4);
    auto keep = [&](int t, const int2 &e) {
        ring[t % kStagedRing] = e;
        xrow[(t + kStagedRing - 1) % kStagedRing] = e.x >= 0 ? (e.x >> 1) * row_units : -1;
        grow[t % kStagedRing] = e.y >= 0 ? (gy_group == 1 ? e.y >> 2 : (e.y >> 2) / gy_group) * row_units : -1;
    };
    int2 ahead = make_int2(-1, -1);
    if (len > 0) {
        keep(lane, entry(lane));
        if (lane < kWalkSteps) ahead = entry(kStagedRing + lane);
    }
    if (adam.m != nullptr && tid == 0) {
        const float t = (float)(adam.state[0] + 1);
        s_step_size = adam.lr / (1.f - powf(adam.beta1, t));
        s_bc2_sqrt = sqrtf(1.f - powf(adam.beta2, t));
    }
    __syncthreads();
    grid_dependency_wait();
    grid_dependents_launch();

    const int64_t col0 = (int64_t)wcol * 128;
    const int cols = (int)min((int64_t)128, batch - col0);
    const bool live = lane * 4 < cols;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 *xcol = reinterpret_cast<const float4 *>(live ? x + col0 + lane * 4 : x);
    const float4 *gcol = reinterpret_cast<const float4 *>(live ? gy + col0 + lane * 4 : gy);
    // rows and coefficients of steps t .. t + 3 into a slot; one group of copies, whatever there is
    auto issue = [&](int t, uint8_t *slot) {
        if (t < len) {
            const int4 xr = *reinterpret_cast<const int4 *>(xrow + t % kStagedRing), gr = *reinterpret_cast<const int4 *>(grow + t % kStagedRing);
            const int to[2 * kStagedSteps] = {xr.x, xr.y, xr.z, xr.w, gr.x, gr.y, gr.z, gr.w};
            uint8_t *mine = slot + lane * 16;
            if ((xr.x | xr.y | xr.z | xr.w | gr.x | gr.y | gr.z | gr.w) >= 0) {
#pragma unroll
                for (int i = 0; i < 2 * kStagedSteps; ++i) async_row16(mine + i * 512, (i < kStagedSteps ? xcol : gcol) + (live ? to[i] : 0), live);
            } else {
#pragma unroll
                for (int i = 0; i < 2 * kStagedSteps; ++i)
                    async_row16(mine + i * 512, (i < kStagedSteps ? xcol : gcol) + (live ? max(to[i], 0) : 0), live && to[i] >= 0);
            }
            if (lane < kStagedSteps) {
                const int edge = ring[(t + lane) % kStagedRing].y;
                async_row16(slot + 2 * kStagedSteps * 512 + lane * 16, coef + max(edge >> 2, 0), edge >= 0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int k = 0; k < kStagedSlots; ++k) issue(k * kStagedSteps, slots + k * kStagedSlot);

    // the row stood on, and what the step in front of this part adds to its gradient
    Quad xin(zero4), dprev(zero4);
    if (len > 0 && live) {
        const int node = ring[0].x;
        if (node >= 0) xin = Quad(__ldg(reinterpret_cast<const float4 *>(x + (int64_t)(node >> 1) * batch + col0) + lane));
        if (GX && q0 > 0) {
            const int2 before = __ldg(walk + q0 - 1);
            if (before.y >= 0) {
                const float4 xh = __ldg(reinterpret_cast<const float4 *>(x + (int64_t)(before.x >> 1) * batch + col0) + lane);
                const float4 gh = __ldg(reinterpret_cast<const float4 *>(gy + (int64_t)((before.y >> 2) / gy_group) * batch + col0) + lane);
                const float4 c = __ldg(coef + (before.y >> 2));
                dprev = term4((before.y & 2) ? c.y : c.z, c.w, xh, gh);
            }
        }
    }
    // one step; what is not there is zeros
    auto step = [&](const uint8_t *slot, int i, int t, float *v) {
        const Quad xn(reinterpret_cast<const float4 *>(slot + i * 512)[lane]), g(reinterpret_cast<const float4 *>(slot + (kStagedSteps + i) * 512)[lane]);
        if (GX) {
            const int2 here = ring[t % kStagedRing];
            const float4 c = *reinterpret_cast<const float4 *>(slot + 2 * kStagedSteps * 512 + i * 16);
            const Quad acc = term4_add((here.y & 2) ? c.z : c.y, c.w, xn, g, dprev);
            dprev = term4((here.y & 2) ? c.y : c.z, c.w, xin, g);
            if ((here.x & 1) && here.x >= 0 && live)
                reinterpret_cast<float4 *>(gx + (int64_t)(here.x >> 1) * batch + col0)[lane] = scale4(acc, scale).values();
        }
        step_sums(xin, xn, g, v);
        xin = xn;
    };
    int my_edge = -1, turn = 0;
    uint8_t *slot = slots;
    const int sum_place = lane % 8 * 4 + lane / 8 % 2 * 2 + lane / 16;
    for (int t0 = 0; t0 < len; t0 += kWalkSteps, turn = turn + 1 == turns ? 0 : turn + 1) {
        if (t0 > 0) {  // the last eight steps' places are free
            if (lane < kWalkSteps) {
                keep(t0 + kStagedRing - kWalkSteps + lane, ahead);
                ahead = entry(t0 + kStagedRing + lane);
            }
            __syncwarp();
        }
        // this warp's turn, four lanes per neuron; the neurons' weights and moments are on their way during the last turn's steps
        const bool last = turn + 1 == turns || t0 + kWalkSteps >= len, mine_to_do = last && wcol <= turn;
        if (turn == wcol) my_edge = ring[(t0 + (lane >> 2)) % kStagedRing].y;
        const bool emit = mine_to_do && my_edge >= 0 && (my_edge & 1);
        const int64_t at = (int64_t)(my_edge >> 2) * 16 + (lane & 3) * 4;
        float4 w4 = zero4, m4 = zero4, v4 = zero4;
        if (emit) {
            w4 = *reinterpret_cast<const float4 *>(w + at);
            if (adam.m != nullptr) {
                m4 = *reinterpret_cast<const float4 *>(adam.m + at);
                v4 = *reinterpret_cast<const float4 *>(adam.v + at);
            }
        }
        float v[4 * kWalkSteps];
#pragma unroll
        for (int half = 0; half < kWalkSteps / kStagedSteps; ++half) {
            const int t = t0 + half * kStagedSteps;
            asm volatile("cp.async.wait_group %0;" ::"n"(kStagedSlots - 1) : "memory");
            __syncwarp();  // the coefficients come from four lanes
#pragma unroll
            for (int i = 0; i < kStagedSteps; ++i) step(slot, i, t + i, v + 4 * (half * kStagedSteps + i));
            __syncwarp();  // everybody has read the slot
            if (half == kWalkSteps / kStagedSteps - 1) {  // the last slot, before it is filled again, serves to add up over the lanes
                sums[(warp * kStagedTurns + turn) * 32 + sum_place] = lane_sums(v, reinterpret_cast<float4 *>(slot), lane);
                __syncwarp();
            }
            issue(t + kStagedSlots * kStagedSteps, slot);
            slot = slot == slots + (kStagedSlots - 1) * kStagedSlot ? slots : slot + kStagedSlot;
        }
        if (!last) continue;
        meet();  // all sums are there
        float mine = 0.f;
        if (mine_to_do)
            for (int r = 0; r < wc; ++r) mine += sums[((group * wc + r) * kStagedTurns + wcol) * 32 + lane];
        meet();  // and have been read
        if (!mine_to_do) continue;
        const int base = lane & 28, q = lane & 3;
        const float s0 = __shfl_sync(0xffffffffu, mine, base), s1 = __shfl_sync(0xffffffffu, mine, base + 1),
                    s2 = __shfl_sync(0xffffffffu, mine, base + 2), sab = __shfl_sync(0xffffffffu, mine, base + 3);
        float4 o = walk_weight_gradient(w4, q, s0, (my_edge & 2) ? s2 : s1, (my_edge & 2) ? s1 : s2, sab);
        if (emit) {
            if (grad_w != nullptr) *reinterpret_cast<float4 *>(grad_w + at) = o;
            if (adam.m != nullptr) walk_adam(w4, o, m4, v4, const_cast<float *>(w) + at, at, adam, s_step_size, s_bc2_sqrt);
        }
    }
    if (adam.m != nullptr && tid == 0) {
        // thread 0 of every CTA has read the step count at its start; the last one to get here advances it
        if (atomicAdd(adam.state + 1, 1) == (int)gridDim.x - 1) {
            adam.state[1] = 0;
            adam.state[0] = adam.state[0] + 1;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Lanes per row (16 lanes, for the rows of 33 .. 64 columns that layers leave to the gather kernels, are not built), warps side by side
// over the columns, column blocks of 4 * G.  As many warps as there are column blocks
// (a power of two, at most 8) share a chunk unless that leaves more than a quarter of them idle.
struct WalkShape {
    int G, wc, ncb;
};
static WalkShape walk_shape(int64_t batch) {
    const int64_t lanes = ceil_div(batch, 4);
    WalkShape s;
    s.G = lanes <= 8 ? 8 : 32;
    s.ncb = (int)ceil_div(batch, 4 * s.G);
    s.wc = kWalkWarps;
    while (s.wc > 1 && ceil_div(s.ncb, s.wc) * s.wc * 4 > (int64_t)s.ncb * 5) s.wc /= 2;
    return s;
}
// The staged backward kernel: rows of whole 16-byte units (the caller sees to that) and at most 16 column blocks, once a warp has two
// turns of eight steps to go; below, its start (two dependent loads and the first copies) shows.  Measured with Adam, us, register /
// staged kernel (steps per warp): 16000 x 128 (7): 7.9 / 8.1; 16000 x 256 (14): 13.1 / 13.5; 20000 x 172 (17): 20.5 / 16.8; 40000 x 128 (17): 22.8 /
// 19.3; 16000 x 512 (27): 21.9 / 20.5; 64000 x 256 (54): 51.8 / 41.3; 128000 x 68: 58 / 42; 128000 x 256 (108): 95 / 79, gradients by class 85 /
// 67, without grad_x 58 / 48; 32000 x 1152: 91 / 83; 12000 x 2048: 65 / 56; 64000 x 1024 (216): 148 / 147, by class 132 / 103, without grad_x 76 / 66.
static bool walk_staged(int64_t batch, int64_t entries, int64_t rows) {
    const int force = tuning(DL_TUNE_WALK_KERNEL);
    const int64_t ncb = ceil_div(batch, 128);
    if (force == 1 || ncb > kStagedWarps || rows * (batch / 4) > INT32_MAX) return false;
    return force == 2 || entries * ncb >= (int64_t)current_sms() * kStagedWarps * 2 * kWalkSteps;
}
static int64_t walk_ctas(int G, int64_t entries) { return ceil_div(entries, (int64_t)kWalkWarps * (32 / G) * kWalkSteps); }

}  // namespace dl

using namespace dl;

// Walk of a layer's connection graph, built on the host from HOST copies of a and b.  out: int32 pairs (format above), room
// for dl_walk_capacity(n_in, n_out) of them.  *entries: how many were written; *complete: 1 when no input feeds more than two
// neurons, so that the walk passes every input row exactly once (grad_x can be formed along it).
extern "C" DL_API int64_t dl_walk_capacity(int64_t n_in, int64_t n_out) { return n_in + 3 * n_out + 1; }

static int build_walk(const int64_t *a, const int64_t *b, int64_t n_in, int64_t n_out, int32_t *out, int64_t *entries, int *complete) {
    DL_REQUIRE(n_in > 0 && n_out > 0 && a && b && out && entries && complete, DL_ERR_INVALID_ARG, "dl_build_walk: null pointer or size");
    DL_REQUIRE(n_in < ((int64_t)1 << 30) && n_out < ((int64_t)1 << 28), DL_ERR_TOO_LARGE, "dl_build_walk: too many rows");
    struct Ends {
        int32_t a, b;
    };
    struct Reach {
        int32_t next, end;
    };
    std::vector<Ends> ends(n_out);
    std::vector<int32_t> degree(n_in, 0);
    int32_t most = 0;
    for (int64_t j = 0; j < n_out; ++j) {
        DL_REQUIRE(a[j] >= 0 && a[j] < n_in && b[j] >= 0 && b[j] < n_in, DL_ERR_INVALID_ARG,
                   "dl_build_walk: connection of neuron %lld outside [0, %lld)", (long long)j, (long long)n_in);
        ends[j] = {(int32_t)a[j], (int32_t)b[j]};
        const int32_t da = ++degree[a[j]], db = ++degree[b[j]];
        most = da > most ? da : most;
        most = db > most ? db : most;
    }
    int64_t n = 0;
    auto put = [&](int32_t node, int store, int32_t edge) {
        out[2 * n] = node << 1 | store;
        out[2 * n + 1] = edge;
        ++n;
    };
    if (most <= 2) {
        // every input lies on one walk, once: from an input the walk goes on by the neuron that it did not come by
        std::vector<Ends> readers(n_in, {-1, -1});
        for (int32_t j = 0; j < (int32_t)n_out; ++j)
            for (const int32_t v : {ends[j].a, ends[j].b}) (readers[v].a < 0 ? readers[v].a : readers[v].b) = j;
        std::vector<uint8_t> seen(n_in, 0);
        auto follow = [&](int32_t v, bool closed) {
            const int32_t home = v;
            const int64_t head = n;
            if (closed) put(v, 0, -1);  // becomes the repetition of the walk's last step
            int32_t came = -1;          // neuron the walk came by (its first neuron at home)
            do {
                seen[v] = 1;
                const int32_t j = readers[v].a != came ? readers[v].a : readers[v].b;
                const bool loop = j >= 0 && ends[j].a == ends[j].b;
                if (j < 0) break;
                const int flip = ends[j].a != v ? 2 : 0;
                put(v, 1, j << 2 | flip | 1);
                v = flip ? ends[j].a : ends[j].b;
                came = j;
                if (loop) break;
            } while (v != home);
            if (closed) {
                out[2 * head] = out[2 * (n - 1)] & ~1;
                out[2 * head + 1] = out[2 * (n - 1) + 1] & ~1;
                put(v, 0, -1);
            } else {
                put(v, 1, -1);
            }
        };
        for (int32_t i = 0; i < (int32_t)n_in; ++i)  // open walks begin and end at inputs that feed one neuron (or none)
            if (degree[i] < 2 && !seen[i]) follow(i, false);
        for (int32_t i = 0; i < (int32_t)n_in; ++i)
            if (!seen[i]) follow(i, true);
        *entries = n;
        *complete = 1;
        return DL_OK;
    }
    std::vector<Reach> reach(n_in);
    std::vector<int32_t> list(2 * n_out);
    int32_t at = 0;
    for (int64_t i = 0; i < n_in; ++i) {
        reach[i] = {at, at};
        at += degree[i];
    }
    for (int32_t j = 0; j < (int32_t)n_out; ++j) {
        list[reach[ends[j].a].end++] = j;
        list[reach[ends[j].b].end++] = j;
    }
    std::vector<uint8_t> used(n_out, 0);
    auto follow = [&](int32_t v) {  // by unused neurons until there are none
        bool any = false;
        for (;;) {
            Reach &r = reach[v];
            while (r.next < r.end && used[list[r.next]]) ++r.next;
            if (r.next == r.end) break;
            const int32_t j = list[r.next++];
            used[j] = 1;
            const int flip = ends[j].a != v ? 2 : 0;
            put(v, 0, j << 2 | flip | 1);
            v = flip ? ends[j].a : ends[j].b;
            any = true;
        }
        if (any) put(v, 0, -1);
        return any;
    };
    for (int32_t i = 0; i < (int32_t)n_in; ++i)  // open walks begin and end at inputs that feed an odd number of neurons
        if (degree[i] % 2 == 1) follow(i);
    for (int32_t i = 0; i < (int32_t)n_in; ++i)
        while (follow(i)) {
        }
    *entries = n;
    *complete = 0;
    return DL_OK;
}

extern "C" DL_API int dl_build_walk(const int64_t *a, const int64_t *b, int64_t n_in, int64_t n_out, int32_t *out, int64_t *entries,
                                    int *complete) {
    try {
        return build_walk(a, b, n_in, n_out, out, entries, complete);
    } catch (const std::bad_alloc &) {  // callers are C
        return fail(DL_ERR_TOO_LARGE, "dl_build_walk: no host memory for %lld inputs and %lld neurons", (long long)n_in, (long long)n_out);
    }
}

static int walk_checks(const char *who, const int32_t *walk, int64_t entries, int64_t n_in, int64_t n_out, int64_t batch) {
    DL_REQUIRE(walk != nullptr && aligned_to(walk, 8) && entries > 0 && entries <= INT32_MAX, DL_ERR_INVALID_ARG, "%s: bad walk", who);
    DL_REQUIRE(n_in > 0 && n_out > 0 && batch > 0, DL_ERR_INVALID_ARG, "%s: sizes must be positive", who);
    DL_REQUIRE(n_in < ((int64_t)1 << 30) && n_out < ((int64_t)1 << 28) && batch < ((int64_t)1 << 31), DL_ERR_TOO_LARGE, "%s: too large", who);
    return DL_OK;
}

extern "C" DL_API int dl_forward_walk_f32(const float *x, const float *w, int w_mode, float *y, float *coef, const int32_t *walk,
                                          int64_t entries, int64_t n_in, int64_t n_out, int64_t batch, int flags, void *stream) {
    if (int s = walk_checks("dl_forward_walk_f32", walk, entries, n_in, n_out, batch)) return s;
    DL_REQUIRE(w_mode >= DL_W_LOGITS && w_mode <= DL_W_ARGMAX, DL_ERR_INVALID_ARG, "dl_forward_walk_f32: unknown w_mode %d", w_mode);
    DL_REQUIRE(x && w && y, DL_ERR_INVALID_ARG, "dl_forward_walk_f32: null pointer");
    DL_REQUIRE(coef == nullptr || aligned_to(coef, 16), DL_ERR_INVALID_ARG, "dl_forward_walk_f32: coef must be 16-byte aligned");
    const WalkShape s = walk_shape(batch);
    const bool vec = batch % 4 == 0 && aligned_to(x, 16) && aligned_to(y, 16);
    const bool overlap = (flags & DL_LAUNCH_OVERLAP_SETUP) != 0;
    const dim3 grid((unsigned)walk_ctas(s.G, entries));
    const int2 *wk = reinterpret_cast<const int2 *>(walk);
    float4 *c4 = reinterpret_cast<float4 *>(coef);
#define DL_WF(GG)                                                                                                                     \
    case GG:                                                                                                                          \
        if (vec) launch_dependent(overlap, walk_forward_kernel<GG, true>, grid, dim3(kThreads), 0, as_stream(stream), x, w, w_mode, y, c4, \
                                  wk, (int)entries, batch, s.wc, s.ncb);                                                              \
        else launch_dependent(overlap, walk_forward_kernel<GG, false>, grid, dim3(kThreads), 0, as_stream(stream), x, w, w_mode, y, c4,    \
                              wk, (int)entries, batch, s.wc, s.ncb);                                                                  \
        break;
    switch (s.G) { DL_WF(8) DL_WF(32) }
#undef DL_WF
    return launch_status("dl_forward_walk_f32");
}

extern "C" DL_API int dl_backward_walk_f32(const float *x, const float *grad_y, const float *coef, float *w, float *grad_w, float *grad_x,
                                           float grad_scale, const int32_t *walk, int64_t entries, int complete, int64_t n_in,
                                           int64_t n_out, int64_t batch, int64_t rows_per_class, float *exp_avg, float *exp_avg_sq,
                                           float lr, float beta1, float beta2, float eps, float adam_grad_scale, int32_t *state, int flags,
                                           void *stream) {
    const char *who = "dl_backward_walk_f32";
    if (int s = walk_checks(who, walk, entries, n_in, n_out, batch)) return s;
    DL_REQUIRE(rows_per_class >= 1 && rows_per_class <= INT32_MAX && n_out % rows_per_class == 0, DL_ERR_INVALID_ARG,
               "%s: n_out (%lld) is not a multiple of the rows per class (%lld)", who, (long long)n_out, (long long)rows_per_class);
    DL_REQUIRE(x && grad_y && coef && w && (grad_w || exp_avg), DL_ERR_INVALID_ARG, "%s: null pointer", who);
    DL_REQUIRE(grad_x == nullptr || complete, DL_ERR_INVALID_ARG, "%s: grad_x needs a walk that passes every input once", who);
    DL_REQUIRE((exp_avg == nullptr) == (exp_avg_sq == nullptr) && (exp_avg == nullptr || state), DL_ERR_INVALID_ARG, "%s: null pointer", who);
    DL_REQUIRE(aligned_to(coef, 16) && aligned_to(w, 16) && aligned_to(grad_w, 16) && aligned_to(exp_avg, 16) && aligned_to(exp_avg_sq, 16),
               DL_ERR_INVALID_ARG, "%s: coef, w, grad_w and the moments must be 16-byte aligned", who);
    const WalkShape s = walk_shape(batch);
    const bool vec = batch % 4 == 0 && aligned_to(x, 16) && aligned_to(grad_y, 16) && aligned_to(grad_x, 16);
    const bool overlap = (flags & DL_LAUNCH_OVERLAP_SETUP) != 0;
    const dim3 grid((unsigned)walk_ctas(s.G, entries));
    const WalkAdam adam = {exp_avg, exp_avg_sq, reinterpret_cast<int *>(state), lr, beta1, beta2, eps, adam_grad_scale};
    auto launch = [&](auto kernel) {
        launch_dependent(overlap, kernel, grid, dim3(kThreads), 0, as_stream(stream), x, grad_y, reinterpret_cast<const float4 *>(coef), w,
                         grad_w, grad_x, grad_scale, reinterpret_cast<const int2 *>(walk), (int)entries, batch, s.wc, s.ncb,
                         (int)rows_per_class, adam);
    };
    if (vec && walk_staged(batch, entries, n_in > n_out ? n_in : n_out)) {
        const int wc = (int)ceil_div(batch, 128), groups = kStagedWarps / wc, warps = wc * groups;
        const int64_t part = ceil_div(ceil_div(entries, (int64_t)current_sms() * groups), kWalkSteps) * kWalkSteps;
        const size_t smem = (size_t)warps * kStagedWarpBytes;
        auto staged = grad_x != nullptr ? walk_backward_staged_kernel<true> : walk_backward_staged_kernel<false>;
        if (cudaFuncSetAttribute(staged, cudaFuncAttributeMaxDynamicSharedMemorySize, kStagedWarps * kStagedWarpBytes) != cudaSuccess)
            return launch_status("dl_backward_walk_f32 (shared memory opt-in)");
        launch_dependent(overlap, staged, dim3((unsigned)ceil_div(entries, part * groups)), dim3(32 * warps), smem, as_stream(stream), x, grad_y,
                         reinterpret_cast<const float4 *>(coef), w, grad_w, grad_x, grad_scale, reinterpret_cast<const int2 *>(walk), (int)entries,
                         batch, wc, (int)part, (int)rows_per_class, adam);
        return launch_status(who);
    }
#define DL_WB(GG)                                                                                                        \
    case GG:                                                                                                             \
        if (grad_x != nullptr) vec ? launch(walk_backward_kernel<GG, true, true>) : launch(walk_backward_kernel<GG, false, true>); \
        else vec ? launch(walk_backward_kernel<GG, true, false>) : launch(walk_backward_kernel<GG, false, false>);       \
        break;
    switch (s.G) { DL_WB(8) DL_WB(32) }
#undef DL_WB
    return launch_status(who);
}
