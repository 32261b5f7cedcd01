// What is left of a packed network once its gates are fixed: layout of the scratch that fold.cu fills.
#pragma once

#include "common.cuh"

namespace dl {

constexpr int kFoldLayers = 32;   // layers per network
// Words in front: gates that are left, by layer (1 .. layers), and behind kFoldDead of them how many values the layer reads last.
constexpr int kFoldHeader = 128, kFoldDead = 64;

// A VALUE is a row of the input (0 .. n[0] - 1) or the output of a neuron (numbered on, layer by layer).  A neuron's output is
// described by a REFERENCE: value << 1 | inverted, or one of two constants; ref ^ 1 is the inverse of any of them.
constexpr int kRefFalse = -2;
__device__ __forceinline__ bool ref_is_constant(int ref) { return ref < 0; }

constexpr int kFoldValueBits = 27;  // of a value; the gate of a neuron lies above the value of its second input

struct FoldShape {
    int layers;
    int n[kFoldLayers + 1];      // rows of the input and of every layer
    int first[kFoldLayers + 2];  // first value of the input (0) and of every layer; behind the last one, their number
};

// Words of the scratch.  ref: by neuron (value - n[0]) what its output is.  in_a, in_b: the values that a gate reads, the gate
// above in_b's (0: the neuron is no gate of its own).  use: by value, the last layer that reads it, 0 when none does.  row: by
// value, where it stands in the list of gates that are left.
struct FoldScratch {
    int32_t *header, *ref, *in_a, *in_b, *use, *row;
};
static inline int64_t fold_words(const FoldShape &sh) {
    const int64_t neurons = sh.first[sh.layers + 1] - sh.n[0];
    return kFoldHeader + 3 * neurons + 2 * (int64_t)sh.first[sh.layers + 1];
}
static inline FoldScratch fold_scratch(const FoldShape &sh, int32_t *work) {
    const int64_t values = sh.first[sh.layers + 1], neurons = values - sh.n[0];
    FoldScratch s;
    s.header = work;
    s.use = work + kFoldHeader;  // cleared together with the header
    s.ref = s.use + values;
    s.in_a = s.ref + neurons;
    s.in_b = s.in_a + neurons;
    s.row = s.in_b + neurons;
    return s;
}

// false: the sizes are outside the range
bool fold_shape(const int64_t *n, int layers, FoldShape *sh);
// Fills the scratch (one launch per layer, there and back).  tail_rows: the last layer's gates are left to the caller -- their
// inputs count as read, they themselves are no part of the list -- else they are gates like all others.
int fold_network(const FoldShape &sh, const int64_t *const *a, const int64_t *const *b, const uint8_t *const *gate, const FoldScratch &s,
                 bool tail_rows, cudaStream_t st);

}  // namespace dl
