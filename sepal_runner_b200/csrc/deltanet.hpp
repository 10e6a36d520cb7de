// The core of the Gated DeltaNet mixer between its projections, with the reference's arithmetic
// (runner/include/sepal/ref/deltanet.hpp:33-330; docs/RUNNER.md:350-361): a depthwise causal convolution over the in-projection's
// `mixed` band (K taps, the LAST tap on the current token, continued from the request's previous K - 1 inputs), SiLU, the split into
// q, k (key heads) and v (value heads), L2 normalisation of q and k per head (x / sqrt(sum x^2 + 1e-6)), value head h reading key head
// h / (value heads / key heads); per token and value head the gated delta rule on a float32 state S [dk, dv]:
//     S <- decay * S;   S <- S + k (x) beta (v - k . S);   read = S^T q / sqrt(dk)
// with decay = exp(-exp(A_log) softplus(a + dt_bias)) and beta = sigmoid(b) (a token reads the state after its own update); then the
// RMSNorm of each head's read scaled by the norm weight itself (not 1 + w) and gated by silu(z), rounded to binary16 for out_proj.
//
// State. A request owns a slot: its recurrent state [value heads, dk, dv] float32 and the last K - 1 rows of `mixed`. A call holds runs
// of consecutive tokens of different requests; a run continues its slot's state and leaves it updated, so a request cut into several
// calls gives what it gives in one. The scan takes a run in chunks of sixteen tokens (warps that each hold 64 rows by 16 columns of the
// float32 state in registers; the chunk's matrix products on the tensor cores with TF32 operands).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "attention.hpp"
#include "context.hpp"

namespace sepal::b200 {

struct DeltaNetShape {
    std::uint32_t key_heads = 0, value_heads = 0;  // value_heads a multiple of key_heads
    std::uint32_t head_dim = 128;                  // dk = dv = 128
    std::uint32_t conv_kernel = 4;
    float eps = 1.0e-6f;                           // of the gated norm
    std::uint32_t key_dim() const { return key_heads * head_dim; }
    std::uint32_t value_dim() const { return value_heads * head_dim; }
    std::uint32_t conv_dim() const { return 2 * key_dim() + value_dim(); }
};

struct DeltaNetRow {
    std::uint32_t q_begin;  // the run's first token in the flat list of the call
    std::uint32_t length;
    std::uint32_t slot;     // the request's state
    std::uint32_t fresh;    // 1: the request starts here: its state and conv tail count as zero whatever the slot holds
};

/// The per-layer weights of the core (device, float32): conv [conv_dim, K]; a_log, dt_bias [value_heads]; norm [head_dim].
struct DeltaNetWeights {
    const float* conv = nullptr;
    const float* a_log = nullptr;
    const float* dt_bias = nullptr;
    const float* norm = nullptr;
};

/// Scratch of one call (device, float32, 16-byte aligned), sized for the call's tokens N: kq [key_heads, N, 264] (a token's k, q and 8
/// floats of padding per key head); v, reads [N, value_dim]; coef [value_heads, N, 56] (the chunk coefficients). The interface asks for
/// 2 N value_heads more, which nothing uses, so that callers' sizes stay what they are.
struct DeltaNetScratch {
    float* kq = nullptr;
    float* v = nullptr;
    float* reads = nullptr;
    float* coef = nullptr;
};

/// Floats of scratch a call of `tokens` tokens needs, and the scratch carved out of one such allocation.
inline std::size_t deltanet_scratch_floats(const DeltaNetShape& s, std::size_t tokens) {
    return tokens * (264 * static_cast<std::size_t>(s.key_heads) + 2 * s.value_dim() + 58 * static_cast<std::size_t>(s.value_heads));
}
inline DeltaNetScratch deltanet_scratch(float* base, const DeltaNetShape& s, std::size_t tokens) {
    DeltaNetScratch sc;
    sc.kq = base;
    sc.v = sc.kq + tokens * s.key_heads * 264;
    sc.reads = sc.v + tokens * s.value_dim();
    sc.coef = sc.reads + tokens * s.value_dim();
    return sc;
}

/// The launches of a layer (prepare with the chunk coefficients, scan with the tails, gated norm). mixed [N, conv_dim], z [N, value_dim], b and a [N, value_heads] are bands of the in-projection's output;
/// states float32 [slots, value_heads, head_dim, head_dim] and tails float32 [slots, K - 1, conv_dim], both updated in place; out
/// binary16 [N, value_dim] with row stride out_stride.
/// `rows` is a HOST array sorted by q_begin.
void launch_deltanet(Context& ctx, const DeltaNetShape& shape, const DeltaNetRow* rows, std::size_t n_rows, Band mixed, Band z, Band b, Band a,
                     const DeltaNetWeights& weights, const DeltaNetScratch& scratch, float* states, float* tails, std::size_t slots,
                     void* out, std::size_t out_stride, cudaStream_t stream);

bool deltanet_supports(const DeltaNetShape& shape);

}  // namespace sepal::b200
