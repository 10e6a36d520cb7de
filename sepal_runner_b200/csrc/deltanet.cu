#include "deltanet.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_fp16.h>

#include "ptx.cuh"

namespace sepal::b200 {

void count_launch();

namespace {

constexpr int kDim = 128;  // dk = dv
constexpr int kPair = 2 * kDim + 8;  // floats of a token's (k, q) row: the pitch that keeps the scan's fragment loads free of bank conflicts

constexpr unsigned kInlineRuns = 64;  // runs whose table travels with the kernels' parameters instead of through a copy

struct DeltaParams {
    const DeltaNetRow* far_runs;    // the table in device memory (null: the one below)
    const unsigned* far_chunks;
    DeltaNetRow near_runs[kInlineRuns];
    unsigned near_chunks[kInlineRuns];  // the number of a run's first chunk of sixteen tokens, counted over all runs
    unsigned char near_order[kInlineRuns];  // the runs, longest first
    unsigned n_rows, n_chunks;
    unsigned key_heads, value_heads, taps;
    unsigned value_dim, conv_dim;
    float eps;
    const void* mixed;
    const void* z;
    const void* b;
    const void* a;
    unsigned long long mixed_stride, z_stride, b_stride, a_stride;
    unsigned mixed_half, z_half, b_half, a_half;
    unsigned wide_norm;  // z and out can be taken four values at a time
    const float* conv;
    const float* a_log;
    const float* dt_bias;
    const float* norm;
    float* kq;  // [key_heads, N, 264]: per token the head's k (128), q (128) and 8 floats of padding
    float* v;
    float* reads;  // [N, value_dim]: the scan's output before the gated norm
    float* coef;   // [value_heads, N, 56]: the chunk coefficients of every token
    unsigned n_tokens;
    int* status;
    float* states;
    float* tails;  // [slots, taps - 1, conv_dim]
    __half* out;
    unsigned long long out_stride;
};

__device__ __forceinline__ DeltaNetRow run_at(const DeltaParams& p, unsigned i) { return p.far_runs != nullptr ? p.far_runs[i] : p.near_runs[i]; }
__device__ __forceinline__ unsigned first_chunk(const DeltaParams& p, unsigned i) { return p.far_chunks != nullptr ? p.far_chunks[i] : p.near_chunks[i]; }

__device__ __forceinline__ float value_of(const void* base, unsigned long long index, unsigned half) {
    return half != 0 ? __half2float(static_cast<const __half*>(base)[index]) : static_cast<const float*>(base)[index];
}
// softplus in the reference's form (runner/include/sepal/ref/primitives.hpp:25-40); sigmoid as 1 / (1 + e^-x), which the reference
// writes as exp(-softplus(-x)): the same function, an ulp or two apart in float32, and a third of the instructions (it runs once per
// element of the convolution's output and of the gate). The quotient is rounded to nearest: beta and the activated k enter a recurrence.
__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid(float x) { return __frcp_rn(__fadd_rn(1.0f, expf(-x))); }
__device__ __forceinline__ float silu(float x) { return __fmul_rn(x, sigmoid(x)); }

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float round_tf32(float x) { return __uint_as_float(to_tf32(x)); }

// The last run that begins at or before `token`, and the last whose first chunk is at or before `chunk`.
__device__ __forceinline__ unsigned run_of_token(const DeltaParams& p, unsigned token) {
    unsigned lo = 0, hi = p.n_rows;
    while (hi - lo > 1) {
        const unsigned mid = (lo + hi) / 2;
        if (run_at(p, mid).q_begin <= token) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ unsigned run_of_chunk(const DeltaParams& p, unsigned chunk) {
    unsigned lo = 0, hi = p.n_rows;
    while (hi - lo > 1) {
        const unsigned mid = (lo + hi) / 2;
        if (first_chunk(p, mid) <= chunk) lo = mid; else hi = mid;
    }
    return lo;
}

// The delta rule in chunks of sixteen tokens. With d_t the decay of token t, c_t its correction beta_t (v_t - k_t . d_t S_{t-1}) and
// S_t = d_t S_{t-1} + k_t (x) c_t, unrolling from the state S_0 before the chunk gives, with P(s, t) = d_{s+1} ... d_t and
// gamma_t = d_0 ... d_t (tokens numbered from 0 inside the chunk), y_t = v_t - gamma_t k_t . S_0 and the strictly lower triangular
// L[t][s] = beta_t P(s, t) (k_t . k_s):
//     c      = (I + L)^-1 diag(beta) y                                  =: T1 y
//     read_t = (gamma_t q_t . S_0 + sum_{s<=t} P(s, t) (q_t . k_s) c_s) / sqrt(dk)   = (gamma_t q_t . S_0 + (W y)_t) / sqrt(dk)
//     S_end  = gamma_last S_0 + sum_s P(s, last) k_s (x) c_s            = gamma_last S_0 + K^T (T2 y)
// so a chunk is four small matrix products per block of columns of the state: K S_0 and Q S_0 (16 x 128 by 128 x columns), T2 y and W y
// (16 x 16 by 16 x columns), K^T (T2 y) (128 x 16 by 16 x columns). The matrices T2 = diag(P(s, last)) T1 and W (both 16 x 16, lower
// triangular) and gamma do not involve the state: deltanet_prepare_kernel forms them per chunk and value head. The products run on the
// tensor cores as mma.sync m16n8k8 with TF32 operands (k, q, the state, y and the coefficients rounded to 10 bits of mantissa, as the
// reference's chunked kernels round theirs to binary16, runner/cuda/src/kernels_deltanet_chunked.cu:262-344) and float32 sums; the
// state itself stays in float32 registers, as the accumulators of the last product, which are at the same time the A operand of the
// first two (the rows of an 8-row block are paired with the k slots t and t + 4 as rows 2 t and 2 t + 1, and B is read accordingly).
constexpr int kChunk = 16;
constexpr int kCols = 16;                  // the M of the products: columns of the state
constexpr int kCoef = 56;                  // floats per (token, value head): T2 row at 0, W row at 24, gamma at 48 (224 bytes)
constexpr int kStatusDeltaNet = 24;        // status code: a wait of the scan kernel ran out
constexpr long long kWaitLimit = 1ll << 30;

// d (16 x 8, float32) += a (16 x 8, TF32, row-major fragments) * b (8 x 8, TF32, column-major fragments).
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The input of the convolution for one channel (below: for two pairs of channels) of the token `t` of a run (negative: before the run,
// from the slot's tail, zeros for a fresh request).
__device__ __forceinline__ float input_at(const DeltaParams& p, const DeltaNetRow& run, const float* tail, int t, unsigned channel) {
    if (t >= 0) return value_of(p.mixed, (static_cast<size_t>(run.q_begin) + t) * p.mixed_stride + channel, p.mixed_half);
    return run.fresh != 0 ? 0.0f : tail[static_cast<size_t>(static_cast<int>(p.taps) - 1 + t) * p.conv_dim + channel];
}
__device__ __forceinline__ uint2 input_pairs(const DeltaParams& p, size_t token, unsigned c0, unsigned c1) {
    const __half* src = static_cast<const __half*>(p.mixed) + token * p.mixed_stride;
    return make_uint2(*reinterpret_cast<const unsigned*>(src + c0), *reinterpret_cast<const unsigned*>(src + c1));
}
__device__ __forceinline__ float4 widen(const uint2& raw) {
    const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 input_pairs_before(const DeltaParams& p, const DeltaNetRow& run, const float* tail, int t, unsigned c0, unsigned c1) {
    if (t >= 0) return widen(input_pairs(p, static_cast<size_t>(run.q_begin) + t, c0, c1));
    if (run.fresh != 0) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* src = tail + static_cast<size_t>(3 + t) * p.conv_dim;
    const float2 lo = *reinterpret_cast<const float2*>(src + c0), hi = *reinterpret_cast<const float2*>(src + c1);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// Everything of a chunk that does not involve the state, in one block per chunk and key head: the convolution (taps in ascending order,
// the last on the token itself), SiLU, q and k normalised, their 2 x 256 dot products, and, for every value head of the key head, decay,
// beta, L and the q-k matrix scaled by the decays, (I + L)^-1 by forward substitution (one thread a column), T2 and W. q and k leave the
// block once, rounded to TF32 for the scan's products; the dot products take them as they are (the first token's read is
// (q . k) beta v, one dot product with heavy cancellation).
//
// A warp takes 128 channels (a head of q or k, or 128 channels of v) of eight consecutive tokens, lane l the channels 2 l, 2 l + 1,
// 64 + 2 l and 65 + 2 l: eleven rows are read for eight tokens, all in flight at once, and the taps once. `Pairs`: binary16 inputs and
// four taps at addresses that allow two channels a load; otherwise channel by channel.
//
// What bounds it is instructions (71 % of the issue slots, the shared-memory pipe at 49 %): 4096 tokens of 32 value heads 116 us under the
// profiler (95 with an approximate quotient in the sigmoid and 1 / norm multiplied, which gives other bits). The convolution and the
// coefficients as two launches, with q and k written and read back between them, took 74 + 65 us for five runs of 2500 tokens in all,
// where one launch took 69. Four blocks to an SM hide one another's barriers (4096 tokens: 98 us against 104 with three, then).
constexpr int kHeadsAtOnce = 2;

template <bool Pairs>
__global__ void __launch_bounds__(256, 4) deltanet_prepare_kernel(const __grid_constant__ DeltaParams p) {
    __shared__ __align__(16) float k_sh[kChunk][kDim + 4], q_sh[kChunk][kDim + 4];
    __shared__ __align__(16) float low[kHeadsAtOnce][kChunk][kChunk + 4];
    __shared__ float qk_sh[kHeadsAtOnce][kChunk][kChunk + 1], inv[kHeadsAtOnce][kChunk][kChunk + 1];
    __shared__ float kk_part[4][kChunk][kChunk + 1], qk_part[4][kChunk][kChunk + 1];
    __shared__ float decay_sh[kHeadsAtOnce][kChunk], beta_sh[kHeadsAtOnce][kChunk], carry_sh[kHeadsAtOnce][kChunk], gamma_sh[kHeadsAtOnce][kChunk];
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const unsigned run_index = run_of_chunk(p, blockIdx.x);
    const DeltaNetRow run = run_at(p, run_index);
    const unsigned t0 = (blockIdx.x - first_chunk(p, run_index)) * kChunk;  // the chunk's first token in the run
    const unsigned count = min(static_cast<unsigned>(kChunk), run.length - t0);
    const size_t token0 = static_cast<size_t>(run.q_begin) + t0;
    const unsigned key_head = blockIdx.y, group = p.value_heads / p.key_heads;
    const unsigned warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const float* tail = p.tails + static_cast<size_t>(run.slot) * (p.taps - 1) * p.conv_dim;
    for (unsigned unit = warp; unit < 2 * (2 + group); unit += 8) {
        const unsigned part = unit / 2, first = unit % 2 * 8;  // q, k, then the value heads; tokens 0-7 or 8-15
        if (first >= count) {
            if (part < 2)
                for (unsigned i = 0; i < 8; ++i)
                    for (unsigned d = lane; d < kDim; d += 32) (part == 0 ? q_sh : k_sh)[first + i][d] = 0.0f;
            continue;
        }
        // q comes first in the convolution's channels
        const unsigned slice = part == 0 ? key_head : part == 1 ? p.key_heads + key_head : 2 * p.key_heads + key_head * group + (part - 2);
        const unsigned c0 = slice * kDim + 2 * lane, c1 = c0 + 64;
        const int t = static_cast<int>(t0 + first);
        float4 act[8];
        if (Pairs) {
            const float4* taps = reinterpret_cast<const float4*>(p.conv);
            const float4 w[4] = {taps[c0], taps[c0 + 1], taps[c1], taps[c1 + 1]};
            uint2 raw[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) raw[i] = first + i < count ? input_pairs(p, token0 + first + i, c0, c1) : make_uint2(0u, 0u);
            float4 x0 = input_pairs_before(p, run, tail, t - 3, c0, c1), x1 = input_pairs_before(p, run, tail, t - 2, c0, c1),
                   x2 = input_pairs_before(p, run, tail, t - 1, c0, c1);
            const auto conv = [](const float4& taps4, float a, float b, float c, float d) {
                float acc = __fadd_rn(0.0f, __fmul_rn(taps4.x, a));
                acc = __fadd_rn(acc, __fmul_rn(taps4.y, b));
                acc = __fadd_rn(acc, __fmul_rn(taps4.z, c));
                return silu(__fadd_rn(acc, __fmul_rn(taps4.w, d)));
            };
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x3 = widen(raw[i]);
                act[i] = make_float4(conv(w[0], x0.x, x1.x, x2.x, x3.x), conv(w[1], x0.y, x1.y, x2.y, x3.y), conv(w[2], x0.z, x1.z, x2.z, x3.z), conv(w[3], x0.w, x1.w, x2.w, x3.w));
                x0 = x1, x1 = x2, x2 = x3;
            }
        } else {
            const unsigned channel[4] = {c0, c0 + 1, c1, c1 + 1};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (first + i < count) {
                    for (unsigned j = 0; j < p.taps; ++j) {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            acc[e] = __fadd_rn(acc[e], __fmul_rn(p.conv[static_cast<size_t>(channel[e]) * p.taps + j],
                                                                 input_at(p, run, tail, t + i + static_cast<int>(j) - static_cast<int>(p.taps - 1), channel[e])));
                    }
                }
                act[i] = make_float4(silu(acc[0]), silu(acc[1]), silu(acc[2]), silu(acc[3]));
            }
        }
        if (part >= 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (first + i < count) {
                    float* dst = p.v + (token0 + first + i) * p.value_dim + (slice - 2 * p.key_heads) * kDim + 2 * lane;
                    *reinterpret_cast<float2*>(dst) = make_float2(act[i].x, act[i].y);
                    *reinterpret_cast<float2*>(dst + 64) = make_float2(act[i].z, act[i].w);
                }
            }
            continue;
        }
        float ss[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) ss[i] = __fmaf_rn(act[i].w, act[i].w, __fmaf_rn(act[i].z, act[i].z, __fmaf_rn(act[i].y, act[i].y, __fmaf_rn(act[i].x, act[i].x, 0.0f))));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) ss[i] += __shfl_xor_sync(0xFFFFFFFFu, ss[i], o);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool live = first + i < count;
            const float norm = __fsqrt_rn(__fadd_rn(ss[i], 1.0e-6f));  // (a division, not a multiplication by 1 / norm, which would round twice)
            const float n[4] = {live ? __fdiv_rn(act[i].x, norm) : 0.0f, live ? __fdiv_rn(act[i].y, norm) : 0.0f, live ? __fdiv_rn(act[i].z, norm) : 0.0f,
                                live ? __fdiv_rn(act[i].w, norm) : 0.0f};
            float* row = (part == 0 ? q_sh : k_sh)[first + i] + 2 * lane;
            *reinterpret_cast<float2*>(row) = make_float2(n[0], n[1]);
            *reinterpret_cast<float2*>(row + 64) = make_float2(n[2], n[3]);
            if (live) {
                float* dst = p.kq + (static_cast<size_t>(key_head) * p.n_tokens + token0 + first + i) * kPair + (part == 0 ? kDim : 0) + 2 * lane;
                *reinterpret_cast<float2*>(dst) = make_float2(round_tf32(n[0]), round_tf32(n[1]));
                *reinterpret_cast<float2*>(dst + 64) = make_float2(round_tf32(n[2]), round_tf32(n[3]));
            }
        }
    }
    __syncthreads();
    // The 2 x 256 dot products: a thread takes tokens (a, a + 8) x (b, b + 8) over a quarter of the 128 dimensions, four dimensions a
    // load (six loads for 32 multiply-adds), and the four quarters meet in shared memory.
    {
        const unsigned quarter = threadIdx.x / 64, pa = threadIdx.x % 8, pb = threadIdx.x / 8 % 8;
        float kk2[2][2] = {}, qk2[2][2] = {};
#pragma unroll 4
        for (unsigned d = 32 * quarter; d < 32 * quarter + 32; d += 4) {
            float4 ka[2], qa[2], kb[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                ka[i] = *reinterpret_cast<const float4*>(&k_sh[pa + 8 * i][d]);
                qa[i] = *reinterpret_cast<const float4*>(&q_sh[pa + 8 * i][d]);
                kb[i] = *reinterpret_cast<const float4*>(&k_sh[pb + 8 * i][d]);
            }
            const auto dot4 = [](const float4& x, const float4& y, float sum) { return __fmaf_rn(x.w, y.w, __fmaf_rn(x.z, y.z, __fmaf_rn(x.y, y.y, __fmaf_rn(x.x, y.x, sum)))); };
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    kk2[i][j] = dot4(ka[i], kb[j], kk2[i][j]);
                    qk2[i][j] = dot4(qa[i], kb[j], qk2[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                kk_part[quarter][pa + 8 * i][pb + 8 * j] = kk2[i][j];
                qk_part[quarter][pa + 8 * i][pb + 8 * j] = qk2[i][j];
            }
        }
    }
    const unsigned s = threadIdx.x / kChunk, t = threadIdx.x % kChunk;  // (row, column) = (s, t) of the 16 x 16 matrices from here on
    float kk = 0.0f, qk = 0.0f;
    for (unsigned h0 = 0; h0 < group; h0 += kHeadsAtOnce) {
        const unsigned heads = min(static_cast<unsigned>(kHeadsAtOnce), group - h0);
        const unsigned first_head = key_head * group + h0;
        if (s < heads) {  // decay and beta of token t of head s
            float decay = 1.0f, beta = 0.0f;
            if (t < count) {
                const unsigned h = first_head + s;
                const float a = value_of(p.a, (token0 + t) * p.a_stride + h, p.a_half), b = value_of(p.b, (token0 + t) * p.b_stride + h, p.b_half);
                decay = expf(-expf(p.a_log[h]) * softplus(a + p.dt_bias[h]));
                beta = sigmoid(b);
            }
            decay_sh[s][t] = decay;
            beta_sh[s][t] = beta;
        }
        __syncthreads();  // (also: the dot products' parts are in place, and the heads before these are done with the shared arrays)
        if (h0 == 0) {
            kk = (kk_part[0][t][s] + kk_part[1][t][s]) + (kk_part[2][t][s] + kk_part[3][t][s]);
            qk = (qk_part[0][t][s] + qk_part[1][t][s]) + (qk_part[2][t][s] + qk_part[3][t][s]);
        }
        for (unsigned h = 0; h < heads; ++h) {
            float product = t > s ? decay_sh[h][t] : 1.0f;  // P(s, t): a running product over the sixteen lanes of row s
#pragma unroll
            for (int o = 1; o < kChunk; o *= 2) {
                const float before = __shfl_up_sync(0xFFFFFFFFu, product, o, kChunk);
                if (t >= static_cast<unsigned>(o)) product = __fmul_rn(product, before);
            }
            const bool live = s < count && t < count;
            low[h][t][s] = live && t > s ? __fmul_rn(beta_sh[h][t], __fmul_rn(product, kk)) : 0.0f;
            qk_sh[h][t][s] = live && t >= s ? __fmul_rn(product, qk) : 0.0f;
            if (s == 0) gamma_sh[h][t] = __fmul_rn(decay_sh[h][0], product);
            if (t == kChunk - 1) carry_sh[h][s] = product;  // (the decay of a token beyond the chunk is 1)
        }
        __syncthreads();
        if (warp < heads && lane < kChunk) {  // column c of T1 = (I + L)^-1 diag(beta), held in registers: the chain is multiply-adds, not loads
            const unsigned c = lane;
            const auto& l = low[warp];
            float column[kChunk];
#pragma unroll
            for (int r = 0; r < kChunk; ++r) {
                float l4[kChunk], value[2] = {r == static_cast<int>(c) ? 1.0f : 0.0f, 0.0f};
#pragma unroll
                for (int m = 0; m < r; m += 4) *reinterpret_cast<float4*>(&l4[m]) = *reinterpret_cast<const float4*>(&l[r][m]);
#pragma unroll
                for (int m = 0; m < r; ++m) value[m % 2] = __fmaf_rn(-l4[m], column[m], value[m % 2]);  // column[m] is 0 above the diagonal
                column[r] = r < static_cast<int>(c) ? 0.0f : value[0] + value[1];
            }
#pragma unroll
            for (int r = 0; r < kChunk; ++r) inv[warp][r][c] = __fmul_rn(column[r], beta_sh[warp][c]);
        }
        __syncthreads();
        if (s < count) {  // row s, column t of T2 and W
            for (unsigned h = 0; h < heads; ++h) {
                float w = 0.0f;
#pragma unroll
                for (unsigned m = 0; m < kChunk; ++m)
                    if (m >= t && m <= s) w = __fmaf_rn(qk_sh[h][s][m], inv[h][m][t], w);
                float* row = p.coef + (static_cast<size_t>(first_head + h) * p.n_tokens + token0 + s) * kCoef;
                row[t] = t <= s ? round_tf32(__fmul_rn(carry_sh[h][s], inv[h][s][t])) : 0.0f;
                row[24 + t] = t <= s ? round_tf32(w) : 0.0f;
                if (t == 0) row[48] = gamma_sh[h][s];
            }
        }
    }
}

// How a block of the scan is laid out: `Parts` warps share the 128 rows of the state, each warp holds `Wide` times sixteen columns of its
// rows, and there are `Sets` such sets of columns side by side.
template <int Parts, int Wide, int Sets>
struct ScanShape {
    static constexpr int kColumns = kCols * Wide * Sets;
    static constexpr int kRows = kDim / Parts, kBlocks = kRows / 8;
    static constexpr int kStateWarps = Parts * Sets, kConsumers = kStateWarps + Sets, kThreads = 32 * (kConsumers + 1);
    static constexpr int kVPitch = kColumns % 32 == 0 ? kColumns + 8 : 24;  // spreads the tokens of a fragment over the banks
    static constexpr int kStages = 4;
    struct Stage {  // what the sixteen tokens of a chunk need from global memory
        float kq[kChunk][kPair];
        float coef[kChunk][kCoef];
        float v[kChunk][kVPitch];
    };
    // A chunk's products with a part of the state's rows: X^T in [0], [1] (tokens 0-7, 8-15) and O^T in [2], [3], each lane's four values
    // together.
    struct Partial {
        float4 value[4][32];
    };
    struct Smem {
        Stage stages[kStages];
        Partial parts[2][Sets][Parts][Wide];
        unsigned long long full[kStages], empty[kStages];
        unsigned abort_flag;
    };
};

// A bounded wait. False when it ran out here or elsewhere in the block. The caller goes on all the same (what it reads is somewhere in
// shared memory), so that every warp meets the others at every barrier; but no state is stored by a block whose flag is up. The flag is up
// before the warp that gave up arrives at the set's barrier, so a sibling that adds up its partial sums behind that barrier finds it when
// it looks, before it stores. (The reads are scratch. Looking before each chunk's cost a twentieth of a long run: 4096 tokens 377 -> 396 us.)
__device__ __forceinline__ bool scan_wait(uint32_t bar, uint32_t parity, unsigned* abort_flag, int* status, unsigned run) {
    if (ptx::mbar_try_wait(bar, parity)) return true;
    const long long began = clock64();
    while (!ptx::mbar_try_wait(bar, parity)) {
        if (*static_cast<volatile unsigned*>(abort_flag) != 0 || clock64() - began > kWaitLimit) {
            *static_cast<volatile unsigned*>(abort_flag) = 1;
            atomicCAS(status, 0, kStatusDeltaNet | (static_cast<int>(run) << 8));
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void add_to(float4& sum, const float4& v) { sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w; }

// The slot's tail becomes the last K - 1 rows of (old tail, then the run's inputs): one warp's share of the channels, `part` of `parts`.
// In the scan, because the launch before it has read the old tail by then and the launch after it may write over the inputs (`out` may lie
// on `mixed`).
__device__ __forceinline__ void leave_tail(const DeltaParams& p, const DeltaNetRow& run, unsigned part, unsigned parts, unsigned lane) {
    const unsigned history = p.taps - 1, share = (p.conv_dim + parts - 1) / parts;
    float* tail = p.tails + static_cast<size_t>(run.slot) * history * p.conv_dim;
    for (unsigned c = part * share + lane; c < min((part + 1) * share, p.conv_dim); c += 32) {
        float x[7];  // all rows before the first is written: a run shorter than the tail moves its old rows up
#pragma unroll
        for (unsigned i = 0; i < 7; ++i) x[i] = i < history ? input_at(p, run, tail, static_cast<int>(run.length + i) - static_cast<int>(history), c) : 0.0f;
#pragma unroll
        for (unsigned i = 0; i < 7; ++i)
            if (i < history) tail[static_cast<size_t>(i) * p.conv_dim + c] = x[i];
    }
}

// One block per run, value head and ScanShape::kColumns columns of the state (columns evolve independently of one another). A chunk's
// chain is state -> products with it -> y -> T2 y -> state. The warps of a set hold their part of the state in registers and exchange
// partial sums through shared memory once a chunk (each then forms y and T2 y for itself). What hangs off the chain is not theirs: one
// more warp a set adds up the reads, a last one brings the chunks and then leaves the tail (two bulk copies a chunk for k, q and the coefficients, which lie in
// global memory as they do here: many small ones take longer to issue than the chunk's arithmetic; cp.async for the block's columns of
// v). The reads go to global memory in float32; the gated norm over a head's 128 reads is the next launch.
//
// One run, 32 value heads: 0.86 us a chunk, 54 ns a token (with one warp to sixteen columns 82 ns), and that is the latency of the chain:
// the same without any copies, issue slots 38 %, tensor pipe 23 %, shared-memory pipe 45 %. Parts 2 and sixteen columns to a warp were
// the best of ten layouts (900 tokens: 53 us; four parts 63; one set of two by two 66; 64 columns to a block 78). Fetching the last
// product's operands in the middle of the first products gave 9 %; 16-byte loads of k and q (fewer instructions) lost 5 %.
//
// Tokens within a tile of eight: column j of an accumulator tile is token (0, 2, 1, 3, 6, 4, 7, 5)[j]. With that order both ways k is
// read (eight tokens' pairs of dimensions as the B operand of the first products, four pairs of tokens as that of the last) touch every
// bank once.
template <int Parts, int Wide, int Sets>
__global__ void __launch_bounds__(ScanShape<Parts, Wide, Sets>::kThreads) deltanet_scan_kernel(const __grid_constant__ DeltaParams p) {
    extern __shared__ __align__(16) unsigned char scan_smem[];
    using Shape = ScanShape<Parts, Wide, Sets>;
    using Stage = typename Shape::Stage;
    auto& sm = *reinterpret_cast<typename Shape::Smem*>(scan_smem);
    constexpr int kStages = Shape::kStages, kBlocks = Shape::kBlocks;
    const unsigned lane = threadIdx.x % 32, warp = threadIdx.x / 32, g = lane / 4, t = lane % 4;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            ptx::mbar_init(ptx::smem_addr(&sm.full[i]), 1 + 32);  // the bulk copies' arrival and each lane's cp.async
            ptx::mbar_init(ptx::smem_addr(&sm.empty[i]), Shape::kConsumers);
        }
        sm.abort_flag = 0;
        ptx::fence_barrier_init();
    }
    ptx::grid_dependency_wait();
    const unsigned columns = blockIdx.x % (kDim / Shape::kColumns), head = blockIdx.x / (kDim / Shape::kColumns) % p.value_heads;
    const unsigned turn_of_run = blockIdx.x / (kDim / Shape::kColumns * p.value_heads), run = p.far_runs != nullptr ? turn_of_run : p.near_order[turn_of_run];
    const DeltaNetRow row = run_at(p, run);
    // What a short last chunk leaves unwritten of its buffer must be finite: an earlier chunk of the run has been there, or it is zeroed.
    // (All four buffers zeroed in every block: 93 us for 48 runs of 66 tokens, 16 heads; so, 86.)
    const unsigned chunks = (row.length + kChunk - 1) / kChunk;
    if (row.length % kChunk != 0 && chunks <= kStages) {
        static_assert(sizeof(Stage) % 16 == 0, "zeroed sixteen bytes at a time");
        float4* last = reinterpret_cast<float4*>(&sm.stages[chunks - 1]);
        for (unsigned e = threadIdx.x; e < sizeof(Stage) / 16; e += blockDim.x) last[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    ptx::fence_proxy_async_smem();
    __syncthreads();
    const unsigned key_head = head / (p.value_heads / p.key_heads);
    if (warp == Shape::kConsumers) {
        const float* v_src = p.v + static_cast<size_t>(row.q_begin) * p.value_dim + head * kDim + columns * Shape::kColumns;
        unsigned issued = 0;  // chunks
        for (unsigned t0 = 0; t0 < row.length; t0 += kChunk, ++issued) {
            const unsigned round = issued, turn = round % kStages;
            if (round >= kStages) {
                const bool ok = scan_wait(ptx::smem_addr(&sm.empty[turn]), (round / kStages - 1) & 1u, &sm.abort_flag, p.status, run);
                // (a warp that gave up goes on to release buffers, the one it gave up on too: nothing is brought into them any more)
                if (!__all_sync(0xFFFFFFFFu, ok && *static_cast<volatile unsigned*>(&sm.abort_flag) == 0)) break;
            }
            Stage& sg = sm.stages[turn];
            const uint32_t bar = ptx::smem_addr(&sm.full[turn]);
            const unsigned count = min(static_cast<unsigned>(kChunk), row.length - t0);
            if (lane == 0) {
                const size_t token0 = static_cast<size_t>(row.q_begin) + t0;
                ptx::mbar_arrive_expect_tx(bar, count * ((kPair + kCoef) * 4));
                ptx::bulk_load(ptx::smem_addr(&sg.kq[0][0]), p.kq + (static_cast<size_t>(key_head) * p.n_tokens + token0) * kPair, count * kPair * 4, bar);
                ptx::bulk_load(ptx::smem_addr(&sg.coef[0][0]), p.coef + (static_cast<size_t>(head) * p.n_tokens + token0) * kCoef, count * kCoef * 4, bar);
            }
            constexpr unsigned kPieces = Shape::kColumns / 4;  // 16-byte pieces of a token's columns
#pragma unroll
            for (unsigned e = lane; e < kChunk * kPieces; e += 32) {
                const unsigned token = e / kPieces, piece = e % kPieces;
                if (token < count) ptx::cp_async_16(ptx::smem_addr(&sg.v[token][4 * piece]), v_src + static_cast<size_t>(t0 + token) * p.value_dim + 4 * piece);
            }
            ptx::cp_async_mbar_arrive(bar);
        }
        leave_tail(p, row, head * (kDim / Shape::kColumns) + columns, p.value_heads * (kDim / Shape::kColumns), lane);
        ptx::grid_launch_dependents();
        // The block's shared memory stays its own until the copies have landed, also when a wait ran out and the other warps are gone.
        if (lane == 0) {
            const long long began = clock64();
            for (unsigned round = issued < kStages ? 0u : issued - kStages; round < issued; ++round)
                while (!ptx::mbar_try_wait(ptx::smem_addr(&sm.full[round % kStages]), (round / kStages) & 1u) && clock64() - began < kWaitLimit) {
                }
        }
        return;
    }
    const bool holds_state = warp < Shape::kStateWarps;
    const unsigned set = holds_state ? warp / Parts : warp - Shape::kStateWarps, part = warp % Parts;
    const unsigned first_row = part * Shape::kRows, set_col = set * (kCols * Wide);
    const unsigned first_col = columns * Shape::kColumns + set_col;
    const unsigned token_of[2] = {t < 2 ? t : t + 4, t + 2};  // the tokens of this lane's two columns of an accumulator tile
    const unsigned token_g = g % 2 != 0 ? g / 2 + 2 : g / 2 < 2 ? g / 2 : g / 2 + 4;  // ... and of column g, as operands have it
    // block b of this warp's rows: rows 8 b + 2 t and 8 b + 2 t + 1 of columns g ([0], [1]) and g + 8 ([2], [3])
    float st[kBlocks][Wide][4] = {};
    float* state = p.states + ((static_cast<size_t>(row.slot) * p.value_heads + head) * kDim + first_row) * kDim + first_col;
    if (holds_state && row.fresh == 0) {
#pragma unroll
        for (int b = 0; b < kBlocks; ++b) {
#pragma unroll
            for (int w = 0; w < Wide; ++w) {
#pragma unroll
                for (int e = 0; e < 4; ++e) st[b][w][e] = state[static_cast<size_t>(8 * b + 2 * t + (e & 1)) * kDim + kCols * w + g + 8 * (e >> 1)];
            }
        }
    }
    const float scale = rsqrtf(static_cast<float>(kDim));
    bool ok = true;
    for (unsigned t0 = 0, round = 0; t0 < row.length; t0 += kChunk, ++round) {
        const unsigned turn = round % kStages;
        const unsigned count = min(static_cast<unsigned>(kChunk), row.length - t0);
        const Stage& sg = sm.stages[turn];
        auto& parts = sm.parts[round & 1u][set];
        ok &= scan_wait(ptx::smem_addr(&sm.full[turn]), (round / kStages) & 1u, &sm.abort_flag, p.status, run);
        __syncwarp();
        // Everything this warp needs of the buffer beside the operands of the first products: v and gamma by token in accumulator layout
        // (element e of tile i is token 8 i + token_of[e & 1], column g + 8 (e >> 1)), T2 or W, lower triangular, as the B operand, K as
        // the last product's operand. Fetched in the middle of the first products, which leave the load pipe idle.
        float v[Wide][2][4], gamma[2][2], gamma_last;
        float2 m[3], ku[kBlocks][2];
        const auto fetch = [&] {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int w = 0; w < Wide; ++w) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[w][i][e] = sg.v[8 * i + token_of[e & 1]][set_col + kCols * w + g + 8 * (e >> 1)];
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) gamma[i][e] = sg.coef[8 * i + token_of[e]][48];
            }
            const unsigned at = holds_state ? 0u : 24u;
            m[0] = make_float2(sg.coef[token_g][at + token_of[0]], sg.coef[token_g][at + token_of[1]]);
            m[1] = make_float2(sg.coef[8 + token_g][at + token_of[0]], sg.coef[8 + token_g][at + token_of[1]]);
            m[2] = make_float2(sg.coef[8 + token_g][at + 8 + token_of[0]], sg.coef[8 + token_g][at + 8 + token_of[1]]);
            gamma_last = sg.coef[count - 1][48];
        };
        if (holds_state) {
            // X^T = S_0^T K^T and O^T = S_0^T Q^T over this warp's rows: [columns, tokens], tokens 0-7 in [0], 8-15 in [1]
            float x[Wide][2][4] = {}, o[Wide][2][4] = {};
#pragma unroll
            for (int b = 0; b < kBlocks; ++b) {
                if (b == kBlocks / 2) {
                    fetch();
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
#pragma unroll
                        for (int d = 0; d < kBlocks; ++d)
                            ku[d][j] = make_float2(sg.kq[8 * j + token_of[0]][first_row + 8 * d + g], sg.kq[8 * j + token_of[1]][first_row + 8 * d + g]);
                    }
                }
                float2 kf[2], qf[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    kf[i] = *reinterpret_cast<const float2*>(&sg.kq[8 * i + token_g][first_row + 8 * b + 2 * t]);
                    qf[i] = *reinterpret_cast<const float2*>(&sg.kq[8 * i + token_g][kDim + first_row + 8 * b + 2 * t]);
                }
#pragma unroll
                for (int w = 0; w < Wide; ++w) {
                    const uint32_t a0 = to_tf32(st[b][w][0]), a1 = to_tf32(st[b][w][2]), a2 = to_tf32(st[b][w][1]), a3 = to_tf32(st[b][w][3]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        mma_tf32(x[w][i], a0, a1, a2, a3, __float_as_uint(kf[i].x), __float_as_uint(kf[i].y));
                        mma_tf32(o[w][i], a0, a1, a2, a3, __float_as_uint(qf[i].x), __float_as_uint(qf[i].y));
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < kBlocks; ++b) {
#pragma unroll
                for (int w = 0; w < Wide; ++w) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) st[b][w][e] = __fmul_rn(st[b][w][e], gamma_last);
                }
            }
#pragma unroll
            for (int w = 0; w < Wide; ++w) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    parts[part][w].value[i][lane] = make_float4(x[w][i][0], x[w][i][1], x[w][i][2], x[w][i][3]);
                    parts[part][w].value[2 + i][lane] = make_float4(o[w][i][0], o[w][i][1], o[w][i][2], o[w][i][3]);
                }
            }
        } else {
            fetch();
        }
        // The set's partial sums are in place: its state warps and its reading warp meet here once a chunk. Two sets of sums alternate,
        // so a warp that writes those of chunk n has seen everyone finish reading those of chunk n - 2.
        ptx::named_barrier_sync(1 + set, 32 * (Parts + 1));
        if (lane == 0) ptx::mbar_arrive(ptx::smem_addr(&sm.empty[turn]));  // (the barrier ordered every lane's reads before this)
#pragma unroll
        for (int w = 0; w < Wide; ++w) {
            float c[2][4] = {};
            uint32_t ya[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float4 sum = parts[0][w].value[i][lane];
#pragma unroll
                for (int r = 1; r < Parts; ++r) add_to(sum, parts[r][w].value[i][lane]);
                const float xs[4] = {sum.x, sum.y, sum.z, sum.w};
                float y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)  // y = v - gamma x, zero beyond the chunk's tokens
                    y[e] = 8u * i + token_of[e & 1] < count ? __fsub_rn(v[w][i][e], __fmul_rn(gamma[i][e & 1], xs[e])) : 0.0f;
                ya[i][0] = to_tf32(y[0]), ya[i][1] = to_tf32(y[2]), ya[i][2] = to_tf32(y[1]), ya[i][3] = to_tf32(y[3]);
                if (!holds_state) {
                    float4 read = parts[0][w].value[2 + i][lane];
#pragma unroll
                    for (int r = 1; r < Parts; ++r) add_to(read, parts[r][w].value[2 + i][lane]);
                    c[i][0] = __fmul_rn(gamma[i][0], read.x), c[i][1] = __fmul_rn(gamma[i][1], read.y);
                    c[i][2] = __fmul_rn(gamma[i][0], read.z), c[i][3] = __fmul_rn(gamma[i][1], read.w);
                }
            }
            // C^T = y T2^T or the reads' two terms gamma o + y W^T: [columns, tokens] again
            mma_tf32(c[1], ya[0][0], ya[0][1], ya[0][2], ya[0][3], __float_as_uint(m[1].x), __float_as_uint(m[1].y));
            mma_tf32(c[0], ya[0][0], ya[0][1], ya[0][2], ya[0][3], __float_as_uint(m[0].x), __float_as_uint(m[0].y));
            mma_tf32(c[1], ya[1][0], ya[1][1], ya[1][2], ya[1][3], __float_as_uint(m[2].x), __float_as_uint(m[2].y));
            if (!holds_state) {
                float* reads = p.reads + (static_cast<size_t>(row.q_begin) + t0) * p.value_dim + head * kDim + first_col + kCols * w;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const unsigned token = 8 * i + token_of[e & 1];
                        if (ok && token < count) reads[static_cast<size_t>(token) * p.value_dim + g + 8 * (e >> 1)] = __fmul_rn(c[i][e], scale);
                    }
                }
                continue;
            }
            // S^T = gamma_last S_0^T + C^T K
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (8u * j + token_of[e & 1] >= count) c[j][e] = 0.0f;  // a row of T2 beyond the chunk is whatever an earlier chunk left there
                const uint32_t a0 = to_tf32(c[j][0]), a1 = to_tf32(c[j][2]), a2 = to_tf32(c[j][1]), a3 = to_tf32(c[j][3]);
#pragma unroll
                for (int b = 0; b < kBlocks; ++b) mma_tf32(st[b][w], a0, a1, a2, a3, __float_as_uint(ku[b][j].x), __float_as_uint(ku[b][j].y));
            }
        }
    }
    ptx::grid_launch_dependents();
    if (!ok || !holds_state || *static_cast<volatile unsigned*>(&sm.abort_flag) != 0) return;
#pragma unroll
    for (int b = 0; b < kBlocks; ++b) {
#pragma unroll
        for (int w = 0; w < Wide; ++w) {
#pragma unroll
            for (int e = 0; e < 4; ++e) state[static_cast<size_t>(8 * b + 2 * t + (e & 1)) * kDim + kCols * w + g + 8 * (e >> 1)] = st[b][w][e];
        }
    }
}

template <int Parts, int Wide, int Sets>
void launch_scan(const Context& ctx, const DeltaParams& p, cudaStream_t stream) {
    using Shape = ScanShape<Parts, Wide, Sets>;
    static std::atomic<bool> configured[64] = {};  // per device; every writer sets the same attribute
    if (ctx.device >= 64 || !configured[ctx.device].load(std::memory_order_relaxed)) {
        check(cudaFuncSetAttribute(deltanet_scan_kernel<Parts, Wide, Sets>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(typename Shape::Smem))), "cudaFuncSetAttribute");
        if (ctx.device < 64) configured[ctx.device].store(true, std::memory_order_relaxed);
    }
    // Overlapped with the launch before it only where that has a block to an SM at most: blocks of the scan that arrive while it still fills
    // the SMs settle wherever room appears first, several to an SM with other SMs left empty, and a run's warps then take twice as long.
    const dim3 grid(p.n_rows * p.value_heads * (kDim / Shape::kColumns)), block(Shape::kThreads);
    if (p.n_chunks * p.key_heads <= static_cast<unsigned>(ctx.sm_count)) {
        launch_kernel(deltanet_scan_kernel<Parts, Wide, Sets>, grid, block, sizeof(typename Shape::Smem), stream, "deltanet_scan_kernel launch", p);
    } else {
        deltanet_scan_kernel<Parts, Wide, Sets><<<grid, block, sizeof(typename Shape::Smem), stream>>>(p);
        check(cudaGetLastError(), "deltanet_scan_kernel launch");
    }
    count_launch();
}

// The gated norm of every token's and value head's 128 reads: x / sqrt(mean(x^2) + eps) * weight * silu(z) (the weight itself, not
// 1 + weight). A warp takes four (token, head) pairs in a row, all their loads in flight together; lane l holds reads 4 l to 4 l + 3;
// squares by fused multiply-add in that order, a butterfly. 4096 tokens, 32 heads, 134 MB: 50 us under the profiler, bound by
// instructions (62 % of the issue slots).
constexpr unsigned kNormUnits = 4;

__global__ void __launch_bounds__(256) deltanet_norm_kernel(const __grid_constant__ DeltaParams p) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const unsigned lane = threadIdx.x % 32;
    const unsigned first = (blockIdx.x * 8 + threadIdx.x / 32) * kNormUnits, units = p.n_tokens * p.value_heads;
    const float4 weight = make_float4(p.norm[4 * lane], p.norm[4 * lane + 1], p.norm[4 * lane + 2], p.norm[4 * lane + 3]);
    float4 x[kNormUnits], gate[kNormUnits];
    bool live[kNormUnits], in_run = false;
    __half* dst[kNormUnits];
    unsigned token = first / p.value_heads, head = first % p.value_heads;
#pragma unroll
    for (unsigned i = 0; i < kNormUnits; ++i) {
        live[i] = false;
        if (first + i >= units) continue;
        if (i > 0 && ++head == p.value_heads) head = 0, ++token;
        if (i == 0 || head == 0) {
            const DeltaNetRow run = run_at(p, run_of_token(p, token));
            in_run = token >= run.q_begin && token - run.q_begin < run.length;
        }
        if (!in_run) continue;  // a gap between runs
        live[i] = true;
        x[i] = *reinterpret_cast<const float4*>(p.reads + static_cast<size_t>(first + i) * kDim + 4 * lane);
        const size_t at = token * p.z_stride + head * kDim + 4 * lane;
        dst[i] = p.out + token * p.out_stride + head * kDim + 4 * lane;
        if (p.wide_norm != 0) {
            const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p.z) + at);
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
            gate[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
        } else {
            gate[i] = make_float4(value_of(p.z, at, p.z_half), value_of(p.z, at + 1, p.z_half), value_of(p.z, at + 2, p.z_half), value_of(p.z, at + 3, p.z_half));
        }
    }
#pragma unroll
    for (unsigned i = 0; i < kNormUnits; ++i) {
        if (!live[i]) continue;  // (the whole warp)
        float ss = __fmaf_rn(x[i].w, x[i].w, __fmaf_rn(x[i].z, x[i].z, __fmaf_rn(x[i].y, x[i].y, __fmaf_rn(x[i].x, x[i].x, 0.0f))));
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
        const float rms = __fsqrt_rn(__fadd_rn(__fmul_rn(ss, 1.0f / kDim), p.eps));
        const auto normed = [&](float read, float w, float z) { return __fmul_rn(__fmul_rn(__fdiv_rn(read, rms), w), silu(z)); };
        const __half2 lo = __floats2half2_rn(normed(x[i].x, weight.x, gate[i].x), normed(x[i].y, weight.y, gate[i].y));
        const __half2 hi = __floats2half2_rn(normed(x[i].z, weight.z, gate[i].z), normed(x[i].w, weight.w, gate[i].w));
        if (p.wide_norm != 0) {
            *reinterpret_cast<uint2*>(dst[i]) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
        } else {
            dst[i][0] = __low2half(lo), dst[i][1] = __high2half(lo), dst[i][2] = __low2half(hi), dst[i][3] = __high2half(hi);
        }
    }
}

}  // namespace

bool deltanet_supports(const DeltaNetShape& s) {
    return s.head_dim == 128 && s.key_heads != 0 && s.value_heads != 0 && s.value_heads % s.key_heads == 0 && s.key_heads <= 32 && s.conv_kernel >= 1 &&
           s.conv_kernel <= 8;
}

void launch_deltanet(Context& ctx, const DeltaNetShape& shape, const DeltaNetRow* rows, std::size_t n_rows, Band mixed, Band z, Band b, Band a,
                     const DeltaNetWeights& weights, const DeltaNetScratch& scratch, float* states, float* tails, std::size_t slots,
                     void* out, std::size_t out_stride, cudaStream_t stream) {
    if (!deltanet_supports(shape))
        throw std::invalid_argument("sepal_b200 deltanet: head_dim must be 128, value_heads a multiple of key_heads (at most 32 key heads), 1 to 8 conv taps");
    if (n_rows == 0) return;
    if (rows == nullptr || mixed.data == nullptr || z.data == nullptr || b.data == nullptr || a.data == nullptr || weights.conv == nullptr ||
        weights.a_log == nullptr || weights.dt_bias == nullptr || weights.norm == nullptr || scratch.kq == nullptr ||
        scratch.v == nullptr || scratch.reads == nullptr || scratch.coef == nullptr || states == nullptr || tails == nullptr || out == nullptr)
        throw std::invalid_argument("sepal_b200 deltanet: null pointer");
    for (std::size_t i = 0; i < n_rows; ++i) {
        if (rows[i].length == 0) throw std::invalid_argument("sepal_b200 deltanet: row " + std::to_string(i) + " is empty");
        if (i > 0 && rows[i].q_begin < rows[i - 1].q_begin + rows[i - 1].length) throw std::invalid_argument("sepal_b200 deltanet: rows must be sorted by their first token and must not overlap");
        if (rows[i].slot >= slots) throw std::invalid_argument("sepal_b200 deltanet: row " + std::to_string(i) + " names a state slot that does not exist");
        for (std::size_t o = 0; o < i; ++o)
            if (rows[o].slot == rows[i].slot) throw std::invalid_argument("sepal_b200 deltanet: two rows of one call share a state slot");
    }
    check(cudaSetDevice(ctx.device), "cudaSetDevice");
    DeltaParams p{};
    // the table of the call: the runs and the numbers of their first chunks
    std::vector<unsigned> chunks(n_rows);
    std::size_t n_chunks = 0;
    for (std::size_t i = 0; i < n_rows; ++i) {
        chunks[i] = static_cast<unsigned>(n_chunks);
        n_chunks += (rows[i].length + kChunk - 1) / kChunk;
    }
    // (what a call may have at most is counted as a row and 16 bytes a chunk, more than the table takes: a limit of the interface)
    const std::size_t rows_bytes = n_rows * sizeof(DeltaNetRow), table_bytes = rows_bytes + n_chunks * 16;
    if (ctx.table == nullptr || table_bytes > ctx.table_bytes / 2) throw std::invalid_argument("sepal_b200 deltanet: too many rows for the context's table");
    if (n_rows <= kInlineRuns) {
        std::memcpy(p.near_runs, rows, rows_bytes);
        std::memcpy(p.near_chunks, chunks.data(), n_rows * sizeof(unsigned));
        for (std::size_t i = 0; i < n_rows; ++i) p.near_order[i] = static_cast<unsigned char>(i);
        std::stable_sort(p.near_order, p.near_order + n_rows, [&](unsigned char a, unsigned char b) { return rows[a].length > rows[b].length; });
    } else {
        std::vector<char> host(rows_bytes + n_rows * sizeof(unsigned));
        std::memcpy(host.data(), rows, rows_bytes);
        std::memcpy(host.data() + rows_bytes, chunks.data(), n_rows * sizeof(unsigned));
        char* table = static_cast<char*>(ctx.table) + (ctx.table_turn++ & 1u) * (ctx.table_bytes / 2);
        check(cudaMemcpyAsync(table, host.data(), host.size(), cudaMemcpyHostToDevice, stream), "cudaMemcpyAsync(rows)");
        p.far_runs = reinterpret_cast<const DeltaNetRow*>(table);
        p.far_chunks = reinterpret_cast<const unsigned*>(table + rows_bytes);
    }
    p.n_rows = static_cast<unsigned>(n_rows);
    p.n_chunks = static_cast<unsigned>(n_chunks);
    p.key_heads = shape.key_heads;
    p.value_heads = shape.value_heads;
    p.taps = shape.conv_kernel;
    p.value_dim = shape.value_dim();
    p.conv_dim = shape.conv_dim();
    p.eps = shape.eps;
    p.mixed = mixed.data;
    p.z = z.data;
    p.b = b.data;
    p.a = a.data;
    p.mixed_stride = mixed.stride;
    p.z_stride = z.stride;
    p.b_stride = b.stride;
    p.a_stride = a.stride;
    p.mixed_half = mixed.half ? 1u : 0u;
    p.z_half = z.half ? 1u : 0u;
    p.b_half = b.half ? 1u : 0u;
    p.a_half = a.half ? 1u : 0u;
    p.conv = weights.conv;
    p.a_log = weights.a_log;
    p.dt_bias = weights.dt_bias;
    p.norm = weights.norm;
    p.kq = scratch.kq;
    p.v = scratch.v;
    p.reads = scratch.reads;
    p.coef = scratch.coef;
    p.status = ctx.status;
    p.states = states;
    p.tails = tails;
    p.out = static_cast<__half*>(out);
    p.out_stride = out_stride;
    const unsigned last = rows[n_rows - 1].q_begin + rows[n_rows - 1].length;
    p.n_tokens = last;
    // (a limit of the interface: no kernel here holds more than 128 channels a warp)
    if (p.conv_dim > 40960) throw std::invalid_argument("sepal_b200 deltanet: the convolution is wider than 40960 channels");
    // two channels a load in the convolution, four values a load and store in the gated norm, where the types and addresses allow it
    const bool pairs = mixed.half && shape.conv_kernel == 4 && mixed.stride % 2 == 0 && reinterpret_cast<std::uintptr_t>(mixed.data) % 4 == 0 &&
                       reinterpret_cast<std::uintptr_t>(weights.conv) % 16 == 0 && reinterpret_cast<std::uintptr_t>(tails) % 8 == 0;
    p.wide_norm = z.half && z.stride % 4 == 0 && reinterpret_cast<std::uintptr_t>(z.data) % 8 == 0 && out_stride % 4 == 0 && reinterpret_cast<std::uintptr_t>(out) % 8 == 0;
    launch_kernel(pairs ? deltanet_prepare_kernel<true> : deltanet_prepare_kernel<false>, dim3(p.n_chunks, shape.key_heads), dim3(256), 0, stream, "deltanet_prepare_kernel launch", p);
    count_launch();
    // Sixteen columns of the state to a block while every block then has an SM of its own (one run of 900 tokens, 16 heads: 46.8 us
    // against 52.1 with 32), otherwise 32, which read k, q and the coefficients half as often (32 heads: 53.2 against 60.3; four runs of
    // 4169 tokens in all: 171 against 248; blocks of 64 columns: 78 and 183).
    if (n_rows * shape.value_heads * (kDim / kCols) <= static_cast<std::size_t>(ctx.sm_count))
        launch_scan<2, 1, 1>(ctx, p, stream);
    else
        launch_scan<2, 1, 2>(ctx, p, stream);
    const std::size_t units = static_cast<std::size_t>(last) * shape.value_heads;
    launch_kernel(deltanet_norm_kernel, dim3(static_cast<unsigned>((units + 8 * kNormUnits - 1) / (8 * kNormUnits))), dim3(256), 0, stream,
                  "deltanet_norm_kernel launch", p);
    count_launch();
}

}  // namespace sepal::b200
