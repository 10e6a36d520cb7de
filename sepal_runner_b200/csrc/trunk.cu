#include "trunk.hpp"

#include "ptx.cuh"

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>

#include <cuda_fp16.h>

namespace sepal::b200 {

void count_launch();

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {  // splitmix64 finaliser
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ float normal_at(unsigned long long seed, unsigned long long i) {
    const unsigned long long h = mix64(seed * 0xD1B54A32D192ED03ull + i);
    const float u1 = (static_cast<float>(static_cast<unsigned>(h >> 40)) + 1.0f) * (1.0f / 16777217.0f);  // (0, 1)
    const float u2 = static_cast<float>(static_cast<unsigned>(h & 0xFFFFFFu)) * (1.0f / 16777216.0f);
    return sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}
__device__ __forceinline__ float to_bf16_grid(float v) {
    const unsigned bits = __float_as_uint(v);
    return __uint_as_float((bits + 0x7FFFu + ((bits >> 16) & 1u)) & 0xFFFF0000u);
}
__global__ void fill_normal_half_kernel(__half* dst, std::size_t count, unsigned long long seed, float stddev) {
    const std::size_t i = static_cast<std::size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count) dst[i] = __float2half_rn(to_bf16_grid(normal_at(seed, i) * stddev));
}
__global__ void fill_normal_float_kernel(float* dst, std::size_t count, unsigned long long seed, float stddev) {
    const std::size_t i = static_cast<std::size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count) dst[i] = to_bf16_grid(normal_at(seed, i) * stddev);
}

// One block per token: a row of the binary16 table widened to the float32 residual stream, 8 values per thread and step.
__global__ void embed_kernel(const __half* table, const std::uint32_t* tokens, float* x, std::size_t hidden, std::size_t vocab) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();  // the kernel before this one may still read the rows this one overwrites
    const std::size_t row = blockIdx.x;
    std::size_t id = tokens[row];
    if (id >= vocab) id = vocab - 1;  // the host checks the ids; never read outside the table
    const uint4* src = reinterpret_cast<const uint4*>(table + id * hidden);
    float4* dst = reinterpret_cast<float4*>(x + row * hidden);
    for (std::size_t v = threadIdx.x; v < hidden / 8; v += blockDim.x) {
        const uint4 raw = src[v];
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
        const float2 a = __half22float2(h[0]), b = __half22float2(h[1]), c = __half22float2(h[2]), d = __half22float2(h[3]);
        dst[2 * v] = make_float4(a.x, a.y, b.x, b.y);
        dst[2 * v + 1] = make_float4(c.x, c.y, d.x, d.y);
    }
}

// The zero-centred RMSNorm, y = (x / rms) * (1 + w) with rms = sqrt(mean(x^2) + eps), every step rounded to float32 and the result to
// binary16. The sum of squares must come out bit for bit as the reference's kernel forms it (runner/cuda/src/kernels_elementwise.cu:6-11,
// 114-141), because a row's bits may depend on nothing but the row: the row in chunks of four consecutive elements, chunk c added (one
// fused multiply-add per element, ascending c) into partial sum number c mod 256; each run of 32 partial sums folded by a butterfly
// (p[l] += p[l ^ o], o = 16, 8, 4, 2, 1); the eight results added in order.
//
// A block of 256 threads owns a row, thread i the partial sum number i. What bounds the launch between two multiplies is the latency of
// a row, not its bytes (which the L2 still holds), so a thread has at most kNormHeld chunks, their loads and the gains' in flight at
// once, and the row meets at one barrier. (A warp to a row, with 80 divisions to a lane: 8.8 us for 29 rows of 1024 under the profiler.)
// Rows wider than the registers hold are read a second time.
constexpr unsigned kNormThreads = 256;
constexpr int kNormHeld = 4;  // chunks a thread keeps: rows up to 4096 wide

__device__ __forceinline__ float square_into(float sum, const float4& v) {
    return __fmaf_rn(v.w, v.w, __fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, __fmaf_rn(v.x, v.x, sum))));
}

__device__ __forceinline__ uint2 normed_chunk(const float4& v, float rms, const float4& g) {
    const __half2 lo = __floats2half2_rn(__fmul_rn(__fdiv_rn(v.x, rms), __fadd_rn(1.0f, g.x)), __fmul_rn(__fdiv_rn(v.y, rms), __fadd_rn(1.0f, g.y)));
    const __half2 hi = __floats2half2_rn(__fmul_rn(__fdiv_rn(v.z, rms), __fadd_rn(1.0f, g.z)), __fmul_rn(__fdiv_rn(v.w, rms), __fadd_rn(1.0f, g.w)));
    return make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}

// `fetch(c)` yields chunk c of the block's row as four floats (from the float32 stream, or widened from the binary16 embedding table and
// written to the stream on the way). All threads of the block call this.
template <class Fetch>
__device__ __forceinline__ void norm_row_in_a_block(Fetch&& fetch, const float* w, __half* yr, std::size_t cols, float eps) {
    __shared__ float folded[kNormThreads / 32];
    const std::size_t chunks = cols / 4;
    const float4* gain = reinterpret_cast<const float4*>(w);
    float4 held[kNormHeld], g[kNormHeld];
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i) {
        const std::size_t c = threadIdx.x + kNormThreads * static_cast<std::size_t>(i);
        if (c < chunks) {
            held[i] = fetch(c);
            g[i] = gain[c];
        }
    }
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i)
        if (threadIdx.x + kNormThreads * static_cast<std::size_t>(i) < chunks) sum = square_into(sum, held[i]);
    for (std::size_t c = threadIdx.x + kNormThreads * static_cast<std::size_t>(kNormHeld); c < chunks; c += kNormThreads) sum = square_into(sum, fetch(c));
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (threadIdx.x % 32 == 0) folded[threadIdx.x / 32] = sum;
    __syncthreads();
    float total = folded[0];
#pragma unroll
    for (unsigned s = 1; s < kNormThreads / 32; ++s) total += folded[s];
    const float rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(cols)), eps));
    uint2* out = reinterpret_cast<uint2*>(yr);
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i) {
        const std::size_t c = threadIdx.x + kNormThreads * static_cast<std::size_t>(i);
        if (c < chunks) out[c] = normed_chunk(held[i], rms, g[i]);
    }
    for (std::size_t c = threadIdx.x + kNormThreads * static_cast<std::size_t>(kNormHeld); c < chunks; c += kNormThreads) out[c] = normed_chunk(fetch(c), rms, gain[c]);
}

__global__ void __launch_bounds__(kNormThreads) rms_norm_half_kernel(const float* x, std::size_t ld_x, const float* w, __half* y, std::size_t ld_y, std::size_t cols,
                                                                     float eps) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();  // x is the output of the multiply launched before this kernel
    const std::size_t row = blockIdx.x;
    const float4* xr = reinterpret_cast<const float4*>(x + row * ld_x);
    norm_row_in_a_block([&](std::size_t c) { return xr[c]; }, w, y + row * ld_y, cols, eps);
}

// The embedding gather and the first layer's input norm in one pass (the reference runs launch_embed and launch_rms_norm back to back,
// runner/cuda/src/cuda_engine.cpp:1676-1692): the row of the binary16 table is widened (exactly) to the float32 stream and normed from
// the registers (a row wider than the registers hold is widened a second time for the second pass).
__global__ void __launch_bounds__(kNormThreads) embed_rms_norm_half_kernel(const __half* table, const std::uint32_t* tokens, float* x, const float* w, __half* y,
                                                                            std::size_t ld_y, std::size_t hidden, std::size_t vocab, float eps) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();  // the kernel before this one may still read the rows this one overwrites
    const std::size_t row = blockIdx.x;
    std::size_t id = tokens[row];
    if (id >= vocab) id = vocab - 1;  // the host checks the ids; never read outside the table
    const uint2* src = reinterpret_cast<const uint2*>(table + id * hidden);
    float4* xr = reinterpret_cast<float4*>(x + row * hidden);
    norm_row_in_a_block(
        [&](std::size_t c) {
            const uint2 raw = src[c];
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
            const float4 v = make_float4(a.x, a.y, b.x, b.y);
            xr[c] = v;  // written twice with the same value when the row is wider than the registers hold
            return v;
        },
        w, y + row * ld_y, hidden, eps);
}

unsigned blocks_for(std::size_t n, unsigned per) { return static_cast<unsigned>((n + per - 1) / per); }

}  // namespace

void launch_embed(const void* table_half, const std::uint32_t* tokens, float* x, std::size_t rows, std::size_t hidden, std::size_t vocab, cudaStream_t stream) {
    if (hidden % 8 != 0) throw std::invalid_argument("launch_embed: the hidden size must be a multiple of 8");
    if (rows == 0) return;
    launch_kernel(embed_kernel, dim3(static_cast<unsigned>(rows)), dim3(128), 0, stream, "embed_kernel launch", static_cast<const __half*>(table_half), tokens, x,
                  hidden, vocab);
    count_launch();
}

void launch_embed_rms_norm_half(const void* table_half, const std::uint32_t* tokens, float* x, const float* w, void* y_half, std::size_t ld_y, std::size_t rows,
                                std::size_t hidden, std::size_t vocab, float eps, cudaStream_t stream) {
    if (hidden % 8 != 0 || ld_y % 4 != 0) throw std::invalid_argument("launch_embed_rms_norm_half: the hidden size must be a multiple of 8 and the stride of y of 4");
    if (rows == 0) return;
    launch_kernel(embed_rms_norm_half_kernel, dim3(static_cast<unsigned>(rows)), dim3(kNormThreads), 0, stream, "embed_rms_norm_half_kernel launch",
                  static_cast<const __half*>(table_half), tokens, x, w, static_cast<__half*>(y_half), ld_y, hidden, vocab, eps);
    count_launch();
}

void launch_rms_norm_half(const float* x, std::size_t ld_x, const float* w, void* y_half, std::size_t ld_y, std::size_t rows, std::size_t cols, float eps,
                          cudaStream_t stream) {
    if (cols % 4 != 0 || ld_x % 4 != 0 || ld_y % 4 != 0) throw std::invalid_argument("launch_rms_norm_half: columns and strides must be multiples of 4");
    if (rows == 0) return;
    launch_kernel(rms_norm_half_kernel, dim3(static_cast<unsigned>(rows)), dim3(kNormThreads), 0, stream, "rms_norm_half_kernel launch", x, ld_x, w,
                  static_cast<__half*>(y_half), ld_y, cols, eps);
    count_launch();
}

void launch_fill_normal_half(void* dst_half, std::size_t count, std::uint64_t seed, float stddev, cudaStream_t stream) {
    if (count == 0) return;
    fill_normal_half_kernel<<<blocks_for(count, 256), 256, 0, stream>>>(static_cast<__half*>(dst_half), count, seed, stddev);
    check(cudaGetLastError(), "fill_normal_half_kernel launch");
    count_launch();
}
void launch_fill_normal_float(float* dst, std::size_t count, std::uint64_t seed, float stddev, cudaStream_t stream) {
    if (count == 0) return;
    fill_normal_float_kernel<<<blocks_for(count, 256), 256, 0, stream>>>(dst, count, seed, stddev);
    check(cudaGetLastError(), "fill_normal_float_kernel launch");
    count_launch();
}

void Trunk::shape_layer(std::uint32_t l) {
    const TrunkConfig& c = cfg_;
    Layer& L = layers_[l];
    L.attention = l % 4 == 3;
    L.mix_in_n = static_cast<std::uint32_t>(L.attention ? c.attn_q + 2 * c.attn_kv : c.dn_in);
    L.mix_out_k = L.attention ? c.attn_o : c.dn_v;
    L.band = L.attention ? 0u : c.dn_v_offset;
}

void* Trunk::alloc(std::size_t bytes) {
    void* p = nullptr;
    check(cudaMalloc(&p, bytes), "cudaMalloc(trunk)");
    allocations_.push_back(p);
    return p;
}

Trunk::Trunk(int device, const TrunkConfig& config, const Checkpoint* checkpoint) : cfg_(config), ctx_(device, 0) {
    ctx_.static_weights = true;  // the weights are in place (and the stream waited for) before the constructor returns

    TrunkConfig& c = cfg_;
    if (c.attn_o == 0) c.attn_o = c.attn_q;
    if (c.layers == 0 || c.hidden % 128 != 0 || c.intermediate % 128 != 0 || c.attn_q % 128 != 0 || c.attn_o % 128 != 0 || c.attn_kv % 8 != 0 ||
        c.dn_in % 8 != 0 || c.dn_v % 128 != 0 || c.dn_v_offset % 8 != 0 || c.dn_v_offset + c.dn_v > c.dn_in || c.attn_o > c.attn_q + 2 * c.attn_kv ||
        c.max_call_tokens == 0 || c.vocab == 0 ||
        (c.attn_heads != 0 && (c.attn_kv_heads == 0 || c.attn_heads % c.attn_kv_heads != 0 || (c.attn_head_dim != 128 && c.attn_head_dim != 256) ||
                               c.attn_q != 2 * c.attn_heads * c.attn_head_dim || c.attn_kv != c.attn_kv_heads * c.attn_head_dim ||
                               c.attn_o != c.attn_heads * c.attn_head_dim || c.attn_rotary_dims % 2 != 0 || c.attn_rotary_dims > c.attn_head_dim)) ||
        (c.dn_value_heads != 0 && (!deltanet_supports(deltanet_shape()) || c.dn_v != c.dn_value_heads * 128 ||
                                   c.dn_in != 2 * c.dn_key_heads * 128 + 2 * c.dn_value_heads * 128 + 2 * c.dn_value_heads)))
        throw std::invalid_argument("sepal_b200 trunk: widths must be multiples of 128 (k and v, the fused in-projection: of 8), the bands the "
                                    "out-projections read inside the in-projections, and layers, vocabulary and call size non-zero; with attn_heads set, attn_q = 2 heads "
                                    "head_dim, attn_kv = kv_heads head_dim, attn_o = heads head_dim, head_dim 128 or 256; with dn_value_heads set, dn_v = 128 value heads "
                                    "and dn_in = 256 key heads + 256 value heads + 2 value heads");
    check(cudaSetDevice(device), "cudaSetDevice");
    check(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
    for (auto& e : ev_) check(cudaEventCreate(&e), "cudaEventCreate");
    const std::size_t H = c.hidden, I = c.intermediate, T = c.max_call_tokens;
    const std::size_t attn_in = c.attn_q + 2 * static_cast<std::size_t>(c.attn_kv);
    p_width_ = static_cast<std::uint32_t>(attn_in > c.dn_in ? attn_in : c.dn_in);
    layers_.resize(c.layers);
    for (std::uint32_t l = 0; l < c.layers; ++l) shape_layer(l);
    if (checkpoint == nullptr)
        place_random();
    else if (checkpoint->metadata("format") == kSavedFormat)
        place_saved(*checkpoint);
    else
        place_checkpoint(*checkpoint);
    x_ = static_cast<float*>(alloc(T * H * 4));
    a1_ = alloc(T * H * 2);
    p_ = alloc(T * static_cast<std::size_t>(p_width_) * 2);
    a3_ = alloc(T * I * 2);
    if (real_attention()) q_ = alloc(T * static_cast<std::size_t>(c.attn_o) * 2);
    if (real_attention() || real_deltanet()) {
        const std::size_t widest = std::max<std::size_t>(real_attention() ? c.attn_o : 0, real_deltanet() ? c.dn_v : 0);
        a2_ = alloc(T * widest * 2);
    }
    if (real_deltanet()) {
        const DeltaNetShape d = deltanet_shape();
        dn_scratch_ = static_cast<float*>(alloc(deltanet_scratch_floats(d, T) * 4));
    }
    tokens_dev_ = static_cast<std::uint32_t*>(alloc(2 * T * 4));
    check(cudaMallocHost(reinterpret_cast<void**>(&tokens_pinned_), 2 * T * 4), "cudaMallocHost");
    check(cudaMallocHost(reinterpret_cast<void**>(&out_pinned_), 2 * kMaxCallRows * H * 4), "cudaMallocHost");
    for (cudaEvent_t& e : call_done_) check(cudaEventCreate(&e), "cudaEventCreate");
    check(cudaStreamSynchronize(stream_), "cudaStreamSynchronize");
}

Trunk::~Trunk() {
    (void)cudaSetDevice(ctx_.device);
    if (stream_ != nullptr) (void)cudaStreamSynchronize(stream_);
    for (void* p : allocations_) (void)cudaFree(p);
    for (Layer& L : layers_) {
        if (L.k_cache != nullptr) (void)cudaFree(L.k_cache);
        if (L.v_cache != nullptr) (void)cudaFree(L.v_cache);
        if (L.dn_states != nullptr) (void)cudaFree(L.dn_states);
        if (L.dn_tails != nullptr) (void)cudaFree(L.dn_tails);
    }
    for (cudaEvent_t e : call_done_)
        if (e != nullptr) (void)cudaEventDestroy(e);
    if (tokens_pinned_ != nullptr) (void)cudaFreeHost(tokens_pinned_);
    if (out_pinned_ != nullptr) (void)cudaFreeHost(out_pinned_);
    for (auto& e : ev_)
        if (e != nullptr) (void)cudaEventDestroy(e);
    if (stream_ != nullptr) (void)cudaStreamDestroy(stream_);
}

std::uint64_t Trunk::gemm_flops_per_token() const {
    std::uint64_t params = 0;
    for (const Layer& L : layers_)
        params += static_cast<std::uint64_t>(L.mix_in_n) * cfg_.hidden + static_cast<std::uint64_t>(cfg_.hidden) * L.mix_out_k +
                  3ull * cfg_.intermediate * cfg_.hidden;
    return 2 * params;
}

// The key/value caches of the attention layers hold `tokens` tokens (all requests of one run or score call, one range each). They
// grow, never shrink, and are zeroed when allocated: the attention kernel reads whole blocks and needs finite numbers everywhere.
void Trunk::reserve_cache(std::size_t tokens) {
    if (!real_attention() || tokens <= cache_tokens_) return;
    check(cudaStreamSynchronize(stream_), "cudaStreamSynchronize");
    const std::size_t bytes = tokens * static_cast<std::size_t>(cfg_.attn_kv) * 2;
    for (Layer& L : layers_) {
        if (!L.attention) continue;
        if (L.k_cache != nullptr) (void)cudaFree(L.k_cache);
        if (L.v_cache != nullptr) (void)cudaFree(L.v_cache);
        L.k_cache = L.v_cache = nullptr;
        check(cudaMalloc(&L.k_cache, bytes), "cudaMalloc(key cache)");
        check(cudaMalloc(&L.v_cache, bytes), "cudaMalloc(value cache)");
        check(cudaMemsetAsync(L.k_cache, 0, bytes, stream_), "cudaMemsetAsync");
        check(cudaMemsetAsync(L.v_cache, 0, bytes, stream_), "cudaMemsetAsync");
    }
    cache_tokens_ = tokens;
}

DeltaNetShape Trunk::deltanet_shape() const {
    DeltaNetShape d;
    d.key_heads = cfg_.dn_key_heads;
    d.value_heads = cfg_.dn_value_heads;
    d.head_dim = 128;
    d.conv_kernel = cfg_.dn_conv_kernel;
    d.eps = cfg_.eps;
    return d;
}

// The recurrent states and convolution tails of the DeltaNet layers, one slot for each request of a run or score call. They grow,
// never shrink; a request's first run starts from zero whatever its slot holds.
void Trunk::reserve_states(std::size_t slots) {
    if (!real_deltanet() || slots <= state_slots_) return;
    check(cudaStreamSynchronize(stream_), "cudaStreamSynchronize");
    const DeltaNetShape d = deltanet_shape();
    const std::size_t state_bytes = slots * d.value_heads * 128 * 128 * 4;
    const std::size_t tail_bytes = slots * std::max<std::size_t>(d.conv_kernel - 1, 1) * d.conv_dim() * 4;
    for (Layer& L : layers_) {
        if (L.attention) continue;
        if (L.dn_states != nullptr) (void)cudaFree(L.dn_states);
        if (L.dn_tails != nullptr) (void)cudaFree(L.dn_tails);
        L.dn_states = L.dn_tails = nullptr;
        check(cudaMalloc(reinterpret_cast<void**>(&L.dn_states), state_bytes), "cudaMalloc(DeltaNet states)");
        check(cudaMalloc(reinterpret_cast<void**>(&L.dn_tails), tail_bytes), "cudaMalloc(DeltaNet tails)");
    }
    state_slots_ = slots;
}

void Trunk::forward_call(const std::uint32_t* tokens_dev, std::size_t rows, const std::vector<AttentionRow>& runs, const std::vector<DeltaNetRow>& dn_runs) {
    const TrunkConfig& c = cfg_;
    const std::size_t H = c.hidden, I = c.intermediate;
    if (layers_.empty()) {
        launch_embed(embedding_, tokens_dev, x_, rows, H, c.vocab, stream_);
        return;
    }
    AttentionShape shape;
    shape.heads = c.attn_heads;
    shape.kv_heads = c.attn_kv_heads;
    shape.head_dim = c.attn_head_dim;
    shape.rotary_dims = c.attn_rotary_dims;
    shape.rope_theta = c.rope_theta;
    shape.eps = c.eps;
    launch_embed_rms_norm_half(embedding_, tokens_dev, x_, layers_.front().norm_in, a1_, H, rows, H, c.vocab, c.eps, stream_);
    for (const Layer& L : layers_) {
        if (&L != &layers_.front()) launch_rms_norm_half(x_, H, L.norm_in, a1_, H, rows, H, c.eps, stream_);
        launch_gemm_f16(ctx_, a1_, H, L.mix_in, H, p_, p_width_, true, rows, L.mix_in_n, H, Epilogue::Store, -1, stream_);
        if (L.attention && real_attention()) {
            // [q + gate; k; v] bands of p -> normed, rotated q; keys and values into the cache; attention times the gate -> a2 -> o_proj
            const __half* pq = static_cast<const __half*>(p_);
            const Band q_gate{pq, p_width_, true}, k{pq + c.attn_q, p_width_, true}, v{pq + c.attn_q + c.attn_kv, p_width_, true};
            launch_attention_prepare(ctx_, shape, runs.data(), runs.size(), q_gate, k, v, L.q_norm, L.k_norm, q_, c.attn_o, L.k_cache, L.v_cache, cache_tokens_, stream_);
            launch_attention(ctx_, shape, runs.data(), runs.size(), rows, q_, c.attn_o, L.k_cache, L.v_cache, cache_tokens_, q_gate, a2_, c.attn_o, stream_);
            launch_gemm_f16(ctx_, a2_, c.attn_o, L.mix_out, L.mix_out_k, x_, H, false, rows, H, L.mix_out_k, Epilogue::Add, -1, stream_);
        } else if (!L.attention && real_deltanet()) {
            // [qkv; z; b; a] bands of p -> the DeltaNet core -> a2 -> out_proj
            const DeltaNetShape d = deltanet_shape();
            const __half* pm = static_cast<const __half*>(p_);
            const Band mixed{pm, p_width_, true}, z{pm + d.conv_dim(), p_width_, true}, b{pm + d.conv_dim() + d.value_dim(), p_width_, true},
                a{pm + d.conv_dim() + d.value_dim() + d.value_heads, p_width_, true};
            const DeltaNetScratch sc = deltanet_scratch(dn_scratch_, d, rows);
            launch_deltanet(ctx_, d, dn_runs.data(), dn_runs.size(), mixed, z, b, a, DeltaNetWeights{L.dn_conv, L.dn_a_log, L.dn_dt_bias, L.dn_norm}, sc, L.dn_states,
                            L.dn_tails, state_slots_, a2_, c.dn_v, stream_);
            launch_gemm_f16(ctx_, a2_, c.dn_v, L.mix_out, L.mix_out_k, x_, H, false, rows, H, L.mix_out_k, Epilogue::Add, -1, stream_);
        } else {
            const __half* band = static_cast<const __half*>(p_) + L.band;
            launch_gemm_f16(ctx_, band, p_width_, L.mix_out, L.mix_out_k, x_, H, false, rows, H, L.mix_out_k, Epilogue::Add, -1, stream_);
        }
        launch_rms_norm_half(x_, H, L.norm_post, a1_, H, rows, H, c.eps, stream_);
        if (c.mlp_int8 == 0) {
            launch_gemm_f16(ctx_, a1_, H, L.gate_up, H, a3_, I, true, rows, 2 * I, H, Epilogue::SwiGLU, -1, stream_);
            launch_gemm_f16(ctx_, a3_, I, L.down, I, x_, H, false, rows, H, I, Epilogue::Add, -1, stream_);
        } else {
            launch_gemm_w8g(ctx_, a1_, H, L.gate_up_q, a3_, I, true, rows, 2 * I, H, Epilogue::SwiGLU, -1, stream_);
            launch_gemm_w8g(ctx_, a3_, I, L.down_q, x_, H, false, rows, H, I, Epilogue::Add, -1, stream_);
        }
    }
}

void Trunk::run(const std::uint32_t* tokens, std::size_t n, float* last_hidden, float* all_hidden, double* times_ms) {
    if (n == 0) throw std::invalid_argument("sepal_b200 trunk: a request needs at least one token");
    if (tokens == nullptr || last_hidden == nullptr) throw std::invalid_argument("sepal_b200 trunk: null pointer");
    for (std::size_t i = 0; i < n; ++i)
        if (tokens[i] >= cfg_.vocab) throw std::invalid_argument("sepal_b200 trunk: token id " + std::to_string(tokens[i]) + " is outside the vocabulary");
    check(cudaSetDevice(ctx_.device), "cudaSetDevice");
    const std::size_t H = cfg_.hidden, T = cfg_.max_call_tokens;
    reserve_cache(n);
    reserve_states(1);
    check(cudaEventRecord(ev_[0], stream_), "cudaEventRecord");
    for (std::size_t start = 0; start < n; start += T) {
        const std::size_t rows = n - start < T ? n - start : T;
        if (start != 0) check(cudaStreamSynchronize(stream_), "cudaStreamSynchronize");  // the pinned token buffer is reused
        std::memcpy(tokens_pinned_, tokens + start, rows * 4);
        check(cudaMemcpyAsync(tokens_dev_, tokens_pinned_, rows * 4, cudaMemcpyHostToDevice, stream_), "cudaMemcpyAsync(tokens)");
        // one run: the request's tokens start .. start + rows, its cache range starting at 0, `start` tokens already in it
        forward_call(tokens_dev_, rows, {AttentionRow{0u, static_cast<std::uint32_t>(rows), 0u, static_cast<std::uint32_t>(start)}},
                     {DeltaNetRow{0u, static_cast<std::uint32_t>(rows), 0u, start == 0 ? 1u : 0u}});
        if (all_hidden != nullptr)
            check(cudaMemcpyAsync(all_hidden + start * H, x_, rows * H * 4, cudaMemcpyDeviceToHost, stream_), "cudaMemcpyAsync(hidden)");
        if (start + rows == n)
            check(cudaMemcpyAsync(out_pinned_, x_ + (rows - 1) * H, H * 4, cudaMemcpyDeviceToHost, stream_), "cudaMemcpyAsync(last hidden)");
    }
    check(cudaEventRecord(ev_[1], stream_), "cudaEventRecord");
    const int status = ctx_.read_status(stream_);  // waits for the stream
    if (status != 0) throw std::runtime_error("sepal_b200 trunk: a kernel gave up waiting (status " + std::to_string(status) + ")");
    std::memcpy(last_hidden, out_pinned_, H * 4);
    if (times_ms != nullptr) {
        float ms = 0.0f;
        check(cudaEventElapsedTime(&ms, ev_[0], ev_[1]), "cudaEventElapsedTime");
        times_ms[0] = ms;
        times_ms[1] = 0.0;
    }
}

void Trunk::score(std::size_t n_requests, const std::uint32_t* tokens, const std::uint64_t* offsets, float* last_hidden, double* times_s) {
    if (n_requests == 0) return;
    if (tokens == nullptr || offsets == nullptr || last_hidden == nullptr) throw std::invalid_argument("sepal_b200 trunk: null pointer");
    const std::size_t H = cfg_.hidden, C = cfg_.max_call_tokens;
    for (std::size_t r = 0; r < n_requests; ++r) {
        if (offsets[r + 1] <= offsets[r]) throw std::invalid_argument("sepal_b200 trunk: request " + std::to_string(r) + " is empty or the offsets decrease");
        for (std::uint64_t i = offsets[r]; i < offsets[r + 1]; ++i)
            if (tokens[i] >= cfg_.vocab) throw std::invalid_argument("sepal_b200 trunk: token id " + std::to_string(tokens[i]) + " is outside the vocabulary");
    }
    // Segments in the order of the requests; a call takes segments until the next one does not fit.
    struct Segment {
        std::size_t request, begin, end;
        bool last;  // the request ends with this segment
    };
    std::vector<Segment> segments;
    for (std::size_t r = 0; r < n_requests; ++r) {
        std::size_t at = offsets[r];
        const std::size_t end = offsets[r + 1];
        while (end - at > C) {
            segments.push_back({r, at, at + C, false});
            at += C;
        }
        segments.push_back({r, at, end, true});
    }
    check(cudaSetDevice(ctx_.device), "cudaSetDevice");
    if (offsets[n_requests] > 0xFFFFFFFFull) throw std::invalid_argument("sepal_b200 trunk: more than 2^32 tokens in one call");
    reserve_cache(offsets[n_requests]);
    reserve_states(n_requests);
    struct Call {
        std::size_t first, count;  // its segments
    };
    std::vector<Call> calls;
    for (std::size_t i = 0, in_call = 0; i < segments.size(); ++i) {
        const std::size_t n = segments[i].end - segments[i].begin;
        if (calls.empty() || in_call + n > C || calls.back().count >= kMaxCallRows) {
            calls.push_back({i, 0});
            in_call = 0;
        }
        ++calls.back().count;
        in_call += n;
    }
    std::vector<cudaEvent_t> stamps;  // one per call, for the completion times
    const auto drop_stamps = [&] {
        for (cudaEvent_t e : stamps) (void)cudaEventDestroy(e);
    };
    try {
        check(cudaEventRecord(ev_[0], stream_), "cudaEventRecord");
        // Results of call c land in half c % 2 of the pinned output; they are copied out when call c + 1 has been enqueued.
        const auto collect = [&](std::size_t c) {
            check(cudaEventSynchronize(call_done_[c % 2]), "cudaEventSynchronize");
            std::size_t slot = 0;
            for (std::size_t i = calls[c].first; i < calls[c].first + calls[c].count; ++i)
                if (segments[i].last) std::memcpy(last_hidden + segments[i].request * H, out_pinned_ + ((c % 2) * kMaxCallRows + slot++) * H, H * 4);
        };
        for (std::size_t c = 0; c < calls.size(); ++c) {
            const std::size_t half = c % 2;
            if (c >= 2) collect(c - 2);  // also: the buffers of this half are free again
            std::uint32_t* pinned = tokens_pinned_ + half * C;
            std::uint32_t* dev = tokens_dev_ + half * C;
            std::size_t rows = 0;
            for (std::size_t i = calls[c].first; i < calls[c].first + calls[c].count; ++i) {
                const std::size_t n = segments[i].end - segments[i].begin;
                std::memcpy(pinned + rows, tokens + segments[i].begin, n * 4);
                rows += n;
            }
            check(cudaMemcpyAsync(dev, pinned, rows * 4, cudaMemcpyHostToDevice, stream_), "cudaMemcpyAsync(tokens)");
            // a request's cache range starts where its tokens start in the flat list; a segment continues what the request's earlier ones left
            std::vector<AttentionRow> runs;
            std::vector<DeltaNetRow> dn_runs;
            std::size_t at = 0;
            for (std::size_t i = calls[c].first; i < calls[c].first + calls[c].count; ++i) {
                const Segment& sg = segments[i];
                runs.push_back(AttentionRow{static_cast<std::uint32_t>(at), static_cast<std::uint32_t>(sg.end - sg.begin), static_cast<std::uint32_t>(offsets[sg.request]),
                                            static_cast<std::uint32_t>(sg.begin - offsets[sg.request])});
                dn_runs.push_back(DeltaNetRow{static_cast<std::uint32_t>(at), static_cast<std::uint32_t>(sg.end - sg.begin), static_cast<std::uint32_t>(sg.request),
                                              sg.begin == offsets[sg.request] ? 1u : 0u});
                at += sg.end - sg.begin;
            }
            forward_call(dev, rows, runs, dn_runs);
            std::size_t row = 0, slot = 0;
            for (std::size_t i = calls[c].first; i < calls[c].first + calls[c].count; ++i) {
                row += segments[i].end - segments[i].begin;
                if (segments[i].last)
                    check(cudaMemcpyAsync(out_pinned_ + (half * kMaxCallRows + slot++) * H, x_ + (row - 1) * H, H * 4, cudaMemcpyDeviceToHost, stream_),
                          "cudaMemcpyAsync(last hidden)");
            }
            check(cudaEventRecord(call_done_[half], stream_), "cudaEventRecord");
            if (times_s != nullptr) {
                cudaEvent_t e = nullptr;
                check(cudaEventCreate(&e), "cudaEventCreate");
                stamps.push_back(e);
                check(cudaEventRecord(e, stream_), "cudaEventRecord");
            }
        }
        if (calls.size() >= 2) collect(calls.size() - 2);
        collect(calls.size() - 1);
        const int status = ctx_.read_status(stream_);
        if (status != 0) throw std::runtime_error("sepal_b200 trunk: a kernel gave up waiting (status " + std::to_string(status) + ")");
        if (times_s != nullptr) {
            for (std::size_t c = 0; c < calls.size(); ++c) {
                float ms = 0.0f;
                check(cudaEventElapsedTime(&ms, ev_[0], stamps[c]), "cudaEventElapsedTime");
                for (std::size_t i = calls[c].first; i < calls[c].first + calls[c].count; ++i)
                    if (segments[i].last) times_s[segments[i].request] = ms * 1e-3;
            }
        }
    } catch (...) {
        (void)cudaStreamSynchronize(stream_);
        drop_stamps();
        throw;
    }
    drop_stamps();
}

std::size_t Trunk::weight(std::uint32_t layer, TrunkWeight which, void* host_out, std::size_t capacity) {
    const TrunkConfig& c = cfg_;
    const std::size_t H = c.hidden, I = c.intermediate;
    const void* src = nullptr;
    std::size_t bytes = 0;
    if (which == TrunkWeight::Embedding) {
        src = embedding_;
        bytes = static_cast<std::size_t>(c.vocab) * H * 2;
    } else {
        if (layer >= c.layers) throw std::invalid_argument("sepal_b200 trunk: no such layer");
        const Layer& L = layers_[layer];
        switch (which) {
        case TrunkWeight::NormIn: src = L.norm_in; bytes = H * 4; break;
        case TrunkWeight::NormPost: src = L.norm_post; bytes = H * 4; break;
        case TrunkWeight::MixIn: src = L.mix_in; bytes = static_cast<std::size_t>(L.mix_in_n) * H * 2; break;
        case TrunkWeight::MixOut: src = L.mix_out; bytes = H * static_cast<std::size_t>(L.mix_out_k) * 2; break;
        case TrunkWeight::GateUp: src = L.gate_up; bytes = 2 * I * H * (c.mlp_int8 ? 1 : 2); break;
        case TrunkWeight::Down: src = L.down; bytes = H * I * (c.mlp_int8 ? 1 : 2); break;
        case TrunkWeight::QNorm: src = L.q_norm; bytes = L.q_norm != nullptr ? static_cast<std::size_t>(c.attn_head_dim) * 4 : 0; break;
        case TrunkWeight::KNorm: src = L.k_norm; bytes = L.k_norm != nullptr ? static_cast<std::size_t>(c.attn_head_dim) * 4 : 0; break;
        case TrunkWeight::DnConv: src = L.dn_conv; bytes = L.dn_conv != nullptr ? static_cast<std::size_t>(deltanet_shape().conv_dim()) * c.dn_conv_kernel * 4 : 0; break;
        case TrunkWeight::DnALog: src = L.dn_a_log; bytes = L.dn_a_log != nullptr ? static_cast<std::size_t>(c.dn_value_heads) * 4 : 0; break;
        case TrunkWeight::DnDtBias: src = L.dn_dt_bias; bytes = L.dn_dt_bias != nullptr ? static_cast<std::size_t>(c.dn_value_heads) * 4 : 0; break;
        case TrunkWeight::DnNorm: src = L.dn_norm; bytes = L.dn_norm != nullptr ? 128 * 4 : 0; break;
        case TrunkWeight::GateUpScales: src = L.gate_up_scales; bytes = L.gate_up_scales != nullptr ? 2 * I * (H / kGroup) * 4 : 0; break;
        case TrunkWeight::DownScales: src = L.down_scales; bytes = L.down_scales != nullptr ? H * (I / kGroup) * 4 : 0; break;
        default: throw std::invalid_argument("sepal_b200 trunk: no such weight");
        }
    }
    if (host_out != nullptr) {
        if (capacity < bytes) throw std::length_error("sepal_b200 trunk: buffer too small: " + std::to_string(bytes) + " bytes needed");
        check(cudaSetDevice(ctx_.device), "cudaSetDevice");
        check(cudaMemcpy(host_out, src, bytes, cudaMemcpyDeviceToHost), "cudaMemcpy(weight)");
    }
    return bytes;
}

}  // namespace sepal::b200
