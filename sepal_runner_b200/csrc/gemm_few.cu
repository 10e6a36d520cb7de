// The trunk projection for few rows of X (a short request, the last tokens of a long one): Y = epilogue(X W^T) with up to 256 rows.
//
// With T rows a weight of two bytes is worth 2 T operations, so below about 250 rows (half that for int8 weights) the multiply is bound
// by reading W once. The kernels in gemm_tc.cu give a CTA 128 rows of X whatever T is and split N in wide tiles: a 7-row multiply by
// 6144 x 2560 weights ran on 24 or 48 CTAs with 40 k steps each, 17.9 us for 31 MB; here 7.8 us behind one like it (alone under the profiler
// 13 us, 30 % of the DRAM's throughput: a launch's start, its cluster's exchange and its end are the rest). Here
//   - the weights are the MMA's first operand (128 rows of W to a CTA) and the tokens its second (N = T rounded up to 16), so nothing is
//     computed for rows that are not there;
//   - the k range of a tile of W is cut over the CTAs of a cluster (`split`, up to eight), so that ceil(N / 128) split CTAs stream their
//     parts of W (every SM from about 2300 rows of W on; 64 CTAs at 1024), and the parts meet through distributed shared memory in the order of their ranges: no scratch in global memory, no
//     counters, the same bits every time;
//   - a CTA takes at most half of an SM up to 64 rows: with the weights static the next multiply's CTAs are resident and have
//     their first boxes of W requested while this one still drains.
//
//   warp 0      TMA producer: per stage a [128 x 64] box of W (int8: [128 x 128] bytes and the group's scales) and the X boxes
//   warp 1      MMA issuer (M 128, N up to 256, K 16); a stage's slot is only committed back when it is loaded again
//   warps 2..9  int8: converters (raw box -> binary16 weights in tensor memory, as in gemm_w8t_pair_kernel: two sets of four warps take
//               the scale groups in turn); then the epilogue: accumulator -> shared memory [token][row of W], the cluster's parts summed
//               in rank order by the CTA whose token it is (token mod split), stored or added in rows of 128 consecutive columns.
#include "gemm_few.hpp"

#include <atomic>
#include <cstdint>
#include <stdexcept>
#include <string>

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gemm_device.cuh"
#include "ptx.cuh"

namespace sepal::b200 {

void count_launch();

namespace {

constexpr unsigned kRows = 128;             // rows of W to a tile
constexpr unsigned kThreads = 320;
constexpr unsigned kMaxStages = 8;
constexpr unsigned kMaxABufs = 4;
constexpr unsigned kWBytes = kRows * 128;   // one box of W: 64 binary16 or 128 int8 values of k
constexpr unsigned kFullBars = 2 * kMaxStages;  // (see barriers_in_turn)
constexpr unsigned kBarriers = kFullBars + kMaxStages + 2 * kMaxABufs + 1;
constexpr unsigned kTailBytes = kBarriers * 8 + 64;
constexpr unsigned kSmemMax = 232448;
constexpr unsigned kSmemHalf = 112 * 1024;  // two CTAs to an SM, with what the system takes of its 228 KB

struct FewParams {
    void* y;
    unsigned long long ld_y;
    unsigned m, n;
    unsigned k_iters, split, n_tok, stages, a_bufs, tmem_cols;
    unsigned epilogue, y_half, vec_ok, early_w;
    int* status;
    const __half* scales_t;
    unsigned long long ld_st;
    const float* descale;
    const float* col_scale;
};

template <bool W8>
__host__ __device__ constexpr unsigned stage_bytes(unsigned n_tok) {
    return kWBytes + n_tok * 128 * (W8 ? 2 : 1);
}

// One token's four (SwiGLU: two) consecutive results of a lane.
template <int V>
__device__ __forceinline__ void store_results(const FewParams& p, unsigned token, unsigned col, unsigned n_out, const float (&v)[V]) {
    const bool add = p.epilogue == 1;
    const size_t at = static_cast<size_t>(token) * p.ld_y + col;
    if (p.vec_ok != 0 && col + V <= n_out) {
        if (p.y_half != 0) {
            __half2* out = reinterpret_cast<__half2*>(static_cast<__half*>(p.y) + at);
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                float a = v[2 * i], b = v[2 * i + 1];
                if (add) {
                    const float2 old = __half22float2(out[i]);
                    a = __fadd_rn(old.x, a), b = __fadd_rn(old.y, b);
                }
                out[i] = __floats2half2_rn(a, b);
            }
        } else if constexpr (V == 4) {
            float4* out = reinterpret_cast<float4*>(static_cast<float*>(p.y) + at);
            float4 r = make_float4(v[0], v[1], v[2], v[3]);
            if (add) {
                const float4 old = *out;
                r = make_float4(__fadd_rn(old.x, r.x), __fadd_rn(old.y, r.y), __fadd_rn(old.z, r.z), __fadd_rn(old.w, r.w));
            }
            *out = r;
        } else {
            *reinterpret_cast<float2*>(static_cast<float*>(p.y) + at) = make_float2(v[0], v[1]);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
        if (col + i >= n_out) break;
        if (p.y_half != 0) {
            __half* out = static_cast<__half*>(p.y) + at + i;
            *out = __float2half_rn(add ? __fadd_rn(__half2float(*out), v[i]) : v[i]);
        } else {
            float* out = static_cast<float*>(p.y) + at + i;
            *out = add ? __fadd_rn(*out, v[i]) : v[i];
        }
    }
}

template <bool W8>
__global__ void __launch_bounds__(kThreads, 2)
gemm_few_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const FewParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = ptx::smem_addr(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (base - raw_addr);
    const unsigned n_tok = p.n_tok, x_box = n_tok * 128, stage = stage_bytes<W8>(n_tok);
    const int stages = static_cast<int>(p.stages);
    const unsigned scale_off = p.stages * stage;  // layout: ring (the parts of the sum take its place at the end) | scales | barriers
    uint8_t* const tail = smem + scale_off + (W8 ? p.stages * 256 : 0);
    const uint32_t bars = ptx::smem_addr(tail);
    const auto full_bar = [&](int s) { return bars + 8u * s; };
    const auto empty_bar = [&](int s) { return bars + 8u * (kFullBars + s); };
    const auto a_full_bar = [&](int s) { return bars + 8u * (kFullBars + kMaxStages + s); };
    const auto a_empty_bar = [&](int s) { return bars + 8u * (kFullBars + kMaxStages + kMaxABufs + s); };
    const uint32_t acc_bar = bars + 8u * (kBarriers - 1);
    unsigned* const words = reinterpret_cast<unsigned*>(tail + kBarriers * 8);
    // Step i arrives on full barrier i % fulls: the two sets of converters take the ring's slots in turn. (What they wait for before they
    // reuse a weight buffer, the one issuing thread's commits, completes in order: a set that has seen the commit two steps back has seen
    // every phase before.)
    const int fulls = static_cast<int>(W8 ? barriers_in_turn(p.stages) : p.stages);
    volatile unsigned* const abort_flag = words + 1;

    const unsigned warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const unsigned rank = blockIdx.x % p.split, row0 = blockIdx.x / p.split * kRows;
    const int k0 = static_cast<int>(p.k_iters * rank / p.split), k1 = static_cast<int>(p.k_iters * (rank + 1) / p.split);
    const int iters = k1 - k0;
    const int a_bufs = static_cast<int>(p.a_bufs);

    if (threadIdx.x == 0) {
        for (int s = 0; s < fulls; ++s) ptx::mbar_init(full_bar(s), 1);
        for (int s = 0; s < stages; ++s) ptx::mbar_init(empty_bar(s), W8 ? 5 : 1);  // the MMAs' commit; int8: and the four converter warps that read the raw box
        for (int s = 0; s < a_bufs; ++s) {
            ptx::mbar_init(a_full_bar(s), 4);
            ptx::mbar_init(a_empty_bar(s), 1);
        }
        ptx::mbar_init(acc_bar, 1);
        words[1] = 0;
        ptx::fence_barrier_init();
        ptx::tma_prefetch_descriptor(&map_x);
        ptx::tma_prefetch_descriptor(&map_w);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(words), p.tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = words[0];
    const uint32_t a_cols = tmem + n_tok;  // the weight buffers (64 columns a scale group) follow the accumulator
    ptx::grid_launch_dependents();

    const auto load_w = [&](int i, int s, int f) {
        ptx::mbar_arrive_expect_tx(full_bar(f), stage + (W8 ? 256u : 0u));
        ptx::tma_load_2d(base + s * stage, &map_w, full_bar(f), (k0 + i) * (W8 ? 128 : 64), static_cast<int>(row0));
        if constexpr (W8) ptx::bulk_load(base + scale_off + s * 256, p.scales_t + static_cast<size_t>(k0 + i) * p.ld_st + row0, 256, full_bar(f));
    };
    const int early = p.early_w != 0 ? min(stages, iters) : 0;
    if (warp == 0 && lane == 0) {
        for (int i = 0; i < early; ++i) load_w(i, i, i);
    }
    ptx::grid_dependency_wait();

    if (warp == 0) {
        if (lane == 0) {
            int s = 0, f = 0;
            unsigned phase = 1;
            for (int i = 0; i < iters; ++i) {
                if (i >= stages && !wait_barrier(empty_bar(s), phase, abort_flag, p.status, kStatusProducerEmpty)) {
                    grace_for_copies_in_flight();
                    break;
                }
                if (i >= early) load_w(i, s, f);
                if constexpr (W8) {
                    ptx::tma_load_2d(base + s * stage + kWBytes, &map_x, full_bar(f), (k0 + i) * 128, 0);
                    ptx::tma_load_2d(base + s * stage + kWBytes + x_box, &map_x, full_bar(f), (k0 + i) * 128 + 64, 0);
                } else {
                    ptx::tma_load_2d(base + s * stage + kWBytes, &map_x, full_bar(f), (k0 + i) * 64, 0);
                }
                if (++f == fulls) f = 0;
                if (++s == stages) s = 0, phase ^= 1u;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = ptx::instr_desc_f16_f32acc(kRows, n_tok);
            int s = 0, f = 0, ab = 0;
            unsigned phase = 0, a_phase = 0;
            bool ok = true;
            for (int i = 0; i < iters; ++i) {
                if ((W8 && !wait_barrier(a_full_bar(ab), a_phase, abort_flag, p.status, kStatusMmaConvFull)) ||
                    !wait_barrier(full_bar(f), phase, abort_flag, p.status, kStatusMmaFull)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint64_t dx = ptx::smem_desc_k_major_sw128(base + s * stage + kWBytes);
                if constexpr (W8) {
                    const uint32_t a = a_cols + static_cast<uint32_t>(ab) * 64u;
#pragma unroll
                    for (unsigned j = 0; j < 8; ++j)
                        ptx::mma_f16_ts(tmem, a + 8 * j, dx + (j / 4) * (x_box >> 4) + 2 * (j % 4), idesc, i != 0 || j != 0 ? 1u : 0u);
                } else {
                    const uint64_t dw = ptx::smem_desc_k_major_sw128(base + s * stage);
#pragma unroll
                    for (unsigned j = 0; j < 4; ++j) ptx::mma_f16_ss(tmem, dw + 2 * j, dx + 2 * j, idesc, i != 0 || j != 0 ? 1u : 0u);
                }
                // a commit holds the issuing thread until its MMAs have drained: only where somebody waits for the slot
                if (i + stages < iters) ptx::mma_commit(empty_bar(s));
                if (W8 && i + a_bufs < iters) ptx::mma_commit(a_empty_bar(ab));
                if (++s == stages) s = 0;
                if (++f == fulls) f = 0, phase ^= 1u;
                if (W8 && ++ab == a_bufs) ab = 0, a_phase ^= 1u;
            }
            if (ok) ptx::mma_commit(acc_bar);
        }
        __syncwarp();
    } else {
        const unsigned worker = warp - 2, quarter = warp % 4, set = worker / 4;
        const unsigned row = quarter * 32 + lane;
        if constexpr (W8) {
            const unsigned sw = row & 7u;
            const __half2 offset = __half2half2(__ushort_as_half(0x6480));  // 1152
            const bool in_n = row0 + row < p.n;  // rows past N multiply by zero
            for (int i = static_cast<int>(set); i < iters; i += 2) {
                const int s = i % stages, ab = i % a_bufs;
                bool got = wait_barrier(full_bar(i % fulls), (i / fulls) & 1, abort_flag, p.status, kStatusConvFull);
                if (got && i >= a_bufs) got = wait_barrier(a_empty_bar(ab), (i / a_bufs - 1) & 1, abort_flag, p.status, kStatusConvEmpty);
                if (!__all_sync(0xFFFFFFFFu, got)) break;
                ptx::tc_fence_after_sync();
                const uint8_t* raw = smem + s * stage + row * 128;
                const __half2 sc = __half2half2(in_n ? reinterpret_cast<const __half*>(smem + scale_off + s * 256)[row] : __ushort_as_half(0));
#pragma unroll
                for (unsigned part = 0; part < 4; ++part) {
                    uint32_t packed[16];
#pragma unroll
                    for (unsigned c = 0; c < 2; ++c) {
                        const uint4 q = *reinterpret_cast<const uint4*>(raw + (((2 * part + c) ^ sw) << 4));
                        const unsigned w[4] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u, q.z ^ 0x80808080u, q.w ^ 0x80808080u};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            unsigned lo = __byte_perm(w[e], 0x64646464u, 0x5140);  // bytes 0, 1 -> two binary16 numbers 1024 + byte
                            unsigned hi = __byte_perm(w[e], 0x64646464u, 0x5342);  // bytes 2, 3
                            const __half2 a = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&lo), offset), sc);
                            const __half2 b = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&hi), offset), sc);
                            packed[8 * c + 2 * e] = *reinterpret_cast<const unsigned*>(&a);
                            packed[8 * c + 2 * e + 1] = *reinterpret_cast<const unsigned*>(&b);
                        }
                    }
                    ptx::tmem_st_32x16(a_cols + ((quarter * 32u) << 16) + static_cast<uint32_t>(ab) * 64u + part * 16, packed);
                }
                __syncwarp();
                if (lane == 0 && i + stages < iters) ptx::mbar_arrive(empty_bar(s));
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(a_full_bar(ab));
            }
        }
        // the accumulator into shared memory, [token][row of W]: the ring is idle once the last MMA has drained
        const bool arrived = wait_barrier(acc_bar, 0, abort_flag, p.status, kStatusEpilogueAccFull);
        if (__all_sync(0xFFFFFFFFu, arrived)) {
            ptx::tc_fence_after_sync();
            float* const mine = reinterpret_cast<float*>(smem) + row;
            for (unsigned c = 16 * set; c < p.m; c += 32) {
                uint32_t v[16];
                ptx::tmem_ld_32x16(tmem + ((quarter * 32u) << 16) + c, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (unsigned j = 0; j < 16; ++j) mine[(c + j) * kRows] = __uint_as_float(v[j]);
            }
            ptx::tc_fence_before_sync();
        }
    }
    __syncwarp();
    ptx::cluster_sync();  // every part of the cluster's sums is in its CTA's shared memory
    if (warp >= 2 && *abort_flag == 0) {
        const unsigned worker = warp - 2;
        const bool gated = p.epilogue == 2;
        const unsigned n_out = gated ? p.n / 2 : p.n;
        // plain: lane l has columns 4 l .. 4 l + 3 of the tile; SwiGLU: gate rows 2 l, 2 l + 1 and the up rows 64 further on
        const unsigned at = gated ? 2 * lane : 4 * lane;
        const unsigned col = gated ? row0 / 2 + at : row0 + at;
        const float descale = W8 ? __ldg(p.descale) : 1.0f;
        float second[4] = {1.0f, 1.0f, 1.0f, 1.0f};
        if (W8 && p.col_scale != nullptr) {
#pragma unroll
            for (unsigned i = 0; i < 4; ++i) {
                const unsigned n = row0 + (gated ? at + i % 2 + (i / 2) * 64 : at + i);
                if (n < p.n) second[i] = __ldg(p.col_scale + n);
            }
        }
        for (unsigned token = rank + p.split * worker; token < p.m; token += 8 * p.split) {
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const uint32_t here = base + token * (kRows * 4) + at * 4;
            float4 part[8];
#pragma unroll
            for (unsigned r = 0; r < 8; ++r) {
                if (r < p.split) {
                    const uint32_t there = ptx::map_to_cta(here, r);
                    if (gated) {
                        const float2 g = ptx::ld_cluster_f32x2(there), u = ptx::ld_cluster_f32x2(there + 256);
                        part[r] = make_float4(g.x, g.y, u.x, u.y);
                    } else {
                        part[r] = ptx::ld_cluster_f32x4(there);
                    }
                }
            }
#pragma unroll
            for (unsigned r = 0; r < 8; ++r) {
                if (r < p.split) {
                    v[0] = __fadd_rn(v[0], part[r].x), v[1] = __fadd_rn(v[1], part[r].y);
                    v[2] = __fadd_rn(v[2], part[r].z), v[3] = __fadd_rn(v[3], part[r].w);
                }
            }
            if (W8) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = p.col_scale != nullptr ? __fmul_rn(__fmul_rn(v[i], descale), second[i]) : __fmul_rn(v[i], descale);
            }
            if (gated) {
                const float r[2] = {swiglu(v[0], v[2]), swiglu(v[1], v[3])};
                store_results(p, token, col, n_out, r);
            } else {
                store_results(p, token, col, n_out, v);
            }
        }
    }
    __syncwarp();
    ptx::cluster_sync();  // nobody reads this CTA's part any more
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, p.tmem_cols);
    }
}

void configure(const Context& ctx) {
    static std::atomic<bool> configured[64] = {};  // per device; every writer sets the same attributes
    if (ctx.device < 64 && configured[ctx.device].load(std::memory_order_relaxed)) return;
    check(cudaFuncSetAttribute(gemm_few_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax), "cudaFuncSetAttribute");
    check(cudaFuncSetAttribute(gemm_few_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax), "cudaFuncSetAttribute");
    if (ctx.device < 64) configured[ctx.device].store(true, std::memory_order_relaxed);
}

// Clusters of `split` CTAs that are resident at once with one CTA to an SM on a GPU of `sm_count` SMs: a GPC's SMs left over by clusters
// that do not divide them stay empty, so that 48 clusters of three do not fit where 144 lone CTAs would. These are what
// cudaOccupancyMaxActiveClusters says of five B200s of 148 SMs, all alike, in proportion for other counts. A function of the SM count, and
// not the driver's answer for the GPU at hand: the parts of k decide the bits of the result, which must be the same on every GPU of a
// kind. (Where fewer fit, the last clusters make a second wave.) With two CTAs to an SM twice as many are resident at least.
unsigned resident_clusters(unsigned sm_count, unsigned split) {
    constexpr unsigned of_148[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    return of_148[split] * sm_count / 148;
}

template <bool W8>
void launch(const Context& ctx, const FewCall& c, FewSchedule sched, cudaStream_t stream) {
    FewParams p{};
    p.y = c.y;
    p.ld_y = c.ld_y;
    p.m = static_cast<unsigned>(c.t);
    p.n = static_cast<unsigned>(c.n);
    p.n_tok = (p.m + 15) / 16 * 16;
    const unsigned per_iter = W8 ? 128 : 64;
    p.k_iters = static_cast<unsigned>((c.k + per_iter - 1) / per_iter);
    p.split = sched.split < p.k_iters ? sched.split : p.k_iters;
    // tensor memory: two CTAs to an SM get 256 columns each, so that neither ever waits for the other's
    p.tmem_cols = sched.slots == 2 ? 256u : 512u;
    p.a_bufs = W8 ? (p.tmem_cols - p.n_tok) / 64 : 0;
    if (p.a_bufs > kMaxABufs) p.a_bufs = kMaxABufs;
    const unsigned room = (sched.slots == 2 ? kSmemHalf : kSmemMax) - 1024 - kTailBytes;
    p.stages = room / (stage_bytes<W8>(p.n_tok) + (W8 ? 256 : 0));
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    // (always more than a third of an SM, or half of it when one CTA is to have it alone: the tensor memory above is only enough for as
    // many CTAs as the shared memory lets in)
    p.epilogue = static_cast<unsigned>(c.epilogue);
    p.y_half = c.y_half ? 1u : 0u;
    p.vec_ok = (reinterpret_cast<std::uintptr_t>(c.y) % 16 == 0 && (c.ld_y * (c.y_half ? 2 : 4)) % 16 == 0) ? 1u : 0u;
    p.early_w = ctx.static_weights ? 1u : 0u;
    p.status = ctx.status;
    p.scales_t = static_cast<const __half*>(c.scales_t);
    p.ld_st = c.ld_st;
    p.descale = c.descale;
    p.col_scale = c.col_scale;
    const unsigned smem = 1024 + p.stages * (stage_bytes<W8>(p.n_tok) + (W8 ? 256 : 0)) + kTailBytes;
    const CUtensorMap map_x = make_tensor_map_2d(ctx, c.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, c.t, c.k, c.ld_x, p.n_tok, 64, true);
    const CUtensorMap map_w = W8 ? make_tensor_map_2d(ctx, c.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.n, c.k, c.ld_w, kRows, 128, true)
                                 : make_tensor_map_2d(ctx, c.w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, c.n, c.k, c.ld_w, kRows, 64, true);
    configure(ctx);
    const unsigned tiles = static_cast<unsigned>((c.n + kRows - 1) / kRows);
    launch_cluster_kernel(gemm_few_kernel<W8>, p.split, dim3(tiles * p.split), dim3(kThreads), smem, stream, "gemm_few_kernel launch", map_x, map_w, p);
    count_launch();
}

}  // namespace

// Up to 64 rows: two CTAs to an SM, and as many parts of k as leave all clusters resident at once (a second wave, or a cluster that
// waits for a GPC with room, costs more than the shorter k loop gives: 6144 x 2560, 7 rows: five parts 7.8 us, six 12.2). Up to 128 rows
// a stage of the half-SM form is down to three or two slots, so a CTA with an SM to itself can be the better one: a k step costs about
// 0.31 us there and 0.42 us, times the CTAs an SM has to feed, with two to an SM (fitted to twelve shapes of up to 148 tiles). Not with
// more tiles than SMs: a second lone CTA starts when the first has ended, where two side by side hide one another's starts and ends (128
// rows: 36864 x 1024 28.3 us alone, 21.9 as two; 65536 x 1024 54.0 and 40.1; 151936 x 2560 193 and 168). From 129 rows up one CTA to an SM.
FewSchedule few_schedule(unsigned sm_count, std::size_t t, std::size_t n, std::size_t k, bool int8) {
    const std::size_t tiles = (n + kRows - 1) / kRows, iters = (k + (int8 ? 127 : 63)) / (int8 ? 128 : 64);
    FewSchedule best;
    double best_cost = 0.0;
    const unsigned most = t <= 128 ? 2u : 1u, least = t <= 64 || (t <= 128 && tiles > sm_count) ? 2u : 1u;
    for (unsigned slots = most; slots >= least; --slots) {
        FewSchedule s;
        s.slots = slots;
        for (unsigned split = 2; split <= 8 && split <= iters; ++split)
            if (tiles <= slots * resident_clusters(sm_count, split)) s.split = split;
        const double steps = static_cast<double>((iters + s.split - 1) / s.split), load = static_cast<double>(tiles * s.split) / sm_count;
        const double cost = steps * (slots == 2 ? 0.42 * (load > 1.0 ? load : 1.0) : 0.31);
        if (best_cost == 0.0 || cost < best_cost) best = s, best_cost = cost;
    }
    return best;
}

void launch_gemm_few(const Context& ctx, const FewCall& call, FewSchedule schedule, cudaStream_t stream) {
    if (call.t == 0 || call.t > kFewMaxRows || schedule.split == 0 || schedule.split > 8 || schedule.slots == 0 || schedule.slots > 2 ||
        (schedule.slots == 2 && call.t > 128))
        throw std::invalid_argument("sepal_b200: the few-rows multiply takes 1 to 256 rows (two CTAs to an SM: 128), its k in 1 to 8 parts");
    if (call.y == nullptr) throw std::invalid_argument("sepal_b200: null output");
    if (call.n > 0x7FFFFFFFu || call.k > 0x7FFFFFFFu) throw std::invalid_argument("sepal_b200: dimension beyond 2^31");
    if (call.int8)
        launch<true>(ctx, call, schedule, stream);
    else
        launch<false>(ctx, call, schedule, stream);
}

}  // namespace sepal::b200
