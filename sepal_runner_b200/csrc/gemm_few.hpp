// The multiply for few rows of X (gemm_few.cu): what the launchers in gemm_tc.cu hand over.
#pragma once

#include <cstddef>

#include "gemm.hpp"

namespace sepal::b200 {

struct FewCall {
    const void* x = nullptr;
    std::size_t ld_x = 0;
    const void* w = nullptr;  // binary16 [N, ld_w], or int8 [N, ld_w] with scales_t
    std::size_t ld_w = 0;
    bool int8 = false;
    const void* scales_t = nullptr;  // int8: as W8gMatrix; ld_st 0: one row of ones serves every group
    std::size_t ld_st = 0;
    const float* descale = nullptr;
    const float* col_scale = nullptr;
    void* y = nullptr;
    std::size_t ld_y = 0;
    bool y_half = true;
    std::size_t t = 0, n = 0, k = 0;
    Epilogue epilogue = Epilogue::Store;
};

inline constexpr std::size_t kFewMaxRows = 256;  // rows of X the kernel takes (the N of one MMA)
inline constexpr int kFewConfig = 1024;          // config: kFewConfig + split (1 .. 8), + 16 for one CTA to an SM

/// CTAs of a cluster that share a tile's k (1 .. 8), and CTAs to an SM (1 or 2), as the automatic schedule has them for a [t x k] by [n x k]
/// multiply on a GPU of `sm_count` SMs. Host arithmetic only.
struct FewSchedule {
    unsigned split = 1, slots = 1;
};
FewSchedule few_schedule(unsigned sm_count, std::size_t t, std::size_t n, std::size_t k, bool int8);

/// Enqueues the multiply. The caller has checked shapes, strides and alignments as for every other kernel (int8: also that scales_t has
/// 16-byte aligned rows padded to a multiple of 128 of N).
void launch_gemm_few(const Context& ctx, const FewCall& call, FewSchedule schedule, cudaStream_t stream);

}  // namespace sepal::b200
