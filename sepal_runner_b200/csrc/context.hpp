// Per-device state shared by every launcher: the properties of the device, the scratch memory of the split-k schedule and the
// device word a kernel writes when one of its bounded waits gives up. Created once (sepal_b200_open); a launch allocates nothing.
#pragma once

#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <utility>

#include <cuda.h>
#include <cuda_runtime.h>

namespace sepal::b200 {

inline void check(cudaError_t status, const char* call) {
    if (status != cudaSuccess) {
        (void)cudaGetLastError();  // reported by the exception: not left for the next call's check
        throw std::runtime_error(std::string(call) + " failed: " + cudaGetErrorString(status));
    }
}

using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

/// Scratch a split-k launch needs: every CTA of the persistent grid may leave the partial sums of two output tiles.
struct Scratch {
    float* partials = nullptr;       // [slots][tile floats]
    std::size_t partial_bytes = 0;
    unsigned* tile_counters = nullptr;  // one per output tile, zero between launches (the last arriver resets its counter)
    std::size_t counter_count = 0;
};

struct Context {
    int device = 0;
    int sm_count = 0;
    int compute_major = 0, compute_minor = 0;
    std::size_t smem_optin = 0;
    Scratch scratch;
    int* status = nullptr;       // device word: 0 = fine; otherwise the code of the first wait that ran out (see kStatus*)
    int* status_host = nullptr;  // pinned host copy for sepal_b200_status
    TensorMapEncodeFn encode = nullptr;
    void* unit_scales = nullptr;  // kUnitScales binary16 ones: the scale table of an int8 multiply whose scales are applied per output column
    float* unit = nullptr;        // device float 1.0
    static constexpr std::size_t kUnitScales = 1u << 16;
    void* table = nullptr;        // device memory for the small per-launch tables of the attention kernels (rows, block lists)
    std::size_t table_bytes = 0;
    unsigned table_turn = 0;
    /// The caller's promise that the weights of a multiply launched through this context are never written by the kernel that runs
    /// before it in the stream (an inference engine's weights are uploaded once). A kernel may then request its first weight tiles
    /// before it waits for that kernel (see launch_overlap below). Off unless set.
    bool static_weights = false;

    Context(int device, std::size_t workspace_bytes);
    /// A context over device memory that somebody else owns: nothing is allocated here, and such a context must never be destroyed
    /// (the destructor would free what it does not own). For callers that cannot allocate; see gemm_tc.cu.
    struct Borrowed {};
    Context(Borrowed, int device, float* partials, std::size_t partial_bytes, unsigned* counters, std::size_t counter_count, int* status_word);
    ~Context();
    Context(const Context&) = delete;
    Context& operator=(const Context&) = delete;

    /// Reads the status word after waiting for `stream`, and clears it. 0 means no kernel reported a problem.
    int read_status(cudaStream_t stream);
};

/// Whether kernels are launched as programmatic dependents of the kernel before them in the stream (on by default): the next
/// kernel's CTAs take the SMs as this one's CTAs leave, set up their barriers and tensor memory, and wait in griddepcontrol.wait until
/// this kernel has completed. Every kernel launched this way executes that wait before it touches global memory.
bool launch_overlap();
void set_launch_overlap(bool on);

/// kernel<<<grid, block, smem, stream>>>(args...), as a programmatic dependent when launch_overlap() is on.
template <class... Params, class... Args>
void launch_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, std::size_t smem, cudaStream_t stream, const char* what, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = launch_overlap() ? 1 : 0;
    check(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...), what);
}

/// The same in clusters of `cluster` consecutive blocks (the grid a multiple of it).
template <class... Params, class... Args>
void launch_cluster_kernel(void (*kernel)(Params...), unsigned cluster, dim3 grid, dim3 block, std::size_t smem, cudaStream_t stream, const char* what, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = launch_overlap() ? 2 : 1;
    check(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...), what);
}

/// Default scratch size: two 128 x 256 float32 tiles for each of `sm_count` CTAs.
std::size_t default_workspace_bytes(int sm_count);

/// A 2-D tensor map over a row-major matrix [rows, cols] of `elem_bytes`-byte elements with row stride `ld` elements, tiled in boxes
/// of [box_rows, box_cols] with the 128-byte swizzle (box_cols * elem_bytes must be 128) or none (swizzle == false). Out-of-range
/// parts of a box read as zeros. Throws std::invalid_argument when the driver rejects the layout.
CUtensorMap make_tensor_map_2d(const Context& ctx, const void* base, CUtensorMapDataType type, std::size_t elem_bytes, std::size_t rows,
                               std::size_t cols, std::size_t ld, unsigned box_rows, unsigned box_cols, bool swizzle128);

}  // namespace sepal::b200
