// host_common.h - host-side helpers shared by the kernel launchers: the per-device status
// word that bounded waits report into, TMA tensor-map encoding through the driver entry point
// (no link-time dependency on libcuda), and cached device properties.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "cai_kernels.h"

namespace cai {

// Error codes returned by the extern "C" launchers (0 = ok, negative = host-side failure).
enum : int {
    CAI_K_OK = 0,
    CAI_K_BAD_ARG = -2,
    CAI_K_CUDA = -6,
};

// Device pointer to this device's status word block (64 ints, zero on creation). Allocated once
// per device on first use; kernels receive it as an argument.
int* status_words(int device);
int current_device();
int sm_count(int device);

// Encode a 2-D bf16 (or other 2-byte / 1-byte / 4-byte) row-major tensor map with a 128-byte
// swizzle. `cols` is the contiguous extent, `ld` the row pitch in elements.
// Returns false if the driver rejected the arguments (alignment, pitch).
bool encode_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_cols, uint32_t box_rows, int elem_bytes, bool swizzle128 = true);
// 3-D variant: dims (cols, rows, batch) with pitches in elements.
bool encode_tmap_3d(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t batch,
                    uint64_t ld_row, uint64_t ld_batch, uint32_t box_cols, uint32_t box_rows,
                    int elem_bytes, uint32_t box_batch = 1);

// Launch a kernel so that it may start while the kernel before it in the stream still runs (grid_dep_wait in sm100.cuh holds
// it back from the data): what the chains of short kernels of a small step or layer wait for is the launch of each, the set-up of its
// barriers and tensor memory and the end of the one before. A step of some 60 launches 546 -> 443 us (400 since grid_dep_launch comes
// behind the last loads), one of 220 launches 5.17 -> 4.76 ms, attention over 8 x 384 tokens 93 -> 85 us. Chains of long kernels take
// the same time (norm, two products and SwiGLU, six times: 16384 tokens of 2048 x 8192 8.5 and 8.5 ms, 4096 of 4096 x 14336 7.0
// and 6.9; runs differ by 3 %).
// Only kernels that call grid_dep_wait in every CTA may be launched like this. Kernels that wait for other GPUs are not, nor are products
// under a limit on their SMs: a CTA that only waits for its turn would hold an SM that another stream may need.
template <typename... Params, typename... Args>
inline cudaError_t launch_early(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Args&&>(args)...);
}

const char* last_error();
void set_last_error(const char* fmt, ...);

}  // namespace cai
