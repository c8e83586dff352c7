// Device helpers shared by the kernels: packed u16x2 arithmetic for the path
// recurrence and explicitly rounded f32 operations for the steps whose f32
// results must match the reference's operation order bit for bit.
#pragma once

#include <cstdint>
#include <utility>

#include <cuda_runtime.h>

namespace nxs {

constexpr unsigned kFullMask = 0xFFFFFFFFu;
constexpr uint32_t kInvalidKey = 0xFFFFFFFFu;
// A path cost no real one reaches (real ones are at most p2 + 48 <= 127); it
// stays below 0x8000 after adding p1, so packed adds never carry.
constexpr uint32_t kInf16 = 0x7FFFu;
constexpr uint32_t kInf2 = 0x7FFF7FFFu;
// A cost above every real one that may still be raised by a real one.
constexpr uint32_t kFar2 = 0x70007000u;

// Per-halfword minimum of two u16x2 words (PTX min.u16x2, sm_90+).
__device__ __forceinline__ uint32_t vmin2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Per-halfword sum of two u16x2 words as f16x2 numbers on their bit patterns. Patterns
// below 2048 are their value times 2^-24 (subnormals and the first normal binade), so
// these adds are the integer adds below that; kInf16 is a NaN pattern, and a sum with
// it is kInf16 again; kFar2's 0x7000 (8192.0) absorbs them. A two-operand FMA-pipe instruction:
// it issues beside the three-operand minimums of the integer pipe, which a multiply-add
// does not (4 + 4 in 8.4 cycles a scheduler, against 13.2 with multiply-adds).
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// f32 operations, each rounded to nearest even on its own: never contracted
// into a fused multiply-add, so results equal the reference's evaluation.
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// Programmatic dependent launch: a kernel launched by launch_after is launched
// as the last block of the kernel before it on the stream exits, before that
// grid's completion is processed, so the launch gap between stages overlaps
// the previous stage's end. Such a kernel calls follow_previous_grid() before
// it touches global memory: it waits until the grid before it has completed
// and its writes are visible (griddepcontrol.wait, which returns at once when
// nothing precedes the kernel programmatically). Since every kernel waits at
// its top, a successor never runs ahead of any earlier kernel's writes, nor
// overwrites what an earlier kernel still reads. No kernel signals its
// successor earlier (griddepcontrol.launch_dependents): blocks launched early
// sat resident while they waited, which with many streams in flight held SMs
// other streams' kernels could use (serving saturation 2,455 -> 2,090 pairs/s).
__device__ __forceinline__ void follow_previous_grid() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The kernels that run beside one another (a segment's two lanes, a batch's streams) ask
// for the same split of the L1 between shared memory and cache: an SM that holds blocks of
// one split takes none of another, so with the driver's choice for each kernel a path scan
// and a selection shut each other out (four 1280x720x128 stream pairs 3,190 us, 2,951 with
// one split; 16 mixed pairs in a batch 2,258 and 2,124). 60% gives the 164 KB split, which
// holds 23 blocks of the path scan (6 KB and the 1 KB an SM reserves for each) and the 32 it
// takes at most of the sweep's; the rest is the room in which the selection's loads land: 40%
// and 100% measured 581 and 553 us for a 1280x720x128 pair against 508. A kernel whose blocks
// are too few there by itself, or that runs by itself, leaves the choice to the driver
// (launch_alone), each for the reason given at its launch.
constexpr int kCarveout = 60, kDriversSplit = 0, kSMs = 148;
constexpr size_t kSplitBytes = 164 * 1024, kBlockReserve = 1024;
template <typename... Params, typename... Args>
inline cudaError_t launch_with(int carveout, void (*kernel)(Params...), dim3 grid, dim3 block,
                               size_t shared, cudaStream_t stream, Args &&...args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = shared;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    attribute[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attribute[1].val.sharedMemCarveout = (unsigned)carveout;
    config.attrs = attribute;
    config.numAttrs = carveout == kDriversSplit ? 1 : 2;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared,
                                cudaStream_t stream, Args &&...args) {
    return launch_with(kCarveout, kernel, grid, block, shared, stream,
                       std::forward<Args>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch_alone(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared,
                                cudaStream_t stream, Args &&...args) {
    return launch_with(kDriversSplit, kernel, grid, block, shared, stream,
                       std::forward<Args>(args)...);
}

}  // namespace nxs
