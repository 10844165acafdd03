// pdl.h -- launches that overlap their set-up with the kernel before them
// (internal to libchy_pot3).
//
// A solve is six to nine kernels, each of which reads what the one before it
// wrote.  With programmatic stream serialization a kernel's CTAs start as soon
// as the one before it has none left to start and leaves room: they stage their
// constant tables, set up barriers and tensor memory, and wait in pdl_wait()
// until that kernel has completed and its writes are visible.  Every thread
// calls pdl_wait() before the kernel's first access to anything but plan
// constants, also where it then has nothing to do, so that a kernel's completion
// implies that of all kernels before it.
//
// Tensor memory is allocated by waiting until it is free, so a kernel that waits
// in pdl_wait() with columns in hand must not be able to reach an SM before an
// earlier kernel has its own there.  A kernel that allocates before pdl_wait()
// therefore hands over (pdl_go()) only after its allocation; one that allocates
// after it (k_thomas_tm, k_wide_sweep_tm) fills its SM's shared memory, so that no
// CTA with columns fits beside it.  The mode solves hand over late, k_mode_mixed at
// its end and the wide products with their last tile: CTAs that wait through a
// long kernel take its registers, L1 and issue slots.  Solves one after the other in
// a graph, hand-over at the start / so (us): mixed 64x32x64 55.4 / 47.6, 256x128x256
// 246.0 / 241.6, 65x32x64 83.7 / 77.5, 512x64x256 464 / 449; one solve waited for:
// 71.5 / 70.1, 265.1 / 262.9, 93.9 / 91.0, 496 / 479 (the wide products at their end:
// 447, but 495 waited for).
//
// Waiting CTAs hold registers and shared memory, and a kernel that starts beside
// one with much shared memory keeps that one's small L1.  So launches overlap
// (Work::pdl) in a solve that has the device to itself and is short: up to
// kPdlCells cells in the launch sequence.  Measured with and without: one solve of
// 64x32x64 FP64 59.4 -> 43.2 us, mixed 61.1 -> 58.8, of 256x128x256 mixed 250.7
// -> 246.7; but eight solves of 256x128x256 FP64 2.20 -> 2.35 ms, four of
// 512x128x512 5.28 -> 5.41, 24 grids on eight streams 1.59 -> 1.61, and a time
// step whose star and source kernels overlapped too 429 -> 470 us.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace chy {

constexpr size_t kPdlCells = (size_t)9 << 20;

// The kernel after this one may start its CTAs (once all of this one's have
// come here).
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The kernels before this one are complete, their writes visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// on = false: an ordinary launch, after the kernel before it has completed.
template <class... P, class... A>
inline cudaError_t launch_pdl(bool on, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = on ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace chy
