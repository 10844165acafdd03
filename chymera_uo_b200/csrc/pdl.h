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
// one with much shared memory keeps that one's small L1 (which is why k_thomas_f64
// and the kernels around it take turns, k_solve.cu).  So launches overlap
// (Work::pdl) in a launch sequence of up to kPdlCells cells that this library runs
// by itself: not beside others of chy_solve_multi, nor in the server.  A caller's
// own streams are not known here; two plans on two streams take the same or less
// time for it (mixed 128x64x128 113 -> 107 us a pair, FP64 114 -> 102, BLKTRI 2.08 ->
// 2.07 ms).  Measured without -> with, us, solves one after the other in a graph, and
// one at a time waited for by the host:
//   0.14 M cells  FP64 64x32x64      39.7 -> 38.2    79.8 -> 63.0
//                 mixed              49.4 -> 47.6    75.8 -> 63.0
//   4.2 M         FP64 128x64x128 x4  155 -> 154      196 -> 180
//   8.2 M         FP64 256x128x256    320 -> 317      354 -> 337
//                 mixed               242 -> 243      270 -> 264
//                 FP64 512x64x256     300 -> 297      334 -> 318
//                 mixed               450 -> 448      492 -> 469
//   8.8 M         mixed 64x32x64 x64  777 -> 774      895 -> 890
//   16.4 M        FP64 256x128x256 x2 576 -> 574      613 -> 597
//                 mixed               424 -> 432      455 -> 455
//   33 M          mixed 256x128x256 x4 738 -> 750     774 -> 777
//   66 M          FP64 256x128x256 x8 2042 -> 2055   2092 -> 2091
//                 mixed              1413 -> 1444    1460 -> 1480
// The line lies between 8.8 M and the first sizes that lose.
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
