// Launch logic of the raymarch kernel (see march.cuh); each march_<mode>_nf<slots>.cu file instantiates launch_nf.
#pragma once

#include <cmath>

#include "march.cuh"
#include "march_pipe.cuh"

namespace phx {

// Launch shapes.  `blocks_per_sm` names a register-cap variant by its resident warps per SM / 4:
//   1: 128-thread blocks, up to 255 registers (the compiler takes 192 in FP32: 2 blocks, 8 warps per SM);
//   3: 168 registers, 12 warps per SM;   4: 128 registers, 16 warps per SM.
// Variants 3 and 4 run as ONE block of 384 / 512 threads per SM when the job list gives every SM such a block, and as
// 3 / 4 blocks of 128 threads otherwise (small images then still spread over all SMs).  On B200 the whole-SM block
// measured faster than the same warps in 128-thread blocks: FP32, 3 x 512^2 bench images, 16 warps 326 ms as one
// block vs 379 ms as four; 12 warps 336 vs 349 ms.
template <Mode M, class PT, int NF, int kBlock, int kMinBlocks>
cudaError_t launch_mb(const MarchArgs<typename Policy<M>::R, PT>& args, int sms, cudaStream_t stream,
                      LaunchShape* shape) {
  auto kern = k_march<M, PT, NF, kBlock, kMinBlocks>;
  // the rays' transfer records (shared-memory kernels; 0 otherwise)
  const size_t smem = Ray<M, PT, NF>::kSmemPerThread * kBlock;
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kern);
  if (e != cudaSuccess) return e;
  if (smem > 48 * 1024) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int bpsm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, kern, kBlock, smem);
  if (e != cudaSuccess) return e;
  if (bpsm < 1) bpsm = 1;
  long long grid = (long long)bpsm * sms;
  const long long need = (args.njobs + kBlock - 1) / kBlock;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  shape->block = kBlock;
  shape->grid = (int)grid;
  shape->regs = fa.numRegs;
  shape->local_bytes = (int)fa.localSizeBytes;
  shape->blocks_per_sm = bpsm;
  if (args.njobs <= 0) return cudaSuccess;
  kern<<<(unsigned)grid, kBlock, smem, stream>>>(args);
  return cudaGetLastError();
}

// Plasma warps of a pipelined block: one for one frequency; more frequencies make the plasma stage the longer one, so two
// (up to 4) or four warps share them.
template <int NF>
constexpr int pipe_plasma_warps() {
  return NF == 1 ? 1 : NF <= 4 ? 2 : 4;
}

// Whether a line of pixels looks along the axis: the central column of an odd width (row of an odd height, turned by 90
// degrees).  Its rays have no angular momentum, circle the poles for as many steps as there are, and make the launch as
// long as they are.
inline bool has_axis_line(int W, int H, double cos_pa, double sin_pa) {
  return (W % 2 == 1 && std::fabs(sin_pa) < 1e-6) || (H % 2 == 1 && std::fabs(cos_pa) < 1e-6);
}

// The pipelined kernel (march_pipe.cuh) takes the launches of few rays per SM.  Its blocks hold one ray per lane of their
// geodesic warp only, so 168 registers leave room for 192 rays an SM against the plain kernel's 512: it wins while a
// launch is as long as its longest rays, and loses once the rays fill the chip several times over; the sooner the longer
// the plasma stage is (one frequency more than the plasma warps share evenly is as long as a whole round more), and the later
// with a line of rays along the axis.  Plain kernel's time over the pipelined one's at 20 / 75 deg (96 x 48 x 48-base snapshot, 3
// levels), by rays per SM, even widths | odd ones:
//   FP32, 1 frequency: 490 1.25 / 1.27, 620 1.04 / 1.17, 700 0.94 / 0.95 | 700 1.15 / 1.32, 850 1.10 / 1.13
//     2: 490 1.15 / 1.15, 600 0.99 / 1.01 | 490 1.33 / 1.46     3: 440 1.06 / 1.09, 490 0.94 / 1.04 | 490 1.17 / 1.30
//     4: 490 1.15 / 1.16, 540 1.03 / 1.10 | 490 1.30 / 1.51     5: 330 1.01 / 1.00 | 330 1.22 / 1.41
//     8: 320 1.13 / 1.33 | 320 1.36 / 1.54
//   mixed, 1: 490 1.27 / 1.37, 620 1.05 / 1.15, 700 0.96 / 0.94 | 780 1.05 / 1.14, 850 1.02 / 1.07
//     2: 390 1.08 / 1.11, 440 1.03 / 0.95, 490 0.91 / 0.93 | 490 1.06 / 1.13, 540 1.01 / 1.14
//     3: 330 1.11 / 1.07, 390 0.97 / 0.99, 490 0.81 / 0.86 | 440 1.06 / 1.10, 490 1.01 / 0.98 (333 x 217: 1.07 / 1.08)
//     4: 390 1.14 / 1.19, 440 1.04 / 0.98, 490 0.97 / 0.98 | 490 1.15 / 1.14     5: 220 1.05 / 1.12, 300 0.94 / 1.03 | 300 1.25 / 1.26
//     8: 300 1.16 / 1.32 | 300 1.41 / 1.55
//   FP64, 1: 300 1.17 / 1.26, 340 1.02 / 1.00 | 300 1.30 / 1.35     3: 110 1.05 / 1.03, 140 1.03 / 1.23 | 140 1.14 / 1.10
//     8: 180 1.05 / 1.35 | 180 1.27 / 1.63
// A variant of 128 registers (256 rays an SM) was at most 4% faster, between 600 and 650 rays an SM, and slower below.
template <Mode M, int NF>
long long pipe_rays_per_sm(int nfreqs, bool axis_line) {
  if (M == Mode::kFP64) return NF == 1 ? 300 : NF <= 4 ? 140 : 180;
  const bool over = nfreqs % pipe_plasma_warps<NF>() == 1;  // NF > 1
  if (M == Mode::kFP32) return NF == 1 ? (axis_line ? 700 : 650) : NF <= 4 ? (over && !axis_line ? 450 : 500) : 320;
  if (axis_line) return NF == 1 ? 850 : NF <= 4 ? 500 : 300;
  return NF == 1 ? 650 : NF <= 4 ? (over ? 360 : 420) : (over ? 240 : 300);
}

template <Mode M, class PT, int NF, int kS, int kMinCtas>
cudaError_t launch_pipe(const MarchArgs<typename Policy<M>::R, PT>& args, int sms, cudaStream_t stream,
                        LaunchShape* shape) {
  auto kern = k_march_pipe<M, PT, NF, kS, kMinCtas>;
  constexpr int kBlock = 32 * (1 + kS);
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kern);
  if (e != cudaSuccess) return e;
  int bpsm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, kern, kBlock, 0);
  if (e != cudaSuccess) return e;
  if (bpsm < 1) bpsm = 1;
  const long long need = (args.njobs + 31) / 32;
  long long grid = (long long)bpsm * sms;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  shape->block = kBlock;
  shape->grid = (int)grid;
  shape->regs = fa.numRegs;
  shape->local_bytes = (int)fa.localSizeBytes;
  shape->blocks_per_sm = bpsm;
  if (args.njobs <= 0) return cudaSuccess;
  kern<<<(unsigned)grid, kBlock, 0, stream>>>(args);
  return cudaGetLastError();
}

// Default variant per mode (measured on B200, 3 x 512^2 bench images): FP32 4 (128 registers, 16 warps); mixed with one
// frequency slot 4 (128 registers, 140 bytes of spills: 474 ms vs 484 ms at 168 registers, 12 warps), mixed with more
// slots 3 (4% faster than uncapped in 128-thread blocks); FP64 uncapped.
template <Mode M, int NF>
constexpr int default_blocks_per_sm() {
  return M == Mode::kFP32 ? 4 : M == Mode::kMixed ? (NF == 1 ? 4 : 3) : 1;
}

// The variant for `blocks_per_sm` (0 = the mode's default).  FP64 is compiled uncapped only; mixed offers 1 and 3, and 4
// with one frequency slot (with more, 128 registers spill 204 bytes: a 333 x 217 image of 3 frequencies 92.5 ms against
// 78.8 ms).
template <Mode M, class PT, int NF>
cudaError_t launch_nf(const MarchArgs<typename Policy<M>::R, PT>& args, int sms, int blocks_per_sm,
                      cudaStream_t stream, LaunchShape* shape) {
  // a launch shape or refill policy named by the caller: always the plain kernel
  const bool axis_line = has_axis_line(args.rc.W, args.rc.H, args.rc.cos_pa, args.rc.sin_pa);
  if (blocks_per_sm <= 0 && args.default_schedule &&
      args.njobs <= pipe_rays_per_sm<M, NF>(args.rc.nfreqs, axis_line) * sms) {
    constexpr int kS = pipe_plasma_warps<NF>(), kThreads = 32 * (1 + kS);
    return launch_pipe<M, PT, NF, kS, (M == Mode::kFP64 ? 256 : 384) / kThreads>(args, sms, stream, shape);
  }
  if constexpr (M == Mode::kFP64) {
    (void)blocks_per_sm;
    return launch_mb<M, PT, NF, 128, 1>(args, sms, stream, shape);
  } else {
    const int bps = blocks_per_sm > 0 ? blocks_per_sm : default_blocks_per_sm<M, NF>();
    const bool whole = args.njobs >= (long long)sms * 128 * bps;  // a whole-SM block for every SM
    if (bps == 3) {
      return whole ? launch_mb<M, PT, NF, 384, 1>(args, sms, stream, shape)
                   : launch_mb<M, PT, NF, 128, 3>(args, sms, stream, shape);
    }
    if constexpr (M == Mode::kFP32 || (M == Mode::kMixed && NF == 1)) {
      if (bps == 4) {
        return whole ? launch_mb<M, PT, NF, 512, 1>(args, sms, stream, shape)
                     : launch_mb<M, PT, NF, 128, 4>(args, sms, stream, shape);
      }
    }
    return launch_mb<M, PT, NF, 128, 1>(args, sms, stream, shape);
  }
}

}  // namespace phx
