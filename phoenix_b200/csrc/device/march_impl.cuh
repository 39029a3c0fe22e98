// Launch logic of the raymarch kernel (see march.cuh); each march_<mode>_nf<slots>.cu file instantiates launch_nf.
#pragma once

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

// The pipelined kernel (march_pipe.cuh) takes the launches of few rays per SM.  Its blocks hold one ray per lane of their
// geodesic warp only, so 168 registers leave room for 192 rays an SM (128: 256) against the plain kernel's 512: it wins
// while a launch is as long as its longest rays, and loses once the rays fill the chip several times over, the sooner the
// longer the plasma stage is.  Plain kernel's time over the pipelined one's at 20 / 75 deg (96 x 48 x 48-base snapshot), by
// rays per SM:
//   FP32, 1 frequency: 28 1.6 / 1.6, 442 1.22 / 1.34, 529 1.10 / 1.17, 691 0.97 / 1.00;  2: 442 1.07 / 1.24;  3: 270 1.22 / 1.16,
//     389 1.12 / 1.18, 492 0.91 / 0.95;  4: 492 1.09 / 1.15;  5: 389 0.94 / 0.94;  8: 172 1.58 / 1.60, 270 1.40 / 1.32;  32: 27 3.1 / 3.3, 270 2.0 / 1.8
//   mixed, 1: 28 1.7 / 1.7, 442 1.33 / 1.52, 691 1.11 / 1.19;  2: 442 1.08 / 1.48;  3: 270 1.30 / 1.30, 492 0.90 / 0.97;  8: 67
//     1.72 / 1.90, 270 1.16 / 1.12
//   FP64, 1: 110 1.28 / 1.19, 297 1.21 / 1.36;  3: 67 1.26 / 1.23, 110 1.09 / 1.08, 172 0.96 / 0.98, 270 0.72 / 0.70;  8: 110 1.38 /
//     1.53, 270 0.92 / 0.82
// Odd widths put a column of rays over the poles that all take the most steps there are, and gain more: FP32, 351 x 333 (789)
// 1.13 / 1.14, 3 frequencies 271 x 269 (492) 1.11 / 1.23; mixed 1.26 / 1.32 and 1.12 / 1.13.  The limits lie between the two.
template <Mode M, int NF>
constexpr long long pipe_rays_per_sm() {
  return M == Mode::kFP64 ? (NF == 1 ? 300 : NF <= 4 ? 140 : 180)
                          : NF == 1 ? (M == Mode::kFP32 ? 700 : 850) : NF <= 4 ? 500 : (M == Mode::kFP32 ? 320 : 300);
}
constexpr int kPipeWideRays = 490;  // rays per SM up to which a pipelined launch takes 168 registers, beyond them 128

// Plasma warps of a pipelined block: one for one frequency; more frequencies make the plasma stage the longer one, so two
// (up to 4) or four warps share them.
template <int NF>
constexpr int pipe_plasma_warps() {
  return NF == 1 ? 1 : NF <= 4 ? 2 : 4;
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
  if (blocks_per_sm <= 0 && args.default_schedule && args.njobs <= pipe_rays_per_sm<M, NF>() * sms) {
    constexpr int kS = pipe_plasma_warps<NF>(), kThreads = 32 * (1 + kS);
    if constexpr (M == Mode::kFP64) {
      return launch_pipe<M, PT, NF, kS, 256 / kThreads>(args, sms, stream, shape);
    } else {
      return args.njobs <= (long long)kPipeWideRays * sms
                 ? launch_pipe<M, PT, NF, kS, 384 / kThreads>(args, sms, stream, shape)
                 : launch_pipe<M, PT, NF, kS, 512 / kThreads>(args, sms, stream, shape);
    }
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
