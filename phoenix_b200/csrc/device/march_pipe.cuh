// The raymarch of a small launch, in a pipeline of warps.
//
// A launch whose rays leave most of the chip's warp slots empty lasts as long as its longest ray: about 10^4 passes of
// a geodesic step and a plasma sample, one after the other in one lane.  Nothing of the geodesic depends on the
// samples, so here a block is one geodesic warp, which marches 32 rays and stores each pass's samples in shared memory,
// and kS plasma warps, which run the plasma stage of the previous chunk of passes meanwhile (lane i: ray i; with more
// than one plasma warp each takes every kS-th frequency).  A pass then costs the longer of the two instead of their sum.
// The arithmetic of a ray is the plain kernel's (march.cuh), but compiled apart: geodesics, samples and FP64 images are the
// same to the bit, optical depths have been in every image compared, and FP32 and mixed Stokes vectors agree to rounding
// (2e-6 of the image's scale at the worst pixel).
//
// Chunks are double-buffered; one barrier of the block per chunk hands a filled buffer over and gets the other one back
// (8 passes of FP32 points, 2 of FP64 ones: 10 to 21 KB of shared memory a block; FP32 with 4: 1 to 2% slower, FP64 with 4:
// the same).
//
// A 64^2 FP32 image takes 10.4 ms against the plain kernel's 15.9 (about 2,040 cycles a pass against 3,215; a march
// without any samples 8.6 ms).  Unrolling the RK4 stages for more parallelism inside the geodesic warp was slower at
// every size (2 stages: 128^2 15.1 -> 15.7 ms, 4: 18.0 ms): the longer code misses the instruction cache.
#pragma once

#include "march.cuh"

namespace phx {

template <Mode M, class PT, int NF, int kS, int kMinCtas>
__global__ void __launch_bounds__(32 * (1 + kS), kMinCtas)
    k_march_pipe(const __grid_constant__ MarchArgs<typename Policy<M>::R, PT> A) {
  using Geo = GeoRay<M, PT>;
  using R = typename Policy<M>::R;
  using G = typename Policy<M>::G;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kPasses = sizeof(G) == 4 ? 8 : 2;  // passes of a chunk
  constexpr int kWords = Geo::kWP ? 9 : 13;        // x1..x3, k, r, step length (FP64: and F)
  __shared__ G word[2][kPasses][kWords][32];
  __shared__ int32_t seed_leaf[2][kPasses][32];
  __shared__ unsigned due[2][kPasses];  // lanes with a sample in the pass
  __shared__ int more[2];               // the chunk is not the rays' last
  __shared__ int32_t head_pix[32];      // the rays of this round: pixel (-1: none) and Walker-Penrose constant
  __shared__ double head_kappa[2][32];
  __shared__ int head_end;
  __shared__ int ray_bad[32];           // bad samples of the rays of this round, over the plasma warps
  auto block_sync = [] {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * (1 + kS)) : "memory");
  };
  const unsigned lane = threadIdx.x & 31u;
  const int role = (int)(threadIdx.x >> 5);
  const SnapView<G, PT>& sg = Geo::geo_view(A.snap, A.snap_d);
  RayCounters ctr{};
  if (role == 0) {
    Geo ray;
    unsigned steps = 0, rays = 0;
    int32_t last = -1;  // the pixel of the round before
    ray_bad[lane] = 0;
    for (;;) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&A.counters[kCtrQueue], 32ull);
      base = __shfl_sync(kFull, base, 0);
      const bool end = base >= (unsigned long long)A.njobs;
      bool live = false;
      int32_t pix = -1;
      if (base + lane < (unsigned long long)A.njobs) {
        pix = A.jobs[base + lane];
        // a job outside the image is skipped, never written (the host checks job lists it uploads itself)
        if (pix >= 0 && pix < A.rc.W * A.rc.H) {
          const RayStart st = ray_start<G>(A.rc, sg.a, sg.hs, pix);
          ray.start(st, pix);
          head_kappa[0][lane] = st.kappa[0];
          head_kappa[1][lane] = st.kappa[1];
          live = true;
        }
      }
      head_pix[lane] = live ? pix : -1;
      if (lane == 0) head_end = end;
      block_sync();
      // the plasma warps are through with the round before: its counts are stored, not added up in global memory, where
      // a pixel that is in the job list twice would get both rays'
      if (A.pixstats && last >= 0) A.pixstats[3 * (size_t)last + 2] = ray_bad[lane];
      ray_bad[lane] = 0;
      last = live ? pix : -1;
      if (end) break;
      for (int b = 0;; b ^= 1) {
#pragma unroll 1
        for (int c = 0; c < kPasses; c++) {
          bool sampled = false;
          if (live) {
            live = ray.template march<1>(sg, A.rc, ctr, [&](const G* x, const G* k, const G* F, G r, G hl, int right,
                                                            const StepTrig<G>&) {
#pragma unroll
              for (int i = 0; i < 3; i++) word[b][c][i][lane] = x[1 + i];
#pragma unroll
              for (int i = 0; i < 4; i++) word[b][c][3 + i][lane] = k[i];
              word[b][c][7][lane] = r;
              word[b][c][8][lane] = hl;
              if constexpr (!Geo::kWP) {
#pragma unroll
                for (int i = 0; i < 4; i++) word[b][c][9 + i][lane] = F[i];
              }
              seed_leaf[b][c][lane] = right;
              sampled = true;
            });
            if (!live) {
              if (A.pixstats) A.pixstats[3 * (size_t)ray.pix] = ray.steps;
              steps += (unsigned)ray.steps;
              rays++;
            }
          }
          const unsigned m = __ballot_sync(kFull, sampled);
          if (lane == 0) due[b][c] = m;
        }
        const bool any = __any_sync(kFull, live);
        if (lane == 0) more[b] = any;
        block_sync();
        if (!any) break;
      }
    }
    const unsigned long long wsteps = warp_sum_u64(steps), wrays = warp_sum_u64(rays);
    const unsigned long long f64s = warp_sum_u64(ctr.fp64_steps);
    if (lane == 0) {
      atomicAdd(&A.counters[kCtrSteps], wsteps);
      atomicAdd(&A.counters[kCtrRays], wrays);
      if (f64s) atomicAdd(&A.counters[kCtrFp64Steps], f64s);
    }
  } else {
    const int first = role - 1;
    PlasmaRay<M, PT, NF, AccRegs<R, Geo::kMixed, (NF + kS - 1) / kS>, kS> ray;
    unsigned nplasma = 0, bad = 0;
    for (;;) {
      block_sync();
      if (head_end) break;
      const int32_t pix = head_pix[lane];
      const double kappa[2] = {head_kappa[0][lane], head_kappa[1][lane]};
      ray.start(kappa);
      for (int b = 0;; b ^= 1) {
        block_sync();
#pragma unroll 1
        for (int c = 0; c < kPasses; c++) {
          if (!((due[b][c] >> lane) & 1u)) continue;
          G x[4], k[4], F[4];
          x[0] = G(0);  // t: not used by a sample
#pragma unroll
          for (int i = 0; i < 3; i++) x[1 + i] = word[b][c][i][lane];
#pragma unroll
          for (int i = 0; i < 4; i++) k[i] = word[b][c][3 + i][lane];
#pragma unroll
          for (int i = 0; i < 4; i++) F[i] = Geo::kWP ? G(0) : word[b][c][(Geo::kWP ? 0 : 9) + i][lane];
          ray.process_sample(A.snap, sg, A.rc, x, k, F, word[b][c][7][lane], word[b][c][8][lane],
                             seed_leaf[b][c][lane], ctr, nullptr, first);
        }
        __syncwarp();
        if (!more[b]) break;
      }
      if (pix >= 0) {
        ray.write(A.out, pix, A.rc.nfreqs, first);
        if (A.pixstats && first == 0) A.pixstats[3 * (size_t)pix + 1] = ray.nplasma;
        if (ray.bad) atomicAdd(&ray_bad[lane], ray.bad);
        nplasma += (unsigned)ray.nplasma;
        bad += (unsigned)ray.bad;
      }
    }
    const unsigned long long wnplasma = warp_sum_u64(nplasma), wbad = warp_sum_u64(bad);
    const unsigned long long f64o = warp_sum_u64(ctr.fp64_ops);
    if (lane == 0) {
      if (first == 0) atomicAdd(&A.counters[kCtrPlasma], wnplasma);
      atomicAdd(&A.counters[kCtrBad], wbad);
      if (f64o) atomicAdd(&A.counters[kCtrFp64Ops], f64o);
    }
  }
  // leaf scans: the step's lookups and, counted once, the samples'
  if (role <= 1) {
    const unsigned long long scans = warp_sum_u64(ctr.scans);
    if (lane == 0 && scans) atomicAdd(&A.counters[kCtrScans], scans);
  }
}

}  // namespace phx
