// Per-frequency image totals on the device: the reference's host::output::compute_spec and compute_tau
// (src/host/io/output.hpp:43-74) without downloading the image.
//
//   I, Q, U, V  summed over the pixels whose I+Q+U+V is finite, times the pixel solid angle and 1e23 (Jy);
//   tau, tauF   means over the pixels whose six values sum to a finite number (0 when there are none).
//
// One thread-block cluster per frequency: each CTA sums a strided share of the pixels into FP64 partials (warp shuffles,
// then its warps in a fixed order) and writes them into CTA 0's shared memory, which adds them up in rank order and
// writes the record.  The result is deterministic (no atomics) and nothing beyond the image and the output records is
// touched.
//
// The kernel is bound by what its SMs can read, so the cluster is the largest set of SMs that can add up partials without
// scratch memory, 16 CTAs (8, the portable size, where the device cannot place 16), and a thread loads kSpecUnroll records
// before it adds the first.  A CTA holds 26,624 of an SM's 65,536 registers: a spectrum starts beside another stream's
// kernel that leaves that much free (up to three blocks of a pipelined render); with 512 threads and six records, all of an
// SM's registers, it waited for half a render of 64^2 pixels, 3.6 ms instead of 0.03.  Measured (records of three images in
// turn; in brackets 512 threads and six records, then 8 CTAs of 512 threads): 1024^2 pixels, 4 frequencies 95 us (93, 177), 1
// frequency 54 (32, 134); 512^2, 3 frequencies 23.6 (23.6, 42.7); 1400 x 1300, 6 frequencies 129 (131, 277); 128^2 6.5
// (6.6, 7.5).  With several frequencies every lane's record is a cache line of its own and the L1's tag lookups hold an SM
// at 33 GB/s; three lanes to a record (shuffled verdicts: 105 us for the first of these; staged through shared memory:
// 86, but 55 and 31 us for the next two) did not pay.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <map>
#include <mutex>
#include <stdexcept>

#include "../host/render_setup.hpp"
#include "internal.hpp"

namespace cg = cooperative_groups;
using namespace phx_capi;

namespace {

constexpr int kSpecCluster = 16, kSpecClusterPortable = 8;
constexpr int kSpecUnroll = 5;  // records a thread has in flight
constexpr int kSpecThreads = 256;
constexpr int kSpecWarps = kSpecThreads / 32;

// Sums of warps, CTAs and the cluster are compensated: s + e is the sum, e what the additions to s rounded off.  Every
// addition there rounds at the size of the total, and the 15 CTAs after the first alone put 1e-16 on it; the threads' and
// the shuffles' roundings are of parts and average out.  Of 288 totals of 512^2 images 96% are the exact sum, rounded
// (without the compensation, 8 CTAs of 512 threads, 65%).
//
// (s, e) += (y, f): Knuth's two-sum, e what the additions to s rounded off (an infinite sum leaves a NaN in e, which total()
// drops).
__device__ __forceinline__ void add_comp(double& s, double& e, double y, double f) {
  const double t = s + y, z = t - s;
  e += f + ((s - (t - z)) + (y - z));
  s = t;
}
__device__ __forceinline__ double total(double s, double e) {
  const double t = s + e;
  return isfinite(t) ? t : s;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(kSpecThreads, 2)
    k_spectrum(const double2* __restrict__ res, long long npix, int nfreqs, double jy_per_unit,
               PhxSpectrum* __restrict__ out) {
  __shared__ double warp_s[6][kSpecWarps];
  __shared__ unsigned warp_n[2][kSpecWarps];
  __shared__ double cta_s[6][kSpecCluster], cta_e[6][kSpecCluster];  // of rank 0: every CTA's partials
  __shared__ unsigned long long cta_n[2][kSpecCluster];
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // waited for before the first access to rank 0's shared memory
  const unsigned rank = cluster.block_rank(), ncta = cluster.num_blocks();
  const int f = blockIdx.y;
  double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  unsigned nflux = 0, ntau = 0;
  const unsigned first = rank * kSpecThreads + threadIdx.x, stride = ncta * kSpecThreads;
  int n = first < npix ? (int)(((unsigned)npix - first + stride - 1) / stride) : 0;
  const size_t step = (size_t)stride * nfreqs * 3;
  const double2* r = res + ((size_t)first * nfreqs + f) * 3;
  for (; n > 0; n -= kSpecUnroll, r += kSpecUnroll * step) {
    double2 v[kSpecUnroll][3];
#pragma unroll
    for (int u = 0; u < kSpecUnroll; u++) {
      if (u < n) {
#pragma unroll
        for (int w = 0; w < 3; w++) v[u][w] = __ldg(r + u * step + w);
      }
    }
    // the records of a round first: all but one of their additions round at their own size, not at the sum's
    double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int u = 0; u < kSpecUnroll; u++) {
      if (u >= n) break;
      const double2 iq = v[u][0], uv = v[u][1], tt = v[u][2];
      const double stokes = iq.x + iq.y + uv.x + uv.y;
      if (isfinite(stokes)) {
        t[0] += iq.x;
        t[1] += iq.y;
        t[2] += uv.x;
        t[3] += uv.y;
        nflux++;
      }
      if (isfinite(stokes + tt.x + tt.y)) {
        t[4] += tt.x;
        t[5] += tt.y;
        ntau++;
      }
    }
#pragma unroll
    for (int q = 0; q < 6; q++) s[q] += t[q];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 6; q++) s[q] = warp_sum(s[q]);
  nflux = __reduce_add_sync(0xffffffffu, nflux);
  ntau = __reduce_add_sync(0xffffffffu, ntau);
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < 6; q++) warp_s[q][warp] = s[q];
    warp_n[0][warp] = nflux;
    warp_n[1][warp] = ntau;
  }
  __syncthreads();
  cluster.barrier_wait();
  const int q = threadIdx.x;
  if (q < 6) {
    double t = warp_s[q][0], e = 0.0;
#pragma unroll
    for (int w = 1; w < kSpecWarps; w++) add_comp(t, e, warp_s[q][w], 0.0);
    *cluster.map_shared_rank(&cta_s[q][rank], 0) = t;
    *cluster.map_shared_rank(&cta_e[q][rank], 0) = e;
  } else if (q < 8) {
    unsigned long long t = 0;
    for (int w = 0; w < kSpecWarps; w++) t += warp_n[q - 6][w];
    *cluster.map_shared_rank(&cta_n[q - 6][rank], 0) = t;
  }
  cluster.sync();
  if (rank != 0 || q >= 8) return;
  unsigned long long m = 0;
  for (unsigned c = 0; c < ncta; c++) m += cta_n[q == 6 ? 0 : 1][c];
  if (q >= 6) {
    (q == 6 ? out[f].n_flux : out[f].n_tau) = (int64_t)m;
    return;
  }
  double t = cta_s[q][0], e = cta_e[q][0];
  for (unsigned c = 1; c < ncta; c++) add_comp(t, e, cta_s[q][c], cta_e[q][c]);
  t = total(t, e);
  if (q < 4) out[f].IQUV[q] = t * jy_per_unit;
  else (q == 4 ? out[f].tau_mean : out[f].tauF_mean) = m ? t / (double)m : 0.0;
}

// Whether the current device can place a cluster of kSpecCluster CTAs of k_spectrum (16 is beyond the portable 8).
bool wide_clusters() {
  int dev = 0;
  ck(cudaGetDevice(&dev), "cudaGetDevice");
  static std::mutex mu;
  static std::map<int, bool> known;  // a property of the device and the kernel
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  bool ok = cudaFuncSetAttribute(k_spectrum, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (ok) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim = {(unsigned)kSpecCluster, 1, 1};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSpecCluster);
    cfg.blockDim = dim3(kSpecThreads);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    ok = cudaOccupancyMaxActiveClusters(&n, k_spectrum, &cfg) == cudaSuccess && n >= 1;
  }
  if (!ok) cudaGetLastError();
  known[dev] = ok;
  return ok;
}

}  // namespace

namespace phx_capi {

void launch_spectrum(const PhxRenderParams& p, const PhxFreqOut* d_res, PhxSpectrum* d_spec, cudaStream_t st) {
  if ((reinterpret_cast<uintptr_t>(d_res) & 15u) != 0) throw std::invalid_argument("d_res must be 16-byte aligned");
  const long long npix = (long long)p.img_width * p.img_height;
  const double jy = phx::pixel_solid_angle(p) * phx::cgs::jansky;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim = {(unsigned)(wide_clusters() ? kSpecCluster : kSpecClusterPortable), 1, 1};
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kSpecThreads);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(attr.val.clusterDim.x, p.nfreqs);
  ck(cudaLaunchKernelEx(&cfg, k_spectrum, reinterpret_cast<const double2*>(d_res), npix, (int)p.nfreqs, jy, d_spec),
     "spectrum launch");
  ck(cudaGetLastError(), "spectrum launch");
}

}  // namespace phx_capi

extern "C" int phx_spectrum_async(const PhxRenderParams* p, const PhxFreqOut* d_res, PhxSpectrum* d_spec,
                                  void* stream) {
  return guarded([&]() -> int {
    if (!p || !d_res || !d_spec) throw std::invalid_argument("null argument");
    phx::check_params(*p);
    launch_spectrum(*p, d_res, d_spec, (cudaStream_t)stream);
    return PHX_OK;
  });
}
