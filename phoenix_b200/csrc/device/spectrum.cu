// Per-frequency image totals on the device: the reference's host::output::compute_spec and compute_tau
// (src/host/io/output.hpp:43-74) without downloading the image.
//
//   I, Q, U, V  summed over the pixels whose I+Q+U+V is finite, times the pixel solid angle and 1e23 (Jy);
//   tau, tauF   means over the pixels whose six values sum to a finite number (0 when there are none).
//
// One thread-block cluster per frequency: each CTA sums a strided share of the pixels into FP64 partials (warp shuffles,
// then its warps in a fixed order); CTA 0 of the cluster then reads the other CTAs' partials through distributed shared
// memory, in rank order, and writes the record.  The result is deterministic (no atomics) and nothing beyond the image
// and the output records is touched.
//
// The kernel is bound by what its SMs can read, so the cluster is the largest set of SMs that can add up partials without
// scratch memory, 16 CTAs (8, the portable size, where the device cannot place 16), and a thread loads kSpecUnroll records
// before it adds the first.  Measured (records of three images in turn): 1024^2 pixels, 4 frequencies 178 -> 96 us, 1
// frequency 132 -> 35 us; 512^2, 3 frequencies 42 -> 25 us; 1400 x 1300, 6 frequencies 281 -> 131 us; images up to 300^2
// stay at the launch's 13 to 17 us.  With several frequencies every lane's record is a cache line of its own and the L1's
// tag lookups hold an SM at 33 GB/s; three lanes to a record (shuffled verdicts: 105 us for the first of these; staged
// through shared memory: 86, but 55 and 31 us for the next two) did not pay.
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
constexpr int kSpecUnroll = 6;  // records a thread has in flight
constexpr int kSpecThreads = 512;
constexpr int kSpecWarps = kSpecThreads / 32;

// Sums of a warp, a CTA or the cluster.  From the warps up they are compensated: s + e is the sum, e what the additions
// to s rounded off.  Every addition there rounds at the size of the total, and the 15 CTAs after the first alone put
// 1e-16 on it; the threads' and the shuffles' roundings are of parts and average out.  Mean error of 24 images' totals against
// an exact sum 9e-18 (8 CTAs without it: 6.7e-17); 2 us of 96.
struct SpecPart {
  double s[6], e[6];        // I, Q, U, V, tau, tauF
  unsigned long long n[2];  // pixels in the flux sum, in the optical-depth means
};

// a += b (Knuth's two-sum; an infinite sum leaves a NaN in e, which total() drops).
__device__ __forceinline__ void add_part(SpecPart& a, const SpecPart& b) {
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const double x = a.s[q], y = b.s[q], t = x + y, z = t - x;
    a.s[q] = t;
    a.e[q] += b.e[q] + ((x - (t - z)) + (y - z));
  }
  a.n[0] += b.n[0];
  a.n[1] += b.n[1];
}
__device__ __forceinline__ double total(const SpecPart& a, int q) {
  const double t = a.s[q] + a.e[q];
  return isfinite(t) ? t : a.s[q];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(kSpecThreads)
    k_spectrum(const double2* __restrict__ res, long long npix, int nfreqs, double jy_per_unit,
               PhxSpectrum* __restrict__ out) {
  __shared__ SpecPart warp_part[kSpecWarps];
  __shared__ SpecPart cta_part;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), ncta = cluster.num_blocks();
  const int f = blockIdx.y;
  double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  unsigned long long nflux = 0, ntau = 0;
  const long long stride = (long long)ncta * kSpecThreads;
  for (long long p0 = (long long)rank * kSpecThreads + threadIdx.x; p0 < npix; p0 += kSpecUnroll * stride) {
    double2 v[kSpecUnroll][3];
#pragma unroll
    for (int u = 0; u < kSpecUnroll; u++) {
      const long long p = p0 + u * stride;
      if (p < npix) {
        const double2* r = res + ((size_t)p * nfreqs + f) * 3;  // one 48-byte record: three 16-byte loads
#pragma unroll
        for (int w = 0; w < 3; w++) v[u][w] = __ldg(r + w);
      }
    }
#pragma unroll
    for (int u = 0; u < kSpecUnroll; u++) {
      if (p0 + u * stride >= npix) break;
      const double2 iq = v[u][0], uv = v[u][1], tt = v[u][2];
      const double stokes = iq.x + iq.y + uv.x + uv.y;
      if (isfinite(stokes)) {
        s[0] += iq.x;
        s[1] += iq.y;
        s[2] += uv.x;
        s[3] += uv.y;
        nflux++;
      }
      if (isfinite(stokes + tt.x + tt.y)) {
        s[4] += tt.x;
        s[5] += tt.y;
        ntau++;
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 6; q++) s[q] = warp_sum(s[q]);
  nflux = warp_sum(nflux);
  ntau = warp_sum(ntau);
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      warp_part[warp].s[q] = s[q];
      warp_part[warp].e[q] = 0.0;
    }
    warp_part[warp].n[0] = nflux;
    warp_part[warp].n[1] = ntau;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    SpecPart t = warp_part[0];
    for (int w = 1; w < kSpecWarps; w++) add_part(t, warp_part[w]);
    cta_part = t;
  }
  cluster.sync();  // every CTA's partial is in its shared memory
  if (rank == 0 && threadIdx.x == 0) {
    SpecPart t = cta_part;
    for (unsigned c = 1; c < ncta; c++) add_part(t, *cluster.map_shared_rank(&cta_part, c));
    PhxSpectrum rec;
    for (int q = 0; q < 4; q++) rec.IQUV[q] = total(t, q) * jy_per_unit;
    rec.tau_mean = t.n[1] ? total(t, 4) / (double)t.n[1] : 0.0;
    rec.tauF_mean = t.n[1] ? total(t, 5) / (double)t.n[1] : 0.0;
    rec.n_flux = (int64_t)t.n[0];
    rec.n_tau = (int64_t)t.n[1];
    out[f] = rec;
  }
  cluster.sync();  // CTA 0 has read the others' shared memory before they exit
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
