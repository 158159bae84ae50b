// Event likelihood on the device: per (hypothesis, module) the extended
// log-likelihood of the module's hit times under a Poisson count and a
// mixture of per-source arrival-time densities (the likelihood of
// example_full.jl:338-449: poisson_dist_per_module, shape_mixture_per_module,
// extended_llh_per_module), FP64.
//
// A module's hits are cut into chunks; blocks take (chunk, hypothesis) items
// from a grid-stride loop (busy modules spread over many blocks, empty ones
// cost one chunk).  A block sums the module's expected photons and stages one
// term per source in shared memory, for its two mixture components
//   c = ln(q w) - lnGamma(alpha) - alpha ln(theta),  alpha - 1,
// and 1 / theta, shift.  Its four warps take a quarter of the sources each,
// for all of the chunk's hits, up to four hits per lane: whatever the number of
// hits, the warps have the same work.  A hit's density is summed as it is,
//   f(x) = sum exp(c + (alpha - 1) ln(x - shift) - (x - shift) / theta),
// one logarithm and two exponentials per source and no branch; a hit whose sum
// is 0, near the ends of the FP64 range or not a number is summed again as a
// log-sum-exp, one source per lane.  Sources beyond one shared-memory tile are
// staged tile by tile for every 128 hits.
//
// Bound by FP64 issue (42 operations per hit, source and hypothesis).  64
// hypotheses of 500 modules x 200 sources with 46,000 hits: 7.07 ms with one
// hit per thread of a 256-thread block (a third of them idle at 92 hits per
// module), an online log-sum-exp whose branches diverge, and CUDA's exp and
// log (some 70 operations); now 2.67 ms, of which the terms (two lgamma and
// three logarithms each, once per hypothesis and module) take a fifth.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "pp_internal.h"
#include "pp_special.cuh"

namespace {

using ppsf::WarpTables;
using ppsf::exp_tab;
using ppsf::log_tab;

constexpr int kThreads = 128, kWarps = kThreads / 32;
constexpr int kTile = 512;           // sources per shared-memory tile
constexpr int kBlockHits = 128;      // hits that a pass over the sources takes: 4 per lane
constexpr int kMaxChunk = 1024;      // hits of a chunk, a multiple of kBlockHits
constexpr unsigned kAll = 0xffffffffu;

struct __align__(16) Term {
  double c1, am1, c2, bm1, inv_theta, shift;
};

__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) t += red[w];
  return t;
}

__device__ __forceinline__ void lse_add(double v, double& m, double& s) {
  if (v == -INFINITY) return;
  if (v > m) {
    s = s * exp(m - v) + 1.0;
    m = v;
  } else {
    s += exp(v - m);
  }
}

// Hits per chunk, from the number of all hits: enough items for every block
// of the grid to have several (a chunk stages the module's terms again), at
// most kMaxChunk.
__device__ __forceinline__ int64_t chunk_hits(int64_t hits, int64_t hyp, int64_t items_wanted) {
  const int64_t c = hits * hyp / max((int64_t)1, items_wanted);
  return min((int64_t)kMaxChunk, max((int64_t)1, c / kBlockHits) * kBlockHits);
}

// chunk_start[k] = first chunk of module k (chunk_start[M + 1] hits each, at
// least one chunk per module); chunk_start[M] = all chunks.  One block; the
// others zero the result.
__global__ void __launch_bounds__(1024) llh_chunk_scan_kernel(const int64_t* __restrict__ offsets, int64_t M, int64_t hyp,
                                                              int64_t items_wanted,
                                                              int64_t* __restrict__ chunk_start,
                                                              double* __restrict__ llh) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ int64_t warp_tot[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x > 0) {
    for (int64_t i = (int64_t)(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < hyp * M;
         i += (int64_t)(gridDim.x - 1) * blockDim.x)
      llh[i] = 0.0;
    return;
  }
  const int64_t per = chunk_hits(offsets[M] - offsets[0], hyp, items_wanted);
  int64_t carry = 0;
  for (int64_t base = 0; base < M; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t n = i < M ? offsets[i + 1] - offsets[i] : 0;
    const int64_t v = i < M ? max((int64_t)1, (n + per - 1) / per) : 0;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(kAll, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? warp_tot[w] : 0;
      all += warp_tot[w];
    }
    __syncthreads();
    if (i < M) chunk_start[i] = carry + before + x - v;
    carry += all;
  }
  if (threadIdx.x == 0) {
    chunk_start[M] = carry;
    chunk_start[M + 1] = per;
  }
}

// Every fourth source's two densities added for Q hits per lane (neighbours
// along a track are lit at about the same time, so quarters would differ in
// how many of their sources are).
template <int Q>
__device__ __forceinline__ void add_sources(const Term* __restrict__ terms, int cnt, const double* x, double* s,
                                            const WarpTables& T) {
#pragma unroll 1
  for (int j = threadIdx.x >> 5; j < cnt; j += kWarps) {
    const Term t = terms[j];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double d = x[q] - t.shift;
      const bool lit = __double2hiint(d) >= 0x00100000;
      if (!__any_sync(kAll, lit)) continue;  // 32 hits before the source's light (a third of them, sorted in time)
      // before the light: a time of some 1e300, whose density is e^-708 or less
      const double y = __hiloint2double(lit ? __double2hiint(d) : 0x7E37E43C, __double2loint(d));
      const double ly = log_tab(y, T);
      const double v1 = fma(t.am1, ly, fma(-t.inv_theta, y, t.c1)), v2 = fma(t.bm1, ly, fma(-t.inv_theta, y, t.c2));
      s[q] += exp_tab(v1, T) + exp_tab(v2, T);
    }
  }
}

__global__ void __launch_bounds__(kThreads, 6) llh_kernel(int mode, int64_t S, int64_t M,
                                                       const double* __restrict__ params,
                                                       const double* __restrict__ photons,
                                                       const int64_t* __restrict__ offsets,
                                                       const double* __restrict__ times,
                                                       const int64_t* chunk_start, double* llh) {
  __shared__ Term terms[kTile];
  __shared__ double part[kWarps][kBlockHits];
  __shared__ double red[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t h = blockIdx.y;
  const WarpTables T = ppsf::warp_tables();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t total = chunk_start[M], per = chunk_start[M + 1];
  for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
    int64_t lo = 0, hi = M;  // the module whose chunks hold g: chunk_start[lo] <= g < chunk_start[hi]
    while (hi - lo > 1) {
      const int64_t step = (hi - lo + 31) / 32, at = lo + (lane + 1) * step;
      const unsigned le = __ballot_sync(kAll, at < hi && chunk_start[at] <= g);
      lo += __popc(le) * step;
      hi = min(hi, lo + step);
    }
    const int64_t k = lo, chunk = g - chunk_start[k];
    const double* P = params + (h * M + k) * S * PP_LLH_PARAMS;
    const double* N = photons ? photons + h * S : nullptr;
    double mu = 0.0, sa = 0.0;
    for (int64_t j = threadIdx.x; j < S; j += blockDim.x) {
      const double a = P[j * PP_LLH_PARAMS];
      mu += a * (N ? N[j] : 1.0);
      sa += a;
    }
    mu = block_sum(mu, red);
    if (mode == PP_LLH_REFERENCE) sa = block_sum(sa, red);
    const int64_t h0 = offsets[k], n = offsets[k + 1] - h0;
    const double norm = mode == PP_LLH_REFERENCE ? sa : mu;
    auto term = [&](int64_t j) {
      const double* q = P + j * PP_LLH_PARAMS;
      const double a = q[0], w = q[1], a1 = q[2], a2 = q[3], th = q[4];
      const double wt = (mode == PP_LLH_REFERENCE ? a : a * (N ? N[j] : 1.0)) / norm;
      const double lth = log(th);
      Term t;
      t.c1 = (wt * w > 0.0 && a1 > 0.0) ? log(wt * w) - lgamma(a1) - a1 * lth : -INFINITY;
      t.c2 = (wt * (1.0 - w) > 0.0 && a2 > 0.0) ? log(wt * (1.0 - w)) - lgamma(a2) - a2 * lth : -INFINITY;
      t.am1 = a1 - 1.0;
      t.bm1 = a2 - 1.0;
      t.inv_theta = 1.0 / th;
      t.shift = q[5];
      return t;
    };
    double acc = 0.0;
    bool odd = false;  // a term that the plain sum is not made for
    const int64_t first = chunk * per, last = min(n, first + per);
    for (int64_t b = first; b < last; b += kBlockHits) {
      const int groups = (int)min((int64_t)4, (last - b + 31) / 32);
      double x[4], s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int64_t i = b + q * 32 + lane;
        x[q] = i < last ? times[h0 + i] : 0.0;
        s[q] = 0.0;
      }
      for (int64_t t0 = 0; t0 < S; t0 += kTile) {
        const int cnt = (int)min((int64_t)kTile, S - t0);
        if (b == first || S > kTile) {  // one tile of sources stays for all the chunk's hits
          __syncthreads();
          for (int j = threadIdx.x; j < cnt; j += blockDim.x) {
            const Term t = term(t0 + j);
            terms[j] = t;
            odd = odd || !(t.c1 < INFINITY) || !(t.c2 < INFINITY) || !(fabs(t.am1) < INFINITY) ||
                  !(fabs(t.bm1) < INFINITY) || !(t.inv_theta > 1e-200 && t.inv_theta < INFINITY) ||
                  !(fabs(t.shift) < INFINITY);
          }
          odd = __syncthreads_or(odd);
        }
        switch (groups) {
          case 1: add_sources<1>(terms, cnt, x, s, T); break;
          case 2: add_sources<2>(terms, cnt, x, s, T); break;
          case 3: add_sources<3>(terms, cnt, x, s, T); break;
          default: add_sources<4>(terms, cnt, x, s, T); break;
        }
      }
      __syncthreads();  // part is free
#pragma unroll
      for (int q = 0; q < 4; ++q) part[warp][q * 32 + lane] = s[q];
      __syncthreads();
      // hit b + threadIdx.x
      const bool has = b + threadIdx.x < last;
      double f = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) f += part[w][threadIdx.x];
      double xt = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) xt = q == warp ? x[q] : xt;
      // x - shift is exact or normal for |x| >= 1e-290; the clamped terms are below 1e-300
      const bool plain = !odd && f > 1e-285 && f < 1e300 && fabs(xt) >= 1e-290 && fabs(xt) < INFINITY;
      if (has && plain) acc += log(f);
      unsigned again = __ballot_sync(kAll, has && !plain);
      while (again) {  // one source per lane, the hit of lane `who`
        const int who = __ffs(again) - 1;
        again &= again - 1;
        const double xx = __shfl_sync(kAll, xt, who);
        double m = -INFINITY, l = 0.0;
        for (int64_t j = lane; j < S; j += 32) {
          const Term t = S <= kTile ? terms[j] : term(j);
          const double y = xx - t.shift;
          if (!(y > 0.0)) continue;
          const double ly = log(y), e = y * t.inv_theta;
          lse_add(t.c1 + t.am1 * ly - e, m, l);
          lse_add(t.c2 + t.bm1 * ly - e, m, l);
        }
        double mm = m;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mm = fmax(mm, __shfl_xor_sync(kAll, mm, o));
        l = m == mm ? l : l * exp(m - mm);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(kAll, l, o);
        if (lane == who) acc += l > 0.0 ? mm + log(l) : -INFINITY;
      }
    }
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) {
      const double nn = (double)n;
      const double pois = chunk > 0 ? 0.0 : (n > 0 ? nn * log(mu) - mu - lgamma(nn + 1.0) : -mu);
      atomicAdd(llh + h * M + k, pois + (n > 0 ? acc : 0.0));
    }
    __syncthreads();
  }
}

}  // namespace

extern "C" pp_status pp_event_llh_device(pp_ctx* c, int32_t mode, int64_t n_hyp, int64_t n_sources,
                                         int64_t n_modules, const double* d_params, const double* d_photons,
                                         const int64_t* d_offsets, const double* d_times, double* d_llh,
                                         void* stream) {
  pp::Range range_("pp_event_llh_device");
  if (!c) return PP_ERR_ARG;
  std::lock_guard<std::mutex> lk(pp::ctx_mutex(c));
  if (mode != PP_LLH_REFERENCE && mode != PP_LLH_SHIFTED) return pp::ctx_fail(c, PP_ERR_ARG, "unknown llh mode");
  if (n_hyp < 0 || n_sources < 1 || n_modules < 0 || n_hyp > 65535 || n_modules > (int64_t)INT32_MAX)
    return pp::ctx_fail(c, PP_ERR_ARG, "need n_sources >= 1, 0 <= n_hyp <= 65535, n_modules >= 0");
  if (n_hyp * n_modules == 0) return PP_OK;
  if (!d_params || !d_offsets || !d_times || !d_llh) return pp::ctx_fail(c, PP_ERR_ARG, "NULL buffer");
  int dev = pp::ctx_device(c), prev = -1;
  cudaGetDevice(&prev);
  if (prev != dev) cudaSetDevice(dev);
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* scratch = nullptr;
  cudaError_t e = pp::ctx_llh_scratch(c, (size_t)(n_modules + 2) * sizeof(int64_t), &scratch);
  if (!e) {
    int64_t* cs = static_cast<int64_t*>(scratch);
    const int64_t blocks = (int64_t)pp::ctx_sm_count(c) * 8;  // on the device at once
    const int64_t zero = std::min<int64_t>((n_hyp * n_modules + 4095) / 4096, 2 * (int64_t)pp::ctx_sm_count(c));
    llh_chunk_scan_kernel<<<1 + (unsigned)zero, 1024, 0, s>>>(d_offsets, n_modules, n_hyp, 4 * blocks, cs, d_llh);
    pp::count_launches(1);
    e = cudaGetLastError();
    // blocks per hypothesis: grid-stride over the chunks
    const dim3 grid((unsigned)std::min<int64_t>(blocks, n_modules * 4), (unsigned)n_hyp);
    if (!e)
      e = pp::launch_dependent(llh_kernel, grid, kThreads, 0, s, mode, n_sources, n_modules, d_params, d_photons,
                               d_offsets, d_times, cs, d_llh);
  }
  if (prev >= 0 && prev != dev) cudaSetDevice(prev);
  if (e) return pp::ctx_cuda_fail(c, e, "event llh");
  return PP_OK;
}
