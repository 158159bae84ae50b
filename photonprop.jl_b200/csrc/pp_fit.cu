// Fit stage on the device: Cherenkov reweighting of hits and weighted Gamma
// maximum-likelihood fits per (pair, observation angle), the caller of the
// hot path in the reference (get_dir_reweight / fit_photon_dist /
// make_photon_fits, src/modelling.jl:46-111; cherenkov_ang_dist,
// src/emission.jl:32-44).
//
// Pipeline on one stream, no host round trip:
//   fit_count_kernel    hits per pair (stored hits only), where a propagation
//                       has not just counted them
//   fit_scan_kernel     exclusive scan in place -> each pair's first record slot
//   fit_scatter_kernel  one 32-byte FitRec per hit, grouped by pair: the
//                       per-hit parts of the weight (cos/sin of the emission
//                       polar angle, 1/n, hit weight / (2 int(n))), tres, ln tres
//   fit_moments_kernel  a warp walks a run of records for 32 or 64 observation
//                       angles, accumulates the four FP64 moments and flushes
//                       them when the pair changes
//   fit_gamma_kernel    Gamma MLE per (pair, angle) from the moments
// fit_columns_kernel builds the records straight from a hit table given as
// FP64 columns (fit_photon_dist over a DataFrame).
//
// The weighted Gamma MLE is the generalised Newton iteration of T. Minka,
// "Estimating a Gamma distribution" (2002), which is how Distributions.jl
// 0.25.62 fits Gamma(x, w) in the reference (fit_mle, src/modelling.jl:75):
// with mx = sum w x / sum w and ml = sum w ln x / sum w,
//   1/a' = 1/a + (ml - ln mx + ln a - psi(a)) / (a^2 (1/a - psi'(a))),
// started at a = (3 - s + sqrt((s - 3)^2 + 24 s)) / (12 s), s = ln mx - ml;
// theta = mx / a.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "pp_device.cuh"
#include "pp_internal.h"
#include "pp_special.cuh"

namespace ppd {

constexpr int kFitWarps = 8;     // warps per block of the moments kernel
constexpr int kFitBlocksPerSm = 4;

__global__ void fit_count_kernel(const pp_hit* __restrict__ hits, const unsigned long long* __restrict__ counters,
                                 unsigned long long cap, int64_t n_pairs, unsigned long long* __restrict__ counts) {
  const unsigned long long n = min(counters[0], cap);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t p = __ldg(&hits[i].pair);
    if ((int64_t)p >= n_pairs) continue;
    // one atomic per pair per warp: hits of one pair sit together in the buffer
    const unsigned grp = __match_any_sync(__activemask(), p);
    if ((threadIdx.x & 31u) == (unsigned)(__ffs(grp) - 1)) atomicAdd(counts + p, (unsigned long long)__popc(grp));
  }
}

// One block: counts[i] becomes the first record slot of pair i (the scatter's
// cursor), the sum of the pairs' hits before it.  Those are counts itself, or,
// where a propagation has just left them there (every hit of it stored), the
// hits of the statistics rows of pairs [lo, hi), the only ones in the buffer.
__global__ void __launch_bounds__(1024) fit_scan_kernel(unsigned long long* __restrict__ counts, int64_t n,
                                                        const double* __restrict__ stats, int64_t lo, int64_t hi) {
  __shared__ unsigned long long warp_tot[32];
  __shared__ unsigned long long carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < n; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    unsigned long long v = 0ull;
    if (i < n) v = !stats ? counts[i] : i >= lo && i < hi ? (unsigned long long)stats[i * PP_STATS] : 0ull;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const int nw = blockDim.x >> 5;
      unsigned long long t = lane < nw ? warp_tot[lane] : 0ull;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
      }
      if (lane < nw) warp_tot[lane] = t;  // inclusive prefix of the warp totals
    }
    __syncthreads();
    const unsigned long long excl = carry + (warp > 0 ? warp_tot[warp - 1] : 0ull) + x - v;
    if (i < n) counts[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
}

__device__ __forceinline__ float ang_norm(const pp::FitConsts& K, const float* normf, float n) {
  // 2 x LinearInterpolation(1.1:0.01:1.5, integral)(n); NaN outside like the reference's BoundsError
  const float x = (n - (float)pp::kAngIntN0) * K.inv_dn;
  if (!(x >= -1e-4f) || !(x <= (float)(pp::kAngIntN - 1) + 1e-4f)) return __int_as_float(0x7fc00000);
  int i = (int)floorf(x);
  i = min(max(i, 0), pp::kAngIntN - 2);
  const float f = x - (float)i;
  return 2.f * fmaf(normf[i + 1] - normf[i], f, normf[i]);
}

// The fit takes tres > 0 (the reference masks tres >= 0, src/modelling.jl:73,
// but a residual of exactly 0, which FP32 rounding makes common for photons
// that fly straight at the sphere, has ln 0 = -inf and no Gamma likelihood).
__device__ __forceinline__ void write_rec(pp::FitRec* r, float ct, float st, float c0, float wn, float tres, int pair) {
  const bool pos = tres > 0.f;
  const float lnt = pos ? logf(tres) : 0.f;
  float4* d = reinterpret_cast<float4*>(r);
  d[0] = make_float4(ct, st, c0, wn);
  d[1] = make_float4(tres, lnt, __int_as_float(pair), __int_as_float(pos ? 1 : 0));
}

__global__ void fit_scatter_kernel(const pp_hit* __restrict__ hits, const unsigned long long* __restrict__ counters,
                                   unsigned long long cap, const pp_pair* __restrict__ pairs, int64_t n_pairs,
                                   int mode, const DevTables* __restrict__ T, const pp::FitConsts K,
                                   unsigned long long* __restrict__ cursor, pp::FitRec* __restrict__ rec) {
  __shared__ float normf[pp::kAngIntN];  // read at a lane's own index
  if (threadIdx.x < pp::kAngIntN) normf[threadIdx.x] = K.normf[threadIdx.x];
  __syncthreads();
  const unsigned long long n = min(counters[0], cap);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float4* h = reinterpret_cast<const float4*>(hits + i);
    const float4 h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2), h3 = __ldg(h + 3);
    const uint32_t p = __float_as_uint(h3.y);
    if ((int64_t)p >= n_pairs) continue;
    const float4* P = reinterpret_cast<const float4*>(pairs + p);
    const float4 pt = __ldg(P), dl = __ldg(P + 1), tg = __ldg(P + 2);
    // emission polar angle about the pair's axis (e_z when the axis is unset)
    const float a2 = fmaf(dl.x, dl.x, fmaf(dl.y, dl.y, dl.z * dl.z));
    float ct = a2 > 0.f ? fmaf(h1.x, dl.x, fmaf(h1.y, dl.y, h1.z * dl.z)) * rsqrtf(a2) : h1.z;
    ct = fminf(fmaxf(ct, -1.f), 1.f);
    const float st = sqrtf(fmaxf(0.f, fmaf(-ct, ct, 1.f)));
    const float wl = h2.w;
    const float n_ph = phase_index(*T, 1.f / wl);
    const float wn = h1.w / ang_norm(K, normf, n_ph);
    const float dx = tg.x - pt.x, dy = tg.y - pt.y, dz = tg.z - pt.z;
    const float d = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    const float tgeo = (d - tg.w) * (mode == kCompat ? K.n800_phase : K.n800_group) / kCVac;
    const float tres = h0.w - (mode == kCompat ? 0.f : pt.w) - tgeo;
    const unsigned grp = __match_any_sync(__activemask(), p);
    const unsigned lane = threadIdx.x & 31u;
    const int lead = __ffs(grp) - 1;
    unsigned long long base = 0;
    if ((int)lane == lead) base = atomicAdd(cursor + p, (unsigned long long)__popc(grp));
    base = __shfl_sync(grp, base, lead);
    write_rec(rec + base + __popc(grp & ((1u << lane) - 1u)), ct, st, 1.f / n_ph, wn, tres, (int)p);
  }
}

__global__ void fit_columns_kernel(int64_t n, const double* __restrict__ tres, const double* __restrict__ theta,
                                   const double* __restrict__ ref_ix, const double* __restrict__ abs_w,
                                   const double* __restrict__ wl, const DevTables* __restrict__ T,
                                   const pp::FitConsts K, pp::FitRec* __restrict__ rec) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double th = theta[i];
    const double nr = ref_ix[i];
    const float pmt = T->n_pmt > 0 ? interp_sorted((float)wl[i], T->pmt_wl, T->pmt_acc, T->n_pmt) : 1.f;
    const float w = (float)abs_w[i] * pmt;
    write_rec(rec + i, (float)cos(th), (float)sin(th), (float)(1.0 / nr), w / ang_norm(K, K.normf, (float)nr),
              (float)tres[i], 0);
  }
}

// A positive normal float as a double, by integer operations: F2F runs on the
// unit that the exponentials and logarithms use.
__device__ __forceinline__ double widen(float w) {
  const uint32_t b = __float_as_uint(w);
  return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// The moments of records [0, n) for kAngles angles per lane.  A block's warps
// are `aw` warps of neighbouring angles times kFitWarps / aw runs of records;
// blockIdx.y counts tiles of aw warps.  The runs divide all the records, so a
// few ten thousand records spread over the chip and a hundred million make
// few flushes.  A warp stages 32 records at a time in its own shared memory,
// with the residual and its logarithm as doubles.
//
// Bound by the special-function unit: three operations per (record, angle)
// for cherenkov_ang_dist.  Three conversions to FP64 beside them took as long
// (two of the record's, once per angle).  7.2e7 records x 250 angles: 28.3 ms,
// now 17.8 ms (that unit 65 % busy; four angles per lane at 96 registers, two at
// 64 20.5 ms); 7.2e5 x 25 (one warp per 2048 records before): 225 us, now 71.
template <int kAngles>
__global__ void __launch_bounds__(kFitWarps * 32) fit_moments_kernel(const pp::FitRec* __restrict__ rec,
                                                                    const unsigned long long* __restrict__ n_ptr,
                                                                    unsigned long long n_fixed,
                                                                    unsigned long long cap,
                                                                    const float2* __restrict__ cs, int n_angles, int aw,
                                                                    const pp::FitConsts K,
                                                                    double* __restrict__ moments) {
  struct Staged {
    float4 geo;   // cos, sin of the emission polar angle, 1/n, weight
    double2 res;  // residual, its logarithm
    int2 who;     // pair; bit 0: the residual is positive, bit 1: not for widen()
  };
  __shared__ Staged tile[kFitWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Staged* mine = tile[warp];
  const unsigned long long n = n_ptr ? min(*n_ptr, cap) : n_fixed;
  const unsigned long long runs = (unsigned long long)gridDim.x * (kFitWarps / aw);
  const unsigned long long run = (unsigned long long)blockIdx.x * (kFitWarps / aw) + warp / aw;
  const unsigned long long per = ((n + runs - 1) / runs + 31) / 32 * 32;  // whole tiles
  const unsigned long long first = min(n, run * per), last = min(n, first + per);
  if (first >= last) return;
  const int a0 = (blockIdx.y * aw + warp % aw) * 32 * kAngles + lane;
  float2 c[kAngles];
  double neg[kAngles], m1[kAngles], m2[kAngles], m3[kAngles];  // sum w over residuals <= 0; sums over the others
#pragma unroll
  for (int q = 0; q < kAngles; ++q) {
    c[q] = a0 + 32 * q < n_angles ? cs[a0 + 32 * q] : make_float2(1.f, 0.f);
    neg[q] = m1[q] = m2[q] = m3[q] = 0.0;
  }
  int cur = -1;
  auto flush = [&]() {
#pragma unroll
    for (int q = 0; q < kAngles; ++q) {
      if (cur >= 0 && a0 + 32 * q < n_angles) {
        double* m = moments + ((int64_t)cur * n_angles + a0 + 32 * q) * PP_FIT_MOMENTS;
        atomicAdd(m + 0, m1[q] + neg[q]);
        atomicAdd(m + 1, m1[q]);
        atomicAdd(m + 2, m2[q]);
        atomicAdd(m + 3, m3[q]);
      }
      neg[q] = m1[q] = m2[q] = m3[q] = 0.0;
    }
  };
  const float4* src = reinterpret_cast<const float4*>(rec);
  float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
  if (first + lane < last) {
    r0 = src[2 * (first + lane)];
    r1 = src[2 * (first + lane) + 1];
  }
  for (unsigned long long t0 = first; t0 < last; t0 += 32) {
    const int cnt = (int)min(32ull, last - t0);
    __syncwarp();
    mine[lane].geo = r0;
    mine[lane].res = make_double2((double)r1.x, (double)r1.y);
    // cherenkov_ang_dist is above 1e-3 for any angles and 1/n of the table's
    // range, so a weight in mid range gives a positive normal product
    const bool odd = !(r0.w >= 1e-30f && r0.w <= 1e30f) || !(fabsf(r0.x) <= 1.001f) || !(fabsf(r0.y) <= 1.001f) ||
                     !(r0.z >= 0.6f && r0.z <= 0.95f);
    mine[lane].who = make_int2(__float_as_int(r1.z), __float_as_int(r1.w) | (odd ? 2 : 0));
    __syncwarp();
    if (t0 + 32 + lane < last) {  // the next tile's records, on their way meanwhile
      r0 = src[2 * (t0 + 32 + lane)];
      r1 = src[2 * (t0 + 32 + lane) + 1];
    }
    for (int j = 0; j < cnt; ++j) {
      const float4 g = mine[j].geo;
      const double2 r = mine[j].res;
      const int2 who = mine[j].who;
      if (who.x != cur) {
        flush();
        cur = who.x;
      }
      // cherenkov_ang_dist(cos(theta0 - a), n) x hit weight / (2 int(n))
      auto weight = [&](int q) {
        const float x = fmaf(g.x, c[q].x, g.y * c[q].y);
        const float pw = ex2(K.c * lg2(fabsf(x - g.z)));
        return fmaf(K.a, ex2(K.b_l2 * pw), K.d) * g.w;
      };
      if (who.y == 1) {
#pragma unroll
        for (int q = 0; q < kAngles; ++q) {
          const double w = widen(weight(q));
          m1[q] += w;
          m2[q] = fma(w, r.x, m2[q]);
          m3[q] = fma(w, r.y, m3[q]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < kAngles; ++q) {
          const double w = (double)weight(q);
          const double p = (who.y & 1) ? w : 0.0;
          neg[q] += (who.y & 1) ? 0.0 : w;
          m1[q] += p;
          m2[q] = (who.y & 1) ? fma(w, r.x, m2[q]) : m2[q];
          m3[q] = (who.y & 1) ? fma(w, r.y, m3[q]) : m3[q];
        }
      }
    }
  }
  flush();
}

__global__ void fit_gamma_kernel(const double* __restrict__ moments, int64_t rows, int n_angles,
                                 const pp_pair* __restrict__ pairs, int64_t n_gen, double* __restrict__ fits) {
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  const double* m = moments + row * PP_FIT_MOMENTS;
  const int64_t N = pairs ? pairs[row / n_angles].n_photons : n_gen;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  double alpha = nan, theta = nan;
  if (m[1] > 0.0) {
    const double mx = m[2] / m[1];
    const double ml = m[3] / m[1];
    const double lmx = log(mx);
    const double s = lmx - ml;
    if (s > 0.0 && isfinite(s) && mx > 0.0) {
      double a = (3.0 - s + sqrt((s - 3.0) * (s - 3.0) + 24.0 * s)) / (12.0 * s);
      for (int it = 0; it < 100; ++it) {
        const double ia = 1.0 / a;
        double psi, psi1;
        ppsf::psi_both(a, psi, psi1);
        const double z = ia + (ml - lmx + log(a) - psi) / (a * a * (ia - psi1));
        const double an = 1.0 / z;
        // the error is squared by each iteration: a step of 1e-9 leaves what
        // rounding leaves (at 1e-14 the rounding of large shapes kept some
        // fits going to the limit)
        const bool done = fabs(an - a) <= 1e-9 * a;
        a = an;
        if (done || !(a > 0.0)) break;
      }
      if (a > 0.0 && isfinite(a)) {
        alpha = a;
        theta = mx / a;
      }
    }
  }
  fits[row * PP_FIT_OUT + 0] = alpha;
  fits[row * PP_FIT_OUT + 1] = theta;
  fits[row * PP_FIT_OUT + 2] = N > 0 ? m[0] / (double)N : nan;
}

}  // namespace ppd

namespace pp {

namespace {
int grid_for(int64_t n, int block, int sm_count) {
  const int64_t want = (n + block - 1) / block;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sm_count * 8));
}

cudaError_t add_moments(const FitConsts& K, const FitRec* rec, const unsigned long long* n_ptr,
                        unsigned long long n_fixed, unsigned long long cap, const float2* cs, int n_angles,
                        double* moments, int sm_count, cudaStream_t s) {
  if ((n_ptr ? cap : n_fixed) == 0) return cudaSuccess;
  // two angles per lane from 33 angles on and four from 65 on (the record's
  // share of the work is divided), and as many warps side by side as the
  // angles need: 1, 2, 4 or 8
  const int per_lane = n_angles > 64 ? 4 : n_angles > 32 ? 2 : 1, warps = (n_angles + 32 * per_lane - 1) / (32 * per_lane);
  int aw = 1;
  while (aw < warps && aw < ppd::kFitWarps) aw *= 2;
  const dim3 grid((unsigned)(sm_count * ppd::kFitBlocksPerSm), (unsigned)((warps + aw - 1) / aw));
  const auto fn = per_lane == 4   ? ppd::fit_moments_kernel<4>
                  : per_lane == 2 ? ppd::fit_moments_kernel<2>
                                  : ppd::fit_moments_kernel<1>;
  fn<<<grid, ppd::kFitWarps * 32, 0, s>>>(rec, n_ptr, n_fixed, cap, cs, n_angles, aw, K, moments);
  count_launches(1);
  return cudaGetLastError();
}
}  // namespace

void fill_fit_consts(FitConsts* K, double n800_phase, double n800_group) {
  K->a = (float)kAngA;
  K->b_l2 = (float)(kAngB / std::log(2.0));  // exp(b v) = 2^(b log2(e) v)
  K->c = (float)kAngC;
  K->d = (float)kAngD;
  K->n800_phase = (float)n800_phase;
  K->n800_group = (float)n800_group;
  K->inv_dn = (float)(1.0 / kAngIntDn);
  double t[kAngIntN];
  cherenkov_ang_dist_int_table(t);
  for (int i = 0; i < kAngIntN; ++i) K->normf[i] = (float)t[i];
}

cudaError_t launch_fit_gamma(const double* moments, int64_t n_pairs, int n_angles, const pp_pair* pairs,
                             int64_t n_gen, double* fits, cudaStream_t s) {
  const int64_t rows = n_pairs * n_angles;
  if (rows == 0) return cudaSuccess;
  // one warp per block: a few hundred serial FP64 fits spread over the chip
  ppd::fit_gamma_kernel<<<(unsigned)((rows + 31) / 32), 32, 0, s>>>(moments, rows, n_angles, pairs, n_gen, fits);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_fit_moments_hits(const FitConsts& K, const void* tables, const pp_pair* pairs, int64_t n_pairs,
                                    int mode, const pp_hit* hits, unsigned long long cap,
                                    const unsigned long long* counters, unsigned long long* counts, FitRec* rec,
                                    const float2* cs, int n_angles, double* moments, int sm_count, cudaStream_t s,
                                    const double* stats, int64_t lo, int64_t hi) {
  cudaError_t e;
  if (n_pairs == 0 || cap == 0) return cudaSuccess;
  const int g = grid_for((int64_t)cap, 256, sm_count);
  if (!stats) {  // hits of unknown pairs: a pass over them to count (2.2 ms for 7.2e7 hits)
    if ((e = cudaMemsetAsync(counts, 0, (size_t)n_pairs * sizeof(unsigned long long), s))) return e;
    ppd::fit_count_kernel<<<g, 256, 0, s>>>(hits, counters, cap, n_pairs, counts);
    count_launches(1);
    if ((e = cudaGetLastError())) return e;
  }
  ppd::fit_scan_kernel<<<1, 1024, 0, s>>>(counts, n_pairs, stats, lo, hi);
  count_launches(1);
  if ((e = cudaGetLastError())) return e;
  ppd::fit_scatter_kernel<<<g, 256, 0, s>>>(hits, counters, cap, pairs, n_pairs, mode,
                                            static_cast<const ppd::DevTables*>(tables), K, counts, rec);
  count_launches(1);
  if ((e = cudaGetLastError())) return e;
  return add_moments(K, rec, counters, 0, cap, cs, n_angles, moments, sm_count, s);
}

cudaError_t launch_fit_columns(const FitConsts& K, const void* tables, int64_t n, const double* tres,
                               const double* theta, const double* ref_ix, const double* abs_w, const double* wl,
                               FitRec* rec, const float2* cs, int n_angles, int64_t n_gen, double* moments,
                               double* fits, int sm_count, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(moments, 0, (size_t)n_angles * PP_FIT_MOMENTS * sizeof(double), s))) return e;
  if (n > 0) {
    ppd::fit_columns_kernel<<<grid_for(n, 256, sm_count), 256, 0, s>>>(
        n, tres, theta, ref_ix, abs_w, wl, static_cast<const ppd::DevTables*>(tables), K, rec);
    count_launches(1);
    if ((e = cudaGetLastError())) return e;
    if ((e = add_moments(K, rec, nullptr, (unsigned long long)n, (unsigned long long)n, cs, n_angles, moments, sm_count,
                         s)))
      return e;
  }
  return launch_fit_gamma(moments, 1, n_angles, nullptr, n_gen, fits, s);
}

}  // namespace pp
