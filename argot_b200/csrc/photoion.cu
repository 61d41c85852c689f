// photoion.cu -- per-cell photo-ionisation and heating rates from the rays
// of each target block (calc_photoion_rate on the device-resident layout).
#include "photoion.cuh"

namespace argot {

int grid_blocks_for_rates(uint64_t n, int threads);
int *err_flag(int dev);

// ------------------------------------------------------------ FP64 rates
// The FP64 loop's tables: sigma_s and sigma_s (nu - nu_s)^+ per bin, nu as
// the reference compares it (a float), and the first bins with sigma_HeI,
// sigma_HeII non-zero.
struct RateTables64 {
  double cs[kNu][3], hw[kNu][3], nu[kNu];
  int first_hei, first_heii;
};
__constant__ RateTables64 c_tab64;

static int ensure_rate_tables64(int device) {
  static std::mutex mu;
  static bool done[64] = {false};
  std::lock_guard<std::mutex> lock(mu);
  if (device < 0 || device >= 64) return ARGOT_B200_EINVAL;
  if (done[device]) return 0;
  double nu[kNu];
  float cs3[3 * kNu];
  host_tables(nu, cs3);
  RateTables64 t;
  const double thr[3] = {kThrHI, kThrHeI, kThrHeII};
  t.first_hei = t.first_heii = kNu;
  for (int k = kNu - 1; k >= 0; k--) {
    t.nu[k] = (double)(float)nu[k];
    for (int q = 0; q < 3; q++) {
      const double c = (double)cs3[3 * k + q];
      t.cs[k][q] = c;
      t.hw[k][q] = t.nu[k] > thr[q] ? c * (t.nu[k] - thr[q]) : 0.0;
      if (c != 0.0 && q >= 1) t.first_hei = k;
      if (c != 0.0 && q == 2) t.first_heii = k;
    }
  }
  ARGOT_CUDA_TRY(cudaMemcpyToSymbol(c_tab64, &t, sizeof(t)));
  ARGOT_CUDA_TRY(cudaStreamSynchronize(0));
  done[device] = true;
  return 0;
}

int ensure_tables(int device) {
  const int rc = ensure_rate_tables(device);
  return rc ? rc : ensure_rate_tables64(device);
}

// Per-species quantities of the target cell for one ray (double):
// the column to the cell's entry face N_s [cm^-2], the cell's own column
// dN_s, and 1/(n_s V_shell + TINY).
struct RayCols {
  double N[3], dN[3], rN[3];
};

__device__ __forceinline__ RayCols ray_columns(const GridDev &g, float t_hi, float t_hei, float t_heii,
                                               float4 raw, RayGeom geo) {
  RayCols c;
  const double cd = __dmul_rn(g.lunit, g.denstonh);
  const double nH = __dmul_rn((double)raw.x, g.denstonh);
  const double nHe = __dmul_rn(nH, kHeliumFact);
  const double n[3] = {__dmul_rn(nH, (double)raw.y), __dmul_rn(nHe, (double)raw.z), __dmul_rn(nHe, (double)raw.w)};
  const float tt[3] = {t_hi, t_hei, t_heii};
  const double a = __dadd_rn((double)geo.dist, __dmul_rn(0.5, (double)geo.delta));
  const double b = __dsub_rn((double)geo.dist, __dmul_rn(0.5, (double)geo.delta));
  const double l3 = __dmul_rn(__dmul_rn(g.lunit, g.lunit), g.lunit);
  const double vsh = __dmul_rn(__dmul_rn(4.0 * kPi / 3.0, __dsub_rn(__dmul_rn(__dmul_rn(a, a), a), __dmul_rn(__dmul_rn(b, b), b))), l3);
#pragma unroll
  for (int s = 0; s < 3; s++) {
    c.dN[s] = __dmul_rn(__dmul_rn(n[s], (double)geo.delta), g.lunit);
    c.N[s] = __dsub_rn(__dmul_rn((double)tt[s], cd), __dmul_rn(0.5, c.dN[s]));
    c.rN[s] = __ddiv_rn(1.0, __dadd_rn(__dmul_rn(n[s], vsh), kTiny));
  }
  return c;
}

// Bins [k0, k1) of the reference's loop in FP64 (calc_photoion_rate.c:285-387)
// with the first kNS species (the others' cross sections are 0 there).  The
// reference forms, per bin and species, (dN_s sigma_s / dtau) pabs rN_s and
// the same times (nu - nu_s); dN_s rN_s does not depend on the bin and is
// applied to the sums, so a bin takes one division instead of three and two
// FMAs per species.
template <int kNS>
__device__ __forceinline__ void rate_bins_f64(const RayCols &c, const double *__restrict__ spec, int k0, int k1,
                                              double (&G)[3], double (&H)[3]) {
#pragma unroll 2
  for (int k = k0; k < k1; k++) {
    double tau = c.N[0] * c_tab64.cs[k][0], dt = c.dN[0] * c_tab64.cs[k][0];
#pragma unroll
    for (int s = 1; s < kNS; s++) {
      tau = fma(c.N[s], c_tab64.cs[k][s], tau);
      dt = fma(c.dN[s], c_tab64.cs[k][s], dt);
    }
    const double w = (__ldg(spec + k) * exp(-tau)) * ((1.0 - exp(-dt)) / (dt + kTiny));
#pragma unroll
    for (int s = 0; s < kNS; s++) {
      G[s] = fma(c_tab64.cs[k][s], w, G[s]);
      H[s] = fma(c_tab64.hw[k][s], w, H[s]);
    }
  }
}

// The same over all bins and species with the reference's operations in its
// order, for rays whose columns or rates are not finite (a source at the
// target's centre, an infinite or undefined field): which of the rates are
// then infinite and which undefined depends on every operation.
static __device__ __noinline__ void rate_bins_f64_in_order(const RayCols &c, const double *__restrict__ spec,
                                                           double out[6]) {
  const double thr[3] = {kThrHI, kThrHeI, kThrHeII};
  double G[3] = {0.0, 0.0, 0.0}, H[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
  for (int k = 0; k < kNu; k++) {
    double cs[3], d[3];
#pragma unroll
    for (int s = 0; s < 3; s++) {
      cs[s] = c_tab64.cs[k][s];
      d[s] = __dmul_rn(c.dN[s], cs[s]);
    }
    const double tau = __dadd_rn(__dadd_rn(__dmul_rn(c.N[0], cs[0]), __dmul_rn(c.N[1], cs[1])),
                                 __dmul_rn(c.N[2], cs[2]));
    const double dtot = __dadd_rn(d[0], __dadd_rn(d[1], d[2]));
    const double pabs = __dmul_rn(__dmul_rn(__ldg(spec + k), exp(-tau)), __dsub_rn(1.0, exp(-dtot)));
    const double den = __dadd_rn(dtot, kTiny), v = c_tab64.nu[k];
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const double w = __dmul_rn(__ddiv_rn(d[s], den), pabs);
      G[s] = __dadd_rn(G[s], __dmul_rn(w, c.rN[s]));
      if (v > thr[s]) H[s] = __dadd_rn(H[s], __dmul_rn(__dmul_rn(w, __dsub_rn(v, thr[s])), c.rN[s]));
    }
  }
#pragma unroll
  for (int s = 0; s < 3; s++) {
    out[s] = G[s];
    out[3 + s] = __dmul_rn(H[s], kHNuL);
  }
}

// The rates of a ray: out[0..2] Gamma, out[3..5] Heat.  75^3 cells, 24 sources
// (the step with the reference-order march): 27.5 ms with three divisions a bin,
// 17.1 ms now; bound by the FP64 operations of the two exponentials.
static __device__ __noinline__ void rate_bins_f64(const RayCols &c, const double *__restrict__ spec, double out[6]) {
  double G[3] = {0.0, 0.0, 0.0}, H[3] = {0.0, 0.0, 0.0};
  const int k1 = c_tab64.first_hei, k2 = c_tab64.first_heii;
  rate_bins_f64<1>(c, spec, 0, k1, G, H);
  rate_bins_f64<2>(c, spec, k1, k2, G, H);
  rate_bins_f64<3>(c, spec, k2, kNu, G, H);
  double all = 0.0;
#pragma unroll
  for (int s = 0; s < 3; s++) {
    const double f = c.dN[s] * c.rN[s];
    out[s] = f * G[s];
    out[3 + s] = f * H[s] * kHNuL;
    all += ((c.N[s] + c.dN[s]) + c.rN[s]) + (out[s] + out[3 + s]);
  }
  if (!isfinite(all)) rate_bins_f64_in_order(c, spec, out);
}

constexpr int kRateWarps = 4;  // warps per CTA in the block-rate kernel

// One warp per target block.  Lanes compute the rates of 32 rays at a time
// into shared memory; then lane j, which owns cell j of the block, adds the
// contributions of the rays that end in its cell in ray order.  No atomics:
// the result does not depend on scheduling.  Each ray's rates are added to
// the existing float value with the reference's float += double rounding
// (calc_photoion_rate.c:403-425).
__global__ void __launch_bounds__(32 * kRateWarps)
    k_rate_blocks(GridDev g, const float4 *__restrict__ raw, const float4 *__restrict__ emit_pos,
                  const double *__restrict__ spec64, uint64_t b0, uint64_t b1,
                  const uint64_t *__restrict__ blk_off, uint64_t base, const uint32_t *__restrict__ rays,
                  uint64_t nray, const float *__restrict__ tau, float *__restrict__ rates6,
                  int *__restrict__ err) {
  __shared__ double buf[kRateWarps][32][7];
  __shared__ int tl[kRateWarps][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t ncell = (uint64_t)g.nx * g.ny * g.nz;
  for (uint64_t b = b0 + warp; b < b1; b += nwarp) {
    int ix, iy, iz;
    const bool own_valid = block_cell(g, b, lane, &ix, &iy, &iz);
    const uint64_t own = own_valid ? cell_index(g, ix, iy, iz) : 0;
    float accf[6];
#pragma unroll
    for (int s = 0; s < 6; s++) accf[s] = own_valid ? rates6[s * ncell + own] : 0.f;
    int bix, biy, biz;
    block_cell(g, b, 0, &bix, &biy, &biz);
    uint64_t r0, r1;
    if (!block_rays(blk_off, b, base, nray, &r0, &r1)) {
      if (lane == 0) atomicExch(err, 1);
      continue;
    }
    for (uint64_t rc = r0; rc < r1; rc += 32) {
      const uint64_t r = rc + lane;
      int t = -1;
      if (r < r1) {
        const uint32_t w = __ldg(rays + r);
        const uint32_t e = w >> 5;
        t = (int)(w & 31u);
        const int lx = bix + (t >> 4), ly = biy + ((t >> 2) & 3), lz = biz + (t & 3);
        const float4 ep = __ldg(emit_pos + e);
        const RayGeom geo = ray_geometry(g, g.ix0 + lx, g.iy0 + ly, g.iz0 + lz, ep.x, ep.y, ep.z);
        const float4 rw = __ldg(raw + cell_index(g, lx, ly, lz));
        const RayCols cols = ray_columns(g, __ldg(tau + r), __ldg(tau + nray + r), __ldg(tau + 2 * nray + r), rw, geo);
        double out[6];
        rate_bins_f64(cols, spec64 + (size_t)e * kNu, out);
#pragma unroll
        for (int s = 0; s < 6; s++) buf[wib][lane][s] = out[s];
      }
      tl[wib][lane] = t;
      __syncwarp();
      const int nk = (int)min((uint64_t)32, r1 - rc);
      for (int k = 0; k < nk; k++) {
        if (tl[wib][k] == lane) {
#pragma unroll
          for (int s = 0; s < 6; s++) accf[s] = __double2float_rn(__dadd_rn((double)accf[s], buf[wib][k][s]));
        }
      }
      __syncwarp();
    }
    if (own_valid) {
#pragma unroll
      for (int s = 0; s < 6; s++) rates6[s * ncell + own] = accf[s];
    }
  }
}

// ------------------------------------------------------------ FP32 rates
// One warp per target block, rays in chunks of 32 (rate_block_f32).  The
// kernel has no FP64 arithmetic.
// Launch shape: ARGOT_RATE_WARPS warps per CTA, at least ARGOT_RATE_MIN_CTAS
// CTAs resident per SM (which caps the registers per thread).  Measured on
// B200 (256^3 cells, 1024 sources): 4 warps x 4 CTAs (124 registers, no
// spills) 0.471 s, the step with the march 0.977 s; x 5 CTAs (96 registers)
// 0.524 s and 1.011 s.
#ifndef ARGOT_RATE_WARPS
#define ARGOT_RATE_WARPS 4
#endif
#ifndef ARGOT_RATE_MIN_CTAS
#define ARGOT_RATE_MIN_CTAS 4
#endif
constexpr int kF32Warps = ARGOT_RATE_WARPS;

template <bool kServed>
__global__ void __launch_bounds__(32 * kF32Warps, ARGOT_RATE_MIN_CTAS)
    k_rate_f32(GridDev g, const float4 *__restrict__ raw, const float4 *__restrict__ emit_pos,
               const float *__restrict__ specn, const double *__restrict__ total, uint64_t b0, uint64_t b1,
               const uint64_t *__restrict__ blk_off, uint64_t base, const uint32_t *__restrict__ rays,
               uint64_t nray, const float *__restrict__ tau, float *__restrict__ rates6,
               const float *__restrict__ pred, int *__restrict__ err) {
  __shared__ RateWarpSmem s_w[kF32Warps];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  RateLane tab;
  load_rate_lane(lane, tab);
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarp = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t b = b0 + warp; b < b1; b += nwarp) {
    uint64_t r0, r1;
    if (!block_rays(blk_off, b, base, nray, &r0, &r1)) {
      if (lane == 0) atomicExch(err, 1);
      continue;
    }
    rate_block_f32<kServed>(g, raw, emit_pos, specn, total, tab, b, r0, r1, rays, nray, tau, rates6, s_w[wib], lane,
                            pred);
  }
}

// The same with a CTA per block (rate_block_f32_cta), for ranges of few blocks.
// When that pays: cta_per_block.
__global__ void __launch_bounds__(32 * kF32Warps, ARGOT_RATE_MIN_CTAS)
    k_rate_f32_cta(GridDev g, const float4 *__restrict__ raw, const float4 *__restrict__ emit_pos,
                   const float *__restrict__ specn, const double *__restrict__ total, uint64_t b0, uint64_t b1,
                   const uint64_t *__restrict__ blk_off, uint64_t base, const uint32_t *__restrict__ rays,
                   uint64_t nray, const float *__restrict__ tau, float *__restrict__ rates6, int *__restrict__ err) {
  __shared__ RateWarpSmem s_w[kF32Warps];
  __shared__ int s_t[kF32Warps][32];
  RateLane tab;
  load_rate_lane(threadIdx.x & 31, tab);
  for (uint64_t b = b0 + blockIdx.x; b < b1; b += gridDim.x) {
    uint64_t r0, r1;
    if (!block_rays(blk_off, b, base, nray, &r0, &r1)) {
      if (threadIdx.x == 0) atomicExch(err, 1);
      continue;
    }
    rate_block_f32_cta<kF32Warps>(g, raw, emit_pos, specn, total, tab, b, r0, r1, rays, nray, tau, rates6, s_w, s_t);
  }
}

// The FP32 rates of blocks [b0, b1) where the rays flagged in pred (7
// planes: six contributions and a flag, see rate_block_f32) keep their
// given contributions: the surrogate's second stage.
int launch_rate_f32_served(const GridDev &g, const float4 *raw, const float4 *emit_pos, const float *specn,
                           const double *total, uint64_t b0, uint64_t b1, const uint64_t *blk_off, uint64_t base,
                           const uint32_t *rays, uint64_t nray, const float *tau, float *rates6, const float *pred,
                           int *err, cudaStream_t st) {
  if (b0 >= b1) return 0;
  k_rate_f32<true><<<grid_blocks_for_rates((b1 - b0) * 32, 32 * kF32Warps), 32 * kF32Warps, 0, st>>>(
      g, raw, emit_pos, specn, total, b0, b1, blk_off, base, rays, nray, tau, rates6, pred, err);
  ARGOT_CUDA_TRY(cudaGetLastError());
  return 0;
}

int grid_blocks_for_rates(uint64_t n, int threads) {
  uint64_t b = (n + threads - 1) / threads;
  const uint64_t cap = (uint64_t)device_sms() * 16;
  return (int)(b < cap ? (b ? b : 1) : cap);
}

}  // namespace argot

using namespace argot;

extern "C" int argot_b200_photoion_rays(const argot_b200_grid *gp, const void *packed,
                                        const argot_b200_dev_tree *t, uint64_t b0, uint64_t b1,
                                        const uint64_t *blk_off, uint64_t base, const uint32_t *rays,
                                        uint64_t nray, const float *tau, int mode, float *rates6,
                                        void *stream) {
  uint64_t nb = 0;
  if (!grid_valid(gp) || !packed || !t || !blk_off || !rates6 || (nray && (!rays || !tau)) ||
      argot_b200_num_blocks(gp, &nb) || b0 > b1 || b1 > nb) {
    set_status(ARGOT_B200_EINVAL);
    return ARGOT_B200_EINVAL;
  }
  if (mode != ARGOT_B200_RATE_EXACT_F64 && mode != ARGOT_B200_RATE_EXACT_F32) {
    set_status(ARGOT_B200_ENOTSUP);
    return ARGOT_B200_ENOTSUP;
  }
  if (b0 == b1) { set_status(0); return 0; }
  int dev = 0;
  ARGOT_CUDA_TRY(cudaGetDevice(&dev));
  int rc = ensure_tables(dev);
  if (rc) return rc;
  int *err = err_flag(dev);
  if (!err) { set_status(ARGOT_B200_ENOMEM); return ARGOT_B200_ENOMEM; }
  GridDev g = make_grid(*gp);
  const uint64_t ncell = (uint64_t)gp->nx * gp->ny * gp->nz;
  const float4 *raw = (const float4 *)packed + ncell;
  cudaStream_t st = (cudaStream_t)stream;
  const int threads = 32 * kRateWarps;
  const int blocks = grid_blocks_for_rates((b1 - b0) * 32, threads);
  const int sms = device_sms();
  if (mode == ARGOT_B200_RATE_EXACT_F64)
    k_rate_blocks<<<blocks, threads, 0, st>>>(g, raw, t->emit_pos, t->emit_spec64, b0, b1, blk_off, base, rays,
                                              nray, tau, rates6, err);
  else if (cta_per_block(b1 - b0, nray, (uint64_t)sms * ARGOT_RATE_MIN_CTAS, kF32Warps))
    k_rate_f32_cta<<<(unsigned)std::min<uint64_t>(b1 - b0, 16ull * sms), 32 * kF32Warps, 0, st>>>(
        g, raw, t->emit_pos, t->emit_specn, t->emit_total, b0, b1, blk_off, base, rays, nray, tau, rates6, err);
  else
    k_rate_f32<false><<<grid_blocks_for_rates((b1 - b0) * 32, 32 * kF32Warps), 32 * kF32Warps, 0, st>>>(
        g, raw, t->emit_pos, t->emit_specn, t->emit_total, b0, b1, blk_off, base, rays, nray, tau, rates6,
        nullptr, err);
  ARGOT_CUDA_TRY(cudaGetLastError());
  set_status(0);
  return 0;
}
