// photoion.cuh -- per-ray photo-ionisation / heating rates
// (calc_photoion_rate, photon-conserving branch, H + He, not cosmological).
#pragma once
#include <algorithm>
#include <mutex>

#include "march.cuh"

namespace argot {

constexpr double kHNuL = kHPlanck * kNuL;  // hplanck*nuL, double

// Frequency tables of the rate kernels.  Every translation unit that
// includes this header has its own copy in its constant bank, filled by its
// own ensure_rate_tables().
__constant__ RateTables c_tab;

// The FP32 bin loop's table: of stage m (bins 64 m .. 64 m + 63) the two bins
// 64 m + l and 64 m + l + 32 of lane l; value s: sigma_s log2(e), value
// 3 + s: sigma_s log2(e) (nu - nu_s)^+.
constexpr int kStages = 4;
struct RateTab {
  float2 v[kStages][6][32];
};
static __device__ RateTab d_rate_tab;

static int ensure_rate_tables(int device) {
  static std::mutex mu;
  static bool done[64] = {false};
  std::lock_guard<std::mutex> lock(mu);
  if (device < 0 || device >= 64) return ARGOT_B200_EINVAL;
  if (done[device]) return 0;
  double nu[kNu];
  float cs3[3 * kNu];
  host_tables(nu, cs3);
  RateTables t;
  RateTab rt;
  const double thr[3] = {kThrHI, kThrHeI, kThrHeII}, l2e = 1.4426950408889634074;
  for (int s = 0; s < 3; s++) {
    float m = 0.f;
    for (int k = kNu - 1; k >= 0; k--) {
      const float c = cs3[3 * k + s];
      t.cs[s][k] = c;
      m = fmaxf(m, c);
      if (k % 64 == 0) t.smax[s][k / 64] = m;
      const double nf = (float)nu[k], w = nf > thr[s] ? nf - thr[s] : 0.0;
      float2 &v = rt.v[k / 64][s][k % 32], &h = rt.v[k / 64][3 + s][k % 32];
      (k % 64 < 32 ? v.x : v.y) = (float)((double)c * l2e);
      (k % 64 < 32 ? h.x : h.y) = (float)((double)c * l2e * w);
    }
  }
  ARGOT_CUDA_TRY(cudaMemcpyToSymbol(c_tab, &t, sizeof(t)));
  ARGOT_CUDA_TRY(cudaMemcpyToSymbol(d_rate_tab, &rt, sizeof(rt)));
  // (a copy from pageable memory may return before it has arrived)
  ARGOT_CUDA_TRY(cudaStreamSynchronize(0));
  done[device] = true;
  return 0;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// FP32 rates.  Per ray: the columns to the target cell's entry face N_s and
// of the cell D_s [cm^-2] and the prefactor P_s = total dN_s / (n_s V_shell)
// (calc_photoion_rate.c:159-246), all in FP32.  With dN_s = n_s delta lunit
// and V_shell = 4 pi / 3 ((r + delta/2)^3 - (r - delta/2)^3) lunit^3 =
// 4 pi (r^2 + delta^2 / 12) delta lunit^3 (the cube difference expanded,
// which has no cancellation), the density cancels:
// P_s = total / (4 pi lunit^2 (r^2 + delta^2 / 12)) for n_s > 0 and 0 for
// n_s = 0 (the reference's TINY only keeps 0/0 away; its n_s V_shell is
// above 1e40 whenever n_s is a positive float).  total (1e48-1e52 photons/s)
// and 1/(4 pi lunit^2) (1e-46) are outside the FP32 range, so their powers
// of two are added as integers and P_s (1e4-1e13) is formed in range.
struct RayParams {
  float N[3], D[3], P[3];
};

// v = m * 2^e for a positive double, m in [1, 2) from the leading 24
// significant bits (integer operations on the bit pattern)
__device__ __forceinline__ float mant_exp2(double v, int &e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  e = (int)((b >> 52) & 0x7ffu) - 1023;
  return __uint_as_float(0x3f800000u | (unsigned)((b >> 29) & 0x7fffffu));
}

constexpr float kHeliumFactF = (float)kHeliumFact;
constexpr float kHNuLf = (float)kHNuL;

// The FP32 parameters of a ray from emitter (sx, sy, sz) to the centre of
// target cell (gix, giy, giz) (global indices) with code-unit columns t_s;
// raw = {dens, fHI, fHeI, fHeII} of the target cell.  A ray that starts at
// its target's centre (r = 0) contributes nothing here (the reference's
// operations, and the FP64 rates, leave infinite and undefined rates there).
__device__ __forceinline__ RayParams ray_params_f32(const GridDev &g, int gix, int giy, int giz, float sx,
                                                    float sy, float sz, float t0, float t1, float t2, float4 raw,
                                                    double total) {
  RayParams p;
  const float x = fmaf((float)gix + 0.5f, g.dx, g.xmin);
  const float y = fmaf((float)giy + 0.5f, g.dy, g.ymin);
  const float z = fmaf((float)giz + 0.5f, g.dz, g.zmin);
  const float dx = x - sx, dy = y - sy, dz = z - sz;
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  // delta_length (calc_photoion_rate.c:52-90): the cell's chord along the
  // ray, min over the axes of the cell side over |cosine|
  const float delta = sqrtf(r2) * fminf(__fdividef(g.dx, fabsf(dx)),
                                        fminf(__fdividef(g.dy, fabsf(dy)), __fdividef(g.dz, fabsf(dz))));
  const float n[3] = {raw.x * raw.y, (raw.x * kHeliumFactF) * raw.z, (raw.x * kHeliumFactF) * raw.w};
  const float tt[3] = {t0, t1, t2};
  const float dc = delta * g.cdf;
  int et;
  const float mt = mant_exp2(total, et);
  const float pv = ldexpf(__fdividef(mt * g.pcm, fmaf(delta * delta, 1.f / 12.f, r2)), et + g.pce);
  const bool ok = r2 > 0.f;
#pragma unroll
  for (int s = 0; s < 3; s++) {
    p.D[s] = ok ? n[s] * dc : 0.f;
    p.N[s] = ok ? fmaf(tt[s], g.cdf, -0.5f * p.D[s]) : 0.f;
    p.P[s] = (ok && n[s] > 0.f) ? pv : 0.f;
  }
  return p;
}

// ---- FP32 bin loop.  A warp integrates one ray at a time; its lanes share
// the 256 bins.  Stage m = 0..3 of a ray covers the bins 64 m .. 64 m + 63,
// lane l the pair (64 m + l, 64 m + l + 32), two bins per instruction with
// the f32x2 FMA and multiply of sm_100.  A lane's bins are the same for
// every ray, so their cross sections stay in 44 registers (RateLane) and the
// spectrum in 8 more until the emitter changes; a ray costs two broadcast
// shared loads and the reduction of its six sums over the warp.
// Stage 0 ends below the HeII threshold (bin 102), so it has no HeII terms;
// they would add exact zeros.
//
// What bounds it: the heavy FMA pipe (62% of its cycles; issue 59%, 16 warps per
// SM) and waits between dependent operations.  A ray takes 62 and 64 packed
// operations in the two thin forms, 69 in form 2 and 70 to 72 beyond, at 2.1
// cycles (f32x2 operations issue on that pipe only) and about a dozen scalar
// ones: about 150 cycles per SM sub-partition, counted from the code, of 245
// in the capture (224^3 cells / 32 sources, 2.6e8 rays, 54.9 ms).  Before, four
// 8-lane groups per warp integrated two rays each and read every bin pair's
// 48-byte table entry from shared memory and its spectrum from global memory: 145
// instructions and 41 L1 data-pipe cycles per ray (that pipe is the march's
// beside it) against 143 and 25 now.  256^3 cells, 1024 clustered sources, 2.17e9
// rays: 0.527 s before, 0.480 s now.  Two rays at a time per warp (for more
// independent chains): 2% faster alone, the step with the march no faster.
// (RateShared reads them from a copy in shared memory instead, for a kernel
// that needs its registers.)
struct RateLane {
  float2 v[kStages][6];
  __device__ __forceinline__ float2 l2e(int m, int s) const { return v[m][s]; }    // sigma_s log2(e)
  __device__ __forceinline__ float2 h(int m, int s) const { return v[m][3 + s]; }  // sigma_s log2(e) (nu - nu_s)^+
};
__device__ __forceinline__ void load_rate_lane(int lane, RateLane &r) {
#pragma unroll
  for (int m = 0; m < kStages; m++)
#pragma unroll
    for (int s = 0; s < 6; s++) r.v[m][s] = __ldg(&d_rate_tab.v[m][s][lane]);
}
struct RateShared {
  const RateTab *tab;
  int lane;
  __device__ __forceinline__ float2 l2e(int m, int s) const { return tab->v[m][s][lane]; }
  __device__ __forceinline__ float2 h(int m, int s) const { return tab->v[m][3 + s][lane]; }
};
// Fills a CTA's copy (all threads; the caller synchronises).
__device__ __forceinline__ void load_rate_tab(RateTab &t) {
  const float2 *from = &d_rate_tab.v[0][0][0];
  float2 *to = &t.v[0][0][0];
  for (int i = threadIdx.x; i < kStages * 6 * 32; i += blockDim.x) to[i] = __ldg(from + i);
}

// The photon-conserving cell factor phi(x) = (1 - e^-x)/x (x the cell's
// optical depth in the bin) enters every bin as e^-tau phi(x), tau the
// optical depth to the cell.  Below x = kPhiXMax the difference 1 - e^-x
// cancels, so the loop forms e^-tau phi(x) = e^-(tau + x/2) sinh(y)/y,
// y = x / 2: the attenuation to the middle of the cell, whose exponent folds
// into the ray's columns, times an even polynomial; above, it takes
// e^-tau (1 - e^-x) / x from the SFU (~2e-7).  Below x = kPhiXThin the
// polynomial is 1 + y^2/6 (the y^4/120 left out is below 7e-9).
constexpr float kPhiXMax = 1.0f;
constexpr float kPhiUMax = 1.44269504088896341f;  // kPhiXMax / ln 2
constexpr float kPhiXThin = 0.06f;

// sinh(y) / y, y = x / 2 = dl ln2 / 2, of the two bins of a pair from
// v = dl^2: a near-minimax fit of degree 3 in v made by argot_b200/fits.py
// (fit_sinhc; times the FP32 mid-cell attenuation 2^(-dl/2) it is within
// 1.5e-7 of phi(x) on [0, 1], checked by the CPU tests); thin: its first two
// terms.
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
template <bool kThin>
__device__ __forceinline__ float2 sinhc_half2(float2 dl) {
  constexpr float kShc[4] = {1.f, 0.0200188775f, 0.000120223514f, 3.4621803e-07f};
  const float2 v = __fmul2_rn(dl, dl);
  if (kThin) return __ffma2_rn(v, both(kShc[1]), both(kShc[0]));
  float2 p = __ffma2_rn(v, both(kShc[3]), both(kShc[2]));
  p = __ffma2_rn(v, p, both(kShc[1]));
  return __ffma2_rn(v, p, both(kShc[0]));
}

// How the stages of a ray with cell columns D form the factor: 0 thin, 1
// the degree-3 polynomial, 2 the SFU form for the bins at or above kPhiXMax
// and the polynomial for the others.  Stage m's x is at most sum_s D_s max
// sigma_s over its bins and those above (smax), so it falls from stage to
// stage.  Four forms of the whole ray are compiled, the cheapest that holds
// is taken: its stages' forms are 0: 1 0 0 0, 1: 1 1 0 0, 2: 2 1 1 1 and, from 3
// on, 2 2 2 2 where stage 2 takes the SFU form from 4 on and stage 3 with 5
// only (a branch in the loop; each of the three compiled by itself cost the
// other forms 2%).  The choice depends on the ray alone, and a ray has the
// warp to itself, so the branches are uniform.
// Measured at 64^3 cells / 16 sources, cells of optical depth 0.5, 2, 7, 20
// and 1000 at the HI edge: 779, 875, 1040, 1041 and 1279 us; with all stages in
// the SFU form once stage 1 needs it 775, 879, 1259, 1258 and 1262 us, with the
// table in shared memory and eight lanes per ray 856, 922, 1021, 1085, 1368 us.
__device__ __forceinline__ int ray_form(float D0, float D1, float D2) {
  int f[kStages];
#pragma unroll
  for (int m = 0; m < kStages; m++) {
    const float x = fmaf(D0, c_tab.smax[0][m], fmaf(D1, c_tab.smax[1][m], D2 * c_tab.smax[2][m]));
    f[m] = x >= kPhiXMax ? 2 : x < kPhiXThin ? 0 : 1;
  }
  if (f[1] == 2) return f[3] == 2 ? 5 : f[2] == 2 ? 4 : 3;
  return f[0] == 2 || f[2] || f[3] ? 2 : f[1];
}

// A ray as the loop reads it: n = the negated mid-cell columns
// -(N_s + D_s / 2), d = the cell's columns D_s [cm^-2], the ray's form, the
// emitter.
struct alignas(16) RayRec {
  float n[3];
  int form;
  float d[3];
  int e;
};
__device__ __forceinline__ RayRec ray_rec(const RayParams &p, int e) {
  RayRec r;
#pragma unroll
  for (int s = 0; s < 3; s++) {
    r.n[s] = -fmaf(0.5f, p.D[s], p.N[s]);
    r.d[s] = p.D[s];
  }
  r.form = ray_form(p.D[0], p.D[1], p.D[2]);
  r.e = e;
  return r;
}

// Stage m of one ray: the lane's two bins.  kNS: species with non-zero cross
// sections; kForm as in ray_form.  ntm = -(tau + x / 2) log2(e), w = s 2^ntm
// sinh(x/2)/(x/2) or, with kForm 2, sfu and x >= kPhiXMax, s 2^(ntm + dl/2)
// (1 - 2^-dl) / x.
template <int m, int kNS, int kForm, class Tab>
__device__ __forceinline__ void rate_stage(const Tab &t, float2 s, const float2 (&n)[3], const float2 (&d)[3],
                                           float2 (&acc)[6], bool sfu = true) {
  float2 ntm = __fmul2_rn(n[kNS - 1], t.l2e(m, kNS - 1));
  float2 dl = __fmul2_rn(d[kNS - 1], t.l2e(m, kNS - 1));
#pragma unroll
  for (int q = kNS - 2; q >= 0; q--) {
    ntm = __ffma2_rn(n[q], t.l2e(m, q), ntm);
    dl = __ffma2_rn(d[q], t.l2e(m, q), dl);
  }
  const float2 e = make_float2(ex2_approx(ntm.x), ex2_approx(ntm.y));
  float2 w = __fmul2_rn(__fmul2_rn(s, e), sinhc_half2<kForm == 0>(dl));
  if (kForm == 2 && sfu) {
    const float kLn2 = 0.69314718055994531f;
    const float2 ntl = __ffma2_rn(dl, both(0.5f), ntm);
    const float q0 = s.x * ex2_approx(ntl.x) * __fdividef(1.0f - ex2_approx(-dl.x), dl.x * kLn2);
    const float q1 = s.y * ex2_approx(ntl.y) * __fdividef(1.0f - ex2_approx(-dl.y), dl.y * kLn2);
    w.x = dl.x < kPhiUMax ? w.x : q0;
    w.y = dl.y < kPhiUMax ? w.y : q1;
  }
#pragma unroll
  for (int q = 0; q < kNS; q++) {
    acc[q] = __ffma2_rn(t.l2e(m, q), w, acc[q]);
    acc[3 + q] = __ffma2_rn(t.h(m, q), w, acc[3 + q]);
  }
}
template <int f0, int f1, int f2, int f3, class Tab>
__device__ __forceinline__ void ray_stages(const Tab &t, const float2 (&sp)[4], const float2 (&n)[3],
                                           const float2 (&d)[3], float2 (&acc)[6], int form = 5) {
  rate_stage<0, 2, f0>(t, sp[0], n, d, acc);
  rate_stage<1, 3, f1>(t, sp[1], n, d, acc);
  rate_stage<2, 3, f2>(t, sp[2], n, d, acc, form >= 4);
  rate_stage<3, 3, f3>(t, sp[3], n, d, acc, form == 5);
}

// The lane's partial sums of one ray: out[s] = (sum (sigma_s log2 e) w, sum
// (sigma_s log2 e) (nu - nu_s)^+ w) over its bins, w = s_nu e^-tau phi(x).
// sp: the lane's spectrum of emitter `cur`, read again when the ray's
// emitter is another one (a block's rays come emitter by emitter).
template <class Tab>
__device__ __forceinline__ void ray_bins(const Tab &t, const RayRec *__restrict__ rec,
                                         const float *__restrict__ specn, int lane, int &cur, float2 (&sp)[4],
                                         float2 (&out)[3]) {
  const float4 ra = *reinterpret_cast<const float4 *>(rec->n), rb = *reinterpret_cast<const float4 *>(rec->d);
  const int form = __float_as_int(ra.w), e = __float_as_int(rb.w);
  if (e != cur) {
    cur = e;
    const float4 *p = reinterpret_cast<const float4 *>(specn + (size_t)e * kNu) + 2 * lane;
    const float4 a = __ldg(p), b = __ldg(p + 1);
    sp[0] = make_float2(a.x, a.y);
    sp[1] = make_float2(a.z, a.w);
    sp[2] = make_float2(b.x, b.y);
    sp[3] = make_float2(b.z, b.w);
  }
  const float2 n[3] = {both(ra.x), both(ra.y), both(ra.z)}, d[3] = {both(rb.x), both(rb.y), both(rb.z)};
  float2 acc[6];
#pragma unroll
  for (int q = 0; q < 6; q++) acc[q] = both(0.f);
  if (form == 0) ray_stages<1, 0, 0, 0>(t, sp, n, d, acc);
  else if (form == 1) ray_stages<1, 1, 0, 0>(t, sp, n, d, acc);
  else if (form == 2) ray_stages<2, 1, 1, 1>(t, sp, n, d, acc);
  else ray_stages<2, 2, 2, 2>(t, sp, n, d, acc, form);
#pragma unroll
  for (int q = 0; q < 3; q++) out[q] = make_float2(acc[q].x + acc[q].y, acc[3 + q].x + acc[3 + q].y);
}

// Per-warp scratch of the FP32 rates: a chunk of 32 rays.
constexpr int kRoundRays = 4;
constexpr int kRedRow = 34;  // float2 per row: 16-byte reads of 8 rows fall on different banks
struct RateChunk {
  RayRec rec[32];
  float2 red[3 * kRoundRays][kRedRow];  // a round's lane sums, row 3 k + s: ray k, species s
  float out[32][6];  // prefactors P_s, then the rays' rates
};

// The rates of nq rays of a chunk (ray i is entry q[i], or i without q), S.out
// holding their prefactors: S.out[ray] = Gamma_s = P_s ln2 a_s, Heat_s = P_s ln2 b_s h nu_L.  All lanes
// of the warp take part; the caller synchronises the warp before and after.
// Rounds of kRoundRays rays: every lane leaves its three pairs of sums per
// ray in shared memory, then lane r and lane r + 16 add the lanes 0..15 and
// 16..31 of row r (a butterfly over the warp takes 60 instructions per ray,
// a recursive halving 25, this 10).
template <class Tab>
__device__ __forceinline__ void chunk_rates(RateChunk &S, const Tab &t, const float *__restrict__ specn,
                                            const int *q, int nq, int lane) {
  const float kLn2 = 0.69314718055994531f;
  const int row = lane & 15, kr = row / 3, s = row - 3 * kr;
  float2 sp[4];
  int cur = -1;
  for (int i = 0; i < nq; i += kRoundRays) {
    const int nr = min(kRoundRays, nq - i);
#pragma unroll 1
    for (int k = 0; k < nr; k++) {
      float2 o[3];
      ray_bins(t, &S.rec[q ? q[i + k] : i + k], specn, lane, cur, sp, o);
#pragma unroll
      for (int c = 0; c < 3; c++) S.red[3 * k + c][lane] = o[c];
    }
    __syncwarp();
    float2 sum = both(0.f);
    if (kr < nr) {
      const float4 *p = reinterpret_cast<const float4 *>(&S.red[row][lane & 16]);
      float4 v[8];
#pragma unroll
      for (int c = 0; c < 8; c++) v[c] = p[c];
#pragma unroll
      for (int o = 4; o; o >>= 1)
#pragma unroll
        for (int c = 0; c < o; c++)
          v[c] = make_float4(v[c].x + v[c + o].x, v[c].y + v[c + o].y, v[c].z + v[c + o].z, v[c].w + v[c + o].w);
      sum = make_float2(v[0].x + v[0].z, v[0].y + v[0].w);
    }
    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, 16);
    sum.y += __shfl_xor_sync(0xffffffffu, sum.y, 16);
    if (kr < nr && lane < 16) {
      const int ray = q ? q[i + kr] : i + kr;
      const float P = S.out[ray][s];
      S.out[ray][s] = P * (kLn2 * sum.x);
      S.out[ray][3 + s] = P * (kLn2 * sum.y) * kHNuLf;
    }
    __syncwarp();
  }
}

// Per-warp scratch of rate_block_f32.
struct RateWarpSmem {
  RateChunk c;
  float acc[12][32]; // per target lane: Kahan sums and compensations (CellSum6Smem)
  int q[32];         // lanes of the chunk's rays that take the quadrature
  int cnt[32], src[32];  // per target lane: rays of the chunk, ray of the round
};

// A cell's six rates summed over its rays in ray order, FP32 with Kahan
// compensation (a cell receives up to a few hundred rays).  CellSum6 keeps
// the sums in registers; CellSum6Smem in the warp's shared memory (word
// [q][lane], conflict-free), which frees twelve registers across the bin
// loop of the rate kernel.
struct CellSum6Smem {
  float (*a)[32];
  int lane;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 12; q++) a[q][lane] = 0.f;
  }
  __device__ __forceinline__ void add(const float *v) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      float s = a[q][lane], c = a[6 + q][lane];
      kahan_add(s, c, v[q]);
      a[q][lane] = s;
      a[6 + q][lane] = c;
    }
  }
  __device__ __forceinline__ float sum(int q) const { return a[q][lane]; }
};
struct CellSum6 {
  float s[6], c[6];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 6; q++) s[q] = c[q] = 0.f;
  }
  __device__ __forceinline__ void add(const float *v) {
#pragma unroll
    for (int q = 0; q < 6; q++) kahan_add(s[q], c[q], v[q]);
  }
  __device__ __forceinline__ float sum(int q) const { return s[q]; }
};

// Phase C of the block-rate kernels: lane k holds ray k of a chunk (its six
// values in out[k], its target lane t, -1 for none); every lane adds the
// rays that end in its cell, in ray order.  __match_any_sync ranks each ray
// among the chunk's rays with the same target; round r hands every cell
// its rank-r ray through `src`, so a chunk whose rays end in distinct cells
// takes one round (instead of every lane scanning the chunk's 32 rays).
template <class Acc>
__device__ __forceinline__ void add_chunk_in_order(Acc &acc, int lane, int t, const float (*out)[6], int *cnt,
                                                   int *src) {
  const unsigned same = __match_any_sync(0xffffffffu, t);
  const int rank = __popc(same & ((1u << lane) - 1u));
  cnt[lane] = 0;
  __syncwarp();
  if (t >= 0 && rank == 0) cnt[t] = __popc(same);
  const int rounds = __reduce_max_sync(0xffffffffu, t >= 0 ? rank + 1 : 0);
  __syncwarp();
  const int mine = cnt[lane];
  for (int r = 0; r < rounds; r++) {
    if (t >= 0 && rank == r) src[t] = lane;
    __syncwarp();
    if (r < mine) acc.add(out[src[lane]]);
    __syncwarp();
  }
}

// Phases A and B of a chunk of 32 rays [rc, min(rc + 32, r1)) of a block whose
// first cell is (bix, biy, biz): S.c.out holds the rays' rates; returns the
// target lane of ray rc + lane (-1: none).  Ends with the warp synchronised.
template <bool kServed>
__device__ __forceinline__ int rate_chunk(const GridDev &g, const float4 *__restrict__ raw,
                                          const float4 *__restrict__ emit_pos, const float *__restrict__ specn,
                                          const double *__restrict__ total, const RateLane &tab, int bix, int biy,
                                          int biz, uint64_t rc, uint64_t r1, const uint32_t *__restrict__ rays,
                                          uint64_t nray, const float *__restrict__ tau, RateWarpSmem &S, int lane,
                                          const float *__restrict__ pred) {
  const uint64_t r = rc + lane;
  int t = -1;
  bool quad = false;
  if (r < r1) {
    const uint32_t w = __ldg(rays + r);
    const uint32_t e = w >> 5;
    t = (int)(w & 31u);
    if (kServed && __ldg(pred + 6 * nray + r) != 0.f) {
#pragma unroll
      for (int s = 0; s < 6; s++) S.c.out[lane][s] = __ldg(pred + s * nray + r);
    } else {
      quad = true;
      const int lx = bix + (t >> 4), ly = biy + ((t >> 2) & 3), lz = biz + (t & 3);
      const float4 ep = __ldg(emit_pos + e);
      const float4 rw = __ldg(raw + cell_index(g, lx, ly, lz));
      const RayParams p = ray_params_f32(g, g.ix0 + lx, g.iy0 + ly, g.iz0 + lz, ep.x, ep.y, ep.z, __ldg(tau + r),
                                         __ldg(tau + nray + r), __ldg(tau + 2 * nray + r), rw, __ldg(total + e));
      S.c.rec[lane] = ray_rec(p, (int)e);
#pragma unroll
      for (int s = 0; s < 3; s++) S.c.out[lane][s] = p.P[s];
    }
  }
  int nq = (int)min((uint64_t)32, r1 - rc);
  if (kServed) {
    const unsigned m = __ballot_sync(0xffffffffu, quad);
    if (quad) S.q[__popc(m & ((1u << lane) - 1u))] = lane;
    nq = __popc(m);
  }
  __syncwarp();
  chunk_rates(S.c, tab, specn, kServed ? S.q : nullptr, nq, lane);
  __syncwarp();
  return t;
}

// The FP32 rates of one target block b whose rays are [r0, r1) of `rays`
// (columns in three planes of nray), written to its cells in rates6; one
// warp.  Phase A: per-ray parameters (ray_params_f32), one lane per ray, 32
// rays at a time.  Phase B: the chunk's rays one after another
// (chunk_rates).  Phase C: lane j adds the rays of cell j of the block in
// ray order (add_chunk_in_order).
// kServed: `pred` holds 7 planes of nray floats, six per-ray contributions
// and a flag; a ray whose flag is non-zero contributes those six values
// and skips the quadrature, which runs over the remaining rays of the
// chunk only (the surrogate's fallback).
template <bool kServed = false>
__device__ __forceinline__ void rate_block_f32(const GridDev &g, const float4 *__restrict__ raw,
                                               const float4 *__restrict__ emit_pos, const float *__restrict__ specn,
                                               const double *__restrict__ total, const RateLane &tab,
                                               uint64_t b, uint64_t r0, uint64_t r1,
                                               const uint32_t *__restrict__ rays, uint64_t nray,
                                               const float *__restrict__ tau, float *__restrict__ rates6,
                                               RateWarpSmem &S, int lane, const float *__restrict__ pred = nullptr) {
  const uint64_t ncell = (uint64_t)g.nx * g.ny * g.nz;
  int ix, iy, iz;
  const bool own_valid = block_cell(g, b, lane, &ix, &iy, &iz);
  const uint64_t own = own_valid ? cell_index(g, ix, iy, iz) : 0;
  CellSum6Smem acc{S.acc, lane};
  acc.zero();
  int bix, biy, biz;
  block_cell(g, b, 0, &bix, &biy, &biz);
  for (uint64_t rc = r0; rc < r1; rc += 32) {
    const int t = rate_chunk<kServed>(g, raw, emit_pos, specn, total, tab, bix, biy, biz, rc, r1, rays, nray, tau, S,
                                      lane, pred);
    add_chunk_in_order(acc, lane, t, S.c.out, S.cnt, S.src);
  }
  if (own_valid) {
#pragma unroll
    for (int s = 0; s < 6; s++) rates6[s * ncell + own] = acc.sum(s);
  }
}

// The same by a CTA of kWarps warps: they take the block's chunks in turn,
// kWarps at a time, then warps 0 to 2 add them in order, two of the six rates
// each (the same sums, bit for bit).  Starts and ends with its shared memory
// free (a barrier after the last use, but for the sums of the warps' own).
struct CellSumPair {
  float (*a)[32];
  int lane, q0;
  __device__ __forceinline__ void add(const float *v) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      float s = a[q0 + i][lane], c = a[6 + q0 + i][lane];
      kahan_add(s, c, v[q0 + i]);
      a[q0 + i][lane] = s;
      a[6 + q0 + i][lane] = c;
    }
  }
};
// Whether nblk blocks with nray rays take a CTA each rather than a warp, on a
// GPU that holds `ctas` CTAs of `warps` warps: when the fills of the GPU times
// the rounds of chunks in each are fewer.  Measured, CTA and warp: 32^3 cells /
// 8 sources (1024 blocks of 7 chunks) 88 and 110 us, 24^3 / 2 (432 of 2) 19 and
// 27, 32^3 / 5 (1024 of 5) 67 and 72, 48^3 / 64 (3456 of 46) 1.32 and 1.54 ms; but
// 32^3 / 1 (1024 of 1) 27 and 19 us, 52^3 / 1 (4394 of 1) 88 and 43, 36^3 / 5 (1458 of
// 5) 90 and 85.  With long blocks the CTAs also even out their differences, an
// eighth: the step of 8 batched problems of 32^3 / 30 in 4 parts (2048 blocks of
// about 19) 2.64 and 3.00 ms.  From two blocks per warp slot on the warps' waits
// for one another outweigh the better split: 64^3 / 16 (8192 of 14) 0.94 and
// 0.82 ms.
static inline bool cta_per_block(uint64_t nblk, uint64_t nray, uint64_t ctas, uint64_t warps) {
  const auto ceil_div = [](uint64_t a, uint64_t b) { return (a + b - 1) / b; };
  if (nblk == 0 || nblk >= 2 * ctas * warps) return false;
  const uint64_t chunks = ceil_div(nray, 32 * nblk);
  const uint64_t by_cta = ceil_div(nblk, ctas) * ceil_div(chunks, warps);
  const uint64_t by_warp = ceil_div(nblk, ctas * warps) * chunks;
  return 8 * by_cta < (chunks > warps ? 9 : 8) * by_warp;
}
template <int kWarps>
__device__ __forceinline__ void rate_block_f32_cta(const GridDev &g, const float4 *__restrict__ raw,
                                                   const float4 *__restrict__ emit_pos,
                                                   const float *__restrict__ specn, const double *__restrict__ total,
                                                   const RateLane &tab, uint64_t b, uint64_t r0, uint64_t r1,
                                                   const uint32_t *__restrict__ rays, uint64_t nray,
                                                   const float *__restrict__ tau, float *__restrict__ rates6,
                                                   RateWarpSmem (&S)[kWarps], int (&t)[kWarps][32]) {
  static_assert(kWarps >= 3, "three warps add a block's rates");
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint64_t ncell = (uint64_t)g.nx * g.ny * g.nz;
  int ix, iy, iz, bix, biy, biz;
  const bool own_valid = block_cell(g, b, lane, &ix, &iy, &iz);
  block_cell(g, b, 0, &bix, &biy, &biz);
  CellSumPair acc{S[0].acc, lane, 2 * wib};
  if (wib < 3) {
#pragma unroll
    for (int i = 0; i < 2; i++) acc.a[acc.q0 + i][lane] = acc.a[6 + acc.q0 + i][lane] = 0.f;
  }
  for (uint64_t rs = r0; rs < r1; rs += 32 * kWarps) {
    const uint64_t rc = rs + 32 * wib;
    t[wib][lane] = rc < r1 ? rate_chunk<false>(g, raw, emit_pos, specn, total, tab, bix, biy, biz, rc, r1, rays, nray,
                                               tau, S[wib], lane, nullptr)
                           : -1;
    __syncthreads();
    if (wib < 3) {
      for (int v = 0; v < kWarps; v++)
        add_chunk_in_order(acc, lane, t[v][lane], S[v].c.out, S[wib].cnt, S[wib].src);
    }
    __syncthreads();
  }
  if (wib < 3 && own_valid) {
    const uint64_t own = cell_index(g, ix, iy, iz);
#pragma unroll
    for (int i = 0; i < 2; i++) rates6[(acc.q0 + i) * ncell + own] = acc.a[acc.q0 + i][lane];
  }
}

}  // namespace argot
