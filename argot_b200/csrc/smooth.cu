// smooth.cu -- the photo-ionisation-rate smoothing of smooth_photoion_rate.c
// on the device, so that the rates stay in HBM through the iteration loop
// (the reference copies them to the host, smooths there and copies back).
//
// Per cell and field: the 27 cells ix-1..ix+1 (outer), iy-1..iy+1,
// iz-1..iz+1 (inner) with the centre weighted by 30, summed in the
// reference's order and precision (smooth_photoion_rate.c:1060-1517): the
// first 13 terms in single precision, the weighted centre and the rest in
// double (its double literal promotes the running sum), times 1/56 in
// double, stored as float.  At the mesh faces: a copy of the nearest cell
// (the reference's default build, `isolated = yes`, with no neighbour rank)
// or the periodic image.  Bit-identical to the reference.
#include <algorithm>

#include "march.cuh"

namespace argot {

// A thread takes two cells next to each other along y and walks kRun planes
// along x.  The two planes behind stay in registers, a plane's four rows are
// one load each (read a plane ahead), the neighbours along z come from the
// lanes beside (the warp's ends load theirs), and a value is converted to
// double once.  The sums keep their order, so nothing of them is shared
// between cells.  Per cell that leaves 2 loads of the 27, 6 conversions of
// 14, and 12 single and 15 double additions.
// Measured, six planes of 256^3 cells: 1.18 ms with 27 loads per cell (each
// two L1 lines per warp), 0.55 ms here (one cell along y per thread 0.68 ms);
// 805 MB, 0.125 ms at the copy rate.
// What bounds it: the latency of a plane's loads and conversions at the 16
// warps per SM that 128 registers allow (issue 48%; 3 CTAs: 0.69 ms, 5: 0.59).
constexpr int kRun = 24, kSmoothThreads = 128;
template <bool kIsolated>
__device__ __forceinline__ int face_index(int i, int n) {
  if (i < 0) return kIsolated ? 0 : n - 1;
  if (i >= n) return kIsolated ? n - 1 : 0;
  return i;
}

template <bool kIsolated>
__global__ void __launch_bounds__(kSmoothThreads, 4)
    k_smooth(int nx, int ny, int nz, int run, const float *__restrict__ in, float *__restrict__ out) {
  const uint32_t nyz = (uint32_t)ny * (uint32_t)nz;
  const uint64_t ncell = (uint64_t)nx * nyz;
  const double kNormal = 1.0 / (30.0 + 26.0);
  const int lane = threadIdx.x & 31;
  // warps over (segment along x, pair of rows, chunk of 32 cells along z)
  const uint32_t nch = (uint32_t)(nz + 31) / 32, npair = (uint32_t)(ny + 1) / 2;
  const uint32_t w = blockIdx.x * (kSmoothThreads / 32) + (threadIdx.x >> 5);
  const uint32_t row = w / nch, seg = row / npair;
  const int x0 = (int)seg * run, y0 = 2 * (int)(row - seg * npair);
  if (x0 >= nx) return;  // (whole warps)
  const int iz = (int)(w - row * nch) * 32 + lane;
  const int z = min(iz, nz - 1), x1 = min(x0 + run, nx);
  // the warp's ends: lane 0 loads its lower neighbour, lane 31 and the lane of
  // the last cell their upper one; `both`: one lane is both
  const bool own_m = lane == 0, own_p = lane == 31 || iz == nz - 1, both = own_m && own_p;
  const int zm = face_index<kIsolated>(z - 1, nz), zp = face_index<kIsolated>(z + 1, nz);
  const float *__restrict__ f = in + blockIdx.y * ncell;
  uint32_t at[4];  // the four rows' offsets in a plane
#pragma unroll
  for (int j = 0; j < 4; j++) at[j] = (uint32_t)face_index<kIsolated>(y0 + j - 1, ny) * (uint32_t)nz;
  struct Rows {
    float c[4], e[4], e2[4];
  };
  auto read = [&](int ix, Rows &r) {
    const float *p = f + (uint64_t)((uint32_t)face_index<kIsolated>(ix, nx) * (uint64_t)nyz);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      r.c[j] = __ldg(p + (at[j] + (uint32_t)z));
      if (own_m || own_p) r.e[j] = __ldg(p + (at[j] + (uint32_t)(own_m ? zm : zp)));
    }
    if (both) {
#pragma unroll
      for (int j = 0; j < 4; j++) r.e2[j] = __ldg(p + (at[j] + (uint32_t)zp));
    }
  };
  auto spread = [&](const Rows &r, float (&v)[12]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float m = __shfl_up_sync(0xffffffffu, r.c[j], 1), q = __shfl_down_sync(0xffffffffu, r.c[j], 1);
      v[3 * j] = own_m ? r.e[j] : m;
      v[3 * j + 1] = r.c[j];
      v[3 * j + 2] = own_p ? (both ? r.e2[j] : r.e[j]) : q;
    }
  };
  // planes ix - 1, ix, ix + 1 in single precision and the last two in double,
  // the arrays' roles rotating with ix
  float v[3][12];
  double d[2][12];
  Rows ahead;
  read(x0 - 1, ahead);
  spread(ahead, v[0]);
  read(x0, ahead);
  spread(ahead, v[1]);
#pragma unroll
  for (int k = 4; k < 12; k++) d[0][k] = (double)v[1][k];
  read(x0 + 1, ahead);
  float *po = out + blockIdx.y * ncell + (uint64_t)x0 * nyz + (uint32_t)y0 * (uint32_t)nz + (uint32_t)iz;
  const bool in_z = iz < nz, two = in_z && y0 + 1 < ny;
  for (int xb = x0; xb < x1; xb += 6) {
#pragma unroll
    for (int u = 0; u < 6; u++) {
      if (xb + u >= x1) break;
      float(&p0)[12] = v[u % 3], (&p1)[12] = v[(u + 1) % 3], (&p2)[12] = v[(u + 2) % 3];
      double(&d1)[12] = d[u % 2], (&d2)[12] = d[(u + 1) % 2];
      spread(ahead, p2);
      read(min(xb + u + 2, x1), ahead);
#pragma unroll
      for (int k = 0; k < 12; k++) d2[k] = (double)p2[k];
#pragma unroll
      for (int h = 0; h < 2; h++) {  // the two cells: rows h, h + 1, h + 2
        float acc = p0[3 * h];
#pragma unroll
        for (int k = 1; k < 9; k++) acc = __fadd_rn(acc, p0[3 * h + k]);
#pragma unroll
        for (int k = 0; k < 4; k++) acc = __fadd_rn(acc, p1[3 * h + k]);
        double s = __dadd_rn((double)acc, __dmul_rn(30.0, d1[3 * h + 4]));
#pragma unroll
        for (int k = 5; k < 9; k++) s = __dadd_rn(s, d1[3 * h + k]);
#pragma unroll
        for (int k = 0; k < 9; k++) s = __dadd_rn(s, d2[3 * h + k]);
        if (h ? two : in_z) po[h ? (uint32_t)nz : 0u] = __double2float_rn(__dmul_rn(kNormal, s));
      }
      po += nyz;
    }
  }
}

// The same with one thread per cell and no sharing between cells: 27 loads
// per cell and plane, but no lane without a cell on a thin mesh.
template <bool kIsolated>
__global__ void __launch_bounds__(256)
    k_smooth_flat(int nx, int ny, int nz, const float *__restrict__ in, float *__restrict__ out, int nplanes) {
  const uint64_t ncell = (uint64_t)nx * ny * nz;
  const double kNormal = 1.0 / (30.0 + 26.0);
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < ncell;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t row = (uint32_t)c / (uint32_t)nz, ix = row / (uint32_t)ny;
    const int at[3] = {(int)ix, (int)(row - ix * (uint32_t)ny), (int)((uint32_t)c - row * (uint32_t)nz)};
    uint32_t jx[3], jy[3], jz[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      jx[a] = (uint32_t)face_index<kIsolated>(at[0] + a - 1, nx);
      jy[a] = (uint32_t)face_index<kIsolated>(at[1] + a - 1, ny);
      jz[a] = (uint32_t)face_index<kIsolated>(at[2] + a - 1, nz);
    }
    uint32_t off[27];
#pragma unroll
    for (int k = 0; k < 27; k++)
      off[k] = (jx[k / 9] * (uint32_t)ny + jy[k / 3 % 3]) * (uint32_t)nz + jz[k % 3];
#pragma unroll 1
    for (int s = 0; s < nplanes; s++) {
      const float *__restrict__ f = in + s * ncell;
      float acc = __ldg(f + off[0]);
#pragma unroll
      for (int k = 1; k < 13; k++) acc = __fadd_rn(acc, __ldg(f + off[k]));
      double d = __dadd_rn((double)acc, __dmul_rn(30.0, (double)__ldg(f + off[13])));
#pragma unroll
      for (int k = 14; k < 27; k++) d = __dadd_rn(d, (double)__ldg(f + off[k]));
      out[s * ncell + c] = __double2float_rn(__dmul_rn(kNormal, d));
    }
  }
}

// Which kernel a mesh takes.  k_smooth's time goes with the slots it fills,
// lanes with or without a cell: fills of the GPU (kSmoothWarps warps per SM)
// times the planes a warp steps through, two of them read ahead, times 64
// cells per warp.  On a thin mesh (few cells along z or y, one plane along
// x) most slots hold no cell.  The line lies at kSlotsPerCell slots per cell
// (measured over 290 meshes: 512 x 512 x 4 195 us in runs against 58 us flat,
// 256 x 256 x 14 53 and 50, 256 x 256 x 16 53 and 54, 256 x 256 x 33 123 and 134);
// up to kFewSteps plane steps in all, both take about 10 us.
constexpr uint64_t kSmoothWarps = 16, kFewSteps = 16;
constexpr double kSlotsPerCell = 2.9;

// Smooths nplanes planes of ncell floats (in -> out).
int launch_smooth_planes(int nx, int ny, int nz, const float *in, float *out, int nplanes, int isolated,
                         cudaStream_t st) {
  const uint64_t ncell = (uint64_t)nx * ny * nz;
  if (!ncell || nplanes <= 0) return 0;
  const int sms = device_sms();
  // shorter segments where the mesh would leave the GPU's warps idle
  const uint64_t columns = (uint64_t)((ny + 1) / 2) * ((nz + 31) / 32), slots = kSmoothWarps * sms;
  int run = kRun;
  while (run > 3 && columns * ((nx + run - 1) / run) * (uint64_t)nplanes < slots) run /= 2;
  const uint64_t warps = columns * ((nx + run - 1) / run);
  const uint64_t steps = (warps * nplanes + slots - 1) / slots * (std::min(run, nx) + 2);
  if (steps > kFewSteps && (double)(steps * slots * 64) > kSlotsPerCell * (double)ncell * nplanes) {
    const unsigned blocks = (unsigned)std::min<uint64_t>((ncell + 255) / 256, (uint64_t)sms * 8);
    if (isolated)
      k_smooth_flat<true><<<blocks, 256, 0, st>>>(nx, ny, nz, in, out, nplanes);
    else
      k_smooth_flat<false><<<blocks, 256, 0, st>>>(nx, ny, nz, in, out, nplanes);
    ARGOT_CUDA_TRY(cudaGetLastError());
    return 0;
  }
  const dim3 grid((unsigned)((warps + kSmoothThreads / 32 - 1) / (kSmoothThreads / 32)), (unsigned)nplanes);
  if (isolated)
    k_smooth<true><<<grid, kSmoothThreads, 0, st>>>(nx, ny, nz, run, in, out);
  else
    k_smooth<false><<<grid, kSmoothThreads, 0, st>>>(nx, ny, nz, run, in, out);
  ARGOT_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace argot

using namespace argot;

extern "C" {

int argot_b200_smooth_rates(const argot_b200_grid *gp, const float *in6, float *out6, int isolated, void *stream) {
  if (!grid_valid(gp) || !in6 || !out6 || in6 == out6 || (isolated != 0 && isolated != 1)) {
    set_status(ARGOT_B200_EINVAL);
    return ARGOT_B200_EINVAL;
  }
  const uint64_t ncell = (uint64_t)gp->nx * gp->ny * gp->nz;
  if (ncell >= (1ull << 32)) { set_status(ARGOT_B200_EINVAL); return ARGOT_B200_EINVAL; }
  const int rc = launch_smooth_planes(gp->nx, gp->ny, gp->nz, in6, out6, 6, isolated, (cudaStream_t)stream);
  if (rc) return rc;
  set_status(0);
  return 0;
}

}  // extern "C"
