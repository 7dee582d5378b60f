// 3D-weighted helical parallel-cone backprojection (plain FP32 and FP64 forms).
//
// Reference: src/Parallel_FDK_Helical_3DWeighting.cpp:42-113 (CPU, the parity
// target) and src/ParallelFDKHelical3DWeightingGPU.cu:14-87 (GPU). For voxel
// (x, y, z): s0 = ceil((2 pi z/h - BetaS)/DeltaFai - 0.5), views
// s0 -/+ ceil(N_pi HSCoef) clamped to [0, PN-1] (the CPU loop; the reference
// GPU loop starts at view 0 and reads w[] out of bounds for far views), and
// per view: UU, Yr, temp1 = sqrt(SO^2 - Yr^2), temp2 = z - h View/2pi,
// Zr = temp2 SO SD/(UU temp1 + SO^2 - Yr^2), U = ceil(Yr/dYL + YLC),
// V = ceil(Zr/dZL + ZLC), bilinear tap if 0 < U < YL and 0 < V < ZL, and the
// 3D weight w[d1] Gama_C^k1 / (w[d2] Gama^k1 + w[d1] Gama_C^k1).
//
// Index selection is bit-exact to the CPU path: x, y, z, s0, UU, Yr, temp1,
// U1 and temp2 are evaluated in double with the reference's operation order
// through non-contracting __d*_rn intrinsics, from per-view cos/sin/h*View/2pi
// tables that the plan computes on the host with the same C library calls. V
// (and, in the kernels with table weights, U) is first located with an estimate
// whose error is known; only when that lies so close to an integer that ceil()
// could disagree is it recomputed with the reference's own operations.
//
// Work decomposition: a thread owns NZ consecutive voxels of one (x, y)
// column. Everything that does not depend on z (the trig, UU, Yr, temp1, U,
// Dey, the projection slope, 1/(temp1 +- UU)) is computed once per column and
// view and reused for the NZ voxels; the NZ windows [s1, s2] are uniform over
// the CTA (all its threads share the z block), so the per-voxel window test
// is a uniform branch. A warp is an 8 x 4 (x, y) tile, which keeps its 32
// detector taps within a few cache lines of one or two rows.
#include <cmath>
#include <vector>

#include "hr_internal.h"
#include "bp_fast.h"

namespace {

constexpr int kBx = 8, kBy = 16;  // CTA tile (x, y); warps are 8 x 4
constexpr double kTwoPiTrunc = 2.0 * 3.14159265358979;         // ..._3DWeighting.cpp:16,62
constexpr double kInvTwoPi = 1.0 / (2.0 * 3.141592653589793);  // :51,79

struct ViewTab {
  double c, s, hv;  // cos(View), sin(View), h*View*invPI
};

struct BpParams {
  int XN, YN, ZN, YL, ZL, PN, N_2pi, half;
  int qcap;  // longest union view window of a z block of the plain kernel (its weight table rows)
  double XNC, YNC, ZNC, dx, dy, dz, YLC, ZLC, dYL, dZL, h, BetaS, DeltaFai, N_pi, SO, SD, k1;
  double SO2, SOSD, SOSDdZL, invdYL;
  float k1f, DeltaFaif;
};

}  // namespace

struct hr_bp_plan {
  BpParams prm;
  int form;
  ViewTab* d_views;
  float* d_w;
  double* d_wd;
  hr::BpFastGeom fg;
  hr::BpFast fast;
};

namespace {

// Voxel centre and central view, exactly as the CPU reference.
struct ZInfo {
  double z;
  int s0, lo, hi;
};

__device__ __forceinline__ ZInfo z_info(const BpParams& P, int zi) {
  ZInfo r;
  r.z = __dmul_rn(__dsub_rn((double)zi, P.ZNC), P.dz);
  const double beta0 = __ddiv_rn(__dmul_rn(kTwoPiTrunc, r.z), P.h);
  const double sarg = __dsub_rn(__ddiv_rn(__dsub_rn(beta0, P.BetaS), P.DeltaFai), 0.5);
  r.s0 = (int)ceil(sarg);
  const int s1 = r.s0 - P.half, s2 = r.s0 + P.half;
  if (zi < P.ZN && s1 < P.PN && s2 > 0) {
    r.lo = s1 < 0 ? 0 : s1;
    r.hi = s2 > P.PN - 1 ? P.PN - 1 : s2;
  } else {
    r.lo = 0x7fffffff;
    r.hi = -0x7fffffff;
  }
  return r;
}

// Per (column, view) quantities.
struct ColView {
  int U;          // channel of the upper tap
  double U1;      // Yr/dYL + YLC
  double denom;   // UU*temp1 + SO^2 - Yr^2
  double A, B;    // temp1 + UU, temp1 - UU
  double slope;   // SO SD / dZL / denom
};

__device__ __forceinline__ ColView col_view(const BpParams& P, double x, double y, const ViewTab& v) {
  ColView r;
  const double UU = __dsub_rn(__dmul_rn(-x, v.c), __dmul_rn(y, v.s));
  const double Yr = __dadd_rn(__dmul_rn(-x, v.s), __dmul_rn(y, v.c));
  const double Yr2 = __dmul_rn(Yr, Yr);
  const double temp1 = __dsqrt_rn(__dsub_rn(P.SO2, Yr2));
  r.denom = __dsub_rn(__dadd_rn(__dmul_rn(UU, temp1), P.SO2), Yr2);
  r.U1 = __dadd_rn(__ddiv_rn(Yr, P.dYL), P.YLC);
  r.U = (int)ceil(r.U1);
  r.A = __dadd_rn(temp1, UU);
  r.B = __dsub_rn(temp1, UU);
  r.slope = P.SOSDdZL / r.denom;
  return r;
}

// Row index V and its fraction Dez = V - V1, bit-exact to the reference.
__device__ __forceinline__ int row_index(const BpParams& P, const ColView& cv, double temp2, double& dez) {
  const double v1a = fma(temp2, cv.slope, P.ZLC);
  int V = (int)ceil(v1a);
  double d = (double)V - v1a;
  if (d < 1e-9 || d > 1.0 - 1e-9) {
    const double Zr = __ddiv_rn(__dmul_rn(temp2, P.SOSD), cv.denom);
    const double V1 = __dadd_rn(__ddiv_rn(Zr, P.dZL), P.ZLC);
    V = (int)ceil(V1);
    d = __dsub_rn((double)V, V1);
  }
  dez = d;
  return V;
}

// ---------------------------------------------------------------------------
// Plain form: FP32 filtered data, FP32 weights and accumulation.
// ---------------------------------------------------------------------------
template <int NZ>
__global__ void __launch_bounds__(kBx* kBy) bp_plain_kernel(float* __restrict__ vol, const float* __restrict__ fp,
                                                           const ViewTab* __restrict__ views,
                                                           const float* __restrict__ gw, BpParams P) {
  extern __shared__ float w_s[];  // [N_2pi]
  for (int t = threadIdx.y * kBx + threadIdx.x; t < P.N_2pi; t += kBx * kBy) w_s[t] = gw[t];
  __syncthreads();
  const int xi = blockIdx.x * kBx + threadIdx.x;
  const int yi = blockIdx.y * kBy + threadIdx.y;
  const int z0 = blockIdx.z * NZ;
  if (xi >= P.XN || yi >= P.YN) return;
  const double x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  const double y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  ZInfo zin[NZ];
  float res[NZ];
  int pstart = 0x7fffffff, pend = -0x7fffffff;
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    zin[m] = z_info(P, z0 + m);
    res[m] = 0.0f;
    pstart = min(pstart, zin[m].lo);
    pend = max(pend, zin[m].hi);
  }
  const size_t plane = (size_t)P.ZL * P.YL;
  for (int p = pstart; p <= pend; ++p) {
    const ViewTab v = views[p];
    const ColView cv = col_view(P, x, y, v);
    if (cv.U <= 0 || cv.U >= P.YL) continue;
    const float dey = (float)((double)cv.U - cv.U1);
    const float invA = 1.0f / (float)cv.A, invB = 1.0f / (float)cv.B;
    const float* col = fp + (size_t)p * plane + (cv.U - 1);
#pragma unroll
    for (int m = 0; m < NZ; ++m) {
      if (p < zin[m].lo || p > zin[m].hi) continue;
      const double temp2 = __dsub_rn(zin[m].z, v.hv);
      double dezd;
      const int V = row_index(P, cv, temp2, dezd);
      if (V <= 0 || V >= P.ZL) continue;
      const float dez = (float)dezd;
      const float* r0 = col + (size_t)(V - 1) * P.YL;
      const float* r1 = r0 + P.YL;
      const float ra = dey * __ldg(r0) + (1.0f - dey) * __ldg(r0 + 1);
      const float rb = dey * __ldg(r1) + (1.0f - dey) * __ldg(r1 + 1);
      const float touying = dez * ra + (1.0f - dez) * rb;
      const int before = p < zin[m].s0;
      const int d1 = (int)(P.N_pi - (double)(zin[m].s0 - p));
      const int d2 = before ? (int)(d1 + P.N_pi) : (int)(d1 - P.N_pi);
      const float w1 = w_s[d1], w2 = w_s[d2];
      const float t2 = (float)temp2;
      const float gama = fabsf(t2) * invA;
      const float gamac = fabsf(before ? t2 - 0.5f : t2 + 0.5f) * invB;
      const float e = exp2f(P.k1f * (log2f(gama) - log2f(gamac)));
      const float weight = w1 / (w1 + w2 * fminf(e, 3.0e38f));
      res[m] += weight * touying;
    }
  }
  float* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
#pragma unroll
  for (int m = 0; m < NZ; ++m)
    if (z0 + m < P.ZN) out[m] = res[m] * P.DeltaFaif;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---- index estimates of the table-weight kernels ----
// Positions are FP64 values read as 64-bit fixed point with 32 fraction bits:
// adding 1.5 * 2^20 leaves them in the low mantissa bits (|x| < 2^19), one
// FP64 add instead of the conversion instructions (an eighth of the FP32 rate).
constexpr double kFixMagic = 1572864.0;            // 1.5 * 2^20
constexpr long long kFixBits = 0x4138000000000000;  // its bit pattern
constexpr double kBig = 1e150;                     // bound of the FP64 weight factors
constexpr double kFixLimit = 262144.0;             // 2^18: positions of a column must lie inside +-this

__device__ __forceinline__ long long to_fix(double x) { return __double_as_longlong(__dadd_rn(x, kFixMagic)) - kFixBits; }

__device__ __forceinline__ double rcp64_approx(double x) {  // ~2^-20 relative
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt64_approx(double x) {  // ~2^-20 relative
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// One update with the reference's own index arithmetic: the weight times the
// bilinear tap of (column, view, slice), 0 outside the detector. The
// table-weight kernel comes here when an estimate lies too close to an integer
// or out of range.
__device__ __forceinline__ float plain_update_exact(const BpParams& P, const float* __restrict__ fp, const ViewTab v,
                                                 int p, double x, double y, double z, float q2) {
  const ColView cv = col_view(P, x, y, v);
  if (cv.U <= 0 || cv.U >= P.YL) return 0.0f;
  double dezd;
  const int V = row_index(P, cv, __dsub_rn(z, v.hv), dezd);
  if (V <= 0 || V >= P.ZL) return 0.0f;
  const float dey = (float)((double)cv.U - cv.U1), dez = (float)dezd;
  const float E = fminf(exp2f(P.k1f * log2f((float)cv.B / (float)cv.A)), 3.0e38f);
  const float* r0 = fp + ((size_t)p * P.ZL + (V - 1)) * P.YL + (cv.U - 1);
  const float* r1 = r0 + P.YL;
  const float ra = dey * r0[0] + (1.0f - dey) * r0[1];
  const float rb = dey * r1[0] + (1.0f - dey) * r1[1];
  return rcp_approx(fmaf(q2, E, 1.0f)) * (dez * ra + (1.0f - dez) * rb);
}

// Plain form with the 3D weight factored (the same split as the fast form):
//   weight = w1 Gc^k1 / (w2 G^k1 + w1 Gc^k1) = 1 / (1 + Q2(view, slice) E(column, view))
//   Q2 = (w2 / w1) (|t2| / |t2 -/+ 0.5|)^k1,   E = ((temp1 - UU) / (temp1 + UU))^k1.
// Each CTA (one z block of NZ slices) first tabulates Q2 for its union view
// window in shared memory (FP64, -1 where the view is outside the slice's
// window), so an update costs one table read, one FMA and one reciprocal for
// its weight instead of two logarithms, an exponential and a division.
//
// What bounds it is instruction issue: its predecessor spent 75 instructions per
// update, a third of them FP64 square roots, divisions and conversions per
// (column, view), the rest conversions and FP64 compares per update. Here the
// per-(column, view) values are FP64 estimates (approximate reciprocal and
// reciprocal square root, one Newton step: 5e-12 relative), and because the
// slices of a column are equally spaced, so are its detector rows: V of slice m
// is a 64-bit fixed-point start plus m steps, two integer adds; its fraction
// becomes a float through one funnel shift and one add. Selection stays exact:
// the estimates are off by less than 64 units of 2^-32 row (half a unit for the
// start, half per step, and the FP64 error, 1.3 units at 64 rows), and where any
// of four slices lies within 7.5e-8 of an integer row, or the channel within
// 1.5e-8, those slices take plain_update_exact. A start carries +256 units so
// that dropping the fraction's low 9 bits rounds to nearest. Rows are linear in
// the slice, so the first and last of four tell whether all lie on the detector
// (no clamps or tests) or all off one side of it (skipped).
// Measured on two rotations of 888 x 64 -> 512 x 512 x 48 (8.4e9 updates):
// 28.8 -> 14.4 ms, 47 instructions per update at 73 % issue, L1 hits 92 %.
// 64 registers (4 CTAs of 256 per SM) 15.24 ms for the chain, 80: 15.53, 96:
// 17.8; CTAs of 128, which tabulate Q2 twice as often, are slower still.
constexpr uint32_t kFixRound = 256;             // half of the 9 dropped fraction bits
constexpr uint32_t kFixNear = 64;               // more than the estimates' error
constexpr int kTx = 8, kTy = 32;                // CTA tile (x, y)

// ---- packed FP32x2 arithmetic (one instruction for two slices) ----
constexpr uint64_t kOne2 = 0x3f8000003f800000ull, kNegOne2 = 0xbf800000bf800000ull;
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void up2(uint64_t r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a + f (b - a). WEIGHTED: (1 - f) a + f b, which stays infinite, with its sign, where one of them is (the
// difference form is then NaN) and does not overflow where both are finite.
template <bool WEIGHTED>
__device__ __forceinline__ uint64_t lerp2(uint64_t f, uint64_t a, uint64_t b) {
  if constexpr (WEIGHTED) return fma2(f, b, mul2(sub2(kOne2, f), a));
  return fma2(f, sub2(b, a), a);
}
template <bool WEIGHTED>
__device__ __forceinline__ double lerp(double f, double a, double b) {
  if constexpr (WEIGHTED) return fma(f, b, (1.0 - f) * a);
  return fma(f, b - a, a);
}

// Data pointer plus a row's bytes in one wide multiply-add.
template <class T>
__device__ __forceinline__ const T* row_ptr(const T* base, uint32_t row, uint32_t pitch_bytes) {
  uint64_t p;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p) : "r"(row), "r"(pitch_bytes), "l"(reinterpret_cast<uint64_t>(base)));
  return reinterpret_cast<const T*>(p);
}
// Four slices of a column, from `first`: their taps, two slices to a packed
// register pair, weighted and added. TEST: slices whose row is off the detector
// or whose q2 is negative are left out (else all are known to count).
template <int NZ, bool TEST, bool WEIGHTED>
__device__ __forceinline__ void plain_group(float (&res)[NZ], int first, const uint32_t (&row)[4], uint32_t rows,
                                            const float (&fz)[4], const float* c0, const float* c1, uint32_t pitch,
                                            uint64_t ux2, uint64_t E2, float4 q4) {
  float a0[4], b0[4], a1[4], b1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t r = TEST ? min(row[i], rows - 1) : row[i];  // a row off the detector reads the last one
    const float* p0 = row_ptr(c0, r, pitch);
    const float* p1 = row_ptr(c1, r, pitch);
    a0[i] = __ldg(p0);
    b0[i] = __ldg(p0 + 1);
    a1[i] = __ldg(p1);
    b1[i] = __ldg(p1 + 1);
  }
  const float q2[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint64_t A0 = pk2(a0[i], a0[i + 1]), A1 = pk2(a1[i], a1[i + 1]);
    const uint64_t ra = lerp2<WEIGHTED>(ux2, A0, pk2(b0[i], b0[i + 1]));
    const uint64_t rb = lerp2<WEIGHTED>(ux2, A1, pk2(b1[i], b1[i + 1]));
    const uint64_t f2 = add2(pk2(fz[i], fz[i + 1]), kNegOne2);  // [1, 2) -> [0, 1)
    float tap[2], den2[2];
    up2(lerp2<WEIGHTED>(f2, ra, rb), tap[0], tap[1]);
    up2(fma2(pk2(q2[i], q2[i + 1]), E2, kOne2), den2[0], den2[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float sum = fmaf(rcp_approx(den2[k]), tap[k], res[first + i + k]);
      if (!TEST || (row[i + k] < rows && q2[i + k] >= 0.0f)) res[first + i + k] = sum;
    }
  }
}

struct PlainColumn {
  const float* fp;        // filtered data
  const ViewTab* views;
  const float* q_s;       // the block's Q2 table, first row = view pstart
  const double* z_s;
  double x, y, z00;       // column, first slice's z
  int pstart;
};

// Views [q0, q1) of the block's union window for one column. ALL: every slice
// of the block has every view of the range in its window (no window tests).
template <int NZ, bool ALL, bool WEIGHTED = false>
__device__ __forceinline__ void plain_views(float (&res)[NZ], const PlainColumn& C, const BpParams& P, int q0, int q1) {
  const size_t plane = (size_t)P.ZL * P.YL;
  const uint32_t rows = (uint32_t)(P.ZL - 1), chans = (uint32_t)(P.YL - 1);
  const uint32_t pitch = (uint32_t)P.YL * (uint32_t)sizeof(float);
  const float* view = C.fp + (size_t)(C.pstart + q0) * plane;
#pragma unroll 1
  for (int q = q0; q < q1; ++q, view += plane) {
    const ViewTab v = C.views[C.pstart + q];
    // ---- per (column, view): channel, row of the first slice, rows per slice ----
    const double UU = fma(-C.x, v.c, -(C.y * v.s));
    const double Yr = fma(-C.x, v.s, C.y * v.c);
    const long long fu = to_fix(fma(Yr, P.invdYL, P.YLC));
    const uint32_t u = (uint32_t)(fu >> 32);
    uint32_t near = ((uint32_t)fu + kFixNear) < 2 * kFixNear ? 0u : 0xffffffffu;
    if (u >= chans && near) continue;  // U <= 0 or U >= YL
    const double t1sq = fma(-Yr, Yr, P.SO2);
    const double ry = rsqrt64_approx(t1sq);
    const double g = t1sq * ry;
    const double temp1 = fma(fma(-g, g, t1sq), 0.5 * ry, g);
    const double den = fma(temp1, UU, t1sq);  // temp1 (temp1 + UU)
    double rd = rcp64_approx(den);
    rd = fma(fma(-den, rd, 1.0), rd, rd);
    const double slope = rd * P.SOSDdZL;
    const double v0 = fma(C.z00 - v.hv, slope, P.ZLC);
    const double dv = slope * P.dz;
    if (!(fabs(v0) + NZ * fabs(dv) < kFixLimit)) near = 0u;  // also NaN
    unsigned long long F = (unsigned long long)to_fix(v0) + kFixRound;
    const unsigned long long S = (unsigned long long)to_fix(dv);
    // (temp1 - UU) / (temp1 + UU) = (temp1 - UU) temp1 / den
    const float E = fminf(exp2f(P.k1f * log2f((float)(fma(-temp1, UU, t1sq) * rd))), 3.0e38f);
    const float ux = (float)(uint32_t)fu * 2.3283064365386963e-10f;  // 2^-32
    const uint64_t ux2 = pk2(ux, ux), E2 = pk2(E, E);
    const float* c0 = view + min(u, chans - 1);
    const float* c1 = c0 + P.YL;
    const float4* qrow = reinterpret_cast<const float4*>(C.q_s + q * NZ);
#pragma unroll
    for (int h = 0; h < NZ / 4; ++h) {
      uint32_t row[4], close = near;
      float fz[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t lo = (uint32_t)F;
        row[i] = (uint32_t)(F >> 32);
        close = __viaddmin_u32(lo, kFixNear, close);
        fz[i] = __uint_as_float(__funnelshift_r(lo, 127u, 9));  // 127 << 23 | lo >> 9: 1 + fraction
        F += S;
      }
      if (!ALL) {
        const float4 t = qrow[h];
        if (fmaxf(fmaxf(t.x, t.y), fmaxf(t.z, t.w)) < 0.0f) continue;  // uniform over the CTA
      }
      if (close < 2 * (kFixRound + kFixNear)) {
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          const float qi = C.q_s[q * NZ + 4 * h + i];
          if (qi < 0.0f) continue;
          const float r = plain_update_exact(P, C.fp, v, C.pstart + q, C.x, C.y, C.z_s[4 * h + i], qi);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k == i) res[4 * h + k] += r;
        }
        continue;
      }
      // rows are linear in the slice: the first and the last decide for all four
      const bool in0 = row[0] < rows, in3 = row[3] < rows;
      if (!in0 && !in3 && (int)(row[0] ^ row[3]) >= 0) continue;  // all on one side of the detector
      const bool inside = in0 && in3;
      if (ALL && inside)
        plain_group<NZ, false, WEIGHTED>(res, 4 * h, row, rows, fz, c0, c1, pitch, ux2, E2, qrow[h]);
      else
        plain_group<NZ, true, WEIGHTED>(res, 4 * h, row, rows, fz, c0, c1, pitch, ux2, E2, qrow[h]);
    }
  }
}

// Shared memory of a table-weight CTA (T: float or double), and the union view
// window of its NZ slices.
template <class T, int NZ>
struct BlockTables {
  double* z;         // [NZ] voxel z of the block's slices
  int *s0, *lo, *hi; // [NZ] central view and clamped window [lo, hi]
  T* q;              // [qcap][NZ]
  __device__ __forceinline__ explicit BlockTables(unsigned char* smem)
      : z(reinterpret_cast<double*>(smem)), s0(reinterpret_cast<int*>(z + NZ)), lo(s0 + NZ), hi(lo + NZ),
        q(reinterpret_cast<T*>(hi + NZ)) {
    static_assert(NZ % 2 == 0, "q on a boundary of 8 bytes");
  }
  __device__ __forceinline__ int first() const {
    int p = lo[0];
    for (int m = 1; m < NZ; ++m) p = min(p, lo[m]);
    return p;
  }
  __device__ __forceinline__ int last() const {
    int p = hi[0];
    for (int m = 1; m < NZ; ++m) p = max(p, hi[m]);
    return p;
  }
};

// An infinite sample among the taps of plain_views' differences gives NaN: the
// thread's NaN voxels again, with weighted taps. (Weighted taps for all would
// cost 4 to 7 % of the kernel's time; this costs 0.3 %, in FP64 1.6 %, and a
// volume of nothing but NaN is computed twice.) Neither inlined nor given what
// it can derive, so that the views' loop keeps its registers.
template <int NZ>
__device__ __noinline__ void plain_nan_voxels(float* vol, const float* fp, const ViewTab* views, const BpParams& P,
                                              unsigned char* smem) {
  const BlockTables<float, NZ> B(smem);
  const int xi = blockIdx.x * kTx + threadIdx.x, yi = blockIdx.y * kTy + threadIdx.y, z0 = blockIdx.z * NZ;
  PlainColumn C;
  C.fp = fp;
  C.views = views;
  C.q_s = B.q;
  C.z_s = B.z;
  C.x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  C.y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  C.z00 = B.z[0];
  C.pstart = B.first();
  float res[NZ];
#pragma unroll
  for (int m = 0; m < NZ; ++m) res[m] = 0.0f;
  plain_views<NZ, false, true>(res, C, P, 0, min(B.last() - C.pstart + 1, P.qcap));
  float* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
#pragma unroll
  for (int m = 0; m < NZ; ++m)
    if (z0 + m < P.ZN && isnan(out[m])) out[m] = res[m] * P.DeltaFaif;
}

template <int NZ>
__global__ void __launch_bounds__(kTx* kTy, 4) bp_plain_q_kernel(float* __restrict__ vol, const float* __restrict__ fp,
                                                             const ViewTab* __restrict__ views,
                                                             const float* __restrict__ gw, const __grid_constant__ BpParams P) {
  static_assert(NZ % 4 == 0, "slices are processed in groups of four");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const BlockTables<float, NZ> B(smem_raw);
  double* z_s = B.z;
  int *s0_s = B.s0, *lo_s = B.lo, *hi_s = B.hi;
  float* q_s = B.q;
  const int tid = threadIdx.y * kTx + threadIdx.x;
  const int z0 = blockIdx.z * NZ;
  // the block's union window (uniform over the CTA; every thread evaluates it)
  int pstart = 0x7fffffff, pend = -0x7fffffff;
  int all0 = -0x7fffffff, all1 = 0x7fffffff;  // views that every slice's window holds
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    const ZInfo zi = z_info(P, z0 + m);
    if (tid == 0) {
      z_s[m] = zi.z;
      s0_s[m] = zi.s0;
      lo_s[m] = zi.lo;
      hi_s[m] = zi.hi;
    }
    pstart = min(pstart, zi.lo);
    pend = max(pend, zi.hi);
    all0 = max(all0, zi.lo);
    all1 = min(all1, zi.hi);
  }
  // views of the union window; 0 for a block whose slices all lie outside the
  // scan (pstart > pend: compared before subtracting, which would overflow).
  // The host sizes qcap from the same expressions; the clamp only keeps the
  // table in bounds.
  int len = pend >= pstart ? pend - pstart + 1 : 0;
  if (len > P.qcap) len = P.qcap;
  __syncthreads();  // the slice data
  for (int e = tid; e < len * NZ; e += kTx * kTy) {
    const int q = e / NZ, m = e - q * NZ;
    const int p = pstart + q;
    float qv = -1.0f;
    if (p >= lo_s[m] && p <= hi_s[m]) {
      const int before = p < s0_s[m];
      const int d1 = (int)(P.N_pi - (double)(s0_s[m] - p));
      const int d2 = before ? (int)(d1 + P.N_pi) : (int)(d1 - P.N_pi);
      const double w1 = __ldg(gw + d1), w2 = __ldg(gw + d2);
      const double t2 = __dsub_rn(z_s[m], views[p].hv);
      const double tc = before ? t2 - 0.5 : t2 + 0.5;
      qv = w2 == 0.0 ? 0.0f : (float)(w2 / w1 * pow(fabs(t2) / fabs(tc), P.k1));
    }
    q_s[e] = qv;
  }
  __syncthreads();
  const int xi = blockIdx.x * kTx + threadIdx.x;
  const int yi = blockIdx.y * kTy + threadIdx.y;
  if (xi >= P.XN || yi >= P.YN) return;
  PlainColumn C;
  C.fp = fp;
  C.views = views;
  C.q_s = q_s;
  C.z_s = z_s;
  C.x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  C.y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  C.z00 = __dmul_rn(__dsub_rn((double)z0, P.ZNC), P.dz);
  C.pstart = pstart;
  float res[NZ];
#pragma unroll
  for (int m = 0; m < NZ; ++m) res[m] = 0.0f;
  // the views every slice has between those that only some have (none of them: all1 < all0)
  const bool common = all1 >= all0;
  const int qa = common ? min(all0 - pstart, len) : len, qb = common ? min(all1 - pstart + 1, len) : len;
  plain_views<NZ, false>(res, C, P, 0, qa);
  plain_views<NZ, true>(res, C, P, qa, qb);
  plain_views<NZ, false>(res, C, P, qb, len);
  float* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
  bool nan = false;
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    if (z0 + m < P.ZN) out[m] = res[m] * P.DeltaFaif;
    nan = nan || isnan(res[m]);
  }
  if (nan) plain_nan_voxels<NZ>(vol, fp, views, P, smem_raw);
}

// ---------------------------------------------------------------------------
// FP64 form: the reference CPU's data path in double on the GPU.
// ---------------------------------------------------------------------------
template <int NZ>
__global__ void __launch_bounds__(kBx* kBy) bp_fp64_kernel(double* __restrict__ vol, const double* __restrict__ fp,
                                                          const ViewTab* __restrict__ views,
                                                          const double* __restrict__ gw, BpParams P) {
  extern __shared__ double wd_s[];  // [N_2pi]
  for (int t = threadIdx.y * kBx + threadIdx.x; t < P.N_2pi; t += kBx * kBy) wd_s[t] = gw[t];
  __syncthreads();
  const int xi = blockIdx.x * kBx + threadIdx.x;
  const int yi = blockIdx.y * kBy + threadIdx.y;
  const int z0 = blockIdx.z * NZ;
  if (xi >= P.XN || yi >= P.YN) return;
  const double x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  const double y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  ZInfo zin[NZ];
  double res[NZ];
  int pstart = 0x7fffffff, pend = -0x7fffffff;
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    zin[m] = z_info(P, z0 + m);
    res[m] = 0.0;
    pstart = min(pstart, zin[m].lo);
    pend = max(pend, zin[m].hi);
  }
  const size_t plane = (size_t)P.ZL * P.YL;
  for (int p = pstart; p <= pend; ++p) {
    const ViewTab v = views[p];
    const ColView cv = col_view(P, x, y, v);
    if (cv.U <= 0 || cv.U >= P.YL) continue;
    const double dey = __dsub_rn((double)cv.U, cv.U1);
    const double* col = fp + (size_t)p * plane + (cv.U - 1);
#pragma unroll
    for (int m = 0; m < NZ; ++m) {
      if (p < zin[m].lo || p > zin[m].hi) continue;
      const double temp2 = __dsub_rn(zin[m].z, v.hv);
      const double Zr = __ddiv_rn(__dmul_rn(temp2, P.SOSD), cv.denom);
      const double V1 = __dadd_rn(__ddiv_rn(Zr, P.dZL), P.ZLC);
      const int V = (int)ceil(V1);
      if (V <= 0 || V >= P.ZL) continue;
      const double dez = __dsub_rn((double)V, V1);
      const double* r0 = col + (size_t)(V - 1) * P.YL;
      const double* r1 = r0 + P.YL;
      const double touying = dey * dez * r0[0] + dey * (1.0 - dez) * r1[0] + (1.0 - dey) * dez * r0[1] +
                             (1.0 - dey) * (1.0 - dez) * r1[1];
      const int before = p < zin[m].s0;
      const int d1 = (int)(P.N_pi - (double)(zin[m].s0 - p));
      const int d2 = before ? (int)(d1 + P.N_pi) : (int)(d1 - P.N_pi);
      const double w1 = wd_s[d1], w2 = wd_s[d2];
      const double gama = fabs(temp2 / cv.A);
      const double gamac = before ? fabs((temp2 - 0.5) / cv.B) : fabs((temp2 + 0.5) / cv.B);
      const double m1 = pow(gama, P.k1);
      const double m2 = pow(gamac, P.k1);
      const double weight = (w1 * m2) / (w2 * m1 + w1 * m2);
      res[m] += weight * touying * P.DeltaFai;
    }
  }
  double* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
#pragma unroll
  for (int m = 0; m < NZ; ++m)
    if (z0 + m < P.ZN) out[m] = res[m];
}

// FP64 form with table weights: weight = 1 / (1 + Q2 E) as in the plain form,
// Q2 tabulated per block in FP64, E one logarithm and one exponential per
// (column, view). The per-update kernel above (kept for blocks whose table
// would not fit: thick slices) evaluates two powers and four divisions per
// update and a square root and a division per (column, view), and the FP64
// units bound it (64 lanes per clock and SM). Here the reciprocals and the root
// start from the approximate instructions and take two Newton steps (1e-16), V
// of slice m is v(first) + m dv and its floor two adds: 51 FP64 operations per
// update, 17 of them per update proper. Where a row lies within 2.4e-7 (a
// channel 1e-9) of an integer the update repeats the reference's own operations
// (fp64_update_exact), so index selection stays exact; elsewhere values differ
// from it by rounding only: against an evaluation in 80 bits, on smooth data,
// 7.4e-16, 7.5e-16 and 5.7e-16 relative (three geometries), the kernel above
// 7.7e-16, 7.5e-16 and 5.5e-16; on noise 4.4e-14, 4.3e-14 and 4.0e-14 against
// 4.8e-14, 4.8e-14 and 4.1e-14.
// Measured on 888 x 16, 3 rotations -> 186 x 171 x 21 (4.5e8 updates): 13.6 ->
// 3.1 ms (FP64 pipe 45 %, issue 57 %); eight slices per thread halve the per-view work but need 117
// registers and leave 1.5 waves of CTAs there: 4.17 ms.
__device__ __noinline__ double fp64_update_exact(const BpParams& P, const double* __restrict__ fp, const ViewTab v,
                                                 int p, double x, double y, double z, double q2) {
  const ColView cv = col_view(P, x, y, v);
  if (cv.U <= 0 || cv.U >= P.YL) return 0.0;
  const double temp2 = __dsub_rn(z, v.hv);
  const double Zr = __ddiv_rn(__dmul_rn(temp2, P.SOSD), cv.denom);
  const double V1 = __dadd_rn(__ddiv_rn(Zr, P.dZL), P.ZLC);
  const int V = (int)ceil(V1);
  if (V <= 0 || V >= P.ZL) return 0.0;
  const double dey = __dsub_rn((double)cv.U, cv.U1), dez = __dsub_rn((double)V, V1);
  const double* r0 = fp + ((size_t)p * P.ZL + (V - 1)) * P.YL + (cv.U - 1);
  const double* r1 = r0 + P.YL;
  const double tap = dey * dez * r0[0] + dey * (1.0 - dez) * r1[0] + (1.0 - dey) * dez * r0[1] +
                     (1.0 - dey) * (1.0 - dez) * r1[1];
  const double E = P.k1 == 0.0 ? 1.0 : fmin(pow(fabs(cv.B) / fabs(cv.A), P.k1), kBig);
  return tap / fma(q2, E, 1.0);
}

constexpr int kDx = 8, kDy = 32;  // CTA tile (x, y)

// The views of a block's union window for one column.
template <int NZ, bool WEIGHTED>
__device__ __forceinline__ void fp64_views(double (&res)[NZ], const double* __restrict__ fp,
                                           const ViewTab* __restrict__ views, const double* q_s, const double* z_s,
                                           const BpParams& P, double x, double y, double z00, int pstart, int len) {
  const size_t plane = (size_t)P.ZL * P.YL;
  const uint32_t rows = (uint32_t)(P.ZL - 1), chans = (uint32_t)(P.YL - 1);
  const uint32_t pitch = (uint32_t)P.YL * (uint32_t)sizeof(double);
  constexpr double kM = 6755399441055744.0;          // 1.5 * 2^52: adding it rounds to an integer
  constexpr uint32_t kTie = 0x3fdfffffu;             // high word of |x| >= 0.5 - 2.4e-7
#pragma unroll 1
  for (int q = 0; q < len; ++q) {
    const ViewTab v = views[pstart + q];
    const double UU = fma(-x, v.c, -(y * v.s));
    const double Yr = fma(-x, v.s, y * v.c);
    const double uc = fma(Yr, P.invdYL, P.YLC) - 0.5;
    const double ur = uc + kM;
    const double ud = uc - (ur - kM);                 // fraction - 1/2
    const uint32_t u = (uint32_t)__double2loint(ur);  // U - 1
    bool near = fabs(ud) > 0.5 - 1e-9;
    if (u >= chans && !near) continue;                // U <= 0 or U >= YL
    const double t1sq = fma(-Yr, Yr, P.SO2);
    double h = rsqrt64_approx(t1sq);
    double g = t1sq * h;
    h *= 0.5;
    const double rr = fma(-g, h, 0.5);
    g = fma(g, rr, g);
    h = fma(h, rr, h);
    const double temp1 = fma(fma(-g, g, t1sq), h, g);
    const double den = fma(temp1, UU, t1sq);          // temp1 (temp1 + UU)
    double rd = rcp64_approx(den);
    rd = fma(fma(-den, rd, 1.0), rd, rd);
    rd = fma(fma(-den, rd, 1.0), rd, rd);
    const double slope = rd * P.SOSDdZL;
    const double v0 = fma(z00 - v.hv, slope, P.ZLC - 0.5);
    const double dv = slope * P.dz;
    if (!(fabs(v0) + NZ * fabs(dv) < kFixLimit)) near = true;  // also NaN
    const double ratio = fabs(fma(-temp1, UU, t1sq) * rd);     // |temp1 - UU| / |temp1 + UU|
    const double E = P.k1 == 0.0 ? 1.0 : fmin(exp(P.k1 * log(ratio)), kBig);
    const double ux = ud + 0.5;
    const double* c0 = fp + (size_t)(pstart + q) * plane + min(u, chans - 1);
    const double* c1 = c0 + P.YL;
    const double* qrow = q_s + q * NZ;
#pragma unroll
    for (int hp = 0; hp < NZ / 2; ++hp) {
      const double2 qq = *reinterpret_cast<const double2*>(qrow + 2 * hp);
      const double q2[2] = {qq.x, qq.y};
      if (q2[0] < 0.0 && q2[1] < 0.0) continue;  // uniform over the CTA
      uint32_t row[2], tie = near ? 0xffffffffu : 0u;
      double vd[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double vc = fma((double)(2 * hp + i), dv, v0);
        const double vr = vc + kM;
        vd[i] = vc - (vr - kM);
        row[i] = (uint32_t)__double2loint(vr);  // V - 1
        tie = max(tie, (uint32_t)__double2hiint(vd[i]) & 0x7fffffffu);
      }
      if (tie >= kTie) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (!(q2[i] < 0.0))
            res[2 * hp + i] += fp64_update_exact(P, fp, v, pstart + q, x, y, z_s[2 * hp + i], q2[i]);
        continue;
      }
      double a0[2], b0[2], a1[2], b1[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t r = min(row[i], rows - 1);  // a row off the detector reads the last one and is not added
        const double* p0 = row_ptr(c0, r, pitch);
        const double* p1 = row_ptr(c1, r, pitch);
        a0[i] = __ldg(p0);
        b0[i] = __ldg(p0 + 1);
        a1[i] = __ldg(p1);
        b1[i] = __ldg(p1 + 1);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double ra = lerp<WEIGHTED>(ux, a0[i], b0[i]);
        const double rb = lerp<WEIGHTED>(ux, a1[i], b1[i]);
        const double tap = lerp<WEIGHTED>(vd[i] + 0.5, ra, rb);
        const double s = fma(q2[i], E, 1.0);
        double w = rcp64_approx(s);
        w = fma(fma(-s, w, 1.0), w, w);
        w = fma(fma(-s, w, 1.0), w, w);
        if (row[i] < rows && !(q2[i] < 0.0)) res[2 * hp + i] = fma(w, tap, res[2 * hp + i]);
      }
    }
  }
}

// The thread's NaN voxels with weighted taps, as in the plain form.
template <int NZ>
__device__ __noinline__ void fp64_nan_voxels(double* vol, const double* fp, const ViewTab* views, const BpParams& P,
                                             unsigned char* smem) {
  const BlockTables<double, NZ> B(smem);
  const int xi = blockIdx.x * kDx + threadIdx.x, yi = blockIdx.y * kDy + threadIdx.y, z0 = blockIdx.z * NZ;
  const double x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  const double y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  const int pstart = B.first();
  double res[NZ];
#pragma unroll
  for (int m = 0; m < NZ; ++m) res[m] = 0.0;
  fp64_views<NZ, true>(res, fp, views, B.q, B.z, P, x, y, B.z[0], pstart, min(B.last() - pstart + 1, P.qcap));
  double* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
#pragma unroll
  for (int m = 0; m < NZ; ++m)
    if (z0 + m < P.ZN && isnan(out[m])) out[m] = res[m] * P.DeltaFai;
}

template <int NZ>
__global__ void __launch_bounds__(kDx* kDy, 3) bp_fp64_q_kernel(double* __restrict__ vol, const double* __restrict__ fp,
                                                               const ViewTab* __restrict__ views,
                                                               const double* __restrict__ gw,
                                                               const __grid_constant__ BpParams P) {
  static_assert(NZ % 2 == 0, "slices are processed in pairs");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const BlockTables<double, NZ> B(smem_raw);
  double* z_s = B.z;
  int *s0_s = B.s0, *lo_s = B.lo, *hi_s = B.hi;
  double* q_s = B.q;
  const int tid = threadIdx.y * kDx + threadIdx.x;
  const int z0 = blockIdx.z * NZ;
  int pstart = 0x7fffffff, pend = -0x7fffffff;
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    const ZInfo zi = z_info(P, z0 + m);
    if (tid == 0) {
      z_s[m] = zi.z;
      s0_s[m] = zi.s0;
      lo_s[m] = zi.lo;
      hi_s[m] = zi.hi;
    }
    pstart = min(pstart, zi.lo);
    pend = max(pend, zi.hi);
  }
  int len = pend >= pstart ? pend - pstart + 1 : 0;  // 0: every slice lies outside the scan
  if (len > P.qcap) len = P.qcap;                    // the host sizes qcap from the same expressions
  __syncthreads();
  for (int e = tid; e < len * NZ; e += kDx * kDy) {
    const int q = e / NZ, m = e - q * NZ;
    const int p = pstart + q;
    double qv = -1.0;
    if (p >= lo_s[m] && p <= hi_s[m]) {
      const int before = p < s0_s[m];
      const int d1 = (int)(P.N_pi - (double)(s0_s[m] - p));
      const int d2 = before ? (int)(d1 + P.N_pi) : (int)(d1 - P.N_pi);
      const double w1 = __ldg(gw + d1), w2 = __ldg(gw + d2);
      const double t2 = __dsub_rn(z_s[m], views[p].hv);
      const double tc = before ? t2 - 0.5 : t2 + 0.5;
      // infinite where w1 or tc is 0 (weight 0: a bound keeps the reciprocal finite), NaN where the
      // reference's weight is
      const double r = w2 / w1 * pow(fabs(t2) / fabs(tc), P.k1);
      qv = r > kBig ? kBig : r;
    }
    q_s[e] = qv;
  }
  __syncthreads();
  const int xi = blockIdx.x * kDx + threadIdx.x;
  const int yi = blockIdx.y * kDy + threadIdx.y;
  if (xi >= P.XN || yi >= P.YN) return;
  const double x = __dmul_rn(__dsub_rn((double)xi, P.XNC), P.dx);
  const double y = __dmul_rn(__dsub_rn((double)yi, P.YNC), P.dy);
  const double z00 = __dmul_rn(__dsub_rn((double)z0, P.ZNC), P.dz);
  double res[NZ];
#pragma unroll
  for (int m = 0; m < NZ; ++m) res[m] = 0.0;
  fp64_views<NZ, false>(res, fp, views, q_s, z_s, P, x, y, z00, pstart, len);
  double* out = vol + ((size_t)yi * P.XN + xi) * P.ZN + z0;
  bool nan = false;
#pragma unroll
  for (int m = 0; m < NZ; ++m) {
    if (z0 + m < P.ZN) out[m] = res[m] * P.DeltaFai;
    nan = nan || isnan(res[m]);
  }
  if (nan) fp64_nan_voxels<NZ>(vol, fp, views, P, smem_raw);
}

constexpr int kNzPlain = 8;
constexpr int kNzFp64 = 4;   // slices per thread of the per-update FP64 kernel
constexpr int kNzFp64Q = 4;  // and of the table-weight one

// Checks a backprojection geometry and fills the kernels' parameter block. Every
// entry that backprojects (the plans and the allocation-free entry) goes through
// it, so they accept exactly the same geometries.
// The geometry checks of every backprojection entry (host only); *half: the window's half width.
int geom_checks(const hr_bp_geom* g, const char* who, int* half_out) {
  HR_REQUIRE(g->XN > 0 && g->YN > 0 && g->ZN > 0 && g->YL > 1 && g->ZL > 1 && g->PN > 0 && g->N_2pi > 1,
             "%s: invalid sizes", who);
  HR_REQUIRE(g->h != 0.0 && g->DeltaFai != 0.0 && g->dYL != 0.0 && g->dZL != 0.0 && g->SO > 0.0,
             "%s: h, DeltaFai, dYL, dZL must be non-zero and SO > 0", who);
  HR_REQUIRE((long long)g->XN * g->YN * g->ZN < (1LL << 40), "%s: volume too large", who);
  HR_REQUIRE(g->N_2pi <= 8192, "%s: N_2pi=%d exceeds 8192", who, g->N_2pi);
  // For views in [s0-half, s0+half] the weight indices are d1 = N_pi-(s0-p)
  // and d1 +/- N_pi; they stay inside [0, N_2pi) iff half <= N_pi and
  // N_pi + half <= N_2pi - 1 (the reference GPU kernel reads outside it).
  const int half = (int)std::ceil(g->N_pi * g->HSCoef);
  HR_REQUIRE(half >= 0 && (double)half <= g->N_pi && g->N_pi + half <= g->N_2pi - 1 &&
                 2.0 * g->N_pi <= g->N_2pi + 1e-9,
             "%s: HSCoef=%g, N_pi=%g give a view window outside the weight table", who, g->HSCoef, g->N_pi);
  *half_out = half;
  return HR_OK;
}

int bp_params_from_geom(const hr_bp_geom* g, const char* who, BpParams* out) {
  int half = 0;
  HR_TRY(geom_checks(g, who, &half));
  HR_TRY(hr::require_device());
  BpParams P{};
  P.XN = g->XN; P.YN = g->YN; P.ZN = g->ZN; P.YL = g->YL; P.ZL = g->ZL; P.PN = g->PN; P.N_2pi = g->N_2pi;
  P.half = half;
  P.XNC = g->XNC; P.YNC = g->YNC; P.ZNC = g->ZNC; P.dx = g->dx; P.dy = g->dy; P.dz = g->dz;
  P.YLC = g->YLC; P.ZLC = g->ZLC; P.dYL = g->dYL; P.dZL = g->dZL; P.h = g->h; P.BetaS = g->BetaS;
  P.DeltaFai = g->DeltaFai; P.N_pi = g->N_pi; P.SO = g->SO; P.SD = g->SD; P.k1 = g->k1;
  P.SO2 = g->SO * g->SO;
  P.SOSD = g->SO * g->SD;
  P.SOSDdZL = P.SOSD / g->dZL;
  P.invdYL = 1.0 / g->dYL;
  P.k1f = (float)g->k1;
  P.DeltaFaif = (float)g->DeltaFai;
  // longest union view window of a z block of kNzPlain slices, with the
  // device's expressions for the central view and the clamped window
  P.qcap = 0;
  for (int z0 = 0; z0 < g->ZN; z0 += kNzPlain) {
    int a = 0x7fffffff, e = -0x7fffffff;
    for (int zi = z0; zi < z0 + kNzPlain && zi < g->ZN; ++zi) {
      const double z = (zi - g->ZNC) * g->dz;
      const double beta0 = kTwoPiTrunc * z / g->h;
      const int s0 = (int)std::ceil((beta0 - g->BetaS) / g->DeltaFai - 0.5);
      const int s1 = s0 - half, s2 = s0 + half;
      if (s1 < g->PN && s2 > 0) {
        a = std::min(a, s1 < 0 ? 0 : s1);
        e = std::max(e, s2 > g->PN - 1 ? g->PN - 1 : s2);
      }
    }
    if (e >= a) P.qcap = std::max(P.qcap, e - a + 1);
  }
  *out = P;
  return HR_OK;
}

// Dynamic shared memory of bp_plain_q_kernel.
size_t plain_q_smem(const BpParams& P) {
  return sizeof(double) * kNzPlain + 3 * sizeof(int) * kNzPlain + sizeof(float) * (size_t)P.qcap * kNzPlain;
}
// Above this the per-CTA weight table would cost too much occupancy (very
// thick slices: long union windows); the per-update weight kernel runs instead.
// The limit on a kernel's dynamic shared memory belongs to the kernel, not to a
// plan: every launch sets it to this most, so that of two plans executed by two
// threads neither lowers it between the other's setting and launch.
constexpr size_t kPlainQSmemMax = 96 * 1024;
bool plain_q_fits(const BpParams& P) { return P.qcap > 0 && plain_q_smem(P) <= kPlainQSmemMax; }

// Dynamic shared memory of bp_fp64_q_kernel, and the most it may take (two CTAs per SM still fit); above
// it (thick slices) the per-update kernel runs.
static_assert(kNzFp64Q <= kNzPlain, "qcap is the longest union window of kNzPlain slices");
size_t fp64_q_smem(const BpParams& P) {
  return sizeof(double) * kNzFp64Q + sizeof(int) * 3 * kNzFp64Q +
         sizeof(double) * (size_t)P.qcap * kNzFp64Q;
}
constexpr size_t kFp64QSmemMax = 100 * 1024;
bool fp64_q_fits(const BpParams& P) { return P.qcap > 0 && fp64_q_smem(P) <= kFp64QSmemMax; }

// The plain-form launch of both the plan and the allocation-free entry (the
// same kernel for the same geometry, so their results are identical).
int launch_plain(const BpParams& P, float* vol, const float* fp, const ViewTab* views, const float* w,
                 cudaStream_t s) {
  dim3 grid((P.XN + kBx - 1) / kBx, (P.YN + kBy - 1) / kBy, (P.ZN + kNzPlain - 1) / kNzPlain);
  HR_REQUIRE(grid.z <= 65535 && grid.y <= 65535, "backprojection: grid too large");
  if (plain_q_fits(P)) {
    grid.x = (P.XN + kTx - 1) / kTx;
    grid.y = (P.YN + kTy - 1) / kTy;
    HR_CUDA_TRY(cudaFuncSetAttribute(bp_plain_q_kernel<kNzPlain>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kPlainQSmemMax));
    bp_plain_q_kernel<kNzPlain><<<grid, dim3(kTx, kTy), plain_q_smem(P), s>>>(vol, fp, views, w, P);
  } else {
    bp_plain_kernel<kNzPlain><<<grid, dim3(kBx, kBy), sizeof(float) * P.N_2pi, s>>>(vol, fp, views, w, P);
  }
  HR_CUDA_TRY(cudaGetLastError());
  return HR_OK;
}

// Per-view tables in the reference's own arithmetic
// (src/Parallel_FDK_Helical_3DWeighting.cpp:73, :76-79): the host C library's
// cos/sin, which the bit-exact index selection depends on.
void fill_view_table(ViewTab* tab, int PN, double BetaS, double DeltaFai, double h) {
  for (int p = 0; p < PN; ++p) {
    const double View = BetaS + p * DeltaFai;
    tab[p] = ViewTab{std::cos(View), std::sin(View), h * View * kInvTwoPi};
  }
}

}  // namespace

void hr::fast_geom_fill(const hr_bp_geom& g, int half, BpFastGeom* f) {
  f->XN = g.XN; f->YN = g.YN; f->ZN = g.ZN; f->YL = g.YL; f->ZL = g.ZL; f->PN = g.PN; f->half = half;
  f->XNC = g.XNC; f->YNC = g.YNC; f->ZNC = g.ZNC; f->dx = g.dx; f->dy = g.dy; f->dz = g.dz;
  f->YLC = g.YLC; f->ZLC = g.ZLC; f->dYL = g.dYL; f->dZL = g.dZL; f->h = g.h; f->BetaS = g.BetaS;
  f->DeltaFai = g.DeltaFai; f->N_pi = g.N_pi; f->SO = g.SO; f->SD = g.SD; f->k1 = g.k1;
  f->ZN_valid = g.ZN;
}

int hr::fast_geom_of(const hr_bp_geom& g, BpFastGeom* f) {
  int half = 0;
  HR_TRY(geom_checks(&g, "backprojection", &half));
  fast_geom_fill(g, half, f);
  return HR_OK;
}

extern "C" int hr_bp_plan_create(hr_bp_plan** plan, const hr_bp_geom* g, const double* w, int form) {
  hr::clear_error();
  HR_REQUIRE(plan != nullptr && g != nullptr && w != nullptr, "hr_bp_plan_create: NULL argument");
  *plan = nullptr;
  HR_REQUIRE(form == HR_FORM_PLAIN || form == HR_FORM_FP64 || form == HR_FORM_FAST,
             "hr_bp_plan_create: unknown form %d", form);
  BpParams P{};
  HR_TRY(bp_params_from_geom(g, "backprojection", &P));
  const int half = P.half;

  std::vector<ViewTab> tab(g->PN);
  fill_view_table(tab.data(), g->PN, g->BetaS, g->DeltaFai, g->h);
  std::vector<float> wf(g->N_2pi);
  for (int i = 0; i < g->N_2pi; ++i) wf[i] = (float)w[i];

  hr_bp_plan* pl = new hr_bp_plan{P, form, nullptr, nullptr, nullptr, hr::BpFastGeom{}, hr::BpFast{}};
  if (form == HR_FORM_FAST) {
    hr::fast_geom_fill(*g, half, &pl->fg);
    const int st = hr::bp_fast_create(&pl->fast, pl->fg, w);
    if (st != HR_OK) {
      hr::bp_fast_destroy(&pl->fast);
      delete pl;
      return st;
    }
    *plan = pl;
    return HR_OK;
  }
  cudaError_t e = cudaMalloc(&pl->d_views, sizeof(ViewTab) * g->PN);
  if (e == cudaSuccess) e = cudaMalloc(&pl->d_w, sizeof(float) * g->N_2pi);
  if (e == cudaSuccess) e = cudaMalloc(&pl->d_wd, sizeof(double) * g->N_2pi);
  if (e == cudaSuccess) e = cudaMemcpy(pl->d_views, tab.data(), sizeof(ViewTab) * g->PN, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(pl->d_w, wf.data(), sizeof(float) * g->N_2pi, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(pl->d_wd, w, sizeof(double) * g->N_2pi, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(pl->d_views);
    cudaFree(pl->d_w);
    cudaFree(pl->d_wd);
    delete pl;
    return hr::fail(e == cudaErrorMemoryAllocation ? HR_ERR_OUT_OF_MEMORY : HR_ERR_CUDA, "bp plan: %s",
                    cudaGetErrorString(e));
  }
  *plan = pl;
  return HR_OK;
}

extern "C" int hr_bp_execute(const hr_bp_plan* pl, void* d_vol, const void* d_fp, void* stream) {
  HR_REQUIRE(pl != nullptr && d_vol != nullptr && d_fp != nullptr, "hr_bp_execute: NULL argument");
  const BpParams& P = pl->prm;
  cudaStream_t s = hr::as_stream(stream);
  if (pl->form == HR_FORM_FAST)
    return hr::bp_fast_execute(pl->fast, pl->fg, static_cast<float*>(d_vol), static_cast<const uint32_t*>(d_fp), s);
  if (pl->form == HR_FORM_PLAIN)
    return launch_plain(P, static_cast<float*>(d_vol), static_cast<const float*>(d_fp), pl->d_views, pl->d_w, s);
  {
    dim3 grid((P.XN + kBx - 1) / kBx, (P.YN + kBy - 1) / kBy, (P.ZN + kNzFp64 - 1) / kNzFp64);
    HR_REQUIRE(grid.z <= 65535 && grid.y <= 65535, "backprojection: grid too large");
    double* vol = static_cast<double*>(d_vol);
    const double* fp = static_cast<const double*>(d_fp);
    if (fp64_q_fits(P)) {
      grid = dim3((P.XN + kDx - 1) / kDx, (P.YN + kDy - 1) / kDy, (P.ZN + kNzFp64Q - 1) / kNzFp64Q);
      HR_CUDA_TRY(cudaFuncSetAttribute(bp_fp64_q_kernel<kNzFp64Q>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kFp64QSmemMax));
      bp_fp64_q_kernel<kNzFp64Q><<<grid, dim3(kDx, kDy), fp64_q_smem(P), s>>>(vol, fp, pl->d_views, pl->d_wd, P);
    } else {
      bp_fp64_kernel<kNzFp64><<<grid, dim3(kBx, kBy), sizeof(double) * P.N_2pi, s>>>(vol, fp, pl->d_views, pl->d_wd,
                                                                                    P);
    }
  }
  HR_CUDA_TRY(cudaGetLastError());
  return HR_OK;
}

int hr::bp_plan_fast_parts(const hr_bp_plan* pl, const BpFastGeom** g, const BpFast** f) {
  HR_REQUIRE(pl != nullptr && pl->form == HR_FORM_FAST, "backprojection plan is not of the fast form");
  *g = &pl->fg;
  *f = &pl->fast;
  return HR_OK;
}

extern "C" int hr_bp_autotune(hr_bp_plan* pl, void* d_vol, const void* d_fp, void* stream) {
  HR_REQUIRE(pl != nullptr && d_vol != nullptr && d_fp != nullptr, "hr_bp_autotune: NULL argument");
  if (pl->form != HR_FORM_FAST) return HR_OK;
  return hr::bp_fast_autotune(&pl->fast, pl->fg, static_cast<float*>(d_vol), static_cast<const uint32_t*>(d_fp),
                              hr::as_stream(stream));
}

extern "C" int hr_bp_select(hr_bp_plan* pl, int variant) {
  HR_REQUIRE(pl != nullptr, "hr_bp_select: NULL plan");
  if (pl->form != HR_FORM_FAST) return variant == 0 ? HR_OK : hr::fail(HR_ERR_INVALID_ARGUMENT, "hr_bp_select: "
                                                                        "only the fast form has variants");
  HR_REQUIRE(variant >= 0 && variant < hr::kFastVariants_n, "hr_bp_select: variant %d out of range [0, %d)",
             variant, hr::kFastVariants_n);
  pl->fast.variant = variant;
  return hr::bp_fast_tex_prepare(&pl->fast, pl->fg);
}

extern "C" int hr_bp_describe(const hr_bp_plan* pl, char* buf, int len) {
  HR_REQUIRE(pl != nullptr, "hr_bp_describe: NULL plan");
  if (pl->form == HR_FORM_FAST) return hr::bp_fast_describe(pl->fast, pl->fg, buf, len);
  if (buf && len > 0) {
    const bool fp64 = pl->form == HR_FORM_FP64, table = fp64 ? fp64_q_fits(pl->prm) : plain_q_fits(pl->prm);
    snprintf(buf, (size_t)len, "%s slices_per_thread=%d tile=%dx%d weights=%s", fp64 ? "fp64" : "plain",
             !fp64 ? kNzPlain : table ? kNzFp64Q : kNzFp64, !table ? kBx : fp64 ? kDx : kTx,
             !table ? kBy : fp64 ? kDy : kTy, table ? "per-block table" : "per update");
  }
  return HR_OK;
}

extern "C" void hr_bp_plan_destroy(hr_bp_plan* pl) {
  if (!pl) return;
  hr::bp_fast_destroy(&pl->fast);
  cudaFree(pl->d_views);
  cudaFree(pl->d_w);
  cudaFree(pl->d_wd);
  delete pl;
}

// ---------------------------------------------------------------------------
// Plain-form backprojection that allocates nothing.
//
// Some callers cannot call cudaMalloc: streaming pipelines that must not
// allocate once they run, because cudaMalloc and cudaFree synchronise the whole
// device and would stall the other streams; hosts whose pooling allocator owns
// all device memory (a MATLAB session, a framework's caching allocator), where
// a second allocator fragments or exhausts the pool; and services that run
// under a fixed device-memory budget. This entry keeps its only scratch -- the
// per-view cos/sin/source-height table -- in a file-scope device array of
// kNoAllocMaxViews entries (768 KiB, held by every GPU that loads the library
// until the process exits) and takes everything else (filtered data, weight
// table, volume) from the caller.
//
// The table is computed on the host with the same C library calls as the plan
// (fill_view_table) and copied into the array, so both entries select the same
// view/row/channel indices and give bit-identical volumes.
// ---------------------------------------------------------------------------
#include <mutex>

namespace {
constexpr int kNoAllocMaxViews = 32768;
constexpr int kNoAllocMaxDevices = 64;
}  // namespace

static __device__ __align__(256) ViewTab g_noalloc_views[kNoAllocMaxViews];

namespace {

std::mutex g_noalloc_mutex;
ViewTab* g_noalloc_ptr[kNoAllocMaxDevices] = {};
// Host staging of the table (pageable, file scope: filled and copied under
// g_noalloc_mutex).
ViewTab g_noalloc_host[kNoAllocMaxViews];

// Device address of g_noalloc_views on the current device, looked up once per
// device (with that device current). In host code the array's name is only a
// host-side stand-in, never a device address. Called with g_noalloc_mutex held.
int noalloc_views(ViewTab** out) {
  int dev = 0;
  HR_CUDA_TRY(cudaGetDevice(&dev));
  HR_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, "hr_bp_plain_noalloc: device %d out of range", dev);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    HR_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_views));
    g_noalloc_ptr[dev] = static_cast<ViewTab*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return HR_OK;
}

}  // namespace

extern "C" int hr_bp_plain_noalloc(float* d_vol, const float* d_fp, const float* d_w, const hr_bp_geom* g,
                                   void* stream) {
  hr::clear_error();
  HR_REQUIRE(d_vol != nullptr && d_fp != nullptr && d_w != nullptr && g != nullptr,
             "hr_bp_plain_noalloc: NULL argument");
  HR_REQUIRE(g->PN <= kNoAllocMaxViews,
             "hr_bp_plain_noalloc: PN=%d views exceed the fixed scratch table of %d views (use hr_bp_plan_create)",
             g->PN, kNoAllocMaxViews);
  BpParams P{};
  HR_TRY(bp_params_from_geom(g, "hr_bp_plain_noalloc", &P));
  cudaStream_t s = hr::as_stream(stream);
  ViewTab* views = nullptr;
  {
    // A copy from pageable host memory returns once the data are staged, so
    // the host buffer may be refilled by the next call as soon as it returns.
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    HR_TRY(noalloc_views(&views));
    fill_view_table(g_noalloc_host, P.PN, P.BetaS, P.DeltaFai, P.h);
    HR_CUDA_TRY(cudaMemcpyAsync(views, g_noalloc_host, sizeof(ViewTab) * P.PN, cudaMemcpyHostToDevice, s));
  }
  return launch_plain(P, d_vol, d_fp, views, d_w, s);
}
