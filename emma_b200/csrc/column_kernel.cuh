// column_kernel.cuh -- the hydro level advance of a complete level without split
// cells (a uniform box, the base level of a tree refined nowhere), periodic or
// transmissive in x, marching through z.
//
// The mixed path's kernel (the FP64 path's: column_fp64.cuh).  A work item is a column
// of 16 x TY cells (TY = 16) in x,y and `nz` cell planes in z.  One
// thread owns each cell of the column's cross-section and of its one-cell ring and
// walks the planes bottom to top; the z direction stays in its registers (the
// states of three planes, the upper face state and the lower flux of the last
// plane), and only what a neighbour in the plane needs goes through shared memory:
// the staged plane (two slots), each cell's +x and +y face state, the x and y
// fluxes.  Per advanced cell that is 25 values written and 45 read; keeping the
// slopes of every cell for its faces, as the brick kernel does, takes 65 and 120.
// Each cell is reconstructed once (MUSCL-Hancock), each face solved once (the -x,
// -y and -z face of each column cell, the +x and +y faces of the column's boundary
// by the ring).  The brick kernel (level_kernel.cuh) stages a 4.5x larger box per
// cell, reconstructs each advanced cell twice and solves 3.5 faces per cell; here
// it is 1.56x, 1.25 and 3.125 (the z halo is two planes per item).
//
// Step z, two barriers:
//   A  reconstruct plane z; solve the -z faces of plane z; update plane z-1 (its x
//      and y fluxes from shared memory);
//   B  solve the x and y faces of plane z; load and stage plane z+2 meanwhile.
// The ring threads also stage the outer halo (x = -2, 17; y = -2, TY+1), four
// column threads the ring's corner columns (+-1 diagonal).  Every face is solved at
// one call site per axis, so a face on the boundary of two columns (or of two z
// chunks) gets the same bits in both.
//
// XS (warp-shuffle x sweep): a warp holds two 16-cell x rows of the column, so the
// left neighbour of a column cell is the next lane down, which passes its +x face
// state up (__shfl_up_sync).  The column's two x boundary faces are solved by the
// x = -1 and x = 16 ring threads at the call site of the shared-memory sweep, so a
// face shared by two columns still gets the same bits in both.
//
// Work: a CTA runs either one item (column, nz planes) or, with
// ColumnArgs::balanced, an equal share of all the level's column-planes (no partial
// last wave), cut into segments where it crosses into the next column.  Each
// segment stages and reconstructs its own z halo; as no face or cell depends on
// where a segment starts, both give the same bits.
//
// Variants as in the level kernel: GRAV (-DWGRAV), DUAL (-DDUAL_E), NTR tracers
// (-DWRADHYD); one at a time.
//
// The reference does the same per oct on a 27-oct copy
// (src/hydro_utils.c:1407-2238, 2973-3303), recomputing each cell's
// reconstruction up to 9 times and each face twice.
#pragma once
#include <type_traits>
#include "hydro_math.cuh"
#include "schedule.h"

namespace emma {

// n entries of 5 (d,u,v,w,p or a flux) in shared memory, entry i by 16-byte
// accesses of consecutive threads: FP32 4 + 1, FP64 2 + 2 + 1
template <class R>
struct Vec5;
template <>
struct Vec5<float> {
  static __device__ __forceinline__ void st(void *b, int n, int i, const float x[5]) {
    reinterpret_cast<float4 *>(b)[i] = make_float4(x[0], x[1], x[2], x[3]);
    (reinterpret_cast<float *>(b) + 4 * n)[i] = x[4];
  }
  static __device__ __forceinline__ void ld(const void *b, int n, int i, float x[5]) {
    const float4 v = reinterpret_cast<const float4 *>(b)[i];
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
    x[4] = (reinterpret_cast<const float *>(b) + 4 * n)[i];
  }
};
template <>
struct Vec5<double> {
  static __device__ __forceinline__ void st(void *b, int n, int i, const double x[5]) {
    reinterpret_cast<double2 *>(b)[i] = make_double2(x[0], x[1]);
    (reinterpret_cast<double2 *>(b) + n)[i] = make_double2(x[2], x[3]);
    (reinterpret_cast<double *>(b) + 4 * n)[i] = x[4];
  }
  static __device__ __forceinline__ void ld(const void *b, int n, int i, double x[5]) {
    const double2 v = reinterpret_cast<const double2 *>(b)[i], w = (reinterpret_cast<const double2 *>(b) + n)[i];
    x[0] = v.x;
    x[1] = v.y;
    x[2] = w.x;
    x[3] = w.y;
    x[4] = (reinterpret_cast<const double *>(b) + 4 * n)[i];
  }
};

// Geometry, threads and shared memory of a column of 16 x TY cells.
template <class R, int TY_, bool DUAL, int NTR>
struct Col {
  static constexpr int TX = kColumnWidth, TY = TY_;
  static constexpr int kInt = TX * TY, kRing = 2 * (TX + TY);  // column and ring cells of a plane
  static constexpr int kThreads = (kInt + kRing + 31) / 32 * 32;
  static constexpr int PW = TX + 4, kP = PW * (TY + 4);  // staged plane: x in -2 .. TX+1, y in -2 .. TY+1
  static constexpr int kSX = kInt + TY, kSY = kInt + TX;  // entries: column cells, then the ring cells of one side
  static constexpr int kExtra = (DUAL ? 2 : 0) + NTR;    // per face: dual energy's flux and u*, the tracer fluxes
  static constexpr size_t a16(size_t x) { return (x + 15) & ~size_t(15); }
  static constexpr size_t v5(int n) { return a16(sizeof(R) * 5 * n); }
  static constexpr size_t plane = v5(kP);                   // bytes of a staged plane
  static constexpr size_t off_P = 0;                        // [2] staged planes
  static constexpr size_t off_SX = off_P + 2 * plane;      // +x face states (XS: the boundary's)
  static constexpr size_t off_SY = off_SX + v5(kSX);        // +y face states
  static constexpr size_t off_FX = off_SY + v5(kSY);        // x fluxes
  static constexpr size_t off_FY = off_FX + v5(kSX);                // y fluxes
  static constexpr size_t off_EX = off_FY + v5(kSY);                // R [kExtra][kSX], then [kExtra][kSY]
  static constexpr size_t off_EY = off_EX + a16(sizeof(R) * kExtra * kSX);
  static constexpr size_t off_TX = off_EY + a16(sizeof(R) * kExtra * kSY);  // tracer fractions R [NTR][kInt + kRing]
  static constexpr size_t off_C0 = off_TX + a16(sizeof(R) * NTR * (kInt + kRing));  // XS: -x face states of x = 0
  static constexpr size_t bytes = off_C0 + v5(TY);
  static_assert(kInt % 32 == 0, "column warps are whole");

  // ring cell r: x = -1 (r < TY), x = TX, y = -1, y = TY
  // out: 1 the ring, 2 the outer halo column beyond it
  static __device__ __forceinline__ void ring_xy(int r, int out, int &x, int &y) {
    if (r < 2 * TY) {
      x = r < TY ? -out : TX - 1 + out;
      y = r < TY ? r : r - TY;
    } else {
      const int i = r - 2 * TY;
      x = i < TX ? i : i - TX;
      y = i < TX ? -out : TY - 1 + out;
    }
  }
  static __device__ __forceinline__ int pidx(int x, int y) { return (y + 2) * PW + (x + 2); }
};

template <bool DUAL, int NTR>
using Col32 = Col<float, column_height(false), DUAL, NTR>;

// The warp's maximum of the next CFL step's |v| + c_s (src/advanceamr.c:122-128) after
// each of its threads wrote the state Wout: exact in FP64 for every cell that may raise
// wmax (warp-uniform); an FP32 estimate (relative error below 2e-6) screens the others
// out, whole warps at a time.  The cell is looked at where the estimate does not hold: it
// underflowed (below 1e-15), the quotient is 0 (densities beyond FP32, or beyond the 2^126
// from which the approximate division gives 0), the density is below FP32's normal numbers
// (c_s > 1e13 then, with pressures >= 1e-10), or it is no number.
__device__ __forceinline__ double column_cfl_max(const double Wout[5], double wmax) {
  const float u = (float)Wout[1], v = (float)Wout[2], w = (float)Wout[3], q = (float)Wout[4] / (float)Wout[0];
  const float s32 = sqrtf(u * u + v * v + w * w) + sqrtf(5.f / 3.f * q);
  const bool cand = !(s32 < (float)wmax * (1.f - 1e-5f)) || !(s32 > 1e-15f && s32 < 1e13f) || !(q > 0.f);
  if (__any_sync(0xffffffffu, cand)) {
    double ex = 0.;
    if (cand) {
      const double va = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(Wout[1], Wout[1]), __dmul_rn(Wout[2], Wout[2])),
                                             __dmul_rn(Wout[3], Wout[3])));
      const double aa = __dsqrt_rn(__ddiv_rn(__dmul_rn(5. / 3., Wout[4]), Wout[0]));
      ex = fmax(0., __dadd_rn(va, aa));  // fmax drops NaN like the reference's FMAX
    }
    for (int o = 16; o > 0; o >>= 1) ex = fmax(ex, __shfl_xor_sync(0xffffffffu, ex, o));
    wmax = fmax(wmax, ex);
  }
  return wmax;
}

// This CTA's range of the level's column-planes (columns in order, each bottom to top):
// an item (one column, nz planes), or an equal share of all of them cut into segments
// where it crosses into the next column.
template <class F>
__device__ __forceinline__ void column_segments(const ColumnArgs &a, const F &segment, int tx, int ty) {
  const int per_col = 2 * a.n, ncols = a.ncol * a.ncoly;
  int p0, p1;
  if (a.balanced) {
    const long long total = (long long)ncols * per_col;
    p0 = (int)(total * blockIdx.x / gridDim.x);
    p1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
  } else {
    const int cz = blockIdx.x / ncols, col = blockIdx.x % ncols;
    p0 = col * per_col + cz * a.nz;
    p1 = p0 + a.nz;
  }
  for (int pos = p0; pos < p1;) {
    const int col = pos / per_col, z = pos - col * per_col;
    const int zend = (p1 - pos < per_col - z) ? z + (p1 - pos) : per_col;
    segment((col % a.ncol) * tx, (col / a.ncol) * ty, z, zend);
    pos += zend - z;
  }
}

// FP32 reconstruction and fluxes, FP64 update; 320 threads at 96 registers (dual energy
// spills 64 bytes, the tracer 28, gravity 8), two CTAs per SM.  Bound by instruction issue
// (57% of cycles at 128^3, 64% at 256^3, 17 and 19 warps an SM: 42.0 warp instructions a
// cell, FP32 pipe 41% of them, minima, compares and selects 31%), not by memory (68 and 81
// bytes a cell of DRAM traffic).  Measured a launch without the time step's maximum,
// against slopes and all three axes through shared memory and the brick kernel: 256^3 0.973
// ms (1.20, 1.66), 128^3 0.139 ms (0.174, 0.223); against the brick kernel, dual energy
// 0.160 ms (0.246) at 128^3, 64^3 with transmissive x 0.030 ms (0.043).  A step of the
// device schedule, with the maximum: 1.038 and 0.155 ms, dual energy 0.174.
template <bool XS, bool GRAV, bool DUAL, int NTR>
__global__ void __launch_bounds__((Col32<DUAL, NTR>::kThreads), column_ctas(false)) column_kernel(const ColumnArgs a) {
  using M = MathF32;
  using C = Col32<DUAL, NTR>;
  using R = float;
  using V = Vec5<R>;
  using TR = Tracers<(NTR > 0 ? NTR : 1)>;
  constexpr int TX = C::TX, TY = C::TY, kInt = C::kInt, PW = C::PW, kP = C::kP;
  constexpr int NT = NTR > 0 ? NTR : 1;
  static_assert((int)GRAV + (int)DUAL + (NTR > 0) <= 1, "one variant at a time");
  static_assert(!XS || (!GRAV && !DUAL && NTR == 0), "the shuffle sweep is the plain variant's");
  extern __shared__ __align__(16) unsigned char smem[];
  if (a.gate != nullptr && *a.gate == 0) return;
  if ((int)blockIdx.x >= a.nitems) return;
  unsigned char *sSX = smem + C::off_SX, *sSY = smem + C::off_SY, *sFX = smem + C::off_FX, *sFY = smem + C::off_FY;
  R *sEX = reinterpret_cast<R *>(smem + C::off_EX), *sEY = reinterpret_cast<R *>(smem + C::off_EY);
  R *sT = reinterpret_cast<R *>(smem + C::off_TX);
  auto sP = [&](int slot) { return smem + C::off_P + slot * C::plane; };

  const LevelArgs &A = *a.lv;
  const double *__restrict__ W = A.W;
  double *__restrict__ Wn = A.Wn;
  const long long N8 = 8LL * A.noct;
  const double dt = A.dt, dtsurdx = dt / A.dx;
  const R hfac = (R)(dtsurdx * 0.5);  // as the brick kernel's
  const int n = a.n, cmask = 2 * n - 1;
  const long long nn = (long long)n * n;
  const int *__restrict__ octidx = a.octidx;

  const int tid = threadIdx.x;
  const bool interior = tid < kInt;
  const int ring = tid - kInt;
  const bool cell = tid < kInt + C::kRing;  // the last threads of a padded warp own no cell
  unsigned st = 0;
  double wmax = 0.;  // exact max signal speed of the cells this warp wrote (warp-uniform)

  // this thread's cell and the second column it stages (ring threads: an outer halo
  // column; four column threads: a ring corner column)
  int rx = 0, ry = 0, hx = 0, hy = 0;
  constexpr int kCornerT0 = kInt - 4;
  const bool conv2 = cell && (!interior || tid >= kCornerT0);
  if (interior) {
    rx = tid % TX;
    ry = tid / TX;
    if (conv2) {
      const int k = tid - kCornerT0;
      hx = (k & 1) ? TX : -1;
      hy = (k & 2) ? TY : -1;
    }
  } else if (cell) {
    C::ring_xy(ring, 1, rx, ry);
    C::ring_xy(ring, 2, hx, hy);
  }
  const int rp = C::pidx(rx, ry), hp = C::pidx(hx, hy);
  // plane-independent parts of the global cell index: periodic, or the boundary
  // cell's copies beyond a transmissive x face (the reference's ghost octs)
  int oxy1 = 0, cxy1 = 0, oxy2 = 0, cxy2 = 0;  // set per segment
  auto xy_part = [&](int x, int y, int &oxy, int &cxy) {
    int xg = x;
    if ((a.trans & 1) && xg < 0) xg = 0;
    if ((a.trans & 2) && xg > cmask) xg = cmask;
    xg &= cmask;
    const int yg = y & cmask;
    oxy = (yg >> 1) * n + (xg >> 1);
    cxy = (xg & 1) | ((yg & 1) << 1);
  };
  auto oct_at = [&](int oxy, int z) { return __ldg(octidx + ((z & cmask) >> 1) * nn + oxy); };
  auto gidx = [](int oct, int cxy, int z) -> long long { return 8LL * oct + (cxy | ((z & 1) << 2)); };
  auto load5 = [&](long long gi, double q[5]) {
#pragma unroll
    for (int v = 0; v < 5; v++) q[v] = __ldg(W + v * N8 + gi);
  };
  auto cvt5 = [](const double q[5], R x[5]) {
#pragma unroll
    for (int v = 0; v < 5; v++) x[v] = (R)q[v];
  };

  // one face normal to axis d between the face states WL, WR (5 values each), flux F
  // (and du, fx as hllc gives them)
  auto solve = [&](auto dc, const R L5[5], const R R5[5], R F[5], R *du, const R *xs, R *fx) {
    constexpr int d = decltype(dc)::value;
    R WL[7], WR[7];
#pragma unroll
    for (int v = 0; v < 5; v++) {
      WL[v] = L5[v];
      WR[v] = R5[v];
    }
    M::face_finish(WL);
    M::face_finish(WR);
    if constexpr (NTR > 0) M::template hllc<NTR>(WL, WR, d, F, st, nullptr, xs, fx);
    else M::hllc(WL, WR, d, F, st, DUAL ? du : nullptr);
  };
  using D0 = std::integral_constant<int, 0>;
  using D1 = std::integral_constant<int, 1>;
  using D2 = std::integral_constant<int, 2>;

  // the x and y faces each thread solves: column cells their -x and -y faces, the +x
  // ring the column's +x boundary faces, the +y ring its +y boundary faces (XS: the
  // -x boundary faces the -x ring)
  const bool ring_xm = !interior && ring < TY, ring_xp = !interior && ring >= TY && ring < 2 * TY;
  const bool ring_ym = cell && !interior && ring >= 2 * TY && ring < 2 * TY + TX;
  const bool ring_yp = cell && !interior && ring >= 2 * TY + TX;
  const int lx = interior ? ((rx == 0) ? kInt + ry : tid - 1) : ry * TX + TX - 1;  // left cell's entry in SX
  const int ex = interior ? tid : kInt + ry;                                      // flux entry in FX
  const int ly = interior ? ((ry == 0) ? kInt + rx : tid - TX) : (TY - 1) * TX + rx;
  const int ey = interior ? tid : kInt + rx;
  // the left cells' places in the tracer fractions
  const int tlx = interior ? ((rx == 0) ? kInt + ry : tid - 1) : lx;
  const int tly = interior ? ((ry == 0) ? kInt + 2 * TY + rx : tid - TX) : ly;
  // the +x and +y fluxes of a column cell
  const int px = (rx == TX - 1) ? kInt + ry : tid + 1, py = (ry == TY - 1) ? kInt + rx : tid + TX;

  // The update of a column cell of plane z-1: q its FP64 state, its x and y fluxes in
  // shared memory, F0/F1 its -z and +z fluxes (d0/d1, f0/f1 their du and tracer
  // fluxes).  The brick kernel's expressions (level_kernel.cuh P3) for a level that
  // receives no corrections.
  auto update = [&](long long gi, const double q[5], const R F0[5], const R F1[5], const R d0[2], const R d1[2],
                    const R f0[NT], const R f1[NT]) {
    double dU[5] = {0., 0., 0., 0., 0.}, dUe = 0., divu = 0., dT[NT] = {};
    const double eold = MathF64::over_g1(q[4]);
    auto add = [&](int k, const R F[5], R fe, R us, const R *fx) {  // faces in the order -x,+x,-y,+y,-z,+z
      const double one = (k & 1) ? -1. : 1.;
#pragma unroll
      for (int v = 0; v < 5; v++) {
        dU[v] = (k & 1) ? dU[v] - (double)F[v] : dU[v] + (double)F[v];  // updatefield (src/hydro_utils.c:3050-3082)
      }
      if constexpr (DUAL) {  // src/hydro_utils.c:2126-2129, 3064, 3167-3177
        dUe += (double)fe * dtsurdx * one;
        const double dl = (kGam - 1.) * (double)us * eold;
        divu += (k & 1) ? dl : -dl;
      }
#pragma unroll
      for (int t = 0; t < NTR; t++) dT[t] += (double)fx[t] * dtsurdx * one;
    };
    auto add_s = [&](int k, const unsigned char *sF, const R *sE, int n, int e) {
      R F[5], fe = (R)0, us = (R)0, fx[NT] = {};
      V::ld(sF, n, e, F);
      if constexpr (DUAL) {
        fe = sE[e];
        us = sE[n + e];
      }
#pragma unroll
      for (int t = 0; t < NTR; t++) fx[t] = sE[t * n + e];
      add(k, F, fe, us, fx);
    };
    add_s(0, sFX, sEX, C::kSX, tid);
    add_s(1, sFX, sEX, C::kSX, px);
    add_s(2, sFY, sEY, C::kSY, tid);
    add_s(3, sFY, sEY, C::kSY, py);
    add(4, F0, DUAL ? d0[0] : (R)0, DUAL ? d0[1] : (R)0, f0);
    add(5, F1, DUAL ? d1[0] : (R)0, DUAL ? d1[1] : (R)0, f1);
    // conserved state W2U(W) + dU (src/hydro_utils.c:3129-3188).  The mixed path's
    // compensated sum of the base state and the flux divergence returns the rounded sum
    // when there are only these two terms.
    const double Ud = q[0] + dU[0] * dtsurdx;
    const double Udu = q[0] * q[1] + dU[1] * dtsurdx;
    const double Udv = q[0] * q[2] + dU[2] * dtsurdx;
    const double Udw = q[0] * q[3] + dU[3] * dtsurdx;
    const double UE =
        (MathF64::over_g1(q[4]) + 0.5 * q[0] * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3])) + dU[4] * dtsurdx;
    // U2W (src/hydro_utils.c:35-64), pressure floor
    const double dl = (Ud == 0. ? 10. : Ud), mm = Udu * Udu + Udv * Udv + Udw * Udw, inv = 1. / dl;
    double Wout[5] = {Ud, Udu * inv, Udv * inv, Udw * inv, (kGam - 1.) * (UE - mm * inv * 0.5)};
    if constexpr (DUAL) {
      // the tracked eint, unless E - Ekin is well resolved against div(u); the
      // floor; the pressure from eint (src/hydro_utils.c:3164-3182, 45-46)
      const double ekin = 0.5 * mm / Ud;
      double eint = eold + dUe;
      eint = eint + (-divu * dtsurdx);
      if ((UE - ekin) > 0.5 * (divu * divu)) eint = UE - ekin;
      eint = MathF64::over_g1(fmax(eint * (kGam - 1.), kPmin));
      Wout[4] = eint * (kGam - 1.);
    }
    Wout[4] = fmax(Wout[4], kPmin);
    if (isnan(Wout[1]) || isnan(Wout[4]) || isnan(Wout[0])) st |= kStNan;
    if constexpr (GRAV) {  // grav_correction (src/hydro_utils.c:2388-2444, PRIMITIVE)
      if (A.gcorr) {
#pragma unroll
        for (int v = 0; v < 3; v++) Wout[1 + v] += (-__ldg(A.F + v * N8 + gi) * dt);
      }
    }
#pragma unroll
    for (int v = 0; v < 5; v++) Wn[v * N8 + gi] = Wout[v];
#pragma unroll
    for (int t = 0; t < NTR; t++) {  // dX in [0, d (1 - YHE)], helium below d YHE (src/hydro_utils.c:3197-3203)
      double x = __ldg(W + (5 + t) * N8 + gi) + dT[t];
      if (t == 0 && x < 0) x = 0.;
      if (x > (Wout[0] * (TR::frac(t)))) x = Wout[0] * (TR::frac(t));
      Wn[(5 + t) * N8 + gi] = x;
    }
    if (a.smax != nullptr) wmax = column_cfl_max(Wout, wmax);
  };

  // One segment: planes [z0, z1) of the column at (x0, y0), the two planes below and
  // above it staged (one of each reconstructed) as its halo.
  auto segment = [&](int x0, int y0, int z0, int z1) {
    xy_part(x0 + rx, y0 + ry, oxy1, cxy1);
    xy_part(x0 + hx, y0 + hy, oxy2, cxy2);
    R qm[5] = {}, qc[5] = {}, qn[5] = {};      // states of the planes z-1, z and z+1
    double fl[3] = {};                         // GRAV: the cell's acceleration at plane z
    R tm[NT] = {}, tc[NT] = {}, tn[NT] = {};   // tracer fractions at planes z-1, z, z+1
    int on1 = 0, on2 = 0;                      // octs of plane z+2
    // plane zz of the cell (oct o) or the second column: loaded, and staged into its slot
    auto fractions_of = [&](long long gi, double d, R f[NT]) {  // X0 = dT / (d frac) (src/hydro_utils.c:1245, 1248-1251)
#pragma unroll
      for (int t = 0; t < NTR; t++) f[t] = (R)(__ldg(W + (5 + t) * N8 + gi) / (d * (TR::frac(t))));
    };
    auto stage = [&](int zz, int p, const double q[5], R x[5]) {
      cvt5(q, x);
      V::st(sP(zz & 1), kP, p, x);
    };
    if (cell) {
      double q[5];
      R x[5];
      load5(gidx(oct_at(oxy1, z0 - 2), cxy1, z0 - 2), q);
      cvt5(q, qm);
      long long gi = gidx(oct_at(oxy1, z0 - 1), cxy1, z0 - 1);
      load5(gi, q);
      stage(z0 - 1, rp, q, qc);
      if constexpr (GRAV)
        for (int v = 0; v < 3; v++) fl[v] = __ldg(A.F + v * N8 + gi);
      fractions_of(gi, q[0], tc);
      gi = gidx(oct_at(oxy1, z0), cxy1, z0);
      load5(gi, q);
      stage(z0, rp, q, qn);
      fractions_of(gi, q[0], tn);
      on1 = oct_at(oxy1, z0 + 1);
      if (conv2) {
        load5(gidx(oct_at(oxy2, z0 - 1), cxy2, z0 - 1), q);
        stage(z0 - 1, hp, q, x);
        load5(gidx(oct_at(oxy2, z0), cxy2, z0), q);
        stage(z0, hp, q, x);
        on2 = oct_at(oxy2, z0 + 1);
      }
    }
    __syncthreads();

    R zhi[5] = {}, Fz[5] = {}, dz[2] = {}, fz[NT] = {};  // +z face state, -z flux (and its du, fx) of the last plane
    R xlo[5] = {}, ylo[5] = {}, xhi[5] = {};             // FP32: this plane's -x, -y (and, XS, +x) face states
    for (int z = z0 - 1; z <= z1; z++) {
      // ---------------------------------------------------------------- A
      const bool xy = z >= z0 && z < z1;  // the halo planes close z faces only
      R Fn[5] = {}, dn[2] = {}, fn[NT] = {};  // the -z flux of plane z
      if (cell) {
        R D[3][5], Wt[5], X[5], gk[3] = {(R)0, (R)0, (R)0};
        {
          const unsigned char *P = sP(z & 1);
          R nm[3][5], np[3][5];
          V::ld(P, kP, rp - 1, nm[0]);
          V::ld(P, kP, rp + 1, np[0]);
          V::ld(P, kP, rp - PW, nm[1]);
          V::ld(P, kP, rp + PW, np[1]);
#pragma unroll
          for (int v = 0; v < 5; v++) {
            nm[2][v] = qm[v];
            np[2][v] = qn[v];
          }
          M::muscl(qc, nm, np, hfac, D, Wt);
        }
        if constexpr (GRAV) {
#pragma unroll
          for (int v = 0; v < 3; v++) gk[v] = (R)(-fl[v] * 0.5 * dt);
        }
#pragma unroll
        for (int v = 0; v < 5; v++) X[v] = qc[v] + Wt[v];
        if constexpr (GRAV) {
#pragma unroll
          for (int v = 0; v < 3; v++) X[1 + v] += gk[v];
        }
        auto face = [&](auto kc, R F5[5]) {
          constexpr int k = decltype(kc)::value;
          R w[7];
          M::face_px5(X, D[k >> 1], k, w, st);
#pragma unroll
          for (int v = 0; v < 5; v++) F5[v] = w[v];
        };
        if (xy) {
          R h[5];
          face(std::integral_constant<int, 0>{}, xlo);
          face(std::integral_constant<int, 2>{}, ylo);
          face(std::integral_constant<int, 1>{}, h);
          if constexpr (XS) {
            if (interior && rx == 0) V::st(smem + C::off_C0, TY, ry, xlo);
            if (interior && rx == TX - 1) V::st(sSX, C::kSX, tid, h);
#pragma unroll
            for (int v = 0; v < 5; v++) xhi[v] = h[v];
          } else if (interior || ring_xm) {
            V::st(sSX, C::kSX, ex, h);
          }
          face(std::integral_constant<int, 3>{}, h);
          if (interior || ring_ym) V::st(sSY, C::kSY, ey, h);
          if constexpr (NTR > 0) {
#pragma unroll
            for (int t = 0; t < NTR; t++) sT[t * (kInt + C::kRing) + tid] = tc[t];
          }
        }
        R zl[5], zh[5];
        face(std::integral_constant<int, 4>{}, zl);
        face(std::integral_constant<int, 5>{}, zh);
        if (interior && z >= z0) {
          R xs[2 * NT];
#pragma unroll
          for (int t = 0; t < NTR; t++) {
            xs[2 * t] = tm[t];
            xs[2 * t + 1] = tc[t];
          }
          solve(D2{}, zhi, zl, Fn, dn, xs, fn);
          if constexpr (DUAL) {  // as the x and y faces keep them: flux, u*
            const R us = dn[0];
            dn[0] = us * dn[1];
            dn[1] = us;
          }
        }
#pragma unroll
        for (int v = 0; v < 5; v++) zhi[v] = zh[v];
#pragma unroll
        for (int v = 0; v < 5; v++) {
          qm[v] = qc[v];
          qc[v] = qn[v];
        }
#pragma unroll
        for (int t = 0; t < NTR; t++) {
          tm[t] = tc[t];
          tc[t] = tn[t];
        }
      }
      if (interior && z > z0) {
        // the FP64 state of plane z-1 again, from L2: loaded here and not ahead of the z
        // face, whose solve would carry its 10 registers (128^3 0.151 against 0.139 ms, dual
        // energy 0.180 against 0.159)
        const long long gu = gidx(oct_at(oxy1, z - 1), cxy1, z - 1);
        double qu[5];
        load5(gu, qu);
        update(gu, qu, Fz, Fn, dz, dn, fz, fn);
      }
      if (interior) {
#pragma unroll
        for (int v = 0; v < 5; v++) Fz[v] = Fn[v];
        if constexpr (DUAL) {
          dz[0] = dn[0];
          dz[1] = dn[1];
        }
#pragma unroll
        for (int t = 0; t < NTR; t++) fz[t] = fn[t];
      }
      __syncthreads();
      // ---------------------------------------------------------------- B
      // the loads of plane z+2 land while the x faces are solved, those of its second
      // column while the y faces are; its slot held plane z, read before the barrier
      const bool next = cell && z < z1, next2 = conv2 && z + 1 < z1;
      double q[5];
      long long gi = 0;
      if (next) {
        gi = gidx(on1, cxy1, z + 2);
        load5(gi, q);
        on1 = oct_at(oxy1, z + 3);
      }
      R F[5], du[2] = {}, fx[NT], xs[2 * NT], L5[5], R5[5];
      auto keep = [&](unsigned char *sF, R *sE, int n, int e) {
        V::st(sF, n, e, F);
        if constexpr (DUAL) {
          sE[e] = du[0] * du[1];  // (Us.m_n / Us.d) ebar (src/hydro_utils.c:2128)
          sE[n + e] = du[0];
        }
#pragma unroll
        for (int t = 0; t < NTR; t++) sE[t * n + e] = fx[t];
      };
      auto fractions = [&](int left) {  // tm: this plane's, after the shift
#pragma unroll
        for (int t = 0; t < NTR; t++) {
          xs[2 * t] = sT[t * (kInt + C::kRing) + left];
          xs[2 * t + 1] = tm[t];
        }
      };
      if constexpr (XS) {
        if (xy && interior) {  // whole warps: every lane takes part in the shuffle
#pragma unroll
          for (int v = 0; v < 5; v++) L5[v] = __shfl_up_sync(0xffffffffu, xhi[v], 1);
          const unsigned st0 = st;
          solve(D0{}, L5, xlo, F, du, xs, fx);
          if (rx != 0) keep(sFX, sEX, C::kSX, ex);
          else st = st0;
        }
      }
      if (xy && (XS ? (ring_xm || ring_xp) : (interior || ring_xp))) {
        int e = ex;
        if (XS && ring_xm) {
#pragma unroll
          for (int v = 0; v < 5; v++) L5[v] = xhi[v];
          V::ld(smem + C::off_C0, TY, ry, R5);
          e = ry * TX;
        } else {
          V::ld(sSX, C::kSX, lx, L5);
#pragma unroll
          for (int v = 0; v < 5; v++) R5[v] = xlo[v];
        }
        fractions(tlx);
        solve(D0{}, L5, R5, F, du, xs, fx);
        keep(sFX, sEX, C::kSX, e);
      }
      if (next) {
        stage(z + 2, rp, q, qn);
        fractions_of(gi, q[0], tn);
      }
      if (next2) {
        load5(gidx(on2, cxy2, z + 2), q);
        on2 = oct_at(oxy2, z + 3);
      }
      if constexpr (GRAV) {
        if (next) {  // the acceleration at plane z+1
          const long long gf = gidx(oct_at(oxy1, z + 1), cxy1, z + 1);
#pragma unroll
          for (int v = 0; v < 3; v++) fl[v] = __ldg(A.F + v * N8 + gf);
        }
      }
      if (xy && (interior || ring_yp)) {
        V::ld(sSY, C::kSY, ly, L5);
        fractions(tly);
        solve(D1{}, L5, ylo, F, du, xs, fx);
        keep(sFY, sEY, C::kSY, ey);
      }
      if (next2) {
        R x[5];
        stage(z + 2, hp, q, x);
      }
      __syncthreads();
    }
  };

  column_segments(a, segment, TX, TY);
  if (a.smax != nullptr && interior && (tid & 31) == 0 && wmax > 0.)
    atomicMax(a.smax + a.L, (unsigned long long)__double_as_longlong(wmax));
  if (st) atomicOr(a.status, st);
  // every thread has read the level's slot
  if (a.end != nullptr && threadIdx.x == 0) batch_end_by_last(a.end, const_cast<LevelArgs *>(a.lv) - a.L);
}

// The launchers have internal linkage, as the level kernel's (level_kernel.cuh): the
// libraries of a process share these object files, each sets its own kernels' limits.
namespace {

constexpr int kColumnMaxDev = 64;

template <class K>
cudaError_t launch_column_kernel(K k, bool *attr_set, int threads, size_t bytes, const ColumnArgs &a, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kColumnMaxDev) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {  // the shared-memory limit is a per-device attribute
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  if (a.nitems <= 0) return cudaSuccess;
  k<<<a.nitems, threads, bytes, s>>>(a);
  return cudaGetLastError();
}

template <bool XS, bool GRAV, bool DUAL, int NTR>
cudaError_t launch_column32(const ColumnArgs &a, cudaStream_t s) {
  using C = Col32<DUAL, NTR>;
  static_assert(column_ctas(false) * (C::bytes + 1024) <= 228 * 1024, "CTAs per SM by shared memory");
  static bool attr_set[kColumnMaxDev] = {false};
  return launch_column_kernel(column_kernel<XS, GRAV, DUAL, NTR>, attr_set, C::kThreads, C::bytes, a, s);
}

}  // namespace
}  // namespace emma
