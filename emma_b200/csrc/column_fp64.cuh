// column_fp64.cuh -- the FP64 column kernel: the hydro level advance of a complete
// level without split cells (periodic, or transmissive in x), marching through z.
//
// The same columns and faces as the mixed path's kernel (column_kernel.cuh) and the
// expressions of the brick kernel (equal bits), laid out for FP64: a face's Riemann
// solve is a chain of dependent FP64 operations that fills no pipe, and a thread that
// also carried its column through z (168 registers) left room for ten warps on an SM:
// 0.51 ms a launch at 128^3, no better than the bricks' 0.53.  Here every face of a plane
// has a thread of its own and the marching state lives in shared memory: 16 x 8-cell
// columns, 13 warps at 72 registers, two CTAs, 26 warps on an SM; 0.371 ms, 0.388 a step
// with the time step's maximum (one 16 x 16-cell CTA of 25 warps: as fast there, but 0.030
// against 0.023 ms at 32^3, where columns are few).  The 72 registers spill: 24 bytes
// stored a thread, with gravity 88, dual energy 72, the tracer 236.  Bound by issue (57% of
// cycles) and the barriers between the two phases; FP64 instructions are 45% of all.
// 64^3: 0.067 ms (bricks 0.081); 32^3: 0.022 (0.041).
//
// Step z, two barriers:
//   A  warps 0-5 reconstruct plane z (128 column cells, 48 ring cells) and write each
//      face's left and right state; warps 6-9 update plane z-2;
//   B  every warp solves faces: 4 warps each the -x, -y and -z faces of plane z, the
//      13th the +x and +y faces of the column's boundary; asynchronous copies bring
//      plane z+2 into the slot of plane z-1.
// Face states are stored in the face's frame (normal velocity first), so that one
// copy of the solver serves the three axes.
#pragma once
#include "column_kernel.cuh"

namespace emma {

template <bool DUAL, int NTR>
struct Col64 {
  static constexpr int TX = kColumnWidth, TY = column_height(true);
  static constexpr int kInt = TX * TY, kRec = kInt + 2 * (TX + TY);
  static constexpr int kUpd = (kRec + 31) / 32 * 32;  // first thread of the update
  static constexpr int kThreads = 3 * kInt + 32;      // a thread for every face of a plane
  static_assert(TX + TY <= 32 && kUpd + kInt <= kThreads, "boundary faces in one warp");
  static constexpr int PW = TX + 4, kP = PW * (TY + 4);
  static constexpr int kSX = kInt + TY, kSY = kInt + TX, kSZ = kInt;  // faces per axis and plane
  static constexpr int kExtra = (DUAL ? 2 : 0) + NTR;
  static constexpr size_t v5(int n) { return 40 * (size_t)n; }
  static constexpr size_t plane = v5(kP), pX = v5(kSX), pY = v5(kSY), pZ = v5(kSZ);
  static constexpr size_t off_P = 0;                 // [3] staged planes
  static constexpr size_t off_LX = off_P + 3 * plane;  // left and right face states
  static constexpr size_t off_RX = off_LX + pX;
  static constexpr size_t off_LY = off_RX + pX;
  static constexpr size_t off_RY = off_LY + pY;
  static constexpr size_t off_RZ = off_RY + pY;
  static constexpr size_t off_LZ = off_RZ + pZ;      // [2], by the plane of the left cell
  static constexpr size_t off_FX = off_LZ + 2 * pZ;  // [2] fluxes, by plane
  static constexpr size_t off_FY = off_FX + 2 * pX;
  static constexpr size_t off_FZ = off_FY + 2 * pY;
  static constexpr int kF = kSX + kSY + kSZ;         // faces of a plane: x, y, z
  static constexpr size_t off_E = off_FZ + 2 * pZ;   // double [2][kExtra][kF]
  static constexpr size_t off_T = off_E + 8 * (size_t)(2 * kExtra * kF);  // tracer fractions, double [2][NTR][kRec]
  struct Shared {  // uniform values of the launch and the segment; the update warps' signal-speed maxima
    const double *W, *F;
    double *Wn;
    long long N8;
    double dt, dtsurdx;
    int gcorr, x0, y0, pad;
    double wmax[kInt / 32];
  };
  static constexpr size_t off_G = off_T + 8 * (size_t)(2 * NTR * kRec);
  static constexpr size_t bytes = (off_G + sizeof(Shared) + 15) & ~size_t(15);
  static_assert(plane % 16 == 0 && pX % 16 == 0 && pY % 16 == 0 && pZ % 16 == 0, "16-byte entries");
  static_assert(column_ctas(true) * (bytes + 1024) <= 228 * 1024, "CTAs per SM by shared memory");
  using Ring = Col<double, TY, DUAL, NTR>;
};

template <bool GRAV, bool DUAL, int NTR>
__global__ void __launch_bounds__((Col64<DUAL, NTR>::kThreads), column_ctas(true)) column_fp64_kernel(const ColumnArgs a) {
  using C = Col64<DUAL, NTR>;
  using M = MathF64;
  using V = Vec5<double>;
  using TR = Tracers<(NTR > 0 ? NTR : 1)>;
  constexpr int TX = C::TX, TY = C::TY, kInt = C::kInt, PW = C::PW, kP = C::kP;
  constexpr int NT = NTR > 0 ? NTR : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  if (a.gate != nullptr && *a.gate == 0) return;
  if ((int)blockIdx.x >= a.nitems) return;
  // What every phase needs and no phase should carry in a register through the others:
  // read again (volatile) where it is used, like the thread's number and all that follows
  // from it.  Held across the face solves, these values cost 25 of the 72 registers.
  typename C::Shared &G = *reinterpret_cast<typename C::Shared *>(smem + C::off_G);
  const volatile typename C::Shared &U = G;
  if (threadIdx.x == 0) {
    const LevelArgs &A = *a.lv;
    G.W = A.W;
    G.Wn = A.Wn;
    G.F = A.F;
    G.N8 = 8LL * A.noct;
    G.dt = A.dt;
    G.dtsurdx = A.dt / A.dx;
    G.gcorr = A.gcorr;
    for (int i = 0; i < kInt / 32; i++) G.wmax[i] = 0.;
  }
  __syncthreads();
  unsigned st = 0;
  auto thread = []() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
  };
  auto sP = [&](int z) { return smem + C::off_P + (((z % 3) + 3) % 3) * C::plane; };
  auto sE = [&](int slot, int k) { return reinterpret_cast<double *>(smem + C::off_E) + (slot * C::kExtra + k) * C::kF; };
  auto sT = [&](int slot, int t) { return reinterpret_cast<double *>(smem + C::off_T) + (slot * NTR + t) * C::kRec; };
  // global index of the cell at (x, y) of the segment's column in plane z: periodic, or
  // the boundary cell's copy beyond a transmissive x face
  auto gidx = [&](int x, int y, int z) -> long long {
    const int n = a.n, cmask = 2 * n - 1;
    int xg = U.x0 + x;
    if ((a.trans & 1) && xg < 0) xg = 0;
    if ((a.trans & 2) && xg > cmask) xg = cmask;
    xg &= cmask;
    const int yg = (U.y0 + y) & cmask, zg = z & cmask;
    const int oct = __ldg(a.octidx + ((long long)(zg >> 1) * n + (yg >> 1)) * n + (xg >> 1));
    return 8LL * oct + ((xg & 1) | ((yg & 1) << 1) | ((zg & 1) << 2));
  };

  // The update of column cell ut in plane u; returns nothing, the warp's signal-speed
  // maximum is kept in shared memory.
  auto update = [&](int ut, int u) {
    const int ux = ut & (TX - 1), uy = ut / TX;
    const long long gi = gidx(ux, uy, u), N8 = U.N8;
    const double *W = const_cast<const double *>(U.W);
    const double dt = U.dt, dtsurdx = U.dtsurdx;
    double q[5];
#pragma unroll
    for (int v = 0; v < 5; v++) q[v] = __ldg(W + v * N8 + gi);
    const int slot = u & 1;
    double dU[5] = {0., 0., 0., 0., 0.}, dUe = 0., divu = 0., dT[NT] = {};
    const double eold = M::over_g1(q[4]);
    // faces in the order -x,+x,-y,+y,-z,+z (updatefield, src/hydro_utils.c:3050-3082)
    auto add = [&](auto kc, const unsigned char *sF, int m, int e, int fs, int fb) {
      constexpr int k = decltype(kc)::value, ax = k >> 1;
      constexpr double one = (k & 1) ? -1. : 1.;
      double f[5];
      V::ld(sF, m, e, f);  // mass, normal, transverse (x,y,z order), energy
      const double F[5] = {f[0], ax == 0 ? f[1] : f[2], ax == 0 ? f[2] : (ax == 1 ? f[1] : f[3]), ax == 2 ? f[1] : f[3],
                           f[4]};
#pragma unroll
      for (int v = 0; v < 5; v++) dU[v] += F[v] * dtsurdx * one;
      if constexpr (DUAL) {  // src/hydro_utils.c:2126-2129, 3064, 3167-3177
        dUe += sE(fs, 0)[fb + e] * dtsurdx * one;
        const double dl = (kGam - 1.) * sE(fs, 1)[fb + e] * eold;
        divu += (k & 1) ? dl : -dl;
      }
#pragma unroll
      for (int t = 0; t < NTR; t++) dT[t] += sE(fs, t)[fb + e] * dtsurdx * one;
    };
    const unsigned char *FX = smem + C::off_FX + slot * C::pX, *FY = smem + C::off_FY + slot * C::pY;
    add(std::integral_constant<int, 0>{}, FX, C::kSX, ut, slot, 0);
    add(std::integral_constant<int, 1>{}, FX, C::kSX, ux == TX - 1 ? kInt + uy : ut + 1, slot, 0);
    add(std::integral_constant<int, 2>{}, FY, C::kSY, ut, slot, C::kSX);
    add(std::integral_constant<int, 3>{}, FY, C::kSY, uy == TY - 1 ? kInt + ux : ut + TX, slot, C::kSX);
    add(std::integral_constant<int, 4>{}, smem + C::off_FZ + slot * C::pZ, C::kSZ, ut, slot, C::kSX + C::kSY);
    add(std::integral_constant<int, 5>{}, smem + C::off_FZ + (slot ^ 1) * C::pZ, C::kSZ, ut, slot ^ 1, C::kSX + C::kSY);
    // conserved state W2U(W) + dU (src/hydro_utils.c:3129-3188)
    const double Ud = q[0] + dU[0], Udu = q[0] * q[1] + dU[1], Udv = q[0] * q[2] + dU[2], Udw = q[0] * q[3] + dU[3];
    const double UE = (M::over_g1(q[4]) + 0.5 * q[0] * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3])) + dU[4];
    // U2W (src/hydro_utils.c:35-64), pressure floor
    const double dl = (Ud == 0. ? 10. : Ud), mm = Udu * Udu + Udv * Udv + Udw * Udw, y = M::rcp(dl);
    double Wout[5] = {Ud, M::div_y(Udu, dl, y), M::div_y(Udv, dl, y), M::div_y(Udw, dl, y),
                      (kGam - 1.) * (UE - M::div_y(mm, dl, y) * 0.5)};
    if (!isfinite(Wout[4])) {  // out of div_y's range: by division
      Wout[1] = Udu / dl;
      Wout[2] = Udv / dl;
      Wout[3] = Udw / dl;
      Wout[4] = (kGam - 1.) * (UE - mm / dl * 0.5);
    }
    if constexpr (DUAL) {
      // the tracked eint, unless E - Ekin is well resolved against div(u); the
      // floor; the pressure from eint (src/hydro_utils.c:3164-3182, 45-46)
      const double ekin = 0.5 * mm / Ud;
      double eint = eold + dUe;
      eint = eint + (-divu * dtsurdx);
      if ((UE - ekin) > 0.5 * (divu * divu)) eint = UE - ekin;
      eint = M::over_g1(fmax(eint * (kGam - 1.), kPmin));
      Wout[4] = eint * (kGam - 1.);
    }
    Wout[4] = fmax(Wout[4], kPmin);
    if (isnan(Wout[1]) || isnan(Wout[4]) || isnan(Wout[0])) st |= kStNan;
    if constexpr (GRAV) {  // grav_correction (src/hydro_utils.c:2388-2444, PRIMITIVE)
      if (U.gcorr) {
        const double *F = const_cast<const double *>(U.F);
#pragma unroll
        for (int v = 0; v < 3; v++) Wout[1 + v] += (-__ldg(F + v * N8 + gi) * dt);
      }
    }
    double *Wn = const_cast<double *>(U.Wn);
#pragma unroll
    for (int v = 0; v < 5; v++) Wn[v * N8 + gi] = Wout[v];
#pragma unroll
    for (int t = 0; t < NTR; t++) {  // dX in [0, d (1 - YHE)], helium below d YHE (src/hydro_utils.c:3197-3203)
      double x = __ldg(W + (5 + t) * N8 + gi) + dT[t];
      if (t == 0 && x < 0) x = 0.;
      if (x > (Wout[0] * (TR::frac(t)))) x = Wout[0] * (TR::frac(t));
      Wn[(5 + t) * N8 + gi] = x;
    }
    if (a.smax != nullptr) {
      const double w0 = U.wmax[ut / 32], w1 = column_cfl_max(Wout, w0);
      if (w1 > w0 && (ut & 31) == 0) G.wmax[ut / 32] = w1;
      __syncwarp();
    }
  };

  auto segment = [&](int x0, int y0, int z0, int z1) {
    if (thread() == 0) {
      G.x0 = x0;
      G.y0 = y0;
    }
    __syncthreads();
    auto stage = [&](int z) {  // 8-byte asynchronous copies into Vec5's places of entry e
      const int e = thread();
      if (e < kP) {
        const long long N8 = U.N8;
        const double *src = const_cast<const double *>(U.W) + gidx(e % PW - 2, e / PW - 2, z);
        double *b = reinterpret_cast<double *>(sP(z));
        double *dst[5] = {b + 2 * e, b + 2 * e + 1, b + 2 * kP + 2 * e, b + 2 * kP + 2 * e + 1, b + 4 * kP + e};
#pragma unroll
        for (int v = 0; v < 5; v++)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst[v])),
                       "l"(src + v * N8)
                       : "memory");
      }
    };
    auto staged = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
    stage(z0 - 2);
    stage(z0 - 1);
    stage(z0);
    staged();
    __syncthreads();
    for (int z = z0 - 1; z <= z1 + 1; z++) {
      // ---------------------------------------------------------------- A
      const int tid = thread(), ring = tid - kInt;
      if (tid < C::kRec && z <= z1) {
        const bool interior = tid < kInt;
        int rx, ry;
        if (interior) {
          rx = tid % TX;
          ry = tid / TX;
        } else {
          C::Ring::ring_xy(ring, 1, rx, ry);
        }
        const int rp = (ry + 2) * PW + (rx + 2);
        const bool ring_xm = !interior && ring < TY, ring_xp = !interior && ring >= TY && ring < 2 * TY;
        const bool ring_ym = !interior && ring >= 2 * TY && ring < 2 * TY + TX, ring_yp = !interior && ring >= 2 * TY + TX;
        const double dtsurdx = U.dtsurdx;
        const unsigned char *P = sP(z);
        double q0[5], nm[3][5], np[3][5], D[3][5], Wt[5];
        V::ld(P, kP, rp, q0);
        V::ld(P, kP, rp - 1, nm[0]);
        V::ld(P, kP, rp + 1, np[0]);
        V::ld(P, kP, rp - PW, nm[1]);
        V::ld(P, kP, rp + PW, np[1]);
        V::ld(sP(z - 1), kP, rp, nm[2]);
        V::ld(sP(z + 1), kP, rp, np[2]);
        double gk[3] = {0., 0., 0.};
        if constexpr (GRAV || NTR > 0) {
          const long long gi = gidx(rx, ry, z), N8 = U.N8;
          const double *W = const_cast<const double *>(U.W);
          if constexpr (GRAV) {
            const double *F = const_cast<const double *>(U.F);
            const double dt = U.dt;
#pragma unroll
            for (int v = 0; v < 3; v++) gk[v] = -__ldg(F + v * N8 + gi) * 0.5 * dt;
          }
#pragma unroll
          for (int t = 0; t < NTR; t++)  // X0 = dT / (d frac) (src/hydro_utils.c:1245, 1248-1251)
            sT(z & 1, t)[tid] = __ldg(W + (5 + t) * N8 + gi) / (q0[0] * (TR::frac(t)));
        }
        M::muscl(q0, nm, np, -dtsurdx * 0.5, D, Wt);
        // face state k in the face's frame: d, normal, transverse (x,y,z order), p
        auto face = [&](auto kc, unsigned char *s, int m, int e) {
          constexpr int k = decltype(kc)::value, ax = k >> 1;
          double w[7];
          M::face_ax(q0, D[ax], Wt, k, w, st, GRAV ? gk : nullptr);
          const double f[5] = {w[0], w[1 + ax], ax == 0 ? w[2] : w[1], ax == 2 ? w[2] : w[3], w[4]};
          V::st(s, m, e, f);
        };
        if (z >= z0 && z < z1) {
          if (interior || ring_xp) face(std::integral_constant<int, 0>{}, smem + C::off_RX, C::kSX, interior ? tid : kInt + ry);
          if (interior || ring_xm)
            face(std::integral_constant<int, 1>{}, smem + C::off_LX, C::kSX,
                 interior ? (rx == TX - 1 ? kInt + ry : tid + 1) : ry * TX);
          if (interior || ring_yp) face(std::integral_constant<int, 2>{}, smem + C::off_RY, C::kSY, interior ? tid : kInt + rx);
          if (interior || ring_ym)
            face(std::integral_constant<int, 3>{}, smem + C::off_LY, C::kSY,
                 interior ? (ry == TY - 1 ? kInt + rx : tid + TX) : rx);
        }
        if (interior) {
          face(std::integral_constant<int, 4>{}, smem + C::off_RZ, C::kSZ, tid);
          face(std::integral_constant<int, 5>{}, smem + C::off_LZ + (z & 1) * C::pZ, C::kSZ, tid);
        }
      }
      if (tid >= C::kUpd && tid < C::kUpd + kInt && z - 2 >= z0) update(tid - C::kUpd, z - 2);
      __syncthreads();
      // ---------------------------------------------------------------- B
      if (z + 2 <= z1 + 1) stage(z + 2);  // into the slot of plane z-1
      // this thread's face: axis and entry (x, y: from kInt on the boundary faces)
      int fe = thread(), fax = fe / kInt;
      bool has_face = true;
      if (fax == 3) {
        const int i = fe - 3 * kInt;
        fax = i < TY ? 0 : 1;
        fe = kInt + (i < TY ? i : i - TY);
        has_face = i < TY + TX;
      } else {
        fe %= kInt;
      }
      if (has_face && z >= z0 && (fax == 2 ? z <= z1 : z < z1)) {
        const unsigned char *sL = smem + (fax == 0 ? C::off_LX : (fax == 1 ? C::off_LY : C::off_LZ + ((z - 1) & 1) * C::pZ));
        const unsigned char *sR = smem + (fax == 0 ? C::off_RX : (fax == 1 ? C::off_RY : C::off_RZ));
        unsigned char *sF = smem + (fax == 0 ? C::off_FX + (z & 1) * C::pX
                                             : (fax == 1 ? C::off_FY + (z & 1) * C::pY : C::off_FZ + (z & 1) * C::pZ));
        const int m = fax == 0 ? C::kSX : (fax == 1 ? C::kSY : C::kSZ), fb = fax == 0 ? 0 : (fax == 1 ? C::kSX : C::kSX + C::kSY);
        double WL[7], WR[7], F[5], du[2] = {0., 0.}, fx[NT] = {}, xs[2 * NT] = {};
        V::ld(sL, m, fe, WL);
        V::ld(sR, m, fe, WR);
        if constexpr (NTR > 0) {
          // the cells of the face: the left one's place (x, y: the ring's beyond the column), the right one's
          int l = fe, r = fe;
          if (fax == 0) {
            l = fe >= kInt ? (fe - kInt) * TX + TX - 1 : (fe % TX == 0 ? kInt + fe / TX : fe - 1);
            r = fe >= kInt ? kInt + TY + (fe - kInt) : fe;
          } else if (fax == 1) {
            l = fe >= kInt ? (TY - 1) * TX + (fe - kInt) : (fe < TX ? kInt + 2 * TY + fe : fe - TX);
            r = fe >= kInt ? kInt + 2 * TY + TX + (fe - kInt) : fe;
          }
#pragma unroll
          for (int t = 0; t < NTR; t++) {
            xs[2 * t] = sT(fax == 2 ? (z - 1) & 1 : z & 1, t)[l];
            xs[2 * t + 1] = sT(z & 1, t)[r];
          }
        }
        M::face_finish(WL);
        M::face_finish(WR);
        M::template hllc_frame<NT>(WL, WR, fax == 2, F, st, DUAL ? du : nullptr, NTR > 0 ? xs : nullptr,
                                   NTR > 0 ? fx : nullptr);
        V::st(sF, m, fe, F);
        if constexpr (DUAL) {
          sE(z & 1, 0)[fb + fe] = du[0] * du[1];  // (Us.m_n / Us.d) ebar (src/hydro_utils.c:2128)
          sE(z & 1, 1)[fb + fe] = du[0];
        }
#pragma unroll
        for (int t = 0; t < NTR; t++) sE(z & 1, t)[fb + fe] = fx[t];
      }
      staged();
      __syncthreads();
    }
  };

  column_segments(a, segment, TX, TY);
  if (a.smax != nullptr && threadIdx.x < kInt / 32 && U.wmax[threadIdx.x] > 0.)  // after the last step's barrier
    atomicMax(a.smax + a.L, (unsigned long long)__double_as_longlong(U.wmax[threadIdx.x]));
  if (st) atomicOr(a.status, st);
  // every thread has read the level's slot
  if (a.end != nullptr && threadIdx.x == 0) batch_end_by_last(a.end, const_cast<LevelArgs *>(a.lv) - a.L);
}

namespace {  // internal linkage, as the other launchers

template <bool GRAV, bool DUAL, int NTR>
cudaError_t launch_column64(const ColumnArgs &a, cudaStream_t s) {
  using C = Col64<DUAL, NTR>;
  static bool attr_set[kColumnMaxDev] = {false};
  return launch_column_kernel(column_fp64_kernel<GRAV, DUAL, NTR>, attr_set, C::kThreads, C::bytes, a, s);
}

}  // namespace
}  // namespace emma
