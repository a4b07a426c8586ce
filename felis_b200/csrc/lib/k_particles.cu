// Particle kernels of the FELIS slice loop, FP64 plain path.
//
// Compiled with --fmad=false: every expression below is evaluated with the
// operand order of the reference (particlePush.cpp, solveField.cpp,
// rearrangeParticles.cpp) and no contraction, so particles and fields equal the
// CPU restatement bit for bit (the diagnostics' sums have an order and sines of
// their own: last bits).  One thread owns one particle; a block owns one
// tile of <= 256 consecutive particles of one (species, slice), so the
// slice's field plane, weight and wake term are uniform per block.
//
// Data layout in HBM: six FP64 structure-of-arrays (x, y, px, py, theta,
// gamma), species-major then slice-major; loads and stores are coalesced
// 8-byte accesses, 2 KB per array per block.
#include "particles.cuh"

namespace felis {

namespace {

// Bessel table lookup with the row clamped to the table (the reference reads
// past the table when H*xi approaches its end; the clamp is flagged).
__device__ __forceinline__ double BJ(const DevGeom& G, int row, int col, int* err) {
  if (row < 0 || row >= G.bn) {
    set_flag(err, ERR_RADIAL);
    row = row < 0 ? 0 : G.bn - 1;
  }
  return __ldg(G.bessel + (size_t)row * G.bcols + col);
}

// a / b for many numerators: three divisions' worth of work saved per quotient
// by the reciprocal y = 1/b, correctly rounded.  q0 = a y is within two ulps;
// one correction makes it faithful, and the second is then exact by
// Markstein's theorem (Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990: for y = RN(1/b) and a faithful q,
// RN(q + RN(a - b q) y) = RN(a / b) while nothing under- or overflows, which
// the caller's window on the operands ensures).  FAST = false divides.
template <bool FAST>
struct Quot {
  double b, y;
  __device__ __forceinline__ explicit Quot(double d) : b(d), y(FAST ? 1.0 / d : 0.0) {}
  __device__ __forceinline__ double operator()(double a) const {
    if (!FAST) return a / b;
    double q = a * y;
    q = fma(fma(-b, q, a), y, q);
    return fma(fma(-b, q, a), y, q);
  }
};
// |v| in [2^-span, 2^span).  With the phase-space coordinates zero or within
// span 400, gamma within 100 and the coefficients within 60, every sum, product
// and quotient of a transverse step is zero or far from the ends of the range.
__device__ __forceinline__ bool within(double v, unsigned span) {
  return ((unsigned)__double2hiint(v) >> 20 & 0x7ffu) - (1023u - span) < 2u * span;
}

// particlePush.cpp:82-110 for one particle.  NARROW: aa and dd are zero (no
// polarisation, ue = 0), whose terms leave the sums as they are.
template <bool FAST, bool NARROW>
__device__ __forceinline__ void transverse_steps(const TransCoef& t, double& x_, double& y_, double& px_, double& py_,
                                                 double gam) {
  const double dz = t.dz, aa = t.aa;
  const int K0_alpha = t.K0_alpha;
  const double x0 = x_, y0 = y_, px0 = px_, py0 = py_;
  const Quot<FAST> over_g(gam), over_g2(NARROW ? 1.0 : gam * gam);
  const double dd = NARROW ? 0.0 : t.ku * t.K0 * t.K0 / (4.0 * gam * gam) * t.ue;
  const double bbg = t.bb / gam, fx = bbg * t.xCoef + t.cc, fy = bbg * t.yCoef - t.cc;
  double kx = 0, ky = 0, kpx = 0, kpy = 0, sx = 0, sy = 0, spx = 0, spy = 0;
#pragma unroll 1
  for (int m = 1; m < 5; ++m) {
    const double c = m == 1 ? 0.0 : (m == 4 ? 1.0 : 0.5);
    const double x = x0 + dz * kx * c;
    const double y = y0 + dz * ky * c;
    const double px = px0 + dz * kpx * c;
    const double py = py0 + dz * kpy * c;
    if (NARROW) {
      kx = over_g(px);
      ky = over_g(py);
      kpx = 0.0 - fx * x;
      kpy = 0.0 - fy * y;
    } else {
      kx = over_g(px) - over_g2(aa * (K0_alpha * x + y));
      ky = over_g(py) + over_g2(aa * (K0_alpha * x - y));
      kpx = K0_alpha * (px - py) * dd - fx * x;
      kpy = K0_alpha * (px + py) * dd - fy * y;
    }
    if (m == 1) {
      sx = kx; sy = ky; spx = kpx; spy = kpy;
    } else if (m < 4) {
      sx = sx + 2 * kx; sy = sy + 2 * ky; spx = spx + 2 * kpx; spy = spy + 2 * kpy;
    } else {
      sx = sx + kx; sy = sy + ky; spx = spx + kpx; spy = spy + kpy;
    }
  }
  const double w = dz / 6.0;
  x_ = x0 + w * sx;
  y_ = y0 + w * sy;
  px_ = px0 + w * spx;
  py_ = py0 + w * spy;
}
// The same with plain divisions, for operands outside the window.
__device__ __noinline__ void transverse_any(const TransCoef* t, double* v, double gam) {
  transverse_steps<false, false>(*t, v[0], v[1], v[2], v[3], gam);
}
__device__ __forceinline__ void transverse_one(const TransCoef& t, double& x, double& y, double& px, double& py,
                                               double gam) {
  auto ok = [](double v) { return v == 0.0 || within(v, 400); };
  if (t.fast && ok(x) && ok(y) && ok(px) && ok(py) && within(gam, 100)) {
    if (t.aa == 0.0 && t.ue == 0.0) transverse_steps<true, true>(t, x, y, px, py, gam);
    else transverse_steps<true, false>(t, x, y, px, py, gam);
  } else {
    double v[4] = {x, y, px, py};
    transverse_any(&t, v, gam);
    x = v[0]; y = v[1]; px = v[2]; py = v[3];
  }
}

// Where a particle sits: cell and weights of the transverse grid, radial bin
// and weight (the same expressions in the push and the deposit).
struct Place {
  int ii, jj, ir;
  double wx1, wy1, wr1, r2;
};
__device__ __forceinline__ Place place_of(const DevGeom& G, double x, double y) {
  Place P;
  const double gx = (x - G.minX) / G.dx, gy = (y - G.minY) / G.dy;
  P.ii = (int)gx;
  P.jj = (int)gy;
  P.wx1 = gx - P.ii;
  P.wy1 = gy - P.jj;
  P.r2 = x * x + y * y;
  const double r = sqrt(P.r2);
  P.ir = r / G.dr + 0.5;
  P.wr1 = (r * r / (G.dr * G.dr) - P.ir * P.ir) / (2.0 * P.ir);
  return P;
}

// Bilinear field gather of particlePush.cpp:306-321 (shared with the drift).
template <int HM>
__device__ __forceinline__ double gather_sumU2(const ParticleLaunch& a, int s, const Place& P, cd* Ux, cd* Uy) {
  const DevGeom& G = a.G;
  const int nx = G.nx;
  const double wx[2] = {1.0 - P.wx1, P.wx1}, wy[2] = {1.0 - P.wy1, P.wy1};
#pragma unroll
  for (int h = 0; h < HM; ++h) {
    if (h >= G.H) break;
    const double2* px_ = a.U + field_plane(G.S, h, 0, s, a.ring_base) * G.N;
    const double2* py_ = a.U + field_plane(G.S, h, 1, s, a.ring_base) * G.N;
    cd ux = C(0, 0), uy = C(0, 0);
#pragma unroll
    for (int ii = 0; ii < 2; ++ii)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int id = (P.jj + jj) * nx + (P.ii + ii);
        const double2 vx = __ldg(px_ + id), vy = __ldg(py_ + id);
        ux = cadd(ux, cscale(cscale(C(vx.x, vx.y), wx[ii]), wy[jj]));
        uy = cadd(uy, cscale(cscale(C(vy.x, vy.y), wx[ii]), wy[jj]));
      }
    Ux[h] = ux;
    Uy[h] = uy;
  }
  double sumU2 = 0.0;
#pragma unroll
  for (int h = 0; h < HM; ++h) {
    if (h >= G.H) break;
    const int H = G.harmony[h];
    sumU2 += (cnorm(Ux[h]) + cnorm(Uy[h])) / (2.0 * H * H);
  }
  return sumU2;
}

// Odd-harmonic / even-harmonic coupling factors fx, fy of the push
// (particlePush.cpp:336-360).
template <bool EVEN>
__device__ __forceinline__ void push_f(const ParticleLaunch& a, int H, double xi, double xi2, double K0_alpha,
                                       cd expP, cd expM, cd* fx, cd* fy) {
  const DevGeom& G = a.G;
  double w[2];
  int idx = (1.0 * H * xi) / G.dBessel;
  w[1] = (H * xi / G.dBessel) - idx;
  w[0] = 1.0 - w[1];
  if (!EVEN || H % 2 == 1) {
    const double sign = ((H - 1) / 2 % 2 == 0) ? 1.0 : -1.0;
    int order = (H - 1) / 2;
    const double J1 = BJ(G, idx, order, a.err) * w[0] + BJ(G, idx + 1, order, a.err) * w[1];
    order = (H + 1) / 2;
    const double J2 = BJ(G, idx, order, a.err) * w[0] + BJ(G, idx + 1, order, a.err) * w[1];
    *fx = C(sign * (K0_alpha * J1 - J2), 0.0);
    *fy = C(sign * (K0_alpha * J1 + J2), 0.0);
  } else {
    const double sign = (H / 2 % 2 == 0) ? 1.0 : -1.0;
    idx = (H * xi) / G.dBessel;
    w[1] = (H * xi / G.dBessel) - idx;
    w[0] = 1.0 - w[1];
    int order = (H - 2) / 2;
    const double J1 = BJ(G, idx, order, a.err) * w[0] + BJ(G, idx + 1, order, a.err) * w[1];
    order = H / 2;
    const double J2 = BJ(G, idx, order, a.err) * w[0] + BJ(G, idx + 1, order, a.err) * w[1];
    order = (H + 2) / 2;
    const double J3 = BJ(G, idx, order, a.err) * w[0] + BJ(G, idx + 1, order, a.err) * w[1];
    const double sx = sign * xi2 * H * 0.5;
    *fx = cscale(cadd(cscale(expP, K0_alpha * J1 - J2), cscale(expM, K0_alpha * J2 - J3)), sx);
    *fy = cscale(cadd(cscale(expP, K0_alpha * J1 + J2), cscale(expM, K0_alpha * J2 + J3)), sx);
  }
}

// xi2 and the polarisation phase B of particlePush.cpp:272-279 and
// solveField.cpp:259-266 (identical expressions in both).
__device__ __noinline__ void pol_terms(double K0, double ue, double K0_alpha, double Phi, double px, double py,
                                       double* xi2, cd* expP) {
  *xi2 = sqrt(2.0) * K0 / (1.0 + K0 * K0 * 0.5 * (1.0 + ue * ue)) *
         sqrt((1 + K0_alpha) * (px * px + ue * ue * py * py) + (1 - K0_alpha) * (px * px * ue * ue + py * py));
  const double B = fm::atan(2.0 * K0_alpha * ue * (px - py) /
                            ((1.0 + K0_alpha) * (px + ue * ue * py) + (1 - K0_alpha) * (px * ue * ue + py)));
  const double ph = B - Phi * 0.5;
  if (ph - ph == 0.0) *expP = cexpi(ph);
  else *expP = C(ph - ph, ph - ph);  // nan in, nan out
}

// particlePush.cpp:261-378 for one particle; outside the push grid theta and
// gamma stay untouched.
template <int HM, int LM, bool EVEN>
__device__ __forceinline__ void push_one(const ParticleLaunch& a, int s, double wakeE, const Place& P, double px,
                                         double py, double& th_, double& ga_) {
  const DevGeom& G = a.G;
  const PushCoef& c = a.pc;
  const int nx = G.nx, ny = G.ny, nr = G.nr, L = G.L, F = G.F;
  const double dz = c.dz, ku = c.ku, ks = c.ks, K0 = c.K0, ue = c.ue, K0_alpha = c.K0_alpha;
  if (!(P.ii >= 0 && P.ii < nx - 1 && P.jj >= 0 && P.jj < ny - 1)) return;
  const int sliceI = s + 1;
  const double pr2 = px * px + py * py;
  const double th0 = th_, gam0 = ga_;
  const double K2 = 1.0 + pr2 + (1.0 + ue * ue) * K0 * K0 * 0.5 * (1.0 + ku * ku * 0.5 * P.r2);
  const double xi = ks / ku * K0 * K0 / (8.0 * gam0 * gam0) * (1.0 - ue * ue);
  double xi2 = 0.0;
  cd expP = C(1.0, 0.0);
  if (EVEN) pol_terms(K0, ue, K0_alpha, c.Phi, px, py, &xi2, &expP);
  const cd expM = cconj(expP);
  const double wr[2] = {1.0 - P.wr1, P.wr1};
  cd Em[LM];
  const double2* Ez = a.Ez + (size_t)sliceI * nr * F;
  const size_t ezs = (size_t)(G.S + 2) * nr * F;
#pragma unroll
  for (int ll = 0; ll < LM; ++ll) Em[ll] = C(0, 0);
  if (P.ir > 0 && P.ir < nr) {
#pragma unroll
    for (int ll = 0; ll < LM; ++ll)
      if (ll < L)
        for (int f = 0; f < F; ++f)
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            const double2 v = Ez[ll * ezs + nr * f + P.ir + jj];
            Em[ll] = cadd(Em[ll], cscale(C(v.x, v.y), wr[jj]));
          }
  } else if (P.ir == 0) {
#pragma unroll
    for (int ll = 0; ll < LM; ++ll)
      if (ll < L)
        for (int f = 0; f < F; ++f)
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            const double2 v = Ez[ll * ezs + nr * f + P.ir + jj];
            Em[ll] = cadd(Em[ll], C(v.x, v.y));
          }
  } else {
    // The reference reuses the previous particle's Em here (carry-over across
    // particles); that sequential dependence is not reproduced: flag it.
    set_flag(a.err, ERR_RADIAL);
  }
  // the coupled field of every harmonic, the same at every RK4 stage
  cd D[HM];
  double sumU2;
  {
    cd Ux[HM], Uy[HM];
    sumU2 = gather_sumU2<HM>(a, s, P, Ux, Uy);
#pragma unroll
    for (int h = 0; h < HM; ++h) {
      if (h >= G.H) break;
      cd fx, fy;
      push_f<EVEN>(a, G.harmony[h], xi, xi2, K0_alpha, expP, expM, &fx, &fy);
      D[h] = csub(cmul(cmul(c.etaX, fx), Ux[h]), cmul(cmul(c.etaY, fy), Uy[h]));
    }
  }
  const double sq = sqrt(ue * ue + 1.0), K2U = K2 + sumU2;
  double kth = 0.0, kg = 0.0, sth = 0.0, sg = 0.0;
#pragma unroll 1
  for (int m = 1; m < 5; ++m) {
    const double cf = m == 1 ? 0.0 : (m == 4 ? 1.0 : 0.5);
    const double th = th0 + dz * kth * cf;
    const double gam = gam0 + dz * kg * cf;
    double sumTh = 0.0, sumG = 0.0, sumEz = 0.0;
#pragma unroll 1
    for (int ll = 0; ll < LM; ++ll) {
      if (ll >= L) break;
      const cd e = cexpi((ll + 1.0) * th);
      sumEz += 2.0 * (Em[ll].re * e.re - Em[ll].im * e.im);
    }
#pragma unroll 1
    for (int h = 0; h < HM; ++h) {
      if (h >= G.H) break;
      const int H = G.harmony[h];
      const cd e = cexpi((1.0 * H) * (th + c.Phi * 0.5));
      const cd t = cmul(e, D[h]);
      const double im = 0.0 * t.re - 1.0 * t.im;
      sumTh += H == 1 ? im : im / (1.0 * H);
      sumG += t.re / (2.0 * gam);
    }
    kth = ku - ks / (2.0 * gam * gam) * (K2U + K0 * sq * sumTh);
    kg = ks * K0 * sq * sumG + c.e_mc2 * sumEz;
    if (m == 1) { sth = kth; sg = kg; }
    else if (m < 4) { sth = sth + 2.0 * kth; sg = sg + 2.0 * kg; }
    else { sth = sth + kth; sg = sg + kg; }
  }
  const double tmpTh = dz / 6.0 * sth;
  if (tmpTh > c.dPhi || tmpTh < -c.dPhi) set_flag(a.err, ERR_THETA_OVERFLOW);
  th_ = th0 + tmpTh;
  const double tmpGam = dz / 6.0 * sg - dz * wakeE;
  ga_ = gam0 + tmpGam;
}

// particlePush.cpp:150-184 for one particle.
template <int HM>
__device__ __forceinline__ void drift_one(const ParticleLaunch& a, int s, double wakeE, const Place& P, double px,
                                          double py, double& th_) {
  const DevGeom& G = a.G;
  const PushCoef& c = a.pc;
  const double pr2 = px * px + py * py;
  const double K2 = 1.0 + pr2;
  if (!(P.ii >= 0 && P.ii < G.nx - 1 && P.jj >= 0 && P.jj < G.ny - 1)) return;
  cd Ux[HM], Uy[HM];
  const double sumU2 = gather_sumU2<HM>(a, s, P, Ux, Uy);
  const double tmp = c.ku - c.ks / (2.0 * c.gamR * c.gamR) * (K2 + sumU2);
  double th = th_;
  th += tmp * c.dz;
  th -= c.dz * wakeE;
  th_ = th;
}

// rearrangeParticles.cpp:301-320 for one particle.
__device__ __forceinline__ void wrap_one(double dTh, double& theta_, int* err) {
  double delTh = 0.0;
  const double theta = theta_;
  int intTh = 0;
  if (theta >= dTh) {
    intTh = theta / dTh;
    delTh = dTh * intTh;
  } else if (theta < 0) {
    intTh = theta / dTh - 1.0;
    delTh = dTh * intTh;
  }
  theta_ = theta - delTh;
  if (theta_ > dTh || theta_ < 0) set_flag(err, ERR_OUT_OF_RANGE);
}

// solveField.cpp:252-301 and 331-357: per-particle deposit records.  e1:
// e^{-i theta}, which the lowest space-charge mode uses.
template <bool EVEN>
__device__ __forceinline__ void prep_one(const ParticleLaunch& a, int64_t n, double macro, const Place& P, double x,
                                         double y, double px, double py, double theta, double gam, cd e1) {
  const DevGeom& G = a.G;
  const PrepCoef& c = a.prep;
  const DevDeposit& D = a.dep;
  const int nx = G.nx, ny = G.ny, nr = G.nr, L = G.L, F = G.F;
  const size_t tot = (size_t)a.P.total;
  double xi2 = 0.0;
  cd expP = C(1.0, 0.0);
  if (EVEN) pol_terms(c.K0, c.ue, c.K0_alpha, c.Phi, px, py, &xi2, &expP);
  const cd expM = cconj(expP);
  D.wx1[n] = P.wx1;
  D.wy1[n] = P.wy1;
  const bool in = P.ii >= 0 && P.ii < nx && P.jj >= 0 && P.jj < ny;
  D.key[n] = in ? P.jj << 16 | P.ii : -1;
  if (in && (P.ii == nx - 1 || P.jj == ny - 1)) atomicAdd(a.err + ERR_EDGE_DEPOSIT, 1);
  if (in) {
#pragma unroll 1
    for (int h = 0; h < G.H; ++h) {
      const int H = G.harmony[h];
      const double dbH = (double)H;
      if (EVEN && H % 2 == 0) {
        double w[2];
        const double sign = (H / 2 % 2 == 0) ? 1.0 : -1.0;
        const int ib = (dbH * c.xi) / G.dBessel;
        w[1] = (dbH * c.xi / G.dBessel) - ib;
        w[0] = 1.0 - w[1];
        int order = (H - 2) / 2;
        const double J1 = BJ(G, ib, order, a.err) * w[0] + BJ(G, ib + 1, order, a.err) * w[1];
        order = H / 2;
        const double J2 = BJ(G, ib, order, a.err) * w[0] + BJ(G, ib + 1, order, a.err) * w[1];
        order = (H + 2) / 2;
        const double J3 = BJ(G, ib, order, a.err) * w[0] + BJ(G, ib + 1, order, a.err) * w[1];
        const double sx = sign * xi2 * dbH * 0.5;
        const cd fx = cscale(cadd(cscale(expM, J1 - c.K0_alpha * J2), cscale(expP, J2 - c.K0_alpha * J3)), sx);
        const cd fy = cscale(cadd(cscale(expM, J1 + c.K0_alpha * J2), cscale(expP, J2 + c.K0_alpha * J3)), sx);
        D.fx[(size_t)h * tot + n] = make_double2(fx.re, fx.im);
        D.fy[(size_t)h * tot + n] = make_double2(fy.re, fy.im);
      }
      const cd e = cexpi((-1.0 * dbH) * (theta + c.Phi * 0.5));
      const cd mc = cdivr(cscale(e, dbH * macro * c.coef_U), gam);
      D.coef[(size_t)h * tot + n] = make_double2(mc.re, mc.im);
    }
  }
  // Ez source (solveField.cpp:331-357): every particle, no grid test.
  const double phi = (F > 1) ? ((x == 0.0) ? 0.0 : fm::atan2(y, x)) : 0.0;
  D.wr1[n] = P.wr1;
  int rk = -1;
  if (P.ir >= 0 && P.ir < nr) {
    rk = P.ir;
    if (rk > 0 && rk == nr - 1 && F > 1) set_flag(a.err, ERR_RADIAL);
#pragma unroll 1
    for (int l = 0; l < L; ++l)
#pragma unroll 1
      for (int f = 0; f < (rk > 0 ? F : 1); ++f) {
        // (l + 1) theta + f phi; the azimuthal term does not enter bin 0
        cd e = e1;
        if (l > 0 || f > 0) e = cexpi(-1.0 * (f > 0 ? (l + 1) * theta + f * phi : (l + 1) * theta));
        const cd ic = C(0.0 * c.coef_Ez * (l + 1.0), 1.0 * c.coef_Ez * (l + 1.0));
        cd cc = cscale(cmul(ic, e), macro);
        if (rk > 0) cc = cdivr(cc, 1.0 * rk);
        D.ez[(size_t)(l * F + f) * tot + n] = make_double2(cc.re, cc.im);
      }
  }
  D.rkey[n] = rk;
}

// e^{i phase} of a phase that nothing has wrapped: the reduction of fm::sincos
// loses accuracy from 2^20 pi/2 on.  A call of its own, so that the usual phases
// do not carry its code.
__device__ __noinline__ void far_phase(double phase, double* s, double* c) { sincos(phase, s, c); }

// Deterministic block sum of `v` (fixed shuffle tree, then warps in order).
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
  return t;
}

// One thread per particle; HM, LM: the most harmonics and space-charge modes
// the instance takes (its register arrays), EVEN: an even harmonic is among them.  The RK4
// stages and the harmonics are loops, so that the whole body stays near the
// size of the instruction caches: unrolled (150 KB of instructions, each run
// once per particle) the kernel waited for instructions.
// Measured at 1024 x 8192 particles (every operation of a step in one launch):
// 2.30 ms with unrolled stages, a division per quotient and the couplings
// inside the stages, 1.08 ms so; the particles' state and deposit records,
// 1.2 GB, would take 0.19 ms, the remaining FP64 operations about 0.6 ms.
template <int HM, int LM, bool EVEN>
__global__ void __launch_bounds__(256, HM == 1 ? 4 : 3) k_particles(const __grid_constant__ ParticleLaunch a) {
  __shared__ double part[8][256];
  __shared__ TransCoef tc[2];
  if (threadIdx.x < 2) tc[threadIdx.x] = threadIdx.x ? a.t1 : a.t0;
  __syncthreads();
  const DevGeom& G = a.G;
  const int4 tile = a.P.tiles[blockIdx.x];
  const int sp = tile.x, s = tile.y;
  const int64_t n = (int64_t)tile.z + threadIdx.x;
  const bool active = n < (int64_t)tile.w;
  const unsigned ops = a.ops;
  const int sliceI = s + 1;
  double wakeE = 0.0;
  if (G.wakeOn) wakeE = G.wakeE[sliceI - 1 + G.minI] / (K_MC2 * 1.0e6);
  const double macro = a.P.weight[(size_t)sp * G.S + s];
  double x = 0, y = 0, px = 0, py = 0, th = 0, ga = 1;
  cd e1 = C(1.0, 0.0);  // e^{-i theta}
  if (active) {
    x = a.P.x[n]; y = a.P.y[n]; px = a.P.px[n]; py = a.P.py[n]; th = a.P.th[n]; ga = a.P.ga[n];
#pragma unroll 1
    for (int p = 0; p < 2; ++p)
      if (ops & (p ? OP_T1 : OP_T0)) transverse_one(tc[p], x, y, px, py, ga);
    Place P{};
    if (ops & (OP_PUSH | OP_DRIFT | OP_PREP)) P = place_of(G, x, y);
    if (ops & OP_PUSH) push_one<HM, LM, EVEN>(a, s, wakeE, P, px, py, th, ga);
    else if (ops & OP_DRIFT) drift_one<HM>(a, s, wakeE, P, px, py, th);
    if (ops & OP_PHASE) th += a.theta_shift;
    if (ops & OP_WRAP) wrap_one(G.numSlice * 2 * M_PI, th, a.err);
    if (ops & (OP_T0 | OP_T1)) {
      a.P.x[n] = x; a.P.y[n] = y; a.P.px[n] = px; a.P.py[n] = py;
    }
    if (ops & (OP_PUSH | OP_DRIFT | OP_PHASE | OP_WRAP)) a.P.th[n] = th;
    if (ops & OP_PUSH) a.P.ga[n] = ga;
    if (!(x - x == 0.0) || !(y - y == 0.0) || !(th - th == 0.0) || !(ga - ga == 0.0)) set_flag(a.err, ERR_NAN);
    if (ops & (OP_PREP | OP_DIAG)) e1 = cexpi(-1.0 * th);
    if (ops & OP_PREP) prep_one<EVEN>(a, n, macro, P, x, y, px, py, th, ga, e1);
  }
  if (ops & OP_DIAG) {
    // twiss.cpp:146-166 and saveFile.cpp:126-137 partial sums of this tile,
    // eight quantities at a time: warp w adds the w-th of them
    double* out = a.diag + (size_t)blockIdx.x * a.diag_stride;
    const int t = threadIdx.x, w = t >> 5, l = t & 31, nq = 7 + 2 * G.H + 1;
    const double on = active ? 1.0 : 0.0, mw = active ? macro : 0.0;
    const double invGam = 1.0 / ga;
    const double xP = px * invGam, yP = py * invGam;
    const double v[7] = {x * x * on, y * y * on, xP * xP * on, yP * yP * on, x * xP * on, y * yP * on, on};
#pragma unroll
    for (int k = 0; k < 7; ++k) part[k][t] = v[k];
    part[7][t] = mw;
    for (int q0 = 0;; q0 += 8) {
      __syncthreads();
      double r = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) r += part[w][l + 32 * k];
      for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
      // the first round holds the twiss sums and the weight, the later ones the bunching sums
      const int q = q0 == 0 ? (w < 7 ? w : nq - 1) : q0 - 1 + w;
      if (l == 0 && (q0 == 0 || q < nq - 1)) out[q] = r;
      if (q0 + 8 >= nq) break;
      __syncthreads();
#pragma unroll 1
      for (int k = 0; k < 8; k += 2) {
        const int h = (q0 + k) >> 1;
        if (h >= G.H) break;
        const int H = G.harmony[h];
        const double a = -1.0 * H * th;
        cd e;
        if (fabs(a) < 0x1p20) e = H == 1 ? e1 : cexpi(a);
        else far_phase(a, &e.im, &e.re);
        part[k][t] = e.re * mw;
        part[k + 1][t] = -e.im * mw;
      }
    }
  }
}

// Level 1: block b sums tiles [b*per, (b+1)*per) of every quantity in a
// fixed order: 7 twiss sums per species, then the 2H+1 bFactor sums.
// The sums of nq quantities over rows [r0, r1) by a CTA of 256 threads, each as
// block_sum forms it over its rows (a thread's rows in order, warp trees, the
// warps in order), eight quantities at a time with their loads in flight
// together and one barrier for all: at one slice a step's reductions took
// 0.0189 ms with two barriers and a load's latency per quantity and a launch of
// their own for the planes, 0.0127 with this.
// value(row, q, &v) adds row's share of quantity q.  Thread q < nq returns its total.
constexpr int kMaxSums = 7 * FELIS_MAX_SPECIES + 2 * FELIS_MAX_HARMONY + 1;
template <class F>
__device__ __forceinline__ double row_sums(int nq, int r0, int r1, F value) {
  static_assert(kMaxSums <= 256, "a thread per quantity");
  __shared__ double part[8][kMaxSums];
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  for (int q0 = 0; q0 < nq; q0 += 8) {
    double v[8] = {};
    for (int r = r0 + threadIdx.x; r < r1; r += 256)
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (q0 + u < nq) value(r, q0 + u, v[u]);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (q0 + u >= nq) break;
      for (int o = 16; o > 0; o >>= 1) v[u] += __shfl_down_sync(0xffffffffu, v[u], o);
      if (ln == 0) part[w][q0 + u] = v[u];
    }
  }
  __syncthreads();
  double t = 0.0;
  if ((int)threadIdx.x < nq)
    for (int k = 0; k < 8; ++k) t += part[k][threadIdx.x];
  return t;
}

// Blocks [0, l1): the beam sums of `per` tiles each; blocks from l1 on: the sum
// of a plane's energies over the slices (launch_sum_planes, in the same launch).
__global__ void __launch_bounds__(256) k_diag_level1(const double* part, int ntiles, int stride, int nspecies,
                                                     int H, const int4* tiles, int per, int l1, double* out,
                                                     const double* planes, int S, int last, double* out_planes) {
  if ((int)blockIdx.x >= l1) {
    const int hp = blockIdx.x - l1;
    const double t = row_sums(1, 0, last, [&](int s, int, double& v) { v += planes[(size_t)hp * S + s]; });
    if (threadIdx.x == 0) out_planes[hp] = t;
    return;
  }
  const int t0 = blockIdx.x * per, t1 = min(ntiles, t0 + per), nb = 7 * nspecies, nq = nb + 2 * H + 1;
  const double r = row_sums(nq, t0, t1, [&](int t, int q, double& v) {
    if (q >= nb) v += part[(size_t)t * stride + 7 + (q - nb)];
    else if (tiles[t].x == q / 7) v += part[(size_t)t * stride + q % 7];
  });
  if ((int)threadIdx.x < nq) out[(size_t)blockIdx.x * nq + threadIdx.x] = r;
}

__global__ void __launch_bounds__(256) k_diag_level2(const double* l1, int nblocks, int nspecies, int H,
                                                     double* twiss, double* bf) {
  const int nq = 7 * nspecies + 2 * H + 1, tid = threadIdx.x;
  __shared__ double tot[kMaxSums];
  const double r = row_sums(nq, 0, nblocks, [&](int b, int q, double& v) { v += l1[(size_t)b * nq + q]; });
  if (tid < nq) tot[tid] = r;
  __syncthreads();
  // species by plane, a warp apart; the bunching factors by the last warps
  for (int k = tid >> 5; k < 2 * nspecies && (tid & 31) == 0; k += 4) {
    if (tid >= 128) break;
    const double* acc = tot + 7 * (k >> 1);
    double* o = twiss + 6 * (k >> 1) + 3 * (k & 1);
    const int y = k & 1;
    o[0] = o[1] = o[2] = 0.0;
    const double cnt = acc[6];
    if (cnt > 0.0) {
      const double a2 = acc[y] / cnt, ap = acc[2 + y] / cnt, ac = acc[4 + y] / cnt;
      const double e = sqrt(a2 * ap - ac * ac);
      o[0] = e; o[1] = a2 / e; o[2] = -ac / e;
    }
  }
  if (tid >= 128 && tid - 128 < 2 * H) bf[tid - 128] = tot[7 * nspecies + tid - 128] / tot[7 * nspecies + 2 * H];
}

}  // namespace

namespace {
template <int HM>
void launch_hm(const ParticleLaunch& a, bool even, cudaStream_t st) {
  if (even) k_particles<HM, 4, true><<<a.P.ntiles, 256, 0, st>>>(a);
  else if (a.G.L > 1) k_particles<HM, 4, false><<<a.P.ntiles, 256, 0, st>>>(a);
  else k_particles<HM, 1, false><<<a.P.ntiles, 256, 0, st>>>(a);
}
}  // namespace

void launch_particles(const ParticleLaunch& a, cudaStream_t st) {
  if (a.P.ntiles <= 0) return;
  bool even = false;
  for (int h = 0; h < a.G.H; ++h) even |= a.G.harmony[h] % 2 == 0;
  if (a.G.H <= 1) launch_hm<1>(a, even, st);
  else if (a.G.H <= 2) launch_hm<2>(a, even, st);
  else if (a.G.H <= 4) launch_hm<4>(a, even, st);
  else launch_hm<FELIS_MAX_HARMONY>(a, even, st);
}

void launch_diag_finalize(const double* partials, int ntiles, int stride, int nspecies, int H, const int4* tiles,
                          double* l1, int l1_blocks, double* out_twiss, double* out_bf, const double* planes, int S,
                          int skip_last, double* out_planes, cudaStream_t st) {
  const int per = (ntiles + l1_blocks - 1) / l1_blocks;
  k_diag_level1<<<l1_blocks + (planes ? 2 * H : 0), 256, 0, st>>>(partials, ntiles, stride, nspecies, H, tiles, per,
                                                                  l1_blocks, l1, planes, S, S - skip_last, out_planes);
  k_diag_level2<<<1, 256, 0, st>>>(l1, l1_blocks, nspecies, H, out_twiss, out_bf);
}

}  // namespace felis
