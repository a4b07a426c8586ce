// ADI and energy kernels of the FELIS slice loop, FP64 plain path
// (--fmad=false); the source deposit is in k_deposit.cu.
#include "field.cuh"
#include "bulk.cuh"

namespace felis {

namespace {

__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)((blockDim.x + 31) >> 5); ++k) t += red[k];
  return t;
}

// ---- ADI -------------------------------------------------------------------
// Each sweep (solveField.cpp:112-181) is a right-hand side from the
// neighbouring lines, its division by alphaP (betaP), a forward and a backward
// recurrence along every line.  Only the recurrences are serial: the
// right-hand sides and their divisions are made first, in place, by all
// threads (two to four per line), so that a line's thread walks a chain of six
// dependent operations forward and four backward per point (48 and 32 cycles
// at 8 per FP64 operation) and waits for nobody.  The reference's operand
// order is kept throughout.

// Coefficients of one direction, by line index.
struct AdiDir {
  const cd *p, *a, *q, *cc, *z;  // alphaP, alpha, Q, CC, H + alphaP + alpha (the other sweep's right-hand side)
  const double *pinv, *qinv, *ccinv;
};

// Right-hand side and its division, in place, of points [k0, k1) of a line
// across the sweep: v_k = -p_k u_{k+1} + z_k u_k - a_k u_{k-1} (+ source),
// with the coefficients D of the line's own direction.  um and ue are u_{k0-1}
// and u_{k1} from before the call.  `div`: divide by dp (its 1 / |dp|^2 given);
// the sweep's last line keeps the plain right-hand side.  src: source values
// by k, stride ss, for k in [s0, s1].
__device__ __forceinline__ void adi_rhs(double2* v, int st, int k0, int k1, const AdiDir& D, double2 um, double2 ue,
                                        bool div, cd dp, double dinv, const double2* __restrict__ src, int ss, int s0,
                                        int s1) {
  if (k0 >= k1) return;
  double2 u0 = v[k0 * st];
  double2 sn = make_double2(0.0, 0.0);
  if (k0 >= s0 && k0 <= s1) sn = src[k0 * ss];
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const double2 up = k + 1 < k1 ? v[(k + 1) * st] : ue;
    const double2 sv = sn;
    const bool in = k >= s0 && k <= s1;
    if (k + 1 < k1 && k + 1 >= s0 && k + 1 <= s1) sn = src[(k + 1) * ss];  // one point ahead
    cd t = cmul(cneg(D.p[k]), C(up.x, up.y));
    t = cadd(t, cmul(D.z[k], C(u0.x, u0.y)));
    t = csub(t, cmul(D.a[k], C(um.x, um.y)));
    if (in) t = cadd(t, C(sv.x, sv.y));
    if (div) t = cdiv_inv(t, dp, dinv);
    v[k * st] = make_double2(t.re, t.im);
    um = u0;
    u0 = up;
  }
}

// The recurrences of one line of n points (interior 1 .. n - 2) whose divided
// right-hand side is in v; out(k, value) receives the solution from the last
// point to the first.  Coefficients and values are read one point ahead of
// the chain.
template <class Out>
__device__ __forceinline__ void adi_solve(double2* v, int st, int n, const AdiDir& D, Out out) {
  double2 x = v[st];
  cd d = C(x.x, x.y);
  x = v[2 * st];
  cd an = D.a[2], qn = D.q[2];
  double in = D.qinv[2];
#pragma unroll 1
  for (int k = 2; k < n - 2; ++k) {
    const cd t = C(x.x, x.y), ak = an, qk = qn;
    const double ik = in;
    x = v[(k + 1) * st];
    an = D.a[k + 1]; qn = D.q[k + 1]; in = D.qinv[k + 1];
    d = csub(t, cdiv_inv(cmul(ak, d), qk, ik));
    v[k * st] = make_double2(d.re, d.im);
  }
  d = csub(C(x.x, x.y), cdiv_inv(d, D.cc[n - 3], D.ccinv[n - 3]));
  cd u = cdiv_inv(d, D.cc[n - 2], D.ccinv[n - 2]);
  x = v[(n - 3) * st];
  cd cn = D.cc[n - 3];
  in = D.ccinv[n - 3];
  out(n - 2, u);
#pragma unroll 1
  for (int k = n - 3; k > 0; --k) {
    const cd t = C(x.x, x.y), ck = cn;
    const double ik = in;
    x = v[(k - 1) * st];
    cn = D.cc[k - 1]; in = D.ccinv[k - 1];
    u = cdiv_inv(csub(t, u), ck, ik);
    out(k, u);
  }
}

__device__ __forceinline__ double norm2(double2 v) { return v.x * v.x + v.y * v.y; }
// nonzero when a component is (its sign apart)
__device__ __forceinline__ int bits_of(double2 v) {
  return ((__double2hiint(v.x) | __double2hiint(v.y)) & 0x7fffffff) | __double2loint(v.x) | __double2loint(v.y);
}

// The recurrence coefficients of a harmonic in shared memory at `at` (they are
// read at every step), 88 bytes per line.
__device__ __forceinline__ void adi_tables(void* at, const AdiTab& T, int nx, int ny, AdiDir& X, AdiDir& Y) {
  cd* tx = reinterpret_cast<cd*>(at);                    // p, a, q, cc [nx each]
  cd* ty = tx + 4 * nx;                                  // p, a, q, cc [ny each]
  double* dx = reinterpret_cast<double*>(ty + 4 * ny);   // pinv, qinv, ccinv [nx each]
  double* dy = dx + 3 * nx;                              // [ny each]
  for (int k = threadIdx.x; k < nx; k += blockDim.x) {
    tx[k] = T.ax_p[k]; tx[nx + k] = T.ax_a[k]; tx[2 * nx + k] = T.ax_q[k]; tx[3 * nx + k] = T.ax_cc[k];
    dx[k] = T.ax_pinv[k]; dx[nx + k] = T.ax_qinv[k]; dx[2 * nx + k] = T.ax_ccinv[k];
  }
  for (int k = threadIdx.x; k < ny; k += blockDim.x) {
    ty[k] = T.ay_p[k]; ty[ny + k] = T.ay_a[k]; ty[2 * ny + k] = T.ay_q[k]; ty[3 * ny + k] = T.ay_cc[k];
    dy[k] = T.ay_pinv[k]; dy[ny + k] = T.ay_qinv[k]; dy[2 * ny + k] = T.ay_ccinv[k];
  }
  X = AdiDir{tx, tx + nx, tx + 2 * nx, tx + 3 * nx, T.ry_0, dx, dx + nx, dx + 2 * nx};
  Y = AdiDir{ty, ty + ny, ty + 2 * ny, ty + 3 * ny, T.rx_0, dy, dy + ny, dy + 2 * ny};
}

// Brings the source of columns [i0, i1] and rows [j0, j1] into this SM's L1,
// so that the right-hand sides, which read it point by point, do not wait for
// L2 at each (half of their time before).
__device__ __forceinline__ void adi_warm(const double2* Sc, int nx, int i0, int i1, int j0, int j1) {
  const int w = i1 - i0 + 1, n = w > 0 && j1 >= j0 ? w * (j1 - j0 + 1) : 0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    [[maybe_unused]] double x, y;
    asm volatile("ld.global.ca.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "l"(Sc + (size_t)(j0 + k / w) * nx + i0 + k % w));
  }
}

// Start of part q of Q of the points [1, n - 2].
__device__ __forceinline__ int adi_part(int n, int q, int Q) { return 1 + (n - 2) * q / Q; }

// One CTA per plane, the plane in shared memory; four threads per line for the
// right-hand sides, one for the recurrences.  The results of the y sweep go
// straight to global memory (edge cells keep their values: the ADI never
// writes them).
//
// Measured at 2048 planes of 102 x 102 (one CTA per SM: 186 KB of shared
// memory): 1.21 ms with the right-hand sides inside the serial sweeps and a
// barrier per column, 0.58 ms so (one plane alone 0.086 and 0.041 ms); the
// planes alone, 682 MB, would take 0.104 ms.  Of a plane's 84,000 cycles the
// chains take 32,000, the right-hand sides 32,000 (10,000 at the FP64 rate),
// staging 16,000; none of them overlaps another, since only one plane fits an
// SM.
constexpr int kAdiParts = 4, kAdiThreads = 512;  // parts per line (fewer on grids wider than 130), threads, at most
__global__ void __launch_bounds__(768, 1) k_adi(AdiLaunch a) {  // 80 registers: three planes of 64 x 64 to an SM
  extern __shared__ double2 Apl[];  // ny rows of nxp complex, then the recurrence tables
  __shared__ double red[16];
  const DevGeom& G = a.G;
  const int S = G.S, nx = G.nx, ny = G.ny, N = G.N, P = a.nxp;
  const int s = blockIdx.x % S;
  const int hp = blockIdx.x / S;  // h*2 + pol
  const int h = hp >> 1, pol = hp & 1;
  const int tid = threadIdx.x;
  const size_t at = field_plane(S, h, pol, s, a.ring_base);
  double2* U = a.U + at * N;
  const double2* Sc = a.Sc + ((size_t)hp * S + s) * N;
  // A plane that holds nothing and receives nothing stays as it is: the sweeps
  // of zeros give zeros.  A planar undulator drives one polarisation, so half
  // of its planes are of this kind (1024 slices of 102 x 102: 0.57 -> 0.30 ms).
  if (a.skip && !a.use_source[pol] && a.lit[at] == 0) {
    if (tid == 0 && a.energy) a.energy[(size_t)hp * S + s] = 0.0;
    return;
  }
  // ---- stage the plane: one bulk copy per row (rows of complex FP64 start on
  // 16-byte boundaries in global and in shared memory) ----
  __shared__ __align__(8) unsigned long long pbar;
  if (tid == 0) bar_init_tx(smem_u32(&pbar), (unsigned)((size_t)N * sizeof(double2)));
  __syncthreads();
  for (int r = tid; r < ny; r += blockDim.x)
    bulk_g2s(Apl + (size_t)r * P, U + (size_t)r * nx, (unsigned)(nx * sizeof(double2)), smem_u32(&pbar));
  AdiDir X, Y;
  adi_tables(Apl + (size_t)ny * P, a.tab[h], nx, ny, X, Y);
  const int4 bx = a.use_source[pol] ? a.box[s] : make_int4(1, 0, 1, 0);
  adi_warm(Sc, nx, bx.x, bx.y, bx.z, bx.w);
  if (!bar_wait0(smem_u32(&pbar), kBulkWaitTries)) {
    set_flag(a.err, ERR_TIMEOUT);
    bar_wait0(smem_u32(&pbar), kBulkWaitTries);  // once more for the copies in flight
  }
  __syncthreads();
  // thread (line l, part q of Q): 32 neighbouring lines to a warp
  const int NL = max(nx, ny) - 2, q = tid / NL, l = tid - q * NL + 1, Q = min(kAdiParts, (int)blockDim.x / NL);
  const double2 zero = make_double2(0.0, 0.0);
  double e = 0.0;
  int any = 0;  // bits of every value of the plane after the solve
  // ---- x sweep, right-hand side: column l, rows of part q ----
  {
    const bool on = q < Q && l <= nx - 2;
    const int k0 = adi_part(ny, q, Q), k1 = adi_part(ny, q + 1, Q);
    double2 um = zero, ue = zero;
    if (on) { um = Apl[(k0 - 1) * P + l]; ue = Apl[k1 * P + l]; }
    __syncthreads();
    if (on) {
      const bool in = l >= bx.x && l <= bx.y;
      adi_rhs(Apl + l, P, k0, k1, Y, um, ue, l < nx - 2, X.p[l], X.pinv[l], Sc + l, nx, in ? bx.z : 1, in ? bx.w : 0);
    }
  }
  __syncthreads();
  // ---- x sweep: row l; the other threads sum |U|^2 of the edge cells ----
  if (q == 0 && l <= ny - 2) {
    double2* row = Apl + (size_t)l * P;
    adi_solve(row, 1, nx, X, [&](int k, cd u) { row[k] = make_double2(u.re, u.im); });
  } else if (q > 0) {
    const int nt = (int)blockDim.x - NL, ne = 2 * nx + 2 * (ny - 2);
    for (int k = tid - NL; k < ne; k += nt) {
      const int m = k - 2 * nx;
      const double2 v = k < nx ? Apl[k] : m < 0 ? Apl[(size_t)(ny - 1) * P + (k - nx)]
                                                : Apl[(size_t)((m >> 1) + 1) * P + ((m & 1) ? nx - 1 : 0)];
      e += norm2(v);
      any |= bits_of(v);
    }
  }
  __syncthreads();
  // ---- y sweep, right-hand side: row l, columns of part q; the x sweep's
  // result is zero beyond the interior ----
  {
    const bool on = q < Q && l <= ny - 2;
    const int k0 = adi_part(nx, q, Q), k1 = adi_part(nx, q + 1, Q);
    double2* row = Apl + (size_t)l * P;
    double2 um = zero, ue = zero;
    if (on) {
      if (k0 > 1) um = row[k0 - 1];
      if (k1 < nx - 1) ue = row[k1];
    }
    __syncthreads();
    if (on) {
      const bool in = l >= bx.z && l <= bx.w;
      adi_rhs(row, 1, k0, k1, X, um, ue, l < ny - 2, Y.p[l], Y.pinv[l], Sc + (size_t)l * nx, 1, in ? bx.x : 1,
              in ? bx.y : 0);
    }
  }
  __syncthreads();
  // ---- y sweep: column l ----
  if (q == 0 && l <= nx - 2)
    adi_solve(Apl + l, P, ny, Y, [&](int k, cd u) {
      const double2 v = make_double2(u.re, u.im);
      U[(size_t)k * nx + l] = v;
      e += cnorm(u);
      any |= bits_of(v);
    });
  any = __syncthreads_or(any);
  if (tid == 0) a.lit[at] = any;
  if (a.energy) {
    const double t = block_sum(e, red);
    if (tid == 0) a.energy[(size_t)hp * S + s] = t;
  }
}

// ADI of planes too large for shared memory: the same steps on tiles, the x
// sweep on bands of kAdiTile rows (with the rows either side), its result in a
// scratch plane per CTA that stays in L2, the y sweep on bands of kAdiTile
// columns; one CTA per plane, planes taken in a grid-stride loop.  (Before, the
// sweeps ran on the planes in global memory, a thread per row, uncoalesced:
// 0.44 ms for 296 planes of 152 x 152, 0.26 ms so.)
constexpr int kAdiTile = 32, kAdiBigParts = 2;
__global__ void __launch_bounds__(640, 1) k_adi_big(AdiLaunch a) {
  extern __shared__ double2 tile[];
  __shared__ double red[16];
  const DevGeom& G = a.G;
  const int S = G.S, nx = G.nx, ny = G.ny, N = G.N;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const double2 zero = make_double2(0.0, 0.0);
  const int NL = max(nx, ny) - 2, q = tid / NL, l = tid - q * NL + 1;
  double2* Xp = a.scratch + (size_t)blockIdx.x * N;
  for (int plane = blockIdx.x; plane < S * G.H * 2; plane += gridDim.x) {
    const int s = plane % S, hp = plane / S, h = hp >> 1, pol = hp & 1;
    const size_t at = field_plane(S, h, pol, s, a.ring_base);
    double2* U = a.U + at * N;
    const double2* Sc = a.Sc + ((size_t)hp * S + s) * N;
    if (a.skip && !a.use_source[pol] && a.lit[at] == 0) {  // as in k_adi
      if (tid == 0 && a.energy) a.energy[(size_t)hp * S + s] = 0.0;
      continue;
    }
    const int4 bx = a.use_source[pol] ? a.box[s] : make_int4(1, 0, 1, 0);
    double e = 0.0;
    int any = 0;  // bits of every value of the plane after the solve
    AdiDir X, Y;
    adi_tables(tile + a.tile_cells, a.tab[h], nx, ny, X, Y);
    // ---- x sweep, rows [j0, j1) ----
    const int P = nx | 1;
    for (int j0 = 1; j0 <= ny - 2; j0 += kAdiTile) {
      const int j1 = min(ny - 1, j0 + kAdiTile), m = j1 - j0;
      double2* B = tile - (ptrdiff_t)(j0 - 1) * P;  // B[j * P + i]: row j, column i
      adi_warm(Sc, nx, bx.x, bx.y, max(bx.z, j0), min(bx.w, j1 - 1));
      for (int r = warp; r < m + 2; r += nw)
        for (int i = lane; i < nx; i += 32) copy16(tile + (size_t)r * P + i, U + (size_t)(j0 - 1 + r) * nx + i);
      copies_done();
      __syncthreads();
      {
        const bool on = q < kAdiBigParts && l <= nx - 2;
        const int k0 = j0 + m * q / kAdiBigParts, k1 = j0 + m * (q + 1) / kAdiBigParts;
        double2 um = zero, ue = zero;
        if (on) { um = B[(k0 - 1) * P + l]; ue = B[k1 * P + l]; }
        __syncthreads();
        if (on) {
          const bool in = l >= bx.x && l <= bx.y;
          adi_rhs(B + l, P, k0, k1, Y, um, ue, l < nx - 2, X.p[l], X.pinv[l], Sc + l, nx, in ? bx.z : 1, in ? bx.w : 0);
        }
      }
      __syncthreads();
      if (tid < m) {
        double2* row = tile + (size_t)(tid + 1) * P;
        adi_solve(row, 1, nx, X, [&](int k, cd u) { row[k] = make_double2(u.re, u.im); });
      }
      __syncthreads();
      for (int r = warp; r < m; r += nw)
        for (int i = lane + 1; i < nx - 1; i += 32) Xp[(size_t)(j0 + r) * nx + i] = tile[(size_t)(r + 1) * P + i];
      __syncthreads();
    }
    // ---- y sweep, columns [i0, i1); the x sweep's result is zero beyond the interior ----
    constexpr int W = kAdiTile + 3;  // odd row pitch of the column tile
    for (int i0 = 1; i0 <= nx - 2; i0 += kAdiTile) {
      const int i1 = min(nx - 1, i0 + kAdiTile), m = i1 - i0;
      double2* B = tile - (i0 - 1);  // B[j * W + i]
      adi_warm(Sc, nx, max(bx.x, i0), min(bx.y, i1 - 1), bx.z, bx.w);
      for (int j = 1 + warp; j <= ny - 2; j += nw)
        for (int c = lane; c < m + 2; c += 32) {
          const int i = i0 - 1 + c;
          if (i == 0 || i == nx - 1) tile[(size_t)j * W + c] = zero;
          else copy16(tile + (size_t)j * W + c, Xp + (size_t)j * nx + i);
        }
      copies_done();
      __syncthreads();
      {
        const bool on = q < kAdiBigParts && l <= ny - 2;
        const int k0 = i0 + m * q / kAdiBigParts, k1 = i0 + m * (q + 1) / kAdiBigParts;
        double2* row = B + (size_t)l * W;
        double2 um = zero, ue = zero;
        if (on) { um = row[k0 - 1]; ue = row[k1]; }
        __syncthreads();
        if (on) {
          const bool in = l >= bx.z && l <= bx.w;
          adi_rhs(row, 1, k0, k1, X, um, ue, l < ny - 2, Y.p[l], Y.pinv[l], Sc + (size_t)l * nx, 1, in ? bx.x : 1,
                  in ? bx.y : 0);
        }
      }
      __syncthreads();
      if (tid < m) {
        const int i = i0 + tid;
        adi_solve(B + i, W, ny, Y, [&](int k, cd u) {
          const double2 v = make_double2(u.re, u.im);
          U[(size_t)k * nx + i] = v;
          e += cnorm(u);
          any |= bits_of(v);
        });
      }
      __syncthreads();
    }
    // ---- |U|^2 of the edge cells, which keep their values ----
    const int ne = 2 * nx + 2 * (ny - 2);
    for (int k = tid; k < ne; k += nt) {
      const int m = k - 2 * nx;
      const double2 v = k < nx ? U[k] : m < 0 ? U[(size_t)(ny - 1) * nx + (k - nx)]
                                              : U[(size_t)((m >> 1) + 1) * nx + ((m & 1) ? nx - 1 : 0)];
      e += norm2(v);
      any |= bits_of(v);
    }
    any = __syncthreads_or(any);
    if (tid == 0) a.lit[at] = any;
    if (a.energy) {
      const double t = block_sum(e, red);
      if (tid == 0) a.energy[(size_t)hp * S + s] = t;
    }
    __syncthreads();
  }
}

// Plane sums of |U|^2 (updateTotalEnergy.cpp:25-33), one block per plane.
__global__ void __launch_bounds__(256) k_energy(DevGeom G, const double2* U, int ring_base, double* out) {
  __shared__ double red[8];
  const int S = G.S;
  const int s = blockIdx.x % S, hp = blockIdx.x / S;
  const double2* P = U + field_plane(S, hp >> 1, hp & 1, s, ring_base) * G.N;
  double e = 0.0;
  for (int k = threadIdx.x; k < G.N; k += blockDim.x) {
    const double2 v = P[k];
    e += v.x * v.x + v.y * v.y;
  }
  const double t = block_sum(e, red);
  if (threadIdx.x == 0) out[(size_t)hp * S + s] = t;
}

// out[hp] = sum over planes s of planes[hp][s], s < S - skip_last (fixed order).
__global__ void __launch_bounds__(256) k_sum_planes(const double* planes, int S, int skip_last, double* out) {
  __shared__ double red[8];
  const int hp = blockIdx.x;
  double e = 0.0;
  for (int s = threadIdx.x; s < S - skip_last; s += blockDim.x) e += planes[(size_t)hp * S + s];
  const double t = block_sum(e, red);
  if (threadIdx.x == 0) out[hp] = t;
}

}  // namespace

cudaError_t adi_set_smem(size_t bytes) { return allow_smem((const void*)k_adi, bytes); }

size_t adi_smem_bytes(int nx, int ny, int nxp) {
  return (size_t)ny * nxp * sizeof(double2) + (size_t)4 * (nx + ny) * sizeof(double2) + (size_t)3 * (nx + ny) * sizeof(double);
}

// `parts` threads per line, whole warps
static int adi_threads(const DevGeom& G, int parts) {
  const int m = (G.nx > G.ny ? G.nx : G.ny) - 2;
  const int p = parts < kAdiThreads / m ? parts : kAdiThreads / m;
  return ((p * m + 31) / 32) * 32;
}

void launch_adi(const AdiLaunch& a, cudaStream_t st) {
  k_adi<<<a.G.S * a.G.H * 2, adi_threads(a.G, kAdiParts), adi_smem_bytes(a.G.nx, a.G.ny, a.nxp), st>>>(a);
}

// cells of a row band or a column band
static size_t adi_tile_cells(int nx, int ny) {
  const size_t rows = (size_t)(kAdiTile + 2) * (nx | 1), cols = (size_t)ny * (kAdiTile + 3);
  return rows > cols ? rows : cols;
}

size_t adi_big_smem_bytes(int nx, int ny) { return adi_tile_cells(nx, ny) * sizeof(double2) + (size_t)88 * (nx + ny); }

cudaError_t adi_big_set_smem(size_t bytes) { return allow_smem((const void*)k_adi_big, bytes); }

void launch_adi_big(AdiLaunch a, int grid, cudaStream_t st) {
  a.tile_cells = (int)adi_tile_cells(a.G.nx, a.G.ny);
  k_adi_big<<<grid, adi_threads(a.G, kAdiBigParts), adi_big_smem_bytes(a.G.nx, a.G.ny), st>>>(a);
}

void launch_energy(const DevGeom& G, const double2* U, int ring_base, double* out_planes, cudaStream_t st) {
  k_energy<<<G.S * G.H * 2, 256, 0, st>>>(G, U, ring_base, out_planes);
}

void launch_sum_planes(const double* planes, int H, int S, int skip_last, double* out, cudaStream_t st) {
  k_sum_planes<<<H * 2, 256, 0, st>>>(planes, S, skip_last, out);
}

}  // namespace felis
