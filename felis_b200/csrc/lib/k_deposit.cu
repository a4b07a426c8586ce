// Ordered source deposit of the FP64 plain path (--fmad=false).
//
// The reference adds each particle's bilinear current into ScUx/ScUy one
// particle after the other (solveField.cpp:233-312), so every cell is a
// sequential sum in particle order, and the radial space-charge bins likewise
// (solveField.cpp:315-357).  The kernel reproduces those sums bit for bit
// without sorting: a slice's particles are taken in chunks, every target (cell
// or bin) gets its contributors' terms in particle order, one after the other
// in shared memory (its chain), and one thread then adds the chain up.
//
// Places in the chains.  Each of sixteen warps owns a consecutive part of the
// chunk and walks it 32 particles at a time.  A target's contributors among
// them sit in two neighbouring rows and two neighbouring columns; ballots over
// the bits of the row pair and of the column pair give every lane the other
// lanes of its pairs.  A popcount below the lane's own bit is the particle's
// rank in the group, and a counter per target and warp carries the rank on
// from group to group.  A prefix sum over targets and warps turns the ranks
// into places.  No sort and no merge.
//
// The block's targets are cut into bands of rows (2-D) or of bins (r) that
// fit the counters; the band of a usual beam (33 x 33 cells) is the whole box.
// Every band walks the slice's particles: a 1 GeV beam on 152 x 152 points (a box
// of about 145 x 145, 13 bands) takes 0.64 ms for a slice of 8192 particles and
// 0.79 for 64 of them (1.14 and 1.26 with the sort).
//
// Measured (B200, 8192 particles per slice, 102 x 102): a single slice 0.415 ms
// with a stable radix sort per chunk and a four-way merge per cell, 0.076 ms
// so; 1024 slices 2.00 ms and 0.63 ms; 96 slices of 2048 particles with
// harmonics 1 to 3, 0.27 and 0.11 ms.  Bound by instruction issue and
// shared-memory latency at two CTAs per SM (64 registers, 106 KB); the
// particles' records, 64 bytes each, would take 0.08 ms from memory.  Shorter
// chunks (512) cost more in prefix sums than their occupancy gives (1.27 ms),
// eight warps of four groups the same time at more registers (0.82 ms).
//
// The two sums of a slice are independent: CTA (s, 0) makes the 2-D source,
// CTA (s, 1) the radial one with its Thomas solve, so that the long serial
// chains of the radial bins (a bin a few sigma wide holds a fifth of the
// slice) run beside other CTAs' work.  The elimination of the radial matrix,
// which no particle enters, is a table made when the lattice changes it.
#include <algorithm>

#include "field.cuh"

namespace felis {

namespace {

constexpr int kWarps = 16;
constexpr int kWork = 32 * kWarps;  // threads of a CTA
constexpr int kCells2 = 1280;       // counters per warp, 2-D (cells of a band)
constexpr int kBins = 512;          // counters per warp, radial
constexpr int kGroups = 2;          // groups of 32 particles per warp and chunk, at most

__device__ __forceinline__ cd C_(double2 v) { return C(v.x, v.y); }

// Maps a slice-local deposit index q (species-major) to the global particle index.
__device__ __noinline__ int q_to_n(const int64_t* soff, int S, int nspecies, int s, int q) {
  for (int sp = 0; sp < nspecies; ++sp) {
    const int b = (int)soff[(size_t)sp * (S + 1) + s], e = (int)soff[(size_t)sp * (S + 1) + s + 1];
    if (q < e - b) return b + q;
    q -= e - b;
  }
  return -1;
}

// Shared memory of a 2-D CTA with C particles per chunk: the chains' terms
// (four per particle) and the counters.
__host__ __device__ inline size_t smem2(int C) { return (size_t)4 * C * 16 + (size_t)(kCells2 + 1) * 2 * kWarps; }
// Shared memory of a radial CTA: the chains' terms (two per particle and
// mode), the counters and the bins.
struct LayR {
  size_t cnt, bins, total;
};
__host__ __device__ inline LayR layr(int C, int LF, int nr) {
  LayR L;
  L.cnt = (size_t)2 * C * 16 * LF;
  L.bins = L.cnt + (size_t)(kBins + 1) * 2 * kWarps;
  L.total = L.bins + (size_t)LF * nr * 16;
  return L;
}

__device__ __forceinline__ int bits_of(int v) { return 32 - __clz(v); }
// Lanes of m whose bit i of v is this lane's.
__device__ __forceinline__ void keep(unsigned& m, int v, int i) {
  const bool p = v >> i & 1;
  const unsigned b = __ballot_sync(0xffffffffu, p);
  m &= p ? b : ~b;
}
// Counter of target t and warp w: sixteen to a target, their order turned with
// the target so that one warp's counters of many targets spread over the banks.
__device__ __forceinline__ int slot(int t, int w) { return t * kWarps + (w ^ ((t >> 2 & 7) << 1)); }

// Turns the counts cnt[slot(t, w)] of targets t < n and warps w into places:
// the chain of target t starts after those of all earlier targets, and warp
// w's part of it after those of the warps before.  cnt[slot(t, 0)] is then the
// start of chain t, cnt[slot(n, 0)] the end of the last.
__device__ __forceinline__ void places(uint16_t* cnt, int n, uint32_t* wsum) {
  constexpr int V = kWarps / 8;  // 16-byte words per target
  const int t = threadIdx.x, K = (n + kWork - 1) / kWork;
  const int i0 = min(n, t * K), i1 = min(n, i0 + K);
  uint32_t sum = 0;  // two 16-bit sums; their total stays below 2^16
#pragma unroll 1
  for (int i = i0 * V; i < i1 * V; ++i) {
    const uint4 c = reinterpret_cast<const uint4*>(cnt)[i];
    sum += c.x + c.y + c.z + c.w;
  }
  sum = (sum & 0xffffu) + (sum >> 16);
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if ((t & 31) >= o) incl += v;
  }
  if ((t & 31) == 31) wsum[t >> 5] = incl;
  __syncthreads();
  // the sums of the warps before this one
  const uint32_t ws = (t & 31) < (t >> 5) ? wsum[t & 31] : 0u;
  uint32_t run = incl - sum + __reduce_add_sync(0xffffffffu, ws);
#pragma unroll 1
  for (int i = i0; i < i1; ++i) {
    uint32_t* c = reinterpret_cast<uint32_t*>(cnt + i * kWarps);
    const int x = i >> 2 & 7;
#pragma unroll
    for (int w = 0; w < kWarps / 2; ++w) {
      const uint32_t v = c[w ^ x], lo = v & 0xffffu;
      c[w ^ x] = run | (run + lo) << 16;
      run += lo + (v >> 16);
    }
  }
  if (t == kWork - 1) cnt[slot(n, 0)] = (uint16_t)run;
}

// acc -= or += the chain t[0], t[stride], ... of n terms, in order.  Four terms
// are read while the four before them are added, so the sum is bound by its
// dependent adds (8 cycles each on this chip).
template <bool SUB>
__device__ __forceinline__ void add_chain(const double2* __restrict__ t, int n, int stride, double2& acc) {
  auto read = [&](double2 (&v)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = t[u * stride];
    t += 4 * stride;
  };
  auto add = [&](const double2& v) {
    acc.x = SUB ? acc.x - v.x : acc.x + v.x;
    acc.y = SUB ? acc.y - v.y : acc.y + v.y;
  };
  auto add4 = [&](const double2 (&v)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) add(v[u]);
  };
  double2 v[4], w[4];
  if (n >= 4) {
    read(v);
    for (n -= 4; n >= 8; n -= 8) {
      read(w);
      add4(v);
      read(v);
      add4(w);
    }
    if (n >= 4) {
      n -= 4;
      read(w);
      add4(v);
      add4(w);
    } else {
      add4(v);
    }
  }
  if (n > 0) v[0] = t[0];
  if (n > 1) v[1] = t[stride];
  if (n > 2) v[2] = t[2 * stride];
  if (n > 0) add(v[0]);
  if (n > 1) add(v[1]);
  if (n > 2) add(v[2]);
}

__device__ void deposit_2d(const DepositLaunch& a, unsigned char* dsm, int s) {
  __shared__ int red_i[4][kWarps];
  __shared__ uint32_t wsum[kWarps];
  const DevGeom& G = a.G;
  const int S = G.S, nx = G.nx, ny = G.ny, N = G.N, H = G.H, CH = a.chunk2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  double2* term = reinterpret_cast<double2*>(dsm);
  uint16_t* cnt = reinterpret_cast<uint16_t*>(dsm + (size_t)4 * CH * 16);
  const size_t tot = (size_t)a.total;
  int Pt = 0;  // a handle holds fewer than 2^31 particles
  for (int sp = 0; sp < G.nspecies; ++sp)
    Pt += (int)(a.soff[(size_t)sp * (S + 1) + s + 1] - a.soff[(size_t)sp * (S + 1) + s]);
  const int first = (int)a.soff[s];
  const bool one = G.nspecies == 1;
  auto index = [&](int q) { return one ? first + q : q_to_n(a.soff, S, G.nspecies, s, q); };
  // ---- box of reachable interior cells over the whole slice ----
  int v[4] = {1 << 30, 1 << 30, 1 << 30, 1 << 30};  // min i, -max i, min j, -max j
  for (int q0 = tid; q0 < Pt; q0 += 8 * kWork) {
    int k[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) k[u] = q0 + u * kWork < Pt ? a.dep.key[index(q0 + u * kWork)] : -1;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k[u] >= 0) {
        const int ki = k[u] & 0xffff, kj = k[u] >> 16;
        v[0] = min(v[0], ki); v[1] = min(v[1], -ki);
        v[2] = min(v[2], kj); v[3] = min(v[3], -kj);
      }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = __reduce_min_sync(0xffffffffu, v[k]);
    if (lane == 0) red_i[k][warp] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k)
    for (int w = 0; w < kWarps; ++w) v[k] = min(v[k], red_i[k][w]);
  const bool found = v[0] < (1 << 30);
  int bi0 = max(1, v[0]), bi1 = min(nx - 2, -v[1] + 1), bj0 = max(1, v[2]), bj1 = min(ny - 2, -v[3] + 1);
  if (!found || bi0 > bi1 || bj0 > bj1) { bi0 = bj0 = 1; bi1 = bj1 = 0; }
  if (tid == 0) a.box[s] = make_int4(bi0, bi1, bj0, bj1);
  const int bw = bi1 - bi0 + 1, bh = bj1 - bj0 + 1;
  if (bw <= 0 || bh <= 0) return;
  // bands of th target rows (grids are at most 256 wide, so several rows fit);
  // targets are counted by row and column of the band
  const int th_max = kCells2 / bw, nband = (bh + th_max - 1) / th_max, th = (bh + nband - 1) / nband;
  const int groups = CH / kWork;  // groups of 32 particles per warp and chunk
  // eta is (c, 0) for one polarisation and (0, s) for the other
  // (particlePush.cpp:222-238): the products with their zero parts leave the
  // terms below as they are.  A planar undulator has c = 1 and s = 0: the
  // second polarisation's source is zero.
  const bool xre = a.etaX.im == 0.0 && a.etaY.re == 0.0;
  const double er = xre ? a.etaX.re : a.etaY.re, ei = xre ? a.etaY.im : a.etaX.im;
  int key[kGroups];  // this lane's particles of the coming chunk
  auto load_keys = [&](int c0) {
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      const int q = c0 + (warp * groups + g) * 32 + lane;
      key[g] = g < groups && q < Pt ? a.dep.key[index(q)] : -1;
    }
  };
  load_keys(0);
  for (int j0 = bj0; j0 <= bj1; j0 += th) {
    const int rows = min(th, bj1 - j0 + 1), n = rows * bw, nb = bits_of((max(rows, bw) + 1) >> 1);
    for (int c0 = 0; c0 < Pt; c0 += CH) {
      for (int i = tid; i < (n + 1) * kWarps / 8; i += kWork) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
      __syncthreads();
      // ---- ranks.  Row r and column c of a particle's cell: 0 is the row /
      // column before the band's first target, so its targets are rows r - 1
      // and r and columns c - 1 and c of the band
      int cell[kGroups];  // target index of (r - 1, c - 1); unused corners masked by `ok`
      unsigned rank[kGroups], ok[kGroups];
      unsigned m[kGroups][4];  // lanes with the same r / 2, (r + 1) / 2, c / 2, (c + 1) / 2
      int r[kGroups], c[kGroups];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        r[g] = (key[g] >> 16) - (j0 - 1);
        c[g] = (key[g] & 0xffff) - (bi0 - 1);
        const bool in = key[g] >= 0 && r[g] >= 0 && r[g] <= rows && c[g] >= 0 && c[g] <= bw;
        ok[g] = !in ? 0u : ((r[g] >= 1 && c[g] >= 1) ? 1u : 0u) | ((r[g] >= 1 && c[g] < bw) ? 2u : 0u) |
                               ((r[g] < rows && c[g] >= 1) ? 4u : 0u) | ((r[g] < rows && c[g] < bw) ? 8u : 0u);
        cell[g] = (r[g] - 1) * bw + c[g] - 1;
        m[g][0] = m[g][1] = __ballot_sync(0xffffffffu, in);
        m[g][2] = m[g][3] = 0xffffffffu;
      }
#pragma unroll 1
      for (int i = 0; i < nb; ++i)
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          keep(m[g][0], r[g] >> 1, i);
          keep(m[g][1], (r[g] + 1) >> 1, i);
          keep(m[g][2], c[g] >> 1, i);
          keep(m[g][3], (c[g] + 1) >> 1, i);
        }
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        // rows {r - 1, r} are the pair of r / 2 for an odd r, else that of (r + 1) / 2
        const unsigned R0 = (r[g] & 1) ? m[g][0] : m[g][1], R1 = (r[g] & 1) ? m[g][1] : m[g][0];
        const unsigned C0 = (c[g] & 1) ? m[g][2] : m[g][3], C1 = (c[g] & 1) ? m[g][3] : m[g][2];
        const unsigned w[4] = {R0 & C0, R0 & C1, R1 & C0, R1 & C1};
        rank[g] = 0;
        unsigned nw[4];
#pragma unroll
        for (int cb = 0; cb < 4; ++cb) {
          nw[cb] = 0;
          if (ok[g] >> cb & 1u) {
            const unsigned before = cnt[slot(cell[g] + (cb & 1) + (cb >> 1) * bw, warp)];
            rank[g] |= (before + __popc(w[cb] & lt)) << (8 * cb);
            if ((w[cb] >> lane) == 1u) nw[cb] = before + __popc(w[cb]);  // the last one moves the counter on
          }
        }
        __syncwarp();
#pragma unroll
        for (int cb = 0; cb < 4; ++cb)
          if (nw[cb]) cnt[slot(cell[g] + (cb & 1) + (cb >> 1) * bw, warp)] = (uint16_t)nw[cb];
        __syncwarp();
      }
      __syncthreads();
      places(cnt, n, wsum);
      __syncthreads();
      // place of every term
      unsigned place[kGroups][2];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        unsigned p[4];
#pragma unroll
        for (int cb = 0; cb < 4; ++cb)
          p[cb] = (ok[g] >> cb & 1u) ? cnt[slot(cell[g] + (cb & 1) + (cb >> 1) * bw, warp)] + (rank[g] >> (8 * cb) & 255u) : 0u;
        place[g][0] = p[0] | p[1] << 16;
        place[g][1] = p[2] | p[3] << 16;
      }
      load_keys(c0 + CH < Pt ? c0 + CH : 0);
      // ---- per harmonic and polarisation: the terms, then the sums ----
      for (int h = 0; h < H; ++h) {
        const bool odd = G.harmony[h] % 2 == 1;
        for (int pol = 0; pol < 2; ++pol) {
          const bool real = odd && (pol == 0) == xre;
          const bool none = odd && !real && ei == 0.0;
          if (!none) {
            const double f = a.fconst[h][pol].x;
            const cd eta = pol ? a.etaY : a.etaX;
#pragma unroll
            for (int g = 0; g < kGroups; ++g) {
              if (!ok[g]) continue;
              const int p = index(c0 + (warp * groups + g) * 32 + lane);
              const double wx1 = a.dep.wx1[p], wy1 = a.dep.wy1[p];
              const double2 m = a.dep.coef[(size_t)h * tot + p];
              const double wx0 = 1.0 - wx1, wy0 = 1.0 - wy1;
              cd fe = C(0.0, 0.0);
              if (!odd) fe = C_((pol ? a.dep.fy : a.dep.fx)[(size_t)h * tot + p]);
#pragma unroll
              for (int cb = 0; cb < 4; ++cb) {
                if (!(ok[g] >> cb & 1u)) continue;
                const double wx = (cb & 1) ? wx1 : wx0, wy = (cb >> 1) ? wy1 : wy0;
                double2 t;
                if (odd) {
                  const double A = (real ? er : ei) * wx * wy * f;
                  t = real ? make_double2(A * m.x, A * m.y) : make_double2(-(A * m.y), A * m.x);
                } else {
                  const cd z = cmul(cmul(cscale(cscale(eta, wx), wy), fe), C_(m));
                  t = make_double2(z.re, z.im);
                }
                term[place[g][cb >> 1] >> (16 * (cb & 1)) & 0xffffu] = t;
              }
            }
          }
          __syncthreads();
          double2* Sc = a.Sc + (((size_t)h * 2 + pol) * S + s) * N;
          for (int i = tid; i < n; i += kWork) {
            const int r = i / bw, t = (j0 + r) * nx + bi0 + (i - r * bw);
            const int k0 = cnt[slot(i, 0)], k1 = none ? k0 : cnt[slot(i + 1, 0)];
            if (k0 == k1 && c0 > 0) continue;
            double2 acc = make_double2(0.0, 0.0);
            if (c0 > 0) acc = Sc[t];
            add_chain<true>(term + k0, k1 - k0, 1, acc);
            Sc[t] = acc;
          }
          __syncthreads();
        }
      }
    }
  }
}

// Radial source of the last species and its Thomas solve (solveField.cpp:315-399).
// Bins are indexed from 0 (bin 0) and 2 (bin 1): bin 0 does not reach bin 1, so
// the empty index between them keeps the neighbour rule one for all bins.
__device__ void deposit_radial(const DepositLaunch& a, unsigned char* dsm, int s) {
  __shared__ uint32_t wsum[kWarps];
  const DevGeom& G = a.G;
  const int S = G.S, nr = G.nr, F = G.F, LF = G.L * F, CH = a.chunkr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const LayR Ly = layr(CH, LF, nr);
  double2* term = reinterpret_cast<double2*>(dsm);
  uint16_t* cnt = reinterpret_cast<uint16_t*>(dsm + Ly.cnt);
  double2* bin = reinterpret_cast<double2*>(dsm + Ly.bins);
  const size_t tot = (size_t)a.total;
  const int64_t* so = a.soff + (size_t)(G.nspecies - 1) * (S + 1) + s;
  const int n0 = (int)so[0], Pl = (int)(so[1] - so[0]);
  for (int i = tid; i < LF * nr; i += kWork) bin[i] = make_double2(0.0, 0.0);
  // the outermost bin that holds a particle
  int top = -1;
  for (int q0 = tid; q0 < Pl; q0 += 8 * kWork) {
    int k[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) k[u] = q0 + u * kWork < Pl ? a.dep.rkey[n0 + q0 + u * kWork] : -1;
#pragma unroll
    for (int u = 0; u < 8; ++u) top = max(top, k[u]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) wsum[warp] = (uint32_t)top;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, (int)wsum[lane & (kWarps - 1)]);
  const int Imax = min(nr, top + 3);        // target indices (bins 0 .. nr - 2) end here
  const int per = CH / kWarps;              // particles per warp and chunk
  const int groups = (per + 31) / 32;
  // bands of target indices [I0, I0 + n); sources from I0 - 1
  for (int I0 = 0; I0 < Imax; I0 += kBins) {
    const int n = min(Imax - I0, kBins), nb = bits_of((n + 2) >> 1);
    int rk[kGroups];
    auto load_keys = [&](int c0) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int q = c0 + warp * per + g * 32 + lane;
        rk[g] = g < groups && g * 32 + lane < per && q < Pl ? a.dep.rkey[n0 + q] : -1;
      }
    };
    load_keys(0);
    for (int c0 = 0; c0 < Pl; c0 += CH) {
      for (int i = tid; i < (n + 1) * kWarps / 8; i += kWork) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
      int b[kGroups];  // index of the particle's bin; 0 is the source below the band
      unsigned rank[kGroups], ok[kGroups], m[kGroups][2];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int I = rk[g] > 0 ? rk[g] + 1 : rk[g];
        b[g] = I - I0 + 1;
        const bool in = rk[g] >= 0 && b[g] >= 0 && b[g] <= n;
        // its own bin (the one below the band is a source only), and the next
        // one but for bin 0, whose next index is no bin
        ok[g] = !in ? 0u : (b[g] >= 1 ? 1u : 0u) | (b[g] < n && I != 0 ? 2u : 0u);
        m[g][0] = m[g][1] = __ballot_sync(0xffffffffu, in);
      }
#pragma unroll 1
      for (int i = 0; i < nb; ++i)
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          keep(m[g][0], b[g] >> 1, i);
          keep(m[g][1], (b[g] + 1) >> 1, i);
        }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const unsigned w[2] = {(b[g] & 1) ? m[g][0] : m[g][1], (b[g] & 1) ? m[g][1] : m[g][0]};
        rank[g] = 0;
        unsigned nw[2];
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          nw[cb] = 0;
          if (ok[g] >> cb & 1u) {
            const unsigned before = cnt[slot(b[g] - 1 + cb, warp)];
            rank[g] |= (before + __popc(w[cb] & lt)) << (16 * cb);
            if ((w[cb] >> lane) == 1u) nw[cb] = before + __popc(w[cb]);
          }
        }
        __syncwarp();
#pragma unroll
        for (int cb = 0; cb < 2; ++cb)
          if (nw[cb]) cnt[slot(b[g] - 1 + cb, warp)] = (uint16_t)nw[cb];
        __syncwarp();
      }
      __syncthreads();
      places(cnt, n, wsum);
      __syncthreads();
      // every (particle, bin) term at its place in the bin's chain
      double wr1[kGroups];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        wr1[g] = ok[g] ? a.dep.wr1[n0 + c0 + warp * per + g * 32 + lane] : 0.0;
        const unsigned p0 = (ok[g] & 1u) ? cnt[slot(b[g] - 1, warp)] + (rank[g] & 0xffffu) : 0u;
        const unsigned p1 = (ok[g] & 2u) ? cnt[slot(b[g], warp)] + (rank[g] >> 16) : 0u;
        rank[g] = p0 | p1 << 16;
      }
#pragma unroll 1
      for (int lf = 0; lf < LF; ++lf)
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          const bool zero = I0 + b[g] == 1;  // bin 0: unweighted, f = 0 modes only
          if (!ok[g] || (zero && lf % F > 0)) continue;
          const double2 v = a.dep.ez[(size_t)lf * tot + n0 + c0 + warp * per + g * 32 + lane];
          const double w0 = 1.0 - wr1[g];
          if (ok[g] & 1u) term[(size_t)(rank[g] & 0xffffu) * LF + lf] = zero ? v : make_double2(v.x * w0, v.y * w0);
          if (ok[g] & 2u) term[(size_t)(rank[g] >> 16) * LF + lf] = make_double2(v.x * wr1[g], v.y * wr1[g]);
        }
      load_keys(c0 + CH < Pl ? c0 + CH : 0);
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i < LF * n; i += kWork) {
        const int lf = i / n, t = i - lf * n, It = I0 + t;
        const int k0 = cnt[slot(t, 0)], k1 = cnt[slot(t + 1, 0)];
        // index 1 is no bin; bin 0 holds f = 0 modes only
        if (k0 == k1 || It == 1 || (It == 0 && lf % F > 0)) continue;
        double2& sum = bin[(size_t)lf * nr + (It > 0 ? It - 1 : 0)];
        double2 x = sum;
        add_chain<false>(term + (size_t)k0 * LF + lf, k1 - k0, LF, x);
        sum = x;
      }
      __syncthreads();
    }
  }
  // ---- Thomas solve in r; the back substitution reads the first slice's
  // ghost, which is zero, so the solution is d_j / b_j ----
  double2* wb = term;  // the elimination's (multiplier, pivot), read beside the bins
  const bool near_tab = nr <= 2 * CH;
  if (near_tab)
    for (int i = tid; i < LF * nr; i += kWork) wb[i] = a.radial[i];
  __syncthreads();
  const double2* e0 = near_tab ? wb : a.radial;
  if (tid < LF) {
    double2* d = bin + (size_t)tid * nr;
    const double2* e = e0 + (size_t)tid * nr;
    if (tid % F != 0) d[0] = make_double2(0.0, 0.0);
    double2 p = d[0], dn = d[1];
    double wn = e[1].x;
    // the next point is read before this one is stored
    for (int j = 1; j < nr - 1; ++j) {
      const double2 dj = dn;
      const double ww = wn;
      dn = d[j + 1];
      wn = e[j + 1].x;
      p = make_double2(dj.x - p.x * ww, dj.y - p.y * ww);
      d[j] = p;
    }
  }
  __syncthreads();
  const size_t ezs = (size_t)(S + 2) * nr * F;
  double2* Ez = a.Ez + (size_t)(s + 1) * F * nr;
  for (int i = tid; i < LF * (nr - 1); i += kWork) {
    const int lf = i / (nr - 1), j = i - lf * (nr - 1), l = lf / F, f = lf - l * F;
    const double2 d = bin[(size_t)lf * nr + j];
    const double b = e0[(size_t)lf * nr + j].y;
    Ez[(size_t)l * ezs + (size_t)f * nr + j] = make_double2(d.x / b, d.y / b);
  }
}

// The radial matrix's elimination for the lattice constant A, one thread per
// mode (l, f): multiplier and pivot of every point (solveField.cpp:361-397).
__global__ void k_radial_elimination(double A, int LF, int F, int nr, const double* logtab, double2* out) {
  const int lf = threadIdx.x;
  if (lf >= LF) return;
  const int l = lf / F, f = lf % F;
  double bp = f == 0 ? -(1.0 + (l + 1.0) * (l + 1.0) * A / 8.0) : 1.0, up = f == 0 ? 1.0 : 0.0;
  out[(size_t)lf * nr] = make_double2(0.0, bp);
  for (int j = 1; j < nr; ++j) {
    const bool last = j == nr - 1;
    const double ww = (last ? 0.0 : j - 0.5) / bp;
    double b = last ? 1.0 : -2.0 * j - (l + 1.0) * (l + 1.0) * A * j - f * f * logtab[j];
    b -= ww * up;
    out[(size_t)lf * nr + j] = make_double2(ww, b);
    bp = b;
    up = last ? 0.0 : j + 0.5;
  }
}

__global__ void __launch_bounds__(kWork, 2) k_deposit(const __grid_constant__ DepositLaunch a) {
  extern __shared__ __align__(16) unsigned char dsm[];
  if (blockIdx.y == 0) deposit_2d(a, dsm, blockIdx.x);
  else deposit_radial(a, dsm, blockIdx.x);
}

}  // namespace

bool deposit_plan(int H, int neven, int L, int F, int nr, size_t dev_smem, DepositPlan* p) {
  const int LF = L * F;
  // the radial grids the library accepts: bins, pivots and bin starts of every
  // mode beside 64 particles' records
  const size_t rec = std::max<size_t>((size_t)1024 * (1 + H + 2 * neven), (size_t)2048 * LF);
  if (16960 + rec + (size_t)8 * (nr + 2) + (size_t)24 * LF * nr > dev_smem) return false;
  p->chunk2 = kGroups * kWork;
  p->chunkr = kGroups * kWork;
  // the radial chunk: as large as fits beside the 2-D one's share, at least
  // 64 particles
  while (p->chunkr > 64 && layr(p->chunkr, LF, nr).total > smem2(p->chunk2)) p->chunkr >>= 1;
  p->smem = std::max(smem2(p->chunk2), layr(p->chunkr, LF, nr).total);
  return p->smem <= dev_smem;
}

void launch_deposit(const DepositLaunch& a, size_t smem, cudaStream_t st) {
  k_deposit<<<dim3(a.G.S, 2), kWork, smem, st>>>(a);
}

void launch_radial_elimination(double A, int L, int F, int nr, const double* logtab, double2* out, cudaStream_t st) {
  k_radial_elimination<<<1, 32, 0, st>>>(A, L * F, F, nr, logtab, out);
}

cudaError_t deposit_set_smem(size_t bytes) { return allow_smem((const void*)k_deposit, bytes); }

}  // namespace felis
