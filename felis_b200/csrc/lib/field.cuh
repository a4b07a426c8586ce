// Field kernels of the FELIS slice loop: declarations.
#pragma once

#include "common.cuh"

namespace felis {

// Coefficient tables of the ADI sweeps for one harmonic (solveField.cpp:
// 110-181), built on the host with the same complex formulas as the CPU
// restatement so the recurrences below reproduce it bit for bit.
struct AdiTab {
  // x-sweep right-hand side (index j): H + betaP + beta (betaP and beta below)
  const cd* rx_0;
  // x-sweep recurrence (index i): alphaP and 1/|alphaP|^2, alpha,
  // Q = alphaP*CC[i-1] and 1/|Q|^2, CC and 1/|CC|^2
  const cd *ax_p, *ax_a, *ax_q, *ax_cc;
  const double *ax_pinv, *ax_qinv, *ax_ccinv;
  // y-sweep right-hand side (index i): H + alphaP + alpha
  const cd* ry_0;
  // y-sweep recurrence (index j)
  const cd *ay_p, *ay_a, *ay_q, *ay_cc;
  const double *ay_pinv, *ay_qinv, *ay_ccinv;
};

struct AdiLaunch {
  DevGeom G;
  double2* U;          // ring of S planes per (h, pol)
  int ring_base;
  const double2* Sc;   // [H][2][S][N]
  const int4* box;     // per slice: {i0, i1, j0, j1} of written source cells
  int use_source[2];   // currentFlag of solveField and a source in this polarisation
  int* lit;            // [H][2][S] ring: 0 if the plane is known to be zero everywhere
  int skip;            // planes may be skipped by it
  const AdiTab* tab;   // [H] (device array of structs)
  double* energy;      // [H][2][S] plane sums of |U|^2 after the solve (may be null)
  int nxp;             // padded row length of the shared-memory plane
  double2* scratch;    // k_adi_big: one plane per CTA
  int tile_cells;      // k_adi_big: cells of the shared-memory tile
  int* err;            // [ERR_SLOTS] (ERR_TIMEOUT: a bounded staging wait ran out)
};

struct DepositLaunch {
  DevGeom G;
  DevDeposit dep;
  const int64_t* soff;  // [nspecies][S+1]
  int64_t total;
  double2* Sc;          // [H][2][S][N]
  int4* box;            // [S]
  double2* Ez;          // [L][(S+2)*F*nr]
  double2 fconst[FELIS_MAX_HARMONY][2];  // odd-harmonic fx, fy (per call constants)
  cd etaX, etaY;
  double A;             // Ez Thomas coefficient (solveField.cpp:320)
  int chunk2, chunkr;   // particles per chunk of the 2-D and the radial sums (DepositPlan)
  const double2* radial;  // [L*F][nr] radial elimination for A (launch_radial_elimination)
};

// Chunk sizes and shared memory of the deposit; false when the radial grid is
// too large for it.
struct DepositPlan {
  int chunk2 = 0, chunkr = 0;
  size_t smem = 0;
};
bool deposit_plan(int H, int neven, int L, int F, int nr, size_t dev_smem, DepositPlan* p);
void launch_deposit(const DepositLaunch& a, size_t smem, cudaStream_t st);
// Multiplier and pivot of every point and mode of the radial Ez solve with
// the coefficient A (DepositLaunch::A): L * F <= 16 modes.
void launch_radial_elimination(double A, int L, int F, int nr, const double* logtab, double2* out, cudaStream_t st);
// The shared memory that launches may take (allow_smem).
cudaError_t deposit_set_smem(size_t bytes);
cudaError_t adi_set_smem(size_t bytes);
void launch_adi(const AdiLaunch& a, cudaStream_t st);
size_t adi_smem_bytes(int nx, int ny, int nxp);
// Planes larger than shared memory: `grid` CTAs, each with one scratch plane.
void launch_adi_big(AdiLaunch a, int grid, cudaStream_t st);
size_t adi_big_smem_bytes(int nx, int ny);
cudaError_t adi_big_set_smem(size_t bytes);
void launch_energy(const DevGeom& G, const double2* U, int ring_base, double* out_planes, cudaStream_t st);
void launch_sum_planes(const double* planes, int H, int S, int skip_last, double* out, cudaStream_t st);

}  // namespace felis
