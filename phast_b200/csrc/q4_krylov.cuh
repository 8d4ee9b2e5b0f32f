// Whole Krylov solves on a structured Q4 grid in one cooperative launch
// (q4_krylov.cu): the bound-projected PCG of the damage solve, and the plain
// and Jacobi CG of its linear (adjoint) system and of the quasi-static
// mechanics.
#pragma once
#include "engine.cuh"

namespace phastb {

// The AT2 damage system of q4_damage_apply_launch (rs = 2), rows with `mask` zero.
struct Q4DamageSys {
  phastb_q4_grid g;
  const double* Hq;
  double rsh;
  const double* rsh_e;
  double gcl0;
  const double* gcl0_e;
  const uint8_t* mask;
};

// The degraded elastic stiffness (linear splits), or the consistent tangent at the displacement u (splits
// whose stress is not linear in the strain), rows with `mask` (per component) zero.
struct Q4MechSys {
  phastb_q4_grid g;
  phastb_q4_material m;
  const double* d;
  const double* u;  // the tangent's displacement; null: the stiffness
  const uint8_t* mask;
};

// ppcg_solve (engine.cuh) on the damage system in one launch: the right-hand side and the inverse
// diagonal stay in registers, w.r to w.Ap carry the exchange.  PHASTB_UNSUPPORTED: the grid does not
// fit the SMs' shared memory, the workspace is not 16-byte aligned (the exchange words are), or the
// device has no cooperative launch (or PHASTB_PERSISTENT_PCG=0); nothing was launched.
int q4_ppcg_persistent(const Q4DamageSys& sys, const PpcgWs& w, const double* d_prev, const double* d_init,
                       const uint8_t* fixed, const double* vals, double tol, int max_iter, int check_every, double* d,
                       int* info, cudaStream_t s);

// PcgLoop bodies (engine.cuh): continue from the state pcg_start_kernel left in w.  `tagged`: 16 bytes of
// scratch per unknown, 16-byte aligned.
int q4_pcg_persistent(const Q4DamageSys& sys, const PcgWs<double>& w, const double* inv_diag, void* tagged, double* x,
                      int maxiter, int check_every, PcgMode mode, cudaStream_t s);
int q4_pcg_persistent(const Q4MechSys& sys, const PcgWs<double>& w, void* tagged, double* x, int maxiter,
                      int check_every, PcgMode mode, cudaStream_t s);

// PHASTB_PERSISTENT_PCG=0 runs every Krylov solve as separate launches per iteration.
bool persistent_pcg_enabled();

}  // namespace phastb
