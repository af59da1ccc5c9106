// Host-visible structures and launchers of the D3Q7 solute kernels.
#pragma once

#include "lbm_internal.h"

namespace lbm {

struct St7Args {
  void* g;                // [6][npad] or [19][npad], stepped in place (kernels_common.cuh)
  int phase;              // Phase of the state
  const int32_t* table;   // D3Q19 pull table [18][npad]; D3Q7: rows 0..5 used
  const int32_t* rows;    // D3Q19: row form of the table (row_table.cuh), or null
  int ahead;              // nodes ahead that a block prefetches into L2, 0 = none
  int chained;            // launched as a programmatic dependent of the step before it
  const void* u;          // [3][npad] advecting velocity
  const void* c_given;    // [npad] C for the first step after init, else null
  void* c_out;            // optional [npad]: C of this step's macro
  int n, npad;
  double tau_s;
  double c2, c4;          // lat_c^2 and lat_c^4 of the D3Q19 equilibrium (1 on the default lattice)
  int nq;                 // 7 (D3Q7, g as [6][npad]) or 19 (D3Q19, g as [19][npad])
};

cudaError_t st7_launch_step(bool f64, const St7Args& a, cudaStream_t st);
cudaError_t st7_launch_step_f64(const St7Args& a, cudaStream_t st);  // st7_faithful.cu, -fmad=false
cudaError_t st19_launch_step_f64(const St7Args& a, cudaStream_t st);  // st7_faithful.cu, -fmad=false
cudaError_t st7_launch_conc(bool f64, const St7Args& a, double* out, cudaStream_t st);
cudaError_t st7_launch_init(bool f64, const St7Args& a, cudaStream_t st);
// the imported (or initial) state is a kPull state
cudaError_t st7_launch_export(bool f64, const St7Args& a, const int32_t* ref_of, double* out, cudaStream_t st);
cudaError_t st7_launch_import(bool f64, const St7Args& a, const int32_t* ref_of, const double* in, cudaStream_t st);

}  // namespace lbm
