// kernels.cuh -- host launchers of the device path (internal).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

struct fpsi_ctx;

namespace fpsi {

// where a residual's norms go: rec[NREC] (device) and, when given, the pinned
// record host[NREC] -- of a run's step *seq (device, counted up) when seq is
// given
struct NormOut {
  double* rec = nullptr;
  double* host = nullptr;
  int32_t* seq = nullptr;
};
// residual chain: boundary states, gradient+limiter, face flux, per-cell
// gather (src, dtau) and, with norms.rec, the norms (else left to the
// launch_assemble that follows)
int launch_residual(fpsi_ctx* x, const NormOut& norms = {});
// the gradient-and-limiter records of the last residual's state, where the
// residual did not write them (!grad_valid: it was inviscid)
int launch_grad_records(fpsi_ctx* x);
// the cells' viscosity and conductivity, for the last residual's state and the
// options in force (the residual of a viscous run leaves them; options may
// have changed since)
int ensure_material(fpsi_ctx* x);
// face Jacobians, diagonal blocks, LU, B and the starting iterate
// (the starting iterate is the block Jacobi start D^-1 B); with norms.rec one
// block finishes the last residual's norms meanwhile
int launch_assemble(fpsi_ctx* x, const NormOut& norms = {});
// block Jacobi start x = D^-1 B on an assembled system
int launch_jacobi_start(fpsi_ctx* x);
// `sweeps` symmetric multi-colour Gauss-Seidel sweeps on the device iterate
int launch_sgs(fpsi_ctx* x, int sweeps);
// out2[0] = ||B||, out2[1] = ||B - A x|| (device), and the pinned host2 too
int launch_linres(fpsi_ctx* x, double* out2, double* host2);
// fills fjp/fjm from the compact face records of the assembled system (a
// no-op when they already hold it)
int ensure_explicit_blocks(fpsi_ctx* x);
// clipped Newton update; per-block minimum alpha into d_amin.  guard
// (device, may be null): the norms of the residual the system came from;
// NaN norms leave the state unchanged
int launch_update(fpsi_ctx* x, const double* guard, const int32_t* flag0 = nullptr,
                  const int32_t* flag1 = nullptr);
// caller-order staging buffer <-> device state (in = staging -> q)
int launch_state(fpsi_ctx* x, bool in);

// rows of w values per cell: device order (map: RCM cell -> row, null RCM
// order; values of 4 or 8 bytes) to or from a caller-order array of doubles
// on the device
int launch_rows_out(fpsi_ctx* x, int w, const int32_t* map, const void* src, int bytes, double* caller);
int launch_rows_in(fpsi_ctx* x, int w, const int32_t* map, const double* caller, void* dst, int bytes);

int launch_batch_flux(int kind, int64_t n, const double* qL, const double* qR, const double* an,
                      const double* area, double pamb, double Rt, double gamma, double us_n,
                      double eta, double* F, cudaStream_t s);
int launch_batch_jac(int64_t n, const double* qL, const double* qR, const double* an,
                     const double* area, double pamb, double Rt, double gamma, double us_n,
                     double eta, int dir, int as_double, void* out, cudaStream_t s);

const char* last_error();

}  // namespace fpsi
