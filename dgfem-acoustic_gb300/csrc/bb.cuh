// Host side of the Bernstein-basis kernels (stage_bb.cuh): basis tables,
// conversions between the reference layout (nodal values) and the tiles of
// Bernstein coefficients, source injection and element means.
#pragma once
#include "ctx.h"

namespace dgc {
// Whether the Bernstein-basis kernels take this context's mesh (straight-sided
// triangles or tetrahedra).
inline bool bb_mesh(const dg_ctx* c) { return c->dim >= 2 && c->ncurved == 0; }
// Index of coefficient n of element e's first variable in a state array, and
// the distance of the next variable's.
int64_t bb_slot(const dg_ctx* c, int64_t e, int n);
int64_t bb_var_stride(const dg_ctx* c);
// Basis tables (c->bb_V, bb_Vinv and their device copies).
int bb_setup_basis(dg_ctx* c);
// reference layout [4][E*np] (c->d_ref or another device array) -> tiles, elements e0 to e1 - 1 (up to E: every
// lane of the padding cleared); and back
cudaError_t bb_from_ref(dg_ctx* c, const double* ref, void* out, int64_t e0, int64_t e1);
cudaError_t bb_to_ref(dg_ctx* c, const void* in, double* ref);
// Hard overwrite of the pressure at source nodes, for elements' coefficients.
cudaError_t bb_inject(dg_ctx* c);
// Element means into out: AoS [E][5] (p, rho, v) or SoA (p [E], rho [E], v [E][3]).
cudaError_t bb_cell_means(dg_ctx* c, double* out, bool soa);
// Many RK4 steps in one launch (persist.cu). Whether the context is in FP64 and
// its tiles fit on the GPU at once; whether it is the faster way then; device lists and buffers of a run (false where memory for them is
// short); n_steps steps on c->stream with residuals and observers to the
// context's result buffers (launched: steps whose launch succeeded); release.
bool persist_fits(const dg_ctx* c);
bool persist_pays(const dg_ctx* c);
bool persist_ready(dg_ctx* c);
cudaError_t persist_run(dg_ctx* c, int64_t n_steps, double dt, int64_t* launched);
void persist_free(dg_ctx* c);
dgk::StageArgs<double> stage_args_f64(dg_ctx* c, int stage, const double* y_in, double* y_out, double dt);
}  // namespace dgc
