// The single-matrix solvers' iterations in one resident kernel (resident.cu).
#pragma once
#include "ofea_internal.cuh"
#include "solver_common.cuh"

namespace ofea {

// Launch shape of the resident solver for one matrix: G CTAs of kResThreads
// threads, CTA b owning the slices [b * spc, (b + 1) * spc); in a matrix
// phase S warps share a slice (S64: FP64 slots, S16: pairs of BF16 slots).
// cluster: the CTAs are one thread-block cluster of that size (small
// matrices); 0: a cooperative grid.
struct ResidentPlan {
    int G = 0, spc = 0, S64 = 1, S16 = 1, cluster = 0;
};

constexpr int kResThreads = 1024;
constexpr int kResMaxM = 1536;  // coarse unknowns the preconditioned form holds in shared memory

// Whether the resident solver takes this matrix (and its plan).  With mixed,
// the coarse level must be set up; elements: a launch per phase would form the
// outer products from the elements.
bool resident_plan(const ofea_ctx *c, bool mixed, bool elements, ResidentPlan &p);

// Enqueues `iters` iterations from fl->itA on (fewer when the solve stops) on
// the context's stream.  MIXED with first != 0 starts with the preconditioner
// applied to b32 / x32 (z_0); with modes its restriction takes K Z
// (solver_modes).  Partials of the kernels before it: G each.
void resident_iterations(ofea_ctx *c, const ResidentPlan &p, bool mixed, bool modes, const Parts &P, Flags *fl, double *d_u,
                         float wsm, double tol2, int iters, int first);

}  // namespace ofea
