// ffvgpu_kernels.h -- host-side launchers of the FP64 kernels.
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

#include "ffvgpu_layout.h"

namespace ffvgpu {


// Parameters every block kernel needs: neighbour table, cell sizes and the
// outer BCs of the field being staged.
// Kernels that take a block range (exchange, unpack, assembly, BC folding)
// cover blocks [first, first + nb); the solver kernels run with first = 0.
struct KCtx {
  const FaceNbr* nbr;  // [blocks][6]
  const double* dx;    // [blocks]
  BCSet bc;
  int nb;
  int first;
  uint64_t wait_ns;    // limit of every bounded device wait (ffvgpu_pool_set_wait_limit)
  // [blocks][8] uniform records of A (launch_urec), or
  // null: every block streams all its coefficients
  const double* urec;
};

// Where a pass takes its blocks' guide layers from: stored (gin [blk][face][p];
// not with sweep and residual together), the neighbours' interiors, or the
// neighbours' interiors with what the sweep before pushed into gin (only with
// the residual).
enum class RbgsGuides { STORED, PULL, PUSHED };
// Fused residual + red-black sweep (rbgs_block.cu); C.urec must be set.  A
// sweep with gout pushes guides for the next pass into it (PUSHED).
// pdl: launched as a programmatic dependent of the previous kernel on the
// stream, which must then be a pass of this kernel.  order: the C.nb blocks in
// the order the grid takes them (null: block order); results do not depend on it.
void launch_rbgs(cudaStream_t s, const KCtx& C, bool res, bool sweep, const double* xin,
                 double* xout, const double* A, const double* b, RbgsGuides from,
                 const double* gin, double* gout, double omega, double* partials, SolveState* st,
                 int fin, int iter, bool pdl = false, const int32_t* order = nullptr);
int rbgs_ordered_blocks();  // pools up to here take an order
// Test hook: the first sweep (stored guides, no residual), in the form that
// launch_rbgs or, ring, launch_rbgs_ring would take, with copies left out that
// it then waits for.
void launch_rbgs_stalled(cudaStream_t s, const KCtx& C, bool ring, const double* xin,
                         double* xout, const double* A, const double* b, const double* gin,
                         double* gout, double omega, double* partials, SolveState* st,
                         const int32_t* order);
// The same pass with the coefficients through a ring of bulk copies
// (rbgs_ring.cu): guides stored (gst) or, gst null, from the neighbours'
// interiors.  pdl as above, after a pass of either kernel.
void launch_rbgs_ring(cudaStream_t s, const KCtx& C, bool res, bool sweep, const double* xin,
                      double* xout, const double* A, const double* b, const double* gst,
                      double omega, double* partials, SolveState* st, int fin, int iter,
                      bool pdl = false, bool stall = false);
int sm_count();  // of the current device
// Each block's uniform record urec[blk][8] (Ap..At of cell 0, then 1.0 when
// every cell has those seven coefficients, else 0.0), adding the uniform
// blocks to *ucount.
void launch_urec(cudaStream_t s, int nb, const double* A, double* urec, int32_t* ucount);
// Jacobi sweep from the zero field, with b.x1 (FIN_CG_RR1): CG's preconditioner
// of one pass.  A block with a set uniform record (C.urec) reads its seven
// coefficients from it.
void launch_jacobi_dot(cudaStream_t s, const KCtx& C, double* xout, const double* A,
                       const double* b, double omega, double* partials, SolveState* st);
void launch_calc_r(cudaStream_t s, const KCtx& C, const double* x, const double* gst,
                   const double* A, const double* b, double* r, SolveState* st);
// Cell-wise steps of the Krylov solvers (krylov_block.cu), with the Jacobi pass
// from zero on the vector formed (C.urec must be set) into z unless z is null,
// the guides of z (launch_cg_p: of p) pushed into gout unless that is null.
// p = r (and r0 = r) on the first iteration of a cycle (st->cycle == 1), else the update.
void launch_bicg_p(cudaStream_t s, const KCtx& C, double* r, double* p, double* q, double* r0,
                   const double* A, double* z, double omega, double* gout, SolveState* st);
void launch_bicg_s(cudaStream_t s, const KCtx& C, double* sv, double* q, double* r,
                   const double* A, double* z, double omega, double* gout, SolveState* st);
// x, r, the residual of iteration iter, and DOT(r, r0) of the next (partials [2][nb]).
void launch_bicg_update(cudaStream_t s, const KCtx& C, double* x, double* pz, double* sz,
                        double* r, double* t, double* sv, double* r0, double* partials,
                        SolveState* st, int iter);
void launch_jacobi_zero(cudaStream_t s, const KCtx& C, double* r, const double* A, double* z,
                        double omega, double* gout, SolveState* st);
void launch_cg_p(cudaStream_t s, const KCtx& C, double* z, double* p, double* gout,
                 SolveState* st, int iter);
void launch_cg_update(cudaStream_t s, const KCtx& C, double* x, double* p, double* r, double* q,
                      const double* A, double* z, double omega, double* gout, double* partials,
                      SolveState* st, int iter);
// Sum of x over the interior (finaliser fin); x += st->alpha.
void launch_sum(cudaStream_t s, const KCtx& C, const double* x, double* partials, SolveState* st,
                int fin);
void launch_shift(cudaStream_t s, const KCtx& C, double* x, SolveState* st);
// r.r0 (setting r0 = r first on the first iteration of a cycle).
void launch_dot_rr0(cudaStream_t s, const KCtx& C, const double* r, double* r0, double* partials,
                    SolveState* st, int fin, int iter);
void launch_dot(cudaStream_t s, const KCtx& C, const double* x, const double* y,
                double* partials, SolveState* st, int fin, int iter);
void launch_exchange(cudaStream_t s, const KCtx& C, const double* x, double* g);
void launch_pack(cudaStream_t s, int nb, const double* stage, int vc, double* dst, size_t stride,
                 double* gdst);
void launch_pack_flag(cudaStream_t s, int nb, const int32_t* stage, int vc, uint8_t* flags,
                      int bit, int mode);
void launch_unpack_flag(cudaStream_t s, int nb, const uint8_t* flags, int vc, int32_t* stage,
                        int bit);
void launch_unpack(cudaStream_t s, const KCtx& C, const double* src, size_t stride, int vc,
                   int with_guides, double* stage);
void launch_assemble(cudaStream_t s, const KCtx& C, const double* ux, const double* uy,
                     const double* uz, const double* gux, const double* guy, const double* guz,
                     const double* cut, const uint8_t* flags, double* A, double* b,
                     double* vface, double rhof, double dt, size_t field_stride);
void launch_fold_bc(cudaStream_t s, const KCtx& C, double* A, double* b);
// bcut_remove_p (corr false) or bcut_corr_u (corr true) on every block.
void launch_projection(cudaStream_t s, const KCtx& C, bool corr, const double* p,
                       const double* gp, const double* cut, const uint8_t* flags, double* ux,
                       double* uy, double* uz, double* vface, double* lapp, double rhof,
                       double dt, size_t field_stride);
void launch_fill(cudaStream_t s, int nb, double* x, size_t stride, double* g, double value);

// Sets the message ffvgpu_last_error() returns on this thread.
void set_last_error(const std::string& msg);

}  // namespace ffvgpu
