// krylov_block.cu -- the cell-wise steps of the FP64 Krylov solvers
// (FFVILS::CG and BiCGSTAB, src/FFV/FFVILS.h:661-974), each with what the
// recurrence does next on the same values: the first pass of the Jacobi
// preconditioner on the vector just formed, the guides the pass after it
// needs, and the dot product the next iteration starts with.
//
// One CTA of 256 threads per block, in the cell order of the stencil kernels
// (ffvgpu_tile.cuh).  Bound by HBM: every vector is read or written once.
// Level-5 sphere grid, BiCGSTAB, us per launch: p with its pass from zero 156
// (86 + 72 as two kernels; 868 MB, 134 us at the measured 6463 GB/s), s with its
// 122 (65 + 72), the update with the next r.r0 182 (174 + 64).  Launched
// normally, not as programmatic dependents: their loads live on the L1 that
// the stencil kernels' shared memory takes, and an overlapped launch keeps the
// stencil kernels' split (24 iterations: 25.0 ms against 27.5).
#include <cfloat>
#include <cuda_runtime.h>

#include "ffvgpu_internal.cuh"
#include "ffvgpu_kernels.h"
#include "ffvgpu_tile.cuh"

namespace ffvgpu {

namespace {

using namespace tile;

// What a kernel forms:
//   P       BiCGSTAB's p (FFVILS.h:853-871): p = r on the first iteration of a
//           cycle (with r0 = r), else t = p + (-gamma) q, p = r + beta t
//   S       s = (-alpha) q + r (FFVILS.h:898-903)
//   CG_P    CG's p = z, or z + beta p (xpay, blas.f90:363-395)
//   CG_XR   x = x + alpha p, r = r + (-alpha) q, r.r (FFVILS.h:760-788)
//   R       nothing: the Jacobi pass reads r
//   BI_XR   x = alpha p_ + gamma s_ + x, r = (-gamma) t + s, r.r and the next
//           iteration's r.r0 (FFVILS.h:938-958, 845-846)
enum Step { P, S, CG_P, CG_XR, R, BI_XR };

struct Vectors {
  double* out;   // P, S, CG_P: the vector formed; CG_XR, BI_XR: x; R: r
  double* r;     // P: r; S: r; CG_P: z; CG_XR, BI_XR: r
  double* q;     // P, S, CG_XR: q; BI_XR: t
  double* a;     // P: r0; CG_XR: p; BI_XR: p_
  double* b;     // BI_XR: s_
  double* c;     // BI_XR: s
  double* d;     // BI_XR: r0
};

// A Jacobi pass from the zero field on right-hand side v (bils.f90:5-55 after
// FFVILS::Fill(z, 0)).  The products with the zero neighbours are kept: they
// decide the sign of a zero residual.
__device__ __forceinline__ double zero_residual(double v, const K7& k) {
  const double z = 0.0;
  return v - k.w * z - k.e * z - k.s * z - k.n * z - k.b * z - k.t * z;
}

// JAC: the Jacobi pass on the vector formed (r for CG_XR and R), into z.
// push: the guides of the last vector written (z, or CG_P's p) into gout.
template <int STEP, bool JAC>
__global__ void __launch_bounds__(NT, 3)
krylov_step_kernel(const __grid_constant__ KCtx C, const Vectors V, const double* __restrict__ A,
                   double* __restrict__ zout, double omega, double* __restrict__ gout,
                   double* __restrict__ partials, SolveState* st, int iter) {
  constexpr int NV = STEP == BI_XR ? 2 : STEP == CG_XR ? 1 : 0;
  __shared__ double T[JAC || STEP == CG_P ? TT : 1];
  __shared__ double ws[2][16];
  __shared__ FaceNbr nbr[6];
  __shared__ int last;
  const int tid = threadIdx.x, blk = blockIdx.x;
  if (gout && tid < 6) nbr[tid] = C.nbr[(size_t)blk * 6 + tid];
  double u[8];
  if (JAC) {
#pragma unroll
    for (int a = 0; a < 8; ++a) u[a] = __ldg(C.urec + (size_t)blk * 8 + a);
  }
  if (*((volatile const int32_t*)&st->done) != 0) return;
  const double alpha = st->alpha, beta = st->beta, gamma = st->gamma;
  const bool first = STEP == P ? st->cycle == 1 : STEP == CG_P ? iter == 1 : false;
  const size_t base = (size_t)blk * BLOCK_CELLS + slot(tid);
  const double* Ab = A + (size_t)blk * 7 * BLOCK_CELLS + slot(tid);
  const bool uni = JAC && u[7] != 0.0;
  const Divisor D(JAC ? u[0] : 1.0);
  double acc[2][2][2] = {};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    double v[NC];
    // the vector, a colour's loads in flight together
    if (STEP == P && first) {
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const size_t s = base + c * HALF_CELLS + plane(n) * 128;
        v[n] = V.r[s];
        V.a[s] = v[n];
      }
    } else if (STEP == CG_P && first) {
#pragma unroll
      for (int n = 0; n < NC; ++n) v[n] = V.r[base + c * HALF_CELLS + plane(n) * 128];
    } else {
      double l0[NC], l1[NC], l2[NC];
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const size_t s = base + c * HALF_CELLS + plane(n) * 128;
        if (STEP == P || STEP == S || STEP == CG_XR || STEP == R || STEP == CG_P) l0[n] = V.r[s];
        if (STEP == P || STEP == S || STEP == CG_XR || STEP == BI_XR) l1[n] = V.q[s];
        if (STEP == P || STEP == CG_P) l2[n] = V.out[s];
        if (STEP == BI_XR) l2[n] = V.c[s];
      }
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        if (STEP == P) {
          const double t = l2[n] + (-gamma) * l1[n];
          v[n] = l0[n] + beta * t;
        } else if (STEP == S) {
          v[n] = (-alpha) * l1[n] + l0[n];
        } else if (STEP == CG_P) {
          v[n] = l0[n] + beta * l2[n];
        } else if (STEP == CG_XR) {
          v[n] = l0[n] + (-alpha) * l1[n];
        } else if (STEP == BI_XR) {
          v[n] = (-gamma) * l1[n] + l2[n];
        } else {
          v[n] = l0[n];
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NC; ++n) {
      const size_t s = base + c * HALF_CELLS + plane(n) * 128;
      if (STEP == P || STEP == S || STEP == CG_P) V.out[s] = v[n];
      if (STEP == CG_XR || STEP == BI_XR) {
        V.r[s] = v[n];
        acc[0][c][n & 1] += v[n] * v[n];
      }
      if (STEP == CG_P && gout) T[own(tid) + c * TH + plane(n) * TP] = v[n];
    }
    if (STEP == CG_XR) {
      double l0[NC], l1[NC];
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const size_t s = base + c * HALF_CELLS + plane(n) * 128;
        l0[n] = V.out[s];
        l1[n] = V.a[s];
      }
#pragma unroll
      for (int n = 0; n < NC; ++n)
        V.out[base + c * HALF_CELLS + plane(n) * 128] = l0[n] + alpha * l1[n];
    }
    if (STEP == BI_XR) {
      double l0[NC], l1[NC], l2[NC];
#pragma unroll
      for (int n = 0; n < NC; ++n) acc[1][c][n & 1] += v[n] * V.d[base + c * HALF_CELLS + plane(n) * 128];
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const size_t s = base + c * HALF_CELLS + plane(n) * 128;
        l0[n] = V.out[s];
        l1[n] = V.a[s];
        l2[n] = V.b[s];
      }
#pragma unroll
      for (int n = 0; n < NC; ++n)
        V.out[base + c * HALF_CELLS + plane(n) * 128] = alpha * l1[n] + gamma * l2[n] + l0[n];
    }
    if (JAC) {
      const double x0 = 0.0;
      if (uni) {
        const K7 k = uniform_coefs(u);
        bool ok = D.normal;
#pragma unroll
        for (int n = 0; n < NC; ++n) {
          v[n] = zero_residual(v[n], k);
          ok = ok && D.ok(v[n]);
        }
        if (ok) {
#pragma unroll
          for (int n = 0; n < NC; ++n) v[n] = D(v[n]);
        } else {
#pragma unroll
          for (int n = 0; n < NC; ++n) v[n] = v[n] / D.d;
        }
      } else {
#pragma unroll  // fully: v stays in registers
        for (int n = 0; n < NC; ++n) {
          const K7 k = stream_coefs(Ab, c * HALF_CELLS + plane(n) * 128);
          v[n] = zero_residual(v[n], k) / k.p;
        }
      }
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const double z = x0 - omega * (x0 - v[n]);
        zout[base + c * HALF_CELLS + plane(n) * 128] = z;
        if (gout) T[own(tid) + c * TH + plane(n) * TP] = z;
      }
    }
  }
  if ((JAC || STEP == CG_P) && gout) {
    __syncthreads();
    push_guides(T, nbr, gout);
  }
  if (NV == 0) return;
#pragma unroll
  for (int k = 0; k < NV; ++k) warp_sums(acc[k], ws[k]);
  __syncthreads();
  const int nb = gridDim.x;
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) __stcg(partials + (size_t)k * nb + blk, block_sum(ws[k]));
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == (unsigned)nb - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double tot[2] = {};
#pragma unroll
  for (int k = 0; k < NV; ++k) tot[k] = cross_block_sum(partials + (size_t)k * nb, nb, ws[0]);
  if (tid == 0) {
    finalize(st, tot[0], STEP == BI_XR ? FIN_BI_RR : FIN_CG_RR, iter);
    // the next iteration's DOT(r, r0); after a restart r0 = r (which its P step
    // writes), so that the product is r.r
    if (STEP == BI_XR && !st->done) finalize(st, st->cycle == 1 ? tot[0] : tot[1], FIN_BI_RR1, iter + 1);
    st->ticket = 0;
    __threadfence();
  }
}

template <int STEP, bool JAC>
void step(cudaStream_t s, const KCtx& C, const Vectors& V, const double* A, double* z,
          double omega, double* gout, double* partials, SolveState* st, int iter) {
  krylov_step_kernel<STEP, JAC><<<C.nb, NT, 0, s>>>(C, V, A, z, omega, gout, partials, st, iter);
}

}  // namespace

void launch_bicg_p(cudaStream_t s, const KCtx& C, double* r, double* p, double* q, double* r0,
                   const double* A, double* z, double omega, double* gout, SolveState* st) {
  const Vectors V{p, r, q, r0, nullptr, nullptr, nullptr};
  z ? step<P, true>(s, C, V, A, z, omega, gout, nullptr, st, 0)
    : step<P, false>(s, C, V, A, z, omega, nullptr, nullptr, st, 0);
}
void launch_bicg_s(cudaStream_t s, const KCtx& C, double* sv, double* q, double* r,
                   const double* A, double* z, double omega, double* gout, SolveState* st) {
  const Vectors V{sv, r, q, nullptr, nullptr, nullptr, nullptr};
  z ? step<S, true>(s, C, V, A, z, omega, gout, nullptr, st, 0)
    : step<S, false>(s, C, V, A, z, omega, nullptr, nullptr, st, 0);
}
void launch_bicg_update(cudaStream_t s, const KCtx& C, double* x, double* pz, double* sz,
                        double* r, double* t, double* sv, double* r0, double* partials,
                        SolveState* st, int iter) {
  const Vectors V{x, r, t, pz, sz, sv, r0};
  step<BI_XR, false>(s, C, V, nullptr, nullptr, 0.0, nullptr, partials, st, iter);
}
void launch_jacobi_zero(cudaStream_t s, const KCtx& C, double* r, const double* A, double* z,
                        double omega, double* gout, SolveState* st) {
  const Vectors V{nullptr, r, nullptr, nullptr, nullptr, nullptr, nullptr};
  step<R, true>(s, C, V, A, z, omega, gout, nullptr, st, 0);
}
void launch_cg_p(cudaStream_t s, const KCtx& C, double* z, double* p, double* gout,
                 SolveState* st, int iter) {
  const Vectors V{p, z, nullptr, nullptr, nullptr, nullptr, nullptr};
  step<CG_P, false>(s, C, V, nullptr, nullptr, 0.0, gout, nullptr, st, iter);
}
void launch_cg_update(cudaStream_t s, const KCtx& C, double* x, double* p, double* r, double* q,
                      const double* A, double* z, double omega, double* gout, double* partials,
                      SolveState* st, int iter) {
  const Vectors V{x, r, q, p, nullptr, nullptr, nullptr};
  z ? step<CG_XR, true>(s, C, V, A, z, omega, gout, partials, st, iter)
    : step<CG_XR, false>(s, C, V, A, z, omega, nullptr, partials, st, iter);
}

}  // namespace ffvgpu
