// matvec_block.cu -- A x with its dot products, and a Jacobi pass, for sm_100a:
// the stencil kernels of the FP64 Krylov solvers (FFVILS::CG and BiCGSTAB,
// src/FFV/FFVILS.h:661-974) on pools of mostly uniform blocks (ring_pool in
// pool.cpp).
//
// y = A x (calc_ax, src/CGMfuncs/bils.f90:162-206) with y.w0 (NV 1: q_.r0 or
// q.p) or y.w0 and y.y (NV 2: t_.s and t_.t_); or, JAC, a Jacobi sweep of x with
// right-hand side w0 (bils.f90:5-55) and, NV 1, w0.y.  Blocks as in the RBGS
// pass: two CTAs of 256 threads per SM, x in registers and a tile, w0 by a bulk
// copy a block ahead, the next block's x loaded while a block's sums are formed.
// A CTA walks the live blocks of its part of the active list; sums are per
// instance, over its blocks in block order.
//
// What bounds it: the loads between a block's barriers (x, guides, a varied
// block's coefficients) against the 28 KB of L1 that two CTAs' shared memory
// leaves.  Level-5 sphere grid, us per launch, one 800-thread warp-specialised
// CTA per SM before -> here: A x with q.r0 154 -> 123, with t.s and t.t
// 164 -> 128, a Jacobi pass 152 -> 140 (87 us at the measured 6463 GB/s for the
// 561 MB that must move).  Tried without gain:
// w0 in registers (more L1, but spills), three CTAs' worth of carve-out.
#include <algorithm>
#include <cstddef>
#include <cuda_runtime.h>

#include "ffvgpu_async.cuh"
#include "ffvgpu_instance.cuh"
#include "ffvgpu_internal.cuh"
#include "ffvgpu_mixed.h"
#include "ffvgpu_tile.cuh"

namespace ffvgpu {

namespace {

using namespace tile;

constexpr int ROLE_MATVEC = 64;  // SolveState::timeout_where bit of this kernel's waits
constexpr int CAP = NT;          // list entries per chunk

struct __align__(128) Smem {
  double w[2][BLOCK_CELLS];  // w0 of the current / next block
  double tile[TT];
  Record rec[3];             // records of the current block and the two after it
  double ws[2][2][16];
  int2 list[CAP];
  uint64_t rbar[3], wbar[2];
  int wcount[NT / 32];
  int nlist, next_from, abort_flag, last_inst;
};
static_assert(2 * (sizeof(Smem) + 1024) <= 228 * 1024, "two CTAs per SM");

struct Row {  // a uniform block's coefficients
  K7 k;
  Divisor D;
  __device__ __forceinline__ Row(const double* u, bool div)
      : k(uniform_coefs(u)), D(div ? u[0] : 1.0) {}
  __device__ __forceinline__ const K7& at(int, int) const { return k; }
};
struct Rows {  // A's rows at the thread's first cell
  const double* Ab;
  __device__ __forceinline__ K7 at(int c, int n) const {
    return stream_coefs(Ab, c * HALF_CELLS + plane(n) * 128);
  }
};
template <int N>
__device__ __forceinline__ void divide(const Row& A, double (&rs)[N], const double (&)[N]) {
  bool ok = A.D.normal;
#pragma unroll
  for (int m = 0; m < N; ++m) ok = ok && A.D.ok(rs[m]);
  if (ok) {
#pragma unroll
    for (int m = 0; m < N; ++m) rs[m] = A.D(rs[m]);
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) rs[m] = rs[m] / A.D.d;
  }
}
template <int N>
__device__ __forceinline__ void divide(const Rows&, double (&rs)[N], const double (&ap)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m) rs[m] = rs[m] / ap[m];
}

// The cells of one staged block; w and y start at the thread's first cell.
// With JAC the new values replace X (a cell's neighbours are of the other
// colour: colour 0 is formed into Y first).
template <int NV, bool JAC, typename COEF>
__device__ __forceinline__ void cells(const double* T, double (&X)[2][NC], const COEF& A,
                                      const double* w, double* __restrict__ y, double omega,
                                      double (&acc)[2][2][2]) {
  constexpr int G = 4;  // cells whose loads are in flight together
  double Y0[JAC ? NC : 1];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const Around N(T, c);
#pragma unroll
    for (int n0 = 0; n0 < NC; n0 += G) {
      double v[G], ap[G], wv[G];
#pragma unroll
      for (int n = n0; n < n0 + G; ++n) {
        const int s = c * HALF_CELLS + plane(n) * 128;
        const K7 k = A.at(c, n);
        const Nbrs b = N.at(n, X[1 - c]);
        wv[n - n0] = (NV > 0 || JAC) ? w[s] : 0.0;
        if (JAC) {
          v[n - n0] = minus_neighbours(wv[n - n0], k, b);
          ap[n - n0] = k.p;
        } else {
          v[n - n0] = k.w * b.w + k.e * b.e + k.s * b.s + k.n * b.n + k.b * b.b + k.t * b.t +
                      k.p * X[c][n];
        }
      }
      if (JAC) {
        divide(A, v, ap);
#pragma unroll
        for (int n = n0; n < n0 + G; ++n) v[n - n0] = X[c][n] - omega * (X[c][n] - v[n - n0]);
      }
#pragma unroll
      for (int n = n0; n < n0 + G; ++n) {
        const double yv = v[n - n0];
        y[c * HALF_CELLS + plane(n) * 128] = yv;
        if (NV > 0) acc[0][c][n & 1] += yv * wv[n - n0];
        if (NV == 2) acc[1][c][n & 1] += yv * yv;
        if (JAC) {
          if (c == 0)
            Y0[JAC ? n : 0] = yv;
          else
            X[1][n] = yv;
        }
      }
    }
  }
  if (JAC)
#pragma unroll
    for (int n = 0; n < NC; ++n) X[0][n] = Y0[JAC ? n : 0];
}

// STALL (test hook): no w0 for the last block of the CTAs with most.
template <int NV, bool JAC, int SRC, bool STALL>
__global__ void __launch_bounds__(NT, 2)
matvec_block_kernel(const __grid_constant__ MixCtx C, const double* __restrict__ x,
                    const double* __restrict__ A, double* __restrict__ y,
                    const double* __restrict__ w0, double omega) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  double* T = S.tile;
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) async::mbar_init(&S.rbar[k], REC_THREADS);
    for (int k = 0; k < 2; ++k) async::mbar_init(&S.wbar[k], 1);
    S.abort_flag = 0;
    async::fence_mbar_init();
  }
  __syncthreads();
  const int n_act = *C.n_active;
  auto fetch_rec = [&](int blk, int m) {  // record of the CTA's m-th block
    if (tid < REC_THREADS)
      fetch_record(S.rec[m % 3], &S.rbar[m % 3], C.nbr, C.ucoef, blk);
  };
  auto stalled = [&](int m) { return STALL && m == (n_act - 1) / (int)gridDim.x; };
  auto fetch_w = [&](int blk, int m) {  // w0 of the CTA's m-th block
    if (tid == 32 && !stalled(m)) {
      async::mbar_expect_tx(&S.wbar[m & 1], BLOCK_CELLS * 8);
      async::bulk_g2s(S.w[m & 1], w0 + (size_t)blk * BLOCK_CELLS, BLOCK_CELLS * 8, &S.wbar[m & 1]);
    }
  };
  auto wait_rec = [&](int m) {
    return async::mbar_wait(&S.rbar[m % 3], (m / 3) & 1, &S.abort_flag, ROLE_MATVEC, C.wait_ns);
  };
  double X[2][NC];
  Staging<SRC, ReadOnly> L;
  int n = 0;      // blocks of this CTA so far
  int run = 0;    // thread 0: blocks of the current instance not yet on its ticket
  int ahead = 0;  // whether block n + 1's record has been fetched
  bool ok = true;
  for (int from = blockIdx.x; ok && from < n_act;) {
    build_live_list<1, false, NT, CAP>(C, from, n_act, S.list, &S.nlist, &S.next_from, S.wcount);
    from = S.next_from;
    const int nl = S.nlist;
    if (nl > 0) {
      fetch_rec(S.list[0].x, n);
      fetch_w(S.list[0].x, n);
      if (nl > 1) fetch_rec(S.list[1].x, n + 1);
      ok = wait_rec(n);
      if (ok) L.load(X, x, S.list[0].x, S.rec[n % 3].nbr, C.gin);
    }
    for (int pos = 0; pos < nl; ++pos, ++n) {
      const int k = n & 1;
      const int2 ent = S.list[pos];
      const int blk = ent.x, inst = ent.y & LF_INST;
      const int next = pos + 1 < nl ? S.list[pos + 1].x : -1;
      const int after = pos + 2 < nl ? S.list[pos + 2].x : -1;
      ahead = next >= 0;
      const Record& R = S.rec[n % 3];
      if (JAC && n > 0) __syncthreads();  // the pushes of the block before are out of the tile
      if (ok) L.put(T, X, x, blk, R.nbr, C.bc, C.dx);
      ok = ok && async::mbar_wait(&S.wbar[k], (n >> 1) & 1, &S.abort_flag, ROLE_MATVEC, C.wait_ns);
      ok = ok && (next < 0 || wait_rec(n + 1));
      if (__syncthreads_or(!ok)) {
        ok = false;
        break;
      }
      // buffers whose last reads were before the previous block's barriers
      if (next >= 0) {
        fetch_w(next, n + 1);
        if (tid == 64)
          async::prefetch_l2(x + (size_t)next * BLOCK_CELLS, BLOCK_CELLS * 8);
        if (tid == 96 && S.rec[(n + 1) % 3].u[7] == 0.0)
          async::prefetch_l2(A + (size_t)next * 7 * BLOCK_CELLS, 7 * BLOCK_CELLS * 8);
      }
      if (after >= 0) fetch_rec(after, n + 2);
      const double* w = S.w[k] + slot(tid);
      double* yb = y + (size_t)blk * BLOCK_CELLS + slot(tid);
      double acc[2][2][2] = {};
      if (R.u[7] != 0.0)
        cells<NV, JAC>(T, X, Row(R.u, JAC), w, yb, omega, acc);
      else
        cells<NV, JAC>(T, X, Rows{A + (size_t)blk * 7 * BLOCK_CELLS + slot(tid)}, w, yb, omega, acc);
      // the next block's loads are in flight over the sums (and pushes)
      if (!JAC && next >= 0) L.load(X, x, next, S.rec[(n + 1) % 3].nbr, C.gin);
      // the warp sums alternate between two buffers: block n + 2 writes its
      // buffer after block n + 1's barrier, which thread 0 passes after its read
#pragma unroll
      for (int v = 0; v < NV; ++v) warp_sums(acc[v], S.ws[k][v]);
      async::fence_proxy_async();  // w[k] is refilled by a bulk copy after the barriers
      __syncthreads();
      if (NV > 0 && tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
          __stcg(C.partials + (size_t)v * C.capacity + blk, block_sum(S.ws[k][v]));
        ++run;
      }
      if (JAC && C.gout) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int m = 0; m < NC; ++m) T[own(tid) + c * TH + plane(m) * TP] = X[c][m];
      }
      if (JAC && next >= 0) L.load(X, x, next, S.rec[(n + 1) % 3].nbr, C.gin);
      if (JAC && C.gout) {
        __syncthreads();
        push_guides(T, R.nbr, C.gout);
      }
      // the instance's ticket, once per run of its blocks in this chunk
      if (NV > 0 && (pos + 1 == nl || (S.list[pos + 1].y & LF_INST) != inst)) {
        if (tid == 0) {
          __threadfence();
          const unsigned t = atomicAdd(&C.inst.st[inst].ticket, (unsigned)run);
          S.last_inst = t + (unsigned)run == (unsigned)C.inst.count[inst] ? inst : -1;
          run = 0;
        }
        __syncthreads();
        const int li = S.last_inst;
        if (li >= 0) {
          __threadfence();
          const int first = C.inst.first[li], cnt = C.inst.count[li];
          double tot[2] = {};
#pragma unroll
          for (int v = 0; v < NV; ++v)
            tot[v] = cross_block_sum(C.partials + (size_t)v * C.capacity + first, cnt, S.ws[k][0]);
          if (tid == 0) {
            SolveState* St = C.inst.st + li;
            finalize(St, tot[0], C.fin, 0);
            if (NV == 2) finalize(St, tot[1], FIN_BI_TT, 0);
            St->ticket = 0;
            __threadfence();
          }
        }
        __syncthreads();  // S.last_inst and S.ws are rewritten
      }
    }
    if (ok) __syncthreads();  // every thread is past the chunk before its list is rebuilt
  }
  if (!ok && tid == 0) {
    // Copies that may still be on their way into this CTA's shared memory:
    // block n's and n + 1's records and block n's w0 (a step issues the ones
    // after them only once its waits have succeeded).
    bool drained = stalled(n) || async::mbar_drain(&S.wbar[n & 1], (n >> 1) & 1);
    drained = async::mbar_drain(&S.rbar[n % 3], (n / 3) & 1) && drained;
    if (ahead) drained = async::mbar_drain(&S.rbar[(n + 1) % 3], ((n + 1) / 3) & 1) && drained;
    // stop every instance of this CTA's chunk and of its later candidates
    const int where = ROLE_MATVEC | (drained ? 0 : async::ROLE_DRAIN);
    auto stop = [&](int i) {
      atomicOr(&C.inst.st[i].timeout_where, where);
      atomicExch(&C.inst.st[i].status, 3);
      atomicExch(&C.inst.st[i].done, 1);
    };
    for (int p = 0; p < S.nlist; ++p) stop(S.list[p].y & LF_INST);
    for (int it = S.next_from; it < n_act; it += gridDim.x) {
      const int i = C.inst.blk_inst[C.active[it]];
      if (i >= 0) stop(i);
    }
  }
}

template <int NV, bool JAC>
void launch(cudaStream_t s, const MixCtx& C, int count, const double* x, const double* A,
            double* y, const double* w0, double omega) {
  constexpr bool FIRST = NV < 2;  // a solve's first stencil launch never has two sums
  auto kernel = C.stall == 2 && FIRST
                    ? (C.gin ? matvec_block_kernel<NV, JAC, PUSHED, FIRST>
                             : matvec_block_kernel<NV, JAC, PULL, FIRST>)
                    : (C.gin ? matvec_block_kernel<NV, JAC, PUSHED, false>
                             : matvec_block_kernel<NV, JAC, PULL, false>);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
  kernel<<<count, NT, sizeof(Smem), s>>>(C, x, A, y, w0, omega);
}

}  // namespace

int matvec_block_grid() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return 2 * std::max(1, sms);
}

void launch_matvec_block(cudaStream_t s, const MixCtx& C, int count, int ndot, const double* x,
                         const double* A, double* y, const double* w0) {
  ndot == 1 ? launch<1, false>(s, C, count, x, A, y, w0, 0.0)
            : launch<2, false>(s, C, count, x, A, y, w0, 0.0);
}

void launch_jacobi_block(cudaStream_t s, const MixCtx& C, int count, bool dot, const double* x,
                         const double* A, const double* b, double* y, double omega) {
  dot ? launch<1, true>(s, C, count, x, A, y, b, omega)
      : launch<0, true>(s, C, count, x, A, y, b, omega);
}

}  // namespace ffvgpu
