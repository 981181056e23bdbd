// rbgs_block.cu -- fused residual + red-black sweep for sm_100a (the hot
// kernel of FFVILS::RBGS).
//
// Per pass over the pool it computes, for every leaf block, the residual
// sum of x_in (calc_r2, src/CGMfuncs/bils.f90:256-304) and the red-black
// SOR sweep x_in -> x_out (rbgs_smoother, bils.f90:57-108, colour 0 then
// colour 1 against guide values from the previous exchange), with the same
// rounding as the reference (compiled with --fmad=false) and the same sum
// tree as the rest of the path.
//
// Two CTAs of 256 threads share an SM, each with one block at a time: its x
// in registers (ffvgpu_tile.cuh: a thread's cells are pairs of planes, so one
// x and one z neighbour of a cell are its own) and in a tile, its b brought by
// a bulk copy while the block before it is computed, its x and A prefetched
// into L2.  What bounds it: the loads and barriers between a block's phases
// (staging, colour-1 residual, colour 0, colour 1) and shared memory, which
// the second CTA overlaps only in part; FP64 arithmetic is a quarter of the
// time.  Level-5 sphere grid (4692 blocks, 4256 uniform), per pass: 147 us (87
// at the measured 6463 GB/s for the 561 MB that must move), 230 us with one cell
// per consumer thread and neighbours chosen by selects (rbgs_ring.cu, which
// brings 254 MB of coefficients and b through a ring; it serves the pools of
// mostly varied blocks); a copy of x through the same structure takes 86 us,
// the pass without guide layers 125 us.  72 blocks: 18.0 -> 13.7 us; 324: 33 ->
// 25.7 us.  Tried and slower at level 5 (us per pass): 128 threads with whole
// k columns in registers 199; 512 threads on strided planes, one CTA per SM
// with everything staged a block ahead 180, two CTAs 163; guides of x and 2:1
// faces read from the neighbours' interiors instead of pushed 176.
#include <algorithm>
#include <cfloat>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <cuda_runtime.h>

#include "ffvgpu_async.cuh"
#include "ffvgpu_internal.cuh"
#include "ffvgpu_kernels.h"
#include "ffvgpu_tile.cuh"

namespace ffvgpu {

namespace {

using namespace tile;

constexpr int ROLE_RBGS = 4;  // SolveState::timeout_where bit (consumer)

// Where a thread's cells take their coefficients from: a uniform block's
// record, with one divisor for all; A's rows; or, with one block per SM, A's
// rows with colour 1's coefficients, which two phases use, held in registers
// (loaded while the block is still being staged).
struct Uniform {
  K7 k;
  Divisor D;
  __device__ __forceinline__ explicit Uniform(const double* u) : k(uniform_coefs(u)), D(u[0]) {}
  __device__ __forceinline__ const K7& at(int, int) const { return k; }
  __device__ __forceinline__ const Uniform& again() const { return *this; }
};
struct Varied {
  const double* Ab;  // at the thread's first cell
  __device__ __forceinline__ explicit Varied(const double* A, bool = true) : Ab(A) {}
  __device__ __forceinline__ K7 at(int c, int n) const {
    return stream_coefs(Ab, c * HALF_CELLS + plane(n) * 128);
  }
  // The same pointer as another value, so that colour 1's coefficients are
  // read again for the update instead of being spilled to keep them.
  __device__ __forceinline__ Varied again() const {
    const double* p = Ab;
    asm volatile("" : "+l"(p));
    return Varied{p};
  }
};
struct Held {
  const double* Ab;
  K7 k1[NC];
  // (a uniform block, which does not use them, loads none: its pass would read
  // 115 KB more)
  __device__ __forceinline__ Held(const double* A, bool varied) : Ab(A), k1() {
    if (varied)
#pragma unroll
      for (int n = 0; n < NC; ++n) k1[n] = stream_coefs(Ab, HALF_CELLS + plane(n) * 128);
  }
  __device__ __forceinline__ K7 at(int c, int n) const {
    return c ? k1[n] : stream_coefs(Ab, plane(n) * 128);
  }
  __device__ __forceinline__ const Held& again() const { return *this; }
};

// rs / ap of N cells, formed together so that their chains overlap.
template <int N>
__device__ __forceinline__ void divide(const Uniform& A, double (&rs)[N], const double (&)[N]) {
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
template <typename V, int N>
__device__ __forceinline__ void divide(const V&, double (&rs)[N], const double (&ap)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m) rs[m] = rs[m] / ap[m];
}

// The sweep and residual of one staged block.  The colour-1 residual, against
// the old colour-0 values, comes first; then the colour-0 cells, whose new
// values replace the old in registers and tile; then the colour-1 update.
// b and xo start at the thread's first cell.
template <bool RES, bool SWEEP, typename COEF>
__device__ __forceinline__ void rbgs_cells(double* T, double (&X)[2][NC], const COEF& A,
                                           const double* b, double* __restrict__ xo,
                                           double omega, double (&acc)[2][2]) {
  constexpr int G = 4;  // cells whose loads are in flight together
  const int t = threadIdx.x;
  if (RES) {
    const Around N(T, 1);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
      const int s = HALF_CELLS + plane(n) * 128;
      const K7 a = A.at(1, n);
      const double r = minus_neighbours(b[s], a, N.at(n, X[0])) - a.p * X[1][n];
      acc[1][n & 1] += r * r;
    }
    if (SWEEP) __syncthreads();  // before the old colour-0 values leave the tile
  }
  {
    const Around N(T, 0);
#pragma unroll
    for (int n0 = 0; n0 < NC; n0 += G) {
      double rs[G], ap[G];
#pragma unroll
      for (int n = n0; n < n0 + G; ++n) {
        const int s = plane(n) * 128;
        const K7 a = A.at(0, n);
        rs[n - n0] = minus_neighbours(b[s], a, N.at(n, X[1]));
        ap[n - n0] = a.p;
        if (RES) {
          const double r = rs[n - n0] - a.p * X[0][n];
          acc[0][n & 1] += r * r;
        }
      }
      if (SWEEP) {
        divide(A, rs, ap);
#pragma unroll
        for (int n = n0; n < n0 + G; ++n) {
          const double xn = X[0][n] - omega * (X[0][n] - rs[n - n0]);
          X[0][n] = xn;
          T[own(t) + plane(n) * TP] = xn;
          xo[plane(n) * 128] = xn;
        }
      }
    }
  }
  if (SWEEP) {
    __syncthreads();
    const Around N(T, 1);
    const auto& A1 = A.again();
#pragma unroll
    for (int n0 = 0; n0 < NC; n0 += G) {
      double rs[G], ap[G];
#pragma unroll
      for (int n = n0; n < n0 + G; ++n) {
        const int s = HALF_CELLS + plane(n) * 128;
        const K7 a = A1.at(1, n);
        rs[n - n0] = minus_neighbours(b[s], a, N.at(n, X[0]));
        ap[n - n0] = a.p;
      }
      divide(A, rs, ap);
#pragma unroll
      for (int n = n0; n < n0 + G; ++n) {
        const double xn = X[1][n] - omega * (X[1][n] - rs[n - n0]);
        T[own(t) + TH + plane(n) * TP] = xn;
        xo[HALF_CELLS + plane(n) * 128] = xn;
      }
    }
  }
}

struct __align__(128) Smem {
  double b[2][BLOCK_CELLS];  // right-hand side of the current / next block
  double tile[TT];
  Record rec[3];             // records of the current block and the two after it
  double ws[2][16];
  uint64_t rbar[3], bbar[2];
  int abort_flag, last, next[2];
};
static_assert(2 * (sizeof(Smem) + 1024) <= 228 * 1024, "two CTAs per SM");

// STALL (test hook): no b for a CTA's third block, its second where no CTA has
// three, its only one where none has two.
template <bool RES, bool SWEEP, int SRC, int PER_SM, bool STALL>
__global__ void __launch_bounds__(NT, PER_SM)
rbgs_block_kernel(const __grid_constant__ KCtx C, const double* xin,
                  double* __restrict__ xout, const double* __restrict__ A,
                  const double* __restrict__ bvec, const double* gst,
                  double* __restrict__ gout, double omega, double* __restrict__ partials,
                  SolveState* st, int fin, int iter,
                  const int32_t* __restrict__ order) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  double* T = S.tile;
  const int tid = threadIdx.x, nb = C.nb, grid = gridDim.x;
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) async::mbar_init(&S.rbar[k], REC_THREADS);
    for (int k = 0; k < 2; ++k) async::mbar_init(&S.bbar[k], 1);
    S.abort_flag = 0;
    async::fence_mbar_init();
  }
  __syncthreads();
  auto block_of = [&](int item) { return item >= nb ? -1 : order ? __ldg(order + item) : item; };
  auto fetch_rec = [&](int b, int m) {  // record of the CTA's m-th block
    if (b >= 0 && tid < REC_THREADS)
      fetch_record(S.rec[m % 3], &S.rbar[m % 3], C.nbr, C.urec, b);
  };
  auto stalled = [&](int m) { return STALL && m == (nb > 2 * grid ? 2 : nb > grid ? 1 : 0); };
  auto fetch_b = [&](int b, int m) {  // b of the CTA's m-th block
    if (b >= 0 && tid == 32 && !stalled(m)) {
      async::mbar_expect_tx(&S.bbar[m & 1], BLOCK_CELLS * 8);
      async::bulk_g2s(S.b[m & 1], bvec + (size_t)b * BLOCK_CELLS, BLOCK_CELLS * 8, &S.bbar[m & 1]);
    }
  };
  auto wait_rec = [&](int m) {
    return async::mbar_wait(&S.rbar[m % 3], (m / 3) & 1, &S.abort_flag, ROLE_RBGS,
                                   C.wait_ns);
  };
  // The first two blocks of a CTA are its own; those after them are handed
  // out as CTAs free up (thread 0 draws one a block ahead).  Records and b do
  // not depend on the pass before this one.
  int blk = block_of(blockIdx.x), next = block_of(grid + blockIdx.x);
  fetch_rec(blk, 0);
  fetch_b(blk, 0);
  fetch_rec(next, 1);
  // a limit of 0 lets nothing be waited for: the pass gives up here, whether or
  // not the record happens to have landed by the time a wait would look
  bool ok = blk < 0 || C.wait_ns != 0;
  std::conditional_t<PER_SM == 1, Held, Varied> AV(
      A + (size_t)blk * 7 * BLOCK_CELLS + slot(tid),
      PER_SM == 1 && __ldg(C.urec + (size_t)blk * 8 + 7) == 0.0);
  pdl_release();
  pdl_wait();
  const bool skip = *((volatile const int32_t*)&st->done) != 0;  // used after the first wait
  const bool draw = 2 * grid < nb;
  int drawn = nb;
  if (tid == 0 && draw) drawn = 2 * grid + (int)atomicAdd(&st->work, 1u);
  ok = ok && (blk < 0 || wait_rec(0));
  int n = 0;
  if (skip) blk = -1;  // the copies in flight are drained below
  double X[2][NC];
  Staging<SRC, Written> L;  // the pass before may still be writing while this one starts
  if (ok && blk >= 0) L.load(X, xin, blk, S.rec[0].nbr, gst);
  while (blk >= 0) {
    const int k = n & 1;
    const Record& R = S.rec[n % 3];
    if (SWEEP && n > 0) __syncthreads();  // the pushes of the block before are out of the tile
    if (ok) L.put(T, X, xin, blk, R.nbr, C.bc, C.dx);
    if (tid == 0) S.next[k] = block_of(drawn);
    ok = ok && async::mbar_wait(&S.bbar[k], (n >> 1) & 1, &S.abort_flag, ROLE_RBGS,
                                       C.wait_ns);
    ok = ok && (next < 0 || wait_rec(n + 1));
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    const int after = S.next[k];
    // buffers whose last reads were before the previous block's barriers
    fetch_b(next, n + 1);
    fetch_rec(after, n + 2);
    if (next >= 0) {
      const Record& Q = S.rec[(n + 1) % 3];
      if (tid == 64) async::prefetch_l2(xin + (size_t)next * BLOCK_CELLS, BLOCK_CELLS * 8);
      if (tid == 96 && Q.u[7] == 0.0)
        async::prefetch_l2(A + (size_t)next * 7 * BLOCK_CELLS, 7 * BLOCK_CELLS * 8);
    }
    if (tid == 0 && after >= 0) drawn = 2 * grid + (int)atomicAdd(&st->work, 1u);
    const double* bb = S.b[k] + slot(tid);
    double* xo = SWEEP ? xout + (size_t)blk * BLOCK_CELLS + slot(tid) : nullptr;
    double acc[2][2] = {};
    if (R.u[7] != 0.0)
      rbgs_cells<RES, SWEEP>(T, X, Uniform(R.u), bb, xo, omega, acc);
    else
      rbgs_cells<RES, SWEEP>(T, X, AV, bb, xo, omega, acc);
    // the warp sums alternate between two buffers: block n + 2 writes its
    // buffer after block n + 1's barrier, which thread 0 passes after its read
    if (RES) warp_sums(acc, S.ws[k]);
    async::fence_proxy_async();  // b[k] is refilled by a bulk copy after the barriers
    __syncthreads();
    // the next block's loads are in flight over the pushes
    if (PER_SM > 1 && next >= 0) L.load(X, xin, next, S.rec[(n + 1) % 3].nbr, gst);
    if (RES && tid == 0) __stcg(partials + blk, block_sum(S.ws[k]));
    if (SWEEP && gout) push_guides(T, R.nbr, gout);
    if constexpr (PER_SM == 1)
      break;  // its only block
    else if (next >= 0)
      AV.Ab = A + (size_t)next * 7 * BLOCK_CELLS + slot(tid);
    blk = next;
    next = after;
    ++n;
  }
  if (!ok || skip) {
    // Copies that may still be on their way into this CTA's shared memory:
    // block n's and n + 1's records and block n's b (a step issues the ones
    // after them only once its waits have succeeded).
    if (tid == 0) {
      bool drained = stalled(n) || async::mbar_drain(&S.bbar[n & 1], (n >> 1) & 1);
      drained = async::mbar_drain(&S.rbar[n % 3], (n / 3) & 1) && drained;
      if (next >= 0) drained = async::mbar_drain(&S.rbar[(n + 1) % 3], ((n + 1) / 3) & 1) && drained;
      if (!ok) {
        atomicOr(&st->timeout_where, ROLE_RBGS | (drained ? 0 : async::ROLE_DRAIN));
        atomicExch(&st->status, 3);
        atomicExch(&st->done, 1);
      }
    }
    return;
  }
  if (!RES && !draw) return;
  if (tid == 0) {
    __threadfence();
    S.last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!S.last) return;
  __threadfence();
  double total = 0.0;
  if (RES) total = cross_block_sum(partials, nb, S.ws[0]);
  if (tid == 0) {
    if (RES) finalize(st, total, fin, iter);
    st->work = 0;
    st->ticket = 0;
    __threadfence();
  }
}

template <bool R, bool W, int G, bool STALL = false>
void launch_one(cudaStream_t s, const KCtx& C, const double* xin, double* xout, const double* A,
                const double* b, const double* gst, double* gout, double omega, double* partials,
                SolveState* st, int fin, int iter, bool pdl, const int32_t* order) {
  const int sms = sm_count();
  // with a block per SM at most, the registers of a second CTA hold a varied
  // block's colour-1 coefficients instead (72 blocks: 13.7 us a pass, 16.8)
  const bool one = C.nb <= sms;
  const int grid = std::min(C.nb, 2 * sms);
  auto kernel = one ? rbgs_block_kernel<R, W, G, 1, STALL> : rbgs_block_kernel<R, W, G, 2, STALL>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
  launch_dep(kernel, grid, NT, sizeof(Smem), s, pdl, C, xin, xout, A, b, gst, gout, omega,
             partials, st, fin, iter, order);
}

}  // namespace

int sm_count() {
  static std::mutex mu;
  static int count[64];
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  int local = 0;
  int& n = dev >= 0 && dev < 64 ? count[dev] : local;
  if (n == 0) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

// With up to twelve blocks per SM the varied blocks, which take three times as
// long, go first so that none is left for the end; with more the order mixes
// them, so that one CTA's coefficient loads overlap the other's arithmetic.
// us per pass, varied first / block order, by blocks per SM: 2.2: 24.0 / 29.0,
// 3.7: 34.4 / 35.8, 4.8: 45.8 / 53.7, 7.9: 59.5 / 68.6, 11.3: 74.5 / 77.9,
// 15.3: 107.6 / 106.2, 21: 108.2 / 105.5, 32: 158.4 / 147.9.
int rbgs_ordered_blocks() { return 12 * sm_count(); }

void launch_rbgs_stalled(cudaStream_t s, const KCtx& C, bool ring, const double* xin,
                         double* xout, const double* A, const double* b, const double* gin,
                         double* gout, double omega, double* partials, SolveState* st,
                         const int32_t* order) {
  if (ring)
    launch_rbgs_ring(s, C, false, true, xin, xout, A, b, gin, omega, partials, st, FIN_RBGS, 0,
                     false, true);
  else
    launch_one<false, true, tile::STORED, true>(s, C, xin, xout, A, b, gin, gout, omega, partials,
                                                st, FIN_RBGS, 0, false, order);
}

void launch_rbgs(cudaStream_t s, const KCtx& C, bool res, bool sweep, const double* xin,
                 double* xout, const double* A, const double* b, RbgsGuides from,
                 const double* gin, double* gout, double omega, double* partials, SolveState* st,
                 int fin, int iter, bool pdl, const int32_t* order) {
#define RBGS(R, W, G) \
  launch_one<R, W, G>(s, C, xin, xout, A, b, gin, gout, omega, partials, st, fin, iter, pdl, order)
  // stored guides are those before a solve's first sweep, pushed ones those of
  // the sweep before
  if (res && sweep)
    from == RbgsGuides::PUSHED ? RBGS(true, true, tile::PUSHED) : RBGS(true, true, tile::PULL);
  else if (sweep)
    from == RbgsGuides::STORED ? RBGS(false, true, tile::STORED) : RBGS(false, true, tile::PULL);
  else
    from == RbgsGuides::STORED ? RBGS(true, false, tile::STORED)
    : from == RbgsGuides::PULL ? RBGS(true, false, tile::PULL)
                               : RBGS(true, false, tile::PUSHED);
#undef RBGS
}

}  // namespace ffvgpu
