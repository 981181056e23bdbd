// ffvgpu_tile.cuh -- one 16^3 block staged in shared memory with its first
// guide layer, the per-block records a kernel reads ahead, and the guides a
// kernel pushes to its block's neighbours; used by the FP64 stencil kernels.
//
// Two or more CTAs of these kernels share an SM, so that one CTA's loads
// overlap another's arithmetic and barriers; inside a CTA the staging issues
// all its loads before it uses any.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "ffvgpu_async.cuh"
#include "ffvgpu_internal.cuh"

namespace ffvgpu {
namespace tile {

// Per colour and plane k in -1..16: rows j = -1..16 of 8 values (i >> 1), then
// 16 x-face guides, one per row -- of the two guide cells beside a row one has
// each colour, so a row of one colour has just one of them, west (i = -1) when
// (j + k + 1) & 1 is the colour, else east (i = 16).  Every neighbour of a cell
// is at a fixed offset in its plane, and rows of 8 put the two rows a half-warp
// reads on disjoint banks.
constexpr int TR = 8, TG = 18 * TR, TP = TG + 16, TH = 18 * TP, TT = 2 * TH;

// Tile position of the guide cell at (face, p = u + 16 v).
__device__ __forceinline__ int guide_at(int face, int p) {
  const int u = p & 15, v = p >> 4, out = (face & 1) ? 16 : -1, c = (u + v + out) & 1;
  return c * TH + (face < 2   ? (v + 1) * TP + TG + u
                   : face < 4 ? (v + 1) * TP + (out + 1) * TR + (u >> 1)
                              : (out + 1) * TP + (v + 1) * TR + (u >> 1));
}
// A CTA of 256 threads holds one block.  Thread t has (j, i / 2) = t & 127 and
// of the planes k the pairs 4 m + 2 h + e (h = t >> 7; e = 0, 1; m = 0..3), both
// colours, in registers: X[c][2 m + e] is storage slot slot(t) + c * 2048 +
// (4 m + e) * 128.  So one z neighbour and one x neighbour of a cell are the
// thread's own; the others come from the tile.  The block tree's virtual thread
// t & 127 + 128 (2 h + e) sums the cells (m = 0..3) of one e.
constexpr int NT = 256, NC = 8;
__device__ __forceinline__ int slot(int t) { return (t >> 7) * 256 + (t & 127); }
__device__ __forceinline__ int own(int t) {  // tile position of (c = 0, m = 0, e = 0)
  return (1 + 2 * (t >> 7)) * TP + TR + (t & 127);
}
__host__ __device__ constexpr int plane(int n) { return 4 * (n >> 1) + (n & 1); }  // cell n of X[c]

// Where a block's guide layer comes from: stored beside the field (gst), the
// neighbours' interiors by the exchange rules, or those with what the kernel
// before pushed (gst: the guide buffer) in place of the scattered reads.
enum Source { STORED, PULL, PUSHED };
__host__ __device__ constexpr bool is_pushed(int f, int kind) {
  return kind >= NB_COARSE || (kind == NB_SAME && f < 2);
}

// Loads of a block's interior and guide layer into registers, all in flight
// together but (PULL) those of 2:1 faces.  LD: how x and gst are read (Written in
// kernels launched as programmatic dependents of the one that wrote them).
template <int SRC, typename LD>
struct Staging {
  double g[3][2];
  __device__ __forceinline__ void load(double (&X)[2][NC], const double* x, int blk,
                                       const FaceNbr* nb, const double* gst) {
    const int t = threadIdx.x, p = t & 127;
    const double* xb = x + (size_t)blk * BLOCK_CELLS + slot(t);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int n = 0; n < NC; ++n) X[c][n] = LD::ld(xb + c * HALF_CELLS + plane(n) * 128);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int f = 2 * r + (t >> 7), kind = nb[f].kind;
      if (SRC == STORED || (SRC == PUSHED && is_pushed(f, kind))) {
        const double* gs = gst + ((size_t)blk * 6 + f) * FACE_CELLS + p;
        g[r][0] = LD::ld(gs);
        g[r][1] = LD::ld(gs + 128);
      } else if (kind <= NB_SAME) {
        const bool outer = kind == NB_OUTER;
        const double* s = x + (size_t)(outer ? blk : nb[f].id[0]) * BLOCK_CELLS;
        g[r][0] = LD::ld(s + face_slot(f, p, outer));
        g[r][1] = LD::ld(s + face_slot(f, p + 128, outer));
      }
    }
  }
  __device__ __forceinline__ void put(double* T, const double (&X)[2][NC], const double* x,
                                      int blk, const FaceNbr* nb, const BCSet& bc,
                                      const double* __restrict__ dxs) {
    const int t = threadIdx.x, p = t & 127;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int n = 0; n < NC; ++n) T[own(t) + c * TH + plane(n) * TP] = X[c][n];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int f = 2 * r + (t >> 7);
      if (SRC != STORED) {
        const int kind = nb[f].kind;
        if (kind == NB_OUTER) {
          const double dx = __ldg(dxs + blk);
          g[r][0] = outer_guide(g[r][0], f, bc, dx);
          g[r][1] = outer_guide(g[r][1], f, bc, dx);
        } else if (SRC == PULL && kind != NB_SAME) {
          guide_pair<LD>(x, blk, f, p, p + 128, nb[f], bc, 0.0, g[r][0], g[r][1]);
        }
      }
      T[guide_at(f, p)] = g[r][0];
      T[guide_at(f, p + 128)] = g[r][1];
    }
  }
};

// ---------------------------------------------------------------------------
// Pushed guides.  A kernel that leaves a block's new values in its tile also
// writes the guides its neighbours will need that they could not read well:
// those of x faces (one 8-byte value per 64-byte row) and of 2:1 faces (eight
// scattered loads per guide).  They go into the neighbour's slot of a guide
// buffer [block][face][p], which the next kernel reads coalesced.  A warp's load
// of an x face touches 32 lines of the 28 KB that two CTAs' shared memory leaves
// to L1, so those loads, and the interior's behind them, wait for lines: reading
// all guides from the neighbours made an RBGS pass of the level-5 sphere grid
// 176 us, pushing these 147 us (without any guides 125 us).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double cell(const double* T, int i, int j, int k) {
  return T[((i + j + k) & 1) * TH + (k + 1) * TP + (j + 1) * TR + (i >> 1)];
}
__device__ __forceinline__ void cells8(const double* T, int i, int j, int k, double (&a)[8]) {
  a[0] = cell(T, i, j, k);
  a[1] = cell(T, i + 1, j, k);
  a[2] = cell(T, i, j + 1, k);
  a[3] = cell(T, i, j, k + 1);
  a[4] = cell(T, i, j + 1, k + 1);
  a[5] = cell(T, i + 1, j, k + 1);
  a[6] = cell(T, i + 1, j + 1, k);
  a[7] = cell(T, i + 1, j + 1, k + 1);
}
// Every thread of the CTA, with the new values of both colours in the tile.
__device__ __forceinline__ void push_guides(const double* T, const FaceNbr* nb,
                                            double* __restrict__ G) {
  const int t = threadIdx.x;
#pragma unroll 1
  for (int f = 0; f < 6; ++f) {
    const int kind = nb[f].kind;
    if (!is_pushed(f, kind)) continue;
    if (kind == NB_SAME) {
      G[((size_t)nb[f].id[0] * 6 + (f ^ 1)) * FACE_CELLS + t] =
          cell(T, (f & 1) ? 15 : 0, t & 15, t >> 4);
    } else if (kind == NB_COARSE) {  // a quarter of the coarse neighbour's face
      if (t < 64) {
        FaceNbr q;
        q.id[0] = q.id[1] = q.id[2] = q.id[3] = 0;
        const int p = ((t & 7) + 8 * nb[f].so_u) + 16 * ((t >> 3) + 8 * nb[f].so_v);
        FineGuide g;
        g.at(f ^ 1, p, q);
        cells8(T, g.i, g.j, g.k, g.a);
        G[((size_t)nb[f].id[0] * 6 + (f ^ 1)) * FACE_CELLS + p] = g.value();
      }
    } else {  // the faces of four fine neighbours
#pragma unroll 1
      for (int h = 0; h < 4; ++h) {
        FaceNbr q;
        q.id[0] = 0;
        q.so_u = h & 1;
        q.so_v = h >> 1;
        CoarseGuide g;
        g.at(f ^ 1, t, q);
        cells8(T, g.i, g.j, g.k, g.a);
        G[((size_t)nb[f].id[h] * 6 + (f ^ 1)) * FACE_CELLS + t] = g.value();
      }
    }
  }
}

// The neighbours of a thread's cells of colour c.  The x neighbour beside the
// thread's own one is east of the cell where the cell's i is odd, else west;
// i alternates with k, so two pointers serve all planes.
struct Around {
  const double *o, *x0, *x1;  // own position in the other colour; x neighbour, even and odd k
  bool odd0;                  // i is odd at even k
  __device__ __forceinline__ Around(const double* T, int c) {
    const int t = threadIdx.x, ih = t & 7, j = (t >> 3) & 15;
    o = T + own(t) + (1 - c) * TH;
    odd0 = ((j + c) & 1) != 0;
    const double* g = T + (1 + 2 * (t >> 7)) * TP + (1 - c) * TH + TG + j;
    x0 = (odd0 ? ih == 7 : ih == 0) ? g : o + (odd0 ? 1 : -1);
    x1 = (odd0 ? ih == 0 : ih == 7) ? g : o + (odd0 ? -1 : 1);
  }
  // cell n; O: the thread's cells of the other colour
  __device__ __forceinline__ Nbrs at(int n, const double (&O)[NC]) const {
    const int e = n & 1, d = plane(n) * TP;
    const bool odd = odd0 != (e != 0);
    const double x = e ? x1[d] : x0[d];
    Nbrs v;
    v.w = odd ? O[n] : x;
    v.e = odd ? x : O[n];
    v.s = o[d - TR];
    v.n = o[d + TR];
    v.b = e ? O[n - e] : o[d - TP];
    v.t = e ? o[d + TP] : O[n + 1 - e];
    return v;
  }
};

// What a kernel reads of a block before its fields: the six face records and
// the uniform record (Ap..At of cell 0, then the flag).
struct __align__(16) Record {
  FaceNbr nbr[6];
  double u[8];
};
static_assert(sizeof(FaceNbr) * 6 == 192 && sizeof(Record) == 256, "copied 16 bytes a thread");
constexpr int REC_THREADS = sizeof(Record) / 16;

// Brings block blk's record into R, completing a phase of *bar (initialised
// for REC_THREADS arrivals): called by threads 0 .. REC_THREADS - 1.
__device__ __forceinline__ void fetch_record(Record& R, uint64_t* bar, const FaceNbr* nbr,
                                             const double* urec, int blk) {
  const int t = threadIdx.x;
  const char* src = t < 12 ? reinterpret_cast<const char*>(nbr + (size_t)blk * 6) + 16 * t
                           : reinterpret_cast<const char*>(urec + (size_t)blk * 8) + 16 * (t - 12);
  char* dst = reinterpret_cast<char*>(&R) + 16 * t;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(async::sa(dst)), "l"(src)
               : "memory");
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(async::sa(bar))
               : "memory");
}

// The seven coefficients of one cell: from the uniform record (in registers)
// or from A's rows, Ab + a * 4096 + s.
struct K7 {
  double p, w, e, s, n, b, t;
};
__device__ __forceinline__ K7 uniform_coefs(const double* u) {
  K7 k;
  k.p = u[0]; k.w = u[1]; k.e = u[2]; k.s = u[3]; k.n = u[4]; k.b = u[5]; k.t = u[6];
  return k;
}
__device__ __forceinline__ K7 stream_coefs(const double* __restrict__ Ab, int s) {
  K7 k;
  k.p = __ldg(Ab + s);
  k.w = __ldg(Ab + 1 * BLOCK_CELLS + s);
  k.e = __ldg(Ab + 2 * BLOCK_CELLS + s);
  k.s = __ldg(Ab + 3 * BLOCK_CELLS + s);
  k.n = __ldg(Ab + 4 * BLOCK_CELLS + s);
  k.b = __ldg(Ab + 5 * BLOCK_CELLS + s);
  k.t = __ldg(Ab + 6 * BLOCK_CELLS + s);
  return k;
}
// b - (the six neighbour terms), in the reference's order (bils.f90:57-108).
__device__ __forceinline__ double minus_neighbours(double b, const K7& k, const Nbrs& v) {
  return b - k.w * v.w - k.e * v.e - k.s * v.s - k.n * v.n - k.b * v.b - k.t * v.t;
}

// Quotients by one divisor, correctly rounded like '/': from y = RN(1 / d),
// q0 = a y is within two ulps, a first correction q1 = q0 + (a - q0 d) y makes
// it faithful, and a second gives RN(a / d) (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990: a
// faithful quotient corrected once with the rounded reciprocal is correctly
// rounded).  Five FP64 operations without a branch, where '/' takes more than
// twice as many instructions and a branch per cell.  Valid while nothing on
// the way can under- or overflow; ok(a) tests that, and the caller divides
// where it fails (zeros, whose sign the corrections would lose, among them).
struct Divisor {
  double d, y;
  bool normal;
  __device__ __forceinline__ explicit Divisor(double dv) : d(dv), y(1.0 / dv) {
    const int e = (__double2hiint(dv) >> 20) & 0x7ff;
    normal = e > 1023 - 250 && e < 1023 + 250;
  }
  __device__ __forceinline__ bool ok(double a) const {
    const unsigned h = __double2hiint(a) & 0x7fffffff;
    return h - ((1023u - 650u) << 20) < (1300u << 20);
  }
  __device__ __forceinline__ double operator()(double a) const {
    const double q0 = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-q0, d, a), y, q0);
    return __fma_rn(__fma_rn(-q1, d, a), y, q1);
  }
};

// Warp sums of the block tree: acc[colour][e] are the two colour sums of
// virtual thread t & 127 + 128 (2 h + e).
__device__ __forceinline__ void warp_sums(const double (&acc)[2][2], double* ws) {
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    double v = acc[0][e] + acc[1][e];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    const int t = threadIdx.x;
    if ((t & 31) == 0) ws[((t & 127) >> 5) + 4 * (2 * (t >> 7) + e)] = v;
  }
}
__device__ __forceinline__ double block_sum(const double* ws) {
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < 16; ++w) s += ws[w];
  return s;
}
// Cross-block sum over n per-block partials in order, one lane per thread (the
// layout header's tree); every thread calls it, thread 0 has the result.
__device__ __forceinline__ double cross_block_sum(const double* part, int n, double* ws) {
  double s = 0.0;
#pragma unroll 8
  for (int b = threadIdx.x; b < n; b += NT) s += __ldcg(part + b);
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  double total = 0.0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int w = 0; w < 8; ++w) total += ws[w];
  return total;
}

// Programmatic dependent launch: the kernels after this one on the stream may
// start their prologue; wait until the kernels before it are complete.
__device__ __forceinline__ void pdl_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace tile

// Launches a kernel, as a programmatic dependent of the kernel before it on
// the stream when pdl is set (that kernel and this one must both run
// tile::pdl_wait in every thread before they touch what an earlier kernel wrote).
template <typename... P, typename... A>
inline void launch_dep(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s,
                       bool pdl, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace ffvgpu
