// Host-side check of how a stencil kernel stages a block (ffvgpu_tile.cuh):
// compiles Staging for the host, stages every block of a grid given on stdin
// (nb, then the neighbour table as kind id0 id1 id2 id3 so_u so_v per face)
// with the 256 threads run one after another, and compares the tile with
// guide_value and the stored guide layer.  Every read through the read-only
// path (__ldg) of x or of the guide buffer is counted.  Prints the wrong tile
// values, then the read-only reads with LD = Written and with LD = ReadOnly.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include <cuda_runtime.h>
#define __noinline__

using std::fabs;
using std::isinf;
using std::isnan;
using std::max;
using std::min;
using std::sqrt;
static std::vector<double> x, g;
static long readonly_reads = 0;
static inline bool within(const std::vector<double>& v, const double* p) {
  return !v.empty() && p >= v.data() && p < v.data() + v.size();
}
static inline double __ldg(const double* p) {
  if (within(x, p) || within(g, p)) ++readonly_reads;
  return *p;
}
// named by device functions of the headers that this check does not call
size_t __cvta_generic_to_shared(const void*);
int atomicOr(int*, int);
double __shfl_xor_sync(unsigned, double, int);
double __ldcg(const double*);
void __syncthreads();
int __double2hiint(double);
double __dmul_rn(double, double);
double __fma_rn(double, double, double);
static struct {
  int x;
} threadIdx;
#include "../../ffv-hc_b200/csrc/ffvgpu_tile.cuh"

using namespace ffvgpu;
using namespace ffvgpu::tile;

static std::vector<FaceNbr> nbr;
static std::vector<double> dxs;
static BCSet bc;

template <int SRC, typename LD>
static long stage_all(int nb) {
  long wrong = 0;
  std::vector<double> T(TT);
  std::vector<Staging<SRC, LD>> L(NT);
  static double X[NT][2][NC];
  for (int blk = 0; blk < nb; ++blk) {
    const FaceNbr* fn = &nbr[(size_t)blk * 6];
    for (threadIdx.x = 0; threadIdx.x < NT; ++threadIdx.x)
      L[threadIdx.x].load(X[threadIdx.x], x.data(), blk, fn, g.data());
    for (threadIdx.x = 0; threadIdx.x < NT; ++threadIdx.x)
      L[threadIdx.x].put(T.data(), X[threadIdx.x], x.data(), blk, fn, bc, dxs.data());
    for (int k = 0; k < 16; ++k)
      for (int j = 0; j < 16; ++j)
        for (int i = 0; i < 16; ++i)
          wrong += cell(T.data(), i, j, k) != x[(size_t)blk * BLOCK_CELLS + sidx(i, j, k)];
    const long before = readonly_reads;  // guide_value's own reads do not count
    for (int f = 0; f < 6; ++f)
      for (int p = 0; p < FACE_CELLS; ++p) {
        const bool stored = SRC == STORED || (SRC == PUSHED && is_pushed(f, fn[f].kind));
        const double want = stored ? g[((size_t)blk * 6 + f) * FACE_CELLS + p]
                                   : guide_value(x.data(), blk, f, p & 15, p >> 4, 1, fn[f], bc,
                                                 dxs[blk]);
        wrong += T[guide_at(f, p)] != want;
      }
    readonly_reads = before;
  }
  return wrong;
}

int main() {
  int nb;
  if (std::scanf("%d", &nb) != 1) return 2;
  nbr.resize((size_t)nb * 6);
  for (FaceNbr& F : nbr)
    if (std::scanf("%d %d %d %d %d %d %d", &F.kind, &F.id[0], &F.id[1], &F.id[2], &F.id[3],
                   &F.so_u, &F.so_v) != 7)
      return 2;
  uint64_t st = 88172645463325252ull;
  auto rnd = [&] {
    st ^= st << 13; st ^= st >> 7; st ^= st << 17;
    return (double)(int64_t)(st >> 11) * 1.0e-15 - 4.0;
  };
  x.resize((size_t)nb * BLOCK_CELLS);
  g.resize((size_t)nb * 6 * FACE_CELLS);
  dxs.resize(nb);
  for (double& v : x) v = rnd();
  for (double& v : g) v = rnd();
  for (double& v : dxs) v = rnd();
  for (int f = 0; f < 6; ++f) {
    bc.type[f] = f & 1;
    bc.value[f] = rnd();
  }
  const long wrong_w = stage_all<STORED, Written>(nb) + stage_all<PULL, Written>(nb) +
                       stage_all<PUSHED, Written>(nb);
  const long written = readonly_reads;
  readonly_reads = 0;
  const long wrong_r = stage_all<STORED, ReadOnly>(nb) + stage_all<PULL, ReadOnly>(nb) +
                       stage_all<PUSHED, ReadOnly>(nb);
  std::printf("%ld %ld %ld\n", wrong_w + wrong_r, written, readonly_reads);
  return 0;
}
