// ffvgpu_instance.cuh -- instances on the device: a CTA's list of live blocks
// and the mixed form's finalisers.
#pragma once
#include <cfloat>
#include <cuda_runtime.h>

#include "ffvgpu_internal.cuh"
#include "ffvgpu_mixed.h"

namespace ffvgpu {

// Per-instance finalisers, run by the CTA that finishes an instance's last
// block.
__device__ inline void mx_finalize(SolveState* S, const double* t, int fin) {
  switch (fin) {
    case FIN_MX_INIT:
      S->bb = t[0];
      if (fabs(t[0]) < (double)FLT_MIN) {  // FFVILS.h:822-826
        S->residual = 0.0;
        S->count = 0;
        S->done = 1;
        break;
      }
      S->rr1 = t[1];
      if (fabs(t[1]) < (double)FLT_MIN) {  // FFVILS.h:847-851 at count = 1
        S->residual = t[1];
        S->count = 0;
        S->done = 1;
        break;
      }
      S->rr0 = 1.0;
      S->alpha = 0.0;
      S->gamma = 1.0;
      S->iter = 1;
      S->cycle = 1;
      S->next_restart = (S->drop > 0.0) ? resid_of(t[1], t[0]) * S->drop : -1.0;
      S->best = resid_of(t[1], t[0]);
      break;
    case FIN_MX_ALPHA:
      S->qp = t[0];
      S->alpha = S->rr1 / t[0];
      break;
    case FIN_MX_GAMMA:
      S->ts = t[0];
      S->gamma = t[0] / t[1];
      break;
    case FIN_MX_UPDATE: {
      const int n = S->iter;
      const double res = resid_of(t[0], S->bb);  // IsConverged, FFVILS.h:24-47
      S->rr = t[0];
      S->residual = res;
      if (S->hist) S->hist[n - 1] = res;
      S->count = n;
      if (res <= S->eps) {
        S->done = 1;
      } else if (isnan(res) || isinf(res)) {
        S->done = 1;
        S->status = 2;
      } else if (n >= S->count_max) {
        S->done = 1;
        S->count = S->count_max + 1;
      } else {
        S->rr0 = S->rr1;  // FFVILS.h:960
        S->cycle += 1;
        double rr1 = t[1];  // next iteration's DOT(r, r0)
        const bool dropped = S->next_restart > 0.0 && res <= S->next_restart;
        const bool grew = S->growth > 0.0 && res > S->growth * S->best;
        const bool aged = S->max_cycle > 0 && S->cycle > S->max_cycle;
        if (res < S->best) S->best = res;
        if (dropped || grew || aged) {
          // restart from the current r: r0 = r (written by the next
          // iteration's first sweep pass), so DOT(r, r0) = r.r
          if (S->drop > 0.0) S->next_restart = res * S->drop;
          S->best = res;
          S->rr0 = 1.0;
          S->alpha = 0.0;
          S->gamma = 1.0;
          S->cycle = 1;
          rr1 = t[0];
        }
        S->rr1 = rr1;
        if (fabs(rr1) < (double)FLT_MIN) {
          S->residual = rr1;
          S->count = 0;
          S->done = 1;
        } else {
          S->beta = rr1 / S->rr0 * S->alpha / S->gamma;
          S->iter = n + 1;
        }
      }
      break;
    }
  }
}

// A CTA's live items, found once per chunk instead of a block ahead: entry
// (block, instance | flags) of the items blockIdx.x + k gridDim.x whose
// instance is still solving (the done flags change between launches only).
constexpr int LIST_CAP = 1024;           // entries per chunk (8 KB of shared memory)
constexpr int LF_UNI = 1 << 30;          // the block is uniform (MixCtx::ucoef)
constexpr int LF_COPY = 1 << 29;         // its instance starts a cycle (p = r, r0 = r)
constexpr int LF_INST = LF_COPY - 1;

// Called by every thread of a CTA of PTS: fills list[0, *n) from the
// candidates from, from + gridDim.x, ... (CAP of them, in item order) and
// sets *next to the first candidate after them.
template <int MODE, bool FIRST, int PTS, int CAP = LIST_CAP>
__device__ inline void build_live_list(const MixCtx& C, int from, int n_act, int2* list, int* n,
                                int* next, int* wcount) {
  static_assert(CAP % PTS == 0, "whole rounds of candidates");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int base = 0;
  for (int r = 0; r < CAP / PTS; ++r) {
    const int it = from + (r * PTS + tid) * gridDim.x;
    int b = -1, e = 0;
    bool live = false;
    if (it < n_act) {
      b = C.active[it];
      const int i = C.inst.blk_inst[b];
      live = i >= 0 && !*((volatile const int32_t*)&C.inst.st[i].done);
      if (live) {
        e = i;
        if (C.ucoef[(size_t)b * 8 + 7] != 0.0) e |= LF_UNI;
        if (FIRST && MODE == 0 && C.inst.st[i].cycle == 1) e |= LF_COPY;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, live);
    if (lane == 0) wcount[warp] = __popc(m);
    __syncthreads();
    int off = base;
    for (int w = 0; w < warp; ++w) off += wcount[w];
    if (live) list[off + __popc(m & ((1u << lane) - 1u))] = make_int2(b, e);
    int tot = 0;
    for (int w = 0; w < PTS / 32; ++w) tot += wcount[w];
    base += tot;
    __syncthreads();  // wcount is refilled by the next round
  }
  if (tid == 0) {
    *n = base;
    *next = from + CAP * gridDim.x;
  }
  __syncthreads();
}

}  // namespace ffvgpu
