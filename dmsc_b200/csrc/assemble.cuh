// Output assembly on the device (cpu/workspace.hxx:86-365), for a batch.
//
// Per image: surviving extrema keep their ascending-cell-id order; surviving
// saddles are listed in minima-sweep order; e_min rows follow the minima sweep
// and e_max rows the maxima sweep, which is the reverse of the minima sweep
// for the same saddles (cpu/arcs_topology.hxx:142). Internal side 0 is the
// faces, side 1 the vertices; in the primal the faces are the maxima, in the
// dual the minima (workspace.hxx:322-362), so every side's per-image output
// goes to the array that image's orientation selects, at an offset the host
// computed from the per-image sizes. All written ids are image-local.
#pragma once

#include "common.cuh"

namespace dmsc {

// Destination of one side's per-image output: the array picked by the
// image's orientation, at the image's offset in it.
struct Route {
  int* primal;
  int* dual;
  const int* off;  // [B]
  __device__ __forceinline__ int* at(bool d, int b) const {
    int* p = d ? dual : primal;
    return p ? p + off[b] : nullptr;
  }
};
struct RouteF {
  float* primal;
  float* dual;
  const int* off;
  __device__ __forceinline__ float* at(bool d, int b) const {
    float* p = d ? dual : primal;
    return p ? p + off[b] : nullptr;
  }
};

// Surviving extrema of both sides (blockIdx.y), image-local cell ids, into the
// routed point lists.
struct PointSide {
  int n;
  const uint8_t* alive;
  const int* rank;
  const int* alive_base;
  const int2* key;
  const int* ext_img;
  Route out;
};

__global__ void points_kernel(PointSide F, PointSide V, Imgs I) {
  const PointSide& S = blockIdx.y ? V : F;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= S.n || !S.alive[x]) return;
  const int b = S.ext_img[x];
  int* dst = S.out.at(I.dual[b], b);
  if (dst) dst[S.rank[x] - S.alive_base[b]] = S.key[x].y - 4 * I.idx_base[b];
}

// Image, global cell and list index of a survivor, in output order.
struct SurvHead {
  int img, cell, sad, pad;
};

// Two 32-bit counts in one word: side 0 in the low half, side 1 in the high
// half (a total of 2^31 or more fails the call).
__device__ __forceinline__ unsigned long long pack2(unsigned f, unsigned v) { return f | (unsigned long long)v << 32; }
__device__ __forceinline__ int half_of(unsigned long long p, int sd) { return (int)(unsigned)(sd ? p >> 32 : p); }

// Everything the host reads back for the sizes, straight to the mapped area:
// the integer bases (first min, saddle, max, survivor, alive ranks and e rows
// of both sides; B + 1 entries each), the geometry starts of both sides and
// the status word. Also leaves the e row and geometry starts on the device.
__global__ void sizes_kernel(int B, const int* __restrict__ surv_base, const unsigned long long* __restrict__ lens,
                             const unsigned long long* __restrict__ rows, const unsigned long long* __restrict__ total,
                             int* __restrict__ bases, long long* __restrict__ gbase0, long long* __restrict__ gbase1,
                             const unsigned* __restrict__ status, int* __restrict__ rb_int,
                             long long* __restrict__ rb_long, unsigned* __restrict__ rb_status) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > B) return;
  const int n = B + 1, f = surv_base[b];
#pragma unroll
  for (int k = 0; k < 6; ++k) rb_int[k * n + b] = bases[k * n + b];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    bases[(6 + sd) * n + b] = half_of(rows[f], sd);
    rb_int[(6 + sd) * n + b] = half_of(rows[f], sd);
    const long long g = b < B ? (long long)half_of(lens[f], sd) : (long long)total[sd];  // the exact total
    (sd ? gbase1 : gbase0)[b] = g;
    rb_long[sd * n + b] = g;
  }
  if (b == 0) *rb_status = *status;
}

// e rows of one survivor (cpu/workspace.hxx:175-195, 197-219) from the out
// ranks of its ends' roots (-1: the void; a thresholded root is always an
// alive extremum, so it always has an out rank): up to two ends.
__device__ __forceinline__ int erow_ends(int r1, int r2, int* o1, int* o2) {
  int n = 0;
  if (r1 != -1) {
    *o1 = r1;
    n = 1;
  }
  if (r1 != r2 && r2 != -1) {
    if (n == 0)
      *o1 = r2;
    else
      *o2 = r2;
    n++;
  }
  return n;
}

// Per-survivor outputs of both sides: the saddle points, persistence, pairs,
// e rows and the CSR offsets of the arcs (cpu/workspace.hxx:247-287: offsets[0]
// = 0, offsets[k+1] = end of survivor k, arc_offsets[k] = end of its first
// arc), all image-local, in the arrays that the image's orientation selects.
struct SurvSideOut {
  RouteF p;
  Route pp, e, off, aoff;
  const int* alive_base;   // [B + 1]
  const long long* gbase;  // [B + 1]
  const int4* out;         // [nsurv] ranks of the ends' roots, persistence bits, rank of the pair's root
  const int4* arc;         // [nsurv] arc ends and raw-arc lengths
  const int4* fin;         // [nsurv] chain lengths and roots of the final arcs (nullptr: no arcs)
};

__global__ void __launch_bounds__(256) survivor_outputs_kernel(int nsurv, Imgs I, const int* __restrict__ surv_base,
                                                               const SurvHead* __restrict__ head,
                                                               const unsigned long long* __restrict__ lens,
                                                               const unsigned long long* __restrict__ rows,
                                                               int* __restrict__ sad_pts, SurvSideOut F,
                                                               SurvSideOut V) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < I.B) {  // one leading zero per image
#pragma unroll
    for (int sd = 0; sd < 2; ++sd)
      if (int* o = (sd ? V : F).off.at(I.dual[i], i)) o[0] = 0;
  }
  if (i >= nsurv) return;
  const int2 ic = *reinterpret_cast<const int2*>(head + i);
  const int b = ic.x;
  const bool d = I.dual[b];
  const int first = surv_base[b], last = surv_base[b + 1], li = i - first;
  if (sad_pts) sad_pts[i] = ic.y - 4 * I.idx_base[b];
  const unsigned long long r0 = rows[i], r1 = rows[i + 1];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    const SurvSideOut& S = sd ? V : F;
    const int4 r = S.out[i];
    const int ab = S.alive_base[b];
    if (float* p = S.p.at(d, b)) p[li] = __int_as_float(r.z);
    if (int* pp = S.pp.at(d, b)) pp[li] = r.w >= 0 ? r.w - ab : -1;
    if (int* e = S.e.at(d, b)) {
      int x = 0, y = 0;
      const int n = erow_ends(r.x, r.y, &x, &y);
      // the vertex side's rows follow the minima sweep (this order), the face
      // side's the maxima sweep, its reverse
      const int o = sd ? half_of(r0, 1) - half_of(rows[first], 1) : half_of(rows[last], 0) - half_of(r1, 0);
      if (n >= 1) {
        e[2 * o] = li;
        e[2 * o + 1] = x - ab;
      }
      if (n == 2) {
        e[2 * o + 2] = li;
        e[2 * o + 3] = y - ab;
      }
    }
    if (!S.fin) continue;
    const int g = (int)S.gbase[b];
    if (int* o = S.off.at(d, b)) o[li + 1] = half_of(lens[i + 1], sd) - g;
    if (int* a = S.aoff.at(d, b)) a[li] = half_of(lens[i], sd) - g + S.arc[i].z + S.fin[i].x;
  }
}

}  // namespace dmsc
