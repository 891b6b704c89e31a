// Persistence pairs as pixel pairs, and the deterministic backward scatter.
//
// A persistence value is the float32 difference of two input pixels: the
// value pixel of the saddle and the value pixel of the extremum that dies at
// it (cpu/persistence.hxx:82-104, 139-161), where a cell's value pixel is its
// highest vertex in the primal, its lowest in the dual, chosen under the
// (value, pixel id) order (cpu/cell_compare.hxx:33-87). On a field without
// ties the pairing is locally constant, so d p / d img is +1 on one pixel and
// -1 on the other; the backward pass scatters dL/dp onto those pixels.
#pragma once

#include "assemble.cuh"
#include "common.cuh"

namespace dmsc {

// Image-local value pixel of cell (t, y, x) (the pixel cell_value reads).
template <bool DUAL>
__device__ __forceinline__ int cell_pixel_g(const float* __restrict__ img, int t, int y, int x, int H, int W) {
  int cy[4], cx[4], n = 0;
  if (t == 0) {
    cy[n] = y;
    cx[n++] = x;
  } else if (t == 1) {
    if (x - 1 >= 0) {
      cy[n] = y;
      cx[n++] = x - 1;
    }
    if (x < W) {
      cy[n] = y;
      cx[n++] = x;
    }
  } else if (t == 2) {
    if (y - 1 >= 0) {
      cy[n] = y - 1;
      cx[n++] = x;
    }
    if (y < H) {
      cy[n] = y;
      cx[n++] = x;
    }
  } else {
    if (y - 1 >= 0 && x - 1 >= 0) {
      cy[n] = y - 1;
      cx[n++] = x - 1;
    }
    if (y - 1 >= 0 && x < W) {
      cy[n] = y - 1;
      cx[n++] = x;
    }
    if (y < H && x - 1 >= 0) {
      cy[n] = y;
      cx[n++] = x - 1;
    }
    if (y < H && x < W) {
      cy[n] = y;
      cx[n++] = x;
    }
  }
  int b = cy[0] * W + cx[0];
  float bv = __ldg(img + b);
  for (int k = 1; k < n; ++k) {
    int id = cy[k] * W + cx[k];
    float v = __ldg(img + id);
    if (value_greater<DUAL>(v, id, bv, b)) {
      b = id;
      bv = v;
    }
  }
  return b;
}

// Value pixel of global cell `cell` of image b.
__device__ __forceinline__ int value_pixel(const float* __restrict__ img_all, const Imgs& I, int b, int cell) {
  const int H = I.H[b], W = I.W[b], Nx = W + 1;
  const int lidx = (cell >> 2) - I.idx_base[b];
  const int y = row_of(I, b, lidx), x = lidx - y * Nx;
  const float* img = img_all + I.px_base[b];
  return I.dual[b] ? cell_pixel_g<true>(img, cell & 3, y, x, H, W) : cell_pixel_g<false>(img, cell & 3, y, x, H, W);
}

// Per surviving saddle of one side, in survivor order (the order of its p
// output), the image-local pixels entering its persistence with sign + and -
// (-1, -1 for a cycle, whose persistence is the constant -1). The sign
// follows persistence_kernel: p = saddle - extremum on the vertex side in the
// primal and on the face side in the dual, extremum - saddle otherwise.
__global__ void pair_pixels_kernel(int nsurv, bool faces, const int* __restrict__ surv_base, Imgs I,
                                   const float* __restrict__ img_all, const SurvHead* __restrict__ head,
                                   const int2* __restrict__ pp, const int2* __restrict__ ext_key, Route PLUS,
                                   Route MINUS) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsurv) return;
  const int4 h = *reinterpret_cast<const int4*>(head + i);
  const int b = h.x;
  const bool d = I.dual[b];
  const int li = i - surv_base[b];
  const int e = pp[2 * (long long)h.z].x;
  int plus = -1, minus = -1;
  if (e >= 0) {
    const int sp = value_pixel(img_all, I, b, h.y);
    const int ep = value_pixel(img_all, I, b, ext_key[e].y);
    const bool saddle_plus = (!faces) != d;
    plus = saddle_plus ? sp : ep;
    minus = saddle_plus ? ep : sp;
  }
  if (int* p = PLUS.at(d, b)) p[li] = plus;
  if (int* m = MINUS.at(d, b)) m[li] = minus;
}

// Every persistence value with its metadata, in the order of the autograd
// outputs: per image its min side's entries, then its max side's, each in
// survivor order. One thread per survivor and side writes an entry whole;
// building the same order from per-side lists took a stable sort of all
// entries and fifteen more passes (8 x 512^2, 1.3 M entries: 1.0 ms of the
// forward, 0.05 ms here).
struct PairEntries {
  float* p;
  long long* image;
  signed char* side;    // 0 min, 1 max
  int* ppairs;
  int* plus;            // image-local pixels
  int* minus;
  int* plus_flat;       // pixels counted over the whole batch
  int* minus_flat;
};
struct PairSide {
  const int2* pp;         // every second record: paired extremum, persistence bits
  const int2* ext_key;    // (value bits, cell) of each extremum
  const int4* out;        // [nsurv] rank of the pair's root in w, persistence bits in z
  const int* alive_base;  // [B + 1]
};

__global__ void __launch_bounds__(256) pair_entries_out_kernel(int nsurv, Imgs I, const int* __restrict__ surv_base,
                                                               const float* __restrict__ img_all,
                                                               const SurvHead* __restrict__ head, PairSide F,
                                                               PairSide V, PairEntries E) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(t >> 1), sd = (int)(t & 1);
  if (i >= nsurv) return;
  const PairSide& S = sd ? V : F;
  const int4 h = *reinterpret_cast<const int4*>(head + i);
  const int b = h.x;
  const bool d = I.dual[b];
  const int first = surv_base[b], n = surv_base[b + 1] - first;
  const bool is_max = (sd == 0) != d;  // faces are maxima in the primal, minima in the dual
  const long long k = 2LL * first + (is_max ? n : 0) + (i - first);
  const int4 o = S.out[i];
  const int e = S.pp[2 * (long long)h.z].x;
  int plus = -1, minus = -1;
  if (e >= 0) {
    const int sp = value_pixel(img_all, I, b, h.y);
    const int ep = value_pixel(img_all, I, b, S.ext_key[e].y);
    const bool saddle_plus = (sd == 1) != d;
    plus = saddle_plus ? sp : ep;
    minus = saddle_plus ? ep : sp;
  }
  E.p[k] = __int_as_float(o.z);
  E.image[k] = b;
  E.side[k] = is_max;
  E.ppairs[k] = o.w >= 0 ? o.w - S.alive_base[b] : -1;
  E.plus[k] = plus;
  E.minus[k] = minus;
  E.plus_flat[k] = plus >= 0 ? plus + I.px_base[b] : plus;
  E.minus_flat[k] = minus >= 0 ? minus + I.px_base[b] : minus;
}

// ---------------------------------------------------------------------------
// backward: grad_img[pix] = sum of +-dL/dp over the pair ends at pix, summed
// in a fixed order (no float atomics), so repeated runs give identical bits.

// Entry k of 2n: pair k >> 1, + end for even k, - end for odd k. Key = pixel
// (npx for an absent end, which sorts last).
__global__ void pair_entries_kernel(long long n, const int* __restrict__ plus, const int* __restrict__ minus,
                                    int npx, int* __restrict__ key, int* __restrict__ idx) {
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 2 * n) return;
  const long long i = k >> 1;
  int p = (k & 1) ? minus[i] : plus[i];
  key[k] = (p >= 0 && p < npx) ? p : npx;
  idx[k] = (int)k;
}

// One thread per sorted entry that starts a run of equal keys: sums the run
// in ascending entry order (the radix sort is stable) and writes the pixel.
__global__ void pair_segments_kernel(long long m, const int* __restrict__ key, const int* __restrict__ idx,
                                     const float* __restrict__ grad_p, int npx, float* __restrict__ grad_img) {
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const int pix = key[k];
  if (pix >= npx || (k > 0 && key[k - 1] == pix)) return;
  float acc = 0.0f;
  for (long long j = k; j < m && key[j] == pix; ++j) {
    const int e = idx[j];
    const float g = grad_p[e >> 1];
    acc = (e & 1) ? acc - g : acc + g;
  }
  grad_img[pix] = acc;
}

}  // namespace dmsc
