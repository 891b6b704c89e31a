// Exclusive scan of V 32-bit counts at once, in one launch.
//
// Single pass with decoupled look-back (Merrill and Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back"): a block takes the next tile
// by a ticket, sums it, publishes the sum, adds up its predecessors' sums until
// one has published its whole prefix, and publishes its own. A count and its
// state share one 64-bit word, so no fence is needed; the state carries the
// launch's epoch, so nothing is cleared between launches, and the last ticket
// resets the counter. Counts wrap at 2^32, which only totals that fail the
// call reach.
//
// The inputs and outputs are an operator's: op.load4(i, v) gives the counts of
// the items i .. i + 3 (i a multiple of 4, the arrays 16-byte aligned),
// op.load(i, v) those of one item (the last few), store4 / store take their
// exclusive sums, op.finish(v) the totals (one thread). The calls here are small (a
// scan's own work is 4 to 50 us), so what counts most is the number of launches:
// the library scan took two per array and a kernel to fetch the totals, ten
// to twelve where one is left.
//
// A tile looks for its predecessors' sums a bounded number of times. One that
// gives up sets the status word and calls op.gave_up(): its sums are wrong, so
// nothing may be addressed by them before the host or a later kernel has seen
// either.
#pragma once

#include "common.cuh"

namespace dmsc {

constexpr int kScanNT = 256, kScanRows = 4, kScanTile = kScanNT * kScanRows * 4;  // rows of 128 items per warp

struct ScanState {
  unsigned* ticket;
  unsigned long long* word;  // [V][tiles] (epoch << 2 | state) << 32 | count
  unsigned epoch;
  int looks;  // bound on a lane's looks at words that are not published yet
  unsigned* status;
};
// Predecessors are running, so no tile comes near it (about half a second).
constexpr int kScanLooks = 1 << 20;

template <int V, class Op>
__global__ void __launch_bounds__(kScanNT) scan_kernel(Op op, long long n, ScanState st) {
  constexpr int NW = kScanNT / 32;
  static_assert(V <= NW, "a warp per count");
  __shared__ unsigned tile, wsum[V][NW], pre[V], tot[V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tiles = (int)gridDim.x;
  if (threadIdx.x == 0) {
    tile = atomicAdd(st.ticket, 1u);
    if (tile == (unsigned)tiles - 1) *st.ticket = 0;  // every ticket is out
  }
  __syncthreads();
  const int t = (int)tile;
  const long long i0 = (long long)t * kScanTile + warp * (128 * kScanRows) + 4 * lane;
  unsigned x[kScanRows][4][V], run[V];
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    const long long i = i0 + 128 * k;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int v = 0; v < V; ++v) x[k][j][v] = 0;
    if (i + 3 < n) {
      op.load4(i, x[k]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i + j < n) op.load(i + j, x[k][j]);
    }
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    run[v] = 0;
#pragma unroll
    for (int k = 0; k < kScanRows; ++k) {
      const unsigned c0 = x[k][0][v], c1 = c0 + x[k][1][v], c2 = c1 + x[k][2][v], c3 = c2 + x[k][3][v];
      unsigned s = c3;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      const unsigned e = run[v] + s - c3;
      x[k][0][v] = e;
      x[k][1][v] = e + c0;
      x[k][2][v] = e + c1;
      x[k][3][v] = e + c2;
      run[v] += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) wsum[v][warp] = run[v];
  }
  __syncthreads();
  if (warp < V) {  // warp v: the tile's sum of count v and its predecessors'
    const int v = warp;
    const unsigned w = lane < NW ? wsum[v][lane] : 0u;
    unsigned s = w;
#pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    const unsigned sum = __shfl_sync(0xffffffffu, s, NW - 1);
    if (lane < NW) wsum[v][lane] = s - w;
    volatile unsigned long long* word = st.word + (long long)v * tiles;
    const unsigned long long agg = (unsigned long long)(st.epoch << 2 | 1u) << 32;
    const unsigned long long whole = (unsigned long long)(st.epoch << 2 | 2u) << 32;
    unsigned before = 0;
    if (t > 0) {
      if (lane == 0) word[t] = agg | sum;
      int looks = 0;
      for (int p0 = t - 1; p0 >= 0; p0 -= 32) {
        const int p = p0 - lane;  // lane 0: the nearest predecessor
        unsigned long long q = whole;
        if (p >= 0) {
          q = 0;
          while (looks < st.looks && (unsigned)((q = word[p]) >> 34) != st.epoch) ++looks;
        }
        const unsigned done = __ballot_sync(0xffffffffu, ((unsigned)(q >> 32) & 3u) == 2u);
        // the counts up to the nearest whole prefix
        const int last = done ? __ffs(done) - 1 : 31;
        before += __reduce_add_sync(0xffffffffu, lane <= last ? (unsigned)q : 0u);
        if (done) break;
      }
      if (looks >= st.looks) {
        set_status(st.status, kStatusRoundCap);
        op.gave_up();
      }
    }
    if (lane == 0) {
      word[t] = whole | (before + sum);
      pre[v] = before;
      tot[v] = before + sum;
    }
  }
  __syncthreads();
  unsigned add[V];
#pragma unroll
  for (int v = 0; v < V; ++v) add[v] = pre[v] + wsum[v][warp];
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    const long long i = i0 + 128 * k;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int v = 0; v < V; ++v) x[k][j][v] += add[v];
    if (i + 3 < n) {
      op.store4(i, x[k]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i + j < n) op.store(i + j, x[k][j]);
    }
  }
  if (t == tiles - 1 && threadIdx.x == 0) op.finish(tot);
}

// Row-segment counts of minima, saddles and maxima; the totals go to the
// mapped readback area, since the host sizes the lists and launches their
// writer from them. So that it can see first whether they hold, two more words
// there take the status word (a gradient tile that gave up has written no
// counts) and whether a tile of this scan gave up (it may end after the last
// one).
struct SegScan {
  const int* in[3];
  int* out[3];
  long long* rb;  // [5]
  const unsigned* status;
  __device__ void load(long long i, unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = (unsigned)in[k][i];
  }
  __device__ void store(long long i, const unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k][i] = (int)v[k];
  }
  __device__ void load4(long long i, unsigned (*v)[3]) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int4 c = *reinterpret_cast<const int4*>(in[k] + i);
      v[0][k] = (unsigned)c.x;
      v[1][k] = (unsigned)c.y;
      v[2][k] = (unsigned)c.z;
      v[3][k] = (unsigned)c.w;
    }
  }
  __device__ void store4(long long i, const unsigned (*v)[3]) const {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      *reinterpret_cast<int4*>(out[k] + i) = make_int4((int)v[0][k], (int)v[1][k], (int)v[2][k], (int)v[3][k]);
  }
  __device__ void finish(const unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) rb[k] = v[k];
    rb[3] = *status;
  }
  __device__ void gave_up() const { rb[4] = kStatusRoundCap; }
};

// Alive flags of both sides' extrema and survivor flags of the saddles.
struct FlagScan {
  const uint8_t* in[2];
  long long n[2];
  int* out[2];
  int* total;  // [2]
  __device__ void load(long long i, unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (i < n[k]) v[k] = in[k][i];
  }
  __device__ void store(long long i, const unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (i < n[k]) out[k][i] = (int)v[k];
  }
  __device__ void load4(long long i, unsigned (*v)[2]) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (i + 3 < n[k]) {
        const uchar4 c = *reinterpret_cast<const uchar4*>(in[k] + i);
        v[0][k] = c.x;
        v[1][k] = c.y;
        v[2][k] = c.z;
        v[3][k] = c.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i + j < n[k]) v[j][k] = in[k][i + j];
      }
    }
  }
  __device__ void store4(long long i, const unsigned (*v)[2]) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (i + 3 < n[k]) {
        *reinterpret_cast<int4*>(out[k] + i) = make_int4((int)v[0][k], (int)v[1][k], (int)v[2][k], (int)v[3][k]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i + j < n[k]) out[k][i + j] = (int)v[j][k];
      }
    }
  }
  __device__ void finish(const unsigned* v) const {
    total[0] = (int)v[0];
    total[1] = (int)v[1];
  }
  __device__ void gave_up() const {}  // the host reads the status word with the counts
};

// Pairs of packed counts (side 0 low, side 1 high), in place.
struct PackedScan {
  unsigned long long* a[2];
  __device__ void load(long long i, unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const unsigned long long p = a[k][i];
      v[2 * k] = (unsigned)p;
      v[2 * k + 1] = (unsigned)(p >> 32);
    }
  }
  __device__ void store(long long i, const unsigned* v) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) a[k][i] = v[2 * k] | (unsigned long long)v[2 * k + 1] << 32;
  }
  __device__ void load4(long long i, unsigned (*v)[4]) const {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int4 c = *reinterpret_cast<const int4*>(a[k] + i + 2 * h);
        v[2 * h][2 * k] = (unsigned)c.x;
        v[2 * h][2 * k + 1] = (unsigned)c.y;
        v[2 * h + 1][2 * k] = (unsigned)c.z;
        v[2 * h + 1][2 * k + 1] = (unsigned)c.w;
      }
  }
  __device__ void store4(long long i, const unsigned (*v)[4]) const {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<int4*>(a[k] + i + 2 * h) =
            make_int4((int)v[2 * h][2 * k], (int)v[2 * h][2 * k + 1], (int)v[2 * h + 1][2 * k],
                      (int)v[2 * h + 1][2 * k + 1]);
  }
  __device__ void finish(const unsigned*) const {}
  __device__ void gave_up() const {}  // the host reads the status word with the sizes
};

}  // namespace dmsc
