// Persistence pairing and cancellation on the device.
//
// Reference semantics: cpu/persistence.hxx:16-182. Each side is a sequential
// union-find sweep over the saddles in sweep order (ascending (s_val, cell id)
// for minima in the primal, the reverse for maxima; flipped in the dual)
// with the elder rule: at a saddle joining two components the one whose
// oldest extremum is younger dies, and the void (-1, one-sided saddles) is
// older than every extremum.
//
// Parallel form (exact). Groups start as single extrema plus the void; a
// group is named by its oldest member. Every round, each group takes the
// first (lowest sweep index) saddle leaving it; a group whose partner group
// has an older oldest member dies at that saddle, which pairs the saddle with
// the group's oldest member, and joins the partner. Saddles whose ends fall
// in one group are cycles (pair -1, persistence -1). Why this equals the
// sweep: a group is always connected, by the time any of its outgoing saddles
// is swept, to its oldest member, so at its first outgoing saddle the dying
// side is exactly known; the globally first remaining saddle is always
// decided, so every round makes progress.
//
#pragma once

#include <cuda/atomic>

#include "common.cuh"
#include "gradient.cuh"
#include "replay.cuh"

namespace dmsc {

constexpr unsigned long long kNoEdge = ~0ull;

// Sweep key of saddle e (list index) on one side: the side sweeps its image's
// saddles in ascending (s_val, cell id) order, or exactly the reverse (desc;
// cpu/arcs_topology.hxx:99-102, 142). List indices ascend with the cell id
// inside an image, so (orderable(s_val), e) orders the ascending sweep and
// (~orderable(s_val), 0x7FFFFFFF - e) the descending one; both stay below
// kNoEdge, and keys of one image never meet another image's.
__device__ __forceinline__ unsigned long long sweep_key(float v, int e, bool desc) {
  const uint32_t o = orderable_key(v);
  return desc ? ((unsigned long long)(~o) << 32) | (uint32_t)(0x7FFFFFFF - e)
              : ((unsigned long long)o << 32) | (uint32_t)e;
}
__device__ __forceinline__ int sweep_key_saddle(unsigned long long k, bool desc) {
  const int lo = (int)(uint32_t)k;
  return desc ? 0x7FFFFFFF - lo : lo;
}

// A saddle's decision on one side: the extremum that dies at it with the arc end
// it dies on (bit 30: the second; extremum indices stay below 2^29), -1 for a
// cycle or a saddle that is not decided yet.
__device__ __forceinline__ int dying_word(int x, bool second) { return second ? x | 0x40000000 : x; }
__device__ __forceinline__ int dying_of(int w) { return w < 0 ? -1 : w & 0x3FFFFFFF; }
__device__ __forceinline__ bool dying_second(int w) { return (w >> 30) & 1; }

// Ends of a saddle as the walks record them for the tile pass below. A local
// saddle has its two ends inside its own 64 x 64 index tile or in the void:
// each end is ~(r * 64 + c) of the extremum's cell in the tile (negative), or
// ~kLocalVoid. Any other saddle holds the ends' groups (>= 0, the void M), a
// cycle kCycleEnd twice.
constexpr int kLocalVoid = 0x7FFF;
constexpr int kCycleEnd = (int)0x80000000;

// K4: per saddle, both face walks and the vertex walks. Writes per saddle and
// side one record {target 0, target 1, cells 0, cells 1}: each arc's dense
// target index (or -1) and its raw arc's cell count (a saddle's two records
// in one 32-byte sector, for the random reads); and the pairing's starting
// state: a saddle whose two ends coincide is a cycle, the others
// record their ends and reduce their sweep key into both ends' minima
// (nothing waits for these reductions), and a saddle that is not local to its
// tile reduces the value part of its key into its ends' `leave` too. Bound by
// instruction issue: the rows of the four ends by multiplication instead of
// division and 32-bit step counts took it from 38 to 32 registers (all 64
// warps of an SM resident) and from 0.373 to 0.266 ms at 4096^2, a step's
// distance from two selects (flow_step) to 0.206 (8192^2 noise: 0.694).
__global__ void __launch_bounds__(256) saddle_walk_kernel(Imgs I, const uint8_t* __restrict__ flow, int nsad,
                                                          const int* __restrict__ crit_sad,
                                                          const int* __restrict__ sad_img,
                                                          const int* __restrict__ off_max,
                                                          const uint32_t* __restrict__ max_bits,
                                                          const int* __restrict__ off_min,
                                                          const uint32_t* __restrict__ min_bits,
                                                          int4* __restrict__ arc, int cap, PairStart ps, unsigned* status) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsad) return;
  const int b = sad_img[s];
  const int H = I.H[b], W = I.W[b], Nx = W + 1;
  const int sc = crit_sad[s];
  const int sl = (sc >> 2) - I.idx_base[b], sy = row_of(I, b, sl), sx = sl - sy * Nx;
  int te[2][2], len[2][2], loc[2][2];  // loc: the end's cell in the saddle's tile, -1 when it lies in another
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    int steps;
    const int end = flow_walk<4>(flow, face_start(sc, j, Nx) >> 2, Nx, cap, &steps, status);
    int y, x;
    const int target = seg_rank(I, b, end, Nx, off_max, max_bits, y, x);
    te[0][j] = target;
    len[0][j] = target >= 0 ? steps + 1 : 0;  // cells of the raw arc, start and end included
    loc[0][j] = ((y ^ sy) | (x ^ sx)) >> 6 ? -1 : (y & 63) << 6 | (x & 63);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int start = vertex_start(sc, j, sy, sx, H, W, Nx);
    int steps = 0;
    int target = -1, at = kLocalVoid;
    if (start >= 0) {
      const int end = flow_walk<0>(flow, start >> 2, Nx, cap, &steps, status);
      int y, x;
      target = seg_rank(I, b, end, Nx, off_min, min_bits, y, x);
      at = ((y ^ sy) | (x ^ sx)) >> 6 ? -1 : (y & 63) << 6 | (x & 63);
    }
    te[1][j] = target;
    len[1][j] = target >= 0 ? steps + 1 : 0;  // an arc that leaves the image is empty
    loc[1][j] = at;
  }
  // a raw arc has fewer cells than the batch (cell ids are int32)
  arc[2 * (long long)s] = make_int4(te[0][0], te[0][1], len[0][0], len[0][1]);
  arc[2 * (long long)s + 1] = make_int4(te[1][0], te[1][1], len[1][0], len[1][1]);
  // descending sweep on the face side in the primal and the vertex side in
  // the dual
  const bool d = I.dual[b];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    const int M = ps.M[sd];
    const int ga = te[sd][0] < 0 ? M : te[sd][0], gb = te[sd][1] < 0 ? M : te[sd][1];
    if (ga == gb) {
      ps.g12[sd][s] = make_int2(kCycleEnd, kCycleEnd);
      continue;
    }
    const bool local = (loc[sd][0] | loc[sd][1]) >= 0;
    ps.g12[sd][s] = local ? make_int2(~loc[sd][0], ~loc[sd][1]) : make_int2(ga, gb);
    const unsigned long long k = sweep_key(ps.sval[s], s, sd == 0 ? !d : d);
    if (ga != M) {
      atomicMin(ps.minedge[sd] + ga, k);  // results unused: reductions
      if (!local) atomicMin(ps.leave[sd] + ga, (unsigned)(k >> 32));
    }
    if (gb != M) {
      atomicMin(ps.minedge[sd] + gb, k);
      if (!local) atomicMin(ps.leave[sd] + gb, (unsigned)(k >> 32));
    }
  }
}

// K5a: the pairing's rounds inside one 64 x 64 index tile and side per block,
// on groups and saddles held in shared memory. A round's decision needs a
// group's first outgoing saddle and the oldest member of the group behind it,
// nothing else, so a block may decide any group whose first outgoing saddle
// is local to the tile, at any time: the saddles that leave the tile enter
// only through the smallest value key among them at each extremum (`leave`,
// from the walks), and a group that reaches it waits for the global rounds.
// Round 0 decides from the walks' minima. The saddles that stay undecided are
// listed again each round, so a round costs what is left of them. After the
// rounds only the first of the saddles between the same two groups is kept
// (when a later one is swept the two are joined already: a cycle); the block
// then writes the decisions (-1 for a cycle, and for now for what stays
// undecided), links every dead group to its root and appends the saddles and
// roots that remain to the lists of the global rounds. A tile with more
// extrema or saddles than fit (kTileNodes, kTileEdges: above those of i.i.d.
// noise, 820 and 1460 of 4096 cells) hands everything on.
//
// Bound: instruction issue (short dependent shared-memory chains and block
// barriers, 48 warps per SM). On the bump fields about 12% of the saddles and 8%
// of the groups are left to the global rounds, on i.i.d. noise 15% and 10%
// (with tiles of 128: 5 to 8%, but one block per SM). Measured, the whole
// pairing stage without and with this pass and the last block's rounds: 4096^2
// bumps 1.13 -> 0.725 ms (this pass 0.43), 8192^2 noise 7.80 -> 4.69, 509 x
// 1531 0.287 -> 0.147.
constexpr int kTileNodes = 896, kTileEdges = 1664;
// Threads per block: 256 when the blocks fill the device several times over,
// 512 when one wave holds them all and a block's own latency counts (24% less
// at 256^2, 8% more at 4096^2).
constexpr int kTilePairNT[2] = {256, 512};
constexpr int kTileRounds = 5;    // 4, 5, 6, 8 rounds: stage of 5.68, 4.69, 4.67, 4.93 ms at 8192^2 noise, 0.765, 0.728, 0.738, 0.763 at 4096^2
constexpr int kTilePairs = 512;   // slots of the table of group pairs
constexpr int tile_list(int warps) { return (kTileEdges / 32 + warps - 1) / warps * 32; }  // a warp's edges
constexpr unsigned kTileVoid = 0xFFFEu;
// `ends` of an edge that is no longer undecided: kTileDead | the dying end (0x8000:
// the second) | the dead node, or a cycle (or not the first between its groups); of one that leaves the tile
constexpr uint32_t kTileDead = 0xFFFF0000u, kTileCycle = 0xFFFFFFFFu, kTileOut = 0xFFFEFFFEu;

template <int NT>
struct PairTileSmem {
  unsigned long long minedge[kTileNodes];  // (value key, edge or its complement) of a root's first local saddle
  float val[kTileNodes];
  uint32_t leave[kTileNodes];   // value key of the group's first saddle out of the tile
  uint32_t ends[kTileEdges];    // nodes of both ends (roots as of the last phase A)
  uint32_t hi[kTileEdges];      // value key
  uint16_t list[NT / 32][tile_list(NT / 32)];  // each warp's undecided edges
  uint16_t link[kTileNodes];
  uint8_t seg[kTileNodes];      // segment of each node
  uint8_t row[kTileEdges];      // row of each edge
  uint32_t bits[2 * kLT];       // extrema of each (row, 32-column segment)
  uint16_t npre[2 * kLT + 1];   // nodes before each segment
  int noff[2 * kLT];            // first rank of each segment
  uint16_t spre[kLT + 1];       // edges before each row
  int sbase[kLT];               // first saddle of each row
  int n_live;
};

struct PairTileArgs {
  PairStart ps;
  const int* off[2];        // segment offsets of each side's extrema
  const uint32_t* bits[2];  // segment bit masks of each side's extrema
  const int2* key[2];       // (value bits, cell) of each extremum
  const int* off_sad;       // segment offsets and counts of the saddles
  const int* seg_sad;
  int* act[2];    // active saddles for the global rounds
  int* roots[2];  // live roots
};

// Root of node x in the tile's forest (path halving; at most kTileNodes steps).
__device__ __forceinline__ unsigned tile_root(volatile uint16_t* link, unsigned x) {
  if (x == kTileVoid) return x;
  unsigned p = link[x];
  for (int k = 0; k <= kTileNodes; ++k) {
    if (p == x || p == kTileVoid) return p;
    const unsigned pp = link[p];
    if (pp == p) return p;
    link[x] = (uint16_t)pp;
    if (pp == kTileVoid) return pp;
    x = pp;
    p = link[x];
  }
  return x;
}

template <int NT>
__global__ void __launch_bounds__(NT, 1536 / NT) pair_tile_kernel(Imgs I, PairTileArgs A) {
  extern __shared__ __align__(16) unsigned char pair_tile_smem[];
  PairTileSmem<NT>& S = *reinterpret_cast<PairTileSmem<NT>*>(pair_tile_smem);
  constexpr int NW = NT / 32, kNodesPer = (kTileNodes + NT - 1) / NT;
  const bool s1 = blockIdx.x & 1;  // consecutive blocks: the two sides of one tile
  const LabelTile g = label_tile_of(I, blockIdx.x >> 1);
  const bool dual = I.dual[g.b];
  const bool desc = s1 ? dual : !dual, older_less = s1 ? !dual : dual;
  unsigned long long* minedge = s1 ? A.ps.minedge[1] : A.ps.minedge[0];
  int* glink = s1 ? A.ps.link[1] : A.ps.link[0];
  int2* g12 = s1 ? A.ps.g12[1] : A.ps.g12[0];
  int* dying = s1 ? A.ps.dying[1] : A.ps.dying[0];
  int* cnt = s1 ? A.ps.cnt[1] : A.ps.cnt[0];
  int* act = s1 ? A.act[1] : A.act[0];
  int* roots = s1 ? A.roots[1] : A.roots[0];
  const int M = s1 ? A.ps.M[1] : A.ps.M[0];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  // ---- segment tables: extrema by (row, segment), saddles by row ----
  const int nsegx = (g.W + kTileX) / kTileX;
  if (tid < 2 * kLT) {
    const int r = tid >> 1, y = g.y0 + r, sx = (g.x0 >> 5) + (tid & 1);
    const bool in = y <= g.H && sx < nsegx;
    const long long q = (long long)I.seg_base[g.b] + (long long)y * nsegx + sx;
    S.bits[tid] = in ? __ldg((s1 ? A.bits[1] : A.bits[0]) + q) : 0u;
    S.noff[tid] = in ? __ldg((s1 ? A.off[1] : A.off[0]) + q) : 0;
    const int so = in ? __ldg(A.off_sad + q) : 0x7FFFFFFF, sn = in ? __ldg(A.seg_sad + q) : 0;
    const int both = sn + __shfl_xor_sync(0xffffffffu, sn, 1);
    if ((tid & 1) == 0) {
      S.sbase[r] = so;
      S.spre[r + 1] = (uint16_t)both;
    }
  } else if (tid == NT - 1) {
    S.n_live = 0;
  }
  __syncthreads();
  if (tid < 32) {  // exclusive sums: 128 segments (4 per lane), 64 rows (2 per lane)
    int c[4], n = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) n += c[k] = __popc(S.bits[4 * lane + k]);
    const int e0 = S.spre[2 * lane + 1], e1 = S.spre[2 * lane + 2];
    int xn = n, xe = e0 + e1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yn = __shfl_up_sync(0xffffffffu, xn, o), ye = __shfl_up_sync(0xffffffffu, xe, o);
      if (lane >= o) {
        xn += yn;
        xe += ye;
      }
    }
    int at = xn - n;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      S.npre[4 * lane + k] = (uint16_t)at;
      at += c[k];
    }
    if (lane == 31) S.npre[2 * kLT] = (uint16_t)at;
    __syncwarp();
    S.spre[2 * lane + 1] = (uint16_t)(xe - e1);
    S.spre[2 * lane + 2] = (uint16_t)xe;
    if (lane == 0) S.spre[0] = 0;
  }
  __syncthreads();
  const int nn = S.npre[2 * kLT], ne = S.spre[kLT];
  auto saddle_in_row = [&](int k, int r) { return S.sbase[r] + k - S.spre[r]; };
  auto edge_of = [&](int s) {  // edge of a saddle of the tile
    int lo = 0;
#pragma unroll
    for (int w = kLT / 2; w > 0; w >>= 1)
      if (S.sbase[lo + w] <= s) lo += w;
    return S.spre[lo] + s - S.sbase[lo];
  };
  auto local_rank = [&](int enc, bool node) -> int {  // node or list rank of a local end
    const int p = ~enc;
    if (p == kLocalVoid) return node ? (int)kTileVoid : M;
    const int q = p >> 5;
    return (node ? S.npre[q] : S.noff[q]) + __popc(S.bits[q] & ((1u << (p & 31)) - 1u));
  };
  if (nn > kTileNodes || ne > kTileEdges) {  // does not fit: all to the global rounds
    for (int k0 = 0; k0 < max(ne, kLTN); k0 += NT) {
      const int k = k0 + tid;
      int s = -1, x = -1;
      if (k < ne) {
        int r = 0;
        for (int w = kLT / 2; w > 0; w >>= 1)
          if (S.spre[r + w] <= k) r += w;
        s = saddle_in_row(k, r);
        dying[s] = -1;
        const int2 e = g12[s];
        if (e.x == kCycleEnd)
          s = -1;
        else if (e.x < 0)
          g12[s] = make_int2(local_rank(e.x, false), local_rank(e.y, false));
      }
      if (k < kLTN) {  // the cell at position k of the tile
        const unsigned m = S.bits[k >> 5];
        if ((m >> (k & 31)) & 1u) {
          x = S.noff[k >> 5] + __popc(m & ((1u << (k & 31)) - 1u));
          minedge[x] = kNoEdge;
        }
      }
      int ps, px;
      block_reserve2(cnt, s >= 0, cnt + 3, x >= 0, ps, px);
      if (s >= 0) act[ps] = s;
      if (x >= 0) roots[px] = x;
    }
    return;
  }
  {  // row of every edge, segment of every node
    constexpr int kR = NT / kLT, kQ = NT / (2 * kLT);  // threads per row and segment
    const int r = tid / kR, q = tid / kQ;
    for (int k = S.spre[r] + tid % kR; k < S.spre[r + 1]; k += kR) S.row[k] = (uint8_t)r;
    for (int i = S.npre[q] + tid % kQ; i < S.npre[q + 1]; i += kQ) S.seg[i] = (uint8_t)q;
  }
  __syncthreads();
  auto saddle_of = [&](int k) { return saddle_in_row(k, S.row[k]); };
  auto rank_of = [&](unsigned i) {
    const int q = S.seg[i];
    return S.noff[q] + (int)i - S.npre[q];
  };
  // ---- nodes i = tid + NT j; edges in chunks of 32, chunk c to warp c % NW ----
  unsigned long long me[kNodesPer];
#pragma unroll
  for (int j = 0; j < kNodesPer; ++j) {
    const int i = tid + NT * j;
    me[j] = kNoEdge;
    if (i >= nn) continue;
    const int x = rank_of(i);
    me[j] = minedge[x];
    S.val[i] = __int_as_float(__ldg(&(s1 ? A.key[1] : A.key[0])[x].x));
    S.leave[i] = (s1 ? A.ps.leave[1] : A.ps.leave[0])[x];
    S.minedge[i] = kNoEdge;
    S.link[i] = (uint16_t)i;
  }
  uint16_t* const list = S.list[warp];
  int n = 0;  // edges in the warp's list
  constexpr int kBatch = 2;  // chunks whose loads are issued together (a warp has three or so; 4 spill)
  for (int c0 = warp; c0 * 32 < ne; c0 += NW * kBatch) {
    int2 en[kBatch];
    float sv[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int k = (c0 + NW * u) * 32 + lane;
      en[u] = make_int2(kCycleEnd, kCycleEnd);
      sv[u] = 0.f;
      if (k < ne) {
        const int sd = saddle_of(k);
        en[u] = g12[sd];
        sv[u] = __ldg(A.ps.sval + sd);
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int k = (c0 + NW * u) * 32 + lane;
      if ((c0 + NW * u) * 32 >= ne) break;  // warp-uniform
      uint32_t e = en[u].x == kCycleEnd ? kTileCycle : kTileOut;
      const bool take = en[u].x < 0 && en[u].x != kCycleEnd;
      if (take) e = (uint32_t)local_rank(en[u].x, true) | (uint32_t)local_rank(en[u].y, true) << 16;
      if (k < ne) {
        const uint32_t o = orderable_key(sv[u]);
        S.hi[k] = desc ? ~o : o;
        S.ends[k] = e;
      }
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) list[n + __popc(m & lt)] = (uint16_t)k;
      n += __popc(m);
    }
  }
  __syncthreads();
  // A root's decision on its first outgoing edge k (value key h1): it dies
  // there when the group behind it is older and no saddle out of the tile
  // comes first. (The other end's root, if this edge is its first too, is the
  // older one: it stays alive, with or without seeing the mark.)
  auto decide = [&](int i, uint32_t h1, int k) -> bool {
    const uint32_t e = S.ends[k];
    if (e >= kTileDead) return false;
    const bool second = (e & 0xFFFFu) != (unsigned)i;
    const unsigned h = second ? e & 0xFFFFu : e >> 16;
    if (h != kTileVoid) {  // nodes are numbered in cell order
      const float vh = S.val[h], vi = S.val[i];
      if (!(older_less ? tie_lt(vh, (int)h, vi, i) : tie_lt(vi, i, vh, (int)h))) return false;
    }
    S.ends[k] = kTileDead | (second ? 0x8000u : 0u) | (uint32_t)i;
    S.link[i] = (uint16_t)h;
    return true;
  };
  unsigned died = 0;  // bit j: node tid + NT j died in the previous round
#pragma unroll
  for (int j = 0; j < kNodesPer; ++j) {
    const int i = tid + NT * j;
    if (i >= nn || me[j] == kNoEdge) continue;
    const uint32_t h1 = (uint32_t)(me[j] >> 32);
    if (S.leave[i] <= h1) continue;  // its first saddle leaves the tile, or may
    if (decide(i, h1, edge_of(sweep_key_saddle(me[j], desc)))) died |= 1u << j;
  }
  int any = __syncthreads_or(died);
  for (int round = 1; any && round < kTileRounds; ++round) {
    // a dead group's first saddle out of the tile now belongs to its root
    if (died) {
#pragma unroll
      for (int j = 0; j < kNodesPer; ++j) {
        if (!((died >> j) & 1u)) continue;
        const int i = tid + NT * j;
        const unsigned r = tile_root(S.link, i);
        if (r != kTileVoid) atomicMin(&S.leave[r], S.leave[i]);
      }
    }
    // phase A: both ends' roots; cycles and the edges decided in the previous
    // round leave the warp's list, the others reduce their key into both
    // roots' minimum
    int kept = 0;
    for (int q0 = 0; q0 < n; q0 += 32) {
      bool keep = false;
      int k = 0;
      if (q0 + lane < n) {
        k = list[q0 + lane];
        const uint32_t e = S.ends[k];
        if (e < kTileDead) {
          const unsigned a = tile_root(S.link, e & 0xFFFFu), b = tile_root(S.link, e >> 16);
          keep = a != b;
          S.ends[k] = keep ? a | b << 16 : kTileCycle;
          if (keep) {
            const unsigned long long m = ((unsigned long long)S.hi[k] << 32) | (uint32_t)(desc ? 0xFFFF - k : k);
            if (a != kTileVoid && m < *(volatile unsigned long long*)&S.minedge[a]) atomicMin(&S.minedge[a], m);
            if (b != kTileVoid && m < *(volatile unsigned long long*)&S.minedge[b]) atomicMin(&S.minedge[b], m);
          }
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      __syncwarp();  // the chunk is read before its slots are written again
      if (keep) list[kept + __popc(m & lt)] = (uint16_t)k;
      kept += __popc(m);
    }
    n = kept;
    __syncthreads();
    // phase B
    died = 0;
#pragma unroll
    for (int j = 0; j < kNodesPer; ++j) {
      const int i = tid + NT * j;
      if (i >= nn || S.link[i] != i) continue;
      const unsigned long long m = S.minedge[i];
      if (m == kNoEdge) continue;
      S.minedge[i] = kNoEdge;
      const uint32_t h1 = (uint32_t)(m >> 32);
      if (S.leave[i] <= h1) continue;
      if (decide(i, h1, desc ? 0xFFFF - (int)(uint32_t)m : (int)(uint32_t)m)) died |= 1u << j;
    }
    any = __syncthreads_or(died);
  }
  // ---- the first edge between each pair of groups, by a hash table (it
  // takes the arrays of the minima and of the keys out of the tile, which
  // are not read any more) ----
  static_assert(kTilePairs <= kTileNodes, "the table reuses the nodes' arrays");
  uint32_t* tab = S.leave;                // group pair of each slot
  unsigned long long* first = S.minedge;  // its first edge's key
  for (int q = tid; q < kTilePairs; q += NT) {
    tab[q] = kTileCycle;
    first[q] = kNoEdge;
  }
  if (lane == 0) atomicAdd(&S.n_live, n);
  __syncthreads();
  const bool dedupe = S.n_live <= kTilePairs;
  for (int q = lane; q < n; q += 32) {
    const int k = list[q];
    const uint32_t e = S.ends[k];
    if (e >= kTileDead) continue;
    const unsigned a = tile_root(S.link, e & 0xFFFFu), b = tile_root(S.link, e >> 16);
    S.ends[k] = a == b ? kTileCycle : a | b << 16;
    if (!dedupe || a == b) continue;
    const uint32_t pr = min(a, b) | max(a, b) << 16;
    unsigned h = (pr * 0x9E3779B1u) >> 23;  // 9 bits; there are no more pairs than slots
    for (int t = 0; t < kTilePairs; ++t) {
      const uint32_t old = atomicCAS(&tab[h], kTileCycle, pr);
      if (old == kTileCycle || old == pr) break;
      h = (h + 1) & (kTilePairs - 1);
    }
    atomicMin(&first[h], ((unsigned long long)S.hi[k] << 32) | (uint32_t)(desc ? 0xFFFF - k : k));
    S.hi[k] = h;
  }
  __syncthreads();
  // ---- decisions, links and what remains for the global rounds ----
  int n_act = 0, n_root = 0;
  if (dedupe) {
    for (int q = lane; q < n; q += 32) {
      const int k = list[q];
      if (S.ends[k] >= kTileDead) continue;
      const int lo = (int)(uint32_t)first[S.hi[k]];
      if ((desc ? 0xFFFF - lo : lo) != k) S.ends[k] = kTileCycle;
    }
  }
  __syncwarp();  // a warp's edges are those of its chunks
  for (int c = warp; c * 32 < ne; c += NW) {
    const int k = c * 32 + lane;
    if (k >= ne) continue;
    const uint32_t e = S.ends[k];
    dying[saddle_of(k)] = e >= kTileDead && e != kTileCycle ? dying_word(rank_of(e & 0x7FFFu), e & 0x8000u) : -1;
    n_act += e < kTileDead;
  }
#pragma unroll
  for (int j = 0; j < kNodesPer; ++j) {
    const int i = tid + NT * j;
    if (i >= nn) continue;
    const unsigned r = tile_root(S.link, i);
    if (r == (unsigned)i)
      ++n_root;
    else
      glink[rank_of(i)] = r == kTileVoid ? M : rank_of(r);
  }
  int pa, pr;
  block_reserve2(cnt, n_act, cnt + 3, n_root, pa, pr);
  for (int c = warp; c * 32 < ne; c += NW) {
    const int k = c * 32 + lane;
    if (k >= ne) continue;
    const uint32_t e = S.ends[k];
    if (e >= kTileDead) continue;
    const int s = saddle_of(k);
    if (e != kTileOut)
      g12[s] = make_int2((e & 0xFFFFu) == kTileVoid ? M : rank_of(e & 0xFFFFu),
                         (e >> 16) == kTileVoid ? M : rank_of(e >> 16));
    act[pa++] = s;
  }
#pragma unroll
  for (int j = 0; j < kNodesPer; ++j) {
    const int i = tid + NT * j;
    if (i >= nn || S.link[i] != i) continue;
    const int x = rank_of(i);
    minedge[x] = kNoEdge;  // the global rounds start empty
    roots[pr++] = x;
  }
}

// Persistence of each decided saddle and cancellation (persistence.hxx:82-104,
// 139-161), both sides of a saddle in one thread, with the saddle's image's
// orientation and threshold: pp[s] = (paired extremum or -1, persistence bits;
// -1 for a cycle) of the face and the vertex side, alive[d] = 0 for an extremum that a cancelled saddle
// kills, survive[s] = 1 when neither side cancels the saddle; and the forest of
// the thresholded roots (ut_tile_kernel).
struct PersistArgs {
  int nsad;
  int M[2];
  const uint8_t* dual;
  const float* thr;
  const int* sad_img;
  const int* crit_sad;
  const float* sval;
  uint8_t* survive;
  int* n_cancel;               // [2]
  const int* dying[2];
  const int2* key[2];          // (value bits, cell) of each extremum
  int4* pp;                    // [nsad] both sides
  uint8_t* alive[2];
  const int4* arc;             // [2 nsad]
  unsigned long long* ckey[2];  // cancellations' replay keys and saddles (nullptr: arcs not simplified)
  int* cval[2];
  ReplayNode* node[2];
  int* par[2];                 // [M + 1] parent of each extremum (itself when it survives)
};

__global__ void __launch_bounds__(256) persistence_kernel(PersistArgs A) {
  // saddles in list order: every per-saddle access is sequential
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  bool canc[2] = {false, false};
  int d[2] = {-1, -1}, w[2] = {-1, -1};
  float p[2] = {-1.0f, -1.0f};
  if (s < A.nsad) {
    const int b = A.sad_img[s];
    const bool du = A.dual[b];
    const float sv = A.sval[s], thr = A.thr[b];
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      w[sd] = A.dying[sd][s];
      d[sd] = dying_of(w[sd]);
    }
    float ev[2];
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) ev[sd] = d[sd] >= 0 ? __int_as_float(A.key[sd][d[sd]].x) : 0.f;
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      if (d[sd] >= 0) {
        // saddle - extremum on the vertex side in the primal and on the face
        // side in the dual, extremum - saddle otherwise
        p[sd] = (sd == 1) != du ? sub_like_host(sv, ev[sd]) : sub_like_host(ev[sd], sv);
        canc[sd] = p[sd] <= thr;
        if (canc[sd]) A.alive[sd][d[sd]] = 0;
      }
    }
    A.pp[s] = make_int4(d[0], __float_as_int(p[0]), d[1], __float_as_int(p[1]));
    A.survive[s] = !(canc[0] || canc[1]);
  }
  // the cancelled edge hangs the extremum it kills under its other end; and,
  // when the side's arcs are simplified, its replay key joins the list
  // (CancelEvent::operator<, cpu/persistence_struct.hxx:16-21): (persistence,
  // saddle cell); a saddle is cancelled at most once per side, so the pair is
  // unique and the target cell never breaks a tie
  int slot[2];
  block_reserve2(A.n_cancel, canc[0] && A.ckey[0], A.n_cancel + 1, canc[1] && A.ckey[1], slot[0], slot[1]);
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    if (!canc[sd]) continue;
    const int4 a = A.arc[2 * (long long)s + sd];
    const int t = dying_second(w[sd]) ? a.x : a.y;
    A.par[sd][d[sd]] = t >= 0 ? t : A.M[sd];
    if (!A.ckey[sd]) continue;
    const unsigned long long key = ((unsigned long long)orderable_key(p[sd]) << 32) | (unsigned)A.crit_sad[s];
    A.ckey[sd][slot[sd]] = key;
    A.cval[sd][slot[sd]] = s;
    // the killed extremum's replay record: its cancellation key, undecided
    // (the other records are never read, see replay.cuh)
    A.node[sd][d[sd]].ctime = key;
    A.node[sd][d[sd]].status = kPending;
  }
}

// Thresholded roots (the reference's uf_min / uf_max, persistence.hxx:90-104,
// 147-161): one component per connected set of cancelled saddles, whose root
// is its one surviving extremum, or the void. No union is needed: every killed
// extremum d hangs under the extremum t at the other end of the saddle that
// kills it.
//   * d and t are in one component: everything that merged into d's pairing
//     group before died younger than d and earlier in the sweep, so with no
//     larger persistence (float subtraction is monotone) and was cancelled too;
//     so d's end of the saddle hangs together with d. The one exception is
//     threshold infinity on a field with infinite values: equal infinities
//     leave NaN, which is never cancelled, where a later, infinite persistence
//     is. The reference's roots depend on the order of its unions there (they
//     may be killed extrema); these are survivors or the void, as everywhere.
//   * There is no cycle: links put both ends into one pairing group for good,
//     and the last link of a cycle would join two ends that the earlier ones had
//     joined already.
// Chains are long (means of 20 to 70 links on the bump fields, up to 350) but
// stay local: followed inside 64 x 64 tiles first (ut_tile_kernel, pointer
// jumping in shared memory), 2 to 6 links are left for root_out_kernel. With
// a lock-free union of the cancelled edges and its flattening instead the
// persistence and rank stage took 0.57 ms at 4096^2, threshold 0.05, now 0.36;
// 0.196 -> 0.128 at 2048^2, threshold 0.25.
struct UtArgs {
  int M[2];                  // the void is node M
  const int* off[2];         // segment offsets and bit masks of each side's extrema
  const uint32_t* bits[2];
  int* par[2];               // [M + 1] parents, then roots
  const int* rank[2];        // [M] alive extrema before each extremum
  int* rout[2];              // [M] rank of each extremum's thresholded root, -1 for the void
  const int* n_cancel;       // [2]
  unsigned* status;
};

// One tile and side per block: every extremum's parent becomes the first
// extremum on its chain that survives or lies in another tile (or the void).
constexpr int kUtNodes = 2048;  // a tile with more is left as it is
__global__ void __launch_bounds__(256) ut_tile_kernel(Imgs I, UtArgs A) {
  __shared__ int target[kUtNodes];     // a chain's end: its rank
  __shared__ uint16_t next[kUtNodes];  // node in the tile, or kUtEnd | itself
  __shared__ int base[kLT], pre[kLT + 1];
  constexpr unsigned kUtEnd = 0x8000u;
  const bool s1 = blockIdx.x & 1;
  const LabelTile g = label_tile_of(I, blockIdx.x >> 1);
  int* par = s1 ? A.par[1] : A.par[0];
  const int tid = threadIdx.x, lane = tid & 31;
  const int nsegx = (g.W + kTileX) / kTileX;
  if (tid < kLT) {  // a row's extrema are consecutive ranks
    const int y = g.y0 + tid, sx = g.x0 >> 5;
    const bool in = y <= g.H;
    const long long q = (long long)I.seg_base[g.b] + (long long)y * nsegx + sx;
    const uint32_t* bits = s1 ? A.bits[1] : A.bits[0];
    base[tid] = in ? __ldg((s1 ? A.off[1] : A.off[0]) + q) : 0x7FFFFFFF;
    int n = in ? __popc(__ldg(bits + q)) + (sx + 1 < nsegx ? __popc(__ldg(bits + q + 1)) : 0) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += v;
    }
    pre[tid + 1] = n;  // inside its half
    if (tid == 0) pre[0] = 0;
  }
  __syncthreads();
  const int half = pre[32];
  __syncthreads();
  if (tid >= 32 && tid < kLT) pre[tid + 1] += half;
  __syncthreads();
  const int nn = pre[kLT];
  if (nn > kUtNodes) return;
  auto row_of = [&](int i) {
    int r = 0;
#pragma unroll
    for (int w = kLT / 2; w > 0; w >>= 1)
      if (pre[r + w] <= i) r += w;
    return r;
  };
  constexpr int kPer = kUtNodes / 256;
  int x[kPer], p[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = tid + 256 * j;
    x[j] = -1;
    if (i < nn) {
      const int r = row_of(i);
      x[j] = base[r] + i - pre[r];
      p[j] = par[x[j]];
    }
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = tid + 256 * j;
    if (x[j] < 0) continue;
    unsigned nx = kUtEnd | (unsigned)i;
    if (p[j] != x[j]) {  // the parent's node, when it lies in the tile
      int r = 0;
#pragma unroll
      for (int w = kLT / 2; w > 0; w >>= 1)
        if (base[r + w] <= p[j]) r += w;
      const int k = p[j] - base[r];
      if (k >= 0 && k < pre[r + 1] - pre[r]) nx = (unsigned)(pre[r] + k);
    }
    target[i] = p[j];
    next[i] = (uint16_t)nx;
  }
  __syncthreads();
  // barrier-free pointer jumping: any value read lies further along the same
  // chain, so a pointer only moves toward the chain's end
  volatile uint16_t* vn = next;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = tid + 256 * j;
    if (x[j] < 0) continue;
    unsigned nx = vn[i];
    const bool moved = !(nx & kUtEnd);
    for (int k = 0; !(nx & kUtEnd) && k <= kUtNodes; ++k) {
      nx = vn[nx];
      vn[i] = (uint16_t)nx;
    }
    if (moved && (nx & kUtEnd)) par[x[j]] = target[nx & (kUtEnd - 1u)];
  }
}

// Rank of each extremum's thresholded root among the alive extrema (-1 for the
// void), kUtBatch extrema per thread with their chains followed in lockstep (a
// written root is further along the same chain for every reader); and the
// images' first alive ranks and survivors (B + 1 entries, the last ones the
// totals), with the counts and the status word for the host straight to the
// mapped readback area.
constexpr int kUtBatch = 4;
struct RankBases {
  int B, nsad;
  const int* first[2];   // [B + 1] first extremum of each image and side
  const int* first_sad;  // [B + 1] first saddle
  const int* pos;        // [nsad] survivors before each saddle
  const int* total;      // alive extrema of both sides, survivors
  int* alive_base[2];
  int* surv_base;
  long long* rb;
};

__global__ void __launch_bounds__(256) root_out_kernel(UtArgs A, RankBases R) {
  const bool s1 = blockIdx.y != 0;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int M = s1 ? A.M[1] : A.M[0];
  if (x <= R.B) {
    // ranks run over both sides' lists, the vertex side's after the faces'
    const int f = (s1 ? R.first[1] : R.first[0])[x];
    const int* rank = s1 ? A.rank[1] : A.rank[0];
    const bool end = f >= M;
    (s1 ? R.alive_base[1] : R.alive_base[0])[x] =
        !end ? rank[f] : s1 || A.M[1] == 0 ? R.total[0] : A.rank[1][0];
    if (!s1) {
      const int q = R.first_sad[x];
      R.surv_base[x] = q < R.nsad ? R.pos[q] : R.total[1];
      if (x == 0) {
        R.rb[0] = R.total[1];
        R.rb[1] = A.n_cancel[0];
        R.rb[2] = A.n_cancel[1];
        R.rb[3] = *A.status;
      }
    }
  }
  int* par = s1 ? A.par[1] : A.par[0];
  const int nt = gridDim.x * blockDim.x;
  int r[kUtBatch];
  unsigned live = 0, own = 0;
#pragma unroll
  for (int u = 0; u < kUtBatch; ++u) {
    const long long i = x + (long long)nt * u;
    r[u] = (int)i;
    if (i < M) own |= 1u << u;
  }
  live = own;
  for (int k = 0; live; ++k) {
    if (k > M) {  // a chain visits a node at most once: never reached
      set_status(A.status, kStatusFindCap);
      break;
    }
    int q[kUtBatch];
#pragma unroll
    for (int u = 0; u < kUtBatch; ++u) q[u] = ((live >> u) & 1u) ? par[r[u]] : r[u];
#pragma unroll
    for (int u = 0; u < kUtBatch; ++u) {
      if (q[u] == r[u]) live &= ~(1u << u);
      r[u] = q[u];
    }
  }
#pragma unroll
  for (int u = 0; u < kUtBatch; ++u) {
    if (!((own >> u) & 1u)) continue;
    const int i = x + nt * u;
    par[i] = r[u];
    (s1 ? A.rout[1] : A.rout[0])[i] = r[u] == M ? -1 : (s1 ? A.rank[1] : A.rank[0])[r[u]];
  }
}

}  // namespace dmsc
