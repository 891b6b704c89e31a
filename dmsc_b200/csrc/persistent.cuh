// Persistent cooperative kernels: the round loops of the pairing, the replay
// and the geometry expansion run entirely on the device, separated by
// grid-wide barriers, with no host round trip per round.
//
// Counters rotate over three slots: round r reads its input count from
// cnt[r % 3], appends its output to cnt[(r + 1) % 3] and clears
// cnt[(r + 2) % 3], which was last read at the top of round r - 1 (before the
// barrier that ended that round). Every loop is capped; hitting a cap sets a
// status bit the host turns into an error, and every thread leaves the loop at
// the same round because the loop condition reads the same counters.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "pairing.cuh"
#include "replay.cuh"

namespace dmsc {

namespace cg = cooperative_groups;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
constexpr int kTimeline = 64;  // timestamps kept per loop (round starts)
// The timeline buffer holds 6 loops' round start times, then each round's
// item count at the same position + kTimelineCounts, then the pairing's
// phase-B start times (faces, vertices) at kTimelinePhaseB.
constexpr int kTimelineCounts = 6 * kTimeline;
constexpr int kTimelinePhaseB = 12 * kTimeline;
constexpr int kTimelineSlots = 14 * kTimeline;

// Root of x in the pairing's group forest. A group links only under an
// older group (ages strictly decrease along links), so a search visits at
// most M + 1 nodes; the loop is capped at `cap` anyway and a cap sets
// kStatusFindCap and returns the node reached (a valid group).
__device__ __forceinline__ int find_halving(int* link, int x, int cap, unsigned* status) {
  for (int k = 0;; ++k) {
    int p = link[x];
    if (p == x) return x;
    if (k >= cap) {
      set_status(status, kStatusFindCap);
      return x;
    }
    int pp = link[p];
    if (pp != p) link[x] = pp;  // path halving: replaces a pointer with an ancestor
    x = pp;
  }
}

// Chunked processing with two output lists: each block takes contiguous
// chunks of items (up to kChunkPer per thread, fewer when there are few
// items, so small rounds still spread over the whole grid; no barrier between
// a thread's items); kept items are gathered in shared memory with shared
// atomics and written out once per chunk with one global reservation per
// list, so a block meets at a barrier a few times per chunk instead of after
// every item.
constexpr int kChunkPer = 8;
constexpr int kChunk = 256 * kChunkPer;  // blocks of 256 threads

struct ChunkLists {
  int n[2];
  int base[2];
  int buf[2][kChunk];
};

__device__ __forceinline__ long long chunk_size(long long n, int blocks) {
  const long long lanes = (long long)blocks * 256;
  return 256LL * max(1LL, min((long long)kChunkPer, (n + lanes - 1) / lanes));
}

// Loops whose active set has shrunk below a threshold leave the grid, whose
// barriers cost several microseconds each: the geometry expansion goes on in
// one block per side (the other blocks leave: all decide alike, from counts
// that are not written any more), the pairing hands over to a kernel that
// holds what is left of a side in one block's shared memory (pair_solo_kernel).
constexpr int kPairSoloEdges = 8192, kPairSoloNodes = 4096;  // per side
constexpr unsigned kSoloVoid = 0x7FFFu;                      // the void's node

__device__ __forceinline__ void chunk_start(ChunkLists& L) {
  if (threadIdx.x < 2) L.n[threadIdx.x] = 0;
  __syncthreads();
}

__device__ __forceinline__ void chunk_keep(ChunkLists& L, int side, int v) { L.buf[side][atomicAdd(&L.n[side], 1)] = v; }

__device__ __forceinline__ void chunk_flush(ChunkLists& L, int* cnt0, int* out0, int* cnt1, int* out1) {
  const int t = threadIdx.x;
  __syncthreads();
  if (t < 2 && L.n[t] > 0) L.base[t] = atomicAdd(t == 0 ? cnt0 : cnt1, L.n[t]);
  __syncthreads();
  for (int k = t; k < L.n[0]; k += 256) out0[L.base[0] + k] = L.buf[0][k];
  for (int k = t; k < L.n[1]; k += 256) out1[L.base[1] + k] = L.buf[1][k];
  __syncthreads();
}

// ---------------------------------------------------------------------------
// pairing rounds (see pairing.cuh for the algorithm)
// ---------------------------------------------------------------------------
struct PairArgs {
  int M;  // void group = M
  // saddles are indexed in list order (ascending cell id); a saddle's sweep
  // key (sweep_key) orders the saddles of its image in this side's sweep
  // and is the atomicMin key, so no sorted copy of the saddles is needed
  const float* sval;  // [nsad] saddle values
  const int* sad_img; // [nsad] image of each saddle
  int2* g12;          // [nsad] groups of the two ends, as of the saddle's last active round
  int* dying;
  int* link;                    // [M+1] group union-find
  unsigned long long* minedge;  // [M+1] smallest sweep key of the group's active saddles
  int* act0;          // active saddles (ping-pong)
  int* act1;
  int* roots0;        // live group roots (ping-pong), [M+1] each
  int* roots1;
  int* cnt;           // [0..2] rotating active counts, [3..5] rotating root counts
  const int2* key;       // [M] (value bits, cell) of each extremum
  const int* idx_base;   // [B + 1] first global index of each image
  int B;
  const uint8_t* dual;   // [B] orientation of each image
  bool faces;            // face side (maxima in the primal) or vertex side
  unsigned* status;
  int max_rounds;
  int* rounds;                   // receives the number of rounds (statistics)
  // what the grid hands over to the solo kernel: the round (-1: it reached its
  // cap), and the side's edges (sweep key; node | node << 16 | descending << 31)
  // and nodes, the live roots in list order
  int* handover;
  unsigned long long* solo_key;  // [kPairSoloEdges]
  uint32_t* solo_ends;           // [kPairSoloEdges]
  int2* solo_ext;                // [kPairSoloNodes] (value bits, cell)
  int* node;                     // [M] node of each live root
  unsigned long long* timeline;  // [kTimeline] round start times (ns), optional
};

// Both sides' persistence pairing in one cooperative launch; each round
// processes both sides' active saddles and live roots, so the two sides share
// their grid barriers. Per round and side: (A) every active saddle finds its
// ends' groups; those whose ends are in one group leave (cycles, whose
// decision is -1 from the start, and the saddles decided in the round before,
// whose ends are joined now), the rest reduce their sweep key into both
// groups' minimum (no returned value needed) and stay active; (B) every
// live root with an outgoing saddle decides whether it dies there, and a
// root that dies links itself under the other group's root at once (phase B
// reads no link, and the next reader is the next round's phase A, behind the
// round's barrier); the others stay live; roots without outgoing saddles
// leave for good. The rounds start from the saddles and roots that the tile
// pass (pair_tile_kernel) left undecided. The void is no list's member: it
// never dies, so nothing is reduced into it. A side with no active saddle
// just idles.
struct PairArgs2 {
  PairArgs s[2];
};

// Items a thread advances together in each phase (U): every load of a stage
// is issued for all of them before any is used, so a thread waits on U
// independent chains of dependent loads at once instead of one after the
// other (the stores and atomics between items would otherwise keep the
// compiler from overlapping them). Two shapes (tuned): U = 2 and U = 4, both
// with at most 4 resident blocks per SM (64 registers).
constexpr int kPairShapes = 2;

// Per-side fields picked by a flag (the parameter struct is only indexed
// with constants, so it stays in the constant bank).
#define PSIDE(f) (s1 ? P.s[1].f : P.s[0].f)

// Phase A for the thread's items i0 + 256 u (u < U) below cend of the active
// lists: side 0's items come first (i < n0); the saddles that stay active are
// appended to the next list.
template <int U>
__device__ __forceinline__ void pair_batch_a(const PairArgs2& P, int r, long long i0, long long cend, int n0,
                                             ChunkLists& L) {
  int e[U], ga[U], gb[U];
  float sv[U];
  unsigned act = 0, s1m = 0, du = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = i0 + 256LL * u;
    e[u] = 0;
    if (i < cend) {
      const bool s1 = i >= n0;
      const long long j = s1 ? i - n0 : i;
      act |= 1u << u;
      s1m |= (unsigned)s1 << u;
      e[u] = ((r & 1) ? PSIDE(act1) : PSIDE(act0))[j];
    }
  }
  int2 g[U];  // the ends' groups of the previous round
#pragma unroll
  for (int u = 0; u < U; ++u) {
    ga[u] = gb[u] = 0;
    g[u] = make_int2(0, 0);
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    g[u] = PSIDE(g12)[e[u]];
    ga[u] = g[u].x;
    gb[u] = g[u].y;
  }
  {
    // the groups' current roots: path-halving finds of all 2U ends in lockstep
    unsigned live = 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((act >> u) & 1u) live |= 3u << (2 * u);
    for (int it = 0; live; ++it) {
      if (it > P.s[0].M + P.s[1].M + 2) {  // ages strictly decrease along links: never reached
        set_status(P.s[0].status, kStatusFindCap);
        break;
      }
      int pa[2 * U], pp[2 * U];
#pragma unroll
      for (int c = 0; c < 2 * U; ++c) {
        const bool s1 = (s1m >> (c >> 1)) & 1u;
        const int x = (c & 1) ? gb[c >> 1] : ga[c >> 1];
        pa[c] = ((live >> c) & 1u) ? PSIDE(link)[x] : x;
      }
#pragma unroll
      for (int c = 0; c < 2 * U; ++c) {
        const bool s1 = (s1m >> (c >> 1)) & 1u;
        const int x = (c & 1) ? gb[c >> 1] : ga[c >> 1];
        if (pa[c] == x) live &= ~(1u << c);
        pp[c] = ((live >> c) & 1u) ? PSIDE(link)[pa[c]] : pa[c];
      }
#pragma unroll
      for (int c = 0; c < 2 * U; ++c) {
        if (!((live >> c) & 1u)) continue;
        const bool s1 = (s1m >> (c >> 1)) & 1u;
        int& x = (c & 1) ? gb[c >> 1] : ga[c >> 1];
        if (pp[c] == pa[c]) {  // pa is the root
          live &= ~(1u << c);
        } else {
          PSIDE(link)[x] = pp[c];  // path halving: replaces a pointer with an ancestor
        }
        x = pp[c];
      }
    }
  }
  // key values (loaded after the finds: fewer registers live across them)
#pragma unroll
  for (int u = 0; u < U; ++u) {
    sv[u] = 0.f;
    if (!((act >> u) & 1u) || ga[u] == gb[u]) continue;
    const bool s1 = (s1m >> u) & 1u;
    sv[u] = PSIDE(sval)[e[u]];
    const bool d = P.s[0].dual[P.s[0].B > 1 ? P.s[0].sad_img[e[u]] : 0];
    du |= (unsigned)(s1 ? d : !d) << u;  // descending sweep: faces in the primal, vertices in the dual
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    if (ga[u] == gb[u]) continue;  // a cycle, or decided in the previous round
    if (ga[u] != g[u].x || gb[u] != g[u].y) PSIDE(g12)[e[u]] = make_int2(ga[u], gb[u]);
    const unsigned long long k = sweep_key(sv[u], e[u], (du >> u) & 1u);
    if (ga[u] != PSIDE(M)) atomicMin(PSIDE(minedge) + ga[u], k);  // result unused: a reduction
    if (gb[u] != PSIDE(M)) atomicMin(PSIDE(minedge) + gb[u], k);
    chunk_keep(L, s1, e[u]);
  }
}

// Phase B for the thread's live roots k0 + 256 u (u < U) below cend (side 0's
// first, k < nr0): each root with an outgoing saddle decides there and a
// dying root links itself under the other group's root; roots without
// outgoing saddles leave for good. The roots that stay live are listed.
template <int U>
__device__ __forceinline__ void pair_batch_b(const PairArgs2& P, int r, long long k0, long long cend, int nr0,
                                             ChunkLists& L) {
  int g[U];
  unsigned act = 0, s1m = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long k = k0 + 256LL * u;
    g[u] = 0;
    if (k < cend) {
      const bool s1 = k >= nr0;
      const long long j = s1 ? k - nr0 : k;
      act |= 1u << u;
      s1m |= (unsigned)s1 << u;
      g[u] = ((r & 1) ? PSIDE(roots1) : PSIDE(roots0))[j];
    }
  }
  unsigned long long me[U];
  int2 kg[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    me[u] = kNoEdge;
    kg[u] = make_int2(0, 0);
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    me[u] = PSIDE(minedge)[g[u]];
    kg[u] = PSIDE(key)[g[u]];
  }
  int e[U];
  unsigned older_less = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    e[u] = 0;
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    if (me[u] == kNoEdge) {  // no outgoing saddle: leaves the list for good
      act &= ~(1u << u);
      continue;
    }
    PSIDE(minedge)[g[u]] = kNoEdge;
    // g is an extremum of one image; its image (from its cell) gives the
    // sweep direction of the key and the age order: value_less on the vertex
    // side in the primal and the face side in the dual
    const bool d = P.s[0].dual[find_image(P.s[0].idx_base, P.s[0].B, kg[u].y >> 2)];
    e[u] = sweep_key_saddle(me[u], s1 ? d : !d);
    older_less |= (unsigned)(s1 ? !d : d) << u;
  }
  int h[U];
  unsigned sec = 0;  // the root's end is the saddle's second
#pragma unroll
  for (int u = 0; u < U; ++u) {
    h[u] = 0;
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    const int2 gg = PSIDE(g12)[e[u]];  // roots as of phase A
    h[u] = gg.x == g[u] ? gg.y : gg.x;
    sec |= (unsigned)(gg.x != g[u]) << u;
  }
  int2 kh[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    kh[u] = make_int2(0, 0);
    const bool s1 = (s1m >> u) & 1u;
    if (((act >> u) & 1u) && h[u] < PSIDE(M)) kh[u] = PSIDE(key)[h[u]];
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    // h older than g: the void is older than any extremum; else (value, cell)
    // under the side's order
    bool dies = h[u] == PSIDE(M);
    if (!dies) {
      const float vh = __int_as_float(kh[u].x), vg = __int_as_float(kg[u].x);
      dies = ((older_less >> u) & 1u) ? tie_lt(vh, kh[u].y, vg, kg[u].y) : tie_lt(vg, kg[u].y, vh, kh[u].y);
    }
    if (dies) {
      PSIDE(dying)[e[u]] = dying_word(g[u], (sec >> u) & 1u);
      PSIDE(link)[g[u]] = h[u];
    } else {
      chunk_keep(L, s1, g[u]);
    }
  }
}
#undef PSIDE

template <int U, int MINB>
__global__ void __launch_bounds__(256, MINB) pairing_persistent_kernel(PairArgs2 P) {
  __shared__ ChunkLists L;
  cg::grid_group grid = cg::this_grid();
  const long long tid = grid.thread_rank();
  const int bid = (int)blockIdx.x, nblk = (int)gridDim.x;
  bool done0 = false, done1 = false;
  for (int r = 0;; ++r) {
    const int n0 = *(volatile int*)(P.s[0].cnt + r % 3), n1 = *(volatile int*)(P.s[1].cnt + r % 3);
    // a side whose active list is empty is finished: its roots are not visited
    const int nr0 = n0 ? *(volatile int*)(P.s[0].cnt + 3 + r % 3) : 0;
    const int nr1 = n1 ? *(volatile int*)(P.s[1].cnt + 3 + r % 3) : 0;
    if (tid == 0) {
      for (int sd = 0; sd < 2; ++sd) {
        const PairArgs& A = P.s[sd];
        const int n = sd ? n1 : n0;
        bool& done = sd ? done1 : done0;
        if (A.timeline && r < kTimeline && !done) {
          A.timeline[r] = global_ns();
          A.timeline[kTimelineCounts + r] = n;
        }
        if (n == 0 && !done && A.rounds) *A.rounds = r;
        done = done || n == 0;
      }
    }
    // both sides fit the solo kernel (or are finished): the whole grid digests
    // the edges and nodes for it (one block gathering them alone took 35 us)
    // and every thread leaves
    if (n0 <= kPairSoloEdges && n1 <= kPairSoloEdges && nr0 <= kPairSoloNodes && nr1 <= kPairSoloNodes) {
      if (tid == 0) *P.s[0].handover = r;
      if (n0 == 0 && n1 == 0) break;
      for (long long j = tid; j < nr0 + nr1; j += grid.size()) {
        const PairArgs& A = j < nr0 ? P.s[0] : P.s[1];
        const int i = (int)(j < nr0 ? j : j - nr0);
        const int g = ((r & 1) ? A.roots1 : A.roots0)[i];
        A.node[g] = i;
        A.solo_ext[i] = A.key[g];
      }
      grid.sync();
      for (long long j = tid; j < n0 + n1; j += grid.size()) {
        const bool s1 = j >= n0;
        const PairArgs& A = s1 ? P.s[1] : P.s[0];
        const int k = (int)(s1 ? j - n0 : j), s = ((r & 1) ? A.act1 : A.act0)[k];
        const int2 e = A.g12[s];
        const float v = A.sval[s];
        const bool d = A.dual[A.B > 1 ? A.sad_img[s] : 0], desc = s1 ? d : !d;
        const int a = find_halving(A.link, e.x, A.M + 2, A.status), b = find_halving(A.link, e.y, A.M + 2, A.status);
        A.solo_key[k] = sweep_key(v, s, desc);
        A.solo_ends[k] = (a == A.M ? kSoloVoid : (unsigned)A.node[a]) | (b == A.M ? kSoloVoid : (unsigned)A.node[b]) << 16 |
                         (unsigned)desc << 31;
      }
      break;
    }
    if (r >= max(P.s[0].max_rounds, P.s[1].max_rounds)) {
      // every thread leaves here in the same round (the counters it read are
      // the same); saddles still undecided stay cycles (-1), so the kernels
      // that run before the host sees the status read valid extremum indices
      if (tid == 0) {
        set_status(P.s[0].status, kStatusRoundCap);
        *P.s[0].handover = -1;
      }
      break;
    }
    if (tid == 0) {
      for (int sd = 0; sd < 2; ++sd) {
        P.s[sd].cnt[(r + 2) % 3] = 0;
        P.s[sd].cnt[3 + (r + 2) % 3] = 0;
      }
    }
    {  // phase A: both sides' active saddles
      const long long n = (long long)n0 + n1, chunk = chunk_size(n, nblk);
      for (long long c0 = (long long)bid * chunk; c0 < n; c0 += (long long)nblk * chunk) {
        chunk_start(L);
        const long long cend = min(n, c0 + chunk);
        for (long long i0 = c0 + threadIdx.x; i0 < cend; i0 += 256LL * U) pair_batch_a<U>(P, r, i0, cend, n0, L);
        chunk_flush(L, P.s[0].cnt + (r + 1) % 3, (r & 1) ? P.s[0].act0 : P.s[0].act1, P.s[1].cnt + (r + 1) % 3,
                    (r & 1) ? P.s[1].act0 : P.s[1].act1);
      }
    }
    grid.sync();
    if (tid == 0 && r < kTimeline)  // side sd's phase-B starts: block 12 + sd
      for (int sd = 0; sd < 2; ++sd)
        if (P.s[sd].timeline) P.s[sd].timeline[kTimelinePhaseB + r] = global_ns();
    {  // phase B: live roots decide on their first outgoing saddle
      const long long n = (long long)nr0 + nr1, chunk = chunk_size(n, nblk);
      for (long long c0 = (long long)bid * chunk; c0 < n; c0 += (long long)nblk * chunk) {
        chunk_start(L);
        const long long cend = min(n, c0 + chunk);
        for (long long k0 = c0 + threadIdx.x; k0 < cend; k0 += 256LL * U) pair_batch_b<U>(P, r, k0, cend, nr0, L);
        chunk_flush(L, P.s[0].cnt + 3 + (r + 1) % 3, (r & 1) ? P.s[0].roots0 : P.s[0].roots1,
                    P.s[1].cnt + 3 + (r + 1) % 3, (r & 1) ? P.s[1].roots0 : P.s[1].roots1);
      }
    }
    grid.sync();
  }
}

// The pairing's last rounds, one block per side: the saddles and live roots
// that the grid (or the tile pass) left, held in shared memory. A round costs
// a few block barriers and shared-memory reads here, 12 to 16 us with grid
// barriers and dependent global loads, however few its saddles are. Phase B
// runs over the edges: the one whose (unique) key is its root's minimum
// decides for that root and clears the minimum.
constexpr int kSoloNT = 1024, kSoloList = kPairSoloEdges / (kSoloNT / 32);

struct PairSoloSmem {
  unsigned long long minedge[kPairSoloNodes];
  unsigned long long key[kPairSoloEdges];  // sweep key of each edge
  uint32_t ends[kPairSoloEdges];           // node | node << 16 | descending sweep << 31
  int2 ext[kPairSoloNodes];                // (value bits, cell) of each node
  int rank[kPairSoloNodes];
  uint16_t link[kPairSoloNodes];
  uint16_t list[kSoloNT / 32][kSoloList];  // each warp's undecided edges
};

__device__ __forceinline__ unsigned solo_root(volatile uint16_t* link, unsigned x) {
  if (x == kSoloVoid) return x;
  unsigned p = link[x];
  for (int k = 0; k <= kPairSoloNodes; ++k) {  // links never form a cycle
    if (p == x || p == kSoloVoid) return p;
    const unsigned pp = link[p];
    if (pp == p) return p;
    link[x] = (uint16_t)pp;
    if (pp == kSoloVoid) return pp;
    x = pp;
    p = link[x];
  }
  return x;
}

__global__ void __launch_bounds__(kSoloNT) pair_solo_kernel(PairArgs2 P) {
  extern __shared__ __align__(16) unsigned char pair_solo_smem[];
  PairSoloSmem& S = *reinterpret_cast<PairSoloSmem*>(pair_solo_smem);
  const bool s1 = blockIdx.x != 0;
  const PairArgs& A = s1 ? P.s[1] : P.s[0];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int r0 = *P.s[0].handover;
  if (r0 < 0) return;  // the grid reached its cap
  const int ne = A.cnt[r0 % 3], nr = A.cnt[3 + r0 % 3];
  if (ne == 0) return;
  const int* roots = (r0 & 1) ? A.roots1 : A.roots0;
  for (int i = tid; i < nr; i += kSoloNT) {
    S.rank[i] = roots[i];
    S.ext[i] = A.solo_ext[i];
    S.minedge[i] = kNoEdge;
    S.link[i] = (uint16_t)i;
  }
  // edges in chunks of 32, chunk c to warp c % 32
  uint16_t* const list = S.list[warp];
  int n = 0;
  for (int c = warp; c * 32 < ne; c += kSoloNT / 32) {
    const int k = c * 32 + lane;
    if (k < ne) {
      S.key[k] = A.solo_key[k];
      S.ends[k] = A.solo_ends[k];
      list[n + lane] = (uint16_t)k;
    }
    n += min(32, ne - c * 32);
  }
  const int max_rounds = max(P.s[0].max_rounds, P.s[1].max_rounds);
  int r = r0;
  while (__syncthreads_or(n > 0)) {
    if (r >= max_rounds) {  // what is undecided stays a cycle (-1)
      if (tid == 0) set_status(A.status, kStatusRoundCap);
      break;
    }
    if (tid == 0 && A.timeline && r < kTimeline && r > r0) A.timeline[r] = global_ns();
    // phase A
    int kept = 0;
    for (int q0 = 0; q0 < n; q0 += 32) {
      bool keep = false;
      int k = 0;
      if (q0 + lane < n) {
        k = list[q0 + lane];
        const uint32_t e = S.ends[k];
        const unsigned a = solo_root(S.link, e & 0x7FFFu), b = solo_root(S.link, (e >> 16) & 0x7FFFu);
        keep = a != b;  // else a cycle, or decided in the previous round
        if (keep) {
          S.ends[k] = a | b << 16 | (e & 0x80000000u);
          const unsigned long long m = S.key[k];
          if (a != kSoloVoid && m < *(volatile unsigned long long*)&S.minedge[a]) atomicMin(&S.minedge[a], m);
          if (b != kSoloVoid && m < *(volatile unsigned long long*)&S.minedge[b]) atomicMin(&S.minedge[b], m);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      __syncwarp();  // the chunk is read before its slots are written again
      if (keep) list[kept + __popc(m & lt)] = (uint16_t)k;
      kept += __popc(m);
    }
    n = kept;
    __syncthreads();
    // phase B (the list is the warp's own: no barrier is needed before it)
    for (int q = lane; q < n; q += 32) {
      const int k = list[q];
      const uint32_t e = S.ends[k];
      const unsigned long long m = S.key[k];
      const bool older_less = !(e >> 31);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const unsigned g = (j ? e >> 16 : e) & 0x7FFFu, h = (j ? e : e >> 16) & 0x7FFFu;
        if (g == kSoloVoid || *(volatile unsigned long long*)&S.minedge[g] != m) continue;
        S.minedge[g] = kNoEdge;
        if (h != kSoloVoid) {
          const int2 kh = S.ext[h], kg = S.ext[g];
          const float vh = __int_as_float(kh.x), vg = __int_as_float(kg.x);
          if (!(older_less ? tie_lt(vh, kh.y, vg, kg.y) : tie_lt(vg, kg.y, vh, kh.y))) continue;
        }
        A.dying[sweep_key_saddle(m, e >> 31)] = dying_word(S.rank[g], j != 0);
        S.link[g] = (uint16_t)h;
      }
    }
    ++r;
  }
  if (tid == 0 && A.rounds) *A.rounds = r;
  if (tid == 0 && A.timeline && r < kTimeline && r > r0) A.timeline[r] = global_ns();
}

// ---------------------------------------------------------------------------
// replay rounds (see replay.cuh)
// ---------------------------------------------------------------------------
struct ReplayArgs {
  const int* n_cancel;               // device count of cancellations
  const unsigned long long* key;     // [C] replay key of each cancellation
  const int* cj;                     // [C] saddle (list index) of each cancellation
  const int* dying;  // [nsad] in saddle list order
  const int4* arc;   // {end 0, end 1, raw-arc cells 0, raw-arc cells 1} of each saddle, list order (every second record)
  const uint8_t* alive;  // [M] extrema that no cancellation kills (their records are never read)
  const int* crit_sad;   // [nsad] global cell id of each saddle
  ReplayState S;
  int max_steps;
  int* act0;
  int* act1;
  int* cnt;  // [0..2]
  int* wx;         // [2C] position of each cancellation's two walks
  long long* wa;   // [2C] path length summed so far by each walk
  unsigned* status;
  int max_rounds;
  int* rounds;
  unsigned long long* timeline;  // [kTimeline] round start times (ns), optional
};

// Rounds of cancellation resolution (replay.cuh) for both sides in one
// cooperative launch (a side with n_cancel == nullptr takes no part). The
// cancellations are in collection order; their keys order the replay.
struct ReplayArgs2 {
  ReplayArgs s[2];
};

// A round that holds every pending cancellation in a thread of its own lets
// the walks wait for the decisions they need instead of ending the round:
// each wait is a re-read of under a microsecond, against 10 to 20 us for a
// round. Measured, the replay stage with rounds only and with waits: 0.37 ->
// 0.14 ms on a 1080 x 1920 field of 256 levels (30 rounds before), 0.34 -> 0.24
// at 2048^2, threshold 0.25, 0.91 -> 0.80 at 4096^2, 0.085 -> 0.045 at 256^2.
// The first round and the rounds with more items than threads do not wait: a
// decision there is as often many strides away (4 looks: 1.16 ms at 4096^2).
constexpr int kReplayWait = 256;

// One batch of a thread's pending cancellations, the items i0 + nt u (u < U)
// below n (side 0's first, i < na): both walks of every item resume where the
// previous round left them and advance in lockstep (2U independent chains of
// node loads at once), then the item decides (link or skip). An item with a
// walk that meets an undecided node keeps its walks' positions and stays
// pending for the next round. With WAIT such a walk looks at the node again,
// up to kReplayWait times, and an item decides inside the loop, as soon as
// both its walks have ended, so that lanes of its own warp may wait for it.
#define RSIDE(f) (s1 ? P.s[1].f : P.s[0].f)
template <int U, bool WAIT>
__device__ __forceinline__ void replay_batch(const ReplayArgs2& P, int rd, long long i0, long long nt,
                                             long long n, int na, ChunkLists& L) {
  int r[U];
  unsigned act = 0, s1m = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = i0 + nt * u;
    r[u] = 0;
    if (i < n) {
      const bool s1 = i >= na;
      act |= 1u << u;
      s1m |= (unsigned)s1 << u;
      const long long j = s1 ? i - na : i;
      r[u] = rd == 0 ? (int)j : ((rd & 1) ? RSIDE(act1) : RSIDE(act0))[j];
    }
  }
  unsigned long long tk[U];
  int sd[U], x[2 * U];
  long long a[2 * U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    tk[u] = 0;
    sd[u] = 0;
    x[2 * u] = x[2 * u + 1] = -1;
    a[2 * u] = a[2 * u + 1] = 0;
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    tk[u] = RSIDE(key)[r[u]];
    sd[u] = RSIDE(cj)[r[u]];
    if (rd > 0) {  // resume where the previous round left the walks
      const int2 w = *reinterpret_cast<const int2*>(RSIDE(wx) + 2 * r[u]);
      const longlong2 aa = *reinterpret_cast<const longlong2*>(RSIDE(wa) + 2 * r[u]);
      x[2 * u] = w.x;
      x[2 * u + 1] = w.y;
      a[2 * u] = aa.x;
      a[2 * u + 1] = aa.y;
    }
  }
  if (rd == 0) {  // the walks start at the saddle's arc ends
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((act >> u) & 1u)) continue;
      const bool s1 = (s1m >> u) & 1u;
      const int4 w = RSIDE(arc)[2 * (long long)sd[u]];
      x[2 * u] = w.x;
      x[2 * u + 1] = w.y;
    }
  }
  int d[U];  // the dying node (issued before the walks, used after them)
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const bool s1 = (s1m >> u) & 1u;
    d[u] = ((act >> u) & 1u) ? dying_of(RSIDE(dying)[sd[u]]) : 0;
  }
  // bit c of `live` is a walk that has not ended (the root as of the step's
  // key is not reached), bit c of `wait` one that met an undecided node
  unsigned live = 0;
#pragma unroll
  for (int c = 0; c < 2 * U; ++c)
    if (((act >> (c >> 1)) & 1u) && x[c] >= 0) live |= 1u << c;
  auto decide = [&](int u) {
    act &= ~(1u << u);
    const bool s1 = (s1m >> u) & 1u;
    const int R0 = x[2 * u], R1 = x[2 * u + 1], dd = d[u], s = sd[u];
    const long long a0 = a[2 * u], a1 = a[2 * u + 1];
    int k = -1;
    if (R0 == dd && R0 != R1)
      k = 0;
    else if (R1 == dd && R0 != R1)
      k = 1;
    ReplayNode* node = RSIDE(S.node);
    if (k >= 0) {
      const int4 ar = RSIDE(arc)[2 * (long long)s];
      *reinterpret_cast<longlong2*>(&node[dd].cl_dy) = make_longlong2(k == 0 ? a0 : a1, k == 0 ? a1 : a0);
      *reinterpret_cast<int4*>(&node[dd].t_dy) =
          make_int4(k == 0 ? ar.x : ar.y, k == 0 ? ar.y : ar.x, k == 0 ? ar.z : ar.w, k == 0 ? ar.w : ar.z);
      // the dying side with what W(d) expands to (its non-empty chains and
      // raw-arc segments), and the saddle
      *reinterpret_cast<int2*>(&node[dd].side) =
          make_int2(side_word(k, (a0 > 0) + (a1 > 0), (ar.z > 0) + (ar.w > 0)), RSIDE(crit_sad)[s]);
      node_link_set(node, dd, NodeLink{kLinked, k == 0 ? R1 : R0, (long long)ar.z + ar.w + a0 + a1});
    } else {
      node_link_set(node, dd, NodeLink{kRootForever, -1, 0});
    }
  };
  // a chain is at most its side's node count long (a side without arcs takes
  // no part and has no bound of its own)
  const int cap = max(P.s[0].max_steps, P.s[1].max_steps);
  int steps = 0, waited = 0;
  while (true) {
    unsigned long long key[2 * U];
    NodeLink w[2 * U];
    bool al[2 * U];
#pragma unroll
    for (int c = 0; c < 2 * U; ++c) {
      const bool s1 = (s1m >> (c >> 1)) & 1u;
      if ((live >> c) & 1u) {  // the alive flag and the record's sector, issued together
        al[c] = RSIDE(alive)[x[c]];
        key[c] = __ldcg(&RSIDE(S.node)[x[c]].ctime);
        w[c] = node_link_live(RSIDE(S.node), x[c]);
      }
    }
    unsigned wait = 0;
#pragma unroll
    for (int c = 0; c < 2 * U; ++c) {
      if (!((live >> c) & 1u)) continue;
      // never cancelled (its record is not written), or not linked before
      // this step: the root
      if (al[c] || key[c] >= tk[c >> 1]) {
        live &= ~(1u << c);
        continue;
      }
      if (w[c].status == kPending) {
        wait |= 1u << c;
        continue;
      }
      if (w[c].status == kRootForever) {
        live &= ~(1u << c);
        continue;
      }
      a[c] += w[c].wlen;
      x[c] = w[c].parent;
      if (x[c] < 0) live &= ~(1u << c);
    }
    if (WAIT) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (((act >> u) & 1u) && !((live >> (2 * u)) & 3u)) decide(u);
      if (!act) return;
      if (wait == live && ++waited >= kReplayWait) break;  // only waiting walks are left
    } else if (wait == live) {
      break;
    }
    if (++steps > 2 * U * (cap + 1) + kReplayWait) {
      set_status(P.s[0].status, kStatusChainCap);
      break;
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!WAIT && ((act >> u) & 1u) && !((live >> (2 * u)) & 3u)) decide(u);
    if (!((act >> u) & 1u)) continue;
    const bool s1 = (s1m >> u) & 1u;
    *reinterpret_cast<int2*>(RSIDE(wx) + 2 * r[u]) = make_int2(x[2 * u], x[2 * u + 1]);
    *reinterpret_cast<longlong2*>(RSIDE(wa) + 2 * r[u]) = make_longlong2(a[2 * u], a[2 * u + 1]);
    chunk_keep(L, s1, r[u]);
  }
}
#undef RSIDE

// Replay shapes (tuned): U = 1 with 4 resident blocks per SM (64 registers,
// which spill 32 bytes; with 3 the stage takes 0.806 ms too at 4096^2, and 0.163
// instead of 0.150 on 1080 x 1920 pixels of 256 levels), U = 2 with 3.
constexpr int kReplayShapes = 2;

template <int U, int MINB>
__global__ void __launch_bounds__(256, MINB) replay_persistent_kernel(ReplayArgs2 P) {
  __shared__ ChunkLists L;
  cg::grid_group grid = cg::this_grid();
  const long long tid = grid.thread_rank(), nth = grid.size();
  for (int sd = 0; sd < 2; ++sd) {
    const ReplayArgs& A = P.s[sd];
    if (!A.n_cancel) continue;
    const int C = *A.n_cancel;
    // the killed nodes' records hold their keys (written by the persistence
    // pass); round 0 takes every cancellation with its walks starting at the
    // saddle's arc ends (no list or walk state yet)
    if (tid == 0) {
      A.cnt[0] = C;
      A.cnt[1] = 0;
      A.cnt[2] = 0;
    }
  }
  grid.sync();
  bool done0 = false, done1 = false;
  for (int rd = 0;; ++rd) {
    const int na = P.s[0].n_cancel ? *(volatile int*)(P.s[0].cnt + rd % 3) : 0;
    const int nb = P.s[1].n_cancel ? *(volatile int*)(P.s[1].cnt + rd % 3) : 0;
    if (tid == 0) {
      if (P.s[0].n_cancel && !done0) {
        if (P.s[0].timeline && rd < kTimeline) {
          P.s[0].timeline[rd] = global_ns();
          P.s[0].timeline[kTimelineCounts + rd] = na;
        }
        if (na == 0 && P.s[0].rounds) *P.s[0].rounds = rd;
      }
      if (P.s[1].n_cancel && !done1) {
        if (P.s[1].timeline && rd < kTimeline) {
          P.s[1].timeline[rd] = global_ns();
          P.s[1].timeline[kTimelineCounts + rd] = nb;
        }
        if (nb == 0 && P.s[1].rounds) *P.s[1].rounds = rd;
      }
    }
    done0 = done0 || na == 0;
    done1 = done1 || nb == 0;
    const long long n = (long long)na + nb;
    if (n == 0) break;
    if (rd >= max(P.s[0].max_rounds, P.s[1].max_rounds)) {
      if (tid == 0) set_status(P.s[0].n_cancel ? P.s[0].status : P.s[1].status, kStatusRoundCap);
      // the cancellations still pending are dropped (their dying nodes
      // become roots), so the chain walks of the kernels that run before the
      // host sees the status meet decided nodes only
      for (long long i = tid; i < n; i += nth) {
        const ReplayArgs& A = i < na ? P.s[0] : P.s[1];
        const long long k = i < na ? i : i - na;
        const int r = rd == 0 ? (int)k : ((rd & 1) ? A.act1 : A.act0)[k];
        A.S.node[dying_of(A.dying[A.cj[r]])].status = kRootForever;
      }
      break;
    }
    if (tid == 0)
      for (int sd = 0; sd < 2; ++sd)
        if (P.s[sd].n_cancel) P.s[sd].cnt[(rd + 2) % 3] = 0;
    // grid-stride over both sides' pending cancellations (the grid works on
    // neighbouring ones at any time, which keeps their nodes in L2: contiguous
    // chunks per block took 366 us instead of 252 for the first round at
    // 4096^2), with one reservation per kChunkPer strides
    const bool wait = rd > 0 && n <= nth;
    for (long long base = 0; base < n; base += nth * kChunkPer) {
      chunk_start(L);
      const long long end = min(n, base + nth * kChunkPer);
      for (long long i0 = base + tid; i0 < end; i0 += nth * U)
        if (wait)
          replay_batch<U, true>(P, rd, i0, nth, end, na, L);
        else
          replay_batch<U, false>(P, rd, i0, nth, end, na, L);
      chunk_flush(L, P.s[0].cnt + (rd + 1) % 3, (rd & 1) ? P.s[0].act0 : P.s[0].act1, P.s[1].cnt + (rd + 1) % 3,
                  (rd & 1) ? P.s[1].act0 : P.s[1].act1);
    }
    grid.sync();
  }
}

// ---------------------------------------------------------------------------
// geometry expansion levels (see replay.cuh)
// ---------------------------------------------------------------------------
struct EmitArgs {
  EmitCtx E;
  int nsurv;
  int4* q0;
  int4* q1;
  int* cnt;  // [8] level counts at emit_slot, raw-arc segment count at kEmitSegs
  int max_levels;
  int* levels;                   // receives the number of levels (statistics)
  unsigned long long* timeline;  // [kTimeline] level start times (ns), optional
};
// Both sides; a side with no geometry has cnt == nullptr.
struct EmitArgs2 {
  EmitArgs s[2];
};

// Where level `lv` counts its tasks: three rotating slots for the levels of the
// whole grid and three others for the last levels, which one block per side
// goes through alone (solo) while the blocks that leave may still be reading
// the last count of the grid's. That one is not written again: a block that
// found it changed could stay and wait for the others for good.
constexpr int kEmitSegs = 3;
__host__ __device__ constexpr int emit_slot(int lv, bool solo) { return lv % 3 + (solo ? kEmitSegs + 1 : 0); }

// One batch of a thread's chain tasks at one expansion level, in[i0 + nt u]
// (u < U) below n: the U chains are counted in lockstep (one node-record load
// per chain and step), the batch reserves its chain tasks and raw-arc
// segments with one block reservation, and the U chains are expanded in
// lockstep: per step, every chain issues its node's loads, then the loads of
// the node's saddle (arc ends and raw-arc lengths), then writes W(node)
// (chain_expand / emit_w, replay.cuh).
template <int U>
__device__ __forceinline__ void emit_batch(const EmitCtx& E, int4* __restrict__ q_out, int* n_out, int* n_base,
                                           const int4* __restrict__ in, long long i0, long long nt, long long n) {
  int x[U], stop[U], z[U], nc[U], nb[U];
  long long pos[U], tot[U];
  unsigned act = 0, rev = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = i0 + nt * u;
    x[u] = stop[u] = -1;
    pos[u] = 0;
    if (i < n) {  // every queued task is a chain task
      const int4 t = in[i];
      if ((t.x & 3) == kTaskChain) {
        act |= 1u << u;
        rev |= (unsigned)((t.x >> 2) & 1) << u;
        x[u] = t.y;
        stop[u] = t.z;
        pos[u] = t.w;
      }
    }
    z[u] = x[u];
    nc[u] = nb[u] = 0;
    tot[u] = 0;
  }
  // counts and total length of each chain (chain_expand_counts)
  unsigned live = 0;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (((act >> u) & 1u) && z[u] != stop[u] && z[u] >= 0) live |= 1u << u;
  for (int k = 0; live; ++k) {
    if (k > E.max_steps) {  // a chain is at most the side's node count long
      set_status(E.status, kStatusChainCap);
      act &= ~live;  // the capped tasks are dropped
      break;
    }
    NodeLink l[U];
    int2 w[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((live >> u) & 1u) {
        l[u] = node_link(E.S.node, z[u]);
        w[u] = node_words(E.S.node, z[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((live >> u) & 1u) {
        tot[u] += l[u].wlen;
        nc[u] += chains_of(w[u].x);  // counts stored at link time
        nb[u] += bases_of(w[u].x);
        z[u] = l[u].parent;
        if (z[u] == stop[u] || z[u] < 0) live &= ~(1u << u);
      }
  }
  int need = 0, nbase = 0;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if ((act >> u) & 1u) {
      need += nc[u];
      nbase += nb[u];
    }
  int p, pb;
  block_reserve2(n_out, need, n_base, nbase, p, pb);
  if (p + (long long)need > E.q_cap || pb + (long long)nbase > E.base_cap) {
    set_status(E.status, kStatusQueueOverflow);
    return;
  }
  // expansion: the slots of chain u follow those of the chains before it
  int pc[U], pbc[U];
  long long off[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    pc[u] = p;
    pbc[u] = pb;
    if ((act >> u) & 1u) {
      p += nc[u];
      pb += nb[u];
    }
    z[u] = x[u];
    off[u] = 0;
  }
  live = 0;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (((act >> u) & 1u) && z[u] != stop[u] && z[u] >= 0) live |= 1u << u;
  while (live) {
    NodeLink l[U];
    int2 w[U];   // (side, saddle)
    int4 te[U];  // (arc ends, raw-arc lengths)
    longlong2 cl[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((live >> u) & 1u) {  // the node's two sectors, issued together
        const ReplayNode* nd = E.S.node + z[u];
        w[u] = node_words(E.S.node, z[u]);
        l[u] = node_link(E.S.node, z[u]);
        cl[u] = *reinterpret_cast<const longlong2*>(&nd->cl_dy);
        te[u] = *reinterpret_cast<const int4*>(&nd->t_dy);
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((live >> u) & 1u)) continue;
      // W(z) = reverse(chain(Tk -> z)) + reverse(arc k) + arc o + chain(To -> R)
      const int d = z[u], k = side_of(w[u].x), s = w[u].y, R = l[u].parent;  // s: the saddle's cell
      const int Tk = te[u].x, To = te[u].y;
      const long long la = cl[u].x, lb = te[u].z, lc = te[u].w, ld = cl[u].y;
      const bool rv = (rev >> u) & 1u;
      const long long at = rv ? pos[u] + tot[u] - off[u] - l[u].wlen : pos[u] + off[u];
      int& q = pc[u];
      int& qb = pbc[u];
      if (!rv) {
        if (la > 0) q_out[q++] = make_task(kTaskChain, 1, Tk, d, at);
        if (lb > 0) E.base_q[qb++] = make_saddle_seg(s, k, 1, lb, at + la);
        if (lc > 0) E.base_q[qb++] = make_saddle_seg(s, 1 - k, 0, lc, at + la + lb);
        if (ld > 0) q_out[q++] = make_task(kTaskChain, 0, To, R, at + la + lb + lc);
      } else {
        if (ld > 0) q_out[q++] = make_task(kTaskChain, 1, To, R, at);
        if (lc > 0) E.base_q[qb++] = make_saddle_seg(s, 1 - k, 1, lc, at + ld);
        if (lb > 0) E.base_q[qb++] = make_saddle_seg(s, k, 0, lb, at + ld + lc);
        if (la > 0) q_out[q++] = make_task(kTaskChain, 0, Tk, d, at + ld + lc + lb);
      }
      off[u] += l[u].wlen;
      z[u] = l[u].parent;
      if (z[u] == stop[u] || z[u] < 0) live &= ~(1u << u);
    }
  }
}
// Expansion shapes (tuned): U = 1 with 4 resident blocks per SM (without
// spills; geometry with 5, 4 and 3: 0.417, 0.390 and 0.384 ms on 1080 x 1920
// pixels of 256 levels, 0.954, 0.945 and 0.986 at 4096^2), U = 2 with 3.
constexpr int kEmitShapes = 2;

// Geometry: breadth-first expansion of both sides' chain and W tasks
// (replay.cuh), collecting the raw-arc segments with their output positions.
// Levels are chain depths and most are bound by the latency of their longest
// chain, so the two sides share every level (and its grid barrier): at each
// level the blocks are split between them by their task counts, and a level's
// tasks go to the warps of all its blocks, 32 at a time. The geometry stage
// with a launch per side and together: 0.344 -> 0.182 ms at 2048^2, threshold
// 0.25, 0.187 -> 0.106 at 256^2, 0.573 -> 0.420 on 1080 x 1920 pixels of 256
// levels, 1.10 -> 0.98 at 4096^2, threshold 0.05.
template <int U, int MINB>
__global__ void __launch_bounds__(256, MINB) emit_persistent_kernel(EmitArgs2 P) {
  cg::grid_group grid = cg::this_grid();
  const long long tid = grid.thread_rank();
  if (tid < 16) {
    const EmitArgs& A = tid < 8 ? P.s[0] : P.s[1];
    if (A.cnt) A.cnt[tid & 7] = 0;
  }
  grid.sync();
  // level 0: the chain of each surviving arc (its own raw arc is a segment
  // item of the writer, read from the survivor records). A block takes
  // kLevel0 survivors per thread at a time: it counts their chains, reserves
  // queue slots once for all of them and then writes the tasks, so the
  // blocks queue on the shared counter once per 4096 arcs instead of once
  // per 256 (each reservation waits on the atomic's return).
  constexpr int kLevel0 = 8;
  const long long span = (long long)blockDim.x * kLevel0;
#pragma unroll 1
  for (int sd = 0; sd < 2; ++sd) {
    const EmitArgs& A = sd ? P.s[1] : P.s[0];
    const EmitCtx& E = A.E;
    if (!A.cnt) continue;
    for (long long base = (long long)blockIdx.x * span; base < A.nsurv; base += (long long)gridDim.x * span) {
      // a chain exists only on arcs that the image's output takes (length 0 otherwise)
      int mine = 0;
#pragma unroll
      for (int k = 0; k < kLevel0; ++k) {
        const long long i = base + (long long)k * blockDim.x + threadIdx.x;
        if (i >= A.nsurv) continue;
        const int2 cl = *reinterpret_cast<const int2*>(E.fin + i);
        mine += (cl.x > 0) + (cl.y > 0);
      }
      // most arcs have no chain (at threshold 0 nearly all): a block reserves
      // queue slots only when one of its threads has a task
      if (!__syncthreads_or(mine > 0)) continue;
      int p, pb;
      block_reserve2(A.cnt + emit_slot(0, false), mine, A.cnt + kEmitSegs, 0, p, pb);
      if (mine == 0) continue;
      for (int k = 0; k < kLevel0; ++k) {
        const long long i = base + (long long)k * blockDim.x + threadIdx.x;
        if (i >= A.nsurv) break;
        const int4 fin = E.fin[i];
        if (fin.x <= 0 && fin.y <= 0) continue;
        const int4 a = E.arc[i];
        const int pos = surv_start(E, (int)i, E.head[i].img);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if ((j ? fin.y : fin.x) <= 0) continue;
          if (p < E.q_cap)
            A.q0[p] = make_task(kTaskChain, 0, j ? a.y : a.x, j ? fin.w : fin.z, pos + a.z + (j ? fin.x + a.w : 0));
          else
            set_status(E.status, kStatusQueueOverflow);
          ++p;
        }
      }
    }
  }
  grid.sync();
  bool solo = false, done[2] = {false, false};
  for (int lv = 0;; ++lv) {
    int n[2];
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const EmitArgs& A = sd ? P.s[1] : P.s[0];
      // in the solo levels the other side's counters are its own block's
      n[sd] = A.cnt && !(solo && (int)blockIdx.x != sd) ? *(volatile int*)(A.cnt + emit_slot(lv, solo)) : 0;
      if (!A.cnt || (solo ? threadIdx.x != 0 || (int)blockIdx.x != sd : tid != 0) || done[sd]) continue;
      if (A.timeline && lv < kTimeline - 2) {
        A.timeline[lv] = global_ns();
        A.timeline[kTimelineCounts + lv] = n[sd];
      }
      if (n[sd] == 0) {
        if (A.levels) *A.levels = lv;
        done[sd] = true;
      }
    }
    if (n[0] == 0 && n[1] == 0) break;
    bool over = false;
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const EmitArgs& A = sd ? P.s[1] : P.s[0];
      if (n[sd] == 0 || (lv < A.max_levels && n[sd] <= A.E.q_cap)) continue;
      over = true;
      if (solo ? threadIdx.x == 0 : tid == 0)
        set_status(A.E.status, lv >= A.max_levels ? kStatusRoundCap : kStatusQueueOverflow);
    }
    if (over) break;  // every thread leaves: the counters are the same for all
    // levels of at most one task per thread of a block finish in one block
    // per side (each task is one thread's work either way)
    if (!solo && n[0] <= 256 && n[1] <= 256) {
      solo = true;
      if (blockIdx.x >= 2) break;
      if (n[blockIdx.x] == 0) break;
    }
    // this block's side, and its place among that side's blocks
    int sd = (int)blockIdx.x, at = 0, blocks = 1;
    if (!solo) {
      const int g = (int)gridDim.x;
      int g0 = (int)((long long)g * n[0] / ((long long)n[0] + n[1]));
      if (n[0] && n[1]) g0 = min(g - 1, max(1, g0));
      sd = (int)blockIdx.x >= g0;
      at = sd ? (int)blockIdx.x - g0 : (int)blockIdx.x;
      blocks = sd ? g - g0 : g0;
    }
    const EmitArgs& A = sd ? P.s[1] : P.s[0];
    const int4* in = (lv & 1) ? A.q1 : A.q0;
    int4* q_out = (lv & 1) ? A.q0 : A.q1;
    if (solo ? threadIdx.x == 0 : tid == 0) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const EmitArgs& C = k ? P.s[1] : P.s[0];
        if (C.cnt && (!solo || k == sd)) C.cnt[emit_slot(lv + 2, solo)] = 0;
      }
    }
    const int ns = sd ? n[1] : n[0];
    const long long nt = (long long)blocks * 256;
    const long long t0 = ((long long)(threadIdx.x >> 5) * blocks + at) * 32 + (threadIdx.x & 31);
    for (long long base = 0; base < ns; base += nt * U)
      emit_batch<U>(A.E, q_out, A.cnt + emit_slot(lv + 1, solo), A.cnt + kEmitSegs, in, base + t0, nt, ns);
    if (solo)
      __syncthreads();
    else
      grid.sync();
  }
}

// Every raw-arc segment collected by emit_persistent_kernel. Segment
// lengths are very uneven, so a lane that finishes its segment takes the next
// one instead of idling until the warp's longest is done: each warp owns
// ranges of kSegRange consecutive segments (grid-stride over the ranges) and,
// every kSegSteps cells, hands the next unstarted segments of its range to its
// idle cursors by ballot (warp-local, no atomics), starting its next range
// while the last one's long segments go on. Each lane drives NC cursors whose
// flow-code loads are issued together, so a lane waits on NC independent
// dependent-load chains at once instead of one.
//
// Bound by instruction issue, so each side has its own body (the codes' shift
// and the arcs' start cells are constants) on 32 instead of 40 registers.
// Geometry, one body for both sides and ranges one after the other -> now:
// 4096^2 dual threshold 0 0.69 -> 0.59 ms, 8192^2 noise 2.91 -> 2.55, 4096^2
// threshold 0.05 0.98 -> 0.95. Blocks in flight beyond those resident even
// out the ranges' lengths: 24 a SM 0.952 ms at 4096^2, 8 0.999, 48 0.975.
constexpr int kSegRange = 128;
constexpr int kSegSteps = 4;
constexpr int kSegBlocks = 24;  // per SM and side
constexpr int kSegCursorShapes = 2;  // NC = 1 or 2 (tuned)

struct SegArgs {
  EmitCtx E[2];
  const int* count[2];  // nullptr: nothing to write on this side
};

template <int NC, bool FACES>
__device__ __forceinline__ void emit_segments(const EmitCtx& E, const int* __restrict__ count) {
  const long long nb = E.nvirt + min((long long)*count, E.base_cap);
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  constexpr int shift = FACES ? 4 : 0, type = FACES ? 3 : 0;
  // the range's unstarted segments (same in every lane)
  long long r0 = warp * kSegRange, next = r0, r1 = min(nb, r0 + kSegRange);
  SegCursor c[NC];
#pragma unroll
  for (int q = 0; q < NC; ++q) c[q].rem = 0;
  while (true) {
    bool busy = false;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const unsigned idle = __ballot_sync(0xffffffffu, c[q].rem <= 0);
      if (c[q].rem <= 0) {
        const long long my = next + __popc(idle & lt);
        if (my < r1) seg_start<FACES>(E, my, c[q]);
      }
      next += __popc(idle);
      busy = busy || c[q].rem > 0;
    }
    if (next >= r1) {
      if (r1 < nb) {  // the next range, while the last one's long segments go on
        next = r0 += nwarps * kSegRange;
        r1 = min(nb, r0 + kSegRange);
      }
      if (next >= r1 && __ballot_sync(0xffffffffu, busy) == 0) break;
    }
#pragma unroll 1
    for (int k = 0; k < kSegSteps; ++k) {
      unsigned f[NC];
#pragma unroll
      for (int q = 0; q < NC; ++q) {  // all loads first: independent chains overlap
        f[q] = 0;
        if (c[q].rem > 1) f[q] = __ldg(E.flow + c[q].idx);
      }
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        if (c[q].rem <= 0) continue;
        *c[q].dst = type + 4 * (c[q].idx - c[q].ibase);
        c[q].dst += c[q].step;
        if (--c[q].rem > 0) c[q].idx += flow_step((f[q] >> shift) & 7u, c[q].Nx);
      }
    }
  }
}

// Both sides in one launch (blockIdx.y).
template <int NC>
__global__ void __launch_bounds__(256) emit_segments_kernel(SegArgs A) {
  if (blockIdx.y == 0) {
    if (A.count[0]) emit_segments<NC, true>(A.E[0], A.count[0]);
  } else {
    if (A.count[1]) emit_segments<NC, false>(A.E[1], A.count[1]);
  }
}

}  // namespace dmsc
