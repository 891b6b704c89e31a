// Arc simplification: replay of the cancellations and emission of the
// simplified arc geometry.
//
// Reference semantics: cpu/arcs_simplification.hxx:310-504. The cancellations
// of one side are replayed in (persistence, saddle cell, target cell) order on
// a union-find whose roots are extrema. For a cancellation of saddle s killing
// extremum d, with arc targets T0 and T1: R0 = Find(T0), R1 = Find(T1); if
// R0 == d != R1 then d is linked under R1 (symmetric for R1 == d); otherwise
// the cancellation is skipped. Every link carries a path: the geometry from d
// back along the dying side's arc through s and on to the other root.
//
// Parallel form (exact). Links never move once made and link times increase
// along every parent chain, so the root of x just before replay step t is the
// first node on x's parent chain that is not linked before t. Each unresolved
// cancellation walks its two chains; it can decide as soon as every node it
// passes has been decided, and decisions are final, so rounds of such walks
// reproduce the sequential replay (including skips, which arise only from
// ties in persistence). Path lengths are summed along the same walks.
//
// Geometry. A link's path W(d) is
//   reverse(chain(T_dying -> d)) + reverse(arc_dying) + arc_other + chain(T_other -> R)
// where chain(x -> R) concatenates W along x's parent chain up to R, and every
// surviving saddle's final arc is arc + chain(T -> root). These are expanded
// breadth-first as chain tasks that each cover a known output range (a chain
// task writes every W along its chain at once: their raw-arc segments and
// their own chains as the next level's tasks); raw arcs are re-walked from
// their start cells when written.
#pragma once

#include "assemble.cuh"
#include "common.cuh"
#include "walks.cuh"

namespace dmsc {

constexpr unsigned long long kNever = ~0ull;  // replay key of a node that is never cancelled
enum : int { kPending = 0, kLinked = 1, kRootForever = 2 };

// A replay node in one 64-byte line. The first 32-byte sector holds all that a
// chain walk reads: its key with the emission's words, and the link (status,
// parent, length of W(node)) in 16 bytes that are written and read as one, so
// a walk that sees the status sees the whole decision, in the round in which
// it is made, with no fence. The second sector holds what the emission needs
// to expand W(node) without touching the saddle's arrays: the two chain
// lengths, the saddle's arc ends on the dying and the other side and their
// raw-arc lengths (written before the kernel ends, read by later kernels).
struct alignas(64) ReplayNode {
  unsigned long long ctime;  // replay key of the cancellation killing the node, kNever if none
  int side;                  // side_word: dying side of the node's cancellation and what W(node) expands to
  int scell;                 // global cell id of the saddle of the node's cancellation
  int status;                // kPending / kLinked / kRootForever
  int parent;                // link target (-1 = void) when kLinked
  long long wlen;            // length of W(node)
  long long cl_dy;           // chain length T_dying -> node at link time
  long long cl_ot;           // chain length T_other -> parent at link time
  int t_dy, t_ot;            // the saddle's arc ends on the dying and the other side
  int len_dy, len_ot;        // their raw-arc lengths (cells; a side's geometry stays below 2^31)
};
static_assert(sizeof(ReplayNode) == 64, "one 64-byte line per node");

struct ReplayState {
  ReplayNode* node;  // [M + 1]
};

struct NodeLink {
  int status, parent;
  long long wlen;
};
// The link while other blocks may be writing it (one 16-byte access through
// L2), and after the replay.
__device__ __forceinline__ NodeLink node_link_live(const ReplayNode* n, int x) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n"
      ".reg .b128 t;\n"
      "ld.relaxed.gpu.global.b128 t, [%2];\n"
      "mov.b128 {%0, %1}, t;\n"
      "}\n"
      : "=l"(lo), "=l"(hi)
      : "l"(__cvta_generic_to_global(&n[x].status))
      );
  return NodeLink{(int)(unsigned)lo, (int)(unsigned)(lo >> 32), (long long)hi};
}
__device__ __forceinline__ void node_link_set(ReplayNode* n, int x, NodeLink l) {
  const unsigned long long lo = (unsigned)l.status | (unsigned long long)(unsigned)l.parent << 32;
  asm volatile(
      "{\n"
      ".reg .b128 t;\n"
      "mov.b128 t, {%1, %2};\n"
      "st.relaxed.gpu.global.b128 [%0], t;\n"
      "}\n" ::"l"(__cvta_generic_to_global(&n[x].status)),
      "l"(lo), "l"((unsigned long long)l.wlen)
      );
}
__device__ __forceinline__ NodeLink node_link(const ReplayNode* n, int x) {
  const int4 v = *reinterpret_cast<const int4*>(&n[x].status);
  return NodeLink{v.x, v.y, (long long)((unsigned long long)(unsigned)v.w << 32 | (unsigned)v.z)};
}
// The emission's words (side, saddle cell).
__device__ __forceinline__ int2 node_words(const ReplayNode* n, int x) {
  return *reinterpret_cast<const int2*>(&n[x].side);
}

// Node records are written only for the nodes a cancellation kills: the
// persistence pass sets their key and kPending, and the replay their decision
// when it is made. Every reader first checks the side's alive flags: an alive
// extremum (no cancellation kills it) is a root forever and its record is
// never read, so no pass initialises the records of the others.
// Side word of a linked node: the dying side k (bit 0), the number of
// non-empty chains of W(node) (bits 1-2) and of its raw-arc segments (bits
// 3-4), so counting a chain's expansion reads one word per node.
__device__ __forceinline__ int side_word(int k, int n_chain, int n_base) { return k | (n_chain << 1) | (n_base << 3); }
__device__ __forceinline__ int side_of(int w) { return w & 1; }
__device__ __forceinline__ int chains_of(int w) { return (w >> 1) & 3; }
__device__ __forceinline__ int bases_of(int w) { return (w >> 3) & 3; }

// Root of x just before the replay step with key t, with the summed path
// length; returns false when a node on the way is still undecided. Replay
// steps are compared by their (persistence, saddle cell) keys, which are
// unique, so no ranks are needed.
__device__ __forceinline__ bool walk_root(const ReplayState& S, const uint8_t* __restrict__ alive, int x,
                                          unsigned long long t, int* root, long long* acc, int max_steps,
                                          unsigned* status) {
  long long a = 0;
  int steps = 0;
  while (x >= 0 && !alive[x]) {
    const unsigned long long key = S.node[x].ctime;
    const NodeLink l = node_link(S.node, x);
    if (key >= t) break;
    if (l.status == kPending) return false;
    if (l.status == kRootForever) break;
    a += l.wlen;
    x = l.parent;
    if (++steps > max_steps) {
      set_status(status, kStatusChainCap);
      break;
    }
  }
  *root = x;
  *acc = a;
  return true;
}

// A survivor's record, one 64-byte line (32 bytes a side): its arc ends, the
// ranks of the thresholded roots of its ends and of its pair (-1 for the
// void), the persistence bits and the raw-arc lengths (15 bits each, with a
// bit for an end that a cancellation kills; kLongArc: look the lengths up).
struct alignas(64) SurvRec {
  struct Side {
    int t0, t1, r0, r1;
    int rp, p;
    unsigned lens;
    int id;  // faces: the saddle's cell, vertices: its list index
  } side[2];
};
constexpr unsigned kLongArc = 0x7FFFu;

struct SurvSource {
  const int4* arc;       // [2 nsad] both sides' records, interleaved
  const int4* pp;        // [nsad] paired extremum and persistence bits of both sides
  const int* rout[2];    // [M] rank of each extremum's root
  const uint8_t* alive[2];
};

// The survivors in list order: their sort keys ((image, s_val) order: the
// image id above the orderable value, so one sort orders every image; a
// 32-bit key of the value alone for one image) and their records. Everything
// is read in list order here, or near it, so that the sort's random
// permutation later costs a survivor one line; gathering the same from the
// saddles' arrays in output order cost it eleven sectors, most of them in DRAM
// for large calls. With 24 M survivors (8192^2 noise, threshold 0) the labels,
// which this pass and the sort run beside, and the final arcs took 5.3 ms
// before and take 3.9 ms.
template <class K>
__global__ void __launch_bounds__(256) survivor_gather_kernel(int nsad, const uint8_t* __restrict__ flag,
                                                              const int* __restrict__ pos,
                                                              const float* __restrict__ sval,
                                                              const int* __restrict__ sad_img,
                                                              const int* __restrict__ crit_sad, SurvSource A,
                                                              K* __restrict__ key_out, int* __restrict__ idx_out,
                                                              SurvRec* __restrict__ rec) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsad || !flag[s]) return;
  const int q = pos[s];
  const uint32_t o = orderable_key(sval[s]);
  key_out[q] = sizeof(K) > 4 ? (K)(((unsigned long long)sad_img[s] << 32) | o) : (K)o;
  idx_out[q] = q;
  const int4 pr = A.pp[s];
  SurvRec r;
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    const int4 a = A.arc[2 * (long long)s + sd];
    const int e = sd ? pr.z : pr.x;
    const bool long_arc = a.z >= (int)kLongArc || a.w >= (int)kLongArc;
    const unsigned l0 = long_arc ? kLongArc : (unsigned)a.z, l1 = long_arc ? kLongArc : (unsigned)a.w;
    const bool d0 = a.x >= 0 && !A.alive[sd][a.x], d1 = a.y >= 0 && !A.alive[sd][a.y];
    SurvRec::Side& v = r.side[sd];
    v.t0 = a.x;
    v.t1 = a.y;
    v.r0 = a.x >= 0 ? A.rout[sd][a.x] : -1;
    v.r1 = a.y >= 0 ? A.rout[sd][a.y] : -1;
    v.rp = e >= 0 ? A.rout[sd][e] : -1;
    v.p = sd ? pr.w : pr.y;
    v.lens = l0 | (d0 ? 0x8000u : 0u) | l1 << 16 | (d1 ? 0x80000000u : 0u);
    v.id = sd ? s : crit_sad[s];
  }
  rec[q] = r;
}

// The survivors in output order and their final arcs, two threads (sides) a
// survivor. `sorted` lists their records by ascending (image, s_val, cell id),
// the vertex side's sweep order (arcs_topology.hxx:99-102); an image whose
// vertex side sweeps descending (dual) takes its range reversed. A side's
// thread reads its half of the record, walks its ends' chains to their final
// roots, and writes everything in output order, so that the later per-survivor
// kernels read in order; the survivor's geometry cells and e rows go to the
// scans (entry nsurv is zero: the totals). Images whose output does not take a
// side's arcs (`primal` / `dual` by orientation) get empty arcs there.
struct FinalSide {
  int4* s_arc;            // [nsurv] arc ends, raw-arc lengths
  int4* s_out;            // [nsurv] ranks of the ends' roots, persistence bits, rank of the pair's root
  int4* s_fin;            // [nsurv] chain lengths and roots; nullptr: no image takes the arcs
  const uint8_t* alive;
  ReplayState S;
  bool primal, dual;
};

__global__ void __launch_bounds__(256) survivor_final_kernel(
    int nsurv, const int* __restrict__ sorted, const SurvRec* __restrict__ rec, const int4* __restrict__ arc, Imgs I,
    const int* __restrict__ surv_base, FinalSide F, FinalSide V, int max_steps, SurvHead* __restrict__ head,
    unsigned long long* __restrict__ lens, unsigned long long* __restrict__ rows,
    unsigned long long* __restrict__ total, unsigned* status) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int p = (int)(t >> 1), sd = (int)(t & 1);
  __shared__ unsigned long long sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  int q = p;
  unsigned n_rows = 0;
  unsigned long long len = 0;
  int4 v0 = make_int4(0, 0, 0, 0), v1 = v0;  // this side's half of the record
  if (p < nsurv) {
    const int4* half = reinterpret_cast<const int4*>(rec + sorted[p]) + 2 * sd;
    v0 = half[0];
    v1 = half[1];
  }
  const int other = __shfl_xor_sync(0xffffffffu, v1.w, 1);
  const int cell = sd ? other : v1.w, s = sd ? v1.w : other;
  if (p < nsurv) {
    const int b = I.B > 1 ? find_image(I.idx_base, I.B, cell >> 2) : 0;
    const bool d = I.dual[b];
    if (d) {
      const int base = surv_base[b], cnt = surv_base[b + 1] - base;
      q = base + cnt - 1 - (p - base);
    }
    const FinalSide& A = sd ? V : F;
    A.s_out[q] = make_int4(v0.z, v0.w, v1.y, v1.x);
    int x, y;
    n_rows = erow_ends(v0.z, v0.w, &x, &y);
    if (A.s_fin) {
      const unsigned l = (unsigned)v1.z;
      int l0 = (int)(l & 0x7FFFu), l1 = (int)(l >> 16 & 0x7FFFu);
      if (l0 == (int)kLongArc) {
        const int4 a = arc[2 * (long long)s + sd];
        l0 = a.z;
        l1 = a.w;
      }
      int4 fin = make_int4(0, 0, -1, -1);
      if (d ? A.dual : A.primal) {
        long long c[2] = {0, 0};
        int root[2] = {v0.x, v0.y};
        // an extremum that no cancellation kills is its own final root; only
        // the others walk their parent chains
        if (l & 0x8000u) walk_root(A.S, A.alive, v0.x, kNever, &root[0], &c[0], max_steps, status);
        if (l >> 31) walk_root(A.S, A.alive, v0.y, kNever, &root[1], &c[1], max_steps, status);
        // a chain beyond 32 bits makes the side's geometry overflow (the
        // exact total says so): its stored length is not used then
        fin = make_int4((int)c[0], (int)c[1], root[0], root[1]);
        len = (unsigned long long)((long long)l0 + l1 + c[0] + c[1]);
      }
      A.s_arc[q] = make_int4(v0.x, v0.y, l0, l1);
      A.s_fin[q] = fin;
    }
    if (sd == 0) *reinterpret_cast<int4*>(head + q) = make_int4(b, cell, s, 0);
  }
  const unsigned other_rows = __shfl_xor_sync(0xffffffffu, n_rows, 1);
  const unsigned other_len = __shfl_xor_sync(0xffffffffu, (unsigned)len, 1);
  if (sd == 0 && p <= nsurv) {  // p == nsurv: q == p, all zero
    lens[q] = pack2((unsigned)len, other_len);
    rows[q] = pack2(n_rows, other_rows);
  }
  // the exact geometry totals
#pragma unroll
  for (int o = 2; o < 32; o <<= 1) len += __shfl_xor_sync(0xffffffffu, len, o);
  if ((threadIdx.x & 31) < 2 && len) atomicAdd(&sum[sd], len);
  __syncthreads();
  if (threadIdx.x < 2 && sum[threadIdx.x]) atomicAdd(total + threadIdx.x, sum[threadIdx.x]);
}

// ---------------------------------------------------------------------------
// geometry emission
// ---------------------------------------------------------------------------
enum : int { kTaskChain = 2 };
// chain task = {kind | dir << 2, start node, stop node (-1 = void), pos}
__device__ __forceinline__ int4 make_task(int kind, int rev, int a, int b, long long pos) {
  return make_int4(kind | (rev << 2), a, b, (int)pos);
}

struct EmitCtx {
  const uint8_t* flow;
  Imgs I;
  bool faces;
  ReplayState S;
  int* out_primal;  // destination of primal images' arcs of this side
  int* out_dual;    // destination of dual images' arcs
  const int* dst_off;  // [B] start of each image's geometry in its destination (positions are image-local)
  long long q_cap;
  int4* base_q;  // raw-arc segments of the chain expansion
  long long base_cap;
  // the survivors' own raw arcs (segment items 0 .. 2 nsurv - 1 of the
  // writer, read from the survivor records instead of a task list)
  int nvirt;                 // 2 nsurv
  const SurvHead* head;      // [nsurv] image and cell of each survivor (output order)
  const int4* arc;           // [nsurv] arc ends and raw-arc lengths
  const int4* fin;           // [nsurv] chain lengths and roots
  const unsigned long long* lens;  // [nsurv + 1] where each survivor's geometry starts (both sides packed)
  const long long* gbase;    // [B + 1] where each image's does
  int max_steps;
  unsigned* status;
};

// Image-local output position of a survivor's first arc.
__device__ __forceinline__ int surv_start(const EmitCtx& E, int i, int b) {
  return half_of(E.lens[i], E.faces ? 0 : 1) - (int)E.gbase[b];
}

// A raw-arc segment task of the chain expansion: {reversed | arc << 1,
// saddle cell, cells, output position}: the writer finds the arc's start
// cell from the saddle's cell with no further load.
template <bool FACES>
__device__ __forceinline__ int arc_start_of_cell(const EmitCtx& E, int sc, int j, int b) {
  const int W = E.I.W[b], Nx = W + 1;
  if (FACES) return face_start(sc, j, Nx) >> 2;
  const int l = (sc >> 2) - E.I.idx_base[b], y = row_of(E.I, b, l);
  return vertex_start(sc, j, y, l - y * Nx, E.I.H[b], W, Nx) >> 2;
}
__device__ __forceinline__ int4 make_saddle_seg(int scell, int j, int rev, long long len, long long pos) {
  return make_int4(rev | (j << 1), scell, (int)len, (int)pos);
}

// A raw arc being written by one lane: the V-path from its start cell, `len`
// cells (cpu/arcs_geometry.hxx:83-111, 133-161), following the flow codes.
// dst is the next output slot, step its stride (-1 for a reversed arc), rem
// the cells left and idx the current index.
struct SegCursor {
  int* dst;
  int step;
  int rem;
  int idx, ibase, Nx;
};

// Starts segment item q: q < nvirt is raw arc (q / 2, q % 2) of a survivor,
// forward at its arc's output position; the others are the chain
// expansion's tasks. rem = 0 when it writes nothing (no arc, or its image's
// output does not take this side's arcs).
template <bool FACES>
__device__ __forceinline__ void seg_start(const EmitCtx& E, long long q, SegCursor& c) {
  c.rem = 0;
  int b, idx, len, pos;
  bool rev;
  if (q < E.nvirt) {
    const int i = (int)(q >> 1), j = (int)(q & 1);
    const int4 a = E.arc[i];
    len = j ? a.w : a.z;
    if ((j ? a.y : a.x) < 0 || len <= 0) return;
    const int2 ic = *reinterpret_cast<const int2*>(E.head + i);
    b = ic.x;
    idx = arc_start_of_cell<FACES>(E, ic.y, j, b);
    pos = surv_start(E, i, b) + (j ? a.z + E.fin[i].x : 0);
    rev = false;
  } else {
    const int4 t = E.base_q[q - E.nvirt];
    const int j = (t.x >> 1) & 1;
    len = t.z;
    b = find_image(E.I.idx_base, E.I.B, t.y >> 2);
    idx = arc_start_of_cell<FACES>(E, t.y, j, b);
    pos = t.w;
    rev = t.x & 1;
  }
  int* out = E.I.dual[b] ? E.out_dual : E.out_primal;
  if (!out || len <= 0) return;
  c.Nx = E.I.W[b] + 1;
  c.ibase = E.I.idx_base[b];
  c.idx = idx;
  c.dst = out + E.dst_off[b] + (rev ? (long long)pos + len - 1 : (long long)pos);
  c.step = rev ? -1 : 1;
  c.rem = len;
}

}  // namespace dmsc
