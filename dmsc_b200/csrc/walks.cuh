// V-path walks: saddle arc targets/lengths and basin/peak labels.
//
// Reference semantics: cpu/arcs_topology.hxx:67-172 (targets and lengths of the
// two face walks and up-to-two vertex walks of each saddle),
// cpu/arcs_geometry.hxx:74-81, 124-131 (arc k = k-th valid start cell) and
// cpu/cell_groups.hxx:96-229 (label = region of the thresholded union-find root
// of the critical cell a cell's V-path reaches). A cell's label depends only on
// its path's endpoint, so the reference's opportunistic label cache is not
// needed for identical results.
#pragma once

#include "common.cuh"

namespace dmsc {

// The j-th valid start cell of saddle `s_cell` on the face side (both cofaces
// are always valid).
__device__ __forceinline__ int face_start(int s_cell, int j, int Nx) {
  int idx = s_cell >> 2;
  if (j == 0) return 3 + 4 * idx;
  return (cell_type(s_cell) == 1) ? 3 + 4 * (idx + Nx) : 3 + 4 * (idx + 1);
}

// The j-th valid start cell on the vertex side, or -1; the saddle lies at
// (ey, ex) of its image (`s_cell` may be a global cell id).
__device__ __forceinline__ int vertex_start(int s_cell, int j, int ey, int ex, int H, int W, int Nx) {
  const int idx = s_cell >> 2;
  const bool h = cell_type(s_cell) == 1;
  const bool low = h ? ex >= 1 : ey >= 1, high = h ? ex < W : ey < H;
  if (j == 0 && low) return 4 * (h ? idx - 1 : idx - Nx);
  return (j == 0 || low) && high ? 4 * idx : -1;
}

// Walks from index `idx` along the flow codes (nibble shift 0 = vertices,
// 4 = faces) to the index of the critical cell; counts the steps.
template <int SHIFT>
__device__ __forceinline__ int flow_walk(const uint8_t* __restrict__ flow, int idx, int Nx, int cap, int* steps,
                                         unsigned* status) {
  int n = 0;
  unsigned c;
  while ((c = (__ldg(flow + idx) >> SHIFT) & 7u) != kFlowNone) {
    idx += flow_step(c, Nx);
    if (++n > cap) {
      set_status(status, kStatusWalkCap);
      break;
    }
  }
  *steps = n;
  return idx;
}

// Dense rank in its critical list of the extremum at global index g of image
// b, whose coordinates (y, x) are returned: its 32-index row segment's first
// rank (the compaction's exclusive scan) plus the extrema before it in the
// segment's bit mask.
__device__ __forceinline__ int seg_rank(const Imgs& I, int b, int g, int Nx, const int* __restrict__ off,
                                        const uint32_t* __restrict__ bits, int& y, int& x) {
  const int l = g - I.idx_base[b];
  y = row_of(I, b, l);
  x = l - y * Nx;
  const int seg = I.seg_base[b] + y * ((Nx + 31) >> 5) + (x >> 5);
  return __ldg(off + seg) + __popc(__ldg(bits + seg) & ((1u << (x & 31)) - 1u));
}

// Where the labels of one side go: image b's block of the output array picked
// by its orientation (faces are peaks in the primal, basins in the dual).
struct LabelOut {
  int* primal;            // output for primal images (nullptr: not requested)
  int* dual;              // output for dual images
  const int* primal_off;  // [B] block offset of image b in `primal`
  const int* dual_off;
};

// ---------------------------------------------------------------------------
// K9 (tiled): labels of both sides through 64 x 64 index tiles. A tile's flow
// codes are staged in shared memory, so every step of a V-path inside the
// tile is a shared-memory read. A path that leaves the tile continues from
// the first cell outside it, which lies on the border of the neighbouring
// tile: label_tile_kernel writes, for every border cell of every tile, its
// label or the border-map entry of the cell its path next enters, and lists
// the cells whose paths leave their tile; label_exit_kernel then crosses each
// further tile of such a path with one lookup in that border map.
constexpr int kLT = 64;
constexpr int kLTN = kLT * kLT;
constexpr int kPerim = 4 * kLT;  // border slots per tile: top row, bottom row, left column, right column

struct LabelTile {
  int b, H, W, Nx, y0, x0;
  long long base;  // global index of the tile's first cell
};

__device__ __forceinline__ LabelTile label_tile_of(const Imgs& I, int t) {
  LabelTile g;
  g.b = find_image(I.ltile_base, I.B, t);
  g.H = I.H[g.b];
  g.W = I.W[g.b];
  g.Nx = g.W + 1;
  const int ntx = (g.W + kLT) / kLT;  // ceil((W + 1) / 64)
  const int tt = t - I.ltile_base[g.b];
  const int ty = tt / ntx, tx = tt - ty * ntx;
  g.y0 = ty * kLT;
  g.x0 = tx * kLT;
  g.base = (long long)I.idx_base[g.b] + (long long)g.y0 * g.Nx + g.x0;
  return g;
}

__device__ __forceinline__ int perim_slot(int r, int c) {
  return r == 0 ? c : r == kLT - 1 ? kLT + c : c == 0 ? 2 * kLT + r : 3 * kLT + r;
}

// In-tile resolution, one side per block. The tile lies in shared memory as
// one signed byte per cell, the distance in the array to the cell its path
// visits next (0: the path ends here), inside a ring of one cell of the
// neighbouring tiles, whose distance is 0: a step of a walk is one byte read
// and one addition, with no test of the code, of the tile's edge or of the
// end. Every cell takes kLabelSteps of them, the thread's cells together, and
// one that has not ended then jumps through the cells that the others reached.
// The state of a final cell is (label << 1) | 1 of its extremum (label -1
// encodes as all ones), or, on the ring, (border-map index of that cell in
// its own tile) << 1.
//
// What bounds it is the instructions: with 16-bit successors and 32-bit states
// for every cell of both sides and a tested loop for each walk it issued 465
// warp instructions for 32 cells of both sides, now 274. Labels at 4096^2
// (smooth, threshold 0.05) 302 -> 205 us, at 8192^2 noise 1461 -> 1107 us, at
// 256^2 29 -> 17 us; the issue slots and the shared-memory pipe are both at
// four fifths. 4 to 12 steps before the jumps are within 3 %, 1536 threads
// per SM instead of 2048 are 9 % slower.
constexpr int kLabelPitch = 72;  // 64 columns from 4 on (words of steps are aligned), the ring in columns 3 and 68
constexpr int kLabelCells = (kLT + 2) * kLabelPitch;
constexpr int kLabelSteps = 8;
__device__ __forceinline__ int label_pos(int r, int c) { return (r + 1) * kLabelPitch + 4 + c; }

// Threads per label tile (the tuner picks one): each thread owns column
// tid % 64 of rows tid / 64 + (NT / 64) k, k < 4096 / NT.
constexpr int kLabelShapes = 2;
constexpr int kLabelNT[kLabelShapes] = {1024, 512};

// Steps of four cells from their four flow codes (one per byte, 0 .. 4): the
// codes, packed to nibbles, select the bytes of a table.
__device__ __forceinline__ unsigned label_steps(unsigned codes) {
  unsigned s = codes & 0x07070707u;
  s = (s | s >> 4) & 0x00FF00FFu;
  s |= s >> 8;
  constexpr unsigned lo = (0xFFu << 8) | (1u << 16) | ((unsigned)(256 - kLabelPitch) << 24);  // none, left, right, up
  return __byte_perm(lo, (unsigned)kLabelPitch, s);                                           // down
}

// Follows border-map entries to a label.
__device__ __forceinline__ int entry_label(int e, const int* __restrict__ perim, int cap, unsigned* status) {
  for (int h = 0; h <= cap; ++h) {
    if (e & 1) return e >> 1;
    e = __ldg(perim + (e >> 1));
  }
  set_status(status, kStatusWalkCap);
  return -1;
}

struct LabelSide {
  const int* off;    // segment offsets of this side's critical list (exclusive scan)
  const uint32_t* bits;  // critical cells of each segment
  const int* rout;   // per critical extremum (batch-wide rank): out rank of its thresholded root, -1 for the void
  const int* abase;  // [B + 1] first out rank of each image's alive extrema
  int* perim;        // border map
  int2* exits;       // cells whose paths leave their tile: (global index, entry)
  int* n_exits;
  LabelOut out;
};

// Label of an extremum from its root's batch-wide out rank: the root's rank
// among its image's surviving extrema, -1 for the void
// (cpu/cell_groups.hxx:128-146, 168-173).
__device__ __forceinline__ int region_label(int rout, int abase) { return rout < 0 ? -1 : rout - abase; }

__device__ __forceinline__ int label_ntx(const LabelTile& g) { return (g.W + kLT) / kLT; }

struct LabelSmem {
  uint32_t st[kLabelCells];      // states of the final cells
  uint16_t ptr[kLabelCells];     // cell reached by each cell's walk
  __align__(4) int8_t step[kLabelCells];
};

// Labels of a tile's cells on one side: face labels over the (H+1) x (W+1)
// indices or vertex labels over the H x W pixels
// (cpu/cell_groups.hxx:151-228). A cell whose path ends inside the tile gets
// its label here; the tile's border cells also get their border-map entries; a
// cell whose path leaves the tile is appended to its side's exit list and
// finished by label_exit_kernel once every tile's border map is written.
template <int NT, bool FACES>
__device__ __forceinline__ void label_tile(LabelSmem& S, const Imgs& I, const uint8_t* __restrict__ flow,
                                           const LabelSide& L, unsigned* status) {
  constexpr int kCells = kLTN / NT, kStep = NT / kLT, kItems = 2 * kLT / (NT / 32);
  const LabelTile g = label_tile_of(I, blockIdx.x);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ntx = label_ntx(g);
  // the (row, 32-cell segment) items of this warp: lane k loads the first rank
  // and the extrema of item k, used once the steps are on their way
  int off = 0;
  unsigned bits = 0;
  if (lane < kItems) {
    const int rs = warp * kItems + lane, y = g.y0 + (rs >> 1), sx = (g.x0 >> 5) + (rs & 1);
    const int nsegx = (g.W + 32) / 32;  // 32-index row segments of the compaction: ceil((W + 1) / 32)
    if (y <= g.H && sx < nsegx) {
      const long long q = (long long)I.seg_base[g.b] + (long long)y * nsegx + sx;
      off = __ldg(L.off + q);
      bits = __ldg(L.bits + q);
    }
  }
  const int abase = __ldg(L.abase + g.b);
  // steps, a word of four cells at a time (rows start at any byte: two aligned
  // words and a shift). A word is read when its first cell lies in the image;
  // what lies beyond is never reached from inside.
#pragma unroll
  for (int k = 0; k < kLTN / 4 / NT + (kLTN / 4 % NT != 0); ++k) {
    const int i = tid + k * NT, r = i >> 4, c = (i & 15) * 4;
    unsigned w = 0;
    if (g.y0 + r <= g.H && g.x0 + c <= g.W) {
      const long long o = g.base + (long long)r * g.Nx + c;
      const unsigned* p = reinterpret_cast<const unsigned*>(flow) + (o >> 2);
      w = __funnelshift_r(__ldg(p), __ldg(p + 1), 8 * (unsigned)(o & 3));
    }
    *reinterpret_cast<unsigned*>(S.step + label_pos(r, c)) = label_steps(FACES ? w >> 4 : w);
  }
  for (int i = tid; i < 4 * kLT; i += NT) {  // the ring
    const int k = i & (kLT - 1), e = i / kLT;
    const int r = e == 0 ? -1 : e == 1 ? kLT : k, c = e == 2 ? -1 : e == 3 ? kLT : k;
    const int nt = blockIdx.x + (e == 0 ? -ntx : e == 1 ? ntx : e == 2 ? -1 : 1);
    S.step[label_pos(r, c)] = 0;
    S.st[label_pos(r, c)] = (unsigned)(nt * kPerim + perim_slot(r & (kLT - 1), c & (kLT - 1))) << 1;
  }
  {  // labels of the extrema
    int lab[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const unsigned m = __shfl_sync(0xffffffffu, bits, k);
      const int o = __shfl_sync(0xffffffffu, off, k);
      lab[k] = (m >> lane) & 1u ? __ldg(L.rout + o + __popc(m & ((1u << lane) - 1u))) : 0;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int rs = warp * kItems + k;
      if ((__shfl_sync(0xffffffffu, bits, k) >> lane) & 1u)
        S.st[label_pos(rs >> 1, (rs & 1) * 32 + lane)] = ((unsigned)region_label(lab[k], abase) << 1) | 1u;
    }
  }
  __syncthreads();
  const int c = tid % kLT, rb = tid / kLT, x = g.x0 + c;
  int pos[kCells];
#pragma unroll
  for (int k = 0; k < kCells; ++k) pos[k] = label_pos(rb + kStep * k, c);
  unsigned pend = 0;
  {
    int last[kCells];
#pragma unroll
    for (int w = 0; w < kLabelSteps; ++w)
#pragma unroll
      for (int k = 0; k < kCells; ++k) {
        last[k] = S.step[pos[k]];
        pos[k] += last[k];
      }
    const int rows = FACES ? g.H + 1 - g.y0 : g.H - g.y0;
    const bool in = FACES ? x <= g.W : x < g.W;
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      S.ptr[label_pos(rb + kStep * k, c)] = (uint16_t)pos[k];
      if (last[k] != 0 && in && rb + kStep * k < rows) pend |= 1u << k;
    }
  }
  __syncthreads();
  // barrier-free pointer jumping of this thread's unfinished cells: a cell's
  // pointer only moves on along its path, whichever thread reads it, so a
  // path's end is reached in at most its length of jumps
  for (int it = 0; pend; ++it) {
    if (it >= kLTN) {
      set_status(status, kStatusWalkCap);
      break;
    }
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      if (!((pend >> k) & 1u)) continue;
      if (S.step[pos[k]] == 0) {
        pend &= ~(1u << k);
      } else {
        pos[k] = *reinterpret_cast<volatile uint16_t*>(S.ptr + pos[k]);
        *reinterpret_cast<volatile uint16_t*>(S.ptr + label_pos(rb + kStep * k, c)) = (uint16_t)pos[k];
      }
    }
  }
  // labels of the paths that end in the tile, entries of the border cells, and
  // a bit per cell whose path leaves the tile if this image outputs the side's
  // labels; those are reserved in the exit list at once and written afterwards
  const bool d = I.dual[g.b];
  int* out = d ? L.out.dual : L.out.primal;
  const int pitch = FACES ? g.Nx : g.W;
  if (out) out += (d ? L.out.dual_off : L.out.primal_off)[g.b] + (g.y0 + rb) * pitch + x;  // image-local: below 2^31
  const bool border_c = c == 0 || c == kLT - 1;
  unsigned xm = 0;
  if (FACES ? x <= g.W : x < g.W) {
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      const int r = rb + kStep * k, y = g.y0 + r;
      if (FACES ? y > g.H : y >= g.H) break;
      const unsigned e = S.st[pos[k]];
      if (border_c || r == 0 || r == kLT - 1) L.perim[blockIdx.x * kPerim + perim_slot(r, c)] = (int)e;
      if (out) {
        if (e & 1u)
          out[k * kStep * pitch] = (int)e >> 1;
        else
          xm |= 1u << k;
      }
    }
  }
  int at = block_reserve(L.n_exits, __popc(xm));
  while (xm) {  // the few cells whose paths leave the tile
    const int k = __ffs(xm) - 1;
    xm &= xm - 1u;
    const int r = rb + kStep * k;
    // global indices stay below 2^29
    L.exits[at++] = make_int2((int)(g.base + (long long)r * g.Nx + c), (int)S.st[S.ptr[label_pos(r, c)]]);
  }
}

// Side `first` (0 faces, 1 vertices), or both (grid y = 2, first = 0).
template <int NT>
__global__ void __launch_bounds__(NT, 2048 / NT) label_tile_kernel(Imgs I, const uint8_t* __restrict__ flow,
                                                                   LabelSide F, LabelSide V, int first,
                                                                   unsigned* status) {
  __shared__ LabelSmem S;
  if (blockIdx.y + first == 0)
    label_tile<NT, true>(S, I, flow, F, status);
  else
    label_tile<NT, false>(S, I, flow, V, status);
}

// Cells whose paths leave their tile: follow the border map to the label
// (both sides in one launch, blockIdx.y).
__global__ void __launch_bounds__(256) label_exit_kernel(Imgs I, LabelSide F, LabelSide V, int first, int cap,
                                                         unsigned* status) {
  const bool faces = blockIdx.y + first == 0;
  const int2* __restrict__ exits = faces ? F.exits : V.exits;
  const int* __restrict__ perim = faces ? F.perim : V.perim;
  const LabelOut& O = faces ? F.out : V.out;
  const int n = faces ? *F.n_exits : *V.n_exits;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int2 e = exits[q];
    const int b = find_image(I.idx_base, I.B, e.x);
    const bool d = I.dual[b];
    int* out = d ? O.dual : O.primal;
    const int W = I.W[b], Nx = W + 1;
    const int lidx = e.x - I.idx_base[b];
    const int y = row_of(I, b, lidx), x = lidx - y * Nx;
    out += (d ? O.dual_off : O.primal_off)[b];
    out[faces ? lidx : y * W + x] = entry_label(e.y, perim, cap, status);
  }
}

}  // namespace dmsc
