// Row-walk matrix assembly: one thread owns one CSR row (the default of FP64 P1
// stiffness from 98,304 cells, P2 from 65,536 cells and P3, see rows_default).
//
// The scatter kernels (fe_kernels.cu) send every element entry to the L2 as
// an FP64 reduction (531 M of them for 205 M nonzeros at P2 n=96) into values
// a zero pass has cleared before; the L2's reduction rate bounds them at any
// occupancy.  Here a thread walks the cells around its row's node instead,
// adds their entries into the row's segment in shared memory, where nothing
// else writes (no atomics, a fixed order: the result is bitwise
// reproducible), and the warp then stores its 32 rows once, coalesced.  There
// is no zero pass and no reduction, and only row i of an element tensor is
// evaluated for row i.
//
// What makes the walk cheap is its plan (built with the slot map when a form
// binds its pattern): the rows of a warp are of one kind (vertex, edge node,
// face node) and of nearly one length, so their code does not diverge; every
// cell is listed with its vertices in the row's own order (its vertex, or its
// edge's or face's vertices, first), so that an entry's formula is fixed at
// compile time; the cells follow one another through their common faces
// (around an edge; around a vertex as strips of the triangles opposite it), so
// that a step fetches one new vertex and keeps the others in registers; and
// the slot bytes of a step's columns stand in the same record.
//
// Element entries, with n_x the gradient of barycentric coordinate x times
// det J, w = k / |det J| and xy = n_x . n_y (for affine cells grad lambda_x .
// grad lambda_y |det J| = xy / |det J|): integrals of products of barycentric
// coordinates are exact rationals, so row i is a few products of the xy.
//
// Reference counterpart: assemble_<I>_c_mat (CUDAFormIntegral.cpp:1103-1226)
// with its zero and set_diagonal passes (CUDAAssembler.cpp:38-164).
#include <cuda_runtime.h>

#include <algorithm>
#include <cub/cub.cuh>
#include <memory>

#define FE_P3_ROW_TABLES
#include "fe_element_code.cuh"
#include "fe_internal.h"
#include "fe_rows.cuh"

namespace fe {
namespace {

constexpr int kMaxStar = 128;           // cells of a vertex row
constexpr int kStripTries = 64;         // beginnings tried for its walk

// marks of an edge row's record: the first and the last cell of a fan around
// the edge; a closed fan ends at the vertex it began with
constexpr uint32_t kFanBegin = 1u, kFanEnd = 2u, kFanClosed = 4u;

// marks of a vertex row's record, beside the vertex it fetches: no cell yet
// (the first two vertices of a strip); the next cell keeps the older one of
// the last two vertices
constexpr uint32_t kStripLoad = 0x80000000u, kStripKeep = 0x40000000u, kStripVertex = 0x3fffffffu;

// kinds of rows
enum { KIND_V = 0, KIND_E = 1, KIND_F = 2 };

__host__ __device__ constexpr int dofs_of(int deg) { return deg == 1 ? 4 : (deg == 2 ? 10 : 20); }

// kind of the node at local index i
__device__ __forceinline__ int kind_of(int deg, int i) { return i < 4 ? KIND_V : (deg < 3 || i < 16 ? KIND_E : KIND_F); }

// local edge {u, v} in the order (2,3),(1,3),(1,2),(0,3),(0,2),(0,1)
__device__ __forceinline__ int edge_id(int u, int v) {
  const int lo = min(u, v), hi = max(u, v);
  return lo == 0 ? 6 - hi : (lo == 1 ? 4 - hi : 0);
}
// local dof of the P2 node of edge {x, y}; of the P3 node near x on it
__device__ __forceinline__ int p2_edge(int x, int y) { return 4 + edge_id(x, y); }
__device__ __forceinline__ int p3_edge(int x, int y) { return 4 + 2 * edge_id(x, y) + (x < y ? 0 : 1); }

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
struct PlanArgs {
  int64_t num_cells, num_rows;
  int k, deg;
  const int32_t* geom;
  const int32_t* dofs;
  const uint8_t* pos;
  const int32_t* row_ptr;
  const int32_t* diag;     // slot of (r, r) or -1
  int32_t* inc_ptr;
  int32_t* inc;
  unsigned* fail;
};

__global__ void k_rows_count(const PlanArgs a, int32_t* __restrict__ cnt, unsigned* __restrict__ kmask) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= a.num_cells) return;
  const int32_t* d = a.dofs + c * a.k;
  for (int i = 0; i < a.k; ++i) {
    const int32_t r = d[i];
    if (r < 0 || r >= a.num_rows) {
      *a.fail = 1u;
      return;
    }
    // a step adds to all its columns at once: they have to differ
    for (int j = 0; j < i; ++j)
      if (d[j] == r) *a.fail = 1u;
    atomicAdd(cnt + r, 1);
    const unsigned bit = 1u << kind_of(a.deg, i);
    if (!(kmask[r] & bit)) atomicOr(kmask + r, bit);
  }
}

__global__ void k_rows_fill(const PlanArgs a, int32_t* __restrict__ cursor) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= a.num_cells * a.k) return;
  const int32_t r = a.dofs[t];
  a.inc[atomicAdd(cursor + r, 1)] = (int32_t)t;
}

// sort key of a row: kind, window of 1024 rows (so that a warp's rows stay
// close in memory), number of cells; per kind its rows and the longest of them
// (totals[kind], totals[3 + kind])
__global__ void k_rows_keys(const PlanArgs a, const int32_t* __restrict__ cnt, const unsigned* __restrict__ kmask,
                            uint32_t* __restrict__ key, int32_t* __restrict__ row, int* __restrict__ totals) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int kind = -1, len = 0;
  if (r < a.num_rows) {
    const unsigned m = kmask[r];
    if (m & (m - 1)) *a.fail = 1u;  // a node that is a vertex here and an edge node there
    kind = m & 4u ? KIND_F : (m & 2u ? KIND_E : KIND_V);
    len = a.row_ptr[r + 1] - a.row_ptr[r];
    const int n = min(cnt[r], 255);
    key[r] = ((uint32_t)kind << 30) | ((uint32_t)(r >> 10) << 8) | (uint32_t)n;
    row[r] = (int32_t)r;
  }
  for (int k = 0; k < 3; ++k) {
    const unsigned here = __ballot_sync(kAll, kind == k);
    if (!here) continue;
    const int most = __reduce_max_sync(kAll, kind == k ? len : 0);
    if ((threadIdx.x & 31) != 0) continue;
    atomicAdd(totals + k, __popc(here));
    if (most > totals[3 + k]) atomicMax(totals + 3 + k, most);
  }
}

// the cell's vertices in the row's order: positions p[0..3]
__device__ __forceinline__ void row_order(int deg, int i, const int (&g)[4], int (&p)[4]) {
  const int lo[6] = {2, 1, 1, 0, 0, 0}, hi[6] = {3, 3, 2, 3, 2, 1};
  if (i < 4) {
    p[0] = i;
    int q = 1;
    for (int v = 0; v < 4; ++v)
      if (v != i) p[q++] = v;
  } else if (deg == 2 || i < 16) {
    const int e = deg == 2 ? i - 4 : (i - 4) / 2;
    int u = lo[e], v = hi[e];
    // P2: the lower mesh vertex first; P3: the vertex the node is near to
    const bool swap = deg == 2 ? g[u] > g[v] : ((i - 4) & 1);
    if (swap) {
      const int t = u;
      u = v;
      v = t;
    }
    p[0] = u;
    p[1] = v;
    int q = 2;
    for (int w = 0; w < 4; ++w)
      if (w != u && w != v) p[q++] = w;
  } else {
    const int f = i - 16;
    int q = 0;
    for (int v = 0; v < 4; ++v)
      if (v != f) p[q++] = v;
    for (int s = 0; s < 2; ++s)  // the face's vertices by their mesh index
      for (int t = 0; t < 2 - s; ++t)
        if (g[p[t]] > g[p[t + 1]]) {
          const int w = p[t];
          p[t] = p[t + 1];
          p[t + 1] = w;
        }
    p[3] = f;
  }
}

// slots of the columns every cell of the row has, packed one byte each
// (V: the row itself; E: a, b, the row, P3: the edge's other node)
__device__ __forceinline__ uint32_t own_slots(int deg, int kind, const uint8_t* q, int i, const int (&p)[4]) {
  if (kind == KIND_V) return q[i];
  uint32_t w = q[p[0]] | ((uint32_t)q[p[1]] << 8) | ((uint32_t)q[i] << 16);
  if (deg == 3) w |= (uint32_t)q[p3_edge(p[1], p[0])] << 24;
  return w;
}

struct PartArgs {
  int kind;
  int64_t nrows, ngroups;
  const int32_t* rows;   // [nrows] rows of this kind in walk order
  int4* own;             // [ngroups*32]
  int32_t* steps;        // [ngroups+1] records of the longest row of each group, then their prefix sum
  uint4* rec;
  uint4* rec2;           // P3: the rest of the records
  int4* own2;            // face rows: their own slots
  uint2* rec1;           // P1 records
  int32_t* cell;
  unsigned* gaps;        // set when a row has slots that no cell adds to
  int parts;             // vertex rows: warps that share a group's cells
};

__device__ __forceinline__ void load_cell(const PlanArgs& a, int32_t t, int64_t& c, int& i, int (&g)[4]) {
  c = t / a.k;
  i = t - (int32_t)c * a.k;
  const int4 v = reinterpret_cast<const int4*>(a.geom)[c];
  g[0] = v.x;
  g[1] = v.y;
  g[2] = v.z;
  g[3] = v.w;
}

// The triangles opposite a vertex in its cells, and for each of their edges
// (opposite corner e) the other triangle that has it.
constexpr int kNoTriangle = 255;
struct Star {
  int n;
  int tv[kMaxStar][3];           // mesh vertices
  uint8_t nb[kMaxStar][3];
  bool simple;                   // no edge is in three triangles, no triangle there twice
};

__device__ void load_star(const PlanArgs& a, const int32_t* inc, int n, Star& S) {
  S.n = n;
  S.simple = true;
  for (int t = 0; t < n; ++t) {
    int64_t c;
    int i, g[4];
    load_cell(a, inc[t], c, i, g);
    int q = 0;
    for (int v = 0; v < 4; ++v)
      if (v != i) S.tv[t][q++] = g[v];
    const int x = S.tv[t][0], y = S.tv[t][1], z = S.tv[t][2];
    if (x == y || x == z || y == z) S.simple = false;
    for (int e = 0; e < 3; ++e) S.nb[t][e] = kNoTriangle;
    for (int o = 0; o < t; ++o) {
      // corners that the other triangle does not have
      const int ox = S.tv[o][0], oy = S.tv[o][1], oz = S.tv[o][2];
      const int miss = (x != ox && x != oy && x != oz ? 1 : 0) | (y != ox && y != oy && y != oz ? 2 : 0) |
                       (z != ox && z != oy && z != oz ? 4 : 0);
      if (miss == 0) S.simple = false;
      if (miss != 1 && miss != 2 && miss != 4) continue;
      const int e = miss >> 1;  // 0, 1, 2
      const int f = ox != x && ox != y && ox != z ? 0 : (oy != x && oy != y && oy != z ? 1 : 2);
      if (S.nb[t][e] != kNoTriangle || S.nb[o][f] != kNoTriangle) S.simple = false;
      S.nb[t][e] = (uint8_t)o;
      S.nb[o][f] = (uint8_t)t;
    }
  }
}

// The cells of a vertex row as strips of the triangles opposite the vertex,
// cut into `parts` of nearly as many cells: emit(part, cell entry, its three
// other vertices, flags) for each step, cell entry -1 for the two steps that
// begin a strip; returns the steps of the longest part.  `code` says how the
// first strip begins: its triangle, which of its vertices is left first, and
// which way it goes at a tie.
template <typename Emit>
__device__ int walk_star(const Star& S, int parts, int code, Emit&& emit) {
  const int n = S.n;
  const int(*tv)[3] = S.tv;
  uint32_t used[kMaxStar / 32];
  for (int q = 0; q < kMaxStar / 32; ++q) used[q] = 0u;
  auto is_used = [&](int t) { return (used[t >> 5] >> (t & 31)) & 1u; };
  auto has = [&](int t, int v) { return tv[t][0] == v || tv[t][1] == v || tv[t][2] == v; };
  // the free triangle with vertices u and v, -1 if there is none
  auto find = [&](int u, int v) {
    for (int t = 0; t < n; ++t)
      if (!is_used(t) && has(t, u) && has(t, v)) return t;
    return -1;
  };
  auto third = [&](int t, int u, int v) {
    for (int q = 0; q < 3; ++q)
      if (tv[t][q] != u && tv[t][q] != v) return tv[t][q];
    return u;
  };
  // across the edge of t opposite its corner `off`, whose ends are u and v: the
  // first free triangle but t, -1 if there is none
  auto across = [&](int t, int off, int u, int v) -> int {
    if (!S.simple) return find(u, v);
    const int e = tv[t][0] == off ? 0 : (tv[t][1] == off ? 1 : 2);
    const int o = S.nb[t][e];
    return o != kNoTriangle && !is_used(o) ? o : -1;
  };
  int steps = 0, longest = 0, left = n, first = 0, part = 0, done = 0;
  auto next_part = [&]() {  // after `done` cells
    if (part + 1 < parts && done >= (part + 1) * n / parts) {
      ++part;
      longest = max(longest, steps);
      steps = 0;
      return true;
    }
    return false;
  };
  bool begun = false;
  while (left > 0) {
    while (begun && is_used(first)) ++first;
    int t = begun ? first : code / 6;
    used[t >> 5] |= 1u << (t & 31);
    --left;
    // its vertices, so that the strip can go on over (q, r)
    int p = tv[t][0], q = tv[t][1], r = tv[t][2];
    if (!begun) {
      const int turn = code / 2 % 3;
      p = tv[t][turn];
      q = tv[t][(turn + 1) % 3];
      r = tv[t][(turn + 2) % 3];
      begun = true;
    } else if (across(t, p, q, r) < 0) {
      if (across(t, q, p, r) >= 0) {
        const int w = p;
        p = q;
        q = w;
      } else if (across(t, r, p, q) >= 0) {
        const int w = p;
        p = r;
        r = w;
      }
    }
    emit(part, -1, p, 0, 0, kStripLoad);
    emit(part, -1, q, 0, 0, kStripLoad);
    steps += 2;
    while (true) {
      const int t1 = across(t, p, q, r), t2 = across(t, q, p, r);
      int next = t1;
      bool keep = false;
      if (t2 >= 0) {
        if (t1 < 0) {
          keep = true;
        } else {
          // towards the triangle with fewer free neighbours
          auto degree = [&](int x, int u, int v) {
            const int w = third(x, u, v);
            if (!S.simple)
              return (find(u, w) != x && find(u, w) >= 0 ? 1 : 0) + (find(v, w) != x && find(v, w) >= 0 ? 1 : 0);
            // (of the two triangles at an edge the search above sees the one listed first)
            const int ou = across(x, v, u, w), ov = across(x, u, v, w);
            return (ou >= 0 && ou < x ? 1 : 0) + (ov >= 0 && ov < x ? 1 : 0);
          };
          keep = degree(t2, p, r) < degree(t1, q, r) + (code & 1);
        }
        if (keep) next = t2;
      }
      emit(part, t, r, p, q, keep ? kStripKeep : 0u);
      ++steps;
      ++done;
      const bool cut = next_part();
      if (next < 0) break;
      if (!keep) p = q;
      q = r;
      r = third(next, p, q);
      t = next;
      if (cut) {
        emit(part, -1, p, 0, 0, kStripLoad);
        emit(part, -1, q, 0, 0, kStripLoad);
        steps += 2;
      }
      used[t >> 5] |= 1u << (t & 31);
      --left;
    }
  }
  return max(longest, steps);
}

// per row: its cells in ascending order, its own vertices and slots; per
// group the longest walk
__global__ void k_rows_head(const PlanArgs a, const PartArgs p) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t g32 = t >> 5;
  if (g32 >= p.ngroups) return;
  int4 own = make_int4(-1, -1, -1, 0), own2 = make_int4(0, 0, 0, 0);
  int n = 0;
  if (t < p.nrows) {
    const int32_t r = p.rows[t];
    const int32_t lo = a.inc_ptr[r];
    n = a.inc_ptr[r + 1] - lo;
    int32_t* inc = a.inc + lo;
    for (int q = 1; q < n; ++q) {
      const int32_t v = inc[q];
      int s = q;
      for (; s > 0 && inc[s - 1] > v; --s) inc[s] = inc[s - 1];
      inc[s] = v;
    }
    own.x = r;
    // a node of no cell: its row, in a pattern of the caller's own, may have its diagonal anywhere, or none
    if (n == 0) own.w = a.diag[r] < 0 ? -1 : a.diag[r] - a.row_ptr[r];
    for (int q = 0; q < n; ++q) {
      int64_t c;
      int i, g[4], o[4];
      load_cell(a, inc[q], c, i, g);
      row_order(a.deg, i, g, o);
      const uint32_t w =
          p.kind == KIND_F ? 0u : own_slots(a.deg, p.kind, a.pos + (c * a.k + i) * a.k, i, o);
      const int va = g[o[0]], vb = p.kind == KIND_V ? -1 : g[o[1]];
      int4 o2 = make_int4(0, 0, 0, 0);
      if (p.kind == KIND_F) {
        // a, b, c, ab ba ac ca bc cb, the face
        const uint8_t* b = a.pos + (c * a.k + i) * a.k;
        auto B = [&](int j) -> uint32_t { return b[j]; };
        o2.x = (int)(B(o[0]) | (B(o[1]) << 8) | (B(o[2]) << 16) | (B(p3_edge(o[0], o[1])) << 24));
        o2.y = (int)(B(p3_edge(o[1], o[0])) | (B(p3_edge(o[0], o[2])) << 8) | (B(p3_edge(o[2], o[0])) << 16) |
                     (B(p3_edge(o[1], o[2])) << 24));
        o2.z = (int)(B(p3_edge(o[2], o[1])) | (B(i) << 8));
      }
      if (q == 0) {
        own.y = va;
        own.z = vb;
        own.w = p.kind == KIND_F ? g[o[2]] : (int)w;
        own2 = o2;
      } else if (own.y != va || own.z != vb || (uint32_t)own.w != (p.kind == KIND_F ? (uint32_t)g[o[2]] : w) ||
                 own2.x != o2.x || own2.y != o2.y || own2.z != o2.z) {
        *a.fail = 1u;  // one dof, several vertices or edges; cells that name a common face's dofs differently
      }
    }
    if (p.kind == KIND_F) p.own2[t] = own2;
    if (p.kind == KIND_V) {
      if (n > kMaxStar) *a.fail = 1u;
      else if (n > 0) {
        // the beginning whose walk has the fewest steps; one strip around the
        // whole star, n + 2 steps, is found in two or three tries as a rule
        Star S;
        load_star(a, inc, n, S);
        auto steps_of = [&](int parts, int code) {
          return walk_star(S, parts, code, [](int, int, int, int, int, uint32_t) {});
        };
        int best = 0, least = steps_of(1, 0);
        for (int code = 1; code < min(6 * n, kStripTries) && least > n + 2; ++code) {
          const int steps = steps_of(1, code);
          if (steps < least) {
            least = steps;
            best = code;
          }
        }
        own.z = best;
        n = p.parts == 1 ? least : steps_of(p.parts, best);
      }
    }
  }
  p.own[t] = own;
  for (int o = 16; o > 0; o >>= 1) n = max(n, __shfl_xor_sync(kAll, n, o));
  if ((t & 31) == 0) p.steps[g32] = n * p.parts;
}

// the records of every (step, lane)
__global__ void k_rows_records(const PlanArgs a, const PartArgs p) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t g32 = t >> 5;
  const int lane = (int)(t & 31);
  if (g32 >= p.ngroups) return;
  int n = 0;
  const int32_t* inc = nullptr;
  int32_t r = -1;
  if (t < p.nrows) {
    r = p.rows[t];
    inc = a.inc + a.inc_ptr[r];
    n = a.inc_ptr[r + 1] - a.inc_ptr[r];
  }
  const int64_t s0 = p.steps[g32];
  const int ns = p.steps[g32 + 1] - p.steps[g32];
  uint64_t used = 0;  // edge rows: cells already listed (all of them below 64)
  int last = -1;      // mesh vertex the next cell around the edge shares
  int fan = -1;       // the vertex its fan began with
  uint2 begun = make_uint2(0u, 0u), left = make_uint2(0u, 0u);  // edge rows: slots of the fan's first and last vertex
  uint32_t seen[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};  // slots some cell adds to
  uint32_t written[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  auto mark = [&](uint32_t b) { seen[b >> 5] |= 1u << (b & 31u); };
  auto write = [&](uint32_t b) {
    if ((written[b >> 5] >> (b & 31u)) & 1u) *a.fail = 1u;
    written[b >> 5] |= 1u << (b & 31u);
  };
  if (p.kind == KIND_V) {
    const int np = ns / p.parts;  // steps of a part
    int at_part = -1, s = 0;
    auto rest = [&]() {  // the part's steps without a cell
      for (; at_part >= 0 && s < np; ++s) {
        const int64_t at = (s0 + at_part * np + s) * 32 + lane;
        p.cell[at] = 0;
        if (a.deg == 1) p.rec1[at] = make_uint2(kStripLoad, 0u);
        else p.rec[at] = make_uint4(kStripLoad, 0u, 0u, 0u);
        if (a.deg == 3) p.rec2[at] = make_uint4(0u, 0u, 0u, 0u);
      }
    };
    if (n > 0 && n <= kMaxStar) {
      Star S;
      load_star(a, inc, n, S);
      walk_star(S, p.parts, p.own[t].z, [&](int part, int t, int r3, int p3, int q3, uint32_t flags) {
        while (at_part < part) {
          rest();
          ++at_part;
          s = 0;
        }
        const int64_t at = (s0 + part * np + s++) * 32 + lane;
        uint4 w = make_uint4((uint32_t)r3 | flags, 0u, 0u, 0u), w2 = make_uint4(0u, 0u, 0u, 0u);
        p.cell[at] = 0;
        if (t >= 0) {
          int64_t c;
          int i, g[4];
          load_cell(a, inc[t], c, i, g);
          int lp = 0, lq = 0, lr = 0;
          for (int v = 0; v < 4; ++v) {
            if (v == i) continue;
            if (g[v] == p3) lp = v;
            else if (g[v] == q3) lq = v;
            else lr = v;
          }
          const uint8_t* q = a.pos + (c * a.k + i) * a.k;
          auto B = [&](int j) -> uint32_t { return q[j]; };
          for (int j = 0; j < a.k; ++j) mark(B(j));
          p.cell[at] = (int32_t)c;
          w.y = B(lp) | (B(lq) << 8) | (B(lr) << 16);
          if (a.deg == 2) {
            w.y |= B(p2_edge(i, lp)) << 24;
            w.z = B(p2_edge(i, lq)) | (B(p2_edge(i, lr)) << 8) | (B(p2_edge(lp, lq)) << 16) |
                  (B(p2_edge(lp, lr)) << 24);
            w.w = B(p2_edge(lq, lr));
          } else if (a.deg == 3) {
            auto E = [&](int x, int y) { return B(p3_edge(x, y)); };
            w.y |= E(i, lp) << 24;
            w.z = E(lp, i) | (E(i, lq) << 8) | (E(lq, i) << 16) | (E(i, lr) << 24);
            w.w = E(lr, i) | (E(lp, lq) << 8) | (E(lq, lp) << 16) | (E(lp, lr) << 24);
            w2.x = E(lr, lp) | (E(lq, lr) << 8) | (E(lr, lq) << 16) | (B(16 + lr) << 24);
            w2.y = B(16 + lq) | (B(16 + lp) << 8) | (B(16 + i) << 16);
          }
        }
        if (a.deg == 1) p.rec1[at] = make_uint2(w.x, w.y);
        else p.rec[at] = w;
        if (a.deg == 3) p.rec2[at] = w2;
      });
    }
    while (at_part < p.parts) {
      rest();
      ++at_part;
      s = 0;
    }
  }
  for (int s = 0; s < (p.kind == KIND_E ? ns : 0); ++s) {
    const int64_t at = (s0 + s) * 32 + lane;
    if (s >= n) {
      p.cell[at] = 0;
      p.rec[at] = make_uint4(kAll, kAll, 0u, 0u);
      if (a.deg == 3) p.rec2[at] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    int64_t c;
    int i, g[4], o[4];
    uint32_t flags = kFanBegin | kFanEnd;  // edge rows: a fan of one cell
    if (n <= 64) {
      // the next unlisted cell with the last vertex; else one that has a
      // vertex no other unlisted cell has (an end of an open fan); else the first
      int pick = -1, end = -1, first = -1;
      for (int q = 0; q < n && pick < 0; ++q) {
        if ((used >> q) & 1u) continue;
        load_cell(a, inc[q], c, i, g);
        row_order(a.deg, i, g, o);
        if (first < 0) first = q;
        if (last >= 0) {
          if (g[o[2]] == last || g[o[3]] == last) pick = q;
          continue;
        }
        int shared[2] = {0, 0};
        for (int q2 = 0; q2 < n; ++q2) {
          if (q2 == q || ((used >> q2) & 1u)) continue;
          int64_t c2;
          int i2, g2[4], o2[4];
          load_cell(a, inc[q2], c2, i2, g2);
          row_order(a.deg, i2, g2, o2);
          for (int e = 0; e < 2; ++e) shared[e] |= g[o[2 + e]] == g2[o2[2]] || g[o[2 + e]] == g2[o2[3]];
        }
        if (end < 0 && !(shared[0] && shared[1])) {
          end = q;
          last = -1;
        }
      }
      if (pick < 0) pick = end >= 0 ? end : first;
      used |= uint64_t(1) << pick;
      load_cell(a, inc[pick], c, i, g);
      row_order(a.deg, i, g, o);
      bool swap = last >= 0 && g[o[3]] == last;
      if (last < 0 || (g[o[2]] != last && g[o[3]] != last)) {
        // a new fan: begin with the vertex that no other unlisted cell has
        bool s2 = false, s3 = false;
        for (int q2 = 0; q2 < n; ++q2) {
          if ((used >> q2) & 1u) continue;
          int64_t c2;
          int i2, g2[4], o2[4];
          load_cell(a, inc[q2], c2, i2, g2);
          row_order(a.deg, i2, g2, o2);
          s2 |= g[o[2]] == g2[o2[2]] || g[o[2]] == g2[o2[3]];
          s3 |= g[o[3]] == g2[o2[2]] || g[o[3]] == g2[o2[3]];
        }
        swap = s2 && !s3;
      }
      if (swap) {
        const int w = o[2];
        o[2] = o[3];
        o[3] = w;
      }
      flags = 0u;
      if (last < 0 || g[o[2]] != last) {
        flags |= kFanBegin;
        fan = g[o[2]];
      }
      last = g[o[3]];
      // the fan ends when no unlisted cell has its last vertex
      bool more = false;
      for (int q2 = 0; q2 < n && !more; ++q2) {
        if ((used >> q2) & 1u) continue;
        int64_t c2;
        int i2, g2[4], o2[4];
        load_cell(a, inc[q2], c2, i2, g2);
        row_order(a.deg, i2, g2, o2);
        more = g2[o2[2]] == last || g2[o2[3]] == last;
      }
      if (!more) {
        flags |= kFanEnd;
        if (last == fan) flags |= kFanClosed;
        last = -1;
      }
    } else {
      load_cell(a, inc[s], c, i, g);
      row_order(a.deg, i, g, o);
    }
    const uint8_t* q = a.pos + (c * a.k + i) * a.k;
    auto B = [&](int j) -> uint32_t { return q[j]; };
    for (int j = 0; j < a.k; ++j) mark(B(j));
    p.cell[at] = (int32_t)c;
    {
      // the walk adds a cell's entries of vertex d (d ad bd, P3: d ad da bd db abd) to the next cell's of c, at
      // the end of a closed fan to the first cell's: both cells have to name those dofs alike
      auto slots_of = [&](int v, int opposite) {
        if (a.deg == 2) return make_uint2(B(o[v]) | (B(p2_edge(o[0], o[v])) << 8) | (B(p2_edge(o[1], o[v])) << 16), 0u);
        return make_uint2(B(o[v]) | (B(p3_edge(o[0], o[v])) << 8) | (B(p3_edge(o[v], o[0])) << 16) |
                              (B(p3_edge(o[1], o[v])) << 24),
                          B(p3_edge(o[v], o[1])) | (B(16 + o[opposite]) << 8));
      };
      const uint2 sc = slots_of(2, 3), sd = slots_of(3, 2);
      if (flags & kFanBegin) begun = sc;
      else if (sc.x != left.x || sc.y != left.y) *a.fail = 1u;
      if ((flags & kFanClosed) && (sd.x != begun.x || sd.y != begun.y)) *a.fail = 1u;
      left = sd;
    }
    if (a.deg == 3) {
      // slots: the six of vertex c (c, ac ca bc cb, abc), the six of d, then cd dc acd bcd
      auto E = [&](int x, int y) { return B(p3_edge(o[x], o[y])); };
      uint4 w, w2;
      w.x = (uint32_t)g[o[2]];
      w.y = (uint32_t)g[o[3]];
      w.z = B(o[2]) | (E(0, 2) << 8) | (E(2, 0) << 16) | (E(1, 2) << 24);
      w.w = E(2, 1) | (B(16 + o[3]) << 8) | (B(o[3]) << 16) | (E(0, 3) << 24);
      w2.x = E(3, 0) | (E(1, 3) << 8) | (E(3, 1) << 16) | (B(16 + o[2]) << 24);
      w2.y = E(2, 3) | (E(3, 2) << 8) | (B(16 + o[1]) << 16) | (B(16 + o[0]) << 24);
      w2.z = flags;
      w2.w = 0u;
      p.rec[at] = w;
      p.rec2[at] = w2;
      const uint32_t cs[6] = {w.z & 0xffu, (w.z >> 8) & 0xffu, (w.z >> 16) & 0xffu,
                              w.z >> 24,   w.w & 0xffu,        (w.w >> 8) & 0xffu};
      const uint32_t ds[6] = {(w.w >> 16) & 0xffu, w.w >> 24,           w2.x & 0xffu,
                              (w2.x >> 8) & 0xffu, (w2.x >> 16) & 0xffu, w2.x >> 24};
      for (int q2 = 0; q2 < 6; ++q2) write(cs[q2]);
      for (int q2 = 0; q2 < 4; ++q2) write((w2.y >> (8 * q2)) & 0xffu);
      if ((flags & kFanEnd) && !(flags & kFanClosed))
        for (int q2 = 0; q2 < 6; ++q2) write(ds[q2]);
    } else {
      uint4 w;
      w.x = (uint32_t)g[o[2]];
      w.y = (uint32_t)g[o[3]];
      w.z = B(o[2]) | (B(o[3]) << 8) | (B(p2_edge(o[0], o[2])) << 16) | (B(p2_edge(o[0], o[3])) << 24);
      w.w = B(p2_edge(o[1], o[2])) | (B(p2_edge(o[1], o[3])) << 8) | (B(p2_edge(o[2], o[3])) << 16) |
            (flags << 24);
      p.rec[at] = w;
      // the walk writes a slot once (twice at the end of a closed fan): cells
      // that overlap, or three at one face, are left to the scatter
      write(w.z & 0xffu);
      write((w.z >> 16) & 0xffu);
      write(w.w & 0xffu);
      write((w.w >> 16) & 0xffu);
      if ((flags & kFanEnd) && !(flags & kFanClosed)) {
        write((w.z >> 8) & 0xffu);
        write(w.z >> 24);
        write((w.w >> 8) & 0xffu);
      }
    }
  }
  for (int s = 0; s < (p.kind == KIND_F ? ns : 0); ++s) {
    const int64_t at = (s0 + s) * 32 + lane;
    uint4 w = make_uint4(kAll, 0u, 0u, 0u);
    p.cell[at] = 0;
    if (s < n) {
      int64_t c;
      int i, g[4], o[4];
      load_cell(a, inc[s], c, i, g);
      row_order(a.deg, i, g, o);
      const uint8_t* q = a.pos + (c * a.k + i) * a.k;
      auto B = [&](int j) -> uint32_t { return q[j]; };
      auto E = [&](int x, int y) { return B(p3_edge(o[x], o[y])); };
      for (int j = 0; j < a.k; ++j) mark(B(j));
      // slots: d, ad da bd db cd dc, abd acd bcd
      w.x = (uint32_t)g[o[3]];
      w.y = B(o[3]) | (E(0, 3) << 8) | (E(3, 0) << 16) | (E(1, 3) << 24);
      w.z = E(3, 1) | (E(2, 3) << 8) | (E(3, 2) << 16) | (B(16 + o[2]) << 24);
      w.w = B(16 + o[1]) | (B(16 + o[0]) << 8);
      p.cell[at] = (int32_t)c;
      for (int q2 = 0; q2 < 4; ++q2) write((w.y >> (8 * q2)) & 0xffu);
      for (int q2 = 0; q2 < 4; ++q2) write((w.z >> (8 * q2)) & 0xffu);
      for (int q2 = 0; q2 < 2; ++q2) write((w.w >> (8 * q2)) & 0xffu);
    }
    p.rec[at] = w;
  }
  if (r >= 0) {
    int covered = 0;
    for (int q = 0; q < 8; ++q) covered += __popc(seen[q]);
    if (covered != a.row_ptr[r + 1] - a.row_ptr[r]) *p.gaps = 1u;
  }
}

__global__ void k_rows_pad_x(const double* __restrict__ x, int64_t n, double4* __restrict__ x4) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v < n) x4[v] = make_double4(x[3 * v], x[3 * v + 1], x[3 * v + 2], 0.0);
}

__global__ void k_rows_same_map(const int32_t* __restrict__ m, const int32_t* __restrict__ g, int64_t n,
                                unsigned* __restrict__ differ) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < n && m[t] != g[t]) *differ = 1u;
}

// ---------------------------------------------------------------------------
// assembly
// ---------------------------------------------------------------------------
struct WalkArgs : RowOut {
  int64_t ngroups;
  const int4* __restrict__ own;
  const int32_t* __restrict__ steps;
  const uint4* __restrict__ rec;
  const uint4* __restrict__ rec2;
  const int4* __restrict__ own2;
  const uint2* __restrict__ rec1;
  const int32_t* __restrict__ cell;
  const double4* __restrict__ x4;
  int gaps;       // some rows have slots that no cell adds to
  const double* __restrict__ coef;   // DG0: [cells]; P1: [vertices]
  double coef_const;
};

struct V3 {
  double x, y, z;
};
__device__ __forceinline__ V3 operator-(const V3& a, const V3& b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot(const V3& a, const V3& b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ V3 cross(const V3& a, const V3& b) {
  return {fma(a.y, b.z, -(a.z * b.y)), fma(a.z, b.x, -(a.x * b.z)), fma(a.x, b.y, -(a.y * b.x))};
}
__device__ __forceinline__ V3 neg_sum(const V3& a, const V3& b, const V3& c) {
  return {-(a.x + b.x + c.x), -(a.y + b.y + c.y), -(a.z + b.z + c.z)};
}
__device__ __forceinline__ V3 load_x(const double4* __restrict__ x4, int v) {
  const double2* p = reinterpret_cast<const double2*>(x4 + v);
  const double2 a = __ldg(p);
  const double b = __ldg(reinterpret_cast<const double*>(p + 1));
  return {a.x, a.y, b};
}

// One warp a CTA: a finished warp's shared memory goes to the next one at once
// (P2 n=96: 1.15 ms against 1.22 ms with CTAs of two and four warps).
// CTAs per SM to fit in registers (fewer registers spill, more leave too few
// warps):
constexpr int kMinV1 = 20, kMinV2 = 13, kMinE = 20, kMinE3 = 16, kMinF3 = 20;

// Vertex rows (P1: all rows): the cells around vertex a as strips, each with
// its three other vertices p, q, r, where r is fetched and p, q are two of
// the cell's before.
// PARTS warps share the rows of a group, each with its part of every row's
// cells and segments of its own, which are added up at the end.
template <int DEG, int COEF, int PARTS>
__global__ void __launch_bounds__(32 * PARTS, (DEG == 1 ? kMinV1 : kMinV2) / PARTS) k_rows_v(const WalkArgs a) {
  let_next_start();
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, part = PARTS == 1 ? 0 : threadIdx.x >> 5;
  const int64_t g = blockIdx.x;
  double* acc = smem + part * (32 * a.stride);
  double* seg = acc + lane * a.stride;
  const int4 own = __ldg(a.own + g * 32 + lane);
  int s0 = __ldg(a.steps + g);
  const int ns = (__ldg(a.steps + g + 1) - s0) / PARTS;
  s0 += part * ns;
  const uint4* rec = a.rec + (int64_t)s0 * 32 + lane;
  const uint2* rec1 = a.rec1 + (int64_t)s0 * 32 + lane;
  const int32_t* cell = a.cell + (int64_t)s0 * 32 + lane;
  int c1 = 0, c2 = 0;  // the records' cells (DG0)
  auto record = [&](int s) {
    uint4 w = make_uint4(kStripLoad, 0u, 0u, 0u);
    c1 = c2;
    if (s < ns) {
      if constexpr (COEF == FE_COEFF_DG0) c2 = __ldg(cell + s * 32);
      if constexpr (DEG == 1) {
        const uint2 h = __ldg(rec1 + s * 32);
        w.x = h.x;
        w.y = h.y;
      } else {
        w = __ldg(rec + s * 32);
      }
    }
    return w;
  };
  // the records run two steps ahead, the coordinates and the coefficient one
  uint4 w1 = record(0), w2 = record(1);
  const RowAt at = row_at(a, own.x);
  V3 xa{0.0, 0.0, 0.0}, xr, ep{0.0, 0.0, 0.0}, eq{0.0, 0.0, 0.0};
  double ka = 1.0, kp = 1.0, kq = 1.0, kn = a.coef_const;
  auto fetch = [&](const uint4& w) {
    const int v = (int)(w.x & kStripVertex);
    xr = load_x(a.x4, v);
    if constexpr (COEF == FE_COEFF_P1) kn = __ldg(a.coef + v);
    if constexpr (COEF == FE_COEFF_DG0) kn = __ldg(a.coef + c1);
  };
  fetch(w1);
  if (own.y >= 0) {
    xa = load_x(a.x4, own.y);
    if constexpr (COEF == FE_COEFF_P1) ka = __ldg(a.coef + own.y);
  }
  for (int s = 0; s < a.stride; ++s) seg[s] = 0.0;
  double diag = 0.0;
  for (int s = 0; s < ns; ++s) {
    const uint4 w = w1;
    w1 = w2;
    w2 = record(s + 2);
    const V3 er = xr - xa;
    const double kr = kn;
    fetch(w1);
    if (!(w.x & kStripLoad)) {
      const V3 gp = cross(eq, er), gq = cross(er, ep), gr = cross(ep, eq);
      const V3 ga = neg_sum(gp, gq, gr);
      const double rdet = 1.0 / fabs(dot(ep, gp));
      const double ap = dot(ga, gp), aq = dot(ga, gq), ar = dot(ga, gr);
      const double aa = -(ap + aq + ar);
      constexpr int NV = DEG == 1 ? 3 : 9;
      double v[NV];  // columns p, q, r, ap, aq, ar, pq, pr, qr
      if constexpr (DEG == 1) {
        // k |T| grad.grad with the cell mean of k (exact: the gradients are constant)
        double f;
        if constexpr (COEF == FE_COEFF_P1) f = (1.0 / 24.0) * ((ka + kp) + (kq + kr)) * rdet;
        else f = (1.0 / 6.0) * kr * rdet;
        v[0] = f * ap;
        v[1] = f * aq;
        v[2] = f * ar;
        diag = fma(f, aa, diag);
      } else if constexpr (COEF == FE_COEFF_P1) {
        const double S = (ka + kp) + (kq + kr);
        const double f = (1.0 / 720.0) * rdet, f4 = 4.0 * f, m2 = -2.0 * S;
        diag = fma(f * fma(14.0, S, 16.0 * ka), aa, diag);
        v[0] = f * fma(-8.0, ka + kp, m2) * ap;
        v[1] = f * fma(-8.0, ka + kq, m2) * aq;
        v[2] = f * fma(-8.0, ka + kr, m2) * ar;
        // column ap: (2S + 10 k_a) ap + (-2S + 4 k_a - 2 k_p) aa
        const double y = fma(10.0, ka, -m2), t = fma(4.0, ka, m2);
        const double tp = fma(-2.0, kp, t), tq = fma(-2.0, kq, t), tr = fma(-2.0, kr, t);
        v[3] = f4 * fma(y, ap, tp * aa);
        v[4] = f4 * fma(y, aq, tq * aa);
        v[5] = f4 * fma(y, ar, tr * aa);
        // column pq: (-2S + 4 k_a - 2 k_p) aq + (-2S + 4 k_a - 2 k_q) ap
        v[6] = f4 * fma(tp, aq, tq * ap);
        v[7] = f4 * fma(tp, ar, tr * ap);
        v[8] = f4 * fma(tq, ar, tr * aq);
      } else {
        const double f = (1.0 / 30.0) * kr * rdet;  // 4 k / 120
        diag = fma(3.0 * f, aa, diag);
        v[0] = -f * ap;
        v[1] = -f * aq;
        v[2] = -f * ar;
        v[3] = f * fma(3.0, ap, -aa);
        v[4] = f * fma(3.0, aq, -aa);
        v[5] = f * fma(3.0, ar, -aa);
        v[6] = -f * (ap + aq);
        v[7] = -f * (ap + ar);
        v[8] = -f * (aq + ar);
      }
      const uint32_t sl[9] = {w.y & 0xffu, (w.y >> 8) & 0xffu, (w.y >> 16) & 0xffu, w.y >> 24, w.z & 0xffu,
                              (w.z >> 8) & 0xffu, (w.z >> 16) & 0xffu, w.z >> 24, w.w};
      // a cell's columns differ: all reads before the writes
      double o[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) o[q] = seg[sl[q]];
#pragma unroll
      for (int q = 0; q < NV; ++q) seg[sl[q]] = o[q] + v[q];
    }
    if (!(w.x & kStripKeep)) {
      ep = eq;
      kp = kq;
    }
    eq = er;
    kq = kr;
  }
  if (own.y >= 0) seg[own.w] += diag;
  if constexpr (PARTS > 1) {
    __syncthreads();
    for (int t = threadIdx.x; t < 32 * a.stride; t += 32 * PARTS) {
      double v = smem[t];
#pragma unroll
      for (int q = 1; q < PARTS; ++q) v += smem[q * (32 * a.stride) + t];
      smem[t] = v;
    }
    __syncthreads();
  }
  constexpr int kRows = 32 / PARTS;
  store_rows(a, smem, at, own.w, lane, part * kRows, kRows);
}

// Edge rows of P2: node ab; the cells around the edge in fans, each with its
// two other vertices c, d, where d is the next cell's c.  The columns c, ac
// and bc take entries of the two cells with the face abc, one after the
// other: their sum runs in registers and is written once, cd belongs to one
// cell, and a, b and ab stay in registers, so the segment is written without
// being read (but for the end of a closed fan).
template <int COEF>
__global__ void __launch_bounds__(32, kMinE) k_rows_e2(const WalkArgs a) {
  extern __shared__ double smem[];
  const int lane = threadIdx.x;
  const int64_t g = blockIdx.x;
  double* acc = smem;
  double* seg = acc + lane * a.stride;
  const int4 own = __ldg(a.own + g * 32 + lane);
  const int s0 = __ldg(a.steps + g), ns = __ldg(a.steps + g + 1) - s0;
  const uint4 none = make_uint4(kAll, kAll, 0u, 0u);
  const uint4* rec = a.rec + (int64_t)s0 * 32 + lane;
  const int32_t* cell = a.cell + (int64_t)s0 * 32 + lane;
  // the records run two cells ahead, the coordinates and the coefficient one
  uint4 wp = ns > 0 ? __ldg(rec) : none, wq = ns > 1 ? __ldg(rec + 32) : none;
  const RowAt at = row_at(a, own.x);
  V3 xa{0.0, 0.0, 0.0}, e1{0.0, 0.0, 0.0}, xd{0.0, 0.0, 0.0};
  double ka = 1.0, kb = 1.0, kn = a.coef_const;
  int c1 = 0, c2 = 0;  // the records' cells (DG0)
  if constexpr (COEF == FE_COEFF_DG0) {
    if (ns > 0) c1 = __ldg(cell);
    if (ns > 1) c2 = __ldg(cell + 32);
  }
  auto fetch = [&](const uint4& w) {
    if (w.y == kAll) return;
    xd = load_x(a.x4, (int)w.y);
    if constexpr (COEF == FE_COEFF_P1) kn = __ldg(a.coef + w.y);
    if constexpr (COEF == FE_COEFF_DG0) kn = __ldg(a.coef + c1);
  };
  if (own.y >= 0) {
    xa = load_x(a.x4, own.y);
    e1 = load_x(a.x4, own.z) - xa;
    if constexpr (COEF == FE_COEFF_P1) {
      ka = __ldg(a.coef + own.y);
      kb = __ldg(a.coef + own.z);
    }
  }
  fetch(wp);
  if (a.gaps)
    for (int s = 0; s < a.stride; ++s) seg[s] = 0.0;
  double va = 0.0, vb = 0.0, vab = 0.0;  // columns a, b and ab
  double rc = 0.0, rac = 0.0, rbc = 0.0; // columns c, ac and bc so far
  // one cell: c, its edge vector from a, e1 x c and its coefficient come from
  // the cell before (or are fetched where a fan begins), d's go to the next
  auto step = [&](const uint4& w, const uint4& wnext, V3& ec, V3& hc, double& kc, V3& ed, V3& hd, double& kd) {
    if (w.y != kAll) {
      if ((w.w >> 24) & kFanBegin) {
        ec = load_x(a.x4, (int)w.x) - xa;
        if constexpr (COEF == FE_COEFF_P1) kc = __ldg(a.coef + w.x);
        rc = rac = rbc = 0.0;
      }
      ed = xd - xa;
      const double k = kn;
      kd = kn;
      fetch(wnext);
      hd = cross(e1, ed);
      hc = cross(e1, ec);
      // times det: grad b = c x d, grad c = -(e1 x d), grad d = e1 x c
      const V3 gb = cross(ec, ed);
      const V3 ga{hd.x - hc.x - gb.x, hd.y - hc.y - gb.y, hd.z - hc.z - gb.z};
      const double rdet = 1.0 / fabs(dot(e1, gb));
      const double ab = dot(ga, gb), ac = -dot(ga, hd), ad = dot(ga, hc), bc = -dot(gb, hd), bd = dot(gb, hc);
      const double aa = -(ab + ac + ad), bb = -(ab + bc + bd);
      double vd, vad, vbd, vcd;
      if constexpr (COEF == FE_COEFF_P1) {
        // integrals of k lambda_x lambda_y, in units of |det| / 720: S + k_x + k_y,
        // twice that for x = y
        const double S = (ka + kb) + (kc + kd);
        const double f4 = (4.0 / 720.0) * rdet, f16 = (16.0 / 720.0) * rdet, m2 = -2.0 * S;
        const double Sa = S + ka, Sb = S + kb;
        const double Maa = fma(4.0, ka, -m2), Mbb = fma(4.0, kb, -m2), Mab = Sa + kb;
        const double Mac = Sa + kc, Mad = Sa + kd, Mbc = Sb + kc, Mbd = Sb + kd;
        vab = fma(f16, fma(Maa, bb, fma(Mbb, aa, 2.0 * Mab * ab)), vab);
        va = fma(f4, fma(fma(10.0, ka, -m2), ab, fma(4.0, ka, fma(-2.0, kb, m2)) * aa), va);
        vb = fma(f4, fma(fma(10.0, kb, -m2), ab, fma(4.0, kb, fma(-2.0, ka, m2)) * bb), vb);
        const double ta = fma(-2.0, ka, m2), tb = fma(-2.0, kb, m2);
        rc = fma(f4, fma(fma(4.0, kc, ta), bc, fma(4.0, kc, tb) * ac), rc);
        vd = f4 * fma(fma(4.0, kd, ta), bd, fma(4.0, kd, tb) * ad);
        rac = fma(f16, fma(Maa, bc, fma(Mac, ab, fma(Mab, ac, Mbc * aa))), rac);
        vad = f16 * fma(Maa, bd, fma(Mad, ab, fma(Mab, ad, Mbd * aa)));
        rbc = fma(f16, fma(Mbb, ac, fma(Mbc, ab, fma(Mab, bc, Mac * bb))), rbc);
        vbd = f16 * fma(Mbb, ad, fma(Mbd, ab, fma(Mab, bd, Mad * bb)));
        vcd = f16 * fma(Mac, bd, fma(Mad, bc, fma(Mbc, ad, Mbd * ac)));
      } else {
        const double f = (1.0 / 30.0) * k * rdet, f16 = 4.0 * f;  // 4 k / 120, 16 k / 120
        vab = fma(2.0 * f16, (aa + bb) + ab, vab);
        va = fma(f, fma(3.0, ab, -aa), va);
        vb = fma(f, fma(3.0, ab, -bb), vb);
        rc = fma(-f, ac + bc, rc);
        vd = -f * (ad + bd);
        rac = fma(f16, fma(2.0, bc, -ad), rac);
        vad = f16 * fma(2.0, bd, -ac);
        rbc = fma(f16, fma(2.0, ac, -bd), rbc);
        vbd = f16 * fma(2.0, ad, -bc);
        vcd = f16 * ((ac + ad) + (bc + bd));
      }
      seg[w.z & 0xffu] = rc;
      seg[(w.z >> 16) & 0xffu] = rac;
      seg[w.w & 0xffu] = rbc;
      seg[(w.w >> 16) & 0xffu] = vcd;
      rc = vd;
      rac = vad;
      rbc = vbd;
      if ((w.w >> 24) & kFanEnd) {
        double* pd = seg + ((w.z >> 8) & 0xffu);
        double* pad = seg + (w.z >> 24);
        double* pbd = seg + ((w.w >> 8) & 0xffu);
        if ((w.w >> 24) & kFanClosed) {
          rc += *pd;
          rac += *pad;
          rbc += *pbd;
        }
        *pd = rc;
        *pad = rac;
        *pbd = rbc;
      }
    }
  };
  V3 ep{0.0, 0.0, 0.0}, eq{0.0, 0.0, 0.0}, hp{0.0, 0.0, 0.0}, hq{0.0, 0.0, 0.0};
  double kp = 1.0, kq = 1.0;
  for (int s = 0; s < ns; ++s) {
    uint4 w = wp;
    wp = wq;
    wq = s + 2 < ns ? __ldg(rec + (s + 2) * 32) : none;
    if constexpr (COEF == FE_COEFF_DG0) {
      c1 = c2;
      if (s + 2 < ns) c2 = __ldg(cell + (s + 2) * 32);
    }
    step(w, wp, ep, hp, kp, eq, hq, kq);
    ep = eq;
    hp = hq;
    kp = kq;
  }
  if (own.y >= 0) {
    seg[own.w & 0xff] = va;
    seg[(own.w >> 8) & 0xff] = vb;
    seg[(own.w >> 16) & 0xff] = vab;
  }
  store_rows(a, acc, at, (own.w >> 16) & 0xff, lane, 0, 32);
  end_after_previous();
}

// ---------------------------------------------------------------------------
// P3 (constant or cellwise k): the same walks with 20 columns a cell, and one
// for face nodes.  An entry is a combination of the six products of the
// gradients (p3_row_v, p3_row_e, p3_row_f, generated from exact integrals).
// Bound by latency at 10 (V), 14 (E) and 16 (F) warps per SM: the FP64 pipe is
// busy 12 % of the time, half of the instructions are integer ones (slots, the
// stores of rows of 20 to 175 entries).  P3 n=36: 0.34 ms against 0.63 ms for
// the warp-coalesced scatter (0.38 ms with one warp for a vertex group).
// ---------------------------------------------------------------------------
template <int COEF>
__device__ __forceinline__ double cell_k(const WalkArgs& a, int c) {
  if constexpr (COEF == FE_COEFF_DG0) return __ldg(a.coef + c);
  else return a.coef_const;
}

// Vertex rows: two warps take the columns of each part (the nodes of vertices
// and of the edges at a, and the others: never the same slot of a row), as the
// segments of 175 slots leave room for few groups.
template <int COEF, int PARTS>
__global__ void __launch_bounds__(64 * PARTS) k_rows_v3(const WalkArgs a) {
  extern __shared__ double smem[];
  let_next_start();
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 6;
  const bool outer = (threadIdx.x >> 5) & 1;
  const int64_t g = blockIdx.x;
  double* acc = smem + part * (32 * a.stride);
  double* seg = acc + lane * a.stride;
  const int4 own = __ldg(a.own + g * 32 + lane);
  int s0 = __ldg(a.steps + g);
  const int ns = (__ldg(a.steps + g + 1) - s0) / PARTS;
  s0 += part * ns;
  const uint4* rec = a.rec + (int64_t)s0 * 32 + lane;
  const uint4* rec2 = a.rec2 + (int64_t)s0 * 32 + lane;
  const int32_t* cell = a.cell + (int64_t)s0 * 32 + lane;
  const uint4 none = make_uint4(kStripLoad, 0u, 0u, 0u), zero4 = make_uint4(0u, 0u, 0u, 0u);
  // records two steps ahead, coordinates and coefficient one
  uint4 w1 = ns > 0 ? __ldg(rec) : none, w2 = ns > 1 ? __ldg(rec + 32) : none;
  uint4 u1 = ns > 0 ? __ldg(rec2) : zero4, u2 = ns > 1 ? __ldg(rec2 + 32) : zero4;
  int c1 = COEF == FE_COEFF_DG0 && ns > 0 ? __ldg(cell) : 0, c2 = COEF == FE_COEFF_DG0 && ns > 1 ? __ldg(cell + 32) : 0;
  const RowAt at = row_at(a, own.x);
  V3 xa{0.0, 0.0, 0.0}, xr = load_x(a.x4, (int)(w1.x & kStripVertex)), ep{0.0, 0.0, 0.0}, eq{0.0, 0.0, 0.0};
  double kn = cell_k<COEF>(a, c1);
  if (own.y >= 0) xa = load_x(a.x4, own.y);
  for (int s = outer ? 1 : 0; s < a.stride; s += 2) seg[s] = 0.0;
  __syncthreads();
  double diag = 0.0;
  for (int s = 0; s < ns; ++s) {
    const uint4 w = w1, u = u1;
    w1 = w2;
    u1 = u2;
    c1 = c2;
    w2 = s + 2 < ns ? __ldg(rec + (s + 2) * 32) : none;
    u2 = s + 2 < ns ? __ldg(rec2 + (s + 2) * 32) : zero4;
    if (COEF == FE_COEFF_DG0 && s + 2 < ns) c2 = __ldg(cell + (s + 2) * 32);
    const V3 er = xr - xa;
    const double k = kn;
    xr = load_x(a.x4, (int)(w1.x & kStripVertex));
    kn = cell_k<COEF>(a, c1);
    if (!(w.x & kStripLoad)) {
      const V3 gp = cross(eq, er), gq = cross(er, ep), gr = cross(ep, eq);
      const V3 ga = neg_sum(gp, gq, gr);
      const double f = k / fabs(dot(ep, gp));
      const double gg[6] = {f * dot(ga, gp), f * dot(ga, gq), f * dot(ga, gr), 0.0, 0.0, 0.0};
      const uint32_t word[6] = {w.y, w.z, w.w, u.x, u.y, 0u};
      auto slot = [&](int j) { return (word[(j - 1) >> 2] >> (8 * ((j - 1) & 3))) & 0xffu; };
      // a cell's columns differ: reads before writes
      if (!outer) {
        double v[10], o[10];
        p3_row_v(gg, [&](int j, double x) {
          if (j < 10) v[j] = x;
        });
        diag += v[0];
#pragma unroll
        for (int j = 1; j < 10; ++j) o[j] = seg[slot(j)];
#pragma unroll
        for (int j = 1; j < 10; ++j) seg[slot(j)] = o[j] + v[j];
      } else {
        double v[10], o[10];
        p3_row_v(gg, [&](int j, double x) {
          if (j >= 10) v[j - 10] = x;
        });
#pragma unroll
        for (int j = 10; j < 20; ++j) o[j - 10] = seg[slot(j)];
#pragma unroll
        for (int j = 10; j < 20; ++j) seg[slot(j)] = o[j - 10] + v[j - 10];
      }
    }
    if (!(w.x & kStripKeep)) ep = eq;
    eq = er;
  }
  // (the row's own column: added by the inner warp alone)
  if (own.y >= 0 && !outer) seg[own.w] += diag;
  __syncthreads();
  if constexpr (PARTS > 1) {
    for (int t = threadIdx.x; t < 32 * a.stride; t += 64 * PARTS) {
      double v = smem[t];
#pragma unroll
      for (int q = 1; q < PARTS; ++q) v += smem[q * (32 * a.stride) + t];
      smem[t] = v;
    }
    __syncthreads();
  }
  constexpr int kRows = 16 / PARTS;
  store_rows(a, smem, at, own.w, lane, (threadIdx.x >> 5) * kRows, kRows);
}

template <int COEF>
__global__ void __launch_bounds__(32, kMinE3) k_rows_e3(const WalkArgs a) {
  extern __shared__ double smem[];
  let_next_start();
  const int lane = threadIdx.x;
  const int64_t g = blockIdx.x;
  double* seg = smem + lane * a.stride;
  const int4 own = __ldg(a.own + g * 32 + lane);
  const int s0 = __ldg(a.steps + g), ns = __ldg(a.steps + g + 1) - s0;
  const uint4 none = make_uint4(kAll, kAll, 0u, 0u);
  const uint4* rec = a.rec + (int64_t)s0 * 32 + lane;
  const uint4* rec2 = a.rec2 + (int64_t)s0 * 32 + lane;
  const int32_t* cell = a.cell + (int64_t)s0 * 32 + lane;
  uint4 w1 = ns > 0 ? __ldg(rec) : none, w2 = ns > 1 ? __ldg(rec + 32) : none;
  int c1 = COEF == FE_COEFF_DG0 && ns > 0 ? __ldg(cell) : 0, c2 = COEF == FE_COEFF_DG0 && ns > 1 ? __ldg(cell + 32) : 0;
  const RowAt at = row_at(a, own.x);
  V3 xa{0.0, 0.0, 0.0}, e1{0.0, 0.0, 0.0}, ec{0.0, 0.0, 0.0}, xd{0.0, 0.0, 0.0};
  double kn = cell_k<COEF>(a, c1);
  if (own.y >= 0) {
    xa = load_x(a.x4, own.y);
    e1 = load_x(a.x4, own.z) - xa;
  }
  if (w1.y != kAll) xd = load_x(a.x4, (int)w1.y);
  if (a.gaps)
    for (int s = 0; s < a.stride; ++s) seg[s] = 0.0;
  uint4 u1 = ns > 0 ? __ldg(rec2) : make_uint4(0u, 0u, 0u, 0u);
  double mine[4] = {0.0, 0.0, 0.0, 0.0};             // columns a, b and the edge's two nodes
  double run[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // the columns of c so far
  for (int s = 0; s < ns; ++s) {
    const uint4 w = w1;
    w1 = w2;
    c1 = c2;
    w2 = s + 2 < ns ? __ldg(rec + (s + 2) * 32) : none;
    if (COEF == FE_COEFF_DG0 && s + 2 < ns) c2 = __ldg(cell + (s + 2) * 32);
    if (w.y == kAll) continue;
    const uint4 u = u1;
    if (s + 1 < ns) u1 = __ldg(rec2 + (s + 1) * 32);
    if (u.z & kFanBegin) {
      ec = load_x(a.x4, (int)w.x) - xa;
#pragma unroll
      for (int q = 0; q < 6; ++q) run[q] = 0.0;
    }
    const V3 ed = xd - xa;
    const double k = kn;
    if (w1.y != kAll) xd = load_x(a.x4, (int)w1.y);
    kn = cell_k<COEF>(a, c1);
    const V3 gb = cross(ec, ed), gc = cross(ed, e1), gd = cross(e1, ec);
    const V3 ga = neg_sum(gb, gc, gd);
    const double f = k / fabs(dot(e1, gb));
    const double gg[6] = {f * dot(ga, gb), f * dot(ga, gc), f * dot(ga, gd), f * dot(gb, gc), f * dot(gb, gd), 0.0};
    double v[20];
    p3_row_e(gg, [&](int j, double x) { v[j] = x; });
#pragma unroll
    for (int q = 0; q < 4; ++q) mine[q] += v[q];
    const uint32_t cs[6] = {w.z & 0xffu, (w.z >> 8) & 0xffu, (w.z >> 16) & 0xffu,
                            w.z >> 24,   w.w & 0xffu,        (w.w >> 8) & 0xffu};
#pragma unroll
    for (int q = 0; q < 6; ++q) seg[cs[q]] = run[q] + v[4 + q];
#pragma unroll
    for (int q = 0; q < 4; ++q) seg[(u.y >> (8 * q)) & 0xffu] = v[16 + q];
#pragma unroll
    for (int q = 0; q < 6; ++q) run[q] = v[10 + q];
    if (u.z & kFanEnd) {
      const uint32_t ds[6] = {(w.w >> 16) & 0xffu, w.w >> 24,          u.x & 0xffu,
                              (u.x >> 8) & 0xffu,  (u.x >> 16) & 0xffu, u.x >> 24};
      if (u.z & kFanClosed) {
#pragma unroll
        for (int q = 0; q < 6; ++q) run[q] += seg[ds[q]];
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) seg[ds[q]] = run[q];
    }
    ec = ed;
  }
  if (own.y >= 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) seg[((uint32_t)own.w >> (8 * q)) & 0xffu] = mine[q];
  }
  store_rows(a, smem, at, (own.w >> 16) & 0xff, lane, 0, 32);
  end_after_previous();
}

// Face rows: one or two cells, which share the face's ten nodes only.
template <int COEF>
__global__ void __launch_bounds__(32, kMinF3) k_rows_f3(const WalkArgs a) {
  extern __shared__ double smem[];
  let_next_start();
  const int lane = threadIdx.x;
  const int64_t g = blockIdx.x;
  double* seg = smem + lane * a.stride;
  const int4 own = __ldg(a.own + g * 32 + lane);
  const int s0 = __ldg(a.steps + g), ns = __ldg(a.steps + g + 1) - s0;
  const uint4 none = make_uint4(kAll, 0u, 0u, 0u);
  const uint4* rec = a.rec + (int64_t)s0 * 32 + lane;
  const int32_t* cell = a.cell + (int64_t)s0 * 32 + lane;
  uint4 w1 = ns > 0 ? __ldg(rec) : none;
  int c1 = COEF == FE_COEFF_DG0 && ns > 0 ? __ldg(cell) : 0;
  const RowAt at = row_at(a, own.x);
  const int4 slots = __ldg(a.own2 + g * 32 + lane);
  V3 xa{0.0, 0.0, 0.0}, e1{0.0, 0.0, 0.0}, e2{0.0, 0.0, 0.0};
  if (own.y >= 0) {
    xa = load_x(a.x4, own.y);
    e1 = load_x(a.x4, own.z) - xa;
    e2 = load_x(a.x4, own.w) - xa;
  }
  const V3 gd = cross(e1, e2);
  if (a.gaps)
    for (int s = 0; s < a.stride; ++s) seg[s] = 0.0;
  double mine[10];
#pragma unroll
  for (int q = 0; q < 10; ++q) mine[q] = 0.0;
  for (int s = 0; s < ns; ++s) {
    const uint4 w = w1;
    const int c = c1;
    if (s + 1 < ns) {
      w1 = __ldg(rec + (s + 1) * 32);
      if (COEF == FE_COEFF_DG0) c1 = __ldg(cell + (s + 1) * 32);
    }
    if (w.x == kAll) continue;
    const V3 e3 = load_x(a.x4, (int)w.x) - xa;
    const double k = cell_k<COEF>(a, c);
    const V3 gb = cross(e2, e3), gc = cross(e3, e1);
    const V3 ga = neg_sum(gb, gc, gd);
    const double f = k / fabs(dot(e1, gb));
    const double gg[6] = {f * dot(ga, gb), f * dot(ga, gc), f * dot(ga, gd),
                          f * dot(gb, gc), f * dot(gb, gd), f * dot(gc, gd)};
    const uint32_t word[3] = {w.y, w.z, w.w};
    p3_row_f(gg, [&](int j, double x) {
      if (j < 10) mine[j] += x;
      else seg[(word[(j - 10) >> 2] >> (8 * ((j - 10) & 3))) & 0xffu] = x;
    });
  }
  if (own.y >= 0) {
    const uint32_t word[3] = {(uint32_t)slots.x, (uint32_t)slots.y, (uint32_t)slots.z};
#pragma unroll
    for (int q = 0; q < 10; ++q) seg[(word[q >> 2] >> (8 * (q & 3))) & 0xffu] = mine[q];
  }
  store_rows(a, smem, at, (slots.z >> 8) & 0xff, lane, 0, 32);
  end_after_previous();
}

int odd_at_least(int n) { return n | 1; }

size_t segment_bytes(int stride) { return sizeof(double) * 32 * (size_t)stride; }

int degree_of(int kind) {
  switch (kind) {
    case FE_FORM_P1_STIFFNESS: return 1;
    case FE_FORM_P2_STIFFNESS: return 2;
    case FE_FORM_P3_STIFFNESS: return 3;
    default: return 0;
  }
}

template <int COEF>
void raise_p3_of() {
  raise_smem(k_rows_v3<COEF, 1>);
  raise_smem(k_rows_v3<COEF, 2>);
  raise_smem(k_rows_v3<COEF, 4>);
  raise_smem(k_rows_e3<COEF>);
  raise_smem(k_rows_f3<COEF>);
}
void raise_p3() {
  raise_p3_of<FE_COEFF_CONSTANT>();
  raise_p3_of<FE_COEFF_DG0>();
}

// a P1 coefficient's dofmap is the mesh's own vertex numbering (then its
// values can be fetched by mesh vertex); asked once per dofmap
bool vertex_numbered(fe_form_s& f, const fe_dofmap_s& map, cudaStream_t s) {
  fe_form_s::RowsPlan& P = *f.rows_plan;
  if (P.map_id == map.id) return P.map_same;
  if (capturing(s)) return false;
  bool same = map.num_cells == f.mesh->num_cells && map.k == 4 && map.num_blocks >= f.mesh->num_nodes;
  if (same && map.num_cells > 0) {
    DevBuf<unsigned> differ(1);
    FE_CUDA(cudaMemsetAsync(differ.p, 0, sizeof(unsigned), s));
    const int64_t n = map.num_cells * 4;
    k_rows_same_map<<<blocks_for(n, 256), 256, 0, s>>>(map.dofs.p, f.mesh->geom.p, n, differ.p);
    FE_CUDA(cudaGetLastError());
    unsigned h = 0;
    FE_CUDA(cudaMemcpyAsync(&h, differ.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    FE_CUDA(cudaStreamSynchronize(s));
    same = h == 0;
  }
  P.map_id = map.id;
  P.map_same = same;
  return same;
}

void build_part(const PlanArgs& a, PartArgs p, fe_form_s::RowsPlan::Part& part, const int32_t* rows, cudaStream_t s) {
  part.ngroups = p.ngroups;
  part.parts = p.parts;
  part.own.alloc((size_t)p.ngroups * 32);
  if (p.kind == KIND_F) {
    part.own2.alloc((size_t)p.ngroups * 32);
    FE_CUDA(cudaMemsetAsync(part.own2.p, 0, part.own2.bytes(), s));
    p.own2 = part.own2.p;
  }
  part.steps.alloc((size_t)p.ngroups + 1);
  DevBuf<unsigned> gaps(1);
  FE_CUDA(cudaMemsetAsync(gaps.p, 0, sizeof(unsigned), s));
  FE_CUDA(cudaMemsetAsync(part.steps.p, 0, part.steps.bytes(), s));
  p.rows = rows;
  p.own = part.own.p;
  p.steps = part.steps.p;
  p.gaps = gaps.p;
  k_rows_head<<<blocks_for(p.ngroups * 32, 128), 128, 0, s>>>(a, p);
  FE_CUDA(cudaGetLastError());
  exclusive_scan(part.steps.p, p.ngroups + 1, s);
  int32_t total = 0;
  FE_CUDA(cudaMemcpyAsync(&total, part.steps.p + p.ngroups, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  unsigned bad = 0;
  FE_CUDA(cudaMemcpyAsync(&bad, a.fail, sizeof(bad), cudaMemcpyDeviceToHost, s));
  FE_CUDA(cudaStreamSynchronize(s));
  if (bad) return;
  const size_t nrec = (size_t)total * 32;
  // 16-byte records first, each array a multiple of 32 records long
  const size_t one = a.deg == 1 ? sizeof(uint2) : (a.deg == 3 && p.kind != KIND_F ? 2 : 1) * sizeof(uint4);
  part.mem.alloc(std::max<size_t>(1, nrec * (one + sizeof(int32_t))));
  if (a.deg == 1) part.rec1 = reinterpret_cast<uint2*>(part.mem.p);
  else part.rec = reinterpret_cast<uint4*>(part.mem.p);
  if (a.deg == 3 && p.kind != KIND_F) part.rec2 = part.rec + nrec;
  part.cell = reinterpret_cast<int32_t*>(part.mem.p + nrec * one);
  p.rec = part.rec;
  p.rec2 = part.rec2;
  p.rec1 = part.rec1;
  p.cell = part.cell;
  k_rows_records<<<blocks_for(p.ngroups * 32, 128), 128, 0, s>>>(a, p);
  FE_CUDA(cudaGetLastError());
  unsigned g = 0;
  FE_CUDA(cudaMemcpyAsync(&g, gaps.p, sizeof(g), cudaMemcpyDeviceToHost, s));
  FE_CUDA(cudaStreamSynchronize(s));
  part.gaps = g != 0;
}

template <int DEG, int COEF>
void raise_v() {
  raise_smem(k_rows_v<DEG, COEF, 1>);
  raise_smem(k_rows_v<DEG, COEF, 2>);
  raise_smem(k_rows_v<DEG, COEF, 4>);
}
template <int DEG>
void raise_all() {
  raise_v<DEG, FE_COEFF_CONSTANT>();
  raise_v<DEG, FE_COEFF_DG0>();
  raise_v<DEG, FE_COEFF_P1>();
}

}  // namespace

void reset_rows_plan(fe_form_s& f) { f.rows_plan.reset(); }

// Small meshes keep the scatter: a call's time is its launches there and the
// plan would not pay.  On B200, us per call, walk / best scatter: P1 n=20
// (48,000 cells) 8.4 / 9.1, n=32 (196,608) 13.7 / 16.7, n=45 28 / 35; P2 n=16
// (24,576) 16 / 18, n=20 25 / 25, n=28 (131,712) 42 / 64; P3 n=3 27 / 59,
// n=12 29 / 65, n=20 86 / 105.
bool rows_default(const fe_form_s& f) {
  const int64_t cells = f.mesh ? f.mesh->num_cells : 0;
  switch (degree_of(f.kind)) {
    case 1: return cells >= 98304;
    case 2: return cells >= 65536;
    case 3: return true;
    default: return false;
  }
}

// Builds the plan of a form bound to a plain pattern; leaves the form without
// one where the walk does not apply (the assembly then takes the scatter):
// kinds without a row walk, two different spaces, dofs that stand for several
// mesh vertices or edges (periodic maps), cells with a repeated dof, neighbours
// that do not share the dofs of a common face (slits), rows too long for a
// warp's shared memory, no memory for the records.
void build_rows_plan(fe_form_s& f, cudaStream_t s) {
  f.rows_plan.reset();
  const int deg = degree_of(f.kind);
  if (!deg || f.precision != FE_PREC_FP64 || f.V0 != f.V1 || f.V0->excluded || f.sp->parent || f.ffcx) return;
  const fe_dofmap_s& V = *f.V0;
  const fe_mesh_s& mesh = *f.mesh;
  const int64_t C = V.num_cells, nR = V.num_blocks;
  if (C == 0 || nR == 0 || V.k != dofs_of(deg) || C != mesh.num_cells || C * V.k > INT32_MAX || nR >= (1 << 30) ||
      mesh.num_nodes > kStripVertex ||
      capturing(s))
    return;
  try {
    auto P = std::make_unique<fe_form_s::RowsPlan>();
    size_t tb = 0;
    FE_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                            (int32_t*)nullptr, (int)nR, 0, 32, s));
    PlanScratch work(*f.ctx, (tb + 3) / 4 + (size_t)C * V.k + 7 * (size_t)(nR + 1) + 8, s);
    int32_t* next = work.p;
    auto take = [&](size_t n) {
      int32_t* q = next;
      next += n;
      return q;
    };
    void* tmp = take((tb + 3) / 4);
    int32_t* cnt = take(nR + 1);
    unsigned* kmask = reinterpret_cast<unsigned*>(take(nR + 1));
    int* totals = take(6);
    unsigned* fail = reinterpret_cast<unsigned*>(take(1));
    FE_CUDA(cudaMemsetAsync(cnt, 0, (2 * (size_t)(nR + 1) + 7) * sizeof(int32_t), s));
    int32_t* cursor = take(nR + 1);
    int32_t* row = take(nR);
    int32_t* row_sorted = take(nR);
    uint32_t* key = reinterpret_cast<uint32_t*>(take(nR));
    uint32_t* key_sorted = reinterpret_cast<uint32_t*>(take(nR));
    int32_t* inc = take((size_t)C * V.k);
    PlanArgs a{};
    a.num_cells = C;
    a.num_rows = nR;
    a.k = V.k;
    a.deg = deg;
    a.geom = mesh.geom.p;
    a.dofs = V.dofs.p;
    a.pos = f.pos.p;
    a.row_ptr = f.sp->row_ptr.p;
    a.diag = f.sp->diag.p;
    a.inc_ptr = cnt;
    a.inc = inc;
    a.fail = fail;
    k_rows_count<<<blocks_for(C, 128), 128, 0, s>>>(a, cnt, kmask);
    FE_CUDA(cudaGetLastError());
    k_rows_keys<<<blocks_for(nR, 256), 256, 0, s>>>(a, cnt, kmask, key, row, totals);
    FE_CUDA(cudaGetLastError());
    exclusive_scan(cnt, nR + 1, s);
    int h[7];  // rows of each kind, their longest, the mark of a failed plan
    FE_CUDA(cudaMemcpyAsync(h, totals, sizeof(h), cudaMemcpyDeviceToHost, s));
    FE_CUDA(cudaMemcpyAsync(cursor, cnt, (size_t)(nR + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    FE_CUDA(cudaStreamSynchronize(s));
    const int *hk = h, *longest = h + 3;
    if (h[6] || std::max({longest[0], longest[1], longest[2]}) > 256) return;
    // segments as long as the longest row of the kind; at least four warps per
    // SM, or the scatter is the better one
    for (int kind = 0; kind < 3; ++kind) {
      P->part[kind].stride = odd_at_least(longest[kind]);
      if (segment_bytes(P->part[kind].stride) + kSmemCta > kSmemSm / 4) return;
    }
    k_rows_fill<<<blocks_for(C * V.k, 256), 256, 0, s>>>(a, cursor);
    FE_CUDA(cudaGetLastError());
    FE_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, key, key_sorted, row, row_sorted, (int)nR, 0, 32, s));
    int64_t first = 0;
    for (int kind = 0; kind < 3; ++kind) {
      PartArgs p{};
      p.kind = kind;
      p.nrows = hk[kind];
      p.ngroups = (hk[kind] + 31) / 32;
      // few groups: their walks are shared by several warps, which shortens
      // the chain of steps (us per call with 1 / 2 / 4: P1 n=12 15.7 / 9.7 /
      // 6.8, n=32 (1,123 groups) 17.0 / 13.7 / 14.8, n=64 83 / 102 / 139; P2
      // n=16 24 / 17 / 16, n=28 (763 groups) 48 / 42 / 46, n=60 320 / 358 / 415)
      p.parts = 1;
      if (kind == KIND_V) p.parts = p.ngroups <= 2 * f.ctx->num_sms ? 4 : (p.ngroups <= 10 * f.ctx->num_sms ? 2 : 1);
      if (p.nrows == 0) continue;
      build_part(a, p, P->part[kind], row_sorted + first, s);
      first += p.nrows;
    }
    P->x4.alloc((size_t)std::max<int64_t>(1, mesh.num_nodes));
    k_rows_pad_x<<<blocks_for(mesh.num_nodes, 256), 256, 0, s>>>(mesh.x.p, mesh.num_nodes, P->x4.p);
    FE_CUDA(cudaGetLastError());
    unsigned bad = 0;
    FE_CUDA(cudaMemcpyAsync(&bad, fail, sizeof(bad), cudaMemcpyDeviceToHost, s));
    FE_CUDA(cudaStreamSynchronize(s));  // the temporaries are freed on return
    if (bad) return;
    for (auto& part : P->part)
      while (part.parts > 1 && part.parts * segment_bytes(part.stride) + kSmemCta > kSmemSm) part.parts /= 2;
    if (deg == 1) raise_all<1>();
    else if (deg == 2) raise_all<2>();
    else raise_p3();
    if (deg == 2) {
      raise_smem(k_rows_e2<FE_COEFF_CONSTANT>);
      raise_smem(k_rows_e2<FE_COEFF_DG0>);
      raise_smem(k_rows_e2<FE_COEFF_P1>);
    }
    f.rows_plan = std::move(P);
    const Coefficient& k = f.coeff[0];
    if (k.kind == FE_COEFF_P1 && k.map) (void)vertex_numbered(f, *k.map, s);
  } catch (const Error& e) {
    if (e.code != FE_ERR_NOMEM) throw;
    f.rows_plan.reset();
  }
}

bool rows_supported(fe_form_s& f, const fe_bc_s* bc0, const fe_bc_s* bc1, cudaStream_t s) {
  if (!f.rows_plan || f.precision != FE_PREC_FP64 || bc0 != bc1) return false;
  const Coefficient& k = f.coeff[0];
  if (k.kind == FE_COEFF_P1) {
    if (f.kind == FE_FORM_P3_STIFFNESS || !k.map || !vertex_numbered(f, *k.map, s)) return false;
  } else if (k.kind != FE_COEFF_DG0 && k.kind != FE_COEFF_CONSTANT && k.kind >= 0) {
    return false;
  }
  if (bc0 && bc0->row_flags.find(f.sp->id) == bc0->row_flags.end() && capturing(s)) return false;
  return true;
}

namespace {
template <int DEG, int COEF>
void launch_parts(const fe_form_s& f, WalkArgs a, cudaStream_t s) {
  const fe_form_s::RowsPlan& P = *f.rows_plan;
  auto set = [&](const fe_form_s::RowsPlan::Part& p) {
    a.ngroups = p.ngroups;
    a.own = p.own.p;
    a.steps = p.steps.p;
    a.rec = p.rec;
    a.rec2 = p.rec2;
    a.own2 = p.own2.p;
    a.rec1 = p.rec1;
    a.cell = p.cell;
    a.stride = p.stride;
    a.gaps = p.gaps ? 1 : 0;
  };
  const auto& pv = P.part[KIND_V];
  if (pv.ngroups) {
    set(pv);
    const unsigned grid = (unsigned)pv.ngroups;
    const size_t seg = segment_bytes(pv.stride);
    if (pv.parts == 4) k_rows_v<DEG, COEF, 4><<<grid, 128, 4 * seg, s>>>(a);
    else if (pv.parts == 2) k_rows_v<DEG, COEF, 2><<<grid, 64, 2 * seg, s>>>(a);
    else k_rows_v<DEG, COEF, 1><<<grid, 32, seg, s>>>(a);
    FE_CUDA(cudaGetLastError());
  }
  const auto& pe = P.part[KIND_E];
  if (DEG == 2 && pe.ngroups) {
    set(pe);
    launch_beside(k_rows_e2<COEF>, (unsigned)pe.ngroups, segment_bytes(pe.stride), pv.ngroups > 0, a, s);
  }
}

template <int COEF>
void launch_p3(const fe_form_s& f, WalkArgs a, cudaStream_t s) {
  const fe_form_s::RowsPlan& P = *f.rows_plan;
  auto set = [&](const fe_form_s::RowsPlan::Part& p) {
    a.ngroups = p.ngroups;
    a.own = p.own.p;
    a.own2 = p.own2.p;
    a.steps = p.steps.p;
    a.rec = p.rec;
    a.rec2 = p.rec2;
    a.cell = p.cell;
    a.stride = p.stride;
    a.gaps = p.gaps ? 1 : 0;
    return (unsigned)p.ngroups;
  };
  bool beside = false;
  const auto& pv = P.part[KIND_V];
  if (pv.ngroups) {
    const unsigned grid = set(pv);
    const size_t seg = segment_bytes(pv.stride);
    if (pv.parts == 4) k_rows_v3<COEF, 4><<<grid, 256, 4 * seg, s>>>(a);
    else if (pv.parts == 2) k_rows_v3<COEF, 2><<<grid, 128, 2 * seg, s>>>(a);
    else k_rows_v3<COEF, 1><<<grid, 64, seg, s>>>(a);
    FE_CUDA(cudaGetLastError());
    beside = true;
  }
  const auto& pe = P.part[KIND_E];
  if (pe.ngroups) {
    const unsigned grid = set(pe);
    launch_beside(k_rows_e3<COEF>, grid, segment_bytes(pe.stride), beside, a, s);
    beside = true;
  }
  const auto& pf = P.part[KIND_F];
  if (pf.ngroups) {
    const unsigned grid = set(pf);
    launch_beside(k_rows_f3<COEF>, grid, segment_bytes(pf.stride), beside, a, s);
  }
}
}  // namespace

void assemble_matrix_rows(fe_form_s& f, double* values, const fe_bc_s* bc, double diagonal, bool zero,
                          cudaStream_t s) {
  const fe_sparsity_s& sp = *f.sp;
  WalkArgs a{};
  a.x4 = f.rows_plan->x4.p;
  const Coefficient& k = f.coeff[0];
  a.coef = k.values;
  a.coef_const = k.kind < 0 ? 1.0 : k.constant[0];
  a.values = values;
  const bool set_diag = set_bc_rows(a, sp, bc, diagonal, zero, s);
  const int kind = k.kind < 0 ? FE_COEFF_CONSTANT : k.kind;
  if (f.kind == FE_FORM_P3_STIFFNESS) {
    if (kind == FE_COEFF_DG0) launch_p3<FE_COEFF_DG0>(f, a, s);
    else launch_p3<FE_COEFF_CONSTANT>(f, a, s);
  } else if (f.kind == FE_FORM_P1_STIFFNESS) {
    if (kind == FE_COEFF_P1) launch_parts<1, FE_COEFF_P1>(f, a, s);
    else if (kind == FE_COEFF_DG0) launch_parts<1, FE_COEFF_DG0>(f, a, s);
    else launch_parts<1, FE_COEFF_CONSTANT>(f, a, s);
  } else {
    if (kind == FE_COEFF_P1) launch_parts<2, FE_COEFF_P1>(f, a, s);
    else if (kind == FE_COEFF_DG0) launch_parts<2, FE_COEFF_DG0>(f, a, s);
    else launch_parts<2, FE_COEFF_CONSTANT>(f, a, s);
  }
  if (set_diag) launch_set_diagonal(sp, *bc, diagonal, values, s);
}

}  // namespace fe
