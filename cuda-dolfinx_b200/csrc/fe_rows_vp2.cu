// Row walk for vector-P2 elasticity with FP32 element tensors: a warp owns
// three nodes at a time, their nine scalar CSR rows.
//
// As in fe_rows.cu the rows are added up in shared memory and stored once,
// without reductions (460 M of them for 150 M nonzeros at n=44) or a zero
// pass.  A step takes one cell of each of the three nodes: lane 10q + j
// evaluates the 3x3 block of node q (the cell's local node i) and the cell's
// node j, from the nine products C_ij^pq = int_ref d_p phi_i d_q phi_j and the
// 54 geometric weights W^{ab}_pq, a <= b, of the cell (W^{ba} is the
// transpose), and adds it to its own three columns of the segments.  The
// weights are formed for ten steps at once, one cell a lane, and passed
// through shared memory: FP64 geometry in every step took more instructions
// than the blocks themselves (a lane a row, ten nodes a warp: 1,600
// instructions a step, 2,125 us at n=44).
//
// Measured (us per call, this walk / the warp-coalesced scatter): n=44 1,328 /
// 1,510, n=32 575 / 574, n=26 361 / 327, n=20 183 / 167, n=12 68 / 55, n=5 31 /
// 30; so it is the default from 196,608 cells (n=32) on.  FP64 tensors take
// twice the shared memory and are slower at every size (n=44 1,693 / 1,526,
// n=32 704 / 593): they keep the scatter.  Bound by
// shared-memory wavefronts (55-58 % of the pipe: 190 a step, half of them the
// block's nine adds into its columns, whose banks meet) and by latency at ten
// warps an SM, which the segments leave room for; evaluating the next step's
// block beside the adds took more registers than it gained (1,468 us).
//
// Entries are evaluated in their pair's upper form (the lower local node as
// the row) in the term order of the warp-coalesced scatter (k_mat_vp2_coal), so
// that FP32 element tensors round alike.  The node-block diagonals are minus
// the mean of the FP64 row and column sums of the FP32 off-diagonal entries;
// these are linear, so they are taken once a node.
//
// Reference counterpart: assemble_<I>_c_mat (CUDAFormIntegral.cpp:1103-1226)
// with its zero and set_diagonal passes (CUDAAssembler.cpp:38-164).
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>

#include "fe_cell.cuh"
#include "fe_element_code.cuh"
#include "fe_internal.h"
#include "fe_rows.cuh"

namespace fe {
namespace {

constexpr int kNodes = 3;   // nodes of a group: 30 lanes
constexpr int kCtas = 12;   // CTAs per SM to fit in registers
constexpr int kBatch = 10;  // steps whose weights are formed together: 30 lanes

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
struct VPlanArgs {
  int64_t num_cells, num_nodes;
  const int32_t* row_ptr;
  const int32_t* diag;  // slot of (r, r) or -1
  const int32_t* dofs;  // [cells][10]
  const uint8_t* pos;   // [cells][10][10]
  int32_t* inc_ptr;
  int32_t* inc;
  unsigned* fail;
};

__global__ void k_nodes_count(const VPlanArgs a, int32_t* __restrict__ cnt, uint8_t* __restrict__ vertex) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= a.num_cells) return;
  const int32_t* d = a.dofs + c * 10;
  for (int i = 0; i < 10; ++i) {
    const int32_t r = d[i];
    if (r < 0 || r >= a.num_nodes) {
      *a.fail = 1u;
      return;
    }
    for (int j = 0; j < i; ++j)  // a step adds to its ten columns at once: they have to differ
      if (d[j] == r) *a.fail = 1u;
    atomicAdd(cnt + r, 1);
    if (i < 4) vertex[r] = 1;
  }
}

__global__ void k_nodes_fill(const VPlanArgs a, int32_t* __restrict__ cursor) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= a.num_cells * 10) return;
  a.inc[atomicAdd(cursor + a.dofs[t], 1)] = (int32_t)t;
}

// sort key: edge nodes after vertices, window of 1024 nodes, number of cells;
// totals: the vertices, then the longest row of the vertices and of the others
__global__ void k_nodes_keys(const VPlanArgs a, const int32_t* __restrict__ cnt, const uint8_t* __restrict__ vertex,
                             uint32_t* __restrict__ key, int32_t* __restrict__ node, int* __restrict__ totals) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int kind = -1, len = 0;
  if (r < a.num_nodes) {
    kind = vertex[r] ? 0 : 1;
    const int32_t* p = a.row_ptr + 3 * r;
    len = p[1] - p[0];
    if (p[2] - p[1] != len || p[3] - p[2] != len) *a.fail = 1u;
    key[r] = ((uint32_t)kind << 30) | ((uint32_t)(r >> 10) << 8) | (uint32_t)min(cnt[r], 255);
    node[r] = (int32_t)r;
  }
  for (int k = 0; k < 2; ++k) {
    const unsigned here = __ballot_sync(kAll, kind == k);
    if (!here) continue;
    const int most = __reduce_max_sync(kAll, kind == k ? len : 0);
    if ((threadIdx.x & 31) != 0) continue;
    if (k == 0) atomicAdd(totals, __popc(here));
    if (most > totals[1 + k]) atomicMax(totals + 1 + k, most);
  }
}

struct VPartArgs {
  int64_t count, ngroups;
  const int32_t* nodes;
  int4* own;       // [groups*3] see NodesPlan
  int32_t* steps;  // [groups+1]
  uint4* rec;      // [steps*3] cell with the local index in the top four bits, ten slot bytes
};

__global__ void k_nodes_head(const VPlanArgs a, const VPartArgs p) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= p.ngroups * kNodes) return;
  int4 own = make_int4(-1, 0, 0, 0);
  int n = 0;
  if (t < p.count) {
    const int32_t r = p.nodes[t], lo = a.inc_ptr[r];
    n = a.inc_ptr[r + 1] - lo;
    int32_t* inc = a.inc + lo;
    for (int q = 1; q < n; ++q) {
      const int32_t v = inc[q];
      int s = q;
      for (; s > 0 && inc[s - 1] > v; --s) inc[s] = inc[s - 1];
      inc[s] = v;
    }
    own.x = 3 * r;
    own.y = a.row_ptr[3 * r];
    own.z = (a.row_ptr[3 * r + 1] - own.y) << 8;
    if (n > 0) {
      own.z |= a.pos[(int64_t)inc[0] * 10 + inc[0] % 10];
    } else if (own.z) {
      // a node of no cell with slots (a pattern of the caller's own): its own column, in the blocks' order
      const int slot = (a.diag[3 * r] - own.y) / 3;
      for (int q = 0; q < 3; ++q)
        if (a.diag[3 * r + q] < 0 || a.diag[3 * r + q] - a.row_ptr[3 * r + q] != 3 * slot + q || slot > 255) *a.fail = 1u;
      own.z |= slot & 0xff;
    }
  }
  atomicMax(p.steps + t / kNodes, max(n, 1));  // every group has a step, its last one stores the rows
  p.own[t] = own;
}

__global__ void k_nodes_records(const VPlanArgs a, const VPartArgs p) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= p.ngroups * kNodes) return;
  const int64_t g = t / kNodes;
  const int q = (int)(t - g * kNodes);
  const int64_t s0 = p.steps[g];
  const int ns = p.steps[g + 1] - p.steps[g];
  int n = 0;
  const int32_t* inc = nullptr;
  if (t < p.count) {
    const int32_t r = p.nodes[t];
    inc = a.inc + a.inc_ptr[r];
    n = a.inc_ptr[r + 1] - a.inc_ptr[r];
  }
  for (int s = 0; s < ns; ++s) {
    uint4 w = make_uint4(kAll, 0u, 0u, 0u);
    if (s < n) {
      const int32_t e = inc[s];
      const uint8_t* b = a.pos + (int64_t)e * 10;
      w.x = (uint32_t)(e / 10) | ((uint32_t)(e % 10) << 28);
      w.y = b[0] | ((uint32_t)b[1] << 8) | ((uint32_t)b[2] << 16) | ((uint32_t)b[3] << 24);
      w.z = b[4] | ((uint32_t)b[5] << 8) | ((uint32_t)b[6] << 16) | ((uint32_t)b[7] << 24);
      w.w = b[8] | ((uint32_t)b[9] << 8);
    }
    p.rec[(s0 + s) * kNodes + q] = w;
  }
  p.own[t].w = p.steps[g + 1];
}

// ---------------------------------------------------------------------------
// assembly
// ---------------------------------------------------------------------------
struct VWalkArgs : RowOut {
  int64_t ngroups;
  int per_warp;  // groups a warp takes one after the other
  const int4* __restrict__ own;
  const int32_t* __restrict__ steps;
  const uint4* __restrict__ rec;
  const double* __restrict__ x;
  const int32_t* __restrict__ geom;
  CoefDev c0, c1;  // lambda, mu
};

// A cell's weights in shared memory: six blocks' first eight, then the ninths,
// padded to an odd number of 16-byte words (lanes write theirs without bank
// conflicts).  C_ij for i <= j: nine values padded to 48 bytes.
constexpr int kW = 60, kC = 12;
constexpr size_t kSmemRec = 30 * sizeof(uint4), kSmemC = 56 * kC;
constexpr size_t nodes_smem(int stride) {
  return kSmemRec + sizeof(float) * (30 * kW + kSmemC) + sizeof(double) * kNodes * (size_t)stride;
}

// N values from 16-byte aligned shared memory
template <int N>
__device__ __forceinline__ void load_n(const float* __restrict__ p, float (&v)[N]) {
  static_assert(N % 4 == 0);
#pragma unroll
  for (int q = 0; q < N / 4; ++q) *reinterpret_cast<float4*>(v + 4 * q) = reinterpret_cast<const float4*>(p)[q];
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// One entry in the scatter's term order: two partial sums, in one packed
// register.  u: the block's weights but the ninth; SWAP: with the transposed weights.
template <bool SWAP>
__device__ __forceinline__ float vp2_entry(const float* c, const float* u, float u8) {
  unsigned long long v = fma2(pack2(c[0], c[1]), pack2(u[0], u[SWAP ? 3 : 1]), 0ull);
  v = fma2(pack2(c[2], c[3]), pack2(u[SWAP ? 6 : 2], u[SWAP ? 1 : 3]), v);
  v = fma2(pack2(c[4], c[5]), pack2(u[4], u[SWAP ? 7 : 5]), v);
  v = fma2(pack2(c[6], c[7]), pack2(u[SWAP ? 2 : 6], u[SWAP ? 5 : 7]), v);
  float v0, v1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v0), "=f"(v1) : "l"(v));
  return fma(c[8], u8, v0) + v1;
}

// A node's three rows are one range of the value array, and of its segment:
// stored (or added) and the segment cleared for the next node.
__device__ __forceinline__ void store_node(const RowOut& a, double* seg, int lo, int len, int own_slot, int fl,
                                           int lane) {
  const int n = 3 * len;
  if (n == 0) return;  // a node of no cell, the padding of the last group
  double* out = a.values + lo;
  if (fl == 0 && a.zero) {
    // the segment begins at the range's own 16-byte phase
    const int head = (int)((reinterpret_cast<uintptr_t>(out) >> 3) & 1);
    const int pairs = (n - head) >> 1;
    double2* from = reinterpret_cast<double2*>(seg + head);
    double2* to = reinterpret_cast<double2*>(out + head);
    for (int t = lane; t < pairs; t += 32) {
      to[t] = from[t];
      from[t] = make_double2(0.0, 0.0);
    }
    // the entry before the pairs and the one after them
    if (lane == 0 && head && n > 0) {
      out[0] = seg[0];
      seg[0] = 0.0;
    }
    if (lane == 1 && n - head > 2 * pairs) {
      out[n - 1] = seg[n - 1];
      seg[n - 1] = 0.0;
    }
    return;
  }
  for (int t = lane; t < n; t += 32) {
    const int r = (t >= len) + (t >= 2 * len);
    const int f = (fl >> (8 * r)) & 0xff, w = lo + t;
    double v = seg[t];
    if (f && ((f & 1) || ((__ldg(a.mask + (w >> 5)) >> (w & 31)) & 1u)))
      v = (f & 1) && t - r * len == 3 * own_slot + r ? a.diagonal : 0.0;
    if (a.zero) out[t] = v;
    else atomicAdd(out + t, v);
    seg[t] = 0.0;
  }
}

// (150 registers; at the 128 of 16 CTAs per SM it spills: 1,402 against 1,361 us)
__global__ void __launch_bounds__(32, kCtas) k_nodes_vp2(const VWalkArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  let_next_start();
  const int lane = threadIdx.x;
  uint4* srec = reinterpret_cast<uint4*>(smem);
  float* sW = reinterpret_cast<float*>(smem + kSmemRec);
  float* sC = sW + 30 * kW;
  double* acc = reinterpret_cast<double*>(sC + kSmemC);
  const int64_t g0 = (int64_t)blockIdx.x * a.per_warp;
  const int64_t g1 = g0 + a.per_warp < a.ngroups ? g0 + a.per_warp : a.ngroups;
  const bool on = lane < 30;
  const int q = on ? lane / 10 : 2, j = on ? lane - 10 * (lane / 10) : 0;
  const uint4 none = make_uint4(kAll, 0u, 0u, 0u);
  const int phase = (int)(reinterpret_cast<uintptr_t>(a.values) >> 3);
  int64_t g = g0;
  int s = __ldg(a.steps + g0);
  const int s1 = __ldg(a.steps + g1);
  int4 own = __ldg(a.own + g * kNodes + q), next = own;  // of this lane's node
  // records run two batches ahead, vertices one
  uint4 wn = lane < kNodes * (s1 - s) && on ? __ldg(a.rec + (int64_t)s * kNodes + lane) : none;
  for (int t = lane; t < 550; t += 32) {
    // pair t / 10 = (i, j), i <= j, row by row
    int pi = 0, pj = t / 10;
    while (pj >= 10 - pi) pj -= 10 - pi, ++pi;
    pj += pi;
    const int pq = t % 10;
    if (pq < 9) sC[(t / 10) * kC + pq] = (float)kP2GradGrad[(pi * 10 + pj) * 9 + pq];
  }
  for (int t = lane; t < kNodes * a.stride; t += 32) acc[t] = 0.0;
  int4 gn = wn.x != kAll ? load_geom(a.geom, wn.x & 0x0fffffffu) : make_int4(0, 0, 0, 0);
  int fl = 0;
  auto begin_group = [&]() {
    // the node's row flags are needed only when its rows are stored
    fl = 0;
    if (a.flags && own.x >= 0)
      fl = __ldg(a.flags + own.x) | (__ldg(a.flags + own.x + 1) << 8) | (__ldg(a.flags + own.x + 2) << 16);
    if (g + 1 < g1) next = __ldg(a.own + (g + 1) * kNodes + q);
  };
  begin_group();
  double* seg = acc + q * a.stride + ((phase + own.y) & 1);
  double sum[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // 00, 11, 22, 01 + 10, 02 + 20, 12 + 21
  while (s < s1) {
    const int nb = s1 - s < kBatch ? s1 - s : kBatch;
    const uint4 w = wn;
    const int4 gv = gn;
    wn = on && lane < kNodes * (s1 - s - nb) ? __ldg(a.rec + (int64_t)(s + nb) * kNodes + lane) : none;
    if (on) srec[lane] = w;
    if (w.x != kAll) {
      const int64_t c = w.x & 0x0fffffffu;
      const double lam = coef_cell(a.c0, c), mu = coef_cell(a.c1, c);
      CellGeo geo;
      cell_geometry(a.x, gv, geo);
      __align__(16) float W[56];
#pragma unroll
      for (int blk = 0; blk < 6; ++blk) {
        const int ca = blk < 3 ? blk : (blk == 5 ? 1 : 0), cb = blk < 3 ? blk : (blk == 3 ? 1 : 2);
        float u[9];
        elasticity_weights<float>(geo, lam, mu, ca, cb, u);
#pragma unroll
        for (int p = 0; p < 8; ++p) W[8 * blk + p] = u[p];
        W[48 + blk] = u[8];
      }
      W[54] = W[55] = 0.f;
#pragma unroll
      for (int p = 0; p < 14; ++p)
        reinterpret_cast<float4*>(sW + lane * kW)[p] = *reinterpret_cast<float4*>(W + 4 * p);
    }
    if (wn.x != kAll) gn = load_geom(a.geom, wn.x & 0x0fffffffu);
    __syncwarp();
    for (int b = 0; b < nb; ++b) {
      const int e = b * kNodes + q;
      const uint32_t head = srec[e].x;
      const int i = (int)(head >> 28);
      if (on && head != kAll && i != j) {
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        __align__(16) float c[12];
        load_n(sC + (lo * (19 - lo) / 2 + hi) * kC, c);
        __align__(16) float W[56];
        load_n(sW + e * kW, W);
        float m[3][3];
        m[0][0] = vp2_entry<false>(c, W, W[48]);
        m[1][1] = vp2_entry<false>(c, W + 8, W[49]);
        m[2][2] = vp2_entry<false>(c, W + 16, W[50]);
        m[0][1] = vp2_entry<false>(c, W + 24, W[51]);
        m[0][2] = vp2_entry<false>(c, W + 32, W[52]);
        m[1][2] = vp2_entry<false>(c, W + 40, W[53]);
        m[1][0] = vp2_entry<true>(c, W + 24, W[51]);
        m[2][0] = vp2_entry<true>(c, W + 32, W[52]);
        m[2][1] = vp2_entry<true>(c, W + 40, W[53]);
        // the block stands in row (i, a), column (j, b), below the diagonal transposed
        const int slot = reinterpret_cast<const uint8_t*>(srec + e)[4 + j];
        double* to = seg + 3 * slot;
        const int len = own.z >> 8, da = i < j ? len : 1, db = i < j ? 1 : len;
        double v[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
          for (int y = 0; y < 3; ++y) v[x][y] = to[x * da + y * db];
        sum[0] += (double)m[0][0];
        sum[1] += (double)m[1][1];
        sum[2] += (double)m[2][2];
        sum[3] += (double)m[0][1] + (double)m[1][0];
        sum[4] += (double)m[0][2] + (double)m[2][0];
        sum[5] += (double)m[1][2] + (double)m[2][1];
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
          for (int y = 0; y < 3; ++y) to[x * da + y * db] = v[x][y] + (double)m[x][y];
      }
      __syncwarp();  // the next step's lanes may add to the same columns
      if (s + b + 1 < own.w) continue;
      // the group's last step: its node-block diagonals, then its rows
      const int len = own.z >> 8, slot = own.z & 0xff;
#pragma unroll
      for (int p = 0; p < 6; ++p) {
        // ten lanes: 5 + 5, then 0 + 2, 1 + 3, then 0 + 1, and 4
        double t = sum[p];
        t += __shfl_down_sync(kAll, t, 5);
        const double last = __shfl_down_sync(kAll, t, 4);
        t += __shfl_down_sync(kAll, t, 2);
        t += __shfl_down_sync(kAll, t, 1);
        sum[p] = t + last;
      }
      if (on && j == 0) {
        double* to = seg + 3 * slot;
        to[0] -= sum[0];
        to[len + 1] -= sum[1];
        to[2 * len + 2] -= sum[2];
        to[1] -= 0.5 * sum[3];
        to[len] -= 0.5 * sum[3];
        to[2] -= 0.5 * sum[4];
        to[2 * len] -= 0.5 * sum[4];
        to[len + 2] -= 0.5 * sum[5];
        to[2 * len + 1] -= 0.5 * sum[5];
      }
#pragma unroll
      for (int p = 0; p < 6; ++p) sum[p] = 0.0;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kNodes; ++k) {
        const int lo = __shfl_sync(kAll, own.y, 10 * k);
        store_node(a, acc + k * a.stride + ((phase + lo) & 1), lo, __shfl_sync(kAll, len, 10 * k),
                   __shfl_sync(kAll, slot, 10 * k), __shfl_sync(kAll, fl, 10 * k), lane);
      }
      ++g;
      if (g < g1) {
        own = next;
        seg = acc + q * a.stride + ((phase + own.y) & 1);
        begin_group();
      }
      __syncwarp();
    }
    s += nb;
  }
  end_after_previous();
}

void launch_vp2(const fe_form_s& f, VWalkArgs a, cudaStream_t s) {
  const fe_form_s::NodesPlan& P = *f.nodes_plan;
  bool beside = false;
  for (int kind = 0; kind < 2; ++kind) {
    const auto& p = P.part[kind];
    if (!p.ngroups) continue;
    a.ngroups = p.ngroups;
    a.own = p.own.p;
    a.steps = p.steps.p;
    a.rec = p.rec.p;
    a.stride = p.stride;
    // several groups a warp fill its batches of ten steps (n=44: 1,328 us with
    // up to 3 and 10, 1,363 with 2 and 6, 1,357 with 6 and 20), as long as the
    // chip is filled twice (n=20: 183 us; once 210, four times 194)
    a.per_warp = (int)std::max<int64_t>(
        1, std::min<int64_t>(kind ? 10 : 3, p.ngroups / (2 * kCtas * (int64_t)f.ctx->num_sms)));
    launch_beside(k_nodes_vp2, (unsigned)((p.ngroups + a.per_warp - 1) / a.per_warp), nodes_smem(p.stride), beside, a,
                  s);
    beside = true;
  }
}

}  // namespace

void reset_nodes_plan(fe_form_s& f) { f.nodes_plan.reset(); }

bool vp2_rows_default(const fe_form_s& f) {
  return f.kind == FE_FORM_VP2_ELASTICITY && f.precision == FE_PREC_FP32 && f.mesh && f.mesh->num_cells >= 196608;
}

// Builds the plan of an elasticity form bound to a plain pattern, or leaves
// the form without one (two spaces, restricted dofs, cells with a repeated
// dof, a node of no cell whose diagonal is not in the blocks' order, rows too
// long for shared memory, no memory for the records).
void build_nodes_plan(fe_form_s& f, cudaStream_t s) {
  f.nodes_plan.reset();
  if (f.kind != FE_FORM_VP2_ELASTICITY || f.precision != FE_PREC_FP32 || f.V0 != f.V1 || f.V0->excluded ||
      f.sp->parent)
    return;
  const fe_dofmap_s& V = *f.V0;
  const int64_t C = V.num_cells, nN = V.num_blocks;
  if (C == 0 || nN == 0 || V.k != 10 || V.bs != 3 || C != f.mesh->num_cells || C >= (1 << 28) ||
      C * 10 > INT32_MAX || nN >= (1 << 30) || capturing(s))
    return;
  try {
    auto P = std::make_unique<fe_form_s::NodesPlan>();
    size_t tb = 0;
    FE_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                            (int32_t*)nullptr, (int)nN, 0, 31, s));
    PlanScratch work(*f.ctx, (tb + 3) / 4 + (size_t)C * 10 + 7 * (size_t)(nN + 1) + 4, s);
    int32_t* next = work.p;
    auto take = [&](size_t n) {
      int32_t* q = next;
      next += n;
      return q;
    };
    void* tmp = take((tb + 3) / 4);
    int32_t* cnt = take(nN + 1);
    uint8_t* vertex = reinterpret_cast<uint8_t*>(take(nN / 4 + 1));
    int* totals = take(3);
    unsigned* fail = reinterpret_cast<unsigned*>(take(1));
    FE_CUDA(cudaMemsetAsync(cnt, 0, (size_t)(next - cnt) * sizeof(int32_t), s));
    int32_t* cursor = take(nN + 1);
    int32_t* node = take(nN);
    int32_t* sorted = take(nN);
    uint32_t* key = reinterpret_cast<uint32_t*>(take(nN));
    uint32_t* key_sorted = reinterpret_cast<uint32_t*>(take(nN));
    int32_t* inc = take((size_t)C * 10);
    VPlanArgs a{};
    a.num_cells = C;
    a.num_nodes = nN;
    a.row_ptr = f.sp->row_ptr.p;
    a.diag = f.sp->diag.p;
    a.dofs = V.dofs.p;
    a.pos = f.pos.p;
    a.inc_ptr = cnt;
    a.inc = inc;
    a.fail = fail;
    k_nodes_count<<<blocks_for(C, 128), 128, 0, s>>>(a, cnt, vertex);
    FE_CUDA(cudaGetLastError());
    k_nodes_keys<<<blocks_for(nN, 256), 256, 0, s>>>(a, cnt, vertex, key, node, totals);
    FE_CUDA(cudaGetLastError());
    exclusive_scan(cnt, nN + 1, s);
    int h[4];  // the vertices, the longest rows, the mark of a failed plan
    FE_CUDA(cudaMemcpyAsync(h, totals, sizeof(h), cudaMemcpyDeviceToHost, s));
    FE_CUDA(cudaMemcpyAsync(cursor, cnt, (size_t)(nN + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    FE_CUDA(cudaStreamSynchronize(s));
    if (h[3]) return;
    k_nodes_fill<<<blocks_for(C * 10, 256), 256, 0, s>>>(a, cursor);
    FE_CUDA(cudaGetLastError());
    FE_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, key, key_sorted, node, sorted, (int)nN, 0, 31, s));
    for (int kind = 0; kind < 2; ++kind) {
      auto& part = P->part[kind];
      const int64_t first = kind ? h[0] : 0, count = kind ? nN - h[0] : h[0];
      if (!count) continue;
      part.stride = (3 * std::max(h[1 + kind], 3) + 2) & ~1;  // and one for the phase of its range
      // (at least two groups per SM)
      if (nodes_smem(part.stride) + kSmemCta > kSmemSm / 2) return;
      part.ngroups = (count + kNodes - 1) / kNodes;
      part.own.alloc((size_t)part.ngroups * kNodes);
      part.steps.alloc((size_t)part.ngroups + 1);
      FE_CUDA(cudaMemsetAsync(part.steps.p, 0, part.steps.bytes(), s));
      VPartArgs p{};
      p.count = count;
      p.ngroups = part.ngroups;
      p.nodes = sorted + first;
      p.own = part.own.p;
      p.steps = part.steps.p;
      k_nodes_head<<<blocks_for(p.ngroups * kNodes, 128), 128, 0, s>>>(a, p);
      FE_CUDA(cudaGetLastError());
      exclusive_scan(part.steps.p, p.ngroups + 1, s);
      int32_t total = 0;
      FE_CUDA(cudaMemcpyAsync(&total, part.steps.p + p.ngroups, sizeof(total), cudaMemcpyDeviceToHost, s));
      FE_CUDA(cudaStreamSynchronize(s));
      part.rec.alloc(std::max<size_t>(1, (size_t)total * kNodes));
      p.rec = part.rec.p;
      k_nodes_records<<<blocks_for(p.ngroups * kNodes, 128), 128, 0, s>>>(a, p);
      FE_CUDA(cudaGetLastError());
    }
    unsigned bad = 0;
    FE_CUDA(cudaMemcpyAsync(&bad, fail, sizeof(bad), cudaMemcpyDeviceToHost, s));
    FE_CUDA(cudaStreamSynchronize(s));  // the temporaries are freed on return
    if (bad) return;
    raise_smem(k_nodes_vp2);
    f.nodes_plan = std::move(P);
  } catch (const Error& e) {
    if (e.code != FE_ERR_NOMEM) throw;
    f.nodes_plan.reset();
  }
}

bool vp2_rows_supported(const fe_form_s& f, const fe_bc_s* bc0, const fe_bc_s* bc1, cudaStream_t s) {
  if (!f.nodes_plan || f.precision != FE_PREC_FP32 || bc0 != bc1) return false;
  for (int q = 0; q < 2; ++q)
    if (f.coeff[q].kind != FE_COEFF_DG0 && f.coeff[q].kind != FE_COEFF_CONSTANT) return false;
  return !(bc0 && bc0->row_flags.find(f.sp->id) == bc0->row_flags.end() && capturing(s));
}

void assemble_matrix_vp2_rows(fe_form_s& f, double* values, const fe_bc_s* bc, double diagonal, bool zero,
                              cudaStream_t s) {
  VWalkArgs a{};
  a.values = values;
  a.x = f.mesh->x.p;
  a.geom = f.mesh->geom.p;
  a.c0 = to_dev(&f.coeff[0]);
  a.c1 = to_dev(&f.coeff[1]);
  const bool set_diag = set_bc_rows(a, *f.sp, bc, diagonal, zero, s);
  launch_vp2(f, a, s);
  if (set_diag) launch_set_diagonal(*f.sp, *bc, diagonal, values, s);
}

}  // namespace fe
