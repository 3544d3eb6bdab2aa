// Shared by the row-walk kernels (fe_rows.cu, fe_rows_vp2.cu): a warp's rows to
// the value array, what a BC does to them, launches side by side.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cub/cub.cuh>
#include <memory>

#include "fe_internal.h"

namespace fe {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr size_t kSmemSm = 227 * 1024;  // shared memory one SM gives to its CTAs
constexpr size_t kSmemCta = 1024;       // the part the system takes of each CTA's share

// where a call's rows go
struct RowOut {
  const int32_t* __restrict__ row_ptr;
  const uint8_t* __restrict__ flags;  // BC flags of the rows, or null
  const uint32_t* __restrict__ mask;  // bit s: the column of slot s is a BC column
  double diagonal;   // stored on BC rows (with zero)
  int zero;
  double* __restrict__ values;
  int stride;     // doubles between the segments of a warp's rows (odd)
};

// a lane's row in the value array, fetched before the walk
struct RowAt {
  int lo = 0, len = 0, fl = 0;
};
__device__ __forceinline__ RowAt row_at(const RowOut& a, int row) {
  RowAt r;
  if (row >= 0) {
    r.lo = __ldg(a.row_ptr + row);
    r.len = __ldg(a.row_ptr + row + 1) - r.lo;
    if (a.flags) r.fl = __ldg(a.flags + row);
  }
  return r;
}

// The warp's 32 row segments (lane l's at acc + l * stride) to their rows.
// First the segments of rows that a BC touches take their zeros (and a BC row
// `diagonal` at its own slot, -1: it has none), then all rows are stored, or added
// with zero == 0 (by reductions, as the scatter's: another call may add to the
// same matrix on another stream).
// A warp takes the `count` rows from `first` on.
__device__ __forceinline__ void store_rows(const RowOut& a, double* acc, const RowAt& at, int own_slot, int lane,
                                           int first, int count) {
  const unsigned mine = count == 32 ? kAll : ((1u << count) - 1u) << first;
  __syncwarp();
  // about every second warp has such rows, a few of them: four at a time, so
  // that their mask words are fetched together
  for (unsigned todo = __ballot_sync(kAll, at.fl != 0) & mine; todo;) {
    int rr[4], rlo[4], rlen[4], rfl[4], rown[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      rr[q] = todo ? __ffs(todo) - 1 : 0;
      rlo[q] = __shfl_sync(kAll, at.lo, rr[q]);
      const int len = __shfl_sync(kAll, at.len, rr[q]);
      rlen[q] = todo ? len : 0;
      rfl[q] = __shfl_sync(kAll, at.fl, rr[q]);
      rown[q] = __shfl_sync(kAll, own_slot, rr[q]);
      todo &= todo - 1;
    }
    const int most = max(max(rlen[0], rlen[1]), max(rlen[2], rlen[3]));
    for (int s = lane; s < most; s += 32) {
      uint32_t m[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int w = rlo[q] + s;
        m[q] = s < rlen[q] ? ((rfl[q] & 1) ? 1u : (__ldg(a.mask + (w >> 5)) >> (w & 31)) & 1u) : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (m[q]) acc[rr[q] * a.stride + s] = (rfl[q] & 1) && s == rown[q] ? a.diagonal : 0.0;
    }
  }
  __syncwarp();
  const int len0 = __shfl_sync(kAll, at.len, first);
  if (a.zero && len0 > 0 && __all_sync(kAll, at.len == len0 || !((mine >> lane) & 1u))) {
    // rows of one length: the lanes go through their entries without a gap
    const int jump = 32 / len0, rest = 32 - jump * len0, end = (first + count) * len0, pad = a.stride - len0;
    // entry t of the group stands at value index t + delta of its row
    const int delta = at.lo - lane * len0;
    int rr = lane / len0, s = lane - rr * len0;
    rr += first;
    const double* from = acc + first * len0 + lane;
#pragma unroll 4
    for (int t = first * len0 + lane; t < end + lane; t += 32, from += 32) {
      const int to = t + __shfl_sync(kAll, delta, rr);
      if (t < end) a.values[to] = from[rr * pad];
      s += rest;
      const bool wrap = s >= len0;
      if (wrap) s -= len0;
      rr += wrap ? jump + 1 : jump;
    }
    return;
  }
#pragma unroll 4
  for (int rr = first; rr < first + count; ++rr) {
    const int rlo = __shfl_sync(kAll, at.lo, rr), rlen = __shfl_sync(kAll, at.len, rr);
    const double* seg = acc + rr * a.stride;
    for (int s = lane; s < rlen; s += 32) {
      const double v = seg[s];
      if (a.zero) a.values[rlo + s] = v;
      else atomicAdd(a.values + rlo + s, v);
    }
  }
}

// The kernels of one call write different rows: the later one starts while
// the earlier one runs (programmatic dependent launch) and ends after it, so
// that what follows in the stream waits for both.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void end_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// bit s of the mask: the column of slot s is a BC column
__global__ void k_rows_bc_mask(const int32_t* __restrict__ col, int64_t nnz, const uint8_t* __restrict__ markers,
                               uint32_t* __restrict__ mask) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const unsigned b = __ballot_sync(kAll, q < nnz && markers[col[q]] != 0);
  if ((threadIdx.x & 31) == 0 && q < nnz) mask[q >> 5] = b;
}
// bit 0: a BC row; bit 1: a row with a BC column
__global__ void k_rows_bc_flags(const int32_t* __restrict__ row_ptr, int64_t num_rows,
                                const uint8_t* __restrict__ markers, const uint32_t* __restrict__ mask,
                                uint8_t* __restrict__ flags) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= num_rows) return;
  const int32_t lo = row_ptr[r], hi = row_ptr[r + 1];
  uint32_t any = 0u;
  for (int32_t w = lo >> 5; w <= (hi - 1) >> 5 && lo < hi; ++w) {
    uint32_t m = mask[w];
    if (w == lo >> 5) m &= kAll << (lo & 31);
    if (w == (hi - 1) >> 5) m &= kAll >> (31 - ((hi - 1) & 31));
    any |= m;
  }
  flags[r] = (uint8_t)((markers[r] ? 1 : 0) | (any ? 2 : 0));
}

unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

template <typename K>
void raise_smem(K kernel) {
  FE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemSm));
}

// The temporaries of a plan in one allocation: small ones from the context's
// scratch pool, which keeps them for the next solve or plan (an allocation of
// some MB takes 0.3 ms, and as long to give back), large ones on their own.
struct PlanScratch {
  static constexpr size_t kPooled = size_t(32) << 20;
  int32_t* p = nullptr;
  cudaStream_t s;
  bool pooled;
  PlanScratch(fe_context_s& ctx, size_t words, cudaStream_t st) : s(st), pooled(words * 4 <= kPooled) {
    cudaMemPool_t pool = pooled ? scratch_pool(ctx) : nullptr;
    const cudaError_t e = pooled ? cudaMallocFromPoolAsync((void**)&p, words * 4, pool, s) : cudaMalloc((void**)&p, words * 4);
    if (e != cudaSuccess) {
      p = nullptr;
      (void)cudaGetLastError();
      throw Error(FE_ERR_NOMEM, std::string("no memory for a plan's temporaries: ") + cudaGetErrorString(e));
    }
  }
  PlanScratch(const PlanScratch&) = delete;
  PlanScratch& operator=(const PlanScratch&) = delete;
  ~PlanScratch() {
    if (p) (void)(pooled ? cudaFreeAsync(p, s) : cudaFree(p));
  }
};

void exclusive_scan(int32_t* v, int64_t n, cudaStream_t s) {
  size_t tb = 0;
  FE_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, v, v, (int)n, s));
  DevBuf<unsigned char> tmp(std::max<size_t>(1, tb));
  FE_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, v, v, (int)n, s));
  FE_CUDA(cudaStreamSynchronize(s));
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  FE_CUDA(cudaStreamIsCapturing(s, &st));
  return st != cudaStreamCaptureStatusNone;
}

// `beside`: the kernel before it in the stream is one of this call's
template <typename K, typename Args>
void launch_beside(K kernel, unsigned grid, size_t smem, bool beside, const Args& a, cudaStream_t s) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(32);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = beside ? 1 : 0;
  FE_CUDA(cudaLaunchKernelEx(&c, kernel, a));
}

// Fills the BC part of `out` (which rows a BC touches is collected once per
// pattern and BC, as the diagonal slots of the zero pass) and says whether
// set_diagonal has to follow.
bool set_bc_rows(RowOut& out, const fe_sparsity_s& sp, const fe_bc_s* bc, double diagonal, bool zero, cudaStream_t s) {
  out.row_ptr = sp.row_ptr.p;
  out.zero = zero ? 1 : 0;
  if (!bc) return false;
  auto& F = bc->row_flags[sp.id];
  if (!F) {
    auto t = std::make_unique<fe_bc_s::RowFlags>();
    t->flags.alloc((size_t)std::max<int64_t>(1, sp.num_rows));
    t->mask.alloc((size_t)(sp.nnz / 32 + 1));
    if (sp.nnz) k_rows_bc_mask<<<blocks_for(sp.nnz, 256), 256, 0, s>>>(sp.col.p, sp.nnz, bc->markers.p, t->mask.p);
    k_rows_bc_flags<<<blocks_for(sp.num_rows, 256), 256, 0, s>>>(sp.row_ptr.p, sp.num_rows, bc->markers.p, t->mask.p,
                                                                 t->flags.p);
    FE_CUDA(cudaGetLastError());
    FE_CUDA(cudaStreamSynchronize(s));  // calls on other streams may read them next
    F = std::move(t);
  }
  out.flags = F->flags.p;
  out.mask = F->mask.p;
  // the marked rows are the owned listed ones: their diagonal goes with the rows
  const bool owned = bc->markers_are_dofs && bc->n_owned == bc->n_bc;
  out.diagonal = owned && zero ? diagonal : 0.0;
  return !owned || !zero;
}

}  // namespace
}  // namespace fe
