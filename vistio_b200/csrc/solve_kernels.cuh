// sm_100a kernels of the global solve A d = r (3 right-hand sides).
//
// A is factored over the supernodes of a merged elimination tree (setup.cpp):
// with F the Schur-complemented block of supernode k (columns K, rows R below
// them), the solve needs two dense matrices of it, N = F_KK^-1 (s x s) and
// W = F_RK N (m x s):
//   forward   r'_K = r_K - (its children's u at K);
//             u_R = W r'_K + (its children's u at R),
//             z_K = N r'_K                         (children before parents)
//   backward  x_K = z_K - W^T x_R                  (parents before children).
// Every step is a dense matrix times a short vector, so a level of the tree is
// one dependent phase. What bounds a solve depends on the batch: a few garments
// are bound by the chain of dependent phases (each a signal or a launch, a
// round trip through L2 for the vector, 32 fused multiply-adds, a store), large
// batches by reading N and W once and W a second time from HBM.
//
// Tasks. Both directions are out[row] = sum over columns c of M(row, c) v(c).
// A task is 32 rows (a tile, one per lane) times 32 columns (a chunk). M is
// stored tile by tile, column by column inside a tile, so that a task is one
// contiguous run of at most 4 KB: one bulk copy into the warp's stage in shared
// memory, issued ahead of everything that has to be waited for. The factor's
// latency then overlaps the dependency wait and the gather of v, no registers
// are held for values in flight (a version that loaded them into registers
// spilled and was 10-50% slower), and what is in flight is 4 KB per resident
// warp. A chunk's sum is one chain of fused multiply-adds from zero in ascending
// column order, and a row's chunks are added in ascending order. Neither depends
// on who runs the task, so every schedule gives the same bits:
//   warp items   a supernode of at most 64 columns, run by one warp;
//   block items  some tiles of one supernode, their tasks shared by the warps.
// W is stored twice (tiles of its rows for the forward product, of its columns
// for the backward one): the same bytes are read either way.
//
// Against inv(L_kk) and L_Rk over a tree of 9 to 11 levels, swept by one
// persistent dependency-driven launch (time of whole plain steps of 10 solves,
// B200): sheet 20x20 721 -> 306 us with the state read back, 97x97 with a
// refinement 3958 -> 946 us for two steps, 24 sheets of sides 17 to 151
// 3.80 -> 1.52 ms, 512 sheets of sides 23 to 121 15.29 -> 12.15 ms. By phase the last
// reads 2.6 to 4.9 TB/s (2.62 GB in 711 us), the small phases at the top less.
#pragma once
#include "pd_kernels.cuh"

namespace vistio {

// The compiled forms of k_level: warps per block and blocks per SM. Untuned
// batches of at most kWideMaxInstances garments use the sixteen-warp form (their
// solves follow one tree's chain), others the eight-warp form.
constexpr uint32_t kWideMaxInstances = 8;
constexpr uint32_t kForms = 3;
constexpr uint32_t kFormWarps[kForms] = {6, 8, 16};
constexpr uint32_t kFormBlocks[kForms] = {5, 4, 2};
constexpr uint32_t kTile = 32;      // rows of a tile and columns of a chunk
constexpr uint32_t kWarpCols = 64;  // columns of a supernode that one warp may take
constexpr uint32_t kMaxTasks = 32;  // tasks of an item whose chunks are shared
// Columns of v staged at a time: what the blocks per SM leave room for. The
// sixteen-warp form takes a supernode of up to 1024 in one piece, so that the
// chunks of its tiles can be shared (97x97 sheet, root of 578 columns: 486 us
// per step with 512, the root's tiles one warp each).
__host__ __device__ constexpr uint32_t vec_cols(uint32_t warps) { return warps == 16 ? 1024 : 512; }
static_assert(vec_cols(6) >= 6 * kWarpCols && vec_cols(8) >= 8 * kWarpCols && vec_cols(16) >= 16 * kWarpCols,
              "the warps' own entries of v fit the block's");
__host__ __device__ constexpr uint32_t level_smem(uint32_t warps) {
  return warps * kTile * kTile * 4 + vec_cols(warps) * 16 + kMaxTasks * kTile * 12;
}
// Default limit of s (s + m) for a warp item; vistio_batch_tune picks one per batch.
constexpr uint32_t kWarpItemLimit = 6144;
__host__ __device__ constexpr bool warp_item(uint32_t s, uint32_t m, uint32_t limit = kWarpItemLimit) {
  return s <= kWarpCols && uint64_t(s) * (s + m) <= limit;
}

// One work item: some tiles of one supernode's product in one direction. All a
// block needs to start its loads, in one read.
struct __align__(16) SweepItem {
  uint64_t mat;        // the direction's panel (float offset in vals)
  uint32_t row0;       // global row (vbase + first) of the supernode's first column
  uint32_t vbase;      // first row of the instance
  uint32_t ncols;      // s
  uint32_t nrows;      // m
  uint32_t rows_off;   // the supernode's rows in rows, and its slots in U
  uint32_t inst;       // owning instance
  uint32_t tile0, ntiles;
  uint32_t pull0;      // the supernode's first pull list (its columns', then its rows')
  uint32_t pulls;      // whether it has children (else every pull list is empty)
};
static_assert(sizeof(SweepItem) == 48, "three 16-byte loads");

// ------------------------------------------------ bulk staging
// A contiguous global range is brought into shared memory with one
// cp.async.bulk whose completion is tracked by an mbarrier transaction count.
// Waits are bounded: after kWaitLimit polls the warp records the timeout status
// bit and goes on.
constexpr uint32_t kWaitLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = kWaitLimit) {
  const uint32_t b = smem_u32(bar);
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(b), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Diagnostic of the failure path: the sweeps' bounded wait on a barrier that
// nothing completes gives up after `polls` polls and records the timeout
// status bit, as a sweep whose staging copy never lands does.
__global__ void k_diag_wait(uint32_t* status, uint32_t polls) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) mbar_init(&bar);
  mbar_fence_init();
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, polls)) atomicOr(status, 4u);
}

// A warp's stage: one task's values in flight or in use at a time.
struct Stage {
  float* buf;      // kTile * kTile floats, 16-byte aligned
  uint64_t* bar;
  uint32_t parity; // phase of the next completion
  // One lane issues the copy once the warp is done with the last task's values;
  // the others reconverge with it before they poll (a warp whose other lanes
  // spin while the issuing lane sits on the other side of a branch was seen to
  // run the spinning side until its poll budget ran out). The values are marked
  // to leave L2 first: a batch's factor is larger than L2, and the lists and
  // vectors every block waits for stay in it (512 sheets 13.67 -> 13.40 ms per
  // step, 24 sheets 1.88 -> 1.83; single garments, whose factor fits, the same).
  __device__ __forceinline__ void issue(const float* src, uint32_t floats) const {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(floats * 4)
                   : "memory");
      asm volatile(
          "{\n .reg .b64 pol;\n createpolicy.fractional.L2::evict_first.b64 pol, 1.0;\n"
          " cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], pol;\n}\n" ::"r"(
              smem_u32(buf)),
          "l"(src), "r"(floats * 4), "r"(smem_u32(bar))
          : "memory");
    }
    __syncwarp();
  }
  __device__ __forceinline__ void wait(uint32_t* status) {
    if (!mbar_wait(bar, parity)) atomicOr(status, 4u);
    parity ^= 1u;
  }
  // The lane's row of the task's product: w rows, nc columns.
  __device__ __forceinline__ float4 sum(const float4* v, uint32_t w, uint32_t nc) const {
    const float* p = buf + min(threadIdx.x & 31, w - 1);
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (uint32_t c = 0; c < nc; ++c) {
      const float a = p[c * w];
      const float4 y = v[c];
      t.x = __fmaf_rn(a, y.x, t.x); t.y = __fmaf_rn(a, y.y, t.y); t.z = __fmaf_rn(a, y.z, t.z);
    }
    return t;
  }
};

// The matrix of an item, in tiles of 32 rows (the last one's rows padded to 8).
template <int DIR> struct Panel {
  const float* m;
  uint32_t rows, cols;
  __device__ __forceinline__ Panel(const BatchDev& B, const SweepItem& I)
      : m(B.vals + I.mat),
        rows(DIR == 0 ? I.nrows + I.ncols : I.ncols),
        cols(DIR == 0 ? I.ncols : I.nrows) {}
  __device__ __forceinline__ uint32_t width(uint32_t t) const { return min(kTile, (rows - t * kTile + 7u) & ~7u); }
  __device__ __forceinline__ uint32_t chunk(uint32_t ch) const { return min(kTile, cols - ch * kTile); }
  // starts the copy of task (t, ch)
  __device__ __forceinline__ void issue(const Stage& st, uint32_t t, uint32_t ch) const {
    const uint32_t w = width(t);
    st.issue(m + size_t(t) * kTile * cols + ch * kTile * w, chunk(ch) * w);
  }
};

// The children's updates at one of a supernode's columns or rows. The list is
// read by prepare(), ahead of the wait; sum() reads the updates, in list order.
// The sixteen-warp form reads four entries ahead (a single garment's sweep waits
// for the rest of the list in every phase: 97x97 329 us per step, 334 with two,
// 348 with one), the others two: four spill there (512 sheets 12.05 ms per step,
// 11.91 with two, 24 sheets 1447 and 1429 us).
// A warp item of a leaf reads no list (its lists are empty; 512 sheets 12.36 ->
// 12.05 ms per step, 24 sheets 1493 -> 1448 us). Block items always do: few are
// leaves, and the test cost single garments, which those bound, 1%.
__host__ __device__ constexpr uint32_t list_ahead(uint32_t warps) { return warps == 16 ? 4 : 2; }
template <uint32_t NP> struct Pull {
  uint32_t q, qe, slot[NP];
  __device__ __forceinline__ void prepare(const BatchDev& B, uint32_t list) {
    q = __ldg(B.pull_ptr + list);
    qe = __ldg(B.pull_ptr + list + 1);
#pragma unroll
    for (uint32_t i = 0; i < NP; ++i) slot[i] = q + i < qe ? __ldg(B.pull + q + i) : 0u;
  }
  __device__ __forceinline__ float4 sum(const BatchDev& B) const {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (uint32_t i = 0; i < NP; ++i)
      if (q + i < qe) t = f4_add(t, B.U[slot[i]]);
#pragma unroll 4
    for (uint32_t e = q + NP; e < qe; ++e) t = f4_add(t, B.U[__ldg(B.pull + e)]);
    return t;
  }
};

// One entry of v: what does not depend on other supernodes is read by prepare(),
// ahead of the wait, the rest by get().
template <int DIR, uint32_t NP, bool LEAVES> struct Entry {
  uint32_t row;
  Pull<NP> p;
  __device__ __forceinline__ void prepare(const BatchDev& B, const SweepItem& I, uint32_t c) {
    if (DIR == 0) {
      row = I.row0 + c;
      p.q = p.qe = 0u;
      if (!LEAVES || I.pulls) p.prepare(B, I.pull0 + c);
    } else {
      row = I.vbase + __ldg(B.rows + I.rows_off + c);
    }
  }
  __device__ __forceinline__ float4 get(const BatchDev& B) const {
    return DIR == 1 ? B.Y[row] : f4_sub(B.T[row], p.sum(B));
  }
};

// One row of the product: begin() ahead of the wait, after() reads what the
// result is combined with, put() writes it.
template <int DIR, uint32_t NP, bool LEAVES> struct OutRow {
  uint32_t row;
  Pull<NP> p;
  float4 with;
  __device__ __forceinline__ bool pulls(const SweepItem& I) const { return DIR == 0 && (!LEAVES || I.pulls) && row < I.nrows; }
  __device__ __forceinline__ void begin(const BatchDev& B, const SweepItem& I, uint32_t r) {
    row = r;
    if (LEAVES) with = make_float4(0.f, 0.f, 0.f, 0.f);
    if (pulls(I)) p.prepare(B, I.pull0 + I.ncols + row);
  }
  __device__ __forceinline__ void after(const BatchDev& B, const SweepItem& I) {
    if (DIR == 1) {
      if (row < I.ncols) with = B.Y[I.row0 + row];
    } else if (pulls(I)) {
      with = p.sum(B);
    }
  }
  __device__ __forceinline__ void put(const BatchDev& B, const SweepItem& I, float4 t) const {
    if (DIR == 1) {
      if (row < I.ncols) B.Y[I.row0 + row] = f4_sub(with, t);
    } else if (row < I.nrows) {
      B.U[I.rows_off + row] = f4_add(t, with);
    } else if (row < I.nrows + I.ncols) {
      B.Y[I.row0 + row - I.nrows] = t;
    }
  }
};

// One item by the whole block. wait() orders the inputs and returns whether the
// garment still takes part. An item of many tiles gives each warp whole tiles,
// whose chunks it adds as they arrive; an item of few (small phases, as long as
// their longest warp) shares the chunks of a tile among the warps and adds their
// sums at the end.
template <int DIR, uint32_t NW, class Wait>
__device__ __forceinline__ void block_item(const BatchDev& B, const SweepItem& I, Stage& st, float4* v, float* part,
                                           Wait wait) {
  const Panel<DIR> M(B, I);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = I.ntiles;
  constexpr uint32_t kVecCols = vec_cols(NW);
  const uint32_t all = (M.cols + kTile - 1) / kTile;
  const bool split = M.cols <= kVecCols && nt * 2 <= NW && all * nt <= kMaxTasks;
  // this warp's first task and its step (split: by chunk, else by tile)
  uint32_t t = split ? 0 : warp, ch = split ? warp : 0;
  auto wrap = [&]() {
    while (ch >= all) { ch -= all; ++t; }
  };
  wrap();
  if (t < nt) M.issue(st, I.tile0 + t, ch);
  OutRow<DIR, list_ahead(NW), false> out;
  if (warp < nt) out.begin(B, I, (I.tile0 + warp) * kTile + lane);
  float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t c0 = 0; c0 < M.cols; c0 += kVecCols) {
    const uint32_t nc = min(kVecCols, M.cols - c0);
    Entry<DIR, list_ahead(NW), false> e;
    if (tid < nc) e.prepare(B, I, c0 + tid);
    if (c0 == 0) {
      if (!wait()) {
        if (t < nt) st.wait(B.status);  // the copy in flight lands before the block ends
        return;
      }
      if (warp < nt) out.after(B, I);
    } else {
      __syncthreads();  // the last segment's readers of v are done
    }
    for (uint32_t c = tid; c < nc; c += 32 * NW) {
      if (c != tid) e.prepare(B, I, c0 + c);
      v[c] = e.get(B);
    }
    __syncthreads();
    if (split) {
      while (t < nt) {
        st.wait(B.status);
        const float4 p = st.sum(v + ch * kTile, M.width(I.tile0 + t), M.chunk(ch));
        float* q = part + (t * all + ch) * kTile * 3 + lane;
        q[0] = p.x; q[kTile] = p.y; q[2 * kTile] = p.z;
        ch += NW;
        wrap();
        if (t < nt) M.issue(st, I.tile0 + t, ch);
      }
      __syncthreads();
      if (warp < nt)
        for (uint32_t k = 0; k < all; ++k) {
          const float* q = part + (warp * all + k) * kTile * 3 + lane;
          const float4 p = make_float4(q[0], q[kTile], q[2 * kTile], 0.f);
          total = k == 0 ? p : f4_add(total, p);
        }
    } else {
      // (an item has more tiles than warps only with one segment of columns)
      const uint32_t last = min(all, (c0 + kVecCols) / kTile);
      while (t < nt) {
        st.wait(B.status);
        const float4 p = st.sum(v + ch * kTile - c0, M.width(I.tile0 + t), M.chunk(ch));
        total = ch == 0 ? p : f4_add(total, p);
        const bool row_done = ++ch == all;
        if (row_done) {
          if (t + NW < nt) {
            out.put(B, I, total);
            M.issue(st, I.tile0 + t + NW, 0);
            out.begin(B, I, (I.tile0 + t + NW) * kTile + lane);
            out.after(B, I);
          }
          t += NW;
          ch = 0;
        } else {
          M.issue(st, I.tile0 + t, ch);
          if (ch == last) break;  // the rest of the row with the next segment
        }
      }
    }
  }
  if (warp < nt) out.put(B, I, total);
}

// One item of a supernode of at most kWarpCols columns by one warp: forward some
// of its tiles, over its one or two chunks; backward one tile. v: kWarpCols
// entries of the warp's own (backward a chunk at a time).
template <int DIR, uint32_t NW, class Wait>
__device__ __forceinline__ void warp_tiles(const BatchDev& B, const SweepItem& I, Stage& st, float4* v, Wait wait) {
  const Panel<DIR> M(B, I);
  const uint32_t lane = threadIdx.x & 31, all = (M.cols + kTile - 1) / kTile;
  M.issue(st, I.tile0, 0);
  OutRow<DIR, list_ahead(NW), true> out;
  float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t t = 0; t < I.ntiles; ++t) {
    out.begin(B, I, (I.tile0 + t) * kTile + lane);
    for (uint32_t ch = 0; ch < all; ++ch) {
      const uint32_t nc = M.chunk(ch);
      float4* vc = DIR == 0 ? v + ch * kTile : v;
      if (t == 0) {
        Entry<DIR, list_ahead(NW), true> e;
        if (lane < nc) e.prepare(B, I, ch * kTile + lane);
        if (ch == 0 && !wait()) {
          st.wait(B.status);  // the copy in flight lands before the block ends
          return;
        }
        if (DIR == 1) __syncwarp();  // the last chunk's readers of v are done
        if (lane < nc) vc[lane] = e.get(B);
        __syncwarp();
      }
      if (ch == 0) out.after(B, I);
      st.wait(B.status);
      const float4 p = st.sum(vc, M.width(I.tile0 + t), nc);
      total = ch == 0 ? p : f4_add(total, p);
      if (ch + 1 < all) M.issue(st, I.tile0 + t, ch + 1);
      else if (t + 1 < I.ntiles) M.issue(st, I.tile0 + t + 1, 0);
    }
    out.put(B, I, total);
  }
}

// One phase of the forward (DIR = 0) or backward (DIR = 1) sweep over every
// instance of the batch: blocks [0, nblock) take one block item each, the rest
// one warp item per warp. The supernodes of a phase are independent; phases are
// ordered by kernel boundaries, and everything up to the wait for the previous
// kernel (griddepcontrol.wait) overlaps it.
template <int DIR, uint32_t FORM>
__global__ void __launch_bounds__(32 * kFormWarps[FORM], kFormBlocks[FORM])
k_level(BatchDev B, const SweepItem* __restrict__ items, uint32_t nblock, uint32_t nwarp) {
  constexpr uint32_t NW = kFormWarps[FORM];
  extern __shared__ float4 level_sm[];
  __shared__ uint64_t bar[NW];
  float* stages = reinterpret_cast<float*>(level_sm);
  float4* v = level_sm + NW * kTile * kTile / 4;
  float* part = reinterpret_cast<float*>(v + vec_cols(NW));
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) mbar_init(&bar[warp]);
  mbar_fence_init();
  __syncwarp();
  Stage st{stages + warp * kTile * kTile, &bar[warp], 0u};
  if (blockIdx.x < nblock) {
    const SweepItem I = items[blockIdx.x];
    block_item<DIR, NW>(B, I, st, v, part, [&]() {
      pdl_begin();
      return !(B.prm->ipc && B.red[I.inst].al_done);
    });
    return;
  }
  const uint32_t q = (blockIdx.x - nblock) * NW + warp;
  if (q >= nwarp) {
    pdl_begin();
    return;
  }
  const SweepItem I = items[nblock + q];
  warp_tiles<DIR, NW>(B, I, st, v + warp * kWarpCols, [&]() {
    pdl_begin();
    return !(B.prm->ipc && B.red[I.inst].al_done);
  });
}

}  // namespace vistio
