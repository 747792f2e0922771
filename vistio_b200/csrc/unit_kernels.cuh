// Sweeps of the global solve by units: connected parts of the supernodal trees
// that one block sweeps level by level out of shared memory.
//
// A solve over one or a few garments is a chain of dependent supernodes, bound by
// the latency of each link. In k_sweep a link is a signal through L2, a staging
// copy, and lists and values gathered one after another. Here a block holds all
// supernodes of a unit at once: their factor values, tables and vector entries are
// brought to shared memory together, the static ones ahead of the wait for the
// kernel before, and a level is one to three barriers. Units that depend on one
// another are phases, one launch each; a unit that holds its tree's root sweeps
// both ways. Against k_sweep (device time of a plain step of 10 iterations, B200):
// sheet 20x20 568 -> 328 us, 97x97 with a refinement 1809 -> 1006, strip 10x40 558 ->
// 306, a contact step of a 64x64 drape 4315 -> 2157.
//
// What is left is the chains: a level of a unit takes 1 to 1.3 us, most of it sums of
// 8 to 60 dependent terms out of shared memory, at 12 to 20 cycles a term with one to
// five warps busy (two reads and three fused multiply-adds of 7 cycles' latency; the
// reads of the next eight terms issued ahead, or 1,024 threads, changed nothing).
//
// The sums are those of sn_forward and sn_backward, term by term in the same
// order, for a warp's supernodes and for a block's (whose column sums run in
// parts, see UnitNode::width): a result does not depend on which kernel sweeps a
// supernode, nor on how the trees are cut.
//
// U holds a forward update at the place that its entry has in the pull lists
// (B.fwd), so that a column's updates are one run.
#pragma once
#include "pd_kernels.cuh"

namespace vistio {

constexpr uint32_t kUnitThreads = 512;
constexpr uint32_t kUnitWarps = kUnitThreads / 32;
constexpr uint32_t kUnitSmem = 224 * 1024;  // of a block's 227 KB
// The block team whose order of sums a block's supernode has (SweepTeams::bn).
constexpr uint32_t kTeam = 32 * kSolveWarps, kTeamFloats = kSolveWarps * kWarpFloats;
// A supernode of one warp whose rows its warp also pushes; the rows of others are
// shared by all warps.
constexpr uint32_t kOwnRows = 64;
__host__ __device__ constexpr bool unit_own_rows(uint32_t s, uint32_t m) { return s <= 32 && m <= kOwnRows; }
// Floats of each of the two buffers that the values of a supernode too large for
// shared memory pass through.
constexpr uint32_t kStreamFloats = 18 * 1024;

struct __align__(16) UnitNode {
  uint64_t src;       // its region [D | P | rows] (float offset among the garment's)
  uint32_t len;       // floats of D and P, a multiple of 4
  uint32_t at;        // where they are in shared memory (float offset)
  uint32_t p_rel;     // P within the region
  uint32_t s, m;
  uint32_t row0;      // its first column's row of the garment
  uint32_t col0;      // first of its columns among the unit's (each node's padded to 8)
  uint32_t r0;        // first of its rows among the unit's
  uint32_t x0;        // first of its rows among its level's (padded to 8)
  uint32_t width;     // 0: column sums of the backward sweep in one chain. Else in kTeam / width
                      // parts (a power of two, at least s): row j of a chunk in part j % parts
  uint32_t chunk;     // rows of a chunk
  uint32_t part0;     // its partial sums among its level's
  uint32_t pad[2];
};
static_assert(sizeof(UnitNode) == 64, "four 16-byte loads");

struct __align__(16) UnitLevel {
  uint32_t col_task, ncol, push_task, npush, x_task, nx, sum_task, nsum;  // ranges in the unit's tasks
  uint32_t flags;
  uint32_t diag;   // 1 + the node whose diagonal product runs in parts too, or 0
  uint32_t pad[2];
  static constexpr uint32_t kWide = 1;   // some node has more than one task of columns
  static constexpr uint32_t kSplit = 2;  // some node's column sums run in parts
};

// A unit: its nodes (the topmost last), its table and its shared memory. The table's
// parts (ntable words), at these word offsets: tasks (the levels come before them),
// per column its row of the garment (kNoRow: padding), the first and the number of the
// updates that are subtracted when the unit starts, and its first kept update (one
// more), the kept updates' places in U (kInside: a node of the unit writes it), the
// rows above the unit, and per row of a node where its x is in z and the kept update
// or, with kAbove, the place in U that it writes.
constexpr uint32_t kInside = 0xffffffffu, kNoRow = 0xffffffffu, kAbove = 0x80000000u;
struct __align__(16) SweepUnitDev {
  uint32_t node0, nnodes, table0, ntable;  // ranges of the global arrays
  uint32_t inst, bytes, nlevels, root;     // bytes: of the factor values; root: holds its tree's root
  uint32_t ncols, nvals, nabove, stream;   // stream: one node, larger than shared memory
  uint32_t tasks, row_of, list0, nlist, val_ptr, slots, above, x_of;
  uint32_t val_of, nodes_at, table_at, vals_at, z_at, t_at, x_at, part_at;  // ..._at: float4 offsets in shared memory
  uint64_t vals0;                          // the garment's first value, row and place in U
  uint32_t vbase, u0;
  uint32_t lists, pad[3];                  // lists: some column has updates to subtract at the start
};
static_assert(sizeof(SweepUnitDev) == 144, "nine 16-byte loads");

// A task: up to 32 columns or rows of a node, and for a column sum one part of it.
__host__ __device__ constexpr uint32_t unit_task(uint32_t node, uint32_t tile, uint32_t part) {
  return node | tile << 12 | part << 24;
}

// Whether the product with inv(L_kk)^T runs in parts (over more columns than the
// team's buffer holds at a time), the columns it takes at a time then, and the
// power of two that holds those of chunk ch.
__host__ __device__ constexpr bool unit_diag_split(uint32_t s) { return s * sn_ld(s) + 8 > kTeamFloats; }
__host__ __device__ constexpr uint32_t unit_diag_cols(uint32_t s) { return (kTeamFloats - 8) / sn_ld(s); }
__device__ __forceinline__ uint32_t unit_diag_width(uint32_t s, uint32_t ch) {
  const uint32_t cw = unit_diag_cols(s), n = min(cw, s - ch * cw);
  return n <= 1 ? 1u : 1u << (32 - __clz(n - 1));
}

__device__ __forceinline__ void f4_fma_rn(float4& t, float a, float4 y) {
  t.x = __fmaf_rn(a, y.x, t.x); t.y = __fmaf_rn(a, y.y, t.y); t.z = __fmaf_rn(a, y.z, t.z);
}

// acc += a(k) v(k) for k = 0 .. 8 n - 1 in that order: a(k) at a[k ld] (or a[k]), v
// contiguous. The vectors of a unit are padded with zeros to eight entries, and what
// is read of the factor beside them is finite, so the last terms add nothing.
template <bool LD>
__device__ __forceinline__ void unit_chain(float4& acc, const float* a, uint32_t ld, const float4* v, uint32_t n) {
  const uint32_t st = LD ? ld : 1u;
#pragma unroll 1
  for (; n; --n, a += 8 * st, v += 8) {
    float t[8];
    float4 w[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      t[i] = a[i * st];
      w[i] = v[i];
    }
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) f4_fma_rn(acc, t[i], w[i]);
  }
}
// The same over the 32 terms of a diagonal tile, for the lanes whose `use(k)` holds.
template <bool LD, class Use>
__device__ __forceinline__ void unit_chain_tile(float4& acc, const float* a, uint32_t ld, const float4* v, uint32_t n, Use use) {
  const uint32_t st = LD ? ld : 1u;
#pragma unroll 1
  for (uint32_t k = 0; k < n; k += 8, a += 8 * st, v += 8) {
    float t[8];
    float4 w[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      t[i] = a[i * st];
      w[i] = v[i];
    }
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
      if (use(k + i)) f4_fma_rn(acc, t[i], w[i]);
  }
}
// acc += a[k ld] v[k] for k = k0, k0 + step, .. below n.
__device__ __forceinline__ void unit_chain_part(float4& acc, const float* a, uint32_t ld, const float4* v, uint32_t k0, uint32_t n,
                                                uint32_t step) {
#pragma unroll 4
  for (uint32_t k = k0; k < n; k += step) f4_fma_rn(acc, a[k * ld], v[k]);
}

struct UnitSmem {
  const float* fac;
  const UnitNode* nd;
  const uint32_t* tb;
  float4 *vals, *z, *t, *x, *part;
  float4 *Y, *U;  // the garment's
};

// y = inv(L_kk) t for the columns of a task.
__device__ __forceinline__ void unit_diag_forward(const UnitSmem& M, const UnitNode& N, uint32_t c0) {
  const uint32_t s = N.s, lane = threadIdx.x & 31, c = c0 + lane, ld = sn_ld(s);
  const float* D = M.fac + N.at + min(c, s - 1);
  const float4* t = M.t + N.col0;
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
  unit_chain<true>(y, D, ld, t, c0 / 8);
  unit_chain_tile<true>(y, D + c0 * ld, ld, t + c0, min(32u, s - c0), [&](uint32_t k) { return k <= lane; });
  if (c < s) {
    M.z[N.col0 + c] = y;
    M.Y[N.row0 + c] = y;
  }
}
// x = inv(L_kk)^T t for the columns of a task.
__device__ __forceinline__ void unit_diag_backward(const UnitSmem& M, const UnitNode& N, uint32_t c0) {
  const uint32_t s = N.s, lane = threadIdx.x & 31, c = c0 + lane;
  const float* D = M.fac + N.at + min(c, s - 1) * sn_ld(s) + c0;
  const float4* t = M.t + N.col0 + c0;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  unit_chain_tile<false>(x, D, 1, t, min(32u, s - c0), [&](uint32_t k) { return k >= lane; });
  if (s > c0 + 32) unit_chain<false>(x, D + 32, 1, t + 32, (s - c0 - 32 + 7) / 8);
  if (c < s) {
    M.z[N.col0 + c] = x;
    M.Y[N.row0 + c] = x;
  }
}

// x from the parts of a split diagonal product.
__device__ __forceinline__ void unit_diag_combine(const UnitSmem& M, const UnitNode& N) {
  const uint32_t s = N.s, cw = unit_diag_cols(s);
  for (uint32_t c = threadIdx.x; c < s; c += kUnitThreads) {
    const uint32_t ch = c / cw, w = unit_diag_width(s, ch), np = kTeam / w;
    const float4* p = M.part + ch * kTeam + (c - ch * cw);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (uint32_t q = 0; q < np; ++q) a = f4_add(a, p[q * w]);
    M.z[N.col0 + c] = a;
    M.Y[N.row0 + c] = a;
  }
}

// u = P y for 32 rows of a node.
__device__ __forceinline__ void unit_push(const UnitSmem& M, const UnitNode& N, const uint32_t* val_of, uint32_t j0) {
  const uint32_t m = N.m, j = j0 + (threadIdx.x & 31);
  float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
  unit_chain<false>(u, M.fac + N.at + N.p_rel + min(j, m - 1) * sn_ld(N.s), 1, M.z + N.col0, (N.s + 7) / 8);
  if (j < m) {
    const uint32_t v = val_of[N.r0 + j];
    if (v & kAbove) M.U[v & ~kAbove] = u;
    else M.vals[v] = u;
  }
}

// The levels of a unit from its leaves: t = the column's entry less what its
// descendants pushed, in list order; y = inv(L_kk) t; u = P y. A warp whose task
// holds all columns of its node goes on from t to y, and to u if the rows are few.
__device__ __forceinline__ void unit_forward(const SweepUnitDev& U, const UnitSmem& M) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nlevels = U.nlevels;
  const uint32_t* tk = M.tb + U.tasks;
  const uint32_t* vp = M.tb + U.val_ptr;
  const uint32_t* val_of = M.tb + U.val_of;
  for (uint32_t l = 0; l < nlevels; ++l) {
    const UnitLevel& L = reinterpret_cast<const UnitLevel*>(M.tb)[l];
    for (uint32_t i = warp, n = L.ncol; i < n; i += kUnitWarps) {
      const uint32_t w = tk[L.col_task + i];
      const UnitNode& N = M.nd[w & 0xfffu];
      const uint32_t s = N.s, c = (w >> 12 & 0xfffu) * 32 + lane, col = N.col0 + min(c, s - 1);
      float4 t = M.z[col];
      for (uint32_t q = vp[col], qe = vp[col + 1]; q < qe; q += 4) {
        float4 v[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) v[e] = M.vals[min(q + e, qe - 1)];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e)
          if (q + e < qe) t = f4_sub(t, v[e]);
      }
      if (c < s) M.t[col] = t;
      if (s > 32) continue;
      __syncwarp();
      unit_diag_forward(M, N, 0);
      if (!unit_own_rows(s, N.m)) continue;
      __syncwarp();
      for (uint32_t j0 = 0; j0 < N.m; j0 += 32) unit_push(M, N, val_of, j0);
    }
    __syncthreads();
    if (L.flags & UnitLevel::kWide) {
      for (uint32_t i = warp, n = L.ncol; i < n; i += kUnitWarps) {
        const uint32_t w = tk[L.col_task + i];
        const UnitNode& N = M.nd[w & 0xfffu];
        if (N.s > 32) unit_diag_forward(M, N, (w >> 12 & 0xfffu) * 32);
      }
      __syncthreads();
    }
    if (!L.npush) continue;
    for (uint32_t i = warp, n = L.npush; i < n; i += kUnitWarps) {
      const uint32_t w = tk[L.push_task + i];
      unit_push(M, M.nd[w & 0xfffu], val_of, (w >> 12 & 0xfffu) * 32);
    }
    __syncthreads();
  }
}

// The levels from the unit's root: t = y - P^T x; x = inv(L_kk)^T t. A warp's
// supernode is one task.
__device__ __forceinline__ void unit_backward(const SweepUnitDev& U, const UnitSmem& M) {
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t* tk = M.tb + U.tasks;
  const uint32_t* x_of = M.tb + U.x_of;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const auto gather = [&](const UnitNode& N, uint32_t j) {
    if (j < ((N.m + 7) & ~7u)) M.x[N.x0 + j] = j < N.m ? M.z[x_of[N.r0 + j]] : zero;
  };
  for (uint32_t l = U.nlevels; l-- > 0;) {
    const UnitLevel& L = reinterpret_cast<const UnitLevel*>(M.tb)[l];
    if (L.nx) {
      for (uint32_t i = warp, n = L.nx; i < n; i += kUnitWarps) {
        const uint32_t w = tk[L.x_task + i];
        gather(M.nd[w & 0xfffu], (w >> 12 & 0xfffu) * 32 + lane);
      }
      __syncthreads();
    }
    for (uint32_t i = warp, n = L.nsum; i < n; i += kUnitWarps) {
      const uint32_t w = tk[L.sum_task + i];
      const UnitNode& N = M.nd[w & 0xfffu];
      const uint32_t c = (w >> 12 & 0xfffu) * 32 + lane, q = w >> 24, s = N.s, ld = sn_ld(s), m = N.m, width = N.width;
      const float* P = M.fac + N.at + N.p_rel + min(c, s - 1);
      const float4* x = M.x + N.x0;
      const uint32_t parts = width ? kTeam / width : 1u;
      float4 a = zero;
      if (!width) {
        for (uint32_t j0 = 0; j0 < m; j0 += 32) gather(N, j0 + lane);
        __syncwarp();
      }
      if (parts == 1) {
        unit_chain<true>(a, P, ld, x, (m + 7) / 8);
      } else {
        for (uint32_t j0 = 0; j0 < m; j0 += N.chunk) unit_chain_part(a, P, ld, x, j0 + q, min(m, j0 + N.chunk), parts);
        if (c < width) M.part[N.part0 + q * width + c] = a;
        continue;
      }
      if (c < s) M.t[N.col0 + c] = f4_sub(M.z[N.col0 + c], a);
      if (!width) {
        __syncwarp();
        unit_diag_backward(M, N, 0);
      }
    }
    __syncthreads();
    if (L.flags & UnitLevel::kSplit) {
      for (uint32_t i = warp, n = L.ncol; i < n; i += kUnitWarps) {
        const uint32_t w = tk[L.col_task + i];
        const UnitNode& N = M.nd[w & 0xfffu];
        const uint32_t c = (w >> 12 & 0xfffu) * 32 + lane, parts = N.width ? kTeam / N.width : 1u;
        if (parts > 1 && c < N.s) {
          float4 a = zero;
#pragma unroll 4
          for (uint32_t q = 0; q < parts; ++q) a = f4_add(a, M.part[N.part0 + q * N.width + c]);
          M.t[N.col0 + c] = f4_sub(M.z[N.col0 + c], a);
        }
      }
      __syncthreads();
    }
    if (!(L.flags & (UnitLevel::kSplit | UnitLevel::kWide))) continue;
    for (uint32_t i = warp, n = L.ncol; i < n; i += kUnitWarps) {
      const uint32_t w = tk[L.col_task + i];
      const UnitNode& N = M.nd[w & 0xfffu];
      if (N.width && !unit_diag_split(N.s)) unit_diag_backward(M, N, (w >> 12 & 0xfffu) * 32);
    }
    if (L.diag) {  // some columns at a time, each column's rows in parts
      const UnitNode& N = M.nd[L.diag - 1];
      const uint32_t s = N.s, ld = sn_ld(s), cw = unit_diag_cols(s), nch = (s + cw - 1) / cw;
      for (uint32_t e = tid; e < nch * kTeam; e += kUnitThreads) {
        const uint32_t ch = e / kTeam, r = e % kTeam, w = unit_diag_width(s, ch), c = ch * cw + r % w;
        float4 a = zero;
        if (c < min(s, (ch + 1) * cw)) unit_chain_part(a, M.fac + N.at + c * ld, 1, M.t + N.col0, c + r / w, s, kTeam / w);
        M.part[e] = a;
      }
      __syncthreads();
      unit_diag_combine(M, N);
    }
    __syncthreads();
  }
}

// The step of a supernode larger than shared memory: its values, columns of D and
// rows of P, pass through two buffers in the order they are used, the next part
// in flight. Thread c holds column c's sum (backward: one of its parts) over the
// parts.
struct UnitStream {
  const float* src;
  float* buf;
  uint64_t* bar;
  uint32_t ld, per;  // vectors of ld floats that a buffer holds
  // the floats that hold vectors [v0, v1) of a matrix at float offset `at` of the
  // region; where vector v0 lands in the buffer
  __device__ __forceinline__ uint32_t issue(uint32_t k, uint32_t at, uint32_t v0, uint32_t v1) const {
    const uint32_t f0 = (at + v0 * ld) & ~3u, f1 = (at + v1 * ld + 3) & ~3u;
    if (threadIdx.x == 0) {
      uint64_t* b = bar + (k & 1);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"((f1 - f0) * 4) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       smem_u32(buf + (k & 1) * kStreamFloats)),
                   "l"(src + f0), "r"((f1 - f0) * 4), "r"(smem_u32(b))
                   : "memory");
    }
    __syncwarp();
    return (at + v0 * ld) & 3u;
  }
};

template <int DIR>
__device__ __forceinline__ void unit_stream(const BatchDev& B, const SweepUnitDev& U, const UnitSmem& M, const UnitStream& S,
                                            bool ahead, bool second) {
  const UnitNode& N = M.nd[0];
  const uint32_t tid = threadIdx.x, s = N.s, m = N.m, ld = S.ld, per = S.per;
  const uint32_t nd = (s + per - 1) / per, np = (m + per - 1) / per, n = nd + np;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // part k of the sequence: D's columns then P's rows (backward: P first)
  const auto is_d = [&](uint32_t k) { return DIR == 0 ? k < nd : k >= np; };
  const auto first = [&](uint32_t k) { return (DIR == 0 ? (k < nd ? k : k - nd) : (k < np ? k : k - np)) * per; };
  const auto issue = [&](uint32_t k) {
    const bool d = is_d(k);
    const uint32_t v0 = first(k);
    S.issue(k, d ? 0u : N.p_rel, v0, min(v0 + per, d ? s : m));
  };
  if (ahead) {  // of the wait for the kernel before
    for (uint32_t k = 0; k < min(2u, n); ++k) issue(k);
    return;
  }
  // times a buffer was filled before (a second pass over the same parts)
  const uint32_t used0 = second ? (n + 1) / 2 : 0u, used1 = second ? n / 2 : 0u;
  const uint32_t* val_of = M.tb + U.val_of;
  const float4* x = M.z + U.ncols;  // backward: its rows are the rows above
  const uint32_t parts = N.width ? kTeam / N.width : 1u, width = N.width ? N.width : 32u;
  const uint32_t c = DIR == 0 ? tid : tid % width, q = DIR == 0 ? 0u : tid / width;
  const bool split = unit_diag_split(s);
  float4 acc = zero;
  if (DIR == 1 && np == 0) {
    if (tid < s) M.t[tid] = M.z[tid];
    __syncthreads();
  }
  for (uint32_t k = 0; k < n; ++k) {
    const bool d = is_d(k);
    const uint32_t v0 = first(k), v1 = min(v0 + per, d ? s : m);
    const float* a = S.buf + (k & 1) * kStreamFloats + (((d ? 0u : N.p_rel) + v0 * ld) & 3u);
    if (!mbar_wait(S.bar + (k & 1), ((k >> 1) + (k & 1 ? used1 : used0)) & 1u)) atomicOr(B.status, 4u);
    if (DIR == 0 && d) {
      if (c < s)
        for (uint32_t i = v0; i < min(v1, c + 1); ++i) f4_fma_rn(acc, a[(i - v0) * ld + c], M.z[i]);
    } else if (DIR == 0) {
      for (uint32_t j = v0 + tid; j < v1; j += kUnitThreads) {
        float4 u = zero;
        for (uint32_t i = 0; i < s; ++i) f4_fma_rn(u, a[(j - v0) * ld + i], M.t[i]);
        M.U[val_of[N.r0 + j] & ~kAbove] = u;
      }
    } else if (!d) {
      if (c < s && q < parts)
        for (uint32_t j0 = v0 / N.chunk * N.chunk; j0 < v1; j0 += N.chunk) {
          uint32_t j = j0 + q;
          if (j < v0) j += (v0 - j + parts - 1) / parts * parts;
          for (const uint32_t je = min(v1, j0 + N.chunk); j < je; j += parts) f4_fma_rn(acc, a[(j - v0) * ld + c], x[j]);
        }
    } else if (!split) {
      if (tid >= v0 && tid < v1) {
        float4 t = zero;
        unit_chain_part(t, a + (tid - v0) * ld, 1, M.t, tid, s, 1);
        M.z[tid] = t;
        M.Y[N.row0 + tid] = t;
      }
    } else {
      const uint32_t cw = unit_diag_cols(s);
      for (uint32_t ch = v0 / cw; ch * cw < v1; ++ch) {
        const uint32_t w = unit_diag_width(s, ch), e = tid, col = ch * cw + e % w;
        if (e < kTeam && col >= v0 && col < min(v1, min(s, (ch + 1) * cw))) {
          float4 p = zero;
          unit_chain_part(p, a + (col - v0) * ld, 1, M.t, col + e / w, s, kTeam / w);
          M.part[ch * kTeam + e] = p;
        }
      }
    }
    __syncthreads();  // every thread is done with the buffer
    if (k + 2 < n) issue(k + 2);
    if (DIR == 0 && k + 1 == nd) {
      if (c < s) {
        M.t[c] = acc;
        M.Y[N.row0 + c] = acc;
      }
      __syncthreads();
    }
    if (DIR == 1 && k + 1 == np) {
      if (c < s && q < parts) M.part[q * width + c] = acc;
      __syncthreads();
      if (tid < s) {
        float4 t = zero;
        for (uint32_t p = 0; p < parts; ++p) t = f4_add(t, M.part[p * width + tid]);
        M.t[tid] = f4_sub(M.z[tid], t);
      }
      __syncthreads();
    }
  }
  if (DIR == 1 && split) unit_diag_combine(M, N);
}

// One phase: block b sweeps unit b, forward (DIR = 0; a unit with its tree's root
// then backward too) or backward (DIR = 1).
template <int DIR>
__global__ void __launch_bounds__(kUnitThreads) k_units(BatchDev B, const SweepUnitDev* __restrict__ units,
                                                        const UnitNode* __restrict__ nodes,
                                                        const uint32_t* __restrict__ tables) {
  extern __shared__ float4 smem4[];
  __shared__ SweepUnitDev U;
  __shared__ uint64_t bar[2];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < sizeof(U) / 16) reinterpret_cast<uint4*>(&U)[tid] = __ldg(reinterpret_cast<const uint4*>(units + blockIdx.x) + tid);
  if (tid < 2) mbar_init(&bar[tid]);
  mbar_fence_init();
  __syncthreads();
  float* fac = reinterpret_cast<float*>(smem4);
  UnitNode* nd = reinterpret_cast<UnitNode*>(smem4 + U.nodes_at);
  uint4* table = reinterpret_cast<uint4*>(smem4 + U.table_at);
  for (uint32_t i = tid; i < U.nnodes * 4; i += kUnitThreads)
    reinterpret_cast<uint4*>(nd)[i] = __ldg(reinterpret_cast<const uint4*>(nodes + U.node0) + i);
  for (uint32_t i = tid; i < U.ntable / 4; i += kUnitThreads)
    table[i] = __ldg(reinterpret_cast<const uint4*>(tables + U.table0) + i);
  __syncthreads();
  const UnitSmem M{fac, nd, reinterpret_cast<const uint32_t*>(table), smem4 + U.vals_at, smem4 + U.z_at, smem4 + U.t_at, smem4 + U.x_at,
                   smem4 + U.part_at, B.Y + U.vbase, B.U + U.u0};
  const float* vals = B.vals + U.vals0;
  const UnitStream S{vals + nd[0].src, fac, bar, sn_ld(nd[0].s), (kStreamFloats - 8) / sn_ld(nd[0].s)};
  if (U.stream) {
    unit_stream<DIR>(B, U, M, S, true, false);
  } else {
    // the factor values of every node, all copies in flight at once
    if (warp == 0) {
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bar[0])), "r"(U.bytes) : "memory");
      __syncwarp();
      for (uint32_t i = lane; i < U.nnodes; i += 32)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(fac + nd[i].at)),
                     "l"(vals + nd[i].src), "r"(nd[i].len * 4), "r"(smem_u32(&bar[0]))
                     : "memory");
      __syncwarp();
    }
    // what pads the factor values and the vectors
    for (uint32_t i = U.bytes / 16 + tid; i < U.nodes_at; i += kUnitThreads) smem4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i = tid; i < U.ncols; i += kUnitThreads) M.t[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  pdl_begin();
  const uint32_t ipc = B.prm->ipc, done = B.red[U.inst].al_done;  // with the loads below in flight
  for (uint32_t c = tid; c < U.ncols; c += kUnitThreads) {
    const uint32_t row = M.tb[U.row_of + c];
    M.z[c] = row == kNoRow ? make_float4(0.f, 0.f, 0.f, 0.f) : M.Y[row];
  }
  if (DIR == 0) {
    for (uint32_t i = tid; i < U.nvals; i += kUnitThreads) {
      const uint32_t at = M.tb[U.slots + i];
      if (at != kInside) M.vals[i] = M.U[at];
    }
  } else {
    for (uint32_t i = tid; i < U.nabove; i += kUnitThreads) M.z[U.ncols + i] = M.Y[M.tb[U.above + i]];
  }
  if (ipc && done) {  // the copies in flight land before the block ends
    if (!mbar_wait(&bar[0], 0u) || (U.stream && !mbar_wait(&bar[1], 0u))) atomicOr(B.status, 4u);
    return;
  }
  if (DIR == 0 && U.lists) {
    __syncthreads();
    // one component of one column per thread, thirty-two updates in flight
    const float* Uf = reinterpret_cast<const float*>(M.U);
    for (uint32_t e = tid; e < 4 * U.ncols; e += kUnitThreads) {
      const uint32_t c = e >> 2, n = M.tb[U.nlist + c];
      if (!n || (e & 3u) == 3u) continue;
      const float* u = Uf + 4ull * M.tb[U.list0 + c] + (e & 3u);
      float t = reinterpret_cast<const float*>(M.z + c)[e & 3u];
      for (uint32_t q = 0; q < n; q += 32) {
        float v[32];
#pragma unroll
        for (uint32_t i = 0; i < 32; ++i) v[i] = u[4 * min(q + i, n - 1)];
#pragma unroll
        for (uint32_t i = 0; i < 32; ++i)
          if (q + i < n) t -= v[i];
      }
      reinterpret_cast<float*>(M.z + c)[e & 3u] = t;
    }
  }
  if (U.stream) {
    __syncthreads();
    unit_stream<DIR>(B, U, M, S, false, false);
    if (DIR == 0 && U.root) {  // the values pass again, in the backward order; no rows above a root
      __syncthreads();
      if (tid < U.ncols) M.z[tid] = M.t[tid];
      __syncthreads();
      unit_stream<1>(B, U, M, S, true, true);
      unit_stream<1>(B, U, M, S, false, true);
    }
    return;
  }
  if (!mbar_wait(&bar[0], 0u)) atomicOr(B.status, 4u);
  __syncthreads();
  if (DIR == 0) unit_forward(U, M);
  if (DIR == 1 || U.root) unit_backward(U, M);
}

}  // namespace vistio
