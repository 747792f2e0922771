// Numeric factorization of P A P^T on the GPU in FP64 (multifrontal), writing
// the FP32 panels the sweeps read. The host does the symbolic analysis
// (ordering, merged supernodes, row structures); the numbers are computed here
// once per garment, material and dt, where the reference uses faer's FP64 LL^T
// (crates/vistio-solver/src/faer_solver.rs:67-93).
//
// Every supernode k (columns f .. f+s, rows R below, n_f = s + m) has a front:
// the lower triangle of an n_f x n_f FP64 matrix, row-major. Supernodes are
// processed by height in the tree, each height over every garment:
//   assemble  the supernode's columns of A plus the update matrices of its
//             children (extend-add through the host-computed map of each child's
//             rows into this front, children one after another);
//   eliminate the first s columns by symmetric Gauss-Jordan steps on 32
//             pivots at a time. With K the block's pivots, P = F_KK^-1 and V the
//             columns F_.K, every other entry becomes F_ij - V_i P V_j^T, the
//             block itself P and its rows and columns -V P. After the last
//             block the front holds N = F_11^-1, -W = -F_21 N and the update
//             matrix F_22 - W F_12 for the parent;
//   emit      N and W in FP32 into the supernode's two panels (SnDev).
// A step is two launches over all fronts of the height: the pivots' inverse
// and V P (k_fpivot), then the lower triangle in 64 x 64 tiles (k_fupdate,
// 32 fused multiply-adds per entry read and written), so that large fronts are
// spread over the SMs. Against one block per front of a tree of many small
// supernodes, with a rank-1 update per column: 512 sheets of sides 23 to 121,
// 184 -> 80 ms for all fronts and panels.
#pragma once
#include "pd_kernels.cuh"

namespace vistio {

constexpr uint32_t kPivots = 32;
constexpr uint32_t kAssembleRows = 16;
constexpr uint32_t kPivotRows = 128;
constexpr uint32_t kUpdateTile = 64;

struct FrontDev {
  const SnDev* sn;
  const uint32_t* rows;       // below-diagonal rows of each supernode (instance-local)
  const uint32_t* a_ptr;      // A in solve order (global rows), f64, both triangles
  const uint32_t* a_col;
  const double* a_val;
  const uint64_t* front_off;  // doubles: where each supernode's front starts
  const uint64_t* work_off;   // doubles: V (n_f x 32), V P (n_f x 32) and P (32 x 32) of a step
  const uint32_t* kid_ptr;    // children of each supernode (global ids)
  const uint32_t* kids;
  const uint32_t* relmap;     // per supernode row (indexed like rows): its position in the parent's front
  const uint64_t* host_p;     // host-factored garments: offsets of L_Rk (m x s, row-major) and
  const uint64_t* host_d;     // inv(L_kk) (s x s, column-major) in host_vals
  const double* host_vals;
  double* fronts;
  double* work;
  float* vals;
  uint32_t* status;           // bit 5: a pivot <= 0 (not positive definite)
};

// One block per (front, kAssembleRows rows).
__global__ void __launch_bounds__(256) k_fassemble(FrontDev D, const uint2* __restrict__ items) {
  const uint2 it = items[blockIdx.x];
  const SnDev S = D.sn[it.x];
  const uint32_t s = S.ncols, nf = s + S.nrows, f = S.first, vb = S.vbase;
  const uint32_t r0 = it.y * kAssembleRows, r1 = min(nf, r0 + kAssembleRows), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* F = D.fronts + D.front_off[it.x];
  for (uint32_t r = r0 + warp; r < r1; r += 8) {
    double* row = F + uint64_t(r) * nf;
    for (uint32_t c = lane; c <= r; c += 32) row[c] = 0.0;
    __syncwarp();
    // the row's entries of A in the supernode's columns, up to the diagonal
    const uint32_t ar = vb + (r < s ? f + r : D.rows[S.rows_off + r - s]);
    const uint32_t last = vb + f + min(r, s - 1);
    for (uint32_t q = D.a_ptr[ar] + lane, qe = D.a_ptr[ar + 1]; q < qe; q += 32) {
      const uint32_t c = D.a_col[q];
      if (c >= vb + f && c <= last) row[c - vb - f] = D.a_val[q];
    }
  }
  for (uint32_t ci = D.kid_ptr[it.x], ce = D.kid_ptr[it.x + 1]; ci < ce; ++ci) {
    __syncthreads();
    const uint32_t ch = D.kids[ci];
    const SnDev C = D.sn[ch];
    const uint32_t sc = C.ncols, mc = C.nrows, nfc = sc + mc;
    const double* Fc = D.fronts + D.front_off[ch];
    const uint32_t* map = D.relmap + C.rows_off;  // ascending
    uint32_t lo = 0, hi = mc;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (map[mid] < r0) lo = mid + 1; else hi = mid;
    }
    for (uint32_t i = lo + warp; i < mc && map[i] < r1; i += 8) {
      double* row = F + uint64_t(map[i]) * nf;
      const double* from = Fc + uint64_t(sc + i) * nfc + sc;
      for (uint32_t j = lane; j <= i; j += 32) row[map[j]] += from[j];
    }
  }
}

// Step `t` of the elimination, first half: one block per (front, kPivotRows
// rows) inverts the pivot block and forms V and V P for its rows. Nothing in the
// front changes here, so the blocks of one front need not wait for each other.
__global__ void __launch_bounds__(kPivotRows) k_fpivot(FrontDev D, const uint2* __restrict__ items, uint32_t t) {
  __shared__ double P[kPivots][kPivots + 1];
  const uint2 it = items[blockIdx.x];
  const SnDev S = D.sn[it.x];
  const uint32_t s = S.ncols, nf = s + S.nrows, k0 = t * kPivots, b = min(kPivots, s - k0), tid = threadIdx.x;
  const double* F = D.fronts + D.front_off[it.x];
  double* V = D.work + D.work_off[it.x];
  double* Q = V + uint64_t(nf) * kPivots;
  // the block, padded to 32 pivots by the identity: thread tid holds column
  // tid & 31 of the rows tid / 32 + 4 u
  constexpr uint32_t kRows = kPivots * kPivots / kPivotRows;
  const uint32_t pj = tid & 31, pi = tid >> 5;
  double x[kRows];
#pragma unroll
  for (uint32_t u = 0; u < kRows; ++u) {
    const uint32_t i = pi + 4 * u;
    x[u] = i < b && pj < b ? F[uint64_t(k0 + max(i, pj)) * nf + k0 + min(i, pj)] : i == pj ? 1.0 : 0.0;
    P[i][pj] = x[u];
  }
  __syncthreads();
  // in-place inverse by Gauss-Jordan steps; the pivots are those of a Cholesky
  bool bad = false;
  for (uint32_t k = 0; k < b; ++k) {
    double d = P[k][k];
    if (!(d > 0.0) || !isfinite(d)) {
      bad = true;
      d = 1.0;  // keep going with finite numbers; the host reports the failure
    }
    const double inv = 1.0 / d, row = P[k][pj] * inv;
#pragma unroll
    for (uint32_t u = 0; u < kRows; ++u) {
      const uint32_t i = pi + 4 * u;
      const double col = P[i][k];
      x[u] = i == k ? (pj == k ? inv : row) : pj == k ? -col * inv : x[u] - col * row;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kRows; ++u) P[pi + 4 * u][pj] = x[u];
    __syncthreads();
  }
  if (bad && tid == 0) atomicOr(D.status, 32u);
  if (it.y == 0) {
    double* Pw = Q + uint64_t(nf) * kPivots;
    for (uint32_t e = tid; e < kPivots * kPivots; e += kPivotRows) Pw[e] = P[e / kPivots][e % kPivots];
  }
  const uint32_t i = it.y * kPivotRows + tid;
  if (i >= nf || (i >= k0 && i < k0 + b)) return;
  // V_i: below the block its row, before it (already eliminated) minus its
  // column of the pivot rows
  double w[kPivots];
#pragma unroll
  for (uint32_t q = 0; q < kPivots; ++q)
    w[q] = q >= b ? 0.0 : i > k0 ? F[uint64_t(i) * nf + k0 + q] : -F[uint64_t(k0 + q) * nf + i];
#pragma unroll
  for (uint32_t q = 0; q < kPivots; ++q) V[uint64_t(i) * kPivots + q] = w[q];
#pragma unroll 4
  for (uint32_t j = 0; j < kPivots; ++j) {
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (uint32_t q = 0; q < kPivots; q += 2) {
      a0 += w[q] * P[q][j];
      a1 += w[q + 1] * P[q + 1][j];
    }
    Q[uint64_t(i) * kPivots + j] = a0 + a1;
  }
}

// Second half: one block per 64 x 64 tile of a front's lower triangle (it.y =
// tile row << 16 | tile column).
__global__ void __launch_bounds__(256) k_fupdate(FrontDev D, const uint2* __restrict__ items, uint32_t t) {
  __shared__ double sv[kPivots][kUpdateTile + 1], sq[kPivots][kUpdateTile + 1];
  const uint2 it = items[blockIdx.x];
  const SnDev S = D.sn[it.x];
  const uint32_t s = S.ncols, nf = s + S.nrows, k0 = t * kPivots, b = min(kPivots, s - k0), k1 = k0 + b;
  const uint32_t i0 = (it.y >> 16) * kUpdateTile, j0 = (it.y & 0xffffu) * kUpdateTile;
  double* F = D.fronts + D.front_off[it.x];
  const double* V = D.work + D.work_off[it.x];
  const double* Q = V + uint64_t(nf) * kPivots;
  const double* Pw = Q + uint64_t(nf) * kPivots;
  auto in_k = [&](uint32_t r) { return r >= k0 && r < k1; };
  for (uint32_t e = threadIdx.x; e < kUpdateTile * kPivots; e += 256) {
    const uint32_t r = e / kPivots, q = e % kPivots, i = i0 + r, j = j0 + r;
    sv[q][r] = i < nf && !in_k(i) ? V[uint64_t(i) * kPivots + q] : 0.0;
    // P F_Kj: V_j P, with the sign of the eliminated columns
    sq[q][r] = j < nf && !in_k(j) ? (j < k0 ? -1.0 : 1.0) * Q[uint64_t(j) * kPivots + q] : 0.0;
  }
  __syncthreads();
  const uint32_t tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[4][4] = {};
  for (uint32_t q = 0; q < b; ++q) {
    double x[4], y[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) { x[u] = sv[q][ty + 16 * u]; y[u] = sq[q][tx + 16 * u]; }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
      for (uint32_t w = 0; w < 4; ++w) acc[u][w] += x[u] * y[w];
  }
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
    for (uint32_t w = 0; w < 4; ++w) {
      const uint32_t i = i0 + ty + 16 * u, j = j0 + tx + 16 * w;
      if (i >= nf || j > i) continue;
      double* p = F + uint64_t(i) * nf + j;
      const bool ik = in_k(i), jk = in_k(j);
      if (ik && jk) *p = Pw[(i - k0) * kPivots + j - k0];
      else if (jk) *p = -Q[uint64_t(i) * kPivots + j - k0];
      else if (ik) *p = -Q[uint64_t(j) * kPivots + i - k0];
      else *p -= acc[u][w];
    }
}

// Garments factored on the host (L_Rk and inv(L_kk) in FP64): N = inv(L_kk)^T
// inv(L_kk) and W = L_Rk inv(L_kk) into the front's layout (-W below N); one
// block per 32 x 32 tile (it.y = tile row << 16 | tile column of (s + m) x s).
__global__ void __launch_bounds__(256) k_ffrom_host(FrontDev D, const uint2* __restrict__ items) {
  __shared__ double sa[32][33], sb[32][33];
  const uint2 it = items[blockIdx.x];
  const SnDev S = D.sn[it.x];
  const uint32_t s = S.ncols, nf = s + S.nrows, i0 = (it.y >> 16) * 32, j0 = (it.y & 0xffffu) * 32;
  const double* Pn = D.host_vals + D.host_p[it.x];
  const double* Dn = D.host_vals + D.host_d[it.x];
  double* F = D.fronts + D.front_off[it.x];
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double acc[4] = {};
  for (uint32_t q0 = 0; q0 < s; q0 += 32) {
    __syncthreads();
    for (uint32_t r = ty; r < 32; r += 8) {
      const uint32_t i = i0 + r, j = j0 + r, q = q0 + tx;
      sa[r][tx] = q < s && i < nf ? (i < s ? Dn[uint64_t(i) * s + q] : Pn[uint64_t(i - s) * s + q]) : 0.0;
      sb[r][tx] = q < s && j < s ? Dn[uint64_t(j) * s + q] : 0.0;
    }
    __syncthreads();
    for (uint32_t q = 0; q < 32; ++q)
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) acc[u] += sa[ty + 8 * u][q] * sb[tx][q];
  }
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u) {
    const uint32_t i = i0 + ty + 8 * u, j = j0 + tx;
    if (i < nf && j < s && j <= i) F[uint64_t(i) * nf + j] = i < s ? acc[u] : -acc[u];
  }
}

// N and W in FP32 into the two panels, tile by tile (SnDev); one block per
// (supernode, 32 forward rows: the m rows of W, then the s rows of N).
__global__ void __launch_bounds__(256) k_femit(FrontDev D, const uint2* __restrict__ items) {
  __shared__ float tile[32][33];
  const uint2 it = items[blockIdx.x];
  const SnDev S = D.sn[it.x];
  const uint32_t s = S.ncols, m = S.nrows, nf = s + m, r0 = it.y * 32;
  const uint32_t wf = min(32u, (nf - r0 + 7u) & ~7u);
  const double* F = D.fronts + D.front_off[it.x];
  float* fwd = D.vals + S.f_off + uint64_t(r0) * s;
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (uint32_t c0 = 0; c0 < s; c0 += 32) {
    const uint32_t wb = min(32u, (s - c0 + 7u) & ~7u);
    float* bwd = D.vals + S.b_off + uint64_t(c0) * m;
    __syncthreads();
    for (uint32_t r = ty; r < 32; r += 8) {
      const uint32_t row = r0 + r, c = c0 + tx;
      float v = 0.f;  // the rows that pad a tile
      if (row < nf && c < s) {
        const uint32_t i = row < m ? 0u : row - m;
        v = row < m ? float(-F[uint64_t(s + row) * nf + c]) : float(F[uint64_t(max(i, c)) * nf + min(i, c)]);
      }
      tile[r][tx] = v;
      if (row < m && tx < wb) bwd[uint64_t(row) * wb + tx] = v;
    }
    __syncthreads();
    for (uint32_t c = ty; c < 32; c += 8)
      if (c0 + c < s && tx < wf) fwd[uint64_t(c0 + c) * wf + tx] = tile[tx][c];
  }
}

}  // namespace vistio
