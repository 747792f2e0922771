// sm_100a kernels of the Projective Dynamics iteration.
//
// Layout (ragged SoA over every instance of a batch): per-vertex float4
// (x, y, z, -) arrays indexed by a global vertex id; triangles and hinges
// hold global vertex ids; each kernel over elements or vertices runs one
// block per "chunk" (instance, first element, count <= blockDim) so a block
// always sees a single instance and its constants.
//
// The iteration is written in delta form: with A the constant PD matrix
// (M/h^2 + sum w S^T S + sum w_b L^T L) and b the reference's right-hand side
// (assembly.rs:157-240), the solve computes d = A^-1 (b - A x) and sets
// x <- x + d, which equals the reference's x <- A^-1 b in exact arithmetic.
// b - A x collapses per element to w g_k . (F_target - F) for a triangle and
// to w s_k s . (target - x) for a hinge, so the residual is formed from small
// differences and FP32 sweeps lose accuracy relative to |d|, not to |x|.
#pragma once
#include <cstdint>
#include <utility>
#include <cuda_runtime.h>

#include "setup.h"

namespace vistio {

// Programmatic dependent launch. The step's kernels are launched with the
// programmatic stream serialization attribute (launch_pdl on the host), so a
// kernel's blocks may be scheduled while the kernel before it in the stream
// is still running. Each such kernel calls pdl_begin() first: it waits until
// the previous kernel has completed and its memory is visible, which orders
// every earlier kernel too (each of them waited for its own predecessor). A
// grid of at most kPdlEarlyBlocks blocks then lets the next kernel launch
// right away, so that kernel's launch overlaps this one's work; larger grids
// leave the SMs to their own blocks. In a kernel launched without the
// attribute both instructions do nothing.
constexpr uint32_t kPdlEarlyBlocks = 148;
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (gridDim.x * gridDim.y * gridDim.z <= kPdlEarlyBlocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches a step kernel with the programmatic stream serialization
// attribute (the kernel calls pdl_begin() first); records errors as a <<<>>>
// launch would.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

struct InstDev {
  uint32_t vbase, nv;
  uint32_t nlvl;               // levels of the supernodal elimination tree
  float kappa;                 // barrier stiffness estimated from this garment's own masses
  int32_t model;
  float warp, weft;
  float inv_hmat2;   // 1 / matrix_dt^2
  int32_t has_ground;
  float ground_h;
  uint32_t sn_base, nsn;
  int32_t unit_stencils;       // every hinge stencil is (-1, -1, 1, 1) (dihedral bending): not loaded
  uint32_t tbase, hbase;       // first triangle and hinge of the garment
  uint32_t inc_ptr;            // its connectivity class's per-vertex offsets in vtri_ptr / vhinge_ptr
  uint32_t tinc_off, hinc_off; // its class's codes in vtri / vhinge
};

// One supernode of the merged elimination tree in HBM: its two panels in vals,
// in tiles of 32 rows (the last tile's rows padded to 8), a tile column by
// column; 32-byte aligned.
//   forward   m + s rows (W, then N) of s columns
//   backward  s rows (W^T) of m columns
struct SnDev {
  uint32_t first;    // first column (instance-local permuted row)
  uint32_t ncols;    // s
  uint32_t nrows;    // m
  uint32_t rows_off; // first of the m row indices of this supernode in rows, and of its slots in U (global)
  uint64_t f_off;    // forward panel (float offset)
  uint64_t b_off;    // backward panel
  uint32_t vbase;    // first vertex (row) of the owning instance
  uint32_t inst;     // owning instance
};

// Per-step constants read from device memory so a captured graph stays valid
// when dt or the contact set-up change.
struct StepParams {
  float dt, inv_dt2;
  float gravity[3];
  float damping;
  float rayleigh;          // alpha_M
  int32_t ipc;             // step_with_ipc semantics
  // contact
  int32_t has_ground;
  float ground_h;
  int32_t has_sphere;
  float sphere_c[3];
  float sphere_r;
  int32_t self_collision;
  float kappa;
  float thickness;
  int32_t has_cyl;
  float cyl[4];            // center x, center z, top y, radius
  int32_t has_box;
  float box_lo[3], box_hi[3];
  float d_hat;             // effective (compliant) d_hat
  float max_vel;           // velocity clamp (0 = off)
  float al_tolerance, al_mu_growth, al_mu_initial;
  float friction, contact_damping, contact_damping_max, contact_vthresh;
  int32_t adaptive_damping;
};

// Per-instance device scalars of the IPC outer loop and reductions.
struct InstRed {
  double diff_sq, norm_sq;   // residual sums of the last solve
  double gdd;                // sum over free vertices of grad . d
  uint32_t toi_bits;         // min CCD time of impact (float bits, >= 0)
  uint32_t active;           // active contacts of the last detect
  uint32_t maxviol_bits;     // max violation (float bits)
  uint32_t al_done;
  float mu;
  float alpha;
  uint32_t last_active;      // active contacts of the last re-detect
  uint32_t al_iters;
  uint32_t iters;
  uint32_t pad;
};

struct BatchDev {
  const InstDev* inst;
  const int4* tri_chunks;
  const int4* hinge_chunks;
  const int4* vtx_chunks;
  // state
  float4* pos;
  float4* vel;
  float4* prev;
  float4* pred;
  const float* mass;       // solver lumped masses (pinned = 1e8)
  const uint8_t* pinned;
  // elements
  const uint4* tri_idx;    // global vertex ids
  const float4* tri_dm;
  const float* tri_w;
  float* tri_out;          // 9 floats per triangle: the three vertex contributions
  const uint4* hinge_idx;
  const float4* hinge_st;
  const float2* hinge_wr;  // (weight, rest angle)
  float4* hinge_out;       // w * s . (target - x)
  // vertex incidence, one CSR per connectivity class over the garment's local
  // vertex ids (InstDev::inc_ptr, tinc_off, hinc_off)
  const uint32_t* vtri_ptr;
  const uint32_t* vtri;    // (local triangle << 2) | slot
  const uint32_t* vhinge_ptr;
  const uint32_t* vhinge;  // (local hinge << 2) | slot
  // solve
  const uint32_t* perm_local;  // vertex -> instance-local permuted row
  const uint32_t* row_vertex;  // global row -> instance-local vertex
  float4* Y;               // solution of the sweeps, indexed by vbase + row
  float4* T;               // their right-hand side
  const SnDev* sn;
  const uint32_t* rows;        // below-diagonal rows of every supernode (instance-local)
  const float* vals;
  const uint32_t* pull_ptr;    // per supernode column, then row: its list in pull
  const uint32_t* pull;        // U slots of its children's rows there
  float4* U;                   // forward updates, one per (supernode, panel row)
  // FP64 refinement: the factored matrix A (f64, rows and columns in each
  // instance's solve order, global row ids), the right-hand side the first
  // sweep solved (R0) and the correction the refinement sweeps solve for (W).
  const uint32_t* a_ptr;
  const uint32_t* a_col;
  const double* a_val;
  float4* R0;
  float4* W;
  // contact / IPC
  float4* grad;            // barrier gradient of the detect at the start of the AL pass
  float4* grad_up;         // gradient of the re-detect
  double4* gacc;           // FP64 accumulator of the self-contact gradient of one detect
  float4* lam;             // AL multipliers
  float4* fin_n;           // final contact normal (ever in contact)
  uint8_t* in_contact;     // of the detect at the start of the AL pass
  uint8_t* in_contact_up;  // of the re-detect
  uint8_t* ever;
  InstRed* red;
  const StepParams* prm;
  uint32_t* status;        // bit 0: non-finite state
};

// ------------------------------------------------------------ math helpers
__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float len3(float3 a) { return sqrtf(dot3(a, a)); }

// double3 arithmetic for the FP64 local projection.
__device__ __forceinline__ double3 operator+(double3 a, double3 b) { return make_double3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ double3 operator-(double3 a, double3 b) { return make_double3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ double3 operator*(double3 a, double s) { return make_double3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ double dot3(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double3 d3(float4 a) { return make_double3(a.x, a.y, a.z); }

// 3x2 column-major matrix (mat3x2.rs:16) in FP64.
struct M32 { double3 c0, c1; };

__device__ __forceinline__ M32 mul2(const M32& f, double a, double b, double c, double d) {
  // f * [[a, c], [b, d]] (column-major [a, b, c, d], mat3x2.rs:62)
  M32 r;
  r.c0 = f.c0 * a + f.c1 * b;
  r.c1 = f.c0 * c + f.c1 * d;
  return r;
}

// polar_decomposition_3x2 (crates/vistio-math/src/decomposition.rs:76-138),
// through the eigen-decomposition of F^T F like the reference. It runs in
// FP64: its rounding grows as 1 / sigma_min^2 in compressed triangles, and in
// FP32 that error dominates a step's error wherever the sheet is pressed
// together. The thresholds are the reference's f32 constants.
struct PolarD {
  M32 rot;
  double s0, s1;
  double2 v0, v1;
};
__device__ __forceinline__ PolarD polar_dev(const M32& f) {
  double a = dot3(f.c0, f.c0), b = dot3(f.c0, f.c1), d = dot3(f.c1, f.c1);
  double ht = 0.5 * (a + d), hd = 0.5 * (a - d);
  double disc = sqrt(hd * hd + b * b);
  double l0 = fmax(ht + disc, 0.0), l1 = fmax(ht - disc, 0.0);
  double s0 = sqrt(l0), s1 = sqrt(l1);
  const double eps = double(1.0e-10f);
  PolarD p;
  if (s0 < eps) {
    p.rot.c0 = make_double3(1.0, 0.0, 0.0);
    p.rot.c1 = make_double3(0.0, 1.0, 0.0);
    p.s0 = p.s1 = 0.0;
    p.v0 = make_double2(1.0, 0.0);
    p.v1 = make_double2(0.0, 1.0);
    return p;
  }
  double2 v0, v1;
  if (fabs(b) > eps) {
    double vx = l0 - d, vy = b;
    double r = 1.0 / sqrt(vx * vx + vy * vy);
    v0 = make_double2(vx * r, vy * r);
    v1 = make_double2(-v0.y, v0.x);
  } else if (a >= d) {
    v0 = make_double2(1.0, 0.0); v1 = make_double2(0.0, 1.0);
  } else {
    v0 = make_double2(0.0, 1.0); v1 = make_double2(1.0, 0.0);
  }
  double is0 = 1.0 / s0, is1 = s1 > eps ? 1.0 / s1 : 0.0;
  double si00 = v0.x * v0.x * is0 + v1.x * v1.x * is1;
  double si01 = v0.x * v0.y * is0 + v1.x * v1.y * is1;
  double si11 = v0.y * v0.y * is0 + v1.y * v1.y * is1;
  p.rot = mul2(f, si00, si01, si01, si11);
  p.s0 = s0; p.s1 = s1; p.v0 = v0; p.v1 = v1;
  return p;
}

// Target deformation gradient of the membrane model
// (element.rs:127-174 and crates/vistio-material/src/*.rs).
__device__ __forceinline__ M32 model_target(int model, const M32& F, float warp_f, float weft_f) {
  if (model == 4) {  // IsotropicLinearModel: identity (isotropic.rs:42-57)
    M32 r; r.c0 = make_double3(1.0, 0.0, 0.0); r.c1 = make_double3(0.0, 1.0, 0.0); return r;
  }
  PolarD p = polar_dev(F);
  if (model == 0) return p.rot;  // ARAP: R
  const double warp = warp_f, weft = weft_f;
  double s0t, s1t;
  if (model == 1) {  // co-rotational, tension field: min(sigma, 1) (decomposition.rs:50-66)
    s0t = fmin(p.s0, 1.0); s1t = fmin(p.s1, 1.0);
  } else if (model == 2) {  // orthotropic (orthotropic.rs:51-79)
    double mk = fmax(fmax(warp, weft), double(1e-6f));
    double kw = warp / mk, kf = weft / mk;
    s0t = p.s0 + (1.0 - p.s0) * kw;
    s1t = p.s1 + (1.0 - p.s1) * kf;
  } else {  // anisotropic co-rotational (anisotropic.rs:78-143)
    double kw = fmin(fmax(warp, 0.0), 1.0), kf = fmin(fmax(weft, 0.0), 1.0);
    double cos2 = p.v0.x * p.v0.x, sin2 = p.v0.y * p.v0.y;
    double k0 = kw * cos2 + kf * sin2, k1 = kw * sin2 + kf * cos2;
    s0t = p.s0 > 1.0 ? 1.0 + (p.s0 - 1.0) * (1.0 - k0) : p.s0;
    s1t = p.s1 > 1.0 ? 1.0 + (p.s1 - 1.0) * (1.0 - k1) : p.s1;
  }
  double t00 = p.v0.x * p.v0.x * s0t + p.v1.x * p.v1.x * s1t;
  double t01 = p.v0.x * p.v0.y * s0t + p.v1.x * p.v1.y * s1t;
  double t11 = p.v0.y * p.v0.y * s0t + p.v1.y * p.v1.y * s1t;
  return mul2(p.rot, t00, t01, t01, t11);
}

// ------------------------------------------------------------- kernels
// Local membrane step of one triangle: w * g_k . (F_target - F) for k = 0..2.
// Compiled once (not inlined): the membrane kernels of both shapes run the
// same instructions, so the compiler's multiply-add contraction cannot differ
// between them and their results are bit-identical.
__device__ __noinline__ void tri_project_one(float* __restrict__ tri_out, int32_t model, float warp, float weft,
                                             uint32_t t, float4 dm, float w, float4 q0, float4 q1, float4 q2) {
  // FP64 from the FP32 positions on (the projection is the ill-conditioned
  // part; the outputs are rounded once).
  const double3 p0 = d3(q0), p1 = d3(q1), p2 = d3(q2);
  M32 ds; ds.c0 = p1 - p0; ds.c1 = p2 - p0;
  M32 F = mul2(ds, dm.x, dm.y, dm.z, dm.w);
  float det = dm.x * dm.w - dm.y * dm.z;
  double3 d0 = make_double3(0.0, 0.0, 0.0), d1 = d0;
  if (fabsf(det) > 1e-12f) {  // element.rs:192-202: degenerate rest shape keeps p
    M32 Ft = model_target(model, F, warp, weft);
    d0 = (Ft.c0 - F.c0) * double(w);
    d1 = (Ft.c1 - F.c1) * double(w);
  }
  // g = [[-(a+b), -(c+d)], [a, c], [b, d]] (assembly.rs:77-81)
  const double g00 = -(double(dm.x) + double(dm.y)), g01 = -(double(dm.z) + double(dm.w));
  const double3 c0 = d0 * g00 + d1 * g01;
  const double3 c1 = d0 * double(dm.x) + d1 * double(dm.z);
  const double3 c2 = d0 * double(dm.y) + d1 * double(dm.w);
  float* o = tri_out + 9ull * t;
  o[0] = float(c0.x); o[1] = float(c0.y); o[2] = float(c0.z);
  o[3] = float(c1.x); o[4] = float(c1.y); o[5] = float(c1.z);
  o[6] = float(c2.x); o[7] = float(c2.y); o[8] = float(c2.z);
}
__device__ __forceinline__ void tri_project(const BatchDev& B, const InstDev& I, uint32_t t, float4 dm, float w,
                                            float4 q0, float4 q1, float4 q2) {
  tri_project_one(B.tri_out, I.model, I.warp, I.weft, t, dm, w, q0, q1, q2);
}

// The membrane step over a chunk of up to 256 triangles with 128 threads:
// each thread loads both of its triangles (indices, rest data, the six
// vertex positions) before it projects either, so twice the loads are in
// flight per warp; eight blocks per SM (64 registers). The loads are
// latency-bound: 0.216 -> 0.176 ms per iteration on 7.9 M triangles against
// one triangle per thread at five 256-thread blocks per SM.
constexpr int kTriThreads = 128;
__global__ void __launch_bounds__(kTriThreads, 8) k_tri(BatchDev B) {
  pdl_begin();
  int4 ch = B.tri_chunks[blockIdx.x];
  const uint32_t i0 = threadIdx.x, i1 = threadIdx.x + kTriThreads;
  if ((int)i0 >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const bool two = (int)i1 < ch.z;
  const uint32_t t0 = uint32_t(ch.y) + i0, t1 = uint32_t(ch.y) + i1;
  const InstDev I = B.inst[ch.x];
  const uint4 a = B.tri_idx[t0], b = two ? B.tri_idx[t1] : a;
  const float4 dma = B.tri_dm[t0], dmb = two ? B.tri_dm[t1] : dma;
  const float wa = B.tri_w[t0], wb = two ? B.tri_w[t1] : wa;
  const float4 qa0 = B.pos[a.x], qa1 = B.pos[a.y], qa2 = B.pos[a.z];
  float4 qb0 = qa0, qb1 = qa1, qb2 = qa2;
  if (two) { qb0 = B.pos[b.x]; qb1 = B.pos[b.y]; qb2 = B.pos[b.z]; }
  tri_project(B, I, t0, dma, wa, qa0, qa1, qa2);
  if (two) tri_project(B, I, t1, dmb, wb, qb0, qb1, qb2);
}

// The same membrane step with one triangle per thread (a chunk of up to 256
// triangles on 256 threads, four blocks per SM): the autotuner's other shape.
__global__ void __launch_bounds__(256, 4) k_tri1(BatchDev B) {
  pdl_begin();
  int4 ch = B.tri_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const uint32_t t = uint32_t(ch.y) + threadIdx.x;
  const InstDev I = B.inst[ch.x];
  const uint4 a = B.tri_idx[t];
  tri_project(B, I, t, B.tri_dm[t], B.tri_w[t], B.pos[a.x], B.pos[a.y], B.pos[a.z]);
}

// Rotation of v = p - centre about `axis` by an angle minus v itself:
// (axis (axis . v) - v)(1 - cos) + (axis x v) sin (bending.rs:231-239), given
// sin and 1 - cos. The two wings turn by +half and -half: the same 1 - cos and
// opposite sines, so one pair of sines serves both.
__device__ __forceinline__ float3 rot_delta(float3 v, float3 axis, float s, float omc) {
  float dt = dot3(axis, v);
  return (axis * dt - v) * omc + cross3(axis, v) * s;
}

// Local bending step of one hinge: w * s . (target - x); only the wings move
// (bending.rs:182-227, discrete_shells.rs:285-337). Compiled once (not
// inlined), so both bending kernels' shapes give bit-identical results.
__device__ __noinline__ float4 hinge_project(float4 st, float2 wr, float3 p0, float3 p1, float3 pa, float3 pb) {
  float3 out = make_float3(0.f, 0.f, 0.f);
  float3 e = p1 - p0;
  float el = len3(e);
  if (el >= 1e-10f) {
    float3 ed = e * (1.f / el);
    float3 ta = pa - p0, tb = pb - p0;
    float3 qa = ta - ed * dot3(ta, ed), qb = tb - ed * dot3(tb, ed);
    float la = len3(qa), lb = len3(qb);
    const float PI = 3.14159265358979323846f;
    float ang = PI;
    if (la >= 1e-10f && lb >= 1e-10f) {
      float c = dot3(qa * (1.f / la), qb * (1.f / lb));
      ang = acosf(fminf(fmaxf(c, -1.f), 1.f));
    }
    float diff = ang - wr.y;
    if (fabsf(diff) >= 1e-8f) {
      float sign = dot3(cross3(qa, qb), ed) >= 0.f ? 1.f : -1.f;
      float half = diff * 0.5f * sign;
      float3 mid = (p0 + p1) * 0.5f;
      const float s = sinf(half), hq = sinf(0.5f * half);
      const float omc = 2.f * hq * hq;  // 1 - cos, without cancellation
      float3 da = rot_delta(pa - mid, ed, s, omc);
      float3 db = rot_delta(pb - mid, ed, -s, omc);
      out = (da * st.z + db * st.w) * wr.x;
    }
  }
  return make_float4(out.x, out.y, out.z, 0.f);
}

// One hinge per thread over a chunk of up to 256 hinges. A garment whose
// stencils are all (-1, -1, 1, 1) skips their load (16 B per hinge), with the
// same products.
__global__ void __launch_bounds__(256) k_hinge(BatchDev B) {
  pdl_begin();
  int4 ch = B.hinge_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  uint32_t h = uint32_t(ch.y) + threadIdx.x;
  uint4 id = B.hinge_idx[h];
  const float4 st = B.inst[ch.x].unit_stencils ? make_float4(-1.f, -1.f, 1.f, 1.f) : B.hinge_st[h];
  float2 wr = B.hinge_wr[h];
  B.hinge_out[h] = hinge_project(st, wr, f3(B.pos[id.x]), f3(B.pos[id.y]), f3(B.pos[id.z]), f3(B.pos[id.w]));
}

// Two hinges per thread (128 threads over a chunk of up to 256), both hinges'
// loads issued before either projection: the autotuner's other shape.
__global__ void __launch_bounds__(128, 8) k_hinge2(BatchDev B) {
  pdl_begin();
  int4 ch = B.hinge_chunks[blockIdx.x];
  const uint32_t i0 = threadIdx.x, i1 = threadIdx.x + 128;
  if ((int)i0 >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const bool two = (int)i1 < ch.z;
  const uint32_t h0 = uint32_t(ch.y) + i0, h1 = two ? uint32_t(ch.y) + i1 : h0;
  const bool unit = B.inst[ch.x].unit_stencils != 0;
  const uint4 a = B.hinge_idx[h0], b = B.hinge_idx[h1];
  const float4 sa = unit ? make_float4(-1.f, -1.f, 1.f, 1.f) : B.hinge_st[h0];
  const float4 sb = unit ? make_float4(-1.f, -1.f, 1.f, 1.f) : B.hinge_st[h1];
  const float2 wa = B.hinge_wr[h0], wb = B.hinge_wr[h1];
  const float3 a0 = f3(B.pos[a.x]), a1 = f3(B.pos[a.y]), a2 = f3(B.pos[a.z]), a3 = f3(B.pos[a.w]);
  const float3 b0 = f3(B.pos[b.x]), b1 = f3(B.pos[b.y]), b2 = f3(B.pos[b.z]), b3 = f3(B.pos[b.w]);
  B.hinge_out[h0] = hinge_project(sa, wa, a0, a1, a2, a3);
  if (two) B.hinge_out[h1] = hinge_project(sb, wb, b0, b1, b2, b3);
}

// Both local steps of a small batch in one launch: blocks [0, ntri) one chunk
// of triangles, the rest one chunk of hinges, one element per thread. A small
// batch's iteration is a chain of launches of 2 to 3 us each, whatever they do
// (sheet 20x20: 10 launches, 29 us); large ones keep a kernel each, in the
// shapes the autotuner times.
__global__ void __launch_bounds__(256, 4) k_local(BatchDev B, uint32_t ntri) {
  pdl_begin();
  const bool tri = blockIdx.x < ntri;
  const int4 ch = tri ? B.tri_chunks[blockIdx.x] : B.hinge_chunks[blockIdx.x - ntri];
  if ((int)threadIdx.x >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const uint32_t e = uint32_t(ch.y) + threadIdx.x;
  if (tri) {
    const InstDev I = B.inst[ch.x];
    const uint4 a = B.tri_idx[e];
    tri_project(B, I, e, B.tri_dm[e], B.tri_w[e], B.pos[a.x], B.pos[a.y], B.pos[a.z]);
  } else {
    const uint4 id = B.hinge_idx[e];
    const float4 st = B.inst[ch.x].unit_stencils ? make_float4(-1.f, -1.f, 1.f, 1.f) : B.hinge_st[e];
    B.hinge_out[e] = hinge_project(st, B.hinge_wr[e], f3(B.pos[id.x]), f3(B.pos[id.y]), f3(B.pos[id.z]), f3(B.pos[id.w]));
  }
}

__device__ __forceinline__ void red_reset(InstRed& R) {
  R.diff_sq = 0.0;
  R.norm_sq = 0.0;
  R.toi_bits = __float_as_uint(1.0f);
  R.gdd = 0.0;
}

// Residual gather: r_i = m_i (pred_i / dt^2 - x_i / h^2) + sum of element
// terms [- (mu grad_i + lambda_i)], written in solve (permuted) order.
// keep_rhs also stores r in R0 for a refinement of this iteration's solve. A
// garment's first block counts the iteration and clears the sums of its solve
// (their readers in the last iteration are done).
__global__ void __launch_bounds__(256) k_gather(BatchDev B, int keep_rhs) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  const InstDev I = B.inst[ch.x];
  uint32_t g = uint32_t(ch.y) + threadIdx.x;
  const StepParams& P = *B.prm;
  InstRed& R = B.red[ch.x];
  if (P.ipc && R.al_done) return;
  if (g == I.vbase) {
    red_reset(R);
    R.iters += 1;
  }
  float m = B.mass[g];
  float3 x = f3(B.pos[g]), q = f3(B.pred[g]);
  float cm = m * I.inv_hmat2, cr = m * P.inv_dt2;
  float3 r = (q - x) * cm + q * (cr - cm);
  // element outputs are read-only here: non-coherent loads, and of a hinge's
  // stencil only this vertex's weight (gather 0.313 -> 0.278 ms per iteration),
  // none where every stencil is (-1, -1, 1, 1): -1 for the edge's ends, 1 for
  // the wings, the same products as the loaded weights
  // the garment's connectivity class's lists (shared by the garments of one
  // mesh topology: read once for all of them, from L2 after the first).
  // Loading the first eight incidences' codes and contributions ahead of the
  // adds was measured slower (62 registers, half the resident warps: 0.264
  // against 0.224 ms per iteration on 512 sheets).
  const uint32_t l = g - I.vbase;
  const uint32_t* tcode = B.vtri + I.tinc_off;
  const uint32_t* hcode = B.vhinge + I.hinc_off;
#pragma unroll 4
  for (uint32_t e = __ldg(B.vtri_ptr + I.inc_ptr + l), ee = __ldg(B.vtri_ptr + I.inc_ptr + l + 1); e < ee; ++e) {
    uint32_t code = __ldg(tcode + e);
    const float* o = B.tri_out + 9ull * (I.tbase + (code >> 2)) + 3 * (code & 3u);
    r.x += __ldg(o); r.y += __ldg(o + 1); r.z += __ldg(o + 2);
  }
#pragma unroll 4
  for (uint32_t e = __ldg(B.vhinge_ptr + I.inc_ptr + l), ee = __ldg(B.vhinge_ptr + I.inc_ptr + l + 1); e < ee; ++e) {
    uint32_t code = __ldg(hcode + e);
    uint32_t h = I.hbase + (code >> 2), k = code & 3u;
    float s = I.unit_stencils ? (k < 2u ? -1.f : 1.f) : __ldg(reinterpret_cast<const float*>(B.hinge_st + h) + k);
    float4 o = __ldg(B.hinge_out + h);
    r.x += s * o.x; r.y += s * o.y; r.z += s * o.z;
  }
  if (P.ipc) {  // assemble_barrier_rhs (assembly.rs:272-282)
    float mu = R.mu;
    float4 gr = B.grad[g], la = B.lam[g];
    r.x -= mu * gr.x + la.x; r.y -= mu * gr.y + la.y; r.z -= mu * gr.z + la.z;
  }
  const uint32_t row = I.vbase + B.perm_local[g];
  B.T[row] = make_float4(r.x, r.y, r.z, 0.f);
  if (keep_rhs) B.R0[row] = make_float4(r.x, r.y, r.z, 0.f);
}

__device__ __forceinline__ void f4_fma(float4& t, float a, float4 y) {
  t.x += a * y.x; t.y += a * y.y; t.z += a * y.z;
}
__device__ __forceinline__ float4 f4_sub(float4 a, float4 b) {
  return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, 0.f);
}
__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, 0.f);
}

// Clears the per-instance residual sums before a solve of its own (without a gather).
__global__ void k_red_reset(BatchDev B, uint32_t ninst) {
  pdl_begin();
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ninst) return;
  InstRed& R = B.red[k];
  if (B.prm->ipc && R.al_done) return;
  red_reset(R);
}

// Iterative refinement of the global solve: T = R0 - A d in FP64, with d the
// sweeps' FP32 solution in Y and A the f64 matrix that was factored. Each
// instance's rows are numbered like its vertices, so the vertex chunks cover
// them. The sweeps then solve A W = T and d + W replaces d.
__global__ void __launch_bounds__(256) k_refine(BatchDev B) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const uint32_t p = uint32_t(ch.y) + threadIdx.x;
  double ax = 0.0, ay = 0.0, az = 0.0;
  for (uint32_t q = B.a_ptr[p], qe = B.a_ptr[p + 1]; q < qe; ++q) {
    const double a = B.a_val[q];
    const float4 d = B.Y[B.a_col[q]];
    ax += a * d.x; ay += a * d.y; az += a * d.z;
  }
  const float4 r = B.R0[p];
  B.T[p] = make_float4(float(double(r.x) - ax), float(double(r.y) - ay), float(double(r.z) - az), 0.f);
}

// d <- d + e between two refinement sweeps.
__global__ void __launch_bounds__(256) k_accum(BatchDev B) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  if (B.prm->ipc && B.red[ch.x].al_done) return;
  const uint32_t p = uint32_t(ch.y) + threadIdx.x;
  B.Y[p] = f4_add(B.Y[p], B.W[p]);
}

// After the sweeps of a plain step: residual sums (pd_solver.rs:403-421) and, with
// do_update, x <- x + d, the pin reset (:429-435) and the ground clamp (:438).
// add_w folds the last refinement correction into d.
__device__ __forceinline__ void update_one(const BatchDev& B, const InstDev& I, uint32_t g, float4 d, float4 x,
                                           int do_update, int add_w, uint32_t row, double& dsq, double& nsq,
                                           bool& bad) {
  if (add_w) d = f4_add(d, B.W[row]);
  dsq += double(d.x) * d.x + double(d.y) * d.y + double(d.z) * d.z;
  nsq += double(x.x) * x.x + double(x.y) * x.y + double(x.z) * x.z;
  bad = bad || !(isfinite(d.x) && isfinite(d.y) && isfinite(d.z));
  if (do_update) {
    float4 nx;
    if (B.pinned[g]) nx = B.prev[g];
    else {
      nx = make_float4(x.x + d.x, x.y + d.y, x.z + d.z, 0.f);
      if (I.has_ground && nx.y < I.ground_h) nx.y = I.ground_h;  // state.rs:180-189
    }
    B.pos[g] = nx;
  }
}

// Two vertices per thread (128 threads over a chunk of up to 256), both
// vertices' loads issued before either update: 0.063 -> about 0.043 ms per
// iteration on 4.05 M vertices (the solve phase 1.315 -> 1.295 ms).
__global__ void __launch_bounds__(128) k_update(BatchDev B, int do_update, int add_w) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  const InstDev I = B.inst[ch.x];
  InstRed& R = B.red[ch.x];
  if (B.prm->ipc && R.al_done) return;
  double dsq = 0.0, nsq = 0.0;
  bool bad = false;
  const uint32_t i0 = threadIdx.x, i1 = threadIdx.x + 128;
  if ((int)i0 < ch.z) {
    const bool two = (int)i1 < ch.z;
    const uint32_t g0 = uint32_t(ch.y) + i0, g1 = uint32_t(ch.y) + i1;
    const uint32_t r0 = I.vbase + B.perm_local[g0], r1 = two ? I.vbase + B.perm_local[g1] : r0;
    const float4 d0 = B.Y[r0], d1 = two ? B.Y[r1] : d0;
    const float4 x0 = B.pos[g0], x1 = two ? B.pos[g1] : x0;
    update_one(B, I, g0, d0, x0, do_update, add_w, r0, dsq, nsq, bad);
    if (two) update_one(B, I, g1, d1, x1, do_update, add_w, r1, dsq, nsq, bad);
  }
  for (int o = 16; o > 0; o >>= 1) {
    dsq += __shfl_down_sync(0xffffffffu, dsq, o);
    nsq += __shfl_down_sync(0xffffffffu, nsq, o);
  }
  if (bad) atomicOr(B.status, 1u);
  if ((threadIdx.x & 31) == 0 && (dsq != 0.0 || nsq != 0.0)) {
    atomicAdd(&R.diff_sq, dsq);
    atomicAdd(&R.norm_sq, nsq);
  }
}

// Whole-batch positions between interleaved xyz (the host layout, one
// contiguous copy) and the float4 state rows.
__global__ void __launch_bounds__(256) k_unpack_pos(float4* pos, const float* __restrict__ xyz, uint64_t n) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    float4 p = pos[i];
    p.x = xyz[3 * i]; p.y = xyz[3 * i + 1]; p.z = xyz[3 * i + 2];
    pos[i] = p;
  }
}
__global__ void __launch_bounds__(256) k_pack_pos(float* __restrict__ xyz, const float4* pos, uint64_t n) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const float4 p = pos[i];
    xyz[3 * i] = p.x; xyz[3 * i + 1] = p.y; xyz[3 * i + 2] = p.z;
  }
}

// save_previous + (IPC) velocity clamp + predict + x <- pred (state.rs:145-169,
// pd_solver.rs:273-283 and 566-603).
__global__ void __launch_bounds__(256) k_predict(BatchDev B) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  const InstDev I = B.inst[ch.x];
  const StepParams& P = *B.prm;
  if (threadIdx.x == 0 && ch.y == int(I.vbase)) {
    InstRed& R = B.red[ch.x];
    R.iters = 0;
    R.al_iters = 0;
    R.al_done = 0;
    R.mu = P.al_mu_initial;
    R.last_active = 0;
    R.alpha = 1.f;
  }
  if ((int)threadIdx.x >= ch.z) return;
  uint32_t g = uint32_t(ch.y) + threadIdx.x;
  float4 x = B.pos[g];
  float4 v = B.vel[g];
  B.prev[g] = x;
  bool pin = B.pinned[g] != 0;
  bool ground = P.ipc ? P.has_ground : I.has_ground;
  float gh = P.ipc ? P.ground_h : I.ground_h;
  if (P.ipc) {
    if (!pin && P.max_vel > 0.f) {
      float vsq = v.x * v.x + v.y * v.y + v.z * v.z;
      if (vsq > P.max_vel * P.max_vel) {
        float sc = P.max_vel / sqrtf(vsq);
        v.x *= sc; v.y *= sc; v.z *= sc;
        B.vel[g] = v;
      }
    }
    B.ever[g] = 0;
    B.fin_n[g] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 q = x;
  if (!pin) {
    float dt = P.dt, dt2 = dt * dt;
    q.x = x.x + dt * v.x + dt2 * P.gravity[0];
    q.y = x.y + dt * v.y + dt2 * P.gravity[1];
    q.z = x.z + dt * v.z + dt2 * P.gravity[2];
    if (ground && q.y < gh) q.y = gh;
  }
  B.pred[g] = q;
  B.pos[g] = q;
}

// update_velocities, (IPC) inelastic velocity filter, ground velocities,
// damping and Rayleigh damping (pd_solver.rs:447-466 and 1027-1147).
__global__ void __launch_bounds__(256) k_finalize(BatchDev B) {
  pdl_begin();
  int4 ch = B.vtx_chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.z) return;
  const InstDev I = B.inst[ch.x];
  const StepParams& P = *B.prm;
  uint32_t g = uint32_t(ch.y) + threadIdx.x;
  float4 x = B.pos[g], pv = B.prev[g];
  float inv_dt = 1.f / P.dt;
  float3 v = make_float3((x.x - pv.x) * inv_dt, (x.y - pv.y) * inv_dt, (x.z - pv.z) * inv_dt);
  bool pin = B.pinned[g] != 0;
  bool ground = P.ipc ? P.has_ground : I.has_ground;
  float gh = P.ipc ? P.ground_h : I.ground_h;
  if (P.ipc) {
    const InstRed& R = B.red[ch.x];
    if (!pin && B.ever[g]) {
      float4 n4 = B.fin_n[g];
      float3 n = f3(n4);
      if (dot3(n, n) >= 0.5f) {
        float vdn = dot3(v, n);
        v = v - n * vdn;
        float vn = fabsf(vdn);
        float vt = len3(v);
        if (vt > 1e-8f) {
          float fi = P.friction * vn;
          if (fi >= vt) v = make_float3(0.f, 0.f, 0.f);
          else v = v * (1.f - fi / vt);
        }
        float cd = P.contact_damping;
        if (P.adaptive_damping) {
          float vm = len3(v);
          float tt = fminf(fmaxf(1.f - vm / fmaxf(P.contact_vthresh, 1e-6f), 0.f), 1.f);
          float ad = cd + tt * (P.contact_damping_max - cd);
          v = v * (1.f - ad);
        } else {
          v = v * (1.f - cd);
        }
      }
    }
    if (R.last_active > 0) v = v * (1.f - 0.05f);
  }
  if (ground && !pin && x.y <= gh) {  // state.rs:195-213
    if (v.y < 0.f) v.y = 0.f;
    pv.y = gh;
    B.prev[g] = pv;
    v.x *= 0.5f; v.z *= 0.5f;
  }
  v = v * (1.f - P.damping);
  if (P.rayleigh > 0.f && !pin) v = v * (1.f / (1.f + P.rayleigh * P.dt));
  B.vel[g] = make_float4(v.x, v.y, v.z, 0.f);
}

}  // namespace vistio
