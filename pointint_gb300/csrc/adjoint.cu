// Adjoint of the Fourier intersection volume: gradients of L = sum_ij C_ij V_ij.
//
// dL/dtheta_n = (1/8 pi^3) sum_q w_q Re( dA_n(k_q)/dtheta_n  conj(B_n(k_q)) ),
// B_n = sum_j W_nj A_j  (the cotangent).  For L = sum_ij C_ij V_ij, W = C + C^T;
// W = e_j 1^T-style single columns give the reference's per-pair gradients
// dV_ij/dtheta_i (B_i = A_j for every i).
//
// Replaces the reference's gradient kernels K4-K6, K8, K10 and K15
// (cpp/src/dof/cuda/affine_dof_cuda.cu:254-576, 693-849;
//  cpp/src/dof/cuda/triangle_mesh_dof_cuda.cu:147-310;
//  cpp/src/compute_intersection_volume.cu:60-101;
//  cpp/src/compute_intersection_volume_multi_object.cu:124-176), which
// materialised dA/dtheta for every k-node (Q x 3V complex doubles for a mesh:
// ~9.5 GB for an icosphere-4 at N_k = 76,928) and reduced it with FP64
// atomics.  Here nothing of size Q x (parameters) exists:
//
//  * cotangent_kernel: forms B^ = W J^ on the sqrt|w|-scaled J (one pass over J)
//    and folds each direction's antipode into it, with the object's origin phase and
//    the quadrature weights, so that one direction of a pair is evaluated;
//  * adj_surf_kernel / adj_tri_kernel: one thread per element; the CTA's
//    elements share one object, so the cotangent of a tile of directions is
//    staged once in shared memory and read as broadcasts.  The small radii enter
//    through sums that a patch of 32 elements shares (beta, below); at the others every
//    thread recomputes its element's form factor and derivatives.  The element's
//    parameter gradient is accumulated in registers, every direction's contribution
//    compensated;
//  * chain kernels turn element gradients into AffineDoF gradients (fixed
//    order FP64 block reduction per object) or TriangleMeshDoF vertex
//    gradients (CSR gather per vertex, no atomics): results are bitwise
//    reproducible.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <vector>
#include "pi_internal.h"
#include "dfmath.cuh"
#include "bessel.cuh"
#include "moments.h"
#include "tri_adjoint.cuh"

namespace pi {

namespace {

constexpr int ADJ_THREADS = 128;
constexpr int ADJ_DT = 8;        // directions staged per shared-memory tile
constexpr int ADJ_LMAX = 256;    // radii per direction held in shared memory
// one copy of the phasor table: the lanes of a warp hold neighbouring elements
// at one direction and radius, whose phases mostly share an entry (a broadcast);
// eight copies, one a lane group, took 7% longer (4.43 against 4.13 ms for 24 bodies)
constexpr int ADJ_COPIES = 1;
constexpr double INV8PI3 = 1.0 / (8.0 * 3.14159265358979323846 * 3.14159265358979323846 * 3.14159265358979323846);

// Kahan-compensated FP32 accumulator.
struct kf {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

// The cotangent of every object, folded for the adjoint kernels: with
// B_n = sum_j W_nj J^_j at the evaluated direction j and its antipode j'
// (KGridDev::dpair),
//   Bt[n][r][e] = s B_n(k_r d_j) e^{-ik.o} - conj(s' B_n(-k_r d_j) e^{ik.o}),
// s = sign(w) sqrt|w| of the node, o the object's origin (zero at k = 0, where
// A = 0 by definition).  A direction's antipode contributes
// Re(conj(B') dA(-k)) with dA(-k) = -conj dA(k) for every real parameter,
// which is Re(conj(-conj B') dA(k)), so it is never evaluated itself.
// Grid (nodes of the evaluated directions, blocks of COT_N objects); one pass
// over J per block.
constexpr int COT_N = 16;
__global__ void __launch_bounds__(256)
cotangent_kernel(KGridDev kg, BatchDev b, const float2* __restrict__ Jw, const float* __restrict__ Cs,
                 float2* __restrict__ Bt) {
  __shared__ float cs[COT_N][64];
  const int n = b.n_obj;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = t < (int64_t)kg.Me * kg.L;
  const int r = in ? (int)(t / kg.Me) : 0, e = in ? (int)(t - (int64_t)r * kg.Me) : 0;
  const int2 jp = in ? kg.dpair[e] : make_int2(0, -1);
  const int64_t q = (int64_t)r * kg.M + jp.x, qm = (int64_t)r * kg.M + max(jp.y, 0);
  const int n0 = blockIdx.y * COT_N;
  float2 acc[COT_N], accm[COT_N];
#pragma unroll
  for (int a = 0; a < COT_N; ++a) acc[a] = accm[a] = make_float2(0.f, 0.f);
  for (int j0 = 0; j0 < n; j0 += 64) {
    __syncthreads();
    for (int i = threadIdx.x; i < COT_N * 64; i += blockDim.x) {
      const int a = i / 64, jj = i % 64;
      cs[a][jj] = (n0 + a < n && j0 + jj < n) ? Cs[(int64_t)(n0 + a) * n + j0 + jj] : 0.f;
    }
    __syncthreads();
    if (!in) continue;
    const int jn = min(64, n - j0);
    for (int jj = 0; jj < jn; ++jj) {
      const float2 v = Jw[(int64_t)(j0 + jj) * kg.Q + q], vm = Jw[(int64_t)(j0 + jj) * kg.Q + qm];
#pragma unroll
      for (int a = 0; a < COT_N; ++a) {
        const float w = cs[a][jj];
        acc[a].x = fmaf(w, v.x, acc[a].x);
        acc[a].y = fmaf(w, v.y, acc[a].y);
        accm[a].x = fmaf(w, vm.x, accm[a].x);
        accm[a].y = fmaf(w, vm.y, accm[a].y);
      }
    }
  }
  if (!in) return;
  const float4 h = kg.dir_hi[jp.x], l = kg.dir_lo[jp.x];
  const float2 km = kg.kmag[r];
  const bool zero = !(km.x * l.w >= 1e-10f);
  const float s = kg.sqrtw[q] * (kg.sign ? kg.sign[q] : 1.f);
  const float sm = jp.y >= 0 ? kg.sqrtw[qm] * (kg.sign ? kg.sign[qm] : 1.f) : 0.f;
#pragma unroll
  for (int a = 0; a < COT_N; ++a) {
    if (n0 + a >= n) break;
    const double* o = b.objs[n0 + a].origin;
    const double so = ((double)h.x + l.x) * o[0] + ((double)h.y + l.y) * o[1] + ((double)h.z + l.z) * o[2];
    const cf p = cis_f64(((double)km.x + (double)km.y) * so);  // e^{ik.o}
    const float2 u = acc[a], um = jp.y >= 0 ? accm[a] : make_float2(0.f, 0.f);
    float2 v = make_float2(s * (u.x * p.re + u.y * p.im) - sm * (um.x * p.re - um.y * p.im),
                           s * (u.y * p.re - u.x * p.im) + sm * (um.y * p.re + um.x * p.im));
    if (zero) v = make_float2(0.f, 0.f);
    Bt[((int64_t)(n0 + a) * kg.L + r) * kg.Me + e] = v;
  }
}

struct AdjWork { int32_t obj, first; };

// A CTA's elements are ADJ_THREADS consecutive pool entries of one object:
// whole patches, whose radii [0, nr) with k rho below the bound enter through
// the patch's expansion (moments.cu).  The cotangent of a direction then
// becomes, for each patch (centre c, k in units of 1/s),
//   beta_m = Re( i^m sum_r conj(Bt_r) e^{i k_r d.c} k_r^m ),   m < ADJ_TERMS,
// 16 real numbers that all its elements share, and an element's contribution
// and its derivatives are sums of beta_m times the moments of moments.cu and
// their derivatives: ~150 FP32 operations per element and direction for all
// those radii instead of ~70 for each.  (24 bodies, N_k = 76,928: adj_tri_kernel
// 13.7 -> 3.80 ms; eight clouds of 50,000 disks: adj_surf_kernel 43.8 -> 8.46.)
constexpr int ADJ_TERMS = MOMENT_TERMS;
// Patches of half a cluster (a warp's elements): the expansions reach 1.4 times
// the k.  A quarter reaches twice the k but its betas, every covered radius for
// every patch and direction, cost more than the radii they save (eight clouds
// 10.2 ms, 24 bodies 4.21).
constexpr int ADJ_PATCH = PI_CLUSTER / 2;
constexpr int ADJ_CL = ADJ_THREADS / ADJ_PATCH;  // patches per CTA
static_assert(ADJ_PATCH % PI_LEAF == 0 && 4 * ADJ_CL * ADJ_DT == ADJ_THREADS, "four threads per patch and direction");
static_assert(ADJ_TERMS == 16, "eight orders per thread");
// Bounds on k rho: the derivatives drop one (centres, vertices) or two (normals)
// orders earlier than the values.  What is dropped, relative to the leading
// term, of a small element on the rim seen along its offset (x^15 / 15!, x^14 /
// 14! and the terms after them) stays below one FP32 rounding: 6.0e-8
// (triangles' vertex derivatives at 2.1), 4.9e-8 (surfels' normal ones at 1.8).
constexpr float ADJ_X_TRI = 2.1f, ADJ_X_SURF = 1.8f;

// Sums over the expansion of one element (scaled units).
struct SurfSums { float F, Fs, Fp; };            // F, dF/dsigma, dF/dp^2
struct TriSums { float F, Fb, Fc, Fsum; };       // t0, its derivatives by b, c and their sum with a's

// Coefficients of the surfels' recurrences, nu = 1 (2 J1(x)/x), 2 (8 J2(x)/x^2)
// or 0 (Gaussian): u_m = lambda_m w_m, w_{m+1} = sigma w_m + K_m q w_{m-1}.
template <int NU>
struct AdjConst {
  float lambda[ADJ_TERMS], K[ADJ_TERMS];
  constexpr AdjConst() : lambda(), K() {
    double g = 1.0, prev = 1.0;
    for (int m = 0; m < ADJ_TERMS; ++m) {
      const double alpha = NU ? (2.0 * m + 2 * NU + 1) / ((m + 1.0) * (m + 2 * NU + 1)) : 1.0 / (m + 1.0);
      const double beta = NU ? 1.0 / ((m + 1.0) * (m + 2 * NU + 1)) : 1.0 / (m + 1.0);
      lambda[m] = (float)g;
      K[m] = m == 0 ? 0.f : (float)(beta / (alpha * prev));
      g *= alpha;
      prev = alpha;
    }
  }
};

__device__ __forceinline__ SurfSums disk_adjoint(const float* be, float sg, float p2) {
  constexpr AdjConst<1> C1{};
  constexpr AdjConst<2> C2{};
  const float q = fmaf(-sg, sg, p2);
  SurfSums f{0.f, 0.f, 0.f};
  float u0 = 0.f, u1 = 1.f, v0 = 0.f, v1 = 1.f;
#pragma unroll
  for (int m = 0; m < ADJ_TERMS; ++m) {
    const float u = C1.lambda[m] * u1;
    f.F = fmaf(be[m], u, f.F);
    if (m + 1 < ADJ_TERMS) f.Fs = fmaf(be[m + 1], u, f.Fs);
    if (m + 2 < ADJ_TERMS) f.Fp = fmaf(be[m + 2], (0.125f * C2.lambda[m]) * v1, f.Fp);
    const float u2 = fmaf(sg, u1, (C1.K[m] * q) * u0), v2 = fmaf(sg, v1, (C2.K[m] * q) * v0);
    u0 = u1; u1 = u2;
    v0 = v1; v1 = v2;
  }
  return f;
}

__device__ __forceinline__ SurfSums gauss_adjoint(const float* be, float sg, float q) {
  constexpr AdjConst<0> C{};
  SurfSums f{0.f, 0.f, 0.f};
  float u0 = 0.f, u1 = 1.f;
#pragma unroll
  for (int m = 0; m < ADJ_TERMS; ++m) {
    const float u = C.lambda[m] * u1;
    f.F = fmaf(be[m], u, f.F);
    if (m + 1 < ADJ_TERMS) f.Fs = fmaf(be[m + 1], u, f.Fs);
    if (m + 2 < ADJ_TERMS) f.Fp = fmaf(be[m + 2], 0.5f * u, f.Fp);
    const float u2 = fmaf(sg, u1, (C.K[m] * q) * u0);
    u0 = u1; u1 = u2;
  }
  return f;
}

__device__ __forceinline__ TriSums tri_adjoint(const float* be, float a, float b, float c) {
  constexpr FmConst<PI_GEOM_TRIANGLE> C{};  // 2/(n+2)!
  TriSums f{0.f, 0.f, 0.f, 0.f};
  float an = 1.f, qn = 1.f, hn = 1.f, hb = 1.f, hc = 1.f;
#pragma unroll
  for (int n = 0; n < ADJ_TERMS; ++n) {
    if (n > 0) {
      an *= a;
      qn = fmaf(b, qn, an);
      hn = fmaf(c, hn, qn);
    }
    f.F = fmaf(be[n] * (-0.5f * C.f[n]), hn, f.F);
    if (n + 1 < ADJ_TERMS) {
      if (n > 0) {
        hb = fmaf(b, hb, hn);
        hc = fmaf(c, hc, hn);
      }
      const float w = be[n + 1] * (-0.5f * C.f[n + 1]);
      f.Fb = fmaf(w, hb, f.Fb);
      f.Fc = fmaf(w, hc, f.Fc);
      f.Fsum = fmaf(w * (float)(n + 3), hn, f.Fsum);
    }
  }
  return f;
}

struct AdjStage {
  float2 B[ADJ_DT * ADJ_LMAX];
  float4 dh[ADJ_DT], dl[ADJ_DT];
  float4 va[ADJ_DT];                          // v = A^T dir and qd = |v|^2 (disks/Gaussians: k' = |k| v)
  float beta[ADJ_DT][ADJ_CL][ADJ_TERMS];
  float4 ctr[ADJ_CL];                         // patch centre and scale s (one for the CTA)
  float4 pw[2 * ADJ_LMAX];                    // (k s)^0, ^2, .. ^14 of each covered radius
  float2 km[ADJ_LMAX], kt[ADJ_LMAX], ctab[PHASOR_ENTRIES * ADJ_COPIES], ctabm[PHASOR_ENTRIES * ADJ_COPIES];
  int nr;
};

// Radii, phasor table and the clusters of this CTA's elements.
__device__ __forceinline__ void adj_setup(AdjStage& st, const KGridDev& kg, const BatchDev& b, const ObjDev& od,
                                          int first) {
  for (int r = threadIdx.x; r < kg.L; r += blockDim.x) {
    st.km[r] = kg.kmag[r];
    st.kt[r] = kg.kt64[r];
  }
  stage_phasors<ADJ_COPIES>(kg.cis_tab, st.ctab);
  stage_phasors<ADJ_COPIES>(kg.cis_tabm, st.ctabm);
  if (threadIdx.x < 32) {
    // a patch's sphere from its leaves'
    const int lane = threadIdx.x, p0 = first + lane * ADJ_PATCH;
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane < ADJ_CL && p0 < od.n_elems) {
      const float4* leaf = b.leaves + od.cl_off * (PI_CLUSTER / PI_LEAF) + p0 / PI_LEAF;
      const int nl = min(ADJ_PATCH, od.n_elems - p0 + PI_LEAF - 1) / PI_LEAF;
      for (int l = 0; l < nl; ++l) { c.x += leaf[l].x; c.y += leaf[l].y; c.z += leaf[l].z; }
      const float inv = 1.0f / nl;
      c = make_float4(c.x * inv, c.y * inv, c.z * inv, 0.f);
      for (int l = 0; l < nl; ++l) {
        const float dx = leaf[l].x - c.x, dy = leaf[l].y - c.y, dz = leaf[l].z - c.z;
        const float reach = sqrtf(dx * dx + dy * dy + dz * dz) * 1.000001f + leaf[l].w;
        c.w = reach > c.w || !(reach == reach) ? reach : c.w;
      }
    }
    float rho = c.w;  // of all patches; NaN stays
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      const float o = __shfl_xor_sync(0xffffffffu, rho, w);
      rho = o > rho || !(o == o) ? o : rho;
    }
    const int ex = rho > 0.f ? min(120, max(-100, ilogbf(rho) + 1)) : 0;
    if (lane < ADJ_CL) st.ctr[lane] = make_float4(c.x, c.y, c.z, __int_as_float((127 + ex) << 23));
    const int n = covered_radii(kg, rho, od.type == PI_GEOM_TRIANGLE ? ADJ_X_TRI : ADJ_X_SURF);
    if (lane == 0) st.nr = n;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < st.nr; r += blockDim.x) {
    const float k = st.km[r].x * st.ctr[0].w, u = k * k, u2 = u * u, u4 = u2 * u2;
    st.pw[2 * r] = make_float4(1.f, u, u2, u2 * u);
    st.pw[2 * r + 1] = make_float4(u4, u4 * u, u4 * u2, u4 * u2 * u);
  }
}

// Stages the cotangent and directions of the tile at e0, then the betas.
__device__ __forceinline__ void stage_tile(AdjStage& st, const KGridDev& kg, const ObjDev& od, const float2* Bt_obj,
                                           int n_cl, int e0) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int jn = min(ADJ_DT, kg.Me - e0);
  if (tid < ADJ_DT) {
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    if (tid < jn) { const int j = kg.dpair[e0 + tid].x; h = kg.dir_hi[j]; l = kg.dir_lo[j]; }
    st.dh[tid] = h;
    st.dl[tid] = l;
    const float* Am = od.A;
    const float vx = Am[0] * h.x + Am[3] * h.y + Am[6] * h.z, vy = Am[1] * h.x + Am[4] * h.y + Am[7] * h.z,
                vz = Am[2] * h.x + Am[5] * h.y + Am[8] * h.z;
    st.va[tid] = make_float4(vx, vy, vz, fmaf(vx, vx, fmaf(vy, vy, vz * vz)));
  }
  for (int t = tid; t < ADJ_DT * kg.L; t += blockDim.x) {
    const int r = t / ADJ_DT, jj = t % ADJ_DT;
    if (jj < jn) st.B[jj * ADJ_LMAX + r] = Bt_obj[(int64_t)r * kg.Me + e0 + jj];
  }
  __syncthreads();
  const int nr = st.nr;
  if (nr > 0) {
    // four threads per patch and direction: the even and the odd orders, of every
    // other pair of radii; the two of a pair each form one radius's term and hand
    // the other its half
    const int jj = tid / (4 * ADJ_CL), c = tid / 4 % ADJ_CL, odd = tid & 1;
    if (jj < jn && c < n_cl) {
      const unsigned quad = 15u << (lane & ~3);
      const float4 h = st.dh[jj], l = st.dl[jj], ct = st.ctr[c];
      const df sc = cdot(make_float3(h.x, h.y, h.z), make_float3(l.x, l.y, l.z), make_float3(ct.x, ct.y, ct.z));
      const float2* Bj = st.B + jj * ADJ_LMAX;
      float p[ADJ_TERMS / 2];
#pragma unroll
      for (int m = 0; m < ADJ_TERMS / 2; ++m) p[m] = 0.f;
      for (int s0 = 0; s0 < nr; s0 += 4) {
        const int ra = s0 + (tid & 2), r0 = min(ra, nr - 1), r = min(ra + odd, nr - 1), r1 = min(ra + 1, nr - 1);
        const float2 Bv = Bj[r];
        const cf P = cis_tab_df<ADJ_COPIES>(st.ctab, st.kt[r], sc);
        const float keep = ra + odd < nr ? 1.f : 0.f;
        const float zr = keep * fmaf(Bv.x, P.re, Bv.y * P.im), zi = keep * (st.km[r].x * ct.w) * fmaf(Bv.x, P.im, -Bv.y * P.re);
        const float got = __shfl_xor_sync(quad, odd ? zr : zi, 1);
        const float za = odd ? got : zr, zb = odd ? zi : got;  // of radii r0 and r1
        const float4 a0 = st.pw[2 * r0], a1 = st.pw[2 * r0 + 1], b0 = st.pw[2 * r1], b1 = st.pw[2 * r1 + 1];
        p[0] = fmaf(za, a0.x, fmaf(zb, b0.x, p[0])); p[1] = fmaf(za, a0.y, fmaf(zb, b0.y, p[1]));
        p[2] = fmaf(za, a0.z, fmaf(zb, b0.z, p[2])); p[3] = fmaf(za, a0.w, fmaf(zb, b0.w, p[3]));
        p[4] = fmaf(za, a1.x, fmaf(zb, b1.x, p[4])); p[5] = fmaf(za, a1.y, fmaf(zb, b1.y, p[5]));
        p[6] = fmaf(za, a1.z, fmaf(zb, b1.z, p[6])); p[7] = fmaf(za, a1.w, fmaf(zb, b1.w, p[7]));
      }
      // Re(i^m z): z's real part for even m, minus its imaginary part for odd m, with the sign of i^(m - m mod 2)
#pragma unroll
      for (int j = 0; j < ADJ_TERMS / 2; ++j) {
        p[j] += __shfl_xor_sync(quad, p[j], 2);
        if ((tid & 2) == 0) st.beta[jj][c][2 * j + odd] = ((2 * j + odd + 1) & 2) ? -p[j] : p[j];
      }
    }
    __syncthreads();
  }
}

// The CTAs of a thread-block cluster (S along x) take the same elements and
// split the tiles of directions; N sums per thread meet through distributed
// shared memory (st.B is free by then), the first CTA writing them.
template <int N>
__device__ __forceinline__ bool adj_total(AdjStage& st, kf (&g)[N], float (&out)[N]) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] = g[i].s;
  if (S == 1) return true;
  float* sums = reinterpret_cast<float*>(st.B);
  static_assert(2 * N * ADJ_THREADS * sizeof(float) <= sizeof(st.B), "sums fit the staged cotangent");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    sums[(2 * i) * ADJ_THREADS + threadIdx.x] = g[i].s;
    sums[(2 * i + 1) * ADJ_THREADS + threadIdx.x] = g[i].c;
  }
  cluster.sync();
  if (rank == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      kbsum t{0.f, 0.f};
      for (int q = 0; q < S; ++q) {
        const float* o = cluster.map_shared_rank(sums, q) + 2 * i * ADJ_THREADS + threadIdx.x;
        t.add(o[0]);
        t.lo -= o[ADJ_THREADS];
      }
      out[i] = t.hi + t.lo;
    }
  cluster.sync();  // no CTA leaves while its sums are read
  return rank == 0;
}

// Per disk / Gaussian: 12 outputs dL/dc (3), dL/dn' (3), dL/dM (6, M = A A^T,
// entries xx xy xz yy yz zz of a symmetric gradient).
//   A = e^{ik.c} S(r) (k.n')/|k|,  r^2 = k^T M k - (k.n')^2,
//   dA/dc  = i k A
//   dA/dn' = e^{ik.c} khat [S - (k.n')^2 (dS/dr)/r]
//   dA/dM  = e^{ik.c} (k.n')/|k| (dS/dr)/(2r) k k^T
// Disk S = area 2 J1(rho r)/(rho r), (dS/dr)/r = -2 area rho^2 J2(x)/x^2;
// Gaussian S = w exp(-sigma^2 r^2/2), (dS/dr)/r = -sigma^2 S.
// Expansion (p = rho |k'_perp| / |k|, sigma the projection from the cluster
// centre): with F = Re sum_r conj(B) e^{ik(d.c + sigma)} S / area|w, i k f has
// the coefficients of f shifted by one, and d(2 J1(x)/x)/d(x^2) = -Lambda_2(x)/8,
// Lambda_2 = 8 J2(x)/x^2, so
//   F = sum beta_m u_m,  dF/dsigma = sum beta_{m+1} u_m,
//   dF/dp^2 = 1/8 sum beta_{m+2} v_m (disk), 1/2 sum beta_{m+2} u_m (Gaussian),
// u_m, v_m the moments of 2 J1(x)/x and of Lambda_2:
//   (m+1)(m+2 nu+1) u_{m+1} = (2m+2 nu+1) sigma u_m + (p^2 - sigma^2) u_{m-1}, nu = 1, 2.
__global__ void __launch_bounds__(ADJ_THREADS)
adj_surf_kernel(KGridDev kg, BatchDev b, const AdjWork* __restrict__ work, const float2* __restrict__ Bt,
                float* __restrict__ out) {
  __shared__ AdjStage st;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S_cta = (int)cluster.num_blocks();
  const AdjWork wk = work[blockIdx.x / S_cta];
  const ObjDev od = b.objs[wk.obj];
  const int e = wk.first + threadIdx.x;
  const bool valid = e < od.n_elems;
  const bool disk = od.type == PI_GEOM_DISK;
  adj_setup(st, kg, b, od, wk.first);
  __syncthreads();
  const int nr = st.nr, n_cl = min(ADJ_CL, (od.n_elems - wk.first + ADJ_PATCH - 1) / ADJ_PATCH);
  const int cl = threadIdx.x / ADJ_PATCH;
  float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0, ql = q0, nr4 = q0;
  if (valid) {
    q0 = b.surf_pool[2 * (od.elem_off + e)];
    q1 = b.surf_pool[2 * (od.elem_off + e) + 1];
    ql = b.surf_lo[od.elem_off + e];
    nr4 = b.surf_nref[od.elem_off + e];
  }
  const float4 ct = valid && nr > 0 ? st.ctr[cl] : make_float4(0.f, 0.f, 0.f, 1.f);
  const float inv_s = 1.0f / ct.w;  // a power of two
  const float3 rel = make_float3(((q0.x - ct.x) + ql.x) * inv_s, ((q0.y - ct.y) + ql.y) * inv_s,
                                 ((q0.z - ct.z) + ql.z) * inv_s);
  const float3 c = make_float3(q0.x, q0.y, q0.z), nn = make_float3(q1.x, q1.y, q1.z);
  const float3 cl3 = make_float3(ql.x, ql.y, ql.z);  // centre low word
  const float p0 = q0.w, p1 = q1.w, ps2 = (p0 * inv_s) * (p0 * inv_s);
  kf g[12];
  const float2* Bt_obj = Bt + (int64_t)wk.obj * kg.L * kg.Me;
  for (int j0 = (int)cluster.block_rank() * ADJ_DT; j0 < kg.Me; j0 += S_cta * ADJ_DT) {
    __syncthreads();
    stage_tile(st, kg, od, Bt_obj, n_cl, j0);
    if (!valid) continue;
    const int jn = min(ADJ_DT, kg.Me - j0);
#pragma unroll 1
    for (int jj = 0; jj < jn; ++jj) {
      const float4 h = st.dh[jj], l = st.dl[jj];
      const float3 dh = make_float3(h.x, h.y, h.z), dl = make_float3(l.x, l.y, l.z);
      const float inv_norm = h.w;
      const float sn = dh.x * nn.x + dh.y * nn.y + dh.z * nn.z;
      // |k'_perp|^2 / |k|^2 = qd (1 - |n|^2) + |n|^2 |v x n/|n||^2 (no cancellation near the normal)
      const float4 va = st.va[jj];
      const float cx = fmaf(va.y, nr4.z, -va.z * nr4.y), cy = fmaf(va.z, nr4.x, -va.x * nr4.z),
                  cz = fmaf(va.x, nr4.y, -va.y * nr4.x);
      const float perp = fmaxf(fmaf(va.w, nr4.w, (1.0f - nr4.w) * fmaf(cx, cx, fmaf(cy, cy, cz * cz))), 0.f);
      const float amp = sn * inv_norm;
      float s_c = 0.f, s_n = 0.f, s_m = 0.f;
      if (nr > 0) {
        const float* be = st.beta[jj][cl];
        const float sg = dh.x * rel.x + dh.y * rel.y + dh.z * rel.z;
        const SurfSums f = disk ? disk_adjoint(be, sg, ps2 * perp) : gauss_adjoint(be, sg, ps2 * perp);
        // dF/dperp = rho^2 (or sigma^2) dF/dp^2, in the scaled units s^2 dF/dp^2
        const float fp = 2.0f * ps2 * f.Fp;  // = sum_r k^2 Re(..) Sr / (area|w)
        s_c = inv_s * p1 * amp * f.Fs;
        s_n = p1 * fmaf(-sn * sn, fp, f.F);
        s_m = 0.5f * p1 * amp * fp;
      }
      const float2* Bj = st.B + jj * ADJ_LMAX;
      if (nr < kg.L) {
        const df sc = cdot2(dh, dl, c, cl3);
        const float rr = p0 * sqrt_fast(perp);
        // with z = conj(B) P, S = C f(k) and (dS/dr)/r = -C p0^2 g(k) (disk: C = 2 p1,
        // J1(x)/x and J2(x)/x^2; Gaussian: C = p1, f = g), sums of k Im(z) f, Re(z) f, k^2 Re(z) g
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        const auto add = [&](int r, float k, float f, float gr) {
          const float2 Bv = Bj[r];
          const cf P = cis_tab_df<ADJ_COPIES>(st.ctab, st.kt[r], sc);
          const float ure = Bv.x * P.re + Bv.y * P.im, uim = Bv.x * P.im - Bv.y * P.re;
          a0 = fmaf(k * uim, f, a0);
          a1 = fmaf(ure, f, a1);
          a2 = fmaf(k * k * ure, gr, a2);
        };
        if (disk) {
          int r = nr;
          // the radii up to the first with x >= 1, without a branch between them; then
          // any (eight clouds of 50,000: 10.5 -> 8.7 ms with these sums)
#pragma unroll 2
          for (; r < kg.L; ++r) {
            const float k = st.km[r].x, x = k * rr;
            if (!(x < 1.0f)) break;
            const J12 j = j12_series(0.25f * x * x);
            add(r, k, j.j1, j.j2);
          }
#pragma unroll 1
          for (; r < kg.L; ++r) {
            const float k = st.km[r].x;
            const J12 j = j12(k * rr);
            add(r, k, j.j1, j.j2);
          }
        } else {
          const float hs = -0.5f * p0 * p0 * perp;
#pragma unroll 2
          for (int r = nr; r < kg.L; ++r) {
            const float k = st.km[r].x, f = __expf(hs * k * k);
            add(r, k, f, f);
          }
        }
        const float C = disk ? 2.0f * p1 : p1, Cp = C * p0 * p0;
        s_c = fmaf(-C * amp, a0, s_c);
        s_n += fmaf(sn * sn * Cp, a2, C * a1);
        s_m = fmaf(-0.5f * amp * Cp, a2, s_m);
      }
      g[0].add(dh.x * s_c); g[1].add(dh.y * s_c); g[2].add(dh.z * s_c);
      const float sn2 = s_n * inv_norm;
      g[3].add(dh.x * sn2); g[4].add(dh.y * sn2); g[5].add(dh.z * sn2);
      const float mx = dh.x * s_m, my = dh.y * s_m, mz = dh.z * s_m;
      g[6].add(dh.x * mx); g[7].add(dh.x * my); g[8].add(dh.x * mz);
      g[9].add(dh.y * my); g[10].add(dh.y * mz); g[11].add(dh.z * mz);
    }
  }
  float sum[12];
  const bool mine = adj_total(st, g, sum);
  if (!valid || !mine) return;
  float* o = out + 12 * (od.elem_off + e);
  const float sc8 = (float)INV8PI3;
#pragma unroll
  for (int i = 0; i < 12; ++i) o[i] = sum[i] * sc8;
}

// Per triangle: 9 outputs dL/dv0, dL/dv1, dL/dv2 (world-frame vertex positions).
// Expansion: t0 = Re sum_r conj(B) e[..] = sum_n -beta_n/(n+2)! h_n(a, b, c) and
// its derivatives by the projections, dh_{n+1}/db = h_n(a, b, b, c) by
// h_n(a, b, b, c) = b h_{n-1}(a, b, b, c) + h_n(a, b, c), and their sum
// (a + b + c derivatives of h_{n+1}) (n+3) h_n by translation.
__global__ void __launch_bounds__(ADJ_THREADS, 4)
adj_tri_kernel(KGridDev kg, BatchDev b, const AdjWork* __restrict__ work, const float2* __restrict__ Bt,
               float* __restrict__ out) {
  __shared__ AdjStage st;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S_cta = (int)cluster.num_blocks();
  const AdjWork wk = work[blockIdx.x / S_cta];
  const ObjDev od = b.objs[wk.obj];
  const int e = wk.first + threadIdx.x;
  const bool valid = e < od.n_elems;
  adj_setup(st, kg, b, od, wk.first);
  __syncthreads();
  const int nr = st.nr, n_cl = min(ADJ_CL, (od.n_elems - wk.first + ADJ_PATCH - 1) / ADJ_PATCH);
  const int cl = threadIdx.x / ADJ_PATCH;
  float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0, q2 = q0, ql = q0;
  if (valid) {
    q0 = b.tri_pool[3 * (od.elem_off + e)];
    q1 = b.tri_pool[3 * (od.elem_off + e) + 1];
    q2 = b.tri_pool[3 * (od.elem_off + e) + 2];
    ql = b.tri_lo[od.elem_off + e];
  }
  const float4 ct = valid && nr > 0 ? st.ctr[cl] : make_float4(0.f, 0.f, 0.f, 1.f);
  const float inv_s = 1.0f / ct.w;  // a power of two
  // A triangle without edges has no gradient wherever it lies.  One with unset vertex
  // ids is stored so at the object's origin, outside its patch's sphere (that of the
  // others): the powers of its projection would overflow, and 0 inf is not 0.
  const bool edges = q1.x != 0.f || q1.y != 0.f || q1.z != 0.f || q2.x != 0.f || q2.y != 0.f || q2.z != 0.f;
  const float3 rel = edges ? make_float3((q0.x - ct.x) + ql.x, (q0.y - ct.y) + ql.y, (q0.z - ct.z) + ql.z)
                           : make_float3(0.f, 0.f, 0.f);
  const float3 ml = make_float3(ql.x, ql.y, ql.z);  // centroid low word
  const float3 m = make_float3(q0.x, q0.y, q0.z), e1 = make_float3(q1.x, q1.y, q1.z),
               e2 = make_float3(q2.x, q2.y, q2.z), S = make_float3(q0.w, q1.w, q2.w);
  kf g[9];
  const float2* Bt_obj = Bt + (int64_t)wk.obj * kg.L * kg.Me;
  for (int j0 = (int)cluster.block_rank() * ADJ_DT; j0 < kg.Me; j0 += S_cta * ADJ_DT) {
    __syncthreads();
    stage_tile(st, kg, od, Bt_obj, n_cl, j0);
    if (!valid) continue;
    const int jn = min(ADJ_DT, kg.Me - j0);
#pragma unroll 1
    for (int jj = 0; jj < jn; ++jj) {
      const float4 h = st.dh[jj], l = st.dl[jj];
      const float3 dh = make_float3(h.x, h.y, h.z), dl = make_float3(l.x, l.y, l.z);
      const float inv_norm = h.w;
      const float gam = (dh.x * S.x + dh.y * S.y + dh.z * S.z) * inv_norm;
      float t0 = 0.f, ta = 0.f, tb = 0.f, tc = 0.f;
      if (nr > 0) {
        const float3 ds = make_float3(dh.x * inv_s, dh.y * inv_s, dh.z * inv_s);
        const float s1 = ds.x * e1.x + ds.y * e1.y + ds.z * e1.z, s2 = ds.x * e2.x + ds.y * e2.y + ds.z * e2.z;
        const float pa = fmaf(s1 + s2, -1.0f / 3.0f, ds.x * rel.x + ds.y * rel.y + ds.z * rel.z);
        const TriSums f = tri_adjoint(st.beta[jj][cl], pa, pa + s1, pa + s2);
        t0 = f.F;
        tb = f.Fb * inv_s;
        tc = f.Fc * inv_s;
        ta = fmaf(f.Fsum, inv_s, -tb - tc);
      }
      if (nr < kg.L) {
        const df sm = cdot2(dh, dl, m, ml), d1 = cdot(dh, dl, e1), d2 = cdot(dh, dl, e2);
        const df sa = df_add(sm, df_div3(df_add(d1, d2)) * -1.0f);
        const float sp = fmaxf(fmaxf(fabsf(d1.hi), fabsf(d2.hi)), fabsf(d2.hi - d1.hi));
        const float kthr = __fdividef(2.0f, sp);  // the series for k sp < 2 (inf when sp = 0)
        const TriSorted ts = tri_sorted(sa, d1, d2);
        float tu = 0.f, tw = 0.f, ti = 0.f;  // sums of k Re(conj(B) D_u), ... D_w, ... i F
        const TriDerPoly cp = tri_der_coeffs(d1.hi, d2.hi);
        const float2* Bj = st.B + jj * ADJ_LMAX;
        for (int r = nr; r < kg.L; ++r) {
          const float2 Bv = Bj[r];
          const float k = st.km[r].x;
          if (k < kthr) {
            // F = P SF, D_v = P SV with the series as polynomials in k; with
            // BP = conj(B) P, Re(conj(B) X) = Re(BP SX) and D_a = i F - D_b - D_c
            const cf P = cis_tab_df<ADJ_COPIES>(st.ctab, st.kt[r], sm);
            const float u = k * k, k3 = u * k;
            const float fre = poly_u(cp.fa, u), fim = k3 * poly_u(cp.fb, u);
            const float bim = poly_u(cp.ba, u), bre = k * poly_u(cp.bb, u);
            const float cim = poly_u(cp.ca, u), cre = k * poly_u(cp.cb, u);
            const float pr = fmaf(Bv.x, P.re, Bv.y * P.im), pi = fmaf(Bv.x, P.im, -Bv.y * P.re);
            const float f_re = fmaf(pr, fre, -pi * fim), f_im = fmaf(pr, fim, pi * fre);
            const float b_re = fmaf(pr, bre, -pi * bim), c_re = fmaf(pr, cre, -pi * cim);
            t0 += f_re;
            ta = fmaf(k, -f_im - b_re - c_re, ta);
            tb = fmaf(k, b_re, tb);
            tc = fmaf(k, c_re, tc);
          } else {
            const cf P = cis_tab_df<ADJ_COPIES>(st.ctab, st.kt[r], ts.sv);
            const TriWideDer d = tri_wide_der<ADJ_COPIES>(st.ctabm, st.kt[r], k, ts);
            const float pr = fmaf(Bv.x, P.re, Bv.y * P.im), pi = fmaf(Bv.x, P.im, -Bv.y * P.re);  // conj(B) P
            t0 = fmaf(pr, d.F.re, fmaf(-pi, d.F.im, t0));
            ti = fmaf(-k, fmaf(pr, d.F.im, pi * d.F.re), ti);
            tu = fmaf(k, fmaf(pr, d.Du.re, -pi * d.Du.im), tu);
            tw = fmaf(k, fmaf(pr, d.Dw.re, -pi * d.Dw.im), tw);
          }
        }
        const float tv = ti - tu - tw;
        ta += ts.u == 0 ? tu : (ts.w == 0 ? tw : tv);
        tb += ts.u == 1 ? tu : (ts.w == 1 ? tw : tv);
        tc += ts.u == 2 ? tu : (ts.w == 2 ? tw : tv);
      }
      // khat x u / 2 terms for grad gamma
      const float3 kh = make_float3(dh.x * inv_norm, dh.y * inv_norm, dh.z * inv_norm);
      const float3 w0 = make_float3(e2.x - e1.x, e2.y - e1.y, e2.z - e1.z);
      const float3 c0 = make_float3(0.5f * (kh.y * w0.z - kh.z * w0.y), 0.5f * (kh.z * w0.x - kh.x * w0.z),
                                    0.5f * (kh.x * w0.y - kh.y * w0.x));
      const float3 c1 = make_float3(-0.5f * (kh.y * e2.z - kh.z * e2.y), -0.5f * (kh.z * e2.x - kh.x * e2.z),
                                    -0.5f * (kh.x * e2.y - kh.y * e2.x));
      const float3 c2 = make_float3(0.5f * (kh.y * e1.z - kh.z * e1.y), 0.5f * (kh.z * e1.x - kh.x * e1.z),
                                    0.5f * (kh.x * e1.y - kh.y * e1.x));
      // dL/dv = -2 (grad gamma t0 + gamma dir t_v), the -2 applied at the end
      const float ga = gam * ta, gb = gam * tb, gc = gam * tc;
      g[0].add(fmaf(dh.x, ga, c0.x * t0)); g[1].add(fmaf(dh.y, ga, c0.y * t0)); g[2].add(fmaf(dh.z, ga, c0.z * t0));
      g[3].add(fmaf(dh.x, gb, c1.x * t0)); g[4].add(fmaf(dh.y, gb, c1.y * t0)); g[5].add(fmaf(dh.z, gb, c1.z * t0));
      g[6].add(fmaf(dh.x, gc, c2.x * t0)); g[7].add(fmaf(dh.y, gc, c2.y * t0)); g[8].add(fmaf(dh.z, gc, c2.z * t0));
    }
  }
  float sum[9];
  const bool mine = adj_total(st, g, sum);
  if (!valid || !mine) return;
  float* o = out + 9 * (od.elem_off + e);
  const float sc8 = -2.0f * (float)INV8PI3;
#pragma unroll
  for (int a = 0; a < 9; ++a) o[a] = sum[a] * sc8;
}

// ---- chain rule to DoF gradients ---------------------------------------------------
struct ChainObj {
  int32_t geom_type, dof_type;
  int64_t n_elems, pool_off, grad_off;   // grad_off: offset (doubles) of this object's DoF gradient
  const unsigned char* src;             // reference-layout packed source
  const double* dofs;
  const int32_t* perm;                  // pool entry -> element, or nullptr
};

struct TriSrcC { double a[3], e1[3], e2[3], S[3]; int32_t vid0, vid1, vid2, pad; };
struct SurfSrcC { double c[3], n[3], p0, p1; };

// AffineDoF: a fixed-order FP64 reduction per object, the CTAs of a
// thread-block cluster sharing its elements (FP64 runs at ~2 operations per SM
// and clock: 116 us for 24 meshes of 5,120 triangles on one CTA each).
//   triangles: dL/dt = sum_v g_v, dL/dA = sum_v g_v v_ref^T  (v = A v_ref + t)
//   surfels:   dL/dt = sum g_c, dL/dA = sum g_c c_ref^T + g_n n_ref^T + 2 G_M A
constexpr int CHAIN_THREADS = 128, CHAIN_SPLIT = 8;
__global__ void __launch_bounds__(CHAIN_THREADS)
chain_affine_kernel(const ChainObj* objs, const float* __restrict__ tri_g, const float* __restrict__ surf_g,
                    double* __restrict__ grad) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const ChainObj o = objs[blockIdx.x / S];
  if (o.dof_type != PI_DOF_AFFINE) return;
  __shared__ double red[18][CHAIN_THREADS / 32];
  __shared__ double total[18];
  double acc[18];
#pragma unroll
  for (int a = 0; a < 18; ++a) acc[a] = 0.0;
  for (int64_t p = rank * CHAIN_THREADS + threadIdx.x; p < o.n_elems; p += S * CHAIN_THREADS) {
    const int64_t e = o.perm ? o.perm[p] : p;
    if (o.geom_type == PI_GEOM_TRIANGLE) {
      const TriSrcC& t = reinterpret_cast<const TriSrcC*>(o.src)[e];
      const float* g = tri_g + 9 * (o.pool_off + p);
      // sum_s g_s v_s^T = (g_0 + g_1 + g_2) a^T + g_1 e1^T + g_2 e2^T
      for (int r = 0; r < 3; ++r) {
        const double g1 = g[3 + r], g2 = g[6 + r], gs = (double)g[r] + g1 + g2;
        acc[r] += gs;
        for (int c = 0; c < 3; ++c) acc[3 + 3 * r + c] += gs * t.a[c] + g1 * t.e1[c] + g2 * t.e2[c];
      }
    } else {
      const SurfSrcC& s = reinterpret_cast<const SurfSrcC*>(o.src)[e];
      const float* g = surf_g + 12 * (o.pool_off + p);
      for (int r = 0; r < 3; ++r) {
        acc[r] += g[r];
        for (int c = 0; c < 3; ++c) acc[3 + 3 * r + c] += (double)g[r] * s.c[c] + (double)g[3 + r] * s.n[c];
      }
      for (int a = 0; a < 6; ++a) acc[12 + a] += g[6 + a];
    }
  }
#pragma unroll
  for (int a = 0; a < 18; ++a)
    for (int w = 16; w > 0; w >>= 1) acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], w);
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 18; ++a) red[a][threadIdx.x >> 5] = acc[a];
  __syncthreads();
  if (threadIdx.x < 18) {
    double t = 0.0;
    for (int w = 0; w < CHAIN_THREADS / 32; ++w) t += red[threadIdx.x][w];
    total[threadIdx.x] = t;
  }
  if (S > 1) {
    cluster.sync();
    double t = 0.0;
    if (rank == 0 && threadIdx.x < 18)
      for (int q = 0; q < S; ++q) t += cluster.map_shared_rank(total, q)[threadIdx.x];
    cluster.sync();  // no CTA leaves, or overwrites it, while its sum is read
    if (rank == 0 && threadIdx.x < 18) total[threadIdx.x] = t;
  }
  __syncthreads();
  if (rank == 0 && threadIdx.x == 0) {
    double* out = grad + o.grad_off;
    for (int a = 0; a < 12; ++a) out[a] = total[a];
    if (o.geom_type != PI_GEOM_TRIANGLE) {
      // + 2 G A with G symmetric (xx xy xz yy yz zz)
      const double G[3][3] = {{total[12], total[13], total[14]},
                              {total[13], total[15], total[16]},
                              {total[14], total[16], total[17]}};
      const double* A = o.dofs + 3;
      for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c)
          out[3 + 3 * r + c] += 2.0 * (G[r][0] * A[c] + G[r][1] * A[3 + c] + G[r][2] * A[6 + c]);
    }
  }
}

// TriangleMeshDoF: one thread per vertex, CSR gather of (triangle, slot) gradients.
__global__ void chain_mesh_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ ent,
                                  const float* __restrict__ tri_g, int64_t nv_total, const int64_t* __restrict__ vmap,
                                  double* __restrict__ grad) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv_total) return;
  double s[3] = {0.0, 0.0, 0.0};
  for (int64_t p = row[v]; p < row[v + 1]; ++p) {
    const int64_t te = ent[p];  // pool triangle * 3 + slot
    const float* g = tri_g + 9 * (te / 3) + 3 * (te % 3);
    s[0] += g[0]; s[1] += g[1]; s[2] += g[2];
  }
  double* o = grad + vmap[v];
  o[0] = s[0]; o[1] = s[1]; o[2] = s[2];
}

}  // namespace

// ---- host side ------------------------------------------------------------------------
int64_t dof_gradient_size(const pi_batch_impl* b) {
  int64_t s = 0;
  for (const HostObjInfo& in : b->info) s += in.n_dofs;
  return s;
}

size_t adjoint_ws_bytes(const pi_kgrid_impl* kg, const pi_batch_impl* b) {
  const size_t nb = (size_t)b->n_obj * kg->Q * sizeof(float2);            // cotangent
  const size_t cs = (size_t)b->n_obj * b->n_obj * sizeof(float);           // C + C^T
  const size_t tg = (size_t)b->n_tri * 9 * sizeof(float), sg = (size_t)b->n_surf * 12 * sizeof(float);
  return 256 + nb + 256 + cs + 256 + tg + 256 + sg + 256;
}

static size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

int launch_adjoint_elements(const pi_kgrid_impl* kg, const pi_batch_impl* b, const float2* Jw, const double* W_host,
                            float** tri_g_out, float** surf_g_out, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (kg->L > ADJ_LMAX) return fail(PI_ERR_UNSUPPORTED, "adjoint supports at most 256 radial nodes");
  if (ws_bytes < adjoint_ws_bytes(kg, b) || !ws) return fail(PI_ERR_WORKSPACE_TOO_SMALL, "adjoint workspace too small");
  const int n = b->n_obj;
  unsigned char* p = static_cast<unsigned char*>(ws);
  float2* Bw = reinterpret_cast<float2*>(p);
  p += up256((size_t)n * kg->Q * sizeof(float2));
  float* Cs = reinterpret_cast<float*>(p);
  p += up256((size_t)n * n * sizeof(float));
  float* tri_g = reinterpret_cast<float*>(p);
  p += up256((size_t)b->n_tri * 9 * sizeof(float));
  float* surf_g = reinterpret_cast<float*>(p);
  std::vector<float> cs((size_t)n * n);
  for (size_t t = 0; t < cs.size(); ++t) cs[t] = (float)W_host[t];
  PI_CUDA(cudaMemcpyAsync(Cs, cs.data(), cs.size() * sizeof(float), cudaMemcpyHostToDevice, s));
  dim3 cg((unsigned)(((int64_t)kg->Me * kg->L + 255) / 256), (unsigned)((n + COT_N - 1) / COT_N));
  cotangent_kernel<<<cg, 256, 0, s>>>(kg->dev, b->dev(), Jw, Cs, Bw);
  PI_LAUNCHED("cotangent_kernel");
  std::vector<AdjWork> wt, ws2;
  for (int i = 0; i < n; ++i) {
    const HostObjInfo& in = b->info[i];
    for (int64_t f = 0; f < in.n_elems; f += ADJ_THREADS)
      (in.geom_type == PI_GEOM_TRIANGLE ? wt : ws2).push_back(AdjWork{i, (int32_t)f});
  }
  AdjWork* dw = nullptr;
  const size_t nw = wt.size() + ws2.size();
  if (nw) {
    PI_CUDA(pool_alloc((void**)&dw, nw * sizeof(AdjWork), s));
    std::vector<AdjWork> all(wt);
    all.insert(all.end(), ws2.begin(), ws2.end());
    PI_CUDA(cudaMemcpyAsync(dw, all.data(), nw * sizeof(AdjWork), cudaMemcpyHostToDevice, s));
    // the directions split over a thread-block cluster until the launch has two
    // waves of four CTAs per SM
    const KGridDev K = kg->dev;
    const BatchDev B = b->dev();
    auto launch = [&](const void* fn, size_t items, const AdjWork* w, float* grad) {
      int S = 1;
      while (S < 16 && (int64_t)S * (int64_t)items < 8 * (int64_t)current_sm_count() && K.Me > 2 * S * ADJ_DT) S *= 2;
      void* args[5] = {const_cast<KGridDev*>(&K), const_cast<BatchDev*>(&B), &w, &Bw, &grad};
      return launch_split(fn, dim3((unsigned)(items * S)), ADJ_THREADS, 0, S, args, s);
    };
    if (!wt.empty()) {
      if (int rc = launch(reinterpret_cast<const void*>(adj_tri_kernel), wt.size(), dw, tri_g)) return rc;
      PI_LAUNCHED("adj_tri_kernel");
    }
    if (!ws2.empty()) {
      if (int rc = launch(reinterpret_cast<const void*>(adj_surf_kernel), ws2.size(), dw + wt.size(), surf_g)) return rc;
      PI_LAUNCHED("adj_surf_kernel");
    }
    PI_CUDA(cudaFreeAsync(dw, s));
  }
  *tri_g_out = tri_g;
  *surf_g_out = surf_g;
  return PI_OK;
}

int launch_dof_gradients(const pi_kgrid_impl* kg, pi_batch_impl* b, const float2* Jw, const double* W_host,
                         double* grad, void* ws, size_t ws_bytes, cudaStream_t s) {
  float *tri_g = nullptr, *surf_g = nullptr;
  int rc = launch_adjoint_elements(kg, b, Jw, W_host, &tri_g, &surf_g, ws, ws_bytes, s);
  if (rc) return rc;
  const int n = b->n_obj;
  std::vector<ChainObj> co(n);
  int64_t goff = 0;
  bool any_mesh = false;
  for (int i = 0; i < n; ++i) {
    const HostObjInfo& in = b->info[i];
    co[i] = ChainObj{in.geom_type, in.dof_type, in.n_elems, in.pool_off, goff,
                     static_cast<const unsigned char*>(b->d_src) + in.src_off, b->d_dofs + in.dof_off,
                     in.perm_off >= 0 ? b->d_perm + in.perm_off : nullptr};
    goff += in.n_dofs;
    any_mesh |= in.dof_type == PI_DOF_TRIANGLE_MESH;
  }
  ChainObj* dco = nullptr;
  PI_CUDA(pool_alloc((void**)&dco, n * sizeof(ChainObj), s));
  PI_CUDA(cudaMemcpyAsync(dco, co.data(), n * sizeof(ChainObj), cudaMemcpyHostToDevice, s));
  int64_t max_elems = 0;
  for (const HostObjInfo& in : b->info) max_elems = std::max(max_elems, in.n_elems);
  const int S = max_elems > 2 * CHAIN_THREADS ? CHAIN_SPLIT : 1;
  void* cargs[4] = {&dco, &tri_g, &surf_g, &grad};
  if (int rc2 = launch_split(reinterpret_cast<const void*>(chain_affine_kernel), dim3((unsigned)(n * S)), CHAIN_THREADS,
                             0, S, cargs, s))
    return rc2;
  PI_LAUNCHED("chain_affine_kernel");
  PI_CUDA(cudaFreeAsync(dco, s));
  if (any_mesh) {
    if (!b->d_vrow) return fail(PI_ERR_UNSUPPORTED, "vertex adjacency missing for TriangleMeshDoF objects");
    chain_mesh_kernel<<<(unsigned)((b->n_mesh_verts + 255) / 256), 256, 0, s>>>(b->d_vrow, b->d_vent, tri_g,
                                                                               b->n_mesh_verts, b->d_vmap, grad);
    PI_LAUNCHED("chain_mesh_kernel");
  }
  return PI_OK;
}

}  // namespace pi
