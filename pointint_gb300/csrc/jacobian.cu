// Jacobian of the form factors with respect to the DoFs, and from it the
// Gauss-Newton Hessian blocks.
//
//   G[d][q] = sqrt|w_q| dA_n(k_q)/dtheta_{n,d}
//
// for every object n and DoF d, rows in the order of the concatenated DoF
// vector, FP32 complex, q-major like J.  The reference's Gauss-Newton blocks
// (hessian_ij of compute_intersection_volume_multi_object.cpp:236-292 / K16
// cpp/src/compute_intersection_volume_multi_object.cu:189-229; hessian_geom1,
// geom2, cross of compute_intersection_volume_cpu.cpp:153-186 / K11
// cpp/src/compute_intersection_volume.cu:109-157) are blocks of
//
//   H = Re(G diag(sign w) G^H) / (8 pi^3),
//
// which the volume contraction forms from G's rows exactly as it forms V from
// J's.  The per-element derivatives are the adjoint's (adjoint.cu); here they
// are summed over elements at every k-node (forward mode) instead of over
// k-nodes for every element.
//
//  * AffineDoF triangles (x = A x0 + t): dA/dt_r = i k_r A; dA/dA_rc =
//    sum_e sum_s (df_e/dv_s)_r x0_{s,c} with df/dv_s = -2 (c_s F + gamma k d D_s),
//    so each thread accumulates sum_e F N0_e (from which sum_e F U_e,
//    U_rc = sum_s c_{s,r} x0_{s,c}, follows per node) and
//    sum_e gamma sum_s D_s x0_s.
//  * AffineDoF disks / Gaussians (c = A c0 + t, n' = A n0, M = A A^T):
//    dA/dA_rc = i k d_r Z_c + khat_r N_c + k^2 d_r (A^T d)_c Y with
//    Z = sum P S a c0, N = sum P (S - k^2 s_n^2 S_r) n0, Y = sum P a S_r.
//  * TriangleMeshDoF: dA/dv_p = sum over the triangles at vertex p of
//    df_e/dv_p (a gather over the batch's vertex adjacency, no atomics).
//
// Thread layouts: the affine-triangle kernel as ff_kernel (a warp owns 32
// directions x JAC_R neighbouring radii); the others one radius per thread (a
// warp owns 32 directions at one radius).  The origin phase e^{ik.o} and
// sqrt|w| are applied once per output.
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

constexpr int JAC_THREADS = 128;
constexpr int JAC_WARPS = JAC_THREADS / 32;
constexpr int JAC_TILE = 128;
// copies of the phasor table: the running sums leave no room for 16
constexpr int JAC_COPIES = 4;

enum { JAC_AFFINE_TRI = 0, JAC_AFFINE_SURF = 1, JAC_MESH_TRI = 2 };

// Radii that the expansions cover (as moment_radii): the n-th term of the
// derivatives' series is at most (k rho)^n / n! of the leading one, as the values'.
constexpr float JAC_X_TRI = MOMENT_X_TRI;
constexpr int JM_RADII = 48;  // radii of a CTA of jac_moment_kernel: its running sums fill shared memory
// Few radii over a multiple of that go to the direct kernel where its threads own
// four radii: they cost it less than another group of CTAs that forms all moments
// again (256 solids 70.2 -> 65.7 ms).  At two radii per thread they cost more (one
// mesh 0.98 -> 1.06 ms).
constexpr int JM_SPARE = 4;
__device__ __forceinline__ int jac_moment_radii(const KGridDev& kg, float rho, int spare) {
  const int n = covered_radii(kg, rho, JAC_X_TRI), over = n % JM_RADII;
  return n > JM_RADII && over <= spare ? n - over : n;
}

struct JacObj {
  int32_t obj, kind;
  int64_t row0;                    // first row of G
  int64_t vstart, nverts;          // TriangleMeshDoF: vertex range in the batch's adjacency
  const unsigned char* src;        // reference-layout source elements
  const double* dofs;              // device DoF vector
};

struct TriSrcJ { double a[3], e1[3], e2[3], S[3]; int32_t vid0, vid1, vid2, pad; };
struct SurfSrcJ { double c[3], n[3], p0, p1; };

// FP32 sum with chunked partials and a compensated running total (complex).
struct kcf {
  float pr = 0.f, pi = 0.f, sr = 0.f, si = 0.f, cr = 0.f, ci = 0.f;
  __device__ __forceinline__ void fma_add(cf a, float s) { pr = fmaf(a.re, s, pr); pi = fmaf(a.im, s, pi); }
  __device__ __forceinline__ void flush() {
    float y = pr - cr, t = sr + y;
    cr = (t - sr) - y; sr = t;
    y = pi - ci; t = si + y;
    ci = (t - si) - y; si = t;
    pr = pi = 0.f;
  }
  __device__ __forceinline__ cf value() const { return cf{sr, si}; }
};

constexpr int JAC_NSUM = 12;  // floats per radius of the affine triangles' sums: NF[3], W[3] (complex)

struct JacThread {
  int j, jm, r;  // direction j evaluated, its antipode jm written from it (or -1)
  bool active;
  float3 dh, dl;
  float inv_norm, dnorm;
  df k;
  float2 kt;  // |k| in 1/64 turns per unit length (double-float), for the table phasors
};

__device__ __forceinline__ JacThread jac_thread(const KGridDev& kg) {
  JacThread t;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * JAC_WARPS + warp;
  const int dt = item / kg.L;
  t.r = item - dt * kg.L;
  const int ei = dt * 32 + lane;
  t.active = dt < (kg.Me + 31) / 32 && ei < kg.Me;
  t.j = 0;
  t.jm = -1;
  if (t.active) { const int2 pr = kg.dpair[ei]; t.j = pr.x; t.jm = pr.y; }
  t.dh = t.dl = make_float3(0.f, 0.f, 0.f);
  t.inv_norm = t.dnorm = 0.f;
  t.k = df{0.f, 0.f};
  t.kt = make_float2(0.f, 0.f);
  if (t.active) {
    const float4 h = kg.dir_hi[t.j], l = kg.dir_lo[t.j];
    t.dh = make_float3(h.x, h.y, h.z);
    t.dl = make_float3(l.x, l.y, l.z);
    t.inv_norm = h.w;
    t.dnorm = l.w;
    const float2 km = kg.kmag[t.r];
    t.k = df{km.x, km.y};
    t.kt = kg.kt64[t.r];
  }
  return t;
}

// The phasor table of cis_tab_df in shared memory; every thread of the CTA
// calls this before its first use (it ends in __syncthreads).
__device__ __forceinline__ void stage_cis_tab(const KGridDev& kg, float2* ctab) {
  stage_phasors<JAC_COPIES>(kg.cis_tab, ctab);
  __syncthreads();
}

// e^{ik.o} for this thread's node (0 at k = 0, where A = 0 by definition).
__device__ __forceinline__ cf jac_origin_phase(const JacThread& t, const ObjDev& od) {
  const double so_d = ((double)t.dh.x + t.dl.x) * od.origin[0] + ((double)t.dh.y + t.dl.y) * od.origin[1] +
                      ((double)t.dh.z + t.dl.z) * od.origin[2];
  const cf e = cis_f64(((double)t.k.hi + (double)t.k.lo) * so_d);
  return (t.k.hi * t.dnorm < 1e-10f) ? cf{0.f, 0.f} : e;
}

// The node of radius r and direction j, and that of its antipode jm: a
// derivative of a real solid's form factor obeys dA(-k) = -conj dA(k) like A,
// so one evaluation gives both outputs, each scaled by its own sqrt|w|.
struct JacOut {
  int64_t q, qm;  // qm < 0: no antipode
  float sw, swm;
  __device__ __forceinline__ void put(float2* row, cf v) const {
    row[q] = make_float2(v.re * sw, v.im * sw);
    if (qm >= 0) row[qm] = make_float2(-v.re * swm, v.im * swm);
  }
};

__device__ __forceinline__ JacOut jac_out(const KGridDev& kg, int r, int j, int jm) {
  JacOut o;
  o.q = (int64_t)r * kg.M + j;
  o.qm = jm >= 0 ? (int64_t)r * kg.M + jm : -1;
  o.sw = kg.sqrtw[o.q];
  o.swm = jm >= 0 ? kg.sqrtw[o.qm] : 0.f;
  return o;
}

// Triangle derivative pieces at one node: F, D_a, D_b, D_c (tri_adjoint.cuh),
// gamma = khat.S and the gradient vectors c_s of gamma with respect to the vertices.
struct TriNode {
  TriDer d;
  float gam;
  float3 c[3];
};

// ml: the centroid's low word, and in .w the longest edge (the series-length bound).
__device__ __forceinline__ TriNode tri_node(const JacThread& t, const float2* ctab, float3 m, float4 ml, float3 e1,
                                            float3 e2, float3 S) {
  TriNode o;
  const df sm = cdot2(t.dh, t.dl, m, make_float3(ml.x, ml.y, ml.z)), d1 = cdot(t.dh, t.dl, e1),
           d2 = cdot(t.dh, t.dl, e2);
  const float sp = fmaxf(fmaxf(fabsf(d1.hi), fabsf(d2.hi)), fabsf(d2.hi - d1.hi));
  const float al = t.k.hi * d1.hi, be = t.k.hi * d2.hi;
  if (t.k.hi * sp < 2.0f) {
    const cf P = cis_tab_df<JAC_COPIES>(ctab, t.kt, sm);
    // the lanes of a warp share the radius and the element: a uniform branch
    if (t.k.hi * t.dnorm * ml.w < 1.0f)
      o.d = tri_series_der<8>(P, al, be);
    else
      o.d = tri_series_der<12>(P, al, be);
  } else {
    const df sa = df_add(sm, df_div3(df_add(d1, d2)) * -1.0f);
    const df sb = df_add(sa, d1), sc = df_add(sa, d2);
    o.d = tri_generic_der(cis_tab_df<JAC_COPIES>(ctab, t.kt, sa), cis_tab_df<JAC_COPIES>(ctab, t.kt, sb), cis_tab_df<JAC_COPIES>(ctab, t.kt, sc), al, be);
  }
  o.gam = (t.dh.x * S.x + t.dh.y * S.y + t.dh.z * S.z) * t.inv_norm;
  const float3 kh = make_float3(t.dh.x * t.inv_norm, t.dh.y * t.inv_norm, t.dh.z * t.inv_norm);
  const float3 w0 = make_float3(e2.x - e1.x, e2.y - e1.y, e2.z - e1.z);
  o.c[0] = make_float3(0.5f * (kh.y * w0.z - kh.z * w0.y), 0.5f * (kh.z * w0.x - kh.x * w0.z),
                       0.5f * (kh.x * w0.y - kh.y * w0.x));
  o.c[1] = make_float3(-0.5f * (kh.y * e2.z - kh.z * e2.y), -0.5f * (kh.z * e2.x - kh.x * e2.z),
                       -0.5f * (kh.x * e2.y - kh.y * e2.x));
  o.c[2] = make_float3(0.5f * (kh.y * e1.z - kh.z * e1.y), 0.5f * (kh.z * e1.x - kh.x * e1.z),
                       0.5f * (kh.x * e1.y - kh.y * e1.x));
  return o;
}

__device__ __forceinline__ float comp(float3 v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : v.z); }

// Writes the 12 derivatives of an affine triangle object at one node and its
// antipode from the sums NF = sum_e F N0 (complex 3-vector) and
// W = sum_e gamma (i F a0 + D_b E1 + D_c E2), both in the object frame:
//   A = -2 sum gamma F = -khat . (cof(A) NF)     (S = cof(A) N0 / 2)
//   dA/dt_r = i k d_r A
//   dA/dA_rc = -2 (MF_rc + k d_r W_c),
//   MF[r][c] = sum_e F_e sum_s grad_s(gamma)_r x0_s[c] = ((khat / 2) x (A (e_c x NF)))_r
struct JacWriter {
  float A[9], cofd[3];  // A row-major, cof(A)^T khat
  float3 dh, kh;        // direction, khat / 2
  double so_d;          // direction . origin
  float dnorm;
  int j, jm;
  int64_t row0;
  __device__ __forceinline__ JacWriter(const JacObj& jo, const ObjDev& od, float3 dh_, float3 dl, float inv_norm,
                                       float dnorm_, int j_, int jm_)
      : dh(dh_), dnorm(dnorm_), j(j_), jm(jm_), row0(jo.row0) {
    const double* M = jo.dofs + 3;
#pragma unroll
    for (int a = 0; a < 9; ++a) A[a] = (float)M[a];
    kh = make_float3(0.5f * dh.x * inv_norm, 0.5f * dh.y * inv_norm, 0.5f * dh.z * inv_norm);
    const float k3[3] = {2.0f * kh.x, 2.0f * kh.y, 2.0f * kh.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
      double v = 0.0;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int r1 = (r + 1) % 3, r2 = (r + 2) % 3;
        v += (double)k3[r] * (M[3 * r1 + c1] * M[3 * r2 + c2] - M[3 * r1 + c2] * M[3 * r2 + c1]);
      }
      cofd[c] = (float)v;
    }
    so_d = ((double)dh.x + dl.x) * od.origin[0] + ((double)dh.y + dl.y) * od.origin[1] +
           ((double)dh.z + dl.z) * od.origin[2];
  }
  __device__ __forceinline__ void put(const KGridDev& kg, float2* G, int r, float2 km, const float (&sv)[JAC_NSUM]) const {
    const JacOut o = jac_out(kg, r, j, jm);
    const float k = km.x;
    // e^{ik.o} (0 at k = 0, where A = 0 by definition); sqrt|w| at the store
    const cf eo = cis_f64(((double)km.x + (double)km.y) * so_d);
    const cf sc = (k * dnorm < 1e-10f) ? cf{0.f, 0.f} : eo;
    const cf Nt[3] = {cf{sv[0], sv[1]}, cf{sv[2], sv[3]}, cf{sv[4], sv[5]}};
    const cf a = cmul(cf{-fmaf(cofd[0], Nt[0].re, fmaf(cofd[1], Nt[1].re, cofd[2] * Nt[2].re)),
                         -fmaf(cofd[0], Nt[0].im, fmaf(cofd[1], Nt[1].im, cofd[2] * Nt[2].im))}, sc);
    float2* out = G + row0 * kg.Q;
#pragma unroll
    for (int rr = 0; rr < 3; ++rr) {  // dA/dt_r = i k d_r A
      const float kd = k * comp(dh, rr);
      o.put(out + (int64_t)rr * kg.Q, cf{-kd * a.im, kd * a.re});
    }
    cf MF[9];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cf v[3];  // e_c x NF
      v[c] = cf{0.f, 0.f};
      v[(c + 1) % 3] = cf{-Nt[(c + 2) % 3].re, -Nt[(c + 2) % 3].im};
      v[(c + 2) % 3] = Nt[(c + 1) % 3];
      cf mv[3];  // A v
#pragma unroll
      for (int a3 = 0; a3 < 3; ++a3) {
        const float x0 = A[3 * a3], x1 = A[3 * a3 + 1], x2 = A[3 * a3 + 2];
        mv[a3] = cf{fmaf(x0, v[0].re, fmaf(x1, v[1].re, x2 * v[2].re)), fmaf(x0, v[0].im, fmaf(x1, v[1].im, x2 * v[2].im))};
      }
      MF[c] = cf{kh.y * mv[2].re - kh.z * mv[1].re, kh.y * mv[2].im - kh.z * mv[1].im};
      MF[3 + c] = cf{kh.z * mv[0].re - kh.x * mv[2].re, kh.z * mv[0].im - kh.x * mv[2].im};
      MF[6 + c] = cf{kh.x * mv[1].re - kh.y * mv[0].re, kh.x * mv[1].im - kh.y * mv[0].im};
    }
#pragma unroll
    for (int rr = 0; rr < 3; ++rr)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const cf mf = MF[3 * rr + c], w = cf{sv[6 + 2 * c], sv[7 + 2 * c]};
        const float kd = k * comp(dh, rr);
        const cf v = cmul(cf{-2.0f * (mf.re + kd * w.re), -2.0f * (mf.im + kd * w.im)}, sc);
        o.put(out + (int64_t)(3 + 3 * rr + c) * kg.Q, v);
      }
  }
};

// Reference-frame values of one element: its first vertex a0, edges E1, E2 and
// doubled area vector N0 = E1 x E2.
struct TriRef { float a0[3], E1[3], E2[3], N0[3]; };

__device__ __forceinline__ TriRef tri_ref(const TriSrcJ& s) {
  TriRef t;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    t.a0[c] = (float)s.a[c];
    t.E1[c] = (float)s.e1[c];
    t.E2[c] = (float)s.e2[c];
    t.N0[c] = (float)(s.e1[(c + 1) % 3] * s.e2[(c + 2) % 3] - s.e1[(c + 2) % 3] * s.e2[(c + 1) % 3]);
  }
  return t;
}

// ---- AffineDoF triangles -------------------------------------------------------------
// A thread owns one direction and R neighbouring radii (the warp 32
// directions, the CTA 4 neighbouring direction blocks of one radial block).
// R = 4 (three CTAs per SM: 168 registers, 70 KB of shared memory each)
// where the launch has at least two waves of CTAs; two radii per thread for
// small launches (one moving mesh of the alignment caller), which would
// otherwise leave SMs idle, and then four CTAs per SM (128 registers without
// spills; three took 1.40 ms an alignment step, four 1.33).
// Per element and direction the small-spread series of F, D_b and D_c are
// formed once as polynomials in k (tri_der_coeffs), so a radius costs a table
// phasor, the Horner chains (cut after h_8 where k |e|max < 1, a test that is
// the same for the whole warp on a tensor grid) and three complex products.
// Radial blocks run heavy-first and the CTA order is re-mapped so that every
// object's heavy blocks start first, as in ff_kernel.  Per radius and node
// six complex sums, chunked in FP32 and Kahan-compensated in shared memory:
//   NF += F N0,  N0 = E1 x E2 (reference edges)
//   W  += gamma (i F a0 + D_b E1 + D_c E2)             (sum_s D_s x0_s, D_a + D_b + D_c = i F)
// (JacWriter forms the 12 derivatives from them.)  The radii of the cluster
// expansions (jac_moment_kernel) are left out; the CTAs of a thread-block
// cluster split the elements, as in ff_kernel.

template <int R>
__global__ void __launch_bounds__(JAC_THREADS, R == 2 ? 4 : 3)
jac_affine_tri_kernel(KGridDev kg, BatchDev b, const JacObj* __restrict__ jobs, float2* __restrict__ G) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const unsigned lin = (blockIdx.y * gridDim.x + blockIdx.x) / (unsigned)S;
  const int slot = (int)(lin % gridDim.y), cta = (int)(lin / gridDim.y);
  const JacObj jo = jobs[slot];
  const ObjDev od = b.objs[jo.obj];
  const int r_first = jac_moment_radii(kg, __uint_as_float(b.cl_rho[jo.obj]), R == 4 ? JM_SPARE : 0);
  const int nrb = (kg.L - r_first + R - 1) / R, ndt = (kg.Me + 31) / 32;
  if (cta * JAC_WARPS >= ndt * nrb) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = cta * JAC_WARPS + warp;
  const int ib = item / ndt, dt = item - ib * ndt;
  const int rlo = kg.L - (ib + 1) * R, skip = max(0, r_first - rlo);  // radii rlo + i, i >= skip
  const int ei = dt * 32 + lane;
  const bool active = item < ndt * nrb && ei < kg.Me;
  int j = 0, jm = -1;  // direction evaluated, its antipode written from it (or -1)
  if (active) { const int2 pr = kg.dpair[ei]; j = pr.x; jm = pr.y; }
  float3 dh = make_float3(0.f, 0.f, 0.f), dl = dh;
  float inv_norm = 0.f, dnorm = 0.f;
  if (active) {
    const float4 h = kg.dir_hi[j], l = kg.dir_lo[j];
    dh = make_float3(h.x, h.y, h.z);
    dl = make_float3(l.x, l.y, l.z);
    inv_norm = h.w;
    dnorm = l.w;
  }
  __shared__ float4 tile[7 * JAC_TILE];
  __shared__ float2 ctab_sm[PHASOR_ENTRIES * JAC_COPIES];
  const float2* ctab = ctab_sm + (threadIdx.x % JAC_COPIES);
  __shared__ float4 krad[JAC_WARPS][R];  // (|k| hi, lo, |k| 64 / 2 pi hi, lo)
  __shared__ float run[2 * JAC_NSUM * R * JAC_THREADS];  // running sums, then compensations
  stage_phasors<JAC_COPIES>(kg.cis_tab, ctab_sm);
  if (lane < R) {
    const int r = rlo + lane;
    const bool ok = item < ndt * nrb && lane >= skip;
    const float2 km = ok ? kg.kmag[r] : make_float2(0.f, 0.f);
    const float2 kt = ok ? kg.kt64[r] : make_float2(0.f, 0.f);
    krad[warp][lane] = make_float4(km.x, km.y, kt.x, kt.y);
  }
  for (int v = 0; v < 2 * JAC_NSUM * R; ++v) run[v * JAC_THREADS + threadIdx.x] = 0.f;
  float acc[R][JAC_NSUM];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int v = 0; v < JAC_NSUM; ++v) acc[i][v] = 0.f;
  // adds the chunk's partials to the compensated running sums
  auto flush = [&]() {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int v = 0; v < JAC_NSUM; ++v) {
        float* ps = run + (i * JAC_NSUM + v) * JAC_THREADS + threadIdx.x;
        float* pc = ps + JAC_NSUM * R * JAC_THREADS;
        const float sum = *ps, y = acc[i][v] - *pc, t = sum + y;
        *pc = (t - sum) - y;
        *ps = t;
        acc[i][v] = 0.f;
      }
  };
  const float4* pool = b.tri_pool + 3 * od.elem_off;
  const float4* pool_lo = b.tri_lo + od.elem_off;
  const TriSrcJ* src = reinterpret_cast<const TriSrcJ*>(jo.src);
  const int per = (od.n_elems + S * 16 - 1) / (S * 16) * 16;  // this CTA's elements, whole chunks
  const int n0 = min(od.n_elems, rank * per), n1 = min(od.n_elems, n0 + per);
  for (int base = n0; base < n1; base += JAC_TILE) {
    const int cnt = min(JAC_TILE, n1 - base);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt; e += JAC_THREADS) {
      tile[6 * e] = pool[3 * (int64_t)(base + e)];
      tile[6 * e + 1] = pool[3 * (int64_t)(base + e) + 1];
      tile[6 * e + 2] = pool[3 * (int64_t)(base + e) + 2];
      const TriRef t = tri_ref(src[od.perm_off >= 0 ? b.perm[od.perm_off + base + e] : base + e]);
      tile[6 * e + 3] = make_float4(t.a0[0], t.a0[1], t.a0[2], t.N0[0]);
      tile[6 * e + 4] = make_float4(t.E1[0], t.E1[1], t.E1[2], t.N0[1]);
      tile[6 * e + 5] = make_float4(t.E2[0], t.E2[1], t.E2[2], t.N0[2]);
      tile[6 * JAC_TILE + e] = pool_lo[base + e];  // centroid low word, longest edge
    }
    __syncthreads();
    if (!active) continue;
    for (int e = 0; e < cnt; ++e) {
      const float4 q0 = tile[6 * e], q1 = tile[6 * e + 1], q2 = tile[6 * e + 2], ql = tile[6 * JAC_TILE + e];
      const float3 m = make_float3(q0.x, q0.y, q0.z), e1 = make_float3(q1.x, q1.y, q1.z),
                   e2 = make_float3(q2.x, q2.y, q2.z);
      const df sm = cdot2(dh, dl, m, make_float3(ql.x, ql.y, ql.z)), d1 = cdot(dh, dl, e1), d2 = cdot(dh, dl, e2);
      const float sp = fmaxf(fmaxf(fabsf(d1.hi), fabsf(d2.hi)), fabsf(d2.hi - d1.hi));
      const float kthr = __fdividef(2.0f, sp);           // the series for k sp < 2 (inf when sp = 0)
      const float kshort = rcp_fast(ql.w * dnorm);       // cut after h_8 for k |e|max < 1
      const float gam = (dh.x * q0.w + dh.y * q1.w + dh.z * q2.w) * inv_norm;
      const TriDerPoly cp = tri_der_coeffs(d1.hi, d2.hi);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (i < skip) continue;
        const float4 kr = krad[warp][i];
        const float k = kr.x;
        cf F, Db, Dc;
        if (k < kthr) {
          const cf P = cis_tab_df<JAC_COPIES>(ctab, make_float2(kr.z, kr.w), sm);
          const float u = k * k;
          float fre, fim, bre, bim, cre, cim;
          if (k < kshort) {
            fre = poly_first<5>(cp.fa, u); fim = poly_first<3>(cp.fb, u);
            bim = poly_first<5>(cp.ba, u); bre = poly_first<4>(cp.bb, u);
            cim = poly_first<5>(cp.ca, u); cre = poly_first<4>(cp.cb, u);
          } else {
            fre = poly_u(cp.fa, u); fim = poly_u(cp.fb, u);
            bim = poly_u(cp.ba, u); bre = poly_u(cp.bb, u);
            cim = poly_u(cp.ca, u); cre = poly_u(cp.cb, u);
          }
          F = cmul(P, cf{fre, u * k * fim});
          Db = cmul(P, cf{k * bre, bim});
          Dc = cmul(P, cf{k * cre, cim});
        } else {
          const df sa = df_add(sm, df_div3(df_add(d1, d2)) * -1.0f);
          const TriDer d = tri_generic_der_at<JAC_COPIES>(ctab, make_float2(kr.z, kr.w), sa, df_add(sa, d1), df_add(sa, d2),
                                              k * d1.hi, k * d2.hi);
          F = d.F;
          Db = d.Db;
          Dc = d.Dc;
        }
        const float4 ta = tile[6 * e + 3], tb = tile[6 * e + 4], tc = tile[6 * e + 5];
        acc[i][0] = fmaf(F.re, ta.w, acc[i][0]);
        acc[i][1] = fmaf(F.im, ta.w, acc[i][1]);
        acc[i][2] = fmaf(F.re, tb.w, acc[i][2]);
        acc[i][3] = fmaf(F.im, tb.w, acc[i][3]);
        acc[i][4] = fmaf(F.re, tc.w, acc[i][4]);
        acc[i][5] = fmaf(F.im, tc.w, acc[i][5]);
        const cf gF = cscale(F, gam), gB = cscale(Db, gam), gC = cscale(Dc, gam);
        const float a0[3] = {ta.x, ta.y, ta.z}, E1[3] = {tb.x, tb.y, tb.z}, E2[3] = {tc.x, tc.y, tc.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[i][6 + 2 * c] = fmaf(-gF.im, a0[c], fmaf(gB.re, E1[c], fmaf(gC.re, E2[c], acc[i][6 + 2 * c])));
          acc[i][7 + 2 * c] = fmaf(gF.re, a0[c], fmaf(gB.im, E1[c], fmaf(gC.im, E2[c], acc[i][7 + 2 * c])));
        }
      }
      if ((e & 15) == 15) flush();
    }
    flush();
  }
  const auto mine = [&](int i) { return (i & (S - 1)) == rank; };  // S is a power of two
  if (S > 1) {
    cluster.sync();
    float tot[R][JAC_NSUM];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!mine(i)) continue;
#pragma unroll
      for (int v = 0; v < JAC_NSUM; ++v) {
        kbsum t{0.f, 0.f};
        for (int q = 0; q < S; ++q) {
          const float* o = cluster.map_shared_rank(run, q) + (i * JAC_NSUM + v) * JAC_THREADS + threadIdx.x;
          t.add(o[0]);
          t.lo -= o[JAC_NSUM * R * JAC_THREADS];
        }
        tot[i][v] = t.hi + t.lo;
      }
    }
    cluster.sync();  // no CTA leaves, or overwrites them, while its sums are read
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (mine(i))
#pragma unroll
        for (int v = 0; v < JAC_NSUM; ++v) run[(i * JAC_NSUM + v) * JAC_THREADS + threadIdx.x] = tot[i][v];
  }
  if (!active) return;
  const JacWriter w(jo, od, dh, dl, inv_norm, dnorm, j, jm);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (i < skip || !mine(i)) continue;
    const float4 kr = krad[warp][i];
    float sv[JAC_NSUM];
#pragma unroll
    for (int v = 0; v < JAC_NSUM; ++v) sv[v] = run[(i * JAC_NSUM + v) * JAC_THREADS + threadIdx.x];
    w.put(kg, G, rlo + i, make_float2(kr.x, kr.y), sv);
  }
}

// The sums NF and W at small k from cluster expansions (moments.cu): with the
// vertices' projections a, b, c from the cluster's centre, F = e^{ik.c} sum_n
// i^{n+2} k^n h_n(a, b, c)/(n+2)! and D_b = e^{ik.c} sum_n i^{n+3} k^n
// h_n(a, b, b, c)/(n+3)!, so
//   NF:  sum_n i^{n+2} k^n / (n+2)! sum_e N0 h_n
//   W: i sum_n i^{n+2} k^n / (n+3)! sum_e gamma (a0 (n+3) h_n + E1 h_n(a,b,b,c) + E2 h_n(a,b,c,c)).
// One CTA owns one object, 32 evaluated directions (one per lane) and up to
// JM_RADII of the covered radii, and alternates between two phases over tiles
// of four clusters: two warps per cluster form its 6 x 16 real moments (the
// recurrences in both, NF and W_x in one, W_y and W_z in the other: ~190 FP32
// operations per element, direction and warp for all radii, where the direct
// sum takes ~190 for each), then each warp sums the tile over its own radii,
// JM_R at a time.  The CTAs of a thread-block cluster split the tiles.
constexpr int JM_WARPS = 8, JM_THREADS = 32 * JM_WARPS, JM_TILE = JM_WARPS / 2;
constexpr int JM_SETS = JAC_NSUM / 2, JM_R = 3;
static_assert(JM_RADII == 2 * JM_R * JM_WARPS, "two batches of radii per warp");
// staged element pairs, as float4: vertices, S, N0, a0, E1, E2 (24 values of
// two elements, and one float4 that spreads the pairs over the banks)
constexpr int JM_PAIR_F4 = 13;

// float4 counts: staged elements, coefficients, running sums (and compensations)
constexpr int JM_F4_ELEM = JM_TILE * PI_CLUSTER / 2 * JM_PAIR_F4, JM_F4_MOM = JM_TILE * JM_SETS * 4 * 32,
              JM_F4_RUN = JM_RADII * JAC_NSUM * 2 * 32 / 4;
constexpr int JM_SMEM = (JM_F4_ELEM + JM_F4_MOM + JM_F4_RUN) * (int)sizeof(float4);

template <int HALF>
__device__ __forceinline__ void jac_moments(const float4* es, int cnt, float3 d, float inv_norm, float4* mom,
                                            kbsum (&zero)[4]) {
  constexpr int NS = HALF == 0 ? 4 : 2;  // sets of this warp: NF, W_x / W_y, W_z
  float2 mu[NS][MOMENT_TERMS];
#pragma unroll
  for (int v = 0; v < NS; ++v)
#pragma unroll
    for (int n = 0; n < MOMENT_TERMS; ++n) mu[v][n] = make_float2(0.f, 0.f);
  float2 zc[NS];  // compensations of the zeroth moments
#pragma unroll
  for (int v = 0; v < NS; ++v) zc[v] = make_float2(0.f, 0.f);
  const float2 dx = dup2(d.x), dy = dup2(d.y), dz = dup2(d.z), in2 = dup2(inv_norm);
#pragma unroll 1
  for (int i = 0; i < cnt; i += 2, es += JM_PAIR_F4) {
    // value c of the two elements
    const auto val = [&](int c) {
      const float4 q = es[c / 2];
      return (c & 1) ? make_float2(q.z, q.w) : make_float2(q.x, q.y);
    };
    const auto dot = [&](int c) { return __ffma2_rn(dx, val(c), __ffma2_rn(dy, val(c + 1), __fmul2_rn(dz, val(c + 2)))); };
    const float2 a = dot(0), bb = dot(3), c = dot(6), g = __fmul2_rn(dot(9), in2);
    const float2 N0[3] = {val(12), val(13), val(14)};
    float2 w0[2], w1[2], w2[2];  // gamma a0, gamma E1, gamma E2
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int x = HALF == 0 ? 0 : 1 + v;
      w0[v] = __fmul2_rn(g, val(15 + x));
      w1[v] = __fmul2_rn(g, val(18 + x));
      w2[v] = __fmul2_rn(g, val(21 + x));
    }
    float2 an = dup2(1.f), qn = an, hn = an, hb = an, hc = an;
#pragma unroll
    for (int n = 0; n < MOMENT_TERMS; ++n) {
      if (n > 0) {
        an = __fmul2_rn(an, a);
        qn = __ffma2_rn(bb, qn, an);
        hn = __ffma2_rn(c, hn, qn);
        hb = __ffma2_rn(bb, hb, hn);
        hc = __ffma2_rn(c, hc, hn);
      }
      const float2 hw = make_float2((float)(n + 3) * hn.x, (float)(n + 3) * hn.y);
      if (n == 0) {  // h's are 1
#pragma unroll
        for (int v = 0; v < NS; ++v) {
          const int x = HALF == 0 ? 0 : v;
          const float2 w3 = make_float2(3.f * w0[x].x, 3.f * w0[x].y);
          kahan2(mu[v][0], zc[v], HALF == 0 && v < 3 ? N0[v] : __fadd2_rn(w3, __fadd2_rn(w1[x], w2[x])));
        }
      } else if (HALF == 0) {
#pragma unroll
        for (int v = 0; v < 3; ++v) mu[v][n] = __ffma2_rn(N0[v], hn, mu[v][n]);
        mu[NS - 1][n] = __ffma2_rn(w0[0], hw, __ffma2_rn(w1[0], hb, __ffma2_rn(w2[0], hc, mu[NS - 1][n])));
      } else {
#pragma unroll
        for (int v = 0; v < 2; ++v)
          mu[v][n] = __ffma2_rn(w0[v], hw, __ffma2_rn(w1[v], hb, __ffma2_rn(w2[v], hc, mu[v][n])));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NS; ++v) {
    zero[v].add(mu[v][0].x);
    zero[v].add(mu[v][0].y);
    zero[v].lo -= zc[v].x + zc[v].y;
  }
  constexpr FmConst<PI_GEOM_TRIANGLE> C{};  // 2/(n+2)!
#pragma unroll
  for (int v = 0; v < NS; ++v) {
    const int set = HALF == 0 ? v : 4 + v;
    float o[MOMENT_TERMS];
#pragma unroll
    for (int n = 0; n < MOMENT_TERMS; ++n) {  // i^{n+2}: real for even n, imaginary for odd n
      const float f = (set < 3 ? 0.5f : 0.5f / (n + 3)) * C.f[n];
      o[(n & 1) * (MOMENT_TERMS / 2) + n / 2] = (mu[v][n].x + mu[v][n].y) * ((n & 2) ? f : -f);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) mom[(set * 4 + t) * 32] = make_float4(o[4 * t], o[4 * t + 1], o[4 * t + 2], o[4 * t + 3]);
  }
}

__global__ void __launch_bounds__(JM_THREADS, 1)
jac_moment_kernel(KGridDev kg, BatchDev b, const JacObj* __restrict__ jobs, float2* __restrict__ G, int groups,
                  int spare) {
  extern __shared__ float4 jsm[];
  float4* elem = jsm;
  float4* mom = elem + JM_F4_ELEM;
  float* run = reinterpret_cast<float*>(mom + JM_F4_MOM);  // [radius][sum or compensation][lane]
  __shared__ float2 ctab_sm[PHASOR_ENTRIES * JAC_COPIES], csc[JM_TILE][32];
  __shared__ float4 krad[JM_RADII];  // |k|, |k| 64 / 2 pi hi, lo
  __shared__ float cscale[JM_TILE];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const unsigned lin = (blockIdx.y * gridDim.x + blockIdx.x) / (unsigned)S;
  const int slot = (int)(lin % gridDim.y), item = (int)(lin / gridDim.y);
  const int dt = item / groups, r0 = (item - dt * groups) * JM_RADII;
  const JacObj jo = jobs[slot];
  const ObjDev od = b.objs[jo.obj];
  const int nr = min(JM_RADII, jac_moment_radii(kg, __uint_as_float(b.cl_rho[jo.obj]), spare) - r0);  // radii r0 .. r0 + nr - 1
  if (nr <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ei = dt * 32 + lane;
  const bool active = ei < kg.Me;
  int j = 0, jm = -1;
  float3 dh = make_float3(0.f, 0.f, 0.f), dl = dh;
  float inv_norm = 0.f, dnorm = 0.f;
  if (active) {
    const int2 pr = kg.dpair[ei];
    j = pr.x;
    jm = pr.y;
    const float4 h = kg.dir_hi[j], l = kg.dir_lo[j];
    dh = make_float3(h.x, h.y, h.z);
    dl = make_float3(l.x, l.y, l.z);
    inv_norm = h.w;
    dnorm = l.w;
  }
  stage_phasors<JAC_COPIES>(kg.cis_tabm, ctab_sm);
  const float2* ctab = ctab_sm + (threadIdx.x % JAC_COPIES);
  // this warp's clusters' zeroth moments: they are the same at every radius, and
  // what they leave of each other is a closed surface's value at small k
  // (moments.cu), so they are summed apart and e^{ik.c} enters less 1
  kbsum zero[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  for (int t = threadIdx.x; t < JM_RADII; t += JM_THREADS) {
    const bool ok = t < nr;
    const float2 km = ok ? kg.kmag[r0 + t] : make_float2(0.f, 0.f), kt = ok ? kg.kt64[r0 + t] : make_float2(0.f, 0.f);
    krad[t] = make_float4(km.x, kt.x, kt.y, km.y);
  }
  for (int t = threadIdx.x; t < JM_F4_RUN; t += JM_THREADS) reinterpret_cast<float4*>(run)[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  const TriSrcJ* src = reinterpret_cast<const TriSrcJ*>(jo.src);
  const int ncl = (od.n_elems + PI_CLUSTER - 1) / PI_CLUSTER;
  for (int t0 = rank * JM_TILE; t0 < ncl; t0 += S * JM_TILE) {
    __syncthreads();  // the last tile's elements and coefficients have been read
    // stage the tile's elements relative to their clusters' centres, in units of s
    for (int t = threadIdx.x; t < JM_TILE * PI_CLUSTER; t += JM_THREADS) {
      const int p = t0 * PI_CLUSTER + t;
      float2* d = reinterpret_cast<float2*>(elem + (size_t)(t / 2) * JM_PAIR_F4);
      const auto put = [&](int c, float v) { reinterpret_cast<float*>(d + c)[t & 1] = v; };
      if (p >= od.n_elems) {  // the missing half of the last pair
        for (int c = 0; c < 24; ++c) put(c, 0.f);
        continue;
      }
      const float4 ctr = b.clusters[od.cl_off + p / PI_CLUSTER];
      const int ex = ctr.w > 0.f ? min(120, max(-100, ilogbf(ctr.w) + 1)) : 0;
      const float inv_s = __int_as_float((127 - ex) << 23);
      const int64_t e = od.elem_off + p;
      const float4 q0 = b.tri_pool[3 * e], q1 = b.tri_pool[3 * e + 1], q2 = b.tri_pool[3 * e + 2], lo = b.tri_lo[e];
      const float m[3] = {(q0.x - ctr.x) + lo.x, (q0.y - ctr.y) + lo.y, (q0.z - ctr.z) + lo.z};
      const float e1[3] = {q1.x, q1.y, q1.z}, e2[3] = {q2.x, q2.y, q2.z};
      const TriRef f = tri_ref(src[od.perm_off >= 0 ? b.perm[od.perm_off + p] : p]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float a = m[c] - (e1[c] + e2[c]) * (1.0f / 3.0f);
        put(c, a * inv_s);
        put(3 + c, (a + e1[c]) * inv_s);
        put(6 + c, (a + e2[c]) * inv_s);
        put(9 + c, c == 0 ? q0.w : (c == 1 ? q1.w : q2.w));
        put(12 + c, f.N0[c]);
        put(15 + c, f.a0[c]);
        put(18 + c, f.E1[c]);
        put(21 + c, f.E2[c]);
      }
    }
    __syncthreads();
    const int c_own = warp >> 1, cl = t0 + c_own;
    if (cl < ncl) {
      const int cnt = min(PI_CLUSTER, od.n_elems - cl * PI_CLUSTER);
      const float4* es = elem + (size_t)c_own * (PI_CLUSTER / 2) * JM_PAIR_F4;
      float4* mo = mom + c_own * JM_SETS * 4 * 32 + lane;
      if (warp & 1) {
        jac_moments<1>(es, cnt, dh, inv_norm, mo, zero);
        const float4 ctr = b.clusters[od.cl_off + cl];
        const int ex = ctr.w > 0.f ? min(120, max(-100, ilogbf(ctr.w) + 1)) : 0;
        const df sc = cdot(dh, dl, make_float3(ctr.x, ctr.y, ctr.z));
        csc[c_own][lane] = make_float2(sc.hi, sc.lo);
        if (lane == 0) cscale[c_own] = __int_as_float((127 + ex) << 23);
      } else {
        jac_moments<0>(es, cnt, dh, inv_norm, mo, zero);
      }
    }
    __syncthreads();
    const int nc = min(JM_TILE, ncl - t0);
    for (int rb = warp * JM_R; rb < nr; rb += JM_WARPS * JM_R) {
      float acc[JM_R][JAC_NSUM];
#pragma unroll
      for (int i = 0; i < JM_R; ++i)
#pragma unroll
        for (int v = 0; v < JAC_NSUM; ++v) acc[i][v] = 0.f;
#pragma unroll 1
      for (int c = 0; c < nc; ++c) {
        const float2 sc = csc[c][lane];
        const float s = cscale[c];
        cf M[JM_R];
        float k[JM_R];
#pragma unroll
        for (int i = 0; i < JM_R; ++i) {
          const float4 kr = krad[rb + i];
          M[i] = cis_tab_m1_df<JAC_COPIES>(ctab, make_float2(kr.y, kr.z), df{sc.x, sc.y});
          k[i] = kr.x * s;
        }
#pragma unroll
        for (int v = 0; v < JM_SETS; ++v) {
          const float4* mo = mom + (c * JM_SETS + v) * 4 * 32 + lane;
          const float4 m0 = mo[0], m1 = mo[32], m2 = mo[64], m3 = mo[96];
#pragma unroll
          for (int i = 0; i < JM_R; ++i) {
            const float u = k[i] * k[i];
            const float xr = u * fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, m1.w, m1.z), m1.y), m1.x), m0.w), m0.z), m0.y);
            const float x = xr + m0.x;
            const float y = k[i] * fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, m3.w, m3.z), m3.y), m3.x), m2.w), m2.z), m2.y), m2.x);
            acc[i][2 * v] += fmaf(M[i].re, x, fmaf(-M[i].im, y, xr));
            acc[i][2 * v + 1] += fmaf(M[i].re, y, fmaf(M[i].im, x, y));
          }
        }
      }
#pragma unroll
      for (int i = 0; i < JM_R; ++i)
#pragma unroll
        for (int v = 0; v < JAC_NSUM; ++v) {
          float* ps = run + ((rb + i) * 2 * JAC_NSUM + 2 * v) * 32 + lane;
          const float sum = ps[0], y = acc[i][v] - ps[32], t = sum + y;
          ps[32] = (t - sum) - y;
          ps[0] = t;
        }
    }
  }
  __syncthreads();  // the last tile's elements have been read: their place takes the zeroth moments
  float2* zs = reinterpret_cast<float2*>(elem);  // [cluster of the tile][set][lane]
#pragma unroll
  for (int v = 0; v < 4; ++v)
    if ((warp & 1) == 0 || v < 2)
      zs[((warp >> 1) * JM_SETS + 4 * (warp & 1) + v) * 32 + lane] = make_float2(zero[v].hi, zero[v].lo);
  if (S > 1) cluster.sync();
  else __syncthreads();
  if (active) {
    const JacWriter w(jo, od, dh, dl, inv_norm, dnorm, j, jm);
    kbsum zt[JM_SETS];
#pragma unroll
    for (int v = 0; v < JM_SETS; ++v) {
      zt[v] = kbsum{0.f, 0.f};
      for (int q = 0; q < S * JM_TILE; ++q) {
        const float2* o = S > 1 ? cluster.map_shared_rank(zs, q / JM_TILE) : zs;
        const float2 z = o[((q % JM_TILE) * JM_SETS + v) * 32 + lane];
        zt[v].add(z.x);
        zt[v].lo += z.y;
      }
      const float f = v < 3 ? -0.5f : -1.0f / 6.0f, p = zt[v].hi * f;  // i^2 / 2!, i^2 / 3!
      zt[v] = kbsum{p, fmaf(zt[v].hi, f, -p) + zt[v].lo * f};
    }
    for (int r = warp * S + rank; r < nr; r += JM_WARPS * S) {
      float sv[JAC_NSUM];
#pragma unroll
      for (int v = 0; v < JAC_NSUM; ++v) {
        kbsum t{0.f, 0.f};
        for (int q = 0; q < S; ++q) {
          const float* o = (S > 1 ? cluster.map_shared_rank(run, q) : run) + (r * 2 * JAC_NSUM + 2 * v) * 32 + lane;
          t.add(o[0]);
          t.lo -= o[32];
        }
        if ((v & 1) == 0) {
          t.add(zt[v / 2].hi);
          t.lo += zt[v / 2].lo;
        }
        sv[v] = t.hi + t.lo;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {  // W = i times the sum
        const float re = sv[6 + 2 * c];
        sv[6 + 2 * c] = -sv[7 + 2 * c];
        sv[7 + 2 * c] = re;
      }
      const float4 kr = krad[r];
      w.put(kg, G, r0 + r, make_float2(kr.x, kr.w), sv);
    }
  }
  if (S > 1) cluster.sync();  // no CTA leaves while its sums are read
}

// ---- AffineDoF disks / Gaussians --------------------------------------------------------
__global__ void __launch_bounds__(JAC_THREADS)
jac_affine_surf_kernel(KGridDev kg, BatchDev b, const JacObj* __restrict__ jobs, float2* __restrict__ G) {
  const JacObj jo = jobs[blockIdx.y];
  const ObjDev od = b.objs[jo.obj];
  const JacThread t = jac_thread(kg);
  const bool disk = od.type == PI_GEOM_DISK;
  __shared__ float4 tile[6 * JAC_TILE];
  __shared__ float2 ctab_sm[PHASOR_ENTRIES * JAC_COPIES];
  const float2* ctab = ctab_sm + (threadIdx.x % JAC_COPIES);
  stage_cis_tab(kg, ctab_sm);
  // v = A^T dir (k' = |k| v), qd = |v|^2
  const float* Af = od.A;
  const float3 v = make_float3(Af[0] * t.dh.x + Af[3] * t.dh.y + Af[6] * t.dh.z,
                               Af[1] * t.dh.x + Af[4] * t.dh.y + Af[7] * t.dh.z,
                               Af[2] * t.dh.x + Af[5] * t.dh.y + Af[8] * t.dh.z);
  const float qd = fmaf(v.x, v.x, fmaf(v.y, v.y, v.z * v.z));
  kcf A, Z[3], N[3], Y;
  const float4* pool = b.surf_pool + 2 * od.elem_off;
  const float4* pool_lo = b.surf_lo + od.elem_off;
  const float4* pool_nref = b.surf_nref + od.elem_off;
  const SurfSrcJ* src = reinterpret_cast<const SurfSrcJ*>(jo.src);
  const float k = t.k.hi, k2 = k * k;
  for (int base = 0; base < od.n_elems; base += JAC_TILE) {
    const int cnt = min(JAC_TILE, od.n_elems - base);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt; e += JAC_THREADS) {
      tile[4 * e] = pool[2 * (int64_t)(base + e)];
      tile[4 * e + 1] = pool[2 * (int64_t)(base + e) + 1];
      const SurfSrcJ& s = src[od.perm_off >= 0 ? b.perm[od.perm_off + base + e] : base + e];  // reference centre c0 and normal n0
      tile[4 * e + 2] = make_float4((float)s.c[0], (float)s.c[1], (float)s.c[2], 0.f);
      tile[4 * e + 3] = make_float4((float)s.n[0], (float)s.n[1], (float)s.n[2], 0.f);
      tile[4 * JAC_TILE + e] = pool_lo[base + e];  // centre low word
      tile[5 * JAC_TILE + e] = pool_nref[base + e];  // (n / |n|, 1 - |n|^2)
    }
    __syncthreads();
    if (!t.active) continue;
    for (int e = 0; e < cnt; ++e) {
      const float4 q0 = tile[4 * e], q1 = tile[4 * e + 1], c0 = tile[4 * e + 2], n0 = tile[4 * e + 3];
      const float4 cl = tile[4 * JAC_TILE + e];
      const df sc = cdot2(t.dh, t.dl, make_float3(q0.x, q0.y, q0.z), make_float3(cl.x, cl.y, cl.z));
      const float sn = t.dh.x * q1.x + t.dh.y * q1.y + t.dh.z * q1.z;
      // |k'_perp|^2 / |k|^2 = qd (1 - |n|^2) + |n|^2 |v x n/|n||^2 (no cancellation near the normal)
      const float4 nr = tile[5 * JAC_TILE + e];
      const float cx = fmaf(v.y, nr.z, -v.z * nr.y), cy = fmaf(v.z, nr.x, -v.x * nr.z),
                  cz = fmaf(v.x, nr.y, -v.y * nr.x);
      const float perp = fmaxf(fmaf(qd, nr.w, (1.0f - nr.w) * fmaf(cx, cx, fmaf(cy, cy, cz * cz))), 0.f);
      const float amp = sn * t.inv_norm;
      const cf P = cis_tab_df<JAC_COPIES>(ctab, t.kt, sc);
      float S, Sr;
      if (disk) {
        const float x = k * q0.w * sqrt_fast(perp);
        S = q1.w * ((x < 1e-10f) ? 1.0f : 2.0f * j1x(x));
        Sr = -2.0f * q1.w * q0.w * q0.w * j2x2(x);
      } else {
        S = q1.w * __expf(-0.5f * q0.w * q0.w * k2 * perp);
        Sr = -q0.w * q0.w * S;
      }
      const float sa = S * amp, sn_t = S - k2 * sn * sn * Sr;
      A.fma_add(P, sa);
      Z[0].fma_add(P, sa * c0.x); Z[1].fma_add(P, sa * c0.y); Z[2].fma_add(P, sa * c0.z);
      N[0].fma_add(P, sn_t * n0.x); N[1].fma_add(P, sn_t * n0.y); N[2].fma_add(P, sn_t * n0.z);
      Y.fma_add(P, amp * Sr);
      if ((e & 15) == 15) {
        A.flush(); Y.flush();
#pragma unroll
        for (int a = 0; a < 3; ++a) { Z[a].flush(); N[a].flush(); }
      }
    }
    A.flush(); Y.flush();
#pragma unroll
    for (int a = 0; a < 3; ++a) { Z[a].flush(); N[a].flush(); }
  }
  if (!t.active) return;
  const JacOut o = jac_out(kg, t.r, t.j, t.jm);
  const cf scl = jac_origin_phase(t, od);
  const double* Am = jo.dofs + 3;  // A row-major
  float atd[3];  // (A^T d)_c = sum_p d_p A_pc
#pragma unroll
  for (int c = 0; c < 3; ++c)
    atd[c] = (float)(t.dh.x * Am[c] + t.dh.y * Am[3 + c] + t.dh.z * Am[6 + c]);
  const cf a = cmul(A.value(), scl), y = Y.value();
  float2* out = G + jo.row0 * kg.Q;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const float kr = k * comp(t.dh, r);
    o.put(out + (int64_t)r * kg.Q, cf{-kr * a.im, kr * a.re});
  }
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float dr = comp(t.dh, r);
      const cf z = Z[c].value(), nn = N[c].value();
      // i k d_r Z_c + khat_r N_c + k^2 d_r (A^T d)_c Y
      const float f = k2 * dr * atd[c], g = dr * t.inv_norm, kd = k * dr;
      const cf v = cmul(cf{-kd * z.im + g * nn.re + f * y.re, kd * z.re + g * nn.im + f * y.im}, scl);
      o.put(out + (int64_t)(3 + 3 * r + c) * kg.Q, v);
    }
}

// ---- TriangleMeshDoF: vertex gather --------------------------------------------------------
__global__ void __launch_bounds__(JAC_THREADS)
jac_mesh_kernel(KGridDev kg, BatchDev b, const JacObj* __restrict__ jobs, const int64_t* __restrict__ vrow,
                const int64_t* __restrict__ vent, const int64_t* __restrict__ vmap, float2* __restrict__ G) {
  const JacObj jo = jobs[blockIdx.y];
  const ObjDev od = b.objs[jo.obj];
  const JacThread t = jac_thread(kg);
  __shared__ float2 ctab_sm[PHASOR_ENTRIES * JAC_COPIES];
  const float2* ctab = ctab_sm + (threadIdx.x % JAC_COPIES);
  stage_cis_tab(kg, ctab_sm);
  if (!t.active) return;
  const JacOut o = jac_out(kg, t.r, t.j, t.jm);
  const cf scl = jac_origin_phase(t, od);
  const float k = t.k.hi;
  for (int64_t v = jo.vstart; v < jo.vstart + jo.nverts; ++v) {
    float gr[3] = {0.f, 0.f, 0.f}, gi[3] = {0.f, 0.f, 0.f};
    for (int64_t p = vrow[v]; p < vrow[v + 1]; ++p) {
      const int64_t te = vent[p];  // pool triangle * 3 + slot
      const int64_t tri = te / 3;
      const int slot = (int)(te - 3 * tri);
      const float4 q0 = b.tri_pool[3 * tri], q1 = b.tri_pool[3 * tri + 1], q2 = b.tri_pool[3 * tri + 2];
      const float4 ql = b.tri_lo[tri];
      const TriNode o = tri_node(t, ctab, make_float3(q0.x, q0.y, q0.z), ql, make_float3(q1.x, q1.y, q1.z),
                                 make_float3(q2.x, q2.y, q2.z), make_float3(q0.w, q1.w, q2.w));
      const cf D = slot == 0 ? o.d.Da : (slot == 1 ? o.d.Db : o.d.Dc);
      const float3 cs = o.c[slot];
#pragma unroll
      for (int r = 0; r < 3; ++r) {  // df/dv = -2 (c_s F + gamma k d D_s)
        const float cr = comp(cs, r), gk = o.gam * k * comp(t.dh, r);
        gr[r] += -2.0f * (cr * o.d.F.re + gk * D.re);
        gi[r] += -2.0f * (cr * o.d.F.im + gk * D.im);
      }
    }
    const int64_t row = vmap[v];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      o.put(G + (row + r) * kg.Q, cmul(cf{gr[r], gi[r]}, scl));
    }
  }
}

}  // namespace

int launch_jacobian(const pi_kgrid_impl* kg, const pi_batch_impl* b, float2* G, cudaStream_t s) {
  std::vector<JacObj> tri, surf, mesh;
  int64_t row = 0, vstart = 0;
  for (int i = 0; i < b->n_obj; ++i) {
    const HostObjInfo& in = b->info[i];
    JacObj o{};
    o.obj = i;
    o.row0 = row;
    o.src = static_cast<const unsigned char*>(b->d_src) + in.src_off;
    o.dofs = b->d_dofs + in.dof_off;
    if (in.dof_type == PI_DOF_TRIANGLE_MESH) {
      o.kind = JAC_MESH_TRI;
      o.vstart = vstart;
      o.nverts = in.n_dofs / 3;
      vstart += o.nverts;
      mesh.push_back(o);
    } else if (in.n_dofs != 12) {
      return fail(PI_ERR_UNSUPPORTED, "the Jacobian supports AffineDoF (12) and TriangleMeshDoF objects");
    } else if (in.geom_type == PI_GEOM_TRIANGLE) {
      o.kind = JAC_AFFINE_TRI;
      tri.push_back(o);
    } else {
      o.kind = JAC_AFFINE_SURF;
      surf.push_back(o);
    }
    row += in.n_dofs;
  }
  if (!mesh.empty() && !b->d_vrow) return fail(PI_ERR_UNSUPPORTED, "vertex adjacency missing for TriangleMeshDoF objects");
  const size_t nj = tri.size() + surf.size() + mesh.size();
  if (nj == 0) return PI_OK;
  if (nj > 65535) return fail(PI_ERR_UNSUPPORTED, "more than 65535 objects in one Jacobian");
  std::vector<JacObj> all(tri);
  all.insert(all.end(), surf.begin(), surf.end());
  all.insert(all.end(), mesh.begin(), mesh.end());
  JacObj* d = nullptr;
  PI_CUDA(pool_alloc((void**)&d, nj * sizeof(JacObj), s));
  PI_CUDA(cudaMemcpyAsync(d, all.data(), nj * sizeof(JacObj), cudaMemcpyHostToDevice, s));
  const KGridDev K = kg->dev;
  const BatchDev B = b->dev();
  const unsigned gx = (unsigned)(((int64_t)((K.Me + 31) / 32) * K.L + JAC_WARPS - 1) / JAC_WARPS);
  if (!tri.empty()) {
    const int n_sm = current_sm_count();
    int64_t n_max = 0, heavy = 0;
    for (const JacObj& o : tri) n_max = std::max(n_max, b->info[o.obj].n_elems);
    for (const JacObj& o : tri) heavy += 4 * b->info[o.obj].n_elems >= n_max;  // as in launch_form_factors
    const int ndt = (K.Me + 31) / 32;
    auto ctas = [&](int R) {
      return (int64_t)(((int64_t)((K.L + R - 1) / R) * ndt + JAC_WARPS - 1) / JAC_WARPS);
    };
    auto busy = [&](int R) { return (K.moments ? (ctas(R) + 3) / 4 : ctas(R)) * heavy; };
    // radii per thread and the split of the elements: two waves of three CTAs
    // per SM, with four radii where sixteen splits give one
    const int R = 16 * busy(4) >= 3 * (int64_t)n_sm ? 4 : 2;
    int S = 1;
    while (S < 16 && S * busy(R) < 6 * (int64_t)n_sm && n_max > 2 * S * 16) S *= 2;
    void* args[4] = {const_cast<KGridDev*>(&K), const_cast<BatchDev*>(&B), &d, &G};
    int rc = launch_split(R == 4 ? reinterpret_cast<const void*>(jac_affine_tri_kernel<4>)
                                 : reinterpret_cast<const void*>(jac_affine_tri_kernel<2>),
                          dim3((unsigned)(ctas(R) * S), (unsigned)tri.size()), JAC_THREADS, 0, S, args, s);
    if (rc) return rc;
    PI_LAUNCHED("jac_affine_tri_kernel");
    if (K.moments) {
      const void* fn = reinterpret_cast<const void*>(jac_moment_kernel);
      if ((rc = ensure_smem_limit(fn, JM_SMEM, "jac_moment_kernel"))) return rc;
      int groups = (K.L + JM_RADII - 1) / JM_RADII;
      int SM = 1;  // one CTA per SM
      while (SM < 8 && (int64_t)SM * ndt * heavy < 2 * (int64_t)n_sm && n_max > SM * JM_TILE * PI_CLUSTER) SM *= 2;
      int spare = R == 4 ? JM_SPARE : 0;  // as the direct kernel
      void* margs[6] = {const_cast<KGridDev*>(&K), const_cast<BatchDev*>(&B), &d, &G, &groups, &spare};
      rc = launch_split(fn, dim3((unsigned)(ndt * groups * SM), (unsigned)tri.size()), JM_THREADS, (size_t)JM_SMEM, SM,
                        margs, s);
      if (rc) return rc;
      PI_LAUNCHED("jac_moment_kernel");
    }
  }
  if (!surf.empty()) {
    jac_affine_surf_kernel<<<dim3(gx, (unsigned)surf.size()), JAC_THREADS, 0, s>>>(K, B, d + tri.size(), G);
    PI_LAUNCHED("jac_affine_surf_kernel");
  }
  if (!mesh.empty()) {
    jac_mesh_kernel<<<dim3(gx, (unsigned)mesh.size()), JAC_THREADS, 0, s>>>(K, B, d + tri.size() + surf.size(),
                                                                             b->d_vrow, b->d_vent, b->d_vmap, G);
    PI_LAUNCHED("jac_mesh_kernel");
  }
  PI_CUDA(cudaFreeAsync(d, s));
  return PI_OK;
}

}  // namespace pi
