// Form factors at small k from cluster expansions.
//
// Most radii of a Gauss-Legendre grid mapped to [0, inf) are small (45 of 64
// below k = 2), and there the elements of a compact patch of an object differ
// by little phase.  The direct sum (ff_kernel) spends ~23 FP32-pipe operations
// per element, direction and radius whatever k is; here each cluster of
// PI_CLUSTER elements is expanded about its centre c once per direction d,
//
//   sum_e A_e(k d) = e^{i k d.c} sum_n (i k)^n mu_n(d),
//
// (73 FP32-pipe operations per triangle and direction for all radii
// together), and a radius then costs one phasor and two Horner chains per
// cluster: about 35 operations per 64 elements.  No reference counterpart.
//
// Moments of an element at projections relative to the cluster centre, in
// units of a power of two s >= rho (so that no power overflows):
//
//  * triangle with vertex projections a, b, c: A = -2 gamma e[ka, kb, kc] and
//    e[..] = sum_n i^{n+2} k^n h_n(a, b, c) / (n+2)!, h_n the complete
//    homogeneous symmetric polynomials, by the nested recurrences
//      a_n = a a_{n-1},  q_n = b q_{n-1} + a_n,  h_n = c h_{n-1} + q_n
//    (every step adds terms of one sign where a, b, c share theirs; the
//    recurrence in the elementary symmetric polynomials loses a few bits at
//    nearly equal vertices).  gamma is folded into the starting values;
//  * disk: amp e^{i k s} 2 J1(kp)/(kp) = amp sum_n i^n k^n u_n with
//      (n+1)(n+3) u_{n+1} = (2n+3) s u_n + (p^2 - s^2) u_{n-1}
//    (from the differential equation of 2 J1(x)/x);
//  * Gaussian: amp e^{i k s - q k^2}, (n+1) u_{n+1} = s u_n + 2 q u_{n-1}.
//    Both with u_n = lambda_n w_n, w_{n+1} = s w_n + K_n q w_{n-1}.
//
// One CTA owns one object and 32 evaluated directions (one per lane); it
// alternates between two phases over tiles of 8 clusters:
//   1. each warp stages one cluster's elements, forms its moments, two
//      elements per packed FP32 instruction, and leaves the 16 coefficients
//      per direction in shared memory;
//   2. each warp sums the tile's clusters over its own radii, 8 at a time in
//      registers (two per packed instruction), and adds them to compensated
//      running sums in shared memory.
//
// Bound by the FP32 pipe (58% busy, its packed instructions holding it two
// cycles) and the waits between the two phases.  256 solids of 5,120 and 12
// triangles, N_k = 76,928: 1.9 ms for 47 to 51 of the 64 radii (42 of a box), where
// the direct sum of all radii took 38.8; one solid of 200,000 triangles on
// 743,680 nodes: 4.4 ms for 115 of its 128.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "pi_internal.h"
#include "dfmath.cuh"
#include "moments.h"

namespace pi {

namespace {

constexpr int FM_WARPS = 8, FM_THREADS = 32 * FM_WARPS;
constexpr int FM_R = 8;                             // radii per warp and batch
constexpr int FM_COPIES = 8;                        // of the phasor table: two CTAs per SM at 128 radii
constexpr int FM_PAIRS = PI_CLUSTER / 2;            // staged element pairs per cluster
constexpr int FM_PAIR_F4 = 6;                       // float4 per pair: 12 values of two elements
static_assert(MOMENT_TERMS == 16, "coefficients are stored as four float4");

// Shared memory, in float4: staged elements, coefficients, phasor table,
// radius constants, then the running sums.
constexpr int FM_F4_ELEM = FM_WARPS * FM_PAIRS * FM_PAIR_F4, FM_F4_MOM = FM_WARPS * 4 * 32, FM_F4_TAB = PHASOR_ENTRIES * FM_COPIES / 2,
              FM_F4_CTR = FM_WARPS * 16;            // cluster phases (hi, lo) per lane

__host__ __device__ constexpr int fm_batches(int L) { return (L + FM_R - 1) / FM_R; }
__host__ __device__ constexpr int fm_smem_f4(int L) {
  return FM_F4_ELEM + FM_F4_MOM + FM_F4_TAB + FM_F4_CTR + fm_batches(L) * FM_R /* kx, kk */ +
         (fm_batches(L) * FM_R + 1) * 32 /* running sums: (re, im, compensations), and of the zeroth moments */;
}

__device__ __forceinline__ float2 f2lo(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 f2hi(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

struct FmDir {
  float3 dh, dl;
  float inv_norm;
  float3 v;    // A^T d (surfels: k' = |k| v)
  float qd;    // |v|^2
};

// Stages cluster cl's elements (values of elements 2i, 2i + 1 in the halves of
// float2s), relative to its centre and scaled by 1/s; missing ones are zeros.
template <int KIND>
__device__ __forceinline__ void fm_stage(const BatchDev& b, const ObjDev& od, int first, int cnt, float4 ctr,
                                         float inv_s, float* es) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < PI_CLUSTER / 32; ++h) {
    const int i = lane + 32 * h;
    float v[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) v[c] = 0.f;
    if (i < cnt) {
      const int64_t e = od.elem_off + first + i;
      if (KIND == PI_GEOM_TRIANGLE) {
        const float4 q0 = b.tri_pool[3 * e], q1 = b.tri_pool[3 * e + 1], q2 = b.tri_pool[3 * e + 2], lo = b.tri_lo[e];
        const float m[3] = {(q0.x - ctr.x) + lo.x, (q0.y - ctr.y) + lo.y, (q0.z - ctr.z) + lo.z};
        const float e1[3] = {q1.x, q1.y, q1.z}, e2[3] = {q2.x, q2.y, q2.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float a = m[c] - (e1[c] + e2[c]) * (1.0f / 3.0f);
          v[c] = a * inv_s;
          v[3 + c] = (a + e1[c]) * inv_s;
          v[6 + c] = (a + e2[c]) * inv_s;
        }
        v[9] = q0.w; v[10] = q1.w; v[11] = q2.w;
      } else {
        const float4 q0 = b.surf_pool[2 * e], q1 = b.surf_pool[2 * e + 1], nr = b.surf_nref[e], lo = b.surf_lo[e];
        v[0] = ((q0.x - ctr.x) + lo.x) * inv_s;
        v[1] = ((q0.y - ctr.y) + lo.y) * inv_s;
        v[2] = ((q0.z - ctr.z) + lo.z) * inv_s;
        v[3] = q1.x * q1.w; v[4] = q1.y * q1.w; v[5] = q1.z * q1.w;  // area|w times A n
        v[6] = nr.x; v[7] = nr.y; v[8] = nr.z;
        const float p = q0.w * inv_s;
        v[9] = nr.w; v[10] = p * p;
      }
    }
    float* d = es + (i >> 1) * (4 * FM_PAIR_F4) + (i & 1);
#pragma unroll
    for (int c = 0; c < 12; ++c) d[2 * c] = v[c];
  }
  __syncwarp();
}

// Sums the moments of the staged elements; mu in the even entries' and odd
// entries' halves.  Returns the zeroth, compensated (hi, lo).
template <int KIND>
__device__ __forceinline__ float2 fm_moments(const float4* es, int pairs, const FmDir& D, float2 mu[MOMENT_TERMS]) {
  constexpr FmConst<KIND> C{};
  float2 z = make_float2(0.f, 0.f), cz0 = z;
#pragma unroll
  for (int n = 0; n < MOMENT_TERMS; ++n) mu[n] = make_float2(0.f, 0.f);
  const float2 dx = dup2(D.dh.x), dy = dup2(D.dh.y), dz = dup2(D.dh.z);
#pragma unroll 1
  for (int i = 0; i < pairs; ++i) {
    const float4 q0 = es[FM_PAIR_F4 * i], q1 = es[FM_PAIR_F4 * i + 1], q2 = es[FM_PAIR_F4 * i + 2],
                 q3 = es[FM_PAIR_F4 * i + 3], q4 = es[FM_PAIR_F4 * i + 4], q5 = es[FM_PAIR_F4 * i + 5];
    const float2 s0 = fma2(dz, f2lo(q1), fma2(dy, f2hi(q0), mul2(dx, f2lo(q0))));
    if (KIND == PI_GEOM_TRIANGLE) {
      const float2 a = s0;
      const float2 bb = fma2(dz, f2hi(q2), fma2(dy, f2lo(q2), mul2(dx, f2hi(q1))));
      const float2 c = fma2(dz, f2lo(q4), fma2(dy, f2hi(q3), mul2(dx, f2lo(q3))));
      const float2 g = fma2(dz, f2hi(q5), fma2(dy, f2lo(q5), mul2(dx, f2hi(q4))));  // gamma |d| (area vector . d)
      tri_moments(a, bb, c, g, mu);
      kahan2(z, cz0, g);
    } else {
      const float2 amp = fma2(dz, f2hi(q2), fma2(dy, f2lo(q2), mul2(dx, f2hi(q1))));
      // |k'_perp|^2 / |k|^2 = qd (1 - |n|^2) + |n|^2 |v x n/|n||^2, as in ff_kernel
      const float2 rx = f2lo(q3), ry = f2hi(q3), rz = f2lo(q4), nw = f2hi(q4), p2 = f2lo(q5);
      const float2 vx = dup2(D.v.x), vy = dup2(D.v.y), vz = dup2(D.v.z);
      const float2 cx = fma2(vy, rz, neg2(mul2(vz, ry))), cy = fma2(vz, rx, neg2(mul2(vx, rz))),
                   cz = fma2(vx, ry, neg2(mul2(vy, rx)));
      const float2 cc = fma2(cx, cx, fma2(cy, cy, mul2(cz, cz)));
      float2 perp = fma2(dup2(D.qd), nw, mul2(add2(dup2(1.0f), neg2(nw)), cc));
      const bool disk = KIND == PI_GEOM_DISK;
      // a disk's is at least 0 (normals longer than 1 make it negative near them), a Gaussian's is not clamped
      if (disk) perp = make_float2(fmaxf(perp.x, 0.f), fmaxf(perp.y, 0.f));
      // disk: q = p^2 - s^2; Gaussian: q = sigma^2 |k'_perp|^2 / |k|^2 (= 2 q' of e^{-q' k^2})
      const float2 q = disk ? fma2(p2, perp, neg2(mul2(s0, s0))) : mul2(p2, perp);
      float2 w0 = amp, w1 = mul2(s0, amp);
      kahan2(z, cz0, w0);
      mu[1] = add2(mu[1], w1);
#pragma unroll
      for (int n = 1; n < MOMENT_TERMS - 1; ++n) {
        const float2 w2 = fma2(s0, w1, mul2(mul2(dup2(C.K[n]), q), w0));
        mu[n + 1] = add2(mu[n + 1], w2);
        w0 = w1;
        w1 = w2;
      }
    }
  }
  mu[0] = z;
  const df s = two_sum(z.x, z.y);
  return make_float2(s.hi, s.lo - (cz0.x + cz0.y));
}

// e^{ik.c} sum_n (i k)^n .. of the cluster: coefficients as Re = sum_j a_j u^j,
// Im = k sum_j b_j u^j (u = k^2, k in units of 1/s).
template <int KIND>
__device__ __forceinline__ void fm_store(const float2 mu[MOMENT_TERMS], float norm, float4* mom) {
  constexpr FmConst<KIND> C{};
  float c[MOMENT_TERMS];
#pragma unroll
  for (int n = 0; n < MOMENT_TERMS; ++n)  // i^n: real for even n, imaginary for odd n
    c[(n & 1) * (MOMENT_TERMS / 2) + n / 2] = (mu[n].x + mu[n].y) * (((n & 2) ? -C.f[n] : C.f[n]) * norm);
#pragma unroll
  for (int t = 0; t < 4; ++t) mom[32 * t] = make_float4(c[4 * t], c[4 * t + 1], c[4 * t + 2], c[4 * t + 3]);
}

// c[1] u + c[2] u^2 + ... + c[7] u^7
__device__ __forceinline__ float2 horner_rest(const float (&c)[8], float2 u) {
  float2 r = dup2(c[7]);
#pragma unroll
  for (int i = 6; i >= 1; --i) r = fma2(r, u, dup2(c[i]));
  return mul2(r, u);
}

__device__ __forceinline__ float2 horner8(const float (&c)[8], float2 u) {
  float2 r = dup2(c[7]);
#pragma unroll
  for (int i = 6; i >= 0; --i) r = fma2(r, u, dup2(c[i]));
  return r;
}

// SERVE and the S CTAs of a thread-block cluster as in ff_kernel: they take
// every S-th tile, and their running sums meet at the end.  The grid is
// (direction groups x S) x (objects or evaluations), re-mapped so that the
// objects (largest first) vary fastest.
template <bool SERVE>
__device__ __forceinline__ void moment_body(const KGridDev& kg, const BatchDev& b, float2* __restrict__ J,
                                            int scale_sqrt_w, const EvalDev* __restrict__ evals,
                                            unsigned* __restrict__ row_amax) {
  extern __shared__ float4 sm[];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const unsigned lin = (blockIdx.y * gridDim.x + blockIdx.x) / (unsigned)S;
  const int slot = (int)(lin % gridDim.y), dt = (int)(lin / gridDim.y);
  const int oi = SERVE ? evals[slot].obj : b.order[slot];
  const ObjDev od = b.objs[oi];
  const int nr = moment_radii(kg, od.type, __uint_as_float(b.cl_rho[oi]));  // radii [0, nr)
  if (nr == 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = fm_batches(nr);
  float4* elem = sm;
  float4* mom = elem + FM_F4_ELEM;
  float2* ctab_sm = reinterpret_cast<float2*>(mom + FM_F4_MOM);
  const float2* ctab = ctab_sm + (threadIdx.x % FM_COPIES);
  float2* csc = ctab_sm + PHASOR_ENTRIES * FM_COPIES;                      // [cluster][lane]: d . c (hi, lo)
  float4* kx = reinterpret_cast<float4*>(csc + 32 * FM_WARPS);  // radii (2p, 2p + 1) in 1/64 turns: (hi, hi', lo, lo')
  float2* kk = reinterpret_cast<float2*>(kx + fm_batches(kg.L) * FM_R / 2);  // (k, k')
  float4* run = kx + fm_batches(kg.L) * FM_R;             // [radius][lane]: sums and compensations
  float4* run0 = run + nb * FM_R * 32;                    // the zeroth moments', in the first and third
  __shared__ float cscale_sm[FM_WARPS];

  const int ei = dt * 32 + lane;
  const bool active = ei < kg.Me;
  int j = 0, jm = -1;
  FmDir D;
  D.dh = D.dl = make_float3(0.f, 0.f, 0.f);
  D.inv_norm = 0.f;
  float dnorm = 0.f;
  if (active) {
    const int2 pr = kg.dpair[ei];
    j = pr.x;
    jm = pr.y;
    const float4 h = kg.dir_hi[j], l = kg.dir_lo[j];
    D.dh = make_float3(h.x, h.y, h.z);
    D.dl = make_float3(l.x, l.y, l.z);
    D.inv_norm = h.w;
    dnorm = l.w;
    if (SERVE && evals[slot].rotate) {  // the unrotated object's form factor at R^T k, as in ff_kernel
      const double* Rm = evals[slot].R;
      const double d0 = (double)h.x + (double)l.x, d1 = (double)h.y + (double)l.y, d2 = (double)h.z + (double)l.z;
      double e[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) e[a] = Rm[a] * d0 + Rm[3 + a] * d1 + Rm[6 + a] * d2;
      D.dh = make_float3((float)e[0], (float)e[1], (float)e[2]);
      D.dl = make_float3((float)(e[0] - (double)D.dh.x), (float)(e[1] - (double)D.dh.y), (float)(e[2] - (double)D.dh.z));
    }
  }
  const float* Am = od.A;
  D.v = make_float3(Am[0] * D.dh.x + Am[3] * D.dh.y + Am[6] * D.dh.z, Am[1] * D.dh.x + Am[4] * D.dh.y + Am[7] * D.dh.z,
                    Am[2] * D.dh.x + Am[5] * D.dh.y + Am[8] * D.dh.z);
  D.qd = fmaf(D.v.x, D.v.x, fmaf(D.v.y, D.v.y, D.v.z * D.v.z));

  stage_phasors<FM_COPIES>(kg.cis_tabm, ctab_sm);
  for (int t = threadIdx.x; t < nb * FM_R / 2; t += FM_THREADS) {
    float2 k[2], kt[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool ok = 2 * t + h < nr;
      k[h] = ok ? kg.kmag[2 * t + h] : make_float2(0.f, 0.f);
      kt[h] = ok ? kg.kt64[2 * t + h] : make_float2(0.f, 0.f);
    }
    kx[t] = make_float4(kt[0].x, kt[1].x, kt[0].y, kt[1].y);
    kk[t] = make_float2(k[0].x, k[1].x);
  }
  for (int t = threadIdx.x; t < (nb * FM_R + 1) * 32; t += FM_THREADS) run[t] = make_float4(0.f, 0.f, 0.f, 0.f);

  const int ncl = (od.n_elems + PI_CLUSTER - 1) / PI_CLUSTER;
  for (int t0 = rank * FM_WARPS; t0 < ncl; t0 += S * FM_WARPS) {
    __syncthreads();  // the last tile's coefficients have been read (and the tables written, before the first)
    const int cl = t0 + warp;
    if (cl < ncl) {
      const float4 ctr = b.clusters[od.cl_off + cl];
      // s: the power of two above rho
      const int ex = ctr.w > 0.f ? min(120, max(-100, ilogbf(ctr.w) + 1)) : 0;
      const float s = __int_as_float((127 + ex) << 23), inv_s = __int_as_float((127 - ex) << 23);
      const int first = cl * PI_CLUSTER, cnt = min(PI_CLUSTER, od.n_elems - first), pairs = (cnt + 1) / 2;
      float4* es = elem + warp * FM_PAIRS * FM_PAIR_F4;
      float2 mu[MOMENT_TERMS], m0;
      float4* mo = mom + warp * 4 * 32 + lane;
      if (od.type == PI_GEOM_TRIANGLE) {
        fm_stage<PI_GEOM_TRIANGLE>(b, od, first, cnt, ctr, inv_s, reinterpret_cast<float*>(es));
        m0 = fm_moments<PI_GEOM_TRIANGLE>(es, pairs, D, mu);
        fm_store<PI_GEOM_TRIANGLE>(mu, D.inv_norm, mo);
      } else if (od.type == PI_GEOM_DISK) {
        fm_stage<PI_GEOM_DISK>(b, od, first, cnt, ctr, inv_s, reinterpret_cast<float*>(es));
        m0 = fm_moments<PI_GEOM_DISK>(es, pairs, D, mu);
        fm_store<PI_GEOM_DISK>(mu, D.inv_norm, mo);
      } else {
        fm_stage<PI_GEOM_GAUSSIAN>(b, od, first, cnt, ctr, inv_s, reinterpret_cast<float*>(es));
        m0 = fm_moments<PI_GEOM_GAUSSIAN>(es, pairs, D, mu);
        fm_store<PI_GEOM_GAUSSIAN>(mu, D.inv_norm, mo);
      }
      const df sc = cdot(D.dh, D.dl, make_float3(ctr.x, ctr.y, ctr.z));
      csc[warp * 32 + lane] = make_float2(sc.hi, sc.lo);
      __syncwarp();  // the cluster's elements have been read: their place takes its zeroth moment
      reinterpret_cast<float2*>(es)[lane] = m0;
      if (lane == 0) cscale_sm[warp] = s;
    }
    __syncthreads();
    const int nc = min(FM_WARPS, ncl - t0);
    if (warp == FM_WARPS - 1) {
      const float4 z = run0[lane];
      kbsum s{z.x, z.z};
      for (int c = 0; c < nc; ++c) {
        const float2 v = reinterpret_cast<const float2*>(elem + c * FM_PAIRS * FM_PAIR_F4)[lane];
        s.add(v.x);
        s.lo += v.y;
      }
      run0[lane] = make_float4(s.hi, 0.f, s.lo, 0.f);
    }
    // Every cluster's value is its zeroth moment, the same at all radii and
    // summed above, and the rest, which vanishes with k: e^{ik.c} enters less 1.
    // A closed surface's form factor at small k is what the zeroth moments leave
    // of each other, ~k of their size, and rounding each cluster's value (all
    // its elements in phase) would leave ten times the error of rounding elements.
    for (int bt = warp; bt < nb; bt += FM_WARPS) {
      // compensated running sums: a cluster's value is as large as all its
      // elements' terms together, so plain partial sums would round coarsely
      float2 re[FM_R / 2], im[FM_R / 2], cre[FM_R / 2], cim[FM_R / 2];
      float4* rp = run + bt * FM_R * 32 + lane;
#pragma unroll
      for (int p = 0; p < FM_R / 2; ++p) {
        const float4 r0 = rp[64 * p], r1 = rp[64 * p + 32];
        re[p] = make_float2(r0.x, r1.x); im[p] = make_float2(r0.y, r1.y);
        cre[p] = make_float2(r0.z, r1.z); cim[p] = make_float2(r0.w, r1.w);
      }
#pragma unroll 1
      for (int c = 0; c < nc; ++c) {
        float a[8], bb[8];
        const float4* mo = mom + c * 4 * 32 + lane;
        const float4 m0 = mo[0], m1 = mo[32], m2 = mo[64], m3 = mo[96];
        a[0] = m0.x; a[1] = m0.y; a[2] = m0.z; a[3] = m0.w; a[4] = m1.x; a[5] = m1.y; a[6] = m1.z; a[7] = m1.w;
        bb[0] = m2.x; bb[1] = m2.y; bb[2] = m2.z; bb[3] = m2.w; bb[4] = m3.x; bb[5] = m3.y; bb[6] = m3.z; bb[7] = m3.w;
        const float2 sc = csc[c * 32 + lane];
        const float2 s2 = dup2(cscale_sm[c]), sh = dup2(sc.x), sl = dup2(sc.y);
#pragma unroll
        for (int p = 0; p < FM_R / 2; ++p) {
          const float4 kt = kx[bt * (FM_R / 2) + p];
          const cf2 M = cis_tab_m1_df2<FM_COPIES>(ctab, f2lo(kt), f2hi(kt), sh, sl);
          const float2 k = mul2(kk[bt * (FM_R / 2) + p], s2), u = mul2(k, k);
          const float2 xr = horner_rest(a, u), x = add2(xr, dup2(a[0])), y = mul2(k, horner8(bb, u));
          kahan2(re[p], cre[p], fma2(M.re, x, fma2(neg2(M.im), y, xr)));
          kahan2(im[p], cim[p], fma2(M.re, y, fma2(M.im, x, y)));
        }
      }
#pragma unroll
      for (int p = 0; p < FM_R / 2; ++p) {
        rp[64 * p] = make_float4(re[p].x, im[p].x, cre[p].x, cim[p].x);
        rp[64 * p + 32] = make_float4(re[p].y, im[p].y, cre[p].y, cim[p].y);
      }
    }
  }
  if (S > 1) cluster.sync();
  else __syncthreads();
  float m = 0.f;
  const double so = ((double)D.dh.x + (double)D.dl.x) * od.origin[0] + ((double)D.dh.y + (double)D.dl.y) * od.origin[1] +
                    ((double)D.dh.z + (double)D.dl.z) * od.origin[2];
  kbsum zero{0.f, 0.f};  // the zeroth moments' sum, its product with 1/|d| split as well
  for (int q = 0; q < S; ++q) {
    const float4 v4 = (S > 1 ? cluster.map_shared_rank(run0, q) : run0)[lane];
    zero.add(v4.x); zero.lo += v4.z;
  }
  {
    const float p = zero.hi * D.inv_norm;
    zero = kbsum{p, fmaf(zero.hi, D.inv_norm, -p) + zero.lo * D.inv_norm};
  }
  for (int r = warp * S + rank; r < nr && active; r += FM_WARPS * S) {
    kbsum re{0.f, 0.f}, im{0.f, 0.f};  // over the cluster, in the order of the ranks
    for (int q = 0; q < S; ++q) {
      const float4 v4 = (S > 1 ? cluster.map_shared_rank(run, q) : run)[r * 32 + lane];
      re.add(v4.x); im.add(v4.y);
      re.lo -= v4.z; im.lo -= v4.w;
    }
    re.add(zero.hi); re.lo += zero.lo;
    cf v{re.hi + re.lo, im.hi + im.lo};
    const float2 km = kg.kmag[r];
    if (!SERVE) {
      const float2 kt = kg.kt64[r];
      v = cmul(cis_f64(((double)kt.x + (double)kt.y) * (6.283185307179586476925 / 64.0) * so), v);
    }
    if (km.x * dnorm < 1e-10f) v = cf{0.f, 0.f};  // A(0) = 0 (affine_dof.cpp:64-65)
    const int64_t q = (int64_t)r * kg.M + j, qm = (int64_t)r * kg.M + jm;
    if (SERVE) {
      const float sw = serve_scale(kg, q, jm >= 0 ? qm : -1);
      const float2 o = make_float2(v.re * sw, v.im * sw);
      m = fmaxf(m, fmaxf(fabsf(o.x), fabsf(o.y)));
      evals[slot].dst[(int64_t)kg.ecol[ei] * kg.L + r] = o;
    } else {
      const float sw = scale_sqrt_w ? kg.sqrtw[q] : 1.0f, swm = scale_sqrt_w && jm >= 0 ? kg.sqrtw[qm] : 1.0f;
      const float2 o = make_float2(v.re * sw, v.im * sw), om = make_float2(-v.re * swm, v.im * swm);
      m = fmaxf(m, fmaxf(fabsf(o.x), fabsf(o.y)));
      J[(int64_t)oi * kg.Q + q] = o;
      if (jm >= 0) {  // the antipode: -conj
        m = fmaxf(m, fmaxf(fabsf(om.x), fabsf(om.y)));
        J[(int64_t)oi * kg.Q + qm] = om;
      }
    }
  }
  if (S > 1) cluster.sync();  // no CTA leaves while its sums are read
  if (!active) return;
  unsigned* amax = SERVE ? reinterpret_cast<unsigned*>(evals[slot].amax) : row_amax ? row_amax + oi : nullptr;
  if (amax) {  // FP32 bits order like the non-negative floats
    const unsigned mask = __activemask();
    const unsigned mb = __reduce_max_sync(mask, __float_as_uint(m));
    if (lane == __ffs(mask) - 1) atomicMax(amax, mb);
  }
}

__global__ void __launch_bounds__(FM_THREADS, 2)
moment_kernel(KGridDev kg, BatchDev b, float2* __restrict__ J, int scale_sqrt_w, const EvalDev* __restrict__ evals,
              unsigned* __restrict__ row_amax) {
  moment_body<false>(kg, b, J, scale_sqrt_w, evals, row_amax);
}

// CTAs per serving evaluation of each class (SERVE_CLASSES).
constexpr int FM_SERVE_SPLIT[SERVE_CLASSES] = {8, 4, 2, 1};

__global__ void __launch_bounds__(FM_THREADS, 2)
moment_serve_kernel(KGridDev kg, BatchDev b, const EvalDev* __restrict__ evals, int n_evals) {
  if (n_evals == 0) return;  // a class that the batch has no evaluation of
  moment_body<true>(kg, b, nullptr, 1, evals, nullptr);
}

}  // namespace

static int moment_smem_bytes(int L) { return fm_smem_f4(L) * (int)sizeof(float4); }

ServeKernel moment_serve(const pi_kgrid_impl* kg, int cls) {
  const int S = FM_SERVE_SPLIT[cls];
  return {reinterpret_cast<const void*>(moment_serve_kernel), (unsigned)((kg->dev.Me + 31) / 32 * S), FM_THREADS, S,
          (size_t)moment_smem_bytes(kg->dev.L)};
}

int moment_setup() {
  int rc = ensure_smem_limit(reinterpret_cast<const void*>(moment_kernel), moment_smem_bytes(MOMENT_MAX_L),
                             "moment_kernel");
  if (rc == PI_OK)
    rc = ensure_smem_limit(reinterpret_cast<const void*>(moment_serve_kernel), moment_smem_bytes(MOMENT_MAX_L),
                           "moment_kernel");
  return rc;
}

int launch_moments(const pi_kgrid_impl* kg, const pi_batch_impl* b, int scale_sqrt_w, float2* J, cudaStream_t s,
                   float* row_amax) {
  if (!kg->dev.moments || b->n_obj == 0) return PI_OK;
  int rc = moment_setup();
  if (rc) return rc;
  // as in launch_form_factors: CTAs of the objects that carry the launch, and
  // a split of their tiles that gives two waves of two CTAs per SM
  const int64_t n_max = b->info[b->order[0]].n_elems, ndt = (kg->dev.Me + 31) / 32;
  int64_t heavy = 0;
  for (int i = 0; i < b->n_obj; ++i) heavy += 4 * b->info[i].n_elems >= n_max;
  int S = 1;
  while (S < 8 && S * ndt * heavy < 4 * (int64_t)current_sm_count() && n_max > S * FM_WARPS * PI_CLUSTER) S *= 2;
  const KGridDev K = kg->dev;
  const BatchDev B = b->dev();
  const EvalDev* no_evals = nullptr;
  void* args[6] = {const_cast<KGridDev*>(&K), const_cast<BatchDev*>(&B), &J, &scale_sqrt_w, &no_evals, &row_amax};
  rc = launch_split(reinterpret_cast<const void*>(moment_kernel), dim3((unsigned)(ndt * S), (unsigned)b->n_obj),
                    FM_THREADS, (size_t)moment_smem_bytes(K.L), S, args, s);
  if (rc) return rc;
  PI_LAUNCHED("moment_kernel");
  return PI_OK;
}

}  // namespace pi
