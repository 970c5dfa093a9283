// Cluster expansions of the form factors at small k (moments.cu): which radii
// of an object they cover.
#pragma once
#include <cuda_runtime.h>
#include "pi_internal.h"

namespace pi {

// An element of a cluster lies within the cluster's bounding radius rho of its
// centre, so its form factor is e^{i k.c} times a power series in k whose
// n-th term is at most (k rho)^n / n! of the element's amplitude (reached by a
// small element on the rim, seen along its offset from the centre).  With the
// MOMENT_TERMS = 16 terms kept, all that is dropped stays below 5.7e-8 of the
// element's amplitude (triangles, k rho <= 2.375) and 2.4e-8 (surfels, k rho
// <= 2.25) there, less than one FP32 rounding (6.0e-8), and orders of
// magnitude below that for the others of its cluster and the smaller radii.
constexpr int MOMENT_TERMS = 16;
constexpr float MOMENT_X_TRI = 2.375f, MOMENT_X_SURF = 2.25f;

// Radii a grid needs for the expansions to pay (an element's moments cost
// about as much as two radii of the direct sum), and at most as many as the
// running sums of moments.cu fit in shared memory.
constexpr int MOMENT_MIN_L = 8, MOMENT_MAX_L = 288;

#ifdef __CUDACC__
// The radii [0, n) with k rho <= bound (radii ascend on a grid with
// kg.moments); every lane of a warp calls this together.
__device__ __forceinline__ int covered_radii(const KGridDev& kg, float rho, float bound) {
  if (!kg.moments) return 0;
  int n = 0;
  for (int r0 = 0; r0 < kg.L; r0 += 32) {
    const int r = r0 + (int)(threadIdx.x & 31);
    n += __popc(__ballot_sync(0xffffffffu, r < kg.L && kg.kmag[r].x * rho <= bound));
  }
  return n;
}

// Scale of a serving row's column (EvalDev): the root of the weights of node q
// and its antipode qm (-1: none).
__device__ __forceinline__ float serve_scale(const KGridDev& kg, int64_t q, int64_t qm) {
  const float sw = kg.sqrtw[q], swm = qm >= 0 ? kg.sqrtw[qm] : 0.f;
  return sqrtf(fmaf(sw, sw, swm * swm));
}

__device__ __forceinline__ int moment_radii(const KGridDev& kg, int type, float rho) {
  return covered_radii(kg, rho, type == PI_GEOM_TRIANGLE ? MOMENT_X_TRI : MOMENT_X_SURF);
}
// Constants of the recurrences: the coefficient of (i k)^n is f[n] times the
// n-th sum (with the triangles' -2 i^2 = 2 folded in), K[n] as above.
template <int KIND>
struct FmConst {
  float f[MOMENT_TERMS], K[MOMENT_TERMS];
  constexpr FmConst() : f(), K() {
    double g = 1.0;  // 2/(n+2)!, lambda_n, 1/n!
    for (int n = 0; n < MOMENT_TERMS; ++n) {
      f[n] = (float)g;
      K[n] = (float)(KIND == PI_GEOM_DISK ? n * (n + 2.0) / ((2.0 * n + 3.0) * (2.0 * n + 1.0)) : (double)n);
      g *= KIND == PI_GEOM_TRIANGLE ? 1.0 / (n + 3.0)
           : KIND == PI_GEOM_DISK   ? (2.0 * n + 3.0) / ((n + 1.0) * (n + 3.0))
                                    : 1.0 / (n + 1.0);
    }
  }
};

// Adds the moments of two triangles (in the halves) to mu: g h_n(a, b, c).
__device__ __forceinline__ void tri_moments(float2 a, float2 b, float2 c, float2 g, float2 mu[MOMENT_TERMS]) {
  float2 an = g, qn = g, hn = g;
  mu[0] = __fadd2_rn(mu[0], hn);
#pragma unroll
  for (int n = 1; n < MOMENT_TERMS; ++n) {
    an = __fmul2_rn(an, a);
    qn = __ffma2_rn(b, qn, an);
    hn = __ffma2_rn(c, hn, qn);
    mu[n] = __fadd2_rn(mu[n], hn);
  }
}
#endif

// Form factors of the radii below moment_radii; ff_kernel evaluates the others.
int launch_moments(const pi_kgrid_impl* kg, const pi_batch_impl* b, int scale_sqrt_w, float2* J, cudaStream_t s,
                   float* row_amax);
// The same of a class of serving evaluations, with the arguments of ff_serve's kernels.
ServeKernel moment_serve(const pi_kgrid_impl* kg, int cls);
int moment_setup();

}  // namespace pi
