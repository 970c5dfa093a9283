// Per-object form factors A_n(k_q) on the device.
//
// Replaces the reference kernels K1-K3 (cpp/src/dof/cuda/affine_dof_cuda.cu:43-250,
// 580-689) and K7 (cpp/src/dof/cuda/triangle_mesh_dof_cuda.cu:34-143), whose
// grid was one CTA per k-node looping over every element in FP64 with a shared
// memory tree reduction.  Here:
//
//  * prepare_*: each object's elements are transformed once per DoF change by
//    its AffineDoF / TriangleMeshDoF into an FP32 object-local frame (origin =
//    centroid of the transformed anchors), centroids (centres) as FP32 hi + lo;
//    the origin phase e^{ik.o} is formed and reduced in FP64 per output.
//  * ff_kernel: the radii that the cluster expansions (moments.cu) leave: 13 to
//    17 of 64 for bodies of 5,120 triangles, whose leaves' expansions cover eight of
//    them (all radii on grids the expansions do not take).
//    One CTA = one object x 4 warps; a warp owns 32 directions
//    (one per lane) x R neighbouring radial nodes of the factored k-grid, so
//    each element's direction dot products and series coefficients are
//    formed once and reused for R radii; where all R radii take the short
//    series, two radii share each packed FP32 instruction; leaves of four
//    triangles have expansions of their own.  The CTAs of a thread-block
//    cluster split the elements where few objects would leave SMs idle.
//    Bound by instruction issue (63-70% active; 256 solids of 5,120 and 12
//    triangles at N_k = 76,928: 38.8 ms for all radii, 12.4 now).  On a centrally
//    symmetric direction set a lane evaluates one direction of an antipodal
//    pair and writes both (A(-k) = -conj A(k) for a real solid: half the
//    evaluations), and a warp's 32 directions form a compact cluster.  Radial
//    blocks start largest-k first, for all objects.  Elements are staged
//    through shared memory and read as broadcasts; each thread accumulates
//    its own outputs (no reduction across threads), 32-element partials in
//    registers and compensated running sums in shared memory; each output
//    element is written once, in the contraction's operand layout.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <algorithm>
#include "pi_internal.h"
#include "dfmath.cuh"
#include "bessel.cuh"
#include "moments.h"

namespace pi {

namespace {

struct TriSrc { double a[3], e1[3], e2[3], S[3]; int32_t vid0, vid1, vid2, pad; };
struct SurfSrc { double c[3], n[3], p0, p1; };

struct PrepObj {
  int32_t geom_type, dof_type;
  int64_t n_elems, n_dofs;
  const unsigned char* src;
  const double* dofs;
  int64_t pool_off, perm_off, cl_off;
};

__device__ __forceinline__ void affine_apply(const double* d, const double* x, double* y, bool translate) {
  for (int r = 0; r < 3; ++r) {
    double v = d[3 + 3 * r] * x[0] + d[3 + 3 * r + 1] * x[1] + d[3 + 3 * r + 2] * x[2];
    y[r] = translate ? v + d[r] : v;
  }
}

// Anchor point of element e before the DoF transform (first vertex / centre;
// the moving vertex of a TriangleMeshDoF).
__device__ __forceinline__ void anchor(const PrepObj& o, int64_t e, double* y) {
  if (o.geom_type == PI_GEOM_TRIANGLE) {
    const TriSrc& t = reinterpret_cast<const TriSrc*>(o.src)[e];
    if (o.dof_type == PI_DOF_TRIANGLE_MESH) {
      int64_t nv = o.n_dofs / 3;
      if (t.vid0 < 0 || t.vid0 >= nv) { y[0] = y[1] = y[2] = 0.0; return; }
      y[0] = o.dofs[3 * t.vid0]; y[1] = o.dofs[3 * t.vid0 + 1]; y[2] = o.dofs[3 * t.vid0 + 2];
    } else {
      y[0] = t.a[0]; y[1] = t.a[1]; y[2] = t.a[2];
    }
  } else {
    const SurfSrc& s = reinterpret_cast<const SurfSrc*>(o.src)[e];
    y[0] = s.c[0]; y[1] = s.c[1]; y[2] = s.c[2];
  }
}

// Fixed-order mean of the anchors (deterministic), plus the object's A for the
// surfel k' = A^T k rule.  FP64 adds run at ~2 per SM and clock, so the map is
// applied to the mean (it is affine) and the S CTAs of a thread-block cluster
// share an object's elements, their sums meeting in the first one (one CTA per
// object and a transform per element: 230 us for 50,000 surfels).
constexpr int ORIGIN_THREADS = 256, ORIGIN_SPLIT = 8;
__global__ void __launch_bounds__(ORIGIN_THREADS)
prepare_origin_kernel(const PrepObj* objs, ObjDev* out, unsigned* cl_rho, int only) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int oi = only >= 0 ? only : blockIdx.x / S;
  const PrepObj o = objs[oi];
  __shared__ double red[3][ORIGIN_THREADS / 32];
  __shared__ double total[3];
  double s[3] = {0.0, 0.0, 0.0};
  for (int64_t e = rank * ORIGIN_THREADS + threadIdx.x; e < o.n_elems; e += S * ORIGIN_THREADS) {
    double y[3];
    anchor(o, e, y);
    s[0] += y[0]; s[1] += y[1]; s[2] += y[2];
  }
  for (int w = 16; w > 0; w >>= 1)
    for (int c = 0; c < 3; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], w);
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 3; ++c) red[c][threadIdx.x >> 5] = s[c];
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < ORIGIN_THREADS / 32; ++w) t += red[threadIdx.x][w];
    total[threadIdx.x] = t;
  }
  if (S > 1) cluster.sync();
  else __syncthreads();
  if (rank == 0 && threadIdx.x == 0) {
    double m[3] = {total[0], total[1], total[2]};
    for (int q = 1; q < S; ++q) {
      const double* t = cluster.map_shared_rank(total, q);
      for (int c = 0; c < 3; ++c) m[c] += t[c];
    }
    ObjDev d;
    const double inv = o.n_elems > 0 ? 1.0 / (double)o.n_elems : 0.0;
    for (int c = 0; c < 3; ++c) m[c] *= inv;
    if (o.dof_type == PI_DOF_AFFINE) {
      const double* A = o.dofs + 3;
      for (int i = 0; i < 9; ++i) d.A[i] = (float)A[i];
      if (o.n_elems > 0) affine_apply(o.dofs, m, d.origin, true);
      else d.origin[0] = d.origin[1] = d.origin[2] = 0.0;
    } else {
      for (int i = 0; i < 9; ++i) d.A[i] = (i % 4 == 0) ? 1.f : 0.f;
      for (int c = 0; c < 3; ++c) d.origin[c] = m[c];
    }
    d.type = o.geom_type;
    d.n_elems = (int32_t)o.n_elems;
    d.elem_off = o.pool_off;
    d.perm_off = o.perm_off;
    d.cl_off = o.cl_off;
    out[oi] = d;
    cl_rho[oi] = 0u;  // prepare_elems_kernel takes the maximum
  }
  if (S > 1) cluster.sync();  // no CTA leaves while its sum is read
}

// Orders one segment of an object's elements (OrderSeg) per CTA by recursive
// bisection of their anchors at the widest coordinate.  Parts of more than one
// cluster: all parts of a level at once, each cut at its exact median, found
// digit by digit (four 6-bit digits of the coordinate scaled to the part's
// bounding box, ties by position) from histograms in shared memory, and moved
// by a stable partition; parts are whole clusters, so a warp's 32 entries
// share a part, and the parts' sizes depend on the count alone, so a warp
// finds its part by walking down from the root.  Within a cluster a warp sorts
// 64, 32, 16 and 8 entries by ranks counted through shuffles.  (Bitonic sorts
// of the whole segment at every level took 185 us for 1,280 elements and 905
// for 5,120; the host ~0.1 us per element.)
constexpr int ORDER_SLOTS = ORDER_SEGMENT / PI_CLUSTER, ORDER_BLOCKS = ORDER_SEGMENT / 32;
constexpr int ORDER_THREADS = 1024;  // segments have 2,048 to ORDER_SEGMENT elements: at most eight entries per thread
constexpr int ORDER_BITS = 6, ORDER_BINS = 1 << ORDER_BITS, ORDER_ROUNDS = 4;

struct OrderShared {
  unsigned mn[3][ORDER_SLOTS], mx[3][ORDER_SLOTS];  // bounding boxes as order-preserving integers
  int axis[ORDER_SLOTS];
  float base[ORDER_SLOTS], scale[ORDER_SLOTS];
  unsigned prefix[ORDER_SLOTS], target[ORDER_SLOTS];
  unsigned less[ORDER_BLOCKS], equal[ORDER_BLOCKS];  // per 32 entries, then their prefix sums
  unsigned hist[ORDER_SLOTS][ORDER_BINS];
};

__host__ __device__ constexpr size_t order_smem(int n2) {
  return sizeof(OrderShared) + (size_t)n2 * (3 * sizeof(float) + 2 * sizeof(unsigned short));
}

// The part of a level that holds entry i: [lo, lo + c).
__device__ __forceinline__ void order_part(int n, int level, int i, int& lo, int& c) {
  lo = 0;
  c = n;
  for (int d = 0; d < level && c > PI_CLUSTER; ++d) {
    const int mid = order_mid(c);
    if (i >= lo + mid) { lo += mid; c -= mid; } else c = mid;
  }
}

__device__ __forceinline__ unsigned order_bits(float v) {
  const unsigned u = __float_as_uint(v);
  return (u >> 31) ? ~u : u | 0x80000000u;
}

__device__ __forceinline__ float order_float(unsigned u) {
  return __uint_as_float((u >> 31) ? u & 0x7fffffffu : ~u);
}

__global__ void __launch_bounds__(ORDER_THREADS)
order_kernel(const OrderSeg* __restrict__ segs, int32_t* __restrict__ perm, int n2) {
  extern __shared__ float4 osm[];
  OrderShared& sh = *reinterpret_cast<OrderShared*>(osm);
  float* ox = reinterpret_cast<float*>(&sh + 1);  // x, y, z of the segment's elements
  unsigned short* ia = reinterpret_cast<unsigned short*>(ox + 3 * n2);  // entry -> element of the segment
  unsigned short* ib = ia + n2;
  const OrderSeg g = segs[blockIdx.x];
  constexpr int T = ORDER_THREADS;
  const int n = g.count, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = T >> 5;
  const int nblk = (n + 31) / 32;
  int32_t* out = perm + g.perm_off;
  for (int i = tid; i < n; i += T) {
    const int64_t e = g.from_perm ? out[i] : i;
    double x[3] = {0.0, 0.0, 0.0};
    if (g.geom_type == PI_GEOM_TRIANGLE) {
      const TriSrc& t = reinterpret_cast<const TriSrc*>(g.src)[e];
      const int64_t nv = g.n_dofs / 3;
      if (g.dof_type == PI_DOF_TRIANGLE_MESH && t.vid0 >= 0 && t.vid1 >= 0 && t.vid2 >= 0 && t.vid0 < nv &&
          t.vid1 < nv && t.vid2 < nv) {
        for (int c = 0; c < 3; ++c)
          x[c] = (g.dofs[3 * (int64_t)t.vid0 + c] + g.dofs[3 * (int64_t)t.vid1 + c] + g.dofs[3 * (int64_t)t.vid2 + c]) / 3.0;
      } else {
        for (int c = 0; c < 3; ++c) x[c] = t.a[c] + (t.e1[c] + t.e2[c]) / 3.0;
      }
    } else {
      const SurfSrc& t = reinterpret_cast<const SurfSrc*>(g.src)[e];
      for (int c = 0; c < 3; ++c) x[c] = t.c[c];
    }
    for (int c = 0; c < 3; ++c) ox[c * n2 + i] = isfinite((float)x[c]) ? (float)x[c] + 0.0f : 0.f;
    ia[i] = (unsigned short)i;
  }
  for (int level = 0; level < 16; ++level) {
    for (int t = tid; t < 3 * ORDER_SLOTS; t += T) { (&sh.mn[0][0])[t] = ~0u; (&sh.mx[0][0])[t] = 0u; }
    bool big = false;
    __syncthreads();
    for (int blk = warp; blk < nblk; blk += nw) {  // bounding boxes
      int lo, c;
      order_part(n, level, blk * 32, lo, c);
      if (c <= PI_CLUSTER) continue;
      big = true;
      const int i = blk * 32 + lane;
      for (int a = 0; a < 3; ++a) {
        const unsigned u = i < n ? order_bits(ox[a * n2 + ia[i]]) : 0u;
        const unsigned l = __reduce_min_sync(0xffffffffu, i < n ? u : ~0u), h = __reduce_max_sync(0xffffffffu, u);
        if (lane == 0) { atomicMin(&sh.mn[a][lo / PI_CLUSTER], l); atomicMax(&sh.mx[a][lo / PI_CLUSTER], h); }
      }
    }
    if (!__syncthreads_or(big)) break;
    for (int t = tid; t < ORDER_SLOTS && t * PI_CLUSTER < n; t += T) {  // one thread per part, at the slot it starts in
      int lo, c;
      order_part(n, level, t * PI_CLUSTER, lo, c);
      if (lo != t * PI_CLUSTER || c <= PI_CLUSTER) continue;
      int ax = 0;
      float best = -1.f, base = 0.f;
      for (int a = 0; a < 3; ++a) {
        const float l = order_float(sh.mn[a][t]), h = order_float(sh.mx[a][t]);
        if (h - l > best) { best = h - l; ax = a; base = l; }
      }
      sh.axis[t] = ax;
      sh.base[t] = base;
      sh.scale[t] = best > 0.f && isfinite(best) ? 16777215.0f / best : 0.f;
      sh.prefix[t] = 0u;
      sh.target[t] = (unsigned)order_mid(c);
    }
    // an entry's coordinate as 24 bits of its part's box
    auto key_of = [&](int slot, int i) {
      const float v = (ox[sh.axis[slot] * n2 + ia[i]] - sh.base[slot]) * sh.scale[slot];
      return (unsigned)fminf(fmaxf(v, 0.f), 16777215.0f);
    };
    for (int round = 0; round < ORDER_ROUNDS; ++round) {
      const int shift = ORDER_BITS * (ORDER_ROUNDS - 1 - round);
      for (int t = tid; t < ORDER_SLOTS * ORDER_BINS; t += T) (&sh.hist[0][0])[t] = 0u;
      __syncthreads();
      for (int blk = warp; blk < nblk; blk += nw) {
        int lo, c;
        order_part(n, level, blk * 32, lo, c);
        const int i = blk * 32 + lane, slot = lo / PI_CLUSTER;
        if (c <= PI_CLUSTER || i >= n) continue;
        const unsigned k = key_of(slot, i);
        if ((k >> shift >> ORDER_BITS) == sh.prefix[slot]) atomicAdd(&sh.hist[slot][(k >> shift) & (ORDER_BINS - 1)], 1u);
      }
      __syncthreads();
      for (int t = warp; t < ORDER_SLOTS && t * PI_CLUSTER < n; t += nw) {  // the digit of the median
        int lo, c;
        order_part(n, level, t * PI_CLUSTER, lo, c);
        if (lo != t * PI_CLUSTER || c <= PI_CLUSTER) continue;
        const unsigned h0 = sh.hist[t][2 * lane], h1 = sh.hist[t][2 * lane + 1], want = sh.target[t];
        unsigned sum = h0 + h1;
        for (int w = 1; w < 32; w <<= 1) {
          const unsigned o = __shfl_up_sync(0xffffffffu, sum, w);
          if (lane >= w) sum += o;
        }
        const unsigned b0 = sum - h0 - h1, b1 = b0 + h0;  // entries below bins 2 lane, 2 lane + 1
        if (b0 <= want && want < b1) { sh.prefix[t] = (sh.prefix[t] << ORDER_BITS) | (2 * lane); sh.target[t] = want - b0; }
        else if (b1 <= want && want < sum) { sh.prefix[t] = (sh.prefix[t] << ORDER_BITS) | (2 * lane + 1); sh.target[t] = want - b1; }
      }
      __syncthreads();
    }
    // stable partition: below the median, and the first `target` equal to it, to the left
    for (int blk = warp; blk < nblk; blk += nw) {
      int lo, c;
      order_part(n, level, blk * 32, lo, c);
      const int i = blk * 32 + lane, slot = lo / PI_CLUSTER;
      const unsigned k = c > PI_CLUSTER && i < n ? key_of(slot, i) : ~0u, med = c > PI_CLUSTER ? sh.prefix[slot] : 0u;
      const unsigned ml = __ballot_sync(0xffffffffu, k < med), me = __ballot_sync(0xffffffffu, k == med);
      if (lane == 0) { sh.less[blk] = __popc(ml); sh.equal[blk] = __popc(me); }
    }
    __syncthreads();
    if (warp == 0) {  // exclusive prefix sums over the blocks
      unsigned carry_l = 0, carry_e = 0;
      for (int b0 = 0; b0 < nblk; b0 += 32) {
        const int blk = b0 + lane;
        const unsigned l = blk < nblk ? sh.less[blk] : 0u, e = blk < nblk ? sh.equal[blk] : 0u;
        unsigned sl = l, se = e;
        for (int w = 1; w < 32; w <<= 1) {
          const unsigned ol = __shfl_up_sync(0xffffffffu, sl, w), oe = __shfl_up_sync(0xffffffffu, se, w);
          if (lane >= w) { sl += ol; se += oe; }
        }
        if (blk < nblk) { sh.less[blk] = carry_l + sl - l; sh.equal[blk] = carry_e + se - e; }
        carry_l += __shfl_sync(0xffffffffu, sl, 31);
        carry_e += __shfl_sync(0xffffffffu, se, 31);
      }
    }
    __syncthreads();
    for (int blk = warp; blk < nblk; blk += nw) {
      int lo, c;
      order_part(n, level, blk * 32, lo, c);
      const int i = blk * 32 + lane, slot = lo / PI_CLUSTER;
      const bool in = c > PI_CLUSTER && i < n;
      const unsigned k = in ? key_of(slot, i) : ~0u, med = c > PI_CLUSTER ? sh.prefix[slot] : 0u;
      const unsigned ml = __ballot_sync(0xffffffffu, k < med), me = __ballot_sync(0xffffffffu, k == med);
      if (i >= n) continue;
      int dest = i;
      if (in) {
        const unsigned below = (1u << lane) - 1u;
        const unsigned nl = sh.less[blk] - sh.less[lo / 32] + __popc(ml & below);
        const unsigned ne = sh.equal[blk] - sh.equal[lo / 32] + __popc(me & below), rem = sh.target[slot];
        const int left = (int)(nl + min(ne, rem));
        const bool is_left = k < med || (k == med && ne < rem);
        dest = is_left ? lo + left : lo + order_mid(c) + (i - lo - left);
      }
      ib[dest] = ia[i];
    }
    __syncthreads();
    unsigned short* t = ia;
    ia = ib;
    ib = t;
  }
  // within each cluster: a warp's lanes hold entries lane and lane + 32
  for (int q = warp; q * PI_CLUSTER < n; q += nw) {
    const int p0 = q * PI_CLUSTER;
    for (int grp = 64; grp >= 2 * PI_LEAF; grp >>= 1) {
      int id[2];
      float x[2][3], v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = p0 + lane + 32 * h;
        id[h] = i < n ? ia[i] : -1;
#pragma unroll
        for (int a = 0; a < 3; ++a) x[h][a] = i < n ? ox[a * n2 + ia[i]] : INFINITY;
      }
      // the widest coordinate of the entry's group (entries past the end do not count)
      float mn[2][3], mx[2][3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int h = 0; h < 2; ++h) { mn[h][a] = x[h][a]; mx[h][a] = id[h] >= 0 ? x[h][a] : -INFINITY; }
        if (grp == 64) {
          mn[0][a] = mn[1][a] = fminf(mn[0][a], mn[1][a]);
          mx[0][a] = mx[1][a] = fmaxf(mx[0][a], mx[1][a]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          for (int w = 1; w < min(grp, 32); w <<= 1) {
            mn[h][a] = fminf(mn[h][a], __shfl_xor_sync(0xffffffffu, mn[h][a], w));
            mx[h][a] = fmaxf(mx[h][a], __shfl_xor_sync(0xffffffffu, mx[h][a], w));
          }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float dx = mx[h][0] - mn[h][0], dy = mx[h][1] - mn[h][1], dz = mx[h][2] - mn[h][2];
        v[h] = dy > dx ? (dz > dy ? x[h][2] : x[h][1]) : (dz > dx ? x[h][2] : x[h][0]);
      }
      int rank[2] = {0, 0};
      if (grp == 64) {
        for (int t = 0; t < 32; ++t) {
          const float u = __shfl_sync(0xffffffffu, v[0], t), w = __shfl_sync(0xffffffffu, v[1], t);
          rank[0] += (u < v[0] || (u == v[0] && t < lane)) + (w < v[0]);
          rank[1] += (u <= v[1]) + (w < v[1] || (w == v[1] && t < lane));
        }
      } else {
        const int g0 = lane & ~(grp - 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          for (int t = 0; t < grp; ++t) {
            const float u = __shfl_sync(0xffffffffu, v[h], g0 + t);
            rank[h] += u < v[h] || (u == v[h] && g0 + t < lane);
          }
          rank[h] += 32 * h + g0;
        }
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (id[h] >= 0) ia[p0 + rank[h]] = (unsigned short)id[h];
      __syncwarp();
    }
  }
  __syncthreads();
  // the ids of all entries are read before any is written (from_perm)
  int32_t id[ORDER_SEGMENT / T];
#pragma unroll
  for (int t = 0; t < ORDER_SEGMENT / T; ++t) {
    const int i = tid + t * T;
    if (i < n) id[t] = g.from_perm ? out[ia[i]] : ia[i];
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < ORDER_SEGMENT / T; ++t) {
    const int i = tid + t * T;
    if (i < n) out[i] = id[t];
  }
}

constexpr int PREP_THREADS = 256;
static_assert(PREP_THREADS % PI_CLUSTER == 0 && PI_CLUSTER == 64, "a cluster is two warps of the preparing CTA");

// grid (x: blocks of pool entries, y: object).  Writes the FP32 local-frame
// pools and the bounding sphere of every cluster and leaf: its centre (that of the
// bounding box, an FP32 point) and its radius, which for a surfel includes the
// reach of its own expansion, rho |A| for a disk and 2.5 sigma |A| for a
// Gaussian (the n-th root of E|Z|^n at n = 16 is 2.48), |A| bounded by the root of
// its squared entries' sum.
__global__ void __launch_bounds__(PREP_THREADS)
prepare_elems_kernel(const PrepObj* objs, const ObjDev* od, float4* tri_pool, float4* surf_pool, float4* tri_lo,
                     float4* surf_lo, float4* surf_nref, const int32_t* perm, float4* clusters, float4* leaves,
                     unsigned* cl_rho, int only) {
  const int oi = only >= 0 ? only : blockIdx.y;
  const PrepObj o = objs[oi];
  if ((int64_t)blockIdx.x * blockDim.x >= o.n_elems) return;
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const double* org = od[oi].origin;
  float v[3][3];        // points that bound the entry (triangles: vertices), object frame
  float reach = 0.f;    // added to their distance from the centre
  bool ok = p < o.n_elems;
  const int64_t e = !ok ? 0 : o.perm_off >= 0 ? perm[o.perm_off + p] : p;
  if (ok && o.geom_type == PI_GEOM_TRIANGLE) {
    const TriSrc& t = reinterpret_cast<const TriSrc*>(o.src)[e];
    double a[3], e1[3], e2[3];
    if (o.dof_type == PI_DOF_TRIANGLE_MESH) {
      int64_t nv = o.n_dofs / 3;
      ok = t.vid0 >= 0 && t.vid1 >= 0 && t.vid2 >= 0 && t.vid0 < nv && t.vid1 < nv && t.vid2 < nv;
      if (ok) {
        const double* v0 = o.dofs + 3 * t.vid0;
        const double* v1 = o.dofs + 3 * t.vid1;
        const double* v2 = o.dofs + 3 * t.vid2;
        for (int c = 0; c < 3; ++c) { a[c] = v0[c]; e1[c] = v1[c] - v0[c]; e2[c] = v2[c] - v0[c]; }
      }
    } else {
      affine_apply(o.dofs, t.a, a, true);
      affine_apply(o.dofs, t.e1, e1, false);
      affine_apply(o.dofs, t.e2, e2, false);
    }
    float4* dst = tri_pool + 3 * (o.pool_off + p);
    if (!ok) {  // unset vertex ids contribute nothing (triangle_mesh_dof.cpp:44-45)
      dst[0] = make_float4(0.f, 0.f, 0.f, 0.f); dst[1] = dst[0]; dst[2] = dst[0];
      tri_lo[o.pool_off + p] = dst[0];
    } else {
      double S[3] = {0.5 * (e1[1] * e2[2] - e1[2] * e2[1]), 0.5 * (e1[2] * e2[0] - e1[0] * e2[2]),
                     0.5 * (e1[0] * e2[1] - e1[1] * e2[0])};
      // centroid m = a + (e1 + e2)/3 relative to the object origin, FP32 hi + lo;
      // beside its low word the longest edge (the series-length bound k |e|max)
      const double l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
      const double l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
      const double l3 = (e2[0] - e1[0]) * (e2[0] - e1[0]) + (e2[1] - e1[1]) * (e2[1] - e1[1]) +
                        (e2[2] - e1[2]) * (e2[2] - e1[2]);
      const float lmax = (float)sqrt(fmax(fmax(l1, l2), l3));
      float mh[3], ml[3];
      for (int c = 0; c < 3; ++c) {
        const double m = a[c] + (e1[c] + e2[c]) / 3.0 - org[c];
        mh[c] = (float)m;
        ml[c] = (float)(m - (double)mh[c]);
        const double r = a[c] - org[c];
        v[0][c] = (float)r; v[1][c] = (float)(r + e1[c]); v[2][c] = (float)(r + e2[c]);
      }
      dst[0] = make_float4(mh[0], mh[1], mh[2], (float)S[0]);
      tri_lo[o.pool_off + p] = make_float4(ml[0], ml[1], ml[2], lmax);
      dst[1] = make_float4((float)e1[0], (float)e1[1], (float)e1[2], (float)S[1]);
      dst[2] = make_float4((float)e2[0], (float)e2[1], (float)e2[2], (float)S[2]);
    }
  } else if (ok) {
    const SurfSrc& s = reinterpret_cast<const SurfSrc*>(o.src)[e];
    double c[3], n[3];
    affine_apply(o.dofs, s.c, c, true);
    affine_apply(o.dofs, s.n, n, false);  // n' = A n so that k'.n = k.(A n) with k' = A^T k
    float4* dst = surf_pool + 2 * (o.pool_off + p);
    float ch[3], cl[3];
    for (int a = 0; a < 3; ++a) {
      const double r = c[a] - org[a];
      ch[a] = (float)r;
      cl[a] = (float)(r - (double)ch[a]);
      v[0][a] = v[1][a] = v[2][a] = ch[a];
    }
    dst[0] = make_float4(ch[0], ch[1], ch[2], (float)s.p0);
    surf_lo[o.pool_off + p] = make_float4(cl[0], cl[1], cl[2], 0.f);
    const double nn = s.n[0] * s.n[0] + s.n[1] * s.n[1] + s.n[2] * s.n[2];
    const double in = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
    surf_nref[o.pool_off + p] =
        make_float4((float)(s.n[0] * in), (float)(s.n[1] * in), (float)(s.n[2] * in), (float)(1.0 - nn));
    dst[1] = make_float4((float)n[0], (float)n[1], (float)n[2], (float)s.p1);
    // |k'_perp|^2 <= |k'|^2 max(1, |1 - |n|^2| + |n|^2) with |k'| <= |A| |k|
    double A2 = 0.0;
    for (int a = 3; a < 12; ++a) A2 += o.dofs[a] * o.dofs[a];
    reach = (float)((o.geom_type == PI_GEOM_DISK ? 1.0 : 2.5) * fabs(s.p0) *
                    sqrt(A2 * fmax(1.0, fabs(1.0 - nn) + nn)));
  }
  // the bounding box: of the leaf, within the warp, then over the cluster's two warps
  float lo[3], hi[3], lctr[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[c] = ok ? fminf(fminf(v[0][c], v[1][c]), v[2][c]) : INFINITY;
    hi[c] = ok ? fmaxf(fmaxf(v[0][c], v[1][c]), v[2][c]) : -INFINITY;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      if (w == PI_LEAF) lctr[c] = lo[c] <= hi[c] ? 0.5f * lo[c] + 0.5f * hi[c] : 0.f;
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], w));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], w));
    }
  }
  float lrho = 0.f;
  if (ok)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float dx = v[i][0] - lctr[0], dy = v[i][1] - lctr[1], dz = v[i][2] - lctr[2];
      lrho = fmaxf(lrho, sqrtf(dx * dx + dy * dy + dz * dz) + reach);
    }
#pragma unroll
  for (int w = 1; w < PI_LEAF; w <<= 1) lrho = fmaxf(lrho, __shfl_xor_sync(0xffffffffu, lrho, w));
  if (threadIdx.x % PI_LEAF == 0 && p < o.n_elems)
    leaves[o.cl_off * (PI_CLUSTER / PI_LEAF) + p / PI_LEAF] = make_float4(lctr[0], lctr[1], lctr[2], lrho);
  __shared__ float box[PREP_THREADS / 32][6];
  __shared__ float rad[PREP_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int c = 0; c < 3; ++c) { box[warp][c] = lo[c]; box[warp][3 + c] = hi[c]; }
  __syncthreads();
  float ctr[3], rho = 0.f;
  bool any = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float l = fminf(box[warp][c], box[warp ^ 1][c]), h = fmaxf(box[warp][3 + c], box[warp ^ 1][3 + c]);
    any = any && l <= h;
    ctr[c] = l <= h ? 0.5f * l + 0.5f * h : 0.f;
  }
  if (ok)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float dx = v[i][0] - ctr[0], dy = v[i][1] - ctr[1], dz = v[i][2] - ctr[2];
      rho = fmaxf(rho, sqrtf(dx * dx + dy * dy + dz * dz) + reach);
    }
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) rho = fmaxf(rho, __shfl_xor_sync(0xffffffffu, rho, w));
  if (lane == 0) rad[warp] = rho;
  __syncthreads();
  if ((threadIdx.x & (PI_CLUSTER - 1)) == 0 && p < o.n_elems) {
    rho = any ? fmaxf(rad[warp], rad[warp + 1]) : 0.f;
    clusters[o.cl_off + p / PI_CLUSTER] = make_float4(ctr[0], ctr[1], ctr[2], rho);
    atomicMax(cl_rho + oi, __float_as_uint(rho));  // non-negative floats order like their bits
  }
}

constexpr int FF_THREADS = 128;
constexpr int FF_WARPS = FF_THREADS / 32;
constexpr int FF_CTAS = 4;  // per SM: 128 registers; at five, 96 registers spill and the kernel is 7% slower
constexpr int FF_TILE = 256;  // elements staged per shared-memory tile (a multiple of FF_CHUNK)
constexpr int FF_CHUNK = 32;  // elements summed in FP32 before the compensated outer sum
static_assert(FF_TILE % FF_CHUNK == 0, "element chunks must not straddle tiles");

// Sums over thousands of elements: each thread adds FF_CHUNK element terms into
// a fresh FP32 partial, then adds the partial to a Kahan-compensated running
// sum, so rounding does not grow with the element count (a plain FP32 sum over
// 1,280 triangles measured ~1e-6 of max|A| per node).  The partials live in
// registers; the running sums and compensations live in shared memory, where
// they are touched once per FF_CHUNK elements, which leaves the registers to
// the element loop.
// A float4 from shared memory, loaded where it is written in the source: the
// element loop reads its radius constants each time instead of keeping them
// in registers across the loop.
__device__ __forceinline__ float4 ld_shared_f4(const float4* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

template <int R>
struct Acc {
  static_assert(R % 2 == 0, "radii are paired for packed FP32");
  // current chunk; radii (2p, 2p + 1) in one float2, the operand of packed FP32
  float2 re2[R / 2], im2[R / 2];
  float* run;  // run[(4 i + v) FF_THREADS]: v = sum re, sum im, compensation re, im
  __device__ __forceinline__ float& re(int i) { return (i & 1) ? re2[i >> 1].y : re2[i >> 1].x; }
  __device__ __forceinline__ float& im(int i) { return (i & 1) ? im2[i >> 1].y : im2[i >> 1].x; }
  __device__ __forceinline__ void init(float* base) {
    run = base + threadIdx.x;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      re(i) = im(i) = 0.f;
#pragma unroll
      for (int v = 0; v < 4; ++v) run[(4 * i + v) * FF_THREADS] = 0.f;
    }
  }
  __device__ __forceinline__ void flush() {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float* p = run + 4 * i * FF_THREADS;
      float sre = p[0], sim = p[FF_THREADS], cre = p[2 * FF_THREADS], cim = p[3 * FF_THREADS];
      float y = re(i) - cre, t = sre + y;
      cre = (t - sre) - y;
      sre = t;
      y = im(i) - cim;
      t = sim + y;
      cim = (t - sim) - y;
      sim = t;
      p[0] = sre; p[FF_THREADS] = sim; p[2 * FF_THREADS] = cre; p[3 * FF_THREADS] = cim;
      re(i) = 0.f;
      im(i) = 0.f;
    }
  }
  __device__ __forceinline__ float& sre(int i) const { return run[4 * i * FF_THREADS]; }
  __device__ __forceinline__ float& sim(int i) const { return run[(4 * i + 1) * FF_THREADS]; }
};

// Adds the triangles [l0, l1) of a leaf to the radii of pairs [p0, np) by the
// leaf's expansion about its centre lf (moments.cu has the formulas), in units
// of a power of two above its radius.
template <int R>
__device__ __forceinline__ void leaf_sum(const float4* tile, int l0, int l1, float4 lf, float3 dh, float3 dl,
                                         float inv_norm, const float2* ctab, const float4* kp, int p0, int np,
                                         Acc<R>& acc) {
  const int ex = lf.w > 0.f ? min(120, max(-100, ilogbf(lf.w) + 1)) : 0;
  const float s = __int_as_float((127 + ex) << 23), inv_s = __int_as_float((127 - ex) << 23);
  const float3 d = make_float3(dh.x * inv_s, dh.y * inv_s, dh.z * inv_s);
  float2 mu[MOMENT_TERMS];
#pragma unroll
  for (int n = 0; n < MOMENT_TERMS; ++n) mu[n] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int e = l0; e < l1; e += 2) {  // two triangles per packed instruction
    float a[2], bv[2], c[2], g[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = min(e + h, l1 - 1);
      const float4 q0 = tile[3 * t], q1 = tile[3 * t + 1], q2 = tile[3 * t + 2], ml = tile[3 * FF_TILE + t];
      const float mx = (q0.x - lf.x) + ml.x, my = (q0.y - lf.y) + ml.y, mz = (q0.z - lf.z) + ml.z;
      const float sm = fmaf(d.x, mx, fmaf(d.y, my, d.z * mz));
      const float s1 = fmaf(d.x, q1.x, fmaf(d.y, q1.y, d.z * q1.z));
      const float s2 = fmaf(d.x, q2.x, fmaf(d.y, q2.y, d.z * q2.z));
      g[h] = e + h < l1 ? dh.x * q0.w + dh.y * q1.w + dh.z * q2.w : 0.f;
      a[h] = fmaf(s1 + s2, -1.0f / 3.0f, sm);
      bv[h] = a[h] + s1;
      c[h] = a[h] + s2;
    }
    tri_moments(make_float2(a[0], a[1]), make_float2(bv[0], bv[1]), make_float2(c[0], c[1]), make_float2(g[0], g[1]), mu);
  }
  constexpr FmConst<PI_GEOM_TRIANGLE> C{};
  float2 cf8[MOMENT_TERMS / 2];  // (real, imaginary) coefficients of u^j
#pragma unroll
  for (int j = 0; j < MOMENT_TERMS / 2; ++j) {
    const float f0 = (j & 1) ? -C.f[2 * j] : C.f[2 * j], f1 = (j & 1) ? -C.f[2 * j + 1] : C.f[2 * j + 1];
    cf8[j] = make_float2((mu[2 * j].x + mu[2 * j].y) * (f0 * inv_norm), (mu[2 * j + 1].x + mu[2 * j + 1].y) * (f1 * inv_norm));
  }
  const df sc = cdot(dh, dl, make_float3(lf.x, lf.y, lf.z));
  const float2 sh = dup2(sc.hi), sl = dup2(sc.lo);
#pragma unroll
  for (int p = 0; p < R / 2; ++p) {
    if (p < p0 || p >= np) continue;
    const float4 kx = ld_shared_f4(kp + 2 * p);
    const float2 kth = make_float2(kx.x, kx.y);
    const cf2 P = cis_tab_df2(ctab, kth, make_float2(kx.z, kx.w), sh, sl);
    const float2 k = __fmul2_rn(kth, dup2(PI_TURN64 * s)), u = __fmul2_rn(k, k);
    const float2 ua = dup2(u.x), ub = dup2(u.y);
    float2 x = cf8[7], y = cf8[7];
#pragma unroll
    for (int j = 6; j >= 0; --j) {
      x = __ffma2_rn(x, ua, cf8[j]);
      y = __ffma2_rn(y, ub, cf8[j]);
    }
    const float2 tr = make_float2(x.x, y.x), ti = __fmul2_rn(k, make_float2(x.y, y.y));
    acc.re2[p] = __ffma2_rn(P.re, tr, __ffma2_rn(neg2(P.im), ti, acc.re2[p]));
    acc.im2[p] = __ffma2_rn(P.re, ti, __ffma2_rn(P.im, tr, acc.im2[p]));
  }
}

// The grid is (CTAs per object) x (objects or evaluations); the CTAs are
// taken in the order the hardware dispatches them (x fastest, then y) and
// re-mapped so that the object slot varies fastest and the CTA index within
// the object slowest: every object's first CTAs (its largest-k radial block,
// below) run before any object's later ones.
// SERVE: the object slot indexes `evals` (serving evaluations: optional rotation of
// the k directions, local-frame direction-major output, row maximum);
// otherwise it indexes the batch's objects (largest first) and J is written
// q-major with the origin phase.
// The CTAs of a thread-block cluster (S along x) take the same object,
// directions and radii and split the elements; their running sums meet
// through distributed shared memory, each CTA writing every S-th radius.
template <int R, bool SERVE>
__device__ __forceinline__ void ff_body(const KGridDev& kg, const BatchDev& b, float2* __restrict__ J,
                                        int scale_sqrt_w, const EvalDev* __restrict__ evals,
                                        unsigned* __restrict__ row_amax) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const unsigned lin = (blockIdx.y * gridDim.x + blockIdx.x) / (unsigned)S;
  const int slot = (int)(lin % gridDim.y), cta = (int)(lin / gridDim.y);
  const int oi = SERVE ? evals[slot].obj : b.order[slot];
  const ObjDev od = b.objs[oi];
  // the radii [0, r_first) are moments.cu's
  const int r_first = moment_radii(kg, od.type, __uint_as_float(b.cl_rho[oi]));
  const int nrb = (kg.L - r_first + R - 1) / R;
  const int ndt = (kg.Me + 31) / 32;
  if (cta * FF_WARPS >= ndt * nrb) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Warps of a CTA take neighbouring direction blocks at the same radial
  // block: they see the same radii, so they take the large-spread branch at
  // the same points of the element loop and reach the tile barriers together.
  // Radial blocks run in descending order of k: on a grid of ascending radii
  // the blocks of large k, whose elements take the long branches, start
  // first (for all objects, by the re-mapping above) and the launch ends on
  // light blocks (with neighbouring radii per warp the blocks differ
  // several-fold in cost).
  // A lane evaluates direction j = dpair[.].x and also writes its antipode
  // jm = dpair[.].y (A(-k) = -conj A(k)), when the grid has one.
  const int item = cta * FF_WARPS + warp;
  const int ib = item / ndt, dt = item - ib * ndt;
  const int rlo = kg.L - (ib + 1) * R;         // the block's radii are rlo .. rlo + R - 1,
  const int skip = max(0, r_first - rlo);      // of which the first `skip` are not its own
  const int ei = dt * 32 + lane;
  const bool busy = item < ndt * nrb, active = busy && ei < kg.Me;
  int j = 0, jm = -1;
  // (lanes past the last direction repeat it, for the votes, and write nothing)
  if (busy) { const int2 pr = kg.dpair[min(ei, kg.Me - 1)]; j = pr.x; jm = pr.y; }

  float3 dh = make_float3(0.f, 0.f, 0.f), dl = dh;
  float inv_norm = 0.f, dnorm = 0.f;
  if (busy) {
    float4 h = kg.dir_hi[j], l = kg.dir_lo[j];
    dh = make_float3(h.x, h.y, h.z); dl = make_float3(l.x, l.y, l.z);
    inv_norm = h.w; dnorm = l.w;
    if (SERVE && evals[slot].rotate) {
      // rotated object: its form factor at k is the unrotated one's at R^T k
      // (|R^T k| = |k|); the direction is turned in FP64 and re-split.
      const double* Rm = evals[slot].R;
      const double d0 = (double)h.x + (double)l.x, d1 = (double)h.y + (double)l.y, d2 = (double)h.z + (double)l.z;
      double e[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) e[a] = Rm[a] * d0 + Rm[3 + a] * d1 + Rm[6 + a] * d2;
      dh = make_float3((float)e[0], (float)e[1], (float)e[2]);
      dl = make_float3((float)(e[0] - (double)dh.x), (float)(e[1] - (double)dh.y), (float)(e[2] - (double)dh.z));
    }
  }
  // radii r = rlo + i: a warp's radii are neighbours, so warps at small k
  // take the short series for every radius of most elements (the lean loop
  // below, chosen once per element for the whole warp), and the branches of
  // the others are taken together more often.
  // The warp's radii as (k 64 / 2 pi hi, lo, k^2, k^3), in shared memory:
  // every lane reads the same entry (a broadcast), once per element and
  // radius, which keeps them out of the registers the element loop needs.
  __shared__ float4 krad[FF_WARPS][R];
  // the phasor table of cis_tab_*
  __shared__ float2 ctab_sm[PHASOR_ENTRIES * PHASOR_COPIES];
  stage_phasors<PHASOR_COPIES>(kg.cis_tab, ctab_sm);
  const float2* ctab = ctab_sm + (threadIdx.x % PHASOR_COPIES);
  __shared__ float2 ctabm_sm[PHASOR_ENTRIES * PHASOR_M1_COPIES];
  stage_phasors<PHASOR_M1_COPIES>(kg.cis_tabm, ctabm_sm);
  const float2* ctabm = ctabm_sm + (threadIdx.x % PHASOR_M1_COPIES);
  if (lane < R) {
    const int r = rlo + lane;
    const bool ok = item < ndt * nrb && lane >= skip;
    const float2 k = ok ? kg.kmag[r] : make_float2(0.f, 0.f);
    const float2 k2 = ok ? kg.kt64[r] : make_float2(0.f, 0.f);
    krad[warp][lane] = make_float4(k2.x, k2.y, k.x * k.x, k.x * k.x * k.x);
  }
  // the same constants paired for packed FP32: radii (2p, 2p + 1) as
  // (kt.hi, kt.hi', kt.lo, kt.lo') and (k^2, k^2', k^3, k^3')
  __shared__ float4 kpair[FF_WARPS][R];
  if (lane < R / 2) {
    float v[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = rlo + 2 * lane + h;
      const bool ok = item < ndt * nrb && 2 * lane + h >= skip;
      const float2 k = ok ? kg.kmag[r] : make_float2(0.f, 0.f);
      const float2 k2 = ok ? kg.kt64[r] : make_float2(0.f, 0.f);
      v[h][0] = k2.x; v[h][1] = k2.y; v[h][2] = k.x * k.x; v[h][3] = k.x * k.x * k.x;
    }
    kpair[warp][2 * lane] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    kpair[warp][2 * lane + 1] = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
  }
  __syncthreads();
  const float4* kw = krad[warp];
  const float4* kp = kpair[warp];
  // (k rho)^2 up to which a leaf's expansion is used (never without kg.moments)
  const float bound2 = kg.moments ? MOMENT_X_TRI * MOMENT_X_TRI : -1.f;
  // the warp's largest k^2 and its smallest (a grid without kg.moments may hold its radii in any order)
  float kmax2 = 0.f, kmin2 = INFINITY;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    kmax2 = fmaxf(kmax2, kw[i].z);
    if (i >= skip) kmin2 = fminf(kmin2, kw[i].z);
  }
  __shared__ float run_sm[4 * R * FF_THREADS];
  Acc<R> acc;
  acc.init(run_sm);
  float2 total[R];

  // tile[0, 3 FF_TILE): the elements' pool entries (surfels use the first
  // 2 FF_TILE and put their unit normals at tile[2 FF_TILE + e]);
  // tile[3 FF_TILE + e]: the low word of element e's centroid (centre).
  __shared__ float4 tile[4 * FF_TILE];
  __shared__ float4 leaf[FF_TILE / PI_LEAF];
  // this CTA's elements [n0, n), whole chunks
  const int per = (od.n_elems + S * FF_CHUNK - 1) / (S * FF_CHUNK) * FF_CHUNK;
  const int n0 = min(od.n_elems, rank * per), n = min(od.n_elems, n0 + per);

  if (od.type == PI_GEOM_TRIANGLE) {
    const float4* src = b.tri_pool + 3 * od.elem_off;
    const float4* lo = b.tri_lo + od.elem_off;
    const float4* leaves = b.leaves + od.cl_off * (PI_CLUSTER / PI_LEAF);
    for (int base = n0; base < n; base += FF_TILE) {
      const int cnt = min(FF_TILE, n - base);
      __syncthreads();
      for (int t = threadIdx.x; t < 3 * cnt; t += FF_THREADS) tile[t] = src[3 * (int64_t)base + t];
      for (int t = threadIdx.x; t < cnt; t += FF_THREADS) tile[3 * FF_TILE + t] = lo[base + t];
      for (int t = threadIdx.x; t * PI_LEAF < cnt; t += FF_THREADS) leaf[t] = leaves[base / PI_LEAF + t];
      __syncthreads();
      if (busy) {  // every lane of a busy warp (the votes below); those without a direction write nothing
        // chunks of FF_CHUNK elements: leaves from all over the tile, since the
        // elements of a compact patch add up in phase and their FP32 partial sum
        // would round coarser
        const int nch = (cnt + FF_CHUNK - 1) / FF_CHUNK;
        for (int ch = 0; ch < nch; ++ch) {
        for (int l0 = ch * PI_LEAF; l0 < cnt; l0 += nch * PI_LEAF) {
        const int l1 = min(l0 + PI_LEAF, cnt);
        int from = skip;  // first radius of the block that the elements are summed at one by one
        {
          // radii ascend: those of the leading pairs lie within the expansion's reach of this leaf
          const float4 lf = leaf[l0 / PI_LEAF];
          const float reach2 = lf.w * lf.w;
          int np = 0;
#pragma unroll
          for (int p = 0; p < R / 2; ++p) np += kp[2 * p + 1].y * reach2 <= bound2 ? 1 : 0;
          // worth it for two pairs, or if nothing else is left (the moments
          // cost about as much as one pair summed directly)
          if (np == R / 2 || np >= skip / 2 + 2) {
            leaf_sum<R>(tile, l0, l1, lf, dh, dl, inv_norm, ctab, kp, skip / 2, np, acc);
            from = 2 * np;
            if (from == R) continue;
          }
        }
        for (int e = l0; e < l1; ++e) {
          const float4 q0 = tile[3 * e], q1 = tile[3 * e + 1], q2 = tile[3 * e + 2];
          const float3 m = make_float3(q0.x, q0.y, q0.z);  // centroid, object frame
          const float3 e1 = make_float3(q1.x, q1.y, q1.z);
          const float3 e2 = make_float3(q2.x, q2.y, q2.z);
          // -2 (khat . S): gamma of the reference times the -2 of Phi = -2 e[..]
          const float g = -2.0f * (dh.x * q0.w + dh.y * q1.w + dh.z * q2.w) * inv_norm;
          const float4 ml = tile[3 * FF_TILE + e];
          const df sm = cdot2_un(dh, dl, m, make_float3(ml.x, ml.y, ml.z));
          const float kl = ml.w * dnorm;  // k kl bounds k sp: the short series below k kl = 1
          const float slim = rcp_fast(kl * kl);  // the short series for k^2 < 1 / kl^2 (inf when kl = 0)
          const float s1 = fmaf(dh.x, e1.x, fmaf(dh.y, e1.y, dh.z * e1.z));
          const float s2 = fmaf(dh.x, e2.x, fmaf(dh.y, e2.y, dh.z * e2.z));
          if (__all_sync(0xffffffffu, kmax2 < slim)) {
            // every radius of this thread takes the short series (the same for
            // all lanes on a tensor grid: unit directions)
            const TriPolyShort tp = tri_series_coeffs_short(s1, s2, g);
            const float2 smh = make_float2(sm.hi, sm.hi), sml = make_float2(sm.lo, sm.lo);
#pragma unroll
            for (int p = 0; p < R / 2; ++p) {
              if (2 * p + 1 < from) continue;
              const float4 kx = ld_shared_f4(kp + 2 * p), ku = ld_shared_f4(kp + 2 * p + 1);
              const cf2 P = cis_tab_df2(ctab, make_float2(kx.x, kx.y), make_float2(kx.z, kx.w), smh, sml);
              const cf2 T = tri_series_eval_short2(tp, make_float2(ku.x, ku.y), make_float2(ku.z, ku.w));
              acc.re2[p] = __ffma2_rn(P.re, T.re, __ffma2_rn(neg2(P.im), T.im, acc.re2[p]));
              acc.im2[p] = __ffma2_rn(P.re, T.im, __ffma2_rn(P.im, T.re, acc.im2[p]));
            }
            continue;
          }
          const TriGaps tg = tri_gaps(s1, s2, sm);
          const float gD = g * rcp_fast(tg.D);
          // the warp's least and greatest spread (positive floats order as their bits):
          // two reductions per element in place of two votes per radius
          const unsigned Db = __float_as_uint(tg.D);
          const float d_lo = __uint_as_float(__reduce_min_sync(0xffffffffu, Db)),
                      d_hi = __uint_as_float(__reduce_max_sync(0xffffffffu, Db));
          const float wide_lo = d_lo * d_lo, wide_hi = 1.0f / 9.0f * d_hi * d_hi;
          // no series where every lane is wide at every radius left
          TriPoly2 tp;
          if ((kg.moments ? kw[from].z : kmin2) * (1.0f / 9.0f * d_lo * d_lo) < 1.0f) tp = tri_series_coeffs2(s1, s2, g);
          // a pair of radii at a time, without a branch between them where both are
          // wide, or both narrow, for every lane: their chains overlap (256 solids
          // 15.37 -> 14.19 ms; the two radii per packed instruction here took longer)
          const auto add = [&](int i, cf P, cf T) {
            acc.re(i) = fmaf(P.re, T.re, fmaf(-P.im, T.im, acc.re(i)));
            acc.im(i) = fmaf(P.re, T.im, fmaf(P.im, T.re, acc.im(i)));
          };
#pragma unroll
          for (int p = 0; p < R / 2; ++p) {
            if (2 * p + 1 < from) continue;
            const float4 ka = ld_shared_f4(kw + 2 * p), kb = ld_shared_f4(kw + 2 * p + 1);
            const float klo = fminf(ka.z, kb.z), khi = fmaxf(ka.z, kb.z);
            if (klo * wide_lo >= 1.0f && klo * wide_hi >= 1.0f) {
              const float2 kta = make_float2(ka.x, ka.y), ktb = make_float2(kb.x, kb.y);
              const cf P0 = cis_tab_df(ctab, kta, tg.sv), P1 = cis_tab_df(ctab, ktb, tg.sv);
              const cf T0 = tri_wide(ctabm, kta, tg, gD * rcp_fast(ka.z)), T1 = tri_wide(ctabm, ktb, tg, gD * rcp_fast(kb.z));
              add(2 * p, P0, T0);
              add(2 * p + 1, P1, T1);
            } else if (khi * wide_hi < 1.0f) {
              const cf P0 = cis_tab_df(ctab, make_float2(ka.x, ka.y), sm), P1 = cis_tab_df(ctab, make_float2(kb.x, kb.y), sm);
              add(2 * p, P0, tri_series_eval(tp, ka.z, ka.w));
              add(2 * p + 1, P1, tri_series_eval(tp, kb.z, kb.w));
            } else {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float4 kr = h ? kb : ka;
                const float2 kt = make_float2(kr.x, kr.y);
                cf P, T;  // the phase's phasor, and the rest with gamma folded in
                if (kr.z * wide_hi < 1.0f) {
                  P = cis_tab_df(ctab, kt, sm);
                  T = tri_series_eval(tp, kr.z, kr.w);  // centroid Taylor series
                } else {
                  P = cis_tab_df(ctab, kt, tg.sv);
                  T = tri_wide(ctabm, kt, tg, gD * rcp_fast(kr.z));
                  if (kr.z * wide_lo < 1.0f) {
                    // lanes of small spread, whose divided differences cancel
                    const bool narrow = kr.z * tg.D * tg.D < 1.0f;
                    const cf Q = cis_tab_df(ctab, kt, sm), U = tri_series_eval(tp, kr.z, kr.w);
                    P = cf{narrow ? Q.re : P.re, narrow ? Q.im : P.im};
                    T = cf{narrow ? U.re : T.re, narrow ? U.im : T.im};
                  }
                }
                add(2 * p + h, P, T);
              }
            }
          }
        }
        }
        acc.flush();
        }
      }
    }
  } else {
    const float4* src = b.surf_pool + 2 * od.elem_off;
    const float4* lo = b.surf_lo + od.elem_off;
    const bool disk = od.type == PI_GEOM_DISK;
    // v = A^T dir, so k' = kmag v and |k'|^2 = kmag^2 qd
    const float* Am = od.A;
    const float3 v = make_float3(Am[0] * dh.x + Am[3] * dh.y + Am[6] * dh.z, Am[1] * dh.x + Am[4] * dh.y + Am[7] * dh.z,
                                 Am[2] * dh.x + Am[5] * dh.y + Am[8] * dh.z);
    const float qd = fmaf(v.x, v.x, fmaf(v.y, v.y, v.z * v.z));
    const float4* nref = b.surf_nref + od.elem_off;
    for (int base = n0; base < n; base += FF_TILE) {
      const int cnt = min(FF_TILE, n - base);
      __syncthreads();
      for (int t = threadIdx.x; t < 2 * cnt; t += FF_THREADS) tile[t] = src[2 * (int64_t)base + t];
      for (int t = threadIdx.x; t < cnt; t += FF_THREADS) {
        tile[2 * FF_TILE + t] = nref[base + t];
        tile[3 * FF_TILE + t] = lo[base + t];
      }
      __syncthreads();
      if (busy) {  // every lane of a busy warp (the votes below); those without a direction write nothing
        const int nch = (cnt + FF_CHUNK - 1) / FF_CHUNK;  // as above
        for (int ch = 0; ch < nch; ++ch) {
        for (int e = ch; e < cnt; e += nch) {
          const float4 q0 = tile[2 * e], q1 = tile[2 * e + 1], nr = tile[2 * FF_TILE + e];
          const float4 cl = tile[3 * FF_TILE + e];
          const df sc = cdot2_un(dh, dl, make_float3(q0.x, q0.y, q0.z), make_float3(cl.x, cl.y, cl.z));
          const float sn = dh.x * q1.x + dh.y * q1.y + dh.z * q1.z;  // dir . (A n)
          // |k'_perp|^2 / kmag^2 = qd (1 - |n|^2) + |n|^2 |v x n/|n||^2: its rounding
          // shrinks with the angle to the normal, where qd - sn^2 would leave ~1e-7
          // (a Bessel argument off by (k rho)^2 1e-7 / (2 x) rad).
          const float cx = fmaf(v.y, nr.z, -v.z * nr.y), cy = fmaf(v.z, nr.x, -v.x * nr.z),
                      cz = fmaf(v.x, nr.y, -v.y * nr.x);
          const float perp = fmaf(qd, nr.w, (1.0f - nr.w) * fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
          const float amp = sn * inv_norm * q1.w;                   // area|w * (k'.n)/|k|
          // two radii per packed FP32 phasor and accumulation (cis_tab_df2)
          const float2 sch = make_float2(sc.hi, sc.hi), scl = make_float2(sc.lo, sc.lo);
          if (disk) {
            const float amp2 = 2.0f * amp;
            const float rr = q0.w * sqrt_fast(fmaxf(perp, 0.f)) * PI_TURN64;  // rho |k'_perp| / kmag, per 1/64 turn
#pragma unroll
            for (int p = 0; p < R / 2; ++p) {
              if (2 * p + 1 < skip) continue;
              const float4 kx = ld_shared_f4(kp + 2 * p);
              const float xa = kx.x * rr, xb = kx.y * rr;
              const float2 S = j1x_pair(xa, xb);
              const cf2 P = cis_tab_df2(ctab, make_float2(kx.x, kx.y), make_float2(kx.z, kx.w), sch, scl);
              const float2 m = make_float2(S.x * amp2, S.y * amp2);
              acc.re2[p] = __ffma2_rn(m, P.re, acc.re2[p]);
              acc.im2[p] = __ffma2_rn(m, P.im, acc.im2[p]);
            }
          } else {
            const float hs = -0.5f * q0.w * q0.w * perp;
#pragma unroll
            for (int p = 0; p < R / 2; ++p) {
              if (2 * p + 1 < skip) continue;
              const float4 kx = ld_shared_f4(kp + 2 * p), ku = ld_shared_f4(kp + 2 * p + 1);
              const float2 m = make_float2(__expf(hs * ku.x) * amp, __expf(hs * ku.y) * amp);
              const cf2 P = cis_tab_df2(ctab, make_float2(kx.x, kx.y), make_float2(kx.z, kx.w), sch, scl);
              acc.re2[p] = __ffma2_rn(m, P.re, acc.re2[p]);
              acc.im2[p] = __ffma2_rn(m, P.im, acc.im2[p]);
            }
          }
        }
        acc.flush();
        }
      }
    }
  }

  acc.flush();
  const auto mine = [&](int i) { return (i & (S - 1)) == rank; };  // S is a power of two
  if (S > 1) {
    cluster.sync();
    // the sums of this CTA's radii over the cluster; compensated, in the
    // order of the ranks
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!mine(i)) continue;
      kbsum re{0.f, 0.f}, im{0.f, 0.f};
      for (int q = 0; q < S; ++q) {
        const float* o = cluster.map_shared_rank(run_sm, q) + 4 * i * FF_THREADS + threadIdx.x;
        re.add(o[0]); im.add(o[FF_THREADS]);
        re.lo -= o[2 * FF_THREADS]; im.lo -= o[3 * FF_THREADS];
      }
      total[i] = make_float2(re.hi + re.lo, im.hi + im.lo);
    }
    cluster.sync();  // no CTA leaves while its sums are read
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (mine(i)) { acc.sre(i) = total[i].x; acc.sim(i) = total[i].y; }
  }
  if (!active) return;
  if (SERVE) {
    const EvalDev& ev = evals[slot];
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rlo + i;
      if (i >= skip && mine(i)) {
        const int64_t q = (int64_t)r * kg.M + j;
        cf v{acc.sre(i), acc.sim(i)};
        if (kw[i].x * PI_TURN64 * dnorm < 1e-10f) v = cf{0.f, 0.f};  // A(0) = 0 (affine_dof.cpp:64-65)
        const float sw = serve_scale(kg, q, jm >= 0 ? (int64_t)r * kg.M + jm : -1);
        ev.dst[(int64_t)kg.ecol[ei] * kg.L + r] = make_float2(v.re * sw, v.im * sw);
        m = fmaxf(m, fmaxf(fabsf(v.re * sw), fabsf(v.im * sw)));
      }
    }
    atomicMax(reinterpret_cast<unsigned*>(ev.amax), __float_as_uint(m));
    return;
  }
  // origin phase e^{i k.o}: formed and reduced in FP64 once per output, so
  // objects far from the frame's origin keep their accuracy.
  const double dox = (double)dh.x + (double)dl.x, doy = (double)dh.y + (double)dl.y,
               doz = (double)dh.z + (double)dl.z;
  const double so_d = dox * od.origin[0] + doy * od.origin[1] + doz * od.origin[2];
  const int64_t Jrow = (int64_t)oi * kg.Q;
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rlo + i;
    if (i >= skip && mine(i)) {
      const int64_t q = (int64_t)r * kg.M + j;
      const double kd = ((double)kw[i].x + (double)kw[i].y) * (6.283185307179586476925 / 64.0);
      cf v = cmul(cis_f64(kd * so_d), cf{acc.sre(i), acc.sim(i)});
      if (kw[i].x * PI_TURN64 * dnorm < 1e-10f) v = cf{0.f, 0.f};  // A(0) = 0 (affine_dof.cpp:64-65)
      if (jm >= 0) {  // the antipode: -conj (the origin phase included)
        const int64_t qm = (int64_t)r * kg.M + jm;
        const float s = scale_sqrt_w ? kg.sqrtw[qm] : 1.0f;
        const float2 u = make_float2(-v.re * s, v.im * s);
        J[Jrow + qm] = u;
        m = fmaxf(m, fmaxf(fabsf(u.x), fabsf(u.y)));
      }
      if (scale_sqrt_w) { const float s = kg.sqrtw[q]; v.re *= s; v.im *= s; }
      J[Jrow + q] = make_float2(v.re, v.im);
      m = fmaxf(m, fmaxf(fabsf(v.re), fabsf(v.im)));
    }
  }
  if (row_amax) {  // the row's largest |Re|, |Im| (FP32 bits order like the non-negative floats)
    const unsigned mask = __activemask();
    const unsigned mb = __reduce_max_sync(mask, __float_as_uint(m));
    if (lane == __ffs(mask) - 1) atomicMax(row_amax + oi, mb);
  }
}

__global__ void to_double2_kernel(const float2* __restrict__ J, int64_t n, double2* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { float2 v = J[i]; out[i] = make_double2(v.x, v.y); }
}

}  // namespace

namespace {

template <int R>
__global__ void __launch_bounds__(FF_THREADS, FF_CTAS)
ff_kernel(KGridDev kg, BatchDev b, float2* __restrict__ J, int scale_sqrt_w, const EvalDev* __restrict__ evals,
          unsigned* __restrict__ row_amax) {
  ff_body<R, false>(kg, b, J, scale_sqrt_w, evals, row_amax);
}

// CTAs per serving evaluation of each class (SERVE_CLASSES).
constexpr int FF_SERVE_SPLIT[SERVE_CLASSES] = {16, 8, 4, 1};

template <int R>
__global__ void __launch_bounds__(FF_THREADS, FF_CTAS)
ff_serve_kernel(KGridDev kg, BatchDev b, const EvalDev* __restrict__ evals, int n_evals) {
  if (n_evals == 0) return;  // a class that the batch has no evaluation of
  ff_body<R, true>(kg, b, nullptr, 1, evals, nullptr);
}

}  // namespace

static int radii_per_thread(int L) { return L >= 32 ? 8 : L >= 4 ? 4 : 2; }  // even: radii are paired
// Serving evaluations: four, since the largest of a batch's few objects sets its
// time (a burst with a fifth of its objects rotated: 12.5 ms at eight, 11.5 at four).
static int serve_radii(int L) { return L >= 4 ? 4 : 2; }

int launch_order(const std::vector<OrderSeg>& segs, int32_t* d_perm, cudaStream_t s) {
  if (segs.empty()) return PI_OK;
  int n_max = 1, n2 = 2;
  for (const OrderSeg& g : segs) n_max = std::max(n_max, (int)g.count);
  while (n2 < n_max) n2 <<= 1;
  int rc = ensure_smem_limit(reinterpret_cast<const void*>(order_kernel), (int)order_smem(ORDER_SEGMENT), "order_kernel");
  if (rc) return rc;
  OrderSeg* d = nullptr;
  PI_CUDA(pool_alloc((void**)&d, segs.size() * sizeof(OrderSeg), s));
  PI_CUDA(cudaMemcpyAsync(d, segs.data(), segs.size() * sizeof(OrderSeg), cudaMemcpyHostToDevice, s));
  order_kernel<<<(unsigned)segs.size(), ORDER_THREADS, order_smem(n2), s>>>(d, d_perm, n2);
  PI_LAUNCHED("order_kernel");
  PI_CUDA(cudaFreeAsync(d, s));
  return PI_OK;
}

int launch_prepare(pi_batch_impl* b, int only_index, cudaStream_t s) {
  std::vector<PrepObj> h(b->n_obj);
  int64_t max_elems = 0;
  for (int i = 0; i < b->n_obj; ++i) {
    const HostObjInfo& in = b->info[i];
    PrepObj& p = h[i];
    p.geom_type = in.geom_type; p.dof_type = in.dof_type; p.n_elems = in.n_elems; p.n_dofs = in.n_dofs;
    p.src = static_cast<const unsigned char*>(b->d_src) + in.src_off;
    p.dofs = b->d_dofs + in.dof_off;
    p.pool_off = in.pool_off;
    p.perm_off = in.perm_off;
    p.cl_off = in.cl_off;
    if (only_index < 0 || only_index == i) max_elems = std::max(max_elems, in.n_elems);
  }
  if (b->n_obj == 0) return PI_OK;
  PrepObj* d = nullptr;
  PI_CUDA(pool_alloc((void**)&d, sizeof(PrepObj) * h.size(), s));
  PI_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(PrepObj) * h.size(), cudaMemcpyHostToDevice, s));
  const int nobj_launch = only_index >= 0 ? 1 : b->n_obj;
  const int S = max_elems > 4 * ORIGIN_THREADS ? ORIGIN_SPLIT : 1;
  void* oargs[4] = {&d, &b->d_objs, &b->d_cl_rho, &only_index};
  if (int rc = launch_split(reinterpret_cast<const void*>(prepare_origin_kernel), dim3((unsigned)(nobj_launch * S)),
                            ORIGIN_THREADS, 0, S, oargs, s))
    return rc;
  PI_LAUNCHED("prepare_origin_kernel");
  if (max_elems > 0) {
    dim3 grid((unsigned)((max_elems + PREP_THREADS - 1) / PREP_THREADS), (unsigned)nobj_launch);
    prepare_elems_kernel<<<grid, PREP_THREADS, 0, s>>>(d, b->d_objs, b->d_tri_pool, b->d_surf_pool, b->d_tri_lo,
                                                       b->d_surf_lo, b->d_surf_nref, b->d_perm, b->d_clusters,
                                                       b->d_leaves, b->d_cl_rho, only_index);
    PI_LAUNCHED("prepare_elems_kernel");
  }
  // The host staging array `h` has been consumed by the copy above once the
  // stream reaches it; cudaMemcpyAsync from pageable memory is synchronous
  // with respect to the host buffer, so it may go out of scope here.
  PI_CUDA(cudaFreeAsync(d, s));
  return PI_OK;
}

int launch_form_factors(const pi_kgrid_impl* kg, const pi_batch_impl* b, int scale_sqrt_w, float2* J,
                        cudaStream_t s, float* row_amax) {
  if (b->n_obj == 0) return PI_OK;
  if (row_amax) PI_CUDA(cudaMemsetAsync(row_amax, 0, (size_t)b->n_obj * sizeof(float), s));
  unsigned* ra = reinterpret_cast<unsigned*>(row_amax);
  const KGridDev K = kg->dev;
  const BatchDev B = b->dev();
  if (b->n_obj > 65535) return fail(PI_ERR_UNSUPPORTED, "more than 65535 objects in one batch");
  int R = radii_per_thread(K.L);
  const int ndt = (K.Me + 31) / 32;
  auto ctas = [&](int r) { return ((int64_t)((K.L + r - 1) / r) * ndt + FF_WARPS - 1) / FF_WARPS; };
  // CTAs that carry the launch: those of the objects of at least a quarter of
  // the largest one's elements, for the fifth of the radii that the cluster
  // expansions usually leave
  const int64_t n_max = b->info[b->order[0]].n_elems;
  int64_t heavy = 0;
  for (int i = 0; i < b->n_obj; ++i) heavy += 4 * b->info[i].n_elems >= n_max;
  auto busy = [&](int r) { return (K.moments ? (ctas(r) + 4) / 5 : ctas(r)) * heavy; };
  const int64_t wave = FF_CTAS * (int64_t)current_sm_count();
  // Four radii per thread where 16 splits at eight give less than 7/4 waves.  Both
  // sides over 14 grids (L = 32 .. 128) and 16 batches: below 0.6 waves four takes 4 to
  // 36% less, above five eight up to 16% less, and between them either may win,
  // triangles and surfels alike: any line from 1 to 4.5 waves loses 1.1 to 1.4% in the
  // mean.  A solid of 200,000 triangles on 5,810 directions,
  // at four and at eight: 17.4 and 19.5 ms at 64 radii (0.97 waves), 23.1 and 24.7 at
  // 112 (1.68), 25.8 and 25.4 at 128 (1.92).
  if (R == 8 && 4 * 16 * busy(8) < 7 * wave) R = 4;
  int S = 1;
  while (S < 16 && S * busy(R) < 2 * wave && n_max > 2 * S * FF_CHUNK) S *= 2;
  const void* fn = R == 8   ? reinterpret_cast<const void*>(ff_kernel<8>)
                   : R == 4 ? reinterpret_cast<const void*>(ff_kernel<4>)
                            : reinterpret_cast<const void*>(ff_kernel<2>);
  const EvalDev* no_evals = nullptr;
  void* args[6] = {const_cast<KGridDev*>(&K), const_cast<BatchDev*>(&B), &J, &scale_sqrt_w, &no_evals, &ra};
  if (int rc = launch_split(fn, dim3((unsigned)(ctas(R) * S), (unsigned)b->n_obj), FF_THREADS, 0, S, args, s)) return rc;
  PI_LAUNCHED("ff_kernel");
  return launch_moments(kg, b, scale_sqrt_w, J, s, row_amax);
}

ServeKernel ff_serve(const pi_kgrid_impl* kg, int cls) {
  const int R = serve_radii(kg->dev.L), S = FF_SERVE_SPLIT[cls];
  const int64_t items = (int64_t)((kg->dev.L + R - 1) / R) * ((kg->dev.Me + 31) / 32);
  return {R == 4 ? reinterpret_cast<const void*>(ff_serve_kernel<4>) : reinterpret_cast<const void*>(ff_serve_kernel<2>),
          (unsigned)((items + FF_WARPS - 1) / FF_WARPS * S), FF_THREADS, S, 0};
}

int ff_serve_setup(const pi_kgrid_impl* kg) { return allow_wide_clusters(ff_serve(kg, 0).fn); }

int launch_form_factors_serve(const pi_kgrid_impl* kg, const pi_batch_impl* lib, const EvalDev* evals,
                              const int (&n_class)[SERVE_CLASSES], cudaStream_t s) {
  KGridDev K = kg->dev;
  BatchDev B = lib->dev();
  int rc = ff_serve_setup(kg);
  if (rc == PI_OK && K.moments) rc = moment_setup();
  for (int c = 0; c < SERVE_CLASSES && rc == PI_OK; evals += n_class[c++]) {
    if (n_class[c] <= 0) continue;
    if (n_class[c] > 65535) return fail(PI_ERR_UNSUPPORTED, "more than 65535 evaluations in one launch");
    int n = n_class[c];
    void* args[4] = {&K, &B, const_cast<EvalDev**>(&evals), &n};
    const ServeKernel k[2] = {ff_serve(kg, c), moment_serve(kg, c)};
    for (int i = 0; i < (K.moments ? 2 : 1) && rc == PI_OK; ++i) {
      rc = launch_split(k[i].fn, dim3(k[i].grid_x, (unsigned)n_class[c]), k[i].threads, k[i].smem, k[i].split, args, s);
      if (rc == PI_OK) count_launch();
    }
  }
  return rc;
}

namespace {
__global__ void amax_commit_kernel(const EvalDev* __restrict__ evals, const int32_t* __restrict__ n_evals) {
  const int n = *n_evals;
  for (int e = threadIdx.x; e < n; e += blockDim.x) *evals[e].amax_keep = *evals[e].amax;
}
}  // namespace

const void* amax_commit_fn() { return reinterpret_cast<const void*>(amax_commit_kernel); }
int amax_commit_threads() { return 256; }

int launch_amax_commit(const EvalDev* evals, const int32_t* n_evals, cudaStream_t s) {
  amax_commit_kernel<<<1, 256, 0, s>>>(evals, n_evals);
  PI_LAUNCHED("amax_commit_kernel");
  return PI_OK;
}

int launch_to_double2(const float2* J, int64_t n, double* out, cudaStream_t s) {
  if (n == 0) return PI_OK;
  to_double2_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(J, n, reinterpret_cast<double2*>(out));
  PI_LAUNCHED("to_double2_kernel");
  return PI_OK;
}

}  // namespace pi
