// evaluate.cu -- upward and downward passes of the KIFMM on the GPU.
//
// Stage map (reference -> here); translation GEMMs: translate.cu, which gathers, scales and scatters the rows:
//   P2M   fmm_scale_invariant.h:163-195 / fmm.h:156-185  k_surf_pot (Laplace mixed: k_surf_pot_lap_f2) check
//                                                        potentials, two tgemm_f64 (pinv factors, scale 0.5^l)
//   M2M   fmm_scale_invariant.h:233-253 / fmm.h:221-241  per level, K = 8 nsurf: tgemm_tc (FP64: tgemm_f64)
//   P2L   fmm_base.h:127-154                             k_surf_pot
//   M2L   fmm_scale_invariant.h:407-440, 560-646;        real kernels, p <= 10: k_m2l_fwd_r + Hadamard + k_m2l_bwd_r
//         fmm.h:395-446, 631-788                         (FP64: k_m2l_bwd); complex kernel, p <= 12: k_m2l_fwd_c +
//                                                        Hadamard + k_m2l_bwd_c; beyond: k_m2l_grid_up + cuFFT +
//                                                        k_transpose(_split) + Hadamard + k_transpose + cuFFT +
//                                                        k_m2l_gather_dn.  Hadamard: k_hadamard_h (opt-in for dense
//                                                        targets: k_hadamard_dc on tcgen05); FP64: k_hadamard_d64
//   L2L   fmm_scale_invariant.h:256-275 / fmm.h:244-263  per level, N = 8 nsurf: tgemm_tc (FP64: tgemm_f64)
//   L2P   fmm_scale_invariant.h:198-230 / fmm.h:188-218  two translation GEMMs (mixed, real kernels: the first
//                                                        tgemm_tc), then the far part of the target evaluation
//   M2P   fmm_base.h:97-124                              far part: k_eval (Laplace: k_far_lap)
//   P2P   fmm_base.h:82-94                               near part: k_near (Laplace mixed: k_near_lap_f2), few
//                                                        leaves: k_near_parts, k_near_lap_f2_parts
// Results stay in tree order until get_values scatters them (python/exafmm.cpp:194-207).
#include <cuda_fp16.h>
#include <cufft.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>
#include <cmath>

#include "kernels.cuh"
#include "tcgen05.cuh"
#include "xfmm_internal.h"

namespace xfmm {

#define XCUFFT2(call)                                                                                \
  do {                                                                                               \
    cufftResult st_ = (call);                                                                        \
    if (st_ != CUFFT_SUCCESS)                                                                        \
      throw Error(XFMM_ERR_CUDA, std::string("cuFFT ") + #call + " failed: " + std::to_string((int)st_)); \
  } while (0)

namespace {

inline int nblk(int64_t n, int t = 256) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }

template <class R> struct R4;
template <> struct R4<float> { using type = float4; };
template <> struct R4<double> { using type = double4; };

template <class Q> __device__ __forceinline__ Q load_charge(const double4& s, const double* qim, int64_t j);
template <> __device__ __forceinline__ float load_charge<float>(const double4& s, const double*, int64_t) {
  return (float)s.w;
}
template <> __device__ __forceinline__ double load_charge<double>(const double4& s, const double*, int64_t) {
  return s.w;
}
template <> __device__ __forceinline__ float2 load_charge<float2>(const double4& s, const double* qim, int64_t j) {
  return make_float2((float)s.w, (float)qim[j]);
}
template <> __device__ __forceinline__ double2 load_charge<double2>(const double4& s, const double* qim, int64_t j) {
  return make_double2(s.w, qim[j]);
}

__device__ __forceinline__ double to64(float v) { return (double)v; }
__device__ __forceinline__ double to64(double v) { return v; }
__device__ __forceinline__ double2 to64(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 to64(double2 v) { return v; }

// FP64 accumulation of FP32/FP64 partials
__device__ __forceinline__ void acc64(double& a, float b) { a += (double)b; }
__device__ __forceinline__ void acc64(double& a, double b) { a += b; }
__device__ __forceinline__ void acc64(double2& a, float2 b) {
  a.x += (double)b.x;
  a.y += (double)b.y;
}
__device__ __forceinline__ void acc64(double2& a, double2 b) {
  a.x += b.x;
  a.y += b.y;
}
template <class Q> struct Acc64 { using type = double; };
template <> struct Acc64<float2> { using type = double2; };
template <> struct Acc64<double2> { using type = double2; };

__device__ __forceinline__ double shfl_x(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double2 shfl_x(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ void put_out(double* o, double v, double s, int acc) { *o = acc ? *o + v * s : v * s; }
__device__ __forceinline__ void put_out(double* o, double2 v, double s, int acc) {
  o[0] = acc ? o[0] + v.x * s : v.x * s;
  o[1] = acc ? o[1] + v.y * s : v.y * s;
}

// ================================================================ far field (M2P + L2P)
struct EvalArgs {
  const int *eval_leafs, *leafs, *ntrgs;
  int n_eval;
  const int64_t* tbeg;
  const double4 *center, *trg4;
  const int64_t* m2p_off;
  const int* m2p;
  const double* surf_base;
  const int* surf_perm;     // surface points in line order (far_surface)
  const double* surf_grid;  // the p grid coordinates of the unit surface
  int nsurf;
  const void* up;  // working values [nnodes][nsurf]
  const void* eq;  // working values [nleafs][nsurf]
  double* out;     // tree order, 4 values per target (complex: interleaved)
  double k_re, k_im;
};

constexpr int EVAL_WARPS = 4;

// Far field (M2P + L2P) of the modified Helmholtz and Helmholtz kernels, in FP64, added to the near field's
// values.  W: value type of the upward equivalent densities (M2P sources); the downward equivalent
// densities (L2P sources) are FP64 (the pinv output).  A leaf by one warp (PARTS 1) or, with few leaves, by
// the CTA's PARTS warps, each taking every PARTS-th chunk of 32 surface points, their sums added in order.
template <int KER, class W, int PARTS>
__global__ void __launch_bounds__(32 * EVAL_WARPS) k_eval(EvalArgs a) {
  // with an FP32 working precision (W), the short form of the FP64 reciprocal square root
  using G = Green<KER, double, std::is_same<typename Base<W>::type, float>::value ? 1 : 2>;
  using Q = typename G::Q;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, part = PARTS > 1 ? wid : 0;
  const int w = PARTS > 1 ? (int)blockIdx.x : blockIdx.x * EVAL_WARPS + wid;
  if (w >= a.n_eval) return;
  __shared__ double4 s_xyz[EVAL_WARPS][32];
  __shared__ Q s_q[EVAL_WARPS][32];
  const G g{a.k_re, a.k_im};
  const int pos = a.eval_leafs[w];
  const int node = a.leafs[pos];
  const int T = a.ntrgs[node], n = a.nsurf;
  const int64_t tb = a.tbeg[node];
  const double4 c = a.center[node];
  const W* upv = (const W*)a.up;
  const Q* eqv = (const Q*)a.eq;
  for (int t0 = 0, Tc = 0; t0 < T; t0 += Tc) {
    // blocks of 32 targets, the last 17..32 as 16 + the rest, so that the split of the sources over
    // 2..32 lanes per target keeps the lanes busy
    Tc = T - t0 > 32 ? 32 : (T - t0 > 16 ? 16 : T - t0);
    int G2 = 1;  // lanes per target: source stride
    while (G2 * 2 * Tc <= 32) G2 *= 2;
    const int tl = lane / G2, sub = lane % G2;
    const bool active = tl < Tc;
    double tx = 0, ty = 0, tz = 0;
    if (active) {
      const double4 t = a.trg4[tb + t0 + tl];
      tx = t.x - c.x;
      ty = t.y - c.y;
      tz = t.z - c.z;
    }
    Q P = vzero<Q>(), GX = vzero<Q>(), GY = vzero<Q>(), GZ = vzero<Q>();
    int chunk = 0;
    // one surface of half size b at offset (ox, oy, oz) from the leaf's centre: den(k) its densities
    auto surface = [&](double ox, double oy, double oz, double b, auto&& den) {
      for (int j0 = 0; j0 < n; j0 += 32) {
        if (PARTS > 1 && (chunk++) % PARTS != part) continue;
        const int cnt = min(32, n - j0), k = j0 + lane;
        __syncwarp();
        if (lane < cnt) {
          s_xyz[wid][lane] = make_double4(ox + a.surf_base[3 * k] * b, oy + a.surf_base[3 * k + 1] * b,
                                          oz + a.surf_base[3 * k + 2] * b, 0.0);
          s_q[wid][lane] = den(k);
        }
        __syncwarp();
        if (!active) continue;
        Q p = vzero<Q>(), gx = vzero<Q>(), gy = vzero<Q>(), gz = vzero<Q>();  // the chunk's sums
        for (int j = sub; j < cnt; j += G2) {
          const double4 s = s_xyz[wid][j];
          g.grad(tx - s.x, ty - s.y, tz - s.z, s_q[wid][j], p, gx, gy, gz);
        }
        P = vadd(P, p);
        GX = vadd(GX, gx);
        GY = vadd(GY, gy);
        GZ = vadd(GZ, gz);
      }
    };
    // M2P: W-list nodes' upward equivalent surfaces (1.05 box, fmm_base.h:103-121)
    for (int64_t e = a.m2p_off[node]; e < a.m2p_off[node + 1]; e++) {
      const int s = a.m2p[e];
      const double4 cs = a.center[s];
      surface(cs.x - c.x, cs.y - c.y, cs.z - c.z, 1.05 * cs.w, [&](int k) { return to64(upv[(int64_t)s * n + k]); });
    }
    // L2P: own downward equivalent surface (2.95 box, fmm_scale_invariant.h:221-228)
    surface(0.0, 0.0, 0.0, 2.95 * c.w, [&](int k) { return eqv[(int64_t)pos * n + k]; });
    for (int o = 1; o < G2; o <<= 1) {
      P = vadd(P, shfl_x(P, o));
      GX = vadd(GX, shfl_x(GX, o));
      GY = vadd(GY, shfl_x(GY, o));
      GZ = vadd(GZ, shfl_x(GZ, o));
    }
    if constexpr (PARTS > 1) {
      __shared__ Q red[PARTS - 1][4][32];
      if (part > 0) {
        red[part - 1][0][lane] = P;
        red[part - 1][1][lane] = GX;
        red[part - 1][2][lane] = GY;
        red[part - 1][3][lane] = GZ;
      }
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int k = 0; k < PARTS - 1; k++) {
          P = vadd(P, red[k][0][lane]);
          GX = vadd(GX, red[k][1][lane]);
          GY = vadd(GY, red[k][2][lane]);
          GZ = vadd(GZ, red[k][3][lane]);
        }
      }
      __syncthreads();
    }
    if (active && sub == 0 && part == 0) {
      const int stride = (KER == K_HELMHOLTZ) ? 8 : 4;
      double* o = a.out + (tb + t0 + tl) * stride;
      const int vs = stride / 4;
      put_out(o, P, INV4PI, 1);
      put_out(o + vs, GX, INV4PI, 1);
      put_out(o + 2 * vs, GY, INV4PI, 1);
      put_out(o + 3 * vs, GZ, INV4PI, 1);
    }
  }
}

// Far field (M2P + L2P) of the Laplace kernel, in FP64 in both precisions: the sums over equivalent densities
// cancel strongly, so every term needs FP64.  Targets map to lanes as in k_eval.  The points of an equivalent
// surface (each W-list node's upward surface, then the leaf's own downward surface) form a p^3 grid's faces,
// and are taken line by line along one axis: 4 p - 4 lines of p points along x (the z faces, then the y
// faces without the z faces' rows), then 2 (p - 2) lines of p - 2 points along y (the x faces' interior).
// On a line the two fixed coordinates' squared distance A is one value, the running coordinate's distances
// and squares are kept in registers for the whole surface, and the gradient along the fixed axes needs only
// the line's sum: per point one add (r^2 = A + d^2), the reciprocal square root and 7 more FP64
// operations, 10 + 6 / p against 17 when every point's separation is formed anew.  The FP64 pipe (2 cycles
// per operation and warp) bounds it: at 4M, p = 8 (1.18e9 pairs) 1.54 -> 1.07 ms;
// FP64 path at 1M 0.70 -> 0.34 (two Newton steps on the instruction, where FP32 gave the seed).
// 1/r: the FP64 reciprocal-square-root approximation instruction (rsqrt_approx64) and NS Newton steps
// y <- y (3 - r^2 y^2) / 2 (1: 2^-39.5, for FP32 densities; 2: full FP64), the powers of two carried in the
// staged densities.  No pair coincides: a target lies at least 1.95 r from its own downward
// surface, and W-list nodes are not adjacent to the leaf.
// Few leaves would leave the chip idle behind the longest of them: FAR_PARTS warps then share a leaf, each
// taking every FAR_PARTS-th line, and their sums meet in shared memory in a fixed order.
template <int NS> struct FarScale;  // yh = KY / r after NS scaled Newton steps
template <> struct FarScale<1> { static constexpr double KY = 2.0; };
template <> struct FarScale<2> { static constexpr double KY = 16.0; };
// q / r -> p and, along a line, q / r^3 -> s (scaled by KY^2) of one point at squared distance r2; q staged as q / KY
template <int NS>
__device__ __forceinline__ double far_point(double r2, double q, double& p) {
  double y = rsqrt_approx64(r2);
  y = y * fma(-r2, y * y, 3.0);
  if constexpr (NS == 2) y = y * fma(-r2, y * y, 12.0);
  const double qi = q * y;
  p += qi;
  return qi * (y * y);
}
// one surface, lines l0, l0 + lstep, ...: den[] the densities in line order, g[] the P grid coordinates in [-1, 1],
// b the half size, u the target relative to the surface's centre; the gradient sums are scaled by KY^2
template <int P, int NS>
__device__ __forceinline__ void far_surface(const double* den, const double* g, double b, double ux, double uy,
                                            double uz, int l0, int lstep, double& p, double& gx, double& gy,
                                            double& gz) {
  double d[P], d2[P];
#pragma unroll
  for (int i = 0; i < P; i++) {
    d[i] = fma(-b, g[i], ux);
    d2[i] = d[i] * d[i];
  }
  int m = l0;
  for (; m < 4 * P - 4; m += lstep) {
    int j, l;
    if (m < 2 * P) {
      l = m < P ? 0 : P - 1;
      j = m < P ? m : m - P;
    } else {
      const int mm = m - 2 * P;
      j = mm < P - 2 ? 0 : P - 1;
      l = 1 + (mm < P - 2 ? mm : mm - (P - 2));
    }
    const double dy = fma(-b, g[j], uy), dz = fma(-b, g[l], uz), A = fma(dz, dz, dy * dy);
    const double* q = den + m * P;
    double s = 0;
#pragma unroll
    for (int i = 0; i < P; i++) {
      const double w = far_point<NS>(A + d2[i], q[i], p);
      gx = fma(-w, d[i], gx);
      s += w;
    }
    gy = fma(-s, dy, gy);
    gz = fma(-s, dz, gz);
  }
  if constexpr (P > 2) {
#pragma unroll
    for (int i = 0; i < P; i++) {
      d[i] = fma(-b, g[i], uy);
      d2[i] = d[i] * d[i];
    }
    const double* q0 = den + (4 * P - 4) * P;
    for (m -= 4 * P - 4; m < 2 * (P - 2); m += lstep) {
      const int i = m < P - 2 ? 0 : P - 1, l = 1 + (m < P - 2 ? m : m - (P - 2));
      const double dx = fma(-b, g[i], ux), dz = fma(-b, g[l], uz), A = fma(dz, dz, dx * dx);
      const double* q = q0 + m * (P - 2);
      double s = 0;
#pragma unroll
      for (int j = 1; j < P - 1; j++) {
        const double w = far_point<NS>(A + d2[j], q[j - 1], p);
        gy = fma(-w, d[j], gy);
        s += w;
      }
      gx = fma(-s, dx, gx);
      gz = fma(-s, dz, gz);
    }
  }
}
constexpr int FAR_PARTS = 4;
// dynamic shared memory of one warp: the surface's densities; and of the CTA: the grid coordinates
inline size_t far_smem(int nsurf, int p) { return sizeof(double) * ((size_t)EVAL_WARPS * nsurf + p); }
// the far field of evaluation leaf w: by one warp (PARTS 1) or as part `part` of FAR_PARTS warps of the CTA
template <class W, int P, int PARTS>
__device__ __forceinline__ void far_leaf_lap(const EvalArgs& a, int w, int lane, int part, double* den, const double* g) {
  constexpr int NS = std::is_same<W, float>::value ? 1 : 2;
  constexpr double KY = FarScale<NS>::KY;
  const int pos = a.eval_leafs[w];
  const int node = a.leafs[pos];
  const int T = a.ntrgs[node];
  const int64_t tb = a.tbeg[node];
  const double4 c = a.center[node];
  const int n = a.nsurf;
  const W* upv = (const W*)a.up;
  const double* eqv = (const double*)a.eq;
  for (int t0 = 0, Tc = 0; t0 < T; t0 += Tc) {
    // blocks of 32 targets, the last 17..32 as 16 + the rest; 2..32 lanes per target split the lines
    Tc = T - t0 > 32 ? 32 : (T - t0 > 16 ? 16 : T - t0);
    int G2 = 1;
    while (G2 * 2 * Tc <= 32) G2 *= 2;
    const int tl = lane / G2, sub = lane % G2;
    const bool active = tl < Tc;
    double tx = 0, ty = 0, tz = 0;
    if (active) {
      const double4 t = a.trg4[tb + t0 + tl];
      tx = t.x - c.x;
      ty = t.y - c.y;
      tz = t.z - c.z;
    }
    double p = 0, gx = 0, gy = 0, gz = 0;
    // M2P: W-list nodes' upward equivalent surfaces (1.05 box, fmm_base.h:103-121)
    for (int64_t e = a.m2p_off[node]; e < a.m2p_off[node + 1]; e++) {
      const int s = a.m2p[e];
      const double4 cs = a.center[s];
      __syncwarp();
      for (int i = lane; i < n; i += 32) den[i] = (1.0 / KY) * (double)upv[(int64_t)s * n + a.surf_perm[i]];
      __syncwarp();
      if (active)
        far_surface<P, NS>(den, g, 1.05 * cs.w, tx - (cs.x - c.x), ty - (cs.y - c.y), tz - (cs.z - c.z),
                           sub * PARTS + part, G2 * PARTS, p, gx, gy, gz);
    }
    // L2P: own downward equivalent surface (2.95 box, fmm_scale_invariant.h:221-228)
    __syncwarp();
    for (int i = lane; i < n; i += 32) den[i] = (1.0 / KY) * eqv[(int64_t)pos * n + a.surf_perm[i]];
    __syncwarp();
    if (active)
      far_surface<P, NS>(den, g, 2.95 * c.w, tx, ty, tz, sub * PARTS + part, G2 * PARTS, p, gx, gy, gz);
    for (int o = 1; o < G2; o <<= 1) {
      p += __shfl_xor_sync(0xffffffffu, p, o);
      gx += __shfl_xor_sync(0xffffffffu, gx, o);
      gy += __shfl_xor_sync(0xffffffffu, gy, o);
      gz += __shfl_xor_sync(0xffffffffu, gz, o);
    }
    if constexpr (PARTS > 1) {
      __shared__ double red[PARTS - 1][4][32];
      if (part > 0) {
        red[part - 1][0][lane] = p;
        red[part - 1][1][lane] = gx;
        red[part - 1][2][lane] = gy;
        red[part - 1][3][lane] = gz;
      }
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int k = 0; k < PARTS - 1; k++) {
          p += red[k][0][lane];
          gx += red[k][1][lane];
          gy += red[k][2][lane];
          gz += red[k][3][lane];
        }
      }
      __syncthreads();
    }
    if (active && sub == 0 && part == 0) {
      double* o = a.out + (tb + t0 + tl) * 4;
      o[0] += p * INV4PI;
      o[1] += gx * (INV4PI / (KY * KY));
      o[2] += gy * (INV4PI / (KY * KY));
      o[3] += gz * (INV4PI / (KY * KY));
    }
  }
}
template <class W, int P, int PARTS>
__global__ void __launch_bounds__(32 * EVAL_WARPS) k_far_lap(EvalArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* g = sm + EVAL_WARPS * a.nsurf;
  if (threadIdx.x < P) g[threadIdx.x] = a.surf_grid[threadIdx.x];
  __syncthreads();
  const int w = PARTS > 1 ? (int)blockIdx.x : blockIdx.x * EVAL_WARPS + wid;
  if (w >= a.n_eval) return;
  far_leaf_lap<W, P, PARTS>(a, w, lane, PARTS > 1 ? wid : 0, sm + wid * a.nsurf, g);
}
// The far field of every system of a batch: each warp takes work items (system, evaluation leaf) from one
// queue (a global counter, zeroed before the launch) in the order of `items` until it runs dry.
template <class W, int P>
__global__ void __launch_bounds__(32 * EVAL_WARPS)
    k_far_lap_queue(const EvalArgs* __restrict__ args, const int2* __restrict__ items, int64_t nitems,
                    unsigned int* __restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nsurf = args[0].nsurf;
  double* g = sm + EVAL_WARPS * nsurf;
  if (threadIdx.x < P) g[threadIdx.x] = args[0].surf_grid[threadIdx.x];
  __syncthreads();
  for (;;) {
    unsigned int k = 0;
    if (lane == 0) k = atomicAdd(counter, 1u);
    k = __shfl_sync(0xffffffffu, k, 0);
    if ((int64_t)k >= nitems) break;
    const int2 it = items[k];
    far_leaf_lap<W, P, 1>(args[it.x], it.y, lane, 0, sm + wid * nsurf, g);
    __syncwarp();
  }
}
// calls fn(std::integral_constant<int, p>) for the supported orders
template <class F>
void order_dispatch(int p, F&& fn) {
  switch (p) {
    case 2: fn(std::integral_constant<int, 2>()); break;
    case 3: fn(std::integral_constant<int, 3>()); break;
    case 4: fn(std::integral_constant<int, 4>()); break;
    case 5: fn(std::integral_constant<int, 5>()); break;
    case 6: fn(std::integral_constant<int, 6>()); break;
    case 7: fn(std::integral_constant<int, 7>()); break;
    case 8: fn(std::integral_constant<int, 8>()); break;
    case 9: fn(std::integral_constant<int, 9>()); break;
    case 10: fn(std::integral_constant<int, 10>()); break;
    case 11: fn(std::integral_constant<int, 11>()); break;
    case 12: fn(std::integral_constant<int, 12>()); break;
    case 13: fn(std::integral_constant<int, 13>()); break;
    case 14: fn(std::integral_constant<int, 14>()); break;
    case 15: fn(std::integral_constant<int, 15>()); break;
    case 16: fn(std::integral_constant<int, 16>()); break;
    default: throw Error(XFMM_ERR_UNSUPPORTED, "expansion order p must be in [2, 16]");
  }
}
// Leaves below which several warps share one (FAR_PARTS, NEAR_PARTS, the surfaces of P2M and P2L): 64 per SM, two
// to three times the warps resident at once.  Near field: 1.5k leaves (Plummer 20k, FP64) 0.49 -> 0.15 ms, 8.4k
// (Plummer 300k, mixed) 0.62 -> 0.29, 4.6k even leaves (Helmholtz 200k) 0.77 -> 0.70, 4.1k even leaves
// (Laplace 100k, FP64) 0.21 -> 0.20: the gain is gone where every SM has several rounds of leaves.
constexpr int SPLIT_LEAVES = 148 * 64;

// ================================================================ near field (P2P)
// Warp per target leaf.  The sources of the leaf's P2P list form one continuous stream that is
// staged 32 at a time in shared memory as leaf-relative coordinates (FP32: hi + lo parts, so the
// separation keeps FP32 relative accuracy); only the stream's last chunk is padded (zero charges,
// far away).  Lanes map to targets in one of two ways:
//   T >= 32 : TPL targets per lane (t = lane + 32 u), every staged source reused TPL times;
//   T <  32 : G lanes per target (G = 32 / 2^ceil(log2 T)), each taking every G-th source of a
//             chunk, partial sums combined with shuffles at the end.
// FP32 chunk sums are accumulated in FP64.
// A system of few leaves would leave the chip idle behind its longest leaves: NEAR_PARTS warps then share a
// leaf, part k taking every NEAR_PARTS-th chunk from the k-th, and the parts' FP64 sums are added in order.
// How many parts a leaf has is fixed by its system's leaf count (NearArgs::parts), and a kernel that has
// one warp per leaf takes the parts one after another, so the results do not depend on the kernel.
constexpr int NEAR_PARTS = 4;
struct NearArgs {
  const int *eval_leafs, *leafs, *nsrcs, *ntrgs;
  int n_eval;
  const int64_t *sbeg, *tbeg, *p2p_off;
  const int* p2p;
  const double4 *center, *src4, *trg4;
  const double* src_qim;
  double* out;
  double k_re, k_im;
  int parts;  // 1 or NEAR_PARTS
};

template <class R> struct Stage4;
template <> struct Stage4<float> { using type = float4; };
template <> struct Stage4<double> { using type = double4; };

constexpr int NEAR_SEG = 64;  // P2P-list entries held per batch

template <class R>
struct NearSmem {
  typename Stage4<R>::type hi[32], lo[32];
  int64_t seg_beg[NEAR_SEG];
  int seg_pre[NEAR_SEG + 1];
};

// PARTS 0: the whole leaf in one pass (systems of one part); 1: its parts one after another (a.parts; the sums kept
// beside the running ones cost registers: Yukawa sphere 300k 0.305 -> 0.340 ms); NEAR_PARTS: part `part` of a
// leaf shared by the warps of the CTA, all of which call this
template <int KER, class R, int TPL, int PARTS = 1>
__device__ __forceinline__ void near_leaf(const NearArgs& a, int node, int lane, NearSmem<R>& sm, int part = 0) {
  using G = Green<KER, R>;
  using Q = typename G::Q;
  using A = typename Acc64<Q>::type;
  constexpr bool CPLX = KER == K_HELMHOLTZ;
  constexpr bool HILO = sizeof(R) == 4;
  const G g{(R)a.k_re, (R)a.k_im};
  const int T = a.ntrgs[node];
  const int64_t tb = a.tbeg[node];
  const double4 c = a.center[node];
  const int64_t e0 = a.p2p_off[node], e1 = a.p2p_off[node + 1];
  // lane -> (target slot, source sub-lane)
  int G2 = 1;
  if (TPL == 1)
    while (G2 * 2 * T <= 32) G2 *= 2;
  const int tl = lane / G2, sub = lane % G2;
  const int nper = 32 / G2;  // sources per lane per chunk
  for (int t0 = 0; t0 < T; t0 += 32 * TPL) {
    R tx[TPL], ty[TPL], tz[TPL], lx[TPL], ly[TPL], lz[TPL];
    A P[TPL], GX[TPL], GY[TPL], GZ[TPL];
    const int np = PARTS == 1 ? a.parts : PARTS > 1 ? PARTS : 1, k0 = PARTS > 1 ? part : 0, k1 = PARTS > 1 ? part + 1 : np;
    A SP[TPL], SX[TPL], SY[TPL], SZ[TPL];  // sums of the parts before
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      const int t = t0 + tl + 32 * u;
      double dx = 0, dy = 0, dz = 0;
      if (t < T) {
        const double4 v = a.trg4[tb + t];
        dx = v.x - c.x;
        dy = v.y - c.y;
        dz = v.z - c.z;
      }
      tx[u] = (R)dx;
      ty[u] = (R)dy;
      tz[u] = (R)dz;
      lx[u] = (R)(dx - (double)tx[u]);
      ly[u] = (R)(dy - (double)ty[u]);
      lz[u] = (R)(dz - (double)tz[u]);
    }
    for (int k = k0; k < k1; k++) {
#pragma unroll
    for (int u = 0; u < TPL; u++) P[u] = GX[u] = GY[u] = GZ[u] = A();
    for (int64_t eb = e0; eb < e1; eb += NEAR_SEG) {
      // segment table of this batch: begin offsets and an inclusive prefix of counts
      const int nseg = (int)(e1 - eb < NEAR_SEG ? e1 - eb : NEAR_SEG);
      __syncwarp();
      int carry = 0;
      for (int q0 = 0; q0 < nseg; q0 += 32) {
        const int q = q0 + lane;
        int cnt = 0;
        if (q < nseg) {
          const int sn = a.p2p[eb + q];
          cnt = a.nsrcs[sn];
          sm.seg_beg[q] = a.sbeg[sn];
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (q < nseg) sm.seg_pre[q + 1] = carry + incl;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) sm.seg_pre[0] = 0;
      __syncwarp();
      const int total = carry;
      int seg = 0;  // per-lane cursor into the segment table
      for (int p0 = 32 * k; p0 < total; p0 += 32 * np) {
        const int pos = p0 + lane;
        __syncwarp();
        if (pos < total) {
          while (sm.seg_pre[seg + 1] <= pos) seg++;
          const int64_t si = sm.seg_beg[seg] + (pos - sm.seg_pre[seg]);
          const double4 sv = a.src4[si];
          const double dx = sv.x - c.x, dy = sv.y - c.y, dz = sv.z - c.z;
          const R hx = (R)dx, hy = (R)dy, hz = (R)dz;
          const R qi = CPLX ? (R)a.src_qim[si] : (R)0;
          sm.hi[lane] = {hx, hy, hz, (R)sv.w};
          if constexpr (HILO || CPLX)
            sm.lo[lane] = {(R)(dx - (double)hx), (R)(dy - (double)hy), (R)(dz - (double)hz), qi};
        } else {
          sm.hi[lane] = {(R)1e3, (R)1e3, (R)1e3, (R)0};  // zero-charge padding, far from every target
          if constexpr (HILO || CPLX) sm.lo[lane] = {(R)0, (R)0, (R)0, (R)0};
        }
        __syncwarp();
        Q p[TPL], gx[TPL], gy[TPL], gz[TPL];
#pragma unroll
        for (int u = 0; u < TPL; u++) p[u] = gx[u] = gy[u] = gz[u] = vzero<Q>();
#pragma unroll 4
        for (int jj = 0; jj < nper; jj++) {
          const int j = jj * G2 + sub;
          const auto h = sm.hi[j];
          typename Stage4<R>::type l{};  // low parts (FP32) and imaginary charges (complex); FP64 real: none
          if constexpr (HILO || CPLX) l = sm.lo[j];
          Q q;
          if constexpr (CPLX) q = Q{h.w, l.w};
          else q = h.w;
#pragma unroll
          for (int u = 0; u < TPL; u++) {
            R dx, dy, dz;
            if constexpr (HILO) {
              dx = (tx[u] - h.x) + (lx[u] - l.x);
              dy = (ty[u] - h.y) + (ly[u] - l.y);
              dz = (tz[u] - h.z) + (lz[u] - l.z);
            } else {
              dx = tx[u] - h.x;
              dy = ty[u] - h.y;
              dz = tz[u] - h.z;
            }
            g.grad(dx, dy, dz, q, p[u], gx[u], gy[u], gz[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < TPL; u++) {
          acc64(P[u], p[u]);
          acc64(GX[u], gx[u]);
          acc64(GY[u], gy[u]);
          acc64(GZ[u], gz[u]);
        }
      }
    }
    if (PARTS == 1 && np > 1) {
#pragma unroll
      for (int u = 0; u < TPL; u++) {
        if (k > k0) {
          P[u] = vadd(SP[u], P[u]);
          GX[u] = vadd(SX[u], GX[u]);
          GY[u] = vadd(SY[u], GY[u]);
          GZ[u] = vadd(SZ[u], GZ[u]);
        }
        SP[u] = P[u];
        SX[u] = GX[u];
        SY[u] = GY[u];
        SZ[u] = GZ[u];
      }
    }
    }
    if constexpr (PARTS > 1) {
      __shared__ A red[PARTS - 1][4 * TPL][32];
      if (part > 0) {
#pragma unroll
        for (int u = 0; u < TPL; u++) {
          red[part - 1][4 * u][lane] = P[u];
          red[part - 1][4 * u + 1][lane] = GX[u];
          red[part - 1][4 * u + 2][lane] = GY[u];
          red[part - 1][4 * u + 3][lane] = GZ[u];
        }
      }
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int q = 0; q < PARTS - 1; q++)
#pragma unroll
          for (int u = 0; u < TPL; u++) {
            P[u] = vadd(P[u], red[q][4 * u][lane]);
            GX[u] = vadd(GX[u], red[q][4 * u + 1][lane]);
            GY[u] = vadd(GY[u], red[q][4 * u + 2][lane]);
            GZ[u] = vadd(GZ[u], red[q][4 * u + 3][lane]);
          }
      }
      __syncthreads();
      if (part > 0) continue;  // the next block of targets
    }
    if (TPL == 1) {
      for (int o = 1; o < G2; o <<= 1) {
        P[0] = vadd(P[0], shfl_x(P[0], o));
        GX[0] = vadd(GX[0], shfl_x(GX[0], o));
        GY[0] = vadd(GY[0], shfl_x(GY[0], o));
        GZ[0] = vadd(GZ[0], shfl_x(GZ[0], o));
      }
    }
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      const int t = t0 + tl + 32 * u;
      if (t < T && sub == 0) {
        const int stride = CPLX ? 8 : 4, vs = stride / 4;
        double* o = a.out + (tb + t) * stride;
        put_out(o, P[u], INV4PI, 0);
        put_out(o + vs, GX[u], INV4PI, 0);
        put_out(o + 2 * vs, GY[u], INV4PI, 0);
        put_out(o + 3 * vs, GZ[u], INV4PI, 0);
      }
    }
  }
}

// ---------------------------------------------------------------- Laplace FP32 near field, paired FP32
// Same mapping and streaming as near_leaf, but two sources are processed per instruction with the
// sm_100 paired FP32 operations (__ffma2_rn / __fadd2_rn / __fmul2_rn): the staged sources are laid
// out structure-of-arrays so that sources (j, j+1) load as one float2, and the target's coordinates
// are duplicated into both halves once per chunk.
// Coordinates are taken relative to the centre of the target leaf: each staged source is moved there in
// FP64 and rounded to FP32 once per chunk (shared by every target of the warp), each target once, so a
// pair's separation is a single FP32 subtraction of two values no larger than the 3 x 3 x 3 leaf
// neighbourhood (a few leaf radii).  Its error is a few FP32 ulps of that neighbourhood's size, not of
// the root's.  That is not enough for the closest pairs (the few pairs a few 1e-5 apart dominate the
// gradient's norm over all targets), so 1/r is taken of max(r^2, d^2), d = NEAR_CLOSE x the leaf
// radius: a pair closer than d (r == 0 among them) contributes a bounded FP32 value.  Those pairs are
// found once per tree with the same FP32 arithmetic (k_close_scan) and, after the near field, k_close_fix
// replaces each one's FP32 contribution with the exact FP64 one (pairs at r == 0 in FP64 contribute
// nothing, laplace.h:57).  The error left in the FP32 pairs, ~2^-24 x (neighbourhood radius /
// separation), is then bounded by separations above d.
constexpr float NEAR_CLOSE = 0.125f;
// the squared close-pair distance of a leaf of radius r (the same FP32 value in every kernel that tests it)
__device__ __forceinline__ float near_close2(double r) {
  const float d = (float)(NEAR_CLOSE * r);
  return d * d;
}
// a source or target relative to the leaf centre, rounded to FP32 (the same in every kernel)
__device__ __forceinline__ float3 leaf_rel(const double4& v, const double4& cn) {
  return make_float3((float)(v.x - cn.x), (float)(v.y - cn.y), (float)(v.z - cn.z));
}
#ifndef XFMM_NEAR_CH
#define XFMM_NEAR_CH 64
#endif
constexpr int NEAR_CH = XFMM_NEAR_CH;  // sources staged per chunk (32 or 64)
static_assert(NEAR_CH == 32 || NEAR_CH == 64, "NEAR_CH");
struct NearSmemF2 {
  // source pair k = sources 2k, 2k+1 relative to the leaf centre: {x, x'}, {y, y'} and {z, z'}, {q, q'}
  float4 pr[NEAR_CH / 2][2];
  int64_t seg_beg[NEAR_SEG];
  int seg_pre[NEAR_SEG + 1];
};

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }

template <int TPL, int PARTS = 1>  // PARTS as in near_leaf (PARTS 1: the whole leaf in one pass)
__device__ __forceinline__ void near_leaf_lap_f2(const NearArgs& a, int node, int lane, NearSmemF2& sm, int part = 0) {
  const int T = a.ntrgs[node];
  const int64_t tb = a.tbeg[node];
  const int64_t e0 = a.p2p_off[node], e1 = a.p2p_off[node + 1];
  const double4 cn = a.center[node];
  int G2 = 1;  // at most 16 lanes per target
  if (TPL == 1)
    while (G2 * 2 * T <= 32 && G2 < 16) G2 *= 2;
  const int tl = lane / G2, sub = lane % G2;
  const int npl = NEAR_CH / 2 / G2;  // source pairs per lane per chunk
  const float2 M1 = make_float2(-1.f, -1.f);
  const float dc2 = near_close2(cn.w);  // close-pair threshold, squared
  for (int t0 = 0; t0 < T; t0 += 32 * TPL) {
    float2 TX[TPL], TY[TPL], TZ[TPL];
    double P[TPL], GX[TPL], GY[TPL], GZ[TPL];
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      const int t = t0 + tl + 32 * u;
      float3 tr = make_float3(0.f, 0.f, 0.f);
      if (t < T) tr = leaf_rel(a.trg4[tb + t], cn);
      TX[u] = dup2(tr.x);
      TY[u] = dup2(tr.y);
      TZ[u] = dup2(tr.z);
      P[u] = GX[u] = GY[u] = GZ[u] = 0.0;
    }
    for (int64_t eb = e0; eb < e1; eb += NEAR_SEG) {
      const int nseg = (int)(e1 - eb < NEAR_SEG ? e1 - eb : NEAR_SEG);
      __syncwarp();
      int carry = 0;
      for (int k0 = 0; k0 < nseg; k0 += 32) {
        const int k = k0 + lane;
        int cnt = 0, sn = -1;
        if (k < nseg) {
          sn = a.p2p[eb + k];
          cnt = a.nsrcs[sn];
          sm.seg_beg[k] = a.sbeg[sn];
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (k < nseg) sm.seg_pre[k + 1] = carry + incl;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) sm.seg_pre[0] = 0;
      __syncwarp();
      const int total = carry;
      int seg = 0;
      for (int p0 = NEAR_CH * part; p0 < total; p0 += NEAR_CH * PARTS) {
        __syncwarp();
#pragma unroll
        for (int h = 0; h < NEAR_CH / 32; h++) {
          const int pos = p0 + 32 * h + lane;
          // zero-charge padding far away: contributes 0 and is never close
          float x = 1e18f, y = 1e18f, z = 1e18f, q = 0.f;
          if (pos < total) {
            while (sm.seg_pre[seg + 1] <= pos) seg++;
            const double4 v = a.src4[sm.seg_beg[seg] + (pos - sm.seg_pre[seg])];
            const float3 sr = leaf_rel(v, cn);
            x = sr.x;
            y = sr.y;
            z = sr.z;
            q = (float)v.w;
          }
          float* r = reinterpret_cast<float*>(sm.pr[16 * h + (lane >> 1)]) + (lane & 1);  // float2 slot
          r[0] = x;
          r[2] = y;
          r[4] = z;
          r[6] = q;
        }
        __syncwarp();
        float2 p2[TPL], gx2[TPL], gy2[TPL], gz2[TPL];
#pragma unroll
        for (int u = 0; u < TPL; u++) p2[u] = gx2[u] = gy2[u] = gz2[u] = make_float2(0.f, 0.f);
        // pairs closer than the threshold (r == 0 among them) give 1/max(r, d): replaced exactly later
#pragma unroll 4
        for (int jj = 0; jj < npl; jj++) {
          const int jp = jj * G2 + sub;  // source pair
          const float4 A0 = sm.pr[jp][0], A1 = sm.pr[jp][1];
          const float2 SX = make_float2(A0.x, A0.y), SY = make_float2(A0.z, A0.w);
          const float2 SZ = make_float2(A1.x, A1.y), Q = make_float2(A1.z, A1.w);
#pragma unroll
          for (int u = 0; u < TPL; u++) {
            const float2 dx = __ffma2_rn(SX, M1, TX[u]);  // t - s
            const float2 dy = __ffma2_rn(SY, M1, TY[u]);
            const float2 dz = __ffma2_rn(SZ, M1, TZ[u]);
            float2 r2 = __fmul2_rn(dx, dx);
            r2 = __ffma2_rn(dy, dy, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            const float2 inv = make_float2(rsqrtf(fmaxf(r2.x, dc2)), rsqrtf(fmaxf(r2.y, dc2)));
            const float2 qi = __fmul2_rn(Q, inv);
            const float2 qi3 = __fmul2_rn(qi, __fmul2_rn(inv, inv));
            p2[u] = __fadd2_rn(p2[u], qi);
            gx2[u] = __ffma2_rn(qi3, dx, gx2[u]);  // sign applied when accumulating
            gy2[u] = __ffma2_rn(qi3, dy, gy2[u]);
            gz2[u] = __ffma2_rn(qi3, dz, gz2[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < TPL; u++) {
          P[u] += (double)(p2[u].x + p2[u].y);
          GX[u] -= (double)(gx2[u].x + gx2[u].y);
          GY[u] -= (double)(gy2[u].x + gy2[u].y);
          GZ[u] -= (double)(gz2[u].x + gz2[u].y);
        }
      }
    }
    if constexpr (PARTS > 1) {
      __shared__ double red[PARTS - 1][4 * TPL][32];
      if (part > 0) {
#pragma unroll
        for (int u = 0; u < TPL; u++) {
          red[part - 1][4 * u][lane] = P[u];
          red[part - 1][4 * u + 1][lane] = GX[u];
          red[part - 1][4 * u + 2][lane] = GY[u];
          red[part - 1][4 * u + 3][lane] = GZ[u];
        }
      }
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int q = 0; q < PARTS - 1; q++)
#pragma unroll
          for (int u = 0; u < TPL; u++) {
            P[u] += red[q][4 * u][lane];
            GX[u] += red[q][4 * u + 1][lane];
            GY[u] += red[q][4 * u + 2][lane];
            GZ[u] += red[q][4 * u + 3][lane];
          }
      }
      __syncthreads();
      if (part > 0) continue;  // the next block of targets
    }
    if (TPL == 1) {
      for (int o = 1; o < G2; o <<= 1) {
        P[0] += __shfl_xor_sync(0xffffffffu, P[0], o);
        GX[0] += __shfl_xor_sync(0xffffffffu, GX[0], o);
        GY[0] += __shfl_xor_sync(0xffffffffu, GY[0], o);
        GZ[0] += __shfl_xor_sync(0xffffffffu, GZ[0], o);
      }
    }
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      const int t = t0 + tl + 32 * u;
      if (t < T && sub == 0) {
        double* o = a.out + (tb + t) * 4;
        o[0] = P[u] * INV4PI;
        o[1] = GX[u] * INV4PI;
        o[2] = GY[u] * INV4PI;
        o[3] = GZ[u] * INV4PI;
      }
    }
  }
}

#ifndef XFMM_NEARF2_MINB
#define XFMM_NEARF2_MINB 6  // minimum resident blocks per SM asked of the register allocator (measured best of 1..8)
#endif
#ifndef XFMM_NEARF2_TPL
#define XFMM_NEARF2_TPL 2  // largest number of targets per lane (2 or 4)
#endif
__global__ void __launch_bounds__(128, XFMM_NEARF2_MINB) k_near_lap_f2(NearArgs a) {
  __shared__ NearSmemF2 sm[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = blockIdx.x * 4 + wid;
  if (w >= a.n_eval) return;
  const int node = a.leafs[a.eval_leafs[w]];
  const int T = a.ntrgs[node];
  if (T <= 32) near_leaf_lap_f2<1>(a, node, lane, sm[wid]);
  else if (T <= 64 || XFMM_NEARF2_TPL == 2) near_leaf_lap_f2<2>(a, node, lane, sm[wid]);
  else near_leaf_lap_f2<XFMM_NEARF2_TPL>(a, node, lane, sm[wid]);
}

// the same with the CTA's warps sharing a leaf (few leaves)
__global__ void __launch_bounds__(32 * NEAR_PARTS, XFMM_NEARF2_MINB) k_near_lap_f2_parts(NearArgs a) {
  __shared__ NearSmemF2 sm[NEAR_PARTS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int node = a.leafs[a.eval_leafs[blockIdx.x]];
  if (a.ntrgs[node] <= 32) near_leaf_lap_f2<1, NEAR_PARTS>(a, node, lane, sm[wid], wid);
  else near_leaf_lap_f2<2, NEAR_PARTS>(a, node, lane, sm[wid], wid);
}

// The near field's close pairs (k_near_lap_f2): every (target, source) of a leaf's U list whose FP32
// leaf-relative separation, computed exactly as the near-field kernel computes it, is not above the
// leaf's close-pair distance.  Warp per target leaf; the U-list sources pass through shared memory 32 at
// a time.  FILL = false counts them (one global counter), FILL = true writes (target position in tree
// order, source position, leaf node, 0) at positions taken from a second counter.
template <bool FILL>
__global__ void __launch_bounds__(128) k_close_scan(NearArgs a, unsigned long long* __restrict__ counter,
                                                    int4* __restrict__ pairs, int64_t capacity) {
  __shared__ float4 ss[4][32];
  __shared__ int sidx[4][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = blockIdx.x * 4 + wid;
  if (w >= a.n_eval) return;
  const int node = a.leafs[a.eval_leafs[w]];
  const int T = a.ntrgs[node];
  const int64_t tb = a.tbeg[node];
  const double4 cn = a.center[node];
  const float dc2 = near_close2(cn.w);
  unsigned long long found = 0;
  for (int64_t e = a.p2p_off[node]; e < a.p2p_off[node + 1]; e++) {
    const int sn = a.p2p[e];
    const int ns = a.nsrcs[sn];
    const int64_t sb = a.sbeg[sn];
    for (int j0 = 0; j0 < ns; j0 += 32) {
      __syncwarp();
      if (j0 + lane < ns) {
        const float3 r = leaf_rel(a.src4[sb + j0 + lane], cn);
        ss[wid][lane] = make_float4(r.x, r.y, r.z, 0.f);
        sidx[wid][lane] = (int)(sb + j0 + lane);
      }
      __syncwarp();
      const int cnt = min(32, ns - j0);
      for (int t = lane; t < T; t += 32) {
        const float3 tr = leaf_rel(a.trg4[tb + t], cn);
        for (int j = 0; j < cnt; j++) {
          const float4 sr = ss[wid][j];
          const float dx = __fmaf_rn(sr.x, -1.f, tr.x), dy = __fmaf_rn(sr.y, -1.f, tr.y),
                      dz = __fmaf_rn(sr.z, -1.f, tr.z);
          float r2 = __fmul_rn(dx, dx);
          r2 = __fmaf_rn(dy, dy, r2);
          r2 = __fmaf_rn(dz, dz, r2);
          if (!(r2 > dc2)) {
            if (FILL) {
              const unsigned long long k = atomicAdd(counter, 1ull);
              if ((int64_t)k < capacity) pairs[k] = make_int4((int)(tb + t), sidx[wid][j], node, 0);
            } else {
              found++;
            }
          }
        }
      }
    }
  }
  if (!FILL) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) found += __shfl_xor_sync(0xffffffffu, found, o);
    if (lane == 0 && found) atomicAdd(counter, found);
  }
}

// For each close pair: the exact FP64 contribution (r == 0 skipped, laplace.h:57) in place of the bounded
// FP32 one that k_near_lap_f2 added (recomputed with the same operations; the gradient's FP32 product is
// taken exactly in FP64, as the fused multiply-add took it).
__global__ void k_close_fix(const int4* __restrict__ pairs, int64_t n, NearArgs a1, const NearArgs* __restrict__ args) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int4 pr = pairs[k];
  const NearArgs& a = args ? args[pr.w] : a1;  // one system, or system pr.w of a batch
  const double4 tv = a.trg4[pr.x], sv = a.src4[pr.y], cn = a.center[pr.z];
  const float dc2 = near_close2(cn.w);
  const float3 tr = leaf_rel(tv, cn), sr = leaf_rel(sv, cn);
  const float dx = __fmaf_rn(sr.x, -1.f, tr.x), dy = __fmaf_rn(sr.y, -1.f, tr.y), dz = __fmaf_rn(sr.z, -1.f, tr.z);
  float r2 = __fmul_rn(dx, dx);
  r2 = __fmaf_rn(dy, dy, r2);
  r2 = __fmaf_rn(dz, dz, r2);
  const float inv = rsqrtf(fmaxf(r2, dc2));
  const float qi = __fmul_rn((float)sv.w, inv);
  const float qi3 = __fmul_rn(qi, __fmul_rn(inv, inv));
  double p = -(double)qi, gx = (double)qi3 * dx, gy = (double)qi3 * dy, gz = (double)qi3 * dz;  // remove FP32
  const double ex = tv.x - sv.x, ey = tv.y - sv.y, ez = tv.z - sv.z;
  const double e2 = ex * ex + ey * ey + ez * ez;
  if (e2 > 0.0) {
    const double ir = rsqrt(e2), qe = sv.w * ir, qe3 = qe * ir * ir;
    p += qe;
    gx -= qe3 * ex;
    gy -= qe3 * ey;
    gz -= qe3 * ez;
  }
  double* o = a.out + (int64_t)pr.x * 4;
  atomicAdd(o, p * INV4PI);
  atomicAdd(o + 1, gx * INV4PI);
  atomicAdd(o + 2, gy * INV4PI);
  atomicAdd(o + 3, gz * INV4PI);
}

#ifndef XFMM_NEAR_MAXTPL
#define XFMM_NEAR_MAXTPL 2  // targets per lane of the FP32 near-field kernel (compile-time tunable)
#endif
#ifndef XFMM_NEAR_MINB
#define XFMM_NEAR_MINB 1  // minimum resident blocks per SM requested from the register allocator
#endif

template <int KER, class R>
__global__ void __launch_bounds__(128, XFMM_NEAR_MINB) k_near(NearArgs a) {
  __shared__ NearSmem<R> sm[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = blockIdx.x * 4 + wid;
  if (w >= a.n_eval) return;
  const int node = a.leafs[a.eval_leafs[w]];
  const int T = a.ntrgs[node];
  if constexpr (sizeof(R) == 4) {
    if (T <= 32 || XFMM_NEAR_MAXTPL == 1) near_leaf<KER, R, 1, 0>(a, node, lane, sm[wid]);
    else if (T <= 64 || XFMM_NEAR_MAXTPL == 2) near_leaf<KER, R, (XFMM_NEAR_MAXTPL >= 2 ? 2 : 1), 0>(a, node, lane, sm[wid]);
    else if (T <= 96 || XFMM_NEAR_MAXTPL == 3) near_leaf<KER, R, (XFMM_NEAR_MAXTPL >= 3 ? 3 : 1), 0>(a, node, lane, sm[wid]);
    else near_leaf<KER, R, (XFMM_NEAR_MAXTPL >= 4 ? 4 : 1), 0>(a, node, lane, sm[wid]);
  } else {
    // FP64: one target per lane keeps occupancy up (two per lane: 134 registers, 27.6 -> 31.3 ms at 4M)
    near_leaf<KER, R, 1, 0>(a, node, lane, sm[wid]);
  }
}

// the same with the CTA's warps sharing a leaf (few leaves)
template <int KER, class R>
__global__ void __launch_bounds__(32 * NEAR_PARTS, XFMM_NEAR_MINB) k_near_parts(NearArgs a) {
  __shared__ NearSmem<R> sm[NEAR_PARTS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int node = a.leafs[a.eval_leafs[blockIdx.x]];
  if (sizeof(R) == 4 && a.ntrgs[node] > 32) near_leaf<KER, R, (sizeof(R) == 4 ? 2 : 1), NEAR_PARTS>(a, node, lane, sm[wid], wid);
  else near_leaf<KER, R, 1, NEAR_PARTS>(a, node, lane, sm[wid], wid);
}

// ================================================================ P2M check potentials and P2L
// Potential at `n` surface points (base * b around centre cn) from body range(s); warp per node.
// The Laplace operators are scale-invariant: computed for root radius pre_r0, they serve a tree of root
// radius r0 = lambda pre_r0 unchanged except for a factor lambda on the check potentials that come straight
// from bodies (P2M, P2L).  With the kernel 1 / (4 pi r), K(lambda x, lambda y) = K(x, y) / lambda: the
// check-to-equivalent pseudo-inverse scales by lambda, M2M and L2L (pseudo-inverse times kernel matrix)
// not at all, and the M2L kernel table by 1 / lambda.  Scaling the P2M check potentials by lambda gives the
// true upward densities; the M2L then yields lambda times the true downward check potentials, which P2L
// must match, and the unscaled pseudo-inverse of L2P maps them to the true downward densities.
inline double op_scale(const Fmm& f, const Tree& t) { return f.kernel == XFMM_LAPLACE ? t.r0 / f.pre_r0 : 1.0; }

struct SurfPotArgs {
  const int* nodes;  // node per warp (P2M: leafs; P2L: p2l_nodes)
  int count;
  const int *nsrcs, *p2l, *level;
  const int64_t *sbeg, *p2l_off;
  const double4 *center, *src4;
  const double* src_qim;
  const double* surf_base;
  int nsurf;
  double alpha;        // 2.95 (P2M check) or 1.05 (P2L dn check)
  void* out;           // working values
  int out_by_node;     // 0: row = warp index (P2M chk[pos]); 1: row = node (P2L into dn, accumulate)
  double k_re, k_im;
  double scale;        // 1 / (4 pi) x op_scale(f, t): the Green's function constant and the operators' r0 scale
};

// The points [k0, k1) of a surface of n that blockIdx.y takes: with few nodes several warps share one, each a
// run of whole 32-point rows (the points are independent: the sums do not depend on the split).
__device__ __forceinline__ void surf_range(int n, int& k0, int& k1) {
  const int per = ((n + (int)gridDim.y - 1) / (int)gridDim.y + 31) & ~31;
  k0 = min(n, (int)blockIdx.y * per);
  k1 = min(n, k0 + per);
}
inline dim3 surf_grid_of(int count) { return dim3(nblk(count, 4), count < SPLIT_LEAVES ? 4 : 1); }

template <int KER, class R>
__global__ void __launch_bounds__(128) k_surf_pot(SurfPotArgs a) {
  using G = Green<KER, R>;
  using Q = typename G::Q;
  using V4 = typename R4<R>::type;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = blockIdx.x * 4 + wid;
  if (w >= a.count) return;
  __shared__ V4 s_xyz[4][32];
  __shared__ Q s_q[4][32];
  const G g{(R)a.k_re, (R)a.k_im};
  const int node = a.nodes[w];
  const double4 c = a.center[node];
  const double b = a.alpha * c.w;
  const int n = a.nsurf;
  int kb, ke;
  surf_range(n, kb, ke);
  if (kb >= ke) return;
  Q* out = (Q*)a.out + (int64_t)(a.out_by_node ? node : w) * n;
  const bool p2l = a.out_by_node;
  const int64_t e0 = p2l ? a.p2l_off[node] : 0, e1 = p2l ? a.p2l_off[node + 1] : 1;
  bool first = !p2l;
  for (int64_t e = e0; e < e1; e++) {
    const int s = p2l ? a.p2l[e] : node;
    const int ns = a.nsrcs[s];
    const int64_t sb = a.sbeg[s];
    for (int j0 = 0; j0 < ns || (first && j0 == 0); j0 += 32) {
      const int cnt = max(0, min(32, ns - j0));
      if (lane < cnt) {
        const double4 sv = a.src4[sb + j0 + lane];
        s_xyz[wid][lane] = V4{(R)(sv.x - c.x), (R)(sv.y - c.y), (R)(sv.z - c.z), (R)0};
        s_q[wid][lane] = load_charge<Q>(sv, a.src_qim, sb + j0 + lane);
      }
      __syncwarp();
      for (int k = kb + lane; k < ke; k += 32) {
        const R px = (R)(a.surf_base[3 * k] * b), py = (R)(a.surf_base[3 * k + 1] * b),
                pz = (R)(a.surf_base[3 * k + 2] * b);
        Q acc = vzero<Q>();
        for (int j = 0; j < cnt; j++) {
          const V4 sx = s_xyz[wid][j];
          g.pot(px - sx.x, py - sx.y, pz - sx.z, s_q[wid][j], acc);
        }
        acc = vscale(acc, (typename Base<Q>::type)a.scale);
        out[k] = first ? acc : vadd(out[k], acc);
      }
      first = false;
      __syncwarp();
    }
  }
}

// P2M check potentials of the Laplace mixed path with paired FP32: two sources per instruction
// (__ffma2_rn etc.), 64 sources staged per chunk as float2 pairs, each lane holding SP_KB check points
// per block.  The check surface (half-width 2.95 r) lies at least 1.95 r from every body of the leaf,
// so no pair coincides (no r == 0 mask) and single FP32 coordinates relative to the leaf centre keep
// the separations accurate to a few ulps.  Padding sources have zero charge.
constexpr int SP_KB = 8;  // check points per lane per block
struct SurfSmemF2 {
  float4 pr[32][2];  // source pair j = sources 2j, 2j + 1: {x, x, y, y}, {z, z, q, q}
};
__global__ void __launch_bounds__(128) k_surf_pot_lap_f2(SurfPotArgs a) {
  __shared__ SurfSmemF2 sm[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = blockIdx.x * 4 + wid;
  if (w >= a.count) return;
  const int node = a.nodes[w];
  const double4 c = a.center[node];
  const double b = a.alpha * c.w;
  const int n = a.nsurf, ns = a.nsrcs[node];
  int kb, ke;
  surf_range(n, kb, ke);
  if (kb >= ke) return;
  const int64_t sb = a.sbeg[node];
  float* out = (float*)a.out + (int64_t)w * n;
  const float2 M1 = make_float2(-1.f, -1.f);
  for (int j0 = 0; j0 < ns || j0 == 0; j0 += 64) {
    const bool first = j0 == 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int j = j0 + 32 * h + lane;
      float x = 0.f, y = 0.f, z = 0.f, q = 0.f;
      if (j < ns) {
        const double4 sv = a.src4[sb + j];
        x = (float)(sv.x - c.x);
        y = (float)(sv.y - c.y);
        z = (float)(sv.z - c.z);
        q = (float)sv.w;
      }
      float* r = reinterpret_cast<float*>(sm[wid].pr[16 * h + (lane >> 1)]) + (lane & 1);
      r[0] = x;
      r[2] = y;
      r[4] = z;
      r[6] = q;
    }
    __syncwarp();
    const int npair = (min(64, max(ns - j0, 0)) + 1) >> 1;
    for (int k0 = kb; k0 < ke; k0 += 32 * SP_KB) {
      const int nk = min(SP_KB, (ke - k0 + 31) >> 5);  // slots of this block holding points (warp-uniform)
      float2 px[SP_KB], py[SP_KB], pz[SP_KB], acc[SP_KB];
#pragma unroll
      for (int i = 0; i < SP_KB; i++) {
        const int k = min(k0 + lane + 32 * i, n - 1);  // lanes past the end repeat the last point
        px[i] = dup2((float)(a.surf_base[3 * k] * b));
        py[i] = dup2((float)(a.surf_base[3 * k + 1] * b));
        pz[i] = dup2((float)(a.surf_base[3 * k + 2] * b));
        acc[i] = make_float2(0.f, 0.f);
      }
      for (int jp = 0; jp < npair; jp++) {
        const float4 A = sm[wid].pr[jp][0], B = sm[wid].pr[jp][1];
        const float2 SX = make_float2(A.x, A.y), SY = make_float2(A.z, A.w);
        const float2 SZ = make_float2(B.x, B.y), Q = make_float2(B.z, B.w);
#pragma unroll
        for (int i = 0; i < SP_KB; i++) {
          if (i >= nk) break;
          const float2 dx = __ffma2_rn(SX, M1, px[i]), dy = __ffma2_rn(SY, M1, py[i]), dz = __ffma2_rn(SZ, M1, pz[i]);
          float2 r2 = __fmul2_rn(dx, dx);
          r2 = __ffma2_rn(dy, dy, r2);
          r2 = __ffma2_rn(dz, dz, r2);
          acc[i] = __ffma2_rn(Q, make_float2(rsqrtf(r2.x), rsqrtf(r2.y)), acc[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < SP_KB; i++) {
        const int k = k0 + lane + 32 * i;
        if (k < ke) {
          const float o = (acc[i].x + acc[i].y) * (float)a.scale;
          out[k] = first ? o : out[k] + o;
        }
      }
    }
    __syncwarp();
  }
}

// ================================================================ M2L grid fallback (cuFFT, p beyond the DFT kernels)
template <class W>
__global__ void k_m2l_grid_up(const int* __restrict__ src, int nsrc, const int* __restrict__ child0,
                              const W* __restrict__ up, int nsurf, const int* __restrict__ conv2surf, int nconv,
                              W* __restrict__ grid) {
  const int64_t total = (int64_t)nsrc * 8 * nconv;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(e % nconv);
    const int64_t sc = e / nconv;
    const int sidx = (int)(sc >> 3), c = (int)(sc & 7);
    const int k = conv2surf[g];
    grid[e] = k >= 0 ? up[((int64_t)child0[src[sidx]] + c) * nsurf + k] : vzero<W>();
  }
}

// out[col][row] = in[row][col] for an R x C matrix of complex values (32x32 tiles)
template <class CT>
__global__ void k_transpose(const CT* __restrict__ in, CT* __restrict__ out, int64_t R, int64_t C) {
  __shared__ CT tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, c0 = (int64_t)blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t r = r0 + i, c = c0 + threadIdx.x;
    if (r < R && c < C) tile[i][threadIdx.x] = in[r * C + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t c = c0 + i, r = r0 + threadIdx.x;
    if (r < R && c < C) out[c * R + r] = tile[threadIdx.x][i];
  }
}
// x rounded to TF32 (10 explicit mantissa bits), to nearest with ties away from zero: half of the 13
// dropped bits' range is added to the magnitude and the dropped bits are cleared (a carry moves into
// the exponent when the rounding crosses a binade).  Integer ALU work, where the conversion instruction
// would run on the much narrower transcendental/conversion pipe.
__device__ __forceinline__ uint32_t tf32_head(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
template <class CT>
void transpose(const CT* in, CT* out, int64_t R, int64_t C, cudaStream_t s) {
  dim3 grid((unsigned)((C + 31) / 32), (unsigned)((R + 31) / 32));
  XREQUIRE(grid.y < 65536, XFMM_ERR_UNSUPPORTED, "transpose too tall");
  k_transpose<CT><<<grid, dim3(32, 8), 0, s>>>(in, out, R, C);
  XLAUNCH();
}

// Hadamard product per frequency (fmm_scale_invariant.h:343-399; intrinsics.h matmult_8x8x2):
//   out[f][t][tc] = sum_ipos sum_sc T[ipos][f][sc*8 + tc] * in[f][src(t, ipos)][sc]
// The FP64 path's form runs on the FP64 tensor cores (k_hadamard_d64), the mixed path's on the FP16 tensor
// cores with split operands (k_hadamard_h below).

// Hadamard product of the FP64 path on the FP64 tensor cores (DMMA, mma.sync m8n8k4 f64), for every target.
// A complex product needs three real ones (Gauss): with a = source, b = operator,
//   k1 = (a.re + a.im) b.re,  k2 = a.re (b.im - b.re),  k3 = a.im (b.re + b.im),  a b = (k1 - k3) + i (k1 + k2),
// and the three sums run over the positions and source components before they are combined: per frequency
// three real GEMMs D_i[target][8] = A_i[target][26 x 8] B_i[26 x 8][8], six DMMAs per 8 targets and position
// (two 4-wide reduction steps) where the 2 x 2 real form takes eight.  The FP64 tensor pipe bounds it (16 cycles per
// DMMA and SM quadrant, measured: the same 64 FMA per SM and clock as the FP64 lanes): 1M bodies, p = 8:
// 5.47 -> 3.83 ms (100k: 0.76 -> 0.57; Helmholtz 50k: 0.95 -> 0.69).
// A warp owns HAD64_TW tiles of 8 targets.  Lane (g, t) supplies components 2 t, 2 t + 1 of its target g's
// source spectrum, 32 contiguous bytes in one load (a row's quad reads a whole 128-byte line), step c taking
// component 2 t + c, and receives the target components 2 t, 2 t + 1.  A position none of a tile's 8 targets
// occupies is skipped (warp ballot); a tile's next spectra are loaded as soon as its products are issued.
// The operator's B fragments are built once per table (k_m2l_fragments64) and copied per CTA.
constexpr int HAD64_NT = 256, HAD64_TW = 4;
constexpr int HAD64_TT = (HAD64_NT / 32) * 8 * HAD64_TW;  // targets per CTA
constexpr int HAD64_B = 26 * 6 * 32;                      // B fragments (doubles) per frequency
constexpr size_t HAD64_SMEM = (size_t)HAD64_B * sizeof(double);

__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
// frag[(f * 26 + ipos) * 6 * 32 + (2 i + c) * 32 + lane] = B_i[component 2 t + c][component g] of the block
// of position ipos, i = 0, 1, 2: b.re, b.im - b.re, b.re + b.im.  One warp per block.
__global__ void k_m2l_fragments64(const double2* __restrict__ T, int nfreq, double* __restrict__ frag) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (w >= 26ll * nfreq) return;
  const int f = (int)(w / 26), ipos = (int)(w % 26);
  const double2* blk = T + ((int64_t)ipos * nfreq + f) * 64;
  double* o = frag + w * 6 * 32 + lane;
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const double2 m = blk[(2 * t + c) * 8 + g];
    o[c * 32] = m.x;
    o[(2 + c) * 32] = m.y - m.x;
    o[(4 + c) * 32] = m.x + m.y;
  }
}
__device__ __forceinline__ double4 ldg_double4(const double* p) {  // 32-byte aligned
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// tab: [26][ld] compact source index of target k at each position (-1: empty or padding); rows: [ld]
// output row of target k (-1: padding); ld a multiple of HAD64_TT
__global__ void __launch_bounds__(HAD64_NT, 2)
    k_hadamard_d64(const double* __restrict__ frag, const double2* __restrict__ in, double2* __restrict__ out,
                   const int* __restrict__ tab, int ld, const int* __restrict__ rows, int nsrc, int ntrg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const double* sB = reinterpret_cast<const double*>(smem_raw);
  const int f = blockIdx.y, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  {
    const uint32_t b0 = tc5::smem_u32(smem_raw);
    const double* src = frag + (int64_t)f * HAD64_B;
    for (int e = tid; e < HAD64_B / 2; e += HAD64_NT) tc5::cp_async16(b0 + 16 * e, src + 2 * e, 16u);
    tc5::cp_async_commit();
  }
  const int g = lane >> 2, t = lane & 3;
  const double* inf = reinterpret_cast<const double*>(in + (int64_t)f * nsrc * 8) + 4 * t;
  auto load4 = [&](int sidx) {
    return sidx >= 0 ? ldg_double4(inf + (int64_t)sidx * 16) : make_double4(0.0, 0.0, 0.0, 0.0);
  };
  const int base = blockIdx.x * HAD64_TT + wid * 8 * HAD64_TW + g;  // this lane's target in tile j: base + 8 j
  double acc[HAD64_TW][3][2];
  int src[HAD64_TW], srcn[HAD64_TW];
  double4 x[HAD64_TW];
#pragma unroll
  for (int j = 0; j < HAD64_TW; j++) {
#pragma unroll
    for (int i = 0; i < 3; i++) acc[j][i][0] = acc[j][i][1] = 0.0;
    src[j] = tab[base + 8 * j];
    srcn[j] = tab[ld + base + 8 * j];
  }
#pragma unroll
  for (int j = 0; j < HAD64_TW; j++) x[j] = load4(src[j]);
  tc5::cp_async_wait<0>();
  __syncthreads();
  for (int ipos = 0; ipos < 26; ipos++) {
    double b[6];
#pragma unroll
    for (int i = 0; i < 6; i++) b[i] = sB[(ipos * 6 + i) * 32 + lane];
#pragma unroll
    for (int j = 0; j < HAD64_TW; j++) {
      if (__ballot_sync(0xffffffffu, src[j] >= 0) != 0u) {  // a target of the tile has a source here
        dmma_884(acc[j][0], x[j].x + x[j].y, b[0]);
        dmma_884(acc[j][1], x[j].x, b[2]);
        dmma_884(acc[j][2], x[j].y, b[4]);
        dmma_884(acc[j][0], x[j].z + x[j].w, b[1]);
        dmma_884(acc[j][1], x[j].z, b[3]);
        dmma_884(acc[j][2], x[j].w, b[5]);
      }
      src[j] = srcn[j];
      x[j] = load4(src[j]);  // the next position's spectra, the index of the one after
      srcn[j] = ipos + 2 < 26 ? tab[(ipos + 2) * ld + base + 8 * j] : -1;
    }
  }
  double2* of = out + (int64_t)f * ntrg * 8;
#pragma unroll
  for (int j = 0; j < HAD64_TW; j++) {
    const int row = rows[base + 8 * j];
    if (row < 0) continue;
#pragma unroll
    for (int i = 0; i < 2; i++)
      of[(int64_t)row * 8 + 2 * t + i] = make_double2(acc[j][0][i] - acc[j][2][i], acc[j][0][i] + acc[j][1][i]);
  }
}

// M2L Hadamard product of the mixed path on the tensor cores (k_hadamard_h, below).  Spectra and products are
// frequency-major, (frequency f, node, child c) at [(f * nrows + node) * 8 + c]: a CTA (one frequency)
// reads its sources from one block of the spectra and writes its rows contiguously.
//
// The mixed path's spectra are stored split: a real x is the pair of FP16 values h = fp16(2^e x) and
// t = fp16(c (2^e x - h)).  A split spectrum has the size of the FP32 one, the products need no conversion (the
// operator's blocks are split the same way, k_m2l_fragments), and an FP16 MMA does twice the work of a TF32 one
// in the same 8 cycles (measured: m16n8k16 f16 and m16n8k8 tf32 both 8.0 cycles per warp and SM quadrant) with
// the same 11-bit significands.  A child's complex value is the 8 bytes {h.re, h.im, t.re, t.im}.
// Every spectrum value of a child is at most the sum of its densities' magnitudes, its bound, and no error may
// show beside the FP32 rounding of what reaches the same targets.  Two forms:
//  * Laplace, Helmholtz with a real wavenumber: c = 1, one exponent per source node, set by its strongest child.
//    22 bits within 2^-17 of the top (2^15), an absolute error below 2^-39 of it elsewhere: far below the
//    rounding of the strongest child's field, which reaches the same targets at a comparable distance.
//  * Screened kernels (modified Helmholtz, complex wavenumbers) show weak sources, for a strong one's field is
//    gone where a weak one's targets are: c = 2^11, which keeps 22 bits down to 2^-29 of the top and an
//    absolute error below 2^-51 of it.  The largest bound of a group's sources (k_source_bounds) sets e0, and the
//    children are sorted into windows of 2^-28 below it, window w with the exponent e0 + 28 w: the error of
//    a value is at most 2^-23 of its own child's bound (the FP32 transform itself rounds at 2^-24 of it).
using SplitC = uint2;
constexpr float SPLIT_TAIL = 2048.f;  // c of the screened kernels
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ float2 h2_float2(uint32_t u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }
__device__ __forceinline__ SplitC split16(float re, float im, float c) {
  const __half2 h = __floats2half2_rn(re, im);
  const float2 hf = __half22float2(h);
  return make_uint2(h2_bits(h), h2_bits(__floats2half2_rn((re - hf.x) * c, (im - hf.y) * c)));
}
__device__ __forceinline__ float pow2f(int e) { return e >= -126 ? __uint_as_float((uint32_t)(127 + e) << 23) : 0.f; }
__device__ __forceinline__ int float_exp(float b) { return (int)(__float_as_uint(b) >> 23) - 127; }  // b >= 0
// The exponent e of a node whose spectrum values are at most `bound` in magnitude: 2^e bound < 2^15 (FP16
// holds 2^16), e odd, as the code k = (127 - e) / 2 in 1..126, so that 2^-e is the float whose exponent
// field is 2 k.  SPLIT_ZERO beside it: a node without values.
__device__ __forceinline__ int split_code(float bound) {
  int e = bound > 0.f ? 14 - float_exp(bound) : 1;
  e = max(-125, min(125, e));
  if (!(e & 1)) e -= 1;
  return (127 - e) >> 1;
}
constexpr int SPLIT_ZERO = 0x100;
__device__ __forceinline__ float split_scale(int code) { return __uint_as_float((uint32_t)(254 - 2 * code) << 23); }
// Screened kernels: e0, a window's exponent, the window of a child.
constexpr int SPLIT_WIN = 28;
__device__ __forceinline__ int split_exp0(float bound) { return bound > 0.f ? min(126, 14 - float_exp(bound)) : 0; }
__device__ __forceinline__ int split_exp(int e0, int w) { return min(126, e0 + SPLIT_WIN * w); }
__device__ __forceinline__ int split_window(float bound, int e0) {
  return bound > 0.f ? max(0, 14 - e0 - float_exp(bound)) / SPLIT_WIN : 0;
}
struct SplitHead {
  unsigned gmax, done;  // largest bound so far (float bits) and finished blocks: zero between uses
  int e0;
  unsigned mask;        // bit w: a child in window w
};
// what a forward transform reads and writes beside the spectra; head null: not screened
struct SplitOut {
  int* code;
  const float* bound;
  uint8_t* win;
  SplitHead* head;
};
// Packed sources: the source row in the low 25 bits (2^25 sources would need 206 GB of spectra at the lowest
// order) and 7 bits of exponent: in the opt-in tcgen05 form's table the source's code (written by
// k_pack_sources after every forward transform), in a tile's slot list the source's distance from the tile's
// largest code in steps (k_tile_codes).  Screened kernels: the row alone.  SPLIT_NONE: no source.
constexpr int SPLIT_ROW_BITS = 25;
constexpr uint32_t SPLIT_ROW_MASK = (1u << SPLIT_ROW_BITS) - 1;
constexpr uint32_t SPLIT_NONE = 0xffffffffu;
__device__ __forceinline__ float split_inv(uint32_t ent) { return __uint_as_float((ent >> 1) & 0x7f000000u); }
__device__ __forceinline__ float split_inv_code(int code) { return __uint_as_float((uint32_t)code << 24); }
__global__ void k_pack_sources(const int* __restrict__ in, int64_t n, const int* __restrict__ scode,
                               uint32_t* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i] >= 0 ? (uint32_t)in[i] | ((uint32_t)(scode[in[i]] & 0x7f) << SPLIT_ROW_BITS) : SPLIT_NONE;
}

// opt-in tcgen05 form (k_hadamard_dc): occupied positions that make a target dense, dense targets a group
// needs; every other target runs in k_hadamard_h
constexpr int HAD_DENSE_MIN = 12, HAD_DENSE_GROUP_MIN = 256;
constexpr int HADC_TT = 512;  // padding of its source table

// Hadamard product on the tensor cores (FP32 accuracy from three FP16 products).
// Per frequency the product is a real GEMM, D[target][16] = A[target][26 x 16] B[26 x 16][16]: a target's
// row of A holds its 26 source spectra (8 complex = 16 reals each, zeros where a position is empty) and B
// holds each position's 8x8 complex block as 2x2 real blocks ([re, im] -> [re, im]).  Warp-level m16n8k16
// FP16 MMAs with FP32 accumulators: A and B are FP16 heads and tails, and each position's
// (At Bh + Ah Bt) / c + Ah Bh (small terms first; the tail-tail product, 2^-22 relative, is dropped) is formed in
// a fresh MMA accumulator, scaled by the block's exponent and added to FP32 running sums in one fused
// multiply-add (the MMA's own accumulation is not rounded to nearest).
//
// A CTA owns a tile of up to 512 targets at one frequency.  The tile's distinct sources (up to 1016, about
// twice the targets of a spatially compact tile, each used by up to 26 of them) are brought into shared
// memory once, on the exponent of the strongest, and every A fragment is read from there with ldmatrix, whose lanes
// address the rows of a fragment freely: a gather without register moves at 8 shared-memory cycles per 16
// targets and position.  Measured, Hadamard stage: 1M bodies, p = 10: 2.8 ms (the same products gathered
// row by row from L1 at 14 cycles per 16 targets: 4.03; the TF32 form with per-use conversions before it:
// 5.26); 4M, p = 8, whose deepest level has ~7 of 26 positions occupied: 4.1 (TF32 with packed rounds of
// pairs and atomics: 6.15); Helmholtz 200k, p = 12: 1.71 (3.55).
// Bank conflicts: a source's slot is 8 k + (octant of the source in its parent).  The sources of 8 sibling
// targets at one relative position have 8 different octants, so their 64-byte rows (four 16-byte chunks,
// swizzled by (slot / 2) % 4) fall on different banks; empty positions read one of 8 zero slots, chosen to
// stay off the banks of the other rows.
// A tile whose sources lie within 2^-18 of the strongest has one pass: all tiles of cubes, Plummer spheres and
// surfaces of up to 4M bodies with charges in (-1, 1), 2 to 9 steps of 2 bits.  Otherwise pass w takes the sources
// 10 w .. 10 w + 9 steps below, the others at zero, over the same accumulators: weak sources keep their bits.  With
// the screened kernels the passes are the windows of the tile's children, each with every window of the operator.
// Tiles with at most 256, 128 or 64 targets split the 26 positions over 2, 4 or 8 warps per 64 targets.
// Bounds per 64 targets and position and SM (cycles): MMAs 24 x 8 / 4 = 48; shared memory 32 (A) + 8 (B).
// At 1M, p = 8 the tensor pipe is 58% and the shared-memory pipe 70% busy: 16 warps per SM hide the rest of
// the latencies only in part.  Smaller tiles at three CTAs per SM (384 targets, 704 slots) close early in
// full volumes (p = 10: 3.83 ms); several tiles per CTA gain nothing.
constexpr int HADH_NT = 256, HADH_TT = 512;      // threads, targets per tile
constexpr int HADH_SLOTS = 1024;                 // source slots, the first 8 zeros
constexpr int HADH_TPC = 1;                      // default tiles per CTA
constexpr int HADH_B = 26 * 2 * 32;              // B fragments (uint4) in shared memory
constexpr int HADH_FB = HADH_B / 2;              // and as stored
constexpr size_t HADH_SMEM = (size_t)HADH_SLOTS * 64 + (size_t)HADH_B * 16 + 32 * sizeof(float);
static_assert(2 * (HADH_SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
constexpr int SPLIT_PASS = 10;                   // steps of 2 bits that one pass over a tile covers
struct HadTile {
  int nslots;   // slots used (a multiple of 8, the zero slots included)
  int groups;   // 1, 2, 4 or 8 groups of 64 targets
  int slot0;    // first entry of the tile in the slot list (source of each slot, -1: none)
  int row0;     // first entry of the tile in the row list (output row of each target, -1: padding)
  int64_t tab0; // first entry of the tile in the table: [position][group][lane] of 4 x 16 bits
};
struct HadSys {
  const SplitC* in;       // split spectra [f][nsrc][child]
  float2* out;            // products [f][target][child]
  const HadTile* tiles;
  const uint32_t* slots;  // packed source of each slot (k_tile_codes)
  const float* tinv;      // per tile: undoes its exponent
  const uint32_t* tpass;  // per tile: bit w: pass w has sources
  const SplitHead* head;  // screened kernels: exponents, and the window of every source's children
  const uint8_t* win;
  const uint2* tab;
  const int* rows;
  int nsrc, ntrg;
};

// not volatile: the compiler interleaves independent accumulators
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same into a fresh accumulator
__device__ __forceinline__ void mma_f16_new(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// head and tail of x: x = head + tail exactly, head a TF32 value
__device__ __forceinline__ void tf32_split(float x, uint32_t& h, uint32_t& t) {
  h = tf32_head(x);
  t = tf32_head(x - __uint_as_float(h));
}

// The operator blocks of frequency f as the kernel's B fragments, built once per operator table from its
// FP64 values: for every (position, output half h, lane) of a warp the four registers {b0 head, b1 head,
// b0 tail, b1 tail}, scaled by the block's exponent; b0 / b1 are the factors of source components t / t + 4
// and half h the target components 4 h .. 4 h + 3 (t = lane % 4).  Stored are the lanes of even g = lane / 4
// (real outputs: (Re, -Im) of a factor), at frag[(v * nfreq + f) * HADH_FB + (ipos * 2 + h) * 16 + 4 (g / 2) + t];
// those of g + 1 (imaginary outputs: (Im, Re)) are the same values swapped (hadh_odd).
// inv[(v * nfreq + f) * 32 + ipos] undoes the exponent.  One warp per block.
// v: the operator's window.  The factors of a screened kernel's child pairs differ by e^(-k (distance)): a
// pair whose largest factor over the frequencies (k_pair_max) is more than 2^-28 below the largest of its
// position goes to the next window, with an exponent of its own, as the sources' children do; pwin[ipos * 64 + pair]
// is the pair's window (null: one window, the unscreened kernels).  Modified Helmholtz takes a second from
// k (box size) of about 7 on.
__global__ void __launch_bounds__(256)
    k_pair_max(const double2* __restrict__ T, int nfreq, unsigned* __restrict__ pmax) {
  const int pair = threadIdx.x & 63, ipos = blockIdx.y;
  float m = 0.f;
  for (int f = blockIdx.x * 4 + (threadIdx.x >> 6); f < nfreq; f += gridDim.x * 4) {
    const double2 q = T[((int64_t)ipos * nfreq + f) * 64 + pair];
    m = fmaxf(m, (float)fmax(fabs(q.x), fabs(q.y)));
  }
  atomicMax(pmax + ipos * 64 + pair, __float_as_uint(m));
}
__global__ void k_m2l_fragments(const double2* __restrict__ T, int nfreq, const uint8_t* __restrict__ pwin, double tail,
                                uint4* __restrict__ frag, float* __restrict__ inv) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, win = blockIdx.y;
  if (w >= 26ll * nfreq) return;
  const int f = (int)(w / 26), ipos = (int)(w % 26);
  const double2* blk = T + ((int64_t)ipos * nfreq + f) * 64;
  auto entry = [&](int pair) { return !pwin || pwin[ipos * 64 + pair] == win ? blk[pair] : make_double2(0.0, 0.0); };
  const double2 u = entry(lane), v = entry(32 + lane);
  float m = (float)fmax(fmax(fabs(u.x), fabs(u.y)), fmax(fabs(v.x), fabs(v.y)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int code = split_code(m);
  const double sc = (double)split_scale(code);
  const int h = lane >> 4, tc = 4 * h + ((lane >> 2) & 3), t = lane & 3;
  uint32_t hd[2], tl[2];
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const double2 q = entry((t + 4 * c) * 8 + tc);
    const double re = q.x * sc, im = -q.y * sc;
    const __half2 hh = __halves2half2(__double2half(re), __double2half(im));
    const float2 hf = __half22float2(hh);
    hd[c] = h2_bits(hh);
    tl[c] = h2_bits(__halves2half2(__double2half((re - hf.x) * tail), __double2half((im - hf.y) * tail)));
  }
  const int64_t row = (int64_t)win * nfreq + f;
  frag[row * HADH_FB + ipos * 32 + lane] = make_uint4(hd[0], hd[1], tl[0], tl[1]);
  if (lane == 0) inv[row * 32 + ipos] = split_inv_code(code);
}
// the registers of lane g + 1 from those of an even g: (Re, -Im) -> (Im, Re) in every half pair
__device__ __forceinline__ uint4 hadh_odd(const uint4& e) {
  auto sw = [](uint32_t v) { return __byte_perm(v, v, 0x1032) ^ 0x8000u; };
  return make_uint4(sw(e.x), sw(e.y), sw(e.z), sw(e.w));
}
// After a forward transform of an unscreened kernel, per tile (one CTA each): the largest exponent code of its
// sources, whose exponent is the tile's, the slot list packed with every source's distance d from it (SPLIT_NONE:
// no source, or one without values), and the passes that the tile needs.
__global__ void __launch_bounds__(256)
    k_tile_codes(const HadTile* __restrict__ tiles, const int* __restrict__ slots, const int* __restrict__ scode,
                 uint32_t* __restrict__ pslots, float* __restrict__ tinv, uint32_t* __restrict__ tpass) {
  __shared__ int smax;
  __shared__ uint32_t spass;
  const HadTile T = tiles[blockIdx.x];
  if (threadIdx.x == 0) {
    smax = 1;
    spass = 1u;
  }
  __syncthreads();
  int src[(HADH_SLOTS + 255) / 256], code[(HADH_SLOTS + 255) / 256], kmax = 1;
#pragma unroll
  for (int i = 0; i < (HADH_SLOTS + 255) / 256; i++) {
    const int q = threadIdx.x + 256 * i;
    src[i] = q < T.nslots ? slots[T.slot0 + q] : -1;
    code[i] = src[i] >= 0 ? scode[src[i]] : SPLIT_ZERO;
    if (code[i] & SPLIT_ZERO) src[i] = -1;
    else kmax = max(kmax, code[i]);
  }
  atomicMax(&smax, __reduce_max_sync(0xffffffffu, kmax));
  __syncthreads();
  kmax = smax;
  uint32_t pass = 0u;
#pragma unroll
  for (int i = 0; i < (HADH_SLOTS + 255) / 256; i++) {
    const int q = threadIdx.x + 256 * i, d = kmax - code[i];
    if (q < T.nslots)
      pslots[T.slot0 + q] = src[i] >= 0 ? (uint32_t)src[i] | (uint32_t)d << SPLIT_ROW_BITS : SPLIT_NONE;
    if (src[i] >= 0) pass |= 1u << (d / SPLIT_PASS);
  }
  pass = __reduce_or_sync(0xffffffffu, pass);
  if ((threadIdx.x & 31) == 0) atomicOr(&spass, pass);
  __syncthreads();
  if (threadIdx.x == 0) {
    tinv[blockIdx.x] = split_inv_code(kmax);
    tpass[blockIdx.x] = spass;
  }
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// Table entry of a slot: 4 slot + swizzle; chunk c of the slot is at 16 (entry ^ c).
__host__ __device__ __forceinline__ uint32_t hadh_entry(int slot) { return (uint32_t)(4 * slot + ((slot >> 1) & 3)); }

// one tile at frequency f; with `fill` it also brings the frequency's B fragments and block scales (frag, binv: those
// of f; bstride frequencies between the operator's nbw windows) into shared memory
template <bool SCREENED>
__device__ __forceinline__ void hadh_tile(const HadSys& S, int tile, int f, unsigned char* sA, uint4* sB, float* sInv,
                                          const uint4* __restrict__ frag, const float* __restrict__ binv, int nbw,
                                          int bstride, bool fill, int tid) {
  const HadTile T = S.tiles[tile];
  const int lane = tid & 31, wid = tid >> 5;
  // ---- the tile's sources: four threads per slot, 16 bytes each
  const uint4* inf = reinterpret_cast<const uint4*>(S.in + (int64_t)f * S.nsrc * 8);
  const uint32_t* slots = S.slots + T.slot0;
  constexpr int QS = HADH_NT / 4, NB = (HADH_SLOTS + QS - 1) / QS;  // slots per round; rounds, all in flight
  const int c = tid & 3;
  constexpr int NF = (HADH_FB + HADH_NT - 1) / HADH_NT;
  // global pieces are children 2c, 2c + 1 as {head, tail, head, tail}; shared chunks are heads of
  // children 0-3 and 4-7, then tails
  auto store_a = [&](int q, const uint4& w) {
    const uint32_t e = hadh_entry(q);
    *reinterpret_cast<uint2*>(sA + 16 * (e ^ (c >> 1)) + 8 * (c & 1)) = make_uint2(w.x, w.z);
    *reinterpret_cast<uint2*>(sA + 16 * (e ^ (2 + (c >> 1))) + 8 * (c & 1)) = make_uint2(w.y, w.w);
  };
  auto store_b = [&](const uint4 (&fb)[NF], const float* bi) {
#pragma unroll
    for (int i = 0; i < NF; i++) {
      const int e = tid + HADH_NT * i, ln = e & 15;  // stored lane 4 (g / 2) + t
      if (e >= HADH_FB) break;
      uint4* o = sB + (e >> 4) * 32 + (ln >> 2) * 8 + (ln & 3);
      o[0] = fb[i];
      o[4] = hadh_odd(fb[i]);
    }
    if (tid < 26) sInv[tid] = bi[tid];
  };
  auto load_b = [&](const uint4* fr, uint4 (&fb)[NF]) {
#pragma unroll
    for (int i = 0; i < NF; i++) fb[i] = __ldg(fr + min(tid + HADH_NT * i, HADH_FB - 1));
  };
  auto scaled = [](uint32_t v, int d) {  // times 2^(-2 d), d < SPLIT_PASS
    const __half2 m = __float2half2_rn(__uint_as_float((uint32_t)(127 - 2 * d) << 23));
    return h2_bits(__hmul2(*reinterpret_cast<__half2*>(&v), m));
  };
  // pass w alone: the sources 10 w .. 10 w + 9 steps below the tile's exponent, at the exponent 20 w above it
  // (stored 2 d above); screened: the children of window w, as they are stored
  auto load_pass = [&](int w) {
    for (int q = tid >> 2; q < T.nslots; q += QS) {
      const uint32_t e = slots[q];
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (e != SPLIT_NONE) {
        if constexpr (SCREENED) {
          const uchar2 cw = reinterpret_cast<const uchar2*>(S.win)[(int64_t)e * 4 + c];
          v = __ldg(inf + (int64_t)e * 4 + c);
          if (cw.x != w) v.x = v.y = 0u;
          if (cw.y != w) v.z = v.w = 0u;
        } else {
          const int d = (int)(e >> SPLIT_ROW_BITS) - SPLIT_PASS * w;
          if (d >= 0 && d < SPLIT_PASS) {
            v = __ldg(inf + (int64_t)(e & SPLIT_ROW_MASK) * 4 + c);
            v = make_uint4(scaled(v.x, d), scaled(v.y, d), scaled(v.z, d), scaled(v.w, d));
          }
        }
      }
      store_a(q, v);
    }
  };
  uint4 fb[NF];
  if (fill) load_b(frag, fb);
  uint32_t todo;  // the passes left, the open one included
  int x0 = 0, xt = 0;
  if constexpr (SCREENED) {
    x0 = S.head->e0;
    todo = S.head->mask;
    if (todo != 1u) {  // the windows of the tile's own sources
      __shared__ uint32_t stodo;
      if (tid == 0) stodo = 0u;
      __syncthreads();
      uint32_t m = 0u;
      for (int q = tid; q < T.nslots; q += HADH_NT) {
        const uint32_t e = slots[q];
        for (int k = 0; e != SPLIT_NONE && k < 8; k++) m |= 1u << S.win[(int64_t)e * 8 + k];
      }
      m = __reduce_or_sync(0xffffffffu, m);
      if (lane == 0) atomicOr(&stodo, m);
      __syncthreads();
      todo = stodo ? stodo : 1u;
    }
    xt = split_exp(x0, __ffs(todo) - 1);  // the sums are formed at the tile's strongest window's exponent
  } else {
    todo = S.tpass[tile];
  }
  if (SCREENED ? S.head->mask == 1u : todo == 1u) {
    uint32_t src[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) {
      const int q = (tid >> 2) + QS * i;
      src[i] = q < T.nslots ? slots[q] : SPLIT_NONE;
    }
    uint4 v[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) {
      const uint32_t e = src[i];
      const int64_t row = SCREENED ? e : e & SPLIT_ROW_MASK;
      v[i] = e != SPLIT_NONE ? __ldg(inf + row * 4 + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < NB; i++) {
      const int q = (tid >> 2) + QS * i;
      if (q >= T.nslots) break;
      uint4 w = v[i];
      if constexpr (!SCREENED) {
        const int d = src[i] != SPLIT_NONE ? (int)(src[i] >> SPLIT_ROW_BITS) : 0;
        if (d > 0) w = make_uint4(scaled(w.x, d), scaled(w.y, d), scaled(w.z, d), scaled(w.w, d));
      }
      store_a(q, w);
    }
  } else {
    load_pass(__ffs(todo) - 1);
  }
  if (fill) store_b(fb, binv);
  __syncthreads();
  float pscale = 1.f;  // of the open pass
  int bw = 0;          // the open window of the operator
  // ---- products: group gr of 64 targets, positions ps, ps + np, ...
  const int gr = wid % T.groups, ps = wid / T.groups, np = (HADH_NT / 32) / T.groups;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t a0 = tc5::smem_u32(sA);
  const uint32_t ch = (uint32_t)(lane >> 4);
  const uint2* tab = S.tab + T.tab0 + gr * 32 + lane;
  const int pstep = T.groups * 32;
  float acc[4][2][4];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[j][h][i] = 0.f;
  for (;;) {
  // table entries two positions ahead
  uint2 e0 = __ldg(tab + ps * pstep), e1 = __ldg(tab + min(ps + np, 25) * pstep);
  for (int ipos = ps; ipos < 26; ipos += np) {
    const uint2 e = e0;
    e0 = e1;
    e1 = __ldg(tab + min(ipos + 2 * np, 25) * pstep);
    const uint4 b[2] = {sB[(ipos * 2) * 32 + lane], sB[(ipos * 2 + 1) * 32 + lane]};
    const float ib = sInv[ipos] * pscale;
#pragma unroll
    for (int jp = 0; jp < 4; jp += 2) {
      uint32_t xh[2][4], xt[2][4];
      const uint32_t ee = jp ? e.y : e.x;
#pragma unroll
      for (int jj = 0; jj < 2; jj++) {
        const uint32_t en16 = (jj ? ee >> 16 : ee & 0xffffu) ^ ch;
        ldsm_x4(a0 + (en16 << 4), xh[jj]);
        ldsm_x4(a0 + ((en16 ^ 2u) << 4), xt[jj]);
      }
      float d[2][2][4];
#pragma unroll
      for (int jj = 0; jj < 2; jj++)
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f16_new(d[jj][h], xt[jj][0], xt[jj][1], xt[jj][2], xt[jj][3], b[h].x, b[h].y);
#pragma unroll
      for (int jj = 0; jj < 2; jj++)
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f16(d[jj][h], xh[jj][0], xh[jj][1], xh[jj][2], xh[jj][3], b[h].z, b[h].w);
#pragma unroll
      for (int jj = 0; jj < 2; jj++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if constexpr (SCREENED)
#pragma unroll
            for (int i = 0; i < 4; i++) d[jj][h][i] *= 1.f / SPLIT_TAIL;
          mma_f16(d[jj][h], xh[jj][0], xh[jj][1], xh[jj][2], xh[jj][3], b[h].x, b[h].y);
        }
#pragma unroll
      for (int jj = 0; jj < 2; jj++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int i = 0; i < 4; i++) acc[jp + jj][h][i] = fmaf(d[jj][h][i], ib, acc[jp + jj][h][i]);
    }
  }
  // ---- the next window of the operator, then the next pass over the sources
  if (++bw == nbw) {
    bw = 0;
    todo &= todo - 1u;
    if (todo == 0u) break;
  }
  __syncthreads();
  if (nbw > 1) {
    load_b(frag + (int64_t)bw * bstride * HADH_FB, fb);
    store_b(fb, binv + (int64_t)bw * bstride * 32);
  }
  if (bw == 0) {
    const int w = __ffs(todo) - 1;
    load_pass(w);
    pscale = pow2f(SCREENED ? xt - split_exp(x0, w) : -2 * SPLIT_PASS * w);
  }
  __syncthreads();
  }
  // ---- the position parts of a group, added in order by its first warp
  if (np > 1) {
    __syncthreads();
    float4* red = reinterpret_cast<float4*>(sA) + wid * 8 * 32 + lane;
    if (ps > 0) {
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          red[(2 * j + h) * 32] = make_float4(acc[j][h][0], acc[j][h][1], acc[j][h][2], acc[j][h][3]);
    }
    __syncthreads();
    if (ps > 0) return;
    for (int k = 1; k < np; k++) {
      const float4* r = red + k * T.groups * 8 * 32;
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const float4 w = r[(2 * j + h) * 32];
          acc[j][h][0] += w.x;
          acc[j][h][1] += w.y;
          acc[j][h][2] += w.z;
          acc[j][h][3] += w.w;
        }
    }
  }
  // D fragment: row g (and g + 8), columns 2t, 2t + 1 of half h = target component 4 h + t (re, im)
  const float inv = SCREENED ? pow2f(-xt) : S.tinv[tile];
  float2* of = S.out + (int64_t)f * S.ntrg * 8;
  const int* rows = S.rows + T.row0 + gr * 64 + g;
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int row = rows[16 * j + 8 * r];
      if (row < 0) continue;
#pragma unroll
      for (int h = 0; h < 2; h++)
        of[(int64_t)row * 8 + 4 * h + t] = make_float2(acc[j][h][2 * r] * inv, acc[j][h][2 * r + 1] * inv);
    }
}

// tiles [blockIdx.x * tpc, ...) at frequency blockIdx.y share one copy of the frequency's B fragments
template <bool SCREENED>
__global__ void __launch_bounds__(HADH_NT, 2)
    k_hadamard_h(const uint4* __restrict__ frag, const float* __restrict__ binv, int nbw, HadSys S, int ntiles, int tpc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* sB = reinterpret_cast<uint4*>(smem_raw + (size_t)HADH_SLOTS * 64);
  float* sInv = reinterpret_cast<float*>(sB + HADH_B);
  const int f = blockIdx.y, tid = threadIdx.x;
  const int te = min(ntiles, ((int)blockIdx.x + 1) * tpc);
  for (int k = blockIdx.x * tpc; k < te; k++) {
    hadh_tile<SCREENED>(S, k, f, smem_raw, sB, sInv, frag + (int64_t)f * HADH_FB, binv + f * 32, nbw, gridDim.y,
                        nbw > 1 || k == (int)blockIdx.x * tpc, tid);
    if (k + 1 < te) __syncthreads();
  }
}
// the same over the tiles of many systems that share one operator table (a batch of Laplace systems):
// tiles[k] = (system, its tile)
__global__ void __launch_bounds__(HADH_NT, 2)
    k_hadamard_h_batch(const uint4* __restrict__ frag, const float* __restrict__ binv, const HadSys* __restrict__ sys,
                       const int2* __restrict__ tiles, int ntiles, int tpc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* sB = reinterpret_cast<uint4*>(smem_raw + (size_t)HADH_SLOTS * 64);
  float* sInv = reinterpret_cast<float*>(sB + HADH_B);
  const int f = blockIdx.y, tid = threadIdx.x;
  const int te = min(ntiles, ((int)blockIdx.x + 1) * tpc);
  for (int k = blockIdx.x * tpc; k < te; k++) {
    const int2 tl = tiles[k];
    hadh_tile<false>(sys[tl.x], tl.y, f, smem_raw, sB, sInv, frag + (int64_t)f * HADH_FB, binv + f * 32, 1, gridDim.y,
                     k == (int)blockIdx.x * tpc, tid);
    if (k + 1 < te) __syncthreads();
  }
}

// Hadamard product, dense form on the sm_100 tensor cores through tcgen05 (FP32 accuracy from three TF32
// products of the spectra's head + tail), as a warp-specialised pipeline.  A CTA owns 128 dense targets (target
// slot i = TMEM lane i) and HADC_FPB frequencies, i.e. a stream of 26 HADC_FPB positions.
//   * Warps 0-3 (one per TMEM lane quarter) produce and consume: per position, the 4 lanes of a quad load
//     one source spectrum as 4 contiguous 16-byte pieces (one position ahead), split it into TF32 head
//     and tail and store both into the position's TMEM stage (operand A, `tcgen05.st.16x256b`), then
//     arrive on the stage's `full` barrier.  Before reusing a stage they wait for its `done` barrier,
//     read the products of the position HADC_S earlier back (`tcgen05.ld`) and add them to FP32 running
//     sums in registers (round-to-nearest adds; the tensor core's own accumulation never spans more than
//     one position); after a frequency's last position they store its 128 output rows.
//   * Warp 4 issues: per frequency one bulk copy of the 26 positions' B blocks (built once per operator
//     in the MMA layout by k_hadc_btab) into shared memory, then per position, once the stage is full,
//     six M128 N16 K8 kind::tf32 MMAs (A tail x B head, A head x B tail, A head x B head per 8-wide
//     step) into the stage's fresh TMEM accumulator, committed to `done`.
// No CTA-wide barrier inside the stream.  Every wait is bounded (about a second); a wait that runs out
// ends the waiting role's loop, the others then run out in turn, the CTA releases its TMEM and *status
// is set.
constexpr int HADC_NT = 160;                                // 4 producer/consumer warps + 1 MMA warp
constexpr int HADC_S = 4;                                   // TMEM stages
constexpr int HADC_D = 4;                                   // positions gathered ahead (cp.async ring)
constexpr int HADC_R = HADC_D + 1;                          // ring slots: 128 rows x 64 bytes each
constexpr int HADC_FPB = 8;                                 // frequencies per CTA
constexpr uint32_t HADC_BBYTES = 26 * 2048;                 // B of one frequency: [position][head, tail] 1 KB each
// dynamic shared memory per CTA: B, then the gather ring; at least 96 KB so that at most two CTAs share an
// SM, whose TMEM (512 columns) holds exactly two allocations of HADC_TMEM_COLS
constexpr size_t HADC_RING = (size_t)HADC_R * 128 * 64;
constexpr size_t HADC_SMEM = HADC_BBYTES + HADC_RING > 96 * 1024 ? HADC_BBYTES + HADC_RING : 96 * 1024;
static_assert(3 * HADC_SMEM > 228 * 1024 && 2 * HADC_SMEM <= 227 * 1024, "two CTAs per SM");
constexpr uint32_t HADC_TMEM_COLS = 256;                    // A: HADC_S x 32 columns, then D: HADC_S x 16
constexpr uint32_t HADC_DCOL = 32 * HADC_S;                 // first D column
constexpr long long HADC_WAIT = 2000000000LL;               // SM cycles (about a second) before a wait gives up
static_assert(HADC_DCOL + 16 * HADC_S <= HADC_TMEM_COLS, "TMEM columns");

// The A columns (reduction index) are a permutation of the 16 input reals fixed by the TMEM store shape
// (16x256b): the 4 lanes of a quad load one source spectrum as 4 contiguous 16-byte pieces, lane q the
// reals 4q .. 4q + 3, which land in columns 2q, 2q + 1, 8 + 2q, 9 + 2q.  Column of input real k:
__host__ __device__ __forceinline__ int hadc_col(int k) {
  const int q = k >> 2, r = k & 3;
  return r < 2 ? 2 * q + r : 8 + 2 * q + (r - 2);
}
// byte offset of B element (output real n, A column c) in the 1 KB block of one (position, part):
// core matrix (c / 4, n / 8) at 256 (c / 4) + 128 (n / 8), its row n % 8 at 16 (n % 8), column c % 4
__host__ __device__ __forceinline__ uint32_t hadc_boff(int n, int c) {
  return (uint32_t)((c >> 2) * 256 + (n >> 3) * 128 + (n & 7) * 16 + (c & 3) * 4);
}
// btab[f] (HADC_BBYTES per frequency): factor m(sc, tc) of position ipos (head + tail of the stored
// fragments) -> the real 2 x 2 block (outputs 2 tc, 2 tc + 1; inputs 2 sc, 2 sc + 1) =
// [[Re m, -Im m], [Im m, Re m]], TF32 head then tail
__global__ void k_hadc_btab(const uint4* __restrict__ frag, const float* __restrict__ binv, int nbw, float itail,
                            int nfreq, unsigned char* __restrict__ btab) {
  const int64_t total = (int64_t)nfreq * 26 * 64;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int f = (int)(e / (26 * 64)), ipos = (int)(e / 64 % 26), sc = (int)(e >> 3 & 7), tc = (int)(e & 7);
    float2 m = make_float2(0.f, 0.f);
    for (int w = 0; w < nbw; w++) {  // the factor stands in one of the operator's windows, zeros in the others
      const int64_t row = (int64_t)w * nfreq + f;
      const uint4 q = frag[row * HADH_FB + (ipos * 2 + (tc >> 2)) * 16 + 4 * (tc & 3) + (sc & 3)];
      const float2 hd = h2_float2(sc < 4 ? q.x : q.y), tl = h2_float2(sc < 4 ? q.z : q.w);
      const float bi = binv[row * 32 + ipos];
      m.x += fmaf(tl.x, itail, hd.x) * bi;
      m.y -= fmaf(tl.y, itail, hd.y) * bi;
    }
    const float v[4] = {m.x, -m.y, m.y, m.x};
    unsigned char* blk = btab + (int64_t)f * HADC_BBYTES + ipos * 2048;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t off = hadc_boff(2 * tc + (j >> 1), hadc_col(2 * sc + (j & 1)));
      uint32_t h, t;
      tf32_split(v[j], h, t);
      *reinterpret_cast<uint32_t*>(blk + off) = h;
      *reinterpret_cast<uint32_t*>(blk + 1024 + off) = t;
    }
  }
}
// a bounded wait whose outcome every lane of the warp shares
__device__ __forceinline__ bool hadc_wait(uint32_t mbar, uint32_t parity) {
  return __all_sync(0xffffffffu, tc5::mbar_wait(mbar, parity, HADC_WAIT));
}

template <bool SCREENED>
__global__ void __launch_bounds__(HADC_NT, 2)
    k_hadamard_dc(const unsigned char* __restrict__ btab, const SplitC* __restrict__ in, float2* __restrict__ out,
                  const SplitHead* __restrict__ head, const uint8_t* __restrict__ win, const uint32_t* __restrict__ tab,
                  int ld, const int* __restrict__ rows, int nsrc, int ntrg, int nfreq, int* __restrict__ status) {
  using namespace tc5;
  extern __shared__ __align__(16) unsigned char smem_raw[];  // B blocks of the current frequency, gather ring
  __shared__ __align__(8) uint64_t mbar[2 * HADC_S + 2];       // full[S], done[S], B half 0, B half 1
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const uint32_t sB = smem_u32(smem_raw);
  const uint32_t full0 = smem_u32(&mbar[0]), done0 = smem_u32(&mbar[HADC_S]), barB0 = smem_u32(&mbar[2 * HADC_S]);
  if (wid == 0) {
    tmem_alloc(smem_u32(&tmem_base), HADC_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int s = 0; s < HADC_S; s++) {
      mbar_init(full0 + 8 * s, 4);
      mbar_init(done0 + 8 * s, 1);
    }
    mbar_init(barB0, 1);
    mbar_init(barB0 + 8, 1);
    fence_mbar_init();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
  const int fbeg = blockIdx.y * HADC_FPB, nf = min(HADC_FPB, nfreq - fbeg);
  const int G = 26 * nf;  // positions in this CTA's stream
  bool ok = true;
  if (wid == 4) {
    // ---------------- MMA warp
    // B in two halves (positions 0-12, 13-25), each refilled for the next frequency as soon as the MMAs
    // that read it have completed: half 0 once position 12 is done (checked before position 12 + S, which
    // reuses its stage), half 1 once position 25 is done (checked before the next frequency's position
    // S - 1); frequency fi waits for half h on phase fi & 1 of its barrier.
    constexpr uint32_t IDESC = idesc_tf32(128, 16);
    constexpr uint32_t HB = HADC_BBYTES / 2;
    static_assert(HADC_S <= 13 && HB % 16 == 0, "B halves");
    auto load_half = [&](int h, int fi) {
      if (elect_one()) {
        mbar_arrive_expect_tx(barB0 + 8 * h, HB);
        bulk_g2s(sB + h * HB, btab + (int64_t)(fbeg + fi) * HADC_BBYTES + h * HB, HB, barB0 + 8 * h);
      }
      __syncwarp();
    };
    load_half(0, 0);
    load_half(1, 0);
    int issued = 0;
    for (int gi = 0; gi < G && ok; gi++) {
      const int fi = gi / 26, p = gi - 26 * fi, s = gi % HADC_S;
      if (gi >= HADC_S && (p == 12 + HADC_S || p == HADC_S - 1)) {
        // the MMAs of position gi - S (12, or the previous frequency's 25) and all before it are done:
        // the half they read takes the next frequency's blocks
        ok = hadc_wait(done0 + 8 * s, ((gi - HADC_S) / HADC_S) & 1);
        if (!ok) break;
        if (p == 12 + HADC_S && fi + 1 < nf) load_half(0, fi + 1);
        if (p == HADC_S - 1) load_half(1, fi);
      }
      if (p == 0 || p == 13) {
        ok = hadc_wait(barB0 + 8 * (p == 13), fi & 1);
        if (!ok) break;
      }
      ok = hadc_wait(full0 + 8 * s, (gi / HADC_S) & 1);
      if (!ok) break;
      fence_after_sync();
      if (elect_one()) {
        const uint32_t dd = tm + HADC_DCOL + 16 * s, aa = tm + 32 * s, bb = sB + p * 2048;
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
          const uint64_t bh = sdesc_nosw(bb + 512 * kk, 256, 128), bt = sdesc_nosw(bb + 1024 + 512 * kk, 256, 128);
          mma_tf32_ts(dd, aa + 16 + 8 * kk, bh, IDESC, kk);  // fresh sums at the first step
          mma_tf32_ts(dd, aa + 8 * kk, bt, IDESC, 1);
          mma_tf32_ts(dd, aa + 8 * kk, bh, IDESC, 1);
        }
        commit(done0 + 8 * s);
      }
      __syncwarp();
      issued = gi + 1;
    }
    // on an early end, the MMAs in flight get a bounded time to finish before the TMEM is released
    if (!ok && issued > 0) hadc_wait(done0 + 8 * ((issued - 1) % HADC_S), ((issued - 1) / HADC_S) & 1);
  } else {
    // ---------------- producer / consumer warps (lane quarter wid)
    const int g = lane >> 2, q = lane & 3;
    const int k = blockIdx.x * 128 + tid;  // this lane's target slot = TMEM lane tid
    const uint32_t tw = tm + ((uint32_t)(wid * 32) << 16);
    const int row = rows[k];
    const int x0 = SCREENED ? head->e0 : 0;
    auto row_of = [](uint32_t e) { return (int64_t)(SCREENED ? e : e & SPLIT_ROW_MASK); };
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; i++) acc[i] = 0.f;
    auto inf_of = [&](int gi) {
      return reinterpret_cast<const uint4*>(in + (int64_t)(fbeg + gi / 26) * nsrc * 8);
    };
    auto take = [&](int gp, int s) {  // products of stream position gp (stage s) into the sums
      fence_after_sync();
      uint32_t d[16];
      ld_32x32b_x16(tw + HADC_DCOL + 16 * s, d);
      wait_ld();
#pragma unroll
      for (int i = 0; i < 16; i++) acc[i] += __uint_as_float(d[i]);
      if (gp % 26 == 25) {  // a frequency's last position: its rows are complete
        if (row >= 0) {
          float4* o = reinterpret_cast<float4*>(out + ((int64_t)(fbeg + gp / 26) * ntrg + row) * 8);
#pragma unroll
          for (int i = 0; i < 4; i++) o[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
        }
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = 0.f;
      }
    };
    // gather ring: slot r holds, per warp and lane, the lane's 4 spectrum pieces (rows g + 8 i) of one
    // position; each lane reads back only what it copied itself
    const uint32_t ring = sB + HADC_BBYTES + (uint32_t)((wid * 4) * 32 + lane) * 16;
    auto gather = [&](int gi, uint32_t ent) {  // cp.async of position gi into its slot (one commit group)
      const uint4* inf = inf_of(gi);
      const uint32_t slot = ring + (uint32_t)(gi % HADC_R) * (128 * 64);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t e = __shfl_sync(0xffffffffu, ent, g + 8 * i);
        cp_async16(slot + i * 32 * 16,
                   e != SPLIT_NONE ? (const void*)(inf + row_of(e) * 4 + q) : (const void*)in,
                   e != SPLIT_NONE ? 16u : 0u);
      }
      cp_async_commit();
    };
    // positions 0 .. D-1 in flight, the index of position D ready
#pragma unroll
    for (int i = 0; i < HADC_D; i++) {
      if (i < G) gather(i, tab[(i % 26) * ld + k]);
      else cp_async_commit();
    }
    uint32_t idxn = HADC_D < G ? tab[(HADC_D % 26) * ld + k] : SPLIT_NONE;
    for (int gi = 0; gi < G && ok; gi++) {
      const int s = gi % HADC_S;
      if (gi + HADC_D < G) gather(gi + HADC_D, idxn);
      else cp_async_commit();  // keep one group per position
      if (gi + HADC_D + 1 < G) idxn = tab[((gi + HADC_D + 1) % 26) * ld + k];
      cp_async_wait<HADC_D>();  // position gi's group has landed
      float4 x[4];
      {
        const uint32_t entg = tab[(gi % 26) * ld + k];
        const uint4* sl = reinterpret_cast<const uint4*>(smem_raw + HADC_BBYTES + (size_t)(gi % HADC_R) * (128 * 64)) +
                           (wid * 4) * 32 + lane;
#pragma unroll
        for (int i = 0; i < 4; i++) {  // head + tail, exponents undone: children 2 q and 2 q + 1
          const uint4 v = sl[i * 32];
          const uint32_t e = __shfl_sync(0xffffffffu, entg, g + 8 * i);
          const float2 h0 = h2_float2(v.x), t0 = h2_float2(v.y), h1 = h2_float2(v.z), t1 = h2_float2(v.w);
          if constexpr (SCREENED) {
            uchar2 cw = make_uchar2(0, 0);
            if (e != SPLIT_NONE) cw = reinterpret_cast<const uchar2*>(win)[row_of(e) * 4 + q];
            const float s0 = pow2f(-split_exp(x0, cw.x)), s1 = pow2f(-split_exp(x0, cw.y));
            constexpr float it = 1.f / SPLIT_TAIL;
            x[i] = make_float4(fmaf(t0.x, it, h0.x) * s0, fmaf(t0.y, it, h0.y) * s0, fmaf(t1.x, it, h1.x) * s1,
                               fmaf(t1.y, it, h1.y) * s1);
          } else {
            const float sc = split_inv(e);
            x[i] = make_float4((h0.x + t0.x) * sc, (h0.y + t0.y) * sc, (h1.x + t1.x) * sc, (h1.y + t1.y) * sc);
          }
        }
      }
      if (gi >= HADC_S) {  // the stage's previous position is done: take its products, then reuse it
        ok = hadc_wait(done0 + 8 * s, ((gi - HADC_S) / HADC_S) & 1);
        if (!ok) break;
        take(gi - HADC_S, s);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {  // rows 16 h + g (x[2h]) and 16 h + g + 8 (x[2h + 1]) of the warp
        const float4 a = x[2 * h], b = x[2 * h + 1];
        const float xs[8] = {a.x, a.y, b.x, b.y, a.z, a.w, b.z, b.w};
        uint32_t ah[8], at[8];
#pragma unroll
        for (int i = 0; i < 8; i++) tf32_split(xs[i], ah[i], at[i]);
        const uint32_t ta = tw + ((uint32_t)(16 * h) << 16) + 32 * s;
        st_16x256b_x2(ta, ah);
        st_16x256b_x2(ta + 16, at);
      }
      wait_st();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(full0 + 8 * s);
    }
    cp_async_wait<0>();
    for (int gp = max(G - HADC_S, 0); gp < G && ok; gp++) {  // the last positions' products
      const int s = gp % HADC_S;
      ok = hadc_wait(done0 + 8 * s, (gp / HADC_S) & 1);
      if (!ok) break;
      take(gp, s);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (wid == 0) {
    fence_after_sync();
    tmem_dealloc(tm, HADC_TMEM_COLS);
  }
  if (!ok && lane == 0) atomicExch(status, 1);
}

// ---------------------------------------------------------------- M2L transforms of the real kernels
// The convolution grid of one child is n1^3 (n1 = 2p), index a + b n1 + c n1^2 (a fastest).  The upward
// equivalent values occupy the corner [0, p)^3 (geometry.h:101-134, up), the downward check values are
// read from the corner [p, 2p)^3 (down).  The forward transform is the real-to-half-complex DFT of the
// grid (factor e^{-2 pi i k n / n1}, unnormalised, frequency f = (kc n1 + kb)(p + 1) + ka), the backward
// one the half-complex-to-real DFT (factor e^{+...}, unnormalised): the transforms of the reference's
// FFTW plans (fmm_scale_invariant.h:560-646).  Because only a p^3 corner of each input is non-zero and
// only a p^3 corner of each output is used, both are computed as three passes of direct sums, one axis
// at a time, in shared memory: no grid is materialised, and each spectrum value is written once by
// the forward transform (k_m2l_fwd_r, below) and read once by the backward one (k_m2l_bwd_r below; FP64:
// k_m2l_bwd here), in the Hadamard product's [frequency][node][child] layout.  A CTA handles FtCpb(R)
// children of one node: their spectrum values of one frequency are contiguous.  The expansion order P
// is a template parameter (2 <= P <= FT_PMAX), so every loop unrolls; k_m2l_bwd keeps each DFT factor
// w^(jk mod n1) in a register chosen at compile time.
constexpr int FT_NT = 256;
constexpr int FT_PMAX = 10;
template <class R> struct FtCpb;
template <> struct FtCpb<float> { static constexpr int v = 8; };   // 64-byte chunks of float2
template <> struct FtCpb<double> { static constexpr int v = 4; };  // 64-byte chunks of double2
template <class R> struct FtMinB;  // k_m2l_bwd (FP64 only)
template <> struct FtMinB<double> { static constexpr int v = 1; };

// calls fn(std::integral_constant<int, p>) for 2 <= p <= FT_PMAX
template <class F>
void ft_dispatch(int p, F&& fn) {
  switch (p) {
    case 2: fn(std::integral_constant<int, 2>()); break;
    case 3: fn(std::integral_constant<int, 3>()); break;
    case 4: fn(std::integral_constant<int, 4>()); break;
    case 5: fn(std::integral_constant<int, 5>()); break;
    case 6: fn(std::integral_constant<int, 6>()); break;
    case 7: fn(std::integral_constant<int, 7>()); break;
    case 8: fn(std::integral_constant<int, 8>()); break;
    case 9: fn(std::integral_constant<int, 9>()); break;
    case 10: fn(std::integral_constant<int, 10>()); break;
    default: throw Error(XFMM_ERR_UNSUPPORTED, "M2L transform kernels cover 2 <= p <= 10");
  }
}

template <class R>
size_t ft_fwd_smem(int p) {  // k_m2l_bwd's shared memory: [CPB][p][n1][H] + [CPB][p][p][H] complex values
  const int n1 = 2 * p, h = p + 1, cpb = FtCpb<R>::v;
  return sizeof(typename C2<R>::type) * ((size_t)cpb * p * p * h + (size_t)cpb * p * n1 * h);
}
template <class R>
size_t ft_bwd_smem(int p) { return ft_fwd_smem<R>(p); }

// Spectrum values as the forward transforms store them and the Hadamard reads them: split FP16 pairs (mixed),
// double2 (FP64).
template <class R> struct Spec;
template <> struct Spec<float> {
  using type = SplitC;
  static __device__ __forceinline__ type make(float2 v, float scale, float c) {
    return split16(v.x * scale, v.y * scale, c);
  }
};
template <> struct Spec<double> {
  using type = double2;
  static __device__ __forceinline__ type make(double2 v, float, float) { return v; }
};
__device__ __forceinline__ float abs1(float v) { return fabsf(v); }
__device__ __forceinline__ float abs1(float2 v) { return fabsf(v.x) + fabsf(v.y); }
// Screened kernels: the bound of every source's children (at child0[src[s]] + 0 .. 7).  Warp per child; the block
// that finishes last sets the group's e0 from the largest.  A pass of its own over the sources' densities, since
// the exponents of all sources stand on it (Yukawa sphere 300k: the forward stage 0.62 ms; with the bounds taken in the
// transform and k_tile_codes after it 0.61).
template <class W>
__global__ void __launch_bounds__(256)
    k_source_bounds(const int* __restrict__ src, int ns, const int* __restrict__ child0, const W* __restrict__ up,
                    int nsurf, float* __restrict__ bound, SplitHead* head) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float b = 0.f;
  for (int64_t e = blockIdx.x * 8ll + wid; e < 8ll * ns; e += gridDim.x * 8ll) {
    const W* u = up + ((int64_t)child0[src[e >> 3]] + (e & 7)) * nsurf;
    float m = 0.f;
    for (int k = lane; k < nsurf; k += 32) m += abs1(__ldg(u + k));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    if (lane == 0) bound[e] = m;
    b = fmaxf(b, m);
  }
  __shared__ float red[8];
  if (lane == 0) red[wid] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; k++) b = fmaxf(b, red[k]);
    atomicMax(&head->gmax, __float_as_uint(b));
    __threadfence();
    if (atomicAdd(&head->done, 1u) == gridDim.x - 1) {
      head->e0 = split_exp0(__uint_as_float(atomicExch(&head->gmax, 0u)));
      head->mask = 1u;
      head->done = 0u;
    }
  }
}
// the window of child r (8 source + child), recorded on request, and its scale
__device__ __forceinline__ float child_scale(const SplitOut& so, int64_t r, bool record) {
  const int e0 = so.head->e0, w = split_window(so.bound[r], e0);
  if (record) {
    so.win[r] = (uint8_t)w;
    if (w > 0) atomicOr(&so.head->mask, 1u << w);
  }
  return pow2f(split_exp(e0, w));
}
// The scale of every child of source node s (children at node0 .. node0 + 7) to csc, ready after the caller's
// next barrier; returns the tails' c.  red: 8 floats of shared memory.  Called by a whole CTA of 256 threads.  Not
// screened: one scale from the bound of the strongest child (one warp per child), and the node's code.
template <class W>
__device__ __forceinline__ float source_scales(const W* __restrict__ up, int64_t node0, int nsurf, float* red, float* csc,
                                               const SplitOut& so, int64_t s) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (so.head) {
    if (threadIdx.x < 8) csc[lane] = child_scale(so, 8 * s + lane, true);
    return SPLIT_TAIL;
  }
  const W* u = up + (node0 + wid) * nsurf;
  float m = 0.f;
  for (int k = lane; k < nsurf; k += 32) m += abs1(__ldg(u + k));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
  if (lane == 0) red[wid] = m;
  __syncthreads();
  if (threadIdx.x < 8) {
    float b = red[0];
#pragma unroll
    for (int c = 1; c < 8; c++) b = fmaxf(b, red[c]);
    const int code = split_code(b);
    csc[lane] = split_scale(code);
    if (lane == 0) so.code[s] = code | (b == 0.f ? SPLIT_ZERO : 0);
  }
  return 1.f;
}
// DFT factors as compile-time constants: where the loops unroll, an index (j k mod N) is known to the compiler and the
// factor becomes an operand of the multiply-add instead of a shared-memory load or a register.  cos and
// sin of 2 pi j / N by their Taylor series on the first octant (|x| <= pi / 4: the last term is below
// 1e-20) and the octant symmetries, so that 0 and 1 are exact.  The transforms' passes had two loads of
// factors for every eight multiply-adds on a busy L1 pipe (67% at p = 10); forward / backward before -> after (ms):
// 1M, p = 10 0.60 / 0.78 -> 0.51 / 0.69; Yukawa sphere 300k 0.74 / 1.00 -> 0.62 / 0.88; FP64 forward, 1M,
// p = 8 0.65 -> 0.51.
constexpr double CX_PI = 3.14159265358979323846264338327950288;
constexpr double cx_series(double x, int first) {  // first 0: cos, 1: sin
  double term = first ? x : 1.0, sum = term;
  for (int k = first + 1; k < 24; k += 2) {
    term *= -x * x / (k * (k + 1));
    sum += term;
  }
  return sum;
}
template <int N>
struct Twiddles {  // N even
  double c[N], s[N];
  constexpr Twiddles() : c{}, s{} {
    for (int j = 0; j < N; j++) {
      // the quarter turn of an N not divisible by 4 is no multiple of the step: fold to j <= N / 4 by hand
      const int h = j <= N / 2 ? j : N - j;              // cos(2 pi j / N) = cos(2 pi h / N), h <= N / 2
      const int q = 4 * h <= N ? h : N / 2 - h;          // = -cos(2 pi (N / 2 - h) / N) beyond the quarter
      const double x = 2.0 * CX_PI * q / N, y = 2.0 * CX_PI * (N - 4 * q) / (4.0 * N);  // q's angle, pi / 2 - it
      const double cc = 4 * q == N ? 0.0 : 8 * q <= N ? cx_series(x, 0) : cx_series(y, 1);
      const double ss = 4 * q == N ? 1.0 : 8 * q <= N ? cx_series(x, 1) : cx_series(y, 0);
      c[j] = 4 * h <= N ? cc : -cc;
      s[j] = j <= N / 2 ? ss : -ss;
    }
  }
};
// w[j] = e^{SIGN 2 pi i j / N}
template <class CT, int N, int SIGN>
struct ConstW {
  __device__ __forceinline__ CT operator[](int j) const {
    constexpr Twiddles<N> T{};
    using R = decltype(CT{}.x);
    return CT{(R)T.c[j], (R)(SIGN * T.s[j])};
  }
};
// acc += a w for a constant w: its zero components cost nothing
template <class CT>
__device__ __forceinline__ void wfma(CT& acc, const CT& a, const CT& w) {
  if (w.x != 0) {
    acc.x = fma(a.x, w.x, acc.x);
    acc.y = fma(a.y, w.x, acc.y);
  }
  if (w.y != 0) {
    acc.x = fma(-a.y, w.y, acc.x);
    acc.y = fma(a.x, w.y, acc.y);
  }
}

// The cuFFT path (orders beyond the DFT kernels): each source's exponent code or windows ...
template <class W>
__global__ void __launch_bounds__(256)
    k_source_codes(const int* __restrict__ src, const int* __restrict__ child0, const W* __restrict__ up, int nsurf,
                   SplitOut so) {
  __shared__ float red[8], csc[8];
  source_scales(up, (int64_t)child0[src[blockIdx.x]], nsurf, red, csc, so, blockIdx.x);
}
// ... and its spectra, rows (source, child) x nfreq, into the split layout [f][source][child]
__global__ void k_transpose_split(const float2* __restrict__ in, SplitC* __restrict__ out, int ns, int nfreq,
                                  SplitOut so) {
  __shared__ float2 tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, c0 = (int64_t)blockIdx.x * 32, nr = (int64_t)ns * 8;
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t r = r0 + i, c = c0 + threadIdx.x;
    if (r < nr && c < nfreq) tile[i][threadIdx.x] = in[r * nfreq + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t c = c0 + i, r = r0 + threadIdx.x;
    if (r >= nr || c >= nfreq) continue;
    const float sc = so.head ? child_scale(so, r, false) : split_scale(so.code[r >> 3] & 0x7f);
    const float2 v = tile[threadIdx.x][i];
    out[c * nr + r] = split16(v.x * sc, v.y * sc, so.head ? SPLIT_TAIL : 1.f);
  }
}

// dn[child of target trg[t]][k] += scale[t] * backward DFT of spec[.][t][child] at map_dn[k]
template <class R, int P>
__global__ void __launch_bounds__(FT_NT, FtMinB<R>::v)
    k_m2l_bwd(const int* __restrict__ trg, int nt, const int* __restrict__ child0,
              const typename C2<R>::type* __restrict__ spec, int nsurf, const int* __restrict__ map_dn,
              const double* __restrict__ tw, const R* __restrict__ scale, R* __restrict__ dn) {
  using CT = typename C2<R>::type;
  constexpr int CPB = FtCpb<R>::v, N = 2 * P, H = P + 1, NC = N * H;
  const int t = blockIdx.x, ch0 = blockIdx.y * CPB, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* sZ1 = reinterpret_cast<CT*>(smem_raw);  // [CPB][c' < P][kb < N][ka < H]
  CT* sZ2 = sZ1 + CPB * P * NC;               // [CPB][c' < P][b' < P][ka < H]
  __shared__ CT sw[2 * FT_PMAX];
  CT w[N];  // in registers: as constants the FP64 factors came slower (1M, p = 8: 0.78 against 0.86 ms)
#pragma unroll
  for (int m = 0; m < N; m++) w[m] = CT{(R)tw[2 * m], (R)tw[2 * m + 1]};
  if (tid < N) sw[tid] = CT{(R)tw[2 * tid], (R)tw[2 * tid + 1]};
  // pass A, along kc, to the outputs c = P + c', one column (ch, kb, ka) per task.  With kc = k + P j
  // (j = 0, 1): w^{(k + P j) m} = (-1)^{j m} w^{k m}, so output m = P + c' is the P-term sum over k of
  // (v[k] + v[k + P]) w^{k m} for even m and (v[k] - v[k + P]) w^{k m} for odd m.
  for (int e = tid; e < NC * CPB; e += FT_NT) {
    const int ch = e % CPB, col = e / CPB;
    const CT* y = spec + ((int64_t)col * nt + t) * 8 + ch0 + ch;
    const int64_t fstride = (int64_t)NC * nt * 8;
    CT up[P], um[P];
#pragma unroll
    for (int k = 0; k < P; k++) {
      const CT a = y[k * fstride], b = y[(k + P) * fstride];
      up[k] = CT{a.x + b.x, a.y + b.y};
      um[k] = CT{a.x - b.x, a.y - b.y};
    }
#pragma unroll
    for (int cc = 0; cc < P; cc++) {
      const bool odd = (P + cc) & 1;
      CT acc = odd ? um[0] : up[0];
#pragma unroll
      for (int k = 1; k < P; k++) vfma(acc, odd ? um[k] : up[k], w[(k * (P + cc)) % N]);
      sZ1[(ch * P + cc) * NC + col] = acc;
    }
  }
  __syncthreads();
  // pass B, along kb, to the outputs b = P + b', one column (ch, c', ka) per task
  for (int e = tid; e < CPB * P * H; e += FT_NT) {  // same pairing of kb and kb + P as pass A
    const int ka = e % H, cc = e / H;
    CT up[P], um[P];
#pragma unroll
    for (int k = 0; k < P; k++) {
      const CT a = sZ1[(cc * N + k) * H + ka], b = sZ1[(cc * N + k + P) * H + ka];
      up[k] = CT{a.x + b.x, a.y + b.y};
      um[k] = CT{a.x - b.x, a.y - b.y};
    }
#pragma unroll
    for (int bb = 0; bb < P; bb++) {
      const bool odd = (P + bb) & 1;
      CT acc = odd ? um[0] : up[0];
#pragma unroll
      for (int k = 1; k < P; k++) vfma(acc, odd ? um[k] : up[k], w[(k * (P + bb)) % N]);
      sZ2[(cc * P + bb) * H + ka] = acc;
    }
  }
  __syncthreads();
  // pass C, along ka (half-complex to real: weight 2 except at ka = 0 and ka = N/2), at the check points;
  // the factor index (ka a mod N) depends on the point, so the factors are read from shared memory
  const int64_t node0 = (int64_t)child0[trg[t]] + ch0;
  const R sc = scale[t];
  for (int e = tid; e < CPB * nsurf; e += FT_NT) {
    const int ch = e / nsurf, k = e - ch * nsurf, g = map_dn[k];
    const int a = g % N, b = g / N % N - P, c = g / (N * N) - P;
    const CT* z = sZ2 + ((ch * P + c) * P + b) * H;
    R y = z[0].x;
    for (int ka = 1, m = a; ka < H; ka++) {
      const R wgt = 2 * ka == N ? (R)1 : (R)2;
      const CT ww = sw[m];
      y += wgt * (z[ka].x * ww.x - z[ka].y * ww.y);
      m += a;
      if (m >= N) m -= N;
    }
    R* d = dn + (node0 + ch) * nsurf + k;
    *d += sc * y;
  }
}

// ---------------------------------------------------------------- M2L transforms of the complex kernel
// The Helmholtz kernel's transforms are full complex DFTs of the n1^3 grid (forward factor
// e^{-2 pi i k n / n1}, backward e^{+...}, both unnormalised; frequency f = (kc n1 + kb) n1 + ka): the
// C2C transforms of the reference's FFTW plans (fmm.h:631-788).  They are pruned as the real ones are
// (input corner [0, p)^3, output corner [p, 2p)^3; three passes of direct sums in shared memory, outputs
// k and k + p of a length-p input from even and odd partial sums).
constexpr int FTC_PMAX = 12;
template <class F>
void ftc_dispatch(int p, F&& fn) {
  switch (p) {
    case 2: fn(std::integral_constant<int, 2>()); break;
    case 3: fn(std::integral_constant<int, 3>()); break;
    case 4: fn(std::integral_constant<int, 4>()); break;
    case 5: fn(std::integral_constant<int, 5>()); break;
    case 6: fn(std::integral_constant<int, 6>()); break;
    case 7: fn(std::integral_constant<int, 7>()); break;
    case 8: fn(std::integral_constant<int, 8>()); break;
    case 9: fn(std::integral_constant<int, 9>()); break;
    case 10: fn(std::integral_constant<int, 10>()); break;
    case 11: fn(std::integral_constant<int, 11>()); break;
    case 12: fn(std::integral_constant<int, 12>()); break;
    default: throw Error(XFMM_ERR_UNSUPPORTED, "complex M2L transform kernels cover 2 <= p <= 12");
  }
}
// y[k] for k < 2P from x[0..P): y[k] = sum_m x[m] w^{k m}, w[j] = e^{sign 2 pi i j / 2P}; outputs k and
// k + P are even + odd and even - odd (w^{(k + P) m} = (-1)^m w^{k m}); out(k, value) stores one output
template <int P, class CT, class WT, class Out>
__device__ __forceinline__ void ftc_dft_p(const CT (&x)[P], const WT& w, Out&& out) {
  constexpr int N = 2 * P;
#pragma unroll
  for (int k = 0; k < P; k++) {
    CT ev = x[0], od{};
#pragma unroll
    for (int m = 2; m < P; m += 2) wfma(ev, x[m], w[(k * m) % N]);
#pragma unroll
    for (int m = 1; m < P; m += 2) wfma(od, x[m], w[(k * m) % N]);
    out(k, CT{ev.x + od.x, ev.y + od.y});
    out(k + P, CT{ev.x - od.x, ev.y - od.y});
  }
}
// y[P + j] for j < P from X[0..2P): y[P + j] = sum_k X[k] w^{k (P + j)}; with k = k' + P i,
// w^{(k' + P i)(P + j)} = (-1)^{i (P + j)} w^{k' (P + j)}: a P-term sum of X[k'] +- X[k' + P]
template <int P, class CT, class WT, class Out>
__device__ __forceinline__ void ftc_idft_upper(const CT (&up)[P], const CT (&um)[P], const WT& w, Out&& out) {
  constexpr int N = 2 * P;
#pragma unroll
  for (int j = 0; j < P; j++) {
    const bool odd = (P + j) & 1;
    CT acc = odd ? um[0] : up[0];
#pragma unroll
    for (int k = 1; k < P; k++) wfma(acc, odd ? um[k] : up[k], w[(k * (P + j)) % N]);
    out(j, acc);
  }
}

// Children per CTA of the complex forward transform: the spectrum values of one frequency of all 8
// children of a node are one 64-byte (float2) or 128-byte (double2) row, written by consecutive lanes.
template <class R> struct FtcCpb;
template <> struct FtcCpb<float> { static constexpr int v = 8; };
template <> struct FtcCpb<double> { static constexpr int v = 4; };
#ifndef XFMM_FTC_JS
#define XFMM_FTC_JS 3
#endif
constexpr int FTC_JS = XFMM_FTC_JS;  // first-axis base frequencies j per slab: outputs ka = j and j + p
#ifndef XFMM_FTC_FWD_MINB
#define XFMM_FTC_FWD_MINB 1  // FP32: resident CTAs per SM the forward transform's registers are set for
#endif
template <class R> struct FtcFwdMinB { static constexpr int v = sizeof(R) == 4 ? XFMM_FTC_FWD_MINB : 1; };
template <class R>
size_t ftc_fwd_smem(int p) {  // per child and slab: [p][p][2 JS] + [p][n1][2 JS] complex values
  return sizeof(typename C2<R>::type) * FtcCpb<R>::v * (size_t)p * (p + 2 * p) * 2 * FTC_JS;
}
#ifndef XFMM_FTC_JSB
#define XFMM_FTC_JSB 2
#endif
constexpr int FTC_JSB = XFMM_FTC_JSB;  // base frequencies per slab of the backward transform
// per CTA: [p][n1][CPB][2 JSB] + [p][p] rows of CPB 2 JSB + 1 (odd: the point-indexed reads of pass C
// fall on different banks) complex values
template <class R>
size_t ftc_bwd_smem(int p) {
  constexpr int ZS = FtcCpb<R>::v * 2 * FTC_JSB;
  return sizeof(typename C2<R>::type) * ((size_t)p * 2 * p * ZS + (size_t)p * p * (ZS + 1));
}

// spec[(f*ns + s)*8 + child] = forward complex DFT of the children ch0 .. ch0 + CPB - 1 of source node
// src[s].  The first-axis frequencies ka are taken in slabs (base frequencies j0 .. j0 + JS - 1 and their
// partners j + p); per slab the three passes run on the slab's columns only, and the grid input is read
// through the grid -> surface map (values outside the surface are zero) from the L1-resident rows of up.
template <class R, int P>
__global__ void __launch_bounds__(FT_NT, FtcFwdMinB<R>::v)
    k_m2l_fwd_c(const int* __restrict__ src, int ns, const int* __restrict__ child0,
                const typename C2<R>::type* __restrict__ up, int nsurf, const int* __restrict__ conv2surf,
                const double* __restrict__ tw, typename Spec<R>::type* __restrict__ spec, SplitOut so) {
  using CT = typename C2<R>::type;
  constexpr int N = 2 * P, CPB = FtcCpb<R>::v, KS = 2 * FTC_JS;
  const int s = blockIdx.x, ch0 = blockIdx.y * CPB, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* sA = reinterpret_cast<CT*>(smem_raw);  // [c < P][b < P][ch][slot < KS]
  CT* sB = sA + P * P * CPB * KS;            // [c < P][kb < N][ch][slot]
  __shared__ int sidx[P * P * P];            // grid corner [c][b][a] -> surface index or -1
  __shared__ CT sw[N];                       // w[m] = e^{-2 pi i m / N}: the same factor in every lane
  if (tid < N) sw[tid] = CT{(R)tw[2 * tid], (R)(-tw[2 * tid + 1])};
  for (int e = tid; e < P * P * P; e += FT_NT) {
    const int a = e % P, b = (e / P) % P, c = e / (P * P);
    sidx[e] = conv2surf[(c * N + b) * N + a];
  }
  const int64_t node0 = (int64_t)child0[src[s]] + ch0;
  __shared__ float csc[8];  // the children's power-of-two scales (mixed)
  float tail = 1.f;
  if constexpr (sizeof(R) == 4) {
    __shared__ float red[8];
    tail = source_scales(up, node0, nsurf, red, csc, so, s);
  }
  const int64_t fstride = (int64_t)N * N * ns * 8;
  for (int j0 = 0; j0 < P; j0 += FTC_JS) {
    __syncthreads();  // sidx and sw ready; the previous slab's sA / sB reads done
    // pass 1, along a: task (c, b, ch); slots 2 q and 2 q + 1 hold ka = j0 + q and j0 + q + P
    for (int e = tid; e < P * P * CPB; e += FT_NT) {
      const int ch = e % CPB, cb = e / CPB;
      const CT* u = up + (node0 + ch) * nsurf;
      CT x[P];
#pragma unroll
      for (int a = 0; a < P; a++) {
        const int k = sidx[cb * P + a];
        x[a] = k >= 0 ? __ldg(u + k) : CT{(R)0, (R)0};
      }
#pragma unroll
      for (int q = 0; q < FTC_JS; q++) {
        const int j = j0 + q;
        if (j >= P) break;
        CT ev = x[0], od{(R)0, (R)0};
#pragma unroll
        for (int a = 1; a < P; a++) vfma(a & 1 ? od : ev, x[a], sw[(j * a) % N]);  // j known at run time only
        sA[(cb * CPB + ch) * KS + 2 * q] = CT{ev.x + od.x, ev.y + od.y};
        sA[(cb * CPB + ch) * KS + 2 * q + 1] = CT{ev.x - od.x, ev.y - od.y};
      }
    }
    __syncthreads();
    // pass 2, along b: task (c, ch, slot)
    for (int e = tid; e < P * CPB * KS; e += FT_NT) {
      const int sl = e % KS, ch = (e / KS) % CPB, c = e / (KS * CPB);
      CT x[P];
#pragma unroll
      for (int b = 0; b < P; b++) x[b] = sA[((c * P + b) * CPB + ch) * KS + sl];
      ftc_dft_p<P>(x, ConstW<CT, N, -1>(), [&](int kb, CT v) { sB[((c * N + kb) * CPB + ch) * KS + sl] = v; });
    }
    __syncthreads();
    // pass 3, along c: task (kb, slot, ch), children fastest: the CPB children of one frequency are
    // written by consecutive lanes
    for (int e = tid; e < N * KS * CPB; e += FT_NT) {
      const int ch = e % CPB, sl = (e / CPB) % KS, kb = e / (CPB * KS);
      const int j = j0 + sl / 2;
      if (j >= P) continue;
      const int ka = j + (sl & 1) * P;
      CT x[P];
#pragma unroll
      for (int c = 0; c < P; c++) x[c] = sB[((c * N + kb) * CPB + ch) * KS + sl];
      auto* o = spec + ((int64_t)(kb * N + ka) * ns + s) * 8 + ch0 + ch;
      ftc_dft_p<P>(x, ConstW<CT, N, -1>(), [&](int kc, CT v) { o[kc * fstride] = Spec<R>::make(v, csc[ch], tail); });
    }
  }
}

// dn[child ch0 + ch of target trg[t]][k] += scale[t] * backward complex DFT of spec[.][t][child] at map_dn[k],
// for the CPB children ch0 .. of the CTA.  The first-axis frequencies ka are taken in slabs as in the
// forward transform: per slab, pass A (along kc, rows of CPB children read by consecutive lanes) and
// pass B (along kb) run on the slab's columns, and pass C adds the slab's terms of the last sum (along
// ka) to per-point sums kept in registers (point i of the thread: k = tid + i FT_NT over CPB nsurf).
template <class R> struct FtcMinB;  // resident CTAs per SM of the backward transform (registers)
template <> struct FtcMinB<float> { static constexpr int v = 2; };
template <> struct FtcMinB<double> { static constexpr int v = 1; };
template <class R, int P>
__global__ void __launch_bounds__(FT_NT, FtcMinB<R>::v)
    k_m2l_bwd_c(const int* __restrict__ trg, int nt, const int* __restrict__ child0,
                const typename C2<R>::type* __restrict__ spec, int nsurf, const int* __restrict__ map_dn,
                const double* __restrict__ tw, const R* __restrict__ scale, typename C2<R>::type* __restrict__ dn) {
  using CT = typename C2<R>::type;
  constexpr int N = 2 * P, CPB = FtcCpb<R>::v, JS = FTC_JSB, KS = 2 * JS, ZS = CPB * KS + 1;
  constexpr int NPT = (CPB * (6 * (P - 1) * (P - 1) + 2) + FT_NT - 1) / FT_NT;  // points per thread
  const int t = blockIdx.x, ch0 = blockIdx.y * CPB, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* sZ1 = reinterpret_cast<CT*>(smem_raw);  // [c' < P][kb < N][ch][slot < KS]
  CT* sZ2 = sZ1 + P * N * CPB * KS;           // [c' < P][b' < P] rows of ZS: [ch][slot], one pad
  __shared__ CT sw[N];                        // w[m] = e^{+2 pi i m / N}, read by broadcast (passes A, B)
  if (tid < N) sw[tid] = CT{(R)tw[2 * tid], (R)tw[2 * tid + 1]};
  CT acc[NPT];
#pragma unroll
  for (int i = 0; i < NPT; i++) acc[i] = CT{(R)0, (R)0};
  const int64_t fstride = (int64_t)N * N * nt * 8;
  for (int j0 = 0; j0 < P; j0 += JS) {
    __syncthreads();  // sw ready; the previous slab's sZ2 reads done
    // pass A, along kc, to c = P + c': task (kb, slot, ch), children fastest (one row per frequency)
    for (int e = tid; e < N * KS * CPB; e += FT_NT) {
      const int ch = e % CPB, sl = (e / CPB) % KS, kb = e / (CPB * KS);
      const int j = j0 + sl / 2;
      if (j >= P) continue;
      const int ka = j + (sl & 1) * P;
      const CT* y = spec + ((int64_t)(kb * N + ka) * nt + t) * 8 + ch0 + ch;
      CT up[P], um[P];
#pragma unroll
      for (int k = 0; k < P; k++) {
        const CT a = y[k * fstride], b = y[(k + P) * fstride];
        up[k] = CT{a.x + b.x, a.y + b.y};
        um[k] = CT{a.x - b.x, a.y - b.y};
      }
      ftc_idft_upper<P>(up, um, ConstW<CT, N, 1>(), [&](int cc, CT v) { sZ1[((cc * N + kb) * CPB + ch) * KS + sl] = v; });
    }
    __syncthreads();
    // pass B, along kb, to b = P + b': task (c', ch, slot)
    for (int e = tid; e < P * CPB * KS; e += FT_NT) {
      const int sl = e % KS, ch = (e / KS) % CPB, cc = e / (KS * CPB);
      if (j0 + sl / 2 >= P) continue;
      CT up[P], um[P];
#pragma unroll
      for (int k = 0; k < P; k++) {
        const CT a = sZ1[((cc * N + k) * CPB + ch) * KS + sl], b = sZ1[((cc * N + k + P) * CPB + ch) * KS + sl];
        up[k] = CT{a.x + b.x, a.y + b.y};
        um[k] = CT{a.x - b.x, a.y - b.y};
      }
      ftc_idft_upper<P>(up, um, ConstW<CT, N, 1>(), [&](int bb, CT v) { sZ2[(cc * P + bb) * ZS + ch * KS + sl] = v; });
    }
    __syncthreads();
    // pass C, this slab's terms of the sum along ka at each point: (Z[j] + (-1)^a Z[j + P]) w^{j a}
#pragma unroll
    for (int i = 0; i < NPT; i++) {
      const int e = tid + i * FT_NT;
      if (e < CPB * nsurf) {
        const int ch = e / nsurf, k = e - ch * nsurf, g = map_dn[k];
        const int a = g % N, b = g / N % N - P, c = g / (N * N) - P;
        const CT* z = sZ2 + (c * P + b) * ZS + ch * KS;
        const R sgn = (a & 1) ? (R)-1 : (R)1;
#pragma unroll
        for (int q = 0; q < JS; q++) {
          const int jj = j0 + q;
          if (jj >= P) break;
          const CT v{z[2 * q].x + sgn * z[2 * q + 1].x, z[2 * q].y + sgn * z[2 * q + 1].y};
          vfma(acc[i], v, sw[(jj * a) % N]);
        }
      }
    }
  }
  const int64_t node0 = (int64_t)child0[trg[t]] + ch0;
  const R sc = scale[t];
#pragma unroll
  for (int i = 0; i < NPT; i++) {
    const int e = tid + i * FT_NT;
    if (e < CPB * nsurf) {
      CT* d = dn + node0 * nsurf + e;  // child ch0 + e / nsurf, point e % nsurf
      *d = CT{d->x + sc * acc[i].x, d->y + sc * acc[i].y};
    }
  }
}

// ---------------------------------------------------------------- slabbed M2L transforms of the real kernels
// The real transforms (half spectrum along the first axis, H = p + 1 frequencies ka) computed as the
// complex ones are: CPB children per CTA (one spectrum row of a frequency read or written by consecutive
// lanes), the first-axis frequencies in slabs of FTR_KS, so that a CTA needs ~37 KB of shared memory
// (p = 8) instead of 110 KB and three or more CTAs share an SM; DFT factors are read from shared memory
// (the same factor in every lane: broadcast).  The backward transform keeps each check point's running
// sum along the last axis in registers across the slabs.
#ifndef XFMM_FTR_KS
#define XFMM_FTR_KS 3
#endif
#ifndef XFMM_FTR_MINB_F
#define XFMM_FTR_MINB_F 4
#endif
constexpr int FTR_KS = XFMM_FTR_KS;
#ifndef XFMM_FTR_BWD_MINB_HI
#define XFMM_FTR_BWD_MINB_HI 3  // backward transform, p >= 9 (more per-point sums per thread; measured at p = 10)
#endif
template <class R> struct FtrMinB;
template <> struct FtrMinB<float> { static constexpr int v = XFMM_FTR_MINB_F; };
template <> struct FtrMinB<double> { static constexpr int v = 1; };
template <class R, int P> struct FtrBwdMinB {
  static constexpr int v = (sizeof(R) == 4 && P >= 9) ? XFMM_FTR_BWD_MINB_HI : FtrMinB<R>::v;
};
template <class R>
size_t ftr_fwd_smem(int p) {  // [p][p][CPB][KS] + [p][n1][CPB][KS] complex values
  return sizeof(typename C2<R>::type) * (size_t)p * 3 * p * FtCpb<R>::v * FTR_KS;
}
template <class R>
size_t ftr_bwd_smem(int p) {  // [p][n1][CPB][KS] + [p][p] rows of CPB KS + 1 complex values
  const size_t zs = (size_t)FtCpb<R>::v * FTR_KS;
  return sizeof(typename C2<R>::type) * ((size_t)p * 2 * p * zs + (size_t)p * p * (zs + 1));
}

// spec[(f*ns + s)*8 + ch0 + ch] = forward real-to-half-complex DFT of the children ch0 .. ch0 + CPB - 1 of
// source node src[s], f = (kc n1 + kb) H + ka
template <class R, int P>
__global__ void __launch_bounds__(FT_NT, FtrMinB<R>::v)
    k_m2l_fwd_r(const int* __restrict__ src, int ns, const int* __restrict__ child0, const R* __restrict__ up,
                int nsurf, const int* __restrict__ conv2surf, const double* __restrict__ tw,
                typename Spec<R>::type* __restrict__ spec, SplitOut so) {
  using CT = typename C2<R>::type;
  constexpr int N = 2 * P, H = P + 1, CPB = FtCpb<R>::v, KS = FTR_KS;
  const int s = blockIdx.x, ch0 = blockIdx.y * CPB, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* sA = reinterpret_cast<CT*>(smem_raw);  // [c < P][b < P][ch][slot < KS]
  CT* sB = sA + P * P * CPB * KS;            // [c < P][kb < N][ch][slot]
  __shared__ int sidx[P * P * P];            // grid corner [c][b][a] -> surface index or -1
  __shared__ CT sw[N];                       // w[m] = e^{-2 pi i m / N}
  if (tid < N) sw[tid] = CT{(R)tw[2 * tid], (R)(-tw[2 * tid + 1])};
  for (int e = tid; e < P * P * P; e += FT_NT) {
    const int a = e % P, b = (e / P) % P, c = e / (P * P);
    sidx[e] = conv2surf[(c * N + b) * N + a];
  }
  const int64_t node0 = (int64_t)child0[src[s]] + ch0;
  __shared__ float csc[8];  // the children's power-of-two scales (mixed)
  float tail = 1.f;
  if constexpr (sizeof(R) == 4) {
    __shared__ float red[8];
    tail = source_scales(up, node0, nsurf, red, csc, so, s);
  }
  const int64_t fstride = (int64_t)N * H * ns * 8;  // kc -> kc + 1
  for (int k0 = 0; k0 < H; k0 += KS) {
    __syncthreads();  // sidx and sw ready; the previous slab's reads done
    // pass 1, along a (real input): task (c, b, ch), slot sl = ka - k0
    for (int e = tid; e < P * P * CPB; e += FT_NT) {
      const int ch = e % CPB, cb = e / CPB;
      const R* u = up + (node0 + ch) * nsurf;
      R x[P];
#pragma unroll
      for (int a = 0; a < P; a++) {
        const int k = sidx[cb * P + a];
        x[a] = k >= 0 ? __ldg(u + k) : (R)0;
      }
#pragma unroll
      for (int sl = 0; sl < KS; sl++) {
        const int ka = k0 + sl;
        if (ka >= H) break;
        R re = x[0], im = 0;
#pragma unroll
        for (int a = 1; a < P; a++) {
          const CT ww = sw[(ka * a) % N];
          re += x[a] * ww.x;
          im += x[a] * ww.y;
        }
        sA[(cb * CPB + ch) * KS + sl] = CT{re, im};
      }
    }
    __syncthreads();
    // pass 2, along b: task (c, ch, slot)
    for (int e = tid; e < P * CPB * KS; e += FT_NT) {
      const int sl = e % KS, ch = (e / KS) % CPB, c = e / (KS * CPB);
      if (k0 + sl >= H) continue;
      CT x[P];
#pragma unroll
      for (int b = 0; b < P; b++) x[b] = sA[((c * P + b) * CPB + ch) * KS + sl];
      ftc_dft_p<P>(x, ConstW<CT, N, -1>(), [&](int kb, CT v) { sB[((c * N + kb) * CPB + ch) * KS + sl] = v; });
    }
    __syncthreads();
    // pass 3, along c: task (kb, slot, ch), children fastest
    for (int e = tid; e < N * KS * CPB; e += FT_NT) {
      const int ch = e % CPB, sl = (e / CPB) % KS, kb = e / (CPB * KS);
      const int ka = k0 + sl;
      if (ka >= H) continue;
      CT x[P];
#pragma unroll
      for (int c = 0; c < P; c++) x[c] = sB[((c * N + kb) * CPB + ch) * KS + sl];
      auto* o = spec + ((int64_t)(kb * H + ka) * ns + s) * 8 + ch0 + ch;
      ftc_dft_p<P>(x, ConstW<CT, N, -1>(), [&](int kc, CT v) { o[kc * fstride] = Spec<R>::make(v, csc[ch], tail); });
    }
  }
}

// dn[child ch0 + ch of target trg[t]][k] += scale[t] * backward half-complex-to-real DFT of spec[.][t][child]
// at map_dn[k] (weight 2 on the half spectrum's interior frequencies 0 < ka < N / 2)
template <class R, int P>
__global__ void __launch_bounds__(FT_NT, (FtrBwdMinB<R, P>::v))
    k_m2l_bwd_r(const int* __restrict__ trg, int nt, const int* __restrict__ child0,
                const typename C2<R>::type* __restrict__ spec, int nsurf, const int* __restrict__ map_dn,
                const double* __restrict__ tw, const R* __restrict__ scale, R* __restrict__ dn) {
  using CT = typename C2<R>::type;
  constexpr int N = 2 * P, H = P + 1, CPB = FtCpb<R>::v, KS = FTR_KS, ZS = CPB * KS + 1;
  constexpr int NPT = (CPB * (6 * (P - 1) * (P - 1) + 2) + FT_NT - 1) / FT_NT;  // points per thread
  const int t = blockIdx.x, ch0 = blockIdx.y * CPB, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* sZ1 = reinterpret_cast<CT*>(smem_raw);  // [c' < P][kb < N][ch][slot < KS]
  CT* sZ2 = sZ1 + P * N * CPB * KS;           // [c' < P][b' < P] rows of ZS: [ch][slot], one pad
  __shared__ CT sw[N];                        // w[m] = e^{+2 pi i m / N}
  if (tid < N) sw[tid] = CT{(R)tw[2 * tid], (R)tw[2 * tid + 1]};
  R acc[NPT];
#pragma unroll
  for (int i = 0; i < NPT; i++) acc[i] = 0;
  const int64_t fstride = (int64_t)N * H * nt * 8;
  for (int k0 = 0; k0 < H; k0 += KS) {
    __syncthreads();  // sw ready; the previous slab's sZ2 reads done
    // pass A, along kc, to c = P + c': task (kb, slot, ch), children fastest
    for (int e = tid; e < N * KS * CPB; e += FT_NT) {
      const int ch = e % CPB, sl = (e / CPB) % KS, kb = e / (CPB * KS);
      const int ka = k0 + sl;
      if (ka >= H) continue;
      const CT* y = spec + ((int64_t)(kb * H + ka) * nt + t) * 8 + ch0 + ch;
      CT up[P], um[P];
#pragma unroll
      for (int k = 0; k < P; k++) {
        const CT a = y[k * fstride], b = y[(k + P) * fstride];
        up[k] = CT{a.x + b.x, a.y + b.y};
        um[k] = CT{a.x - b.x, a.y - b.y};
      }
      ftc_idft_upper<P>(up, um, ConstW<CT, N, 1>(), [&](int cc, CT v) { sZ1[((cc * N + kb) * CPB + ch) * KS + sl] = v; });
    }
    __syncthreads();
    // pass B, along kb, to b = P + b': task (c', ch, slot)
    for (int e = tid; e < P * CPB * KS; e += FT_NT) {
      const int sl = e % KS, ch = (e / KS) % CPB, cc = e / (KS * CPB);
      if (k0 + sl >= H) continue;
      CT up[P], um[P];
#pragma unroll
      for (int k = 0; k < P; k++) {
        const CT a = sZ1[((cc * N + k) * CPB + ch) * KS + sl], b = sZ1[((cc * N + k + P) * CPB + ch) * KS + sl];
        up[k] = CT{a.x + b.x, a.y + b.y};
        um[k] = CT{a.x - b.x, a.y - b.y};
      }
      ftc_idft_upper<P>(up, um, ConstW<CT, N, 1>(), [&](int bb, CT v) { sZ2[(cc * P + bb) * ZS + ch * KS + sl] = v; });
    }
    __syncthreads();
    // pass C, this slab's terms along ka at each point: wgt Re(Z[ka] w^{ka a})
#pragma unroll
    for (int i = 0; i < NPT; i++) {
      const int e = tid + i * FT_NT;
      if (e < CPB * nsurf) {
        const int ch = e / nsurf, k = e - ch * nsurf, g = map_dn[k];
        const int a = g % N, b = g / N % N - P, c = g / (N * N) - P;
        const CT* z = sZ2 + (c * P + b) * ZS + ch * KS;
#pragma unroll
        for (int sl = 0; sl < KS; sl++) {
          const int ka = k0 + sl;
          if (ka >= H) break;
          const CT ww = sw[(ka * a) % N];
          const R wgt = (ka == 0 || 2 * ka == N) ? (R)1 : (R)2;
          acc[i] += wgt * (z[sl].x * ww.x - z[sl].y * ww.y);
        }
      }
    }
  }
  const int64_t node0 = (int64_t)child0[trg[t]] + ch0;
  const R sc = scale[t];
#pragma unroll
  for (int i = 0; i < NPT; i++) {
    const int e = tid + i * FT_NT;
    if (e < CPB * nsurf) dn[node0 * nsurf + e] += sc * acc[i];  // child ch0 + e / nsurf, point e % nsurf
  }
}

// dn[child c of target t][k] += scale[t] * grid[(t*8 + c)*nconv + map_dn[k]]   (fmm_scale_invariant.h:639-643)
template <class W, class RB>
__global__ void k_m2l_gather_dn(const int* __restrict__ trg, int ntrg, const int* __restrict__ child0,
                                const W* __restrict__ grid, int nconv, const int* __restrict__ map_dn, int nsurf,
                                const RB* __restrict__ scale, W* __restrict__ dn) {
  const int64_t total = (int64_t)ntrg * 8 * nsurf;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(e % nsurf);
    const int64_t tc = e / nsurf;
    const int t = (int)(tc >> 3), c = (int)(tc & 7);
    W* d = dn + ((int64_t)child0[trg[t]] + c) * nsurf + k;
    *d = vadd(*d, vscale(grid[tc * nconv + map_dn[k]], scale[t]));
  }
}

// ================================================================ misc
// Sources of the Laplace paired-FP32 near field: hi/lo FP32 parts of (x - o), FP32 charge.
// *bad becomes nonzero if any of v[0, n) is NaN or infinite
__global__ void k_count_nonfinite(const double* __restrict__ v, int64_t n, int* __restrict__ bad) {
  int found = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    found |= !isfinite(v[i]);
  if (__syncthreads_or(found) && threadIdx.x == 0) atomicOr(bad, 1);
}
__global__ void k_set_charges(const double* __restrict__ q, const int* __restrict__ perm, int64_t n, int cplx,
                              double4* __restrict__ src4, double* __restrict__ qim) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t j = perm[i];
  if (cplx) {
    src4[i].w = q[2 * j];
    qim[i] = q[2 * j + 1];
  } else {
    src4[i].w = q[j];
  }
}
__global__ void k_scatter_out(const double* __restrict__ in, const int* __restrict__ perm, int64_t n, int width,
                              double* __restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t j = perm[i];
  for (int c = 0; c < width; c++) out[j * width + c] = in[i * width + c];
}

}  // namespace

// ================================================================ workspace
// Rows of one batch of translation GEMMs (translate.cu): per row its A and C offsets in real elements of
// the buffers (complex values count twice) and its scale.
struct GemmRows {
  int M = 0;
  DBuf<int64_t> a, c;
  DBuf<double> al64;
};

struct Workspace {
  int precision = -1, kernel = -1, p = 0;
  size_t vsz = 0;
  DBuf<char> up, dn, chk;  // working precision
  DBuf<double> tc_scratch;  // tile counters and partial sums of the split-K translations
  DBuf<int4> close_pairs;   // Laplace mixed near field: the close pairs (k_close_scan), found once per tree
  int64_t n_close = -1;     // -1: not searched yet
  DBuf<char> ybuf, eq;     // FP64: pinv intermediate (rows of the kept singular directions), downward
                           // equivalent densities of the leaves
  DBuf<double> out;
  DBuf<int> status;   // set by a kernel whose bounded wait ran out (0: none)
  // leaves grouped by level (P2M / L2P operators are per level except for Laplace)
  std::vector<int> leaf_level_off;
  GemmRows p2m1, p2m2, l2p1, l2p2;  // two factors each (rows grouped by leaf level)
  std::vector<GemmRows> m2m, l2l;  // per level of the parent
  // M2L
  DBuf<char> grid, specA, specB;
  std::vector<cufftHandle> fwd, bwd;
  std::vector<int> had_tile0;  // first tile of each group (ngroups + 1; k_hadamard_h)
  // mixed path: tiles of k_hadamard_h (per group [had_tile0[g], had_tile0[g + 1])), their source slots,
  // tables and output rows; every source's exponent code (screened kernels: its children's bounds and windows)
  // of the last forward transform (one group at a time)
  DBuf<HadTile> hadh_tile;
  DBuf<int> hadh_slots, hadh_rows, scode;
  DBuf<float> sbound;
  DBuf<uint8_t> swin;
  DBuf<SplitHead> shead;
  DBuf<uint32_t> hadh_pslots, hadh_tpass;  // k_tile_codes
  DBuf<float> hadh_tinv;
  DBuf<uint2> hadh_tab;
  // FP64, and the dense targets of the tcgen05 form: per group a [26][ld] source table and ld output rows
  // (hadd_tabp: the table packed with the exponent codes)
  DBuf<int> hadd_tab, hadd_row;
  DBuf<uint32_t> hadd_tabp;
  std::vector<int64_t> hadd_tab0, hadd_row0;
  std::vector<int> hadd_ld;
  bool hadh_attr = false, hadc_attr = false, had64_attr = false;
  // dense Hadamard targets on tcgen05 (k_hadamard_dc) instead of mma.sync (k_hadamard_h): chosen when the
  // workspace is created, by XFMM_HADAMARD_TCGEN05=1 in the environment
  bool had_tc5 = false;
  DBuf<unsigned char> hadc_btab;      // its B blocks per frequency (k_hadc_btab), built for one operator table
  uint64_t hadc_btab_id = 0;          // LevelOps::m2l_id of that table
  // M2L transforms: own pruned DFT kernels (real p <= 10, complex p <= 12, shared memory permitting) or
  // cuFFT on the grid
  bool fused = false;
  size_t ft_fwd_smem = 0, ft_bwd_smem = 0;
  int64_t launches = 0;  // kernels of this library launched by the last evaluate
  cudaEvent_t ev[9] = {};
  std::vector<cudaEvent_t> m2l_ev;  // 4 per M2L group
  bool ev_ok = false;
  ~Workspace() {
    for (auto h : fwd) cufftDestroy(h);
    for (auto h : bwd) cufftDestroy(h);
    if (ev_ok) {
      for (auto& e : ev) cudaEventDestroy(e);
      for (auto& e : m2l_ev) cudaEventDestroy(e);
    }
  }
};

void release_workspace(Tree& t) {
  for (auto& w : t.ws) {
    delete w;
    w = nullptr;
  }
}

namespace {

template <class RB>
void upload_rows(GemmRows& g, const std::vector<int64_t>& a, const std::vector<int64_t>& c,
                 const std::vector<double>& al, cudaStream_t s) {
  g.M = (int)a.size();
  g.a.upload(a, s);
  g.c.upload(c, s);
  g.al64.upload(al, s);
}

inline const LevelOps& level_ops(const Fmm& f, int level) { return f.ops[f.kernel == XFMM_LAPLACE ? 0 : level]; }

Workspace& workspace(Fmm& f, Tree& t, cudaStream_t s) {
  Workspace*& w = t.ws[f.precision];
  if (w && w->kernel == f.kernel && w->p == f.p) return *w;
  delete w;
  w = new Workspace();
  Workspace& W = *w;
  W.precision = f.precision;
  W.kernel = f.kernel;
  W.p = f.p;
  const bool cplx = f.is_complex();
  W.vsz = (f.mixed() ? 4 : 8) * (cplx ? 2 : 1);
  const int n = f.nsurf;
  W.up.alloc((size_t)t.nnodes * n * W.vsz);
  W.dn.alloc((size_t)t.nnodes * n * W.vsz);
  W.chk.alloc((size_t)std::max(t.nleafs, 1) * n * W.vsz);
  W.ybuf.alloc((size_t)std::max(t.nleafs, 1) * n * 8 * (cplx ? 2 : 1));
  W.eq.alloc((size_t)std::max(t.nleafs, 1) * n * 8 * (cplx ? 2 : 1));
  W.out.alloc((size_t)t.ntrg * 4 * (cplx ? 2 : 1));
  W.status.alloc(1);
  {
    const char* e = std::getenv("XFMM_HADAMARD_TCGEN05");
    W.had_tc5 = e && e[0] == '1';
  }
  XCUDA(cudaMemsetAsync(W.status.p, 0, sizeof(int), s));
  // leaf rows grouped by level: P2M (chk[pos] -> up[node]) and L2P (dn[node] -> eq[pos])
  const bool lap = f.kernel == XFMM_LAPLACE;
  std::vector<int> order(t.nleafs);
  for (int i = 0; i < t.nleafs; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return t.h_level[t.h_leafs[x]] < t.h_level[t.h_leafs[y]]; });
  W.leaf_level_off.assign(t.depth + 2, 0);
  {
    std::vector<int64_t> idn, nodes;
    std::vector<double> al, one;
    int cur = 0;
    for (int l = 0; l <= t.depth; l++) {
      W.leaf_level_off[l] = cur;
      while (cur < t.nleafs && t.h_level[t.h_leafs[order[cur]]] == l) cur++;
    }
    W.leaf_level_off[t.depth + 1] = cur;
    const int64_t rn = (int64_t)n * (cplx ? 2 : 1);  // row length in real elements
    for (int i : order) {
      const int node = t.h_leafs[i];
      idn.push_back((int64_t)i * rn);
      nodes.push_back((int64_t)node * rn);
      al.push_back(lap ? std::pow(0.5, t.h_level[node]) : 1.0);
      one.push_back(1.0);
    }
    // P2M: chk[i] -U^H-> eq[i] (scratch) -V S+, 0.5^l-> up[node];  L2P: dn[node] -> chk[i] (scratch) -> eq[i]
    upload_rows<double>(W.p2m1, idn, idn, one, s);
    upload_rows<double>(W.p2m2, idn, nodes, al, s);
    upload_rows<double>(W.l2p1, nodes, idn, one, s);
    upload_rows<double>(W.l2p2, idn, idn, al, s);
  }
  W.m2m.clear();
  W.l2l.clear();
  W.m2m.resize(t.depth + 1);
  W.l2l.resize(t.depth + 1);
  for (int l = 0; l <= t.depth; l++) {
    std::vector<int64_t> ma, mc, la, lc;
    std::vector<double> one;
    for (int k : t.h_nonleafs)
      if (t.h_level[k] == l) {
        const int64_t rn = (int64_t)n * (cplx ? 2 : 1);
        ma.push_back((int64_t)t.h_child0[k] * rn);
        mc.push_back((int64_t)k * rn);
        la.push_back((int64_t)k * rn);
        lc.push_back((int64_t)t.h_child0[k] * rn);
        one.push_back(1.0);
      }
    upload_rows<double>(W.m2m[l], ma, mc, one, s);
    upload_rows<double>(W.l2l[l], la, lc, one, s);
  }
  {
    // scratch of the split-K translations (one at a time on the tree's stream), its counters zeroed once
    const int cw = cplx ? 2 : 1, lap_rows = lap ? t.nleafs : 0;
    int64_t need = 0;
    for (int l = 0; l <= t.depth; l++) {
      if (f.mixed()) {
        need = std::max(need, tgemm_tc_scratch(W.m2m[l].M, cw * n, cw * 8 * n, 1));
        need = std::max(need, tgemm_tc_scratch(W.l2l[l].M, cw * 8 * n, cw * n, 1));
      } else {
        need = std::max(need, tgemm_f64_scratch(W.m2m[l].M, cw * n, cw * 8 * n));
        need = std::max(need, tgemm_f64_scratch(W.l2l[l].M, cw * 8 * n, cw * n));
      }
      // the pseudo-inverse factors (FP64 in both precisions), between n and the kept rank
      const int m = lap ? lap_rows : W.leaf_level_off[l + 1] - W.leaf_level_off[l];
      const int rk = cw * level_ops(f, l).rank;
      need = std::max({need, tgemm_f64_scratch(m, rk, cw * n), tgemm_f64_scratch(m, cw * n, rk)});
    }
    if (need > 0) {
      W.tc_scratch.alloc((size_t)need);
      XCUDA(cudaMemsetAsync(W.tc_scratch.p, 0, W.tc_scratch.bytes(), s));
    }
  }
  // M2L buffers and FFT plans
  const int ng = (int)t.m2l_src_off.size() - 1;
  int maxn = 1;
  for (int g = 0; g < ng; g++) {
    maxn = std::max(maxn, t.m2l_src_off[g + 1] - t.m2l_src_off[g]);
    maxn = std::max(maxn, t.m2l_trg_off[g + 1] - t.m2l_trg_off[g]);
  }
  const size_t rsz = f.mixed() ? 4 : 8;  // real scalar size
  {
    constexpr size_t kMaxSmem = 227 * 1024;
    const size_t fw = f.mixed() ? ftr_fwd_smem<float>(f.p) : ftr_fwd_smem<double>(f.p);
    const size_t bw = f.mixed() ? ft_bwd_smem<float>(f.p) : ft_bwd_smem<double>(f.p);
    const size_t cw = std::max(f.mixed() ? ftc_fwd_smem<float>(f.p) : ftc_fwd_smem<double>(f.p),
                               f.mixed() ? ftc_bwd_smem<float>(f.p) : ftc_bwd_smem<double>(f.p));
    W.fused = cplx ? (f.p <= FTC_PMAX && cw <= kMaxSmem) : (f.p <= FT_PMAX && fw <= kMaxSmem && bw <= kMaxSmem);
  }
  W.specA.alloc((size_t)maxn * 8 * f.nfreq * 2 * rsz);
  W.specB.alloc((size_t)maxn * 8 * f.nfreq * 2 * rsz);
  if (f.mixed()) {
    XREQUIRE(maxn < (int)SPLIT_ROW_MASK, XFMM_ERR_UNSUPPORTED, "too many M2L sources");
    W.scode.alloc(maxn);
    if (f.kernel != XFMM_LAPLACE) {
      W.sbound.alloc((size_t)maxn * 8);
      W.swin.alloc((size_t)maxn * 8);
      W.shead.alloc(1);
      XCUDA(cudaMemsetAsync(W.shead.p, 0, W.shead.bytes(), s));
    }
  }
  int dims[3] = {f.n1, f.n1, f.n1};
  cufftType tf = cplx ? (f.mixed() ? CUFFT_C2C : CUFFT_Z2Z) : (f.mixed() ? CUFFT_R2C : CUFFT_D2Z);
  cufftType tb = cplx ? (f.mixed() ? CUFFT_C2C : CUFFT_Z2Z) : (f.mixed() ? CUFFT_C2R : CUFFT_Z2D);
  if (!W.fused) W.grid.alloc((size_t)maxn * 8 * f.nconv * rsz * (cplx ? 2 : 1));
  for (int g = 0; g < ng && !W.fused; g++) {
    const int ns = t.m2l_src_off[g + 1] - t.m2l_src_off[g], nt = t.m2l_trg_off[g + 1] - t.m2l_trg_off[g];
    cufftHandle hf = 0, hb = 0;
    if (ns > 0) {
      XCUFFT2(cufftPlanMany(&hf, 3, dims, nullptr, 1, f.nconv, nullptr, 1, f.nfreq, tf, 8 * ns));
      XCUFFT2(cufftSetStream(hf, s));
    }
    if (nt > 0) {
      XCUFFT2(cufftPlanMany(&hb, 3, dims, nullptr, 1, f.nfreq, nullptr, 1, f.nconv, tb, 8 * nt));
      XCUFFT2(cufftSetStream(hb, s));
    }
    W.fwd.push_back(hf);
    W.bwd.push_back(hb);
  }
  if (f.mixed()) {
    // Tiles of k_hadamard_h over the targets of each group, level by level (node order within a level is
    // Morton order: the targets of a tile are spatially compact and share most of their sources).  A tile
    // closes at HADH_TT targets or when a class of its source slots (the octant of the source in its
    // parent) is full.  In the tcgen05 mode the dense targets go to its table instead.
    std::vector<HadTile> tiles;
    std::vector<int> slots, rows, dtab, drow;
    std::vector<uint2> tab;
    W.had_tile0.assign(ng + 1, 0);
    W.hadd_tab0.assign(ng, 0);
    W.hadd_row0.assign(ng, 0);
    W.hadd_ld.assign(ng, 0);
    const std::vector<int> oct = t.octant.download(s, (size_t)t.nnodes);
    const std::vector<int> msrc = t.m2l_src.download(s, (size_t)t.n_m2l_src);
    std::vector<int> slot_of(maxn, -1), used;  // slot of each source in the open tile; its sources
    std::vector<uint32_t> ent(26 * (size_t)HADH_TT);
    for (int g = 0; g < ng; g++) {
      W.had_tile0[g] = (int)tiles.size();
      const int tb = t.m2l_trg_off[g], te = t.m2l_trg_off[g + 1];
      const int* snode = msrc.data() + t.m2l_src_off[g];
      std::vector<int> dense, rest;
      for (int tt = tb; tt < te; tt++) {
        int cnt = 0;
        for (int ipos = 0; ipos < 26; ipos++) cnt += t.h_m2l_tab[26 * (size_t)tt + ipos] >= 0;
        (W.had_tc5 && cnt >= HAD_DENSE_MIN ? dense : rest).push_back(tt);
      }
      if ((int)dense.size() < HAD_DENSE_GROUP_MIN) {
        rest.insert(rest.end(), dense.begin(), dense.end());
        std::sort(rest.begin(), rest.end());
        dense.clear();
      }
      auto by_level = [&](int a, int b) { return t.h_level[t.h_m2l_trg[a]] < t.h_level[t.h_m2l_trg[b]]; };
      std::stable_sort(dense.begin(), dense.end(), by_level);
      std::stable_sort(rest.begin(), rest.end(), by_level);
      const int ld = (int)((dense.size() + HADC_TT - 1) / HADC_TT) * HADC_TT;
      W.hadd_ld[g] = ld;
      W.hadd_tab0[g] = (int64_t)dtab.size();
      W.hadd_row0[g] = (int64_t)drow.size();
      dtab.resize(dtab.size() + (size_t)26 * ld, -1);
      drow.resize(drow.size() + ld, -1);
      for (size_t k = 0; k < dense.size(); k++) {
        const int tt = dense[k];
        drow[W.hadd_row0[g] + k] = tt - tb;
        for (int ipos = 0; ipos < 26; ipos++)
          dtab[W.hadd_tab0[g] + (size_t)ipos * ld + k] = t.h_m2l_tab[26 * (size_t)tt + ipos];
      }
      for (size_t k0 = 0; k0 < rest.size();) {
        int fill[8] = {1, 1, 1, 1, 1, 1, 1, 1};  // slots 0 .. 7 are the zeros
        size_t k1 = k0;
        for (; k1 < rest.size() && k1 - k0 < (size_t)HADH_TT; k1++) {
          const int* src = t.h_m2l_tab.data() + 26 * (size_t)rest[k1];
          int need[8] = {0, 0, 0, 0, 0, 0, 0, 0};
          bool fits = true;
          for (int ipos = 0; ipos < 26; ipos++)
            if (src[ipos] >= 0 && slot_of[src[ipos]] < 0) {
              const int c = oct[snode[src[ipos]]] & 7;
              if (fill[c] + ++need[c] > HADH_SLOTS / 8) fits = false;
            }
          if (!fits) break;
          for (int ipos = 0; ipos < 26; ipos++)
            if (src[ipos] >= 0 && slot_of[src[ipos]] < 0) {
              const int c = oct[snode[src[ipos]]] & 7;
              slot_of[src[ipos]] = 8 * fill[c]++ + c;
              used.push_back(src[ipos]);
            }
        }
        HadTile T;
        T.nslots = 8 * *std::max_element(fill, fill + 8);
        const int nt = (int)(k1 - k0);
        T.groups = (nt + 63) / 64;
        while ((HADH_NT / 32) % T.groups) T.groups++;
        T.slot0 = (int)slots.size();
        T.row0 = (int)rows.size();
        T.tab0 = (int64_t)tab.size();
        slots.resize(slots.size() + T.nslots, -1);
        for (int src : used) slots[T.slot0 + slot_of[src]] = src;
        for (int k = 0; k < 64 * T.groups; k++) rows.push_back(k < nt ? rest[k0 + k] - tb : -1);
        // per position the slot of every target; empty rows of a fragment's 8 take zero slots off the
        // others' banks
        for (int ipos = 0; ipos < 26; ipos++)
          for (int k = 0; k < 64 * T.groups; k += 8) {
            uint32_t classes = 0;
            int sl[8];
            for (int i = 0; i < 8; i++) {
              const int src = k + i < nt ? t.h_m2l_tab[26 * (size_t)rest[k0 + k + i] + ipos] : -1;
              sl[i] = src >= 0 ? slot_of[src] : -1;
              if (src >= 0) classes |= 1u << (sl[i] & 7);
            }
            int c = 0;
            for (int i = 0; i < 8; i++) {
              if (sl[i] < 0) {
                while (c < 7 && (classes >> c & 1)) c++;
                sl[i] = c;
                classes |= 1u << c;
              }
              ent[(size_t)ipos * HADH_TT + k + i] = hadh_entry(sl[i]);
            }
          }
        tab.resize(tab.size() + (size_t)26 * T.groups * 32);
        uint2* o = tab.data() + T.tab0;
        for (int ipos = 0; ipos < 26; ipos++)
          for (int gr = 0; gr < T.groups; gr++)
            for (int ln = 0; ln < 32; ln++) {
              const uint32_t* e = ent.data() + (size_t)ipos * HADH_TT + 64 * gr + (ln & 15);
              *o++ = make_uint2(e[0] | e[16] << 16, e[32] | e[48] << 16);
            }
        tiles.push_back(T);
        for (int src : used) slot_of[src] = -1;
        used.clear();
        k0 = k1;
      }
    }
    W.had_tile0[ng] = (int)tiles.size();
    if (!tiles.empty()) {
      W.hadh_tile.upload(tiles, s);
      W.hadh_slots.upload(slots, s);
      W.hadh_rows.upload(rows, s);
      W.hadh_tab.upload(tab, s);
      W.hadh_pslots.alloc(slots.size());
      W.hadh_tinv.alloc(tiles.size());
      W.hadh_tpass.alloc(tiles.size());
    }
    if (!dtab.empty()) {
      W.hadd_tab.upload(dtab, s);
      W.hadd_row.upload(drow, s);
      W.hadd_tabp.alloc(dtab.size());
    }
    XCUDA(cudaStreamSynchronize(s));  // the host tables are released here
  } else {
    // FP64: every target in the dense form on the FP64 tensor cores (k_hadamard_d64): per group a [26][ld]
    // source table and ld output rows, targets level by level (Morton order inside a level), padded to
    // whole CTA tiles
    std::vector<int> dtab, drow;
    W.had_tile0.assign(ng + 1, 0);
    W.hadd_tab0.assign(ng, 0);
    W.hadd_row0.assign(ng, 0);
    W.hadd_ld.assign(ng, 0);
    for (int g = 0; g < ng; g++) {
      const int tb = t.m2l_trg_off[g], te = t.m2l_trg_off[g + 1];
      std::vector<int> all;
      for (int tt = tb; tt < te; tt++) all.push_back(tt);
      std::stable_sort(all.begin(), all.end(),
                       [&](int a, int b) { return t.h_level[t.h_m2l_trg[a]] < t.h_level[t.h_m2l_trg[b]]; });
      const int ld = (int)((all.size() + HAD64_TT - 1) / HAD64_TT) * HAD64_TT;
      W.hadd_ld[g] = ld;
      W.hadd_tab0[g] = (int64_t)dtab.size();
      W.hadd_row0[g] = (int64_t)drow.size();
      dtab.resize(dtab.size() + (size_t)26 * ld, -1);
      drow.resize(drow.size() + ld, -1);
      for (size_t k = 0; k < all.size(); k++) {
        const int tt = all[k];
        drow[W.hadd_row0[g] + k] = tt - tb;
        for (int ipos = 0; ipos < 26; ipos++)
          dtab[W.hadd_tab0[g] + (size_t)ipos * ld + k] = t.h_m2l_tab[26 * (size_t)tt + ipos];
      }
    }
    if (dtab.empty()) dtab.push_back(-1);
    if (drow.empty()) drow.push_back(-1);
    W.hadd_tab.upload(dtab, s);
    W.hadd_row.upload(drow, s);
  }
  for (auto& e : W.ev) XCUDA(cudaEventCreate(&e));
  W.m2l_ev.resize(4 * (size_t)ng);
  for (auto& e : W.m2l_ev) XCUDA(cudaEventCreate(&e));
  W.ev_ok = true;
  XCUDA(cudaStreamSynchronize(s));
  return W;
}

template <class RB> const RB* m2l_scale_of(const Tree& t);
template <> const float* m2l_scale_of<float>(const Tree& t) { return t.m2l_scale.p; }
template <> const double* m2l_scale_of<double>(const Tree& t) { return t.m2l_scale64.p; }

// The near field's close pairs of this tree (count, then fill), once per workspace; no allocation while
// evaluating afterwards.
void find_close_pairs(Workspace& ws, const NearArgs& na, int n_eval, cudaStream_t s) {
  DBuf<unsigned long long> cnt(2);
  XCUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), s));
  if (n_eval > 0) {
    k_close_scan<false><<<nblk(n_eval, 4), 128, 0, s>>>(na, cnt.p, nullptr, 0);
    XLAUNCH();
  }
  unsigned long long n = 0;
  XCUDA(cudaMemcpyAsync(&n, cnt.p, sizeof(n), cudaMemcpyDeviceToHost, s));
  XCUDA(cudaStreamSynchronize(s));
  ws.close_pairs.alloc(std::max<unsigned long long>(n, 1));
  if (n > 0) {
    k_close_scan<true><<<nblk(n_eval, 4), 128, 0, s>>>(na, cnt.p + 1, ws.close_pairs.p, (int64_t)n);
    XLAUNCH();
    XCUDA(cudaStreamSynchronize(s));  // cnt is released on return
  }
  ws.n_close = (int64_t)n;
}

constexpr int DOWN_PRE = 1, DOWN_NEAR = 2, DOWN_FAR = 4, DOWN_ALL = 7;
constexpr int M2L_FWD = 1, M2L_HAD_TILES = 2, M2L_HAD_DENSE = 4, M2L_BWD = 8, M2L_ALL = 15;
// parts of the downward pass before the near field: the M2L parts above (P2L with the forward transforms),
// then L2L, then L2P's check-to-equivalent step
constexpr int PRE_L2L = 16, PRE_DC2E = 32, PRE_ALL = M2L_ALL | PRE_L2L | PRE_DC2E;
// parts of the upward pass: P2M's check potentials, its two pseudo-inverse GEMMs, M2M
constexpr int UP_CHK = 1, UP_M2M = 2, UP_PINV = 4, UP_P2M = UP_CHK | UP_PINV, UP_ALL = 7;

// ------------------------------------------------------------------ engine, per kernel and precision
template <int KER, class R>
struct Engine {
  using W = typename Green<KER, R>::Q;          // working value: R or complex
  using V64 = typename Green<KER, double>::Q;   // FP64 value (pinv GEMMs, downward equivalent densities)
  using CT = typename C2<R>::type;              // spectrum value
  static constexpr int CW = KER == K_HELMHOLTZ ? 2 : 1;  // reals per value

  static void split_scratch(TGemm& g, Workspace& ws) {
    g.scratch = ws.tc_scratch.p;
    g.scratch_len = (int64_t)ws.tc_scratch.n;
  }
  static void upward(Fmm& f, Tree& t, Workspace& ws, cudaStream_t s, int parts = UP_ALL) {
    const int n = f.nsurf;
    if (parts & UP_P2M) {
      if (parts & UP_CHK) {
        ws.launches = 0;
        XCUDA(cudaEventRecord(ws.ev[0], s));
      }
      // P2M: check potentials of every leaf, then the pinv (UC2E) GEMM per leaf level
      if (t.nleafs && (parts & UP_CHK)) {
        SurfPotArgs a{t.leafs.p,  t.nleafs, t.nsrcs.p,     nullptr,  t.level.p, t.sbeg.p,   nullptr, t.center.p,
                      t.src4.p,   t.src_qim.p, f.surf_base.p, n,      2.95,      ws.chk.p, 0,         f.k_re, f.k_im,
                      INV4PI * op_scale(f, t)};
        if constexpr (KER == K_LAPLACE && sizeof(R) == 4)
          k_surf_pot_lap_f2<<<surf_grid_of(t.nleafs), 128, 0, s>>>(a);
        else
          k_surf_pot<KER, R><<<surf_grid_of(t.nleafs), 128, 0, s>>>(a);
        XLAUNCH();
        ws.launches++;
      }
      if (t.nleafs && (parts & UP_PINV)) {
        // e = 0.5^l (V S+) (U^H c) per leaf level, two FP64 GEMMs on the tensor cores: y over the kept
        // singular directions only, then e scattered to the leaves' up rows with the level's scale.
        // (An FP32 first factor, as in L2P below, measured 1.4e-7 more potential error at p = 8 and 3e-7
        // at p = 10: the upward densities feed every later translation.)
        for (int l = 0; l <= t.depth; l++) {
          if (KER == K_LAPLACE && l > 0) break;
          const int r0 = ws.leaf_level_off[l], r1 = ws.leaf_level_off[l + 1];
          const int m = KER == K_LAPLACE ? ws.p2m1.M : r1 - r0;
          const int off = KER == K_LAPLACE ? 0 : r0;
          if (m <= 0) continue;
          const LevelOps& op = level_ops(f, l);
          const int rk = op.rank;
          TGemm g1{m, CW * rk, CW * n, ws.p2m1.a.p + off, ws.p2m1.c.p + off, nullptr, (int64_t)CW * n, 0, (int64_t)CW * n};
          split_scratch(g1, ws);
          tgemm_f64<R, double>(g1, (const R*)ws.chk.p, op.tg_p2m1.p, (double*)ws.ybuf.p, s);
          TGemm g2{m, CW * n, CW * rk, ws.p2m2.a.p + off, ws.p2m2.c.p + off, ws.p2m2.al64.p + off, (int64_t)CW * n, 0,
                   (int64_t)CW * n};
          split_scratch(g2, ws);
          tgemm_f64<double, R>(g2, (const double*)ws.ybuf.p, op.tg_p2m2.p, (R*)ws.up.p, s);
          ws.launches += 2;
        }
      }
      if (parts & UP_PINV) XCUDA(cudaEventRecord(ws.ev[1], s));
    }
    if (!(parts & UP_M2M)) return;
    // M2M: deepest parents first (post-order); per level one GEMM of the parents' 8 children rows
    // (contiguous per parent) with the [8n][n] operator, written to the parents' rows
    for (int l = t.depth - 1; l >= 0; l--) {
      const GemmRows& g = ws.m2m[l];
      if (g.M <= 0) continue;
      const LevelOps& op = level_ops(f, l);
      // the parents' rows start at zero (clear_values): the products are added to them, as the reference
      // adds each child's contribution (fmm_scale_invariant.h:243-251)
      TGemm gm{g.M, CW * n, CW * 8 * n, g.a.p, g.c.p, nullptr, (int64_t)CW * n, 1, (int64_t)CW * n};
      gm.status = ws.status.p;
      split_scratch(gm, ws);
      if constexpr (sizeof(R) == 4)
        tgemm_tc<float>(gm, (const float*)ws.up.p, op.tg_m2m_h.p, op.tg_m2m_l.p, op.ld_m2m, (float*)ws.up.p, s);
      else
        tgemm_f64<double, double>(gm, (const double*)ws.up.p, op.tg_m2m.p, (double*)ws.up.p, s);
      ws.launches++;
    }
    XCUDA(cudaEventRecord(ws.ev[2], s));
  }

  // phase: which parts of every group's M2L to run (M2L_FWD, M2L_HAD_TILES, M2L_HAD_DENSE, M2L_BWD)
  static void m2l(Fmm& f, Tree& t, Workspace& ws, cudaStream_t s, int phase = M2L_ALL) {
    const int n = f.nsurf, nconv = f.nconv, nfreq = f.nfreq;
    const int ng = (int)t.m2l_src_off.size() - 1;
    for (int g = 0; g < ng; g++) {
      cudaEvent_t* ev = ws.m2l_ev.data() + 4 * g;
      const int ns = t.m2l_src_off[g + 1] - t.m2l_src_off[g], nt = t.m2l_trg_off[g + 1] - t.m2l_trg_off[g];
      if (ns == 0 || nt == 0) continue;
      const int* src = t.m2l_src.p + t.m2l_src_off[g];
      const int* trg = t.m2l_trg.p + t.m2l_trg_off[g];
      const int tab_level = KER == K_LAPLACE ? 0 : g + 1;
      using SP = typename Spec<R>::type;
      SP* spec = (SP*)ws.specB.p;
      const bool screened = KER != K_LAPLACE && f.screened();
      const SplitOut so{ws.scode.p, ws.sbound.p, ws.swin.p, screened ? ws.shead.p : nullptr};
      if (phase & M2L_FWD) {
        XCUDA(cudaEventRecord(ev[0], s));
        if constexpr (sizeof(R) == 4) {
          if (screened) {
            k_source_bounds<W><<<std::min(ns, 148 * 8), 256, 0, s>>>(src, ns, t.child0.p, (const W*)ws.up.p, n,
                                                                   ws.sbound.p, ws.shead.p);
            XLAUNCH();
            ws.launches++;
          }
        }
        // upward equivalent DFT (fmm_scale_invariant.h:560-604) -> specB [f][s][c]
        if constexpr (KER != K_HELMHOLTZ) {
          if (ws.fused) {
            ft_dispatch(f.p, [&](auto pc) {
              constexpr int PP = decltype(pc)::value;
              const size_t smem = ftr_fwd_smem<R>(PP);
              if (ws.ft_fwd_smem < smem) {
                XCUDA(cudaFuncSetAttribute(k_m2l_fwd_r<R, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                ws.ft_fwd_smem = smem;
              }
              k_m2l_fwd_r<R, PP><<<dim3(ns, 8 / FtCpb<R>::v), FT_NT, smem, s>>>(
                  src, ns, t.child0.p, (const R*)ws.up.p, n, f.conv_to_surf_up.p, f.dft_tw.p, spec, so);
            });
            XLAUNCH();
            ws.launches++;
          }
        } else if (ws.fused) {
          ftc_dispatch(f.p, [&](auto pc) {
            constexpr int PP = decltype(pc)::value;
            const size_t smem = ftc_fwd_smem<R>(PP);
            if (ws.ft_fwd_smem < smem) {
              XCUDA(cudaFuncSetAttribute(k_m2l_fwd_c<R, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
              ws.ft_fwd_smem = smem;
            }
            k_m2l_fwd_c<R, PP><<<dim3(ns, 8 / FtcCpb<R>::v), FT_NT, smem, s>>>(
                src, ns, t.child0.p, (const CT*)ws.up.p, n, f.conv_to_surf_up.p, f.dft_tw.p, spec, so);
          });
          XLAUNCH();
          ws.launches++;
        }
        if (!ws.fused) {
          k_m2l_grid_up<W><<<std::min<int64_t>(nblk((int64_t)ns * 8 * nconv), 148 * 32), 256, 0, s>>>(
              src, ns, t.child0.p, (const W*)ws.up.p, n, f.conv_to_surf_up.p, nconv, (W*)ws.grid.p);
          XLAUNCH();
          ws.launches++;
          XCUFFT2(cufftSetStream(ws.fwd[g], s));
          exec_fwd(ws.fwd[g], ws.grid.p, ws.specA.p);
          ws.launches++;
          if constexpr (sizeof(R) == 4) {  // -> [f][s][c], split
            k_source_codes<W><<<ns, 256, 0, s>>>(src, t.child0.p, (const W*)ws.up.p, n, so);
            XLAUNCH();
            const dim3 grid((nfreq + 31) / 32, ((int64_t)ns * 8 + 31) / 32);
            XREQUIRE(grid.y < 65536, XFMM_ERR_UNSUPPORTED, "transpose too tall");
            k_transpose_split<<<grid, dim3(32, 8), 0, s>>>((const float2*)ws.specA.p, spec, ns, nfreq, so);
            XLAUNCH();
            ws.launches++;
          } else {
            transpose<CT>((const CT*)ws.specA.p, (CT*)ws.specB.p, (int64_t)ns * 8, nfreq, s);  // -> [f][s][c]
          }
        }
        if (const int nht = ws.had_tile0[g + 1] - ws.had_tile0[g]; sizeof(R) == 4 && nht > 0 && !screened) {
          k_tile_codes<<<nht, 256, 0, s>>>(ws.hadh_tile.p + ws.had_tile0[g], ws.hadh_slots.p, ws.scode.p,
                                           ws.hadh_pslots.p, ws.hadh_tinv.p + ws.had_tile0[g],
                                           ws.hadh_tpass.p + ws.had_tile0[g]);
          XLAUNCH();
          ws.launches++;
        }
        if (sizeof(R) == 4 && ws.hadd_ld[g] > 0 && !screened) {  // the tcgen05 form's table
          const int64_t nd = (int64_t)26 * ws.hadd_ld[g];
          k_pack_sources<<<std::min<int64_t>(nblk(nd), 148 * 8), 256, 0, s>>>(
              ws.hadd_tab.p + ws.hadd_tab0[g], nd, ws.scode.p, ws.hadd_tabp.p + ws.hadd_tab0[g]);
          XLAUNCH();
          ws.launches++;
        }
        XCUDA(cudaEventRecord(ev[1], s));
      }
      if (phase & (M2L_HAD_TILES | M2L_HAD_DENSE)) {
        // Hadamard product
        const int ntiles = ws.had_tile0[g + 1] - ws.had_tile0[g];
        if constexpr (sizeof(CT) == 8) {
          XREQUIRE(nfreq < 65536, XFMM_ERR_UNSUPPORTED, "too many frequencies for the Hadamard grid");
          if (ntiles > 0 && (phase & M2L_HAD_TILES)) {
            if (!ws.hadh_attr) {
              for (auto kern : {k_hadamard_h<false>, k_hadamard_h<true>})
                XCUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HADH_SMEM));
              ws.hadh_attr = true;
            }
            const int tpc = t.hadr_tpc > 0 ? t.hadr_tpc : HADH_TPC;
            const HadSys S = had_sys(ws, g, ns, nt, screened);
            const LevelOps& op = f.ops[tab_level];
            const auto kern = screened ? k_hadamard_h<true> : k_hadamard_h<false>;
            kern<<<dim3((ntiles + tpc - 1) / tpc, nfreq), HADH_NT, HADH_SMEM, s>>>(
                (const uint4*)op.m2l_frag.p, op.m2l_binv.p, op.m2l_windows, S, ntiles, tpc);
            XLAUNCH();
            ws.launches++;
          }
          if (ws.hadd_ld[g] > 0 && (phase & M2L_HAD_DENSE)) {
            if (!ws.hadc_attr) {
              for (auto kern : {k_hadamard_dc<false>, k_hadamard_dc<true>})
                XCUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HADC_SMEM));
              ws.hadc_attr = true;
            }
            const LevelOps& op = f.ops[tab_level];
            if (ws.hadc_btab_id != op.m2l_id) {  // B blocks in the MMA layout
              ws.hadc_btab.reserve((size_t)nfreq * HADC_BBYTES);
              k_hadc_btab<<<std::min<int64_t>(nblk((int64_t)nfreq * 26 * 64), 148 * 16), 256, 0, s>>>(
                  (const uint4*)op.m2l_frag.p, op.m2l_binv.p, op.m2l_windows, screened ? 1.f / SPLIT_TAIL : 1.f, nfreq,
                  ws.hadc_btab.p);
              XLAUNCH();
              ws.launches++;
              ws.hadc_btab_id = op.m2l_id;
            }
            const auto kern = screened ? k_hadamard_dc<true> : k_hadamard_dc<false>;
            const uint32_t* tab = screened ? (const uint32_t*)ws.hadd_tab.p : ws.hadd_tabp.p;  // -1 is SPLIT_NONE
            kern<<<dim3(ws.hadd_ld[g] / 128, (nfreq + HADC_FPB - 1) / HADC_FPB), HADC_NT, HADC_SMEM, s>>>(
                ws.hadc_btab.p, spec, (CT*)ws.specA.p, ws.shead.p, ws.swin.p, tab + ws.hadd_tab0[g], ws.hadd_ld[g],
                ws.hadd_row.p + ws.hadd_row0[g], ns, nt, nfreq, ws.status.p);
            XLAUNCH();
            ws.launches++;
          }
        } else {
          XREQUIRE(nfreq < 65536, XFMM_ERR_UNSUPPORTED, "too many frequencies for the Hadamard grid");
          if (ws.hadd_ld[g] > 0 && (phase & M2L_HAD_DENSE)) {
            if (!ws.had64_attr) {
              XCUDA(cudaFuncSetAttribute(k_hadamard_d64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HAD64_SMEM));
              ws.had64_attr = true;
            }
            k_hadamard_d64<<<dim3(ws.hadd_ld[g] / HAD64_TT, nfreq), HAD64_NT, HAD64_SMEM, s>>>(
                (const double*)f.ops[tab_level].m2l_frag.p, spec, (CT*)ws.specA.p, ws.hadd_tab.p + ws.hadd_tab0[g], ws.hadd_ld[g],
                ws.hadd_row.p + ws.hadd_row0[g], ns, nt);
            XLAUNCH();
            ws.launches++;
          }
        }
        XCUDA(cudaEventRecord(ev[2], s));
      }
      if (phase & M2L_BWD) {
        // inverse DFT of specA [f][t][c] to the downward check potentials (fmm_scale_invariant.h:606-646)
        if constexpr (KER != K_HELMHOLTZ) {
          if (ws.fused) {
            ft_dispatch(f.p, [&](auto pc) {
              constexpr int PP = decltype(pc)::value;
            if constexpr (sizeof(R) == 4) {  // FP64: the unslabbed form (measured faster at 1 CTA per SM)
              const size_t smem = ftr_bwd_smem<R>(PP);
              if (ws.ft_bwd_smem < smem) {
                XCUDA(cudaFuncSetAttribute(k_m2l_bwd_r<R, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                ws.ft_bwd_smem = smem;
              }
              k_m2l_bwd_r<R, PP><<<dim3(nt, 8 / FtCpb<R>::v), FT_NT, smem, s>>>(
                  trg, nt, t.child0.p, (const CT*)ws.specA.p, n, f.map_dn.p, f.dft_tw.p,
                  m2l_scale_of<R>(t) + t.m2l_trg_off[g], (R*)ws.dn.p);
            } else {
              const size_t smem = ft_bwd_smem<R>(PP);
              if (ws.ft_bwd_smem < smem) {
                XCUDA(cudaFuncSetAttribute(k_m2l_bwd<R, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                ws.ft_bwd_smem = smem;
              }
              k_m2l_bwd<R, PP><<<dim3(nt, 8 / FtCpb<R>::v), FT_NT, smem, s>>>(
                  trg, nt, t.child0.p, (const CT*)ws.specA.p, n, f.map_dn.p, f.dft_tw.p,
                  m2l_scale_of<R>(t) + t.m2l_trg_off[g], (R*)ws.dn.p);
            }
            });
            XLAUNCH();
            ws.launches++;
          }
        } else if (ws.fused) {
          ftc_dispatch(f.p, [&](auto pc) {
            constexpr int PP = decltype(pc)::value;
            const size_t smem = ftc_bwd_smem<R>(PP);
            if (ws.ft_bwd_smem < smem) {
              XCUDA(cudaFuncSetAttribute(k_m2l_bwd_c<R, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
              ws.ft_bwd_smem = smem;
            }
            k_m2l_bwd_c<R, PP><<<dim3(nt, 8 / FtcCpb<R>::v), FT_NT, smem, s>>>(trg, nt, t.child0.p, (const CT*)ws.specA.p, n,
                                                               f.map_dn.p, f.dft_tw.p,
                                                               m2l_scale_of<R>(t) + t.m2l_trg_off[g], (CT*)ws.dn.p);
          });
          XLAUNCH();
          ws.launches++;
        }
        if (!ws.fused) {
          ws.launches++;
          transpose<CT>((const CT*)ws.specA.p, (CT*)ws.specB.p, nfreq, (int64_t)nt * 8, s);  // -> [t][c][f]
          XCUFFT2(cufftSetStream(ws.bwd[g], s));
          exec_bwd(ws.bwd[g], ws.specB.p, ws.grid.p);
          k_m2l_gather_dn<W, R><<<std::min<int64_t>(nblk((int64_t)nt * 8 * n), 148 * 32), 256, 0, s>>>(
              trg, nt, t.child0.p, (const W*)ws.grid.p, nconv, f.map_dn.p, n,
              m2l_scale_of<R>(t) + t.m2l_trg_off[g], (W*)ws.dn.p);
          XLAUNCH();
          ws.launches += 2;
        }
        XCUDA(cudaEventRecord(ev[3], s));
      }
    }
  }

  static void exec_fwd(cufftHandle h, void* in, void* out) {
    if (KER == K_HELMHOLTZ) {
      if (sizeof(R) == 4) XCUFFT2(cufftExecC2C(h, (cufftComplex*)in, (cufftComplex*)out, CUFFT_FORWARD));
      else XCUFFT2(cufftExecZ2Z(h, (cufftDoubleComplex*)in, (cufftDoubleComplex*)out, CUFFT_FORWARD));
    } else {
      if (sizeof(R) == 4) XCUFFT2(cufftExecR2C(h, (cufftReal*)in, (cufftComplex*)out));
      else XCUFFT2(cufftExecD2Z(h, (cufftDoubleReal*)in, (cufftDoubleComplex*)out));
    }
  }
  static void exec_bwd(cufftHandle h, void* in, void* out) {
    if (KER == K_HELMHOLTZ) {
      if (sizeof(R) == 4) XCUFFT2(cufftExecC2C(h, (cufftComplex*)in, (cufftComplex*)out, CUFFT_INVERSE));
      else XCUFFT2(cufftExecZ2Z(h, (cufftDoubleComplex*)in, (cufftDoubleComplex*)out, CUFFT_INVERSE));
    } else {
      if (sizeof(R) == 4) XCUFFT2(cufftExecC2R(h, (cufftComplex*)in, (cufftReal*)out));
      else XCUFFT2(cufftExecZ2D(h, (cufftDoubleComplex*)in, (cufftDoubleReal*)out));
    }
  }

  // the tiles of group g of the mixed path's Hadamard
  static HadSys had_sys(Workspace& ws, int g, int ns, int nt, bool screened = false) {
    return HadSys{(const SplitC*)ws.specB.p,         (float2*)ws.specA.p,
                  ws.hadh_tile.p + ws.had_tile0[g],  screened ? (const uint32_t*)ws.hadh_slots.p : ws.hadh_pslots.p,
                  ws.hadh_tinv.p + ws.had_tile0[g],  ws.hadh_tpass.p + ws.had_tile0[g],
                  ws.shead.p,                        ws.swin.p,
                  ws.hadh_tab.p,                     ws.hadh_rows.p,
                  ns,                                nt};
  }

  // the far field (M2P + L2P evaluation), added to the near field's values
  static EvalArgs far_args(Fmm& f, Tree& t, Workspace& ws) {
    return EvalArgs{t.eval_leafs.p, t.leafs.p,     t.ntrgs.p,     t.n_eval_leafs, t.tbeg.p, t.center.p,
                    t.trg4.p,       t.m2p_off.p,   t.m2p.p,       f.surf_base.p,  f.surf_perm.p, f.surf_grid.p,
                    f.nsurf,        ws.up.p,       ws.eq.p,       ws.out.p,       f.k_re,   f.k_im};
  }

  static NearArgs near_args(Fmm& f, Tree& t, Workspace& ws) {
    return NearArgs{t.eval_leafs.p, t.leafs.p, t.nsrcs.p,   t.ntrgs.p, t.n_eval_leafs, t.sbeg.p, t.tbeg.p,
                    t.p2p_off.p,    t.p2p.p,   t.center.p,  t.src4.p,  t.trg4.p,       t.src_qim.p, ws.out.p,
                    f.k_re,         f.k_im,    t.n_eval_leafs < SPLIT_LEAVES ? NEAR_PARTS : 1};
  }

  // phases: DOWN_PRE (P2L, M2L, L2L, L2P check-to-equivalent), DOWN_NEAR (P2P), DOWN_FAR (M2P + L2P
  // evaluation, added to the near field's values); an evaluate runs all three in this order
  static void downward(Fmm& f, Tree& t, Workspace& ws, cudaStream_t s, int phases = DOWN_ALL, int m2l_phase = PRE_ALL) {
    const int n = f.nsurf;
    if (phases & DOWN_PRE) downward_pre(f, t, ws, s, m2l_phase);
    if (t.n_eval_leafs && (phases & DOWN_NEAR)) {
      NearArgs na = near_args(f, t, ws);
      if constexpr (KER == K_LAPLACE && sizeof(R) == 4) {
        if (ws.n_close < 0) find_close_pairs(ws, na, t.n_eval_leafs, s);
        if (na.parts > 1) k_near_lap_f2_parts<<<t.n_eval_leafs, 32 * NEAR_PARTS, 0, s>>>(na);
        else k_near_lap_f2<<<nblk(t.n_eval_leafs, 4), 128, 0, s>>>(na);
        XLAUNCH();
        ws.launches++;
        if (ws.n_close > 0) {
          k_close_fix<<<nblk(ws.n_close, 256), 256, 0, s>>>(ws.close_pairs.p, ws.n_close, na, nullptr);
          XLAUNCH();
          ws.launches++;
        }
      } else {
        if (na.parts > 1) k_near_parts<KER, R><<<t.n_eval_leafs, 32 * NEAR_PARTS, 0, s>>>(na);
        else k_near<KER, R><<<nblk(t.n_eval_leafs, 4), 128, 0, s>>>(na);
        XLAUNCH();
        ws.launches++;
      }
    }
    if (phases & DOWN_NEAR) XCUDA(cudaEventRecord(ws.ev[8], s));
    if (t.n_eval_leafs && (phases & DOWN_FAR)) {
      const EvalArgs a = far_args(f, t, ws);
      const int blocks = nblk(t.n_eval_leafs, EVAL_WARPS);
      if constexpr (KER == K_LAPLACE) {
        order_dispatch(f.p, [&](auto pc) {
          constexpr int PP = decltype(pc)::value;
          const size_t smem = far_smem(n, PP);
          if (t.n_eval_leafs < SPLIT_LEAVES)
            k_far_lap<W, PP, FAR_PARTS><<<t.n_eval_leafs, 32 * EVAL_WARPS, smem, s>>>(a);
          else
            k_far_lap<W, PP, 1><<<blocks, 32 * EVAL_WARPS, smem, s>>>(a);
        });
      } else {
        if (t.n_eval_leafs < SPLIT_LEAVES) k_eval<KER, W, EVAL_WARPS><<<t.n_eval_leafs, 32 * EVAL_WARPS, 0, s>>>(a);
        else k_eval<KER, W, 1><<<blocks, 32 * EVAL_WARPS, 0, s>>>(a);
      }
      XLAUNCH();
      ws.launches++;
    }
    if (phases & DOWN_FAR) XCUDA(cudaEventRecord(ws.ev[7], s));
  }

  // m2l_phase: the parts to run (PRE_ALL for an evaluate): the M2L parts (P2L with the forward transforms),
  // L2L (PRE_L2L) and L2P's check-to-equivalent step (PRE_DC2E)
  static void downward_pre(Fmm& f, Tree& t, Workspace& ws, cudaStream_t s, int m2l_phase = PRE_ALL) {
    const int n = f.nsurf;
    // P2L (X list) into downward check potentials
    if (t.n_p2l_nodes && (m2l_phase & M2L_FWD)) {
      SurfPotArgs a{t.p2l_nodes.p, t.n_p2l_nodes, t.nsrcs.p,     t.p2l.p, t.level.p, t.sbeg.p, t.p2l_off.p, t.center.p,
                    t.src4.p,      t.src_qim.p,   f.surf_base.p, n,       1.05,      ws.dn.p,  1,           f.k_re,
                    f.k_im,        INV4PI * op_scale(f, t)};
      k_surf_pot<KER, R><<<surf_grid_of(t.n_p2l_nodes), 128, 0, s>>>(a);
      XLAUNCH();
      ws.launches++;
    }
    if (m2l_phase & M2L_FWD) XCUDA(cudaEventRecord(ws.ev[3], s));
    // M2L
    if (t.n_m2l_trg) m2l(f, t, ws, s, m2l_phase);
    if (m2l_phase & M2L_BWD) XCUDA(cudaEventRecord(ws.ev[4], s));
    if (m2l_phase & PRE_L2L) {
      // L2L: shallowest parents first (pre-order); per level one GEMM of the parents' rows with the
      // [n][8n] operator, added to the 8 children rows (contiguous per parent)
      for (int l = 0; l < t.depth; l++) {
        const GemmRows& g = ws.l2l[l];
        if (g.M <= 0) continue;
        const LevelOps& op = level_ops(f, l);
        TGemm gl{g.M, CW * 8 * n, CW * n, g.a.p, g.c.p, nullptr, (int64_t)CW * 8 * n, 1, (int64_t)CW * n};
        gl.status = ws.status.p;
        split_scratch(gl, ws);
        if constexpr (sizeof(R) == 4)
          tgemm_tc<float>(gl, (const float*)ws.dn.p, op.tg_l2l_h.p, op.tg_l2l_l.p, op.ld_l2l, (float*)ws.dn.p, s);
        else
          tgemm_f64<double, double>(gl, (const double*)ws.dn.p, op.tg_l2l.p, (double*)ws.dn.p, s);
        ws.launches++;
      }
      XCUDA(cudaEventRecord(ws.ev[5], s));
    }
    if (!(m2l_phase & PRE_DC2E)) return;
    // L2P part 1: downward check -> equivalent (DC2E) per leaf level, e = conj(U) S+ (conj(VH) 0.5^l c):
    // y over the kept singular directions, then e to the leaf positions (FP64).
    if (t.nleafs) {
      for (int l = 0; l <= t.depth; l++) {
        if (KER == K_LAPLACE && l > 0) break;
        const int r0 = ws.leaf_level_off[l], r1 = ws.leaf_level_off[l + 1];
        const int m = KER == K_LAPLACE ? ws.l2p1.M : r1 - r0;
        const int off = KER == K_LAPLACE ? 0 : r0;
        if (m <= 0) continue;
        const LevelOps& op = level_ops(f, l);
        const int rk = op.rank;
        TGemm g1{m, CW * rk, CW * n, ws.l2p1.a.p + off, ws.l2p1.c.p + off, ws.l2p2.al64.p + off, (int64_t)CW * n, 0,
                 (int64_t)CW * n};
        // The mixed path's downward check values are FP32 and conj(VH) is orthogonal: y = conj(VH) c runs
        // at FP32 accuracy (TF32 x 3), then e = conj(U) S+ y, whose 1/s amplification needs FP64.  These
        // densities feed only the leaf's own targets (measured: +0.5e-7 potential error at p = 8, +1e-7
        // at p = 10).
        g1.status = ws.status.p;
        split_scratch(g1, ws);
        if constexpr (sizeof(R) == 4 && KER != K_HELMHOLTZ)
          tgemm_tc<double>(g1, (const float*)ws.dn.p, op.tg_l2p1_h.p, op.tg_l2p1_l.p, op.ld_l2p1, (double*)ws.ybuf.p, s);
        else
          tgemm_f64<R, double>(g1, (const R*)ws.dn.p, op.tg_l2p1.p, (double*)ws.ybuf.p, s);
        TGemm g2{m, CW * n, CW * rk, ws.l2p2.a.p + off, ws.l2p2.c.p + off, nullptr, (int64_t)CW * n, 0, (int64_t)CW * n};
        split_scratch(g2, ws);
        tgemm_f64<double, double>(g2, (const double*)ws.ybuf.p, op.tg_l2p2.p, (double*)ws.eq.p, s);
        ws.launches += 2;
      }
    }
    XCUDA(cudaEventRecord(ws.ev[6], s));
  }
};

template <class F>
void dispatch(const Fmm& f, F&& fn) {
  if (f.kernel == XFMM_LAPLACE) {
    if (f.mixed()) fn(Engine<K_LAPLACE, float>());
    else fn(Engine<K_LAPLACE, double>());
  } else if (f.kernel == XFMM_MODIFIED_HELMHOLTZ) {
    if (f.mixed()) fn(Engine<K_YUKAWA, float>());
    else fn(Engine<K_YUKAWA, double>());
  } else {
    if (f.mixed()) fn(Engine<K_HELMHOLTZ, float>());
    else fn(Engine<K_HELMHOLTZ, double>());
  }
}

void check_ready(const Fmm& f, const Tree& t) {
  XREQUIRE(t.lists_built, XFMM_ERR_STATE, "evaluate before build_list");
  XREQUIRE(t.m2l_ready, XFMM_ERR_STATE, "evaluate before M2L_setup");
  XREQUIRE(f.precomputed, XFMM_ERR_STATE, "evaluate before precompute");
  XREQUIRE(f.pre_r0 == t.r0 || f.kernel == XFMM_LAPLACE, XFMM_ERR_STATE,
           "operators were precomputed for another root radius");
  XREQUIRE(f.kernel == XFMM_LAPLACE || f.pre_depth >= t.depth, XFMM_ERR_STATE,
           "operators were precomputed for a shallower tree");
  XREQUIRE(t.nsurf_lists == f.nsurf, XFMM_ERR_STATE, "lists were built for another expansion order");
  XREQUIRE((t.m2l_grouped_by_level != 0) == (f.kernel != XFMM_LAPLACE), XFMM_ERR_STATE,
           "M2L_setup was done for another kernel family");
}

}  // namespace

// ================================================================ public (internal API)
void m2l_fragments(LevelOps& op, const double* T64, int nfreq, bool mixed, bool screened, cudaStream_t s) {
  static std::atomic<uint64_t> tables{0};
  op.m2l_id = ++tables;
  if (!mixed) {
    op.m2l_frag.alloc((size_t)nfreq * HAD64_B * sizeof(double));
    k_m2l_fragments64<<<nblk(26ll * nfreq * 32), 256, 0, s>>>((const double2*)T64, nfreq, (double*)op.m2l_frag.p);
    XLAUNCH();
    return;
  }
  DBuf<uint8_t> pwin;
  op.m2l_windows = 1;
  if (screened) {  // every child pair's window (k_m2l_fragments)
    DBuf<unsigned> pmax(26 * 64);
    XCUDA(cudaMemsetAsync(pmax.p, 0, pmax.bytes(), s));
    k_pair_max<<<dim3(std::min((nfreq + 3) / 4, 64), 26), 256, 0, s>>>((const double2*)T64, nfreq, pmax.p);
    XLAUNCH();
    const std::vector<unsigned> hm = pmax.download(s);  // the bits of floats >= 0
    std::vector<uint8_t> hw(26 * 64, 255);              // 255: no factors, or below the FP32 range
    for (int i = 0; i < 26; i++) {
      const int top = (int)(*std::max_element(hm.begin() + 64 * i, hm.begin() + 64 * (i + 1)) >> 23);
      for (int k = 64 * i; k < 64 * (i + 1); k++) {
        const int x = (int)(hm[k] >> 23);
        if (x == 0) continue;
        hw[k] = (uint8_t)((top - x) / SPLIT_WIN);
        op.m2l_windows = std::max(op.m2l_windows, (int)hw[k] + 1);
      }
    }
    pwin.upload(hw, s);
  }
  op.m2l_frag.alloc((size_t)op.m2l_windows * nfreq * HADH_FB * sizeof(uint4));
  op.m2l_binv.alloc((size_t)op.m2l_windows * nfreq * 32);
  k_m2l_fragments<<<dim3(nblk(26ll * nfreq * 32), op.m2l_windows), 256, 0, s>>>(
      (const double2*)T64, nfreq, pwin.p, screened ? SPLIT_TAIL : 1.0, (uint4*)op.m2l_frag.p, op.m2l_binv.p);
  XLAUNCH();
  if (screened) XCUDA(cudaStreamSynchronize(s));  // pwin is released here
}
void set_charges(Fmm& f, Tree& t, const double* q, bool on_device, cudaStream_t s) {
  const int64_t n = t.nsrc;
  const int vs = f.is_complex() ? 2 : 1;
  const double* dq = q;
  if (!on_device) {
    // host charges: copied to a grow-only staging buffer owned by the tree and checked there for
    // non-finite values before any of them replaces the current charges; the call returns once the
    // caller's buffer has been read
    t.stage_q.upload(q, n * vs, s);
    dq = t.stage_q.p;
    t.stage_flag.reserve(1);
    XCUDA(cudaMemsetAsync(t.stage_flag.p, 0, sizeof(int), s));
    k_count_nonfinite<<<std::max<int64_t>(1, std::min<int64_t>(nblk(n * vs), 4 * 148)), 256, 0, s>>>(
        dq, n * vs, t.stage_flag.p);
    XLAUNCH();
    int bad = 0;
    XCUDA(cudaMemcpyAsync(&bad, t.stage_flag.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    XCUDA(cudaStreamSynchronize(s));
    if (bad) throw Error(XFMM_ERR_NUMERIC, "non-finite value in charges");
  }
  k_set_charges<<<nblk(n), 256, 0, s>>>(dq, t.src_perm.p, n, f.is_complex(), t.src4.p, t.src_qim.p);
  XLAUNCH();
}

void clear_values(Fmm& f, Tree& t, cudaStream_t s) {
  check_ready(f, t);
  Workspace& ws = workspace(f, t, s);
  XCUDA(cudaMemsetAsync(ws.up.p, 0, ws.up.bytes(), s));
  XCUDA(cudaMemsetAsync(ws.dn.p, 0, ws.dn.bytes(), s));
}

void upward_pass(Fmm& f, Tree& t, cudaStream_t s) {
  check_ready(f, t);
  Workspace& ws = workspace(f, t, s);
  dispatch(f, [&](auto e) { decltype(e)::upward(f, t, ws, s); });
}

void downward_pass(Fmm& f, Tree& t, cudaStream_t s) {
  check_ready(f, t);
  Workspace& ws = workspace(f, t, s);
  dispatch(f, [&](auto e) { decltype(e)::downward(f, t, ws, s); });
}

// ================================================================ many systems in one evaluate
// Persistent near field over the target leaves of every system of a batch: each warp takes work items
// (system, target leaf) from one queue (a global counter, zeroed before the launch) in the order of
// `items` (largest pair count first) until it runs dry.  tpl: the largest number of targets a lane holds
// (1 or 2), the height of the warp's target tile.
__global__ void __launch_bounds__(128, XFMM_NEARF2_MINB)
    k_near_lap_f2_queue(const NearArgs* __restrict__ args, const int2* __restrict__ items, int64_t nitems,
                        unsigned int* __restrict__ counter, int tpl) {
  __shared__ NearSmemF2 sm[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (;;) {
    unsigned int k = 0;
    if (lane == 0) k = atomicAdd(counter, 1u);
    k = __shfl_sync(0xffffffffu, k, 0);
    if ((int64_t)k >= nitems) break;
    const int2 it = items[k];
    const NearArgs& a = args[it.x];
    const int node = a.leafs[a.eval_leafs[it.y]];
    const int T = a.ntrgs[node];
    if (T <= 32 || tpl == 1) near_leaf_lap_f2<1>(a, node, lane, sm[wid]);
    else near_leaf_lap_f2<2>(a, node, lane, sm[wid]);
    __syncwarp();
  }
}
template <int KER, class R>
__global__ void __launch_bounds__(128, XFMM_NEAR_MINB)
    k_near_queue(const NearArgs* __restrict__ args, const int2* __restrict__ items, int64_t nitems,
                 unsigned int* __restrict__ counter, int tpl) {
  __shared__ NearSmem<R> sm[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (;;) {
    unsigned int k = 0;
    if (lane == 0) k = atomicAdd(counter, 1u);
    k = __shfl_sync(0xffffffffu, k, 0);
    if ((int64_t)k >= nitems) break;
    const int2 it = items[k];
    const NearArgs& a = args[it.x];
    const int node = a.leafs[a.eval_leafs[it.y]];
    const int T = a.ntrgs[node];
    if (sizeof(R) == 4 && T > 32 && tpl >= 2) near_leaf<KER, R, 2>(a, node, lane, sm[wid]);
    else near_leaf<KER, R, 1>(a, node, lane, sm[wid]);
    __syncwarp();
  }
}
// pairs of one system, tagged with its index in .w, appended to a batch list
__global__ void k_tag_pairs(const int4* __restrict__ src, int64_t n, int sys, int4* __restrict__ dst) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) {
    int4 v = src[k];
    v.w = sys;
    dst[k] = v;
  }
}

struct Batch {
  Uses uses;
  std::vector<Fmm*> fmm;
  std::vector<Tree*> tree;
  int kernel = 0, precision = 0;
  DBuf<NearArgs> args;
  DBuf<int2> items;
  int64_t nitems = 0;
  DBuf<unsigned int> counter;
  DBuf<int4> close;
  int64_t nclose = 0;
  std::vector<int> order;  // systems, most bodies first (dealt to the streams in this order)
  std::vector<cudaStream_t> streams;
  std::vector<cudaEvent_t> events;
  int near_ctas_per_sm = 0, near_tpl = 2;  // tuning (0: the kernel's resident limit)
  // mixed Laplace systems sharing one operator table: the M2L Hadamard of every system in one launch
  bool had_batched = false;
  const LevelOps* had_op = nullptr;
  int had_nfreq = 0, had_tpc = HADH_TPC, nhtiles = 0;
  DBuf<HadSys> hsys;
  DBuf<int2> htiles;
  // with the shared table also the M2M and L2L of every system, per level one GEMM over all systems' rows
  std::vector<GemmRows> bm2m, bl2l;  // row offsets rebased onto system 0's up / dn arrays
  DBuf<double> bscratch;             // FP64 scratch of their split K (zero between uses)
  GemmRows bp2m1, bp2m2, bl2p1, bl2p2;  // P2M and L2P pseudo-inverse factors of every system's leaves
  int* bstatus = nullptr;            // system 0's device status flag (bounded waits)
  // mixed Laplace: the far field of every system as one persistent launch over (system, leaf) items
  DBuf<EvalArgs> fargs;
  DBuf<int2> fitems;
  int64_t nfitems = 0;
  DBuf<unsigned int> fcounter;
  ~Batch() {
    for (auto e : events) cudaEventDestroy(e);
    for (auto st : streams) cudaStreamDestroy(st);
  }
};

Batch* batch_create(Fmm** fmms, Tree** trees, int n, cudaStream_t s) {
  XREQUIRE(n > 0, XFMM_ERR_ARG, "a batch needs at least one system");
  auto* b = new Batch();
  try {
    b->kernel = fmms[0]->kernel;
    b->precision = fmms[0]->precision;
    std::vector<NearArgs> hargs(n);
    std::vector<std::pair<int64_t, int2>> work;
    std::vector<int64_t> bodies(n);
    for (int k = 0; k < n; k++) {
      Fmm& f = *fmms[k];
      Tree& t = *trees[k];
      XREQUIRE(f.kernel == b->kernel && f.precision == b->precision, XFMM_ERR_ARG,
               "the systems of a batch share one kernel and one precision");
      check_ready(f, t);
      Workspace& ws = workspace(f, t, s);
      b->fmm.push_back(&f);
      b->tree.push_back(&t);
      dispatch(f, [&](auto e) { hargs[k] = decltype(e)::near_args(f, t, ws); });
      bodies[k] = t.ntrg;
      // work items: target leaves, costed by their pair counts
      std::vector<int64_t> poff = t.p2p_off.download(s);
      std::vector<int> pl = t.p2p.download(s, (size_t)t.np2p);
      std::vector<int> el = t.eval_leafs.download(s, (size_t)t.n_eval_leafs);
      for (int i = 0; i < t.n_eval_leafs; i++) {
        const int node = t.h_leafs[el[i]];
        int64_t ns = 0;
        for (int64_t e = poff[node]; e < poff[node + 1]; e++) ns += t.h_nsrcs[pl[e]];
        work.push_back({(int64_t)t.h_ntrgs[node] * ns, make_int2(k, i)});
      }
      if (f.kernel == XFMM_LAPLACE && f.mixed() && ws.n_close < 0 && t.n_eval_leafs > 0)
        find_close_pairs(ws, hargs[k], t.n_eval_leafs, s);
      if (f.kernel == XFMM_LAPLACE && f.mixed()) b->nclose += std::max<int64_t>(ws.n_close, 0);
    }
    if (b->kernel == XFMM_LAPLACE && b->precision == XFMM_MIXED) {
      // far-field items: evaluation leaves costed by targets x surface points evaluated (own + W list)
      std::vector<EvalArgs> fa(n);
      std::vector<std::pair<int64_t, int2>> fw;
      for (int k = 0; k < n; k++) {
        Fmm& f = *fmms[k];
        Tree& t = *trees[k];
        Workspace& ws = workspace(f, t, s);
        fa[k] = Engine<K_LAPLACE, float>::far_args(f, t, ws);
        std::vector<int64_t> moff = t.m2p_off.download(s);
        std::vector<int> el = t.eval_leafs.download(s, (size_t)t.n_eval_leafs);
        for (int i = 0; i < t.n_eval_leafs; i++) {
          const int node = t.h_leafs[el[i]];
          fw.push_back({(int64_t)t.h_ntrgs[node] * f.nsurf * (1 + moff[node + 1] - moff[node]), make_int2(k, i)});
        }
      }
      std::stable_sort(fw.begin(), fw.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
      std::vector<int2> fi(fw.size());
      for (size_t i = 0; i < fw.size(); i++) fi[i] = fw[i].second;
      b->nfitems = (int64_t)fi.size();
      if (!fi.empty()) b->fitems.upload(fi, s);
      b->fargs.upload(fa, s);
      b->fcounter.alloc(1);
    }
    std::stable_sort(work.begin(), work.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    std::vector<int2> items(work.size());
    for (size_t i = 0; i < work.size(); i++) items[i] = work[i].second;
    b->nitems = (int64_t)items.size();
    b->items.upload(items, s);
    b->args.upload(hargs, s);
    b->counter.alloc(1);
    if (b->nclose > 0) {
      b->close.alloc((size_t)b->nclose);
      int64_t off = 0;
      for (int k = 0; k < n; k++) {
        Workspace& ws = *trees[k]->ws[fmms[k]->precision];
        if (ws.n_close <= 0) continue;
        k_tag_pairs<<<nblk(ws.n_close, 256), 256, 0, s>>>(ws.close_pairs.p, ws.n_close, k, b->close.p + off);
        XLAUNCH();
        off += ws.n_close;
      }
    }
    // one operator table for every system (one Fmm), mixed Laplace (one M2L group): the Hadamard
    // tiles of all systems as one list
    bool shared = b->kernel == XFMM_LAPLACE && b->precision == XFMM_MIXED;
    for (int k = 1; k < n && shared; k++) shared = fmms[k] == fmms[0];
    if (shared) {
      std::vector<HadSys> hs(n);
      std::vector<int2> tl;
      for (int k = 0; k < n; k++) {
        Tree& t = *trees[k];
        Workspace& ws = *t.ws[fmms[k]->precision];
        HadSys& h = hs[k];
        h = HadSys{};
        if (t.n_m2l_trg == 0 || t.m2l_src_off.size() != 2) continue;
        h = Engine<K_LAPLACE, float>::had_sys(ws, 0, t.m2l_src_off[1] - t.m2l_src_off[0],
                                              t.m2l_trg_off[1] - t.m2l_trg_off[0]);
        for (int j = 0; j < ws.had_tile0[1] - ws.had_tile0[0]; j++) tl.push_back(make_int2(k, j));
      }
      // per-level translations over all systems' rows: offsets rebased onto system 0's up / dn arrays (every
      // system's arrays are separate allocations, 256-byte aligned: the rebased offsets keep 16-byte rows).
      // A rebased offset reaches from system 0's array into another system's allocation: this relies on the
      // device's single flat address space (every allocation of the context is addressed from one base),
      // not on C++ pointer rules, and the offsets are only ever applied on the device.
      int maxd = 0;
      for (int k = 0; k < n; k++) maxd = std::max(maxd, trees[k]->depth);
      const int prec = fmms[0]->precision, ns = fmms[0]->nsurf;
      Workspace& w0 = *trees[0]->ws[prec];
      const float* up0 = (const float*)w0.up.p;
      const float* dn0 = (const float*)w0.dn.p;
      b->bm2m.resize(maxd);
      b->bl2l.resize(maxd);
      int64_t need = 0;
      for (int l = 0; l < maxd; l++) {
        std::vector<int64_t> ma, mc, la, lc;
        for (int k = 0; k < n; k++) {
          Tree& t = *trees[k];
          Workspace& ws = *t.ws[prec];
          if (l >= t.depth) continue;
          const int64_t du = (const float*)ws.up.p - up0, dd = (const float*)ws.dn.p - dn0;
          const GemmRows& gm = ws.m2m[l];
          const GemmRows& gl = ws.l2l[l];
          if (gm.M > 0) {
            const std::vector<int64_t> a = gm.a.download(s, (size_t)gm.M), c = gm.c.download(s, (size_t)gm.M);
            for (int i = 0; i < gm.M; i++) {
              ma.push_back(a[i] + du);
              mc.push_back(c[i] + du);
            }
          }
          if (gl.M > 0) {
            const std::vector<int64_t> a = gl.a.download(s, (size_t)gl.M), c = gl.c.download(s, (size_t)gl.M);
            for (int i = 0; i < gl.M; i++) {
              la.push_back(a[i] + dd);
              lc.push_back(c[i] + dd);
            }
          }
        }
        upload_rows<double>(b->bm2m[l], ma, mc, std::vector<double>(ma.size(), 1.0), s);
        upload_rows<double>(b->bl2l[l], la, lc, std::vector<double>(la.size(), 1.0), s);
        need = std::max(need, tgemm_tc_scratch((int)ma.size(), ns, 8 * ns, 1));
        need = std::max(need, tgemm_tc_scratch((int)la.size(), 8 * ns, ns, 1));
      }
      // the pseudo-inverse factors of P2M and L2P over every system's leaves (one leaf group for Laplace):
      // A and C offsets rebased onto system 0's arrays, each in its own element unit
      {
        auto rel = [](const DBuf<char>& x, const DBuf<char>& x0, size_t es) {
          return (int64_t)((x.p - x0.p) / (int64_t)es);
        };
        std::vector<int64_t> a1, c1, a2, c2, la1, lc1, la2, lc2;
        std::vector<double> al2, lal1;
        for (int k = 0; k < n; k++) {
          Workspace& ws = *trees[k]->ws[prec];
          const int64_t dchk = rel(ws.chk, w0.chk, sizeof(float)), dy = rel(ws.ybuf, w0.ybuf, sizeof(double)),
                        dup = rel(ws.up, w0.up, sizeof(float)), ddn = rel(ws.dn, w0.dn, sizeof(float)),
                        deq = rel(ws.eq, w0.eq, sizeof(double));
          auto take = [&](const GemmRows& g, int64_t da, int64_t dc, std::vector<int64_t>& va,
                          std::vector<int64_t>& vc, std::vector<double>* val) {
            if (g.M <= 0) return;
            const std::vector<int64_t> a = g.a.download(s, (size_t)g.M), c = g.c.download(s, (size_t)g.M);
            std::vector<double> al;
            if (val) al = g.al64.download(s, (size_t)g.M);
            for (int i = 0; i < g.M; i++) {
              va.push_back(a[i] + da);
              vc.push_back(c[i] + dc);
              if (val) val->push_back(al[i]);
            }
          };
          XREQUIRE(ws.p2m1.M == ws.p2m2.M && ws.l2p1.M == ws.l2p2.M, XFMM_ERR_STATE,
                   "pseudo-inverse factor rows differ");
          take(ws.p2m1, dchk, dy, a1, c1, nullptr);
          take(ws.p2m2, dy, dup, a2, c2, &al2);
          take(ws.l2p1, ddn, dy, la1, lc1, nullptr);
          // L2P's first factor takes its per-row scale from the second factor's rows (as in the evaluate)
          take(ws.l2p2, dy, deq, la2, lc2, &lal1);
        }
        upload_rows<double>(b->bp2m1, a1, c1, std::vector<double>(a1.size(), 1.0), s);
        upload_rows<double>(b->bp2m2, a2, c2, al2, s);
        upload_rows<double>(b->bl2p1, la1, lc1, lal1, s);
        upload_rows<double>(b->bl2p2, la2, lc2, std::vector<double>(la2.size(), 1.0), s);
        need = std::max(need, tgemm_tc_scratch((int)la1.size(), fmms[0]->ops[0].rank, ns, 0));
      }
      if (need > 0) {
        b->bscratch.alloc((size_t)need);
        XCUDA(cudaMemsetAsync(b->bscratch.p, 0, b->bscratch.bytes(), s));
      }
      b->bstatus = w0.status.p;
      b->had_batched = true;
      b->had_op = &fmms[0]->ops[0];
      b->had_nfreq = fmms[0]->nfreq;
      b->nhtiles = (int)tl.size();
      b->hsys.upload(hs, s);
      if (!tl.empty()) b->htiles.upload(tl, s);
      XREQUIRE(b->had_nfreq < 65536, XFMM_ERR_UNSUPPORTED, "too many frequencies for the Hadamard grid");
      XCUDA(cudaFuncSetAttribute(k_hadamard_h_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HADH_SMEM));
    }
    b->order.resize(n);
    for (int k = 0; k < n; k++) b->order[k] = k;
    std::stable_sort(b->order.begin(), b->order.end(), [&](int x, int y) { return bodies[x] > bodies[y]; });
    XCUDA(cudaStreamSynchronize(s));
  } catch (...) {
    delete b;
    throw;
  }
  return b;
}

// The batch's own buffers were written when it was created, and its evaluates use them with the systems'.
void batch_free(Batch* b) {
  if (!b) return;
  FreeScope free(b->uses);
  delete b;
}
std::vector<Uses*> batch_uses(Batch* b) {
  std::vector<Uses*> u{&b->uses};
  for (size_t k = 0; k < b->fmm.size(); k++) u.insert(u.end(), {&b->fmm[k]->uses, &b->tree[k]->uses});
  return u;
}

void batch_schedule(const int64_t* sizes, int n, int nstreams, int* stream_of) {
  XREQUIRE(n >= 0 && nstreams >= 1, XFMM_ERR_ARG, "batch schedule needs n >= 0 and nstreams >= 1");
  std::vector<int> order(n);
  for (int k = 0; k < n; k++) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return sizes[x] > sizes[y]; });
  std::vector<int64_t> load(std::max(1, std::min(nstreams, std::max(n, 1))), 0);
  for (int k : order) {
    const int j = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    stream_of[k] = j;
    load[j] += sizes[k];
  }
}

void batch_set_tuning(Batch* b, int option, int value) {
  if (option == XFMM_BATCH_NEAR_CTAS_PER_SM) {
    XREQUIRE(value >= 0 && value <= 32, XFMM_ERR_ARG, "CTAs per SM out of range (0..32)");
    b->near_ctas_per_sm = value;
  } else if (option == XFMM_BATCH_NEAR_TARGETS_PER_LANE) {
    XREQUIRE(value == 1 || value == 2, XFMM_ERR_ARG, "targets per lane must be 1 or 2");
    b->near_tpl = value;
  } else if (option == XFMM_BATCH_HADAMARD_TILES_PER_CTA) {
    XREQUIRE(value >= 0 && value <= 64, XFMM_ERR_ARG, "Hadamard tiles per CTA must be 0..64");
    b->had_tpc = value > 0 ? value : HADH_TPC;
  } else {
    XREQUIRE(false, XFMM_ERR_ARG, "unknown batch tuning option");
  }
}

// One evaluate of every system: charges (device, caller's order; null: keep the current ones) in,
// potentials and gradients out (device, caller's order).  The per-system stages before and after the
// near field run on `nstreams` streams forked from s (systems dealt largest first, each to the stream
// with the fewest bodies so far); the near field of all systems is one persistent launch on s.
void batch_evaluate(Batch* b, const double* const* charges, double* const* outs, int nstreams, cudaStream_t s) {
  const int n = (int)b->fmm.size();
  nstreams = std::max(1, std::min(nstreams, n));
  while ((int)b->streams.size() < nstreams) {
    cudaStream_t st;
    XCUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    b->streams.push_back(st);
  }
  while (b->events.size() < (size_t)5 * (nstreams + 1)) {
    cudaEvent_t e;
    XCUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    b->events.push_back(e);
  }
  std::vector<int64_t> sizes(n);
  for (int k = 0; k < n; k++) sizes[k] = b->tree[k]->ntrg;
  std::vector<int> stream_of(n);
  batch_schedule(sizes.data(), n, nstreams, stream_of.data());
  std::vector<std::vector<int>> lists(nstreams);
  for (int k : b->order) lists[stream_of[k]].push_back(k);
  auto fork_join = [&](int evbase, auto&& body) {
    if (nstreams == 1) {
      for (int k : lists[0]) body(k, s);
      return;
    }
    XCUDA(cudaEventRecord(b->events[evbase], s));
    for (int j = 0; j < nstreams; j++) {
      XCUDA(cudaStreamWaitEvent(b->streams[j], b->events[evbase], 0));
      for (int k : lists[j]) body(k, b->streams[j]);
      XCUDA(cudaEventRecord(b->events[evbase + 1 + j], b->streams[j]));
      XCUDA(cudaStreamWaitEvent(s, b->events[evbase + 1 + j], 0));
    }
  };
  // before the near field: upward pass, P2L, M2L and L2L per system.  With one shared operator table (mixed
  // Laplace) the parts that share it run as one launch over all systems: the M2M and L2L of each level, and
  // the M2L Hadamard between the systems' forward and backward transforms.
  const int E = nstreams + 1;
  Fmm& f0 = *b->fmm[0];
  auto per_system = [&](int evbase, int up_parts, int pre_parts, bool first) {
    fork_join(evbase, [&](int k, cudaStream_t st) {
      Fmm& f = *b->fmm[k];
      Tree& t = *b->tree[k];
      if (first) {
        if (charges && charges[k]) set_charges(f, t, charges[k], true, st);
        clear_values(f, t, st);
      }
      Workspace& ws = workspace(f, t, st);
      dispatch(f, [&](auto e) {
        if (up_parts) decltype(e)::upward(f, t, ws, st, up_parts);
        if (pre_parts) decltype(e)::downward(f, t, ws, st, DOWN_PRE, pre_parts);
      });
    });
  };
  auto batched_tr = [&](const GemmRows& g, bool m2m) {
    if (g.M <= 0) return;
    const int nn = f0.nsurf;
    const LevelOps& op = f0.ops[0];
    float* up0 = (float*)b->tree[0]->ws[f0.precision]->up.p;
    float* dn0 = (float*)b->tree[0]->ws[f0.precision]->dn.p;
    TGemm gg = m2m ? TGemm{g.M, nn, 8 * nn, g.a.p, g.c.p, nullptr, (int64_t)nn, 1, (int64_t)nn}
                   : TGemm{g.M, 8 * nn, nn, g.a.p, g.c.p, nullptr, (int64_t)8 * nn, 1, (int64_t)nn};
    gg.status = b->bstatus;
    gg.scratch = b->bscratch.p;
    gg.scratch_len = (int64_t)b->bscratch.n;
    if (m2m) tgemm_tc<float>(gg, up0, op.tg_m2m_h.p, op.tg_m2m_l.p, op.ld_m2m, up0, s);
    else tgemm_tc<float>(gg, dn0, op.tg_l2l_h.p, op.tg_l2l_l.p, op.ld_l2l, dn0, s);
  };
  if (!b->had_batched) {
    per_system(0, UP_ALL, PRE_ALL, true);
  } else {
    Workspace& w0 = *b->tree[0]->ws[f0.precision];
    const int nn = f0.nsurf, rk = f0.ops[0].rank;
    const LevelOps& op = f0.ops[0];
    per_system(0, UP_CHK, 0, true);
    if (b->bp2m1.M > 0) {  // P2M's pseudo-inverse factors of every system's leaves
      TGemm g1{b->bp2m1.M, rk, nn, b->bp2m1.a.p, b->bp2m1.c.p, nullptr, (int64_t)nn, 0, (int64_t)nn};
      tgemm_f64<float, double>(g1, (const float*)w0.chk.p, op.tg_p2m1.p, (double*)w0.ybuf.p, s);
      TGemm g2{b->bp2m2.M, nn, rk, b->bp2m2.a.p, b->bp2m2.c.p, b->bp2m2.al64.p, (int64_t)nn, 0, (int64_t)nn};
      tgemm_f64<double, float>(g2, (const double*)w0.ybuf.p, op.tg_p2m2.p, (float*)w0.up.p, s);
    }
    for (int l = (int)b->bm2m.size() - 1; l >= 0; l--) batched_tr(b->bm2m[l], true);
    per_system(E, 0, M2L_FWD | M2L_HAD_DENSE, false);
    if (b->nhtiles > 0) {
      const int tpc = std::max(1, b->had_tpc);
      k_hadamard_h_batch<<<dim3((b->nhtiles + tpc - 1) / tpc, b->had_nfreq), HADH_NT, HADH_SMEM, s>>>(
          (const uint4*)b->had_op->m2l_frag.p, b->had_op->m2l_binv.p, b->hsys.p, b->htiles.p, b->nhtiles, tpc);
      XLAUNCH();
    }
    per_system(2 * E, 0, M2L_BWD, false);
    for (int l = 0; l < (int)b->bl2l.size(); l++) batched_tr(b->bl2l[l], false);
    if (b->bl2p1.M > 0) {  // L2P's check-to-equivalent factors of every system's leaves
      TGemm g1{b->bl2p1.M, rk, nn, b->bl2p1.a.p, b->bl2p1.c.p, b->bl2p1.al64.p, (int64_t)nn, 0, (int64_t)nn};
      g1.status = b->bstatus;
      g1.scratch = b->bscratch.p;
      g1.scratch_len = (int64_t)b->bscratch.n;
      tgemm_tc<double>(g1, (const float*)w0.dn.p, op.tg_l2p1_h.p, op.tg_l2p1_l.p, op.ld_l2p1, (double*)w0.ybuf.p, s);
      TGemm g2{b->bl2p2.M, nn, rk, b->bl2p2.a.p, b->bl2p2.c.p, nullptr, (int64_t)nn, 0, (int64_t)nn};
      tgemm_f64<double, double>(g2, (const double*)w0.ybuf.p, op.tg_l2p2.p, (double*)w0.eq.p, s);
    }
  }
  // the near field of every system: one persistent launch draining the work queue
  if (b->nitems > 0) {
    int dev = 0, nsm = 148;
    XCUDA(cudaGetDevice(&dev));
    XCUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    XCUDA(cudaMemsetAsync(b->counter.p, 0, sizeof(unsigned int), s));
    const bool lapf2 = b->kernel == XFMM_LAPLACE && b->precision == XFMM_MIXED;
    auto launch = [&](auto kern) {
      int per_sm = 0;
      XCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, 0));
      if (b->near_ctas_per_sm > 0) per_sm = std::min(per_sm, b->near_ctas_per_sm);
      const int64_t need = (b->nitems + 3) / 4;
      const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::max(per_sm, 1) * nsm, need));
      kern<<<grid, 128, 0, s>>>(b->args.p, b->items.p, b->nitems, b->counter.p, b->near_tpl);
      XLAUNCH();
    };
    if (lapf2) launch(k_near_lap_f2_queue);
    else if (b->kernel == XFMM_LAPLACE) launch(k_near_queue<K_LAPLACE, double>);
    else if (b->kernel == XFMM_MODIFIED_HELMHOLTZ)
      b->precision == XFMM_MIXED ? launch(k_near_queue<K_YUKAWA, float>) : launch(k_near_queue<K_YUKAWA, double>);
    else
      b->precision == XFMM_MIXED ? launch(k_near_queue<K_HELMHOLTZ, float>) : launch(k_near_queue<K_HELMHOLTZ, double>);
    if (lapf2 && b->nclose > 0) {
      NearArgs none{};
      k_close_fix<<<nblk(b->nclose, 256), 256, 0, s>>>(b->close.p, b->nclose, none, b->args.p);
      XLAUNCH();
    }
  }
  // the far field (one persistent launch over every system's leaves for mixed Laplace), then the results
  const bool far_queue = b->nfitems > 0;
  if (far_queue) {
    int dev = 0, nsm = 148, per_sm = 0;
    XCUDA(cudaGetDevice(&dev));
    XCUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    order_dispatch(f0.p, [&](auto pc) {
      constexpr int PP = decltype(pc)::value;
      const size_t smem = far_smem(f0.nsurf, PP);
      XCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_far_lap_queue<float, PP>, 32 * EVAL_WARPS, smem));
      const int grid = (int)std::max<int64_t>(
          1, std::min<int64_t>((int64_t)std::max(per_sm, 1) * nsm, (b->nfitems + EVAL_WARPS - 1) / EVAL_WARPS));
      XCUDA(cudaMemsetAsync(b->fcounter.p, 0, sizeof(unsigned int), s));
      k_far_lap_queue<float, PP>
          <<<grid, 32 * EVAL_WARPS, smem, s>>>(b->fargs.p, b->fitems.p, b->nfitems, b->fcounter.p);
    });
    XLAUNCH();
  }
  fork_join(4 * E, [&](int k, cudaStream_t st) {
    Fmm& f = *b->fmm[k];
    Tree& t = *b->tree[k];
    Workspace& ws = workspace(f, t, st);
    if (!far_queue) dispatch(f, [&](auto e) { decltype(e)::downward(f, t, ws, st, DOWN_FAR); });
    get_values(f, t, outs[k], st);
  });
}

// Device times of the last upward + downward pass (ms): 0 P2M, 1 M2M, 2 P2L, 3 M2L, 4 L2L,
// 5 L2P check->equivalent, 6 target evaluation (P2P + M2P + L2P), 7 total, 8-10 M2L FFT / Hadamard / iFFT.
namespace {
// An mbarrier (expecting one arrival) whose phase nothing completes; the wait runs out after `limit`
// cycles and the kernel reports it through *status, as the pipelined kernels do.
__global__ void k_selftest_wait(long long limit, int* status) {
  __shared__ __align__(8) uint64_t bar;
  const uint32_t b = tc5::smem_u32(&bar);
  if (threadIdx.x == 0) {
    tc5::mbar_init(b, 1);
    tc5::fence_mbar_init();
  }
  __syncthreads();
  const bool ok = __all_sync(0xffffffffu, tc5::mbar_wait(b, 0, limit));
  if (!ok && threadIdx.x == 0) atomicExch(status, 1);
}
}  // namespace

void selftest_bounded_wait(int64_t limit_cycles) {
  XREQUIRE(limit_cycles >= 1 && limit_cycles <= 1000000000LL, XFMM_ERR_ARG, "limit_cycles outside 1..1e9");
  DBuf<int> status(1);
  XCUDA(cudaMemset(status.p, 0, sizeof(int)));
  k_selftest_wait<<<1, 32>>>(limit_cycles, status.p);
  XLAUNCH();
  XCUDA(cudaDeviceSynchronize());
  int h = 0;
  XCUDA(cudaMemcpy(&h, status.p, sizeof(int), cudaMemcpyDeviceToHost));
  XREQUIRE(!h, XFMM_ERR_TIMEOUT, "bounded device-side wait ran out (self-test)");
}

// After the caller's stream has been synchronised: XFMM_ERR_TIMEOUT when a bounded device-side wait of the
// last pass ran out (the flag is cleared for the next pass).
void check_device_status(Fmm& f, Tree& t) {
  Workspace* ws = t.ws[f.precision];
  if (!ws) return;
  int dev_status = 0;
  XCUDA(cudaMemcpy(&dev_status, ws->status.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (dev_status) {
    XCUDA(cudaMemset(ws->status.p, 0, sizeof(int)));
    XREQUIRE(false, XFMM_ERR_TIMEOUT, "a bounded device-side wait ran out in the last pass (results incomplete)");
  }
}

void stage_times(Fmm& f, Tree& t, double* ms14) {
  Workspace* ws = t.ws[f.precision];
  XREQUIRE(ws, XFMM_ERR_STATE, "no evaluate has run");
  XCUDA(cudaEventSynchronize(ws->ev[7]));
  int dev_status = 0;
  XCUDA(cudaMemcpy(&dev_status, ws->status.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (dev_status) {
    XCUDA(cudaMemset(ws->status.p, 0, sizeof(int)));
    XREQUIRE(false, XFMM_ERR_TIMEOUT, "a bounded device-side wait ran out in the last pass (results incomplete)");
  }
  auto el = [](cudaEvent_t a, cudaEvent_t b) {
    float ms = 0;
    return cudaEventElapsedTime(&ms, a, b) == cudaSuccess ? (double)ms : 0.0;
  };
  const int pairs[8][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 4}, {4, 5}, {5, 6}, {6, 7}, {0, 7}};
  for (int i = 0; i < 8; i++) ms14[i] = el(ws->ev[pairs[i][0]], ws->ev[pairs[i][1]]);
  ms14[8] = ms14[9] = ms14[10] = 0;
  const int ng = (int)ws->m2l_ev.size() / 4;
  for (int g = 0; g < ng; g++) {
    const int ns = t.m2l_src_off[g + 1] - t.m2l_src_off[g], nt = t.m2l_trg_off[g + 1] - t.m2l_trg_off[g];
    if (ns == 0 || nt == 0) continue;
    cudaEvent_t* e = ws->m2l_ev.data() + 4 * g;
    ms14[8] += el(e[0], e[1]);
    ms14[9] += el(e[1], e[2]);
    ms14[10] += el(e[2], e[3]);
  }
  for (int i = 0; i < 11; i++) f.stage_ms[i] = ms14[i];
  ms14[11] = (double)ws->launches;
  ms14[12] = el(ws->ev[6], ws->ev[8]);  // near field (P2P)
  ms14[13] = el(ws->ev[8], ws->ev[7]);  // far field (M2P + L2P)
}

void get_values(Fmm& f, Tree& t, double* out_dev, cudaStream_t s) {
  Workspace& ws = workspace(f, t, s);
  const int width = 4 * (f.is_complex() ? 2 : 1);
  k_scatter_out<<<nblk(t.ntrg), 256, 0, s>>>(ws.out.p, t.trg_perm.p, t.ntrg, width, out_dev);
  XLAUNCH();
  ws.launches++;
}

// xfmm_gradient_p2p: one "leaf" of all targets against one "leaf" of all sources
namespace {
struct RawP2P {
  DBuf<double4> s4, t4;
  DBuf<double> qim;
};
__global__ void k_pack_raw(const double* xyz, const double* q, int64_t n, int cplx, double4* out, double* qim) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_double4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], q ? (cplx ? q[2 * i] : q[i]) : 0.0);
  if (q && cplx) qim[i] = q[2 * i + 1];
}
template <int KER, class R>
__global__ void __launch_bounds__(128) k_raw_p2p(const double4* __restrict__ s4, const double* __restrict__ qim,
                                                  int64_t ns, const double4* __restrict__ t4, int64_t nt,
                                                  double k_re, double k_im, double* __restrict__ out) {
  using G = Green<KER, R>;
  using Q = typename G::Q;
  using A = typename Acc64<Q>::type;
  using V4 = typename R4<R>::type;
  __shared__ double4 sx[128];
  __shared__ Q sq[128];
  const G g{(R)k_re, (R)k_im};
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const double4 tv = t < nt ? t4[t] : make_double4(0, 0, 0, 0);
  A P, GX, GY, GZ;
  P = GX = GY = GZ = A();
  for (int64_t j0 = 0; j0 < ns; j0 += 128) {
    const int cnt = (int)(ns - j0 < 128 ? ns - j0 : 128);
    __syncthreads();
    if (threadIdx.x < cnt) {
      const double4 sv = s4[j0 + threadIdx.x];
      sx[threadIdx.x] = sv;
      sq[threadIdx.x] = load_charge<Q>(sv, qim, j0 + threadIdx.x);
    }
    __syncthreads();
    Q p = vzero<Q>(), gx = vzero<Q>(), gy = vzero<Q>(), gz = vzero<Q>();
    for (int j = 0; j < cnt; j++) {
      const double4 s = sx[j];  // differences in FP64, the kernel in R
      g.grad((R)(tv.x - s.x), (R)(tv.y - s.y), (R)(tv.z - s.z), sq[j], p, gx, gy, gz);
    }
    acc64(P, p);
    acc64(GX, gx);
    acc64(GY, gy);
    acc64(GZ, gz);
  }
  if (t < nt) {
    const int stride = (KER == K_HELMHOLTZ) ? 8 : 4, vs = stride / 4;
    double* o = out + t * stride;
    put_out(o, P, INV4PI, 1);
    put_out(o + vs, GX, INV4PI, 1);
    put_out(o + 2 * vs, GY, INV4PI, 1);
    put_out(o + 3 * vs, GZ, INV4PI, 1);
  }
}
}  // namespace

void gradient_p2p_raw(int kernel, double k_re, double k_im, int precision, const double* src, int64_t ns,
                      const double* q, const double* trg, int64_t nt, double* out, cudaStream_t s) {
  const int cplx = kernel == XFMM_HELMHOLTZ;
  RawP2P r;
  r.s4.alloc(std::max<int64_t>(ns, 1));
  r.t4.alloc(std::max<int64_t>(nt, 1));
  r.qim.alloc(std::max<int64_t>(ns, 1));
  k_pack_raw<<<nblk(ns), 256, 0, s>>>(src, q, ns, cplx, r.s4.p, r.qim.p);
  k_pack_raw<<<nblk(nt), 256, 0, s>>>(trg, nullptr, nt, 0, r.t4.p, nullptr);
  XLAUNCH();
  const int blocks = nblk(nt, 128);
  const bool m = precision == XFMM_MIXED;
  if (kernel == XFMM_LAPLACE) {
    if (m) k_raw_p2p<K_LAPLACE, float><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
    else k_raw_p2p<K_LAPLACE, double><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
  } else if (kernel == XFMM_MODIFIED_HELMHOLTZ) {
    if (m) k_raw_p2p<K_YUKAWA, float><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
    else k_raw_p2p<K_YUKAWA, double><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
  } else {
    if (m) k_raw_p2p<K_HELMHOLTZ, float><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
    else k_raw_p2p<K_HELMHOLTZ, double><<<blocks, 128, 0, s>>>(r.s4.p, r.qim.p, ns, r.t4.p, nt, k_re, k_im, out);
  }
  XLAUNCH();
  XCUDA(cudaStreamSynchronize(s));
}

// The evaluation of gradient_p2p_raw with the packed bodies in device scratch that the caller owns
// (s4: ns double4, qim: ns doubles, t4: nt double4, each 32-byte aligned).  Asynchronous on s; no
// allocation and no synchronisation.  The packing kernels write every scratch entry the P2P kernel
// reads, so the scratch needs no initial contents.
void gradient_p2p_scratch(int kernel, double k_re, double k_im, int precision, const double* src, int64_t ns,
                          const double* q, const double* trg, int64_t nt, double* out, double4* s4, double* qim,
                          double4* t4, cudaStream_t s) {
  const int cplx = kernel == XFMM_HELMHOLTZ;
  if (ns > 0) k_pack_raw<<<nblk(ns), 256, 0, s>>>(src, q, ns, cplx, s4, qim);
  k_pack_raw<<<nblk(nt), 256, 0, s>>>(trg, nullptr, nt, 0, t4, nullptr);
  XLAUNCH();
  const int blocks = nblk(nt, 128);
  const bool m = precision == XFMM_MIXED;
  if (kernel == XFMM_LAPLACE) {
    if (m) k_raw_p2p<K_LAPLACE, float><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
    else k_raw_p2p<K_LAPLACE, double><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
  } else if (kernel == XFMM_MODIFIED_HELMHOLTZ) {
    if (m) k_raw_p2p<K_YUKAWA, float><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
    else k_raw_p2p<K_YUKAWA, double><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
  } else {
    if (m) k_raw_p2p<K_HELMHOLTZ, float><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
    else k_raw_p2p<K_HELMHOLTZ, double><<<blocks, 128, 0, s>>>(s4, qim, ns, t4, nt, k_re, k_im, out);
  }
  XLAUNCH();
}

// FmmBase::verify (fmm_base.h:208-267) on the device: FP64 direct sum over all sources
void verify(Fmm& f, Tree& t, int sample, double* err2, cudaStream_t s) {
  Workspace& ws = workspace(f, t, s);
  std::vector<int> trg_leaves;
  if (sample) {
    const int stride = t.nleafs / 10;
    for (int i = 0; i < 10 && i * stride < t.nleafs; i++) trg_leaves.push_back(t.h_leafs[i * stride]);
  } else {
    trg_leaves = t.h_leafs;
  }
  std::vector<int64_t> tb = t.tbeg.download(s);
  std::vector<int64_t> rows;
  for (int node : trg_leaves)
    for (int k = 0; k < t.h_ntrgs[node]; k++) rows.push_back(tb[node] + k);
  const int cplx = f.is_complex();
  const int width = 4 * (cplx ? 2 : 1);
  std::vector<double4> htrg = t.trg4.download(s);
  std::vector<double> hout = ws.out.download(s);
  std::vector<double> txyz(3 * rows.size());
  for (size_t i = 0; i < rows.size(); i++) {
    txyz[3 * i] = htrg[rows[i]].x;
    txyz[3 * i + 1] = htrg[rows[i]].y;
    txyz[3 * i + 2] = htrg[rows[i]].z;
  }
  std::vector<double4> hsrc = t.src4.download(s);
  std::vector<double> hqim = t.src_qim.download(s);
  std::vector<double> sxyz(3 * t.nsrc), q(t.nsrc * (cplx ? 2 : 1));
  for (int64_t i = 0; i < t.nsrc; i++) {
    sxyz[3 * i] = hsrc[i].x;
    sxyz[3 * i + 1] = hsrc[i].y;
    sxyz[3 * i + 2] = hsrc[i].z;
    if (cplx) {
      q[2 * i] = hsrc[i].w;
      q[2 * i + 1] = hqim[i];
    } else {
      q[i] = hsrc[i].w;
    }
  }
  DBuf<double> ds, dq, dt, dout;
  ds.upload(sxyz, s);
  dq.upload(q, s);
  dt.upload(txyz, s);
  dout.alloc(std::max<size_t>(rows.size(), 1) * width);
  XCUDA(cudaMemsetAsync(dout.p, 0, dout.bytes(), s));
  gradient_p2p_raw(f.kernel, f.k_re, f.k_im, XFMM_FP64, ds.p, t.nsrc, dq.p, dt.p, (int64_t)rows.size(), dout.p, s);
  std::vector<double> ex = dout.download(s);
  double pd = 0, pn = 0, gd = 0, gn = 0;
  const int vs = cplx ? 2 : 1;
  for (size_t i = 0; i < rows.size(); i++)
    for (int c = 0; c < 4; c++)
      for (int v = 0; v < vs; v++) {
        const double e = ex[i * width + c * vs + v], a = hout[rows[i] * width + c * vs + v];
        (c == 0 ? pd : gd) += (e - a) * (e - a);
        (c == 0 ? pn : gn) += e * e;
      }
  err2[0] = std::sqrt(pd / pn);
  err2[1] = std::sqrt(gd / gn);
}

}  // namespace xfmm
