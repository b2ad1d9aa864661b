// CUDA kernels of libtwos.so (sm_100a).
//
//   wos_kernel       persistent walk-on-spheres: every lane runs one walk at a
//                    time and refills from a device work queue when its walk
//                    ends on the epsilon shell, so walks of very different
//                    lengths do not idle a warp.  Replaces the OpenMP site loop
//                    + evaluate_site/paired_site + walk of the reference
//                    (wih_twos.cpp:635-717, 1825-1841; adjoint.cpp:18-42).
//   nearest()        plain BVH closest-point query: nearest-child-first order,
//                    pruning on push and pop.  Replaces rtcPointQuery +
//                    point_query_callback (wih_twos.cpp:339-359, 416-430).
//                    nearest_geo() and the walk kernel run the same search in
//                    units with one set of loads for nodes and triangles;
//                    warp_search() takes one query with a whole warp.
//   finalize_kernel  one warp per site: FP64 U-statistic, means and the
//                    leave-one-out jackknife SE over the per-walk samples with
//                    warp-shuffle reductions in a fixed order (wih_twos.cpp:
//                    691-715; adjoint.cpp:36-41).
//   closest_kernel   batched closest point, a lane (or closest_warp_kernel: a
//                    warp) per point.
//   list_*_kernel    the candidate lists of the grid cells near the surface.
//   grid_build_kernel / grid_bound_kernel
//                    the mixed form's distance-bound grid: one FP32 closest-
//                    point query per grid vertex at mesh open, and the bound
//                    a walk step would use at given points.
//   topk kernels     block-local bitonic top-k then a merge block.
//
// Compiled with -fmad=false: FP64 arithmetic is evaluated exactly as written
// (no contraction), so it matches a plain IEEE FP64 evaluation on the host;
// the FP32 path asks for FMAs explicitly where it wants them.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>

#include "twos_internal.h"

namespace twos {

// ================================================================ random stream
// Philox4x32-10 (Salmon, Moraes, Dror & Shaw, "Parallel random numbers: as
// easy as 1, 2, 3", SC'11): counter = (step, walk, site, repeat*8 + block).
struct Philox4 {
  uint32_t x, y, z, w;
};

__device__ __forceinline__ Philox4 philox(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                          uint32_t c3) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
    const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return {c0, c1, c2, c3};
}

// Blocks c3, c3 + 1, .. c3 + N - 1 of one counter together, round by round: a
// step that draws several blocks spends a tenth of the instructions' bytes
// (the walk kernels' stalls on instruction fetch) and has N independent chains.
template <int N>
__device__ __forceinline__ void philox_blocks(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                              uint32_t c3, Philox4 (&q)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) q[i] = {c0, c1, c2, c3 + static_cast<uint32_t>(i)};
#pragma unroll 1
  for (int r = 0; r < 10; ++r) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint32_t lo0 = 0xD2511F53u * q[i].x, hi0 = __umulhi(0xD2511F53u, q[i].x);
      const uint32_t lo1 = 0xCD9E8D57u * q[i].z, hi1 = __umulhi(0xCD9E8D57u, q[i].z);
      q[i] = {hi1 ^ q[i].y ^ k0, lo1, hi0 ^ q[i].w ^ k1, lo0};
    }
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

// Uniforms in [0,1): FP64 takes the top 53 bits of (hi:lo); FP32 takes the
// top 24, i.e. the FP64 value truncated, so both forms share samples.
template <typename T> __device__ __forceinline__ T uniform(uint32_t hi, uint32_t lo);
template <> __device__ __forceinline__ double uniform<double>(uint32_t hi, uint32_t lo) {
  const uint64_t v = (static_cast<uint64_t>(hi) << 32) | lo;
  return static_cast<double>(v >> 11) * 0x1.0p-53;
}
template <> __device__ __forceinline__ float uniform<float>(uint32_t hi, uint32_t) {
  return static_cast<float>(hi >> 8) * 0x1.0p-24f;
}

template <typename T> struct Vec {
  T x, y, z;
};

__device__ __forceinline__ void sincos_pi(double a, double *s, double *c) { sincospi(a, s, c); }
__device__ __forceinline__ void sincos_pi(float a, float *s, float *c) { sincospif(a, s, c); }

// Uniform direction on S^2: z = 1 - 2a, phi = 2*pi*b (the parametrisation of
// random_unit_vector, wih_twos.cpp:536-542).
template <typename T> __device__ __forceinline__ Vec<T> direction(T a, T b) {
  const T z = T(1) - T(2) * a;
  const T zz = z * z;
  const T radial = sqrt(fmax(T(0), T(1) - zz));
  T s, c;
  sincos_pi(T(2) * b, &s, &c);
  return {radial * c, radial * s, z};
}

template <typename T> __device__ __forceinline__ T median3(T a, T b, T c) {
  return fmax(fmin(a, b), fmin(fmax(a, b), c));
}

// ================================================================ arithmetic helpers
// madd: FMA in FP32, plain multiply-add in FP64 (bit-identical to host FP64).
__device__ __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double madd(double a, double b, double c) { return a * b + c; }

__device__ __forceinline__ float dot3(const Vec<float> &a, const Vec<float> &b) {
  return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, a.z * b.z));
}
__device__ __forceinline__ double dot3(const Vec<double> &a, const Vec<double> &b) {
  return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <typename T> __device__ __forceinline__ Vec<T> sub(const Vec<T> &a, const Vec<T> &b) {
  return {a.x - b.x, a.y - b.y, a.z - b.z};
}
// a*b + c: one fused multiply-add in FP32 (the mixed form's arithmetic);
// separately rounded in FP64, so the plain form keeps the host's operations
// (the library is built without contraction).
template <typename T> __device__ __forceinline__ T mad_t(T a, T b, T c) { return a * b + c; }
template <> __device__ __forceinline__ float mad_t<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }

template <typename T> __device__ __forceinline__ Vec<T> add_scaled(const Vec<T> &a, const Vec<T> &d, T s) {
  return {mad_t(d.x, s, a.x), mad_t(d.y, s, a.y), mad_t(d.z, s, a.z)};
}

// Squared distance from p to the closest point of triangle (a, b, c):
// Ericson's Voronoi-region case analysis (Real-Time Collision Detection,
// 5.1.5), the algorithm of closest_point_triangle (wih_twos.cpp:247-289).
template <typename T>
__device__ __forceinline__ Vec<T> tri_closest(const Vec<T> &p, const Vec<T> &a, const Vec<T> &b, const Vec<T> &c) {
  const Vec<T> ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
  const T d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  Vec<T> q;
  if (d1 <= T(0) && d2 <= T(0)) {
    q = a;
  } else {
    const Vec<T> bp = sub(p, b);
    const T d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3 >= T(0) && d4 <= d3) {
      q = b;
    } else {
      const T vc = mad_t(d1, d4, -(d3 * d2));
      if (vc <= T(0) && d1 >= T(0) && d3 <= T(0)) {
        const T v = d1 / (d1 - d3);
        q = add_scaled(a, ab, v);
      } else {
        const Vec<T> cp = sub(p, c);
        const T d5 = dot3(ab, cp), d6 = dot3(ac, cp);
        if (d6 >= T(0) && d5 <= d6) {
          q = c;
        } else {
          const T vb = mad_t(d5, d2, -(d1 * d6));
          if (vb <= T(0) && d2 >= T(0) && d6 <= T(0)) {
            const T w = d2 / (d2 - d6);
            q = add_scaled(a, ac, w);
          } else {
            const T va = mad_t(d3, d6, -(d5 * d4));
            if (va <= T(0) && (d4 - d3) >= T(0) && (d5 - d6) >= T(0)) {
              const T w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
              q = add_scaled(b, sub(c, b), w);
            } else {
              const T denom = T(1) / (va + vb + vc);
              const T v = vb * denom, w = vc * denom;
              const Vec<T> t = add_scaled(a, ab, v);
              q = add_scaled(t, ac, w);
            }
          }
        }
      }
    }
  }
  return q;
}

template <typename T>
__device__ __forceinline__ T tri_dist2(const Vec<T> &p, const Vec<T> &a, const Vec<T> &b, const Vec<T> &c) {
  const Vec<T> d = sub(p, tri_closest(p, a, b, c));
  return dot3(d, d);
}

// ================================================================ BVH traversal
template <typename T> struct Layout;
template <> struct Layout<float> {
  using Node = NodeF;
  using Tri = TriF;
};
template <> struct Layout<double> {
  using Node = NodeD;
  using Tri = TriD;
};

__device__ __forceinline__ float gap(float lo, float hi, float p) { return fmaxf(fmaxf(lo - p, p - hi), 0.f); }
__device__ __forceinline__ double gap(double lo, double hi, double p) { return fmax(fmax(lo - p, p - hi), 0.0); }

// Lower bound on the squared distance from p to each child: the larger of
// the box bound and the normal-slab bound (the child's triangles lie between
// the planes n.x = smin and n.x = smax, so |n.p - [smin, smax]| bounds the
// distance from below; for a nearly flat patch the slab is thin and the
// bound is close to the true distance, where the box bound is off by up to
// the box size).
// 32-byte read-only load (two float4) of 32-byte aligned data: one L1
// request instead of two.
__device__ __forceinline__ void ldg32(const void *p, float4 &a, float4 &b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// ldg32 under a condition; a and b are left alone without it.
__device__ __forceinline__ void ldg32_if(bool cond, const void *p, float4 &a, float4 &b) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %9, 0;\n\t"
      "@q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
      : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w), "+f"(b.x), "+f"(b.y), "+f"(b.z), "+f"(b.w)
      : "l"(p), "r"(static_cast<int>(cond)));
}

// The bounds from a loaded node (its six float4 in order).
__device__ __forceinline__ void node_bounds(const float4 &x, const float4 &y, const float4 &z, const float4 &nl,
                                            const float4 &nr, const float4 &t, const Vec<float> &p, float &dl,
                                            float &dr, int &cl, int &cr) {
  const float lx = gap(x.x, x.z, p.x), rx = gap(x.y, x.w, p.x);
  const float ly = gap(y.x, y.z, p.y), ry = gap(y.y, y.w, p.y);
  const float lz = gap(z.x, z.z, p.z), rz = gap(z.y, z.w, p.z);
  const float sl = __fmaf_rn(nl.x, p.x, __fmaf_rn(nl.y, p.y, nl.z * p.z));
  const float sr = __fmaf_rn(nr.x, p.x, __fmaf_rn(nr.y, p.y, nr.z * p.z));
  const float gl = gap(nl.w, t.x, sl), gr = gap(nr.w, t.y, sr);
  dl = fmaxf(__fmaf_rn(lx, lx, __fmaf_rn(ly, ly, lz * lz)), gl * gl);
  dr = fmaxf(__fmaf_rn(rx, rx, __fmaf_rn(ry, ry, rz * rz)), gr * gr);
  cl = __float_as_int(t.z);
  cr = __float_as_int(t.w);
}

__device__ __forceinline__ void node_dist2(const NodeF *__restrict__ nodes, int idx, const Vec<float> &p,
                                           float &dl, float &dr, int &cl, int &cr) {
  const NodeF *n = nodes + idx;
  float4 x, y, z, nl, nr, t;
  ldg32(&n->x, x, y);
  ldg32(&n->z, z, nl);
  ldg32(&n->nr, nr, t);
  node_bounds(x, y, z, nl, nr, t, p, dl, dr, cl, cr);
}

__device__ __forceinline__ void node_dist2(const NodeD *__restrict__ nodes, int idx, const Vec<double> &p,
                                           double &dl, double &dr, int &cl, int &cr) {
  const NodeD *n = nodes + idx;
  const double2 xl = __ldg(&n->xlo), xh = __ldg(&n->xhi);
  const double2 yl = __ldg(&n->ylo), yh = __ldg(&n->yhi);
  const double2 zl = __ldg(&n->zlo), zh = __ldg(&n->zhi);
  const double2 l0 = __ldg(&n->nl_xy), l1 = __ldg(&n->nl_zmin);
  const double2 r0 = __ldg(&n->nr_xy), r1 = __ldg(&n->nr_zmin);
  const double2 smax = __ldg(&n->smax);
  const int4 ch = __ldg(&n->child);
  const double lx = gap(xl.x, xh.x, p.x), rx = gap(xl.y, xh.y, p.x);
  const double ly = gap(yl.x, yh.x, p.y), ry = gap(yl.y, yh.y, p.y);
  const double lz = gap(zl.x, zh.x, p.z), rz = gap(zl.y, zh.y, p.z);
  const double sl = l0.x * p.x + l0.y * p.y + l1.x * p.z;
  const double sr = r0.x * p.x + r0.y * p.y + r1.x * p.z;
  const double gl = gap(l1.y, smax.x, sl), gr = gap(r1.y, smax.y, sr);
  dl = fmax(lx * lx + ly * ly + lz * lz, gl * gl);
  dr = fmax(rx * rx + ry * ry + rz * rz, gr * gr);
  cl = ch.x;
  cr = ch.y;
}

// The same bounds for the four children of a four-wide node (six 32-byte
// loads); slot k's squared lower bound in d[k], its child code in c[k].  An
// empty slot's inverted box gives +inf.
__device__ __forceinline__ void node4_dist2(const Node4F *__restrict__ nodes, int idx, const Vec<float> &p,
                                            float d[4], int c[4]) {
  const Node4F *n = nodes + idx;
  float4 xlo, xhi, ylo, yhi, zlo, zhi, nx, ny, nz, smin, smax, ch;
  ldg32(&n->xlo, xlo, xhi);
  ldg32(&n->ylo, ylo, yhi);
  ldg32(&n->zlo, zlo, zhi);
  ldg32(&n->nx, nx, ny);
  ldg32(&n->nz, nz, smin);
  ldg32(&n->smax, smax, ch);
  auto slot = [&](float xl, float xh, float yl, float yh, float zl, float zh, float a, float b, float e, float s0,
                  float s1) {
    const float gx = gap(xl, xh, p.x), gy = gap(yl, yh, p.y), gz = gap(zl, zh, p.z);
    const float s = __fmaf_rn(a, p.x, __fmaf_rn(b, p.y, e * p.z));
    const float gs = gap(s0, s1, s);
    return fmaxf(__fmaf_rn(gx, gx, __fmaf_rn(gy, gy, gz * gz)), gs * gs);
  };
  d[0] = slot(xlo.x, xhi.x, ylo.x, yhi.x, zlo.x, zhi.x, nx.x, ny.x, nz.x, smin.x, smax.x);
  d[1] = slot(xlo.y, xhi.y, ylo.y, yhi.y, zlo.y, zhi.y, nx.y, ny.y, nz.y, smin.y, smax.y);
  d[2] = slot(xlo.z, xhi.z, ylo.z, yhi.z, zlo.z, zhi.z, nx.z, ny.z, nz.z, smin.z, smax.z);
  d[3] = slot(xlo.w, xhi.w, ylo.w, yhi.w, zlo.w, zhi.w, nx.w, ny.w, nz.w, smin.w, smax.w);
  c[0] = __float_as_int(ch.x);
  c[1] = __float_as_int(ch.y);
  c[2] = __float_as_int(ch.z);
  c[3] = __float_as_int(ch.w);
}

__device__ __forceinline__ void order2(float &da, int &ca, float &db, int &cb) {
  if (db < da) {
    const float t = da;
    da = db;
    db = t;
    const int u = ca;
    ca = cb;
    cb = u;
  }
}

// Plane-slab lower bound of a triangle (one or two 16-byte loads); the full
// closest-point test loads the vertices only when this bound is below best.
__device__ __forceinline__ float tri_plane_gap2(const TriF *__restrict__ tris, uint32_t i, const Vec<float> &p) {
  const float4 P = __ldg(&tris[i].plane);
  const float dmax = __ldg(&tris[i].a.w);
  const float s = __fmaf_rn(P.x, p.x, __fmaf_rn(P.y, p.y, P.z * p.z));
  const float g = gap(P.w, dmax, s);
  return g * g;
}
__device__ __forceinline__ double tri_plane_gap2(const TriD *__restrict__ tris, uint32_t i, const Vec<double> &p) {
  const double2 n = __ldg(&tris[i].nxy), z = __ldg(&tris[i].nzmin);
  const double dmax = __ldg(&tris[i].dmax_id.x);
  const double s = n.x * p.x + n.y * p.y + z.x * p.z;
  const double g = gap(z.y, dmax, s);
  return g * g;
}

__device__ __forceinline__ void load_tri(const TriF *__restrict__ tris, uint32_t i, Vec<float> &a, Vec<float> &b,
                                         Vec<float> &c) {
  const float4 A = __ldg(&tris[i].a), B = __ldg(&tris[i].b), C = __ldg(&tris[i].c);
  a = {A.x, A.y, A.z};
  b = {B.x, B.y, B.z};
  c = {C.x, C.y, C.z};
}
__device__ __forceinline__ void load_tri(const TriD *__restrict__ tris, uint32_t i, Vec<double> &a,
                                         Vec<double> &b, Vec<double> &c) {
  const double2 p0 = __ldg(&tris[i].axy), p1 = __ldg(&tris[i].azbx), p2 = __ldg(&tris[i].bybz);
  const double2 p3 = __ldg(&tris[i].cxy), p4 = __ldg(&tris[i].czpad);
  a = {p0.x, p0.y, p1.x};
  b = {p1.y, p2.x, p2.y};
  c = {p3.x, p3.y, p4.x};
}

// One triangle against the current best: the plane-slab bound first, the
// full closest-point test only when the bound is below best.  Returns true
// when the triangle is strictly closer (best2 updated); `full` counts full tests.
__device__ __forceinline__ float plane_gap2(const float4 &P, const float4 &A, const Vec<float> &p) {
  const float s = __fmaf_rn(P.x, p.x, __fmaf_rn(P.y, p.y, P.z * p.z));
  const float g = gap(P.w, A.w, s);
  return g * g;
}
__device__ __forceinline__ bool tri_test(const TriF *__restrict__ tris, uint32_t i, const Vec<float> &p, float &best2,
                                         uint32_t &full) {
  float4 P, A;
  ldg32(&tris[i].plane, P, A);
  if (!(plane_gap2(P, A, p) < best2)) return false;
  ++full;
  float4 B, C;
  ldg32(&tris[i].b, B, C);
  const float d2 = tri_dist2(p, Vec<float>{A.x, A.y, A.z}, Vec<float>{B.x, B.y, B.z}, Vec<float>{C.x, C.y, C.z});
  if (d2 < best2) {
    best2 = d2;
    return true;
  }
  return false;
}
__device__ __forceinline__ bool tri_test(const TriD *__restrict__ tris, uint32_t i, const Vec<double> &p,
                                         double &best2, uint32_t &full) {
  if (!(tri_plane_gap2(tris, i, p) < best2)) return false;
  ++full;
  Vec<double> a, b, c;
  load_tri(tris, i, a, b, c);
  const double d2 = tri_dist2(p, a, b, c);
  if (d2 < best2) {
    best2 = d2;
    return true;
  }
  return false;
}

__device__ __forceinline__ float lower_f(float v) { return v; }
__device__ __forceinline__ float lower_f(double v) { return __double2float_rd(v); }

// Closest-point query: on return best2 holds the squared distance to the
// nearest triangle strictly closer than sqrt(best2) on entry; returns false
// when there is none.  The stack lives in shared memory, `stack` pointing at
// this thread's column (stride `stride` entries).  Bounded: at most kStack
// pushes outstanding and `max_iter` node/leaf visits; overruns set `err`.
template <typename T>
__device__ bool nearest(const typename Layout<T>::Node *__restrict__ nodes,
                        const typename Layout<T>::Tri *__restrict__ tris, uint32_t max_iter, const Vec<T> &p,
                        T &best2, uint32_t &best_tri, uint2 *stack, int stride, uint32_t &err, int node = 0) {
  bool found = false;
  int sp = 0;
  bool have = true;
  uint32_t iter = 0;
  while (have) {
    if (++iter > max_iter) {
      err |= TWOS_DEVERR_ITER;
      break;
    }
    if (node >= 0) {
      T dl, dr;
      int cl, cr;
      node_dist2(nodes, node, p, dl, dr, cl, cr);
      const bool vl = dl < best2, vr = dr < best2;
      if (vl && vr) {
        if (dr < dl) {
          const T td = dl;
          dl = dr;
          dr = td;
          const int tc = cl;
          cl = cr;
          cr = tc;
        }
        if (sp >= kStack) {
          err |= TWOS_DEVERR_STACK;
          break;
        }
        stack[sp * stride] = make_uint2(static_cast<uint32_t>(cr), __float_as_uint(lower_f(dr)));
        ++sp;
        node = cl;
        continue;
      }
      if (vl) {
        node = cl;
        continue;
      }
      if (vr) {
        node = cr;
        continue;
      }
    } else {
      const uint32_t enc = ~static_cast<uint32_t>(node);
      const uint32_t first = enc >> 3, count = enc & 7u;
      for (uint32_t i = 0; i < count; ++i) {
        uint32_t full = 0;
        if (tri_test(tris, first + i, p, best2, full)) {
          best_tri = first + i;
          found = true;
        }
      }
    }
    // Pop the next entry still closer than the current best.
    have = false;
    while (sp > 0) {
      --sp;
      const uint2 e = stack[sp * stride];
      if (static_cast<T>(__uint_as_float(e.y)) < best2) {
        node = static_cast<int>(e.x);
        have = true;
        break;
      }
    }
  }
  return found;
}

// ================================================================ sources
template <typename T> struct TermT {
  int kind, axis;
  T amp, offset, div;
  T c[3], w[3];
};

template <typename T> __device__ __forceinline__ T coord(const Vec<T> &v, int a) {
  return a == 0 ? v.x : (a == 1 ? v.y : v.z);
}

template <typename T> __device__ __forceinline__ T term_value(const TermT<T> &t, const Vec<T> &x) {
  switch (t.kind) {
    case TWOS_TERM_CONST:
      return t.amp;
    case TWOS_TERM_LINEAR:
      return t.amp * (coord(x, t.axis) + t.offset);
    case TWOS_TERM_GAUSS: {
      const T a = (x.x - t.c[0]) / t.w[0], b = (x.y - t.c[1]) / t.w[1], c = (x.z - t.c[2]) / t.w[2];
      return t.amp * exp(-(a * a) - (b * b) - (c * c));
    }
    case TWOS_TERM_BUMP: {
      const Vec<T> d{x.x - t.c[0], x.y - t.c[1], x.z - t.c[2]};
      const T dd = d.x * d.x + d.y * d.y + d.z * d.z;
      const T s = fmax(T(0), T(1) - dd / (t.w[0] * t.w[0]));
      return t.amp * (s * s) / t.div;
    }
    case TWOS_TERM_BOX:
      return (x.x >= t.c[0] && x.x <= t.w[0] && x.y >= t.c[1] && x.y <= t.w[1] && x.z >= t.c[2] &&
              x.z <= t.w[2])
                 ? t.amp
                 : T(0);
    case TWOS_TERM_BALL: {
      const Vec<T> d{x.x - t.c[0], x.y - t.c[1], x.z - t.c[2]};
      const T dd = d.x * d.x + d.y * d.y + d.z * d.z;
      return dd <= t.w[0] * t.w[0] ? t.amp : T(0);
    }
    case TWOS_TERM_QUAD: {
      const T a = x.x - t.c[0], b = x.y - t.c[1], c = x.z - t.c[2];
      return t.amp * (t.w[0] * (a * a) + t.w[1] * (b * b) + t.w[2] * (c * c));
    }
    default:
      return T(0);
  }
}

template <typename T>
__device__ __forceinline__ T source_value(const TermT<T> *terms, uint32_t begin, uint32_t n, const Vec<T> &x) {
  T s = T(0);
#pragma unroll 1
  for (uint32_t i = 0; i < n; ++i) {
    const T v = term_value(terms[begin + i], x);
    s = i == 0 ? v : s + v;
  }
  return s;
}

// Two sources at one point, through one copy of the terms' code.
template <typename T>
__device__ __forceinline__ void source_values(const TermT<T> *terms, uint32_t begin0, uint32_t n0, uint32_t begin1,
                                              uint32_t n1, const Vec<T> &x, T &s0, T &s1) {
  s0 = s1 = T(0);
#pragma unroll 1
  for (uint32_t i = 0; i < n0 + n1; ++i) {
    const bool second = i >= n0;
    const T v = term_value(terms[second ? begin1 + (i - n0) : begin0 + i], x);
    if (second)
      s1 = i == n0 ? v : s1 + v;
    else
      s0 = i == 0 ? v : s0 + v;
  }
}

}  // namespace twos
#include "ball_green.cuh"
namespace twos {

// One step's EXACT source integral over B_r(x), accumulated into acc as the
// analytic study backend does (study.cpp:96-104): the harmonic (CONST and
// LINEAR) terms as r^2/6 f(x) in one product, then each bump's closed-form
// ball integral added in term order.  Bumps are evaluated in FP64 (double-
// double inside) from the frame coordinates.
template <typename T>
__device__ __forceinline__ T exact_source(T acc, const TermT<T> *terms, uint32_t begin, uint32_t n,
                                          const Vec<T> &x, T r, uint32_t &err) {
  T harmonic = T(0);
  bool any = false;
  for (uint32_t i = 0; i < n; ++i) {
    const TermT<T> &t = terms[begin + i];
    if (t.kind == TWOS_TERM_CONST || t.kind == TWOS_TERM_LINEAR) {
      harmonic = any ? harmonic + term_value(t, x) : term_value(t, x);
      any = true;
    }
  }
  if (any) acc = acc + r * r / T(6) * harmonic;
  for (uint32_t i = 0; i < n; ++i) {
    const TermT<T> &t = terms[begin + i];
    if (t.kind != TWOS_TERM_BUMP) continue;
    const double dx = static_cast<double>(x.x) - static_cast<double>(t.c[0]);
    const double dy = static_cast<double>(x.y) - static_cast<double>(t.c[1]);
    const double dz = static_cast<double>(x.z) - static_cast<double>(t.c[2]);
    bool negative = false;
    const double v = exact_bump_green(sqrt(dx * dx + dy * dy + dz * dz), static_cast<double>(r),
                                      static_cast<double>(t.w[0]),
                                      static_cast<double>(t.amp) / static_cast<double>(t.div), negative);
    if (negative) err |= TWOS_DEVERR_SOURCE;
    acc = acc + static_cast<T>(v);
  }
  return acc;
}

// ================================================================ WoS kernel
constexpr int kWosBlock = 128;

template <typename T> __device__ __forceinline__ T to_T(double v);
template <> __device__ __forceinline__ double to_T<double>(double v) { return v; }
template <> __device__ __forceinline__ float to_T<float>(double v) { return static_cast<float>(v); }

// Position of a site/cavity in the geometry frame: FP64 keeps the original
// coordinates; FP32 is taken about the geometry centre.
template <typename T> __device__ __forceinline__ Vec<T> to_frame(const double *xyz, const GeoDesc &g);
template <> __device__ __forceinline__ Vec<double> to_frame<double>(const double *xyz, const GeoDesc &) {
  return {xyz[0], xyz[1], xyz[2]};
}
template <> __device__ __forceinline__ Vec<float> to_frame<float>(const double *xyz, const GeoDesc &g) {
  return {static_cast<float>(xyz[0] - g.center[0]), static_cast<float>(xyz[1] - g.center[1]),
          static_cast<float>(xyz[2] - g.center[2])};
}

template <typename T> __device__ __forceinline__ const typename Layout<T>::Node *geo_nodes(const GeoDesc &g);
template <> __device__ __forceinline__ const NodeF *geo_nodes<float>(const GeoDesc &g) { return g.nodes_f; }
template <> __device__ __forceinline__ const NodeD *geo_nodes<double>(const GeoDesc &g) { return g.nodes_d; }
template <typename T> __device__ __forceinline__ const typename Layout<T>::Tri *geo_tris(const GeoDesc &g);
template <> __device__ __forceinline__ const TriF *geo_tris<float>(const GeoDesc &g) { return g.tris_f; }
template <> __device__ __forceinline__ const TriD *geo_tris<double>(const GeoDesc &g) { return g.tris_d; }

// An upper bound on sqrtf(x) for x > 0 from rsqrtf, whose stated maximum
// error is 2 ulp: x rsqrtf(x) is within 1.25 * 2^-22 of sqrt(x) (relative),
// so raising it by 2^-20 puts it above the correctly rounded sqrtf(x).  The
// grid bounds only need |p - v| from above (a larger distance lowers the
// lower bound and raises the upper one), and this takes fewer instructions
// than the correctly rounded square root.  x = 0 gives NaN, which the
// bounds' fmaxf / fminf skip: that corner is left out, which only loosens
// them.
__device__ __forceinline__ float sqrt_up(float x) { return x * rsqrtf(x) * (1.0f + 0x1.0p-20f); }

// Distance-grid vertex (i, j, k) in the FP32 frame, rounded the same way in
// the grid build and in the walk step.
__device__ __forceinline__ Vec<float> grid_vertex(const GeoDesc &g, uint32_t i, uint32_t j, uint32_t k) {
  return {__fadd_rn(g.grid_lo[0], __fmul_rn(static_cast<float>(i), g.grid_h)),
          __fadd_rn(g.grid_lo[1], __fmul_rn(static_cast<float>(j), g.grid_h)),
          __fadd_rn(g.grid_lo[2], __fmul_rn(static_cast<float>(k), g.grid_h))};
}

// An integer below 2^23 as a float, exactly: one integer and one float
// operation instead of a conversion, which has a sixteenth of their rate.
__device__ __forceinline__ float small_float(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.f; }

// The grid cell of `p` (FP32 frame): its lower corner (clamped so the cell
// lies inside the grid) and record; false when p lies outside the grid (or is
// NaN).  A grid has fewer than 2^32 cells.
__device__ __forceinline__ bool grid_cell(const GeoDesc &g, const Vec<float> &p, uint32_t (&c)[3], uint32_t &cell) {
  const float fx = (p.x - g.grid_lo[0]) * g.grid_inv_h;
  const float fy = (p.y - g.grid_lo[1]) * g.grid_inv_h;
  const float fz = (p.z - g.grid_lo[2]) * g.grid_inv_h;
  if (!(fx >= 0.f && fy >= 0.f && fz >= 0.f && fx <= g.grid_top[0] && fy <= g.grid_top[1] && fz <= g.grid_top[2]))
    return false;
  c[0] = min(static_cast<uint32_t>(fx), g.grid_n[0] - 2);
  c[1] = min(static_cast<uint32_t>(fy), g.grid_n[1] - 2);
  c[2] = min(static_cast<uint32_t>(fz), g.grid_n[2] - 2);
  cell = (c[0] * (g.grid_n[1] - 1) + c[1]) * (g.grid_n[2] - 1) + c[2];
  return true;
}

// The grid's bounds of the mesh distance at `p`.  Lower: the
// largest D(v) - |p - v| over the eight corners v of p's cell (the distance
// is 1-Lipschitz, so each is a bound).  Upper (with UPPER; before the FP32
// allowance the caller adds): the smallest (D(v) + 1) q + |p - v| over the
// corners whose value is held exactly -- a vertex stores
// floor((d_FP32 - 2 delta)/q), so its distance is below (D + 1) q + 3 delta.
// `word` is the record's last word (entry_of).  False when p lies outside the
// grid.  One 16-byte record per cell (GeoDesc::grid).
template <bool UPPER>
__device__ __forceinline__ bool grid_bounds(const GeoDesc &g, const Vec<float> &p, float &bound, float &upper,
                                            int &word) {
  uint32_t c0[3], cell;
  if (!grid_cell(g, p, c0, cell)) return false;
  float best = -CUDART_INF_F, up = CUDART_INF_F;
  const uint4 rec = __ldg(g.grid + cell);
  const uint32_t base = rec.z & 0xffffu;
  // The vertices' coordinates, rounded as grid_vertex rounds them.
  float d[3][2];
  const float x[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float f = small_float(c0[a]);
    d[a][0] = x[a] - __fadd_rn(g.grid_lo[a], __fmul_rn(f, g.grid_h));
    d[a][1] = x[a] - __fadd_rn(g.grid_lo[a], __fmul_rn(f + 1.f, g.grid_h));
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const Vec<float> dv{d[0][c >> 2], d[1][(c >> 1) & 1], d[2][c & 1]};
    const uint32_t off = ((c < 4 ? rec.x : rec.y) >> (8 * (c & 3))) & 0xffu;
    const float dist = sqrt_up(dot3(dv, dv));
    const float dq = small_float(off == 0xffu ? base : base + off) * g.grid_q;
    best = fmaxf(best, dq - dist);
    if (UPPER && off != 0xffu) up = fminf(up, dq + g.grid_q + dist);
  }
  bound = best;
  if (UPPER) upper = up;
  word = static_cast<int>(rec.w);
  return true;
}

// The upper bound alone, at a point of the grid (a rolled loop: the mixed
// form's walk steps seldom need it).
__device__ __forceinline__ float grid_upper(const GeoDesc &g, const Vec<float> &p) {
  uint32_t c0[3], cell;
  float up = CUDART_INF_F;
  if (!grid_cell(g, p, c0, cell)) return up;
  const uint4 rec = __ldg(g.grid + cell);
  const uint32_t base = rec.z & 0xffffu;
#pragma unroll 1
  for (uint32_t c = 0; c < 8; ++c) {
    const uint32_t off = ((c < 4 ? rec.x : rec.y) >> (8 * (c & 3))) & 0xffu;
    if (off == 0xffu) continue;
    const Vec<float> dv = sub(p, grid_vertex(g, c0[0] + (c >> 2), c0[1] + ((c >> 1) & 1u), c0[2] + (c & 1u)));
    up = fminf(up, small_float(base + off) * g.grid_q + g.grid_q + sqrt_up(dot3(dv, dv)));
  }
  return up;
}

constexpr float kListReach = 1.7f;  // spacings from the surface up to which cells have lists
// A cell record's last word: an entry node (-1: none), or the start of the
// cell's candidate list, whose first entry holds the entry node.
__device__ __forceinline__ bool is_list(int word) { return word < -1; }
__device__ __forceinline__ uint32_t list_start(int word) { return static_cast<uint32_t>(word) & 0x7fffffffu; }
__device__ __forceinline__ int entry_of(const GeoDesc &g, int word) {
  return is_list(word) ? static_cast<int>(__ldg(&g.lists[list_start(word)].x)) : word;
}
// The last word of the record of p's cell (p inside the grid).
__device__ __forceinline__ int cell_word(const GeoDesc &g, const Vec<float> &p) {
  uint32_t c[3], cell = 0;
  return grid_cell(g, p, c, cell) ? static_cast<int>(__ldg(&g.grid[cell].w)) : -1;
}
// Distance from p to the centre of its grid cell (p inside the grid), from above.
__device__ __forceinline__ float cell_offset(const GeoDesc &g, const Vec<float> &p) {
  uint32_t c[3] = {0u, 0u, 0u}, cell;
  grid_cell(g, p, c, cell);
  float d2 = 0.f;
  const float x[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float e = x[a] - __fmaf_rn(small_float(c[a]) + 0.5f, g.grid_h, g.grid_lo[a]);
    d2 = __fmaf_ru(e, e, d2);
  }
  return __fsqrt_ru(d2);
}

__device__ __forceinline__ bool grid_bound(const GeoDesc &g, const Vec<float> &p, float &bound) {
  float upper;
  int entry_node;
  return grid_bounds<false>(g, p, bound, upper, entry_node);
}

// (sqrt(d2) + by)^2, rounded up.
__device__ __forceinline__ float widen2(float d2, float by) {
  const float t = __fadd_ru(__fsqrt_ru(d2), by);
  return __fmul_ru(t, t);
}

// ---------------------------------------------------------------- FP64 queries
// The FP64 form's closest-point query searches the FP32 BVH: whatever only
// prunes need not be FP64, as long as it leaves room for its error.  `margin`
// bounds the difference between an FP32 distance bound at p (node boxes,
// normal slabs, triangle planes, the two bounds of a triangle below) and the
// FP64 distance: the session's delta (vertices, boxes and slabs rounded to
// FP32, the arithmetic) plus the rounding of the point itself.  The search
// keeps the triangles whose lower bound stays below the smallest upper bound
// plus two margins -- nearly always one or two -- and only those get the FP64
// closest-point test, together with the warp's next walk step.  Every triangle
// that could hold the FP64 minimum is among them, so the result is the
// minimum an FP64 search gives, bit for bit, at half the node bytes and
// full-rate arithmetic.
struct Cull {
  Vec<float> p;   // the query point in the FP32 frame
  float margin;
  float limit;    // squared FP32 pruning threshold
  int count;      // candidates held
};

// (sqrt(best2) + margin)^2 rounded up (infinite for an unbounded query).
__device__ __forceinline__ float cull_limit(double best2, float margin) {
  const float t = __fadd_ru(__fsqrt_ru(__double2float_ru(best2)), margin);
  return __fmul_ru(t, t);
}

// Sets up the search at p for distances below sqrt(best2); false when FP32
// cannot hold the geometry or the point (cull_margin 0: see open_impl; a
// coordinate beyond 2^50, whose square would overflow, or NaN; a distance
// whose product with an edge may be beyond 2^60, where the squares of such
// products overflow: cull_margin is at least 2^-19 half extents), or where the
// margin, which grows with the point's distance, prunes too little: beyond
// `most` times the mesh's own.  The caller then takes the FP64 nodes.  Bulk
// calls of 30,000 points on 81,920 triangles, ms by distance in half extents,
// FP32 / FP64 nodes: 300 3.6 / 5.1, 1,000 4.9 / 5.1, 10,000 13.3 / 5.1 (6.3
// where the line runs through a call); a warp per point, 16,384 points: 30,000
// 2.3 / 1.7 (warp_plain64).
constexpr float kFarLane = 512.f, kFarWarp = 32768.f;  // about 1,000 and 64,000 half extents
__device__ __forceinline__ bool cull_begin(const GeoDesc &g, const Vec<double> &p, double best2, Cull &c,
                                           float most = kFarLane) {
  const double xyz[3] = {p.x, p.y, p.z};
  c.p = to_frame<float>(xyz, g);
  const float norm1 = fabsf(c.p.x) + fabsf(c.p.y) + fabsf(c.p.z);
  c.margin = __fmaf_ru(norm1, 0x1.0p-20f, g.cull_margin);
  c.limit = cull_limit(best2, c.margin);
  c.count = 0;
  return g.cull_margin > 0.f && norm1 < 0x1.0p50f && c.margin < most * g.cull_margin &&
         (norm1 + 0x1.0p20f * g.cull_margin) * g.box_extent < 0x1.0p60f;
}

// A point of the triangle at (nearly) its closest to p: Ericson's regions as
// tri_closest, with the interior weights clamped so that the point stays in
// the triangle whatever their rounding (degenerate triangles included).
__device__ __forceinline__ Vec<float> tri_point(const Vec<float> &ap, const Vec<float> &bp, const Vec<float> &cp,
                                                const Vec<float> &ab, const Vec<float> &ac) {
  // Returned as the vector from the point to p.
  const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  if (d1 <= 0.f && d2 <= 0.f) return ap;
  const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
  if (d3 >= 0.f && d4 <= d3) return bp;
  const float vc = mad_t(d1, d4, -(d3 * d2));
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) return add_scaled(ap, ab, -__saturatef(__fdividef(d1, d1 - d3)));
  const float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
  if (d6 >= 0.f && d5 <= d6) return cp;
  const float vb = mad_t(d5, d2, -(d1 * d6));
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) return add_scaled(ap, ac, -__saturatef(__fdividef(d2, d2 - d6)));
  const float va = mad_t(d3, d6, -(d5 * d4));
  if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f)
    return add_scaled(bp, sub(ac, ab), -__saturatef(__fdividef(d4 - d3, (d4 - d3) + (d5 - d6))));
  const float denom = __fdividef(1.f, va + vb + vc);
  const float v = __saturatef(vb * denom);
  const float w = fminf(__saturatef(vc * denom), 1.f - v);
  return add_scaled(add_scaled(ap, ab, -v), ac, -w);
}

// Of two triangles at the same FP64 distance from p, the one that a search of
// the FP64 nodes, nearer child first, meets first: it decides the closest point
// returned, and the two points can be far apart.  Where the points are the same
// (a common vertex: most ties; within `near` of their size) i stands for both,
// which `ties` notes (kTieSame); a triangle with another point cannot then be
// compared with i alone, and kTieOpen leaves the decision to the search itself
// (first_of_tied).  Out of line: ties are few.
constexpr uint32_t kTieSame = 1u, kTieOpen = 2u;
struct Tied {
  uint32_t tri, ties;
};
__device__ __noinline__ Tied first_met(const GeoDesc *g, double x, double y, double z, uint32_t i, uint32_t j,
                                       double near, uint32_t ties) {
  const Vec<double> p{x, y, z};
  Vec<double> a, b, c;
  load_tri(g->tris_d, i, a, b, c);
  const Vec<double> q = tri_closest(p, a, b, c);
  load_tri(g->tris_d, j, a, b, c);
  const Vec<double> r = tri_closest(p, a, b, c);
  const double apart = fmax(fabs(q.x - r.x), fmax(fabs(q.y - r.y), fabs(q.z - r.z)));
  if (apart <= near * (fabs(q.x) + fabs(q.y) + fabs(q.z))) return {i, ties | kTieSame};
  if (ties & kTieSame) return {i, ties | kTieOpen};
  const uint32_t lo = min(i, j), hi = max(i, j);
  int node = 0;
  for (int depth = 0; node >= 0 && depth <= kMaxDepth; ++depth) {
    const int4 ch = __ldg(&g->nodes_d[node].child);
    const uint32_t right = ~static_cast<uint32_t>(ch.y);  // of a leaf: first triangle and count
    const uint32_t mid = ch.y >= 0 ? __ldg(g->node_first + ch.y) : (right & 7u) ? right >> 3 : 0xffffffffu;
    if (lo < mid && hi >= mid) {  // the subtree where they part
      double dl, dr;
      int cl, cr;
      node_dist2(g->nodes_d, node, p, dl, dr, cl, cr);
      return {dr < dl ? hi : lo, ties};
    }
    node = hi < mid ? ch.x : ch.y;
  }
  return {lo, ties};
}

// The same for points that are the same but for rounding, nearly always.
__device__ __forceinline__ float point_mark(const Vec<double> &q) {
  return static_cast<float>(q.x + 0.7548776662466927 * q.y + 0.5698402909980532 * q.z);
}

// FP64 closest-point test of the held candidates (TIES: the triangle of several
// at the same distance as first_met, its notes in *ties, the mark of its point
// in *mark).  A lane's search of the FP32 nodes meets the same one first but for
// symmetric points, so points that differ by rounding count as the same (bulk
// call of 122,591 points: 1.88 ms without a look at ties, 1.95 so, 2.11 with
// every rounding looked at).
template <bool TIES = false>
__device__ __forceinline__ bool cull_flush(const GeoDesc &g, const Vec<double> &p, Cull &c, double &best2,
                                           uint32_t &best_tri, const uint2 *cand, int stride,
                                           uint32_t *ties = nullptr, float *mark = nullptr) {
  bool found = false;
  for (int k = 0; k < c.count; ++k) {
    const uint2 e = cand[k * stride];
    if (!(__uint_as_float(e.y) < c.limit)) continue;  // the limit fell below its bound since
    Vec<double> ta, tb, tc;
    load_tri(g.tris_d, e.x, ta, tb, tc);
    const Vec<double> q = tri_closest(p, ta, tb, tc), dv = sub(p, q);
    const double d2 = dot3(dv, dv);
    if (d2 < best2) {
      best2 = d2;
      best_tri = e.x;
      found = true;
      if (TIES) *ties = 0u, *mark = point_mark(q);
    } else if (TIES && d2 == best2) {
      if (point_mark(q) == *mark) {
        *ties |= kTieSame;
      } else {
        const Tied t = first_met(&g, p.x, p.y, p.z, best_tri, e.x, 0x1.0p-48, *ties);
        if (t.tri == e.x) *mark = point_mark(q);
        best_tri = t.tri;
        *ties = t.ties;
      }
    }
  }
  c.count = 0;
  return found;
}

// Squared lower bound of the distance from p to a triangle along a direction
// w: the plane through the vertex nearest along w separates them by the
// smallest w.(p - vertex) / |w|.  Holds for any w; near 0 it bounds nothing.
__device__ __forceinline__ float support2(const Vec<float> &w, const Vec<float> &ap, const Vec<float> &bp,
                                          const Vec<float> &cp, float w2) {
  const float m = fmaxf(fminf(dot3(w, ap), fminf(dot3(w, bp), dot3(w, cp))), 0.f);
  return w2 > 1e-30f ? __fdividef(m, w2) * m * (1.f - 0x1.0p-18f) : 0.f;
}

// One triangle of the search: the plane slab, then the bound along the
// direction to its centroid (it leaves 2.9 of 15.3 triangles a query for the
// tests below on the 81,920-triangle noise sphere), then two bounds from the
// vector w from a point of the triangle near its closest to p: |w| from
// above, and w's own direction from below, whatever the point's rounding.  A
// triangle within the threshold is held as a candidate; true when the list
// is full and the caller has to flush it first.
__device__ __forceinline__ bool cull_tri(uint32_t i, const float4 &P, const float4 &A, const float4 &B,
                                         const float4 &C, Cull &c, uint2 *cand, int stride, uint32_t &full) {
  if (!(plane_gap2(P, A, c.p) < c.limit)) return false;
  if (c.count >= kCand) return true;
  const Vec<float> a{A.x, A.y, A.z}, b{B.x, B.y, B.z}, cc{C.x, C.y, C.z};
  const Vec<float> ap = sub(c.p, a), bp = sub(c.p, b), cp = sub(c.p, cc);
  const Vec<float> t{ap.x + bp.x + cp.x, ap.y + bp.y + cp.y, ap.z + bp.z + cp.z};
  if (!(support2(t, ap, bp, cp, dot3(t, t)) < c.limit)) return false;
  ++full;
  const Vec<float> w = tri_point(ap, bp, cp, sub(b, a), sub(cc, a));
  const float w2 = dot3(w, w);
  const float low2 = support2(w, ap, bp, cp, w2);
  if (!(low2 < c.limit)) return false;
  cand[c.count * stride] = make_uint2(i, __float_as_uint(low2));
  ++c.count;
  const float up = __fmaf_ru(2.f, c.margin, __fsqrt_ru(w2));
  c.limit = fminf(c.limit, __fmul_ru(up, up));
  return false;
}

// Bound and start node of a query from the distance grid: the grid's upper
// bound plus 6 delta (its 3 delta and the query's own error, with room) is
// above the distance, so the traversal may prune with it before any triangle
// is found; when the initial bound is below one entry cell, it starts at the
// cell's entry node (every triangle outside that subtree is farther).  A
// geometry FP32 cannot hold (cull_margin 0) has no bounds: its FP32 distances
// overflow for some triangles, at a grid vertex for others than at p.
//
// The grid's upper bound comes from FP32 distances at its vertices.  Where FP32
// cannot evaluate a triangle (edges a thousand times longer than its height;
// products below the smallest normal number) its interior point is anywhere
// in its plane, and the bound can be below the distance.  So a search takes
// the bound as a distance to be found below, and one that finds none below it
// is made again without it.
__device__ __forceinline__ void grid_start(const GeoDesc &g, const Vec<float> &p, float radius, float &upper,
                                           int &node) {
  float bound;
  int entry = -1;
  upper = CUDART_INF_F;
  node = 0;
  if (!g.grid || !(g.cull_margin > 0.f) || !grid_bounds<true>(g, p, bound, upper, entry)) {
    upper = CUDART_INF_F;
    return;
  }
  upper = __fmaf_ru(6.f, g.delta, upper);
  if (fminf(radius, upper) < g.entry_radius) node = max(entry_of(g, entry), 0);
}

// nearest() over the FP64 nodes, for what the FP32 bounds cannot hold; out of
// line and by value, so it costs the callers no registers.
struct Plain64 {
  double best2;
  uint32_t tri;
  uint32_t flags;  // error bits | found << 31
};
// `warm`: a triangle to be tested first (kNoTri: none).
constexpr uint32_t kNoTri = 0xffffffffu;
__device__ __noinline__ Plain64 nearest_plain64(const GeoDesc *g, double x, double y, double z, double best2,
                                                uint32_t warm = kNoTri) {
  uint2 stack[kStack];
  Plain64 r{best2, 0u, 0u};
  const Vec<double> p{x, y, z};
  uint32_t err = 0, full = 0;
  bool found = warm != kNoTri && tri_test(g->tris_d, warm, p, r.best2, full);
  if (found) r.tri = warm;
  found |= nearest<double>(g->nodes_d, g->tris_d, g->max_iter, p, r.best2, r.tri, stack, 1, err);
  r.flags = err | (found ? 0x80000000u : 0u);
  return r;
}

// The triangle at the smallest FP64 distance best2 that the search of the FP64
// nodes meets first (`tri`, one of them, should it meet none).
__device__ __forceinline__ uint32_t first_of_tied(const GeoDesc &g, const Vec<double> &p, double best2, uint32_t tri) {
  const Plain64 r = nearest_plain64(&g, p.x, p.y, p.z, best2 * (1.0 + 0x1.0p-40) + 0x1.0p-1000);
  return r.flags >> 31 && r.best2 == best2 ? r.tri : tri;
}

// The same, as nearest_geo().
__device__ __forceinline__ bool nearest_plain(const GeoDesc &g, const Vec<double> &p, double &best2,
                                              uint32_t &best_tri, uint32_t &err) {
  const Plain64 r = nearest_plain64(&g, p.x, p.y, p.z, best2);
  err |= r.flags & 0x7fffffffu;
  if (!(r.flags >> 31)) return false;
  best2 = r.best2;
  best_tri = r.tri;
  return true;
}

// Closest-point query outside the walk kernel, as nearest(), from the distance
// grid's bound and entry node; the FP64 form searches in FP32.  A loop of
// units with one set of loads for nodes and triangles, as the walk kernel's.
// `stack`: this thread's column of kNearShared traversal entries and, in the
// FP64 form, kCand candidates; deeper entries are local.  A leaf may be reached
// with kStack entries held, so an overrun is one entry more, which there is
// room for until the next unit notices it (likewise in closest_kernel and
// cert_walk_kernel).
constexpr int kNearShared = 8;
template <typename T> __host__ __device__ constexpr int near_entries() {
  return kNearShared + (sizeof(T) == 8 ? kCand : 0);
}
template <typename T>
__device__ __forceinline__ bool nearest_geo(const GeoDesc &g, const Vec<T> &p, T &best2, uint32_t &best_tri,
                                            uint2 *stack, int stride, uint32_t &err) {
  Cull c{{0.f, 0.f, 0.f}, 0.f, 0.f, 0};
  uint2 *cand = stack + kNearShared * stride;
  uint2 deep[kStack + 1 - kNearShared];
  float upper;
  int node;
  bool found = false;
  const T from = best2;
  if constexpr (sizeof(T) == 4) {
    c.p = p;
    grid_start(g, c.p, sqrtf(best2), upper, node);
    best2 = fminf(best2, upper * upper);
  } else {
    if (!cull_begin(g, p, best2, c)) return nearest_plain(g, p, best2, best_tri, err);
    grid_start(g, c.p, sqrtf(c.limit), upper, node);
    const float reach = __fadd_ru(upper, c.margin), reach2 = __fmul_ru(reach, reach);
    c.limit = fminf(c.limit, reach2);
    best2 = fmin(best2, static_cast<double>(reach2));
  }
#pragma unroll 1
  for (;;) {
    uint32_t tri_cur = 0, tri_end = 0, iter = 0;
    int sp = 0;
    bool have = true;
#pragma unroll 1
    for (;;) {
      const float limit = [&]() -> float {
        if constexpr (sizeof(T) == 4)
          return best2;
        else
          return c.limit;
      }();
      bool flush = false, done = false;
      if (tri_cur >= tri_end) {
        while (!have && sp > 0) {
          --sp;
          const uint2 e = sp < kNearShared ? stack[sp * stride] : deep[sp - kNearShared];
          if (__uint_as_float(e.y) < limit) {
            node = static_cast<int>(e.x);
            have = true;
          }
        }
        done = !have;
        if (have && node < 0) {
          const uint32_t enc = ~static_cast<uint32_t>(node);
          tri_cur = enc >> 3;
          tri_end = tri_cur + (enc & 7u);
          have = false;
        }
      }
      if (!done && (++iter > g.max_iter || sp > kStack)) {
        err |= sp > kStack ? TWOS_DEVERR_STACK : TWOS_DEVERR_ITER;
        done = true;
        best2 = fmax(best2, from);  // no second search
      }
      if (!done) {
        const bool on_tri = tri_cur < tri_end;
        const char *at = on_tri ? reinterpret_cast<const char *>(g.tris_f + tri_cur)
                                : reinterpret_cast<const char *>(g.nodes_f + node);
        float4 r0, r1, r2, r3, r4{}, r5{};
        ldg32(at, r0, r1);
        ldg32(at + 32, r2, r3);
        ldg32_if(!on_tri, at + 64, r4, r5);
        if (on_tri) {
          if constexpr (sizeof(T) == 4) {
            if (plane_gap2(r0, r1, c.p) < best2) {
              const float d2 = tri_dist2(c.p, Vec<float>{r1.x, r1.y, r1.z}, Vec<float>{r2.x, r2.y, r2.z},
                                         Vec<float>{r3.x, r3.y, r3.z});
              if (d2 < best2) {
                best2 = d2;
                best_tri = tri_cur;
                found = true;
              }
            }
            ++tri_cur;
          } else {
            // A full candidate list is tested first; the triangle comes again.
            uint32_t full = 0;
            flush = cull_tri(tri_cur, r0, r1, r2, r3, c, cand, stride, full);
            if (!flush) ++tri_cur;
          }
        } else {
          float dl, dr;
          int cl, cr;
          node_bounds(r0, r1, r2, r3, r4, r5, c.p, dl, dr, cl, cr);
          const bool vl = dl < limit, vr = dr < limit, swap = dr < dl;
          if (vl && vr) {
            const uint2 e = make_uint2(static_cast<uint32_t>(swap ? cl : cr), __float_as_uint(swap ? dl : dr));
            if (sp < kNearShared)
              stack[sp * stride] = e;
            else
              deep[sp - kNearShared] = e;
            ++sp;
          }
          have = vl || vr;
          node = vl && !(vr && swap) ? cl : cr;
        }
      }
      if constexpr (sizeof(T) == 8) {
        if (flush || done) found |= cull_flush(g, p, c, best2, best_tri, cand, stride);
      }
      if (done) break;
    }
    if (found || !(best2 < from)) return found;
    // None below the grid's bound (grid_start): without it, from the root.
    best2 = from;
    if constexpr (sizeof(T) == 8) c.limit = cull_limit(from, c.margin);
    node = 0;
  }
}

__device__ __forceinline__ uint32_t find_job(const JobDesc *jobs, uint32_t n, uint64_t wid) {
  uint32_t lo = 0, hi = n - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (jobs[mid].walk_begin <= wid)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Dynamic shared memory: the launch's job, geometry and term tables.
// Job and geometry descriptors are copied to shared memory when they take at
// most kTableSmem bytes, which keeps 8 blocks of 128 threads (with their
// traversal stacks) resident per SM; a launch with more jobs reads them from
// global memory (through L1) instead of giving up resident blocks.
constexpr uint32_t kTableSmem = 2048;
struct SmemPlan {
  uint32_t geo_offset, term_offset, bytes;
  bool tables;  // jobs and geometries in shared memory
};
template <typename T> __host__ __device__ inline SmemPlan smem_plan(uint32_t n_jobs, uint32_t n_geos, uint32_t n_terms) {
  SmemPlan p;
  const uint32_t jobs = n_jobs * static_cast<uint32_t>(sizeof(JobDesc));
  const uint32_t geo_offset = (jobs + 15u) & ~15u;
  const uint32_t geos = geo_offset + n_geos * static_cast<uint32_t>(sizeof(GeoDesc));
  p.tables = geos <= kTableSmem;
  p.geo_offset = p.tables ? geo_offset : 0u;
  p.term_offset = p.tables ? (geos + 15u) & ~15u : 0u;
  p.bytes = p.term_offset + n_terms * static_cast<uint32_t>(sizeof(TermT<T>));
  return p;
}

bool launch_tables_in_smem(int precision, uint32_t n_jobs, uint32_t n_geos, uint32_t n_terms) {
  return precision == TWOS_PREC_MIXED ? smem_plan<float>(n_jobs, n_geos, n_terms).tables
                                      : smem_plan<double>(n_jobs, n_geos, n_terms).tables;
}

constexpr int kShared = 8;  // traversal-stack entries per thread in shared memory; the deeper ones are local
// Shared-memory entries per thread: the traversal stack and, in the FP64
// form, the candidates of its search.
template <typename T> __host__ __device__ constexpr int wos_stack_entries() {
  return sizeof(T) == 4 ? kShared : kShared + kCand;
}

// A walk's state that its traversal does not touch (position, sums, ids).
// Its ids are in shared memory (one word per thread and field, consecutive
// threads on consecutive words), and so is the rest in the FP64 form, whose
// state is twice as wide; the mixed form keeps what every step changes in
// registers.
template <typename V, bool SHARED> struct Cell {
  V v;
  __device__ __forceinline__ operator V() const { return v; }
  __device__ __forceinline__ void operator=(V x) { v = x; }
};
template <typename V> struct Cell<V, true> {
  volatile V *p;
  __device__ __forceinline__ operator V() const { return *p; }
  __device__ __forceinline__ void operator=(V x) { *p = x; }
};
// Shared-memory bytes of that state per thread (both forms: ids, the nearest
// cavity's distance and index).
template <typename T> __host__ __device__ constexpr int wos_cold_bytes(bool gradient) {
  return sizeof(T) == 4 ? 24 : 88 + (gradient ? 96 : 0);
}

enum : int { kIdle = 0, kTraverse = 1, kStep = 2, kBegin = 3, kFirst = 4, kAgain = 5 };

// Persistent walk-on-spheres kernel as a per-lane state machine.  Each loop
// iteration every traversing lane runs up to `units` units of work back to
// back -- BVH node tests or triangle tests of its current closest-point query
// -- and stops early when its query ends.  A lane whose query
// has finished waits in kStep until at least `step_threshold` lanes of its
// warp are ready (or no lane is still traversing); those lanes then take
// their walk step together and start their next query, and lanes whose walk
// ended refill from the work queue once `refill` lanes are idle.  So lanes
// never wait for the slowest traversal of the warp, only for the batched
// step.  In the mixed form a step first tries the geometry's distance-bound
// grid and skips the query when the grid's bound is large enough.  MODE:
// TWOS_MODE_*; the per-walk value type is T (FP32 accumulation in the mixed
// form, FP64 in the plain form).  SRC: TWOS_SOURCE_* (a
// template argument, so the exact-integral code of TWOS_SOURCE_EXACT adds no
// registers to the other forms).
//
// What bounds it: instruction issue under the traversal's divergence (7 to 9
// of 32 lanes per instruction) and, between issues, the dependent loads of
// nodes and triangles.  Hence: one set of loads per unit for both kinds (a
// warp used to wait for its node lanes, its triangle lanes and its full tests
// one after another; 50 M walks of the 327,680-triangle noise sphere, mixed:
// 201 -> 184 ms); every piece of the loop emitted once -- query set-up, grid
// lookup, candidate test -- because the FP64 kernel stalled on instruction
// fetch with two copies of them (1.02 M walks, 81,920 triangles: 47 -> 38
// ms); and few stack entries in shared memory, which leaves it to the L1
// (FP64 52 -> 47 ms, mixed 204 -> 201).
// Residency: the FP32 form with the centre-point source fits 64 registers, so
// 1024 threads (8 blocks of 128) stay resident per SM; the other FP32 forms
// take up to 80 (768 threads), the FP64 form and the exact ball integrals
// (double-double) 128 (512 threads: they spill below, and their local memory
// then shares the L1 with the BVH; 2,000 x 512 FP64 walks on 81,920 triangles
// 39 ms with 80 registers and 32 with 120, the gradient form 4.2 and 2.7).
// The FP64 forms and the mixed compliance and hot forms (on the binary BVH) do
// not spill; of the mixed forms, boundary mode spills 4 bytes, paired
// centre-source walks 12 (28 with claims), four-wide ones 12 to 18, and the
// gradient 20 to 64.
template <typename T, int MODE, int SRC>
constexpr int wos_min_blocks(int block) {
  const int threads = sizeof(T) == 8 || SRC == TWOS_SOURCE_EXACT           ? 512
                      : SRC == TWOS_SOURCE_CENTER && MODE != kModeGradient ? 1024
                                                                           : 768;
  return threads / block > 1 ? threads / block : 1;
}

// Walks a lane claims from the work queue at once.
__host__ __device__ __forceinline__ uint32_t lane_walks_of(const WosLaunch &L) {
  return L.lane_walks > 1 ? static_cast<uint32_t>(L.lane_walks) : 1u;
}

template <typename T, int MODE, int SRC, int BLOCK, bool TRACE = false, bool GRID64 = false, bool WIDE = false,
          bool CLAIM = false>
__global__ void __launch_bounds__(BLOCK, wos_min_blocks<T, MODE, SRC>(BLOCK)) wos_kernel(const WosLaunch L) {
  constexpr bool GREEN = SRC == TWOS_SOURCE_GREEN;
  constexpr bool EXACT = SRC == TWOS_SOURCE_EXACT && MODE != kModeBoundary;
  constexpr bool GRAD = MODE == kModeGradient;
  constexpr bool PAIRED = MODE == TWOS_MODE_PAIRED || GRAD;
  // Dynamic shared memory: per thread the first kShared entries of the
  // traversal stack and, in the FP64 form, kCand candidates (column-major so a
  // warp's accesses hit distinct banks), then the walks' state (Cell), then
  // the tables.
  extern __shared__ __align__(16) unsigned char s_dyn[];
  uint2 *s_stack = reinterpret_cast<uint2 *>(s_dyn);
  unsigned char *s_cold = s_dyn + wos_stack_entries<T>() * BLOCK * sizeof(uint2);
  unsigned char *s_tab = s_cold + wos_cold_bytes<T>(GRAD) * BLOCK;
  const SmemPlan plan = smem_plan<T>(L.n_jobs, L.n_geos, L.n_terms);
  const JobDesc *s_jobs = plan.tables ? reinterpret_cast<const JobDesc *>(s_tab) : L.jobs;
  const GeoDesc *s_geos = plan.tables ? reinterpret_cast<const GeoDesc *>(s_tab + plan.geo_offset) : L.geos;
  TermT<T> *s_terms = reinterpret_cast<TermT<T> *>(s_tab + plan.term_offset);

  if (plan.tables) {
    JobDesc *tj = reinterpret_cast<JobDesc *>(s_tab);
    GeoDesc *tg = reinterpret_cast<GeoDesc *>(s_tab + plan.geo_offset);
    for (uint32_t i = threadIdx.x; i < L.n_jobs; i += blockDim.x) tj[i] = L.jobs[i];
    for (uint32_t i = threadIdx.x; i < L.n_geos; i += blockDim.x) tg[i] = L.geos[i];
  }
  for (uint32_t i = threadIdx.x; i < L.n_terms; i += blockDim.x) {
    const TermDev &d = L.terms[i];
    TermT<T> t;
    t.kind = d.kind;
    t.axis = d.axis;
    t.amp = to_T<T>(d.amp);
    t.offset = to_T<T>(d.offset);
    t.div = to_T<T>(d.div);
    for (int k = 0; k < 3; ++k) {
      t.c[k] = to_T<T>(d.c[k]);
      t.w[k] = to_T<T>(d.w[k]);
    }
    s_terms[i] = t;
  }
  __syncthreads();

  const unsigned lane = threadIdx.x & 31u;
  const unsigned full = 0xffffffffu;
  const bool on = static_cast<int>(lane) < L.lanes;  // lanes that take walks
  const unsigned on_mask = __ballot_sync(full, on);
  uint2 *stack = s_stack + threadIdx.x;
  uint2 deep[kStack - kShared];
  auto push = [&](int &sp, uint2 e) {
    if (sp < kShared)
      stack[sp * BLOCK] = e;
    else
      deep[sp - kShared] = e;
    ++sp;
  };
  uint32_t err = 0;
  // Per-thread traversal counters (32-bit: a thread's share of one launch
  // stays far below 2^32), summed in 64 bits at the end.
  uint32_t c_nodes = 0, c_planes = 0, c_tris = 0, c_grid = 0;

  int phase = kIdle;
  bool exhausted = false;  // warp-uniform
  const int units = L.units > 0 ? L.units : 1;
  // Walk state.
  constexpr bool COLD = sizeof(T) == 8;
  auto word8 = [&](auto &c, int word) {  // 8-byte words of the thread's column
    c.p = reinterpret_cast<decltype(c.p)>(s_cold + (word * BLOCK + threadIdx.x) * 8);
  };
  auto word4 = [&](auto &c, int word, int h) {  // 4-byte halves of a word, in separate rows
    c.p = reinterpret_cast<decltype(c.p)>(s_cold + word * BLOCK * 8 + (h * BLOCK + threadIdx.x) * 4);
  };
  auto cell = [&](auto &c, int word) {
    if constexpr (COLD)
      word8(c, word);
    else
      c.v = 0;
  };
  auto half = [&](auto &c, int word, int h) {
    if constexpr (COLD)
      word4(c, word, h);
    else
      c.v = 0;
  };
  // Distance to the nearest cavity (infinite without one) and, in boundary
  // mode, its index.
  Cell<T, true> dcav;
  Cell<int, true> icav;
  constexpr int kCavWord = COLD ? 9 : 0;
  dcav.p = reinterpret_cast<volatile T *>(s_cold + (kCavWord * BLOCK) * 8 + threadIdx.x * sizeof(T));
  icav.p = reinterpret_cast<volatile int *>(s_cold + (kCavWord * BLOCK) * 8 + BLOCK * sizeof(T) + threadIdx.x * 4);

  uint32_t job = 0;
  Cell<T, COLD> px, py, pz, u, pv, best2;
  Cell<uint64_t, true> wid;
  Cell<uint32_t, true> site, walk;
  Cell<uint32_t, COLD> steps, best_tri;  // best_tri: leaf-order index of the walk's nearest triangle
  cell(px, 0);
  cell(py, 1);
  cell(pz, 2);
  cell(u, 3);
  cell(pv, 4);
  cell(best2, 5);
  word8(wid, COLD ? 6 : 1);
  word4(site, COLD ? 7 : 2, 0);
  word4(walk, COLD ? 7 : 2, 1);
  half(steps, 8, 0);
  half(best_tri, 8, 1);
  // Gradient mode: first-ball radius, payoff increments and direction, and
  // the ball source terms of grad U / grad P.
  Cell<T, COLD> g_r0, g_u0, g_p0, g_w0[3], g_su[3], g_sp[3];
  if constexpr (GRAD) {
    cell(g_r0, 11);
    cell(g_u0, 12);
    cell(g_p0, 13);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      cell(g_w0[k], 14 + k);
      cell(g_su[k], 17 + k);
      cell(g_sp[k], 20 + k);
    }
  }
  // Query state.  The FP64 form prunes in FP32 (cull.p, cull.limit); the
  // mixed form's position and best2 are FP32 themselves.
  Cull cull{{0.f, 0.f, 0.f}, 0.f, 0.f, 0};
  int node = 0, sp = 0;
  bool have = false, found = false;
  // Four-wide form: this query continues on the binary BVH (set when a
  // four-wide visit would overflow the stack).
  bool narrow = false;
  // The query reads its cell's candidate list: node = the entry at hand (its
  // triangle in tri_cur, the bits of its centre distance in tri_end), sp = the
  // bits of the distance from the cell centre; FP32: have = a triangle, iter,
  // improved best2, second = the smallest distance of another one.
  constexpr bool LISTS = !WIDE;
  bool list = false;
  float second = CUDART_INF_F;
  bool resume = false;  // FP64 form: back to the traversal after the candidates' test
  bool tri_ok = false;    // best_tri belongs to this walk
  uint32_t tri_cur = 0, tri_end = 0, iter = 0;
  // CLAIM: walks a lane claims from the queue at once, run one after
  // another: s_claim[thread] of them, wid + 1 onwards, are not yet started
  // (shared memory, read only at refills).  A compile-time variant, so the
  // default kernel's refill stays one atomic per warp and one start per lane.
  __shared__ uint32_t s_claim[CLAIM ? BLOCK : 1];
  if (CLAIM) s_claim[threadIdx.x] = 0u;

  // Squared bound that prunes a subtree.
  auto prune_limit = [&]() -> float {
    if constexpr (sizeof(T) == 4)
      return LISTS && list ? cull.limit : best2.v;
    else
      return cull.limit;
  };
  auto set_best2 = [&](T v) { best2 = v; };
  // FP64 form: the held candidates' FP64 test.
  auto flush = [&](const GeoDesc &G, const Vec<T> &pos) {
    if constexpr (sizeof(T) == 8) {
      if (cull.count == 0) return;
      double b2 = best2;
      uint32_t tri = best_tri;
      if (cull_flush(G, pos, cull, b2, tri, stack + kShared * BLOCK, BLOCK)) {
        best2 = b2;
        best_tri = tri;
        found = tri_ok = true;
      }
    }
  };
  // The grid's bounds and record word at pos (the mixed form's upper bound
  // comes later: begin_query).
  auto walk_grid = [&](const GeoDesc &G, const Vec<T> &pos, float &bound, float &upper, int &entry_node) {
    if (!G.grid) return false;
    if constexpr (sizeof(T) == 4) {
      return grid_bounds<false>(G, pos, bound, upper, entry_node);
    } else {
      const double p3[3] = {pos.x, pos.y, pos.z};
      return grid_bounds<true>(G, to_frame<float>(p3, G), bound, upper, entry_node);
    }
  };
  // Starts the query at pos; `in_grid`: with the grid's upper bound and entry
  // node there.
  auto begin_query = [&](const JobDesc &J, const GeoDesc &G, const Vec<T> &pos, bool in_grid, float bound,
                         float upper, int entry_node, T dc) {
    T best2 = static_cast<T>(J.query_radius2);
    found = false;
    node = 0;
    // Entry node: with an initial bound b below one entry cell, every triangle
    // outside the cell's entry subtree is farther than b (the table keeps every
    // triangle within a cell size plus 4 delta), so the traversal starts there.
    // The grid's upper bound plus 6 delta (its 3 delta and the query's own
    // error, with room) serves as b before any triangle is found.  (The
    // four-wide form starts at its root: the table holds binary nodes.)
    if constexpr (sizeof(T) == 8) {
      if (!cull_begin(G, pos, best2, cull)) {
        const uint32_t warm = L.warm && tri_ok ? static_cast<uint32_t>(best_tri) : kNoTri;
        const Plain64 r = nearest_plain64(&G, pos.x, pos.y, pos.z, best2, warm);
        err |= r.flags & 0x7fffffffu;
        found = tri_ok = r.flags >> 31;
        set_best2(r.best2);
        best_tri = r.tri;
        phase = kStep;
        return;
      }
    }
    list = false;
    if constexpr (sizeof(T) == 4) {
      // A point of a cell with a list is at most kListReach spacings and half
      // a cell's diagonal from the surface: bound enough for its short search.
      if (in_grid) upper = LISTS && is_list(entry_node) ? (kListReach + 0.9f) * G.grid_h : grid_upper(G, pos);
    }
    const float ubs = __fmaf_ru(6.f, G.delta, upper);
    // A cavity nearer than the mesh decides the step, so the search goes no
    // farther than the cavity, and with a mesh known to be beyond there is
    // none -- once the mesh is known to lie within the query radius.  (Design
    // loop around an inserted cavity, 262,144 walks on 5,120 triangles with
    // the grid steps off: 29 ms without, 5 with.)
    if (dc < static_cast<T>(CUDART_INF_F) &&
        ((in_grid && static_cast<T>(ubs) * static_cast<T>(ubs) < best2) || J.query_radius2 == CUDART_INF)) {
      if (dc <= static_cast<T>(in_grid ? fmaxf(bound, 0.f) : 0.f)) {
        set_best2(static_cast<T>(CUDART_INF_F));
        found = true;
        if (sizeof(T) == 8) cull.count = 0;
        phase = kStep;
        return;
      }
      const T lim = dc * dc * (T(1) + T(0x1.0p-20));
      if (lim < best2) {
        best2 = lim;
        found = true;
        if constexpr (sizeof(T) == 8) cull.limit = fminf(cull.limit, cull_limit(best2, cull.margin));
      }
    }
    if (in_grid) {
      if constexpr (LISTS) {
        list = is_list(entry_node);
        if (!list && entry_node >= 0 && ubs < G.entry_radius) node = entry_node;
      }
      // A triangle is to be found below the bound (see the step).
      if constexpr (sizeof(T) == 4) {
        best2 = fminf(best2, ubs * ubs);
      } else {
        const float reach = __fadd_ru(ubs, cull.margin), reach2 = __fmul_ru(reach, reach);
        cull.limit = fminf(cull.limit, reach2);
        if (static_cast<double>(reach2) < best2) {
          best2 = static_cast<double>(reach2);
          found = false;
        }
      }
    }
    set_best2(best2);
    iter = 0;
    phase = kTraverse;
    if (LISTS && list) {
      // The candidates hold every triangle that can be nearest (or within 3
      // delta of it) at a point of the cell, nearest to the cell's centre
      // first.
      const Vec<float> q = [&]() -> Vec<float> {
        if constexpr (sizeof(T) == 4)
          return pos;
        else
          return cull.p;
      }();
      sp = __float_as_int(__fmaf_ru(2.f, G.delta, cell_offset(G, q)));
      node = static_cast<int>(list_start(entry_node)) + 1;
      const uint2 e = __ldg(G.lists + node);
      tri_cur = e.x;
      tri_end = e.y;
      have = false;
      second = CUDART_INF_F;
      if constexpr (sizeof(T) == 4) cull.limit = best2;
      return;
    }
    sp = 0;
    have = true;
    narrow = false;
    // Warm start: the walk's previous nearest triangle is tested first, so
    // the search prunes with its distance from the first node on.  (In the
    // FP64 form the grid's bound prunes as well: 38.0 against 39.3 ms with
    // both on 1.02 M walks of the 81,920-triangle noise sphere.)
    tri_cur = tri_end = 0;
    if (L.warm && tri_ok && (sizeof(T) == 4 || !in_grid)) {
      tri_cur = best_tri;
      tri_end = tri_cur + 1;
    }
  };

  for (;;) {
    // Starts walk `wid` on this lane (its first radius from the per-site
    // pre-pass when there is one).
    auto start_walk = [&]() {
      const uint64_t id = wid;
      job = find_job(s_jobs, L.n_jobs, id);
      const JobDesc &J = s_jobs[job];
      // (A 64-bit division takes four times as long as a 32-bit one.)
      const uint64_t local = id - J.walk_begin;
      const uint32_t at = local >> 32 ? static_cast<uint32_t>(local / J.walks) : static_cast<uint32_t>(local) / J.walks;
      site = at;
      walk = static_cast<uint32_t>(local - static_cast<uint64_t>(at) * J.walks);
      const GeoDesc &G = s_geos[J.geo];
      bool skip = false;
      Vec<T> pos;
      if (L.walk_start) {
        const double *st = L.walk_start + 3ull * id;
        skip = isnan(st[0]);
        pos = to_frame<T>(st, G);
      } else {
        pos = to_frame<T>(L.sites + 3ull * (J.site_begin + at), G);
      }
      px = pos.x;
      py = pos.y;
      pz = pos.z;
      u = T(0);
      pv = T(0);
      steps = 0;
      tri_ok = false;
      if (GRAD) g_r0 = T(0);
      if (!skip && (J.flags & kJobSkipCavitySites)) {
        const T R = to_T<T>(J.cavity_radius);
        for (uint32_t c = 0; c < J.n_cav; ++c) {
          const Vec<T> cc = to_frame<T>(L.cavities + 3ull * (J.cav_begin + c), G);
          const Vec<T> dv = sub(pos, cc);
          if (sqrt(dot3(dv, dv)) <= R) skip = true;
        }
      }
      if (skip) {
        if (MODE != kModeBoundary) static_cast<T *>(L.u_out)[id] = T(0);
        if (PAIRED) static_cast<T *>(L.p_out)[id] = T(0);
        if (GRAD)
          for (int k = 0; k < 6; ++k) static_cast<T *>(L.grad_out)[6ull * id + k] = T(0);
        if (MODE == kModeBoundary) L.hits[id].cavity = -2;
        L.steps_out[id] = 0u;
      } else if (L.site_best2 && (MODE != kModeBoundary || L.site_tri)) {
        // First query answered by the per-site pre-pass.
        best2 = static_cast<const T *>(L.site_best2)[J.site_rank + at];
        found = best2 >= T(0);
        if (MODE == kModeBoundary && found) {
          best_tri = L.site_tri[J.site_rank + at];
          tri_ok = true;
        }
        dcav = CUDART_INF_F;
        phase = J.n_cav ? kFirst : kStep;
      } else {
        phase = kBegin;
      }
    };

    // ---- refill idle lanes from the work queue (CLAIM: from their own
    // claims first)
    const unsigned idle = __ballot_sync(full, on && phase == kIdle);
    if constexpr (CLAIM) {
      if (idle != 0u) {
        const unsigned pending = __ballot_sync(full, s_claim[threadIdx.x] != 0u);
        if ((!exhausted || pending != 0u) && (__popc(idle) >= L.refill || idle == on_mask)) {
          uint32_t claim_left = s_claim[threadIdx.x];
          const unsigned claim = __ballot_sync(full, on && phase == kIdle && claim_left == 0u);
          if (!exhausted && claim != 0u) {
            const uint64_t span = static_cast<uint64_t>(lane_walks_of(L)) * __popc(claim);
            unsigned long long base = 0;
            const int leader = __ffs(claim) - 1;
            if (static_cast<int>(lane) == leader) base = atomicAdd(L.counter, static_cast<unsigned long long>(span));
            base = __shfl_sync(full, base, leader);
            if (base + span >= L.total_walks) exhausted = true;
            if (on && phase == kIdle && claim_left == 0u) {
              const uint64_t first =
                  base + static_cast<uint64_t>(lane_walks_of(L)) * __popc(claim & ((1u << lane) - 1u));
              if (first < L.total_walks) {
                wid = first - 1;  // wraps for the first walk of the queue; wid + 1 is exact
                const uint64_t left = L.total_walks - first;
                claim_left = left < lane_walks_of(L) ? static_cast<uint32_t>(left) : lane_walks_of(L);
              }
            }
          }
          if (phase == kIdle && claim_left != 0u) {
            wid = wid + 1;
            --claim_left;
            start_walk();
          }
          s_claim[threadIdx.x] = claim_left;
        }
      }
    } else if (!exhausted && idle != 0u && (__popc(idle) >= L.refill || idle == on_mask)) {
      unsigned long long base = 0;
      const int leader = __ffs(idle) - 1;
      if (static_cast<int>(lane) == leader)
        base = atomicAdd(L.counter, static_cast<unsigned long long>(__popc(idle)));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= L.total_walks) exhausted = true;
      if (on && phase == kIdle) {
        const uint64_t id = base + __popc(idle & ((1u << lane) - 1u));
        if (id < L.total_walks) {
          wid = id;
          start_walk();
        }
      }
    }

    // ---- batched walk step for lanes whose query has finished
    const unsigned ready = __ballot_sync(full, phase >= kStep);
    const unsigned trav = __ballot_sync(full, phase == kTraverse);
    if (ready != 0u && (__popc(ready) >= L.step_threshold || trav == 0u) && phase >= kStep) {
      const JobDesc &J = s_jobs[job];
      const GeoDesc &G = s_geos[J.geo];
      // One pass; `break` leaves it once the lane's next phase is set.
      do {
        Vec<T> pos{px, py, pz};
        if (phase == kStep) {
          flush(G, pos);
          if (resume) {
            // Only the full candidate list was due; the search goes on.
            resume = false;
            phase = kTraverse;
            break;
          }
          if (!found && static_cast<T>(best2) < static_cast<T>(J.query_radius2)) {
            // None below the grid's bound (grid_start).  Where a mixed
            // search has gone on from the previous triangle and an entry node,
            // the bound is the distance; else the search is made without it.
            if (sizeof(T) == 4 && L.warm && tri_ok && sqrtf(static_cast<float>(best2)) < G.entry_radius)
              found = true;
            else
              phase = kAgain;
          }
        }
        if (phase == kStep) {
          T d = sqrt(static_cast<T>(best2));
          if (!found) {
            err |= TWOS_DEVERR_QUERY;
            d = T(0);  // ends the walk; the call reports the failure
          }
          const T dmesh = d, dc = dcav;
          if (dc < d) d = dc;
          // Boundary mode: the first strictly nearer cavity (closest_boundary,
          // wih_twos.cpp:612-624).  Gradient mode: the exit is on a cavity.
          const int hit_cav = dc < dmesh ? static_cast<int>(icav) : -1;
          const bool cav_nearer = dc < dmesh;
          // The mixed form shrinks the radius by the FP32 distance error bound;
          // the FP64 form uses the distance itself (wih_twos.cpp:645-647).
          const T r = sizeof(T) == 4 ? d - static_cast<T>(G.delta) : d;
          bool done = !(r > to_T<T>(J.epsilon));
          bool cap = false;
          if (!done) {
            const uint32_t ctr3 = J.repeat << 3;
            const uint32_t step = steps, wk = walk, key = J.site_offset + site;
            Philox4 q0;
            Vec<T> a = pos;
            if constexpr (!GREEN) {
              Philox4 q[1];
              philox_blocks(J.k0, J.k1, step, wk, key, ctr3, q);
              q0 = q[0];
            } else {
              Philox4 q[4];
              philox_blocks(J.k0, J.k1, step, wk, key, ctr3, q);
              q0 = q[0];
              const Philox4 q1 = q[1], q2 = q[2], q3 = q[3];
              const T beta = median3(uniform<T>(q2.x, q2.y), uniform<T>(q2.z, q2.w), uniform<T>(q3.x, q3.y));
              const Vec<T> g = direction<T>(uniform<T>(q1.x, q1.y), uniform<T>(q1.z, q1.w));
              a = add_scaled(pos, g, r * beta);
            }
            if (EXACT) {
              u = exact_source(static_cast<T>(u), s_terms, J.src_begin, J.n_src, pos, r, err);
              if (PAIRED) pv = exact_source(static_cast<T>(pv), s_terms, J.adj_begin, J.n_adj, pos, r, err);
            } else {
              const T w = r * r / T(6);
              if constexpr (PAIRED) {
                T su, sp;
                source_values(s_terms, J.src_begin, J.n_src, J.adj_begin, J.n_adj, a, su, sp);
                const T du = w * su, dp = w * sp;
                u = u + du;
                pv = pv + dp;
                if (GRAD && step == 0) {
                  g_u0 = du;
                  g_p0 = dp;
                }
              } else if (MODE != kModeBoundary) {
                u = u + w * source_value(s_terms, J.src_begin, J.n_src, a);
              }
            }
            const Vec<T> dir = direction<T>(uniform<T>(q0.x, q0.y), uniform<T>(q0.z, q0.w));
            if (GRAD && step == 0) {
              // First ball: the sphere term's radius and direction, and one draw
              // (blocks 4-5) for the ball source term of the gradient,
              // R (1 - t^3) f(x + t R w') w' with t ~ U(0,1), w' uniform.
              Philox4 qb[2];
              philox_blocks(J.k0, J.k1, 0u, wk, key, ctr3 | 4u, qb);
              const Philox4 q4 = qb[0], q5 = qb[1];
              const T t = uniform<T>(q4.x, q4.y);
              const Vec<T> wp = direction<T>(uniform<T>(q4.z, q4.w), uniform<T>(q5.x, q5.y));
              const Vec<T> z = add_scaled(pos, wp, t * r);
              const T wt = r * (T(1) - t * t * t);
              T su, sq;
              source_values(s_terms, J.src_begin, J.n_src, J.adj_begin, J.n_adj, z, su, sq);
              const T fs = wt * su, fq = wt * sq;
              g_su[0] = wp.x * fs;
              g_su[1] = wp.y * fs;
              g_su[2] = wp.z * fs;
              g_sp[0] = wp.x * fq;
              g_sp[1] = wp.y * fq;
              g_sp[2] = wp.z * fq;
              g_r0 = r;
              g_w0[0] = dir.x;
              g_w0[1] = dir.y;
              g_w0[2] = dir.z;
            }
            pos = add_scaled(pos, dir, r);
            px = pos.x;
            py = pos.y;
            pz = pos.z;
            steps = step + 1;
            if (static_cast<int>(step + 1) >= J.max_steps) {
              done = true;
              cap = true;
            }
          }
          if (done) {
            if (MODE == kModeBoundary) {
              HitRec h;
              h.pad = 0;
              Vec<T> q{T(0), T(0), T(0)}, nrm{T(0), T(0), T(0)};
              if (cap || !found) {
                h.cavity = -2;
              } else if (hit_cav >= 0) {
                // Point on the sphere along the radial direction; the domain
                // excludes the sphere, so the outward normal points into it.
                const Vec<T> cc = to_frame<T>(L.cavities + 3ull * (J.cav_begin + hit_cav), G);
                const Vec<T> dv = sub(pos, cc);
                const T inv = T(1) / sqrt(dot3(dv, dv));
                const Vec<T> dir{dv.x * inv, dv.y * inv, dv.z * inv};
                q = add_scaled(cc, dir, to_T<T>(J.cavity_radius));
                nrm = {dir.x * T(-1), dir.y * T(-1), dir.z * T(-1)};
                h.cavity = hit_cav;
              } else {
                Vec<T> ta, tb, tc;
                load_tri(geo_tris<T>(G), best_tri, ta, tb, tc);
                q = tri_closest(pos, ta, tb, tc);
                if (dmesh > T(0)) {
                  const T inv = T(1) / dmesh;
                  const Vec<T> dq = sub(q, pos);
                  nrm = {dq.x * inv, dq.y * inv, dq.z * inv};
                }
                h.cavity = -1;
              }
              const bool f32 = sizeof(T) == 4;
              h.point[0] = static_cast<double>(q.x) + (f32 ? G.center[0] : 0.0);
              h.point[1] = static_cast<double>(q.y) + (f32 ? G.center[1] : 0.0);
              h.point[2] = static_cast<double>(q.z) + (f32 ? G.center[2] : 0.0);
              h.normal[0] = static_cast<double>(nrm.x);
              h.normal[1] = static_cast<double>(nrm.y);
              h.normal[2] = static_cast<double>(nrm.z);
              L.hits[wid] = h;
            } else {
              if (GRAD) {
                // Dirichlet data of u at the exit point on the mesh.
                if (!cap && found && J.n_bnd > 0 && !cav_nearer) {
                  Vec<T> q = pos;
                  if (tri_ok) {
                    Vec<T> ta, tb, tc;
                    load_tri(geo_tris<T>(G), best_tri, ta, tb, tc);
                    q = tri_closest(pos, ta, tb, tc);
                  }
                  u = u + source_value(s_terms, J.bnd_begin, J.n_bnd, q);
                }
                T *go = static_cast<T *>(L.grad_out) + 6ull * wid;
                const T r0 = g_r0;
                if (r0 > T(0)) {
                  const T k = T(3) / r0;
                  const T cu = k * (u - g_u0), cp = k * (pv - g_p0);
#pragma unroll
                  for (int a = 0; a < 3; ++a) {
                    go[a] = g_w0[a] * cu + g_su[a];
                    go[3 + a] = g_w0[a] * cp + g_sp[a];
                  }
                } else {
                  for (int k = 0; k < 6; ++k) go[k] = T(0);
                }
              }
              static_cast<T *>(L.u_out)[wid] = u;
            }
            if (PAIRED) static_cast<T *>(L.p_out)[wid] = pv;
            L.steps_out[wid] = steps | (cap ? 0x80000000u : 0u);
            phase = kIdle;
            break;
          }
        }
        // The nearest cavity at the new position.
        T dc = CUDART_INF_F;
        if (J.n_cav) {
          const T R = to_T<T>(J.cavity_radius);
          int nearest_cav = -1;
          for (uint32_t c = 0; c < J.n_cav; ++c) {
            const Vec<T> cc = to_frame<T>(L.cavities + 3ull * (J.cav_begin + c), G);
            const Vec<T> dv = sub(pos, cc);
            const T len = sqrt(dot3(dv, dv));
            if (len - R < dc && (MODE != kModeBoundary || len > T(0))) {
              dc = len - R;
              nearest_cav = static_cast<int>(c);
            }
          }
          if (MODE == kModeBoundary) icav = nearest_cav;
        }
        dcav = dc;
        if (phase == kFirst) {
          phase = kStep;
          break;
        }
        // Distance-bound grid: D(v) - |x - v| over the corners v of x's cell
        // bounds the mesh distance from below; a bound of at least grid_tau
        // spacings is the next ball's radius and no query is needed.  A grid
        // step never ends a walk: the bound must clear the termination shell
        // with room to spare.  The FP64 form takes no grid steps (with GRID64
        // it does, a comparison of precision alone); its queries only start
        // from the grid's upper bound and entry node.  It evaluates the grid
        // at the FP32 image of the position, within a few 1e-8 of it, and
        // bound <= d - delta covers that.
        float bound = 0.f, upper = CUDART_INF_F;
        int entry_node = -1;
        bool in_grid = false;
        if (L.entry || ((sizeof(T) == 4 || GRID64) && L.grid_tau > 0.f))
          in_grid = walk_grid(G, pos, bound, upper, entry_node);
        if constexpr (sizeof(T) == 4 || GRID64) {
          const T b = static_cast<T>(bound);
          if (in_grid && L.grid_tau > 0.f && bound >= L.grid_tau * G.grid_h &&
              bound > 2.f * (static_cast<float>(J.epsilon) + G.delta) && b * b < static_cast<T>(J.query_radius2) &&
              phase == kStep) {
            best2 = b * b;
            found = true;
            ++c_grid;
            if constexpr (TRACE) {
              const unsigned long long slot = atomicAdd(L.trace_count, 1ull);
              if (slot < L.trace_cap) L.trace[slot] = make_float4(pos.x, pos.y, pos.z, bound);
            }
            // The step itself comes with the warp's next batch.
            break;
          }
        }
        begin_query(J, G, pos, in_grid && L.entry && phase != kAgain, bound, upper, entry_node, dc);
      } while (false);
    }

    if (__ballot_sync(full, phase != kIdle) == 0u) {
      if (exhausted && (!CLAIM || __ballot_sync(full, s_claim[threadIdx.x] != 0u) == 0u)) break;
      continue;
    }

    // ---- a batch of traversal units for every traversing lane.  With `vote`
    // only the lanes whose next unit is of the commoner kind -- triangle, or
    // node and pops -- take it.
    bool take = phase == kTraverse;
    if (L.vote) {  // warp-uniform; the ballots cost nothing when it is off
      const bool want_tri = phase == kTraverse && tri_cur < tri_end;
      const unsigned vt = __ballot_sync(full, want_tri);
      const unsigned vn = __ballot_sync(full, phase == kTraverse && !want_tri);
      const bool tri_turn = __popc(vt) >= __popc(vn);
      take = take && want_tri == tri_turn;
    }
    if (take) {
      const GeoDesc &G = s_geos[s_jobs[job].geo];
      const Vec<float> pos = [&]() -> Vec<float> {  // the FP32 query point
        if constexpr (sizeof(T) == 4)
          return {px, py, pz};
        else
          return cull.p;
      }();
      // Up to `units` units back to back before the warp returns to the
      // refill and step ballots: the loop overhead is paid once per batch.
      auto fail = [&](uint32_t bit) {
        err |= bit;
        found = false;
        set_best2(static_cast<T>(CUDART_INF_F));
        cull.count = 0;
        resume = false;
        phase = kStep;
      };
#pragma unroll 1
      for (int unit = 0; unit < units; ++unit) {
        if constexpr (LISTS) {
          if (list) {
            const float low = __uint_as_float(tri_end) - __int_as_float(sp);
            if (tri_end == 0x7f800000u || (low > 0.f && !(low * low < prune_limit()))) {
              // No later candidate is nearer.  FP32: with another triangle
              // within rounding of the minimum, the value depends on the
              // order of the tests, and the traversal's is the one to return.
              list = false;
              if (sizeof(T) == 8 || (found && !(have && second < cull.limit))) {
                if (sizeof(T) == 4 && have) {
                  best_tri = iter;
                  tri_ok = true;
                }
                phase = kStep;
                break;
              }
              if constexpr (sizeof(T) == 4) {
                if (have) {
                  best2 = cull.limit;
                  found = false;
                }
                const int start = entry_of(G, cell_word(G, pos));
                node = start >= 0 && sqrtf(best2) < G.entry_radius ? start : 0;
                sp = 0;
                have = true;
                iter = 0;
                tri_cur = tri_end = 0;
                if (L.warm && tri_ok) {
                  tri_cur = best_tri;
                  tri_end = tri_cur + 1;
                }
              }
            }
          }
        }
        // The unit's triangle or node: the leaf at hand, else the current
        // node or the next stack entry still closer than the current best.
        if (!(LISTS && list) && tri_cur >= tri_end) {
          while (!have && sp > 0) {
            --sp;
            const uint2 e = sp < kShared ? stack[sp * BLOCK] : deep[sp - kShared];
            if (__uint_as_float(e.y) < prune_limit()) {
              node = static_cast<int>(e.x);
              have = true;
            }
          }
          if (!have) {
            phase = kStep;
            break;
          }
          if (node < 0) {
            const uint32_t enc = ~static_cast<uint32_t>(node);
            tri_cur = enc >> 3;
            tri_end = tri_cur + (enc & 7u);
            have = false;
          }
        }
        if ((sizeof(T) == 8 || !(LISTS && list)) && ++iter > G.max_iter) {
          fail(TWOS_DEVERR_ITER);
          break;
        }
        if constexpr (WIDE) {
          if (tri_cur >= tri_end && have && !narrow) {
            // Four-wide node: its valid children sorted nearest first (a
            // five-comparator network); the nearest is next, the others are
            // pushed farthest first.
            ++c_nodes;
            float d[4];
            int c[4];
            node4_dist2(G.nodes4_f, node, pos, d, c);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (!(d[k] < prune_limit())) d[k] = CUDART_INF_F;
            order2(d[0], c[0], d[1], c[1]);
            order2(d[2], c[2], d[3], c[3]);
            order2(d[0], c[0], d[2], c[2]);
            order2(d[1], c[1], d[3], c[3]);
            order2(d[1], c[1], d[2], c[2]);
            const int nv =
                (d[0] < CUDART_INF_F) + (d[1] < CUDART_INF_F) + (d[2] < CUDART_INF_F) + (d[3] < CUDART_INF_F);
            if (nv == 0) {
              have = false;
            } else if (sp + nv - 1 > kStack) {
              // Up to three pushes per level can outgrow the stack on a
              // root-started query with a loose bound.  The query goes on
              // from the binary root with the bound found so far (one push
              // per level there): every triangle nearer than best2 is still
              // reached.
              narrow = true;
              sp = 0;
              node = 0;
            } else {
              if (nv > 3) push(sp, make_uint2(static_cast<uint32_t>(c[3]), __float_as_uint(d[3])));
              if (nv > 2) push(sp, make_uint2(static_cast<uint32_t>(c[2]), __float_as_uint(d[2])));
              if (nv > 1) push(sp, make_uint2(static_cast<uint32_t>(c[1]), __float_as_uint(d[1])));
              node = c[0];
            }
            continue;
          }
        }
        // One set of loads for either kind (64 bytes of a triangle or 96 of a
        // node): lanes on nodes and lanes on triangles wait for memory
        // together, once per unit, before the warp splits on the arithmetic.
        const bool on_tri = (LISTS && list) || tri_cur < tri_end;
        const char *at = on_tri ? reinterpret_cast<const char *>(G.tris_f + tri_cur)
                                : reinterpret_cast<const char *>(G.nodes_f + node);
        float4 r0, r1, r2, r3, r4{}, r5{};
        ldg32(at, r0, r1);
        ldg32(at + 32, r2, r3);
        ldg32_if(!on_tri, at + 64, r4, r5);
        uint2 next = make_uint2(tri_cur + 1u, tri_end);
        if (LISTS && list) next = __ldg(G.lists + node + 1);
        if (on_tri) {
          ++c_planes;
          if constexpr (sizeof(T) == 4) {
            if (plane_gap2(r0, r1, pos) < prune_limit()) {
              ++c_tris;
              const float d2 = tri_dist2(pos, Vec<float>{r1.x, r1.y, r1.z}, Vec<float>{r2.x, r2.y, r2.z},
                                         Vec<float>{r3.x, r3.y, r3.z});
              const bool nearer = d2 < best2;
              if (LISTS && list) {
                if (!nearer || have) second = fminf(second, nearer ? best2.v : d2);
                if (nearer) {
                  cull.limit = widen2(d2, 3.f * G.delta);
                  iter = tri_cur;
                  have = true;
                }
              } else if (nearer) {
                best_tri = tri_cur;
                tri_ok = true;
              }
              if (nearer) {
                best2 = d2;
                found = true;
              }
            }
          } else {
            // A full candidate list is tested first; the triangle comes again.
            if (cull_tri(tri_cur, r0, r1, r2, r3, cull, stack + kShared * BLOCK, BLOCK, c_tris)) {
              resume = true;
              phase = kStep;
              break;
            }
          }
          tri_cur = next.x;
          tri_end = next.y;
          if (LISTS && list) ++node;
        } else {
          ++c_nodes;
          float dl, dr;
          int cl, cr;
          node_bounds(r0, r1, r2, r3, r4, r5, pos, dl, dr, cl, cr);
          const float limit = prune_limit();
          const bool vl = dl < limit, vr = dr < limit;
          const bool swap = dr < dl;
          if (vl && vr) {
            if (sp >= kStack) {
              fail(TWOS_DEVERR_STACK);
              break;
            }
            push(sp, make_uint2(static_cast<uint32_t>(swap ? cl : cr), __float_as_uint(swap ? dl : dr)));
          }
          have = vl || vr;
          node = vl && !(vr && swap) ? cl : cr;
        }
      }
    }
  }
  if (err) atomicOr(L.error, err);
  if (L.counters) {
    unsigned long long n_nodes = c_nodes, n_planes = c_planes, n_tris = c_tris, n_grid = c_grid;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      n_nodes += __shfl_xor_sync(full, n_nodes, o);
      n_planes += __shfl_xor_sync(full, n_planes, o);
      n_tris += __shfl_xor_sync(full, n_tris, o);
      n_grid += __shfl_xor_sync(full, n_grid, o);
    }
    if (lane == 0) {
      atomicAdd(&L.counters[0], n_nodes);
      atomicAdd(&L.counters[1], n_planes);
      atomicAdd(&L.counters[2], n_tris);
      if (n_grid) atomicAdd(&L.counters[3], n_grid);
    }
  }
}

// ---------------------------------------------------------------- warp search
// One query by a whole warp, for the few long queries a call starts with (a
// site deep inside visits hundreds of nodes, and one lane waits for memory at
// each): up to 32 entries of a common stack are taken at once, a lane each.
// The grid's bound is close to the distance, so almost all of them have to be
// visited in any order.  `limit` is the squared pruning threshold at entry;
// leaf(i, rows, limit) tests triangle i (its four float4) and returns the
// lane's new threshold.  SLABS: node bounds with the normal slabs (distances
// to triangles) or boxes only.
//
// The stack holds kWarpStack entries per warp; near its end one entry at a
// time is taken, which needs at most one more per level.
constexpr int kWarpStack = 512;
template <bool SLABS, typename Leaf>
__device__ __forceinline__ void warp_search(const GeoDesc &g, const Vec<float> &p, int root, float &limit,
                                            uint2 *stack, uint32_t &err, Leaf &&leaf) {
  const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
  __syncwarp();
  if (lane == 0) stack[0] = make_uint2(static_cast<uint32_t>(root), 0u);
  __syncwarp();
  uint32_t iter = 0;
  for (int size = 1; size > 0;) {
    if (++iter > g.max_iter) {
      err |= TWOS_DEVERR_ITER;
      break;
    }
    const int take = size > kWarpStack - 64 ? 1 : min(size, 32);
    size -= take;
    uint2 e = make_uint2(0u, 0x7f800000u);
    if (static_cast<int>(lane) < take) e = stack[size + take - 1 - static_cast<int>(lane)];
    const bool live = static_cast<int>(lane) < take && __uint_as_float(e.y) < limit;
    const int node = static_cast<int>(e.x);
    float dn = CUDART_INF_F, df = CUDART_INF_F;
    int cn = 0, cf = 0;
    if (live && node < 0) {
      const uint32_t enc = ~static_cast<uint32_t>(node);
      for (uint32_t i = enc >> 3, end = (enc >> 3) + (enc & 7u); i < end; ++i) {
        float4 r[4];
        ldg32(&g.tris_f[i].plane, r[0], r[1]);
        ldg32(&g.tris_f[i].b, r[2], r[3]);
        limit = fminf(limit, leaf(i, r, limit));
      }
    } else if (live) {
      const NodeF *n = g.nodes_f + node;
      float4 x, y, z, nl, nr, t;
      ldg32(&n->x, x, y);
      ldg32(&n->z, z, nl);
      ldg32(&n->nr, nr, t);
      if (!SLABS) nl = nr = t = make_float4(0.f, 0.f, 0.f, 0.f);
      int cl, cr;
      node_bounds(x, y, z, nl, nr, t, p, dn, df, cl, cr);
      if (!SLABS) {
        cl = __float_as_int(__ldg(&n->tail.z));
        cr = __float_as_int(__ldg(&n->tail.w));
      }
      const bool swap = df < dn;
      cn = swap ? cr : cl;
      cf = swap ? cl : cr;
      const float d = dn;
      dn = fminf(d, df);
      df = fmaxf(d, df);
    }
    // Nearer children above the farther ones, the first lane's on top.
    limit = __uint_as_float(__reduce_min_sync(full, __float_as_uint(limit)));
    const unsigned mf = __ballot_sync(full, df < limit), mn = __ballot_sync(full, dn < limit);
    const unsigned above = lane == 31u ? 0u : full << (lane + 1u);
    if (df < limit) stack[size + __popc(mf & above)] = make_uint2(static_cast<uint32_t>(cf), __float_as_uint(df));
    size += __popc(mf);
    if (dn < limit) stack[size + __popc(mn & above)] = make_uint2(static_cast<uint32_t>(cn), __float_as_uint(dn));
    size += __popc(mn);
    __syncwarp();
  }
}

// The smallest value of the warp and its triangle, to every lane (ties: the
// lower leaf-order index).
template <typename T> __device__ __forceinline__ void warp_best(T &best, uint32_t &tri) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const T b = __shfl_xor_sync(0xffffffffu, best, o);
    const uint32_t t = __shfl_xor_sync(0xffffffffu, tri, o);
    if (b < best || (b == best && t < tri)) {
      best = b;
      tri = t;
    }
  }
}

// nearest_geo() by a warp (all lanes with the same arguments).
//
// FP32: which of several triangles within rounding of the minimum a lane's
// traversal returns depends on its order, because a node bound can exceed a
// contained triangle's distance by rounding.  A site's first distance moves
// all its walks, so the warp's search returns the very value: it collects
// the triangles within 3 delta of the minimum, and if there are several,
// replays the lane's traversal on the nodes that hold them (node_first: a
// node's first triangle), which are few.  No other triangle can change the
// outcome while a node bound and a triangle's distance are together off by
// less than 3 delta, that is 96 * 2^-24 of the mesh's half extent.  Each is off
// by some 4 * 2^-24 (|p|_1 + half the box's diagonal), so points within eight
// half extents (|p|_1 <= 2^22 delta) are searched this way and one lane takes
// the others.  (A cube of 768 triangles and this search at any distance:
// another triangle, or none, from 48 half extents on.)  Distances to triangles
// so small beside their distance that FP32 cannot resolve them can be off by
// more: where the replay then ends without a triangle, the traversal follows.
constexpr int kContend = 256;
constexpr int kWarpEntries = kWarpStack + kContend + 1;  // shared-memory entries per warp
// The search and the replay: 1 with the nearest triangle, 0 with none below
// sqrt(from), -1 where the traversal has to decide, below sqrt(cut) if that
// finds a triangle.
__device__ __forceinline__ int warp_contenders(const GeoDesc &g, const Vec<float> &p, int root, float from, float &cut,
                                               float &best2, uint32_t &best_tri, uint2 *stack, uint32_t &err) {
  const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
  uint2 *list = stack + kWarpStack;
  uint32_t *count = &list[kContend].x;
  float limit = from, mine = CUDART_INF_F;
  __syncwarp();  // the previous call's reads of the list are done
  if (lane == 0) *count = 0u;
  warp_search<true>(g, p, root, limit, stack, err, [&](uint32_t i, const float4 *r, float lim) {
    if (!(plane_gap2(r[0], r[1], p) < lim)) return lim;
    const float d2 = tri_dist2(p, Vec<float>{r[1].x, r[1].y, r[1].z}, Vec<float>{r[2].x, r[2].y, r[2].z},
                               Vec<float>{r[3].x, r[3].y, r[3].z});
    if (!(d2 < lim)) return lim;
    const uint32_t at = atomicAdd(count, 1u);
    if (at < kContend) list[at] = make_uint2(i, __float_as_uint(d2));
    mine = fminf(mine, d2);
    return widen2(d2, 4.f * g.delta);
  });
  mine = __uint_as_float(__reduce_min_sync(full, __float_as_uint(mine)));
  if (!(mine < best2)) return 0;
  // The contenders, one per lane.
  cut = fminf(best2, widen2(mine, 3.f * g.delta));
  const uint32_t n = *count;
  uint32_t held = 0;
  if (n <= kContend) {
    for (uint32_t k = 0; k < n; k += 32) {  // in place: an entry moves only forward
      uint2 c = make_uint2(0u, 0x7f800000u);
      if (k + lane < n) c = list[k + lane];
      const bool keep = __uint_as_float(c.y) < cut;
      const unsigned m = __ballot_sync(full, keep);
      __syncwarp();
      if (keep) list[held + __popc(m & ((1u << lane) - 1u))] = c;
      held += __popc(m);
      __syncwarp();
    }
  }
  if (n > kContend || held > 32u) return -1;  // too many to replay
  uint32_t tri = 0xffffffffu;
  float d2 = CUDART_INF_F, plane2 = CUDART_INF_F;
  if (lane < held) {
    tri = list[lane].x;
    d2 = __uint_as_float(list[lane].y);
    plane2 = tri_plane_gap2(g.tris_f, tri, p);
  }
  if (held == 1u) {
    best2 = mine;
    best_tri = __shfl_sync(full, tri, 0);
    return 1;
  }
  // Replay, by all lanes alike; entries: (node, bound) and the end of the
  // node's triangle range.  The lanes share the stack, so none stores an entry
  // before all have read the last one there, or reads it before it is stored.
  float r = cut;
  bool found = false;
  int sp = 0, node = root;
  uint32_t end = 0xffffffffu;
  for (bool have = true; have;) {
    if (node < 0) {
      const uint32_t enc = ~static_cast<uint32_t>(node), first = enc >> 3, last = first + (enc & 7u);
      for (uint32_t i = first; i < last; ++i) {
        const unsigned who = __ballot_sync(full, tri == i);
        if (who == 0u) continue;
        const int src = __ffs(who) - 1;
        const float pg = __shfl_sync(full, plane2, src), dd = __shfl_sync(full, d2, src);
        if (pg < r && dd < r) {
          r = dd;
          best_tri = i;
          found = true;
        }
      }
    } else {
      float dl, dr;
      int cl, cr;
      node_dist2(g.nodes_f, node, p, dl, dr, cl, cr);
      // (An empty right child: all triangles are on the left.)
      const uint32_t mid = cr >= 0                               ? __ldg(g.node_first + cr)
                           : (~static_cast<uint32_t>(cr) & 7u) ? ~static_cast<uint32_t>(cr) >> 3
                                                               : end;
      const uint32_t begin = cl >= 0 ? __ldg(g.node_first + cl) : ~static_cast<uint32_t>(cl) >> 3;
      const bool vl = __ballot_sync(full, tri >= begin && tri < mid) != 0u && dl < r;
      const bool vr = __ballot_sync(full, tri >= mid && tri < end && lane < held) != 0u && dr < r;
      if (vl || vr) {
        const bool swap = dr < dl;
        if (vl && vr) {
          const int far = swap ? cl : cr;
          __syncwarp();
          stack[2 * sp] = make_uint2(static_cast<uint32_t>(far), __float_as_uint(swap ? dl : dr));
          stack[2 * sp + 1].x = swap ? mid : end;
          __syncwarp();
          ++sp;
        }
        const bool left = vl && !(vr && swap);
        node = left ? cl : cr;
        if (left) end = mid;
        continue;
      }
    }
    have = false;
    while (sp > 0) {
      --sp;
      const uint2 e = stack[2 * sp];
      if (__uint_as_float(e.y) < r) {
        node = static_cast<int>(e.x);
        end = stack[2 * sp + 1].x;
        have = true;
        break;
      }
    }
  }
  if (!found) {
    cut = from;
    return -1;
  }
  best2 = r;
  return 1;
}

__device__ __forceinline__ bool warp_nearest(const GeoDesc &g, const Vec<float> &p, float &best2, uint32_t &best_tri,
                                             uint2 *stack, uint32_t &err, bool = true) {
  const unsigned full = 0xffffffffu;
  float upper;
  int root;
  grid_start(g, p, sqrtf(best2), upper, root);
  const float given = best2, from = fminf(given, upper * upper);
  float cut = from;
  int state = -1;
  if ((fabsf(p.x) + fabsf(p.y) + fabsf(p.z)) * 0x1.0p-22f <= g.delta)
    state = warp_contenders(g, p, root, from, cut, best2, best_tri, stack, err);
  if (state > 0 || (state == 0 && !(from < given))) return state > 0;
  if (state == 0) {  // none below the grid's bound: without it, from the root
    cut = given;
    root = 0;
  }
  // The traversal itself, by one lane (its stack in the warp's memory).
  uint32_t bits = 0;
  bool found = false;
  __syncwarp();
  if ((threadIdx.x & 31u) == 0u) {
#pragma unroll 1
    for (;;) {
      best2 = cut;
      found = nearest<float>(g.nodes_f, g.tris_f, g.max_iter, p, best2, best_tri, stack, 1, bits, root);
      if (found || bits != 0u || !(cut < given)) break;
      if (!(cut < from)) root = 0;
      cut = cut < from ? from : given;
    }
  }
  best2 = __shfl_sync(full, best2, 0);
  best_tri = __shfl_sync(full, best_tri, 0);
  err |= __shfl_sync(full, bits, 0);
  return __shfl_sync(full, static_cast<int>(found), 0) != 0;
}

// The nearest triangle of lanes that hold their own nearest (0xffffffff: none)
// at `own`, `mine` and `tri` the warp's (warp_best).
__device__ __forceinline__ uint32_t warp_tied(const GeoDesc &g, const Vec<double> &p, double own, uint32_t own_tri,
                                              double mine, uint32_t tri, uint32_t ties) {
  const unsigned full = 0xffffffffu;
  const bool holds = own == mine && own_tri != 0xffffffffu;
  ties = __reduce_or_sync(full, holds ? ties : 0u);
  for (unsigned m = __ballot_sync(full, holds && own_tri != tri); m != 0u; m &= m - 1u) {
    const Tied t = first_met(&g, p.x, p.y, p.z, tri, __shfl_sync(full, own_tri, __ffs(m) - 1), 0.0, ties);
    tri = t.tri;
    ties = t.ties;
  }
  return ties & kTieOpen ? first_of_tied(g, p, mine, tri) : tri;
}

// warp_search on the FP64 nodes, for what FP32 cannot hold (16,384 points a
// million half extents away, 81,920 triangles: 6.6 ms with one lane's search
// in each warp).  Entries' bounds are rounded down and the threshold up to FP32.
// Out of line, as nearest_plain64.
__device__ __noinline__ Plain64 warp_plain64(const GeoDesc *g, double x, double y, double z, double best2, bool which,
                                             uint2 *stack) {
  const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
  const Vec<double> p{x, y, z};
  double mine = best2;
  uint32_t tri = 0xffffffffu, ties = 0, bits = 0;
  __syncwarp();
  if (lane == 0) stack[0] = make_uint2(0u, 0u);
  __syncwarp();
  float limit = __double2float_ru(best2);
  uint32_t iter = 0;
  for (int size = 1; size > 0;) {
    if (++iter > g->max_iter) {
      bits = TWOS_DEVERR_ITER;
      break;
    }
    const int take = size > kWarpStack - 64 ? 1 : min(size, 32);
    size -= take;
    uint2 e = make_uint2(0u, 0x7f800000u);
    if (static_cast<int>(lane) < take) e = stack[size + take - 1 - static_cast<int>(lane)];
    const bool live = static_cast<int>(lane) < take && __uint_as_float(e.y) <= limit;
    const int node = static_cast<int>(e.x);
    float dn = CUDART_INF_F, df = CUDART_INF_F;
    int cn = 0, cf = 0;
    if (live && node < 0) {
      const uint32_t enc = ~static_cast<uint32_t>(node);
      for (uint32_t i = enc >> 3, end = (enc >> 3) + (enc & 7u); i < end; ++i) {
        if (!(tri_plane_gap2(g->tris_d, i, p) <= mine)) continue;
        Vec<double> a, b, c;
        load_tri(g->tris_d, i, a, b, c);
        const double d2 = tri_dist2(p, a, b, c);
        if (d2 < mine) {
          mine = d2;
          tri = i;
          ties = 0u;
        } else if (which && d2 == mine && tri != 0xffffffffu) {
          const Tied t = first_met(g, x, y, z, tri, i, 0.0, ties);
          tri = t.tri;
          ties = t.ties;
        }
      }
    } else if (live) {
      double dl, dr;
      int cl, cr;
      node_dist2(g->nodes_d, node, p, dl, dr, cl, cr);
      const bool swap = dr < dl;
      cn = swap ? cr : cl;
      cf = swap ? cl : cr;
      dn = __double2float_rd(swap ? dr : dl);
      df = __double2float_rd(swap ? dl : dr);
    }
    limit = __uint_as_float(__reduce_min_sync(full, __float_as_uint(fminf(limit, __double2float_ru(mine)))));
    // (<=: the bound of a triangle at the smallest distance can round to the threshold.)
    const bool far = df <= limit && df < CUDART_INF_F, near = dn <= limit && dn < CUDART_INF_F;
    const unsigned mf = __ballot_sync(full, far), mn = __ballot_sync(full, near);
    const unsigned above = lane == 31u ? 0u : full << (lane + 1u);
    if (far) stack[size + __popc(mf & above)] = make_uint2(static_cast<uint32_t>(cf), __float_as_uint(df));
    size += __popc(mf);
    if (near) stack[size + __popc(mn & above)] = make_uint2(static_cast<uint32_t>(cn), __float_as_uint(dn));
    size += __popc(mn);
    __syncwarp();
  }
  const double own = mine;
  const uint32_t own_tri = tri;
  warp_best(mine, tri);
  if (tri == 0xffffffffu) return {best2, 0u, bits};
  if (which) tri = warp_tied(*g, p, own, own_tri, mine, tri, ties);
  return {mine, tri, bits | 0x80000000u};
}

// `which`: of several triangles at the distance, the one of first_met is wanted.
__device__ __forceinline__ bool warp_nearest(const GeoDesc &g, const Vec<double> &p, double &best2,
                                             uint32_t &best_tri, uint2 *stack, uint32_t &err, bool which = true) {
  Cull c;
  if (!cull_begin(g, p, best2, c, kFarWarp)) {
    const Plain64 r = warp_plain64(&g, p.x, p.y, p.z, best2, which, stack);
    err |= r.flags & 0x7fffffffu;
    if (!(r.flags >> 31)) return false;
    best2 = r.best2;
    best_tri = r.tri;
    return true;
  }
  float upper;
  int node;
  grid_start(g, c.p, sqrtf(c.limit), upper, node);
  const float reach = __fadd_ru(upper, c.margin), reach2 = __fmul_ru(reach, reach);
  float limit = fminf(c.limit, reach2);
  double mine = fmin(best2, static_cast<double>(reach2));
  uint32_t tri = 0xffffffffu, overrun = 0, ties = 0;
  warp_search<true>(g, c.p, node, limit, stack, overrun, [&](uint32_t i, const float4 *r, float lim) {
    if (!(plane_gap2(r[0], r[1], c.p) < lim)) return lim;
    Vec<double> ta, tb, tc;
    load_tri(g.tris_d, i, ta, tb, tc);
    const double d2 = tri_dist2(p, ta, tb, tc);
    if (!(d2 < mine)) {
      if (which && d2 == mine && tri != 0xffffffffu) {
        const Tied t = first_met(&g, p.x, p.y, p.z, tri, i, 0.0, ties);
        tri = t.tri;
        ties = t.ties;
      }
      return lim;
    }
    mine = d2;
    tri = i;
    ties = 0u;
    return cull_limit(d2, c.margin);
  });
  const double own = mine;
  const uint32_t own_tri = tri;
  warp_best(mine, tri);
  err |= overrun;
  if (tri == 0xffffffffu)
    return overrun == 0u && reach2 < best2 && nearest_plain(g, p, best2, best_tri, err);
  if (which) tri = warp_tied(g, p, own, own_tri, mine, tri, ties);
  best2 = mine;
  best_tri = tri;
  return true;
}

// Per-site first query: one closest-point traversal per site of the launch
// (the N walks of a site all start there), written as the squared mesh
// distance, or -1 when no surface point lies within the query radius.
//
// A warp per site: one thread per site took 634 us for 384 sites of the
// 20,480-triangle noise sphere (426 with the grid's bound), as long as half
// their walks; with a warp each the whole call fell from 1.31 to 1.03 ms.
template <typename T>
__global__ void __launch_bounds__(kWosBlock) site_prepass_kernel(const WosLaunch L) {
  __shared__ uint2 s_stack[kWarpEntries * (kWosBlock / 32)];
  uint2 *stack = s_stack + kWarpEntries * (threadIdx.x >> 5);
  uint32_t err = 0;
  T *out = static_cast<T *>(L.site_best2);
  const uint32_t warps = gridDim.x * (kWosBlock / 32);
  for (uint32_t g = blockIdx.x * (kWosBlock / 32) + (threadIdx.x >> 5); g < L.total_sites; g += warps) {
    uint32_t lo = 0, hi = L.n_jobs - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (L.jobs[mid].site_rank <= g)
        lo = mid;
      else
        hi = mid - 1;
    }
    const JobDesc &J = L.jobs[lo];
    const GeoDesc &G = L.geos[J.geo];
    const Vec<T> p = to_frame<T>(L.sites + 3ull * (J.site_begin + (g - J.site_rank)), G);
    T best2 = static_cast<T>(J.query_radius2);
    uint32_t tri = 0;
    const bool found = warp_nearest(G, p, best2, tri, stack, err, L.site_tri != nullptr);
    if ((threadIdx.x & 31u) == 0) {
      out[g] = found ? best2 : T(-1);
      if (L.site_tri) L.site_tri[g] = tri;
    }
  }
  if (err) atomicOr(L.error, err);
}

cudaError_t launch_site_prepass(int precision, const WosLaunch &L, cudaStream_t s) {
  if (!L.site_best2 || L.total_sites == 0) return cudaSuccess;
  const int grid = static_cast<int>(std::min<uint32_t>((L.total_sites + kWosBlock / 32 - 1) / (kWosBlock / 32), 148u * 16));
  if (precision == TWOS_PREC_MIXED)
    site_prepass_kernel<float><<<grid, kWosBlock, 0, s>>>(L);
  else
    site_prepass_kernel<double><<<grid, kWosBlock, 0, s>>>(L);
  return cudaGetLastError();
}

template <typename T, int MODE, int SRC, int BLOCK> static const void *wos_fn() {
  return reinterpret_cast<const void *>(&wos_kernel<T, MODE, SRC, BLOCK>);
}

template <typename T, int MODE, int BLOCK> static const void *select_src(int src) {
  if (src == TWOS_SOURCE_GREEN) return wos_fn<T, MODE, TWOS_SOURCE_GREEN, BLOCK>();
  if (src == TWOS_SOURCE_EXACT) return wos_fn<T, MODE, TWOS_SOURCE_EXACT, BLOCK>();
  return wos_fn<T, MODE, TWOS_SOURCE_CENTER, BLOCK>();
}

template <int MODE, int BLOCK> static const void *select_wide_src(int src) {
  if (src == TWOS_SOURCE_GREEN)
    return reinterpret_cast<const void *>(&wos_kernel<float, MODE, TWOS_SOURCE_GREEN, BLOCK, false, false, true>);
  return reinterpret_cast<const void *>(&wos_kernel<float, MODE, TWOS_SOURCE_CENTER, BLOCK, false, false, true>);
}

template <int MODE, int BLOCK> static const void *claim_fn() {
  return reinterpret_cast<const void *>(
      &wos_kernel<float, MODE, TWOS_SOURCE_CENTER, BLOCK, false, false, false, true>);
}

template <int BLOCK>
static const void *select_wos_block(int precision, int mode, int src, int grid64, int wide, int claim) {
  // Walk claims (lane_walks > 1): the mixed centre-source modes on the binary BVH.
  if (claim && !wide && precision == TWOS_PREC_MIXED && src == TWOS_SOURCE_CENTER) {
    if (mode == TWOS_MODE_COMPLIANCE) return claim_fn<TWOS_MODE_COMPLIANCE, BLOCK>();
    if (mode == TWOS_MODE_PAIRED) return claim_fn<TWOS_MODE_PAIRED, BLOCK>();
    if (mode == TWOS_MODE_HOT) return claim_fn<TWOS_MODE_HOT, BLOCK>();
  }
  if (wide && precision == TWOS_PREC_MIXED && (src == TWOS_SOURCE_CENTER || src == TWOS_SOURCE_GREEN)) {
    if (mode == TWOS_MODE_COMPLIANCE) return select_wide_src<TWOS_MODE_COMPLIANCE, BLOCK>(src);
    if (mode == TWOS_MODE_PAIRED) return select_wide_src<TWOS_MODE_PAIRED, BLOCK>(src);
    if (mode == TWOS_MODE_HOT) return select_wide_src<TWOS_MODE_HOT, BLOCK>(src);
  }
  if (grid64 && precision == TWOS_PREC_FP64 && mode == TWOS_MODE_COMPLIANCE && src == TWOS_SOURCE_CENTER)
    return reinterpret_cast<const void *>(
        &wos_kernel<double, TWOS_MODE_COMPLIANCE, TWOS_SOURCE_CENTER, BLOCK, false, true>);
  if (mode == kModeBoundary)
    return precision == TWOS_PREC_MIXED ? wos_fn<float, kModeBoundary, TWOS_SOURCE_CENTER, BLOCK>()
                                        : wos_fn<double, kModeBoundary, TWOS_SOURCE_CENTER, BLOCK>();
#define TWOS_PICK(T)                                                                 \
  if (mode == TWOS_MODE_COMPLIANCE) return select_src<T, TWOS_MODE_COMPLIANCE, BLOCK>(src); \
  if (mode == TWOS_MODE_PAIRED) return select_src<T, TWOS_MODE_PAIRED, BLOCK>(src);         \
  if (mode == kModeGradient) return select_src<T, kModeGradient, BLOCK>(src);               \
  return select_src<T, TWOS_MODE_HOT, BLOCK>(src);
  if (precision == TWOS_PREC_MIXED) {
    TWOS_PICK(float)
  }
  TWOS_PICK(double)
#undef TWOS_PICK
}

// Walk kernel instantiations: block sizes 128, 256 and 512 threads.
static const void *select_wos(int precision, int mode, int src, int block, int grid64, int wide, int claim) {
  switch (block) {
    case 128:
      return select_wos_block<128>(precision, mode, src, grid64, wide, claim);
    case 256:
      return select_wos_block<256>(precision, mode, src, grid64, wide, claim);
    case 512:
      return select_wos_block<512>(precision, mode, src, grid64, wide, claim);
    default:
      return nullptr;
  }
}

static uint32_t wos_dyn_smem(int precision, int mode, const WosLaunch &L, int block) {
  const int entries = precision == TWOS_PREC_MIXED ? wos_stack_entries<float>() : wos_stack_entries<double>();
  const int cold = precision == TWOS_PREC_MIXED ? wos_cold_bytes<float>(mode == kModeGradient)
                                                : wos_cold_bytes<double>(mode == kModeGradient);
  const uint32_t stack = static_cast<uint32_t>((entries * sizeof(uint2) + cold) * block);
  return stack + (precision == TWOS_PREC_MIXED ? smem_plan<float>(L.n_jobs, L.n_geos, L.n_terms).bytes
                                               : smem_plan<double>(L.n_jobs, L.n_geos, L.n_terms).bytes);
}

// The mixed compliance walk kernel (centre source, 128 threads) with a
// record of every grid step's position and bound (L.trace): used by tests to
// check each bound against the FP64 distance.
cudaError_t launch_wos_traced(const WosLaunch &L, int grid, cudaStream_t s) {
  if (L.n_jobs == 0 || L.n_geos == 0 || !L.trace || !L.trace_count) return cudaErrorInvalidValue;
  const uint32_t dyn = wos_dyn_smem(TWOS_PREC_MIXED, TWOS_MODE_COMPLIANCE, L, kWosBlock);
  const void *fn = reinterpret_cast<const void *>(&wos_kernel<float, TWOS_MODE_COMPLIANCE, TWOS_SOURCE_CENTER,
                                                              kWosBlock, true>);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn));
  if (e != cudaSuccess) return e;
  WosLaunch copy = L;
  copy.lanes = 32;
  void *args[] = {&copy};
  return cudaLaunchKernel(fn, dim3(grid), dim3(kWosBlock), args, dyn, s);
}

cudaError_t launch_wos(int precision, int mode, int src, const WosLaunch &L, int grid, int block,
                       cudaStream_t s) {
  if (L.n_jobs == 0 || L.n_geos == 0) return cudaErrorInvalidValue;
  const uint32_t dyn = wos_dyn_smem(precision, mode, L, block);
  if (dyn > 200 * 1024) return cudaErrorInvalidValue;
  const void *fn = select_wos(precision, mode, src, block, L.grid64, L.wide, L.lane_walks > 1);
  if (!fn) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn));
  if (e != cudaSuccess) return e;
  // A launch with fewer walks than resident lanes spreads them over all warps:
  // a warp's divergent lanes take turns, so the fewer the better (256 FP64
  // walks: 1.88 ms with full warps, 1.57 with 16 lanes, 1.18 with 4, 0.76 with
  // one; 65,536: 4.8 ms full, 4.4 with 19; 98,304 mixed: 1.28 and 1.18).
  WosLaunch copy = L;
  const uint64_t warps = static_cast<uint64_t>(grid) * (block / 32);
  const uint64_t claims = (L.total_walks + lane_walks_of(L) - 1) / lane_walks_of(L);
  copy.lanes = static_cast<int>(std::min<uint64_t>(32, std::max<uint64_t>(1, (claims + warps - 1) / warps)));
  void *args[] = {&copy};
  return cudaLaunchKernel(fn, dim3(grid), dim3(block), args, dyn, s);
}

int wos_max_blocks_per_sm(int precision, int mode, int src, int block, const WosLaunch &L) {
  const uint32_t dyn = wos_dyn_smem(precision, mode, L, block);
  const void *fn = select_wos(precision, mode, src, block, L.grid64, L.wide, L.lane_walks > 1);
  if (!fn || dyn > 200 * 1024) return 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn)) != cudaSuccess)
    return 0;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, dyn) != cudaSuccess) return 0;
  return n;
}

// ================================================================ finalize
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename V, int MODE>
__global__ void __launch_bounds__(256) finalize_kernel(const FinalizeLaunch F) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t g = warp; g < F.total_sites; g += nwarps) {
    // Job of launch site g (jobs ordered by site_rank).
    uint32_t lo = 0, hi = F.n_jobs - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (F.jobs[mid].site_rank <= g)
        lo = mid;
      else
        hi = mid - 1;
    }
    const JobDesc &J = F.jobs[lo];
    const uint32_t s = g - J.site_rank;
    const uint64_t base = J.walk_begin + static_cast<uint64_t>(s) * J.walks;
    const V *U = static_cast<const V *>(F.u) + base;
    const V *P = static_cast<const V *>(F.p) + base;
    const uint32_t *S = F.steps + base;
    const uint32_t n = J.walks;
    const double nd = static_cast<double>(n);
    double a = 0.0, b = 0.0, c = 0.0;
    unsigned long long st = 0, caps = 0;
    for (uint32_t w = lane; w < n; w += 32) {
      const double x = static_cast<double>(U[w]);
      const uint32_t sw = S[w];
      st += sw & 0x7fffffffu;
      caps += sw >> 31;
      if (MODE == TWOS_MODE_PAIRED) {
        const double y = static_cast<double>(P[w]);
        a += x;
        b += y;
        c += x * y;
      } else {
        a += x;
        b += x * x;
      }
    }
    a = warp_sum(a);
    b = warp_sum(b);
    c = warp_sum(c);
    st = warp_sum_u64(st);
    caps = warp_sum_u64(caps);
    twos_site_result r;
    r.steps = st;
    r.caps = caps;
    // Leave-one-out values, their mean and spread (two more passes over the
    // samples, which are L2-resident at this point).
    double lsum = 0.0;
    for (uint32_t w = lane; w < n; w += 32) {
      const double x = static_cast<double>(U[w]);
      double leave;
      if (MODE == TWOS_MODE_COMPLIANCE) {
        const double ls = a - x, ls2 = b - x * x;
        leave = (ls * ls - ls2) / ((nd - 1.0) * (nd - 2.0));
      } else if (MODE == TWOS_MODE_PAIRED) {
        const double y = static_cast<double>(P[w]);
        leave = ((a - x) * (b - y) - (c - x * y)) / ((nd - 1.0) * (nd - 2.0));
      } else {
        leave = (a - x) / (nd - 1.0);
      }
      lsum += leave;
    }
    const double lmean = warp_sum(lsum) / nd;
    double spread = 0.0;
    for (uint32_t w = lane; w < n; w += 32) {
      const double x = static_cast<double>(U[w]);
      double leave;
      if (MODE == TWOS_MODE_COMPLIANCE) {
        const double ls = a - x, ls2 = b - x * x;
        leave = (ls * ls - ls2) / ((nd - 1.0) * (nd - 2.0));
      } else if (MODE == TWOS_MODE_PAIRED) {
        const double y = static_cast<double>(P[w]);
        leave = ((a - x) * (b - y) - (c - x * y)) / ((nd - 1.0) * (nd - 2.0));
      } else {
        leave = (a - x) / (nd - 1.0);
      }
      const double dv = leave - lmean;
      spread += dv * dv;
    }
    spread = warp_sum(spread);
    const double se = n >= 4 ? sqrt((nd - 1.0) / nd * spread) : CUDART_NAN;
    if (MODE == TWOS_MODE_COMPLIANCE) {
      r.u = a / nd;
      r.p = r.u;
      r.score = (a * a - b) / (nd * (nd - 1.0));
      r.same_index = b / nd;
    } else if (MODE == TWOS_MODE_PAIRED) {
      r.u = a / nd;
      r.p = b / nd;
      r.score = (a * b - c) / (nd * (nd - 1.0));
      r.same_index = c / nd;
    } else {
      r.u = a / nd;
      r.p = 0.0;
      r.score = a / nd;
      r.same_index = 0.0;
    }
    r.score_se = se;
    if (lane == 0) {
      F.out[J.site_begin + s] = r;
      if (F.totals) {
        atomicAdd(&F.totals[0], st);
        atomicAdd(&F.totals[1], caps);
      }
    }
  }
}

// Gradient mode: one warp per site (warp_sum: a fixed xor-tree order).  Pass 1: sums of u, p, grad u, grad p
// and grad u . grad p; pass 2: the leave-one-out cross statistics and their
// mean; pass 3: the jackknife variance.  FP64 throughout.
template <typename V> __global__ void __launch_bounds__(256) grad_finalize_kernel(const GradFinalizeLaunch F) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warp = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
  const V *u = static_cast<const V *>(F.u), *p = static_cast<const V *>(F.p), *g = static_cast<const V *>(F.grad);
  const uint32_t N = F.walks;
  const double n = static_cast<double>(N);
  for (uint64_t site = warp; site < F.n_sites; site += nwarps) {
    const uint64_t base = site * N;
    double su = 0, sp = 0, sgu[3] = {0, 0, 0}, sgp[3] = {0, 0, 0}, sdot = 0;
    unsigned long long steps = 0, caps = 0;
    for (uint32_t w = lane; w < N; w += 32) {
      const uint64_t i = base + w;
      su += static_cast<double>(u[i]);
      sp += static_cast<double>(p[i]);
      double d = 0;
      for (int k = 0; k < 3; ++k) {
        const double a = static_cast<double>(g[6 * i + k]), b = static_cast<double>(g[6 * i + 3 + k]);
        sgu[k] += a;
        sgp[k] += b;
        d += a * b;
      }
      sdot += d;
      const uint32_t st = F.steps[i];
      steps += st & 0x7fffffffu;
      caps += st >> 31;
    }
    su = warp_sum(su);
    sp = warp_sum(sp);
    for (int k = 0; k < 3; ++k) {
      sgu[k] = warp_sum(sgu[k]);
      sgp[k] = warp_sum(sgp[k]);
    }
    sdot = warp_sum(sdot);
    const double den = n * (n - 1.0);
    const double cross = (sgu[0] * sgp[0] + sgu[1] * sgp[1] + sgu[2] * sgp[2] - sdot) / den;
    // Leave-one-out: ((S_u - g_i).(S_p - h_i) - (S_dot - g_i.h_i)) / ((N-1)(N-2)).
    const double den1 = (n - 1.0) * (n - 2.0);
    double s1 = 0, s2 = 0;
    if (N > 2) {
      for (uint32_t w = lane; w < N; w += 32) {
        const uint64_t i = base + w;
        double a[3], b[3], d = 0;
        for (int k = 0; k < 3; ++k) {
          a[k] = static_cast<double>(g[6 * i + k]);
          b[k] = static_cast<double>(g[6 * i + 3 + k]);
          d += a[k] * b[k];
        }
        const double c = ((sgu[0] - a[0]) * (sgp[0] - b[0]) + (sgu[1] - a[1]) * (sgp[1] - b[1]) +
                          (sgu[2] - a[2]) * (sgp[2] - b[2]) - (sdot - d)) / den1;
        s1 += c;
      }
      s1 = warp_sum(s1);
      const double mean = s1 / n;
      for (uint32_t w = lane; w < N; w += 32) {
        const uint64_t i = base + w;
        double a[3], b[3], d = 0;
        for (int k = 0; k < 3; ++k) {
          a[k] = static_cast<double>(g[6 * i + k]);
          b[k] = static_cast<double>(g[6 * i + 3 + k]);
          d += a[k] * b[k];
        }
        const double c = ((sgu[0] - a[0]) * (sgp[0] - b[0]) + (sgu[1] - a[1]) * (sgp[1] - b[1]) +
                          (sgu[2] - a[2]) * (sgp[2] - b[2]) - (sdot - d)) / den1;
        s2 += (c - mean) * (c - mean);
      }
      s2 = warp_sum(s2);
    }
    // Standard errors of the means of u and p (two-pass sample variance).
    const double mu = su / n, mp = sp / n;
    double vu = 0, vp = 0;
    for (uint32_t w = lane; w < N; w += 32) {
      const double du = static_cast<double>(u[base + w]) - mu, dp = static_cast<double>(p[base + w]) - mp;
      vu += du * du;
      vp += dp * dp;
    }
    vu = warp_sum(vu);
    vp = warp_sum(vp);
    for (int o = 16; o > 0; o >>= 1) {
      steps += __shfl_xor_sync(0xffffffffu, steps, o);
      caps += __shfl_xor_sync(0xffffffffu, caps, o);
    }
    if (lane == 0) {
      twos_gradient_result r;
      r.u = su / n;
      r.p = sp / n;
      for (int k = 0; k < 3; ++k) {
        r.grad_u[k] = sgu[k] / n;
        r.grad_p[k] = sgp[k] / n;
      }
      r.cross = cross;
      r.cross_se = N > 2 ? sqrt((n - 1.0) / n * s2) : 0.0;
      r.steps = steps;
      r.caps = caps;
      r.u_se = N > 1 ? sqrt(vu / (n * (n - 1.0))) : 0.0;
      r.p_se = N > 1 ? sqrt(vp / (n * (n - 1.0))) : 0.0;
      F.out[site] = r;
      atomicAdd(&F.totals[0], steps);
      atomicAdd(&F.totals[1], caps);
    }
  }
}

cudaError_t launch_grad_finalize(int precision, const GradFinalizeLaunch &F, cudaStream_t s) {
  if (F.n_sites == 0) return cudaSuccess;
  const int grid = static_cast<int>(std::min<uint64_t>((static_cast<uint64_t>(F.n_sites) * 32 + 255) / 256,
                                                       148ull * 16));
  if (precision == TWOS_PREC_MIXED)
    grad_finalize_kernel<float><<<grid, 256, 0, s>>>(F);
  else
    grad_finalize_kernel<double><<<grid, 256, 0, s>>>(F);
  return cudaGetLastError();
}

cudaError_t launch_finalize(int precision, int mode, const FinalizeLaunch &F, cudaStream_t s) {
  if (F.total_sites == 0) return cudaSuccess;
  const int block = 256;
  const uint64_t warps = F.total_sites;
  int grid = static_cast<int>(std::min<uint64_t>((warps * 32 + block - 1) / block, 148ull * 16));
  FinalizeLaunch copy = F;
  void *args[] = {&copy};
  const void *fn;
  if (precision == TWOS_PREC_MIXED) {
    fn = mode == TWOS_MODE_COMPLIANCE ? reinterpret_cast<const void *>(&finalize_kernel<float, 0>)
         : mode == TWOS_MODE_PAIRED   ? reinterpret_cast<const void *>(&finalize_kernel<float, 1>)
                                      : reinterpret_cast<const void *>(&finalize_kernel<float, 2>);
  } else {
    fn = mode == TWOS_MODE_COMPLIANCE ? reinterpret_cast<const void *>(&finalize_kernel<double, 0>)
         : mode == TWOS_MODE_PAIRED   ? reinterpret_cast<const void *>(&finalize_kernel<double, 1>)
                                      : reinterpret_cast<const void *>(&finalize_kernel<double, 2>);
  }
  return cudaLaunchKernel(fn, dim3(grid), dim3(block), args, 0, s);
}

// ================================================================ L2 read probe
// Streams an L2-resident buffer with the walk kernel's load form (32-byte
// read-only vector loads, one per lane, consecutive lanes on consecutive
// sectors), `passes` times over.  The measured rate is the L2 read roof for a
// working set that fits the L2 (the distance grid and the BVH of one mesh).
__global__ void __launch_bounds__(256) l2_read_kernel(const float4 *__restrict__ buf, uint64_t n32, int passes,
                                                      uint32_t *sink) {
  float acc = 0.f;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (int p = 0; p < passes; ++p) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n32; i += stride) {
      float4 a, b;
      ldg32(buf + 2 * i, a, b);
      acc += (a.x + a.y + a.z + a.w) + (b.x + b.y + b.z + b.w);
    }
  }
  // The buffer holds zeros, so this store never happens; the compiler cannot
  // know that and keeps every load.
  if (acc != 0.f) sink[0] = __float_as_uint(acc);
}

cudaError_t launch_l2_read(const void *buf, uint64_t bytes, int passes, uint32_t *sink, int blocks, cudaStream_t s) {
  l2_read_kernel<<<blocks, 256, 0, s>>>(static_cast<const float4 *>(buf), bytes / 32, passes, sink);
  return cudaGetLastError();
}

// ================================================================ batched closest point
// The result of point i: distance (infinite when nothing is within the query
// radius) and, if wanted, the nearest point.
template <typename T>
__device__ __forceinline__ void closest_store(const GeoDesc &G, const Vec<T> &p, bool found, T best2, uint32_t best_tri,
                                              uint64_t i, double *dist, double *closest) {
  dist[i] = found ? static_cast<double>(sqrt(best2)) : CUDART_INF;
  if (!closest) return;
  double q[3] = {CUDART_NAN, CUDART_NAN, CUDART_NAN};
  if (found) {
    Vec<T> a, b, c;
    load_tri(geo_tris<T>(G), best_tri, a, b, c);
    const Vec<T> cp = tri_closest(p, a, b, c);
    const bool f32 = sizeof(T) == 4;
    q[0] = static_cast<double>(cp.x) + (f32 ? G.center[0] : 0.0);
    q[1] = static_cast<double>(cp.y) + (f32 ? G.center[1] : 0.0);
    q[2] = static_cast<double>(cp.z) + (f32 ? G.center[2] : 0.0);
  }
  for (int a = 0; a < 3; ++a) closest[3 * i + a] = q[a];
}

// A warp per point: a call with few points is as long as its longest query,
// and a lane alone waits for memory at every node (5,000 points, 81,920
// triangles, FP64: 1.69 ms with a lane each, 0.25 with a warp, of which 0.03
// settle ties).
template <typename T>
__global__ void __launch_bounds__(kWosBlock) closest_warp_kernel(const GeoDesc *geo, const double *pts, uint64_t n,
                                                                 double query_radius2, double *dist, double *closest,
                                                                 uint32_t *error) {
  __shared__ uint2 s_stack[kWarpEntries * (kWosBlock / 32)];
  __shared__ GeoDesc G;
  if (threadIdx.x == 0) G = *geo;
  __syncthreads();
  uint32_t err = 0;
  uint2 *stack = s_stack + kWarpEntries * (threadIdx.x >> 5);
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (kWosBlock / 32);
  for (uint64_t i = blockIdx.x * (kWosBlock / 32) + (threadIdx.x >> 5); i < n; i += warps) {
    const Vec<T> p = to_frame<T>(pts + 3 * i, G);
    T best2 = static_cast<T>(query_radius2);
    uint32_t best_tri = 0;
    const bool found = warp_nearest(G, p, best2, best_tri, stack, err, closest != nullptr);
    if ((threadIdx.x & 31u) == 0) closest_store(G, p, found, best2, best_tri, i, dist, closest);
  }
  if (err) atomicOr(error, err);
}

// A point per lane, for many points: as the walk kernel, a lane runs units of
// its search, one set of loads per unit, and takes the next point from the
// queue when it ends, so a warp does not wait for its longest query (call of
// 122,591 points, 81,920 triangles, FP64: 3.1 ms with a fixed point per
// thread, 1.96 with the queue).
template <typename T>
__global__ void __launch_bounds__(kWosBlock) closest_kernel(const GeoDesc *geo, const double *pts, uint64_t n,
                                                            double query_radius2, double *dist, double *closest,
                                                            unsigned long long *counter, uint32_t *error) {
  constexpr int kLaneStack = 8;
  __shared__ uint2 s_stack[(kLaneStack + kCand) * kWosBlock];
  __shared__ GeoDesc G;
  if (threadIdx.x == 0) G = *geo;
  __syncthreads();
  uint2 *stack = s_stack + threadIdx.x, *cand = stack + kLaneStack * kWosBlock;
  uint2 deep[kStack + 1 - kLaneStack];
  const unsigned lane = threadIdx.x & 31u, full = 0xffffffffu;
  uint32_t err = 0;
  uint64_t i = 0;
  Vec<T> p{T(0), T(0), T(0)};
  Cull c{{0.f, 0.f, 0.f}, 0.f, 0.f, 0};  // FP32: p and the threshold best2
  T best2 = T(0);
  uint32_t best_tri = 0, tri_cur = 0, tri_end = 0, iter = 0, ties = 0;
  int node = 0, sp = 0;
  bool have = false, found = false, exhausted = false;  // exhausted is warp-uniform
  float mark = 0.f;
  int phase = kIdle;
  for (;;) {
    if (phase == kStep) {
      if constexpr (sizeof(T) == 8) found |= cull_flush<true>(G, p, c, best2, best_tri, cand, kWosBlock, &ties, &mark);
      if (have || tri_cur < tri_end || sp > 0) {
        phase = kTraverse;  // the candidate list was full: the search goes on
      } else {
        if (!found && best2 < static_cast<T>(query_radius2)) {
          // None below the grid's bound (grid_start): without it, from the root.
          best2 = static_cast<T>(query_radius2);
          if constexpr (sizeof(T) == 8) c.limit = cull_limit(best2, c.margin);
          node = 0;
          have = true;
          iter = 0;
          phase = kTraverse;
        } else {
          if constexpr (sizeof(T) == 8) {
            if (found && closest && (ties & kTieOpen)) best_tri = first_of_tied(G, p, best2, best_tri);
          }
          closest_store(G, p, found, best2, best_tri, i, dist, closest);
          phase = kIdle;
        }
      }
    }
    const unsigned idle = __ballot_sync(full, phase == kIdle);
    if (!exhausted && idle != 0u) {
      unsigned long long base = 0;
      const int leader = __ffs(idle) - 1;
      if (static_cast<int>(lane) == leader) base = atomicAdd(counter, static_cast<unsigned long long>(__popc(idle)));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= n) exhausted = true;
      const uint64_t next = base + __popc(idle & ((1u << lane) - 1u));
      if (phase == kIdle && next < n) {
        i = next;
        p = to_frame<T>(pts + 3 * i, G);
        best2 = static_cast<T>(query_radius2);
        found = false;
        sp = 0;
        tri_cur = tri_end = iter = ties = 0;
        bool search = true;
        if constexpr (sizeof(T) == 4) {
          c.p = p;
        } else {
          if (!cull_begin(G, p, best2, c)) {
            found = nearest_plain(G, p, best2, best_tri, err);
            have = search = false;
            phase = kStep;
          }
        }
        if (search) {
          float upper;
          if constexpr (sizeof(T) == 4) {
            grid_start(G, c.p, sqrtf(best2), upper, node);
            best2 = fminf(best2, upper * upper);
          } else {
            grid_start(G, c.p, sqrtf(c.limit), upper, node);
            const float reach = __fadd_ru(upper, c.margin), reach2 = __fmul_ru(reach, reach);
            c.limit = fminf(c.limit, reach2);
            best2 = fmin(best2, static_cast<double>(reach2));
          }
          have = true;
          phase = kTraverse;
        }
      }
    }
    if (__ballot_sync(full, phase != kIdle) == 0u) {
      if (exhausted) break;
      continue;
    }
    if (phase != kTraverse) continue;
#pragma unroll 1
    for (int unit = 0; unit < 8; ++unit) {
      const float limit = [&]() -> float {
        if constexpr (sizeof(T) == 4)
          return best2;
        else
          return c.limit;
      }();
      if (tri_cur >= tri_end) {
        while (!have && sp > 0) {
          --sp;
          const uint2 e = sp < kLaneStack ? stack[sp * kWosBlock] : deep[sp - kLaneStack];
          if (__uint_as_float(e.y) < limit) {
            node = static_cast<int>(e.x);
            have = true;
          }
        }
        if (!have) {
          phase = kStep;
          break;
        }
        if (node < 0) {
          const uint32_t enc = ~static_cast<uint32_t>(node);
          tri_cur = enc >> 3;
          tri_end = tri_cur + (enc & 7u);
          have = false;
        }
      }
      if (++iter > G.max_iter || sp > kStack) {
        err |= sp > kStack ? TWOS_DEVERR_STACK : TWOS_DEVERR_ITER;
        best2 = static_cast<T>(CUDART_INF_F);  // no second search
        have = false;
        sp = 0;
        tri_cur = tri_end;
        phase = kStep;
        break;
      }
      const bool on_tri = tri_cur < tri_end;
      const char *at = on_tri ? reinterpret_cast<const char *>(G.tris_f + tri_cur)
                              : reinterpret_cast<const char *>(G.nodes_f + node);
      float4 r0, r1, r2, r3, r4{}, r5{};
      ldg32(at, r0, r1);
      ldg32(at + 32, r2, r3);
      ldg32_if(!on_tri, at + 64, r4, r5);
      if (on_tri) {
        if constexpr (sizeof(T) == 4) {
          if (plane_gap2(r0, r1, c.p) < best2) {
            const float d2 = tri_dist2(c.p, Vec<float>{r1.x, r1.y, r1.z}, Vec<float>{r2.x, r2.y, r2.z},
                                       Vec<float>{r3.x, r3.y, r3.z});
            if (d2 < best2) {
              best2 = d2;
              best_tri = tri_cur;
              found = true;
            }
          }
        } else {
          uint32_t full_tests = 0;
          if (cull_tri(tri_cur, r0, r1, r2, r3, c, cand, kWosBlock, full_tests)) {
            phase = kStep;  // a full candidate list is tested first; the triangle comes again
            break;
          }
        }
        ++tri_cur;
      } else {
        float dl, dr;
        int cl, cr;
        node_bounds(r0, r1, r2, r3, r4, r5, c.p, dl, dr, cl, cr);
        const bool vl = dl < limit, vr = dr < limit, swap = dr < dl;
        if (vl && vr) {
          const uint2 e = make_uint2(static_cast<uint32_t>(swap ? cl : cr), __float_as_uint(swap ? dl : dr));
          if (sp < kLaneStack)
            stack[sp * kWosBlock] = e;
          else
            deep[sp - kLaneStack] = e;
          ++sp;
        }
        have = vl || vr;
        node = vl && !(vr && swap) ? cl : cr;
      }
    }
  }
  if (err) atomicOr(error, err);
}

__global__ void ball_green_kernel(const double *__restrict__ cases, uint32_t n, double *__restrict__ out,
                                  uint32_t *error) {
  uint32_t err = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    bool negative = false;
    out[i] = exact_bump_green(cases[4ull * i], cases[4ull * i + 1], cases[4ull * i + 2], cases[4ull * i + 3],
                              negative);
    if (negative) err |= TWOS_DEVERR_SOURCE;
  }
  if (err) atomicOr(error, err);
}

cudaError_t launch_ball_green(const double *cases, uint32_t n, double *out, uint32_t *error, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int grid = static_cast<int>(std::min<uint32_t>((n + 127) / 128, 148u * 8));
  ball_green_kernel<<<grid, 128, 0, s>>>(cases, n, out, error);
  return cudaGetLastError();
}

// Points up to which each gets a warp.  The warp's search costs more
// instructions in all, so it wins where a call is as long as its longest query
// (calls, ms, lane / warp, FP64, 327,680 triangles: 3,000 points of the solid
// 2.5 / 0.34, 30,000 2.8 / 1.4, 60,000 3.2 / 2.7, 122,591 3.9 / 5.2; near the
// surface 10,000 0.15 / 0.16, 30,000 0.24 / 0.33, 122,591 0.68 / 1.28).  The
// line lies between the two: calls in the solid would gain by a warp up to
// some 80,000 points, those near the surface lose from 10,000 on.
constexpr uint64_t kWarpPoints = 16384;

cudaError_t launch_closest(int precision, const GeoDesc *geo_dev, const double *pts, uint64_t n,
                           double query_radius2, double *dist, double *closest, unsigned long long *counter,
                           uint32_t *error, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int block = kWosBlock;
  if (n <= kWarpPoints) {
    const int grid = static_cast<int>((n + block / 32 - 1) / (block / 32));
    if (precision == TWOS_PREC_MIXED)
      closest_warp_kernel<float><<<grid, block, 0, s>>>(geo_dev, pts, n, query_radius2, dist, closest, error);
    else
      closest_warp_kernel<double><<<grid, block, 0, s>>>(geo_dev, pts, n, query_radius2, dist, closest, error);
    return cudaGetLastError();
  }
  const cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 148ull * 8));
  if (precision == TWOS_PREC_MIXED)
    closest_kernel<float><<<grid, block, 0, s>>>(geo_dev, pts, n, query_radius2, dist, closest, counter, error);
  else
    closest_kernel<double><<<grid, block, 0, s>>>(geo_dev, pts, n, query_radius2, dist, closest, counter, error);
  return cudaGetLastError();
}

// ================================================================ distance-bound grid
// One thread per grid vertex: its FP32 closest-point distance, less `margin`,
// rounded down to a multiple of grid_q and saturated at 65535 multiples.  A
// vertex whose query fails keeps 0 (a bound no step uses).
__global__ void __launch_bounds__(kWosBlock) grid_build_kernel(const GeoDesc *geo, double margin, uint16_t *out,
                                                               uint32_t *error) {
  __shared__ uint2 s_stack[kStack * kWosBlock];
  __shared__ GeoDesc G;
  if (threadIdx.x == 0) G = *geo;
  __syncthreads();
  uint32_t err = 0;
  uint2 *stack = s_stack + threadIdx.x;
  const uint64_t n = static_cast<uint64_t>(G.grid_n[0]) * G.grid_n[1] * G.grid_n[2];
  for (uint64_t v = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; v < n;
       v += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t gk = static_cast<uint32_t>(v % G.grid_n[2]);
    const uint64_t ij = v / G.grid_n[2];
    const uint32_t gj = static_cast<uint32_t>(ij % G.grid_n[1]), gi = static_cast<uint32_t>(ij / G.grid_n[1]);
    const Vec<float> p = grid_vertex(G, gi, gj, gk);
    float best2 = CUDART_INF_F;
    uint32_t tri = 0;
    uint16_t q = 0;
    if (nearest<float>(geo_nodes<float>(G), geo_tris<float>(G), G.max_iter, p, best2, tri, stack, kWosBlock, err)) {
      const double m = floor((static_cast<double>(sqrtf(best2)) - margin) / static_cast<double>(G.grid_q));
      q = m <= 0.0 ? 0 : m >= 65535.0 ? 65535 : static_cast<uint16_t>(m);
    }
    out[v] = q;
  }
  if (err) atomicOr(error, err);
}

// The grid's lower bound at each point (original coordinates), NaN where the
// point lies outside the grid or the geometry has none.
__global__ void __launch_bounds__(256) grid_bound_kernel(const GeoDesc *geo, const double *pts, uint64_t n,
                                                         double *out) {
  const GeoDesc G = *geo;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    float b = 0.f;
    out[i] = G.grid && grid_bound(G, to_frame<float>(pts + 3 * i, G), b) ? static_cast<double>(b) : CUDART_NAN;
  }
}

cudaError_t launch_grid_bound(const GeoDesc *geo_dev, const double *pts, uint64_t n, double *out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int grid = static_cast<int>(std::min<uint64_t>((n + 255) / 256, 148ull * 16));
  grid_bound_kernel<<<grid, 256, 0, s>>>(geo_dev, pts, n, out);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) grid_pack_kernel(const uint16_t *__restrict__ v, uint32_t n0, uint32_t n1,
                                                         uint32_t n2, const int32_t *__restrict__ table,
                                                         uint32_t shift, uint32_t e1, uint32_t e2,
                                                         uint4 *__restrict__ cells) {
  const uint64_t m1 = n1 - 1, m2 = n2 - 1, count = static_cast<uint64_t>(n0 - 1) * m1 * m2;
  for (uint64_t cell = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; cell < count;
       cell += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t k = static_cast<uint32_t>(cell % m2);
    const uint64_t ij = cell / m2;
    const uint32_t j = static_cast<uint32_t>(ij % m1), i = static_cast<uint32_t>(ij / m1);
    uint32_t d[8], base = 0xffffu;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      d[c] = v[(static_cast<uint64_t>(i + (c >> 2)) * n1 + (j + ((c >> 1) & 1))) * n2 + (k + (c & 1))];
      base = min(base, d[c]);
    }
    // Byte offsets above the base; 255 for a saturated corner or one too far
    // above the base (the reader then uses the base: a lower bound still).
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t off = d[c] == 0xffffu || d[c] - base > 254u ? 0xffu : d[c] - base;
      if (c < 4)
        lo |= off << (8 * c);
      else
        hi |= off << (8 * (c - 4));
    }
    const int32_t entry = table ? table[(static_cast<uint64_t>(i >> shift) * e1 + (j >> shift)) * e2 + (k >> shift)]
                                : -1;
    cells[cell] = make_uint4(lo, hi, base, static_cast<uint32_t>(entry));
  }
}

cudaError_t launch_grid_pack(const uint16_t *vertices, const uint32_t n[3], const int32_t *table, uint32_t shift,
                             const uint32_t entry_n[3], uint4 *cells, cudaStream_t s) {
  if (n[0] < 2 || n[1] < 2 || n[2] < 2) return cudaErrorInvalidValue;
  if (table && (((n[0] - 2) >> shift) >= entry_n[0] || ((n[1] - 2) >> shift) >= entry_n[1] ||
                ((n[2] - 2) >> shift) >= entry_n[2]))
    return cudaErrorInvalidValue;
  const uint64_t count = static_cast<uint64_t>(n[0] - 1) * (n[1] - 1) * (n[2] - 1);
  const int grid = static_cast<int>(std::min<uint64_t>((count + 255) / 256, 148ull * 64));
  grid_pack_kernel<<<grid, 256, 0, s>>>(vertices, n[0], n[1], n[2], table, shift, table ? entry_n[1] : 0,
                                        table ? entry_n[2] : 0, cells);
  return cudaGetLastError();
}

// Candidate lists (GeoDesc::lists).  A cell whose centre lies within
// kListReach spacings of the surface -- beyond, a mixed-form step takes its
// radius from the grid -- lists every triangle that can be nearest, or within
// 8 delta of it, at a point of the cell: with rho half the cell's diagonal
// (grown by the 0.01 h of the point-to-cell rounding), those within
// d(centre) + 2 rho of the centre.  At most kListMost triangles; denser cells
// keep their entry node.
constexpr int kListMost = 30;

// The cells near the surface, in `cells` (cells[0 .. *count)).
__global__ void __launch_bounds__(256) list_cells_kernel(const GeoDesc *geo, uint32_t *cells, uint32_t capacity,
                                                         uint32_t *count) {
  const GeoDesc G = *geo;
  const uint64_t m1 = G.grid_n[1] - 1, m2 = G.grid_n[2] - 1, n = (G.grid_n[0] - 1) * m1 * m2;
  const float most = (kListReach + 0.8661f) * 128.f + 1.f;  // corner values of such a cell are below
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t threads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t base = blockIdx.x * static_cast<uint64_t>(blockDim.x); base < n; base += threads) {
    const uint64_t cell = base + threadIdx.x;
    const bool take = cell < n && static_cast<float>(G.grid[cell].z & 0xffffu) <= most;
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (m == 0u) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(count, static_cast<uint32_t>(__popc(m)));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (take && cells && at < capacity) cells[at] = static_cast<uint32_t>(cell);
  }
}

// FILL 0: adds the entries of all lists to *cursor; 1: writes the lists at
// positions taken from *cursor, each list's cell in its first entry and its
// position in place of the cell in `cells` (kNoList: none).  The records are
// pointed at the lists by list_point_kernel: this kernel's searches read them.
constexpr uint32_t kNoList = 0xffffffffu;
template <int FILL>
__global__ void __launch_bounds__(kWosBlock) list_build_kernel(const GeoDesc *geo, uint32_t *cells, uint32_t n,
                                                               uint2 *lists, uint32_t *cursor, uint32_t *error) {
  __shared__ uint2 s_stack[near_entries<double>() * kWosBlock];
  const GeoDesc G = *geo;
  const uint64_t m1 = G.grid_n[1] - 1, m2 = G.grid_n[2] - 1;
  uint32_t err = 0;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const uint64_t cell = cells[t];
    if (FILL) cells[t] = kNoList;
    const float h = G.grid_h;
    const Vec<float> c{__fmaf_rn(static_cast<float>(cell / (m1 * m2)) + 0.5f, h, G.grid_lo[0]),
                       __fmaf_rn(static_cast<float>(cell / m2 % m1) + 0.5f, h, G.grid_lo[1]),
                       __fmaf_rn(static_cast<float>(cell % m2) + 0.5f, h, G.grid_lo[2])};
    // The centre's FP64 distance, and lower bounds for the triangles that hold
    // however degenerate they are.
    double best2 = CUDART_INF;
    uint32_t tri = 0;
    const Vec<double> c64{static_cast<double>(c.x) + G.center[0], static_cast<double>(c.y) + G.center[1],
                          static_cast<double>(c.z) + G.center[2]};
    if (!nearest_geo(G, c64, best2, tri, s_stack + threadIdx.x, kWosBlock, err)) continue;
    const float d = __double2float_ru(sqrt(best2));
    if (!(d <= kListReach * h)) continue;
    const float radius = d + 1.7668f * h + 8.f * G.delta;  // 2 rho = sqrt(3) * 1.02 h
    const float limit = radius * radius;
    uint32_t id[kListMost];
    float dist[kListMost];
    int held = 0;
    uint2 stack[kStack];
    int sp = 0, node = 0;
    uint32_t iter = 0;
    bool fits = true;
    for (bool have = true; have && fits;) {
      if (++iter > G.max_iter) {
        fits = false;
        break;
      }
      if (node < 0) {
        const uint32_t enc = ~static_cast<uint32_t>(node);
        for (uint32_t i = enc >> 3, e = (enc >> 3) + (enc & 7u); i < e && fits; ++i) {
          if (!(tri_plane_gap2(G.tris_f, i, c) < limit)) continue;
          Vec<float> ta, tb, tc;
          load_tri(G.tris_f, i, ta, tb, tc);
          const Vec<float> ap = sub(c, ta), bp = sub(c, tb), cp = sub(c, tc);
          const Vec<float> w = tri_point(ap, bp, cp, sub(tb, ta), sub(tc, ta));
          const float d2 = support2(w, ap, bp, cp, dot3(w, w));
          if (!(d2 < limit)) continue;
          if (held == kListMost) {
            fits = false;
          } else if (FILL) {
            const float dd = sqrtf(d2);
            int k = held;
            for (; k > 0 && (dist[k - 1] > dd || (dist[k - 1] == dd && id[k - 1] > i)); --k) {
              dist[k] = dist[k - 1];
              id[k] = id[k - 1];
            }
            dist[k] = dd;
            id[k] = i;
          }
          ++held;
        }
      } else {
        float dl, dr;
        int cl, cr;
        node_dist2(G.nodes_f, node, c, dl, dr, cl, cr);
        if (dl < limit || dr < limit) {
          if (dl < limit && dr < limit) stack[sp++] = make_uint2(static_cast<uint32_t>(cr), 0u);
          node = dl < limit ? cl : cr;
          continue;
        }
      }
      have = sp > 0;
      if (have) node = static_cast<int>(stack[--sp].x);
    }
    if (!fits) continue;
    // Header (entry node), the triangles, a terminator.
    const uint32_t at = atomicAdd(cursor, static_cast<uint32_t>(held + 2));
    if (FILL) {
      uint2 *out = lists + at;
      out[0] = make_uint2(G.grid[cell].w, static_cast<uint32_t>(cell));
      for (int k = 0; k < held; ++k) out[1 + k] = make_uint2(id[k], __float_as_uint(dist[k]));
      out[1 + held] = make_uint2(0u, 0x7f800000u);
      cells[t] = at;
    }
  }
  if (err) atomicOr(error, err);
}

// Points the records of the cells with lists (positions in `at`) at them and
// counts them in *listed.
__global__ void __launch_bounds__(256) list_point_kernel(const uint32_t *at, uint32_t n, uint2 *lists, uint4 *grid,
                                                         uint32_t *listed) {
  uint32_t count = 0;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    if (at[t] == kNoList) continue;
    uint2 *head = lists + at[t];
    grid[head->y].w = 0x80000000u | at[t];
    head->y = 0u;
    ++count;
  }
  if (count) atomicAdd(listed, count);
}

cudaError_t launch_list_cells(const GeoDesc *geo_dev, uint32_t *cells, uint32_t capacity, uint32_t *count,
                              cudaStream_t s) {
  list_cells_kernel<<<148 * 8, 256, 0, s>>>(geo_dev, cells, capacity, count);
  return cudaGetLastError();
}

cudaError_t launch_list_build(const GeoDesc *geo_dev, uint32_t *cells, uint32_t n, uint4 *grid, uint2 *lists,
                              uint32_t *cursor, uint32_t *listed, uint32_t *error, cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<uint32_t>((n + kWosBlock - 1) / kWosBlock, 148u * 32));
  if (!lists) {
    list_build_kernel<0><<<blocks, kWosBlock, 0, s>>>(geo_dev, cells, n, nullptr, cursor, error);
    return cudaGetLastError();
  }
  list_build_kernel<1><<<blocks, kWosBlock, 0, s>>>(geo_dev, cells, n, lists, cursor, error);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  list_point_kernel<<<static_cast<int>(std::min<uint32_t>((n + 255) / 256, 148u * 8)), 256, 0, s>>>(cells, n, lists,
                                                                                                 grid, listed);
  return cudaGetLastError();
}

cudaError_t launch_grid_build(const GeoDesc *geo_dev, uint64_t n, double margin, uint16_t *out, uint32_t *error,
                              cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int block = kWosBlock;
  const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 148ull * 32));
  grid_build_kernel<<<grid, block, 0, s>>>(geo_dev, margin, out, error);
  return cudaGetLastError();
}

// ================================================================ top-k
// Keys compare by (value desc, index asc); NaN sorts last.
struct KeyIdx {
  double v;
  uint32_t i;
};
__device__ __forceinline__ bool before(const KeyIdx &a, const KeyIdx &b) {
  const bool an = isnan(a.v), bn = isnan(b.v);
  if (an != bn) return bn;
  if (a.v != b.v) return a.v > b.v;
  return a.i < b.i;
}

constexpr int kTopkTile = 2048;

// Sorts one tile of kTopkTile keys in shared memory (bitonic) and writes its
// first k entries.
__global__ void __launch_bounds__(1024) topk_tile_kernel(const double *keys, uint32_t n, uint32_t k,
                                                         KeyIdx *partial) {
  __shared__ double sv[kTopkTile];
  __shared__ uint32_t si[kTopkTile];
  const uint32_t base = blockIdx.x * kTopkTile;
  for (uint32_t t = threadIdx.x; t < kTopkTile; t += blockDim.x) {
    const uint32_t g = base + t;
    sv[t] = g < n ? keys[g] : -CUDART_INF;
    si[t] = g < n ? g : 0xffffffffu;
  }
  __syncthreads();
  for (uint32_t size = 2; size <= kTopkTile; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t t = threadIdx.x; t < kTopkTile / 2; t += blockDim.x) {
        const uint32_t pos = 2 * t - (t & (stride - 1));
        const uint32_t a = pos, b = pos + stride;
        const bool up = ((pos & size) == 0);
        const KeyIdx ka{sv[a], si[a]}, kb{sv[b], si[b]};
        const bool swap = up ? before(kb, ka) : before(ka, kb);
        if (swap) {
          sv[a] = kb.v;
          si[a] = kb.i;
          sv[b] = ka.v;
          si[b] = ka.i;
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t t = threadIdx.x; t < k; t += blockDim.x) partial[blockIdx.x * k + t] = {sv[t], si[t]};
}

// Merges the per-tile candidates by repeated selection of the best remaining
// (k <= 1024, candidates <= a few hundred thousand).
__global__ void __launch_bounds__(1024) topk_merge_kernel(const KeyIdx *partial, uint32_t m, uint32_t k,
                                                          uint32_t *index) {
  __shared__ KeyIdx red[32];
  __shared__ KeyIdx last;
  if (threadIdx.x == 0) last = {CUDART_INF, 0u};
  __syncthreads();
  for (uint32_t r = 0; r < k; ++r) {
    KeyIdx best{-CUDART_INF, 0xffffffffu};
    bool have = false;
    for (uint32_t t = threadIdx.x; t < m; t += blockDim.x) {
      const KeyIdx c = partial[t];
      if (c.i == 0xffffffffu) continue;
      if (r > 0 && !before(last, c)) continue;  // already taken
      if (!have || before(c, best)) {
        best = c;
        have = true;
      }
    }
    // Block reduction.
    for (int o = 16; o > 0; o >>= 1) {
      KeyIdx other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      if (other.i != 0xffffffffu && (best.i == 0xffffffffu || before(other, best))) best = other;
    }
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x < 32) {
      KeyIdx b2 = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : KeyIdx{-CUDART_INF, 0xffffffffu};
      for (int o = 16; o > 0; o >>= 1) {
        KeyIdx other{__shfl_xor_sync(0xffffffffu, b2.v, o), __shfl_xor_sync(0xffffffffu, b2.i, o)};
        if (other.i != 0xffffffffu && (b2.i == 0xffffffffu || before(other, b2))) b2 = other;
      }
      if (threadIdx.x == 0) {
        index[r] = b2.i;
        last = b2;
      }
    }
    __syncthreads();
  }
}

size_t topk_scratch_bytes(uint32_t n, uint32_t k) {
  const uint32_t tiles = (n + kTopkTile - 1) / kTopkTile;
  return static_cast<size_t>(tiles) * k * sizeof(KeyIdx);
}

cudaError_t launch_topk(const double *keys, uint32_t n, uint32_t k, uint32_t *index, void *scratch,
                        size_t scratch_bytes, cudaStream_t s) {
  if (n == 0 || k == 0) return cudaSuccess;
  if (k > 1024 || k > static_cast<uint32_t>(kTopkTile)) return cudaErrorInvalidValue;
  if (scratch_bytes < topk_scratch_bytes(n, k)) return cudaErrorInvalidValue;
  const uint32_t tiles = (n + kTopkTile - 1) / kTopkTile;
  KeyIdx *partial = static_cast<KeyIdx *>(scratch);
  topk_tile_kernel<<<tiles, 1024, 0, s>>>(keys, n, k, partial);
  topk_merge_kernel<<<1, 1024, 0, s>>>(partial, tiles * k, k, index);
  return cudaGetLastError();
}

}  // namespace twos

// Differential WoS kernels (use nearest_geo and cull_begin above).
#include "diffwos.cuh"

// Certified validation kernels (use the stream, direction, warp_nearest and warp_search above).
#include "validate.cuh"

// Array-RQMC / matched MC lockstep walks (use nearest_geo, warp_nearest, the stream and warp sums above).
#include "rqmc.cuh"

#include "wavefront.cuh"
