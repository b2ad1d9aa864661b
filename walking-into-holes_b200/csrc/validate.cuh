// Certified fresh-sample validation on the device (run_minimum_benefit and
// cert_walk, benchmarks/compiled_bunny/src/minimum_benefit.hpp:13-188).
//
// Every quantity the certificate relies on is a rigorous bound computed the
// way the reference computes it: round to nearest, then step one ulp toward
// the safe side (nextafter), in FP64 without contraction (the library is
// built with -fmad=false).  The mesh distance is the distance to the union
// of the triangles' bounding boxes -- the minimum over triangles of a
// rounded-down box distance, which does not depend on traversal order, so it
// equals the reference's CertDistanceTree value bit for bit.  The FP64 BVH's
// node boxes (padded outward at build) contain those triangle boxes, so
// their rounded-down distances are lower bounds that prune exactly.
//
// cert_walk_kernel runs the walks as the walk kernel does: a state machine per
// lane, units of traversal work, a work queue.  Its search prunes in FP32
// (boxes only -- the slabs bound distances to triangles, not to their boxes)
// with the margin of the FP64 closest-point queries, and only the triangles
// whose FP32 box distance is within two margins of the smallest get the
// rounded-down FP64 box distance.  Geometries FP32 cannot hold run
// validate_kernel, one thread per walk on the FP64 nodes.  Every loop is
// bounded by the session's iteration limit or max_steps.
//
// Included at the end of kernels.cu (one translation unit with the random
// stream, direction and closest-point helpers).
#pragma once

namespace twos {

namespace {

__device__ __forceinline__ double cv_dn(double x) { return nextafter(x, -CUDART_INF); }
__device__ __forceinline__ double cv_up(double x) { return nextafter(x, CUDART_INF); }
__device__ __forceinline__ double cv_pdn(double x) { return fmax(0.0, cv_dn(x)); }

__device__ __forceinline__ double cv_box_lower(double lx, double ly, double lz, double hx, double hy, double hz,
                                               double x, double y, double z) {
  const double lo[3] = {lx, ly, lz}, hi[3] = {hx, hy, hz}, p[3] = {x, y, z};
  double sum = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double g = fmax(fmax(0.0, cv_dn(lo[a] - p[a])), cv_dn(p[a] - hi[a]));
    sum = cv_pdn(sum + cv_pdn(g * g));
  }
  return cv_pdn(sqrt(sum));
}

// point_distance_bound: rounded up (upper) or down.
__device__ __forceinline__ double cv_point_distance(const double *a, const double *b, bool upper) {
  double sum = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double d = fabs(a[k] - b[k]);
    d = upper ? cv_up(d) : cv_pdn(d);
    const double q = upper ? cv_up(d * d) : cv_pdn(d * d);
    sum = upper ? cv_up(sum + q) : cv_pdn(sum + q);
  }
  return upper ? cv_up(sqrt(sum)) : cv_pdn(sqrt(sum));
}

// Minimum over triangles of the rounded-down distance to the triangle's box.
__device__ double cv_mesh_distance(const GeoDesc &G, const double *p, uint32_t &err) {
  double best = CUDART_INF;
  int32_t stack[64];
  int sp = 0;
  stack[sp++] = 0;
  uint32_t iter = 0;
  while (sp > 0) {
    if (++iter > G.max_iter) {
      err |= TWOS_DEVERR_ITER;
      return 0.0;  // fail closed: a zero distance ends the walk
    }
    const int32_t code = stack[--sp];
    if (code < 0) {
      const uint32_t enc = ~static_cast<uint32_t>(code);
      for (uint32_t i = enc >> 3, e = (enc >> 3) + (enc & 7u); i < e; ++i) {
        Vec<double> a, b, c;
        load_tri(G.tris_d, i, a, b, c);
        const double v = cv_box_lower(fmin(fmin(a.x, b.x), c.x), fmin(fmin(a.y, b.y), c.y), fmin(fmin(a.z, b.z), c.z),
                                      fmax(fmax(a.x, b.x), c.x), fmax(fmax(a.y, b.y), c.y), fmax(fmax(a.z, b.z), c.z),
                                      p[0], p[1], p[2]);
        best = fmin(best, v);
      }
      continue;
    }
    const NodeD &n = G.nodes_d[code];
    const double2 xl = __ldg(&n.xlo), xh = __ldg(&n.xhi), yl = __ldg(&n.ylo), yh = __ldg(&n.yhi);
    const double2 zl = __ldg(&n.zlo), zh = __ldg(&n.zhi);
    const int4 ch = __ldg(&n.child);
    const double dl = cv_box_lower(xl.x, yl.x, zl.x, xh.x, yh.x, zh.x, p[0], p[1], p[2]);
    const double dr = cv_box_lower(xl.y, yl.y, zl.y, xh.y, yh.y, zh.y, p[0], p[1], p[2]);
    // Nearer child on top of the stack; a child whose bound is >= best
    // cannot hold a smaller triangle bound.
    const bool left_first = dl < dr;
    const double d_far = left_first ? dr : dl, d_near = left_first ? dl : dr;
    const int32_t c_far = left_first ? ch.y : ch.x, c_near = left_first ? ch.x : ch.y;
    if (d_far < best) {
      if (sp >= 64) {
        err |= TWOS_DEVERR_STACK;
        return 0.0;
      }
      stack[sp++] = c_far;
    }
    if (d_near < best) {
      if (sp >= 64) {
        err |= TWOS_DEVERR_STACK;
        return 0.0;
      }
      stack[sp++] = c_near;
    }
  }
  return best;
}

__device__ double cv_domain_distance(const ValidateLaunch &V, const GeoDesc &G, const double *p, uint32_t &err) {
  double d = cv_mesh_distance(G, p, err);
  for (uint32_t i = 0; i < V.n_cav; ++i) d = fmin(d, cv_dn(cv_point_distance(p, V.cavities + 3 * i, false) - V.cavity_radius));
  return fmax(0.0, d);
}

// (1 - t/1024)^1024 <= exp(-t), every step rounded down.
__device__ double cv_exp_lower(double t_upper) {
  double a = fmax(0.0, cv_dn(1.0 - cv_up(t_upper / 1024.0)));
  for (int i = 0; i < 10; ++i) a = cv_pdn(a * a);
  return a;
}

// Rounded-down source: a leading constant, then linear and Gaussian terms
// in order (cert_source_lower's affine and housing sequences).
__device__ double cv_source_lower(const ValidateLaunch &V, const double *p) {
  uint32_t i = 0;
  double value = 0.0;
  if (V.n_terms > 0 && V.terms[0].kind == TWOS_TERM_CONST) value = V.terms[i++].amp;
  for (; i < V.n_terms; ++i) {
    const TermDev &t = V.terms[i];
    if (t.kind == TWOS_TERM_LINEAR) {
      value = cv_dn(value + cv_dn(t.amp * cv_dn(p[t.axis] + t.offset)));
    } else if (t.kind == TWOS_TERM_GAUSS) {
      double exponent = 0.0;
      for (int a = 0; a < 3; ++a) {
        const double q = cv_up(cv_up(fabs(p[a] - t.c[a])) / t.w[a]);
        exponent = cv_up(exponent + cv_up(q * q));
      }
      value = cv_dn(value + cv_pdn(t.amp * cv_exp_lower(exponent)));
    } else if (t.kind == TWOS_TERM_CONST) {
      value = cv_dn(value + t.amp);
    }
  }
  return fmax(0.0, value);
}

}  // namespace

// Rounded-down distance of p to the box of triangle i.
__device__ __forceinline__ double cv_tri_box(const GeoDesc &G, uint32_t i, const double *p) {
  Vec<double> a, b, c;
  load_tri(G.tris_d, i, a, b, c);
  return cv_box_lower(fmin(fmin(a.x, b.x), c.x), fmin(fmin(a.y, b.y), c.y), fmin(fmin(a.z, b.z), c.z),
                      fmax(fmax(a.x, b.x), c.x), fmax(fmax(a.y, b.y), c.y), fmax(fmax(a.z, b.z), c.z), p[0], p[1],
                      p[2]);
}

constexpr int kCertBlock = 128;
constexpr int kCertStack = 8;  // traversal-stack entries per thread in shared memory; the deeper ones are local

// Certified walks, one per lane at a time.  One walk per thread on the FP64
// nodes took 170 ms for 65,536 walks (5.5 M steps, 20,480 triangles): twelve
// round-and-nextafter chains per node, root starts, a local-memory stack, and
// every walk of a site repeating its first query.
// Here a node costs two FP32 boxes; a query starts from the smaller of the
// grid's upper bound and the previous distance plus the step (the distance is
// 1-Lipschitz), at the grid's entry node; each site's first distance comes
// from V.mesh_distance.  With that the same walks took 40 ms, bound by the
// ~100 units of a query far from the surface, whose triangles' boxes are nearly
// equidistant.  But a distance d matters only below radius_cap / 0.95: beyond,
// the step is radius_cap and its points lie within d whatever d is.  So a query
// looks no farther, and there is none where the distance is known to be beyond
// -- by the previous distance less the steps since, or by the grid's lower
// bound of the distance to the triangles less the largest extent of a
// triangle's box: 6.3 ms.  What is left is the chain of up to max_steps FP64
// steps and near-surface queries of the longest walks.  Six blocks per SM leave
// 80 registers a thread, which spill 40 bytes.
__global__ void __launch_bounds__(kCertBlock, 6) cert_walk_kernel(const ValidateLaunch V, int lanes) {
  __shared__ uint2 s_stack[(kCertStack + kCand) * kCertBlock];
  __shared__ GeoDesc G;
  if (threadIdx.x == 0) G = *V.geo;
  __syncthreads();
  uint2 *stack = s_stack + threadIdx.x, *cand = stack + kCertStack * kCertBlock;
  uint2 deep[kStack + 1 - kCertStack];
  const unsigned lane = threadIdx.x & 31u, full = 0xffffffffu;
  const bool on = static_cast<int>(lane) < lanes;
  const unsigned on_mask = __ballot_sync(full, on);
  const uint64_t total = static_cast<uint64_t>(V.n_sites) * V.walks;
  uint32_t err = 0;
  unsigned long long failures = 0, total_steps = 0;
  int phase = kIdle;
  bool exhausted = false, resume = false;  // exhausted is warp-uniform
  uint64_t wid = 0;
  uint32_t site = 0, walk = 0, steps = 0, clipped = 0;
  double pt[3] = {0.0, 0.0, 0.0}, value = 0.0, best = 0.0;
  // Mesh distances from `far` on give the same step; `low` bounds the
  // distance from below.
  const double far = fmax(V.radius_cap / 0.95, V.epsilon) * (1.0 + 0x1.0p-20);
  double low = 0.0;
  Cull c{{0.f, 0.f, 0.f}, 0.f, 0.f, 0};
  int node = 0, sp = 0;
  bool have = false;
  uint32_t tri_cur = 0, tri_end = 0, iter = 0;
  float within = CUDART_INF_F;  // the grid's upper bound, where the query relies on it
  for (;;) {
    const unsigned idle = __ballot_sync(full, on && phase == kIdle);
    if (!exhausted && idle != 0u) {
      unsigned long long base = 0;
      const int leader = __ffs(idle) - 1;
      if (static_cast<int>(lane) == leader) base = atomicAdd(V.counter, static_cast<unsigned long long>(__popc(idle)));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= total) exhausted = true;
      if (on && phase == kIdle) {
        wid = base + __popc(idle & ((1u << lane) - 1u));
        if (wid < total) {
          site = static_cast<uint32_t>(wid / V.walks);
          walk = static_cast<uint32_t>(wid - static_cast<uint64_t>(site) * V.walks);
          for (int a = 0; a < 3; ++a) pt[a] = V.sites[3ull * site + a];
          value = 0.0;
          steps = clipped = 0;
          best = low = V.mesh_distance[site];
          c.count = 0;
          phase = kStep;
        }
      }
    }
    if (phase == kStep) {
      // The candidates' FP64 boxes, then the step.
      for (int k = 0; k < c.count; ++k) {
        const uint2 e = cand[k * kCertBlock];
        if (__uint_as_float(e.y) < c.limit) best = fmin(best, cv_tri_box(G, e.x, pt));
      }
      c.count = 0;
      if (resume && best > 0.0) {
        resume = false;
        phase = kTraverse;  // `best` is the smallest so far: no bound from below yet
      } else if (best > within) {
        // None within the grid's bound (grid_start): without it, from the root.
        resume = false;
        within = CUDART_INF_F;
        const float reach = __fmaf_ru(2.f, c.margin, __double2float_ru(far));
        c.limit = __fmul_ru(reach, reach);
        node = sp = 0;
        have = true;
        tri_cur = tri_end = iter = 0;
        phase = kTraverse;
      } else {
        resume = false;
        low = fmax(low, fmin(best, far));
        double d = fmin(best, fmax(low, far));
        for (uint32_t i = 0; i < V.n_cav; ++i)
          d = fmin(d, cv_dn(cv_point_distance(pt, V.cavities + 3 * i, false) - V.cavity_radius));
        d = fmax(0.0, d);
        bool done = d <= V.epsilon, capped = false, contained = true;
        double s = 0.0;
        if (!done) {
          s = fmin(V.radius_cap, cv_pdn(0.95 * d));
          const uint32_t ctr3 = V.repeat << 3, key = V.site_offset + site;
          const Philox4 q0 = philox(V.k0, V.k1, steps, walk, key, ctr3 | 0u);
          double to[2][3];  // the sampled points: the next position and the source point
          for (int a = 0; a < 3; ++a) to[1][a] = pt[a];
          if (V.green) {
            const Philox4 q1 = philox(V.k0, V.k1, steps, walk, key, ctr3 | 1u);
            const Philox4 q2 = philox(V.k0, V.k1, steps, walk, key, ctr3 | 2u);
            const Philox4 q3 = philox(V.k0, V.k1, steps, walk, key, ctr3 | 3u);
            const double beta = median3(uniform<double>(q2.x, q2.y), uniform<double>(q2.z, q2.w),
                                        uniform<double>(q3.x, q3.y));
            const Vec<double> g = direction<double>(uniform<double>(q1.x, q1.y), uniform<double>(q1.z, q1.w));
            const double sc = s * beta;
            to[1][0] = pt[0] + g.x * sc;
            to[1][1] = pt[1] + g.y * sc;
            to[1][2] = pt[2] + g.z * sc;
          }
          const Vec<double> dir = direction<double>(uniform<double>(q0.x, q0.y), uniform<double>(q0.z, q0.w));
          to[0][0] = pt[0] + dir.x * s;
          to[0][1] = pt[1] + dir.y * s;
          to[0][2] = pt[2] + dir.z * s;
          if (!(cv_point_distance(pt, to[0], true) < d) || !(cv_point_distance(pt, to[1], true) < d)) {
            contained = false;  // fail closed: this record must not be used
            ++failures;
            done = true;
          } else {
            const double weight = cv_pdn(cv_pdn(s * s) / 6.0);
            const double increment = cv_pdn(weight * cv_source_lower(V, to[1]));
            value = cv_pdn(value + increment);
            ++steps;
            if (value >= V.value_cap) {
              value = V.value_cap;
              clipped = 1;
              done = true;
            } else {
              for (int a = 0; a < 3; ++a) pt[a] = to[0][a];
              if (static_cast<int>(steps) >= V.max_steps) done = capped = true;
            }
          }
        }
        if (done) {
          twos_cert_sample out{};
          out.value = value;
          out.steps = steps;
          out.capped = capped;
          out.clipped = static_cast<uint8_t>(clipped);
          out.contained = contained;
          V.samples[wid] = out;
          total_steps += steps;
          phase = kIdle;
        } else {
          // Next query: below the previous mesh distance plus the step, and
          // below `far`.
          cull_begin(G, Vec<double>{pt[0], pt[1], pt[2]}, CUDART_INF, c);
          float ub = __fadd_ru(__double2float_ru(best), __double2float_ru(s));
          low -= s * (1.0 + 0x1.0p-40);
          best = CUDART_INF;
          within = CUDART_INF_F;
          float bound, upper;
          int entry = -1;
          if (G.grid && grid_bounds<true>(G, c.p, bound, upper, entry)) {
            upper = __fmaf_ru(6.f, G.delta, upper);
            if (upper < ub && upper < far) within = upper;
            ub = fminf(ub, upper);
            low = fmax(low, static_cast<double>(bound - G.box_extent - 2.f * c.margin));
          }
          if (low >= far) {
            within = CUDART_INF_F;
          } else {
            low = 0.0;
            node = ub < G.entry_radius ? max(entry_of(G, entry), 0) : 0;
            const float reach = __fmaf_ru(2.f, c.margin, fminf(ub, __double2float_ru(far)));
            c.limit = __fmul_ru(reach, reach);
            sp = 0;
            have = true;
            tri_cur = tri_end = 0;
            iter = 0;
            phase = kTraverse;
          }
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
      if (tri_cur >= tri_end) {
        while (!have && sp > 0) {
          --sp;
          const uint2 e = sp < kCertStack ? stack[sp * kCertBlock] : deep[sp - kCertStack];
          if (__uint_as_float(e.y) < c.limit) {
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
        best = 0.0;  // fail closed: a zero distance ends the walk
        c.count = 0;
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
        const float gx = gap(fminf(fminf(r1.x, r2.x), r3.x), fmaxf(fmaxf(r1.x, r2.x), r3.x), c.p.x);
        const float gy = gap(fminf(fminf(r1.y, r2.y), r3.y), fmaxf(fmaxf(r1.y, r2.y), r3.y), c.p.y);
        const float gz = gap(fminf(fminf(r1.z, r2.z), r3.z), fmaxf(fmaxf(r1.z, r2.z), r3.z), c.p.z);
        const float g2 = __fmaf_rn(gx, gx, __fmaf_rn(gy, gy, gz * gz));
        if (g2 < c.limit) {
          if (c.count >= kCand) {
            // A full candidate list is tested first; the triangle comes again.
            resume = true;
            phase = kStep;
            break;
          }
          cand[c.count * kCertBlock] = make_uint2(tri_cur, __float_as_uint(g2));
          ++c.count;
          const float up = __fmaf_ru(2.f, c.margin, __fsqrt_ru(g2));
          c.limit = fminf(c.limit, __fmul_ru(up, up));
        }
        ++tri_cur;
      } else {
        const float lx = gap(r0.x, r0.z, c.p.x), rx = gap(r0.y, r0.w, c.p.x);
        const float ly = gap(r1.x, r1.z, c.p.y), ry = gap(r1.y, r1.w, c.p.y);
        const float lz = gap(r2.x, r2.z, c.p.z), rz = gap(r2.y, r2.w, c.p.z);
        const float dl = __fmaf_rn(lx, lx, __fmaf_rn(ly, ly, lz * lz));
        const float dr = __fmaf_rn(rx, rx, __fmaf_rn(ry, ry, rz * rz));
        const int cl = __float_as_int(r5.z), cr = __float_as_int(r5.w);
        const bool vl = dl < c.limit, vr = dr < c.limit, swap = dr < dl;
        if (vl && vr) {
          const uint2 e = make_uint2(static_cast<uint32_t>(swap ? cl : cr), __float_as_uint(swap ? dl : dr));
          if (sp < kCertStack)
            stack[sp * kCertBlock] = e;
          else
            deep[sp - kCertStack] = e;
          ++sp;
        }
        have = vl || vr;
        node = vl && !(vr && swap) ? cl : cr;
      }
    }
  }
  if (err) atomicOr(V.error, err);
  if (failures) atomicAdd(&V.totals[0], failures);
  if (total_steps) atomicAdd(&V.totals[1], total_steps);
}

__global__ void __launch_bounds__(128) validate_kernel(const ValidateLaunch V) {
  const GeoDesc G = *V.geo;
  uint32_t err = 0;
  unsigned long long failures = 0, total_steps = 0;
  const uint64_t total = static_cast<uint64_t>(V.n_sites) * V.walks;
  for (uint64_t wid = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; wid < total;
       wid += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t site = static_cast<uint32_t>(wid / V.walks);
    const uint32_t walk = static_cast<uint32_t>(wid - static_cast<uint64_t>(site) * V.walks);
    double pt[3] = {V.sites[3ull * site], V.sites[3ull * site + 1], V.sites[3ull * site + 2]};
    twos_cert_sample out{};
    out.contained = 1;
    bool done = false;
    for (int k = 0; k < V.max_steps && !done; ++k) {
      const double d = cv_domain_distance(V, G, pt, err);
      if (d <= V.epsilon) {
        done = true;
        break;
      }
      const double s = fmin(V.radius_cap, cv_pdn(0.95 * d));
      const uint32_t ctr3 = V.repeat << 3;
      const Philox4 q0 = philox(V.k0, V.k1, static_cast<uint32_t>(k), walk, V.site_offset + site, ctr3 | 0u);
      double y[3] = {pt[0], pt[1], pt[2]};
      if (V.green) {
        const Philox4 q1 = philox(V.k0, V.k1, static_cast<uint32_t>(k), walk, V.site_offset + site, ctr3 | 1u);
        const Philox4 q2 = philox(V.k0, V.k1, static_cast<uint32_t>(k), walk, V.site_offset + site, ctr3 | 2u);
        const Philox4 q3 = philox(V.k0, V.k1, static_cast<uint32_t>(k), walk, V.site_offset + site, ctr3 | 3u);
        const double beta = median3(uniform<double>(q2.x, q2.y), uniform<double>(q2.z, q2.w),
                                    uniform<double>(q3.x, q3.y));
        const Vec<double> g = direction<double>(uniform<double>(q1.x, q1.y), uniform<double>(q1.z, q1.w));
        const double sc = s * beta;
        y[0] = pt[0] + g.x * sc;
        y[1] = pt[1] + g.y * sc;
        y[2] = pt[2] + g.z * sc;
      }
      const Vec<double> dir = direction<double>(uniform<double>(q0.x, q0.y), uniform<double>(q0.z, q0.w));
      const double next[3] = {pt[0] + dir.x * s, pt[1] + dir.y * s, pt[2] + dir.z * s};
      if (!(cv_point_distance(pt, next, true) < d) || !(cv_point_distance(pt, y, true) < d)) {
        out.contained = 0;  // fail closed: this record must not be used
        ++failures;
        done = true;
        break;
      }
      const double weight = cv_pdn(cv_pdn(s * s) / 6.0);
      const double increment = cv_pdn(weight * cv_source_lower(V, y));
      out.value = cv_pdn(out.value + increment);
      ++out.steps;
      if (out.value >= V.value_cap) {
        out.value = V.value_cap;
        out.clipped = 1;
        done = true;
        break;
      }
      pt[0] = next[0];
      pt[1] = next[1];
      pt[2] = next[2];
    }
    if (!done) out.capped = 1;
    total_steps += out.steps;
    V.samples[wid] = out;
  }
  if (err) atomicOr(V.error, err);
  if (failures) atomicAdd(&V.totals[0], failures);
  if (total_steps) atomicAdd(&V.totals[1], total_steps);
}

// Distances at each site, a warp per site: the exact FP64 one, and the
// certified ones to the mesh (every walk's first query) and to the domain.
__global__ void __launch_bounds__(kWosBlock) validate_center_kernel(const ValidateLaunch V) {
  __shared__ uint2 s_stack[kWarpStack * (kWosBlock / 32)];
  uint2 *stack = s_stack + kWarpStack * (threadIdx.x >> 5);
  const GeoDesc G = *V.geo;
  uint32_t err = 0;
  const uint32_t warps = gridDim.x * (kWosBlock / 32);
  for (uint32_t site = blockIdx.x * (kWosBlock / 32) + (threadIdx.x >> 5); site < V.n_sites; site += warps) {
    const double *p = V.sites + 3ull * site;
    const Vec<double> v{p[0], p[1], p[2]};
    double best2 = CUDART_INF;
    uint32_t tri = 0;
    double d = CUDART_INF;
    if (warp_nearest(G, v, best2, tri, stack, err, false)) d = sqrt(best2);
    double dm = CUDART_INF;
    Cull c;
    if (cull_begin(G, v, best2, c)) {
      // Boxes contain their triangles: the exact distance bounds this one.
      float limit = c.limit;
      uint32_t overrun = 0;
      warp_search<false>(G, c.p, 0, limit, stack, overrun, [&](uint32_t i, const float4 *r, float lim) {
        const float gx = gap(fminf(fminf(r[1].x, r[2].x), r[3].x), fmaxf(fmaxf(r[1].x, r[2].x), r[3].x), c.p.x);
        const float gy = gap(fminf(fminf(r[1].y, r[2].y), r[3].y), fmaxf(fmaxf(r[1].y, r[2].y), r[3].y), c.p.y);
        const float gz = gap(fminf(fminf(r[1].z, r[2].z), r[3].z), fmaxf(fmaxf(r[1].z, r[2].z), r[3].z), c.p.z);
        if (!(__fmaf_rn(gx, gx, __fmaf_rn(gy, gy, gz * gz)) < lim)) return lim;
        dm = fmin(dm, cv_tri_box(G, i, p));
        return cull_limit(dm * dm, c.margin);
      });
      warp_best(dm, tri);
      err |= overrun;
      if (overrun) dm = 0.0;  // fail closed, as cv_mesh_distance: the site's walks end at once
    } else {
      dm = cv_mesh_distance(G, p, err);
    }
    if ((threadIdx.x & 31u) != 0) continue;
    double clear = dm;
    for (uint32_t i = 0; i < V.n_cav; ++i) {
      const double dx = p[0] - V.cavities[3 * i], dy = p[1] - V.cavities[3 * i + 1], dz = p[2] - V.cavities[3 * i + 2];
      d = fmin(d, sqrt(dx * dx + dy * dy + dz * dz) - V.cavity_radius);
      clear = fmin(clear, cv_dn(cv_point_distance(p, V.cavities + 3 * i, false) - V.cavity_radius));
    }
    V.center_distance[site] = d;
    V.mesh_distance[site] = dm;
    V.clearance[site] = fmax(0.0, clear);
  }
  if (err) atomicOr(V.error, err);
}

cudaError_t launch_validate(const ValidateLaunch &V, cudaStream_t s) {
  const uint64_t total = static_cast<uint64_t>(V.n_sites) * V.walks;
  if (total == 0) return cudaSuccess;
  const int grid_c = static_cast<int>(std::min<uint32_t>((V.n_sites + kWosBlock / 32 - 1) / (kWosBlock / 32), 148u * 4));
  validate_center_kernel<<<grid_c, kWosBlock, 0, s>>>(V);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (V.cull) {
    int per_sm = 0, sms = 0, device = 0;
    if ((e = cudaGetDevice(&device)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cert_walk_kernel, kCertBlock, 0)) != cudaSuccess)
      return e;
    if (per_sm <= 0) return cudaErrorLaunchOutOfResources;
    // Fewer walks than lanes: spread over all warps, as launch_wos does.
    const uint64_t grid = static_cast<uint64_t>(per_sm) * sms, warps = grid * (kCertBlock / 32);
    const int lanes = static_cast<int>(std::min<uint64_t>(32, (total + warps - 1) / warps));
    cert_walk_kernel<<<static_cast<unsigned>(grid), kCertBlock, 0, s>>>(V, lanes);
  } else {
    const int grid = static_cast<int>(std::min<uint64_t>((total + 127) / 128, 148ull * 16));
    validate_kernel<<<grid, 128, 0, s>>>(V);
  }
  return cudaGetLastError();
}

}  // namespace twos
