/*
 * geo_fp32.cuh - device access to the FP32 geometry blob and the bounds that
 * the safe balls and the BVH searches of both precisions are built on: the
 * FP32 transport reads its surfaces here, the FP64 transport only bounds
 * (which flights cannot meet a surface, which nodes a ray cannot enter).
 */
#ifndef PTG_GEO_FP32_CUH
#define PTG_GEO_FP32_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace ptg {

namespace {

constexpr unsigned FULL = 0xffffffffu;
extern __shared__ float4 sblob[];

#ifdef PT_CHECK
/* Bounds-checked build: [0] violations, [1] code of the first, [2] its
   index, one set per file of kernels.  A failed check is recorded and the
   access is redirected to a valid element; the kernel never traps. */
__device__ int g_check[3];
cudaError_t check_read(long long* count, int* code, int* index, bool reset) {
  int v[3] = {0, 0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(v, g_check, sizeof(v));
  if (e != cudaSuccess) return e;
  *count = v[0];
  *code = v[1];
  *index = v[2];
  if (reset) {
    const int z[3] = {0, 0, 0};
    e = cudaMemcpyToSymbol(g_check, z, sizeof(z));
  }
  return e;
}
__device__ __noinline__ void check_fail(int code, int index) {
  if (atomicAdd(&g_check[0], 1) == 0) {
    g_check[1] = code;
    g_check[2] = index;
  }
}
#endif

/* Geometry blob accessor: SMEM = true reads the copy staged in shared
   memory (shared-memory loads), false reads global memory through the
   read-only path. */
template <bool SMEM>
struct Geo {
  const float4* base;   /* global blob (SMEM = false) */
  BlobLayout lay;
  int nstage = 0;       /* SMEM = false: BVH node units staged in shared memory */
  __device__ __forceinline__ float4 ld(int i) const {
#ifdef PT_CHECK
    if ((unsigned)i >= (unsigned)lay.total) { check_fail(1, i); i = 0; }
#endif
    if (SMEM) return sblob[i];
    return __ldg(base + i);
  }
  __device__ __forceinline__ int ldi(int unit, int k) const {
#ifdef PT_CHECK
    if (k < 0 || (unsigned)(unit + k / 4) >= (unsigned)lay.total) { check_fail(1, unit + k / 4); unit = 0; k = 0; }
#endif
    if (SMEM) return reinterpret_cast<const int*>(sblob + unit)[k];
    return __ldg(reinterpret_cast<const int*>(base + unit) + k);
  }
  __device__ __forceinline__ float4 hotA(int s) const { return ld(lay.hot + 2 * s); }
  __device__ __forceinline__ int4 hotB(int s) const {
    const float4 v = ld(lay.hot + 2 * s + 1);
    return make_int4(__float_as_int(v.x), __float_as_int(v.y), __float_as_int(v.z),
                     __float_as_int(v.w));
  }
  __device__ __forceinline__ float4 cold(int s, int i) const { return ld(lay.cold + 3 * s + i); }
  __device__ __forceinline__ float4 edge(int e) const { return ld(lay.edge + e); }
  __device__ __forceinline__ int cand_begin(int g) const { return ldi(lay.cand_begin, g); }
  __device__ __forceinline__ int cand(int k) const { return ldi(lay.cand, k); }
  __device__ __forceinline__ float4 start(int i) const { return ld(lay.start + i); }
  __device__ __forceinline__ int bvh_root(int g) const { return ldi(lay.bvh_root, g); }
  __device__ __forceinline__ int plane_begin(int g) const { return ldi(lay.plane_begin, g); }
  __device__ __forceinline__ float4 plane(int i) const { return ld(lay.plane + i); }
  __device__ __forceinline__ float4 node(int i) const {
    if (!SMEM && i < nstage) return sblob[i];  /* a top level, staged */
    return ld(lay.bvh_node + i);
  }
};

/* Square root from the hardware approximation (relative error ~2^-22). */
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

/* Entry distance of the ray into a node box (+inf when it misses the box
   or enters beyond tmax); inverse direction components are finite. */
__device__ __forceinline__ float box_entry(float4 lo, float4 hi, float px, float py, float pz,
                                           float ix, float iy, float iz, float tmax, float eps) {
  const float ax = (lo.x - px) * ix, bx = (hi.x - px) * ix;
  const float ay = (lo.y - py) * iy, by = (hi.y - py) * iy;
  const float az = (lo.z - pz) * iz, bz = (hi.z - pz) * iz;
  const float t0 = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
  const float t1 = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
  return (t0 <= t1 && t1 >= -eps && t0 <= tmax) ? t0 : 3.0e38f;
}

__device__ __forceinline__ float inv_dir(float d) {
  return __fdividef(1.0f, fabsf(d) > 1.0e-20f ? d : copysignf(1.0e-20f, d));
}

/* Traversal depth bound: the builder limits the depth to 30. */
constexpr int kBvhStack = 32;

/* Lower bound of the distance from p to one candidate surface (planes bound
   polygons from below, the infinite cylinder bounds the clipped one).  The
   square roots are the hardware approximation: its relative error (< 2^-22
   of a distance below the box diagonal) is far inside the 4 eps the callers
   take off, so the bound stays a bound. */
template <int EXT, class G_t>
__device__ __forceinline__ float surface_lb(const G_t& G, int s, float px, float py, float pz) {
  const float4 A = G.hotA(s);
  const int4 B = G.hotB(s);
  const int type = B.x & 0xff;
  if (type == REC_POLY) return fabsf(A.w - fmaf(A.x, px, fmaf(A.y, py, A.z * pz)));
  if (EXT && type == REC_CAP) {
    /* inside: the nearer of mantle and caps; outside: the larger excess */
    const float4 E = G.edge(B.y);
    const float wx = px - A.x, wy = py - A.y, wz = pz - A.z;
    const float sa = fmaf(wx, E.x, fmaf(wy, E.y, wz * E.z));
    const float ux = fmaf(-sa, E.x, wx), uy = fmaf(-sa, E.y, wy), uz = fmaf(-sa, E.z, wz);
    const float er = sqrt_approx(fmaf(ux, ux, fmaf(uy, uy, uz * uz))) - A.w;
    const float ea = fabsf(sa) - E.w;
    return (er <= 0.0f && ea <= 0.0f) ? fminf(-er, -ea) : fmaxf(er, ea);
  }
  if (type == REC_SPHERE) {
    const float wx = px - A.x, wy = py - A.y, wz = pz - A.z;
    return fabsf(sqrt_approx(fmaf(wx, wx, fmaf(wy, wy, wz * wz))) - A.w);
  }
  const float wx = px - A.x, wy = py - A.y;
  return fabsf(sqrt_approx(fmaf(wx, wx, wy * wy)) - A.z);
}

/* Distance from p to a node box (0 inside; approximate square root, as in
   surface_lb). */
__device__ __forceinline__ float box_dist(float4 lo, float4 hi, float px, float py, float pz) {
  const float ex = fmaxf(fmaxf(lo.x - px, px - hi.x), 0.0f);
  const float ey = fmaxf(fmaxf(lo.y - py, py - hi.y), 0.0f);
  const float ez = fmaxf(fmaxf(lo.z - pz, pz - hi.z), 0.0f);
  return sqrt_approx(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
}

/* BVH range query for the safe ball: the smallest lower bound d of the
   distance from p to a surface of the grain, the surface it belongs to
   (near) and the smallest bound d2 of every other surface, searched below
   the initial d (nodes no nearer than the second bound so far are pruned:
   they cannot change either; a surface's bound is the larger of the
   distance to its leaf's box and its own plane / quadric bound).  Out of
   line, like scan_bvh. */
template <int EXT, class G_t>
__device__ __noinline__ float safety_bvh(const G_t& G, int root, float px, float py, float pz,
                                         float d, float& d2, int& near) {
  int stk[kBvhStack];
  float std_[kBvhStack];
  int sp = 0;
  int node = root;
  d2 = d;
  near = -1;
  while (true) {
    const float4 n0 = G.node(2 * node), n1 = G.node(2 * node + 1);
    const int cnt = __float_as_int(n1.w);
    const int a = __float_as_int(n0.w);
    bool descended = false;
    if (cnt > 0) {
      const float bd = box_dist(n0, n1, px, py, pz);
      for (int k = a; k < a + cnt; ++k) {
        const int sk = G.cand(k);
        const float e = fmaxf(bd, surface_lb<EXT>(G, sk, px, py, pz));
        const bool nearer = e < d;
        d2 = nearer ? d : fminf(d2, e);
        near = nearer ? sk : near;
        d = nearer ? e : d;
      }
    } else {
      const float dl = box_dist(G.node(2 * a), G.node(2 * a + 1), px, py, pz);
      const float dg = box_dist(G.node(2 * a + 2), G.node(2 * a + 3), px, py, pz);
      const bool lf = dl <= dg;
      const float dn = lf ? dl : dg, df = lf ? dg : dl;
      if (dn < d2) {
        if (df < d2 && sp < kBvhStack) {
          stk[sp] = lf ? a + 1 : a;
          std_[sp] = df;
          ++sp;
        }
        node = lf ? a : a + 1;
        descended = true;
      }
    }
    if (descended) continue;
    bool found = false;
    while (sp > 0) {
      --sp;
      if (std_[sp] < d2) {
        node = stk[sp];
        found = true;
        break;
      }
    }
    if (!found) break;
  }
  return d;
}

/* Lower bound of the distance from p to every box face and to every
   candidate surface of the grain, less 4 eps.  A grain with a BVH is
   searched only within `cap` (the radius the safe ball needs).  dgrain
   receives the bound over the candidate surfaces alone (the grain ball: a
   flight inside it needs the box-face test only); for a BVH grain it is
   searched no farther than the full bound, so it costs no extra nodes. */
template <int EXT, class G_t>
__device__ __forceinline__ float safety(const G_t& G, int grain, float px, float py, float pz,
                                        float X, float Y, float Z, float eps, float cap,
                                        float& dgrain, float& dgrain2, int& near) {
  const float dbox = fminf(fminf(fminf(px, X - px), fminf(py, Y - py)), fminf(pz, Z - pz));
  float dc = 3.0e38f, dc2 = 3.0e38f;
  near = -1;
  if (grain > 0) {
    const int root = EXT ? G.bvh_root(grain) : -1;
    if (root < 0) {
      /* the nearest candidate and the bound of all the others */
      const int kb = G.cand_begin(grain), ke = G.cand_begin(grain + 1);
      for (int k = kb; k < ke; ++k) {
        const int sk = G.cand(k);
        const float d = surface_lb<EXT>(G, sk, px, py, pz);
        const bool nearer = d < dc;
        dc2 = nearer ? dc : fminf(dc2, d);
        near = nearer ? sk : near;
        dc = nearer ? d : dc;
      }
    } else {
      const int kb = EXT == 2 ? G.plane_begin(grain) : 0;
      const int ke = EXT == 2 ? G.plane_begin(grain + 1) : 0;
      if (ke > kb) {
        for (int k = kb; k < ke; ++k) {
          const float4 A = G.plane(k);
          dc = fminf(dc, fabsf(fmaf(A.x, px, fmaf(A.y, py, A.z * pz)) - A.w));
        }
        dc2 = dc;
      } else {
        dc = safety_bvh<EXT>(G, root, px, py, pz, fminf(dbox, cap), dc2, near);
      }
    }
  }
  dgrain = dc - 4.0f * eps;
  dgrain2 = dc2 - 4.0f * eps;
  return fminf(dbox, dc) - 4.0f * eps;
}

/* Whether a flight of length fp from p along d ends behind every facet plane
   of a BVH grain that has them: a polygon is met only from behind (along its
   outward normal), so none is met up to fp.  The margin covers the polygons'
   distance from their plane (eps / 4), the tests' eps and the rounding of the
   direction times fp.  A ballistic flight (infinite, 1e10 in FP64) ends behind
   none: 8000 ballistic phonons in a small mesh 0.48 -> 0.44 ms without asking.
   This and the plane bounds of the balls replace nearly
   every tree walk in a polyhedral grain: 5 Voronoi grains as 43 000 triangles,
   2.5e6 phonons: 160 -> 54 ms (drain 60 -> 22, tail 93 -> 27). */
template <class G_t>
__device__ __forceinline__ bool behind_planes(const G_t& G, int grain, float px, float py, float pz,
                                              float dx, float dy, float dz, float fp, float eps) {
  if (fp >= 1.0e10f) return false;
  const int kb = G.plane_begin(grain), ke = G.plane_begin(grain + 1);
  const float m = -fmaf(5.0e-7f, fp, 4.0f * eps);
  bool behind = ke > kb;
  for (int k = kb; k < ke; ++k) {
    const float4 A = G.plane(k);
    const float s = fmaf(A.x, px, fmaf(A.y, py, A.z * pz)) - A.w;
    behind = behind && fmaf(fp, fmaf(A.x, dx, fmaf(A.y, dy, A.z * dz)), s) < m;
  }
  return behind;
}

/* Buckets of the tail order: a quarter octave of the expected walk each. */
constexpr int kOrderBuckets = 128;
static_assert(2 * kOrderBuckets == kTailOrderExtra, "tail order histogram and cursors");

/* Bucket of a phonon's expected remaining walk.  A diffusive phonon at x
   between the baths at 0 and L takes about 1.5 x (L - x) / MFP^2 more flights
   to leave (the exit time of a random walk whose flights move it by
   2 MFP^2 / 3 squared along x); walls and holes stretch the walk, but the
   phonons the tail phase waits for are those that rank high on it. */
__device__ __forceinline__ int order_bucket(float x, float x_len, float lam) {
  const float w = __fdividef(fmaxf(x * (x_len - x), 0.0f), lam * lam);
  return w > 1.0f ? min(kOrderBuckets - 1, (int)(4.0f * __log2f(w))) : 0;
}

/* Chunk c of the work queue: (task, first local particle, count). */
__device__ __forceinline__ int3 queue_chunk(const ChunkQueue& q, int c) {
  const int k = c / q.per_task;
  const int j = (c - k * q.per_task) * q.size;
  return make_int3(q.order ? __ldg(q.order + k) : k, j, min(q.size, q.np_local - j));
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

}  // namespace

}  // namespace ptg

#endif
