// render.cu -- wavefront path tracing, path-replay adjoint and edge sampling.
//
// Forward (path_integrator.cc:80-186 trace2light, :355-372 render_interior,
// camera.h:75-87 Film::add) as wavefront kernels over a tile of path samples:
//   k_camera  : sampler stream, pixel jitter, camera ray, primary closest hit
//   per depth : k_shade (hit-light test, light / BSDF / indirect sampling, ray write
//               with warp-aggregated compaction) -> k_trace (closest hit per ray)
//               -> k_accum (NEE + MIS contributions, throughput, compaction)
//   k_film    : per-pixel average of its spp paths (deterministic, no atomics).
// Backward (Wrap2torch.backward + enoki reverse sweep, torch_psdr.py:48-72): from the hit
// records that the forward kept (or that re-tracing the tile from its seeds gives),
// k_adjoint replays every path's sampler stream and applies the hand-written adjoint of
// the estimator, scattering into fixed-point accumulators (warp-aggregated where a warp
// shares the target). Primary-edge (path_integrator.cc:188-272) and direct-edge (:274-353)
// boundary terms follow the reference formulas (PSDR_EST_REFERENCE).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include "render.h"

namespace psdr {

// ------------------------------------------------------------------ helpers
PSDR_D unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Warp-aggregated append: all lanes of the warp must call it together.
PSDR_D int warp_append(int* counter, bool pred) {
  const unsigned m = __ballot_sync(0xffffffffu, pred);
  if (!m) return -1;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  return pred ? base + __popc(m & lanemask_lt()) : -1;
}

// Warp-aggregated append of n entries per lane: the lane's first entry. All lanes call it.
PSDR_D int warp_reserve(int* counter, int n) {
  const int lane = threadIdx.x & 31;
  int sum = n;
  for (int k = 1; k < 32; k <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, k);
    if (lane >= k) sum += v;
  }
  const int total = __shfl_sync(0xffffffffu, sum, 31);
  if (total == 0) return 0;
  int base = 0;
  if (lane == 0) base = atomicAdd(counter, total);
  return __shfl_sync(0xffffffffu, base, 0) + sum - n;
}

PSDR_D void xform_pos(const float* m, float3 p, float3& out) {
  const float w = m[12] * p.x + m[13] * p.y + m[14] * p.z + m[15];
  out = f3((m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3]) / w, (m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7]) / w,
           (m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11]) / w);
}
PSDR_D float3 xform_dir(const float* m, float3 p) {
  return f3(m[0] * p.x + m[1] * p.y + m[2] * p.z, m[4] * p.x + m[5] * p.y + m[6] * p.z,
            m[8] * p.x + m[9] * p.y + m[10] * p.z);
}

// camera.h:260-276 gen_camera_ray_with_point: visibility in the raster + pixel.
PSDR_D bool project(const DevView& V, float3 pt, int& px, int& py) {
  float3 pc, p;
  xform_pos(V.w2c, pt, pc);
  xform_pos(V.c2r, pc, p);
  px = (int)floorf(p.x);
  py = (int)floorf(p.y);
  return pc.z < 0.f && p.x > 0.f && p.x < (float)V.W && p.y > 0.f && p.y < (float)V.H;
}

// camera.h:121 look direction c2w (0, 0, -1).
PSDR_D float3 view_look_dir(const DevView& V) { return f3(-V.c2w[2], -V.c2w[6], -V.c2w[10]); }

// camera.h:336-353 orthographic ray toward world point pt: origin c2w (w2c pt).xy0 (in
// the same rounded operations as the float oracle), direction the look direction.
PSDR_D float3 ortho_origin_rn(const DevView& V, float3 pt) {
  const float3 pc = xform_pos_rn(V.w2c, pt);
  return xform_pos_rn(V.c2w, f3(pc.x, pc.y, 0.f));
}

// Transposed Jacobian of that origin w.r.t. the point, applied to a: M^T a with
// M = C diag(1, 1, 0) W (C, W the rotation parts of c2w, w2c).
PSDR_D float3 ortho_origin_jt(const DevView& V, float3 a) {
  const float ux = V.c2w[0] * a.x + V.c2w[4] * a.y + V.c2w[8] * a.z;
  const float uy = V.c2w[1] * a.x + V.c2w[5] * a.y + V.c2w[9] * a.z;
  return f3(V.w2c[0] * ux + V.w2c[4] * uy, V.w2c[1] * ux + V.w2c[5] * uy, V.w2c[2] * ux + V.w2c[6] * uy);
}

PSDR_D int find_view(const DevView* __restrict__ views, int nv, long long g) {
  int lo = 0, hi = nv - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (views[mid].sample_off <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}
PSDR_D int find_view_pix(const DevView* __restrict__ views, int nv, long long g) {
  int lo = 0, hi = nv - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (views[mid].pix_off <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Replay record k of path s: 0 its primary hit; 1 + d R + r the hit of ray r of depth d;
// 1 + D R + 2 d and the next the depth's contribution C and throughput factor beta. Records lie
// field by field, so that a warp's neighbouring paths read and write whole lines (path by
// path, 264 B apart, each access of a depth-3 path moved a 32-byte sector for 16 bytes).
PSDR_D float4& rec_at(const WF& w, int s, int k) { return w.rec[(size_t)k * w.rec_plane + s]; }
PSDR_D float4& rec_hit(const WF& w, int s, int d, int r) { return rec_at(w, s, 1 + d * w.R + r); }
PSDR_D float4& rec_c(const WF& w, int s, int d) { return rec_at(w, s, 1 + w.D * w.R + 2 * d); }
PSDR_D float4& rec_beta(const WF& w, int s, int d) { return rec_at(w, s, 2 + w.D * w.R + 2 * d); }

PSDR_D float4 hit4(const HitRec& h) { return make_float4(__int_as_float(h.tri), h.b1, h.b2, h.t); }

// Out of line: the adjoint kernels scatter vertex and texel gradients from many call
// sites, and one copy of the three fixed-point conversions keeps their loops smaller in
// the instruction cache.
static __device__ __noinline__ void atomic_add3(GradAcc* p, float3 v) {
  acc_add(p, v.x);
  acc_add(p + 1, v.y);
  acc_add(p + 2, v.z);
}

// Vertex gradients are accumulated only for the vertices the caller asked for.
PSDR_D bool vert_wanted(const DevScene& sc, int v) { return sc.grad_verts && (!sc.vmask || sc.vmask[v]); }
PSDR_D void vert_add(const DevScene& sc, int v, float3 a) {
  if (vert_wanted(sc, v)) atomic_add3(sc.grad_verts + 3 * (size_t)v, a);
}

// ------------------------------------------------------------------ camera kernel
// ORTHO: the instance for jobs with an orthographic view (it handles both camera types).
// 64 registers (8 blocks of 128 threads per SM): the record writes of the replay instances
// otherwise take 76.
template <int MODE, bool ORTHO>
__global__ void __launch_bounds__(128, 8) k_camera(WF w, const DevScene* __restrict__ scenes,
                                                const DevView* __restrict__ views, Tile tile) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (tile.n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < tile.n) {
      const long long g = tile.begin + s;
      const int v = find_view(views, w.nviews, g);
      const DevView& V = views[v];
      const DevScene& sc = scenes[V.scene];
      const long long i = g - V.sample_off;
      Rng rng = make_rng((unsigned long long)i + w.seed);
      const float jx = rng.next_float(), jy = rng.next_float();
      const int pix = V.spp > 1 ? (int)(i / V.spp) : (int)i;
      const int x = pix % V.W, y = pix / V.W;
      float3 pc;
      xform_pos(V.r2c, f3(jx + (float)x, jy + (float)y, 1.0f), pc);
      float3 o = V.pos, d;
      if (ORTHO && V.ortho) {
        // camera.h:313-334: origin on the camera plane, direction the look direction
        xform_pos(V.c2w, f3(pc.x, pc.y, 0.f), o);
        d = view_look_dir(V);
      } else {
        d = normalize(xform_dir(V.c2w, pc));
      }
      w.org[s] = make_float4(o.x, o.y, o.z, 0.f);  // before the out-of-line trace: o dies there
      const HitRec h = trace_closest(sc, o, d, kTmin, INFINITY);
      w.rs[s] = rng.state;
      w.ri[s] = rng.inc;
      w.view[s] = v;
      w.pix[s] = pix;
      w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
      w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      w.cur[s] = hit4(h);
      if (MODE != MODE_FWD) rec_at(w, s, 0) = hit4(h);
      alive = h.tri >= 0;
    }
    const int k = warp_append(&w.cnt[0], alive);
    if (alive) w.q0[k] = s;
  }
}

// ------------------------------------------------------------------ shade kernel
// A MIS BSDF-sample ray counts only if it ends on a light (the accumulate and adjoint kernels
// skip any other hit): the closest light triangle along it, by the traversal's test and tie
// rule, bounds an occlusion query of k_trace, and a ray with no light along it (nineteen in
// twenty under a small lamp) needs none. For lights of at most this many triangles in all.
constexpr int kMisLightTris = 16;

// Returns the bound of the query: the light's distance; < 0: no light along the ray; infinity: too
// many light triangles, trace for the closest hit.
PSDR_D float mis_light_bound(const DevScene& sc, float3 o, float3 d) {
  int nlt = 0;
  for (int l = 0; l < sc.nlight; ++l) nlt += sc.lights[l].ntri;
  if (sc.nlight == 0 || nlt > kMisLightTris) return INFINITY;
  const RayPre rp = ray_pre(o, d);
  float tl = INFINITY;
  int best = -1;
  for (int l = 0; l < sc.nlight; ++l) {
    const DevLight& Lt = sc.lights[l];
    for (int t = Lt.tri0; t < Lt.tri0 + Lt.ntri; ++t) {
      const float4* q = sc.tri + 6 * (size_t)t;
      float tt, b1, b2;
      if (tri_test(rp, xyz(__ldg(q)), xyz(__ldg(q + 1)), xyz(__ldg(q + 2)), kTmin, tl, tt, b1, b2) &&
          (tt < tl || best < 0 || t < best)) {
        tl = tt;
        best = t;
      }
    }
  }
  return best < 0 ? -1.f : tl;
}

// Hit-light test and all samples of one depth; rays are written to the shaded slot. From
// kListMin paths on, the BSDF-sample rays that need a traversal are listed (slots past
// nL * cap, in ra[].y from slot nL * cap on, counted in cnt[2D+3]) and the others get their miss
// here, where 32 lanes make the light test together; below, k_trace makes it as a lane takes
// the ray, while the other rays of the warp wait. The test adds 6 us to a small launch of this
// kernel, which is what k_trace saves on 2^18 paths (plain 128^2 x 16 spp render); 2^20 paths
// of 256^2 x 16 spp: k_trace 595 -> 566 us for 11 us more here; 2^22 of 256^2 x 64 spp: 1.18 ->
// 1.05 ms for 0.02. The form holds for every depth of a loop, since it pays at the late ones too:
// with the list at the first depth only, the first two, the first three and all, the large
// render (depth 5) takes 17.78, 17.72, 17.68 and 17.67 ms, its batched step 87.5, 87.3, 87.2, 87.1.
constexpr int kListMin = 1 << 19;
template <int MODE, bool BSDF, bool LIST>
__global__ void __launch_bounds__(256) k_shade(WF w, const DevScene* __restrict__ scenes,
                                               const DevView* __restrict__ views, int d) {
  const int* qin = (d & 1) ? w.q1 : w.q0;
  const int n = w.cnt[2 * d];
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const bool last = d == w.D - 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) w.cnt[2 * w.D + 2] = 0;  // ray fetch counter of k_trace
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n32; q += stride) {
    bool go = false;
    int s = -1;
    Surf x;
    const DevScene* sc = nullptr;
    if (q < n) {
      s = qin[q];
      sc = &scenes[views[w.view[s]].scene];
      const float4 c = w.cur[s];
      x = make_surf(*sc, __float_as_int(c.x), c.y, c.z, xyz(w.org[s]));
      if (x.is_light) {
        if (MODE != MODE_REPLAY && w.light_vis && d == 0) {
          const DevLight& Lt = sc->lights[x.light];
          float4 L = w.L[s];
          const float4 T = w.T[s];
          const float3 e = light_emit<BSDF>(Lt, x);
          L.x += T.x * e.x; L.y += T.y * e.y; L.z += T.z * e.z;
          w.L[s] = L;
        }
      } else {
        go = true;
      }
    }
    const int k = warp_append(&w.cnt[2 * d + 1], go);
    Rng rng{0, 0};
    float3 Ns;
    if (go) {
      w.qs[k] = s;
      rng.state = w.rs[s];
      rng.inc = w.ri[s];
      float3 mm;
      bool mapped;
      Ns = BSDF ? shading_normal(sc->objs[x.obj], x, mm, mapped) : x.n;
    }
    // rays are stored type-major (slot r * cap + k): a warp of k_trace then traces
    // rays of one kind from neighbouring paths
    const size_t cs = (size_t)w.cap;
    for (int i = 0; go && i < w.nL; ++i) {
      const float rx = rng.next_float(), ry = rng.next_float();
      const LightSample ls = sample_light(*sc, rx, ry);
      const float3 dv = ls.y - x.p;
      const float3 dir = normalize(dv);
      const float dist = norm(dv);
      const size_t slot = i * cs + k;
      w.ro[slot] = make_float4(x.p.x, x.p.y, x.p.z, dist * 1.0001f + 4e-3f);
      w.rd[slot] = make_float4(dir.x, dir.y, dir.z, __int_as_float(ls.light));
      w.ra[slot] = make_float4(ls.y.x, ls.y.y, ls.y.z, ls.pdf);
    }
    unsigned listed = 0;  // samples to list (kMaxRays bounds them)
    for (int j = 0; j < w.nB; ++j) {
      if (go) {
        const float rx = rng.next_float(), ry = rng.next_float();
        float ct, st, sp, cp;
        const float3 wo =
            BSDF ? material_dir(x, Ns, rx, ry, ct, st, sp, cp) : diffuse_dir(x.n, x.t, rx, ry, ct, st, sp, cp);
        const float tl = LIST ? mis_light_bound(*sc, x.p, wo) : INFINITY;
        const size_t slot = (w.nL + j) * cs + k;
        if (!(tl < 0.f)) {
          listed |= 1u << j;
          w.ro[slot] = make_float4(x.p.x, x.p.y, x.p.z, tl);
          w.rd[slot] = make_float4(wo.x, wo.y, wo.z, 0.f);
          w.ra[slot].x = ct;
        } else {
          w.hit[slot] = make_float4(__int_as_float(-1), 0.f, 0.f, INFINITY);
        }
      }
    }
    if (LIST) {
      int i = warp_reserve(&w.cnt[2 * w.D + 3], __popc(listed));  // one atomic per warp
      for (; listed; listed &= listed - 1)
        w.ra[w.nL * cs + i++].y = __uint_as_float((unsigned)((__ffs(listed) - 1) * cs + k));
    }
    if (go) {
      const float rx = rng.next_float(), ry = rng.next_float();
      if (!last) {
        float ct, st, sp, cp;
        const float3 wo =
            BSDF ? material_dir(x, Ns, rx, ry, ct, st, sp, cp) : diffuse_dir(x.n, x.t, rx, ry, ct, st, sp, cp);
        const size_t slot = (w.nL + w.nB) * cs + k;
        w.ro[slot] = make_float4(x.p.x, x.p.y, x.p.z, INFINITY);
        w.rd[slot] = make_float4(wo.x, wo.y, wo.z, 0.f);
        w.ra[slot] = make_float4(ct, 0.f, 0.f, 0.f);
      }
      w.rs[s] = rng.state;
    }
  }
}

// ------------------------------------------------------------------ trace kernel
// Closest hit of every queued ray of a depth (light-sample rays r < nL stop at the first
// hit short of the light). Persistent warps with dynamic ray fetch: the lanes whose rays
// have finished take the next unclaimed rays of the queue together once there are kRefill
// of them, so a warp keeps its lanes busy instead of waiting for its longest ray (the rays
// of a warp differ in traversal length by an order of magnitude) and the ray set-up runs on
// at least half a warp. The fetch counter is w.cnt[2D+2], reset by k_shade.
//
// Bound by instruction issue and divergence, not by memory: on 256^2 x 32 spp rays of the
// icosphere scene the SMs issue on 79 % of the cycles with 18.6 of 32 lanes active at the first
// depth, 68 % and 16 at the third (11 before lanes waited for one another at leaves,
// trav_step); L1 64-82 %, L2 11-18 %, DRAM 2-3 % of their peaks. Traversal
// of the 512^2 x 32 spp icosphere step: 14.0 ms before, 12.2 ms now (2^20-path tiles).
constexpr int kRefill = 16;
// Per-lane memory of k_trace: the first kShort stack entries, the ray as the triangle test
// takes it and the hit's barycentrics live in shared memory (one column per lane, so a
// warp's accesses hit 32 banks), which keeps them out of the registers of the node visits;
// deeper stack entries are in local memory.
constexpr int kShort = 16;
// Resident blocks asked for: 64 registers, no spills. 6 and 7 blocks take 1-3 % longer, 9 and
// more spill (+16 % and up).
constexpr int kTraceBlocks = 8;
struct TraceShared {
  int stack[kShort][128];
  float ray[8][128];  // origin, shear constants, barycentrics
};
struct TraceMem {
  TraceShared* sh;
  int lane;
  int kz;
  int deep[kStack - kShort];
  PSDR_D void set_ray(const RayPre& r) {
    sh->ray[0][lane] = r.o.x; sh->ray[1][lane] = r.o.y; sh->ray[2][lane] = r.o.z;
    sh->ray[3][lane] = r.Sx; sh->ray[4][lane] = r.Sy; sh->ray[5][lane] = r.Sz;
    kz = r.kz;
    bary(0.f, 0.f);
  }
  PSDR_D RayPre ray() const {
    RayPre r;
    r.o = f3(sh->ray[0][lane], sh->ray[1][lane], sh->ray[2][lane]);
    r.Sx = sh->ray[3][lane]; r.Sy = sh->ray[4][lane]; r.Sz = sh->ray[5][lane];
    r.kz = kz;
    return r;
  }
  PSDR_D void bary(float u, float v) { sh->ray[6][lane] = u; sh->ray[7][lane] = v; }
  PSDR_D float b1() const { return sh->ray[6][lane]; }
  PSDR_D float b2() const { return sh->ray[7][lane]; }
  PSDR_D void put(int i, int v) { if (i < kShort) sh->stack[i][lane] = v; else deep[i - kShort] = v; }
  PSDR_D void push3(int sp, int n, int c1, int c2, int c3) {
    if (sp + 3 <= kShort) {
      // a slot above the new top may be overwritten: three stores, no branch
      sh->stack[sp + 2][lane] = c1;
      sh->stack[sp + (n > 2 ? 1 : 0)][lane] = n > 2 ? c2 : (n > 1 ? c2 : c1);
      sh->stack[sp + (n > 2 ? 0 : 1)][lane] = n > 2 ? c3 : c1;
    } else {
      if (n > 2) put(sp, c3);
      if (n > 1) put(sp + n - 2, c2);
      if (n > 0) put(sp + n - 1, c1);
    }
  }
  PSDR_D int pop(int i) const { return i < kShort ? sh->stack[i][lane] : deep[i - kShort]; }
};
template <bool LIST>
__global__ void __launch_bounds__(128, kTraceBlocks) k_trace(WF w, const DevScene* __restrict__ scenes,
                                                             const DevView* __restrict__ views, int d,
                                                             unsigned long long* __restrict__ ray_count) {
  const unsigned nk = (unsigned)w.cnt[2 * d + 1];
  const int Rd = (d == w.D - 1) ? w.R - 1 : w.R;
  if (ray_count && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(ray_count, (unsigned long long)nk * Rd);
  // the queue: light-sample rays, BSDF-sample rays (all or those k_shade listed), indirect rays
  const unsigned n_light = nk * (unsigned)w.nL, n_list = n_light + (LIST ? (unsigned)w.cnt[2 * w.D + 3] : nk * (unsigned)w.nB);
  const unsigned total = n_list + (d == w.D - 1 ? 0u : nk);
  unsigned* fetch = reinterpret_cast<unsigned*>(w.cnt + 2 * w.D + 2);
  __shared__ TraceShared sh;
  TraceMem mem;
  mem.sh = &sh;
  mem.lane = threadIdx.x;
  Trav s;
  s.node = kNoNode;
  const DevScene* sc = scenes;
  size_t slot = 0;
  bool open = false;  // the lane's ray has been traversed and its hit is not written yet
  unsigned next = 0;  // last index this warp claimed: beyond `total` the queue is empty
  const float4* nodes = nullptr;
  const float4* leaf = nullptr;
  while (true) {
    if (open && s.node == kNoNode) {
      w.hit[slot] = make_float4(__int_as_float(s.tri), mem.b1(), mem.b2(), s.t);
      open = false;
    }
    const unsigned idle = __ballot_sync(0xffffffffu, !open);
    if (next < total && (__popc(idle) >= kRefill)) {
      const int lane = threadIdx.x & 31, leader = __ffs(idle) - 1;
      unsigned base = 0;
      if (lane == leader) base = atomicAdd(fetch, (unsigned)__popc(idle));
      base = __shfl_sync(0xffffffffu, base, leader);
      next = base + __popc(idle);
      const unsigned idx = base + __popc(idle & lanemask_lt());
      if (!open && idx < total) {
        unsigned k;
        if (idx < (LIST ? n_light : n_list)) {
          const unsigned r = idx / nk;
          k = idx - r * nk;
          slot = (size_t)r * w.cap + k;
        } else if (LIST && idx < n_list) {
          const unsigned loc = __float_as_uint(w.ra[(size_t)w.nL * w.cap + (idx - n_light)].y);
          k = loc % (unsigned)w.cap;
          slot = (size_t)w.nL * w.cap + loc;
        } else {
          k = idx - n_list;
          slot = (size_t)(w.nL + w.nB) * w.cap + k;
        }
        sc = scenes + (w.one_scene >= 0 ? w.one_scene : views[w.view[w.qs[k]]].scene);
        const float4 o = w.ro[slot], dd = w.rd[slot];
        // a bounded ray stops at the first hit short of its light: a light sample's target, or
        // the closest light triangle along a BSDF sample
        float tmax = o.w;
        if (!LIST && idx >= n_light && idx < n_list) tmax = mis_light_bound(*sc, xyz(o), xyz(dd));
        const bool none = tmax < 0.f;
        if (none) tmax = INFINITY;
        const float t_occ = idx < n_light ? (tmax - 4e-3f) / 1.0001f - 4e-3f : (tmax < INFINITY ? tmax : -INFINITY);
        mem.set_ray(ray_pre(xyz(o), xyz(dd)));
        trav_begin(s, xyz(o), xyz(dd), tmax, t_occ, sc->ntri > 0 && !none ? sc->root : kNoNode);
        nodes = sc->nodes;
        leaf = sc->leaf;
        open = true;
      }
      continue;
    }
    if (idle == 0xffffffffu) break;
    trav_step(0xffffffffu, nodes, leaf, s, kTmin, mem, sc->err);
  }
}

// ------------------------------------------------------------------ accumulate kernel
// Per shaded path: the depth's contribution C (light samples + MIS-weighted BSDF
// samples, path_integrator.cc:103-160) and throughput factor beta (indirect bounce,
// :163-181). FWD folds them into L and T; REPLAY also stores the hit records and
// (C, beta) of the depth, which is all the adjoint needs besides the sampler stream.
template <int MODE, bool BSDF>
__global__ void __launch_bounds__(256) k_accum(WF w, const DevScene* __restrict__ scenes,
                                               const DevView* __restrict__ views, int d) {
  const int n = w.cnt[2 * d + 1];
  int* qout = (d & 1) ? w.q0 : w.q1;
  if (blockIdx.x == 0 && threadIdx.x == 0) w.cnt[2 * w.D + 3] = 0;  // listed rays of k_shade
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const bool last = d == w.D - 1;
  const float fL = (float)w.nL, fB = (float)w.nB;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n32; k += stride) {
    bool cont = false;
    int s = -1;
    if (k < n) {
      s = w.qs[k];
      const DevScene& sc = scenes[views[w.view[s]].scene];
      const size_t cs = (size_t)w.cap;
      const float4 c = w.cur[s];
      const Surf x = make_surf(sc, __float_as_int(c.x), c.y, c.z, xyz(w.org[s]));
      const DevObj& ob = sc.objs[x.obj];
      const float3 color = tex_rgb(ob.color, texel_offset(ob.color, x.u, x.v));
      const float3 bsdf = color * kInvPi;
      // DiffuseBsdfMaterial: the value depends on the outgoing direction
      const bool rough = BSDF && ob.mat == kMatDiffuseBsdf;
      float3 Ns = x.n;
      float sigma = 0.f;
      if (rough) {
        float3 mm;
        bool mapped;
        Ns = shading_normal(ob, x, mm, mapped);
        sigma = material_sigma(ob, x);
      }
      auto fr = [&](float3 L) { return rough ? bsdf_value(ob, color, sigma, Ns, x.wi, L) : bsdf; };
      float3 C = f3(0.f, 0.f, 0.f), beta = f3(0.f, 0.f, 0.f);
      for (int i = 0; i < w.nL; ++i) {
        const float4 h = w.hit[i * cs + k];
        const int tri = __float_as_int(h.x);
        if (tri < 0) continue;
        const float4 dd = w.rd[i * cs + k], aux = w.ra[i * cs + k];
        const float3 dir = xyz(dd);
        const Surf q = make_surf(sc, tri, h.y, h.z, x.p);
        if (!(q.is_light && sqnorm(q.p - xyz(aux)) < kEps)) continue;
        const DevLight& Lt = sc.lights[__float_as_int(dd.w)];
        const float tmp = dot(q.n, -dir) / q.sqd;
        const float G = dot(x.n, dir) * tmp;
        const float pdf_l = aux.w;
        float wgt = 1.0f / fL;
        if (w.nB > 0) wgt *= mis_power(pdf_l, dot(x.n, dir) * kInvPi * tmp, fL, fB);
        const float3 f = fr(dir);
        C += mul(light_emit<BSDF>(Lt, q), f) * (G / pdf_l * wgt);
      }
      for (int j = 0; j < w.nB; ++j) {
        const size_t slot = (w.nL + j) * cs + k;
        const float4 h = w.hit[slot];
        const int tri = __float_as_int(h.x);
        if (tri < 0) continue;
        const float3 wo = xyz(w.rd[slot]);
        const float ct = w.ra[slot].x;
        const Surf q = make_surf(sc, tri, h.y, h.z, x.p);
        if (!q.is_light) continue;
        const DevLight& Lt = sc.lights[q.light];
        const float tmp = dot(q.n, -wo) / q.sqd;
        const float G = dot(x.n, wo) * tmp;
        const float pdf_b = ct * kInvPi * tmp;
        float wgt = 1.0f / fB;
        if (w.nL > 0) wgt *= mis_power(pdf_b, __ldg(sc.light_pmf + q.light) * Lt.inv_area, fB, fL);
        const float3 f = fr(wo);
        C += mul(light_emit<BSDF>(Lt, q), f) * (G / pdf_b * wgt);
      }
      float4 hn = make_float4(__int_as_float(-1), 0.f, 0.f, 0.f);
      bool more = false;  // the next depth shades the path
      if (!last) {
        const size_t slot = (w.nL + w.nB) * cs + k;
        hn = w.hit[slot];
        const int tri = __float_as_int(hn.x);
        if (tri >= 0) {
          const float3 wo = xyz(w.rd[slot]);
          const float ct = w.ra[slot].x;
          const Surf nx = make_surf(sc, tri, hn.y, hn.z, x.p);
          const float tmp = dot(nx.n, -wo) / nx.sqd;
          const float G = dot(x.n, wo) * tmp;
          const float pdf = ct * kInvPi * tmp;
          beta = fr(wo) * (G / pdf);
          w.cur[s] = hn;
          w.org[s] = make_float4(x.p.x, x.p.y, x.p.z, 0.f);
          cont = true;
          more = !nx.is_light;
        }
      }
      if (MODE != MODE_FWD) {
        const int Rd = last ? w.R - 1 : w.R;
        for (int r = 0; r < Rd; ++r) rec_hit(w, s, d, r) = w.hit[r * cs + k];
        rec_c(w, s, d) = make_float4(C.x, C.y, C.z, 0.f);
        rec_beta(w, s, d) = make_float4(beta.x, beta.y, beta.z, 0.f);
        // a path that is not shaded again: nothing comes from the depths it does not reach (the
        // records of paths that miss the scene, or see a light, are never read past the first)
        if (!more) {
          for (int q = d + 1; q < w.D; ++q) {
            rec_c(w, s, q) = make_float4(0.f, 0.f, 0.f, 0.f);
            rec_beta(w, s, q) = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      }
      if (MODE != MODE_REPLAY) {
        const float3 T = xyz(w.T[s]);
        const float3 L = xyz(w.L[s]) + mul(T, C);
        const float3 Tn = mul(T, beta);
        w.T[s] = make_float4(Tn.x, Tn.y, Tn.z, 0.f);
        w.L[s] = make_float4(L.x, L.y, L.z, 0.f);
      }
    }
    const int kk = warp_append(&w.cnt[2 * (d + 1)], cont);
    if (cont) qout[kk] = s;
  }
}

// ------------------------------------------------------------------ film
// Per pixel: sum of its spp path radiances (non-finite paths count as 0), / spp,
// then the n_pass average of identical passes (path_integrator.cc:381-406).
__global__ void k_film(WF w, const DevView* __restrict__ views, Tile tile, int n_pass, float* samples_out) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < tile.npix; p += gridDim.x * blockDim.x) {
    const long long gp = tile.pix_begin + p;
    const int v = find_view_pix(views, w.nviews, gp);
    const DevView& V = views[v];
    const long long lp = gp - V.pix_off;
    const long long s0 = V.sample_off + lp * V.spp - tile.begin;
    float3 acc = f3(0.f, 0.f, 0.f);
    for (int k = 0; k < V.spp; ++k) {
      const long long s = s0 + k;
      float3 L = xyz(w.L[s]);
      if (!finite3(L)) L = f3(0.f, 0.f, 0.f);
      if (samples_out) {
        samples_out[3 * (lp * V.spp + k)] = L.x;
        samples_out[3 * (lp * V.spp + k) + 1] = L.y;
        samples_out[3 * (lp * V.spp + k) + 2] = L.z;
      }
      acc += L;
    }
    float3 val = acc / (float)V.spp;
    if (n_pass > 1) {
      float3 a = f3(0.f, 0.f, 0.f);
      for (int i = 0; i < n_pass; ++i) a += val;
      val = a / (float)n_pass;
    }
    if (V.image) {
      float* o = V.image + 3 * lp;
      o[0] = val.x; o[1] = val.y; o[2] = val.z;
    }
  }
}

// ------------------------------------------------------------------ adjoint helpers
struct SurfAdj {
  float3 p, n, t;
  float area;
};
PSDR_D SurfAdj zero_adj() {
  SurfAdj a;
  a.p = a.n = a.t = f3(0.f, 0.f, 0.f);
  a.area = 0.f;
  return a;
}

// A lane's own sums (own_add3) of the gradients that most of its paths share: the vertices of
// the scene's only light (DevScene::light_nv) and the emission of its first kHotLights lights.
// They belong to one scene; a lane that goes on to another scene's paths adds them to the
// accumulators first. (In jobs with several scenes the emission gradients used to go to the
// accumulators one by one, every lane of the GPU adding to the same few words: a 9-view step
// over three scenes took 67.2 ms, 51.5 with sums per lane.) Against fp32 sums, which lose small
// terms and depend on how paths are dealt to lanes, the exact ones cost k_adjoint up to 5 % (489
// and 510 us, 250^2 x 16 spp with every gradient; 2.78 and 2.75 ms, 512^2 x 32 spp with vertices)
// and k_adjoint_ext 1 to 7 % (2.85 and 3.04 ms, 377 x 97 x 96 spp). Only the sums in use are cleared
// and flushed: all 36 of a lane, at each change of scene too, took 1 to 3 % more.
constexpr int kHotLights = 4;
constexpr int kHotEmit = 3 * kMaxLightVerts;  // first emission sum
constexpr int kHotSums = kHotEmit + 3 * kHotLights;
struct HotAcc {
  const DevScene* sc;
  int lv0, nlv;  // light vertex range; nlv = 0: none
  int nlt;       // lights whose emission gradient is summed here
  bool high;     // hi is in use (large contributions, carries)
  long long lo[kHotSums], hi[kHotSums];
};
PSDR_D void hot_init(HotAcc& hot) {
  hot.sc = nullptr;
  hot.lv0 = hot.nlv = hot.nlt = 0;
  hot.high = false;
}
static __device__ __noinline__ void hot_carry(HotAcc& hot, int k, float3 v) {
  if (!hot.high) {
    for (int q = 0; q < kHotSums; ++q) hot.hi[q] = 0;
    hot.high = true;
  }
  hot.lo[k] = own_carry(hot.lo[k], hot.hi + k, v.x);
  hot.lo[k + 1] = own_carry(hot.lo[k + 1], hot.hi + k + 1, v.y);
  hot.lo[k + 2] = own_carry(hot.lo[k + 2], hot.hi + k + 2, v.z);
}
// Adds v to sums k, k + 1, k + 2 (a dynamic index: the sums live in local memory, L1).
PSDR_D void hot_add(HotAcc& hot, int k, float3 v) {
  if (!own_add3(hot.lo + k, v)) hot_carry(hot, k, v);
}
PSDR_D GradAcc* hot_target(const HotAcc& hot, int k) {
  if (k < kHotEmit) return hot.sc->grad_verts + 3 * (size_t)hot.lv0 + k;
  GradAcc* e = hot.sc->lights[(k - kHotEmit) / 3].grad_emit;
  return e ? e + (k - kHotEmit) % 3 : nullptr;
}
// Calls f(sum) for the sums in use.
template <class F>
PSDR_D void hot_each(const HotAcc& hot, F f) {
  for (int k = 0; k < 3 * hot.nlv; ++k) f(k);
  for (int k = kHotEmit; k < kHotEmit + 3 * hot.nlt; ++k) f(k);
}
static __device__ __noinline__ void hot_spill(HotAcc& hot) {
  if (!hot.sc) return;
  hot_each(hot, [&](int k) {
    const long long hi = hot.high ? hot.hi[k] : 0;
    if (hi | hot.lo[k]) acc_put(hot_target(hot, k), hi, hot.lo[k]);
  });
  hot_init(hot);
}
static __device__ __noinline__ void hot_rebind(HotAcc& hot, const DevScene* sc) {
  hot_spill(hot);
  hot.sc = sc;
  hot.lv0 = sc->light_v0;
  hot.nlv = sc->light_nv > 0 && vert_wanted(*sc, sc->light_v0) ? sc->light_nv : 0;
  hot.nlt = min(sc->nlight, kHotLights);
  hot_each(hot, [&](int k) { hot.lo[k] = 0; });
}
PSDR_D void hot_bind(HotAcc& hot, const DevScene* sc) {
  if (hot.sc != sc) hot_rebind(hot, sc);
}
// End of a kernel (all lanes together): one addition per warp when its lanes share the scene.
PSDR_D void hot_flush(HotAcc& hot) {
  const unsigned have = __ballot_sync(0xffffffffu, hot.sc != nullptr);
  if (!have) return;
  const unsigned long long own = (unsigned long long)hot.sc;
  const unsigned long long first = __shfl_sync(0xffffffffu, own, __ffs(have) - 1);
  if (!__all_sync(0xffffffffu, !own || own == first)) {
    hot_spill(hot);
    return;
  }
  if (!own) hot_bind(hot, reinterpret_cast<const DevScene*>(first));
  hot_each(hot, [&](int k) {
    if (GradAcc* to = hot_target(hot, k)) acc_put_warp(to, hot.high ? hot.hi[k] : 0, hot.lo[k]);
  });
}

// Adjoint ae of an environment light's radiance at box uv (u, v), incoming direction wi:
// scatters into the cube-map texel or the SH coefficients and returns the adjoint of wi.
static __device__ __noinline__ float3 env_emit_adj(const DevLight* L, float u, float v, float3 wi, float3 ae) {
  if (L->kind == kLightEnv) {
    if (L->tex.grad) atomic_add3(L->tex.grad + texel_offset(L->tex, u, v), ae);
    return f3(0.f, 0.f, 0.f);
  }
  float Y[9];
  sh9_basis(wi, Y);
  float s[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    if (L->grad_sh) atomic_add3(L->grad_sh + 3 * k, ae * Y[k]);
    s[k] = ae.x * L->sh[3 * k] + ae.y * L->sh[3 * k + 1] + ae.z * L->sh[3 * k + 2];
  }
  const float x = wi.x, y = wi.y, z = wi.z;
  return f3(kSh1 * s[3] + kSh2 * (s[4] * y + s[7] * z) - 2.f * kSh3 * s[6] * x + 2.f * kSh4 * s[8] * x,
            kSh1 * s[1] + kSh2 * (s[4] * x + s[5] * z) - 2.f * kSh3 * s[6] * y - 2.f * kSh4 * s[8] * y,
            kSh1 * s[2] + kSh2 * (s[5] * y + s[7] * x) + 4.f * kSh3 * s[6] * z);
}

// Emission adjoint of light hit q reached from x: area lights into the emission
// accumulator, environment lights into their parameters, and the SH9 direction's share
// into the point x (wi = -normalize(q - x)).
PSDR_D void add_emit(const DevScene& sc, HotAcc& hot, int light, float3 a) {
  GradAcc* to = sc.lights[light].grad_emit;
  if (!to) return;
  if (light < hot.nlt) hot_add(hot, kHotEmit + 3 * light, a);
  else atomic_add3(to, a);
}

template <bool EXT>
PSDR_D void add_light_emit(const DevScene& sc, HotAcc& hot, int light, const Surf& q, float3 ae, SurfAdj& ax) {
  const DevLight& Lt = sc.lights[light];
  if (!EXT || Lt.kind == kLightArea) {
    add_emit(sc, hot, light, ae);
    return;
  }
  const float3 aw = env_emit_adj(&Lt, q.u, q.v, q.wi, ae);
  if (Lt.kind == kLightSh9) ax.p += (aw - q.wi * dot(q.wi, aw)) / sqrtf(q.sqd);
}

PSDR_D void add_vertex(const DevScene& sc, HotAcc& hot, int v, float3 a) {
  if (!sc.grad_verts) return;
  const int rel = v - hot.lv0;
  if (hot.nlv > 0 && rel >= 0 && rel < hot.nlv) {
    hot_add(hot, 3 * rel, a);
    return;
  }
  vert_add(sc, v, a);
}

// Adjoint of Scene::hit's surface attributes (point, flipped normal and tangent,
// area) w.r.t. the triangle vertices (mesh.cc:27-67; area via |cross|/2, the same
// function as Heron's formula).
static __device__ __noinline__ void surf_vertex_adj(const DevScene& sc, int tri, float b1, float b2, bool front,
                                                    const SurfAdj& a, float3& g0, float3& g1, float3& g2) {
  const float4* r = sc.tri + 6 * (size_t)tri;
  const float4 q0 = __ldg(r), q1 = __ldg(r + 1), q2 = __ldg(r + 2), q3 = __ldg(r + 3), q5 = __ldg(r + 5);
  const float3 p0 = xyz(q0), p1 = xyz(q1), p2 = xyz(q2);
  const float sgn = front ? 1.f : -1.f;
  g0 = a.p * (1.f - b1 - b2);
  g1 = a.p * b1;
  g2 = a.p * b2;
  const float3 c = p1 - p0, b = p0 - p2;
  const float3 cr = cross(c, b);
  const float crn = norm(cr);
  const float3 n = cr / crn;
  const float3 an = a.n * sgn;
  float3 acr = (an - n * dot(n, an)) / crn + n * (0.5f * a.area);
  // tangent
  const float du1y = q5.x - q3.w, du2y = q5.z - q3.w;
  const float3 tw = c * du2y + b * du1y;
  const float twn = norm(tw);
  const float3 t = tw / twn;
  const float3 at = a.t * sgn;
  const float3 atw = (at - t * dot(t, at)) / twn;
  float3 ac = cross(b, acr) + atw * du2y;
  float3 ab = cross(acr, c) + atw * du1y;
  g1 += ac; g0 -= ac;
  g0 += ab; g2 -= ab;
}

PSDR_D void scatter_surf(const DevScene& sc, HotAcc& hot, int tri, float b1, float b2, bool front,
                         const SurfAdj& a) {
  if (!sc.grad_verts) return;
  const int4 tv = __ldg(sc.tri_v + tri);
  if (!vert_wanted(sc, tv.x) && !vert_wanted(sc, tv.y) && !vert_wanted(sc, tv.z)) return;
  float3 g0, g1, g2;
  surf_vertex_adj(sc, tri, b1, b2, front, a, g0, g1, g2);
  add_vertex(sc, hot, tv.x, g0);
  add_vertex(sc, hot, tv.y, g1);
  add_vertex(sc, hot, tv.z, g2);
}

// scatter_surf for a triangle that is not a light's: path vertices past the camera hit
// (paths end at lights), whose vertices never fall in the light-vertex register range.
// Out of line: the adjoint scatters from several depths' call sites.
PSDR_D void scatter_verts(const DevScene& sc, int tri, float b1, float b2, bool front, const SurfAdj& a) {
  if (!sc.grad_verts) return;
  const int4 tv = __ldg(sc.tri_v + tri);
  if (!vert_wanted(sc, tv.x) && !vert_wanted(sc, tv.y) && !vert_wanted(sc, tv.z)) return;
  float3 g0, g1, g2;
  surf_vertex_adj(sc, tri, b1, b2, front, a, g0, g1, g2);
  vert_add(sc, tv.x, g0);
  vert_add(sc, tv.y, g1);
  vert_add(sc, tv.z, g2);
}
static __device__ __noinline__ void scatter_mesh(const DevScene& sc, int tri, float b1, float b2, bool front, SurfAdj a) {
  scatter_verts(sc, tri, b1, b2, front, a);
}

PSDR_D void scatter_tex(const DevTex& tx, int off, float3 a, bool /*unused*/) {
  if (!tx.grad) return;
  if (tx.ch == 1) acc_add(tx.grad + off, a.x + a.y + a.z);
  else atomic_add3(tx.grad + off, a);
}

// Adjoint of G = dot(Nx, w) dot(Nq, -w) / d2 with d2 = |q - x|^2, w given.
PSDR_D void geom_adj(float adjG, float3 Nx, float3 Nq, float3 w, float3 xp, float3 qp, float d2, float G,
                     SurfAdj& ax, SurfAdj& aq, float3& adj_w) {
  const float a = dot(Nx, w), bq = -dot(Nq, w);
  const float adj_a = adjG * bq / d2, adj_b = adjG * a / d2, adj_d2 = -adjG * G / d2;
  ax.n += w * adj_a;
  aq.n += w * (-adj_b);
  adj_w = Nx * adj_a - Nq * adj_b;
  const float3 dq = (qp - xp) * (2.f * adj_d2);
  aq.p += dq;
  ax.p -= dq;
}

// Adjoint of wo = normalize(u T + v B + ct N), B = N x T, w.r.t. N and T.
PSDR_D void dir_adj(float3 adj_wo, float3 wo, float3 N, float3 T, float u, float v, float ct, SurfAdj& ax) {
  const float3 B = cross(N, T);
  const float3 m = T * u + B * v + N * ct;
  const float3 am = (adj_wo - wo * dot(wo, adj_wo)) / norm(m);
  const float3 aB = am * v;
  ax.t += am * u + cross(aB, N);
  ax.n += am * ct + cross(T, aB);
}

// ------------------------------------------------------------------ material adjoints
// Material state of a shaded vertex (DiffuseBsdfMaterial, diffuse_bsdf.cc:3-88).
struct MatPt {
  float3 color;  // color texel
  float3 N;      // shading normal
  float3 m;      // normal-map vector 2 texel - 1
  float sigma;   // roughness texel
  bool rough, mapped;
};
PSDR_D MatPt mat_point(const DevObj& ob, const Surf& x) {
  MatPt mp;
  mp.color = tex_rgb(ob.color, texel_offset(ob.color, x.u, x.v));
  mp.rough = ob.mat == kMatDiffuseBsdf;
  mp.N = shading_normal(ob, x, mp.m, mp.mapped);
  mp.sigma = material_sigma(ob, x);
  return mp;
}

// Adjoints gathered at a vertex before they are folded into the surface and textures.
struct MatAdj {
  float3 color, N, V;
  float sigma;
};
PSDR_D MatAdj zero_mat_adj() {
  MatAdj a;
  a.color = a.N = a.V = f3(0.f, 0.f, 0.f);
  a.sigma = 0.f;
  return a;
}

// f = bsdf_value(color, sigma, N, V, L): returns f and accumulates the adjoints of
// color, sigma, N, V (ma) and L (adj_L) for the adjoint adj_f of f.
PSDR_D float3 bsdf_adj(const MatPt& mp, float3 V, float3 L, float3 adj_f, MatAdj& ma, float3& adj_L) {
  if (!mp.rough) {
    ma.color += adj_f * kInvPi;
    return mp.color * kInvPi;
  }
  const float a = 1.0f / (kPi + kOrenC * mp.sigma), b = mp.sigma * a;
  const float nlr = dot(mp.N, L), nvr = dot(mp.N, V);
  const float nl = fmaxf(nlr, 0.f), nv = fmaxf(nvr, 0.f);
  const float t0 = dot(V, L) - nl * nv;
  const float t = t0 > 0.f ? fmaxf(nl, nv) + kEps : t0;
  const float g = a + b * t;
  ma.color += adj_f * g;
  const float adj_g = dot(adj_f, mp.color);
  const float da = -kOrenC * a * a, db = a + mp.sigma * da;
  ma.sigma += adj_g * (da + db * t);
  const float adj_t = adj_g * b;
  float adj_nl = 0.f, adj_nv = 0.f;
  if (t0 > 0.f) {
    if (nl >= nv) adj_nl = adj_t;
    else adj_nv = adj_t;
  } else {
    adj_L += V * adj_t;
    ma.V += L * adj_t;
    adj_nl = -adj_t * nv;
    adj_nv = -adj_t * nl;
  }
  if (nlr >= 0.f) { ma.N += L * adj_nl; adj_L += mp.N * adj_nl; }
  if (nvr >= 0.f) { ma.N += V * adj_nv; ma.V += mp.N * adj_nv; }
  return mp.color * g;
}

// Adjoint of a sampled direction wo = normalize(u T + v B + ct N), B = Ng x T, about
// the shading normal N (its adjoint goes to adjN).
PSDR_D void dir_adj_mat(float3 adj_wo, float3 wo, const Surf& x, float3 N, float u, float v, float ct, SurfAdj& ax,
                        float3& adjN) {
  const float3 B = cross(x.n, x.t);
  const float3 m = x.t * u + B * v + N * ct;
  const float3 am = (adj_wo - wo * dot(wo, adj_wo)) / norm(m);
  const float3 aB = am * v;
  ax.t += am * u + cross(aB, x.n);
  ax.n += cross(x.t, aB);
  adjN += am * ct;
}

// Folds a vertex's material adjoints into its surface adjoint (shading normal through
// the normal map's frame, incoming direction into the point and the ray origin) and
// scatters the roughness and normal-map texel adjoints. Returns the ray origin's adjoint.
PSDR_D float3 mat_finalize(const DevObj& ob, const Surf& x, const MatPt& mp, const MatAdj& ma, SurfAdj& ax) {
  if (mp.mapped) {
    const float3 B = cross(x.n, x.t);
    const float3 nn = x.t * mp.m.x + B * mp.m.y + x.n * mp.m.z;
    const float3 am = (ma.N - mp.N * dot(mp.N, ma.N)) / norm(nn);
    const float3 aB = am * mp.m.y;
    ax.t += am * mp.m.x + cross(aB, x.n);
    ax.n += am * mp.m.z + cross(x.t, aB);
    if (ob.normal.grad)
      atomic_add3(ob.normal.grad + texel_offset(ob.normal, x.u, x.v), f3(dot(am, x.t), dot(am, B), dot(am, x.n)) * 2.f);
  } else {
    ax.n += ma.N;
  }
  if (mp.rough && ob.rough.grad && ma.sigma != 0.f)
    acc_add(ob.rough.grad + texel_offset(ob.rough, x.u, x.v), ma.sigma);
  // V = -normalize(x.p - o)
  const float3 au = (ma.V - x.wi * dot(x.wi, ma.V)) * (-1.f / sqrtf(x.sqd));
  ax.p += au;
  return -au;
}

// Adjoint of a BSDF-sampled segment's G in the unbiased estimator: the direction is
// that of the segment's end points, w = normalize(q - x), so it back-propagates into
// both points instead of the sampling frame.
PSDR_D void geom_adj_points(float adjG, const Surf& x, const Surf& q, SurfAdj& ax, SurfAdj& aq,
                            float3 adj_w_extra = f3(0.f, 0.f, 0.f)) {
  const float3 rv = q.p - x.p;
  const float rn = norm(rv);
  const float3 wg = rv / rn;
  const float G = dot(x.n, wg) * (dot(q.n, -wg) / q.sqd);
  float3 adj_w;
  geom_adj(adjG, x.n, q.n, wg, x.p, q.p, q.sqd, G, ax, aq, adj_w);
  adj_w += adj_w_extra;
  const float3 ar = (adj_w - wg * dot(wg, adj_w)) / rn;
  aq.p += ar;
  ax.p -= ar;
}

// The adjoint of one depth of trace2light in three parts: a light sample, a BSDF sample and the
// continuation, each recomputed from its two sampler draws (rx, ry) and its hit record h.
// They back-propagate adjC (of the depth's contribution) or adjB (of its throughput factor)
// into the surface x (ax), the color texel (adj_tex), the emission and the light vertices.
// UNB (unbiased estimator): BSDF-sampled segments differentiate G through their end
// points (geom_adj_points); the reference differentiates it through the sampled
// direction's frame.
// BSDF (DiffuseBsdfMaterial in the scene): the BSDF value depends on the shading normal
// (mp), the incoming direction x.wi and the outgoing direction; their adjoints and the
// color / roughness adjoints gather in ma (adj_tex is unused).
// VERTS: some vertex gradient is wanted; without it only the texel and emission adjoints are
// formed (a material of direction-dependent value also passes adjoints on through
// directions, so its kernel always has VERTS).
template <bool BSDF, bool VERTS>
PSDR_D void light_sample_adj(const WF& w, const DevScene& sc, const Surf& x, float3 bsdf, float rx, float ry, float4 h,
                             float3 adjC, SurfAdj& ax, HotAcc& hot, float3& adj_tex, const MatPt* mp, MatAdj* ma) {
  const int tri = __float_as_int(h.x);
  if (tri < 0) return;
  const float fL = (float)w.nL, fB = (float)w.nB;
  const LightSample ls = sample_light(sc, rx, ry);
  const float3 rv = ls.y - x.p;
  const float3 dir = normalize(rv);
  const Surf q = make_surf(sc, tri, h.y, h.z, x.p);
  if (!(q.is_light && sqnorm(q.p - ls.y) < kEps)) return;
  const DevLight& Lt = sc.lights[ls.light];
  const float3 emit = light_emit<BSDF>(Lt, q);
  const float tmp = dot(q.n, -dir) / q.sqd;
  const float G = dot(x.n, dir) * tmp;
  float wgt = 1.0f / fL;
  if (w.nB > 0) wgt *= mis_power(ls.pdf, dot(x.n, dir) * kInvPi * tmp, fL, fB);
  const float3 av = adjC * wgt;
  const float s_ = G / ls.pdf;
  float3 adjL = f3(0.f, 0.f, 0.f);
  float3 f = bsdf;
  if (BSDF) f = bsdf_adj(*mp, x.wi, dir, mul(av, emit) * s_, *ma, adjL);
  else adj_tex += mul(av, emit) * (s_ * kInvPi);
  const float3 eb = mul(emit, f);
  const float3 ae = mul(av, f) * s_;
  add_light_emit<BSDF>(sc, hot, ls.light, q, ae, ax);
  if (!VERTS) return;
  const float adj_gam = dot(av, eb) / ls.pdf;
  SurfAdj aq = zero_adj();
  aq.area = adj_gam * G / q.area;
  float3 adj_dir;
  geom_adj(adj_gam, x.n, q.n, dir, x.p, q.p, q.sqd, G, ax, aq, adj_dir);
  if (BSDF) adj_dir += adjL;
  const float3 ar = (adj_dir - dir * dot(dir, adj_dir)) / norm(rv);
  ax.p -= ar;
  // light sample point y = p0 + (p1-p0) su + (p2-p0) sv
  if (sc.grad_verts) {
    const int4 tv = __ldg(sc.tri_v + ls.tri);
    add_vertex(sc, hot, tv.x, ar * (1.f - ls.su - ls.sv));
    add_vertex(sc, hot, tv.y, ar * ls.su);
    add_vertex(sc, hot, tv.z, ar * ls.sv);
  }
  scatter_surf(sc, hot, tri, h.y, h.z, q.front, aq);
}

template <bool UNB, bool BSDF, bool VERTS>
PSDR_D void bsdf_sample_adj(const WF& w, const DevScene& sc, const Surf& x, float3 bsdf, float rx, float ry, float4 h,
                            float3 adjC, SurfAdj& ax, HotAcc& hot, float3& adj_tex, const MatPt* mp, MatAdj* ma) {
  const int tri = __float_as_int(h.x);
  if (tri < 0) return;
  const float fL = (float)w.nL, fB = (float)w.nB;
  const float3 Ns = BSDF ? mp->N : x.n;
  const Surf q = make_surf(sc, tri, h.y, h.z, x.p);
  if (!q.is_light) return;
  float ct, st, sp, cp;
  const float3 wo = BSDF ? material_dir(x, Ns, rx, ry, ct, st, sp, cp) : diffuse_dir(x.n, x.t, rx, ry, ct, st, sp, cp);
  const DevLight& Lt = sc.lights[q.light];
  const float3 emit = light_emit<BSDF>(Lt, q);
  const float tmp = dot(q.n, -wo) / q.sqd;
  const float G = dot(x.n, wo) * tmp;
  const float pdf_b = ct * kInvPi * tmp;
  float wgt = 1.0f / fB;
  if (w.nL > 0) wgt *= mis_power(pdf_b, __ldg(sc.light_pmf + q.light) * Lt.inv_area, fB, fL);
  const float3 av = adjC * wgt;
  const float s_ = G / pdf_b;
  // the BSDF's outgoing direction: the sampled one, or the segment's (unbiased)
  float3 adjL = f3(0.f, 0.f, 0.f);
  float3 f = bsdf;
  if (BSDF) f = bsdf_adj(*mp, x.wi, UNB ? normalize(q.p - x.p) : wo, mul(av, emit) * s_, *ma, adjL);
  else adj_tex += mul(av, emit) * (s_ * kInvPi);
  const float3 eb = mul(emit, f);
  const float3 ae = mul(av, f) * s_;
  add_light_emit<BSDF>(sc, hot, q.light, q, ae, ax);
  if (!VERTS) return;
  const float adj_gam = dot(av, eb) / pdf_b;
  SurfAdj aq = zero_adj();
  aq.area = adj_gam * G / q.area;
  if (UNB) {
    geom_adj_points(adj_gam, x, q, ax, aq, adjL);
  } else {
    float3 adj_wo;
    geom_adj(adj_gam, x.n, q.n, wo, x.p, q.p, q.sqd, G, ax, aq, adj_wo);
    if (BSDF) dir_adj_mat(adj_wo + adjL, wo, x, Ns, cp * st, sp * st, ct, ax, ma->N);
    else dir_adj(adj_wo, wo, x.n, x.t, cp * st, sp * st, ct, ax);
  }
  scatter_surf(sc, hot, tri, h.y, h.z, q.front, aq);
}

// Returns false when the path ends here; otherwise carry = the adjoint of the next vertex nx,
// passed to the next depth.
template <bool UNB, bool BSDF, bool VERTS>
PSDR_D bool continuation_adj(const DevScene& sc, const Surf& x, float3 bsdf, float rx, float ry, float4 h, float3 adjB,
                             SurfAdj& ax, SurfAdj& carry, Surf& nx, float3& adj_tex, const MatPt* mp, MatAdj* ma) {
  const int tri = __float_as_int(h.x);
  if (tri < 0) return false;
  const float3 Ns = BSDF ? mp->N : x.n;
  float ct, st, sp, cp;
  const float3 wo = BSDF ? material_dir(x, Ns, rx, ry, ct, st, sp, cp) : diffuse_dir(x.n, x.t, rx, ry, ct, st, sp, cp);
  nx = make_surf(sc, tri, h.y, h.z, x.p);
  const float tmp = dot(nx.n, -wo) / nx.sqd;
  const float G = dot(x.n, wo) * tmp;
  const float pdf = ct * kInvPi * tmp;
  const float s_ = G / pdf;
  float3 adjL = f3(0.f, 0.f, 0.f);
  float3 f = bsdf;
  if (BSDF) f = bsdf_adj(*mp, x.wi, UNB ? normalize(nx.p - x.p) : wo, adjB * s_, *ma, adjL);
  else adj_tex += adjB * (s_ * kInvPi);
  if (!VERTS) return true;
  const float adj_gam = dot(adjB, f) / pdf;
  carry = zero_adj();
  carry.area = adj_gam * G / nx.area;
  if (UNB) {
    geom_adj_points(adj_gam, x, nx, ax, carry, adjL);
  } else {
    float3 adj_wo;
    geom_adj(adj_gam, x.n, nx.n, wo, x.p, nx.p, nx.sqd, G, ax, carry, adj_wo);
    if (BSDF) dir_adj_mat(adj_wo + adjL, wo, x, Ns, cp * st, sp * st, ct, ax, ma->N);
    else dir_adj(adj_wo, wo, x.n, x.t, cp * st, sp * st, ct, ax);
  }
  return true;
}

// Warp-aggregated scatter of a surface adjoint: reduced over the warp when every
// lane targets the same triangle of the same scene (the spp samples of a pixel).
PSDR_D void scatter_surf_warp(const DevScene* scp, HotAcc& hot, int tri, float b1, float b2, bool front,
                              const SurfAdj& a, bool active) {
  const int t0 = __shfl_sync(0xffffffffu, active ? tri : -1, 0);
  const unsigned long long p0 = __shfl_sync(0xffffffffu, (unsigned long long)scp, 0);
  const bool uni = __all_sync(0xffffffffu, active && tri == t0 && (unsigned long long)scp == p0);
  if (!uni) {
    if (active) scatter_surf(*scp, hot, tri, b1, b2, front, a);
    return;
  }
  if (!scp->grad_verts) return;
  {
    const int4 tv = __ldg(scp->tri_v + tri);
    if (!vert_wanted(*scp, tv.x) && !vert_wanted(*scp, tv.y) && !vert_wanted(*scp, tv.z)) return;
  }
  float3 g0, g1, g2;
  surf_vertex_adj(*scp, tri, b1, b2, front, a, g0, g1, g2);
  float v[9] = {g0.x, g0.y, g0.z, g1.x, g1.y, g1.z, g2.x, g2.y, g2.z};
#pragma unroll
  for (int o = 16; o; o >>= 1)
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if ((threadIdx.x & 31) == 0) {
    const int4 tv = __ldg(scp->tri_v + tri);
    add_vertex(*scp, hot, tv.x, f3(v[0], v[1], v[2]));
    add_vertex(*scp, hot, tv.y, f3(v[3], v[4], v[5]));
    add_vertex(*scp, hot, tv.z, f3(v[6], v[7], v[8]));
  }
}

PSDR_D void scatter_tex_warp(const DevTex* tx, int off, float3 a, bool active) {
  const bool has = active && tx && tx->grad;
  const unsigned long long key = has ? (unsigned long long)(tx->grad + off) : 0ull;
  const unsigned long long k0 = __shfl_sync(0xffffffffu, key, 0);
  const bool uni = __all_sync(0xffffffffu, has && key == k0);
  if (!uni) {
    if (has) scatter_tex(*tx, off, a, false);
    return;
  }
  float v0 = a.x, v1 = a.y, v2 = a.z;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    v2 += __shfl_xor_sync(0xffffffffu, v2, o);
  }
  if ((threadIdx.x & 31) == 0) scatter_tex(*tx, off, f3(v0, v1, v2), false);
}

// ------------------------------------------------------------------ adjoint kernels
// The records hold each depth's contribution C_d and throughput factor beta_d, so the suffix
// radiances S_d = C_d + beta_d S_{d+1} come straight from them; every path's vertices are then
// visited from the camera on, replaying its sampler stream, and every depth's reverse-mode
// adjoint is applied (PSDR_EST_REFERENCE: pdfs and MIS weights are constants, jacobi =
// area/detach(area), barycentrics are not differentiated), scattering into the fixed-point
// accumulators: k_adjoint, from per-warp lists, and k_adjoint_ext, one thread per path.
PSDR_D float3 suffix_radiance(const WF& w, int s, int from) {
  float3 S = f3(0.f, 0.f, 0.f);
  for (int k = w.D - 1; k >= from; --k) S = xyz(rec_c(w, s, k)) + mul(xyz(rec_beta(w, s, k)), S);
  return S;
}

// Camera-origin adjoint summed per lane while consecutive samples share a view.
struct CamAcc {
  const DevView* v = nullptr;
  GradAcc* to = nullptr;  // its accumulators or null
  Own3 g;
  PSDR_D void add(const DevView* view, float3 a) {
    if (view != v) {
      flush();
      v = view;
      to = view->grad_pos;
    }
    if (to) g.add(a);
  }
  PSDR_D void flush() {
    if (to) {
      g.put(to);
      g = Own3();
    }
    v = nullptr;
    to = nullptr;
  }
  // End of a kernel: one addition per warp when the warp shares the view.
  PSDR_D void flush_warp() {
    const unsigned long long key = (unsigned long long)to;
    const unsigned long long k0 = __shfl_sync(0xffffffffu, key, 0);
    if (!__all_sync(0xffffffffu, key == k0)) { flush(); return; }
    if (to) g.put_warp(to);
  }
};

// Viewing direction (camera -z axis in world space) and fx*fy of the map from world
// directions to raster coordinates: the camera's right and up axes are not normalised
// (camera.h:7-40), so c2r's scale is multiplied by the norms of w2c's first two rows.
PSDR_D float3 view_look(const DevView& V) { return f3(-V.c2w[2], -V.c2w[6], -V.c2w[10]); }
PSDR_D float view_fxfy(const DevView& V) {
  const float r0 = sqrtf(V.w2c[0] * V.w2c[0] + V.w2c[1] * V.w2c[1] + V.w2c[2] * V.w2c[2]);
  const float r1 = sqrtf(V.w2c[4] * V.w2c[4] + V.w2c[5] * V.w2c[5] + V.w2c[6] * V.w2c[6]);
  return fabsf(V.c2r[0] * V.c2r[5]) * r0 * r1;
}

// Unbiased estimator, primary vertex: adjoint of the camera Jacobian ratio J/detach(J),
// J = |n.(x-o)| / z^3, z = (x-o).look, scaled by phi = dot(dI, L). Returns the camera origin's share.
PSDR_D float3 cam_jacobian_adj(const DevView& V, const Surf& x, float phi, SurfAdj& ax) {
  if (V.ortho) {
    // J = |n.look|: only the normal moves it
    const float3 look = view_look(V);
    ax.n += look * (phi / dot(x.n, look));
    return f3(0.f, 0.f, 0.f);
  }
  const float3 rel = x.p - V.pos;
  const float nr = dot(x.n, rel);
  const float3 look = view_look(V);
  const float z = dot(rel, look);
  ax.n += rel * (phi / nr);
  const float3 ap = x.n * (phi / nr) - look * (3.f * phi / z);
  ax.p += ap;
  return -ap;
}

// The camera end of a path (depth 0): its view, primary surface and pixel gradient.
// Returns false when the path contributes nothing (missed the scene, no image gradient).
PSDR_D bool primary_point(const WF& w, const DevScene* __restrict__ scenes, const DevView* __restrict__ views,
                          const Tile& tile, int s, const DevView*& Vp, const DevScene*& scp, float4& h0, float3& g,
                          Surf& x0, float3& o0) {
  const DevView& V = views[w.view[s]];
  Vp = &V;
  scp = &scenes[V.scene];
  h0 = rec_at(w, s, 0);
  const int tri0 = __float_as_int(h0.x);
  if (tri0 < 0 || !V.dimage) return false;
  const float* gp = V.dimage + 3 * (size_t)w.pix[s];
  g = f3(gp[0], gp[1], gp[2]) / (float)V.spp;
  o0 = V.pos;
  if (V.ortho) {
    // the camera ray's origin on the camera plane, as k_camera formed it
    Rng r0 = make_rng((unsigned long long)(tile.begin + s - V.sample_off) + w.seed);
    const float jx = r0.next_float(), jy = r0.next_float();
    const int pix = w.pix[s];
    float3 pc;
    xform_pos(V.r2c, f3(jx + (float)(pix % V.W), jy + (float)(pix / V.W), 1.0f), pc);
    xform_pos(V.c2w, f3(pc.x, pc.y, 0.f), o0);
  }
  x0 = make_surf(*scp, tri0, h0.y, h0.z, o0);
  return true;
}

// Work lists of one warp of k_adjoint in shared memory, field by field (a column per entry).
// Path vertices past the first: path, depth, ray origin, throughput, sampler, carried adjoint.
// BSDF samples that hit a light: path, depth, sample, draws, ray origin, adjoint of C.
constexpr int kVertCap = 64;     // at most 31 waiting + 32 new
constexpr int kVertFields = 22;
constexpr int kHitFields = 11;
constexpr int kAdjWarps = 8;
__host__ __device__ constexpr int adj_hit_cap(int nB) { return 32 + 32 * (nB > 0 ? nB : 1); }
__host__ __device__ constexpr int adj_warp_words(int nB) { return kVertFields * kVertCap + kHitFields * adj_hit_cap(nB); }

// Adjoint of the interior paths of a tile (DiffuseMaterial scenes). A warp takes 32 paths at
// their camera vertices; the vertices they go on to, and the BSDF samples that hit a light
// (about one in twenty), go to the warp's lists and are worked on 32 at a time. Walking
// each path to its end instead (one thread per path over all depths) ran every depth's code
// for the few paths still alive, and the BSDF-sample code for two lanes of a warp on average:
// 5.8 ms per 512^2 x 32 spp x depth 3 step against 2.9 ms with lists; 2.3 ms with the warps of a
// block starting together (2.8 ms in tiles of 2^22 paths whose records lie in HBM, with fp32
// or with exact sums per thread). Bound by the latency of its record loads (5.9 cycles
// per issued instruction at 24 % occupancy, 128 registers; DRAM 8 % busy); instruction fetch is
// down from 7.2 cycles to 1.3, for 3.0 at the block's barrier.
// Without vertex gradients (VERTS false: texture and emission optimisation) the lists carry no
// surface adjoint and the vertex scatters go; 256^2 x 64 spp: 0.83 -> 0.55 ms (three blocks per
// SM spill: 0.63 ms).
template <bool UNB, bool VERTS>
__global__ void __launch_bounds__(32 * kAdjWarps, 2) k_adjoint(WF w, const DevScene* __restrict__ scenes,
                                                               const DevView* __restrict__ views, Tile tile) {
  extern __shared__ float adj_lists[];
  const int lane = threadIdx.x & 31;
  float* vl = adj_lists + (threadIdx.x >> 5) * adj_warp_words(w.nB);
  const int hcap = adj_hit_cap(w.nB);
  float* hl = vl + kVertFields * kVertCap;
  auto vput = [&](int f, int e, float v) { vl[f * kVertCap + e] = v; };
  auto vget = [&](int f, int e) { return vl[f * kVertCap + e]; };
  auto hput = [&](int f, int e, float v) { hl[f * hcap + e] = v; };
  auto hget = [&](int f, int e) { return hl[f * hcap + e]; };
  int nv = 0, nh = 0;  // entries of the lists

  CamAcc cam;
  HotAcc hot;
  hot_init(hot);
  const int stride = gridDim.x * blockDim.x;
  int s0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31);  // first path of the warp's next 32
  while (true) {
    // The block's warps start each batch together: the kernel is bound by instruction fetch, and
    // warps that run the same code at the same time share it.
    const bool more = s0 < tile.n;
    if (!__syncthreads_or(more || nv > 0 || nh > 0)) break;
    if (nh >= 32 || (nh > 0 && nv == 0 && !more)) {
      // ---- BSDF samples that hit a light
      const int take = min(32, nh);
      nh -= take;
      if (lane < take) {
        const int e = nh + lane;
        const int s = __float_as_int(hget(0, e)), dj = __float_as_int(hget(1, e));
        const int d = dj >> 8, j = dj & 255;
        const float rx = hget(2, e), ry = hget(3, e);
        const float3 org = f3(hget(4, e), hget(5, e), hget(6, e)), adjC = f3(hget(7, e), hget(8, e), hget(9, e));
        const DevScene& sc = scenes[__float_as_int(hget(10, e))];
        hot_bind(hot, &sc);
        const float4 hx = d == 0 ? rec_at(w, s, 0) : rec_hit(w, s, d - 1, w.nL + w.nB);
        const int tri = __float_as_int(hx.x);
        const Surf x = make_surf(sc, tri, hx.y, hx.z, org);
        const DevObj& ob = sc.objs[x.obj];
        const int off = texel_offset(ob.color, x.u, x.v);
        SurfAdj ax = zero_adj();
        float3 atx = f3(0.f, 0.f, 0.f);
        bsdf_sample_adj<UNB, false, VERTS>(w, sc, x, tex_rgb(ob.color, off) * kInvPi, rx, ry,
                                    rec_hit(w, s, d, w.nL + j), adjC, ax, hot, atx, nullptr, nullptr);
        scatter_tex(ob.color, off, atx, false);
        if (VERTS) scatter_mesh(sc, tri, hx.y, hx.z, x.front, ax);
      }
      __syncwarp();
      continue;
    }
    const bool fresh = nv < 32 && more;
    if (!fresh && nv == 0) continue;
    bool act = false, has0 = false;  // act: a vertex to work on; has0: a fresh path with something to scatter
    int s = 0, d = 0, tri = -1;
    float4 hx = make_float4(0.f, 0.f, 0.f, 0.f);
    float3 g = f3(0.f, 0.f, 0.f), T = f3(1.f, 1.f, 1.f), org = f3(0.f, 0.f, 0.f);
    Rng rng{0, 0};
    SurfAdj ax = zero_adj();
    Surf x;
    x.front = true;
    const DevScene* scp = nullptr;
    if (fresh) {
      s = s0 + lane;
      s0 += stride;
      const DevView* Vp = nullptr;
      if (s < tile.n && primary_point(w, scenes, views, tile, s, Vp, scp, hx, g, x, org)) {
        const DevView& V = *Vp;
        tri = __float_as_int(hx.x);
        hot_bind(hot, scp);
        if (x.is_light) {
          // camera ray on a light: L = emit at depth 0 when lights are visible
          if (w.light_vis) {
            const DevLight& Lt = scp->lights[x.light];
            const float3 L = light_emit<false>(Lt, x);
            has0 = true;
            ax.area = dot(g, L) / x.area;
            if (UNB) cam.add(&V, cam_jacobian_adj(V, x, dot(g, L), ax));
            add_emit(*scp, hot, x.light, g);
          }
        } else {
          const float3 L = suffix_radiance(w, s, 0);
          if (finite3(L)) {
            act = has0 = true;
            rng = make_rng((unsigned long long)(tile.begin + s - V.sample_off) + w.seed);
            rng.next_float();
            rng.next_float();
            ax.area = dot(g, L) / x.area;  // jacobi of the primary hit
            if (UNB) cam.add(&V, cam_jacobian_adj(V, x, dot(g, L), ax));
          }
        }
      }
    } else {
      const int take = min(32, nv);
      nv -= take;
      if (lane < take) {
        const int e = nv + lane;
        act = true;
        s = __float_as_int(vget(0, e));
        d = __float_as_int(vget(1, e));
        org = f3(vget(2, e), vget(3, e), vget(4, e));
        T = f3(vget(5, e), vget(6, e), vget(7, e));
        rng.state = (unsigned long long)__float_as_uint(vget(8, e)) | (unsigned long long)__float_as_uint(vget(9, e)) << 32;
        rng.inc = (unsigned long long)__float_as_uint(vget(10, e)) | (unsigned long long)__float_as_uint(vget(11, e)) << 32;
        if (VERTS) {
          ax.p = f3(vget(12, e), vget(13, e), vget(14, e));
          ax.n = f3(vget(15, e), vget(16, e), vget(17, e));
          ax.t = f3(vget(18, e), vget(19, e), vget(20, e));
          ax.area = vget(21, e);
        }
        const DevView& V = views[w.view[s]];
        scp = &scenes[V.scene];
        hot_bind(hot, scp);
        const float* gp = V.dimage + 3 * (size_t)w.pix[s];
        g = f3(gp[0], gp[1], gp[2]) / (float)V.spp;
        hx = rec_hit(w, s, d - 1, w.nL + w.nB);
        tri = __float_as_int(hx.x);
        x = make_surf(*scp, tri, hx.y, hx.z, org);
      }
      __syncwarp();
    }
    const DevTex* tx = nullptr;
    int toff = 0;
    float3 atx = f3(0.f, 0.f, 0.f), bsdf = atx;
    const float3 adjC = mul(g, T);
    if (act) {
      tx = &scp->objs[x.obj].color;
      toff = texel_offset(*tx, x.u, x.v);
      bsdf = tex_rgb(*tx, toff) * kInvPi;
      for (int i = 0; i < w.nL; ++i) {
        const float rx = rng.next_float(), ry = rng.next_float();
        light_sample_adj<false, VERTS>(w, *scp, x, bsdf, rx, ry, rec_hit(w, s, d, i), adjC, ax, hot, atx, nullptr, nullptr);
      }
    }
    for (int j = 0; j < w.nB; ++j) {
      bool hit = false;
      float rx = 0.f, ry = 0.f;
      if (act) {
        rx = rng.next_float();
        ry = rng.next_float();
        const int t = __float_as_int(rec_hit(w, s, d, w.nL + j).x);
        hit = t >= 0 && scp->objs[__ldg(scp->tri_v + t).w].light >= 0;
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int e = nh + __popc(m & lanemask_lt());
        hput(0, e, __int_as_float(s));
        hput(1, e, __int_as_float(d << 8 | j));
        hput(2, e, rx);
        hput(3, e, ry);
        hput(4, e, org.x); hput(5, e, org.y); hput(6, e, org.z);
        hput(7, e, adjC.x); hput(8, e, adjC.y); hput(9, e, adjC.z);
        hput(10, e, __int_as_float((int)(scp - scenes)));
      }
      nh += __popc(m);
    }
    bool go = false;
    SurfAdj carry;
    Surf nx;
    if (act && d < w.D - 1) {
      const float rx = rng.next_float(), ry = rng.next_float();
      const float3 adjB = mul(adjC, suffix_radiance(w, s, d + 1));
      go = continuation_adj<UNB, false, VERTS>(*scp, x, bsdf, rx, ry, rec_hit(w, s, d, w.nL + w.nB), adjB, ax, carry, nx, atx,
                                        nullptr, nullptr) &&
           !nx.is_light;  // a path that ends on a light has nothing downstream
    }
    if (fresh) {
      if (VERTS) scatter_surf_warp(scp, hot, tri, hx.y, hx.z, x.front, ax, has0);
      scatter_tex_warp(tx, toff, atx, has0);
    } else if (act) {
      scatter_tex(*tx, toff, atx, false);
      if (VERTS) scatter_mesh(*scp, tri, hx.y, hx.z, x.front, ax);
    }
    const unsigned m = __ballot_sync(0xffffffffu, go);
    if (go) {
      const int e = nv + __popc(m & lanemask_lt());
      const float3 Tn = mul(T, xyz(rec_beta(w, s, d)));
      vput(0, e, __int_as_float(s));
      vput(1, e, __int_as_float(d + 1));
      vput(2, e, x.p.x); vput(3, e, x.p.y); vput(4, e, x.p.z);
      vput(5, e, Tn.x); vput(6, e, Tn.y); vput(7, e, Tn.z);
      vput(8, e, __uint_as_float((unsigned)rng.state)); vput(9, e, __uint_as_float((unsigned)(rng.state >> 32)));
      vput(10, e, __uint_as_float((unsigned)rng.inc)); vput(11, e, __uint_as_float((unsigned)(rng.inc >> 32)));
      if (VERTS) {
        vput(12, e, carry.p.x); vput(13, e, carry.p.y); vput(14, e, carry.p.z);
        vput(15, e, carry.n.x); vput(16, e, carry.n.y); vput(17, e, carry.n.z);
        vput(18, e, carry.t.x); vput(19, e, carry.t.y); vput(20, e, carry.t.z);
        vput(21, e, carry.area);
      }
    }
    nv += __popc(m);
    __syncwarp();
  }
  if (UNB) cam.flush_warp();
  hot_flush(hot);
}

// The same for jobs with a DiffuseBsdfMaterial mesh or an environment light, one thread per
// path over all depths: the incoming direction of a vertex depends on the previous vertex (or
// the camera origin), so a vertex's surface adjoint is scattered one depth later.
template <bool UNB>
__global__ void __launch_bounds__(128, 2) k_adjoint_ext(WF w, const DevScene* __restrict__ scenes,
                                                        const DevView* __restrict__ views, Tile tile) {
  const int stride = gridDim.x * blockDim.x;
  CamAcc cam;
  const int n32 = (tile.n + 31) & ~31;
  HotAcc hot;
  hot_init(hot);
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool has0 = false;
    SurfAdj ax0 = zero_adj();
    float3 atex0 = f3(0.f, 0.f, 0.f);
    const DevTex* tx0 = nullptr;
    int toff0 = 0;
    const DevScene* scp = nullptr;
    const DevView* Vp = nullptr;
    float4 h0 = make_float4(__int_as_float(-1), 0.f, 0.f, 0.f);
    float3 g, o0;
    Surf x0;
    x0.front = true;
    if (s < tile.n && primary_point(w, scenes, views, tile, s, Vp, scp, h0, g, x0, o0)) {
      const DevView& V = *Vp;
      const DevScene& sc = *scp;
      hot_bind(hot, scp);
      float3 co = f3(0.f, 0.f, 0.f);  // the path's share of the camera origin's adjoint
      if (x0.is_light) {
        // camera ray on a light: L = emit at depth 0 when lights are visible
        if (w.light_vis) {
          const DevLight& Lt = sc.lights[x0.light];
          const float3 L = light_emit<true>(Lt, x0);
          has0 = true;
          ax0.area = dot(g, L) / x0.area;
          if (UNB) cam.add(&V, cam_jacobian_adj(V, x0, dot(g, L), ax0));
          if (Lt.kind == kLightArea) {
            add_emit(sc, hot, x0.light, g);
          } else {
            // an SH9 light's radiance depends on wi = -normalize(x0 - o): its share goes
            // to the ray origin, which moves with the camera
            const float3 aw = env_emit_adj(&Lt, x0.u, x0.v, x0.wi, g);
            if (Lt.kind == kLightSh9) cam.add(&V, (aw - x0.wi * dot(x0.wi, aw)) / sqrtf(x0.sqd));
          }
        }
      } else {
        const float3 L = suffix_radiance(w, s, 0);
        if (finite3(L)) {
          has0 = true;
          Rng rng = make_rng((unsigned long long)(tile.begin + s - V.sample_off) + w.seed);
          rng.next_float();
          rng.next_float();
          SurfAdj ax = zero_adj();
          ax.area = dot(g, L) / x0.area;  // jacobi of the primary hit
          if (UNB) co = cam_jacobian_adj(V, x0, dot(g, L), ax);
          Surf xc = x0;
          int tric = __float_as_int(h0.x);
          float4 hc = h0;
          float3 T = f3(1.f, 1.f, 1.f);
          // the surface adjoint of depth d-1 >= 1, scattered after depth d
          SurfAdj axq = zero_adj();
          int triq = -1;
          float4 hq = h0;
          bool frontq = true;
          for (int d = 0; d < w.D; ++d) {
            const float3 adjC = mul(g, T);
            const float3 adjB = mul(adjC, suffix_radiance(w, s, d + 1));
            const DevObj& ob = sc.objs[xc.obj];
            const MatPt mp = mat_point(ob, xc);
            MatAdj ma = zero_mat_adj();
            SurfAdj nextc = zero_adj();
            Surf nx;
            float3 none;
            for (int i = 0; i < w.nL; ++i) {
              const float rx = rng.next_float(), ry = rng.next_float();
              light_sample_adj<true, true>(w, sc, xc, mp.color * kInvPi, rx, ry, rec_hit(w, s, d, i), adjC, ax, hot, none, &mp,
                                     &ma);
            }
            for (int j = 0; j < w.nB; ++j) {
              const float rx = rng.next_float(), ry = rng.next_float();
              bsdf_sample_adj<UNB, true, true>(w, sc, xc, mp.color * kInvPi, rx, ry, rec_hit(w, s, d, w.nL + j), adjC, ax, hot, none,
                                         &mp, &ma);
            }
            const float rx = rng.next_float(), ry = rng.next_float();
            const bool next = d < w.D - 1 && continuation_adj<UNB, true, true>(sc, xc, mp.color * kInvPi, rx, ry,
                                                                         rec_hit(w, s, d, w.nL + w.nB), adjB, ax, nextc, nx, none, &mp, &ma);
            const float3 aorg = mat_finalize(ob, xc, mp, ma, ax);
            if (d == 0) cam.add(&V, co + aorg);
            else if (d == 1) ax0.p += aorg;
            else axq.p += aorg;
            if (triq >= 0) scatter_mesh(sc, triq, hq.y, hq.z, frontq, axq);
            triq = -1;
            const int off = texel_offset(ob.color, xc.u, xc.v);
            if (d == 0) {
              ax0 = ax;
              atex0 = ma.color;
              tx0 = &ob.color;
              toff0 = off;
            } else {
              if (ob.color.grad) scatter_tex(ob.color, off, ma.color, false);
              axq = ax;
              triq = tric;
              hq = hc;
              frontq = xc.front;
            }
            if (!next) break;
            T = mul(T, xyz(rec_beta(w, s, d)));
            hc = rec_hit(w, s, d, w.nL + w.nB);
            tric = __float_as_int(hc.x);
            xc = nx;
            if (xc.is_light) break;  // the path ends on a light: nothing downstream
            ax = nextc;
          }
          if (triq >= 0) scatter_mesh(sc, triq, hq.y, hq.z, frontq, axq);
        }
      }
    }
    scatter_surf_warp(scp, hot, __float_as_int(h0.x), h0.y, h0.z, x0.front, ax0, has0);
    scatter_tex_warp(tx0, toff0, atex0, has0);
  }
  cam.flush_warp();
  hot_flush(hot);
}

// ------------------------------------------------------------------ hypercube
struct HCube {
  const float* pmf;
  const float* cmf;
  const double* w;    // cell masses (double)
  const double* pre;  // inclusive prefix sums of w
  int ncells;
  int res[3];
  float unit[3];
};

// Unbiased estimator: the cell is the first whose double-precision prefix sum exceeds
// s * total (a float CDF cannot resolve cells below 2^-24 of the mass nor place a sample
// inside them); the caller draws a fresh uniform for the position inside the cell.
PSDR_D int hc_cell_unb(const HCube& hc, float s, double& pmf) {
  const double tot = hc.pre[hc.ncells - 1];
  const double t = (double)s * tot;
  int lo = 0, hi = hc.ncells - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (hc.pre[mid] > t) hi = mid;
    else lo = mid + 1;
  }
  pmf = hc.w[lo] / tot;
  return lo;
}

// ------------------------------------------------------------------ primary edges
// True when triangle tri is one of the faces of the edge with vertices ev.
PSDR_D bool tri_has_edge(const DevScene& sc, int tri, int2 ev) {
  if (tri < 0) return false;
  const int4 tv = __ldg(sc.tri_v + tri);
  return (tv.x == ev.x || tv.y == ev.x || tv.z == ev.x) && (tv.x == ev.y || tv.y == ev.y || tv.z == ev.y);
}

// path_integrator.cc:188-272. PRE=true is the preprocess pass over the hypercube
// cells (sample index = cell, the sampler stream persists across rounds); PRE=false
// samples the cell from the preprocessed mass.
// unb (unbiased estimator, PRE=false): one offset ray must hit a face of the edge
// (foreground); the path of the other side (background, possibly a miss) is traced,
// and eb.hb keeps that background hit with flag 1 (background on the +eps side) or 2.
template <bool PRE>
__global__ void __launch_bounds__(128, 6) k_edge_init(WF w, const DevScene* __restrict__ scenes,
                                                   const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                   long long begin, int n, HCube hc, int round, int unb) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < n) {
      const long long i = begin + s;
      const DevView& V = views[v];
      const DevScene& sc = scenes[V.scene];
      Rng rng;
      float s1, hpdf = 1.f;
      bool ok = true;
      if (PRE) {
        if (round == 0) rng = make_rng((unsigned long long)i);
        else { rng.state = w.rs[s]; rng.inc = w.ri[s]; }
        s1 = ((float)i + rng.next_float()) * hc.unit[0];
      } else {
        rng = make_rng((unsigned long long)i + w.seed);
        s1 = rng.next_float();
        if (unb) {
          double pm;
          const int cell = hc_cell_unb(hc, s1, pm);
          hpdf = (float)pm;
          ok = pm > 0.0;
          s1 = (rng.next_float() + (float)cell) * hc.unit[0];
        } else {
          const int cell = discrete_sample(hc.pmf, hc.cmf, hc.ncells, s1, hpdf);
          ok = hpdf > 0.f;
          s1 = (s1 + (float)cell) * hc.unit[0];
        }
      }
      const int ne = *sc.n_edges;
      float ss = s1, pe;
      const int e = discrete_sample(sc.edge_pmf, sc.edge_cmf, ne, ss, pe);
      const float4 E0 = __ldg(sc.edge + 4 * (size_t)e), E1 = __ldg(sc.edge + 4 * (size_t)e + 1);
      // ray construction in explicitly rounded ops (bit-identical to the float oracle)
      const float3 p0 = xyz(E0), p1 = xyz(E1);
      const float3 xe = add_rn(p0, scale_rn(sub_rn(p1, p0), ss));
      const float pdf_e = __fdiv_rn(pe, E0.w);
      const float3 pc = xform_pos_rn(V.w2c, xe);
      const float3 pr = xform_pos_rn(V.c2r, pc);
      const int px = (int)floorf(pr.x), py = (int)floorf(pr.y);
      bool valid = ok && pc.z < 0.f && pr.x > 0.f && pr.x < (float)V.W && pr.y > 0.f && pr.y < (float)V.H;
      // camera.h:260-276 / 336-353: the ray through the edge point
      const bool ortho = V.ortho;
      const float3 eo = ortho ? xform_pos_rn(V.c2w, f3(pc.x, pc.y, 0.f)) : V.pos;
      const float3 rd = ortho ? view_look_dir(V) : normalize_rn(sub_rn(xe, V.pos));
      const float3 nrm = cross_rn(rd, normalize_rn(sub_rn(p1, p0)));
      HitRec ha, hb;
      ha.tri = hb.tri = -1;
      ha.b1 = ha.b2 = hb.b1 = hb.b2 = 0.f;
      if (valid) {
        const float3 da = sub_rn(rd, scale_rn(nrm, kEps)), db = add_rn(rd, scale_rn(nrm, kEps));
        const int2 ef = (!PRE && unb) ? __ldg(sc.edge_f + e) : make_int2(kEdgeNonManifold, -1);
        if (ef.x == kEdgeNonManifold) {
          ha = trace_closest(sc, eo, da, kTmin, INFINITY);
          hb = trace_closest(sc, eo, db, kTmin, INFINITY);
        } else {
          // Unbiased silhouette sample: valid only when exactly one offset ray's closest hit
          // is a face of the edge. Test each ray against the edge's faces first (the
          // traversal's test and tie rule): a ray that misses both cannot have one as its
          // closest hit, and for a ray that hits one at t an occlusion query bounded at t
          // decides. Only the other ray of a valid sample needs its full closest hit (its
          // background).
          auto face_hit = [&](float3 d, float& tf) {
            const RayPre rp = ray_pre(eo, d);
            int best = -1;
            tf = INFINITY;
            for (int k = 0; k < 2; ++k) {
              const int f = k == 0 ? ef.x : ef.y;
              if (f < 0) continue;
              const float4* q = sc.tri + 6 * (size_t)f;
              float tt, b1, b2;
              if (tri_test(rp, xyz(__ldg(q)), xyz(__ldg(q + 1)), xyz(__ldg(q + 2)), kTmin, tf, tt, b1, b2) &&
                  (tt < tf || best < 0 || f < best)) {
                tf = tt;
                best = f;
              }
            }
            return best >= 0;
          };
          float tfa, tfb;
          const bool fa = face_hit(da, tfa), fb = face_hit(db, tfb);
          if (fa && fb) {
            // both rays reach the faces: bounded queries decide each ray; only a ray whose
            // face is hidden while the other's is seen needs its full closest hit
            const int2 ev = __ldg(sc.edge_v + e);
            ha = trace_closest(sc, eo, da, kTmin, tfa, tfa);
            hb = trace_closest(sc, eo, db, kTmin, tfb, tfb);
            const bool na = tri_has_edge(sc, ha.tri, ev), nb = tri_has_edge(sc, hb.tri, ev);
            if (na && !nb) hb = trace_closest(sc, eo, db, kTmin, INFINITY);
            else if (nb && !na) ha = trace_closest(sc, eo, da, kTmin, INFINITY);
          } else if (fa) {
            ha = trace_closest(sc, eo, da, kTmin, tfa, tfa);
            if (tri_has_edge(sc, ha.tri, __ldg(sc.edge_v + e))) hb = trace_closest(sc, eo, db, kTmin, INFINITY);
          } else if (fb) {
            hb = trace_closest(sc, eo, db, kTmin, tfb, tfb);
            if (tri_has_edge(sc, hb.tri, __ldg(sc.edge_v + e))) ha = trace_closest(sc, eo, da, kTmin, INFINITY);
          }
        }
      }
      int flag;
      HitRec hcur = ha;
      if (!PRE && unb) {
        const int2 ev = __ldg(sc.edge_v + e);
        const bool na = tri_has_edge(sc, ha.tri, ev), nb = tri_has_edge(sc, hb.tri, ev);
        const HitRec& hg = na ? hb : ha;
        valid = valid && na != nb && hg.tri >= 0;
        flag = valid ? (na ? 1 : 2) : 0;
        hcur = hg;
        eb.hb[s] = make_float4(__int_as_float(hg.tri), hg.b1, hg.b2, __int_as_float(flag));
      } else {
        const Surf a = make_surf(sc, ha.tri, ha.b1, ha.b2, eo);
        const Surf b = make_surf(sc, hb.tri, hb.b1, hb.b2, eo);
        valid = valid && a.valid && b.valid && (norm(a.p - xe) < 10.f * kEps || norm(b.p - xe) < 10.f * kEps);
        flag = valid ? 1 : 0;
        eb.hb[s] = make_float4(__int_as_float(hb.tri), hb.b1, hb.b2, __int_as_float(flag));
      }
      eb.a[s] = make_float4(__int_as_float(e), ss, pdf_e, hpdf);
      eb.n[s] = make_float4(nrm.x, nrm.y, nrm.z, __int_as_float(py * V.W + px));
      w.rs[s] = rng.state;
      w.ri[s] = rng.inc;
      w.view[s] = v;
      w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
      w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      w.cur[s] = hit4(hcur);
      w.org[s] = make_float4(eo.x, eo.y, eo.z, 0.f);
      eb.La[s] = w.org[s];  // the ray origin, for the second path (k_edge_mid)
      alive = valid;
    }
    const int k = warp_append(&w.cnt[0], alive);
    if (alive) w.q0[k] = s;
  }
}

// Unbiased silhouette term: -sgn L_bg K (d_rel . n) with d_rel = (dx_e - do) -
// (r_e / r_bg)(dx_bg - do), K = fx fy r_e / z_e^3 / (pdf_e hc_density H W spp); the
// background point moves with its triangle, the edge point with the edge's vertices.
__global__ void __launch_bounds__(256) k_edge_final_unb(WF w, const DevScene* __restrict__ scenes,
                                                        const DevView* __restrict__ views, int v, EdgeBuf eb, int n,
                                                        float cells, int spp) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  const float3 look = view_look(V);
  const float fxfy = view_fxfy(V);
  GradAcc* const gpos = V.grad_pos;
  Own3 go;  // camera origin
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n || !V.dimage) continue;
    const float4 hg = eb.hb[s];
    const int flag = __float_as_int(hg.w);
    if (flag == 0) continue;
    const float4 a = eb.a[s], nn = eb.n[s];
    const float* gp = V.dimage + 3 * (size_t)__float_as_int(nn.w);
    const float3 L = xyz(w.L[s]);
    const float phi = gp[0] * L.x + gp[1] * L.y + gp[2] * L.z;
    if (!(phi != 0.f) || !isfinite(phi)) continue;
    const int e = __float_as_int(a.x);
    const float ss = a.y;
    const float4 E0 = __ldg(sc.edge + 4 * (size_t)e), E1 = __ldg(sc.edge + 4 * (size_t)e + 1);
    const float3 xe = add_rn(xyz(E0), scale_rn(sub_rn(xyz(E1), xyz(E0)), ss));
    const float3 re3 = xe - V.pos;
    const float re = norm(re3), z = dot(re3, look);
    const int tri = __float_as_int(hg.x);
    const Surf g = make_surf(sc, tri, hg.y, hg.z, V.pos);
    // orthographic: no depth scaling, and a camera translation moves both points alike
    const float ratio = V.ortho ? 1.f : re / sqrtf(g.sqd);
    const float K = fxfy * (V.ortho ? 1.f : re / (z * z * z)) / (a.z * a.w * cells * (float)V.H * (float)V.W *
                                                                  (float)spp);
    const float3 av = xyz(nn) * (-(flag == 1 ? 1.f : -1.f) * phi * K);
    if (!finite3(av)) continue;
    if (sc.grad_verts) {
      const int2 ev = __ldg(sc.edge_v + e);
      vert_add(sc, ev.x, av * (1.f - ss));
      vert_add(sc, ev.y, av * ss);
      const int4 tv = __ldg(sc.tri_v + tri);
      const float3 ag = av * (-ratio);
      vert_add(sc, tv.x, ag * (1.f - hg.y - hg.z));
      vert_add(sc, tv.y, ag * hg.y);
      vert_add(sc, tv.z, ag * hg.z);
    }
    if (gpos) go.add(-(av * (1.f - ratio)));
  }
  if (gpos) go.put_warp(gpos);
}

// Between the two trace2light calls: keep L_a, restart the slot at the +eps hit with
// the sampler stream continuing where the first path left it.
__global__ void __launch_bounds__(256) k_edge_mid(WF w, const DevView* __restrict__ views, int v, EdgeBuf eb, int n) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < n) {
      const float4 hb = eb.hb[s];
      alive = __float_as_int(hb.w) != 0;
      if (alive) {
        const float4 eo = eb.La[s];  // the ray origin k_edge_init left there
        eb.La[s] = w.L[s];
        w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
        w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        w.cur[s] = make_float4(hb.x, hb.y, hb.z, 0.f);
        w.org[s] = eo;
      }
    }
    const int k = warp_append(&w.cnt[0], alive);
    if (alive) w.q0[k] = s;
  }
}

// PRE: mass[cell] += |dL / pdf_e|. Otherwise the gradient of the zero-valued term
// (x_e - detach(x_e)).n + (o - detach(o)).(n*[1,1,-1]) times dL / pdf_e / pdf_hc / spp.
template <bool PRE>
__global__ void __launch_bounds__(256) k_edge_final(WF w, const DevScene* __restrict__ scenes,
                                                    const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                    long long begin, int n, float* mass, int spp) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  GradAcc* const gpos = V.grad_pos;
  Own3 go;  // camera origin
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n) continue;
    const float4 hb = eb.hb[s];
    if (__float_as_int(hb.w) == 0) continue;
    const float3 La = xyz(eb.La[s]), Lb = xyz(w.L[s]);
    const float3 dL = sub_rn(La, Lb);
    const float4 a = eb.a[s];
    const float pdf_e = a.z;
    if (PRE) {
      const float3 val = f3(__fdiv_rn(dL.x, pdf_e), __fdiv_rn(dL.y, pdf_e), __fdiv_rn(dL.z, pdf_e));
      if (finite3(val)) mass[begin + s] = __fadd_rn(mass[begin + s], norm_rn(val));
    } else {
      if (!finite3(dL * 0.0f)) continue;
      const float4 nn = eb.n[s];
      const int pix = __float_as_int(nn.w);
      if (!V.dimage) continue;
      const float* gp = V.dimage + 3 * (size_t)pix;
      const float K = (gp[0] * dL.x + gp[1] * dL.y + gp[2] * dL.z) / (pdf_e * a.w * (float)spp);
      const float3 nrm = xyz(nn);
      // x_dot_n = (x_e - detach(x_e)).n + (o - detach(o)).nflip; an orthographic ray's
      // origin o is x_e's foot on the camera plane and moves with x_e as well
      const float3 nflip = f3(nrm.x, nrm.y, -nrm.z);
      const float3 jo = V.ortho ? ortho_origin_jt(V, nflip) : f3(0.f, 0.f, 0.f);
      const float3 ax = (nrm + jo) * K;
      const int e = __float_as_int(a.x);
      const float ss = a.y;
      if (sc.grad_verts) {
        const int2 ev = __ldg(sc.edge_v + e);
        vert_add(sc, ev.x, ax * (1.f - ss));
        vert_add(sc, ev.y, ax * ss);
      }
      if (gpos) go.add((nflip - jo) * K);
    }
  }
  if (!PRE && gpos) go.put_warp(gpos);
}

// ------------------------------------------------------------------ pixel borders
// Unbiased estimator: material crossing the pixel borders. The border segments are the
// (W+1) x H vertical and W x (H+1) horizontal unit segments of the pixel grid; segment q
// contributes (dI[hi] - dI[lo]) . Int L v dl, L the radiance seen through the border
// point and v the raster velocity of its primary vertex across the segment (material
// flows into pixel hi and out of pixel lo; outside the image dI = 0). Segments are
// importance-sampled by m_q = |dI[hi] - dI[lo]|_1 (zero where the term is zero) with
// stratified inversion of the double-precision CDF: sample i of N takes
// u = (i + xi) / N, its segment is the first with prefix > u * total and its position
// along the segment the remainder, so every segment gets N m_q / total samples spread
// evenly along it.
PSDR_D void border_pixels(const DevView& V, long long q, bool& vert, int& k, int& j, int& lo, int& hi) {
  const long long nv = (long long)(V.W + 1) * V.H;
  vert = q < nv;
  lo = hi = -1;
  if (vert) {
    k = (int)(q % (V.W + 1));
    j = (int)(q / (V.W + 1));
    if (k >= 1) lo = j * V.W + k - 1;
    if (k < V.W) hi = j * V.W + k;
  } else {
    const long long r = q - nv;
    k = (int)(r % V.W);
    j = (int)(r / V.W);
    if (j >= 1) lo = (j - 1) * V.W + k;
    if (j < V.H) hi = j * V.W + k;
  }
}

PSDR_D float3 dimage_at(const DevView& V, int p) {
  if (p < 0) return f3(0.f, 0.f, 0.f);
  const float* g = V.dimage + 3 * (size_t)p;
  return f3(g[0], g[1], g[2]);
}

__global__ void k_border_mass(const DevView* __restrict__ views, int v, float* __restrict__ mass, long long S) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= S) return;
  const DevView& V = views[v];
  bool vert;
  int k, j, lo, hi;
  border_pixels(V, q, vert, k, j, lo, hi);
  const float3 d = dimage_at(V, hi) - dimage_at(V, lo);
  mass[q] = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
}

// Segment and position of border sample i of N (explicitly rounded double arithmetic,
// identical in the oracle).
PSDR_D long long border_locate(const double* __restrict__ w, const double* __restrict__ pre, long long S,
                               long long i, long long N, float xi, float& t, double& pmf) {
  const double tot = pre[S - 1];
  const double u = __ddiv_rn(__dadd_rn((double)i, (double)xi), (double)N);
  const double tt = __dmul_rn(u, tot);
  long long lo = 0, hi = S - 1;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (pre[mid] > tt) hi = mid;
    else lo = mid + 1;
  }
  const double base = lo > 0 ? pre[lo - 1] : 0.0;
  double r = __ddiv_rn(__dsub_rn(tt, base), w[lo]);
  r = r < 0.0 ? 0.0 : r;
  t = fminf((float)r, 0.99999994f);
  pmf = __ddiv_rn(w[lo], tot);
  return lo;
}

__global__ void __launch_bounds__(128) k_border_init(WF w, const DevScene* __restrict__ scenes,
                                                     const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                     const double* __restrict__ mw, const double* __restrict__ mpre,
                                                     long long S, long long begin, int n, long long N) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < n) {
      const long long i = begin + s;
      const DevView& V = views[v];
      const DevScene& sc = scenes[V.scene];
      Rng rng = make_rng((unsigned long long)i + w.seed);
      const float xi = rng.next_float();
      float t;
      double pmf;
      const long long q = border_locate(mw, mpre, S, i, N, xi, t, pmf);
      bool vert;
      int k, j, lo, hi;
      border_pixels(V, q, vert, k, j, lo, hi);
      const float3 fp = vert ? f3((float)k, t + (float)j, 1.0f) : f3(t + (float)k, (float)j, 1.0f);
      float3 pc;
      xform_pos(V.r2c, fp, pc);
      float3 o = V.pos, d;
      if (V.ortho) {
        xform_pos(V.c2w, f3(pc.x, pc.y, 0.f), o);
        d = view_look_dir(V);
      } else {
        d = normalize(xform_dir(V.c2w, pc));
      }
      const HitRec h = trace_closest(sc, o, d, kTmin, INFINITY);
      w.rs[s] = rng.state;
      w.ri[s] = rng.inc;
      w.view[s] = v;
      w.pix[s] = -1;
      w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
      w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      w.cur[s] = hit4(h);
      w.org[s] = make_float4(o.x, o.y, o.z, 0.f);
      eb.hb[s] = hit4(h);
      eb.a[s] = make_float4(__int_as_float((int)q), t, (float)pmf, 0.f);
      alive = h.tri >= 0 && pmf > 0.0;
    }
    const int k = warp_append(&w.cnt[0], alive);
    if (alive) w.q0[k] = s;
  }
}

__global__ void __launch_bounds__(256) k_border_final(WF w, const DevScene* __restrict__ scenes,
                                                      const DevView* __restrict__ views, int v, EdgeBuf eb, int n,
                                                      long long N) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  GradAcc* const gpos = V.grad_pos;
  Own3 go;  // camera origin
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n || !V.dimage) continue;
    const float4 h = eb.hb[s];
    const int tri = __float_as_int(h.x);
    if (tri < 0) continue;
    const float4 a = eb.a[s];
    if (!(a.z > 0.f)) continue;
    bool vert;
    int k, j, lo, hi;
    border_pixels(V, __float_as_int(a.x), vert, k, j, lo, hi);
    const float3 L = xyz(w.L[s]);
    const float3 dg = dimage_at(V, hi) - dimage_at(V, lo);
    const float wgt = dot(dg, L) / ((float)N * a.z);
    if (!(wgt != 0.f) || !isfinite(wgt)) continue;
    // raster coordinate c (x for vertical borders, y for horizontal) of the material
    // point and its gradient w.r.t. the point
    const Surf x = make_surf(sc, tri, h.y, h.z, V.pos);
    float3 pc;
    xform_pos(V.w2c, x.p, pc);
    const float* m = V.c2r;
    const int c = vert ? 0 : 1;
    const float wden = m[12] * pc.x + m[13] * pc.y + m[14] * pc.z + m[15];
    const float u = (m[4 * c] * pc.x + m[4 * c + 1] * pc.y + m[4 * c + 2] * pc.z + m[4 * c + 3]) / wden;
    const float3 gpc = f3(m[4 * c] - u * m[12], m[4 * c + 1] - u * m[13], m[4 * c + 2] - u * m[14]) / wden;
    const float* r = V.w2c;
    const float3 gx = f3(r[0] * gpc.x + r[4] * gpc.y + r[8] * gpc.z, r[1] * gpc.x + r[5] * gpc.y + r[9] * gpc.z,
                         r[2] * gpc.x + r[6] * gpc.y + r[10] * gpc.z);
    const float3 ag = gx * wgt;
    if (!finite3(ag)) continue;
    if (sc.grad_verts) {
      const int4 tv = __ldg(sc.tri_v + tri);
      vert_add(sc, tv.x, ag * (1.f - h.y - h.z));
      vert_add(sc, tv.y, ag * h.y);
      vert_add(sc, tv.z, ag * h.z);
    }
    if (gpos) go.add(-ag);
  }
  if (gpos) go.put_warp(gpos);
}

// ------------------------------------------------------------------ camera lens
// Unbiased estimator, perspective views: derivative of the image with respect to the
// camera's basis and field of view (look_at, up, fov, and look_from through the basis).
// With the camera origin fixed, the world direction seen at raster point u (taken from
// the image centre) is M [u; 1], M = C diag(2 tan(fov/2) / W, -2 tan(fov/2) / H, -1), C the
// camera basis (right, up, dir) of camera.h:35-52. A change dM moves the image content
// with the raster velocity V(u) = (h_3 u_x - h_1, h_3 u_y - h_2), h = G [u; 1],
// G = M^-1 dM. A box-filtered pixel then changes by the content flowing in across its
// borders (the integral the pixel-border samples estimate, with V in place of the
// material point's raster velocity) plus Int_P L div V du, where
// div V = 3 (G_31 u_x + G_32 u_y) + 2 G_33 - G_11 - G_22.
// Per view: grad_lens[0..2] = sum over camera samples of g.L {1, u_x, u_y} / spp (g the
// pixel's dPhi/dI), grad_lens[3..11] = dPhi/dG of the border part (row-major 3x3).
struct LensAcc {
  const DevView* v = nullptr;
  Own3 s;
  PSDR_D void add(const DevView* view, float gl, float ux, float uy) {
    if (view != v) {
      flush();
      v = view;
    }
    s.add(f3(gl, gl * ux, gl * uy));  // (views without grad_lens are skipped)
  }
  PSDR_D void flush() {
    if (v) s.put(v->grad_lens);
    v = nullptr;
    s = Own3();
  }
  PSDR_D void flush_warp() {
    const unsigned long long key = (unsigned long long)v;
    const unsigned long long k0 = __shfl_sync(0xffffffffu, key, 0);
    if (!__all_sync(0xffffffffu, key == k0) || !v) { flush(); return; }
    s.put_warp(v->grad_lens);
    v = nullptr;
  }
};

// Interior moments from the replay records of a tile (after its adjoint): the sample's
// radiance is the film's value (the emission of a visible light, or the path's suffix
// radiance from depth 0); its raster position replays the two jitter draws of k_camera.
template <bool BSDF>
__global__ void __launch_bounds__(256) k_lens_interior(WF w, const DevScene* __restrict__ scenes,
                                                       const DevView* __restrict__ views, Tile tile) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (tile.n + 31) & ~31;
  LensAcc acc;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= tile.n) continue;
    const DevView& V = views[w.view[s]];
    if (!V.grad_lens || !V.dimage) continue;
    const float4 h0 = rec_at(w, s, 0);
    const int tri0 = __float_as_int(h0.x);
    if (tri0 < 0) continue;
    const DevScene& sc = scenes[V.scene];
    const Surf x0 = make_surf(sc, tri0, h0.y, h0.z, V.pos);
    float3 L;
    if (x0.is_light) {
      if (!w.light_vis) continue;
      L = light_emit<BSDF>(sc.lights[x0.light], x0);
    } else {
      L = suffix_radiance(w, s, 0);
    }
    if (!finite3(L)) continue;
    const int pix = w.pix[s];
    const float* gp = V.dimage + 3 * (size_t)pix;
    const float gl = (gp[0] * L.x + gp[1] * L.y + gp[2] * L.z) / (float)V.spp;
    Rng rng = make_rng((unsigned long long)(tile.begin + s - V.sample_off) + w.seed);
    const float jx = rng.next_float(), jy = rng.next_float();
    acc.add(&V, gl, jx + (float)(pix % V.W) - 0.5f * (float)V.W, jy + (float)(pix / V.W) - 0.5f * (float)V.H);
  }
  acc.flush_warp();
}

// Border part from the pixel-border samples of view v (after k_border_final): the
// sample's weight times dV_c/dG at its raster point, c the coordinate across the border.
__global__ void __launch_bounds__(256) k_lens_border(WF w, const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                     int n, long long N) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  Own3 bv, bh, bc;  // rows of dPhi/dG
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n || !V.dimage || !V.grad_lens) continue;
    if (__float_as_int(eb.hb[s].x) < 0) continue;  // the border ray left the scene: no radiance
    const float4 a = eb.a[s];
    if (!(a.z > 0.f)) continue;
    bool vert;
    int k, j, lo, hi;
    border_pixels(V, __float_as_int(a.x), vert, k, j, lo, hi);
    const float3 L = xyz(w.L[s]);
    const float3 dg = dimage_at(V, hi) - dimage_at(V, lo);
    const float wgt = dot(dg, L) / ((float)N * a.z);
    if (!(wgt != 0.f) || !isfinite(wgt)) continue;
    const float ux = (vert ? (float)k : a.y + (float)k) - 0.5f * (float)V.W;
    const float uy = (vert ? a.y + (float)j : (float)j) - 0.5f * (float)V.H;
    const float wc = wgt * (vert ? ux : uy);
    if (vert) bv.add(f3(-wgt * ux, -wgt * uy, -wgt));
    else bh.add(f3(-wgt * ux, -wgt * uy, -wgt));
    bc.add(f3(wc * ux, wc * uy, wc));
  }
  if (!V.grad_lens) return;
  bv.put_warp(V.grad_lens + 3);
  bh.put_warp(V.grad_lens + 6);
  bc.put_warp(V.grad_lens + 9);
}

// dPhi/dtheta_j = <Gamma, P_j>, Gamma = B + the interior part of dPhi/dG.
__global__ void k_lens_out(const GradAcc* __restrict__ acc, LensChain ch, float* __restrict__ out, int accumulate) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double G[9];
  for (int m = 0; m < 9; ++m) G[m] = acc_value(acc[3 + m].hi, acc[3 + m].lo);
  const double s0 = acc_value(acc[0].hi, acc[0].lo), sx = acc_value(acc[1].hi, acc[1].lo),
               sy = acc_value(acc[2].hi, acc[2].lo);
  G[0] -= s0;
  G[4] -= s0;
  G[6] += 3.0 * sx;
  G[7] += 3.0 * sy;
  G[8] += 2.0 * s0;
  for (int j = 0; j < 10; ++j) {
    double d = 0.0;
    for (int m = 0; m < 9; ++m) d += G[m] * ch.P[j][m];
    out[j] = accumulate ? out[j] + (float)d : (float)d;
  }
}

// ------------------------------------------------------------------ interpenetration creases
// Unbiased estimator: where the surfaces of two different meshes cut into each other (a
// noisy icosphere sunk into the ground), the visible surface switches from one mesh to the
// other along their intersection curve. That curve is not a mesh edge, so neither the
// silhouette nor the shadow-boundary samples see it; it moves when either mesh moves. Its
// term (primary visibility): with surface 1 seen on one side of the projected curve and
// surface 2 on the other, n the raster normal from 1 to 2, the image changes by
//   Int_curve g [L1 (v_c - v_1) - L2 (v_c - v_2)] . n dl
// (raster velocities: v_c of the curve, v_k of surface k's material point at it). With
// J = d(raster)/d(world), w = J^T n, c = n1.n2 and the curve's world velocity taken in the
// plane of the two normals (it stays on both surfaces), the adjoint of surface k's material
// point is K [(G1 - G2) A_k n_k -+ G_k w] (minus for 1), A_1 = (w.n1 - c w.n2) / (1 - c^2),
// A_2 = (w.n2 - c w.n1) / (1 - c^2), G_k = g . L_k, K = raster length per sample.
constexpr int kCreaseCap = 16384;          // intersection segments kept per scene
constexpr int kCreaseSamplesPerSpp = 16384;  // crease samples per primary-edge spp
constexpr unsigned long long kCreaseStream = 0xC0000000ull;  // sampler streams of the crease samples

// Meshes whose boxes the crease extraction keeps (a triangle of a mesh beyond this many
// walks the tree without the box test).
constexpr int kCreaseBoxObjs = 4096;

struct CreaseBuf {
  float4* a;   // segment start xyz, length (ordered by the triangle pair)
  float4* b;   // segment end xyz, -
  int2* tris;  // the two triangles (different meshes)
  float4* ra;  // the same, in the order the extraction found them
  float4* rb;
  int2* rtris;
  int* count;  // segments found (may exceed kCreaseCap: the rest are dropped)
  int* obox;   // per mesh: its box (min xyz, max xyz as order-preserving ints), kCreaseBoxObjs
  int* later;  // per mesh m: the box of meshes m+1 .. (the ones its triangles are tested against)
};

// Order-preserving int image of a float (for atomicMin / atomicMax on boxes).
PSDR_D int f2ord(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
PSDR_D float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void k_crease_box_init(const DevScene* __restrict__ scenes, int si, CreaseBuf cb) {
  const int n = min(scenes[si].nobj, kCreaseBoxObjs);
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < n; o += gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) {
      cb.obox[6 * o + k] = 0x7fffffff;
      cb.obox[6 * o + 3 + k] = (int)0x80000000;
    }
}

// Box of every mesh (lights excluded): one thread per triangle, reduced over the warp when
// its triangles belong to one mesh (meshes are contiguous ranges of triangles).
__global__ void k_crease_boxes(const DevScene* __restrict__ scenes, int si, CreaseBuf cb) {
  const DevScene& sc = scenes[si];
  const int nmesh = min(sc.nobj - sc.nlight, kCreaseBoxObjs);
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (sc.ntri + 31) & ~31;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n32; t += stride) {
    int o = -1;
    int v[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000, (int)0x80000000};
    if (t < sc.ntri) {
      o = __ldg(sc.tri_v + t).w;
      if (o < nmesh) {
        const float4* R = sc.tri + 6 * (size_t)t;
        const float3 p0 = xyz(__ldg(R)), p1 = xyz(__ldg(R + 1)), p2 = xyz(__ldg(R + 2));
        v[0] = f2ord(fminf(p0.x, fminf(p1.x, p2.x)));
        v[1] = f2ord(fminf(p0.y, fminf(p1.y, p2.y)));
        v[2] = f2ord(fminf(p0.z, fminf(p1.z, p2.z)));
        v[3] = f2ord(fmaxf(p0.x, fmaxf(p1.x, p2.x)));
        v[4] = f2ord(fmaxf(p0.y, fmaxf(p1.y, p2.y)));
        v[5] = f2ord(fmaxf(p0.z, fmaxf(p1.z, p2.z)));
      } else {
        o = -1;
      }
    }
    const int o0 = __shfl_sync(0xffffffffu, o, 0);
    if (__all_sync(0xffffffffu, o == o0)) {
      if (o0 < 0) continue;
      for (int k = 0; k < 3; ++k) {
        const int mn = __reduce_min_sync(0xffffffffu, v[k]);
        const int mx = __reduce_max_sync(0xffffffffu, v[3 + k]);
        if ((threadIdx.x & 31) == 0) {
          atomicMin(cb.obox + 6 * o0 + k, mn);
          atomicMax(cb.obox + 6 * o0 + 3 + k, mx);
        }
      }
    } else if (o >= 0) {
      for (int k = 0; k < 3; ++k) {
        atomicMin(cb.obox + 6 * o + k, v[k]);
        atomicMax(cb.obox + 6 * o + 3 + k, v[3 + k]);
      }
    }
  }
}

// later[m] = union of the boxes of meshes m+1 .. nmesh-1 (empty for the last).
__global__ void k_crease_later(const DevScene* __restrict__ scenes, int si, CreaseBuf cb) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const DevScene& sc = scenes[si];
  const int nmesh = min(sc.nobj - sc.nlight, kCreaseBoxObjs);
  int u[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000, (int)0x80000000};
  for (int m = nmesh - 1; m >= 0; --m) {
    for (int k = 0; k < 6; ++k) cb.later[6 * m + k] = u[k];
    for (int k = 0; k < 3; ++k) {
      u[k] = min(u[k], cb.obox[6 * m + k]);
      u[3 + k] = max(u[3 + k], cb.obox[6 * m + 3 + k]);
    }
  }
}

// The segment where triangles a and b cross (false when they do not, or are coplanar).
// Double precision; a vertex exactly on the other plane counts as on its positive side.
PSDR_D bool tri_tri_segment(const double3* A, const double3* B, double3& s0, double3& s1) {
  auto sub = [](double3 p, double3 q) { return make_double3(p.x - q.x, p.y - q.y, p.z - q.z); };
  auto dotd = [](double3 p, double3 q) { return p.x * q.x + p.y * q.y + p.z * q.z; };
  auto crs = [](double3 p, double3 q) {
    return make_double3(p.y * q.z - p.z * q.y, p.z * q.x - p.x * q.z, p.x * q.y - p.y * q.x);
  };
  // the two points where triangle T's edges cross the plane (n, d); false if none
  auto cut = [&](const double3* T, double3 n, double d, double3& p, double3& q) {
    double s[3];
    for (int k = 0; k < 3; ++k) s[k] = dotd(n, T[k]) + d;
    const bool pos0 = s[0] >= 0.0, pos1 = s[1] >= 0.0, pos2 = s[2] >= 0.0;
    if (pos0 == pos1 && pos1 == pos2) return false;
    // the lone vertex on its side
    const int k = (pos0 != pos1 && pos0 != pos2) ? 0 : (pos1 != pos0 && pos1 != pos2) ? 1 : 2;
    const int i = (k + 1) % 3, j = (k + 2) % 3;
    const double ti = s[k] / (s[k] - s[i]), tj = s[k] / (s[k] - s[j]);
    p = make_double3(T[k].x + (T[i].x - T[k].x) * ti, T[k].y + (T[i].y - T[k].y) * ti, T[k].z + (T[i].z - T[k].z) * ti);
    q = make_double3(T[k].x + (T[j].x - T[k].x) * tj, T[k].y + (T[j].y - T[k].y) * tj, T[k].z + (T[j].z - T[k].z) * tj);
    return true;
  };
  const double3 na = crs(sub(A[1], A[0]), sub(A[2], A[0])), nb = crs(sub(B[1], B[0]), sub(B[2], B[0]));
  const double3 D = crs(na, nb);
  const double dd = dotd(D, D);
  if (!(dd > 1e-30 * dotd(na, na) * dotd(nb, nb))) return false;
  double3 pa, qa, pb, qb;
  if (!cut(A, nb, -dotd(nb, B[0]), pa, qa) || !cut(B, na, -dotd(na, A[0]), pb, qb)) return false;
  double ta0 = dotd(pa, D), ta1 = dotd(qa, D), tb0 = dotd(pb, D), tb1 = dotd(qb, D);
  if (ta0 > ta1) { const double t = ta0; ta0 = ta1; ta1 = t; const double3 x = pa; pa = qa; qa = x; }
  if (tb0 > tb1) { const double t = tb0; tb0 = tb1; tb1 = t; const double3 x = pb; pb = qb; qb = x; }
  const double lo = fmax(ta0, tb0), hi = fmin(ta1, tb1);
  if (!(lo < hi)) return false;
  s0 = ta0 >= tb0 ? pa : pb;
  s1 = ta1 <= tb1 ? qa : qb;
  return true;
}

// One thread per triangle of a mesh: the LBVH is walked with the triangle's box, and every
// triangle of a later mesh (lights excluded) that it crosses adds one segment.
__global__ void __launch_bounds__(128) k_crease_pairs(const DevScene* __restrict__ scenes, int si, CreaseBuf cb) {
  const DevScene& sc = scenes[si];
  const int nmesh = sc.nobj - sc.nlight;
  const int stride = gridDim.x * blockDim.x;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < sc.ntri; t += stride) {
    const int4 tv = __ldg(sc.tri_v + t);
    if (tv.w >= nmesh || sc.root == 0x7fffffff) continue;
    const float4* R = sc.tri + 6 * (size_t)t;
    const float3 p0 = xyz(__ldg(R)), p1 = xyz(__ldg(R + 1)), p2 = xyz(__ldg(R + 2));
    const float3 lo = f3(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)), fminf(p0.z, fminf(p1.z, p2.z)));
    const float3 hi = f3(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)), fmaxf(p0.z, fmaxf(p1.z, p2.z)));
    if (tv.w < kCreaseBoxObjs) {
      // a triangle clear of every later mesh's box crosses none of its triangles
      const int* L = cb.later + 6 * tv.w;
      if (__ldg(L) == 0x7fffffff || ord2f(__ldg(L)) > hi.x || ord2f(__ldg(L + 3)) < lo.x || ord2f(__ldg(L + 1)) > hi.y ||
          ord2f(__ldg(L + 4)) < lo.y || ord2f(__ldg(L + 2)) > hi.z || ord2f(__ldg(L + 5)) < lo.z)
        continue;
    }
    const double3 A[3] = {make_double3(p0.x, p0.y, p0.z), make_double3(p1.x, p1.y, p1.z), make_double3(p2.x, p2.y, p2.z)};
    int stack[64];
    int sp = 0;
    int node = sc.root;
    while (true) {
      if (node >= 0) {
        const float4* nd = sc.nodes + kNodeF4 * (size_t)node;
        const float4 lx = __ldg(nd), hx = __ldg(nd + 1), ly = __ldg(nd + 2), hy = __ldg(nd + 3);
        const float4 lz = __ldg(nd + 4), hz = __ldg(nd + 5);
        const int4 e = __ldg(reinterpret_cast<const int4*>(nd + 6));
        const float clx[4] = {lx.x, lx.y, lx.z, lx.w}, chx[4] = {hx.x, hx.y, hx.z, hx.w};
        const float cly[4] = {ly.x, ly.y, ly.z, ly.w}, chy[4] = {hy.x, hy.y, hy.z, hy.w};
        const float clz[4] = {lz.x, lz.y, lz.z, lz.w}, chz[4] = {hz.x, hz.y, hz.z, hz.w};
        const int ch[4] = {e.x, e.y, e.z, e.w};
        for (int c = 0; c < 4; ++c) {
          if (ch[c] == kNoNode) continue;
          if (clx[c] > hi.x || chx[c] < lo.x || cly[c] > hi.y || chy[c] < lo.y || clz[c] > hi.z || chz[c] < lo.z)
            continue;
          if (sp < 64) stack[sp++] = ch[c];
          else atomicOr(sc.err, 1);
        }
      } else {
        const int code = ~node;
        const int first = code >> 3, cnt = (code & 7) + 1;
        for (int k = 0; k < cnt; ++k) {
          const float4* lt = sc.leaf + 3 * (size_t)(first + k);
          const float4 q0 = __ldg(lt), q1 = __ldg(lt + 1), q2 = __ldg(lt + 2);
          const int u = __float_as_int(q0.w);
          const int ou = __ldg(sc.tri_v + u).w;
          if (ou <= tv.w || ou >= nmesh) continue;
          const double3 B[3] = {make_double3(q0.x, q0.y, q0.z), make_double3(q1.x, q1.y, q1.z),
                                make_double3(q2.x, q2.y, q2.z)};
          double3 s0, s1;
          if (!tri_tri_segment(A, B, s0, s1)) continue;
          const double len = sqrt((s1.x - s0.x) * (s1.x - s0.x) + (s1.y - s0.y) * (s1.y - s0.y) +
                                  (s1.z - s0.z) * (s1.z - s0.z));
          if (!(len > 0.0)) continue;
          const int slot = atomicAdd(cb.count, 1);
          if (slot >= kCreaseCap) continue;
          cb.ra[slot] = make_float4((float)s0.x, (float)s0.y, (float)s0.z, (float)len);
          cb.rb[slot] = make_float4((float)s1.x, (float)s1.y, (float)s1.z, 0.f);
          cb.rtris[slot] = make_int2(t, u);
        }
      }
      if (sp == 0) break;
      node = stack[--sp];
    }
  }
}

// The extraction appends in whatever order the threads reach the counter; each segment's
// rank by its (triangle, triangle) pair puts them in one fixed order, so the samples (and
// the gradients) do not depend on scheduling.
__global__ void k_crease_order(CreaseBuf cb) {
  const int n = min(*cb.count, kCreaseCap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int2 ti = cb.rtris[i];
    const unsigned long long ki = ((unsigned long long)(unsigned)ti.x << 32) | (unsigned)ti.y;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const int2 tj = cb.rtris[j];
      const unsigned long long kj = ((unsigned long long)(unsigned)tj.x << 32) | (unsigned)tj.y;
      rank += kj < ki;
    }
    cb.a[rank] = cb.ra[i];
    cb.b[rank] = cb.rb[i];
    cb.tris[rank] = ti;
  }
}

// Segment lengths (0 past the segments found) as the masses of the length CDF.
__global__ void k_crease_mass(CreaseBuf cb, double* __restrict__ w) {
  const int n = min(*cb.count, kCreaseCap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kCreaseCap; i += gridDim.x * blockDim.x)
    w[i] = i < n ? (double)cb.a[i].w : 0.0;
}

// World-space gradients of the raster coordinates (J's rows) at camera-space point pc.
PSDR_D void raster_grad(const DevView& V, float3 pc, float3& gx, float3& gy) {
  const float* m = V.c2r;
  const float* r = V.w2c;
  const float wden = m[12] * pc.x + m[13] * pc.y + m[14] * pc.z + m[15];
  float3 g[2];
  for (int c = 0; c < 2; ++c) {
    const float u = (m[4 * c] * pc.x + m[4 * c + 1] * pc.y + m[4 * c + 2] * pc.z + m[4 * c + 3]) / wden;
    const float3 gpc = f3(m[4 * c] - u * m[12], m[4 * c + 1] - u * m[13], m[4 * c + 2] - u * m[14]) / wden;
    g[c] = f3(r[0] * gpc.x + r[4] * gpc.y + r[8] * gpc.z, r[1] * gpc.x + r[5] * gpc.y + r[9] * gpc.z,
              r[2] * gpc.x + r[6] * gpc.y + r[10] * gpc.z);
  }
  gx = g[0];
  gy = g[1];
}

// Crease point of sample i (stratified by length over all segments) and its projection.
struct CreasePt {
  float3 x, tang;
  float2 u;     // raster position
  float2 n;     // unit raster normal of the projected curve
  float rlen;   // raster length per unit world length along the curve
  float wgt;    // world length per sample (total length / N)
  int seg;
  bool ok;
};

PSDR_D CreasePt crease_point(const DevView& V, CreaseBuf cb, const double* mw, const double* mpre, long long i,
                             long long N, float xi) {
  CreasePt c;
  c.ok = false;
  if (!(mpre[kCreaseCap - 1] > 0.0)) return c;
  float t;
  double pmf;
  c.seg = (int)border_locate(mw, mpre, kCreaseCap, i, N, xi, t, pmf);
  if (!(pmf > 0.0)) return c;
  const float4 a = cb.a[c.seg], b = cb.b[c.seg];
  const float3 s0 = xyz(a), s1 = xyz(b);
  c.x = s0 + (s1 - s0) * t;
  c.tang = (s1 - s0) * (1.f / a.w);
  c.wgt = (float)(mw[c.seg] / (pmf * (double)N));
  float3 pc, pr;
  xform_pos(V.w2c, c.x, pc);
  xform_pos(V.c2r, pc, pr);
  if (!(pc.z < 0.f && pr.x > 0.f && pr.x < (float)V.W && pr.y > 0.f && pr.y < (float)V.H)) return c;
  c.u = make_float2(pr.x, pr.y);
  float3 gx, gy;
  raster_grad(V, pc, gx, gy);
  const float mx = dot(gx, c.tang), my = dot(gy, c.tang);
  c.rlen = sqrtf(mx * mx + my * my);
  if (!(c.rlen > 0.f)) return c;
  c.n = make_float2(-my / c.rlen, mx / c.rlen);
  c.ok = true;
  return c;
}

// Offset rays on both sides of the projected curve; both must reach the two meshes next to
// the crease point (else something hides it). Paths from both hits give L1 and L2 (slots
// 2s: the -n side, surface 1; 2s + 1: the +n side, surface 2). The offset is 5 ray epsilons
// (tmin) in world units: closer to the crease, rays leaving one surface skip the other
// within tmin and the rendered radiance there is not the image's limit at the crease.
constexpr float kCreaseOffset = 5.f * kTmin;  // world units
__global__ void __launch_bounds__(128) k_crease_init(WF w, const DevScene* __restrict__ scenes,
                                                     const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                     CreaseBuf cb, const double* __restrict__ mw,
                                                     const double* __restrict__ mpre, long long begin, int n,
                                                     long long N) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    HitRec hs[2];
    hs[0].tri = hs[1].tri = -1;
    const DevView& V = views[v];
    if (s < n && !V.ortho) {
      const long long i = begin + s;
      const DevScene& sc = scenes[V.scene];
      Rng rng = make_rng(kCreaseStream + (unsigned long long)i + w.seed);
      const CreasePt c = crease_point(V, cb, mw, mpre, i, N, rng.next_float());
      bool ok = c.ok;
      int flag = 0;
      if (ok) {
        const int2 tp = cb.tris[c.seg];
        const int oa = __ldg(sc.tri_v + tp.x).w, ob = __ldg(sc.tri_v + tp.y).w;
        const float tol = 10.f * kCreaseOffset;
        int objs[2];
        for (int side = 0; side < 2; ++side) {
          const float sg = (side ? kCreaseOffset : -kCreaseOffset) * c.rlen;  // pixels
          float3 pcam;
          xform_pos(V.r2c, f3(c.u.x + sg * c.n.x, c.u.y + sg * c.n.y, 1.0f), pcam);
          const float3 d = normalize(xform_dir(V.c2w, pcam));
          hs[side] = trace_closest(sc, V.pos, d, kTmin, INFINITY);
          objs[side] = -1;
          if (hs[side].tri >= 0) {
            const Surf x = make_surf(sc, hs[side].tri, hs[side].b1, hs[side].b2, V.pos);
            if (norm(x.p - c.x) < tol) objs[side] = x.obj;
          }
        }
        ok = objs[0] >= 0 && objs[1] >= 0 && objs[0] != objs[1] && (objs[0] == oa || objs[0] == ob) &&
             (objs[1] == oa || objs[1] == ob);
        flag = ok ? (objs[0] == oa ? 1 : 2) : 0;  // 1: surface 1 is the segment's first triangle
      }
      const int px = ok ? min(V.W - 1, (int)floorf(c.u.x)) : 0, py = ok ? min(V.H - 1, (int)floorf(c.u.y)) : 0;
      eb.a[s] = make_float4(__int_as_float(c.seg), c.wgt * c.rlen, c.n.x, c.n.y);
      eb.n[s] = make_float4(c.x.x, c.x.y, c.x.z, __int_as_float(py * V.W + px));
      eb.hb[s] = make_float4(0.f, 0.f, 0.f, __int_as_float(flag));
      for (int side = 0; side < 2; ++side) {
        const int slot = 2 * s + side;
        const Rng r = make_rng(kCreaseStream + 0x10000000ull + 2 * (unsigned long long)i + side + w.seed);
        w.rs[slot] = r.state;
        w.ri[slot] = r.inc;
        w.view[slot] = v;
        w.pix[slot] = -1;
        w.T[slot] = make_float4(1.f, 1.f, 1.f, 0.f);
        w.L[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
        w.cur[slot] = hit4(hs[side]);
        w.org[slot] = make_float4(V.pos.x, V.pos.y, V.pos.z, 0.f);
      }
      alive = ok;
    }
    for (int side = 0; side < 2; ++side) {
      const int k = warp_append(&w.cnt[0], alive);
      if (alive) w.q0[k] = 2 * s + side;
    }
  }
}

// Barycentric weights of point x in triangle tri (of its vertices v0, v1, v2).
PSDR_D float3 bary_of(const DevScene& sc, int tri, float3 x) {
  const float4* R = sc.tri + 6 * (size_t)tri;
  const float3 p0 = xyz(__ldg(R)), p1 = xyz(__ldg(R + 1)), p2 = xyz(__ldg(R + 2));
  const float3 e1 = p1 - p0, e2 = p2 - p0, q = x - p0;
  const float d11 = dot(e1, e1), d12 = dot(e1, e2), d22 = dot(e2, e2), q1 = dot(q, e1), q2 = dot(q, e2);
  const float den = d11 * d22 - d12 * d12;
  const float b1 = (d22 * q1 - d12 * q2) / den, b2 = (d11 * q2 - d12 * q1) / den;
  return f3(1.f - b1 - b2, b1, b2);
}

__global__ void __launch_bounds__(256) k_crease_final(WF w, const DevScene* __restrict__ scenes,
                                                      const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                      CreaseBuf cb, int n) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  GradAcc* const gpos = V.grad_pos;
  Own3 go;  // camera origin
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n || !V.dimage) continue;
    const int flag = __float_as_int(eb.hb[s].w);
    if (flag == 0) continue;
    const float4 a = eb.a[s], xn = eb.n[s];
    const float* gp = V.dimage + 3 * (size_t)__float_as_int(xn.w);
    const float3 L1 = xyz(w.L[2 * s]), L2 = xyz(w.L[2 * s + 1]);
    const float G1 = gp[0] * L1.x + gp[1] * L1.y + gp[2] * L1.z, G2 = gp[0] * L2.x + gp[1] * L2.y + gp[2] * L2.z;
    if (!isfinite(G1) || !isfinite(G2) || (G1 == 0.f && G2 == 0.f)) continue;
    const int2 tp = cb.tris[__float_as_int(a.x)];
    const int t1 = flag == 1 ? tp.x : tp.y, t2 = flag == 1 ? tp.y : tp.x;
    const float3 x = xyz(xn);
    const float3 n1 = normalize(xyz(__ldg(sc.tri + 6 * (size_t)t1 + 3)));
    const float3 n2 = normalize(xyz(__ldg(sc.tri + 6 * (size_t)t2 + 3)));
    float3 pc, gx, gy;
    xform_pos(V.w2c, x, pc);
    raster_grad(V, pc, gx, gy);
    const float3 wv = gx * a.z + gy * a.w;  // J^T n
    const float c = dot(n1, n2), sn2 = 1.f - c * c;
    if (!(sn2 > 1e-6f)) continue;
    const float w1 = dot(wv, n1), w2 = dot(wv, n2);
    const float A1 = (w1 - c * w2) / sn2, A2 = (w2 - c * w1) / sn2;
    const float K = a.y;
    const float3 a1 = (n1 * ((G1 - G2) * A1) - wv * G1) * K;
    const float3 a2 = (n2 * ((G1 - G2) * A2) + wv * G2) * K;
    if (!finite3(a1) || !finite3(a2)) continue;
    if (sc.grad_verts) {
      const float3 b1 = bary_of(sc, t1, x), b2 = bary_of(sc, t2, x);
      const int4 v1 = __ldg(sc.tri_v + t1), v2 = __ldg(sc.tri_v + t2);
      vert_add(sc, v1.x, a1 * b1.x);
      vert_add(sc, v1.y, a1 * b1.y);
      vert_add(sc, v1.z, a1 * b1.z);
      vert_add(sc, v2.x, a2 * b2.x);
      vert_add(sc, v2.y, a2 * b2.y);
      vert_add(sc, v2.z, a2 * b2.z);
    }
    if (gpos) go.add(-(a1 + a2));  // moving the camera by d is moving both surfaces by -d
  }
  if (gpos) go.put_warp(gpos);
}

// ------------------------------------------------------------------ BSDF jumps
// Unbiased estimator, DiffuseBsdfMaterial with roughness > 0 (diffuse_bsdf.cc:56-88).
// With N.L >= 0 and N.V >= 0 the rough-diffuse value jumps by color b (max(N.L, N.V) +
// 1e-5) where t = m.L crosses 0, m = V - (N.V) N: over the shading hemisphere, the half
// great circle through N perpendicular to m. The rendered value at x_k changes at
// Int_arc dF L_i (Ng.L) d/dtheta[m . L_att] / |m| dl, L_att the direction from the material
// point x_k to the material point x_{k+1} seen along L. One pass per depth k:
// k_jump_init replays camera sample i to its k-th vertex (stream i: 2 jitter draws, then
// per vertex the arc draw and two direction draws), draws the arc direction there
// (uniform, pdf 1/pi) and starts a path along it on stream 16 i + k; the path kernels
// estimate L_i with D - k bounces; k_jump_final scatters the adjoint of the carrier
// m . normalize(x_{k+1} - x_k). Side buffers: a = weight (prefix throughput x color x dF x
// (Ng.L) pi / (|m| spp)) and pixel; n = x_k's hit (w: 1 when the sample is live);
// hb = x_{k+1}'s hit; La = x_{k-1}'s hit (tri -1: the camera).
constexpr unsigned long long kJumpStreams = 16;  // max_bounce <= 16

__global__ void __launch_bounds__(128) k_jump_init(WF w, const DevScene* __restrict__ scenes,
                                                   const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                   long long begin, int n, int k, int D) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < n) {
      const long long i = begin + s;
      const DevView& V = views[v];
      const DevScene& sc = scenes[V.scene];
      Rng rng = make_rng((unsigned long long)i + w.seed);
      const float jx = rng.next_float(), jy = rng.next_float();
      const int pix = V.spp > 1 ? (int)(i / V.spp) : (int)i;
      float3 pc;
      xform_pos(V.r2c, f3(jx + (float)(pix % V.W), jy + (float)(pix / V.W), 1.0f), pc);
      float3 o = V.pos, d;
      if (V.ortho) {
        xform_pos(V.c2w, f3(pc.x, pc.y, 0.f), o);
        d = view_look_dir(V);
      } else {
        d = normalize(xform_dir(V.c2w, pc));
      }
      HitRec h = trace_closest(sc, o, d, kTmin, INFINITY);
      Surf x = make_surf(sc, h.tri, h.b1, h.b2, o);
      HitRec hp;
      hp.tri = -1; hp.b1 = hp.b2 = hp.t = 0.f;
      float3 T = f3(1.f, 1.f, 1.f);
      eb.n[s] = make_float4(__int_as_float(-1), 0.f, 0.f, __int_as_float(0));
      w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int kk = 1; kk <= k; ++kk) {
        if (!x.valid || x.is_light) break;
        const float u_arc = rng.next_float();
        const DevObj& ob = sc.objs[x.obj];
        const MatPt mp = mat_point(ob, x);
        if (kk == k) {
          const float nv = dot(mp.N, x.wi);
          const float3 m = x.wi - mp.N * nv;
          const float mlen = norm(m);
          if (!(mp.rough && mp.sigma > 0.f && nv >= 0.f && mlen > 1e-7f)) break;
          const float3 wa = normalize(cross(mp.N, m));
          float sp, cp;
          sincosf((u_arc - 0.5f) * kPi, &sp, &cp);
          const float3 L = normalize(mp.N * cp + wa * sp);
          const float nl = fmaxf(dot(mp.N, L), 0.f);
          const float a = 1.0f / (kPi + kOrenC * mp.sigma);
          const float dF = mp.sigma * a * (fmaxf(nl, nv) + kEps);
          const float3 wv = mul(T, mp.color) * (dF * dot(x.n, L) * kPi / (mlen * (float)V.spp));
          const HitRec ha = trace_closest(sc, x.p, L, kTmin, INFINITY);
          if (ha.tri < 0 || !finite3(wv)) break;
          eb.a[s] = make_float4(wv.x, wv.y, wv.z, __int_as_float(pix));
          eb.n[s] = make_float4(__int_as_float(h.tri), h.b1, h.b2, __int_as_float(1));
          eb.hb[s] = hit4(ha);
          eb.La[s] = hit4(hp);
          const Surf xa = make_surf(sc, ha.tri, ha.b1, ha.b2, x.p);
          if (k < D && !xa.is_light) {
            const Rng rl = make_rng((unsigned long long)i * kJumpStreams + (unsigned long long)k + w.seed);
            w.rs[s] = rl.state;
            w.ri[s] = rl.inc;
            w.view[s] = v;
            w.pix[s] = -1;
            w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
            w.cur[s] = hit4(ha);
            w.org[s] = make_float4(x.p.x, x.p.y, x.p.z, 0.f);
            alive = true;
          }
          break;
        }
        // continue the camera path: cosine sampling about the shading normal
        const float rx = rng.next_float(), ry = rng.next_float();
        float ct, st, sphi, cphi;
        const float3 wo = material_dir(x, mp.N, rx, ry, ct, st, sphi, cphi);
        const HitRec hn = trace_closest(sc, x.p, wo, kTmin, INFINITY);
        const Surf nx = make_surf(sc, hn.tri, hn.b1, hn.b2, x.p);
        if (!nx.valid) break;
        const float tmp = dot(nx.n, -wo) / nx.sqd;
        const float G = dot(x.n, wo) * tmp;
        const float pdf = ct * kInvPi * tmp;
        T = mul(T, surf_bsdf(sc, x, wo)) * (G / pdf);
        if (!finite3(T)) break;
        hp = h;
        h = hn;
        x = nx;
      }
    }
    const int kq = warp_append(&w.cnt[0], alive);
    if (alive) w.q0[kq] = s;
  }
}

__global__ void __launch_bounds__(256) k_jump_final(WF w, const DevScene* __restrict__ scenes,
                                                    const DevView* __restrict__ views, int v, EdgeBuf eb, int n,
                                                    int k) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  GradAcc* const gpos = V.grad_pos;
  Own3 go;  // camera origin
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    if (s >= n || !V.dimage) continue;
    const float4 hk = eb.n[s];
    if (__float_as_int(hk.w) != 1) continue;
    const float4 a = eb.a[s], hn = eb.hb[s], hp = eb.La[s];
    const int pix = __float_as_int(a.w);
    const int tp = __float_as_int(hp.x);
    // the vertex before x_k: the camera (k = 1) or the material point of the last hit
    float3 op = V.pos;
    if (tp >= 0) op = make_surf(sc, tp, hp.y, hp.z, V.pos).p;
    const int tk = __float_as_int(hk.x);
    float3 ok = op;
    if (tp < 0 && V.ortho) {
      const Surf x0 = make_surf(sc, tk, hk.y, hk.z, V.pos);
      ok = ortho_origin_rn(V, x0.p);
    }
    const Surf x = make_surf(sc, tk, hk.y, hk.z, ok);
    const int ta = __float_as_int(hn.x);
    const Surf xa = make_surf(sc, ta, hn.y, hn.z, x.p);
    if (!x.valid || !xa.valid) continue;
    const float3 Li = xa.is_light ? light_emit<true>(sc.lights[xa.light], xa) : xyz(w.L[s]);
    const float* gp = V.dimage + 3 * (size_t)pix;
    const float wgt = gp[0] * a.x * Li.x + gp[1] * a.y * Li.y + gp[2] * a.z * Li.z;
    if (!(wgt != 0.f) || !isfinite(wgt)) continue;
    // q = m . l, m = V - (N.V) N, l = normalize(x_{k+1} - x_k)
    const DevObj& ob = sc.objs[x.obj];
    const MatPt mp = mat_point(ob, x);
    const bool fixed_v = tp < 0 && V.ortho;  // orthographic primary vertex: V = -look
    const float3 Vd = fixed_v ? -view_look_dir(V) : x.wi;
    const float3 u = xa.p - x.p;
    const float r = norm(u);
    const float3 l = u / r;
    const float nv = dot(mp.N, Vd), nl = dot(mp.N, l);
    const float3 m = Vd - mp.N * nv;
    const float3 du = (m - l * dot(m, l)) * (wgt / r);
    MatAdj ma = zero_mat_adj();
    ma.N = (Vd * nl + l * nv) * (-wgt);
    if (!fixed_v) ma.V = (l - mp.N * nl) * wgt;
    if (!finite3(du) || !finite3(ma.N) || !finite3(ma.V)) continue;
    SurfAdj ax = zero_adj(), aa = zero_adj();
    aa.p = du;
    ax.p = -du;
    const float3 ao = mat_finalize(ob, x, mp, ma, ax);
    scatter_verts(sc, tk, hk.y, hk.z, x.front, ax);
    scatter_verts(sc, ta, hn.y, hn.z, xa.front, aa);
    if (tp >= 0) {
      SurfAdj ap = zero_adj();
      ap.p = ao;
      scatter_verts(sc, tp, hp.y, hp.z, true, ap);
    } else if (!fixed_v && gpos) {
      go.add(ao);
    }
  }
  if (gpos) go.put_warp(gpos);
}

// ------------------------------------------------------------------ direct edges
// path_integrator.cc:274-353 and the boundary_term / hit_triangle adjoint (:11-78).
// UNB (unbiased estimator, PRE=false): the same samples and edge/light visibility
// tests; the edge point x_b, light point y and receiver x_d lie on one line and the
// shadow boundary moves over the receiver at d_eff = dx_b - dx_d / lam - dy (1 - 1/lam),
// lam = |x_d - y| / |x_b - y|. Per camera connection: -T |n_y.w| / |x_b - y|^2 J_cam
// (d_eff . (w x e)) / (pdf_e pdf_y hc_density H W spp), e oriented by the edge's outward
// vector so that the occluding faces lie on the -(w x e) side, T = f_r(x_d) L_e times the
// albedos of the diffuse bounces between x_d and the camera-visible vertex.
// BSDF: the DiffuseBsdfMaterial instance (direction-dependent f at the receiver and
// along the bounce chain); the other instance is the DiffuseMaterial one.
// The draws of shadow-boundary sample i: hypercube cell and position (PRE: the three draws of
// preprocess round `round` in the cell's sampler stream; each round takes three), edge point
// x_b, light point y; returns the silhouette test (the edge's faces see y on opposite sides).
struct DirDraw {
  Rng rng;
  float hpdf, sx, pdf_e;
  int e;
  float3 p0, p1, out, nl, nr, xb, dir;
  LightSample ls;
};

template <bool PRE, bool UNB>
PSDR_D bool direct_draw(const WF& w, const DevScene& sc, const HCube& hc, int round, long long i, DirDraw& o) {
  float s3[3];
  o.hpdf = 1.f;
  if (PRE) {
    o.rng = make_rng((unsigned long long)i);
    o.rng.skip(3ull * (unsigned)round);
    const int r12 = hc.res[1] * hc.res[2];
    const int c0 = (int)(i / r12);
    const int rem = (int)(i - (long long)c0 * r12);
    const int c1 = rem / hc.res[2], c2 = rem - c1 * hc.res[2];
    const float d0 = o.rng.next_float(), d1 = o.rng.next_float(), d2 = o.rng.next_float();
    s3[0] = ((float)c0 + d0) * hc.unit[0];
    s3[1] = ((float)c1 + d1) * hc.unit[1];
    s3[2] = ((float)c2 + d2) * hc.unit[2];
  } else {
    o.rng = make_rng((unsigned long long)i + w.seed);
    s3[0] = o.rng.next_float(); s3[1] = o.rng.next_float(); s3[2] = o.rng.next_float();
    int cell;
    if (UNB) {
      double pm;
      cell = hc_cell_unb(hc, s3[2], pm);
      o.hpdf = (float)pm;
      s3[2] = o.rng.next_float();
    } else {
      cell = discrete_sample(hc.pmf, hc.cmf, hc.ncells, s3[2], o.hpdf);
    }
    if (!(o.hpdf > 0.f)) return false;
    const int r12 = hc.res[1] * hc.res[2];
    const int c0 = cell / r12, rem = cell - c0 * r12;
    const int c1 = rem / hc.res[2], c2 = rem - c1 * hc.res[2];
    s3[0] = (s3[0] + (float)c0) * hc.unit[0];
    s3[1] = (s3[1] + (float)c1) * hc.unit[1];
    s3[2] = (s3[2] + (float)c2) * hc.unit[2];
  }
  const int ne = *sc.n_edges;
  float pe;
  o.sx = s3[0];
  o.e = discrete_sample(sc.edge_pmf, sc.edge_cmf, ne, o.sx, pe);
  const float4 E0 = __ldg(sc.edge + 4 * (size_t)o.e), E1 = __ldg(sc.edge + 4 * (size_t)o.e + 1),
               E2 = __ldg(sc.edge + 4 * (size_t)o.e + 2), E3 = __ldg(sc.edge + 4 * (size_t)o.e + 3);
  o.p0 = xyz(E0);
  o.p1 = xyz(E1);
  o.out = f3(E1.w, E2.x, E2.y);
  o.nl = f3(E2.z, E2.w, E3.x);
  o.nr = f3(E3.y, E3.z, E3.w);
  o.xb = o.p0 + (o.p1 - o.p0) * o.sx;
  o.pdf_e = pe / E0.w;
  o.ls = sample_light(sc, s3[1], s3[2]);
  o.dir = normalize(o.xb - o.ls.y);
  return dot(o.nl, o.dir) * dot(o.nr, o.dir) < 0.f && norm(o.nl - o.nr) > kEps;
}

// The queue of the samples that pass the silhouette test: the ray origins' array (unused by these
// samples), which holds four entries per path of the tile.
PSDR_D int* direct_queue(const WF& w) { return reinterpret_cast<int*>(w.ro); }
constexpr int kDirectPerPath = 4;

// Index k of a preprocess launch: cell k % cells of round round0 + k / cells.
PSDR_D long long direct_index(bool pre, const HCube& hc, int round0, long long k, int& round) {
  if (!pre) return k;
  const int cells = hc.res[0] * hc.res[1] * hc.res[2];
  const long long r = k / cells;
  round = round0 + (int)r;
  return k - r * cells;
}

// First stage of the shadow-boundary samples [begin, begin + n): the draws and the
// silhouette test only; the samples that pass are queued (direct_queue, count in w.cnt[0]) for
// k_direct, whose warps then start with every lane on a sample that traces (most samples
// fail the test, and a lane that fails would idle while its warp traces).
template <bool PRE, bool UNB>
__global__ void __launch_bounds__(256) k_direct_pick(WF w, const DevScene* __restrict__ scenes,
                                                     const DevView* __restrict__ views, int v, long long begin,
                                                     int n, HCube hc, int round0) {
  const DevScene& sc = scenes[views[v].scene];
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n32; k += stride) {
    bool ok = false;
    if (k < n) {
      int round = 0;
      const long long i = direct_index(PRE, hc, round0, begin + k, round);
      DirDraw o;
      ok = direct_draw<PRE, UNB>(w, sc, hc, round, i, o);
    }
    const int q = warp_append(&w.cnt[0], ok);
    if (ok) direct_queue(w)[q] = k;
  }
}

template <bool PRE, bool UNB, bool BSDF>
__global__ void __launch_bounds__(128) k_direct(WF w, const DevScene* __restrict__ scenes,
                                                const DevView* __restrict__ views, int v, long long begin, HCube hc,
                                                int round0, float* mass, int spp) {
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  const int nq = w.cnt[0];
  const int stride = gridDim.x * blockDim.x;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
    const long long k = begin + direct_queue(w)[q];  // PRE: also the sample's entry in `mass`
    int round = 0;
    const long long i = direct_index(PRE, hc, round0, k, round);
    DirDraw o;
    if (!direct_draw<PRE, UNB>(w, sc, hc, round, i, o)) continue;
    Rng& rng = o.rng;
    const float hpdf = o.hpdf, sx = o.sx, pdf_e = o.pdf_e;
    const int e = o.e;
    const float3 p0 = o.p0, p1 = o.p1, out = o.out, xb = o.xb, dir = o.dir;
    const LightSample& ls = o.ls;
    // edge -> light: the same occlusion shortcut as the NEE rays (valid needs the
    // closest hit to be the light within sqrt(1e-5) of y)
    const float dist_l = norm(xb - ls.y);
    const HitRec hs = trace_closest(sc, xb, -dir, kTmin, dist_l * 1.0001f + 4e-3f, dist_l - 4e-3f);
    const Surf s0 = make_surf(sc, hs.tri, hs.b1, hs.b2, xb);
    if (!(s0.valid && s0.is_light && sqnorm(s0.p - ls.y) < kEps)) continue;
    const HitRec hd = trace_closest(sc, xb, dir, kTmin, INFINITY);
    const Surf d0 = make_surf(sc, hd.tri, hd.b1, hd.b2, xb);
    if (!(d0.valid && !d0.is_light)) continue;
    if (UNB) {
      // PRE: the guiding mass is the sum over camera connections of |weight| |w x e|
      // (the bounce chain draws from the sampler after its persisted state)
      if (!PRE && (!V.dimage || !sc.grad_verts)) continue;
      float3 ev = normalize(p1 - p0);
      if (dot(cross(dir, ev), out) < 0.f) ev = -ev;
      const float3 nsv = cross(dir, ev);
      const float dby = norm(xb - ls.y), lam = norm(d0.p - ls.y) / dby;
      const float cos_y = fabsf(dot(s0.n, dir));
      const float k0 = -cos_y / (dby * dby) / (pdf_e * ls.pdf * (float)V.H * (float)V.W);
      const float fxfy = view_fxfy(V);
      const float3 look = view_look(V);
      const DevLight& Lt = sc.lights[s0.light];
      // running throughput: the emission times pi f_r at every vertex the chain leaves
      // (DiffuseMaterial: f_r / pi of the receiver folded in up front, then the albedos)
      float3 T = light_emit<BSDF>(Lt, s0);
      if (!BSDF) {
        const DevObj& ob = sc.objs[d0.obj];
        T = mul(tex_rgb(ob.color, texel_offset(ob.color, d0.u, d0.v)) * kInvPi, T);
      }
      float wsum = 0.f, msum = 0.f;
      // camera connection of a vertex whose reflection hemisphere faces the camera:
      // T times its BSDF toward the camera times its camera Jacobian
      auto connect = [&](const Surf& v) {
        // from the camera position, or (orthographic) from v's foot on the camera plane
        // along the look direction
        const float3 co = V.ortho ? ortho_origin_rn(V, v.p) : V.pos;
        const float3 rel = v.p - co;
        const float dist = norm(rel);
        const float3 dir = V.ortho ? look : rel / dist;
        if (dot(v.n, dir) >= 0.f) return;
        int qx, qy;
        if (!project(V, v.p, qx, qy)) return;
        // the closest hit must be v itself: stop at the first hit short of it (same
        // outcome as a full closest-hit query followed by the distance test)
        const HitRec hc2 = trace_closest(sc, co, dir, kTmin, dist * 1.0001f + 4e-3f, dist - 4e-3f);
        const Surf iv = make_surf(sc, hc2.tri, hc2.b1, hc2.b2, co);
        if (!(iv.valid && !iv.is_light && sqnorm(iv.p - v.p) < kEps)) return;
        const float z = dot(rel, look);
        const float Jc = V.ortho ? fxfy * fabsf(dot(v.n, look)) : fxfy * fabsf(dot(v.n, rel)) / (z * z * z);
        const float3 Tf = BSDF ? mul(T, surf_bsdf(sc, v, -dir)) : T;
        if (PRE) {
          msum += norm(Tf) * fabsf(k0 * Jc);
        } else {
          const float* gp = V.dimage + 3 * ((size_t)qy * V.W + qx);
          wsum += (gp[0] * Tf.x + gp[1] * Tf.y + gp[2] * Tf.z) * (k0 * Jc);
        }
      };
      connect(d0);
      // the change of the radiance leaving the receiver, carried to the camera through
      // up to max_bounce - 1 bounces cosine-sampled about the geometric normal (each
      // multiplies pi f_r: G / pdf = pi)
      Surf v = d0;
      for (int j = 1; j < w.D; ++j) {
        const float ru = rng.next_float(), rv = rng.next_float();
        float ct, st, sp, cp;
        const float3 wo = diffuse_dir(v.n, v.t, ru, rv, ct, st, sp, cp);
        const HitRec hn = trace_closest(sc, v.p, wo, kTmin, INFINITY);
        const Surf nx = make_surf(sc, hn.tri, hn.b1, hn.b2, v.p);
        if (!nx.valid || nx.is_light) break;
        if (BSDF) {
          T = mul(T, surf_bsdf(sc, v, wo)) * kPi;
        } else {
          const DevObj& on = sc.objs[nx.obj];
          T = mul(T, tex_rgb(on.color, texel_offset(on.color, nx.u, nx.v)));
        }
        connect(nx);
        v = nx;
      }
      if (PRE) {
        const float m = msum * norm(nsv);
        if (isfinite(m)) mass[k] = m;
        continue;
      }
      const float3 a = nsv * (wsum / (hpdf * (float)hc.ncells * (float)spp));
      if (!finite3(a) || wsum == 0.f) continue;
      const int2 evv = __ldg(sc.edge_v + e);
      vert_add(sc, evv.x, a * (1.f - sx));
      vert_add(sc, evv.y, a * sx);
      const int4 td = __ldg(sc.tri_v + hd.tri);
      const float3 ad = a * (-1.f / lam);
      vert_add(sc, td.x, ad * (1.f - hd.b1 - hd.b2));
      vert_add(sc, td.y, ad * hd.b1);
      vert_add(sc, td.z, ad * hd.b2);
      const int4 tl = __ldg(sc.tri_v + ls.tri);
      const float3 al = a * (1.f / lam - 1.f);
      vert_add(sc, tl.x, al * (1.f - ls.su - ls.sv));
      vert_add(sc, tl.y, al * ls.su);
      vert_add(sc, tl.z, al * ls.sv);
      continue;
    }
    int px, py;
    if (!project(V, d0.p, px, py)) continue;
    float3 co = V.pos, cd;
    if (V.ortho) {
      co = ortho_origin_rn(V, d0.p);
      cd = view_look_dir(V);
    } else {
      cd = normalize(d0.p - V.pos);
    }
    const HitRec h2 = trace_closest(sc, co, cd, kTmin, INFINITY);
    const Surf i2 = make_surf(sc, h2.tri, h2.b1, h2.b2, co);
    if (!(i2.valid && !i2.is_light && sqnorm(i2.p - d0.p) < kEps)) continue;
    const float pdf_xw = s0.sqd * pdf_e * ls.pdf / dot(s0.n, dir);
    // boundary_term (detached quantities)
    const float3 xs = s0.p, xd = d0.p, ns = s0.n, nd = d0.n;
    const float3 rb = xb - xs;
    const float3 db = normalize(rb);
    float3 ev = normalize(p1 - p0);
    if (dot(cross(db, ev), out) < 0.f) ev = -ev;
    const float3 npl = cross(db, ev);
    const float3 ep = cross(nd, npl);
    const float cos_s = fabsf(dot(ns, db));
    const float cos_b = dot(ev, db), cos_d = dot(ep, db);
    const float sb2 = 1.f - cos_b * cos_b, sd2 = 1.f - cos_d * cos_d;
    const float sin_b = sb2 > 0.f ? sqrtf(sb2) : 0.f, sin_d = sd2 > 0.f ? sqrtf(sd2) : 0.f;
    const float len_sb = norm(xb - xs), len_sd = norm(xd - xs);
    const float Jb = len_sd * len_sb * sin_b / (sin_d * cos_s);
    const float dG = cos_s * dot(nd, -db) / (len_sd * len_sd);
    const DevLight& Lt = sc.lights[s0.light];
    const float3 Ts = light_emit<BSDF>(Lt, s0);
    float3 Td;
    if (BSDF) {
      Td = surf_bsdf(sc, d0, -cd);
    } else {
      const DevObj& ob = sc.objs[d0.obj];
      Td = tex_rgb(ob.color, texel_offset(ob.color, d0.u, d0.v)) * kInvPi;
    }
    if (PRE) {
      float3 val = mul(mul(f3(dG, dG, dG) * Jb / pdf_xw, Ts), Td);
      if (!finite3(val)) continue;
      val.x = val.x < kEps ? kEps : val.x;
      val.y = val.y < kEps ? kEps : val.y;
      val.z = val.z < kEps ? kEps : val.z;
      mass[k] = norm(val);
    } else {
      const float3 nep = cross(nd, ep);
      const float3 z = mul(mul(mul(f3(0.f, 0.f, 0.f), nep * dG) * Jb / pdf_xw, Ts), Td);
      if (!finite3(z) || !V.dimage || !sc.grad_verts) continue;
      const float* gp = V.dimage + 3 * ((size_t)py * V.W + px);
      const float c = Jb / pdf_xw * dG / (hpdf * (float)spp);
      const float3 wv = f3(gp[0] * nep.x * Ts.x * Td.x, gp[1] * nep.y * Ts.y * Td.y, gp[2] * nep.z * Ts.z * Td.z) * c;
      // hit_triangle(xs, d, xd, ep, nep) adjoint w.r.t. d
      const float3 e1 = ep, e2 = nep;
      const float3 T = xs - xd;
      const float3 P = cross(db, e2), Q = cross(T, e1);
      const float det = dot(P, e1);
      const float dcl = fminf(fmaxf(det, kEps), 1.f - kEps);
      const float inv = 1.f / dcl;
      const float u = dot(P, T) * inv, vv = dot(Q, db) * inv;
      const float au = dot(wv, e1), avv = dot(wv, e2);
      float3 ad = cross(e2, T) * (au * inv) + Q * (avv * inv);
      if (det > kEps && det < 1.f - kEps) ad += cross(e2, e1) * (-(au * u + avv * vv) * inv);
      const float3 axb = (ad - db * dot(db, ad)) / norm(rb);
      const int2 evv = __ldg(sc.edge_v + e);
      vert_add(sc, evv.x, axb * (1.f - sx));
      vert_add(sc, evv.y, axb * sx);
    }
  }
}

// ------------------------------------------------------------------ indirect shadow boundaries
// Unbiased estimator: shadow boundaries of light that other surfaces reflect. The geometry
// is the shadow-boundary term's with the light point replaced by the first surface y seen
// from the edge point x_b in a direction w sampled inside the edge's silhouette lune: the
// directions w = cos(t) e + sin(t) m(psi) for which exactly one of the two faces at the edge
// faces w, two opposite wedges of angle alpha (the angle between the face normals) around
// the edge, solid angle 4 alpha, sampled uniformly (pdf 1 / (4 alpha)). Measured this way
// the geometric factor cos_y / |x_b - y|^2 of the area form cancels, so sample weights stay
// bounded. y must be a mesh surface (light sources are the shadow-boundary term's); the
// receiver x_d is the first hit from x_b away from y and must be seen by the camera. The
// radiance leaving y toward x_b is a path traced from y with max_bounce - 1 bounces (y is
// the second vertex of the camera path through x_d); the boundary moves over the receiver at
// d_eff = dx_b - dx_d / lam - dy (1 - 1/lam) as for the light. Receivers that reach the
// camera only through further bounces are left out (their source paths would be one bounce
// shorter per chain vertex).
constexpr unsigned long long kIndirectStream = 0xE0000000ull;  // streams of the source paths
// Its per-sample variance is an order of magnitude below the light-source term's, so it takes
// a quarter of the shadow-boundary samples and a quarter of the guiding cells along the edge
// axis.
constexpr int kIndirectSampleDiv = 4, kIndirectCellDiv = 4;
// Preprocess rounds of the unbiased estimator's light-source shadow-boundary guide per
// requested round. One sample per cell (the reference's preprocess) leaves most of the 360k
// cells of the default guide with a single noisy estimate; the term's per-sample weights
// are heavy-tailed, and with four samples per cell its standard deviation on the 512²
// icosphere workload drops by a third (about 2.5x less variance) for ~1 ms.
constexpr int kDirectGuideRounds = 4;
// Preprocess rounds of the shadow-boundary guide that run in one launch (a launch of 360k cells
// traces few enough samples to be bound by its longest chain of rays).
constexpr int kGuideRounds = 8;

// Direction of lune coordinates (u2, u3) in [0, 1)^2 at an edge with unit direction ev and
// unit face normals nl, nr (both perpendicular to ev); alpha gets the wedge angle.
PSDR_D float3 lune_dir(float3 ev, float3 nl, float3 nr, float u2, float u3, float& alpha) {
  const float3 b = cross(ev, nl);
  const float ar = atan2f(dot(nr, b), dot(nr, nl));  // nr's angle from nl around ev
  alpha = fabsf(ar);
  const bool second = u2 >= 0.5f;
  const float t = second ? 2.f * u2 - 1.f : 2.f * u2;
  const float psi = (second ? -0.5f * kPi : 0.5f * kPi) + t * ar;
  const float ct = 1.f - 2.f * u3, st = sqrtf(fmaxf(0.f, 1.f - ct * ct));
  float sp, cp;
  sincosf(psi, &sp, &cp);
  return ev * ct + (nl * cp + b * sp) * st;
}

// PRE: guiding mass per hypercube cell (|k0 J_cam| |f_r(x_d)| |w x e|; the source radiance
// is not known yet). Otherwise: one sample per thread, side buffers for k_indirect_final and
// a path from y (slot s) whose radiance toward x_b the depth loop computes.
template <bool PRE>
__global__ void __launch_bounds__(128) k_indirect(WF w, const DevScene* __restrict__ scenes,
                                                  const DevView* __restrict__ views, int v, EdgeBuf eb,
                                                  long long begin, int n, HCube hc, int round, float* mass) {
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (n + 31) & ~31;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n32; s += stride) {
    bool alive = false;
    if (s < n) {
      const long long i = begin + s;
      Rng rng;
      float s3[3], hpdf = 1.f;
      bool ok = true;
      if (PRE) {
        if (round == 0) rng = make_rng(kIndirectStream + (unsigned long long)i);
        else { rng.state = w.rs[s]; rng.inc = w.ri[s]; }
        const int r12 = hc.res[1] * hc.res[2];
        const int c0 = (int)(i / r12);
        const int rem = (int)(i - (long long)c0 * r12);
        const int c1 = rem / hc.res[2], c2 = rem - c1 * hc.res[2];
        const float d0 = rng.next_float(), d1 = rng.next_float(), d2 = rng.next_float();
        s3[0] = ((float)c0 + d0) * hc.unit[0];
        s3[1] = ((float)c1 + d1) * hc.unit[1];
        s3[2] = ((float)c2 + d2) * hc.unit[2];
        w.rs[s] = rng.state;
        w.ri[s] = rng.inc;
      } else {
        rng = make_rng(kIndirectStream + (unsigned long long)i + w.seed);
        s3[0] = rng.next_float(); s3[1] = rng.next_float(); s3[2] = rng.next_float();
        double pm;
        const int cell = hc_cell_unb(hc, s3[2], pm);
        hpdf = (float)pm;
        ok = pm > 0.0;
        s3[2] = rng.next_float();
        const int r12 = hc.res[1] * hc.res[2];
        const int c0 = cell / r12, rem = cell - c0 * r12;
        const int c1 = rem / hc.res[2], c2 = rem - c1 * hc.res[2];
        s3[0] = (s3[0] + (float)c0) * hc.unit[0];
        s3[1] = (s3[1] + (float)c1) * hc.unit[1];
        s3[2] = (s3[2] + (float)c2) * hc.unit[2];
      }
      const int ne = *sc.n_edges;
      float sx = s3[0], pe;
      const int e = ok ? discrete_sample(sc.edge_pmf, sc.edge_cmf, ne, sx, pe) : 0;
      float3 xb = f3(0.f, 0.f, 0.f), nsv = f3(0.f, 0.f, 0.f);
      HitRec hy, hd;
      hy.tri = hd.tri = -1;
      hy.b1 = hy.b2 = 0.f;
      if (ok) {
        const float4 E0 = __ldg(sc.edge + 4 * (size_t)e), E1 = __ldg(sc.edge + 4 * (size_t)e + 1),
                     E2 = __ldg(sc.edge + 4 * (size_t)e + 2), E3 = __ldg(sc.edge + 4 * (size_t)e + 3);
        const float3 p0 = xyz(E0), p1 = xyz(E1);
        const float3 out = f3(E1.w, E2.x, E2.y), nl = f3(E2.z, E2.w, E3.x), nr = f3(E3.y, E3.z, E3.w);
        xb = p0 + (p1 - p0) * sx;
        const float pdf_e = pe / E0.w;
        float3 ev = normalize(p1 - p0);
        float alpha;
        const float3 wy = lune_dir(ev, nl, nr, s3[1], s3[2], alpha);  // toward the source
        const float3 dir = -wy;                                       // from the source through x_b
        ok = alpha > kEps && dot(nl, dir) * dot(nr, dir) < 0.f;
        if (ok) {
          hy = trace_closest(sc, xb, wy, kTmin, INFINITY);
          const Surf s0 = make_surf(sc, hy.tri, hy.b1, hy.b2, xb);
          ok = s0.valid && !s0.is_light;
          if (ok) {
            hd = trace_closest(sc, xb, dir, kTmin, INFINITY);
            const Surf d0 = make_surf(sc, hd.tri, hd.b1, hd.b2, xb);
            ok = d0.valid && !d0.is_light;
            if (ok) {
              if (dot(cross(dir, ev), out) < 0.f) ev = -ev;
              nsv = cross(dir, ev);
              // the receiver seen by the camera (perspective views)
              const float3 rel = d0.p - V.pos;
              const float dist = norm(rel);
              const float3 cd = rel / dist;
              int qx = 0, qy = 0;
              ok = !V.ortho && dot(d0.n, cd) < 0.f && project(V, d0.p, qx, qy);
              if (ok) {
                const HitRec hc2 = trace_closest(sc, V.pos, cd, kTmin, dist * 1.0001f + 4e-3f, dist - 4e-3f);
                const Surf iv = make_surf(sc, hc2.tri, hc2.b1, hc2.b2, V.pos);
                ok = iv.valid && !iv.is_light && sqnorm(iv.p - d0.p) < kEps;
              }
              if (ok) {
                const float3 look = view_look(V);
                const float z = dot(rel, look);
                const float Jc = view_fxfy(V) * fabsf(dot(d0.n, rel)) / (z * z * z);
                const float k0 = -4.f * alpha / (pdf_e * (float)V.H * (float)V.W) * Jc;
                const float lam = norm(d0.p - s0.p) / norm(xb - s0.p);
                if (PRE) {
                  const float3 fr = surf_bsdf(sc, d0, -cd);
                  const float m = fabsf(k0) * norm(fr) * norm(nsv);
                  if (isfinite(m)) mass[i] = mass[i] + m;
                  ok = false;  // no path in the preprocess
                } else {
                  eb.a[s] = make_float4(__int_as_float(e), sx, hpdf, __int_as_float(qy * V.W + qx));
                  eb.n[s] = make_float4(__int_as_float(hy.tri), hy.b1, hy.b2, k0);
                  eb.hb[s] = make_float4(__int_as_float(hd.tri), hd.b1, hd.b2, lam);
                  eb.La[s] = make_float4(nsv.x, nsv.y, nsv.z, 0.f);
                }
              }
            }
          }
        }
      }
      if (!PRE) {
        eb.La[s].w = __int_as_float(ok ? 1 : 0);
        const Rng r = make_rng(kIndirectStream + 0x10000000ull + (unsigned long long)i + w.seed);
        w.rs[s] = r.state;
        w.ri[s] = r.inc;
        w.view[s] = v;
        w.pix[s] = -1;
        w.T[s] = make_float4(1.f, 1.f, 1.f, 0.f);
        w.L[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        w.cur[s] = make_float4(__int_as_float(ok ? hy.tri : -1), hy.b1, hy.b2, 0.f);
        w.org[s] = make_float4(xb.x, xb.y, xb.z, 0.f);
        alive = ok;
      }
    }
    if (!PRE) {
      const int k = warp_append(&w.cnt[0], alive);
      if (alive) w.q0[k] = s;
    }
  }
}

// N: the samples of the view (the per-sample estimate is divided by N / (H W)).
__global__ void __launch_bounds__(128) k_indirect_final(WF w, const DevScene* __restrict__ scenes,
                                                        const DevView* __restrict__ views, int v, EdgeBuf eb, int n,
                                                        float cells, long long N) {
  const DevView& V = views[v];
  const DevScene& sc = scenes[V.scene];
  const int stride = gridDim.x * blockDim.x;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += stride) {
    if (!V.dimage || !sc.grad_verts) continue;
    const float4 nv = eb.La[s];
    if (__float_as_int(nv.w) != 1) continue;
    const float4 a = eb.a[s], yn = eb.n[s], hd = eb.hb[s];
    const float3 Lo = xyz(w.L[s]);
    const int dtri = __float_as_int(hd.x);
    const float4 E0 = __ldg(sc.edge + 4 * (size_t)__float_as_int(a.x)), E1 = __ldg(sc.edge + 4 * (size_t)__float_as_int(a.x) + 1);
    const float3 xb = xyz(E0) + (xyz(E1) - xyz(E0)) * a.y;
    // the receiver lit from the edge side, reflecting toward the camera
    const Surf d0 = make_surf(sc, dtri, hd.y, hd.z, xb);
    const float3 fr = surf_bsdf(sc, d0, normalize(V.pos - d0.p));
    const float* gp = V.dimage + 3 * (size_t)__float_as_int(a.w);
    const float wsum = (gp[0] * fr.x * Lo.x + gp[1] * fr.y * Lo.y + gp[2] * fr.z * Lo.z) * yn.w;
    const float3 ag = xyz(nv) * (wsum / (a.z * cells * (float)((double)N / ((double)V.H * V.W))));
    if (!finite3(ag) || wsum == 0.f) continue;
    const int e = __float_as_int(a.x);
    const float sx = a.y, lam = hd.w;
    const int2 evv = __ldg(sc.edge_v + e);
    vert_add(sc, evv.x, ag * (1.f - sx));
    vert_add(sc, evv.y, ag * sx);
    const int4 td = __ldg(sc.tri_v + dtri);
    const float3 ad = ag * (-1.f / lam);
    vert_add(sc, td.x, ad * (1.f - hd.y - hd.z));
    vert_add(sc, td.y, ad * hd.y);
    vert_add(sc, td.z, ad * hd.z);
    const int4 ty = __ldg(sc.tri_v + __float_as_int(yn.x));
    const float3 ay = ag * (1.f / lam - 1.f);
    vert_add(sc, ty.x, ay * (1.f - yn.y - yn.z));
    vert_add(sc, ty.y, ay * yn.y);
    vert_add(sc, ty.z, ay * yn.z);
  }
}

// ------------------------------------------------------------------ small utilities
__global__ void k_mass_rounds(const float* __restrict__ rm, int cells, int rounds, float* __restrict__ mass) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cells) return;
  float m = mass[i];
  for (int r = 0; r < rounds; ++r) m = m + rm[(size_t)r * cells + i];
  mass[i] = m;
}
__global__ void k_mass_cdf(const float* __restrict__ mass, int n, double* __restrict__ w) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) w[i] = (double)mass[i];
}
// Unbiased estimator: add a uniform share (a quarter of the mean mass, 20% of the
// samples) to every cell, bounding sample weights at 5x the uniform one.
__global__ void k_mass_floor(float* __restrict__ mass, const double* __restrict__ pre, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double tot = pre[n - 1];
  const float f = tot > 0.0 ? (float)(0.25 * tot / (double)n) : 1.0f;
  mass[i] = mass[i] + f;
}
__global__ void k_mass_finalize(const double* __restrict__ w, const double* __restrict__ pre, int n,
                                float* __restrict__ pmf, float* __restrict__ cmf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double tot = pre[n - 1];
  if (!(tot > 0.0)) { pmf[i] = 0.f; cmf[i] = 1.f; return; }
  pmf[i] = (float)(w[i] / tot);
  cmf[i] = (float)(pre[i] / tot);
}
__global__ void k_grad_out(const GradAcc* __restrict__ acc, float* __restrict__ out, long long n, int accumulate) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const longlong2 a = __ldg(reinterpret_cast<const longlong2*>(acc) + i);
  out[i] = (accumulate ? out[i] : 0.f) + (float)acc_value(a.x, a.y);
}


// ================================================================== host side
namespace {
// per_sm caps the grid; kEachBlock leaves it uncapped. The kernels that trace a ray per thread
// (k_camera and the *_init of the boundary terms) take a block per 128 samples: threads end
// at very different times, and a grid of a few blocks per SM, each over several batches, ends
// with most SMs waiting for their last blocks. k_camera 2.65 -> 2.03 ms (1.31 M triangles,
// 1024^2 x 16 spp), k_edge_init 1.15 -> 1.02 and k_border_init 0.43 -> 0.37 ms (512^2 x 32 spp
// step) against 8 blocks of 256 per SM. k_direct, whose queue is mostly shorter than its
// launch, takes 64 blocks per SM (1.48 -> 1.33 ms against 16). k_shade and k_accum stay at 8:
// every thread does the same work, and uncapped they take 10-15 % longer on a single job.
constexpr int kEachBlock = 1 << 20;
inline int grid_for(long long n, int threads, int per_sm) {
  const long long want = (n + threads - 1) / threads;
  const long long cap = (long long)num_sms() * per_sm;
  return (int)std::max<long long>(1, std::min(want, cap));
}
}  // namespace

// camera.h:7-64, :111-124; psdr.cc:24-29 (near -0.01, far -1000). Row-major floats.
void make_view(const psdr_camera_desc& c, int spp, DevView& v) {
  auto nrm = [](double* a) { double n = std::sqrt(a[0]*a[0]+a[1]*a[1]+a[2]*a[2]); a[0]/=n; a[1]/=n; a[2]/=n; };
  auto crs = [](const double* a, const double* b, double* r) {
    r[0] = a[1]*b[2]-a[2]*b[1]; r[1] = a[2]*b[0]-a[0]*b[2]; r[2] = a[0]*b[1]-a[1]*b[0]; };
  double o[3] = {c.look_from[0], c.look_from[1], c.look_from[2]};
  double t[3] = {c.look_at[0], c.look_at[1], c.look_at[2]};
  double u[3] = {c.up[0], c.up[1], c.up[2]};
  double dir[3] = {o[0]-t[0], o[1]-t[1], o[2]-t[2]};
  nrm(dir); nrm(u);
  double right[3], nup[3];
  crs(u, dir, right);
  crs(dir, right, nup);
  double cw[4][4] = {{0}}, cs[4][4] = {{0}}, sr[4][4] = {{0}}, tr[4][4] = {{0}};
  for (int i = 0; i < 3; ++i) { cw[i][0] = right[i]; cw[i][1] = nup[i]; cw[i][2] = dir[i]; cw[i][3] = o[i]; }
  cw[3][3] = 1;
  const double nearv = -0.01, farv = -1000.0, inv_nf = 1.0 / (nearv - farv);
  v.ortho = c.type == PSDR_CAM_ORTHOGRAPHIC;
  if (v.ortho) {
    // camera.h:19-31 orthographic(left, right, bottom, top, near, far) = scale * translate
    // over the view box of camera.h:290-300 (width fov = view_width, height width H / W)
    const double hw = (double)c.fov / 2, hh = (double)c.height * hw / (double)c.width;
    cs[0][0] = 2 / (2 * hw);
    cs[1][1] = 2 / (2 * hh);
    cs[2][2] = 2 / (nearv - farv);
    cs[2][3] = cs[2][2] * (-(nearv + farv) / 2);
    cs[3][3] = 1;
  } else {
    const double cot = 1.0 / std::tan((double)c.fov * 0.5);
    cs[0][0] = -cot; cs[1][1] = -cot; cs[2][2] = (nearv + farv) * inv_nf; cs[2][3] = -2 * farv * nearv * inv_nf;
    cs[3][2] = 1;
  }
  sr[0][0] = 0.5 * c.width; sr[1][1] = -0.5 * c.height; sr[2][2] = 1; sr[3][3] = 1;
  tr[0][0] = tr[1][1] = tr[2][2] = tr[3][3] = 1; tr[0][3] = 1; tr[1][3] = -1;
  auto mm = [](const double a[4][4], const double b[4][4], double r[4][4]) {
    for (int i = 0; i < 4; ++i) for (int j = 0; j < 4; ++j) { double s = 0; for (int k = 0; k < 4; ++k) s += a[i][k] * b[k][j]; r[i][j] = s; } };
  auto inv = [](const double a[4][4], double r[4][4]) {
    double m[4][8];
    for (int i = 0; i < 4; ++i) for (int j = 0; j < 8; ++j) m[i][j] = j < 4 ? a[i][j] : (j - 4 == i ? 1.0 : 0.0);
    for (int col = 0; col < 4; ++col) {
      int p = col;
      for (int rr = col + 1; rr < 4; ++rr) if (std::fabs(m[rr][col]) > std::fabs(m[p][col])) p = rr;
      for (int j = 0; j < 8; ++j) std::swap(m[col][j], m[p][j]);
      const double iv = 1.0 / m[col][col];
      for (int j = 0; j < 8; ++j) m[col][j] *= iv;
      for (int rr = 0; rr < 4; ++rr) { if (rr == col) continue; const double f = m[rr][col]; for (int j = 0; j < 8; ++j) m[rr][j] -= f * m[col][j]; }
    }
    for (int i = 0; i < 4; ++i) for (int j = 0; j < 4; ++j) r[i][j] = m[i][j + 4];
  };
  double t1[4][4], c2r[4][4], r2c[4][4], w2c[4][4];
  mm(sr, tr, t1);
  mm(t1, cs, c2r);
  inv(c2r, r2c);
  inv(cw, w2c);
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      v.r2c[4 * i + j] = (float)r2c[i][j];
      v.c2w[4 * i + j] = (float)cw[i][j];
      v.w2c[4 * i + j] = (float)w2c[i][j];
      v.c2r[4 * i + j] = (float)c2r[i][j];
    }
  v.pos = make_float3(c.look_from[0], c.look_from[1], c.look_from[2]);
  v.H = c.height;
  v.W = c.width;
  v.spp = spp;
  v.scene = 0;
  v.image = nullptr;
  v.dimage = nullptr;
  v.grad_pos = nullptr;
  v.grad_lens = nullptr;
  v.scene_ntri = 0;
}

// Forward-mode derivative of the raster-to-direction map M = C diag(2 t / W, -2 t / H, -1),
// t = tan(fov / 2), C = (right, up, dir) built as camera.h:35-52 does (dir = normalize(from -
// at), right = cross(normalize(up), dir) unnormalised, up' = cross(dir, right)), with
// respect to the ten camera parameters (from, at, up, fov); P_j = M^-1 dM/dtheta_j.
namespace {
struct Dual10 {
  double v;
  double d[10];
};
Dual10 dconst(double v) { Dual10 r{v, {0}}; return r; }
Dual10 dvar(double v, int j) { Dual10 r = dconst(v); r.d[j] = 1.0; return r; }
Dual10 operator+(const Dual10& a, const Dual10& b) { Dual10 r{a.v + b.v, {0}}; for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] + b.d[j]; return r; }
Dual10 operator-(const Dual10& a, const Dual10& b) { Dual10 r{a.v - b.v, {0}}; for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] - b.d[j]; return r; }
Dual10 operator*(const Dual10& a, const Dual10& b) { Dual10 r{a.v * b.v, {0}}; for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] * b.v + a.v * b.d[j]; return r; }
Dual10 operator*(const Dual10& a, double k) { Dual10 r{a.v * k, {0}}; for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] * k; return r; }
Dual10 dinv(const Dual10& a) { Dual10 r{1.0 / a.v, {0}}; for (int j = 0; j < 10; ++j) r.d[j] = -a.d[j] / (a.v * a.v); return r; }
Dual10 dsqrt(const Dual10& a) { Dual10 r{std::sqrt(a.v), {0}}; for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] / (2.0 * r.v); return r; }
Dual10 dtan(const Dual10& a) {
  const double t = std::tan(a.v);
  Dual10 r{t, {0}};
  for (int j = 0; j < 10; ++j) r.d[j] = a.d[j] * (1.0 + t * t);
  return r;
}
void dnormalize(Dual10* a) {
  const Dual10 n = dinv(dsqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]));
  for (int k = 0; k < 3; ++k) a[k] = a[k] * n;
}
void dcross(const Dual10* a, const Dual10* b, Dual10* r) {
  r[0] = a[1] * b[2] - a[2] * b[1];
  r[1] = a[2] * b[0] - a[0] * b[2];
  r[2] = a[0] * b[1] - a[1] * b[0];
}
bool inv3(const double* m, double* r) {
  const double c00 = m[4] * m[8] - m[5] * m[7], c01 = m[5] * m[6] - m[3] * m[8], c02 = m[3] * m[7] - m[4] * m[6];
  const double det = m[0] * c00 + m[1] * c01 + m[2] * c02;
  if (!(std::fabs(det) > 0.0) || !std::isfinite(det)) return false;
  const double id = 1.0 / det;
  r[0] = c00 * id; r[1] = (m[2] * m[7] - m[1] * m[8]) * id; r[2] = (m[1] * m[5] - m[2] * m[4]) * id;
  r[3] = c01 * id; r[4] = (m[0] * m[8] - m[2] * m[6]) * id; r[5] = (m[2] * m[3] - m[0] * m[5]) * id;
  r[6] = c02 * id; r[7] = (m[1] * m[6] - m[0] * m[7]) * id; r[8] = (m[0] * m[4] - m[1] * m[3]) * id;
  return true;
}
}  // namespace

void lens_chain(const psdr_camera_desc& c, LensChain& out, double* m9) {
  Dual10 from[3], at[3], up[3];
  for (int k = 0; k < 3; ++k) {
    from[k] = dvar(c.look_from[k], k);
    at[k] = dvar(c.look_at[k], 3 + k);
    up[k] = dvar(c.up[k], 6 + k);
  }
  const Dual10 fov = dvar(c.fov, 9);
  Dual10 dir[3] = {from[0] - at[0], from[1] - at[1], from[2] - at[2]};
  dnormalize(dir);
  dnormalize(up);
  Dual10 right[3], nup[3];
  dcross(up, dir, right);
  dcross(dir, right, nup);
  const Dual10 t = dtan(fov * 0.5);
  const Dual10 sx = t * (2.0 / c.width), sy = t * (-2.0 / c.height);
  Dual10 M[9];
  for (int i = 0; i < 3; ++i) {
    M[3 * i] = right[i] * sx;
    M[3 * i + 1] = nup[i] * sy;
    M[3 * i + 2] = dir[i] * -1.0;
  }
  double m[9], mi[9];
  for (int q = 0; q < 9; ++q) m[q] = M[q].v;
  if (m9) std::copy(m, m + 9, m9);
  PSDR_CHECK(inv3(m, mi), "degenerate camera basis (look_at equals look_from, or up parallel to the view)");
  for (int j = 0; j < 10; ++j)
    for (int r = 0; r < 3; ++r)
      for (int q = 0; q < 3; ++q) {
        double acc = 0.0;
        for (int k = 0; k < 3; ++k) acc += mi[3 * r + k] * M[3 * k + q].d[j];
        out.P[j][3 * r + q] = acc;
      }
}

void lens_out(const GradAcc* acc, const LensChain& ch, float* out, int accumulate, cudaStream_t st) {
  k_lens_out<<<1, 32, 0, st>>>(acc, ch, out, accumulate);
  profiler().launches += 1;
  PSDR_CUDA(cudaGetLastError());
}

// Pixels that hold whole groups of 32 paths: the adjoint kernels reduce the camera vertices of 32
// consecutive paths of a tile over the warp, in fp32.
static int group_pixels(int spp) {
  int g = 32;
  while (spp % g) g >>= 1;
  return 32 / g;
}

// Tiles of whole pixels, and of whole groups of 32 paths of the job where a tile holds one: those
// groups, and with them the gradients, are then the same for any such tile size.
std::vector<Tile> plan_tiles(const std::vector<DevView>& views, int cap) {
  std::vector<Tile> tiles;
  long long total = 0;
  for (const DevView& v : views) total += (long long)v.H * v.W * v.spp;
  if (total > cap) {  // (the views of a job share their spp)
    const int spp = views[0].spp, unit = group_pixels(spp);
    const int pixels = cap / spp;
    if (pixels > unit) cap = spp * (pixels / unit * unit);
  }
  Tile cur{0, 0, 0, 0};
  for (const DevView& v : views) {
    long long rem = (long long)v.H * v.W;
    while (rem > 0) {
      const long long room = (cap - cur.n) / v.spp;
      if (room <= 0) {
        tiles.push_back(cur);
        cur = Tile{cur.begin + cur.n, 0, cur.pix_begin + cur.npix, 0};
        continue;
      }
      const long long take = std::min(room, rem);
      cur.n += (int)(take * v.spp);
      cur.npix += (int)take;
      rem -= take;
    }
  }
  if (cur.n > 0) tiles.push_back(cur);
  return tiles;
}

void assign_offsets(std::vector<DevView>& views) {
  long long so = 0, po = 0;
  for (DevView& v : views) {
    v.sample_off = so;
    v.pix_off = po;
    so += (long long)v.H * v.W * v.spp;
    po += (long long)v.H * v.W;
  }
}

Profiler& profiler() {
  static Profiler p;
  return p;
}
void Profiler::begin_trace(cudaStream_t st) {
  if (!on) return;
  if (capture_ev) {
    cudaEvent_t a, b;
    PSDR_CUDA(cudaEventCreate(&a));
    PSDR_CUDA(cudaEventCreate(&b));
    capture_ev->emplace_back(a, b);
    // External: becomes an event-record node of the graph (re-recorded every replay)
    PSDR_CUDA(cudaEventRecordWithFlags(a, st, cudaEventRecordExternal));
    return;
  }
  if (used == ev.size()) {
    cudaEvent_t a, b;
    PSDR_CUDA(cudaEventCreate(&a));
    PSDR_CUDA(cudaEventCreate(&b));
    ev.emplace_back(a, b);
  }
  PSDR_CUDA(cudaEventRecord(ev[used].first, st));
}
void Profiler::end_trace(cudaStream_t st) {
  if (!on) return;
  if (capture_ev) {
    PSDR_CUDA(cudaEventRecordWithFlags(capture_ev->back().second, st, cudaEventRecordExternal));
    return;
  }
  PSDR_CUDA(cudaEventRecord(ev[used].second, st));
  ++used;
  ++trace_launches;
}
void Profiler::replayed(std::vector<EvPair>* graph_ev, long long n_trace) {
  if (!on || graph_ev->empty()) return;
  trace_launches += n_trace;
  for (auto& r : replays)
    if (r.first == graph_ev) { ++r.second; return; }
  replays.emplace_back(graph_ev, 1);
}
#define PSDR_LAUNCHED(n) (profiler().launches += (n))
void count_launches(int n) { profiler().launches += n; }

// The scene of every view of a job, or -1 when its views have several.
static int job_scene(const std::vector<DevView>& views) {
  for (const DevView& v : views)
    if (v.scene != views[0].scene) return -1;
  return views.empty() ? -1 : views[0].scene;
}

static int any_ortho(const std::vector<DevView>& views) {
  for (const DevView& v : views)
    if (v.ortho) return 1;
  return 0;
}

// Shadow-boundary samples [0, n) in chunks of four tile capacities: the pick stage queues the
// samples that pass the silhouette test, then the k_direct instance for the job's
// materials (w.bsdf) traces them. PRE: n = cells x rounds, from round0 on.
template <bool PRE, bool UNB>
static void launch_direct(const WF& w, cudaStream_t st, const DevScene* scenes, const DevView* vd, int v,
                          long long n, const HCube& hc, int round0, float* mass, int spp) {
  const long long chunk = std::min<long long>((long long)kDirectPerPath * w.cap, 1 << 30);
  for (long long b = 0; b < n; b += chunk) {
    const int nb = (int)std::min<long long>(chunk, n - b);
    PSDR_CUDA(cudaMemsetAsync(w.cnt, 0, sizeof(int), st));
    k_direct_pick<PRE, UNB><<<grid_for(nb, 256, 8), 256, 0, st>>>(w, scenes, vd, v, b, nb, hc, round0);
    const int g = grid_for(nb, 128, 64);
    if (w.bsdf) k_direct<PRE, UNB, true><<<g, 128, 0, st>>>(w, scenes, vd, v, b, hc, round0, mass, spp);
    else k_direct<PRE, UNB, false><<<g, 128, 0, st>>>(w, scenes, vd, v, b, hc, round0, mass, spp);
    PSDR_LAUNCHED(2);
  }
  PSDR_CUDA(cudaGetLastError());
}

// Zeroes the queue counters of a wavefront before a new set of paths enters its depth
// loop (k_shade resets the ray fetch counter of k_trace itself).
static void clear_counts(const WF& w, cudaStream_t st) {
  PSDR_CUDA(cudaMemsetAsync(w.cnt, 0, sizeof(int) * 2 * (w.D + 2), st));
}

template <int MODE, bool LIST>
static void depth_loop_t(WF& w, const DevScene* scenes, const DevView* views, cudaStream_t st) {
  const int cap = w.cap;
  Profiler& pf = profiler();
  for (int d = 0; d < w.D; ++d) {
    const int gs = grid_for(cap, 256, 8);
    if (w.bsdf) k_shade<MODE, true, LIST><<<gs, 256, 0, st>>>(w, scenes, views, d);
    else k_shade<MODE, false, LIST><<<gs, 256, 0, st>>>(w, scenes, views, d);
    pf.begin_trace(st);
    k_trace<LIST><<<num_sms() * w.trace_bps, 128, 0, st>>>(w, scenes, views, d, pf.on ? pf.d_rays : nullptr);
    pf.end_trace(st);
    PSDR_LAUNCHED(3);
    if (w.bsdf) k_accum<MODE, true><<<gs, 256, 0, st>>>(w, scenes, views, d);
    else k_accum<MODE, false><<<gs, 256, 0, st>>>(w, scenes, views, d);
  }
  PSDR_CUDA(cudaGetLastError());
}

// n paths at most enter the loop.
static void depth_loop(WF& w, const DevScene* scenes, const DevView* views, int mode, int n, cudaStream_t st) {
  const bool list = n >= kListMin && w.nB > 0;
  auto run = [&](auto m) {
    if (list) depth_loop_t<m.value, true>(w, scenes, views, st);
    else depth_loop_t<m.value, false>(w, scenes, views, st);
  };
  if (mode == MODE_REPLAY) run(std::integral_constant<int, MODE_REPLAY>{});
  else if (mode == MODE_KEEP) run(std::integral_constant<int, MODE_KEEP>{});
  else run(std::integral_constant<int, MODE_FWD>{});
}

template <int MODE>
static void launch_camera(const WF& w, const DevScene* scenes, const DevView* views, const Tile& tile, int g,
                          cudaStream_t st) {
  if (w.ortho) k_camera<MODE, true><<<g, 128, 0, st>>>(w, scenes, views, tile);
  else k_camera<MODE, false><<<g, 128, 0, st>>>(w, scenes, views, tile);
}

static void run_tile(WF& w, const DevScene* scenes, const DevView* views, const Tile& tile, int mode,
                     cudaStream_t st) {
  clear_counts(w, st);
  const int g = grid_for(tile.n, 128, kEachBlock);
  if (mode == MODE_REPLAY) launch_camera<MODE_REPLAY>(w, scenes, views, tile, g, st);
  else if (mode == MODE_KEEP) launch_camera<MODE_KEEP>(w, scenes, views, tile, g, st);
  else launch_camera<MODE_FWD>(w, scenes, views, tile, g, st);
  PSDR_LAUNCHED(1);
  depth_loop(w, scenes, views, mode, tile.n, st);
}

// Device bytes of a workspace per path of tile capacity (psdr_workspace::ensure).
static size_t path_bytes(const psdr_config& cfg, bool records) {
  const size_t R = (size_t)cfg.mis_light_samples + std::max(cfg.mis_bsdf_samples, 1) + 1, D = cfg.max_bounce;
  return 2 * 8 + 2 * 4 + 4 * 16 + 3 * 4 + 4 * 16 * R + (records ? 16 * (1 + D * R + 2 * D) : 0);
}

// Paths of a wavefront tile when the caller leaves it to the library: 2^22, halved until the
// workspace is at most kTileBytes and an eighth of the free device memory (down to 2^20, the
// smallest). Every launch over a tile ends with its warps draining their last rays (50 to
// 120 node visits for the longest against 14 on average), about 60 us in which the lanes
// empty out; larger tiles pay for it less often. 1.31 M triangles, 1024^2 x 16 spp, depth 5:
// traversal 18.2 ms with 2^20-path tiles, 14.7 with 2^21, 13.0 with 2^22. A workspace's first job
// maps its memory, 0.3 KB per path of the tile: at 2^22 about 5 ms more than at 2^20, once (first
// pass of a new integrator against its later ones: 256^2 x 64 spp step 11.1 and 3.3 ms,
// 1024^2 x 16 spp render 20.5 and 17.7 ms).
// A workspace that already holds such a tile keeps it without asking for the free memory. The
// choice changes no image and no gradient (plan_tiles): samples per pixel for which the smallest
// tile could cut a group of 32 paths get that tile always.
constexpr long long kTileMax = 1 << 22, kTileBatch = 1 << 21, kTileMin = 1 << 20;
constexpr size_t kTileBytes = size_t(4) << 30;
static long long auto_tile(const psdr_config& cfg, long long need, bool records, const psdr_workspace* ws) {
  if (need <= kTileMin || (long long)group_pixels(cfg.spp_interior) * cfg.spp_interior > kTileMin) return kTileMin;
  const size_t pb = path_bytes(cfg, records);
  long long t = kTileMax;
  while (t > kTileMin && (size_t)t * pb > kTileBytes) t >>= 1;
  if (t == kTileMin) return t;
  const size_t held = (size_t)std::min(t, need);
  if (ws && (size_t)ws->cap >= held && ws->R >= cfg.mis_light_samples + std::max(cfg.mis_bsdf_samples, records ? 1 : 0) + 1 &&
      ws->D >= cfg.max_bounce && (!records || ws->rec.bytes >= held * (pb - path_bytes(cfg, false))))
    return t;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
    cudaGetLastError();
    return kTileMin;
  }
  while (t > kTileMin && (size_t)t * pb > free_b / 8) t >>= 1;
  return t;
}

// lanes: concurrent tiles of a batch; its automatic tile is small enough for each lane to
// get one, and at most 2^21 (the lanes' tiles fill one another's tails: 2^22 is no faster), but no
// smaller than 2^20. 512^2 x 32 spp step in four lanes: 15.6 ms at 2^20, 14.9 at 2^21, for 1.4 GB
// more memory and 34 ms to create the batch against 29; 1024^2 x 32 spp: 91.5 and 87.3 ms.
int choose_cap(const psdr_config& cfg, const std::vector<DevView>& views, bool backward, int lanes,
               const psdr_workspace* ws, bool records) {
  int maxspp = 1;
  long long total = 0, need = 0;
  for (auto& v : views) {
    maxspp = std::max(maxspp, v.spp);
    total += (long long)v.H * v.W * v.spp;
    if (!backward) continue;
    // the largest boundary term of the view (backward_unit)
    const long long px = (long long)v.H * v.W;
    need = std::max({need, px * cfg.spp_primary_edge, px * cfg.spp_secondary_edge});
    if (cfg.estimator == PSDR_EST_UNBIASED)
      need = std::max({need, border_segments(v) * cfg.spp_pixel_boundary,
                       2ll * kCreaseSamplesPerSpp * cfg.spp_primary_edge, px * v.spp});
  }
  need = std::max(need, total);
  long long cap = cfg.tile_paths > 0 ? cfg.tile_paths : auto_tile(cfg, need, backward && records, ws);
  if (backward) {
    if (cfg.tile_paths == 0) {
      // (as few tiles as one per lane, of whole groups of paths, but no smaller than 2^20)
      const long long group = (long long)group_pixels(cfg.spp_interior) * cfg.spp_interior;
      const long long share = ((total + lanes - 1) / lanes + group - 1) / group * group;
      if (lanes > 1) cap = std::min({cap, kTileBatch, std::max(kTileMin, share)});
      cap = std::min(cap, need);
    }
    long long cells = std::max<long long>(cfg.primary_edge_hypercube_resolution,
                                          (long long)cfg.secondary_edge_hypercube_resolution[0] *
                                              cfg.secondary_edge_hypercube_resolution[1] *
                                              cfg.secondary_edge_hypercube_resolution[2]);
    cap = std::max(cap, cells);
  } else {
    cap = std::min<long long>(cap, std::max<long long>(total, maxspp));
  }
  cap = std::max<long long>(cap, maxspp);
  cap = (cap + 31) / 32 * 32;
  return (int)cap;
}

}  // namespace psdr

// Mass / prefix-sum buffers of the hypercube cells and pixel-border segments.
void psdr_workspace::ensure_mass(long long n, cudaStream_t st) {
  if (n <= mass_cap) return;
  mass_cap = 0;  // (until all of them are there: an allocation may fail)
  mass.alloc(4 * (size_t)n, st);
  mass_d.alloc(8 * (size_t)n, st);
  mass_pre.alloc(8 * (size_t)n, st);
  scan_tmp.alloc(8 * (psdr::scan_tmp_doubles((int)n) + 64), st);
  mass_cap = n;
}

void psdr_workspace::ensure(int c, int r, int d, int nv, int rec_needed, cudaStream_t st) {
  using namespace psdr;
  stream = st;
  if (c > cap || r > R || d > D) {
    const int cap1 = std::max(c, cap), R1 = std::max(r, R), D1 = std::max(d, D);
    cap = 0;  // until all of the buffers are there: an allocation may fail
    const size_t n = (size_t)cap1;
    rs.alloc(8 * n, st); ri.alloc(8 * n, st); view.alloc(4 * n, st); pix.alloc(4 * n, st);
    T.alloc(16 * n, st); L.alloc(16 * n, st); cur.alloc(16 * n, st); org.alloc(16 * n, st);
    q0.alloc(4 * n, st); q1.alloc(4 * n, st); qs.alloc(4 * n, st);
    cnt.alloc(sizeof(int) * 2 * (kMaxDepth + 2), st);
    ro.alloc(16 * n * R1, st); rd.alloc(16 * n * R1, st); ra.alloc(16 * n * R1, st); hit.alloc(16 * n * R1, st);
    cap = cap1;
    R = R1;
    D = D1;
  }
  // the records of the job's tile, which may be smaller than what an earlier job left
  if (rec_needed) rec.alloc(16 * (size_t)c * (1 + (size_t)d * r + 2 * (size_t)d), st);
  if (nv > nviews_cap) {
    nviews_cap = 0;
    views.alloc(sizeof(DevView) * nv, st);
    nviews_cap = nv;
  }
  wf.cap = cap;
  wf.rs = rs.as<unsigned long long>(); wf.ri = ri.as<unsigned long long>();
  wf.view = view.as<int>(); wf.pix = pix.as<int>();
  wf.T = T.as<float4>(); wf.L = L.as<float4>(); wf.cur = cur.as<float4>(); wf.org = org.as<float4>();
  wf.q0 = q0.as<int>(); wf.q1 = q1.as<int>(); wf.qs = qs.as<int>(); wf.cnt = cnt.as<int>();
  wf.ro = ro.as<float4>(); wf.rd = rd.as<float4>(); wf.ra = ra.as<float4>(); wf.hit = hit.as<float4>();
  wf.rec = rec.as<float4>();
  wf.rec_plane = c;
}

namespace psdr {

void upload_views(psdr_workspace* ws, const std::vector<DevView>& views, cudaStream_t st) {
  ws->h_views = views;
  PSDR_CUDA(cudaMemcpyAsync(ws->views.p, ws->h_views.data(), sizeof(DevView) * views.size(), cudaMemcpyHostToDevice, st));
}

void set_wf(WF& w, const psdr_config& cfg, int nviews, int nB_override, int light_vis) {
  w.D = cfg.max_bounce;
  w.nL = cfg.mis_light_samples;
  w.nB = nB_override >= 0 ? nB_override : cfg.mis_bsdf_samples;
  w.R = w.nL + w.nB + 1;
  w.light_vis = light_vis;
  w.nviews = nviews;
  w.one_scene = -1;
  // seed s offsets every sample stream by s * 2654435761 (mod 2^32, the width of the
  // stream index): jobs of different seeds draw from disjoint stream ranges
  w.seed = cfg.seed * 2654435761ull;
  w.trace_bps = cfg.trace_queue > 0 ? cfg.trace_queue : 8;
}

void forward_tile(const DevScene* scenes_dev, const std::vector<DevView>& views, const DevView* vd, const Tile& t,
                  const psdr_config& cfg, psdr_workspace* ws, cudaStream_t st, float* samples_out,
                  const KeptRecords* keep) {
  WF w = ws->wf;
  w.cap = ws->cap;
  set_wf(w, cfg, (int)views.size(), -1, cfg.enable_light_visable);
  w.bsdf = ws->bsdf;
  w.ortho = any_ortho(views);
  w.one_scene = job_scene(views);
  if (keep) {
    w.rec = keep->rec + t.begin;
    w.rec_plane = keep->plane;
    w.view = keep->view + t.begin;
    w.pix = keep->pix + t.begin;
  }
  run_tile(w, scenes_dev, vd, t, keep ? MODE_KEEP : MODE_FWD, st);
  k_film<<<grid_for(t.npix, 256, 8), 256, 0, st>>>(w, vd, t, std::max(1, cfg.n_pass), samples_out);
  PSDR_LAUNCHED(1);
  PSDR_CUDA(cudaGetLastError());
}

// Forward: the interior estimate of every view into V.image (and per-sample radiance
// of view 0 into samples_out when given).
// Device work of a forward job whose views are already in ws->views (tiles of `cap`
// paths). Makes no allocation and no host copy, so it can be recorded into a graph.
void forward_launch(const DevScene* scenes_dev, const std::vector<DevView>& views, const psdr_config& cfg, int cap,
                    psdr_workspace* ws, cudaStream_t st, float* samples_out, const KeptRecords* keep) {
  const DevView* vd = ws->views.as<DevView>();
  for (const Tile& t : plan_tiles(views, cap)) forward_tile(scenes_dev, views, vd, t, cfg, ws, st, samples_out, keep);
}

void render_forward_impl(const DevScene* scenes_dev, std::vector<DevView>& views, const psdr_config& cfg,
                         psdr_workspace* ws, cudaStream_t st, float* samples_out, const KeptRecords* keep) {
  assign_offsets(views);
  const int cap = choose_cap(cfg, views, false, 1, ws);
  const int R = cfg.mis_light_samples + cfg.mis_bsdf_samples + 1;
  ws->ensure(cap, R, cfg.max_bounce, (int)views.size(), 0, st);
  upload_views(ws, views, st);
  forward_launch(scenes_dev, views, cfg, cap, ws, st, samples_out, keep);
}

static void edge_phase(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb, long long begin,
                       int n, const HCube& hc, int round, bool pre, float* mass, int spp, cudaStream_t st) {
  clear_counts(w, st);
  if (pre) k_edge_init<true><<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, begin, n, hc, round, 0);
  else k_edge_init<false><<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, begin, n, hc, round, 0);
  PSDR_LAUNCHED(1);
  depth_loop(w, scenes, vd, MODE_FWD, n, st);
  clear_counts(w, st);
  k_edge_mid<<<grid_for(n, 256, 8), 256, 0, st>>>(w, vd, v, eb, n);
  PSDR_LAUNCHED(1);
  depth_loop(w, scenes, vd, MODE_FWD, n, st);
  if (pre) k_edge_final<true><<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, begin, n, mass, spp);
  else k_edge_final<false><<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, begin, n, mass, spp);
  PSDR_LAUNCHED(1);
  PSDR_CUDA(cudaGetLastError());
}

// Unbiased silhouette samples: one path per sample (the background side).
static void edge_phase_unb(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb,
                           long long begin, int n, const HCube& hc, int spp, cudaStream_t st) {
  clear_counts(w, st);
  k_edge_init<false><<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, begin, n, hc, 0, 1);
  PSDR_LAUNCHED(2);
  depth_loop(w, scenes, vd, MODE_FWD, n, st);
  k_edge_final_unb<<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, n, (float)hc.ncells, spp);
  PSDR_CUDA(cudaGetLastError());
}

// Pixel-border samples [begin, begin + n) of the N of view v (segment masses in w/pre).
static void border_phase(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb,
                         const double* mw, const double* mpre, long long S, long long begin, int n, long long N,
                         bool lens, cudaStream_t st) {
  clear_counts(w, st);
  k_border_init<<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, mw, mpre, S, begin, n, N);
  PSDR_LAUNCHED(2);
  depth_loop(w, scenes, vd, MODE_FWD, n, st);
  k_border_final<<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, n, N);
  if (lens) {
    k_lens_border<<<grid_for(n, 256, 8), 256, 0, st>>>(w, vd, v, eb, n, N);
    PSDR_LAUNCHED(1);
  }
  PSDR_CUDA(cudaGetLastError());
}

// Indirect shadow-boundary samples [begin, begin + n) of view v: one source path each.
static void indirect_phase(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb,
                           long long begin, int n, const HCube& hc, long long N, cudaStream_t st) {
  clear_counts(w, st);
  k_indirect<false><<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, begin, n, hc, 0, nullptr);
  PSDR_LAUNCHED(1);
  WF wy = w;
  wy.D = w.D - 1;  // the source y is the second vertex of the camera path
  wy.light_vis = 0;
  depth_loop(wy, scenes, vd, MODE_FWD, n, st);
  k_indirect_final<<<grid_for(n, 128, 16), 128, 0, st>>>(w, scenes, vd, v, eb, n, (float)hc.ncells, N);
  PSDR_LAUNCHED(1);
  PSDR_CUDA(cudaGetLastError());
}

// Interpenetration-crease samples [begin, begin + n) of the N of view v: two paths per
// sample (slots 2s, 2s + 1), so n is at most half the tile.
static void crease_phase(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb,
                         const CreaseBuf& cb, const double* mw, const double* mpre, long long begin, int n,
                         long long N, cudaStream_t st) {
  clear_counts(w, st);
  k_crease_init<<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, cb, mw, mpre, begin, n, N);
  PSDR_LAUNCHED(1);
  depth_loop(w, scenes, vd, MODE_FWD, n, st);
  k_crease_final<<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, cb, n);
  PSDR_LAUNCHED(1);
  PSDR_CUDA(cudaGetLastError());
}

static CreaseBuf crease_buf(psdr_workspace* ws) {
  unsigned char* p = ws->crease.as<unsigned char>();
  CreaseBuf cb;
  cb.a = reinterpret_cast<float4*>(p);
  cb.b = reinterpret_cast<float4*>(p + 16 * (size_t)kCreaseCap);
  cb.tris = reinterpret_cast<int2*>(p + 32 * (size_t)kCreaseCap);
  cb.ra = reinterpret_cast<float4*>(p + 40 * (size_t)kCreaseCap);
  cb.rb = reinterpret_cast<float4*>(p + 56 * (size_t)kCreaseCap);
  cb.rtris = reinterpret_cast<int2*>(p + 72 * (size_t)kCreaseCap);
  cb.count = reinterpret_cast<int*>(p + 80 * (size_t)kCreaseCap);
  cb.obox = reinterpret_cast<int*>(p + 80 * (size_t)kCreaseCap + 256);
  cb.later = cb.obox + 6 * kCreaseBoxObjs;
  return cb;
}

// BSDF-jump samples [begin, begin + n) of view v at depth k (1 <= k <= D): the arc
// paths run D - k bounces (none at k = D, where only a light seen along the arc counts).
static void jump_phase(WF w, const DevScene* scenes, const DevView* vd, int v, const EdgeBuf& eb, long long begin,
                       int n, int k, cudaStream_t st) {
  const int D = w.D;
  clear_counts(w, st);
  k_jump_init<<<grid_for(n, 128, kEachBlock), 128, 0, st>>>(w, scenes, vd, v, eb, begin, n, k, D);
  PSDR_LAUNCHED(1);
  if (k < D) {
    WF wk = w;
    wk.D = D - k;
    wk.light_vis = 0;
    depth_loop(wk, scenes, vd, MODE_FWD, n, st);
  }
  k_jump_final<<<grid_for(n, 256, 8), 256, 0, st>>>(w, scenes, vd, v, eb, n, k);
  PSDR_LAUNCHED(1);
  PSDR_CUDA(cudaGetLastError());
}

long long border_segments(const DevView& V) {
  return (long long)(V.W + 1) * V.H + (long long)V.W * (V.H + 1);
}

// Indirect shadow-boundary samples of a view.
static long long indirect_samples(const DevView& V, const psdr_config& cfg) {
  return std::max(1LL, (long long)V.H * V.W * cfg.spp_secondary_edge / kIndirectSampleDiv);
}

// Buffers of the boundary terms, sized for the job: the side buffers for the largest launch of
// its units (a tile of `cap` samples at most), the masses and prefix sums for the guides' cells
// and the border segments.
void ensure_border(psdr_workspace* ws, const psdr_config& cfg, const std::vector<DevView>& views,
                   const SceneGradInfo& gi, int cap, cudaStream_t st) {
  const bool unb = cfg.estimator == PSDR_EST_UNBIASED;
  const int* r3 = cfg.secondary_edge_hypercube_resolution;
  const long long cells1 = cfg.primary_edge_hypercube_resolution, cells2 = (long long)r3[0] * r3[1] * r3[2];
  const int rounds = std::min(kGuideRounds, cfg.secondary_edge_preprocess_rounds * (unb ? kDirectGuideRounds : 1));
  long long samples = 0, mass = std::max(cells1, cells2);
  for (const BwdUnit& u : backward_units(views, cfg, cap, gi)) samples = std::max(samples, u.samples);
  for (const DevView& v : views)
    if (unb) mass = std::max({mass, border_segments(v), (long long)kCreaseCap, (long long)v.scene_ntri});
  const size_t n = (size_t)std::max(ws->eb_cap, std::min<long long>(samples, cap));
  ws->eb_cap = 0;
  ws->eb_a.alloc(16 * n, st);
  ws->eb_n.alloc(16 * n, st);
  ws->eb_hb.alloc(16 * n, st);
  ws->eb_La.alloc(16 * n, st);
  ws->eb_cap = (long long)n;
  ws->hc_pmf.alloc(4 * (size_t)std::max(cells1, cells2), st);
  ws->hc_cmf.alloc(4 * (size_t)std::max(cells1, cells2), st);
  ws->ensure_mass(mass, st);
  ws->mass_rounds.alloc(sizeof(float) * (size_t)cells2 * rounds, st);
  if (unb) ws->crease.alloc(80 * (size_t)kCreaseCap + 256 + 2 * 24 * (size_t)kCreaseBoxObjs, st);
}

void set_scene_ntri(std::vector<DevView>& views, const psdr_scene* const* scenes) {
  for (DevView& v : views) v.scene_ntri = scenes[v.scene]->ntri;
}

static HCube build_hcube(psdr_workspace* ws, int ncells, const int* res, int N, bool floor, cudaStream_t st) {
  HCube hc;
  const int b = (ncells + 255) / 256;
  if (floor) {
    k_mass_cdf<<<b, 256, 0, st>>>(ws->mass.as<float>(), ncells, ws->mass_d.as<double>());
    PSDR_LAUNCHED(5);
    inclusive_scan_double(ws->mass_d.as<double>(), ws->mass_pre.as<double>(), ncells, ws->scan_tmp.as<double>(), st);
    k_mass_floor<<<b, 256, 0, st>>>(ws->mass.as<float>(), ws->mass_pre.as<double>(), ncells);
  }
  k_mass_cdf<<<b, 256, 0, st>>>(ws->mass.as<float>(), ncells, ws->mass_d.as<double>());
  PSDR_LAUNCHED(5);
  inclusive_scan_double(ws->mass_d.as<double>(), ws->mass_pre.as<double>(), ncells, ws->scan_tmp.as<double>(), st);
  k_mass_finalize<<<b, 256, 0, st>>>(ws->mass_d.as<double>(), ws->mass_pre.as<double>(), ncells,
                                     ws->hc_pmf.as<float>(), ws->hc_cmf.as<float>());
  PSDR_CUDA(cudaGetLastError());
  hc.pmf = ws->hc_pmf.as<float>();
  hc.cmf = ws->hc_cmf.as<float>();
  hc.w = ws->mass_d.as<double>();
  hc.pre = ws->mass_pre.as<double>();
  hc.ncells = ncells;
  for (int k = 0; k < 3; ++k) {
    hc.res[k] = k < N ? res[k] : 1;
    hc.unit[k] = 1.0f / (float)hc.res[k];
  }
  return hc;
}

// Backward: interior path replay + adjoint, then the primary- and direct-edge terms
// of every view. Views must carry dimage (and grad_pos when wanted).
void render_backward_impl(const DevScene* scenes_dev, std::vector<DevView>& views, const psdr_config& cfg,
                          psdr_workspace* ws, const SceneGradInfo& gi, cudaStream_t st, const KeptRecords* keep) {
  assign_offsets(views);
  const int cap = choose_cap(cfg, views, true, 1, ws, keep == nullptr);
  const int Rmax = cfg.mis_light_samples + std::max(cfg.mis_bsdf_samples, 1) + 1;
  ws->ensure(cap, Rmax, cfg.max_bounce, (int)views.size(), keep ? 0 : 1, st);
  ensure_border(ws, cfg, views, gi, cap, st);
  upload_views(ws, views, st);
  backward_launch(scenes_dev, views, cfg, cap, ws, gi, st, keep);
}

// The terms of a backward job: cfg.terms, or by default interior + primary + direct edges
// (reference estimator), and for the unbiased estimator also the pixel borders, creases,
// indirect shadow boundaries and, when a DiffuseBsdfMaterial mesh is in the job, its BRDF
// jumps.
static int job_terms(const psdr_config& cfg, const SceneGradInfo& gi) {
  if (cfg.terms) return cfg.terms;
  return cfg.estimator == PSDR_EST_UNBIASED ? (111 | (gi.jump ? 16 : 0)) : 7;
}

// The units of a backward job, in the serial order: every interior tile, then per view
// its boundary terms (primary edges, direct edges, pixel borders, indirect shadow
// boundaries, creases, BRDF jumps). Costs count traced rays.
std::vector<BwdUnit> backward_units(const std::vector<DevView>& views, const psdr_config& cfg, int cap,
                                    const SceneGradInfo& gi) {
  std::vector<BwdUnit> u;
  const bool unb = cfg.estimator == PSDR_EST_UNBIASED;
  const int terms = job_terms(cfg, gi);
  const double D = cfg.max_bounce;
  const double R = cfg.mis_light_samples + cfg.mis_bsdf_samples + 1;
  const double R1 = cfg.mis_light_samples + 2;  // boundary paths of the reference estimator: one BSDF sample
  if (terms & 1)
    for (const Tile& t : plan_tiles(views, cap)) u.push_back(BwdUnit{1, -1, t, 2.0 * t.n * (1 + D * R), 0});
  for (int v = 0; v < (int)views.size(); ++v) {
    const DevView& V = views[v];
    const double px = (double)V.H * V.W;
    const long long npx = (long long)V.H * V.W;
    if (terms & 2) {
      const double pre = (double)cfg.primary_edge_hypercube_resolution * cfg.primary_edge_preprocess_rounds *
                         2.0 * (1 + D * R1);
      const double n = px * cfg.spp_primary_edge * (unb ? 2 + D * R : 2.0 * (1 + D * R1));
      u.push_back(BwdUnit{2, v, Tile{}, pre + n,
                          std::max<long long>(cfg.primary_edge_hypercube_resolution, npx * cfg.spp_primary_edge)});
    }
    if (terms & 4) {
      const int* r3 = cfg.secondary_edge_hypercube_resolution;
      const double per = unb ? 3.0 + 2.0 * (D - 1) : 3.0;
      const double pre = (double)r3[0] * r3[1] * r3[2] * cfg.secondary_edge_preprocess_rounds *
                         (unb ? kDirectGuideRounds : 1) * per;
      u.push_back(BwdUnit{4, v, Tile{}, pre + px * cfg.spp_secondary_edge * per, 0});
    }
    if (unb && (terms & 8) && cfg.spp_pixel_boundary > 0 && V.dimage)
      u.push_back(BwdUnit{8, v, Tile{}, (double)border_segments(V) * cfg.spp_pixel_boundary * (1 + D * R),
                          border_segments(V) * cfg.spp_pixel_boundary});
    if (unb && (terms & 64) && V.dimage && !V.ortho && cfg.max_bounce >= 2) {
      const int* rs = cfg.secondary_edge_hypercube_resolution;
      const double cells = (double)std::max(1, rs[0] / kIndirectCellDiv) * rs[1] * rs[2];
      const double n = (double)indirect_samples(V, cfg);
      u.push_back(BwdUnit{64, v, Tile{}, (cells * cfg.secondary_edge_preprocess_rounds + n) * 3.0 +
                                             n * (D - 1) * R,
                          indirect_samples(V, cfg)});
    }
    if (unb && (terms & 32) && V.dimage && !V.ortho)
      u.push_back(BwdUnit{32, v, Tile{}, 8.0 * V.scene_ntri +
                                             (double)cfg.spp_primary_edge * kCreaseSamplesPerSpp * 2.0 * (1 + D * R),
                          (long long)cfg.spp_primary_edge * kCreaseSamplesPerSpp});
    // (without a DiffuseBsdfMaterial mesh the term is zero)
    if (unb && (terms & 16) && gi.jump && V.dimage) {
      double c = 0.0;
      for (int k = 1; k <= cfg.max_bounce; ++k) c += k + 1 + (D - k) * R;
      u.push_back(BwdUnit{16, v, Tile{}, px * V.spp * c, npx * V.spp});
    }
  }
  return u;
}

std::vector<std::vector<BwdUnit>> schedule_units(const std::vector<BwdUnit>& units, int lanes) {
  lanes = std::max(1, lanes);
  std::vector<int> order(units.size());
  for (size_t i = 0; i < units.size(); ++i) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return units[a].cost > units[b].cost; });
  std::vector<double> load(lanes, 0.0);
  std::vector<int> lane_of(units.size(), 0);
  for (int i : order) {
    const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    lane_of[i] = k;
    load[k] += units[i].cost;
  }
  std::vector<std::vector<BwdUnit>> out(lanes);
  for (size_t i = 0; i < units.size(); ++i) out[lane_of[i]].push_back(units[i]);
  return out;
}

std::vector<std::vector<Tile>> schedule_tiles(const std::vector<Tile>& tiles, int lanes) {
  std::vector<BwdUnit> u;
  for (const Tile& t : tiles) u.push_back(BwdUnit{1, -1, t, (double)t.n, 0});
  std::vector<std::vector<Tile>> out;
  for (const auto& l : schedule_units(u, lanes)) {
    out.emplace_back();
    for (const BwdUnit& x : l) out.back().push_back(x.tile);
  }
  return out;
}

// Interior adjoint of a tile: persistent blocks (their warps' work lists fill better over many
// paths), as many as are resident.
template <bool UNB, bool VERTS>
static void launch_adjoint(const WF& w, const DevScene* scenes, const DevView* vd, const Tile& t, cudaStream_t st) {
  // fewer warps where many BSDF samples make the lists long (nB > 13)
  int warps = kAdjWarps;
  constexpr int kMost = 200 << 10;  // shared memory of a block
  while (warps > 1 && (int)sizeof(float) * warps * adj_warp_words(w.nB) > kMost) warps >>= 1;
  const int bytes = (int)sizeof(float) * warps * adj_warp_words(w.nB);
  PSDR_CUDA(cudaFuncSetAttribute(k_adjoint<UNB, VERTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  k_adjoint<UNB, VERTS><<<grid_for(t.n, 32 * warps, 2), 32 * warps, bytes, st>>>(w, scenes, vd, t);
}

// Device work of one backward unit on workspace ws (views at vd); no allocation, no
// host copy.
void backward_unit(const DevScene* scenes_dev, const std::vector<DevView>& views, const DevView* vd,
                   const BwdUnit& u, const psdr_config& cfg, int cap, psdr_workspace* ws, const SceneGradInfo& gi,
                   cudaStream_t st, const KeptRecords* keep) {
  const bool unb = cfg.estimator == PSDR_EST_UNBIASED;
  bool lens = false;  // a view wants the camera-lens gradient
  for (const DevView& V : views) lens = lens || V.grad_lens != nullptr;
  // ---- interior tile
  if (u.term == 1) {
    WF w = ws->wf;
    w.cap = ws->cap;
    set_wf(w, cfg, (int)views.size(), -1, cfg.enable_light_visable);
    w.bsdf = ws->bsdf;
    w.ortho = any_ortho(views);
    w.one_scene = job_scene(views);
    const Tile& t = u.tile;
    if (keep) {
      w.rec = keep->rec + t.begin;
      w.rec_plane = keep->plane;
      w.view = keep->view + t.begin;
      w.pix = keep->pix + t.begin;
    } else {
      run_tile(w, scenes_dev, vd, t, MODE_REPLAY, st);
    }
    const int g = grid_for(t.n, 128, 16);
    if (gi.bsdf) {
      if (unb) k_adjoint_ext<true><<<g, 128, 0, st>>>(w, scenes_dev, vd, t);
      else k_adjoint_ext<false><<<g, 128, 0, st>>>(w, scenes_dev, vd, t);
    } else if (unb) {
      if (gi.verts) launch_adjoint<true, true>(w, scenes_dev, vd, t, st);
      else launch_adjoint<true, false>(w, scenes_dev, vd, t, st);
    } else {
      if (gi.verts) launch_adjoint<false, true>(w, scenes_dev, vd, t, st);
      else launch_adjoint<false, false>(w, scenes_dev, vd, t, st);
    }
    PSDR_LAUNCHED(1);
    if (lens) {
      if (gi.bsdf) k_lens_interior<true><<<grid_for(t.n, 256, 8), 256, 0, st>>>(w, scenes_dev, vd, t);
      else k_lens_interior<false><<<grid_for(t.n, 256, 8), 256, 0, st>>>(w, scenes_dev, vd, t);
      PSDR_LAUNCHED(1);
    }
    PSDR_CUDA(cudaGetLastError());
    return;
  }
  // ---- boundary terms of view v
  PSDR_CHECK(std::min<long long>(u.samples, cap) <= ws->eb_cap, "a boundary term has more samples than side buffers");
  WF w = ws->wf;
  w.cap = ws->cap;
  set_wf(w, cfg, (int)views.size(), 1, 0);
  w.bsdf = ws->bsdf;
  w.ortho = any_ortho(views);
  w.one_scene = job_scene(views);
  // paths of the unbiased boundary samples carry the interior estimator's radiance
  WF wi = ws->wf;
  wi.cap = ws->cap;
  set_wf(wi, cfg, (int)views.size(), -1, cfg.enable_light_visable);
  wi.bsdf = ws->bsdf;
  wi.ortho = any_ortho(views);
  wi.one_scene = w.one_scene;
  EdgeBuf eb{ws->eb_a.as<float4>(), ws->eb_n.as<float4>(), ws->eb_hb.as<float4>(), ws->eb_La.as<float4>(), nullptr};
  const int v = u.view;
  const DevView& V = views[v];
  switch (u.term) {
    case 2: {  // primary edges: preprocess over the hypercube cells, then the edge samples
      const int cells = cfg.primary_edge_hypercube_resolution;
      PSDR_CUDA(cudaMemsetAsync(ws->mass.p, 0, sizeof(float) * cells, st));
      HCube none{};
      none.unit[0] = 1.0f / (float)cells;
      for (int r = 0; r < cfg.primary_edge_preprocess_rounds; ++r)
        edge_phase(w, scenes_dev, vd, v, eb, 0, cells, none, r, true, ws->mass.as<float>(), 1, st);
      const int res[1] = {cells};
      const HCube hc = build_hcube(ws, cells, res, 1, unb, st);
      const long long N = (long long)V.H * V.W * cfg.spp_primary_edge;
      for (long long b = 0; b < N; b += cap) {
        const int nb = (int)std::min<long long>(cap, N - b);
        if (unb) edge_phase_unb(wi, scenes_dev, vd, v, eb, b, nb, hc, cfg.spp_primary_edge, st);
        else edge_phase(w, scenes_dev, vd, v, eb, b, nb, hc, 0, false, nullptr, cfg.spp_primary_edge, st);
      }
      break;
    }
    case 4: {  // direct edges
      const int* r3 = cfg.secondary_edge_hypercube_resolution;
      const int cells = r3[0] * r3[1] * r3[2];
      PSDR_CUDA(cudaMemsetAsync(ws->mass.p, 0, sizeof(float) * cells, st));
      HCube pre{};
      for (int k = 0; k < 3; ++k) { pre.res[k] = r3[k]; pre.unit[k] = 1.0f / (float)r3[k]; }
      const int rounds = cfg.secondary_edge_preprocess_rounds * (unb ? kDirectGuideRounds : 1);
      PSDR_LAUNCHED(1);
      // the rounds' samples draw from known places of their cells' streams: up to kGuideRounds of
      // them run in one launch, and their masses are added up in order
      float* rm = ws->mass_rounds.as<float>();
      for (int r = 0; r < rounds; r += kGuideRounds) {
        const int nr = std::min(kGuideRounds, rounds - r);
        PSDR_CUDA(cudaMemsetAsync(rm, 0, sizeof(float) * (size_t)cells * nr, st));
        if (unb) launch_direct<true, true>(w, st, scenes_dev, vd, v, (long long)cells * nr, pre, r, rm, 1);
        else launch_direct<true, false>(w, st, scenes_dev, vd, v, (long long)cells * nr, pre, r, rm, 1);
        k_mass_rounds<<<(cells + 255) / 256, 256, 0, st>>>(rm, cells, nr, ws->mass.as<float>());
        PSDR_LAUNCHED(1);
      }
      const HCube hc = build_hcube(ws, cells, r3, 3, unb, st);
      const long long N = (long long)V.H * V.W * cfg.spp_secondary_edge;
      if (unb) launch_direct<false, true>(w, st, scenes_dev, vd, v, N, hc, 0, nullptr, cfg.spp_secondary_edge);
      else launch_direct<false, false>(w, st, scenes_dev, vd, v, N, hc, 0, nullptr, cfg.spp_secondary_edge);
      PSDR_CUDA(cudaGetLastError());
      break;
    }
    case 8: {  // pixel borders (unbiased estimator): segment masses, their prefix sums, samples
      const long long S = border_segments(V);
      const long long N = S * cfg.spp_pixel_boundary;
      const int b = (int)((S + 255) / 256);
      k_border_mass<<<b, 256, 0, st>>>(vd, v, ws->mass.as<float>(), S);
      k_mass_cdf<<<b, 256, 0, st>>>(ws->mass.as<float>(), (int)S, ws->mass_d.as<double>());
      PSDR_LAUNCHED(2);
      inclusive_scan_double(ws->mass_d.as<double>(), ws->mass_pre.as<double>(), (int)S, ws->scan_tmp.as<double>(),
                            st);
      for (long long b0 = 0; b0 < N; b0 += cap)
        border_phase(wi, scenes_dev, vd, v, eb, ws->mass_d.as<double>(), ws->mass_pre.as<double>(), S, b0,
                     (int)std::min<long long>(cap, N - b0), N, V.grad_lens != nullptr, st);
      break;
    }
    case 64: {  // indirect shadow boundaries: the guiding preprocess, then the samples
      const int* rs = cfg.secondary_edge_hypercube_resolution;
      const int r3[3] = {std::max(1, rs[0] / kIndirectCellDiv), rs[1], rs[2]};
      const int cells = r3[0] * r3[1] * r3[2];
      PSDR_CUDA(cudaMemsetAsync(ws->mass.p, 0, sizeof(float) * cells, st));
      HCube pre{};
      for (int k = 0; k < 3; ++k) { pre.res[k] = r3[k]; pre.unit[k] = 1.0f / (float)r3[k]; }
      for (int r = 0; r < cfg.secondary_edge_preprocess_rounds; ++r) {
        k_indirect<true><<<grid_for(cells, 128, kEachBlock), 128, 0, st>>>(w, scenes_dev, vd, v, eb, 0, cells, pre, r,
                                                                   ws->mass.as<float>());
        PSDR_LAUNCHED(1);
      }
      const HCube hc = build_hcube(ws, cells, r3, 3, true, st);
      const long long N = indirect_samples(V, cfg);
      for (long long b0 = 0; b0 < N; b0 += cap)
        indirect_phase(wi, scenes_dev, vd, v, eb, b0, (int)std::min<long long>(cap, N - b0), hc, N, st);
      break;
    }
    case 32: {  // creases: the segments where two meshes cross, a length CDF over them, samples
      const CreaseBuf cb = crease_buf(ws);
      PSDR_CUDA(cudaMemsetAsync(cb.count, 0, sizeof(int), st));
      k_crease_box_init<<<kCreaseBoxObjs / 256, 256, 0, st>>>(scenes_dev, V.scene, cb);
      k_crease_boxes<<<grid_for(V.scene_ntri, 256, 8), 256, 0, st>>>(scenes_dev, V.scene, cb);
      k_crease_later<<<1, 32, 0, st>>>(scenes_dev, V.scene, cb);
      PSDR_LAUNCHED(3);
      k_crease_pairs<<<num_sms() * 4, 128, 0, st>>>(scenes_dev, V.scene, cb);
      k_crease_order<<<kCreaseCap / 128, 128, 0, st>>>(cb);
      k_crease_mass<<<kCreaseCap / 256, 256, 0, st>>>(cb, ws->mass_d.as<double>());
      PSDR_LAUNCHED(3);
      inclusive_scan_double(ws->mass_d.as<double>(), ws->mass_pre.as<double>(), kCreaseCap,
                            ws->scan_tmp.as<double>(), st);
      const long long N = (long long)cfg.spp_primary_edge * kCreaseSamplesPerSpp;
      const int chunk = cap / 2;
      for (long long b0 = 0; b0 < N; b0 += chunk)
        crease_phase(wi, scenes_dev, vd, v, eb, cb, ws->mass_d.as<double>(), ws->mass_pre.as<double>(), b0,
                     (int)std::min<long long>(chunk, N - b0), N, st);
      break;
    }
    case 16: {  // BSDF jumps (DiffuseBsdfMaterial scenes)
      const long long N = (long long)V.H * V.W * V.spp;
      for (int k = 1; k <= cfg.max_bounce; ++k)
        for (long long b0 = 0; b0 < N; b0 += cap)
          jump_phase(wi, scenes_dev, vd, v, eb, b0, (int)std::min<long long>(cap, N - b0), k, st);
      break;
    }
    default:
      throw Error{PSDR_ERR_INVALID_ARG, "unknown backward unit"};
  }
}

// Device work of a backward job (views already uploaded); no allocation, no host copy.
// The units run one after another on st with one workspace.
void backward_launch(const DevScene* scenes_dev, const std::vector<DevView>& views, const psdr_config& cfg,
                     int cap, psdr_workspace* ws, const SceneGradInfo& gi, cudaStream_t st, const KeptRecords* keep) {
  const DevView* vd = ws->views.as<DevView>();
  for (const BwdUnit& u : backward_units(views, cfg, cap, gi))
    backward_unit(scenes_dev, views, vd, u, cfg, cap, ws, gi, st, keep);
}

void grad_out(const GradAcc* acc, float* out, long long n, int accumulate, cudaStream_t st) {
  if (!out || n <= 0) return;
  k_grad_out<<<(int)((n + 255) / 256), 256, 0, st>>>(acc, out, n, accumulate);
  PSDR_LAUNCHED(1);
}

}  // namespace psdr

// ---------------------------------------------------------------- profiler C entry points
using psdr::profiler;
extern "C" {
PSDR_API psdr_status psdr_profile_enable(int32_t on) {
  try {
    psdr::Profiler& p = profiler();
    if (on && !p.d_rays) {
      PSDR_CUDA(cudaMalloc(&p.d_rays, sizeof(unsigned long long)));
      PSDR_CUDA(cudaMemset(p.d_rays, 0, sizeof(unsigned long long)));
    }
    p.on = on != 0;
  } catch (const psdr::Error& e) {
    psdr::set_error(e.msg);
    return e.code;
  }
  return PSDR_OK;
}
PSDR_API psdr_status psdr_profile_reset(void) {
  try {
    psdr::Profiler& p = profiler();
    p.used = 0;
    p.launches = 0;
    p.trace_launches = 0;
    p.replays.clear();
    if (p.d_rays) PSDR_CUDA(cudaMemset(p.d_rays, 0, sizeof(unsigned long long)));
  } catch (const psdr::Error& e) {
    psdr::set_error(e.msg);
    return e.code;
  }
  return PSDR_OK;
}
PSDR_API psdr_status psdr_profile_read(int64_t* out3, double* trace_ms) {
  try {
    psdr::Profiler& p = profiler();
    double ms = 0;
    for (size_t i = 0; i < p.used; ++i) {
      PSDR_CUDA(cudaEventSynchronize(p.ev[i].second));
      float t = 0;
      PSDR_CUDA(cudaEventElapsedTime(&t, p.ev[i].first, p.ev[i].second));
      ms += t;
    }
    for (auto& r : p.replays) {
      double g = 0;
      for (auto& e : *r.first) {
        PSDR_CUDA(cudaEventSynchronize(e.second));
        float t = 0;
        PSDR_CUDA(cudaEventElapsedTime(&t, e.first, e.second));
        g += t;
      }
      ms += g * (double)r.second;
    }
    unsigned long long rays = 0;
    if (p.d_rays) PSDR_CUDA(cudaMemcpy(&rays, p.d_rays, sizeof(rays), cudaMemcpyDeviceToHost));
    if (out3) { out3[0] = p.launches; out3[1] = p.trace_launches; out3[2] = (int64_t)rays; }
    if (trace_ms) *trace_ms = ms;
  } catch (const psdr::Error& e) {
    psdr::set_error(e.msg);
    return e.code;
  }
  return PSDR_OK;
}
}

// ================================================================== allocation-free forward
// psdr_render_fwd_noalloc renders one camera without allocating device memory: the
// wavefront buffers of each tile live in one file-scope __device__ array that every
// GPU loading this library holds until the process exits. It exists for callers that
// cannot call cudaMalloc at render time -- hosts that hand the library a fixed memory
// budget up front (plugin hosts, engines with their own pools), and latency-critical
// loops where cudaMalloc's implicit device synchronisation is not acceptable.
namespace psdr {
namespace {

// Writes the view record into the scratch from a kernel argument, so the call issues no
// host-to-device copy from host memory.
__global__ void k_put_view(DevView* dst, DevView v) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *dst = v;
}

constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;  // 32 MiB per device
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};

// Device address of the scratch array for the current device. The first call on a
// device looks it up with cudaGetSymbolAddress (the host-side symbol is only a
// stand-in and must never be passed to a kernel).
unsigned char* noalloc_scratch() {
  int dev = 0;
  PSDR_CUDA(cudaGetDevice(&dev));
  PSDR_CHECK(dev >= 0 && dev < kNoAllocMaxDevices, "device index out of range for the allocation-free path");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    PSDR_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
  }
  return g_noalloc_ptr[dev];
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Bytes of scratch a tile of `cap` paths needs with R rays per path and depth D.
size_t noalloc_bytes(size_t cap, int R, int D) {
  size_t b = align256(sizeof(DevView));
  b += align256(sizeof(int) * 2 * (D + 2));
  b += 2 * align256(8 * cap);              // sampler state, stream increment
  b += 2 * align256(4 * cap);              // view, pixel
  b += 4 * align256(16 * cap);             // T, L, current vertex, origin
  b += 3 * align256(4 * cap);              // queues
  b += 4 * align256(16 * cap * (size_t)R); // ray origin/direction/aux, hits
  return b;
}

}  // namespace
}  // namespace psdr

extern "C" PSDR_API psdr_status psdr_render_fwd_noalloc(psdr_scene* scene, const psdr_camera_desc* cam,
                                                        const psdr_config* cfg, float* image, void* stream) {
  using namespace psdr;
  try {
    PSDR_CHECK(scene != nullptr && cam != nullptr && cfg != nullptr && image != nullptr, "null argument");
    PSDR_CHECK(cfg->n_pass > 0 && cfg->spp_interior > 0, "n_pass and spp_interior must be > 0");
    PSDR_CHECK(cfg->max_bounce > 0 && cfg->max_bounce <= kMaxDepth, "max_bounce must be in [1, 16]");
    PSDR_CHECK(cfg->mis_light_samples >= 0 && cfg->mis_bsdf_samples >= 0, "mis sample counts must be >= 0");
    PSDR_CHECK(cam->type == PSDR_CAM_PERSPECTIVE, "only perspective cameras are supported");
    PSDR_CHECK(cam->height > 0 && cam->width > 0, "camera height and width must be > 0");
    PSDR_CHECK(scene->nlight > 0 || cfg->mis_light_samples == 0, "scene has no light to sample");
    const int R = cfg->mis_light_samples + cfg->mis_bsdf_samples + 1;
    PSDR_CHECK(R <= kMaxRays, "too many mis samples");
    const int D = cfg->max_bounce;
    // largest tile (multiple of 32 paths) that fits the fixed scratch
    size_t cap = kNoAllocScratchBytes / (100 + 64 * (size_t)R);
    cap &= ~size_t(31);
    while (cap > 32 && noalloc_bytes(cap, R, D) > kNoAllocScratchBytes) cap -= 32;
    if ((size_t)cfg->spp_interior > cap) {
      set_error("psdr_render_fwd_noalloc: spp_interior " + std::to_string(cfg->spp_interior) +
                " exceeds the allocation-free tile of " + std::to_string(cap) + " paths (32 MiB scratch)");
      return PSDR_ERR_INVALID_ARG;
    }
    int cur_dev = 0;
    PSDR_CUDA(cudaGetDevice(&cur_dev));
    if (cur_dev != scene->device) {
      set_error("psdr_render_fwd_noalloc: the scene was created on device " + std::to_string(scene->device) +
                " but device " + std::to_string(cur_dev) + " is current");
      return PSDR_ERR_INVALID_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char* base = noalloc_scratch();
    size_t off = 0;
    auto take = [&](size_t bytes) { unsigned char* p = base + off; off += align256(bytes); return p; };
    DevView* vd = reinterpret_cast<DevView*>(take(sizeof(DevView)));
    WF w{};
    w.cap = (int)cap;
    w.cnt = reinterpret_cast<int*>(take(sizeof(int) * 2 * (D + 2)));
    w.rs = reinterpret_cast<unsigned long long*>(take(8 * cap));
    w.ri = reinterpret_cast<unsigned long long*>(take(8 * cap));
    w.view = reinterpret_cast<int*>(take(4 * cap));
    w.pix = reinterpret_cast<int*>(take(4 * cap));
    w.T = reinterpret_cast<float4*>(take(16 * cap));
    w.L = reinterpret_cast<float4*>(take(16 * cap));
    w.cur = reinterpret_cast<float4*>(take(16 * cap));
    w.org = reinterpret_cast<float4*>(take(16 * cap));
    w.q0 = reinterpret_cast<int*>(take(4 * cap));
    w.q1 = reinterpret_cast<int*>(take(4 * cap));
    w.qs = reinterpret_cast<int*>(take(4 * cap));
    w.ro = reinterpret_cast<float4*>(take(16 * cap * R));
    w.rd = reinterpret_cast<float4*>(take(16 * cap * R));
    w.ra = reinterpret_cast<float4*>(take(16 * cap * R));
    w.hit = reinterpret_cast<float4*>(take(16 * cap * R));
    w.rec = nullptr;
    set_wf(w, *cfg, 1, -1, cfg->enable_light_visable);
    w.bsdf = scene->has_bsdf || scene->env_light >= 0 ? 1 : 0;
    w.ortho = cam->type == PSDR_CAM_ORTHOGRAPHIC ? 1 : 0;
    w.one_scene = 0;
    // the view record goes into the scratch too (the previous call's view is overwritten)
    DevView V;
    make_view(*cam, cfg->spp_interior, V);
    V.sample_off = 0;
    V.pix_off = 0;
    V.image = image;
    k_put_view<<<1, 32, 0, st>>>(vd, V);
    count_launches(1);
    // tiles of whole pixels, walked without building a host-side list
    const long long npix = (long long)cam->height * cam->width;
    const long long pix_per_tile = (long long)cap / cfg->spp_interior;
    for (long long p0 = 0; p0 < npix; p0 += pix_per_tile) {
      const long long np = std::min(pix_per_tile, npix - p0);
      Tile t{p0 * cfg->spp_interior, (int)(np * cfg->spp_interior), p0, (int)np};
      run_tile(w, scene->d_dev.as<DevScene>(), vd, t, MODE_FWD, st);  // clears the queue counters first
      k_film<<<grid_for(t.npix, 256, 8), 256, 0, st>>>(w, vd, t, std::max(1, cfg->n_pass), nullptr);
    }
    PSDR_CUDA(cudaGetLastError());
  } catch (const psdr::Error& e) {
    psdr::set_error(e.msg);
    return e.code;
  } catch (const std::exception& e) {
    psdr::set_error(e.what());
    return PSDR_ERR_CUDA;
  }
  return PSDR_OK;
}
