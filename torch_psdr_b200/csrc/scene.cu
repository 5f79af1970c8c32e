// scene.cu -- scene construction on the device.
//
// Replaces Scene::Scene (scene.cc:3-104), TriangleMesh (mesh.cc:5-204) and the OptiX
// GAS build (scene_optix.cc:187-238):
//  * flattened vertex array and 96-byte per-triangle shading records,
//  * the edge list via a stable sort of half-edges by (min,max) vertex id (the
//    reference hashes them on the host; grouping by sorted key gives the same
//    left/right face assignment, in (min,max) order per mesh),
//  * discrete CDFs over edges (length), lights (power) and light triangles (area),
//  * an LBVH: 30-bit Morton codes of triangle-box centres (large triangles split off
//    by a top key bit), radix sort, Karras (2012) hierarchy, boxes of its leaf ranges, then
//    a 4-wide layout (greedy collapse of the binary tree) with child boxes in the
//    parent and leaves of up to `leaf_size` triangles.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "psdr_internal.h"

namespace psdr {

namespace {

// Last entry of the table whose offset is at most i.
template <class F>
__device__ __forceinline__ int table_find(int n, int i, F off) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off(mid) <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The flattened vertices and the triangle records (mesh.cc:27-67: normal, uv tangent, Heron
// area) of every object in one launch; a copy and a launch per object took longer than the
// work of small meshes (17 objects: 34 launches, 110 us).
__global__ void k_records(int nobj, const DevSrc* __restrict__ src, int nvert, int ntri, float* __restrict__ verts,
                          float4* __restrict__ out, int4* __restrict__ out_v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nvert) {
    const DevSrc& s = src[table_find(nobj, i, [&](int o) { return src[o].vert_off; })];
    const float* v = s.verts + 3 * (size_t)(i - s.vert_off);
    verts[3 * (size_t)i] = v[0];
    verts[3 * (size_t)i + 1] = v[1];
    verts[3 * (size_t)i + 2] = v[2];
  }
  if (i >= ntri) return;
  const int obj = table_find(nobj, i, [&](int o) { return src[o].tri_off; });
  const DevSrc& s = src[obj];
  const int f = i - s.tri_off;
  const int j0 = s.faces[3 * f], j1 = s.faces[3 * f + 1], j2 = s.faces[3 * f + 2];
  const float* V = s.verts;
  const float3 p0 = f3(V[3 * j0], V[3 * j0 + 1], V[3 * j0 + 2]);
  const float3 p1 = f3(V[3 * j1], V[3 * j1 + 1], V[3 * j1 + 2]);
  const float3 p2 = f3(V[3 * j2], V[3 * j2 + 1], V[3 * j2 + 2]);
  float uv[6] = {0.f, 0.f, 0.f, 1.f, 1.f, 0.f};
  if (s.uvs) {
    for (int c = 0; c < 3; ++c) {
      const int u = s.uvi[3 * f + c];
      uv[2 * c] = s.uvs[2 * u];
      uv[2 * c + 1] = s.uvs[2 * u + 1];
    }
  }
  const float3 a = p2 - p1, b = p0 - p2, c = p1 - p0;
  const float3 cr = cross(c, b);
  const float3 n = cr / sqrtf(sqnorm(cr));
  const float du1y = uv[3] - uv[1], du2y = uv[5] - uv[1];
  const float3 tw = c * du2y + b * du1y;
  const float3 t = tw / sqrtf(sqnorm(tw));
  const float la = norm(a), lb = norm(b), lc = norm(c);
  const float hp = (la + lb + lc) / 2.0f;
  const float q = hp * (hp - la) * (hp - lb) * (hp - lc);
  const float area = q > 0.f ? sqrtf(q) : 0.f;
  float4* r = out + 6 * (size_t)i;
  r[0] = make_float4(p0.x, p0.y, p0.z, area);
  r[1] = make_float4(p1.x, p1.y, p1.z, __int_as_float(obj));
  r[2] = make_float4(p2.x, p2.y, p2.z, uv[0]);
  r[3] = make_float4(n.x, n.y, n.z, uv[1]);
  r[4] = make_float4(t.x, t.y, t.z, uv[2]);
  r[5] = make_float4(uv[3], uv[4], uv[5], 0.f);
  out_v[i] = make_int4(j0 + s.vert_off, j1 + s.vert_off, j2 + s.vert_off, obj);
}

// emitter.cc:4-14 + sampler.h:86-96: per-light area, power and triangle CDF.
__global__ void k_light_setup(DevLight* lights, int nlight, const float4* __restrict__ tri, float* ltri_pmf,
                              float* ltri_cmf, int ltri_base, float* light_pmf, float* light_cmf) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double all_power = 0;
  for (int l = 0; l < nlight; ++l) {
    DevLight& L = lights[l];
    double tot = 0;
    for (int k = 0; k < L.ntri; ++k) tot += (double)tri[6 * (size_t)(L.tri0 + k)].w;
    double acc = 0;
    for (int k = 0; k < L.ntri; ++k) {
      double a = (double)tri[6 * (size_t)(L.tri0 + k)].w;
      acc += a;
      ltri_pmf[L.tri0 - ltri_base + k] = (float)(a / tot);
      ltri_cmf[L.tri0 - ltri_base + k] = (float)(acc / tot);
    }
    L.area = (float)tot;
    L.inv_area = 1.0f / (float)tot;
    const double lum = (double)L.emit[0] * 0.2126 + (double)L.emit[1] * 0.7152 + (double)L.emit[2] * 0.0722;
    // environment lights: 4 pi (emitter.cc:130, 243)
    const double pw = L.kind == 0 ? 2.0 * 3.14159265358979323846 * lum * tot : 4.0 * 3.14159265358979323846;
    L.power = (float)pw;
    all_power += pw;
  }
  double acc = 0;
  for (int l = 0; l < nlight; ++l) {
    const double lum = (double)lights[l].emit[0] * 0.2126 + (double)lights[l].emit[1] * 0.7152 +
                       (double)lights[l].emit[2] * 0.0722;
    const double p = lights[l].kind == 0 ? 2.0 * 3.14159265358979323846 * lum * (double)lights[l].area
                                         : 4.0 * 3.14159265358979323846;
    acc += p;
    light_pmf[l] = (float)(p / all_power);
    light_cmf[l] = (float)(acc / all_power);
  }
}

// ---------------------------------------------------------------- edges
// Half-edge h = 3f + slot: slot 0 (F0,F1,third F2), 1 (F1,F2,F0), 2 (F2,F0,F1). Its key is
// (min << vbits) | max of its vertex ids (vbits bits each): 32-bit keys up to 65,536 vertices.
template <class K>
__global__ void k_halfedges(int nF, const int4* __restrict__ tri_v, int vbits, K* __restrict__ keys,
                            uint32_t* __restrict__ vals) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int n = 3 * nF;
  if (h >= n) return;
  const int f = h / 3, slot = h - 3 * f;
  const int4 v = tri_v[f];
  const int a = slot == 0 ? v.x : (slot == 1 ? v.y : v.z);
  const int b = slot == 0 ? v.y : (slot == 1 ? v.z : v.x);
  keys[h] = ((K)min(a, b) << vbits) | (K)max(a, b);
  vals[h] = (uint32_t)h;
}

PSDR_D float3 ldv(const float* v, int i) { return f3(v[3 * i], v[3 * i + 1], v[3 * i + 2]); }

// mesh.cc:97-204 build_edges: left face = first half-edge of the group, right face =
// last one (a boundary edge uses the left face twice), normals, out direction and the
// orientation fix, length.
template <class K>
__global__ void k_edge_build(const K* __restrict__ keys, int vbits, const uint32_t* __restrict__ vals, int n,
                             const int* __restrict__ eidx, const int4* __restrict__ tri_v, const float* __restrict__ verts,
                             float4* __restrict__ edge, int2* __restrict__ edge_v, int2* __restrict__ edge_f,
                             float* __restrict__ elen, int* __restrict__ n_edges) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool start = i == 0 || keys[i] != keys[i - 1];
  if (i == n - 1) *n_edges = eidx[i] + (start ? 1 : 0);
  if (!start) return;
  int j = i;
  while (j + 1 < n && keys[j + 1] == keys[i]) ++j;
  const uint32_t hl = vals[i], hr = vals[j];
  auto third = [&](uint32_t h) {
    const int f = h / 3, slot = h - 3 * f;
    const int4 v = tri_v[f];
    return slot == 0 ? v.z : (slot == 1 ? v.x : v.y);
  };
  const int fl = hl / 3, fr = hr / 3;
  const bool shared = j > i && fl != fr;
  const int kl = third(hl), kr = j > i ? third(hr) : kl;
  const int v0 = (int)(keys[i] >> vbits), v1 = (int)(keys[i] & (((K)1 << vbits) - 1));
  const float3 p0 = ldv(verts, v0), p1 = ldv(verts, v1), p2l = ldv(verts, kl), p2r = ldv(verts, kr);
  float3 nl = normalize(cross(p1 - p0, p2l - p1));
  float3 nr = normalize(cross(p2r - p1, p1 - p0));
  float3 out = shared ? normalize(nl + nr) : normalize(cross(p1 - p0, nl));
  const float3 cp = normalize((p0 + p1) - (p2l + p2r));
  if (dot(cp, out) < 0.f && shared && norm(nl - nr) > kEps) { nl = -nl; nr = -nr; out = -out; }
  const float len = norm_rn(sub_rn(p0, p1));  // exact: the edge CDF matches the float oracle
  const int e = eidx[i];
  edge[4 * e + 0] = make_float4(p0.x, p0.y, p0.z, len);
  edge[4 * e + 1] = make_float4(p1.x, p1.y, p1.z, out.x);
  edge[4 * e + 2] = make_float4(out.y, out.z, nl.x, nl.y);
  edge[4 * e + 3] = make_float4(nl.z, nr.x, nr.y, nr.z);
  edge_v[e] = make_int2(v0, v1);
  edge_f[e] = j > i + 1 ? make_int2(kEdgeNonManifold, -1) : make_int2(fl, shared ? fr : -1);
  elen[e] = len;
}

__global__ void k_cdf_finalize(const float* __restrict__ w, const double* __restrict__ pre,
                               const int* __restrict__ n_dev, int cap, float* __restrict__ pmf,
                               float* __restrict__ cmf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = *n_dev;
  if (i >= n || i >= cap) return;
  const double tot = pre[n - 1];
  pmf[i] = (float)((double)w[i] / tot);
  cmf[i] = (float)(pre[i] / tot);
}

// ---------------------------------------------------------------- LBVH
PSDR_D unsigned int f2ord(float f) {
  unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
PSDR_D float ord2f(unsigned int u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

// n_core: triangles before the environment light's box (the box, 1000 times the scene,
// would squeeze the scene into a few Morton cells); the geometry box covers all n.
__global__ void k_centroid_box(int n, int n_core, const float4* __restrict__ tri, unsigned int* __restrict__ cbox) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  float3 lo = f3(INFINITY, INFINITY, INFINITY), hi = f3(-INFINITY, -INFINITY, -INFINITY);
  float3 glo = lo, ghi = hi;
  if (i < n) {
    const float4* r = tri + 6 * (size_t)i;
    const float3 p0 = xyz(r[0]), p1 = xyz(r[1]), p2 = xyz(r[2]);
    const float3 bl = f3(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)), fminf(p0.z, fminf(p1.z, p2.z)));
    const float3 bh = f3(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)), fmaxf(p0.z, fmaxf(p1.z, p2.z)));
    const float3 c = (bl + bh) * 0.5f;
    if (i < n_core) { lo = c; hi = c; }
    glo = bl; ghi = bh;
  }
  // 12 order-preserving integers (min of six, max of six), reduced over the block: one set of
  // atomics per block (per warp they serialise on the 12 words: 330 us for 1.31 M triangles)
  unsigned v[12] = {f2ord(lo.x), f2ord(lo.y), f2ord(lo.z), f2ord(hi.x), f2ord(hi.y), f2ord(hi.z),
                    f2ord(glo.x), f2ord(glo.y), f2ord(glo.z), f2ord(ghi.x), f2ord(ghi.y), f2ord(ghi.z)};
  __shared__ unsigned red[12];
  if (threadIdx.x < 12) red[threadIdx.x] = (threadIdx.x % 6) < 3 ? 0xffffffffu : 0u;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const unsigned r = (k % 6) < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
    if ((threadIdx.x & 31) == 0) {
      if ((k % 6) < 3) atomicMin(&red[k], r);
      else atomicMax(&red[k], r);
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    if ((threadIdx.x % 6) < 3) atomicMin(cbox + threadIdx.x, red[threadIdx.x]);
    else atomicMax(cbox + threadIdx.x, red[threadIdx.x]);
  }
}

PSDR_D unsigned int expand_bits(unsigned int v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__global__ void k_morton(int n, int n_core, const float4* __restrict__ tri, const unsigned int* __restrict__ cbox,
                         uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 lo = f3(ord2f(cbox[0]), ord2f(cbox[1]), ord2f(cbox[2]));
  const float3 hi = f3(ord2f(cbox[3]), ord2f(cbox[4]), ord2f(cbox[5]));
  const float4* r = tri + 6 * (size_t)i;
  const float3 p0 = xyz(r[0]), p1 = xyz(r[1]), p2 = xyz(r[2]);
  const float3 bl = f3(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)), fminf(p0.z, fminf(p1.z, p2.z)));
  const float3 bh = f3(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)), fmaxf(p0.z, fmaxf(p1.z, p2.z)));
  const float3 c = (bl + bh) * 0.5f;
  const float3 ext = hi - lo;
  auto q = [](float x, float l, float e) {
    float t = e > 0.f ? (x - l) / e : 0.5f;
    return (unsigned int)fminf(fmaxf(t * 1024.0f, 0.0f), 1023.0f);
  };
  unsigned int m = (expand_bits(q(c.x, lo.x, ext.x)) << 2) | (expand_bits(q(c.y, lo.y, ext.y)) << 1) |
                   expand_bits(q(c.z, lo.z, ext.z));
  // Triangles whose box spans more than a quarter of the scene (ground planes, walls)
  // get the top key bit, so the root splits them off instead of letting them inflate
  // the box of whatever small-triangle cluster shares their centroid cell.
  const float3 glo = f3(ord2f(cbox[6]), ord2f(cbox[7]), ord2f(cbox[8]));
  const float3 ghi = f3(ord2f(cbox[9]), ord2f(cbox[10]), ord2f(cbox[11]));
  const float sext = fmaxf(fmaxf(ghi.x - glo.x, ghi.y - glo.y), ghi.z - glo.z);
  const float text = fmaxf(fmaxf(bh.x - bl.x, bh.y - bl.y), bh.z - bl.z);
  if (text > 0.25f * sext || i >= n_core) m |= 1u << 30;
  keys[i] = m;
  vals[i] = (uint32_t)i;
}

// Common prefix of the (morton, index) pair keys at sorted positions i and j.
PSDR_D int delta(const uint32_t* __restrict__ k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const uint32_t a = k[i], b = k[j];
  if (a == b) return 32 + __clz((unsigned)(i ^ j));
  return __clz(a ^ b);
}

// ---- node boxes. An internal node's box is the union over its range of sorted leaves. Instead
// of climbing the tree (an atomic, two fences and dependent loads per level: 47 us for 1,284
// triangles, 310 us for 1.31 M), groups of 32 entries keep running unions from their start
// (pre) and to their end (suf), level upon level (an entry of level l + 1 is a group of level
// l); any range is then the union of at most two of them per level and a few entries inside
// one group. Minima and maxima are exact, so the boxes are those of the climb.
struct Box {
  float lo[3], hi[3];
};
constexpr int kBoxLevels = 7;  // 32^7 > 2^31 leaves
struct BoxLevels {
  const float* leaf;              // leaf boxes, 6 floats each
  float* pre[kBoxLevels];         // per level, 6 floats per entry
  float* suf[kBoxLevels];
  int cnt[kBoxLevels];            // entries of the level
};
__device__ __forceinline__ Box box_load(const float* p, int i) {
  const float2* q = reinterpret_cast<const float2*>(p + 6 * (size_t)i);
  const float2 a = q[0], b = q[1], c = q[2];
  return Box{{a.x, a.y, b.x}, {b.y, c.x, c.y}};
}
__device__ __forceinline__ void box_store(float* p, int i, const Box& b) {
  float2* q = reinterpret_cast<float2*>(p + 6 * (size_t)i);
  q[0] = make_float2(b.lo[0], b.lo[1]);
  q[1] = make_float2(b.lo[2], b.hi[0]);
  q[2] = make_float2(b.hi[1], b.hi[2]);
}
__device__ __forceinline__ Box box_union(Box a, const Box& b) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.lo[k] = fminf(a.lo[k], b.lo[k]);
    a.hi[k] = fmaxf(a.hi[k], b.hi[k]);
  }
  return a;
}
__device__ __forceinline__ Box box_empty() {
  return Box{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
}
__device__ __forceinline__ float box_area(const Box& b) {
  const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
  return dx * dy + dy * dz + dz * dx;
}

// Running unions of a warp's 32 entries (lanes past the end hold empty boxes).
__device__ __forceinline__ void warp_unions(const Box& own, int i, int n, float* pre, float* suf) {
  const int lane = threadIdx.x & 31;
  Box p = own, q = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    Box a, b;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      a.lo[k] = __shfl_up_sync(0xffffffffu, p.lo[k], o);
      a.hi[k] = __shfl_up_sync(0xffffffffu, p.hi[k], o);
      b.lo[k] = __shfl_down_sync(0xffffffffu, q.lo[k], o);
      b.hi[k] = __shfl_down_sync(0xffffffffu, q.hi[k], o);
    }
    if (lane >= o) p = box_union(p, a);
    if (lane + o < 32) q = box_union(q, b);
  }
  if (i < n) {
    box_store(pre, i, p);
    box_store(suf, i, q);
  }
}

// Leaf boxes and records in tree order, the kept order, and level 0 of the running unions.
__global__ void __launch_bounds__(256) k_leaves(int n, const uint32_t* __restrict__ order, const float4* __restrict__ tri,
                                                float4* __restrict__ leaf, uint32_t* __restrict__ order_out,
                                                float* __restrict__ box, float* __restrict__ pre,
                                                float* __restrict__ suf) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  Box b = box_empty();
  if (k < n) {
    const uint32_t t = order[k];
    const float4* r = tri + 6 * (size_t)t;
    const float4 p0 = r[0], p1 = r[1], p2 = r[2];
    leaf[3 * (size_t)k + 0] = make_float4(p0.x, p0.y, p0.z, __int_as_float((int)t));
    leaf[3 * (size_t)k + 1] = make_float4(p1.x, p1.y, p1.z, 0.f);
    leaf[3 * (size_t)k + 2] = make_float4(p2.x, p2.y, p2.z, 0.f);
    if (order_out) order_out[k] = t;
    b.lo[0] = fminf(p0.x, fminf(p1.x, p2.x)); b.lo[1] = fminf(p0.y, fminf(p1.y, p2.y)); b.lo[2] = fminf(p0.z, fminf(p1.z, p2.z));
    b.hi[0] = fmaxf(p0.x, fmaxf(p1.x, p2.x)); b.hi[1] = fmaxf(p0.y, fmaxf(p1.y, p2.y)); b.hi[2] = fmaxf(p0.z, fmaxf(p1.z, p2.z));
    box_store(box, k, b);
  }
  warp_unions(b, k, n, pre, suf);
}

// Level l >= 1: entry e is group e of the level below (its union stands at the group's end).
__global__ void __launch_bounds__(256) k_box_level(int n, int n_below, const float* __restrict__ pre_below,
                                                   float* __restrict__ pre, float* __restrict__ suf) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  Box b = box_empty();
  if (e < n) b = box_load(pre_below, min(32 * e + 31, n_below - 1));
  warp_unions(b, e, n, pre, suf);
}

// Box of the sorted leaves [lo, hi].
__device__ Box range_box(const BoxLevels& L, int lo, int hi) {
  Box b = box_empty();
  for (int l = 0; l < kBoxLevels; ++l) {
    if ((lo >> 5) == (hi >> 5)) {
      if ((lo & 31) == 0) return box_union(b, box_load(L.pre[l], hi));
      if ((hi & 31) == 31 || hi == L.cnt[l] - 1) return box_union(b, box_load(L.suf[l], lo));
      for (int e = lo; e <= hi; ++e)
        b = box_union(b, l == 0 ? box_load(L.leaf, e) : box_load(L.pre[l - 1], min(32 * e + 31, L.cnt[l - 1] - 1)));
      return b;
    }
    b = box_union(b, box_union(box_load(L.suf[l], lo), box_load(L.pre[l], hi)));
    lo = (lo >> 5) + 1;
    hi = (hi >> 5) - 1;
    if (lo > hi) return b;
  }
  return b;
}

// Karras 2012: internal node i covers the sorted leaves range[i]; its children are internal
// nodes (< n-1) or leaves (n-1 + k). `box` holds the internal nodes' boxes, then the leaves'.
__global__ void k_karras(int n, const uint32_t* __restrict__ k, BoxLevels L, int2* __restrict__ child,
                         int2* __restrict__ range, float* __restrict__ box) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = delta(k, n, i, i - d);
  int lmax = 2;
  while (delta(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = delta(k, n, i, j);
  int s = 0;
  for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
    if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
  }
  const int g = i + s * d + min(d, 0);
  const int lo = min(i, j), hi = max(i, j);
  child[i] = make_int2((lo == g) ? (n - 1 + g) : g, (hi == g + 1) ? (n - 1 + g + 1) : (g + 1));
  range[i] = make_int2(lo, hi);
  box_store(box, i, range_box(L, lo, hi));
}

// The internal nodes' boxes alone, for a tree kept from an earlier build.
__global__ void k_node_boxes(int n, BoxLevels L, const int2* __restrict__ range, float* __restrict__ box) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int2 r = range[i];
  box_store(box, i, range_box(L, r.x, r.y));
}

// ---- 4-wide BVH: greedy collapse of the binary tree. Starting from the root, a 4-wide
// node takes the two children of its binary node and keeps replacing the internal child
// with the largest surface area by that child's two children until it holds four (or
// only leaves are left); every internal child left in it becomes a 4-wide node of its own.
// A binary node whose range holds at most leaf_size triangles is a leaf.
//
// Two kernels: one block walks the nodes of more than `small` triangles level by level
// (k_collapse_top) and hands every smaller subtree to a warp (k_collapse_sub), which walks it
// with a queue in the slice of the queue array that its range of leaves owns. One block for
// the whole tree took 135 us for 20,484 triangles and 5.6 ms for 1.31 M. Nodes take their
// indices from a counter, so the layout depends on scheduling; hits do not.
struct Collapse {
  int n, leaf_size, small;
  const int2* child;
  const int2* range;
  const float* box;
  const unsigned* cbox;
  float4* nodes;
  int* slots;     // per 4-wide node: its four children (binary ids), -1 for none
  int* counters;  // [0] 4-wide nodes, [1] subtrees handed to warps, [2] subtrees taken
  int2* tasks;    // subtree roots: (binary id, 4-wide index)
  int2* queue;    // (binary id, 4-wide index)
};
__device__ __forceinline__ int leaves_of(const Collapse& c, int node) {
  if (node >= c.n - 1) return 1;
  const int2 r = c.range[node];
  return r.y - r.x + 1;
}
__device__ __forceinline__ int leaf_code(const Collapse& c, int node) {
  if (node >= c.n - 1) return ~((node - (c.n - 1)) << 3);
  const int2 r = c.range[node];
  return ~((r.x << 3) | (r.y - r.x));
}

// Node boxes are padded so that no triangle the exact test would accept is culled.
__device__ __forceinline__ float box_pad(const unsigned* cbox) {
  const float3 glo = f3(ord2f(cbox[6]), ord2f(cbox[7]), ord2f(cbox[8]));
  const float3 ghi = f3(ord2f(cbox[9]), ord2f(cbox[10]), ord2f(cbox[11]));
  const float ext = fmaxf(fmaxf(ghi.x - glo.x, ghi.y - glo.y), ghi.z - glo.z);
  return ext * 2e-6f + 1e-20f;
}
__device__ __forceinline__ void write_node(float4* o, const Box* b, const int* enc, float apad) {
  float lo[3][4], hi[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const bool none = enc[k] == kNoNode;
      lo[q][k] = none ? INFINITY : b[k].lo[q] - (fabsf(b[k].lo[q]) * 2e-6f + apad);
      hi[q][k] = none ? -INFINITY : b[k].hi[q] + (fabsf(b[k].hi[q]) * 2e-6f + apad);
    }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    o[2 * q] = make_float4(lo[q][0], lo[q][1], lo[q][2], lo[q][3]);
    o[2 * q + 1] = make_float4(hi[q][0], hi[q][1], hi[q][2], hi[q][3]);
  }
  o[6] = make_float4(__int_as_float(enc[0]), __int_as_float(enc[1]), __int_as_float(enc[2]), __int_as_float(enc[3]));
}

// The children of the 4-wide node of binary node i, with their boxes and leaf counts.
__device__ __forceinline__ int gather4(const Collapse& c, int i, int* sl, Box* bx, int* cnt) {
  const int2 ch = c.child[i];
  sl[0] = ch.x;
  sl[1] = ch.y;
  int ns = 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    bx[k] = box_load(c.box, sl[k]);
    cnt[k] = leaves_of(c, sl[k]);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    int best = -1;
    float ba = -1.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k < ns && cnt[k] > c.leaf_size) {
        const float a = box_area(bx[k]);
        if (a > ba) { ba = a; best = k; }
      }
    if (best < 0) break;
    int open = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k == best) open = sl[k];
    const int2 g = c.child[open];
    const Box bx0 = box_load(c.box, g.x), bx1 = box_load(c.box, g.y);
    const int c0 = leaves_of(c, g.x), c1 = leaves_of(c, g.y);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == best) { sl[k] = g.x; bx[k] = bx0; cnt[k] = c0; }
      if (k == ns) { sl[k] = g.y; bx[k] = bx1; cnt[k] = c1; }
    }
    ++ns;
  }
  return ns;
}

// Writes the 4-wide node of index w from its gathered children; its inner children take the
// indices from `base` on (enc: their links).
__device__ __forceinline__ void finish4(const Collapse& c, int w, int base, int ns, float apad, const Box* bx, int* sl,
                                        int* cnt, int* enc) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= ns) { enc[k] = kNoNode; sl[k] = -1; cnt[k] = 0; }
    else enc[k] = cnt[k] > c.leaf_size ? base++ : leaf_code(c, sl[k]);
  }
  write_node(c.nodes + kNodeF4 * (size_t)w, bx, enc, apad);
  reinterpret_cast<int4*>(c.slots)[w] = make_int4(sl[0], sl[1], sl[2], sl[3]);
}
__device__ __forceinline__ int inner_children(const Collapse& c, int ns, const int* cnt) {
  int inner = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) inner += k < ns && cnt[k] > c.leaf_size;
  return inner;
}

// c.counters[0] starts at 1 (the root's index is 0), the others at 0.
__global__ void __launch_bounds__(256) k_collapse_top(Collapse c) {
  __shared__ int next_n;
  const float apad = box_pad(c.cbox);
  int2* cur = c.queue;
  int2* nxt = c.queue + c.n;
  if (threadIdx.x == 0) cur[0] = make_int2(0, 0);
  int m = 1;
  __syncthreads();
  while (m > 0) {
    if (threadIdx.x == 0) next_n = 0;
    __syncthreads();
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
      const int2 job = cur[q];
      int sl[4], cnt[4], enc[4];
      Box bx[4];
      const int ns = gather4(c, job.x, sl, bx, cnt);
      const int inner = inner_children(c, ns, cnt);
      finish4(c, job.y, inner ? atomicAdd(c.counters, inner) : 0, ns, apad, bx, sl, cnt, enc);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (cnt[k] <= c.leaf_size) continue;
        if (cnt[k] > c.small) nxt[atomicAdd(&next_n, 1)] = make_int2(sl[k], enc[k]);
        else c.tasks[atomicAdd(c.counters + 1, 1)] = make_int2(sl[k], enc[k]);
      }
    }
    __syncthreads();
    m = next_n;
    int2* t = cur;
    cur = nxt;
    nxt = t;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(128) k_collapse_sub(Collapse c) {
  const int lane = threadIdx.x & 31;
  const float apad = box_pad(c.cbox);
  const int ntask = c.counters[1];
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(c.counters + 2, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntask) return;
    const int2 root = c.tasks[t];
    // a subtree of r leaves has fewer than r inner nodes: its queue is the slice [lo, hi] of the array
    int2* q = c.queue + c.range[root.x].x;
    if (lane == 0) q[0] = root;
    int head = 0, tail = 1;
    __syncwarp();
    while (head < tail) {
      const int take = min(32, tail - head);
      int sl[4], cnt[4] = {0, 0, 0, 0}, enc[4], ns = 0, inner = 0;
      Box bx[4];
      int2 job = make_int2(0, 0);
      if (lane < take) {
        job = q[head + lane];
        ns = gather4(c, job.x, sl, bx, cnt);
        inner = inner_children(c, ns, cnt);
      }
      // one allocation per warp
      int x = inner;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      int base = 0;
      if (lane == 31 && x) base = atomicAdd(c.counters, x);
      base = __shfl_sync(0xffffffffu, base, 31) + x - inner;
      if (lane < take) finish4(c, job.y, base, ns, apad, bx, sl, cnt, enc);
      head += take;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = cnt[k] > c.leaf_size;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) q[tail + __popc(b & ((1u << lane) - 1u))] = make_int2(sl[k], enc[k]);
        tail += __popc(b);
      }
      __syncwarp();
    }
  }
}

// New boxes of the 4-wide nodes of a kept tree (links unchanged).
__global__ void k_refit4(const int* __restrict__ counters, const int* __restrict__ slots, const float* __restrict__ box,
                         const unsigned* __restrict__ cbox, float4* __restrict__ nodes) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= counters[0]) return;
  const int4 s4 = reinterpret_cast<const int4*>(slots)[w];
  const int sl[4] = {s4.x, s4.y, s4.z, s4.w};
  float4* o = nodes + kNodeF4 * (size_t)w;
  const float4 e = o[6];
  const int enc[4] = {__float_as_int(e.x), __float_as_int(e.y), __float_as_int(e.z), __float_as_int(e.w)};
  Box bx[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) bx[k] = sl[k] >= 0 ? box_load(box, sl[k]) : box_empty();
  write_node(o, bx, enc, box_pad(cbox));
}

__global__ void k_bvh_init(unsigned int* cbox, int* counters) {
  const int i = threadIdx.x;
  if (i < 12) cbox[i] = ((i % 6) < 3) ? 0xffffffffu : 0u;
  if (counters && i < 3) counters[i] = i == 0 ? 1 : 0;
}

inline int nblk(int64_t n, int t = 256) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }

}  // namespace

struct DevicePool {
  std::mutex m;
  cudaMemPool_t pool = nullptr;
  long long live = 0;
};

static DevicePool* device_pool() {
  constexpr int kMaxDevices = 64;
  static DevicePool pools[kMaxDevices];
  int dev = 0;
  PSDR_CUDA(cudaGetDevice(&dev));
  PSDR_CHECK(dev >= 0 && dev < kMaxDevices, "device index out of range");
  DevicePool& P = pools[dev];
  std::lock_guard<std::mutex> lock(P.m);
  if (!P.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    PSDR_CUDA(cudaMemPoolCreate(&P.pool, &props));
    unsigned long long keep = kPoolKeep;
    PSDR_CUDA(cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep));
  }
  return &P;
}

DevicePool* pool_alloc(void** p, size_t bytes, cudaStream_t st) {
  DevicePool* P = device_pool();
  {
    std::lock_guard<std::mutex> lock(P->m);
    ++P->live;
  }
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, P->pool, st);
  if (e == cudaErrorMemoryAllocation) {
    // what the pool keeps may be what is missing
    cudaGetLastError();
    cudaMemPoolTrimTo(P->pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes, P->pool, st);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    std::lock_guard<std::mutex> lock(P->m);
    --P->live;
    PSDR_CUDA(e);
  }
  return P;
}

void pool_free(DevicePool* P, void* p, cudaStream_t st) {
  cudaFreeAsync(p, st);
  bool last;
  {
    std::lock_guard<std::mutex> lock(P->m);
    last = --P->live == 0;
  }
  if (last) {
    cudaStreamSynchronize(st);
    cudaMemPoolTrimTo(P->pool, 0);
  }
}

int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// Bits of a vertex id in the half-edge keys.
static int vertex_bits(const psdr_scene* s) {
  int b = 1;
  while ((1ll << b) < (long long)s->nvert) ++b;
  return b;
}

// Builds everything that depends on vertex positions (records, edges, CDFs, BVH) on
// stream `st`. Device work only (after the first build sized the scratch), so it can
// also be recorded into a graph.
// Vertices, triangle records, light tables and the edge list (everything but the BVH).
// Returns the number of triangles outside the environment light's box.
static int build_records_and_edges(psdr_scene* s, cudaStream_t st) {
  k_records<<<nblk(std::max(s->nvert, s->ntri)), 256, 0, st>>>(s->nobj, s->srcs.as<DevSrc>(), s->nvert, s->ntri,
                                                                s->verts.as<float>(), s->tri.as<float4>(),
                                                                s->tri_v.as<int4>());
  PSDR_CUDA(cudaGetLastError());
  // lights (the table was uploaded at creation; area, power and CDFs are recomputed)
  if (s->nlight > 0) {
    k_light_setup<<<1, 1, 0, st>>>(s->lights_buf.as<DevLight>(), s->nlight, s->tri.as<float4>(), s->ltri_pmf.as<float>(),
                                   s->ltri_cmf.as<float>(), s->dev.ltri_base, s->light_pmf.as<float>(),
                                   s->light_cmf.as<float>());
  }
  // edges: sort half-edges by (min,max) vertex id; the environment light's box (the last
  // triangles) has no edges (scene.cc:59-62 takes them from the other meshes only)
  const int n_edge_tri = s->env_light >= 0 ? s->obj_tri_off[s->meshes.size() + s->env_light] : s->ntri;
  const int nh = 3 * n_edge_tri;
  const int vbits = vertex_bits(s);
  uint32_t* vals = s->vals.as<uint32_t>();
  const int gh = nblk(std::max(1, nh));
  SortedKeys he;
  if (2 * vbits <= 32) {
    k_halfedges<<<gh, 256, 0, st>>>(n_edge_tri, s->tri_v.as<int4>(), vbits, s->keys.as<uint32_t>(), vals);
    he = radix_sort_pairs(s->keys.as<uint32_t>(), vals, nh, 2 * vbits, s->sort_tmp, st);
  } else {
    k_halfedges<<<gh, 256, 0, st>>>(n_edge_tri, s->tri_v.as<int4>(), vbits, s->keys.as<uint64_t>(), vals);
    he = radix_sort_pairs(s->keys.as<uint64_t>(), vals, nh, 2 * vbits, s->sort_tmp, st);
  }
  int* eidx = s->aux_i2.as<int>();
  exclusive_scan_runs(he, eidx, nh, s->flags.as<int>(), st);
  float* elen = reinterpret_cast<float*>(s->aux_d2.as<double>() + nh);  // scratch tail
  if (he.k32)
    k_edge_build<<<gh, 256, 0, st>>>(he.k32, vbits, he.vals, nh, eidx, s->tri_v.as<int4>(), s->verts.as<float>(),
                                     s->edge.as<float4>(), s->edge_v.as<int2>(), s->edge_f.as<int2>(), elen,
                                     s->n_edges.as<int>());
  else
    k_edge_build<<<gh, 256, 0, st>>>(he.k64, vbits, he.vals, nh, eidx, s->tri_v.as<int4>(), s->verts.as<float>(),
                                     s->edge.as<float4>(), s->edge_v.as<int2>(), s->edge_f.as<int2>(), elen,
                                     s->n_edges.as<int>());
  inclusive_scan_widen(elen, s->n_edges.as<int>(), s->aux_d2.as<double>(), nh,
                       reinterpret_cast<double*>(s->flags.as<int>()), st);
  k_cdf_finalize<<<gh, 256, 0, st>>>(elen, s->aux_d2.as<double>(), s->n_edges.as<int>(), nh, s->edge_pmf.as<float>(),
                                     s->edge_cmf.as<float>());
  PSDR_CUDA(cudaGetLastError());
  // records, lights, half-edges, run scan (3), edges, length CDF (4)
  count_launches(1 + (s->nlight > 0) + 9);
  return n_edge_tri;
}

// Floats of the running-union arrays (pre and suf) over n leaves.
static size_t box_level_floats(size_t n) {
  size_t t = 0;
  for (size_t c = n; ; c = (c + 31) / 32) {
    t += 6 * ((c + 31) / 32 * 32);
    if (c <= 32) break;
  }
  return t;
}

// Leaf records and boxes of the leaves in `order`, and the levels of running unions over them.
static BoxLevels build_leaves(psdr_scene* s, const uint32_t* order, uint32_t* order_out, cudaStream_t st) {
  const int n = s->ntri;
  BoxLevels L{};
  float* leaf_box = s->aabb.as<float>() + 6 * (size_t)(n - 1);
  float* pre = s->box_levels.as<float>();
  float* suf = pre + box_level_floats(n);
  L.leaf = leaf_box;
  int cnt = n;
  for (int l = 0; l < kBoxLevels; ++l) {
    L.pre[l] = pre;
    L.suf[l] = suf;
    L.cnt[l] = cnt;
    if (l == 0)
      k_leaves<<<nblk(cnt), 256, 0, st>>>(cnt, order, s->tri.as<float4>(), s->leaf.as<float4>(), order_out, leaf_box, pre,
                                          suf);
    else
      k_box_level<<<nblk(cnt), 256, 0, st>>>(cnt, L.cnt[l - 1], L.pre[l - 1], pre, suf);
    count_launches(1);
    if (cnt <= 32) break;
    pre += 6 * (size_t)((cnt + 31) / 32 * 32);
    suf += 6 * (size_t)((cnt + 31) / 32 * 32);
    cnt = (cnt + 31) / 32;
  }
  return L;
}

void scene_build_geometry(psdr_scene* s, cudaStream_t st) {
  const int n_edge_tri = build_records_and_edges(s, st);
  // BVH
  const int n = s->ntri;
  uint32_t* vals = s->vals.as<uint32_t>();
  unsigned int* cbox = s->cbox.as<unsigned int>();
  int* counters = s->bvh_counters.as<int>();
  k_bvh_init<<<1, 32, 0, st>>>(cbox, counters);
  k_centroid_box<<<nblk(n), 256, 0, st>>>(n, n_edge_tri, s->tri.as<float4>(), cbox);
  k_morton<<<nblk(n), 256, 0, st>>>(n, n_edge_tri, s->tri.as<float4>(), cbox, s->keys.as<uint32_t>(), vals);
  const SortedKeys mo = radix_sort_pairs(s->keys.as<uint32_t>(), vals, n, 31, s->sort_tmp, st);
  const BoxLevels L = build_leaves(s, mo.vals, s->bvh_order.as<uint32_t>(), st);
  if (n > 1) {
    int2* child = s->aux_i.as<int2>();
    int2* range = s->range.as<int2>();
    float* box = s->aabb.as<float>();
    k_karras<<<nblk(n - 1), 256, 0, st>>>(n, mo.k32, L, child, range, box);
    // the root (node 0) must stay an internal node: leaves hold fewer than n triangles. Subtrees
    // of at most 1/1024 of the triangles go to warps of their own.
    Collapse c{n, std::min(s->leaf_size, n - 1), std::max(32, n / 1024), child, range, box, cbox, s->nodes.as<float4>(),
               s->bvh_slots.as<int>(), counters, s->aux_d.as<int2>(), s->aux_d2.as<int2>()};
    k_collapse_top<<<1, 256, 0, st>>>(c);
    k_collapse_sub<<<std::max(1, std::min(n / 128, 2 * num_sms())), 128, 0, st>>>(c);
    count_launches(3);
  }
  count_launches(3);
  PSDR_CUDA(cudaGetLastError());
}

// Same as scene_build_geometry for records, lights and edges, but the BVH keeps the tree
// of the last full build and only its boxes are recomputed. Any tree whose boxes bound
// their triangles gives the same closest hits.
void scene_refit_geometry(psdr_scene* s, cudaStream_t st) {
  const int n_edge_tri = build_records_and_edges(s, st);
  const int n = s->ntri;
  unsigned int* cbox = s->cbox.as<unsigned int>();
  k_bvh_init<<<1, 32, 0, st>>>(cbox, nullptr);  // the scene extent pads the node boxes
  k_centroid_box<<<nblk(n), 256, 0, st>>>(n, n_edge_tri, s->tri.as<float4>(), cbox);
  const BoxLevels L = build_leaves(s, s->bvh_order.as<uint32_t>(), nullptr, st);
  if (n > 1) {
    float* box = s->aabb.as<float>();
    k_node_boxes<<<nblk(n - 1), 256, 0, st>>>(n, L, s->range.as<int2>(), box);
    k_refit4<<<nblk(n - 1), 256, 0, st>>>(s->bvh_counters.as<int>(), s->bvh_slots.as<int>(), box, cbox,
                                          s->nodes.as<float4>());
    count_launches(2);
  }
  count_launches(2);
  PSDR_CUDA(cudaGetLastError());
}

// One allocation for all of a scene's buffers (45 stream-ordered allocations took as long as
// building a small scene's geometry).
void psdr_scene_alloc(psdr_scene* s) {
  cudaStream_t st = s->stream;
  const int n = std::max(1, s->ntri), nh = 3 * n;
  int nlt = 0;
  for (auto& l : s->h_lights) nlt += l.ntri;
  std::vector<std::pair<DBuf*, size_t>> plan;
  auto want = [&](DBuf& b, size_t bytes) { plan.emplace_back(&b, bytes); };
  // the tables uploaded at creation come first (upload_tables copies them in one piece)
  want(s->objs, sizeof(DevObj) * std::max(1, s->nobj));
  want(s->srcs, sizeof(DevSrc) * std::max(1, s->nobj));
  want(s->lights_buf, sizeof(DevLight) * std::max(1, s->nlight));
  want(s->d_dev, sizeof(DevScene));
  want(s->err, sizeof(int));
  want(s->verts, sizeof(float) * 3 * std::max(1, s->nvert));
  want(s->tri, sizeof(float4) * 6 * n);
  want(s->tri_v, sizeof(int4) * n);
  want(s->light_pmf, sizeof(float) * std::max(1, s->nlight));
  want(s->light_cmf, sizeof(float) * std::max(1, s->nlight));
  want(s->ltri_pmf, sizeof(float) * std::max(1, nlt));
  want(s->ltri_cmf, sizeof(float) * std::max(1, nlt));
  want(s->n_edges, sizeof(int));
  want(s->edge, sizeof(float4) * 4 * nh);
  want(s->edge_v, sizeof(int2) * nh);
  want(s->edge_f, sizeof(int2) * nh);
  want(s->edge_pmf, sizeof(float) * nh);
  want(s->edge_cmf, sizeof(float) * nh);
  want(s->nodes, sizeof(float4) * kNodeF4 * n);
  want(s->leaf, sizeof(float4) * 3 * n);
  want(s->bvh_order, sizeof(uint32_t) * n);
  want(s->range, sizeof(int2) * n);
  want(s->bvh_slots, sizeof(int) * 4 * (size_t)n);
  want(s->bvh_counters, sizeof(int) * 3);
  // build scratch
  const size_t key = 2 * vertex_bits(s) <= 32 ? sizeof(uint32_t) : sizeof(uint64_t);
  want(s->keys, key * nh);
  want(s->vals, sizeof(uint32_t) * nh);
  want(s->sort_tmp.keys2, key * nh);
  want(s->sort_tmp.vals2, sizeof(uint32_t) * nh);
  want(s->sort_tmp.hist, sizeof(int) * std::max(sort_hist_ints(nh, 2 * vertex_bits(s)), sort_hist_ints(n, 31)));
  want(s->aux_i, sizeof(int2) * n);
  want(s->aux_i2, sizeof(int) * nh);
  want(s->aux_d, sizeof(int2) * n);
  want(s->aux_d2, sizeof(double) * nh + sizeof(float) * nh);
  want(s->aabb, sizeof(float) * 6 * (2 * (size_t)n));
  want(s->box_levels, 2 * sizeof(float) * box_level_floats(n));
  want(s->flags, sizeof(int) * (2 * scan_tmp_ints(nh) + 64));
  want(s->cbox, sizeof(unsigned int) * 12);
  // gradient accumulators
  want(s->g_verts, sizeof(GradAcc) * 3 * std::max(1, s->nvert));
  want(s->g_tex, sizeof(GradAcc) * std::max<size_t>(1, s->grad_texels));
  want(s->g_emit, sizeof(GradAcc) * 3 * std::max(1, s->nlight));
  want(s->vmask, std::max(1, s->nvert));
  size_t total = 0;
  for (auto& w : plan) total += (w.second + 255) & ~size_t(255);
  s->slab.alloc(total, st);
  size_t off = 0;
  for (auto& w : plan) {
    w.first->place(s->slab.as<unsigned char>() + off, w.second, st);
    off += (w.second + 255) & ~size_t(255);
  }
  PSDR_CUDA(cudaMemsetAsync(s->err.p, 0, sizeof(int), st));
  DevScene& d = s->dev;
  d.ntri = s->ntri; d.nvert = s->nvert; d.nobj = s->nobj; d.nlight = s->nlight;
  const int nm = (int)s->meshes.size();
  const bool hot = s->nlight == 1 && s->obj_nvert[nm] <= kMaxLightVerts;
  d.light_v0 = hot ? s->obj_vert_off[nm] : 0;
  d.light_nv = hot ? s->obj_nvert[nm] : 0;
  d.tri = s->tri.as<float4>(); d.tri_v = s->tri_v.as<int4>(); d.verts = s->verts.as<float>();
  d.objs = s->objs.as<DevObj>(); d.lights = s->lights_buf.as<DevLight>();
  d.light_pmf = s->light_pmf.as<float>(); d.light_cmf = s->light_cmf.as<float>();
  d.ltri_pmf = s->ltri_pmf.as<float>(); d.ltri_cmf = s->ltri_cmf.as<float>();
  d.edge_cap = nh; d.n_edges = s->n_edges.as<int>(); d.edge = s->edge.as<float4>(); d.edge_v = s->edge_v.as<int2>();
  d.edge_f = s->edge_f.as<int2>();
  d.edge_pmf = s->edge_pmf.as<float>(); d.edge_cmf = s->edge_cmf.as<float>();
  d.nodes = s->nodes.as<float4>(); d.leaf = s->leaf.as<float4>();
  d.root = s->ntri > 1 ? 0 : ~0;  // a single triangle makes the root a leaf
  d.grad_verts = nullptr;
  d.vmask = nullptr;
  d.err = s->err.as<int>();
}

}  // namespace psdr

// Host -> device uploads of the object and light tables and the scene record; done
// once at creation so that the geometry rebuild (psdr_scene_update, or a rebuild
// recorded into a batch graph) is made of device work only.
void psdr_scene::upload_tables() {
  using namespace psdr;
  h_srcs.clear();
  for (int o = 0; o < nobj; ++o) {
    const bool is_mesh = o < (int)meshes.size();
    const int l = o - (int)meshes.size();
    DevSrc d{};
    d.verts = is_mesh ? meshes[o].vertices : lights[l].vertices;
    d.faces = is_mesh ? meshes[o].faces : lights[l].faces;
    if (is_mesh && meshes[o].uvs && meshes[o].uv_indices) {
      d.uvs = meshes[o].uvs;
      d.uvi = meshes[o].uv_indices;
    } else if (!is_mesh && l == env_light && lights[l].type == PSDR_LIGHT_ENV) {
      // the EnvLight box carries the cube-map uvs
      d.uvs = env_uv.as<float>();
      d.uvi = env_uvi.as<int>();
    }
    d.vert_off = obj_vert_off[o];
    d.tri_off = obj_tri_off[o];
    h_srcs.push_back(d);
  }
  unsigned char* base = slab.as<unsigned char>();
  std::vector<unsigned char> tables(d_dev.as<unsigned char>() - base + sizeof(DevScene), 0);
  auto put = [&](const DBuf& b, const void* src, size_t bytes) {
    if (bytes) memcpy(tables.data() + (b.as<unsigned char>() - base), src, bytes);
  };
  put(objs, h_objs.data(), sizeof(DevObj) * h_objs.size());
  put(srcs, h_srcs.data(), sizeof(DevSrc) * h_srcs.size());
  put(lights_buf, h_lights.data(), sizeof(DevLight) * h_lights.size());
  put(d_dev, &dev, sizeof(DevScene));
  PSDR_CUDA(cudaMemcpyAsync(base, tables.data(), tables.size(), cudaMemcpyHostToDevice, stream));
}
