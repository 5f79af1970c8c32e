// psdr_internal.h -- host-side objects behind the C ABI handles.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "psdr.h"
#include "psdr_common.cuh"

namespace psdr {

void set_error(const std::string& msg);
struct Error {
  psdr_status code;
  std::string msg;
};

#define PSDR_CUDA(call)                                                                       \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      throw ::psdr::Error{e_ == cudaErrorMemoryAllocation ? PSDR_ERR_OOM : PSDR_ERR_CUDA,     \
                          std::string(#call) + ": " + cudaGetErrorString(e_)};                \
  } while (0)
#define PSDR_CHECK(cond, msg) \
  do { if (!(cond)) throw ::psdr::Error{PSDR_ERR_INVALID_ARG, msg}; } while (0)

// The library's stream-ordered memory pool of one device. It keeps up to kPoolKeep bytes of freed
// memory while any of the library's allocations is alive (a program that makes a new scene per
// step would otherwise map its memory anew each time: 7.8 ms for 1.31 M triangles, 0.5 ms from
// kept memory) and gives everything back when the last one is freed.
struct DevicePool;
constexpr unsigned long long kPoolKeep = 2ull << 30;
DevicePool* pool_alloc(void** p, size_t bytes, cudaStream_t st);  // on the current device
void pool_free(DevicePool* pool, void* p, cudaStream_t st);

// Device allocation owned by the library (stream-ordered allocator).
struct DBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaStream_t st = nullptr;
  bool view = false;  // a part of another allocation (place)
  DevicePool* pool = nullptr;
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  ~DBuf() { release(); }
  void release() {
    if (p && !view) pool_free(pool, p, st);
    p = nullptr;
    bytes = 0;
    view = false;
  }
  void place(void* q, size_t n, cudaStream_t s) {
    release();
    p = q;
    bytes = n;
    st = s;
    view = true;
  }
  void alloc(size_t n, cudaStream_t s) {
    if (n <= bytes && p) return;
    release();
    st = s;
    size_t nb = n ? n : 16;
    pool = pool_alloc(&p, nb, s);
    bytes = nb;
  }
  template <class T> T* as() const { return reinterpret_cast<T*>(p); }
};

int num_sms();
void count_launches(int n);  // profiler launch counter (psdr_profile_read)

// Scan / sort primitives (sort.cu). Temporary sizes: scan_tmp_ints(n) ints, scan_tmp_doubles(n)
// doubles.
size_t scan_tmp_ints(int n);
size_t scan_tmp_doubles(int n);
void inclusive_scan_double(const double* in, double* out, int n, double* tmp_blocks, cudaStream_t st);
// Prefix sums of (double)in[i], zero from *n_dev on.
void inclusive_scan_widen(const float* in, const int* n_dev, double* out, int n, double* tmp_blocks, cudaStream_t st);
struct SortTmp {
  DBuf keys2, vals2, hist;
};
size_t sort_hist_ints(int n, int bits);  // ints of SortTmp::hist for n pairs
// Sorted pairs: in the caller's arrays or in the temporary ones, whichever the last pass wrote.
struct SortedKeys {
  uint64_t* k64 = nullptr;  // 64-bit keys, or
  uint32_t* k32 = nullptr;  // 32-bit keys
  uint32_t* vals = nullptr;
};
// Stable LSD radix sort of (key, value) pairs over the low `bits` bits of the keys.
SortedKeys radix_sort_pairs(uint64_t* keys, uint32_t* vals, int n, int bits, SortTmp& tmp, cudaStream_t st);
SortedKeys radix_sort_pairs(uint32_t* keys, uint32_t* vals, int n, int bits, SortTmp& tmp, cudaStream_t st);
// out[i] = number of runs of equal keys that start before entry i.
void exclusive_scan_runs(const SortedKeys& k, int* out, int n, int* tmp_blocks, cudaStream_t st);

// The caller's buffers of one object, for the geometry build (k_records).
struct DevSrc {
  const float* verts;
  const int* faces;
  const float* uvs;  // null: the default uvs
  const int* uvi;
  int vert_off, tri_off;
};

}  // namespace psdr

struct psdr_scene {
  cudaStream_t stream = nullptr;
  int device = 0;  // the CUDA device current at psdr_scene_create (holds every buffer below)
  std::vector<psdr_mesh_desc> meshes;
  std::vector<psdr_area_light_desc> lights;
  int ntri = 0, nvert = 0, nobj = 0, nlight = 0, nnode = 0;
  // BVH leaves of up to this many triangles. Two against one: 11 % fewer visits per ray for 40 %
  // more triangle tests (tests are paid for in warps that gather them); traversal of the 512^2
  // icosphere step 12.3 -> 11.8 ms, of 1.31 M triangles 18.6 -> 17.9 ms. Three and four: slower.
  int leaf_size = 2;
  std::vector<int> obj_vert_off, obj_tri_off, obj_nvert, obj_ntri;
  std::vector<psdr::DevObj> h_objs;
  std::vector<psdr::DevLight> h_lights;
  std::vector<psdr::DevSrc> h_srcs;
  // device storage: one allocation, the buffers below are parts of it
  psdr::DBuf slab;
  size_t grad_texels = 0;  // entries of g_tex
  psdr::DBuf verts, tri, tri_v, objs, srcs, lights_buf, light_pmf, light_cmf, ltri_pmf, ltri_cmf;
  psdr::DBuf n_edges, edge, edge_v, edge_f, edge_pmf, edge_cmf;
  psdr::DBuf nodes, leaf, err;
  // tree of the last full build, kept for psdr_scene_refit: leaf triangle order, the leaf
  // ranges of the binary nodes (range), the children of every 4-wide node (binary ids, -1 for
  // none) and the number of 4-wide nodes (bvh_counters[0])
  psdr::DBuf bvh_order, range, bvh_slots, bvh_counters;
  // build scratch
  psdr::DBuf keys, vals, aux_i, aux_i2, aux_d, aux_d2, aabb, box_levels, flags, cbox;
  psdr::SortTmp sort_tmp;
  // fixed-point gradient accumulators (GradAcc), parts of the slab
  psdr::DBuf g_verts, g_tex, g_emit;
  psdr::DBuf vmask;  // per-vertex gradient mask (set from the gradient targets of a backward)
  std::vector<size_t> tex_grad_off;  // per object offset into g_tex (doubles), SIZE_MAX if none
  // DiffuseBsdfMaterial roughness / normal-map accumulators (after every color texture)
  std::vector<size_t> rough_grad_off, nrm_grad_off;
  bool has_bsdf = false;
  // environment light (EnvLight / SH9Light): its index (the last light) or -1, the box
  // mesh the library builds for it, and each light's parameter accumulator offset in g_tex
  int env_light = -1;
  float env_host_v[24];
  psdr::DBuf env_v, env_f, env_uv, env_uvi;
  std::vector<size_t> light_grad_off;
  bool grads_ready = false;
  psdr::DevScene dev{};
  psdr::DBuf d_dev;  // device copy of `dev`
  void upload_tables();
};
