// Ray-batch kernels: closest hit and any hit over caller-supplied rays.  These
// back pfxt_trace_rays / pfxt_occluded (the parity entry on identical ray
// batches) and the traversal benchmark.
//
// Persistent warps with per-lane refill: the grid fills the GPU once (SM count
// x resident blocks), and whenever lanes of a warp finish their query they
// take the next ray indices from one atomic counter (one atomic per warp per
// refill).  A warp therefore keeps its lanes busy instead of idling behind its
// slowest ray, which is what limits a one-ray-per-thread launch on incoherent
// batches.  Inside a lane the walk alternates an inner-node phase and a leaf
// phase (the "while-while" loop), so lanes of a warp tend to run the same
// phase together.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "traverse.cuh"

namespace pfxt {

namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ void load_ray(const pfxt_ray* __restrict__ rays, uint32_t i, v3& o, v3& d, float& tmax) {
  const float4* p = reinterpret_cast<const float4*>(rays + i);
  float4 a = __ldg(p), b = __ldg(p + 1);
  o = mk3(a.x, a.y, a.z);
  tmax = a.w;
  d = mk3(b.x, b.y, b.z);
}

// The output word that marks a ray the first walk handed over to the IEEE
// walk (closest hit: the `hit` field; any hit: the flag).
constexpr uint32_t RETRY = QuadWalker<true>::RETRY;

// MODE 0: closest hit -> pfxt_hit; MODE 1: any hit -> u32 flag.  Rays that the
// four-box walk cannot take are marked RETRY for k_trace_retry.
template <int MODE, bool GUARD = false>
__global__ void __launch_bounds__(kThreads, TRACE_WARPS_PER_SM * 32 / kThreads) k_trace(SceneView s, const pfxt_ray* __restrict__ rays, uint32_t n,
                                                    void* __restrict__ out, uint32_t* __restrict__ counter, uint32_t lanes) {
  constexpr bool ANY = MODE == 1;
  constexpr unsigned FULL = 0xffffffffu;
  QuadStack st;
  QuadWalker<ANY, GUARD> w;
  w.idle();
  const int lane = threadIdx.x & 31;
  uint32_t idx = 0;
  bool have = false, retired = lane >= (int)lanes;
  for (;;) {
    bool need = !have && !retired;
    unsigned m = __ballot_sync(FULL, need);
    if (m) {
      int leader = __ffs(m) - 1;
      uint32_t first = 0;
      if (lane == leader) first = atomicAdd(counter, (uint32_t)__popc(m));
      first = __shfl_sync(FULL, first, leader);
      if (need) {
        idx = first + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (idx < n) {
          v3 o, d;
          float tmax;
          load_ray(rays, idx, o, d, tmax);
          w.start(s, o, d, tmax);
          have = true;
        } else {
          retired = true;
        }
      }
    }
    if (__all_sync(FULL, retired)) break;
    w.inner_phase(s, st, [&](v3& o, v3& d) {
      float tmax;
      load_ray(rays, idx, o, d, tmax);
    });
    if (w.leaf_ready()) w.leaf_phase(s, st);
    if (have && w.finished()) {
      if (MODE == 0)
        reinterpret_cast<uint4*>(out)[idx] =
            make_uint4(__float_as_uint(w.hit.t), w.hit.slot, w.record(s), w.hit.hit);
      else
        reinterpret_cast<uint32_t*>(out)[idx] = w.hit.hit;
      have = false;
    }
  }
}

// The rays k_trace marked RETRY, walked again from the start with IEEE
// division throughout (rare: a direction component above 2^20 or an origin
// component beyond the bounded range, in world or instance space).
template <int MODE, bool FLAT>
__global__ void __launch_bounds__(kThreads) k_trace_retry(SceneView s, const pfxt_ray* __restrict__ rays, uint32_t n,
                                                          void* __restrict__ out) {
  constexpr bool ANY = (MODE == 1);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t marker = MODE == 0 ? reinterpret_cast<const uint4*>(out)[i].w : reinterpret_cast<const uint32_t*>(out)[i];
    if (marker != RETRY) continue;
    RefStack st;
    Walker<ANY, false, BOX_IEEE> w;
    v3 o, d;
    float tmax;
    load_ray(rays, i, o, d, tmax);
    w.start(s, o, d, tmax);
    w.template run<FLAT>(s, st, [&](v3& wo, v3& wd) {
      wo = o;
      wd = d;
    });
    if (MODE == 0)
      reinterpret_cast<uint4*>(out)[i] = make_uint4(__float_as_uint(w.hit.t), w.hit.slot, w.hit.record, w.hit.hit);
    else
      reinterpret_cast<uint32_t*>(out)[i] = w.hit.hit;
  }
}

// Box and triangle tests of every ray as the reference counts them, one ray a
// thread on the two-box nodes (a measurement, not a hot path).
template <bool ANY>
__global__ void __launch_bounds__(kThreads) k_trace_counts(SceneView s, const pfxt_ray* __restrict__ rays, uint32_t n,
                                                           uint2* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    RefStack st;
    Walker<ANY, true, BOX_EITHER> w;
    v3 o, d;
    float tmax;
    load_ray(rays, i, o, d, tmax);
    w.start(s, o, d, tmax);
    w.run(s, st, [&](v3& wo, v3& wd) {
      wo = o;
      wd = d;
    });
    out[i] = make_uint2(w.counts.boxes, w.counts.tris);
  }
}

// The four-box node of every two-box node: its grandchildren, or a child
// itself where that is a leaf; for a pseudo-parent (one child, a subtree's
// root) the root's.  Nodes that only another node's expansion reaches are
// written too and never read: an index per two-box node needs no numbering
// pass, and the lines the walk does not touch cost no cache.
__global__ void __launch_bounds__(kThreads) k_collapse(const WideNode* __restrict__ wide, uint32_t n,
                                                       QuadNode* __restrict__ quad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  QuadNode q;
  for (int k = 0; k < 4; ++k) {
    for (int x = 0; x < 3; ++x) {
      q.axis[x].lo[k] = INFINITY;
      q.axis[x].hi[k] = -INFINITY;
    }
    q.child[k] = REF_NONE;
    q.pad[k] = 0u;
  }
  int count = 0;
  auto add = [&](const WideNode& w, int c) {
    const float* f = &w.b0[0] + 6 * c;
    for (int x = 0; x < 3; ++x) {
      q.axis[x].lo[count] = f[x];
      q.axis[x].hi[count] = f[3 + x];
    }
    q.child[count++] = w.child[c];
  };
  const uint32_t top = wide[i].child[1] == REF_NONE && !(wide[i].child[0] & REF_LEAF) ? wide[i].child[0] : i;
  for (int c = 0; c < 2; ++c) {
    const uint32_t child = wide[top].child[c];
    if (child == REF_NONE) continue;
    if (child & REF_LEAF) {
      add(wide[top], c);
    } else {
      add(wide[child], 0);
      if (wide[child].child[1] != REF_NONE) add(wide[child], 1);
    }
  }
  quad[i] = q;
}

// Traversal triangles from the triangle records, which are on the device for
// shading anyway; bound by HBM (164 bytes a triangle).  Made on the host they were
// 64 bytes a triangle to write and to upload: a scene of 1.19 M triangles and its
// tracer take 64 ms to build where they took 111 (99 with the 48-byte triangles,
// without boxes, of the two-box walk).  The upload of the leaves is 4 bytes.
__global__ void __launch_bounds__(kThreads) k_lay_triangles(const GpuTriangle* __restrict__ records,
                                                            const uint32_t* __restrict__ leaf_of, uint32_t n,
                                                            const WideNode* __restrict__ wide,
                                                            TravTri* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const GpuTriangle& r = records[i];
  TravTri t;
  for (int k = 0; k < 3; ++k) {
    t.a[k] = r.a[k];
    t.e1[k] = r.b[k] - r.a[k];  // tri_hit: e1 = tri.b.xyz - tri.a.xyz
    t.e2[k] = r.c[k] - r.a[k];  // e2 = tri.c.xyz - tri.a.xyz
    t.lo[k] = t.hi[k] = 0.0f;
  }
  t.pad = 0.0f;
  const uint32_t at = leaf_of[i];
  if (at != REF_NONE) {
    const float* f = &wide[at >> 1].b0[0] + 6u * (at & 1u);
    for (int k = 0; k < 3; ++k) {
      t.lo[k] = f[k];
      t.hi[k] = f[3 + k];
    }
  }
  out[i] = t;
}

// Narrow 32-bit flags to bytes (separate input and output regions).
__global__ void k_pack(const uint32_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i] ? 1 : 0;
}

constexpr int kMaxDevices = 64;

// Blocks of a persistent launch on the current device (SM count x resident
// blocks), computed once per device.  Threads that race on a device's first
// launch compute the same number, so the relaxed store is enough.
template <int MODE, bool GUARD = false>
int persistent_blocks() {
  static std::atomic<int> cached[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int>* slot = (dev >= 0 && dev < kMaxDevices) ? &cached[dev] : nullptr;
  int blocks = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (blocks == 0) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_trace<MODE, GUARD>, kThreads, 0);
    blocks = (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
    if (slot) slot->store(blocks, std::memory_order_relaxed);
  }
  return blocks;
}

template <int MODE, bool GUARD>
cudaError_t launch(const SceneView& s, const pfxt_ray* rays, uint32_t n, void* out, uint32_t* counter,
                   cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  const uint32_t most = (uint32_t)persistent_blocks<MODE, GUARD>();
  const uint32_t lanes = lanes_per_warp(n, most * (kThreads / 32));
  const uint32_t blocks = std::min(most, (n + lanes * (kThreads / 32) - 1) / (lanes * (kThreads / 32)));
  k_trace<MODE, GUARD><<<blocks, kThreads, 0, stream>>>(s, rays, n, out, counter, lanes);
  // Few rays a thread, as a thread with several holds its warp up (2^21 rays of two axes
  // in a room of 100k triangles, one batch of resident blocks and four: 767 and 740 us),
  // but not one: 16 batches cost the scan of a batch without any 3 us at 1.5 M rays.
  const uint32_t scan = std::min(4u * most, (n + kThreads - 1) / kThreads);
  if (s.insts)
    k_trace_retry<MODE, false><<<scan, kThreads, 0, stream>>>(s, rays, n, out);
  else
    k_trace_retry<MODE, true><<<scan, kThreads, 0, stream>>>(s, rays, n, out);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_closest(const SceneView& s, const pfxt_ray* rays, uint32_t n, pfxt_hit* hits, uint32_t* counter,
                           cudaStream_t stream) {
  return s.small == 2u ? launch<0, true>(s, rays, n, hits, counter, stream)
                       : launch<0, false>(s, rays, n, hits, counter, stream);
}

cudaError_t launch_any(const SceneView& s, const pfxt_ray* rays, uint32_t n, uint32_t* blocked, uint32_t* counter,
                       cudaStream_t stream) {
  return s.small == 2u ? launch<1, true>(s, rays, n, blocked, counter, stream)
                       : launch<1, false>(s, rays, n, blocked, counter, stream);
}

cudaError_t launch_counts(const SceneView& s, const pfxt_ray* rays, uint32_t n, bool any, uint2* counts,
                          cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const uint32_t blocks = (n + kThreads - 1) / kThreads;
  if (any)
    k_trace_counts<true><<<blocks, kThreads, 0, stream>>>(s, rays, n, counts);
  else
    k_trace_counts<false><<<blocks, kThreads, 0, stream>>>(s, rays, n, counts);
  return cudaGetLastError();
}

cudaError_t launch_collapse(const WideNode* wide, uint32_t n, QuadNode* quad, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_collapse<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(wide, n, quad);
  return cudaGetLastError();
}

cudaError_t launch_lay_triangles(const GpuTriangle* records, const uint32_t* leaf_of, uint32_t n,
                                 const WideNode* wide, TravTri* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_lay_triangles<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(records, leaf_of, n, wide, out);
  return cudaGetLastError();
}

cudaError_t prepare_any_queries() {
  persistent_blocks<1>();
  persistent_blocks<1, true>();
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, k_trace<1>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, k_trace<1, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, k_trace_retry<1, false>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, k_trace_retry<1, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, k_pack);
  return e;
}

cudaError_t launch_pack_flags(const uint32_t* flags, uint8_t* bytes, uint32_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_pack<<<(n + 255u) / 256u, 256, 0, stream>>>(flags, bytes, n);
  return cudaGetLastError();
}

}  // namespace pfxt
