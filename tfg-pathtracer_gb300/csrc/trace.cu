// er_trace_closest: closest-hit queries on caller rays, the parity gate for
// BVH::transverse (BVH.hpp:120-157) as throwRay uses it (kernel.cu:152-173).
#include <cstring>

#include "internal.h"
#include "traverse.cuh"

namespace er {
namespace {

template <int NODES, bool STATS>
__global__ void __launch_bounds__(kTravBlock, kTravMinBlocks)
    k_trace_rays(DevScene S, const float* __restrict__ rays, int32_t n, int normalize, int32_t* tri, float* dist,
                 float* uv, unsigned long long* stats, int32_t* counter, uint32_t* err) {
  __shared__ int2 stk[kSmemStack * kTravBlock];
  TravStats st{0, 0, 0};
  persistent_traverse<kClosest, NODES, STATS>(
      S, n, counter, stk + threadIdx.x, st, err,
      rays_per_warp(n, gridDim.x * (kTravBlock / 32), kLoneWidth),
      [&](int32_t i, auto& tr) {
        const float* q = rays + 6 * (int64_t)i;
        f3 o = mk(q[0], q[1], q[2]);
        f3 d = mk(q[3], q[4], q[5]);
        if (normalize) d = xnormalize(d);  // Ray.hpp:17
        tr.init(S, o, d, mk1(0.f), 0.f);
      },
      [&](int32_t i, auto& tr) {
        tri[i] = tr.slot >= 0 ? __float_as_int(__ldg(S.tri_v + 3 * (size_t)tr.slot).w) : -1;
        if (dist) dist[i] = tr.slot >= 0 ? tr.best : 0.0f;
        if (uv) {
          uv[2 * (int64_t)i] = tr.slot >= 0 ? tr.u : 0.0f;
          uv[2 * (int64_t)i + 1] = tr.slot >= 0 ? tr.v : 0.0f;
        }
      });
  if (STATS) {
    atomicAdd(&stats[8], (unsigned long long)st.nodes);
    atomicAdd(&stats[9], (unsigned long long)st.boxes);
    atomicAdd(&stats[10], (unsigned long long)st.tris);
  }
}

template <int NODES, bool STATS>
void launch(er_scene* s, const float* rays, int64_t n, int normalize, int32_t* tri, float* dist, float* uv) {
  const int grid = blocks_per_sm((const void*)k_trace_rays<NODES, STATS>, kTravBlock) * s->num_sms;
  int64_t need = (n + kTravBlock / 32 * kLoneWidth - 1) / (kTravBlock / 32 * kLoneWidth);
  int g = (int)(need < grid ? need : grid);
  if (g < 1) g = 1;
  int32_t* counter = (int32_t*)((char*)s->err_word + 32);
  cudaMemsetAsync(counter, 0, sizeof(int32_t), s->stream);
  k_trace_rays<NODES, STATS><<<g, kTravBlock, 0, s->stream>>>(s->dev, rays, (int32_t)n, normalize, tri, dist, uv,
                                                          s->d_stats, counter, s->err_word);
}

}  // namespace
}  // namespace er

using namespace er;

extern "C" er_status er_trace_closest(er_scene* s, const float* rays, int64_t n, int32_t* tri_id, float* dist,
                                      float* uv, uint32_t flags, er_trace_stats* stats) {
  return guarded("er_trace_closest", [&]() -> er_status {
    if (!s || n < 0 || (n > 0 && (!rays || !tri_id))) return fail(ER_ERR_INVALID_ARG, "bad argument");
    if (n > 0x7FFFFFFF) return fail(ER_ERR_INVALID_ARG, "more than 2^31-1 rays in one call");
    ER_CUDA(cudaSetDevice(s->device));
    if (n == 0) return ER_OK;
    const bool dev = flags & ER_TRACE_DEVICE_PTRS;
    const bool want_stats = (flags & ER_TRACE_STATS) && stats;
    const float* d_rays = rays;
    int32_t* d_tri = tri_id;
    float *d_dist = dist, *d_uv = uv;
    // Host arrays.  Few rays (kTracePinned) are copied into page-locked memory
    // of the scene, where it has it, which the kernel reads and writes in
    // place: no transfers and nothing to allocate.  Others go through one
    // device block, rays first; up to kTraceKept it stays with the scene for
    // its next call.  4,099 rays take 58 us a call, 88 through the block; with
    // an allocation per array, a transfer each and two waits they took 114.
    const size_t n4 = ((size_t)n * 4 + 255) & ~(size_t)255;
    const size_t in_bytes = 6 * n4, bytes = in_bytes + (1 + (dist ? 1 : 0) + (uv ? 2 : 0)) * n4;
    const bool pinned = !dev && s->pin_rays && bytes <= kTracePinned;
    char* block = (char*)s->h_pin + 128;
    void* own = nullptr;  // a block of this call alone
    if (!dev) {
      if (!pinned && bytes > s->trace_cap) {
        const bool keep = bytes <= kTraceKept;
        if (keep) {
          cudaFree(s->trace_dev);
          s->trace_dev = nullptr;
          s->trace_cap = 0;
        }
        const size_t cap = keep ? (bytes + 0xFFFFF) & ~(size_t)0xFFFFF : bytes;
        if (cudaMalloc(&own, cap) != cudaSuccess) {
          cudaGetLastError();
          return fail(ER_ERR_OOM, "trace buffers");
        }
        if (keep) {
          s->trace_dev = own;
          s->trace_cap = cap;
          own = nullptr;
        }
      }
      if (!pinned) block = (char*)(own ? own : s->trace_dev);
      d_rays = (const float*)block;
      d_tri = (int32_t*)(block + in_bytes);
      if (dist) d_dist = (float*)(block + in_bytes + n4);
      if (uv) d_uv = (float*)(block + in_bytes + (dist ? 2 : 1) * n4);
      if (pinned) std::memcpy(block, rays, (size_t)n * 6 * sizeof(float));
      else cudaMemcpyAsync(block, rays, (size_t)n * 6 * sizeof(float), cudaMemcpyHostToDevice, s->stream);
    }
    auto cleanup = [&]() { cudaFree(own); };
    unsigned long long s0[16] = {0};
    if (want_stats) cudaMemcpyAsync(s0, s->d_stats, sizeof s0, cudaMemcpyDeviceToHost, s->stream);
    cudaEventRecord(s->ev0, s->stream);
    int norm = (flags & ER_TRACE_NORMALIZED) ? 0 : 1;
    const NodeKind kind = node_kind(s->dev);
    if (kind == kQ8Nodes) {
      if (want_stats) launch<kQ8Nodes, true>(s, d_rays, n, norm, d_tri, d_dist, d_uv);
      else launch<kQ8Nodes, false>(s, d_rays, n, norm, d_tri, d_dist, d_uv);
    } else if (want_stats) {
      launch<kPlainNodes, true>(s, d_rays, n, norm, d_tri, d_dist, d_uv);
    } else if (kind == kTexNodes) {
      launch<kTexNodes, false>(s, d_rays, n, norm, d_tri, d_dist, d_uv);
    } else {
      launch<kPlainNodes, false>(s, d_rays, n, norm, d_tri, d_dist, d_uv);
    }
    cudaEventRecord(s->ev1, s->stream);
    cudaError_t ce = cudaGetLastError();
    if (ce != cudaSuccess) {
      cleanup();
      return cuda_fail(ce, "k_trace_rays launch");
    }
    if (!dev && !pinned) {
      cudaMemcpyAsync(tri_id, d_tri, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream);
      if (dist) cudaMemcpyAsync(dist, d_dist, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, s->stream);
      if (uv) cudaMemcpyAsync(uv, d_uv, (size_t)n * 2 * sizeof(float), cudaMemcpyDeviceToHost, s->stream);
    }
    // one wait for the results, the device error word and the call's end
    uint32_t* h_err = (uint32_t*)s->h_pin;
    *h_err = 0;
    cudaMemcpyAsync(h_err, s->err_word, 4, cudaMemcpyDeviceToHost, s->stream);
    ce = cudaStreamSynchronize(s->stream);
    cleanup();
    if (ce != cudaSuccess) return cuda_fail(ce, "er_trace_closest");
    if (pinned) {
      std::memcpy(tri_id, d_tri, (size_t)n * sizeof(int32_t));
      if (dist) std::memcpy(dist, d_dist, (size_t)n * sizeof(float));
      if (uv) std::memcpy(uv, d_uv, (size_t)n * 2 * sizeof(float));
    }
    er_status st = *h_err != 0 ? check_device_error(s) : ER_OK;
    if (st != ER_OK) return st;
    if (stats) {
      float ms = 0;
      cudaEventElapsedTime(&ms, s->ev0, s->ev1);
      stats->ms = ms;
      stats->node_visits = stats->box_tests = stats->tri_tests = 0;
      if (want_stats) {
        unsigned long long s1[16];
        cudaMemcpy(s1, s->d_stats, sizeof s1, cudaMemcpyDeviceToHost);
        stats->node_visits = (int64_t)(s1[8] - s0[8]);
        stats->box_tests = (int64_t)(s1[9] - s0[9]);
        stats->tri_tests = (int64_t)(s1[10] - s0[10]);
      }
    }
    return ER_OK;
  });
}
