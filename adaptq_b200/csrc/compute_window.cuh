// Attention over the FP32 window: the first tokens of a conversation, up to hybrid_thresh of them
// (512 by default), attended to as they came.
//
// Replaces the hybrid branch of upstream AttentionHead::compute (attention/attention.cpp:491-523)
// for head dimensions of whole float4 up to 128; other dimensions take compute_general.cuh.
//
// What bounds it: latency.  At the default threshold the window of a head is at most 512 KB, and a
// call has few heads, so the time is the chain launch, row loads, softmax, combination of the parts
// (longer windows and large calls: window_applies in adaptq_b200.cu).  A cluster of up to eight
// blocks shares a (head, query), 64 tokens each at 512; a warp takes eight tokens at a time
// with their keys and values all in flight (one lane per float4), keeps its own running maximum,
// sum and accumulator, and the parts are combined through shared memory, first in the block, then
// over the cluster: no partials in global memory, no arrival counter.  In the general kernel the
// values came after the softmax, in a loop of four loads at a time, and the parts were merged
// through global memory: 8 heads x 300 tokens x 128, back to back, 18.5 us a call there and 9.6 us
// here, of which the host's part (call, launch) is most.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace aq {

constexpr int WK_THREADS = 256, WK_WARPS = WK_THREADS / 32;
constexpr int WK_MAX_DIM = 128; // one float4 per lane
constexpr int WK_BATCH = 8;     // tokens a warp has in flight
constexpr int WK_TOKENS = 64;   // tokens per block up to a full cluster
constexpr int WK_MAX_CLUSTER = 8;

__global__ void __launch_bounds__(WK_THREADS) window_kernel(CacheView c, const float *q, float *out, int head0, int nq, int n, int *status) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank();
  const int item = (int)blockIdx.x / parts; // head and query
  const int h = head0 + item / nq, dim = c.dim, d4 = dim >> 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ __align__(16) float s_acc[WK_WARPS][WK_MAX_DIM];
  __shared__ float s_m[WK_WARPS], s_l[WK_WARPS];
  __shared__ float p_acc[WK_MAX_DIM], p_ml[2]; // this block's part, read by the cluster's first block

  const bool col = lane < d4;
  float qv[4] = {0.f, 0.f, 0.f, 0.f};
  if (col) { // the caller's query need not lie on a 16-byte boundary
#pragma unroll
    for (int e = 0; e < 4; ++e) qv[e] = __ldg(q + (size_t)item * dim + 4 * lane + e);
  }
  const float attn_s = 1.f / sqrtf((float)dim);
  const int per = (n + parts - 1) / parts;
  const int t0 = min(n, part * per), t1 = min(n, t0 + per);
  const float4 *rows = reinterpret_cast<const float4 *>(c.mirror + (size_t)h * c.mirror_stride);
  griddep_wait(); // the window is read from here on

  float m = -1e30f, l = 0.f; // the running maximum starts where upstream's does (attention.cpp:498)
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int t = t0 + warp; t < t1; t += WK_BATCH * WK_WARPS) {
    float4 kr[WK_BATCH], vr[WK_BATCH];
    float s[WK_BATCH];
#pragma unroll
    for (int b = 0; b < WK_BATCH; ++b) {
      const int tok = t + b * WK_WARPS;
      const bool live = tok < t1 && col && AQ_CHECK(status, tok < c.hyb && h >= 0 && h < c.n_heads, 12);
      kr[b] = live ? __ldcg(rows + (size_t)tok * 2 * d4 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
      vr[b] = live ? __ldcg(rows + (size_t)tok * 2 * d4 + d4 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float top = m;
#pragma unroll
    for (int b = 0; b < WK_BATCH; ++b) {
      const float dot = (qv[0] * kr[b].x + qv[1] * kr[b].y) + (qv[2] * kr[b].z + qv[3] * kr[b].w);
      s[b] = warp_sum(dot) * attn_s;
      if (t + b * WK_WARPS < t1) top = fmaxf(top, s[b]);
    }
    const float scale = expf(m - top);
    m = top;
    l *= scale;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] *= scale;
#pragma unroll
    for (int b = 0; b < WK_BATCH; ++b) {
      if (t + b * WK_WARPS >= t1) break;
      const float w = expf(s[b] - m);
      l += w;
      acc[0] += w * vr[b].x;
      acc[1] += w * vr[b].y;
      acc[2] += w * vr[b].z;
      acc[3] += w * vr[b].w;
    }
  }
  if (col) *reinterpret_cast<float4 *>(&s_acc[warp][4 * lane]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
  __syncthreads();
  if (tid < dim) {
    float M = s_m[0];
#pragma unroll
    for (int w = 1; w < WK_WARPS; ++w) M = fmaxf(M, s_m[w]);
    float L = 0.f, x = 0.f;
#pragma unroll
    for (int w = 0; w < WK_WARPS; ++w) {
      const float f = expf(s_m[w] - M);
      L += s_l[w] * f;
      x += s_acc[w][tid] * f;
    }
    p_acc[tid] = x;
    if (tid == 0) { p_ml[0] = M; p_ml[1] = L; }
  }
  cluster.sync();
  if (part == 0 && tid < dim) {
    float pm[WK_MAX_CLUSTER], pl[WK_MAX_CLUSTER], px[WK_MAX_CLUSTER];
    float M = -INFINITY;
#pragma unroll
    for (int r = 0; r < WK_MAX_CLUSTER; ++r) {
      pm[r] = -INFINITY;
      pl[r] = px[r] = 0.f;
      if (r < parts) {
        const float *ml = cluster.map_shared_rank(p_ml, r);
        pm[r] = ml[0];
        pl[r] = ml[1];
        px[r] = cluster.map_shared_rank(p_acc, r)[tid];
        M = fmaxf(M, pm[r]);
      }
    }
    float L = 0.f, x = 0.f;
#pragma unroll
    for (int r = 0; r < WK_MAX_CLUSTER; ++r) {
      if (r < parts) {
        const float f = expf(pm[r] - M);
        L += pl[r] * f;
        x += px[r] * f;
      }
    }
    // a sum that is zero or not finite is replaced by n (attention.cpp:513)
    out[(size_t)item * dim + tid] = x * ((L > 0.f && L < INFINITY) ? 1.f / L : 1.f / (float)n);
  }
  cluster.sync(); // the other blocks' shared memory stays until it has been read
}

} // namespace aq
