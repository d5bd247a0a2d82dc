// Canary attention-error estimator: for b in {2, 4, 8},
//   delta_b = mean over (query head, query) of KL( softmax(q . K~_b^T * s) || softmax(q . K_ref^T * s) )
// where K~_b is the storage round trip of the K_ref window at b bits in the cache's exact K
// format (per channel over consecutive groups of k_group tokens) -- echokv_vllm/canary.py:59-89,
// echokv_vllm/quant.py:82-96.  One CTA per layer; the whole problem of a layer lives in shared
// memory, so the estimator is one launch (the reference issues about a dozen small kernels).  The KV heads of a layer
// are independent until the final mean: a thread-block cluster of up to 8 CTAs per layer takes one head (or every
// eighth) each, and the cluster's first CTA adds the per-CTA sums in CTA order through distributed shared memory, so
// the result does not depend on timing.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace echokv {

constexpr int CK_THREADS = 256;
constexpr int CK_WARPS = CK_THREADS / 32;
constexpr int CK_RPW = 4;                    // query rows a warp scores at once
constexpr int CK_ROWS = CK_WARPS * CK_RPW;   // query rows (queries x query heads of one KV head) per pass

struct CanaryArgs {
  const void* q; int q_dt; int64_t q_sl, q_sq, q_sh;
  const float* kref; int64_t k_sl, k_sw, k_sh;
  int ring_pos, ring_fill, window;
  int nq, Hq, H, D, KG;
  float scale;
  float* out;
  int k_vec;  // K_ref rows can be read with 16-byte loads
};

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < CK_THREADS / 32; ++i) t += red[i];
  return t;
}

// Scores of CK_RPW query rows (`a`, stride SD) against keys t and t + 32 of `k` (stride SD): lanes are keys, so a
// query value is a broadcast and the padded key rows (SD = D + 4 floats) are read without bank conflicts.
__device__ __forceinline__ void score_rows(const float* a, const float* k, int t, int w, int D, int SD, float scale,
                                           float* dst, int row0, int nr) {
  const float4* b0 = reinterpret_cast<const float4*>(k + min(t, w - 1) * SD);
  const float4* b1 = reinterpret_cast<const float4*>(k + min(t + 32, w - 1) * SD);
  float acc[CK_RPW][2];
#pragma unroll
  for (int r = 0; r < CK_RPW; ++r) acc[r][0] = acc[r][1] = 0.f;
#pragma unroll 2
  for (int d4 = 0; d4 < D / 4; ++d4) {
    const float4 y0 = b0[d4], y1 = b1[d4];
#pragma unroll
    for (int r = 0; r < CK_RPW; ++r) {
      const float4 x = reinterpret_cast<const float4*>(a + r * SD)[d4];
      acc[r][0] += x.x * y0.x + x.y * y0.y + x.z * y0.z + x.w * y0.w;
      acc[r][1] += x.x * y1.x + x.y * y1.y + x.z * y1.z + x.w * y1.w;
    }
  }
#pragma unroll
  for (int r = 0; r < CK_RPW; ++r) {
    if (row0 + r >= nr) break;
    if (t < w) dst[(row0 + r) * w + t] = acc[r][0] * scale;
    if (t + 32 < w) dst[(row0 + r) * w + t + 32] = acc[r][1] * scale;
  }
}

// Bound by the chain of its phases (load, four times: round trip, scores, log-softmax), not by any unit: 256 CTAs of
// 8 warps at 32 layers x 8 heads.  A warp keeps its four query rows from the scores to the KL, so a pass has two
// CTA-wide barriers (around the round trip); the key rows are padded by 16 bytes because lanes read the same channel of 32
// keys (without the padding every such load was a 32-way bank conflict), and the round trip quantizes with one reciprocal per
// group.  8 queries x 4 heads per KV head, 64-key window, 32 layers, block 64 / K group 32:
// 52 us a measurement, 570 us before (16 / 16: 40 us, 155 us before, at one query).
__global__ void __launch_bounds__(CK_THREADS) canary_kl_kernel(CanaryArgs A) {
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int layer = blockIdx.y;
  const int crank = (int)cluster.block_rank(), csize = (int)cluster.num_blocks();
  const int D = A.D, KG = A.KG, SD = D + 4;
  const int w = (A.ring_fill / KG) * KG;       // whole groups only; the newest w keys
  const int gqa = A.Hq / A.H;
  const int rows_total = A.nq * gqa;
  float* kr = sm;                    // [w][SD] K_ref window of this head
  float* kq = kr + w * SD;           // [w][SD] its round trip at the current tier
  float* qs = kq + w * SD;           // [CK_ROWS][SD] query rows
  float* lr = qs + CK_ROWS * SD;     // [CK_ROWS][w] reference log-weights
  float* lq = lr + CK_ROWS * w;      // [CK_ROWS][w] quantized log-weights
  __shared__ float red[CK_WARPS];
  __shared__ float cta_total[3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float total[3] = {0.f, 0.f, 0.f};

  for (int h = crank; h < A.H; h += csize) {
    __syncthreads();
    {
      const int per = A.k_vec ? D / 4 : D;  // loads per row
      const float* kh = A.kref + layer * A.k_sl + h * A.k_sh;
#pragma unroll 8
      for (int i = threadIdx.x; i < w * per; i += CK_THREADS) {
        const int t = i / per, c = i - t * per;
        const int v = A.ring_fill - w + t;  // index in the oldest-first view
        const int row = A.ring_fill < A.window ? v : (A.ring_pos + v) % A.window;
        const float* src = kh + (int64_t)row * A.k_sw;
        if (A.k_vec) reinterpret_cast<float4*>(kr + t * SD)[c] = reinterpret_cast<const float4*>(src)[c];
        else kr[t * SD + c] = src[c];
      }
    }
    for (int r0 = 0; r0 < rows_total; r0 += CK_ROWS) {
      const int nr = min(CK_ROWS, rows_total - r0);
      __syncthreads();
#pragma unroll 4
      for (int i = threadIdx.x; i < CK_ROWS * D; i += CK_THREADS) {  // rows past the end are zero
        const int r = i / D, d = i - r * D;
        float x = 0.f;
        if (r < nr) {
          const int rr = r0 + r, qi = rr / gqa, g = rr - qi * gqa;
          x = ld_dt(A.q, A.q_dt, layer * A.q_sl + (int64_t)qi * A.q_sq + (int64_t)(h * gqa + g) * A.q_sh + d);
        }
        qs[r * SD + d] = x;
      }
      const int row0 = warp * CK_RPW;  // this warp's rows
      for (int pass = 0; pass < 4; ++pass) {  // 0: reference, 1..3: tiers 2, 4, 8
        __syncthreads();
        const float* kk = kr;
        float* dst = lr;
        if (pass) {
          const int bits = 1 << pass;
          const float levels = (float)((1 << bits) - 1);
          for (int i = threadIdx.x; i < (w / KG) * D; i += CK_THREADS) {
            const int grp = i / D, d = i - grp * D;
            const float* src = kr + grp * KG * SD + d;
            float* to = kq + grp * KG * SD + d;
            float mn = INFINITY, mx = -INFINITY;
#pragma unroll 8
            for (int p = 0; p < KG; ++p) { const float x = src[p * SD]; mn = fminf(mn, x); mx = fmaxf(mx, x); }
            __half s16, m16;
            group_stats(mn, mx, levels, s16, m16);
            const float sc = __half2float(s16), m = __half2float(m16), rsc = __frcp_rn(sc);
#pragma unroll 8
            for (int p = 0; p < KG; ++p) {
              const float code = __fsub_rn(__uint_as_float(quant_u(src[p * SD], m, sc, rsc, levels)), QMAGIC);
              to[p * SD] = __fadd_rn(__fmul_rn(code, sc), m);
            }
          }
          __syncthreads();
          kk = kq;
          dst = lq;
        }
        if (row0 < nr) {
          for (int t = lane; t < w + lane; t += 64) score_rows(qs + row0 * SD, kk, t, w, D, SD, A.scale, dst, row0, nr);
        }
        __syncwarp();
        // log-softmax per row, and for tiers the row's KL
        float part = 0.f;
        for (int rr = row0; rr < min(row0 + CK_RPW, nr); ++rr) {
          float mx = -INFINITY;
          for (int t = lane; t < w; t += 32) mx = fmaxf(mx, dst[rr * w + t]);
#pragma unroll
          for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          float se = 0.f;
          for (int t = lane; t < w; t += 32) se += expf(dst[rr * w + t] - mx);
#pragma unroll
          for (int o = 16; o; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
          const float lse = mx + logf(se);
          float kl = 0.f;
          for (int t = lane; t < w; t += 32) {
            const float v = dst[rr * w + t] - lse;
            dst[rr * w + t] = v;
            if (pass) kl += expf(v) * (v - lr[rr * w + t]);
          }
          part += kl;
        }
        if (pass) total[pass - 1] += block_sum(part, red);
      }
    }
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < 3; ++b) cta_total[b] = total[b];
  }
  cluster.sync();  // every CTA's sums are in its shared memory
  if (crank == 0 && threadIdx.x == 0) {
    const float inv = 1.f / (float)(A.Hq * A.nq);
    for (int b = 0; b < 3; ++b) {
      float t = 0.f;
      for (int r = 0; r < csize; ++r) t += cluster.map_shared_rank(cta_total, r)[b];  // in CTA order = head order
      A.out[layer * 3 + b] = fmaxf(t * inv, 0.f);
    }
  }
  cluster.sync();  // no CTA leaves (and gives up its shared memory) before the first one has read it
}

}  // namespace echokv

using namespace echokv;

extern "C" int echokv_canary_kl(const void* query, int32_t q_dtype, int64_t q_sl, int64_t q_sq, int64_t q_sh,
                                const float* kref, int64_t k_sl, int64_t k_sw, int64_t k_sh, int32_t ring_pos,
                                int32_t ring_fill, int32_t window, int32_t num_layers, int32_t nq, int32_t num_q_heads,
                                int32_t num_kv_heads, int32_t head_size, int32_t k_group, float softmax_scale,
                                float* out, void* stream) {
  if (num_layers <= 0) return ECHOKV_OK;
  if (!query || !kref || !out) return set_error(ECHOKV_E_ARGUMENT, "canary_kl: null pointer");
  if (q_dtype < 0 || q_dtype > 2) return set_error(ECHOKV_E_ARGUMENT, "canary_kl: bad dtype");
  if (nq <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads || head_size % 4 || k_group <= 0 || window <= 0 ||
      ring_fill > window || ring_pos < 0 || ring_pos >= window)
    return set_error(ECHOKV_E_ARGUMENT, "canary_kl: bad shape");
  const int w = (ring_fill / k_group) * k_group;
  if (w == 0) return set_error(ECHOKV_E_ARGUMENT, "canary_kl: K_ref has %d keys, fewer than k_group=%d", ring_fill, k_group);
  if ((reinterpret_cast<uintptr_t>(kref) & 3) != 0) return set_error(ECHOKV_E_ARGUMENT, "canary_kl: misaligned K_ref");
  const size_t smem = (size_t)(2 * w * (head_size + 4) + CK_ROWS * (head_size + 4) + 2 * CK_ROWS * w) * sizeof(float);
  if (smem > 48 * 1024) {  // per call: the attribute belongs to the current device
    cudaError_t e = cudaFuncSetAttribute(canary_kl_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(ECHOKV_E_UNSUPPORTED, "canary_kl: window %d x head %d needs %zu bytes of shared memory", w, head_size, smem);
  }
  CanaryArgs A;
  A.q = query; A.q_dt = q_dtype; A.q_sl = q_sl; A.q_sq = q_sq; A.q_sh = q_sh;
  A.kref = kref; A.k_sl = k_sl; A.k_sw = k_sw; A.k_sh = k_sh;
  A.ring_pos = ring_pos; A.ring_fill = ring_fill; A.window = window;
  A.nq = nq; A.Hq = num_q_heads; A.H = num_kv_heads; A.D = head_size; A.KG = k_group;
  A.scale = softmax_scale; A.out = out;
  A.k_vec = ((reinterpret_cast<uintptr_t>(kref) & 15) | ((k_sl | k_sw | k_sh) & 3)) == 0;
  const int csize = num_kv_heads < 8 ? num_kv_heads : 8;  // 8 = the portable cluster size
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)csize, (unsigned)num_layers);
  cfg.blockDim = dim3(CK_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, canary_kl_kernel, A) != cudaSuccess) return check_launch("canary_kl");
  return check_launch("canary_kl");
}
