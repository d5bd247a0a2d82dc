// C ABI of split-K paged decode attention: argument checks and kernel selection.
#include <type_traits>

#include "decode_generic.cuh"

using namespace echokv;

namespace echokv {
int launch_decode_mma(const LayoutDev& L, const ResidualDev& R, const uint8_t* pages, const DecodeArgs& A,
                      int64_t num_seqs, int* counter, bool zero_counter, int* status, cudaStream_t st, bool* handled);
int decode_mma_teams(int H, int D, int VG, int KG, int BS, int gqa, int chunks);
int decode_status_take(bool clear);
int prefill_status_take(bool clear);

// out[q_rows[seq], head] = splits merged in split order (kernels/decode.py:226-262).  One warp per (sequence, query
// head), four heads per CTA: lane s holds split s's running maximum and denominator (further rounds when there are more
// than 32), the weights are exchanged by shuffles and a lane sums VEC channels over the splits, with the loads of
// eight splits in flight.  A sequence's result is a function of its own splits alone.
//
// Bound by its latency (split partials just written sit in L2): launch, one round of loads, the sum.  A thread per channel
// and a CTA per head (before) made 8,192 CTAs of a batch of 256 sequences x 32 heads: 27.8 us, now 6.7 us; one sequence x 8 splits 3.75 -> 2.5 us,
// 528 rows x 24 splits 54 -> 11 us.
constexpr int MERGE_HEADS = 4;
template <int VEC>
__global__ void __launch_bounds__(MERGE_HEADS * 32) decode_merge_kernel(DecodeArgs A, int BS, int D) {
  constexpr int BATCH = 8;
  using V = typename std::conditional<VEC == 4, float4, float2>::type;
  const int seq = blockIdx.x, head = blockIdx.y * MERGE_HEADS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int d = (blockIdx.z * 32 + lane) * VEC;  // this lane's channels
  pdl_launch_dependents();
  pdl_wait();  // the split kernel has completed
  if (seq == 0 && head == 0 && blockIdx.z == 0 && lane == 0) A.state[0] = 0;  // its item counter, for the next call
  if (head >= A.Hq) return;
  const int64_t base = ((int64_t)seq * A.Hq + head) * A.num_splits;
  const float* src = A.acc + base * D + min(d, D - VEC);
  // The first splits' partials are read along with the length that says how many there are (the rows exist either way).
  V x[BATCH];
  float2 ml = make_float2(-INFINITY, 0.f);
  if (lane < A.num_splits) ml = *reinterpret_cast<const float2*>(A.ml + (base + lane) * 2);
#pragma unroll
  for (int k = 0; k < BATCH; ++k) x[k] = *reinterpret_cast<const V*>(src + (int64_t)min(k, A.num_splits - 1) * D);
  const int64_t seq_len = A.lens[seq];
  const int64_t o_row = A.q_rows ? A.q_rows[seq] : seq;
  if (seq_len == 0) return;  // CUDA-graph padding: leave the row alone
  const int n_blocks = (int)((seq_len + BS - 1) / BS);
  const int bps = max(bps_floor(A), (n_blocks + A.num_splits - 1) / A.num_splits);
  const int used = (n_blocks + bps - 1) / bps;
  float m = lane < used ? ml.x : -INFINITY;
  for (int s0 = 32; s0 < used; s0 += 32)
    if (s0 + lane < used) m = fmaxf(m, A.ml[(base + s0 + lane) * 2]);
  m = warp_max(m);  // the overall maximum
  float acc[VEC];
#pragma unroll
  for (int k = 0; k < VEC; ++k) acc[k] = 0.f;
  float lt = 0.f;
  for (int s0 = 0; s0 < used; s0 += 32) {
    const bool on = s0 + lane < used;
    if (s0 > 0 && on) ml = *reinterpret_cast<const float2*>(A.ml + (base + s0 + lane) * 2);
    const float w = on ? exp2f(ml.x - m) : 0.f;
    lt += on ? ml.y * w : 0.f;
    const int n = min(32, used - s0);
    for (int s = 0; s < n; s += BATCH) {
      if (s0 + s > 0) {
#pragma unroll
        for (int k = 0; k < BATCH; ++k) x[k] = *reinterpret_cast<const V*>(src + (int64_t)min(s0 + s + k, used - 1) * D);
      }
#pragma unroll
      for (int k = 0; k < BATCH; ++k) {
        const float wk = __shfl_sync(0xffffffffu, w, s + k);
        if (s + k < n) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[e] += reinterpret_cast<const float*>(&x[k])[e] * wk;
        }
      }
    }
  }
  lt = warp_sum(lt);
  if (d >= D) return;
  const int64_t o = o_row * A.o_s0 + (int64_t)head * A.o_s1 + d;
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] /= lt;
  if (A.out_vec) {  // 16-bit rows that take a lane's channels as one store
    uint32_t w[VEC / 2];
#pragma unroll
    for (int e = 0; e < VEC / 2; ++e) {
      if (A.out_dt == ECHOKV_DT_BF16) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(acc[2 * e], acc[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&p);
      } else {
        const __half2 p = __floats2half2_rn(acc[2 * e], acc[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&p);
      }
    }
    uint16_t* dst = reinterpret_cast<uint16_t*>(A.out) + o;
    if constexpr (VEC == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    else *reinterpret_cast<uint32_t*>(dst) = w[0];
  } else {
#pragma unroll
    for (int e = 0; e < VEC; ++e) st_dt(A.out, A.out_dt, o + e, acc[e]);
  }
}

}  // namespace echokv

template <int GQ>
static int launch_generic_gq(const LayoutDev& L, const ResidualDev& R, const uint8_t* pages, const DecodeArgs& A,
                             dim3 grid, cudaStream_t st) {
  switch (L.D) {
    case 64: decode_generic_kernel<GQ, 2><<<grid, DG_WARPS * 32, 0, st>>>(L, R, pages, A); break;
    case 128: decode_generic_kernel<GQ, 4><<<grid, DG_WARPS * 32, 0, st>>>(L, R, pages, A); break;
    case 256:
      if constexpr (GQ <= 8) {
        decode_generic_kernel<GQ, 8><<<grid, DG_WARPS * 32, 0, st>>>(L, R, pages, A);
        break;
      } else {
        return set_error(ECHOKV_E_UNSUPPORTED, "decode: head_size 256 supports at most 8 query heads per KV head");
      }
    default: return set_error(ECHOKV_E_UNSUPPORTED, "decode: head_size %d is not one of 64/128/256", L.D);
  }
  return ECHOKV_OK;
}

extern "C" {

int64_t echokv_decode_scratch_bytes(int64_t num_seqs, int32_t num_q_heads, int32_t head_size, int32_t num_splits) {
  if (num_seqs <= 0 || num_q_heads <= 0 || head_size <= 0 || num_splits <= 0) return 0;
  // 256 bytes of work-queue state, then the split partials (accumulators + running max / sum)
  const int64_t partials = num_seqs * num_q_heads * (int64_t)num_splits * (head_size + 2) * (int64_t)sizeof(float);
  return (partials + 15) / 16 * 16 + 256;
}

static int decode_impl(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                       const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                       const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                       void* scratch, int64_t scratch_bytes, void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype,
                       float softmax_scale, int32_t num_splits, int32_t blocks_per_split,
                       const int32_t* blocks_per_split_dev, bool zero_state, bool planned, int64_t num_seqs,
                       int32_t num_q_heads, void* stream, const int64_t* groups = nullptr, int64_t num_groups = 0,
                       int32_t group_tokens = 1, const int64_t* split_lens = nullptr) {
  if (num_seqs <= 0) return ECHOKV_OK;
  LayoutDev L;
  ResidualDev R;
  int rc = make_layout(layout, pages, &L);
  if (rc) return rc;
  rc = make_residual(residual, &R);
  if (rc) return rc;
  if (!query || !block_table || !lens || !scratch || !out) return set_error(ECHOKV_E_ARGUMENT, "decode: null pointer");
  if (num_splits < 1 || blocks_per_split < 1) return set_error(ECHOKV_E_ARGUMENT, "decode: num_splits and blocks_per_split must be >= 1");
  if (num_q_heads % L.H) return set_error(ECHOKV_E_ARGUMENT, "decode: %d query heads not a multiple of %d KV heads", num_q_heads, L.H);
  if (q_dtype < 0 || q_dtype > 2 || out_dtype < 0 || out_dtype > 2) return set_error(ECHOKV_E_ARGUMENT, "decode: bad dtype");
  const int gqa = num_q_heads / L.H;
  if (scratch_bytes < echokv_decode_scratch_bytes(num_seqs, num_q_heads, L.D, num_splits) || (reinterpret_cast<uintptr_t>(scratch) & 15))
    return set_error(ECHOKV_E_ARGUMENT, "decode: scratch too small (%lld bytes) or misaligned", (long long)scratch_bytes);
  if (gqa > 16) return set_error(ECHOKV_E_UNSUPPORTED, "decode: %d query heads per KV head (max 16)", gqa);

  DecodeArgs A;
  A.q = query; A.q_s0 = q_s0; A.q_s1 = q_s1; A.q_dt = q_dtype; A.q_rows = q_rows;
  A.bt = block_table; A.bt_s0 = bt_s0; A.bt_rows = bt_rows; A.lens = lens;
  // scratch = [256 bytes of work-queue state][split partials: accumulators, then running max / sum]
  A.state = reinterpret_cast<int*>(scratch);
  A.acc = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(scratch) + 256);
  A.ml = A.acc + num_seqs * num_q_heads * (int64_t)num_splits * L.D;
  A.out = out; A.o_s0 = o_s0; A.o_s1 = o_s1; A.out_dt = out_dtype;
  A.scale_log2e = softmax_scale * 1.4426950408889634f;
  A.num_splits = num_splits; A.bps_min = blocks_per_split; A.gqa = gqa; A.Hq = num_q_heads;
  A.bps_dev = blocks_per_split_dev;
  A.planned = planned;
  A.groups = nullptr; A.tok = 1;
  cudaStream_t st = (cudaStream_t)stream;
  const uint8_t* pg = (const uint8_t*)pages->base;

  bool handled = false;
  // Groups of consecutive tokens, where the query heads of two or more tokens fit the columns of the tensor-core kernel's MMAs (a step
  // of 16 chunks of 33 tokens, 32 / 8 heads: 1.72 -> 1.10 ms).  Their partials are those of the tokens one by one, so the merge is too.
  if (num_groups > 0 && group_tokens > 1) {
    DecodeArgs G = A;
    G.groups = groups; G.tok = group_tokens;
    rc = launch_decode_mma(L, R, pg, G, num_groups, A.state, zero_state, nullptr, st, &handled);
    if (rc) return rc;
    if (handled) A.lens = split_lens;
  }
  if (!handled) {
    rc = launch_decode_mma(L, R, pg, A, num_seqs, A.state, zero_state, nullptr, st, &handled);
    if (rc) return rc;
  }
  if (!handled) {
    dim3 grid((unsigned)num_seqs, (unsigned)L.H, (unsigned)num_splits);
    if (gqa == 1) rc = launch_generic_gq<1>(L, R, pg, A, grid, st);
    else if (gqa == 2) rc = launch_generic_gq<2>(L, R, pg, A, grid, st);
    else if (gqa <= 4) rc = launch_generic_gq<4>(L, R, pg, A, grid, st);
    else if (gqa <= 8) rc = launch_generic_gq<8>(L, R, pg, A, grid, st);
    else rc = launch_generic_gq<16>(L, R, pg, A, grid, st);
    if (rc) return rc;
    rc = check_launch("decode");
    if (rc) return rc;
  }
  dim3 mgrid((unsigned)num_seqs, (unsigned)((num_q_heads + MERGE_HEADS - 1) / MERGE_HEADS), (unsigned)((L.D + 127) / 128));
  const int vec = L.D == 64 ? 2 : 4;
  A.out_vec = out_dtype != ECHOKV_DT_F32 && ((o_s0 | o_s1) % vec) == 0 && (reinterpret_cast<uintptr_t>(out) % (2 * vec)) == 0;
  cudaError_t e;
  if (L.D == 64) e = launch_pdl(decode_merge_kernel<2>, mgrid, dim3(MERGE_HEADS * 32), 0, st, A, L.BS, L.D);
  else e = launch_pdl(decode_merge_kernel<4>, mgrid, dim3(MERGE_HEADS * 32), 0, st, A, L.BS, L.D);
  if (e != cudaSuccess) return check_launch("decode merge");
  return check_launch("decode merge");
}

int echokv_decode_ex(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                     const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                     const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                     void* scratch, int64_t scratch_bytes, void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype,
                     float softmax_scale, int32_t num_splits, int32_t blocks_per_split,
                     const int32_t* blocks_per_split_dev, int64_t num_seqs, int32_t num_q_heads, void* stream) {
  return decode_impl(layout, pages, residual, query, q_s0, q_s1, q_dtype, q_rows, block_table, bt_s0, bt_rows, lens, scratch,
                     scratch_bytes, out, o_s0, o_s1, out_dtype, softmax_scale, num_splits, blocks_per_split,
                     blocks_per_split_dev, false, false, num_seqs, num_q_heads, stream);
}

int echokv_decode_step(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                       const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                       const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                       void* scratch, int64_t scratch_bytes, void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype,
                       float softmax_scale, int32_t num_splits, int32_t blocks_per_split,
                       const int32_t* blocks_per_split_dev, int64_t num_seqs, int32_t num_q_heads, void* stream) {
  return decode_impl(layout, pages, residual, query, q_s0, q_s1, q_dtype, q_rows, block_table, bt_s0, bt_rows, lens, scratch,
                     scratch_bytes, out, o_s0, o_s1, out_dtype, softmax_scale, num_splits, blocks_per_split,
                     blocks_per_split_dev, false, true, num_seqs, num_q_heads, stream);
}

int echokv_decode_chunks(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                         const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                         const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                         void* scratch, int64_t scratch_bytes, void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype,
                         float softmax_scale, int32_t num_splits, int32_t blocks_per_split, const int64_t* groups,
                         int64_t num_groups, int32_t group_tokens, const int64_t* split_lens, int64_t num_seqs, int32_t num_q_heads,
                         void* stream) {
  if (num_groups > 0 && (!groups || !split_lens || group_tokens < 1))
    return set_error(ECHOKV_E_ARGUMENT, "decode_chunks: groups need their records, their tokens' split lengths and a size");
  return decode_impl(layout, pages, residual, query, q_s0, q_s1, q_dtype, q_rows, block_table, bt_s0, bt_rows, lens, scratch,
                     scratch_bytes, out, o_s0, o_s1, out_dtype, softmax_scale, num_splits, blocks_per_split,
                     nullptr, false, false, num_seqs, num_q_heads, stream, groups, num_groups, group_tokens, split_lens);
}

int echokv_decode(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                  const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                  const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                  void* scratch, int64_t scratch_bytes, void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype,
                  float softmax_scale, int32_t num_splits, int32_t blocks_per_split, int64_t num_seqs,
                  int32_t num_q_heads, void* stream) {
  return decode_impl(layout, pages, residual, query, q_s0, q_s1, q_dtype, q_rows, block_table, bt_s0, bt_rows, lens, scratch,
                     scratch_bytes, out, o_s0, o_s1, out_dtype, softmax_scale, num_splits, blocks_per_split, nullptr, true, false,
                     num_seqs, num_q_heads, stream);
}

// Work items the tensor-core split kernel processes at the same time on the current device for this shape (its
// teams: one per group of H consumer warps), or 0 when the shape takes the generic kernel.
int32_t echokv_decode_parallelism(const echokv_layout* layout, int32_t num_q_heads) {
  if (!layout || layout->num_kv_heads <= 0 || num_q_heads <= 0 || num_q_heads % layout->num_kv_heads) return 0;
  return decode_mma_teams(layout->num_kv_heads, layout->head_size, layout->v_group, layout->k_group, layout->block_size,
                          num_q_heads / layout->num_kv_heads, layout->mem_bits / 2);
}


// ---- decode without any allocation by the caller ------------------------------------------------
// Some callers of echokv_decode cannot provide scratch memory: code that runs inside another
// framework's memory pool with allocation forbidden at that point (for example while that
// framework is capturing or replaying its own graphs, or in a plugin that is handed only the
// input and output buffers), or a C host that links this library but not a CUDA allocator.  For
// them the split partials live in a fixed array inside the library itself.
#define ECHOKV_STATIC_SCRATCH_BYTES (8u << 20)
static __device__ __align__(256) unsigned char g_static_decode_scratch[ECHOKV_STATIC_SCRATCH_BYTES];

int64_t echokv_decode_static_scratch_bytes(void) { return (int64_t)ECHOKV_STATIC_SCRATCH_BYTES; }

int echokv_decode_static(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                         const void* query, int64_t q_s0, int64_t q_s1, int32_t q_dtype, const int64_t* q_rows,
                         const int32_t* block_table, int64_t bt_s0, const int64_t* bt_rows, const int64_t* lens,
                         void* out, int64_t o_s0, int64_t o_s1, int32_t out_dtype, float softmax_scale,
                         int32_t num_splits, int32_t blocks_per_split, int64_t num_seqs, int32_t num_q_heads,
                         void* stream) {
  if (num_seqs <= 0) return ECHOKV_OK;
  if (!layout) return set_error(ECHOKV_E_ARGUMENT, "decode_static: layout is null");
  if (num_q_heads <= 0 || layout->head_size <= 0 || num_splits <= 0)
    return set_error(ECHOKV_E_ARGUMENT, "decode_static: num_q_heads, head_size and num_splits must be positive");
  const int64_t need = echokv_decode_scratch_bytes(num_seqs, num_q_heads, layout->head_size, num_splits);
  if (need > (int64_t)ECHOKV_STATIC_SCRATCH_BYTES)
    return set_error(ECHOKV_E_UNSUPPORTED,
                     "decode_static: %lld sequences x %d query heads x %d splits need %lld bytes of split partials, "
                     "the built-in scratch holds %lld; use echokv_decode with caller-provided scratch",
                     (long long)num_seqs, num_q_heads, num_splits, (long long)need,
                     (long long)ECHOKV_STATIC_SCRATCH_BYTES);
  // The array's name is only a host-side handle; its device address is looked up once per device,
  // with that device current.
  constexpr int MAX_DEVICES = 64;
  static void* device_ptr[MAX_DEVICES] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error(ECHOKV_E_CUDA, "decode_static: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= MAX_DEVICES) return set_error(ECHOKV_E_UNSUPPORTED, "decode_static: device index %d", dev);
  if (!device_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_decode_scratch);
    if (e != cudaSuccess || !p)
      return set_error(ECHOKV_E_CUDA, "decode_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    device_ptr[dev] = p;
  }
  return echokv_decode(layout, pages, residual, query, q_s0, q_s1, q_dtype, q_rows, block_table, bt_s0, bt_rows, lens,
                       device_ptr[dev], (int64_t)ECHOKV_STATIC_SCRATCH_BYTES, out, o_s0, o_s1, out_dtype, softmax_scale,
                       num_splits, blocks_per_split, num_seqs, num_q_heads, stream);
}

int echokv_kernel_status(int clear) {
  const int d = decode_status_take(clear != 0), p = prefill_status_take(clear != 0);
  if (d < 0 || p < 0) return set_error(ECHOKV_E_CUDA, "kernel_status: cannot read the status words"), -1;
  return (d == 1 ? 1 : 0) | (d == 2 ? 2 : 0) | (p ? 4 : 0);
}

}  // extern "C"
