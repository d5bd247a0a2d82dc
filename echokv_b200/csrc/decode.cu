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

// out[q_rows[seq], head] = the splits' partials weighted by their maxima and added up (kernels/decode.py:226-262).  W warps
// share a (sequence, query head): lane s holds the running maximum and denominator of splits s and s + 32 (further rounds
// when there are more than 64), the weights are exchanged by shuffles and a lane sums VEC channels.  The sum has one order
// whatever W is: splits s, s + 8, s + 16, ... one after the other for each of s = 0 .. 7, then these eight as a tree; so a
// sequence's result is a function of its own splits alone, and the batch may choose W.
//
// Bound by its latency (split partials just written sit in L2): launch, the rounds of loads, the sum.  With a warp per head
// 64 splits were eight rounds of loads one after the other, of more than a microsecond each.  From the merge to the next
// layer's write in a decode step, a warp per head throughout and now: 8 sequences x 32 heads, 33 splits 7.0 -> 2.7 us;
// 16 x 8, 62 splits 12.7 -> 3.1; 48 x 16, 11 splits 6.3 -> 3.5; 64 x 32, 9 splits 5.1 -> 3.7; 256 x 32, 1 or 2 splits 7.1 -> 6.8.
// W is the largest with heads x W <= MERGE_WARPS (16 warps an SM) that leaves a warp more than two of the splits there may be:
// 48 x 16 heads take 3.6 us at W = 2 and 5.0 at 4, 64 x 32 take 3.6 at 1 and 4.8 at 2.
// The rule sees the grid, not the splits in use: a layer's step of two sequences x 32 heads in blocks of 64 takes 18.9 us at 3,000 tokens
// (20.8 with a warp per head), but at 60 to 500 tokens 17.7 - 18.7 (16.3 - 17.0).  Registers for the merge beside a split CTA (80, or 40 at W = 8)
// do not pay: steps of 1 to 256 sequences 0.4 and 3 % slower.
constexpr int MERGE_SUMS = 8;      // independent sums over the splits
constexpr int MERGE_ROUND = 64;    // splits whose maxima and denominators a warp holds at a time
constexpr int64_t MERGE_WARPS = 2400;
// FEW (W = 1): calls of at most FEW_SPLITS splits, whose sums are a product each: 48 registers instead of 94, more warps
// (528 tokens x 32 heads, 2 splits: 13.1 us before, 10.2 now, under ncu).
constexpr int FEW_SPLITS = 4;
template <int VEC, int W, bool FEW>
__global__ void __launch_bounds__(W == 8 ? 256 : 128, W == 1 ? (FEW ? 8 : 5) : 1) decode_merge_kernel(DecodeArgs A, int BS, int D) {
  constexpr int HEADS = W == 8 ? 1 : 4 / W;   // per CTA
  constexpr int OWN = MERGE_SUMS / W;         // sums of this warp
  constexpr int LOADS = W == 1 ? FEW_SPLITS : MERGE_SUMS;  // splits in flight; with a warp per head the heads are many and registers limit the warps
  using V = typename std::conditional<VEC == 4, float4, float2>::type;
  __shared__ __align__(16) float part[W == 1 ? 1 : HEADS * W][32 * VEC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, me = warp % W;
  const int seq = blockIdx.x, slot = blockIdx.y * HEADS + warp / W, head = min(slot, A.Hq - 1);
  const int d = (blockIdx.z * 32 + lane) * VEC;  // this lane's channels
  pdl_launch_dependents();
  // In a planned step the lengths were final before the step's first write (see common.cuh): they are read ahead of the wait,
  // and only partials that exist are read behind it.  Otherwise the first splits' partials are read along with the length
  // that says how many there are (the rows exist either way); with a warp per head, whose warps hide one another's
  // latency, behind it.
  int64_t seq_len = 0, o_row = seq;
  int used = A.num_splits;
  auto plan = [&]() {
    seq_len = A.lens[seq];
    if (A.q_rows) o_row = A.q_rows[seq];
    const int n_blocks = (int)((seq_len + BS - 1) / BS);
    const int bps = max(bps_floor(A), (n_blocks + A.num_splits - 1) / A.num_splits);
    used = (n_blocks + bps - 1) / bps;
  };
  if (A.planned) plan();
  pdl_wait();  // the split kernel has completed
  if (W == 1 && !A.planned) plan();
  if (seq == 0 && slot == 0 && blockIdx.z == 0 && me == 0 && lane == 0) A.state[0] = 0;  // its item counter, for the next call
  const int64_t base = ((int64_t)seq * A.Hq + head) * A.num_splits;
  const float* src = A.acc + base * D + min(d, D - VEC);
  // Split of this warp's load k of the batch that starts at split s: sums me * OWN .. of W consecutive groups of eight.
  auto split_of = [&](int s, int k) { return s + (k / OWN) * MERGE_SUMS + me * OWN + k % OWN; };
  V x[LOADS];
  float2 ml[2] = {make_float2(-INFINITY, 0.f), make_float2(-INFINITY, 0.f)};
#pragma unroll
  for (int r = 0; r < 2; ++r)
    if (r * 32 + lane < used) ml[r] = *reinterpret_cast<const float2*>(A.ml + (base + r * 32 + lane) * 2);
#pragma unroll
  for (int k = 0; k < LOADS; ++k)
    if (split_of(0, k) < used) x[k] = *reinterpret_cast<const V*>(src + (int64_t)split_of(0, k) * D);
  if (W > 1 && !A.planned) plan();
  if (seq_len == 0) return;  // CUDA-graph padding: leave the row alone
  float m = fmaxf(lane < used ? ml[0].x : -INFINITY, 32 + lane < used ? ml[1].x : -INFINITY);
  for (int s0 = MERGE_ROUND; s0 < used; s0 += 32)
    if (s0 + lane < used) m = fmaxf(m, A.ml[(base + s0 + lane) * 2]);
  m = warp_max(m);  // the overall maximum
  __align__(16) float sum[VEC];
  float lt = 0.f;
  if constexpr (FEW) {
    const float w = lane < used ? exp2f(ml[0].x - m) : 0.f;
    lt = lane < used ? ml[0].y * w : 0.f;
    float t[FEW_SPLITS][VEC];
#pragma unroll
    for (int k = 0; k < FEW_SPLITS; ++k) {
      const float wk = __shfl_sync(0xffffffffu, w, k);
#pragma unroll
      for (int e = 0; e < VEC; ++e) t[k][e] = k < used ? __fmul_rn(reinterpret_cast<const float*>(&x[k])[e], wk) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) sum[e] = __fadd_rn(__fadd_rn(t[0][e], t[1][e]), __fadd_rn(t[2][e], t[3][e]));
  } else {
    float acc[OWN][VEC];
#pragma unroll
    for (int i = 0; i < OWN; ++i)
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[i][e] = 0.f;
    for (int s0 = 0; s0 < used; s0 += MERGE_ROUND) {
      float w[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int s = s0 + r * 32 + lane;
        if (s0 > 0 && s < used) ml[r] = *reinterpret_cast<const float2*>(A.ml + (base + s) * 2);
        w[r] = s < used ? exp2f(ml[r].x - m) : 0.f;
        lt += s < used ? ml[r].y * w[r] : 0.f;
      }
      const int end = min(s0 + MERGE_ROUND, used);
      for (int s = s0; s < end; s += MERGE_SUMS * W) {
#pragma unroll
        for (int k0 = 0; k0 < MERGE_SUMS; k0 += LOADS) {
          if (s > 0 || k0 > 0) {
#pragma unroll
            for (int k = 0; k < LOADS; ++k)
              if (split_of(s, k0 + k) < used) x[k] = *reinterpret_cast<const V*>(src + (int64_t)split_of(s, k0 + k) * D);
          }
#pragma unroll
          for (int k = 0; k < LOADS; ++k) {
            const int sk = split_of(s, k0 + k), at = sk - s0;
            const float wk = __shfl_sync(0xffffffffu, at < 32 ? w[0] : w[1], at & 31);
            if (sk < used) {
#pragma unroll
              for (int e = 0; e < VEC; ++e) acc[(k0 + k) % OWN][e] += reinterpret_cast<const float*>(&x[k])[e] * wk;
            }
          }
          if (s + k0 + LOADS >= end) break;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      float t[OWN];
#pragma unroll
      for (int i = 0; i < OWN; ++i) t[i] = acc[i][e];
#pragma unroll
      for (int n = OWN / 2; n >= 1; n /= 2)
#pragma unroll
        for (int i = 0; i < n; ++i) t[i] = t[2 * i] + t[2 * i + 1];
      sum[e] = t[0];
    }
  }
  lt = warp_sum(lt);
  if constexpr (W > 1) {
    *reinterpret_cast<V*>(&part[warp][lane * VEC]) = *reinterpret_cast<const V*>(sum);
    __syncthreads();
    if (me != 0) return;
    __align__(16) float t[W][VEC];
#pragma unroll
    for (int i = 0; i < W; ++i) *reinterpret_cast<V*>(t[i]) = *reinterpret_cast<const V*>(&part[warp + i][lane * VEC]);
#pragma unroll
    for (int n = W / 2; n >= 1; n /= 2)
#pragma unroll
      for (int i = 0; i < n; ++i)
#pragma unroll
        for (int e = 0; e < VEC; ++e) t[i][e] = t[2 * i][e] + t[2 * i + 1][e];
#pragma unroll
    for (int e = 0; e < VEC; ++e) sum[e] = t[0][e];
  }
  if (slot >= A.Hq || d >= D) return;
  const int64_t o = o_row * A.o_s0 + (int64_t)head * A.o_s1 + d;
#pragma unroll
  for (int e = 0; e < VEC; ++e) sum[e] /= lt;
  if (A.out_vec) {  // 16-bit rows that take a lane's channels as one store
    uint32_t w[VEC / 2];
#pragma unroll
    for (int e = 0; e < VEC / 2; ++e) {
      if (A.out_dt == ECHOKV_DT_BF16) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(sum[2 * e], sum[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&p);
      } else {
        const __half2 p = __floats2half2_rn(sum[2 * e], sum[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&p);
      }
    }
    uint16_t* dst = reinterpret_cast<uint16_t*>(A.out) + o;
    if constexpr (VEC == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    else *reinterpret_cast<uint32_t*>(dst) = w[0];
  } else {
#pragma unroll
    for (int e = 0; e < VEC; ++e) st_dt(A.out, A.out_dt, o + e, sum[e]);
  }
}

template <int VEC, int W, bool FEW = false>
static cudaError_t launch_merge_w(const DecodeArgs& A, int64_t num_seqs, int BS, int D, cudaStream_t st) {
  constexpr int HEADS = W == 8 ? 1 : 4 / W;
  return launch_pdl(decode_merge_kernel<VEC, W, FEW>, dim3((unsigned)num_seqs, (unsigned)((A.Hq + HEADS - 1) / HEADS), (unsigned)((D + 127) / 128)),
                    dim3(W == 8 ? 256 : 128), 0, st, A, BS, D);
}
template <int VEC>
static cudaError_t launch_merge(const DecodeArgs& A, int64_t num_seqs, int BS, int D, cudaStream_t st) {
  const int64_t heads = num_seqs * A.Hq;
  if (A.num_splits > 16 && heads * 8 <= MERGE_WARPS) return launch_merge_w<VEC, 8>(A, num_seqs, BS, D, st);
  if (A.num_splits > 8 && heads * 4 <= MERGE_WARPS) return launch_merge_w<VEC, 4>(A, num_seqs, BS, D, st);
  if (A.num_splits > 4 && heads * 2 <= MERGE_WARPS) return launch_merge_w<VEC, 2>(A, num_seqs, BS, D, st);
  if (A.num_splits <= FEW_SPLITS) return launch_merge_w<VEC, 1, true>(A, num_seqs, BS, D, st);
  return launch_merge_w<VEC, 1>(A, num_seqs, BS, D, st);
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
  const int vec = L.D == 64 ? 2 : 4;
  A.out_vec = out_dtype != ECHOKV_DT_F32 && ((o_s0 | o_s1) % vec) == 0 && (reinterpret_cast<uintptr_t>(out) % (2 * vec)) == 0;
  const cudaError_t e = L.D == 64 ? launch_merge<2>(A, num_seqs, L.BS, L.D, st) : launch_merge<4>(A, num_seqs, L.BS, L.D, st);
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
