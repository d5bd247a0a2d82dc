// Read-side dequantization kernels: arbitrary token gather (the store's oracle read), dense
// dequantization of whole contexts for chunked prefill, and LRU demotion to INT2.
#include "common.cuh"

namespace echokv {

// Dequantize 8 channels [d0, d0+8) of head h of token (blk, off): K and V as float.
// Mirrors TieredKVCache.gather (echokv_vllm/tiered_cache.py:451-478) / load_kv_tile
// (kernels/common.py:50-109): K comes from the residual when the token's group is the
// block's open group.  `zero_unopened`: blocks with tier 0 give zeros (gather) instead of
// being read as INT2 (the attention kernels).
__device__ __forceinline__ void dequant8(const LayoutDev& L, const ResidualDev& R, const uint8_t* pages, int64_t blk,
                                         int off, int h, int d0, bool zero_unopened, float (&k)[8], float (&v)[8]) {
  const uint8_t* page = pages + blk * L.PS;
  int bits = page[0];
  if (bits == 0) {
    if (zero_unopened) {
#pragma unroll
      for (int i = 0; i < 8; ++i) k[i] = v[i] = 0.f;
      return;
    }
    bits = 2;
  }
  const int64_t ro = row_offset(pages, L, blk, off, bits);
  const int side_bytes = (L.H * L.D * bits) / 8;
  const int head_bytes = (L.D * bits) / 8;
  const uint8_t* krow = pages + ro + h * head_bytes;
  const uint8_t* vrow = krow + side_bytes;
  // V: per-token stats per group of VG channels
  const int g = d0 / L.VG;
  const int64_t ve = ((int64_t)off * L.H + h) * L.NG + g;
  const float vs = __half2float(reinterpret_cast<const __half*>(page + L.o_vs)[ve]);
  const float vm = __half2float(reinterpret_cast<const __half*>(page + L.o_vm)[ve]);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __fadd_rn(__fmul_rn((float)extract_code(vrow, d0 + i, bits), vs), vm);
  // K
  const int grp = off / L.KG;
  const int64_t slot = R.block_res[blk];
  if (slot >= 0 && R.res_group[slot] == grp) {
    const int64_t o = slot * R.s_slot + (int64_t)(off % L.KG) * R.s_pos + h * R.s_head + d0;
#pragma unroll
    for (int i = 0; i < 8; ++i) k[i] = ld_dt(R.base, R.dtype, o + i);
  } else {
    const int64_t ke = ((int64_t)grp * L.H + h) * L.D + d0;
    const __half* ks = reinterpret_cast<const __half*>(page + L.o_ks) + ke;
    const __half* km = reinterpret_cast<const __half*>(page + L.o_km) + ke;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      k[i] = __fadd_rn(__fmul_rn((float)extract_code(krow, d0 + i, bits), __half2float(ks[i])), __half2float(km[i]));
  }
}

__global__ void gather_kernel(LayoutDev L, ResidualDev R, const uint8_t* __restrict__ pages,
                              const int64_t* __restrict__ blk, const int64_t* __restrict__ off, int64_t n,
                              float* __restrict__ k_out, float* __restrict__ v_out) {
  const int cpt = (L.H * L.D) / 8;  // chunks per token
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= n * cpt) return;
  const int64_t i = idx / cpt;
  const int c = (int)(idx % cpt);
  const int h = (c * 8) / L.D, d0 = (c * 8) % L.D;
  float k[8], v[8];
  dequant8(L, R, pages, blk[i], (int)off[i], h, d0, true, k, v);
  float* ko = k_out + (i * L.H + h) * L.D + d0;
  float* vo = v_out + (i * L.H + h) * L.D + d0;
#pragma unroll
  for (int j = 0; j < 8; ++j) { ko[j] = k[j]; vo[j] = v[j]; }
}

// One CTA per work item (request, block index, dense row, ctx) -- kernels/prefill.py:329-369.
template <typename T>
__global__ void __launch_bounds__(256)
dequant_dense_kernel(LayoutDev L, ResidualDev R, const uint8_t* __restrict__ pages, const int32_t* __restrict__ work,
                     const int32_t* __restrict__ bt, int64_t bt_s0, T* __restrict__ k_out, T* __restrict__ v_out,
                     int64_t o_s0, int64_t o_s1) {
  const int32_t* w = work + blockIdx.x * 4;
  const int req = w[0], bi = w[1], ctx = w[3];
  const int64_t row0 = w[2];
  const int64_t blk = bt[(int64_t)req * bt_s0 + bi];
  const int nvalid = min(L.BS, ctx - bi * L.BS);
  const int cpt = (L.H * L.D) / 8;
  for (int idx = threadIdx.x; idx < nvalid * cpt; idx += blockDim.x) {
    const int t = idx / cpt, c = idx % cpt;
    const int h = (c * 8) / L.D, d0 = (c * 8) % L.D;
    float k[8], v[8];
    dequant8(L, R, pages, blk, t, h, d0, false, k, v);
    const int64_t o = (row0 + t) * o_s0 + h * o_s1 + d0;
#pragma unroll
    for (int j = 0; j < 8; ++j) { Elem<T>::st(k_out, o + j, k[j]); Elem<T>::st(v_out, o + j, v[j]); }
  }
}

// The same for 16-bit outputs whose rows allow 16-byte stores: one CTA per 16 tokens of a work item, one thread per
// 8 channels and every (256 / (H * D / 8))-th of the tokens.  The arithmetic is dequant8's: code * scale + min in fp32, two
// roundings, two values per instruction.
//
// Bound by its instructions, and for few blocks by the chain work item -> block table -> header -> rows, so a CTA is
// as small as keeps that chain worth it (a 64-token block as one CTA left 34 CTAs of 32 rounds each for a 2,112-token context:
// 60 us, now 6.5 us), a thread stays on its channels (its K group's statistics are read once) with four tokens' loads
// in flight, and a code becomes a float with one byte permute.  8 x 8,704 tokens x 8 heads x 128 at INT4 / INT8
// alternating: 96 us, 156 us before = 0.61 of the measured copy peak at INT4 + INT8's mean of 383 MB.
template <typename T> __device__ __forceinline__ uint32_t pack2_rn(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2_rn<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2_rn<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 8 codes as four float pairs.  A code c < 2^23 placed in the mantissa of 2^23 is the float 2^23 + c (one byte permute),
// and subtracting 2^23 is exact.
__device__ __forceinline__ float code_byte(uint32_t w, int k) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k));
}
__device__ __forceinline__ float2 code_pair(uint32_t wa, int ka, uint32_t wb, int kb) {
  return __fadd2_rn(make_float2(code_byte(wa, ka), code_byte(wb, kb)), make_float2(-8388608.f, -8388608.f));
}
template <int BITS> struct Codes8;  // 8 packed codes as loaded
template <> struct Codes8<8> { using W = uint2; };
template <> struct Codes8<4> { using W = uint32_t; };
template <> struct Codes8<2> { using W = uint16_t; };
template <int BITS>
__device__ __forceinline__ void unpack8(const typename Codes8<BITS>::W& w, float2 (&q)[4]) {
  if constexpr (BITS == 8) {
    q[0] = code_pair(w.x, 0, w.x, 1); q[1] = code_pair(w.x, 2, w.x, 3);
    q[2] = code_pair(w.y, 0, w.y, 1); q[3] = code_pair(w.y, 2, w.y, 3);
  } else if constexpr (BITS == 4) {
    const uint32_t e = w & 0x0F0F0F0Fu, o = (w >> 4) & 0x0F0F0F0Fu;
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = code_pair(e, i, o, i);
  } else {
    const uint32_t x = w, c0 = x & 0x0303u, c1 = (x >> 2) & 0x0303u, c2 = (x >> 4) & 0x0303u, c3 = (x >> 6) & 0x0303u;
    q[0] = code_pair(c0, 0, c1, 0); q[1] = code_pair(c2, 0, c3, 0);
    q[2] = code_pair(c0, 1, c1, 1); q[3] = code_pair(c2, 1, c3, 1);
  }
}

constexpr int DENSE_TOK = 16;   // tokens per CTA
constexpr int DENSE_BATCH = 4;  // of which a thread has this many in flight

template <typename T>
struct DenseArgs {
  LayoutDev L;
  ResidualDev R;
  const uint8_t* pages;
  const int32_t* work;
  const int32_t* bt;
  int64_t bt_s0;
  T *k_out, *v_out;
  int64_t o_s0, o_s1;
  int slices;  // CTAs per block
};

// Tokens [t0, t1) of one block of tier BITS; `s_row`: byte offset of each token's row from the pool base.  The loads of
// a batch of tokens are issued together; the K statistics are read again only where the K group changes.
template <typename T, int BITS>
__device__ __forceinline__ void dense_rows(const DenseArgs<T>& A, const uint8_t* page, int64_t row0, int t0, int t1, int64_t slot,
                                           int open_grp, const int64_t* s_row) {
  using W = typename Codes8<BITS>::W;
  constexpr int BATCH = DENSE_BATCH;
  const LayoutDev& L = A.L;
  const int cpt = (L.H * L.D) / 8, cph = L.D / 8;
  const int side_bytes = (L.H * L.D * BITS) / 8;
  const int threads = blockDim.x, lanes_t = cpt < threads ? threads / cpt : 1;  // tokens in work at once
  const int t_off = cpt < threads ? (int)threadIdx.x / cpt : 0;
  if (t_off >= lanes_t) return;
  for (int c = (int)threadIdx.x - t_off * cpt; c < cpt; c += threads) {
    const int h = c / cph, d0 = (c - h * cph) * 8;
    const __half* vs_p = reinterpret_cast<const __half*>(page + L.o_vs) + h * L.NG + d0 / L.VG;
    const __half* vm_p = reinterpret_cast<const __half*>(page + L.o_vm) + h * L.NG + d0 / L.VG;
    T* ko_p = A.k_out + row0 * A.o_s0 + h * A.o_s1 + d0;
    T* vo_p = A.v_out + row0 * A.o_s0 + h * A.o_s1 + d0;
    for (int g0 = t0; g0 < t1;) {  // tokens [g0, g1) share a K group
      const int grp = g0 / L.KG, g1 = min(t1, (grp + 1) * L.KG);
      const bool open = grp == open_grp;
      const int ke = (grp * L.H + h) * L.D + d0;
      const uint4 s8 = *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(page + L.o_ks) + ke);
      const uint4 m8 = *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(page + L.o_km) + ke);
      for (int tb = g0 + t_off; tb < g1; tb += BATCH * lanes_t) {
        W kw[BATCH], vw[BATCH];
        __half vs[BATCH], vm[BATCH];
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
          const int t = min(tb + b * lanes_t, g1 - 1);
          const uint8_t* krow = A.pages + s_row[t - t0] + c * BITS;  // 8 channels * BITS / 8 bytes per chunk of 8
          kw[b] = *reinterpret_cast<const W*>(krow);
          vw[b] = *reinterpret_cast<const W*>(krow + side_bytes);
          vs[b] = vs_p[t * L.H * L.NG];
          vm[b] = vm_p[t * L.H * L.NG];
        }
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
          const int t = tb + b * lanes_t;
          if (t >= g1) break;
          uint4 ko, vo;
          uint32_t* ki = reinterpret_cast<uint32_t*>(&ko);
          uint32_t* vi = reinterpret_cast<uint32_t*>(&vo);
          float2 q[4];
          if (open) {
            const int64_t o = slot * A.R.s_slot + (int64_t)(t - grp * L.KG) * A.R.s_pos + h * A.R.s_head + d0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              ki[i] = pack2_rn<T>(ld_dt(A.R.base, A.R.dtype, o + 2 * i), ld_dt(A.R.base, A.R.dtype, o + 2 * i + 1));
            }
          } else {
            unpack8<BITS>(kw[b], q);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 ks = __half22float2(reinterpret_cast<const __half2*>(&s8)[i]);
              const float2 km = __half22float2(reinterpret_cast<const __half2*>(&m8)[i]);
              const float2 k = __fadd2_rn(__fmul2_rn(q[i], ks), km);
              ki[i] = pack2_rn<T>(k.x, k.y);
            }
          }
          unpack8<BITS>(vw[b], q);
          const float fs = __half2float(vs[b]), fm = __half2float(vm[b]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 v = __fadd2_rn(__fmul2_rn(q[i], make_float2(fs, fs)), make_float2(fm, fm));
            vi[i] = pack2_rn<T>(v.x, v.y);
          }
          *reinterpret_cast<uint4*>(ko_p + t * A.o_s0) = ko;
          *reinterpret_cast<uint4*>(vo_p + t * A.o_s0) = vo;
        }
      }
      g0 = g1;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) dequant_dense_vec_kernel(const DenseArgs<T> A) {
  __shared__ int64_t s_row[DENSE_TOK];
  const LayoutDev& L = A.L;
  const int item = blockIdx.x / A.slices, t0 = (blockIdx.x - item * A.slices) * DENSE_TOK;
  const int4 w = reinterpret_cast<const int4*>(A.work)[item];
  const int req = w.x, bi = w.y, row0 = w.z, ctx = w.w;  // block of the context, dense row of its first token
  const int t1 = min(min(L.BS, ctx - bi * L.BS), t0 + DENSE_TOK);
  if (t0 >= t1) return;
  const int64_t blk = A.bt[(int64_t)req * A.bt_s0 + bi];
  const uint8_t* page = A.pages + blk * L.PS;
  int bits = page[0];
  if (bits == 0) bits = 2;  // an unopened block reads as INT2, like the attention kernels
  const int64_t slot = A.R.block_res[blk];
  const int open_grp = slot >= 0 ? (int)A.R.res_group[slot] : -1;
  if (t0 + (int)threadIdx.x < t1) s_row[threadIdx.x] = row_offset(A.pages, L, blk, t0 + threadIdx.x, bits);
  __syncthreads();
  if (bits == 4) dense_rows<T, 4>(A, page, row0, t0, t1, slot, open_grp, s_row);
  else if (bits == 8) dense_rows<T, 8>(A, page, row0, t0, t1, slot, open_grp, s_row);
  else dense_rows<T, 2>(A, page, row0, t0, t1, slot, open_grp, s_row);
}

// Demotion, phase 2: requantize a block's dequantized contents (scratch: K then V, float
// [n, BS, H, D]) to INT2 into chunk 0 of its own page (tiered_cache.py:322-340).
__global__ void __launch_bounds__(256)
demote_requant_kernel(LayoutDev L, uint8_t* __restrict__ pages, const int64_t* __restrict__ victims, int64_t n,
                      const float* __restrict__ scratch) {
  const int64_t b = victims[blockIdx.x];
  const float* ksrc = scratch + (int64_t)blockIdx.x * L.BS * L.H * L.D;
  const float* vsrc = scratch + (n + blockIdx.x) * (int64_t)L.BS * L.H * L.D;
  uint8_t* page = pages + b * L.PS;
  const float levels = 3.f;
  const int bits = 2;
  const int side_bytes = (L.H * L.D * bits) / 8, head_bytes = (L.D * bits) / 8;
  const int64_t row_bytes = 2 * side_bytes;
  uint8_t* data = page + L.o_data;  // INT2: every token row lives in chunk 0 of the own page
  if (threadIdx.x == 0) page[0] = 2;
  // K: per channel over each group of KG tokens
  const int cph = (L.H * L.D) / 8;
  for (int idx = threadIdx.x; idx < L.KGPB * cph; idx += blockDim.x) {
    const int grp = idx / cph, c = idx % cph;
    const int h = (c * 8) / L.D, d0 = (c * 8) % L.D;
    float mn[8], mx[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { mn[k] = INFINITY; mx[k] = -INFINITY; }
    for (int p = 0; p < L.KG; ++p) {
      const float* x = ksrc + ((int64_t)(grp * L.KG + p) * L.H + h) * L.D + d0;
#pragma unroll
      for (int k = 0; k < 8; ++k) { mn[k] = fminf(mn[k], x[k]); mx[k] = fmaxf(mx[k], x[k]); }
    }
    __align__(16) __half s16[8], m16[8];
    float sc[8], m[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      group_stats(mn[k], mx[k], levels, s16[k], m16[k]);
      sc[k] = __half2float(s16[k]); m[k] = __half2float(m16[k]);
    }
    const int64_t e = ((int64_t)grp * L.H + h) * L.D + d0;
    *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(page + L.o_ks) + e) = *reinterpret_cast<uint4*>(s16);
    *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(page + L.o_km) + e) = *reinterpret_cast<uint4*>(m16);
    for (int p = 0; p < L.KG; ++p) {
      const int t = grp * L.KG + p;
      const float* x = ksrc + ((int64_t)t * L.H + h) * L.D + d0;
      uint32_t q[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = quant_code(x[k], m[k], sc[k], levels);
      store_packed8(data + t * row_bytes + h * head_bytes + (d0 * bits) / 8, pack8(q, bits), bits);
    }
  }
  // V: per token, groups of VG channels
  for (int idx = threadIdx.x; idx < L.BS * L.H * L.NG; idx += blockDim.x) {
    const int t = idx / (L.H * L.NG), r = idx % (L.H * L.NG);
    const int h = r / L.NG, g = r % L.NG;
    const float* x = vsrc + ((int64_t)t * L.H + h) * L.D + g * L.VG;
    float mn = INFINITY, mx = -INFINITY;
    for (int c = 0; c < L.VG; ++c) { mn = fminf(mn, x[c]); mx = fmaxf(mx, x[c]); }
    __half s16, m16;
    group_stats(mn, mx, levels, s16, m16);
    const float sc = __half2float(s16), m = __half2float(m16);
    const int64_t e = ((int64_t)t * L.H + h) * L.NG + g;
    reinterpret_cast<__half*>(page + L.o_vs)[e] = s16;
    reinterpret_cast<__half*>(page + L.o_vm)[e] = m16;
    uint8_t* dst = data + t * row_bytes + side_bytes + h * head_bytes + (g * L.VG * bits) / 8;
    for (int c = 0; c < L.VG; c += 8) {
      uint32_t q[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = quant_code(x[c + k], m, sc, levels);
      store_packed8(dst + (c * bits) / 8, pack8(q, bits), bits);
    }
  }
}

// Demotion in one launch, for blocks whose codes fit a CTA's shared memory: one CTA per victim copies the block's token
// rows (chunk 0, which the INT2 rows go to, among them) to shared memory, then every thread dequantizes and
// requantizes the groups it owns, reading a group's old statistics before it stores the new ones.  The same
// arithmetic as the three launches above (index list, gather to fp32 in global memory, requantize), which took 60 us for
// about 95 victims of 16 tokens x 8 heads x 128 at INT8; now 19 us, the two passes of one thread over its group's tokens.
struct DemoteArgs {
  LayoutDev L;
  ResidualDev R;
  uint8_t* pages;
  const int64_t* victims;
};
__device__ __forceinline__ void smem_codes8(const uint8_t* p, int bits, float (&q)[8]) {
  uint64_t w;
  if (bits == 8) w = *reinterpret_cast<const uint64_t*>(p);
  else if (bits == 4) w = *reinterpret_cast<const uint32_t*>(p);
  else w = *reinterpret_cast<const uint16_t*>(p);
  const uint32_t mask = (1u << bits) - 1u;
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = __uint_as_float(0x4B000000u | ((uint32_t)(w >> (i * bits)) & mask)) - 8388608.f;
}
__device__ __forceinline__ uint32_t code2(float x, float m, float sc, float rsc) {
  return quant_u(x, m, sc, rsc, 3.f) - QMAGIC_BITS;
}
__global__ void __launch_bounds__(256) demote_block_kernel(const DemoteArgs A) {
  extern __shared__ __align__(16) uint8_t rows[];  // the block's token rows [BS][K codes | V codes] at its old tier
  const LayoutDev& L = A.L;
  const int64_t b = A.victims[blockIdx.x];
  uint8_t* page = A.pages + b * L.PS;
  const int old = page[0], bits = old == 0 ? 2 : old;
  const int row_bytes = (2 * L.H * L.D * bits) / 8, side = row_bytes / 2;
  {
    const int per = row_bytes / 16;
    const uint4 hd = *reinterpret_cast<const uint4*>(page);
    const int tpc = (2 * L.BS) / bits;
    for (int i = threadIdx.x; i < L.BS * per; i += blockDim.x) {
      const int t = i / per, c = i - t * per, j = t / tpc;
      int64_t pg = b, slot = 0;
      if (j > 0) {
        const int id = j == 1 ? (int)hd.y : (j == 2 ? (int)hd.z : (int)hd.w);
        pg = id / L.KC;
        slot = id - pg * L.KC;
      }
      const uint4* src = reinterpret_cast<const uint4*>(A.pages + pg * L.PS + L.o_data + slot * L.CB + (int64_t)(t - j * tpc) * row_bytes);
      reinterpret_cast<uint4*>(rows + t * row_bytes)[c] = src[c];
    }
  }
  const int64_t rslot = A.R.block_res[b];
  const int open_grp = rslot >= 0 ? (int)A.R.res_group[rslot] : -1;
  __syncthreads();  // every row is here (and the header has been read): from now on the page may change
  if (threadIdx.x == 0) page[0] = 2;
  const int side2 = (L.H * L.D * 2) / 8;
  uint8_t* data = page + L.o_data;  // INT2: every token row lies in chunk 0 of the own page
  const int cph = (L.H * L.D) / 8;
  // K: 8 channels of one group of KG tokens per thread
  for (int i = threadIdx.x; i < L.KGPB * cph; i += blockDim.x) {
    const int grp = i / cph, c = i - grp * cph, h = (c * 8) / L.D, d0 = (c * 8) % L.D;
    const int e = (grp * L.H + h) * L.D + d0;
    __half* ks = reinterpret_cast<__half*>(page + L.o_ks) + e;
    __half* km = reinterpret_cast<__half*>(page + L.o_km) + e;
    float so[8], mo[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { so[k] = __half2float(ks[k]); mo[k] = __half2float(km[k]); }
    auto load = [&](int p, float (&x)[8]) {
      const int t = grp * L.KG + p;
      if (old == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = 0.f;
      } else if (grp == open_grp) {
        const int64_t o = rslot * A.R.s_slot + (int64_t)p * A.R.s_pos + h * A.R.s_head + d0;
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = ld_dt(A.R.base, A.R.dtype, o + k);
      } else {
        smem_codes8(rows + t * row_bytes + c * bits, bits, x);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = __fadd_rn(__fmul_rn(x[k], so[k]), mo[k]);
      }
    };
    float mn[8], mx[8], x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { mn[k] = INFINITY; mx[k] = -INFINITY; }
    for (int p = 0; p < L.KG; ++p) {
      load(p, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) { mn[k] = fminf(mn[k], x[k]); mx[k] = fmaxf(mx[k], x[k]); }
    }
    __align__(16) __half s16[8], m16[8];
    float sc[8], m[8], rsc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      group_stats(mn[k], mx[k], 3.f, s16[k], m16[k]);
      sc[k] = __half2float(s16[k]); m[k] = __half2float(m16[k]); rsc[k] = __frcp_rn(sc[k]);
    }
    *reinterpret_cast<uint4*>(ks) = *reinterpret_cast<uint4*>(s16);
    *reinterpret_cast<uint4*>(km) = *reinterpret_cast<uint4*>(m16);
    for (int p = 0; p < L.KG; ++p) {
      load(p, x);
      uint32_t w = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) w |= code2(x[k], m[k], sc[k], rsc[k]) << (2 * k);
      *reinterpret_cast<uint16_t*>(data + (grp * L.KG + p) * 2 * side2 + c * 2) = (uint16_t)w;
    }
  }
  // V: one group of VG channels of one token per thread
  for (int i = threadIdx.x; i < L.BS * L.H * L.NG; i += blockDim.x) {
    const int t = i / (L.H * L.NG), hg = i - t * (L.H * L.NG);
    __half* vs = reinterpret_cast<__half*>(page + L.o_vs) + i;
    __half* vm = reinterpret_cast<__half*>(page + L.o_vm) + i;
    const float so = __half2float(*vs), mo = __half2float(*vm);
    const int c0 = hg * (L.VG / 8);  // first 8-channel piece
    float mn = INFINITY, mx = -INFINITY, x[8];
    auto load = [&](int c) {
      smem_codes8(rows + t * row_bytes + side + (c0 + c) * bits, bits, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = old == 0 ? 0.f : __fadd_rn(__fmul_rn(x[k], so), mo);
    };
    for (int c = 0; c < L.VG / 8; ++c) {
      load(c);
#pragma unroll
      for (int k = 0; k < 8; ++k) { mn = fminf(mn, x[k]); mx = fmaxf(mx, x[k]); }
    }
    __half s16, m16;
    group_stats(mn, mx, 3.f, s16, m16);
    const float sc = __half2float(s16), m = __half2float(m16), rsc = __frcp_rn(sc);
    *vs = s16;
    *vm = m16;
    for (int c = 0; c < L.VG / 8; ++c) {
      load(c);
      uint32_t w = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) w |= code2(x[k], m, sc, rsc) << (2 * k);
      *reinterpret_cast<uint16_t*>(data + t * 2 * side2 + side2 + (c0 + c) * 2) = (uint16_t)w;
    }
  }
}
constexpr int DEMOTE_MAX_SMEM = 200 * 1024;

__global__ void demote_index_kernel(const int64_t* victims, int64_t n, int BS, int64_t* blk, int64_t* off) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * BS) return;
  blk[i] = victims[i / BS];
  off[i] = i % BS;
}

}  // namespace echokv

using namespace echokv;

extern "C" {

int echokv_gather(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                  const int64_t* blk, const int64_t* off, int64_t n, float* k_out, float* v_out, void* stream) {
  if (n <= 0) return ECHOKV_OK;
  LayoutDev L;
  ResidualDev R;
  int rc = make_layout(layout, pages, &L);
  if (rc) return rc;
  rc = make_residual(residual, &R);
  if (rc) return rc;
  if (!blk || !off || !k_out || !v_out) return set_error(ECHOKV_E_ARGUMENT, "gather: null pointer");
  const int64_t total = n * (L.H * L.D / 8);
  gather_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      L, R, (const uint8_t*)pages->base, blk, off, n, k_out, v_out);
  return check_launch("gather");
}

int echokv_dequant_dense(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                         const int32_t* work, int64_t n_work, const int32_t* block_table, int64_t bt_s0, void* k_out,
                         void* v_out, int64_t out_s0, int64_t out_s1, int32_t out_dtype, void* stream) {
  if (n_work <= 0) return ECHOKV_OK;
  LayoutDev L;
  ResidualDev R;
  int rc = make_layout(layout, pages, &L);
  if (rc) return rc;
  rc = make_residual(residual, &R);
  if (rc) return rc;
  if (!work || !block_table || !k_out || !v_out) return set_error(ECHOKV_E_ARGUMENT, "dequant_dense: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
#define LAUNCH(T)                                                                                              \
  dequant_dense_kernel<T><<<(unsigned)n_work, 256, 0, st>>>(L, R, (const uint8_t*)pages->base, work, block_table, \
                                                           bt_s0, (T*)k_out, (T*)v_out, out_s0, out_s1)
  // 16-byte loads and stores need the stat arrays, the rows of the outputs and 8-channel chunks aligned
  const int slices = (L.BS + DENSE_TOK - 1) / DENSE_TOK;
  const int64_t ctas = n_work * slices;
  const bool vec = out_dtype != ECHOKV_DT_F32 && ctas < (1ll << 31) && L.D % 8 == 0 && L.VG % 8 == 0 &&
                   ((L.o_ks | L.o_km | L.PS | L.o_data | L.CB) % 16) == 0 && (out_s0 % 8) == 0 && (out_s1 % 8) == 0 &&
                   ((reinterpret_cast<uintptr_t>(k_out) | reinterpret_cast<uintptr_t>(v_out) |
                     reinterpret_cast<uintptr_t>(pages->base) | reinterpret_cast<uintptr_t>(work)) % 16) == 0;
  // Threads for DENSE_TOK / DENSE_BATCH tokens at once where the rows are so short that 256 threads would have a token each
  // (and three repeated loads) and there are more CTAs than run at once (two per SM): one KV head of 128 channels, 16 x 500
  // tokens 6.5 -> 4.2 us, 8 x 8,704 tokens 31 -> 13 us.  With fewer CTAs a token per thread is the shorter chain (700 tokens 3.6 us
  // against 4.2).
  const int chunks = L.H * L.D / 8 * (DENSE_TOK / DENSE_BATCH);
  const unsigned threads = chunks < 256 && ctas > 2 * 148 ? (unsigned)(chunks + 31) / 32 * 32 : 256u;
#define LAUNCH_VEC(T)                                                                                         \
  {                                                                                                           \
    DenseArgs<T> A = {L, R, (const uint8_t*)pages->base, work, block_table, bt_s0, (T*)k_out, (T*)v_out, out_s0, \
                      out_s1, slices};                                                                                \
    dequant_dense_vec_kernel<T><<<(unsigned)ctas, threads, 0, st>>>(A);                                       \
  }
  if (vec) {
    if (out_dtype == ECHOKV_DT_F16) LAUNCH_VEC(__half) else LAUNCH_VEC(__nv_bfloat16)
    return check_launch("dequant_dense");
  }
#undef LAUNCH_VEC
  switch (out_dtype) {
    case ECHOKV_DT_F32: LAUNCH(float); break;
    case ECHOKV_DT_F16: LAUNCH(__half); break;
    case ECHOKV_DT_BF16: LAUNCH(__nv_bfloat16); break;
    default: return set_error(ECHOKV_E_ARGUMENT, "dequant_dense: bad dtype %d", out_dtype);
  }
#undef LAUNCH
  return check_launch("dequant_dense");
}

int64_t echokv_demote_scratch_bytes(const echokv_layout* layout, int64_t n) {
  if (!layout || n <= 0) return 0;
  const int64_t tok = n * layout->block_size;
  // dequantized K and V (float) + the (blk, off) index of every token
  return tok * layout->num_kv_heads * layout->head_size * 2 * (int64_t)sizeof(float) + tok * 2 * (int64_t)sizeof(int64_t);
}

int echokv_demote_blocks(const echokv_layout* layout, const echokv_pages* pages, const echokv_residual* residual,
                         const int64_t* victims, int64_t n, void* scratch, int64_t scratch_bytes, void* stream) {
  if (n <= 0) return ECHOKV_OK;
  LayoutDev L;
  ResidualDev R;
  int rc = make_layout(layout, pages, &L);
  if (rc) return rc;
  rc = make_residual(residual, &R);
  if (rc) return rc;
  if (!victims || !scratch) return set_error(ECHOKV_E_ARGUMENT, "demote_blocks: null pointer");
  if (scratch_bytes < echokv_demote_scratch_bytes(layout, n) || (reinterpret_cast<uintptr_t>(scratch) & 15))
    return set_error(ECHOKV_E_ARGUMENT, "demote_blocks: scratch too small or misaligned");
  cudaStream_t st = (cudaStream_t)stream;
  // one launch when a block's rows at INT8 fit a CTA's shared memory and every row is made of 16-byte pieces at any tier
  const int64_t smem = 2 * (int64_t)L.BS * L.H * L.D;
  if (smem <= DEMOTE_MAX_SMEM && (L.H * L.D) % 32 == 0 && L.NG * L.VG == L.D &&
      ((L.PS | L.o_data | L.CB | L.o_ks | L.o_km) % 16) == 0) {
    // per call: the attribute belongs to the current device
    if (smem > 48 * 1024 && cudaFuncSetAttribute(demote_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return check_launch("demote_blocks");
    const DemoteArgs A = {L, R, (uint8_t*)pages->base, victims};
    demote_block_kernel<<<(unsigned)n, 256, (size_t)smem, st>>>(A);
    return check_launch("demote_blocks");
  }
  const int64_t tok = n * L.BS;
  float* kf = (float*)scratch;
  float* vf = kf + tok * L.H * L.D;
  int64_t* bi = (int64_t*)(vf + tok * L.H * L.D);
  int64_t* oi = bi + tok;
  demote_index_kernel<<<(unsigned)((tok + 255) / 256), 256, 0, st>>>(victims, n, L.BS, bi, oi);
  const int64_t total = tok * (L.H * L.D / 8);
  gather_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(L, R, (const uint8_t*)pages->base, bi, oi, tok, kf, vf);
  demote_requant_kernel<<<(unsigned)n, 256, 0, st>>>(L, (uint8_t*)pages->base, victims, n, kf);
  return check_launch("demote_blocks");
}

}  // extern "C"
