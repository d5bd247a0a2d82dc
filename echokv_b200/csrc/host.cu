// Host-side pieces of the C ABI: error text, layout arithmetic, argument checks.
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <exception>
#include <numeric>
#include <vector>

#include "common.cuh"

namespace echokv {

static thread_local char g_err[512] = "";

int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

// TieredLayout.__post_init__ / offsets / per_token_bytes (echokv_vllm/tiered_cache.py:85-147).
int describe(const echokv_layout* l, echokv_layout_info* out) {
  if (!l || !out) return set_error(ECHOKV_E_ARGUMENT, "layout/out is null");
  const int64_t h = l->num_kv_heads, d = l->head_size, bs = l->block_size, kg = l->k_group, vg = l->v_group;
  const int mb = l->mem_bits;
  if (h <= 0 || d <= 0 || bs <= 0 || kg <= 0 || vg <= 0)
    return set_error(ECHOKV_E_LAYOUT, "layout fields must be positive");
  if (!(mb == 2 || mb == 4 || mb == 6 || mb == 8))
    return set_error(ECHOKV_E_LAYOUT, "mem_bits must be one of 2/4/6/8, got %d", mb);
  if (bs % 16 != 0) return set_error(ECHOKV_E_LAYOUT, "block_size must be a multiple of 16, got %d", (int)bs);
  if (bs % kg != 0 || bs / kg > 8)
    return set_error(ECHOKV_E_LAYOUT, "block_size %d must be 1-8 multiples of k_group %d", (int)bs, (int)kg);
  if (d % vg != 0 || d % 4 != 0)
    return set_error(ECHOKV_E_LAYOUT, "head_size %d must be divisible by v_group %d and by 4", (int)d, (int)vg);
  const int64_t ng = d / vg, kgpb = bs / kg;
  out->o_v_scale = bs;
  out->o_v_min = out->o_v_scale + bs * h * ng * 2;
  out->o_k_scale = out->o_v_min + bs * h * ng * 2;
  out->o_k_min = out->o_k_scale + kgpb * h * d * 2;
  out->o_data = out->o_k_min + kgpb * h * d * 2;
  out->chunk_bytes = bs * h * d / 2;
  out->chunks_per_page = mb / 2;
  out->page_bytes = out->o_data + out->chunks_per_page * out->chunk_bytes;
  const int64_t raw = 1 + 4 * h * ng + 4 * h * d / kg + (mb / 2) * h * d / 2;
  out->per_token_bytes = (raw + 3) / 4 * 4;
  out->k_groups_per_block = (int32_t)kgpb;
  out->v_groups = (int32_t)ng;
  out->reserved = 0;
  return ECHOKV_OK;
}

int make_layout(const echokv_layout* l, const echokv_pages* p, LayoutDev* L) {
  echokv_layout_info info;
  int rc = describe(l, &info);
  if (rc) return rc;
  if (!p || !p->base) return set_error(ECHOKV_E_ARGUMENT, "pages is null");
  if (p->page_stride_bytes < info.page_bytes)
    return set_error(ECHOKV_E_ARGUMENT, "page stride %lld is smaller than the layout's page (%lld bytes)",
                     (long long)p->page_stride_bytes, (long long)info.page_bytes);
  if (p->page_stride_bytes % 16 != 0 || (reinterpret_cast<uintptr_t>(p->base) % 16) != 0)
    return set_error(ECHOKV_E_ARGUMENT, "pages must be 16-byte aligned with a 16-byte aligned row stride");
  if (l->head_size % 16 != 0 || l->v_group % 8 != 0)
    return set_error(ECHOKV_E_UNSUPPORTED, "kernels need head_size %% 16 == 0 and v_group %% 8 == 0 (got %d, %d)",
                     l->head_size, l->v_group);
  L->H = l->num_kv_heads; L->D = l->head_size; L->BS = l->block_size; L->KG = l->k_group; L->VG = l->v_group;
  L->KC = info.chunks_per_page; L->NG = info.v_groups; L->KGPB = info.k_groups_per_block;
  L->o_vs = info.o_v_scale; L->o_vm = info.o_v_min; L->o_ks = info.o_k_scale; L->o_km = info.o_k_min;
  L->o_data = info.o_data; L->CB = info.chunk_bytes; L->PS = p->page_stride_bytes; L->NB = p->num_blocks;
  return ECHOKV_OK;
}

int make_residual(const echokv_residual* r, ResidualDev* R) {
  if (!r || !r->base || !r->block_res || !r->res_group)
    return set_error(ECHOKV_E_ARGUMENT, "residual buffer / block_res / res_group is null");
  if (r->dtype < ECHOKV_DT_F32 || r->dtype > ECHOKV_DT_BF16)
    return set_error(ECHOKV_E_ARGUMENT, "bad residual dtype %d", r->dtype);
  R->base = r->base; R->dtype = r->dtype;
  R->s_slot = r->s_slot; R->s_pos = r->s_pos; R->s_head = r->s_head;
  R->block_res = r->block_res; R->res_group = r->res_group;
  return ECHOKV_OK;
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(ECHOKV_E_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return ECHOKV_OK;
}

}  // namespace echokv

extern "C" {

int echokv_abi_version(void) { return ECHOKV_ABI_VERSION; }

const char* echokv_last_error(void) { return echokv::g_err; }

int echokv_layout_describe(const echokv_layout* layout, echokv_layout_info* out) {
  return echokv::describe(layout, out);
}

// A group ends where a token, taken alone, would be worked off in another way than the one before it: where another tile of 16 tokens
// is full (full tiles go in pairs, and then share a reference of the exponentials), and where the split size may change.  That is behind
// a multiple of 32 blocks (the calls have 32 splits where the size follows the context at all), and a block is 16 tokens or a
// multiple.  So a token's bits follow from its own context, however its chunk was cut.  A chunk of 33 tokens has one group of up to 2
// tokens more at most, as it has of 4 or 8 (17, 9 and 5 without the rule); 16 such chunks behind 740 - 1,472: 1.099 ms a step
// instead of 1.064.
int64_t echokv_chunk_groups(const int64_t* chunks, int64_t num_chunks, int64_t num_tokens, const int64_t* widths, int32_t num_widths,
                            int64_t* rows, int64_t* split_lens, int64_t* groups, int64_t* num_groups) {
  const int64_t n = num_tokens;
  std::vector<int64_t> order, place;  // chunks from the longest context to the shortest; where a chunk's tokens begin in the list
  try {
    order.resize(num_chunks);
    place.resize(num_chunks + 1);
  } catch (const std::exception&) {  // no memory, or a negative count
    return echokv::set_error(ECHOKV_E_ARGUMENT, "chunk_groups: no memory for %lld chunks", (long long)num_chunks);
  }
  std::iota(order.begin(), order.end(), 0);
  std::sort(order.begin(), order.end(), [&](int64_t a, int64_t b) {
    return chunks[4 * a + 2] != chunks[4 * b + 2] ? chunks[4 * a + 2] > chunks[4 * b + 2] : a < b;
  });
  for (int64_t c = 0; c < num_chunks; ++c) {
    if (chunks[4 * c + 1] < 0) return echokv::set_error(ECHOKV_E_ARGUMENT, "chunk_groups: a chunk of %lld tokens", (long long)chunks[4 * c + 1]);
    place[c + 1] = place[c] + chunks[4 * c + 1];
  }
  if (place[num_chunks] != n)
    return echokv::set_error(ECHOKV_E_ARGUMENT, "chunk_groups: %lld tokens, not %lld", (long long)place[num_chunks], (long long)n);
  for (int64_t c = 0, at = 0; c < num_chunks; ++c)
    for (int64_t i = 0; i < chunks[4 * c + 1]; ++i, ++at) {
      rows[at] = chunks[4 * c] + i;
      rows[n + at] = chunks[4 * c + 3];
      rows[2 * n + at] = chunks[4 * c + 2] - chunks[4 * c + 1] + 1 + i;
    }
  int64_t total = 0;
  for (int32_t k = 0; k < num_widths; ++k) {
    const int64_t before = total;
    for (const int64_t c : order)
      for (int64_t first = place[c], end = place[c + 1]; first < end;) {
        int64_t next = first + 1;
        const int64_t* len = rows + 2 * n;
        while (next < end && next - first < widths[k] && len[next] % 16 != 0 && len[next] % 512 != 1) ++next;
        int64_t* g = groups + 5 * total++;
        g[0] = rows[first]; g[1] = rows[n + first]; g[2] = rows[2 * n + next - 1]; g[3] = next - first; g[4] = first;
        for (int64_t i = first; i < next; ++i) split_lens[k * n + i] = g[2];
        first = next;
      }
    num_groups[k] = total - before;
  }
  return total;
}

}  // extern "C"
