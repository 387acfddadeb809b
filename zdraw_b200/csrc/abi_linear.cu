// extern "C" entry points next to the attention path: the projection GEMM (plain, with the q/k
// prologue as epilogue, three products in one launch) and the wide-head attention built from it.
// See include/zdraw_cuda.h for the contract and the reference entry points each one replaces.
#include <cmath>

#include "abi_internal.cuh"
#include "linear.cuh"
#include "prologue.cuh"
#include "wide_attention.cuh"

namespace {

using namespace zdraw::abi;

// One product of a projection launch as the entry points describe it.
struct PartSpec {
  const void* w;
  void* c;
  uint32_t epilogue;  // zdraw::kEpilogue*: 0 plain, 1 qk; 2 row max and 3 exp are internal (wide attention)
  const float *w_txt, *w_img;
  unsigned int* row_key = nullptr;   // row max / exp: ordered keys of the row maxima
  float* row_sum = nullptr;          // exp: partial row sums; plain: the rows are divided by their sum
  int n_partial = 0;                 // partial sums per row
  float exp_scale = 0.0f;
  float* shift = nullptr;            // exp: see LinearPart
  unsigned int *row_missed = nullptr, *any_missed = nullptr;
  uint32_t n_valid = 0;              // row max / exp: real columns (0 = all n); W then has n_valid rows
};

// What the wide attention's launches say beyond the parameters of the entry points.
struct WideSpec {
  uint32_t w_k_valid = 0;         // columns of W that exist when fewer than k (A has all k)
  const unsigned int* norms = nullptr;  // row max: see LinearArgs; all of W is n_valid_all rows of k
  uint32_t n_valid_all = 0;
  unsigned int *all_rows = nullptr, *norms_done = nullptr;
  float* zero = nullptr;  // zero_n floats set to zero beside the product
  size_t zero_n = 0;
  bool rows_first = false;        // tile order: across the column blocks of a row block first
  bool early_dependents = false;  // (projections: true)
  int k_splits = 1;               // 2: C holds zeros and each tile's K is walked by two pairs (linear.cuh)
};

WideSpec projection() {
  WideSpec s;
  s.early_dependents = true;
  return s;
}

// Shared body of zdraw_cuda_linear and zdraw_cuda_qkv_projection: validates, builds the tensor
// maps and launches one kernel that computes every part from the same A.
int run_linear(Ctx* cx, void* stream, const void* a, int n_parts, const PartSpec* parts, const float* rope_cos,
               const float* rope_sin, const zdraw_cuda_linear_params* p, const WideSpec& wide) {
  if (!p) return fail(cx, ZDRAW_CUDA_E_ARG, "params is null");
  if (p->reserved != 0 || p->m == 0 || p->n == 0 || p->k == 0) return fail(cx, ZDRAW_CUDA_E_ARG, "zero size or reserved != 0");
  if (p->c_dtype != ZDRAW_DTYPE_F16 && p->c_dtype != ZDRAW_DTYPE_F32) return fail(cx, ZDRAW_CUDA_E_ARG, "bad c_dtype");
  if (!a || !aligned16(a)) return fail(cx, ZDRAW_CUDA_E_ARG, "null or misaligned matrix");
  bool any_qk = false;
  for (int i = 0; i < n_parts; ++i) {
    if (parts[i].epilogue > 3) return fail(cx, ZDRAW_CUDA_E_ARG, "bad epilogue");
    if (!parts[i].w || !parts[i].c || !aligned16(parts[i].w) || !aligned16(parts[i].c))
      return fail(cx, ZDRAW_CUDA_E_ARG, "null or misaligned matrix");
    any_qk = any_qk || parts[i].epilogue == 1;
  }
  // Shapes and types outside the kernel: declined, nothing enqueued (the reference's fast GEMMs
  // admit 32-aligned dims only, src/metal/mres_util.zig:30-38).
  if (p->a_dtype != ZDRAW_DTYPE_F16 || p->w_dtype != ZDRAW_DTYPE_F16) return fail(cx, ZDRAW_CUDA_DECLINED, "A and W must be f16");
  // (Tiles are 256 columns x 64 of K; what lies beyond n or k is zero-filled on the way in and
  // clipped on the way out, so only the 16-byte granularity of the copy engine remains.)
  if (p->n % 32 != 0 || p->k % 32 != 0) return fail(cx, ZDRAW_CUDA_DECLINED, "n and k must be multiples of 32");
  if (p->m > (1u << 30) || p->n > (1u << 30) || p->k > (1u << 30)) return fail(cx, ZDRAW_CUDA_DECLINED, "shape too large");
  const long long ld_a = p->ld_a ? static_cast<long long>(p->ld_a) : p->k;
  const long long ld_w = p->ld_w ? static_cast<long long>(p->ld_w) : (wide.w_k_valid ? wide.w_k_valid : p->k);
  const long long ld_c = p->ld_c ? static_cast<long long>(p->ld_c) : p->n;
  if (ld_a < p->k || ld_w < static_cast<long long>(wide.w_k_valid ? wide.w_k_valid : p->k) || ld_c < p->n)
    return fail(cx, ZDRAW_CUDA_E_ARG, "row stride smaller than the row");
  if (ld_a % 8 != 0 || ld_w % 8 != 0 || ld_c % 8 != 0)  // TMA strides are multiples of 16 bytes
    return fail(cx, ZDRAW_CUDA_DECLINED, "row strides must be multiples of 8 elements");
  zdraw::LinearArgs la = {};
  la.m = static_cast<int>(p->m);
  la.n = static_cast<int>(p->n);
  la.k = static_cast<int>(p->k);
  la.n_parts = n_parts;
  la.status = cx->d_status;
  la.norms = wide.norms;
  la.norm_scale = parts[0].exp_scale;
  la.n_valid_all = static_cast<int>(wide.n_valid_all);
  la.n_all = (la.n_valid_all + 255) / 256 * 256;
  la.all_rows = wide.all_rows;
  la.norms_done = wide.norms_done;
  la.zero = reinterpret_cast<float4*>(wide.zero);
  la.zero_n4 = static_cast<long long>(wide.zero_n / 4);
  la.rows_first = wide.rows_first ? 1 : 0;
  la.k_splits = wide.k_splits;
  la.early_dependents = wide.early_dependents ? 1 : 0;
  if (any_qk) {
    if (p->tokens == 0 || p->heads == 0 || p->m % p->tokens != 0 || p->n != p->heads * 128u || p->txt_tokens > p->tokens)
      return fail(cx, ZDRAW_CUDA_E_ARG, "qk epilogue needs m = images * tokens and n = heads * 128");
    if (!rope_cos || !rope_sin || !aligned16(rope_cos) || !aligned16(rope_sin) || p->rope_batch_stride % 4 != 0)
      return fail(cx, ZDRAW_CUDA_E_ARG, "qk epilogue needs aligned tables");
    if (!(p->norm_eps >= 0.0f)) return fail(cx, ZDRAW_CUDA_E_ARG, "norm_eps must be >= 0");
    la.tokens = static_cast<int>(p->tokens);
    la.heads = static_cast<int>(p->heads);
    la.txt_tokens = static_cast<int>(p->txt_tokens);
    la.norm_eps = p->norm_eps;
    la.rope_cos = rope_cos;
    la.rope_sin = rope_sin;
    la.rope_batch_stride = static_cast<long long>(p->rope_batch_stride);
  }
  for (int i = 0; i < n_parts; ++i) {
    zdraw::LinearPart& lp = la.part[i];
    lp.epilogue = static_cast<int>(parts[i].epilogue);
    lp.c = parts[i].c;
    if (parts[i].epilogue == 1) {
      if (!parts[i].w_txt || !parts[i].w_img || !aligned16(parts[i].w_txt) || !aligned16(parts[i].w_img))
        return fail(cx, ZDRAW_CUDA_E_ARG, "qk epilogue needs aligned norm weights");
      lp.w_txt = parts[i].w_txt;
      lp.w_img = parts[i].w_img;
    } else {
      lp.c_f32 = p->c_dtype == ZDRAW_DTYPE_F32;
      lp.ld_c = ld_c;
      lp.row_key = parts[i].row_key;
      lp.row_sum = parts[i].row_sum;
      lp.n_partial = parts[i].n_partial;
      lp.exp_scale = parts[i].exp_scale;
      lp.shift = parts[i].shift;
      lp.row_missed = parts[i].row_missed;
      lp.any_missed = parts[i].any_missed;
      lp.n_valid = static_cast<int>(parts[i].n_valid ? parts[i].n_valid : p->n);
    }
  }
  ZD_CUDA(cx, cudaSetDevice(cx->device));
  int pairs = 0;
  ZD_CUDA(cx, zdraw::linear_pairs(cx->sm_count, &pairs));
  // Row-major matrices [rows][ld] as tiled tensor maps: boxes of 128 bytes (64 halves) x 128 rows.
  zdraw::LinearMaps maps;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  // Rows and columns beyond what a matrix has are filled with zeros by the copy engine.
  auto encode = [&](CUtensorMap* tm, const void* base_ptr, uint64_t rows, long long ld, uint64_t cols) {
    const cuuint64_t dims[4] = {cols, rows, 1, 1};
    const cuuint64_t strides[3] = {2u * static_cast<cuuint64_t>(ld), 2u * static_cast<cuuint64_t>(ld) * rows,
                                   2u * static_cast<cuuint64_t>(ld) * rows};
    const cuuint32_t box[4] = {64u, 128u, 1, 1};
    return cx->encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base_ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  if (encode(&maps.a, a, p->m, ld_a, p->k) != CUDA_SUCCESS)
    return fail(cx, ZDRAW_CUDA_E_CUDA, "cuTensorMapEncodeTiled failed");
  for (int i = 0; i < zdraw::kMaxLinearParts; ++i) {
    maps.w[i] = maps.w[0];  // unused entries
    if (i >= n_parts) continue;
    const PartSpec& ps = parts[i];
    if (encode(&maps.w[i], ps.w, ps.n_valid ? ps.n_valid : p->n, ld_w, wide.w_k_valid ? wide.w_k_valid : p->k) !=
        CUDA_SUCCESS)
      return fail(cx, ZDRAW_CUDA_E_CUDA, "cuTensorMapEncodeTiled failed");
  }
  if (wide.norms && encode(&maps.w[1], parts[0].w, wide.n_valid_all, p->k, p->k) != CUDA_SUCCESS)
    return fail(cx, ZDRAW_CUDA_E_CUDA, "cuTensorMapEncodeTiled failed");
  // Plain parts: C for the epilogue's tile stores (32 columns x 32 rows, swizzle of the row size).
  for (int i = 0; i < zdraw::kMaxLinearParts; ++i) {
    maps.c[i] = maps.a;  // any valid map where none is used
    if (i >= n_parts || (parts[i].epilogue != 0 && parts[i].epilogue != 3)) continue;
    const bool f32 = p->c_dtype == ZDRAW_DTYPE_F32;
    const cuuint64_t dims[2] = {p->n, p->m};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_c) * (f32 ? 4u : 2u)};
    const cuuint32_t box[2] = {f32 ? 32u : 64u, 32u};  // 128-byte rows either way: 32 f32 or 64 f16 columns
    const cuuint32_t es[2] = {1, 1};
    if (cx->encode(&maps.c[i], f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, parts[i].c, dims,
                   strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return fail(cx, ZDRAW_CUDA_E_CUDA, "cuTensorMapEncodeTiled failed for C");
  }
  ZD_CUDA(cx, zdraw::launch_linear(static_cast<cudaStream_t>(stream), maps, la, pairs));
  return ZDRAW_CUDA_OK;
}

}  // namespace

extern "C" {

int zdraw_cuda_linear(void* ctx, void* stream, const void* a, const void* w, void* c, const float* norm_w_txt,
                      const float* norm_w_img, const float* rope_cos, const float* rope_sin,
                      const zdraw_cuda_linear_params* p) {
  Ctx* cx = as_ctx(ctx);
  if (!cx) return ZDRAW_CUDA_E_ARG;
  if (!p) return fail(cx, ZDRAW_CUDA_E_ARG, "params is null");
  if (p->epilogue > 1) return fail(cx, ZDRAW_CUDA_E_ARG, "bad epilogue");
  if (p->epilogue == 1 && p->c_dtype != ZDRAW_DTYPE_F16) return fail(cx, ZDRAW_CUDA_E_ARG, "the qk epilogue writes f16");
  const PartSpec part = {w, c, p->epilogue, norm_w_txt, norm_w_img};
  return run_linear(cx, stream, a, 1, &part, rope_cos, rope_sin, p, projection());
}

int zdraw_cuda_wide_attention(void* ctx, void* stream, const float* q, const float* k, const float* v, float* o,
                              size_t tokens, size_t head_dim) {
  Ctx* cx = as_ctx(ctx);
  if (!cx) return ZDRAW_CUDA_E_ARG;
  if (!q || !k || !v || !o || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o))
    return fail(cx, ZDRAW_CUDA_E_ARG, "null or misaligned tensor");
  if (tokens == 0 || head_dim == 0) return fail(cx, ZDRAW_CUDA_E_ARG, "zero tokens or head_dim");
  // Shapes outside the kernels are declined: the reference's own admission, tokens % 32 and
  // head_dim % 32 (src/metal/mvattn_owned.zig:271-272); the token bound keeps the tokens^2 half
  // scratch below 9 GB.
  if (tokens % 32 != 0 || head_dim % 32 != 0 || tokens > 65536 || head_dim > 4096)
    return fail(cx, ZDRAW_CUDA_DECLINED, "tokens (<= 65536) and head_dim (<= 4096) must be multiples of 32");
  ZD_CUDA(cx, cudaSetDevice(cx->device));
  const size_t n = tokens * head_dim;
  // The score matrix is tiled in blocks of up to 256 keys: its columns are padded to that (the padding
  // is stored as zeros and skipped by the row maximum).
  const size_t n_pad = (tokens + 255) / 256 * 256;
  const size_t n_partial = n_pad / 128;  // partial row sums: one per 128 columns
  const size_t aux_bytes = 4 * (2 * tokens * n_partial + 2 * tokens);  // partial sums, offsets, row keys, row flags
  int rc;
  if ((rc = ensure(cx, cx->wa_q16, n * 2)) || (rc = ensure(cx, cx->wa_k16, n * 2)) || (rc = ensure(cx, cx->wa_vt16, n * 2)) ||
      (rc = ensure(cx, cx->wa_aux, aux_bytes)) || (rc = ensure(cx, cx->wa_p, tokens * n_pad * 2)))
    return rc;
  float* row_sum = static_cast<float*>(cx->wa_aux.p);
  float* shift = row_sum + tokens * n_partial;
  unsigned int* row_key = reinterpret_cast<unsigned int*>(shift + tokens * n_partial);
  unsigned int* row_missed = row_key + tokens;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  zdraw::WideCast cast = {};
  cast.q = q;
  cast.k = k;
  cast.v = v;
  cast.q16 = cx->wa_q16.p;
  cast.k16 = cx->wa_k16.p;
  cast.vt16 = cx->wa_vt16.p;
  cast.tokens = static_cast<int>(tokens);
  cast.ch = static_cast<int>(head_dim);
  cast.row_key = row_key;
  cast.row_missed = row_missed;
  cast.state = cx->wa_state;
  // O = P V has few tiles (tokens / 256 x head_dim / 256): where a second half-length round of work items
  // fits the chip better, K is split and the halves are added to an O that idle warps of the two launches before have
  // zeroed. By then the operands have been read, so that the result is the same with O in the place of one of them.
  // (Zeroed by the cast launch, with P V in one piece for such an O: 60.3 us at 4096 x 512, 66.9 in place; now 59.)
  int pairs = 0;
  ZD_CUDA(cx, zdraw::linear_pairs(cx->sm_count, &pairs));
  const bool split = zdraw::linear_split_pays(zdraw::linear_tiles(static_cast<int>(tokens), static_cast<int>(head_dim), 1), pairs);
  // kf32_to_h x2, kvt_transpose_h (mvattn_owned.zig:322-330)
  ZD_CUDA(cx, zdraw::launch_wide_cast(st, cast));
  cx->wa_ran = true;
  // The scores S = Q K^T (K is already [n][k]) are never stored. One product keeps only row maxima; a
  // second one turns its accumulator into exp(scale (S - max)) in half and keeps partial row sums:
  // recomputing S (k = head_dim is short) costs less than writing and re-reading tokens^2 f32 scores.
  // Softmax does not change when another number than the maximum is subtracted, as long as nothing
  // overflows, so the maxima come from some 512 keys spread over the image (every stride-th one, through
  // the tensor map's row stride). Where a row's largest score lies 2^16 or more above the sample's (in the
  // exponentials), the exp product stores the 128 columns concerned under an offset of their own and a
  // last pass brings such rows to one scale (wide_rescale_kernel). All of it depends on the data alone. (The
  // reference takes the exact f32 maximum of half products, krow_softmax_h, src/metal/mvattn_owned.zig:95-128.)
  // A call with a row missed in each block of 256 takes 60.2 us at 4096 x 512 and 533 at 16384 (59 and 530 with none;
  // 99 and 1050 when such blocks were multiplied again under exact maxima), with every row missed 64 and 610 to 710.
  // Below 1024 tokens every key is in the sample: its maxima are exact and the last pass is left out.
  // Operands of large norms (scores beyond kMaxSampledScore possible) get the maxima of all keys from the same launch.
  const size_t stride = tokens < 1024 ? 1 : tokens / 512;
  const size_t n_sample = (tokens + stride - 1) / stride;
  zdraw_cuda_linear_params ps = {};
  ps.m = static_cast<uint32_t>(tokens);
  ps.n = static_cast<uint32_t>((n_sample + 255) / 256 * 256);
  ps.k = static_cast<uint32_t>(head_dim);
  ps.ld_w = stride * head_dim;
  ps.ld_c = n_pad;
  ps.a_dtype = ps.w_dtype = ps.c_dtype = ZDRAW_DTYPE_F16;
  PartSpec part_s = {cx->wa_k16.p, cx->wa_p.p, static_cast<uint32_t>(zdraw::kEpilogueRowMax), nullptr, nullptr};
  part_s.row_key = row_key;
  part_s.row_sum = row_sum;
  part_s.n_partial = static_cast<int>(n_partial);
  part_s.exp_scale = 1.4426950408889634f / std::sqrt(static_cast<float>(head_dim));
  part_s.n_valid = static_cast<uint32_t>(n_sample);
  WideSpec max_spec;
  max_spec.norms = cx->wa_state + zdraw::kWideNorms;
  max_spec.n_valid_all = static_cast<uint32_t>(tokens);
  max_spec.all_rows = cx->wa_state + zdraw::kWideAllKeys;
  max_spec.zero = split ? o : nullptr;
  max_spec.zero_n = n / 2;
  if ((rc = run_linear(cx, stream, cx->wa_q16.p, 1, &part_s, nullptr, nullptr, &ps, max_spec)) != 0) return rc;
  ps.n = static_cast<uint32_t>(n_pad);
  ps.ld_w = head_dim;
  part_s.n_valid = static_cast<uint32_t>(tokens);
  part_s.epilogue = static_cast<uint32_t>(zdraw::kEpilogueExp);
  if (stride > 1) {
    part_s.shift = shift;
    part_s.row_missed = row_missed;
    part_s.any_missed = cx->wa_state + zdraw::kWideMissed;
  }
  WideSpec exp_spec;
  exp_spec.norms_done = cx->wa_state + zdraw::kWideNorms;
  exp_spec.zero = split ? o + n / 2 : nullptr;
  exp_spec.zero_n = n / 2;
  if ((rc = run_linear(cx, stream, cx->wa_q16.p, 1, &part_s, nullptr, nullptr, &ps, exp_spec)) != 0) return rc;
  if (stride > 1) {
    zdraw::WideRescale rs = {};
    rs.p = cx->wa_p.p;
    rs.ld_p = static_cast<long long>(n_pad);
    rs.tokens = static_cast<int>(tokens);
    rs.n_partial = static_cast<int>(n_partial);
    rs.row_sum = row_sum;
    rs.shift = shift;
    rs.row_missed = row_missed;
    rs.any_missed = cx->wa_state + zdraw::kWideMissed;
    ZD_CUDA(cx, zdraw::launch_wide_rescale(st, rs, cx->sm_count));
  }
  // O[tokens, head_dim] = (P (V^T)^T) / row sum, f32 out
  zdraw_cuda_linear_params po = {};
  po.m = static_cast<uint32_t>(tokens);
  po.n = static_cast<uint32_t>(head_dim);
  po.k = static_cast<uint32_t>(n_pad);   // P with its zero padding; V^T has `tokens` columns, the rest reads as zeros
  po.ld_w = tokens;
  po.a_dtype = po.w_dtype = ZDRAW_DTYPE_F16;
  po.c_dtype = ZDRAW_DTYPE_F32;
  PartSpec part_o = {cx->wa_vt16.p, o, 0, nullptr, nullptr};
  part_o.row_sum = row_sum;
  part_o.n_partial = static_cast<int>(n_partial);
  WideSpec last;
  last.w_k_valid = static_cast<uint32_t>(tokens);
  last.rows_first = true;
  last.k_splits = split ? 2 : 1;
  return run_linear(cx, stream, cx->wa_p.p, 1, &part_o, nullptr, nullptr, &po, last);
}

int zdraw_cuda_wide_attention_route(void* ctx, void* stream, uint32_t* exact_row_max) {
  Ctx* cx = as_ctx(ctx);
  if (!cx || !exact_row_max) return ZDRAW_CUDA_E_ARG;
  *exact_row_max = 0;
  if (!cx->wa_ran) return fail(cx, ZDRAW_CUDA_E_ARG, "no wide attention call has run on this context");
  ZD_CUDA(cx, cudaSetDevice(cx->device));
  ZD_CUDA(cx, cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  uint32_t state[zdraw::kWideStateWords] = {};
  ZD_CUDA(cx, cudaMemcpy(state, cx->wa_state, sizeof(state), cudaMemcpyDeviceToHost));
  *exact_row_max = state[zdraw::kWideAllKeys] | state[zdraw::kWideMissed];
  return ZDRAW_CUDA_OK;
}

int zdraw_cuda_qkv_projection(void* ctx, void* stream, const void* x, const void* wq, const void* wk, const void* wv,
                              void* q16, void* k16, void* v, const float* q_w_txt, const float* q_w_img,
                              const float* k_w_txt, const float* k_w_img, const float* rope_cos,
                              const float* rope_sin, const zdraw_cuda_linear_params* p) {
  Ctx* cx = as_ctx(ctx);
  if (!cx) return ZDRAW_CUDA_E_ARG;
  if (!p) return fail(cx, ZDRAW_CUDA_E_ARG, "params is null");
  if (p->epilogue != 1) return fail(cx, ZDRAW_CUDA_E_ARG, "the q/k/v projection takes epilogue = 1 (q and k get the prologue)");
  const PartSpec parts[3] = {{wq, q16, 1, q_w_txt, q_w_img}, {wk, k16, 1, k_w_txt, k_w_img}, {wv, v, 0, nullptr, nullptr}};
  return run_linear(cx, stream, x, 3, parts, rope_cos, rope_sin, p, projection());
}

}  // extern "C"
