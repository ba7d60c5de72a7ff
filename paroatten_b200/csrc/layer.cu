// One self-attention layer per call: the pre-attention passes and the attention kernel of
// paro_attention, issued from one C entry point on one caller-provided work space.
//
// A layer is eight to ten launches.  Composed from Python (one ctypes call, its argument checks and two or three
// tensor allocations per pass) they cost about 190 us of host time, which is what a call of a few thousand
// tokens took; the device needs a fraction of that.  Here the host side is one call and the launches: 187 -> 74 us
// for 2 heads x 1024 tokens, 194 -> 158 us for 6 x 5960 (where the device is what remains); 63 and 140 us since K and V
// share their statistics launches and the passes themselves became shorter.
#include "attn_common.cuh"
#include "common.cuh"
#include "norm.cuh"
#include "rope.cuh"

using namespace paro;

namespace {

// Sections of the work space, each on a 256-byte boundary.
struct Sections {
  size_t q8, k8, v16, qs, ks, vs, vm, km, kp, rms_q, rms_k, tab32, stats, total;
};

// Elements of Q from which the passes get the fp32 copy of an interleaved fp64 table, made for the call: a launch of 2 us.
// Layers without it and with it, bf16: 4 x 2080 x 128 63.4 and 65.1 us, 8 x 4160 x 128 91.8 and 92.0, 8 x 6240 x 128 136.4 and
// 130.9, 24 x 6240 x 128 302 and 290 (fp16 300 and 292; with RMS norm level from here on).
constexpr int64_t FP32_TABLE_ELEMS = 4 << 20;
bool fp32_table(const paro_layer_args& a) {
  return a.rope_mode == PARO_ROPE_COMPLEX_F64 && a.cos_tab && !a.sin_tab && a.F > 0 && a.Hh > 0 && a.W > 0 &&
         (int64_t)a.B * a.H * a.N * a.D >= FP32_TABLE_ELEMS;
}
int64_t table_pairs(const paro_layer_args& a) { return ((int64_t)a.F + a.Hh + a.W) * (a.D / 2); }

Sections sections(const paro_layer_args& a) {
  const size_t BH = (size_t)a.B * a.H, rows = BH * a.N, D = a.D, nb = ((size_t)a.N + 63) / 64;
  Sections s{};
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) / 256 * 256;
    return here;
  };
  s.q8 = take(rows * D);
  s.k8 = take(rows * D);
  s.v16 = take(BH * D * nb * 64 * 2);
  s.qs = take(BH * nb * 2 * sizeof(float));
  s.ks = take(BH * nb * sizeof(float));
  s.vs = take(BH * D * sizeof(float));
  s.vm = take(BH * D * sizeof(float));
  s.km = take(BH * D * 2);
  s.kp = take(a.smooth_k ? rows * D * 2 : 0);
  s.rms_q = take(a.q_norm_mode == PARO_NORM_RMS_ALL ? (size_t)a.B * a.N * sizeof(float) : 0);
  s.rms_k = take(a.k_norm_mode == PARO_NORM_RMS_ALL ? (size_t)a.B * a.N * sizeof(float) : 0);
  s.tab32 = take(fp32_table(a) ? table_pairs(a) * sizeof(float2) : 0);
  s.stats = take(layer_kv_scratch_bytes(a.B, a.H, a.N, a.D));
  s.total = at;
  return s;
}

}  // namespace

extern "C" size_t paro_layer_workspace_bytes(const paro_layer_args* a) {
  if (!a || a->B <= 0 || a->H <= 0 || a->N <= 0 || (a->D != 64 && a->D != 128)) return 0;
  return sections(*a).total;
}

extern "C" int paro_layer(const paro_layer_args* args, paro_stream_t stream) {
  PARO_REQUIRE(args, PARO_EINVAL, "paro_layer: null arguments");
  const paro_layer_args& a = *args;
  PARO_REQUIRE(a.B > 0 && a.H > 0 && a.N > 0 && (a.D == 64 || a.D == 128), PARO_ESHAPE, "paro_layer: bad sizes");
  const Sections at = sections(a);
  PARO_REQUIRE(a.workspace && aligned16(a.workspace) && a.workspace_bytes >= at.total, PARO_ECAP,
               "paro_layer: work space too small or unaligned (%zu < %zu)", a.workspace_bytes, at.total);
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t* w = static_cast<uint8_t*>(a.workspace);
  int8_t* q8 = reinterpret_cast<int8_t*>(w + at.q8);
  int8_t* k8 = reinterpret_cast<int8_t*>(w + at.k8);
  uint16_t* v16 = reinterpret_cast<uint16_t*>(w + at.v16);
  float *qs = reinterpret_cast<float*>(w + at.qs), *ks = reinterpret_cast<float*>(w + at.ks);
  float *vs = reinterpret_cast<float*>(w + at.vs), *vm = reinterpret_cast<float*>(w + at.vm);

  // what the pre-attention passes would refuse, before the first of them
  if (int rc = check_tensor("paro_layer(q)", a.q, a.dtype, a.B, a.H, a.N, a.D, a.q_strides[0], a.q_strides[1], a.q_strides[2])) return rc;
  if (int rc = check_tensor("paro_layer(k)", a.k, a.dtype, a.B, a.H, a.N, a.D, a.k_strides[0], a.k_strides[1], a.k_strides[2])) return rc;
  if (int rc = check_tensor("paro_layer(v)", a.v, a.dtype, a.B, a.H, a.N, a.D, a.v_strides[0], a.v_strides[1], a.v_strides[2])) return rc;
  PARO_REQUIRE(a.F > 0 && a.Hh > 0 && a.W > 0 && a.n_text >= 0 && (int64_t)a.n_text + (int64_t)a.F * a.Hh * a.W == a.N,
               PARO_ESHAPE, "paro_layer: n_text + F*H*W = %lld != N = %d", (long long)a.n_text + (long long)a.F * a.Hh * a.W, a.N);
  if (int rc = check_rope("paro_layer", a.rope_mode, a.cos_tab, a.sin_tab, a.pairs_f, a.pairs_h, a.D)) return rc;
  const float* const section = reinterpret_cast<const float*>(w);   // (stands for the RMS statistics, computed below)
  if (int rc = check_norm("paro_layer(q)", a.q_norm_mode, a.q_norm_weight, a.q_norm_bias, section, a.q_norm_eps)) return rc;
  if (int rc = check_norm("paro_layer(k)", a.k_norm_mode, a.k_norm_weight, a.k_norm_bias, section, a.k_norm_eps)) return rc;

  int rope_mode = a.rope_mode;
  const void* sin_tab = a.sin_tab;
  if (fp32_table(a)) {
    rope_mode = PARO_ROPE_COMPLEX_F64_APPROX;
    sin_tab = w + at.tab32;
    if (int rc = launch_round_table(a.cos_tab, w + at.tab32, table_pairs(a), s)) return rc;
  }

  // the per-token statistic of an RMS norm over all heads
  auto inv_rms = [&](const void* x, const int64_t* st, int mode, float eps, size_t section, const float** out) -> int {
    *out = nullptr;
    if (mode != PARO_NORM_RMS_ALL) return PARO_OK;
    float* buf = reinterpret_cast<float*>(w + section);
    *out = buf;
    return paro_row_inv_rms(x, a.dtype, a.B, a.H, a.N, a.D, st[0], st[1], st[2], eps, buf, stream);
  };
  // RoPE + reorder + INT8 of one tensor in one pass
  auto prep = [&](const void* x, const int64_t* st, int group, int norm, const void* weight, const void* bias,
                  const float* rms, float eps, int8_t* out, float* scale) -> int {
    if (norm != PARO_NORM_NONE)
      return paro_prep_qk_int8_norm(x, a.dtype, a.B, a.H, a.N, a.D, st[0], st[1], st[2], a.n_text, a.F, a.Hh, a.W,
                                    a.order_ids, rope_mode, a.cos_tab, sin_tab, a.pairs_f, a.pairs_h, group, out, scale,
                                    norm, weight, bias, rms, eps, stream);
    return paro_prep_qk_int8(x, a.dtype, a.B, a.H, a.N, a.D, st[0], st[1], st[2], a.n_text, a.F, a.Hh, a.W, a.order_ids,
                             rope_mode, a.cos_tab, sin_tab, a.pairs_f, a.pairs_h, group, 0, nullptr, out, scale,
                             nullptr, 0, stream);
  };

  const float* rms = nullptr;
  if (int rc = inv_rms(a.q, a.q_strides, a.q_norm_mode, a.q_norm_eps, at.rms_q, &rms)) return rc;
  if (int rc = prep(a.q, a.q_strides, 32, a.q_norm_mode, a.q_norm_weight, a.q_norm_bias, rms, a.q_norm_eps, q8, qs)) return rc;

  if (int rc = inv_rms(a.k, a.k_strides, a.k_norm_mode, a.k_norm_eps, at.rms_k, &rms)) return rc;
  void* kp = nullptr;   // K's rotated and reordered copy, where it is smoothed
  if (!a.smooth_k) {
    if (int rc = prep(a.k, a.k_strides, 64, a.k_norm_mode, a.k_norm_weight, a.k_norm_bias, rms, a.k_norm_eps, k8, ks)) return rc;
  } else {
    // The mean to subtract is that of the rotated values.  The rotated copy is written once and read twice: 127 us for
    // 5 x 75600 x 128 with the fp64 rotation, 227 us for 2 x 48 x 17776 x 64 with the fp32 one, against 152 and 264 us for
    // rotating K in the statistics pass and again in the quantiser.
    kp = w + at.kp;
    const int rc = a.k_norm_mode == PARO_NORM_NONE
        ? paro_rope_permute(a.k, kp, a.dtype, a.B, a.H, a.N, a.D, a.k_strides[0], a.k_strides[1], a.k_strides[2], a.n_text,
                            a.F, a.Hh, a.W, a.order_ids, 0, rope_mode, a.cos_tab, sin_tab, a.pairs_f, a.pairs_h, stream)
        : paro_rope_permute_norm(a.k, kp, a.dtype, a.B, a.H, a.N, a.D, a.k_strides[0], a.k_strides[1], a.k_strides[2],
                                 a.n_text, a.F, a.Hh, a.W, a.order_ids, rope_mode, a.cos_tab, sin_tab, a.pairs_f,
                                 a.pairs_h, a.k_norm_mode, a.k_norm_weight, a.k_norm_bias, rms, a.k_norm_eps, stream);
    if (rc) return rc;
  }
  // (these passes clear the redo counter as well)
  const bool fast = a.attn_mode == PARO_ATTN_FAST && a.redo && a.redo_bytes >= sizeof(int32_t);
  if (int rc = layer_kv_passes(a, kp, w + at.km, k8, ks, v16, vs, vm, w + at.stats, fast ? a.redo : nullptr, s)) return rc;

  if (a.ev_start) PARO_CUDA_OK(cudaEventRecord((cudaEvent_t)a.ev_start, s));
  if (int rc = sparse_attn_launch(q8, k8, v16, qs, 32, ks, vs, a.smooth_v ? vm : nullptr, a.pair_ptr, a.sched, a.sched_cnt,
                                  a.plan_slices, a.inv_idx, a.n_text, a.out, a.dtype, a.out_strides[0], a.out_strides[1],
                                  a.out_strides[2], a.lse, a.B, a.H, a.N, a.D, a.sm_scale, a.attn_mode, a.redo, a.redo_bytes,
                                  a.status, a.host_status, fast, s))
    return rc;
  if (a.ev_stop) PARO_CUDA_OK(cudaEventRecord((cudaEvent_t)a.ev_stop, s));
  return PARO_OK;
}
