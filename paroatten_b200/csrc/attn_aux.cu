// Two small companions of the attention kernel:
//   paro_plan_validate      checks walk lists that were not built by this library (loaded from a file,
//                           handed over the C ABI) before the attention kernel follows them;
//   paro_merge_attn_states  combines two partial attention results (O, LSE) computed over disjoint sets
//                           of key blocks into the result over their union -- what the LSE output is for
//                           (sequence-parallel / ring composition, reference core.py:55-57).
#include <type_traits>

#include "common.cuh"

namespace paro {

enum PlanFault : int32_t {
  PLAN_OK = 0,
  PLAN_BAD_OFFSETS = 1,     // pair_ptr not starting at 0, not monotone, or beyond the schedule's length
  PLAN_BAD_COUNT = 2,       // more steps than slots, a negative count, or steps for a q-block that does not exist
  PLAN_BAD_BLOCK = 3,       // a k-block id >= nbk inside a q-block's steps
  PLAN_BAD_FILLER = 4,      // an entry past a q-block's steps that is not the 0xFFFF filler
  PLAN_BAD_ORDER = 5,       // k-blocks of a section (shared / own) not strictly ascending
};

// One warp per pair of q-blocks.  report[0] = fault, [1] = pair row, [2] = step, [3] = offending value;
// the first fault found wins.
__global__ void plan_validate_kernel(const int32_t* __restrict__ pair_ptr, const uint32_t* __restrict__ sched,
                                     const int32_t* __restrict__ cnt, int prows, int npairs, int nbq, int nbk,
                                     long long sched_len, int32_t* __restrict__ report) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  auto fault = [&](int code, int row, int step, int value) {
    if (atomicCAS(report, 0, code) == 0) {
      report[1] = row;
      report[2] = step;
      report[3] = value;
    }
  };
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < prows; r += warps) {
    const long long e0 = pair_ptr[r], e1 = pair_ptr[r + 1];
    if ((r == 0 && e0 != 0) || e0 < 0 || e1 < e0 || e1 > sched_len) {
      if (lane == 0) fault(PLAN_BAD_OFFSETS, r, 0, (int)e1);
      continue;
    }
    const int slots = (int)(e1 - e0);
    const int na = cnt[2 * r] & 0xFFFF, nb = cnt[2 * r + 1] & 0xFFFF;   // (high halves: optional q-block ids)
    const bool has_second = 2 * (r % npairs) + 1 < nbq;
    const int qa = (int)((uint32_t)cnt[2 * r] >> 16), qb = (int)((uint32_t)cnt[2 * r + 1] >> 16);
    if (qa > nbq || qb > nbq) {   // q-block id + 1 of a half, 0 = none given
      if (lane == 0) fault(PLAN_BAD_BLOCK, r, -1, qa > nbq ? qa - 1 : qb - 1);
      continue;
    }
    if (na < 0 || nb < 0 || na > slots || nb > slots || (!has_second && nb != 0)) {
      if (lane == 0) fault(PLAN_BAD_COUNT, r, 0, na > slots || na < 0 ? na : nb);
      continue;
    }
    for (int i = lane; i < slots; i += 32) {
      const uint32_t e = sched[e0 + i];
      const int ka = (int)(e & 0xFFFFu), kb = (int)(e >> 16);
      if (i < na ? ka >= nbk : ka != 0xFFFF) fault(i < na ? PLAN_BAD_BLOCK : PLAN_BAD_FILLER, r, i, ka);
      if (i < nb ? kb >= nbk : kb != 0xFFFF) fault(i < nb ? PLAN_BAD_BLOCK : PLAN_BAD_FILLER, r, i, kb);
      if (i > 0 && i < max(na, nb)) {
        // sections: shared steps (ka == kb) first, then each q-block's own steps; ascending inside a section
        const uint32_t ep = sched[e0 + i - 1];
        const int pa = (int)(ep & 0xFFFFu), pb = (int)(ep >> 16);
        const bool sh = i < na && i < nb && ka == kb, psh = (i - 1) < na && (i - 1) < nb && pa == pb;
        if (sh && !psh) fault(PLAN_BAD_ORDER, r, i, ka);                 // a shared step after an own step
        if (sh == psh) {
          if (i < na && ka <= pa) fault(PLAN_BAD_ORDER, r, i, ka);
          if (i < nb && kb <= pb) fault(PLAN_BAD_ORDER, r, i, kb);
        }
      }
    }
  }
}

// out = (o_a * w_a + o_b * w_b), w_x = exp(lse_x - lse), lse = log(exp(lse_a) + exp(lse_b)); a side whose
// LSE is -inf (no kept block for that row) contributes nothing.
// HBM-bound (6 bytes per element): 16 bytes = 8 channels of a row per load, MERGE_ROWS rows of both tensors in
// flight per thread.  A row's weights take two exponentials, a logarithm and two divisions: one lane computes
// them, from LSEs requested before the rows, and hands them to the D/8 lanes of the row (computed by every lane, with
// the row found by 64-bit divisions, they took about as long as the loads).
// Two rows in bf16, four in fp16, whose conversions take fewer instructions: 12 x 32760 x 128 with one, two, four rows 68,
// 53, 57 us in bf16 and 64, 49, 47 in fp16 (one row per thread, weights by every lane: 70, 68).  46 us are its bytes.
// Two rows as well where a CTA's four would be past a short sequence's end: 2000 x 16 x 128 in fp16 8.3 and 11 us.
template <typename T, int D, int MERGE_ROWS>
__global__ void __launch_bounds__(256)
merge_states_kernel(const T* __restrict__ oa, const float* __restrict__ la, const T* __restrict__ ob,
                    const float* __restrict__ lb, T* __restrict__ out, float* __restrict__ lo, int H, int N, int BH,
                    int64_t sb, int64_t sh, int64_t sn) {
  constexpr int TPR = D / 8, RPW = 32 / TPR;      // lanes per row, rows a warp covers with one load
  constexpr int WROWS = RPW * MERGE_ROWS;         // rows per warp, consecutive
  const int lane = threadIdx.x & 31, c8 = (lane % TPR) * 8;
  const int n0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * WROWS;
  for (int bh = blockIdx.y; bh < BH; bh += gridDim.y) {
    const int64_t base = (bh / H) * sb + (bh % H) * sh + c8;
    const size_t row0 = (size_t)bh * N;
    const bool mine = lane < WROWS && n0 + lane < N;
    const float a = mine ? la[row0 + n0 + lane] : 0.f, c = mine ? lb[row0 + n0 + lane] : 0.f;
    Pack8<T> pa[MERGE_ROWS], pb[MERGE_ROWS];
#pragma unroll
    for (int u = 0; u < MERGE_ROWS; ++u) {
      const int n = n0 + u * RPW + lane / TPR;
      if (n < N) {
        pa[u].v = *reinterpret_cast<const uint4*>(oa + base + (int64_t)n * sn);
        pb[u].v = *reinterpret_cast<const uint4*>(ob + base + (int64_t)n * sn);
      }
    }
    float wa = 0.f, wb = 0.f;                     // of row n0 + lane
    if (mine) {
      const float m = fmaxf(a, c);
      float l = -INFINITY;
      if (m > -INFINITY) {
        const float ea = expf(a - m), eb = expf(c - m);   // exp(-inf) = 0
        const float s = ea + eb;
        wa = ea / s;
        wb = eb / s;
        l = m + logf(s);
      }
      if (lo) lo[row0 + n0 + lane] = l;
    }
#pragma unroll
    for (int u = 0; u < MERGE_ROWS; ++u) {
      const int n = n0 + u * RPW + lane / TPR;
      const float ua = __shfl_sync(0xffffffffu, wa, u * RPW + lane / TPR), ub = __shfl_sync(0xffffffffu, wb, u * RPW + lane / TPR);
      Pack8<T> po;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // a weight of exactly 0 drops that side even when it holds Inf or NaN (unwritten rows)
        const float va = ua != 0.f ? ua * F16Traits<T>::to_float(pa[u].e[j]) : 0.f;
        const float vb = ub != 0.f ? ub * F16Traits<T>::to_float(pb[u].e[j]) : 0.f;
        po.e[j] = F16Traits<T>::from_float(va + vb);
      }
      if (n < N) *reinterpret_cast<uint4*>(out + base + (int64_t)n * sn) = po.v;
    }
  }
}

template <typename T, int D>
void launch_merge(const void* oa, const float* la, const void* ob, const float* lb, void* out, float* lo, int B, int H, int N,
                  int64_t sb, int64_t sh, int64_t sn, cudaStream_t s) {
  auto launch = [&](auto rows) {
    constexpr int R = decltype(rows)::value, CTA_ROWS = 8 * R * (256 / D);
    const dim3 grid((N + CTA_ROWS - 1) / CTA_ROWS, (unsigned)min((long long)B * H, 65535ll));
    merge_states_kernel<T, D, R><<<grid, 256, 0, s>>>((const T*)oa, la, (const T*)ob, lb, (T*)out, lo, H, N, B * H, sb, sh, sn);
  };
  if (std::is_same<T, __half>::value && N >= 256) launch(std::integral_constant<int, 4>{});
  else launch(std::integral_constant<int, 2>{});
}

}  // namespace paro

using namespace paro;

extern "C" int paro_plan_validate(const int32_t* pair_ptr, const uint32_t* sched, const int32_t* sched_cnt, int slices,
                                  int nbq, int nbk, int64_t sched_len, int32_t* report, paro_stream_t stream) {
  PARO_REQUIRE(pair_ptr && sched && sched_cnt && report, PARO_EINVAL, "paro_plan_validate: null pointer");
  PARO_REQUIRE(slices > 0 && nbq > 0 && nbk > 0 && nbk < 0xFFFF && sched_len >= 0, PARO_ESHAPE,
               "paro_plan_validate: bad sizes (slices %d, nbq %d, nbk %d)", slices, nbq, nbk);
  cudaStream_t s = (cudaStream_t)stream;
  const int npairs = (nbq + 1) / 2;
  const long long prows = (long long)slices * npairs;
  PARO_REQUIRE(prows < (1ll << 31), PARO_ESHAPE, "paro_plan_validate: too many pairs");
  PARO_CUDA_OK(cudaMemsetAsync(report, 0, 4 * sizeof(int32_t), s));
  plan_validate_kernel<<<(unsigned)min(4096ll, (prows + 7) / 8), 256, 0, s>>>(pair_ptr, sched, sched_cnt, (int)prows,
                                                                              npairs, nbq, nbk, sched_len, report);
  if (int rc = check_launch("plan_validate_kernel")) return rc;
  int32_t w[4] = {0, 0, 0, 0};
  PARO_CUDA_OK(cudaMemcpyAsync(w, report, sizeof(w), cudaMemcpyDeviceToHost, s));
  PARO_CUDA_OK(cudaStreamSynchronize(s));
  static const char* const what[] = {"", "offsets not monotone from 0 or beyond the schedule", "step count out of range",
                                     "k-block id out of range", "entry past a q-block's steps is not the filler",
                                     "k-blocks of a section not strictly ascending"};
  if (w[0] != 0)
    return fail(PARO_EINVAL, "sparse plan rejected: %s (pair row %d, step %d, value %d)",
                what[w[0] >= 1 && w[0] <= 5 ? w[0] : 0], w[1], w[2], w[3]);
  return PARO_OK;
}

extern "C" int paro_merge_attn_states(const void* o_a, const float* lse_a, const void* o_b, const float* lse_b, void* out,
                                      float* lse_out, int dtype, int B, int H, int N, int D, int64_t stride_b,
                                      int64_t stride_h, int64_t stride_n, paro_stream_t stream) {
  PARO_REQUIRE(lse_a && lse_b, PARO_EINVAL, "paro_merge_attn_states: null pointer");
  if (int rc = check_tensor("paro_merge_attn_states(o_a)", o_a, dtype, B, H, N, D, stride_b, stride_h, stride_n)) return rc;
  if (int rc = check_tensor("paro_merge_attn_states(o_b)", o_b, dtype, B, H, N, D, stride_b, stride_h, stride_n)) return rc;
  if (int rc = check_tensor("paro_merge_attn_states(out)", out, dtype, B, H, N, D, stride_b, stride_h, stride_n)) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  auto merge = [&](auto tag) {
    using T = decltype(tag);
    if (D == 128) launch_merge<T, 128>(o_a, lse_a, o_b, lse_b, out, lse_out, B, H, N, stride_b, stride_h, stride_n, s);
    else launch_merge<T, 64>(o_a, lse_a, o_b, lse_b, out, lse_out, B, H, N, stride_b, stride_h, stride_n, s);
  };
  if (dtype == PARO_F16) merge(__half{});
  else merge(__nv_bfloat16{});
  return check_launch("merge_states_kernel");
}
