// Compaction of a boolean block mask into walk lists, with the q-blocks of a pair chosen by the k-blocks they
// share.  Integer work only; every list is compared bit for bit with the CPU oracle.
//
//   pack      mask bytes -> one bit per block (1/8 of the bytes, and all later passes work on whole words)
//   overlap   shared k-blocks of every two q-blocks of a slice, the product of the 0/1 matrix with its transpose, on the
//             tensor cores
//   pair      greedy pairing, one CTA per slice
//   count     kept blocks per q-block and per pair; two scans turn them into offsets
//   lists     the CSR lists, the merged lists and the walk schedule of a pair, written by one warp
//
// The host reads three totals back between count and lists (the lists' lengths), once per call.
// Measured on a 40 x 1182 x 1182 mask at density 0.2: 0.58 ms on the device (pack 48 us, overlap 98, pair 290, count and
// scans 17, lists 110) and 0.8 ms for the whole call; a fp32 bmm with 591 rounds of small torch kernels took 67 ms.
#include "common.cuh"
#include "umma.cuh"

namespace paro {

using namespace umma;

// Layout of the scratch buffer of paro_plan_offsets / paro_plan_lists.
struct PlanScratch {
  uint32_t* bits;      // [slices*nbq][words]
  int32_t* row_cnt;    // [slices*nbq] kept blocks per q-block, mask order
  int32_t* part;       // [2][scan blocks] partial sums of the two scans
  uint16_t* ov;        // [slices*nbq][pitch] overlaps (pairing by overlap only); entries left of the diagonal tile are not written
  int words, pitch, scan_blocks;
  size_t bytes;
};

constexpr int SCAN_ITEMS = 1024;   // elements one block scans

static PlanScratch plan_scratch(void* base, int slices, int nbq, int nbk, int overlap) {
  PlanScratch s;
  const size_t rows = (size_t)slices * nbq;
  s.words = (nbk + 127) / 128 * 4;   // 16-byte rows; the padding bits are 0
  s.pitch = (nbq + 7) & ~7;          // 16-byte rows
  s.scan_blocks = (int)((rows + SCAN_ITEMS - 1) / SCAN_ITEMS);
  size_t off = 0;
  auto take = [&](size_t n) {
    const size_t at = off;
    off += (n + 255) & ~size_t(255);
    return static_cast<char*>(base) + at;
  };
  s.bits = reinterpret_cast<uint32_t*>(take(rows * s.words * 4));
  s.row_cnt = reinterpret_cast<int32_t*>(take(rows * 4));
  s.part = reinterpret_cast<int32_t*>(take(2 * (size_t)s.scan_blocks * 4));
  s.ov = reinterpret_cast<uint16_t*>(take(overlap ? rows * s.pitch * 2 : 0));
  s.bytes = off;
  return s;
}

// One warp per mask row; bound by the mask's bytes.  A row starts at any byte, so lanes read single bytes (32 of them are
// one sector) and a ballot makes the word; eight words are in flight per warp.
__global__ void __launch_bounds__(256)
plan_pack_kernel(const uint8_t* __restrict__ mask, int rows, int nbk, int words, uint32_t* __restrict__ bits,
                 int32_t* __restrict__ row_cnt) {
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
    const uint8_t* src = mask + (size_t)r * nbk;
    int cnt = 0;
    for (int w0 = 0; w0 < words; w0 += 8) {
      uint8_t v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int kb = (w0 + u) * 32 + lane;
        v[u] = kb < nbk ? src[kb] : 0;
      }
      uint32_t mine = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t b = __ballot_sync(0xffffffffu, v[u] != 0);
        cnt += __popc(b);
        if (lane == u) mine = b;
      }
      if (lane < 8 && w0 + lane < words) bits[(size_t)r * words + w0 + lane] = mine;
    }
    if (lane == 0) row_cnt[r] = cnt;
  }
}

// Overlaps of 128 x 128 pairs of rows per CTA on kind::i8 (0/1 bytes, int32 accumulators in TMEM), only tiles on or above
// the diagonal: the pairing asks for the partners AFTER a row.  The operands are expanded from the bit rows by the
// CTA itself -- one thread turns 128 bits of a row into the row of a 128-byte-swizzled K-major tile -- so nothing but the
// bits (1/8 of the mask) is read; two stages, the next one is expanded while the MMAs of the last one run.  The same sums
// by AND + POPC (16 per clock and SM) took about 250 us where this takes 98.
constexpr int OV_TILE = 128, OV_THREADS = 256, OV_STAGE = 2 * OV_TILE * 128;   // bytes of a stage: A and B, 128 k-blocks deep
constexpr int OV_SMEM = 2 * OV_STAGE + 1024;
constexpr long long OV_WAIT_LIMIT = 400000000;   // SM clocks before a wait gives up
__global__ void __launch_bounds__(OV_THREADS)
plan_overlap_kernel(const uint32_t* __restrict__ bits, int slices, int nbq, int words, int pitch, uint16_t* __restrict__ ov,
                    int32_t* __restrict__ error) {
  extern __shared__ uint8_t ov_smem[];
  __shared__ uint64_t s_bar[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_failed;
  const int tj = blockIdx.x, ti = blockIdx.y;
  if (tj < ti) return;
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ov_smem) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    s_failed = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&s_tmem, OV_TILE);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t acc = s_tmem;
  constexpr uint32_t IDESC = instr_desc(2, 1, 1, OV_TILE, OV_TILE);   // s32 += s8 * s8
  const int r = threadIdx.x & (OV_TILE - 1);
  const int row = (threadIdx.x < OV_TILE ? ti : tj) * OV_TILE + r;   // threads 0-127 expand A, 128-255 B
  uint8_t* const my_row = tiles + (threadIdx.x < OV_TILE ? 0 : OV_TILE * 128) + r * 128;
  const int chunks = words / 4;
  int done = 0;   // stages handed to the tensor cores so far
  bool ok = true;
  for (int slice = blockIdx.z; slice < slices && ok; slice += gridDim.z) {
    const uint32_t* src = bits + ((size_t)slice * nbq + (row < nbq ? row : 0)) * words;
    for (int c = 0; c < chunks; ++c, ++done) {
      const int st = done & 1;
      uint4 v = row < nbq ? *reinterpret_cast<const uint4*>(src + 4 * c) : make_uint4(0, 0, 0, 0);
      if (done >= 2 && !mbar_wait_plain_bounded(&s_bar[st], ((done >> 1) - 1) & 1, OV_WAIT_LIMIT)) s_failed = 1;
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {   // 16 bits -> 16 bytes: a nibble times (1 + 2^7 + 2^14 + 2^21) puts its bits 8 apart
        const uint32_t h = w[k >> 1] >> (16 * (k & 1));
        uint4 e;
        e.x = (h & 15u) * 0x00204081u & 0x01010101u;
        e.y = (h >> 4 & 15u) * 0x00204081u & 0x01010101u;
        e.z = (h >> 8 & 15u) * 0x00204081u & 0x01010101u;
        e.w = (h >> 12 & 15u) * 0x00204081u & 0x01010101u;
        *reinterpret_cast<uint4*>(my_row + st * OV_STAGE + ((k ^ (r & 7)) << 4)) = e;
      }
      fence_proxy_async();
      tc_fence_before();
      __syncthreads();
      if (s_failed) {
        ok = false;
        break;
      }
      if (threadIdx.x == 0) {
        tc_fence_after();
        const uint64_t da = smem_desc(smem_u32(tiles + st * OV_STAGE), 128), db = smem_desc(smem_u32(tiles + st * OV_STAGE + OV_TILE * 128), 128);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_i8_ss(acc, desc_advance(da, 32 * k), desc_advance(db, 32 * k), IDESC, c > 0 || k > 0);
        mma_commit(&s_bar[st]);
      }
    }
    // the last stage's commit covers all of the slice's MMAs; both stages are free afterwards
    if (ok && !mbar_wait_plain_bounded(&s_bar[(done - 1) & 1], ((done - 1) >> 1) & 1, OV_WAIT_LIMIT)) s_failed = 1;
    tc_fence_after();
    // warp w: lanes (rows) of quadrant w & 3, 64 of the 128 columns
    const int orow = ti * OV_TILE + (warp & 3) * 32 + lane, col0 = tj * OV_TILE + (warp >> 2) * 64;
    uint16_t* dst = ov + ((size_t)slice * nbq + orow) * pitch;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t o[32];
      tmem_ld32(acc + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 64 + 32 * q), o);
      tmem_wait_ld();
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int c8 = col0 + 32 * q + 8 * g;   // (the pitch is a multiple of 8: a group is inside or outside as a whole)
        if (orow < nbq && c8 < pitch)
          *reinterpret_cast<uint4*>(dst + c8) = make_uint4(o[8 * g] | o[8 * g + 1] << 16, o[8 * g + 2] | o[8 * g + 3] << 16,
                                                           o[8 * g + 4] | o[8 * g + 5] << 16, o[8 * g + 6] | o[8 * g + 7] << 16);
      }
    }
    tc_fence_before();
    __syncthreads();   // the accumulator is read before the next slice's first MMA overwrites it
    tc_fence_after();
    ok = ok && !s_failed;
  }
  if (threadIdx.x == 0 && s_failed) *error = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(acc, OV_TILE);
  }
}

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
               : "memory");
}

// Greedy pairing of one slice per CTA: the first q-block not yet paired takes the free q-block it shares most
// k-blocks with (ties: the lowest index).  The nbq/2 rounds are a serial chain, so the latency of a round is what
// counts: one barrier per round (the bit of the q-block taken last may not have reached every thread yet; it is
// carried in a register instead), eight candidates per thread and load, the word of the free map around the current row in a
// register, and, since the first free q-block only moves forward, the overlap rows are brought to shared memory
// `1 << chunk_log` rows at a time, one chunk ahead.  chunk_log < 0: rows too long for shared memory, read where they are.
// (591 rounds: 290 us; with two-byte candidates and the free map searched in shared memory 500 us.)
// A pairing that does not need fewer tiles than adjacency is replaced by adjacency; any[0] = 1 if one was kept.
constexpr int PAIR_THREADS = 256, PAIR_MAX_ROWS = 65536;
__global__ void __launch_bounds__(PAIR_THREADS)
plan_pair_kernel(const uint16_t* __restrict__ ov, int nbq, int pitch, int npairs, int chunk_log, int32_t* __restrict__ pair_q,
                 int32_t* __restrict__ any) {
  extern __shared__ __align__(16) uint16_t s_rows[];
  __shared__ uint32_t s_free[PAIR_MAX_ROWS / 32];   // bit per q-block, as words and as bytes (byte t: rows 8t..8t+7)
  __shared__ __align__(16) uint32_t s_part[2][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const uint8_t* s_free8 = reinterpret_cast<const uint8_t*>(s_free);
  const uint16_t* o = ov + (size_t)blockIdx.x * nbq * pitch;
  int32_t* out = pair_q + (size_t)blockIdx.x * npairs * 2;
  for (int w = tid; w < (nbq + 31) / 32; w += threads)
    s_free[w] = nbq - 32 * w >= 32 ? 0xffffffffu : (1u << (nbq - 32 * w)) - 1u;
  if (tid < 16) s_part[tid >> 3][tid & 7] = 0;

  int loaded = -1;   // newest chunk requested
  auto load = [&](int c) {
    loaded = c;
    const int r0 = c << chunk_log;
    if (r0 >= nbq) return;
    const int n16 = min(1 << chunk_log, nbq - r0) * (pitch / 8);
    const uint4* src = reinterpret_cast<const uint4*>(o + (size_t)r0 * pitch);
    uint4* dst = reinterpret_cast<uint4*>(s_rows + (size_t)(c & 1) * ((size_t)pitch << chunk_log));
    for (int k = tid; k < n16; k += threads) cp_async16(dst + k, src + k);
  };
  if (chunk_log >= 0) load(0);
  __syncthreads();

  int cur = -1, i = -1, gone = -1;
  long long shared_greedy = 0;
  int fw = 0;                      // word of the free map that holds the next free q-block after i, as far as known
  uint32_t fm = s_free[0];         // its bits after i
  auto next_free = [&]() {         // (the caller knows there is one)
    for (;;) {
      if (gone >= 0 && (gone >> 5) == fw) fm &= ~(1u << (gone & 31));
      if (fm) {
        const int bit = __ffs(fm) - 1;
        fm &= fm - 1;
        return fw * 32 + bit;
      }
      fm = s_free[++fw];           // all but the bit of `gone` are up to date: the round before last is behind a barrier
    }
  };
  for (int p = 0; p < nbq / 2; ++p) {
    i = next_free();
    const uint16_t* row = o + (size_t)i * pitch;
    if (chunk_log >= 0) {
      const int c = i >> chunk_log;
      if (c != cur) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (c != loaded) {          // (the chunks in between held no free q-block)
          load(c);
          asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncthreads();            // the chunk before this one was last read before the previous round's barrier
        load(c + 1);
        cur = c;
      }
      row = s_rows + (size_t)(c & 1) * ((size_t)pitch << chunk_log) + (size_t)(i - (c << chunk_log)) * pitch;
    }
    uint32_t best = 0;
    for (int j8 = tid * 8; j8 < nbq; j8 += threads * 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + j8);
      uint32_t m = s_free8[j8 >> 3];
      if (j8 + 7 <= i) m = 0;
      else if (j8 <= i) m &= 0xFFu << (i - j8 + 1);
      if ((gone >> 3) == (j8 >> 3)) m &= ~(1u << (gone & 7));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t key = ((k & 1 ? w[k >> 1] >> 16 : w[k >> 1] & 0xFFFFu) << 16) | (uint32_t)(0xFFFF - j8 - k);
        best = max(best, m >> k & 1u ? key : 0u);
      }
    }
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) s_part[p & 1][warp] = best;
    __syncthreads();
    const uint4 x = *reinterpret_cast<const uint4*>(s_part[p & 1]), y = *reinterpret_cast<const uint4*>(s_part[p & 1] + 4);
    best = max(max(max(x.x, x.y), max(x.z, x.w)), max(max(y.x, y.y), max(y.z, y.w)));
    gone = 0xFFFF - (int)(best & 0xFFFFu);
    shared_greedy += best >> 16;
    if (tid == 0) {
      s_free[i >> 5] &= ~(1u << (i & 31));
      s_free[gone >> 5] &= ~(1u << (gone & 31));
      *reinterpret_cast<int2*>(out + 2 * p) = make_int2(i, gone);
    }
  }
  if (nbq & 1) {
    i = next_free();
    if (tid == 0) *reinterpret_cast<int2*>(out + nbq - 1) = make_int2(i, -1);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // adjacency's shared blocks
  __syncthreads();
  uint32_t mine = 0;
  for (int p = tid; p < nbq / 2; p += threads) mine += o[(size_t)(2 * p) * pitch + 2 * p + 1];
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) s_part[0][warp] = mine;
  __syncthreads();
  long long shared_adjacent = 0;
  for (int k = 0; k < threads / 32; ++k) shared_adjacent += s_part[0][k];
  if (shared_greedy > shared_adjacent) {
    if (tid == 0) *any = 1;
  } else {
    for (int k = tid; k < 2 * npairs; k += threads) out[k] = k < nbq ? k : -1;
  }
}

// The q-blocks of pair row r (qb = -1: none).
__device__ __forceinline__ void pair_rows(const int32_t* pair_q, int r, int npairs, int nbq, int& qa, int& qb) {
  if (pair_q) {
    qa = pair_q[2 * r];
    qb = pair_q[2 * r + 1];
  } else {
    const int p = r % npairs;
    qa = 2 * p;
    qb = 2 * p + 1 < nbq ? 2 * p + 1 : -1;
  }
}

// One warp per pair: kept blocks of its two q-blocks and of their union, at the places the scans run over.
__global__ void __launch_bounds__(256)
plan_pair_count_kernel(const uint32_t* __restrict__ bits, const int32_t* __restrict__ row_cnt, int nbq, int words, int npairs,
                       int prows, const int32_t* __restrict__ pair_q, int32_t* __restrict__ row_ptr,
                       int32_t* __restrict__ pair_ptr) {
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < prows; r += warps) {
    int qa, qb;
    pair_rows(pair_q, r, npairs, nbq, qa, qb);
    const size_t row0 = (size_t)(r / npairs) * nbq;
    const uint32_t *a = bits + (row0 + qa) * words, *b = bits + (row0 + (qb < 0 ? qa : qb)) * words;
    uint32_t n = 0;
    for (int w = lane; w < words; w += 32) n += __popc(a[w] | b[w]);
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) {
      const size_t at = row0 + 2 * (size_t)(r % npairs);
      row_ptr[at + 1] = row_cnt[row0 + qa];
      if (qb >= 0) row_ptr[at + 2] = row_cnt[row0 + qb];
      pair_ptr[r + 1] = (int)n;
    }
  }
}

__device__ __forceinline__ int block_sum_1024(int v, int* s32) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s32[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, s32[threadIdx.x & 31]);
}

// In-place inclusive scans of row_ptr[1..n0] (blockIdx.y = 0) and pair_ptr[1..n1] (1) in two launches: the sums of
// 1024-element blocks, then every block adds up the sums before its own and scans its elements.
__global__ void __launch_bounds__(1024)
plan_scan_sums_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ pair_ptr, int n0, int n1,
                      int32_t* __restrict__ part) {
  __shared__ int s32[32];
  const int n = blockIdx.y ? n1 : n0, i = blockIdx.x * SCAN_ITEMS + threadIdx.x;
  const int32_t* a = blockIdx.y ? pair_ptr : row_ptr;
  const int sum = block_sum_1024(i < n ? a[i + 1] : 0, s32);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = sum;
}

__global__ void __launch_bounds__(1024)
plan_scan_kernel(int32_t* __restrict__ row_ptr, int32_t* __restrict__ pair_ptr, int n0, int n1,
                 const int32_t* __restrict__ part, int32_t* __restrict__ totals) {
  __shared__ int s32[2][32];
  const int n = blockIdx.y ? n1 : n0, i = blockIdx.x * SCAN_ITEMS + threadIdx.x, lane = threadIdx.x & 31;
  int32_t* a = blockIdx.y ? pair_ptr : row_ptr;
  int before = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += 1024) before += part[blockIdx.y * gridDim.x + k];
  before = block_sum_1024(before, s32[0]);
  int v = i < n ? a[i + 1] : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) s32[1][threadIdx.x >> 5] = v;
  __syncthreads();
  const int w = threadIdx.x >> 5;
  v += before + __reduce_add_sync(0xffffffffu, lane < w ? s32[1][lane] : 0);
  if (i < n) a[i + 1] = v;
  if (i == 0) a[0] = 0;
  if (i == n - 1) totals[blockIdx.y] = v;
}

// One warp per pair writes everything that is read of it: cols of its two q-blocks, the merged list, the schedule and the
// step counts.  A lane owns one word (32 k-blocks) of the two bit rows, expands its set bits into per-list staging in
// shared memory at offsets from a warp scan, and the lists are copied out in whole lines (expanding straight to
// global memory writes each sector once per entry).  1024 k-blocks are staged at a time.
constexpr int LIST_WARPS = 4, LIST_CHUNK = 1024;
__global__ void __launch_bounds__(32 * LIST_WARPS)
plan_lists_kernel(const uint32_t* __restrict__ bits, int nbq, int words, int npairs, int prows,
                  const int32_t* __restrict__ pair_q, const int32_t* __restrict__ row_ptr,
                  const int32_t* __restrict__ pair_ptr, int32_t* __restrict__ cols, int32_t* __restrict__ pair_ent,
                  uint32_t* __restrict__ sched, int32_t* __restrict__ cnt, int32_t* __restrict__ cnt_kernel) {
  __shared__ uint16_t s_list[LIST_WARPS][6][LIST_CHUNK];
  const int lane = threadIdx.x & 31, warps = gridDim.x * LIST_WARPS;
  auto& L = s_list[threadIdx.x >> 5];   // 0/1 q-block A/B, 2 merged (local id * 4 + flags), 3 both, 4/5 only A/B
  uint16_t* sched16 = reinterpret_cast<uint16_t*>(sched);
  for (int r = blockIdx.x * LIST_WARPS + (threadIdx.x >> 5); r < prows; r += warps) {
    int qa, qb;
    pair_rows(pair_q, r, npairs, nbq, qa, qb);
    const size_t row0 = (size_t)(r / npairs) * nbq, at = row0 + 2 * (size_t)(r % npairs);
    const uint32_t *pa = bits + (row0 + qa) * words, *pb = bits + (row0 + (qb < 0 ? qa : qb)) * words;
    uint32_t both = 0;
    if (qb >= 0) {
      for (int w = lane; w < words; w += 32) both += __popc(pa[w] & pb[w]);
      both = __reduce_add_sync(0xffffffffu, both);
    }
    const int e0 = pair_ptr[r], slots = pair_ptr[r + 1] - e0, ns = (int)both;
    int at_a = row_ptr[at], at_b = qb >= 0 ? row_ptr[at + 1] : 0, at_u = e0, at_s = e0, at_1 = e0 + ns, at_2 = e0 + ns;
    for (int w0 = 0; w0 < words; w0 += 32) {
      const uint32_t a = w0 + lane < words ? pa[w0 + lane] : 0u, b = qb >= 0 && w0 + lane < words ? pb[w0 + lane] : 0u;
      // inclusive warp scans of |a|, |b| (16 bits each: at most 1024) and |a & b|
      uint32_t nab = (uint32_t)__popc(a) | ((uint32_t)__popc(b) << 16), nsh = (uint32_t)__popc(a & b);
      uint32_t sab = nab, ssh = nsh;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t0 = __shfl_up_sync(0xffffffffu, sab, o), t1 = __shfl_up_sync(0xffffffffu, ssh, o);
        if (lane >= o) { sab += t0; ssh += t1; }
      }
      const uint32_t tab = __shfl_sync(0xffffffffu, sab, 31), tsh = __shfl_sync(0xffffffffu, ssh, 31);
      const int t_a = (int)(tab & 0xFFFFu), t_b = (int)(tab >> 16), t_s = (int)tsh, t_u = t_a + t_b - t_s;
      sab -= nab;
      ssh -= nsh;
      int i_a = (int)(sab & 0xFFFFu), i_b = (int)(sab >> 16), i_s = (int)ssh;
      for (uint32_t u = a | b; u; u &= u - 1) {
        const int bit = __ffs(u) - 1, kb = lane * 32 + bit;
        const int in_a = (a >> bit) & 1u, in_b = (b >> bit) & 1u;
        L[2][i_a + i_b - i_s] = (uint16_t)(kb * 4 + in_a + 2 * in_b);
        if (in_a & in_b) L[3][i_s] = (uint16_t)kb;
        else if (in_a) L[4][i_a - i_s] = (uint16_t)kb;
        else L[5][i_b - i_s] = (uint16_t)kb;
        if (in_a) L[0][i_a] = (uint16_t)kb;
        if (in_b) L[1][i_b] = (uint16_t)kb;
        i_a += in_a;
        i_b += in_b;
        i_s += in_a & in_b;
      }
      __syncwarp();
      const int k0 = w0 * 32;
      for (int k = lane; k < t_a; k += 32) cols[at_a + k] = k0 + L[0][k];
      for (int k = lane; k < t_b; k += 32) cols[at_b + k] = k0 + L[1][k];
      for (int k = lane; k < t_u; k += 32) pair_ent[at_u + k] = 4 * k0 + L[2][k];
      for (int k = lane; k < t_s; k += 32) sched[at_s + k] = (uint32_t)(k0 + L[3][k]) * 0x10001u;
      for (int k = lane; k < t_a - t_s; k += 32) sched16[2 * (size_t)(at_1 + k)] = (uint16_t)(k0 + L[4][k]);
      for (int k = lane; k < t_b - t_s; k += 32) sched16[2 * (size_t)(at_2 + k) + 1] = (uint16_t)(k0 + L[5][k]);
      __syncwarp();
      at_a += t_a; at_b += t_b; at_u += t_u; at_s += t_s; at_1 += t_a - t_s; at_2 += t_b - t_s;
    }
    // steps past the end of a q-block's list hold the filler
    for (int k = at_1 + lane; k < e0 + slots; k += 32) sched16[2 * (size_t)k] = 0xFFFFu;
    for (int k = at_2 + lane; k < e0 + slots; k += 32) sched16[2 * (size_t)k + 1] = 0xFFFFu;
    if (lane == 0) {
      const int na = at_1 - e0, nb = at_2 - e0;
      *reinterpret_cast<int2*>(cnt + 2 * (size_t)r) = make_int2(na, nb);
      if (cnt_kernel) *reinterpret_cast<int2*>(cnt_kernel + 2 * (size_t)r) = make_int2(na | ((qa + 1) << 16), nb | ((qb + 1) << 16));
    }
  }
}

static int check_plan_args(const char* who, int slices, int nbq, int nbk, int overlap, const void* scratch, size_t scratch_bytes,
                           PlanScratch* s) {
  PARO_REQUIRE(slices > 0 && nbq > 0 && nbk > 0, PARO_ESHAPE, "%s: empty mask", who);
  PARO_REQUIRE((int64_t)slices * nbq * nbk < (1ll << 31), PARO_ESHAPE, "%s: mask too large", who);
  PARO_REQUIRE(nbk < 0xFFFF, PARO_ESHAPE, "%s: nbk = %d does not fit 16 bits", who, nbk);
  PARO_REQUIRE(!overlap || nbq < 0xFFFF, PARO_ESHAPE, "%s: nbq = %d does not fit 16 bits", who, nbq);
  *s = plan_scratch(const_cast<void*>(scratch), slices, nbq, nbk, overlap);
  PARO_REQUIRE(scratch && aligned16(scratch) && scratch_bytes >= s->bytes, PARO_ECAP, "%s: scratch too small (%zu < %zu)", who,
               scratch_bytes, s->bytes);
  return PARO_OK;
}

}  // namespace paro

using namespace paro;

extern "C" size_t paro_plan_scratch_bytes(int slices, int nbq, int nbk, int overlap) {
  if (slices <= 0 || nbq <= 0 || nbk <= 0) return 0;
  return plan_scratch(nullptr, slices, nbq, nbk, overlap).bytes;
}

extern "C" int paro_plan_offsets(const uint8_t* mask, int slices, int nbq, int nbk, int overlap, int32_t* row_ptr,
                                 int32_t* pair_ptr, int32_t* pair_q, int32_t* totals, void* scratch, size_t scratch_bytes,
                                 paro_stream_t stream) {
  PARO_REQUIRE(mask && row_ptr && pair_ptr && totals && (!overlap || pair_q), PARO_EINVAL, "paro_plan_offsets: null pointer");
  PARO_REQUIRE(!overlap || aligned8(pair_q), PARO_EALIGN, "paro_plan_offsets: pair_q not 8-byte aligned");
  PlanScratch sc;
  if (int rc = check_plan_args("paro_plan_offsets", slices, nbq, nbk, overlap, scratch, scratch_bytes, &sc)) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const int npairs = (nbq + 1) / 2, rows = slices * nbq, prows = slices * npairs;
  plan_pack_kernel<<<min(8192, (rows + 7) / 8), 256, 0, s>>>(mask, rows, nbk, sc.words, sc.bits, sc.row_cnt);
  PARO_CUDA_OK(cudaMemsetAsync(totals, 0, 4 * sizeof(int32_t), s));
  if (overlap) {
    const int tiles = (nbq + OV_TILE - 1) / OV_TILE;
    PARO_CUDA_OK(cudaFuncSetAttribute(plan_overlap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OV_SMEM));
    plan_overlap_kernel<<<dim3(tiles, tiles, min(slices, 65535)), OV_THREADS, OV_SMEM, s>>>(sc.bits, slices, nbq, sc.words,
                                                                                            sc.pitch, sc.ov, totals + 3);
    int chunk_log = 5;   // two chunks of rows within 200 KB
    while (chunk_log >= 0 && (size_t)sc.pitch * 4 << chunk_log > 200 * 1024) --chunk_log;
    const size_t smem = chunk_log >= 0 ? (size_t)sc.pitch * 4 << chunk_log : 0;
    PARO_CUDA_OK(cudaFuncSetAttribute(plan_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    const int threads = min(PAIR_THREADS, (nbq + 255) / 256 * 32);   // eight rows per thread
    plan_pair_kernel<<<slices, threads, smem, s>>>(sc.ov, nbq, sc.pitch, npairs, chunk_log, pair_q, totals + 2);
  }
  plan_pair_count_kernel<<<min(8192, (prows + 7) / 8), 256, 0, s>>>(sc.bits, sc.row_cnt, nbq, sc.words, npairs, prows,
                                                                    overlap ? pair_q : nullptr, row_ptr, pair_ptr);
  const dim3 scan_grid(sc.scan_blocks, 2);
  plan_scan_sums_kernel<<<scan_grid, 1024, 0, s>>>(row_ptr, pair_ptr, rows, prows, sc.part);
  plan_scan_kernel<<<scan_grid, 1024, 0, s>>>(row_ptr, pair_ptr, rows, prows, sc.part, totals);
  return check_launch("plan_offsets", overlap ? 6 : 4);
}

extern "C" int paro_plan_lists(int slices, int nbq, int nbk, int overlap, const int32_t* row_ptr, const int32_t* pair_ptr,
                               const int32_t* pair_q, int32_t* cols, int32_t* pair_ent, uint32_t* sched, int32_t* sched_cnt,
                               int32_t* sched_cnt_kernel, const void* scratch, size_t scratch_bytes, paro_stream_t stream) {
  PARO_REQUIRE(row_ptr && pair_ptr && cols && pair_ent && sched && sched_cnt && (!overlap || pair_q), PARO_EINVAL,
               "paro_plan_lists: null pointer");
  PARO_REQUIRE(aligned8(sched_cnt) && aligned8(sched_cnt_kernel), PARO_EALIGN,
               "paro_plan_lists: sched_cnt / sched_cnt_kernel not 8-byte aligned");
  PlanScratch sc;
  if (int rc = check_plan_args("paro_plan_lists", slices, nbq, nbk, overlap, scratch, scratch_bytes, &sc)) return rc;
  const int npairs = (nbq + 1) / 2, prows = slices * npairs;
  plan_lists_kernel<<<min(16384, (prows + LIST_WARPS - 1) / LIST_WARPS), 32 * LIST_WARPS, 0, (cudaStream_t)stream>>>(
      sc.bits, nbq, sc.words, npairs, prows, overlap ? pair_q : nullptr, row_ptr, pair_ptr, cols, pair_ent, sched, sched_cnt,
      sched_cnt_kernel);
  return check_launch("plan_lists_kernel");
}
