// Causal flash attention of prompt portions on the 5th-generation tensor cores (head_dim 64 or 128).
//
// Persistent CTAs walk items: 128 consecutive query rows of one request and one query head, over the request's keys in tiles of 128
// ABSOLUTE positions. Every CTA lists the step's (request, query tile) pairs by falling work and takes items in turn; requests of
// few rows cost nothing (a grid over all requests and query tiles spent 130 us on CTAs that only left, beside 60 decoding rows). Roles:
//   softmax warps        a thread owns one query ROW: it reads its row of S from tensor memory (no shuffles for max or sum),
//                        masks on absolute positions, exponentiates in the exp2 domain in fp32, and writes P as bf16 into shared
//                        memory in the swizzled K-major layout the tensor core reads. The output row stays in tensor memory over all
//                        the tiles (the products accumulate); it is in units of 2^m, where m follows the row's maximum
//                        lazily: only a maximum that exceeds m by more than 8 raises it, and only then is the row read, rescaled and
//                        written back;
//   a warp each for Q and K, and for V:  TMA through a ring of their own; a page is one box of the cache's tensor map (128-byte
//                        swizzle, no multicast), a lane holds its number, asked for a tile ahead;
//   MMA warps            tcgen05.mma: S = Q K^T into tensor memory one tile ahead, and, once P is written, O += P V (V is read as
//                        an MN-major operand straight from its [key][d] page layout).
// Because tiles are cut at absolute positions and a row's running max and sum are its own, a row's result does not depend on how the
// prompt was cut or on what else is in the batch. Replaces flash_prefill_mma_kernel of the reference (src/kernels.cuh:1335-1482).
// Every wait is bounded.
//
// head_dim 128 (flash_prefill_tc_kernel): a CTA an SM, with TWO softmax warpgroups that take the tiles in turn, so that one's exponentials run while the
// other reads scores, stores P or waits. A row's maximum goes from tile to tile through shared memory as soon as it is known, its sum when the tile is
// done, and there is one output accumulator an item, whose products are issued in the tiles' order: all sums have the order of one warpgroup that
// walks all tiles, and the same bits (a head of 64 padded with zeros gives what the kernel for 64 gives). Accumulators alternate item by item, so the
// next item's products need not wait until the last one is written, each warpgroup half of its columns. Scores and products have an MMA warp each.
// head_dim 64 (flash_prefill_tc64_kernel): items are short beside their ends, so two CTAs of one softmax warpgroup share an SM, each within
// 113 KB of shared memory, 256 columns of tensor memory and 128 registers (a row of S is read in two halves of 64, the first one twice:
// once for the maximum, once for the exponentials).
//
// What bounds it: the softmax warps, some 2,500 cycles a tile of a warpgroup alone, 1,024 of them exponentials (16 a cycle an SM, so two
// cannot fall below 1,024 cycles a tile; the MMAs take 900 to 1,250). Measured against its forerunner (a CTA per query tile of a grid over
// all requests, one warpgroup, MMAs issued behind "lane == 0", page numbers loaded when they were needed), us: 32 heads over 8 of 128, 2,048
// rows 74.7 -> 52, behind 2,048 more 182 -> 115 (900 TFLOP/s); 24 heads of 128, 512 rows behind 1,536 34.9 -> 24.4, with bias and sink 58 -> 40; 32 heads over 8 of
// 64, 2,048 rows 40.7 -> 40.0, four portions of 512 23.9 -> 20.4, 1,988 rows beside 60 decoding requests 173 -> 39.7. With two chains of their own (a
// maximum, sum and accumulator for the even tiles and for the odd ones, joined at the item's end) the 128 kernel was 1 to 8 % faster (behind 2,048 113 us,
// 512 behind 1,536 22.6), but every result differed in its last bits from one chain's. At head_dim 64 that form was slower (45 us at 2,048 rows: an item of 8.5 tiles
// spends a third of its time at its ends), and so was one that joined the chains later, behind the next item's first tile (49 us).
//
// EX: a distance bias, r1 ln(1 + r2 (i - j)) off the score of query i and key j (r1, r2 >= 0, a number per head), and a
// sink, exp(sink) in the denominator (a number per head). The bias grows with the distance, so the unbiased maximum of a
// tile less the bias of its nearest key bounds the tile's scores from above; that bound takes the maximum's place (any
// reference value gives the same quotient; the caller keeps the bias's spread within a tile far from the exponent's range),
// and a score meets its bias once, in the exponent.
#include "tc_common.cuh"

constexpr int FT_BM = 128, FT_BN = 128;
constexpr int FT_TILE = 128 * 64 * 2;  // one [128][64] bf16 tile: 16 KB; a [128][head_dim] operand is head_dim / 64 of them, 64 columns each
constexpr int FT_THREADS = 384;        // 168 registers each: a row of S is 128 of them
// A launch lists up to FT_MAX_PAIRS (request, query tile) pairs, in the place of P, and a CTA keeps the pairs of its own items, FT_OWN at most; the
// launcher cuts steps of more. (When every CTA kept all pairs, 200 of them at head_dim 64, one request of 32,768 rows was 43 launches and took
// 10.8 ms, now 6.7; 16,000 rows beside 300 single rows 3.1 ms, now 1.6.)
constexpr int FT_MAX_PAIRS = 4096, FT_OWN = 420, FT_OWN64 = 200;

// MN-major operand with the 128-byte swizzle: 64 contiguous elements of the MN dimension per row,
// eight K rows per 1,024-byte group (stride SBO); further MN atoms would lie LBO apart (one here).
__device__ __forceinline__ uint64_t ft_desc_mn128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(FT_TILE >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::f16 instruction descriptor as hb_umma_idesc_bf16, with B read MN-major.
__host__ __device__ constexpr uint32_t ft_idesc_b_mn(int M, int N) { return hb_umma_idesc_bf16(M, N) | (1u << 16); }

__device__ __forceinline__ uint64_t ft_pack2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void ft_unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t ft_fma2(uint64_t a, uint64_t b, uint64_t c) {   // two fmaf, each rounded by itself
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t ft_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// 32 columns of this thread's lane, not waited for (see hb_tmem_ld64_nowait), and back.
__device__ __forceinline__ void ft_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]) : "r"(taddr));
}
__device__ __forceinline__ void ft_ld32_fence(uint32_t* r) { asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]) :: "memory"); }
__device__ __forceinline__ void ft_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}

// head_dim 128: Q, P of both warpgroups, rings of two K and two V tiles, and the list of the items.
struct FtBars {
  uint64_t q_full, q_free, k_full[2], k_free[2], v_full[2], v_free[2], s_full[2], s_free[2], p_full[2], pv_done[2], o_free[2];
  uint64_t m_full[2][4], l_full[2][4];   // a warp's rows have their maximum, and their sum, behind its tile
  float m[128], l[128];                  // a row's running maximum and sum, handed from tile to tile
  uint32_t own[FT_OWN];              // request << 16 | query tile of this CTA's items, in their order
  int n_entries;
  uint32_t tmem_slot;
  int abort_flag;
};
constexpr int FT_SMEM = 14 * FT_TILE + (int)sizeof(FtBars);
// head_dim 64: Q, P, rings of two K and two V tiles.
struct FtBars64 {
  uint64_t q_full, q_free, k_full[2], k_free[2], v_full[2], v_free[2], s_full, s_free, p_full, pv_done;
  uint32_t own[FT_OWN64];
  int n_entries;
  uint32_t tmem_slot;
  int abort_flag;
};
constexpr int FT_SMEM64 = 7 * FT_TILE + (int)sizeof(FtBars64);
static_assert(FT_SMEM <= 227 * 1024 && 2 * (FT_SMEM64 + 1024) <= 228 * 1024, "shared memory of one block and of two");
static_assert(FT_MAX_PAIRS * sizeof(uint2) <= 2 * FT_TILE, "the unordered pairs lie where P will");

// Item k of this CTA: CTAs take the items in turn, back and forth (the items come by falling work).
__device__ __forceinline__ int ft_item(int k) { return k * (int)gridDim.x + ((k & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x); }

// (first row, rows, position of the first row, request) of a (request, query tile) pair.
__device__ __forceinline__ int4 ft_entry(uint32_t e, const int* q_start, const int* q_len, const int* ctx_len) {
  const int r = e >> 16, row = (int)(e & 0xffffu) * FT_BM;
  return make_int4(q_start[r] + row, min(FT_BM, q_len[r] - row), ctx_len[r] + row, r);
}
// Key tiles of an item: the first and how many.
struct FtSpan { int kt_lo, n, lo, p_last; };
__device__ __forceinline__ FtSpan ft_span(const int4& e, int window) {
  FtSpan s;
  s.p_last = e.z + e.y - 1;
  s.lo = window > 0 ? max(0, e.z - window + 1) : 0;
  s.kt_lo = s.lo / FT_BN;
  s.n = s.p_last / FT_BN - s.kt_lo + 1;
  return s;
}

// One warp: the (request, query tile) pairs of this launch and their key tiles, unordered. The numbers of 128 requests are asked for together: one
// trip to memory after another, a step of 64 requests took 0.7 us longer (portions of 16 rows, 4 heads of 64: 9.0 us, now 8.3; a block per query tile 7.6).
__device__ __forceinline__ void ft_list(uint2* raw, int* n_entries, int most, const int* q_len, const int* ctx_len, int window, int min_rows,
                                        int req0, int reqs, int qt0, int qts) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int base = 0; base < reqs; base += 128) {
    int q_lens[4], ctxs[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = base + 32 * j + lane;
      q_lens[j] = i < reqs ? q_len[req0 + i] : 0;
      ctxs[j] = i < reqs ? ctx_len[req0 + i] : 0;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (base + 32 * j >= reqs) break;
      const int r = req0 + base + 32 * j + lane, len = q_lens[j] < min_rows ? 0 : q_lens[j], ctx = ctxs[j];
      const int tiles = max(0, min((len + FT_BM - 1) / FT_BM - qt0, qts));
      int at = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
      }
      const int total = __shfl_sync(0xffffffffu, at, 31);
      at += n - tiles;
      for (int t = 0; t < tiles && at + t < most; t++) {
        const int row = (qt0 + t) * FT_BM;
        raw[at + t] = make_uint2((uint32_t)r << 16 | (uint32_t)(qt0 + t), ft_span(make_int4(0, min(FT_BM, len - row), ctx + row, r), window).n);
      }
      n += total;
    }
  }
  if (lane == 0) *n_entries = min(n, most);
}
// All threads: the pairs by falling work; a pair's place is the number of pairs with more key tiles to walk, its items are Hq in a row from place *
// Hq on, and those of them that are this CTA's are kept (at most one in gridDim.x items).
__device__ __forceinline__ void ft_sort(const uint2* raw, uint32_t* own, int n_entries, int Hq) {
  for (int i = threadIdx.x; i < n_entries; i += blockDim.x) {
    const uint2 e = raw[i];
    int place = 0;
    for (int j = 0; j < n_entries; j++) {
      const uint32_t w = raw[j].y;
      place += w > e.y || (w == e.y && j < i);
    }
    const int u0 = place * Hq, u1 = u0 + Hq;
    for (int k = u0 / (int)gridDim.x; k * (int)gridDim.x < u1; k++) {
      const int u = ft_item(k);
      if (u >= u0 && u < u1) own[k] = e.x;
    }
  }
}
// The loader of K or V: a warp brings the tiles of an item, page by page, through a ring of two; lane l holds the page of a tile's place l. The
// places behind the item's last page, and ahead of a window's first, have none. `fill` (V): they get boxes beyond the cache, which
// arrive as zeros, since P is 0 there and 0 times what an earlier item left (another request's, perhaps an infinity or NaN) need not be 0. K
// leaves them as they are: their scores are masked, whatever they are.
template <int FT_D>
__device__ __forceinline__ bool ft_bring(const FtSpan& sp, const int* table, int page_size, int Hkv, int h, bool fill, const CUtensorMap* map, uint8_t* ring,
                                         uint64_t* full, uint64_t* free, uint32_t& it, volatile int* abort_flag) {
  constexpr int NH = FT_D / 64, OPND = NH * FT_TILE;
  const int lane = threadIdx.x & 31, places = FT_BN / page_size, first = sp.lo / page_size, last = sp.p_last / page_size;
  // the page of this lane's place in tile t, asked for one tile ahead
  auto page = [&](int t) {
    const int pg = (sp.kt_lo + t) * places + lane;
    return lane < places && pg >= first && pg <= last ? table[pg] : -1;
  };
  int next = page(0);
  for (int t = 0; t < sp.n; t++, it++) {
    const uint32_t s = it & 1, ph = (it >> 1) & 1;
    const uint32_t boxes = __ballot_sync(0xffffffffu, lane < places && (fill || next >= 0));
    const int row = next >= 0 ? (next * Hkv + h) * page_size : -page_size;
    next = t + 1 < sp.n ? page(t + 1) : 0;
    if (!__all_sync(0xffffffffu, hb_mbar_wait(&free[s], ph ^ 1, abort_flag))) return false;
    if (hb_elect()) hb_mbar_expect_tx(&full[s], (uint32_t)__popc(boxes) * page_size * FT_D * 2);
    __syncwarp();
    for (int p = 0; p < places; p += 4) {       // four boxes an election (pages of 8 one by one: 2,048 rows behind 2,048 106 us, now 102)
      int from[4];
#pragma unroll
      for (int j = 0; j < 4; j++) from[j] = __shfl_sync(0xffffffffu, row, p + j);
      if (hb_elect()) {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (boxes >> (p + j) & 1) {
            uint8_t* dst = ring + s * OPND + (p + j) * page_size * 128;            // rows of 128 bytes in each 64-column tile
#pragma unroll
            for (int hf = 0; hf < NH; hf++) hb_tma_load_2d(dst + hf * FT_TILE, map, &full[s], hf * 64, from[j]);
          }
      }
      __syncwarp();
    }
  }
  return true;
}
// The exponentials of two scores.
template <bool EX>
__device__ __forceinline__ void ft_exp(uint32_t s0, uint32_t s1, uint64_t scale2, uint64_t sub2, float r1, float r2, float dist, float& p0, float& p1) {
  float e0, e1;
  ft_unpack2(ft_fma2(ft_pack2(s0, s1), scale2, sub2), e0, e1);
  if (EX) {   // (a key behind the row is masked: any finite bias will do)
    e0 = fmaf(-r1, __log2f(fmaxf(fmaf(r2, dist, 1.f), 1.f)), e0);
    e1 = fmaf(-r1, __log2f(fmaxf(fmaf(r2, dist - 1.f, 1.f), 1.f)), e1);
  }
  p0 = hb_exp2(e0);
  p1 = hb_exp2(e1);
}
// m_run follows the row's maximum lazily: it is raised (and the row of O rescaled) only when a tile's maximum exceeds it by
// more than FT_SLACK, so P <= 2^FT_SLACK; the sum l_run is in the same units, and O / l_run is exact whichever maxima were used.
constexpr float FT_SLACK = 8.f;

template <bool EX>
__global__ void __launch_bounds__(FT_THREADS, 1) flash_prefill_tc_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const int* __restrict__ bt, int bt_stride, const int* __restrict__ q_start,
    const int* __restrict__ q_len, const int* __restrict__ ctx_len, __nv_bfloat16* __restrict__ out, int Hq, int Hkv,
    int page_size, int window, float scale_log2, int min_rows, int* status, const float* __restrict__ r1p,
    const float* __restrict__ r2p, const float* __restrict__ sink, int req0, int reqs, int qt0, int qts, int most) {
  constexpr int FT_D = 128, NH = FT_D / 64, OPND = NH * FT_TILE;
  // the 128-byte swizzle wants the tiles on 1 KB boundaries, and there is no room for slack: checked below
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                      // [128][head_dim]
  uint8_t* sP = sQ + OPND;                 // per warpgroup two K blocks of [128 rows][64 keys]
  uint8_t* sK = sP + 4 * FT_TILE;          // two stages of [128 keys][head_dim]
  uint8_t* sV = sK + 2 * OPND;             // and two more
  FtBars* bar = (FtBars*)(sV + 2 * OPND);
  volatile int* abort_flag = &bar->abort_flag;

  // the step's own metadata (lengths, tables) was copied before the step's first kernel began; everything else
  // that an earlier kernel wrote is read after hb_pdl_wait() below
  hb_pdl_launch();
  if (hb_smem_u32(smem) & 1023) {   // never seen; the tiles would not be where the tensor core expects them
    if (threadIdx.x == 0) atomicExch(status, 1);
    hb_pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) ft_list((uint2*)sP, &bar->n_entries, most, q_len, ctx_len, window, min_rows, req0, reqs, qt0, qts);
  if (threadIdx.x == 32) {
    hb_mbar_init(&bar->q_full, 1); hb_mbar_init(&bar->q_free, 1);
    for (int b = 0; b < 2; b++) {
      hb_mbar_init(&bar->k_full[b], 1); hb_mbar_init(&bar->k_free[b], 1);
      hb_mbar_init(&bar->v_full[b], 1); hb_mbar_init(&bar->v_free[b], 1);
    }
    for (int c = 0; c < 2; c++) {
      hb_mbar_init(&bar->s_full[c], 1); hb_mbar_init(&bar->s_free[c], 4);
      hb_mbar_init(&bar->p_full[c], 4); hb_mbar_init(&bar->pv_done[c], 1);
      hb_mbar_init(&bar->o_free[c], 8);
      for (int w = 0; w < 4; w++) { hb_mbar_init(&bar->m_full[c][w], 1); hb_mbar_init(&bar->l_full[c][w], 1); }
    }
    bar->abort_flag = 0;
    hb_fence_barrier_init();
  }
  if (warp == 8 && lane == 0) { hb_tma_prefetch_desc(&map_q); hb_tma_prefetch_desc(&map_k); hb_tma_prefetch_desc(&map_v); }
  __syncthreads();
  const int n_entries = bar->n_entries, n_items = n_entries * Hq;
  if ((int)blockIdx.x >= n_items) {   // the grid is made for the most items there can be
    hb_pdl_wait();
    return;
  }
  ft_sort((const uint2*)sP, bar->own, n_entries, Hq);
  if (warp == 10) {
    hb_tmem_alloc(&bar->tmem_slot, 512);
    hb_tmem_relinquish();
  }
  hb_tc_fence_before();
  __syncthreads();
  hb_tc_fence_after();
  const uint32_t tmem = bar->tmem_slot;   // S of warpgroup c: 128 columns at c * 128; O of the CTA's item k: head_dim columns at 256 + (k & 1) * 128
  hb_pdl_wait();   // barriers, shared and tensor memory were set up while the kernel ahead was still running

  // an item's numbers are fetched while the one before it is worked on
  auto entry = [&](int k) { const int u = ft_item(k); return ft_entry(bar->own[u < n_items ? k : 0], q_start, q_len, ctx_len); };

  // The CTA's tiles are numbered through all its items: tile t has warpgroup, S, P and ring stages t & 1, and is their use t >> 1. A barrier is
  // waited for use after use by one warp, or behind another's word that the use before is over, so a parity can only mean the use that is wanted.
  if (warp == 8 || warp == 9) {  // ---------------- TMA: lane l brings page l of a tile
    const bool is_k = warp == 8;
    const CUtensorMap* map = is_k ? &map_k : &map_v;
    uint64_t *full = is_k ? bar->k_full : bar->v_full, *free = is_k ? bar->k_free : bar->v_free;
    uint8_t* ring = is_k ? sK : sV;
    uint32_t it = 0;
    bool ok = true;
    int4 ahead = entry(0);
    for (int k = 0, u; (u = ft_item(k)) < n_items && ok; k++) {
      const int4 e = ahead;
      ahead = entry(k + 1);
      const int hq = u % Hq, h = hq / (Hq / Hkv);
      const FtSpan sp = ft_span(e, window);
      if (is_k) {
        if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->q_free, (k & 1) ^ 1, abort_flag))) break;
        if (hb_elect()) {
          hb_mbar_expect_tx(&bar->q_full, OPND);
#pragma unroll
          for (int hf = 0; hf < NH; hf++) hb_tma_load_2d(sQ + hf * FT_TILE, &map_q, &bar->q_full, hq * FT_D + hf * 64, e.x);
        }
        __syncwarp();
      }
      ok = ft_bring<FT_D>(sp, bt + (size_t)e.w * bt_stride, page_size, Hkv, h, !is_k, map, ring, full, free, it, abort_flag);
    }
  } else if (warp == 10) {  // ---------------- tensor cores: S = Q K^T of every tile
    if (hb_elect()) {
      constexpr uint32_t idesc = hb_umma_idesc_bf16(FT_BM, FT_BN);
      uint32_t t = 0;
      bool ok = true;
      int4 ahead = entry(0);
      for (int k = 0; ft_item(k) < n_items && ok; k++) {
        const int n = ft_span(ahead, window).n;
        ahead = entry(k + 1);
        ok = hb_mbar_wait(&bar->q_full, k & 1, abort_flag);
        for (int i = 0; i < n && ok; i++, t++) {
          const uint32_t c = t & 1, ph = (t >> 1) & 1;
          ok = hb_mbar_wait(&bar->k_full[c], ph, abort_flag) && hb_mbar_wait(&bar->s_free[c], ph ^ 1, abort_flag);
          if (!ok) break;
          hb_tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < FT_D / 16; kk++) {   // 16 columns a step: four steps in each 64-column tile
            const uint64_t dq = hb_umma_desc_k128(hb_smem_u32(sQ + (kk >> 2) * FT_TILE)) + 2 * (kk & 3);
            const uint64_t dk = hb_umma_desc_k128(hb_smem_u32(sK + c * OPND + (kk >> 2) * FT_TILE)) + 2 * (kk & 3);
            hb_umma_bf16(tmem + c * FT_BN, dq, dk, idesc, kk != 0);
          }
          hb_umma_commit(&bar->s_full[c]);
          hb_umma_commit(&bar->k_free[c]);
          if (i == n - 1) hb_umma_commit(&bar->q_free);
        }
      }
    }
  } else if (warp == 11) {  // ---------------- tensor cores: O += P V, tile after tile
    if (hb_elect()) {
      constexpr uint32_t idesc = ft_idesc_b_mn(FT_BM, FT_D);
      uint32_t t = 0;
      bool ok = true;
      int4 ahead = entry(0);
      for (int k = 0; ft_item(k) < n_items && ok; k++) {
        const int n = ft_span(ahead, window).n;
        ahead = entry(k + 1);
        ok = hb_mbar_wait(&bar->o_free[k & 1], ((k >> 1) & 1) ^ 1, abort_flag);     // the item before the last one is written
        for (int i = 0; i < n && ok; i++, t++) {
          const uint32_t c = t & 1, ph = (t >> 1) & 1;
          ok = hb_mbar_wait(&bar->v_full[c], ph, abort_flag) && hb_mbar_wait(&bar->p_full[c], ph, abort_flag);
          if (!ok) break;
          hb_tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < FT_BN / 16; kk++) {
            const uint64_t dp = hb_umma_desc_k128(hb_smem_u32(sP + (2 * c + (kk >> 2)) * FT_TILE)) + 2 * (kk & 3);
            const uint64_t dv = ft_desc_mn128(hb_smem_u32(sV + c * OPND + kk * 16 * 128));   // 16 keys on; the second 64 columns lie FT_TILE further (the descriptor's leading offset)
            hb_umma_bf16(tmem + 256 + (k & 1) * 128, dp, dv, idesc, i > 0 || kk != 0);      // O stays in tensor memory over the item's tiles
          }
          hb_umma_commit(&bar->v_free[c]);
          hb_umma_commit(&bar->pv_done[c]);
        }
      }
    }
  } else {  // ---------------- softmax: warpgroup c has every second tile; thread = query row
    const int c = warp >> 2, w = warp & 3, r = threadIdx.x & 127;
    const uint32_t lane_base = (uint32_t)(w * 32) << 16, tmem_s = tmem + c * FT_BN + lane_base;
    uint32_t t0 = 0;       // the item's first tile
    bool ok = true;        // every wait's outcome is made uniform over the warp: the tensor-memory accesses below are warp-wide
    auto wait = [&](uint64_t* b, uint32_t parity) { ok = __all_sync(0xffffffffu, hb_mbar_wait(b, parity, abort_flag)); return ok; };
    int4 ahead = entry(0);
    for (int k = 0, u; (u = ft_item(k)) < n_items && ok; k++) {
      const int4 e = ahead;
      ahead = entry(k + 1);
      const int hq = u % Hq;
      const FtSpan sp = ft_span(e, window);
      const int qp = e.z + min(r, e.y - 1);      // rows past the portion's end are computed, never stored
      const float r1 = EX && r1p ? r1p[hq] : 0.f, r2 = EX && r1p ? r2p[hq] : 0.f;
      const uint32_t tmem_o = tmem + 256 + (k & 1) * 128 + lane_base;
      float m_run = -INFINITY, l_run = 0.f;
      for (int i = (t0 ^ c) & 1; i < sp.n; i += 2) {
        const uint32_t t = t0 + i, ph = (t >> 1) & 1, ph_before = ((t - 1) >> 1) & 1;     // this tile's use, and that of the tile before
        const int k_base = (sp.kt_lo + i) * FT_BN;
        const bool need_mask = k_base + FT_BN - 1 > e.z || (window > 0 && k_base < sp.p_last - window + 1);
        if (!wait(&bar->s_full[c], ph)) break;
        hb_tc_fence_after();
        // a row of S in one read; in two with a bias (EX), whose chains are longer and want registers of their own: the second half stays, the first is read again
        constexpr int H = EX ? 64 : 128;
        uint32_t sr[H];
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        const int hi_j = qp - k_base, lo_j = window > 0 ? qp - window - k_base : -1;  // key j of the tile is visible iff lo_j < j <= hi_j
        auto read = [&](int at) {
#pragma unroll
          for (int q = 0; q < H; q += 32) ft_ld32(tmem_s + at + q, sr + q);
          hb_tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < H; q += 32) ft_ld32_fence(sr + q);
        };
        auto mask = [&](int at) {
          if (need_mask) {
#pragma unroll
            for (int j = 0; j < H; j++)
              if (!(j + at <= hi_j && j + at > lo_j)) sr[j] = __float_as_uint(-INFINITY);
          }
        };
        auto free_s = [&] {        // the scores of the warpgroup's next tile may overwrite S
          hb_tc_fence_before();
          __syncwarp();
          if (lane == 0) hb_mbar_arrive(&bar->s_free[c]);
        };
#pragma unroll
        for (int at = 0; at < 128; at += H) {
          read(at);
          if (!EX) free_s();
          mask(at);
#pragma unroll
          for (int j = 0; j < H; j += 2) mx[(j >> 1) & 3] = fmaxf(fmaxf(mx[(j >> 1) & 3], __uint_as_float(sr[j])), __uint_as_float(sr[j + 1]));
        }
        float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;
        const float dist0 = (float)(qp - k_base);                     // of the tile's first key
        if (EX) m_tile -= r1 * __log2f(fmaf(r2, fmaxf(dist0 - (FT_BN - 1), 0.f), 1.f));
        if (i > 0) {       // the maximum so far, from the other warpgroup's tile
          if (!wait(&bar->m_full[c ^ 1][w], ph_before)) break;
          m_run = bar->m[r];
        }
        const bool grow = m_tile > m_run + FT_SLACK;   // also the first tile with a visible key: m_run is -inf
        float corr = 1.f;
        if (grow) {
          corr = hb_exp2(m_run - m_tile);   // 0 while nothing has been summed
          m_run = m_tile;
        }
        bar->m[r] = m_run;
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->m_full[c][w]);
        const float sub = m_run == -INFINITY ? 0.f : m_run;
        const uint64_t scale2 = ft_pack2(__float_as_uint(scale_log2), __float_as_uint(scale_log2)), sub2 = ft_pack2(__float_as_uint(-sub), __float_as_uint(-sub));
        uint64_t sum2[2] = {0ull, 0ull};   // four sums of pairs, of keys 64-127 first (the order that one warpgroup with half a row in registers has)
#pragma unroll
        for (int hh = 1; hh >= 0; hh--) {
          if (EX && hh == 0) {
            read(0);
            free_s();
            mask(0);
          }
          uint32_t* x = sr + (EX ? 0 : hh * 64);
#pragma unroll
          for (int j = 0; j < 64; j += 4) {  // masked scores are -inf: 2^-inf = 0
            float p0, p1, p2, p3;
            ft_exp<EX>(x[j], x[j + 1], scale2, sub2, r1, r2, dist0 - (float)(j + hh * 64), p0, p1);
            ft_exp<EX>(x[j + 2], x[j + 3], scale2, sub2, r1, r2, dist0 - (float)(j + 2 + hh * 64), p2, p3);
            sum2[(j >> 2) & 1] = ft_add2(sum2[(j >> 2) & 1], ft_pack2(__float_as_uint(p0 + p1), __float_as_uint(p2 + p3)));
            x[j >> 1] = hb_pack_bf16(p0, p1);
            x[(j >> 1) + 1] = hb_pack_bf16(p2, p3);
          }
          // (without a bias the exponentials of the whole row come first: half by half they were 10 % slower)
          if (EX || hh == 0) {
            // the product of the tile two before has read P
            if ((!EX || hh == 1) && t >= 2 && !wait(&bar->pv_done[c], ph ^ 1)) break;
            // 64 keys = eight 16-byte chunks of this row in K block hh of P
#pragma unroll
            for (int cc = EX ? hh * 8 : 0; cc < (EX ? hh * 8 + 8 : 16); cc++) {
              const uint32_t dst = hb_smem_u32(sP + (2 * c + (cc >> 3)) * FT_TILE) + r * 128 + (((cc & 7) ^ (r & 7)) << 4);
              const uint32_t* y = sr + (EX ? 0 : (cc >> 3) * 64) + 4 * (cc & 7);
              asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]) : "memory");
            }
          }
        }
        if (!ok) break;
        if (i > 0) {       // the sum so far
          if (!wait(&bar->l_full[c ^ 1][w], ph_before)) break;
          l_run = bar->l[r];
        }
        float s0, s1, s2, s3;
        ft_unpack2(sum2[0], s0, s1);
        ft_unpack2(sum2[1], s2, s3);
        l_run = l_run * corr + ((s0 + s1) + (s2 + s3));
        bar->l[r] = l_run;
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->l_full[c][w]);
        if (i > 0 && __any_sync(0xffffffffu, grow)) {   // a raised maximum: the rows of O so far, when the product of the tile before has written them
          if (!wait(&bar->pv_done[c ^ 1], ph_before)) break;   // (its warpgroup's sum came behind the use before)
          hb_tc_fence_after();
#pragma unroll
          for (int q = 0; q < FT_D / 32; q++) {
            uint32_t o[32];
            ft_ld32(tmem_o + q * 32, o);
            hb_tmem_ld_wait();
            ft_ld32_fence(o);
#pragma unroll
            for (int d = 0; d < 32; d++) o[d] = __float_as_uint(__uint_as_float(o[d]) * corr);
            ft_st32(tmem_o + q * 32, o);
          }
          hb_tmem_st_wait();
        }
        hb_tc_fence_before();
        hb_fence_proxy_async();
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->p_full[c]);
      }
      // ---- the item's end: each warpgroup writes half of the columns; the next item's products go to the other accumulator
      const uint32_t last = t0 + sp.n - 1, cl = last & 1, ph_last = (last >> 1) & 1;
      t0 += sp.n;
      if (ok && cl != c && wait(&bar->m_full[cl][w], ph_last) && wait(&bar->l_full[cl][w], ph_last)) {
        m_run = bar->m[r];
        l_run = bar->l[r];
      }
      if (ok && wait(&bar->pv_done[cl], ph_last)) {
        hb_tc_fence_after();
        if (EX && sink) l_run += hb_exp2(fmaf(sink[hq], 1.4426950408889634f, -m_run));
        const float inv = 1.f / l_run;
        constexpr int HC = FT_D / 2;                                 // this warpgroup's columns: c * HC ..
        uint32_t o[HC];
        hb_tmem_ld64_nowait(tmem_o + c * HC, o);
        hb_tmem_ld_wait();
        hb_tmem_ld_fence64(o);
        hb_tc_fence_before();
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->o_free[k & 1]);
        if (r < e.y) {
          __nv_bfloat16* dst = out + ((size_t)(e.x + r) * Hq + hq) * FT_D + c * HC;
#pragma unroll
          for (int d = 0; d < HC; d += 8) {
            uint4 v;
            v.x = hb_pack_bf16(__uint_as_float(o[d]) * inv, __uint_as_float(o[d + 1]) * inv);
            v.y = hb_pack_bf16(__uint_as_float(o[d + 2]) * inv, __uint_as_float(o[d + 3]) * inv);
            v.z = hb_pack_bf16(__uint_as_float(o[d + 4]) * inv, __uint_as_float(o[d + 5]) * inv);
            v.w = hb_pack_bf16(__uint_as_float(o[d + 6]) * inv, __uint_as_float(o[d + 7]) * inv);
            *(uint4*)(dst + d) = v;
          }
        }
      }
    }
  }

  hb_tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    __nanosleep(100000);
  }
  if (warp == 10) {
    __syncwarp();
    hb_tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------
// head_dim 64: one chain, two CTAs an SM.
// ---------------------------------------------------------------------------------------
template <bool EX>
__global__ void __launch_bounds__(256, 2) flash_prefill_tc64_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const int* __restrict__ bt, int bt_stride, const int* __restrict__ q_start,
    const int* __restrict__ q_len, const int* __restrict__ ctx_len, __nv_bfloat16* __restrict__ out, int Hq, int Hkv,
    int page_size, int window, float scale_log2, int min_rows, int* status, const float* __restrict__ r1p,
    const float* __restrict__ r2p, const float* __restrict__ sink, int req0, int reqs, int qt0, int qts, int most) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                 // [128][64]
  uint8_t* sP = sQ + FT_TILE;         // two K blocks of [128 rows][64 keys]
  uint8_t* sK = sP + 2 * FT_TILE;     // two stages of [128 keys][64]
  uint8_t* sV = sK + 2 * FT_TILE;     // and two more
  FtBars64* bar = (FtBars64*)(sV + 2 * FT_TILE);
  volatile int* abort_flag = &bar->abort_flag;

  hb_pdl_launch();
  if (hb_smem_u32(smem) & 1023) {   // as above
    if (threadIdx.x == 0) atomicExch(status, 1);
    hb_pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) ft_list((uint2*)sP, &bar->n_entries, most, q_len, ctx_len, window, min_rows, req0, reqs, qt0, qts);
  if (threadIdx.x == 32) {
    hb_mbar_init(&bar->q_full, 1); hb_mbar_init(&bar->q_free, 1);
    for (int b = 0; b < 2; b++) {
      hb_mbar_init(&bar->k_full[b], 1); hb_mbar_init(&bar->k_free[b], 1);
      hb_mbar_init(&bar->v_full[b], 1); hb_mbar_init(&bar->v_free[b], 1);
    }
    hb_mbar_init(&bar->s_full, 1); hb_mbar_init(&bar->s_free, 4);
    hb_mbar_init(&bar->p_full, 4); hb_mbar_init(&bar->pv_done, 1);
    bar->abort_flag = 0;
    hb_fence_barrier_init();
  }
  if (warp == 4 && lane == 0) { hb_tma_prefetch_desc(&map_q); hb_tma_prefetch_desc(&map_k); hb_tma_prefetch_desc(&map_v); }
  __syncthreads();
  const int n_entries = bar->n_entries, n_items = n_entries * Hq;
  if ((int)blockIdx.x >= n_items) {
    hb_pdl_wait();
    return;
  }
  ft_sort((const uint2*)sP, bar->own, n_entries, Hq);
  if (warp == 6) {
    hb_tmem_alloc(&bar->tmem_slot, 256);
    hb_tmem_relinquish();
  }
  hb_tc_fence_before();
  __syncthreads();
  hb_tc_fence_after();
  const uint32_t tmem_s = bar->tmem_slot, tmem_o = tmem_s + FT_BN;  // S: 128 columns, O: 64 columns
  hb_pdl_wait();

  auto entry = [&](int k) { const int u = ft_item(k); return ft_entry(bar->own[u < n_items ? k : 0], q_start, q_len, ctx_len); };
  if (warp == 4 || warp == 5) {  // ---------------- TMA
    const bool is_k = warp == 4;
    uint32_t it = 0;
    bool ok = true;
    int4 ahead = entry(0);
    for (int k = 0, u; (u = ft_item(k)) < n_items && ok; k++) {
      const int4 e = ahead;
      ahead = entry(k + 1);
      const int hq = u % Hq, h = hq / (Hq / Hkv);
      if (is_k) {
        if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->q_free, (k & 1) ^ 1, abort_flag))) break;
        if (hb_elect()) {
          hb_mbar_expect_tx(&bar->q_full, FT_TILE);
          hb_tma_load_2d(sQ, &map_q, &bar->q_full, hq * 64, e.x);
        }
        __syncwarp();
      }
      ok = ft_bring<64>(ft_span(e, window), bt + (size_t)e.w * bt_stride, page_size, Hkv, h, !is_k, is_k ? &map_k : &map_v, is_k ? sK : sV,
                        is_k ? bar->k_full : bar->v_full, is_k ? bar->k_free : bar->v_free, it, abort_flag);
    }
  } else if (warp == 6) {  // ---------------- tensor cores: S_i is issued before O_{i-1}, so it overlaps the softmax of tile i - 1
    constexpr uint32_t idesc_s = hb_umma_idesc_bf16(FT_BM, FT_BN), idesc_o = ft_idesc_b_mn(FT_BM, 64);
    uint32_t base = 0;      // tiles of the items before
    bool ok = true;
    int4 ahead = entry(0);
    for (int k = 0; ft_item(k) < n_items && ok; k++) {
      const int n = ft_span(ahead, window).n;
      ahead = entry(k + 1);
      ok = __all_sync(0xffffffffu, hb_mbar_wait(&bar->q_full, k & 1, abort_flag));
      for (int i = 0; i <= n && ok; i++) {
        if (i < n) {
          const uint32_t it = base + i, s = it & 1, ph = (it >> 1) & 1;
          ok = hb_mbar_wait(&bar->k_full[s], ph, abort_flag) && hb_mbar_wait(&bar->s_free, (it & 1) ^ 1, abort_flag);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          hb_tc_fence_after();
          if (hb_elect()) {
            const uint64_t dq = hb_umma_desc_k128(hb_smem_u32(sQ)), dk = hb_umma_desc_k128(hb_smem_u32(sK + s * FT_TILE));
#pragma unroll
            for (int kk = 0; kk < 4; kk++) hb_umma_bf16(tmem_s, dq + 2 * kk, dk + 2 * kk, idesc_s, kk != 0);
            hb_umma_commit(&bar->s_full);
            hb_umma_commit(&bar->k_free[s]);
            if (i == n - 1) hb_umma_commit(&bar->q_free);
          }
          __syncwarp();
        }
        if (i > 0) {
          const uint32_t it = base + i - 1, s = it & 1, ph = (it >> 1) & 1;
          ok = hb_mbar_wait(&bar->v_full[s], ph, abort_flag) && hb_mbar_wait(&bar->p_full, it & 1, abort_flag);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          hb_tc_fence_after();
          if (hb_elect()) {
#pragma unroll
            for (int kk = 0; kk < FT_BN / 16; kk++) {
              const uint64_t dp = hb_umma_desc_k128(hb_smem_u32(sP + (kk >> 2) * FT_TILE)) + 2 * (kk & 3);
              const uint64_t dv = ft_desc_mn128(hb_smem_u32(sV + s * FT_TILE + kk * 16 * 128));   // 16 keys on
              hb_umma_bf16(tmem_o, dp, dv, idesc_o, i > 1 || kk != 0);
            }
            hb_umma_commit(&bar->v_free[s]);
            hb_umma_commit(&bar->pv_done);
          }
          __syncwarp();
        }
      }
      base += n;
    }
  } else if (warp < 4) {  // ---------------- softmax: thread = query row
    const int r = threadIdx.x;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    uint32_t cnt = 0;      // tiles so far, over all items
    bool ok = true;        // every wait's outcome is made uniform over the warp
    int4 ahead = entry(0);
    for (int k = 0, u; (u = ft_item(k)) < n_items && ok; k++) {
      const int4 e = ahead;
      ahead = entry(k + 1);
      const int hq = u % Hq;
      const FtSpan sp = ft_span(e, window);
      const int qp = e.z + min(r, e.y - 1);      // rows past the portion's end are computed, never stored
      const float r1 = EX && r1p ? r1p[hq] : 0.f, r2 = EX && r1p ? r2p[hq] : 0.f;
      float m_run = -INFINITY, l_run = 0.f;
      for (int i = 0; i < sp.n && ok; i++, cnt++) {
        const int k_base = (sp.kt_lo + i) * FT_BN;
        const bool need_mask = k_base + FT_BN - 1 > e.z || (window > 0 && k_base < sp.p_last - window + 1);
        const int hi_j = qp - k_base, lo_j = window > 0 ? qp - window - k_base : -1;  // key j of the tile is visible iff lo_j < j <= hi_j
        if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->s_full, cnt & 1, abort_flag))) { ok = false; break; }
        hb_tc_fence_after();
        uint32_t sr[64];
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          hb_tmem_ld64_nowait(tmem_s + lane_base + hh * 64, sr);
          hb_tmem_ld_wait();
          hb_tmem_ld_fence64(sr);
          if (need_mask) {
#pragma unroll
            for (int j = 0; j < 64; j++)
              if (!(j + hh * 64 <= hi_j && j + hh * 64 > lo_j)) sr[j] = __float_as_uint(-INFINITY);
          }
#pragma unroll
          for (int j = 0; j < 64; j += 2) mx[(j >> 1) & 3] = fmaxf(fmaxf(mx[(j >> 1) & 3], __uint_as_float(sr[j])), __uint_as_float(sr[j + 1]));
        }
        float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;
        const float dist0 = (float)(qp - k_base);                     // of the tile's first key
        if (EX) m_tile -= r1 * __log2f(fmaf(r2, fmaxf(dist0 - (FT_BN - 1), 0.f), 1.f));
        const bool grow = m_tile > m_run + FT_SLACK;   // also the first tile with a visible key: m_run is -inf
        float corr = 1.f;
        if (grow) {
          corr = hb_exp2(m_run - m_tile);   // 0 while nothing has been summed
          m_run = m_tile;
        }
        const float sub = m_run == -INFINITY ? 0.f : m_run;
        const uint64_t scale2 = ft_pack2(__float_as_uint(scale_log2), __float_as_uint(scale_log2)), sub2 = ft_pack2(__float_as_uint(-sub), __float_as_uint(-sub));
        uint64_t sum2[2] = {0ull, 0ull};   // four sums of pairs
        // the exponentials: keys 64-127 are still in the registers (masked), keys 0-63 are read again
#pragma unroll
        for (int hh = 1; hh >= 0; hh--) {
          if (hh == 0) {
            hb_tmem_ld64_nowait(tmem_s + lane_base, sr);
            hb_tmem_ld_wait();
            hb_tmem_ld_fence64(sr);
            hb_tc_fence_before();
            __syncwarp();
            if (lane == 0) hb_mbar_arrive(&bar->s_free);  // the last read of S: the scores of the next tile may overwrite it
            if (need_mask) {
#pragma unroll
              for (int j = 0; j < 64; j++)
                if (!(j <= hi_j && j > lo_j)) sr[j] = __float_as_uint(-INFINITY);
            }
          }
#pragma unroll
          for (int j = 0; j < 64; j += 4) {  // masked scores are -inf: 2^-inf = 0
            float p0, p1, p2, p3;
            ft_exp<EX>(sr[j], sr[j + 1], scale2, sub2, r1, r2, dist0 - (float)(j + hh * 64), p0, p1);
            ft_exp<EX>(sr[j + 2], sr[j + 3], scale2, sub2, r1, r2, dist0 - (float)(j + 2 + hh * 64), p2, p3);
            sum2[(j >> 2) & 1] = ft_add2(sum2[(j >> 2) & 1], ft_pack2(__float_as_uint(p0 + p1), __float_as_uint(p2 + p3)));
            sr[j >> 1] = hb_pack_bf16(p0, p1);
            sr[(j >> 1) + 1] = hb_pack_bf16(p2, p3);
          }
          // the product of the tile before has read its P and written its O
          if (hh == 1 && cnt > 0 && !__all_sync(0xffffffffu, hb_mbar_wait(&bar->pv_done, (cnt - 1) & 1, abort_flag))) { ok = false; break; }
          // 64 keys = eight 16-byte chunks of this row in K block hh of P
#pragma unroll
          for (int cc = 0; cc < 8; cc++) {
            const uint32_t dst = hb_smem_u32(sP + hh * FT_TILE) + r * 128 + ((cc ^ (r & 7)) << 4);
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(sr[4 * cc]), "r"(sr[4 * cc + 1]),
                         "r"(sr[4 * cc + 2]), "r"(sr[4 * cc + 3]) : "memory");
          }
        }
        if (!ok) break;
        float s0, s1, s2, s3;
        ft_unpack2(sum2[0], s0, s1);
        ft_unpack2(sum2[1], s2, s3);
        l_run = l_run * corr + ((s0 + s1) + (s2 + s3));
        if (i > 0 && __any_sync(0xffffffffu, grow)) {   // a raised maximum: the row of O so far
          hb_tc_fence_after();
          hb_tmem_ld64_nowait(tmem_o + lane_base, sr);
          hb_tmem_ld_wait();
          hb_tmem_ld_fence64(sr);
#pragma unroll
          for (int d = 0; d < 64; d++) sr[d] = __float_as_uint(__uint_as_float(sr[d]) * corr);
          hb_tmem_st64(tmem_o + lane_base, sr);
          hb_tmem_st_wait();
        }
        hb_tc_fence_before();
        hb_fence_proxy_async();
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->p_full);
      }
      // the item's end: the next one's first product comes behind the arrivals of these warps, so O is theirs until then
      if (ok) ok = __all_sync(0xffffffffu, hb_mbar_wait(&bar->pv_done, (cnt - 1) & 1, abort_flag));
      if (ok) {
        hb_tc_fence_after();
        if (EX && sink) l_run += hb_exp2(fmaf(sink[hq], 1.4426950408889634f, -m_run));
        const float inv = 1.f / l_run;
        uint32_t o[64];
        hb_tmem_ld64_nowait(tmem_o + lane_base, o);
        hb_tmem_ld_wait();
        hb_tmem_ld_fence64(o);
        hb_tc_fence_before();
        if (r < e.y) {
          __nv_bfloat16* dst = out + ((size_t)(e.x + r) * Hq + hq) * 64;
#pragma unroll
          for (int d = 0; d < 64; d += 8) {
            uint4 w;
            w.x = hb_pack_bf16(__uint_as_float(o[d]) * inv, __uint_as_float(o[d + 1]) * inv);
            w.y = hb_pack_bf16(__uint_as_float(o[d + 2]) * inv, __uint_as_float(o[d + 3]) * inv);
            w.z = hb_pack_bf16(__uint_as_float(o[d + 4]) * inv, __uint_as_float(o[d + 5]) * inv);
            w.w = hb_pack_bf16(__uint_as_float(o[d + 6]) * inv, __uint_as_float(o[d + 7]) * inv);
            *(uint4*)(dst + d) = w;
          }
        }
      }
    }
  }

  hb_tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    __nanosleep(100000);
  }
  if (warp == 6) {
    __syncwarp();
    hb_tmem_dealloc(tmem_s, 256);
  }
}

HB_EXPORT int hb_flash_prefill_tc_supported(int Hq, int Hkv, int D, int page_size) {
  return Hkv > 0 && Hq % Hkv == 0 && (D == 64 || D == 128) && page_size >= 8 && page_size <= FT_BN && (page_size & (page_size - 1)) == 0;
}

static int ft_sms() {
  static int n[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n[dev] = 148;
  return n[dev];
}

// How a step is cut into launches. Portions of T rows in all have at most T / 128 (request, query tile) pairs and one more each, and there are at
// most T / min_rows portions; a launch takes `most` pairs (as many as a CTA has places for its share of the items). A step that may have more is cut
// into launches of req_step requests, or of req_step requests and qt_step query tiles.
struct FtCut { int req_step, qt_step, tiles, most, ctas; long bound; };
static FtCut ft_cut(int T, int R, int max_q_len, int Hq, int D, int min_rows) {
  FtCut c;
  c.tiles = (max_q_len + FT_BM - 1) / FT_BM;
  c.ctas = (D == 64 ? 2 : 1) * ft_sms();
  const long share = (long)(D == 64 ? FT_OWN64 : FT_OWN) * c.ctas / Hq;
  c.most = share < FT_MAX_PAIRS ? (int)share : FT_MAX_PAIRS;
  const long full = T / FT_BM, portions = min_rows > 1 && T / min_rows < R ? T / min_rows : R;
  c.bound = full + portions;
  c.req_step = R;
  c.qt_step = c.tiles;
  if (c.most > 0 && c.bound > c.most && (long)R * c.tiles > c.most) {
    if (full <= c.most / 2) c.req_step = c.most - (int)full;
    else {
      c.req_step = R < 32 ? R : 32;
      if (c.req_step > c.most) c.req_step = c.most;
      c.qt_step = c.most / c.req_step;
    }
  }
  return c;
}
// The launches that a step of these sizes is.
HB_EXPORT int hb_flash_prefill_tc_launches(int T, int R, int max_q_len, int Hq, int D, int min_rows) {
  if (R <= 0 || max_q_len <= 0 || T <= 0) return 0;
  const FtCut c = ft_cut(T, R, max_q_len, Hq, D, min_rows);
  return ((R + c.req_step - 1) / c.req_step) * ((c.tiles + c.qt_step - 1) / c.qt_step);
}

// q, out [T, Hq, D] bf16; caches [num_pages, Hkv, page_size, D] bf16 (D 64 or 128); per request q_start, q_len,
// ctx_len and a block table row, as hb_flash_prefill. Requests with fewer than min_rows rows are
// skipped. `status` is set to 1 if a bounded wait ran out.
HB_EXPORT int hb_flash_prefill_tc(const void* q, const void* kc, const void* vc, long num_pages, const int* bt, int bt_stride,
                                  const int* q_start, const int* q_len, const int* ctx_len, void* out, int T, int R,
                                  int max_q_len, int Hq, int Hkv, int D, int page_size, int window, float scale,
                                  int min_rows, int* status, const float* r1, const float* r2, const float* sink,
                                  cudaStream_t st) {
  if (R <= 0 || max_q_len <= 0 || T <= 0) return 0;
  if (!hb_flash_prefill_tc_supported(Hq, Hkv, D, page_size))
    HB_FAIL("hb_flash_prefill_tc: %d/%d heads of %d with pages of %d are not supported", Hq, Hkv, D, page_size);
  if (R > 65535 || max_q_len > 65535 * FT_BM) HB_FAIL("hb_flash_prefill_tc: %d requests / portions of %d rows are beyond the grid limit", R, max_q_len);
  if (!status) HB_FAIL("hb_flash_prefill_tc: no status word");
  const bool ex = r1 || sink;
  if ((r1 != nullptr) != (r2 != nullptr) || (ex && window > 0)) HB_FAIL("hb_flash_prefill_tc: a distance bias needs both of its vectors, and no window");
  CUtensorMap mq, mk, mv;
  if (hb_make_tensor_map_bf16(&mq, q, (uint64_t)T, (uint64_t)Hq * D, (uint64_t)Hq * D, FT_BM)) return -1;
  const uint64_t rows = (uint64_t)num_pages * Hkv * page_size;
  if (hb_make_tensor_map_bf16(&mk, kc, rows, (uint64_t)D, (uint64_t)D, (uint32_t)page_size)) return -1;
  if (hb_make_tensor_map_bf16(&mv, vc, rows, (uint64_t)D, (uint64_t)D, (uint32_t)page_size)) return -1;
  const float sl2 = scale * 1.4426950408889634f;
  cudaError_t e = cudaSuccess;
  const FtCut c = ft_cut(T, R, max_q_len, Hq, D, min_rows);
  if (c.most < 1) HB_FAIL("hb_flash_prefill_tc: %d heads are beyond the list of items", Hq);
#define FT_LAUNCH(KERN, THREADS, SMEM)                                                                                           \
  do {                                                                                                                          \
    static bool configured = false;                                                                                             \
    if (!configured) {                                                                                                          \
      e = cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);                                        \
      if (e != cudaSuccess) HB_FAIL("hb_flash_prefill_tc: %s", cudaGetErrorString(e));                                          \
      configured = true;                                                                                                        \
    }                                                                                                                           \
    e = hb_launch(KERN, grid, THREADS, SMEM, st, mq, mk, mv, bt, bt_stride, q_start, q_len, ctx_len, (__nv_bfloat16*)out, Hq,   \
                  Hkv, page_size, window, sl2, min_rows, status, r1, r2, sink, req0, reqs, qt0, qts, most);         \
  } while (0)
  for (int req0 = 0; req0 < R && e == cudaSuccess; req0 += c.req_step)
    for (int qt0 = 0; qt0 < c.tiles && e == cudaSuccess; qt0 += c.qt_step) {
      const int reqs = R - req0 < c.req_step ? R - req0 : c.req_step, qts = c.tiles - qt0 < c.qt_step ? c.tiles - qt0 : c.qt_step;
      const long items = ((long)reqs * qts < c.bound ? (long)reqs * qts : c.bound) * Hq;
      const int grid = (int)(items < c.ctas ? (items > 0 ? items : 1) : c.ctas);
      const long share = (long)(D == 64 ? FT_OWN64 : FT_OWN) * grid / Hq;      // (of a smaller grid: whatever the lengths say, a CTA's items have places)
      const int most = share < c.most ? (int)share : c.most;
      if (D == 64 && !ex) FT_LAUNCH(flash_prefill_tc64_kernel<false>, 256, FT_SMEM64);
      else if (D == 64) FT_LAUNCH(flash_prefill_tc64_kernel<true>, 256, FT_SMEM64);
      else if (!ex) FT_LAUNCH(flash_prefill_tc_kernel<false>, FT_THREADS, FT_SMEM);
      else FT_LAUNCH(flash_prefill_tc_kernel<true>, FT_THREADS, FT_SMEM);
    }
#undef FT_LAUNCH
  if (e != cudaSuccess) HB_FAIL("hb_flash_prefill_tc: %s", cudaGetErrorString(e));
  HB_CHECK_LAUNCH("hb_flash_prefill_tc");
  return 0;
}
