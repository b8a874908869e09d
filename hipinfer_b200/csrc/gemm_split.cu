// C[M,N] (+)= A[M,K] W[N,K]^T for 32-bit operands, to 32-bit accuracy, on the tensor cores: every operand is the exact sum of three
// bf16 numbers (x1 = round(x), x2 = round(x - x1), x3 = x - x1 - x2: 24 bits), and the six products of the nine that reach the last bit
// of a 32-bit product are summed: w1 a1, w1 a2, w2 a1, w2 a2, w1 a3, w3 a1 (the rest is below 2^-26 of |w a|).
//
// The tensor cores' sums do not round to nearest, so they are kept short: an accumulator in tensor memory takes 64 k, smallest
// products first (only the last four MMAs meet a sum of full size), and is then added to the running sum in registers, rounded to
// nearest. The error against 64 bits is smaller than that of gemm_simt.cu, whose FFMA chains are 512 and longer:
// 512 x 2,048 x 8,192 1.7e-7 against 5.8e-7 (2-norm), 301 x 16,384 x 2,048 1.3e-7 against 4.1e-7.
//
// The weights are the MMA's 128-row side and the rows of A its N side (up to 160: what two stages leave in 227 KB of shared memory). A's three planes
// are written by a small kernel ahead (split_rows_kernel) and come by TMA; W is read as it is, 32 bits, and split on its way into
// shared memory. A CTA makes one tile of 128 weights x NT rows, over all of K or a slice of it (few tiles: the slices' sums go to
// a workspace and are added lowest first). Warps:
//   0-7    W: 128 x 64 floats a stage, asked for a stage ahead, split into three swizzled K-major bf16 tiles; and, while those loads are
//          on their way, the running sums of the stage before: a thread owns one weight row (TMEM lane) and half of the tile's columns
//   8      TMA of A's planes;  9  tcgen05.mma, 24 a stage
// Where the sum of three does not hold, the row is flagged and its outputs are FFMA chains in the order of gemm_simt.cu: numbers that are
// not finite, or round to no finite bf16 (they would turn into NaN where FFMA gives an infinity), and rows whose numbers are all below
// 2^-100 (the tensor cores do not see all of their remainders, which lie below the normal range). In a row that has a number of 2^-100 or more the
// small ones lose those remainders: some 2^-120 of an error for each, beside a row of at least 2^-100. It shows only where all the large numbers meet zeros.
//
// What bounds it: a gate/up of 301 rows (119 us) is 256 tiles on 148 SMs, two rounds of 32 stages. The MMAs of a stage, 24 of 93 cycles at N = 160, are
// 74 us of that (73 us would be six products at the measured burst rate of 1,666 TFLOP/s, 89 at the sustained one); the rest is what a stage's
// workers, copies and MMAs wait for one another. From some 64 rows down the workers bound it (some 1,100 cycles a stage for the split of 128 x 64 weights and
// the running sums). us, gemm_simt.cu / here, with the kernels ahead and behind: 301 rows x 16,384 x 2,048 455 / 119, x 2,048 x 8,192
// 250 / 80, x 3,072 x 2,048 107 / 29; 64 rows x 16,384 x 2,048 109 / 55; 9 rows x 16,384 x 2,048 101 / 52, x 3,072 x 2,048 43 / 19, x 256 x 256 16 / 8.4.
// Tried: sums in warps of their own (120 us more for the gate/up: four warps cannot split W as fast), the weights' lines asked into L2
// five stages ahead (5 % slower).
#include "tc_common.cuh"

#include <string.h>

constexpr int GS_WR = 128, GS_NT = 160, GS_BK = 64, GS_STAGES = 2, GS_MAX_SPLITS = 8;
constexpr int GS_WTILE = GS_WR * GS_BK * 2, GS_ATILE = GS_NT * GS_BK * 2, GS_STAGE = 3 * (GS_WTILE + GS_ATILE);
constexpr int GS_THREADS = 10 * 32;
struct GsBars {
  uint64_t w_full[GS_STAGES], a_full[GS_STAGES], stage_free[GS_STAGES], acc_full[2], acc_free[2];
  uint32_t tmem_slot;
  int abort_flag;
  int w_odd[GS_WR], a_odd[GS_NT], any_odd;    // rows whose outputs are FFMA chains, and whether there are some
};
constexpr int GS_SMEM = GS_STAGES * GS_STAGE + (int)sizeof(GsBars) + 1024;
static_assert(GS_SMEM <= 227 * 1024 && GS_WTILE % 1024 == 0 && GS_ATILE % 1024 == 0, "shared memory of a block, swizzled tiles on 1 KB");

// x = hi + mid + lo and the same of y, each bf16. `odd` becomes NaN where that does not hold: x, y (or a rounding of them to bf16) is not
// finite, and the remainder of the remainder then is not a number.
__device__ __forceinline__ void gs_split2(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo, float& odd) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float rx = x - __low2float(h), ry = y - __high2float(h);
  const __nv_bfloat162 m = __floats2bfloat162_rn(rx, ry);
  const float sx = rx - __low2float(m), sy = ry - __high2float(m);
  const __nv_bfloat162 l = __floats2bfloat162_rn(sx, sy);
  hi = *(const uint32_t*)&h;
  mid = *(const uint32_t*)&m;
  lo = *(const uint32_t*)&l;
  odd += sx + sy;
}

constexpr float GS_TINY = 7.8886090522101181e-31f;      // 2^-100
__device__ __forceinline__ float gs_most(const float4& v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))); }

// Row m of A (4-element aligned) as rows m, M + m and 2 M + m of planes [3 M, Kp], zero beyond K; odd[m]: the row has a number that is no such sum.
__global__ void __launch_bounds__(128) split_rows_kernel(const float* A, long lda, __nv_bfloat16* planes, int* odd, int M, int K, int Kp) {
  __shared__ int any, size;      // size: 1 a number below GS_TINY, 2 one above
  hb_pdl_launch();
  const int m = blockIdx.x;
  if (threadIdx.x == 0) any = size = 0;
  __syncthreads();
  hb_pdl_wait();
  float bad = 0.f, most = 0.f;
  for (int k = threadIdx.x * 4; k < Kp; k += 512) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < K) v = *(const float4*)(A + (size_t)m * lda + k);
    uint2 h, d, l;
    gs_split2(v.x, v.y, h.x, d.x, l.x, bad);
    gs_split2(v.z, v.w, h.y, d.y, l.y, bad);
    most = fmaxf(most, gs_most(v));
    __nv_bfloat16* p = planes + (size_t)m * Kp + k;
    *(uint2*)p = h;
    *(uint2*)(p + (size_t)M * Kp) = d;
    *(uint2*)(p + (size_t)2 * M * Kp) = l;
  }
  if (bad != bad) any = 1;
  if (most > 0.f) atomicOr(&size, most < GS_TINY ? 1 : 2);
  __syncthreads();
  if (threadIdx.x == 0) odd[m] = any || size == 1;
}

__global__ void __launch_bounds__(GS_THREADS, 1) gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const float* A, long lda,
                                                                   const float* W, long ldw, float* C, long ldc, const int* odd, float* ws,
                                                                   int M, int N, int K, int NT, int kbs, int accumulate, int depth, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  GsBars* bar = (GsBars*)(smem + GS_STAGES * GS_STAGE);
  volatile int* abort_flag = &bar->abort_flag;
  hb_pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * GS_WR, m0 = blockIdx.y * NT, num_kb = (K + GS_BK - 1) / GS_BK;
  const int kb0 = blockIdx.z * kbs, kb1 = min(num_kb, kb0 + kbs), n_kb = kb1 - kb0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GS_STAGES; s++) { hb_mbar_init(&bar->w_full[s], 8); hb_mbar_init(&bar->a_full[s], 1); hb_mbar_init(&bar->stage_free[s], 1); }
    for (int b = 0; b < 2; b++) { hb_mbar_init(&bar->acc_full[b], 1); hb_mbar_init(&bar->acc_free[b], 8); }
    bar->abort_flag = 0;
    bar->any_odd = 0;
    hb_fence_barrier_init();
  }
  for (int i = threadIdx.x; i < GS_WR; i += GS_THREADS) bar->w_odd[i] = 0;
  if (warp == 9) {
    hb_tmem_alloc(&bar->tmem_slot, 512);
    hb_tmem_relinquish();
  }
  if (warp == 8 && lane == 0) hb_tma_prefetch_desc(&map_a);
  hb_tc_fence_before();
  __syncthreads();
  hb_tc_fence_after();
  const uint32_t tmem = bar->tmem_slot;      // two accumulators, 256 columns apart
  if (warp < 8) {  // ---------------- W: lane = four k of one row, 16 lanes a row, the block's 128 rows in 8 steps; and the running sums
    const int row = warp * 2 + (lane >> 4), kq = (lane & 15) * 4;
    const float* src = W + (size_t)(n0 + row) * ldw + kq;
    float4 v[8];
    auto fetch = [&](int i, int kb) {
      const int k = kb * GS_BK;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (kb < kb1 && n0 + row + 16 * i < N && k + kq < K) v[i] = *(const float4*)(src + (size_t)(16 * i) * ldw + k);
    };
    const int quarter = warp & 3, half = warp >> 2, chunks = NT / 16, per = (chunks + 1) / 2;
    const int c0 = half * per, mine = min(per, chunks - c0);          // this warp's chunks of 16 columns
    const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16) + c0 * 16;
    float acc[5][16];
#pragma unroll
    for (int q = 0; q < 5; q++)
#pragma unroll
      for (int j = 0; j < 16; j++) acc[q][j] = 0.f;
    bool ok = true;
    uint32_t sizes = 0;                          // of the thread's 8 rows: bit i a number below GS_TINY, bit 8 + i one above
#pragma unroll
    for (int i = 0; i < 8; i++) fetch(i, kb0);   // (the weights do not depend on the kernel ahead)
    for (int it = 0; it <= n_kb; it++) {
      if (it < n_kb) {
        const uint32_t s = it % GS_STAGES, ph = (it / GS_STAGES) & 1;
        if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->stage_free[s], ph ^ 1, abort_flag))) { ok = false; break; }
        const uint32_t dst = hb_smem_u32(smem + s * GS_STAGE) + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8;
        // four rows at a time: their chains run side by side, and the next block's are asked for as registers fall free
#pragma unroll
        for (int g = 0; g < 8; g += 4) {
          uint32_t x[4][6];
          float bad[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            bad[i] = 0.f;
            gs_split2(v[g + i].x, v[g + i].y, x[i][0], x[i][2], x[i][4], bad[i]);
            gs_split2(v[g + i].z, v[g + i].w, x[i][1], x[i][3], x[i][5], bad[i]);
            const float m = gs_most(v[g + i]);
            if (m > 0.f) sizes |= m < GS_TINY ? 1u << (g + i) : 256u << (g + i);
          }
#pragma unroll
          for (int i = 0; i < 4; i++) fetch(g + i, kb0 + it + 1);
#pragma unroll
          for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int p = 0; p < 3; p++)
              asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst + (g + i) * 2048 + p * GS_WTILE), "r"(x[i][2 * p]), "r"(x[i][2 * p + 1]));
            if (bad[i] != bad[i]) bar->w_odd[row + 16 * (g + i)] = 1;
          }
        }
        hb_fence_proxy_async();
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->w_full[s]);
      }
      if (it > 0) {      // the sums of the stage before
        const uint32_t b = (it - 1) & 1, aph = ((it - 1) >> 1) & 1;
        if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->acc_full[b], aph, abort_flag))) { ok = false; break; }
        hb_tc_fence_after();
#pragma unroll
        for (int q = 0; q < 5; q++)
          if (q < mine) {
            float t[16];
            hb_tmem_ld16(t0 + b * 256 + q * 16, t);
#pragma unroll
            for (int j = 0; j < 16; j++) acc[q][j] += t[j];
          }
        hb_tc_fence_before();
        __syncwarp();
        if (lane == 0) hb_mbar_arrive(&bar->acc_free[b]);
      }
    }
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) sizes |= __shfl_xor_sync(0xffffffffu, sizes, o);     // a row is 16 lanes'
    if ((lane & 15) == 0)
      for (int i = 0; i < 8; i++)
        if ((sizes >> i & 0x101u) == 1u) bar->w_odd[row + 16 * i] = 1;
    hb_pdl_wait();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    for (int i = threadIdx.x; i < NT; i += 256)
      if ((bar->a_odd[i] = m0 + i < M ? odd[m0 + i] : 0)) bar->any_odd = 1;
    if (threadIdx.x < GS_WR && bar->w_odd[threadIdx.x]) bar->any_odd = 1;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const int n = n0 + quarter * 32 + lane;
    if (ok && n < N) {
      const bool slice = ws != nullptr, add = !slice && accumulate;
      const long ld = slice ? N : ldc;
      float* out = (slice ? ws + (size_t)blockIdx.z * M * N : C) + (size_t)(m0 + c0 * 16) * ld + n;
      const int rows = min(mine * 16, M - m0 - c0 * 16);        // of this warp's columns
#pragma unroll
      for (int q = 0; q < 5; q++)
        if (q * 16 < rows) {
          float old[16];
#pragma unroll
          for (int j = 0; j < 16; j++) old[j] = add && q * 16 + j < rows ? out[(size_t)(q * 16 + j) * ld] : 0.f;
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (q * 16 + j < rows) out[(size_t)(q * 16 + j) * ld] = add ? old[j] + acc[q][j] : acc[q][j];
          if (bar->any_odd) {
#pragma unroll 1
            for (int j = 0; j < 16 && q * 16 + j < rows; j++) {
              const int m = m0 + (c0 + q) * 16 + j;
              if (!(bar->w_odd[quarter * 32 + lane] | bar->a_odd[m - m0])) continue;
              const float *a = A + (size_t)m * lda, *w = W + (size_t)n * ldw;
              float sum = 0.f, was = 0.f;
#pragma unroll
              for (int z = 0; z < 16; z++) was = z == j ? old[z] : was;
              for (int k = kb0 * GS_BK, end = min(K, kb1 * GS_BK); k < end;) {
                const int stop = min(end, slice ? end : (k / depth + 1) * depth);
                float chain = 0.f;
                for (; k < stop; k++) chain = fmaf(a[k], w[k], chain);
                sum += chain;
              }
              out[(size_t)(q * 16 + j) * ld] = add ? was + sum : sum;
            }
          }
        }
    }
  } else if (warp == 8) {  // ---------------- TMA of A's planes
    hb_pdl_wait();
    for (int it = 0; it < n_kb; it++) {
      const uint32_t s = it % GS_STAGES, ph = (it / GS_STAGES) & 1;
      if (!__all_sync(0xffffffffu, hb_mbar_wait(&bar->stage_free[s], ph ^ 1, abort_flag))) break;
      if (hb_elect()) {
        hb_mbar_expect_tx(&bar->a_full[s], 3 * NT * GS_BK * 2);
#pragma unroll
        for (int p = 0; p < 3; p++)
          hb_tma_load_2d(smem + s * GS_STAGE + 3 * GS_WTILE + p * GS_ATILE, &map_a, &bar->a_full[s], (kb0 + it) * GS_BK, p * M + m0);
      }
      __syncwarp();
    }
  } else if (warp == 9) {  // ---------------- tensor cores
    const uint32_t idesc = hb_umma_idesc_bf16(GS_WR, NT);
    for (int it = 0; it < n_kb; it++) {
      const uint32_t s = it % GS_STAGES, ph = (it / GS_STAGES) & 1, b = it & 1, aph = (it >> 1) & 1;
      const bool ok = hb_mbar_wait(&bar->acc_free[b], aph ^ 1, abort_flag) && hb_mbar_wait(&bar->w_full[s], ph, abort_flag) &&
                      hb_mbar_wait(&bar->a_full[s], ph, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
      hb_tc_fence_after();
      if (hb_elect()) {
        const uint64_t w1 = hb_umma_desc_k128(hb_smem_u32(smem + s * GS_STAGE)), a1 = hb_umma_desc_k128(hb_smem_u32(smem + s * GS_STAGE + 3 * GS_WTILE));
        constexpr uint64_t WP = GS_WTILE >> 4, AP = GS_ATILE >> 4;      // a plane further, in the descriptor's units
        const uint32_t d = tmem + b * 256;
        auto product = [&](int wp, int ap, bool first) {
#pragma unroll
          for (int k = 0; k < GS_BK / 16; k++) hb_umma_bf16(d, w1 + wp * WP + 2 * k, a1 + ap * AP + 2 * k, idesc, !first || k != 0);
        };
        product(2, 0, true);
        product(0, 2, false);
        product(1, 1, false);
        product(1, 0, false);
        product(0, 1, false);
        product(0, 0, false);
        hb_umma_commit(&bar->stage_free[s]);
        hb_umma_commit(&bar->acc_full[b]);
      }
      __syncwarp();
    }
  }

  hb_tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    __nanosleep(100000);  // let copies that may still be in flight land before the shared memory is given up
  }
  if (warp == 9) {
    __syncwarp();
    hb_tmem_dealloc(tmem, 512);
  }
}

// C (+)= the slices' sums, lowest first; four columns a thread.
__global__ void __launch_bounds__(256) split_reduce_kernel(const float* ws, float* C, long ldc, int M, int N, int slices, int accumulate) {
  hb_pdl_launch();
  hb_pdl_wait();
  const size_t MN = (size_t)M * N, i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= MN) return;
  float4 v[GS_MAX_SPLITS];
#pragma unroll
  for (int s = 0; s < GS_MAX_SPLITS; s++)
    if (s < slices) v[s] = *(const float4*)(ws + s * MN + i);
  float4 t = v[0];
#pragma unroll
  for (int s = 1; s < GS_MAX_SPLITS; s++)
    if (s < slices) { t.x += v[s].x; t.y += v[s].y; t.z += v[s].z; t.w += v[s].w; }
  float* o = C + i / N * ldc + i % N;
  if (accumulate) { const float4 c = *(const float4*)o; t.x += c.x; t.y += c.y; t.z += c.z; t.w += c.w; }
  *(float4*)o = t;
}

// ---------------------------------------------------------------------------------------
// The K blocks of a slice and the slices, by N and K alone, so that a row's bits do not depend on how many rows there are: 512 k deep or deeper, one
// row of tiles at most a round of 148 SMs, and of those the number whose rounds take least for one row of tiles and for two together. (With the slices chosen for the rows there
// are, three rows of tiles or more would be up to 30 % faster where they are few, us: 400 rows x 2,048 x 2,048 28 / 39, x 2,048 x 8,192 88 / 107, 2,048
// rows x 2,048 x 2,048 110 / 128. One rule for one row of tiles alone takes 301 rows x 3,072 x 2,048 from 28 to 41, 9 rows from 19 to 15.)
// nt: the tile's rows of A, a multiple of 16; an output's bits do not depend on it.
static void gs_plan(int M, int N, int K, int* nt, int* kbs, int* splits) {
  const int tiles = (M + GS_NT - 1) / GS_NT, num_kb = (K + GS_BK - 1) / GS_BK;
  *nt = ((M + tiles - 1) / tiles + 15) / 16 * 16;
  const long cols = (N + GS_WR - 1) / GS_WR;
  long least = -1;
  for (int n = 1; n <= GS_MAX_SPLITS && (n == 1 || (n * cols <= 148 && n <= K / 512 && !(N & 3))); n++) {
    const int blocks = (num_kb + n - 1) / n, slices = (num_kb + blocks - 1) / blocks;
    const long time = blocks * ((cols * slices + 147) / 148 + (2 * cols * slices + 147) / 148);
    if (least < 0 || time < least) { least = time; *kbs = blocks; *splits = slices; }
  }
}
static size_t gs_planes(int M, int K) { return (size_t)3 * M * ((K + GS_BK - 1) / GS_BK * GS_BK) * 2; }
static size_t gs_flags(int M) { return ((size_t)M * 4 + 15) / 16 * 16; }

// Bytes of workspace of a product, and (launches) the kernels it is.
HB_EXPORT long hb_gemm_split_workspace(int M, int N, int K, int* launches) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  int nt, kbs, splits;
  gs_plan(M, N, K, &nt, &kbs, &splits);
  if (launches) *launches = splits > 1 ? 3 : 2;
  return (long)(gs_planes(M, K) + gs_flags(M) + (splits > 1 ? (size_t)splits * M * N * 4 : 0));
}

// A [M, K], W [N, K], C [M, N], fp32 with contiguous rows on 16 bytes; K and, where C is written by the slices' reader, N a multiple of 4.
HB_EXPORT int hb_gemm_split(const float* A, long lda, const float* W, long ldw, float* C, long ldc, int M, int N, int K, int accumulate, void* ws,
                            long ws_bytes, int* status, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 3)) HB_FAIL("hb_gemm_split: K = %d must be a positive multiple of 4", K);
  if ((((uintptr_t)A | (uintptr_t)W | (uintptr_t)C | (uintptr_t)ws) & 15) || ((lda | ldw | ldc) & 3)) HB_FAIL("hb_gemm_split: operands and rows must lie on 16 bytes");
  if (!status || !ws) HB_FAIL("hb_gemm_split: no status word or workspace");
  int nt, kbs, splits;
  gs_plan(M, N, K, &nt, &kbs, &splits);
  if ((M + nt - 1) / nt > 65535) HB_FAIL("hb_gemm_split: M = %d is beyond the grid limit", M);
  if (ws_bytes < hb_gemm_split_workspace(M, N, K, nullptr)) HB_FAIL("hb_gemm_split: workspace of %ld bytes", ws_bytes);
  int chains = (K + 511) / 512;      // the chains of the plain kernels (slice_plan in gemm_simt.cu): at most eight, 512 deep or more
  if (chains > 8) chains = 8;
  const int depth = ((K + chains - 1) / chains + 63) / 64 * 64;
  const int Kp = (K + GS_BK - 1) / GS_BK * GS_BK;
  __nv_bfloat16* planes = (__nv_bfloat16*)ws;
  int* odd = (int*)((char*)ws + gs_planes(M, K));
  float* part = splits > 1 ? (float*)((char*)odd + gs_flags(M)) : nullptr;
  CUtensorMap ma;
  if (hb_make_tensor_map_bf16(&ma, planes, (uint64_t)3 * M, (uint64_t)Kp, (uint64_t)Kp, (uint32_t)nt)) return -1;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM);
    if (e != cudaSuccess) HB_FAIL("hb_gemm_split: %s", cudaGetErrorString(e));
    configured = true;
  }
  cudaError_t e = hb_launch(split_rows_kernel, M, 128, 0, s, A, lda, planes, odd, M, K, Kp);
  const dim3 grid((N + GS_WR - 1) / GS_WR, (M + nt - 1) / nt, splits);
  if (e == cudaSuccess)
    e = hb_launch(gemm_split_kernel, grid, GS_THREADS, GS_SMEM, s, ma, A, lda, W, ldw, C, ldc, (const int*)odd, part, M, N, K, nt, kbs, accumulate, depth, status);
  if (e == cudaSuccess && splits > 1)
    e = hb_launch(split_reduce_kernel, (unsigned)(((size_t)M * N / 4 + 255) / 256), 256, 0, s, (const float*)part, C, ldc, M, N, splits, accumulate);
  if (e != cudaSuccess) HB_FAIL("hb_gemm_split: %s", cudaGetErrorString(e));
  HB_CHECK_LAUNCH("hb_gemm_split");
  return 0;
}
