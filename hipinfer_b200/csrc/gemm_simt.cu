// The plain matrix product C[M,N] = A[M,K] W[N,K]^T in true 32-bit arithmetic (FFMA chains, no tensor cores), W row-major
// with K contiguous as the reference stores weights (src/api.cu:81-83). It is the 32-bit engine's product of up to eight rows (more rows
// go to gemm_split.cu where that takes their sizes) and serves whatever the tensor-core kernels do not take.
//
// K is cut into slices by a rule on K alone (slice_plan): at most eight, 512 deep or more. An output is the sum of its
// slices' FFMA chains, each running its k in order from zero, added lowest slice first. Every kernel below adds in that
// order, so a row's result is the same bits whatever M is and whichever kernel of this file ran, and the chains are no longer than K / 8.
//
// Three ways through the same sum:
//   simt_rows_kernel   up to 8 rows (a decode step: W is read once, the floor is its bytes).
//   simt_tile_kernel   64 x 128 tiles, 8 x 8 outputs a thread in packed pairs (fma.rn.f32x2), shared memory double-buffered
//                      through registers. WHOLE: a block walks all slices and keeps their running sum in registers;
//                      else blockIdx.z is the slice, partial sums go to a workspace and simt_reduce_kernel adds them: for
//                      products of so few tiles that whole-K blocks would leave SMs idle.
// EPI 0: C = sum;  EPI 1: C += sum (32-bit C: the residual stream);  EPI 2: C += colscale[n] * sum (the same with a scale
// vector over the output columns, of the weight's element type).
#include "tc_common.cuh"

constexpr int SM_TM = 64, SM_TN = 128, SM_TK = 16, SM_MAX_SLICES = 8, SM_MIN_SLICE = 512;

// The slices of K: a function of K alone.
__host__ __device__ static inline void slice_plan(int K, int* depth, int* count) {
  int n = (K + SM_MIN_SLICE - 1) / SM_MIN_SLICE;
  if (n > SM_MAX_SLICES) n = SM_MAX_SLICES;
  const int d = ((K + n - 1) / n + 63) / 64 * 64;
  *depth = d;
  *count = (K + d - 1) / d;
}

template <typename TC, typename TW, int EPI>
__device__ __forceinline__ void simt_put(TC* c, float sum, const TW* colscale, int n) {
  if (EPI == 2) *c = hb_from_float<TC>(__fadd_rn(hb_to_float(*c), __fmul_rn(hb_to_float(colscale[n]), sum)));
  else if (EPI == 1) *c = hb_from_float<TC>(hb_to_float(*c) + sum);
  else *c = hb_from_float<TC>(sum);
}

__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {   // two fmaf, each rounded by itself
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Four elements k .. k + 3 of row r, zero beyond the matrix or the slice. VEC: rows are 4-element aligned and k_end a
// multiple of 4, so that an access is whole or absent.
template <typename T, bool VEC>
__device__ __forceinline__ float4 simt_load(const T* p, long ld, int r, int rows, int k, int k_end) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r >= rows) return v;
  const T* q = p + (size_t)r * ld + k;
  if (VEC) {
    if (k < k_end) v = hb_load4(q);
  } else {
    if (k < k_end) v.x = hb_to_float(q[0]);
    if (k + 1 < k_end) v.y = hb_to_float(q[1]);
    if (k + 2 < k_end) v.z = hb_to_float(q[2]);
    if (k + 3 < k_end) v.w = hb_to_float(q[3]);
  }
  return v;
}

template <typename TA, typename TW, typename TC, int EPI, bool WHOLE, bool VEC>
__global__ void __launch_bounds__(128, 2) simt_tile_kernel(const TA* A, long lda, const TW* __restrict__ W, long ldw,
                                                           TC* C, long ldc, int M, int N, int K,
                                                           const TW* __restrict__ colscale, float* ws, int depth) {
  // rows of 64 + 4 and 128 + 4: a float4 read of one k by a warp meets no bank twice (the transposing stores below do: two passes each)
  __shared__ __align__(16) float As[2][SM_TK][SM_TM + 4], Ws[2][SM_TK][SM_TN + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * SM_TM, n0 = blockIdx.x * SM_TN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;          // this thread's row (of every 32) and first k of a staged tile
  const int k_lo = WHOLE ? 0 : blockIdx.z * depth, k_hi = WHOLE ? K : min(K, k_lo + depth);
  uint64_t acc[8][4], tot[WHOLE ? 8 : 1][4];            // [row][pair of columns]
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
  if (WHOLE)
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) tot[WHOLE ? i : 0][j] = 0ull;
  // no hb_pdl_launch(): a kernel of few blocks behind this one would be placed two an SM beside its tiles (a delta-rule walk
  // of 64 blocks took 683 us instead of 598)
  hb_pdl_wait();
  float4 ra[2], rw[4];
  auto fetch = [&](int k) {
#pragma unroll
    for (int i = 0; i < 2; i++) ra[i] = simt_load<TA, VEC>(A, lda, m0 + lr + 32 * i, M, k + lk, k_hi);
#pragma unroll
    for (int i = 0; i < 4; i++) rw[i] = simt_load<TW, VEC>(W, ldw, n0 + lr + 32 * i, N, k + lk, k_hi);
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      As[b][lk][lr + 32 * i] = ra[i].x; As[b][lk + 1][lr + 32 * i] = ra[i].y;
      As[b][lk + 2][lr + 32 * i] = ra[i].z; As[b][lk + 3][lr + 32 * i] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      Ws[b][lk][lr + 32 * i] = rw[i].x; Ws[b][lk + 1][lr + 32 * i] = rw[i].y;
      Ws[b][lk + 2][lr + 32 * i] = rw[i].z; Ws[b][lk + 3][lr + 32 * i] = rw[i].w;
    }
  };
  fetch(k_lo);
  stage(0);
  __syncthreads();
  int b = 0, left = depth;
  for (int k0 = k_lo; k0 < k_hi; k0 += SM_TK) {
    const bool more = k0 + SM_TK < k_hi;
    if (more) fetch(k0 + SM_TK);
#pragma unroll
    for (int k = 0; k < SM_TK; k++) {
      float a[8];
      uint64_t w[4];
      *(float4*)(a) = *(const float4*)&As[b][k][ty * 4];
      *(float4*)(a + 4) = *(const float4*)&As[b][k][32 + ty * 4];
      *(ulonglong2*)(w) = *(const ulonglong2*)&Ws[b][k][tx * 4];
      *(ulonglong2*)(w + 2) = *(const ulonglong2*)&Ws[b][k][64 + tx * 4];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint64_t aa = f2_pack(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = f2_fma(aa, w[j], acc[i][j]);
      }
    }
    if (WHOLE) {
      left -= SM_TK;
      if (left == 0 || !more) {      // the slice's end (its depth is a multiple of the tile's)
        left = depth;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) { tot[WHOLE ? i : 0][j] = f2_add(tot[WHOLE ? i : 0][j], acc[i][j]); acc[i][j] = 0ull; }
      }
    }
    if (more) {
      stage(b ^ 1);
      __syncthreads();
      b ^= 1;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int m = m0 + (i >> 2) * 32 + ty * 4 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + (j >> 1) * 64 + tx * 4 + (j & 1) * 2;
      float lo, hi;
      f2_unpack(WHOLE ? tot[WHOLE ? i : 0][j] : acc[i][j], lo, hi);
      if (WHOLE) {
        TC* c = C + (size_t)m * ldc + n;
        if (n < N) simt_put<TC, TW, EPI>(c, lo, colscale, n);
        if (n + 1 < N) simt_put<TC, TW, EPI>(c + 1, hi, colscale, n + 1);
      } else {
        float* c = ws + ((size_t)blockIdx.z * M + m) * N + n;
        if (n < N) c[0] = lo;
        if (n + 1 < N) c[1] = hi;
      }
    }
  }
}

template <typename TW, typename TC, int EPI>
__global__ void __launch_bounds__(256) simt_reduce_kernel(const float* ws, TC* C, long ldc, int M, int N,
                                                          int slices, const TW* __restrict__ colscale) {
  hb_pdl_launch();
  hb_pdl_wait();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x, MN = (size_t)M * N;
  if (i >= MN) return;
  float v[SM_MAX_SLICES], sum = 0.f;
#pragma unroll
  for (int s = 0; s < SM_MAX_SLICES; s++)
    if (s < slices) v[s] = ws[s * MN + i];
#pragma unroll
  for (int s = 0; s < SM_MAX_SLICES; s++)
    if (s < slices) sum += v[s];
  const size_t m = i / N, n = i - m * N;
  simt_put<TC, TW, EPI>(C + m * ldc + n, sum, colscale, (int)n);
}

// Up to 8 rows: W streams once through rings of shared memory, by cp.async. Persistent blocks (two an SM) walk groups of 16
// columns; warp w of a block makes slice w by itself: it asks for its slice's next piece (16 columns x KC), waits for the oldest
// and multiplies, with no barrier until the slices are added. Lane l makes column l & 15 of the rows (l >> 4), (l >> 4) + 2,
// ...: a 16-byte read of W serves RP rows, whose chains are independent. The first pieces of W are asked for before the wait
// for the kernel ahead. RING: the pieces of a warp's ring, five where two blocks then fit an SM, else four (32-bit operands, from
// five rows on, from four with more than four slices: with five pieces only one block fitted, and the blocks, dealt two an SM, ran
// in two rounds). Bound by HBM up to four rows, by the reads of shared memory above: 16,384 x 2,048 at 1, 4 and 8 rows 24.4, 28.5 and
// 41.6 us (8 rows with five pieces: 46.8), 4,096 x 14,336 45.4, 44.9 and 62.1 (4 and 8 rows with five pieces: 55.4 and 77.3).
constexpr int SR_COLS = 16, SR_ROWS = 8;
template <typename TA, typename TW, int KC> struct RowsPiece {
  static constexpr int PW = 16 / sizeof(TW), PA = 16 / sizeof(TA);        // elements of a 16-byte access
  // a column's piece is padded by 16 bytes: the 16-byte reads of eight columns meet no bank twice
  static constexpr int W_BYTES = SR_COLS * (KC + PW) * sizeof(TW);
  __host__ __device__ static constexpr int bytes(int M) { return W_BYTES + M * KC * (int)sizeof(TA); }
};
constexpr int SR_STATIC = 2 * SM_MAX_SLICES * SR_ROWS * SR_COLS * (int)sizeof(float), SR_MOST = 228 * 512 - 1024 - SR_STATIC;   // dynamic bytes of a block of two
template <typename TA, typename TW, typename TC, int EPI, int RP, int KC, int RING>
__global__ void __launch_bounds__(256, 2) simt_rows_kernel(const TA* A, long lda, const TW* __restrict__ W, long ldw, TC* C, long ldc,
                                                           int M, int N, int K, const TW* __restrict__ colscale, int depth) {
  using P = RowsPiece<TA, TW, KC>;
  extern __shared__ __align__(16) uint8_t sr_smem[];
  __shared__ float part[2][SM_MAX_SLICES][SR_ROWS][SR_COLS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slices = blockDim.x >> 5;
  const int per_tile = depth / KC, tiles = (N + SR_COLS - 1) / SR_COLS, k_lo = warp * depth, k_hi = min(K, k_lo + depth);
  const int total = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * per_tile;      // this block's pieces
  const int piece = P::bytes(M);
  const uint8_t* ring = sr_smem + (size_t)warp * RING * piece;
  const uint32_t ring_s = hb_smem_u32(ring);
  // this lane's place in a piece: LW lanes a column, LA lanes a row of A
  constexpr int LW = KC / P::PW, LA = KC / P::PA;
  static_assert(LW <= 32 && LA <= 32, "a piece's row is at most a warp wide");
  int wi = 0, wt = blockIdx.x, wk = k_lo;              // the next piece of W to ask for: its count, tile and k
  auto load_w = [&]() {
    const uint32_t dst = ring_s + (uint32_t)(wi % RING) * piece + (uint32_t)((lane / LW) * (KC + P::PW) + lane % LW * P::PW) * sizeof(TW);
    const int k = wk + lane % LW * P::PW, n = wt * SR_COLS + lane / LW;
    const TW* src = W + (size_t)n * ldw + k;
    if (k < k_hi) {
#pragma unroll
      for (int c = 0; c < SR_COLS; c += 32 / LW)
        if (n + c < N) hb_cp_async16(dst + (uint32_t)(c * (KC + P::PW)) * sizeof(TW), src + (size_t)c * ldw);
    }
    wi++;
    wk += KC;
    if (wk == k_lo + depth) { wk = k_lo; wt += gridDim.x; }
  };
  int ai = 0, ak = k_lo;
  auto load_a = [&]() {
    const uint32_t dst = ring_s + (uint32_t)(ai % RING) * piece + P::W_BYTES + (uint32_t)(lane % LA * P::PA) * sizeof(TA);
    const int k = ak + lane % LA * P::PA;
    if (k < k_hi)
      for (int m = lane / LA; m < M; m += 32 / LA) hb_cp_async16(dst + (uint32_t)(m * KC) * sizeof(TA), A + (size_t)m * lda + k);
    ai++;
    ak += KC;
    if (ak == k_lo + depth) ak = k_lo;
  };
  for (int i = 0; i < RING - 1 && i < total; i++) load_w();
  hb_pdl_wait();
  hb_pdl_launch();      // not earlier: blocks of kernels further on would hold room on the SMs ahead of those that can run
#pragma unroll
  for (int i = 0; i < RING - 1; i++) {
    if (i < total) load_a();
    hb_cp_async_commit();
  }
  const int n = lane & 15, h = lane >> 4;
  float acc[RP];
#pragma unroll
  for (int r = 0; r < RP; r++) acc[r] = 0.f;
  int step = 0, tile = blockIdx.x, buf = 0;
  for (int i = 0; i < total; i++) {
    hb_cp_async_wait<RING - 2>();
    __syncwarp();
    const uint8_t* st = ring + (size_t)(i % RING) * piece;
    const TW* wr = (const TW*)st + n * (KC + P::PW);
    const TA* ar = (const TA*)(st + P::W_BYTES);
    const int len = min(KC, k_hi - k_lo - step * KC);      // a multiple of 4, or none
    if (len == KC) {
#pragma unroll 4
      for (int k = 0; k < KC; k += 4) {
        const float4 w = hb_load4(wr + k);
#pragma unroll
        for (int r = 0; r < RP; r++) {
          const float4 a = hb_load4(ar + min(h + 2 * r, M - 1) * KC + k);
          acc[r] = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, acc[r]))));
        }
      }
    } else {
      for (int k = 0; k < len; k += 4) {
        const float4 w = hb_load4(wr + k);
#pragma unroll
        for (int r = 0; r < RP; r++) {
          const float4 a = hb_load4(ar + min(h + 2 * r, M - 1) * KC + k);
          acc[r] = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, acc[r]))));
        }
      }
    }
    __syncwarp();                                          // the piece before this one is free: its lanes are all done with it
    if (wi < total) load_w();
    if (ai < total) load_a();
    hb_cp_async_commit();
    if (++step == per_tile) {
#pragma unroll
      for (int r = 0; r < RP; r++) { part[buf][warp][h + 2 * r][n] = acc[r]; acc[r] = 0.f; }
      __syncthreads();                                     // (two buffers: the next tile's sums need not wait for these reads)
      for (int j = tid; j < M * SR_COLS; j += blockDim.x) {
        const int m = j / SR_COLS, c = j % SR_COLS;
        float sum = 0.f;
        for (int sl = 0; sl < slices; sl++) sum += part[buf][sl][m][c];
        if (tile * SR_COLS + c < N) simt_put<TC, TW, EPI>(C + (size_t)m * ldc + tile * SR_COLS + c, sum, colscale, tile * SR_COLS + c);
      }
      step = 0;
      tile += gridDim.x;
      buf ^= 1;
    }
  }
}

static int simt_sms() {
  static int n[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n[dev] = 148;
  return n[dev];
}
// Whether slices get blocks of their own: while the tiles are at most three rounds of two an SM, since a whole-K block of the last,
// partly filled round takes as long as the whole round. us whole / split: 640 tiles (301 x 16,384 x 2,048) 500 / 455, 768 (1,531 x 4,096 x
// 14,336) 4,114 / 3,475, but 1,024 of four slices (512 x 16,384 x 2,048) 699 / 713. Beyond, eight slices still gain some 5 % (2,048 x
// 4,096 x 14,336: 4,841 / 4,628), for 268 MB of partial sums; up to the line they are at most 233 MB. Two slices only where
// the tiles are more than the SMs: 64 x 4,096 x 1,024 took 60 / 77, 301 x 4,096 x 1,024 105 / 84.
static bool simt_splits(int M, int N, int slices) {
  const long tiles = (long)((M + SM_TM - 1) / SM_TM) * ((N + SM_TN - 1) / SM_TN);
  return slices > 1 && tiles <= 6l * simt_sms() && (slices > 2 || tiles > simt_sms());
}

// Floats of workspace that a product of more than SR_ROWS rows can use (0: none; without one it runs unsplit, same bits).
HB_EXPORT long hb_gemm_simt_workspace(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  int depth, slices;
  slice_plan(K, &depth, &slices);
  return simt_splits(M, N, slices) ? (long)slices * M * N : 0;
}

template <typename TA, typename TW, typename TC, int EPI>
static int simt_launch(const TA* A, long lda, const TW* W, long ldw, TC* C, long ldc, int M, int N, int K, const TW* colscale,
                       float* ws, cudaStream_t s) {
  int depth, slices;
  slice_plan(K, &depth, &slices);
  const bool bytes16 = !(((uintptr_t)A | (uintptr_t)W) & 15) && !((lda * sizeof(TA)) & 15) && !((ldw * sizeof(TW)) & 15);
  cudaError_t e;
  // 16-byte pieces of both operands' rows: a slice starts at a multiple of 64, so K alone decides about the last one
  if (M <= SR_ROWS && bytes16 && (K * sizeof(TA)) % 16 == 0 && (K * sizeof(TW)) % 16 == 0) {
    const int tiles = (N + SR_COLS - 1) / SR_COLS, most = 2 * simt_sms(), blocks = tiles < most ? tiles : most;
    // pieces 64 deep with up to four slices, 32 deep with more
#define HB_SIMT_ROWS(RP, KC, RING)                                                                                            \
  do {                                                                                                                        \
    auto kern = simt_rows_kernel<TA, TW, TC, EPI, RP, KC, RING>;                                                              \
    static_assert((KC == 64 ? 4 : 8) * 4 * RowsPiece<float, float, KC>::bytes(8) <= SR_MOST, "two blocks an SM");              \
    const size_t smem = (size_t)slices * RING * RowsPiece<TA, TW, KC>::bytes(M);                                              \
    e = smem > 40 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SR_MOST) : cudaSuccess;    \
    if (e == cudaSuccess) e = hb_launch(kern, blocks, 32 * slices, smem, s, A, lda, W, ldw, C, ldc, M, N, K, colscale, depth); \
  } while (0)
    if (slices <= 4) {
      if (M <= 2) HB_SIMT_ROWS(1, 64, 5);
      else if (M <= 4) HB_SIMT_ROWS(2, 64, 5);
      else HB_SIMT_ROWS(4, 64, 4);
    } else {
      if (M <= 2) HB_SIMT_ROWS(1, 32, 5);
      else if (slices * 5 * RowsPiece<TA, TW, 32>::bytes(M) <= SR_MOST && M <= 4) HB_SIMT_ROWS(2, 32, 5);
      else if (M <= 4) HB_SIMT_ROWS(2, 32, 4);
      else HB_SIMT_ROWS(4, 32, 4);
    }
#undef HB_SIMT_ROWS
    if (e != cudaSuccess) HB_FAIL("hb_gemm_simt: %s", cudaGetErrorString(e));
    return 0;
  }
  const bool vec = bytes16 && (K & 3) == 0, split = ws && simt_splits(M, N, slices);
  const dim3 grid((N + SM_TN - 1) / SM_TN, (M + SM_TM - 1) / SM_TM, split ? slices : 1);
#define HB_SIMT_ARGS grid, 128, 0, s, A, lda, W, ldw, C, ldc, M, N, K, colscale, ws, depth
  if (split) {
    e = vec ? hb_launch(simt_tile_kernel<TA, TW, float, 0, false, true>, grid, 128, 0, s, A, lda, W, ldw, (float*)nullptr, ldc, M, N, K, colscale, ws, depth)
            : hb_launch(simt_tile_kernel<TA, TW, float, 0, false, false>, grid, 128, 0, s, A, lda, W, ldw, (float*)nullptr, ldc, M, N, K, colscale, ws, depth);
    if (e == cudaSuccess)
      e = hb_launch(simt_reduce_kernel<TW, TC, EPI>, (unsigned)(((size_t)M * N + 255) / 256), 256, 0, s, (const float*)ws, C, ldc, M, N, slices, colscale);
  } else {
    e = vec ? hb_launch(simt_tile_kernel<TA, TW, TC, EPI, true, true>, HB_SIMT_ARGS) : hb_launch(simt_tile_kernel<TA, TW, TC, EPI, true, false>, HB_SIMT_ARGS);
  }
#undef HB_SIMT_ARGS
  if (e != cudaSuccess) HB_FAIL("hb_gemm_simt: %s", cudaGetErrorString(e));
  return 0;
}

static int simt_check(const char* name, int M, int K) {
  if (K <= 0) HB_FAIL("%s: K must be positive", name);
  if ((M + 63) / 64 > 65535) HB_FAIL("%s: M = %d is beyond the grid limit", name, M);
  return 0;
}

// colscale: N values of the weight's element type. workspace: hb_gemm_simt_workspace(M, N, K) floats, or null.
HB_EXPORT int hb_gemm_simt_scaled(const void* A, int a_dt, long lda, const void* W, int w_dt, long ldw, float* C, long ldc,
                                  int M, int N, int K, const void* colscale, float* workspace, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (simt_check("hb_gemm_simt_scaled", M, K)) return -1;
  if (!colscale) HB_FAIL("hb_gemm_simt_scaled: no scale vector");
  int r = -1;
  HB_DISPATCH_2(a_dt, w_dt, "hb_gemm_simt_scaled",
                (r = simt_launch<TA, TB, float, 2>((const TA*)A, lda, (const TB*)W, ldw, C, ldc, M, N, K, (const TB*)colscale, workspace, s)));
  if (r) return r;
  HB_CHECK_LAUNCH("hb_gemm_simt_scaled");
  return 0;
}

HB_EXPORT int hb_gemm_simt(const void* A, int a_dt, long lda, const void* W, int w_dt, long ldw, void* C, int c_dt, long ldc,
                           int M, int N, int K, int epi, float* workspace, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (simt_check("hb_gemm_simt", M, K)) return -1;
  if (epi != 0 && epi != 1) HB_FAIL("hb_gemm_simt: unknown epilogue %d", epi);
  if (epi == 1 && c_dt != HB_F32) HB_FAIL("hb_gemm_simt: accumulating into C needs a 32-bit C");
  if (c_dt != HB_F32 && c_dt != HB_BF16) HB_FAIL("hb_gemm_simt: unknown C dtype code %d", c_dt);
  int r = -1;
#define HB_SIMT_CALL(TC, EPI) (r = simt_launch<TA, TB, TC, EPI>((const TA*)A, lda, (const TB*)W, ldw, (TC*)C, ldc, M, N, K, (const TB*)nullptr, workspace, s))
  if (epi == 1) HB_DISPATCH_2(a_dt, w_dt, "hb_gemm_simt", HB_SIMT_CALL(float, 1));
  else if (c_dt == HB_F32) HB_DISPATCH_2(a_dt, w_dt, "hb_gemm_simt", HB_SIMT_CALL(float, 0));
  else HB_DISPATCH_2(a_dt, w_dt, "hb_gemm_simt", HB_SIMT_CALL(__nv_bfloat16, 0));
#undef HB_SIMT_CALL
  if (r) return r;
  HB_CHECK_LAUNCH("hb_gemm_simt");
  return 0;
}
