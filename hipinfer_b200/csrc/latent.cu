// The helpers of latent attention: keys and values of all heads are functions of one latent vector per token, so that
// the cache keeps the latent (R wide) and one rotated key part (Dr wide, shared by all heads) per token, and attention
// runs in the latent's space: with k_h = Wuk_h c and v_h = Wuv_h c,
//     q_h . k_h = (Wuk_h^T q_h) . c          the query is taken into the latent's space, once per row
//     sum_j p_j v_hj = Wuv_h (sum_j p_j c_j)  the values are projected after the sum over keys, once per row
// so a row's attention is one pass over [c | kr] rows with queries R + Dr wide and values the first R columns.
//
// latent_prepare_kernel: from the 32-bit result of the first product (row = [.. cq_raw (Rq) .. c_raw (R) .. kr_raw (Dr) ..])
//   cq = cq_raw / rms(cq_raw) * wq      -> cq_out [T][Rq]
//   c  = c_raw / rms(c_raw) * wc        -> the token's cache row, columns [0, R)
//   kr = rotated(kr_raw)                -> the token's cache row, columns [R, R + Dr)   (pairs (2i, 2i + 1), i < rot / 2,
//                                          with pairing 1; pairs (i, i + rot / 2) with pairing 0)
//   root mean squares with eps inside the root, all 32-bit, rounded once.
// heads_linear_kernel: out[t, h, n] = sum_k a[t, h, k] Wt[h][k][n] (32-bit a, 32-bit sums), optionally times
//   sigmoid(gate[t, h, n]) (or of one number per head, gate[t, h]); and, where asked, the `tail` columns after a's K are
//   rotated the same way and copied behind out's N columns (the rotated part of a query).
#include "common.cuh"

template <typename TW, typename TO>
__global__ void __launch_bounds__(256) latent_prepare_kernel(const float* proj, long ld, int cq_off, int c_off,
                                                             int kr_off, const TW* __restrict__ wq, const TW* __restrict__ wc,
                                                             const int* __restrict__ pos, const int* __restrict__ slot_map,
                                                             const float2* __restrict__ table, int rot, float eps,
                                                             TO* __restrict__ cq_out, TO* __restrict__ cache, int Rq, int R,
                                                             int Dr, int page_size, int pairing) {
  __shared__ float sh[32];
  hb_pdl_launch();
  hb_pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x;
  const float* row = proj + (size_t)t * ld;
  float ss = 0.f;
  for (int i = tid; i < Rq; i += 256) ss = fmaf(row[cq_off + i], row[cq_off + i], ss);
  const float fq = rsqrtf(hb_block_sum(ss, sh) / (float)Rq + eps);
  for (int i = tid; i < Rq; i += 256) cq_out[(size_t)t * Rq + i] = hb_from_float<TO>(row[cq_off + i] * fq * hb_to_float(wq[i]));
  const int slot = slot_map ? slot_map[t] : -1;
  if (slot < 0) return;
  ss = 0.f;
  for (int i = tid; i < R; i += 256) ss = fmaf(row[c_off + i], row[c_off + i], ss);
  const float fc = rsqrtf(hb_block_sum(ss, sh) / (float)R + eps);
  TO* dst = cache + (size_t)slot * (R + Dr);      // one head a page: the slot is the row
  for (int i = tid; i < R; i += 256) dst[i] = hb_from_float<TO>(row[c_off + i] * fc * hb_to_float(wc[i]));
  const int half = rot >> 1;
  const float2* cs = table + (size_t)pos[t] * half;
  for (int i = tid; i < half; i += 256) {
    const int ia = pairing ? 2 * i : i, ib = pairing ? 2 * i + 1 : i + half;
    const float u = row[kr_off + ia], v = row[kr_off + ib];
    const float2 c = cs[i];
    dst[R + ia] = hb_from_float<TO>(__fsub_rn(__fmul_rn(u, c.x), __fmul_rn(v, c.y)));
    dst[R + ib] = hb_from_float<TO>(__fadd_rn(__fmul_rn(v, c.x), __fmul_rn(u, c.y)));
  }
  for (int i = rot + tid; i < Dr; i += 256) dst[R + i] = hb_from_float<TO>(row[kr_off + i]);
}

HB_EXPORT int hb_latent_prepare(const float* proj, long ld, int cq_off, int c_off, int kr_off, const void* wq, const void* wc,
                                int w_dt, const int* pos, const int* slot_map, const void* table, int rot, float eps,
                                void* cq_out, void* cache, int o_dt, int T, int Rq, int R, int Dr, int page_size, int pairing,
                                cudaStream_t s) {
  if (T <= 0) return 0;
  if (rot < 0 || rot > Dr || (rot & 1)) HB_FAIL("hb_latent_prepare: %d rotated dimensions of %d", rot, Dr);
  HB_DISPATCH_2(w_dt, o_dt, "hb_latent_prepare",
                (hb_launch(latent_prepare_kernel<TA, TB>, T, 256, 0, s, proj, ld, cq_off, c_off, kr_off, (const TA*)wq,
                           (const TA*)wc, pos, slot_map, (const float2*)table, rot, eps, (TB*)cq_out, (TB*)cache, Rq, R, Dr,
                           page_size, pairing)));
  HB_CHECK_LAUNCH("hb_latent_prepare");
  return 0;
}

constexpr int HL_TM = 8, HL_THREADS = 128, HL_TN = 32, HL_KZ = HL_THREADS / HL_TN;

// A block owns HL_TM rows, one head and HL_TN output columns; its threads are HL_TN columns x HL_KZ interleaved slices of
// k, which meet in shared memory: few rows still fill the machine, and a thread's loads of the weight are independent of one
// another. The sums are those of heads_linear_vec_kernel, bit for bit: a row's result does not depend on how many rows there are.
template <typename TW, typename TO>
__global__ void __launch_bounds__(HL_THREADS) heads_linear_kernel(const float* a, long lda, long a_head,
                                                                  const TW* __restrict__ wt, TO* __restrict__ out, long ldo,
                                                                  long o_head, int T, int K, int N,
                                                                  const float* gate, long ld_gate, int gate_off,
                                                                  int tail, int rot, const int* __restrict__ pos,
                                                                  const float2* __restrict__ table,
                                                                  const int* __restrict__ row_list, const int* __restrict__ row_req,
                                                                  const int* __restrict__ q_len, int row_limit, int pairing,
                                                                  int gate_per_head) {
  extern __shared__ float hl_a[];      // [HL_TM][K + tail], then [HL_KZ][HL_TM][HL_TN] partial sums
  hb_pdl_launch();
  hb_pdl_wait();
  const int h = blockIdx.y, t0 = blockIdx.z * HL_TM, nl = threadIdx.x % HL_TN, kz = threadIdx.x / HL_TN;
  const int n = blockIdx.x * HL_TN + nl;
  const int KT_ = K + tail, rows = min(HL_TM, T - t0);
  float* red = hl_a + HL_TM * KT_;
  auto row_of = [&](int r) { return row_list ? row_list[t0 + r] : t0 + r; };      // the row's place in a, out, gate and pos
  // rows of requests that bring row_limit rows or more belong to another path: a block all of whose rows do is idle
  unsigned skip = 0;
  if (q_len)
    for (int r = 0; r < rows; r++) skip |= (q_len[row_req[row_of(r)]] >= row_limit ? 1u : 0u) << r;
  if (q_len && skip == (1u << rows) - 1u) return;
  for (int i = threadIdx.x; i < rows * KT_; i += HL_THREADS) {
    const int r = i / KT_, k = i - r * KT_;
    hl_a[r * KT_ + k] = a[(size_t)row_of(r) * lda + (size_t)h * a_head + k];
  }
  __syncthreads();
  // partial sums as the lanes of heads_linear_vec_kernel make them: chain l of a row has the k = l, l + 32, ..; chain kz + 4 u is acc[.][u]
  float acc[HL_TM][8];
#pragma unroll
  for (int r = 0; r < HL_TM; r++)
#pragma unroll
    for (int u = 0; u < 8; u++) acc[r][u] = 0.f;
  if (n < N) {
    const TW* w = wt + (size_t)h * K * N + n;
    int k = kz;
    for (; k + 28 < K; k += 32) {
      float wv[8];
#pragma unroll
      for (int u = 0; u < 8; u++) wv[u] = hb_to_float(w[(size_t)(k + 4 * u) * N]);
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int r = 0; r < HL_TM; r++) acc[r][u] = fmaf(hl_a[r * KT_ + k + 4 * u], wv[u], acc[r][u]);
    }
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (k + 4 * u < K) {
        const float wv = hb_to_float(w[(size_t)(k + 4 * u) * N]);
#pragma unroll
        for (int r = 0; r < HL_TM; r++) acc[r][u] = fmaf(hl_a[r * KT_ + k + 4 * u], wv, acc[r][u]);
      }
  }
  // .. and added as the lanes' butterfly adds them: chains 16 apart, then 8, 4, 2 and 1 (the last two between the threads)
#pragma unroll
  for (int r = 0; r < HL_TM; r++)
    red[(kz * HL_TM + r) * HL_TN + nl] = ((acc[r][0] + acc[r][4]) + (acc[r][2] + acc[r][6])) + ((acc[r][1] + acc[r][5]) + (acc[r][3] + acc[r][7]));
  __syncthreads();
  if (n < N) {
    // thread (nl, kz) finishes rows kz, kz + HL_KZ, ...
    for (int r = kz; r < rows; r += HL_KZ) {
      if (skip >> r & 1) continue;
      const float* z = red + r * HL_TN + nl;
      float o = (z[0] + z[2 * HL_TM * HL_TN]) + (z[HL_TM * HL_TN] + z[3 * HL_TM * HL_TN]);
      if (gate) o *= 1.f / (1.f + expf(-gate[(size_t)row_of(r) * ld_gate + gate_off + (gate_per_head ? (size_t)h : (size_t)h * N + n)]));
      out[(size_t)row_of(r) * ldo + (size_t)h * o_head + n] = hb_from_float<TO>(o);
    }
  } else if (n < N + tail && kz == 0) {
    const int j = n - N, half = rot >> 1;
    for (int r = 0; r < rows; r++) {
      if (skip >> r & 1) continue;
      const float* src = hl_a + r * KT_ + K;
      float y = src[j];
      if (j < rot) {
        const int i = pairing ? j >> 1 : (j < half ? j : j - half);
        const bool second = pairing ? (j & 1) : (j >= half);
        const float2 c = table[(size_t)pos[row_of(r)] * half + i];
        const float u = src[pairing ? 2 * i : i], v = src[pairing ? 2 * i + 1 : i + half];
        y = second ? __fadd_rn(__fmul_rn(v, c.x), __fmul_rn(u, c.y)) : __fsub_rn(__fmul_rn(u, c.x), __fmul_rn(v, c.y));
      }
      out[(size_t)row_of(r) * ldo + (size_t)h * o_head + n] = hb_from_float<TO>(y);
    }
  }
}

// The same for N a multiple of 8 and rows of the weight on 16-byte boundaries: a warp owns HV_ROWS rows, one head and eight output
// columns, its lanes the k's lane, lane + 32, ..: a lane's loads of the weight are 16 bytes each, eight of them in flight, and
// asked for before the wait for the kernel ahead. The lanes' sums meet by a transposing butterfly that leaves lane l the sum
// of (row l / 8, column l % 8): 31 shuffles for 32 sums, no shared memory, no barrier. Bound by latency: the weight of a head is
// 32 KB (4 rows, 32 heads of 256 x 64: 13.5 us with two-byte loads of one k after the other, 4.4 now). row_list: the rows the
// call is for (indices in a, out, gate and pos), or null: all T.
constexpr int HV_ROWS = 4, HV_K = 8;
struct HeadsVec {
  const float* a; long lda, a_head;
  const void* wt;
  void* out; long ldo, o_head;
  int T, K, N;
  const float* gate; long ld_gate;
  int gate_off, tail, rot;
  const int* pos; const float2* table;
  const int *row_list, *row_req, *q_len;
  int row_limit, pairing, gate_per_head;
};

template <typename TW> __device__ __forceinline__ void hv_load8(const TW* p, float* v);
template <> __device__ __forceinline__ void hv_load8<float>(const float* p, float* v) {
  *(float4*)v = *(const float4*)p;
  *(float4*)(v + 4) = *(const float4*)(p + 4);
}
template <> __device__ __forceinline__ void hv_load8<__nv_bfloat16>(const __nv_bfloat16* p, float* v) {
  const uint4 r = *(const uint4*)p;
  const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] = __uint_as_float(u[i] << 16);
    v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
  }
}

template <typename TW, typename TO>
__global__ void __launch_bounds__(256) heads_linear_vec_kernel(HeadsVec A) {
  hb_pdl_launch();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i0 = blockIdx.z * HV_ROWS;
  const int n0 = (blockIdx.x * 8 + warp) * 8, K = A.K, N = A.N;
  const bool tail_block = (int)blockIdx.x * 64 >= N;
  int row[HV_ROWS];
  bool on[HV_ROWS], any = false;
#pragma unroll
  for (int r = 0; r < HV_ROWS; r++) {
    on[r] = i0 + r < A.T;
    row[r] = on[r] ? (A.row_list ? A.row_list[i0 + r] : i0 + r) : 0;
    if (on[r] && A.q_len && A.q_len[A.row_req[row[r]]] >= A.row_limit) on[r] = false;
    any |= on[r];
  }
  if (!any || (!tail_block && n0 >= N)) {
    if ((blockIdx.x | blockIdx.y | blockIdx.z) == 0) hb_pdl_wait();      // the grid never ends before the one ahead of it
    return;
  }
  if (tail_block) {                       // the rotated columns behind the product's
    hb_pdl_wait();
    const int half = A.rot >> 1;
#pragma unroll
    for (int r = 0; r < HV_ROWS; r++) {
      if (!on[r]) continue;
      const float* src = A.a + (size_t)row[r] * A.lda + (size_t)h * A.a_head + K;
      for (int j = threadIdx.x; j < A.tail; j += 256) {
        float y = src[j];
        if (j < A.rot) {
          const int i = A.pairing ? j >> 1 : (j < half ? j : j - half);
          const bool second = A.pairing ? (j & 1) : (j >= half);
          const float2 c = A.table[(size_t)A.pos[row[r]] * half + i];
          const float u = src[A.pairing ? 2 * i : i], v = src[A.pairing ? 2 * i + 1 : i + half];
          y = second ? __fadd_rn(__fmul_rn(v, c.x), __fmul_rn(u, c.y)) : __fsub_rn(__fmul_rn(u, c.x), __fmul_rn(v, c.y));
        }
        ((TO*)A.out)[(size_t)row[r] * A.ldo + (size_t)h * A.o_head + N + j] = hb_from_float<TO>(y);
      }
    }
    return;
  }
  const TW* w = (const TW*)A.wt + (size_t)h * K * N + n0;
  float acc[HV_ROWS * 8];
#pragma unroll
  for (int i = 0; i < HV_ROWS * 8; i++) acc[i] = 0.f;
  for (int k0 = 0; k0 < K; k0 += 32 * HV_K) {
    float wv[HV_K][8];
#pragma unroll
    for (int i = 0; i < HV_K; i++) {
      const int k = k0 + i * 32 + lane;
      if (k < K) hv_load8<TW>(w + (size_t)k * N, wv[i]);
    }
    if (k0 == 0) hb_pdl_wait();
    float av[HV_ROWS][HV_K];
#pragma unroll
    for (int r = 0; r < HV_ROWS; r++)
#pragma unroll
      for (int i = 0; i < HV_K; i++) {
        const int k = k0 + i * 32 + lane;
        av[r][i] = on[r] && k < K ? A.a[(size_t)row[r] * A.lda + (size_t)h * A.a_head + k] : 0.f;
      }
#pragma unroll
    for (int i = 0; i < HV_K; i++)
      if (k0 + i * 32 + lane < K)
#pragma unroll
        for (int r = 0; r < HV_ROWS; r++)
#pragma unroll
          for (int c = 0; c < 8; c++) acc[r * 8 + c] = fmaf(av[r][i], wv[i][c], acc[r * 8 + c]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {      // after the step of o a lane keeps the sums whose bit o is its own
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < 16; i++)
      if (i < o) {
        const float send = up ? acc[i] : acc[i + o], kept = up ? acc[i + o] : acc[i];
        acc[i] = kept + __shfl_xor_sync(0xffffffffu, send, o);
      }
  }
  const int r = lane >> 3, n = n0 + (lane & 7);
  bool mine = false;
  int t = 0;
#pragma unroll
  for (int i = 0; i < HV_ROWS; i++)
    if (i == r) { mine = on[i]; t = row[i]; }
  if (!mine) return;
  float y = acc[0];
  if (A.gate) y *= 1.f / (1.f + expf(-A.gate[(size_t)t * A.ld_gate + A.gate_off + (A.gate_per_head ? (size_t)h : (size_t)h * N + n)]));
  ((TO*)A.out)[(size_t)t * A.ldo + (size_t)h * A.o_head + n] = hb_from_float<TO>(y);
}

// Whether the rows are so few that latency bounds them. The kernel above pays 31 shuffles for 32 sums, whatever K is, and reads
// a head's weight once for 4 rows; the one before it fills the SMs better when there are many. The line lies where the two took
// the same time, in warps of the kernel above: up to K = 64 between 1,280 and 1,536 (32 heads of 64 x 64, 16 rows: 2.3 us against
// 3.2; 24 rows 3.7 against 3.4), at K = 128 between 3,072 and 4,096 (16 heads of 128 x 512, 8 rows: 5.2 against 6.4; 16 rows 10.0
// against 9.4), at K = 256 and 512 between 5,120 and 6,144 (32 heads of 256 x 64, 64 rows: 12.4 against 17.5; 128 rows 23.7
// against 23.2, 2,048 rows 398 against 189).
static_assert(HL_KZ == 4, "the order of the sums");
static bool hv_few(int T, int H, int K, int N) {
  const long warps = (long)((T + HV_ROWS - 1) / HV_ROWS) * H * (N / 8);
  return warps < 24l * (K < 64 ? 64 : K < 216 ? K : 216);
}

// a float32 [T][lda], head h's K (+ tail) inputs at column h * a_head; wt [H][K][N]; out [T][ldo], head h's N (+ tail)
// outputs at column h * o_head.
HB_EXPORT int hb_heads_linear(const float* a, long lda, long a_head, const void* wt, int w_dt, void* out, int o_dt, long ldo,
                              long o_head, int T, int H, int K, int N, const float* gate, long ld_gate, int gate_off, int tail,
                              int rot, const int* pos, const void* table, const int* row_req, const int* q_len, int row_limit,
                              int pairing, int gate_per_head, const int* row_list, cudaStream_t s) {
  if (T <= 0 || H <= 0) return 0;
  if (tail && (!pos || !table || rot > tail || (rot & 1))) HB_FAIL("hb_heads_linear: a rotated tail needs positions and a table");
  const size_t smem = ((size_t)HL_TM * (K + tail) + (size_t)HL_KZ * HL_TM * HL_TN) * sizeof(float);
  if (smem > 96 * 1024) HB_FAIL("hb_heads_linear: K = %d is too wide", K);      // (whichever kernel: the rule below goes by the rows)
  if (N % 8 == 0 && ((uintptr_t)wt & 15) == 0 && H <= 65535 && hv_few(T, H, K, N)) {     // (a row of 8 is 16 or 32 bytes)
    const HeadsVec A{a, lda, a_head, wt, out, ldo, o_head, T, K, N, gate, ld_gate, gate_off, tail, rot, pos, (const float2*)table, row_list,
                     row_req, q_len, row_limit, pairing, gate_per_head};
    const dim3 grid((N + 63) / 64 + (tail ? 1 : 0), H, (T + HV_ROWS - 1) / HV_ROWS);
    HB_DISPATCH_2(w_dt, o_dt, "hb_heads_linear", (hb_launch(heads_linear_vec_kernel<TA, TB>, grid, 256, 0, s, A)));
    HB_CHECK_LAUNCH("hb_heads_linear");
    return 0;
  }
  if ((T + HL_TM - 1) / HL_TM > 65535 || H > 65535) HB_FAIL("hb_heads_linear: the grid is too large");
  dim3 grid((N + tail + HL_TN - 1) / HL_TN, H, (T + HL_TM - 1) / HL_TM);
#define HL_LAUNCH(TW, TO)                                                                                       \
  do {                                                                                                          \
    auto kern = heads_linear_kernel<TW, TO>;                                                                    \
    if (smem + 4096 > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    hb_launch(kern, grid, dim3(HL_THREADS), smem, s, a, lda, a_head, (const TW*)wt, (TO*)out, ldo, o_head, T, K, N, gate,  \
              ld_gate, gate_off, tail, rot, pos, (const float2*)table, row_list, row_req, q_len, row_limit, pairing,     \
              gate_per_head);                                                                                   \
  } while (0)
  HB_DISPATCH_2(w_dt, o_dt, "hb_heads_linear", HL_LAUNCH(TA, TB));
#undef HL_LAUNCH
  HB_CHECK_LAUNCH("hb_heads_linear");
  return 0;
}

// The rows of one request's tokens [0, n) of a cache plane with one head ([page][1][page_size][W]) copied, in the
// order of their positions, into a contiguous buffer [n][W]: the input of a product over a request's whole context.
template <typename TC>
__global__ void __launch_bounds__(256) gather_rows_kernel(const TC* plane, const int* __restrict__ table,
                                                          TC* __restrict__ dst, int n, int W, int page_size) {
  hb_pdl_launch();
  hb_pdl_wait();
  const int vec = 16 / sizeof(TC), cw = W / vec;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < (long)n * cw; i += (long)gridDim.x * 256) {
    const int t = (int)(i / cw), c = (int)(i - (long)t * cw);
    const size_t row = (size_t)table[t / page_size] * page_size + t % page_size;
    ((uint4*)(dst + (size_t)t * W))[c] = ((const uint4*)(plane + row * W))[c];
  }
}

HB_EXPORT int hb_gather_rows(const void* plane, int dt, const int* table, void* dst, int n, int W, int page_size, cudaStream_t s) {
  if (n <= 0) return 0;
  const int esz = dt == HB_F32 ? 4 : 2;
  if ((W * esz) % 16 || (((uintptr_t)plane | (uintptr_t)dst) & 15)) HB_FAIL("hb_gather_rows: rows of %d elements are no whole 16-byte chunks", W);
  const long chunks = (long)n * (W * esz / 16);
  const int blocks = (int)((chunks + 255) / 256 < 2048 ? (chunks + 255) / 256 : 2048);
  HB_DISPATCH_1(dt, "hb_gather_rows", (hb_launch(gather_rows_kernel<TA>, blocks, 256, 0, s, (const TA*)plane, table, (TA*)dst, n, W, page_size)));
  HB_CHECK_LAUNCH("hb_gather_rows");
  return 0;
}
