// The generalized delta rule: a linear recurrence with a state matrix per head, carried from token to token.
//
// Per head, with state S [D key channels][D value channels] (32-bit, in a state slot of the request):
//     u  = k / sqrt(sum(k^2) + unit_eps)
//     S' = diag(w) S - (a * u) (u^T S) + k v^T          (both terms read the old state)
//     o  = S'^T r
//     w  = exp(-decay_scale * sigmoid(w_raw + w_bias)),   a = sigmoid(a_raw + a_bias)
// and then the head's output: o / sqrt(mean(o^2) + eps) * norm_weight * sigmoid(gate_raw).
// r, k, v, a_raw, gate_raw are columns of the 32-bit result of one projection, w_raw of another; everything here
// is 32-bit (expf, the sums, the state); the output is rounded once.
//
// Value channel j of the state, S[:, j], never meets another channel: u^T S and S^T r are sums over key channels.
// So a block owns (request, head) and its threads own value channels; the tokens of the request's portion run in
// order, the state stays on chip from the first to the last of them, and is written back once. Which requests
// and how many tokens comes from device arrays (first row, row count and state slot of each request), so the
// launch is the same for every batch of as many requests and replays from a CUDA graph.
//
//   delta_rule_kernel      four threads share two value channels, each with D / 4 key channels of them in registers; tokens
//                          in chunks, what does not depend on the state a chunk at a time (D = 32, 64, 128); two forms.
//   delta_rule_any_kernel  any D: the state in shared memory, a thread per value channel.
#include "common.cuh"

struct DeltaArgs {
  const float* proj;     // [T][ld]: columns r_off, k_off, v_off, a_off, g_off (each heads * D wide)
  long ld;
  int r_off, k_off, v_off, a_off, g_off;
  const float* w_raw;    // [T][ldw]
  long ldw;
  const void* w_bias;    // [heads * D]
  const void* a_bias;    // [heads * D]
  const void* norm_w;    // [heads * D]
  float* state;          // [slots][heads][D][D]
  const int* q_start;    // [R]
  const int* q_len;      // [R]
  const int* slot;       // [R]
  void* out;             // [T][heads * D]
  int heads, D;
  float decay_scale, unit_eps, eps;
};

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

// Sum over the first `n` threads' values of a block of up to 256 threads, in a fixed order.
__device__ __forceinline__ float head_sum(float v, float* sh, int nwarps) {
  v = hb_warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < nwarps; i++) t += sh[i];
  return t;
}

template <typename TW, typename TO>
__global__ void delta_rule_any_kernel(DeltaArgs A) {
  extern __shared__ float smem[];
  hb_pdl_launch();
  hb_pdl_wait();
  const int D = A.D, h = blockIdx.x, req = blockIdx.y, j = threadIdx.x;
  const int nw = (blockDim.x + 31) >> 5;
  float* S = smem;                 // [D][D]
  float* vr = S + (size_t)D * D;   // r, w, au, k, u: [5][D]
  float* vw = vr + D, *vau = vw + D, *vk = vau + D, *vu = vk + D;
  float* sh = vu + D;              // [32]
  const bool on = j < D;
  float* Sg = A.state + ((size_t)A.slot[req] * A.heads + h) * D * D;
  if (on) for (int i = 0; i < D; i++) S[i * D + j] = Sg[i * D + j];
  const int t0 = A.q_start[req], n = A.q_len[req];
  const TW* wb = (const TW*)A.w_bias, *ab = (const TW*)A.a_bias, *nwt = (const TW*)A.norm_w;
  const int c = h * D + j;
  for (int t = t0; t < t0 + n; t++) {
    const float* row = A.proj + (size_t)t * A.ld;
    float kj = 0.f, vj = 0.f;
    if (on) {
      kj = row[A.k_off + c];
      vj = row[A.v_off + c];
    }
    const float kk = head_sum(kj * kj, sh, nw);     // (its first barrier also ends the token before)
    if (on) {
      const float uj = kj / sqrtf(kk + A.unit_eps);
      vr[j] = row[A.r_off + c];
      vw[j] = expf(-A.decay_scale * sigmoidf_(A.w_raw[(size_t)t * A.ldw + c] + hb_to_float(wb[c])));
      vau[j] = sigmoidf_(row[A.a_off + c] + hb_to_float(ab[c])) * uj;
      vk[j] = kj;
      vu[j] = uj;
    }
    __syncthreads();
    float o = 0.f;
    if (on) {
      float sa = 0.f;
      for (int i = 0; i < D; i++) sa = fmaf(vu[i], S[i * D + j], sa);
      for (int i = 0; i < D; i++) {
        const float s = fmaf(vk[i], vj, fmaf(vw[i], S[i * D + j], -vau[i] * sa));
        S[i * D + j] = s;
        o = fmaf(s, vr[i], o);
      }
    }
    const float oo = head_sum(o * o, sh, nw);
    if (on) {
      const float y = o * rsqrtf(oo / (float)D + A.eps) * hb_to_float(nwt[c]) * sigmoidf_(row[A.g_off + c]);
      ((TO*)A.out)[(size_t)t * A.heads * D + c] = hb_from_float<TO>(y);
    }
  }
  if (on) for (int i = 0; i < D; i++) Sg[i * D + j] = S[i * D + j];
}

// A thread holds S[q * NR + i][j], i < NR, of two neighbouring value channels j in registers; the four threads q of a channel
// pair (D = 4 NR) are neighbouring lanes, so the parts of u^T S meet by shuffles (each lane fetches all four and adds them in the
// order of q) and no thread waits for another warp while the state walks. Two channels a thread halve the reads of the token's
// vectors, which (with a barrier a token before that) bounded the walk: one read of 16 bytes serves 8 products instead of 4.
//
// The tokens go by in chunks of CH. What does not depend on the state is made for a chunk at once, a warp per token (the unit
// key, decay and removal rate: a warp sum and two expf), the raw values of a later chunk on their way from global memory
// meanwhile; the chunk's outputs are finished (their parts added, head norm, gate) a warp per token too.
//
// HELP: the first D / 16 warps only WALK, 10 NR multiply-adds a thread and its share of the reads a token, and DR_HELP further warps
// prepare the next chunk and finish the one before beside them, one barrier a chunk: for few blocks, where the walk must not
// stand still (32 heads of 64, two requests, 2,048 tokens: 598 us with a barrier a token, 556 without, 551 with the helpers: the walk
// itself is what is left). It keeps two chunks of 16 in shared memory, two blocks an SM at D = 64. Without (HELP false) the same warps
// do both in turn, for short chunks in an eighth of the shared memory, so that an SM holds more blocks: for many of them (64
// requests of a token each, 32 heads of 64, took 35 us with the helpers, 16 without). Both do the same arithmetic in the same order.
constexpr int DR_Q = 4, DR_HELP = 4;

template <int NR, bool HELP, int CH> struct DeltaCfg {
  static constexpr int D = NR * DR_Q, WALKERS = D / 2 * DR_Q, THREADS = WALKERS + (HELP ? 32 * DR_HELP : 0);
  static constexpr int NW = HELP ? DR_HELP : WALKERS / 32, TPW = CH / NW, CPL = D / 32;      // warps that prepare and finish, tokens of each
  // a vector lies in four parts of NR + 4: the lanes of a warp read four places at once, of banks of their own; the rows of the
  // output's parts are D + 8 apart for the same reason
  static constexpr int SEG = NR + 4, VS = DR_Q * SEG, OS = D + 8, VEC = CH * VS, IN = 5 * VEC + CH * D, OUT = CH * DR_Q * OS;
  static constexpr size_t SMEM = (size_t)(HELP ? 2 : 1) * (IN + OUT) * sizeof(float);
  static_assert(WALKERS % 32 == 0 && TPW * NW == CH && CPL >= 1 && NR % 4 == 0, "chunk, warps and head size must fit");
};

template <typename TW, typename TO, int NR, bool HELP, int CH>
__global__ void __launch_bounds__(DeltaCfg<NR, HELP, CH>::THREADS, HELP || NR > 16 ? 1 : 512 / (8 * NR)) delta_rule_kernel(DeltaArgs A) {
  using C = DeltaCfg<NR, HELP, CH>;
  constexpr int D = C::D, NW = C::NW, TPW = C::TPW, CPL = C::CPL, SEG = C::SEG, VS = C::VS, OS = C::OS, VEC = C::VEC, IN = C::IN, OUT = C::OUT;
  // HELP: [2] inputs of a chunk (r, w, au, k, u [CH][VS] each, v [CH][D]), [2] outputs; else one of each
  extern __shared__ __align__(16) float dr_smem[];
  hb_pdl_launch();
  hb_pdl_wait();
  const int h = blockIdx.x, req = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
  const int t0 = A.q_start[req], n = A.q_len[req], chunks = (n + CH - 1) / CH;
  const int hc = h * D;
  const bool helper = HELP && tid >= C::WALKERS;
  auto inputs = [&](int c) { return dr_smem + (HELP ? (c & 1) * IN : 0); };
  auto outputs = [&](int c) { return dr_smem + (HELP ? 2 * IN + (c & 1) * OUT : IN); };

  // ---------------- what a warp does for its tokens of a chunk (HELP: the helpers alone): warp, warp + NW, ..
  const int warp = HELP ? (tid - C::WALKERS) >> 5 : tid >> 5;
  const TW* wb = (const TW*)A.w_bias, *ab = (const TW*)A.a_bias, *nwt = (const TW*)A.norm_w;
  float pre[TPW][CPL][5];              // raw values: k, r, v, a_raw, w_raw of channels lane, lane + 32, ..
  float gate[TPW][CPL];                // the gate's raw values of the chunk to be finished next
  float cab[CPL], cwb[CPL], cnw[CPL];  // this lane's channels of the two biases and the norm weight
  auto fetch_gate = [&](int base) {
#pragma unroll
    for (int x = 0; x < TPW; x++) {
      const int tt = warp + x * NW;
      if (base + tt < n) {
        const float* row = A.proj + (size_t)(t0 + base + tt) * A.ld;
#pragma unroll
        for (int y = 0; y < CPL; y++) gate[x][y] = row[A.g_off + hc + lane + 32 * y];
      }
    }
  };
  auto fetch = [&](int base) {
#pragma unroll
    for (int x = 0; x < TPW; x++) {
      const int tt = warp + x * NW;
      if (base + tt < n) {
        const float* row = A.proj + (size_t)(t0 + base + tt) * A.ld;
        const float* wrow = A.w_raw + (size_t)(t0 + base + tt) * A.ldw;
#pragma unroll
        for (int y = 0; y < CPL; y++) {
          const int c = hc + lane + 32 * y;
          pre[x][y][0] = row[A.k_off + c];
          pre[x][y][1] = row[A.r_off + c];
          pre[x][y][2] = row[A.v_off + c];
          pre[x][y][3] = row[A.a_off + c];
          pre[x][y][4] = wrow[c];
        }
      }
    }
  };
  auto prepare = [&](int c) {          // the fetched chunk's vectors into shared memory
    float* vr = inputs(c), *vw = vr + VEC, *vau = vw + VEC, *vk = vau + VEC, *vu = vk + VEC, *vv = vu + VEC;
#pragma unroll
    for (int x = 0; x < TPW; x++) {
      const int tt = warp + x * NW;
      if (c * CH + tt < n) {                                 // (uniform over the warp)
        float kk = 0.f;
#pragma unroll
        for (int y = 0; y < CPL; y++) kk = fmaf(pre[x][y][0], pre[x][y][0], kk);
        kk = hb_warp_sum(kk);
        const float inv = 1.f / sqrtf(kk + A.unit_eps);
#pragma unroll
        for (int y = 0; y < CPL; y++) {
          const int cl = lane + 32 * y, at = tt * VS + cl / NR * SEG + cl % NR;
          const float kj = pre[x][y][0], uj = kj * inv;
          vk[at] = kj;
          vu[at] = uj;
          vr[at] = pre[x][y][1];
          vv[tt * D + cl] = pre[x][y][2];
          vau[at] = sigmoidf_(pre[x][y][3] + cab[y]) * uj;
          vw[at] = expf(-A.decay_scale * sigmoidf_(pre[x][y][4] + cwb[y]));
        }
      }
    }
  };
  auto finish = [&](int c) {           // a walked chunk's outputs: head norm, weight and gate
    const float* vo = outputs(c);
#pragma unroll
    for (int x = 0; x < TPW; x++) {
      const int tt = warp + x * NW;
      if (c * CH + tt < n) {
        float ov[CPL], oo = 0.f;
#pragma unroll
        for (int y = 0; y < CPL; y++) {
          ov[y] = vo[tt * DR_Q * OS + lane + 32 * y];
#pragma unroll
          for (int qq = 1; qq < DR_Q; qq++) ov[y] += vo[(tt * DR_Q + qq) * OS + lane + 32 * y];
          oo = fmaf(ov[y], ov[y], oo);
        }
        oo = hb_warp_sum(oo);
        const float f = rsqrtf(oo / (float)D + A.eps);
        const size_t t = (size_t)(t0 + c * CH + tt);
#pragma unroll
        for (int y = 0; y < CPL; y++) {
          const int cc = hc + lane + 32 * y;
          ((TO*)A.out)[t * A.heads * D + cc] = hb_from_float<TO>(ov[y] * f * cnw[y] * sigmoidf_(gate[x][y]));
        }
      }
    }
  };
  if (!HELP || helper) {
    fetch(0);
#pragma unroll
    for (int y = 0; y < CPL; y++) {
      cab[y] = hb_to_float(ab[hc + lane + 32 * y]);
      cwb[y] = hb_to_float(wb[hc + lane + 32 * y]);
      cnw[y] = hb_to_float(nwt[hc + lane + 32 * y]);
    }
  }
  if (helper) {
    prepare(0);
    fetch(CH);
    __syncthreads();
    for (int c = 0; c < chunks; c++) {
      if (c > 0) finish(c - 1);
      fetch_gate(c * CH);
      if (c + 1 < chunks) {
        prepare(c + 1);
        fetch((c + 2) * CH);
      }
      __syncthreads();
    }
    if (chunks > 0) finish(chunks - 1);
    return;
  }

  // ---------------- the walk
  const int q = lane & 3, j = (tid >> 2) * 2;
  float* Sg = A.state + ((size_t)A.slot[req] * A.heads + h) * D * D;
  float S[NR][2];
#pragma unroll
  for (int i = 0; i < NR; i++) {
    const float2 v = *(const float2*)(Sg + (q * NR + i) * D + j);
    S[i][0] = v.x;
    S[i][1] = v.y;
  }
  if (HELP) __syncthreads();
  for (int ch = 0; ch < chunks; ch++) {
    if (!HELP) {
      prepare(ch);
      __syncthreads();
      fetch_gate(ch * CH);                                   // both in flight during the walk
      if (ch + 1 < chunks) fetch((ch + 1) * CH);
    }
    const float* vr = inputs(ch), *vw = vr + VEC, *vau = vw + VEC, *vk = vau + VEC, *vu = vk + VEC, *vv = vu + VEC;
    float* vo = outputs(ch);
    const int m = min(CH, n - ch * CH);
    for (int tt = 0; tt < m; tt++) {
      const int at = tt * VS + q * SEG;
      float4 u[NR / 4];
#pragma unroll
      for (int i = 0; i < NR / 4; i++) u[i] = *(const float4*)(vu + at + 4 * i);
      const float2 v2 = *(const float2*)(vv + tt * D + j);
      const float vj[2] = {v2.x, v2.y};
      float part[2], sa[2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int i = 0; i < NR / 4; i++) {
          s0 = fmaf(u[i].x, S[4 * i][c], s0); s1 = fmaf(u[i].y, S[4 * i + 1][c], s1);
          s2 = fmaf(u[i].z, S[4 * i + 2][c], s2); s3 = fmaf(u[i].w, S[4 * i + 3][c], s3);
        }
        part[c] = (s0 + s1) + (s2 + s3);
      }
      float all[2][DR_Q];
#pragma unroll
      for (int qq = 0; qq < DR_Q; qq++)
#pragma unroll
        for (int c = 0; c < 2; c++) all[c][qq] = __shfl_sync(0xffffffffu, part[c], qq, DR_Q);
#pragma unroll
      for (int c = 0; c < 2; c++) {
        sa[c] = all[c][0];
#pragma unroll
        for (int qq = 1; qq < DR_Q; qq++) sa[c] += all[c][qq];
      }
      float o[2][4] = {};
#pragma unroll
      for (int i = 0; i < NR / 4; i++) {
        const float4 kk = *(const float4*)(vk + at + 4 * i), ww = *(const float4*)(vw + at + 4 * i);
        const float4 aa = *(const float4*)(vau + at + 4 * i), rr = *(const float4*)(vr + at + 4 * i);
#pragma unroll
        for (int c = 0; c < 2; c++) {
          S[4 * i][c] = fmaf(kk.x, vj[c], fmaf(ww.x, S[4 * i][c], -aa.x * sa[c]));             o[c][0] = fmaf(S[4 * i][c], rr.x, o[c][0]);
          S[4 * i + 1][c] = fmaf(kk.y, vj[c], fmaf(ww.y, S[4 * i + 1][c], -aa.y * sa[c]));     o[c][1] = fmaf(S[4 * i + 1][c], rr.y, o[c][1]);
          S[4 * i + 2][c] = fmaf(kk.z, vj[c], fmaf(ww.z, S[4 * i + 2][c], -aa.z * sa[c]));     o[c][2] = fmaf(S[4 * i + 2][c], rr.z, o[c][2]);
          S[4 * i + 3][c] = fmaf(kk.w, vj[c], fmaf(ww.w, S[4 * i + 3][c], -aa.w * sa[c]));     o[c][3] = fmaf(S[4 * i + 3][c], rr.w, o[c][3]);
        }
      }
      *(float2*)(vo + (tt * DR_Q + q) * OS + j) = make_float2((o[0][0] + o[0][1]) + (o[0][2] + o[0][3]), (o[1][0] + o[1][1]) + (o[1][2] + o[1][3]));
    }
    __syncthreads();
    if (!HELP) finish(ch);
  }
#pragma unroll
  for (int i = 0; i < NR; i++) *(float2*)(Sg + (q * NR + i) * D + j) = make_float2(S[i][0], S[i][1]);
}

enum { DR_RULE = 0, DR_ANY = 1, DR_HELPERS = 2, DR_SHORT = 3 };
// Which form a launch takes. Portions: with helpers while the blocks that an SM then holds (four, two, one for heads of 32, 64, 128)
// are enough for one round; at 128 always, where both hold one and the helpers are 1 to 3 % ahead. 300 tokens of 32 heads, us with
// helpers / without: of 64, 4 requests 122 / 236, 8 280 / 326, 12 420 / 338; of 32, 12 requests 210 / 245; of 128, 4 291 / 306.
// Single tokens: without, but for the few block counts at which the wider block is ahead (32 heads of 64: 1 request 3.30 / 3.07, 4
// 3.33 / 3.95, 8 5.66 / 4.80, 64 35.3 / 16.0; of 32, 8 requests 2.68 / 2.86, 64 14.0 / 6.1; of 128, 4 6.2 / 5.7).
static int dr_form(int D, long blocks, bool single) {
  if (single) return D <= 64 && blocks > 74 && blocks <= (D <= 32 ? 296 : 148) ? DR_HELPERS : DR_SHORT;
  return D > 64 || blocks <= 148 * (D <= 32 ? 4 : 2) ? DR_HELPERS : DR_SHORT;
}

constexpr int dr_short(int NR) { return NR > 16 ? NR / 4 : 4; }      // tokens of a chunk without helpers: one a warp, at least four

template <typename TW, typename TO, int NR, bool HELP, int CH>
static int delta_rule_launch_form(const DeltaArgs& A, dim3 grid, cudaStream_t s) {
  using C = DeltaCfg<NR, HELP, CH>;
  auto kern = delta_rule_kernel<TW, TO, NR, HELP, CH>;
  if (C::SMEM > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) HB_FAIL("hb_delta_rule: %s", cudaGetErrorString(e));
  }
  hb_launch(kern, grid, C::THREADS, C::SMEM, s, A);
  return 0;
}

template <typename TW, typename TO, int NR>
static int delta_rule_launch_reg(const DeltaArgs& A, dim3 grid, int rows, int form, cudaStream_t s) {
  if (form == DR_RULE) form = dr_form(4 * NR, (long)grid.x * grid.y, rows == (int)grid.y);
  if (form == DR_HELPERS) return delta_rule_launch_form<TW, TO, NR, true, 16>(A, grid, s);
  return delta_rule_launch_form<TW, TO, NR, false, dr_short(NR)>(A, grid, s);
}

template <typename TW, typename TO>
static int delta_rule_launch(const DeltaArgs& A, int R, int rows, int form, cudaStream_t s) {
  const dim3 grid(A.heads, R);
  if (!((uintptr_t)A.state & 7)) switch (A.D) {      // (the register kernels read the state in pairs)
    case 32: return delta_rule_launch_reg<TW, TO, 8>(A, grid, rows, form, s);
    case 64: return delta_rule_launch_reg<TW, TO, 16>(A, grid, rows, form, s);
    case 128: return delta_rule_launch_reg<TW, TO, 32>(A, grid, rows, form, s);
    default: break;
  }
  const int threads = (A.D + 31) / 32 * 32;
  const size_t smem = ((size_t)A.D * A.D + 5 * (size_t)A.D + 32) * sizeof(float);
  if (threads > 1024 || smem > 200 * 1024) HB_FAIL("hb_delta_rule: heads of %d are too wide for one block's shared memory", A.D);
  auto kern = delta_rule_any_kernel<TW, TO>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) HB_FAIL("hb_delta_rule: %s", cudaGetErrorString(e));
  }
  hb_launch(kern, grid, threads, smem, s, A);
  return 0;
}

// rows: the step's rows (as many as requests: every portion is a single token). form: 0 by the rule, or the form to run (tests compare
// them): 1 the shared-memory kernel, 2 and 3 the register kernel with and without helpers.
HB_EXPORT int hb_delta_rule(const float* proj, long ld, int r_off, int k_off, int v_off, int a_off, int g_off,
                            const float* w_raw, long ldw, const void* w_bias, const void* a_bias, const void* norm_w,
                            int w_dt, float* state, const int* q_start, const int* q_len, const int* slot, void* out,
                            int out_dt, int R, int heads, int D, float decay_scale, float unit_eps, float eps,
                            int rows, int form, cudaStream_t s) {
  if (R <= 0) return 0;
  if (heads <= 0 || D <= 0) HB_FAIL("hb_delta_rule: %d heads of %d", heads, D);
  if (R > 65535) HB_FAIL("hb_delta_rule: %d requests are beyond the grid limit", R);
  DeltaArgs A{proj, ld, r_off, k_off, v_off, a_off, g_off, w_raw, ldw, w_bias, a_bias, norm_w, state, q_start, q_len, slot,
              out, heads, D, decay_scale, unit_eps, eps};
  int r = -1;
  HB_DISPATCH_2(w_dt, out_dt, "hb_delta_rule", {
    if (form == DR_ANY) {
      const int threads = (D + 31) / 32 * 32;
      const size_t smem = ((size_t)D * D + 5 * (size_t)D + 32) * sizeof(float);
      if (threads > 1024 || smem > 200 * 1024) HB_FAIL("hb_delta_rule: heads of %d are too wide for one block's shared memory", D);
      auto kern = delta_rule_any_kernel<TA, TB>;
      if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) HB_FAIL("hb_delta_rule: %s", cudaGetErrorString(e));
      }
      hb_launch(kern, dim3(heads, R), threads, smem, s, A);
      r = 0;
    } else {
      r = delta_rule_launch<TA, TB>(A, R, rows, form, s);
    }
  });
  if (r) return r;
  HB_CHECK_LAUNCH("hb_delta_rule");
  return 0;
}
