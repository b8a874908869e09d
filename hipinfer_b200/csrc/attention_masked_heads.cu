// Attention of single rows (decoded tokens, short portions) over the paged cache on warp tensor-core instructions: the
// heads that share a kv head are the rows of the MMA tiles, so a key tile is read once for all of them. Mask, sink and
// gate as in attention_masked.cu (the same visibility rule; see there). bfloat16 queries, keys and values.
//
// One CTA of four warps per (tile of 64 ABSOLUTE positions, kv head and tile of 16 MT heads of the group, row); MT = 1 (up to 16
// heads a tile) or 2 (up to 32). The CTAs of HS_SPLIT_TILES = 8 neighbouring tiles are one cluster: a decode step of few
// requests has few tiles, and a CTA that walked four of them in a row kept 20 of 148 SMs busy for 36 us (4 rows of 1,200 keys, 32
// heads, a latent of 256 + 32; 14 us now). CTAs of a cluster that have no tile leave at once, and where no row of the call
// has as many as eight tiles the cluster is smaller; while the call's CTAs are fewer than two an SM, some without a tile stay and share
// the join. With all eight kept to the end many short rows paid for them: 64 rows of 40 keys, 32 heads over 8 kv heads of 64,
// took 35 us, 10.5 before the tiles had CTAs of their own, 7.5 now; 64 rows of 600 keys 78, 62 and 60 us. Within a CTA the warps split the keys for the scores (16 keys each, all heads)
// and the value columns for the sums; scores and probabilities pass through shared memory. The keys are read as soon as the
// block runs, ahead of the wait for the kernel before it, where the whole tile is of earlier steps. Queries lie in shared memory
// (any D that is a multiple of 16); the values may be the first E columns of the key rows (a latent that serves as both), in
// which case no value tile is loaded.
// A cluster joins its tiles through distributed shared memory, every CTA its share of the columns, in the tiles' order; a row
// that one cluster covers is finished there (sink, gate, one rounding), the partial results of a longer row are joined, in the
// splits' order, by a second kernel over the whole machine. What is added to what is a matter of the row's position alone.
#include "tc_common.cuh"

#define HK 64
constexpr int HS_THREADS = 128, HS_SPLIT_TILES = 8;      // (the largest portable cluster)

struct HeadsArgs {
  const __nv_bfloat16* q; long ldq;
  const __nv_bfloat16* kc; long k_page, k_head, k_row;
  const __nv_bfloat16* vc; long v_page, v_head, v_row;
  int alias;                            // values are the first E columns of the key rows
  const int* bt; int bt_stride;
  const int* row_req; const int* pos;
  const int* row_list;                  // the rows this call is for (indices in q, pos, row_req and out), or null: all T
  const int* ctx_len;                   // per request, or null: tokens in the cache before this step
  const float* sink;
  const float* gate; long ld_gate; int gate_off; int gate_mode;
  void* out; long ldo;
  int H, G, D, E, MT, page_size, mask, window, keep_first, chunk;
  float scale;
  const int* q_len; int row_limit;
  float* part;                          // [T][G][ZT][splits][16 MT][E + 4], T by the place in the list
  int G_ZT;                             // head tiles: G * ZT
  int splits, cs, join;                 // clusters of a row, their CTAs, and how many of those stay for the join where they have no tile
  const float* r1; const float* r2;     // [H] or null: r1 ln(1 + r2 (p - j)) is taken off the score
};

__device__ __forceinline__ void hs_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void hs_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t hs_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *(uint32_t*)&v;
}
__host__ __device__ __forceinline__ int hs_tile_count(int p, int lo, int keep) {
  const int last = p / HK, first_win = lo / HK, last_keep = keep > 0 ? (keep - 1) / HK : -1;
  if (first_win <= last_keep + 1) return last + 1;
  return (last_keep + 1) + (last - first_win + 1);
}
__device__ __forceinline__ int hs_tile_at(int i, int lo, int keep) {
  const int first_win = lo / HK, last_keep = keep > 0 ? (keep - 1) / HK : -1;
  if (first_win <= last_keep + 1 || i <= last_keep) return i;
  return first_win + (i - (last_keep + 1));
}

// EU: units of 16 value columns a warp owns.
template <int EU, int MT, typename TO>
__global__ void __launch_bounds__(HS_THREADS) attn_masked_heads_kernel(HeadsArgs A) {
  extern __shared__ __align__(16) uint8_t hs_smem[];
  constexpr int MR = 16 * MT, SP = HK + 4, PP = HK + 8;
  __shared__ long kofs[HK], vofs[HK];
  __shared__ __align__(8) float mls[HS_SPLIT_TILES][MR][2];   // every CTA's maxima and weight sums, put here by that CTA
  hb_pdl_launch();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = lane >> 2, qi = lane & 3;
  const int rank = blockIdx.x % A.cs, split = blockIdx.x / A.cs, ZT = A.G_ZT / A.G, g = blockIdx.y / ZT, z = blockIdx.y % ZT;
  const int tw = blockIdx.z, t = A.row_list ? A.row_list[tw] : tw, rq = A.row_req[t], p = A.pos[t];
  int lo = 0, keep = 0;
  if (A.mask == 1 && A.window > 0) { lo = max(0, p - A.window + 1); keep = min(A.keep_first, p + 1); }
  else if (A.mask == 2 && A.chunk > 0) lo = (p / A.chunk) * A.chunk;
  const int n_tiles = hs_tile_count(p, lo, keep);
  const int n_splits_row = (n_tiles + HS_SPLIT_TILES - 1) / HS_SPLIT_TILES;       // a matter of the row's position alone
  const int n_here = min(A.cs, n_tiles - split * HS_SPLIT_TILES);                 // (one cluster a row where cs is less than eight)
  const int n_join = n_here > 0 ? max(n_here, A.join) : 0;
  const bool has = rank < n_here;
  // nothing for this CTA to do: it leaves (the cluster's barriers are of the CTAs that have not left, and nobody writes to it)
  if ((A.q_len && A.q_len[rq] >= A.row_limit) || rank >= n_join) {
    if ((blockIdx.x | blockIdx.y | blockIdx.z) == 0) hb_pdl_wait();                // the grid never ends before the one ahead of it
    return;
  }
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");            // this CTA runs: the others may write to it
  const int D = A.D, E = A.E, HG = A.H / A.G, ps = A.page_size;
  const int KP = D + 8, VP = A.alias ? KP : E + 8;
  const int h0 = z * MR, nh = min(MR, HG - h0);
  __nv_bfloat16* Qs = (__nv_bfloat16*)hs_smem;              // [MR][KP]
  __nv_bfloat16* Ks = Qs + MR * KP;                          // [HK][KP]
  __nv_bfloat16* Vs = A.alias ? Ks : Ks + HK * KP;           // [HK][VP]
  float* Ss = (float*)(A.alias ? Ks + HK * KP : Vs + HK * VP);     // [MR][SP]
  __nv_bfloat16* Ps = (__nv_bfloat16*)(Ss + MR * SP);        // [MR][PP]
  const int RS = E + 4;                 // a row's sums, then its maximum and weight sum; rows stay 16-byte aligned
  float* stage = (float*)hs_smem;       // [MR][RS] over queries and keys, when these are done with
  const int k0 = has ? hs_tile_at(split * HS_SPLIT_TILES + rank, lo, keep) * HK : 0;
  // where the tile's 64 keys lie, one thread a key
  if (tid < HK) {
    const int kp = k0 + tid;
    const bool vis = has && kp <= p && (kp >= lo || kp < keep);
    const int page = vis ? A.bt[(size_t)rq * A.bt_stride + kp / ps] : -1, off = kp % ps;
    kofs[tid] = page >= 0 ? (long)page * A.k_page + (long)g * A.k_head + (long)off * A.k_row : -1;
    vofs[tid] = page >= 0 ? (long)page * A.v_page + (long)g * A.v_head + (long)off * A.v_row : -1;
  }
  __syncthreads();
  auto load_rows = [&](__nv_bfloat16* dst, int pitch, int pieces, const __nv_bfloat16* src, const long* ofs) {
    const int dk = HS_THREADS / pieces, dc = HS_THREADS - dk * pieces;
    int kr = tid / pieces, c = tid - kr * pieces;
    while (kr < HK) {
      __nv_bfloat16* d = dst + kr * pitch + c * 8;
      const long o = ofs[kr];
      if (o >= 0) hs_cp16((uint32_t)__cvta_generic_to_shared(d), src + o + c * 8);
      else *(uint4*)d = make_uint4(0u, 0u, 0u, 0u);
      kr += dk;
      c += dc;
      if (c >= pieces) { c -= pieces; kr++; }
    }
  };
  const bool early = has && A.ctx_len && k0 + HK <= A.ctx_len[rq];     // every key of the tile is of an earlier step
  if (early) {
    load_rows(Ks, KP, D / 8, A.kc, kofs);
    if (!A.alias) load_rows(Vs, VP, E / 8, A.vc, vofs);
  }
  hb_pdl_wait();
  if (has && !early) {
    load_rows(Ks, KP, D / 8, A.kc, kofs);
    if (!A.alias) load_rows(Vs, VP, E / 8, A.vc, vofs);
  }
  if (has) {    // the queries of the tile's heads (rows beyond the group's heads are zero)
    const __nv_bfloat16* qrow = A.q + (size_t)t * A.ldq + ((size_t)g * HG + h0) * D;
    const int CQ = D / 8, dr = HS_THREADS / CQ, dc = HS_THREADS - dr * CQ;
    int r = tid / CQ, c = tid - r * CQ;
    while (r < MR) {
      if (r < nh) hs_cp16((uint32_t)__cvta_generic_to_shared(Qs + r * KP + c * 8), qrow + (size_t)r * D + c * 8);
      else *(uint4*)(Qs + r * KP + c * 8) = make_uint4(0u, 0u, 0u, 0u);
      r += dr;
      c += dc;
      if (c >= CQ) { c -= CQ; r++; }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // scores: this warp's 16 keys against all heads, in units of log 2 (scale * log2(e) folded into one factor)
    float sc[MT][2][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int j = 0; j < 2; j++) sc[m][j][0] = sc[m][j][1] = sc[m][j][2] = sc[m][j][3] = 0.f;
    const uint32_t q_addr = (uint32_t)__cvta_generic_to_shared(Qs + (lane & 15) * KP + (lane >> 4) * 8);
    // lane l gives the row of matrix l / 8: keys (l / 16) * 8 + l % 8, columns ((l / 8) & 1) * 8
    const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(Ks + (warp * 16 + (lane >> 4) * 8 + (lane & 7)) * KP + ((lane >> 3) & 1) * 8);
#pragma unroll 2
    for (int ks = 0; ks < D / 16; ks++) {
      uint32_t b[4];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(k_addr + ks * 32));
#pragma unroll
      for (int m = 0; m < MT; m++) {
        uint32_t a[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(q_addr + (uint32_t)(m * 16 * KP * 2 + ks * 32)));
        hs_mma(sc[m][0], a, b[0], b[1]);
        hs_mma(sc[m][1], a, b[2], b[3]);
      }
    }
    const float sl2 = A.scale * 1.4426950408889634f;
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int kc = warp * 16 + j * 8 + qi * 2 + (c & 1), key = k0 + kc, r = m * 16 + quad + (c >> 1) * 8;
          const bool vis = key <= p && (key >= lo || key < keep);
          float v = vis ? sc[m][j][c] * sl2 : -INFINITY;
          if (A.r1 && vis && r < nh) {
            const size_t head = (size_t)g * HG + h0 + r;
            v -= A.r1[head] * __log2f(fmaf(A.r2[head], (float)(p - key), 1.f));
          }
          Ss[r * SP + kc] = v;
        }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    // a warp per row: probabilities against the tile's maximum, rounded for the value product; their 32-bit sum
#pragma unroll
    for (int i = 0; i < MR / 4; i++) {
      const int r = warp * (MR / 4) + i;
      const float a = Ss[r * SP + lane], b = Ss[r * SP + 32 + lane];
      const float m = hb_warp_max(fmaxf(a, b));
      const float ea = m == -INFINITY ? 0.f : exp2f(a - m), eb = m == -INFINITY ? 0.f : exp2f(b - m);
      const float l = hb_warp_sum(ea + eb);
      Ps[r * PP + lane] = __float2bfloat16_rn(ea);
      Ps[r * PP + 32 + lane] = __float2bfloat16_rn(eb);
      // to every CTA of the join, the CTA itself included
      if (lane < n_join)
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(hb_mapa(&mls[rank][r][0], lane)), "f"(m), "f"(l) : "memory");
    }
    __syncthreads();
    float o[MT][2 * EU][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < 2 * EU; n++) o[m][n][0] = o[m][n][1] = o[m][n][2] = o[m][n][3] = 0.f;
    // lane l gives the row of matrix l / 8: keys (l & 7) + ((l >> 3) & 1) * 8 of a group of 16, columns (l >> 4) * 8 of a pair
    const uint32_t v_addr = (uint32_t)__cvta_generic_to_shared(Vs + ((lane & 7) + ((lane >> 3) & 1) * 8) * VP + warp * EU * 16 + (lane >> 4) * 8);
    const uint32_t p_addr = (uint32_t)__cvta_generic_to_shared(Ps + (lane & 15) * PP + (lane >> 4) * 8);
#pragma unroll
    for (int kk = 0; kk < HK / 16; kk++) {
      uint32_t pf[MT][4];
#pragma unroll
      for (int m = 0; m < MT; m++)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(pf[m][0]), "=r"(pf[m][1]), "=r"(pf[m][2]), "=r"(pf[m][3]) : "r"(p_addr + (uint32_t)((m * 16 * PP + kk * 16) * 2)));
#pragma unroll
      for (int n = 0; n < EU; n++) {
        if ((warp * EU + n) * 16 >= E) break;
        uint32_t b[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(v_addr + (uint32_t)((kk * 16 * VP + n * 16) * 2)));
#pragma unroll
        for (int m = 0; m < MT; m++) {
          hs_mma(o[m][2 * n], pf[m], b[0], b[1]);
          hs_mma(o[m][2 * n + 1], pf[m], b[2], b[3]);
        }
      }
    }
    __syncthreads();                    // queries and keys are done with
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < 2 * EU; n++) {
        const int e = warp * EU * 16 + n * 8 + qi * 2, ra = m * 16 + quad;
        if (e >= E) break;
        *(float2*)(stage + ra * RS + e) = make_float2(o[m][n][0], o[m][n][1]);
        *(float2*)(stage + (ra + 8) * RS + e) = make_float2(o[m][n][2], o[m][n][3]);
      }
  } else {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  hb_cluster_sync();                    // every CTA's sums lie in its stage, its maxima and weight sums in all CTAs' mls
  const uint32_t stage_s = hb_smem_u32(stage);
  const int C4 = E / 4;
  const size_t slot = ((size_t)tw * A.G + g) * ZT + z;
  float* part = n_splits_row > 1 ? A.part + (slot * A.splits + split) * (size_t)MR * RS : nullptr;
  for (int i = rank * HS_THREADS + tid; i < nh * C4; i += n_join * HS_THREADS) {
    const int r = i / C4, e = (i - r * C4) * 4;
    float4 v[HS_SPLIT_TILES];
#pragma unroll
    for (int c = 0; c < HS_SPLIT_TILES; c++)
      if (c < n_here) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(stage_s + (uint32_t)(r * RS + e) * 4), "r"(c));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[c].x), "=f"(v[c].y), "=f"(v[c].z), "=f"(v[c].w) : "r"(at) : "memory");
      }
    float m = -INFINITY, l = 0.f;
#pragma unroll
    for (int c = 0; c < HS_SPLIT_TILES; c++)
      if (c < n_here) m = fmaxf(m, mls[c][r][0]);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < HS_SPLIT_TILES; c++)
      if (c < n_here) {
        const float w = m == -INFINITY ? 0.f : exp2f(mls[c][r][0] - m);
        l = fmaf(mls[c][r][1], w, l);
        a.x = fmaf(v[c].x, w, a.x); a.y = fmaf(v[c].y, w, a.y); a.z = fmaf(v[c].z, w, a.z); a.w = fmaf(v[c].w, w, a.w);
      }
    if (part) {                         // the merge kernel joins the splits of such a row
      *(float4*)(part + r * RS + e) = a;
      if (e == 0) { part[r * RS + E] = m; part[r * RS + E + 1] = l; }
      continue;
    }
    const size_t head = (size_t)g * HG + h0 + r;
    float f = 1.f;
    if (A.sink) {
      const float sk = A.sink[head] * 1.4426950408889634f, m2 = fmaxf(m, sk);     // the maxima are in units of log 2
      f = exp2f(m - m2);
      l = fmaf(l, f, exp2f(sk - m2));
    }
    f = l > 0.f ? f / l : 0.f;
    if (A.gate_mode == 2) f *= 1.f / (1.f + expf(-A.gate[(size_t)t * A.ld_gate + A.gate_off + head]));
    a.x *= f; a.y *= f; a.z *= f; a.w *= f;
    if (A.gate_mode == 1) {
      const float* gp = A.gate + (size_t)t * A.ld_gate + A.gate_off + head * E + e;
      a.x *= 1.f / (1.f + expf(-gp[0])); a.y *= 1.f / (1.f + expf(-gp[1]));
      a.z *= 1.f / (1.f + expf(-gp[2])); a.w *= 1.f / (1.f + expf(-gp[3]));
    }
    TO* op = (TO*)A.out + (size_t)t * A.ldo + head * E + e;
    op[0] = hb_from_float<TO>(a.x); op[1] = hb_from_float<TO>(a.y); op[2] = hb_from_float<TO>(a.z); op[3] = hb_from_float<TO>(a.w);
  }
  hb_cluster_sync();                    // no CTA leaves while its sums may still be read
}

// Joins the key splits of rows that were walked by several CTAs: one thread a (head, 4 value columns). It finds the row's
// maximum and weight sum over the splits (a few cached loads), adds the sink, and sums the splits' columns times
// exp2(split maximum - row maximum) in the splits' order, all loads independent of one another; gate and one rounding
// on the way out. The whole machine takes part: the partial sums of a latent layer's row are as large as a third of
// the keys it read, too much for one CTA to pull through its own loads.
template <typename TO>
__global__ void __launch_bounds__(HS_THREADS) attn_masked_heads_merge_kernel(HeadsArgs A) {
  hb_pdl_launch();
  hb_pdl_wait();
  const int tw = blockIdx.z, t = A.row_list ? A.row_list[tw] : tw, ZT = gridDim.y / A.G, g = blockIdx.y / ZT, z = blockIdx.y % ZT;
  if (A.q_len && A.q_len[A.row_req[t]] >= A.row_limit) return;
  const int E = A.E, MR = 16 * A.MT, HG = A.H / A.G, RS = E + 4, C4 = E / 4;
  const int h0 = z * MR, nh = min(MR, HG - h0);
  const int p = A.pos[t];
  int lo = 0, keep = 0;
  if (A.mask == 1 && A.window > 0) { lo = max(0, p - A.window + 1); keep = min(A.keep_first, p + 1); }
  else if (A.mask == 2 && A.chunk > 0) lo = (p / A.chunk) * A.chunk;
  const int n_parts = (hs_tile_count(p, lo, keep) + HS_SPLIT_TILES - 1) / HS_SPLIT_TILES;
  if (n_parts <= 1) return;                                   // finished by the CTA that walked it
  const int i = blockIdx.x * HS_THREADS + threadIdx.x;
  if (i >= nh * C4) return;
  const int r = i / C4, e = (i - r * C4) * 4;
  const size_t slot = ((size_t)tw * A.G + g) * ZT + z, pstride = (size_t)MR * RS;
  const float* all = A.part + slot * A.splits * pstride + (size_t)r * RS;
  const size_t head = (size_t)g * HG + h0 + r;
  float m = -INFINITY;
  for (int sp = 0; sp < n_parts; sp++) m = fmaxf(m, all[sp * pstride + E]);
  float l = 0.f;
  for (int sp = 0; sp < n_parts; sp++) l = fmaf(all[sp * pstride + E + 1], exp2f(all[sp * pstride + E] - m), l);
  float f = 1.f;
  if (A.sink) {
    const float sk = A.sink[head] * 1.4426950408889634f, m2 = fmaxf(m, sk);     // the maxima are in units of log 2
    f = exp2f(m - m2);
    l = fmaf(l, f, exp2f(sk - m2));
  }
  f = l > 0.f ? f / l : 0.f;
  if (A.gate_mode == 2) f *= 1.f / (1.f + expf(-A.gate[(size_t)t * A.ld_gate + A.gate_off + head]));
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int sp = 0; sp < n_parts; sp++) {
    const float4 v = *(const float4*)(all + sp * pstride + e);
    const float w = exp2f(all[sp * pstride + E] - m);
    a.x = fmaf(v.x, w, a.x); a.y = fmaf(v.y, w, a.y); a.z = fmaf(v.z, w, a.z); a.w = fmaf(v.w, w, a.w);
  }
  a.x *= f; a.y *= f; a.z *= f; a.w *= f;
  if (A.gate_mode == 1) {
    const float* gp = A.gate + (size_t)t * A.ld_gate + A.gate_off + head * E + e;
    a.x *= 1.f / (1.f + expf(-gp[0])); a.y *= 1.f / (1.f + expf(-gp[1]));
    a.z *= 1.f / (1.f + expf(-gp[2])); a.w *= 1.f / (1.f + expf(-gp[3]));
  }
  TO* op = (TO*)A.out + (size_t)t * A.ldo + head * E + e;
  op[0] = hb_from_float<TO>(a.x); op[1] = hb_from_float<TO>(a.y); op[2] = hb_from_float<TO>(a.z); op[3] = hb_from_float<TO>(a.w);
}

static int hs_mt(int HG) { return HG > 16 ? 2 : 1; }
static size_t hs_smem_bytes(int MT, int D, int E, int alias) {
  const size_t MR = 16 * MT;
  const size_t tiles = MR * (D + 8) * 2 + (size_t)HK * (D + 8) * 2 + (alias ? 0 : (size_t)HK * (E + 8) * 2) + MR * (HK + 4) * 4 + MR * (HK + 8) * 2;
  const size_t stage = MR * (E + 4) * 4;
  return tiles > stage ? tiles : stage;
}
// The most tiles a row up to max_pos can have.
static int hs_most_tiles(int mask, int window, int keep_first, int chunk, int max_pos) {
  int worst = max_pos / HK + 1;
  if (mask == 1 && window > 0) {
    const int w = (window - 1 + HK - 1) / HK + 1 + (keep_first > 0 ? (keep_first - 1) / HK + 1 : 0);
    if (w < worst) worst = w;
  } else if (mask == 2 && chunk > 0) {
    const int w = chunk % HK == 0 ? chunk / HK : (chunk - 1 + HK - 1) / HK + 1;
    if (w < worst) worst = w;
  }
  return worst < 1 ? 1 : worst;
}
static int hs_splits(int most_tiles) { return (most_tiles + HS_SPLIT_TILES - 1) / HS_SPLIT_TILES; }

// units of 16 value columns a warp owns for these sizes; 0: not a size the kernel takes
static int hs_units(int H, int G, int D, int E, int alias) {
  if (G <= 0 || H % G || D <= 0 || E <= 0 || D % 16 || E % 16 || D > 1024) return 0;
  const int MT = hs_mt(H / G);
  int eu = 1;
  while (eu <= 16 / MT && eu * 64 < E) eu *= 2;
  if (eu > 16 / MT) return 0;
  if (alias && E > D) return 0;
  if (hs_smem_bytes(MT, D, E, alias) > 200 * 1024) return 0;
  return eu;
}

HB_EXPORT int hb_attn_masked_heads_supported(int H, int G, int D, int E, int alias) { return hs_units(H, G, D, E, alias) ? 1 : 0; }

HB_EXPORT long hb_attn_masked_heads_workspace(int T, int H, int G, int E, int mask, int window, int keep_first, int chunk, int max_pos) {
  const int HG = H / G, MT = hs_mt(HG), ZT = (HG + 16 * MT - 1) / (16 * MT);
  const int splits = hs_splits(hs_most_tiles(mask, window, keep_first, chunk, max_pos));
  if (splits <= 1) return 0;
  return (long)T * G * ZT * splits * 16 * MT * (E + 4);
}
HB_EXPORT int hb_attn_masked_heads(const void* q, long ldq, const void* kc, long k_page, long k_head, long k_row, const void* vc,
                                   long v_page, long v_head, long v_row, int alias, const int* bt, int bt_stride,
                                   const int* row_req, const int* pos, const float* sink, const float* gate, long ld_gate,
                                   int gate_off, int gate_mode, void* out, int o_dt, long ldo, int T, int H, int G, int D, int E,
                                   int page_size, int mask, int window, int keep_first, int chunk, float scale, const int* q_len,
                                   int row_limit, float* part, long n_part, int max_pos, const float* r1, const float* r2,
                                   const int* row_list, const int* ctx_len, cudaStream_t s) {
  if (T <= 0) return 0;
  const int eu = hs_units(H, G, D, E, alias);
  if (!eu) HB_FAIL("hb_attn_masked_heads: %d heads over %d kv heads with keys of %d and values of %d are not sizes it takes", H, G, D, E);
  if (T > 65535) HB_FAIL("hb_attn_masked_heads: %d rows are beyond the grid limit", T);
  if ((ldq | k_page | k_head | k_row | v_page | v_head | v_row) & 7 || (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) & 15))
    HB_FAIL("hb_attn_masked_heads: rows of q, keys and values must start on 16-byte boundaries");
  if ((r1 != nullptr) != (r2 != nullptr)) HB_FAIL("hb_attn_masked_heads: a distance bias needs both of its vectors");
  HeadsArgs A;
  A.r1 = r1; A.r2 = r2; A.q = (const __nv_bfloat16*)q; A.ldq = ldq; A.kc = (const __nv_bfloat16*)kc; A.k_page = k_page; A.k_head = k_head; A.k_row = k_row;
  A.vc = (const __nv_bfloat16*)vc; A.v_page = v_page; A.v_head = v_head; A.v_row = v_row; A.alias = alias; A.bt = bt;
  A.bt_stride = bt_stride; A.row_req = row_req; A.pos = pos; A.sink = sink; A.gate = gate; A.ld_gate = ld_gate; A.gate_off = gate_off;
  A.gate_mode = gate ? gate_mode : 0; A.out = out; A.ldo = ldo; A.H = H; A.G = G; A.D = D; A.E = E; A.page_size = page_size;
  A.mask = mask; A.window = window; A.keep_first = keep_first; A.chunk = chunk; A.scale = scale; A.q_len = q_len;
  A.row_limit = row_limit; A.part = part; A.row_list = row_list; A.ctx_len = ctx_len;
  const int HG = H / G;
  A.MT = hs_mt(HG);
  const int ZT = (HG + 16 * A.MT - 1) / (16 * A.MT);
  A.G_ZT = G * ZT;
  const int most = hs_most_tiles(mask, window, keep_first, chunk, max_pos);
  A.splits = hs_splits(most);
  // the join's CTAs: a power of two, two an SM at most over the whole call, no more than there are columns for
  A.join = HS_SPLIT_TILES;
  while (A.join > 1 && ((long)T * A.G_ZT * A.splits * A.join > 296 || A.join * HS_THREADS / 2 >= (HG < 16 * A.MT ? HG : 16 * A.MT) * (E / 4))) A.join /= 2;
  A.cs = most > 4 ? HS_SPLIT_TILES : most > 2 ? 4 : most;
  if (A.cs < A.join) A.cs = A.join;
  if (A.splits > 1 && (!part || n_part < (long)T * G * ZT * A.splits * 16 * A.MT * (E + 4)))
    HB_FAIL("hb_attn_masked_heads: rows of up to %d key tiles need a workspace", A.splits * HS_SPLIT_TILES);
  if ((long)ZT * G > 65535) HB_FAIL("hb_attn_masked_heads: the grid is too large");
  const size_t smem = hs_smem_bytes(A.MT, D, E, alias);
  const dim3 grid(A.cs * A.splits, G * ZT, T);
  cudaError_t e = cudaErrorInvalidValue;
#define HS_RUN(EU, MT)                                                                                                            \
  do {                                                                                                                            \
    auto kern = o_dt == HB_BF16 ? attn_masked_heads_kernel<EU, MT, __nv_bfloat16> : attn_masked_heads_kernel<EU, MT, float>;      \
    e = smem + 8192 > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess; \
    if (e == cudaSuccess) e = hb_launch_cluster(kern, grid, dim3(HS_THREADS), smem, s, dim3(A.cs, 1, 1), A);            \
  } while (0)
  if (A.MT == 2) {
    if (eu == 1) HS_RUN(1, 2);
    else if (eu == 2) HS_RUN(2, 2);
    else if (eu == 4) HS_RUN(4, 2);
    else HS_RUN(8, 2);
  } else {
    if (eu == 1) HS_RUN(1, 1);
    else if (eu == 2) HS_RUN(2, 1);
    else if (eu == 4) HS_RUN(4, 1);
    else if (eu == 8) HS_RUN(8, 1);
    else HS_RUN(16, 1);
  }
#undef HS_RUN
  if (e != cudaSuccess) HB_FAIL("hb_attn_masked_heads: %s", cudaGetErrorString(e));
  HB_CHECK_LAUNCH("hb_attn_masked_heads");
  if (A.splits > 1) {
    dim3 mgrid((16 * A.MT * (E / 4) + HS_THREADS - 1) / HS_THREADS, G * ZT, T);
    if (o_dt == HB_BF16) hb_launch(attn_masked_heads_merge_kernel<__nv_bfloat16>, mgrid, dim3(HS_THREADS), 0, s, A);
    else hb_launch(attn_masked_heads_merge_kernel<float>, mgrid, dim3(HS_THREADS), 0, s, A);
    HB_CHECK_LAUNCH("hb_attn_masked_heads (merge)");
  }
  return 0;
}
