// prefill_mx8.cu - grouped expert products on MXFP4 weights and f32 activations for small groups (a few tokens an
// expert): tcgen05.mma kind::mxf8f6f4 with block scales. The tensor cores take the E2M1 codes and their E8M0
// scales as they are stored (src/oss_kernels.rs:41-55: code * 2^(e - 127)), so nothing is decoded, and the weights' boxes are
// expanding copies (16 codes of 4 bits into a place of 16 bytes: the tensor map's 16U4_ALIGN16B): they land as operand A.
//
// The activations are exact sums of E4M3 pieces with block scales of their own: x = x1 + x2 + ..., xi the
// nearest E4M3 of what is left of x, in units of 2^(E - 7 - 5 (i - 1)), E the exponent of the block's largest value.
// What a piece leaves is at most a 32nd of what it was given: 5 pieces hold all 24 bits of the values within 13 octaves of the
// block's largest and leave 2^-37 of that of the smaller ones (calls of fewer than PM_MX_PROMPT tokens), 4 leave 2^-19 of
// it (prompts; the two bf16 pieces of prefill_mx.cu leave 2^-17 of a value). No unit is below 2^-126: in blocks whose largest is
// below 2^-99 the last pieces hold less, down to 2^-136. The pieces of a
// tile's tokens are columns of ONE product: N = pieces x tokens, a sum each, added up smallest first. With 5 pieces
// the sums are folded into f32 registers every 256 K values (the tensor cores' own sums lose the low bits
// of a long chain: 1e-5 of the RMS over 2,880 values against 1e-7).
//
// A persistent pipeline as in prefill_mx.cu; two CTAs an SM, 128 weight rows (64 of gate and 64 of up, or 128 of down) x
// 16 tokens (5 pieces) or 32 (4), stages of 128 K values that four warps hand on: one thread issues every copy, one warp brings
// the weights' scales, one issues the products, eight read the sums.
// Bound by the weights' bytes and, above 8 tokens a tile, the products (whole layers of 32 experts, d = ff = 2880, us a layer, before: workers moved the codes
// from packed boxes to operand A, 900 cycles of latency a stage, and a launch between the products split h): 1 token 53 -> 37.5, 8 tokens
// 144 -> 90, 31 tokens 183 -> 126, 224 tokens 239 -> 176.
#include <cuda_fp16.h>

#include "mxsum.cuh"

#define M8_M 128
#define M8_KS 128     /* K values of a stage: four products of 32 */
#define M8_AST (M8_M * 128)    /* operand A of a stage: 16 codes = 8 bytes and 8 unused, rows of 128 bytes, swizzled */
#define M8_ABYTES (M8_M * 64)  /* ... the bytes of it that are copied */
#define M8_NW 8
#define M8_NT (32 * (M8_NW + 3))
#define M8_IT 4
#define M8_END 0xfffffffeu

template <int NP> struct M8Shape {
  static constexpr int NTOK = NP == 5 ? 16 : 32;
  static constexpr bool FOLD = NP == 5;
  static constexpr int NSR = NP == 5 ? 4 : 3;          // stages: the weights with their scales, the tokens' pieces with theirs
  static constexpr int BST = NP * NTOK * M8_KS + 512;  // the pieces of a stage and their scales
  static constexpr uint32_t SET = NP * NTOK;           // columns of a set of sums (folded: two sets)
  // columns of the scales, a place a stage: nothing orders a copy of scales behind the products that
  // read the ones before it but the commit that frees the place
  static constexpr uint32_t SFA = 256 - 8 * NSR, SFB = 256 - 4 * NSR;
  static constexpr int NACC = FOLD ? 2 : 1;
};
static_assert(2 * M8Shape<5>::SET <= M8Shape<5>::SFA && M8Shape<4>::SET <= M8Shape<4>::SFA, "sums and scales share 256 columns");

struct M8Args {
  CUtensorMap m0, m1;     // nibble planes of gate or down, of up (expanding boxes of 64 rows; down: of 128)
  const uint8_t *s0, *s1; // their planes of scale bytes
  size_t s0_stride, s1_stride;
  const uint4 *tiles;
  const int *n_tiles;
  unsigned int *next;
  const uint8_t *rec;     // the tokens' pieces (k_mx8_rows)
  const uint8_t *w0, *w1;       // the nibbles, the f32 rows and the row of each pair (null: its own), for mx_repair
  size_t w0_stride, w1_stride;
  const float *x;
  const uint32_t *src_row;
  const float *bias0, *bias1;
  const float *wts;
  const uint32_t *pair_src;
  float *out;             // gate/up: h [P][ff]; down: eo [splits][P][d]
  uint8_t *hrec;          // gate/up: the pieces of h, for the down products
  size_t split_stride;
  int *err;
  unsigned long long wait_ns;
  uint32_t zero;  // 0 (see tc_mbar_arrive_used)
  int row_tiles, splits, split_stages;
  int cols, rows;
  int act;
  float act_limit, act_alpha;
};

__device__ __forceinline__ void m8_mma(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n\t}\n" ::"r"(tmem_c),
      "l"(da), "l"(db), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
// 512 bytes of scales (row r, K block k at (r & 31) * 16 + (r >> 5) * 4 + k) -> four columns of every lane quarter
__device__ __forceinline__ void m8_cp_scales(uint32_t tmem_c, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_c), "l"(desc) : "memory");
}
__device__ __forceinline__ uint32_t m8_e4m3x2(float hi, float lo) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 m8_from_e4m3x2(uint32_t v) {
  uint32_t h;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"((uint16_t)v));
  return __half22float2(*reinterpret_cast<const __half2 *>(&h));
}
__device__ __forceinline__ float m8_pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 .. 127

// the tokens' f32 rows (of pair p: row src_row[p]) -> their pieces: per tile and stage [4 K blocks][2 groups of 16][pieces x rows][16], then the scales. A block's 32
// values lie as the packed codes come apart: group 0 holds values 0, 16, 1, 17 .. 7, 23, group 1 the others. A thread
// a (row, block).
template <int NP>
__global__ void __launch_bounds__(128) k_mx8_rows(const int *__restrict__ n_tiles, const uint4 *__restrict__ tiles,
                                                  const uint32_t *__restrict__ src_row, int cols, const float *__restrict__ x,
                                                  uint8_t *__restrict__ rec) {
#pragma unroll 1
  for (int practice = gridDim.x * gridDim.y <= PM_PRACTICE_CTAS; practice >= 0; practice--) {
    uint4 T = make_uint4(0, 0, 0, 0);
    if (!practice) {
      pm_pdl();
      T = tiles[blockIdx.y];  // (read beside the count: the list has room for every row of the grid)
      if ((int)blockIdx.y >= *n_tiles) return;
    }
    const int npad = practice ? 128 : ((int)T.z + 7) & ~7, nst = (cols + M8_KS - 1) / M8_KS, nb = practice ? 1 : cols / 32, N = NP * npad;
    uint8_t *base = rec + (size_t)(T.w >> 4) * nst * (2048 * NP + 512);
    for (int u = practice ? (int)threadIdx.x : (int)(blockIdx.x * 128 + threadIdx.x); u < nb * npad; u += gridDim.x * 128) {
      const int b = u / npad, r = u - b * npad;
      float v[32];
      uint32_t top = 0;
      const bool on = r < (int)T.z;
      const size_t row = on ? src_row[T.y + r] : 0;
      const float4 *src = (const float4 *)(x + row * cols + 32 * b);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float z = practice ? 1.0f : 0.0f;
        const float4 f = on ? __ldg(src + i) : make_float4(z, z, z, z);
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
      }
#pragma unroll
      for (int i = 0; i < 32; i++) top = max(top, __float_as_uint(v[i]) & 0x7fffffffu);
      const int E = (int)(top >> 23) - 127;
      uint8_t *dst = base + (size_t)(b >> 2) * (N * M8_KS + 512) + (size_t)(b & 3) * (N * 32);
      uint8_t *sf = base + (size_t)(b >> 2) * (N * M8_KS + 512) + N * M8_KS + (b & 3);
      // (what is left is kept in units of the next piece: exact, and in range also where x1, rounded up, is 2^128)
      const float unit = m8_pow2(-max(E - 7, -126));
#pragma unroll
      for (int i = 0; i < 32; i++) v[i] = __fmul_rn(v[i], unit);
#pragma unroll
      for (int p = 0; p < NP; p++) {
        const int S = max(E - 7 - 5 * p, -126);
        const float next = m8_pow2(S - max(E - 12 - 5 * p, -126));  // 32, or less at the bottom of the range
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i++) {  // (16 times: values i and i + 16)
          const uint32_t c = m8_e4m3x2(v[i + 16], v[i]);
          const float2 f = m8_from_e4m3x2(c);
          v[i] = __fmul_rn(__fsub_rn(v[i], f.x), next);
          v[i + 16] = __fmul_rn(__fsub_rn(v[i + 16], f.y), next);
          if (i & 1) w[i >> 1] |= c << 16;
          else w[i >> 1] = c;
        }
        if (top >= 0x7f800000u) {  // an infinity or a NaN in the block: NaN (what it spoils is summed again, mxsum.cuh)
#pragma unroll
          for (int i = 0; i < 8; i++) w[i] = 0x7f7f7f7fu;
        }
        const int n = p * npad + r;
        if (!practice) {
          *(uint4 *)(dst + (size_t)n * 16) = make_uint4(w[0], w[1], w[2], w[3]);
          *(uint4 *)(dst + (size_t)(N + n) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
          sf[(n & 31) * 16 + (n >> 5) * 4] = (uint8_t)(S + 127);
        }
      }
    }
  }
}

struct M8Item {
  uint4 t;
  int r0, s0, s1, split;  // first row, stages [s0, s1), which cut of K
};

template <bool DOWN, int NP>
__global__ void __launch_bounds__(M8_NT, 2) k_tc_mx8(const __grid_constant__ M8Args A) {
  using S = M8Shape<NP>;
  constexpr int MW = M8_NW, NSR = S::NSR, NACC = S::NACC;
  constexpr int RPC = DOWN ? M8_M : M8_M / 2;  // matrix rows of an item
  constexpr int HX = S::NTOK / 4;              // gate/up: sums that a thread hands to its partner
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sA = smem, *sB = sA + NSR * M8_AST, *sSA = sB + NSR * S::BST;
  float *sX = (float *)(sSA + NSR * 512);  // gate/up: [2 halves of the tokens][HX][128 rows]
  M8Item *items = (M8Item *)((uint8_t *)sX + (DOWN ? 0 : 2 * HX * M8_M * 4));
  // the rings: full_raw / empty_raw: operand A and its scales, a_ready / a_free: the activations' pieces
  uint64_t *full_raw = (uint64_t *)(items + M8_IT), *empty_raw = full_raw + NSR;
  uint64_t *a_ready = empty_raw + NSR, *a_free = a_ready + NSR, *acc_full = a_free + NSR;
  uint64_t *acc_free = acc_full + NACC, *it_full = acc_free + NACC, *it_empty = it_full + M8_IT;
  uint32_t *tmem_slot = (uint32_t *)(it_empty + M8_IT);
  const int nbk = A.cols / 32, rows = A.rows, nst = (A.cols + M8_KS - 1) / M8_KS;
  const int tid = threadIdx.x, warp = __shfl_sync(PM_FULL, tid >> 5, 0), lane = tid & 31;

  // (gate/up lets the down products in only after its own wait: they read the tile list before theirs)
  if (DOWN) pm_pdl_trigger();
  if (warp == MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_s32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NSR; i++) {
      tc_mbar_init(full_raw + i, 2);   // the box(es); the scales
      tc_mbar_init(empty_raw + i, 1);  // the products' commits
      tc_mbar_init(a_ready + i, 1);
      tc_mbar_init(a_free + i, 1);
    }
    for (int i = 0; i < NACC; i++) {
      tc_mbar_init(acc_full + i, 1);
      tc_mbar_init(acc_free + i, MW);
    }
    for (int i = 0; i < M8_IT; i++) {
      tc_mbar_init(it_full + i, 1);
      tc_mbar_init(it_empty + i, 2 + MW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __reduce_max_sync(PM_FULL, *tmem_slot);
  if (warp != MW + 1) {  // (the producer waits later)
    pm_pdl_wait();
    if (!DOWN) pm_pdl_trigger();
  }
  auto next_item = [&](int k, M8Item &it) -> bool {
    const int s = k & (M8_IT - 1);
    const bool ok = tc_wait(it_full + s, (uint32_t)((k / M8_IT) & 1), A.err, A.wait_ns);
    it = items[s];
    __syncwarp();
    if (lane == 0) tc_mbar_arrive_used(it_empty + s, it.t.x ^ (uint32_t)it.r0, A.zero);
    return ok && it.t.x != M8_END;
  };

  if (warp == MW) {
    // ================= the issuing warp =================
    const uint32_t el = tc_elect() ? 1u : 0u;
    const uint32_t sA_a = tc_s32(sA), sB_a = tc_s32(sB), sSA_a = tc_s32(sSA);
    uint32_t st = 0, pf = 0, set = 0, ps = 1;  // the rings' place (they go round together) and its phase; the sums' set
    M8Item it;
    for (int k = 0; next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      const uint32_t npad = (__reduce_max_sync(PM_FULL, it.t.z) + 7u) & ~7u, N = NP * npad;
      const int s0 = (int)__reduce_max_sync(PM_FULL, (uint32_t)it.s0), s1 = (int)__reduce_max_sync(PM_FULL, (uint32_t)it.s1);
      // instruction descriptor: A E2M1 (5), B E4M3 (0), both K-major, UE8M0 scales, N (of 16: 40 columns are followed by 8
      // of whatever lies behind them, which nobody reads), M = 128; bits 4..5 and 29..30: which byte of the scale columns
      const uint32_t idesc = (5u << 7) | (((N + 15u) >> 4) << 18) | (1u << 23) | (1u << 27);
      for (int s = s0; s < s1; s++) {
        const bool first = S::FOLD ? ((s - s0) & 1) == 0 : s == s0;
        const bool last = S::FOLD ? ((s - s0) & 1) == 1 || s == s1 - 1 : s == s1 - 1;
        // operand A: rows of 128 bytes, 128-byte swizzle (layout type 2), groups of 8 rows 1024 bytes apart
        const uint64_t dA = (tc_desc(sA_a + st * M8_AST, 16u, 1024u)) | (2ull << 61);
        const uint64_t dB = tc_desc(sB_a + st * S::BST, N * 16u, 128u);
        const int ksteps = min(4, (A.cols - s * M8_KS) / 32);
        if (first) tc_wait(acc_free + set, ps, A.err, A.wait_ns);
        tc_wait(a_ready + st, pf, A.err, A.wait_ns);
        tc_wait(full_raw + st, pf, A.err, A.wait_ns);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (el) {
          m8_cp_scales(tmem + S::SFA + 4u * st, tc_desc(sSA_a + st * 512u, 128u, 128u));
          m8_cp_scales(tmem + S::SFB + 4u * st, tc_desc(sB_a + st * S::BST + N * M8_KS, 128u, 128u));
#pragma unroll
          for (uint32_t ks = 0; ks < 4; ks++)
            if ((int)ks < ksteps)
              m8_mma(tmem + set * S::SET, dA + 2u * ks, dB + (uint64_t)(ks * N * 2u), idesc | (ks << 4) | (ks << 29), tmem + S::SFA + 4u * st,
                     tmem + S::SFB + 4u * st, !first || ks > 0 ? 1u : 0u);
          tc_commit(empty_raw + st);
          tc_commit(a_free + st);
          if (last) tc_commit(acc_full + set);
        }
        __syncwarp();
        if (++st == NSR) { st = 0; pf ^= 1; }
        if (last && ++set == NACC) { set = 0; ps ^= 1; }
      }
    }
  } else if (warp == MW + 1) {
    // ================= one thread: work items, the weights' boxes, the activations' pieces =================
    if (tc_elect()) {
      const uint32_t sA_a = tc_s32(sA), sB_a = tc_s32(sB);
      const int per_tile = A.row_tiles * A.splits, G = (int)gridDim.x;
      int cur = (int)blockIdx.x, nxt = cur + G;
      uint4 Tc = __ldcg(A.tiles + cur / per_tile), Tn = make_uint4(M8_END, 0, 0, 0);  // (the list has room for every item of the grid)
      const int n_items = __ldcg(A.n_tiles) * per_tile;
      uint32_t sr = 0, pr = 1, nr = 0, nb = 0;
      bool ok = true;
      auto weights = [&](int el, int r0, int q) {  // stage q of the item's rows (a box past the matrix reads zeros)
        const uint32_t s = nr % NSR, a = sA_a + s * M8_AST;
        tc_mbar_expect(full_raw + s, (uint32_t)M8_ABYTES);  // (an expanding copy counts the bytes it has read)
        tc_tma3(a, &A.m0, q * M8_KS, r0, el, full_raw + s);  // boxes of 128 rows (down) or 64
        if (!DOWN) tc_tma3(a + M8_AST / 2, &A.m1, q * M8_KS, r0, el, full_raw + s);
        nr++;
      };
      // the first item's weights, under the launch before this one (TC_EARLY_WEIGHTS, prefill_tc.cuh)
      int early = 0;
      if (cur < n_items && (int)Tc.x >= 0) {
        const int in = cur % per_tile, rt = in / A.splits, s0 = (in - rt * A.splits) * A.split_stages;
        for (; early < min(NSR, min(nst - s0, A.split_stages)); early++) weights((int)Tc.x, rt * RPC, s0 + early);
      }
      pm_pdl_wait();
      for (int k = 0; ok; k++) {
        const int s = k & (M8_IT - 1);
        if (k >= M8_IT && !tc_wait(it_empty + s, (uint32_t)((k / M8_IT - 1) & 1), A.err, A.wait_ns)) break;
        const bool end = cur >= n_items;
        const int in = cur % per_tile, rt = in / A.splits, sp = in - rt * A.splits;
        const int r0 = rt * RPC, s0 = sp * A.split_stages, s1 = min(nst, s0 + A.split_stages);
        M8Item it;
        it.t = end ? make_uint4(M8_END, 0, 0, 0) : Tc;
        it.r0 = r0;
        it.s0 = s0;
        it.s1 = s1;
        it.split = sp;
        items[s] = it;
        tc_mbar_arrive(it_full + s);
        if (end) break;
        const int fut = 2 * G + (int)atomicAdd(A.next, 1u);  // (needed an item later)
        if (nxt < n_items) Tn = __ldcg(A.tiles + nxt / per_tile);
        if ((int)Tc.x >= 0) {
          const uint32_t bytes = ((Tc.z + 7) >> 3) * (8u * M8_KS * NP) + 512u;
          const uint8_t *rec = A.rec + (size_t)(Tc.w >> 4) * nst * (2048 * NP + 512);
          for (int q = s0; q < s1; q++) {  // (a box past the matrix reads zeros)
            if (early > 0) {
              early--;
            } else {
              if (nr >= NSR && !tc_wait(empty_raw + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
              weights((int)Tc.x, r0, q);
            }
            if (nb >= NSR && !tc_wait(a_free + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
            tc_mbar_expect(a_ready + sr, bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sB_a + sr * S::BST),
                         "l"(rec + (size_t)q * bytes), "r"(bytes), "r"(tc_s32(a_ready + sr))
                         : "memory");
            nb++;
            if (++sr == NSR) { sr = 0; pr ^= 1; }
          }
        }
        cur = nxt;
        nxt = fut;
        Tc = Tn;
      }
      // the last copies have landed before the CTA gives up its shared memory (full_raw: also the scales' arrival, which
      // comes when a wait has not run out; a copy takes microseconds, so the bounded wait covers it in any case)
      for (uint32_t i = 1; i <= NSR && i <= nr; i++) {
        const uint32_t q = nr - i;
        tc_landed(full_raw + q % NSR, (q / NSR) & 1);
      }
      for (uint32_t i = 1; i <= NSR && i <= nb; i++) {
        const uint32_t q = nb - i;
        tc_landed(a_ready + q % NSR, (q / NSR) & 1);
      }
    }
    __syncwarp();
  } else if (warp == MW + 2) {
    // ================= the weights' scales: lane l brings those of the tile's rows l, l + 32, l + 64, l + 96 =================
    // (gate/up: rows 0..63 are gate's, 64..127 up's). 512 bytes a stage: row r, K block k at (r & 31) * 16 + (r >> 5) * 4 + k.
    uint32_t sr = 0, pr = 1, n = 0;
    bool ok = true;
    M8Item it;
    for (int k = 0; ok && next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      const size_t el = it.t.x;
      const uint8_t *sp[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool up = !DOWN && i >= 2;
        const int row = it.r0 + lane + 32 * (DOWN ? i : (i & 1));
        sp[i] = (up ? A.s1 + el * A.s1_stride : A.s0 + el * A.s0_stride) + (size_t)min(row, rows - 1) * nbk;
      }
      TcBytes8 nx[2][4];  // eight blocks (two stages) at a time, two such ahead
#pragma unroll
      for (int i = 0; i < 4; i++) {
        nx[0][i].load(sp[i] + 4 * it.s0);
        nx[1][i].load(sp[i] + 4 * min(it.s0 + 2, nst - 1));
      }
#pragma unroll 1
      for (int s2 = it.s0; s2 < it.s1 && ok; s2 += 2) {
        unsigned long long sc[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          sc[i] = nx[0][i].get();
          nx[0][i] = nx[1][i];
          if (s2 + 4 < it.s1) nx[1][i].load(sp[i] + 4 * (s2 + 4));
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (s2 + h < it.s1 && ok) {
            if (n >= NSR) ok = __all_sync(PM_FULL, tc_wait(empty_raw + sr, pr, A.err, A.wait_ns));
            if (!ok) break;
            // (255 is a NaN to the tensor cores, 2^127 of the doubled codes elsewhere: mx_repair's)
            *(uint4 *)(sSA + sr * 512 + lane * 16) =
                make_uint4((uint32_t)(sc[0] >> (32 * h)), (uint32_t)(sc[1] >> (32 * h)), (uint32_t)(sc[2] >> (32 * h)), (uint32_t)(sc[3] >> (32 * h)));
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(full_raw + sr);
            n++;
            if (++sr == NSR) { sr = 0; pr ^= 1; }
          }
      }
    }
  } else {
    // ================= the workers: lane m of the sums, half `part` of the tokens =================
    // row m of the tile: gate's row m (m < 64) or up's row m - 64; down: row m
    const int m = tid & 127;
    const int part = (int)__reduce_max_sync(PM_FULL, (unsigned)warp >> 2);
    const bool up = !DOWN && m >= 64;
    const uint32_t tlane = tmem + (__reduce_max_sync(PM_FULL, 32u * (warp & 3)) << 16);
    uint32_t set = 0, pf = 0;
    M8Item it;
    for (int k = 0; next_item(k, it); k++) {
      const uint4 T = it.t;
      const int el = (int)T.x, nvalid = (int)__reduce_max_sync(PM_FULL, T.z), r0 = it.r0;
      const uint32_t npad = ((uint32_t)nvalid + 7u) & ~7u;
      const int ew = (int)npad >> 1, e0 = part * ew, row = r0 + (DOWN ? m : (m & 63));
      if (el < 0) {  // an expert another rank holds: zeros (down) / nothing to do (gate/up)
        if (DOWN)
          for (int i = tid; i < nvalid * RPC; i += 32 * M8_NW) {
            const int n = i / RPC, mm = i - n * RPC;
            if (r0 + mm < rows) A.out[(size_t)it.split * A.split_stride + (size_t)(T.y + n) * rows + r0 + mm] = 0.0f;
          }
        continue;
      }
      float acc[S::NTOK / 2];
#pragma unroll
      for (int u = 0; u < S::NTOK / 2; u++) acc[u] = 0.0f;
      auto fold = [&] {  // the pieces' sums of the thread's tokens, smallest piece first
        tc_wait(acc_full + set, pf, A.err, A.wait_ns);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t at = tlane + set * S::SET + (uint32_t)e0;
        auto columns = [&](int c, auto width) {
          constexpr int W = decltype(width)::value;
          uint32_t v[NP][W];
#pragma unroll
          for (int p = 0; p < NP; p++) {
            if constexpr (W == 8) tc_ld8<0>(at + (uint32_t)c + p * npad, v[p]);
            else tc_ld4<0>(at + (uint32_t)c + p * npad, v[p]);
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int u = 0; u < W; u++) {
            float t = __uint_as_float(v[NP - 1][u]);
#pragma unroll
            for (int p = NP - 2; p >= 0; p--) t = __fadd_rn(t, __uint_as_float(v[p][u]));
            acc[c + u] = __fadd_rn(acc[c + u], t);
          }
        };
#pragma unroll
        for (int c = 0; c < S::NTOK / 2; c += 8) {
          if (c + 8 <= ew) columns(c, PassC<8>());
          else if (c < ew) columns(c, PassC<4>());
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(acc_free + set);
        if (++set == NACC) { set = 0; pf ^= 1; }
      };
      if (S::FOLD) {
#pragma unroll 1
        for (int s2 = it.s0; s2 < it.s1; s2 += 2) fold();
      } else {
        fold();
      }
      // ---- epilogue ----
      // (columns past the tile's tokens: of whatever their pieces' places hold)
#pragma unroll
      for (int u = 0; u < S::NTOK / 2; u++)
        if (e0 + u >= nvalid) acc[u] = 0.0f;
      const bool on = row < rows && *(volatile int *)A.err == 0;
      mx_repair(
          acc, [&](int u) { return row < rows && u < ew && e0 + u < nvalid; },
          [&](int u) {
            const uint32_t p = T.y + (uint32_t)(e0 + u);
            return mx_sum_f32((up ? A.w1 + (size_t)el * A.w1_stride : A.w0 + (size_t)el * A.w0_stride) + row * mx_row_bytes(A.cols),
                              (up ? A.s1 + (size_t)el * A.s1_stride : A.s0 + (size_t)el * A.s0_stride) + (size_t)row * nbk,
                              A.x + (size_t)(A.src_row ? A.src_row[p] : p) * A.cols, 4 * it.s0, min(4 * it.s1, nbk));
          });
      __syncwarp();
      const bool bias = A.bias0 && it.split == 0;
      const float b0 = bias && row < rows ? A.bias0[(size_t)el * rows + row] : 0.0f;
      float *out = A.out + (size_t)it.split * A.split_stride + (size_t)T.y * rows + row;
      if constexpr (DOWN) {
#pragma unroll
        for (int u = 0; u < S::NTOK / 2; u++)
          if (u < ew && on && e0 + u < nvalid) out[(size_t)(e0 + u) * rows] = bias ? __fadd_rn(acc[u], b0) : acc[u];
      } else {
        // the warps w and w ^ 2 hold gate's and up's sums of the same rows: a gate thread activates the even columns of its
        // half of the tokens, the up thread the odd ones, each on the other's sum out of shared memory
        const float b1 = bias && row < rows ? A.bias1[(size_t)el * rows + row] : 0.0f;
        float *sx = sX + part * HX * M8_M;
#pragma unroll
        for (int i = 0; i < HX; i++)
          if (2 * i < ew) sx[i * M8_M + m] = up ? acc[2 * i] : acc[2 * i + 1];
        asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");
#pragma unroll
        for (int i = 0; i < HX; i++) {
          const int n = e0 + 2 * i + (up ? 1 : 0);
          if (2 * i < ew && n < nvalid) {
            const float other = sx[i * M8_M + (m ^ 64)];
            float gv = up ? other : acc[2 * i], uv = up ? acc[2 * i + 1] : other;
            if (bias) {
              gv = __fadd_rn(gv, b0);
              uv = __fadd_rn(uv, b1);
            }
            const float wt = A.wts ? A.wts[A.pair_src[T.y + n]] : 1.0f;
            const float h = pm_act(A.act, A.act_limit, A.act_alpha, gv, uv, wt, A.wts != nullptr);
            if (on) out[(size_t)n * rows] = h;
            // the warp holds a block of 32 values of token n: its pieces (k_mx8_rows), as the down products read them
            if (r0 + 32 * (warp & 1) < rows) {  // (rows: a multiple of 32)
              const uint32_t top = __reduce_max_sync(PM_FULL, __float_as_uint(h) & 0x7fffffffu), N = NP * npad;
              const int E = (int)(top >> 23) - 127, kb = (r0 >> 5) + (warp & 1), o = (lane & 15) * 2 + (lane >> 4);
              uint8_t *stage = A.hrec + (size_t)(T.w >> 4) * ((rows + M8_KS - 1) / M8_KS) * (2048 * NP + 512) +
                               (size_t)(kb >> 2) * (N * M8_KS + 512);
              uint8_t *dst = stage + (kb & 3) * (N * 32) + (o >> 4) * (N * 16) + (o & 15) + n * 16, *sf = stage + N * M8_KS + (kb & 3);
              float v = __fmul_rn(h, m8_pow2(-max(E - 7, -126)));
#pragma unroll
              for (int p = 0; p < NP; p++) {
                const int S = max(E - 7 - 5 * p, -126);
                const uint32_t c = m8_e4m3x2(0.0f, v), nn = (uint32_t)n + p * npad;
                v = __fmul_rn(__fsub_rn(v, m8_from_e4m3x2(c).x), m8_pow2(S - max(E - 12 - 5 * p, -126)));
                dst[p * npad * 16] = top >= 0x7f800000u ? 0x7f : (uint8_t)c;
                if (lane == 0) sf[(nn & 31) * 16 + (nn >> 5) * 4] = (uint8_t)(S + 127);
              }
            }
          }
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");  // both have read before the next item's sums
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

// bytes of the pieces of a call of T tokens: n_pairs rows of `cols` values in at most max_groups groups
size_t mx8_rec_bytes(int T, int n_pairs, int max_groups, int cols) {
  const size_t groups = (size_t)(max_groups < n_pairs ? max_groups : n_pairs), pieces = T < PM_MX_PROMPT ? 5 : 4;
  return (((size_t)n_pairs + 15 * groups) / 16 + 1) * ((cols + M8_KS - 1) / M8_KS) * (2048 * pieces + 512);
}
void launch_mx8_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x, uint8_t *rec) {
  const long units = ((long)n_rows + 15 * t.max_tiles) * (cols / 32);
  const long gx = (units / t.max_tiles + 127) / 128;
  const dim3 grid((unsigned)(gx < 1 ? 1 : gx), (unsigned)t.max_tiles);
  if (t.ntok == M8Shape<5>::NTOK) pm_launch(L, k_mx8_rows<5>, grid, 128, 0, t.n, t.tiles, src_row, cols, x, rec);
  else pm_launch(L, k_mx8_rows<4>, grid, 128, 0, t.n, t.tiles, src_row, cols, x, rec);
}

template <bool DOWN, int NP> static cudaError_t mx8_start(const Launch &L, const M8Args &A, long items) {
  using S = M8Shape<NP>;
  constexpr size_t smem = (size_t)S::NSR * (M8_AST + S::BST + 512) + (DOWN ? 0 : 2 * (S::NTOK / 4) * M8_M * 4) + M8_IT * sizeof(M8Item) +
                          (4 * S::NSR + 2 * S::NACC + 2 * M8_IT) * 8 + 16;
  static_assert(smem <= 115712, "two CTAs an SM");
  static SmemOptIn opt;
  const cudaError_t e = smem_optin(opt, k_tc_mx8<DOWN, NP>, smem);
  if (e != cudaSuccess) return e;
  const long ctas = 2L * L.n_sm;
  return pm_launch(L, k_tc_mx8<DOWN, NP>, dim3((unsigned)(items < ctas ? items : ctas)), M8_NT, smem, A);
}

// Tokens of a tile of a call of T tokens whose n_groups groups hold n_pairs / n_groups pairs on average; 128: prefill_mx.cu. Here a group makes
// a tile every 32 pairs, there mostly one. us a call of one layer, here : there, at 48 / 56 / 60 / 64 / 72 / 88 pairs a group (median of three runs):
//   24 experts x 2880 x 2880  198 : 232   209 : 246   241 : 250   258 : 255   288 : 259   314 : 287
//   32 experts x 2880 x 2880  257 : 305   266 : 305   299 : 312   332 : 326   373 : 346   402 : 384
//   32 experts x 4096 x 1536  199 : 256   219 : 274   239 : 279   267 : 280   297 : 291   336 : 310
//   64 experts x 2048 x 1024  166 : 201   175 : 211   185 : 216   205 : 218   233 : 227   261 : 258
//  128 experts x 2880 x 2880  882 : 1035  980 : 1068  1193 : 1133 1197 : 1233 1328 : 1203 1601 : 1417
// (two layers of 32 x 2880 x 2880 at 80 pairs 785 : 722, at 96 928 : 793; 16 x 4096 x 4096 at 65 / 80 pairs 340 : 317, 378 : 339; 32 x 1024 x 512 at
// 56 / 64 / 80 59 : 63, 68 : 64, 74 : 72; these kernels run into the power limit, a time repeats within 10 %): the line is at 64, two tiles a group.
// Up to 88 where the tiles of 128 tokens would leave a sixth of the SMs without work (their gate/up items: 128 rows each, waves of one item an SM):
//    4 experts x 2880 x 2880 (62 % of a wave)           74 : 99 at 64, 76 : 102 at 72, 78 : 108 at 88
//    8 experts x 2880 x 2880 (62 % of two)             106 : 143, 112 : 147, 122 : 159
//    8 experts x 2048 x 1024 (43 % of one)              62 : 75, 63 : 75, 66 : 80
//   16 experts x 2880 x 2880 (83 % of three)           181 : 210, 192 : 221, 225 : 242
// and not above (86 % and more: 8 x 4096 x 4096 209 : 204 at 88; 32 x 1024 x 512 76 : 72 at 87).
// (Sums from four fp8 pieces are 6e-7 of the RMS from 64 bits, from two bf16 pieces 1.0e-5.)
int mx_tile_tokens(int T, int n_pairs, int n_groups, int ff) {
  if (T < PM_MX_PROMPT) return M8Shape<5>::NTOK;
  const int groups = n_groups < n_pairs ? n_groups : n_pairs, avg = n_pairs / groups;
  const long places = 148, items = (long)groups * ((ff + M8_M - 1) / M8_M), waves = (items + places - 1) / places;
  const bool idle = 6 * items < 5 * waves * places;
  return avg <= 64 || (idle && avg <= 88) ? M8Shape<4>::NTOK : 128;
}

// Cuts of K of the down products: a few tokens make ceil(d / 128) items an expert, each a chain of ff / 128 stages;
// while that leaves CTAs without work, K is cut in up to four (the combine step adds the parts in order).
static int mx8_split_stages(int nst, int splits) { return ((nst + splits - 1) / splits + 1) & ~1; }  // whole boxes
int mx_splits(const pm_layer_desc &D, int n_pairs) {
  const int nst = (D.ff + M8_KS - 1) / M8_KS;
  // (a pair is at most a tile of its own; two CTAs on each of a B200's 148 SMs, also where the device offers fewer: the
  // number of parts is part of how a sum rounds)
  const long items = (long)((D.d + M8_M - 1) / M8_M) * n_pairs;
  long s = 296 / (items > 0 ? items : 1);
  s = s > 4 ? 4 : s;
  s = s > nst / 4 ? nst / 4 : s;  // at least four stages each
  if (s <= 1) return 1;
  const int ss = mx8_split_stages(nst, (int)s);
  return (nst + ss - 1) / ss;  // (rounding up may leave fewer)
}

// Tensor-core form of launch_gateup / launch_down for MXFP4 weights and f32 activations given as the pieces of
// the grouping's rows. x, src_row: the rows the pieces were made of (as in launch_mx8_rows). splits: cuts of K (down only); split s
// goes to out + s * split_stride.
cudaError_t launch_tc_mx8(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                          const uint8_t *rec, const float *x, const uint32_t *src_row, const float *wts, float *out, uint8_t *hrec, int splits,
                          size_t split_stride, int *err, unsigned long long wait_ns) {
  if (t.max_tiles == 0) return cudaSuccess;
  const WMat &W0 = down ? ly.down : ly.gate, &W1 = ly.up;
  M8Args A;
  A.hrec = hrec;
  A.m0 = (down ? ly.maps->down : ly.maps->gate).m[0];  // boxes of 128 or 64 rows
  A.m1 = ly.maps->up.m[0];
  A.s0 = W0.plane[1];
  A.s0_stride = W0.stride[1];
  A.s1 = W1.plane[1];
  A.s1_stride = W1.stride[1];
  A.tiles = t.tiles;
  A.n_tiles = t.n;
  A.next = t.next + (down ? 1 : 0);
  A.rec = rec;
  A.w0 = W0.plane[0];
  A.w0_stride = W0.stride[0];
  A.w1 = W1.plane[0];
  A.w1_stride = W1.stride[0];
  A.x = x;
  A.src_row = src_row;
  A.bias0 = down ? ly.bias_down : ly.bias_gate;
  A.bias1 = down ? nullptr : ly.bias_up;
  A.wts = !down && ly.desc.weight_fold == PM_FOLD_BEFORE_DOWN ? wts : nullptr;
  A.pair_src = pair_src;
  A.out = out;
  A.split_stride = split_stride;
  A.err = err;
  A.wait_ns = wait_ns;
  A.zero = 0;
  const int rpc = down ? M8_M : M8_M / 2, nst = (W0.cols + M8_KS - 1) / M8_KS;
  A.row_tiles = (W0.rows + rpc - 1) / rpc;
  A.split_stages = mx8_split_stages(nst, splits);
  A.splits = splits;
  A.cols = W0.cols;
  A.rows = W0.rows;
  A.act = ly.desc.act;
  A.act_limit = ly.desc.act_limit;
  A.act_alpha = ly.desc.act_alpha;
  const long items = (long)A.row_tiles * A.splits * t.max_tiles;
  if (t.ntok == M8Shape<5>::NTOK) return down ? mx8_start<true, 5>(L, A, items) : mx8_start<false, 5>(L, A, items);
  return down ? mx8_start<true, 4>(L, A, items) : mx8_start<false, 4>(L, A, items);
}
