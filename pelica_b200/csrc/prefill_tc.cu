// prefill_tc.cu - grouped expert products for many tokens per expert on the 5th-gen
// tensor cores (tcgen05.mma kind::i8, operand A and the accumulators in TMEM), exact in
// the integer domain of the reference's CPU path (src/ds4_cpu.rs:59-83).
//
// A work item = (128 weight rows of one active expert) x (up to 128 of its tokens); a persistent CTA an SM
// (16 worker warps, one warp that issues the tensor-core instructions, one producer warp) runs one item
// after another, all rings and counters running on across items. Per 256-value block b of the rows:
//   1. the producer brings the block's weight bytes in by TMA (boxes of 64 rows x one block) and the
//      tokens' operand by one bulk copy; each worker unpacks 64 values of one row into two u8 operand
//      planes IN REGISTERS and stores them to tensor memory, where the products read operand A from:
//      shared memory carries only the tokens' activations. Q4_K: A_hi = nibble * (sc >> 3),
//      A_lo = nibble * (sc & 7), so that with the token's int8 activations xq
//        isum = 8 * (A_hi . xq) + (A_lo . xq) = sum_j sc_j * sum_i nib_ji * xq_ji
//      (6-bit scales do not fit one u8 product with a nibble; two 3-bit halves do), and
//      msum = sum_j m_j * bsum_j comes from one K=16 f16 product (see k_tc).
//   2. the issuing warp runs the block's tcgen05.mma in one or two PASSES of at most 64 tokens; pass p
//      of the CTA writes accumulator set p & 1 (2 sets x 3 accumulators x 64 columns; operand A has the
//      other 128 columns of tensor memory), so the products of one pass run under the float terms of
//      the one before;
//   3. every worker reads its TMEM lane (tcgen05.ld) and adds the block's float term
//      total += x.d[b] * (d * isum - dmin * msum) in block order, as `row_scalar`.
// Operand A of block b + 1 goes out in quarters of K, each as soon as the last products that read the
// quarter's columns are complete. Gate and up rows share an item (64 + 64 rows) so SwiGLU is fused in
// the epilogue; down rows write the pair outputs. Waits are time-bounded; TMEM is freed on every path.
//
// What bounds a block of 128 rows x 128 tokens: tensor pipe 2 x 17 products of N = 64 = 1,150 cycles;
// CUDA cores about 350 (unpack) + 100 (operand store) + 2 x 450 (float terms: five rounded steps an
// output, as f32x2 pairs, behind an integer add and a conversion).
#include <cuda_fp16.h>

#include "prefill_tc.cuh"

// The two shapes of the kernel. PARTS: worker threads a row.
//  4 (tiles of up to 128 tokens): one CTA an SM of 16 worker warps, passes of 64 tokens.
//  2 (tiles of up to 64 tokens): two CTAs an SM of 8 worker warps and half of the tensor memory each, passes of
//    16 tokens. With few tokens a block is a chain of short steps - wait, unpack, store, hand over, fold - that
//    one set of warps runs in lockstep; two CTAs interleave theirs, and half as many warps wait at each barrier.
template <int PARTS> struct TcShape {
  static constexpr int NW = PARTS * TC_M;                // worker threads
  static constexpr int NT = NW + 64;                     // ... the warp that issues the products, the producer warp
  static constexpr int CTAS = PARTS == 4 ? 1 : 2;        // an SM
  static constexpr int NTOK = PARTS == 4 ? TC_NMAX : 64; // tokens of a tile
  static constexpr int PN = PARTS == 4 ? 64 : 16;        // tokens of a pass
  static constexpr int MP = NTOK / PN;                   // passes of a block at most
  static constexpr int CW = PN / PARTS;                  // columns of a pass that a thread folds, at most
  // tensor memory: two sets of the accumulators hi, lo, mins (PN columns each), then operand A (64 columns a plane)
  static constexpr uint32_t COLS = PARTS == 4 ? 512 : 256, SET = 3 * PN, A_HI = COLS - 128, A_LO = COLS - 64;
  static constexpr int BST = NTOK / 8 * TC_REC;          // the tokens' operand of a block
  static constexpr int XB = PN * TC_M * 4;               // gate/up: exchange of a pass's sums
};
// stages of the weights' and of the tokens' ring: what fits an SM
template <int PARTS, bool Q6, bool DOWN> struct TcStages {
  static constexpr int raw = PARTS == 4 ? (Q6 ? (DOWN ? 4 : 3) : (DOWN ? 5 : 4)) : 2;
  static constexpr int tok = PARTS == 2 && Q6 && !DOWN ? 2 : 3;
};

// Compile with -DPM_TC_TRACE=1 (gate/up launches) or =2 (down launches) to stamp the phases of CTA 0's second
// item with the SM clock: [worker thread 0 | thread 511 | issuing warp | producer][block][stamp], read back with
// pm_debug_tc_trace.
#ifdef PM_TC_TRACE
__device__ unsigned long long g_tc_trace[4 * 32 * 8];
#define TC_STAMP(who, b, i)                                                                                        \
  if (blockIdx.x == 0 && k == 1 && (b) < 32 && (int)DOWN + 1 == PM_TC_TRACE &&                          \
      ((who) == 3 || (who) == 2 ? (who) == 3 || lane == 0 : (tid == ((who) ? 511 : 0))))                                                        \
    g_tc_trace[((who) * 32 + (b)) * 8 + (i)] = clock64();
extern "C" __attribute__((visibility("default"))) int pm_debug_tc_trace(unsigned long long *out) {
  return (int)cudaMemcpyFromSymbol(out, g_tc_trace, sizeof(g_tc_trace));
}
#else
#define TC_STAMP(who, b, i)
#endif
#define TC_STAMP_W(b, i) TC_STAMP(0, b, i) TC_STAMP(1, b, i)

// The token tiles of a grouping: group a contributes ceil(count / ntok) tiles. tiles[i] = (expert slot, or
// ~0 for an expert another rank holds; first pair; pairs; first record row). The records' rows keep a group's
// pairs together and start every group on a multiple of 16 rows. One CTA; groups <= 512.
__global__ void __launch_bounds__(512) k_tc_tiles(Groups g, int first_local, int n_local, int *head,
                                                  uint4 *tiles, int ntok, int even, int max_tiles) {
  pm_pdl();
  __shared__ uint32_t s_t[16], s_r[16];
  const int a = threadIdx.x, lane = a & 31, warp = a >> 5;
  const int ng = min(*g.n_groups, 512);
  const uint32_t cnt = a < ng ? g.count[a] : 0;
  const uint32_t tc = (cnt + ntok - 1) / ntok, rp = tc_group_rows(ntok, cnt, tc);
  uint32_t t = tc, r = rp;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t ut = __shfl_up_sync(PM_FULL, t, o), ur = __shfl_up_sync(PM_FULL, r, o);
    if (lane >= o) { t += ut; r += ur; }
  }
  if (lane == 31) { s_t[warp] = t; s_r[warp] = r; }
  __syncthreads();
  uint32_t bt = 0, br = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 16; w++) {
    if (w < warp) { bt += s_t[w]; br += s_r[w]; }
    all += s_t[w];
  }
  const uint32_t first = bt + t - tc, r0 = br + r - rp;
  if (a < ng) {
    int el = (int)g.expert[a] - first_local;
    if (el < 0 || el >= n_local) el = -1;
    const uint32_t off = g.offset[a];
    const uint32_t nt = tc_tile_tokens(cnt, tc, ntok, even);
    for (uint32_t i = 0; i < tc && (int)(first + i) < max_tiles; i++)
      tiles[first + i] = make_uint4((uint32_t)el, off + i * nt, min(cnt - i * nt, nt), r0 + i * tc_tile_rows(ntok, nt));
  }
  if (a == 0) {  // [0] tiles, [1], [2] the item counters of the two products
    head[0] = min((int)all, max_tiles);
    head[1] = 0;
    head[2] = 0;
  }
}

// Rows of f32 values -> the records the products read: `Q8x::new` (src/ds4_cpu.rs:13-35) of every 256-value
// block, a CTA column a token tile, one warp per (8 rows, block). Row i of a tile comes from row src_row[first + i] of
// x (null: row first + i itself), first = the tile's first pair; rows past the tile's count are zeros. A token
// is read and quantised once per expert that serves it: a launch less for small calls, but four times the
// bytes of a gather of quantised rows (4096 tokens x 8 experts x 7168 values: 280 us against 48 + 60), so large
// calls quantise first (k_quant_q8x) and gather (k_tc_rows; the line and its figures: dev_experts).
// FEW: tiles of prefill_few.cu. 1: one record a block (its 8 rows serve all 16 columns); 2 (Q6_K): the rows twice, record g with
// the sub-blocks of 16 whose number has the other parity than g as zeros. 0: two records every 16 rows.
template <int FEW>
__global__ void __launch_bounds__(256) k_tc_quant_rows(const int *__restrict__ n_tiles, const uint4 *__restrict__ tiles,
                                                       const uint32_t *__restrict__ src_row, int cols,
                                                       const float *__restrict__ x, uint8_t *__restrict__ rec) {
  __shared__ __align__(16) uint8_t s_rec[8][TC_REC];
#pragma unroll 1
  for (int practice = gridDim.x * gridDim.y <= PM_PRACTICE_CTAS; practice >= 0; practice--) {
    uint4 T = make_uint4(0, 0, 0, 0);
    if (!practice) {
      pm_pdl();
      T = tiles[blockIdx.y];  // (read beside the count: the list has room for every row of the grid)
      if ((int)blockIdx.y >= *n_tiles) return;
    }
    const int nb = cols / 256;
    const uint32_t off = T.y, cnt = T.z;
    const int lane = threadIdx.x & 31;
    uint8_t *S = s_rec[threadIdx.x >> 5];
    const int nrg = FEW ? FEW : (int)((cnt + 15u) / 16u) * 2, units = practice ? 8 : nrg * nb;  // (row group, block) pairs of this tile
    uint8_t *rec0 = rec + (size_t)(T.w >> 3) * nb * TC_REC;
    for (int u = practice ? (int)(threadIdx.x >> 5) : (int)(blockIdx.x * 8 + (threadIdx.x >> 5)); u < units; u += gridDim.x * 8) {
      const int b = u / max(nrg, 1), rgl = u - b * nrg;  // (the tile's records lie block by block)
      // lane = values 8 lane .. 8 lane + 7 of every row = half of K chunk lane / 2; row r of chunk c waits in shared memory in place
      // r ^ (c & 7) of the chunk's eight (no bank conflicts). Two times four rows through the same code: executed once a warp it is
      // fetched cold, so half as much of it counts (8 tokens through 48 layers of 128 experts 3,147 -> 3,120 us; prompts the same).
      const int ch = lane >> 1;
#pragma unroll 1
      for (int h = 0; h < 2; h++) {
        float v[4][8];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const uint32_t i = (uint32_t)((FEW ? 0 : rgl * 8) + 4 * h + r);
          if (i < cnt) {
            const size_t row = src_row ? src_row[off + i] : off + i;
            const float4 *src = (const float4 *)(x + row * cols + (size_t)b * 256 + 8 * lane);
            const float4 p = __ldg(src), w = __ldg(src + 1);
            v[r][0] = p.x; v[r][1] = p.y; v[r][2] = p.z; v[r][3] = p.w;
            v[r][4] = w.x; v[r][5] = w.y; v[r][6] = w.z; v[r][7] = w.w;
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[r][j] = practice ? 1.0f : 0.0f;
          }
        }
        float mx[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          float m = 0.0f;
#pragma unroll
          for (int j = 0; j < 8; j++) m = fmaxf(m, fabsf(v[r][j]));
          mx[r] = __uint_as_float(__reduce_max_sync(PM_FULL, __float_as_uint(m)));  // (non-negative floats order like integers)
        }
        // lane r divides for row r
        const float mine = lane == 0 ? mx[0] : (lane == 1 ? mx[1] : (lane == 2 ? mx[2] : mx[3]));
        const float idv = mine != 0.0f ? __fdiv_rn(127.0f, mine) : 0.0f;
        if (lane < 4) *(float *)(S + TC_REC_XD + (4 * h + lane) * 4) = mine != 0.0f ? __fdiv_rn(mine, 127.0f) : 0.0f;
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int r8 = 4 * h + r;
          uint32_t w0, w1;
          pm_q8_pack8(v[r], __shfl_sync(PM_FULL, idv, r), w0, w1);
          int s = __dp4a((int)w1, 0x01010101, __dp4a((int)w0, 0x01010101, 0));
          s += __shfl_xor_sync(PM_FULL, s, 1);  // the sum of 32 values: lanes 4 j .. 4 j + 3 hold group j
          s += __shfl_xor_sync(PM_FULL, s, 2);
          if ((lane & 3) == 0) {  // s = 64 * (s >> 6) + (s & 63), both parts exact in f16
            __half *bm = (__half *)(S + TC_REC_BM + r8 * 16) + (lane >> 2);
            bm[0] = __int2half_rn((s >> 6) * 64);
            bm[64] = __int2half_rn(s & 63);
          }
          const int tot = __reduce_add_sync(PM_FULL, s);  // (four times the block's sum)
          if (lane == 0) *(int32_t *)(S + TC_REC_XS + r8 * 4) = -4128 * tot;
          if (FEW == 2 && (ch & 1) != rgl) w0 = w1 = 0u;
          *(uint2 *)(S + ch * 128 + ((r8 ^ (ch & 7)) << 4) + ((lane & 1) << 3)) = make_uint2(w0, w1);
        }
      }
      __syncwarp();
      uint4 *R = (uint4 *)(rec0 + (size_t)u * TC_REC);
      if (!practice) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int p = 32 * k + lane, c = p >> 3;
          R[p] = *(const uint4 *)(S + c * 128 + (((p & 7) ^ (c & 7)) << 4));
        }
        if (lane < (TC_REC - 2048) / 16 - 4) R[128 + lane] = *(const uint4 *)(S + 2048 + lane * 16);
      }
      __syncwarp();
    }
  }
}

// The same records from rows that are quantised already (rows another rank sent): one warp per
// (8 rows, block), xbm / xs as k_q8x_aux makes them.
template <int FEW>
__global__ void __launch_bounds__(256) k_tc_rows(const int *__restrict__ n_tiles, const uint4 *__restrict__ tiles,
                                                 const uint32_t *__restrict__ src_row, int cols,
                                                 const int8_t *__restrict__ xq, const float *__restrict__ xd,
                                                 const uint16_t *__restrict__ xbm, const int32_t *__restrict__ xs,
                                                 uint8_t *__restrict__ rec) {
  pm_pdl();
  const uint4 T = tiles[blockIdx.y];  // (read beside the count: the list has room for every row of the grid)
  if ((int)blockIdx.y >= *n_tiles) return;
  const int nb = cols / 256;
  const uint32_t off = T.y, cnt = T.z;
  const int lane = threadIdx.x & 31;
  const int nrg = FEW ? FEW : (int)((cnt + 15u) / 16u) * 2, units = nrg * nb;
  uint8_t *rec0 = rec + (size_t)(T.w >> 3) * nb * TC_REC;
  for (int u = blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += gridDim.x * 8) {
    const int b = u / nrg, rgl = u - b * nrg;
    uint8_t *R = rec0 + (size_t)u * TC_REC;
    {  // int8 values: lane = (row of the group, quarter of the block's 16 chunks)
      const int r8 = lane >> 2, q = lane & 3;
      const uint32_t i = (uint32_t)(FEW ? 0 : rgl * 8) + r8;
      uint4 v[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      if (i < cnt) {
        const size_t row = src_row ? src_row[off + i] : off + i;
        const uint4 *src = (const uint4 *)(xq + row * cols + (size_t)b * 256 + 64 * q);
#pragma unroll
        for (int c = 0; c < 4; c++)
          if (FEW != 2 || (c & 1) == rgl) v[c] = __ldg(src + c);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) *(uint4 *)(R + ((4 * q + c) * 8 + r8) * 16) = v[c];
    }
    const int r8 = lane < 16 ? lane >> 1 : (lane & 7);
    const uint32_t i = (uint32_t)(FEW ? 0 : rgl * 8) + r8;
    const size_t row = i < cnt ? (src_row ? (size_t)src_row[off + i] : (size_t)(off + i)) : 0;
    if (lane < 16) {  // the f16 form of the sub-block sums: lane = (row, K chunk of the mins product)
      const int k = lane & 1;
      *(uint4 *)(R + TC_REC_BM + (k * 8 + r8) * 16) =
          i < cnt ? __ldg((const uint4 *)(xbm + (row * nb + b) * 16 + 8 * k)) : make_uint4(0, 0, 0, 0);
    } else if (lane < 24) {
      *(float *)(R + TC_REC_XD + r8 * 4) = i < cnt ? xd[row * nb + b] : 0.0f;
    } else {
      *(int32_t *)(R + TC_REC_XS + r8 * 4) = i < cnt ? -16512 * xs[row * nb + b] : 0;
    }
  }
}

// WT: the weight type of the product's matrices.
//  PM_TYPE_Q4_K: u8 planes hi = nibble * (sc >> 3), lo = nibble * (sc & 7) and one
//    kind::f16 product for the mins: A_m = (m_0..m_7, m_0..m_7) against the token's
//    (64 * (bsum_j >> 6), bsum_j & 63) - every product and the sum (< 2^22) are exact in
//    f32, so the accumulator holds msum = sum_j m_j * bsum_j as an integer-valued float.
//  PM_TYPE_Q6_K: the product v = sc * (q - 32) in [-4064, 4096] is split after the
//    multiplication: v + 4128 = 64 * th + tl with th in [1, 128], tl in [0, 63] - two u8
//    planes, and isum = 64 * (th . xq) + (tl . xq) - 4128 * sum(xq) exactly. The planes are
//    th and 4 * tl (the two bytes of 4 * (v + 4128)), so the products give 4 * isum and the
//    fold multiplies by d / 4: both scalings are by a power of two, the rounding is that of
//    d * float(isum).
// Work items are handed out by the producers: two a CTA by position, the rest from a counter in global
// memory (tiles hold 1 to 128 tokens, so a fixed share would leave SMs idle: 22 % of the cycles at 128
// tokens an expert), requested an item ahead and passed to the other warps through a ring of four slots.
// Barriers (all mbarriers, phases counted over the CTA's life): full / empty per stage of the rings;
// a_ready[q]: quarter q of operand A of a block is in tensor memory (its four worker warps); a_free[q]: the last
// products that read quarter q of operand A are complete; acc_full[s] / acc_free[s]: a pass's products
// into set s are complete / have been read by every worker warp.
template <int WT, bool DOWN, int PARTS>
__global__ void __launch_bounds__(TcShape<PARTS>::NT, TcShape<PARTS>::CTAS) k_tc(const __grid_constant__ TcArgs A) {
  constexpr bool Q6 = WT == PM_TYPE_Q6_K;
  using S = TcShape<PARTS>;
  constexpr int NS = TcStages<PARTS, Q6, DOWN>::raw, NSB = TcStages<PARTS, Q6, DOWN>::tok, MW = S::NW / 32;  // MW: the first warp behind the workers
  constexpr int RAWB = Q6 ? TC_RAW_Q6 : TC_RAW_Q4;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sRaw = smem;                                  // [NS] blocks of the 128 rows (boxes of 64 rows)
  uint8_t *sB = sRaw + NS * RAWB;                        // [NSB] x [npad / 8 records]
  uint8_t *sAm = sB + NSB * S::BST;                   // Q4_K: [2][2 chunks][128 rows][8 f16]
  float *sX = (float *)(sAm + (Q6 ? 0 : 2 * 2 * TC_M * 16));  // gate/up: exchange [64 tokens][128 rows]
  TcItem *items = (TcItem *)((uint8_t *)sX + (DOWN ? 0 : S::XB));
  uint64_t *full_raw = (uint64_t *)(items + TC_IT), *empty_raw = full_raw + NS;
  uint64_t *full_b = empty_raw + NS, *empty_b = full_b + NSB;
  uint64_t *acc_full = empty_b + NSB, *acc_free = acc_full + 2, *a_free = acc_free + 2, *a_ready = a_free + 4;
  uint64_t *it_full = a_ready + 4, *it_empty = it_full + TC_IT;
  uint32_t *tmem_slot = (uint32_t *)(it_empty + TC_IT);

  const int nb = A.cols / 256, rows = A.rows;
  const int tid = threadIdx.x, warp = __shfl_sync(PM_FULL, tid >> 5, 0), lane = tid & 31;

  pm_pdl_trigger();
  if (warp == MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc_s32(tmem_slot)),
                 "r"((uint32_t)S::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NS; i++) {
      tc_mbar_init(full_raw + i, 1);  // the producer's expect_tx; the copies complete the bytes
      tc_mbar_init(empty_raw + i, MW);
    }
    for (int i = 0; i < NSB; i++) {
      tc_mbar_init(full_b + i, 1);
      tc_mbar_init(empty_b + i, 1 + MW);  // the products' commit and every worker warp after its last float term
    }
    for (int i = 0; i < 2; i++) {
      tc_mbar_init(acc_full + i, 1);
      tc_mbar_init(acc_free + i, MW);
    }
    for (int i = 0; i < 4; i++) {
      tc_mbar_init(a_free + i, 1);
      tc_mbar_init(a_ready + i, 4);  // the warps of the quarter
    }
    for (int i = 0; i < TC_IT; i++) {
      tc_mbar_init(it_full + i, 1);
      tc_mbar_init(it_empty + i, 1 + MW);  // the issuing warp and the workers have read the slot
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // (a warp reduction leaves its result in a uniform register: what is computed from it - descriptors, addresses,
  // the passes of a block - stays on the uniform datapath instead of being moved there product by product)
  const uint32_t tmem = __reduce_max_sync(PM_FULL, *tmem_slot);
  if (warp != MW + 1) pm_pdl_wait();  // (barriers and tensor memory were prepared under the kernel before; the producer waits later)
  // the CTA's k-th item, as the issuing warp and the workers take it from the ring (false: no more)
  auto next_item = [&](int k, TcItem &it) -> bool {
    const int s = k & (TC_IT - 1);
    const bool ok = tc_wait(it_full + s, (uint32_t)((k / TC_IT) & 1), A.err, A.wait_ns);
    it.t = items[s].t;
    it.r0 = items[s].r0;
    __syncwarp();
    if (lane == 0) tc_mbar_arrive_used(it_empty + s, it.t.x ^ (uint32_t)it.r0, A.zero);
    return ok && it.t.x != TC_END;
  };

  if (warp == MW) {
    // ================= the issuing warp =================
    const uint32_t el = tc_elect() ? 1u : 0u;
    const uint32_t sB_a = tc_s32(sB), sAm_a = tc_s32(sAm);
    uint32_t gb = 0, gp = 0;  // blocks and passes this CTA has run so far
    uint32_t sb = 0, pb = 0;  // the tokens' stage and its phase
    TcItem it;
    for (int k = 0; next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      const int npad = ((int)__reduce_max_sync(PM_FULL, it.t.z) + 15) & ~15, np = (npad + S::PN - 1) / S::PN;
      for (int b = 0; b < nb; b++, gb++) {
        const uint32_t bs = sB_a + sb * S::BST, am = sAm_a + (gb & 1) * (2 * TC_M * 16);
        if (A.fault_block >= 0 && b >= A.fault_block) break;  // (test hook: the workers' waits run out)
        tc_wait(full_b + sb, pb, A.err, A.wait_ns);  // the tokens' block is in shared memory
        TC_STAMP(2, b, 0)
        for (int p = 0; p < np; p++, gp++) {
          const uint32_t set = gp & 1;
          const int n = min(npad - p * S::PN, S::PN);
          // instruction descriptors: D s32, A u8, B s8, K-major; and the f16 one (D f32)
          const uint32_t nm = ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
          const uint32_t idesc = (2u << 4) | (1u << 10) | nm, idesc_h = (1u << 4) | nm;
          const uint32_t bp = bs + (uint32_t)p * (S::PN / 8) * TC_REC, acc = tmem + set * S::SET;
          const uint64_t dB = tc_desc(bp, 128u, (uint32_t)TC_REC);  // K chunks 128 B apart, 8-token groups a record apart
          const uint64_t dAm = tc_desc(am, TC_M * 16u, 128u), dBm = tc_desc(bp + TC_REC_BM, 128u, (uint32_t)TC_REC);
          const bool last = p == np - 1;
          if (gp >= 2) tc_wait(acc_free + set, ((gp >> 1) - 1) & 1, A.err, A.wait_ns);
          TC_STAMP(2, b, 1 + 2 * p)
          auto quarter = [&](int q) {
#pragma unroll
            for (int ks = 2 * q; ks < 2 * q + 2; ks++) {
              const uint64_t db = dB + (uint64_t)(ks * 16);  // two K chunks a step
              tc_mma_i8_ta(acc, tmem + S::A_HI + 8u * ks, db, idesc, ks > 0 ? 1u : 0u);
              tc_mma_i8_ta(acc + S::PN, tmem + S::A_LO + 8u * ks, db, idesc, ks > 0 ? 1u : 0u);
            }
            if (!Q6 && q == 1) tc_mma_f16(acc + 2u * S::PN, dAm, dBm, idesc_h, 0u);  // (the warps of quarters 0 and 1 write the mins)
            if (last) tc_commit(a_free + q);
          };
          if (p == 0) {
            // a quarter of K at a time, each as soon as its operand A is in tensor memory: the first quarters of a
            // block are stored while the last ones of the block before are still being multiplied
#pragma unroll
            for (int q = 0; q < 4; q++) {
              tc_wait(a_ready + q, gb & 1, A.err, A.wait_ns);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              if (el) quarter(q);
              __syncwarp();
            }
          } else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (el) {
#pragma unroll
              for (int q = 0; q < 4; q++) quarter(q);
            }
          }
          if (el) {
            tc_commit(acc_full + set);
            if (last) tc_commit(empty_b + sb);
          }
          __syncwarp();
          TC_STAMP(2, b, 2 + 2 * p)
        }
        if (++sb == NSB) { sb = 0; pb ^= 1; }
      }
    }
  } else if (warp == MW + 1) {
    // ================= the producer: one thread =================
    if (tc_elect()) {
      const uint32_t sRaw_a = tc_s32(sRaw), sB_a = tc_s32(sB);
      const int G = (int)gridDim.x;
      int cur = (int)blockIdx.x, nxt = cur + G;
      uint4 Tc = __ldcg(A.tiles + cur / A.row_tiles), Tn = make_uint4(TC_END, 0, 0, 0);  // (the list has room for every item of the grid)
      const int n_items = __ldcg(A.n_tiles) * A.row_tiles;
      uint32_t sr = 0, pr = 1, sb = 0, pb = 1;  // stages and the phases of their empty barriers (1: the first round does not wait)
      uint32_t nr = 0, nbk = 0;                 // copies issued per ring (for the end)
      bool ok = true;
      auto weights = [&](const uint4 &T, int ra, int b) {  // block b of the item's rows -> the next raw area (a box past the matrix reads zeros)
        const bool sh = T.x == TC_SHARED;
        const int el = sh ? 0 : (int)T.x;
        const CUtensorMap *m0 = sh ? A.ms0 : A.m0, *m1 = sh ? A.ms1 : A.m1;
        const uint32_t r = sRaw_a + sr * RAWB;
        uint64_t *fr = full_raw + sr;
        tc_mbar_expect(fr, (uint32_t)RAWB);
        // (a box costs the copy engine about 100 cycles + 3-4 a row: down tiles come as boxes of 128 rows)
        if (!Q6) {
          tc_tma3(r, m0, b * 144, ra, el, fr);
          if (!DOWN) tc_tma3(r + 64 * 144, m1, b * 144, ra, el, fr);
        } else {
          tc_tma3(r, m0, b * 128, ra, el, fr);
          if (!DOWN) tc_tma3(r + 64 * 128, m1, b * 128, ra, el, fr);
          tc_tma3(r + 16384, m0 + 1, b * 64, ra, el, fr);
          if (!DOWN) tc_tma3(r + 16384 + 64 * 64, m1 + 1, b * 64, ra, el, fr);
        }
        nr++;
        if (++sr == NS) { sr = 0; pr ^= 1; }
      };
      // the first item's weights, under the launch before this one (TC_EARLY_WEIGHTS)
      int early = 0;
      if (cur < n_items && (int)Tc.x >= 0)
        for (; early < min(NS, nb); early++) weights(Tc, (cur % A.row_tiles) * (DOWN ? TC_M : TC_M / 2), early);
      pm_pdl_wait();
      for (int k = 0; ok; k++) {
        const int s = k & (TC_IT - 1);
        if (k >= TC_IT && !tc_wait(it_empty + s, (uint32_t)((k / TC_IT - 1) & 1), A.err, A.wait_ns)) break;
        const bool end = cur >= n_items;
        const int rt = cur % A.row_tiles, ra = rt * (DOWN ? TC_M : TC_M / 2);  // first row of the box(es)
        items[s].t = end ? make_uint4(TC_END, 0, 0, 0) : Tc;
        items[s].r0 = ra;
        tc_mbar_arrive(it_full + s);
        if (end) break;
        // the item after next, and the next one's tile: asked for now, needed an item later
        const int fut = 2 * G + (int)atomicAdd(A.next, 1u);
        if (nxt < n_items) Tn = __ldcg(A.tiles + nxt / A.row_tiles);
        if ((int)Tc.x >= 0) {
          const uint32_t bytes = ((Tc.z + 15) >> 4) * (2u * TC_REC);
          const uint8_t *rec = A.rec + (size_t)(Tc.w >> 3) * nb * TC_REC;  // the tile's first record
          for (int b = 0; b < nb; b++) {
            // ---- the weights of block b ----
            if (early > 0) {
              early--;
            } else {
              if (nr >= NS && !tc_wait(empty_raw + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
              TC_STAMP(3, b, 0)
              weights(Tc, ra, b);
            }
            // ---- the tokens' records of block b -> their area ----
            if (nbk >= NSB && !tc_wait(empty_b + sb, pb, A.err, A.wait_ns)) { ok = false; break; }
            TC_STAMP(3, b, 1)
            tc_mbar_expect(full_b + sb, bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             sB_a + sb * S::BST),
                         "l"(rec + (size_t)b * bytes), "r"(bytes), "r"(tc_s32(full_b + sb))
                         : "memory");
            nbk++;
            if (++sb == NSB) { sb = 0; pb ^= 1; }
          }
        }
        cur = nxt;
        nxt = fut;
        Tc = Tn;
      }
      // the last copies have landed before the CTA gives up its shared memory
      for (uint32_t i = 1; i <= NS && i <= nr; i++) {
        const uint32_t g = nr - i;
        tc_landed(full_raw + g % NS, (g / NS) & 1);
      }
      for (uint32_t i = 1; i <= NSB && i <= nbk; i++) {
        const uint32_t g = nbk - i;
        tc_landed(full_b + g % NSB, (g / NSB) & 1);
      }
    }
    __syncwarp();
  } else if (warp < MW) {
    // ================= the workers =================
    // unpack: thread = (row m of the tile, part of the block): the quarters q of K that are the part's, K values
    // 64 q .. 64 q + 63 = TMEM columns 16 q .. 16 q + 15 of each plane. The same thread adds row m's float terms
    // (TMEM lane m) for its part of a pass's token columns, so the row's (d, dmin) stay in registers.
    constexpr int QN = 4 / PARTS;  // quarters a thread
    // (redux results live in uniform registers, as the addresses of tensor memory have to: large tiles 1 to 2 % faster,
    // and the small shape, which has other registers to spare, slower)
    const int m = tid & 127, part = PARTS == 4 ? (int)__reduce_max_sync(PM_FULL, (unsigned)warp >> 2) : warp >> 2;
    const uint32_t tlane = tmem + (PARTS == 4 ? __reduce_max_sync(PM_FULL, 32u * (warp & 3)) << 16 : (uint32_t)(32 * (warp & 3)) << 16);
    const float nz = __uint_as_float((uint32_t)A.neg_zero2);
    const uint64_t nz2 = tc_pack2(nz, nz);
    uint32_t gb = 0, gp = 0;  // blocks whose operand A this CTA has stored, passes whose float terms it has added
    uint32_t sr = 0, pr = 0;  // the next raw stage and its phase
    uint32_t sf = 0, pf = 0;  // the tokens' stage of the block whose float terms come next, and its phase
    TcItem it;
    for (int k = 0; next_item(k, it); k++) {
      const uint4 T = it.t;
      const bool sh = T.x == TC_SHARED;  // the shared expert: no biases, no routing weight
      const int el = sh ? 0 : (int)T.x, nvalid = (int)T.z, npad = (nvalid + 15) & ~15, r0 = it.r0;
      if (el < 0) {  // an expert another rank holds: zeros (down) / nothing to do (gate/up)
        if (DOWN)
          for (int i = tid; i < nvalid * TC_M; i += S::NW) {
            const int n = i / TC_M, mm = i % TC_M;
            if (r0 + mm < rows) A.out[(size_t)(T.y + n) * rows + r0 + mm] = 0.0f;
          }
        continue;
      }
      const bool second = !DOWN && m >= 64;  // the row belongs to the up matrix
      const int mrow = r0 + (second ? m - 64 : m);
      // (the item's code exists once per number of passes a block: with one loop for all the row sums moved
      // between registers at every join)
      const float *bias0 = sh ? nullptr : A.bias0, *wts = sh ? nullptr : A.wts;
      auto run = [&](auto passes) {
        constexpr int NP = decltype(passes)::value, CH = S::CW / 2;
        // columns of the last pass that are this thread's (the others have all CW)
        const int ewl = PARTS == 4 ? (npad - (NP - 1) * S::PN) / PARTS : S::CW;
        // gate/up: the routing weight of the columns this thread will activate (half of its own: see the epilogue),
        // pass p in lanes CH p ...
        float wreg = 1.0f;
        if (!DOWN && wts && lane < NP * CH) {
          const int p = lane / CH, i = lane % CH, ew = p == NP - 1 ? ewl : S::CW;
          const int n = p * S::PN + part * ew + (second ? ew >> 1 : 0) + i;
          if (i < (ew >> 1) && n < nvalid) wreg = wts[A.pair_src[T.y + n]];
        }
        const uint8_t *dptr = nullptr, *sptr = nullptr;  // Q6_K: the row's f16 scales and the thread's sub-scales, a block ahead
        uint32_t scw_n[QN], d_n = 0;
        if (Q6) {
          const size_t row = (size_t)min(mrow, rows - 1) * nb;
          dptr = (second ? (sh ? A.ds1 : A.d1 + (size_t)el * A.d1_stride) : (sh ? A.ds0 : A.d0 + (size_t)el * A.d0_stride)) + row * 2;
          sptr = (second ? (sh ? A.ss1 : A.s1 + (size_t)el * A.s1_stride) : (sh ? A.ss0 : A.s0 + (size_t)el * A.s0_stride)) + row * 16 +
                 4 * QN * part;
#pragma unroll
          for (int i = 0; i < QN; i++) scw_n[i] = __ldg((const uint32_t *)sptr + i);
          d_n = __ldg((const uint16_t *)dptr);
        }
        float rd = 0.0f, rdmin = 0.0f;  // the scales of the block at hand
        // quarter q of a block's weights in `raw` -> the two planes (and, quarters 0 and 1, a K chunk of the mins'
        // product). Rows past the matrix: the boxes hold zeros there (what Q6_K gives is never written out).
        auto unpack_q6 = [&](const uint8_t *raw, int q, uint32_t scw, uint32_t *ah, uint32_t *al) {
          // (TMA swizzles: 16-byte piece c of a ql row sits at c ^ (row & 7), of a qh row at c ^ ((row >> 1) & 3))
          const int hf = q >> 1, p2 = q & 1;
          const uint8_t *rq = raw + m * 128, *rh = raw + 16384 + m * 64;
          uint4 qlv[4], qhv[2];
#pragma unroll
          for (int j = 0; j < 4; j++) qlv[j] = *(const uint4 *)(rq + (((4 * hf + j) ^ (m & 7)) << 4));
#pragma unroll
          for (int j = 0; j < 2; j++) qhv[j] = *(const uint4 *)(rh + (((2 * hf + j) ^ ((m >> 1) & 3)) << 4));
#pragma unroll
          for (int qq = 0; qq < 2; qq++) {
#pragma unroll
            for (int lh = 0; lh < 2; lh++) {
              // 16 values: sub-block 8 hf + 2 qt + lh of the block, qt = 2 p2 + qq
              const uint4 qlw = qlv[2 * qq + lh];
              const uint4 qhw = qhv[lh];
              const int sv = (int)(int8_t)((scw >> (8 * (2 * qq + lh))) & 0xff);
              // z4 = 4 * (sv * (q - 32) + 4128) in [256, 32896]: its high byte is th, its low byte 4 * tl
              // (v + 4128 = 64 th + tl). The low plane holds 4 * tl, the fold takes a quarter of d.
              const uint32_t sv4 = (uint32_t)(4 * sv);
              const uint32_t kk = (uint32_t)(4 * (4128 - 32 * sv)) * 0x00010001u;
              const uint32_t ws[4] = {qlw.x, qlw.y, qlw.z, qlw.w}, hs[4] = {qhw.x, qhw.y, qhw.z, qhw.w};
              const int rot = (4 * p2 + 2 * qq - 4) & 31;  // brings the pair of high bits to bits 4, 5 of its byte
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const uint32_t qv = ((ws[i] >> (4 * p2)) & 0x0f0f0f0fu) | (__funnelshift_r(hs[i], hs[i], rot) & 0x30303030u);
                // two values per 32-bit product (16-bit lanes, each lane's result positive): values 0, 2 and 1, 3
                const uint32_t ze = __byte_perm(qv, 0u, 0x4240) * sv4 + kk;
                const uint32_t zo = __byte_perm(qv, 0u, 0x4341) * sv4 + kk;
                al[4 * (2 * qq + lh) + i] = __byte_perm(ze, zo, 0x6240);
                ah[4 * (2 * qq + lh) + i] = __byte_perm(ze, zo, 0x7351);
              }
            }
          }
        };
        auto unpack_q4 = [&](const uint8_t *raw, int q, uint32_t sc03, uint32_t sc47, uint32_t m03, uint32_t m47, uint32_t *ah,
                             uint32_t *al) {
          const uint8_t *rp = raw + m * 144 + 16 + 32 * q;
          const uint4 w0 = *(const uint4 *)rp, w1 = *(const uint4 *)(rp + 16);
          if (q < 2)  // the eight mins as f16, K chunk q of the f16 product (both hold m_0..m_7)
            *(uint4 *)(sAm + (gb & 1) * (2 * TC_M * 16) + (q * TC_M + m) * 16) =
                make_uint4(pm_bytes_to_half2(m03, 0x4140), pm_bytes_to_half2(m03, 0x4342),
                           pm_bytes_to_half2(m47, 0x4140), pm_bytes_to_half2(m47, 0x4342));
          const uint32_t scw = ((q & 2) ? sc47 : sc03) >> (16 * (q & 1));
          const uint32_t sc0 = scw & 0xffu, sc1 = (scw >> 8) & 0xffu;  // scales of sub-blocks 2q, 2q+1
          const uint32_t M4 = 0x0f0f0f0fu;
          // sub-block 2q = low nibbles -> K 64q .. 64q+31 ; sub-block 2q+1 = high -> K 64q+32 .. 64q+63
          const uint32_t v[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
          const uint32_t sh0 = sc0 >> 3, sl0 = sc0 & 7, sh1 = sc1 >> 3, sl1 = sc1 & 7;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint32_t lo = v[i] & M4, hi = (v[i] >> 4) & M4;
            ah[i] = lo * sh0;
            al[i] = lo * sl0;
            ah[8 + i] = hi * sh1;
            al[8 + i] = hi * sl1;
          }
        };

        uint64_t tot[NP * CH];  // row sums: pairs of columns, pass p in CH p ..
#pragma unroll
        for (int i = 0; i < NP * CH; i++) tot[i] = 0ull;
        // the float terms of the next pass (pass P of its block), in block order: TMEM lane m, the part's columns.
        // x.d of the block is visible once this thread has seen the tokens' barrier (long complete).
        uint32_t used = 0;  // of every word that the folds of a block read from the tokens' area (tc_mbar_arrive_used)
        auto fold = [&](auto pass, float d, float dm) {
          constexpr int P = decltype(pass)::value;
          if (P == 0) used = 0;
          constexpr bool LAST = P == NP - 1;
          const uint32_t set = gp & 1;
          const int ew = LAST ? ewl : S::CW, c0 = part * ew;
          if (P == 0) tc_wait(full_b + sf, pf, A.err, A.wait_ns);
          tc_wait(acc_full + set, (gp >> 1) & 1, A.err, A.wait_ns);
          gp++;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t acc = tlane + set * S::SET + (uint32_t)c0;
          const uint8_t *rcd = sB + sf * S::BST + P * (S::PN / 8) * TC_REC;
          const uint64_t rd2 = tc_pack2(d, d), nm2 = tc_pack2(-dm, -dm);  // (x - y = x + (-y), -(a * b) = (-a) * b, to the bit)
          auto term2 = [&](uint32_t h0, uint32_t h1, uint32_t l0, uint32_t l1, uint32_t m0, uint32_t m1, uint64_t xd2, int xs0,
                           int xs1, uint64_t &t) {
            if (Q6) {
              // 4 * isum (exact in int32; (d / 4) * float(4 isum) rounds as d * float(isum) does)
              const int i0 = 256 * (int)h0 + ((int)l0 + xs0), i1 = 256 * (int)h1 + ((int)l1 + xs1);
              t = tc_add2(t, tc_fma2(xd2, tc_mul2(rd2, tc_pack2((float)i0, (float)i1)), nz2));
            } else {
              const int i0 = 8 * (int)h0 + (int)l0, i1 = 8 * (int)h1 + (int)l1;
              const uint64_t p = tc_fma2(rd2, tc_pack2((float)i0, (float)i1), nz2);
              const uint64_t q = tc_fma2(nm2, tc_pack2(__uint_as_float(m0), __uint_as_float(m1)), nz2);
              t = tc_add2(t, tc_fma2(xd2, tc_add2(p, q), nz2));
            }
          };
          // four columns (n: the first of them; column n: record n / 8, slot n % 8)
          auto cols4 = [&](const uint32_t *v0, const uint32_t *v1, const uint32_t *v2, int n, uint64_t &ta, uint64_t &tb) {
            const uint8_t *rx = rcd + (n >> 3) * TC_REC + (n & 7) * 4;
            const ulonglong2 x4 = *(const ulonglong2 *)(rx + TC_REC_XD);
            int4 s4 = make_int4(0, 0, 0, 0);
            if (Q6) s4 = *(const int4 *)(rx + TC_REC_XS);
            used ^= (uint32_t)x4.x ^ (uint32_t)s4.x;
            term2(v0[0], v0[1], v1[0], v1[1], v2[0], v2[1], x4.x, s4.x, s4.y, ta);
            term2(v0[2], v0[3], v1[2], v1[3], v2[2], v2[3], x4.y, s4.z, s4.w, tb);
          };
          auto group = [&](auto first) {  // columns C8 .. C8 + 7 of the thread, as far as there are that many
            constexpr int C8 = decltype(first)::value;
            uint64_t *t = tot + P * CH + C8 / 2;
            if (!LAST || PARTS == 2 || C8 + 8 <= ew) {
              uint32_t v0[8], v1[8], v2[8];
              tc_ld8<C8>(acc, v0);
              tc_ld8<S::PN + C8>(acc, v1);
              if (!Q6) tc_ld8<2 * S::PN + C8>(acc, v2);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              cols4(v0, v1, v2, c0 + C8, t[0], t[1]);
              cols4(v0 + 4, v1 + 4, v2 + 4, c0 + C8 + 4, t[2], t[3]);
            } else if (C8 < ew) {
              uint32_t v0[4], v1[4], v2[4];
              tc_ld4<C8>(acc, v0);
              tc_ld4<S::PN + C8>(acc, v1);
              if (!Q6) tc_ld4<2 * S::PN + C8>(acc, v2);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              cols4(v0, v1, v2, c0 + C8, t[0], t[1]);
            }
          };
          group(PassC<0>{});
          if constexpr (S::CW == 16) group(PassC<8>{});
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            tc_mbar_arrive(acc_free + set);
            if (LAST) tc_mbar_arrive_used(empty_b + sf, used, A.zero);  // this warp has read the block's x.d
          }
          if (LAST)
            if (++sf == NSB) { sf = 0; pf ^= 1; }
        };

        float rd_p = 0.0f, rdmin_p = 0.0f;  // the scales of the block before
        for (int b = 0; b < nb; b++, gb++) {
          // ---- operand A of block b -> registers -> tensor memory, each quarter once the last products that read
          // its columns are done (unpacked here, not before the float terms that run under the products: the 32
          // registers are not live there) ----
          uint32_t sc03, sc47, m03, m47, scw[QN];
          if (Q6) {
            rd = __fmul_rn(pm_f16(d_n), 0.25f);  // the products come out times 4
            const int bn = min(b + 1, nb - 1);
#pragma unroll
            for (int i = 0; i < QN; i++) {
              scw[i] = scw_n[i];
              scw_n[i] = __ldg((const uint32_t *)(sptr + 16 * bn) + i);
            }
            d_n = __ldg((const uint16_t *)(dptr + 2 * bn));
          }
          tc_wait(full_raw + sr, pr, A.err, A.wait_ns);
          const uint8_t *raw = sRaw + sr * RAWB;
          if (!Q6) {
            const uint4 hdr = *(const uint4 *)(raw + m * 144);
            rd = pm_f16(hdr.x);
            rdmin = pm_f16(hdr.x >> 16);
            pm_q4k_scmin_packed(hdr.y, hdr.z, hdr.w, sc03, sc47, m03, m47);
          }
#pragma unroll
          for (int i = 0; i < QN; i++) {
            const int q = part * QN + i;
            uint32_t ah[16], al[16];
            if (Q6) unpack_q6(raw, q, scw[i], ah, al);
            else unpack_q4(raw, q, sc03, sc47, m03, m47, ah, al);
            // (computed before the wait: left alone the compiler moves the arithmetic behind it)
#pragma unroll
            for (int j = 0; j < 16; j++) asm volatile("" : "+r"(ah[j]), "+r"(al[j]));
            TC_STAMP_W(b, 0)
            if (gb > 0) {
              tc_wait(a_free + q, (gb - 1) & 1, A.err, A.wait_ns);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            TC_STAMP_W(b, 1)
            tc_st16(tlane + S::A_HI + 16u * q, ah);
            tc_st16(tlane + S::A_LO + 16u * q, al);
            if (i == QN - 1) {  // the whole warp has read the area (its words are stored: an arrival is not ordered
              __syncwarp();     // behind loads whose registers nobody has read yet)
              if (lane == 0) tc_mbar_arrive(empty_raw + sr);
              if (++sr == NS) { sr = 0; pr ^= 1; }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            if (!Q6) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the mins
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(a_ready + q);
          }
          TC_STAMP_W(b, 2)
          // ---- the last pass of the block before (its products ran under this block's unpack), then all but the
          // last of this one ----
          if (b > 0) fold(PassC<NP - 1>{}, rd_p, rdmin_p);
          TC_STAMP_W(b, 3)
          if constexpr (NP > 1) fold(PassC<0>{}, rd, rdmin);
          if constexpr (NP > 2) fold(PassC<1>{}, rd, rdmin);
          if constexpr (NP > 3) fold(PassC<2>{}, rd, rdmin);
          TC_STAMP_W(b, 5)
          rd_p = rd;
          rdmin_p = rdmin;
        }
        fold(PassC<NP - 1>{}, rd_p, rdmin_p);

        const bool dead = *(volatile int *)A.err != 0;
        if (DOWN) {
          if (!dead && mrow < rows) {
            const float bd = bias0 ? bias0[(size_t)el * rows + mrow] : 0.0f;
            float *o = A.out + (size_t)T.y * rows + mrow;
#pragma unroll
            for (int i = 0; i < NP * CH; i++) {
              const int p = i / CH, c = 2 * (i % CH), ew = p == NP - 1 ? ewl : S::CW, n = p * S::PN + part * ew + c;
              float v0, v1;
              tc_unpack2(tot[i], v0, v1);
              if (bias0) {
                v0 = __fadd_rn(v0, bd);
                v1 = __fadd_rn(v1, bd);
              }
              if (c < ew && n < nvalid) o[(size_t)n * rows] = v0;
              if (c < ew && n + 1 < nvalid) o[(size_t)(n + 1) * rows] = v1;
            }
          }
        } else {
          // gate rows in tile rows 0..63, up rows in 64..127: a pass at a time the warps that hold the same
          // columns of both (w and w ^ 2) exchange their sums through shared memory; the gate warp activates
          // the first half of the columns, the up warp the second
          const float bg = bias0 && mrow < rows ? bias0[(size_t)el * rows + mrow] : 0.0f;
          const float bu = bias0 && mrow < rows ? A.bias1[(size_t)el * rows + mrow] : 0.0f;
          float *sx = sX + part * S::CW * TC_M;  // (the area of these warps, whatever the pass holds)
          const int mg = m & 63;
#pragma unroll
          for (int p = 0; p < NP; p++) {
            const int ew = p == NP - 1 ? ewl : S::CW;
            if (p) asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");  // the pass before has been read
#pragma unroll
            for (int i = 0; i < CH; i++)
              if (2 * i < ew) {
                float v0, v1;
                tc_unpack2(tot[CH * p + i], v0, v1);
                sx[(2 * i) * TC_M + m] = v0;
                sx[(2 * i + 1) * TC_M + m] = v1;
              }
            asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");
            const int h0 = second ? ew >> 1 : 0;
#pragma unroll 2
            for (int i = 0; i < (ew >> 1); i++) {
              const int c = h0 + i, n = p * S::PN + part * ew + c;
              float gv = sx[c * TC_M + mg], uv = sx[c * TC_M + 64 + mg];
              const float wt = __shfl_sync(PM_FULL, wreg, CH * p + i);
              if (bias0) {
                gv = __fadd_rn(gv, bg);
                uv = __fadd_rn(uv, bu);
              }
              if (!dead && n < nvalid && mrow < rows)
                A.out[(size_t)(T.y + n) * rows + mrow] = pm_act(A.act, A.act_limit, A.act_alpha, gv, uv, wt, wts != nullptr);
            }
          }
          // (nobody writes the area again before every warp has stored operand A of the next item)
        }
      };
      const int np = (npad + S::PN - 1) / S::PN;
      if (np == 1) run(PassC<1>{});
      else if (np == 2) run(PassC<2>{});
      else if constexpr (S::MP == 4) {
        if (np == 3) run(PassC<3>{});
        else run(PassC<4>{});
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MW)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)S::COLS) : "memory");
}

#define TC_FEW_AVG 6
static int tc_max_tiles(int n_pairs, int max_groups, int ntok = TC_FEW_TOKENS) {  // (the default: of every shape)
  int groups = max_groups < n_pairs ? max_groups : n_pairs;
  return n_pairs / ntok + groups;
}
size_t tc_tile_words(int n_pairs, int max_groups) { return 4 + 4 * (size_t)(tc_max_tiles(n_pairs, max_groups) + 1); }
// bytes of the records of n_pairs rows of `cols` values in at most max_groups groups (every group
// starts on a multiple of 16 rows)
size_t tc_rec_bytes(int n_pairs, int max_groups, int cols) {
  size_t groups = (size_t)(max_groups < n_pairs ? max_groups : n_pairs);
  size_t few = (size_t)n_pairs < TC_FEW_AVG * groups + TC_FEW_TOKENS * groups ? (size_t)n_pairs : 0;  // (tiles of few tokens: 16 rows each)
  size_t rows = (size_t)n_pairs + few + 16 * groups + 16;
  return (rows / 8 + 1) * (size_t)(cols / 256) * TC_REC;
}
TcTiles tc_tiles_of(uint32_t *buf, int n_pairs, int max_groups, int n_groups, int tokens, int shared_tokens, int ntok) {
  TcTiles t;
  // Tiles of at most 8 tokens (prefill_few.cu) where no group can have more, and while the groups hold up to 6 pairs on average: a
  // tile costs it 0.55 to 0.75 of one of k_tc's, and a group of more than 8 pairs makes two. A layer, there : here at 2 / 3 / 4 / 6 / 8
  // pairs a group: 256 experts x 7168 x 2048 963 : 1270, 1065 : 1382, 1161 : 1435, 1380 : 1478, 1654 : 1543; at 2 / 4 / 6 / 8 / 10: 128
  // experts x 2048 x 768, down Q6_K (four layers) 504 : 626, 531 : 632, 581 : 639, 653 : 681, 738 : 698; at 2 / 4 / 6 / 8 / 12: 64 x 2048 x
  // 1024 80 : 95, 95 : 108, 100 : 112, 109 : 115, 134 : 126.
  // Above that, tiles of up to 64 tokens and the two-CTA shape while the groups hold up to 16 pairs on average. A layer, this shape :
  // the one-CTA shape, us at 2 / 8 / 16 / 20 / 24 / 32 / 64 pairs a group:
  //   128 experts x 2048 x 768   152 : 190   164 : 213   207 : 222   221 : 232   238 : 241   273 : 250   388 : 330
  //    64 experts x 2048 x 1024  102 : 125   115 : 136   141 : 146   148 : 148   160 : 153   182 : 155   257 : 215
  //    32 experts x 7168 x 2048  234 : 301   252 : 322   313 : 335   332 : 343   333 : 349   407 : 363   611 : 487
  // (the line is below every crossing, 20 to 30 pairs: an average says little of the largest group)
  const int avg = n_pairs / (n_groups < n_pairs ? n_groups : n_pairs);
  t.ntok = ntok                                             ? ntok
           : tokens <= TC_FEW_TOKENS || avg <= TC_FEW_AVG ? TC_FEW_TOKENS
           : avg <= 16                                      ? TcShape<2>::NTOK
                                                            : TC_NMAX;
  t.even = ntok != 0;
  t.shared = shared_tokens > 0;
  t.max_tiles = tc_max_tiles(n_pairs, max_groups, t.ntok) + (shared_tokens + t.ntok - 1) / t.ntok;
  t.n = (int *)buf;
  t.next = (unsigned int *)buf + 1;
  t.tiles = (uint4 *)(buf + 4);
  return t;
}
cudaError_t launch_tc_tiles(const Launch &L, const LayerDev &ly, Groups g, const TcTiles &t) {
  return pm_launch(L, k_tc_tiles, 1, 512, 0, g, ly.first_local, ly.n_local, t.n, t.tiles, t.ntok, t.even, t.max_tiles);
}
static dim3 rows_grid(int n_rows, const TcTiles &t, int cols) {
  const long units = ((long)n_rows / 8 + 2 * t.max_tiles) * (cols / 256);  // (row group, block) records in all
  long gx = (units / t.max_tiles + 7) / 8;  // a warp writes about one record
  return dim3((unsigned)(gx < 1 ? 1 : gx), (unsigned)t.max_tiles);
}
static int few_records(const TcTiles &t, int weight_type) {
  return t.ntok == TC_FEW_TOKENS ? (weight_type == PM_TYPE_Q6_K ? 2 : 1) : 0;
}
void launch_tc_quant_rows(const Launch &L, int weight_type, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x,
                          uint8_t *rec) {
  const int few = few_records(t, weight_type);
  pm_launch(L, few == 0 ? k_tc_quant_rows<0> : (few == 1 ? k_tc_quant_rows<1> : k_tc_quant_rows<2>), rows_grid(n_rows, t, cols), 256, 0, t.n,
            t.tiles, src_row, cols, x, rec);
}
void launch_tc_rows(const Launch &L, int weight_type, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const int8_t *xq,
                    const float *xd, const uint16_t *xbm, const int32_t *xs, uint8_t *rec) {
  const int few = few_records(t, weight_type);
  pm_launch(L, few == 0 ? k_tc_rows<0> : (few == 1 ? k_tc_rows<1> : k_tc_rows<2>), rows_grid(n_rows, t, cols), 256, 0, t.n, t.tiles, src_row,
            cols, xq, xd, xbm, xs, rec);
}

template <int WT, bool DOWN, int PARTS> static cudaError_t tc_start(const Launch &L, const TcArgs &A, long items) {
  using S = TcShape<PARTS>;
  constexpr bool Q6 = WT == PM_TYPE_Q6_K;
  constexpr int NS = TcStages<PARTS, Q6, DOWN>::raw, NSB = TcStages<PARTS, Q6, DOWN>::tok;
  constexpr size_t smem = (size_t)NS * (Q6 ? TC_RAW_Q6 : TC_RAW_Q4) + (size_t)NSB * S::BST + (Q6 ? 0 : 2 * 2 * TC_M * 16) +
                          (DOWN ? 0 : S::XB) + (2 * NS + 2 * NSB + 12 + 2 * TC_IT) * 8 + TC_IT * sizeof(TcItem) + 16;
  static_assert(smem <= (S::CTAS == 1 ? 232448 : 115712), "more than an SM's shared memory");
  static SmemOptIn opt;
  const cudaError_t e = smem_optin(opt, k_tc<WT, DOWN, PARTS>, smem);
  if (e != cudaSuccess) return e;
  const long ctas = (long)S::CTAS * L.n_sm;
  return pm_launch(L, k_tc<WT, DOWN, PARTS>, dim3((unsigned)(items < ctas ? items : ctas)), S::NT, smem, A);
}
template <int WT, bool DOWN> static cudaError_t tc_start_shape(const Launch &L, const TcArgs &A, int ntok, long items) {
  return ntok == TC_NMAX ? tc_start<WT, DOWN, 4>(L, A, items) : tc_start<WT, DOWN, 2>(L, A, items);
}

// Tensor-core form of launch_gateup / launch_down for Q4_K or Q6_K weights and Q8x activations given as
// the records of the grouping's rows.
// shared_only: the list holds the shared expert's tiles alone (its width may differ).
cudaError_t launch_tc(const Launch &L, const LayerDev &ly, bool shared_only, bool down, const uint32_t *pair_src, const TcTiles &t,
                      const uint8_t *rec, const float *wts, float *out, int *err, unsigned long long wait_ns, int fault_block) {
  if (t.max_tiles == 0) return cudaSuccess;
  const WMat &W0 = down ? (shared_only ? ly.sdown : ly.down) : (shared_only ? ly.sgate : ly.gate), &W1 = ly.up;
  const WMat &S0 = down ? ly.sdown : ly.sgate, &S1 = ly.sup;
  const LayerMaps &M = *ly.maps;
  const WMaps &M0 = down ? M.down : M.gate, &MS0 = down ? M.sdown : M.sgate;
  const bool q6 = W0.type == PM_TYPE_Q6_K;
  TcArgs A;
  for (int i = 0; i < 2; i++) {
    A.m0[i] = M0.m[i];
    A.m1[i] = M.up.m[i];
    A.ms0[i] = MS0.m[i];
    A.ms1[i] = M.sup.m[i];
  }
  A.ss0 = S0.plane[2];
  A.ss1 = S1.plane[2];
  A.ds0 = S0.plane[3];
  A.ds1 = S1.plane[3];
  A.tiles = t.tiles;
  A.n_tiles = t.n;
  A.next = t.next + (down ? 1 : 0);
  A.rec = rec;
  A.s0 = W0.plane[2];
  A.s0_stride = W0.stride[2];
  A.s1 = W1.plane[2];
  A.s1_stride = W1.stride[2];
  A.d0 = W0.plane[3];
  A.d0_stride = W0.stride[3];
  A.d1 = W1.plane[3];
  A.d1_stride = W1.stride[3];
  A.bias0 = down ? ly.bias_down : ly.bias_gate;
  A.bias1 = down ? nullptr : ly.bias_up;
  A.wts = !down && ly.desc.weight_fold == PM_FOLD_BEFORE_DOWN ? wts : nullptr;
  A.pair_src = pair_src;
  A.out = out;
  A.err = err;
  A.wait_ns = wait_ns;
  A.zero = 0;
  A.fault_block = fault_block;
  A.neg_zero2 = 0x8000000080000000ull;
  A.row_tiles = down ? (W0.rows + TC_M - 1) / TC_M : (W0.rows + 63) / 64;
  A.cols = W0.cols;
  A.rows = W0.rows;
  A.act = ly.desc.act;
  A.act_limit = ly.desc.act_limit;
  A.act_alpha = ly.desc.act_alpha;
  const long items = (long)A.row_tiles * t.max_tiles;
  if (t.ntok == TC_FEW_TOKENS) return launch_tc_few(L, A, W0.type, down, items);
  cudaError_t e = q6 ? (down ? tc_start_shape<PM_TYPE_Q6_K, true>(L, A, t.ntok, items)
                             : tc_start_shape<PM_TYPE_Q6_K, false>(L, A, t.ntok, items))
                     : (down ? tc_start_shape<PM_TYPE_Q4_K, true>(L, A, t.ntok, items)
                             : tc_start_shape<PM_TYPE_Q4_K, false>(L, A, t.ntok, items));
  return e;
}
