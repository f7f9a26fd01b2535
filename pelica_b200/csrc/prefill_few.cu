// prefill_few.cu - the products of prefill_tc.cu for tiles of at most 8 tokens: decode of a few sequences, and calls that
// give an expert a few tokens. Same weights, same integer sums, same order of the float terms, so the same bits.
//
// With so few tokens a product of 16 columns is mostly padding and the unpack of the weights decides. Here the codes go to
// the tensor cores WITHOUT their sub-block scales and every product step of 32 K values has its own accumulator:
//   Q4_K: a step is one sub-block, D_j = sum_i nib_ji * xq_ji; isum = sum_j sc_j * D_j is the worker's, eight multiply-adds
//         an output. One u8 plane in place of two and no multiplication of the codes. msum as in k_tc.
//   Q6_K: a step is two sub-blocks of 16. The tokens' record comes twice, once with the second sub-block of every step zero
//         and once with the first: columns 0..7 hold the sums of sub-block 2 j, columns 8..15 of 2 j + 1, at no
//         further cost (16 columns are the least a step has). Operand A is q - 32 as s8, so no offset term.
// A warp spends about 180 instructions on a block of 128 rows (of Q4_K and up to 4 tokens) where k_tc's small shape, whose
// issue slots were three quarters full, takes 315; what is left to wait for are the weights' bytes. A layer, k_tc : here:
//   256 experts x 7168 x 2048 (Q4_K), shared expert: 1 token 93 : 73 us, 64 tokens 1,409 : 1,077 us (6.2 GB of weights)
//   128 experts x 2048 x 768 (Q4_K, down Q6_K), 8 tokens 93 : 75 us
#include <cuda_fp16.h>

#include "prefill_tc.cuh"

#define FW_NW 8                     /* worker warps: 128 rows x two halves of K (and of the tokens) */
#define FW_NT (32 * (FW_NW + 2))
#define FW_COLS 256u
// tensor memory: the sums of eight steps (16 columns each), the mins' product, operand A
#define FW_MINS 128u
#define FW_A 192u
template <bool Q6, bool DOWN> struct FewShape {
  static constexpr int NREC = Q6 ? 2 : 1;
  static constexpr int BST = NREC * TC_REC;
  static constexpr int RAWB = Q6 ? TC_RAW_Q6 : TC_RAW_Q4;
  static constexpr int NS = Q6 ? 4 : 5;                 // weights' stages
  static constexpr int NSB = Q6 ? (DOWN ? 3 : 2) : 4;   // tokens' stages: what fits two CTAs an SM
  static constexpr int AM = Q6 ? 0 : TC_M * 32;         // the mins' operand, two of them
  static constexpr int XB = DOWN ? 0 : TC_FEW_TOKENS * TC_M * 4;
  static constexpr size_t SMEM = (size_t)NS * RAWB + NSB * BST + 2 * AM + XB + (2 * NS + 2 * NSB + 3 + 2 * TC_IT) * 8 +
                                 TC_IT * sizeof(TcItem) + 16;
};

template <int OFF> __device__ __forceinline__ void fw_ld2(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2 + %3];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr), "n"(OFF));
}
// CPT columns of the thread's lane
template <int CPT, int OFF> __device__ __forceinline__ void fw_ld(uint32_t taddr, uint32_t *r) {
  if constexpr (CPT == 4) tc_ld4<OFF>(taddr, r);
  else fw_ld2<OFF>(taddr, r);
}
template <int CPT, int J, int N, int STEP> __device__ __forceinline__ void fw_ld_all(uint32_t taddr, uint32_t (*r)[CPT]) {
  if constexpr (J < N) {
    fw_ld<CPT, J * STEP>(taddr, r[J]);
    fw_ld_all<CPT, J + 1, N, STEP>(taddr, r);
  }
}
// signed byte I of w
template <int I> __device__ __forceinline__ int fw_sbyte(uint32_t w) {
  int r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"(I | ((8 | I) << 4) | ((8 | I) << 8) | ((8 | I) << 12)));
  return r;
}

template <int WT, bool DOWN>
__global__ void __launch_bounds__(FW_NT, 2) k_tc_few(const __grid_constant__ TcArgs A) {
  constexpr bool Q6 = WT == PM_TYPE_Q6_K;
  using S = FewShape<Q6, DOWN>;
  constexpr int NS = S::NS, NSB = S::NSB, MW = FW_NW;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sRaw = smem;                                  // [NS] blocks of the 128 rows
  uint8_t *sB = sRaw + NS * S::RAWB;                     // [NSB] x [1 or 2 records]
  uint8_t *sAm = sB + NSB * S::BST;                      // Q4_K: [2][2 chunks][128 rows][8 f16]
  float *sX = (float *)(sAm + 2 * S::AM);                // gate/up: exchange [8 tokens][128 rows]
  TcItem *items = (TcItem *)((uint8_t *)sX + S::XB);
  uint64_t *full_raw = (uint64_t *)(items + TC_IT), *empty_raw = full_raw + NS;
  uint64_t *full_b = empty_raw + NS, *empty_b = full_b + NSB;
  // a_ready: operand A of a block is in tensor memory; done: its products are complete; read: so are the reads of their sums
  uint64_t *a_ready = empty_b + NSB, *done = a_ready + 1, *read = done + 1;
  uint64_t *it_full = read + 1, *it_empty = it_full + TC_IT;
  uint32_t *tmem_slot = (uint32_t *)(it_empty + TC_IT);

  const int nb = A.cols / 256, rows = A.rows;
  const int tid = threadIdx.x, warp = __shfl_sync(PM_FULL, tid >> 5, 0), lane = tid & 31;

  pm_pdl_trigger();
  if (warp == MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_s32(tmem_slot)), "r"(FW_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NS; i++) {
      tc_mbar_init(full_raw + i, 1);
      tc_mbar_init(empty_raw + i, MW);
    }
    for (int i = 0; i < NSB; i++) {
      tc_mbar_init(full_b + i, 1);
      tc_mbar_init(empty_b + i, MW);  // (after the float terms, behind the block's products)
    }
    tc_mbar_init(a_ready, MW);
    tc_mbar_init(done, 1);
    tc_mbar_init(read, MW);
    for (int i = 0; i < TC_IT; i++) {
      tc_mbar_init(it_full + i, 1);
      tc_mbar_init(it_empty + i, 1 + MW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __reduce_max_sync(PM_FULL, *tmem_slot);
  if (warp != MW + 1) pm_pdl_wait();  // (the producer's weights do not wait: see there)
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
    // instruction descriptors (k_tc): D s32, A u8 or (Q6_K) s8, B s8, N = 16; the f16 one of the mins
    constexpr uint32_t nm = (2u << 17) | ((uint32_t)(TC_M >> 4) << 24);
    constexpr uint32_t idesc = (2u << 4) | (Q6 ? 1u << 7 : 0u) | (1u << 10) | nm, idesc_h = (1u << 4) | nm;
    uint32_t gb = 0, sb = 0, pb = 0;
    TcItem it;
    for (int k = 0; next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      for (int b = 0; b < nb; b++, gb++) {
        if (A.fault_block >= 0 && b >= A.fault_block) break;  // (test hook: the workers' waits run out)
        const uint32_t bs = sB_a + sb * S::BST;
        // K chunks 128 B apart; columns 8..15: the second record (Q6_K), the same one once more (Q4_K)
        const uint64_t dB = tc_desc(bs, 128u, Q6 ? (uint32_t)TC_REC : 0u);
        const uint64_t dAm = tc_desc(sAm_a + (gb & 1) * S::AM, TC_M * 16u, 128u), dBm = tc_desc(bs + TC_REC_BM, 128u, 0u);
        tc_wait(full_b + sb, pb, A.err, A.wait_ns);
        if (gb > 0) tc_wait(read, (gb - 1) & 1, A.err, A.wait_ns);
        tc_wait(a_ready, gb & 1, A.err, A.wait_ns);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (el) {
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc_mma_i8_ta(tmem + 16u * ks, tmem + FW_A + 8u * ks, dB + (uint64_t)(ks * 16), idesc, 0u);
          if (!Q6) tc_mma_f16(tmem + FW_MINS, dAm, dBm, idesc_h, 0u);
          tc_commit(done);
        }
        __syncwarp();
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
      auto weights = [&](const uint4 &T, int ra, int b) {  // block b of the item's rows -> the next stage
        const bool sh = T.x == TC_SHARED;
        const int el = sh ? 0 : (int)T.x;
        const CUtensorMap *m0 = sh ? A.ms0 : A.m0, *m1 = sh ? A.ms1 : A.m1;
        const uint32_t r = sRaw_a + sr * S::RAWB;
        uint64_t *fr = full_raw + sr;
        tc_mbar_expect(fr, (uint32_t)S::RAWB);  // (a box past the matrix reads zeros)
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
      // The first item's weights, under the launch before this one, which makes the tokens' records (TC_EARLY_WEIGHTS)
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
        const int fut = 2 * G + (int)atomicAdd(A.next, 1u);  // (needed an item later)
        if (nxt < n_items) Tn = __ldcg(A.tiles + nxt / A.row_tiles);
        if ((int)Tc.x >= 0) {
          const uint8_t *rec = A.rec + (size_t)(Tc.w >> 3) * nb * TC_REC;  // the tile's first record
          for (int b = 0; b < nb; b++) {
            if (early > 0) {
              early--;
            } else {
              if (nr >= NS && !tc_wait(empty_raw + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
              weights(Tc, ra, b);
            }
            if (nbk >= NSB && !tc_wait(empty_b + sb, pb, A.err, A.wait_ns)) { ok = false; break; }
            tc_mbar_expect(full_b + sb, (uint32_t)S::BST);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             sB_a + sb * S::BST),
                         "l"(rec + (size_t)b * S::BST), "r"((uint32_t)S::BST), "r"(tc_s32(full_b + sb))
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
  } else {
    // ================= the workers =================
    // thread = (row m of the tile, half `part` of a block's K values, and of the tile's tokens when it comes to the sums)
    const int m = tid & 127, part = (int)__reduce_max_sync(PM_FULL, (unsigned)warp >> 2);
    const uint32_t tlane = tmem + (__reduce_max_sync(PM_FULL, 32u * (warp & 3)) << 16);
    const float nz = __uint_as_float((uint32_t)A.neg_zero2);
    const uint64_t nz2 = tc_pack2(nz, nz);
    uint32_t gb = 0;          // blocks whose operand A has been stored
    uint32_t sr = 0, pr = 0;  // the next weights' stage and its phase
    uint32_t sf = 0, pf = 0;  // the tokens' stage of the block whose float terms come next, and its phase
    TcItem it;
    for (int k = 0; next_item(k, it); k++) {
      const uint4 T = it.t;
      const bool sh = T.x == TC_SHARED;  // the shared expert: no biases, no routing weight
      const int el = sh ? 0 : (int)T.x, nvalid = (int)__reduce_max_sync(PM_FULL, T.z), r0 = it.r0;
      if (el < 0) {  // an expert another rank holds: zeros (down) / nothing to do (gate/up)
        if (DOWN)
          for (int i = tid; i < nvalid * TC_M; i += 32 * FW_NW) {
            const int n = i / TC_M, mm = i % TC_M;
            if (r0 + mm < rows) A.out[(size_t)(T.y + n) * rows + r0 + mm] = 0.0f;
          }
        continue;
      }
      const bool second = !DOWN && m >= 64;  // the row belongs to the up matrix
      const int mrow = r0 + (second ? m - 64 : m);
      const float *bias0 = sh ? nullptr : A.bias0, *wts = sh ? nullptr : A.wts;
      auto run = [&](auto columns) {
        constexpr int CPT = decltype(columns)::value;  // columns of the tile a thread folds
        const int c0 = part * CPT;
        const bool mine = c0 < nvalid;  // (one part's columns may all be padding)
        // gate/up: the routing weight of the columns this thread will activate (half of its own: see the epilogue)
        float wt[CPT / 2];
        if (!DOWN)
#pragma unroll
          for (int i = 0; i < CPT / 2; i++) {
            const int n = c0 + (second ? CPT / 2 : 0) + i;
            wt[i] = wts && n < nvalid ? wts[A.pair_src[T.y + n]] : 1.0f;
          }
        const uint8_t *dptr = nullptr, *sptr = nullptr;  // Q6_K: the row's f16 scales and sub-scales, a block ahead
        uint4 sc_n = make_uint4(0, 0, 0, 0);
        uint32_t d_n = 0;
        if (Q6) {
          const size_t row = (size_t)min(mrow, rows - 1) * nb;
          dptr = (second ? (sh ? A.ds1 : A.d1 + (size_t)el * A.d1_stride) : (sh ? A.ds0 : A.d0 + (size_t)el * A.d0_stride)) + row * 2;
          sptr = (second ? (sh ? A.ss1 : A.s1 + (size_t)el * A.s1_stride) : (sh ? A.ss0 : A.s0 + (size_t)el * A.s0_stride)) + row * 16;
          sc_n = __ldg((const uint4 *)sptr);
          d_n = __ldg((const uint16_t *)dptr);
        }
        uint64_t tot[CPT / 2];  // row sums: pairs of columns
#pragma unroll
        for (int i = 0; i < CPT / 2; i++) tot[i] = 0ull;
        // the float terms of a block whose products are complete, in block order
        auto fold = [&](const uint4 &sc, float d, float dm) {
          uint32_t used = 0;
          if (mine) {
            tc_wait(full_b + sf, pf, A.err, A.wait_ns);  // (long complete: makes x.d visible to this thread)
            const float *rx = (const float *)(sB + sf * S::BST + TC_REC_XD) + c0;
            uint64_t xd2[CPT / 2];
            if constexpr (CPT == 4) {
              const ulonglong2 x4 = *(const ulonglong2 *)rx;
              xd2[0] = x4.x;
              xd2[1] = x4.y;
            } else {
              xd2[0] = *(const uint64_t *)rx;
            }
            used = (uint32_t)xd2[0];
            int isum[CPT];
            [[maybe_unused]] uint32_t mins[CPT];
#pragma unroll
            for (int c = 0; c < CPT; c++) isum[c] = 0;
            uint32_t v[8][CPT];
            if constexpr (!Q6) {
              fw_ld_all<CPT, 0, 8, 16>(tlane + (uint32_t)c0, v);
              fw_ld<CPT, (int)FW_MINS>(tlane + (uint32_t)c0, mins);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 8; j++) {
                const int s = (int)__byte_perm(j < 4 ? sc.x : sc.y, 0u, 0x4440 | (j & 3));
#pragma unroll
                for (int c = 0; c < CPT; c++) isum[c] += s * (int)v[j][c];
              }
            } else {
              // sub-blocks 2 j, then sub-blocks 2 j + 1
              const uint32_t w[4] = {sc.x, sc.y, sc.z, sc.w};
              fw_ld_all<CPT, 0, 8, 16>(tlane + (uint32_t)c0, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 8; j++) {
                const int s = (j & 1) ? fw_sbyte<2>(w[j >> 1]) : fw_sbyte<0>(w[j >> 1]);
#pragma unroll
                for (int c = 0; c < CPT; c++) isum[c] += s * (int)v[j][c];
              }
              fw_ld_all<CPT, 0, 8, 16>(tlane + (uint32_t)c0 + 8u, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 8; j++) {
                const int s = (j & 1) ? fw_sbyte<3>(w[j >> 1]) : fw_sbyte<1>(w[j >> 1]);
#pragma unroll
                for (int c = 0; c < CPT; c++) isum[c] += s * (int)v[j][c];
              }
            }
            const uint64_t rd2 = tc_pack2(d, d), nm2 = tc_pack2(-dm, -dm);  // (x - y = x + (-y), -(a * b) = (-a) * b, to the bit)
#pragma unroll
            for (int i = 0; i < CPT / 2; i++) {
              const uint64_t p = tc_fma2(rd2, tc_pack2((float)isum[2 * i], (float)isum[2 * i + 1]), nz2);
              if constexpr (Q6) {
                tot[i] = tc_add2(tot[i], tc_fma2(xd2[i], p, nz2));
              } else {
                const uint64_t q = tc_fma2(nm2, tc_pack2(__uint_as_float(mins[2 * i]), __uint_as_float(mins[2 * i + 1])), nz2);
                tot[i] = tc_add2(tot[i], tc_fma2(xd2[i], tc_add2(p, q), nz2));
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane < 2) tc_mbar_arrive_used(lane == 0 ? read : empty_b + sf, used, A.zero);  // (the sums; x.d)
          if (++sf == NSB) { sf = 0; pf ^= 1; }
        };

        uint4 sc = make_uint4(0, 0, 0, 0), sc_p = sc;  // scales of the block at hand and of the one before (Q4_K: eight bytes)
        float rd = 0.0f, rdmin = 0.0f, rd_p = 0.0f, rdmin_p = 0.0f;
        for (int b = 0; b < nb; b++, gb++) {
          uint32_t w[32];  // the part's K values: quarters 2 part, 2 part + 1 (16 columns of operand A each)
          if (Q6) {
            sc = sc_n;
            rd = pm_f16(d_n);
            const int bn = min(b + 1, nb - 1);
            sc_n = __ldg((const uint4 *)(sptr + 16 * bn));
            d_n = __ldg((const uint16_t *)(dptr + 2 * bn));
          }
          tc_wait(full_raw + sr, pr, A.err, A.wait_ns);
          const uint8_t *raw = sRaw + sr * S::RAWB;
          if constexpr (Q6) {
            // (TMA swizzles: 16-byte piece c of a ql row sits at c ^ (row & 7), of a qh row at c ^ ((row >> 1) & 3))
            const uint8_t *rq = raw + m * 128, *rh = raw + 16384 + m * 64;
            uint4 qlv[4], qhv[2];
#pragma unroll
            for (int j = 0; j < 4; j++) qlv[j] = *(const uint4 *)(rq + (((4 * part + j) ^ (m & 7)) << 4));
#pragma unroll
            for (int j = 0; j < 2; j++) qhv[j] = *(const uint4 *)(rh + (((2 * part + j) ^ ((m >> 1) & 3)) << 4));
#pragma unroll
            for (int p2 = 0; p2 < 2; p2++)
#pragma unroll
              for (int qq = 0; qq < 2; qq++)
#pragma unroll
                for (int lh = 0; lh < 2; lh++) {
                  const uint4 qlw = qlv[2 * qq + lh], qhw = qhv[lh];
                  const uint32_t ws[4] = {qlw.x, qlw.y, qlw.z, qlw.w}, hs[4] = {qhw.x, qhw.y, qhw.z, qhw.w};
                  const int rot = (4 * p2 + 2 * qq - 4) & 31;  // brings the pair of high bits to bits 4, 5 of its byte
#pragma unroll
                  for (int i = 0; i < 4; i++) {
                    const uint32_t qv = ((ws[i] >> (4 * p2)) & 0x0f0f0f0fu) | (__funnelshift_r(hs[i], hs[i], rot) & 0x30303030u);
                    w[16 * p2 + 4 * (2 * qq + lh) + i] = (qv + 0x60606060u) ^ 0x80808080u;  // q - 32 (no byte carries: q < 64)
                  }
                }
          } else {
            const uint4 hdr = *(const uint4 *)(raw + m * 144);
            uint32_t m03, m47;
            rd = pm_f16(hdr.x);
            rdmin = pm_f16(hdr.x >> 16);
            pm_q4k_scmin_packed(hdr.y, hdr.z, hdr.w, sc.x, sc.y, m03, m47);
            // the eight mins as f16: K chunk `part` of the f16 product (both hold m_0..m_7)
            *(uint4 *)(sAm + (gb & 1) * S::AM + (part * TC_M + m) * 16) =
                make_uint4(pm_bytes_to_half2(m03, 0x4140), pm_bytes_to_half2(m03, 0x4342),
                           pm_bytes_to_half2(m47, 0x4140), pm_bytes_to_half2(m47, 0x4342));
            const uint8_t *rp = raw + m * 144 + 16 + 64 * part;
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const uint4 v0 = *(const uint4 *)(rp + 32 * q), v1 = *(const uint4 *)(rp + 32 * q + 16);
              const uint32_t v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
              for (int i = 0; i < 8; i++) {  // low nibbles: sub-block 4 part + 2 q; high ones: the next
                w[16 * q + i] = v[i] & 0x0f0f0f0fu;
                w[16 * q + 8 + i] = (v[i] >> 4) & 0x0f0f0f0fu;
              }
            }
          }
          // (computed before the wait: left alone the compiler moves the arithmetic behind it)
#pragma unroll
          for (int j = 0; j < 32; j++) asm volatile("" : "+r"(w[j]));
          if (gb > 0) {
            tc_wait(done, (gb - 1) & 1, A.err, A.wait_ns);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          tc_st32(tlane + FW_A + 32u * part, w);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          if (!Q6) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the mins
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          // operand A is there; the whole warp has read the weights' stage (its words are stored)
          if (lane < 2) tc_mbar_arrive(lane == 0 ? a_ready : empty_raw + sr);
          if (++sr == NS) { sr = 0; pr ^= 1; }
          // the float terms of the block before: its products ran under this block's unpack, and this block's start once
          // its sums have been read
          if (b > 0) fold(sc_p, rd_p, rdmin_p);
          sc_p = sc;
          rd_p = rd;
          rdmin_p = rdmin;
        }
        tc_wait(done, (gb - 1) & 1, A.err, A.wait_ns);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        fold(sc_p, rd_p, rdmin_p);

        const bool dead = *(volatile int *)A.err != 0;
        if (DOWN) {
          if (!dead && mrow < rows) {
            const float bd = bias0 ? bias0[(size_t)el * rows + mrow] : 0.0f;
            float *o = A.out + (size_t)T.y * rows + mrow;
#pragma unroll
            for (int i = 0; i < CPT / 2; i++) {
              float v[2];
              tc_unpack2(tot[i], v[0], v[1]);
#pragma unroll
              for (int u = 0; u < 2; u++) {
                const int n = c0 + 2 * i + u;
                if (bias0) v[u] = __fadd_rn(v[u], bd);
                if (n < nvalid) o[(size_t)n * rows] = v[u];
              }
            }
          }
        } else {
          // gate rows in tile rows 0..63, up rows in 64..127: the warps w and w ^ 2 exchange their sums through shared memory;
          // the gate warp activates the first half of the columns, the up warp the second
          const float bg = bias0 && mrow < rows ? bias0[(size_t)el * rows + mrow] : 0.0f;
          const float bu = bias0 && mrow < rows ? A.bias1[(size_t)el * rows + mrow] : 0.0f;
          float *sx = sX + c0 * TC_M;
          const int mg = m & 63;
#pragma unroll
          for (int i = 0; i < CPT / 2; i++) {
            float v0, v1;
            tc_unpack2(tot[i], v0, v1);
            sx[(2 * i) * TC_M + m] = v0;
            sx[(2 * i + 1) * TC_M + m] = v1;
          }
          asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");
#pragma unroll
          for (int i = 0; i < CPT / 2; i++) {
            const int c = (second ? CPT / 2 : 0) + i, n = c0 + c;
            if (n < nvalid) {
              float gv = sx[c * TC_M + mg], uv = sx[c * TC_M + 64 + mg];
              if (bias0) {
                gv = __fadd_rn(gv, bg);
                uv = __fadd_rn(uv, bu);
              }
              if (!dead && mrow < rows)
                A.out[(size_t)(T.y + n) * rows + mrow] = pm_act(A.act, A.act_limit, A.act_alpha, gv, uv, wt[i], wts != nullptr);
            }
          }
          // (nobody writes the area again before every warp has stored operand A of the next item)
        }
      };
      if (nvalid <= 4) run(PassC<2>{});
      else run(PassC<4>{});
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(FW_COLS) : "memory");
}

template <int WT, bool DOWN> static cudaError_t few_start(const Launch &L, const TcArgs &A, long items) {
  constexpr size_t smem = FewShape<WT == PM_TYPE_Q6_K, DOWN>::SMEM;
  static_assert(smem <= 115712, "two CTAs an SM");
  static SmemOptIn opt;
  const cudaError_t e = smem_optin(opt, k_tc_few<WT, DOWN>, smem);
  if (e != cudaSuccess) return e;
  const long ctas = 2L * L.n_sm;
  return pm_launch(L, k_tc_few<WT, DOWN>, dim3((unsigned)(items < ctas ? items : ctas)), FW_NT, smem, A);
}
cudaError_t launch_tc_few(const Launch &L, const TcArgs &A, int weight_type, bool down, long items) {
  if (weight_type == PM_TYPE_Q6_K) return down ? few_start<PM_TYPE_Q6_K, true>(L, A, items) : few_start<PM_TYPE_Q6_K, false>(L, A, items);
  return down ? few_start<PM_TYPE_Q4_K, true>(L, A, items) : few_start<PM_TYPE_Q4_K, false>(L, A, items);
}
