// prefill_q32.cu - grouped expert products on Q8_0 / IQ4_NL / IQ4_XS weights and 32-value int8 activation blocks
// (src/q4x_cpu.rs:85-117) on the 5th-gen tensor cores: tcgen05.mma kind::i8, operand A and the int32 sums in tensor
// memory.
//
// One product of 128 x N x 32 is one block of every (row, token): its sums are exact integers, so the workers
// read them, convert and add (d_w * d_x) * sum in block order, each step rounded, and the result has the bits of the row
// kernels. A persistent pipeline like the other two (prefill_tc.cu, prefill_mx.cu): a producer thread brings the
// weights in by TMA (boxes of 128 K values) and the tokens' blocks by bulk copies; eight worker warps expand
// the weights into tensor memory and fold the sums of the stage before; two CTAs an SM.
//
// Bound by issue slots: the folds' 2.5 instructions an integer sum on pipes that do 64 a cycle, the expansion of the codes, and what
// a block costs whatever its columns; so a tile of at most 16 (32) tokens reads the sums of four (two) blocks at once, and one of at
// most 8 folds a quarter of the product's 16 columns. The row kernels took 8 dp4a a sum and read every weight once a token. 32 experts,
// 2560 x 640, top-8, IQ4_XS, a layer of 4 / 33 / 200 / 600 tokens: 78 / 144 / 218 / 410 us folding block by block behind one loop for
// every tile, 65 / 119 / 188 / 342 us here (gate/up + down on the row kernels: 33 tokens 585 us alone).
#include "tcgen.cuh"

#define Q32_M 128
#define Q32_N 64     /* tokens of a tile */
#define Q32_NW 8     /* worker warps */
#define Q32_NT (32 * (Q32_NW + 2))
#define Q32_KB 4     /* blocks of a stage */
#define Q32_NSR 3
#define Q32_NSB 3
#define Q32_NACC 3   /* slots of 64 columns of sums */
#define Q32_ACC 64u  /* tensor memory: two stages of operand A, then the sums */
#define Q32_BST (Q32_N * 36 * Q32_KB)
#define Q32_IT 4
#define Q32_END 0xfffffffeu

struct Q32Args {
  CUtensorMap m0, m1;     // values of gate or down, of up
  const uint8_t *s0, *s1; // their planes of scales
  size_t s0_stride, s1_stride;
  const uint4 *tiles;
  const int *n_tiles;
  unsigned int *next;
  const uint8_t *rec;     // the tokens' blocks (k_q32_rows)
  const float *bias0, *bias1;
  const float *wts;
  const uint32_t *pair_src;
  float *out;             // gate/up: h [P][ff]; down: eo [P][d]
  int *err;
  unsigned long long wait_ns;
  uint32_t zero;  // 0 (see tc_mbar_arrive_used)
  uint64_t neg_zero2;     // (-0, -0): see tc_fma2
  int row_tiles;
  int cols, rows;
  int act;
  float act_limit, act_alpha;
};

// f32 rows -> 32-value int8 blocks (`Q8::new`, src/q4x_cpu.rs:23-37, the steps of k_quant_q8_32) in the products'
// order: per tile and block [2 K groups][rows][16 values], then the rows' scales, rows padded to 16 with zeros.
// nibbles: the order in which the codes of a 4-bit block come apart (q32_codes): 8 i + k holds value
// 4 i + k / 2 + 16 (k & 1). A thread a (row, block); neighbouring lanes write neighbouring 16 bytes.
__global__ void __launch_bounds__(128) k_q32_rows(const int *__restrict__ n_tiles, const uint4 *__restrict__ tiles,
                                                  const uint32_t *__restrict__ src_row, int cols, const float *__restrict__ x,
                                                  int nibbles, int f16_scale, uint8_t *__restrict__ rec) {
#pragma unroll 1
  for (int practice = gridDim.x * gridDim.y <= PM_PRACTICE_CTAS; practice >= 0; practice--) {
    uint4 T = make_uint4(0, 0, 0, 0);
    if (!practice) {
      pm_pdl();
      T = tiles[blockIdx.y];  // (read beside the count: the list has room for every row of the grid)
      if ((int)blockIdx.y >= *n_tiles) return;
    }
    const int npad = practice ? 128 : ((int)T.z + 15) & ~15, nb = practice ? 1 : cols / 32;
    uint8_t *base = rec + (size_t)T.w * nb * 36;
    for (int u = practice ? (int)threadIdx.x : (int)(blockIdx.x * 128 + threadIdx.x); u < nb * npad; u += gridDim.x * 128) {
      const int b = u / npad, r = u - b * npad;
      float v[32], a = 0.0f;
      const bool on = r < (int)T.z;
      const size_t row = on ? (src_row ? src_row[T.y + r] : T.y + r) : 0;
      const float4 *src = (const float4 *)(x + row * cols + 32 * b);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float z = practice ? 1.0f : 0.0f;
        const float4 f = on ? __ldg(src + i) : make_float4(z, z, z, z);
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
      }
#pragma unroll
      for (int i = 0; i < 32; i++) a = fmaxf(a, fabsf(v[i]));
      float s = 0.0f;
      uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (a != 0.0f) {
        const float id = __fdiv_rn(127.0f, a);
        s = __fdiv_rn(a, 127.0f);
        if (f16_scale) s = __half2float(__float2half_rn(s));
        uint32_t q[32];
#pragma unroll
        for (int i = 0; i < 32; i++) q[i] = (uint32_t)(int)fminf(fmaxf(roundf(__fmul_rn(v[i], id)), -127.0f), 127.0f) & 0xffu;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int c = 4 * (i >> 1) + 2 * (i & 1);  // (4-bit blocks: values c, c + 16, c + 1, c + 17)
          w[i] = nibbles ? q[c] | (q[c + 16] << 8) | (q[c + 1] << 16) | (q[c + 17] << 24)
                         : q[4 * i] | (q[4 * i + 1] << 8) | (q[4 * i + 2] << 16) | (q[4 * i + 3] << 24);
        }
      }
      uint8_t *dst = base + (size_t)b * npad * 36;
      if (!practice) {
        *(uint4 *)(dst + r * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        *(uint4 *)(dst + (npad + r) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
        *(float *)(dst + npad * 32 + r * 4) = s;
      }
    }
  }
}

// eight 4-bit codes -> two words of codebook values, nibble 0 first (src/q4x_cpu.rs:453-461): look-ups of both halves
// of the table by prmt, the third prmt takes a byte of one or the other by the code's top bit
__device__ __forceinline__ void q32_codes(uint32_t q, uint32_t &w0, uint32_t &w1) {
  const uint32_t s = q & 0x77777777u, p = ((q >> 1) & 0x44444444u) | 0x32103210u;
  w0 = __byte_perm(__byte_perm(0xbfad9881u, 0xf6eaddcfu, s), __byte_perm(0x26190d01u, 0x71594535u, s), p);
  w1 = __byte_perm(__byte_perm(0xbfad9881u, 0xf6eaddcfu, s >> 16), __byte_perm(0x26190d01u, 0x71594535u, s >> 16), p >> 16);
}

// blocks whose sums share a slot of 64 columns, of a tile of npad columns: fewer barriers for small tiles (the issuing warp fills the slots,
// the workers read them)
__host__ __device__ constexpr uint32_t q32_slot_blocks(uint32_t npad) { return npad <= 16 ? 4u : (npad <= 32 ? 2u : 1u); }

struct Q32Item {
  uint4 t;
  int r0;
  int pad[3];
};

template <int WT> struct Q32Raw {
  static constexpr bool NIB = WT != PM_TYPE_Q8_0;
  static constexpr int ROW = NIB ? 64 : 128;  // bytes of a row's 128 values
  static constexpr int BYTES = Q32_M * ROW;
};

template <int WT, bool DOWN>
__global__ void __launch_bounds__(Q32_NT, 2) k_tc_q32(const __grid_constant__ Q32Args A) {
  constexpr bool NIB = Q32Raw<WT>::NIB, XS = WT == PM_TYPE_IQ4_XS;
  constexpr int RAWB = Q32Raw<WT>::BYTES, RROW = Q32Raw<WT>::ROW, MW = Q32_NW;
  constexpr int RPC = DOWN ? Q32_M : Q32_M / 2;  // matrix rows of an item
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sRaw = smem, *sB = sRaw + Q32_NSR * RAWB;
  float *sX = (float *)(sB + Q32_NSB * Q32_BST);  // gate/up: exchange [64 tokens][128 rows]
  Q32Item *items = (Q32Item *)((uint8_t *)sX + (DOWN ? 0 : Q32_N * Q32_M * 4));
  uint64_t *full_raw = (uint64_t *)(items + Q32_IT), *empty_raw = full_raw + Q32_NSR, *full_b = empty_raw + Q32_NSR;
  uint64_t *empty_b = full_b + Q32_NSB, *a_ready = empty_b + Q32_NSB, *a_free = a_ready + 2, *acc_full = a_free + 2;
  uint64_t *acc_free = acc_full + Q32_NACC, *it_full = acc_free + Q32_NACC, *it_empty = it_full + Q32_IT;
  uint32_t *tmem_slot = (uint32_t *)(it_empty + Q32_IT);
  const int nb = A.cols / 32, rows = A.rows, nst = (nb + Q32_KB - 1) / Q32_KB;
  const int tid = threadIdx.x, warp = __shfl_sync(PM_FULL, tid >> 5, 0), lane = tid & 31;

  pm_pdl_trigger();
  if (warp == MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_s32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < Q32_NSR; i++) {
      tc_mbar_init(full_raw + i, 1);
      tc_mbar_init(empty_raw + i, MW);
    }
    for (int i = 0; i < Q32_NSB; i++) {
      tc_mbar_init(full_b + i, 1);
      tc_mbar_init(empty_b + i, 1 + MW);  // the products' commit and the workers (scales)
    }
    for (int i = 0; i < 2; i++) {
      tc_mbar_init(a_ready + i, MW);
      tc_mbar_init(a_free + i, 1);
    }
    for (int i = 0; i < Q32_NACC; i++) {
      tc_mbar_init(acc_full + i, 1);
      tc_mbar_init(acc_free + i, MW);
    }
    for (int i = 0; i < Q32_IT; i++) {
      tc_mbar_init(it_full + i, 1);
      tc_mbar_init(it_empty + i, 1 + MW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __reduce_max_sync(PM_FULL, *tmem_slot);
  if (warp != MW + 1) pm_pdl_wait();  // (the producer waits later)
  auto next_item = [&](int k, Q32Item &it) -> bool {
    const int s = k & (Q32_IT - 1);
    const bool ok = tc_wait(it_full + s, (uint32_t)((k / Q32_IT) & 1), A.err, A.wait_ns);
    it = items[s];
    __syncwarp();
    if (lane == 0) tc_mbar_arrive_used(it_empty + s, it.t.x ^ (uint32_t)it.r0, A.zero);
    return ok && it.t.x != Q32_END;
  };

  if (warp == MW) {
    // ================= the issuing warp =================
    const uint32_t el = tc_elect() ? 1u : 0u;
    const uint32_t sB_a = tc_s32(sB);
    uint32_t st = 0, sb = 0, pb = 0, slot = 0, ps = 1;
    Q32Item it;
    for (int k = 0; next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      const uint32_t npad = (__reduce_max_sync(PM_FULL, it.t.z) + 15u) & ~15u, G = q32_slot_blocks(npad);
      // instruction descriptor: D s32, A and B s8, both K-major, N = npad, M = 128
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((npad >> 3) << 17) | ((uint32_t)(Q32_M >> 4) << 24);
      for (int s = 0; s < nst; s++, st++) {
        const uint32_t a = st & 1, nblk = (uint32_t)min(Q32_KB, nb - s * Q32_KB);
        const uint64_t dB = tc_desc(sB_a + sb * Q32_BST, npad * 16u, 128u);
        tc_wait(full_b + sb, pb, A.err, A.wait_ns);
        tc_wait(a_ready + a, (st >> 1) & 1, A.err, A.wait_ns);
        for (uint32_t b0 = 0; b0 < nblk; b0 += G) {
          tc_wait(acc_free + slot, ps, A.err, A.wait_ns);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (el) {
            for (uint32_t b = b0; b < b0 + G && b < nblk; b++)
              tc_mma_i8_ta(tmem + Q32_ACC + slot * 64u + (b - b0) * npad, tmem + a * 32u + b * 8u, dB + (uint64_t)(b * npad * 36u >> 4),
                           idesc, 0u);
            tc_commit(acc_full + slot);
          }
          __syncwarp();
          if (++slot == Q32_NACC) { slot = 0; ps ^= 1; }
        }
        if (el) {
          tc_commit(a_free + a);
          tc_commit(empty_b + sb);
        }
        __syncwarp();
        if (++sb == Q32_NSB) { sb = 0; pb ^= 1; }
      }
    }
  } else if (warp == MW + 1) {
    // ================= the producer: one thread =================
    if (tc_elect()) {
      const uint32_t sRaw_a = tc_s32(sRaw), sB_a = tc_s32(sB);
      const int G = (int)gridDim.x;
      int cur = (int)blockIdx.x, nxt = cur + G;
      uint4 Tc = __ldcg(A.tiles + cur / A.row_tiles), Tn = make_uint4(Q32_END, 0, 0, 0);  // (the list has room for every item of the grid)
      const int n_items = __ldcg(A.n_tiles) * A.row_tiles;
      uint32_t sr = 0, pr = 1, sb = 0, pb = 1, nr = 0, ntk = 0;  // (copies issued per ring)
      bool ok = true;
      auto weights = [&](int el, int r0, int q) {  // stage q of the item's rows (a box past the matrix reads zeros)
        const uint32_t r = sRaw_a + sr * RAWB;
        tc_mbar_expect(full_raw + sr, (uint32_t)RAWB);
        tc_tma3(r, &A.m0, q * RROW, r0, el, full_raw + sr);  // boxes of 128 rows (down) or 64
        if (!DOWN) tc_tma3(r + RAWB / 2, &A.m1, q * RROW, r0, el, full_raw + sr);
        nr++;
        if (++sr == Q32_NSR) { sr = 0; pr ^= 1; }
      };
      // the first item's weights, under the launch before this one (TC_EARLY_WEIGHTS, prefill_tc.cuh)
      int early = 0;
      if (cur < n_items && (int)Tc.x >= 0)
        for (; early < min(Q32_NSR, nst); early++) weights((int)Tc.x, (cur % A.row_tiles) * RPC, early);
      pm_pdl_wait();
      for (int k = 0; ok; k++) {
        const int s = k & (Q32_IT - 1);
        if (k >= Q32_IT && !tc_wait(it_empty + s, (uint32_t)((k / Q32_IT - 1) & 1), A.err, A.wait_ns)) break;
        const bool end = cur >= n_items;
        const int r0 = (cur % A.row_tiles) * RPC;
        Q32Item it;
        it.t = end ? make_uint4(Q32_END, 0, 0, 0) : Tc;
        it.r0 = r0;
        items[s] = it;
        tc_mbar_arrive(it_full + s);
        if (end) break;
        const int fut = 2 * G + (int)atomicAdd(A.next, 1u);  // (needed an item later)
        if (nxt < n_items) Tn = __ldcg(A.tiles + nxt / A.row_tiles);
        if ((int)Tc.x >= 0) {
          const int el = (int)Tc.x;
          const uint32_t per_block = ((Tc.z + 15) >> 4) * (16u * 36u);
          const uint8_t *rec = A.rec + (size_t)Tc.w * nb * 36;
          for (int q = 0; q < nst; q++) {
            if (early > 0) {
              early--;
            } else {
              if (nr >= Q32_NSR && !tc_wait(empty_raw + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
              weights(el, r0, q);
            }
            if (ntk >= Q32_NSB && !tc_wait(empty_b + sb, pb, A.err, A.wait_ns)) { ok = false; break; }
            const uint32_t bytes = per_block * (uint32_t)min(Q32_KB, nb - q * Q32_KB);
            tc_mbar_expect(full_b + sb, bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sB_a + sb * Q32_BST),
                         "l"(rec + (size_t)q * (per_block * Q32_KB)), "r"(bytes), "r"(tc_s32(full_b + sb))
                         : "memory");
            ntk++;
            if (++sb == Q32_NSB) { sb = 0; pb ^= 1; }
          }
        }
        cur = nxt;
        nxt = fut;
        Tc = Tn;
      }
      // the last copies have landed before the CTA gives up its shared memory
      for (uint32_t i = 1; i <= Q32_NSR && i <= nr; i++) tc_landed(full_raw + (nr - i) % Q32_NSR, ((nr - i) / Q32_NSR) & 1);
      for (uint32_t i = 1; i <= Q32_NSB && i <= ntk; i++) tc_landed(full_b + (ntk - i) % Q32_NSB, ((ntk - i) / Q32_NSB) & 1);
    }
    __syncwarp();
  } else {
    // ================= the workers =================
    // expand: thread = (row m of the tile; blocks 2 part, 2 part + 1 of a stage); fold: row m, half `part` of the tokens
    const int m = tid & 127, part = (int)__reduce_max_sync(PM_FULL, (unsigned)warp >> 2);
    const bool up = !DOWN && m >= 64;
    // (redux results live in uniform registers, as the addresses of tensor memory have to)
    const uint32_t tlane = tmem + (__reduce_max_sync(PM_FULL, 32u * (warp & 3)) << 16);
    uint32_t st = 0, sr = 0, pr = 0, sb = 0, slot = 0, pf = 0;
    Q32Item it;
    for (int k = 0; next_item(k, it); k++) {
      const uint4 T = it.t;
      const int el = (int)T.x, nvalid = (int)__reduce_max_sync(PM_FULL, T.z), r0 = it.r0;
      const uint32_t npad = ((uint32_t)nvalid + 15u) & ~15u;
      // columns this thread folds: half of the tokens (of a tile of at most 8: a quarter of the product's 16 columns)
      const int ew = nvalid <= 8 ? 4 : (int)npad >> 1, e0 = part * ew;
      const int row = r0 + (DOWN ? m : (m & 63));
      float *out = A.out + (size_t)T.y * rows + row;
      if (el < 0) {  // an expert another rank holds: zeros (down) / nothing to do (gate/up)
        if (DOWN)
          for (int i = tid; i < nvalid * RPC; i += 32 * Q32_NW) {
            const int n = i / RPC, mm = i - n * RPC;
            if (r0 + mm < rows) A.out[(size_t)(T.y + n) * rows + r0 + mm] = 0.0f;
          }
        continue;
      }
      // the scales of a stage: four f16, or the 8-byte header of
      // the stage's 256-value block
      const uint8_t *sp = (up ? A.s1 + (size_t)el * A.s1_stride : A.s0 + (size_t)el * A.s0_stride) +
                          (size_t)min(row, rows - 1) * (XS ? nb : 2 * nb);
      TcBytes8 sc_n;
      auto load_scales = [&](int s) {
        if (XS) sc_n.a = __ldg((const unsigned long long *)(sp + (s >> 1) * 8));
        else sc_n.load(sp + 8 * s);
      };
      uint64_t acc[Q32_N / 4];
#pragma unroll
      for (int i = 0; i < Q32_N / 4; i++) acc[i] = 0;
      // the sums of a stage for tiles of at most 16 and at most 32 tokens, W columns a thread: the blocks of a slot are read at once
      auto fold_slots = [&](auto width, auto blocks, int s, unsigned long long sc) {
        constexpr int W = decltype(width)::value, B = decltype(blocks)::value, NC = 64 / B;  // columns of a block
        const int nblk = min(Q32_KB, nb - s * Q32_KB);
        const uint8_t *xd = sB + sb * Q32_BST + NC * 32 + e0 * 4;
        const float d = XS ? pm_f16((uint32_t)sc) : 0.0f;
        // XS: the codes of the stage's four scales, low nibbles and two high bits; else four f16 scales
        uint32_t low = (uint32_t)(sc >> 32) >> (16 * (s & 1)), high = (uint32_t)sc >> (16 + 8 * (s & 1));
        uint32_t used = 0;
#pragma unroll 1
        for (int b0 = 0; b0 < nblk; b0 += B) {
          tc_wait(acc_full + slot, pf, A.err, A.wait_ns);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = tlane + Q32_ACC + slot * 64u + (uint32_t)e0;
          uint32_t v[B][W];
#pragma unroll
          for (int b = 0; b < B; b++) {  // (a block that is not there: whatever its columns hold)
            if (W == 4) tc_ld4<0>(at + NC * b, v[b]);
#pragma unroll
            for (int u = 0; u < W / 8; u++) tc_ld8<0>(at + NC * b + 8 * u, v[b] + 8 * u);
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int b = 0; b < B; b++)
            if (b0 + b < nblk) {
              float dw;
              if (XS) dw = __fmul_rn(d, (float)((int)(((low >> (4 * b)) & 15u) | (((high >> (2 * b)) & 3u) << 4)) - 32));
              else dw = pm_f16((uint32_t)(sc >> (16 * b)));
              const uint64_t dw2 = tc_pack2(dw, dw);
#pragma unroll
              for (int u = 0; u < W; u += 4) {
                const ulonglong2 x2 = *(const ulonglong2 *)(xd + b * (NC * 36) + u * 4);
                used ^= (uint32_t)x2.x;
                const uint64_t s0 = tc_pack2(__int2float_rn((int)v[b][u]), __int2float_rn((int)v[b][u + 1]));
                const uint64_t s1 = tc_pack2(__int2float_rn((int)v[b][u + 2]), __int2float_rn((int)v[b][u + 3]));
                acc[u / 2] = tc_add2(acc[u / 2], tc_fma2(tc_mul2(dw2, x2.x), s0, A.neg_zero2));
                acc[u / 2 + 1] = tc_add2(acc[u / 2 + 1], tc_fma2(tc_mul2(dw2, x2.y), s1, A.neg_zero2));
              }
            }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(acc_free + slot);
          if (++slot == Q32_NACC) { slot = 0; pf ^= 1; }
          if (B < Q32_KB) {
            xd += B * (NC * 36);
            low >>= 4 * B;
            high >>= 2 * B;
            sc >>= 16 * (B & 3);
          }
        }
        if (lane == 0) tc_mbar_arrive_used(empty_b + sb, used, A.zero);
        if (++sb == Q32_NSB) sb = 0;
      };
      auto fold = [&](int s, unsigned long long sc) {
        if (npad == 16u) {
          if (ew == 4) fold_slots(PassC<4>(), PassC<(int)q32_slot_blocks(16)>(), s, sc);
          else fold_slots(PassC<8>(), PassC<(int)q32_slot_blocks(16)>(), s, sc);
          return;
        }
        if (npad == 32u) {
          fold_slots(PassC<16>(), PassC<(int)q32_slot_blocks(32)>(), s, sc);
          return;
        }
        static_assert(q32_slot_blocks(48) == 1 && q32_slot_blocks(Q32_N) == 1, "one block a slot from here on");
        const int nblk = min(Q32_KB, nb - s * Q32_KB);
        const uint8_t *xd = sB + sb * Q32_BST + npad * 32u + e0 * 4;
        // (a slot a block; not unrolled: with four copies the workers waited for instructions, not for the pipes)
#pragma unroll 1
        for (int b = 0; b < nblk; b++) {
          tc_wait(acc_full + slot, pf, A.err, A.wait_ns);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = tlane + Q32_ACC + slot * 64u + (uint32_t)e0;
          float dw;
          if (XS) {  // d * (ls - 32) of sub-block ib (src/q4x_cpu.rs:102-117)
            const int ib = 4 * (s & 1) + b;
            const uint32_t lo = (uint32_t)sc, hi = (uint32_t)(sc >> 32);
            const int ls = (int)((hi >> (4 * ib)) & 15) | (int)((((lo >> 16) >> (2 * ib)) & 3) << 4);
            dw = __fmul_rn(pm_f16(lo), (float)(ls - 32));
          } else {
            dw = pm_f16((uint32_t)(sc >> (16 * b)));
          }
          const uint64_t dw2 = tc_pack2(dw, dw);
          auto half = [&](int c) {  // columns c .. c + 15
            uint32_t v[16];
            tc_ld8<0>(at + c, v);
            tc_ld8<8>(at + c, v + 8);
            ulonglong2 x2[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x2[u] = *(const ulonglong2 *)(xd + (c + 4 * u) * 4);
#pragma unroll
            for (int u = 0; u < 4; u++) {
              x2[u].x = tc_mul2(dw2, x2[u].x);
              x2[u].y = tc_mul2(dw2, x2[u].y);
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int u = 0; u < 16; u += 4) {
              const uint64_t s0 = tc_pack2(__int2float_rn((int)v[u]), __int2float_rn((int)v[u + 1]));
              const uint64_t s1 = tc_pack2(__int2float_rn((int)v[u + 2]), __int2float_rn((int)v[u + 3]));
              uint64_t *ac = acc + (c + u) / 2;
              ac[0] = tc_add2(ac[0], tc_fma2(x2[u / 4].x, s0, A.neg_zero2));
              ac[1] = tc_add2(ac[1], tc_fma2(x2[u / 4].y, s1, A.neg_zero2));
            }
          };
          half(0);
          half(16);  // (24 columns: the last 8 are not used)
          xd += npad * 36u;
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(acc_free + slot);
          if (++slot == Q32_NACC) { slot = 0; pf ^= 1; }
        }
        __syncwarp();
        uint32_t used = 0;  // (every read of the scales - of four tokens - went into their sums)
#pragma unroll
        for (int i = 0; i < Q32_N / 4; i += 2) used ^= (uint32_t)acc[i];
        if (lane == 0) tc_mbar_arrive_used(empty_b + sb, used, A.zero);
        if (++sb == Q32_NSB) sb = 0;
      };
      unsigned long long sc = 0;
      load_scales(0);
      for (int s = 0; s < nst; s++, st++) {
        const unsigned long long sc_p = sc;
        sc = XS ? sc_n.a : sc_n.get();
        if (s + 1 < nst) load_scales(s + 1);
        tc_wait(full_raw + sr, pr, A.err, A.wait_ns);
        const uint8_t *raw = sRaw + sr * RAWB + m * RROW;
        uint32_t w[16];
        if constexpr (NIB) {
          uint4 q[2];
#pragma unroll
          for (int j = 0; j < 2; j++)  // (TMA swizzle of 64-byte rows: 16-byte piece i sits at i ^ (row / 2 & 3))
            q[j] = *(const uint4 *)(raw + (((2 * part + j) ^ ((m >> 1) & 3)) << 4));
#pragma unroll
          for (int j = 0; j < 2; j++) {
            q32_codes(q[j].x, w[8 * j], w[8 * j + 1]);
            q32_codes(q[j].y, w[8 * j + 2], w[8 * j + 3]);
            q32_codes(q[j].z, w[8 * j + 4], w[8 * j + 5]);
            q32_codes(q[j].w, w[8 * j + 6], w[8 * j + 7]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) {  // (of 128-byte rows: at i ^ (row & 7))
            const uint4 q = *(const uint4 *)(raw + (((4 * part + j) ^ (m & 7)) << 4));
            w[4 * j] = q.x; w[4 * j + 1] = q.y; w[4 * j + 2] = q.z; w[4 * j + 3] = q.w;
          }
        }
        const uint32_t a = st & 1;
        if (st >= 2) {
          tc_wait(a_free + a, ((st >> 1) - 1) & 1, A.err, A.wait_ns);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        tc_st16(tlane + a * 32u + 16u * part, w);
        __syncwarp();  // (an arrival is not ordered behind loads whose registers nobody has read yet)
        if (lane == 0) tc_mbar_arrive(empty_raw + sr);
        if (++sr == Q32_NSR) { sr = 0; pr ^= 1; }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(a_ready + a);
        if (s > 0) fold(s - 1, sc_p);
      }
      fold(nst - 1, sc);
      // ---- epilogue ----
      const bool on = row < rows && *(volatile int *)A.err == 0;
      const float b0 = A.bias0 && row < rows ? A.bias0[(size_t)el * rows + row] : 0.0f;
      if constexpr (DOWN) {
#pragma unroll
        for (int i = 0; i < Q32_N / 4; i++)
          if (2 * i < ew) {
            float v[2];
            tc_unpack2(acc[i], v[0], v[1]);
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const int n = e0 + 2 * i + u;
              if (A.bias0) v[u] = __fadd_rn(v[u], b0);  // src/oss_batch.rs:89
              if (on && n < nvalid) out[(size_t)n * rows] = v[u];
            }
          }
      } else {  // gate rows in lanes 0..63, up rows in 64..127: the warps w and w ^ 2 exchange through shared memory
        float *sx = sX + part * (Q32_N / 2) * Q32_M;
        const float b1 = A.bias0 && row < rows ? A.bias1[(size_t)el * rows + row] : 0.0f;
#pragma unroll
        for (int i = 0; i < Q32_N / 4; i++)
          if (2 * i < ew) {
            float v[2];
            tc_unpack2(acc[i], v[0], v[1]);
            sx[(2 * i) * Q32_M + m] = v[0];
            sx[(2 * i + 1) * Q32_M + m] = v[1];
          }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * part + (warp & 1)) : "memory");
        const int f = up ? ew >> 1 : 0;
#pragma unroll 2
        for (int i = f; i < f + (ew >> 1); i++) {
          const int n = e0 + i;
          if (on && n < nvalid) {
            float gv = sx[i * Q32_M + (m & 63)], uv = sx[i * Q32_M + 64 + (m & 63)];
            if (A.bias0) {
              gv = __fadd_rn(gv, b0);
              uv = __fadd_rn(uv, b1);
            }
            const float wt = A.wts ? A.wts[A.pair_src[T.y + n]] : 1.0f;
            out[(size_t)n * rows] = pm_act(A.act, A.act_limit, A.act_alpha, gv, uv, wt, A.wts != nullptr);
          }
        }
        // (nobody writes the area again before every warp has expanded the next item's first stage)
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

bool q32_weights(int type) { return type == PM_TYPE_Q8_0 || type == PM_TYPE_IQ4_NL || type == PM_TYPE_IQ4_XS; }
int q32_tile_tokens() { return Q32_N; }
size_t q32_rec_bytes(int n_pairs, int max_groups, int cols) {
  const size_t groups = (size_t)(max_groups < n_pairs ? max_groups : n_pairs);
  return ((size_t)n_pairs + 15 * groups + 16) * (cols / 32) * 36;
}
void launch_q32_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x, int weight_type,
                     bool f16_scale, uint8_t *rec) {
  const long units = ((long)n_rows + 15 * t.max_tiles) * (cols / 32);
  const long gx = (units / t.max_tiles + 127) / 128;
  pm_launch(L, k_q32_rows, dim3((unsigned)(gx < 1 ? 1 : gx), (unsigned)t.max_tiles), 128, 0, t.n, t.tiles, src_row, cols, x,
            (int)(weight_type != PM_TYPE_Q8_0), (int)f16_scale, rec);
}

template <int WT, bool DOWN> static cudaError_t q32_start(const Launch &L, const Q32Args &A, long items) {
  constexpr size_t smem = (size_t)Q32_NSR * Q32Raw<WT>::BYTES + (size_t)Q32_NSB * Q32_BST + (DOWN ? 0 : Q32_N * Q32_M * 4) +
                          Q32_IT * sizeof(Q32Item) + (2 * Q32_NSR + 2 * Q32_NSB + 4 + 2 * Q32_NACC + 2 * Q32_IT) * 8 + 16;
  static_assert(smem <= 115712, "two CTAs an SM");
  static SmemOptIn opt;
  const cudaError_t e = smem_optin(opt, k_tc_q32<WT, DOWN>, smem);
  if (e != cudaSuccess) return e;
  const long ctas = 2L * L.n_sm;
  return pm_launch(L, k_tc_q32<WT, DOWN>, dim3((unsigned)(items < ctas ? items : ctas)), Q32_NT, smem, A);
}

// Tensor-core form of launch_gateup / launch_down for 32-value activation blocks given as the grouping's records.
cudaError_t launch_tc_q32(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                          const uint8_t *rec, const float *wts, float *out, int *err, unsigned long long wait_ns) {
  if (t.max_tiles == 0) return cudaSuccess;
  const WMat &W0 = down ? ly.down : ly.gate, &W1 = ly.up;
  Q32Args A;
  A.m0 = (down ? ly.maps->down : ly.maps->gate).m[down ? 1 : 0];  // boxes of 128 or 64 rows
  A.m1 = ly.maps->up.m[0];
  A.s0 = W0.plane[1];
  A.s0_stride = W0.stride[1];
  A.s1 = W1.plane[1];
  A.s1_stride = W1.stride[1];
  A.tiles = t.tiles;
  A.n_tiles = t.n;
  A.next = t.next + (down ? 1 : 0);
  A.rec = rec;
  A.bias0 = down ? ly.bias_down : ly.bias_gate;
  A.bias1 = down ? nullptr : ly.bias_up;
  A.wts = !down && ly.desc.weight_fold == PM_FOLD_BEFORE_DOWN ? wts : nullptr;
  A.pair_src = pair_src;
  A.out = out;
  A.err = err;
  A.wait_ns = wait_ns;
  A.zero = 0;
  A.neg_zero2 = 0x8000000080000000ull;
  const int rpc = down ? Q32_M : Q32_M / 2;
  A.row_tiles = (W0.rows + rpc - 1) / rpc;
  A.cols = W0.cols;
  A.rows = W0.rows;
  A.act = ly.desc.act;
  A.act_limit = ly.desc.act_limit;
  A.act_alpha = ly.desc.act_alpha;
  const long items = (long)A.row_tiles * t.max_tiles;
  switch (W0.type) {
    case PM_TYPE_Q8_0: return down ? q32_start<PM_TYPE_Q8_0, true>(L, A, items) : q32_start<PM_TYPE_Q8_0, false>(L, A, items);
    case PM_TYPE_IQ4_NL: return down ? q32_start<PM_TYPE_IQ4_NL, true>(L, A, items) : q32_start<PM_TYPE_IQ4_NL, false>(L, A, items);
    case PM_TYPE_IQ4_XS: return down ? q32_start<PM_TYPE_IQ4_XS, true>(L, A, items) : q32_start<PM_TYPE_IQ4_XS, false>(L, A, items);
  }
  return cudaErrorInvalidValue;
}
