// prefill_mx.cu - grouped expert products on MXFP4 weights and f32 activations (the gpt-oss path,
// src/oss_prefill.rs:237,548) on the 5th-gen tensor cores: tcgen05.mma kind::f16 with bf16 operands, operand A
// and the f32 accumulators in tensor memory.
//
// MXFP4 weights are exact in bf16 (a one-bit mantissa times a power of two: the E2M1 code
// doubled, times the halved E8M0 scale, src/oss_kernels.rs:41-55), the f32 activations are
// not: each is split into bf16 pieces, x = x1 + x2, xi = bf16(what is left), and every K step runs once a
// piece into the same accumulator. Products of two bf16 values are exact in f32: what differs from the f32 reference
// path (src/oss_batch.rs:774-789) is the 2^-17 relative residue and the summation order; parity is the layer
// tolerance (1e-3 relative + 1e-4 of the RMS), not bits. For prompts whose experts get many tokens; calls with fewer
// tokens an expert run on prefill_mx8.cu.
//
// A persistent pipeline like the int8 kernel's (prefill_tc.cu): a producer thread brings the weights' nibbles in
// by TMA (boxes of 256 K values) and the tokens' pieces by one bulk copy a chunk of 64 K values; the workers decode
// a block of 32 codes a thread and store it to tensor memory, up to four chunks ahead of the products; work items
// come from a counter. One accumulator for the whole K (the block scale lives in the bf16 weight).
// A CTA takes 256 weight rows (128 gate rows and the same 128 rows of up, or 256 down rows) x 128 tokens. Both
// halves multiply one staging of the tokens' pieces, which halves what comes from L2: 31 bytes a cycle an SM; with 128
// rows it would be the limit, 62. Gate and up sums of an output sit in the same thread. Bound by the tensor pipe
// (1,050 cycles a chunk, 60 % of the time at 2048 tokens, 32 experts, d = ff = 2880) and by what the workers' decode
// adds where the two do not overlap: gate/up + down 2,110 -> 750 us against a kernel that staged decoded weights
// in shared memory and took 128 rows.
#include <cuda_bf16.h>

#include "mxsum.cuh"

#define MX_M 128
#define MX_KC 64   /* K values of a chunk */
#define MX_NA 4    /* chunks of operand A in tensor memory */
#define NPC 2      /* bf16 pieces of an activation */
#define MX_BOX (MX_M * 128)   /* nibbles of 128 rows x 256 K values */

struct MxShape {
  static constexpr int MT = 2;                 // 128-row halves of a CTA
  static constexpr int NW = 512, NT = NW + 64;
  static constexpr int NTOK = 128;
  static constexpr uint32_t COLS = 512;        // tensor memory: accumulators, then MX_NA chunks of operand A
  static constexpr uint32_t A0 = 256, ACH = MT * MX_KC / 2;  // first column, columns a chunk
  static constexpr int RAWB = MT * MX_BOX, NSR = 3;
  static constexpr int BST = NTOK * MX_KC * 2 * NPC, NSB = 4;
};

__device__ __forceinline__ void mx_mma_ta(uint32_t tmem_c, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_c),
      "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

// A block: 16 bytes of E2M1 codes (value j in the low nibble of byte j, value j + 16 in the high one) and its E8M0
// scale e -> 32 bf16. Two codes a word, 16 bits apart as they lie: word 2 j holds nibbles 0 and 4 of the j-th word (values
// 4 j, 4 j + 2), word 2 j + 1 nibbles 2 and 6 (4 j + 1, 4 j + 3), words 8 .. the same of the high nibbles (values 16 ..);
// k_mx_rows puts the tokens' values into the same order. The code's three magnitude bits at bits 8..6 of
// a bf16 are the code times 2^-126 (its subnormal included), so one multiplication by 2^(e - 1) makes the value; four
// ALU instructions and a multiplication a word, where look-ups of both bytes by prmt took ten (and the prmt, shifts
// and logic, 64 lanes a cycle, were what the workers waited for: 2,070 -> 1,150 cycles a chunk).
__device__ __forceinline__ uint32_t mx_mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void mx_codes(const uint4 q, uint32_t scale2, uint32_t *w) {
  const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    w[2 * j] = mx_mul2(((v[j] << 6) & 0x01c001c0u) | ((v[j] << 12) & 0x80008000u), scale2);
    w[8 + 2 * j] = mx_mul2(((v[j] << 2) & 0x01c001c0u) | ((v[j] << 8) & 0x80008000u), scale2);
    w[2 * j + 1] = mx_mul2(((v[j] >> 2) & 0x01c001c0u) | ((v[j] << 4) & 0x80008000u), scale2);
    w[8 + 2 * j + 1] = mx_mul2(((v[j] >> 6) & 0x01c001c0u) | (v[j] & 0x80008000u), scale2);
  }
}
// scales outside 2 .. 128
__device__ __forceinline__ void mx_codes_any(const uint4 q, uint32_t e, uint32_t *w) {
  if (e >= 2u && e < 250u) {  // 2^(e - 1) in two steps: 2^127 is the largest power a bf16 holds
    mx_codes(q, min(e + 126u, 254u) * 0x00800080u, w);
    const uint32_t more2 = (e > 128u ? e - 1u : 127u) * 0x00800080u;
#pragma unroll
    for (int i = 0; i < 16; i++) w[i] = mx_mul2(w[i], more2);
  } else {  // the scale's own subnormal branch (src/oss_kernels.rs:42-45) and scales near the top of the range: through f32
    const uint32_t v[4] = {q.x, q.y, q.z, q.w};
    const float s = pm_e8(e);
    auto cv = [&](uint32_t c) { return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(__fmul_rn(s, pm_e2m1(c & 15u)))); };
#pragma unroll
    for (int i = 0; i < 16; i++) {  // word i: nibbles n and n + 4 of word j
      const int j = (i & 7) >> 1, n = 2 * (i & 1) + (i >> 3);
      w[i] = cv(v[j] >> (4 * n)) | (cv(v[j] >> (4 * n + 16)) << 16);
    }
  }
}

struct MxArgs {
  CUtensorMap m0, m1;     // nibble planes of gate or down, of up
  const uint8_t *s0, *s1; // their planes of scale bytes
  size_t s0_stride, s1_stride;
  const uint4 *tiles;
  const int *n_tiles;
  unsigned int *next;
  const uint8_t *rec;     // the tokens' pieces (k_mx_rows)
  const uint8_t *w0, *w1;       // the nibbles, the f32 rows and the row of each pair (null: its own), for mx_repair
  size_t w0_stride, w1_stride;
  const float *x;
  const uint32_t *src_row;
  const float *bias0, *bias1;
  const float *wts;
  const uint32_t *pair_src;
  float *out;             // gate/up: h [P][ff]; down: eo [P][d]
  int *err;
  unsigned long long wait_ns;
  uint32_t zero;  // 0 (see tc_mbar_arrive_used)
  int row_tiles;
  int cols, rows;
  int act;
  float act_limit, act_alpha;
};

// f32 rows -> the products' operand: per tile and chunk of 64 K values [piece][8 K groups][rows][8 bf16], rows padded
// to 16 with zeros; the 8 values of a K group in the order the decoded weights have (0, 2, 1, 3, 4, 6, 5, 7). A thread a
// (row, K group), a warp 8 rows x 4 K groups: 128 neighbouring bytes of a row read, 128 neighbouring bytes of a K group written
// (a warp of 32 rows touched 32 lines a load, which is what bound it: 8192 rows x 2880 values 33 us).
__global__ void __launch_bounds__(256) k_mx_rows(const int *__restrict__ n_tiles, const uint4 *__restrict__ tiles,
                                                 const uint32_t *__restrict__ src_row, int cols, const float *__restrict__ x,
                                                 uint8_t *__restrict__ rec) {
  pm_pdl();
  const uint4 T = tiles[blockIdx.y];  // (read beside the count: the list has room for every row of the grid)
  if ((int)blockIdx.y >= *n_tiles) return;
  const int npad = ((int)T.z + 15) & ~15, nch = (cols + MX_KC - 1) / MX_KC;
  uint8_t *base = rec + (size_t)T.w * nch * (MX_KC * 2 * NPC);
  for (int u = blockIdx.x * 256 + threadIdx.x; u < nch * 8 * npad; u += gridDim.x * 256) {
    const int w = u >> 5, q = w / (npad >> 3), g = 4 * q + (u & 3), r = 8 * (w - q * (npad >> 3)) + ((u >> 2) & 7);  // K group of 8 values, row of the tile
    float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (r < (int)T.z && 8 * g < cols) {
      const size_t row = src_row ? src_row[T.y + r] : T.y + r;
      const float4 *src = (const float4 *)(x + row * cols + 8 * g);
      const float4 a = __ldg(src), b = __ldg(src + 1);  // (the order of mx_codes)
      v[0] = a.x; v[1] = a.z; v[2] = a.y; v[3] = a.w; v[4] = b.x; v[5] = b.z; v[6] = b.y; v[7] = b.w;
    }
    uint8_t *dst = base + (size_t)(g >> 3) * (npad * MX_KC * 2 * NPC) + ((g & 7) * npad + r) * 16;
#pragma unroll
    for (int p = 0; p < NPC; p++) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const __nv_bfloat16 a = __float2bfloat16_rn(v[2 * i]), b = __float2bfloat16_rn(v[2 * i + 1]);
        v[2 * i] = __fsub_rn(v[2 * i], __bfloat162float(a));
        v[2 * i + 1] = __fsub_rn(v[2 * i + 1], __bfloat162float(b));
        w[i] = (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
      }
      *(uint4 *)(dst + (size_t)p * npad * MX_KC * 2) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

struct MxItem {
  uint4 t;
  int r0;  // first row
  int pad[3];
};
#define MX_IT 4
#define MX_END 0xfffffffeu

template <bool DOWN>
__global__ void __launch_bounds__(MxShape::NT, 1) k_tc_mx(const __grid_constant__ MxArgs A) {
  using S = MxShape;
  constexpr int MW = S::NW / 32, NSR = S::NSR, NSB = S::NSB, MT = S::MT;
  constexpr int RPC = DOWN ? MT * MX_M : MX_M;  // matrix rows of an item
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sRaw = smem, *sB = sRaw + NSR * S::RAWB;
  MxItem *items = (MxItem *)(sB + NSB * S::BST);
  uint64_t *full_raw = (uint64_t *)(items + MX_IT), *empty_raw = full_raw + NSR, *full_b = empty_raw + NSR, *empty_b = full_b + NSB;
  uint64_t *a_ready = empty_b + NSB, *a_free = a_ready + MX_NA, *acc_full = a_free + MX_NA, *acc_free = acc_full + 1;
  uint64_t *it_full = acc_free + 1, *it_empty = it_full + MX_IT;
  uint32_t *tmem_slot = (uint32_t *)(it_empty + MX_IT);
  const int nbk = A.cols / 32, rows = A.rows, nch = (A.cols + MX_KC - 1) / MX_KC;
  const int tid = threadIdx.x, warp = __shfl_sync(PM_FULL, tid >> 5, 0), lane = tid & 31;

  pm_pdl_trigger();
  if (warp == MW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_s32(tmem_slot)), "r"(S::COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NSR; i++) {
      tc_mbar_init(full_raw + i, 1);
      tc_mbar_init(empty_raw + i, MW);
    }
    for (int i = 0; i < NSB; i++) {
      tc_mbar_init(full_b + i, 1);
      tc_mbar_init(empty_b + i, 1);  // the products' commit (nobody else reads the tokens' pieces)
    }
    for (int i = 0; i < MX_NA; i++) {
      tc_mbar_init(a_ready + i, MW / 2);
      tc_mbar_init(a_free + i, 1);
    }
    tc_mbar_init(acc_full, 1);
    tc_mbar_init(acc_free, MW);
    for (int i = 0; i < MX_IT; i++) {
      tc_mbar_init(it_full + i, 1);
      tc_mbar_init(it_empty + i, 1 + MW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __reduce_max_sync(PM_FULL, *tmem_slot);
  pm_pdl_wait();  // (barriers and tensor memory were prepared under the kernel before)
  auto next_item = [&](int k, MxItem &it) -> bool {
    const int s = k & (MX_IT - 1);
    const bool ok = tc_wait(it_full + s, (uint32_t)((k / MX_IT) & 1), A.err, A.wait_ns);
    it = items[s];
    __syncwarp();
    if (lane == 0) tc_mbar_arrive_used(it_empty + s, it.t.x ^ (uint32_t)it.r0, A.zero);
    return ok && it.t.x != MX_END;
  };

  if (warp == MW) {
    // ================= the issuing warp =================
    const uint32_t el = tc_elect() ? 1u : 0u;
    const uint32_t sB_a = tc_s32(sB);
    uint32_t st = 0, sb = 0, pb = 0, n_acc = 0;
    MxItem it;
    for (int k = 0; next_item(k, it); k++) {
      if ((int)it.t.x < 0) continue;
      const uint32_t npad = (__reduce_max_sync(PM_FULL, it.t.z) + 15u) & ~15u;
      // instruction descriptor: D f32, A and B bf16, both K-major, N = npad, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((npad >> 3) << 17) | ((uint32_t)(MX_M >> 4) << 24);
      if (n_acc > 0) tc_wait(acc_free, (n_acc - 1) & 1, A.err, A.wait_ns);  // the item before has been read
      for (int c = 0; c < nch; c++) {
        const uint32_t a = (uint32_t)c & 3u;
        const uint64_t dB = tc_desc(sB_a + sb * S::BST, npad * 16u, 128u);
        const int ksteps = min(4, (A.cols - c * MX_KC) / 16);  // (a trailing single block: 2 steps)
        tc_wait(full_b + sb, pb, A.err, A.wait_ns);
        tc_wait(a_ready + a, st & 1, A.err, A.wait_ns);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (el) {
#pragma unroll
          for (int h = 0; h < MT; h++)
#pragma unroll
            for (int ks = 0; ks < 4; ks++)
              if (ks < ksteps) {
#pragma unroll
                for (int p = 0; p < NPC; p++) {  // (a piece is npad * 128 bytes, a K step two groups of npad * 16)
                  const uint32_t at = tmem + S::A0 + a * S::ACH + h * (MX_KC / 2) + 8u * ks;
                  const uint64_t db = dB + (uint64_t)(p * npad * 8 + ks * npad * 2);
                  mx_mma_ta(tmem + h * 128u, at, db, idesc, (c > 0 || ks > 0 || p > 0) ? 1u : 0u);
                }
              }
          tc_commit(a_free + a);
          tc_commit(empty_b + sb);
          if (c == nch - 1) tc_commit(acc_full);
        }
        __syncwarp();
        if (a == 3) st++;
        if (++sb == NSB) { sb = 0; pb ^= 1; }
      }
      // (a last group of fewer than four chunks: its other places in the ring go round empty)
      n_acc++;
      for (uint32_t a = (uint32_t)nch & 3u; a != 0 && a < 4; a++) {
        tc_wait(a_ready + a, st & 1, A.err, A.wait_ns);
        if (el) tc_mbar_arrive(a_free + a);
        if (a == 3) st++;
      }
    }
  } else if (warp == MW + 1) {
    // ================= the producer: one thread =================
    if (tc_elect()) {
      const uint32_t sRaw_a = tc_s32(sRaw), sB_a = tc_s32(sB);
      const int n_items = *A.n_tiles * A.row_tiles, G = (int)gridDim.x;
      int cur = (int)blockIdx.x, nxt = cur + G;
      uint4 Tc = make_uint4(MX_END, 0, 0, 0), Tn = Tc;
      if (cur < n_items) Tc = __ldg(A.tiles + cur / A.row_tiles);
      uint32_t sr = 0, pr = 1, sb = 0, pb = 1, nr = 0, nbk_ = 0;
      bool ok = true;
      for (int k = 0; ok; k++) {
        const int s = k & (MX_IT - 1);
        if (k >= MX_IT && !tc_wait(it_empty + s, (uint32_t)((k / MX_IT - 1) & 1), A.err, A.wait_ns)) break;
        const bool end = cur >= n_items;
        const int r0 = (cur % A.row_tiles) * RPC;
        MxItem it;
        it.t = end ? make_uint4(MX_END, 0, 0, 0) : Tc;
        it.r0 = r0;
        items[s] = it;
        tc_mbar_arrive(it_full + s);
        if (end) break;
        const int fut = 2 * G + (int)atomicAdd(A.next, 1u);  // (needed an item later)
        if (nxt < n_items) Tn = __ldg(A.tiles + nxt / A.row_tiles);
        if ((int)Tc.x >= 0) {
          const int el = (int)Tc.x;
          const uint32_t bytes = ((Tc.z + 15) >> 4) * (16u * MX_KC * 2 * NPC);
          const uint8_t *rec = A.rec + (size_t)Tc.w * nch * (MX_KC * 2 * NPC);
          for (int c = 0; c < nch; c++) {
            if ((c & 3) == 0) {  // nibbles of four chunks (a box past the matrix reads zeros)
              const uint32_t r = sRaw_a + sr * S::RAWB;
              if (nr >= NSR && !tc_wait(empty_raw + sr, pr, A.err, A.wait_ns)) { ok = false; break; }
              tc_mbar_expect(full_raw + sr, (uint32_t)S::RAWB);
              if (DOWN) {
                tc_tma3(r, &A.m0, c * 32, r0, el, full_raw + sr);
                tc_tma3(r + MX_BOX, &A.m0, c * 32, r0 + MX_M, el, full_raw + sr);
              } else {
                tc_tma3(r, &A.m0, c * 32, r0, el, full_raw + sr);
                tc_tma3(r + MX_BOX, &A.m1, c * 32, r0, el, full_raw + sr);
              }
              nr++;
              if (++sr == NSR) { sr = 0; pr ^= 1; }
            }
            if (nbk_ >= NSB && !tc_wait(empty_b + sb, pb, A.err, A.wait_ns)) { ok = false; break; }
            tc_mbar_expect(full_b + sb, bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sB_a + sb * S::BST),
                         "l"(rec + (size_t)c * bytes), "r"(bytes), "r"(tc_s32(full_b + sb))
                         : "memory");
            nbk_++;
            if (++sb == NSB) { sb = 0; pb ^= 1; }
          }
        }
        cur = nxt;
        nxt = fut;
        Tc = Tn;
      }
      // the last copies have landed before the CTA gives up its shared memory
      for (uint32_t i = 1; i <= NSR && i <= nr; i++) {
        const uint32_t q = nr - i;
        tc_landed(full_raw + q % NSR, (q / NSR) & 1);
      }
      for (uint32_t i = 1; i <= NSB && i <= nbk_; i++) {
        const uint32_t q = nbk_ - i;
        tc_landed(full_b + q % NSB, (q / NSB) & 1);
      }
    }
    __syncwarp();
  } else {
    // ================= the workers =================
    // decode: thread = (row m of a 128-row half, half h); the even chunks or the odd ones (two blocks of 32 codes each)
    const int m = tid & 127, part = warp >> 2, h = part >> 1, par = part & 1;
    const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    uint32_t st = 0, sr = 0, pr = 0, n_acc = 0;
    MxItem it;
    for (int k = 0; next_item(k, it); k++) {
      const uint4 T = it.t;
      const int el = (int)T.x, nvalid = (int)T.z, npad = (nvalid + 15) & ~15, r0 = it.r0;
      float *out = A.out + (size_t)T.y * rows;
      if (el < 0) {  // an expert another rank holds: zeros (down) / nothing to do (gate/up)
        if (DOWN)
          for (int i = tid; i < nvalid * RPC; i += S::NW) {
            const int n = i / RPC, mm = i - n * RPC;
            if (r0 + mm < rows) out[(size_t)n * rows + r0 + mm] = 0.0f;
          }
        continue;
      }
      const bool up = !DOWN && h == 1;  // the up matrix is half 1
      const int drow = DOWN ? r0 + h * MX_M + m : r0 + m;
      // its scale bytes, eight blocks (four chunks) at a time
      const uint8_t *sp = (up ? A.s1 + (size_t)el * A.s1_stride : A.s0 + (size_t)el * A.s0_stride) + (size_t)min(drow, rows - 1) * nbk;
      TcBytes8 sc_n;
      sc_n.load(sp);
      for (int c4 = 0; c4 < nch; c4 += 4) {
        const unsigned long long sc = sc_n.get();
        if (c4 + 4 < nch) sc_n.load(sp + 2 * (c4 + 4));
        tc_wait(full_raw + sr, pr, A.err, A.wait_ns);
        const uint8_t *raw = sRaw + sr * S::RAWB + h * MX_BOX + m * 128;
        uint4 q[4];
#pragma unroll
        for (int j = 0; j < 4; j++)  // (TMA swizzle: 16-byte piece i of a row sits at i ^ (row & 7))
          q[j] = *(const uint4 *)(raw + (((4 * (j >> 1) + 2 * par + (j & 1)) ^ (m & 7)) << 4));
        auto stored = [&](int a) {  // the stores to operand A's chunk a are done
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(a_ready + a);
        };
        const uint32_t ew4[2] = {(uint32_t)sc >> (16 * par), (uint32_t)(sc >> 32) >> (16 * par)};
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int a = 2 * j + par;
          const bool on = c4 + a < nch;
          uint32_t w[32];
          if (on) {
            const uint32_t e0 = ew4[j] & 0xffu, e1 = (ew4[j] >> 8) & 0xffu;
            if (__any_sync(PM_FULL, max(e0 - 2u, e1 - 2u) > 126u)) {
              mx_codes_any(q[2 * j], e0, w);
              mx_codes_any(q[2 * j + 1], e1, w + 16);
            } else {
              mx_codes(q[2 * j], (e0 + 126u) * 0x00800080u, w);
              mx_codes(q[2 * j + 1], (e1 + 126u) * 0x00800080u, w + 16);
            }
          }
          if (j > 0) stored(par);  // (the wait for a chunk's stores comes after the next one's decode)
          tc_wait(a_free + a, (st & 1) ^ 1, A.err, A.wait_ns);
          if (on) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tc_st32(tlane + S::A0 + a * S::ACH + h * (MX_KC / 2), w);
          }
        }
        __syncwarp();  // (an arrival is not ordered behind loads whose registers nobody has read yet)
        if (lane == 0) tc_mbar_arrive(empty_raw + sr);
        if (++sr == NSR) { sr = 0; pr ^= 1; }
        stored(2 + par);
        st++;
      }
      // ---- epilogue: TMEM lane m, the part's token columns ----
      tc_wait(acc_full, n_acc & 1, A.err, A.wait_ns);
      n_acc++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool dead = *(volatile int *)A.err != 0;
      // (The columns are read a second time where a sum was not finite: looked for eight columns at a time, the branch cost
      // 2.5 % of a prompt.) A sum once more in f32: matrix `second`, row r, token n of the tile
      auto again = [&](bool second, int r, int n) {
        const uint32_t p = T.y + (uint32_t)n;
        return mx_sum_f32((second ? A.w1 + (size_t)el * A.w1_stride : A.w0 + (size_t)el * A.w0_stride) + r * mx_row_bytes(A.cols),
                          (second ? A.s1 + (size_t)el * A.s1_stride : A.s0 + (size_t)el * A.s0_stride) + (size_t)r * nbk,
                          A.x + (size_t)(A.src_row ? A.src_row[p] : p) * A.cols, 0, nbk);
      };
      if (DOWN) {
        const float bd = A.bias0 && drow < rows ? A.bias0[(size_t)el * rows + drow] : 0.0f;
        const bool on = !dead && drow < rows, bias = A.bias0 != nullptr;
        auto put = [&](int n, float o) {
          if (bias) o = __fadd_rn(o, bd);
          if (on && n < nvalid) out[(size_t)n * rows + drow] = o;
        };
        {
          const int hw = npad >> 1, c0 = par * hw;  // half of the columns: a multiple of 8
          float poison = 0.0f;  // a NaN once a sum is not finite
          auto columns = [&](bool repair) {
            for (int c8 = 0; c8 < hw; c8 += 8) {
              uint32_t v[8];
              tc_ld8<0>(tlane + h * 128u + (uint32_t)(c0 + c8), v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              float o[8];
#pragma unroll
              for (int u = 0; u < 8; u++) o[u] = __uint_as_float(v[u]);
              if (repair)
                mx_repair(o, [&](int u) { return on && c0 + c8 + u < nvalid; }, [&](int u) { return again(false, drow, c0 + c8 + u); });
#pragma unroll
              for (int u = 0; u < 8; u++) {
                put(c0 + c8 + u, o[u]);
                poison = __fmaf_rn(o[u], 0.0f, poison);
              }
              if (repair) __syncwarp();
            }
          };
          columns(false);
          if (__any_sync(PM_FULL, poison != 0.0f)) columns(true);
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(acc_free);
        }
      } else {
        const int hrow = r0 + m;  // the h row this thread activates
        const bool on = !dead && hrow < rows;
        const float bg = A.bias0 && hrow < rows ? A.bias0[(size_t)el * rows + hrow] : 0.0f;
        const float bu = A.bias0 && hrow < rows ? A.bias1[(size_t)el * rows + hrow] : 0.0f;
        auto put = [&](int n, float gv, float uv) {
          if (A.bias0) {
            gv = __fadd_rn(gv, bg);
            uv = __fadd_rn(uv, bu);
          }
          const float wt = A.wts ? A.wts[A.pair_src[T.y + n]] : 1.0f;
          out[(size_t)n * rows + hrow] = pm_act(A.act, A.act_limit, A.act_alpha, gv, uv, wt, A.wts != nullptr);
        };
        {  // gate sums in columns 0 .., up sums in 128 ..: a quarter of the tokens a thread
          const int qw = npad >> 2, c0 = part * qw;
          float poison = 0.0f;
          auto columns = [&](bool repair) {
            for (int c4 = 0; c4 < qw; c4 += 4) {
              uint32_t vg[4], vu[4];
              tc_ld4<0>(tlane + (uint32_t)(c0 + c4), vg);
              tc_ld4<128>(tlane + (uint32_t)(c0 + c4), vu);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              float o[8];  // gate, then up
#pragma unroll
              for (int u = 0; u < 4; u++) {
                o[u] = __uint_as_float(vg[u]);
                o[4 + u] = __uint_as_float(vu[u]);
              }
              if (repair)
                mx_repair(o, [&](int u) { return on && c0 + c4 + (u & 3) < nvalid; },
                          [&](int u) { return again(u >= 4, hrow, c0 + c4 + (u & 3)); });
#pragma unroll
              for (int u = 0; u < 4; u++) {
                if (on && c0 + c4 + u < nvalid) put(c0 + c4 + u, o[u], o[4 + u]);
                poison = __fmaf_rn(o[u], 0.0f, __fmaf_rn(o[4 + u], 0.0f, poison));
              }
              if (repair) __syncwarp();
            }
          };
          columns(false);
          if (__any_sync(PM_FULL, poison != 0.0f)) columns(true);
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(acc_free);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS) : "memory");
}

// bytes of the pieces of n_pairs rows of `cols` values in at most max_groups groups
size_t mx_rec_bytes(int n_pairs, int max_groups, int cols) {
  const size_t groups = (size_t)(max_groups < n_pairs ? max_groups : n_pairs);
  return ((size_t)n_pairs + 15 * groups + 16) * ((cols + MX_KC - 1) / MX_KC) * (MX_KC * 2 * NPC);
}
void launch_mx_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x,
                    uint8_t *rec) {
  const long units = ((long)n_rows + 15 * t.max_tiles) * ((cols + 7) / 8);
  const long gx = (units / t.max_tiles + 511) / 512;  // two units a thread
  const dim3 grid((unsigned)(gx < 1 ? 1 : gx), (unsigned)t.max_tiles);
  pm_launch(L, k_mx_rows, grid, 256, 0, t.n, t.tiles, src_row, cols, x, rec);
}

template <bool DOWN> static cudaError_t mx_start(const Launch &L, const MxArgs &A, long items) {
  using S = MxShape;
  constexpr size_t smem = (size_t)S::NSR * S::RAWB + (size_t)S::NSB * S::BST + MX_IT * sizeof(MxItem) +
                          (2 * S::NSR + 2 * S::NSB + 2 * MX_NA + 2 + 2 * MX_IT) * 8 + 16;
  static_assert(smem <= 232448, "more than an SM's shared memory");
  static SmemOptIn opt;
  const cudaError_t e = smem_optin(opt, k_tc_mx<DOWN>, smem);
  if (e != cudaSuccess) return e;
  const long ctas = L.n_sm;
  return pm_launch(L, k_tc_mx<DOWN>, dim3((unsigned)(items < ctas ? items : ctas)), S::NT, smem, A);
}

// Tensor-core form of launch_gateup / launch_down for MXFP4 weights and f32 activations given as the pieces of
// the grouping's rows. x, src_row: the rows the pieces were made of (as in launch_mx_rows).
cudaError_t launch_tc_mx(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                         const uint8_t *rec, const float *x, const uint32_t *src_row, const float *wts, float *out, int *err, unsigned long long wait_ns) {
  if (t.max_tiles == 0) return cudaSuccess;
  const WMat &W0 = down ? ly.down : ly.gate, &W1 = ly.up;
  const WMaps &M0 = down ? ly.maps->down : ly.maps->gate, &M1 = ly.maps->up;
  MxArgs A;
  A.m0 = M0.m[1];  // boxes of 128 rows
  A.m1 = M1.m[1];
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
  A.err = err;
  A.wait_ns = wait_ns;
  A.zero = 0;
  const int rpc = down ? 2 * MX_M : MX_M;
  A.row_tiles = (W0.rows + rpc - 1) / rpc;
  A.cols = W0.cols;
  A.rows = W0.rows;
  A.act = ly.desc.act;
  A.act_limit = ly.desc.act_limit;
  A.act_alpha = ly.desc.act_alpha;
  const long items = (long)A.row_tiles * t.max_tiles;
  return down ? mx_start<true>(L, A, items) : mx_start<false>(L, A, items);
}
