// prefill_tc.cuh - what the two kernels of products on 256-value blocks share: the tokens' records, the launch's
// arguments, the work items (prefill_tc.cu; prefill_few.cu: tiles of at most 8 tokens).
#pragma once

#include "tcgen.cuh"

// The tokens' operand is read from records laid out for the products (k_tc_quant_rows writes them):
// record (8 rows, block b) = [16 K chunks][8 rows][16 B] int8 activations, [2 K chunks][8 rows][8 f16]
// sub-block sums for the Q4_K mins product, [8] f32 x.d, [8] i32 offset term of Q6_K, padded to a
// multiple of 128 bytes so that every 8 x 16 B core matrix sits in one 128-byte line of shared memory.
// The records of a token tile lie block by block, so that a tile's operand of a block is ONE copy
// (a copy costs its issuing warp about 70 cycles whatever its size).
#define TC_REC 2432
#define TC_REC_BM 2048
#define TC_REC_XD 2304
#define TC_REC_XS 2336
#define TC_M 128
#define TC_NMAX 128               /* tokens of the largest tile */
#define TC_RAW_Q4 (TC_M * 144)                       /* bytes of a block's weights: as stored */
#define TC_RAW_Q6 (TC_M * (128 + 64))                /* ql, qh (the scales and d come straight to the registers) */
struct TcArgs {
  CUtensorMap m0[2], m1[2];    // planes of the tile's matrices as [expert][row][bytes]: gate or down, up
  CUtensorMap ms0[2], ms1[2];  // ... of the shared expert
  const uint4 *tiles;        // see k_tc_tiles
  const int *n_tiles;        // [1]
  unsigned int *next;        // [1] zero at launch: work items handed out so far (beyond two a CTA)
  const uint8_t *rec;        // the tokens' operand as records (TC_REC)
  const uint8_t *s0, *s1, *d0, *d1;  // Q6_K: the planes of the 16 sub-scales and of the f16 scales
  const uint8_t *ss0, *ss1, *ds0, *ds1;  // ... of the shared expert
  size_t s0_stride, s1_stride, d0_stride, d1_stride;
  const float *bias0, *bias1;  // expert biases or null
  const float *wts;            // routing weights by pair source (gate/up with fold) or null
  const uint32_t *pair_src;
  float *out;                  // gate/up: h [P][ff]; down: eo [P][d]
  int *err;
  unsigned long long wait_ns;  // limit of every wait on an mbarrier
  uint32_t zero;  // 0 (see tc_mbar_arrive_used)
  uint64_t neg_zero2;          // (-0, -0): see tc_fma2
  int fault_block;             // test hook: no products are issued or signalled from this block on (-1 = off)
  int row_tiles;               // tiles of rows of the matrix (128 rows, or 64 gate + 64 up)
  int cols, rows;
  int act;
  float act_limit, act_alpha;
};

// TC_EARLY_WEIGHTS. The product kernels let their producer thread begin before griddepcontrol.wait: it reads the tile list and fills the
// weights' ring. Allowed because the launch before each of them - a k_*_rows kernel, or k_tc_mx8's gate/up before its down - lets the
// next one in only after its own wait: the plan, and all else before that launch, is complete by then, and the weights are nobody's output. (Read
// past L1: __ldcg.) The tokens' operand and every write come after the wait.
// (48 layers of 128 experts x 2048 x 768, 8 tokens 3,475 -> 3,326 us; 256 x 7168 x 2048, 1 token 72.4 -> 69.1 us; 64 x 2048 x 1024, 64 tokens
// 174.5 -> 169.9 us; prompts within 1 %.)
struct TcItem {
  uint4 t;   // the tile (k_tc_tiles); t.x = ~1: no more items
  int r0;    // first row of the item's matrix rows
  int pad[3];
};
#define TC_IT 4
#define TC_END 0xfffffffeu

// The products of a tile list of at most 8 tokens a tile (prefill_few.cu)
cudaError_t launch_tc_few(const Launch &L, const TcArgs &A, int weight_type, bool down, long items);
