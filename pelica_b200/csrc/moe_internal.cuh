// moe_internal.cuh - device-side descriptions shared by the kernels and the C ABI.
#pragma once

#include <cuda.h>  // CUtensorMap

#include "common.cuh"
#include "optin.h"

// One expert tensor family ([n_local experts][rows][cols]) in its device layout.
//  Q4_K : plane 0 = the GGUF blocks unchanged (144 B, 16-byte aligned rows)
//  Q6_K : plane 0 = ql (128 B/block), 1 = qh (64 B), 2 = scales (16 B),
//         3 = d (2 B): the block's four fields split into planes so every
//         field is aligned; 210 B/block in total, as stored (no padding)
//  MXFP4: plane 0 = E2M1 nibbles (16 B/block, rows padded to an even number of blocks: the expanding tensor
//         copies of prefill_mx8.cu take rows 32 bytes apart), 1 = E8M0 scale bytes (1 B/block)
//         (the reference splits gpt-oss tensors the same way, src/oss.rs:241-253)
//  Q8_0 : plane 0 = int8 values (32 B/block), 1 = f16 scales (2 B/block)
//  IQ4_NL: plane 0 = codebook indices (16 B/block), 1 = f16 scales (2 B/block)
//  IQ4_XS: plane 0 = codebook indices (128 B/block), 1 = the 8-byte header (f16 d, u16 high
//          scale bits, 4 bytes of low scale nibbles)
//  Q5_K : plane 0 = the GGUF blocks unchanged (176 B)
//  IQ3_S: plane 0 = qs, qh, signs, scales as stored (108 B/block), 1 = f16 d (2 B/block)
//  GLM_Q4: plane 0 = nibbles (32 B per group of 64), 1 = f32 group scales: the container's two regions
struct WMat {
  int type;
  int rows, cols;
  uint8_t *plane[4];
  size_t stride[4];  // bytes per expert in each plane
};

// TMA descriptions of a family's planes as [expert][row][bytes of the row], boxes of 64 rows (gate, up) or 128 rows
// (down) x one 256-value block (Q4_K: plane 0; Q6_K: ql, qh; MXFP4: the nibbles of
// 128 values, each 16 in a place of 16 bytes, and of 256 values x 128 rows as stored; Q8_0,
// IQ4_NL, IQ4_XS: the values, with 64 and with 128 rows). Host memory of the layer: launchers copy them into parameters.
struct WMaps {
  CUtensorMap m[2];
};
struct LayerMaps {
  WMaps gate, up, down, sgate, sup, sdown;
};

struct LayerDev {
  pm_layer_desc desc;
  int n_local, first_local;
  const float *router;       // [E][d]
  const float *logit_bias;   // [E] or null
  const float *select_bias;  // [E] or null
  WMat gate, up, down;
  const float *bias_gate, *bias_up, *bias_down;  // [n_local][ff|d] or null
  WMat sgate, sup, sdown;                        // shared expert (1 "expert")
  const float *shared_gate_inp;                  // [d] or null
  uint32_t *usage;                               // [E]
  const LayerMaps *maps;                         // host pointer
};

// pair_pos of a pair whose expert id was refused by the plan (combine reads a zero row)
#define PM_PAIR_NONE 0xffffffffu
// values of a context's device error word (0 = none; 1..99 = a bounded wait gave up)
#define PM_DEVERR_BAD_EXPERT_ID 100

// A grouping of pairs by expert (the dispatch plan, or the trivial one-group
// plan of the shared expert).
struct Groups {
  const int *n_groups;         // [1]
  const uint32_t *expert;      // [g] global expert id
  const uint32_t *offset;      // [g]
  const uint32_t *count;       // [g]
  const uint32_t *pair_token;  // [P]
  const uint32_t *pair_src;    // [P] index t*K+k of the pair (or null)
  int max_groups;
};

struct PlanDev {
  int *n_active;
  uint32_t *active, *offset, *count;  // [E]
  uint32_t *base;                     // [E] first pair of expert e
  uint32_t *cnt;                      // [E] scratch counters
  uint32_t *pair_token, *pair_pos, *pair_src;  // [P]
};

// bytes of an MXFP4 row in plane 0
__host__ __device__ inline size_t mx_row_bytes(int cols) { return ((size_t)(cols / 32) + 1) / 2 * 32; }
// bytes of one expert's tensor in plane p
static inline size_t wmat_plane_bytes(int type, int rows, int cols, int p) {
  size_t nb;
  switch (type) {
    case PM_TYPE_Q4_K:
      nb = (size_t)rows * (cols / 256);
      return p == 0 ? nb * 144 : 0;
    case PM_TYPE_Q6_K: {
      nb = (size_t)rows * (cols / 256);
      const size_t f[4] = {128, 64, 16, 2};
      return nb * f[p];
    }
    case PM_TYPE_MXFP4:
      nb = (size_t)rows * (cols / 32);
      return p == 0 ? rows * mx_row_bytes(cols) : (p == 1 ? nb : 0);
    case PM_TYPE_Q8_0:
      nb = (size_t)rows * (cols / 32);
      return p == 0 ? nb * 32 : (p == 1 ? nb * 2 : 0);
    case PM_TYPE_IQ4_NL:
      nb = (size_t)rows * (cols / 32);
      return p == 0 ? nb * 16 : (p == 1 ? nb * 2 : 0);
    case PM_TYPE_IQ4_XS:
      nb = (size_t)rows * (cols / 256);
      return p == 0 ? nb * 128 : (p == 1 ? nb * 8 : 0);
    case PM_TYPE_Q5_K:
      nb = (size_t)rows * (cols / 256);
      return p == 0 ? nb * 176 : 0;
    case PM_TYPE_IQ3_S:
      nb = (size_t)rows * (cols / 256);
      return p == 0 ? nb * 108 : (p == 1 ? nb * 2 : 0);
    case PM_TYPE_GLM_Q4:
      nb = (size_t)rows * (cols / 64);
      return p == 0 ? nb * 32 : (p == 1 ? nb * 4 : 0);
  }
  return 0;
}

// ---- launchers (kernels_basic.cu) -----------------------------------------
struct Launch {
  cudaStream_t stream;
  int64_t *count;  // kernels launched
  int n_sm = 148;  // SMs of the device
};

// Launch of a kernel that begins with pm_pdl(): it may start while the kernel before it in the stream is still
// running (a layer of a small call is six to nine kernels of a few us each; started one by one they left 1-2 us
// between any two).
template <typename... P, typename... A>
static inline cudaError_t pm_launch(const Launch &L, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = L.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (L.count) ++*L.count;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// the current device's opt-in of `kern` to at least `bytes` of dynamic shared memory (a launch within the 48 KB every kernel
// has needs none)
template <typename... P> static inline cudaError_t smem_optin(SmemOptIn &o, void (*kern)(P...), size_t bytes) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  return (cudaError_t)o.raise(
      dev, (int)bytes, [&](int b) { return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, b); });
}

// cols: of the matrix's rows (0: blocks one after another, whatever row they are of)
void launch_repack(const Launch &L, int type, int cols, const uint8_t *raw, size_t n_blocks, uint8_t *p0,
                   uint8_t *p1, uint8_t *p2, uint8_t *p3);
void launch_unpack(const Launch &L, int type, int cols, uint8_t *raw, size_t n_blocks, const uint8_t *p0,
                   const uint8_t *p1, const uint8_t *p2, const uint8_t *p3);
void launch_dequant(const Launch &L, int type, size_t n_values, const uint8_t *p0,
                    const uint8_t *p1, const uint8_t *p2, const uint8_t *p3, float *out);
// bm (optional): per block 16 f16 values, 64 * (bsum_j >> 6) for the 8 sub-blocks, then
// bsum_j & 63: the operand the tensor-core kernel multiplies the Q4_K mins with;
// xs (optional): per block the sum of its 256 values (the Q6_K offset term)
void launch_quant_q8x(const Launch &L, const float *x, size_t rows, int n, int8_t *q, float *d,
                      int32_t *bsum, uint16_t *bm = nullptr, int32_t *xs = nullptr);
void launch_quant_q8_32(const Launch &L, const float *x, size_t rows, int n, int8_t *q, float *d, bool f16_scale);
// The launches that route and plan return their status: what runs behind them takes positions and counts from their
// results, so a call stops at the first that was refused.
cudaError_t launch_router(const Launch &L, const LayerDev &ly, const float *x, int T, float *logits);
cudaError_t launch_route(const Launch &L, const LayerDev &ly, const float *logits, int T, uint32_t *ids,
                  float *w);
// err: the context's error word (an expert id outside the layer is reported there, never used)
cudaError_t launch_plan(const Launch &L, const LayerDev &ly, const uint32_t *ids, int T, PlanDev plan, int *err);
// router + top-k + plan (+ tile list) of T <= PM_SMALL_ROUTE_TOKENS tokens in one launch (ticket: a zeroed word the
// kernel leaves zeroed; slot_table: expert -> slot of an expert-parallel placement, or null)
#define PM_SMALL_ROUTE_TOKENS 8
// the token tiles of a grouping for the tensor-core products (prefill_tc.cu)
struct TcTiles {
  int *n;              // [1] tiles
  unsigned int *next;  // [2] item counters of the gate/up and the down launch (each list serves one of each)
  uint4 *tiles;        // (expert slot or ~0, first pair, pairs, first record row)
  int ntok;            // tokens of a full tile (128; 64 where the groups are small, TC_FEW_TOKENS where they are a few pairs)
  int even;            // a group's tiles have the same number of tokens (of 16) instead of ntok and a remainder
  int shared;          // the list holds the shared expert as one more group (pairs P .. P + T - 1)
  int max_tiles;
};
#define TC_FEW_TOKENS 8  // tokens of a tile of prefill_few.cu
// record rows from one tile of a group to the next, and of a group of cnt pairs in n tiles (every group starts on a multiple
// of 16; a tile of few tokens has 16 rows of its own)
__host__ __device__ inline uint32_t tc_tile_rows(int ntok, uint32_t tokens) { return ntok == TC_FEW_TOKENS ? 16u : tokens; }
__host__ __device__ inline uint32_t tc_group_rows(int ntok, uint32_t cnt, uint32_t n) {
  return ntok == TC_FEW_TOKENS ? 16u * n : (cnt + 15u) & ~15u;
}
// tokens of each of the n tiles that cnt pairs make. Even tiles for the bf16 products: a weight tile is decoded once a
// token tile at a cost that a tile of a few tokens does not hide.
__host__ __device__ inline uint32_t tc_tile_tokens(uint32_t cnt, uint32_t n, int ntok, int even) {
  return even && n > 1 ? ((cnt + n - 1) / n + 15u) & ~15u : (uint32_t)ntok;
}
bool route_plan_small_takes(const LayerDev &ly, const float *x, int T);
cudaError_t launch_route_plan_small(const Launch &L, const LayerDev &ly, const float *x, int T, float *logits, uint32_t *ids,
                                    float *w, PlanDev pl, const int32_t *slot_table, unsigned int *ticket, const TcTiles &tt, int *err,
                                    unsigned long long wait_ns);
// top-k, weights and plan of any number of tokens from their logits (seg: route_seg_words words of scratch)
size_t route_seg_words(int T, int E);
cudaError_t launch_route_plan(const Launch &L, const LayerDev &ly, const float *logits, int T, uint32_t *ids, float *w, PlanDev pl,
                              uint32_t *seg, const TcTiles &tt);
cudaError_t launch_shared_groups(const Launch &L, int *one, uint32_t *zero, uint32_t *count, uint32_t *token, int T, const TcTiles &tt);
void launch_gateup(const Launch &L, const LayerDev &ly, bool shared, Groups g, int n_pairs,
                   const float *x, const int8_t *xq, const float *xd, const int32_t *xbsum,
                   const float *w, float *h);
void launch_down(const Launch &L, const LayerDev &ly, bool shared, Groups g, int n_pairs,
                 const float *h, const int8_t *hq, const float *hd, const int32_t *hbsum,
                 float *eo);
#define PM_MX_PROMPT 32  // tokens of a call from which the MXFP4 products need not hold every bit of an activation
#define TC_SHARED 0x40000000u  // expert slot of a tile of the shared expert
// tensor-core (tcgen05 int8) form of launch_gateup / launch_down for Q4_K / Q6_K x Q8x (prefill_tc.cu):
// the token tiles of a grouping (one list serves both products), the activation rows regrouped by expert
// in the products' layout (rec: tc_rec_bytes(n_pairs, max_groups, cols) bytes), the products.
// src_row: row of the activations that holds pair p (null: row p itself)
size_t tc_tile_words(int n_pairs, int max_groups);
// n_groups: groups that can have pairs (the experts this GPU holds)
// tokens: of the call, the most a group can have; shared_tokens: of the shared expert's group in the same list (0: none)
// ntok: tokens of a full tile, 0 for launch_tc's own rule (anything else: even tiles)
TcTiles tc_tiles_of(uint32_t *buf, int n_pairs, int max_groups, int n_groups, int tokens, int shared_tokens, int ntok);  // buf: tc_tile_words words, 16-byte aligned
size_t tc_rec_bytes(int n_pairs, int max_groups, int cols);
cudaError_t launch_tc_tiles(const Launch &L, const LayerDev &ly, Groups g, const TcTiles &t);
// weight_type: of the matrix that the rows meet (it decides the records of tiles of few tokens)
void launch_tc_quant_rows(const Launch &L, int weight_type, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x,
                          uint8_t *rec);
void launch_tc_rows(const Launch &L, int weight_type, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const int8_t *xq,
                    const float *xd, const uint16_t *xbm, const int32_t *xs, uint8_t *rec);
cudaError_t launch_tc(const Launch &L, const LayerDev &ly, bool shared_only, bool down, const uint32_t *pair_src, const TcTiles &t,
                      const uint8_t *rec, const float *wts, float *out, int *err, unsigned long long wait_ns, int fault_block);
// tensor-core forms for MXFP4 weights and f32 activations: tiles of 128 tokens on bf16 pieces (prefill_mx.cu), smaller
// ones (mx_tile_tokens) on block-scaled fp8 pieces (prefill_mx8.cu). The rows are regrouped by tile and split into their
// pieces (rec: mx_rec_bytes / mx8_rec_bytes bytes); the fp8 gate/up products write the pieces of h themselves (hrec). The down
// products of the second may be cut along K into mx_splits parts: part s goes to out + s * split_stride.
size_t mx_rec_bytes(int n_pairs, int max_groups, int cols);
size_t mx8_rec_bytes(int T, int n_pairs, int max_groups, int cols);
int mx_tile_tokens(int T, int n_pairs, int n_groups, int ff);
int mx_splits(const pm_layer_desc &D, int n_pairs);
void launch_mx_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x, uint8_t *rec);
void launch_mx8_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x, uint8_t *rec);
cudaError_t launch_tc_mx(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                         const uint8_t *rec, const float *x, const uint32_t *src_row, const float *wts, float *out, int *err, unsigned long long wait_ns);
cudaError_t launch_tc_mx8(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                          const uint8_t *rec, const float *x, const uint32_t *src_row, const float *wts, float *out, uint8_t *hrec, int splits,
                          size_t split_stride, int *err, unsigned long long wait_ns);
// tensor-core (tcgen05 int8) form for Q8_0 / IQ4_NL / IQ4_XS weights and 32-value activation blocks (prefill_q32.cu)
bool q32_weights(int type);
int q32_tile_tokens();
size_t q32_rec_bytes(int n_pairs, int max_groups, int cols);
void launch_q32_rows(const Launch &L, int n_rows, const TcTiles &t, const uint32_t *src_row, int cols, const float *x, int weight_type,
                     bool f16_scale, uint8_t *rec);
cudaError_t launch_tc_q32(const Launch &L, const LayerDev &ly, bool down, const uint32_t *pair_src, const TcTiles &t,
                          const uint8_t *rec, const float *wts, float *out, int *err, unsigned long long wait_ns);
// expert parallelism (kernels_basic.cu): per-rank pair counts, the wire records of a dispatch,
// the received (expert, weight) records, the derived forms of received Q8x group sums
cudaError_t launch_ep_slots(const Launch &L, uint32_t *ids, int P, int E, const int32_t *table, uint32_t *usage);
void launch_ep_rank_counts(const Launch &L, const uint32_t *cnt, int E, int W, int32_t *out);
void launch_ep_pack(const Launch &L, int P, int row_bytes, int nd, int nbs, const void *rows, const float *xd,
                    const int32_t *xbs, const uint32_t *pair_token, const uint32_t *pair_src, const uint32_t *ids,
                    const float *w, void *srows, float *sd, int32_t *sbs, uint32_t *smeta);
void launch_ep_unmeta(const Launch &L, int R, const uint32_t *meta, int first, int n_local, uint32_t *eids, float *w,
                      int *err);
void launch_q8x_aux(const Launch &L, size_t n_blocks, const int32_t *bsum, uint16_t *bm, int32_t *xs);
// xn: null, or where the rows go normed (the next layer of a stack)
cudaError_t launch_combine(const Launch &L, const LayerDev &ly, const float *eo, const uint32_t *pair_pos,
                           const float *w, const float *shared_out, const float *shared_logit, int T,
                           float *y, bool accumulate, int parts = 1, float *xn = nullptr, float eps = 0.0f);
void launch_rmsnorm(const Launch &L, const float *x, int T, int d, float eps, float *out);
void launch_shared_gate_logit(const Launch &L, const LayerDev &ly, const float *x, int T,
                              float *out);
