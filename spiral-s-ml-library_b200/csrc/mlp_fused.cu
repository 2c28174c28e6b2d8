// Persistent fused multi-layer forward for narrow policy networks (the Leduc-sized
// 32-256-256-256-3 net of the benchmark): one launch runs every layer, and hidden
// activations never leave the SM.
//
// The reference runs such a net as block_matmul -> block_map -> block_row_map device
// functions with a global-memory round trip per node (ml/layers.spi:181-252,
// generated ml/layers.py:4500-4546).  Here a CTA owns 128 batch rows at a time:
//   warp 0         : TMA producer -- the input tile, then every layer's weights in
//                    64-column K-chunks through a ring of shared-memory stages
//                    (weights come from L2: the whole net is a few hundred KB).
//   warp 1         : tcgen05.mma issuer -- layer l multiplies the activation tile in
//                    shared memory (A, K-major, 128-byte swizzle) by the weight chunk
//                    (B) into one TMEM accumulator of up to 256 fp32 columns.
//   warp 2         : training forward -- stores the delivered activation chunks (TMA).
//   warp 3         : biases to shared memory.
//   warps 4..11    : epilogue -- read the accumulator (one row per thread), add bias,
//                    ReLU, round to the 16-bit storage type and write the result back
//                    into the activation tile in exactly the swizzled K-major layout
//                    the next layer's MMAs read.
//   warps 12..15   : the last layer's row head (masked softmax / regret matching /
//                    argmax) written to global, beside the next tile's first layers.
//                    A single-layer net has no epilogue warps and two such groups.
// 16-bit arithmetic classes (SB_F16, SB_BF16), and TF32 storage for layer graphs (below); widths: input <= 512 and a
// multiple of 8 (inputs beyond 256 as far as shared memory allows: the reference's Hold'em
// policy net is 512 -> 64, game/nl_hu_holdem/model_cem.spi:71-98), hidden layers multiples of 64 up to 256, output <= 64 (<= 256 when a
// prefix mask confines the head to its first 64 columns, the shape of the reference's
// own policy nets, game/leduc/model_cem.spi:37,52-60).
//
// Layer graphs (sb_layers_forward_fused) run in TF32 storage: K-chunks of 32 values, inputs and hidden layers up to 256,
// hidden outputs stored as in the training forward.  8192 rows, 128-128-128-128 with ln_l2 and a sampling head: 29.6 us as
// three launches (each waits for the last tile of the one before, loads one tile per SM, and stores it), 14.0 as one.
//
// Optional, for the reference's graphs: ln_l2 before every ReLU (ml/layers.spi:562-568), a
// sampling head that draws from a Philox stream per row (ml/layers.spi:422-431), and the
// per-decision tail of ml/models.spi:51-76 (pick a member per row, report its action and the
// probabilities every member gave that action), done by whichever CTA finishes the last member
// of a row tile.
#include "common.cuh"
#include "row_head.cuh"

namespace {

constexpr int FM_MAX_LAYERS = 8;
// Storage of activations and weights: 16 bits, or TF32 in 32 bits (layer graphs).  A K-chunk is 128 bytes of a row.
constexpr int FM_F16 = 0, FM_BF16 = 1, FM_TF32 = 2;
__host__ __device__ constexpr int fm_chunk_cols(int cls) { return cls == FM_TF32 ? 32 : 64; }
constexpr int FM_HIDDEN_NONE = 0, FM_HIDDEN_RELU = 1, FM_HIDDEN_NORM = 2;
constexpr int FM_HEAD_BIAS = 64;                        // floats kept for the head's biases, zero beyond the outputs
// Warps of an instance: four with a job each (producer, issuer, activation stores, biases), eight for the epilogue of the
// hidden layers, and groups of four that finish head rows (a single-layer net is nothing but heads: two groups take turns).
__host__ __device__ constexpr int fm_epi_warps(int hidden) { return hidden == FM_HIDDEN_NONE ? 0 : 8; }
__host__ __device__ constexpr int fm_head_groups(int hidden) { return hidden == FM_HIDDEN_NONE ? 2 : 1; }
__host__ __device__ constexpr int fm_threads(int hidden) { return 32 * (4 + fm_epi_warps(hidden) + 4 * fm_head_groups(hidden)); }
constexpr size_t FM_SMEM_LIMIT = 225 * 1024;            // dynamic shared memory; the static part stays below 2 KB
constexpr int FM_W_STAGES = 4;                         // stages of the weight ring that decide which nets fit
constexpr int FM_W_STAGES_MAX = 8;                     // stages taken where shared memory is left
constexpr uint32_t FM_CHUNK_BYTES = 128u * 128u;       // activation chunk: 128 rows x 128 bytes
// A weight stage holds one K-chunk of a layer: (widest layer's rows) x 128 bytes, at most 256 rows.

struct FusedMaps {
  CUtensorMap x;                      // [batch, in] box {chunk, 128}
  CUtensorMap w[FM_MAX_LAYERS];       // W_l [members, out_l, in_l] box {chunk, rows_l, 1}
  CUtensorMap act[FM_MAX_LAYERS];     // training forward, layer graph: hidden activations of layer l, [batch, width_l] box {chunk, 128}
};

struct FusedParams {
  int n_layers;
  int batch;
  int width[FM_MAX_LAYERS + 1];       // width[0] = input features
  int n_pad[FM_MAX_LAYERS];           // MMA N of layer l (hidden: width; last: what the head needs, a multiple of 16)
  int k_chunks[FM_MAX_LAYERS];        // ceil(in_l / chunk)
  int k_steps[FM_MAX_LAYERS];         // MMAs of the layer, 32 bytes of K each
  uint32_t idesc[FM_MAX_LAYERS];
  uint32_t w_bytes[FM_MAX_LAYERS];    // bytes of one weight chunk of layer l
  const float* bias[FM_MAX_LAYERS];   // may be null
  int tmem_cols;
  int acc_stride;                     // TMEM columns between the two accumulators (layers alternate between them)
  int num_tiles;                      // 128-row tiles of the batch
  int num_items;                      // work items = tiles x ensemble members
  long long member_stride;            // elements between two members' parameter vectors
  long long out_stride;               // elements between two members' outputs (batch x n_out)
  uint32_t x_chunks;                  // chunks of the input tile
  uint32_t stage_bytes;               // bytes of one weight stage
  uint32_t act_offset, w_offset;      // byte offsets of the activation tile and the weight ring
  int x_shared;                       // 1: the input tile lies in the activation tile (act_offset = 0); layer graphs of wide layers
  int w_stages;                       // stages of the weight ring
  uint32_t bias_offset;               // byte offset of the biases: all layers of a member one behind the other
  uint32_t bias_bytes;                // bytes of one member's biases; two such buffers take turns when there are several members
  uint32_t bias_pos[FM_MAX_LAYERS];   // byte offset of a layer's biases in a buffer
  // head
  float* out;
  SbRowHead head;                     // n, flags, prefix, mask, seed, ...; argmax_out / sample_out are [members, batch]
  int head_width;                     // columns of a row that the head holds in registers (sb_row_head_width)
  // training forward: the hidden activations and their ReLU sign words are also written to global
  // memory for the backward pass (single net only)
  int store_acts;
  uint32_t* bits[FM_MAX_LAYERS];      // uint32 [width_l / 32, batch] per hidden layer, or null
  // decision tail (null counters = off)
  int members;
  int* tile_counters;                 // int32 [num_tiles], zero between calls
  int32_t* ensemble_id;               // [batch]
  int32_t* action;                    // [batch]
  float* prob_selected;               // [batch]
  float* prob_ensemble;               // [batch, members]
};

// The last layer: a thread takes the first W values of its row out of tensor memory (all that the head needs,
// sb_row_head_columns), adds the bias (from the warp's buffer) and hands over to the shared row head.  The accumulator
// is handed back (`bar_done`) as soon as the row is in registers.
template <int W>
__device__ __noinline__ void fused_head(const SbRowHead& h, unsigned long long legal, bool has_bias, uint32_t bias_smem,
                                        float* out, uint32_t t_row, long long row, int batch, uint32_t bar_done) {
  uint32_t raw[W];
  tmem_ld_head<W>(t_row, raw);
  tmem_ld_wait();
  tc_fence_before_sync();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar_done);
  if (row >= batch) return;
  float* v = reinterpret_cast<float*>(raw);
  if (has_bias) {
#pragma unroll
    for (int j = 0; j < W; j += 4) {
      float4 b;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                   : "r"(bias_smem + 4u * (uint32_t)j) : "memory");
      v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
    }
  }
  sb_row_head_finish<W>(h, v, (typename SbLegalWord<W>::type)legal, row, out + row * h.n);
}

// Finishes 32 columns of a row: bias, ReLU, rounding to the storage type, and the swizzled store into the activation
// tile (`dst` = the row's 128 bytes of the activation chunk, `piece0` = first of its four 16-byte pieces there, all eight
// in 32-bit storage, `key` the row's swizzle).  `word` (or null) takes the sign word of the row and chunk.
template <int CLS, bool NORM>
__device__ __forceinline__ void hidden_chunk(uint32_t* raw, float sumsq, float inv, bool has_bias, uint32_t bias_addr,
                                             uint32_t* word, uint32_t dst, uint32_t piece0, uint32_t key) {
  float* v = reinterpret_cast<float*>(raw);
  if (NORM) divide_row32(v, sumsq, inv);
  if (has_bias) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      unsigned long long b0, b1;       // the same address for the whole warp
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(b0), "=l"(b1) : "r"(bias_addr + 16u * (uint32_t)q) : "memory");
      unpack_f32x2(add_f32x2(pack_f32x2(v[4 * q], v[4 * q + 1]), b0), v[4 * q], v[4 * q + 1]);
      unpack_f32x2(add_f32x2(pack_f32x2(v[4 * q + 2], v[4 * q + 3]), b1), v[4 * q + 2], v[4 * q + 3]);
    }
  }
  if (word) *word = positive_bits32(v);
  if constexpr (CLS == FM_TF32) {
    auto one = [&](int j) { return __float_as_uint(round_tf32_rn(fmaxf(v[j], 0.f))); };
#pragma unroll
    for (int q = 0; q < 8; ++q)
      st_shared_v4(dst + (((uint32_t)q ^ key) << 4), make_uint4(one(4 * q), one(4 * q + 1), one(4 * q + 2), one(4 * q + 3)));
  } else {
    constexpr bool BF16 = CLS == FM_BF16;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 out = make_uint4(relu_pack2<BF16>(v[8 * q], v[8 * q + 1]), relu_pack2<BF16>(v[8 * q + 2], v[8 * q + 3]),
                                   relu_pack2<BF16>(v[8 * q + 4], v[8 * q + 5]), relu_pack2<BF16>(v[8 * q + 6], v[8 * q + 7]));
      st_shared_v4(dst + (((piece0 + (uint32_t)q) ^ key) << 4), out);
    }
  }
}

// One warp's share of a hidden layer: chunks `half`, half + 2, ... of 32 columns (at most four).
// Writes relu(acc + bias) in the storage type into the activation tile, in the
// 128-byte-swizzled K-major layout the next layer's A descriptors expect:
// element (row, j) -> chunk j / 64, byte row * 128 + (((j % 64) / 8) ^ (row % 8)) * 16 + (j % 8) * 2
// (32-bit storage: chunk j / 32, byte row * 128 + (((j % 32) / 4) ^ (row % 8)) * 16 + (j % 4) * 4).
// After each 32-column chunk the warp arrives on the barrier of the activation chunk it belongs to
// (`chunk_bar0` + 8 bytes per chunk): the next layer's MMAs on that K-chunk start as soon as all its
// warps (eight, four in 32-bit storage) have delivered it, while the later chunks are still being finished.
//
// A tile's time is the chain of these chunks.  Clock stamps of a tile of the Leduc net (262144 rows): 3860 clocks a hidden
// layer, of which a chunk takes 640 (85 instructions 460, proxy fence 110, the next chunk's wait 70) and the way from the
// last chunk over its MMAs to the next accumulator 920 + 210.  What kept other warps waiting before: the head, finished by
// half of these warps (2300 for the mask bytes, 2200 for the rows), and the biases, 1200 to 2000 per layer from global
// memory.  Heads and biases now have warps of their own: 262144 rows 129.1 -> 91.7 us, 16384 rows 13.3 -> 12.3, training
// forward of 65536 rows 47.8 -> 38.9, 128-256-256-17 155 -> 113; 16 members of 512-64, 4096 states 59 -> 48.
// Tried: sixteen warps of two chunks each (80 registers: 106 us); the last K-chunk by halves of the columns, so that the
// epilogue starts on the left one (101: MMAs of 128 columns read A twice).
// False when a wait expired.
template <int CLS, bool NORM>
__device__ __forceinline__ bool fused_hidden(uint32_t t_row, int n_cols, bool has_bias, uint32_t bias_smem, uint32_t act_base,
                                          int row_in_tile, int half,
                                          uint32_t chunk_bar0, uint32_t* bits_out, long long row, int batch,
                                          uint32_t bar_full, uint32_t parity, uint32_t bar_act_free, uint32_t act_parity,
                                          volatile int* abortp) {
  const int lane = (int)(threadIdx.x & 31);
  const int chunks = n_cols >> 5;
  if (!mbar_wait_warp(bar_full, parity, abortp, SB_SITE_MLP_ACC)) return false;
  tc_fence_after_sync();
  // Row normalisation (local_ln_l2, ml/primitives.spi:701-703; no bias in this mode): a first pass
  // over the whole accumulator row sums the squares; both warps of a quadrant do it for themselves.
  float sumsq = 0.f;
  uint32_t raw_a[32], raw_b[32];
  if (NORM) {
    for (int c = 0; c < chunks; ++c) {
      tmem_ld32(t_row + (uint32_t)(c * 32), raw_a);
      tmem_ld_wait32(raw_a);
#pragma unroll
      for (int j = 0; j < 32; ++j) sumsq = fmaf(__uint_as_float(raw_a[j]), __uint_as_float(raw_a[j]), sumsq);
    }
  }
  const float inv = NORM ? row_reciprocal(sumsq) : 0.f;
  tmem_ld32(t_row + (uint32_t)(half * 32), raw_a);
  // Training forward: the stores of the previous layer's activations must have read the tile before it is overwritten.
  if (bar_act_free && !mbar_wait_warp(bar_act_free, act_parity, abortp, SB_SITE_MLP_ACT)) return false;
  const uint32_t key = (uint32_t)row_in_tile & 7u;
  const uint32_t dst0 = act_base + (uint32_t)row_in_tile * 128u;
  uint32_t* word = bits_out && row < batch ? bits_out + row : nullptr;
  // Chunk c of 32 columns: the left or right half of activation chunk c / 2, all of chunk c in 32-bit storage.
  auto finish = [&](uint32_t* raw, int c) {
    const uint32_t chunk = (uint32_t)(CLS == FM_TF32 ? c : c >> 1);
    hidden_chunk<CLS, NORM>(raw, sumsq, inv, has_bias, bias_smem + 128u * (uint32_t)c,
                       word ? word + (long long)c * batch : nullptr, dst0 + chunk * FM_CHUNK_BYTES, 4u * (uint32_t)(c & 1), key);
    // generic-proxy writes of the activation tile must be visible to the MMA's async-proxy reads
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(chunk_bar0 + 8u * chunk);
  };
  // The next chunk is on its way out of tensor memory while this one is finished.
#pragma unroll 1
  for (int c = half; c < chunks; c += 4) {
    tmem_ld_wait32(raw_a);
    if (c + 2 < chunks) tmem_ld32(t_row + (uint32_t)((c + 2) * 32), raw_b);
    finish(raw_a, c);
    if (c + 2 >= chunks) break;
    tmem_ld_wait32(raw_b);
    if (c + 4 < chunks) tmem_ld32(t_row + (uint32_t)((c + 4) * 32), raw_a);
    finish(raw_b, c + 2);
  }
  return true;
}

// The per-decision tail for one state, once every member's probabilities and sampled index are in
// global memory: draw a member, report its action, the probability it gave the action and the
// probability every member gave it (ml/models.spi:51-76).
__device__ __noinline__ void decide_row(const FusedParams& p, long long row) {
  if (row >= p.batch) return;
  const int n = p.head.n;
  const unsigned long long stream = p.head.row_offset + (unsigned long long)row;
  // drawn after the members' sampling draws (outputs position .. position + members - 1 of the stream)
  const int e_id = (int)sb_philox_below(p.head.seed, stream, p.head.position + (unsigned long long)p.members,
                                        (uint32_t)p.members);
  const int a = __ldcg(p.head.sample_out + (long long)e_id * p.batch + row);
  p.ensemble_id[row] = e_id;
  p.action[row] = a;
  const float* prow = p.out + row * n + (a >= 0 ? a : 0);
  p.prob_selected[row] = a >= 0 ? __ldcg(prow + (long long)e_id * p.out_stride) : 0.f;
  float* by_member = p.prob_ensemble + row * p.members;
  // The members' probabilities lie a whole output apart: eight are on their way at a time (a load and a store in turn
  // took a memory round trip per member; 16 members, 256 states: 19.8 -> 19.1 us).
  for (int e0 = 0; e0 < p.members; e0 += 8) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = a >= 0 && e0 + j < p.members ? __ldcg(prow + (long long)(e0 + j) * p.out_stride) : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (e0 + j < p.members) by_member[e0 + j] = v[j];
  }
}

// HIDDEN: what the hidden layers are, FM_HIDDEN_NONE (a single layer), FM_HIDDEN_RELU or FM_HIDDEN_NORM (x / sum(x^2) over
// the row before every ReLU, no bias).  Instances of their own: with the divisions of
// the one and the chunk loop of the other in every kernel, registers went short where they are not used.  Leduc net,
// 262144 rows 137 -> 129 us, 16384 rows 13.9 -> 13.3; one layer of 512-64, 16 members, 512 states 23 -> 18.5.
template <int CLS, int HIDDEN>
__global__ void __launch_bounds__(fm_threads(HIDDEN), 1)
mlp_fused_kernel(const __grid_constant__ FusedMaps maps, const __grid_constant__ FusedParams p) {
  constexpr int EW = fm_epi_warps(HIDDEN), HG = fm_head_groups(HIDDEN), CHUNK = fm_chunk_cols(CLS);
  constexpr bool TF32 = CLS == FM_TF32;
  extern __shared__ uint8_t fm_smem_raw[];
  __shared__ __align__(8) uint64_t bar_x_full, bar_x_empty, bar_act_free, bar_tail_in[HG], bar_tail_out[HG];
  __shared__ __align__(8) uint64_t bar_bias_full[2], bar_bias_empty[2];
  __shared__ __align__(8) uint64_t bar_acc_full[2], bar_head_full[2], bar_head_done[2];      // per accumulator: a hidden layer's or a head's, and its rows read
  __shared__ __align__(8) uint64_t bar_chunk[8];       // chunk k of the activation tile is written (8 warps each, 4 in 32-bit storage)
  __shared__ __align__(8) uint64_t bar_w_full[FM_W_STAGES_MAX], bar_w_empty[FM_W_STAGES_MAX];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ int tile_is_complete[HG];
  __shared__ SbRowHead head_slot[4 * HG];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(fm_smem_raw) + 1023u) & ~1023u;
  const uint32_t x_base = base;                      // input tile: x_chunks x 16 KB
  const uint32_t act_base = base + p.act_offset;     // activation tile: up to 4 chunks
  const uint32_t w_base = base + p.w_offset;         // weight ring
  const uint32_t bias_base = base + p.bias_offset;

  if (tid == 0) {
    mbar_init(smem_u32(&bar_x_full), 1);
    mbar_init(smem_u32(&bar_x_empty), p.x_shared ? 2 : 1);   // the MMAs that read it last; shared: and the stores of the last hidden layer
    mbar_init(smem_u32(&bar_act_free), 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_acc_full[a]), 1);
      mbar_init(smem_u32(&bar_head_full[a]), 1);
      mbar_init(smem_u32(&bar_head_done[a]), 4);    // the four warps that finish head rows
      mbar_init(smem_u32(&bar_bias_full[a]), 1);
      mbar_init(smem_u32(&bar_bias_empty[a]), EW + 4);   // every warp that reads an item's biases
    }
    for (int k = 0; k < 8; ++k) mbar_init(smem_u32(&bar_chunk[k]), TF32 ? 4 : 8);
    for (int g = 0; g < HG; ++g) {
      mbar_init(smem_u32(&bar_tail_in[g]), 4);       // the four warps that finish head rows
      mbar_init(smem_u32(&bar_tail_out[g]), 1);
    }
    for (int s = 0; s < p.w_stages; ++s) {
      mbar_init(smem_u32(&bar_w_full[s]), 1);
      mbar_init(smem_u32(&bar_w_empty[s]), 1);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), (uint32_t)p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile int* abortp = &abort_flag;
  const int L = HIDDEN == FM_HIDDEN_NONE ? 1 : p.n_layers;
  // Set-up above touched only this CTA's shared and tensor memory; everything below reads or writes
  // global memory and therefore waits for the kernel before it on the stream.
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();

  // The producer and the issuer are whole warps that run their loops together; single instructions are predicated on
  // `one` (see umma_issue).
  const bool one = elect_one_lane();
  if (warp == 0) {
    int stage = 0;
    uint32_t w_phase = 0, x_phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x) {
      const int member = item / p.num_tiles, tile = item - member * p.num_tiles;
      if (!mbar_wait_warp(smem_u32(&bar_x_empty), x_phase ^ 1u, abortp, SB_SITE_MLP_ACT)) break;
      x_phase ^= 1u;
      if (one) mbar_arrive_expect_tx(smem_u32(&bar_x_full), p.x_chunks * FM_CHUNK_BYTES);
      for (uint32_t c = 0; c < p.x_chunks; ++c)
        tma_load_2d(x_base + c * FM_CHUNK_BYTES, &maps.x, (int)c * CHUNK, tile * 128, smem_u32(&bar_x_full), one);
      for (int l = 0; ok && l < L; ++l) {
        for (int c = 0; c < p.k_chunks[l]; ++c) {
          if (!mbar_wait_warp(smem_u32(&bar_w_empty[stage]), w_phase ^ 1u, abortp, SB_SITE_MLP_WEIGHTS)) {
            ok = false;
            break;
          }
          if (one) mbar_arrive_expect_tx(smem_u32(&bar_w_full[stage]), p.w_bytes[l]);
          tma_load_3d(w_base + (uint32_t)stage * p.stage_bytes, &maps.w[l], c * CHUNK, 0, member, smem_u32(&bar_w_full[stage]), one);
          if (++stage == p.w_stages) {
            stage = 0;
            w_phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    int stage = 0;
    uint32_t w_phase = 0, x_phase = 0, chunk_phase = 0, head_phase = 0;     // chunk_phase, head_phase: one parity bit per barrier
    uint32_t acc = 0;
    bool ok = true;
    const uint32_t hi = (uint32_t)(umma_smem_desc(0u, 16u, 1024u, 2u) >> 32);
    const uint32_t x_lo = (uint32_t)umma_smem_desc(x_base, 16u, 1024u, 2u);
    const uint32_t act_lo = (uint32_t)umma_smem_desc(act_base, 16u, 1024u, 2u);
    const uint32_t w_lo0 = (uint32_t)umma_smem_desc(w_base, 16u, 1024u, 2u);
    const uint32_t w_full0 = smem_u32(&bar_w_full[0]), w_empty0 = smem_u32(&bar_w_empty[0]), chunk0 = smem_u32(&bar_chunk[0]);
    const uint32_t w_step = p.stage_bytes >> 4;
    const int w_stages = p.w_stages;
    uint32_t w_lo = w_lo0;
    int done = 0;                               // items before this one
    for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x, ++done) {
      for (int l = 0; ok && l < L; ++l, acc ^= 1u) {
        const uint32_t idesc = p.idesc[l];
        const int chunks = p.k_chunks[l];
        int steps = p.k_steps[l];
        uint32_t a_lo = l == 0 ? x_lo : act_lo;
        if (l == 0) {
          if (!mbar_wait_warp(smem_u32(&bar_x_full), x_phase, abortp, SB_SITE_MLP_ACT)) { ok = false; break; }
          x_phase ^= 1u;
        }
        // Layers alternate between two accumulators, across items too: the epilogue of layer l-1 still reads its
        // own while this layer's first MMAs run, and the next item's first layer runs beside the head of this one.
        // The accumulator of two layers ago is free: a hidden layer's because all of its chunks were delivered
        // before the layer after it began, a head's when its four warps have said so.
        if (L > 1 ? (l == 1 && done > 0) : done > 1) {
          if (!mbar_wait_warp(smem_u32(&bar_head_done[acc]), (head_phase >> acc) & 1u, abortp, SB_SITE_MLP_ACT)) { ok = false; break; }
          head_phase ^= 1u << acc;
        }
        const uint32_t d_tmem = tmem_base + acc * (uint32_t)p.acc_stride;
        uint32_t accumulate = 0u;
        for (int c = 0; c < chunks; ++c, steps -= 4) {
          // The weights first: they have usually been there for long when the activations come, and a wait for
          // what is there already costs the issuer some 100 clocks all the same (the other order: 91.7 -> 95 us).
          if (!mbar_wait_warp(w_full0 + 8u * (uint32_t)stage, w_phase, abortp, SB_SITE_MLP_WEIGHTS)) { ok = false; break; }
          if (l > 0) {
            // K-chunk c of this layer's input = activation chunk c of the previous layer's output
            if (!mbar_wait_warp(chunk0 + 8u * (uint32_t)c, (chunk_phase >> c) & 1u, abortp, SB_SITE_MLP_ACT)) { ok = false; break; }
            chunk_phase ^= 1u << c;
          }
          tc_fence_after_sync();
          umma_issue<false, TF32>(d_tmem, a_lo, hi, w_lo, hi, idesc, accumulate, one);
          umma_issue<false, TF32>(d_tmem, a_lo + 2u, hi, w_lo + 2u, hi, idesc, 1u, one && steps > 1);   // beyond the layer's inputs both tiles are zero
          umma_issue<false, TF32>(d_tmem, a_lo + 4u, hi, w_lo + 4u, hi, idesc, 1u, one && steps > 2);
          umma_issue<false, TF32>(d_tmem, a_lo + 6u, hi, w_lo + 6u, hi, idesc, 1u, one && steps > 3);
          accumulate = 1u;
          a_lo += FM_CHUNK_BYTES >> 4;
          tc_commit(w_empty0 + 8u * (uint32_t)stage, one);
          w_lo += w_step;
          if (++stage == w_stages) {
            stage = 0;
            w_lo = w_lo0;
            w_phase ^= 1u;
          }
        }
        if (!ok) break;
        tc_commit(l < L - 1 ? smem_u32(&bar_acc_full[acc]) : smem_u32(&bar_head_full[acc]), one);
        if (l == (p.x_shared ? L - 1 : 0)) tc_commit(smem_u32(&bar_x_empty), one);     // the input tile may be refilled
      }
    }
  } else if (warp == 2) {
    // Training forward: every delivered chunk of a hidden layer's output also leaves for global memory; the tile in shared
    // memory already has the layout of a TMA box.  The epilogue overwrites the tile once the layer's stores have read it,
    // so the chunk barriers cannot move on before this warp has seen them.
    if (HIDDEN != FM_HIDDEN_NONE && p.store_acts) {
      uint32_t chunk_phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x) {
        const int tile = item % p.num_tiles;
        for (int l = 0; ok && l < L - 1; ++l) {
          for (int c = 0; c < p.k_chunks[l + 1]; ++c) {
            if (!mbar_wait_warp(smem_u32(&bar_chunk[c]), (chunk_phase >> c) & 1u, abortp, SB_SITE_MLP_ACT)) { ok = false; break; }
            chunk_phase ^= 1u << c;
            if (one) {
              tma_store_2d(&maps.act[l], act_base + (uint32_t)c * FM_CHUNK_BYTES, c * CHUNK, tile * 128);
              bulk_commit_group();
            }
          }
          if (!ok) break;
          if (one) {
            bulk_wait_group_read<0>();
            mbar_arrive(smem_u32(&bar_act_free));
            if (p.x_shared && l == L - 2) mbar_arrive(smem_u32(&bar_x_empty));
          }
        }
      }
      if (one) bulk_wait_group<0>();      // bulk groups belong to the lane that issued the stores
    }
  } else if (warp == 3) {
    // Biases: a member's go to shared memory as a whole, once for a single net, and per item (two buffers that take turns)
    // for an ensemble.  A first tile waits for them, so two layers' are on their way at a time: with one a single tile of
    // 64-128-128-3 took 6.56 us, this way 5.3 (5.1 without biases); by cp.async, all layers' at a time, as much, but 262144 rows of
    // the Leduc net 92.4 us instead of 90.4.
    if (p.bias_bytes) {
      int n = 0;
      for (int item = blockIdx.x; item < p.num_items; item += gridDim.x, ++n) {
        if (n > 0 && p.members == 1) break;
        const long long pofs = (long long)(item / p.num_tiles) * p.member_stride;
        const uint32_t buf = (uint32_t)(n & 1);
        if (n > 1 && !mbar_wait_warp(smem_u32(&bar_bias_empty[buf]), ((n >> 1) & 1) ^ 1u, abortp, SB_SITE_MLP_ACT)) break;
        for (int l0 = 0; l0 < L; l0 += 2) {
          float b[2][8];                       // layers of up to 256 columns; of a wider output the head needs the first 64
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int l = l0 + q;
            const float* src = l < L ? p.bias[l] + pofs : nullptr;
            const int live = l < L ? p.width[l + 1] : 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) b[q][i] = lane + 32 * i < live ? __ldg(src + lane + 32 * i) : 0.f;
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int l = l0 + q;
            if (l < L) {
              const uint32_t dst = bias_base + buf * p.bias_bytes + p.bias_pos[l] + 4u * (uint32_t)lane;
              const int n_pad = l < L - 1 ? p.width[l + 1] : FM_HEAD_BIAS;
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (lane + 32 * i < n_pad) asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + 128u * (uint32_t)i), "f"(b[q][i]) : "memory");
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_bias_full[buf]));
      }
    }
  } else {
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
    const bool has_bias = p.bias_bytes != 0u, rebias = has_bias && p.members > 1;
    bool ok = true;
    int n = 0;                            // items of this CTA before this one
    // The biases of the item: in place before the first read, and for an ensemble handed back after the last.
    bool bias_seen = false;
    auto bias_wait = [&]() -> uint32_t {
      const uint32_t buf = rebias ? (uint32_t)(n & 1) : 0u;
      if (has_bias && (rebias || !bias_seen)) {
        if (!mbar_wait_warp(smem_u32(&bar_bias_full[buf]), rebias ? (uint32_t)(n >> 1) & 1u : 0u, abortp, SB_SITE_MLP_ACT)) ok = false;
        bias_seen = true;
      }
      return bias_base + buf * p.bias_bytes;
    };
    auto bias_done = [&]() {
      if (rebias) {
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_bias_empty[n & 1]));
      }
    };
    if (EW > 0 && warp < 4 + EW) {
      if constexpr (EW > 0) {
        const int half = (warp - 4) >> 2;
        uint32_t layer = 0, acc_phase = 0;   // layers across items (the last bit is the accumulator), a parity bit per accumulator
        uint32_t act_phase = 1;              // the first tile finds the activation tile free
        const uint32_t act_free = p.store_acts ? smem_u32(&bar_act_free) : 0u;
        for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x, ++n) {
          const int tile = item % p.num_tiles;
          const long long grow = (long long)tile * 128 + row_in_tile;
          const uint32_t bias_smem = bias_wait();
          if (!ok) break;
          for (int l = 0; l < L - 1; ++l, ++layer) {
            const uint32_t acc = layer & 1u;
            ok = fused_hidden<CLS, HIDDEN == FM_HIDDEN_NORM>(t_row + acc * (uint32_t)p.acc_stride, p.n_pad[l], has_bias,
                     bias_smem + p.bias_pos[l], act_base, row_in_tile, half, smem_u32(&bar_chunk[0]), p.bits[l], grow,
                     p.batch, smem_u32(&bar_acc_full[acc]), (acc_phase >> acc) & 1u, act_free, act_phase, abortp);
            acc_phase ^= 1u << acc;
            act_phase ^= 1u;
            if (!ok) break;
          }
          ++layer;                        // the head's
          bias_done();
        }
      }
    } else {
      const int hw = warp - 4 - EW, hg = hw >> 2;
      // This warp's copy of the head description (in shared memory: the head code reads a field where it
      // needs it instead of holding the whole structure in registers); member-specific fields are set per item.
      SbRowHead& h = head_slot[hw];
      if (lane == 0) h = p.head;
      __syncwarp();
      uint32_t layer = (uint32_t)(L - 1), acc_phase = 0, tail_phase = 0;
      for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x, ++n, layer += (uint32_t)L) {
        if (HG == 2 && (n & 1) != hg) continue;
        const int member = item / p.num_tiles, tile = item - member * p.num_tiles;
        const long long grow = (long long)tile * 128 + row_in_tile;
        float* out_m = p.out + (long long)member * p.out_stride;
        __syncwarp();                 // every lane is done with its row of the item before: with `h`
        if (lane == 0) {
          h.argmax_out = p.head.argmax_out ? p.head.argmax_out + (long long)member * p.batch : nullptr;
          h.sample_out = p.head.sample_out ? p.head.sample_out + (long long)member * p.batch : nullptr;
          h.position = p.head.position + (unsigned long long)member;      // one draw per member from the row's stream
        }
        __syncwarp();
        // What the head needs beside the accumulator is asked for before the wait.
        unsigned long long legal = 0ull;
        if (grow < p.batch) {
          if (p.head_width <= 4) legal = sb_row_head_legal<4>(h, grow);
          else if (p.head_width <= 16) legal = sb_row_head_legal<16>(h, grow);
          else legal = sb_row_head_legal<64>(h, grow);
        }
        const uint32_t bias_smem = bias_wait() + p.bias_pos[L - 1];
        if (!ok) break;
        const uint32_t acc = layer & 1u;
        if (!mbar_wait_warp(smem_u32(&bar_head_full[acc]), (acc_phase >> acc) & 1u, abortp, SB_SITE_MLP_ACC)) break;
        acc_phase ^= 1u << acc;
        tc_fence_after_sync();
        const uint32_t head_done = smem_u32(&bar_head_done[acc]);
        const uint32_t t_acc = t_row + acc * (uint32_t)p.acc_stride;
        switch (p.head_width) {
          case 4: fused_head<4>(h, legal, has_bias, bias_smem, out_m, t_acc, grow, p.batch, head_done); break;
          case 8: fused_head<8>(h, legal, has_bias, bias_smem, out_m, t_acc, grow, p.batch, head_done); break;
          case 16: fused_head<16>(h, legal, has_bias, bias_smem, out_m, t_acc, grow, p.batch, head_done); break;
          case 32: fused_head<32>(h, legal, has_bias, bias_smem, out_m, t_acc, grow, p.batch, head_done); break;
          default: fused_head<64>(h, legal, has_bias, bias_smem, out_m, t_acc, grow, p.batch, head_done); break;
        }
        bias_done();
        if (p.tile_counters) {
          // Decision tail (ml/models.spi:51-76).  The four head warps publish their rows of this member, count
          // the member in; the CTA that counts the last member of the tile in sees every member's results.
          // The two meeting points are mbarriers with bounded waits, like every other wait of the kernel.
          __threadfence();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_tail_in[hg]));
          if ((hw & 3) == 0 && lane == 0) {
            if (mbar_wait(smem_u32(&bar_tail_in[hg]), tail_phase, abortp, SB_SITE_MLP_ACT)) {
              __threadfence();
              const int before = atomicAdd(p.tile_counters + tile, 1);
              __threadfence();
              tile_is_complete[hg] = before == p.members - 1 ? 1 : 0;
            } else {
              tile_is_complete[hg] = 0;
            }
            mbar_arrive(smem_u32(&bar_tail_out[hg]));
          }
          if (!mbar_wait_warp(smem_u32(&bar_tail_out[hg]), tail_phase, abortp, SB_SITE_MLP_ACT)) break;
          tail_phase ^= 1u;
          if (tile_is_complete[hg]) {
            __threadfence();
            decide_row(p, grow);
            if ((hw & 3) == 0 && lane == 0) p.tile_counters[tile] = 0;        // ready for the next call
          }
          // tile_is_complete is rewritten only after all four warps have arrived for the next item.
        }
      }
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abortp != 0) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) { }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

}  // namespace

// 3-D tensor map over the weights of one layer of every ensemble member: [members, rows, cols] with
// `member_stride` elements between members, box {128 bytes of columns, box_rows, 1 member}, 128-byte swizzle.
static int make_tmap_members(CUtensorMap* map, const void* base, int in_dtype, int members, long long member_stride,
                             int rows, int cols, int box_rows) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return sb_fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  CUtensorMapDataType dt = in_dtype == SB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                           : in_dtype == SB_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const cuuint64_t es = (cuuint64_t)sb_dtype_size(in_dtype);
  cuuint64_t gdim[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)members};
  cuuint64_t gstride[2] = {(cuuint64_t)cols * es, (cuuint64_t)member_stride * es};
  cuuint32_t box[3] = {(cuuint32_t)(128u / es), (cuuint32_t)box_rows, 1u};
  cuuint32_t estr[3] = {1, 1, 1};
  if (members == 1) gstride[1] = (cuuint64_t)rows * cols * es;      // unused dimension: any legal stride
  gstride[1] = (gstride[1] + 15u) / 16u * 16u;
  CUresult r = enc(map, dt, 3, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return sb_fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled (3-D) failed with CUresult %d (members=%d rows=%d cols=%d)",
                   (int)r, members, rows, cols);
  return SB_OK;
}

// Layer graphs that the fused kernel takes: two layers or more, a TF32 input of up to 256 columns in 16-byte rows, hidden
// layers of multiples of 64 up to 256, outputs as for any head.  Where the input tile, the activation tile and four weight
// stages do not fit side by side (32-bit values: from 192 columns on), the input shares the activation tile and three
// stages do: the next tile's input then waits for this one's last layer.
static bool fused_graph_separate(int x_chunks, int act_chunks, int max_n) {
  return (size_t)(x_chunks + act_chunks) * FM_CHUNK_BYTES + (size_t)FM_W_STAGES * max_n * 128u + 1024 <= FM_SMEM_LIMIT;
}
static bool fused_graph_ok(int n_layers, const int* sizes, int prefix) {
  if (n_layers < 2 || n_layers > FM_MAX_LAYERS || !sizes) return false;
  if (sizes[0] < 4 || sizes[0] > 256 || sizes[0] % 4) return false;
  for (int i = 1; i < n_layers; ++i)
    if (sizes[i] < 64 || sizes[i] > 256 || sizes[i] % 64) return false;
  const int n_out = sizes[n_layers];
  return n_out >= 1 && prefix <= n_out && (n_out <= 64 || (n_out <= 256 && prefix >= 0 && prefix <= 64));
}

// What the per-decision tail writes (all null = no tail).
struct FusedDecide {
  int* tile_counters;
  int32_t* ensemble_id;
  int32_t* action;
  float* prob_selected;
  float* prob_ensemble;
};

// Validates and launches the fused kernel.  `head`: n is set here; argmax_out / sample_out are
// [members, batch].  `who` names the entry point in error texts.  `layer_weights`: a layer graph in TF32 storage, the
// weights of every layer on their own instead of one parameter vector (the hidden activations then go to `acts_out`).
static int fused_launch(const char* who, int n_layers, const int* sizes, int batch, int members, int in_dtype,
                        const void* x, const void* w_compute, const float* params, SbRowHead head, int hidden_norm,
                        float* out, const FusedDecide* decide, void* stream, void* const* acts_out = nullptr,
                        void* const* bits_out = nullptr, const void* const* layer_weights = nullptr) {
  const bool graph = layer_weights != nullptr;
  if (members < 1 || members > 1024) return sb_fail(SB_ERR_BAD_ARG, "%s: 1..1024 ensemble members", who);
  if (n_layers < 1 || n_layers > FM_MAX_LAYERS) return sb_fail(SB_ERR_UNSUPPORTED, "%s: 1..%d layers", who, FM_MAX_LAYERS);
  if (!sizes) return sb_fail(SB_ERR_BAD_ARG, "%s: sizes is null", who);
  if (graph ? in_dtype != SB_TF32 : in_dtype != SB_F16 && in_dtype != SB_BF16)
    return sb_fail(SB_ERR_UNSUPPORTED, graph ? "%s: TF32 storage only" : "%s: 16-bit arithmetic classes only (SB_F16, SB_BF16)", who);
  if (batch < 0) return sb_fail(SB_ERR_BAD_ARG, "%s: negative batch", who);
  if (head.flags & ~(SB_EPI_MASKED_SOFTMAX | SB_EPI_REGRET_MATCHING | SB_EPI_ARGMAX | SB_EPI_SAMPLE))
    return sb_fail(SB_ERR_BAD_ARG, "%s: the head may hold softmax, regret matching, arg-max and sampling", who);
  if (graph) {
    if (!fused_graph_ok(n_layers, sizes, head.prefix))
      return sb_fail(SB_ERR_UNSUPPORTED, "%s: widths that the fused graph does not take", who);
  } else if (sizes[0] < 8 || sizes[0] > 512 || sizes[0] % 8) return sb_fail(SB_ERR_UNSUPPORTED, "%s: input width %d (8..512, multiple of 8)", who, sizes[0]);
  for (int i = 1; i < n_layers; ++i)
    if (sizes[i] < 64 || sizes[i] > 256 || sizes[i] % 64)
      return sb_fail(SB_ERR_UNSUPPORTED, "%s: hidden width %d (64..256, multiple of 64)", who, sizes[i]);
  const int n_out = sizes[n_layers];
  if (head.prefix > n_out) return sb_fail(SB_ERR_BAD_ARG, "%s: prefix %d beyond the %d output columns", who, head.prefix, n_out);
  if (n_out < 1 || !(n_out <= 64 || (n_out <= 256 && head.prefix >= 0 && head.prefix <= 64)))
    return sb_fail(SB_ERR_UNSUPPORTED, "%s: output width %d (1..64, or up to 256 under a prefix mask of at most 64 columns)", who, n_out);
  if (hidden_norm && params) return sb_fail(SB_ERR_UNSUPPORTED, "%s: row-normalised hidden layers take no bias (params must be null)", who);
  if (batch == 0) return SB_OK;
  if (!x || (!w_compute && !graph) || !out) return sb_fail(SB_ERR_BAD_ARG, "%s: null pointer", who);
  if ((head.flags & SB_EPI_ARGMAX) && !head.argmax_out) return sb_fail(SB_ERR_BAD_ARG, "%s: SB_EPI_ARGMAX without an actions buffer", who);
  if ((head.flags & SB_EPI_SAMPLE) && !head.sample_out) return sb_fail(SB_ERR_BAD_ARG, "%s: SB_EPI_SAMPLE without an indices buffer", who);
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_compute)) & 15)
    return sb_fail(SB_ERR_MISALIGNED, "%s: x and w_compute must be 16-byte aligned", who);

  long long off[2 * FM_MAX_LAYERS + 1];
  int rc = sb_mlp_param_offsets(n_layers, sizes, off);
  if (rc != SB_OK) return rc;

  FusedMaps maps;
  FusedParams p;
  memset(&p, 0, sizeof(p));
  head.n = n_out;
  const int head_cols = sb_row_head_columns(head);      // columns that the head turns into zeros are not multiplied
  p.n_layers = n_layers;
  p.batch = batch;
  p.num_tiles = (batch + 127) / 128;
  p.num_items = p.num_tiles * members;
  p.member_stride = off[2 * n_layers];
  p.out_stride = (long long)batch * n_out;
  const int es = sb_dtype_size(in_dtype), chunk = 128 / es;
  int max_n = 32;
  uint32_t max_act_chunks = 1;
  for (int l = 0; l <= n_layers; ++l) p.width[l] = sizes[l];
  for (int l = 0; l < n_layers; ++l) {
    const bool last = l == n_layers - 1;
    p.n_pad[l] = last ? (head_cols + 15) / 16 * 16 : sizes[l + 1];
    p.k_chunks[l] = (sizes[l] + chunk - 1) / chunk;
    p.k_steps[l] = (sizes[l] * es + 31) / 32;
    p.idesc[l] = sb_umma_idesc(in_dtype, 0, 0, 128, p.n_pad[l]);
    p.w_bytes[l] = (uint32_t)p.n_pad[l] * 128u;
    p.bias[l] = params ? params + off[2 * l + 1] : nullptr;
    if (p.n_pad[l] > max_n) max_n = p.n_pad[l];
    if (l > 0 && (uint32_t)p.k_chunks[l] > max_act_chunks) max_act_chunks = (uint32_t)p.k_chunks[l];
    const void* w = graph ? layer_weights[l] : reinterpret_cast<const char*>(w_compute) + off[2 * l] * 2;
    if (graph && (!w || (reinterpret_cast<uintptr_t>(w) & 15)))
      return sb_fail(SB_ERR_MISALIGNED, "%s: weights[%d] is null or not 16-byte aligned", who, l);
    rc = make_tmap_members(&maps.w[l], w, in_dtype, members, p.member_stride, sizes[l + 1], sizes[l], p.n_pad[l]);
    if (rc != SB_OK) return rc;
  }
  for (int l = n_layers; l < FM_MAX_LAYERS; ++l) maps.w[l] = maps.w[0];
  if (acts_out) {
    if (members != 1) return sb_fail(SB_ERR_UNSUPPORTED, "%s: the training forward runs one net", who);
    for (int l = 0; l + 1 < n_layers; ++l) {
      if (!acts_out[l] || (reinterpret_cast<uintptr_t>(acts_out[l]) & 15))
        return sb_fail(SB_ERR_BAD_ARG, "%s: activations[%d] is null or not 16-byte aligned", who, l);
      rc = make_tmap_2d(&maps.act[l], acts_out[l], in_dtype, batch, sizes[l + 1], 128, chunk, SWZ_128);
      if (rc != SB_OK) return rc;
      p.bits[l] = (bits_out && bits_out[l]) ? reinterpret_cast<uint32_t*>(bits_out[l]) : nullptr;
    }
    p.store_acts = 1;
  }
  for (int l = acts_out ? (n_layers > 1 ? n_layers - 1 : 0) : 0; l < FM_MAX_LAYERS; ++l) maps.act[l] = maps.w[0];
  rc = make_tmap_2d(&maps.x, x, in_dtype, batch, sizes[0], 128, chunk, SWZ_128);
  if (rc != SB_OK) return rc;
  p.x_chunks = (uint32_t)p.k_chunks[0];
  p.x_shared = graph && !fused_graph_separate((int)p.x_chunks, (int)max_act_chunks, max_n);
  p.act_offset = p.x_shared ? 0u : p.x_chunks * FM_CHUNK_BYTES;
  p.w_offset = p.x_shared && p.x_chunks > max_act_chunks ? p.x_chunks * FM_CHUNK_BYTES : p.act_offset + max_act_chunks * FM_CHUNK_BYTES;
  p.acc_stride = 32;
  while (p.acc_stride < max_n) p.acc_stride <<= 1;
  p.tmem_cols = 2 * p.acc_stride;            // two accumulators (at most 2 x 256 columns)
  p.out = out; p.head = head; p.head_width = sb_row_head_width(head);
  p.members = members;
  if (decide) {
    p.tile_counters = decide->tile_counters; p.ensemble_id = decide->ensemble_id; p.action = decide->action;
    p.prob_selected = decide->prob_selected; p.prob_ensemble = decide->prob_ensemble;
  }
  p.stage_bytes = ((uint32_t)max_n * 128u + 1023u) / 1024u * 1024u;     // stages stay 1024-byte aligned (swizzle atoms)
  // Which nets are taken depends on the widths alone, not on how few columns the head of a call needs.
  const uint32_t full_n = p.x_shared ? 0u : graph ? (uint32_t)max_n : (uint32_t)((n_out + 15) / 16 * 16 > max_n ? (n_out + 15) / 16 * 16 : max_n);
  const size_t smem_needed = (size_t)p.w_offset + (size_t)FM_W_STAGES * (full_n * 128u) + 1024;
  if (smem_needed > FM_SMEM_LIMIT)
    return sb_fail(SB_ERR_UNSUPPORTED, "%s: the input tile, the widest hidden tile and the weight ring need %zu bytes of "
                                       "shared memory (inputs wider than 256 fit with hidden layers of at most 128)", who, smem_needed);
  // The ring takes what is left beside the biases: more than the four stages of the rule above for narrow layers; three
  // where tiles and four stages fill the limit to the byte and biases come on top (65 to 128 inputs with 256-wide layers, 257 to 320
  // with 192, 449 to 512 with 128), and at least three where a graph's input shares the activation tile.
  if (params) {
    for (int l = 0; l < n_layers; ++l) {
      p.bias_pos[l] = p.bias_bytes;
      p.bias_bytes += 4u * (uint32_t)(l < n_layers - 1 ? sizes[l + 1] : FM_HEAD_BIAS);
    }
  }
  const uint32_t bias_bytes = p.bias_bytes * (members > 1 ? 2u : 1u);
  p.w_stages = (int)((FM_SMEM_LIMIT - 1024 - p.w_offset - bias_bytes) / p.stage_bytes);
  if (p.w_stages > FM_W_STAGES_MAX) p.w_stages = FM_W_STAGES_MAX;
  p.bias_offset = p.w_offset + (uint32_t)p.w_stages * p.stage_bytes;
  const size_t smem = (size_t)p.bias_offset + bias_bytes + 1024;

  static void (*const kernels[3][3])(FusedMaps, FusedParams) = {
      {mlp_fused_kernel<FM_F16, FM_HIDDEN_NONE>, mlp_fused_kernel<FM_F16, FM_HIDDEN_RELU>, mlp_fused_kernel<FM_F16, FM_HIDDEN_NORM>},
      {mlp_fused_kernel<FM_BF16, FM_HIDDEN_NONE>, mlp_fused_kernel<FM_BF16, FM_HIDDEN_RELU>, mlp_fused_kernel<FM_BF16, FM_HIDDEN_NORM>},
      {nullptr, mlp_fused_kernel<FM_TF32, FM_HIDDEN_RELU>, mlp_fused_kernel<FM_TF32, FM_HIDDEN_NORM>}};   // a graph has hidden layers
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  SB_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev].load(std::memory_order_acquire)) {
    for (int b = 0; b < 3; ++b)
      for (int k = 0; k < 3; ++k)
        if (kernels[b][k]) SB_CUDA(cudaFuncSetAttribute(kernels[b][k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FM_SMEM_LIMIT));
    attr_set[dev].store(true, std::memory_order_release);
  }
  const int sms = sb_sm_count();
  const int grid = p.num_items < sms ? p.num_items : sms;
  double flops = 0.0;
  for (int l = 0; l < n_layers; ++l) flops += 2.0 * batch * (double)sizes[l] * sizes[l + 1] * members;
  sb_prof_before((cudaStream_t)stream);
  const int hidden = n_layers == 1 ? FM_HIDDEN_NONE : hidden_norm ? FM_HIDDEN_NORM : FM_HIDDEN_RELU;
  SB_CUDA(sb_launch(kernels[in_dtype == SB_TF32 ? FM_TF32 : in_dtype == SB_BF16 ? FM_BF16 : FM_F16][hidden], dim3(grid), dim3(fm_threads(hidden)), smem, (cudaStream_t)stream, 1, maps, p));
  sb_prof_after((cudaStream_t)stream, flops);
  SB_COUNT_LAUNCH();
  SB_CUDA(cudaGetLastError());
  return SB_OK;
}

static SbRowHead fused_head_from_spec(const sb_head_spec* spec) {
  SbRowHead h;
  memset(&h, 0, sizeof(h));
  h.flags = spec->flags; h.prefix = spec->prefix < 0 ? -1 : spec->prefix; h.mask = spec->mask;
  h.argmax_out = spec->argmax_out; h.sample_out = spec->sample_out;
  h.seed = spec->seed; h.row_offset = spec->row_offset; h.position = spec->position;
  return h;
}

extern "C" int sb_mlp_forward_fused_ensemble(int n_layers, const int* sizes, int batch, int members, int in_dtype,
                                             const void* x, const void* w_compute, const float* params, int head,
                                             const uint8_t* mask, float* out, int32_t* actions, void* stream) {
  if (head & ~(SB_EPI_MASKED_SOFTMAX | SB_EPI_REGRET_MATCHING | SB_EPI_ARGMAX))
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward_fused: head may hold only row-head flags");
  SbRowHead h;
  memset(&h, 0, sizeof(h));
  h.flags = head; h.prefix = -1; h.mask = mask; h.argmax_out = actions;
  return fused_launch("sb_mlp_forward_fused", n_layers, sizes, batch, members, in_dtype, x, w_compute, params, h, 0, out,
                      nullptr, stream);
}

extern "C" int sb_mlp_forward_fused(int n_layers, const int* sizes, int batch, int in_dtype, const void* x,
                                    const void* w_compute, const float* params, int head, const uint8_t* mask,
                                    float* out, int32_t* actions, void* stream) {
  return sb_mlp_forward_fused_ensemble(n_layers, sizes, batch, 1, in_dtype, x, w_compute, params, head, mask, out,
                                       actions, stream);
}

extern "C" int sb_mlp_forward_fused_head(int n_layers, const int* sizes, int batch, int members, int in_dtype,
                                         const void* x, const void* w_compute, const float* params, int hidden_norm,
                                         const sb_head_spec* head, float* out, void* stream) {
  if (!head) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward_fused_head: head is null");
  if (head->flags & SB_EPI_BINARIZE) return sb_fail(SB_ERR_UNSUPPORTED, "sb_mlp_forward_fused_head: no sign hash in the fused kernel");
  return fused_launch("sb_mlp_forward_fused_head", n_layers, sizes, batch, members, in_dtype, x, w_compute, params,
                      fused_head_from_spec(head), hidden_norm, out, nullptr, stream);
}

extern "C" int sb_policy_decide(const sb_decide_args* a, void* stream) {
  if (!a) return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: null arguments");
  if (a->rows < 0 || a->rows > 0x7fffffffLL) return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: rows out of range");
  if (a->rows == 0) return SB_OK;
  if (!a->sizes || a->n_layers < 1) return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: no network");
  if (!a->output_probs || !a->output_indices || !a->ensemble_id || !a->action || !a->sampling_prob_selected ||
      !a->sampling_prob_ensemble || !a->tile_counters || !a->x)
    return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: every output buffer, the input workspace x and tile_counters are required");
  if (a->head_flags & ~(SB_EPI_MASKED_SOFTMAX | SB_EPI_REGRET_MATCHING))
    return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: head_flags may hold SB_EPI_MASKED_SOFTMAX and SB_EPI_REGRET_MATCHING");
  int rc;
  if (a->fields) {
    int features = a->n_dense;
    for (int j = 0; j < a->n_fields; ++j) features += a->widths ? a->widths[j] : 0;
    if (features != a->sizes[0])
      return sb_fail(SB_ERR_BAD_ARG, "sb_policy_decide: the state layout describes %d features, the net takes %d", features, a->sizes[0]);
    rc = sb_encode_states(a->fields, a->n_fields, a->widths, a->dense, a->n_dense, a->x, a->rows, a->in_dtype, stream);
    if (rc != SB_OK) return rc;
  }
  SbRowHead h;
  memset(&h, 0, sizeof(h));
  h.flags = a->head_flags | SB_EPI_SAMPLE;
  h.prefix = a->prefix < 0 ? -1 : a->prefix;
  h.mask = a->mask;
  h.sample_out = a->output_indices;
  h.seed = a->seed; h.row_offset = a->row_offset; h.position = 0;
  FusedDecide d;
  d.tile_counters = a->tile_counters; d.ensemble_id = a->ensemble_id; d.action = a->action;
  d.prob_selected = a->sampling_prob_selected; d.prob_ensemble = a->sampling_prob_ensemble;
  return fused_launch("sb_policy_decide", a->n_layers, a->sizes, (int)a->rows, a->members, a->in_dtype, a->x, a->w_compute,
                      a->params, h, a->hidden_norm, a->output_probs, &d, stream);
}

extern "C" int sb_layers_fused_supported(int n_layers, const int* sizes, int prefix) {
  return fused_graph_ok(n_layers, sizes, prefix < 0 ? -1 : prefix) ? 1 : 0;
}

extern "C" int sb_layers_forward_fused(int n_layers, const int* sizes, int rows, const float* x, const void* const* weights,
                                       int hidden_norm, void* const* hidden, const sb_head_spec* head, float* out, void* stream) {
  if (!head || !weights || !hidden) return sb_fail(SB_ERR_BAD_ARG, "sb_layers_forward_fused: null pointer");
  if (head->flags & SB_EPI_BINARIZE) return sb_fail(SB_ERR_UNSUPPORTED, "sb_layers_forward_fused: no sign hash in the fused kernel");
  return fused_launch("sb_layers_forward_fused", n_layers, sizes, rows, 1, SB_TF32, x, nullptr, nullptr, fused_head_from_spec(head),
                      hidden_norm, out, nullptr, stream, hidden, nullptr, weights);
}

// True when the fused kernel can run this net (the checks of fused_launch that depend on the shape only).
static bool fused_shape_ok(int n_layers, const int* sizes, int in_dtype) {
  if (n_layers < 1 || n_layers > FM_MAX_LAYERS || !sizes) return false;
  if (in_dtype != SB_F16 && in_dtype != SB_BF16) return false;
  if (sizes[0] < 8 || sizes[0] > 512 || sizes[0] % 8) return false;
  uint32_t max_act_chunks = 1;
  int max_n = 32;
  for (int i = 1; i < n_layers; ++i) {
    if (sizes[i] < 64 || sizes[i] > 256 || sizes[i] % 64) return false;
    if ((uint32_t)(sizes[i] / 64) > max_act_chunks) max_act_chunks = (uint32_t)(sizes[i] / 64);
    if (sizes[i] > max_n) max_n = sizes[i];
  }
  const int n_out = sizes[n_layers];
  if (n_out < 1 || n_out > 64) return false;
  if ((n_out + 15) / 16 * 16 > max_n) max_n = (n_out + 15) / 16 * 16;
  const size_t stage = ((size_t)max_n * 128 + 1023) / 1024 * 1024;
  const size_t smem = (size_t)((sizes[0] + 63) / 64 + max_act_chunks) * FM_CHUNK_BYTES + FM_W_STAGES * stage + 1024;
  return smem <= FM_SMEM_LIMIT;
}

extern "C" int sb_mlp_fused_supported(int n_layers, const int* sizes, int in_dtype) {
  return fused_shape_ok(n_layers, sizes, in_dtype) ? 1 : 0;
}

extern "C" int sb_mlp_forward_fused_train(int n_layers, const int* sizes, int batch, int in_dtype, const void* x,
                                          const void* w_compute, const float* params, void* const* activations,
                                          void* const* relu_bits, int head, const uint8_t* mask, float* out,
                                          int32_t* actions, void* stream) {
  if (head & ~(SB_EPI_MASKED_SOFTMAX | SB_EPI_REGRET_MATCHING | SB_EPI_ARGMAX))
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward_fused_train: head may hold only row-head flags");
  if (n_layers > 1 && !activations) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward_fused_train: activations is null");
  for (int l = 0; l + 1 < n_layers; ++l)
    if (relu_bits && relu_bits[l] && sizes && sizes[l + 1] % 32 != 0)
      return sb_fail(SB_ERR_UNSUPPORTED, "sb_mlp_forward_fused_train: sign words need widths that are multiples of 32");
  SbRowHead h;
  memset(&h, 0, sizeof(h));
  h.flags = head; h.prefix = -1; h.mask = mask; h.argmax_out = actions;
  static void* const no_acts[1] = {nullptr};
  return fused_launch("sb_mlp_forward_fused_train", n_layers, sizes, batch, 1, in_dtype, x, w_compute, params, h, 0, out,
                      nullptr, stream, n_layers > 1 ? activations : no_acts, relu_bits);
}
