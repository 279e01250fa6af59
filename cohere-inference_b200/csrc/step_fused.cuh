// One decoding step of up to 16 rows as ONE cooperative kernel: embedding, every layer, vocabulary projection and pick.
//
// What bounds it. At 1-16 rows a step has 135 MB of int8 weights to read (21 us) and hardly any arithmetic, but it is a
// chain of 8 dependent stages per layer in which every output depends on every input of the stage before. As 67 launches
// that chain cost 3.7 us per stage (boundary, start-up of the CTAs, operand staging, split-K exchange inside a cluster,
// epilogue): 0.26 ms at 1 row. Here 128 CTAs stay resident for the whole step and a stage costs one trip through L2:
//   * A CTA owns 8 output channels of every 1024-wide projection (24 of qkv, 32 of fc1) over the whole of K, so there is
//     no split-K exchange between CTAs; its 16 warps split K (64 values each, 256 for fc2) and add up through shared
//     memory in a fixed order.
//   * Results travel through self-flagging words: every exchange buffer is filled with 0xffffffff beforehand (no
//     value the kernel stores has that pattern: conversions and fp32 arithmetic give the canonical NaNs), producers
//     store words, consumers load 16-byte pieces and look again while a word still holds the fill pattern. No flag, no
//     fence, no barrier; measured alone, a round of "store 8 columns, poll all 1024" costs 1.1 us at 1 row.
//     A step uses one of two buffer sets (by the parity of a device counter) and refills the other one; the kernel
//     boundary orders the refill against the next step.
//   * The operand a warp polls IS its mma fragment (the buffers are laid out so that a warp-wide load takes whole
//     sectors): nothing is staged in shared memory. The residual stream lives in registers of the CTA that owns its
//     columns for the whole step.
//   * Weights never wait: every thread copies (cp.async) exactly the 16-byte fragment pieces it will multiply by into
//     slots of its own, one layer ahead, so a wait is its own cp.async group and no barrier.
//   * Attention: one CTA per (row, head) of up to 128, two per CTA above that; caches are asked into L2 a stage early and
//     the first keys are in registers before the query arrives. (Splitting the keys of 1-2 rows over idle CTAs made every
//     CTA poll 16 KB of partial outputs instead of 2 KB and cost more than it gave.)
// Where the time goes, from clock stamps (1 row, 16 x 64 heads, bf16 caches, 175 frames, 152 us): the 64 stages take 119 us,
// 0.4-0.8 us each from the last barrier to the first poll (sums, epilogue, publishing, the next stage's prologue), 0.15 in
// the hold below, 0.4-0.6 polling (the same few lines go to 128 SMs through L2), 0.1-0.7 multiplying or attending; the
// vocabulary projection 9.7; the rest is the launch, the embedding, the first layer's copies and the pick. So the code is kept
// short between two exchanges and in itself. 8 x 128 heads over int8 caches take 196 us: the two attention stages of a layer
// wait 2.2 us each in front of the first keys, whose scales nobody has asked into L2 (bf16 caches: 0.6). The loop over the layers runs through ONE
// copy each of the LayerNorm-folding projection, the output projection, fc2 and the attention, driven by a table in
// shared memory: with a copy per stage it was 120 KB of instructions that every layer fetched again (265 us at 1 row).
// And each copy does only what its kind needs: one general projection for all six executed 935 instructions per warp
// and stage (222 us).
// Measured (8 layers, 16 x 64 heads, int8 weights, bf16 caches, a step of the kernel sequence against this one): 251 ->
// 151 us at 1 row, 262 -> 184 at 8, 298 -> 224 at 16; bf16 weights at 8 rows 0.326 -> 0.243 ms.
// Every wait is bounded (B200DEC_ST_TIMEOUT); after one has run out the others only look once, so the kernel ends.
#pragma once
#include <type_traits>

#include "linear_kernel.cuh"

namespace b200dec_detail {

constexpr int FC = 128, FT = 512, FW = 16;  // CTAs, threads, warps
constexpr int F_MAX_ROWS = 16, F_MAX_LAYERS = 16;
constexpr uint32_t F_EMPTY = 0xffffffffu;

enum { FM_INT8 = 0, FM_INT8_24 = 1, FM_F16 = 2, FM_BF16 = 3 };

struct FProj {
  const uint8_t* w;
  const uint32_t* meta;
  const float* scale;
  const float* bias;
  const float* ln_g;
  const float* ln_bias;
};
struct FLayer {
  FProj qkv, o, cq, co, fc1, fc2;
  const float* gamma[3];
  float eps[3];
  int pad;
  void *sk, *sv, *ck, *cv;
  float *sks, *svs, *cks, *cvs;
};
struct FArgs {
  int layers, rows, heads, act, slots, seq, frames, vocab, max_prompt, out_cols, eos, max_pos, head_umma;
  uint32_t wait_limit;
  int withhold;
  const __nv_bfloat16* embed;
  const __nv_bfloat16* ptab;
  b200dec_norm ln0;
  FProj head;
  const float* gamma_f;
  float eps_f, scale_log2;
  const int* active;
  int64_t* tok;
  int* pos;
  const int* plen;
  const int* limit;
  const int* cross_len;
  uint8_t* finished;
  const int64_t* forced;
  int64_t* out;
  uint8_t* flags_host;
  int* status;
  float* logits;
  int64_t* argmax;
  uint32_t* ws;  // counter (16 words), then two sets of exchange buffers
  size_t set_words;
  FLayer layer[F_MAX_LAYERS];
};

// Words of one layer's exchange buffers (and the order they lie in) for a number of rows. wide: the attention
// output, the feed-forward intermediate and the residual rows travel as fp32 (bf16 weights); else the first two as fp16
// pairs and the rows as the next LayerNorm's operand, fp16(row * gamma), with every CTA's share of the rows' sums.
struct FLayout {
  int x, qkv, cq, att, mid, layer;
  __host__ __device__ FLayout(int rows, bool wide) {
    x = rows * (wide ? 1024 : 512 + 2 * FC), qkv = rows * 3072, cq = rows * 1024;
    att = wide ? rows * 1024 : rows * 512;
    mid = wide ? rows * 4096 : rows * 2048;
    layer = 3 * x + qkv + cq + 2 * att + mid;
  }
  // offsets inside a layer; the rows that fc2 leaves come last, so that the next layer finds them right before its own
  // buffers, and the first layer the embedding's
  __host__ __device__ int o_x_o() const { return 0; }
  __host__ __device__ int o_x_co() const { return x; }
  __host__ __device__ int o_qkv() const { return 2 * x; }
  __host__ __device__ int o_cq() const { return 2 * x + qkv; }
  __host__ __device__ int o_att_s() const { return 2 * x + qkv + cq; }
  __host__ __device__ int o_att_c() const { return o_att_s() + att; }
  __host__ __device__ int o_mid() const { return o_att_c() + att; }
  __host__ __device__ int o_x_f() const { return o_mid() + mid; }
};
// One set: the embedding's rows, the layers, the vocabulary projection's (max, index) per row and CTA.
__host__ __device__ inline size_t fused_set_words(int layers, int rows, bool wide) {
  const FLayout l(rows, wide);
  return (size_t)l.x + (size_t)layers * l.layer + (size_t)rows * FC * 2;
}

// Ring slots (8 KB: 16 bytes per thread) of a layer's six projections. A tile is 8 channels; a warp's share of K = 1024
// is one 64-block, of K = 4096 four. int8: one slot per tile and 64-block; 16-bit weights: two; 2:4 (feed-forward): one
// slot (and one selector word) per tile and 128-block, which two warps share at K = 1024. 16-bit weights keep a quarter
// of fc2 in the ring; the rest is asked into L2 a stage early and loaded when its stage begins.
template <int MODE, bool R16>
struct FTraits {
  static constexpr bool BF = MODE == FM_BF16, W16 = MODE == FM_F16 || BF, S24 = MODE == FM_INT8_24;
  static constexpr int CH = W16 ? 2 : 1;  // slots of a tile's 64-block
  static constexpr int S_QKV = 0, S_O = 3 * CH, S_CQ = 4 * CH, S_CO = 5 * CH, S_FC1 = 6 * CH, S_FC2 = S_FC1 + 4 * CH;
  static constexpr int N_FC2 = S24 || W16 ? 2 : 4;
  static constexpr int SLOTS = S_FC2 + N_FC2, SLOT_BYTES = FT * 16;
  static constexpr int HT = SLOTS / CH / 4 * 4;  // tiles of the vocabulary projection that wait in the ring
  static constexpr int NTP = R16 && W16 ? 2 : 4;                      // tiles multiplied per pass: what `red` holds
  static constexpr int RM = R16 ? 16 : 8;
  static constexpr int RED_BYTES = FW * NTP * RM * 8 * 4;             // [warp][tile][row][8]
  static constexpr int OFF_SEL = SLOTS * SLOT_BYTES, SEL_BYTES = S24 ? 6 * FT * 4 : 0;
  static constexpr int OFF_RED = OFF_SEL + SEL_BYTES, OFF_STAT = OFF_RED + 2 * RED_BYTES,
                       OFF_TAB = OFF_STAT + (BF ? FW * RM * 8 : 0), OFF_CACHES = OFF_TAB + (F_MAX_LAYERS * 6 + 1) * 64,
                       BYTES = OFF_CACHES + F_MAX_LAYERS * 64;
  static_assert(BYTES + 1024 <= 227 * 1024, "fits an SM");
  static_assert(RED_BYTES >= (FW * (128 + 4) + 2 * FW) * 4, "the attention merge fits");
};

// One projection of one layer, as the table in shared memory holds it: the weights and the gamma of the LayerNorm that
// reads the rows it updates (or, bf16 weights, of the LayerNorm folded into it).
struct FStage {
  FProj w;
  const float* gamma;
  float eps;
  int pad;
};
static_assert(sizeof(FStage) == 64, "");

DEVI uint4 ld_poll16(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
DEVI uint32_t ld_poll4(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
DEVI void st_word(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
DEVI bool has_empty(const uint4& v) { return max(max(v.x, v.y), max(v.z, v.w)) == F_EMPTY; }
DEVI float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
DEVI void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr_u32(smem)), "l"(gmem) : "memory");
}

// Position of value k inside its 64-block in an exchange buffer, so that piece i (16 bytes) of the four lanes t of a row
// lies together. A lane's 16 values of a block are k = 16 t + .. with int8 weights (mapping 0), 32 j + 8 t + .. with
// 16-bit and 2:4 weights (mapping 1): see the tiled layouts in linear.cu.
DEVI int perm32(int k, bool map) {  // fp32 words
  const int b = k & 63, i = map ? 2 * (b >> 5) + ((b >> 2) & 1) : (b >> 2) & 3, t = map ? (b >> 3) & 3 : b >> 4;
  return (k & ~63) + i * 16 + t * 4 + (b & 3);
}
DEVI int perm16(int k, bool map) {  // fp16 pairs: word index of the pair that k (even) starts
  const int b = k & 63, j = map ? b >> 5 : (b >> 3) & 1, t = map ? (b >> 3) & 3 : b >> 4;
  return ((k & ~63) >> 1) + j * 16 + t * 4 + ((b & 7) >> 1);
}

struct FWait {
  uint32_t limit;
  int* status;
};
// v[i] = the piece at addr(i): all requested at once; those that still hold the fill pattern are requested again together
// (one trip per round, not one per piece)
template <int N, class Addr>
DEVI void poll(uint4 (&v)[N], FWait& w, Addr addr) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = ld_poll16(addr(i));
#pragma unroll 1
  for (uint32_t n = 0;; ++n) {
    bool again = false;
#pragma unroll
    for (int i = 0; i < N; ++i) again |= has_empty(v[i]);
    if (!again) break;
    if (n >= w.limit) {
      atomicOr(w.status, B200DEC_ST_TIMEOUT);
      w.limit = 0;  // from here on every wait looks once
      break;
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (has_empty(v[i])) v[i] = ld_poll16(addr(i));
  }
}

// the operand of one warp: 16 rows x 64 k as the A fragments of four k-steps (and the low halves for bf16 weights)
template <bool BF>
struct FOperand {
  uint32_t hi[4][4];
  uint32_t lo[BF ? 4 : 1][4];
};


template <int MODE, int D, bool Q8, bool R16>
struct FusedStep {
  using T = FTraits<MODE, R16>;
  static constexpr bool BF = T::BF, W16 = T::W16, S24 = T::S24;
  static constexpr int CH = T::CH, NTP = T::NTP, RM = T::RM, HALVES = R16 ? 2 : 1;
  static constexpr bool MAP_A = W16, MAP_F = W16 || S24;  // k mapping of the attention / feed-forward projections
  static constexpr int PC = BF ? 4 : 2, PW = BF ? 64 : 32;  // 16-byte pieces and words of a row's 64 values
  using Op = FOperand<BF>;

  const FArgs& p;
  unsigned char* ring;     // [slot][thread][16 bytes], at this thread's own
  uint32_t* sel;           // 2:4: [piece][thread], at this thread's own
  float* red;              // two buffers: [warp][tile][row][8], or the attention merge
  float2* stat;            // bf16 weights: [warp][row] sums
  const uint32_t* lut;
  const FStage* tab;
  char* const* caches;     // per layer: self keys, values, cross keys, values, then their scales
  const int tid, warp, lane, g, t, cta, R;
  int row0, row1;          // the operand rows of this lane: g and g + 8, or row 0 again where there is no such row (what
                           // the multiply makes of those is not looked at)
  FWait wait;
  int par = 0;             // which half of `red` the next stage uses
  float resid = 0.f;       // residual stream: row `warp`, channel 8 cta + (lane & 7)
  float best = -INFINITY;  // vocabulary: row `warp`'s best logit over this lane's channels so far
  int arg = 0x7fffffff;

  DEVI FusedStep(const FArgs& a, unsigned char* smem, const uint32_t* l)
      : p(a), ring(smem + threadIdx.x * 16), sel(reinterpret_cast<uint32_t*>(smem + T::OFF_SEL) + threadIdx.x),
        red(reinterpret_cast<float*>(smem + T::OFF_RED)), stat(reinterpret_cast<float2*>(smem + T::OFF_STAT)), lut(l),
        tab(reinterpret_cast<const FStage*>(smem + T::OFF_TAB)), caches(reinterpret_cast<char* const*>(smem + T::OFF_CACHES)), tid(threadIdx.x), warp(threadIdx.x >> 5),
        lane(threadIdx.x & 31), g(lane >> 2), t(lane & 3), cta(blockIdx.x), R(a.rows), wait{a.wait_limit, a.status} {
    row0 = g < R ? g : 0, row1 = g + 8 < R ? g + 8 : 0;
  }
  // Nothing another CTA publishes can be here before it has had the time of a trip through L2 since this CTA's own last
  // result, and looking earlier costs the others: polls of lines that every CTA reads queue up in front of the stores to
  // them. A trip through L2 is what it is on this chip at its full clock: us a step with a hold of 0 / 700 / 1400 / 2100
  // cycles, 16 x 64 heads and bf16 caches, 1 row 194 / 163 / 152 / 168, 8 rows 258 / 218 / 186 / 188, 16 rows 236 / 238 / 240 /
  // 239 (there the polls are slower than the hold); 8 x 128 heads over int8 caches 240 / 207 / 196 / 211, 290 / 251 / 215 / 225,
  // 250 / 250 / 252 / 249.
  // IDLE: more where the CTA has had no (row, head) to attend. 0, 1500 and 3000 cycles are the same within 0.3 us except at
  // 16 rows over int8 caches (252.7, 251.6, 252.0).
  static constexpr uint32_t HOP = 1400, IDLE = 1500;  // cycles
  uint32_t since = 0;      // clock at the last barrier
  DEVI static uint32_t now() {
    uint32_t c;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
    return c;
  }
  DEVI void hold(uint32_t cycles) const {
    while (now() - since < cycles) {}
  }
  DEVI void barrier() {
    __syncthreads();
    since = now();
  }
  DEVI float* red_buf() { return red + par * (T::RED_BYTES / 4); }

  // ---- weights: this thread's own pieces, global -> its ring slots. Byte offsets inside one matrix fit 32 bits --------
  DEVI void fill_slot(int slot, const uint8_t* src) { cp_async16(ring + slot * T::SLOT_BYTES, src); }
  DEVI uint32_t at_k1024(int tile) const {  // 64-block `warp` of a K = 1024 projection
    return W16 ? ((tile >> 1) * 32 + 2 * warp) * 1024 + (tile & 1) * 512 + lane * 16
               : ((tile >> 1) * 16 + warp) * 1024 + (tile & 1) * 512 + lane * 16;
  }
  DEVI void fill_k1024(const uint8_t* w, int slot, int tile0, int n) {
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const uint8_t* s = w + at_k1024(tile0 + i);
#pragma unroll
      for (int j = 0; j < CH; ++j) fill_slot(slot + i * CH + j, s + j * 1024);
    }
  }
  DEVI uint32_t at_fc2() const {  // 64-block 4 warp of tile `cta` (16-bit weights: piece 8 warp); the next ones follow
    return W16 ? ((cta >> 1) * 128 + 8 * warp) * 1024 + (cta & 1) * 512 + lane * 16
               : ((cta >> 1) * 64 + 4 * warp) * 1024 + (cta & 1) * 512 + lane * 16;
  }
  DEVI void fill_fc1(const FProj& w) {
    if constexpr (S24) {
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const uint32_t b = (2 * cta + (i >> 1)) * 8 + (warp >> 1);
        fill_slot(T::S_FC1 + i, w.w + b * 1024 + (i & 1) * 512 + lane * 16);
        cp_async4(sel + i * FT, w.meta + b * 64 + (i & 1) * 32 + lane);
      }
    } else {
      fill_k1024(w.w, T::S_FC1, 4 * cta, 4);
    }
  }
  DEVI void fill_fc2(const FProj& w) {
    if constexpr (S24) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t b = (cta >> 1) * 32 + 2 * warp + i;
        fill_slot(T::S_FC2 + i, w.w + b * 1024 + (cta & 1) * 512 + lane * 16);
        cp_async4(sel + (4 + i) * FT, w.meta + b * 64 + (cta & 1) * 32 + lane);
      }
    } else {
      const uint8_t* s = w.w + at_fc2();
#pragma unroll
      for (int i = 0; i < T::N_FC2; ++i) fill_slot(T::S_FC2 + i, s + i * 1024);
    }
  }
  // tile i of this CTA's share of the vocabulary waits in slots (i % HT) * CH ..
  DEVI void fill_head(int i0, int n, int tiles, int per) {
#pragma unroll 1
    for (int i = i0; i < i0 + n; ++i) {
      const int tile = cta * per + i, slot = (i % T::HT) * CH;
      if (i >= per || tile >= tiles) return;
      if (!p.head_umma) {
        fill_k1024(p.head.w, slot, tile, 1);
      } else {  // the block layouts of the tcgen05 kernels
        const int ch = (tile & 15) * 8 + g;
        const uint32_t blk = (tile >> 4) * 16 + warp;
        if constexpr (W16) {
          fill_slot(slot, p.head.w + blk * 16384 + ch * 128 + ((t ^ (ch & 7)) << 4));
          fill_slot(slot + 1, p.head.w + blk * 16384 + ch * 128 + (((4 + t) ^ (ch & 7)) << 4));
        } else {
          fill_slot(slot, p.head.w + blk * 8192 + t * 2048 + ch * 16);
        }
      }
    }
  }

  // ---- multiply ------------------------------------------------------------------------------------------------------
  DEVI uint4 slot16(int slot) const { return *reinterpret_cast<const uint4*>(ring + slot * T::SLOT_BYTES); }
  DEVI void mma_step(float (&acc)[4], const Op& a, int s, uint32_t b0, uint32_t b1) {
    if constexpr (BF) {
      mma_bf16(acc, a.hi[s], b0, b1);
      mma_bf16(acc, a.lo[s], b0, b1);
    } else {
      mma_f16(acc, a.hi[s], b0, b1);
    }
  }
  DEVI void mma_int8(float (&acc)[4], const Op& a, const uint4& b) {
    const uint32_t r[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      uint32_t b0, b1;
      widen_u8(r[s], b0, b1);
      mma_step(acc, a, s, b0, b1);
    }
  }
  DEVI void mma_w16(float (&acc)[4], const Op& a, int j, const uint4& b) {  // piece j: k-steps 2 j, 2 j + 1
    mma_step(acc, a, 2 * j, b.x, b.y);
    mma_step(acc, a, 2 * j + 1, b.z, b.w);
  }
  DEVI void mma_24(float (&acc)[4], const Op& a, uint32_t q0, uint32_t q1, uint32_t m) {  // 64 k: 8 kept bytes, 4 selectors
    const uint32_t r[2] = {q0 ^ 0x80808080u, q1 ^ 0x80808080u};
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t c = lut[((m >> (4 * s)) & 15u) | ((s & 1) << 4)];
      uint32_t b0, b1;
      widen_u8(__byte_perm(r[s >> 1], 0x80808080u, c), b0, b1);
      mma_step(acc, a, s, b0, b1);
    }
  }
  struct Tile {  // one tile's 64 k of weights
    uint4 w[CH];
  };
  DEVI Tile tile_at(int slot) const {
    Tile b;
#pragma unroll
    for (int j = 0; j < CH; ++j) b.w[j] = slot16(slot + j);
    return b;
  }
  DEVI void mma_tile(float (&acc)[4], const Op& a, const Tile& b) {
    if constexpr (W16) {
      mma_w16(acc, a, 0, b.w[0]);
      mma_w16(acc, a, 1, b.w[1]);
    } else {
      mma_int8(acc, a, b.w[0]);
    }
  }

  // ---- operands ------------------------------------------------------------------------------------------------------
  // one 64-block's pieces (PC per half) as fragments
  DEVI void operand(const uint4* v, Op& a) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h < HALVES) {
        const uint4* u = v + h * PC;
        if constexpr (BF) {
#pragma unroll
          for (int i = 0; i < 4; ++i) put(a, h, i, u[i]);
        } else {
          a.hi[0][h] = u[0].x, a.hi[0][2 + h] = u[0].y, a.hi[1][h] = u[0].z, a.hi[1][2 + h] = u[0].w;
          a.hi[2][h] = u[1].x, a.hi[2][2 + h] = u[1].y, a.hi[3][h] = u[1].z, a.hi[3][2 + h] = u[1].w;
        }
      } else {
        clear_half1(a);
      }
    }
  }
  DEVI void clear_half1(Op& a) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a.hi[i][1] = a.hi[i][3] = 0;
      if constexpr (BF) a.lo[i][1] = a.lo[i][3] = 0;
    }
  }
  DEVI void put(Op& a, int h, int s, const uint4& f) {  // four fp32 values of k-step s, rows of half h
    uint2 hi, lo;
    to_operand<BF, BF>(make_float4(__uint_as_float(f.x), __uint_as_float(f.y), __uint_as_float(f.z), __uint_as_float(f.w)), hi, lo);
    a.hi[s][h] = hi.x, a.hi[s][2 + h] = hi.y;
    if constexpr (BF) a.lo[s][h] = lo.x, a.lo[s][2 + h] = lo.y;
  }
  // The rows a LayerNorm reads, as the ready operand with the sums of row `warp` (s1, s2: this lane's part) ...
  DEVI void ln_linked(const uint32_t* x, Op& a, float& s1, float& s2) {
    uint4 v[HALVES * 2 + 2];
    const uint32_t* r0 = x + row0 * 512 + warp * 32 + t * 4;
    const uint32_t* r1 = x + row1 * 512 + warp * 32 + t * 4;
    const uint32_t* st = warp < R ? x + R * 512 + (warp * FC + lane * 4) * 2 : r0;  // no such row: anything
    const int st1 = warp < R ? 4 : 0;
    hold(HOP);
    poll(v, wait, [&](int i) {
      return i >= HALVES * 2 ? st + (i - HALVES * 2) * st1 : i < 2 ? r0 + i * 16 : r1 + (i - 2) * 16;
    });
    operand(v, a);
    const uint4 b = v[HALVES * 2], c = v[HALVES * 2 + 1];
    s1 = (__uint_as_float(b.x) + __uint_as_float(b.z)) + (__uint_as_float(c.x) + __uint_as_float(c.z));
    s2 = (__uint_as_float(b.y) + __uint_as_float(b.w)) + (__uint_as_float(c.y) + __uint_as_float(c.w));
  }
  // ... or (bf16 weights) from the fp32 rows: (x - shift) * gamma, the rows' sums over this warp's 64 k into `stat`
  DEVI void ln_rows(const uint32_t* x, const float* gamma, Op& a) {
    float4 gm[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) gm[i] = __ldg(reinterpret_cast<const float4*>(gamma + warp * 64 + 32 * (i >> 1) + 8 * t + 4 * (i & 1)));
    uint4 v[HALVES * 5];  // per half: four pieces of 4 values, and the row's first four for its shift
    hold(HOP);
    poll(v, wait, [&](int i) { return x + (i < 5 ? row0 : row1) * 1024 + (i % 5 == 4 ? 0 : warp * 64 + t * 4 + (i % 5) * 16); });
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      const uint4 f = v[5 * h + 4];
      const float c = 0.25f * ((__uint_as_float(f.x) + __uint_as_float(f.y)) + (__uint_as_float(f.z) + __uint_as_float(f.w)));
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 u = v[5 * h + i];
        const float x0 = __uint_as_float(u.x) - c, x1 = __uint_as_float(u.y) - c, x2 = __uint_as_float(u.z) - c,
                    x3 = __uint_as_float(u.w) - c;
        s1 += (x0 + x1) + (x2 + x3);
        s2 += (x0 * x0 + x1 * x1) + (x2 * x2 + x3 * x3);
        put(a, h, i, make_uint4(__float_as_uint(x0 * gm[i].x), __float_as_uint(x1 * gm[i].y), __float_as_uint(x2 * gm[i].z),
                                __float_as_uint(x3 * gm[i].w)));
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (t == 0) stat[warp * RM + g + 8 * h] = make_float2(s1, s2);
    }
    if constexpr (!R16) clear_half1(a);
  }
  // ---- results -----------------------------------------------------------------------------------------------------------
  DEVI void store_partial(int tile, const float (&acc)[4]) {  // this warp's sums of a tile
    float* o = red_buf() + ((warp * NTP + tile) * RM + g) * 8 + 2 * t;
    *reinterpret_cast<float2*>(o) = make_float2(acc[0], acc[1]);
    if constexpr (R16) *reinterpret_cast<float2*>(o + 64) = make_float2(acc[2], acc[3]);
  }
  // warp r finishes row r. Several tiles: lane = 8 tile + channel ...
  DEVI float sum_tiles() {
    const float* b = red_buf() + ((lane >> 3) * RM + warp) * 8 + (lane & 7);
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < FW; ++w) s[w & 3] += b[w * NTP * RM * 8];
    return (s[0] + s[1]) + (s[2] + s[3]);
  }
  // ... one tile: four lanes share a channel's sum, every lane gets channel lane & 7
  DEVI float sum_one() {
    const float* b = red_buf() + (4 * (lane >> 3) * NTP * RM + warp) * 8 + (lane & 7);
    float s = (b[0] + b[NTP * RM * 8]) + (b[2 * NTP * RM * 8] + b[3 * NTP * RM * 8]);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    return s;
  }
  // row `warp`, channel 8 cta + (lane & 7) of the residual stream to the LayerNorm that reads it next (gn: its gamma)
  DEVI void publish_x(uint32_t* x, float gn, bool map) {
    if constexpr (BF) {
      if (lane < 8) st_word(x + warp * 1024 + perm32(8 * cta + lane, map), __float_as_uint(resid));
    } else {
      const float v = resid * gn, o = __shfl_xor_sync(0xffffffffu, v, 1);
      float s1 = resid, s2 = resid * resid;
#pragma unroll
      for (int k = 1; k < 8; k <<= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, k);
        s2 += __shfl_xor_sync(0xffffffffu, s2, k);
      }
      if (lane < 8 && !(lane & 1)) st_word(x + warp * 512 + perm16(8 * cta + lane, map), pack_f16(v, o));
      if (lane < 2) st_word(x + R * 512 + (warp * FC + cta) * 2 + lane, __float_as_uint(lane ? s2 : s1));
    }
  }
  DEVI void first_max(float& b, int& a) const {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, b, o);
      const int oa = __shfl_xor_sync(0xffffffffu, a, o);
      if (ob > b || (ob == b && oa < a)) b = ob, a = oa;
    }
  }

  // ---- a LayerNorm-folding projection: nt tiles from tile0 ------------------------------------------------------------------
  // what: 0 qkv / 1 cross-q: fp32 rows of `pitch` to out; 2 fc1: activation, 16-bit rows to out; 3 vocabulary
  DEVI void ln_projection(int what, const FStage& st, const uint32_t* x, uint32_t* out, int pitch, int tile0, int nt, int slot) {
    constexpr int PASSES = 4 / NTP;
    float scale[PASSES], bias[PASSES], lg[PASSES], lb[PASSES];
#pragma unroll
    for (int ps = 0; ps < PASSES; ++ps) {  // the channel's epilogue values, requested before anything waits
      const int c = ps * NTP * 8 + lane, ch = tile0 * 8 + c;
      scale[ps] = 1.f, bias[ps] = lg[ps] = lb[ps] = 0.f;
      if (warp < R && lane < NTP * 8 && c < nt * 8) {
        if (!W16) scale[ps] = __ldg(st.w.scale + ch);
        if (st.w.bias) bias[ps] = __ldg(st.w.bias + ch);
        lg[ps] = __ldg(st.w.ln_g + ch), lb[ps] = __ldg(st.w.ln_bias + ch);
      }
    }
    Op a;
    float s1 = 0.f, s2 = 0.f;
    if constexpr (BF) ln_rows(x, st.gamma, a);
    else ln_linked(x, a, s1, s2);
    if (what == 3) cp_async_wait_group<0>();
    else cp_async_wait_group<5>();
#pragma unroll 1
    for (int ps = 0; ps * NTP < nt; ++ps) {
      if (nt == 1) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_tile(acc, a, tile_at(slot));
        store_partial(0, acc);
      } else if (S24 && what == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
          const uint4 q = slot16(slot + i);
          const uint32_t m = sel[i * FT];
          if (warp & 1) mma_24(acc, a, q.z, q.w, m >> 16);
          else mma_24(acc, a, q.x, q.y, m);
          store_partial(i, acc);
        }
      } else {  // NTP tiles side by side; a tile past nt is some other weights' product, and not looked at
        Tile b[NTP];
#pragma unroll
        for (int i = 0; i < NTP; ++i) b[i] = tile_at(slot + (ps * NTP + i) * CH);
        float acc[NTP][4];
#pragma unroll
        for (int i = 0; i < NTP; ++i) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
          mma_tile(acc[i], a, b[i]);
        }
#pragma unroll
        for (int i = 0; i < NTP; ++i) store_partial(i, acc[i]);
      }
      if constexpr (!BF) {
        if (ps == 0 && warp < R) s1 = warp_sum(s1), s2 = warp_sum(s2);
      }
      barrier();
      if (warp < R) {
        if constexpr (BF) {
          const float2 f = stat[(lane & 15) * RM + warp];
          s1 = warp_sum(lane < 16 ? f.x : 0.f), s2 = warp_sum(lane < 16 ? f.y : 0.f);
        }
        const float dm = s1 * (1.f / D_MODEL);
        const float rstd = rsqrtf(fmaxf(s2 * (1.f / D_MODEL) - dm * dm, 0.f) + st.eps);
        const int c = ps * NTP * 8 + lane, ch = tile0 * 8 + c;
        float y = rstd * (sum_tiles() * scale[PASSES == 1 ? 0 : ps] - dm * lg[PASSES == 1 ? 0 : ps]) + lb[PASSES == 1 ? 0 : ps] +
                  bias[PASSES == 1 ? 0 : ps];
        const bool mine = lane < NTP * 8 && c < nt * 8;
        if (what == 2) {
          y = act_fn(y, p.act);
          if constexpr (BF) {
            if (mine) st_word(out + warp * 4096 + perm32(ch, MAP_F), __float_as_uint(y));
          } else {
            const float o = __shfl_xor_sync(0xffffffffu, y, 1);
            if (mine && !(lane & 1)) st_word(out + warp * 2048 + perm16(ch, MAP_F), pack_f16(y, o));
          }
        } else if (mine) {
          if (what == 3) {
            if (p.logits) p.logits[(size_t)warp * p.vocab + ch] = y;
            if (y > best) best = y, arg = ch;  // a lane's channels ascend: the first maximum stays, NaN never wins
          } else {
            st_word(out + warp * pitch + ch, __float_as_uint(y));
          }
        }
      }
      par ^= 1;
    }
  }

  // ---- a projection that updates the residual stream: channels 8 cta .. + 7 ----------------------------------------------------
  struct Residual {
    float scale, bias, gn;
  };
  DEVI Residual residual_values(const FStage& st) const {
    Residual r{1.f, 0.f, 1.f};
    if (warp < R) {
      const int ch = 8 * cta + (lane & 7);
      if (!W16) r.scale = __ldg(st.w.scale + ch);
      if (st.w.bias) r.bias = __ldg(st.w.bias + ch);
      if (!BF) r.gn = __ldg(st.gamma + ch);
    }
    return r;
  }
  DEVI void residual_update(const Residual& r, uint32_t* x, bool map, bool publish) {
    barrier();
    if (warp < R) {
      resid += sum_one() * r.scale + r.bias;
      if (publish) publish_x(x, r.gn, map);
    }
    par ^= 1;
  }
  DEVI void out_projection(const FStage& st, const uint32_t* att, uint32_t* x, int slot, bool map, bool publish) {
    const Residual r = residual_values(st);
    Op a;
    const uint32_t* r0 = att + row0 * (BF ? 1024 : 512) + warp * PW + t * 4;
    const uint32_t* r1 = att + row1 * (BF ? 1024 : 512) + warp * PW + t * 4;
    uint4 v[HALVES * PC];
    hold(item.live ? HOP : HOP + IDLE);
    poll(v, wait, [&](int i) { return i < PC ? r0 + i * 16 : r1 + (i - PC) * 16; });
    operand(v, a);
    cp_async_wait_group<5>();
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tile(acc, a, tile_at(slot));
    store_partial(0, acc);
    residual_update(r, x, map, publish);
  }
  DEVI void fc2_projection(const FStage& st, const uint32_t* mid, uint32_t* x) {
    const Residual r = residual_values(st);
    uint4 late[W16 ? 6 : 1];  // 16-bit weights: the pieces that are not in the ring
    if constexpr (W16) {
#pragma unroll
      for (int i = 0; i < 6; ++i) late[i] = ld_stream16(st.w.w + at_fc2() + (2 + i) * 1024);
    }
    constexpr int NB = BF ? (R16 ? 1 : 2) : 4;  // 64-blocks polled at once
    const uint32_t* r0 = mid + row0 * (BF ? 4096 : 2048) + warp * 4 * PW + t * 4;
    const uint32_t* r1 = mid + row1 * (BF ? 4096 : 2048) + warp * 4 * PW + t * 4;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int b0 = 0; b0 < 4; b0 += NB) {
      uint4 v[NB * HALVES * PC];
      if (b0 == 0) hold(HOP);
      poll(v, wait, [&](int i) {
        const int b = i / (HALVES * PC), h = (i / PC) % HALVES;
        return (h ? r1 : r0) + (b0 + b) * PW + (i % PC) * 16;
      });
      if (b0 == 0) cp_async_wait_group<5>();
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        Op a;
        operand(v + b * HALVES * PC, a);
        const int blk = b0 + b;
        float(&ac)[4] = acc[blk & 1];
        if constexpr (S24) {
          const uint4 q = slot16(T::S_FC2 + (blk >> 1));
          const uint32_t m = sel[(4 + (blk >> 1)) * FT];
          if (blk & 1) mma_24(ac, a, q.z, q.w, m >> 16);
          else mma_24(ac, a, q.x, q.y, m);
        } else if constexpr (W16) {
          mma_w16(ac, a, 0, blk == 0 ? slot16(T::S_FC2) : late[2 * blk - 2]);
          mma_w16(ac, a, 1, blk == 0 ? slot16(T::S_FC2 + 1) : late[2 * blk - 1]);
        } else {
          mma_int8(ac, a, slot16(T::S_FC2 + blk));
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[0][e] += acc[1][e];
    store_partial(0, acc[0]);
    residual_update(r, x, MAP_A, true);
  }

  // ---- attention: this CTA's (row, head), or two of them on eight warps each ------------------------------------------------
  // The cache passes are those of attention.cu (attend_range, attend_range_q8) with one running maximum per warp.
  static constexpr int LD = Q8 ? 16 : 8;                    // dims per lane (a 16-byte load)
  static constexpr int VB = D * (Q8 ? 1 : 2);               // bytes of a cached vector
  static constexpr int LPK = D / LD, GPW = 32 / LPK, U = Q8 ? 2 : 4, SET = D + 4;
  struct Item {
    int r, h, nw, wi, half;       // row, head; nw warps share it, this one is warp wi; half: which of the CTA's two
    int n_self, n_cross;          // cached keys
    uint32_t vec_self, vec_cross;  // index of its key 0 in the two caches
    bool live;
  };
  Item item;
  DEVI void setup_item(const int* s_slot, const int* s_self, const int* s_cross) {
    const int items = R * p.heads;
    item.nw = items > FC ? FW / 2 : FW;
    item.half = warp / item.nw, item.wi = warp % item.nw;
    const int it = cta + FC * item.half, i = it < items ? it : 0;
    item.live = it < items;
    item.h = i % p.heads, item.r = i / p.heads;
    const uint32_t head = s_slot[item.r] * p.heads + item.h;
    item.n_self = s_self[item.r], item.n_cross = s_cross[item.r];
    item.vec_self = head * p.seq, item.vec_cross = head * p.frames;
  }
  DEVI void prefetch_cache(int li, bool self) const {  // towards L2, a stage or more before the keys are read
    if (!item.live) return;
    char* const* c = caches + li * 8 + (self ? 0 : 2);
    const int bytes = (self ? item.n_self : item.n_cross) * VB;
    const size_t at = (size_t)(self ? item.vec_self : item.vec_cross) * VB;
    for (int o = (item.wi * 32 + lane) * 128; o < bytes; o += item.nw * 4096) prefetch_l2_line(c[0] + at + o), prefetch_l2_line(c[1] + at + o);
  }
  DEVI static float2 fma2(float2 a, float2 b, float2 c) {  // two fp32 multiply-adds in one instruction
    float2 d;
    asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmov.b64 z, {%6, %7};\n"
        "fma.rn.f32x2 z, x, y, z;\nmov.b64 {%0, %1}, z;\n}\n"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
  }
  DEVI static float2 unpack(uint32_t w) { return make_float2(bf16_lo(w), bf16_hi(w)); }

  DEVI void attention(int li, bool self, const uint32_t* q0, uint32_t* att) {
    if (item.live) {
      const int grp = lane / LPK, gl = lane % LPK;
      char* const* c = caches + li * 8 + (self ? 0 : 2);
      const int n = self ? item.n_self : item.n_cross;
      const uint32_t vec0 = self ? item.vec_self : item.vec_cross;
      char* kc = c[0] + (size_t)vec0 * VB + gl * 16;
      char* vc = c[1] + (size_t)vec0 * VB + gl * 16;
      float* ksc = Q8 ? reinterpret_cast<float*>(c[4]) + vec0 : nullptr;
      float* vsc = Q8 ? reinterpret_cast<float*>(c[5]) + vec0 : nullptr;
      const int step = item.nw * GPW;
      int j = item.wi * GPW + grp;  // this lane's key of u = 0
      uint4 kk[U], vv[U];
      float ks[Q8 ? U : 1], vs[Q8 ? U : 1];
      auto fetch = [&]() {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int ju = j + u * step;
          kk[u] = vv[u] = make_uint4(0, 0, 0, 0);
          if constexpr (Q8) ks[u] = 1.f, vs[u] = 0.f;
          if (ju < n) {
            kk[u] = ld_stream16(kc + ju * VB), vv[u] = ld_stream16(vc + ju * VB);
            if constexpr (Q8) ks[u] = __uint_as_float(ld_stream4(ksc + ju)), vs[u] = __uint_as_float(ld_stream4(vsc + ju));
          }
        }
      };
      fetch();
      // the query, and for the warp that appends (its share of the keys is the smallest) the new key and value
      const bool append = self && item.wi == item.nw - 1;
      constexpr int QP = LD / 4;
      uint4 qv[3 * QP];
      const uint32_t* src = q0 + item.r * (self ? 3072 : 1024) + item.h * D + gl * LD;
      const int kv = append ? 1024 : 0;  // the others look at the query again
      hold(HOP);
      poll(qv, wait, [&](int i) { return src + (i / QP) * kv + (i % QP) * 4; });
      float m = -1e30f, sum = 0.f;
      float2 q[LD / 2], acc[LD / 2];
      __half2 qh[Q8 ? 8 : 1], ah[Q8 ? 8 : 1];
      auto value = [&](int which, int i) {  // dims 2 i, 2 i + 1 of the query, new key or new value
        const uint4 u = qv[which * QP + i / 2];
        return i & 1 ? make_float2(__uint_as_float(u.z), __uint_as_float(u.w)) : make_float2(__uint_as_float(u.x), __uint_as_float(u.y));
      };
#pragma unroll
      for (int i = 0; i < LD / 2; ++i) {
        q[i] = value(0, i);
        q[i].x *= p.scale_log2, q[i].y *= p.scale_log2;
        acc[i] = make_float2(0.f, 0.f);
        if constexpr (Q8) qh[i] = __floats2half2_rn(q[i].x, q[i].y), ah[i] = __float2half2_rn(0.f);
      }
      auto over_lanes = [&](float d) {
#pragma unroll
        for (int o = 1; o < LPK; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        return d;
      };
      if (append) {  // rounded into the cache; attended as the bf16 values
        uint32_t kn[LD / 2], vn[LD / 2];
        float2 d = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LD / 2; ++i) {
          const float2 k = value(1, i), v = value(2, i);
          kn[i] = pack_bf16(k.x, k.y), vn[i] = pack_bf16(v.x, v.y);
          d = fma2(q[i], unpack(kn[i]), d);
        }
        m = over_lanes(d.x + d.y);  // every lane group has the score; one counts the key
        if constexpr (Q8) {
          quantise(kn, kc + n * VB, ksc + n, grp, gl);
          quantise(vn, vc + n * VB, vsc + n, grp, gl);
        } else if (grp == 0) {
          *reinterpret_cast<uint4*>(kc + n * VB) = make_uint4(kn[0], kn[1], kn[2], kn[3]);
          *reinterpret_cast<uint4*>(vc + n * VB) = make_uint4(vn[0], vn[1], vn[2], vn[3]);
        }
        if (grp == 0) {
          sum = 1.f;
#pragma unroll
          for (int i = 0; i < LD / 2; ++i) {
            acc[i] = unpack(vn[i]);
            if constexpr (Q8) ah[i] = __floats2half2_rn(acc[i].x, acc[i].y);
          }
        }
      }
      const int rounds = (n - item.wi * GPW + U * step - 1) / (U * step);  // the same for the whole warp
#pragma unroll 1
      for (int r = 0; r < rounds; ++r, j += U * step) {
        if (r) fetch();
        float sc[U], mx = m;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float d;
          const uint32_t w[4] = {kk[u].x, kk[u].y, kk[u].z, kk[u].w};
          if constexpr (Q8) {
            __half2 a0 = __float2half2_rn(0.f), a1 = a0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t lo, hi;
              widen_u8(w[i] ^ 0x80808080u, lo, hi);
              a0 = __hfma2(qh[2 * i], *reinterpret_cast<const __half2*>(&lo), a0);
              a1 = __hfma2(qh[2 * i + 1], *reinterpret_cast<const __half2*>(&hi), a1);
            }
            const float2 f = __half22float2(__hadd2(a0, a1));
            d = (f.x + f.y) * ks[u];
          } else {
            float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) d2 = fma2(q[i], unpack(w[i]), d2);
            d = d2.x + d2.y;
          }
          d = over_lanes(d);
          sc[u] = j + u * step < n ? d : -INFINITY;
          mx = fmaxf(mx, sc[u]);
        }
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float a = ex2f(m - mx);
        sum *= a;
        if constexpr (Q8) {
          const __half2 a2 = __float2half2_rn(a);
#pragma unroll
          for (int i = 0; i < 8; ++i) ah[i] = __hmul2(ah[i], a2);
        } else {
#pragma unroll
          for (int i = 0; i < LD / 2; ++i) acc[i].x *= a, acc[i].y *= a;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float e = ex2f(sc[u] - mx);
          sum += e;
          const uint32_t w[4] = {vv[u].x, vv[u].y, vv[u].z, vv[u].w};
          if constexpr (Q8) {
            const __half2 eh = __float2half2_rn(e * vs[u]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t lo, hi;
              widen_u8(w[i] ^ 0x80808080u, lo, hi);
              ah[2 * i] = __hfma2(eh, *reinterpret_cast<const __half2*>(&lo), ah[2 * i]);
              ah[2 * i + 1] = __hfma2(eh, *reinterpret_cast<const __half2*>(&hi), ah[2 * i + 1]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = fma2(make_float2(e, e), unpack(w[i]), acc[i]);
          }
        }
        m = mx;
      }
      if constexpr (Q8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = __half22float2(ah[i]);
      }
      // the warp's (max, sum, output) set, merged over its lane groups
#pragma unroll
      for (int o = LPK; o < 32; o <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int i = 0; i < LD / 2; ++i) {
          acc[i].x += __shfl_xor_sync(0xffffffffu, acc[i].x, o);
          acc[i].y += __shfl_xor_sync(0xffffffffu, acc[i].y, o);
        }
      }
      float* b = red_buf();
      if (grp == 0) {
#pragma unroll
        for (int i = 0; i < LD / 2; i += 2)
          *reinterpret_cast<float4*>(b + warp * SET + gl * LD + 2 * i) = make_float4(acc[i].x, acc[i].y, acc[i + 1].x, acc[i + 1].y);
        if (gl == 0) *reinterpret_cast<float2*>(b + FW * SET + 2 * warp) = make_float2(m, sum);
      }
    }
    barrier();
    const int d = item.wi * 32 + lane;
    if (item.live && d < D) {  // a thread per dim; the sets' weights once per warp, lane w holding set w's
      const int w0 = item.half * item.nw;
      const float* b = red_buf();
      float2 f = *reinterpret_cast<const float2*>(b + FW * SET + 2 * (w0 + (lane & (item.nw - 1))));
      float M = f.x;
#pragma unroll
      for (int o = 1; o < FW; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));  // eight sets: each counted twice
      const float e = ex2f(f.x - M);
      float L = e * f.y;
      for (int o = 1; o < item.nw; o <<= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
      float O[4] = {0.f, 0.f, 0.f, 0.f};
      const float* ob = b + w0 * SET + d;
#pragma unroll 1
      for (int w = 0; w < item.nw; w += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) O[k & 3] += __shfl_sync(0xffffffffu, e, w + k) * ob[(w + k) * SET];
      const float v = ((O[0] + O[1]) + (O[2] + O[3])) / L;
      const int k = item.h * D + d;
      if constexpr (BF) {
        st_word(att + item.r * 1024 + perm32(k, MAP_A), __float_as_uint(v));
      } else {
        const float o = __shfl_xor_sync(0xffffffffu, v, 1);
        if (!(d & 1)) st_word(att + item.r * 512 + perm16(k, MAP_A), pack_f16(v, o));
      }
    }
    par ^= 1;
  }
  // the reference's int8 cache format (see attend_range_q8)
  DEVI void quantise(const uint32_t (&bf)[LD / 2], char* dst, float* scale, int grp, int gl) {
    float f[LD], mx = 0.f;
#pragma unroll
    for (int i = 0; i < LD / 2; ++i) f[2 * i] = bf16_lo(bf[i]), f[2 * i + 1] = bf16_hi(bf[i]);
#pragma unroll
    for (int i = 0; i < LD; ++i) mx = fmaxf(mx, fabsf(f[i]));
#pragma unroll
    for (int o = 1; o < LPK; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float sc = mx > 0.f ? __fdiv_rn(mx, 127.f) : 1.f, inv = __fdiv_rn(1.f, sc);
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < LD; ++i)
      w[i >> 2] |= (uint32_t)(__float2int_rn(fminf(fmaxf(__fmul_rn(f[i], inv), -127.f), 127.f)) & 0xff) << ((i & 3) * 8);
    if (grp == 0) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
      if (gl == 0) *scale = sc;
    }
  }

  // ---- the step ------------------------------------------------------------------------------------------------------------
  // row `warp`: the embedding's LayerNorm, this CTA's 8 channels of it
  DEVI void embedding(const int* s_slot, uint32_t* x, float gn) {
    if (warp < R) {
      const int s = s_slot[warp];
      int64_t tk = p.tok[s];
      int ps = p.pos[s];
      const bool report = cta == 0 && lane == 0;
      if (tk < 0 || tk >= p.vocab) {
        if (report) atomicOr(p.status, B200DEC_ST_TOKEN_RANGE);
        tk = 0;
      }
      if (ps < 0 || ps >= p.max_pos) {
        if (report) atomicOr(p.status, B200DEC_ST_POS_RANGE);
        ps = 0;
      }
      float v[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = i * 128 + lane * 4;
        const uint2 e = *reinterpret_cast<const uint2*>(p.embed + (size_t)tk * D_MODEL + c);
        const uint2 q = *reinterpret_cast<const uint2*>(p.ptab + (size_t)ps * D_MODEL + c);
        v[4 * i] = bf16_lo(e.x) + bf16_lo(q.x), v[4 * i + 1] = bf16_hi(e.x) + bf16_hi(q.x);
        v[4 * i + 2] = bf16_lo(e.y) + bf16_lo(q.y), v[4 * i + 3] = bf16_hi(e.y) + bf16_hi(q.y);
      }
      float s1 = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) s1 += v[i];
      const float mean = warp_sum(s1) * (1.f / D_MODEL);
      float s2 = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) s2 += (v[i] - mean) * (v[i] - mean);
      const float rstd = rsqrtf(warp_sum(s2) * (1.f / D_MODEL) + p.ln0.eps);
      // channel 8 cta + (lane & 7): the value itself again, from the tables
      const int ch = 8 * cta + (lane & 7);
      const float mine = __bfloat162float(p.embed[(size_t)tk * D_MODEL + ch]) + __bfloat162float(p.ptab[(size_t)ps * D_MODEL + ch]);
      resid = (mine - mean) * rstd * __ldg(p.ln0.w + ch) + __ldg(p.ln0.b + ch);
      publish_x(x, gn, MAP_A);
    }
  }

  DEVI void pick(const uint32_t* parts, int s) {  // warp 0 of CTA r: row r; see pick_kernel (rowops.cu)
    uint4 v[2];
    poll(v, wait, [&](int i) { return parts + (cta * FC + lane * 4) * 2 + 4 * i; });
    float b = __uint_as_float(v[0].x);
    int a = (int)v[0].y;
    const float ob[3] = {__uint_as_float(v[0].z), __uint_as_float(v[1].x), __uint_as_float(v[1].z)};
    const int oa[3] = {(int)v[0].w, (int)v[1].y, (int)v[1].w};
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (ob[i] > b || (ob[i] == b && oa[i] < a)) b = ob[i], a = oa[i];
    first_max(b, a);
    if (lane != 0 || s < 0 || s >= p.slots) return;  // the dummy slot never advances
    if (a < 0 || a >= p.vocab) a = 0;                // a row of NaN
    if (p.argmax) p.argmax[s] = a;
    if (p.finished[s]) return;
    const int at = p.pos[s] + 1;
    const bool in_prompt = at < p.plen[s];
    const int64_t nt = in_prompt ? p.forced[(size_t)s * p.max_prompt + min(at, p.max_prompt - 1)] : (int64_t)a;
    if (at < p.out_cols) p.out[(size_t)s * p.out_cols + at] = nt;
    p.tok[s] = nt;
    p.pos[s] = at;
    const uint8_t done = (!in_prompt && (nt == p.eos || at >= p.limit[s])) ? 1 : 0;
    p.finished[s] = done;
    if (done && p.flags_host) p.flags_host[s] = 1;
  }

  DEVI void run(const int* s_slot, const int* s_self, const int* s_cross) {
    const FLayout lay(R, BF);
    const int parity = (int)(ld_poll4(p.ws) & 1u);
    uint32_t* base = p.ws + 16 + (size_t)parity * p.set_words + lay.x;  // the first layer's buffers
    // the first layer's weights, one cp.async group per projection
    fill_k1024(tab[0].w.w, T::S_QKV, 3 * cta, 3), cp_async_commit();
    fill_k1024(tab[1].w.w, T::S_O, cta, 1), cp_async_commit();
    fill_k1024(tab[2].w.w, T::S_CQ, cta, 1), cp_async_commit();
    fill_k1024(tab[3].w.w, T::S_CO, cta, 1), cp_async_commit();
    fill_fc1(tab[4].w), cp_async_commit();
    fill_fc2(tab[5].w), cp_async_commit();
    embedding(s_slot, base - lay.x, __ldg(p.layer[0].gamma[0] + 8 * cta + (lane & 7)));
    setup_item(s_slot, s_self, s_cross);
    prefetch_cache(0, true);
    {  // the other set is next step's: fill it again
      uint4* o = reinterpret_cast<uint4*>(p.ws + 16 + (size_t)(parity ^ 1) * p.set_words);
      for (uint32_t i = cta * FT + tid; i < (uint32_t)(p.set_words / 4); i += FC * FT)
        o[i] = make_uint4(F_EMPTY, F_EMPTY, F_EMPTY, F_EMPTY);
    }
    const int tiles = p.vocab / 8, per = (tiles + FC - 1) / FC, passes = (per + 3) / 4, blocks = p.layers * 3;
    // A layer is three blocks: qkv, self-attention, o; cross-q, cross-attention, cross-o; fc1, fc2. Behind the last
    // layer the vocabulary projection goes through the same LayerNorm-folding code, four tiles at a time.
    int li = 0, k = 0;
#pragma unroll 1
    for (int s = 0; s < blocks + passes; ++s) {
      const bool head = s >= blocks, last = li + 1 >= p.layers;
      const FStage* e = tab + (head ? p.layers * 6 : li * 6 + 2 * k);
      const int ps = s - blocks, tile0 = head ? cta * per + ps * 4 : (k == 0 ? 3 : k == 1 ? 1 : 4) * cta;
      const int nt = head ? max(0, min(min(4, per - ps * 4), tiles - tile0)) : k == 0 ? 3 : k == 1 ? 1 : 4;
      const int slot = head ? (ps * 4 % T::HT) * CH : k == 0 ? T::S_QKV : k == 1 ? T::S_CQ : T::S_FC1;
      const uint32_t* x = base + (head || k == 0 ? -lay.x : k == 1 ? lay.o_x_o() : lay.o_x_co());
      uint32_t* out = base + (k == 0 ? lay.o_qkv() : k == 1 ? lay.o_cq() : lay.o_mid());
      ln_projection(head ? 3 : k, *e, x, out, k == 0 ? 3072 : 1024, tile0, nt, slot);
      // the slots just read: the same projection of the next layer; from the last layer on, the vocabulary projection
      if (head) fill_head(ps * 4 + T::HT, 4, tiles, per);
      else if (last) fill_head(slot / CH, min(nt, T::HT - slot / CH), tiles, per);
      else if (k == 2) fill_fc1(e[6].w);
      else fill_k1024(e[6].w.w, slot, tile0, nt);
      cp_async_commit();
      if (head) continue;
      if (k < 2) {
        uint32_t* att = base + (k == 0 ? lay.o_att_s() : lay.o_att_c());
        attention(li, k == 0, out, att);
        // the caches that the next attention reads
        if (k == 0) prefetch_cache(li, false);
        else if (!last) prefetch_cache(li + 1, true);
        const int so = k == 0 ? T::S_O : T::S_CO;
        out_projection(e[1], att, base + (k == 0 ? lay.o_x_o() : lay.o_x_co()), so, k == 0 ? MAP_A : MAP_F,
                       !(p.withhold && s == 0 && cta == 1));
        if (last) fill_head(so / CH, 1, tiles, per);
        else fill_k1024(e[7].w.w, so, cta, 1);
        if constexpr (W16) {
          if (k == 1)  // fc2's pieces past the ring
#pragma unroll
            for (int i = 2; i < 8; ++i) prefetch_l2_line(e[3].w.w + at_fc2() + i * 1024);
        }
        ++k;
      } else {
        fc2_projection(e[1], out, base + lay.o_x_f());
        if (last) fill_head(T::S_FC2 / CH, T::HT - T::S_FC2 / CH, tiles, per);
        else fill_fc2(e[7].w);
        k = 0, ++li, base += lay.layer;
      }
      cp_async_commit();
    }
    if (warp < R) {
      first_max(best, arg);
      if (lane < 2) st_word(base + (warp * FC + cta) * 2 + lane, lane ? (uint32_t)arg : __float_as_uint(best));
    }
    if (cta < R && warp == 0) {
      pick(base, s_slot[cta]);
      if (cta == 0 && lane == 0) p.ws[0] = (uint32_t)(parity ^ 1);  // every CTA has published, so every CTA has read it
    }
  }
};

template <int MODE, int D, bool Q8, bool R16>
__global__ void __launch_bounds__(FT, 1) fused_step_kernel(const __grid_constant__ FArgs p) {
  using T = FTraits<MODE, R16>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_slot[F_MAX_ROWS], s_self[F_MAX_ROWS], s_cross[F_MAX_ROWS];
  __shared__ uint32_t lut[32];
  const int tid = threadIdx.x;
  if (tid < p.rows) {  // slots and lengths, clamped into range (a bad value is reported through the status word)
    int s = p.active[tid];
    const bool report = blockIdx.x == 0;
    if (s < 0 || s > p.slots) {
      if (report) atomicOr(p.status, B200DEC_ST_SLOT_RANGE);
      s = p.slots;
    }
    int n = p.pos[s], f = p.cross_len[s];
    if (n < 0 || n >= p.seq) {
      if (report) atomicOr(p.status, B200DEC_ST_POS_RANGE);
      n = max(0, min(n, p.seq - 1));
    }
    if (f < 1 || f > p.frames) {
      if (report) atomicOr(p.status, B200DEC_ST_FRAMES_RANGE);
      f = max(1, min(f, p.frames));
    }
    s_slot[tid] = s, s_self[tid] = n, s_cross[tid] = f;
  }
  if (T::S24 && tid < 32) {  // byte-permute controls of the 2:4 selectors, as in linear_kernel.cuh
    const int i0 = tid & 3, i1 = (tid >> 2) & 3, odd = tid >> 4;
    uint32_t ctl = 0;
    for (int q = 0; q < 4; ++q) {
      uint32_t sl = 4;
      if (q == i1) sl = odd ? 3 : 1;
      if (q == i0) sl = odd ? 2 : 0;
      ctl |= sl << (4 * q);
    }
    lut[tid] = ctl;
  }
  // the stage table: one thread per (layer, projection)
  FStage* tab = reinterpret_cast<FStage*>(smem + T::OFF_TAB);
  for (int i = tid; i < p.layers * 6; i += FT) {
    const FLayer& l = p.layer[i / 6];
    const int k = i % 6;
    const bool last = i / 6 + 1 == p.layers;
    FStage s{k == 0 ? l.qkv : k == 1 ? l.o : k == 2 ? l.cq : k == 3 ? l.co : k == 4 ? l.fc1 : l.fc2, nullptr, 0.f, 0};
    if (k == 0 || k == 2 || k == 4) s.gamma = l.gamma[k / 2], s.eps = l.eps[k / 2];
    else s.gamma = k == 1 ? l.gamma[1] : k == 3 ? l.gamma[2] : last ? p.gamma_f : p.layer[i / 6 + 1].gamma[0];
    tab[i] = s;
  }
  char** caches = reinterpret_cast<char**>(smem + T::OFF_CACHES);
  for (int i = tid; i < p.layers * 8; i += FT) {
    const FLayer& l = p.layer[i >> 3];
    void* c = l.sk;  // self keys, values, cross keys, values, then their scales in the same order
    switch (i & 7) {
      case 1: c = l.sv; break;
      case 2: c = l.ck; break;
      case 3: c = l.cv; break;
      case 4: c = l.sks; break;
      case 5: c = l.svs; break;
      case 6: c = l.cks; break;
      case 7: c = l.cvs; break;
    }
    caches[i] = reinterpret_cast<char*>(c);
  }
  if (tid == FT - 1) {  // the vocabulary projection's entry
    FStage s{p.head, p.gamma_f, p.eps_f, 0};
    tab[p.layers * 6] = s;
  }
  __syncthreads();
  FusedStep<MODE, D, Q8, R16> step(p, smem, lut);
  step.run(s_slot, s_self, s_cross);
}

template <int MODE>
int launch_fused_mode(const FArgs& a, int head_dim, bool q8, cudaStream_t stream) {
  auto go = [&](auto kern, int bytes) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return fail(B200DEC_ECUDA, "fused step: smem attribute: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(FC), cfg.blockDim = dim3(FT), cfg.dynamicSmemBytes = bytes, cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // its CTAs wait for one another: all or none are resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, a);
    if (e != cudaSuccess) return fail(B200DEC_ECUDA, "fused step launch: %s", cudaGetErrorString(e));
    return 0;
  };
  auto rows = [&](auto d, auto q) {
    constexpr int D = decltype(d)::value;
    constexpr bool Q = decltype(q)::value;
    if (a.rows <= 8) return go(fused_step_kernel<MODE, D, Q, false>, FTraits<MODE, false>::BYTES);
    if constexpr (FTraits<MODE, true>::W16 && D == 64)  // 16 heads: 128 items and more, not fused (fused_mode)
      return fail(B200DEC_EINVAL, "fused step: no kernel for %d rows of 16-bit weights and 16 heads", a.rows);
    else
      return go(fused_step_kernel<MODE, D, Q, true>, FTraits<MODE, true>::BYTES);
  };
  using i64 = std::integral_constant<int, 64>;
  using i128 = std::integral_constant<int, 128>;
  if (head_dim == 64) return q8 ? rows(i64{}, std::true_type{}) : rows(i64{}, std::false_type{});
  return q8 ? rows(i128{}, std::true_type{}) : rows(i128{}, std::false_type{});
}

int launch_fused_int8(const FArgs& a, int head_dim, bool q8, cudaStream_t s);
int launch_fused_24(const FArgs& a, int head_dim, bool q8, cudaStream_t s);
int launch_fused_f16(const FArgs& a, int head_dim, bool q8, cudaStream_t s);
int launch_fused_bf16(const FArgs& a, int head_dim, bool q8, cudaStream_t s);

}  // namespace b200dec_detail
