// Backward kernel.  A work item is one (batch, head, 128-key tile): its K_j and V_j stay in shared
// memory, dK_j and dV_j in TMEM, and the query tiles Q_i, dO_i are streamed past them.  The kernel
// is persistent: one CTA per SM takes items from a ticket counter until none are left, so that
// the loads and first products of the next item overlap the dK/dV epilogue of the current one and
// uneven items (causal, ragged lengths) balance themselves.
//
// Takes over the work of the reference's _bwd_dense_dq_kernel / _bwd_dense_dkdv_kernel
// (src/triton_sigmoid/sigmoid_triton_dense.py:162-467) and the padded pair
// (src/triton_sigmoid/sigmoid_triton_padded.py:179-509).  The reference recomputes S and dP
// in both of its kernels (7 GEMMs per tile pair); here each tile pair costs 5:
//
//   S^T  = K_j Q_i^T            (smem x smem -> TMEM, fp32)   [key rows on TMEM lanes]
//   dP^T = V_j dO_i^T           (smem x smem -> TMEM, fp32)
//   P^T  = sigmoid(scale S^T + bias), dS^T = P^T (1 - P^T) dP^T        (registers)
//   dV_j += P^T  dO_i           (TMEM x smem -> TMEM)
//   dK_j += dS^T Q_i            (TMEM x smem -> TMEM)
//   dQ_i  = dS K_j              (smem x smem -> TMEM), then added into an fp32 accumulator in
//                                global memory by bulk reductions out of shared memory (see acc_piece)
//
// Warp roles (28 warps):
//   warps 0-15  compute: warp w owns TMEM lanes (key rows) 32 (w & 3) .. +31 and the query
//               columns 32 (w >> 2) .. +31 of every tile
//   warp  16    item scheduler + TMA producer (also clears padded rows of tiles that straddle a valid length)
//   warp  17    tcgen05 issuer A: S^T and dP^T; owns the TMEM allocation
//   warp  18    tcgen05 issuer B: dV, dK, dQ
//   warp  19    idle
//   warps 20-27 dQ drain: take finished dQ tiles out of TMEM (freeing the columns at once) and feed the reductions
//               while the compute warps are on the next tile.  At D = 64 they also take the epilogue (dK_j, dV_j) of
//               short items, see kDrainEpilogueMaxTiles.
//               Registers are re-balanced with setmaxnreg.  To fit, the compute warps of D = 64 do not keep P in
//               registers between their two phases but read its 16-bit copy back from TMEM.
// What bounds it (timeline of one SM, B=4 T=4096 H=16): D = 128 shared memory - the operands of S, dP and dQ, which
// saturate its 128 bytes per clock while they run, the tiles coming in, dS, and dQ going out: 3800 of a tile's 4200
// clocks (1.70 -> 1.42 ms for the backward when the drain moved from the compute warps to these); D = 64 the two phases
// of the compute warps with the barriers between them, 2900 clocks (0.85 -> 0.77 ms).  Times in these two are of single calls, at 1.8 to 1.9 GHz, bf16.
// Repeated calls of that size run at the board's power limit, at 1.5 to 1.65 GHz, where a step saves what it saves in energy: B=4 T=4096 H=16 D = 64 takes 850 us
// at 993 W (time x nvidia-smi's power.draw over a second); left out of it for the purpose, the phases' arithmetic was 107 mJ and dQ's way out 86.
// Figures of several steps in this file are from different boards and are not to be added up; each pair was timed in turn.
// Two issuing warps, because one warp's instruction stream (waits, 32 MMAs, commits per tile
// pair) is a serial chain that otherwise bounds the kernel.  Everything the two exchange goes
// through mbarriers: "S columns free" after dV, "dP columns free" after dK.
// dQ = scale * accumulator is rounded to the 16-bit type by sigattn_dq_convert_kernel; in the kByHead form by the drain warps.
#pragma once

#include "ptx.cuh"
#include "sigmoid_math.cuh"

namespace sigattn {

struct BwdParams {
  // fp32, zero-filled before the launch: one region of (rows of the sequence) x D floats per batch element and head,
  // see acc_piece()
  // (kByHead: one region per CTA, not filled)
  float* dq_acc;
  int64_t acc_sb, acc_sh;  // floats from one batch element / head to the next (packed: acc_sb = 0)
  void* dk;
  void* dv;
  int64_t dk_sb, dk_st, dk_sh;
  int64_t dv_sb, dv_st, dv_sh;
  const int* lens_q;
  const int* lens_k;
  // Packed (variable-length) layout: sequence b occupies rows cu_q[b] .. cu_q[b+1]-1 of a (total, H, D)
  // tensor (likewise cu_k for keys / values); Tq, Tk are then upper bounds of the lengths and dq_acc has
  // one region per head and sequence.  nullptr = (B, T, H, D).
  const int* cu_q;
  const int* cu_k;
  const float* bias;
  const float* score_mod;
  float scale;
  float bias_scalar;
  int B, H, Tq, Tk;
  int d_cols;   // columns of the tensors in memory (<= D; the rest reads as zeros and is not written)
  int causal;
  int n_kvblk;  // ceil(Tk / 128)
  int n_items;  // B * H * n_kvblk
  int group;    // (batch, head) pairs per scheduling group, >= 1 (see bwd_decode_item)
  void* dq;     // kByHead only (else sigattn_dq_convert_kernel writes dQ)
  int64_t dq_sb, dq_st, dq_sh;
  // two counters, zero between launches: [0] items handed out beyond the first per CTA,
  // [1] CTAs that have finished (the last one clears both)
  unsigned int* ticket;
};

constexpr int kBwdComputeWarps = 16;
constexpr int kBwdProducerWarp = 16;
constexpr int kBwdIssuerA = 17;
constexpr int kBwdIssuerB = 18;
constexpr int kBwdDrainWarps = 8;
// D = 64: the drain warps also take the epilogue (dK_j, dV_j out of TMEM and to global memory) of items with at most
// this many query tiles, so that the compute warps go straight on to the next item; for longer items, whose
// epilogue is a small share, the compute warps do it themselves (the drain warps, busy with it, would fall
// behind with the next item's dQ tiles: measured -1.5 % at 32 tiles per item, +7 % at 4).
// (D = 128: the compute warps always do; the drain warps have no shared memory to turn rows in.)
template <int D> constexpr int kDrainEpilogueMaxTiles = (D == 64) ? 8 : 0;
constexpr int kBwdFirstDrainWarp = 20;
constexpr int kBwdThreads = (kBwdFirstDrainWarp + kBwdDrainWarps) * 32;
constexpr int kBwdTileKV = 128;
constexpr int kBwdTileQ = 128;

template <int D>
struct BwdSmem {
  static constexpr int kStages = 2;                      // Q tiles
  static constexpr int kDoStages = (D == 64) ? 2 : 1;      // dO tiles (one at D = 128: the room goes to the drain's patches)
  static constexpr int kTileBytes = 128 * D * 2;
  // K_j / V_j buffers: two at D = 64 (the next item's are loaded while this item still computes), one at
  // D = 128 (no room for more)
  static constexpr int kKvBufs = (D == 64) ? 2 : 1;
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kKOff + kKvBufs * kTileBytes;
  static constexpr int kQOff = kVOff + kKvBufs * kTileBytes;
  static constexpr int kDoOff = kQOff + kStages * kTileBytes;
  static constexpr int kDsOff = kDoOff + kDoStages * kTileBytes;
  static constexpr int kDsBytes = 128 * 128 * 2;
  // a private 4 KB patch per drain warp: 32 query rows x 32 head columns of dQ on their way to the accumulator; at
  // D = 64 also 32 rows x 64 bytes of dK / dV in the epilogue of short items, turned there so that four adjacent lanes
  // write one row (16 bytes of padding per row keep the 16-byte accesses of different rows off each other's banks)
  static constexpr int kPatchRow = 64 + 16;
  static constexpr int kDqPatchOff = kDsOff + kDsBytes;
  static constexpr int kDqPatchBytes = 4096;
  static constexpr int kBarOff = kDqPatchOff + kBwdDrainWarps * kDqPatchBytes;
  static constexpr int kKvFull = 0;                   // [2] per K/V buffer
  static constexpr int kQFull = 2;                    // [2]
  static constexpr int kQEmpty = kQFull + kStages;    // [2]  both issuers release a stage
  static constexpr int kDoFull = kQEmpty + kStages;     // [kDoStages]
  static constexpr int kDoEmpty = kDoFull + kDoStages;  // [kDoStages]
  static constexpr int kSFull = kDoEmpty + kDoStages;   // [2] S^T written (per S buffer)
  static constexpr int kDpFull = kSFull + 2;          // dP^T written
  static constexpr int kPReady = kDpFull + 1;         // [2] P^T in TMEM (16 warps; per S buffer)
  static constexpr int kDsReady = kPReady + 2;        // dS^T in TMEM and shared memory (16 warps)
  static constexpr int kSFree = kDsReady + 1;         // dV has consumed P^T: S columns reusable
  static constexpr int kDpFree = kSFree + 1;          // dK has consumed dS^T: dP columns reusable
  static constexpr int kDqFull = kDpFree + 1;         // [2] dQ tile complete in TMEM
  static constexpr int kDqEmpty = kDqFull + 2;        // [2] dQ tile read out (8 drain warps)
  static constexpr int kDkvFull = kDqEmpty + 2;       // every MMA of the CTA complete
  static constexpr int kKvFix = kDkvFull + 1;         // [2] per K/V buffer: padded rows of K_j zeroed
  static constexpr int kQdoFix = kKvFix + 2;          // [2] per stage: padded rows of the last Q_i / dO_i zeroed
  static constexpr int kKvEmpty = kQdoFix + 2;        // [2] per K/V buffer, both issuers: every product that reads it is complete
  static constexpr int kDkvEmpty = kKvEmpty + 2;      // [2] dK_j, dV_j read out of TMEM: [0] by the 16 compute warps, [1] by the 8 drain warps (short items at D = 64)
  static constexpr int kItemFull = kDkvEmpty + 2;     // [2] item index published
  static constexpr int kItemEmpty = kItemFull + 2;    // [2] item index read by every consumer warp
  static constexpr int kNumBars = kItemEmpty + 2;
  static constexpr int kMiscOff = (kBarOff + 8 * kNumBars + 15) & ~15;  // tmem base (u32), abort flag (int), 2 x item record (16 int each)
  static constexpr int kTotal = kMiscOff + 16 + 2 * 64;
  static constexpr int kDynBytes = kTotal + 1024;
};

// Masked tiles (a key or query beyond the valid ones, the causal diagonal): a logit of minus infinity makes a probability of exactly zero on every
// way, and has no say in the form that a chunk takes, whatever lies in the padded rows (padded batch of 16 <= 2048, H=8, 243 -> 237 us against a general
// polynomial for all masked tiles, 24 packed sequences, D=128, 231 -> 226, B=40 T=500 H=16 D=128 410 -> 369).  One instantiation for
// masked and other tiles, with the mask behind a branch, took 205 us for B=40 T=500 H=16 D=64 where this took 218, but 5 to 9 % more where few tiles are masked.
// Bit i: column q0 + i is a valid query, q_lo <= q < q_hi.
__device__ __forceinline__ uint32_t bwd_valid_columns(int q0, int q_lo, int q_hi) {
  const int a = min(max(q_lo - q0, 0), 32), b = min(max(q_hi - q0, 0), 32);
  const uint32_t below_b = b < 32 ? (1u << b) - 1u : 0xffffffffu, below_a = a < 32 ? (1u << a) - 1u : 0xffffffffu;
  return below_b & ~below_a;
}
__device__ __forceinline__ void bwd_mask_logits(float2 (&t)[16], uint32_t valid) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    t[i].x = (valid & (1u << (2 * i))) ? t[i].x : -INFINITY;
    t[i].y = (valid & (2u << (2 * i))) ? t[i].y : -INFINITY;
  }
}

// The two phases of one tile for one thread (its key row, 32 query columns) in the D = 128 kernel.
//
// Phase A: scores -> probabilities, kept in registers for phase B; their 16-bit packing is written over the first 16
// of the 32 columns read (the operand of dV).  Both phases move 16 columns at a time, so that besides the 32
// probabilities only few registers are live.
// masked: only columns with their bit in `valid` count.
template <bool kBF16, bool kMask, bool kAccurate, DeepTest kTest>
__device__ __forceinline__ void bwd_phase_a(uint32_t s_addr, float c1, float c0, uint32_t valid,
                                            float2 (&pv)[16], DeepWatch& watch) {
  // tested tiles work on logits shifted up (see sigmoid2_far)
  const float c0s = kTest == kNoTest ? c0 : c0 + kFarShift;
  {
    uint32_t r[32];
    tmem_ld32_sync(s_addr, r);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      pv[i] = __ffma2_rn(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), make_float2(c1, c1),
                         make_float2(c0s, c0s));
  }
  if constexpr (kMask) bwd_mask_logits(pv, valid);
  // f(logits) -> probabilities, in place; eight pairs at a time leave for TMEM
  auto emit = [&](auto f) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t pk[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 pe = f(pv[8 * h + i]);
        pv[8 * h + i] = pe;
        pk[i] = pack2<kBF16>(pe.x, pe.y);
      }
      tmem_st8(s_addr + 8 * h, pk);
    }
  };
  if constexpr (kAccurate) {
    // exponential and reciprocal both on the special-function unit (see sigmoid2_accurate_from_log2)
    emit([](float2 x) { return sigmoid2_accurate_from_log2(x); });
  } else if (kTest != kNoTest && warp_all_negative(pv)) {
    watch.passed();
    // all logits far below zero (the usual case under the default bias): short series, no compare / select per element
    emit([](float2 x) { return sigmoid2_far<kBF16>(x); });
  } else {
    bool all_neg = false;
    if constexpr (kTest != kNoTest) {
#pragma unroll
      for (int i = 0; i < 16; ++i) pv[i] = __fadd2_rn(pv[i], make_float2(-kFarShift, -kFarShift));
      // Negative but not far below zero: full polynomial, still no select.  Not looked for in masked tiles, whose code is shorter for it: with it B=8 T=8192
      // H=32 causal is 11.50 ms instead of 11.20, B=4 T=4096 H=8 736 us instead of 708, and no masked call is faster.
      if constexpr (kTest == kTestAll && !kMask) all_neg = warp_all_negative(pv);
      if constexpr (kTest == kTestNow) watch.failed();
    }
    if (all_neg) emit([](float2 x) { return sigmoid2_from_log2_neg<kBF16>(x); });
    else         emit([](float2 x) { return sigmoid2_from_log2<kBF16>(x); });
  }
}

// Phase B: dS = P (1 - P) dP for the same 32 columns; 16-bit dS^T goes to TMEM (over the first
// 16 dP columns read) and to the swizzled shared-memory copy the dQ GEMM reads.
template <bool kBF16, bool kMask>
__device__ __forceinline__ void bwd_phase_b(uint32_t dp_addr, uint32_t ds_line, uint32_t chunk0, uint32_t sw,
                                            const float2 (&pv)[16]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t r[16], pk[8];
    tmem_ld16(dp_addr + 16 * h, r);
    tmem_ld_wait_for(r);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 pp = pv[8 * h + i];
      const float2 w = __ffma2_rn(make_float2(-pp.x, -pp.y), pp, pp);  // P - P^2
      float2 d = __fmul2_rn(w, make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
      if constexpr (kMask) {
        d.x = (pp.x != 0.0f) ? d.x : 0.0f;  // masked elements have P exactly 0; keeps NaN/Inf padding out
        d.y = (pp.y != 0.0f) ? d.y : 0.0f;
      }
      pk[i] = pack2<kBF16>(d.x, d.y);
    }
    tmem_st8(dp_addr + 8 * h, pk);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const uint32_t chunk = (chunk0 + 2 * h + m) ^ sw;  // 128-byte swizzle: 16-byte chunk index XOR (row & 7)
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ds_line + chunk * 16), "r"(pk[4 * m]),
                   "r"(pk[4 * m + 1]), "r"(pk[4 * m + 2]), "r"(pk[4 * m + 3])
                   : "memory");
    }
  }
}

// The two phases for the D = 64 kernel.  The probabilities are not kept in registers between the phases
// (32 registers per thread that the drain warps' share of the register file cannot spare) but read back
// from TMEM in the 16-bit form they were stored in for the dV product, and dS = P (1 - P) dP is formed on
// packed 16-bit pairs.
template <bool kBF16, bool kMask, bool kAccurate, DeepTest kTest, DeepRange kRange>
__device__ __forceinline__ void bwd_phase_a16(uint32_t s_addr, float c1, float c0, uint32_t valid, DeepWatch& watch) {
  uint32_t r[32];
  tmem_ld32_sync(s_addr, r);
  uint32_t pk[16];
  float2 t[16];
  // Masked tiles of short sequences (the near range) are tested by their largest logit, unshifted, so that those that fail pay no way back from the
  // shift and no second look at all signs: such calls have many masked tiles, and with scores of larger deviation most fail.  B=40 T=500 H=16 bf16, deviation
  // 3: 246 us with the general polynomial in all masked tiles, 258 with the shift, 227 so; deviation 1 265, 230, 222; B=16 T=1000, deviation 3, 330, 322, 304.
  // In the far range no such call got slower by the shift, and this test would move the code of whole tiles: B=4 T=4096 H=16 fp16 891 against 910.
  constexpr bool kByLargest = kMask && kTest != kNoTest && kRange == kNear;
  const float c0s = kTest == kNoTest || kByLargest ? c0 : c0 + kDeepShift<kRange, kBF16>;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    t[i] = __ffma2_rn(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), make_float2(c1, c1),
                      make_float2(c0s, c0s));
  if constexpr (kMask) bwd_mask_logits(t, valid);
  float most = 0.0f;
  if constexpr (kByLargest) most = largest(t);
  if constexpr (kAccurate) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 pe = sigmoid2_accurate_from_log2(t[i]);
      pk[i] = pack2<kBF16>(pe.x, pe.y);
    }
  } else if (kByLargest && __all_sync(0xffffffffu, most < -kNearShift<kBF16>)) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 pe = sigmoid2_near<kBF16, false>(t[i]);
      pk[i] = pack2<kBF16>(pe.x, pe.y);
    }
  } else if (kTest != kNoTest && !kByLargest && warp_all_negative(t)) {
    watch.passed();
    // the usual case under the default bias: short polynomial, no compare / select per element
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if constexpr (kRange == kFar && !kMask) {
        pk[i] = sigmoid2_far_packed<kBF16>(t[i], false);
      } else if constexpr (kRange == kFar) {  // (in single precision: no further from the sigmoid than the general polynomial)
        const float2 pe = sigmoid2_far<kBF16>(t[i]);
        pk[i] = pack2<kBF16>(pe.x, pe.y);
      } else {
        const float2 pe = sigmoid2_near<kBF16>(t[i]);
        pk[i] = pack2<kBF16>(pe.x, pe.y);
      }
    }
  } else {
    bool all_neg = false;
    if constexpr (kByLargest) {
      all_neg = __all_sync(0xffffffffu, most < 0.0f);
    } else if constexpr (kTest != kNoTest) {
#pragma unroll
      for (int i = 0; i < 16; ++i) t[i] = __fadd2_rn(t[i], make_float2(-kDeepShift<kRange, kBF16>, -kDeepShift<kRange, kBF16>));
      if constexpr (kTest == kTestAll) all_neg = warp_all_negative(t);
      else watch.failed();
    }
    if (all_neg) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 pe = sigmoid2_from_log2_neg<kBF16>(t[i]);
        pk[i] = pack2<kBF16>(pe.x, pe.y);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 pe = sigmoid2_from_log2<kBF16>(t[i]);
        pk[i] = pack2<kBF16>(pe.x, pe.y);
      }
    }
  }
  tmem_st16(s_addr, pk);
}

template <bool kBF16, bool kMask>
__device__ __forceinline__ void bwd_phase_b16(uint32_t p_addr, uint32_t dp_addr, uint32_t ds_line, uint32_t chunk0,
                                              uint32_t sw) {
  uint32_t pp[16], r[32];
  tmem_ld16(p_addr, pp);
  tmem_ld32(dp_addr, r);
  tmem_ld_wait_for(pp);
  tmem_ld_wait_for(r);
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t ph = pp[i];
    const uint32_t w = hfma2<kBF16>(ph ^ 0x80008000u, ph, ph);  // P - P^2
    uint32_t d = hmul2<kBF16>(w, pack2<kBF16>(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
    if constexpr (kMask) {
      // masked elements have P exactly 0: force dS to 0 there, whatever (NaN, Inf) the padding put into dP
      const uint32_t keep = ((ph & 0x00007fffu) ? 0x0000ffffu : 0u) | ((ph & 0x7fff0000u) ? 0xffff0000u : 0u);
      d &= keep;
    }
    pk[i] = d;
  }
  tmem_st16(dp_addr, pk);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const uint32_t chunk = (chunk0 + m) ^ sw;  // 128-byte swizzle: 16-byte chunk index XOR (row & 7)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ds_line + chunk * 16), "r"(pk[4 * m]),
                 "r"(pk[4 * m + 1]), "r"(pk[4 * m + 2]), "r"(pk[4 * m + 3])
                 : "memory");
  }
}

// The fp32 dQ accumulator.  Each (batch element, head) has a region of its rows x D floats.  A quarter (32 rows, fewer
// at the region's end) of query tile i starts at (128 i + 32 quarter) D and holds [D / 32][8][rows][4] floats: blocks of
// 32 columns, in them the four-column pieces, in those the rows.  That is the order in which a drain warp, one query row
// per lane, writes 32 columns to shared memory without bank conflicts, and one bulk reduction adds the 4 KB to global
// memory.  (Reductions issued lane by lane, red.global.add, reach the same 5.8 TB/s of the L2, but they wait for it in
// the load/store queue of the SM, and every barrier and shared-memory access of the other warps waits behind them: 250
// to 450 clocks per barrier in a timeline of one SM.)
__device__ __forceinline__ int acc_piece(int rows, int c4, int row) { return ((c4 * rows) + row) * 4; }

// One work item.  The producer warp decodes it once (integer divisions, length and bias loads from global
// memory) and publishes the record through shared memory; every other role reads it from there.
struct BwdItem {
  int b, h, kv0;
  int bc;               // batch coordinate of the tensor maps and strides (0 when packed)
  int tq0, tk0;         // first row of the sequence in the token dimension (0 unless packed)
  int key_lim;          // key rows below this exist in this sequence's tensors (Tk; packed: Lk)
  int64_t acc_base;     // start of the (batch element, head) in the dQ accumulator, in floats
  int Lq, Lk;
  int i_begin, n_q;     // first query tile that sees this key tile, number of query tiles
  bool ragged_kv;       // the key tile straddles Lk
  // rows beyond the valid length have to be cleared: of K_j, of the last Q_i and dO_i (not where the tensors end there: those come as zeros)
  bool clear_k, clear_q;
  float bias;           // additive bias of the item's batch element
};
// record layout in shared memory: 16 ints, the first the item index (-1: no more work).  Read and written 16 bytes at a time: 27 warps read each, and
// int by int that was 430 accesses an item (24 packed sequences <= 1500, H=8, D=128 267 -> 260 us, B=512 T=512 H=16 2315 -> 2280).
__device__ __forceinline__ void bwd_publish_item(int4* rec, int item, const BwdItem& it) {
  rec[0] = make_int4(item, it.b, it.h, it.kv0);
  rec[1] = make_int4(it.bc, it.tq0, it.tk0, it.key_lim);
  rec[2] = make_int4((int)(uint32_t)((uint64_t)it.acc_base & 0xffffffffull), (int)(uint32_t)((uint64_t)it.acc_base >> 32), it.Lq, it.Lk);
  rec[3] = make_int4(it.i_begin, it.n_q, (it.ragged_kv ? 1 : 0) | (it.clear_k ? 2 : 0) | (it.clear_q ? 4 : 0), __float_as_int(it.bias));
}
// (behind the barrier that says that the record is there: the wait is a compiler barrier)
__device__ __forceinline__ int bwd_load_item(const int4* rec, BwdItem& it) {
  const int4 a = rec[0], b = rec[1], c = rec[2], d = rec[3];
  it.b = a.y; it.h = a.z; it.kv0 = a.w;
  it.bc = b.x; it.tq0 = b.y; it.tk0 = b.z; it.key_lim = b.w;
  it.acc_base = (int64_t)(((uint64_t)(uint32_t)c.y << 32) | (uint64_t)(uint32_t)c.x);
  it.Lq = c.z; it.Lk = c.w;
  it.i_begin = d.x; it.n_q = d.y;
  it.ragged_kv = (d.z & 1) != 0; it.clear_k = (d.z & 2) != 0; it.clear_q = (d.z & 4) != 0; it.bias = __int_as_float(d.w);
  return a.x;
}
template <int D>
__device__ __forceinline__ BwdItem bwd_decode_item(const BwdParams& p, int item) {
  BwdItem it;
  // Groups of `group` (batch, head) pairs: within a group every pair's key tile 0 comes first, then
  // every pair's tile 1, ... (under a causal mask the early tiles are the heavy ones, so this is a
  // longest-first order), while the Q / dO of one group still fit the L2.  group = 1: (batch, head)-major.
  const int per_group = p.group * p.n_kvblk;
  const int grp = item / per_group;
  const int r = item - grp * per_group;
  const int g_eff = min(p.group, p.B * p.H - grp * p.group);
  const int j = r / g_eff;  // key tile
  const int bh = grp * p.group + (r - j * g_eff);
  it.b = bh / p.H;
  it.h = bh - it.b * p.H;
  it.kv0 = j * kBwdTileKV;
  it.Lq = p.Tq;
  it.Lk = p.Tk;
  if (p.lens_q) it.Lq = min(max(p.lens_q[it.b], 0), p.Tq);
  if (p.lens_k) it.Lk = min(max(p.lens_k[it.b], 0), p.Tk);
  it.bc = it.b;
  it.tq0 = it.tk0 = 0;
  it.key_lim = p.Tk;
  if (p.cu_q) {
    it.tq0 = p.cu_q[it.b];
    it.tk0 = p.cu_k[it.b];
    it.Lq = min(max(p.cu_q[it.b + 1] - it.tq0, 0), p.Tq);
    it.Lk = min(max(p.cu_k[it.b + 1] - it.tk0, 0), p.Tk);
    it.bc = 0;
    it.key_lim = it.Lk;
  }
  it.acc_base = (int64_t)it.bc * p.acc_sb + (int64_t)it.h * p.acc_sh + (int64_t)it.tq0 * D;
  const int i_end = (it.Lq + kBwdTileQ - 1) / kBwdTileQ;
  it.i_begin = p.causal ? j : 0;  // query tiles that can see this key tile (top-left aligned)
  it.n_q = (it.kv0 < it.Lk) ? max(i_end - it.i_begin, 0) : 0;
  it.ragged_kv = it.kv0 + kBwdTileKV > it.Lk;
  it.clear_k = it.ragged_kv && (p.cu_q || it.Lk < p.Tk);
  it.clear_q = (it.i_begin + it.n_q) * kBwdTileQ > it.Lq && (p.cu_q || it.Lq < p.Tq);  // only the last query tile can straddle Lq
  it.bias = item_bias(p.bias, p.bias_scalar, it.b, it.Lk);
  return it;
}

// kByHead: a CTA takes all key tiles of a (batch element, head), in order, and finishes its dQ itself (see the drain
// warps), so that the accumulator needs neither the fill nor the conversion pass and stays in the L2.  group is 1 and the
// tickets count (batch, head) pairs.  (This form spills more, see the registers below.)
// kForm: as in the forward kernel (at D = 128, where P is in single precision, the far range only).
template <int D, bool kBF16, bool kAccurate, bool kByHead, DeepForm kForm>
__global__ void __launch_bounds__(kBwdThreads, 1)
sigattn_bwd_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                   const __grid_constant__ CUtensorMap v_map, const __grid_constant__ CUtensorMap do_map,
                   const BwdParams p) {
  using L = BwdSmem<D>;
  constexpr int kTileBytes = L::kTileBytes;
  constexpr uint32_t kTmemCols = 512;
  // TMEM plan.  D = 64: two S^T buffers (tiles alternate), so that the scores of the next tile are
  // computed while this one is still being processed; dQ_i is written over the S^T buffer of its
  // own tile once dV has read P^T from it:   S0 0 | S1 128 | dP 256 | dV 384 | dK 448.
  // D = 128: no room for that: one S^T buffer, dQ over the dP^T columns:  S 0 | dP 128 | dV 256 | dK 384.
  // Column group c keeps its 16-bit P^T in S columns 32c + [0,16), dS^T likewise in the dP columns.
  constexpr bool kTwoS = (D == 64);
  // Products per pass of the loops that issue them.  The roles' code together is more than the SM's instruction caches hold: at D = 128 loops of
  // two passes are 1 to 3 % faster for it (B=8 T=8192 H=32 causal 11.21 -> 10.92 ms, B=128 T=512 H=8 573 -> 563 us; four passes or eight 1 to 20 %
  // slower), at D = 64, whose products are half as long, none is, nor in the forms whose elementwise phases are longer: bias above -3, B=4 T=4096
  // H=16 D=128 bias 0 1502 us in loops of two passes, 1461 unrolled (fp16 1526, 1449); accurate sigmoid, B=1 T=20224 H=8 4440, 4188.
  constexpr int kMmaUnroll = (D == 64 || kForm == kDeepWatched || kAccurate) ? 8 : 4;
  constexpr uint32_t kColS = 0;
  constexpr uint32_t kColDp = kTwoS ? 256 : 128;
  constexpr uint32_t kColDv = kTwoS ? 384 : 256;
  constexpr uint32_t kColDk = kColDv + D;
  static_assert(kColDk + D <= kTmemCols, "TMEM budget");
  // Query tiles are numbered through the whole life of the CTA (g = tiles of earlier items + index
  // within the item): stages, S buffers and barrier parities simply run on from item to item.
  // index and parity of the per-S-buffer barriers for tile g
  auto sbuf = [](int g) -> int { return kTwoS ? (g & 1) : 0; };
  auto spar = [](int g) -> uint32_t { return kTwoS ? (uint32_t)(g >> 1) & 1u : (uint32_t)g & 1u; };
  // stage of dO of tile g and the parity of that stage's "full" barrier
  auto do_stage = [](int g) -> int { return L::kDoStages == 2 ? (g & 1) : 0; };
  auto do_par = [](int g) -> uint32_t { return L::kDoStages == 2 ? (uint32_t)(g >> 1) & 1u : (uint32_t)g & 1u; };
  // where dQ of tile g is written
  auto dq_col = [&](int g) -> uint32_t { return kTwoS ? kColS + 128u * (uint32_t)(g & 1) : kColDp; };
  constexpr int kSiteBase = 0x20000;
  // compute warps, the two issuing warps and the drain warps read the item ring
  constexpr int kItemReaders = kBwdComputeWarps + 2 + kBwdDrainWarps;

  extern __shared__ uint8_t smem_dyn[];
  const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
  const uint32_t bars = smem_base + L::kBarOff;
  auto bar = [&](int slot) -> uint32_t { return bars + 8u * slot; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + L::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + L::kMiscOff + 4);
  int4* item_ring = reinterpret_cast<int4*>(smem_gen + L::kMiscOff + 16);  // 2 records of 16 ints

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // a kernel of this library already gave up on a wait: do not pile more work on a sick device
  // (looked at behind the set-up, where the warps meet anyway)
  const bool sick = *reinterpret_cast<volatile int*>(&g_status_word) != 0;

  // (without a second item, or pair, for any CTA nobody asks for one, and the counters stay as they are)
  const int n_tickets = kByHead ? p.B * p.H : p.n_items;
  const bool tickets = n_tickets > (int)gridDim.x;

  // ---------------------------------------------------------------- setup
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(L::kKvFull + i), 1);
      mbar_init(bar(L::kKvFix + i), 1);
      mbar_init(bar(L::kQdoFix + i), 1);
      mbar_init(bar(L::kKvEmpty + i), 2);  // issuer A (S^T, dP^T) and issuer B (dQ)
    }
    for (int i = 0; i < L::kStages; ++i) {
      mbar_init(bar(L::kQFull + i), 1);
      mbar_init(bar(L::kQEmpty + i), 2);   // S^T (issuer A) and dK (issuer B) both read Q_i
    }
    for (int i = 0; i < L::kDoStages; ++i) {
      mbar_init(bar(L::kDoFull + i), 1);
      mbar_init(bar(L::kDoEmpty + i), 2);  // dP^T (issuer A) and dV (issuer B) both read dO_i
    }
    mbar_init(bar(L::kSFull + 0), 1);
    mbar_init(bar(L::kSFull + 1), 1);
    mbar_init(bar(L::kDpFull), 1);
    mbar_init(bar(L::kPReady + 0), kBwdComputeWarps);
    mbar_init(bar(L::kPReady + 1), kBwdComputeWarps);
    mbar_init(bar(L::kDsReady), kBwdComputeWarps);
    mbar_init(bar(L::kSFree), 1);
    mbar_init(bar(L::kDpFree), 1);
    mbar_init(bar(L::kDqFull + 0), 1);
    mbar_init(bar(L::kDqFull + 1), 1);
    mbar_init(bar(L::kDqEmpty + 0), kBwdDrainWarps);
    mbar_init(bar(L::kDqEmpty + 1), kBwdDrainWarps);
    mbar_init(bar(L::kDkvFull), 1);
    mbar_init(bar(L::kDkvEmpty + 0), kBwdComputeWarps);
    mbar_init(bar(L::kDkvEmpty + 1), kBwdDrainWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(L::kItemFull + i), 1);
      mbar_init(bar(L::kItemEmpty + i), kItemReaders);
    }
    fence_mbar_init();
  }
  if (warp == kBwdProducerWarp && lane == 0) {
    tma_prefetch_desc(&q_map);
    tma_prefetch_desc(&k_map);
    tma_prefetch_desc(&v_map);
    tma_prefetch_desc(&do_map);
  }
  if (warp == kBwdIssuerA) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  // one answer for the CTA: the word may change while its warps read it
  const bool leave = __syncthreads_or(sick);
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  if (leave) {
    if (warp == kBwdIssuerA) tmem_dealloc(tmem, kTmemCols);
    return;
  }

  // Consumer side of the item ring: returns the k-th item of this CTA, or -1 when there is none
  // (also on a failed wait).  Called by all 32 lanes of a reader warp.
  auto read_item = [&](int k, BwdItem& it) -> int {
    const int slot = k & 1;
    if (!mbar_wait_warp(bar(L::kItemFull + slot), (uint32_t)(k >> 1) & 1u, abort_flag, kSiteBase + 30)) return -1;
    // (Of the last record only the -1 holds.  The general form of D = 64 looks at it before it reads on: B=4 T=4096 H=16 fp16 893 us so, 912 without, T=1024 bf16 534
    // and 551, 16 padded sequences 246 and 251.  The others read on at once, which spares them registers: by head B=128 T=512 H=16 fp16 598 us so, 618 with
    // the look, D = 128 B=8 T=8192 H=32 causal 11.4 and 11.8 ms, 24 packed sequences 235 and 238 us.)
    int item = 0;
    if constexpr (D == 64 && !kByHead) item = *reinterpret_cast<const volatile int*>(item_ring + 4 * slot);
    if (item >= 0) item = bwd_load_item(item_ring + 4 * slot, it);
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(L::kItemEmpty + slot));
    return item;
  };

  // 896 threads get 72 registers each at launch.  Each aligned group of four warps executes one instruction; the counts add up to
  // exactly what the CTA holds:
  //   D = 64:  compute 80, role 56, drain 64 (512 x 80 + 128 x 56 + 256 x 64);
  //   D = 128: compute 72, role 56, drain 80 (a dQ tile goes from the drain warps' registers, 64 per thread, to the
  //            accumulator in two steps, so that its TMEM columns are free for the next dP at once; 512 x 72 + 128 x 56 + 256 x 80).
  // The instructions stand inside the roles' branches: the compiler allocates registers up to a count only in code that it alone leads to.
  // Before a join it kept to 72 everywhere, and all roles spilled.  Bytes of stores / loads by -Xptxas -v, general and by head, bf16: D = 64 68 / 80
  // and 132 / 192 then, 20 / 16 and 68 / 80 now (bias above -3: 32 / 52 and 84 / 96); D = 128 120 / 188 and 208 / 300 then, 56 / 72 and 156 / 188 now (fp16
  // 40 / 40 and 140 / 156; bias above -3: 80 / 108 and 188 / 236).  Backward, B=512 T=512 H=16 bf16 2190 -> 2060 us, 24 packed sequences <= 1500, H=8, D=128
  // 287 -> 278, B=8 T=8192 H=32 D=128 causal 11.91 -> 11.45 ms at the power cap.
  if (warp >= kBwdFirstDrainWarp) {
    if constexpr (D == 64) setmaxnreg_dec<64>(); else setmaxnreg_inc<80>();
    // ============================================================ dQ drain
    // Warp d = warp - 20: lane quarter d & 3 (32 query rows, one per lane), half of the head columns d >> 2.  Per tile:
    // wait for the dQ product, take the block into registers, release the TMEM columns, then add it into the
    // accumulator (see acc_piece).
    {
      const int dw = warp - kBwdFirstDrainWarp;
      const int quarter = dw & 3, half = dw >> 2;
      constexpr int kCols = D / 2;  // head columns per warp
      const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
      uint8_t* patch = smem_gen + L::kDqPatchOff + dw * L::kDqPatchBytes;
      int g = 0;
      int act = 0;  // items with work so far
      bool ok = true;
      for (int k = 0; ok; ++k) {
        BwdItem it;
        const int item = read_item(k, it);
        if (item < 0) break;
        const int row_lim = p.cu_q ? it.Lq : p.Tq;
        // kByHead: the first key tile of a query tile stores its dQ instead of adding it (no fill before the launch), the
        // last one adds the accumulator to its own and writes the rounded rows (no conversion after it).  All of a
        // block's traffic is this warp's, so waiting for its own bulk operations orders it.
        uint8_t* dq_rows = nullptr;  // row 0 of the sequence, this warp's columns
        int last_j = 0;              // last key tile with keys
        if constexpr (kByHead) {
          dq_rows = reinterpret_cast<uint8_t*>(p.dq) +
                    2 * ((int64_t)it.bc * p.dq_sb + (int64_t)it.h * p.dq_sh + (int64_t)it.tq0 * p.dq_st + kCols * half);
          last_j = (it.Lk + kBwdTileKV - 1) / kBwdTileKV - 1;
          if (it.kv0 == 0) {
            // rows of query tiles that no product is computed for
            for (int row = it.n_q * kBwdTileQ + quarter * 32 + lane; row < row_lim; row += 128)
              for (int c = 0; c < kCols && kCols * half + c < p.d_cols; c += 8)
                *reinterpret_cast<uint4*>(dq_rows + 2 * ((int64_t)row * p.dq_st + c)) = make_uint4(0, 0, 0, 0);
          } else {
            if (lane == 0) {
              bulk_wait_all();  // what earlier key tiles stored and added is in memory
              fence_proxy_async_global();
            }
            __syncwarp();
          }
        }
        if (it.n_q == 0) continue;
        for (int t = 0; t < it.n_q; ++t) {
          const int gt = g + t;
          ok = mbar_wait_warp(bar(L::kDqFull + sbuf(gt)), spar(gt), abort_flag, kSiteBase + 14);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t addr = tmem + lane_addr + dq_col(gt) + (uint32_t)(kCols * half);
          uint32_t r[kCols / 32][32];
#pragma unroll
          for (int c = 0; c < kCols / 32; ++c) tmem_ld32(addr + 32 * c, r[c]);
#pragma unroll
          for (int c = 0; c < kCols / 32; ++c) tmem_ld_wait_for(r[c]);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(L::kDqEmpty + sbuf(gt)));  // the TMEM columns are free again
          const int row0 = (it.i_begin + t) * kBwdTileQ + quarter * 32;
          const int rows = min(row_lim - row0, 32);  // rows at or beyond Lq hold zeros, which do no harm
          if (rows <= 0) continue;
          float* dst = p.dq_acc + (kByHead ? (int64_t)blockIdx.x * p.acc_sh : it.acc_base) + (int64_t)row0 * D +
                       (kCols / 32) * half * (rows * 32);
          const bool store = kByHead && it.kv0 == 0;
          if (kByHead && it.kv0 == kBwdTileKV * (p.causal ? min(it.i_begin + t, last_j) : last_j)) {
            const bool live = row0 + lane < it.Lq;
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c) {
              if (lane == 0) bulk_wait_read();
              __syncwarp();
              uint4* mine = reinterpret_cast<uint4*>(patch + lane * L::kPatchRow);
#pragma unroll
              for (int c8 = 0; c8 < 4; ++c8) {
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
                if (!store && lane < rows) {
                  a = __ldcg(reinterpret_cast<const float4*>(dst + c * (rows * 32) + acc_piece(rows, 2 * c8, lane)));
                  b = __ldcg(reinterpret_cast<const float4*>(dst + c * (rows * 32) + acc_piece(rows, 2 * c8 + 1, lane)));
                }
                const uint32_t* x = r[c] + 8 * c8;
                uint4 w;
                w.x = pack2<kBF16>(p.scale * (a.x + __uint_as_float(x[0])), p.scale * (a.y + __uint_as_float(x[1])));
                w.y = pack2<kBF16>(p.scale * (a.z + __uint_as_float(x[2])), p.scale * (a.w + __uint_as_float(x[3])));
                w.z = pack2<kBF16>(p.scale * (b.x + __uint_as_float(x[4])), p.scale * (b.y + __uint_as_float(x[5])));
                w.w = pack2<kBF16>(p.scale * (b.z + __uint_as_float(x[6])), p.scale * (b.w + __uint_as_float(x[7])));
                if (!live) w = make_uint4(0, 0, 0, 0);
                mine[c8] = w;
              }
              __syncwarp();
              // four lanes per row, as in the epilogue below
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int r8 = 8 * i + (lane >> 2);
                const uint4 w = *reinterpret_cast<const uint4*>(patch + r8 * L::kPatchRow + 16 * (lane & 3));
                if (r8 < rows && kCols * half + 32 * c + 8 * (lane & 3) < p.d_cols)
                  *reinterpret_cast<uint4*>(dq_rows + 2 * ((int64_t)(row0 + r8) * p.dq_st + 32 * c + 8 * (lane & 3))) = w;
              }
              __syncwarp();
            }
            continue;
          }
#pragma unroll
          for (int c = 0; c < kCols / 32; ++c) {
            if (lane == 0) bulk_wait_read();  // the patch's previous content has been read
            __syncwarp();
            if (lane < rows) {
#pragma unroll
              for (int c4 = 0; c4 < 8; ++c4)
                reinterpret_cast<uint4*>(patch)[acc_piece(rows, c4, lane) / 4] =
                    make_uint4(r[c][4 * c4], r[c][4 * c4 + 1], r[c][4 * c4 + 2], r[c][4 * c4 + 3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (store) bulk_store(dst + c * (rows * 32), smem_u32(patch), (uint32_t)rows * 128u);
              else bulk_reduce_add_f32(dst + c * (rows * 32), smem_u32(patch), (uint32_t)rows * 128u);
            }
          }
        }
        if (!ok) break;
        g += it.n_q;

        // ---- epilogue of the item: dV_j, then dK_j, out of TMEM, rounded, through the patch (so that four
        // lanes cover a row's 64 bytes and an instruction 8 rows; a lane writing its own row would touch 32
        // lines per instruction, which the load/store unit takes one at a time) and out to global memory,
        // while the compute warps are already on the next item's first tiles.
        ++act;
        if (it.n_q > kDrainEpilogueMaxTiles<D>) continue;  // the compute warps' business
        if constexpr (D == 64) {
        if (lane == 0) bulk_wait_read();  // the patch is about to be rewritten
        ok = mbar_wait_warp(bar(L::kDkvFull), (uint32_t)(act - 1) & 1u, abort_flag, kSiteBase + 15);
        if (!ok) break;
        tc_fence_after_sync();
        const bool row_ok = it.kv0 + quarter * 32 + lane < it.Lk;  // padded key rows get zero gradients
#pragma unroll
        for (int which = 0; which < 2; ++which) {  // 0: dV, 1: dK
          const uint32_t acc_addr = tmem + lane_addr + (which ? kColDk : kColDv) + 32u * (uint32_t)half;
          const float mul = which ? p.scale : 1.0f;
          uint4* mine = reinterpret_cast<uint4*>(patch + lane * L::kPatchRow);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint32_t r[16];
            tmem_ld(acc_addr + 16 * u, r);
            tmem_ld_wait_for(r);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              uint4 w;
              w.x = pack2<kBF16>(mul * __uint_as_float(r[8 * m + 0]), mul * __uint_as_float(r[8 * m + 1]));
              w.y = pack2<kBF16>(mul * __uint_as_float(r[8 * m + 2]), mul * __uint_as_float(r[8 * m + 3]));
              w.z = pack2<kBF16>(mul * __uint_as_float(r[8 * m + 4]), mul * __uint_as_float(r[8 * m + 5]));
              w.w = pack2<kBF16>(mul * __uint_as_float(r[8 * m + 6]), mul * __uint_as_float(r[8 * m + 7]));
              if (!row_ok) w = make_uint4(0, 0, 0, 0);
              mine[2 * u + m] = w;
            }
          }
          if (which == 1) {
            // both accumulators are out of TMEM: the next item's first dV / dK products may overwrite them
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(L::kDkvEmpty + 1));
          }
          __syncwarp();
          const int64_t out_st = which ? p.dk_st : p.dv_st;
          uint8_t* out = which ? reinterpret_cast<uint8_t*>(p.dk) + 2 * ((int64_t)it.bc * p.dk_sb + (int64_t)it.h * p.dk_sh + (int64_t)it.tk0 * p.dk_st)
                               : reinterpret_cast<uint8_t*>(p.dv) + 2 * ((int64_t)it.bc * p.dv_sb + (int64_t)it.h * p.dv_sh + (int64_t)it.tk0 * p.dv_st);
          out += 64 * half + 16 * (lane & 3);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r8 = 8 * i + (lane >> 2);
            const uint4 x = *reinterpret_cast<const uint4*>(patch + r8 * L::kPatchRow + 16 * (lane & 3));
            const int krow = it.kv0 + quarter * 32 + r8;
            if (krow < it.key_lim && 32 * half + 8 * (lane & 3) < p.d_cols) *reinterpret_cast<uint4*>(out + 2 * (int64_t)krow * out_st) = x;
          }
          __syncwarp();  // the patch is rewritten by the next pass
        }
        }
      }
      if (lane == 0) bulk_wait_all();  // every reduction has been performed when the kernel ends
    }
  } else if (warp >= kBwdComputeWarps) {  // (producer, issuers and the idle warp, down to the compute warps' branch)
  setmaxnreg_dec<56>();
  if (warp == kBwdProducerWarp) {
    // ============================================================ item scheduler + TMA producer
    // Rows beyond the valid lengths may hold anything (NaN included).  Masked probabilities are
    // exactly zero, but 0 * NaN is NaN inside an MMA, so the padded rows of every tile that is
    // contracted over its rows (K_j for dQ, Q_i for dK, dO_i for dV) are cleared in shared memory - unless the tensor ends with the
    // valid rows, as beyond it TMA has written zeros.  The products that mind wait for this: with a division per 16 bytes, and all products behind
    // it, up to 16,000 clocks an item (backward of 24 packed sequences <= 1500, H=8, D=128 260 -> 232 us; B=8 T=300 H=8 D=32 31.0 -> 26.8).  (The loop
    // stays rolled: unrolled it moves the other roles' code so that B=4 T=4096 H=16 fp16 takes 924 us instead of 890.  The form for bias above -3 at D = 128 is
    // the other way round, without a row to clear: bf16, bias 0, B=1 T=16384 H=8 2752 us rolled, 2609 unrolled, T=20224 4292, 4099, B=4 T=4096 H=16 1467, 1412; fp16
    // the same.)
    constexpr int kClearUnroll = D == 128 && kForm == kDeepWatched ? 4 : 1;
    auto zero_rows = [&](uint8_t* tile, int first_bad) {
#pragma unroll kClearUnroll
      for (int at = 128 * first_bad + 16 * lane; at < 128 * 128; at += 512) {
#pragma unroll
        for (int c = 0; c < D / 64; ++c) *reinterpret_cast<uint4*>(tile + c * 16384 + at) = make_uint4(0, 0, 0, 0);
      }
    };
    int g = 0;    // query tiles loaded so far (all items)
    int act = 0;  // items with work so far
    int head = 0, tile = 0;  // kByHead: the pair this CTA is on and its next key tile
    bool ok = true;
    for (int k = 0; ok; ++k) {
      const int slot = k & 1;
      ok = mbar_wait_warp(bar(L::kItemEmpty + slot), ((uint32_t)(k >> 1) & 1u) ^ 1u, abort_flag, kSiteBase + 31);
      if (!ok) break;
      int item = blockIdx.x;  // the first item needs no ticket
      if (kByHead && tile > 0 && tile < p.n_kvblk) {
        item = head * p.n_kvblk + tile++;
      } else {
        if (k > 0) {
          item = -1;
          if (lane == 0 && tickets) {
            const unsigned int tk = atomicAdd(p.ticket, 1u) + gridDim.x;
            item = tk < (unsigned int)n_tickets ? (int)tk : -1;
          }
          item = __shfl_sync(0xffffffffu, item, 0);
        }
        if (kByHead && item >= 0) {
          head = item;
          tile = 1;
          item = head * p.n_kvblk;
        }
      }
      BwdItem it = {};
      if (item >= 0) it = bwd_decode_item<D>(p, item);
      if (lane == 0) {
        bwd_publish_item(item_ring + 4 * slot, item, it);
        mbar_arrive(bar(L::kItemFull + slot));  // (release: the record is visible to whoever sees the phase)
      }
      if (item < 0) break;
      if (it.n_q == 0) continue;

      for (int t = 0; t < it.n_q && ok; ++t) {
        const int gt = g + t;
        const int st = gt & 1;
        const uint32_t ph = (uint32_t)(gt >> 1) & 1u;
        const int qrow = (it.i_begin + t) * kBwdTileQ;
        ok = mbar_wait_warp(bar(L::kQEmpty + st), ph ^ 1u, abort_flag, kSiteBase + 1);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(L::kQFull + st), kTileBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem_base + L::kQOff + st * kTileBytes + c * 16384, &q_map, bar(L::kQFull + st), c * 64, it.h, it.tq0 + qrow, it.bc);
        }
        const int dst = do_stage(gt);
        const uint32_t dph = do_par(gt);
        ok = mbar_wait_warp(bar(L::kDoEmpty + dst), dph ^ 1u, abort_flag, kSiteBase + 2);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(L::kDoFull + dst), kTileBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem_base + L::kDoOff + dst * kTileBytes + c * 16384, &do_map, bar(L::kDoFull + dst), c * 64, it.h, it.tq0 + qrow, it.bc);
        }
        if (t == 0) {
          // K_j, V_j of this item into buffer kb, once the products of the item that used it last have
          // finished reading it (the first Q / dO tiles above are already on their way)
          const int kb = act % L::kKvBufs;
          const uint32_t kph = (uint32_t)(act / L::kKvBufs) & 1u;
          ok = mbar_wait_warp(bar(L::kKvEmpty + kb), kph ^ 1u, abort_flag, kSiteBase + 32);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(bar(L::kKvFull + kb), 2 * kTileBytes);
#pragma unroll
            for (int c = 0; c < D / 64; ++c) {
              tma_load_4d(smem_base + L::kKOff + kb * kTileBytes + c * 16384, &k_map, bar(L::kKvFull + kb), c * 64, it.h, it.tk0 + it.kv0, it.bc);
              tma_load_4d(smem_base + L::kVOff + kb * kTileBytes + c * 16384, &v_map, bar(L::kKvFull + kb), c * 64, it.h, it.tk0 + it.kv0, it.bc);
            }
          }
          if (it.clear_k) {
            ok = mbar_wait_warp(bar(L::kKvFull + kb), kph, abort_flag, kSiteBase + 17);
            if (!ok) break;
            zero_rows(smem_gen + L::kKOff + kb * kTileBytes, it.Lk - it.kv0);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(L::kKvFix + kb));
          }
        }
        if (t == it.n_q - 1 && it.clear_q) {
          ok = mbar_wait_warp(bar(L::kQFull + st), ph, abort_flag, kSiteBase + 18);
          ok = ok && mbar_wait_warp(bar(L::kDoFull + dst), dph, abort_flag, kSiteBase + 19);
          if (!ok) break;
          zero_rows(smem_gen + L::kQOff + st * kTileBytes, it.Lq - qrow);
          zero_rows(smem_gen + L::kDoOff + dst * kTileBytes, it.Lq - qrow);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(L::kQdoFix + st));
        }
      }
      g += it.n_q;
      ++act;
    }
  }
  else if (warp == kBwdIssuerA) {
    // ============================================================ issuer A: S^T = K Q^T, dP^T = V dO^T
    const bool leader = elect_one();
    constexpr uint32_t idesc_st = make_idesc(128, 128, kBF16, false, false);
    constexpr uint32_t kStageStep = kTileBytes >> 4;
    // operands with rows = M / N and the 64 contiguous elements = contraction
    const uint64_t k_km = smem_desc_sw128(smem_base + L::kKOff, 16, 1024);
    const uint64_t v_km = smem_desc_sw128(smem_base + L::kVOff, 16, 1024);
    const uint64_t q_km0 = smem_desc_sw128(smem_base + L::kQOff, 16, 1024);
    const uint64_t do_km0 = smem_desc_sw128(smem_base + L::kDoOff, 16, 1024);
    const uint32_t k_lo = (uint32_t)k_km, v_lo = (uint32_t)v_km, q_lo0 = (uint32_t)q_km0, do_lo0 = (uint32_t)do_km0;
    const uint32_t hi = (uint32_t)(k_km >> 32);  // identical for all four (same layout parameters)
    auto issue = [&](uint32_t dcol, uint32_t a_lo, uint32_t b_lo) {
#pragma unroll kMmaUnroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (uint32_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
        mma_ss(leader, tmem + dcol, make_desc(a_lo + off, hi), make_desc(b_lo + off, hi), idesc_st, kk > 0);
      }
    };
    int g = 0;                // query tiles issued so far (all items)
    int act = 0;              // items with work so far
    bool ok = true;
    for (int k = 0; ok; ++k) {
      BwdItem it;
      const int item = read_item(k, it);
      if (item < 0) break;
      if (it.n_q == 0) continue;
      const int kb = act % L::kKvBufs;
      const uint32_t kv_off = (uint32_t)kb * kStageStep;  // this item's K_j / V_j buffer, in descriptor address units
      ok = mbar_wait_warp(bar(L::kKvFull + kb), (uint32_t)(act / L::kKvBufs) & 1u, abort_flag, kSiteBase + 3);
      for (int t = 0; t < it.n_q && ok; ++t) {
        const int gt = g + t;
        const int st = gt & 1;
        const uint32_t ph = (uint32_t)(gt >> 1) & 1u;  // parity of the stage's "full" barriers
        const uint32_t prev = (uint32_t)(gt - 1) & 1u;
        ok = mbar_wait_warp(bar(L::kQFull + st), ph, abort_flag, kSiteBase + 4);
        if constexpr (kTwoS) {
          // this S buffer last held tile g-2: its P^T (read by dV) and then its dQ, until that was drained
          if (gt >= 2) ok = ok && mbar_wait_warp(bar(L::kDqEmpty + sbuf(gt)), spar(gt - 2), abort_flag, kSiteBase + 5);
        } else {
          // the S columns still hold P^T of the previous tile until its dV GEMM has read them
          if (gt > 0) ok = ok && mbar_wait_warp(bar(L::kSFree), prev, abort_flag, kSiteBase + 5);
        }
        if (!ok) break;
        tc_fence_after_sync();
        issue(kColS + 128u * (uint32_t)sbuf(gt), k_lo + kv_off, q_lo0 + (uint32_t)st * kStageStep);
        mma_commit(leader, bar(L::kSFull + sbuf(gt)));
        mma_commit(leader, bar(L::kQEmpty + st));
        ok = mbar_wait_warp(bar(L::kDoFull + do_stage(gt)), do_par(gt), abort_flag, kSiteBase + 6);
        if (gt > 0) {
          // the dP columns hold dS^T of the previous tile (read by dK) and, when dQ shares them,
          // the previous dQ tile until it has been drained
          ok = ok && mbar_wait_warp(bar(kTwoS ? L::kDpFree : L::kDqEmpty), prev, abort_flag, kSiteBase + 7);
        }
        if (!ok) break;
        tc_fence_after_sync();
        issue(kColDp, v_lo + kv_off, do_lo0 + (uint32_t)do_stage(gt) * kStageStep);
        mma_commit(leader, bar(L::kDpFull));
        mma_commit(leader, bar(L::kDoEmpty + do_stage(gt)));
      }
      if (!ok) break;
      mma_commit(leader, bar(L::kKvEmpty + kb));  // this warp's products no longer read K_j, V_j once they complete
      g += it.n_q;
      ++act;
    }
  } else if (warp == kBwdIssuerB) {
    // ============================================================ issuer B: dV, dK, dQ
    const bool leader = elect_one();
    constexpr uint32_t idesc_acc = make_idesc(128, D, kBF16, false, true);  // A in TMEM, B rows = contraction
    constexpr uint32_t idesc_dq = make_idesc(128, D, kBF16, true, true);  // dQ: both operands rows = contraction
    constexpr uint32_t kStageStep = kTileBytes >> 4;
    // operands whose rows are the contraction index; the next 64-column block lies 16 KB further
    const uint64_t k_mn = smem_desc_sw128(smem_base + L::kKOff, 16384, 1024);
    const uint64_t ds_mn = smem_desc_sw128(smem_base + L::kDsOff, 16384, 1024);
    const uint64_t q_mn0 = smem_desc_sw128(smem_base + L::kQOff, 16384, 1024);
    const uint64_t do_mn0 = smem_desc_sw128(smem_base + L::kDoOff, 16384, 1024);
    const uint32_t k_lo = (uint32_t)k_mn, ds_lo = (uint32_t)ds_mn, q_lo0 = (uint32_t)q_mn0, do_lo0 = (uint32_t)do_mn0;
    const uint32_t hi = (uint32_t)(k_mn >> 32);
    // acc[key, d] (+)= A^T[key, query] (16-bit, TMEM) . B[query, d]
    auto issue_acc = [&](uint32_t dcol, uint32_t acol, uint32_t b_lo, uint32_t acc0) {
#pragma unroll kMmaUnroll
      for (int kk = 0; kk < kBwdTileQ / 16; ++kk) {
        // queries 32c .. 32c+31 sit, 16-bit packed, in columns 32c + [0,16) of the source
        mma_ts(leader, tmem + dcol, tmem + acol + 32 * (kk >> 1) + 8 * (kk & 1), make_desc(b_lo + kk * (2048 >> 4), hi),
               idesc_acc, kk > 0 ? 1u : acc0);
      }
    };
    int g = 0;    // query tiles issued so far (all items)
    int act = 0;  // items with work so far
    uint32_t kvfix_par = 0u;  // bit kb: parity of buffer kb's "padded K rows cleared" (one phase per ragged key tile in it)
    uint32_t qfix_par = 0u;   // bit st: parity of stage st's "padded Q / dO rows cleared"
    // who reads the accumulators of an item (0: compute warps, 1: drain warps), for the previous item, and the
    // parity of each of the two hand-back barriers' next phase
    int prev_kind = 0;
    uint32_t empty_par = 0u;  // bit kind
    bool ok = true;
    for (int k = 0; ok; ++k) {
      BwdItem it;
      const int item = read_item(k, it);
      if (item < 0) break;
      if (it.n_q == 0) continue;
      const int kb = act % L::kKvBufs;
      const uint32_t kv_off = (uint32_t)kb * kStageStep;
      ok = mbar_wait_warp(bar(L::kKvFull + kb), (uint32_t)(act / L::kKvBufs) & 1u, abort_flag, kSiteBase + 24);  // K_j for dQ
      // the accumulators still hold the previous item's dK, dV until its epilogue has read them
      if (ok && act > 0) {
        ok = mbar_wait_warp(bar(L::kDkvEmpty + prev_kind), (empty_par >> prev_kind) & 1u, abort_flag, kSiteBase + 33);
        empty_par ^= 1u << prev_kind;
      }
      prev_kind = it.n_q <= kDrainEpilogueMaxTiles<D> ? 1 : 0;
      for (int t = 0; t < it.n_q && ok; ++t) {
        const int gt = g + t;
        const int st = gt & 1;
        const uint32_t par = (uint32_t)gt & 1u;
        const uint32_t acc0 = t > 0 ? 1u : 0u;
        // dV += P^T dO.  The probabilities only prove that Q_i has landed (they come from S^T = K Q^T): this
        // product is the first of this warp's to read dO_i and waits for that tile itself - without it a row
        // of the stage could still hold the tile of two steps earlier (seen once in some hundred runs on one
        // shape, as dV rows carrying dO of query q - 256 instead of q).
        ok = mbar_wait_warp(bar(L::kDoFull + do_stage(gt)), do_par(gt), abort_flag, kSiteBase + 22);
        // Rows that are cleared (see the producer): the first products to mind are this warp's.  Scores and dP of padded queries or keys are
        // masked, whatever their rows hold or change to.
        if (t == it.n_q - 1 && it.clear_q) {
          ok = ok && mbar_wait_warp(bar(L::kQdoFix + st), (qfix_par >> st) & 1u, abort_flag, kSiteBase + 21);
          qfix_par ^= 1u << st;
        }
        if (t == 0 && it.clear_k) {
          ok = ok && mbar_wait_warp(bar(L::kKvFix + kb), (kvfix_par >> kb) & 1u, abort_flag, kSiteBase + 20);
          kvfix_par ^= 1u << kb;
        }
        ok = ok && mbar_wait_warp(bar(L::kPReady + sbuf(gt)), spar(gt), abort_flag, kSiteBase + 8);
        if (!ok) break;
        tc_fence_after_sync();
        issue_acc(kColDv, kColS + 128u * (uint32_t)sbuf(gt), do_lo0 + (uint32_t)do_stage(gt) * kStageStep, acc0);
        if (!kTwoS) mma_commit(leader, bar(L::kSFree));
        mma_commit(leader, bar(L::kDoEmpty + do_stage(gt)));
        // dK += dS^T Q  (no wait for Q_i of this warp's own: dS exists only because S^T = K Q^T was computed
        // from the landed tile, so its arrival precedes the barrier below)
        ok = mbar_wait_warp(bar(L::kDsReady), par, abort_flag, kSiteBase + 9);
        if (!ok) break;
        tc_fence_after_sync();
        if constexpr (kTwoS) {
          // dQ first: the compute warps wait for it before they rewrite the shared-memory copy of dS, its
          // drain starts earlier, and at the last tile of an item it is complete before dK is, so that the
          // epilogue may use the dS buffer as scratch as soon as dK_j, dV_j are complete
#pragma unroll kMmaUnroll
          for (int kk = 0; kk < kBwdTileKV / 16; ++kk) {
            const uint64_t kd = make_desc(k_lo + kv_off + kk * (2048 >> 4), hi), dsd = make_desc(ds_lo + kk * (2048 >> 4), hi);
            mma_ss(leader, tmem + dq_col(gt), dsd, kd, idesc_dq, kk > 0);
          }
          mma_commit(leader, bar(L::kDqFull + sbuf(gt)));
        }
        issue_acc(kColDk, kColDp, q_lo0 + (uint32_t)st * kStageStep, acc0);
        if (kTwoS) mma_commit(leader, bar(L::kDpFree));
        mma_commit(leader, bar(L::kQEmpty + st));
        // dK_j, dV_j are complete with the last tile's dK: to take them out of TMEM the epilogue need not wait for the last dQ.  (At D = 128 it
        // waits for that before it writes over the shared-memory copy of dS, which the product still reads.)
        if (t == it.n_q - 1) mma_commit(leader, bar(L::kDkvFull));
        if constexpr (!kTwoS) {
          // the dQ GEMM needs the previous dQ tile read out of its columns
          ok = mbar_wait_warp(bar(L::kDqEmpty), par ^ 1u, abort_flag, kSiteBase + 10);
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll kMmaUnroll
          for (int kk = 0; kk < kBwdTileKV / 16; ++kk) {
            const uint64_t kd = make_desc(k_lo + kv_off + kk * (2048 >> 4), hi), dsd = make_desc(ds_lo + kk * (2048 >> 4), hi);
            mma_ss(leader, tmem + dq_col(gt), dsd, kd, idesc_dq, kk > 0);
          }
          mma_commit(leader, bar(L::kDqFull + sbuf(gt)));
        }
      }
      if (!ok) break;
      mma_commit(leader, bar(L::kKvEmpty + kb));  // the dQ products were this warp's readers of K_j
      g += it.n_q;
      ++act;
    }
  }  // (issuer B)
  } else {
    if constexpr (D == 64) setmaxnreg_inc<80>();
    // ============================================================ compute warps
    const int quarter = warp & 3;                         // TMEM lane quarter this warp may access
    const int cg = warp >> 2;                             // query-column group: columns 32 cg .. 32 cg + 31
    const int lane_row = quarter * 32 + lane;             // key row within the tile == TMEM lane
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr0 = tmem + lane_addr + kColS + 32 * cg;  // + 128 for the second S buffer
    const uint32_t dp_addr = tmem + lane_addr + kColDp + 32 * cg;
    const float c1 = p.scale * kLog2e;
    // shared-memory copy of dS^T: [2 blocks of 64 queries][128 key rows][128 bytes], 128-byte swizzle
    const uint32_t ds_line = smem_base + L::kDsOff + (cg >> 1) * 16384 + lane_row * 128;
    const uint32_t chunk0 = (uint32_t)(cg & 1) * 4;
    const uint32_t sw = (uint32_t)(lane_row & 7);
    int g = 0;    // query tiles processed so far (all items)
    int act = 0;  // items with work so far
    bool ok = true;
    DeepWatch watch;

    for (int k = 0; ok; ++k) {
      BwdItem it;
      const int item = read_item(k, it);
      if (item < 0) break;
      const int b = it.b, h = it.h, kv0 = it.kv0, Lq = it.Lq, Lk = it.Lk, i_begin = it.i_begin, n_q = it.n_q;
      const int kv = kv0 + lane_row;
      if (n_q == 0) {
        // no query sees this key tile: its gradients are zero
        uint8_t* dk_base = reinterpret_cast<uint8_t*>(p.dk) +
                           2 * ((int64_t)it.bc * p.dk_sb + (int64_t)h * p.dk_sh + (int64_t)it.tk0 * p.dk_st);
        uint8_t* dv_base = reinterpret_cast<uint8_t*>(p.dv) +
                           2 * ((int64_t)it.bc * p.dv_sb + (int64_t)h * p.dv_sh + (int64_t)it.tk0 * p.dv_st);
        constexpr int kChunksPerRow = D * 2 / 16;
        for (int i = threadIdx.x; i < kBwdTileKV * kChunksPerRow; i += kBwdComputeWarps * 32) {
          const int row = kv0 + i / kChunksPerRow;
          if (row < it.key_lim && 8 * (i % kChunksPerRow) < p.d_cols) {
            *reinterpret_cast<uint4*>(dk_base + 2 * (int64_t)row * p.dk_st + 16 * (i % kChunksPerRow)) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(dv_base + 2 * (int64_t)row * p.dv_st + 16 * (i % kChunksPerRow)) = make_uint4(0, 0, 0, 0);
          }
        }
        continue;
      }
      float c0 = it.bias;
      if (p.score_mod && kv < it.key_lim) c0 += p.score_mod[(p.cu_k ? (int64_t)it.tk0 : (int64_t)b * p.Tk) + kv];
      c0 *= kLog2e;
      const bool row_ok = kv < Lk;
      watch.start();

      for (int t = 0; t < n_q; ++t) {
        const int gt = g + t;
        const int q0 = (i_begin + t) * kBwdTileQ + 32 * cg;  // first query index of my columns
        // valid queries for this key row: q_lo <= q < q_hi (empty when the key row is padding)
        const int q_lo = p.causal ? kv : 0;
        const int q_hi = row_ok ? Lq : 0;
        // warp-uniform on purpose: the two instantiations contain warp-collective TMEM accesses.  True for every tile with rows that the producer
        // clears (clear_k implies ragged_kv, clear_q reaches columns from Lq on only): those rows may change while S^T and dP^T are computed from them.
        const bool need_mask = it.ragged_kv || (q0 + 32 > Lq) || (p.causal && q0 < kv0 + kBwdTileKV - 1);
        float2 pv[16];  // D = 128 only: the probabilities of this tile
        ok = mbar_wait_warp(bar(L::kSFull + sbuf(gt)), spar(gt), abort_flag, kSiteBase + 12);
        const uint32_t s_addr = s_addr0 + 128u * (uint32_t)sbuf(gt);
        if (!ok) break;
        tc_fence_after_sync();
        constexpr DeepTest kTest = kForm != kDeepWatched && !kAccurate ? kTestAll : kNoTest;
        constexpr DeepRange kRange = kForm == kDeepNear ? kNear : kFar;
        const bool test_now = kForm == kDeepWatched && !kAccurate && watch.due();
        if constexpr (D == 64) {
          if (need_mask)     bwd_phase_a16<kBF16, true, kAccurate, kTest, kRange>(s_addr, c1, c0, bwd_valid_columns(q0, q_lo, q_hi), watch);
          else if (test_now) bwd_phase_a16<kBF16, false, kAccurate, kTestNow, kRange>(s_addr, c1, c0, 0u, watch);
          else               bwd_phase_a16<kBF16, false, kAccurate, kTest, kRange>(s_addr, c1, c0, 0u, watch);
        } else {
          if (need_mask)     bwd_phase_a<kBF16, true, kAccurate, kTest>(s_addr, c1, c0, bwd_valid_columns(q0, q_lo, q_hi), pv, watch);
          else if (test_now) bwd_phase_a<kBF16, false, kAccurate, kTestNow>(s_addr, c1, c0, 0u, pv, watch);
          else               bwd_phase_a<kBF16, false, kAccurate, kTest>(s_addr, c1, c0, 0u, pv, watch);
        }
        if (kForm == kDeepWatched && !need_mask && !test_now) watch.skipped();
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(L::kPReady + sbuf(gt)));

        // (Phase B rewrites the shared-memory copy of dS, which the dQ product of the previous tile reads.  That
        // product is complete when dP^T of this tile is: issuer A started the latter only after the previous tile's
        // dK (D = 64), which its issuer committed after dQ, or after its dQ had been drained (D = 128).)
        ok = mbar_wait_warp(bar(L::kDpFull), (uint32_t)gt & 1u, abort_flag, kSiteBase + 13);
        if (!ok) break;
        tc_fence_after_sync();
        if constexpr (D == 64) {
          if (need_mask) bwd_phase_b16<kBF16, true>(s_addr, dp_addr, ds_line, chunk0, sw);
          else           bwd_phase_b16<kBF16, false>(s_addr, dp_addr, ds_line, chunk0, sw);
        } else {
          if (need_mask) bwd_phase_b<kBF16, true>(dp_addr, ds_line, chunk0, sw, pv);
          else           bwd_phase_b<kBF16, false>(dp_addr, ds_line, chunk0, sw, pv);
        }
        fence_proxy_async_smem();
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(L::kDsReady));
      }
      if (!ok) break;

      // ------------------------------------------------------------ epilogue of the item
      // (before the drain of the last dQ tile; at D = 128 its product may still be running while the accumulators are read, but not while rows
      // are turned through dS); short items' at D = 64 is the drain warps' (kDrainEpilogueMaxTiles<D>): nothing of the accumulators is needed here then
      // column groups 0,1 store dV, groups 2,3 store dK (each half of the head dimension)
      if (n_q <= kDrainEpilogueMaxTiles<D>) {
        // (no arrival either: each of the two hand-back barriers is arrived on only by the warps that read the
        // accumulators of that item - a group that runs ahead must not add arrivals to a phase that still
        // waits for the other group's)
      } else {
      ok = mbar_wait_warp(bar(L::kDkvFull), (uint32_t)act & 1u, abort_flag, kSiteBase + 15);
      if (!ok) break;
      {
        tc_fence_after_sync();
        const bool is_dk = cg >= 2;
        const int col0 = (cg & 1) * (D / 2);
        const uint32_t acc_addr = tmem + lane_addr + (is_dk ? kColDk : kColDv) + col0;
        const float mul = is_dk ? p.scale : 1.0f;
        // out of TMEM already rounded to 16 bits, so that few registers are live across the hand-over
        uint4 w[D / 64][4];
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          uint32_t r[32];
          tmem_ld32_sync(acc_addr + c * 32, r);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            w[c][q4].x = pack2<kBF16>(mul * __uint_as_float(r[8 * q4 + 0]), mul * __uint_as_float(r[8 * q4 + 1]));
            w[c][q4].y = pack2<kBF16>(mul * __uint_as_float(r[8 * q4 + 2]), mul * __uint_as_float(r[8 * q4 + 3]));
            w[c][q4].z = pack2<kBF16>(mul * __uint_as_float(r[8 * q4 + 4]), mul * __uint_as_float(r[8 * q4 + 5]));
            w[c][q4].w = pack2<kBF16>(mul * __uint_as_float(r[8 * q4 + 6]), mul * __uint_as_float(r[8 * q4 + 7]));
            if (!row_ok) w[c][q4] = make_uint4(0, 0, 0, 0);
          }
        }
        // the accumulators are in registers: the next item's first dV / dK products may overwrite them
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(L::kDkvEmpty + 0));
        // row 0 of this sequence's dK or dV, at this warp's columns
        const int64_t out_st = is_dk ? p.dk_st : p.dv_st;
        uint8_t* out_base = is_dk ? reinterpret_cast<uint8_t*>(p.dk) + 2 * ((int64_t)it.bc * p.dk_sb + (int64_t)h * p.dk_sh + (int64_t)it.tk0 * p.dk_st)
                                  : reinterpret_cast<uint8_t*>(p.dv) + 2 * ((int64_t)it.bc * p.dv_sb + (int64_t)h * p.dv_sh + (int64_t)it.tk0 * p.dv_st);
        out_base += 2 * col0;
        // A lane holds 64 bytes of its key row (D = 128: twice); written as they are, one store instruction would touch 32
        // lines, and the load/store unit takes them one at a time: about 2000 clocks per item for the CTA at D = 64; at D = 128 8000 went by
        // before the slowest warp could go on to the next item.
        // Each warp therefore turns its 32 x 64-byte block through its own part of the shared-memory copy
        // of dS - the rows and 16-byte slots it writes in phase B - so that four lanes cover a row and an instruction 8 rows.  No product reads
        // that any more at D = 64, where dQ is issued before the item's last dK; at D = 128 the last dQ has to be complete first.
        if constexpr (D == 128) {
          ok = mbar_wait_warp(bar(L::kDqFull), (uint32_t)(g + n_q - 1) & 1u, abort_flag, kSiteBase + 16);
          if (!ok) break;
        }
        uint8_t* ds_gen = smem_gen + L::kDsOff + (cg >> 1) * 16384 + quarter * 32 * 128;  // row 0 of this warp's quarter
        const int sub = lane >> 2, piece = lane & 3;
        const int left = it.key_lim - (kv0 + quarter * 32 + sub);  // rows from this lane's first on
        uint8_t* out = out_base + 2 * (int64_t)(kv0 + quarter * 32 + sub) * out_st + 16 * piece;
        const int64_t out_step = 16 * out_st;
#pragma unroll
        for (int cc = 0; cc < D / 64; ++cc) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(ds_gen + lane * 128 + (((chunk0 + q4) ^ sw) << 4)) = w[cc][q4];
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // (row sub + 8 i of the quarter, which begins at a multiple of 8 rows: one swizzle phase)
            const uint4 x = *reinterpret_cast<const uint4*>(ds_gen + (sub + 8 * i) * 128 + (((chunk0 + piece) ^ (uint32_t)sub) << 4));
            if (8 * i < left && col0 + 32 * cc + 8 * piece < p.d_cols) *reinterpret_cast<uint4*>(out + i * out_step + 64 * cc) = x;
          }
          __syncwarp();  // the slots are rewritten by the next pass, or phase B of the next item
        }
      }
      }
      g += n_q;
      ++act;
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kBwdIssuerA) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (tickets && threadIdx.x == 0) {
    // the last CTA to finish leaves both counters at zero for the next launch that uses them
    __threadfence();
    const unsigned int done = atomicAdd(p.ticket + 1, 1u);
    if (done == gridDim.x - 1) {
      p.ticket[0] = 0u;
      p.ticket[1] = 0u;
      __threadfence();
    }
  }
}

// Padded batches: zero-fills the accumulator's query tiles with valid rows, which a fill of everything does not know: 16 sequences of 256 to
// 2048, H=8, D = 64 266 -> 258 us for the backward (with a conversion that reads valid rows only), D = 128 (8 of them) 198 -> 189; 64 sequences of 10 to
// 4096, H=4, 1340 -> 1273.
template <int D>
__global__ void __launch_bounds__(256) sigattn_dq_fill_kernel(float* acc, const int* lens_q, int n_tiles, int T, int H) {
  const int i = (int)(blockIdx.x % (unsigned)n_tiles), bh = (int)(blockIdx.x / (unsigned)n_tiles);
  if (128 * i >= min(lens_q[bh / H], T)) return;
  float4* dst = reinterpret_cast<float4*>(acc + ((int64_t)bh * T + 128 * i) * D);
  const int n = min(128, T - 128 * i) * (D / 4);
#pragma unroll 4
  for (int k = threadIdx.x; k < n; k += 256) dst[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// dQ = scale * accumulator, cast to the 16-bit type.  One block per (batch element, head, query tile): the accumulator's
// pieces in as they lie, turned through shared memory, whole rows out.
struct DqConvertParams {
  const float* acc;
  int64_t acc_sb, acc_sh;
  void* dq;
  int64_t sb, st, sh;
  const int* lens_q;
  const int* cu_q;
  int n_tiles, T, H;
  int d_cols;  // columns of dQ (the accumulator has D)
  float scale;
};

template <int D, bool kBF16>
__global__ void __launch_bounds__(256) sigattn_dq_convert_kernel(const DqConvertParams p) {
  constexpr int kRowBytes = 2 * D + 16;
  __shared__ __align__(16) uint8_t tile[128 * kRowBytes];
  const int i = (int)(blockIdx.x % (unsigned)p.n_tiles);
  const int bh = (int)(blockIdx.x / (unsigned)p.n_tiles);
  const int b = bh / p.H, h = bh - b * p.H;
  int tq0 = 0, limit = p.T, bc = b;
  if (p.cu_q) {
    tq0 = p.cu_q[b];
    limit = min(max(p.cu_q[b + 1] - tq0, 0), p.T);
    bc = 0;
  }
  const int rows = min(limit - 128 * i, 128);
  if (rows <= 0) return;
  const int live = (p.lens_q ? min(max(p.lens_q[b], 0), p.T) : limit) - 128 * i;  // rows beyond get no gradient
  const int r = threadIdx.x & 127;
  if (r < rows) {
    const int quarter = r >> 5;
    const int qrows = min(rows - 32 * quarter, 32);
    const float4* src = reinterpret_cast<const float4*>(p.acc + (int64_t)bc * p.acc_sb + (int64_t)h * p.acc_sh +
                                                        (int64_t)(tq0 + 128 * i + 32 * quarter) * D);
    if (r < live) {
#pragma unroll 8
      for (int c = threadIdx.x >> 7; c < D / 4; c += 2) {
        const float4 a = __ldg(src + acc_piece(qrows, c, r & 31) / 4);
        *reinterpret_cast<uint2*>(tile + r * kRowBytes + 8 * c) = make_uint2(pack2<kBF16>(a.x * p.scale, a.y * p.scale), pack2<kBF16>(a.z * p.scale, a.w * p.scale));
      }
    } else {  // (the accumulator may not have been filled there, see sigattn_dq_fill_kernel)
#pragma unroll 8
      for (int c = threadIdx.x >> 7; c < D / 4; c += 2) *reinterpret_cast<uint2*>(tile + r * kRowBytes + 8 * c) = make_uint2(0u, 0u);
    }
  }
  __syncthreads();
  uint8_t* out = reinterpret_cast<uint8_t*>(p.dq) + 2 * ((int64_t)bc * p.sb + (int64_t)h * p.sh + (int64_t)(tq0 + 128 * i) * p.st);
  constexpr int kLanes = D / 8;  // 16-byte pieces of a row
  const int piece = threadIdx.x % kLanes;
  if (8 * piece >= p.d_cols) return;
  for (int row = threadIdx.x / kLanes; row < rows; row += 256 / kLanes)
    *reinterpret_cast<uint4*>(out + 2 * (int64_t)row * p.st + 16 * piece) =
        *reinterpret_cast<const uint4*>(tile + row * kRowBytes + 16 * piece);
}

}  // namespace sigattn
