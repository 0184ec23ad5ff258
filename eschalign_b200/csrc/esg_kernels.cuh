// esg_kernels.cuh -- device code of the B200 panel scorer (sm_100a).
//
// The kernels, in the order a batch launches them:
//
//   k2_batched   the product: every (query, reference pair) of the panel in
//                16-bit lanes.  One warp is a 32-lane systolic array: each
//                lane holds a 16-, 28- or 32-row stripe of one query (two
//                state words and the row's score-record address in
//                registers) and walks the columns of a reference pair; the
//                stripe's bottom row goes to the next lane by shuffle, so no
//                DP state ever leaves the register file.  The two 16-bit
//                halves of every register are two references (a
//                length-sorted pair).  Substitution is one shared-memory load
//                from the lane's per-column score record; the recurrence is
//                three DPX instructions plus two adds on the FMA pipe.  The
//                argmax / tie / XS reduction is folded in per query, online,
//                in shared memory.
//                Pairs that may have left int16 are flagged and their query
//                is re-scored by the int32 kernel.
//   k3_lanes     the exact int32 path: the recurrence of
//                crates/eschalign/src/scalar.rs:120-163 on chains of lanes
//                (28- or 32-row stripes, bottom rows passed by shuffle, several
//                references a warp for short queries); what k2 cannot take
//                or flags.  With one lane a chain it is the one-thread-per-
//                pair comparison arm.
//   k4_rows      per-query reduction of k3's rows (mapper.rs:444-472).
//   k5_merge     per read: forward and reverse-complement query states
//                merged into the read's result (k5_merge_chunks: straight
//                from the panel chunks' states).
//   k6_pairs     paired batches: per pair, the (reference, template strand)
//                candidates of crates/eschalign/src/mapper/pair.rs:195-234
//                ranked from the four mate rows (one warp per pair).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace esg {

constexpr int kMaxStripes = 32;       // a query spans at most one warp (k2)
constexpr int kNeg16 = -31500;        // int16 stand-in for -infinity (biased domain)
constexpr int kBiasLocal = 2048;      // local: H + B >= B >= |o|, |e|
constexpr int kBiasSemiGlobal = -16384;  // semi-global: H + B < 0 while |H| < 12000
constexpr int kNeg32 = -(1 << 29);    // int32 stand-in for -infinity, i32::MIN / 4 (scalar.rs:42)
// k2 CTA shape: 4 warps, 4 resident CTAs per SM (16 warps, <= 128
// registers; 3 for 28- and 32-row stripes).  Measured on B200 on the C2
// workload (reads of ~110 nt x 164 references, both strands):
//   ESG_K2_WARPS / ESG_K2_MIN_BLOCKS  CTA shape (4 x 4 beat 4 x 5 at 96
//       registers, and 8 warps x 2 CTAs)
//   ESG_K2_R32_BLOCKS  resident CTAs of 28- and 32-row stripes (3; at 4 they
//       spill 124-212 bytes and lose 2-5 %, at 2 -4.6 %)
#ifndef ESG_K2_WARPS
#define ESG_K2_WARPS 4
#endif
#ifndef ESG_K2_MIN_BLOCKS
#define ESG_K2_MIN_BLOCKS 4
#endif
#ifndef ESG_K2_R32_BLOCKS
#define ESG_K2_R32_BLOCKS 3
#endif
constexpr int kK2Warps = ESG_K2_WARPS;  // warps per k2 CTA
constexpr int kK2Threads = kK2Warps * 32;
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kNoRef = 0xffffffffu;
constexpr uint32_t kMaxCap = 32;       // largest tie capacity (ESG_MAX_TIE_CAPACITY)
// per-thread shared words of the column score record (one per row code
// 0-5), word c of thread t at c * kK2Threads + t: every thread in its own bank
constexpr int kScrWords = 6;
constexpr uint32_t kScrStride = (uint32_t)kK2Threads * 4;  // bytes between code words
// What the 16-bit halves of k2's registers hold (see pair_pass).
enum K2Lanes {
  kLanesInt,      // biased int16
  kLanesChecked,  // the same, semi-global, every cell watched for an overflow
  kLanesHalf,     // local: unbiased whole numbers 0..2047 as f16 subnormals
};
constexpr int kHalfMax = 2047;           // largest score kLanesHalf holds exactly
constexpr uint32_t kHalfOne = 0x3c003c00u;  // 1.0 in both halves
// Unroll of k2's unchecked column loop.  Unrolled once, the loop spends up to
// 1.4 register moves a cell pair (of 7.9 instructions) on the rotated state;
// unrolled past about 16 KB of code it outruns the instruction cache.  Swept
// 1-8 on B200, 150 000 C2 reads on one shape: local f16, 32 rows 133 / 121 /
// 125 / 122 ms at 1 / 2 / 3 / 4; semi-global, 28 + 32 rows 115 / 114 / 115 at 2 /
// 3 / 4; reading the panel through L2, semi-global 183 at 3, 181 at 5; int16
// local 28 + 32 rows 138 / 128 / 130 at 1 / 2 / 3; long queries 53.5 / 63 /
// 80 at 2 / 4 / 6 (two stripe heights share the cache).
template <int R, bool kSmem, bool kLong>
__host__ __device__ constexpr int steady_unroll(bool local, int lanes) {
  if (kLong) return 2;
  if (R == 8) return 4;
  if (lanes == kLanesHalf) return R == 16 ? 3 : kSmem ? 2 : 4;
  if (!local) return R == 16 || kSmem ? 3 : 5;
  return R == 16 ? 8 : kSmem ? 2 : 4;
}

// error bits in counters[2]
constexpr uint32_t kErrPanelWait = 1u;
constexpr uint32_t kErrRedoOverflow = 2u;

// query-state flags (device side, mirrored into esg_read_result.flags)
constexpr int kQRedo = 8;       // k2 flagged a pair; the query is re-scored by k3
constexpr int kQRescored = 4;   // == ESG_RESULT_RESCORED32

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v));
}
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// a * b + c as a 32-bit IMAD, which issues to the FMA pipe and so keeps the
// integer ALU free for the DPX ops
__device__ __forceinline__ uint32_t mad_lo(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// max(a + b, 0) and a + b per f16 half, on the FMA pipe.  Whole numbers n
// with |n| <= 2047 are kept as n * 2^-24 (sign and magnitude n; exact sums),
// so a result >= 0 is the integer n itself to the integer min / max ops.
__device__ __forceinline__ uint32_t add_relu_f16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(kHalfOne), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t add_f16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// the whole number n (|n| <= 1023) as a pair of f16 subnormals
__host__ __device__ __forceinline__ uint32_t half_pair(int n) {
  return (n < 0 ? 0x8000u | (uint32_t)(-n) : (uint32_t)n) * 0x10001u;
}
__device__ __forceinline__ uint32_t max16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ int lo16(uint32_t v) { return (int)(int16_t)(v & 0xffffu); }
__device__ __forceinline__ int hi16(uint32_t v) { return ((int)v) >> 16; }
__host__ __device__ __forceinline__ uint32_t pack16x2(int lo, int hi) {
  return (uint32_t)(uint16_t)(int16_t)lo | ((uint32_t)(uint16_t)(int16_t)hi << 16);
}

// Online reduction of one query's candidates (mapper.rs:444-472): best, XS,
// n_tied counted in full, and the `cap` smallest tie candidates in order.
// Candidates may arrive in any order; the result does not depend on it.
// slot = {best, suboptimal, n_tied, flags}; ties = cap entries.
__device__ __forceinline__ void slot_add(int* slot, uint32_t* ties, uint32_t cap, uint32_t idx,
                                         int score) {
  const int best = slot[0];
  if (score > best) {
    if (slot[2] > 0) slot[1] = max(slot[1], best);
    slot[0] = score;
    slot[2] = 1;
    ties[0] = idx;
  } else if (score == best) {
    const uint32_t n = (uint32_t)slot[2];
    slot[2] = (int)(n + 1);
    const uint32_t listed = n < cap ? n : cap;
    if (listed < cap || idx < ties[cap - 1]) {
      uint32_t pos = listed < cap ? listed : cap - 1;
      while (pos > 0 && ties[pos - 1] > idx) {
        ties[pos] = ties[pos - 1];
        --pos;
      }
      ties[pos] = idx;
    }
  } else {
    slot[1] = max(slot[1], score);
  }
}

// ---------------------------------------------------------------- k2
struct K2Params {
  // panel blob: n_pairs uint4 {sel offset, mA | mB << 16, refA, refB} then the
  // 16-bit PRMT selectors of every pair's columns
  const uint4* blob;
  uint32_t blob_bytes;   // multiple of 16
  uint32_t n_pairs;
  uint32_t sel_base;     // uint16 index of the first selector in the blob
  // reads (codes 0..4); query q < n_reads is read q forward, else the
  // reverse complement of read q - n_reads
  const uint8_t* codes;
  const uint64_t* off;
  const uint32_t* len;
  uint32_t n_reads;
  // work tiles: tasks[t] = {start in order[], count | smax << 16}
  const uint32_t* order;
  const uint2* tasks;
  uint32_t n_tasks;
  uint32_t* counters;    // [1] redo count, [2] error bits (and the task counters)
  uint32_t* task_counter;  // this launch's task counter
  // outputs
  int4* qhead;           // per query {best, suboptimal, n_tied, flags}
  uint32_t* qties;       // per query cap candidates
  int32_t* rows;         // optional [q * n_refs + r]
  uint32_t n_refs;
  uint32_t* redo_list;   // k3 list; redo entries go after redo_base
  uint32_t redo_base;
  uint32_t redo_cap;
  // panel chunks: with n_chunks > 1 a task is (tile, chunk), the chunk's
  // reference pairs are chunk_lo[c] .. chunk_lo[c + 1], and each query's
  // partial state goes to part_head / part_ties [q * n_chunks + c] for
  // k2_merge_chunks; with n_chunks == 1 a task is a tile over every pair
  uint32_t n_chunks;
  const uint32_t* chunk_lo;
  int4* part_head;
  uint32_t* part_ties;
  // scoring, pre-shifted by the gap open (see k2_batched)
  uint32_t tab_a[6];
  uint32_t tab_b[6];
  uint32_t rec2;         // kLanesHalf: added to a table's score to give s (see pair_pass)
  int32_t borrow;        // kLanesChecked: some s - o is negative
  uint32_t e2;           // e in both halves
  int32_t o, e;
  int32_t bias;          // value bias of the int16 lanes
  uint32_t one;          // the constant 1 (a multiplier the compiler cannot fold)
  uint2* lbuf;           // long queries: per-warp column buffer (G, F), lbuf_cols each
  uint32_t lbuf_cols;
  int32_t sat;           // local: a best (unbiased) at or above this may have wrapped
  uint32_t cap;
};

// Bounded wait on an mbarrier phase (a TMA bulk copy's completion).  Gives
// up after 2^26 polls, setting an error bit the host reads.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, uint32_t* err) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(bar);
  // 2^26 polls; past them the thread that issued the copies (thread 0)
  // keeps polling up to 2^24 more so that its copies in flight land before
  // the CTA's shared memory is released
  const uint32_t limit = (1u << 26) + (threadIdx.x == 0 ? (1u << 24) : 0u);
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) {
      if (it < (1u << 26)) return true;
      break;  // landed only in thread 0's extra polls: still a timeout
    }
  }
  atomicOr(err, kErrPanelWait);
  return false;
}

// Stage the panel blob into shared memory with TMA bulk copies, each CTA
// its own: one thread arms an mbarrier with the byte count and issues
// cp.async.bulk in chunks; every thread waits on the phase.
__device__ __forceinline__ bool stage_panel(void* smem, const void* gsrc, uint32_t bytes,
                                            uint64_t* bar, uint32_t* err) {
  const uint32_t bar_a = (uint32_t)__cvta_generic_to_shared(bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a), "r"(bytes)
                 : "memory");
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    const char* src = (const char*)gsrc;
    constexpr uint32_t kChunk = 32768;
    for (uint32_t at = 0; at < bytes; at += kChunk) {
      const uint32_t n = (bytes - at) < kChunk ? (bytes - at) : kChunk;
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              dst + at),
          "l"(src + at), "r"(n), "r"(bar_a)
          : "memory");
    }
  }
  const bool ok = mbar_wait(bar, 0, err);
  // One decision for the whole CTA: a thread that gave up and one that saw
  // the phase flip must not part ways (the survivors' warp-wide shuffles
  // would then run with exited lanes).
  return __syncthreads_and(ok) != 0;
}

// One systolic pass of a warp over the columns of one reference pair, two
// references per register (low half: the longer one of the pair, high half:
// the shorter one).
//
// What bounds it is the integer ALU (every DPX instruction, PRMT and plain
// MAX takes the same 64-lane-a-clock issue port; the FMA pipe beside it is
// as wide), and behind it the F chain down a stripe's rows (three dependent
// instructions a row), which 12-16 warps an SM hide.  So a cell pair is
// written for the fewest ALU instructions -- E, F and H, one DPX instruction
// each, and half a VIMNMX3 for the running best where there is one -- with
// both remaining adds (the diagonal term, G = H + open) on the FMA pipe:
//
//   kLanesHalf (local, scores up to 2047)  Halves hold H, E, F >= 0 as whole
//     numbers, which are also the f16 subnormals n * 2^-24: sums of those are
//     exact and HFMA2.relu gives max(a + b, 0), the local floor, for free.
//     d = relu(H_diag + s), H = max3(d, E, F), G = relu(H + o),
//     E = max(E + e, G), F = max(F + e, G).  E and F floored at 0 change no H
//     (the floor is 0).  3.5 ALU.  g[r] holds d of the row's next column (its
//     record is written a column ahead), so that nothing old outlives the
//     update and the registers need no rotation.  The best is taken over d:
//     E and F never exceed an earlier H.
//   kLanesInt, semi-global  Halves hold value + B (B = -16384) in int16.
//     d = G_diag + (s - o) and G = H + o are 32-bit IMADs, exact in both
//     halves: the low half's sums stay negative (static bound, or watched, see
//     kLanesChecked), so a negative addend's carry out is the rule, cancelled
//     by o * 65537 (and, where some s - o is negative, by a record word built
//     with one less above it: kLanesChecked alone spends the instructions on
//     that), and the high half's carry is discarded.  Padding columns (garbage
//     that may wrap) are only ever in the high half.  3 ALU.  g[r] is d of the
//     row's next column in the unchecked loop, as above, and G of its last one
//     in the checked one, which takes the columns' ends from it.
//   kLanesInt, local  B = 2048; d takes the ALU (max(G_diag + (s - o), E)) as
//     nothing else gives the floor.  4.5 ALU.  For scores past 2047.
//
// C2 local, 150 000 reads: 115.8 ms; with 4.5 ALU on 16-row stripes (the best
// of before) 137.5.  Semi-global 107.9 against 130.7 (5 ALU, 32 rows).
//
// Score records: at each column the lane writes the column's score word for
// each read code (PRMT of that code's tables by the column's selector, which
// picks a byte per half and sign-extends it; codes 0-3, and the wildcard code
// 4 when the warp holds a wildcard row) to its own record in shared memory,
// then each row loads its code's word: ta[r] is that word's address.  Tables
// {tb, ta}: byte x is s(c, x) - o for reference code x = 0..3, 4 (wildcard),
// and a padding column's score at x = 5; for kLanesHalf s + off (0..127, off
// taken off again by P.rec2, padding columns 0).  The padding code's word is a
// constant.  The words of one code are kK2Threads apart, so every lane reads
// and writes its own bank.
//
// The lane with skew k works on column j = t - k at step t; its top input
// (G and F of the row above) is the previous lane's bottom output of step
// t-1, fetched by shuffle.  A query's first lane takes the border instead.
// In a long pass (kLong), lane 0 takes its top input from `buf` (the bottom
// row of the previous pass) when `from_buf`, and lane 31 writes its bottom
// row to `buf` when `to_buf`: lane 0 reads column j at step j, lane 31
// overwrites it at step j + 31, so one buffer serves every pass.
//
// Returns, per lane, the pass's local best (H + B) or semi-global last-column
// maximum (G, the short half's taken at its own end) in `v`, and the
// semi-global maximum of the last row over the lane's columns (H + B) in `lr`.
struct PassConst {
  uint32_t g0, f0, neg2, e2, o32, one, bias2;
};

// A column's 16-bit PRMT selector: an explicit shared-memory load when the
// panel is staged in shared memory, a read-only global load otherwise.
template <bool kSmem>
__device__ __forceinline__ uint32_t load_sel(const uint16_t* sp, int j) {
  if constexpr (kSmem) {
    uint16_t v;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(sp + j);
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
  } else {
    return __ldg(sp + j);
  }
}

template <int V>
struct IntConst {
  static constexpr int value = V;
};

template <int R, bool kLocal, bool kLong, bool kSmem, int kLanes>
__device__ __forceinline__ void pair_pass(const K2Params& P, uint32_t scr, bool wild,
                                          const uint32_t (&ta)[R], int skew,
                                          bool active_lane, bool first, uint32_t padmask, int m,
                                          int jshort, const uint16_t* __restrict__ sp, int steps,
                                          const PassConst& K, uint2* buf, bool from_buf,
                                          bool to_buf, uint32_t& v, uint32_t& lr, uint32_t& am) {
  const int lane = threadIdx.x & 31;
  constexpr bool kCheck = kLanes == kLanesChecked;
  constexpr bool kHalf = kLanes == kLanesHalf;
  constexpr bool kPre = kLocal && (kSmem || !kHalf);
  // padding rows: local, -128 (kLanesHalf: 0) against every column, so H
  // stays 0 under the floor; semi-global, s = 0 (H = 0 exactly against real
  // columns; the short half's columns past its end are never read)
  st_shared_u32(scr + 5 * kScrStride,
                kHalf ? 0u : kLocal ? 0xff80ff80u : pack16x2(-P.o, -P.o));
  uint32_t g[R], ev[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    g[r] = K.g0;
    ev[r] = K.f0;
  }
  uint32_t gdc = K.g0;  // G of the row above, previous column
  uint32_t gbot = K.g0, fbot = K.f0;
  // local: max H + B over this lane's cells; checked semi-global: the same
  // without the floor (the short half's taken at its own end)
  uint32_t best = kLocal ? K.bias2 : K.neg2, s_best = K.neg2;
  uint32_t lastrow = K.neg2;               // semi-global: max H + B of the last row
  uint32_t s_col = K.neg2, s_last = K.neg2;  // semi-global short-half snapshot
  // inactive lanes of a tile sit at a skew no step reaches; only the long
  // path needs the per-lane bound (its lanes past the query's last stripe)
  const int mlim = (kLong && !active_lane) ? 0 : m;
  // (kPre: +2 % where the panel is in shared memory)
  uint32_t seln = kPre ? load_sel<kSmem>(sp, 0) : 0u;

  // a column's score record: one word per read code, in this thread's own
  // bank, read back per row (wildcard rows only when the warp has some)
  auto record = [&](uint32_t sel) {
    auto word = [&](int c) {
      uint32_t w = prmt(P.tab_a[c], P.tab_b[c], sel);
      if constexpr (kHalf) w = add_f16x2(w, P.rec2);
      if constexpr (kCheck)
        if (P.borrow) w -= (w << 1) & 0x10000u;
      st_shared_u32(scr + c * kScrStride, w);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) word(c);
    if (wild) word(4);
  };
  if constexpr (kHalf) {
    // column 0's diagonal terms, from the zero border
    record(kPre ? seln : load_sel<kSmem>(sp, 0));
#pragma unroll
    for (int r = 0; r < R; ++r) g[r] = add_relu_f16x2(K.g0, ld_shared_u32(ta[r]));
    if constexpr (kPre) seln = load_sel<kSmem>(sp, 1);
  }
  uint2 bnext = make_uint2(0u, 0u);
  if constexpr (kLong)
    if (from_buf && lane == 0) bnext = buf[0];
  // One column of the lane's stripe, given the top input (G, F of the row
  // above at this column).
  auto column = [&](auto snap, int j, uint32_t gt, uint32_t ft) {
    constexpr bool kSnap = decltype(snap)::value != 0;
    if constexpr (kLong) {
      if (from_buf && lane == 0) {
        gt = bnext.x;
        ft = bnext.y;
        bnext = buf[min(j + 1, m - 1)];  // a column ahead: its latency is off the chain
      }
    }
    // columns of a lane come in order: with kPre the next one's selector is
    // loaded a column ahead
    constexpr int kAhead = kHalf || (!kLocal && !kSnap) ? 1 : 0;
    uint32_t sel;
    if constexpr (kPre) {
      sel = seln;
      seln = load_sel<kSmem>(sp, j + kAhead + 1);
    } else {
      sel = load_sel<kSmem>(sp, j + kAhead);
    }
    record(sel);
    if constexpr (kHalf || (!kLocal && !kSnap)) {
      // g[r]: the row's diagonal term at this column, then at the next
      uint32_t f = ft, up = gt, prev = 0, h = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t d = g[r];
        h = __vimax3_s16x2(d, ev[r], f);
        if constexpr (kLocal || kCheck) {
          const uint32_t x = kLocal ? d : h;
          if (r & 1)
            best = __vimax3_s16x2(best, prev, x);
          else
            prev = x;
        }
        const uint32_t sc = ld_shared_u32(ta[r]);
        g[r] = kHalf ? add_relu_f16x2(up, sc) : mad_lo(up, K.one, sc);
        const uint32_t gr = kHalf ? add_relu_f16x2(h, K.o32) : mad_lo(h, K.one, K.o32);
        ev[r] = __viaddmax_s16x2(ev[r], K.e2, gr);
        f = __viaddmax_s16x2(f, K.e2, gr);
        up = kHalf ? h : gr;
      }
      gbot = up;
      fbot = f;
      if constexpr (!kLocal) lastrow = max16x2(lastrow, h);
      if constexpr (kLong) {
        if (to_buf && lane == 31) buf[j] = make_uint2(gbot, fbot);
      }
      return;
    }
    uint32_t f = ft, h15 = 0, hprev = 0, gd = gdc;
    gdc = gt;
    if constexpr (kLocal) {
      uint32_t gup = gt;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        ev[r] = __viaddmax_s16x2(ev[r], K.e2, g[r]);
        f = __viaddmax_s16x2(f, K.e2, gup);
        const uint32_t h1 = __viaddmax_s16x2(gd, ld_shared_u32(ta[r]), ev[r]);
        gd = g[r];
        const uint32_t h = __vimax3_s16x2(h1, f, K.bias2);
        if (r & 1)
          best = __vimax3_s16x2(best, hprev, h);
        else
          hprev = h;
        g[r] = mad_lo(h, K.one, K.o32);
        gup = g[r];
      }
    } else {
      // (a row's diagonal term is taken before the row above overwrites the G
      // it reads)
      auto diag = [&](int r) {
        return mad_lo(r ? g[r ? r - 1 : 0] : gd, K.one, ld_shared_u32(ta[r]));
      };
      uint32_t dn = diag(0);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t d = dn;
        if (r + 1 < R) dn = diag(r + 1 < R ? r + 1 : r);
        const uint32_t h = __vimax3_s16x2(d, ev[r], f);
        if constexpr (kCheck) {
          if (r & 1)
            best = __vimax3_s16x2(best, hprev, h);
          else
            hprev = h;
        }
        g[r] = mad_lo(h, K.one, K.o32);
        ev[r] = __viaddmax_s16x2(ev[r], K.e2, g[r]);
        f = __viaddmax_s16x2(f, K.e2, g[r]);
        if (r == R - 1) h15 = h;
      }
    }
    gbot = g[R - 1];
    fbot = f;
    if constexpr (kLong) {
      if (to_buf && lane == 31) buf[j] = make_uint2(gbot, fbot);
    }
    if constexpr (!kLocal) {
      lastrow = max16x2(lastrow, h15);
      if (kSnap && j == jshort) {
        // the short half's last column, padding rows left out.  Padding
        // rows hold G = o + B exactly (H = 0), so a maximum above that is a
        // read row's and the unmasked maximum stands; only a maximum equal
        // to it takes the masked one.  (Masking every time kept the pad
        // mask's selects live across the column loop: 40-52 bytes of spill
        // in the 32-row kernel.)
        uint32_t cm = K.neg2;
#pragma unroll
        for (int r = 0; r < R; ++r) cm = max16x2(cm, g[r]);
        if (padmask && (cm >> 16) == (K.g0 >> 16)) {
          cm = K.neg2;
#pragma unroll
          for (int r = 0; r < R; ++r) cm = max16x2(cm, ((padmask >> r) & 1u) ? K.neg2 : g[r]);
        }
        s_col = cm;
        s_last = lastrow;
        if constexpr (kCheck) s_best = best;
      }
    }
  };
  // The top input: the previous lane's bottom row of the previous step, or
  // the border for a query's first lane.
  auto top = [&](uint32_t& gt, uint32_t& ft) {
    gt = __shfl_up_sync(kFull, gbot, 1);
    ft = __shfl_up_sync(kFull, fbot, 1);
    if (first) {
      gt = K.g0;
      ft = K.f0;
    }
  };

  int t = 0;
  // Steps fill .. m - 1, where fill = steps - m is the largest skew, have
  // every lane of the task's queries inside the pair's columns: they run
  // without the column check, and in semi-global mode (up to the first lane's
  // snapshot column) without the snapshot, whose code would fill the
  // instruction cache.  Lanes past the queries take skew 0 there (columns in
  // range, values nobody reads: only later lanes, also past the queries, see
  // them, and a pass's results are taken from the queries' own lanes; a long
  // query's local best takes padding rows in too, which add nothing to H).
  const int fill = steps - m;
  const int full = (kLocal || jshort < 0) ? m : jshort;
  if (fill < full) {
#pragma unroll 1
    for (; t < fill; ++t) {
      uint32_t gt, ft;
      top(gt, ft);
      const int j = t - skew;
      if ((unsigned)j < (unsigned)mlim) column(IntConst<kLocal ? 0 : 1>{}, j, gt, ft);
    }
    const int sk = active_lane ? skew : 0;
    if constexpr (!kLocal) {
      // from G of the last column to the diagonal terms of the next
      record(load_sel<kSmem>(sp, t - sk));
#pragma unroll
      for (int r = R - 1; r >= 0; --r)
        g[r] = mad_lo(r ? g[r ? r - 1 : 0] : gdc, K.one, ld_shared_u32(ta[r]));
    }
    constexpr int kUnroll = steady_unroll<R, kSmem, kLong>(kLocal, kLanes);
#pragma unroll kUnroll
    for (; t < full; ++t) {
      uint32_t gt, ft;
      top(gt, ft);
      column(IntConst<0>{}, t - sk, gt, ft);
    }
    if constexpr (!kLocal) {
      // and back: the next column's record is in place
      gdc = g[0] - ld_shared_u32(ta[0]);
#pragma unroll
      for (int r = 0; r + 1 < R; ++r) g[r] = g[r + 1 < R ? r + 1 : r] - ld_shared_u32(ta[r + 1 < R ? r + 1 : r]);
      g[R - 1] = gbot;
    }
  }
#pragma unroll 1
  for (; t < steps; ++t) {
    uint32_t gt, ft;
    top(gt, ft);
    const int j = t - skew;
    if ((unsigned)j < (unsigned)mlim) column(IntConst<1>{}, j, gt, ft);
  }
  am = K.neg2;
  if constexpr (kLocal) {
    v = best;
    lr = 0;
  } else {
    if constexpr (kCheck)
      am = active_lane ? (jshort >= 0 ? (best & 0xffffu) | (s_best & 0xffff0000u) : best) : K.neg2;
    uint32_t cm = K.neg2;
#pragma unroll
    for (int r = 0; r < R; ++r) cm = max16x2(cm, ((padmask >> r) & 1u) ? K.neg2 : g[r]);
    if (jshort >= 0) {
      // the short (high) half's last column and last row, taken at its end
      cm = (cm & 0xffffu) | (s_col & 0xffff0000u);
      lastrow = (lastrow & 0xffffu) | (s_last & 0xffff0000u);
    }
    v = active_lane ? cm : K.neg2;
    lr = lastrow;
  }
}

// Record addresses of stripe `s` of a query (n codes at q, reverse complement
// if rc): row r is read row i = R s + r - pad; rows before the read are
// padding.  Returns whether any lane of the warp has a wildcard row.
template <int R>
__device__ __forceinline__ bool row_records(const uint8_t* q, uint32_t n, bool rc, bool valid,
                                            int s, int pad, uint32_t scr, uint32_t (&ta)[R]) {
  bool wild = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = s * R + r - pad;
    uint32_t c = 5;  // padding row
    if (valid && i >= 0) {
      uint32_t x = rc ? q[n - 1 - i] : q[i];
      x = x > 4 ? 4 : x;
      c = (rc && x < 4) ? 3 - x : x;
    }
    wild |= c == 4;
    ta[r] = scr + c * kScrStride;  // the row code's word in the column record
  }
  return __any_sync(kFull, wild);
}

// The last lane of a query folds one reference pair's two scores into the
// query's slot (and its rows, when asked for).  A pair that may have left
// the int16 lanes flags its query for the int32 re-score: in local mode a
// best at or above P.sat; in checked semi-global mode any cell with
// H + B >= 0 (H >= 16384), where G's IMAD may borrow wrongly (see
// pair_pass) -- the first such cell is itself exact, its inputs being below
// the mark, so the maximum over every cell, `am`, catches it.
template <bool kLocal, int kLanes>
__device__ __forceinline__ void fold_pair(const K2Params& P, int* slot, uint32_t* sties,
                                          uint32_t cap, uint4 pm, int mB, bool rc, uint32_t qid,
                                          uint32_t v, uint32_t lr, uint32_t am, int bias) {
  int scA, scB;
  if constexpr (kLocal) {
    scA = lo16(v) - bias;
    scB = hi16(v) - bias;
    if constexpr (kLanes == kLanesInt)
      if (scA >= P.sat || (mB > 0 && scB >= P.sat)) slot[3] |= kQRedo;
  } else {
    scA = max(lo16(v) - P.o, lo16(lr)) - bias;
    scB = max(hi16(v) - P.o, hi16(lr)) - bias;
    if constexpr (kLanes == kLanesChecked)
      if (lo16(am) >= 0 || (mB > 0 && hi16(am) >= 0)) slot[3] |= kQRedo;
  }
  const uint32_t rbit = rc ? 1u : 0u;
  slot_add(slot, sties, cap, (pm.z << 1) | rbit, scA);
  if (P.rows) P.rows[(size_t)qid * P.n_refs + pm.z] = scA;
  if (pm.w != kNoRef) {
    slot_add(slot, sties, cap, (pm.w << 1) | rbit, scB);
    if (P.rows) P.rows[(size_t)qid * P.n_refs + pm.w] = scB;
  }
}

// A query's state at the end of a task: its final state (and a re-score
// request if it may have wrapped), or with panel chunks its partial state
// for k2_merge_chunks.
__device__ __forceinline__ void flush_query(const K2Params& P, uint32_t qid, uint32_t chunk,
                                            const int* slot, const uint32_t* sties,
                                            uint32_t cap) {
  const int fl = slot[3];
  const uint32_t nl = min((uint32_t)slot[2], cap);
  if (P.n_chunks > 1) {
    const size_t at = (size_t)qid * P.n_chunks + chunk;
    P.part_head[at] = make_int4(slot[0], slot[1], slot[2], fl);
    for (uint32_t k = 0; k < nl; ++k) P.part_ties[at * cap + k] = sties[k];
    return;
  }
  P.qhead[qid] = make_int4(slot[0], slot[1], slot[2], fl);
  for (uint32_t k = 0; k < nl; ++k) P.qties[(size_t)qid * cap + k] = sties[k];
  if (fl & kQRedo) {
    const uint32_t at = atomicAdd(&P.counters[1], 1u);
    if (at < P.redo_cap)
      P.redo_list[P.redo_base + at] = qid;
    else
      atomicOr(&P.counters[2], kErrRedoOverflow);
  }
}

// One warp, one task at a time, tasks pulled from an atomic counter.
// kLong = false takes tiles of up to 32 queries whose stripes fill the warp's
// lanes (a query of n rows takes S = ceil(n / R) lanes), scored in one pass
// per reference pair; kLong = true takes one long query (S > 32) per task,
// scored in ceil(S / 32) passes per pair chained through a per-warp column
// buffer in global memory, the last one on 16-row stripes when that is enough
// (half the lanes' rows would be idle: 600 reads of 1100-5000 nt against 48
// references, with the unrolled loop, 74.6 -> 47.1 ms semi-global, 75.0 ->
// 55.2 local).  Instantiations of their own keep the register allocation of
// the short-read path free of the long path's state.
// Stripes are aligned so the read's last row is the last row of its last
// stripe; the rows before the read's first row score 0 against every real
// column and hold H = 0 exactly, the top border the first real row needs.
template <int R, bool kLocal, bool kSmemPanel, bool kLong, int kLanes>
__global__ void __launch_bounds__(kK2Threads, R > 16 ? ESG_K2_R32_BLOCKS : ESG_K2_MIN_BLOCKS)
    k2_batched(const K2Params P) {
  constexpr bool kCheck = kLanes == kLanesChecked;
  constexpr bool kHalf = kLanes == kLanesHalf;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t panel_bar;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const uint32_t cap = P.cap;

  const uint4* pairs;
  const uint16_t* sels;
  int* slots;
  if constexpr (kSmemPanel) {
    if (!stage_panel(smem_raw, P.blob, P.blob_bytes, &panel_bar, &P.counters[2])) return;
    pairs = reinterpret_cast<const uint4*>(smem_raw);
    sels = reinterpret_cast<const uint16_t*>(smem_raw) + P.sel_base;
    slots = reinterpret_cast<int*>(smem_raw + P.blob_bytes);
  } else {
    pairs = P.blob;
    sels = reinterpret_cast<const uint16_t*>(P.blob) + P.sel_base;
    slots = reinterpret_cast<int*>(smem_raw);
  }
  // this lane's query slot: {best, suboptimal, n_tied, flags, ties[cap]}
  int* slot = slots + (size_t)(wib * 32 + lane) * (4 + cap);
  uint32_t* sties = reinterpret_cast<uint32_t*>(slot + 4);
  // column score records: word c * kK2Threads + thread (bank = lane)
  const uint32_t scr = (uint32_t)__cvta_generic_to_shared(slots + (size_t)kK2Threads * (4 + cap)) +
                       threadIdx.x * 4u;
  uint2* lbuf = P.lbuf ? P.lbuf + ((size_t)blockIdx.x * kK2Warps + wib) * P.lbuf_cols : nullptr;

  const int bias = P.bias;
  PassConst K;
  // a zero border cell's G (kLanesHalf: its H) and its E and F
  K.g0 = kHalf ? 0u : pack16x2(bias + P.o, bias + P.o);
  K.neg2 = kHalf ? 0u : pack16x2(kNeg16, kNeg16);
  // E of column 1 and F of row 1: semi-global, opened at the zero border;
  // int16 local takes them a cell later (its E and F are the last column's and
  // the row above's)
  K.f0 = kHalf || kLocal ? K.neg2 : K.g0;
  K.bias2 = pack16x2(bias, bias);  // H = 0 (the local floor)
  // + o in both halves: one 32-bit add, or one f16x2 add
  K.o32 = kHalf ? half_pair(P.o) : (uint32_t)(P.o * 65537);
  K.e2 = P.e2;
  K.one = P.one;  // 1, opaque to the compiler: keeps G's add an IMAD

  for (;;) {
    uint32_t task = 0;
    if (lane == 0) task = atomicAdd(P.task_counter, 1u);
    task = __shfl_sync(kFull, task, 0);
    if (task >= P.n_tasks) break;
    const uint32_t tile = P.n_chunks > 1 ? task / P.n_chunks : task;
    const uint32_t chunk = task - tile * P.n_chunks;
    const uint32_t p_lo = P.n_chunks > 1 ? P.chunk_lo[chunk] : 0u;
    const uint32_t p_hi = P.n_chunks > 1 ? P.chunk_lo[chunk + 1] : P.n_pairs;
    const uint2 tk = P.tasks[tile];
    const uint32_t count = tk.y & 0xffffu;
    const int smax = (int)(tk.y >> 16);

    if constexpr (kLong) {
      // ---------------- one long query, ceil(S / 32) passes per pair
      const uint32_t qid = P.order[tk.x];
      const bool rc = qid >= P.n_reads;
      const uint32_t rd = rc ? qid - P.n_reads : qid;
      const uint32_t n = P.len[rd];
      // passes of 32 R-row stripes; a last pass of at most 16 rows a lane
      // takes 16-row stripes
      const int passes = (smax + 31) / 32;
      const int before = (passes - 1) * 32 * R;  // rows of the passes before the last
      const bool narrow = (int)n - before <= 32 * 16;
      const int RL = narrow ? 16 : R;
      const int SL = ((int)n - before + RL - 1) / RL;  // stripes of the last pass
      const int pad = before + SL * RL - (int)n;
      const int owner = SL - 1;  // lane holding the last stripe
      const uint8_t* q = P.codes + P.off[rd];
      if (lane == owner) {
        slot[0] = INT32_MIN;
        slot[1] = INT32_MIN;
        slot[2] = 0;
        slot[3] = 0;
      }
      for (uint32_t p = p_lo; p < p_hi; ++p) {
        const uint4 pm = pairs[p];
        const int mA = (int)(pm.y & 0xffffu), mB = (int)(pm.y >> 16);  // mA >= mB
        const int jshort = (mB > 0 && mB < mA) ? mB - 1 : -1;
        const uint16_t* sp = sels + pm.x;
        uint32_t acc = kLocal ? K.bias2 : K.neg2, lr_last = K.neg2, amacc = K.neg2;
        auto run = [&](auto rows, int pass, bool last) {
          constexpr int RP = decltype(rows)::value;
          const int s = before / RP * (last ? 1 : 0) + (last ? 0 : pass * 32) + lane;
          const bool valid = !last || lane < SL;
          uint32_t ta[RP];
          const bool wild = row_records<RP>(q, n, rc, valid, s, pad, scr, ta);
          const uint32_t padmask = (s == 0) ? ((1u << pad) - 1u) : 0u;
          uint32_t v, lr, am;
          pair_pass<RP, kLocal, true, kSmemPanel, kLanes>(
              P, scr, wild, ta, lane, valid, s == 0, padmask, mA, jshort, sp, mA + 31, K, lbuf,
              pass > 0, !last, v, lr, am);
          acc = max16x2(acc, v);
          if constexpr (kCheck) amacc = max16x2(amacc, am);
          if (last) lr_last = lr;
          __syncwarp();  // the buffer's writes are visible to the next pass
        };
        for (int pass = 0; pass + 1 < passes; ++pass) run(IntConst<R>{}, pass, false);
        if (narrow)
          run(IntConst<16>{}, passes - 1, true);
        else
          run(IntConst<R>{}, passes - 1, true);
#pragma unroll
        for (int d = 16; d; d >>= 1) acc = max16x2(acc, __shfl_xor_sync(kFull, acc, d));
        if constexpr (kCheck) {
#pragma unroll
          for (int d = 16; d; d >>= 1) amacc = max16x2(amacc, __shfl_xor_sync(kFull, amacc, d));
        }
        if (lane == owner)
          fold_pair<kLocal, kLanes>(P, slot, sties, cap, pm, mB, rc, qid, acc, lr_last, amacc,
                                    bias);
      }
      if (lane == owner) flush_query(P, qid, chunk, slot, sties, cap);
      __syncwarp();
      continue;
    } else {
    // ---------------- up to 32 queries, one pass per pair
    uint32_t kq = 0, kn = 0, kS = 0;
    if ((uint32_t)lane < count) {
      kq = P.order[tk.x + lane];
      const uint32_t rd = kq < P.n_reads ? kq : kq - P.n_reads;
      kn = P.len[rd];
      kS = (kn + R - 1) / R;
    }
    uint32_t incl = kS;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += v;
    }
    uint32_t qid = 0, n = 0;
    int s = 1 << 20, S = 0;  // lanes past the task's queries never become active
    bool valid = false;
    for (uint32_t k = 0; k < count; ++k) {
      const uint32_t ek = __shfl_sync(kFull, incl, k);
      const uint32_t sk = __shfl_sync(kFull, kS, k);
      const uint32_t qk = __shfl_sync(kFull, kq, k);
      const uint32_t nk = __shfl_sync(kFull, kn, k);
      if ((uint32_t)lane >= ek - sk && (uint32_t)lane < ek) {
        qid = qk;
        n = nk;
        s = lane - (int)(ek - sk);
        S = (int)sk;
        valid = true;
      }
    }
    const bool first = valid ? (s == 0) : true;
    const bool last = valid && (s == S - 1);
    const int pad = valid ? S * R - (int)n : 0;
    const bool rc = qid >= P.n_reads;
    const uint32_t rd = rc ? qid - P.n_reads : qid;

    uint32_t ta[R];
    const bool wild =
        row_records<R>(valid ? P.codes + P.off[rd] : P.codes, n, rc, valid, s, pad, scr, ta);
    // rows of the read's top padding (first lane only): excluded from the
    // semi-global last-column maximum
    const uint32_t padmask = (valid && first) ? ((1u << pad) - 1u) : 0u;

    if (last) {
      slot[0] = INT32_MIN;
      slot[1] = INT32_MIN;
      slot[2] = 0;
      slot[3] = 0;
    }

    for (uint32_t p = p_lo; p < p_hi; ++p) {
      const uint4 pm = pairs[p];
      const int mA = (int)(pm.y & 0xffffu), mB = (int)(pm.y >> 16);  // mA >= mB
      const int jshort = (mB > 0 && mB < mA) ? mB - 1 : -1;
      uint32_t v, lr, am;
      pair_pass<R, kLocal, false, kSmemPanel, kLanes>(
          P, scr, wild, ta, s, valid, first, padmask, mA, jshort, sels + pm.x, mA + smax - 1, K,
          nullptr, false, false, v, lr, am);
      // per-query maximum, to the query's last lane
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t w = __shfl_up_sync(kFull, v, d);
        if (s >= d) v = max16x2(v, w);
        if constexpr (kCheck) {
          const uint32_t wa = __shfl_up_sync(kFull, am, d);
          if (s >= d) am = max16x2(am, wa);
        }
      }
      if (last) fold_pair<kLocal, kLanes>(P, slot, sties, cap, pm, mB, rc, qid, v, lr, am, bias);
    }

    // --- flush the query states of this task
    if (last) flush_query(P, qid, chunk, slot, sties, cap);
    __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- chunk merge
// The 32 smallest of two sorted lists of 32 (lane k holds a list's k-th
// smallest, kNoRef past its end), sorted: the lanewise minimum of one list
// and the other reversed is bitonic and holds them.
__device__ __forceinline__ uint32_t merge_lists(uint32_t a, uint32_t b, int lane) {
  uint32_t x = min(a, __shfl_sync(kFull, b, 31 - lane));
#pragma unroll
  for (int d = 16; d; d >>= 1) {
    const uint32_t y = __shfl_xor_sync(kFull, x, d);
    x = (lane & d) ? max(x, y) : min(x, y);
  }
  return x;
}

// One warp: a query's panel chunks' states (heads and tie lists of the query,
// n_chunks of them) into the state over their union (mapper.rs:444-472): the
// highest best, its ties counted in full, the best score outside them.  Lane
// k returns the k-th tie in candidate order.  The chunks go a lane each, so a
// small batch cut into a chunk per reference pair pays a few loads here, not
// a chain of them (one thread a query walked 20 chunks in about 25 us).
__device__ __forceinline__ int4 merge_chunks(const int4* head, const uint32_t* ties,
                                             uint32_t n_chunks, uint32_t cap, int lane,
                                             uint32_t& tie) {
  int best = INT32_MIN;
  for (uint32_t c = lane; c < n_chunks; c += 32) best = max(best, head[c].x);
  best = __reduce_max_sync(kFull, best);
  int sub = INT32_MIN;
  uint32_t n = 0, flags = 0;
  tie = kNoRef;
  for (uint32_t c0 = 0; c0 < n_chunks; c0 += 32) {
    const uint32_t c = c0 + lane;
    const int4 b = c < n_chunks ? head[c] : make_int4(INT32_MIN, INT32_MIN, 0, 0);
    const bool on = c < n_chunks && b.x == best;
    sub = max(sub, on ? b.y : b.x);
    n += on ? (uint32_t)b.z : 0u;
    flags |= (uint32_t)b.w;
    for (uint32_t m = __ballot_sync(kFull, on); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const uint32_t nl = min((uint32_t)__shfl_sync(kFull, b.z, src), cap);
      const uint32_t t = (uint32_t)lane < nl ? ties[(size_t)(c0 + src) * cap + lane] : kNoRef;
      tie = merge_lists(tie, t, lane);
    }
  }
  return make_int4(best, __reduce_max_sync(kFull, sub), (int)__reduce_add_sync(kFull, n),
                   (int)__reduce_or_sync(kFull, flags));
}

struct KMParams {
  const uint32_t* order;   // the queries k2 scored
  uint32_t n_order;
  uint32_t n_chunks;
  const int4* part_head;   // [q * n_chunks + c]
  const uint32_t* part_ties;
  int4* qhead;
  uint32_t* qties;
  uint32_t cap;
  uint32_t* counters;      // [1] redo count, [2] error bits
  uint32_t* redo_list;
  uint32_t redo_base;
  uint32_t redo_cap;
};

// One warp per query: its panel chunks' partial states merged, and a re-score
// request where any chunk may have wrapped.
static __global__ void __launch_bounds__(128) k2_merge_chunks(const KMParams P) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < P.n_order; i += warps) {
    const uint32_t q = P.order[i];
    const size_t base = (size_t)q * P.n_chunks;
    uint32_t tie;
    const int4 acc = merge_chunks(P.part_head + base, P.part_ties + base * P.cap, P.n_chunks,
                                  P.cap, lane, tie);
    if ((uint32_t)lane < P.cap) P.qties[(size_t)q * P.cap + lane] = tie;
    if (lane) continue;
    P.qhead[q] = acc;
    if (acc.w & kQRedo) {
      const uint32_t at = atomicAdd(&P.counters[1], 1u);
      if (at < P.redo_cap)
        P.redo_list[P.redo_base + at] = q;
      else
        atomicOr(&P.counters[2], kErrRedoOverflow);
    }
  }
}

// ---------------------------------------------------------------- k3
// k3_lanes: the exact int32 path.  It scores a list of queries against every
// reference of the panel and writes the rows (k4 reduces them).  The work
// unit is (query, a run of references); one warp takes one unit at a time.
//
// Lanes hold 28- or 32-row stripes of the query, whichever k3_cost says its
// length fills better.  A query of S stripes is scored
// against a reference by a chain of W = min(S, wmax) lanes: the lane at
// position w of the chain holds stripes w, W + w, 2W + w, ... in successive
// passes, walks the reference's columns one per step, lagging the lane
// before it by one step, and takes its top input (G and F of the row above)
// from that lane by shuffle.  The chain's first lane takes the zero border
// in the first pass and, in later passes, the bottom row the chain's last
// lane left in the warp's column buffer (global memory) in the pass before.
// A warp runs 32 / W chains side by side, one reference each, so short
// queries fill the warp with references instead of idle lanes.  wmax = 32 is
// the product setting; wmax = 1 makes every lane a chain of its own -- one
// thread per (query, reference) pair, the stripes' bottom row through the
// buffer -- the plain comparison arm.
//
// What bounds it is the integer ALU, so a cell takes the fewest DPX
// instructions: E, F and H one each (and half one for the local best), the
// diagonal term G_diag + (s - o) and G = H + o as IMADs on the FMA pipe.
// Local mode's floor comes with E (VIADDMNMX.RELU: E >= 0 changes no H), and
// its g[r] holds the diagonal term of the row's next column.  The substitution
// s - o comes from the lane's per-column record in shared memory (word c = the
// score of read code c against this column, one 16-byte table load and four
// stores per column), one load per cell.  The query is padded at the top to
// whole stripes with rows that score 0, which hold H = 0 exactly -- the top
// border -- and are left out of the semi-global last-column maximum.
// Columns that every chain is inside run without the column check; unrolled
// twice that loop measured 121 ms against 108 (both stripe heights' loops
// share the instruction cache).  60 000 C2 reads x 164 references, both
// strands: 143 -> 108 ms local, 150 -> 105 semi-global, one thread per pair
// 154 -> 116, against four ALU-bound DPX instructions on 16-row stripes.
constexpr int kK3Warps = 4;
constexpr int kK3Threads = kK3Warps * 32;
constexpr uint32_t kK3Stride = (uint32_t)kK3Threads * 4;  // bytes between record words

struct K3Params {
  // queries: list entry p is query list[p] (q < n_reads: read q forward,
  // else the reverse complement of read q - n_reads); without a list, entry
  // p is read p forward
  const uint8_t* codes;
  const uint64_t* off;
  const uint32_t* len;
  uint32_t n_reads;
  const uint32_t* list;
  uint32_t host_count;         // entries listed by the host
  const uint32_t* redo_count;  // device count of entries after them (may be null)
  uint32_t redo_cap;           // capacity after host_count
  // references: slot k is panel reference ridx[k] (identity without ridx)
  const uint8_t* rcodes;
  const uint32_t* roff;
  const uint32_t* rlen;
  const uint32_t* ridx;
  uint32_t n_refs;
  uint32_t max_cols;           // longer references score kNoScore (no room in colbuf)
  int32_t* out;                // [p * n_refs + ref] (may be null)
  int32_t* rows;               // [q * n_refs + ref] (may be null)
  uint32_t wmax;               // lanes per chain at most: 32, or 1 (one thread per pair)
  uint32_t refs_per_task;
  unsigned long long* task_counter;  // null: units taken warp-strided
  int2* colbuf;                // per warp (32 / wmax) * max_cols int2
  int32_t ma, mi, o, e;
  int32_t one;                 // 1, opaque to the compiler (keeps G's add an IMAD)
};

constexpr int32_t kNoScore = INT32_MIN;

// Work of a query of n rows in R-row stripes, per reference: passes over the
// columns, at R rows and about 4 rows' worth of per-column work each, shared
// by the warp's chains.
__device__ __forceinline__ float k3_cost(int n, int R, int wmax) {
  const int S = n > 0 ? (n + R - 1) / R : 1, W = min(S, wmax);
  return (float)(((S + W - 1) / W) * (R + 4)) / (float)(32 / W);
}

// References per unit: 32 when the units then fill the resident warps twice,
// fewer for a short list, whose time is one unit's.
__host__ __device__ inline uint32_t k3_refs_per_task(uint64_t queries, uint32_t n_refs,
                                                     uint64_t warps) {
  uint32_t r = 32;
  while (r > 4 && queries * ((n_refs + r - 1) / r) < 2 * warps) r /= 2;
  return r;
}

// One query (n rows at qc) against references [k_lo, k_hi) of the panel.
template <int R, bool kLocal>
__device__ __forceinline__ void k3_unit(const K3Params& P, const int4* tab, uint32_t my, int2* buf,
                                        uint32_t pos, uint32_t q, int n, const uint8_t* qc, bool rc,
                                        uint32_t u, uint32_t tpq) {
  const int lane = threadIdx.x & 31;
  const int o = P.o, e = P.e;
  const int S = n > 0 ? (n + R - 1) / R : 1;
  const int W = min(S, (int)P.wmax);
  const int C = 32 / W;                // chains in the warp
  const int passes = (S + W - 1) / W;
  const int c = lane / W, w = lane - c * W;
  const int pad = S * R - n;
  // this unit's references: its share of the query's groups of C (whole
  // groups, so only the query's very last group can be short)
  const uint32_t groups = (P.n_refs + (uint32_t)C - 1) / (uint32_t)C;
  const uint32_t k_lo = (uint32_t)((uint64_t)u * groups / tpq) * (uint32_t)C;
  const uint32_t k_hi = min((uint32_t)((uint64_t)(u + 1) * groups / tpq) * (uint32_t)C, P.n_refs);

  for (uint32_t k0 = k_lo; k0 < k_hi; k0 += (uint32_t)C) {
    const uint32_t k = k0 + (uint32_t)c;
    const bool has = c < C && k < k_hi;
    const uint32_t mref = has ? P.rlen[k] : 0u;
    // (a reference longer than the column buffer's rows, or a query that
    // needs passes without a buffer, is not scored)
    const bool fits = mref <= P.max_cols && (passes == 1 || buf != nullptr);
    const int m = (fits && n > 0) ? (int)mref : 0;
    const int M = (int)__reduce_max_sync(kFull, (unsigned)m);
    const uint8_t* rcs = has ? P.rcodes + P.roff[k] : P.rcodes;
    // every chain's columns (chains without a reference aside): steps before
    // this one, and past the fill, need no column check
    const int mmin = (int)__reduce_min_sync(kFull, m > 0 ? (unsigned)m : 0xffffffffu);
    // local: the best H over the chain's cells; semi-global: the best of
    // the last column and (on the lane of the last stripe) the last row
    int acc = kLocal ? 0 : kNeg32;
    for (int pass = 0; pass < passes; ++pass) {
      const int s = pass * W + w;
      const bool valid = m > 0 && s < S;
      uint32_t addr[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = s * R + r - pad;
        uint32_t code = 5;  // padding row
        if (valid && i >= 0) {
          uint32_t x = rc ? qc[n - 1 - i] : qc[i];
          x = x > 4 ? 4 : x;
          code = (rc && x < 4) ? 3 - x : x;
        }
        addr[r] = my + code * kK3Stride;
      }
      const uint32_t padmask = (valid && s == 0) ? ((1u << pad) - 1u) : 0u;
      const bool from_buf = valid && pass > 0 && w == 0;
      const bool to_buf = valid && pass + 1 < passes && w == W - 1;
      // local: d of the row's next column; semi-global: G of its last one
      int g[R], ev[R];
      // this column's record: the score (s - o) of read codes 0-3
      auto record = [&](int x) {
        const int4 tw = tab[min(x, 4)];
        st_shared_u32(my, (uint32_t)tw.x);
        st_shared_u32(my + kK3Stride, (uint32_t)tw.y);
        st_shared_u32(my + 2 * kK3Stride, (uint32_t)tw.z);
        st_shared_u32(my + 3 * kK3Stride, (uint32_t)tw.w);
      };
      auto score = [&](int r) { return ld_shared_u32(addr[r]); };
      auto add = [&](int a, uint32_t b) {  // on the FMA pipe
        return (int)mad_lo((uint32_t)a, (uint32_t)P.one, b);
      };
      const int last = max(m - 1, 0);
      int x1 = valid ? rcs[0] : 0;  // the next column's code, loaded a column ahead
      if constexpr (kLocal) {
        record(x1);
        x1 = valid ? rcs[min(1, last)] : 0;
#pragma unroll
        for (int r = 0; r < R; ++r) g[r] = add(o, score(r));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) g[r] = o;  // G of a zero border cell
      }
#pragma unroll
      for (int r = 0; r < R; ++r) ev[r] = kLocal ? 0 : kNeg32;
      int gdc = o, gbot = o, fbot = kNeg32;
      int best = kLocal ? 0 : kNeg32;
      int lastrow = kNeg32, lastcol = kNeg32;
      int2 bnext = make_int2(0, 0);
      if (from_buf) bnext = buf[c];
      auto column = [&](auto check, int j, int gt, int ft) {
        constexpr bool kLast = decltype(check)::value != 0;
        if (from_buf) {
          gt = bnext.x;
          ft = bnext.y;
          bnext = buf[(size_t)min(j + 1, last) * C + c];
        }
        record(x1);
        x1 = rcs[min(j + (kLocal ? 2 : 1), last)];
        int f = ft, prev = 0, h = 0;
        if constexpr (kLocal) {
          int up = gt;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int d = g[r];
            h = __vimax3_s32(d, ev[r], f);
            if (r & 1)
              best = __vimax3_s32(best, prev, d);
            else
              prev = d;
            g[r] = add(up, score(r));
            up = add(h, (uint32_t)o);
            ev[r] = __viaddmax_s32_relu(ev[r], e, up);  // E >= 0: the floor of H
            f = __viaddmax_s32(f, e, up);
          }
          gbot = up;
        } else {
          int gup = gt, dn = add(gdc, score(0));
          gdc = gt;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int d = dn;
            if (r + 1 < R) dn = add(g[r], score(r + 1 < R ? r + 1 : r));
            ev[r] = __viaddmax_s32(ev[r], e, g[r]);
            f = __viaddmax_s32(f, e, gup);
            h = __vimax3_s32(d, ev[r], f);
            g[r] = gup = add(h, (uint32_t)o);
          }
          gbot = gup;
        }
        fbot = f;
        if (to_buf) buf[(size_t)j * C + c] = make_int2(gbot, fbot);
        if constexpr (!kLocal) {
          lastrow = max(lastrow, h);
          if (kLast && j == m - 1) {
            int cm = kNeg32;
#pragma unroll
            for (int r = 0; r < R; ++r) cm = max(cm, ((padmask >> r) & 1u) ? kNeg32 : g[r]);
            lastcol = cm - o;
          }
        }
      };
      auto top = [&](int& gt, int& ft) {
        gt = __shfl_up_sync(kFull, gbot, 1);
        ft = __shfl_up_sync(kFull, fbot, 1);
        if (w == 0) {
          gt = o;
          ft = kNeg32;
        }
      };
      const int steps = M + W - 1;
      int t = 0;
      // (semi-global: short of any chain's last column)
      const int full = min(M, mmin - (kLocal ? 0 : 1));
      if (W - 1 < full) {
#pragma unroll 1
        for (; t < W - 1; ++t) {
          int gt, ft;
          top(gt, ft);
          const int j = t - w;
          if (valid && (unsigned)j < (unsigned)m) column(IntConst<0>{}, j, gt, ft);
        }
        const int sk = valid ? w : 0;
#pragma unroll 1
        for (; t < full; ++t) {
          int gt, ft;
          top(gt, ft);
          column(IntConst<0>{}, t - sk, gt, ft);
        }
      }
#pragma unroll 1
      for (; t < steps; ++t) {
        int gt, ft;
        top(gt, ft);
        const int j = t - w;
        if (valid && (unsigned)j < (unsigned)m) column(IntConst<1>{}, j, gt, ft);
      }
      __syncwarp();  // the buffer's writes are seen by the next pass
      if (valid) {
        if constexpr (kLocal) {
          acc = max(acc, best);
        } else {
          acc = max(acc, lastcol);
          if (s == S - 1) acc = max(acc, lastrow);
        }
      }
    }
    // the chain's maximum, to its first lane
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_down_sync(kFull, acc, d);
      if (w + d < W) acc = max(acc, v);
    }
    if (has && w == 0) {
      // scalar.rs:123-125: an empty query or reference scores 0
      const int score = !fits ? kNoScore : (m == 0 ? 0 : acc);
      const uint32_t ref = P.ridx ? P.ridx[k] : k;
      if (P.out) P.out[(size_t)pos * P.n_refs + ref] = score;
      if (P.rows) P.rows[(size_t)q * P.n_refs + ref] = score;
    }
  }
}

template <bool kLocal>
__global__ void __launch_bounds__(kK3Threads, 3) k3_lanes(const K3Params P) {
  __shared__ int4 tab[5];                      // words of read codes 0-3 against reference code x
  __shared__ uint32_t rec[6 * kK3Threads];     // word c of thread t at c * kK3Threads + t
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int mao = P.ma - P.o, mio = P.mi - P.o;
  if (threadIdx.x < 5) {
    const int x = threadIdx.x;  // 4: a wildcard reference base matches every read code
    tab[x] = make_int4((x == 0 || x == 4) ? mao : mio, (x == 1 || x == 4) ? mao : mio,
                       (x == 2 || x == 4) ? mao : mio, (x == 3 || x == 4) ? mao : mio);
  }
  const uint32_t my = (uint32_t)__cvta_generic_to_shared(rec) + threadIdx.x * 4u;
  st_shared_u32(my + 4 * kK3Stride, (uint32_t)mao);   // read wildcard: a match everywhere
  st_shared_u32(my + 5 * kK3Stride, (uint32_t)-P.o);  // padding row: s = 0
  __syncthreads();

  const uint32_t n_list =
      P.host_count + (P.redo_count ? min(*P.redo_count, P.redo_cap) : 0u);
  const uint32_t tpq = (P.n_refs + P.refs_per_task - 1) / P.refs_per_task;
  const unsigned long long n_units = (unsigned long long)n_list * tpq;
  const size_t warp_id = (size_t)blockIdx.x * kK3Warps + wib;
  const size_t n_warps = (size_t)gridDim.x * kK3Warps;
  const int cmax = 32 / (int)P.wmax;
  int2* const buf = P.colbuf ? P.colbuf + warp_id * (size_t)cmax * P.max_cols : nullptr;

  unsigned long long unit = warp_id;
  for (;; unit += P.task_counter ? 0ull : n_warps) {
    if (P.task_counter) {
      unsigned long long u = 0;
      if (lane == 0) u = atomicAdd(P.task_counter, 1ull);
      unit = __shfl_sync(kFull, u, 0);
    }
    if (unit >= n_units) break;
    const uint32_t pos = (uint32_t)(unit / tpq);
    const uint32_t u = (uint32_t)(unit - (unsigned long long)pos * tpq);
    const uint32_t q = P.list ? P.list[pos] : pos;
    const bool rc = q >= P.n_reads;
    const uint32_t rd = rc ? q - P.n_reads : q;
    const int n = (int)P.len[rd];
    const uint8_t* qc = P.codes + P.off[rd];
    if (k3_cost(n, 28, (int)P.wmax) < k3_cost(n, 32, (int)P.wmax))
      k3_unit<28, kLocal>(P, tab, my, buf, pos, q, n, qc, rc, u, tpq);
    else
      k3_unit<32, kLocal>(P, tab, my, buf, pos, q, n, qc, rc, u, tpq);
  }
}

// ---------------------------------------------------------------- k4
struct K4Params {
  const uint32_t* list;
  uint32_t host_count;
  const uint32_t* redo_count;
  uint32_t redo_cap;
  const int32_t* rows;  // k3 output, [pos * n_refs + r]
  uint32_t n_refs;
  uint32_t n_reads;
  int4* qhead;
  uint32_t* qties;
  uint32_t cap;
};

// One warp per listed query: mapper.rs:444-472 over its row.
static __global__ void __launch_bounds__(256) k4_rows(const K4Params P) {
  const uint32_t n_list = P.host_count + (P.redo_count ? min(*P.redo_count, P.redo_cap) : 0u);
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t pos = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; pos < n_list; pos += warps) {
    const uint32_t q = P.list[pos];
    const uint32_t rbit = q >= P.n_reads ? 1u : 0u;
    const int32_t* row = P.rows + (size_t)pos * P.n_refs;
    int best = INT32_MIN;
    for (uint32_t r = lane; r < P.n_refs; r += 32) best = max(best, row[r]);
#pragma unroll
    for (int d = 16; d; d >>= 1) best = max(best, __shfl_xor_sync(kFull, best, d));
    int sub = INT32_MIN;
    uint32_t n_tied = 0, listed = 0;
    for (uint32_t base = 0; base < P.n_refs; base += 32) {
      const uint32_t r = base + lane;
      const int v = r < P.n_refs ? row[r] : INT32_MIN;
      const bool tie = r < P.n_refs && v == best;
      if (r < P.n_refs && !tie) sub = max(sub, v);
      const uint32_t bal = __ballot_sync(kFull, tie);
      if (tie) {
        const uint32_t rank = listed + __popc(bal & ((1u << lane) - 1u));
        if (rank < P.cap) P.qties[(size_t)q * P.cap + rank] = (r << 1) | rbit;
      }
      listed += __popc(bal);
      n_tied += __popc(bal);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) sub = max(sub, __shfl_xor_sync(kFull, sub, d));
    if (lane == 0) P.qhead[q] = make_int4(best, sub, (int)n_tied, kQRescored);
  }
}

// ---------------------------------------------------------------- k0
// Reads travel host to device packed at 2 bits a base (base i of a byte in
// bits 2i..2i+1, each read starting on a byte); these two kernels run once
// after the upload.  k0_unpack writes one byte a base: each thread takes a
// 32-bit word (16 bases) and stores 16 bytes.  k0_exceptions then sets the
// listed positions -- read bases that were not A/C/G/T -- to the wildcard
// code 4.
__device__ __forceinline__ uint32_t spread4(uint32_t b) {
  return (b & 3u) | ((b >> 2) & 3u) << 8 | ((b >> 4) & 3u) << 16 | ((b >> 6) & 3u) << 24;
}

static __global__ void __launch_bounds__(256) k0_unpack(const uint32_t* __restrict__ packed,
                                                        uint64_t n_words, uint4* __restrict__ codes) {
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
       w += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = packed[w];
    codes[w] = make_uint4(spread4(p & 0xffu), spread4((p >> 8) & 0xffu), spread4((p >> 16) & 0xffu),
                          spread4(p >> 24));
  }
}

static __global__ void __launch_bounds__(256) k0_exceptions(const uint64_t* __restrict__ at,
                                                            uint64_t n, uint8_t* __restrict__ codes) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    codes[at[i]] = 4;
}

// ---------------------------------------------------------------- k5
struct K5Params {
  const uint32_t* len;
  uint32_t n_reads;
  int both;
  const int4* qhead;
  const uint32_t* qties;
  uint32_t cap;
  int4* results;       // esg_read_result layout
  uint32_t* ties;      // [read * cap + k]
  int32_t* rows;       // optional rows: an empty read's rows score 0 (no cell)
  uint32_t n_refs;
};

static __global__ void __launch_bounds__(256) k5_merge(const K5Params P) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < P.n_reads;
       r += gridDim.x * blockDim.x) {
    const uint32_t cap = P.cap;
    uint32_t* out_t = P.ties + (size_t)r * cap;
    if (P.len[r] == 0) {
      P.results[r] = make_int4(INT32_MIN, INT32_MIN, 0, 1 /* ESG_RESULT_EMPTY */);
      for (uint32_t k = 0; k < cap; ++k) out_t[k] = kNoRef;
      if (P.rows) {
        for (uint32_t j = 0; j < P.n_refs; ++j) P.rows[(size_t)r * P.n_refs + j] = 0;
        if (P.both)
          for (uint32_t j = 0; j < P.n_refs; ++j)
            P.rows[((size_t)P.n_reads + r) * P.n_refs + j] = 0;
      }
      continue;
    }
    const int4 a = P.qhead[r];
    const uint32_t* ta = P.qties + (size_t)r * cap;
    int best = a.x, sub = a.y, flags = a.w & kQRescored;
    uint32_t n_tied = (uint32_t)a.z;
    if (!P.both) {
      const uint32_t nl = min(n_tied, cap);
      for (uint32_t k = 0; k < nl; ++k) out_t[k] = ta[k];
    } else {
      const uint32_t qb = P.n_reads + r;
      const int4 b = P.qhead[qb];
      const uint32_t* tb = P.qties + (size_t)qb * cap;
      flags |= b.w & kQRescored;
      const uint32_t na = min((uint32_t)a.z, cap), nb = min((uint32_t)b.z, cap);
      if (a.x > b.x) {
        sub = max(max(a.y, b.y), b.x);
        for (uint32_t k = 0; k < na; ++k) out_t[k] = ta[k];
      } else if (b.x > a.x) {
        best = b.x;
        n_tied = (uint32_t)b.z;
        sub = max(max(a.y, b.y), a.x);
        for (uint32_t k = 0; k < nb; ++k) out_t[k] = tb[k];
      } else {
        n_tied = (uint32_t)a.z + (uint32_t)b.z;
        sub = max(a.y, b.y);
        uint32_t i = 0, k2 = 0, w = 0;
        while (w < cap && (i < na || k2 < nb)) {
          if (k2 >= nb || (i < na && ta[i] < tb[k2]))
            out_t[w++] = ta[i++];
          else
            out_t[w++] = tb[k2++];
        }
      }
    }
    for (uint32_t k = min(n_tied, cap); k < cap; ++k) out_t[k] = kNoRef;  // ESG_NO_TIE
    if (n_tied > cap) flags |= 2;  // ESG_RESULT_TIES_TRUNCATED
    P.results[r] = make_int4(best, sub, (int)n_tied, flags);
  }
}

// Batches in panel chunks whose queries all ran on k2 and cannot be flagged:
// k2_merge_chunks and k5_merge in one, a warp per read.
struct K5ChunkParams {
  K5Params M;
  uint32_t n_chunks;
  const int4* part_head;
  const uint32_t* part_ties;
};

static __global__ void __launch_bounds__(128) k5_merge_chunks(const K5ChunkParams P) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5, cap = P.M.cap;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < P.M.n_reads; r += warps) {
    uint32_t tie = kNoRef;
    int4 out = make_int4(INT32_MIN, INT32_MIN, 0, 1 /* ESG_RESULT_EMPTY */);
    if (P.M.len[r] == 0) {
      if (P.M.rows)
        for (uint32_t j = lane; j < P.M.n_refs; j += 32) {
          P.M.rows[(size_t)r * P.M.n_refs + j] = 0;
          if (P.M.both) P.M.rows[((size_t)P.M.n_reads + r) * P.M.n_refs + j] = 0;
        }
    } else {
      size_t base = (size_t)r * P.n_chunks;
      int4 a = merge_chunks(P.part_head + base, P.part_ties + base * cap, P.n_chunks, cap, lane,
                            tie);
      if (P.M.both) {
        base += (size_t)P.M.n_reads * P.n_chunks;
        uint32_t tb;
        const int4 b = merge_chunks(P.part_head + base, P.part_ties + base * cap, P.n_chunks, cap,
                                    lane, tb);
        const int sub = max(a.y, b.y);
        if (a.x == b.x) {
          a = make_int4(a.x, sub, a.z + b.z, 0);
          tie = merge_lists(tie, tb, lane);
        } else if (a.x > b.x) {
          a = make_int4(a.x, max(sub, b.x), a.z, 0);
        } else {
          a = make_int4(b.x, max(sub, a.x), b.z, 0);
          tie = tb;
        }
      }
      out = make_int4(a.x, a.y, a.z, (uint32_t)a.z > cap ? 2 : 0 /* ESG_RESULT_TIES_TRUNCATED */);
    }
    if ((uint32_t)lane < cap) P.M.ties[(size_t)r * cap + lane] = tie;  // kNoRef: ESG_NO_TIE
    if (lane == 0) P.M.results[r] = out;
  }
}

// ---------------------------------------------------------------- k6_pairs
// One warp per read pair.  Rows: mate m of pair p is read 2p + m; its
// forward row is query 2p + m, its reverse-complement row n_reads + 2p + m.
// Candidate (r, t): t = 0 pairs mate 1 forward with mate 2 reverse-
// complemented, t = 1 mate 1 reverse-complemented with mate 2 forward
// (pair.rs:135-137); eligible when both mate scores are >= min_score.
// Pass 1 takes the best eligible sum; pass 2 walks the references in
// 32-wide chunks and, in (r, t) order, lists the first tier (ballots give
// each tie its rank), and takes the next tier's sum and the per-mate best
// over candidates outside the tier (pair.rs:297-314).
struct K6Params {
  const int32_t* rows;   // [q * n_refs + r], q < 2 n_reads
  const uint32_t* len;   // trimmed mate lengths [n_reads]
  const int4* mates;     // k5's per-mate results (for RESCORED32)
  uint32_t n_pairs;
  uint32_t n_reads;
  uint32_t n_refs;
  uint32_t cap;
  int32_t min_score;
  int both;              // both template strands
  int4* out;             // [2 p]: best, next, n_tied, flags; [2 p + 1]: xs[2], primary[2]
  uint32_t* ties;        // [p * cap + k]
};

static __global__ void __launch_bounds__(256) k6_pairs(const K6Params P) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t wpb = blockDim.x >> 5;
  const int32_t ms = P.min_score;
  for (uint32_t p = blockIdx.x * wpb + (threadIdx.x >> 5); p < P.n_pairs; p += gridDim.x * wpb) {
    uint32_t* out_t = P.ties + (size_t)p * P.cap;
    const size_t nr = P.n_refs;
    const int32_t* f0 = P.rows + (size_t)(2 * p) * nr;
    const int32_t* f1 = f0 + nr;
    const int32_t* r0 = P.rows + (size_t)(P.n_reads + 2 * p) * nr;
    const int32_t* r1 = r0 + nr;
    const bool empty = P.len[2 * p] == 0 || P.len[2 * p + 1] == 0;
    int32_t best = INT32_MIN;
    if (!empty) {
      for (uint32_t r = lane; r < P.n_refs; r += 32) {
        const int32_t a = f0[r], b = r1[r];
        if (a >= ms && b >= ms) best = max(best, a + b);
        if (P.both) {
          const int32_t c = r0[r], d = f1[r];
          if (c >= ms && d >= ms) best = max(best, c + d);
        }
      }
    }
    best = __reduce_max_sync(kFull, best);
    const bool any = best != INT32_MIN;
    int32_t next = INT32_MIN, xs0 = INT32_MIN, xs1 = INT32_MIN, pa = INT32_MIN, pb = INT32_MIN;
    uint32_t n = 0;
    if (!empty) {
      for (uint32_t c0 = 0; c0 < P.n_refs; c0 += 32) {
        const uint32_t r = c0 + lane;
        const bool valid = r < P.n_refs;
        int32_t a = 0, b = 0, c = 0, d = 0;
        bool tie0 = false, tie1 = false;
        if (valid) {
          a = f0[r];
          b = r1[r];
          const bool e0 = a >= ms && b >= ms;
          tie0 = e0 && a + b == best;
          if (!tie0) {
            if (e0) next = max(next, a + b);
            xs0 = max(xs0, a);
            xs1 = max(xs1, b);
          }
          if (P.both) {
            c = r0[r];
            d = f1[r];
            const bool e1 = c >= ms && d >= ms;
            tie1 = e1 && c + d == best;
            if (!tie1) {
              if (e1) next = max(next, c + d);
              xs0 = max(xs0, c);
              xs1 = max(xs1, d);
            }
          }
        }
        const uint32_t b0 = __ballot_sync(kFull, tie0), b1 = __ballot_sync(kFull, tie1);
        if ((b0 | b1) == 0) continue;
        if (n == 0) {  // the primary: the first tie in (r, t) order
          const int src = __ffs(b0 | b1) - 1;
          const bool t0 = (b0 >> src) & 1u;
          pa = __shfl_sync(kFull, t0 ? a : c, src);
          pb = __shfl_sync(kFull, t0 ? b : d, src);
        }
        const uint32_t pre = n + __popc(b0 & lt) + __popc(b1 & lt);
        if (tie0 && pre < P.cap) out_t[pre] = r << 1;
        if (tie1 && pre + tie0 < P.cap) out_t[pre + tie0] = (r << 1) | 1u;
        n += __popc(b0) + __popc(b1);
      }
    }
    next = __reduce_max_sync(kFull, next);
    xs0 = __reduce_max_sync(kFull, xs0);
    xs1 = __reduce_max_sync(kFull, xs1);
    for (uint32_t k = min(n, P.cap) + lane; k < P.cap; k += 32) out_t[k] = kNoRef;  // ESG_NO_TIE
    if (lane == 0) {
      int flags = (any ? 0 : 1) | (n > P.cap ? 2 : 0);  // ESG_RESULT_EMPTY / _TIES_TRUNCATED
      if (!empty) flags |= (P.mates[2 * p].w | P.mates[2 * p + 1].w) & kQRescored;
      P.out[2 * p] = make_int4(best, next, (int)n, flags);
      P.out[2 * p + 1] = make_int4(xs0, xs1, pa, pb);
    }
  }
}

}  // namespace esg
