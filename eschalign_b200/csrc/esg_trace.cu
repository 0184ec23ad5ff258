// esg_trace.cu -- traceback of winners on the device: the alignment
// (coordinates and CIGAR) of chosen (read, reference, strand) jobs, as
// crates/eschalign/src/scalar.rs:182-364 computes it.
//
// k7_tags: tiles of jobs of at most 1024 rows whose scores fit 16 bits; the
// trace rides in the low bits of the recurrence's values (see below).
// k7_trace: one warp per task.  A task is a tile of jobs whose 16-row
// stripes fill the warp's lanes (a job of n rows takes ceil(n / 16) lanes;
// each job has its own reference), or one long job (over 32 stripes) run in
// passes of 32 stripes chained through a per-warp column buffer.  Lanes
// walk their job's reference columns as a systolic array (lane l one step
// behind lane l - 1, the stripe's bottom row passed down by shuffle) in
// int32 -- the recurrence of scalar.rs:213-289 exactly, no saturation --
// and write one 4-bit trace code per cell (source: stop / diagonal /
// insertion / deletion, plus the E- and F-extended bits) to a per-warp
// scratch: 8 bytes per lane per column, lane-contiguous, so a warp writes
// 256 coalesced bytes a column and the scratch of the resident warps stays
// in L2.  Reads are top-padded so the last row sits at row 15 of the last
// stripe; pad rows hold H = 0, the zero border.  Each lane keeps its first
// maximum in column-major order (local: every cell; semi-global: the last
// row and the last column); a segmented shuffle reduction gives the job's
// end cell, and the job's last lane follows the trace codes back
// (scalar.rs:292-364), writing run-length CIGAR words.  k7_sums and
// k7_pack put the jobs' words and records into the caller's layout.
#include "../../include/eschalign_b200.h"
#include "esg_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

extern "C" void esg_internal_set_error(esg_status st, const char* msg);

namespace {

constexpr int kTR = 16;                 // rows per lane stripe
constexpr int kTWarps = 4;              // warps per CTA
constexpr int kTThreads = kTWarps * 32;
constexpr int kNegT = INT32_MIN / 4;    // scalar.rs's NEG
constexpr uint32_t kFullT = 0xffffffffu;
// trace codes (scalar.rs:167-175)
constexpr uint32_t kStop = 0, kDiag = 1, kIns = 2, kDel = 3, kEExt = 4, kFExt = 8;
// cigar ops (BAM)
constexpr uint32_t kOpM = 0, kOpI = 1, kOpD = 2;

struct K7Params {
  const uint8_t* codes;       // reads, 1 B codes
  const uint64_t* off;
  const uint32_t* len;
  const uint8_t* rcodes;      // panel, longest first (slot order)
  const uint32_t* roff;
  const uint32_t* rlen;
  const uint32_t* job_q;      // read | reverse << 31
  const uint32_t* job_slot;   // panel slot of the job's reference
  const uint64_t* job_at;     // the job's first word in the ops staging
  const uint32_t* order;      // jobs in task order
  const uint2* tasks;         // {start in order, count | stripes << 16}; stripes > 32: one long job
  uint32_t n_tasks;
  uint32_t* task_counter;
  uint2* trace;               // per warp: trace_words uint2
  size_t trace_words;
  uint32_t mcols;             // columns of one pass in the trace scratch
  uint2* colbuf;              // per warp: mcols (H, F), long jobs
  int ma, mi, o, e;
  int4* res;                  // per job {score, query_start, query_end, ref_start}
  int4* res2;                 // per job {ref_end, n_ops, 0, 0}
  uint32_t* ops;              // staging
};

__device__ __forceinline__ uint32_t mask4(uint32_t c) { return c < 4 ? 1u << c : 0xfu; }

// (b1, j1, i1) better than (b0, j0, i0): higher score, then smaller column,
// then smaller row -- the first maximum of a column-major scan.
__device__ __forceinline__ bool better(int b1, int j1, int i1, int b0, int j0, int i0) {
  return b1 > b0 || (b1 == b0 && (j1 < j0 || (j1 == j0 && i1 < i0)));
}

template <bool kLocal>
__global__ void __launch_bounds__(kTThreads) k7_trace(const K7Params P) {
  const int lane = threadIdx.x & 31;
  const size_t warp = (size_t)blockIdx.x * kTWarps + (threadIdx.x >> 5);
  uint2* trace = P.trace + warp * P.trace_words;
  uint2* colbuf = P.colbuf + warp * P.mcols;
  for (;;) {
    uint32_t task = 0;
    if (lane == 0) task = atomicAdd(P.task_counter, 1u);
    task = __shfl_sync(kFullT, task, 0);
    if (task >= P.n_tasks) break;
    const uint2 tk = P.tasks[task];
    const uint32_t count = tk.y & 0xffffu;
    const int smax = (int)(tk.y >> 16);
    const bool long_job = smax > 32;

    // --- lane -> (job, first lane of the job, stripes)
    uint32_t job = 0, n = 0;
    int S = 0, s0 = 0;
    bool has_job = false;
    if (long_job) {
      job = P.order[tk.x];
      n = P.len[P.job_q[job] & 0x7fffffffu];
      S = smax;
      has_job = true;
    } else {
      uint32_t kj = 0, kn = 0, kS = 0;
      if ((uint32_t)lane < count) {
        kj = P.order[tk.x + lane];
        kn = P.len[P.job_q[kj] & 0x7fffffffu];
        kS = (kn + kTR - 1) / kTR;
      }
      uint32_t incl = kS;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kFullT, incl, d);
        if (lane >= d) incl += v;
      }
      for (uint32_t k = 0; k < count; ++k) {
        const uint32_t ek = __shfl_sync(kFullT, incl, k);
        const uint32_t sk = __shfl_sync(kFullT, kS, k);
        const uint32_t jk = __shfl_sync(kFullT, kj, k);
        const uint32_t nk = __shfl_sync(kFullT, kn, k);
        if ((uint32_t)lane >= ek - sk && (uint32_t)lane < ek) {
          job = jk;
          n = nk;
          S = (int)sk;
          s0 = (int)(ek - sk);
          has_job = true;
        }
      }
    }
    const uint32_t jq = has_job ? P.job_q[job] : 0u;
    const uint32_t rd = jq & 0x7fffffffu;
    const bool rc = (jq >> 31) != 0;
    const uint32_t slot = has_job ? P.job_slot[job] : 0u;
    const int m = has_job ? (int)P.rlen[slot] : 0;
    const uint8_t* rp = P.rcodes + (has_job ? P.roff[slot] : 0u);
    const uint8_t* q = P.codes + (has_job ? P.off[rd] : 0ull);
    const int pad = S * kTR - (int)n;
    const int passes = long_job ? (S + 31) / 32 : 1;

    int best = kLocal ? 0 : kNegT, bj = 0, bi = 0;  // 1-based end cell, 0: none
    for (int pass = 0; pass < passes; ++pass) {
      const int s = long_job ? pass * 32 + lane : lane - s0;  // stripe of the job
      const bool valid = has_job && s >= 0 && s < S;
      const bool first = valid && s == 0;
      const bool from_buf = long_job && pass > 0 && lane == 0;
      const bool to_buf = long_job && pass + 1 < passes && lane == 31;
      const int padrows = (valid && s == 0) ? pad : 0;
      uint32_t qm[kTR];
#pragma unroll
      for (int r = 0; r < kTR; ++r) {
        const int i = s * kTR + r - pad;  // 0-based read row
        uint32_t c = 4;
        if (valid && i >= 0) {
          uint32_t x = rc ? q[n - 1 - i] : q[i];
          x = x > 4 ? 4 : x;
          c = (rc && x < 4) ? 3 - x : x;
        }
        qm[r] = mask4(c);
      }
      int H[kTR], E[kTR];
#pragma unroll
      for (int r = 0; r < kTR; ++r) {
        H[r] = 0;
        E[r] = kNegT;
      }
      int hbot = 0, fbot = kNegT, hdg = 0;
      // the pass's first maximum (its columns come in order)
      int pb = kLocal ? 0 : kNegT, pj = 0, pi = 0;
      const int skew = long_job ? lane : s;
      int steps = valid ? m + skew : 0;
#pragma unroll
      for (int d = 16; d; d >>= 1) steps = max(steps, __shfl_xor_sync(kFullT, steps, d));
#pragma unroll 1
      for (int t = 0; t < steps; ++t) {
        const int j = t - skew;
        int ht = __shfl_up_sync(kFullT, hbot, 1);
        int ft = __shfl_up_sync(kFullT, fbot, 1);
        if (first) {
          ht = 0;
          ft = kNegT;
        }
        if (valid && (unsigned)j < (unsigned)m) {
          if (from_buf) {
            const uint2 b = colbuf[j];
            ht = (int)b.x;
            ft = (int)b.y;
          }
          const uint32_t rm = mask4(rp[j]);
          int hup = ht, f = ft, hdiag = hdg;
          hdg = ht;
          uint32_t w0 = 0, w1 = 0;
#pragma unroll
          for (int r = 0; r < kTR; ++r) {
            const int hleft = H[r];
            const int e_ext = E[r] + P.e, e_open = hleft + P.o;
            const int ev = max(e_open, e_ext);
            const int f_ext = f + P.e, f_open = hup + P.o;
            f = max(f_open, f_ext);
            const int hd = hdiag + ((qm[r] & rm) ? P.ma : P.mi);
            int h = max(max(hd, ev), f);
            if (kLocal) h = max(h, 0);
            if (r < padrows) h = 0;  // the zero border above the read
            uint32_t t4 = h == f ? kIns : kDel;
            if (h == hd) t4 = kDiag;
            if (kLocal && h == 0) t4 = kStop;
            t4 |= (ev == e_ext ? kEExt : 0u) | (f == f_ext ? kFExt : 0u);
            if (r < 8)
              w0 |= t4 << (4 * r);
            else
              w1 |= t4 << (4 * (r - 8));
            E[r] = ev;
            hdiag = hleft;
            H[r] = h;
            hup = h;
            if (kLocal && h > pb) {  // pad rows hold 0: never above it
              pb = h;
              pi = s * kTR + r - pad + 1;
              pj = j + 1;
            }
          }
          trace[((size_t)pass * P.mcols + j) * 32 + lane] = make_uint2(w0, w1);
          hbot = H[kTR - 1];
          fbot = f;
          if (to_buf) colbuf[j] = make_uint2((uint32_t)hbot, (uint32_t)fbot);
          if (!kLocal) {
            if (j < m - 1) {
              if (s == S - 1 && hbot > pb) {  // the last row
                pb = hbot;
                pi = (int)n;
                pj = j + 1;
              }
            } else {
#pragma unroll
              for (int r = 0; r < kTR; ++r) {  // the last column, rows in order
                const int i = s * kTR + r - pad + 1;
                if (i >= 1 && H[r] > pb) {
                  pb = H[r];
                  pi = i;
                  pj = m;
                }
              }
            }
          }
        }
      }
      // (a later pass starts at the first column again)
      if (better(pb, pj, pi, best, bj, bi)) {
        best = pb;
        bj = pj;
        bi = pi;
      }
      __syncwarp();  // trace and column buffer writes visible to the warp
    }

    // --- the job's end cell: first maximum over its lanes
    {
      const int sj = long_job ? lane : lane - s0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int b2 = __shfl_up_sync(kFullT, best, d);
        const int j2 = __shfl_up_sync(kFullT, bj, d);
        const int i2 = __shfl_up_sync(kFullT, bi, d);
        if (has_job && sj >= d && better(b2, j2, i2, best, bj, bi)) {
          best = b2;
          bj = j2;
          bi = i2;
        }
      }
    }
    // --- the walk, by the job's last lane
    const bool walker = has_job && (long_job ? lane == 31 : lane - s0 == S - 1);
    if (walker) {
      int i = bi, j = bj;
      uint32_t* out = P.ops + P.job_at[job];
      uint32_t runs = 0, cur = 4, cnt = 0;
      int state = 0;  // 0 H, 1 E (deletion), 2 F (insertion)
      while (i > 0 && j > 0) {
        const int ip = i - 1 + pad;
        const int st = ip >> 4, r = ip & 15;
        const int ln = long_job ? (st & 31) : s0 + st;
        const int ps = long_job ? (st >> 5) : 0;
        const uint2 w = trace[((size_t)ps * P.mcols + (j - 1)) * 32 + ln];
        const uint32_t t4 = ((r < 8 ? w.x : w.y) >> (4 * (r & 7))) & 0xfu;
        uint32_t op = 4;
        if (state == 0) {
          const uint32_t src = t4 & 3u;
          if (src == kStop) break;
          if (src == kDiag) {
            op = kOpM;
            --i;
            --j;
          } else if (src == kIns) {
            state = 2;
          } else {
            state = 1;
          }
        } else if (state == 2) {
          op = kOpI;
          if (!(t4 & kFExt)) state = 0;
          --i;
        } else {
          op = kOpD;
          if (!(t4 & kEExt)) state = 0;
          --j;
        }
        if (op != 4) {
          if (op == cur) {
            ++cnt;
          } else {
            if (cnt) out[runs++] = (cnt << 4) | cur;
            cur = op;
            cnt = 1;
          }
        }
      }
      if (cnt) out[runs++] = (cnt << 4) | cur;
      for (uint32_t a = 0, b = runs ? runs - 1 : 0; a < b; ++a, --b) {  // first to last
        const uint32_t x = out[a];
        out[a] = out[b];
        out[b] = x;
      }
      const bool none = bi == 0 || bj == 0;
      P.res[job] = none ? make_int4(0, 0, 0, 0) : make_int4(best, i, bi, j);
      P.res2[job] = make_int4(none ? 0 : bj, (int)runs, 0, 0);
    }
    __syncwarp();  // the walk is done before the scratch is reused
  }
}

// ---------------------------------------------------------------- k7_tags
// The traceback of jobs of at most 1024 rows whose scores fit 16 bits (what
// is left takes k7_trace): tiles of jobs on 28- or 32-row stripes, one pass.
//
// k7_trace compares its way to a trace code, some 25 ALU instructions a cell.
// Here the maxima of the recurrence carry it: every value is
//     (score - 1) << 16 | source << 14 | length
// with source 1 deletion, 2 insertion, 3 diagonal -- the order that breaks
// ties as scalar.rs:259-285 does -- and length the gap's extensions so far.
// Extending adds (e << 16) + 1, so on a tie the extension wins, and a gap's
// end holds its whole length: the 16 low bits of H are all the walk needs of a
// cell, two cells to a stored word.  A local score of 0 is the floor value 0
// (VIADDMNMX.RELU on E), source 0: stop.  The score alone, for the next
// cells, is (value + 0xc000) & 0xffff0000; semi-global, where no value is 0,
// it is the high half itself (score - 1).  5 ALU instructions a cell local, 4
// semi-global, the adds on the FMA pipe.
// Stored words are indexed by step, not by column, so that a warp's stores
// are contiguous: word q of lane l at step t at ((t * 4 + q) * 32 + l) * 16
// bytes, rows 8 q .. 8 q + 7 of the stripe.
// What bounds it: issue slots (11 instructions a cell) and the walk's loads;
// the scratch (2 bytes a cell) is written once, 3.5 GB of DRAM traffic here.
// 100 000 jobs of ~110 nt x 70-180 nt: 2.9 -> 1.4 ms semi-global, 3.7 -> 1.4
// local (on 330 CTAs; 1.2 on 444, whose scratch is 0.77 GB).
constexpr int kTagRows = 1024;    // longest read
constexpr int kTagCols = 1700;    // longest reference: 592 warps' scratch in kTagBytes
constexpr uint64_t kTagBytes = 2ull << 30;
constexpr uint64_t kTagOwn = 64ull << 20;  // scratch up to this: the scorer's own pool
constexpr int kTagScore = 30000;  // bound on |score|, gap floors included
constexpr int kAhead = 8;         // cells of the walk read at once (4, 8, 16: 1.24, 1.19, 1.27 ms)
constexpr int kTagNeg = -31000 * 65536;
constexpr uint32_t kTag28 = 0x8000u;  // in a task's count: 28-row stripes

template <bool kOn>
struct TagCheck {
  static constexpr bool value = kOn;
};

struct K7TagParams {
  K7Params J;
  uint4* trace;     // per warp: steps * 128 uint4
  uint32_t steps;   // of a tile at most
  int one;          // 1, opaque to the compiler (keeps adds on the FMA pipe)
};

__device__ __forceinline__ uint32_t tag_lds(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void tag_sts(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v));
}

template <int R, bool kLocal>
__device__ __forceinline__ void tag_tile(const K7TagParams& P, const int4* tab, uint32_t my,
                                         uint4* trace, uint2 tk) {
  constexpr uint32_t kStride = kTThreads * 4;
  const K7Params& J = P.J;
  const int lane = threadIdx.x & 31;
  const uint32_t count = tk.y & 0x7fffu;
  const int smax = (int)(tk.y >> 16);
  // --- lane -> (job, stripe)
  uint32_t job = 0, n = 0;
  int S = 0, s0 = 0;
  bool valid = false;
  {
    uint32_t kj = 0, kn = 0, kS = 0;
    if ((uint32_t)lane < count) {
      kj = J.order[tk.x + lane];
      kn = J.len[J.job_q[kj] & 0x7fffffffu];
      kS = (kn + R - 1) / R;
    }
    uint32_t incl = kS;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(kFullT, incl, d);
      if (lane >= d) incl += v;
    }
    for (uint32_t k = 0; k < count; ++k) {
      const uint32_t ek = __shfl_sync(kFullT, incl, k);
      const uint32_t sk = __shfl_sync(kFullT, kS, k);
      const uint32_t jk = __shfl_sync(kFullT, kj, k);
      const uint32_t nk = __shfl_sync(kFullT, kn, k);
      if ((uint32_t)lane >= ek - sk && (uint32_t)lane < ek) {
        job = jk;
        n = nk;
        S = (int)sk;
        s0 = (int)(ek - sk);
        valid = true;
      }
    }
  }
  const uint32_t jq = valid ? J.job_q[job] : 0u;
  const uint32_t rd = jq & 0x7fffffffu;
  const bool rc = (jq >> 31) != 0;
  const uint32_t slot = valid ? J.job_slot[job] : 0u;
  const int m = valid ? (int)J.rlen[slot] : 0;
  const uint8_t* rp = J.rcodes + (valid ? J.roff[slot] : 0u);
  const uint8_t* q = J.codes + (valid ? J.off[rd] : 0ull);
  const int pad = S * R - (int)n;
  const int s = valid ? lane - s0 : 0;
  const bool first = !valid || s == 0;
  const int padrows = (valid && s == 0) ? pad : 0;
  uint32_t addr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = s * R + r - pad;
    uint32_t c = 5;  // padding row
    if (valid && i >= 0) {
      uint32_t x = rc ? q[n - 1 - i] : q[i];
      x = x > 4 ? 4 : x;
      c = (rc && x < 4) ? 3 - x : x;
    }
    addr[r] = my + c * kStride;
  }
  auto add = [&](int a, int b) {  // on the FMA pipe
    int d;
    asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(P.one), "r"(b));
    return d;
  };
  const int last = max(m - 1, 0);
  // a zero cell's score as the next cells take it
  constexpr int kZero = kLocal ? 0 : -65536;
  const int cE = J.o * 65536 + (kLocal ? -0xc000 : 0x4000);
  const int cF = J.o * 65536 + (kLocal ? -0x8000 : 0x8000);
  const int ext = J.e * 65536 + 1;
  auto record = [&](int x) {
    const int4 tw = tab[min(x, 4)];
    tag_sts(my, (uint32_t)tw.x);
    tag_sts(my + kStride, (uint32_t)tw.y);
    tag_sts(my + 2 * kStride, (uint32_t)tw.z);
    tag_sts(my + 3 * kStride, (uint32_t)tw.w);
  };
  // d of the row's next column, and E of the first one: opened at the border,
  // as F of a first row is (local, where an open from 0 is under the floor: the floor)
  int g[R], ev[R];
  record(valid ? rp[0] : 0);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    g[r] = add(kZero, (int)tag_lds(addr[r]));
    ev[r] = kLocal ? 0 : add(kZero, cE);
  }
  int x1 = rp[min(1, last)];
  int hbot = kZero, fbot = add(kZero, cF);
  const int ftop = fbot;  // F of a first row: opened at the border
  int best = kLocal ? 0 : kNegT, bj = 0, bi = 0;  // 1-based end cell, 0: none
  const int steps = [&] {
    int v = valid ? m + s : 0;
    return __reduce_max_sync(kFullT, v);
  }();
  // columns every job's lanes are inside, short of any last column
  const int full = (int)__reduce_min_sync(kFullT, valid ? (unsigned)(m - 1) : 0x7fffffffu);
  auto column = [&](auto check, int t, int j, int up, int f) {
    constexpr bool kCheck = decltype(check)::value;
    record(x1);
    x1 = rp[min(j + 2, last)];
    int hc[R];
    uint32_t w[R / 2];
    int prev = 0, xp = 0, cm = kTagNeg;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int x = __vimax3_s32(g[r], ev[r], f);
      const int h = (kLocal ? add(x, 0xc000) : x) & (int)0xffff0000;
      g[r] = add(up, (int)tag_lds(addr[r]));
      ev[r] = kLocal ? __viaddmax_s32_relu(ev[r], ext, add(h, cE))
                     : __viaddmax_s32(ev[r], ext, add(h, cE));
      f = __viaddmax_s32(f, ext, add(h, cF));
      up = h;
      // the column's best, the smallest row first
      if constexpr (kLocal) {
        const int y = add(h, R - 1 - r);
        if (r & 1)
          cm = __vimax3_s32(cm, prev, y);
        else
          prev = y;
      }
      if (kCheck && !kLocal) hc[r] = h;
      if (r & 1)
        w[r / 2] = __byte_perm((uint32_t)xp, (uint32_t)x, 0x5410);
      else
        xp = x;
    }
    hbot = up;
    fbot = f;
    uint4* at = trace + (size_t)t * 128 + lane;
#pragma unroll
    for (int k = 0; k < R / 8; ++k)
      at[k * 32] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    if constexpr (R % 8 != 0)
      *reinterpret_cast<uint2*>(at + R / 8 * 32) = make_uint2(w[R / 8 * 4], w[R / 8 * 4 + 1]);
    if constexpr (kLocal) {
      if ((cm >> 16) > best) {  // padding rows hold 0: never above best
        best = cm >> 16;
        bi = s * R + (R - 1 - (cm & 0xffff)) - pad + 1;
        bj = j + 1;
      }
    } else {
      if (!kCheck || j < m - 1) {
        if (s == S - 1 && (up >> 16) + 1 > best) {  // the last row
          best = (up >> 16) + 1;
          bi = (int)n;
          bj = j + 1;
        }
      } else if constexpr (kCheck) {
#pragma unroll
        for (int r = 0; r < R; ++r)  // the last column, rows in order
          if (r >= padrows && (hc[r] >> 16) + 1 > best) {
            best = (hc[r] >> 16) + 1;
            bi = s * R + r - pad + 1;
            bj = m;
          }
      }
    }
  };
  auto top = [&](int& ht, int& ft) {
    ht = __shfl_up_sync(kFullT, hbot, 1);
    ft = __shfl_up_sync(kFullT, fbot, 1);
    if (first) {
      ht = kZero;
      ft = ftop;
    }
  };
  int t = 0;
  const int fill = smax - 1;
  if (fill < full) {
#pragma unroll 1
    for (; t < fill; ++t) {
      int ht, ft;
      top(ht, ft);
      const int j = t - s;
      if (valid && (unsigned)j < (unsigned)m) column(TagCheck<true>{}, t, j, ht, ft);
    }
#pragma unroll 1
    for (; t < full; ++t) {
      int ht, ft;
      top(ht, ft);
      column(TagCheck<false>{}, t, t - s, ht, ft);
    }
  }
#pragma unroll 1
  for (; t < steps; ++t) {
    int ht, ft;
    top(ht, ft);
    const int j = t - s;
    if (valid && (unsigned)j < (unsigned)m) column(TagCheck<true>{}, t, j, ht, ft);
  }
  __syncwarp();  // trace writes visible to the warp
  // --- the job's end cell: first maximum over its lanes
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int b2 = __shfl_up_sync(kFullT, best, d);
    const int j2 = __shfl_up_sync(kFullT, bj, d);
    const int i2 = __shfl_up_sync(kFullT, bi, d);
    if (valid && s >= d && better(b2, j2, i2, best, bj, bi)) {
      best = b2;
      bj = j2;
      bi = i2;
    }
  }
  // --- the walk, by the job's last lane.  Up to kAhead cells down the
  // diagonal at a time -- most steps are diagonal, and their loads then wait together
  // -- and one gap.  The walkers of a tile stay together: a branch a step for
  // each of them took as long as the columns (34 000 instructions a tile).
  const bool walker = valid && s == S - 1;
  int i = walker ? bi : 0, j = walker ? bj : 0;
  uint32_t* out = J.ops + (walker ? J.job_at[job] : 0ull);
  uint32_t runs = 0, cur = 4, cnt = 0;
  auto emit = [&](uint32_t op, uint32_t len) {
    const bool flush = len && op != cur;
    if (flush && cnt) out[runs] = (cnt << 4) | cur;
    runs += flush && cnt;
    cnt = (flush ? 0u : cnt) + len;
    cur = flush ? op : cur;
  };
  auto code = [&](int k) -> uint32_t {  // k cells down the diagonal; 0 past the border
    const int ip = i - k - 1 + pad, st = ip / R, r = ip - st * R;
    const uint4* cell = trace + (size_t)(j - k - 1 + st) * 128 + (r >> 3) * 32 + (s0 + st);
    return i > k && j > k ? (uint32_t)reinterpret_cast<const uint16_t*>(cell)[r & 7] : 0u;
  };
  while (__any_sync(kFullT, i > 0 && j > 0)) {
    uint32_t cell[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) cell[k] = code(k);
    int nm = 0;
    uint32_t c = 0xc000u;  // the first that is not diagonal
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      c = c >= 0xc000u ? cell[k] : c;
      nm += c >= 0xc000u;
    }
    emit(kOpM, (uint32_t)nm);
    i -= nm;
    j -= nm;
    const bool on = i > 0 && j > 0, ins = c >= 0x8000u, stop = on && c < 0x4000u;
    // (a gap from the border may count padding rows above the read)
    const int len = on && !stop && nm < kAhead ? min((int)(c & 0x3fffu) + 1, ins ? i : j) : 0;
    emit(ins ? kOpI : kOpD, (uint32_t)len);
    i -= ins ? len : 0;
    j -= ins ? 0 : len;
    if (__any_sync(kFullT, stop)) {
      if (stop) {  // the alignment starts here
        const bool none = bi == 0 || bj == 0;
        J.res[job] = none ? make_int4(0, 0, 0, 0) : make_int4(best, i, bi, j);
        i = -1;
      }
    }
  }
  if (walker) {
    if (cnt) out[runs++] = (cnt << 4) | cur;
    for (uint32_t a = 0, b = runs ? runs - 1 : 0; a < b; ++a, --b) {  // first to last
      const uint32_t x = out[a];
      out[a] = out[b];
      out[b] = x;
    }
    const bool none = bi == 0 || bj == 0;
    if (i >= 0) J.res[job] = none ? make_int4(0, 0, 0, 0) : make_int4(best, i, bi, j);
    J.res2[job] = make_int4(none ? 0 : bj, (int)runs, 0, 0);
  }
  __syncwarp();  // the walk is done before the scratch is reused
}

template <bool kLocal>
__global__ void __launch_bounds__(kTThreads, 3) k7_tags(const K7TagParams P) {
  __shared__ int4 tab[5];                   // words of read codes 0-3 against reference code x
  __shared__ uint32_t rec[6 * kTThreads];   // word c of thread t at c * kTThreads + t
  const int lane = threadIdx.x & 31;
  // a diagonal step's addend: the score and the source
  const int dg = kLocal ? -0x4000 : 0xc000;
  const int ma = P.J.ma * 65536 + dg, mi = P.J.mi * 65536 + dg;
  if (threadIdx.x < 5) {
    const int x = threadIdx.x;  // 4: a wildcard reference base matches every read code
    tab[x] = make_int4((x == 0 || x == 4) ? ma : mi, (x == 1 || x == 4) ? ma : mi,
                       (x == 2 || x == 4) ? ma : mi, (x == 3 || x == 4) ? ma : mi);
  }
  const uint32_t my = (uint32_t)__cvta_generic_to_shared(rec) + threadIdx.x * 4u;
  tag_sts(my + 4 * kTThreads * 4, (uint32_t)ma);  // read wildcard: a match everywhere
  tag_sts(my + 5 * kTThreads * 4, (uint32_t)dg);  // padding row: s = 0
  __syncthreads();
  uint4* trace = P.trace + ((size_t)blockIdx.x * kTWarps + (threadIdx.x >> 5)) *
                               (size_t)P.steps * 128;
  for (;;) {
    uint32_t task = 0;
    if (lane == 0) task = atomicAdd(P.J.task_counter, 1u);
    task = __shfl_sync(kFullT, task, 0);
    if (task >= P.J.n_tasks) break;
    const uint2 tk = P.J.tasks[task];
    if (tk.y & kTag28)
      tag_tile<28, kLocal>(P, tab, my, trace, tk);
    else
      tag_tile<32, kLocal>(P, tab, my, trace, tk);
  }
}

// ---------------------------------------------------------------- results
// The caller's records and packed words, made on the device: each block's
// words counted (k7_sums), then placed after the blocks before it (k7_pack).
// Copying the kernels' results out and walking the jobs on the host for the
// offsets, back up for the packing and again for the records took 1.3 ms a
// 100 000 jobs.
constexpr uint32_t kPackThreads = 256;
constexpr uint32_t kPackJobs = 4 * kPackThreads;  // jobs a block

__global__ void __launch_bounds__(kPackThreads) k7_sums(const int4* __restrict__ res2,
                                                        uint32_t n_jobs,
                                                        unsigned long long* __restrict__ sums) {
  __shared__ unsigned long long sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  uint32_t v = 0;
  for (uint32_t i = threadIdx.x; i < kPackJobs; i += kPackThreads) {
    const uint64_t k = (uint64_t)blockIdx.x * kPackJobs + i;
    if (k < n_jobs) v += (uint32_t)res2[k].y;
  }
  v = __reduce_add_sync(kFullT, v);
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, (unsigned long long)v);
  __syncthreads();
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kPackThreads) k7_pack(const int4* __restrict__ res,
                                                        const int4* __restrict__ res2,
                                                        uint32_t n_jobs,
                                                        const unsigned long long* __restrict__ sums,
                                                        const uint32_t* __restrict__ staging,
                                                        const uint64_t* __restrict__ at,
                                                        esg_alignment* __restrict__ rec,
                                                        uint32_t* __restrict__ words) {
  __shared__ unsigned long long before;
  __shared__ uint32_t warp_sum[kPackThreads / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  unsigned long long b = 0;
  for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kPackThreads) b += sums[i];
  if (b) atomicAdd(&before, b);
  const uint64_t k0 = (uint64_t)blockIdx.x * kPackJobs + 4 * threadIdx.x;
  int4 r2[4];
  uint32_t mine = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    r2[i] = k0 + i < n_jobs ? res2[k0 + i] : make_int4(0, 0, 0, 0);
    mine += (uint32_t)r2[i].y;
  }
  uint32_t incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(kFullT, incl, d);
    if (lane >= (uint32_t)d) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  unsigned long long o = before + incl - mine;
  for (uint32_t w = 0; w < warp; ++w) o += warp_sum[w];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t k = k0 + i;
    if (k >= n_jobs) break;
    const int4 r = res[k];
    const uint32_t nr = (uint32_t)r2[i].y;
    rec[k] = {r.x, (uint32_t)r.y, (uint32_t)r.z, (uint32_t)r.w, (uint32_t)r2[i].x, nr, o};
    const uint32_t* src = staging + at[k];
    for (uint32_t w = 0; w < nr; ++w) words[o + w] = src[w];
    o += nr;
  }
}

esg_status terr(esg_status st, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  esg_internal_set_error(st, buf);
  return st;
}

#define TCUDA(call)                                                          \
  do {                                                                       \
    cudaError_t e_ = (call);                                                 \
    if (e_ != cudaSuccess) {                                                 \
      if (mem) cudaFreeAsync(mem, st);                                       \
      return terr(ESG_ERR_DRIVER, "%s: %s", #call, cudaGetErrorString(e_));  \
    }                                                                        \
  } while (0)

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// Align the jobs against reads already on the device.
esg_status align_impl(esg_scorer* sc, const uint8_t* d_codes, const uint64_t* d_off,
                      const uint32_t* d_len, uint32_t n_reads, const uint32_t* h_len,
                      const esg_align_job* jobs, uint32_t n_jobs, esg_alignment* out,
                      uint32_t* ops, uint64_t ops_capacity, uint64_t* ops_needed,
                      std::vector<uint32_t>* grow = nullptr, cudaStream_t stream = nullptr) {
  esg_internal_panel P{};
  esg_internal_panel_of(sc, &P);
  if (n_jobs && (!jobs || !out)) return terr(ESG_ERR_BAD_ARGUMENT, "jobs/out must not be NULL");
  // --- plan on the host
  std::vector<uint32_t> job_q(n_jobs), job_slot(n_jobs), S(n_jobs);
  std::vector<uint64_t> job_at(n_jobs);
  uint64_t staging = 0;
  uint32_t mcols = 1, passes_max = 1, tag_cols = 1, tag_stripes = 1;
  uint32_t all_cols = 1, all_passes = 1;  // over every job, as k7_trace would hold them
  // jobs by kernel and stripe height: k7_tags on 28 and 32 rows, k7_trace
  enum { kT28, kT32, kFull, kKinds };
  std::vector<uint32_t> live[kKinds];
  live[kT28].reserve(n_jobs);
  live[kT32].reserve(n_jobs);
  const int64_t mm = std::max(std::abs(P.scoring.match_score), std::abs(P.scoring.mismatch)),
                go = std::abs(P.scoring.gap_open), ge = std::abs(P.scoring.gap_extend);
  for (uint32_t k = 0; k < n_jobs; ++k) {
    const esg_align_job& jb = jobs[k];
    if (jb.read >= n_reads) return terr(ESG_ERR_BAD_ARGUMENT, "job %u: no read %u", k, jb.read);
    if (jb.ref >= P.n_refs) return terr(ESG_ERR_BAD_ARGUMENT, "job %u: no reference %u", k, jb.ref);
    if (jb.reverse > 1) return terr(ESG_ERR_BAD_ARGUMENT, "job %u: reverse must be 0 or 1", k);
    const uint32_t n = h_len[jb.read], m = P.len_of[jb.ref];
    job_q[k] = jb.read | (jb.reverse << 31);
    job_slot[k] = P.slot_of[jb.ref];
    job_at[k] = staging;
    staging += (uint64_t)n + m + 1;
    S[k] = (n + kTR - 1) / kTR;
    if (S[k] > 0xffffu) return terr(ESG_ERR_BAD_ARGUMENT, "job %u: read too long", k);
    if (!n || !m) continue;
    all_cols = std::max(all_cols, m);
    all_passes = std::max(all_passes, (S[k] + 31) / 32);
    if (n <= kTagRows && m <= kTagCols &&
        (int64_t)std::min(n, m) * (mm + ge) + 2 * go + mm <= kTagScore) {
      // 28-row stripes where they pad enough less (a row costs 1.045 of a
      // 32-row stripe's in the scoring kernel, whose loop this is)
      const bool r28 = n <= 28 * 8 && (n + 27) / 28 * 28 * 1045 < (n + 31) / 32 * 32 * 1000;
      S[k] = r28 ? (n + 27) / 28 : (n + 31) / 32;
      live[r28 ? kT28 : kT32].push_back(k);
      tag_stripes = std::max(tag_stripes, S[k]);
      tag_cols = std::max(tag_cols, m);
    } else {
      live[kFull].push_back(k);
      mcols = std::max(mcols, m);
      if (S[k] > 32) passes_max = std::max(passes_max, (S[k] + 31) / 32);
    }
  }
  // tiles of jobs up to 32 stripes (next fit, longest first); longer jobs
  // alone.  Tasks of a kernel lie together: k7_tags' first.
  std::vector<uint32_t> order;
  std::vector<uint2> tasks;
  order.reserve(n_jobs);
  uint32_t n_tag = 0;
  for (int kind = 0; kind < kKinds; ++kind) {
    if (kind == kFull) n_tag = (uint32_t)tasks.size();
    std::vector<uint32_t>& lv = live[kind];
    if (lv.empty()) continue;
    // longest first, stable: a counting sort on the stripes (long jobs, over
    // 32 stripes, are few and sorted apart).  k7_tags' jobs by reference
    // length before that: a tile runs for its longest reference, and with
    // references of 70-180 nt in any order 30 % of its lanes' steps were idle
    std::vector<uint32_t> cnt(34, 0), start(34, 0), sorted(lv.size());
    if (kind != kFull) {
      std::vector<uint32_t> first(tag_cols + 2, 0);
      auto len = [&](uint32_t k) { return P.len_of[jobs[k].ref]; };
      for (uint32_t k : lv) ++first[tag_cols - len(k) + 1];
      for (uint32_t v = 1; v < tag_cols + 2; ++v) first[v] += first[v - 1];
      for (uint32_t k : lv) sorted[first[tag_cols - len(k)]++] = k;
      lv.swap(sorted);
    }
    for (uint32_t k : lv) ++cnt[std::min<uint32_t>(S[k], 33)];
    uint32_t at = 0;
    for (int v = 33; v >= 1; --v) {
      start[v] = at;
      at += cnt[v];
    }
    for (uint32_t k : lv) sorted[start[std::min<uint32_t>(S[k], 33)]++] = k;
    std::stable_sort(sorted.begin(), sorted.begin() + cnt[33],
                     [&](uint32_t a, uint32_t b) { return S[a] > S[b]; });
    const uint32_t mark = kind == kT28 ? kTag28 : 0u;
    uint32_t open_start = 0, open_count = 0, open_free = 0, open_smax = 0;
    auto close_tile = [&]() {
      if (open_count) tasks.push_back(make_uint2(open_start, open_count | mark | (open_smax << 16)));
      open_count = 0;
    };
    for (uint32_t k : sorted) {
      if (S[k] > 32) {
        tasks.push_back(make_uint2((uint32_t)order.size(), 1u | (S[k] << 16)));
        order.push_back(k);
        continue;
      }
      if (!open_count || S[k] > open_free) {
        close_tile();
        open_start = (uint32_t)order.size();
        open_free = 32;
        open_smax = S[k];
      }
      order.push_back(k);
      open_free -= S[k];
      ++open_count;
    }
    close_tile();
  }
  const uint32_t n_full = (uint32_t)tasks.size() - n_tag;
  const uint32_t n_tasks = (uint32_t)tasks.size();

  // --- geometry and scratch: per warp passes x columns x 32 lanes of 8 B,
  // capped at 4 GiB in all
  if ((size_t)all_passes * all_cols * 32 * 8 > (1ull << 30))
    return terr(ESG_ERR_BAD_ARGUMENT,
                "a job of %u stripes x %u columns needs over 1 GiB of trace per warp",
                all_passes * 32, all_cols);
  const size_t trace_words = (size_t)passes_max * mcols * 32;
  cudaSetDevice(P.device);
  const bool local = P.mode == ESG_MODE_LOCAL;
  const void* fn = local ? (const void*)k7_trace<true> : (const void*)k7_trace<false>;
  const void* tag_fn = local ? (const void*)k7_tags<true> : (const void*)k7_tags<false>;
  auto grid = [&](const void* f, uint32_t n, size_t warp_bytes, uint64_t most) -> uint64_t {
    if (!n) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kTThreads, 0) != cudaSuccess)
      per_sm = 1;
    uint64_t w = std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * P.sm_count * kTWarps, n);
    w = std::min<uint64_t>(w, std::max<uint64_t>(kTWarps, most / warp_bytes / kTWarps * kTWarps));
    return (w + kTWarps - 1) / kTWarps;
  };
  const uint32_t tag_steps = tag_cols + tag_stripes - 1;
  const size_t tag_bytes = (size_t)tag_steps * 128 * sizeof(uint4);
  const uint64_t blocks = grid(fn, n_full, trace_words * 8, 4ull << 30);
  // k7_tags' scratch: the least of 512 MiB, 1 and 2 GiB that holds four warps
  // an SM, in eighths of it (what the shared pool keeps then fits the next
  // call, whose jobs need a little more)
  uint64_t tag_room = kTagBytes / 4;
  while (tag_room < kTagBytes && tag_room / tag_bytes < 4ull * P.sm_count) tag_room *= 2;
  const uint64_t tag_blocks = grid(tag_fn, n_tag, tag_bytes, tag_room);
  const uint64_t tag_need = tag_blocks * kTWarps * tag_bytes;
  const uint64_t tag_alloc = (tag_need + tag_room / 8 - 1) / (tag_room / 8) * (tag_room / 8);
  const uint64_t warps = blocks * kTWarps;
  const size_t scratch = warps * trace_words * 8;

  const size_t nj = std::max<uint32_t>(n_jobs, 1);
  const uint32_t pack_blocks = (uint32_t)((nj + kPackJobs - 1) / kPackJobs);
  const size_t sizes[] = {
      align256(nj * 4),                          // job_q
      align256(nj * 4),                          // job_slot
      align256(nj * 8),                          // job_at
      align256(std::max<size_t>(order.size(), 1) * 4),
      align256(std::max<uint32_t>(n_tasks, 1) * 8),
      align256(8),                               // task counters
      align256(nj * 16),                         // res
      align256(nj * 16),                         // res2
      align256(std::max<uint64_t>(staging, 1) * 4),
      align256(scratch),
      align256(warps * (size_t)mcols * 8),
      align256(nj * sizeof(esg_alignment)),
      align256(pack_blocks * 8),                 // words per block
  };
  size_t total = 0;
  for (size_t v : sizes) total += v;
  cudaStream_t st = stream ? stream : P.stream;
  void* mem = nullptr;
  TCUDA(cudaMallocFromPoolAsync(&mem, total, P.pool, st));
  char* at = (char*)mem;
  auto take = [&](size_t i) {
    char* p = at;
    at += sizes[i];
    return p;
  };
  uint32_t* d_job_q = (uint32_t*)take(0);
  uint32_t* d_job_slot = (uint32_t*)take(1);
  uint64_t* d_job_at = (uint64_t*)take(2);
  uint32_t* d_order = (uint32_t*)take(3);
  uint2* d_tasks = (uint2*)take(4);
  uint32_t* d_counter = (uint32_t*)take(5);
  int4* d_res = (int4*)take(6);
  int4* d_res2 = (int4*)take(7);
  uint32_t* d_staging = (uint32_t*)take(8);
  uint2* d_trace = (uint2*)take(9);
  uint2* d_colbuf = (uint2*)take(10);
  esg_alignment* d_rec = (esg_alignment*)take(11);
  unsigned long long* d_sums = (unsigned long long*)take(12);
  if (n_jobs) {
    TCUDA(cudaMemcpyAsync(d_job_q, job_q.data(), n_jobs * 4, cudaMemcpyHostToDevice, st));
    TCUDA(cudaMemcpyAsync(d_job_slot, job_slot.data(), n_jobs * 4, cudaMemcpyHostToDevice, st));
    TCUDA(cudaMemcpyAsync(d_job_at, job_at.data(), n_jobs * 8, cudaMemcpyHostToDevice, st));
  }
  if (!order.empty())
    TCUDA(cudaMemcpyAsync(d_order, order.data(), order.size() * 4, cudaMemcpyHostToDevice, st));
  if (n_tasks)
    TCUDA(cudaMemcpyAsync(d_tasks, tasks.data(), n_tasks * 8, cudaMemcpyHostToDevice, st));
  TCUDA(cudaMemsetAsync(d_counter, 0, 8, st));
  TCUDA(cudaMemsetAsync(d_res, 0, nj * 16, st));   // empty jobs stay all zero
  TCUDA(cudaMemsetAsync(d_res2, 0, nj * 16, st));
  if (n_tasks) {
    K7Params K{};
    K.codes = d_codes;
    K.off = d_off;
    K.len = d_len;
    K.rcodes = P.rcodes;
    K.roff = P.roff;
    K.rlen = P.rlen;
    K.job_q = d_job_q;
    K.job_slot = d_job_slot;
    K.job_at = d_job_at;
    K.order = d_order;
    K.tasks = d_tasks;
    K.trace = d_trace;
    K.trace_words = trace_words;
    K.mcols = mcols;
    K.colbuf = d_colbuf;
    K.ma = P.scoring.match_score;
    K.mi = P.scoring.mismatch;
    K.o = P.scoring.gap_open;
    K.e = P.scoring.gap_extend;
    K.res = d_res;
    K.res2 = d_res2;
    K.ops = d_staging;
    if (n_tag) {
      // its scratch comes from a pool the device's scorers share: mapping it
      // anew for each of them took longer (25 ms for 0.6 GB) than the tracing.
      // Small scratch from the scorer's own: making the shared pool takes 0.3 ms
      // of a first call (1000 jobs: 0.8 ms, 1.2 with it)
      const bool own = tag_need <= kTagOwn;
      cudaMemPool_t pool = own ? P.pool : esg_internal_trace_pool(P.device, kTagBytes, P.pool);
      uint64_t ctas = tag_blocks, bytes = own ? tag_need : tag_alloc;
      uint4* d_tags = nullptr;
      cudaError_t e = cudaMallocFromPoolAsync((void**)&d_tags, bytes, pool, st);
      while (e == cudaErrorMemoryAllocation && ctas > 1) {
        cudaGetLastError();  // short of memory: fewer warps take the tasks
        ctas = (ctas + 1) / 2;
        bytes = ctas * kTWarps * tag_bytes;
        e = cudaMallocFromPoolAsync((void**)&d_tags, bytes, pool, st);
      }
      TCUDA(e);
      K7TagParams T{K, d_tags, tag_steps, 1};
      T.J.n_tasks = n_tag;
      T.J.task_counter = d_counter;
      void* args[] = {&T};
      e = cudaLaunchKernel(tag_fn, dim3((unsigned)ctas), dim3(kTThreads), args, 0, st);
      cudaFreeAsync(d_tags, st);
      TCUDA(e);
    }
    if (n_full) {
      K.tasks = d_tasks + n_tag;
      K.n_tasks = n_full;
      K.task_counter = d_counter + 1;
      void* args[] = {&K};
      TCUDA(cudaLaunchKernel(fn, dim3((unsigned)blocks), dim3(kTThreads), args, 0, st));
    }
  }
  // --- how many words there are, then records and words packed
  k7_sums<<<pack_blocks, kPackThreads, 0, st>>>(d_res2, n_jobs, d_sums);
  TCUDA(cudaGetLastError());
  std::vector<uint64_t> sums(pack_blocks);
  TCUDA(cudaMemcpyAsync(sums.data(), d_sums, pack_blocks * 8, cudaMemcpyDeviceToHost, st));
  TCUDA(cudaStreamSynchronize(st));
  uint64_t need = 0;
  for (uint64_t v : sums) need += v;
  if (ops_needed) *ops_needed = need;
  if (grow) {
    grow->resize(need);
    ops = grow->data();
    ops_capacity = need;
  }
  if (need > ops_capacity || (need && !ops)) {
    cudaFreeAsync(mem, st);
    return terr(ESG_ERR_BAD_ARGUMENT, "the alignments need %llu CIGAR words, room for %llu",
                (unsigned long long)need, (unsigned long long)ops_capacity);
  }
  if (n_jobs) {
    uint32_t* d_out = nullptr;
    if (need) TCUDA(cudaMallocFromPoolAsync((void**)&d_out, need * 4, P.pool, st));
    k7_pack<<<pack_blocks, kPackThreads, 0, st>>>(d_res, d_res2, n_jobs, d_sums, d_staging,
                                                  d_job_at, d_rec, d_out);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(out, d_rec, n_jobs * sizeof(esg_alignment), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && need)
      e = cudaMemcpyAsync(ops, d_out, need * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (d_out) cudaFreeAsync(d_out, st);
    TCUDA(e);
  }
  cudaFreeAsync(mem, st);
  esg_internal_set_error(ESG_OK, "");
  return ESG_OK;
}

}  // namespace

esg_status esg_internal_align_batch(esg_scorer* sc, esg_batch* b, const esg_align_job* jobs,
                                    uint32_t n_jobs, esg_alignment* out,
                                    std::vector<uint32_t>* ops, cudaStream_t stream) {
  const uint8_t* codes = nullptr;
  const uint64_t* off = nullptr;
  const uint32_t* len = nullptr;
  const uint32_t* h_len = nullptr;
  uint32_t n_reads = 0;
  esg_internal_batch_reads(b, &codes, &off, &len, &n_reads, &h_len);
  if (!codes) return terr(ESG_ERR_BAD_ARGUMENT, "the batch is not submitted");
  return align_impl(sc, codes, off, len, n_reads, h_len, jobs, n_jobs, out, nullptr, 0, nullptr,
                    ops, stream);
}

extern "C" {

esg_status esg_align_batch(esg_scorer* sc, esg_batch* b, const esg_align_job* jobs,
                           uint32_t n_jobs, esg_alignment* out, uint32_t* ops,
                           uint64_t ops_capacity, uint64_t* ops_needed) {
  if (!sc || !b) return terr(ESG_ERR_BAD_ARGUMENT, "NULL scorer or batch");
  const uint8_t* codes = nullptr;
  const uint64_t* off = nullptr;
  const uint32_t* len = nullptr;
  const uint32_t* h_len = nullptr;
  uint32_t n_reads = 0;
  esg_internal_batch_reads(b, &codes, &off, &len, &n_reads, &h_len);
  if (!codes) return terr(ESG_ERR_BAD_ARGUMENT, "the batch is not submitted");
  return align_impl(sc, codes, off, len, n_reads, h_len, jobs, n_jobs, out, ops, ops_capacity,
                    ops_needed);
}

esg_status esg_align_reads(esg_scorer* sc, const uint8_t* codes, const uint64_t* off,
                           const uint32_t* len, uint32_t n_reads, const esg_align_job* jobs,
                           uint32_t n_jobs, esg_alignment* out, uint32_t* ops,
                           uint64_t ops_capacity, uint64_t* ops_needed) {
  if (!sc) return terr(ESG_ERR_BAD_ARGUMENT, "NULL scorer");
  if (n_reads && (!off || !len)) return terr(ESG_ERR_BAD_ARGUMENT, "off/len must not be NULL");
  esg_internal_panel P{};
  esg_internal_panel_of(sc, &P);
  // the reads to the device (no scoring): packed first, unless they already
  // lie one after the other
  std::vector<uint64_t> poff(std::max<uint32_t>(n_reads, 1), 0);
  uint64_t total = 0;
  bool together = true;
  for (uint32_t k = 0; k < n_reads; ++k) {
    poff[k] = total;
    together = together && off[k] == off[0] + total;
    total += len[k];
  }
  if (total && !codes) return terr(ESG_ERR_BAD_ARGUMENT, "codes must not be NULL");
  std::vector<uint8_t> pc;
  const uint8_t* src = nullptr;
  if (total && together) {
    src = codes + off[0];
  } else if (total) {
    pc.resize(total);
    for (uint32_t k = 0; k < n_reads; ++k)
      if (len[k]) memcpy(pc.data() + poff[k], codes + off[k], len[k]);
    src = pc.data();
  }
  cudaSetDevice(P.device);
  cudaStream_t st = P.stream;
  const size_t b0 = align256(std::max<uint64_t>(total, 1)), b1 = align256(poff.size() * 8),
               b2 = align256(std::max<uint32_t>(n_reads, 1) * 4);
  void* mem = nullptr;
  TCUDA(cudaMallocFromPoolAsync(&mem, b0 + b1 + b2, P.pool, st));
  uint8_t* d_codes = (uint8_t*)mem;
  uint64_t* d_off = (uint64_t*)((char*)mem + b0);
  uint32_t* d_len = (uint32_t*)((char*)mem + b0 + b1);
  if (total) TCUDA(cudaMemcpyAsync(d_codes, src, total, cudaMemcpyHostToDevice, st));
  TCUDA(cudaMemcpyAsync(d_off, poff.data(), poff.size() * 8, cudaMemcpyHostToDevice, st));
  if (n_reads) TCUDA(cudaMemcpyAsync(d_len, len, n_reads * 4, cudaMemcpyHostToDevice, st));
  const esg_status s = align_impl(sc, d_codes, d_off, d_len, n_reads, len, jobs, n_jobs, out,
                                  ops, ops_capacity, ops_needed);
  cudaFreeAsync(mem, st);
  cudaStreamSynchronize(st);
  return s;
}

}  // extern "C"
