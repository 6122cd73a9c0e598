// Tensor-core form of the polyphase engine (tcgen05 + TMA, sm_103a).
//
// The fused shift + polyphase contraction of the decimation groups of an
// apply runs as persistent launches of matrix products over 128-row tiles,
// one per launch pack (as many groups as the launch records hold; the
// planner, fdsp_tc_plan.h, describes the operands):
//
//     Y[j][n] = sum_k A[j][k] B[k][n]
//
//   A  input samples j D' + a + k of [history | block] as 16-bit {hi, lo}
//      parts (4 K elements a sample), loaded 16 samples at a time by TMA
//      into the 128-byte-swizzled K-major layout: a tensor map whose rows
//      are D' samples apart (rows overlap when D' < 16) turns the Hankel
//      matrix of each tile into one TMA copy per K chunk, no staging code;
//   B  the NCO-modulated taps of the merge set's output streams ("slots"),
//      hi taps in the first half of the columns and lo taps in the second,
//      prebuilt per apply in the same swizzled image and copied per chunk;
//   Y  FP32 in tensor memory; the epilogue adds the hi and lo halves,
//      rotates by the NCO phase of each window start (exact integer phase)
//      and stores.  Windows across the NCO rollover are stored unrotated and
//      rotated exactly (split sum) by tc_fix_kernel, launched after the
//      filter bank: keeping that rare path out of the filter-bank kernel
//      roughly halved its MMA issue time.
//
// Per CTA (one per SM, 608 threads):
//   warp 0      producer: takes the CTA's items from the scheduler's queue
//               and announces each in a ring with its first stage; per
//               item (R tiles of one merge set) and K chunk,
//               waits for a free stage, then R TMA tile loads of A and one
//               bulk copy of the B chunk, completing on the stage barrier;
//   warp 1      MMA issuer: per chunk 4 MMAs (K = 16) per tile into the
//               item's accumulator slot, commit frees the stage; the last
//               chunk's commit hands the slot to the epilogue;
//   warps 2-17  epilogue: four warps per TMEM lane quarter; each reads its
//               (at most two) neighbouring 8-slot column chunks out of tensor memory,
//               releases the slot, then rotates and stores;
//   warp 18     scheduler: queues the CTA's items for warp 0, from the list
//               that the prep kernel sorted by first input sample.
// Warps 0 and 1 run their loops in lane 0 alone.
// Two accumulator slots of 256 columns (R tiles x N columns each) let the
// MMAs of one item run while the epilogue drains the previous one.
//
// The items of every merge set are listed in input order and cut into one run
// of equal cost per CTA, so the split input is read from HBM about once and
// every group reuses it from L2.
//
// Every mbarrier wait is bounded (TcLaunch::poll); a wait that runs out sets
// the error flag (mapped host memory, read by fdsp_channelizer_status),
// drains the copies and MMAs this CTA issued and exits.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fdsp_internal.h"
#include "fdsp_nco.cuh"
#include "fdsp_tc.cuh"

namespace fdsp {

constexpr int kTcEpiPerQ = kTcEpiWarps / 4;           // epilogue warps per TMEM lane quarter
constexpr int kTcEpiOwn = 8 / kTcEpiPerQ;             // most column chunks a warp reads per item (R NS <= 64)
constexpr int kTcSchedWarp = 2 + kTcEpiWarps;         // the item scheduler (after the epilogue warps)
constexpr int kTcThreads = 96 + 32 * kTcEpiWarps;     // producer, MMA, epilogue and scheduler warps
constexpr int kTcRing = 16;                           // items announced ahead (> stages + 2)
constexpr int kTcQueue = 64;                          // items the scheduler warp finds ahead
constexpr uint32_t kTmemCols = 512;

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
template <int FMT>
__device__ __forceinline__ void split2(float2 x, uint32_t& hi, uint32_t& lo) {
  if constexpr (FMT == 0) {
    const __half2 h = __float22half2_rn(x);
    const float2 hf = __half22float2(h);
    const __half2 l = __float22half2_rn(make_float2(x.x - hf.x, x.y - hf.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  } else {
    const __nv_bfloat162 h = __float22bfloat162_rn(x);
    const float2 hf = __bfloat1622float2(h);
    const __nv_bfloat162 l = __float22bfloat162_rn(make_float2(x.x - hf.x, x.y - hf.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  }
}

__device__ __forceinline__ float2 tc_load_x(const TcLaunch& L, int64_t v) {
  if (v < 0) {
    const int64_t hv = v + L.H;
    return hv >= 0 ? L.hist[hv] : make_float2(0.f, 0.f);
  }
  if (v >= L.N) return make_float2(0.f, 0.f);
  if (L.block16 != nullptr) {
    const short2 s = L.block16[v];
    return make_float2((float)s.x, (float)s.y);
  }
  return __ldg(L.block + v);
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: 8-row atoms of
// 128-byte rows 1024 bytes apart (stride byte offset), version 1, layout 2.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) |
         ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int32_t x, int32_t y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(tc::smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Position in the stage ring: stage s of round r (chunk r * stages + s),
// advanced without a division per chunk.
struct TcRing {
  int s = 0, r = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) {
      s = 0;
      ++r;
    }
  }
};

// ---------------------------------------------------------------------------
// prep: split [history | block] into {hi, lo} parts, build the B images and
// the item list
// ---------------------------------------------------------------------------
// B image of merge set m, chunk c: N = 4 NS rows (columns of B) of 128
// bytes, the 16-byte piece q of row n (taps 2q, 2q + 1 of the chunk) at
// (q ^ (n & 7)) 16, the 128-byte swizzle of a 1024-byte-aligned atom.
// Column n: hi/lo half h = n / (2 NS), slot s = (n mod 2 NS) / 2, part
// p = n & 1 (Re, Im).  For the input elements (x_re, x_im) of either half
// (hi or lo) the Re column holds (g_re, -g_im) and the Im column (g_im, g_re)
// of the tap's hi or lo part.
template <int FMT>
__global__ void __launch_bounds__(256) tc_prep_kernel(const __grid_constant__ TcLaunch L, int nb_build) {
  if (blockIdx.x == 0) {  // the record, for the filter-bank kernel
    const uint4* src = reinterpret_cast<const uint4*>(&L);
    uint4* dst = reinterpret_cast<uint4*>(L.rec_out);
    for (int i = (int)threadIdx.x; i < (int)(sizeof(TcLaunch) / 16); i += 256) dst[i] = src[i];
  }
  if ((int)blockIdx.x < nb_build) {
    const int total = L.bprefix[L.nmsets];
    for (int p = (int)blockIdx.x * 256 + (int)threadIdx.x; p < total; p += nb_build * 256) {
      int lo = 0, hi = L.nmsets;  // largest m with bprefix[m] <= p
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (L.bprefix[mid] <= p) lo = mid;
        else hi = mid;
      }
      const TcMset& M = L.ms[lo];
      const int NS = M.NS, N = 4 * NS;
      const int lp = p - L.bprefix[lo];
      const int c = lp / (N * 8);
      const int rem = lp - c * N * 8;
      const int n = rem >> 3, q = rem & 7;
      const int h = n / (2 * NS);
      const int s = (n - h * 2 * NS) >> 1, part = n & 1;
      const TcSlot& S = L.slots[M.slot0 + s];
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (S.J > 0) {
        const float2* g = L.ctaps[S.ch] + (size_t)S.phi * S.T;
        for (int u = 0; u < 2; ++u) {
          const int t = c * kTcChunkTaps + 2 * q + u - (int)S.o;
          if (t < 0 || t >= (int)S.T) continue;
          uint32_t gh, gl;
          split2<FMT>(__ldg(g + t), gh, gl);
          const uint32_t v = h ? gl : gh;  // {re, im} of the tap's hi or lo part
          const uint32_t re = v & 0xFFFFu, im = v >> 16;
          const uint32_t e0 = part ? (im | (re << 16)) : (re | ((im ^ 0x8000u) << 16));
          w[2 * u] = e0;       // x_hi elements
          w[2 * u + 1] = e0;   // x_lo elements
        }
      }
      uint8_t* dst = L.bbuf + M.b + ((size_t)c * N + n) * 128 + (size_t)((q ^ (n & 7)) * 16);
      *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    // the items in the order of their first input sample, each with the cost
    // of all items before it
    const int nitems = L.iprefix[L.nmsets];
    for (int p = (int)blockIdx.x * 256 + (int)threadIdx.x; p < nitems; p += nb_build * 256) {
      int m = 0, hi = L.nmsets;  // largest m with iprefix[m] <= p
      while (hi - m > 1) {
        const int mid = (m + hi) >> 1;
        if (L.iprefix[mid] <= p) m = mid;
        else hi = mid;
      }
      const int t = p - L.iprefix[m];
      uint32_t place, cost;
      tc_item_place(L.ms, L.nmsets, L.groups, m, t, L.cost_shift, &place, &cost);
      L.items[place] = make_uint2(((uint32_t)m << 26) | (uint32_t)t, cost);
    }
    return;
  }
  const int64_t stride = (int64_t)(gridDim.x - nb_build) * 256;
  const int64_t NH = L.N + L.H;
  for (int64_t u = (int64_t)(blockIdx.x - nb_build) * 256 + threadIdx.x; u < L.xhl_n; u += stride) {
    float2 x = make_float2(0.f, 0.f);
    if (u < L.H) {
      x = L.hist[u];
    } else if (u < NH) {
      if (L.block16 != nullptr) {
        const short2 s = L.block16[u - L.H];
        x = make_float2((float)s.x, (float)s.y);
      } else {
        x = L.block[u - L.H];
      }
    }
    uint2 hl;
    split2<FMT>(x, hl.x, hl.y);
    L.xhl[u] = hl;
  }
}

// ---------------------------------------------------------------------------
// epilogue constants and the exact NCO path
// ---------------------------------------------------------------------------
// Per-slot epilogue constants, staged in shared memory at CTA start (read
// with warp-uniform addresses: broadcasts, no constant-cache traffic).
struct TcEpiSlot {
  uint64_t out;   // float2*: output of row 0
  uint64_t om;    // NCO turns per sample (2^-64 units); 0: no rotation
  uint64_t fm;    // ceil(2^64 / R): (a mod R) as one multiply-high (Lemire et al. 2019)
  int64_t x0;     // NCO counter argument of row 0's window start (base + w0, unreduced)
  uint32_t R;     // counter rollover; 0: every output takes the exact path
  int32_t J;      // rows with an output
  uint32_t stride;  // bytes from an output to the next row's
  uint16_t flags;   // how its outputs are stored (TcSlot::flags the addresses allow)
  uint16_t Tm1;     // taps - 1
};
static_assert(sizeof(TcEpiSlot) == kTcEpiSlotBytes, "epilogue slot table layout");
static_assert(offsetof(TcEpiSlot, om) == 8 && offsetof(TcEpiSlot, fm) == 16 && offsetof(TcEpiSlot, x0) == 24 &&
                  offsetof(TcEpiSlot, R) == 32 && offsetof(TcEpiSlot, J) == 36 && offsetof(TcEpiSlot, stride) == 40 &&
                  offsetof(TcEpiSlot, flags) == 44 && offsetof(TcEpiSlot, Tm1) == 46,
              "the epilogue reads a slot's table entry as three 16-byte parts");

// What a warp needs of a slot for one block of 32 rows: made by one lane per
// slot, read by every lane as 16-byte broadcasts.
//   {address of the first row's output, row stride in bytes, scratch address}
//   {counter of the first row, turns per sample (64 bits), -}
//   {rollover, counters below this do not straddle it, rows (0-32), -}
constexpr uint32_t kTcRec = 48;
static_assert(kTcEpiRecs == 16 * (int)kTcRec && kTcEpiRows == 2048, "epilogue scratch: 32 rows x 8 outputs, 16 records");

// Outputs whose window crosses the NCO rollover (or whose counter leaves the
// fast path's 32-bit range) were stored unrotated; rotate_prep/rotate_apply
// split the window sum at the rollover exactly, from the FP32 modulated taps.
__device__ __noinline__ void tc_fix_exact(const TcLaunch& L, int slot, int64_t j, int64_t D, float2* dst) {
  const TcSlot& S = L.slots[slot];
  const NcoConst nc = L.nco[S.ch];
  OutMeta cm;
  cm.omega64 = nc.omega64;
  cm.wrap64 = nc.wrap64;
  cm.fastmod = nc.fastmod;
  cm.out = nullptr;
  cm.rollover = nc.rollover;
  cm.base = L.nco_base[S.ch];
  cm.enabled = nc.enabled;
  cm.step32 = 0;
  const int64_t w0 = (int64_t)S.w0 + j * D;
  const ExactRot er = rotate_prep(cm, w0, S.T);
  float2 B = make_float2(0.f, 0.f);
  if (er.straddle) {
    const float2* g = L.ctaps[S.ch] + (size_t)S.phi * S.T;
    // eight taps' loads in flight at a time (one after another, each tap cost
    // a memory latency); the sum runs in tap order
    for (int k = er.k0; k < (int)S.T; k += 8) {
      float2 x[8], gk[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = min(k + i, (int)S.T - 1);
        x[i] = tc_load_x(L, w0 + t);
        gk[i] = __ldg(g + t);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (k + i >= (int)S.T) break;
        B.x = fmaf(gk[i].x, x[i].x, B.x);
        B.x = fmaf(-gk[i].y, x[i].y, B.x);
        B.y = fmaf(gk[i].x, x[i].y, B.y);
        B.y = fmaf(gk[i].y, x[i].x, B.y);
      }
    }
  }
  *dst = rotate_apply(er, *dst, B);
}

// Most rows of a slot (T taps, rows Dp samples apart) whose windows straddle
// one rollover point.
__host__ __device__ __forceinline__ int64_t tc_fix_rows(int64_t T, int64_t Dp) { return (T - 1 + Dp - 1) / Dp; }

// Whether the filter-bank epilogue rotates slot S's rows itself (its fast
// path); when not, every row of the slot was stored unrotated.
__device__ __forceinline__ bool tc_slot_fast(const TcLaunch& L, const NcoConst& nc, int64_t Dp, int T) {
  return !L.exact_all && nc.rollover < 0x80000000u && (int64_t)31 * Dp + T < (int64_t)nc.rollover;
}

// Exact rotation of the rows that the filter-bank kernel stored unrotated:
// windows that straddle the NCO rollover (the phase restarts inside the
// window, so the product splits into the taps before and after it), or every
// row of a slot whose rollover is too short (or too long) for the epilogue's
// 32-bit counters.  Blocks (slot, y): the gridDim.y blocks of a slot take its
// rows in turn.  Runs after the filter-bank launch on the same stream.  Bound
// by latency: a thread a rollover point, its rows one after another and a load
// at a time, after a search for its merge set, took 27 us for 64 channels of
// 4 M samples.
__global__ void __launch_bounds__(128) tc_fix_kernel(const __grid_constant__ TcLaunch L) {
  const int s = blockIdx.x;
  if (s >= L.nslots) return;
  const TcSlot& S = L.slots[s];
  if (S.J <= 0 || S.T == 0) return;
  const NcoConst nc = L.nco[S.ch];
  if (!nc.enabled || nc.omega64 == 0 || nc.rollover == 0) return;
  const int64_t Dp = S.D;
  float2* out = reinterpret_cast<float2*>(S.out);
  const int64_t J = S.J, T = S.T, R = nc.rollover;
  const int64_t t0 = (int64_t)blockIdx.y * blockDim.x + threadIdx.x, tstep = (int64_t)gridDim.y * blockDim.x;
  if (!tc_slot_fast(L, nc, Dp, (int)T)) {
    for (int64_t j = t0; j < J; j += tstep) tc_fix_exact(L, s, j, Dp, out + (uint64_t)S.U * (uint64_t)j);
    return;
  }
  // rollover points n (block relative): (nco_base + n) mod R == 0; row j's
  // window [w0 + j D', w0 + j D' + T - 1] straddles n when it holds n - 1 and n
  const int64_t w0 = S.w0;
  const int64_t base = L.nco_base[S.ch];
  const int64_t first = w0 + 1;                            // smallest n a window can straddle
  const int64_t last = w0 + (J - 1) * Dp + T - 1;          // largest
  int64_t r0 = (base + first) % R;
  if (r0 < 0) r0 += R;
  const int64_t n0 = first + (r0 == 0 ? 0 : R - r0);
  // a thread a row: at most tc_fix_rows rows straddle a point, those with
  // n - T + 1 <= w0 + j D' <= n - 1
  const int64_t per = tc_fix_rows(T, Dp), points = last < n0 ? 0 : (last - n0) / R + 1;
  for (int64_t i = t0; i < points * per; i += tstep) {
    const int64_t n = n0 + i / per * R, lo = n - T + 1 - w0;
    const int64_t j = (lo <= 0 ? 0 : (lo + Dp - 1) / Dp) + i % per;
    if (j < J && w0 + j * Dp <= n - 1) tc_fix_exact(L, s, j, Dp, out + (uint64_t)S.U * (uint64_t)j);
  }
}

// 16-byte shared-memory load (one instruction for four fields of a slot record).
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};\n" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
// 32-byte global store (32-byte aligned).
__device__ __forceinline__ void stg256(void* p, const float2 (&o)[4]) {
  asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(o[0].x), "f"(o[0].y),
               "f"(o[1].x), "f"(o[1].y), "f"(o[2].x), "f"(o[2].y), "f"(o[3].x), "f"(o[3].y)
               : "memory");
}
// ---------------------------------------------------------------------------
// the filter-bank kernel
// ---------------------------------------------------------------------------
template <int FMT>
__global__ void __launch_bounds__(kTcThreads, 1) tc_filter_kernel(const __grid_constant__ TcFilterParams P) {
  const TcLaunch& L = *P.rec;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kTcMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kTcMaxStages];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ __align__(8) uint64_t drain_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int2 ring[kTcRing];       // item k: (merge set, item index); merge set -1 ends the sequence
  __shared__ int2 q_items[kTcQueue];   // scheduler -> producer: item i at i % kTcQueue
  __shared__ int q_prod, q_cons;       // items written / taken
  __shared__ TcMset s_ms[kTcMaxMsets];       // merge sets and groups of the launch (read per item)
  __shared__ TcGroup s_groups[kTcMaxGroups];
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t sbase = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  // launch constants in registers (L lives in device memory, and the inline
  // PTX's memory clobbers would otherwise reload them every chunk)
  const int stages = L.stages;
  const uint32_t poll = L.poll;
  const uint32_t stage_bytes = (uint32_t)L.stage_bytes;
  const bool hold = L.hold != 0;
  const uint8_t* const bbuf = L.bbuf;

  if (warp == 0) {
    tc::tmem_alloc(&tmem_base_s, kTmemCols);
    tc::tmem_relinquish();
  }
  if (tid == 0) q_prod = q_cons = 0;
  if (tid == 32) {
    for (int i = 0; i < stages; ++i) {
      tc::mbar_init(&full_bar[i], 1);
      tc::mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&acc_full[i], 1);
      tc::mbar_init(&acc_empty[i], kTcEpiWarps);
    }
    tc::mbar_init(&drain_bar, 1);
    tc::mbar_fence_init();
  }
  for (int i = tid; i < L.nmsets; i += kTcThreads) s_ms[i] = L.ms[i];
  for (int i = tid; i < L.ngroups; i += kTcThreads) s_groups[i] = L.groups[i];
  // epilogue constants of every slot of the launch (after the stages)
  TcEpiSlot* etab =
      reinterpret_cast<TcEpiSlot*>(smem_raw + (sbase - tc::smem_u32(smem_raw)) + (size_t)L.table_off);
  for (int s = tid; s < L.nslots; s += kTcThreads) {
    const TcSlot& S = L.slots[s];
    const int64_t D = S.D;
    TcEpiSlot e;
    e.out = S.out;
    e.J = S.J;
    e.stride = 8u * S.U;
    // runs leave in 16-byte pieces from their first output, pairs and quads
    // are single stores (rows 32 apart keep the alignment)
    const uint64_t lo = e.out | e.stride;
    uint32_t flags = S.flags;
    if (((e.out - 8u * (uint32_t)tc_run_pos((int)flags)) & 15u) != 0u) flags &= ~(uint32_t)kTcRun;
    if ((flags & kTcRun) || (lo & 15u) != 0u) flags &= ~(uint32_t)kTcPair;
    if ((lo & 31u) != 0u) flags &= ~(uint32_t)kTcQuad;
    e.flags = (uint16_t)flags;
    e.Tm1 = (uint16_t)(S.T > 0 ? S.T - 1u : 0u);
    e.om = 0;
    e.fm = 0;
    e.x0 = 0;
    e.R = 0xFFFFFFFFu;
    if (S.J > 0) {
      const NcoConst nc = L.nco[S.ch];
      if (nc.enabled) {
        // fast path: row counters (P0 + lane D) stay below 2 R < 2^32 with one
        // conditional subtraction; otherwise every output goes exact (R = 0)
        const bool fast = tc_slot_fast(L, nc, D, S.T);
        e.om = nc.omega64;
        e.fm = nc.fastmod;
        e.x0 = (int64_t)L.nco_base[S.ch] + S.w0;
        e.R = fast ? nc.rollover : 0u;
      }
    }
    etab[s] = e;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base_s;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    // Lane 0 alone waits and issues the copies (keeping the other lanes in
    // warp-synchronous calls around every wait slowed the MMA stream to less
    // than half its rate); its items come from the scheduler warp's queue.
    if (lane == 0) {
      int64_t ci = 0;  // chunks issued
      TcRing rg;       // their stage and round
      int64_t k = 0;   // items announced
      bool failed = false;
      while (!hold && !failed) {
        // item k from the scheduler (bounded wait)
        uint32_t polls = 0;
        while (*reinterpret_cast<volatile int*>(&q_prod) <= k) {
          if (++polls > poll) {
            failed = true;
            break;
          }
          __nanosleep(32);
        }
        if (failed) break;
        __threadfence_block();  // the item was written before the count
        const volatile int* qi = reinterpret_cast<volatile int*>(&q_items[k % kTcQueue]);
        const int2 item = make_int2(qi[0], qi[1]);
        __threadfence_block();
        *reinterpret_cast<volatile int*>(&q_cons) = (int)(k + 1);
        const bool more = item.x >= 0;
        // announce item k (or the end of the sequence) with its first stage
        if (rg.r > 0 && !tc::mbar_wait_bounded_fast(&empty_bar[rg.s], (uint32_t)((rg.r - 1) & 1), poll)) {
          failed = true;
          break;
        }
        ring[k % kTcRing] = item;
        ++k;
        if (!more) {
          tc::mbar_arrive(&full_bar[rg.s]);  // no copies: the consumers read the end marker
          ++ci;
          rg.next(stages);
          break;
        }
        const int m = item.x, t = item.y;
        const TcMset& M = s_ms[m];
        const int D = s_groups[M.group].D;
        const CUtensorMap* map = &P.maps[M.group];
        const int R = M.R;
        const uint32_t bbytes = (uint32_t)(4 * M.NS * 128);
        const uint32_t tx = (uint32_t)R * kTcTileBytes + bbytes;
        const int32_t x0 = 4 * (M.a % D);
        const int32_t y0 = t * R * kTcRows + M.a / D;
        const uint8_t* bsrc = bbuf + M.b;
        const int nchunks = M.nchunks;
        for (int c = 0; c < nchunks; ++c, ++ci, rg.next(stages)) {
          const int s = rg.s;
          // (the first chunk's stage was claimed with the announcement)
          if (c > 0 && rg.r > 0 && !tc::mbar_wait_bounded_fast(&empty_bar[s], (uint32_t)((rg.r - 1) & 1), poll)) {
            failed = true;
            break;
          }
          const uint32_t st = sbase + (uint32_t)s * stage_bytes;
          const uint32_t fb = tc::smem_u32(&full_bar[s]);
          mbar_expect_tx(&full_bar[s], tx);
          for (int r = 0; r < R; ++r)
            tma_load_2d(st + (uint32_t)r * kTcTileBytes, map, x0 + 64 * c, y0 + r * kTcRows, fb);
          bulk_load(st + (uint32_t)R * kTcTileBytes, bsrc + (size_t)c * bbytes, bbytes, fb);
        }
      }
      // every copy issued lands before the CTA can exit
      for (int64_t i = (ci > stages ? ci - stages : 0); i < ci; ++i)
        if (!tc::mbar_wait_bounded_fast(&full_bar[i % stages], (uint32_t)((i / stages) & 1), poll)) failed = true;
      if (failed) atomicExch(L.err, 1);
    }
  } else if (warp == kTcSchedWarp) {
    // ------------------------------------------------------------ scheduler
    // The CTA's part of the item list, up to 32 items a round, into the
    // producer's queue; an item with merge set -1 ends it.  The list is cut by
    // cost, not by input range: with few, uneven items (64 channels of 4 M
    // samples: 17 an SM of 4 to 65 chunks) equal ranges left the slowest SM
    // 2.5 times the average work.
    const int nitems = L.iprefix[L.nmsets];
    // first item whose cost before it is at least lim
    auto lower = [&](uint32_t lim) {
      int lo = 0, hi = nitems;  // 32 probes a round
      while (hi > lo) {
        const int step = (hi - lo + 32) / 33, p = lo + step * (lane + 1) - 1;
        const bool less = p < hi && __ldg(&L.items[p].y) < lim;
        const int n = __popc(__ballot_sync(0xffffffffu, less));  // (costs only grow along the list)
        const int nlo = lo + step * n;
        if (n < 32) hi = min(hi, nlo + step - 1);  // (probe n is not less)
        lo = min(nlo, hi);
      }
      return lo;
    };
    const uint32_t end = tc_cost_bound(L.ctotal, (int)blockIdx.x + 1, L.G);  // the items before this cost are ours
    const int first = lower(tc_cost_bound(L.ctotal, (int)blockIdx.x, L.G));
    bool failed = false, more = !hold;
    for (int done = 0; more;) {
      const int at = first + done + lane;
      const uint2 v = at < nitems ? __ldg(&L.items[at]) : make_uint2(0u, 0xFFFFFFFFu);
      int room = 0;
      if (lane == 0) {
        uint32_t polls = 0;
        while ((room = kTcQueue - (done - *reinterpret_cast<volatile int*>(&q_cons))) <= 0) {
          if (++polls > poll) {
            failed = true;
            break;
          }
          __nanosleep(64);
        }
      }
      failed = __shfl_sync(0xffffffffu, failed ? 1 : 0, 0) != 0;
      if (failed) break;
      const bool item = v.y < end;
      const int count = __popc(__ballot_sync(0xffffffffu, item));  // (a run from lane 0 on: costs grow)
      const int n = min(min(__shfl_sync(0xffffffffu, room, 0), 32), count + 1);
      if (lane < n) {
        volatile int* qi = reinterpret_cast<volatile int*>(&q_items[(done + lane) % kTcQueue]);
        qi[0] = item ? (int)(v.x >> 26) : -1;
        qi[1] = (int)(v.x & 0x3FFFFFFu);
      }
      more = n <= count;  // the end marker is not yet among them
      __threadfence_block();  // the items are written before the count
      __syncwarp();
      done += n;
      if (lane == 0) *reinterpret_cast<volatile int*>(&q_prod) = done;
    }
    if (failed && lane == 0) atomicExch(L.err, 1);
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // (lane 0 alone, for the same reason)
    if (lane == 0) {
      int64_t ci = 0;
      TcRing rg;
      int k = 0;
      bool failed = false, issued = false;
      auto wait1 = [&](uint64_t* bar, uint32_t parity) {
        const bool ok = tc::mbar_wait_bounded_fast(bar, parity, poll);
        tc::fence_after_sync();
        return ok;
      };
      while (true) {
        // the first stage of item k also announces it (ring entry k)
        if (!wait1(&full_bar[rg.s], (uint32_t)(rg.r & 1))) {
          failed = true;
          break;
        }
        const int2 it = ring[k % kTcRing];
        const int a = k & 1;
        if (k >= 2 && !wait1(&acc_empty[a], (uint32_t)(((k >> 1) - 1) & 1))) {
          failed = true;
          break;
        }
        if (it.x < 0) {  // end of the sequence: pass it on through the accumulator slot
          tc::mbar_arrive(&acc_full[a]);
          break;
        }
        const TcMset& M = s_ms[it.x];
        const int R = M.R, N = 4 * M.NS, nchunks = M.nchunks;
        const uint32_t idesc = tc::idesc_f16(FMT, 128, (uint32_t)N);
        const uint32_t dcol = tbase + (uint32_t)a * 256u;
        const uint32_t rstep = R == 2 ? 128u : 256u;  // accumulator columns of a tile
        for (int c = 0; c < nchunks; ++c, ++ci, rg.next(stages)) {
          const int s = rg.s;
          if (c > 0 && !wait1(&full_bar[s], (uint32_t)(rg.r & 1))) {
            failed = true;
            break;
          }
          const uint32_t st = sbase + (uint32_t)s * stage_bytes;
          const uint64_t bdesc = desc_sw128(st + (uint32_t)R * kTcTileBytes);
          for (int r = 0; r < R; ++r) {
            const uint64_t adesc = desc_sw128(st + (uint32_t)r * kTcTileBytes);
            const uint32_t d = dcol + (uint32_t)r * rstep;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_f16_ss(d, adesc + (uint64_t)(2 * kk), bdesc + (uint64_t)(2 * kk), idesc, (c | kk) != 0 ? 1u : 0u);
          }
          tc::mma_commit(&empty_bar[s]);
          issued = true;
        }
        if (failed) break;
        tc::mma_commit(&acc_full[a]);
        ++k;
      }
      // every MMA this CTA issued completes before its TMEM is released
      if (issued) {
        tc::mma_commit(&drain_bar);
        if (!tc::mbar_wait_bounded(&drain_bar, 0u, poll)) failed = true;
      }
      if (failed) atomicExch(L.err, 1);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // It used to bound the kernel: 16 warps took ~9000 cycles an item (87
    // instructions per 32 outputs at one in 6 cycles a warp), while the
    // accumulator waited for them.  So one lane per slot prepares what a block
    // of 32 rows needs, and a block whose rows all exist and whose counters do
    // not roll over (all but a few in a hundred) runs without a test per
    // output; its stores are chosen by warp-uniform masks.  Rows of 3, 5, 6 or
    // 7 outputs go through shared memory and leave in whole lines, rows of a
    // multiple of 4 as 32-byte stores: the sectors written fell from 2.5 times
    // the outputs to 1.1 times.  The 256-channel step of 2^26 samples went from
    // 5.14 to 4.83 ms, 64 taps over 2^24 samples from 156 to 140 us; the MMA
    // side now sets the pace (~7000 cycles an item: 12 KB of operands read and
    // 12 KB filled per MMA are 192 cycles of shared memory for 128 of tensor
    // work).  Nothing here may spill: with the stages in shared memory the L1
    // is too small, and 20 spilled registers doubled the kernel's time.
    const int q = warp & 3;           // TMEM lane quarter this warp may read
    const int h = (warp - 2) >> 2;    // which of the item's column chunks
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const uint32_t etab_s = tc::smem_u32(etab);
    const uint32_t scr = sbase + (uint32_t)L.scratch_off + (uint32_t)(warp - 2) * (uint32_t)L.scratch_warp;  // 32 rows x 8 outputs (where the launch has runs)
    const uint32_t rec = scr + (uint32_t)L.scratch_warp - 16u * kTcRec;  // a record per slot
    bool failed = false;
    for (int k = 0;; ++k) {
      const int a = k & 1;
      bool ok = true;
      if (lane == 0) ok = tc::mbar_wait_bounded(&acc_full[a], (uint32_t)((k >> 1) & 1), poll);
      if (!__shfl_sync(0xffffffffu, ok ? 1 : 0, 0)) {
        failed = true;
        break;
      }
      tc::fence_after_sync();
      const int2 it = ring[k % kTcRing];
      if (it.x < 0) break;
      const int m = it.x, t = it.y;
      const TcMset& M = s_ms[m];
      const int R = M.R, NS = M.NS, nch = NS >> 3;
      const int D = s_groups[M.group].D;
      // the warp's column chunks (8 slots of a tile each, at most kTcEpiOwn:
      // R NS <= 64) are read out of tensor memory together and the accumulator
      // slot released, so the MMAs of a later item run while this warp rotates
      // and stores
      const int per = (R * nch + kTcEpiPerQ - 1) / kTcEpiPerQ;  // 1 or 2
      const int idx0 = h * per, n_own = min(per, R * nch - idx0);
      float yv[kTcEpiOwn][16];  // (hi + lo) sums of those chunks
#pragma unroll
      for (int u = 0; u < kTcEpiOwn; ++u) {
        if (u < n_own) {
          const int idx = idx0 + u, r = idx >= nch ? 1 : 0, cc = idx - r * nch;
          const uint32_t col = tbase + lane_off + (uint32_t)a * 256u + (uint32_t)(r * 128 + 16 * cc);
          uint32_t vh[16], vl[16];
          tc::tmem_ld16(col, vh);
          tc::tmem_ld16(col + (uint32_t)(2 * NS), vl);
          tc::tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) yv[u][i] = __uint_as_float(vh[i]) + __uint_as_float(vl[i]);
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[a]);
      // the records: lane e makes the one of slot e & 7 of chunk e >> 3
      uint32_t rows = 0, flags = 0;
      bool plain = true;   // every row or none, no rollover in any window of the block
      bool first = false;  // the first slot of a run
      if ((lane >> 3) < n_own) {
        const int idx = idx0 + (lane >> 3), r = idx >= nch ? 1 : 0, cc = idx - r * nch;
        const int row0 = (t * R + r) * kTcRows + q * 32;  // row of lane 0
        const uint32_t e = etab_s + (uint32_t)(M.slot0 + cc * 8 + (lane & 7)) * kTcEpiSlotBytes;
        const uint4 ea = lds128(e), eb = lds128(e + 16u), ec = lds128(e + 32u);
        const uint64_t out = (uint64_t)ea.x | ((uint64_t)ea.y << 32);
        const uint32_t Rr = ec.x, Tm1 = ec.w >> 16;
        rows = (uint32_t)min(max((int)ec.y - row0, 0), 32);
        const uint64_t ptr = out + (uint64_t)ec.z * (uint64_t)(uint32_t)row0;
        // NCO counter of the first row's window start, (x0 + row0 D) mod R:
        // 0 <= x0 + row0 D < 2^32 or > -R on the fast path
        uint32_t p0 = 0, lim = 0xFFFFFFFFu, Rc = 0xFFFFFFFFu;
        if ((ea.z | ea.w) != 0u) {
          const int64_t v = (int64_t)((uint64_t)eb.z | ((uint64_t)eb.w << 32)) + (int64_t)row0 * D;
          const uint64_t fm = (uint64_t)eb.x | ((uint64_t)eb.y << 32);
          Rc = Rr;
          lim = Rr > Tm1 ? Rr - Tm1 : 0u;  // (R = 0: every row of the slot is left to tc_fix_kernel)
          if (Rr != 0u)
            p0 = v < 0 ? (uint32_t)(v + (int64_t)Rr) : (uint32_t)__umul64hi(fm * (uint64_t)(uint32_t)v, (uint64_t)Rr);
        }
        plain = rows == 0u || (rows == 32u && (uint64_t)p0 + 31u * (uint32_t)D < (uint64_t)lim);
        flags = ec.w & 0xFFFFu;
        const uint32_t pos = (uint32_t)tc_run_pos((int)flags);
        const uint32_t ra = rec + (uint32_t)lane * kTcRec;
        sts128(ra, (uint32_t)ptr, (uint32_t)(ptr >> 32), ec.z, scr + (uint32_t)(lane & 7) * 256u - pos * 248u);
        sts128(ra + 16u, p0, ea.z, ea.w, 0u);
        sts128(ra + 32u, Rc, lim, rows, 0u);
        first = (flags & kTcRun) != 0u && pos == 0u;
      }
      const uint32_t m_plain = __ballot_sync(0xffffffffu, plain);
      const uint32_t m_live = __ballot_sync(0xffffffffu, rows > 0u);
      const uint32_t m_run = __ballot_sync(0xffffffffu, (flags & kTcRun) != 0u);
      const uint32_t m_first = __ballot_sync(0xffffffffu, first);
      const uint32_t m_pair = __ballot_sync(0xffffffffu, (flags & kTcPair) != 0u);
      const uint32_t m_quad = __ballot_sync(0xffffffffu, (flags & kTcQuad) != 0u);
      const uint32_t laneD = (uint32_t)lane * (uint32_t)D;
      // one chunk of 8 slots; kPlain: every lane has its row and no counter
      // rolls over (else both are tested per output)
      auto chunk = [&](int u, auto plain_tag) {
        constexpr bool kPlain = decltype(plain_tag)::value;
        const uint32_t rc = rec + (uint32_t)u * 8u * kTcRec;
        const uint32_t live = m_live >> (8 * u), run = m_run >> (8 * u), pair = m_pair >> (8 * u),
                       quad = m_quad >> (8 * u);
#pragma unroll
        for (int g = 0; g < 8; g += 4) {  // four slots at a time
          if (((live >> g) & 15u) == 0u) continue;  // padding slots: nothing to do
          float2 o[4];
          bool v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint4 rb = lds128(rc + (uint32_t)(g + e) * kTcRec + 16u);
            const float2 y0 = make_float2(yv[0][2 * (g + e)], yv[0][2 * (g + e) + 1]);
            uint32_t pc = rb.x + laneD;
            bool fast = true;
            v[e] = true;
            if constexpr (!kPlain) {
              const uint4 rr = lds128(rc + (uint32_t)(g + e) * kTcRec + 32u);
              pc = pc >= rr.x ? pc - rr.x : pc;
              fast = pc < rr.y;
              v[e] = (uint32_t)lane < rr.z;
            }
            const uint32_t turns = __umulhi(pc, rb.y) + pc * rb.z;  // bits 32..63 of pc * om: 2^-32 turns
            float sn, cs;
            __sincosf((float)(int32_t)turns * 1.4629180792671596e-09f, &sn, &cs);  // 2 pi / 2^32
            o[e] = cmul_nco(y0, make_float2(cs, sn));
            if constexpr (!kPlain) o[e] = fast ? o[e] : y0;  // windows across the rollover: unrotated, for tc_fix_kernel
          }
          auto dst = [&](int e) {
            const uint4 r0 = lds128(rc + (uint32_t)(g + e) * kTcRec);
            return reinterpret_cast<float2*>(((uint64_t)r0.x | ((uint64_t)r0.y << 32)) +
                                             (uint64_t)r0.z * (uint64_t)(uint32_t)lane);
          };
          if ((quad >> g) & 1u) {
            if (v[3]) {
              stg256(dst(0), o);
              continue;
            }
          }
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            if ((pair >> (g + e)) & 1u) {
              if (v[e + 1])
                __stcs(reinterpret_cast<float4*>(dst(e)), make_float4(o[e].x, o[e].y, o[e + 1].x, o[e + 1].y));
              else if (v[e])
                __stcs(dst(e), o[e]);
              continue;
            }
#pragma unroll
            for (int f = e; f < e + 2; ++f) {
              if ((run >> (g + f)) & 1u) {  // rows of the run follow one another in the scratch
                const uint4 r0 = lds128(rc + (uint32_t)(g + f) * kTcRec);
                if (v[f]) sts64(r0.w + r0.z * (uint32_t)lane, o[f]);
              } else if ((live >> (g + f)) & 1u) {
                if (v[f]) __stcs(dst(f), o[f]);
              }
            }
          }
        }
      };
      // one copy of the chunk code of either kind (kept small: the warps of
      // every role share the SM's instruction cache); the chunks move down
      // into yv[0] in turn
#pragma unroll 1
      for (int u = 0; u < n_own; ++u) {
        if (u > 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) yv[0][i] = yv[1][i];
        }
        __syncwarp();  // the records; the scratch rows of the last chunk are read
        if (((m_plain >> (8 * u)) & 255u) == 255u)
          chunk(u, std::true_type());
        else
          chunk(u, std::false_type());
        // complete runs leave in whole lines: 32 rows of len outputs follow one
        // another in the scratch as they do in the channel's output
        uint32_t firsts = (m_first >> (8 * u)) & 255u;
        if (firsts != 0u) {
          __syncwarp();
          do {
            const uint32_t e = (uint32_t)__ffs((int)firsts) - 1u, ra = rec + (8u * (uint32_t)u + e) * kTcRec;
            firsts &= firsts - 1u;
            const uint4 r0 = lds128(ra);
            const uint64_t ptr = (uint64_t)r0.x | ((uint64_t)r0.y << 32);
            const uint32_t len = r0.z >> 3, src = scr + e * 256u;
            if (lds128(ra + (len - 1u) * kTcRec + 32u).z == 32u) {
              for (uint32_t i = (uint32_t)lane; i < 16u * len; i += 32u)
                __stcs(reinterpret_cast<uint4*>(ptr) + i, lds128(src + 16u * i));
            } else {  // the last rows of the channel
              uint32_t count = 0;
              for (uint32_t f = 0; f < len; ++f) count += lds128(ra + f * kTcRec + 32u).z;
              for (uint32_t i = (uint32_t)lane; i < count; i += 32u) {
                float2 w;
                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(w.x), "=f"(w.y) : "r"(src + 8u * i));
                __stcs(reinterpret_cast<float2*>(ptr) + i, w);
              }
            }
          } while (firsts != 0u);
        }
      }
      __syncwarp();  // the records are read before the next item's are made
    }
    if (failed && lane == 0) atomicExch(L.err, 1);
  }

  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, kTmemCols);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

void PolyEngine::free_tc() {
  if (d_ctaps_) dfree(d_ctaps_);
  if (d_ctab_) dfree(d_ctab_);
  if (d_xhl_) dfree(d_xhl_);
  if (d_bbuf_) dfree(d_bbuf_);
  if (d_items_) dfree(d_items_);
  if (d_tcrec_) dfree(d_tcrec_);
  for (cudaEvent_t e : pack_ev_) cudaEventDestroy(e);
  pack_ev_.clear();
  for (cudaStream_t q : side_) cudaStreamDestroy(q);
  side_.clear();
  if (h_err_) cudaFreeHost(h_err_);
  d_ctaps_ = nullptr;
  d_ctab_ = nullptr;
  d_xhl_ = nullptr;
  d_bbuf_ = nullptr;
  d_items_ = nullptr;
  items_cap_ = 0;
  d_tcrec_ = nullptr;
  h_err_ = nullptr;
  d_err_ = nullptr;
  xhl_cap_ = 0;
  bbuf_cap_ = 0;
}

// FP32 NCO-modulated taps of every channel, [U][T] per channel, and the
// per-channel pointer table the kernels read; the error flag in mapped host
// memory.
int PolyEngine::build_tc(int fmt) {
  free_tc();
  tc_fmt_ = fmt;
  std::vector<size_t> off(chans_.size());
  size_t total = 0;
  for (size_t c = 0; c < chans_.size(); ++c) {
    off[c] = total;
    total += (size_t)chans_[c].up * chans_[c].T;
  }
  std::vector<float2> g(total);
  for (size_t c = 0; c < chans_.size(); ++c) {
    const EngineChannel& e = chans_[c];
    int64_t fm = 0;
    if (e.nco.enabled) {
      fm = (int64_t)e.shift_hz % (int64_t)fs_;
      if (fm < 0) fm += fs_;
    }
    for (uint32_t ph = 0; ph < e.up; ++ph) {
      for (uint32_t k = 0; k < e.T; ++k) {
        const float2 h = e.flipped[(size_t)ph * e.T + k];
        double gr = h.x, gi = h.y;
        if (e.nco.enabled) {
          // e^{j w k}, w k reduced exactly: 2 pi ((f mod fs) k mod fs) / fs
          const uint64_t red = (uint64_t)(((unsigned __int128)(uint64_t)fm * (uint64_t)k) % fs_);
          const double ang = 2.0 * M_PI * (double)red / (double)fs_;
          const double cs = std::cos(ang), sn = std::sin(ang);
          gr = (double)h.x * cs - (double)h.y * sn;
          gi = (double)h.x * sn + (double)h.y * cs;
        }
        g[off[c] + (size_t)ph * e.T + k] = make_float2((float)gr, (float)gi);
      }
    }
  }
  cudaError_t err = dalloc(reinterpret_cast<void**>(&d_ctaps_), total * sizeof(float2));
  if (err == cudaSuccess) err = cudaMemcpy(d_ctaps_, g.data(), total * sizeof(float2), cudaMemcpyHostToDevice);
  std::vector<const float2*> tab(chans_.size());
  for (size_t c = 0; c < chans_.size(); ++c) tab[c] = d_ctaps_ + off[c];
  if (err == cudaSuccess) err = dalloc(reinterpret_cast<void**>(&d_ctab_), tab.size() * sizeof(float2*));
  if (err == cudaSuccess) err = cudaMemcpy(d_ctab_, tab.data(), tab.size() * sizeof(float2*), cudaMemcpyHostToDevice);
  // one device record per launch pack (packs <= groups)
  if (err == cudaSuccess) err = dalloc(reinterpret_cast<void**>(&d_tcrec_), kTcMaxGroups * sizeof(TcLaunch));
  for (int i = 0; i < kTcSideStreams && err == cudaSuccess; ++i) {
    cudaStream_t q = nullptr;
    err = cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking);
    if (err == cudaSuccess) side_.push_back(q);
  }
  for (int i = 0; i <= kTcSideStreams && err == cudaSuccess; ++i) {
    cudaEvent_t e = nullptr;
    err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (err == cudaSuccess) pack_ev_.push_back(e);
  }
  if (err == cudaSuccess) err = cudaHostAlloc(&h_err_, sizeof(int), cudaHostAllocMapped);
  if (err == cudaSuccess) {
    *h_err_ = 0;
    err = cudaHostGetDevicePointer(reinterpret_cast<void**>(&d_err_), h_err_, 0);
  }
  if (err != cudaSuccess) return cuda_status(err);
  if (!tensor_map_encoder()) return FDSP_ERR_UNSUPPORTED;
  return FDSP_OK;
}

int PolyEngine::tc_error() {
  if (!h_err_) return 0;
  const int v = *reinterpret_cast<volatile int*>(h_err_);
  *reinterpret_cast<volatile int*>(h_err_) = 0;
  return v;
}

// Plans and enqueues the tensor-core form of the groups in `tc_groups`
// (engine group indices).  Groups are packed greedily into launches whose
// records fit the kernel parameter block; per pack one prep (the first also
// splits the input, which every pack then reads), one filter-bank launch and
// the exact rotation pass.  Each pack has its own device record and B-image
// region, so the packs run at the same time: pack 0 on the caller's stream,
// pack k > 0 on side stream (k - 1) mod kTcSideStreams once the split is
// done, and a pack's filter-bank CTAs take the SMs that the earlier packs'
// CTAs leave as they finish (one launch's tail instead of one per pack).
// With kernel timing on (each launch timed alone), or with a completion hook
// (apply_host: the first packs' device-to-host copies then start while the
// later packs compute, where concurrent packs would all end together), the
// packs run one after another on the caller's stream.  Groups no launch can
// hold are returned in `fallback` for the FP32 kernel.
int PolyEngine::launch_tc(const float2* d_in, uint64_t n, float2* const* out, const std::vector<int>& tc_groups,
                          std::vector<int>& fallback, cudaStream_t stream) {
  fallback.clear();
  std::vector<TcGroupIn> gin;
  std::vector<int> gmap;
  for (int gi : tc_groups) {
    const EngineGroup& g = groups_[gi];
    TcGroupIn in;
    in.D = (int)g.D;
    in.max_split = std::max(1, g.tc_split);
    for (size_t ki = 0; ki < classes_.size(); ++ki) {
      const EngineClass& k = classes_[ki];
      if (k.down != g.D) continue;
      const uint32_t U = k.up;
      for (uint32_t r = 0; r < U; ++r) {
        if (k.M <= r) continue;
        const uint64_t tt = (uint64_t)k.phase + (uint64_t)r * g.D;
        for (int c : k.chans) {
          TcSlotIn s;
          s.ch = c;
          s.T = (int)chans_[c].T;
          s.U = (int)U;
          s.r = (int)r;
          s.phi = (int)(tt % U);
          s.delta = (int64_t)(k.xoffset + tt / U);
          s.J = (int64_t)((k.M - r + U - 1) / U);
          in.slots.push_back(s);
        }
      }
    }
    if (!in.slots.empty()) {
      gin.push_back(in);
      gmap.push_back(gi);
    }
  }
  if (gin.empty()) return FDSP_OK;
  if (num_sms_ == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev);
    if (num_sms_ <= 0) num_sms_ = 1;
  }
  // Plan each group once, then fill launches with them in turn.  The row split
  // is chosen when the block size, the slots or the split limit change (the
  // choice plans every split: most of the planning time); between blocks of a
  // stream only the windows' offsets move.
  std::vector<std::vector<int>> packs;  // indices into gin
  std::vector<TcPlan> plans;
  for (int i = 0; i < (int)gin.size(); ++i) {
    EngineGroup& eg = groups_[gmap[i]];
    const bool known = eg.tc_plan_n == n && eg.tc_plan_slots == gin[i].slots.size() && eg.tc_plan_max == gin[i].max_split;
    TcGroupPlan gp;
    bool ok = known && tc_plan_group(gin[i], H_, eg.tc_plan_split, gp) == 0;
    if (!ok) ok = tc_plan_group(gin[i], H_, 0, gp) == 0;
    if (ok && !gp.ms.empty()) {
      eg.tc_plan_n = n;
      eg.tc_plan_slots = gin[i].slots.size();
      eg.tc_plan_max = gin[i].max_split;
      eg.tc_plan_split = gp.g.S;
      if (plans.empty() || !tc_append(plans.back(), gp)) {
        plans.emplace_back();
        packs.emplace_back();
        ok = tc_append(plans.back(), gp);
      }
      if (ok) packs.back().push_back(i);
    }
    if (!ok) fallback.push_back(gmap[i]);
  }
  for (TcPlan& p : plans)
    if (tc_finish(p, (int64_t)n, H_, num_sms_) != 0) return FDSP_ERR_UNSUPPORTED;
  if (plans.empty()) return FDSP_OK;
  if (plans.size() > (size_t)kTcMaxGroups) return FDSP_ERR_UNSUPPORTED;
  // scratch (grow only): the split input, which every pack reads, the B images
  // and the item list of every pack
  const TcScratch sc = tc_scratch(plans);
  auto grow = [&](auto** p, size_t* cap, size_t need, size_t slack) {
    return grow_scratch(
        p, cap, need, slack,
        // a pool gives a released range to other engines, on other streams,
        // while earlier applies queued on this stream may still read it
        // (without a pool cudaFree waits for them)
        [&]() { return pool_ ? cuda_status(cudaStreamSynchronize(stream)) : (int)FDSP_OK; },
        [&](void* q) { dfree(q); },
        [&](auto** q, size_t n) {
          const int st = cuda_status(dalloc(reinterpret_cast<void**>(q), n * sizeof(**q)));
          if (st != FDSP_OK) cudaGetLastError();
          return st;
        });
  };
  FDSP_TRY(grow(&d_xhl_, &xhl_cap_, sc.xhl, sc.xhl_slack));
  FDSP_TRY(grow(&d_bbuf_, &bbuf_cap_, sc.b, sc.b_slack));
  FDSP_TRY(grow(&d_items_, &items_cap_, sc.items, sc.items_slack));
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return FDSP_ERR_UNSUPPORTED;
  // (side streams and events made by build_tc, outside any stream capture)
  if (side_.empty() || pack_ev_.size() < side_.size() + 1) return FDSP_ERR_UNSUPPORTED;
  const bool concurrent = !kprof_ && !done_fn_ && plans.size() > 1;
  std::vector<char> side_used(side_.size(), 0);
  static thread_local TcLaunch L;
  for (size_t li = 0; li < plans.size(); ++li) {
    const TcPlan& plan = plans[li];
    cudaStream_t ps = stream;  // this pack's stream
    if (concurrent && li > 0) {
      const size_t si = (li - 1) % side_.size();
      ps = side_[si];
      if (!side_used[si]) {  // after the split (recorded below by pack 0)
        FDSP_TRY(cuda_status(kwait(ps, pack_ev_[0])));
        side_used[si] = 1;
      }
    }
    std::memset(&L, 0, sizeof(L));
    L.block = in16_ ? nullptr : d_in;
    L.block16 = in16_;
    L.hist = d_hist_[hist_cur_];
    L.nco = d_nco_;
    L.ctaps = d_ctab_;
    L.xhl = d_xhl_;
    L.bbuf = d_bbuf_ + sc.b_off[li];
    L.err = d_err_;
    L.rec_out = d_tcrec_ + li;
    L.N = (int64_t)n;
    L.xhl_n = (int64_t)sc.xhl;
    L.H = H_;
    L.G = plan.G;
    L.nmsets = (int32_t)plan.ms.size();
    L.ngroups = (int32_t)plan.groups.size();
    L.stages = plan.stages;
    L.stage_bytes = plan.stage_bytes;
    L.table_off = plan.table_off;
    L.scratch_off = plan.scratch_off;
    L.scratch_warp = plan.scratch_warp;
    L.nslots = (int32_t)plan.slots.size();
    L.poll = tc_poll_;
    L.hold = tc_hold_;
    L.exact_all = tc_exact_all_;
    for (size_t c = 0; c < chans_.size(); ++c) {
      const uint32_t R = chans_[c].nco.rollover;
      L.nco_base[c] = R ? (uint32_t)(abs0_ % R) : 0u;
    }
    int pieces = 0;
    for (size_t m = 0; m < plan.ms.size(); ++m) {
      L.ms[m] = plan.ms[m];
      L.bprefix[m] = pieces;
      pieces += plan.ms[m].nchunks * 4 * plan.ms[m].NS * 8;
    }
    L.bprefix[plan.ms.size()] = pieces;
    L.items = d_items_ + sc.item_off[li];
    int items = 0;
    for (size_t m = 0; m < plan.ms.size(); ++m) {
      L.iprefix[m] = items;
      items += plan.ms[m].items;
    }
    L.iprefix[plan.ms.size()] = items;
    L.ctotal = plan.ctotal;
    L.cost_shift = plan.cost_shift;
    for (size_t s = 0; s < plan.slots.size(); ++s) {
      L.slots[s] = plan.slots[s];
      if (plan.slots[s].J > 0)
        L.slots[s].out = (uint64_t)(uintptr_t)(out[plan.slots[s].ch] + plan.slot_r[s]);
    }
    for (size_t g = 0; g < plan.groups.size(); ++g) {
      const TcPlanGroup& pg = plan.groups[g];
      L.groups[g].D = pg.D;
      L.groups[g].S = pg.S;
      groups_[gmap[packs[li][g]]].tc_split_used = pg.S;
      // rows of D' samples; a row spans Wx samples (4 16-bit elements each);
      // (rows - 1) D' + Wx <= xhl_samples keeps every address inside xhl
      const cuuint64_t rows = (cuuint64_t)((plan.xhl_samples - pg.Wx) / pg.D + 1);
      const cuuint64_t dims[2] = {(cuuint64_t)(4 * pg.Wx), rows};
      const cuuint64_t strides[1] = {(cuuint64_t)pg.D * 8u};
      const cuuint32_t box[2] = {64u, (cuuint32_t)kTcRows};
      const cuuint32_t estr[2] = {1u, 1u};
      const CUresult r = enc(&L.maps[g], CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, d_xhl_, dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS) return FDSP_ERR_UNSUPPORTED;
    }
    // prep: B images (few blocks), then, for the first launch, the split
    const int nb_build = std::max(1, std::min(num_sms_, (std::max(pieces, items) + 255) / 256));
    const int64_t nb_split = li == 0 ? std::min<int64_t>(((int64_t)sc.xhl + 255) / 256, (int64_t)num_sms_ * 8) : 0;
    auto prep = tc_fmt_ == 0 ? tc_prep_kernel<0> : tc_prep_kernel<1>;
    int nbb = nb_build;
    cudaError_t e = klaunch(reinterpret_cast<const void*>(prep), dim3((unsigned)(nb_build + nb_split)), dim3(256), 0,
                            ps, L, nbb);
    if (e != cudaSuccess) return cuda_status(e);
    launches_last_++;
    if (concurrent && li == 0) FDSP_TRY(cuda_status(krecord(pack_ev_[0], stream)));
    auto kern = tc_fmt_ == 0 ? tc_filter_kernel<0> : tc_filter_kernel<1>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, plan.smem);
    if (e != cudaSuccess) return cuda_status(e);
    if (kprof_) cudaEventRecord(kprof_event(), ps);
    static thread_local TcFilterParams FP;
    std::memcpy(FP.maps, L.maps, sizeof(FP.maps));
    FP.rec = d_tcrec_ + li;
    e = klaunch(reinterpret_cast<const void*>(kern), dim3((unsigned)plan.G), dim3(kTcThreads), (size_t)plan.smem, ps,
                FP);
    if (kprof_) cudaEventRecord(kprof_event(), ps);
    if (e != cudaSuccess) return cuda_status(e);
    launches_last_++;
    // exact pass: blocks per slot for the most rows a slot of this launch may
    // have to fix, one per thread (the pass is latency bound: each row is a
    // serial sum of up to T taps, and the last pack's pass ends the step)
    int64_t work = 1;
    for (size_t si = 0; si < plan.slots.size(); ++si) {
      const TcSlot& S = plan.slots[si];
      if (S.J <= 0) continue;
      const NcoConst& nc = chans_[S.ch].nco;
      if (!nc.enabled || nc.omega64 == 0 || nc.rollover == 0) continue;
      const int64_t Dp = S.D;
      const bool fast = !tc_exact_all_ && nc.rollover < 0x80000000u && 31 * Dp + S.T < (int64_t)nc.rollover;
      work = std::max<int64_t>(
          work, fast ? (((int64_t)S.J * Dp + S.T) / nc.rollover + 1) * tc_fix_rows(S.T, Dp) : (int64_t)S.J);
    }
    const unsigned fix_y = (unsigned)std::min<int64_t>(4096, (work + 127) / 128);
    e = klaunch(reinterpret_cast<const void*>(tc_fix_kernel), dim3((unsigned)plan.slots.size(), fix_y), dim3(128), 0,
                ps, L);
    if (e != cudaSuccess) return cuda_status(e);
    launches_last_++;
    tc_groups_last_ += (int)packs[li].size();
    if (done_fn_) {
      std::vector<int> egs;
      for (int gi : packs[li]) egs.push_back(gmap[gi]);
      notify_done(egs, ps);
    }
  }
  // the side streams join the caller's stream (before the history update)
  for (size_t si = 0; si < side_.size(); ++si) {
    if (!side_used[si]) continue;
    FDSP_TRY(cuda_status(krecord(pack_ev_[1 + si], side_[si])));
    FDSP_TRY(cuda_status(kwait(stream, pack_ev_[1 + si])));
  }
  return FDSP_OK;
}

}  // namespace fdsp
