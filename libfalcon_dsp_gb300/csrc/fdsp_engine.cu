// Polyphase engine: fused per-channel NCO shift + polyphase up/down resampling
// for any number of channels sharing one input stream (plain FP32 form).
//
// Reference behaviour reproduced (paths relative to the reference project):
//   shift      src/transform/falcon_dsp_freq_shift.cc:164-192, :194-235
//   resample   src/transform/falcon_dsp_polyphase_resampler.cc:114-162, :256-346
//   channelize src/transform/falcon_dsp_multi_rate_channelizer.cc:146-164
//
// Design (GB300-first, not a translation of the Jetson kernels):
//  * Channels are grouped by decimation factor D.  For one group, one CTA owns
//    a tile of Qt output rows and stages the RAW input span the tile needs in
//    shared memory exactly once, de-interleaved by D (sample s at
//    [s mod D][s div D]) so that 32 lanes computing 32 consecutive rows read
//    32 consecutive words: no bank conflicts, whatever D is.
//  * The NCO is folded into the taps.  For a window starting at input s with
//    no counter rollover inside it,
//        sum_k h[k] x[s+k] e^{j w ((s+k) mod R)} = e^{j w (s mod R)} sum_k g[k] x[s+k]
//    with g[k] = h[k] e^{j w k}.  All channels of a group therefore read the
//    same unshifted samples, and each output pays one rotation by an exact
//    integer phase (64-bit fixed point turns).  A window that straddles a
//    rollover (the reference's phase jump) is corrected exactly by splitting
//    its sum at the rollover.
//  * Channels with the same (up, down) share streaming state, so their outputs
//    sit at the same input positions.  They are packed NB at a time into tap
//    batches: one shared-memory load of x feeds NB complex MACs, which keeps
//    the kernel FMA-bound instead of shared-memory bound.
//  * All per-launch parameters ride in the kernel parameter block; the launch
//    needs no host->device copy and is safe to capture in a CUDA graph.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <type_traits>

#include "fdsp_internal.h"
#include "fdsp_nco.cuh"

namespace fdsp {

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
using ChanMeta = OutMeta;

// Counter value (n mod R) of the sample at block-relative index w: one
// multiply-high below 2^32 (Lemire, Kaser & Kurz, "Faster remainder by direct
// computation", 2019).
__device__ __forceinline__ uint32_t nco_counter(const ChanMeta& cm, int64_t w) {
  const int64_t pv = (int64_t)cm.base + w;
  if (pv < 0) return (uint32_t)(pv + (int64_t)cm.rollover);
  if ((pv >> 32) == 0) return (uint32_t)__umul64hi(cm.fastmod * (uint64_t)(uint32_t)pv, (uint64_t)cm.rollover);
  return (uint32_t)((uint64_t)pv % cm.rollover);
}

// e^{j 2 pi t} for t in 2^-32 turns, on the SFU: the reduced argument lies in
// [-pi, pi), where __sincosf is accurate to ~4e-7 absolute.
__device__ __forceinline__ float2 phasor32(uint32_t turns) {
  const float a = (float)(int32_t)turns * 1.4629180792671596e-09f;  // 2 pi / 2^32
  float s, c;
  __sincosf(a, &s, &c);
  return make_float2(c, s);
}


// Packed FP32 pairs: one instruction, two IEEE multiply-adds.  The FMA rate is
// that of the scalar form (74 TFLOP/s of either measured); half the issue
// slots stay free for the shared-memory reads.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// kRows rows (jl, jl + 32, ...) of one work set with NB live channels: T
// complex MACs per row and channel (taps and samples from shared memory), then
// rotation and store.  Packed taps are stored [T][NB] as (re, re, im, im), so a
// complex MAC is two packed multiply-adds of the sample as it lies in memory:
// a += (re, re) x, b += (im, im) x, and the output is (a.x - b.y, a.y + b.x).
// Compact taps (re, im) take half the room and the same multiply-adds one
// component at a time (packed ones too where four rows share the copies).
// Bound: issue slots and shared-memory reads.  A tap read (a broadcast) feeds
// kRows samples, a sample read NB channels.  Sums run over the taps in order
// whatever kRows is, so an output's bits do not depend on the tile height.
constexpr int kShortRun = 5;  // phases of a run that is walked tap by tap
template <int NB, int kRows, bool kPacked>
__device__ __forceinline__ void process_rows(const float2* __restrict__ xs, const float4* __restrict__ tp,
                                             const ChanMeta* __restrict__ meta, int T, int D, int P, int nph, int b0,
                                             int q0, int64_t j, int64_t J, int U, int r, int delta) {
  const f32x2* xp = reinterpret_cast<const f32x2*>(xs + b0 * P + q0);
  constexpr int kPitch = (NB + 1) & ~1;  // compact taps of a row
  const ulonglong2* tq = reinterpret_cast<const ulonglong2*>(tp);
  const float2* tc = reinterpret_cast<const float2*>(tp);
  f32x2 sa[kRows][NB], sb[kRows][NB];
#pragma unroll
  for (int q = 0; q < kRows; ++q)
#pragma unroll
    for (int n = 0; n < NB; ++n) sa[q][n] = sb[q][n] = 0ull;
  auto tap = [&]() {
    f32x2 x[kRows];
#pragma unroll
    for (int q = 0; q < kRows; ++q) x[q] = xp[32 * q];
    if constexpr (kPacked) {
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        const ulonglong2 g = tq[n];
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          sa[q][n] = fma2(g.x, x[q], sa[q][n]);
          sb[q][n] = fma2(g.y, x[q], sb[q][n]);
        }
      }
      tq += NB;
    } else {
      float2 g[kPitch];
#pragma unroll
      for (int n = 0; n < NB; n += 2) {
        if (n + 1 < NB) {
          const float4 v = *reinterpret_cast<const float4*>(tc + n);
          g[n] = make_float2(v.x, v.y);
          g[n + 1] = make_float2(v.z, v.w);
        } else {
          g[n] = tc[n];
        }
      }
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          if constexpr (kRows >= 4) {
            sa[q][n] = fma2(pack2(g[n].x, g[n].x), x[q], sa[q][n]);
            sb[q][n] = fma2(pack2(g[n].y, g[n].y), x[q], sb[q][n]);
          } else {
            const float2 v = unpack2(x[q]), a = unpack2(sa[q][n]), b = unpack2(sb[q][n]);
            sa[q][n] = pack2(fmaf(g[n].x, v.x, a.x), fmaf(g[n].x, v.y, a.y));
            sb[q][n] = pack2(fmaf(g[n].y, v.x, b.x), fmaf(g[n].y, v.y, b.y));
          }
        }
      tc += kPitch;
    }
  };
  // The taps of a window are runs of nph samples between the wraps of the
  // de-interleaved tile.  Compact taps of wide batches, and short runs, are
  // walked with a test per tap; the others run by run.  (Measured both ways over
  // D = 1 to 100, 5 to 16 % apart: 64 taps of 16 channels by 2 over 2^20
  // samples 190 us run by run, 160 tap by tap.)
  if ((!kPacked && NB > 2) || (nph > 1 && nph <= kShortRun)) {
    const int step = nph == 1 ? 1 : P, wrap = 1 - (nph - 1) * P;
    int b = b0;
#pragma unroll(NB > 4 ? 1 : 2)
    for (int k = 0; k < T; ++k) {
      tap();
      const bool last = ++b == nph;
      xp += last ? wrap : step;
      b = last ? 0 : b;
    }
  } else {
    const int run = nph == 1 ? T : nph, step = nph == 1 ? 1 : P, wrap = nph == 1 ? 0 : 1 - nph * P;
    for (int k = 0, end = min(T, run - b0); k < T; end = min(T, k + run), xp += wrap) {
#pragma unroll(NB > 4 ? 1 : 2)
      for (; k < end; ++k) {
        tap();
        xp += step;
      }
    }
  }

  float2 acc[kRows][NB];
#pragma unroll
  for (int q = 0; q < kRows; ++q)
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      const float2 va = unpack2(sa[q][n]), vb = unpack2(sb[q][n]);
      acc[q][n] = make_float2(va.x - vb.y, va.y + vb.x);
    }

  // Epilogue: rotate by the NCO phase of the window start, store; windows that
  // straddle the NCO rollover are stored unrotated and then take the exact
  // split-sum path, so no accumulator stays live through the fix-up.  The
  // counter of a channel's first row is one modulo, the next rows (32 D
  // samples on) step it by 32 D mod R.
  uint32_t slow = 0;  // bit q * NB + n
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const ChanMeta& cm = meta[n];
    const uint32_t R = cm.rollover, step = cm.step32;
    const uint32_t om_lo = (uint32_t)cm.omega64, om_hi = (uint32_t)(cm.omega64 >> 32);
    const bool en = cm.enabled != 0;
    float2* const out = cm.out;
    uint32_t p = en ? nco_counter(cm, (int64_t)delta + j * D - T + 1) : 0u;
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const float2 e0 = phasor32(__umulhi(p, om_lo) + p * om_hi);  // bits 32..63 of p * omega64
      const float2 e = en ? e0 : make_float2(1.f, 0.f);
      const bool ok = !en || (uint64_t)p + (uint64_t)T - 1 < (uint64_t)R;
      const float2 y = cmul_nco(acc[q][n], e);
      if (j + 32 * q < J) {
        out[(int64_t)r + (int64_t)U * (j + 32 * q)] = ok ? y : acc[q][n];
        slow |= ok ? 0u : (1u << (q * NB + n));
      }
      p += step;
      p -= (p >= R || p < step) ? R : 0u;
    }
  }
  // The exact path takes the warp's slow outputs row block by channel, so that
  // at any time its lanes are at one tap (a broadcast) of neighbouring rows;
  // each lane's sum starts at its own first tap past the rollover.  Lane by
  // lane, the lanes' taps lay D apart, 16 to 32 bank cycles a read, and a tile
  // at the rollover set the time of the launch (4000 taps of two channels by 4
  // over 2^20 samples: 2.6 ms so, 0.71 this way).
  for (uint32_t all = __reduce_or_sync(0xffffffffu, slow); all != 0u; all &= all - 1u) {
    const int bit = __ffs(all) - 1;
    const int q = bit / NB, n = bit - q * NB;
    const bool mine = ((slow >> bit) & 1u) != 0u;
    const OutMeta& cm = meta[n];
    const int64_t jq = j + 32 * q;
    const ExactRot er = rotate_prep(cm, (int64_t)delta + jq * D - T + 1, T);
    const bool sum = mine && er.straddle;
    const int first = __reduce_min_sync(0xffffffffu, sum ? er.k0 : T);
    const int last = __reduce_max_sync(0xffffffffu, sum ? er.k0 : first);  // from here on every such lane sums
    float2 B = make_float2(0.f, 0.f);
    const int kq = (b0 + first) / nph;
    int bb = b0 + first - kq * nph;
    const float2* x = xs + bb * P + kq + q0 + 32 * q;
    auto mac = [&](int k) {
      float2 gk;
      if constexpr (kPacked) {
        const float4 g4 = tp[k * NB + n];
        gk = make_float2(g4.x, g4.z);
      } else {
        gk = reinterpret_cast<const float2*>(tp)[k * kPitch + n];
      }
      const float2 v = *x;
      x += P;
      if (++bb == nph) {
        bb = 0;
        x += 1 - nph * P;
      }
      return make_float4(gk.x, gk.y, v.x, v.y);
    };
    auto add = [&](float4 m) {
      B.x = fmaf(m.x, m.z, B.x);
      B.x = fmaf(-m.y, m.w, B.x);
      B.y = fmaf(m.x, m.w, B.y);
      B.y = fmaf(m.y, m.z, B.y);
    };
    int k = first;
    for (; k < last; ++k) {
      const float4 m = mac(k);
      if (k >= er.k0) add(m);
    }
    for (; k < T; ++k) add(mac(k));
    if (mine) {
      float2* o = cm.out + ((int64_t)r + (int64_t)U * jq);
      *o = rotate_apply(er, *o, B);
    }
  }
}

// The row blocks of one work set: two rows a thread where the tile height
// allows (four in engines of one or two channels a batch), one otherwise.
template <int NB, bool kPacked>
__device__ __forceinline__ void process_block(int rows, const float2* __restrict__ xs, const float4* __restrict__ tp,
                                              const ChanMeta* __restrict__ meta, int T, int D, int P, int nph, int b0,
                                              int q0, int64_t j, int64_t J, int U, int r, int delta) {
  if (NB <= 2 && rows == 4) {
    process_rows<NB, NB <= 2 ? 4 : 2, kPacked>(xs, tp, meta, T, D, P, nph, b0, q0, j, J, U, r, delta);
  } else if (rows >= 2) {
    process_rows<NB, 2, kPacked>(xs, tp, meta, T, D, P, nph, b0, q0, j, J, U, r, delta);
  } else {
    process_rows<NB, 1, kPacked>(xs, tp, meta, T, D, P, nph, b0, q0, j, J, U, r, delta);
  }
}

// Single-channel work sets with long filters: each thread computes kWinRows
// consecutive output rows.  Taps are visited phase by phase (k = v, v + D,
// ...), where the samples of consecutive taps and consecutive rows are
// consecutive in the de-interleaved tile, so the rows share one sliding
// window of samples held in registers: one shared-memory load per tap step
// serves kWinRows outputs (the per-row path loads a sample per tap and
// output).  kWinRows is odd so the lanes of a warp (row blocks kWinRows
// apart) read distinct bank pairs.  Real taps (no NCO shift, resampler
// semantics) take 2 FMAs per tap instead of 4.
constexpr int kWinRows = 7;
// Forms of the kernel: rows; sliding window with two CTAs an SM, whose registers
// hold complex taps or a block of real ones read ahead; sliding window of real
// taps with three CTAs an SM and nothing read ahead.  The last is faster where
// three fit or the phases are few (1000 taps over 2^23 samples 762 -> 696 us,
// 8000 of one phase 6.2 -> 5.5 ms, 100 a phase at 3/2 over 2^22 108 -> 84 us);
// with fewer CTAs and more phases reading ahead is (4095 taps by 10 over 2^24
// samples 1.13 ms, 1.20 without).
constexpr int kRowForm = 0, kWinTwo = 1, kWinReal = 2;

// Shared memory of a CTA that leaves room for two more, or one more, on the SM.
constexpr int kSmem3 = 75 * 1024;
constexpr int kSmem2 = 112 * 1024;
// Taps are staged while the CTA stays within this, the SM's limit; longer
// filters of many phases read them through L1, of which the tile leaves little
// (3000 taps of four channels by 100 over 2^22 samples: 0.80 ms so, 0.41
// staged, one CTA an SM).
constexpr int kSmemTaps = 227 * 1024;
// Complex multiply-adds that a launch of their own pays for (about 60 us).
constexpr int64_t kSplitWork = 1 << 28;

// Rotation and store of one single-channel output (the per-row epilogue
// for NB = 1).
__device__ __forceinline__ void win_finish(float2 acc, const ChanMeta& cm, const float2* __restrict__ xs,
                                           const float4* __restrict__ tp, int T, int D, int P, int a0, int jl,
                                           int64_t j, int U, int r, int delta) {
  const int64_t m = (int64_t)r + (int64_t)U * j;
  const int64_t w = (int64_t)delta + j * D - T + 1;
  float2 y = acc;
  if (rotate_fast(cm, w, T, y)) {
    cm.out[m] = y;
    return;
  }
  const ExactRot er = rotate_prep(cm, w, T);
  float2 B = make_float2(0.f, 0.f);
  if (er.straddle) {
    const int kb = a0 + er.k0;
    int qq = kb / D;
    int bb = kb - qq * D;
    qq += jl;
    for (int k = er.k0; k < T; ++k) {
      const float2 x = xs[bb * P + qq];
      const float4 g4 = tp[k];
      const float2 gk = make_float2(g4.x, g4.z);
      B.x = fmaf(gk.x, x.x, B.x);
      B.x = fmaf(-gk.y, x.y, B.x);
      B.y = fmaf(gk.x, x.y, B.y);
      B.y = fmaf(gk.y, x.x, B.y);
      if (++bb == D) {
        bb = 0;
        ++qq;
      }
    }
  }
  cm.out[m] = rotate_apply(er, acc, B);
}

template <bool kReal, bool kAhead>
__device__ __forceinline__ void win_sums(const float2* __restrict__ xs, const float4* __restrict__ tp, int T, int D,
                                         int P, int a0, int jl0, f32x2 (&acc)[kWinRows]) {
  // packed multiply-adds in the scalar form's order: (re, re) (x, y), then
  // (-im, im) (y, x) for complex taps
#pragma unroll
  for (int q = 0; q < kWinRows; ++q) acc[q] = 0ull;
  const int bq = a0 / D, b0 = a0 - bq * D;
  const int nv = T < D ? T : D;
  for (int vp = 0; vp < nv; ++vp) {
    int ph = b0 + vp, q0 = bq + jl0;
    if (ph >= D) {
      ph -= D;
      ++q0;
    }
    const f32x2* xr = reinterpret_cast<const f32x2*>(xs + ph * P + q0);  // row jl0 + q, tap vp + m D: xr[m + q]
    const ulonglong2* tk = reinterpret_cast<const ulonglong2*>(tp + vp);
    const int nm = (T - 1 - vp) / D + 1;
    f32x2 w[kWinRows], sw[kReal ? 1 : kWinRows];  // samples, and with re and im exchanged
    auto put = [&](int i, f32x2 v) {
      w[i] = v;
      if constexpr (!kReal) {
        const float2 f = unpack2(v);
        sw[i] = pack2(f.y, f.x);
      }
    };
    auto tap = [&](int m, f32x2& gr, f32x2& gi) {
      if constexpr (kReal) {
        gr = tk[m * D].x;
      } else {
        const ulonglong2 g = tk[m * D];
        const float2 f = unpack2(g.y);
        gr = g.x;
        gi = pack2(-f.x, f.y);
      }
    };
#pragma unroll
    for (int q = 0; q < kWinRows - 1; ++q) put(q, xr[q]);
    int m = 0;
    for (; m + kWinRows <= nm; m += kWinRows) {
      // circular window: sample m + u + q sits in slot (u + q) % kWinRows; real
      // taps leave two CTAs the registers to read the block's taps and samples first
      f32x2 xn[kAhead ? kWinRows : 1], gn[kAhead ? kWinRows : 1];
      if constexpr (kAhead) {
#pragma unroll
        for (int u = 0; u < kWinRows; ++u) {
          xn[u] = xr[m + u + kWinRows - 1];
          gn[u] = tk[(m + u) * D].x;
        }
      }
#pragma unroll
      for (int u = 0; u < kWinRows; ++u) {
        f32x2 gr, gi = 0ull;
        if constexpr (kAhead) {
          put((u + kWinRows - 1) % kWinRows, xn[u]);
          gr = gn[u];
        } else {
          put((u + kWinRows - 1) % kWinRows, xr[m + u + kWinRows - 1]);
          tap(m + u, gr, gi);
        }
#pragma unroll
        for (int q = 0; q < kWinRows; ++q) {
          acc[q] = fma2(gr, w[(u + q) % kWinRows], acc[q]);
          if constexpr (!kReal) acc[q] = fma2(gi, sw[(u + q) % kWinRows], acc[q]);
        }
      }
    }
    for (; m < nm; ++m) {
      put(kWinRows - 1, xr[m + kWinRows - 1]);
      f32x2 gr, gi = 0ull;
      tap(m, gr, gi);
#pragma unroll
      for (int q = 0; q < kWinRows; ++q) {
        acc[q] = fma2(gr, w[q], acc[q]);
        if constexpr (!kReal) acc[q] = fma2(gi, sw[q], acc[q]);
      }
#pragma unroll
      for (int q = 0; q < kWinRows - 1; ++q) {
        w[q] = w[q + 1];
        if constexpr (!kReal) sw[q] = sw[q + 1];
      }
    }
  }
}

// History after a block: the last H samples of [old history | block], sample
// i of the new buffer.
__device__ __forceinline__ void hist_sample(const float2* __restrict__ old_hist, const float2* __restrict__ block,
                                            const short2* __restrict__ block16, int64_t N, int H,
                                            float2* __restrict__ new_hist, int i) {
  const int64_t v = N + i;
  if (v < H) {
    new_hist[i] = old_hist[v];
  } else if (block16 != nullptr) {
    const short2 s = block16[v - H];
    new_hist[i] = make_float2((float)s.x, (float)s.y);
  } else {
    new_hist[i] = block[v - H];
  }
}

// One CTA = one tile of Qt output rows of a decimation group; the tiles of the
// launch's groups (fuse_map[first ..]) follow one another in blockIdx.x, and
// the blocks past the last tile write the history of the next block.  Shared
// memory: [input tile, de-interleaved: nph x P float2][taps of every work set
// of the group][ChanMeta per (work set, channel)].
//
// One launch over all groups: a group alone has 100-400 tiles, 1-2 a SM, so
// launches one after another each ended in a nearly empty wave (64 channels of
// 2^20 samples: 12 launches 165 us, one launch 82 us).
//
// The tile holds the input phases that some window reads: all D of them where
// windows overlap or wrap, else (long decimations) only the groups' windows,
// up to kMaxSegs segments of them (seg_at / seg_gap map a staged phase to its
// place in the row).
template <int NBMAX, int kTaps, int kForm>
__global__ void __launch_bounds__(kThreads, kForm == kWinTwo || (kForm == kRowForm && NBMAX == 8) ? 2 : 3)
    poly_fp32_kernel(const __grid_constant__ PolyLaunch<NBMAX> L, int first, int tiles) {
  extern __shared__ __align__(16) float2 xs[];
  grid_dependency();
  int tile = blockIdx.x;
  if (tile >= tiles) {
    const int i = (tile - tiles) * kThreads + (int)threadIdx.x;
    if (i < L.H) hist_sample(L.hist, L.block, L.block16, L.N, L.H, L.new_hist, i);
    return;
  }
  for (; tile >= L.groups[L.fuse_map[first]].ntiles; ++first) tile -= L.groups[L.fuse_map[first]].ntiles;
  const GroupDesc& G = L.groups[L.fuse_map[first]];
  const int D = G.D, Qt = G.Qt, P = G.P, nph = G.nph;
  const int64_t row0 = (int64_t)tile * Qt;
  const int64_t sb = row0 * D + G.delta_min - G.tmax + 1 + G.seg_first;  // first staged input (block relative)
  const int len = G.len;
  float4* taps_s = reinterpret_cast<float4*>(xs + G.taps_off);
  ChanMeta* meta_s = reinterpret_cast<ChanMeta*>(xs + G.meta_off);
  const int nws = G.ws_end - G.ws_begin;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // Stage the raw input span, de-interleaved by D, with asynchronous 8-byte
  // copies (every copy of the tile in flight at once).  Negative indices come
  // from the history (the H samples before the block); past the block end the
  // copy reads 0 bytes and zero-fills.
  // Sample t of the tile is phase b = t mod nph of row q = t / nph, stepped
  // by kThreads; a tile inside the block skips the range checks.
  {
    int q = (int)(((uint64_t)threadIdx.x * G.inv_nph) >> 32);
    int b = (int)threadIdx.x - q * nph;
    const int dq = G.step_q, db = G.step_b;
    const int at0 = G.seg_at[0], at1 = G.seg_at[1], at2 = G.seg_at[2];
    const int gap0 = G.seg_gap[0], gap1 = G.seg_gap[1], gap2 = G.seg_gap[2];
    const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(xs);
    auto place = [&]() {  // sample of the tile's span
      return q * D + b + (b >= at0 ? gap0 : 0) + (b >= at1 ? gap1 : 0) + (b >= at2 ? gap2 : 0);
    };
    auto advance = [&]() {
      b += db;
      q += dq;
      if (b >= nph) {
        b -= nph;
        ++q;
      }
    };
    if (L.block16 == nullptr && sb >= 0 && sb + G.span <= L.N) {
      const float2* src = L.block + sb;
      if (nph == D) {
        src += threadIdx.x;
        for (int t = threadIdx.x; t < len; t += kThreads, src += kThreads, advance())
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst0 + 8u * (uint32_t)(b * P + q)), "l"(src)
                       : "memory");
      } else {
        for (int t = threadIdx.x; t < len; t += kThreads, advance())
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst0 + 8u * (uint32_t)(b * P + q)),
                       "l"(src + place())
                       : "memory");
      }
    } else if (L.block16 == nullptr) {
      for (int t = threadIdx.x; t < len; t += kThreads, advance()) {
        const int64_t v = sb + place();
        const float2* src = L.block;
        uint32_t bytes = 0;
        if (v < 0) {
          const int64_t hv = v + L.H;
          if (hv >= 0) {
            src = L.hist + hv;
            bytes = 8;
          }
        } else if (v < L.N) {
          src = L.block + v;
          bytes = 8;
        }
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst0 + 8u * (uint32_t)(b * P + q)),
                     "l"(src), "r"(bytes)
                     : "memory");
      }
    } else {
      // int16 front end: block samples are converted on the way in (the
      // history is already float), four loads in flight a thread
      for (int t = threadIdx.x; t < len;) {
        float2 x[4];
        int at[4];
#pragma unroll
        for (int u = 0; u < 4; ++u, t += kThreads, advance()) {
          at[u] = -1;
          x[u] = make_float2(0.f, 0.f);
          if (t >= len) continue;
          at[u] = b * P + q;
          const int64_t v = sb + place();
          if (v < 0) {
            const int64_t hv = v + L.H;
            if (hv >= 0) x[u] = L.hist[hv];
          } else if (v < L.N) {
            const short2 s = L.block16[v];
            x[u] = make_float2((float)s.x, (float)s.y);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (at[u] >= 0) xs[at[u]] = x[u];
      }
    }
  }
  // Stage the taps of every work set (when they fit) and the per-channel NCO
  // constants: a warp a work set, every copy in flight at once (one work set
  // after another with plain loads took a memory latency each).
  for (int wi = warp; wi < nws; wi += kThreads / 32) {
    const WorkSet<NBMAX>& W = L.ws[G.ws_begin + wi];
    if constexpr (kTaps != kTapsGlobal) {
      const int cnt = kTaps == kTapsPacked ? W.T * W.nb : W.T * ((W.nb + 1) >> 1);
      const float4* src = W.taps;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(taps_s + W.soff);
      for (int i = lane; i < cnt; i += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16u * (uint32_t)i), "l"(src + i)
                     : "memory");
    }
    if (lane < W.nb) {
      const int c = W.ch[lane];
      const NcoConst nc = L.nco[c];
      ChanMeta m;
      m.omega64 = nc.omega64;
      m.wrap64 = nc.wrap64;
      m.fastmod = nc.fastmod;
      m.out = L.out[c];
      m.rollover = nc.rollover;
      m.base = L.nco_base[c];
      m.enabled = nc.enabled;
      m.step32 = nc.rollover ? (32u * (uint32_t)D) % nc.rollover : 0u;
      meta_s[wi * NBMAX + lane] = m;
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  if constexpr (kForm != kRowForm) {
    // single-channel work sets: items are (work set, block of kWinRows rows),
    // blocks fastest (Qt is a multiple of 32 kWinRows)
    const int nblk = Qt / kWinRows;
    const int nitems = nws * nblk;
    f32x2 acc[kWinRows];
    // One unshifted channel, a block a thread: the tile's outputs (every phase
    // of every row, contiguous in the channel) go back through shared memory
    // and leave in whole lines.  Stored from the registers, neighbouring lanes
    // are 7 rows apart (a sector per 8 bytes), and each output paid a rotation:
    // 64 complex taps over 2^20 samples, 26 us so, 18 us here.
    if (G.lines) {
      const int wq = (int)threadIdx.x / nblk, U = nws;
      const int jl0 = ((int)threadIdx.x - wq * nblk) * kWinRows;
      const WorkSet<NBMAX>& W = L.ws[G.ws_begin + min(wq, nws - 1)];
      const bool mine = wq < nws && row0 + jl0 < W.J;
      if (mine) {
        const int a0 = (W.delta - G.delta_min) + (G.tmax - W.T);
        const float4* tp = kTaps != kTapsGlobal ? taps_s + W.soff : W.taps;
        if (kForm == kWinReal || G.real_taps)
          win_sums<true, kForm == kWinTwo>(xs, tp, W.T, D, P, a0, jl0, acc);
        else
          win_sums<false, false>(xs, tp, W.T, D, P, a0, jl0, acc);
      }
      float2* const out = meta_s[0].out + row0 * U;
      __syncthreads();  // every window is summed: the tile is free
      if (mine) {
#pragma unroll
        for (int q = 0; q < kWinRows; ++q)
          xs[(jl0 + q) * U + W.r] = cmul_nco(unpack2(acc[q]), make_float2(1.f, 0.f));
      }
      __syncthreads();
      const int count = (int)min((int64_t)Qt * U, G.outs - row0 * U);
      for (int i = threadIdx.x; i < count; i += kThreads) out[i] = xs[i];
      return;
    }
    for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
      const int wq = it / nblk;
      const int jl0 = (it - wq * nblk) * kWinRows;
      const WorkSet<NBMAX>& W = L.ws[G.ws_begin + wq];
      const int64_t j0 = row0 + jl0;
      if (j0 >= W.J) continue;
      const int T = W.T;
      const int a0 = (W.delta - G.delta_min) + (G.tmax - T);
      const float4* tp = kTaps != kTapsGlobal ? taps_s + W.soff : W.taps;
      const ChanMeta* mt = meta_s + wq * NBMAX;
      if (kForm == kWinReal || G.real_taps)
        win_sums<true, kForm == kWinTwo>(xs, tp, T, D, P, a0, jl0, acc);
      else
        win_sums<false, false>(xs, tp, T, D, P, a0, jl0, acc);
#pragma unroll
      for (int q = 0; q < kWinRows; ++q)
        if (j0 + q < W.J)
          win_finish(unpack2(acc[q]), mt[0], xs, tp, T, D, P, a0, jl0 + q, j0 + q, W.U, W.r, W.delta);
    }
    return;
  }

  // Items are (work set, block of 32 kRows rows), a warp each, so every tap
  // load is a broadcast.
  const int rows = G.rows;
  const int nblk = Qt / (32 * rows);
  const int nitems = nws * nblk;
  for (int it = warp; it < nitems; it += kThreads / 32) {
    const int wq = it / nblk;
    const int jl = (it - wq * nblk) * 32 * rows;
    const WorkSet<NBMAX>& W = L.ws[G.ws_begin + wq];
    if (row0 + jl >= W.J) continue;
    const int64_t j = row0 + jl + lane;
    const int T = W.T, b0 = W.b0, q0 = W.q0 + jl + lane;
    const float4* tp = kTaps != kTapsGlobal ? taps_s + W.soff : W.taps;
    const ChanMeta* mt = meta_s + wq * NBMAX;
#define FDSP_NB(n)                                                                                        \
  case n:                                                                                                 \
    if constexpr (NBMAX >= n)                                                                             \
      process_block<n, kTaps == kTapsPacked>(rows, xs, tp, mt, T, D, P, nph, b0, q0, j, (int64_t)W.J, W.U, W.r, W.delta);       \
    break;
    switch (W.nb) {
      FDSP_NB(1)
      FDSP_NB(2)
      FDSP_NB(3)
      FDSP_NB(4)
      FDSP_NB(5)
      FDSP_NB(6)
      FDSP_NB(7)
      FDSP_NB(8)
      default: break;
    }
#undef FDSP_NB
  }
}

// Rational resampling of one unshifted channel with many output phases
// (kNatMinUp to kNatMaxUp): consecutive outputs on consecutive lanes.  Their windows
// start D / U samples apart, so sample reads of the tile as it lies in memory
// hardly conflict, the taps lie in output order (column r of [T][U]: phase r D
// mod U; conflict-free, staged as they lie), and stores are contiguous.  The row form gives each of the U phases its own work
// set: outputs U apart on neighbouring lanes (a sector per 8-byte store) and a
// tile 160 x 34 samples that leaves one CTA an SM.  Bound: shared-memory reads
// (a sample per output and tap; a tap read feeds the thread's four outputs,
// whose windows lie whole periods apart).  147/160 of 2^20 samples, 24 taps
// a phase: 31 us in row form, 17 us here (cold cache).  Sums run in the row form's order.
// kCheck keeps that form's products with the taps' zero imaginary parts: an
// infinite or NaN sample then marks both parts of an output, as it did there.
constexpr int kNatMinUp = 16;
constexpr int kNatMaxUp = kMaxWorkSets;  // an apply builds a work set per phase first, and refuses more
constexpr int kNatMaxTaps = 8192;  // U T: 32 KB of taps in shared memory
constexpr int kNatPer = 4;         // outputs a thread of a full tile
constexpr int kNatMaxCols = 512;   // threads of a CTA: a multiple of U columns, rounded up to warps

template <bool kCheck>
__global__ void __launch_bounds__(kNatMaxCols) nat_resample_kernel(const __grid_constant__ NatLaunch L, int tiles) {
  extern __shared__ __align__(16) float2 xs[];
  grid_dependency();
  const int threads = (int)blockDim.x;
  if ((int)blockIdx.x >= tiles) {
    const int i = ((int)blockIdx.x - tiles) * threads + (int)threadIdx.x;
    if (i < L.H) hist_sample(L.hist, L.block, L.block16, L.N, L.H, L.new_hist, i);
    return;
  }
  const int U = L.U, D = L.D, T = L.T, cols = L.cols;
  const int64_t m0 = (int64_t)blockIdx.x * (L.per * cols);  // a multiple of U: every tile starts at the same phase
  const int count = (int)min((int64_t)L.per * cols, L.M - m0);
  const int64_t s0 = L.xoffset + (m0 / U) * D - T + 1;  // first sample of output m0's window
  const uint32_t ph0 = L.phase;
  float* const taps = reinterpret_cast<float*>(xs + L.len);
  const int len = (int)((ph0 + (uint64_t)(count - 1) * D) / U) + T;  // samples the outputs read (<= L.len)
  for (int i = threadIdx.x; i < len; i += threads) {
    const int64_t v = s0 + i;
    if (L.block16 == nullptr) {
      const float2* src = L.block;
      uint32_t bytes = 0;
      if (v < 0) {
        if (v + L.H >= 0) {
          src = L.hist + (v + L.H);
          bytes = 8;
        }
      } else if (v < L.N) {
        src = L.block + v;
        bytes = 8;
      }
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(xs + i)),
                   "l"(src), "r"(bytes)
                   : "memory");
    } else {
      float2 x = make_float2(0.f, 0.f);
      if (v < 0) {
        if (v + L.H >= 0) x = L.hist[v + L.H];
      } else if (v < L.N) {
        const short2 s = L.block16[v];
        x = make_float2((float)s.x, (float)s.y);
      }
      xs[i] = x;
    }
  }
  for (int i = threadIdx.x; i < (U * T + 3) / 4; i += threads)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(taps) + 16u * (uint32_t)i),
                 "l"(reinterpret_cast<const float4*>(L.taps) + i)
                 : "memory");
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  // column c of the tile: outputs c, c + cols, ..., whose windows lie
  // cols / U * D samples apart and share their taps
  const int c = (int)threadIdx.x;
  if (c >= cols || c >= count) return;
  const f32x2* xp = reinterpret_cast<const f32x2*>(xs) + (ph0 + (uint32_t)c * (uint32_t)D) / (uint32_t)U;
  const float* tp = taps + (uint32_t)(L.r_first + c) % (uint32_t)U;
  auto run = [&](auto outs) {
    constexpr int kOuts = decltype(outs)::value;
    f32x2 acc[kOuts], chk[kOuts];
    int off[kOuts];
#pragma unroll
    for (int q = 0; q < kOuts; ++q) {
      off[q] = c + q * cols < count ? q * (cols / U * D) : 0;  // (past the end: a valid window, not stored)
      acc[q] = chk[q] = 0ull;
    }
#pragma unroll 2
    for (int k = 0; k < T; ++k) {
      const float h = tp[k * U];
      const f32x2 hh = pack2(h, h);
#pragma unroll
      for (int q = 0; q < kOuts; ++q) {
        const f32x2 x = xp[k + off[q]];
        acc[q] = fma2(hh, x, acc[q]);
        if constexpr (kCheck) chk[q] = fma2(0ull, x, chk[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < kOuts; ++q) {
      if (c + q * cols >= count) continue;
      float2 y = unpack2(acc[q]);
      if constexpr (kCheck) {
        const float2 z = unpack2(chk[q]);
        y = make_float2(y.x - z.y, y.y + z.x);
      }
      L.out[m0 + c + q * cols] = y;
    }
  };
  if (L.per == kNatPer) run(std::integral_constant<int, kNatPer>());
  else run(std::integral_constant<int, 1>());
}

// The history update alone (applies whose groups all ran on the tensor cores).
__global__ void hist_update_kernel(const float2* __restrict__ old_hist, const float2* __restrict__ block,
                                   const short2* __restrict__ block16, int64_t N, int H, float2* __restrict__ new_hist) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < H) hist_sample(old_hist, block, block16, N, H, new_hist, i);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
cudaError_t launch_overlapped(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t s, void** args) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const bool known = cudaStreamIsCapturing(s, &cs) == cudaSuccess;
  if (!known) cudaGetLastError();
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = known && cs == cudaStreamCaptureStatusNone ? 1u : 0u;
  return cudaLaunchKernelExC(&cfg, func, args);
}

NcoConst make_nco(uint32_t fs, int32_t f) {
  NcoConst n;
  std::memset(&n, 0, sizeof(n));
  if (f == 0 || fs == 0) return n;
  // rollover index: falcon_dsp_freq_shift.cc:216-229
  double r = (double)fs / (double)std::llabs((long long)f);
  while (r < 1e5) r *= 10.0;
  const uint32_t R = (uint32_t)std::round(r);
  int64_t fm = (int64_t)f % (int64_t)fs;
  if (fm < 0) fm += fs;
  const unsigned __int128 num = ((unsigned __int128)(uint64_t)fm << 64) + (fs / 2);
  const uint64_t w = (uint64_t)(num / fs);
  n.omega64 = w;
  n.wrap64 = (uint64_t)R * w;
  n.rollover = R;
  n.fastmod = R ? (~0ull / R + 1) : 0;
  n.enabled = (R != 0) ? 1u : 0u;
  return n;
}

PolyEngine::~PolyEngine() {
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  if (graph_) cudaGraphDestroy(graph_);
  for (auto e : kprof_ev_)
    if (e) cudaEventDestroy(e);
  free_tc();
  for (auto& b : batches_) {
    if (b.d_taps) dfree(b.d_taps);
  }
  if (d_nco_) dfree(d_nco_);
  if (d_nat_) dfree(d_nat_);
  for (auto& h : d_hist_) {
    if (h) dfree(h);
  }
}

// ---------------------------------------------------------------------------
// device memory: the engine's own buffers come from its pool when it has one
// ---------------------------------------------------------------------------
cudaError_t PolyEngine::dalloc(void** p, size_t bytes) {
  if (!pool_) return cudaMalloc(p, bytes);
  *p = pool_->alloc(bytes);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}

void PolyEngine::dfree(void* p) {
  if (!p) return;
  if (pool_) pool_->release(p);
  else cudaFree(p);
}

DevPool::~DevPool() {
  if (base_) cudaFree(base_);
}

int DevPool::init(size_t bytes) {
  std::lock_guard<std::mutex> lk(mu_);
  if (base_ || bytes < RangePool::kAlign) return FDSP_ERR_INVALID_ARG;
  bytes &= ~(RangePool::kAlign - 1);
  const cudaError_t e = cudaMalloc(&base_, bytes);
  if (e != cudaSuccess) {
    base_ = nullptr;
    return cuda_status(e);
  }
  ranges_.init(bytes);
  return FDSP_OK;
}

void* DevPool::alloc(size_t bytes) {
  std::lock_guard<std::mutex> lk(mu_);
  if (!base_) return nullptr;
  const size_t off = ranges_.alloc(bytes);
  return off == RangePool::kNone ? nullptr : base_ + off;
}

void DevPool::release(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(mu_);
  if (base_) ranges_.release((size_t)(static_cast<char*>(p) - base_));
}

static int choose_qt(uint32_t D, int tmax) {
  // ~4K input samples per tile (three CTAs per SM), two warps' rows where that
  // stays within ~8K samples (a thread then computes two rows or more), at
  // least one; shared memory (tile + halo + offset spread, de-interleaved)
  // under ~200 KB.
  int qt = (int)((4096 / D) & ~63u);
  if (qt < 64) qt = D <= 128 ? 64 : 32;
  auto bytes = [&](int q) {
    const int64_t len = (int64_t)q * D + 3LL * D + tmax;
    const int64_t P = len / D + 2;
    return (int64_t)D * P * 8;
  };
  while (qt > 32 && bytes(qt) > 200 * 1024) qt -= 32;
  if (bytes(qt) > 200 * 1024) return -1;
  return qt;
}

int PolyEngine::init(uint32_t fs, const fdsp_channel_cfg* ch, uint32_t nch, bool complex_taps, cudaStream_t stream) {
  if (nch == 0 || ch == nullptr) return FDSP_ERR_INVALID_ARG;
  if (nch > (uint32_t)kMaxChannels) return FDSP_ERR_UNSUPPORTED;
  fs_ = fs;
  complex_taps_ = complex_taps;
  chans_.resize(nch);
  cls_of_.assign(nch, -1);
  int tmax_all = 1;
  for (uint32_t c = 0; c < nch; ++c) {
    const fdsp_channel_cfg& cc = ch[c];
    if (cc.up_rate == 0 || cc.down_rate == 0 || cc.num_coeffs == 0 || cc.resample_filter_coeffs == nullptr)
      return FDSP_ERR_INVALID_ARG;
    EngineChannel& e = chans_[c];
    e.up = cc.up_rate;
    e.down = cc.down_rate;
    // polyphase_resampler.cc:131-157 -- pad to a multiple of up, transpose, flip
    uint32_t padded = cc.num_coeffs;
    while (padded % e.up) padded++;
    e.T = padded / e.up;
    e.flipped.assign((size_t)padded, make_float2(0.f, 0.f));
    for (uint32_t ph = 0; ph < e.up; ++ph) {
      for (uint32_t jj = 0; jj < e.T; ++jj) {
        const uint64_t src = (uint64_t)jj * e.up + ph;
        if (src < cc.num_coeffs) {
          const fdsp_cf32 v = cc.resample_filter_coeffs[src];
          e.flipped[(size_t)ph * e.T + (e.T - 1 - jj)] = make_float2(v.re, complex_taps ? v.im : 0.f);
        }
      }
    }
    e.shift_hz = (int32_t)cc.freq_shift_in_hz;  // initialize(uint32_t, int32_t) truncation
    e.nco = make_nco(fs, e.shift_hz);
    if (e.nco.enabled && e.T > e.nco.rollover) return FDSP_ERR_UNSUPPORTED;
    tmax_all = std::max(tmax_all, (int)e.T);
    // class by (up, down)
    int k = -1;
    for (size_t i = 0; i < classes_.size(); ++i) {
      if (classes_[i].up == e.up && classes_[i].down == e.down) k = (int)i;
    }
    if (k < 0) {
      EngineClass nc;
      nc.up = e.up;
      nc.down = e.down;
      nc.phase = 0;
      nc.xoffset = 0;
      nc.M = 0;
      classes_.push_back(nc);
      k = (int)classes_.size() - 1;
    }
    classes_[k].chans.push_back((int)c);
    cls_of_[c] = k;
  }
  H_ = tmax_all - 1;

  // NB: channels per tap batch (largest class decides).  Four: the kernel then
  // keeps three CTAs an SM (eight leave two: 256 channels of 2^26 samples took
  // 18.9 ms by eight and 15.9 by four); eight only where batches of four would
  // exceed a launch's work sets.
  size_t maxcls = 1, sets4 = 0;
  for (auto& k : classes_) {
    maxcls = std::max(maxcls, k.chans.size());
    sets4 += (k.chans.size() + 3) / 4 * k.up;
  }
  nb_ = maxcls >= 8 && sets4 > (size_t)kMaxWorkSets ? 8 : maxcls >= 4 ? 4 : maxcls >= 2 ? 2 : 1;

  // decimation groups
  std::map<uint32_t, int> gidx;
  for (auto& k : classes_) {
    if (!gidx.count(k.down)) {
      gidx[k.down] = (int)groups_.size();
      EngineGroup g;
      g.D = k.down;
      g.Qt = 0;
      groups_.push_back(g);
    }
  }
  if (groups_.size() > (size_t)kMaxGroups) return FDSP_ERR_UNSUPPORTED;

  // batches: within a class, channels sorted by taps per phase (descending)
  for (size_t ki = 0; ki < classes_.size(); ++ki) {
    std::vector<int> cs = classes_[ki].chans;
    std::stable_sort(cs.begin(), cs.end(), [&](int a, int b) { return chans_[a].T > chans_[b].T; });
    for (size_t i = 0; i < cs.size(); i += nb_) {
      EngineBatch bt;
      bt.cls = (int)ki;
      bt.group = gidx[classes_[ki].down];
      bt.chans.assign(cs.begin() + i, cs.begin() + std::min(cs.size(), i + nb_));
      bt.T = (int)chans_[bt.chans[0]].T;
      bt.d_taps = nullptr;
      groups_[bt.group].batches.push_back((int)batches_.size());
      batches_.push_back(bt);
    }
  }
  for (size_t gi = 0; gi < groups_.size(); ++gi) group_of_d_[groups_[gi].D] = (int)gi;
  for (auto& g : groups_) {
    int tmax = 1;
    for (int b : g.batches) tmax = std::max(tmax, batches_[b].T);
    g.Qt = choose_qt(g.D, tmax);
    if (g.Qt < 0) return FDSP_ERR_UNSUPPORTED;
    g.Qt_default = g.Qt;
    // sliding-window form: every batch of the group holds one channel and
    // the filter is long enough for row blocks to pay; tiles of a multiple
    // of 32 x kWinRows rows within the same shared-memory budget
    bool single = true, real = true;
    for (int b : g.batches) {
      single = single && batches_[b].chans.size() == 1;
      for (int c : batches_[b].chans) {
        real = real && !chans_[c].nco.enabled;
        for (const float2& h : chans_[c].flipped) real = real && h.y == 0.f;
      }
    }
    const int unit = 32 * kWinRows;
    if (single && tmax >= 16) {
      auto bytes = [&](int q) {
        const int64_t len = (int64_t)q * g.D + 3LL * g.D + tmax;
        return (int64_t)g.D * (len / g.D + 2) * 8;
      };
      // enough row blocks for every thread of the CTA: kThreads blocks of
      // kWinRows rows spread over the group's work sets (U output phases each
      // class), as far as shared memory allows
      size_t nws = 0;
      for (int b : g.batches) nws += classes_[batches_[b].cls].up;
      const int want = (int)((kThreads + std::max<size_t>(nws, 1) - 1) / std::max<size_t>(nws, 1)) * kWinRows;
      int q = std::max(unit, (want + unit - 1) / unit * unit);
      while (q > unit && bytes(q) > 200 * 1024) q -= unit;
      if (bytes(q) <= 200 * 1024) {
        g.win = 1;
        g.real_taps = real ? 1 : 0;
        g.Qt_win = q;
      }
    }
  }

  // modulated, padded taps of every batch: [up][T][channels] as (re, re, im,
  // im), then as (re, im) with the channels padded to an even number
  for (auto& bt : batches_) {
    const uint32_t U = classes_[bt.cls].up;
    const size_t nb = bt.chans.size();
    const size_t packed = (size_t)U * bt.T * nb, pitch = (nb + 1) & ~(size_t)1;
    std::vector<float4> host(packed + (size_t)U * bt.T * pitch / 2, make_float4(0.f, 0.f, 0.f, 0.f));
    float2* const compact = reinterpret_cast<float2*>(host.data() + packed);
    for (size_t n = 0; n < bt.chans.size(); ++n) {
      const EngineChannel& e = chans_[bt.chans[n]];
      const int pad = bt.T - (int)e.T;
      int64_t fm = 0;
      if (e.nco.enabled) {
        fm = (int64_t)e.shift_hz % (int64_t)fs;
        if (fm < 0) fm += fs;
      }
      for (uint32_t ph = 0; ph < U; ++ph) {
        for (int k = pad; k < bt.T; ++k) {
          const float2 h = e.flipped[(size_t)ph * e.T + (k - pad)];
          double gr = h.x, gi = h.y;
          if (e.nco.enabled) {
            // e^{j w k} with w k reduced exactly: 2 pi ((f mod fs) k mod fs) / fs
            const uint64_t red = (uint64_t)(((unsigned __int128)(uint64_t)fm * (uint64_t)k) % fs);
            const double ang = 2.0 * M_PI * (double)red / (double)fs;
            const double c = std::cos(ang), s = std::sin(ang);
            gr = (double)h.x * c - (double)h.y * s;
            gi = (double)h.x * s + (double)h.y * c;
          }
          host[((size_t)ph * bt.T + k) * nb + n] = make_float4((float)gr, (float)gr, (float)gi, (float)gi);
          compact[((size_t)ph * bt.T + k) * pitch + n] = make_float2((float)gr, (float)gi);
        }
      }
    }
    cudaError_t e = dalloc(reinterpret_cast<void**>(&bt.d_taps), host.size() * sizeof(float4));
    if (e != cudaSuccess) return cuda_status(e);
    e = cudaMemcpy(bt.d_taps, host.data(), host.size() * sizeof(float4), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_status(e);
  }

  // one unshifted channel of many phases, every phase in turn (up and down
  // coprime), whose windows move slowly (a tile of outputs spans at most 4
  // samples an output): the many-phase form, its taps in output order
  const uint32_t U0 = chans_[0].up, D0 = chans_[0].down;
  uint32_t g0 = U0;
  for (uint32_t b = D0, r; b; b = r) {
    r = g0 % b;
    g0 = b;
  }
  if (nch == 1 && !complex_taps && !chans_[0].nco.enabled && U0 >= (uint32_t)kNatMinUp && U0 <= (uint32_t)kNatMaxUp && g0 == 1 &&
      D0 <= 4u * U0 && (uint64_t)U0 * chans_[0].T <= (uint64_t)kNatMaxTaps) {
    const uint32_t T0 = chans_[0].T;
    std::vector<float> host(((size_t)U0 * T0 + 3) & ~(size_t)3, 0.f);
    nat_col_.assign(U0, 0);
    for (uint32_t r = 0; r < U0; ++r) {
      const uint32_t phi = (uint32_t)((uint64_t)r * D0 % U0);
      nat_col_[phi] = (int32_t)r;
      for (uint32_t k = 0; k < T0; ++k) host[(size_t)k * U0 + r] = chans_[0].flipped[(size_t)phi * T0 + k].x;
    }
    cudaError_t e = dalloc(reinterpret_cast<void**>(&d_nat_), host.size() * sizeof(float));
    if (e != cudaSuccess) return cuda_status(e);
    e = cudaMemcpy(d_nat_, host.data(), host.size() * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_status(e);
  }

  std::vector<NcoConst> nco(nch);
  for (uint32_t c = 0; c < nch; ++c) nco[c] = chans_[c].nco;
  cudaError_t e = dalloc(reinterpret_cast<void**>(&d_nco_), nch * sizeof(NcoConst));
  if (e != cudaSuccess) return cuda_status(e);
  e = cudaMemcpy(d_nco_, nco.data(), nch * sizeof(NcoConst), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_status(e);
  if (H_ > 0) {
    for (auto& h : d_hist_) {
      e = dalloc(reinterpret_cast<void**>(&h), (size_t)H_ * sizeof(float2));
      if (e != cudaSuccess) return cuda_status(e);
      e = stream ? cudaMemsetAsync(h, 0, (size_t)H_ * sizeof(float2), stream)
                 : cudaMemset(h, 0, (size_t)H_ * sizeof(float2));
      if (e != cudaSuccess) return cuda_status(e);
    }
  }
  // with a stream the engine's applies on it follow the fill; without one
  // every later stream must see it
  if (!stream) {
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_status(e);
  }
  return FDSP_OK;
}

// Outputs the reference loop emits for n inputs from (phase, xoffset):
// the m >= 0 with xoffset + floor((phase + m*down)/up) < n.
uint64_t polyphase_out_count(uint32_t up, uint32_t down, uint32_t phase, uint64_t xoffset, uint64_t n) {
  if (xoffset >= n) return 0;
  const unsigned __int128 lim = (unsigned __int128)up * (n - xoffset);  // > phase
  return (uint64_t)((lim - phase + down - 1) / down);
}

// State after M outputs of an apply of n inputs (polyphase_resampler.cc:303-312).
void polyphase_advance(uint32_t up, uint32_t down, uint32_t& phase, uint64_t& xoffset, uint64_t n, uint64_t M) {
  if (xoffset >= n) {
    xoffset -= n;
    return;
  }
  const unsigned __int128 t = (unsigned __int128)phase + (unsigned __int128)M * down;
  const uint64_t x_new = xoffset + (uint64_t)(t / up);
  phase = (uint32_t)(t % up);
  xoffset = x_new - n;
}

static uint64_t class_out_count(const EngineClass& k, uint64_t n) {
  return polyphase_out_count(k.up, k.down, k.phase, k.xoffset, n);
}

int PolyEngine::out_counts(uint64_t n_in, uint64_t* n_out) const {
  if (!n_out) return FDSP_ERR_INVALID_ARG;
  for (size_t c = 0; c < chans_.size(); ++c) n_out[c] = class_out_count(classes_[cls_of_[c]], n_in);
  return FDSP_OK;
}

int PolyEngine::set_precision(int mode) {
  if (mode == precision_) return FDSP_OK;
  if (mode == FDSP_PRECISION_FP32) {
    precision_ = mode;
    return FDSP_OK;
  }
  if (mode != FDSP_PRECISION_FP16X3 && mode != FDSP_PRECISION_BF16X3) return FDSP_ERR_INVALID_ARG;
  const int st = build_tc(mode == FDSP_PRECISION_FP16X3 ? 0 : 1);
  if (st != FDSP_OK) return st;
  precision_ = mode;
  return FDSP_OK;
}

void PolyEngine::notify_done(const std::vector<int>& egroups, cudaStream_t stream) {
  if (!done_fn_ || egroups.empty()) return;
  std::vector<int> ch;
  for (int eg : egroups)
    for (const EngineClass& k : classes_)
      if (k.down == groups_[eg].D && k.M > 0) ch.insert(ch.end(), k.chans.begin(), k.chans.end());
  if (!ch.empty()) done_fn_(done_ctx_, ch.data(), (int)ch.size(), stream);
}

void PolyEngine::set_graph(bool on) {
  use_graph_ = on;
  graph_replays_ = 0;
  if (!on) {
    if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
    graph_exec_ = nullptr;
    if (graph_) cudaGraphDestroy(graph_);
    graph_ = nullptr;
    knodes_.clear();
  }
}

void PolyEngine::set_profile(bool on) {
  kprof_ = on;
  kprof_used_ = 0;
}

cudaEvent_t PolyEngine::kprof_event() {
  if (kprof_used_ == kprof_ev_.size()) {
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    kprof_ev_.push_back(e);
  }
  return kprof_ev_[kprof_used_++];
}

int PolyEngine::read_profile(double* ms, uint32_t* launches) {
  if (!ms || !launches) return FDSP_ERR_INVALID_ARG;
  *ms = 0.0;
  *launches = 0;
  for (size_t i = 0; i + 1 < kprof_used_; i += 2) {
    if (!kprof_ev_[i] || !kprof_ev_[i + 1]) continue;
    FDSP_TRY(cuda_status(cudaEventSynchronize(kprof_ev_[i + 1])));
    float t = 0.f;
    FDSP_TRY(cuda_status(cudaEventElapsedTime(&t, kprof_ev_[i], kprof_ev_[i + 1])));
    *ms += t;
    ++*launches;
  }
  return FDSP_OK;
}

bool PolyEngine::use_tc_for(int eg) const {
  if (precision_ == FDSP_PRECISION_FP32 || force_ == 0) return false;
  return force_ == 1 || groups_[eg].use_tc != 0;
}

int PolyEngine::autotune(uint64_t n, cudaStream_t stream) {
  if (n == 0 || n >= (1ull << 31)) return FDSP_ERR_INVALID_ARG;
  const size_t ng = groups_.size();
  float2* d_in = nullptr;
  std::vector<float2*> outs(chans_.size(), nullptr);
  int st = cuda_status(cudaMalloc(&d_in, n * sizeof(float2)));
  if (st == FDSP_OK) st = cuda_status(cudaMemsetAsync(d_in, 0, n * sizeof(float2), stream));
  for (size_t c = 0; c < chans_.size() && st == FDSP_OK; ++c) {
    const uint64_t cap = (n * chans_[c].up + chans_[c].down - 1) / chans_[c].down + 2;
    st = cuda_status(cudaMalloc(&outs[c], cap * sizeof(float2)));
  }
  prof_ev_.assign(2 * ng, nullptr);
  prof_hit_.assign(ng, 0);
  for (size_t i = 0; i < prof_ev_.size() && st == FDSP_OK; ++i) st = cuda_status(cudaEventCreate(&prof_ev_[i]));
  std::vector<uint64_t> counts(chans_.size());
  // minimum over 3 timed applies (after one untimed) of each group's time
  auto run = [&](int force, std::vector<float>& t) -> int {
    t.assign(ng, 3.4e38f);
    reset();
    force_ = force;
    for (int rep = 0; rep < 4; ++rep) {
      std::fill(prof_hit_.begin(), prof_hit_.end(), 0);
      int s2 = apply(d_in, n, outs.data(), nullptr, counts.data(), stream);
      if (s2 == FDSP_OK) s2 = cuda_status(cudaStreamSynchronize(stream));
      if (s2 != FDSP_OK) return s2;
      if (rep == 0) continue;
      for (size_t g = 0; g < ng; ++g) {
        if (!prof_hit_[g]) continue;
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, prof_ev_[2 * g], prof_ev_[2 * g + 1]) == cudaSuccess) t[g] = std::min(t[g], ms);
      }
    }
    return FDSP_OK;
  };
  std::vector<float> best(ng, 3.4e38f), t;
  std::vector<int> best_qt(ng);
  for (size_t g = 0; g < ng; ++g) best_qt[g] = groups_[g].Qt_default;
  // FP32 tile height: the default, half, double and four times where shared memory allows
  // (large decimations start from small default tiles, where staging the
  // input span and taps dominates: four times the default is tried too)
  const int factor_num[4] = {1, 1, 2, 4}, factor_den[4] = {1, 2, 1, 1};
  for (int ci = 0; ci < 4 && st == FDSP_OK; ++ci) {
    std::vector<char> valid(ng, 0);
    for (size_t g = 0; g < ng; ++g) {
      EngineGroup& eg = groups_[g];
      const int q = (eg.Qt_default * factor_num[ci] / factor_den[ci]) & ~31;
      const int64_t len = (int64_t)q * eg.D + 3LL * eg.D + 64;
      valid[g] = q >= 32 && (int64_t)eg.D * (len / eg.D + 2) * 8 <= 200 * 1024;
      eg.Qt = valid[g] ? q : eg.Qt_default;
    }
    st = run(0, t);
    for (size_t g = 0; g < ng && st == FDSP_OK; ++g)
      if (valid[g] && t[g] < best[g]) {
        best[g] = t[g];
        best_qt[g] = groups_[g].Qt;
      }
  }
  for (size_t g = 0; g < ng; ++g) groups_[g].Qt = best_qt[g];
  force_ = -1;
  for (auto ev : prof_ev_)
    if (ev) cudaEventDestroy(ev);
  prof_ev_.clear();
  cudaStreamSynchronize(stream);
  if (d_in) cudaFree(d_in);
  for (auto p : outs)
    if (p) cudaFree(p);
  reset();
  return st;
}

void PolyEngine::reset() {
  if (d_err_) cudaMemset(d_err_, 0, sizeof(int));
  for (auto& k : classes_) {
    k.phase = 0;
    k.xoffset = 0;
  }
  abs0_ = 0;
  cudaDeviceSynchronize();
  for (auto& h : d_hist_) {
    if (h) cudaMemset(h, 0, (size_t)H_ * sizeof(float2));
  }
  hist_cur_ = 0;
  cudaDeviceSynchronize();
}

// Tile of Qt rows of one group: which input phases it stages, its pitch, and
// its shared-memory layout.  keep_packed: packed taps wherever they fit.
// Returns whether they do.
template <int NB>
static bool layout_group(PolyLaunch<NB>& L, GroupDesc& gd, int Qt, bool keep_packed = false) {
  const int D = gd.D;
  gd.Qt = Qt;
  gd.nph = D;
  for (int i = 0; i < kMaxSegs - 1; ++i) {
    gd.seg_at[i] = INT32_MAX;
    gd.seg_gap[i] = 0;
  }
  int64_t len = (int64_t)Qt * D + gd.delta_span + gd.tmax - 1;
  for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) {
    WorkSet<NB>& W = L.ws[wi];
    const int a0 = (W.delta - gd.delta_min) + (gd.tmax - W.T);  // first tap of row 0 in the tile
    W.q0 = a0 / D;
    W.b0 = a0 - W.q0 * D;
  }
  // Long decimations: the windows of a row lie inside one period of D samples
  // and leave gaps, which are not staged (64 taps of one phase at D = 320 read
  // a fifth of the input) where that saves an eighth or more.
  if (!gd.win && gd.delta_span + gd.tmax <= D) {
    int lo[kMaxSegs], hi[kMaxSegs], ns = 0;
    bool fits = true;
    // union of the windows [b0, b0 + T): work sets in order of start, by
    // repeated selection of the earliest start past the last segment
    for (int at = 0; fits;) {
      int best = INT32_MAX;
      for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi)
        if (L.ws[wi].b0 + L.ws[wi].T > at) best = std::min(best, std::max(at, L.ws[wi].b0));
      if (best == INT32_MAX) break;
      int end = best;
      for (bool grew = true; grew;) {
        grew = false;
        for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi)
          if (L.ws[wi].b0 <= end && L.ws[wi].b0 + L.ws[wi].T > end) {
            end = L.ws[wi].b0 + L.ws[wi].T;
            grew = true;
          }
      }
      if (ns == kMaxSegs) {
        fits = false;
        break;
      }
      lo[ns] = best;
      hi[ns++] = end;
      at = end;
    }
    int nph = 0;
    for (int i = 0; fits && i < ns; ++i) nph += hi[i] - lo[i];
    if (fits && nph > 0 && 8 * nph <= 7 * D) {
      for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) {
        WorkSet<NB>& W = L.ws[wi];
        int base = 0;
        for (int i = 0; i < ns; base += hi[i] - lo[i], ++i)
          if (W.b0 >= lo[i] && W.b0 < hi[i]) {
            W.b0 = base + (W.b0 - lo[i]);
            break;
          }
      }
      // phase b of the row is staged sample b + seg_first + the gaps before it
      gd.seg_first = lo[0];
      for (int i = 1, at = hi[0] - lo[0]; i < ns; at += hi[i] - lo[i], ++i) {
        gd.seg_at[i - 1] = at;
        gd.seg_gap[i - 1] = lo[i] - hi[i - 1];
      }
      gd.nph = nph;
      len = (int64_t)Qt * nph;
    }
  }
  if (gd.nph == D) gd.seg_first = 0;
  gd.len = (int32_t)len;
  gd.step_q = kThreads / gd.nph;
  gd.step_b = kThreads % gd.nph;
  gd.span = (int32_t)(gd.nph == D ? len : (int64_t)Qt * D);
  gd.inv_nph = ((1ull << 32) + (uint64_t)gd.nph - 1) / (uint64_t)gd.nph;  // exact quotients: len * nph < 2^32
  int64_t P = (len + gd.nph - 1) / gd.nph;
  if ((P & 1) == 0) P++;  // odd pitch: the staging scatter spreads over banks
  gd.P = (int32_t)P;
  // shared-memory layout: input tile | taps of each work set | channel constants
  int64_t off = ((int64_t)gd.nph * P + 1) & ~1LL;  // float2 units, 16-byte aligned
  if (gd.lines) off = std::max(off, (int64_t)Qt * (gd.ws_end - gd.ws_begin));  // the tile's outputs take its place
  gd.taps_off = (int32_t)off;
  const int64_t meta_bytes = (int64_t)(gd.ws_end - gd.ws_begin) * NB * 48;
  int64_t packed = 0, compact = 0, tsum = 0;  // taps of all work sets: float4 packed, compact; taps of a channel each
  int long_t = 0, long_nb = 0;                // the longest work set
  for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) {
    const WorkSet<NB>& W = L.ws[wi];
    packed += (int64_t)W.T * W.nb;
    compact += (int64_t)W.T * ((W.nb + 1) >> 1);
    tsum += W.T;
    if ((int64_t)W.T * W.nb > (int64_t)long_t * long_nb) {
      long_t = W.T;
      long_nb = W.nb;
    }
  }
  auto bytes = [&](int64_t taps) { return (off + 2 * taps) * (int64_t)sizeof(float2) + meta_bytes; };
  auto ctas = [&](int64_t b) { return b <= kSmem3 ? 3 : b <= kSmem2 ? 2 : b <= kSmemTaps ? 1 : 0; };
  // Packed taps take fewer instructions; compact ones where the SM then holds
  // more CTAs or only one packed one, and for wide batches of short runs, whose
  // reads bound the kernel (64 taps of 16 channels by 3 over 2^20 samples: 137
  // us packed, 122 compact; by 10: 43 and 53).
  gd.taps = ctas(bytes(packed)) > 0 ? kTapsPacked : kTapsGlobal;
  const bool packed_fits = gd.taps == kTapsPacked;
  if (!gd.win && ctas(bytes(compact)) > 0 && !(keep_packed && packed_fits) &&
      (ctas(bytes(packed)) <= 1 || ctas(bytes(compact)) > ctas(bytes(packed)) ||
       (NB >= 4 && gd.nph > 1 && gd.nph <= kShortRun)))
    gd.taps = kTapsCompact;
  int64_t toff = 0;
  for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) {
    L.ws[wi].soff = (int32_t)toff;
    toff += (int64_t)L.ws[wi].T * (gd.taps == kTapsPacked ? L.ws[wi].nb : (L.ws[wi].nb + 1) >> 1);
  }
  if (gd.taps != kTapsGlobal) off += 2 * toff;
  gd.meta_off = (int32_t)off;
  gd.smem_bytes = (int32_t)(off * (int64_t)sizeof(float2) + meta_bytes);
  // Rows a thread.  A warp's item takes the instructions of a tap: a sample
  // read a row, the tap reads, the multiply-adds (packed taps, and four rows
  // that share the copies, two components at a time) and the walk.  A tile
  // takes the SM's issue slots for all of its items, or, where its warps are
  // few, their rounds at one instruction in three cycles a warp (9000 taps of
  // two channels by 10 over 2^22 samples: 7.2 ms with a row a thread, 4.2 with
  // two; 300 taps by 6 over 2^20: 68 us and 47).
  const int ctas_sm = std::max(1, std::min(ctas(gd.smem_bytes), NB == 8 ? 2 : 3)), warps = kThreads / 32;
  const bool pk = gd.taps == kTapsPacked;
  auto tap = [&](int r, int64_t t, int64_t n, int64_t half) {  // of t taps, n of all channels, half of channel pairs
    return (double)(t * (r + 3) + (pk ? n * (1 + 2 * r) : half + n * (r >= 4 ? 2 * r + 4 : 4 * r)));
  };
  double best_time = 0;
  for (int r = NB <= 2 ? 4 : 2; r >= 1 && !gd.win; r /= 2) {
    if (Qt % (32 * r) != 0) continue;
    const int blocks = Qt / (32 * r), items = blocks * (gd.ws_end - gd.ws_begin);
    const double work = blocks * tap(r, tsum, packed, compact);
    const double round = tap(r, long_t, (int64_t)long_t * long_nb, (int64_t)long_t * ((long_nb + 1) >> 1));
    const double time = std::max(work / 4, (items + warps - 1) / warps * round * 3 / ctas_sm);
    if (best_time == 0 || time < best_time) {
      best_time = time;
      gd.rows = r;
    }
  }
  return packed_fits;
}

template <int NB>
int PolyEngine::launch(const float2* d_in, uint64_t n, float2* const* out, cudaStream_t stream) {
  static thread_local PolyLaunch<NB> L;  // ~20 KB: keep it off the stack
  std::memset(&L, 0, sizeof(L));
  if (num_sms_ == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev);
    if (num_sms_ <= 0) num_sms_ = 1;
  }
  L.block = in16_ ? nullptr : d_in;
  L.block16 = in16_;
  L.hist = d_hist_[hist_cur_];
  L.new_hist = d_hist_[hist_cur_ ^ 1];
  L.N = (int64_t)n;
  L.H = H_;
  L.nco = d_nco_;
  for (size_t c = 0; c < chans_.size(); ++c) {
    L.out[c] = out[c];
    const uint32_t R = chans_[c].nco.rollover;
    L.nco_base[c] = R ? (uint32_t)(abs0_ % R) : 0u;
  }
  int ng = 0, nws = 0;
  int64_t work = 0;  // complex multiply-adds
  int64_t rows_of[kMaxGroups];
  int qt_of[kMaxGroups];
  bool fixed_qt[kMaxGroups];
  const float4* compact_of[kMaxWorkSets];  // the work sets' compact taps
  for (auto& g : groups_) {
    GroupDesc& gd = L.groups[ng];
    gd.D = (int32_t)g.D;
    gd.ws_begin = nws;
    int dmin = INT32_MAX, dmax = INT32_MIN, tmax = 1;
    int64_t rows = 0;
    for (int bi : g.batches) {
      const EngineBatch& bt = batches_[bi];
      const EngineClass& k = classes_[bt.cls];
      const uint32_t U = k.up;
      for (uint32_t r = 0; r < U; ++r) {
        if (k.M <= r) continue;
        const uint64_t J = (k.M - r + U - 1) / U;
        const uint64_t t = (uint64_t)k.phase + (uint64_t)r * g.D;
        const uint64_t delta = k.xoffset + t / U;
        const uint32_t phi = (uint32_t)(t % U);
        if (nws >= kMaxWorkSets) return FDSP_ERR_UNSUPPORTED;
        WorkSet<NB>& W = L.ws[nws++];
        W.taps = bt.d_taps + (size_t)phi * bt.T * bt.chans.size();
        compact_of[nws - 1] = bt.d_taps + (size_t)U * bt.T * bt.chans.size() + (size_t)phi * bt.T * ((bt.chans.size() + 1) / 2);
        W.T = bt.T;
        W.delta = (int32_t)delta;
        W.J = (int32_t)J;
        W.U = (int32_t)U;
        W.r = (int32_t)r;
        W.nb = (int32_t)bt.chans.size();
        for (size_t i = 0; i < bt.chans.size(); ++i) W.ch[i] = (int16_t)bt.chans[i];
        dmin = std::min(dmin, (int)delta);
        dmax = std::max(dmax, (int)delta);
        tmax = std::max(tmax, bt.T);
        rows = std::max<int64_t>(rows, (int64_t)J);
        work += (int64_t)bt.T * W.nb * (int64_t)J;
      }
    }
    gd.ws_end = nws;
    if (gd.ws_end == gd.ws_begin) continue;
    gd.tmax = tmax;
    gd.delta_min = dmin;
    gd.delta_span = dmax - dmin;
    // the sliding-window form where it fills the GPU with its larger tiles
    // (short blocks keep the per-row form, whose smaller tiles spread wider)
    const bool win = g.win && rows >= (int64_t)g.Qt_win * num_sms_;
    gd.win = win ? 1 : 0;
    gd.real_taps = g.real_taps;
    // one unshifted channel whose every phase has outputs, a block of rows a
    // thread, the outputs within the tile's budget
    const int nsets = nws - gd.ws_begin, unit = 32 * kWinRows;
    const int qt_lines = std::min(g.Qt_win, std::max(1, kThreads / nsets) * kWinRows / unit * unit);
    gd.lines = win && g.batches.size() == 1 && !chans_[batches_[g.batches[0]].chans[0]].nco.enabled &&
               nsets == (int)classes_[batches_[g.batches[0]].cls].up && qt_lines >= unit &&
               (int64_t)nsets * qt_lines * 8 <= 64 * 1024;
    gd.outs = gd.lines ? (int64_t)classes_[batches_[g.batches[0]].cls].M : 0;
    rows_of[ng] = rows;
    qt_of[ng] = gd.lines ? qt_lines : win ? g.Qt_win : g.Qt;
    if (!win && g.Qt == g.Qt_default && g.Qt == 32) {  // two rows a thread where the windows' phases alone fit
      layout_group<NB>(L, gd, 64);
      if (gd.smem_bytes <= kSmem3) qt_of[ng] = 64;
    }
    fixed_qt[ng] = win || g.Qt != g.Qt_default;
    ng++;
  }
  // Blocks too short to give every SM three tiles of the default height take
  // lower tiles (latency: more of the GPU stages and computes at once), but not
  // so low that a tile stages more halo than rows (4095 taps by 10 over 2^20
  // samples: 0.93 ms with 32 rows, 0.34 with 384).
  for (int shift = 1; shift <= 5; ++shift) {
    int64_t tiles = 0;
    for (int gi = 0; gi < ng; ++gi) tiles += (rows_of[gi] + qt_of[gi] - 1) / qt_of[gi];
    if (tiles >= 3LL * num_sms_) break;
    for (int gi = 0; gi < ng; ++gi)
      if (!fixed_qt[gi] &&
          (int64_t)(qt_of[gi] / 2) * L.groups[gi].D >= (int64_t)L.groups[gi].tmax + L.groups[gi].delta_span)
        qt_of[gi] = std::max(32, (qt_of[gi] / 2) & ~31);
  }
  // Chooses the tile of a group; false: it fits at no height.
  bool packed_fits[kMaxGroups];
  auto fit = [&](int gi, bool keep_packed) {
    GroupDesc& gd = L.groups[gi];
    const int qt0 = qt_of[gi], nsets = gd.ws_end - gd.ws_begin;
    packed_fits[gi] = layout_group<NB>(L, gd, qt0, keep_packed);
    // A lower tile where this one's samples leave no room for two more CTAs on
    // the SM, or one more, and a lower one does: not below one that stages as
    // much halo as rows or leaves a warp without rows (9700 taps of two
    // channels over 2^20 samples: 211 ms with 32 rows, 8.3 with 4096)
    if (!fixed_qt[gi] && 16 * (int64_t)gd.taps_off > gd.smem_bytes) {
      const int64_t halo = (int64_t)gd.tmax + gd.delta_span;
      const int base = std::max(32, (4096 / gd.D) & ~31);
      // (registers allow two CTAs of 8-channel batches, three of others)
      for (int room : {NB == 8 ? kSmem2 : kSmem3, kSmem2}) {
        for (int q = qt0 - 32; gd.smem_bytes > room; q -= 32) {
          if (q < 32 || (q < base && ((int64_t)q * gd.D < halo || nsets * q < kThreads))) {
            layout_group<NB>(L, gd, qt0, keep_packed);
            break;
          }
          layout_group<NB>(L, gd, q, keep_packed);
        }
        if (gd.smem_bytes <= room) break;
      }
    }
    while (gd.smem_bytes > 227 * 1024) {
      if (gd.win || gd.Qt <= 32) return false;
      layout_group<NB>(L, gd, gd.Qt - 32, keep_packed);
    }
    gd.ntiles = (int32_t)((rows_of[gi] + gd.Qt - 1) / gd.Qt);
    return true;
  };
  // Groups that would gain by compact taps leave the launch of the others only
  // for work that pays for one more (about 10 us with its tail: 64 channels
  // over 300 k samples took 68 us in three launches, 60 in one).
  const bool one_launch = ng > 1 && work < kSplitWork;
  int64_t gain = 0;
  bool others = false;
  for (int gi = 0; gi < ng; ++gi) {
    if (!fit(gi, one_launch)) return FDSP_ERR_UNSUPPORTED;
    const GroupDesc& gd = L.groups[gi];
    if (one_launch || gd.win || use_tc_for(group_of_d_[gd.D])) continue;
    if (gd.taps == kTapsPacked) others = true;
    if (gd.taps == kTapsCompact && packed_fits[gi])
      for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) gain += (int64_t)L.ws[wi].T * L.ws[wi].nb * L.ws[wi].J;
  }
  if (!one_launch && others && gain > 0 && gain < kSplitWork)
    for (int gi = 0; gi < ng; ++gi)
      if (L.groups[gi].taps == kTapsCompact && packed_fits[gi] && !fit(gi, true)) return FDSP_ERR_UNSUPPORTED;
  for (int gi = 0; gi < ng; ++gi)
    if (!L.groups[gi].win && L.groups[gi].taps != kTapsPacked)
      for (int wi = L.groups[gi].ws_begin; wi < L.groups[gi].ws_end; ++wi) L.ws[wi].taps = compact_of[wi];
  // tensor-core groups: one prep launch and one filter-bank launch for all of
  // them; groups the tensor-core plan cannot hold stay on the FP32 kernel
  std::vector<char> on_tc(ng, 0);
  {
    std::vector<int> tcg, fallback;
    for (int gi = 0; gi < ng; ++gi) {
      const int eg = group_of_d_[L.groups[gi].D];
      if (L.groups[gi].ntiles > 0 && use_tc_for(eg)) tcg.push_back(eg);
    }
    if (!tcg.empty()) {
      FDSP_TRY(launch_tc(d_in, n, out, tcg, fallback, stream));
      for (int gi = 0; gi < ng; ++gi) {
        const int eg = group_of_d_[L.groups[gi].D];
        on_tc[gi] = std::find(tcg.begin(), tcg.end(), eg) != tcg.end() &&
                    std::find(fallback.begin(), fallback.end(), eg) == fallback.end();
      }
    }
  }
  if (d_nat_ && ng == 1 && !on_tc[0] && prof_ev_.empty())
    return launch_nat(d_in, n, out[0], L.groups[0].win == 0, stream);
  // The FP32 groups in one launch per kernel variant (how the taps lie,
  // sliding window or rows) and shared-memory size (three CTAs an
  // SM or fewer), tallest work first; the last launch also writes the history.
  // Group by group only for the autotuner, and for blocks of several waves
  // whose outputs are copied back as groups finish (apply_host).
  struct Batch {
    const void* kern;
    int first, count, tiles;
    size_t smem;
  };
  Batch lb[kMaxGroups];
  int nlb = 0, nm = 0;
  {
    int order[kMaxGroups], nfp = 0;
    int64_t cost[kMaxGroups], tiles = 0;
    for (int gi = 0; gi < ng; ++gi) {
      const GroupDesc& gd = L.groups[gi];
      if (on_tc[gi] || gd.ntiles <= 0) continue;
      cost[gi] = 0;
      for (int wi = gd.ws_begin; wi < gd.ws_end; ++wi) cost[gi] += (int64_t)L.ws[wi].T * L.ws[wi].nb * gd.Qt;
      tiles += gd.ntiles;
      order[nfp++] = gi;
    }
    std::sort(order, order + nfp, [&](int a, int b) { return cost[a] != cost[b] ? cost[a] > cost[b] : a < b; });
    const bool single = !prof_ev_.empty() || (done_fn_ && tiles > 3LL * num_sms_);
    constexpr int kKinds = 7;
    const void* const kernels[kKinds] = {reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsPacked, kRowForm>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsCompact, kRowForm>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsGlobal, kRowForm>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsPacked, kWinTwo>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsGlobal, kWinTwo>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsPacked, kWinReal>),
                                    reinterpret_cast<const void*>(poly_fp32_kernel<NB, kTapsGlobal, kWinReal>)};
    // (kind of kernel, and CTAs that fit an SM: three or more, two, one)
    int variant_of[kMaxGroups];
    uint32_t variants = 0;
    for (int i = 0; i < nfp; ++i) {
      const GroupDesc& gd = L.groups[order[i]];
      int kind = gd.taps == kTapsPacked ? 0 : gd.taps == kTapsCompact ? 1 : 2;
      if (gd.win) kind = (gd.taps == kTapsPacked ? 3 : 4) + (gd.real_taps && (gd.smem_bytes <= kSmem3 || gd.D <= kShortRun) ? 2 : 0);
      variant_of[i] = kind + kKinds * ((gd.smem_bytes > kSmem3) + (gd.smem_bytes > kSmem2));
      variants |= 1u << variant_of[i];
    }
    for (; variants != 0u; variants &= variants - 1u) {
      const int variant = __builtin_ctz(variants);
      bool open = false;
      for (int i = 0; i < nfp; ++i) {
        if (variant_of[i] != variant) continue;
        const GroupDesc& gd = L.groups[order[i]];
        if (!open || single) {
          Batch& nb = lb[nlb++];
          nb.kern = kernels[variant % kKinds];
          nb.first = nm;
          nb.count = nb.tiles = 0;
          nb.smem = 0;
          open = true;
        }
        Batch& cb = lb[nlb - 1];
        L.fuse_map[nm++] = (int8_t)order[i];
        cb.count++;
        cb.tiles += gd.ntiles;
        cb.smem = std::max(cb.smem, (size_t)gd.smem_bytes);
      }
    }
  }
  bool hist_done = false;
  for (int li = 0; li < nlb; ++li) {
    const Batch& bt = lb[li];
    const int eg = group_of_d_[L.groups[L.fuse_map[bt.first]].D];
    cudaError_t e = cudaFuncSetAttribute(bt.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bt.smem);
    if (e != cudaSuccess) return cuda_status(e);
    if (!prof_ev_.empty()) {
      cudaEventRecord(prof_ev_[2 * eg], stream);
      prof_hit_[eg] = 1;
    }
    if (kprof_) cudaEventRecord(kprof_event(), stream);
    int first = bt.first, tiles = bt.tiles, hist_blocks = 0;
    if (li + 1 == nlb && H_ > 0) {
      hist_blocks = (H_ + kThreads - 1) / kThreads;
      hist_done = true;
    }
    e = klaunch_overlapped(bt.kern, dim3((unsigned)(tiles + hist_blocks)), dim3(kThreads), bt.smem, stream, L, first, tiles);
    if (kprof_) cudaEventRecord(kprof_event(), stream);
    if (e != cudaSuccess) return cuda_status(e);
    launches_last_++;
    if (!prof_ev_.empty()) cudaEventRecord(prof_ev_[2 * eg + 1], stream);
    if (done_fn_) {
      std::vector<int> egs;
      for (int i = 0; i < bt.count; ++i) egs.push_back(group_of_d_[L.groups[L.fuse_map[bt.first + i]].D]);
      notify_done(egs, stream);
    }
  }
  if (hist_done) {
    hist_cur_ ^= 1;
    return FDSP_OK;
  }
  if (H_ > 0) {
    const float2* a0 = d_hist_[hist_cur_];
    const float2* a1 = in16_ ? nullptr : d_in;
    const short2* a2 = in16_;
    int64_t a3 = (int64_t)n;
    int a4 = H_;
    float2* a5 = d_hist_[hist_cur_ ^ 1];
    cudaError_t e = klaunch(reinterpret_cast<const void*>(hist_update_kernel), dim3((unsigned)((H_ + 255) / 256)),
                            dim3(256), 0, stream, a0, a1, a2, a3, a4, a5);
    if (e != cudaSuccess) return cuda_status(e);
    hist_cur_ ^= 1;
    launches_last_++;
  }
  return FDSP_OK;
}

// The many-phase form of the engine's only channel.
int PolyEngine::launch_nat(const float2* d_in, uint64_t n, float2* out, bool check, cudaStream_t stream) {
  const EngineClass& k = classes_[0];
  NatLaunch L;
  std::memset(&L, 0, sizeof(L));
  L.block = in16_ ? nullptr : d_in;
  L.block16 = in16_;
  L.hist = d_hist_[hist_cur_];
  L.new_hist = d_hist_[hist_cur_ ^ 1];
  L.taps = d_nat_;
  L.r_first = nat_col_[k.phase];
  L.out = out;
  L.N = (int64_t)n;
  L.M = (int64_t)k.M;
  L.xoffset = (int64_t)k.xoffset;
  L.phase = k.phase;
  L.U = (int32_t)k.up;
  L.D = (int32_t)k.down;
  L.T = batches_[0].T;
  L.H = H_;
  // Columns: whole periods of U, about a thread each of a CTA; a period more
  // where that leaves fewer than six warps (U of 129 to 191 or 65 to 95: 131/100
  // of 2^22 samples 58 us with 131 columns, 52 with 262; 150/7 662 and 629;
  // more columns than these gain nothing).  Full tiles where they give every SM
  // two, one output a thread otherwise.
  L.cols = (int32_t)(k.up * std::max(1u, (uint32_t)kThreads / k.up));
  if (L.cols < 192 && L.cols + (int32_t)k.up <= kNatMaxCols) L.cols += (int32_t)k.up;
  L.per = L.M >= 2LL * num_sms_ * kNatPer * L.cols ? kNatPer : 1;
  const int64_t outs = (int64_t)L.per * L.cols;
  const int threads = (L.cols + 31) & ~31;
  L.len = (int32_t)((((outs - 1) * L.D + L.U - 1) / L.U + L.T + 1) & ~1LL);
  const size_t smem = (size_t)L.len * sizeof(float2) + (((size_t)L.U * L.T + 3) & ~(size_t)3) * sizeof(float);
  int tiles = (int)((L.M + outs - 1) / outs);
  const int hist_blocks = (H_ + threads - 1) / threads;
  const void* kern = check ? reinterpret_cast<const void*>(nat_resample_kernel<true>)
                           : reinterpret_cast<const void*>(nat_resample_kernel<false>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_status(e);
  if (kprof_) cudaEventRecord(kprof_event(), stream);
  e = klaunch_overlapped(kern, dim3((unsigned)(tiles + hist_blocks)), dim3((unsigned)threads), smem, stream, L, tiles);
  if (kprof_) cudaEventRecord(kprof_event(), stream);
  if (e != cudaSuccess) return cuda_status(e);
  launches_last_++;
  if (H_ > 0) hist_cur_ ^= 1;
  if (done_fn_) notify_done(std::vector<int>(1, 0), stream);
  return FDSP_OK;
}

int PolyEngine::apply_ci16(const int16_t* d_in, uint64_t n, float2* const* out, const uint64_t* cap,
                           uint64_t* n_out, cudaStream_t stream) {
  in16_ = reinterpret_cast<const short2*>(d_in);
  // the float pointer is only checked for NULL; every kernel reads in16_
  const int st = apply(reinterpret_cast<const float2*>(d_in), n, out, cap, n_out, stream);
  in16_ = nullptr;
  return st;
}

int PolyEngine::apply(const float2* d_in, uint64_t n, float2* const* out, const uint64_t* cap, uint64_t* n_out,
                      cudaStream_t stream) {
  launches_last_ = 0;
  tc_groups_last_ = 0;
  if (n > 0 && d_in == nullptr) return FDSP_ERR_INVALID_ARG;
  if (n >= (1ull << 31)) return FDSP_ERR_UNSUPPORTED;
  for (auto& k : classes_) k.M = class_out_count(k, n);
  for (size_t c = 0; c < chans_.size(); ++c) {
    const uint64_t M = classes_[cls_of_[c]].M;
    if (n_out) n_out[c] = M;
    if (M > 0 && (out == nullptr || out[c] == nullptr)) return FDSP_ERR_INVALID_ARG;
    if (cap && cap[c] < M) return FDSP_ERR_CAPACITY;
  }
  if (n == 0) return FDSP_OK;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  const bool graph = use_graph_ && !kprof_ && !done_fn_ && stream != nullptr &&
                     cudaStreamIsCapturing(stream, &capturing) == cudaSuccess &&
                     capturing == cudaStreamCaptureStatusNone;
  auto run = [&]() {
    switch (nb_) {
      case 1: return launch<1>(d_in, n, out, stream);
      case 2: return launch<2>(d_in, n, out, stream);
      case 4: return launch<4>(d_in, n, out, stream);
      default: return launch<8>(d_in, n, out, stream);
    }
  };
  int st = FDSP_OK;
  bool done = false;
  if (graph && graph_exec_ && !knodes_.empty()) {
    // replay: the same launch sequence with this apply's arguments written
    // into the recorded kernel nodes (no capture)
    const int hist_save = hist_cur_;
    kmode_ = 2;
    kcur_ = 0;
    kshape_ok_ = true;
    st = run();
    kmode_ = 0;
    if (st != FDSP_OK) return st;
    if (kshape_ok_ && kcur_ == knodes_.size()) {
      const cudaError_t e = cudaGraphLaunch(graph_exec_, stream);
      if (e != cudaSuccess) return cuda_status(e);
      graph_replays_++;
      done = true;
    } else {  // another launch sequence: capture it afresh
      hist_cur_ = hist_save;
      launches_last_ = 0;
      tc_groups_last_ = 0;
    }
  }
  if (!done && graph) {
    cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) return cuda_status(e);
    kmode_ = 1;
    knodes_.clear();
    kfuncs_.clear();
    kshape_ok_ = true;
    st = run();
    kmode_ = 0;
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(stream, &g);
    if (st == FDSP_OK && e != cudaSuccess) st = cuda_status(e);
    if (st == FDSP_OK && kshape_ok_) {
      // a fresh executable graph whose kernel nodes the next applies update
      if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
      graph_exec_ = nullptr;
      if (graph_) cudaGraphDestroy(graph_);
      graph_ = g;
      g = nullptr;
      e = cudaGraphInstantiate(&graph_exec_, graph_, 0);
      if (e != cudaSuccess) {
        graph_exec_ = nullptr;
        knodes_.clear();
        st = cuda_status(e);
      }
    } else if (st == FDSP_OK) {
      // nodes not recorded: update the executable graph from each capture
      knodes_.clear();
      if (graph_exec_) {
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(graph_exec_, g, &info) != cudaSuccess) {
          cudaGetLastError();
          cudaGraphExecDestroy(graph_exec_);
          graph_exec_ = nullptr;
        }
      }
      if (!graph_exec_) {
        e = cudaGraphInstantiate(&graph_exec_, g, 0);
        if (e != cudaSuccess) {
          graph_exec_ = nullptr;
          st = cuda_status(e);
        }
      }
    }
    if (st == FDSP_OK) {
      e = cudaGraphLaunch(graph_exec_, stream);
      if (e != cudaSuccess) st = cuda_status(e);
      else graph_replays_++;
    }
    if (g) cudaGraphDestroy(g);
    done = true;
  }
  if (!done) st = run();
  if (st != FDSP_OK) return st;
  // advance the streaming state (polyphase_resampler.cc:303-312)
  for (auto& k : classes_) polyphase_advance(k.up, k.down, k.phase, k.xoffset, n, k.M);
  abs0_ += n;
  return FDSP_OK;
}

}  // namespace fdsp
