// sieve.cu -- wheel-30 segmented sieve with fused reductions, for sm_103a.
//
// One CTA owns one segment of S bytes (30*S integers) at a time, entirely in
// shared memory, and takes (request, segment) items from a device work queue
// (one global atomic per item; requests come heaviest first).  Per segment:
//   1. fill: AND of four presieve tiles (primes 7..17, 19..31, 37..43,
//      47..59) read at the segment's phase, 16 bytes per load from the tile
//      copy in which that phase is aligned -- replaces the reference's memset + per-prime
//      launches for the smallest primes (context.cu:404-414);
//   2. mark with shared-memory atomicAnd, in work units handed out by a
//      shared counter: primes 61 <= p < split one warp each (lane = residue
//      class x stream, fixed bit mask per stream); split <= p < S/16 four per
//      warp-round (lane = prime x class); from S/16 on a lane per prime, 32
//      primes of one class mod 30 at a time (the wheel tier); primes from the
//      request's bucket split on come from the segment's bucket list, 1024
//      entries per unit, read coalesced from HBM (filled by
//      bucket_fill_kernel).  The reference's sieve_w30_seg_kernel starts each
//      stream at p^2 (sieve.cu:10-37, start offsets context.cu:354-388); here
//      they start at the segment, and a low segment's own sieving primes are
//      set again;
//   3. reduce in the same CTA: popcount (count), masked popcount (p mod 4,
//      p mod 3), and an ordered gap scan with a warp max-scan carrying the
//      previous prime, byte values and gaps counted in shared memory -- replaces extract +
//      thrust::sort + mod4 + gaps kernels (extract.cu:10-39,
//      chebyshev.cu:11-25, gaps.cu:31-75).  Count-only requests skip the
//      gap scan.
// Segment boundaries, 2/3/5 and request totals are stitched by
// finalize_kernel (the reference does this on the host, context.cu:462-524);
// combine_kernel rebuilds requests that shared atoms of a batch.  A lone request
// without lists runs in one launch: solo_kernel with at most a wave of segments,
// lone_kernel or lone_count_kernel with more.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "attr_cache.h"
#include "sieve.cuh"

namespace vg {

__device__ __forceinline__ uint32_t w30(uint32_t o) {
  return (uint32_t)((kW30Packed >> (o << 3)) & 0xFFu);
}

__constant__ ConstPrimeTable cTab = make_const_prime_table();
__constant__ WheelClasses cWheel = make_wheel_classes();

// x mod p by Barrett reduction with m = floor((2^64-1)/p).
__device__ __forceinline__ uint32_t mod_barrett(uint64_t x, uint32_t p, uint64_t m) {
  uint64_t q = __umul64hi(x, m);
  uint64_t r = x - q * (uint64_t)p;
  return (uint32_t)(r >= p ? r - p : r);
}

// First hit (segment-local byte) of class o of prime p, moved up so that the
// number it stands for is >= p*p.  Returns >= nbytes if there is none.
__device__ __forceinline__ uint32_t lift_to_square(uint32_t s, uint64_t k0, uint32_t p,
                                                   uint32_t o, uint32_t nbytes) {
  const uint64_t n = 30ull * (k0 + s) + w30(o);
  const uint64_t p2 = (uint64_t)p * p;
  if (n >= p2) return s;
  const uint64_t step = 30ull * p;
  const uint64_t add = ((p2 - n + step - 1) / step) * p;
  const uint64_t s2 = s + add;
  return s2 < nbytes ? (uint32_t)s2 : nbytes;
}

// A value that is the same in every lane, as a warp-uniform register: the
// compiler then branches on it without divergence bookkeeping (a quarter of the
// marking's instructions went there when units and bounds were read by shuffle
// or from shared memory).
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __reduce_max_sync(0xFFFFFFFFu, x); }

// Clear the candidate at shared address j (the segment's start plus its byte;
// the start is a multiple of four), given keep = ~(1 << class): the mask is keep
// with its low byte moved to byte j & 3 of the word, which a byte permute in
// backward-extract mode does from j itself (it reads two selector bits).
__device__ __forceinline__ void clear_at(uint32_t j, uint32_t keep) {
  asm volatile(
      "{\n\t.reg .b32 m, a;\n\t"
      "prmt.b32.b4e m, %1, %1, %0;\n\t"
      "and.b32 a, %0, -4;\n\t"
      "red.shared.and.b32 [a], m;\n\t}"
      :: "r"(j), "r"(keep) : "memory");
}

// The same where j < end, as one predicated instruction: a branch around it
// costs more issue slots than the address and mask that idle lanes compute.
__device__ __forceinline__ void clear_below(uint32_t j, uint32_t keep, uint32_t end) {
  asm volatile(
      "{\n\t.reg .b32 m, a;\n\t.reg .pred p;\n\t"
      "setp.lt.u32 p, %0, %2;\n\t"
      "prmt.b32.b4e m, %1, %1, %0;\n\t"
      "and.b32 a, %0, -4;\n\t"
      "@p red.shared.and.b32 [a], m;\n\t}"
      :: "r"(j), "r"(keep), "r"(end) : "memory");
}

// A word at shared address a with a mask at hand, always or where on.
__device__ __forceinline__ void and_word(uint32_t a, uint32_t mask) {
  asm volatile("red.shared.and.b32 [%0], %1;" :: "r"(a), "r"(mask) : "memory");
}
__device__ __forceinline__ void and_word_if(uint32_t a, uint32_t mask, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.shared.and.b32 [%0], %1;\n\t}"
               :: "r"(a), "r"(mask), "r"((uint32_t)on) : "memory");
}

// A candidate given as bit index v = 8 * byte + class of the segment at shared
// address seg, where it lies below send: its word is v / 32 and its mask
// 0xFFFFFFFE rotated by v (a funnel shift takes its count mod 32).  The test is
// made on the word's address, so up to 31 bits past the segment's end may be
// cleared: send is the address past the last word, whose spare bits are masked
// when it is scanned.
__device__ __forceinline__ void clear_bit_below(uint32_t seg, uint32_t v, uint32_t send) {
  const uint32_t a = seg + 4u * (v >> 5), m = __funnelshift_l(0xFFFFFFFEu, 0xFFFFFFFEu, v);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %0, %2;\n\t@p red.shared.and.b32 [%0], %1;\n\t}"
               :: "r"(a), "r"(m), "r"(send) : "memory");
}

// The eight class residues of table prime i (32 bytes, two vector loads).
__device__ __forceinline__ void load_residues(const uint32_t* __restrict__ R, uint32_t i, uint32_t r[8]) {
  const uint4 lo = __ldg(reinterpret_cast<const uint4*>(R) + 2u * i);
  const uint4 hi = __ldg(reinterpret_cast<const uint4*>(R) + 2u * i + 1u);
  r[0] = lo.x; r[1] = lo.y; r[2] = lo.z; r[3] = lo.w;
  r[4] = hi.x; r[5] = hi.y; r[6] = hi.z; r[7] = hi.w;
}

struct GapSink {
  uint32_t* shist;           // this warp's shared histogram copy
  ReqAccum* acc;             // this request's global accumulators
  LargeGapRec* large;
  unsigned int* n_large;
  uint32_t cap;
  uint32_t req;
  uint64_t base;             // 30 * k0: absolute value of relative 0
};

// Count the gap v - vprev.  Shared bins hold gap/2 < kSmemBins; one extra
// shared bin (never flushed) absorbs larger gaps, which take the rare path
// together with a new maximum and gaps >= kLargeGap.  The gap starts before any
// that (maxg, maxgs) stands for (it leads into their run), so it wins a tie.
__device__ __forceinline__ void record_gap(const GapSink& sk, uint32_t vprev, uint32_t v,
                                           uint32_t& maxg, uint32_t& maxgs) {
  const uint32_t g = v - vprev;
  const uint32_t bin = g >> 1;
  atomicAdd(sk.shist + min(bin, (uint32_t)kSmemBins), 1u);
  // rare: a new maximum or g >= 2 * kSmemBins (which covers g >= kLargeGap)
  if (g >= min(maxg, 2u * (uint32_t)kSmemBins)) {
    if (g >= maxg) { maxg = g; maxgs = vprev; }
    if (bin >= (uint32_t)kSmemBins)
      atomicAdd(&sk.acc->hist[bin < (uint32_t)kHistBins ? bin : kHistBins - 1], 1ull);
    if (g >= kLargeGap) {
      const unsigned idx = atomicAdd(sk.n_large, 1u);
      if (idx < sk.cap) {
        LargeGapRec r; r.pos = sk.base + v; r.gap = g; r.req = sk.req;
        sk.large[idx] = r;
      }
    }
  }
}

static_assert(2u * (uint32_t)kSmemBins <= kLargeGap, "gaps from kLargeGap on must leave the shared bins");

// Value of bit b of a word, relative to the word's first integer.
__device__ __forceinline__ uint32_t word_value(uint32_t b) { return 30u * (b >> 3) + w30(b & 7u); }

// A thread's run of words, prime by prime: its largest gap (the earliest on
// ties), and the gaps beyond the shared bins.
__device__ __noinline__ uint2 walk_run(GapSink sk, const uint32_t* seg, uint32_t wbeg, uint32_t wend) {
  uint32_t best = 0, at = 0, pv = 0;
  bool any = false;
  for (uint32_t wi = wbeg; wi < wend; ++wi) {
    for (uint32_t w = seg[wi]; w; w &= w - 1u) {
      const uint32_t v = 120u * wi + word_value(__ffs(w) - 1u);
      const uint32_t g = v - pv;
      if (any && g > best) { best = g; at = pv; }
      if (any && g >= 2u * (uint32_t)kSmemBins) {
        const uint32_t bin = g >> 1;
        atomicAdd(&sk.acc->hist[bin < (uint32_t)kHistBins ? bin : kHistBins - 1], 1ull);
        if (g >= kLargeGap) {
          const unsigned idx = atomicAdd(sk.n_large, 1u);
          if (idx < sk.cap) {
            LargeGapRec r; r.pos = sk.base + v; r.gap = g; r.req = sk.req;
            sk.large[idx] = r;
          }
        }
      }
      pv = v;
      any = true;
    }
  }
  return make_uint2(best, at);
}

// Add one to the 32-bit counter at shared address a.
__device__ __forceinline__ void count_one(uint32_t a) {
  asm volatile("red.shared.add.u32 [%0], 1;" :: "r"(a) : "memory");
}

// A claimed (request, segment) work item with what the CTA needs of it.
// The edge masks fix the segment's first word, w = ((w & and0) | or0) &
// keep0, and its last word, w &= keepl: the tile primes themselves (7..29
// live in wheel byte 0, 31 in byte 1), 1, and the request's ends.
struct SegItem {
  uint64_t item, k0, bbase;
  uint32_t req, nbytes, np, split, wheel, rflags, bcnt, valid, mix;
  uint32_t and0, or0, keep0, keepl;
};

// What follows from a work item's request R: the tiers, the flags and the edge
// masks (keep0 and keepl where the segment is the first or the last).
__device__ __forceinline__ void set_item(SegItem& d, const ReqDesc& R, uint32_t keep0, uint32_t keepl) {
  d.split = R.tier_split; d.wheel = R.tier_wheel; d.rflags = R.rflags;
  d.and0 = d.k0 == 0 ? ~1u : ~0u;                                        // 1 is not prime
  d.or0 = d.k0 < 3 ? (uint32_t)(kTilePrimeBits >> (8u * d.k0)) : 0u;     // the tile primes are
  d.keep0 = keep0;                                                       // numbers below a
  d.keepl = keepl;                                                       // numbers from b on
}

// Number of leading i in [0, n) for which pred(i) holds (pred holds on a
// prefix), by a 32-ary search of one warp: each step probes 32 evenly spaced
// points, so about log32(n) dependent loads instead of log2(n).
template <class Pred>
__device__ __forceinline__ uint32_t warp_count_leading(uint32_t n, uint32_t lane, Pred pred) {
  uint32_t lo = 0, hi = n;                      // the answer is in [lo, hi]
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31u) / 32u;
    const uint32_t idx = lo + lane * step;
    const bool t = idx < hi && pred(idx);
    const uint32_t k = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, t));
    if (k == 0) break;                          // pred(lo) fails: the answer is lo
    const uint32_t last_true = lo + (k - 1u) * step;
    hi = min(hi, lo + k * step);                // first probe that failed (or the end)
    lo = last_true + 1u;
  }
  return lo;
}

// Claim the next work item and look it up, by one whole warp: its request
// (the last with seg_base <= item), its bytes, the table primes with p*p
// below its upper end, and its bucket list.  Lane 0 writes d.
__device__ __noinline__ void claim_item(unsigned long long* queue, const ReqDesc* __restrict__ reqs,
                                        const uint32_t* __restrict__ P, const uint32_t* __restrict__ bcount,
                                        uint64_t item_lo, uint64_t item_end, uint64_t list_seg0,
                                        uint32_t nreq, SegItem& d, uint32_t lane) {
  unsigned long long it = 0;
  if (lane == 0) it = atomicAdd(queue, 1ull);
  const uint64_t item = item_lo + __shfl_sync(0xFFFFFFFFu, it, 0);
  if (item >= item_end) {
    if (lane == 0) { d.item = item; d.valid = 0; }
    return;
  }
  const uint32_t r = warp_count_leading(nreq, lane, [&](uint32_t i) { return reqs[i].seg_base <= item; }) - 1u;
  const ReqDesc& R = reqs[r];
  const uint64_t si = item - R.seg_base;
  const uint64_t k0 = R.k_lo + si * R.seg_bytes;
  const uint64_t left = R.k_hi - k0;
  const uint32_t nb = left < R.seg_bytes ? (uint32_t)left : R.seg_bytes;
  const uint64_t hi_num = 30ull * (k0 + nb);
  // only primes up to the bucket split matter (the rest come from the list)
  const uint32_t lim = R.bucket_idx < R.nprimes ? R.bucket_idx + 1u : R.nprimes;
  uint32_t a = warp_count_leading(lim, lane, [&](uint32_t i) {
    const uint64_t p = P[i];
    return p * p < hi_num;
  });
  if (lane == 0) {
    d.bcnt = 0;
    d.bbase = 0;
    if (R.bucket_idx < a) {
      a = R.bucket_idx;
      d.bcnt = min(bcount[item], R.bucket_cap);
      d.bbase = R.bucket_base + (si - list_seg0) * (uint64_t)R.bucket_cap;
    }
    d.item = item; d.valid = 1;
    d.req = r; d.k0 = k0; d.nbytes = nb; d.np = a;
    d.mix = a && P[a - 1u] >= 2u * nb;
    set_item(d, R, si == 0 ? first_word_mask(R) : ~0u, k0 + nb == R.k_hi ? last_word_mask(R, nb) : ~0u);
  }
}

// The same for a lone request without lists (lone_kernel): the next of its
// segments and the table primes with p*p below the segment's upper end.
__device__ __noinline__ void claim_lone(const SieveParams& prm, SegItem& d, uint32_t lane) {
  const ReqDesc& R = prm.solo;
  unsigned long long it = 0;
  if (lane == 0) it = atomicAdd(&prm.ctl->queue, 1ull);
  const uint64_t si = __shfl_sync(0xFFFFFFFFu, it, 0);
  if (si >= R.nseg) {
    if (lane == 0) d.valid = 0;
    return;
  }
  const uint64_t k0 = R.k_lo + si * R.seg_bytes;
  const uint32_t nb = (uint32_t)min((uint64_t)R.seg_bytes, R.k_hi - k0);
  const uint64_t hi_num = 30ull * (k0 + nb);
  const uint32_t np = warp_count_leading(R.nprimes, lane, [&](uint32_t i) {
    const uint64_t p = prm.P[i];
    return p * p < hi_num;
  });
  if (lane == 0) {
    d.k0 = k0; d.nbytes = nb; d.item = si; d.valid = 1; d.req = 0; d.np = np; d.bcnt = 0; d.bbase = 0;
    d.mix = np && prm.P[np - 1u] >= 2u * nb;
    set_item(d, R, si == 0 ? prm.keep0 : ~0u, si + 1u == R.nseg ? prm.keepl : ~0u);
  }
}

// Shared-memory per-warp record used to stitch warps inside a segment.
struct WarpRec {
  uint32_t first1, last1;    // relative value + 1 (0 = none)
  uint32_t cnt, c41, c31;
  uint32_t maxg, maxgs;
  uint32_t pad;
};

__device__ __forceinline__ SegRec seg_rec(const SegRec* s) {
  const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2*>(s));
  const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2*>(s) + 1);
  SegRec r;
  r.first = a.x; r.last = a.y; r.max_gap_start = b.x;
  r.max_gap = (uint32_t)b.y; r.pad = 0;
  return r;
}
static_assert(sizeof(SegRec) == 32 && alignof(SegRec) == 16, "read as two 16-byte halves");

// Shared memory of finalize_request: 32-bit words.
constexpr uint32_t kFinalWords = kHistBins + 1u + 8u * 32u;

// The whole CTA finishes request r: seeds 2, 3, 5, gaps across segment
// boundaries, the largest gap, and the final counts (the reference's host-side
// conventions, context.cu:321-322,462-524, restated for a half-open [a, b)).
// Records and accumulators are read past L1: other CTAs of the same launch may
// have written them.  kClean: the accumulators are left at zero.
template <bool kClean>
__device__ __forceinline__ void finalize_request(const ReqDesc& R, uint32_t r, const SegRec* S, ReqAccum* A,
                                                 LargeGapRec* large, unsigned int* n_large, uint32_t large_cap,
                                                 ReqResult* O, uint32_t* tmp) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t* const joins = tmp;                       // gaps between segments and seeds, per bin
  uint64_t* const part = reinterpret_cast<uint64_t*>(tmp + kHistBins + 1);     // per warp: four values
  const bool in2 = R.a <= 2 && 2 < R.b, in3 = R.a <= 3 && 3 < R.b, in5 = R.a <= 5 && 5 < R.b;
  const uint64_t seed_first = in2 ? 2 : in3 ? 3 : in5 ? 5 : 0;
  const uint64_t seed_last = in5 ? 5 : in3 ? 3 : in2 ? 2 : 0;
  const bool gaps = (R.rflags & kReqGaps) != 0;
  // the accumulators of other CTAs, loaded while the records are folded
  uint64_t wc = 0, a41 = 0, a31 = 0;
  if (tid == 0) { wc = __ldcg(&A->count); a41 = __ldcg(&A->c41); a31 = __ldcg(&A->c31); }
  const uint64_t h0 = tid < (uint32_t)kHistBins ? __ldcg(&A->hist[tid]) : 0;
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += blockDim.x) joins[b] = 0;
  __syncthreads();

  uint64_t bg = 0, bs = 0, first = ~0ull, last = 0;
  auto consider = [&](uint64_t g, uint64_t st) {
    if (g > bg || (g == bg && g && st < bs)) { bg = g; bs = st; }
  };
  if (tid == 0 && gaps) {
    if (in2 && in3) { atomicAdd(&joins[0], 1u); consider(1, 2); }
    if (in3 && in5) { atomicAdd(&joins[1], 1u); consider(2, 3); }
  }
  for (uint64_t i = tid; i < R.nseg; i += blockDim.x) {
    const SegRec s = seg_rec(S + i);
    if (!s.first) continue;
    first = s.first < first ? s.first : first;
    last = s.last > last ? s.last : last;
    if (!gaps) continue;
    if (s.max_gap) consider(s.max_gap, s.max_gap_start);
    uint64_t prev = 0;
    for (uint64_t j = i; j-- > 0;) {
      if (__ldcg(&S[j].first)) { prev = __ldcg(&S[j].last); break; }
    }
    if (!prev) prev = seed_last;
    if (!prev) continue;
    const uint64_t g = s.first - prev;
    const uint64_t bin = g >> 1;
    atomicAdd(&joins[bin < (uint64_t)kHistBins ? bin : kHistBins - 1], 1u);
    consider(g, prev);
    if (g >= kLargeGap) {
      const unsigned idx = atomicAdd(n_large, 1u);
      if (idx < large_cap) {
        LargeGapRec lr; lr.pos = s.first; lr.gap = (uint32_t)g; lr.req = r;
        large[idx] = lr;
      }
    }
  }
  // the largest gap (the earliest on ties), the first and the last prime
  auto fold = [&](uint64_t g2, uint64_t s2, uint64_t f2, uint64_t l2) {
    consider(g2, s2);
    first = f2 < first ? f2 : first;
    last = l2 > last ? l2 : last;
  };
  const uint32_t warps = (uint32_t)min((uint64_t)(blockDim.x >> 5), (R.nseg + 31u) / 32u);   // those with records
  if (warp < max(warps, 1u)) {
#pragma unroll 1
    for (int d = 16; d > 0; d >>= 1) {
      const uint64_t g2 = __shfl_down_sync(0xFFFFFFFFu, bg, d), s2 = __shfl_down_sync(0xFFFFFFFFu, bs, d);
      const uint64_t f2 = __shfl_down_sync(0xFFFFFFFFu, first, d), l2 = __shfl_down_sync(0xFFFFFFFFu, last, d);
      fold(g2, s2, f2, l2);
    }
    if (lane == 0) { part[4 * warp] = bg; part[4 * warp + 1] = bs; part[4 * warp + 2] = first; part[4 * warp + 3] = last; }
  }
  __syncthreads();
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += blockDim.x) {
    O->hist[b] = (b == tid ? h0 : __ldcg(&A->hist[b])) + joins[b];
    if (kClean) A->hist[b] = 0;
  }
  if (tid == 0) {
    for (uint32_t w = 1; w < warps; ++w) fold(part[4 * w], part[4 * w + 1], part[4 * w + 2], part[4 * w + 3]);
    const uint64_t ns = (uint64_t)in2 + in3 + in5;
    const uint64_t count = wc + ns;
    O->count = count;
    O->c41 = a41 + (in5 ? 1 : 0);
    O->c43 = (wc - a41) + (in3 ? 1 : 0);
    O->c31 = a31;
    O->c32 = (wc - a31) + (in2 ? 1 : 0) + (in5 ? 1 : 0);
    O->first = seed_first ? seed_first : first != ~0ull ? first : 0;
    O->last = last ? last : seed_last;
    O->max_gap = bg;
    O->max_gap_start = bg ? bs : 0;
    O->num_gaps = count ? count - 1 : 0;
    if (kClean) A->count = A->c41 = A->c31 = 0;
  }
}

// The three forms of the sieve: work items of a plan's requests, and a lone
// request in one launch, with at most a wave of segments (solo_kernel) or with
// more (lone_kernel), there with gaps or counts alone.
constexpr int kFormBatch = 0, kFormSolo = 1, kFormLone = 2, kFormLoneCount = 3;

template <int kForm>
__device__ __forceinline__ void sieve_body(const SieveParams& prm) {
  constexpr bool kSolo = kForm == kFormSolo, kLone = kForm == kFormLone || kForm == kFormLoneCount;
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* seg = smem;
  const uint32_t sseg = (uint32_t)__cvta_generic_to_shared(seg);
  uint32_t* shist = seg + (prm.seg_bytes >> 2);
  WarpRec* wrec = reinterpret_cast<WarpRec*>(shist + kSmemHistCopies * kSmemStride);
  uint32_t* bhist = reinterpret_cast<uint32_t*>(wrec + kMaxThreads / 32);    // byte values, kSmemHistCopies copies
  uint8_t* btab = reinterpret_cast<uint8_t*>(bhist + kSmemHistCopies * kByteValues);   // the gap scan's byte table

  // the segment in hand, s_item[cur], and the next one, s_item[cur ^ 1],
  // claimed and looked up by warp 0 while the others mark (so no thread
  // waits on that lookup)
  __shared__ SegItem s_item[2];
  __shared__ uint32_t s_ctr;
  __shared__ uint32_t s_filled;                    // the segment in hand has been filled by the warps

  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t nthr = blockDim.x, nwarps = nthr >> 5;

  for (uint32_t i = tid; i < kSmemHistCopies * kSmemStride; i += nthr) shist[i] = 0;
  for (uint32_t i = tid; i < kSmemHistCopies * kByteValues; i += nthr) bhist[i] = 0;
  for (uint32_t x = tid; x < kByteValues; x += nthr)
    btab[x] = x ? (uint8_t)((__ffs(x) - 1) | ((31 - __clz(x)) << 4)) : 0;
  if (tid == 0) s_ctr = s_filled = 0;
  int cur_req = -1;
  bool cur_gaps = false;
  // Add the histograms to the current request's accumulators and clear them:
  // the byte values give the primes, those 1 mod 3 and the gaps inside bytes
  // (added to the first gap histogram).
  auto flush = [&] {
    ReqAccum* acc = prm.acc + cur_req;
    for (uint32_t x = tid; x < kByteValues; x += nthr) {
      uint32_t n = 0;
#pragma unroll
      for (int c = 0; c < kSmemHistCopies; ++c) { n += bhist[c * kByteValues + x]; bhist[c * kByteValues + x] = 0; }
      // whole warps (kByteValues and the thread count are multiples of 32);
      // sums of 32 products below 2^35 in two parts
      const unsigned long long all = (unsigned long long)n * __popc(x);
      const unsigned long long c1 = (unsigned long long)n * __popc(x & 0x2Bu);
      const uint32_t all0 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)all & 0xFFFFFFu);
      const uint32_t all1 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(all >> 24));
      const uint32_t c10 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)c1 & 0xFFFFFFu);
      const uint32_t c11 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(c1 >> 24));
      if (lane == 0 && (all0 | all1)) {
        atomicAdd(&acc->count, ((unsigned long long)all1 << 24) + all0);
        atomicAdd(&acc->c31, ((unsigned long long)c11 << 24) + c10);
      }
      if (!n) continue;
      for (uint32_t b = x; b & (b - 1u);) {
        const uint32_t lo = __ffs(b) - 1u;
        b &= b - 1u;
        atomicAdd(&shist[(w30(__ffs(b) - 1u) - w30(lo)) >> 1], n);
      }
    }
    __syncthreads();
    for (uint32_t bn = tid; bn < (uint32_t)kSmemBins; bn += nthr) {
      uint32_t s = 0;
#pragma unroll
      for (int c = 0; c < kSmemHistCopies; ++c) { s += shist[c * kSmemStride + bn]; shist[c * kSmemStride + bn] = 0; }
      if (s && bn) atomicAdd(&acc->hist[bn], (unsigned long long)s);     // bin 0: the runs' first primes
    }
  };

  // The presieve tiles' AND in 16-byte units v, v + step, .. below end of the
  // segment at k0 (up to 3 words past its end: never read), and in the solo
  // form into the words that the slices left.
  auto fill = [&](uint64_t k0, uint32_t v, uint32_t end, uint32_t step, const uint32_t* merged) {
    // copy (phase mod 16) of each tile holds the phase on a 16-byte boundary
    uint32_t toff[kTiles];                         // 16-byte units from each tile's start
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      const uint32_t ph = (uint32_t)(k0 % tile_period(t));
      toff[t] = (ph & 15u) * prm.tile_stride16[t] + (ph >> 4);
    }
    uint4* seg4 = reinterpret_cast<uint4*>(seg);
#pragma unroll 4
    for (; v < end; v += step) {
      uint4 x = __ldg(reinterpret_cast<const uint4*>(prm.tile[0]) + toff[0] + v);
#pragma unroll
      for (int t = 1; t < kTiles; ++t) {
        const uint4 y = __ldg(reinterpret_cast<const uint4*>(prm.tile[t]) + toff[t] + v);
        x.x &= y.x; x.y &= y.y; x.z &= y.z; x.w &= y.w;
      }
      if (kSolo && merged) {
        const uint4 y = __ldcg(reinterpret_cast<const uint4*>(merged) + v);
        x.x &= y.x; x.y &= y.y; x.z &= y.z; x.w &= y.w;
      }
      seg4[v] = x;
    }
  };

  uint64_t item_end = 0;
  uint32_t nreq = 1, cur = 0;
  // solo: this CTA's segment and its share of the segment's units
  const uint32_t slices = kSolo ? prm.slices : 1u;
  const uint32_t slice = kSolo ? blockIdx.x % slices : 0u;
  if constexpr (kSolo) {
    if (tid == 0) {
      const ReqDesc& R = prm.solo;
      SegItem& d = s_item[0];
      const uint32_t si = blockIdx.x / slices;
      d.k0 = R.k_lo + (uint64_t)si * R.seg_bytes;
      d.nbytes = (uint32_t)min((uint64_t)R.seg_bytes, R.k_hi - d.k0);
      d.item = si; d.valid = 1; d.req = 0; d.np = R.nprimes; d.bcnt = 0; d.bbase = 0; d.mix = 0;
      set_item(d, R, si == 0 ? prm.keep0 : ~0u, si + 1u == (uint32_t)R.nseg ? prm.keepl : ~0u);
      s_item[1].valid = 0;
    }
  } else if constexpr (kLone) {
    if (warp == 0) claim_lone(prm, s_item[0], lane);
  } else {
    const uint64_t total_segs = prm.hdr->total_segs;
    item_end = prm.item_hi ? min(total_segs, prm.item_hi) : total_segs;
    nreq = prm.hdr->nreq;
    if (warp == 0)
      claim_item(prm.queue, prm.reqs, prm.P, prm.bcount, prm.item_lo, item_end, prm.list_seg0, nreq, s_item[0], lane);
  }
  __syncthreads();
  // Two or three barriers per segment: after a fill by all threads, after the
  // marking, before the warps are stitched.  No thread reads the segment after
  // the last one, so the next fill or marking follows it directly.
  for (;; cur ^= 1u) {
    // work queue: the next (request, segment) item, heaviest requests first
    const SegItem& S = s_item[cur];
    if (!S.valid) break;
    const uint64_t item = S.item;
    const uint32_t req = S.req;
    const uint64_t k0 = S.k0;
    const uint32_t nbytes = S.nbytes;
    const uint32_t nwords = (nbytes + 3u) >> 2;
    const uint32_t np = S.np;

    if ((int)req != cur_req) {
      if (cur_req >= 0 && cur_gaps) {               // flush the previous request's counts
        __syncthreads();                            // after warp 0's last stitching gaps
        flush();
      }
      cur_req = (int)req;
      cur_gaps = kLone ? kForm == kFormLone : (S.rflags & kReqGaps) != 0;
    }

    // 1. presieve fill, of all words (unless the warps have filled them after
    //    scanning the segment before) or, solo, after the slices are merged,
    //    into what the slices left
    if (kSolo && slices > 1u) {
      const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
      for (uint32_t v = tid; v < (nbytes + 15u) >> 4; v += nthr) reinterpret_cast<uint4*>(seg)[v] = ones;
      __syncthreads();
    } else if (kSolo || !s_filled) {
      fill(k0, tid, (nbytes + 15u) >> 4, nthr, nullptr);
      __syncthreads();
    }

    // 2. marking.  Work units handed out by a shared counter:
    //    units [0, nsmall): one prime each, p < split: a warp per prime, lane
    //      = (class o, stream h of 4); a stream steps 4p bytes = p words, so
    //      its bit mask never changes;
    //    then 32 primes each up to the wheel tier: lanes = (prime q of 4, class
    //      o), eight rounds of four primes, loads of all rounds issued before
    //      any marking so their latency overlaps;
    //    then 2^wlog primes of one class mod 30 each (the wheel tier, one per
    //      lane at a time), then kBucketUnit entries of the segment's bucket
    //      list each.
    {
      const uint32_t unp = uniform(np), unb = uniform(nbytes);
      const uint32_t wheel = uniform(S.wheel);
      const uint32_t nsmall = min(uniform(S.split), unp);
      const uint32_t mend = wheel < unp ? max(wheel, nsmall) : unp;
      const uint32_t nmidu = (mend - nsmall + 31u) / 32u;
      // the wheel tier's run of each class (lane = class): positions wbeg ..
      // wend - 1 of the wheel table, and the units of classes 0 .. lane.  The
      // end is rounded up to a row: the primes past np that this adds clear
      // composites only (and themselves, see the restoring below).
      uint32_t wbeg = 0, wend = 0;
      if (lane < 8u && wheel < unp) {
        wbeg = __ldg(prm.Woff + 8u * (wheel / kWheelRow) + lane);
        wend = __ldg(prm.Woff + 8u * ((unp + kWheelRow - 1u) / kWheelRow) + lane);
      }
      // primes per unit, 2^wlog: claiming a unit costs about as much as
      // marking 32 primes, but every warp should get several units
      uint32_t wlog = 5;
      while (wlog < kWheelUnitLog2Max && mend + ((256u * slices) << wlog) <= unp) ++wlog;
      uint32_t wincl = (wend - wbeg + (1u << wlog) - 1u) >> wlog;
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wincl, d);
        if ((int)lane >= d) wincl += t;
      }
      const uint32_t nscan = nsmall + nmidu + uniform(lane == 7u ? wincl : 0u);
      // x mod p for the wheel tier (p > 2^10): q = hi32((x >> 10) * floor(2^42
      // / p)) is x / p or up to 2 less, so 32 bits of remainder suffice
      const uint32_t k0s = uniform((uint32_t)(k0 >> 10)), k0l = uniform((uint32_t)k0);
      const uint32_t bcnt = uniform(S.bcnt);
      const uint64_t bbase = S.bbase;
      if (!kSolo && warp == 0) {                    // overlaps the marking
        if constexpr (kLone)
          claim_lone(prm, s_item[cur ^ 1u], lane);
        else
          claim_item(prm.queue, prm.reqs, prm.P, prm.bcount, prm.item_lo, item_end, prm.list_seg0, nreq,
                     s_item[cur ^ 1u], lane);
      }
      const uint32_t nunits = nscan + (bcnt + kBucketUnit - 1) / kBucketUnit;
      // Where many primes lie above the segment, the units that shared memory
      // bounds (below it) alternate with the wheel tier's, which issue bounds
      // above it: [9*10^11, 9.1*10^11) 1.459 -> 1.417 ms.  Elsewhere the
      // heaviest come first ([0, 10^10): 1.075 ms, alternating 1.088).
      const bool mix = uniform(S.mix) != 0u;
      const uint32_t nlow = nsmall + nmidu, nwheel = nscan - nlow;
      const uint32_t o = lane & 7u, h = lane >> 3;
      const uint32_t send = sseg + unb;             // shared address past the segment's end
      for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(&s_ctr, 1u);
        u = uniform(u);
        if (kSolo) u = u * slices + slice;
        if (u >= nunits) break;
        if (!kSolo && mix && u < nscan) {
          if (u < 2u * min(nlow, nwheel)) u = (u & 1u) ? nlow + (u >> 1) : u >> 1;
          else if (nlow > nwheel) u -= nwheel;
        }
        if (u < nsmall) {
          const bool cst = u < kConstPrimes;
          const uint32_t p = cst ? cTab.p[u] : __ldg(prm.P + u);
          const uint64_t M = cst ? (uint64_t)cTab.m[u] : __ldg(prm.M + u);
          const uint32_t minv = (uint32_t)(M >> 32) + 1u;
          const uint32_t m = mod_barrett(k0, p, M);
          const uint32_t r = __ldg(prm.R + 8u * u + o);
          uint32_t s = r - m;
          s = min(s, s + p);
          // This lane's stream: bytes j0 + 4 p i = words w0 + p i with one
          // mask, n of them in the segment.  All 32 streams step p words, so
          // their banks shift alike: lanes that start on 32 different banks
          // stay on banks of their own while every lane walks on, and each
          // atomic of the warp takes one shared-memory wavefront instead of
          // one per lane sharing a bank.  With u = w0 / p mod 32 the bank after
          // i steps is p (u + i) mod 32, so the lanes, in the order of their u,
          // skip to u + rot = rank + shift, the shift being the least that
          // makes every rot >= 0: 3 steps on average, the longest of a warp
          // about 6 (to a fixed bank per lane: 16 and 31).  A lane walks steps
          // rot .. n-1, then wraps to 0 .. rot-1 (wrapped lanes may meet
          // another lane on a bank, and test for their wrap at each step).
          // [0, 10^10) takes 1.042 ms with the order and 1.074 with fixed
          // banks; with it the tier pays up to 2048 (1.039 ms, up to 1400..1700
          // 1.042; [10^12, 1.01*10^12) 1.390 and 1.408).
          const uint32_t j0 = s + h * p;
          const uint32_t c = j0 & 3u;
          const uint32_t mask = ~(1u << ((c << 3) | o));
          const uint32_t lim = (unb - c + 3u) >> 2;         // word w holds byte 4w + c < nbytes
          const uint32_t w0 = j0 >> 2;
          // steps: w0 < p, so floor(whole words / p) or one more, the floor by a
          // multiplication, exact for factors below 2^16 ([0, 10^10) 1.033 ms;
          // with a division, a remainder and two reductions 1.037)
          const uint32_t nmin = __umulhi(unb >> 2, minv);
          const uint32_t n = nmin + (w0 + nmin * p < lim ? 1u : 0u);
          const uint32_t pinv = p * (2u - p * p);           // p^-1 mod 64 (p odd, p*p = 1 mod 8)
          const uint32_t u32 = (w0 * pinv) & 31u;
          uint32_t less = 0, same = 0xFFFFFFFFu;             // lanes with a smaller u, with this u
#pragma unroll
          for (int t = 4; t >= 0; --t) {
            const bool bit = (u32 >> t) & 1u;
            const uint32_t set = __ballot_sync(0xFFFFFFFFu, bit);
            less |= bit ? same & ~set : 0u;
            same &= bit ? set : ~set;
          }
          const uint32_t rank = (uint32_t)__popc(less | (same & ((1u << lane) - 1u)));
          const int off = (int)u32 - (int)rank;
          uint32_t rot = (uint32_t)(__reduce_max_sync(0xFFFFFFFFu, off) - off);
          if (rot >= n) rot = 0;
          const uint32_t first = n - rot;                    // steps before the wrap
          const uint32_t k1 = __reduce_min_sync(0xFFFFFFFFu, first);
          const uint32_t k2 = nmin, k3 = nmin + 1u;
          const uint32_t p4 = 4u * p, turn = n * p4;
          uint32_t q = sseg + 4u * w0 + p4 * rot;
          uint32_t k = 0;
#pragma unroll 16
          for (; k < k1; ++k, q += p4) and_word(q, mask);
#pragma unroll 8
          for (; k < k2; ++k, q += p4) {                     // some lanes have wrapped
            if (k == first) q -= turn;
            and_word(q, mask);
          }
          for (; k < k3; ++k, q += p4) {                     // some lanes are done
            if (k == first) q -= turn;
            and_word_if(q, mask, k < n);
          }
        } else if (u >= nscan) {
          // bucket list of this segment: primes >= the bucket split whose
          // hits were listed by bucket_fill_kernel; entries read coalesced
          const uint64_t base = bbase + (uint64_t)(u - nscan) * kBucketUnit;
          const uint32_t lim = min(kBucketUnit, bcnt - (u - nscan) * kBucketUnit);
#pragma unroll 8
          for (uint32_t e = lane; e < lim; e += 32) {
            // entry = bit index: word v / 32, and ~(1 << (v mod 32)) is
            // 0xFFFFFFFE rotated by v (a funnel shift takes its count mod 32)
            const uint32_t v = __ldg(prm.bucket + base + e);
            atomicAnd(seg + (v >> 5), __funnelshift_l(0xFFFFFFFEu, 0xFFFFFFFEu, v));
          }
        } else if (u >= nsmall + nmidu) {
          // wheel tier: a lane per prime of one class mod 30, its eight hits
          // per turn of p bytes in the order of their cofactors w mod 30: the
          // first lies at t w + const - k0 (mod p), the next ones follow by p.
          // What bounds it: shared-memory wavefronts (3.5 per atomic on random
          // banks) below the segment size, at 6 instructions per clear; issue
          // above, at about 100 instructions per prime and segment, 60 from 2.5
          // segments on.  Reading a prime's eight residues instead costs 44
          // bytes where this takes 8, and with a 64-bit reduction and a branch
          // per clear 168 and 13 instructions ([9*10^11, 10^12) 20.8 ms to 16.5
          // when that was the difference).
          const uint32_t wu = u - nsmall - nmidu;
          const uint32_t cls = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, lane < 8u && wu >= wincl));
          const uint32_t ubeg = __shfl_sync(0xFFFFFFFFu, wincl, (cls + 31u) & 31u);
          const uint32_t cend = __shfl_sync(0xFFFFFFFFu, wend, cls);
          uint32_t i = __shfl_sync(0xFFFFFFFFu, wbeg, cls) + ((wu - (cls ? ubeg : 0u)) << wlog) + lane;
          const uint32_t cc = w30(cls);
          const WheelClass& C = cWheel.c[cls];
          const uint2* __restrict__ W = reinterpret_cast<const uint2*>(prm.W);
          // past the class's end a lane repeats its last prime: the same
          // clears again
          uint2 e = __ldg(W + min(i, cend - 1u));
          const uint32_t pfirst = __reduce_min_sync(0xFFFFFFFFu, 30u * e.x + cc);
          uint32_t left = 1u << (wlog - 5u);            // batches of 32 primes
          const uint32_t wend4 = sseg + ((unb + 3u) & ~3u);       // address past the last word
          if (pfirst >= 15u * unb) {
            // at most one hit at all (cofactors coprime to 30 lie 2 apart or
            // more): the first multiple p (30 a + w) of the segment is found
            // directly, from 30 (k0 mod p) / p and the next w from there: 16
            // operations on the integer pipe (as the smallest of the eight
            // classes' hits, below, 40, twice its share).
            constexpr uint32_t kCoprime = 0xA08A2882u;    // residues 1 7 11 13 17 19 23 29, and 31 for the next turn's 1
            auto mark = [&](uint2 q) {
              const uint32_t p = 30u * q.x + cc, inv = q.y;
              uint32_t m = k0l - __umulhi(k0s, inv) * p;
              m = min(m, m - p);
              m = min(m, m - p);
              const uint32_t m30 = 30u * m;
              uint32_t r = __umulhi(m30, inv) >> 10;      // 30 m / p, or one less
              r += m30 - r * p >= p ? 2u : 1u;            // cofactors from r on give numbers >= 30 k0
              const uint32_t w = r + (uint32_t)__ffs(kCoprime >> r) - 1u;
              const uint32_t n = w * p - m30;             // the hit's number in the segment, at most 6 p
              const uint32_t byte = __umulhi(n, 143165577u);            // n / 30 (exact below 3 * 10^8)
              clear_bit_below(sseg, 8u * byte + (((n - 30u * byte) * 17477u) >> 16), wend4);   // W30[o] * 4 / 15 = o
            };
            // (So few operations per prime leave the table's L2 reads to bound
            // the loop at 6 TB/s over the chip; more batches in flight per
            // warp than one ahead gain nothing.)
            for (;;) {
              const uint2 now = e;
              if (--left) e = __ldg(W + min(i += 32u, cend - 1u));
              mark(now);
              if (!left) break;
            }
          } else if (pfirst >= unb) {
            // at most one hit per class: positions as bit indices 8 * byte +
            // class, whose low bits also give the mask
            uint32_t step[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) step[j] = C.bstep[j];
            // Hits of cofactors w and w' (mod 30) lie at least |w - w'| / 30 and
            // 1 - |w - w'| / 30 of p apart, so of a group of classes whose
            // cofactors keep a distance of 12 or 6 round the circle at most one
            // hit is inside, from 2.5 or 5 segments on: one clear for the
            // smallest of the group.
            const uint32_t group = pfirst >= 5u * unb ? 4u : 2u * pfirst >= 5u * unb ? 2u : 1u;
            for (;;) {
              const uint32_t p = 30u * e.x + cc;
              uint32_t m = k0l - __umulhi(k0s, e.y) * p;
              const uint32_t t2 = 16u * e.x, t4 = 32u * e.x, t6 = 48u * e.x, p8 = 8u * p;
              uint32_t y = 8u * e.x + step[0];
              if (--left) e = __ldg(W + min(i += 32u, cend - 1u));
              m = min(m, m - p);
              m = min(m, m - p);
              y -= 8u * m;
              uint32_t v[8];
              v[0] = min(y, y + p8);
#pragma unroll
              for (int j = 1; j < 8; ++j) {
                // W30 steps 6 4 2 4 2 4 6
                y += (j == 1 || j == 7 ? t6 : j == 3 || j == 5 ? t2 : t4) + step[j];
                v[j] = min(y, y + p8);
              }
              if (group == 4u) {                   // w = 1 7 13 19 and 11 17 23 29
                clear_bit_below(sseg, min(min(v[0], v[1]), min(v[3], v[5])), wend4);
                clear_bit_below(sseg, min(min(v[2], v[4]), min(v[6], v[7])), wend4);
              } else if (group == 2u) {                   // w_j and w_(j+4): 16, 12, 12, 16 apart
#pragma unroll
                for (int j = 0; j < 4; ++j) clear_bit_below(sseg, min(v[j], v[j + 4]), wend4);
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) clear_bit_below(sseg, v[j], wend4);
              }
              if (!left) break;
            }
          } else {
            // several hits per class; whole turns of the batch's largest
            // prime need no test
            uint32_t step[8], keep[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) { step[j] = C.step[j]; keep[j] = C.keep[j]; }
            for (;;) {
              const uint32_t p = 30u * e.x + cc;
              uint32_t m = k0l - __umulhi(k0s, e.y) * p;
              m = min(m, m - p);
              m = min(m, m - p);
              const uint32_t t2 = 2u * e.x, t4 = 4u * e.x, t6 = 6u * e.x;
              uint32_t pos[8];
              uint32_t y = e.x - m;                     // offset of the hit of w = 1, mod p
              pos[0] = min(y, y + p);
#pragma unroll
              for (int j = 1; j < 8; ++j) {
                y += (j == 1 || j == 7 ? t6 : j == 3 || j == 5 ? t2 : t4) + step[j];
                pos[j] = min(y, y + p);
              }
              uint32_t n = __umulhi(unb, e.y) >> 10;
              if ((n + 1u) * p <= unb) ++n;             // floor(nbytes / p)
              if (--left) e = __ldg(W + min(i += 32u, cend - 1u));
#pragma unroll
              for (int j = 0; j < 8; ++j) pos[j] += sseg;
              const uint32_t nall = __reduce_min_sync(0xFFFFFFFFu, n);
              const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, n) + 1u;
              uint32_t k = 0;
#pragma unroll 1
              for (; k < nall; ++k) {
#pragma unroll
                for (int j = 0; j < 8; ++j) { clear_at(pos[j], keep[j]); pos[j] += p; }
              }
#pragma unroll 1
              for (; k < nmax; ++k) {
#pragma unroll
                for (int j = 0; j < 8; ++j) { clear_below(pos[j], keep[j], send); pos[j] += p; }
              }
              if (!left) break;
            }
          }
        } else {
          // mid tier: p, k0 mod p and the whole turns of p once per prime (lane
          // = prime), then shuffled to the (prime, class) lanes of each round.
          // Past the tier's end a lane repeats its last prime.
          const uint32_t base = nsmall + 32u * (u - nsmall);
          const uint32_t im = min(base + lane, mend - 1u);
          const uint32_t pm = __ldg(prm.P + im);
          const uint32_t mm = mod_barrett(k0, pm, __ldg(prm.M + im));
          const uint32_t nm = unb / pm;
          const uint32_t keep = ~(1u << o);
          uint32_t rr[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) rr[t] = __ldg(prm.R + 8u * min(base + 4u * t + h, mend - 1u) + o);
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const uint32_t p = __shfl_sync(0xFFFFFFFFu, pm, 4 * t + h);
            const uint32_t m = __shfl_sync(0xFFFFFFFFu, mm, 4 * t + h);
            uint32_t s = rr[t] - m;
            s = min(s, s + p);
            const bool mine = (lane >> 2) == (uint32_t)t;
            const uint32_t nall = __reduce_min_sync(0xFFFFFFFFu, mine ? nm : ~0u);
            const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, mine ? nm : 0u) + 1u;
            uint32_t j = sseg + s, k = 0;
#pragma unroll 8
            for (; k < nall; ++k, j += p) clear_at(j, keep);
#pragma unroll 2
            for (; k < nmax; ++k, j += p) clear_below(j, keep, send);
          }
        }
      }
    }
    __syncthreads();
    // Multiples of p below p*p are cleared too; they are composite anyway, but
    // for p itself.  Only a segment that starts below 128 bytes can hold a
    // prime that sieves it (p*p < 30 (k0 + nbytes) and p >= 30 k0 need k0 <=
    // 86; the rounding to a row adds primes of less than 3840): there they are
    // set again.  This spares every hit a p*p test.
    // (Solo sieves every segment with the request's last prime; its host gives
    // the bound.)
    if (kSolo && slices > 1u) {
      // merge the slices; the last one to arrive goes on
      uint32_t* const words = prm.merge + (uint64_t)item * (prm.seg_bytes >> 2);
      for (uint32_t w = tid; w < nwords; w += nthr)
        if (seg[w] != ~0u) atomicAnd(words + w, seg[w]);
      __threadfence();
      __syncthreads();
      if (tid == 0) s_ctr = atomicAdd(&prm.ctl->seg_done[item], 1u);
      __syncthreads();
      if (s_ctr != slices - 1u) return;
      __threadfence();
      fill(k0, tid, (nbytes + 15u) >> 4, nthr, words);
      __syncthreads();
      uint4* const w4 = reinterpret_cast<uint4*>(words);
      for (uint32_t v = tid; v < (nbytes + 15u) >> 4; v += nthr) w4[v] = make_uint4(~0u, ~0u, ~0u, ~0u);
      if (tid == 0) prm.ctl->seg_done[item] = 0;
    }
    if (k0 < (kSolo ? prm.low_k : 128u)) {
      const uint32_t nset = min((np + kWheelRow - 1u) / kWheelRow * kWheelRow, prm.ntab);
      for (uint32_t i = tid; i < nset; i += nthr) {
        const uint32_t p = __ldg(prm.P + i), k = p / 30u;
        if (k < k0 || k - (uint32_t)k0 >= nbytes) continue;
        const uint32_t v = 8u * (k - (uint32_t)k0) + (p % 30u) * 4u / 15u;    // W30[o] * 4 / 15 = o
        atomicOr(seg + (v >> 5), 1u << (v & 31u));
      }
      __syncthreads();
    }
    if (tid == 0) s_ctr = 0;                        // every unit is taken: reset for the next segment

    // 3. reductions: each thread scans one contiguous run of words (odd
    //    length, so the lanes of a warp hit distinct banks); lanes are
    //    stitched with a warp max-scan of their last prime, warps by warp 0.
    {
      const uint32_t run = ((nwords + nthr - 1) / nthr) | 1u;
      const uint32_t wbeg = min(tid * run, nwords);
      const uint32_t wend = min(wbeg + run, nwords);
      // edge fix-ups, each by the thread whose run holds the word
      if (wbeg == 0 && wend > 0) seg[0] = ((seg[0] & S.and0) | S.or0) & S.keep0;
      if (wbeg < wend && wend == nwords) seg[nwords - 1u] &= S.keepl;
      if (prm.flags & kFlagBitmap) {
        __syncthreads();
        uint32_t* dst = prm.bitmap + ((k0 - (kForm != kFormBatch ? prm.solo.k_lo : prm.reqs[0].k_lo)) >> 2);
        for (uint32_t w = tid; w < nwords; w += nthr) dst[w] = seg[w];
      }
      GapSink sk;
      sk.shist = shist + (warp % kSmemHistCopies) * kSmemStride;
      sk.acc = prm.acc + req;
      sk.large = prm.large; sk.n_large = prm.n_large; sk.cap = prm.large_cap;
      sk.req = req; sk.base = 30ull * k0;
      const uint32_t m41 = (k0 & 1ull) ? 0x99669966u : 0x66996699u;
      uint32_t first1 = 0, last1 = 0, cnt = 0, c41 = 0, c31 = 0, maxg = 0, maxgs = 0;
      const bool gaps = kLone ? kForm == kFormLone : uniform(S.rflags & kReqGaps) != 0;
      if (gaps) {
        // Byte by byte, four fixed steps per word, so the lanes of a warp
        // stay in step whatever their primes.  A byte's value is counted in
        // the byte histogram (its primes and the gaps inside it follow from
        // that when the request is flushed), the gap into it from the
        // previous prime in the gap histogram, and the largest such gap is
        // kept as g << 23 | (2^23 - 1 - end), the earliest first on ties
        // (nv and npv are 2^23 - 1 - the gap's end and start).
        // 7 shared-memory wavefronts and 24 instructions per byte and warp,
        // and issue bounds it (a 16-byte table entry per byte with the inner
        // gaps as packed counters: 12 and 35, [9*10^11, 10^12) 16.5 ms to 14.8).
        // A run is walked prime by prime only where it holds a gap beyond the
        // shared bins, or where no gap between bytes of the whole warp exceeds
        // 28, the largest inside a byte.
        const uint32_t hb = (uint32_t)__cvta_generic_to_shared(sk.shist);
        const uint32_t bb = (uint32_t)__cvta_generic_to_shared(bhist + (warp % kSmemHistCopies) * kByteValues);
        constexpr uint32_t kWlo = (uint32_t)kW30Packed, kWhi = (uint32_t)(kW30Packed >> 32);
        constexpr uint32_t kEnd = (1u << 23) - 1u;
        static_assert(30u * kMaxSegBytes < kEnd && 2 * kSmemBins < 512, "a gap and its end share 32 bits");
        const uint32_t tb = (uint32_t)__cvta_generic_to_shared(btab);
        uint32_t fi = wbeg;                         // the run's first prime is its first "previous" one (gap 0)
        while (fi < wend && !seg[fi]) ++fi;
        uint32_t pv = fi < wend ? 120u * fi + word_value(__ffs(seg[fi]) - 1u) : 0u;
        if (fi < wend) first1 = pv + 1u;
        uint32_t top = 0, npv = kEnd - pv;
        const uint32_t nsteps = uniform(run);
#pragma unroll 4
        for (uint32_t i = 0; i < nsteps; ++i) {
          const uint32_t wi = wbeg + i;
          const uint32_t w = wi < wend ? seg[wi] : 0u;
          c41 += __popc(w & m41);
          const int nvb = (int)(kEnd - 120u * wi);
#pragma unroll
          for (uint32_t b = 0; b < 4; ++b) {
            const uint32_t x = (w >> (8u * b)) & 0xFFu;
            if (x) {
              uint32_t e;
              asm volatile("ld.shared.u8 %0, [%1];" : "=r"(e) : "r"(tb + x));
              count_one(bb + 4u * x);
              const int r = (int)__byte_perm(kWlo, kWhi, e);      // bytes: W30 of the lowest, of the highest bit
              const uint32_t nv = (uint32_t)__dp4a(r, 0x000000FF, nvb - 30 * (int)b);
              const uint32_t g = min(npv - nv, 2u * (uint32_t)kSmemBins);
              npv = (uint32_t)__dp4a(r, 0x0000FF00, nvb - 30 * (int)b);
              count_one(hb + 2u * g);
              top = max(top, g * (1u << 23) + nv);
            }
          }
        }
        if (first1) {
          last1 = kEnd - npv + 1u;
          maxg = top >> 23;
          maxgs = kEnd - (top & kEnd) - maxg;
        }
        const uint32_t wmax = __reduce_max_sync(0xFFFFFFFFu, maxg);
        if (first1 && (wmax <= 28u || maxg >= 2u * (uint32_t)kSmemBins)) {
          const uint2 m = walk_run(sk, seg, wbeg, wend);
          maxg = m.x;
          maxgs = m.y;
        }
      } else {
        // Count only: the run's words are added bit by bit (carry-save, eight
        // words per step), so three masked popcounts per step of eight words
        // give the primes and those 1 mod 4 and 1 mod 3; popcounts run at a
        // quarter of the integer rate (of every word, a count to 3*10^10 takes
        // 2.83 ms to 2.71).
        uint32_t ones = 0, twos = 0, fours = 0, n8 = 0, a8 = 0, b8 = 0;
        constexpr uint32_t m31 = 0x2B2B2B2Bu;
        auto add = [](uint32_t& s, uint32_t x, uint32_t y) {      // s + x + y per bit: the sum, and the carry
          const uint32_t c = (s & x) | (s & y) | (x & y);
          s ^= x ^ y;
          return c;
        };
        const uint32_t nsteps = uniform(run);
        for (uint32_t i = 0; i < nsteps; i += 8u) {
          uint32_t w[8];
#pragma unroll
          for (uint32_t t = 0; t < 8; ++t) w[t] = wbeg + i + t < wend ? seg[wbeg + i + t] : 0u;
          const uint32_t t0 = add(ones, w[0], w[1]), t1 = add(ones, w[2], w[3]);
          const uint32_t t2 = add(ones, w[4], w[5]), t3 = add(ones, w[6], w[7]);
          const uint32_t f0 = add(twos, t0, t1), f1 = add(twos, t2, t3);
          const uint32_t e = add(fours, f0, f1);
          n8 += __popc(e);
          a8 += __popc(e & m41);
          b8 += __popc(e & m31);
        }
        cnt = 8u * n8 + 4u * __popc(fours) + 2u * __popc(twos) + __popc(ones);
        c41 = 8u * a8 + 4u * __popc(fours & m41) + 2u * __popc(twos & m41) + __popc(ones & m41);
        c31 = 8u * b8 + 4u * __popc(fours & m31) + 2u * __popc(twos & m31) + __popc(ones & m31);
        if (cnt) {
          uint32_t wi = wbeg, wl = wend - 1u;
          while (!seg[wi]) ++wi;                    // the run holds a prime
          while (!seg[wl]) --wl;
          first1 = 120u * wi + word_value(__ffs(seg[wi]) - 1u) + 1u;
          last1 = 120u * wl + word_value(31u - __clz(seg[wl])) + 1u;
        }
      }
      // lane stitching: previous lane's last prime (values grow with the lane)
      uint32_t sc = last1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, sc, d);
        if ((int)lane >= d) sc = max(sc, t);
      }
      uint32_t prev1 = __shfl_up_sync(0xFFFFFFFFu, sc, 1);
      if (lane == 0) prev1 = 0;
      if (gaps && first1 && prev1) record_gap(sk, prev1 - 1u, first1 - 1u, maxg, maxgs);
      const uint32_t wlast = __shfl_sync(0xFFFFFFFFu, sc, 31);
      const uint32_t wfirst = __reduce_min_sync(0xFFFFFFFFu, first1 ? first1 : 0xFFFFFFFFu);
      cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
      c41 = __reduce_add_sync(0xFFFFFFFFu, c41);
      c31 = __reduce_add_sync(0xFFFFFFFFu, c31);
      const uint32_t gm = __reduce_max_sync(0xFFFFFFFFu, maxg);
      const uint32_t gs = __reduce_min_sync(0xFFFFFFFFu, (maxg == gm && gm) ? maxgs : 0xFFFFFFFFu);
      if (lane == 0) {
        WarpRec r;
        r.first1 = wfirst == 0xFFFFFFFFu ? 0u : wfirst;
        r.last1 = wlast; r.cnt = cnt; r.c41 = c41; r.c31 = c31;
        r.maxg = gm; r.maxgs = gs; r.pad = 0;
        wrec[warp] = r;
      }
      // After a gap scan a warp fills its words for the next segment, where
      // that has runs as long (and no other warp still copies them out): the
      // fill's loads from L2 overlap the other warps' scan, and the segment
      // needs a barrier less (10^10 numbers at 0 1.033 -> 1.023 ms, at 10^12
      // 1.383 -> 1.372).  After a count's short scan, which leaves little to
      // overlap, filling in turn costs 0.5 % more than all threads do.
      if constexpr (!kSolo && kForm != kFormLoneCount) {
        const SegItem& N = s_item[cur ^ 1u];
        const bool filled = gaps && N.valid && !(prm.flags & kFlagBitmap) &&
                            ((((N.nbytes + 3u) >> 2) + nthr - 1) / nthr | 1u) == run;
        if (tid == 0) s_filled = filled;
        if (filled) {
          __syncwarp();
          fill(N.k0, 8u * run * warp + lane, min(8u * run * (warp + 1u), (N.nbytes + 15u) >> 4), 32u, nullptr);
        }
      }
      __syncthreads();
      // warps are stitched like lanes, lane = warp: the gap from the last
      // prime before a warp to its first prime, the largest gap (ties: the
      // first), the sums
      if (warp == 0) {
        WarpRec r = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        if (lane < nwarps) r = wrec[lane];
        uint32_t sw = r.last1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, sw, d);
          if ((int)lane >= d) sw = max(sw, t);
        }
        uint32_t before = __shfl_up_sync(0xFFFFFFFFu, sw, 1);
        if (lane == 0) before = 0;
        uint32_t bg = 0, bs = 0;
        if (gaps && r.first1 && before) record_gap(sk, before - 1u, r.first1 - 1u, bg, bs);
        if (r.maxg > bg) { bg = r.maxg; bs = r.maxgs; }   // on a tie the joining gap starts first
        const uint32_t gm = __reduce_max_sync(0xFFFFFFFFu, bg);
        const uint32_t gs = __reduce_min_sync(0xFFFFFFFFu, (bg == gm && gm) ? bs : 0xFFFFFFFFu);
        const uint32_t fst1 = __reduce_min_sync(0xFFFFFFFFu, r.first1 ? r.first1 : 0xFFFFFFFFu);
        const uint32_t run1 = __shfl_sync(0xFFFFFFFFu, sw, 31);
        const uint32_t tc = __reduce_add_sync(0xFFFFFFFFu, r.cnt);
        const uint32_t t41 = __reduce_add_sync(0xFFFFFFFFu, r.c41);
        const uint32_t t31 = __reduce_add_sync(0xFFFFFFFFu, r.c31);
        if (lane == 0) {
          SegRec sr;
          sr.first = fst1 != 0xFFFFFFFFu ? sk.base + fst1 - 1u : 0;
          sr.last = run1 ? sk.base + run1 - 1u : 0;
          sr.max_gap = gm;
          sr.max_gap_start = gm ? sk.base + gs : 0;
          sr.pad = 0;
          prm.segs[item] = sr;
          if (t41) atomicAdd(&sk.acc->c41, (unsigned long long)t41);
          if (tc) {                                   // with gaps: from the byte histogram
            atomicAdd(&sk.acc->count, (unsigned long long)tc);
            atomicAdd(&sk.acc->c31, (unsigned long long)t31);
          }
        }
      }
    }
  }
  __syncthreads();
  if (cur_req >= 0 && cur_gaps) flush();
  if constexpr (kForm != kFormBatch) {
    // the last segment to be reduced (the last CTA to run out of segments)
    // writes the result and leaves the accumulators and the control words
    // clear for the next run
    const uint32_t parts = kSolo ? (uint32_t)prm.solo.nseg : gridDim.x;
    if (parts > 1) {
      __threadfence();
      __syncthreads();
      if (tid == 0) s_ctr = atomicAdd(&prm.ctl->done, 1u);
      __syncthreads();
      if (s_ctr != parts - 1u) return;
      __threadfence();
    } else {
      __syncthreads();
    }
    // (the segment is done with: its memory serves)
    finalize_request<true>(prm.solo, 0u, prm.segs, prm.acc, prm.large, &prm.ctl->n_large, prm.large_cap,
                           &prm.out->res, smem);
    __syncthreads();
    if (tid == 0) {
      prm.out->n_large = __ldcg(&prm.ctl->n_large);
      prm.ctl->n_large = 0;
      prm.ctl->done = 0;
      prm.ctl->queue = 0;
    }
  }
}

__global__ void __launch_bounds__(kMaxThreads, 1) sieve_segments_kernel(const SieveParams prm) {
  sieve_body<kFormBatch>(prm);
}

// A lone request in one launch.  A range of one wave or less leaves most of
// its time in launches, copies and, at high offsets, in one CTA per segment
// walking all sieving primes (a 4096-wide window at 10^12: 82 us in one CTA).
// Here the request comes as a parameter, `slices` CTAs share each segment's
// units and merge what they cleared in L2, the last of them reduces the
// segment, and the last segment writes the result to host memory.  No CTA
// waits for another.
__global__ void __launch_bounds__(kMaxThreads, 1) solo_kernel(const __grid_constant__ SieveParams prm) {
  sieve_body<kFormSolo>(prm);
}

// A lone request of more segments than a wave, without lists, in one launch:
// one CTA per SM takes segments from a queue, and the last CTA to find it empty
// writes the result to host memory.  As a plan the same request takes a copy up,
// a zeroing launch, the sieve, a launch of one block that folds the records
// and two copies down with a wait each: Context(10^10) 1079 us instead of 1052,
// 2*10^9 numbers at 0 234 instead of 221, Context(10^12) 125.5 ms instead of
// 124.3.
__global__ void __launch_bounds__(kMaxThreads, 1) lone_kernel(const __grid_constant__ SieveParams prm) {
  sieve_body<kFormLone>(prm);
}
// The same for counts alone: without the gap scan's code in the kernel a count
// of [0, 3*10^10) takes 2456 us instead of 2462.
__global__ void __launch_bounds__(kMaxThreads, 1) lone_count_kernel(const __grid_constant__ SieveParams prm) {
  sieve_body<kFormLoneCount>(prm);
}

// A CTA per request; a lone one's records are folded by 1024 threads (150 000
// records: 0.18 ms, by 256 threads 0.54).
__global__ void __launch_bounds__(kMaxThreads)
finalize_kernel(const ReqDesc* __restrict__ reqs, const BatchHdr* __restrict__ hdr,
                const SegRec* __restrict__ segs, ReqAccum* __restrict__ acc, LargeGapRec* large,
                unsigned int* n_large, uint32_t large_cap, ReqResult* __restrict__ out) {
  const uint32_t r = blockIdx.x;
  if (r >= hdr->nreq) return;       // fixed-size launches (graph replay) cover capacity
  __shared__ __align__(8) uint32_t tmp[kFinalWords];
  const ReqDesc R = reqs[r];
  finalize_request<false>(R, r, segs + R.seg_base, acc + r, large, n_large, large_cap, out + r, tmp);
}

// Bucket fill: one CTA per work item (a request, a run of its bucket primes
// and a run of its segments; heavy runs of small primes are split over
// several items so that items carry similar numbers of hits), a thread per
// prime walking its eight classes as eight independent chains.  A chain is the
// hit's byte k in the item's segments; its segment is k / S by a
// multiplication, and its entry goes to the next place of that segment's bin
// in shared memory.  Then one global atomic per segment reserves room in that
// segment's list, and a warp per segment copies its bin there: 3 write requests
// per 32 entries.  What bounds it: shared-memory wavefronts and issue, half and
// half (a returning atomic and a store on random banks per hit).
// [10^14, 10^14 + 10^9) 82 us of 325, [10^14 - 10^11, 10^14) 24.4 ms in all;
// counting in a first walk and storing each entry from its lane in a second one,
// with 16 write requests per 32 entries as the bound, 97 of 342 us and 26.8 ms.
// The bins hold 1.54 times an item's expected hits: with at most kFillSegs
// segments their mean is 54 entries and the margin 4 standard deviations.
// Primes near sqrt(b) have their hits in clusters (p q = s^2 / 4 - d^2 / 4
// hardly moves with p for a fixed sum s = p + q), and other items can draw an
// overfull bin too: such an item walks again and stores its entries from the
// lanes, at the places that the counts of the first walk reserve.
// A list that would overflow its capacity raises *overflow and drops the
// entries past it (the host then reruns without lists).
struct FillShared {
  uint32_t cnt[kFillSegs];
  uint32_t gpos[kFillSegs];      // the next place in the segment's list
  uint32_t stage[kFillStage];    // the bins, kFillStage / (the item's segments) entries each
};

__global__ void __launch_bounds__(kFillPrimes)
bucket_fill_kernel(const FillParams fp) {
  extern __shared__ __align__(16) uint32_t smem[];
  FillShared& sh = *reinterpret_cast<FillShared*>(smem);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t nitems = fp.nitems ? fp.nitems : fp.hdr->nfill;
  for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
    const FillItem item = fp.items[it];
    const ReqDesc R = fp.reqs[item.req];
    // segments g0..g1 of the window that starts at segment seg0 of the
    // request; byte numbers below are relative to segment g0, at k0
    const uint32_t g0 = item.segs & 0xFFFFu, g1 = item.segs >> 16;
    const uint32_t nseg = g1 - g0;
    const uint32_t cap = R.bucket_cap, S = R.seg_bytes;
    const uint64_t k0 = R.k_lo + (uint64_t)(fp.seg0 + g0) * S;
    const uint32_t h = (uint32_t)min(R.k_hi - k0, (uint64_t)nseg * S);
    // k / S = hi32(k mag) >> shift, exact for k < 2^12 S and S <= 2^19: mag S -
    // 2^(32 + shift) < S, and 2^12 S S < 2^(32 + shift), 2^shift < S <= 2^(shift + 1)
    static_assert(kFillSegs < 4096 && kMaxSegBytes <= 1u << 19, "k / S by one multiplication");
    const uint32_t shift = 31u - (uint32_t)__clz(S - 1u);
    const uint32_t mag = (uint32_t)(((1ull << (32u + shift)) + S - 1u) / S);
    // the item's lists, segment g at g * cap (the host keeps a window's
    // entries below 2^32)
    uint32_t* const list = fp.bucket + R.bucket_base + (uint64_t)g0 * cap;
    unsigned int* const gcount = fp.bcount + R.seg_base + fp.seg0 + g0;
    const uint32_t bin = kFillStage / nseg;
    for (uint32_t g = tid; g < nseg; g += kFillPrimes) sh.cnt[g] = 0;
    const uint32_t i = item.p0 + tid;
    uint32_t start[8], step = 0, whole = 0;
    bool low = false;
#pragma unroll
    for (int o = 0; o < 8; ++o) start[o] = h;
    if (i < item.p1) {
      load_residues(fp.R, i, start);
      const uint32_t p = __ldg(fp.P + i);
      const uint32_t m = mod_barrett(k0, p, __ldg(fp.M + i));
      low = 30ull * k0 < (uint64_t)p * p;
      step = min(p, h);                            // (k stays below 2 h)
      whole = low ? 0u : h / p;
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        start[o] = start[o] >= m ? start[o] - m : start[o] + p - m;
        if (low) start[o] = lift_to_square(start[o], k0, p, o, h);
        start[o] = min(start[o], h);
      }
    }
    __syncthreads();
    {
      uint32_t k[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) k[o] = start[o];
      auto put = [&](uint32_t x, uint32_t o) {
        const uint32_t g = __umulhi(x, mag) >> shift;
        const uint32_t pos = min(atomicAdd(&sh.cnt[g], 1u), bin - 1u);
        sh.stage[g * bin + pos] = bucket_entry(x - g * S, o);
      };
      for (uint32_t t = 0; t < whole; ++t) {
#pragma unroll
        for (uint32_t o = 0; o < 8; ++o) { put(k[o], o); k[o] += step; }
      }
      do {
#pragma unroll
        for (uint32_t o = 0; o < 8; ++o)
          if (k[o] < h) { put(k[o], o); k[o] += step; }
      } while (low && min(min(min(k[0], k[1]), min(k[2], k[3])), min(min(k[4], k[5]), min(k[6], k[7]))) < h);
    }
    __syncthreads();
    bool mine = false;
    for (uint32_t g = tid; g < nseg; g += kFillPrimes) mine |= sh.cnt[g] > bin;
    const bool full = __syncthreads_or(mine);
    for (uint32_t g = tid; g < nseg; g += kFillPrimes) {
      const uint32_t c = sh.cnt[g];
      const uint32_t at = c ? atomicAdd(gcount + g, c) : 0u;
      if (at + c > cap) atomicOr(fp.overflow, 1u);
      sh.gpos[g] = at;
    }
    __syncthreads();
    if (!full) {
      for (uint32_t g = warp; g < nseg; g += kFillPrimes / 32) {
        const uint32_t at = sh.gpos[g], n = min(sh.cnt[g], cap - min(at, cap));
        uint32_t* const to = list + ((uint64_t)g * cap + at);
        const uint32_t* const from = sh.stage + g * bin;
#pragma unroll 2
        for (uint32_t e = lane; e < n; e += 32) to[e] = from[e];
      }
    } else {
#pragma unroll
      for (uint32_t o = 0; o < 8; ++o) {
#pragma unroll 1
        for (uint32_t k = start[o]; k < h; k += step) {
          const uint32_t g = __umulhi(k, mag) >> shift;
          const uint32_t pos = atomicAdd(&sh.gpos[g], 1u);
          if (pos < cap) list[(uint64_t)g * cap + pos] = bucket_entry(k - g * S, o);
        }
      }
    }
    __syncthreads();
  }
}

// Rebuild caller requests from shared atoms (disjoint pieces of the batch's
// ranges, each sieved once).  A request is the ordered run of its atoms:
// counts add; its gaps are the atoms' inner gaps plus one junction gap
// between each atom holding primes and the next such atom; the maximal gap
// is the largest of those, the earliest on ties, as within one range.  Each
// thread folds a contiguous run of atoms, thread 0 joins the runs in order.
// A request that asked for counts only gets no gap outputs even where its
// atoms were scanned for another request's gaps, so its result is the one
// it gets alone.
__global__ void __launch_bounds__(256)
combine_kernel(const BatchHdr* __restrict__ hdr, const ReqSpan* __restrict__ spans,
               const uint32_t* __restrict__ apos, const ReqResult* __restrict__ ares,
               ReqResult* __restrict__ out) {
  const uint32_t r = blockIdx.x, tid = threadIdx.x;
  if (r >= hdr->nout) return;
  const ReqSpan sp = spans[r];
  const bool gaps = (sp.rflags & kReqGaps) != 0;
  __shared__ uint32_t jh[kHistBins];
  __shared__ uint64_t t_first[256], t_last[256], t_bg[256], t_bs[256];
  __shared__ uint64_t t_sum[5][256];
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += blockDim.x) jh[b] = 0;
  __syncthreads();

  auto add_gap = [&](uint64_t g, uint64_t st, uint64_t& bg, uint64_t& bs) {
    const uint64_t bin = g >> 1;
    atomicAdd(&jh[bin < (uint64_t)kHistBins ? bin : kHistBins - 1], 1u);
    if (g > bg || (g == bg && st < bs)) { bg = g; bs = st; }
  };
  const uint32_t n = sp.e - sp.s;
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t j0 = sp.s + min(n, tid * per), j1 = sp.s + min(n, (tid + 1) * per);
  uint64_t c[5] = {0, 0, 0, 0, 0};
  uint64_t first = 0, last = 0, bg = 0, bs = 0;
  for (uint32_t j = j0; j < j1; ++j) {
    const ReqResult* A = ares + apos[j];
    const uint64_t ac = A->count;
    c[0] += ac; c[1] += A->c41; c[2] += A->c43; c[3] += A->c31; c[4] += A->c32;
    if (!ac) continue;
    if (!first) first = A->first;
    if (gaps) {
      if (last) add_gap(A->first - last, last, bg, bs);
      const uint64_t mg = A->max_gap;
      if (mg && (mg > bg || (mg == bg && A->max_gap_start < bs))) { bg = mg; bs = A->max_gap_start; }
    }
    last = A->last;
  }
  t_first[tid] = first; t_last[tid] = last; t_bg[tid] = bg; t_bs[tid] = bs;
#pragma unroll
  for (int q = 0; q < 5; ++q) t_sum[q][tid] = c[q];
  __syncthreads();
  ReqResult* O = out + r;
  if (tid == 0) {
    uint64_t s5[5] = {0, 0, 0, 0, 0};
    uint64_t f = 0, l = 0, g = 0, gs = 0;
    for (uint32_t t = 0; t < blockDim.x; ++t) {
#pragma unroll
      for (int q = 0; q < 5; ++q) s5[q] += t_sum[q][t];
      if (!t_first[t]) continue;
      if (!f) f = t_first[t];
      if (gaps) {
        if (l) add_gap(t_first[t] - l, l, g, gs);
        if (t_bg[t] && (t_bg[t] > g || (t_bg[t] == g && t_bs[t] < gs))) { g = t_bg[t]; gs = t_bs[t]; }
      }
      l = t_last[t];
    }
    O->count = s5[0]; O->c41 = s5[1]; O->c43 = s5[2]; O->c31 = s5[3]; O->c32 = s5[4];
    O->first = f;
    O->last = l;
    O->max_gap = g;
    O->max_gap_start = g ? gs : 0;
    O->num_gaps = s5[0] ? s5[0] - 1 : 0;
  }
  __syncthreads();
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += blockDim.x) {
    uint64_t h = 0;
    if (gaps) {
      h = jh[b];
      for (uint32_t j = sp.s; j < sp.e; ++j) h += ares[apos[j]].hist[b];
    }
    O->hist[b] = h;
  }
}

// Zero up to three regions in one launch (a plan's accumulators, control
// words and bucket counts, before each run).
__global__ void zero_kernel(ZeroSpan z0, ZeroSpan z1, ZeroSpan z2) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (uint64_t i = t0; i < z0.n16; i += stride) static_cast<uint4*>(z0.p)[i] = zero;
  for (uint64_t i = t0; i < z1.n16; i += stride) static_cast<uint4*>(z1.p)[i] = zero;
  for (uint64_t i = t0; i < z2.n16; i += stride) static_cast<uint4*>(z2.p)[i] = zero;
}

// ---------------------------------------------------------------------------
// host-side launchers (called by the engine)
// ---------------------------------------------------------------------------
size_t sieve_smem_bytes(uint32_t seg_bytes, uint32_t /*threads*/) {
  // segment, gap histogram copies, warp records (room for 32 warps), byte
  // histogram copies, byte table
  return (size_t)seg_bytes + sizeof(uint32_t) * kSmemHistCopies * kSmemStride +
         sizeof(WarpRec) * (kMaxThreads / 32) + sizeof(uint32_t) * kSmemHistCopies * kByteValues + kByteValues;
}

size_t sieve_static_smem_bytes() {
  cudaFuncAttributes a{};
  return cudaFuncGetAttributes(&a, sieve_segments_kernel) == cudaSuccess ? a.sharedSizeBytes : 1024;
}

cudaError_t launch_sieve(const SieveParams& prm, uint32_t grid, uint32_t threads,
                         cudaStream_t stream) {
  const size_t smem = sieve_smem_bytes(prm.seg_bytes, threads);
  // the attribute is per device: raised once per (device, size), outside
  // stream capture (plans raise it before they capture)
  static AttrCache attr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int rc = attr.ensure(dev, smem, [](size_t n) {
    return (int)cudaFuncSetAttribute(sieve_segments_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  });
  if (rc) return (cudaError_t)rc;
  if (grid == 0) return cudaSuccess;
  sieve_segments_kernel<<<grid, threads, smem, stream>>>(prm);
  return cudaGetLastError();
}

cudaError_t launch_solo(const SieveParams& prm, uint32_t threads, cudaStream_t stream) {
  const size_t smem = std::max(sieve_smem_bytes(prm.seg_bytes, threads), sizeof(uint32_t) * (size_t)kFinalWords);
  static AttrCache attr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int rc = attr.ensure(dev, smem, [](size_t n) {
    return (int)cudaFuncSetAttribute(solo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  });
  if (rc) return (cudaError_t)rc;
  solo_kernel<<<(uint32_t)prm.solo.nseg * prm.slices, threads, smem, stream>>>(prm);
  return cudaGetLastError();
}

cudaError_t launch_lone(const SieveParams& prm, uint32_t grid, uint32_t threads, cudaStream_t stream) {
  const size_t smem = std::max(sieve_smem_bytes(prm.seg_bytes, threads), sizeof(uint32_t) * (size_t)kFinalWords);
  const bool gaps = (prm.solo.rflags & kReqGaps) != 0;
  static AttrCache attr, attr_count;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int rc = gaps ? attr.ensure(dev, smem, [](size_t n) {
    return (int)cudaFuncSetAttribute(lone_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  }) : attr_count.ensure(dev, smem, [](size_t n) {
    return (int)cudaFuncSetAttribute(lone_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  });
  if (rc) return (cudaError_t)rc;
  if (gaps) lone_kernel<<<grid, threads, smem, stream>>>(prm);
  else lone_count_kernel<<<grid, threads, smem, stream>>>(prm);
  return cudaGetLastError();
}

cudaError_t launch_combine(const BatchHdr* hdr, const ReqSpan* spans, const uint32_t* apos,
                           const ReqResult* ares, ReqResult* out, uint32_t grid, cudaStream_t stream) {
  if (grid == 0) return cudaSuccess;
  combine_kernel<<<grid, 256, 0, stream>>>(hdr, spans, apos, ares, out);
  return cudaGetLastError();
}

cudaError_t launch_zero(ZeroSpan z0, ZeroSpan z1, ZeroSpan z2, uint32_t max_grid, cudaStream_t stream) {
  const uint64_t n = std::max(z0.n16, std::max(z1.n16, z2.n16));
  if (n == 0) return cudaSuccess;
  const uint32_t grid = (uint32_t)std::min<uint64_t>((n + 255) / 256, max_grid);
  zero_kernel<<<grid, 256, 0, stream>>>(z0, z1, z2);
  return cudaGetLastError();
}

// the attribute is per device, as in launch_sieve
static cudaError_t fill_attributes() {
  static AttrCache attr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  return (cudaError_t)attr.ensure(dev, sizeof(FillShared), [](size_t n) {
    return (int)cudaFuncSetAttribute(bucket_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  });
}

cudaError_t bucket_fill_ctas_per_sm(uint32_t* out) {
  if (cudaError_t e = fill_attributes()) return e;
  int n = 0;
  if (cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, bucket_fill_kernel, kFillPrimes,
                                                                    sizeof(FillShared)))
    return e;
  *out = n < 1 ? 1u : (uint32_t)n;
  return cudaSuccess;
}

cudaError_t launch_bucket_fill(const FillParams& fp, uint32_t grid, cudaStream_t stream) {
  if (cudaError_t e = fill_attributes()) return e;
  if (grid == 0) return cudaSuccess;
  bucket_fill_kernel<<<grid, kFillPrimes, sizeof(FillShared), stream>>>(fp);
  return cudaGetLastError();
}

cudaError_t launch_finalize(const ReqDesc* reqs, const BatchHdr* hdr, const SegRec* segs,
                            ReqAccum* acc, LargeGapRec* large, unsigned int* n_large,
                            uint32_t large_cap, ReqResult* out, uint32_t grid,
                            cudaStream_t stream) {
  if (grid == 0) return cudaSuccess;
  finalize_kernel<<<grid, grid == 1 ? 1024 : 256, 0, stream>>>(reqs, hdr, segs, acc, large, n_large, large_cap, out);
  return cudaGetLastError();
}

}  // namespace vg
