// Group form of the classification: reads that the dual-strand warp tiers do not take (over kLeanQ
// bases, or more postings than they hold) and every read of the plain form. A block takes a read;
// its two halves of H threads take one strand each, side by side, and synchronise on a named
// barrier each; a strand that does not fit its half's share of the shared memory makes the whole
// block take the strands in turn with all of it. What does not fit then goes to a second class of block
// (RestSmem), and what that does not hold to the next tier.
//
// The strand's bases are hashed from global memory (a seed's window is five aligned words), so
// shared memory holds postings only, 8 bytes each plus a 2-byte index, in seed order.
//   links              a posting is linked when its reference also has a posting under the found seed
//                      before its own (found indices f and f - 1, Analyser.cpp:2057-2115). A reference
//                      with no linked posting has no occurrence run of 2 and so no diagonal run of 2
//                      (one diagonal, consecutive seeds), which a candidate needs (:2402): only
//                      references with a link matter, and a strand without any is done. The search
//                      goes through the previous seed's bucket from just before the posting's own
//                      place in its bucket: copies of a repeat keep their order from bucket to bucket,
//                      so they meet in a few comparisons; buckets of random hits are one or two long. The
//                      worst, neighbouring buckets of 2,000 (4,000) postings with no reference in common,
//                      takes 2.2 (9.1) us a read in a batch of 1,000; the global-memory tier 11 (26) us.
//   occurrence filter  per linked reference a bitmap of the found indices where it occurs; its longest
//                      run of ones is occMax; references with max(2, hs - 1) or more stay (:2115)
//   order              the kept postings by reference, each one's in seed order (a posting's place is
//                      the number of ones before its found index in the bitmap): that is (position,
//                      seed) order unless a stray hit interferes, which is checked; then each
//                      reference's postings are ranked by a warp, or, when one has more than kRankMax,
//                      sorted by the block
//   runs, walks        run starts as a bit mask; a run's length reaches back to the last start
//                      (:2337-2490); a thread walks a run end's head and tail and adds its length,
//                      triangle and covered bases to its reference's sums and bitmap (MatrixCPU.cpp:18-214)
//
// What bounds it: latency, of the slots' DRAM pages and of some twenty group-wide steps a strand, with
// eight strands in flight per SM (10,000 reads of 1-20 kb: issue slots 37% used, DRAM 1.7 TB/s; the
// barriers hold the warps longest). Measured on a B200 against the form before it (two sizes of block, one strand at a time on 256 threads, a hash set of (refID, found
// index) pairs, then a block per SM with two full sorts for what they left): 20,000 reads of 1-20 kb
// on 5,000 references 5.86 -> 1.66 ms, 200,000 reads of 250 bases on references sharing repeats (36
// copies of a segment) 4.50 -> 1.69 ms, 4,001 reads of 75 bases to 20 kb from host memory 1.28 -> 0.65 ms.
#pragma once
#include "mg_lean.cuh"

namespace mg {

constexpr uint32_t kLgEmpty = 0xFFFFFFFFu;
constexpr uint32_t kLgKeepAll = 64;       // see long_strand's `keeps_all`
constexpr uint32_t kRankMax = 128;        // postings of a reference that a warp ranks
constexpr uint32_t kNone = 0xFFFFu;       // no link (long_strand, step 2)
constexpr uint32_t kRunEnd = 0x8000u;     // a run's length in place of its last posting's link

// Shared memory of a block: two halves of H threads, each with room for E postings, NS seeds and RM
// kept references per strand (RT table slots); the whole block uses both shares of the postings and
// seeds for one strand. Rest: the class for what the others leave, which has the keep rule ahead of the
// table on the whole block (keep_by_runs).
template <int H_, int E_, int NS_, int RT_, int RM_, bool Rest_ = false>
struct alignas(16) LongSm {
  static constexpr int H = H_, E = E_, NS = NS_, RT = RT_, RM = RM_;
  static constexpr bool Rest = Rest_;
  static constexpr uint32_t kIdBits = RM > 126 ? 8 : 7, kNoId = (1u << kIdBits) - 1;  // a reference's order of insertion
  static constexpr int NSP = NS + 1, NW = (NS + 31) / 32, BW = E / 64;  // BW: words of E / 2 bits
  struct Half {
    unsigned long long sumr[RM];  // sums of a candidate's runs; before: the linked references' best
    uint32_t sumc[RM];            // runs (sumr), their refIDs (sumc), the ranges' bounds
    uint32_t segmax[RM];          // longest diagonal run of a kept reference; then its covered bases
    uint32_t kref[RM];            // kept references by refID
    uint32_t rt[RT];              // table of linked references
    uint8_t rid[RT];              // a slot's reference: order of insertion
    uint16_t cnt[RM];             // kept postings (by order of insertion)
    uint8_t rk[RM], kid[RM];      // rank among the kept references (kNoId: none) by order of insertion, and back
  };
  uint32_t rs[2 * E];  // refID << 11 | seed
  uint32_t ps[2 * E];  // reference position
  // per share: sorted order (E / 2), kept postings (E / 2), first posting and postings of each seed
  // (NSP each); the seeds with more than a slot's postings and then the linked references' bitmaps lie
  // over the first two, the candidates' coverage over the last two
  uint16_t pool[2 * (E + 2 * NSP)];
  uint32_t fm[2 * NW];  // found seeds
  uint16_t fp[2 * NW];  // found seeds before each word of fm
  uint32_t bk[2 * BW];  // starts of diagonal runs
  uint32_t red[2][2][2 * H / 32];
  uint32_t ne[2], nx[2], n_rt[2], over[2], dup[2], n_ends[2], n_out[2], keeps_all;
  float hi[2];
  int status[2];
  uint32_t cand_at, ahead;
  Half h[2];
  mg_candidate cb[2][RM];
  uint8_t comp[256];  // complement(upper(byte)), 0 where there is none
  static_assert(E % 64 == 0 && E % 4 == 0 && NSP % 2 == 0 && 2 * E <= 8192 && NS <= E / 2 && 2 * NS <= 2047 && RM < kNoId && 3 * RM <= E / 2 && (!Rest || 2 * E / 32 <= RT), "sizes");
  static_assert(RM * 8 >= 2 * (RM + 1), "tables over the sums");
};

// The classes of reads: the batched forms' tier (reads to 20,480 bases and 4,096 postings per strand)
// with four blocks per SM, and the plain form's kernel, one block of two warps per read, up to 15 per
// SM (11,000 reads of 150 bases: 97 us; a block of 256 threads per read with two bitonic sorts per
// strand, the form before, 1,010 us; room for 256 postings instead of 512 makes no difference). Then
// what the first leaves: two blocks per SM, 8,192 postings (4,096 kept), 2,046 seeds (reads of 20,480
// bases down to k = 20) and 224 kept references, whatever the number of linked ones.
using LongSmem = LongSm<128, 2048, 703, 256, 88>;
using PlainSmem = LongSm<32, 512, 255, 64, 32>;
using RestSmem = LongSm<128, 4096, 1023, 512, 224, true>;
constexpr uint32_t kLgQ = 20480;
static_assert(4 * (sizeof(LongSmem) + 1024) <= 233472, "four blocks per SM");
static_assert(2 * (sizeof(RestSmem) + 1024) <= 233472, "two blocks per SM");

__device__ __forceinline__ uint32_t lg_mix(uint32_t x) { return (x * 2654435761u) ^ (x >> 15); }

// Barrier over a group: the block (bar 0), or half bar - 1 of H threads. The ids are immediates: with
// an id in a register a block is given all 16 barriers, and four blocks fill the SM.
template <int H>
__device__ __forceinline__ void lg_sync(int bar) {
  if (bar == 0)
    asm volatile("bar.sync 0;" ::: "memory");
  else if (H == 32)
    __syncwarp();
  else if (bar == 1)
    asm volatile("bar.sync 1, %0;" ::"n"(H) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"n"(H) : "memory");
}

// hash28_dev of the 17-byte window a..a+16 of an ACGT read in upper case (strand 0), or of its
// reverse complement (strand 1). The five aligned words loaded each hold a byte of the window
// ((a & 3) + 17 <= 20).
__device__ __forceinline__ uint32_t hash17_acgt(const uint8_t* a, int strand) {
  const uint32_t* w = (const uint32_t*)((uintptr_t)a & ~(uintptr_t)3);
  const uint32_t sh = ((uint32_t)(uintptr_t)a & 3u) * 8u;
  const uint32_t x0 = __ldg(w), x1 = __ldg(w + 1), x2 = __ldg(w + 2), x3 = __ldg(w + 3), x4 = __ldg(w + 4);
  uint32_t y[5] = {__funnelshift_r(x0, x1, sh), __funnelshift_r(x1, x2, sh), __funnelshift_r(x2, x3, sh),
                   __funnelshift_r(x3, x4, sh), x4 >> sh};
#pragma unroll
  for (int i = 0; i < 5; i++) y[i] = upper4(y[i]);
  uint32_t h = 2166136261u;
  if (strand == 0) {
#pragma unroll
    for (int i = 0; i < 17; i++) h = (h * 16777619u) ^ ((y[i >> 2] >> (8 * (i & 3))) & 0xFFu);
  } else {
#pragma unroll
    for (int i = 0; i < 5; i++) y[i] = comp4(y[i]);
#pragma unroll
    for (int i = 16; i >= 0; i--) h = (h * 16777619u) ^ ((y[i >> 2] >> (8 * (i & 3))) & 0xFFu);
  }
  return ((h >> 28) ^ h) & 0x0FFFFFFFu;
}

// n (1 to 8) bytes p..p+n-1 as a little-endian number, zeros above; only aligned words that hold one
// of them are read.
__device__ __forceinline__ uint64_t load_bytes(const uint8_t* p, uint32_t n) {
  const uintptr_t a = (uintptr_t)p;
  const uint32_t* w = (const uint32_t*)(a & ~(uintptr_t)3);
  const uint32_t o = (uint32_t)(a & 3u), e = o + n;
  const uint32_t w0 = w[0], w1 = e > 4 ? w[1] : 0u, w2 = e > 8 ? w[2] : 0u;
  const uint64_t v = ((uint64_t)__funnelshift_r(w1, w2, 8 * o) << 32) | __funnelshift_r(w0, w1, 8 * o);
  return v & (~0ull >> (64 - 8 * n));
}
// complement(upper(byte)) of four bytes, by table for those outside ACGT.
__device__ __forceinline__ uint32_t comp_any4(uint32_t w, const uint8_t* comp) {
  const uint32_t u = upper4(w);
  if (acgt4(u)) return comp4(u);
  return (uint32_t)comp[u & 0xFFu] | ((uint32_t)comp[(u >> 8) & 0xFFu] << 8) |
         ((uint32_t)comp[(u >> 16) & 0xFFu] << 16) | ((uint32_t)comp[u >> 24] << 24);
}

// The head and tail walks of a run (head_walk, tail_walk) on the strand's bases, read from the batch
// (raw, L bytes; the reverse complement backwards, through the complement table). The run: reference
// position of its first seed sr and reference end of its last seed lr, first query base sq and query
// end lq. Returns the run's query start << 16 | its extended length T, or 0 when T < k.
// Both walks advance eight bytes per round trip to memory, with the loads of a step (query and
// reference, head and tail) in flight together: most walks end in the first or second step, and a
// step's cost is the reference's DRAM latency, once for both. Sixteen bytes a step cost more in
// registers and instructions than the round trips they save (the finishing pass of 1 M reads of
// 75-300 bases: 278 us, against 226 us at eight).
__device__ __forceinline__ uint32_t walk_run(const DevIndex& ix, const uint8_t* comp, const uint8_t* raw, uint32_t L,
                                             int strand, uint32_t ref, uint32_t sr, uint32_t lr, uint32_t sq,
                                             uint32_t lq, uint32_t k) {
  const uint8_t* rs = ix.bases + ix.ref_off[ref];
  const uint32_t rlen = ix.ref_len[ref];
  // strand bases p..p+n-1 (1 <= n <= 8) as a number, base p in the low byte
  auto query = [&](uint32_t p, uint32_t n) -> uint64_t {
    if (!strand) {
      const uint64_t v = load_bytes(raw + p, n);
      return ((uint64_t)upper4((uint32_t)(v >> 32)) << 32) | upper4((uint32_t)v);
    }
    const uint64_t v = load_bytes(raw + (L - p - n), n);  // base p is the last byte of these
    const uint32_t lo = __byte_perm((uint32_t)v, 0, 0x0123), hi = __byte_perm((uint32_t)(v >> 32), 0, 0x0123);
    const uint64_t m = (((uint64_t)lo << 32) | hi) >> (64 - 8 * n);
    // zeros above base p+n-1 map to the table's entry of 0: zero, as on the reference's side
    return ((uint64_t)comp_any4((uint32_t)(m >> 32), comp) << 32) | comp_any4((uint32_t)m, comp);
  };
  const uint32_t tl = lq < L && lr < rlen ? min(min(rlen - lr, k), L - lq) : 0u;  // most that the tail takes
  const uint32_t hz = min(sr, k);
  const uint32_t hl = sq != 0 && hz != 0 ? min(sq - 1, hz - 1) : 0u;  // most that the head takes
  uint32_t tail = 0, head = 0;
  bool t_on = tl > 0, h_on = hl > 0;
#pragma unroll 1
  while (t_on || h_on) {  // a walk that goes on takes at least one base
    const uint32_t tn = t_on ? min(8u, tl - tail) : 0u, hn = h_on ? min(8u, hl - head) : 0u;
    uint64_t tq = 0, tr = 0, hq = 0, hr = 0;
    if (tn) tr = load_bytes(rs + lr + tail, tn);
    if (hn) hr = load_bytes(rs + (sr - head - hn + 1), hn);
    if (tn) tq = query(lq + tail, tn);
    if (hn) hq = query(sq - head - hn, hn);
    if (tn) {
      const uint64_t d = tq ^ tr;
      const uint32_t same = d ? (uint32_t)(__ffsll((long long)d) - 1) >> 3 : tn;
      tail += same;
      t_on = same == tn && tail < tl;
    }
    if (hn) {
      const uint64_t d = (hq ^ hr) << (64 - 8 * hn);  // the walk goes down from the last byte
      const uint32_t same = d ? (uint32_t)__clzll((long long)d) >> 3 : hn;
      head += same;
      h_on = same == hn && head < hl;
    }
  }
  const uint32_t tot = tail + head + (lq - sq);
  return tot >= k ? ((sq - head) << 16) | tot : 0u;
}

// Longest run of ones of a bitmap of nw words (nw <= 64), on a warp; every lane gets it. before[w]
// receives the number of ones in the words before w, *total that of all.
__device__ __forceinline__ uint32_t warp_longest_run(const uint32_t* bm, uint32_t nw, uint16_t* before, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t n0 = 2 * lane < nw ? __popc(bm[2 * lane]) : 0u, n1 = 2 * lane + 1 < nw ? __popc(bm[2 * lane + 1]) : 0u;
  uint32_t x = n0 + n1;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (2 * lane < nw) before[2 * lane] = (uint16_t)(x - n0 - n1);
  if (2 * lane + 1 < nw) before[2 * lane + 1] = (uint16_t)(x - n1);
  *total = __shfl_sync(0xffffffffu, x, 31);
  // a span's (bits, leading ones, trailing ones, longest run); two words a lane, then lanes combined
  uint32_t len = 0, pre = 0, suf = 0, best = 0;
  auto join = [&](uint32_t l2, uint32_t p2, uint32_t s2, uint32_t b2) {  // this span, then the other
    best = max(max(best, b2), suf + p2);
    pre = pre == len ? len + p2 : pre;
    suf = s2 == l2 ? l2 + suf : s2;
    len += l2;
  };
#pragma unroll
  for (uint32_t u = 0; u < 2; u++) {
    const uint32_t w = 2 * lane + u;
    if (w < nw) {
      const uint32_t m = bm[w];
      join(32, (uint32_t)__ffs(~m) ? (uint32_t)__ffs(~m) - 1u : 32u, (uint32_t)__clz(~m), (uint32_t)longest_run(m));
    }
  }
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t l2 = __shfl_down_sync(0xffffffffu, len, o), p2 = __shfl_down_sync(0xffffffffu, pre, o);
    const uint32_t s2 = __shfl_down_sync(0xffffffffu, suf, o), b2 = __shfl_down_sync(0xffffffffu, best, o);
    if (lane + o < 32) join(l2, p2, s2, b2);
  }
  return __shfl_sync(0xffffffffu, best, 0);
}

// A posting under the found seed before posting i's (x = rs[i]) with its reference; kNone: there is none
// (or !on). The warp reconverges.
__device__ __forceinline__ uint32_t link_of(const uint32_t* rs, const uint16_t* st, const uint16_t* cn,
                                            const uint32_t* fm, uint32_t i, uint32_t x, bool on) {
  const uint32_t j = x & 2047u;
  uint32_t w = j >> 5, m = on ? fm[w] & ((1u << (j & 31u)) - 1u) : 0u;
#pragma unroll 1
  while (!m && w && on) m = fm[--w];
  uint32_t a = 0, c = 0, t = 0, at = kNone;
  if (m) {
    const uint32_t pj = w * 32 + 31 - __clz(m);
    a = st[pj];
    c = cn[pj];
    t = i - st[j];  // a stray hit in either bucket shifts the copies by one
    t = t < 2 ? 0 : t - 2;
    if (t >= c) t = 0;
  }
#pragma unroll 1
  for (uint32_t n = 0; n < c && at == kNone; n++) {
    if ((rs[a + t] ^ x) < 2048u) at = a + t;
    if (++t == c) t = 0;
  }
  __syncwarp();
  return at;
}

// A reference (on) into the strand's table, with the next number; S.over: more than RM. The warp
// reconverges.
template <class SM>
__device__ __forceinline__ void add_ref(SM& S, int half, uint32_t ref, bool on) {
  typename SM::Half& T = S.h[half];
  uint32_t s = lg_mix(ref) & (SM::RT - 1), left = on ? (uint32_t)SM::RT : 0u;  // each slot once
#pragma unroll 1
  while (left) {
    uint32_t old = *(volatile uint32_t*)&T.rt[s];
    if (old == kLgEmpty && !*(volatile uint32_t*)&S.over[half]) {  // the table stays free to end probes
      old = atomicCAS(&T.rt[s], kLgEmpty, ref);
      if (old == kLgEmpty) {
        const uint32_t id = atomicAdd(&S.n_rt[half], 1u);
        if (id < (uint32_t)SM::RM) {
          T.rid[s] = (uint8_t)id;
          T.sumc[id] = ref;
        } else {
          S.over[half] = 1;
        }
      }
    }
    left = old == ref || old == kLgEmpty ? 0u : left - 1;
    s = (s + 1) & (SM::RT - 1);
  }
  __syncwarp();
}

// The keep rule ahead of the table, on the whole block, for a strand of ne postings with more linked
// references than the table or the bitmaps hold: most are copies of a repeat that the rule drops beside
// the strand's own reference. A posting's links, followed back, are the occurrence run that ends at it;
// only references with a run long enough go to the table. Returns how many (above RM: too many), the
// longest run at each of them in `best`. Reads of 250 bases on the flank of a segment with 100 (200)
// copies and inside it, 10,000 each: 1.2 (3.0) and 2.2 (3.7) ms; through the global-memory tier, which
// took what LongSmem does not hold, 28 (67) and 112 (237) ms. 2,000 reads of 16 kb across several
// segments of 30 copies: 1.0 ms, 28.5 ms so. Not in the first class: there the call's registers
// spill in the common strands (20,000 reads of 1-20 kb: 1.70 ms, 1.67 ms without).
template <class SM>
__device__ __forceinline__ uint32_t keep_by_runs(SM& S, uint32_t ne) {
  constexpr uint32_t G = 2 * SM::H, kE = 2 * SM::E, kRT = SM::RT;
  const uint32_t tid = threadIdx.x;
  const uint32_t* rs = S.rs;
  const uint16_t* st = S.pool + kE;
  const uint16_t* cn = st + 2 * SM::NSP;
  typename SM::Half& T = S.h[0];
  uint16_t* ln = S.pool;     // each posting's link, over sx and kl; then at a run's last posting its length
  uint32_t* on = S.h[1].rt;  // postings that a run goes on from, a bit each (the other half's table is free)
  uint16_t* best = reinterpret_cast<uint16_t*>(T.sumr);
  __syncthreads();  // every thread has read the table's count
#pragma unroll 1
  for (uint32_t i = tid; i < kE / 32; i += G) on[i] = 0;
#pragma unroll 1
  for (uint32_t i = tid; i < kRT; i += G) T.rt[i] = kLgEmpty;
  if (tid == 0) {
    S.n_rt[0] = 0;
    S.over[0] = 0;
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < ne; i0 += G) {
    const uint32_t i = i0 + tid, l = link_of(rs, st, cn, S.fm, i, i < ne ? rs[i] : 0u, i < ne);
    if (i < ne) ln[i] = (uint16_t)l;
    if (l != kNone) atomicOr(&on[l >> 5], 1u << (l & 31u));
  }
  __syncthreads();
  uint32_t hs = 0;
#pragma unroll 1
  for (uint32_t i = tid; i < ne; i += G) {
    uint32_t p = ln[i], len = 1;
    if (p == kNone || ((on[i >> 5] >> (i & 31u)) & 1u)) continue;
#pragma unroll 1
    for (; p != kNone; p = ln[p]) len++;  // fewer steps than seeds: a link leads to an earlier one
    ln[i] = (uint16_t)(kRunEnd | len);    // no other run passes here
    hs = max(hs, len);
  }
  hs = __reduce_max_sync(0xFFFFFFFFu, hs);
  if ((tid & 31u) == 0) S.red[0][0][tid >> 5] = hs;
  __syncthreads();
#pragma unroll 1
  for (uint32_t w = 0; w < G / 32; w++) hs = max(hs, S.red[0][0][w]);
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < ne; i0 += G) {
    const uint32_t i = i0 + tid, v = i < ne ? ln[i] : kNone;
    add_ref(S, 0, i < ne ? rs[i] >> 11 : 0u, v != kNone && (v & kRunEnd) && (v & (kRunEnd - 1)) >= max(2u, hs - 1));
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t id = tid; id < (uint32_t)SM::RM; id += G) best[id] = (uint16_t)hs;
  return S.n_rt[0];
}

// One strand of a read (raw bytes, L of them, no byte without a complement; acgt: all of them letters
// of ACGT in either case) on G threads with room for kE postings and kNS seeds: half `half` of the
// block (G = H), or all of it (whole: G = 2 H, half 0). On kStrandOk the strand's *n_out scored candidates
// are in cb, in ascending refID, and *highest is its HighestScore. kStrandOverflow: it does not fit.
// *keeps_all: the keep rule keeps every reference with a posting (hs = 2), the strand has more than
// kLgKeepAll postings and a diagonal run. Only counted (mg_last_tier_counts): such a strand has its
// candidates among the linked references like any other.
// One instance for both, and loops kept rolled: the code runs through once per strand, so that its
// size is paid in instruction fetches. With an instance each and the compiler's unrolling it was
// 355 KB, and four blocks per SM slowed each other from 64,000 to 119,000 cycles a read (20,000 reads
// of 1-20 kb: 2.25 ms); at 98 KB, from 64,000 to 84,000 (1.75 ms).
template <class SM>
__device__ __forceinline__ int long_strand(const DevIndex& ix, const uint8_t* raw, uint32_t L, int strand, bool acgt,
                                           SM& S, bool whole, int half, mg_candidate* cb, int* err, uint32_t* n_out,
                                           float* highest, bool* keeps_all) {
  constexpr uint32_t kRT = SM::RT, kRM = SM::RM;
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t sh = whole ? 1u : 0u;  // twice the threads and the room
  const uint32_t G = SM::H << sh, kE = SM::E << sh, kNS = SM::NS << sh, kNW = SM::NW << sh, kW = G / 32;
  const int bar = whole ? 0 : 1 + half;
  const uint32_t tid = whole ? threadIdx.x : threadIdx.x - half * SM::H;
  const uint32_t lane = tid & 31u, warp = tid >> 5;
  const uint32_t k = (uint32_t)ix.k, step = (uint32_t)ix.step;
  uint32_t* rs = S.rs + half * SM::E;
  uint32_t* ps = S.ps + half * SM::E;
  uint16_t* sx = S.pool + half * (SM::E + 2 * SM::NSP);  // sorted order of the kept postings
  uint16_t* kl = sx + kE / 2;                        // the kept postings
  uint16_t* st = sx + kE;                            // first posting of each seed
  uint16_t* cn = st + (SM::NSP << sh);               // its number of postings
  uint32_t* fm = S.fm + half * SM::NW;
  uint16_t* fp = S.fp + half * SM::NW;
  uint32_t* bk = S.bk + half * SM::BW;
  typename SM::Half& T = S.h[half];
  uint32_t* iref = T.sumc;                                      // linked references in order of insertion
  uint16_t* best = reinterpret_cast<uint16_t*>(T.sumr);         // their longest occurrence runs
  uint16_t* boff = reinterpret_cast<uint16_t*>(T.sumr);         // then: the kept references' ranges
  uint32_t* bfill = T.sumc;                                     // (counts, then fill)
  uint32_t(*red)[2 * SM::H / 32] = S.red[half];
  *n_out = 0;
  *highest = -1.0f;
  if (L <= k) return kStrandOk;
  const uint32_t ns = (L - k + step - 1) / step;
  const uint32_t kCovWords = SM::NSP << sh;  // over st and cn
  if (ns > kNS || (L + 31) / 32 > kCovWords) return kStrandOverflow;
#pragma unroll 1
  for (uint32_t i = tid; i < kRT; i += G) T.rt[i] = kLgEmpty;
  if (tid == 0) {
    S.n_rt[half] = 0;
    S.over[half] = 0;
    S.ne[half] = 0;
    S.nx[half] = 0;
  }
  lg_sync<SM::H>(bar);
  // 1. seeds, probe, postings. A seed's slot is read once (random DRAM sectors bound this step: with
  //    a prefetch, a pass over the counts and one over the postings the tier took 1.70 ms for 20,000 reads
  //    of 1-20 kb, 1.58 ms so), two seeds in flight per thread; a warp takes room for its seeds' postings from
  //    the group's cursor, so nothing waits for another warp and the postings lie in no order.
  uint16_t* xl = kl;                              // seeds with more than a slot's postings (at most kE / 8)
  uint32_t* xo = reinterpret_cast<uint32_t*>(sx);  // their first posting in the index
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < ns; j0 += 2 * G) {
    uint4 v0[2], v1[2];
    uint32_t cnt[2], o0[2], hash[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t j = j0 + u * G + tid, p = j * step;
      v0[u] = v1[u] = make_uint4(0u, 0u, 0u, 0u);
      cnt[u] = o0[u] = 0;
      hash[u] = kLgEmpty;
      if (j < ns) {
        uint32_t h;
        if (acgt && ix.hlen == 17) {
          h = hash17_acgt(raw + (strand ? L - 17 - p : p), strand);
        } else {
          h = 2166136261u;
#pragma unroll 1
          for (int t = 0; t < ix.hlen; t++) {
            const uint8_t c = strand ? S.comp[raw[L - 1 - p - t]] : upper_dev(raw[p + t]);
            h = (h * 16777619u) ^ c;
          }
          h = ((h >> 28) ^ h) & 0x0FFFFFFFu;
        }
        hash[u] = h;
        if (ix.slots) {
          const uint4* sl = ix.slots + (size_t)h * kSlotVecs;
          v0[u] = __ldg(sl);
          v1[u] = __ldg(sl + 1);
        } else {
          o0[u] = __ldg(ix.dir + h);
          cnt[u] = __ldg(ix.dir + h + 1) - o0[u];
        }
      }
    }
#pragma unroll 1
    for (int u = 0; u < 2; u++) {
      const uint32_t jw = j0 + u * G + warp * 32;  // the warp's first seed
      if (jw >= ns) break;                         // warp-uniform
      const uint32_t j = jw + lane, h = u ? hash[1] : hash[0];
      const uint4 a = u ? v0[1] : v0[0], b = u ? v1[1] : v1[0];
      uint4 c = make_uint4(0u, 0u, 0u, 0u), d = c;
      const uint32_t full = ix.slots ? a.x : u ? cnt[1] : cnt[0], o = ix.slots ? a.y : u ? o0[1] : o0[0];
      if (ix.slots && full > 3) {
        const uint4* sl = ix.slots + (size_t)h * kSlotVecs;
        c = __ldg(sl + 2);
        d = __ldg(sl + 3);
      }
      const uint32_t fb = __ballot_sync(FULL, full > 0 || h == ix.empty_hash);
      const uint32_t n = min(full, kE + 1);
      uint32_t x = n;
      for (int t = 1; t < 32; t <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, t);
        if (lane >= (uint32_t)t) x += y;
      }
      const uint32_t tot = __shfl_sync(FULL, x, 31);
      uint32_t base = 0;
      if (lane == 0) {
        fm[jw >> 5] = fb;
        base = atomicAdd(&S.ne[half], tot);  // at most kNS (kE + 1) over a strand: fits 32 bits
      }
      base = __shfl_sync(FULL, base, 0);
      if (base + tot > kE) continue;  // warp-uniform; the strand overflows, seen below
      const uint32_t e = base + x - n;
      if (j < ns) {
        st[j] = (uint16_t)e;
        cn[j] = (uint16_t)n;
      }
      auto put = [&](uint32_t t, uint32_t ref, uint32_t pos) {
        if (t < n) {
          rs[e + t] = (ref << 11) | j;
          ps[e + t] = pos;
        }
      };
      if (ix.slots) {
        put(0, a.z, a.w);
        put(1, b.x, b.y);
        put(2, b.z, b.w);
        put(3, c.x, c.y);
        put(4, c.z, c.w);
        put(5, d.x, d.y);
        put(6, d.z, d.w);
      } else {
#pragma unroll 1
        for (uint32_t t = 0; t < (uint32_t)kSlotPosts && t < n; t++) {
          const uint2 v = __ldg(ix.post + o + t);
          put(t, v.x, v.y);
        }
      }
      if (n > (uint32_t)kSlotPosts) {  // at most kE / 8 seeds of the strand
        const uint32_t i = atomicAdd(&S.nx[half], 1u);
        xl[i] = (uint16_t)j;
        xo[i] = o;
      }
    }
  }
  lg_sync<SM::H>(bar);
  const uint32_t ne = S.ne[half], nx = S.nx[half];
  if (ne > kE) return kStrandOverflow;  // group-uniform
  if (ne == 0) return kStrandOk;        // nothing found: the reference skips the strand
  if (warp == kW - 1) {  // found seeds before each word: at most 64 words, two a lane
    const uint32_t nw = (ns + 31) >> 5;
    const uint32_t c0 = 2 * lane < nw ? __popc(fm[2 * lane]) : 0u, c1 = 2 * lane + 1 < nw ? __popc(fm[2 * lane + 1]) : 0u;
    uint32_t f = c0 + c1;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, f, o);
      if (lane >= (uint32_t)o) f += y;
    }
    if (2 * lane < nw) fp[2 * lane] = (uint16_t)(f - c0 - c1);
    if (2 * lane + 1 < nw) fp[2 * lane + 1] = (uint16_t)(f - c1);
  }
  // the postings past the slots', a warp per eight seeds with four lanes on each
#pragma unroll 1
  for (uint32_t i0 = 8 * warp; i0 < nx; i0 += 8 * kW) {
    const uint32_t i = i0 + (lane >> 2);
    if (i < nx) {
      const uint32_t j = xl[i], e = st[j], n = cn[j], o = xo[i];
#pragma unroll 4
      for (uint32_t t = (uint32_t)kSlotPosts + (lane & 3u); t < n; t += 4) {
        const uint2 v = __ldg(ix.post + o + t);
        rs[e + t] = (v.x << 11) | j;
        ps[e + t] = v.y;
      }
    }
  }
  lg_sync<SM::H>(bar);
  const uint32_t fw = (ns - 1) >> 5;
  const uint32_t nf = fp[fw] + __popc(fm[fw]), nfw = (nf + 31) >> 5;
  // 2. the linked references (the warps reconverge between the two searches)
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < ne; i0 += G) {
    const uint32_t i = i0 + tid, x = i < ne ? rs[i] : 0u;
    const bool linked = link_of(rs, st, cn, fm, i, x, i < ne) != kNone;
    add_ref(S, half, x >> 11, linked);
  }
  lg_sync<SM::H>(bar);
  uint32_t R = S.n_rt[half];
  if (R == 0) return kStrandOk;  // no reference at two found seeds in a row: no candidate
  // the bitmaps (R of nfw words) and, behind them, the ones before each word (R nfw half-words) lie over sx
  if (R > kRM || 3 * R * nfw > kE / 2) {
    if (!SM::Rest || !whole) return kStrandOverflow;
    R = keep_by_runs(S, ne);
    if (R > kRM) return kStrandOverflow;
  }
  const bool nobm = SM::Rest && 3 * R * nfw > kE / 2;  // no room for bitmaps: the kept postings are counted and ranked one by one
  // 3. occurrence filter; from here on the postings hold, in place of the refID, its reference's order
  //    of insertion (kNoId: not linked, not needed any more)
  constexpr uint32_t kNoId = SM::kNoId, kPlace = 11 + SM::kIdBits;  // id << 11 | seed, and a place above it
  uint32_t* bm = reinterpret_cast<uint32_t*>(sx);
  uint16_t* pw = sx + 2 * R * nfw;
#pragma unroll 1
  for (uint32_t i = tid; i < R * nfw && !nobm; i += G) bm[i] = 0;
  if (tid == 0) S.dup[half] = nobm;
  lg_sync<SM::H>(bar);
  const uint32_t only = iref[0];
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < ne; i0 += G) {
    const uint32_t i = i0 + tid, x = i < ne ? rs[i] : kLgEmpty, ref = x >> 11, j = x & 2047u;
    uint32_t id = kNoId;
    if (R == 1) {
      if (i < ne && ref == only) id = 0;
    } else {
      uint32_t s = lg_mix(ref) & (kRT - 1), left = i < ne ? kRT : 0u;  // the table has free slots: R <= kRM < kRT
#pragma unroll 1
      while (left) {
        const uint32_t v = T.rt[s];
        if (v == ref) id = T.rid[s];
        left = v == ref || v == kLgEmpty ? 0u : left - 1;
        s = (s + 1) & (kRT - 1);
      }
    }
    __syncwarp();
    if (i < ne) {
      rs[i] = (id << 11) | j;
      if (id != kNoId && !nobm) {
        const uint32_t f = fp[j >> 5] + __popc(fm[j >> 5] & ((1u << (j & 31u)) - 1u)), bit = 1u << (f & 31u);
        if (atomicOr(&bm[id * nfw + (f >> 5)], bit) & bit) S.dup[half] = 1;  // twice under one seed
      }
    }
  }
  lg_sync<SM::H>(bar);
  if (nfw == 1) {
#pragma unroll 1
    for (uint32_t id = tid; id < R; id += G) {
      best[id] = (uint16_t)longest_run(bm[id]);
      T.cnt[id] = (uint16_t)__popc(bm[id]);
      pw[id] = 0;
    }
  } else if (!nobm) {
#pragma unroll 1
    for (uint32_t id = warp; id < R; id += kW) {
      uint32_t n;
      const uint32_t b = warp_longest_run(bm + id * nfw, nfw, pw + id * nfw, &n);
      if (lane == 0) {
        best[id] = (uint16_t)b;
        T.cnt[id] = (uint16_t)n;
      }
    }
  }
  lg_sync<SM::H>(bar);
  uint32_t hs = 0;
#pragma unroll 1
  for (uint32_t id = lane; id < R; id += 32) hs = max(hs, (uint32_t)best[id]);
  hs = __reduce_max_sync(FULL, hs);
  const uint32_t keep_min = max(2u, hs - 1);  // max(1, hs - 1) (Analyser.cpp:2115), among the linked
  uint32_t nk = 0;  // kept references
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < R; i0 += 32) nk += __popc(__ballot_sync(FULL, i0 + lane < R && best[i0 + lane] >= keep_min));
#pragma unroll 1
  for (uint32_t id = tid; id < R; id += G) {
    uint32_t r = kNoId;
    if (best[id] >= keep_min) {
      const uint32_t ref = iref[id];
      r = 0;
#pragma unroll 4
      for (uint32_t u = 0; u < R; u++) r += (best[u] >= keep_min && iref[u] < ref) ? 1u : 0u;
      T.kref[r] = ref;
      T.kid[r] = (uint8_t)id;
    }
    T.rk[id] = (uint8_t)r;
  }
#pragma unroll 1
  for (uint32_t i = tid; i < kRM; i += G) T.segmax[i] = 0;
  lg_sync<SM::H>(bar);
  auto rank_of = [&](uint32_t x) -> uint32_t { return T.rk[(x >> 11) & kNoId]; };  // of a linked posting
  // 4. the kept postings in (refID, position, seed) order, as indices in sx[0 .. T2)
  auto key_of = [&](uint32_t i) { return ((uint64_t)ps[i] << 11) | (rs[i] & 2047u); };
  uint32_t T2 = 0;
  // a range [a, b) of kept postings ranked by a warp into dst: an entry's place is the number of
  // smaller keys (the keys are distinct)
  auto rank_range = [&](const uint16_t* src, uint16_t* dst, uint32_t a, uint32_t b) {
#pragma unroll 1
    for (uint32_t e0 = a; e0 < b; e0 += 32) {
      const uint32_t e = e0 + lane;
      const uint32_t mine = e < b ? src[e] : 0u;
      const uint64_t key = e < b ? key_of(mine) : 0ull;
      uint32_t r = 0;
#pragma unroll 1
      for (uint32_t f0 = a; f0 < b; f0 += 32) {
        const uint64_t other = f0 + lane < b ? key_of(src[f0 + lane]) : ~0ull;
        const uint32_t n = min(32u, b - f0);
#pragma unroll 4
        for (uint32_t u = 0; u < n; u++) r += __shfl_sync(FULL, other, u) < key ? 1u : 0u;
      }
      if (e < b) dst[a + r] = (uint16_t)mine;
    }
  };
  const bool dup = S.dup[half] != 0;
  uint32_t* badr = bk;  // ranges with postings out of order, a bit each
  if (dup) {  // a reference twice under a seed: the postings are counted one by one
#pragma unroll 1
    for (uint32_t id = tid; id < R; id += G) bfill[id] = 0;
    lg_sync<SM::H>(bar);
#pragma unroll 1
    for (uint32_t i = tid; i < ne; i += G) {  // a posting's place in its range goes beside its id
      const uint32_t x = rs[i];
      if ((x >> 11) != kNoId && rank_of(x) != kNoId) rs[i] = x | (atomicAdd(&bfill[x >> 11], 1u) << kPlace);
    }
    lg_sync<SM::H>(bar);
#pragma unroll 1
    for (uint32_t id = tid; id < R; id += G) T.cnt[id] = (uint16_t)bfill[id];
    lg_sync<SM::H>(bar);
  }
  uint32_t bmax = 0;
#pragma unroll 1
  for (uint32_t b0 = 0; b0 < nk; b0 += 32) {  // every warp: the ranges' starts; warp 0 writes them
    const uint32_t b = b0 + lane, c = b < nk ? T.cnt[T.kid[b]] : 0u;
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (warp == 0 && b < nk) boff[b] = (uint16_t)(T2 + x - c);
    T2 += __shfl_sync(FULL, x, 31);
    bmax = max(bmax, __reduce_max_sync(FULL, c));
  }
  if (T2 > kE / 2) return kStrandOverflow;  // group-uniform
  if (tid == 0) boff[nk] = (uint16_t)T2;
  if (tid < (kRM + 31) / 32) badr[tid] = 0;
  lg_sync<SM::H>(bar);
#pragma unroll 1
  for (uint32_t i = tid; i < ne; i += G) {  // into the ranges, in seed order unless dup
    const uint32_t x = rs[i], id = (x >> 11) & kNoId;
    if (id == kNoId) continue;
    const uint32_t b = T.rk[id];
    if (b == kNoId) continue;
    uint32_t at = x >> kPlace;
    if (!dup) {
      const uint32_t j = x & 2047u, f = fp[j >> 5] + __popc(fm[j >> 5] & ((1u << (j & 31u)) - 1u));
      const uint32_t w = id * nfw + (f >> 5);
      at = pw[w] + __popc(bm[w] & ((1u << (f & 31u)) - 1u));
    }
    kl[boff[b] + at] = (uint16_t)i;
  }
  lg_sync<SM::H>(bar);
  bool bad = dup;  // seed order is not position order: a stray hit, or copies within the reference
#pragma unroll 1
  for (uint32_t i = tid; i < T2; i += G) {
    const uint32_t a = kl[i];
    if (i > 0) {
      const uint32_t p = kl[i - 1];
      const uint32_t b = rank_of(rs[a]);
      if (rank_of(rs[p]) == b && key_of(p) > key_of(a)) {
        bad = true;
        atomicOr(&badr[b >> 5], 1u << (b & 31u));
      }
    }
    sx[i] = (uint16_t)a;
  }
  bad = __any_sync(FULL, bad);
  if (lane == 0) red[1][warp] = bad;
  lg_sync<SM::H>(bar);
  uint32_t any = 0;
#pragma unroll 1
  for (uint32_t w = 0; w < kW; w++) any |= red[1][w];
  bool sorted = !any;
  if (!sorted && bmax <= kRankMax) {
#pragma unroll 1
    for (uint32_t b = warp; b < nk; b += kW)
      if (dup || ((badr[b >> 5] >> (b & 31u)) & 1u)) rank_range(kl, sx, boff[b], boff[b + 1]);
    sorted = true;
    lg_sync<SM::H>(bar);
  }
  if (!sorted) {  // a reference with many postings out of order: bitonic sort of the indices
    uint32_t N = 2;
#pragma unroll 1
    while (N < T2) N <<= 1;
#pragma unroll 1
    for (uint32_t i = T2 + tid; i < N; i += G) sx[i] = 0xFFFFu;
    lg_sync<SM::H>(bar);
#pragma unroll 1
    for (uint32_t kk = 2; kk <= N; kk <<= 1) {
#pragma unroll 1
      for (uint32_t jj = kk >> 1; jj > 0; jj >>= 1) {
#pragma unroll 1
        for (uint32_t c = tid; c < N / 2; c += G) {
          const uint32_t i = 2 * c - (c & (jj - 1)), p = i + jj;  // the pairs i, i ^ jj with i the lower
          const uint32_t a = sx[i], b = sx[p];
          bool gt;
          if (a == 0xFFFFu || b == 0xFFFFu) {
            gt = a > b;
          } else {
            const uint32_t ra = rank_of(rs[a]), rb = rank_of(rs[b]);
            gt = ra > rb || (ra == rb && key_of(a) > key_of(b));
          }
          if (gt == ((i & kk) == 0) && a != b) {
            sx[i] = (uint16_t)b;
            sx[p] = (uint16_t)a;
          }
        }
        lg_sync<SM::H>(bar);
      }
    }
  }
  // 5. diagonal runs (Analyser.cpp:2337-2490): run starts, and each reference's longest run
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < T2; i0 += G) {
    const uint32_t i = i0 + tid;
    bool start = true;
    if (i < T2 && i > 0) {
      const uint32_t a = sx[i - 1], b = sx[i];
      // one reference and seed + 1: one addition on the packed word
      const uint32_t xa = rs[a] & ((1u << kPlace) - 1u), xb = rs[b] & ((1u << kPlace) - 1u);
      start = !((uint64_t)ps[a] + step == ps[b] && xa + 1u == xb && (xb & 2047u) != 0);
    }
    const uint32_t w = __ballot_sync(FULL, start);
    if (lane == 0 && (i0 + warp * 32) < T2) bk[(i0 >> 5) + warp] = w;
  }
  lg_sync<SM::H>(bar);
  auto run_end = [&](uint32_t i) { return i + 1 == T2 || ((bk[(i + 1) >> 5] >> ((i + 1) & 31u)) & 1u); };
  auto run_first = [&](uint32_t i) {  // bit 0 is set: the search ends there at the latest
    uint32_t w = i >> 5, m = bk[w] & (0xFFFFFFFFu >> (31u - (i & 31u)));
#pragma unroll 1
    while (!m) m = bk[--w];
    return w * 32 + 31 - __clz(m);
  };
  if (tid == 0) S.n_ends[half] = 0;
#pragma unroll 1
  for (uint32_t i = tid; i < T2; i += G)
    if (run_end(i)) atomicMax(&T.segmax[rank_of(rs[sx[i]])], i - run_first(i) + 1);
  lg_sync<SM::H>(bar);
  uint32_t M = 0;
#pragma unroll 1
  for (uint32_t b = lane; b < nk; b += 32) M = max(M, T.segmax[b]);
  M = __reduce_max_sync(FULL, M);
  if (M < 2) return kStrandOk;  // Analyser.cpp:2402
  *keeps_all = hs == 2 && ne > kLgKeepAll;
  // 6. candidates: the kept references whose longest run is M, in rank order (every warp has the
  //    masks); the walks of all their runs, a run end a thread, summed per candidate, as many
  //    candidates at a time as their coverage bitmaps have room
  constexpr uint32_t kCM = (kRM + 31) / 32;
  uint32_t cm[kCM];
  uint32_t nc = 0;
#pragma unroll
  for (uint32_t u = 0; u < kCM; u++) {
    const uint32_t b = u * 32 + lane;
    cm[u] = __ballot_sync(FULL, b < nk && T.segmax[b] == M);
    nc += __popc(cm[u]);
  }
  auto cand_of = [&](uint32_t b) -> int {  // a rank's candidate, -1: none
    uint32_t before = 0;
    int c = -1;
#pragma unroll
    for (uint32_t u = 0; u < kCM; u++) {
      if ((b >> 5) == u && ((cm[u] >> (b & 31u)) & 1u)) c = (int)(before + __popc(cm[u] & ((1u << (b & 31u)) - 1u)));
      before += __popc(cm[u]);
    }
    return c;
  };
  const uint32_t nw = (L + 31) / 32;
  uint32_t* cov = reinterpret_cast<uint32_t*>(st);
  const uint32_t per = kCovWords / nw;
#pragma unroll 1
  for (uint32_t c = tid; c < nc; c += G) {
    T.sumc[c] = 0;
    T.sumr[c] = 0;
  }
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < T2; i0 += G) {  // the candidates' run ends, listed (in kl) to fill the warps
    const uint32_t i = i0 + tid;
    const bool end = i < T2 && run_end(i) && T.segmax[rank_of(rs[sx[i]])] == M;
    const uint32_t m = __ballot_sync(FULL, end);
    if (!m) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&S.n_ends[half], (uint32_t)__popc(m));
    at = __shfl_sync(FULL, at, 0);
    if (end) kl[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)i;
  }
  lg_sync<SM::H>(bar);  // every warp has its masks: segmax holds the covered bases from here on
  const uint32_t n_ends = S.n_ends[half];
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < nc; c0 += per) {
    const uint32_t cn = min(per, nc - c0);
#pragma unroll 1
    for (uint32_t i = tid; i < cn * nw; i += G) cov[i] = 0;
    lg_sync<SM::H>(bar);
#pragma unroll 1
    for (uint32_t t0 = 0; t0 < n_ends; t0 += G) {
      const uint32_t t = t0 + tid;
      int c = -1;
      uint32_t z = 0, i = 0, xe = 0, rank = 0;
      if (t < n_ends) {
        i = kl[t];
        xe = rs[sx[i]];
        rank = rank_of(xe);
        c = cand_of(rank);
      }
      if (c >= (int)c0 && c < (int)(c0 + cn)) {
        const uint32_t s = sx[run_first(i)];
        z = walk_run(ix, S.comp, raw, L, strand, T.kref[rank], ps[s], ps[sx[i]] + step,
                     (rs[s] & 2047u) * step, (xe & 2047u) * step + step, k);
      }
      __syncwarp();
      if (!z) continue;
      const uint32_t len = z & 0xFFFFu, a = z >> 16, bnd = a + len;
      atomicAdd(&T.sumc[c], len);
      atomicAdd(&T.sumr[c], (unsigned long long)len * (len + 1) / 2);
      uint32_t* cv = cov + (c - c0) * nw;
#pragma unroll 1
      for (uint32_t wd = a >> 5; wd <= (bnd - 1) >> 5; wd++) {
        const uint32_t w0 = wd * 32;
        const uint32_t lo = a > w0 ? a : w0, up = bnd < w0 + 32 ? bnd : w0 + 32;
        const uint32_t n = up - lo;
        atomicOr(&cv[wd], (n == 32 ? 0xFFFFFFFFu : ((1u << n) - 1u)) << (lo - w0));
      }
    }
    lg_sync<SM::H>(bar);
#pragma unroll 1
    for (uint32_t c = warp; c < cn; c += kW) {
      uint32_t hits = 0;
#pragma unroll 1
      for (uint32_t w = lane; w < nw; w += 32) hits += __popc(cov[c * nw + w]);
      hits = __reduce_add_sync(FULL, hits);
      if (lane == 0) T.segmax[c0 + c] = hits;
    }
    lg_sync<SM::H>(bar);
  }
  // 7. scores, a lane per candidate (MatrixCPU.cpp:18-214); one whose runs all fell short of k keeps
  //    Score -2 and is not scored
  if (warp == 0) {
    uint32_t n_sc = 0;
    float hi = -1.0f;
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < nc; c0 += 32) {
      const uint32_t c = c0 + lane;
      const bool ok = c < nc && T.sumc[c] > 0;
      uint32_t ref = 0;
      float score = 0.0f, pct = 0.0f, rel = -1.0f;
      if (ok) {
        uint32_t n = c;  // the candidate's rank: the c-th set bit of the masks
        bool have = false;
#pragma unroll
        for (uint32_t u = 0; u < kCM; u++) {
          const uint32_t pc = __popc(cm[u]);
          if (!have && n < pc) {
            ref = T.kref[u * 32 + __fns(cm[u], 0, (int)n + 1)];
            have = true;
          }
          if (!have) n -= pc;
        }
        final_score(T.sumr[c], (uint64_t)T.sumc[c], T.segmax[c], L, &score, &pct);
        rel = relative_score_tab(ix, L, ix.ref_len[ref], score, err);
      }
      const uint32_t m = __ballot_sync(FULL, ok);
      if (ok) cb[n_sc + __popc(m & ((1u << lane) - 1u))] = mg_candidate{ref, rel, score, pct};
      n_sc += __popc(m);
      hi = fmaxf(hi, rel);
    }
    for (int o = 16; o; o >>= 1) hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
    if (lane == 0) {
      S.n_out[half] = n_sc;
      S.hi[half] = hi;
    }
  }
  lg_sync<SM::H>(bar);
  *n_out = S.n_out[half];
  *highest = S.hi[half];
  return kStrandOk;
}

// Whether the read's L bytes are all letters of ACGT in either case (1), or else all have a
// complement (0), or not (-1); on the whole block.
template <class SM>
__device__ int read_letters(const uint8_t* raw, uint32_t L, const SM& S) {
  const uintptr_t a = (uintptr_t)raw, e = a + L;
  bool other = false;
#pragma unroll 1
  for (uintptr_t w = (a & ~(uintptr_t)3) + 4 * threadIdx.x; L && w < e; w += 4 * blockDim.x) {
    uint32_t x = *(const uint32_t*)w;  // an aligned word holding at least one byte of the read
    if (w < a) x = (x & (0xFFFFFFFFu << (8 * (uint32_t)(a - w)))) | (0x41414141u >> (32 - 8 * (uint32_t)(a - w)));
    if (w + 4 > e) {
      const uint32_t o = 8 * (uint32_t)(w + 4 - e);
      x = (x & (0xFFFFFFFFu >> o)) | (0x41414141u << (32 - o));
    }
    other |= !acgt4(upper4(x));
  }
  if (!__syncthreads_or(other)) return 1;
  bool bad = false;
#pragma unroll 1
  for (uint32_t i = threadIdx.x; i < L; i += blockDim.x) bad |= S.comp[raw[i]] == 0;
  return __syncthreads_or(bad) ? -1 : 0;
}

// Both strands of read r, the strand merge and the staging write; false when the read must go to the
// next tier. n_small, n_large (optional): counters of the reads that the halves, and the whole block,
// could not take, and of those with a strand that keeps every reference (long_strand). ahead (thread 0's): the entry of list that the block
// takes next; while the first warp writes this read's result, the last one asks for that read's bases.
template <class SM>
__device__ bool process_read_long(const DevIndex& ix, const BatchDev& b, uint32_t r, SM& S, mg_candidate* stage,
                                  mg_candidate* arena, uint64_t arena_cap, unsigned long long* arena_n, int* errw,
                                  unsigned* n_small, unsigned* n_large, const uint32_t* list = nullptr,
                                  uint32_t n_list = 0, uint32_t ahead = 0) {
  constexpr int H = SM::H;
  const uint64_t o0 = b.offs[r];
  const uint64_t Lr = b.offs[r + 1] - o0;
  if (Lr > (uint64_t)kLgQ || ix.n_refs > (1u << 21)) {  // the packed postings hold refID << 11
    if (threadIdx.x == 0 && n_small) {
      atomicAdd(n_small, 1u);
      atomicAdd(n_large, 1u);
    }
    return false;
  }
  const uint32_t L = (uint32_t)Lr;
  const uint8_t* raw = b.bases + o0;
  const int letters = read_letters(raw, L, S);
  if (letters < 0) {
    if (threadIdx.x == 0) {
      b.reads[r] = mg_read_result{-1.0f, 0, 0, 0, MG_READ_BAD_BYTE, 0, 0};
      atomicOr(errw, kErrBadInput);
    }
    return true;
  }
  int err = 0;
  uint32_t n[2] = {0, 0};
  float h[2] = {-1.0f, -1.0f};
  bool keeps_all = false, over = false;
  // first the strands side by side, then, when one does not fit its half, in turn on the whole block (what
  // the first class leaves, the reads without n_small, seldom fits a half of the second: on the whole block
  // at once 2,000 reads of 14 kb on five strains take 0.98 ms, 1.22 ms with the halves first)
#pragma unroll 1
  for (int pass = SM::Rest && !n_small ? 1 : 0; pass < 3; pass++) {
    const bool whole = pass > 0;
    const int half = whole ? 0 : threadIdx.x / H, strand = whole ? pass - 1 : half;
    uint32_t n1;
    float h1;
    bool w = false;
    const int s = long_strand(ix, raw, L, strand, letters == 1, S, whole, half, S.cb[strand], &err, &n1, &h1, &w);
    __syncthreads();
    if (threadIdx.x % H == 0 && (!whole || threadIdx.x == 0)) {
      S.status[strand] = s;
      S.n_out[strand] = n1;
      S.hi[strand] = h1;
      if (w) S.keeps_all = 1;
      if (threadIdx.x == 0) S.ahead = ahead;
    }
    __syncthreads();
    if (!whole) {
      n[0] = S.n_out[0];
      n[1] = S.n_out[1];
      h[0] = S.hi[0];
      h[1] = S.hi[1];
      over = S.status[0] != kStrandOk || S.status[1] != kStrandOk;
    } else {
      over = S.status[strand] != kStrandOk;
      (strand ? n[1] : n[0]) = S.n_out[strand];
      (strand ? h[1] : h[0]) = S.hi[strand];
    }
    keeps_all = S.keeps_all != 0;
    __syncthreads();
    if (pass == 0 && threadIdx.x == 0 && n_small && (over || keeps_all)) atomicAdd(n_small, 1u);
    if (over == whole) break;  // both strands done on the halves, or one does not fit at all
    if (pass == 0 && threadIdx.x == 0) S.keeps_all = 0;
  }
  if (threadIdx.x == 0) S.keeps_all = 0;
  if (threadIdx.x == 0 && n_large && (over || keeps_all)) atomicAdd(n_large, 1u);
  if (err) atomicOr(errw, err);  // any thread's: the scoring lanes record bits per thread
  if (over) return false;
  // the strand merge (Analyser.cpp:592-611), the log skip rule (:388) and the staging write
  const int ch = h[0] < h[1] ? 1 : 0;  // Analyser.cpp:601
  const uint32_t tot = n[0] + n[1];
  if (threadIdx.x < 32) {
    uint32_t top = 0;
#pragma unroll 1
    for (uint32_t c = threadIdx.x; c < n[ch]; c += 32) top += S.cb[ch][c].rel == h[ch];
    top = __reduce_add_sync(0xffffffffu, top);
    if (threadIdx.x == 0) {
      unsigned long long at = 0;
      bool fits = true;
      if (tot > (uint32_t)kSlots) {
        at = atomicAdd(arena_n, (unsigned long long)tot);
        fits = at + tot <= arena_cap;
        if (!fits) atomicOr(errw, kErrArena);
      }
      S.cand_at = fits ? (uint32_t)at : kLgEmpty;
      b.reads[r] = mg_read_result{h[ch], fits ? (uint32_t)at : 0u, (uint16_t)n[0], (uint16_t)n[1], (uint8_t)ch,
                                  (uint8_t)((n[ch] > 0 && h[ch] != 0.0f) ? 1 : 0), (uint16_t)top};
    }
  } else if (list && threadIdx.x >= 2 * H - 32 && S.ahead < n_list) {
    const uint32_t r2 = list[S.ahead];
    const uint64_t a = b.offs[r2], e = b.offs[r2 + 1];
    if (e - a <= (uint64_t)kLgQ)
#pragma unroll 1
      for (uint64_t o = a + 128 * (threadIdx.x & 31u); o < e; o += 128 * 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(b.bases + o));
  }
  __syncthreads();
  if (S.cand_at != kLgEmpty) {
    mg_candidate* dst = tot > (uint32_t)kSlots ? arena + S.cand_at : stage + (uint64_t)r * kSlots;
#pragma unroll 1
    for (uint32_t c = threadIdx.x; c < tot; c += 2 * H) dst[c] = c < n[0] ? S.cb[0][c] : S.cb[1][c - n[0]];
  }
  return true;
}

}  // namespace mg
