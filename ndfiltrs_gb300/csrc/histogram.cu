// Rank-histogram median, rank and percentile for windows of rank 1 to 3
// (method="histogram"; also the large-window path of "direct").
//
// Replaces order_statistic_into / Geometry::block / Histogram
// (src/histogram.rs:93-631). As in the reference, each block of outputs
// ranks its support (the block plus the window halo, through the boundary
// modes) so that every retained sample gets a unique block-local rank; a
// window is then a set of ranks, kept as a bit histogram, and a k-th
// order statistic is the k-th set bit. Results equal direct selection bit
// for bit: equal keys are interchangeable, so the tie order of the ranks
// does not matter.
//
// GB300 design:
//  * one thread block per output tile (a persistent grid where slots are used);
//  * ranking: a block-level LSD radix sort of the support's keys over the bits
//    on which the retained ones differ, in shared memory where it fits (boxes)
//    or through a per-block scratch slot in global memory (L2-resident); rank
//    codes are u16 (support <= 65534);
//  * boxes: a warp selects for a patch of 32 outputs whose windows share one
//    threshold rank (PatchWalk), at a few ranks and support rows per patch;
//  * footprints: each half-warp (16 lanes) owns a strip of output columns and
//    walks it in boustrophedon order, so a warp advances two windows per
//    step; a step removes and adds the ends of the footprint's runs, spread
//    over the 16 lanes with shared-memory atomics on the half-warp's private
//    bitset; a selection scans 512 ranks per step from a tracked pivot (the
//    previous window's order statistic) and ends with a 5-step select in the
//    final word. Tile widths are multiples of 32 columns, so every half-warp's
//    columns lie inside the tile's support.
// Walking every box window through a bitset of its own cost 238 warp
// instructions per output at 65 x 65 whatever the window; patches took the
// 65 x 65 median of a 4096^2 float32 star field from 6.59 to 3.07 ms and the
// (9, 33, 33) median of a 64 x 512 x 512 cube from 61.2 to 33.0 ms; sorting a box's
// support in shared memory, and sharing it among several planes (eight for that
// cube), to 2.40 and 13.2 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/ndfiltrs_gb300.h"
#include "common.cuh"
#include "plan.h"

namespace ndf {

int fail(int code, const std::string& message);
int cuda_fail(cudaError_t e, const char* what);

namespace {

constexpr int kHThreads = 512;
constexpr int kHWarps = kHThreads / 32;
constexpr uint16_t kOmitted = 0xFFFF;
constexpr uint16_t kPropagated = 0xFFFE;
constexpr int kMaxSupport = 65534;
constexpr unsigned int kFull = 0xffffffffu;

struct HistArgs {
  Geom3 g;
  int TW, TH, TZ, SW, SH, SZ, S;
  int plane;                // SH * SW: one support plane (the support is SZ of them)
  long long tiles_x, tiles_yx, tiles;
  int cols_per_warp;        // columns walked by each half-warp segment
  int words;                // per-segment bit histogram: 32-bit words
  long long slot_bytes;     // scratch bytes per block slot (sorts through a slot)
  int digit_bits;           // largest radix digit width of the block sort (8 to 11)
  int patch_w;              // boxes: columns of a warp's patch of outputs (8 or 32)
  int sideways;             // patches of one row are walked along it (else down)
  int in_smem;              // boxes: the support is sorted in shared memory (else through a slot)
  int column_map;           // the columns' offsets lie in a table (else mapped as they go)
  unsigned int row_magic;   // ceil(2^32 / SW): row of an in-plane support index
  unsigned int plane_magic; // ceil(2^32 / plane): plane of a support index
  Reduce r;
  // Footprint windows: support-linear offsets (y * SW + x) of the taps
  // (nf), of the top and bottom ends of every vertical run of taps (nv
  // each) and of the left and right ends of every horizontal run (nh
  // each), in that order. Unused (nullptr) for rectangular windows.
  const uint16_t* lists;
  int nf, nv, nh;
};

// A block's sort slot: two arrays of keys with their support indices. A key and
// its index lie together, so that the scatter of a pass writes one 32-byte
// sector per sample (apart they wrote two, and those stores bound the sort:
// 6.9 of the 14.0 ms of a (9, 33, 33) median of a 64 x 512 x 512 cube; 13.1 ms now).
template <typename K>
struct Entry;
template <>
struct __align__(8) Entry<uint32_t> {
  uint32_t key;
  uint32_t at;
};
template <>
struct __align__(16) Entry<unsigned long long> {
  unsigned long long key;
  unsigned long long at;
};

// The sorted keys of a footprint's support: the decode table, or every second
// word of a slot's entries.
template <typename K>
struct SortedKeys {
  const K* p;
  int step;
  __device__ __forceinline__ K operator[](int rank) const { return p[rank * step]; }
};

template <typename K>
struct Slot {
  Entry<K>* a;
  Entry<K>* b;
};

__host__ __device__ inline long long align16(long long v) { return (v + 15) & ~15ll; }

// Bytes of a tile's axis maps: 64-bit offsets of its rows and planes, and of
// its columns where those have a table.
__host__ __device__ inline long long axis_map_bytes(int SH, int SZ, int SW, bool column_map) {
  return align16(8ll * (SH + SZ + (column_map ? SW : 0)));
}

template <typename K>
__host__ __device__ inline long long slot_bytes_for(int S) {
  return 2 * align16((long long)S * sizeof(Entry<K>));
}

template <typename K>
__device__ inline Slot<K> slot_at(unsigned char* base, int S) {
  return {reinterpret_cast<Entry<K>*>(base), reinterpret_cast<Entry<K>*>(base + align16((long long)S * sizeof(Entry<K>)))};
}

// Accesses to the sort slots in global memory with an L2 evict-last policy.
// A block rewrites its slot on every radix pass; the hint keeps the slots in
// L2 against the input stream (the support's samples), so that most of the
// ping-pong does not reach DRAM.
__device__ __forceinline__ unsigned long long keep_policy() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void st_keep(Entry<uint32_t>* a, Entry<uint32_t> v, unsigned long long p) {
  asm volatile("st.global.L2::cache_hint.v2.b32 [%0], {%1, %2}, %3;" ::"l"(a), "r"(v.key), "r"(v.at), "l"(p) : "memory");
}
__device__ __forceinline__ void st_keep(Entry<unsigned long long>* a, Entry<unsigned long long> v, unsigned long long p) {
  asm volatile("st.global.L2::cache_hint.v2.b64 [%0], {%1, %2}, %3;" ::"l"(a), "l"(v.key), "l"(v.at), "l"(p) : "memory");
}
__device__ __forceinline__ Entry<uint32_t> ld_keep(const Entry<uint32_t>* a, unsigned long long p) {
  Entry<uint32_t> v;
  asm volatile("ld.global.L2::cache_hint.v2.b32 {%0, %1}, [%2], %3;" : "=r"(v.key), "=r"(v.at) : "l"(a), "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ Entry<unsigned long long> ld_keep(const Entry<unsigned long long>* a, unsigned long long p) {
  Entry<unsigned long long> v;
  asm volatile("ld.global.L2::cache_hint.v2.b64 {%0, %1}, [%2], %3;" : "=l"(v.key), "=l"(v.at) : "l"(a), "l"(p) : "memory");
  return v;
}

// Shared-memory words of the sort's counter tables for `nd` digits: one
// table of nd counters per warp plus the nd digit totals.
__host__ __device__ inline long long sort_table_words(int nd) { return (long long)(kHWarps + 1) * nd; }

// One stable counting pass over `nd`-valued digits. `table` holds
// kHWarps x nd counters, `totals` nd. Each warp owns a contiguous segment
// and ranks its 32-entry chunks in order, so equal digits keep their order. Loads are batched (kBatch entries per lane in registers) so a
// pass costs one memory round trip per batch rather than one per chunk.
template <typename K, typename Digit>
__device__ void radix_pass(const Entry<K>* src, Entry<K>* dst, int S, unsigned int* table, unsigned int* totals,
                           int nd, Digit digit, unsigned long long keep) {
  constexpr int kBatch = sizeof(K) == 4 ? 8 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kHWarps * nd; i += blockDim.x) table[i] = 0;
  __syncthreads();
  const int chunk = (((S + kHWarps - 1) / kHWarps) + 31) & ~31;
  const int begin = warp * chunk;
  const int end = min(S, begin + chunk);
  unsigned int* wt = table + warp * nd;
  for (int b = begin; b < end; b += 32 * kBatch) {
    Entry<K> e[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int i = b + j * 32 + lane;
      e[j] = i < end ? ld_keep(src + i, keep) : Entry<K>{0, 0};
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      // A digit that many lanes share (the top ones are alike) is added once.
      const bool valid = b + j * 32 + lane < end;
      const int d = valid ? (int)digit(e[j].key) : -1;
      const int first = __shfl_sync(kFull, d, 0);
      const unsigned int same = __ballot_sync(kFull, d == first);
      const bool shared = __popc(same) >= 8;
      if (shared && lane == 0 && valid) atomicAdd(&wt[d], (unsigned int)__popc(same));
      if (valid && (!shared || d != first)) atomicAdd(&wt[d], 1u);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nd; d += blockDim.x) {
    unsigned int sum = 0;
    for (int w = 0; w < kHWarps; ++w) sum += table[w * nd + d];
    totals[d] = sum;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // Exclusive scan of the nd totals by one warp (nd / 32 per lane).
    const int per = nd >> 5;
    unsigned int run = 0;
    for (int j = 0; j < per; ++j) {
      const unsigned int t = totals[lane * per + j];
      totals[lane * per + j] = run;
      run += t;
    }
    unsigned int inc = run;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    const unsigned int excl = inc - run;
    for (int j = 0; j < per; ++j) totals[lane * per + j] += excl;
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nd; d += blockDim.x) {
    unsigned int run = totals[d];
    for (int w = 0; w < kHWarps; ++w) {
      const unsigned int c = table[w * nd + d];
      table[w * nd + d] = run;
      run += c;
    }
  }
  __syncthreads();
  for (int b = begin; b < end; b += 32 * kBatch) {
    Entry<K> e[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int i = b + j * 32 + lane;
      e[j] = i < end ? ld_keep(src + i, keep) : Entry<K>{0, 0};
    }
    // Lanes with equal digits by a ballot per digit bit (the match instruction
    // takes its pipe some 46 clocks a warp).
    unsigned int peers[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) peers[j] = __ballot_sync(kFull, b + j * 32 + lane < end);
    for (int bit = 1; bit < nd; bit <<= 1) {
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const bool set = (digit(e[j].key) & bit) != 0;
        const unsigned int with = __ballot_sync(kFull, set);
        peers[j] &= set ? with : ~with;
      }
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const bool valid = b + j * 32 + lane < end;
      const unsigned int d = digit(e[j].key);
      unsigned int at = 0;
      if (valid) at = wt[d];
      __syncwarp();
      if (valid && lane == 31 - __clz(peers[j])) wt[d] = at + __popc(peers[j]);
      __syncwarp();
      if (valid) st_keep(dst + at + __popc(peers[j] & ((1u << lane) - 1u)), e[j], keep);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ int select_in_word32(unsigned int word, int k) {
  int position = 0;
#pragma unroll
  for (int width = 16; width >= 1; width >>= 1) {
    int low = __popc(word & ((1u << width) - 1u));
    if (k >= low) {
      k -= low;
      word >>= width;
      position += width;
    }
  }
  return position;
}

// Each half-warp (16 lanes, a "segment") owns one bit histogram of the
// ranks in its window, so a warp advances two windows per step. The segment
// tracks the rank `m` of its last selected order statistic and the number
// `lt` of window samples ranked below it, kept up to date by every histogram
// update. A selection walks from m word by word (every lane loads the same
// word, so the walk costs what one thread's would); the next window's order
// statistic is usually a few window samples away, within a word or two. A
// walk longer than kSeqWords words continues as a parallel scan of 16 words
// per iteration (sixteen sequential words measured 2-5% faster than four,
// and four faster than one or two, on full windows from 13 x 13 to 65 x 65 when
// boxes came this way too; 32 no faster than 16). Every loop
// that contains warp-synchronous operations runs until both segments of the
// warp are done, so the two halves stay converged.
constexpr int kSeg = 16;
constexpr int kSegs = kHThreads / kSeg;
constexpr int kSeqWords = 16;

struct SegHist {
  unsigned int* words;
  int nwords;
  int m;      // tracked rank (the last order statistic selected)
  int lt;     // window samples ranked below m
  int count;  // retained samples in the window
  int nan;    // propagated NaN samples in the window
};

__device__ __forceinline__ int seg_lane() { return threadIdx.x & (kSeg - 1); }

__device__ __forceinline__ unsigned int seg_ballot(bool p) {
  return (__ballot_sync(kFull, p) >> (threadIdx.x & kSeg)) & 0xFFFFu;
}

__device__ __forceinline__ int seg_sum(int v) {
#pragma unroll
  for (int o = kSeg / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(kFull, v, o, kSeg);
  return v;
}

__device__ __forceinline__ unsigned int seg_scan(unsigned int v) {
  const int hl = seg_lane();
#pragma unroll
  for (int o = 1; o < kSeg; o <<= 1) {
    const unsigned int t = __shfl_up_sync(kFull, v, o, kSeg);
    if (hl >= o) v += t;
  }
  return v;
}

template <typename V>
__device__ __forceinline__ V seg_bcast(V v, int src) {
  return __shfl_sync(kFull, v, src, kSeg);
}

// Parallel continuation of a walk. Forward: the rem-th (0-based) set bit at
// or above word wi. Backward: the rem-th (1-based) set bit counting down
// from the top of word wi. `active` false takes part for convergence only
// and returns r unchanged.
__device__ __noinline__ int seg_scan_select(const SegHist& h, int wi, int rem, bool fwd, bool active, int r) {
  const int hl = seg_lane();
  bool found = !active;
  for (int guard = 0; guard < 8192; ++guard) {
    if (!__any_sync(kFull, !found)) break;
    const int widx = fwd ? wi + hl : wi - hl;
    const unsigned int word = (widx >= 0 && widx < h.nwords) ? h.words[widx] : 0u;
    const unsigned int pc = __popc(word);
    const unsigned int incl = seg_scan(pc);
    const int total = (int)seg_bcast(incl, kSeg - 1);
    const unsigned int ball = seg_ballot(fwd ? (int)incl > rem : (int)incl >= rem);
    const int L = ball ? __ffs(ball) - 1 : 0;
    const unsigned int w = seg_bcast(word, L);
    const int excl = (int)seg_bcast(incl - pc, L);
    if (!found) {
      if (ball) {
        const int within = rem - excl;
        r = ((fwd ? wi + L : wi - L) << 5) + select_in_word32(w, fwd ? within : __popc(w) - within);
        found = true;
      } else {
        rem -= total;
        wi = fwd ? wi + kSeg : wi - kSeg;
        if (wi < 0 || wi >= h.nwords) found = true;  // no such bit: leave r
      }
    }
  }
  return r;
}

// Rank of the k-th (0-based) retained sample of the segment's window; the
// tracked rank moves to it. `active` false leaves the state untouched.
__device__ __forceinline__ int seg_select(SegHist& h, int k, bool active) {
  int r = 0, wi = 0, rem = 0;
  bool fwd = true, done = !active;
  if (active) {
    int d = k - h.lt;
    wi = h.m >> 5;
    const int bit = h.m & 31;
    if (d >= 0) {
      unsigned int w = h.words[wi] & (~0u << bit);
      int pc = __popc(w);
#pragma unroll 1
      for (int s = 0; d >= pc && s < kSeqWords; ++s) {
        d -= pc;
        ++wi;
        w = wi < h.nwords ? h.words[wi] : 0u;
        pc = __popc(w);
      }
      if (d < pc) {
        r = (wi << 5) + select_in_word32(w, d);
        done = true;
      } else {
        rem = d - pc;
        ++wi;
      }
    } else {
      int e = -d;
      unsigned int w = h.words[wi] & ((1u << bit) - 1u);
      int pc = __popc(w);
#pragma unroll 1
      for (int s = 0; e > pc && s < kSeqWords; ++s) {
        e -= pc;
        --wi;
        w = wi >= 0 ? h.words[wi] : 0u;
        pc = __popc(w);
      }
      if (e <= pc) {
        r = (wi << 5) + select_in_word32(w, pc - e);
        done = true;
      } else {
        rem = e - pc;
        --wi;
        fwd = false;
      }
    }
  }
  if (__any_sync(kFull, !done)) r = seg_scan_select(h, wi, rem, fwd, !done, r);
  if (active) {
    h.m = r;
    h.lt = k;
  }
  return r;
}

// Rank of the first retained sample above `rank` (the next order statistic).
__device__ __forceinline__ int seg_next(const SegHist& h, int rank, bool active) {
  int r = rank, wi = 0;
  bool done = !active;
  if (active) {
    wi = rank >> 5;
    unsigned int w = h.words[wi] & ~((2u << (rank & 31)) - 1u);
#pragma unroll 1
    for (int s = 0; w == 0u && s < kSeqWords; ++s) {
      ++wi;
      w = wi < h.nwords ? h.words[wi] : 0u;
    }
    if (w) {
      r = (wi << 5) + __ffs(w) - 1;
      done = true;
    } else {
      ++wi;
    }
  }
  if (__any_sync(kFull, !done)) r = seg_scan_select(h, wi, 0, true, !done, r);
  return r;
}

// Per-step bookkeeping of a lane: retained, below-m and propagated-NaN
// deltas.
struct StepDelta {
  int kept = 0, below = 0, nans = 0;
};

template <bool PROPAGATE>
__device__ __forceinline__ void update(const SegHist& h, int c, int sign, StepDelta& d) {
  const bool valid = c < (int)kPropagated;
  // Unconditional: a dropped code XORs zero into a word of the segment's own
  // bitset (the lane's, within its bounds), so the update has no branch (and
  // no reconvergence) around its atomic.
  atomicXor(&h.words[valid ? (c >> 5) : min(seg_lane(), h.nwords - 1)], valid ? 1u << (c & 31) : 0u);
  d.kept += valid ? sign : 0;
  d.below += c < h.m ? sign : 0;  // codes below m are retained (dropped codes are the largest)
  if (PROPAGATE) d.nans += c == (int)kPropagated ? sign : 0;
}

// Apply a step's deltas. Under the omit policy the retained and below-m
// deltas share one reduction in two 16-bit halves biased by 1024 per lane,
// valid while a lane handles fewer than 512 codes (`narrow`).
template <bool PROPAGATE>
__device__ __forceinline__ void finish_update(SegHist& h, const StepDelta& d, bool narrow) {
  if (PROPAGATE || !narrow) {
    h.count += seg_sum(d.kept);
    h.lt += seg_sum(d.below);
    if (PROPAGATE) h.nan += seg_sum(d.nans);
  } else {
    const int packed = (d.kept + 1024) | ((d.below + 1024) << 16);
    const unsigned int sum = (unsigned int)seg_sum(packed);
    h.count += (int)(sum & 0xFFFFu) - kSeg * 1024;
    h.lt += (int)(sum >> 16) - kSeg * 1024;
  }
  __syncwarp();
}

// Footprint windows: remove the codes at rbase + rlist[i] and add those at
// abase + alist[i] (n each).
template <bool PROPAGATE>
__device__ __forceinline__ void step_lists(const uint16_t* codes, int rbase, const uint16_t* rlist,
                                           int abase, const uint16_t* alist, int n, SegHist& h) {
  const int hl = seg_lane();
  StepDelta d;
  const int iters = (n + kSeg - 1) / kSeg;
  for (int it = 0, i = hl; it < iters; ++it, i += kSeg) {
    const bool in = i < n;
    const int rc = in ? codes[rbase + rlist[i]] : (int)kOmitted;
    const int ac = in ? codes[abase + alist[i]] : (int)kOmitted;
    update<PROPAGATE>(h, rc, -1, d);
    update<PROPAGATE>(h, ac, +1, d);
  }
  finish_update<PROPAGATE>(h, d, n <= 8 * 1024);
}

// Footprint windows: add every tap of the window whose origin is `base`.
template <bool PROPAGATE>
__device__ __forceinline__ void add_taps(const uint16_t* codes, int base, const uint16_t* taps, int n,
                                        SegHist& h) {
  const int hl = seg_lane();
  StepDelta d;
  for (int i = hl; i < n; i += kSeg) update<PROPAGATE>(h, codes[base + taps[i]], +1, d);
  finish_update<PROPAGATE>(h, d, false);
}

// The ranks a window's statistic is read from: lo (and hi for an even
// median or an interpolated percentile), the retained count, and whether
// the window has a value at all.
struct Ranks {
  int lo = 0, hi = 0, n = 0;
  bool valid = false, two = false;
};

// Select the ranks of the segment's window. Every branch on per-segment data
// calls the same sequence of selections, so the warp stays converged.
__device__ __forceinline__ Ranks hist_ranks(SegHist& h, const HistArgs& a) {
  const Reduce& r = a.r;
  Ranks o;
  o.n = h.count;
  const bool valid = !((!r.omit && h.nan > 0) || (r.omit && h.count < r.min_count) || h.count == 0);
  const int last = max(h.count - 1, 0);
  switch (r.kind) {
    case kRank:
    case kRankHistogram: {
      const bool ok = valid && r.param < h.count;
      o.lo = o.hi = seg_select(h, ok ? (int)r.param : 0, ok);
      o.valid = ok;
      return o;
    }
    case kMin:
      o.lo = o.hi = seg_select(h, 0, valid);
      o.valid = valid;
      return o;
    case kMax:
      o.lo = o.hi = seg_select(h, last, valid);
      o.valid = valid;
      return o;
    case kPercentile: {
      if (r.q_is_max) {
        o.lo = o.hi = seg_select(h, last, valid);
        o.valid = valid;
        return o;
      }
      const PctSplit ps = pct_split(r, max(h.count, 1));
      o.lo = seg_select(h, valid ? ps.lower : 0, valid);
      o.two = ps.upper != ps.lower;
      o.hi = seg_next(h, o.lo, valid && o.two);
      o.valid = valid;
      return o;
    }
    default: {
      const bool even = (h.count & 1) == 0;
      const int k = even ? h.count / 2 - 1 : h.count / 2;
      o.lo = seg_select(h, valid ? k : 0, valid);
      o.hi = seg_next(h, o.lo, valid && even);
      o.two = even;
      o.valid = valid;
      return o;
    }
  }
}

// The statistic of a window from the samples of its ranks lo and hi.
template <typename T>
__device__ __forceinline__ T hist_value(const Ranks& o, const HistArgs& a, T vlo, T vhi) {
  if (!o.valid) return nan_of(T());
  switch (a.r.kind) {
    case kPercentile: {
      if (a.r.q_is_max) return vlo;
      const PctSplit ps = pct_split(a.r, max(o.n, 1));
      return pct_value<T>(ps, vlo, o.two ? vhi : vlo);
    }
    case kRank:
    case kRankHistogram:
    case kMin:
    case kMax:
      return vlo;
    default:
      if (!o.two) return vlo;
      if constexpr (sizeof(T) == 4) {
        return midpoint_f32(vlo, vhi);
      } else {
        return midpoint(vlo, vhi);
      }
  }
}

// Outputs of a walk, one per lane of the segment: the ranks are selected in
// order (one window after another) and parked in lane i % 16; every 16
// outputs the batch's keys are loaded (one independent load per lane), and
// the previous batch's values are computed and stored, so the loads' latency
// overlaps the next 16 windows.
template <typename T>
struct OutPipe {
  using K = typename KeyOf<T>::K;
  Ranks next;             // ranks parked in this lane
  long long next_at = -1; // its output index (-1: none / not stored)
  Ranks held;             // the previous batch: ranks and loaded keys
  long long held_at = -1;
  K kl = 0, kh = 0;

  __device__ __forceinline__ void park(const Ranks& o, long long at, int slot) {
    if (seg_lane() == slot) {
      next = o;
      next_at = at;
    }
  }
  __device__ __forceinline__ void complete(const HistArgs& a, T* __restrict__ out) {
    if (held_at >= 0) out[held_at] = canonical(hist_value<T>(held, a, KeyOf<T>::value(kl), KeyOf<T>::value(kh)));
    held_at = -1;
  }
  // Complete the held batch, then load the parked one's keys and hold it.
  __device__ __forceinline__ void rotate(const HistArgs& a, SortedKeys<K> sorted, T* __restrict__ out) {
    complete(a, out);
    if (next_at >= 0) {
      kl = next.valid ? sorted[next.lo] : K(0);
      kh = next.valid && next.two ? sorted[next.hi] : kl;
    }
    held = next;
    held_at = next_at;
    next_at = -1;
  }
};

// A segment's boustrophedon walk over columns [c_begin, c_begin + ncols)
// of its tile (footprint windows); columns at or beyond `tw_eff` are computed
// for convergence but not stored. A window's origin is its top-left support
// position o = row * SW + c, and a step moves the run ends in `lists`: down
// removes o + top[i] and adds o + SW + bottom[i], up removes o + bottom[i] and
// adds o - SW + top[i], right removes o + left[i] and adds o + 1 + right[i].
template <typename T, bool PROPAGATE>
__device__ __forceinline__ void walk(const uint16_t* codes, const uint16_t* lists, int c_begin,
                                     int ncols, int tw_eff, int th_eff, int SW,
                                     long long y0, long long x0, const Geom3& g, const HistArgs& a,
                                     SortedKeys<typename KeyOf<T>::K> sorted, T* __restrict__ out,
                                     SegHist& h) {
  const uint16_t* top = lists + a.nf;
  const uint16_t* bottom = top + a.nv;
  const uint16_t* left = bottom + a.nv;
  const uint16_t* right = left + a.nh;
  add_taps<PROPAGATE>(codes, c_begin, lists, a.nf, h);
  OutPipe<T> pipe;
  int slot = 0;
  int row = 0;
  int dir = 1;
  for (int j = 0; j < ncols; ++j) {
    const int c = c_begin + j;
    for (int i = 0; i < th_eff; ++i) {
      const Ranks o = hist_ranks(h, a);
      pipe.park(o, c < tw_eff ? (y0 + row) * g.W + x0 + c : -1, slot);
      if (++slot == kSeg) {
        pipe.rotate(a, sorted, out);
        slot = 0;
      }
      if (i + 1 < th_eff) {
        const int o = row * SW + c;
        if (dir > 0) {
          step_lists<PROPAGATE>(codes, o, top, o + SW, bottom, a.nv, h);
          ++row;
        } else {
          step_lists<PROPAGATE>(codes, o, bottom, o - SW, top, a.nv, h);
          --row;
        }
      }
    }
    if (j + 1 < ncols) {
      const int o = row * SW + c;
      step_lists<PROPAGATE>(codes, o, left, o + 1, right, a.nh, h);
    }
    dir = -dir;
  }
  pipe.rotate(a, sorted, out);
  pipe.complete(a, out);
}

// ---------------------------------------------------------------------------
// A tile's support: its samples in the array, each axis mapped through its
// boundary mode once per tile. (A single row maps its columns as it goes, as do
// supports so wide that a table would leave no room for their codes.)
template <typename T>
struct Support {
  using K = typename KeyOf<T>::K;
  const HistArgs& a;
  const T* in;
  long long* row_map;     // SH row offsets, then SZ plane offsets (-1: outside)
  long long* column_map;  // SW column offsets
  long long x0;
  T outside;

  __device__ __forceinline__ long long column(int sx) const {
    long long m;
    return map_index(x0 + sx - a.g.ax, a.g.W, a.g.mx, &m) ? m : -1;
  }

  // Fill the tables (the caller synchronizes).
  __device__ __forceinline__ void build(long long z0, long long y0) {
    const Geom3& g = a.g;
    const int lines = a.SH + a.SZ;
    for (int i = threadIdx.x; i < lines + (a.column_map ? a.SW : 0); i += blockDim.x) {
      long long m;
      if (i < a.SH)
        row_map[i] = map_index(y0 + i - g.ay, g.H, g.my, &m) ? m * g.W : -1;
      else if (i < lines)
        row_map[i] = map_index(z0 + (i - a.SH) - g.az, g.D, g.mz, &m) ? m * g.H * g.W : -1;
      else
        column_map[i - lines] = column(i - lines);
    }
  }

  // f(support index, key) for every sample, rows to warps (without a table of columns:
  // samples to threads).
  template <typename F>
  __device__ __forceinline__ void each(F&& f) const {
    const bool drop_inf = a.r.drop_inf;
    const K out_key = sample_key<T>(outside, drop_inf);
    if (!a.column_map) {
      if (a.SZ * a.SH > 1) {
        for (int e = threadIdx.x; e < a.S; e += blockDim.x) f(e, sample_key<T>(value(e), drop_inf));
        return;
      }
      const bool inside = row_map[0] >= 0 && row_map[1] >= 0;
      const T* src = in + (inside ? row_map[0] + row_map[1] : 0);
      for (int sx = threadIdx.x; sx < a.SW; sx += blockDim.x) {
        const long long ox = column(sx);
        f(sx, inside && ox >= 0 ? sample_key<T>(__ldg(src + ox), drop_inf) : out_key);
      }
      return;
    }
    const int lane = threadIdx.x & 31, rows = a.SZ * a.SH;
    for (int row = threadIdx.x >> 5; row < rows; row += kHWarps) {
      const int sz = a.SZ > 1 ? row / a.SH : 0;
      const long long oy = row_map[row - sz * a.SH], oz = row_map[a.SH + sz];
      const bool inside = oy >= 0 && oz >= 0;
      const T* src = in + (inside ? oy + oz : 0);
      const int e = row * a.SW;
#pragma unroll 4
      for (int sx = lane; sx < a.SW; sx += 32) {
        const long long ox = column_map[sx];
        f(e + sx, inside && ox >= 0 ? sample_key<T>(__ldg(src + ox), drop_inf) : out_key);
      }
    }
  }

  __device__ __forceinline__ T value(unsigned int e) const {
    unsigned int sz = 0;
    if (a.SZ > 1) {
      sz = __umulhi(e, a.plane_magic);
      e -= sz * a.plane;
    }
    const unsigned int sy = __umulhi(e, a.row_magic);
    const int sx = (int)(e - sy * a.SW);
    const long long oy = row_map[sy], oz = row_map[a.SH + sz];
    const long long ox = a.column_map ? column_map[sx] : column(sx);
    return oy >= 0 && oz >= 0 && ox >= 0 ? __ldg(in + oy + oz + ox) : outside;
  }
};

// The bits on which the support's retained keys differ (AND and OR over the
// block) and the number of dropped samples.
template <typename K>
struct KeyBits {
  K varying;
  int sent;
};

template <typename K>
__device__ __forceinline__ KeyBits<K> block_bits(K k_and, K k_or, int sent, int S) {
  __shared__ K red_and[kHWarps], red_or[kHWarps];
  __shared__ int red_sent[kHWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int o = 16; o >= 1; o >>= 1) {
    k_and &= __shfl_xor_sync(0xffffffffu, k_and, o);
    k_or |= __shfl_xor_sync(0xffffffffu, k_or, o);
    sent += __shfl_xor_sync(0xffffffffu, sent, o);
  }
  if (lane == 0) {
    red_and[warp] = k_and;
    red_or[warp] = k_or;
    red_sent[warp] = sent;
  }
  __syncthreads();
  k_and = ~K(0);
  k_or = 0;
  sent = 0;
  for (int w = 0; w < kHWarps; ++w) {
    k_and &= red_and[w];
    k_or |= red_or[w];
    sent += red_sent[w];
  }
  return {sent == S ? K(0) : (K)(k_and ^ k_or), sent};
}

template <typename K>
__device__ __forceinline__ int lowest_set(K v) {
  return (sizeof(K) == 8 ? __ffsll((long long)v) : __ffs((int)v)) - 1;
}
template <typename K>
__device__ __forceinline__ int highest_set(K v) {
  return (int)sizeof(K) * 8 - 1 - (sizeof(K) == 8 ? __clzll((long long)v) : __clz((int)v));
}

// ---------------------------------------------------------------------------
// Block sort of a support within shared memory (boxes).
//
// Sorting keys and payloads through a slot in global memory scatters a key and
// a payload per sample and pass, a 32-byte sector each: 1.7 of the 3.1 ms of a
// 65 x 65 median of 4096^2 went there, at 21% issue. Here the samples' order (16-bit
// indices) ping-pongs between the two arrays that the walk needs anyway, and
// only the 16 key bits that the next digits come from lie beside them; they are
// taken from the array again (it is in L2) when those are used up. A key is
// never moved, so a sample costs 6 bytes of shared memory whatever its type.
// Per pass of four bits each thread counts the digits of a run of consecutive
// samples in sixteen counters of its own, one scan over (digit, thread) makes
// them first positions, and the thread places its samples in order: no atomics
// and no search for equal digits within a warp, which made wide digits dear
// (ranking 8-bit digits with match_any kept that pipe 61% busy and took 1.9 ms
// of a 65 x 65 median of 4096^2, with ballots 1.5 ms at 149 warp instructions per
// 32 samples and pass). Counters of the digits d and d + 8 share a word in the
// thread's bank; a run has twice an odd number of samples, so that the runs'
// words lie in different banks too.
// Returns with the sorted order in `order` (S indices).
constexpr int kDigitBits = 4;
constexpr int kCounterWords = (1 << kDigitBits) / 2 * kHThreads;

template <typename T>
__device__ void sort_in_smem(const Support<T>& sup, uint16_t* other, uint16_t* order, uint16_t* seg,
                             unsigned int* table, typename KeyOf<T>::K varying) {
  using K = typename KeyOf<T>::K;
  __shared__ unsigned int warp_sum[kHWarps];
  const HistArgs& a = sup.a;
  const int S = a.S, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (varying == 0) {
    for (int i = tid; i < S; i += blockDim.x) order[i] = (uint16_t)i;
    __syncthreads();
    return;
  }
  // The last pass writes `order`.
  const int lo = lowest_set(varying), nbits = highest_set(varying) - lo + 1;
  const int passes = (nbits + kDigitBits - 1) / kDigitBits;
  constexpr int kPerFill = 16 / kDigitBits;
  constexpr int kRake = kCounterWords / kHThreads;  // 8
  const int run = 2 * (((S + 2 * kHThreads - 1) / (2 * kHThreads)) | 1);
  const int begin = min(S, tid * run), end = min(S, begin + run);
  uint16_t* counters = reinterpret_cast<uint16_t*>(table + tid);
  auto counter = [&](unsigned int d) -> uint16_t& { return counters[(d & 7) * 2 * kHThreads + (d >> 3)]; };
  for (int pass = 0; pass < passes; ++pass) {
    const int in_seg = pass % kPerFill;
    if (in_seg == 0) {
      const int shift = lo + pass * kDigitBits;
      sup.each([&](int e, K key) { seg[e] = (uint16_t)(key >> shift); });
    }
    const int shift = in_seg * kDigitBits;
    const bool to_order = ((passes - 1 - pass) & 1) == 0;
    const uint16_t* src = to_order ? other : order;
    uint16_t* dst = to_order ? order : other;
#pragma unroll
    for (int j = 0; j < kRake; ++j) table[j * kHThreads + tid] = 0;
    __syncthreads();
    // Two samples at a time: i and i + 1 (runs start at even places).
    auto samples = [&](int i) -> unsigned int {
      return pass == 0 ? (unsigned int)i | (unsigned int)(i + 1) << 16 : *reinterpret_cast<const unsigned int*>(src + i);
    };
    auto digit = [&](unsigned int e) -> unsigned int { return (unsigned int)(seg[e] >> shift) & 15u; };
#pragma unroll 2
    for (int i = begin; i + 1 < end; i += 2) {
      const unsigned int e = samples(i);
      const unsigned int d0 = digit(e & 0xFFFFu), d1 = digit(e >> 16);
      ++counter(d0);
      ++counter(d1);
    }
    if ((end - begin) & 1) ++counter(digit(samples(end - 1) & 0xFFFFu));
    __syncthreads();
    // Exclusive scan in the order (digit, thread); thread r rakes the words
    // 8 r to 8 r + 7. The low halves (digits 0 to 7) come before all high ones.
    uint4* mine = reinterpret_cast<uint4*>(table + tid * kRake);
    uint4 u = mine[0], v = mine[1];
    const unsigned int c[kRake] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    unsigned int sum = 0;
#pragma unroll
    for (int j = 0; j < kRake; ++j) sum += c[j];
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    unsigned int base = incl - sum, total = 0;
#pragma unroll
    for (int w = 0; w < kHWarps; ++w) {
      const unsigned int t = warp_sum[w];
      base += w < warp ? t : 0;
      total += t;
    }
    base += total << 16;
    unsigned int p[kRake];
#pragma unroll
    for (int j = 0; j < kRake; ++j) {
      p[j] = base;
      base += c[j];
    }
    mine[0] = make_uint4(p[0], p[1], p[2], p[3]);
    mine[1] = make_uint4(p[4], p[5], p[6], p[7]);
    __syncthreads();
#pragma unroll 2
    for (int i = begin; i + 1 < end; i += 2) {
      const unsigned int e = samples(i);
      const unsigned int d0 = digit(e & 0xFFFFu), d1 = digit(e >> 16);
      uint16_t& c0 = counter(d0);
      const uint16_t at0 = c0;
      c0 = at0 + 1;
      uint16_t& c1 = counter(d1);
      const uint16_t at1 = c1;
      c1 = at1 + 1;
      dst[at0] = (uint16_t)e;
      dst[at1] = (uint16_t)(e >> 16);
    }
    if ((end - begin) & 1) {
      const unsigned int e = samples(end - 1) & 0xFFFFu;
      dst[counter(digit(e))] = (uint16_t)e;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Box windows (1-D to 3-D): a warp selects for a patch of 32 outputs at once.
//
// The 32 windows of a patch overlap almost entirely, so their order statistics
// lie close together among the tile's ranks. The warp keeps one threshold rank
// t near them. Each lane knows how many samples of its window rank below t,
// and reads its order statistic off the ranks around t, which every lane looks
// through together:
//  * counts: a support row becomes one bit per sample (code < t) by ballots;
//    a lane's share of the row is a shifted, masked popcount. When the patch
//    moves down by its height the rows that leave and enter are counted, or
//    all rows when those are fewer;
//  * ranks: lane i takes the sample of rank r + i and works out which of the
//    32 windows hold it (a mask of lanes). The 32 x 32 bits are transposed in
//    five shuffle stages, after which lane L has the word of the 32 ranks that
//    its own window holds: a popcount advances its count and the word that
//    reaches its order statistic is kept and searched once at the end.
// The work per output is the rows' ballots over 32 outputs plus the rank
// distance between the patch's least and largest result, instead of the
// window's faces per output and a walk through a private bitset (16 lanes a
// window). A patch of 8 x 4 outputs keeps that distance short on slopes (rows
// of 32 x 1 serve single-row tiles). Deep (3-D) windows take patches of 8 columns
// in 4 planes and move them down by a row: of each plane one row leaves and one
// enters, where 8 x 4 in a plane would count 14.

// Bits [lo, lo + width) of a word; lo and width at least 0.
__device__ __forceinline__ unsigned int bit_run(int lo, int width) {
  unsigned int m;
  asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(m) : "r"(lo), "r"(width));
  return m;
}

// Transpose of the 32 x 32 bit matrix whose row i lane i holds: five exchanges
// of halves. Moving the other lane's half into place is a byte permute for the
// first two and a rotation for the rest; what a lane keeps follows from its
// number, so the constants are made once.
struct Transpose {
  unsigned int bytes16, bytes8;    // __byte_perm selectors
  unsigned int rot4, rot2, rot1;   // left rotations
  unsigned int keep4, keep2, keep1;

  __device__ __forceinline__ Transpose() {
    const unsigned int lane = threadIdx.x & 31;
    bytes16 = lane & 16 ? 0x3276u : 0x5410u;
    bytes8 = lane & 8 ? 0x3715u : 0x6240u;
    rot4 = lane & 4 ? 28 : 4;
    rot2 = lane & 2 ? 30 : 2;
    rot1 = lane & 1 ? 31 : 1;
    keep4 = lane & 4 ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
    keep2 = lane & 2 ? 0xCCCCCCCCu : 0x33333333u;
    keep1 = lane & 1 ? 0xAAAAAAAAu : 0x55555555u;
  }
  __device__ __forceinline__ static unsigned int swap(unsigned int x, int j, unsigned int rot, unsigned int keep) {
    const unsigned int y = __shfl_xor_sync(kFull, x, j);
    return (x & keep) | (__funnelshift_l(y, y, rot) & ~keep);
  }
  __device__ __forceinline__ unsigned int operator()(unsigned int x) const {
    x = __byte_perm(x, __shfl_xor_sync(kFull, x, 16), bytes16);
    x = __byte_perm(x, __shfl_xor_sync(kFull, x, 8), bytes8);
    x = swap(x, 4, rot4, keep4);
    x = swap(x, 2, rot2, keep2);
    return swap(x, 1, rot1, keep1);
  }
};

// PW columns by 32 / PW rows (or planes, if DEEP) of outputs.
template <typename T, int PW, bool DEEP, bool DROPS>
struct PatchWalk {
  static constexpr int PZ = DEEP ? 32 / PW : 1;
  static constexpr int PH = DEEP ? 1 : 32 / PW;

  const HistArgs& a;
  const uint16_t* codes;  // rank of each support sample (or a dropped code)
  const uint16_t* place;  // support index of each rank (65535 up to 32 before and after)
  const Support<T>& sup;
  int lx, ly, lz;         // the lane's output within the patch
  int px, py, pz;         // the patch's first column, row and plane in the tile
  int t;                  // threshold rank
  int below, dropped;     // the lane's window: samples of rank below t, dropped samples
  Transpose transpose;

  // Add to the lane's counts those of two support rows (`width` columns from
  // px + lx), negated for the first if FLIP; `first` and `second` say whether
  // the rows lie in (or leave and enter) the lane's window. `row` is the first
  // one's start, the second lies `apart` codes further.
  template <bool FLIP>
  __device__ __forceinline__ void add_rows(const uint16_t* row, int width, int apart, bool first, bool second) {
    const uint16_t* at = row + px + (threadIdx.x & 31);
    int u = at[0], v = at[apart];
    unsigned int a0 = __ballot_sync(kFull, u < t), b0 = __ballot_sync(kFull, v < t), c0 = 0, d0 = 0;
    if (DROPS) {
      c0 = __ballot_sync(kFull, u >= (int)kPropagated);
      d0 = __ballot_sync(kFull, v >= (int)kPropagated);
    }
    int na = 0, nb = 0, nc = 0, nd = 0;
    int left = width;
#pragma unroll 1
    for (; left >= 32; left -= 32) {
      at += 32;
      u = at[0];
      v = at[apart];
      const unsigned int a1 = __ballot_sync(kFull, u < t), b1 = __ballot_sync(kFull, v < t);
      na += __popc(__funnelshift_r(a0, a1, lx));
      nb += __popc(__funnelshift_r(b0, b1, lx));
      a0 = a1;
      b0 = b1;
      if (DROPS) {
        const unsigned int c1 = __ballot_sync(kFull, u >= (int)kPropagated);
        const unsigned int d1 = __ballot_sync(kFull, v >= (int)kPropagated);
        nc += __popc(__funnelshift_r(c0, c1, lx));
        nd += __popc(__funnelshift_r(d0, d1, lx));
        c0 = c1;
        d0 = d1;
      }
    }
    if (left > 0) {
      const unsigned int mask = (1u << left) - 1u;
      unsigned int a1 = 0, b1 = 0, c1 = 0, d1 = 0;
      if (left + PW - 1 > 32) {
        u = at[32];
        v = at[apart + 32];
        a1 = __ballot_sync(kFull, u < t);
        b1 = __ballot_sync(kFull, v < t);
        if (DROPS) {
          c1 = __ballot_sync(kFull, u >= (int)kPropagated);
          d1 = __ballot_sync(kFull, v >= (int)kPropagated);
        }
      }
      na += __popc(__funnelshift_r(a0, a1, lx) & mask);
      nb += __popc(__funnelshift_r(b0, b1, lx) & mask);
      if (DROPS) {
        nc += __popc(__funnelshift_r(c0, c1, lx) & mask);
        nd += __popc(__funnelshift_r(d0, d1, lx) & mask);
      }
    }
    below += (second ? nb : 0) + (first ? (FLIP ? -na : na) : 0);
    if (DROPS) dropped += (second ? nd : 0) + (first ? (FLIP ? -nc : nc) : 0);
  }

  // Whether the lane's window holds plane pz + dz of the support.
  __device__ __forceinline__ bool in_depth(int dz) const { return !DEEP || (unsigned)(dz - lz) < (unsigned)a.g.kd; }

  // Support planes that the patch's windows reach (tiles of fewer planes than a
  // patch end earlier; the lanes beyond have no output).
  __device__ __forceinline__ int depth() const { return DEEP ? min(a.g.kd + PZ - 1, a.SZ - pz) : 1; }

  // Count the whole windows, two rows at a time (the row after the last is
  // read but lies in no window; it ends within the places that follow).
  __device__ __forceinline__ void count_all() {
    below = dropped = 0;
    for (int dz = 0; dz < depth(); ++dz) {
      const uint16_t* row = codes + (pz + dz) * a.plane + py * a.SW;
      const bool deep = in_depth(dz);
      for (int q = 0; q < a.g.kh + PH - 1; q += 2, row += 2 * a.SW)
        add_rows<false>(row, a.g.kw, a.SW, deep && (unsigned)(q - ly) < (unsigned)a.g.kh,
                        deep && (unsigned)(q + 1 - ly) < (unsigned)a.g.kh);
    }
  }

  // Move the windows down by the patch height or, those of a patch of one row, along
  // it by the patch width: of each support row 32 columns leave and 32 enter.
  __device__ __forceinline__ void move(bool sideways) {
    if (PW == 32) {
      const uint16_t* row = codes + py * a.SW;
      const int rows = sideways ? a.g.kh : 1, width = sideways ? PW : a.g.kw, apart = sideways ? a.g.kw : a.g.kh * a.SW;
#pragma unroll 1
      for (int q = 0; q < rows; ++q, row += a.SW) add_rows<true>(row, width, apart, true, true);
      if (sideways)
        px += PW;
      else
        py += PH;
      return;
    }
    for (int dz = 0; dz < depth(); ++dz) {
      const uint16_t* row = codes + (pz + dz) * a.plane + py * a.SW;
      const bool deep = in_depth(dz);
#pragma unroll 1
      for (int q = 0; q < 2 * PH - 1; ++q, row += a.SW) {
        const bool mine = deep && (PH == 1 || (unsigned)(q - ly) < (unsigned)PH);
        add_rows<true>(row, a.g.kw, a.g.kh * a.SW, mine, mine);
      }
    }
    py += PH;
  }

  // Which of the ranks [start, start + 32) the lane's window holds (bit i:
  // rank start + i). Ranks outside the support are in no window.
  __device__ __forceinline__ unsigned int ranks_in(int start) const {
    unsigned int e = place[start + (int)(threadIdx.x & 31)];
    int dz = 0;
    if (DEEP) {
      // (The planes end below 65535, so its plane is in no window.)
      const int sz = (int)__umulhi(e, a.plane_magic);
      e -= sz * a.plane;
      dz = sz - pz;
    }
    const int sy = (int)__umulhi(e, a.row_magic);
    const int dx = (int)e - sy * a.SW - px, dy = sy - py;
    bool in = (unsigned)dx < (unsigned)(a.g.kw + PW - 1) && (unsigned)dy < (unsigned)(a.g.kh + PH - 1);
    if (DEEP) in = in && (unsigned)dz < (unsigned)(a.g.kd + PZ - 1);
    if (!__any_sync(kFull, in)) return 0u;
    unsigned int lanes = 0;
    if (in) {
      // Columns dx - kw + 1 .. dx and rows dy - kh + 1 .. dy (planes, if deep)
      // of the patch.
      const int cl = max(dx - a.g.kw + 1, 0), ch = min(dx, PW - 1);
      lanes = bit_run(cl, ch - cl + 1);
      if (PW < 32) {
        static_assert(PW == 8 || PW == 32, "column masks are repeated per byte");
        lanes *= 0x01010101u;
        const int d = DEEP ? dz : dy, k = DEEP ? a.g.kd : a.g.kh;
        const int rl = max(d - k + 1, 0), rh = min(d, 32 / PW - 1);
        lanes &= bit_run(rl * PW, (rh - rl + 1) * PW);
      }
    }
    return transpose(lanes);
  }

  // Move the threshold to rank `to` (the counts follow).
  __device__ __forceinline__ void move_threshold(int to) {
    const int lo = min(t, to), hi = max(t, to);
    int count = 0;
    for (int start = lo; start < hi; start += 32) count += __popc(ranks_in(start) & bit_run(0, hi - start));
    below += to > t ? count : -count;
    t = to;
  }

  // The patch's order statistics: which ranks, and whether there is a value.
  // Lanes outside the image (`live` false) ask for nothing.
  __device__ __forceinline__ Ranks select(bool live) {
    const Reduce& r = a.r;
    Ranks o;
    const int volume = a.g.kd * a.g.kh * a.g.kw;
    o.n = volume - dropped;
    o.valid = live && !((!r.omit && dropped > 0) || (r.omit && o.n < r.min_count) || o.n == 0);
    int k1 = 0, k2;
    switch (r.kind) {
      case kRank:
      case kRankHistogram:
        o.valid = o.valid && r.param < o.n;
        k1 = o.valid ? (int)r.param : 0;
        break;
      case kMin:
        break;
      case kMax:
        k1 = o.n - 1;
        break;
      case kPercentile:
        if (r.q_is_max) {
          k1 = o.n - 1;
        } else {
          const PctSplit ps = pct_split(r, max(o.n, 1));
          k1 = ps.lower;
          o.two = ps.upper != ps.lower;
        }
        break;
      default:
        o.two = (o.n & 1) == 0;
        k1 = o.two ? o.n / 2 - 1 : o.n / 2;
    }
    k2 = k1 + (o.two ? 1 : 0);
    // The word that holds order statistic k starts at rank s and has it as
    // its k'-th set bit.
    int s1 = 0, s2 = 0, i1 = 0, i2 = 0;
    unsigned int w1 = 0, w2 = 0;
    const bool pairs = __any_sync(kFull, o.two);
    // Lanes without a value wait for nothing and find nothing.
    k1 = o.valid ? k1 : -1;
    k2 = o.valid ? k2 : -1;
    const int least = o.valid ? k1 : INT_MAX;
    auto look = [&](int start, int base, unsigned int word, int count) {
      if ((unsigned)(k1 - base) < (unsigned)count) {
        s1 = start;
        i1 = k1 - base;
        w1 = word;
      }
      if (pairs && (unsigned)(k2 - base) < (unsigned)count) {
        s2 = start;
        i2 = k2 - base;
        w2 = word;
      }
    };
    int base = below;
    for (int start = t; __any_sync(kFull, k2 >= base) && start < a.S; start += 32) {
      const unsigned int word = ranks_in(start);
      const int count = __popc(word);
      look(start, base, word, count);
      base += count;
    }
    base = below;
    for (int start = t; __any_sync(kFull, least < base) && start > 0;) {
      start -= 32;
      const unsigned int word = ranks_in(start);
      const int count = __popc(word);
      base -= count;
      look(start, base, word, count);
    }
    o.lo = s1 + select_in_word32(w1, i1);
    o.hi = o.two ? s2 + select_in_word32(w2, i2) : o.lo;
    return o;
  }

  // Walk `patches` patches from (px, py, pz) on, down the tile's rows or along one.
  __device__ __forceinline__ void walk(int patches, int tw_eff, int th_eff, int tz_eff, T* __restrict__ out) {
    const bool sideways = PW == 32 && a.sideways;
    // Counting whole windows costs kh + PH - 1 rows a plane, moving them down
    // 2 (2 PH - 1).
    const bool recount = !sideways && a.g.kh + PH - 1 <= 2 * (2 * PH - 1);
    Ranks held;
    T vl = 0, vh = 0;
    long long held_at = -1;
    for (int i = 1;; ++i) {
      if (i == 1 || recount) count_all();
      const bool live = px + lx < tw_eff && py + ly < th_eff && pz + lz < tz_eff;
      const Ranks o = select(live);
      // The previous patch's samples have arrived by now.
      if (held_at >= 0) out[held_at] = canonical(hist_value<T>(held, a, vl, vh));
      held = o;
      held_at = live ? ((long long)(pz + lz) * a.g.H + py + ly) * a.g.W + px + lx : -1;
      if (o.valid) {
        vl = sup.value(place[o.lo]);
        vh = o.two ? sup.value(place[o.hi]) : vl;
      }
      const int least = __reduce_min_sync(kFull, o.valid ? o.lo : INT_MAX);
      const int most = __reduce_max_sync(kFull, o.valid ? o.hi : -1);
      if (i == patches) {
        if (most >= 0) t = (least + most) >> 1;
        break;
      }
      if (recount) {
        if (most >= 0) t = (least + most) >> 1;
        py += PH;
      } else {
        if (most >= 0 && (t < least || t > most)) move_threshold((least + most) >> 1);
        move(sideways);
      }
    }
    if (held_at >= 0) out[held_at] = canonical(hist_value<T>(held, a, vl, vh));
  }
};

// Every patch of a tile: columns of patches split into runs of rows, or rows into
// runs of columns, so that the block's warps all have work. `out` is the tile's
// first output.
template <typename T, int PW, bool DEEP, bool DROPS>
__device__ __forceinline__ void walk_patches(const HistArgs& a, const uint16_t* codes, const uint16_t* place,
                                             const Support<T>& sup, int nret, int tw_eff, int th_eff, int tz_eff,
                                             T* __restrict__ out) {
  using Walk = PatchWalk<T, PW, DEEP, DROPS>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int across = (tw_eff + PW - 1) / PW, columns = across * ((tz_eff + Walk::PZ - 1) / Walk::PZ);
  const int rows = (th_eff + Walk::PH - 1) / Walk::PH;
  const bool sideways = PW == 32 && a.sideways;
  const int lines = sideways ? rows : columns, length = sideways ? across : rows;
  const int runs = min(length, max(1, kHWarps / lines));
  Walk p{a, codes, place, sup, lane % PW, DEEP ? 0 : lane / PW, DEEP ? lane / PW : 0, 0, 0, 0, 0, 0, 0};
  const Reduce& r = a.r;
  p.t = r.kind == kMin ? 0 : r.kind == kMax ? nret : r.kind == kPercentile ? (int)(nret * r.q_fraction) : nret / 2;
  if (r.kind == kRank || r.kind == kRankHistogram)
    p.t = (int)min((long long)nret, r.param * nret / max(1, a.g.kd * a.g.kh * a.g.kw));
  for (int item = warp; item < lines * runs; item += kHWarps) {
    const int run = item / lines, line = item - run * lines;
    const int begin = length * run / runs, end = length * (run + 1) / runs;
    if (sideways) {
      p.px = begin * PW;
      p.py = line;
    } else {
      const int deep = line / across;
      p.px = (line - deep * across) * PW;
      p.pz = deep * Walk::PZ;
      p.py = begin * Walk::PH;
    }
    p.walk(end - begin, tw_eff, th_eff, tz_eff, out);
  }
}

// One output tile (index `tile` of the plan's tile list) of the sliding
// rank-histogram filter: gather the support, rank it, slide. `scratch_slot`
// is the calling block's sort slot; `smem` the dynamic shared memory, whose
// footprint-list region the caller has filled for FP windows.
template <typename T, bool SDEC, bool FP>
__device__ __forceinline__ void histogram_tile(const T* __restrict__ in, T* __restrict__ out, const HistArgs& a,
                                               long long tile, unsigned char* scratch_slot, unsigned char* smem) {
  using K = typename KeyOf<T>::K;
  const K kSent = KeyOf<T>::kSentinel;
  const Geom3& g = a.g;
  const int S = a.S;
  // Shared memory. Footprints: rank codes [S] u16 | run lists | decode table
  // [S] keys (SDEC) | work (the axis maps while gathering, radix tables during
  // the sort, half-warp histograms while sliding). Boxes: axis maps | rank codes
  // [S + 64] u16 (patches read up to 32 codes past a row's end, and the row
  // after the last) | places of the ranks [32 + S + 32] u16 (no window holds
  // the outer ones) | key bits [S] u16 and counters of the sort in shared
  // memory. A sort through a slot has its counters where the codes come.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long map_bytes = FP ? 0 : axis_map_bytes(a.SH, a.SZ, a.SW, a.column_map);
  uint16_t* codes_s = reinterpret_cast<uint16_t*>(smem + map_bytes);
  const long long code_bytes = align16((long long)(FP ? a.S : a.S + 64) * 2);
  const long long list_bytes = FP ? align16((long long)(a.nf + 2 * a.nv + 2 * a.nh) * 2) : code_bytes;
  uint16_t* lists_s = reinterpret_cast<uint16_t*>(smem + map_bytes + code_bytes);
  uint16_t* place_s = lists_s + 32;
  unsigned char* rest = smem + map_bytes + code_bytes + list_bytes;
  K* decode_s = reinterpret_cast<K*>(rest);
  unsigned int* work = reinterpret_cast<unsigned int*>(
      FP ? rest + (SDEC ? align16((long long)a.S * sizeof(K)) : 0) : smem + map_bytes);
  const long long tz = tile / a.tiles_yx, z = tz * a.TZ;
  const long long tyx = tile - tz * a.tiles_yx;
  const long long y0 = (tyx / a.tiles_x) * a.TH;
  const long long x0 = (tyx % a.tiles_x) * a.TW;
  long long* maps = reinterpret_cast<long long*>(FP ? reinterpret_cast<unsigned char*>(work) : smem);
  Support<T> sup{a, in, maps, maps + a.SH + a.SZ, x0, (T)a.r.cval};
  sup.build(z, y0);
  __syncthreads();
  const uint16_t dropped = a.r.omit ? kOmitted : kPropagated;
  K k_and = kSent, k_or = 0;
  int sent = 0;
  auto note = [&](K key) {
    if (key != kSent) {
      k_and &= key;
      k_or |= key;
    } else {
      ++sent;
    }
  };
  SortedKeys<K> sorted{nullptr, 0};
  if (!FP && a.in_smem) {
    sup.each([&](int, K key) { note(key); });
    const KeyBits<K> bits = block_bits<K>(k_and, k_or, sent, S);
    sent = bits.sent;
    uint16_t* seg = reinterpret_cast<uint16_t*>(rest);
    unsigned int* table = reinterpret_cast<unsigned int*>(rest + align16((long long)S * 2));
    sort_in_smem<T>(sup, codes_s, place_s, seg, table, bits.varying);
    if (sent > 0) {
      sup.each([&](int e, K key) { seg[e] = key == kSent ? 1 : 0; });
      __syncthreads();
    }
    for (int r = threadIdx.x; r < S; r += blockDim.x) {
      // A dropped sample (its key can tie with the largest retained one's
      // sorted bits) lies in no window: place 65535 is below the last row.
      const uint16_t e = place_s[r];
      const bool drop = sent > 0 && seg[e] != 0;
      codes_s[e] = drop ? dropped : (uint16_t)r;
      if (drop) place_s[r] = 0xFFFF;
    }
  } else {
    Slot<K> slot = slot_at<K>(scratch_slot, S);
    const unsigned long long keep = keep_policy();
    sup.each([&](int e, K key) {
      st_keep(slot.a + e, Entry<K>{key, (K)e}, keep);
      note(key);
    });
    const KeyBits<K> bits = block_bits<K>(k_and, k_or, sent, S);
    sent = bits.sent;
    // Sort keys (LSD over the bits on which the retained keys differ). The
    // dropped samples' all-ones keys take part like any other key: an LSD
    // sort orders the retained keys among themselves whatever lies between
    // them, and a dropped sample's position is never set in a histogram.
    Entry<K>* src = slot.a;
    Entry<K>* dst = slot.b;
    if (bits.varying != 0) {
      const int lo = lowest_set(bits.varying), hi = highest_set(bits.varying);
      // The fewest passes, with the smallest digits that still cover the bits.
      const int passes = (hi - lo + a.digit_bits) / a.digit_bits;
      const int digits = max(5, (hi - lo + passes) / passes);
      const int nd = 1 << digits;
      const K mask = (K)(nd - 1);
      for (int shift = lo; shift <= hi; shift += digits) {
        radix_pass<K>(src, dst, S, work, work + kHWarps * nd, nd,
                      [shift, mask](K key) { return (unsigned int)((key >> shift) & mask); }, keep);
        Entry<K>* t = src;
        src = dst;
        dst = t;
      }
    }
    for (int pos = threadIdx.x; pos < S; pos += blockDim.x) {
      const Entry<K> e = ld_keep(src + pos, keep);
      const K key = e.key;
      const uint16_t at = (uint16_t)e.at;
      codes_s[at] = key == kSent ? dropped : (uint16_t)pos;
      if (!FP) place_s[pos] = key == kSent ? (uint16_t)0xFFFF : at;
      if (SDEC) decode_s[pos] = key;
    }
    sorted = {SDEC ? decode_s : &src->key, SDEC ? 1 : 2};
  }
  if (!FP && threadIdx.x < 64) lists_s[threadIdx.x < 32 ? (int)threadIdx.x : S + (int)threadIdx.x] = 0xFFFF;
  __syncthreads();
  const int th_eff = (int)min((long long)a.TH, g.H - y0);
  const int tw_eff = (int)min((long long)a.TW, g.W - x0);
  T* plane_out = out + z * g.H * g.W;
  if constexpr (!FP) {
    const int tz_eff = (int)min((long long)a.TZ, g.D - z);
    auto walk_all = [&](auto width, auto deep, auto drops) {
      walk_patches<T, decltype(width)::value, decltype(deep)::value, decltype(drops)::value>(
          a, codes_s, place_s, sup, S - sent, tw_eff, th_eff, tz_eff, plane_out + y0 * g.W + x0);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    using P8 = std::integral_constant<int, 8>;
    using P32 = std::integral_constant<int, 32>;
    if (g.kd > 1)
      sent > 0 ? walk_all(P8{}, Yes{}, Yes{}) : walk_all(P8{}, Yes{}, No{});
    else if (a.patch_w == 8)
      sent > 0 ? walk_all(P8{}, No{}, Yes{}) : walk_all(P8{}, No{}, No{});
    else
      sent > 0 ? walk_all(P32{}, No{}, Yes{}) : walk_all(P32{}, No{}, No{});
  } else {
    // Slide: each half-warp walks its columns in boustrophedon order.
    const int seg = threadIdx.x / kSeg;
    SegHist h;
    h.words = work + seg * a.words;
    h.nwords = a.words;
    h.m = 0;
    h.lt = 0;
    h.count = 0;
    h.nan = 0;
    for (int i = seg_lane(); i < a.words; i += kSeg) h.words[i] = 0u;
    __syncwarp();
    // Both halves of a warp have columns iff the warp's first column is in
    // the tile's valid width; whole warps beyond it sit out.
    const int warp_first = (threadIdx.x / 32) * 2 * a.cols_per_warp;
    if (warp_first < tw_eff) {
      if (!a.r.omit)
        walk<T, true>(codes_s, lists_s, seg * a.cols_per_warp, a.cols_per_warp, tw_eff, th_eff, a.SW, y0, x0, g, a,
                      sorted, plane_out, h);
      else
        walk<T, false>(codes_s, lists_s, seg * a.cols_per_warp, a.cols_per_warp, tw_eff, th_eff, a.SW, y0, x0, g, a,
                       sorted, plane_out, h);
    }
  }
  __syncthreads();
}

// Copy a footprint window's run lists into their shared-memory region (made
// visible by the first barrier of the next tile).
__device__ __forceinline__ void load_lists(const HistArgs& a, unsigned char* smem) {
  uint16_t* lists_s = reinterpret_cast<uint16_t*>(smem + align16((long long)a.S * 2));
  const int n = a.nf + 2 * a.nv + 2 * a.nh;
  for (int i = threadIdx.x; i < n; i += blockDim.x) lists_s[i] = a.lists[i];
}

template <typename T, bool SDEC, bool FP>
__global__ void __launch_bounds__(kHThreads, FP ? 1 : 2)
    histogram_kernel(const T* __restrict__ in, T* __restrict__ out, const __grid_constant__ HistArgs a,
                     unsigned char* scratch) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (FP) load_lists(a, smem);
  unsigned char* slot = scratch + (long long)blockIdx.x * a.slot_bytes;
  for (long long tile = blockIdx.x; tile < a.tiles; tile += gridDim.x)
    histogram_tile<T, SDEC, FP>(in, out, a, tile, slot, smem);
}

// Batched images (float32): one persistent launch walks the concatenated
// tile lists of every image of a family (same SDEC / FP variant); a block
// finds a tile's image by binary search over the images' first tiles and
// keeps that image's arguments in shared memory until the image changes.
struct HistTask {
  const float* in;
  float* out;
  long long first_tile;
  HistArgs a;
};

template <bool SDEC, bool FP>
__global__ void __launch_bounds__(kHThreads, FP ? 1 : 2)
    histogram_family_kernel(const HistTask* __restrict__ tasks, int ntasks, long long total_tiles,
                            unsigned char* scratch, long long slot_bytes) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ HistTask task;
  __shared__ int current, found;
  if (threadIdx.x == 0) current = -1;
  __syncthreads();
  unsigned char* slot = scratch + (long long)blockIdx.x * slot_bytes;
  for (long long tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
    if (threadIdx.x == 0) {
      int lo = 0, hi = ntasks - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].first_tile <= tile)
          lo = mid;
        else
          hi = mid - 1;
      }
      found = lo;
    }
    __syncthreads();
    const int index = found;
    if (index != current) {
      const long long* src = reinterpret_cast<const long long*>(tasks + index);
      long long* dst = reinterpret_cast<long long*>(&task);
      for (int i = threadIdx.x; i < (int)(sizeof(HistTask) / 8); i += blockDim.x) dst[i] = src[i];
      __syncthreads();
      if (FP) load_lists(task.a, smem);
      if (threadIdx.x == 0) current = index;
    }
    __syncthreads();
    histogram_tile<float, SDEC, FP>(task.in, task.out, task.a, tile - task.first_tile, slot, smem);
  }
}

struct HistChoice {
  int TW = 0, TH = 0, TZ = 1;
  bool sdec = false;     // footprints: sorted keys in shared memory
  bool in_smem = false;  // boxes: sorted in shared memory
  bool column_map = false;
  size_t smem = 0;
};

constexpr size_t kSmemBudget = 225 * 1024;
constexpr size_t kSmemPair = 113 * 1024 - 640;  // two blocks per SM (with 1 KB and the static variables each)

// Run-list entries of a footprint window (0 for a rectangular one).
struct Runs {
  int nf = 0, nv = 0, nh = 0;
  bool footprint = false;
  int entries() const { return footprint ? nf + 2 * nv + 2 * nh : 0; }
};

// Footprints: bytes of the work region, the largest of its three uses in turn:
// the axis maps while gathering, the sort's 8-bit-digit tables, and the
// segments' bit histograms while sliding. (Supports of two wide rows need 8 bytes
// a column for the maps and for the histograms alike, and the maps the offsets of
// the rows besides.)
size_t work_bytes_for(int SH, int SZ, int SW, bool column_map) {
  const size_t maps = (size_t)axis_map_bytes(SH, SZ, SW, column_map);
  const size_t sort = (size_t)sort_table_words(256) * 4;
  const size_t hist = (size_t)kSegs * (((long long)SZ * SH * SW + 31) / 32) * 4;
  return std::max(maps, std::max(sort, hist));
}

size_t footprint_smem(int SH, int SZ, int SW, bool column_map, bool sdec, size_t key_bytes, const Runs& runs) {
  const long long S = (long long)SZ * SH * SW;
  const size_t codes = (size_t)align16(S * 2);
  const size_t lists = (size_t)align16((long long)runs.entries() * 2);
  const size_t decode = sdec ? (size_t)align16(S * (long long)key_bytes) : 0;
  return codes + lists + decode + work_bytes_for(SH, SZ, SW, column_map);
}

size_t box_smem(const Geom3& g, int tw, int th, int tz, bool column_map, bool in_smem) {
  const int SH = th + g.kh - 1, SW = tw + g.kw - 1, SZ = tz + g.kd - 1;
  const long long S = (long long)SZ * SH * SW;
  const size_t maps = (size_t)axis_map_bytes(SH, SZ, SW, column_map), codes = 2 * (size_t)align16((S + 64) * 2);
  if (in_smem) return maps + codes + (size_t)align16(S * 2) + (size_t)kCounterWords * 4;
  return maps + std::max(codes, (size_t)sort_table_words(256) * 4);
}

// Sorts through a slot take digits of up to 11 bits (three passes cover 32
// varying bits) as far as their tables fit in the bytes they share.
int slot_digit_bits(size_t room) {
  int bits = 8;
  while (bits < 11 && (size_t)sort_table_words(2 << bits) * 4 <= room) ++bits;
  return bits;
}

// Count the taps and the vertical and horizontal runs (within each plane)
// of a kd x kh x kw footprint mask (row-major).
Runs count_runs(const std::vector<uint8_t>& mask, int kd, int kh, int kw) {
  Runs r;
  r.footprint = true;
  for (int zz = 0; zz < kd; ++zz)
    for (int y = 0; y < kh; ++y)
      for (int x = 0; x < kw; ++x) {
        const size_t at = ((size_t)zz * kh + y) * kw + x;
        if (!mask[at]) continue;
        ++r.nf;
        if (y == 0 || !mask[at - kw]) ++r.nv;
        if (x == 0 || !mask[at - 1]) ++r.nh;
      }
  return r;
}

// The patch width of a box window's tile of height th: rows of 32 outputs
// where a tile has single rows, else 8 columns.
int patch_width(const Geom3& g, int th) { return th % 4 != 0 && g.kd == 1 ? 32 : 8; }

// The walk over a box window's tile in warp instructions (measured on windows
// from 13 x 13 to 129 x 129 and 9 x 33 x 33): pairs of rows counted per patch, and
// the ranks looked through, which grow with the support over the window and with
// the spread of the patch's order statistics (that of windows shifted across the
// patch, for independent samples, and 1% of the support for a slope). Patches of one
// row are walked along it where the windows are so wide that moving them beats
// counting them again. (Counted anew for every patch, a median over 20,001 samples of
// a line of 2^20 took 1.01 ms and one of 2 x 10001 over 512 x 2048 11.5 ms, the
// latter in tiles of at most 128 columns too; walked along rows of up to 1,024
// columns 0.24 and 1.03.)
struct BoxWalk {
  double cost;
  bool sideways;
};

BoxWalk box_walk(const Geom3& g, int tw, int th, int tz, double S) {
  const int pw = patch_width(g, th), lines = 32 / pw;
  const bool deep = g.kd > 1;
  const int ph = deep ? 1 : lines, pz = deep ? lines : 1;
  const double outputs = (double)tw * th * tz, volume = (double)g.kd * g.kh * g.kw;
  const double words = (g.kw + pw - 1 + 31) / 32;
  const double pair = 20.0 * words + 25.0;
  const double planes = g.kd + pz - 1;
  const double shifted = deep ? (double)g.kh * g.kw * (pz - 1) : (double)g.kw * (ph - 1);
  const double moves = std::min(std::sqrt(0.5 * ((double)g.kd * g.kh * (pw - 1) + shifted)), 1.5 * std::sqrt(volume));
  const double ranks = std::min(S, 1.6 * moves * S / volume + 0.01 * S);
  const double patches = outputs / 32.0 * (deep ? (double)pz * ((tz + pz - 1) / pz) / tz : 1.0);
  // Patches in `lines` lines of `length`, whose first one costs `all` pairs of rows
  // and the others `moved`, or `all` too if those are fewer.
  auto walk = [&](double lines, double length, double all, double moved) {
    const double runs = std::min(length, std::max(1.0, kHWarps / lines));
    const double steps = std::max(1.0, length / runs);
    const double pairs = std::min(all, moved + all / steps);
    const double idle = std::max(1.0, kHWarps / (lines * runs));
    return idle * patches * (pairs * pair + 65.0 * (ranks / 32.0 + 2.0) + 250.0);
  };
  const double across = tw / pw, columns = across * ((tz + pz - 1) / pz), rows = std::max(1, th / ph);
  const double down = walk(columns, rows, planes * (g.kh + ph - 1) / 2, planes * (2 * ph - 1));
  if (pw != 32) return {down, false};
  // Moving a patch along its row counts two words of each support row.
  const double right = walk(rows, across, (g.kh + 1) / 2, g.kh * 65.0 / pair);
  return {std::min(down, right), right < down};
}

// Pick the output tile by a cost model: for boxes in warp instructions, the walk's
// and the block sort's (13 per support sample in shared memory, 29 through a slot, and
// a share of the passes' scans and barriers per tile); for footprints in
// units of one histogram update per output: vertical steps, the first window
// of each segment's walk, the column moves, the block sort (about 8 units per
// support sample) and a global decode when the sorted keys do not fit in
// shared memory. Or the given tw x th when it fits (an autotuner candidate; 0
// when it does not).
HistChoice choose_tile(const Geom3& g, size_t key_bytes, int sm_count, const Runs& runs = Runs{}, int force_tw = 0,
                       int force_th = 0) {
  HistChoice best;
  if ((long long)g.kw > kMaxSupport || (long long)g.kh > kMaxSupport || (long long)g.kd > kMaxSupport)
    return best;
  double best_cost = 1e300;
  // Columns go through a table, but for single rows and where no tile has room for
  // one: 8 bytes a column beside the 4 of each sample's code and place would shut
  // out boxes of two rows beyond 14,350 columns and of three beyond 11,473, which fit
  // without it (up to some 28,000 and 19,000).
  bool tables = true;
  auto consider = [&](int tw, int th, int tz = 1) {
    const int SH = th + g.kh - 1, SZ = tz + g.kd - 1, SW = tw + g.kw - 1;
    const long long S = (long long)SZ * SW * SH;
    if (S > kMaxSupport) return;
    const bool column_map = tables && SH * SZ > 1;
    if (runs.footprint) {
      for (int sdec = 1; sdec >= 0; --sdec) {
        const size_t smem = footprint_smem(SH, SZ, SW, column_map, sdec != 0, key_bytes, runs);
        if (smem > kSmemBudget) continue;
        const double cpw = (tw + kSegs - 1) / kSegs;
        const double outputs = (double)tw * th;
        double cost = 2.0 * runs.nv + runs.nf / (cpw * th) + 2.0 * runs.nh / th + 8.0 * (double)S / outputs +
                      (sdec ? 0.0 : 12.0);
        if (smem * 2 <= kSmemBudget) cost *= 0.9;  // two resident blocks per SM
        if (cost < best_cost) {
          best_cost = cost;
          best.TW = tw;
          best.TH = th;
          best.sdec = sdec != 0;
          best.column_map = column_map;
          best.smem = smem;
        }
        return;
      }
      return;
    }
    if (box_smem(g, tw, th, tz, column_map, false) > kSmemBudget) return;
    // Tiles that an SM takes one after the other, whole ones: small arrays
    // prefer tiles that leave no SM idle. Two resident blocks overlap.
    const double tiles = (double)((g.W + tw - 1) / tw * ((g.H + th - 1) / th) * ((g.D + tz - 1) / tz));
    const double turns = std::ceil(tiles / std::max(1, sm_count));
    if (turns * (turns > 1 ? 0.75 : 1.0) * (13.0 * (double)S + 12000.0) >= best_cost) return;  // the sort alone
    const double walk = box_walk(g, tw, th, tz, (double)S).cost;
    for (int in_smem = 1; in_smem >= 0; --in_smem) {
      const size_t smem = box_smem(g, tw, th, tz, column_map, in_smem != 0);
      if (smem > kSmemBudget) continue;
      const double cost = turns * (smem <= kSmemPair && turns > 1 ? 0.75 : 1.0) *
                          ((in_smem ? 13.0 : 29.0) * (double)S + 12000.0 + walk);
      if (cost < best_cost) {
        best_cost = cost;
        best.TW = tw;
        best.TH = th;
        best.TZ = tz;
        best.in_smem = in_smem != 0;
        best.column_map = column_map;
        best.smem = smem;
      }
    }
  };
  if (force_tw > 0) {
    consider(force_tw, force_th);
    return best;
  }
  if (g.H == 1 && g.kh == 1) {
    for (int tw : {8192, 4096, 2048, 1024, 512, 256, 128, 64, 32})
      if (tw <= 32 || tw / 2 < g.W) consider(tw, 1);
    return best;
  }
  auto consider_all = [&] {
    // Flat windows thousands of columns wide: longer rows share their support among
    // more outputs.
    if (!runs.footprint && g.kd == 1 && g.kw >= 1024)
      for (int tw : {1024, 512, 256})
        for (int th : {1, 2})
          if (tw / 2 < g.W && th <= g.H) consider(tw, th);
    for (int tw : {128, 64, 32, 16}) {
      if (tw > 32 && tw / 2 >= g.W) continue;
      if (tw == 16 && (runs.footprint || g.kd == 1)) continue;
      for (int th : {256, 192, 128, 96, 64, 48, 32, 16, 8, 4, 2, 1}) {
        if (th > 1 && th / 2 >= g.H) continue;
        consider(tw, th);
      }
      if (runs.footprint) continue;
      // Boxes also take the heights between, where a support just fits, and deep
      // ones several planes.
      for (int th = 120; th > 8; th -= 4)
        if (th / 2 < g.H) consider(tw, th);
      if (g.kd > 1)
        for (int tz : {2, 4, 8, 16})
          for (int th = 64; th >= 4; th -= 4)
            if (th / 2 < g.H && tz / 2 < g.D) consider(tw, th, tz);
    }
  };
  consider_all();
  if (best.TW == 0) {
    tables = false;
    consider_all();
  }
  return best;
}

HistArgs make_args_core(const Geom3& g, const HistChoice& c, int dtype, const Runs& runs, const Reduce& r) {
  HistArgs a{};
  a.g = g;
  a.TW = c.TW;
  a.TH = c.TH;
  a.SW = a.TW + a.g.kw - 1;
  a.SH = a.TH + a.g.kh - 1;
  a.TZ = c.TZ;
  a.SZ = a.TZ + a.g.kd - 1;
  a.plane = a.SW * a.SH;
  a.S = a.SZ * a.plane;
  a.tiles_x = (a.g.W + a.TW - 1) / a.TW;
  a.tiles_yx = a.tiles_x * ((a.g.H + a.TH - 1) / a.TH);
  a.tiles = a.tiles_yx * ((a.g.D + a.TZ - 1) / a.TZ);
  a.cols_per_warp = (a.TW + kSegs - 1) / kSegs;  // columns per half-warp segment
  a.words = (a.S + 31) / 32;
  a.slot_bytes = dtype == 0 ? slot_bytes_for<uint32_t>(a.S) : slot_bytes_for<unsigned long long>(a.S);
  a.in_smem = c.in_smem;
  a.column_map = c.column_map;
  a.digit_bits = c.in_smem ? kDigitBits
                           : slot_digit_bits(runs.footprint
                                                 ? work_bytes_for(a.SH, a.SZ, a.SW, c.column_map)
                                                 : c.smem - (size_t)axis_map_bytes(a.SH, a.SZ, a.SW, c.column_map));
  a.patch_w = patch_width(g, c.TH);
  a.sideways = !runs.footprint && box_walk(g, c.TW, c.TH, c.TZ, a.S).sideways;
  a.plane_magic = (unsigned int)(((1ull << 32) + a.plane - 1) / (unsigned long long)a.plane);
  a.row_magic = (unsigned int)(((1ull << 32) + a.SW - 1) / (unsigned long long)a.SW);
  a.r = r;
  a.lists = nullptr;
  a.nf = runs.nf;
  a.nv = runs.nv;
  a.nh = runs.nh;
  return a;
}

Runs plan_runs(const Plan& p) {
  Runs runs;
  runs.footprint = p.hist_footprint;
  runs.nf = p.hist_nf;
  runs.nv = p.hist_nv;
  runs.nh = p.hist_nh;
  return runs;
}

HistChoice plan_choice(const Plan& p) {
  HistChoice c;
  c.TW = p.hist_block_w;
  c.TH = p.hist_block_h;
  c.TZ = p.hist_block_d;
  c.sdec = p.hist_sdec;
  c.in_smem = p.hist_in_smem;
  c.column_map = p.hist_column_map;
  c.smem = p.hist_smem;
  return c;
}

HistArgs make_args(const Plan& p) {
  HistArgs a = make_args_core(p.tile.g, plan_choice(p), p.dtype, plan_runs(p), p.r);
  if (p.hist_footprint) a.lists = p.d_hist_lists;
  return a;
}

template <typename T>
void* kernel_for(bool sdec, bool fp = false) {
  if (fp) return sdec ? (void*)histogram_kernel<T, true, true> : (void*)histogram_kernel<T, false, true>;
  return (void*)histogram_kernel<T, false, false>;
}

template <typename T>
cudaError_t launch_t(const Plan& p, const T* in, T* out, cudaStream_t s) {
  HistArgs a = make_args(p);
  // Sorts in shared memory: a block per tile; through slots: a block per slot.
  const long long grid = a.in_smem ? std::min<long long>(a.tiles, INT_MAX)
                                   : std::min<long long>(a.tiles, (long long)(p.scratch_bytes / (size_t)a.slot_bytes));
  if (grid < 1) return cudaErrorInvalidValue;
  unsigned char* scratch = (unsigned char*)p.d_scratch;
  const unsigned blocks = (unsigned)grid;
  if (p.hist_footprint) {
    if (p.hist_sdec)
      histogram_kernel<T, true, true><<<blocks, kHThreads, p.smem_bytes, s>>>(in, out, a, scratch);
    else
      histogram_kernel<T, false, true><<<blocks, kHThreads, p.smem_bytes, s>>>(in, out, a, scratch);
  } else {
    histogram_kernel<T, false, false><<<blocks, kHThreads, p.smem_bytes, s>>>(in, out, a, scratch);
  }
  return cudaGetLastError();
}

}  // namespace

namespace {

// The footprint of a plan as a kd x kh x kw mask in the tile's (z, y, x)
// orientation, from the taps' box positions (all ones for a box).
std::vector<uint8_t> footprint_mask(const Plan& p) {
  const Geom3& g = p.tile.g;
  std::vector<uint8_t> mask((size_t)g.kd * g.kh * g.kw, 0);
  for (int i = 0; i < p.r.count; ++i) {
    const int* bt = &p.box_taps[(size_t)i * 3];
    mask[((size_t)bt[0] * g.kh + bt[1]) * g.kw + bt[2]] = 1;
  }
  return mask;
}

// Run lists for footprint windows; none for boxes.
Runs runs_of(const Plan& p) {
  const Geom3& g = p.tile.g;
  if (p.footprint.empty()) return Runs{};
  if ((long long)g.kd * g.kh * g.kw > (1ll << 24)) return Runs{};  // too large to list
  return count_runs(footprint_mask(p), g.kd, g.kh, g.kw);
}

}  // namespace

bool histogram_configure(Plan& p, int tw, int th) {
  if (p.ndim > 3 || p.r.count < 1) return false;
  const int k = p.r.kind;
  if (k != kMedian && k != kMedianNetwork && k != kMedianHistogram && k != kRank &&
      k != kRankHistogram && k != kMin && k != kMax && k != kPercentile)
    return false;
  const Runs runs = runs_of(p);
  HistChoice c = choose_tile(p.tile.g, p.dtype == 0 ? 4 : 8, p.sm_count, runs, tw, th);
  if (c.TW == 0) return false;
  p.hist_block_w = c.TW;
  p.hist_block_h = c.TH;
  p.hist_block_d = c.TZ;
  p.hist_sdec = c.sdec;
  p.hist_in_smem = c.in_smem;
  p.hist_column_map = c.column_map;
  p.hist_smem = c.smem;
  p.hist_footprint = runs.footprint;
  p.hist_nf = runs.nf;
  p.hist_nv = runs.nv;
  p.hist_nh = runs.nh;
  p.hist_lists.clear();
  if (runs.footprint) {
    // Support-linear offsets (zz * plane + y * SW + x) of the taps and of
    // the run ends; below the support size, so they fit 16 bits.
    const Geom3& g = p.tile.g;
    const int SW = c.TW + g.kw - 1;
    const int plane = SW * (c.TH + g.kh - 1);
    const std::vector<uint8_t> mask = footprint_mask(p);
    auto at = [&](int zz, int y, int x) {
      return y >= 0 && y < g.kh && x >= 0 && x < g.kw && mask[((size_t)zz * g.kh + y) * g.kw + x] != 0;
    };
    std::vector<uint16_t> taps, top, bottom, left, right;
    for (int zz = 0; zz < g.kd; ++zz)
      for (int y = 0; y < g.kh; ++y)
        for (int x = 0; x < g.kw; ++x) {
          if (!at(zz, y, x)) continue;
          const uint16_t off = (uint16_t)(zz * plane + y * SW + x);
          taps.push_back(off);
          if (!at(zz, y - 1, x)) top.push_back(off);
          if (!at(zz, y + 1, x)) bottom.push_back(off);
          if (!at(zz, y, x - 1)) left.push_back(off);
          if (!at(zz, y, x + 1)) right.push_back(off);
        }
    // A step removes one list and adds the other; the pairing of entries
    // does not matter, only that both lists of an axis have one entry per run.
    p.hist_lists = taps;
    p.hist_lists.insert(p.hist_lists.end(), top.begin(), top.end());
    p.hist_lists.insert(p.hist_lists.end(), bottom.begin(), bottom.end());
    p.hist_lists.insert(p.hist_lists.end(), left.begin(), left.end());
    p.hist_lists.insert(p.hist_lists.end(), right.begin(), right.end());
  }
  HistArgs a = make_args(p);
  p.hist_blocks_x = a.tiles_x;
  p.hist_blocks_y = a.tiles / a.tiles_x;
  return true;
}

size_t histogram_smem(const Plan& p) { return p.hist_smem; }

// Scratch slots for a block sort through them: one per resident block
// (occupancy x SMs), capped by the number of tiles.
cudaError_t histogram_allocate(Plan& p) {
  HistArgs a = make_args(p);
  void* kernel = p.dtype == 0 ? kernel_for<float>(p.hist_sdec, p.hist_footprint)
                              : kernel_for<double>(p.hist_sdec, p.hist_footprint);
  cudaError_t e = allow_max_smem((const void*)kernel);
  if (e != cudaSuccess) return e;
  if (p.hist_footprint) {
    e = cudaMalloc(&p.d_hist_lists, p.hist_lists.size() * sizeof(uint16_t));
    if (e != cudaSuccess) return e;
    e = cudaMemcpy(p.d_hist_lists, p.hist_lists.data(), p.hist_lists.size() * sizeof(uint16_t),
                   cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) return e;
  p.scratch_bytes = 0;
  if (a.in_smem) return cudaSuccess;
  int per_sm = 1;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kHThreads, p.smem_bytes);
  if (e != cudaSuccess) return e;
  long long slots = std::min<long long>(a.tiles, (long long)std::max(per_sm, 1) * p.sm_count);
  p.scratch_bytes = (size_t)slots * (size_t)a.slot_bytes;
  return cudaMalloc(&p.d_scratch, p.scratch_bytes);
}

namespace {

int hist_family_variant(const Plan& p) {
  if (p.algo != Algo::kHistogram || p.dtype != 0) return -1;
  return p.hist_footprint ? (p.hist_sdec ? 3 : 2) : 0;
}

long long hist_family_tiles(const Plan& p) { return make_args(p).tiles; }

long long hist_family_slot_bytes(const Plan& p) { return p.hist_in_smem ? 0 : make_args(p).slot_bytes; }

void hist_family_write_task(const Plan& p, const void* in, void* out, long long first_tile, void* task) {
  HistTask t{};
  t.in = (const float*)in;
  t.out = (float*)out;
  t.first_tile = first_tile;
  t.a = make_args(p);
  std::memcpy(task, &t, sizeof(t));
}

const void* hist_family_kernel(int v) {
  switch (v) {
    case 0: return (const void*)histogram_family_kernel<false, false>;
    case 2: return (const void*)histogram_family_kernel<false, true>;
    default: return (const void*)histogram_family_kernel<true, true>;
  }
}

cudaError_t hist_family_launch(int v, const void* d_tasks, int ntasks, long long tiles, unsigned char* scratch,
                               long long slot_bytes, size_t smem, int grid, cudaStream_t s) {
  void* args[] = {(void*)&d_tasks, &ntasks, &tiles, &scratch, &slot_bytes};
  return cudaLaunchKernel(hist_family_kernel(v), dim3(grid), dim3(kHThreads), args, smem, s);
}

}  // namespace

const FamilyOps& histogram_family_ops() {
  static const FamilyOps ops{sizeof(HistTask), hist_family_variant, hist_family_tiles, hist_family_slot_bytes,
                             hist_family_write_task, hist_family_kernel, hist_family_launch};
  return ops;
}

cudaError_t launch_histogram(const Plan& p, const void* in, void* out, cudaStream_t s) {
  if (p.dtype == 0) return launch_t<float>(p, (const float*)in, (float*)out, s);
  return launch_t<double>(p, (const double*)in, (double*)out, s);
}


// ---------------------------------------------------------------------------
// Allocation-free variant of the histogram kernel.
//
// Some callers cannot let a library allocate device memory: code that runs
// while a CUDA stream is being captured (cudaMalloc is not allowed there),
// frameworks that own all device memory through their own pool, and real-time
// pipelines where an allocation's implicit device synchronization is not
// acceptable. For them, ndf_histogram_filter_noalloc takes the caller's
// device input and output and keeps its only scratch (the per-block sort
// slots) in the file-scope array below, so it never calls cudaMalloc,
// cudaFree or any allocating routine.
//
// Limits and sharing:
//  * the array holds kNoAllocScratchBytes (16 MiB) on every GPU that loads
//    the library, until the process exits;
//  * supports sorted in shared memory do not use it; for the others the number
//    of concurrently working thread blocks is the number of sort slots that
//    fit in it (a slot is 2 x S entries of a key and its index for a support
//    of S samples), capped by the device's resident capacity; a support whose
//    slot does not fit is rejected with NDF_ERR_MEMORY;
//  * every call shares the array and it keeps the last call's contents; the
//    kernel writes every slot word before reading it, so nothing needs
//    clearing; calls that overlap on the GPU (other streams, other host
//    threads) race on it and must be serialized by the caller;
//  * the first call on a device looks up the array's device address
//    (cudaGetSymbolAddress) with that device current; make that first call
//    before any stream capture;
//  * the address is kept for the life of the process: do not use the entry
//    point on a device after cudaDeviceReset (or another teardown of its
//    primary context), which can move the array.

constexpr size_t kNoAllocScratchBytes = 16u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {

constexpr int kMaxDevices = 64;

struct NoAllocDevices {
  std::mutex lock;
  void* address[kMaxDevices] = {};
};

NoAllocDevices& noalloc_devices() {
  static NoAllocDevices d;
  return d;
}

// Device address of g_noalloc_scratch on the current device (set-up once
// per device, with that device current).
cudaError_t noalloc_scratch(int device, void** out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  NoAllocDevices& d = noalloc_devices();
  std::lock_guard<std::mutex> guard(d.lock);
  if (!d.address[device]) {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    d.address[device] = ptr;
  }
  *out = d.address[device];
  return cudaSuccess;
}

int noalloc_fail(int code, const char* message) {
  return fail(code, message);
}

// a * b into *out; false when the product does not fit in 64 bits.
bool mul_fits(unsigned long long a, unsigned long long b, unsigned long long* out) {
  if (a != 0 && b > ~0ull / a) return false;
  *out = a * b;
  return true;
}

}  // namespace
}  // namespace ndf

extern "C" int ndf_histogram_filter_noalloc(const void* d_in, void* d_out, int32_t dtype, int32_t ndim,
                                            const uint64_t* shape, const uint64_t* size,
                                            const int64_t* origin, const int32_t* modes, double cval,
                                            int32_t kind, int32_t omit_nan, int32_t ignore_inf,
                                            uint64_t min_count, uint64_t parameter, double percentile,
                                            void* stream) {
  using namespace ndf;
  if (dtype != NDF_FLOAT32 && dtype != NDF_FLOAT64)
    return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION, "array dtype must be float32 or float64");
  if (ndim < 1 || ndim > 2)
    return noalloc_fail(NDF_ERR_UNSUPPORTED, "the allocation-free histogram filter takes 1-D or 2-D arrays");
  if (!shape || !size || !origin || !modes)
    return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION, "missing shape, size, origin or mode");
  if (kind != kMedian && kind != kMedianNetwork && kind != kMedianHistogram && kind != kRank &&
      kind != kRankHistogram && kind != kMin && kind != kMax && kind != kPercentile)
    return noalloc_fail(NDF_ERR_UNSUPPORTED, "the allocation-free histogram filter computes order statistics");
  long long shp[2] = {1, 1}, sz[2] = {1, 1}, org[2] = {0, 0};
  int md[2] = {kNearest, kNearest};
  const int pad = 2 - ndim;
  unsigned long long volume = 1, n_out = 1;
  for (int a = 0; a < ndim; ++a) {
    if (modes[a] < 0 || modes[a] > 4) return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION, "unsupported boundary mode");
    if (size[a] == 0) return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION, "window sizes must be positive");
    if (size[a] > 65534 || shape[a] > (1ull << 40))
      return noalloc_fail(NDF_ERR_OVERFLOW, "shape or index arithmetic overflowed");
    const long long length = (long long)size[a];
    if (origin[a] < -(length / 2) || origin[a] > (length - 1) / 2)
      return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION,
                          "origin must satisfy -(size // 2) <= origin <= (size - 1) // 2");
    shp[a + pad] = (long long)shape[a];
    sz[a + pad] = length;
    org[a + pad] = origin[a];
    md[a + pad] = modes[a];
    if (!mul_fits(volume, size[a], &volume) || !mul_fits(n_out, shape[a], &n_out))
      return noalloc_fail(NDF_ERR_OVERFLOW, "shape or index arithmetic overflowed");
  }
  if (omit_nan && (min_count == 0 || min_count > volume))
    return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION,
                        "min_count must be between 1 and the number of window elements");
  if (kind == kPercentile && (!std::isfinite(percentile) || percentile < 0.0 || percentile > 100.0))
    return noalloc_fail(NDF_ERR_INVALID_CONFIGURATION, "percentile must be finite and between zero and 100");
  if (n_out == 0) return NDF_OK;
  if (!d_in || !d_out) return noalloc_fail(NDF_ERR_LENGTH_MISMATCH, "missing input or output buffer");
  Geom3 g{};
  g.D = 1;
  g.H = shp[0];
  g.W = shp[1];
  g.kd = 1;
  g.kh = (int)sz[0];
  g.kw = (int)sz[1];
  g.az = 0;
  g.ay = (int)(sz[0] / 2 + org[0]);
  g.ax = (int)(sz[1] / 2 + org[1]);
  g.mz = kNearest;
  g.my = md[0];
  g.mx = md[1];
  Reduce r{};
  r.kind = kind;
  r.omit = omit_nan != 0;
  r.drop_inf = r.omit && ignore_inf != 0;
  r.count = (int)std::min<unsigned long long>(volume, 1ull << 30);
  r.min_count = r.omit ? (long long)min_count : 1;
  r.param = (long long)std::min<uint64_t>(parameter, (uint64_t)(1ull << 62));
  r.q = percentile;
  r.q_fraction = percentile / 100.0;
  r.q_is_max = percentile == 100.0;
  r.pct = nullptr;
  r.cval = dtype == NDF_FLOAT32 ? (double)(float)cval : cval;
  int device = 0, sm_count = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  HistChoice c = choose_tile(g, dtype == 0 ? 4 : 8, sm_count);
  if (c.TW == 0) return noalloc_fail(NDF_ERR_UNSUPPORTED, "window too large for the histogram kernel");
  HistArgs a = make_args_core(g, c, dtype, Runs{}, r);
  if ((size_t)a.slot_bytes > kNoAllocScratchBytes)
    return noalloc_fail(NDF_ERR_MEMORY,
                        "the window's sort slot exceeds the 16 MiB allocation-free scratch");
  if (e != cudaSuccess) {
    cudaGetLastError();
    return noalloc_fail(NDF_ERR_NO_DEVICE, "no usable CUDA device");
  }
  const size_t smem = c.smem;
  if (smem > (size_t)optin) return noalloc_fail(NDF_ERR_UNSUPPORTED, "window too large for shared memory");
  void* scratch = nullptr;
  e = noalloc_scratch(device, &scratch);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
  const void* kernel = dtype == 0 ? kernel_for<float>(c.sdec) : kernel_for<double>(c.sdec);
  e = allow_max_smem(kernel);
  int per_sm = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kHThreads, smem);
  if (e != cudaSuccess) return cuda_fail(e, "histogram (allocation-free) set-up");
  long long slots = (long long)(kNoAllocScratchBytes / (size_t)a.slot_bytes);
  const long long grid = a.in_smem ? std::min<long long>(a.tiles, INT_MAX)
                                   : std::min<long long>(std::min<long long>(a.tiles, slots),
                                                         (long long)std::max(per_sm, 1) * sm_count);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == 0)
    histogram_kernel<float, false, false><<<(unsigned)grid, kHThreads, smem, s>>>(
        (const float*)d_in, (float*)d_out, a, (unsigned char*)scratch);
  else
    histogram_kernel<double, false, false><<<(unsigned)grid, kHThreads, smem, s>>>(
        (const double*)d_in, (double*)d_out, a, (unsigned char*)scratch);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "histogram (allocation-free)");
  return NDF_OK;
}
