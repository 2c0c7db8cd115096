// Team rounds: LP rounds of whole instances inside one launch, sm_103a.
//
// A team of T CTAs refines one instance: one CTA (T = 1), a thread-block
// cluster (T <= 16) or the whole cooperative grid. Every phase of a sub-round
// (sweep, target- and source-side selection, commit, hindsight reverts,
// rollback) runs in the same kernel, separated by team barriers instead of
// launch boundaries, and so do all rounds of the launch. The phases follow the
// rules of the multi-launch pipeline (the same lane-per-vertex sweep, the same
// selection thresholds, the same CTA-flat commit), so every instance ends
// exactly as there.
//
// What bounds it: a sub-round of a small instance is a chain of dependent L2
// accesses (0.5 us each) and barriers (a grid barrier about 2 us, a cluster
// barrier 1.2 us). The multi-launch form pays six launches for it, 30 us per
// sub-round on 1,024 vertices; a team pays four to six barriers. Per refine,
// before (multi-launch) and now: 1,024 vertices 1,130 -> 435 us, 131,071
// (k = 64) 3,552 -> 2,009 us, 1M (k = 32) 5,830 -> 4,601 us. A 1,280-instance
// batch (clusters, CTA selection in one pass, CTA-wide heavy vertices) takes
// 42.1 -> 28.7 ms end to end and 24 stepped sessions 38.2 -> 6.2 ms.
//
// A vertex is swept, selected, moved and undone by one CTA per sub-round, whose
// candidate and kept-move lists live in its own part of the instance's scratch
// arrays; CTAs meet in per-block totals and selection segments (global memory)
// only. The 1-CTA-per-SM builds deal the vertices out once, in 32-vertex chunks
// (chunk c to CTA c mod T), and so can keep them in shared memory. The others
// list a round's active vertices per sub-round for the whole team and cut each
// sub-round's list into equal parts: a CTA's chunks fall into a sub-round by a
// hash, 15 +- 4 of them where 304 CTAs share a million vertices, and the
// slowest CTA had 1.7 times the mean.
#pragma once

#include <cstddef>
#include <type_traits>

#include "lp_device.cuh"

namespace lpgpu {

constexpr int kTeamThreads = kFlatThreads;  // the CTA-flat helpers are written for this width
constexpr int kTeamWarps = kTeamThreads / 32;

enum TeamSync : int { kSyncCta = 0, kSyncCluster = 1, kSyncGrid = 2 };

// Global scratch of a team (64-bit words): barrier arrivals, abort flag, work
// item, wide nets, then three slots of per-block totals (sub-rounds take them in turn: in
// sub-round s, after its first barrier, nobody reads the slot of s - 1 any
// more and nobody adds to it before the first barrier of s + 1, so it is
// cleared then), then the selection thresholds.
struct TeamGlob {
  int64_t* g;
  int K;
  __device__ ull* arrivals() const { return reinterpret_cast<ull*>(g); }
  __device__ int64_t* abort_flag() const { return g + 1; }
  __device__ int64_t* item() const { return g + 2; }
  __device__ ull* wide() const { return reinterpret_cast<ull*>(g + 3); }  // wide nets listed by an expansion
  __device__ int64_t* slot(int q) const { return g + 8 + (int64_t)q * (5 * K + 8); }
  __device__ ull* in_w(int q) const { return reinterpret_cast<ull*>(slot(q)); }
  __device__ ull* in_cnt(int q) const { return in_w(q) + K; }
  __device__ ull* out_w(int q) const { return in_w(q) + 2 * K; }
  __device__ ull* acc_w(int q) const { return in_w(q) + 3 * K; }
  __device__ ull* acc_cnt(int q) const { return in_w(q) + 4 * K; }
  __device__ ull* delta(int q) const { return in_w(q) + 5 * K; }
  __device__ ull* nrev(int q) const { return in_w(q) + 5 * K + 1; }
  __device__ ull* active(int q) const { return in_w(q) + 5 * K + 2; }
  __device__ uint64_t* thr_to() const { return reinterpret_cast<uint64_t*>(g + 32 + 15 * (int64_t)K); }
  __device__ uint64_t* thr_from() const { return thr_to() + K; }
  // active vertices per sub-round, for three rounds in turn
  __device__ ull* count(int r) const { return reinterpret_cast<ull*>(thr_from() + K) + r * kMaxSubrounds; }
};

// Selection keys a CTA holds in registers and shared memory; more leave the L1
// cache less (1M vertices, k = 32, 1,024 / 2,048 / 4,096 keys: 4,575 / 4,558 /
// 4,895 us; 131,071 1,975 / 1,986 / 2,060; row-net 4.2M 10,995 / 11,020 / 11,370).
constexpr int kTeamStage = 1024;
constexpr int kSelBits = 11;      // key bits per pass of the CTA selection
constexpr size_t kSelArea = (size_t)kTeamStage * 12 + (sizeof(unsigned) << kSelBits);
constexpr size_t kWarpSelArea = (size_t)kTeamWarps * 256 * sizeof(unsigned);
constexpr size_t kTeamArea = sizeof(FlatSmem) > kSelArea ? sizeof(FlatSmem) : kSelArea;
static_assert(kTeamArea >= kWarpSelArea, "every warp's selection histogram fits the shared area");
#ifndef LPGPU_PX_WARP_SEL
#define LPGPU_PX_WARP_SEL 512  // segments of at most this many keys get one warp when blocks outnumber CTAs
#endif
constexpr int kTeamWarpSelKeys = LPGPU_PX_WARP_SEL;

// Candidates whose records stay in shared memory (the others in I.rec).
constexpr int kCandCache = 512;

// The 1-CTA-per-SM builds (OWN) keep a CTA's part of the instance in shared
// memory; the 2-CTA builds have 64 registers, where the code for it costs more
// than it gives (4.2M vertices 11,360 us without, 12,210 us with it).
//
// A CTA's part of the instance. Its vertices are named by their index li in
// the CTA (32 per chunk). off / wv / part / list / inets are copies in shared
// memory when they fit (off null: not resident): nobody else reads or changes
// them, so a sweep's chain of dependent accesses is one L2 trip (the net's
// record) instead of four. Whole refine, without -> with (GB300, us): 1,024
// vertices 577 -> 544, 16,384 996 -> 912, 65,536 (k = 32) 1,810 -> 1,708,
// 131,071 (k = 64) 2,117 -> 2,032, 262,144 1,409 -> 1,352.
struct TeamPart {
  int4* rec;
  uint8_t* status;
  int32_t *list, *heavy, *kept;
  int32_t *off, *wv, *part;
  uint32_t* masks;  // active vertices per chunk while the list is built (free until the round's first kept move)
  int beg, cnt;     // this CTA's part of the sub-round's list
  int len, vbits, chunks, own_nets;  // own_nets: bit 0 the records, 1 the pin counts are in shared memory
};

// KM: room for blocks.
template <int KM>
struct TeamShared {
  static constexpr int kBlocks = KM;
  PxInst I;
  TeamPart V;
  RoundCtx c;
  int64_t bw[KM], lmax[KM], perf[KM];
  int64_t tot_cnt[KM];  // candidates of the team per block
  int64_t seg[KM];
  uint64_t thr_to[KM], thr_from[KM];
  ull in_w[KM], out_w[KM], dw[KM];  // of this CTA
  unsigned in_cnt[KM];
  unsigned base[KM], cur[KM];  // this CTA's range inside a block's segment
  int slack[KM];
  int pen[KM];
  int over_ids[KM];
  uint32_t fmask[kLvWeights * KM / 32];
  uint8_t over[KM];
  int off[kMaxSubrounds + 1], fill[kMaxSubrounds];
  int kbeg[kMaxSubrounds], kpre[kMaxSubrounds + 1];  // kept moves of the round's sub-rounds: place, count before
  long long st[kStats];
  uint64_t red_and[kTeamWarps], red_or[kTeamWarps];
  unsigned wsum[kTeamWarps];
  uint64_t thr;
  long long below, delta, gdelta, tdelta;
  ull hint;
  int hborder;
  int nover, any;  // any: bit 0 a target block overflows, 1 a source block may empty, 2 a candidate exists
  int sel_bin, sel_n;
  int maxdeg;  // of the collected moves
  int ncand, nrev, grev, nkept, rolled, tile, nheavy, nhuge, item, abort;
  // builds with resident parts only (kTeamShortAt: the end for the others)
  alignas(16) int4 crec[kCandCache];  // (li, gain, to | from << 16, weight)
  uint8_t cst[kCandCache];            // 1 committed, 2 reverted, 3 rolled back
};
constexpr size_t kTeamSharedAt = (kTeamArea + 15) & ~size_t(15);
// Room for blocks by the words of Λ, and where the CTA's part of the instance starts.
template <int W>
constexpr int kTeamBlocks = W <= 4 ? 128 : 32 * W;
template <int KM>
constexpr size_t kTeamOwnAt = (kTeamSharedAt + sizeof(TeamShared<KM>) + 15) & ~size_t(15);
struct Team {
  TeamGlob G;
  int T, rank, sync;
  ull arrivals;  // barrier arrivals expected so far (grid barrier, thread 0)
  int builds;    // active lists built so far
};

// Limit of a grid barrier's wait: clocks (about 20 s: a barrier waits for the slowest
// CTA's phase, one net of a billion pins takes a second, and a GPU that is shared in
// time counts its absence), looked at every so many polls (a power of two).
#ifndef LPGPU_TEAM_WAIT_CLOCKS
#define LPGPU_TEAM_WAIT_CLOCKS 40000000000ll
#endif
#ifndef LPGPU_TEAM_WAIT_POLLS
#define LPGPU_TEAM_WAIT_POLLS 1024u
#endif

// Barrier of the team: everything its CTAs wrote before is visible after. The
// grid barrier (one arrival per CTA on a counter that only grows) gives up at
// its limit and then raises the team's abort flag, which ends the kernel in
// every CTA; false: aborted.
template <typename TS>
__device__ __forceinline__ bool team_sync(Team& tm, TS& s) {
  if (tm.sync == kSyncCta) {
    __syncthreads();
    return true;
  }
  if (tm.sync == kSyncCluster) {
    __syncwarp();  // .aligned wants whole warps, and the callers' thread-0 and strided code diverges
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // release and acquire on the counter order the whole CTA's accesses
    // (through the CTA barriers); separate fences only add to the latency
    tm.arrivals += (ull)tm.T;
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(tm.G.arrivals()) : "memory");
    const long long t0 = clock64();
    for (unsigned polls = 0;; ++polls) {
      ull seen;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(tm.G.arrivals()) : "memory");
      if (seen >= tm.arrivals) break;
      if ((polls & (LPGPU_TEAM_WAIT_POLLS - 1)) == LPGPU_TEAM_WAIT_POLLS - 1) {
        if (*(volatile int64_t*)tm.G.abort_flag() || clock64() - t0 > LPGPU_TEAM_WAIT_CLOCKS) {
          *(volatile int64_t*)tm.G.abort_flag() = 1;
          s.abort = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  return s.abort == 0;
}
#define TEAM_SYNC()                      \
  do {                                   \
    if (!team_sync(tm, s)) return false; \
  } while (0)

// (gain, local vertex) as one integer in the order of move_key, without the
// constant bits between the two fields: the selection's first pass then covers
// the differing gain bits and the top vertex bits together.
__device__ __forceinline__ uint64_t team_key(int gain, int lv, int vbits) {
  return ((uint64_t)((uint32_t)((int64_t)gain - 1) ^ 0x80000000u) << vbits) | (uint32_t)lv;
}

// First key whose inclusive weighted prefix exceeds `budget` among up to 32
// keys, one per lane (lanes >= n hold none); every lane returns it.
__device__ __forceinline__ uint64_t warp_rank_select(uint64_t key, int w, int n, int64_t budget) {
  const int lane = lane_id();
  int64_t excl = 0;
  for (int j = 0; j < n; ++j) {
    const uint64_t kj = __shfl_sync(FULLMASK, key, j);
    const int wj = __shfl_sync(FULLMASK, w, j);
    if (kj < key) excl += wj;
  }
  const unsigned hit = __ballot_sync(FULLMASK, lane < n && excl <= budget && excl + w > budget);
  return hit ? __shfl_sync(FULLMASK, key, __ffs(hit) - 1) : ~0ull;
}

__device__ __forceinline__ void warp_and_or(uint64_t& a, uint64_t& o) {
  const uint32_t al = __reduce_and_sync(FULLMASK, (uint32_t)a), ah = __reduce_and_sync(FULLMASK, (uint32_t)(a >> 32));
  const uint32_t ol = __reduce_or_sync(FULLMASK, (uint32_t)o), oh = __reduce_or_sync(FULLMASK, (uint32_t)(o >> 32));
  a = ((uint64_t)ah << 32) | al;
  o = ((uint64_t)oh << 32) | ol;
}

// Gain-sorted prefix without sorting, by one CTA: the first of `cnt` distinct
// keys whose inclusive weighted prefix exceeds `budget` (keys below it are
// accepted; all ones when the total stays within the budget, 0 for a negative
// budget). Each pass bins the keys by their topmost differing kSelBits bits,
// keeps the bin the budget ends in, and gathers that bin's keys; up to 32 keys
// left are ranked by one warp. Keys are few per block (a sub-round's candidates
// into it), so the time is barriers: one pass and the ranking usually, against
// four byte passes of a plain radix selection. `area`: kSelArea bytes.
template <typename TS>
__device__ uint64_t team_cta_select(const uint64_t* gk, const int32_t* gw, int64_t cnt, int64_t budget,
                                    unsigned char* area, TS& s) {
  constexpr int PER = kTeamStage / kTeamThreads, BINS = 1 << kSelBits, BPT = BINS / kTeamThreads;
  uint64_t* sk = reinterpret_cast<uint64_t*>(area);
  int32_t* sw = reinterpret_cast<int32_t*>(sk + kTeamStage);
  unsigned* hist = reinterpret_cast<unsigned*>(sw + kTeamStage);
  const int t = threadIdx.x, lane = lane_id(), wid = t >> 5;
  if (budget < 0 || cnt <= 0) return budget < 0 ? 0ull : ~0ull;
  bool held = cnt <= kTeamStage;  // the keys still in play are in registers
  int n = held ? (int)cnt : 0;
  uint64_t mask = 0, prefix = 0, kr[PER];
  int wr[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = t + q * kTeamThreads;
    kr[q] = held && i < n ? *(gk + i) : 0;
    wr[q] = held && i < n ? *(gw + i) : 0;
  }
  for (;;) {
    uint64_t ka = ~0ull, ko = 0;
    if (held) {
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (t + q * kTeamThreads < n) {
          ka &= kr[q];
          ko |= kr[q];
        }
    } else {
      for (int64_t i = t; i < cnt; i += kTeamThreads) {
        const uint64_t key = *(gk + i);
        if ((key & mask) == prefix) {
          ka &= key;
          ko |= key;
        }
      }
    }
    warp_and_or(ka, ko);
    if (lane == 0) {
      s.red_and[wid] = ka;
      s.red_or[wid] = ko;
    }
    for (int i = t; i < BINS; i += kTeamThreads) hist[i] = 0;
    if (t == 0) {
      s.sel_bin = -1;
      s.sel_n = 0;
    }
    __syncthreads();
    ka = s.red_and[lane % kTeamWarps];
    ko = s.red_or[lane % kTeamWarps];
    warp_and_or(ka, ko);
    const uint64_t diff = ka ^ ko;
    const int hi = diff ? 63 - __clzll(diff) : 0, lo = hi >= kSelBits ? hi - kSelBits + 1 : 0;
    if (held) {
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (t + q * kTeamThreads < n) atomicAdd(&hist[(unsigned)(kr[q] >> lo) & (BINS - 1)], (unsigned)wr[q]);
    } else {
      for (int64_t i = t; i < cnt; i += kTeamThreads) {
        const uint64_t key = *(gk + i);
        if ((key & mask) == prefix) atomicAdd(&hist[(unsigned)(key >> lo) & (BINS - 1)], (unsigned)*(gw + i));
      }
    }
    __syncthreads();
    unsigned h[BPT], sum = 0;
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
      h[j] = hist[BPT * t + j];
      sum += h[j];
    }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(FULLMASK, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s.wsum[wid] = incl;
    __syncthreads();
    int64_t run = (int64_t)incl - sum;
    for (int w = 0; w < wid; ++w) run += s.wsum[w];
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
      if (run <= budget && run + h[j] > budget) {  // one bin at most
        s.sel_bin = BPT * t + j;
        s.below = run;
      }
      run += h[j];
    }
    __syncthreads();
    const int bin = s.sel_bin;
    if (bin < 0) return ~0ull;  // the total stays within the budget
    budget -= s.below;
    const uint64_t above = hi >= 63 ? 0 : ~((2ull << hi) - 1);  // bits above the differing ones
    mask = lo > 0 ? ~((1ull << lo) - 1) : ~0ull;
    prefix = (ka & above) | ((uint64_t)bin << lo);
    if (held) {
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (t + q * kTeamThreads < n && (kr[q] & mask) == prefix) {
          const int at = atomicAdd(&s.sel_n, 1);
          sk[at] = kr[q];
          sw[at] = wr[q];
        }
    } else {
      for (int64_t i = t; i < cnt; i += kTeamThreads) {
        const uint64_t key = *(gk + i);
        if ((key & mask) == prefix) {
          const int at = atomicAdd(&s.sel_n, 1);
          if (at < kTeamStage) {
            sk[at] = key;
            sw[at] = *(gw + i);
          }
        }
      }
    }
    __syncthreads();
    n = s.sel_n;
    held = held || n <= kTeamStage;
    if (!held) {
      __syncthreads();  // s.sel_n is cleared by the next pass
      continue;
    }
    if (n <= 32) {
      if (wid == 0) {
        const uint64_t r = warp_rank_select(lane < n ? sk[lane] : ~0ull, lane < n ? sw[lane] : 0, n, budget);
        if (lane == 0) s.thr = r;
      }
      __syncthreads();
      return s.thr;
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int i = t + q * kTeamThreads;
      kr[q] = i < n ? sk[i] : 0;
      wr[q] = i < n ? sw[i] : 0;
    }
    __syncthreads();  // the list and the counters are reused by the next pass
  }
}

// The same threshold by one warp (at most a few hundred keys), 8 bits per
// pass. `hist`: 256 words of this warp's shared scratch.
static __device__ uint64_t team_warp_select(const uint64_t* gk, const int32_t* gw, int cnt, int64_t budget, unsigned* hist) {
  const int lane = lane_id();
  if (budget < 0 || cnt <= 0) return budget < 0 ? 0ull : ~0ull;
  uint64_t mask = 0, prefix = 0;
  for (;;) {
    // the keys in play: their differing bits, and the first 32 of them
    uint64_t ka = ~0ull, ko = 0;
    uint64_t* lk = reinterpret_cast<uint64_t*>(hist);
    int* lw = reinterpret_cast<int*>(hist + 64);
    int n = 0;
    for (int i0 = 0; i0 < cnt; i0 += 32) {
      const int i = i0 + lane;
      const uint64_t key = i < cnt ? *(gk + i) : 0;
      const bool in = i < cnt && (key & mask) == prefix;
      const unsigned bal = __ballot_sync(FULLMASK, in);
      if (in) {
        ka &= key;
        ko |= key;
        const int at = n + __popc(bal & lanemask_lt());
        if (at < 32) {
          lk[at] = key;
          lw[at] = *(gw + i);
        }
      }
      n += __popc(bal);
    }
    __syncwarp();
    if (n <= 32) return warp_rank_select(lane < n ? lk[lane] : ~0ull, lane < n ? lw[lane] : 0, n, budget);
    warp_and_or(ka, ko);
    __syncwarp();
    const uint64_t diff = ka ^ ko;
    const int hi = 63 - __clzll(diff), lo = hi >= 8 ? hi - 7 : 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) hist[32 * j + lane] = 0;
    __syncwarp();
    for (int i = lane; i < cnt; i += 32) {
      const uint64_t key = *(gk + i);
      if ((key & mask) == prefix) atomicAdd(&hist[(unsigned)(key >> lo) & 255u], (unsigned)*(gw + i));
    }
    __syncwarp();
    unsigned h[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      h[j] = hist[8 * lane + j];
      sum += h[j];
    }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(FULLMASK, incl, o);
      if (lane >= o) incl += y;
    }
    int bin = -1;
    int64_t run = (int64_t)incl - sum, below = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (run <= budget && run + h[j] > budget) {
        bin = 8 * lane + j;
        below = run;
      }
      run += h[j];
    }
    const unsigned found = __ballot_sync(FULLMASK, bin >= 0);
    if (!found) return ~0ull;
    const int src = __ffs(found) - 1;
    bin = __shfl_sync(FULLMASK, bin, src);
    budget -= __shfl_sync(FULLMASK, below, src);
    const uint64_t above = hi >= 63 ? 0 : ~((2ull << hi) - 1);
    mask = lo > 0 ? ~((1ull << lo) - 1) : ~0ull;
    prefix = (ka & above) | ((uint64_t)bin << lo);
    __syncwarp();  // the histogram is reused by the next pass
  }
}

// Segments of the blocks flagged in s.over: s.seg (starts, from s.tot_cnt) and
// the list of flagged blocks. Whole CTA.
template <typename TS>
__device__ __forceinline__ void team_plan(const PxInst& I, TS& s) {
  if (threadIdx.x < 32) {
    constexpr int PER = TS::kBlocks / 32;
    const int lane = threadIdx.x;
    int64_t sum = 0;
    int nov = 0;
    for (int j = 0; j < PER; ++j) {
      const int b = PER * lane + j;
      if (b < I.k && s.over[b]) {
        sum += s.tot_cnt[b];
        ++nov;
      }
    }
    int64_t inc = sum;
    int ino = nov;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t y = __shfl_up_sync(FULLMASK, inc, d);
      const int z = __shfl_up_sync(FULLMASK, ino, d);
      if (lane >= d) {
        inc += y;
        ino += z;
      }
    }
    int64_t run = inc - sum;
    int at = ino - nov;
    for (int j = 0; j < PER; ++j) {
      const int b = PER * lane + j;
      if (b < I.k && s.over[b]) {
        s.seg[b] = run;
        run += s.tot_cnt[b];
        s.over_ids[at++] = b;
      }
    }
    if (lane == 31) s.nover = ino;
  }
  __syncthreads();
}

// Thresholds of the flagged blocks from the filled segments, the blocks dealt
// to the team's CTAs (a warp each for small segments when they outnumber the
// CTAs), into the team's table `gthr` (T > 1) or `thr`.
template <typename Budget, typename TS>
__device__ __forceinline__ void team_select(const PxInst& I, Team& tm, TS& s, unsigned char* area,
                                            uint64_t* gthr, uint64_t* thr, Budget budget) {
  const int nover = s.nover, wid = threadIdx.x >> 5;
  const int64_t warp_keys = nover > tm.T ? kTeamWarpSelKeys : -1;
  unsigned* whist = reinterpret_cast<unsigned*>(area) + 256 * wid;
  if (warp_keys >= 0) {
    for (int j = wid * tm.T + tm.rank; j < nover; j += tm.T * kTeamWarps) {
      const int b = s.over_ids[j];
      if (s.tot_cnt[b] > warp_keys) continue;
      const uint64_t t = team_warp_select(I.keys + s.seg[b], I.kw + s.seg[b], (int)s.tot_cnt[b], budget(b), whist);
      if (lane_id() == 0) (tm.T > 1 ? gthr : thr)[b] = t;
    }
    __syncthreads();
  }
  for (int j = tm.rank; j < nover; j += tm.T) {
    const int b = s.over_ids[j];
    if (s.tot_cnt[b] <= warp_keys) continue;  // the same for the whole CTA
    const uint64_t t = team_cta_select(I.keys + s.seg[b], I.kw + s.seg[b], s.tot_cnt[b], budget(b), area, s);
    if (threadIdx.x == 0) (tm.T > 1 ? gthr : thr)[b] = t;
    __syncthreads();
  }
}

template <bool OWN>
__device__ __forceinline__ int team_lv(const Team& tm, int li) {
  return !OWN ? li : (((li >> kChunkShift) * tm.T + tm.rank) << kChunkShift) | (li & 31);
}
template <bool OWN, typename TS>
__device__ __forceinline__ void team_degree(const Team& tm, const TS& s, int li, int64_t& o0, int64_t& d) {
  if (OWN && s.V.off) {
    o0 = s.V.off[li];
    d = s.V.off[li + 1] - o0;
  } else {
    const int64_t v = s.I.v0 + team_lv<OWN>(tm, li);
    o0 = s.I.vtx_off[v];
    d = s.I.vtx_off[v + 1] - o0;
  }
}
template <bool OWN, typename TS>
__device__ __forceinline__ void team_vertex(const Team& tm, const TS& s, int li, int64_t& o0, int64_t& d,
                                            int& from, int& wv) {
  team_degree<OWN>(tm, s, li, o0, d);
  if (OWN && s.V.off) {
    from = s.V.part[li];
    wv = s.V.wv[li];
  } else {
    const int64_t v = s.I.v0 + team_lv<OWN>(tm, li);
    from = s.I.part[v] - s.I.boff;
    wv = s.I.w_v[v];
  }
}

// Candidate i of the CTA's list and its status.
template <bool OWN, typename TS>
__device__ __forceinline__ int4 team_rec(const TS& s, int i) { return OWN && i < kCandCache ? s.crec[i] : s.V.rec[i]; }
template <bool OWN, typename TS>
__device__ __forceinline__ int team_status(const TS& s, int i) {
  return OWN && i < kCandCache ? s.cst[i] : s.V.status[i];
}
template <bool OWN, typename TS>
__device__ __forceinline__ void team_set_status(TS& s, int i, int x) {
  (OWN && i < kCandCache ? s.cst : s.V.status)[i] = (uint8_t)x;
}

// Appends the warp's candidate moves (lanes with `has`) to the CTA's list and
// adds them to its per-block totals.
template <bool OWN, typename TS>
__device__ __forceinline__ void team_candidates(TS& s, bool has, int li, int gain, int from, int to, int wv) {
  const int slot = flat_append_to(&s.ncand, has);
  if (has) {
    (OWN && slot < kCandCache ? s.crec : s.V.rec)[slot] = make_int4(li, gain, to | (from << 16), wv);
    atomicAdd(&s.in_w[to], (ull)(int64_t)wv);
    atomicAdd(&s.in_cnt[to], 1u);
    atomicAdd(&s.out_w[from], (ull)(int64_t)wv);
  }
}

// cnt += x (bit-sliced).
template <int PL>
__device__ __forceinline__ void lv_add_counters(uint32_t (&cnt)[PL], const uint32_t (&x)[PL]) {
  uint32_t cy = 0;
#pragma unroll
  for (int p = 0; p < PL; ++p) {
    const uint32_t t = cnt[p];
    cnt[p] = t ^ x[p] ^ cy;
    cy = (t & x[p]) | (cy & (t ^ x[p]));
  }
}

// Best move of a vertex by the G = 1, 2 or 4 lanes of its group (lane `sub`
// takes every G-th step of U incidences; the counters are summed over the
// group, so every lane decides alike). All lanes of the warp take part; d = 0:
// nothing to evaluate.
template <int W, bool UNIT, int PL, int U, typename TS>
__device__ __forceinline__ void team_lv_vertex(const RoundCtx& c, const TS& s, int64_t o0, int d, int from,
                                               int wv, int G, int sub, int zero_gain, int& to, int& gain) {
  uint32_t cnt[W][PL];
#pragma unroll
  for (int t = 0; t < W; ++t)
#pragma unroll
    for (int p = 0; p < PL; ++p) cnt[t][p] = 0;
  int internal = 0;
  const int fw = from >> 5;
  const uint32_t fbit = 1u << (from & 31);
  int32_t ee[U];
  lv_ids<U, false>(c, o0, d, U * sub, ee);
  for (int j = U * sub; j < d; j += U * G) {
    uint32_t wd[U][W], l1[U];
    int we[U];
    lv_records<W, UNIT, U, false>(c, ee, fw, fbit, wd, l1, we);
    lv_ids<U, false>(c, o0, d, j + U * G, ee);  // in flight with the records
    lv_add<W, UNIT, PL, U>(wd, l1, we, fbit, cnt, internal);
  }
  __syncwarp();
  for (int g = 1; g < G; g <<= 1) {
#pragma unroll
    for (int t = 0; t < W; ++t) {
      uint32_t x[PL];
#pragma unroll
      for (int p = 0; p < PL; ++p) x[p] = __shfl_xor_sync(FULLMASK, cnt[t][p], g);
      lv_add_counters<PL>(cnt[t], x);
    }
    internal += __shfl_xor_sync(FULLMASK, internal, g);
  }
  bool border = false;
  if (d > 0)
    lv_decide<W, PL>(c, cnt, internal, from, wv, 0, 0, false, zero_gain, s.fmask, s.slack, s.bw, s.perf, to, gain,
                     border);
}

// Best move of a vertex for k > 128 by the W / 4 lanes of its group: lane `wl`
// counts the blocks of words 4 wl .. 4 wl + 3, so a net's record is one
// contiguous load of the group and the counters stay in registers; the
// decision of lv_decide with its tests joined over the group. All lanes of the
// warp take part; d = 0: nothing to evaluate.
template <int W, bool UNIT, int PL, int U, typename TS>
__device__ __forceinline__ void team_lv_wide(const RoundCtx& c, const TS& s, int64_t o0, int d, int from, int wv,
                                             int wl, int zero_gain, int& to, int& gain) {
  constexpr int LG = W / 4;
  uint32_t cnt[4][PL];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int p = 0; p < PL; ++p) cnt[t][p] = 0;
  int internal = 0;
  const int fw = from >> 5, fl = (fw >> 2) == wl ? fw & 3 : -1;  // the from word, when this lane holds it
  const uint32_t fbit = 1u << (from & 31);
  int32_t ee[U];
  lv_ids<U, false>(c, o0, d, 0, ee);
  for (int j = 0; j < d; j += U) {
    uint32_t wd[U][4], l1[U];
    int we[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int t = 0; t < 4; ++t) wd[u][t] = 0;
      l1[u] = fbit;
      we[u] = 0;
      if (ee[u] >= 0) {
        const uint32_t* rec = c.conn + (int64_t)ee[u] * 2 * W;
        load_words<4, false>(rec + 4 * wl, wd[u]);
        if (fl >= 0) l1[u] = rec[W + fw];
        we[u] = UNIT ? 1 : c.w_e[ee[u]];
      }
    }
    lv_ids<U, false>(c, o0, d, j + U, ee);  // in flight with the records
    lv_add<4, UNIT, PL, U>(wd, l1, we, fbit, cnt, internal);
  }
  __syncwarp();
  uint32_t cand[4];
  if (wv >= 1 && wv <= kLvWeights) {
#pragma unroll
    for (int t = 0; t < 4; ++t) cand[t] = s.fmask[(wv - 1) * W + 4 * wl + t];
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      cand[t] = 0;
      for (int l = 0; l < 32; ++l) {
        const int b = 32 * (4 * wl + t) + l;
        if (b < c.k && s.slack[b] >= wv) cand[t] |= 1u << l;
      }
    }
  }
  // isBorderNode: some incident net holds a block other than `from`
  uint32_t other = 0, anyc = 0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint32_t fm = t == fl ? ~fbit : ~0u;
    uint32_t o = 0;
#pragma unroll
    for (int p = 0; p < PL; ++p) o |= cnt[t][p];
    other |= o & fm;
    cand[t] &= fm;
    anyc |= cand[t];
  }
  auto joined = [&](uint32_t x) {
#pragma unroll
    for (int g = 1; g < LG; g <<= 1) x |= __shfl_xor_sync(FULLMASK, x, g);
    return x;
  };
#pragma unroll
  for (int g = 1; g < LG; g <<= 1) internal += __shfl_xor_sync(FULLMASK, internal, g);
  other = joined(other);  // every lane takes part in every join
  anyc = joined(anyc);
  const bool open = other != 0 && anyc != 0;
  // maximum penalty over the candidates, plane by plane from the top
  int val = 0;
#pragma unroll
  for (int p = PL - 1; p >= 0; --p) {
    uint32_t tt[4], o = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      tt[t] = cand[t] & cnt[t][p];
      o |= tt[t];
    }
    if (joined(o)) {
#pragma unroll
      for (int t = 0; t < 4; ++t) cand[t] = tt[t];
      val |= 1 << p;
    }
  }
  int b = INT_MAX;  // lowest block of maximum penalty
#pragma unroll
  for (int t = 3; t >= 0; --t)
    if (cand[t]) b = 32 * (4 * wl + t) + __ffs(cand[t]) - 1;
#pragma unroll
  for (int g = 1; g < LG; g <<= 1) b = min(b, __shfl_xor_sync(FULLMASK, b, g));
  if (d == 0 || !open || val < internal) return;
  if (val > internal) {
    to = b;
    gain = internal - val;
  } else if (zero_gain && s.bw[from] - 1 > s.bw[b] + 1 && s.bw[b] < s.perf[b]) {
    to = b;
    gain = 0;
  }
}

// Penalties of the blocks 32 t + lane over the 32-incidence windows start,
// start + step, ... of a vertex (lane = incidence, Λ words transposed across
// the warp); `internal` is this lane's part.
template <int W, bool UNIT>
__device__ __forceinline__ void team_windows(const RoundCtx& c, int64_t o0, int d, int from, int start, int step,
                                             int (&pen)[W], int& internal, bool& border) {
  const int lane = lane_id(), fw = from >> 5;
  const uint32_t fbit = 1u << (from & 31);
#pragma unroll
  for (int t = 0; t < W; ++t) pen[t] = 0;
  for (int w0 = start; w0 < d; w0 += step) {
    uint32_t wd[W];
    int we = 0, lam = 0;
#pragma unroll
    for (int t = 0; t < W; ++t) wd[t] = 0;
    if (w0 + lane < d) {
      const int64_t e = c.inets[o0 + w0 + lane];
      we = UNIT ? 1 : c.w_e[e];
      const uint32_t* rec = c.conn + e * 2 * W;
      load_words<W, false>(rec, wd);
      internal += (rec[W + fw] & fbit) ? 0 : we;  // Φ(e, from) > 1
#pragma unroll
      for (int t = 0; t < W; ++t) lam += __popc(wd[t]);
    }
    border = border || __ballot_sync(FULLMASK, lam > 1) != 0;
    if constexpr (UNIT) {
#pragma unroll
      for (int t = 0; t < W; ++t) pen[t] += __popc(transpose32(wd[t]));
    } else {
      const Planes wp = make_planes(we, 32 - __clz(__reduce_or_sync(FULLMASK, (unsigned)we)));
#pragma unroll
      for (int t = 0; t < W; ++t) pen[t] += plane_sum(wp, transpose32(wd[t]), we);
    }
  }
}

template <int W, bool UNIT, bool OWN, typename TS>
__device__ __forceinline__ void team_heavy_decide(const PxParams& P, TS& s, int li, int from, int wv,
                                                  int internal, const int (&pen)[W]) {
  const int lane = lane_id(), k = s.I.k;
  int sl[W];
#pragma unroll
  for (int t = 0; t < W; ++t) sl[t] = 32 * t + lane < k ? s.slack[32 * t + lane] : -1;
  int to = from, gain = 0;
  decide<W, UNIT>(k, from, wv, internal, P.zero_gain, pen, sl, s.bw, s.perf, to, gain);
  team_candidates<OWN>(s, lane == 0 && to != from, li, gain, from, to, wv);
}

// Heavy vertices (summed net weight beyond the lane counters): a warp each up
// to kTeamHuge incidences, the whole CTA above.
constexpr int kTeamHuge = 1024;
template <int W, bool UNIT, bool OWN, typename TS>
__device__ void team_heavy(const PxParams& P, const RoundCtx& c, const Team& tm, TS& s) {
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int nheavy = s.nheavy, nhuge = s.nhuge;
  int64_t o0, d;
  int from, wv;
  for (int i = wid; i < nheavy; i += kTeamWarps) {
    const int li = s.V.heavy[i];
    team_vertex<OWN>(tm, s, li, o0, d, from, wv);
    int pen[W], internal = 0;
    bool border = false;
    team_windows<W, UNIT>(c, o0, (int)d, from, 0, 32, pen, internal, border);
    internal = warp_sum(internal);
    if (border) team_heavy_decide<W, UNIT, OWN>(P, s, li, from, wv, internal, pen);
  }
  for (int i = 0; i < nhuge; ++i) {
    const int li = s.V.heavy[s.V.len - 1 - i];
    team_vertex<OWN>(tm, s, li, o0, d, from, wv);
    __syncthreads();  // the previous vertex's sums are read
    for (int b = threadIdx.x; b < 32 * W; b += blockDim.x) s.pen[b] = 0;
    if (threadIdx.x == 0) {
      s.hint = 0;
      s.hborder = 0;
    }
    __syncthreads();
    int pen[W], internal = 0;
    bool border = false;
    team_windows<W, UNIT>(c, o0, (int)d, from, 32 * wid, 32 * kTeamWarps, pen, internal, border);
    internal = warp_sum(internal);
    if (lane == 0) {
      if (internal) atomicAdd(&s.hint, (ull)internal);
      if (border) s.hborder = 1;
    }
#pragma unroll
    for (int t = 0; t < W; ++t)
      if (pen[t]) atomicAdd(&s.pen[32 * t + lane], pen[t]);
    __syncthreads();
    if (wid == 0 && s.hborder) {
#pragma unroll
      for (int t = 0; t < W; ++t) pen[t] = s.pen[32 * t + lane];
      team_heavy_decide<W, UNIT, OWN>(P, s, li, from, wv, (int)s.hint, pen);
    }
  }
}

// Incidences a thread handles per step of the CTA-flat walks (1M vertices, k =
// 32: 1 4,596, 2 4,558, 4 4,648, 8 5,126 us per refine; row-net 4.2M 10,980 /
// 11,010 / 11,030 / 11,400).
constexpr int kTeamGroup = 2;

// Collects into f the candidates [c0, c0 + kFlatItems) of the CTA's list that
// pass `take(i, rec)`, as moves from `from` to `to` (back: the reverse), and
// sets their status to `set` (0: unchanged); with `move`, their part and the
// CTA's block-weight deltas follow.
template <bool OWN, typename Take, typename TS>
__device__ __forceinline__ void team_gather(const Team& tm, TS& s, FlatSmem& f, int c0, int ncand, bool back,
                                            int set, bool move, Take take) {
  constexpr int PER = kFlatItems / kTeamThreads;
  if (threadIdx.x == 0) f.n = s.maxdeg = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = c0 + q * kTeamThreads + threadIdx.x;
    bool sel = false;
    int4 r = make_int4(0, 0, 0, 0);
    if (i < ncand) {
      r = team_rec<OWN>(s, i);
      sel = take(i, r);
    }
    const int slot = flat_append(f, sel);
    if (sel) {
      const int to = r.z & 0xffff, from = r.z >> 16;
      int64_t o0, d;
      team_degree<OWN>(tm, s, r.x, o0, d);
      f.o0[slot] = o0;
      f.pre[slot] = (int)d;
      if (OWN) atomicMax(&s.maxdeg, (int)d);
      f.ft[slot] = back ? r.z : (from | (to << 16));  // low half: the block left
      f.att[slot] = 0;
      f.pos[slot] = i;
      if (set) team_set_status<OWN>(s, i, set);
      if (move) {
        const int a = back ? to : from, b = back ? from : to;
        s.I.part[s.I.v0 + team_lv<OWN>(tm, r.x)] = s.I.boff + b;
        if (OWN && s.V.off) s.V.part[r.x] = b;
        atomicAdd(&s.dw[b], (ull)(int64_t)r.w);
        atomicAdd(&s.dw[a], (ull)(-(int64_t)r.w));
      }
    }
  }
  __syncthreads();
}

// Few moves of small degree, as most CTAs of a team have in a sub-round: eight
// lanes take a move's incidences directly, without the scan and the searches of
// the flat walk, whose barriers and instructions were half of such a phase
// (16,384 vertices on 16 CTAs, 27 moves each: 873 -> 821 us per refine; 1,024 on
// one CTA 490 -> 457 us).
constexpr int kShortMoves = kTeamThreads / 8, kShortDegree = 32;
template <bool OWN, typename TS>
__device__ __forceinline__ bool team_short(const TS& s, int n) {
  return OWN && n <= kShortMoves && s.maxdeg <= kShortDegree;
}

// Moves every incidence of the collected items between their blocks; returns
// this thread's attributed delta, and the items' degrees in *degrees (summed
// over the threads). After a flat walk *total is the sum of the degrees.
template <bool OWN, typename TS>
__device__ __forceinline__ int64_t team_commit(const RoundCtx& c, const TS& s, FlatSmem& f, int n, int* total,
                                               int64_t* degrees, int64_t* toggles) {
  if (team_short<OWN>(s, n)) {
    const int it = threadIdx.x >> 3;
    int64_t att = 0;
    int tg = 0;
    if (it < n) {
      const int64_t o0 = f.o0[it];
      const int d = f.pre[it], ft = f.ft[it];
      if ((threadIdx.x & 7) == 0 && degrees) *degrees += d;
      for (int j = threadIdx.x & 7; j < d; j += 16) {
        const bool h[2] = {true, j + 8 < d};
        const int64_t e[2] = {c.inets[o0 + j], h[1] ? c.inets[o0 + j + 8] : 0};
        const int fr[2] = {ft & 0xffff, ft & 0xffff}, to[2] = {ft >> 16, ft >> 16};
        int a[2];
        commit_group<2>(c, h, e, fr, to, a, tg);
        att += a[0] + a[1];
      }
    }
    if (toggles) *toggles += tg;
    return att;
  }
  *total = flat_scan(f, n);
  if (degrees && threadIdx.x == 0) *degrees += *total;
  return flat_commit<kTeamGroup>(c, f, n, *total, false, toggles);
}

// Adds this thread's attributed delta to the CTA's, flushes the CTA's block
// weight deltas and delta (T > 1), and meets the team. Afterwards s.dw is
// zero, and for T = 1 s.bw holds the new weights.
template <typename TS>
__device__ __forceinline__ bool team_close_moves(const PxInst& I, Team& tm, TS& s, int q, int64_t att) {
  att = warp_sum(att);
  if (lane_id() == 0 && att) atomicAdd(reinterpret_cast<ull*>(&s.delta), (ull)att);
  __syncthreads();
  for (int b = threadIdx.x; b < I.k; b += blockDim.x) {
    const ull d = s.dw[b];
    if (d) {
      if (tm.T > 1)
        atomicAdd(reinterpret_cast<ull*>(&I.bw[I.boff + b]), d);
      else
        s.bw[b] += (int64_t)d;
      s.dw[b] = 0;
    }
  }
  if (threadIdx.x == 0) {
    if (tm.T > 1 && s.delta != s.gdelta) atomicAdd(tm.G.delta(q), (ull)(s.delta - s.gdelta));
    s.gdelta = s.delta;  // what the team has of this CTA's delta
  }
  return team_sync(tm, s);
}

// Block weights, reverts and delta of the team after a barrier (T > 1; for
// T = 1 they are the CTA's own), in one round trip.
template <typename TS>
__device__ __forceinline__ void team_state(const PxInst& I, const Team& tm, TS& s, int q) {
  if (tm.T > 1) {
    for (int b = threadIdx.x; b < I.k; b += blockDim.x) s.bw[b] = I.bw[I.boff + b];
    if (threadIdx.x == kTeamThreads - 1) {
      s.grev = (int)*tm.G.nrev(q);
      s.tdelta = (long long)*tm.G.delta(q);
    }
  } else if (threadIdx.x == 0) {
    s.grev = s.nrev;
    s.tdelta = s.delta;
  }
  __syncthreads();
}

// The round's active vertices grouped by sub-round, from the flags (which are
// cleared): sub-round j is list[s.off[j] .. s.off[j + 1]), of the CTA's own
// vertices (by their index in the CTA) or, for a team that shares its list, of
// all of the team's. Returns their number, -1: aborted.
template <bool OWN, typename TS>
__device__ int team_build_list(const PxInst& I, const PxParams& P, Team& tm, TS& s, int round) {
  const bool shared = !OWN && tm.T > 1;
  int32_t* list = s.V.list;
  uint32_t* masks = s.V.masks;
  const int chunks = s.V.chunks;
  const int lane = lane_id(), wid = threadIdx.x >> 5, S = P.S;
  const int ni = (int)(I.v1 - I.v0);
  for (int j = threadIdx.x; j < S; j += blockDim.x) s.fill[j] = 0;
  __syncthreads();
  for (int i = wid; i < chunks; i += kTeamWarps) {
    const int lv = ((i * tm.T + tm.rank) << kChunkShift) + lane;
    const bool f = lv < ni && I.flag[I.v0 + lv] != 0;
    if (f) I.flag[I.v0 + lv] = 0;
    const unsigned m = __ballot_sync(FULLMASK, f);
    if (lane == 0) {
      masks[i] = m;
      if (m) atomicAdd(&s.fill[subround_of(lv, round, S)], __popc(m));
    }
  }
  __syncthreads();
  if (shared) {
    const int r = tm.builds % 3;
    for (int j = threadIdx.x; j < S; j += blockDim.x)
      s.kbeg[j] = s.fill[j] ? (int)atomicAdd(tm.G.count(r) + j, (ull)s.fill[j]) : 0;
    if (!team_sync(tm, s)) return -1;
    if (tm.rank == 0)  // nobody reads the counts of the round before last any more
      for (int j = threadIdx.x; j < kMaxSubrounds; j += blockDim.x) tm.G.count(r == 2 ? 0 : r + 1)[j] = 0;
    for (int j = threadIdx.x; j < S; j += blockDim.x) s.fill[j] = (int)tm.G.count(r)[j];
    __syncthreads();
  }
  ++tm.builds;
  if (threadIdx.x < 32) {  // S <= 64: two bins per lane
    const int a = 2 * lane < S ? s.fill[2 * lane] : 0, b = 2 * lane + 1 < S ? s.fill[2 * lane + 1] : 0;
    int incl = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULLMASK, incl, o);
      if (lane >= o) incl += y;
    }
    const int excl = incl - a - b;
    __syncwarp();
    if (2 * lane < S) {
      s.off[2 * lane] = excl;
      s.fill[2 * lane] = excl + (shared ? s.kbeg[2 * lane] : 0);
    }
    if (2 * lane + 1 < S) {
      s.off[2 * lane + 1] = excl + a;
      s.fill[2 * lane + 1] = excl + a + (shared ? s.kbeg[2 * lane + 1] : 0);
    }
    if (lane == 31) s.off[S] = incl;
  }
  __syncthreads();
  for (int i = wid; i < chunks; i += kTeamWarps) {
    const unsigned m = masks[i];
    if (!m) continue;
    const int lv = (i * tm.T + tm.rank) << kChunkShift;
    int at = 0;
    if (lane == 0) at = atomicAdd(&s.fill[subround_of(lv, round, S)], __popc(m));
    at = __shfl_sync(FULLMASK, at, 0);
    if ((m >> lane) & 1u) list[at + __popc(m & lanemask_lt())] = (OWN ? i << kChunkShift : lv) + lane;
  }
  if (shared) {
    if (!team_sync(tm, s)) return -1;
  } else {
    __syncthreads();
  }
  return s.off[S];
}

// One sub-round; `q` is its slot of the team's totals. False: aborted or, with
// *idle set, the round has no active vertex in the whole team.
template <int W, bool UNIT, int U, bool OWN, typename TS>
__device__ bool team_subround(const PxInst& I, const PxParams& P, const RoundCtx& c, Team& tm, TS& s,
                              unsigned char* area, int sub, int q, int64_t& t_pins, int64_t& t_moved_pins,
                              int64_t& t_toggles, bool* idle) {
  constexpr int PL = UNIT ? 6 : 8;
  FlatSmem& f = *reinterpret_cast<FlatSmem*>(area);
  const int lane = lane_id(), k = I.k, T = tm.T, vbits = s.V.vbits;
  const TeamGlob& G = tm.G;
  // ---- slack, feasibility masks, per-block totals
  for (int b = threadIdx.x; b < k; b += blockDim.x) {
    const int64_t sl = s.lmax[b] - s.bw[b];
    s.slack[b] = sl < 0 ? -1 : (sl > INT_MAX ? INT_MAX : (int)sl);
    s.in_w[b] = s.out_w[b] = 0;
    s.in_cnt[b] = s.cur[b] = s.base[b] = 0;
    s.thr_to[b] = s.thr_from[b] = ~0ull;
  }
  if (threadIdx.x == 0) {
    s.ncand = s.nrev = s.rolled = s.tile = s.nheavy = s.nhuge = 0;
    s.any = 0;
    s.delta = s.gdelta = 0;
    const int beg = s.off[sub], cnt = s.off[sub + 1] - beg;
    s.V.beg = beg;
    s.V.cnt = cnt;
    if (!OWN && T > 1) {  // an equal part of the team's list, and of the scratch arrays at its place
      const int lo = (int)((int64_t)cnt * tm.rank / T), hi = (int)((int64_t)cnt * (tm.rank + 1) / T);
      s.V.beg = beg + lo;
      s.V.cnt = s.V.len = hi - lo;
      s.V.rec = I.rec + I.v0 + beg + lo;
      s.V.status = I.status + I.v0 + beg + lo;
      s.V.heavy = I.kw + beg + lo;
      s.V.kept = I.cand + beg + lo;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x >> 5; i < kLvWeights * W; i += kTeamWarps) {
    const int w = i / W + 1, b = 32 * (i % W) + lane;
    const unsigned m = __ballot_sync(FULLMASK, b < k && s.slack[b] >= w);
    if (lane == 0) s.fmask[i] = m;
  }
  __syncthreads();
  // ---- sweep: warps take tiles of 32 / G vertices, G lanes evaluate one: few
  // vertices leave warps idle, which then shorten the longest incidence walk
  // (131,071 vertices on 152 CTAs, 123 per CTA and sub-round: sweep 6.8 -> 5.6
  // us together with the resident part, the wait for its slowest CTA 4.7 -> 4.2
  // us); heavy vertices are set aside and evaluated by a warp or the CTA
  {
    const int beg = s.V.beg, cnt = s.V.cnt;
    constexpr int wide = W <= 4 ? 0 : W == 8 ? 1 : W == 16 ? 2 : 3;  // k > 128: log2 of the W / 4 lanes per vertex
    const int gs = wide ? wide : !OWN ? 0 : cnt <= 8 * kTeamWarps ? 2 : cnt <= 16 * kTeamWarps ? 1 : 0;  // log2 G
    const int vi = OWN ? lane >> gs : lane, part_of = lane & ((1 << gs) - 1);
    for (;;) {
      int tile = 0;
      if (lane == 0) tile = atomicAdd(&s.tile, 32 >> gs);
      tile = __shfl_sync(FULLMASK, tile, 0);
      if (tile >= cnt) break;
      int li = 0, from = 0, to = 0, gain = 0, wv = 0, d = 0;
      int64_t o0 = 0;
      if (tile + vi < cnt) {
        li = s.V.list[beg + tile + vi];
        int64_t dd;
        team_vertex<OWN>(tm, s, li, o0, dd, from, wv);
        to = from;
        if (!OWN || part_of == 0) t_pins += dd;
        d = dd > kHighDegree ? 0 : (int)dd;  // isBorderNode is false above the threshold
        if ((int64_t)d * I.max_we >= (1 << PL)) {  // beyond the lane counters
          if (!OWN || part_of == 0) {
            if (d <= kTeamHuge)
              s.V.heavy[atomicAdd(&s.nheavy, 1)] = li;
            else
              s.V.heavy[s.V.len - 1 - atomicAdd(&s.nhuge, 1)] = li;
          }
          d = 0;
        }
        if constexpr (!OWN) {
          bool border = false;
          if (d > 0)
            lv_vertex<W, UNIT, PL, U, false>(c, o0, d, from, wv, 0, 0, false, P.zero_gain, s.fmask, s.slack, s.bw,
                                             s.perf, to, gain, border);
        }
      }
      if constexpr (W > 4)
        team_lv_wide<W, UNIT, PL, U>(c, s, o0, d, from, wv, part_of, P.zero_gain, to, gain);
      else if constexpr (OWN)
        team_lv_vertex<W, UNIT, PL, U>(c, s, o0, d, from, wv, 1 << gs, part_of, P.zero_gain, to, gain);
      team_candidates<OWN>(s, (!OWN || part_of == 0) && to != from, li, gain, from, to, wv);
    }
    __syncthreads();
    if (s.nheavy | s.nhuge) {
      team_heavy<W, UNIT, OWN>(P, c, tm, s);
      __syncthreads();
    }
  }
  const int ncand = s.ncand;
  if (T > 1) {
    for (int b = threadIdx.x; b < k; b += blockDim.x) {
      if (s.in_cnt[b]) {
        atomicAdd(G.in_w(q) + b, s.in_w[b]);
        s.base[b] = (unsigned)atomicAdd(G.in_cnt(q) + b, (ull)s.in_cnt[b]);
      }
      if (s.out_w[b]) atomicAdd(G.out_w(q) + b, s.out_w[b]);
    }
    if (OWN && sub == 0 && threadIdx.x == 0 && s.off[P.S]) atomicAdd(G.active(q), (ull)s.off[P.S]);
  }
  TEAM_SYNC();
  // ---- plan: target blocks whose candidates weigh more than the slack, and
  // whether some source block could lose its whole weight
  if (T > 1 && tm.rank == 0) {  // the previous sub-round's slot is free again
    const int z = q == 0 ? 2 : q - 1;
    for (int b = threadIdx.x; b < 5 * G.K + 8; b += blockDim.x) G.slot(z)[b] = 0;
  }
  for (int b = threadIdx.x; b < k; b += blockDim.x) {
    const int64_t in_w = T > 1 ? (int64_t)*(G.in_w(q) + b) : (int64_t)s.in_w[b];
    const int64_t out = T > 1 ? (int64_t)*(G.out_w(q) + b) : (int64_t)s.out_w[b];
    const int64_t cnt = T > 1 ? (int64_t)*(G.in_cnt(q) + b) : (int64_t)s.in_cnt[b];
    const bool over = in_w > s.lmax[b] - s.bw[b];
    s.over[b] = over;
    s.tot_cnt[b] = cnt;
    const int bits = (over ? 1 : 0) | (out >= s.bw[b] ? 2 : 0) | (cnt > 0 ? 4 : 0);
    if (bits) atomicOr(&s.any, bits);
  }
  if (sub == 0) {
    const int64_t act = OWN && T > 1 ? (int64_t)*(G.active(q)) : (int64_t)s.off[P.S];
    if (act == 0) {  // the same in every CTA
      *idle = true;
      __syncthreads();
      return false;
    }
  }
  __syncthreads();
  const int flags = s.any;
  if (!(flags & 4)) {  // no candidate in the team
    if (threadIdx.x == 0) s.kpre[sub] = s.nkept;
    __syncthreads();
    return true;
  }
  // ---- target side (the atomic weight check of changeNodePart, h:548-562):
  // per block the longest (gain, vertex) prefix within L_max
  if (flags & 1) {
    team_plan(I, s);
    for (int i = threadIdx.x; i < ncand; i += blockDim.x) {
      const int4 r = team_rec<OWN>(s, i);
      const int b = r.z & 0xffff;
      if (s.over[b]) {
        const int64_t slot = s.seg[b] + s.base[b] + atomicAdd(&s.cur[b], 1u);
        I.keys[slot] = team_key(r.y, team_lv<OWN>(tm, r.x), vbits);
        I.kw[slot] = r.w;
      }
    }
    TEAM_SYNC();
    team_select(I, tm, s, area, G.thr_to(), s.thr_to, [&](int b) { return s.lmax[b] - s.bw[b]; });
    TEAM_SYNC();
    if (T > 1) {
      for (int j = threadIdx.x; j < s.nover; j += blockDim.x)
        s.thr_to[s.over_ids[j]] = *(G.thr_to() + s.over_ids[j]);
      __syncthreads();
    }
  }
  // ---- source side (from_weight_after > 0, h:551): per block the longest
  // prefix of its target-accepted moves that leaves weight >= 1
  if (flags & 2) {
    for (int b = threadIdx.x; b < k; b += blockDim.x) {
      s.in_w[b] = 0;
      s.in_cnt[b] = s.cur[b] = s.base[b] = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ncand; i += blockDim.x) {
      const int4 r = team_rec<OWN>(s, i);
      if (team_key(r.y, team_lv<OWN>(tm, r.x), vbits) < s.thr_to[r.z & 0xffff]) {
        atomicAdd(&s.in_w[r.z >> 16], (ull)(int64_t)r.w);
        atomicAdd(&s.in_cnt[r.z >> 16], 1u);
      }
    }
    __syncthreads();
    if (T > 1) {
      for (int b = threadIdx.x; b < k; b += blockDim.x)
        if (s.in_cnt[b]) {
          atomicAdd(G.acc_w(q) + b, s.in_w[b]);
          s.base[b] = (unsigned)atomicAdd(G.acc_cnt(q) + b, (ull)s.in_cnt[b]);
        }
      TEAM_SYNC();
    }
    bool any = false;
    for (int b = threadIdx.x; b < k; b += blockDim.x) {
      const int64_t w = T > 1 ? (int64_t)*(G.acc_w(q) + b) : (int64_t)s.in_w[b];
      const int64_t n = T > 1 ? (int64_t)*(G.acc_cnt(q) + b) : (int64_t)s.in_cnt[b];
      s.tot_cnt[b] = n;
      s.over[b] = n > 0 && s.bw[b] - w < 1;
      any |= s.over[b] != 0;
    }
    if (__syncthreads_or(any)) {
      team_plan(I, s);
      for (int i = threadIdx.x; i < ncand; i += blockDim.x) {
        const int4 r = team_rec<OWN>(s, i);
        const int b = r.z >> 16;
        const uint64_t key = team_key(r.y, team_lv<OWN>(tm, r.x), vbits);
        if (s.over[b] && key < s.thr_to[r.z & 0xffff]) {
          const int64_t slot = s.seg[b] + s.base[b] + atomicAdd(&s.cur[b], 1u);
          I.keys[slot] = key;
          I.kw[slot] = r.w;
        }
      }
      TEAM_SYNC();
      team_select(I, tm, s, area, G.thr_from(), s.thr_from, [&](int b) { return s.bw[b] - 1; });
      TEAM_SYNC();
      if (T > 1) {
        for (int j = threadIdx.x; j < s.nover; j += blockDim.x)
          s.thr_from[s.over_ids[j]] = *(G.thr_from() + s.over_ids[j]);
        __syncthreads();
      }
    }
  }
  // ---- commit of the accepted moves
  int64_t att = 0;
  int total = 0, n = 0;
  for (int c0 = 0; c0 < ncand; c0 += kFlatItems) {
    team_gather<OWN>(tm, s, f, c0, ncand, false, 0, true, [&](int i, const int4& r) {
      const uint64_t key = team_key(r.y, team_lv<OWN>(tm, r.x), vbits);
      const bool acc = key < s.thr_to[r.z & 0xffff] && key < s.thr_from[r.z >> 16];
      team_set_status<OWN>(s, i, acc ? 1 : 0);
      return acc;
    });
    n = f.n;
    att += team_commit<OWN>(c, s, f, n, &total, &t_moved_pins, &t_toggles);
    if (c0 + kFlatItems < ncand) __syncthreads();
  }
  if (!team_close_moves(I, tm, s, q, att)) return false;
  if (!P.revert) team_state(I, tm, s, q);
  // ---- hindsight reverts: every committed move is evaluated on the
  // post-commit state before any is undone (moveVertex,
  // label_propagation_refiner.h:100-137, made deterministic)
  if (P.revert) {
    for (int c0 = 0; c0 < ncand; c0 += kFlatItems) {
      if (ncand > kFlatItems) {  // otherwise the commit's items are still there
        team_gather<OWN>(tm, s, f, c0, ncand, false, 0, false,
                    [&](int i, const int4&) { return team_status<OWN>(s, i) == 1; });
        n = f.n;
        total = flat_scan(f, n);
      } else if (team_short<OWN>(s, n)) {
        const int it = threadIdx.x >> 3;
        int g = 0;
        if (it < n) {
          const int64_t o0 = f.o0[it];
          const int d = f.pre[it], ft = f.ft[it];
          for (int j = threadIdx.x & 7; j < d; j += 8) {
            const int64_t e = c.inets[o0 + j];
            const uint32_t* r = c.conn + e * 2 * W;
            const uint32_t lf = (r[(ft & 0xffff) >> 5] >> (ft & 31)) & 1u;
            const uint32_t l1 = (r[W + (ft >> 21)] >> ((ft >> 16) & 31)) & 1u;
            const int we = UNIT ? 1 : c.w_e[e];
            if (l1 == lf) g += l1 ? -we : we;
          }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) g += __shfl_xor_sync(FULLMASK, g, o);
        if (it < n && (threadIdx.x & 7) == 0 && g < 0) {
          team_set_status<OWN>(s, f.pos[it], 2);
          atomicAdd(&s.nrev, 1);
        }
        __syncthreads();
        continue;
      }
      // gain of moving back: + w(e) if Φ(e, to) > 1, - w(e) if from is in Λ(e)
      for (int x0 = threadIdx.x; x0 < total; x0 += kTeamGroup * kTeamThreads) {
        int it[kTeamGroup], e[kTeamGroup];
        uint32_t l1[kTeamGroup], lf[kTeamGroup];
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u) {
          const int x = x0 + u * kTeamThreads;
          it[u] = x < total ? flat_find(f, n, x) : -1;
          e[u] = it[u] >= 0 ? c.inets[f.o0[it[u]] + (x - f.pre[it[u]])] : 0;
        }
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u) {
          l1[u] = lf[u] = 0;
          if (it[u] >= 0) {
            const int ft = f.ft[it[u]];
            const uint32_t* r = c.conn + (int64_t)e[u] * 2 * W;
            lf[u] = (r[(ft & 0xffff) >> 5] >> (ft & 31)) & 1u;
            l1[u] = (r[W + (ft >> 21)] >> ((ft >> 16) & 31)) & 1u;
          }
        }
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u)
          if (it[u] >= 0 && l1[u] == lf[u]) {
            const int we = UNIT ? 1 : c.w_e[e[u]];
            atomicAdd(&f.att[it[u]], l1[u] ? -we : we);
          }
      }
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (f.att[i] < 0) {
          team_set_status<OWN>(s, f.pos[i], 2);
          atomicAdd(&s.nrev, 1);
        }
      __syncthreads();
    }
    if (T > 1) {
      if (threadIdx.x == 0 && s.nrev) atomicAdd(G.nrev(q), (ull)s.nrev);
      TEAM_SYNC();
    }
    team_state(I, tm, s, q);
    if (s.grev) {
      att = 0;
      if (s.nrev)
        for (int c0 = 0; c0 < ncand; c0 += kFlatItems) {
          team_gather<OWN>(tm, s, f, c0, ncand, true, 0, true,
                      [&](int i, const int4&) { return team_status<OWN>(s, i) == 2; });
          att += team_commit<OWN>(c, s, f, f.n, &total, nullptr, nullptr);
          __syncthreads();
        }
      if (!team_close_moves(I, tm, s, q, att)) return false;
      team_state(I, tm, s, q);
    }
  }
  // ---- rollback of a sub-round whose summed delta is positive
  if (P.rollback && s.tdelta > 0) {
    // every CTA has read the delta before any adds the rollback's part
    TEAM_SYNC();
    att = 0;
    for (int c0 = 0; c0 < ncand; c0 += kFlatItems) {
      team_gather<OWN>(tm, s, f, c0, ncand, true, 3, true,
                  [&](int i, const int4&) { return team_status<OWN>(s, i) == 1; });
      if (threadIdx.x == 0) s.rolled += f.n;
      att += team_commit<OWN>(c, s, f, f.n, &total, nullptr, nullptr);
      __syncthreads();
    }
    if (!team_close_moves(I, tm, s, q, att)) return false;
    team_state(I, tm, s, q);
  }
  // ---- kept moves (they activate the next round's vertices), statistics
  const bool shared = !OWN && T > 1;
  const int at0 = s.nkept;
  __syncthreads();
  for (int i0 = 0; i0 < ncand; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    const bool keep = i < ncand && team_status<OWN>(s, i) == 1;
    const int slot = flat_append_to(&s.nkept, keep);
    if (keep) s.V.kept[shared ? slot - at0 : slot] = team_rec<OWN>(s, i).x;
  }
  if (threadIdx.x == 0) {
    s.st[kStCands] += ncand;
    s.st[kStReverted] += s.nrev + s.rolled;
    s.st[kStDelta] += s.delta;
    if (shared) {
      s.kbeg[sub] = s.V.beg;
      s.kpre[sub] = at0;
    }
  }
  __syncthreads();
  return true;
}

// Nets of more than kTeamWideNet pins are listed by an expansion (P.wide: some can be
// stamped) and then dealt to the CTAs: where they lie side by side, one CTA's tile
// held them all (400 nets of 8,192 pins beside 400,000 of 4, k = 2, no threshold:
// 14,232 us, now 2,113; multi-launch pipeline 9,294. Zipf 1M, k = 32 4,010 -> 4,033,
// row-net 1M, k = 61 3,780 -> 3,726, 4.2M 10,301 -> 10,165). Above kTeamBigNet they do
// not fit the flat sums.
constexpr int kTeamBigNet = 65536;

// Copies `words` 32-bit words from src to dst (whole CTA).
__device__ __forceinline__ void team_copy(uint32_t* dst, const uint32_t* src, int64_t words) {
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < words; i += kTeamThreads) dst[i] = src[i];
}

// This CTA's part of the instance (s.V) and the pointers its phases use (s.c).
// The scratch arrays hold 32 entries per chunk; the CTA with the last,
// possibly partial chunk comes last. What fits into the launch's P.resident
// bytes of shared memory at `own` is copied there: the vertices' arrays, and
// for a team of one CTA whose arrays start at net 0 also the nets' records and
// pin counts.
template <typename TS>
__device__ void team_part(const PxInst& I, int resident, bool shared, const Team& tm, TS& s, unsigned char* own) {
  const int T = tm.T, ni = (int)(I.v1 - I.v0), lane = lane_id(), wid = threadIdx.x >> 5;
  const int nch = (ni + 31) >> kChunkShift, base = nch / T, rem = nch % T;
  const int chunks = base + (tm.rank < rem ? 1 : 0);
  const int last = rem ? rem - 1 : T - 1;
  const int64_t r0 = 32ll * (tm.rank > last ? (int64_t)(tm.rank - last - 1) * base
                                            : (int64_t)(T - 1 - last) * base + (int64_t)tm.rank * (base + (rem ? 1 : 0)));
  const int len = chunks == 0 ? 0 : (tm.rank == last ? ni - (int)r0 : 32 * chunks);
  int32_t* off = reinterpret_cast<int32_t*>(own);
  int32_t *wv = off + len + 1, *part = wv + len, *list = part + len, *inets = list + len;
  int64_t left = (int64_t)resident - 4 * (4 * (int64_t)len + 1);
  // incidences per chunk, then the chunks' starts
  int64_t run = 0;
  const bool room = left > 0;
  if (room)
    for (int c0 = 0; c0 < chunks; c0 += kTeamThreads) {
      const int i = c0 + threadIdx.x;
      int64_t size = 0;
      if (i < chunks) {
        const int v = team_lv<true>(tm, i << kChunkShift);
        size = I.vtx_off[I.v0 + min(v + 32, ni)] - I.vtx_off[I.v0 + v];
      }
      int64_t total;
      const int64_t at = run + block_scan_excl_i64(size, &total);
      if (i < chunks) off[i << kChunkShift] = (int)min(at, (int64_t)INT_MAX);
      run += total;
    }
  left -= 4 * run;
  const bool res = room && left >= 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    RoundCtx c{};
    c.inets = res ? inets : I.inets;
    c.w_e = I.w_e;
    c.phi = I.phi;
    c.conn = I.conn;
    c.k = I.k;
    c.W = I.W;
    c.kmax = I.kstride;
    c.unit_nets = I.unit_nets;
    c.phi16 = I.phi16;
    c.max_we = I.max_we;
    s.c = c;
    s.V.rec = I.rec + I.v0 + r0;
    s.V.status = I.status + I.v0 + r0;
    s.V.list = res ? list : shared ? I.list : I.list + r0;  // a shared list holds the whole team's vertices
    s.V.heavy = I.kw + r0;
    s.V.kept = I.cand + r0;
    s.V.masks = reinterpret_cast<uint32_t*>(I.cand + r0);
    s.V.off = res ? off : nullptr;
    s.V.wv = wv;
    s.V.part = part;
    s.V.len = len;
    s.V.chunks = chunks;
    s.V.vbits = 32 - __clz(ni > 1 ? ni - 1 : 1);
    s.V.own_nets = 0;
  }
  if (res) {
    for (int i = wid; i < chunks; i += kTeamWarps) {
      const int lv = team_lv<true>(tm, i << kChunkShift) + lane, li = (i << kChunkShift) + lane;
      const int64_t v = I.v0 + min(lv, ni - 1);
      const int at = off[i << kChunkShift];
      const int64_t g = I.vtx_off[v], g0 = __shfl_sync(FULLMASK, g, 0);
      const int64_t size = __shfl_sync(FULLMASK, I.vtx_off[v + 1], 31) - g0;
      __syncwarp();
      if (lv < ni) {
        off[li] = at + (int)(g - g0);
        wv[li] = I.w_v[v];
        part[li] = I.part[v] - I.boff;
      }
      for (int64_t x = lane; x < size; x += 32) inets[at + x] = I.inets[g0 + x];
    }
    if (threadIdx.x == 0) off[len] = (int)run;
  }
  __syncthreads();
  if (T == 1 && res && I.e0 == 0) {
    // 16-byte boundary for the record loads
    uint32_t* at = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(inets + run) + 15) & ~(uintptr_t)15);
    left -= 16;
    const int64_t cw = I.e1 * 2 * I.W, pe = I.e1 * I.kstride, pw = I.phi16 ? (pe + 1) / 2 : pe;
    int nets = 0;
    if (left >= 4 * cw) {
      left -= 4 * cw;
      team_copy(at, I.conn, cw);
      if (threadIdx.x == 0) s.c.conn = at;
      at += cw;
      nets |= 1;
    }
    if (left >= 4 * pw) {
      team_copy(at, reinterpret_cast<const uint32_t*>(I.phi), pw);
      if (threadIdx.x == 0) s.c.phi = reinterpret_cast<int32_t*>(at);
      nets |= 2;
    }
    if (threadIdx.x == 0) s.V.own_nets = nets;
    __syncthreads();
  }
}

// Writes the nets' records and pin counts back.
template <typename TS>
__device__ void team_put_back(const PxInst& I, const TS& s) {
  if (s.V.own_nets & 1) team_copy(I.conn, s.c.conn, I.e1 * 2 * I.W);
  if (s.V.own_nets & 2) {
    const int64_t pe = I.e1 * I.kstride;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(s.c.phi);
    team_copy(reinterpret_cast<uint32_t*>(I.phi), src, I.phi16 ? pe / 2 : pe);
    if (I.phi16 && (pe & 1) && threadIdx.x == 0)  // the last word's other half may be another instance's
      reinterpret_cast<uint16_t*>(I.phi)[pe - 1] = reinterpret_cast<const uint16_t*>(src)[pe - 1];
  }
}

// All rounds of one instance (P.rounds, fewer when no vertex is active). `q`
// continues over instances. False: aborted.
template <int W, bool UNIT, int U, bool OWN, typename TS>
__device__ bool team_instance(const PxInst& I, const PxParams& P, Team& tm, TS& s, unsigned char* area,
                              int& q) {
  FlatSmem& f = *reinterpret_cast<FlatSmem*>(area);
  const int k = I.k, T = tm.T, lane = lane_id();
  const bool shared = !OWN && T > 1;
  team_part(I, OWN ? P.resident : 0, shared, tm, s, area + kTeamOwnAt<TS::kBlocks>);
  // with 64 registers and 4-word records the pointers are better re-read from
  // shared memory than spilled (4.2M vertices 11,880 -> 11,270 us)
  typename std::conditional<(OWN || W < 4), const RoundCtx, const RoundCtx&>::type c = s.c;
  const int32_t* kept = s.V.kept;
  for (int b = threadIdx.x; b < k; b += blockDim.x) {
    s.bw[b] = I.bw[I.boff + b];
    s.lmax[b] = I.lmax[I.boff + b];
    s.perf[b] = I.perfect[I.boff + b];
    s.dw[b] = 0;
  }
  const int first = P.round >= 0 ? P.round : I.round;
  for (int round = first; round < first + P.rounds; ++round) {
    if (threadIdx.x < kStats) s.st[threadIdx.x] = 0;
    if (threadIdx.x == 0) s.nkept = 0;
    const int active = team_build_list<OWN>(I, P, tm, s, round);
    if (active < 0) return false;
    int64_t t_pins = 0, t_moved_pins = 0, t_toggles = 0;
    bool idle = false;
    for (int sub = 0; sub < P.S; ++sub) {
      const bool ok = team_subround<W, UNIT, U, OWN>(I, P, c, tm, s, area, sub, q, t_pins, t_moved_pins, t_toggles,
                                                       &idle);
      q = q == 2 ? 0 : q + 1;
      if (idle) break;
      if (!ok) return false;
    }
    if (idle) break;
    // ---- round statistics
    t_pins = warp_sum(t_pins);
    t_toggles = warp_sum(t_toggles);
    t_moved_pins = warp_sum(t_moved_pins);
    if (lane == 0) {
      atomicAdd(reinterpret_cast<ull*>(&s.st[kStMovedPins]), (ull)t_moved_pins);
      atomicAdd(reinterpret_cast<ull*>(&s.st[kStPins]), (ull)t_pins);
      atomicAdd(reinterpret_cast<ull*>(&s.st[kStToggles]), (ull)t_toggles);
    }
    if (threadIdx.x == 0) {
      s.st[kStActive] = !shared || tm.rank == 0 ? active : 0;
      s.kpre[P.S] = s.nkept;
      s.st[kStMoved] = s.nkept;
    }
    __syncthreads();
    if (threadIdx.x < kStats && s.st[threadIdx.x])
      atomicAdd(reinterpret_cast<ull*>(&I.stats[(int64_t)round * kStats + threadIdx.x]), (ull)s.st[threadIdx.x]);
    if (round + 1 == first + P.rounds && !P.activate_last) break;
    // ---- activation of the kept moves (label_propagation_refiner.h:112-128):
    // the vertex, and the pins of its nets with |e| <= threshold through a stamp
    const int stamp = round + 1, nkept = s.nkept;
    for (int c0 = 0; c0 < nkept; c0 += kFlatItems) {
      const int n = min(kFlatItems, nkept - c0);
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int li;
        if (shared) {  // the sub-rounds' kept moves lie apart
          int j = 0;
          while (s.kpre[j + 1] <= c0 + i) ++j;
          li = I.cand[s.kbeg[j] + c0 + i - s.kpre[j]];
        } else {
          li = kept[c0 + i];
        }
        int64_t o0, d;
        team_degree<OWN>(tm, s, li, o0, d);
        f.o0[i] = o0;
        f.pre[i] = (int)d;
        I.flag[I.v0 + team_lv<OWN>(tm, li)] = 1;
      }
      __syncthreads();
      const int total = flat_scan(f, n);
      for (int x0 = threadIdx.x; x0 < total; x0 += kTeamGroup * kTeamThreads) {
        int e[kTeamGroup];
        int64_t size[kTeamGroup];
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u) {
          const int x = x0 + u * kTeamThreads;
          const int it = x < total ? flat_find(f, n, x) : 0;
          e[u] = x < total ? c.inets[f.o0[it] + (x - f.pre[it])] : -1;
        }
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u) size[u] = e[u] >= 0 ? I.net_off[e[u] + 1] - I.net_off[e[u]] : INT64_MAX;
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u)
          if (e[u] >= 0 && size[u] <= P.act_threshold) I.net_epoch[e[u]] = stamp;
      }
      __syncthreads();
    }
    TEAM_SYNC();
    // expansion: the pins of the stamped nets, CTA-flat over tiles of nets
    ull* wide = T > 1 ? tm.G.wide() : reinterpret_cast<ull*>(&s.hint);
    if (T == 1 && threadIdx.x == 0) s.hint = 0;
    const int room = (int)(I.v1 - I.v0);  // entries of I.cand, whose kept moves are read
    for (int64_t b0 = I.e0 + (int64_t)tm.rank * kFlatItems; b0 < I.e1; b0 += (int64_t)T * kFlatItems) {
      if (threadIdx.x == 0) f.n = 0;
      __syncthreads();
      constexpr int PER = kFlatItems / kTeamThreads;
      int64_t o0[PER], o1[PER];
      bool hit[PER];
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int64_t e = b0 + p * kTeamThreads + threadIdx.x;
        const bool in = e < I.e1;
        hit[p] = in && I.net_epoch[e] == stamp;
        o0[p] = in ? I.net_off[e] : 0;
        o1[p] = in ? I.net_off[e + 1] : 0;
      }
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        if (P.wide && hit[p] && o1[p] - o0[p] > kTeamWideNet) {
          const int at = (int)atomicAdd(wide, 1ull);
          if (at < room) {
            I.cand[at] = (int)(b0 - I.e0) + p * kTeamThreads + (int)threadIdx.x;
            hit[p] = false;
          } else if (o1[p] - o0[p] > kTeamBigNet) {  // no room in either
            for (int64_t j = o0[p]; j < o1[p]; ++j) I.flag[I.pins[j]] = 1;
            hit[p] = false;
          }
        }
        const int slot = flat_append(f, hit[p]);
        if (slot >= 0) {
          f.o0[slot] = o0[p];
          f.pre[slot] = (int)(o1[p] - o0[p]);
        }
      }
      __syncthreads();
      const int n = f.n, total = flat_scan(f, n);
      for (int x0 = threadIdx.x; x0 < total; x0 += kTeamGroup * kTeamThreads) {
        int pin[kTeamGroup];
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u) {
          const int x = x0 + u * kTeamThreads;
          const int it = x < total ? flat_find(f, n, x) : 0;
          pin[u] = x < total ? I.pins[f.o0[it] + (x - f.pre[it])] : -1;
        }
#pragma unroll
        for (int u = 0; u < kTeamGroup; ++u)
          if (pin[u] >= 0) I.flag[pin[u]] = 1;
      }
      __syncthreads();
    }
    TEAM_SYNC();
    if (P.wide) {
      const int listed = (int)min((ull)room, *wide);
      int64_t p0 = 0, p1 = 0;
      for (int i = tm.rank - T; i < listed; i += T) {  // the next net's range in flight with a net's pins
        int64_t q0 = 0, q1 = 0;
        if (i + T < listed) {
          const int64_t e = I.e0 + I.cand[i + T];
          q0 = I.net_off[e];
          q1 = I.net_off[e + 1];
        }
        for (int64_t j = p0 + threadIdx.x; j < p1; j += kTeamThreads) I.flag[I.pins[j]] = 1;
        p0 = q0;
        p1 = q1;
      }
      TEAM_SYNC();
      if (T > 1 && tm.rank == 0 && threadIdx.x == 0) *wide = 0;  // nobody lists before the next round's barriers
    }
  }
  __syncthreads();
  if (T == 1) {
    for (int b = threadIdx.x; b < k; b += blockDim.x) I.bw[I.boff + b] = s.bw[b];
    if (OWN) team_put_back(I, s);
  }
  return true;
}

template <int W, bool UNIT, int U, int MINB>
__global__ void __launch_bounds__(kTeamThreads, MINB) k_team(const PxInst* __restrict__ insts,
                                                             const int32_t* __restrict__ order, int32_t count,
                                                             PxParams P, int sync, int64_t* scratch, int64_t* queue,
                                                             int64_t* err) {
  extern __shared__ __align__(16) unsigned char team_smem[];
  auto& s = *reinterpret_cast<TeamShared<kTeamBlocks<W>>*>(team_smem + kTeamSharedAt);
  Team tm;
  tm.T = P.T;
  tm.rank = blockIdx.x % P.T;
  tm.sync = sync;
  tm.arrivals = 0;
  tm.builds = 0;
  tm.G.K = P.kcap;
  tm.G.g = scratch ? scratch + (int64_t)(blockIdx.x / P.T) * team_scratch_words(P.kcap) : nullptr;
  if (threadIdx.x == 0) s.abort = 0;
  __syncthreads();
  int q = 0;
  for (;;) {
    int it = 0;
    if (sync == kSyncGrid) {
      it = 0;  // one instance
    } else {
      if (tm.rank == 0 && threadIdx.x == 0) {
        it = (int)atomicAdd(reinterpret_cast<ull*>(queue), 1ull);
        if (P.T > 1)
          *(volatile int64_t*)tm.G.item() = it;
        else
          s.item = it;
      }
      team_sync(tm, s);
      it = P.T > 1 ? (int)*(tm.G.item()) : s.item;
    }
    if (it >= count) break;
    const PxInst* src = insts + (order ? order[it] : it);
    for (int i = threadIdx.x; i < (int)(sizeof(PxInst) / 8); i += blockDim.x)
      reinterpret_cast<int64_t*>(&s.I)[i] = reinterpret_cast<const int64_t*>(src)[i];
    __syncthreads();
    if (!team_instance<W, UNIT, U, MINB == 1>(s.I, P, tm, s, team_smem, q)) {
      if (threadIdx.x == 0) *(volatile int64_t*)err = 1;
      break;
    }
    if (sync == kSyncGrid) break;
    team_sync(tm, s);  // the item word and s.item are written again
  }
}

// Kernel variant: unit net weights, sweep unroll 4 or 8 (the 2-CTA builds up to
// k = 64), compiled for 1 resident CTA per SM (up to 128 registers) or 2 (64
// registers; k <= 128).
template <int W, bool UNIT>
static const void* team_kernel_wu(int unroll, int minb) {
  (void)unroll;
  if constexpr (W <= 4) {
    if (minb >= 2) {
      if constexpr (W <= 2) {
        if (unroll == 8) return (const void*)k_team<W, UNIT, 8, 2>;
      }
      return (const void*)k_team<W, UNIT, 4, 2>;
    }
  }
  return (const void*)k_team<W, UNIT, 4, 1>;
}

}  // namespace lpgpu
