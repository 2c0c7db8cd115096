// Device helpers shared by the kernel files: warp and CTA reductions, packed
// incidence walks, the lane-per-vertex best-move evaluation and the CTA-flat
// commit. Everything here is inlined or internal to the including file.
#pragma once

#include "common.cuh"

namespace lpgpu {

#define FULLMASK 0xffffffffu


__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned lanemask_lt() { return (1u << lane_id()) - 1u; }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLMASK, v, o);
  return v;
}

// Block-wide sum of an int64 (any blockDim multiple of 32, <= 1024). All threads get the total.
static __device__ int64_t block_sum_i64(int64_t v) {
  __shared__ int64_t ws[32];
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane_id() == 0) ws[w] = v;
  __syncthreads();
  int64_t t = lane_id() < nw ? ws[lane_id()] : 0;
  t = warp_sum(t);
  return t;
}

// Block-wide exclusive scan of an int64 (blockDim multiple of 32, <= 1024).
static __device__ int64_t block_scan_excl_i64(int64_t v, int64_t* total) {
  __shared__ int64_t ws[32];
  const int lane = lane_id(), w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(FULLMASK, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    int64_t s = lane < nw ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(FULLMASK, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) ws[lane] = s;
  }
  __syncthreads();
  const int64_t prefix = w > 0 ? ws[w - 1] : 0;
  *total = ws[nw - 1];
  return prefix + x - v;
}

// Incidence packing shared by the kernels that walk the incidences of a set
// of vertices (one per lane). Vertices of degree 1..32 are packed greedily
// into groups of <= 32 incidences (lane = incidence, contiguous per vertex);
// longer vertices are walked alone in 32-incidence chunks. For every group
// `body(has, ow, j, seg_end)` runs on all lanes: lane `has` holds incidence j
// (index into inets) of the vertex held by lane `ow`. The return value is, on
// each selected lane, the sum over its vertex's incidences of the ints
// returned by body (segmented sums inside a group).
template <typename Body>
__device__ __forceinline__ int packed_incidences(bool sel, int64_t o0, int deg,
                                                 unsigned char* __restrict__ s_owner, Body&& body) {
  const int lane = lane_id();
  int my_total = 0;
  const bool small = sel && deg >= 1 && deg <= 32;
  const int dsm = small ? deg : 0;
  int incl = dsm;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULLMASK, incl, o);
    if (lane >= o) incl += y;
  }
  const int excl = incl - dsm;
  unsigned rem = __ballot_sync(FULLMASK, small);
  while (rem) {
    const int q = __ffs(rem) - 1;
    const int start = __shfl_sync(FULLMASK, excl, q);
    const bool inpack = ((rem >> lane) & 1u) && incl - start <= 32;
    const unsigned pmask = __ballot_sync(FULLMASK, inpack);
    const int D = __shfl_sync(FULLMASK, incl, 31 - __clz(pmask)) - start;
    const int st = excl - start;
    __syncwarp();
    if (inpack) s_owner[__popc(pmask & lanemask_lt())] = (unsigned char)lane;
    const unsigned starts = __reduce_or_sync(FULLMASK, inpack ? (1u << st) : 0u);
    __syncwarp();
    const bool has = lane < D;
    const int ow = has ? s_owner[__popc(starts & ((2u << lane) - 1u)) - 1] : lane;
    const int64_t o_ow = __shfl_sync(FULLMASK, o0, ow);
    const int st_ow = __shfl_sync(FULLMASK, st, ow);
    const int d_ow = __shfl_sync(FULLMASK, deg, ow);
    const int seg_end = has ? st_ow + d_ow : lane + 1;
    int x = body(has, ow, has ? o_ow + lane - st_ow : (int64_t)0);
    // segmented suffix sums: the first lane of every vertex gets its total
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_down_sync(FULLMASK, x, o);
      if (lane + o < seg_end) x += y;
    }
    const int tot = __shfl_sync(FULLMASK, x, inpack ? st : 0);
    if (inpack) my_total = tot;
    rem &= ~pmask;
  }
  unsigned bigm = __ballot_sync(FULLMASK, sel && deg > 32);
  while (bigm) {
    const int j = __ffs(bigm) - 1;
    bigm &= bigm - 1;
    const int64_t oj = __shfl_sync(FULLMASK, o0, j);
    const int dj = __shfl_sync(FULLMASK, deg, j);
    int acc = 0;
    for (int base = 0; base < dj; base += 32) {
      const bool has = base + lane < dj;
      acc += body(has, j, has ? oj + base + lane : (int64_t)0);
    }
    acc = warp_sum(acc);
    if (lane == j) my_total = acc;
  }
  return my_total;
}

// ====================================================== sweep / best move

// 32 x 32 bit transpose across a warp (recursive block swap with shuffles):
// on return lane j holds the word whose bit i is bit j of lane i's input.
__device__ __forceinline__ uint32_t transpose32(uint32_t x) {
  const int lane = lane_id();
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const uint32_t m = s == 16 ? 0x0000FFFFu : s == 8 ? 0x00FF00FFu : s == 4 ? 0x0F0F0F0Fu
                     : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(FULLMASK, x, s);
    x = (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y << s) & ~m));
  }
  return x;
}

// W words of a Λ record. NC: through the read-only data path (records that
// no thread of the running kernel changes); otherwise plain coherent loads.
template <int W, bool NC = true>
__device__ __forceinline__ void load_words(const uint32_t* __restrict__ p, uint32_t (&w)[W]) {
  if constexpr (W % 4 == 0) {
#pragma unroll
    for (int i = 0; i < W / 4; ++i) {
      const uint4 q = NC ? __ldg(reinterpret_cast<const uint4*>(p) + i) : reinterpret_cast<const uint4*>(p)[i];
      w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
    }
  } else if constexpr (W == 2) {
    const uint2 q = NC ? __ldg(reinterpret_cast<const uint2*>(p)) : *reinterpret_cast<const uint2*>(p);
    w[0] = q.x; w[1] = q.y;
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = NC ? __ldg(p + i) : p[i];
  }
}

// Weighted sum over the lanes in `mask` from weight bit-planes:
// sum_p popc(bits[p] & mask) << p (planes beyond kPlanes recomputed by the caller).
constexpr int kPlanes = 4;

struct Planes {
  uint32_t b[kPlanes];
  int n;  // number of planes in use (<= 31)
};

// Bit-planes of a per-lane non-negative weight `w` (all lanes participate).
__device__ __forceinline__ Planes make_planes(int w, int nplanes) {
  Planes p;
  p.n = nplanes;
#pragma unroll
  for (int i = 0; i < kPlanes; ++i) p.b[i] = i < nplanes ? __ballot_sync(FULLMASK, (w >> i) & 1) : 0u;
  return p;
}

// sum over lanes in mask of w; warp-uniform call (extra planes via ballot).
__device__ __forceinline__ int plane_sum(const Planes& p, uint32_t mask, int w) {
  int s = 0;
#pragma unroll
  for (int i = 0; i < kPlanes; ++i) s += __popc(p.b[i] & mask) << i;
  for (int i = kPlanes; i < p.n; ++i) s += __popc(__ballot_sync(FULLMASK, (w >> i) & 1) & mask) << i;
  return s;
}

// Decision of Km1Policy::computeMaxGainMoveImpl (gain_policy.h:147-166,
// disable_randomization) from penalties held by block-owning lanes: lane l
// owns blocks l + 32 t and pen[t] = sum of w(e) over incident nets with that
// block in Λ(e). score(b) = internal - pen(b); the move goes to the feasible
// block (slack(b) >= w(v), b != from) of minimum score < 0, lowest id on ties.
// Without one, and with zero_gain, the lowest feasible block of score 0 is
// taken if the rebalancing rule of label_propagation_refiner.h:88-95 holds.
template <int W, bool PACKED>
__device__ __forceinline__ void decide(int k, int from, int wv, int internal, int zero_gain,
                                       const int (&pen)[W], const int (&slack)[W],
                                       const int64_t* __restrict__ s_bw,
                                       const int64_t* __restrict__ s_perf, int& to, int& gain) {
  const int lane = lane_id();
  // quick reject: neither an improving move (pen > internal) nor a zero-gain
  // candidate (pen == internal) exists when every other block's penalty is
  // below the internal weight
  int any = -1;
#pragma unroll
  for (int t = 0; t < W; ++t) {
    const int blk = 32 * t + lane;
    if (blk != from && pen[t] > any) any = pen[t];
  }
  if (__reduce_max_sync(FULLMASK, any) < internal) return;
  int zb = INT_MAX;
  if constexpr (PACKED) {
    // penalties below 2^20: one max over (pen << 11 | 2047 - blk) gives the
    // largest penalty and, on ties, the lowest block; 0 = no feasible block
    unsigned key = 0;
#pragma unroll
    for (int t = 0; t < W; ++t) {
      const int blk = 32 * t + lane;
      if (blk < k && blk != from && slack[t] >= wv) {
        const unsigned kk = ((unsigned)pen[t] << 11) | (unsigned)(2047 - blk);
        key = kk > key ? kk : key;
        if (zb == INT_MAX && pen[t] == internal) zb = blk;
      }
    }
    const unsigned mk = __reduce_max_sync(FULLMASK, key);
    if (mk != 0 && (int)(mk >> 11) > internal) {
      to = 2047 - (int)(mk & 2047u);
      gain = internal - (int)(mk >> 11);
      return;
    }
  } else {
    int bp = -1, bb = INT_MAX;
#pragma unroll
    for (int t = 0; t < W; ++t) {
      const int blk = 32 * t + lane;
      if (blk < k && blk != from && slack[t] >= wv) {
        if (pen[t] > bp) { bp = pen[t]; bb = blk; }
        if (zb == INT_MAX && pen[t] == internal) zb = blk;
      }
    }
    const int mp = __reduce_max_sync(FULLMASK, bp);
    if (mp > internal) {
      to = __reduce_min_sync(FULLMASK, bp == mp ? bb : INT_MAX);
      gain = internal - mp;
      return;
    }
  }
  if (zero_gain) {
    const int z = __reduce_min_sync(FULLMASK, zb);
    if (z != INT_MAX && s_bw[from] - 1 > s_bw[z] + 1 && s_bw[z] < s_perf[z]) {
      to = z;
      gain = 0;
    }
  }
}



// ---- lane-per-vertex sweep (k <= 128)
//
// A lane evaluates its own vertex: it walks the vertex's incident nets and adds
// each net's Λ(e) bit vector (times w(e)) into bit-sliced counters, one
// 32-block word t and plane p per register cnt[t][p], so that bit l of plane p
// is bit p of the penalty of block 32 t + l. The best target then comes from a
// bit-sliced maximum over the feasible blocks. Vertices whose summed incident
// net weight stays below 2^PL take this path; the others take the
// warp-cooperative windows below.
constexpr int kLvWeights = 16;  // vertex weights 1..16 have precomputed feasibility masks
// Incidences per lane whose gathers are issued together (a multiple of 4), and
// resident CTAs per SM the k <= 128 sweep is compiled for.
#ifndef LPGPU_LV_UNROLL
#define LPGPU_LV_UNROLL 4
#endif
#ifndef LPGPU_SWEEP_MIN_BLOCKS
#define LPGPU_SWEEP_MIN_BLOCKS 3
#endif
static_assert(LPGPU_LV_UNROLL % 4 == 0, "the carry-save adder takes four vectors at a time");

// cnt += s0 + 2 s1 + 4 s2 (bit-sliced, ripple carry).
template <int PL>
__device__ __forceinline__ void lv_add3(uint32_t (&cnt)[PL], uint32_t s0, uint32_t s1, uint32_t s2) {
  uint32_t cy = cnt[0] & s0;
  cnt[0] ^= s0;
  uint32_t t = cnt[1];
  cnt[1] = t ^ s1 ^ cy;
  cy = (t & s1) | (cy & (t ^ s1));
  t = cnt[2];
  cnt[2] = t ^ s2 ^ cy;
  cy = (t & s2) | (cy & (t ^ s2));
#pragma unroll
  for (int p = 3; p < PL; ++p) {
    const uint32_t c2 = cnt[p] & cy;
    cnt[p] ^= cy;
    cy = c2;
  }
}

// cnt += w * x (bit-sliced; w < 2^PL).
template <int PL>
__device__ __forceinline__ void lv_add_weighted(uint32_t (&cnt)[PL], uint32_t x, int w) {
  uint32_t cy = 0;
#pragma unroll
  for (int p = 0; p < PL; ++p) {
    const uint32_t a = ((w >> p) & 1) ? x : 0u;
    const uint32_t t = cnt[p];
    cnt[p] = t ^ a ^ cy;
    cy = (t & a) | (cy & (t ^ a));
  }
}

// The next U incident nets (from index j) of the vertex with incidences
// [o0, o0 + d); -1 past its end.
template <int U, bool NC>
__device__ __forceinline__ void lv_ids(const RoundCtx& c, int64_t o0, int d, int j, int32_t (&ee)[U]) {
#pragma unroll
  for (int u = 0; u < U; ++u) ee[u] = j + u < d ? (NC ? __ldg(&c.inets[o0 + j + u]) : c.inets[o0 + j + u]) : -1;
}

// Records of U incident nets: Λ words and the Λ1 word of block word fw. A
// record of up to 16 bytes (k <= 64) comes in one load: the lanes' records lie
// in different lines, so every load instruction costs a pass per lane.
template <int W, bool UNIT, int U, bool NC>
__device__ __forceinline__ void lv_records(const RoundCtx& c, const int32_t (&ee)[U], int fw, uint32_t fbit,
                                           uint32_t (&wd)[U][W], uint32_t (&l1)[U], int (&we)[U]) {
#pragma unroll
  for (int u = 0; u < U; ++u) {
#pragma unroll
    for (int t = 0; t < W; ++t) wd[u][t] = 0;
    l1[u] = fbit;
    we[u] = 0;
    if (ee[u] >= 0) {
      const uint32_t* rec = c.conn + (int64_t)ee[u] * 2 * W;
      if constexpr (W <= 2) {
        uint32_t r[2 * W];
        load_words<2 * W, NC>(rec, r);
#pragma unroll
        for (int t = 0; t < W; ++t) wd[u][t] = r[t];
        l1[u] = W == 2 && fw ? r[2 * W - 1] : r[W];
      } else {
        load_words<W, NC>(rec, wd[u]);
        l1[u] = NC ? __ldg(rec + W + fw) : rec[W + fw];
      }
      we[u] = UNIT ? 1 : (NC ? __ldg(&c.w_e[ee[u]]) : c.w_e[ee[u]]);
    }
  }
}

// Adds U records into the bit-sliced counters and the internal weight.
template <int W, bool UNIT, int PL, int U>
__device__ __forceinline__ void lv_add(const uint32_t (&wd)[U][W], const uint32_t (&l1)[U], const int (&we)[U],
                                       uint32_t fbit, uint32_t (&cnt)[W][PL], int& internal) {
#pragma unroll
  for (int u = 0; u < U; ++u) internal += (l1[u] & fbit) ? 0 : we[u];
  if constexpr (UNIT) {
    // carry-save sum of each four vectors, then one 3-bit ripple add
#pragma unroll
    for (int g = 0; g < U; g += 4)
#pragma unroll
      for (int t = 0; t < W; ++t) {
        const uint32_t a = wd[g][t], b = wd[g + 1][t], e = wd[g + 2][t], f = wd[g + 3][t];
        const uint32_t s = a ^ b ^ e;
        const uint32_t c1 = (a & b) | (e & (a ^ b));
        const uint32_t c2 = s & f;
        lv_add3<PL>(cnt[t], s ^ f, c1 ^ c2, c1 & c2);
      }
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int t = 0; t < W; ++t) lv_add_weighted<PL>(cnt[t], wd[u][t], we[u]);
  }
}

// Best move of one vertex from its counters: the same decision as `decide`
// (Km1Policy::computeMaxGainMoveImpl with disable_randomization, plus the
// zero-gain rebalancing rule of label_propagation_refiner.h:88-95). `from`,
// `to` are local block ids; `bo` is the instance's first global block.
template <int W, int PL>
__device__ __forceinline__ void lv_decide(const RoundCtx& c, const uint32_t (&cnt)[W][PL], int internal, int from,
                                          int wv, int bo, int inst, bool batched, int zero_gain,
                                          const uint32_t* __restrict__ s_fmask, const int* __restrict__ s_slack,
                                          const int64_t* __restrict__ s_bw, const int64_t* __restrict__ s_perf,
                                          int& to, int& gain, bool& border) {
  const int fw = from >> 5;
  const uint32_t fbit = 1u << (from & 31);
  // feasible targets: c(V_b) + w(v) <= L_max(b)
  uint32_t cand[W];
  if (!batched && wv >= 1 && wv <= kLvWeights) {
#pragma unroll
    for (int t = 0; t < W; ++t) cand[t] = s_fmask[(wv - 1) * W + t];
  } else {
    const int kk = batched ? c.inst_k[inst] : c.k;
#pragma unroll
    for (int t = 0; t < W; ++t) {
      uint32_t msk = 0;
      for (int l = 0; l < 32; ++l) {
        const int b = 32 * t + l;
        if (b < kk) {
          const int64_t sl = batched ? c.lmax[bo + b] - c.bw[bo + b] : (int64_t)s_slack[b];
          if (sl >= wv) msk |= 1u << l;
        }
      }
      cand[t] = msk;
    }
  }
  // isBorderNode: some incident net holds a block other than `from`
  uint32_t other = 0, anyc = 0;
#pragma unroll
  for (int t = 0; t < W; ++t) {
    const uint32_t fm = t == fw ? ~fbit : ~0u;
    uint32_t o = 0;
#pragma unroll
    for (int p = 0; p < PL; ++p) o |= cnt[t][p];
    other |= o & fm;
    cand[t] &= fm;
    anyc |= cand[t];
  }
  if (!other) return;
  border = true;
  if (!anyc) return;
  // maximum penalty over the candidates, plane by plane from the top
  int val = 0;
#pragma unroll
  for (int p = PL - 1; p >= 0; --p) {
    uint32_t tt[W], o = 0;
#pragma unroll
    for (int t = 0; t < W; ++t) {
      tt[t] = cand[t] & cnt[t][p];
      o |= tt[t];
    }
    if (o) {
#pragma unroll
      for (int t = 0; t < W; ++t) cand[t] = tt[t];
      val |= 1 << p;
    }
  }
  if (val < internal || (val == internal && !zero_gain)) return;
  int b = 0;  // lowest block of maximum penalty
#pragma unroll
  for (int t = W - 1; t >= 0; --t)
    if (cand[t]) b = 32 * t + __ffs(cand[t]) - 1;
  if (val > internal) {
    to = b;
    gain = internal - val;
    return;
  }
  const int64_t* bwp = batched ? c.bw + bo : s_bw;
  const int64_t* pfp = batched ? c.perfect + bo : s_perf;
  if (bwp[from] - 1 > bwp[b] + 1 && bwp[b] < pfp[b]) {
    to = b;
    gain = 0;
  }
}

// Best move of one vertex by its own lane (accumulate all incidences, decide);
// U incidences per step have their gathers in flight together; NC as in
// load_words.
template <int W, bool UNIT, int PL, int U = LPGPU_LV_UNROLL, bool NC = true>
__device__ __forceinline__ void lv_vertex(const RoundCtx& c, int64_t o0, int d, int from, int wv, int bo,
                                          int inst, bool batched, int zero_gain,
                                          const uint32_t* __restrict__ s_fmask, const int* __restrict__ s_slack,
                                          const int64_t* __restrict__ s_bw, const int64_t* __restrict__ s_perf,
                                          int& to, int& gain, bool& border) {
  static_assert(U % 4 == 0, "the carry-save adder takes four vectors at a time");
  uint32_t cnt[W][PL];
#pragma unroll
  for (int t = 0; t < W; ++t)
#pragma unroll
    for (int p = 0; p < PL; ++p) cnt[t][p] = 0;
  int internal = 0;  // Σ w(e) over incident nets with Φ(e, from) > 1
  const int fw = from >> 5;
  const uint32_t fbit = 1u << (from & 31);
  int32_t ee[U];
  for (int j = 0; j < d; j += U) {
    uint32_t wd[U][W], l1[U];
    int we[U];
    lv_ids<U, NC>(c, o0, d, j, ee);
    lv_records<W, UNIT, U, NC>(c, ee, fw, fbit, wd, l1, we);
    lv_add<W, UNIT, PL, U>(wd, l1, we, fbit, cnt, internal);
  }
  lv_decide<W, PL>(c, cnt, internal, from, wv, bo, inst, batched, zero_gain, s_fmask, s_slack, s_bw, s_perf, to,
                   gain, border);
}


// ---- CTA-flat incidence walks
//
// A CTA collects the selected vertices of a range of list positions in shared
// memory (first incidence and degree), scans the degrees, and then spreads
// every incidence of every collected vertex over all its threads: thread t
// takes incidences t, t + blockDim, ... and finds its vertex by binary search
// in the scanned degrees. Hub vertices are split across the whole CTA, and the
// gathers and atomics of different vertices are in flight together.
#ifndef LPGPU_FLAT_THREADS
#define LPGPU_FLAT_THREADS 512
#endif
constexpr int kFlatThreads = LPGPU_FLAT_THREADS;
constexpr int kFlatItems = 1024;  // list positions (and so at most this many vertices) per CTA pass
static_assert(kFlatItems % kFlatThreads == 0, "whole items per thread");

struct FlatSmem {
  int64_t o0[kFlatItems];    // first incidence
  int pre[kFlatItems + 1];   // degrees, then their exclusive prefix sums
  int ft[kFlatItems];        // local from | local to << 16
  int att[kFlatItems];       // per-vertex sums (attributed delta, or the reverse move's gain)
  int inst[kFlatItems];      // instance (batched)
  int pos[kFlatItems];       // list position
  int wsum[kFlatThreads / 32];
  int n;
};

// Warp-aggregated append to a shared counter; returns each selected lane's slot.
__device__ __forceinline__ int flat_append_to(int* counter, bool sel) {
  const unsigned m = __ballot_sync(FULLMASK, sel);
  if (!m) return -1;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane_id() == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(FULLMASK, base, leader);
  return sel ? base + __popc(m & lanemask_lt()) : -1;
}

// Appends the lanes with `sel` to the CTA's item list; returns each lane's slot.
__device__ __forceinline__ int flat_append(FlatSmem& f, bool sel) { return flat_append_to(&f.n, sel); }

// In-place exclusive scan of f.pre[0 .. n) (n <= kFlatItems); f.pre[n] = total.
__device__ __forceinline__ int flat_scan(FlatSmem& f, int n) {
  constexpr int PER = kFlatItems / kFlatThreads;
  const int t = threadIdx.x, lane = lane_id(), wid = t >> 5;
  int v[PER], sum = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = t * PER + q;
    v[q] = i < n ? f.pre[i] : 0;
    sum += v[q];
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULLMASK, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) f.wsum[wid] = incl;
  __syncthreads();
  int wbase = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kFlatThreads / 32; ++w) {
    const int x = f.wsum[w];
    if (w < wid) wbase += x;
    total += x;
  }
  int run = wbase + incl - sum;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = t * PER + q;
    if (i < n) f.pre[i] = run;
    run += v[q];
  }
  if (t == 0) f.pre[n] = total;
  __syncthreads();
  return total;
}

// Vertex of flat incidence index x: the largest i with pre[i] <= x.
__device__ __forceinline__ int flat_find(const FlatSmem& f, int n, int x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (f.pre[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Commit of Q incidences (e[q], from f[q], to t[q]; h[q]: present): all 2Q Φ
// atomics are issued before any result is used, then per incidence the
// decrement of Φ(e, f) and increment of Φ(e, t) toggle Λ when Φ(e, f) reaches
// 0 or Φ(e, t) leaves 0, and Λ1 when either passes through 1. The attributed
// delta (km1Delta, hypergraph_common.h:133-140) is -w(e) when Φ(e, f) reaches
// 0 and +w(e) when Φ(e, t) reaches 1; a[q] is each incidence's part.
template <int Q>
__device__ __forceinline__ void commit_group(const RoundCtx& c, const bool (&h)[Q], const int64_t (&e)[Q],
                                             const int (&f)[Q], const int (&t)[Q], int (&a)[Q], int& toggles) {
  const int W = c.W;
  const int64_t k = c.kmax;
  int of[Q], ot[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    of[q] = ot[q] = 0;
    if (h[q]) {
      of[q] = phi_add(c, e[q] * k + f[q], -1);
      ot[q] = phi_add(c, e[q] * k + t[q], 1);
    }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    a[q] = 0;
    if (!h[q]) continue;
    const int we = c.unit_nets ? 1 : c.w_e[e[q]];
    uint32_t* rec = c.conn + e[q] * 2 * W;
    const uint32_t fb = 1u << (f[q] & 31), tb = 1u << (t[q] & 31);
    if (of[q] == 1) { atomicXor(&rec[f[q] >> 5], fb); a[q] -= we; ++toggles; }
    if (of[q] == 1 || of[q] == 2) atomicXor(&rec[W + (f[q] >> 5)], fb);
    if (ot[q] == 0) { atomicXor(&rec[t[q] >> 5], tb); a[q] += we; ++toggles; }
    if (ot[q] == 0 || ot[q] == 1) atomicXor(&rec[W + (t[q] >> 5)], tb);
  }
}

// Incidences a thread of the CTA-flat commit handles per step.
#ifndef LPGPU_COMMIT_GROUP
#define LPGPU_COMMIT_GROUP 2  // 4 and 8 measured slower on rownet
#endif

// Moves every incidence of the CTA's collected vertices from their `from` to
// their `to` block (flat over the CTA). Returns this thread's summed delta;
// per-vertex sums go to f.att when `per_item`; *toggles counts this thread's
// Λ bit changes.
template <int Q = LPGPU_COMMIT_GROUP>
__device__ __forceinline__ int64_t flat_commit(const RoundCtx& c, FlatSmem& f, int n, int total, bool per_item,
                                               int64_t* toggles = nullptr) {
  int64_t att = 0;
  int tg = 0;
  for (int x0 = threadIdx.x; x0 < total; x0 += Q * kFlatThreads) {
    bool h[Q];
    int64_t e[Q];
    int fr[Q], to[Q], it[Q], a[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int x = x0 + q * kFlatThreads;
      h[q] = x < total;
      it[q] = h[q] ? flat_find(f, n, x) : 0;
      e[q] = h[q] ? c.inets[f.o0[it[q]] + (x - f.pre[it[q]])] : 0;
      const int ft = h[q] ? f.ft[it[q]] : 0;
      fr[q] = ft & 0xffff;
      to[q] = ft >> 16;
    }
    commit_group<Q>(c, h, e, fr, to, a, tg);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      att += a[q];
      if (per_item && a[q]) atomicAdd(&f.att[it[q]], a[q]);
    }
  }
  if (toggles) *toggles += tg;
  return att;
}

}  // namespace lpgpu
