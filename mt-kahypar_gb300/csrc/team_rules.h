// How many CTAs refine an instance (team rounds, team_kernel.cuh), and where the
// multi-launch pipeline is the better form: plain host arithmetic, no CUDA.
#pragma once

#include <stdint.h>

namespace lpgpu {

// CTAs per team of a launch over one instance (1: a CTA; up to kTeamMaxCluster:
// a thread-block cluster; more: the whole cooperative grid).
constexpr int kTeamMaxCluster = 16;

struct TeamShape {
  int per_sm;  // kernel build: resident CTAs per SM
  int unroll;
  int T;       // CTAs of the team; kTeamAll: as many as are resident; kTeamNone: the pipeline
};
constexpr int kTeamAll = 0, kTeamNone = -1;

// One instance of n vertices and `pins` pins. Few vertices can carry any number
// of pins (coarse levels, dense hypergraphs), so both count. Measured (GB300,
// whole refine in us, one CTA / cluster of 16 / one CTA per SM / two per SM;
// multi-launch pipeline in brackets).
// About five pins per vertex: 1,024 vertices (k = 2) 467 / 556 / - / - [1,094];
// 2,048 (k = 4) 608 / 617 / - / -; 4,096 (k = 2) 976 / 681 / - / -; 10,007 (k = 8)
// 1,634 / 797 / 888 / -; 16,384 (k = 64, weighted) 5,508 / 1,852 / 1,660 / -
// [2,917]; 65,536 (k = 32) - / 2,678 / 1,703 / 2,015; 262,144 (k = 16) - / 5,877 /
// 2,184 / 2,242 [3,203]; 524,288 (k = 32) - / 11,319 / 2,924 / 2,887, unweighted k
// = 8 1,777 / 1,903; 1M (k = 32) - / - / 5,195 / 4,641 [5,563]; 4.2M (k = 128) - /
// - / 12,145 / 11,015 [11,371].
// More pins (k = 32, weighted): 1,024 vertices, 16,357 pins 610 / 661 / 796 / -
// [1,314], 30,673 1,231 / 763 / 920 / - [1,833]; 2,048 and 12,279 648 / 676 / 735 /
// - [1,287], 20,460 785 / 673 / 783 / - [1,366], 204,633 4,426 / 1,259 / 1,156 / -
// [3,226], 4.1M 35,617 / 7,390 / 4,362 / - [5,419]; 8,192 and 131,046 3,112 / 991 /
// 968 / - [2,188]; 12,288 and 368,579 9,505 / 1,681 / 1,179 / - [3,300], 11.0M
// 144,494 / 15,743 / 6,794 / - [9,912].
// A team deals out whole vertices, 32 at a time, and the pipeline the incidences
// of all of them: with thousands of pins per vertex on few vertices it wins (256
// vertices, 0.76M pins 8,554 / 4,979 / 4,939 / - [5,398], 14.5M 115,542 / 65,058 /
// 64,541 / - [61,421], k = 2 22,972 / 17,365 / 17,107 / - [7,787]; 1,024 and 3.1M
// 30,016 / 8,592 / 6,859 / - [6,543], 20.2M 205,846 / 54,539 / 43,137 / -
// [35,790]), except where one or two CTAs hold them all (64 vertices, 3.8M
// 45,912 / 26,496 / 25,476 / - [57,563]).
inline TeamShape team_shape(int64_t n, int64_t pins) {
  if (n <= 2048 && pins + 4 * n <= 24576) return {1, 4, 1};
  if (n <= 12288 && pins <= 131072) return {1, 4, kTeamMaxCluster};
  if (n > 128 && pins > 4096 * n) return {1, 4, kTeamNone};
  return {n < 655360 ? 1 : 2, 4, kTeamAll};
}

// The same on a device with `all` refines in progress (this one included), `grids` of
// which want the whole grid. A cooperative grid on every SM keeps the others out until
// it ends: beside one of 131,071 vertices (k = 64) a 1,024-vertex refine takes 2,347
// instead of 430 us, a pipeline 50 ms, and the grid gains nothing (2,347 us).
// - One grid beside other refines leaves them room: with two CTAs per SM half of the
//   GPU, a third of the CTAs from three refines on (us, the grid / the others. 131,071
//   vertices and a small one: half 2,231 / 478, a third 2,248 / 487, a quarter 2,395 /
//   472; and three clusters: 2,410 / 815, 2,272 / 820, 2,426 / 794; 1M and three small
//   ones: 6,105 / 451, 6,313 / 447, 7,574 / 441). For k > 128 an SM holds one CTA:
//   three quarters of the SMs, then two thirds (131,071 vertices in that build: 2,049 /
//   480 and one cluster 2,026 / 794).
// - Several grids take equal shares, of whole SMs up to 200,000 vertices and for 33 to
//   64 blocks, of CTAs two to an SM above (us per refine, 2 / 4 / 8 threads, whole SMs |
//   two CTAs per SM [pipeline]): 16,384 vertices 405 / 220 / 127 | 472 / 252 / 139 [780 /
//   410 / 223]; 131,071, k = 64 1,177 / 841 / 617 | 1,317..1,811 / 991 / 681 [1,904 / 1,146 /
//   784]; 400,003, k = 64 2,054 / 1,666 / 1,512 | 1,969 / 1,791 / 1,578 [2,434 / 1,679 /
//   1,465]; 262,144, k = 16 1,376 / 1,022 / 824 | 1,252 / 885 / 684 [1,947 / 1,206 / 897];
//   524,288, k = 8 1,178 / 897 / 766 | 1,076 / 737 / 592 [1,419 / 896 / 720]; 250,007, k =
//   300 1,407 / 1,041 / 847 | - [2,365 / 1,721 / 1,558].
// - The pipeline serves several large ones as well or better, from 589,824 vertices on
//   (600,011 2,410 / 1,953 / 1,852 | 2,153..2,937 / 1,878 / 1,706 [2,550 / 1,813 / 1,660]; 1M
//   4,171 / 3,764 / 3,853 | 3,905 / 3,214 / 3,314 [3,879 / 3,131 / 3,045]), and three from
//   393,216 on for more than 32 blocks (500,000, k = 128: 1,277 / 1,217 / 994 [1,591 / 1,096 /
//   995]).
inline TeamShape shared_team_shape(int64_t n, int64_t pins, int k, int num_sms, int grids, int all) {
  TeamShape t = team_shape(n, pins);
  if (t.T != kTeamAll || all <= 1) return t;
  if (grids > 1 && k <= 128 && (n >= 589824 || (grids > 2 && n >= 393216 && k > 32)))
    return {t.per_sm, t.unroll, kTeamNone};
  if (grids <= 1) {
    t.per_sm = k > 128 ? 1 : 2;
    t.T = k > 128 ? (all == 2 ? 3 * num_sms / 4 : 2 * num_sms / 3) : 2 * num_sms / (all < 3 ? all : 3);
  } else {
    t.per_sm = k <= 128 && n >= 200000 && (k <= 32 || k > 64) ? 2 : 1;
    t.T = t.per_sm * num_sms / (all < 8 ? all : 8);
  }
  if (t.T <= kTeamMaxCluster) t.T = kTeamMaxCluster + 1;
  return t;
}

// Several instances, the largest of max_n vertices and of max_pins pins: CTAs per
// team, with about `per_sm` CTAs' worth of teams per SM at most (stepped rounds, which
// leave room for other sessions' work, ask for 2; a batch for 5, of which two are
// resident at once). Larger teams finish the largest instance sooner, more of them
// keep the SMs busy. Whole refine, T = 1 / 2 / 4 / 8 / 16 (GB300, ms): 1,280 instances
// of up to 65,536 vertices 16.1 / 20.2 / 27.3 / 42.1 / 87.9 (multi-launch pipeline
// 33.8); 320: 11.3 / 6.9 / 7.2 / 10.7 / 22.3 (9.0); 80: 9.3 / 5.5 / 3.5 / 3.2 / 5.9
// (3.9); 24: 8.9 / 5.2 / 3.1 / 2.0 / 2.2 (2.6); 1,280 of up to 4,096: 4.0 / 7.9 / 14.4
// / 27.9 / 68.1 (7.9).
// One CTA serves what it serves alone (team_shape). Few vertices with many pins take
// teams that are all resident: 37 of 2,048 vertices and 61,384 pins 1.89 / 1.54 / 1.39
// / 2.03 / 3.04 (4.5), 204,633 pins 5.1 / 3.1 / 2.1 / 2.5 / 3.4 (8.4).
inline int team_of_many(int64_t count, int64_t max_n, int64_t max_pins, int64_t num_sms, int per_sm) {
  if (max_n <= 2048) {
    if (max_pins + 4 * max_n <= 24576) return 1;
    per_sm = 1;
  }
  int T = 1;
  while (T < 8 && count * 2 * T <= per_sm * num_sms) T *= 2;
  return T;
}

// The team of a batch of several instances. Clusters of 16 where every one of them
// finds its SMs and the instances are large (us, clusters of 8 / 16): 2 of 16,384
// vertices 1,037 / 931, 2 of 65,536 1,890 / 1,350, 8 of 65,536 k = 2 / 8 / 64 1,779 /
// 1,570, 1,939 / 1,717, 2,640 / 2,362, but 8 of 4,096 831 / 870; for k > 128 an SM holds
// one CTA, and 8 of 16,384 and k = 300 take 1,919 / 2,797.
inline int team_of_batch(int64_t count, int64_t max_n, int64_t max_pins, int64_t num_sms, int kmax) {
  const int T = team_of_many(count, max_n, max_pins, num_sms, 5);
  return T == 8 && kmax <= 128 && max_pins > 65536 && count * 16 <= num_sms ? kTeamMaxCluster : T;
}

// A team's time is about 33 ns per pin of its instance and CTA. Where the largest
// instance so outlasts the whole pipeline (its 1.1 ms of extra launches and 0.6 ns per
// pin of the batch), the pipeline refines the batch. Pipeline / teams, us: 2 of 262,144
// vertices and 5 pins each 3,012 / 5,467, 4 4,123 / 3,390 (16 CTAs), 8 7,270 / 6,205; 2
// of 1M 9,190 / 21,508, 4 15,487 / 12,798 (16), 8 33,278 / 26,758; one of 65,536 beside 20
// of 1,024 1,978 / 1,835, one of 262,144 2,338 / 5,414, one of 1M 4,887 / 20,318, beside
// 200 5,785 / 77,412 (one CTA each).
inline bool batch_wants_pipeline(int64_t max_pins, int64_t sum_pins, int T) {
  return max_pins / T > 34000 + sum_pins / 55;
}

}  // namespace lpgpu
