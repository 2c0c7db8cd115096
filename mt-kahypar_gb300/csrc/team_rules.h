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

}  // namespace lpgpu
