// Launch rules of the team rounds (team_kernel.cuh).
#include <algorithm>

#include "team_kernel.cuh"

namespace lpgpu {

// One file per Λ word count (team_w*.cu), compiled in parallel.
const void* team_kernel_w1(bool unit, int unroll, int minb);
const void* team_kernel_w2(bool unit, int unroll, int minb);
const void* team_kernel_w4(bool unit, int unroll, int minb);
const void* team_kernel_w8(bool unit, int unroll, int minb);
const void* team_kernel_w16(bool unit, int unroll, int minb);
const void* team_kernel_w32(bool unit, int unroll, int minb);

static const void* team_kernel_for(int W, bool unit, int unroll, int minb) {
  switch (W) {
    case 1: return team_kernel_w1(unit, unroll, minb);
    case 2: return team_kernel_w2(unit, unroll, minb);
    case 4: return team_kernel_w4(unit, unroll, minb);
    case 8: return team_kernel_w8(unit, unroll, minb);
    case 16: return team_kernel_w16(unit, unroll, minb);
    default: return team_kernel_w32(unit, unroll, minb);
  }
}

// Shared memory of a launch without the CTA's part of the instance (own: the
// build can hold it).
static size_t team_smem_base(int W, bool own) {
  switch (W) {
    case 1:
    case 2:
    case 4: return own ? kTeamOwnAt<128> : kTeamSharedAt + offsetof(TeamShared<128>, crec);
    case 8: return kTeamOwnAt<256>;
    case 16: return kTeamOwnAt<512>;
    default: return kTeamOwnAt<1024>;
  }
}

// k > 128 has the 1-CTA-per-SM build only (its per-block tables).
static int team_min_blocks(int W, int ctas_per_sm) { return W > 4 || ctas_per_sm < 2 ? 1 : 2; }

static int team_occupancy(const void* kern, int minb, size_t smem) {
  allow_dyn_smem_of(kern, smem);
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, kTeamThreads, smem) != cudaSuccess) return 1;
  return std::max(1, std::min(blocks, minb));
}

// Shared memory for a CTA's part of the instance. A team of several CTAs leaves
// half of the SM's memory to the L1 cache, which holds the record gathers in
// flight (400K vertices with 170 KB of parts: 3,030 -> 3,690 us).
static int64_t team_own_most(int minb, int T, int W) {
  return minb >= 2 ? 0 : (T == 1 ? 224 : W > 4 ? 160 : 128) * 1024 - (int64_t)team_smem_base(W, true);
}

// Shared memory of a launch: what a CTA's part of the instance wants with a
// quarter to spare (the CTAs' shares differ), if an SM holds it; a part that
// does not fit stays in global memory and leaves the SM's memory to the L1
// cache.
static size_t team_smem_bytes(int minb, int T, int W, int64_t own_bytes) {
  const size_t base = team_smem_base(W, minb < 2);
  const int64_t most = team_own_most(minb, T, W);
  if (own_bytes <= 0 || own_bytes > most) return base;
  return base + (size_t)std::min(most, own_bytes + own_bytes / 4 + 1024);
}

int64_t team_own_bytes(int64_t n, int64_t m, int64_t pins, int T, int k, int W, bool phi16, int per_sm) {
  const int64_t own = 4 * (pins / T) + 16 * (n / T + 32);
  if (T > 1) return own;
  const int64_t nets = own + 16 + 8 * m * W, all = nets + (phi16 ? 2 : 4) * m * k;
  const int64_t most = team_own_most(team_min_blocks(W, per_sm), T, W);
  return all <= most ? all : nets <= most ? nets : own;
}

int team_slots(const Launch& L, int64_t count, int T) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(count, 2 * (int64_t)L.num_sms / T));
}

int team_resident(const Launch& L, int W, bool unit, int unroll, int ctas_per_sm) {
  const int minb = team_min_blocks(W, ctas_per_sm);
  return L.num_sms * team_occupancy(team_kernel_for(W, unit, unroll, minb), minb,
                                       team_smem_base(W, minb < 2));
}

// Active vertices of every instance's last persistent round (its round's
// statistics), for the host's stop rule.
__global__ void k_px_active(const PxInst* __restrict__ insts, int32_t count, int64_t* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const PxInst& I = insts[i];
    out[i] = I.stats[(int64_t)I.round * kStats + kStActive];
  }
}

cudaError_t launch_px_active(const Launch& L, const PxInst* insts, int32_t count, int64_t* out) {
  if (count <= 0) return cudaSuccess;
  k_px_active<<<(count + 255) / 256, 256, 0, L.st>>>(insts, count, out);
  return launched("k_px_active");
}

// One launch of the kernel: build, shared memory, how its teams meet.
namespace {
struct TeamLaunch {
  const void* kern;
  size_t smem, base;
  int resident;  // CTAs of the build that the GPU holds
  TeamSync sync;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  TeamLaunch(const Launch& L, int T, int W, bool unit, int unroll, int ctas_per_sm, int64_t own_bytes) {
    const int minb = team_min_blocks(W, ctas_per_sm);
    kern = team_kernel_for(W, unit, unroll, minb);
    smem = team_smem_bytes(minb, T, W, own_bytes);
    base = team_smem_base(W, minb < 2);
    resident = L.num_sms * team_occupancy(kern, minb, smem);
    sync = T == 1 ? kSyncCta : T > kTeamMaxCluster ? kSyncGrid : kSyncCluster;
    cfg.gridDim = dim3((unsigned)T);
    cfg.blockDim = dim3(kTeamThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = L.st;
  }
  // Attributes of the launch, once the object has its place.
  cudaError_t attributes(int T) {
    if (sync == kSyncCta) return cudaSuccess;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (sync == kSyncGrid) {
      at.id = cudaLaunchAttributeCooperative;
      at.val.cooperative = 1;
      return cudaSuccess;
    }
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)T;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    return T > 8 ? cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
  }
};
}  // namespace

// Most CTAs a team may have; a smaller limit stands in for a GPU partition.
#ifndef LPGPU_TEAM_MOST
#define LPGPU_TEAM_MOST (1 << 20)
#endif

bool team_fits(const Launch& L, int T, int W, bool unit, int unroll, int ctas_per_sm, int64_t own_bytes) {
  if (T <= 1) return true;
  if (T > LPGPU_TEAM_MOST) return false;
  TeamLaunch t(L, T, W, unit, unroll, ctas_per_sm, own_bytes);
  if (t.sync == kSyncGrid) return T <= t.resident;
  int clusters = 0;
  if (t.attributes(T) != cudaSuccess || cudaOccupancyMaxActiveClusters(&clusters, t.kern, &t.cfg) != cudaSuccess) {
    cudaGetLastError();  // no cluster of this size: the answer, not a failure
    return false;
  }
  return clusters > 0;
}

cudaError_t launch_px_round(const Launch& L, const PxInst* insts, const int32_t* order, int32_t count, PxParams P,
                            int W, bool unit, int ctas_per_sm, int teams, int64_t* scratch, int64_t* queue,
                            int64_t* err, int64_t own_bytes, bool cleared) {
  if (count <= 0 || P.rounds <= 0) return cudaSuccess;
  if (W < 1 || W > 32 || (W & (W - 1)) || P.T < 1 || P.kcap > kTeamMaxK) return cudaErrorInvalidValue;
  const bool grid = P.T > kTeamMaxCluster;
  if (grid && (count != 1 || teams != 1)) return cudaErrorInvalidValue;
  cudaError_t e = cleared ? cudaSuccess : cudaMemsetAsync(queue, 0, sizeof(int64_t), L.st);
  if (e != cudaSuccess) return e;
  if (P.T > 1) {
    if (!scratch) return cudaErrorInvalidValue;
    if (!cleared) e = cudaMemsetAsync(scratch, 0, sizeof(int64_t) * teams * team_scratch_words(P.kcap), L.st);
    if (e != cudaSuccess) return e;
  } else {
    scratch = nullptr;
  }
  TeamLaunch t(L, P.T, W, unit, P.unroll, ctas_per_sm, own_bytes);
  P.resident = (int32_t)(t.smem - t.base);
  if (grid && P.T > t.resident) return cudaErrorCooperativeLaunchTooLarge;
  teams = std::max(1, std::min(teams, std::min<int>(count, std::max(1, t.resident / P.T))));
  t.cfg.gridDim = dim3((unsigned)(teams * P.T));
  if ((e = t.attributes(P.T)) != cudaSuccess) return e;
  int sync = t.sync;
  void* args[] = {(void*)&insts, (void*)&order, (void*)&count, (void*)&P, (void*)&sync, (void*)&scratch,
                  (void*)&queue, (void*)&err};
  e = cudaLaunchKernelExC(&t.cfg, t.kern, args);
  if (e != cudaSuccess) {
    set_error(std::string("k_team: ") + cudaGetErrorString(e));
    return e;
  }
  return launched("k_team");
}

}  // namespace lpgpu
