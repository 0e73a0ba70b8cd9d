// One trajectory per group of lanes (pyst_group.cuh) for a single model:
// runs too small to fill the GPU thread by thread.  Built once per
// (PYST_TAU, PYST_SCORE) flavour.
#include "pyst_group.cuh"
#include "pyst_launch.cuh"

namespace pyst {
// see pyst_k_thread.cu: per-flavour namespace, not an anonymous one
namespace PYST_CAT(group_flavour_, PYST_TAU, PYST_SCORE) {

constexpr bool kTau = (bool)PYST_TAU, kScore = (bool)PYST_SCORE;
#ifndef PYST_GROUP_MINB
#define PYST_GROUP_MINB 4
#endif

template <int R, int FC, int LG>
__global__ void __launch_bounds__(128, PYST_GROUP_MINB)
    k_group(const uint32_t* __restrict__ gblob, int blob_words,
            int64_t n_traj, uint64_t id_base, RunArgs ra, OutBase ob,
            unsigned long long* queue) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* sblob = (uint32_t*)smem;
  uint64_t* bar = (uint64_t*)(smem + (size_t)blob_words * 4);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const bool ok = stage_blob(sblob, gblob, blob_words, bar, 0,
                             ra.stage_polls);
  // first trajectory by group index, later ones from the shared queue
  const int64_t ngroups = (int64_t)gridDim.x * blockDim.x / LG;
  const int64_t u0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LG;
  const bool leader = (threadIdx.x & (LG - 1)) == 0;
  if (!ok) {
    mbar_drain(bar, 0);  // let a late copy land before the block exits
    if (leader)
      for (int64_t u = u0; u < n_traj;
           u = ngroups + (int64_t)atomicAdd(queue, 1ull))
        mark_staging_failure(ob, u);
    return;
  }
  ModelView m;
  m.load(sblob);
  auto next = [&](bool first, bool want) {
    if (first) return u0;
    long long v = 0;
    if (want && leader) v = (long long)atomicAdd(queue, 1ull);
    return ngroups + (int64_t)__shfl_sync(0xffffffffu, v, 0, LG);
  };
  auto out = [&](int64_t u) { return ob.at(0, u, 0, 0, ob.stride, m.R); };
  run_groups<R, FC, LG, kTau, kScore>(m, ra, id_base, n_traj, next, out);
}

template <int R, int FC, int LG>
int launch_one(const uint32_t* d_blob, const HostModelInfo& mi, int64_t n,
               uint64_t id_base, const RunArgs& ra, const OutBase& ob,
               unsigned long long* queue, cudaStream_t st) {
  auto kf = k_group<R, FC, LG>;
  const int bs = 128;
  const size_t smem = (size_t)mi.words * 4 + 16;
  const int rc = set_smem(kf, smem);
  if (rc) return rc;
  if (cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st) !=
      cudaSuccess)
    return PYST_ECUDA;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, bs, smem);
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (n * LG + bs - 1) / bs;
  const int64_t cap = (int64_t)num_sms() * per_sm;
  if (grid > cap) grid = cap;
  kf<<<(unsigned)grid, bs, smem, st>>>(d_blob, mi.words, n, id_base, ra, ob,
                                       queue);
  return cudaGetLastError() == cudaSuccess ? PYST_OK : PYST_ECUDA;
}

// (16 lanes in tau-leaping: models of 9 to 16 species only.  Six factor slots:
// models of four to six factors, 32 trajectories per SM, 6 reactions: 0.44 ms
// against 1.22 for a thread each, tau-leaping 0.63 against 2.12.)
template <int R, int FC>
int launch_lanes(int lanes, const uint32_t* d_blob, const HostModelInfo& mi,
                 int64_t n, uint64_t id_base, const RunArgs& ra,
                 const OutBase& ob, unsigned long long* queue,
                 cudaStream_t st) {
  if constexpr (R <= 4)
    if (lanes == 4)
      return launch_one<R, FC, 4>(d_blob, mi, n, id_base, ra, ob, queue, st);
  if (lanes == 8)
    return launch_one<R, FC, 8>(d_blob, mi, n, id_base, ra, ob, queue, st);
  if (lanes == 16)
    return launch_one<R, FC, 16>(d_blob, mi, n, id_base, ra, ob, queue, st);
  return launch_one<R, FC, 32>(d_blob, mi, n, id_base, ra, ob, queue, st);
}

}  // namespace (flavour)
using namespace PYST_CAT(group_flavour_, PYST_TAU, PYST_SCORE);

int PYST_CAT(launch_group_, PYST_TAU, PYST_SCORE)(
    int lanes, const uint32_t* d_blob, const HostModelInfo& mi, int64_t n,
    uint64_t id_base, const RunArgs& ra, const OutBase& ob,
    unsigned long long* queue, cudaStream_t st) {
  if (n <= 0) return PYST_OK;
#define PYST_GO(r, fc) \
  return launch_lanes<r, fc>(lanes, d_blob, mi, n, id_base, ra, ob, queue, st)
#define PYST_GO_R(r)                  \
  do {                                \
    if (mi.factors == 1) PYST_GO(r, 1); \
    if (mi.factors == 2) PYST_GO(r, 2); \
    if (mi.factors == 3) PYST_GO(r, 3); \
    PYST_GO(r, 6);                    \
  } while (0)
  if (mi.R <= 3) PYST_GO_R(3);
  if (mi.R <= 4) PYST_GO_R(4);
  if (mi.R <= 6) PYST_GO_R(6);
  PYST_GO_R(8);
#undef PYST_GO_R
#undef PYST_GO
}

}  // namespace pyst
