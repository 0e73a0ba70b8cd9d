// Batched persistent kernel: many models of uneven size in one launch.
// Blocks take work items (one model, its trajectories and output offsets)
// from a device queue (an atomic counter in caller workspace), stage the
// item's model blob into shared memory with one bulk-async copy, and run its
// trajectories thread-per-trajectory or warp-per-trajectory as the item
// says (PYST_GROUPS: for batches too small to fill the GPU thread by thread,
// a group of lanes per trajectory where the item's model allows it).
// Replaces the reference's one-JIT-and-launch-sequence-per-model sweep
// (examples/*_sim.py loops over CuTauLeaping().run, e.g.
// examples/schlogl_sim.py:66-80).  Built once per (PYST_GROUPS, PYST_SCORE)
// flavour.
#include "pyst_group.cuh"
#include "pyst_launch.cuh"

// Blocks of 128 threads per SM the register allocation must allow: 6 (at most
// 80 registers) measured 11% faster than no bound on the Schlogl /
// Lotka-Volterra sweep (2,048 models, scores, statistics) and 1.5% slower on
// synthetic networks of up to 256 reactions, with every form inlined; with
// the tau-leaping forms out of line scored batches take 5 (at most 96: 40
// models of 10 to 24 reactions x 250 trajectories, tau-leaping 26.9 -> 19.4
// ms, direct method 20.0 -> 18.2; the sweep 719 -> 712).
#ifndef PYST_BATCH_MINB
#if PYST_GROUPS
#define PYST_BATCH_MINB 4  // as k_group
#else
#define PYST_BATCH_MINB (PYST_SCORE ? 5 : 6)
#endif
#endif
#if PYST_BATCH_MINB > 0
#define PYST_BATCH_BOUNDS __launch_bounds__(128, PYST_BATCH_MINB)
#else
#define PYST_BATCH_BOUNDS __launch_bounds__(128)
#endif

namespace pyst {
// nvcc gives template functions of an anonymous namespace weak external
// linkage on the host side, so the flavours built from this file would be
// merged at link time; a per-flavour namespace keeps them apart.
namespace PYST_CAT(batch_flavour_, PYST_GROUPS, PYST_SCORE) {

// Summary statistics and score Jacobians of one finished model (U
// trajectories), computed by the block that ran it -- or, for a model split
// into chunks, ran its last chunk -- from the samples (and scores) written
// for it, sums over trajectories in trajectory order.  Loads bypass L1
// (other blocks wrote part of the data).  Means and variances go to shared
// scratch `ms` when 2*kappa*ita doubles fit, else they are recomputed.
__device__ void item_epilogue(const ModelView& m, const pyst_batch_item& item,
                              int64_t U, const OutBase& ob, double* ms,
                              int ms_bytes) {
  const int ita = m.ita, KF = m.kappa * m.ita, R = m.R;
  if (U <= 0) return;
  const int32_t* smp = ob.samples + item.sample_offset;
  const double dU = (double)U;
  const bool keep = (size_t)KF * 16 <= (size_t)ms_bytes;
  auto row_moments = [&](int kf, double& mean, double& var) {
    const int32_t* row = smp + (int64_t)kf * U;
    double s = 0.0, s2 = 0.0;
    for (int64_t u = 0; u < U; ++u) {
      const double x = (double)__ldcg(row + u);
      s = __dadd_rn(s, x);
      s2 = __dadd_rn(s2, __dmul_rn(x, x));
    }
    mean = __ddiv_rn(s, dU);
    var = __dsub_rn(__ddiv_rn(s2, dU), __dmul_rn(mean, mean));
  };
  for (int kf = threadIdx.x; kf < KF; kf += blockDim.x) {
    double mean, var;
    row_moments(kf, mean, var);
    if (keep) {
      ms[2 * kf] = mean;
      ms[2 * kf + 1] = var;
    }
    if (ob.stats) {
      double corr = 0.0;
      const int f = kf % ita;
      if (f + 1 < ita) {
        double mb, vb;
        row_moments(kf + 1, mb, vb);
        const int32_t* ra_ = smp + (int64_t)kf * U;
        const int32_t* rb = ra_ + U;
        double sab = 0.0;
        for (int64_t u = 0; u < U; ++u)
          sab = __dadd_rn(sab, __dmul_rn((double)__ldcg(ra_ + u),
                                         (double)__ldcg(rb + u)));
        const double cov = __dsub_rn(__ddiv_rn(sab, dU), __dmul_rn(mean, mb));
        const double den = __dmul_rn(var, vb);
        if (den > 0.0) corr = __ddiv_rn(cov, __dsqrt_rn(den));
      }
      double* o = ob.stats + item.stats_offset + (int64_t)kf * 3;
      o[0] = mean;
      o[1] = var;
      o[2] = corr;
    }
  }
  if (!ob.jac || !ob.score) return;
  __syncthreads();
  const double* sc = ob.score + item.score_offset;
  for (int idx = threadIdx.x; idx < KF * R; idx += blockDim.x) {
    const int kf = idx / R, j = idx - kf * R;
    double mean, var;
    if (keep) {
      mean = ms[2 * kf];
      var = ms[2 * kf + 1];
    } else {
      row_moments(kf, mean, var);
    }
    const int32_t* row = smp + (int64_t)kf * U;
    double gm = 0.0, gv = 0.0;
    for (int64_t u = 0; u < U; ++u) {
      const double d = __dsub_rn((double)__ldcg(row + u), mean);
      const double s = __ldcg(sc + u * R + j);
      gm = __dadd_rn(gm, __dmul_rn(d, s));
      gv = __dadd_rn(gv, __dmul_rn(__dsub_rn(__dmul_rn(d, d), var), s));
    }
    double* o = ob.jac + item.jac_offset;
    o[(int64_t)kf * R + j] = __ddiv_rn(gm, dU);
    o[((int64_t)KF + kf) * R + j] = __ddiv_rn(gv, dU);
  }
}

#if !PYST_GROUPS
// One trajectory of an item with direct forms.  The tau-leaping forms are
// functions of their own (arguments by value: the model view stays in
// registers): inlined into this large kernel their spills depended on what
// else was in it (2,048 sweep sets x 256 trajectories, ms, inlined and out of
// line: 809 and 615, with scores 747 and 712; the direct method with scores
// loses, 600 telegraph and 600 Schlogl models of 256 14 and 22).
template <int R, bool TAU, bool SCORE>
__device__ __noinline__ void run_exact_call(ModelView m, int32_t* xcol,
                                            int64_t* slot, int bs, RunArgs ra,
                                            uint64_t id, TrajOut o) {
  run_thread<R, TAU, SCORE, kPkPacked, R, 3>(m, xcol, slot, bs, ra, id, o);
}
template <int R, bool TAU, bool SCORE>
__device__ __forceinline__ void run_exact(const ModelView& m, int32_t* xcol,
                                          int64_t* slot, int bs,
                                          const RunArgs& ra, uint64_t id,
                                          const TrajOut& o) {
  if constexpr (TAU)
    run_exact_call<R, TAU, SCORE>(m, xcol, slot, bs, ra, id, o);
  else
    run_thread<R, TAU, SCORE, kPkPacked, R, 3>(m, xcol, slot, bs, ra, id, o);
}
#endif

template <bool SCORE>
__global__ void PYST_BATCH_BOUNDS
    k_batch(const uint32_t* __restrict__ gblobs,
            const pyst_batch_item* __restrict__ items, int64_t n_items,
            RunArgs ra, OutBase ob, unsigned long long* queue, unsigned* done,
            int max_blob_words, int warp_bytes, int dyn_bytes, int pk_bytes,
            int fd_bytes, int wide_cap) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long s_item;
  __shared__ int s_last;
#if PYST_GROUPS
  __shared__ int s_next;
#endif
  uint32_t* sblob = (uint32_t*)smem;
  uint64_t* bar = (uint64_t*)(smem + (size_t)max_blob_words * 4);
  // packed reaction descriptors of the current item (thread mapping)
  uint32_t* spk = (uint32_t*)(smem + (size_t)max_blob_words * 4 + 16);
  // and its direct forms (fd_bytes 0: the launch has no room for them)
  uint4* sfd = (uint4*)((unsigned char*)spk + pk_bytes);
  // reaction words of large networks (wide_cap 0: no room for them)
  uint4* sfw = (uint4*)((unsigned char*)sfd + fd_bytes);
  unsigned char* dyn = (unsigned char*)sfw + wide_bytes(wide_cap);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const int bs = blockDim.x, nw = bs >> 5, wid = threadIdx.x >> 5;
  uint32_t parity = 0;
  while (true) {
    if (threadIdx.x == 0) s_item = (long long)atomicAdd(queue, 1ull);
    __syncthreads();
    const long long it = s_item;
    if (it >= n_items) break;
    const pyst_batch_item item = items[it];
    // the model's trajectory count (a split model's chunks share it) and
    // this item's first trajectory in it
    const int64_t U = item.model_n_traj > 0 ? item.model_n_traj : item.n_traj;
    const int64_t cb = item.model_n_traj > 0 ? item.chunk_begin : 0;
    const uint32_t* blob = gblobs + item.blob_offset;
    const int words = (int)__ldg(blob + PYST_H_WORDS);
    const bool ok = stage_blob(sblob, blob, words, bar, parity,
                               ra.stage_polls);
    if (!ok) {
      mbar_drain(bar, parity);
      for (int64_t v = threadIdx.x; v < item.n_traj; v += bs)
        mark_staging_failure(ob, item.traj_offset + cb + v);
      break;
    }
    parity ^= 1u;
    ModelView m;
    m.load(sblob);
    if (SCORE && ob.score && m.nlaw > 0) {
      // (block-uniform) scores need a_j proportional to rate_j (mass
      // action): the item is not simulated; its samples read -1 and its
      // scores NaN
      const int KF = m.kappa * m.ita;
      const double nan = __longlong_as_double(0x7ff8000000000000ll);
      for (int64_t v = threadIdx.x; v < item.n_traj; v += bs) {
        const TrajOut o = ob.at(item.sample_offset, cb + v, item.traj_offset,
                                item.score_offset, U, m.R);
        for (int kf = 0; kf < KF; ++kf) o.samples[(int64_t)kf * o.stride] = -1;
        if (o.status) *o.status = (uint8_t)PYST_TRAJ_UNSUPPORTED;
        if (o.events) *o.events = 0;
        if (o.seqhash) *o.seqhash = 0;
        if (o.t_final) *o.t_final = 0.0;
        for (int j = 0; j < m.R; ++j) o.score[j] = nan;
      }
    } else {
      if (item.mapping == PYST_MAP_THREAD &&
          packed_bytes(m.R) <= (size_t)pk_bytes) {
        // (uniform over the block: every thread reads the same item)
        m.pk = spk;
#if !PYST_GROUPS
        if (fd_bytes && m.nlaw == 0 &&
            has_direct_forms(m.R, blob_direct_factors(sblob))) {
          m.fd = sfd;
          build_direct(m, sfd, bs);
        }
#endif
        m.fast = __syncthreads_and(pack_reactions(m, spk)) != 0;
      }
      // (uniform: items beyond the register arrays, or warp-mapped)
      if (m.nlaw == 0 && m.R <= wide_cap &&
          (item.mapping != PYST_MAP_THREAD ||
           m.R > PYST_THREAD_MAX_REACTIONS))
        if (__syncthreads_and(build_wide(m, sfw))) m.fw = sfw;
      const bool tau = item.method == PYST_METHOD_TAU_LEAP;
#if PYST_GROUPS
      // (block-uniform)
      const int lanes =
          item.mapping == PYST_MAP_THREAD && m.nlaw == 0 && m.fast
              ? batch_lanes(blob_direct_factors(sblob), m.S, m.R) : 0;
      if (lanes) {
        auto out = [&](int64_t u) {
          return ob.at(item.sample_offset, u, item.traj_offset,
                       item.score_offset, U, m.R);
        };
        // trajectories of the item in order, to the groups as they ask
        if (threadIdx.x == 0) s_next = 0;
        __syncthreads();
        auto next = [&](bool first, bool want) {
          (void)first;
          const int lg = lanes;
          int v = 0;
          if (want && (threadIdx.x & (lg - 1)) == 0)
            v = atomicAdd(&s_next, 1);
          v = __shfl_sync(0xffffffffu, v, 0, lg);
          return v < item.n_traj ? cb + v : cb + item.n_traj;
        };
        const uint64_t idb = (uint64_t)item.traj_id_base;
        const int64_t end = cb + item.n_traj;
        if (lanes == 4) {
          if (tau)
            run_groups<4, 3, 4, true, SCORE>(m, ra, idb, end, next, out);
          else
            run_groups<4, 3, 4, false, SCORE>(m, ra, idb, end, next, out);
        } else {
          if (tau)
            run_groups<8, 3, 8, true, SCORE>(m, ra, idb, end, next, out);
          else
            run_groups<8, 3, 8, false, SCORE>(m, ra, idb, end, next, out);
        }
      } else
#endif
      if (item.mapping == PYST_MAP_THREAD) {
        int32_t* xcol = (int32_t*)dyn + threadIdx.x;
        const bool direct = !PYST_GROUPS && m.fast && m.fd != nullptr;
        int64_t* slot =
            (int64_t*)((int32_t*)dyn + (size_t)(m.S + (direct ? 1 : 0)) * bs) +
            threadIdx.x;
        for (int64_t v = threadIdx.x; v < item.n_traj; v += bs) {
          const int64_t u = cb + v;
          const TrajOut o = ob.at(item.sample_offset, u, item.traj_offset,
                                  item.score_offset, U, m.R);
          const uint64_t id = (uint64_t)item.traj_id_base + (uint64_t)u;
          if (direct) {
            // (block-uniform) an item with direct forms: the reaction count
            // (2 to 8) fixed at compile time, three factor slots (one form
            // for all items keeps the kernel's size)
#if !PYST_GROUPS
            switch (m.R) {
#define PYST_EXACT_CASE(r)                                                 \
  case r:                                                                  \
    if (tau)                                                               \
      run_exact<r, true, SCORE>(m, xcol, slot, bs, ra, id, o);             \
    else                                                                   \
      run_exact<r, false, SCORE>(m, xcol, slot, bs, ra, id, o);            \
    break;
              PYST_EXACT_CASE(2)
              PYST_EXACT_CASE(3)
              PYST_EXACT_CASE(4)
              PYST_EXACT_CASE(5)
              PYST_EXACT_CASE(6)
              PYST_EXACT_CASE(7)
              PYST_EXACT_CASE(8)
#undef PYST_EXACT_CASE
            }
#endif
          } else if (m.R <= 8) {
            if (tau) run_thread<8, true, SCORE>(m, xcol, slot, bs, ra, id, o);
            else run_thread<8, false, SCORE>(m, xcol, slot, bs, ra, id, o);
          } else if (SCORE || m.R <= PYST_THREAD_MAX_REACTIONS) {
            // (the host maps scored items with more reactions to warps)
            if (tau) run_thread<32, true, SCORE>(m, xcol, slot, bs, ra, id, o);
            else run_thread<32, false, SCORE>(m, xcol, slot, bs, ra, id, o);
          } else {
            if (tau) run_thread_big<true>(m, xcol, slot, bs, ra, id, o);
            else run_thread_big<false>(m, xcol, slot, bs, ra, id, o);
          }
        }
      } else {
        unsigned char* mine = dyn + (size_t)wid * warp_bytes;
        const WarpSmem ws = warp_smem(mine, m.S, m.R);
        double* sacc = (double*)(mine + warp_smem_bytes(m.S, m.R));
        for (int64_t v = wid; v < item.n_traj; v += nw) {
          const int64_t u = cb + v;
          const TrajOut o = ob.at(item.sample_offset, u, item.traj_offset,
                                  item.score_offset, U, m.R);
          const uint64_t id = (uint64_t)item.traj_id_base + (uint64_t)u;
          if (tau) run_warp<true, SCORE>(m, ws, ra, id, o, sacc);
          else run_warp<false, SCORE>(m, ws, ra, id, o, sacc);
        }
      }
    }
    if (ob.stats || ob.jac) {
      // a split model: every thread makes its outputs visible device-wide
      // before the chunk is counted (uniform branch)
      if (item.group_chunks > 1) __threadfence();
      __syncthreads();  // the item's samples are all written
      bool last = true;
      if (item.group_chunks > 1) {
        // the block finishing the model's last chunk reduces the model
        if (threadIdx.x == 0) {
          s_last = atomicAdd(done + item.group, 1u) + 1u ==
                   (unsigned)item.group_chunks;
          if (s_last) __threadfence();
        }
        __syncthreads();
        last = s_last != 0;
      }
      if (last) item_epilogue(m, item, U, ob, (double*)dyn, dyn_bytes);
    }
    __syncthreads();  // everyone done with sblob and dyn before restaging
  }
}

}  // namespace (flavour)
using namespace PYST_CAT(batch_flavour_, PYST_GROUPS, PYST_SCORE);

int PYST_CAT(launch_batch_, PYST_GROUPS, PYST_SCORE)(
    const uint32_t* d_blobs, const pyst_batch_item* d_items, int64_t n_items,
    const pyst_batch_limits* lim, const RunArgs& ra, const OutBase& ob,
    unsigned long long* queue, unsigned* done, int bs, cudaStream_t st) {
  const size_t wb =
      host_warp_bytes(lim->max_species, lim->max_reactions, PYST_SCORE);
  const size_t thread_bytes = (size_t)bs * lim->max_species * 12;
  const size_t wbytes = wb * (size_t)(bs / 32);
  const size_t dyn = thread_bytes > wbytes ? thread_bytes : wbytes;
  const int maxr_pk = lim->max_reactions < PYST_THREAD_MAX_REACTIONS
                          ? lim->max_reactions
                          : PYST_THREAD_MAX_REACTIONS;
  const size_t pk_bytes = packed_bytes(maxr_pk);
  size_t smem = (size_t)lim->max_blob_words * 4 + 16 + pk_bytes + dyn;
  if (smem > kMaxDynSmem) return PYST_EUNSUPPORTED;
  // room for the direct forms and their columns' extra element, if it fits
  const size_t fd = direct_bytes(kDirectMaxR), one = (size_t)bs * 4;
  const size_t fd_bytes =
      !PYST_GROUPS && smem + fd + one <= kMaxDynSmem ? fd : 0;
  if (fd_bytes) smem += fd + one;
  const size_t wide = (size_t)lim->max_reactions * 16;
  const int wide_cap = smem + wide <= kMaxDynSmem ? lim->max_reactions : 0;
  if (wide_cap) smem += wide;
  auto kf = k_batch<(bool)PYST_SCORE>;
  const int rc = set_smem(kf, smem);
  if (rc) return rc;
  if (cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st) !=
      cudaSuccess)
    return PYST_ECUDA;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, bs, smem);
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (int64_t)num_sms() * per_sm;
  if (grid > n_items) grid = n_items;
  kf<<<(unsigned)grid, bs, smem, st>>>(d_blobs, d_items, n_items, ra, ob,
                                       queue, done, lim->max_blob_words,
                                       (int)wb, (int)dyn, (int)pk_bytes,
                                       (int)fd_bytes, wide_cap);
  return cudaGetLastError() == cudaSuccess ? PYST_OK : PYST_ECUDA;
}

}  // namespace pyst
