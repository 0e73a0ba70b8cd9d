// One trajectory per group of lanes: the engine of runs too small to fill
// the GPU thread by thread.
//
// A trajectory is one dependent chain of steps, so a run of few trajectories
// is bound by the latency of a step (about 4 cycles per instruction of a
// lone warp), not by issue.  Here LG adjacent lanes (4 to 32) share a
// trajectory, and a step's chain is what remains when its work is laid out
// over them, with no shared memory on it:
//   * lane j owns reaction j: it holds the rate, the counts of the (up to
//     three) factors' species and, packed a byte each, what every reaction's
//     firing changes them by, and computes only its own propensity;
//   * the propensities are gathered by shuffles and every lane adds them up
//     in reaction order (FP64), so totals, selections and clocks are those of
//     one thread per trajectory, bit for bit;
//   * lane i owns species i: its count, its samples, its mean and variance
//     sums and its tau candidate (in reaction order, as the thread loop);
//   * lane g generates the random block and exponential variate of every
//     LG-th step, and lane j the Poisson draw of reaction j;
//   * lane j keeps reaction j's firing count and propensity integral
//     (scores).
// kSteps direct-method steps are run in a row before one vote asks whether
// any of them met something rare (a sample time, a zero or infinite total, a
// count out of range); if so the saved state comes back and as many exact
// single steps run instead.  All control flow is uniform over the warp:
// groups in the other mode sit a part out with their results dropped, so
// every shuffle has the full mask and groups meet again in each round.
//
// Measured (one B200, ms; before: the mode-sorted scheduler for tau-leaping,
// a warp-wide tree of speculated steps for the direct method up to 2,368
// trajectories, a thread each above): tau Schlogl 4,999 trajectories 20.2 ->
// 9.3, 1,184 20.3 -> 3.9; tau Lotka-Volterra 20,011 85 -> 31, 1,184 75 -> 17;
// direct Lotka-Volterra 1,024 72 -> 41, 4,700 119 -> 47; direct telegraph
// 1,024 7.6 -> 1.6; a 64-set sweep of 256 trajectories with scores 236 ->
// 123.  A step takes about 210 cycles of a lone warp, a leap about 4,000; past
// 4 lanes x 112 trajectories per SM issue bounds it.
//
// Same algorithms and reference sources as pyst_engine.cuh.  Models: at most
// 8 packable reactions (blob_direct_factors), at most LG species.
#pragma once
#include "pyst_engine.cuh"

namespace pyst {

// Direct-method steps per vote (at most the group's lanes).  The direct method
// on Lotka-Volterra, 1,024 trajectories: 50.4 ms at 4 steps, 39.9 at 8, 38.9
// at 16, but 16 lose on Schlogl, whose sample times are 25 to 90 steps apart
// (1,700 trajectories: 9.0, 8.4, 9.0); tau-leaping's fallback rounds with
// their samples and leaps between lose from 5 up (Schlogl 1,024: 3.9 at 4,
// 4.4 at 10).
constexpr int kGroupStepsDirect = 8, kGroupStepsTau = 4;
// votes per round of the loop: a leap costs about as much as 16 steps, so
// that groups in either mode wait little for the others
constexpr int kGroupVotes = 4;

// R: at most 8, at least the model's reaction count (missing reactions have
// rate 0: their propensities add nothing and are never selected).  FC:
// factor slots.  first(): this group's first trajectory, next(): the one
// after (both called by all lanes of the warp, `want` telling whose result
// is used); out(u): where trajectory u's results go.
template <int R, int FC, int LG, bool TAU, bool SCORE, class Next, class Out>
__device__ void run_groups(const ModelView& m, const RunArgs& ra,
                           uint64_t id_base, int64_t n_traj, Next next,
                           Out out) {
  constexpr int kMost = TAU ? kGroupStepsTau : kGroupStepsDirect;
  constexpr int kGroupSteps = kMost < LG ? kMost : LG;
  static_assert(R <= LG && LG <= 32 && R <= 8 && kGroupSteps <= LG, "");
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, gl = lane & (LG - 1);
  const unsigned gm =
      LG == 32 ? kAll : ((1u << (LG & 31)) - 1u) << (lane & ~(LG - 1));
  auto gany = [&](bool c) { return (__ballot_sync(kAll, c) & gm) != 0u; };
  auto gshfl = [&](auto v, int src) {
    return __shfl_sync(kAll, v, src, LG);
  };
  const int Rm = m.R, S = m.S, ita = m.ita, kappa = m.kappa;

  // ---- this lane's reaction and species --------------------------------
  // change of species sp by a firing of reaction j
  auto delta = [&](int sp, int j) {
    int v = 0;
    for (int e = m.netptr(j); e < m.netptr(j + 1); ++e)
      if (ent_lo(m.net(e)) == sp) v = ent_hi_s16(m.net(e));
    return v;
  };
  // the changes of species sp by reactions 0..7, a byte each
  auto changes = [&](int sp) {
    uint32_t lo = 0, hi = 0;
    for (int j = 0; j < Rm && j < 8; ++j) {
      const uint32_t b = (uint32_t)delta(sp, j) & 0xFFu;
      if (j < 4) lo |= b << (8 * j);
      else hi |= b << (8 * (j - 4));
    }
    return make_uint2(lo, hi);
  };
  const float rate = gl < Rm ? m.rate(gl) : 0.0f;
  int fsp[FC], fsub[FC];
  uint2 fch[FC];
#pragma unroll
  for (int q = 0; q < FC; ++q) {
    fsp[q] = -1;
    fsub[q] = 0;
    fch[q] = make_uint2(0u, 0u);
  }
  int neg_sp[2] = {0, 0}, neg_v[2] = {0, 0};  // what a firing takes (TAU)
  if (gl < Rm) {
    int k = 0;
    for (int e = m.facptr(gl); e < m.facptr(gl + 1); ++e) {
      const uint32_t fe = m.fac(e);
      for (int q = 0; q < fac_order(fe); ++q, ++k) {
#pragma unroll
        for (int c = 0; c < FC; ++c)
          if (c == k) {
            fsp[c] = ent_lo(fe);
            fsub[c] = q * fac_falling(fe);
            fch[c] = changes(ent_lo(fe));
          }
      }
    }
    int k2 = 0;
    for (int e = m.netptr(gl); e < m.netptr(gl + 1) && k2 < 2; ++e) {
      const int v = ent_hi_s16(m.net(e));
      if (v < 0) {
        neg_sp[k2] = ent_lo(m.net(e));
        neg_v[k2++] = -v;
      }
    }
  }
  const uint2 own = gl < S ? changes(gl) : make_uint2(0u, 0u);
  const int x0 = gl < S ? m.x0(gl) : 0;
  const uint32_t gw = gl < S ? m.g(gl) : 0u;
  const double t_end = m.time(ita - 1);

  // ---- the trajectory's state -------------------------------------------
  bool active = false, more = true, first = true;
  Stream rs = make_stream(ra.seed, 0);
  TrajOut o;
  int x = 0, xf[FC];
  double t = 0.0, tf = 0.0;
  int f = 0;
  int64_t steps = 0, events = 0;
  int nst = 0, nev = 0, lim = 0;  // 32-bit parts of steps, events; the limit
  uint64_t h = 0;
  bool ssa_mode = !TAU;
  int ssa_left = 0, exact = 0;
  uint32_t leap_q = 0;
  double integ = 0.0;
  int cnt = 0;  // (as the thread engine's)
  int status = PYST_TRAJ_DONE;
  bool done = false, fill_state = false;
  // variates: this lane's of blocks vb + gl (c) and vb + LG + gl (n; valid
  // when have_n); off: the next step's place in the window
  uint64_t vb = 0;
  int off = 0;
  bool have_n = false;
  double e_c = 0.0, u_c = 0.0, e_n = 0.0, u_n = 0.0;
#pragma unroll
  for (int q = 0; q < FC; ++q) xf[q] = 0;

  auto variates_of = [&](uint64_t blk, double& e, double& u) {
    rs.n = blk;
    const uint4 w = next_block(rs);
    e = -pyst_log(u53(w.x, w.y));
    u = u53(w.z, w.w);
  };
  // Move a window that is used up on by LG blocks.  When a group lacks its
  // next block's variates, every group that does generates them, so that
  // groups out of phase still share the work.
  auto advance = [&]() {
    if (__any_sync(kAll, off >= LG && !have_n)) {
      if (!have_n) {
        variates_of(vb + (uint64_t)(LG + gl), e_n, u_n);
        have_n = true;
      }
    }
    if (off >= LG) {
      e_c = e_n;
      u_c = u_n;
      vb += LG;
      off -= LG;
      have_n = false;
    }
  };
  auto steps_left = [&]() {
    const int64_t left = ra.step_budget - steps;
    return (int)(left < (1ll << 30) ? left : (1ll << 30));
  };
  // the propensity and the sums over the reactions (P[R - 1]: the total)
  auto propensity_own = [&]() {
    float a = __fmul_rn(rate, (float)xf[0]);
#pragma unroll
    for (int q = 1; q < FC; ++q)
      a = __fmul_rn(a, (float)(xf[q] - fsub[q]));
    return a;
  };
  auto gather = [&](float a, double (&P)[R]) {
    const double y = rate_bits(a);
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      s = __fma_rn(gshfl(y, j), 0x1.0p896, s);
      P[j] = s;
    }
    return s;
  };
  auto select = [&](const double (&P)[R], double r) {
    int sel = 0;
#pragma unroll
    for (int j = 0; j < R - 1; ++j) sel += P[j] < r ? 1 : 0;
    return sel;
  };
  // byte sel of a change word pair, sign extended
  auto change = [&](uint2 c, uint32_t pick) {
    int v;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(c.x), "r"(c.y), "r"(pick));
    return v;
  };
  auto fire = [&](int sel) {
    const uint32_t pick = (uint32_t)sel * 0x1111u + 0x8880u;
    x += change(own, pick);
#pragma unroll
    for (int q = 0; q < FC; ++q) xf[q] += change(fch[q], pick);
  };

  while (true) {
    // ---- new trajectories ------------------------------------------------
    const bool want = !active && more;
    if (__any_sync(kAll, want)) {
      const int64_t u = next(first, want);
      first = false;
      if (want) {
        if (u < n_traj) {
          active = true;
          rs = make_stream(ra.seed, id_base + (uint64_t)u);
          o = out(u);
          x = x0;
#pragma unroll
          for (int q = 0; q < FC; ++q)
            xf[q] = fsp[q] >= 0 ? m.x0(fsp[q]) : 1;
          t = 0.0;
          f = 0;
          tf = m.time(0);
          steps = events = 0;
          nst = nev = 0;
          lim = steps_left();
          h = PYST_FNV_OFFSET;
          ssa_mode = !TAU;
          ssa_left = exact = 0;
          leap_q = 0;
          integ = 0.0;
          cnt = 0;
          status = PYST_TRAJ_DONE;
          done = fill_state = false;
          vb = 0;
          off = 0;
          have_n = false;
          variates_of((uint64_t)gl, e_c, u_c);
        } else {
          more = false;
        }
      }
    }
    if (!__any_sync(kAll, active)) break;

    // ---- direct-method steps ---------------------------------------------
    if (!TAU || __any_sync(kAll, active && ssa_mode)) {
      for (int rep = 0; rep < kGroupVotes; ++rep) {
        const bool ssa = active && ssa_mode && !done;
        // variates for the window's steps (a group that wants some lets the
        // others fill theirs)
        if (__any_sync(kAll, ssa && !have_n && off + kGroupSteps > LG)) {
          if (!have_n) {
            variates_of(vb + (uint64_t)(LG + gl), e_n, u_n);
            have_n = true;
          }
        }
        const bool row = ssa && exact == 0 && nst + kGroupSteps <= lim &&
                         (!TAU || ssa_left >= kGroupSteps);
        if (ssa && !row && exact == 0) exact = kGroupSteps;
        const double e_w = gl >= off ? e_c : e_n;
        const double u_w = gl >= off ? u_c : u_n;
        if (__any_sync(kAll, row)) {
          const int sx = x;
          int sxf[FC];
#pragma unroll
          for (int q = 0; q < FC; ++q) sxf[q] = xf[q];
          const double s_integ = integ;
          const int s_cnt = cnt;
          double tt = t;
          bool bad = false;
          int sels[kGroupSteps];
#pragma unroll
          for (int b = 0; b < kGroupSteps; ++b) {
            const float a = propensity_own();
            double P[R];
            const double a0 = gather(a, P);
            const int src = (off + b) & (LG - 1);
            const double e = gshfl(e_w, src), u = gshfl(u_w, src);
            const int sel = select(P, __dmul_rn(u, a0));
            sels[b] = sel;
            fire(sel);
            const double tau = ddiv_normal(e, a0);
            bad |= !rate_sum_usable(a0) || x < 0;
            if (SCORE) {
              integ = __dadd_rn(integ, __dmul_rn(rate_bits(a),
                                                 __dmul_rn(tau, 0x1.0p896)));
              cnt += sel == gl ? 1 : 0;
            }
            tt = __dadd_rn(tt, tau);
          }
          // (the clock does not decrease: its last value tells for all)
          bad = gany(bad || !(tt < tf));
          if (row && !bad) {
            t = tt;
            nst += kGroupSteps;
            nev += kGroupSteps;
            off += kGroupSteps;
            if (TAU) {
              ssa_left -= kGroupSteps;
              if (ssa_left <= 0) ssa_mode = false;
            }
            if (o.seqhash) {
#pragma unroll
              for (int b = 0; b < kGroupSteps; ++b)
                h = seq_mix(h, (uint64_t)sels[b]);
            }
          } else {
            x = sx;
#pragma unroll
            for (int q = 0; q < FC; ++q) xf[q] = sxf[q];
            integ = s_integ;
            cnt = s_cnt;
            if (row) exact = kGroupSteps;
          }
        }
        // ---- exact single steps -----------------------------------------
        while (__any_sync(kAll, exact > 0)) {
          const bool ex = exact > 0;
          const float a = propensity_own();
          double P[R];
          double a0 = gather(a, P);
          const int src = off & (LG - 1);
          const double e_x = gl >= off ? e_c : e_n;
          const double u_x = gl >= off ? u_c : u_n;
          const double e = gshfl(e_x, src), u = gshfl(u_x, src);
          double tau = ddiv_normal(e, a0);
          int sel = select(P, __dmul_rn(u, a0));
          const bool plain = ex && !rate_sum_usable(a0) && a0 != 0.0;
          if (__any_sync(kAll, plain)) {
            // an infinite or NaN propensity: plain conversions and division
            double s = 0.0, Q[R];
            int lastnz = -1;
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float aj = gshfl(a, j);
              if (j < Rm) s = __dadd_rn(s, (double)aj);
              if (j < Rm && aj > 0.0f) lastnz = j;
              Q[j] = s;
            }
            const double rx = __dmul_rn(u, s);
            int sx = -1;
#pragma unroll
            for (int j = R - 1; j >= 0; --j)
              if (j < Rm && Q[j] >= rx) sx = j;
            if (plain) {
              a0 = s;
              tau = __ddiv_rn(e, s);
              sel = sx < 0 ? lastnz : sx;
            }
          }
          bool stop = !ex;
          if (ex) {
            --exact;
            if (a0 == 0.0) {
              status = PYST_TRAJ_ABSORBED;
              fill_state = true;
              done = stop = true;
            } else if (nst >= lim) {
              steps += nst;
              events += nev;
              nst = nev = 0;
              lim = steps_left();
              if (lim <= 0) {
                status = PYST_TRAJ_STEP_BUDGET;
                done = stop = true;
              }
            }
          }
          if (!stop) {
            const double tn = __dadd_rn(t, tau);
            while (tn >= tf) {
              for (int k = 0; k < kappa; ++k)
                if (m.out(k) == gl) store_sample(o, ita, k, f, x);
              f++;
              if (f == ita) {
                done = true;
                break;
              }
              tf = m.time(f);
            }
            nst++;
            off++;
            if (SCORE) {
              const double dt = (tn >= t_end) ? __dsub_rn(t_end, t) : tau;
              const double w =
                  plain ? __dmul_rn((double)a, dt)
                        : __dmul_rn(rate_bits(a), __dmul_rn(dt, 0x1.0p896));
              integ = __dadd_rn(integ, w);
            }
            t = tn;
            stop = done;
          }
          if (!stop && sel >= 0) fire(sel);  // (-1: as thread_round's)
          if (gany(!stop && x < 0)) {
            status = PYST_TRAJ_OVERFLOW;
            done = stop = true;
          }
          if (!stop) {
            nev++;
            if (o.seqhash) h = seq_mix(h, (uint64_t)sel);
            if (SCORE) cnt += sel == gl ? 1 : 0;
            if (TAU && --ssa_left <= 0) {
              ssa_mode = false;
              exact = 0;
            }
          }
          if (done) exact = 0;
          advance();
        }
        advance();
        if (!__any_sync(kAll, active && ssa_mode && !done)) break;
      }
    }

    // ---- DECIDE and leap -------------------------------------------------
    if constexpr (TAU) {
      bool lp = active && !ssa_mode && !done;
      if (__any_sync(kAll, lp)) {
        const float a = propensity_own();
        float av[R];
        double a0 = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          av[j] = gshfl(a, j);
          a0 = add_rate(a0, av[j]);
        }
        const bool usable = rate_sum_usable(a0);
        if (lp && !usable) {
          if (a0 == 0.0) {
            status = PYST_TRAJ_ABSORBED;
            fill_state = true;
            done = true;
            lp = false;
          } else {
            a0 = 0.0;
#pragma unroll
            for (int j = 0; j < R; ++j)
              if (j < Rm) a0 = __dadd_rn(a0, (double)av[j]);
          }
        }
        if (lp && nst >= lim) {
          steps += nst;
          events += nev;
          nst = nev = 0;
          lim = steps_left();
          if (lim <= 0) {
            status = PYST_TRAJ_STEP_BUDGET;
            done = true;
            lp = false;
          }
        }
        // critical reactions: lane j looks at what reaction j takes
        bool cj = false;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int xs = gshfl(x, neg_sp[q]);
          cj |= neg_v[q] > 0 &&
                (int64_t)neg_v[q] * m.n_c > (int64_t)xs;
        }
        const unsigned crit =
            (__ballot_sync(kAll, cj && gl < Rm) & gm) >> (lane & ~(LG - 1));
        // lane i: mean and variance of species i's change, its tau
        float mu = 0.0f, s2 = 0.0f;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int v = change(own, (uint32_t)j * 0x1111u + 0x8880u);
          if (v != 0 && !((crit >> j) & 1u)) {
            mu = __fadd_rn(mu, __fmul_rn((float)v, av[j]));
            s2 = __fadd_rn(s2, __fmul_rn((float)(v * v), av[j]));
          }
        }
        float tau1 = __int_as_float(0x7f800000);
        if ((gw >> 16) & 1u) {
          const float c = tau_candidate(m.eta, gw, x, mu, s2);
          if (c < tau1) tau1 = c;
        }
#pragma unroll
        for (int d = LG / 2; d > 0; d >>= 1)
          tau1 = fminf(tau1, __shfl_xor_sync(kAll, tau1, d));
        const bool to_ssa = (double)tau1 < __ddiv_rn(10.0, a0);
        if (lp && to_ssa) {
          ssa_mode = true;
          ssa_left = ra.ssa_fallback_steps;
          lp = false;
        }
        if (__any_sync(kAll, lp)) {
          if (lp) nst++;
          double a0c = 0.0;
#pragma unroll
          for (int j = 0; j < R; ++j)
            if (j < Rm && ((crit >> j) & 1u))
              a0c = __dadd_rn(a0c, (double)av[j]);
          double tau2 = __longlong_as_double(0x7ff0000000000000ll);
          const double ec = gshfl(e_c, off & (LG - 1));
          const double uc = gshfl(u_c, off & (LG - 1));
          const bool use = lp && a0c > 0.0;
          if (use) {
            tau2 = __ddiv_rn(ec, a0c);
            off++;
          }
          const double tau1d = (double)tau1;
          double tau = (tau2 < tau1d) ? tau2 : tau1d;
          int kcrit = -1;
          if (tau1d > tau2) {
            const double r = __dmul_rn(uc, a0c);
            double cum = 0.0;
            int lastnz = -1;
#pragma unroll
            for (int j = 0; j < R; ++j) {
              if (j < Rm && ((crit >> j) & 1u)) {
                cum = __dadd_rn(cum, (double)av[j]);
                if (av[j] > 0.0f) lastnz = j;
                if (kcrit < 0 && cum >= r) kcrit = j;
              }
            }
            if (kcrit < 0) kcrit = lastnz;
          }
          int K[R];
          int64_t d = 0;
          int retry = 0;
          bool trying = lp;
          while (__any_sync(kAll, trying)) {
            int kj = 0;
            if (trying && gl < Rm) {
              if ((crit >> gl) & 1u)
                kj = gl == kcrit ? 1 : 0;
              else
                kj = poisson(__fmul_rn(a, (float)tau),
                             leap_key(rs, leap_q, gl, retry));
            }
            __syncwarp();
            bool bad = false;
            int64_t dn = 0;
            int Kn[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const int kq = gshfl(kj, j);
              bad |= kq < 0;
              Kn[j] = kq < 0 ? 0 : kq;
              dn += (int64_t)Kn[j] *
                    change(own, (uint32_t)j * 0x1111u + 0x8880u);
            }
            const int64_t nx = (int64_t)x + dn;
            const bool over = gany(nx > PYST_I32MAX);
            const bool neg = gany(nx < 0);
            if (trying) {
              d = dn;
#pragma unroll
              for (int j = 0; j < R; ++j) K[j] = Kn[j];
              if (bad || over) {
                status = bad ? PYST_TRAJ_SAMPLER : PYST_TRAJ_OVERFLOW;
                done = true;
                lp = trying = false;
              } else if (!neg) {
                trying = false;
              } else {
                tau = __dmul_rn(tau, 0.5);
                retry++;
                if (retry > ra.max_leap_retries) {
                  status = PYST_TRAJ_LEAP_RETRY;
                  done = true;
                  lp = trying = false;
                }
              }
            }
          }
          if (lp) {
            leap_q++;
            const double tn = __dadd_rn(t, tau);
            int64_t fired = 0;
#pragma unroll
            for (int j = 0; j < R; ++j) fired += K[j];
            if (o.seqhash) {
              h = seq_mix(h, PYST_LEAP_TAG);
#pragma unroll
              for (int j = 0; j < R; ++j)
                if (K[j] != 0)
                  h = seq_mix(h, ((uint64_t)j << 32) | (uint32_t)K[j]);
            }
            if (SCORE) {
              int kown = 0;
#pragma unroll
              for (int j = 0; j < R; ++j) kown = j == gl ? K[j] : kown;
              cnt = (int)((uint32_t)cnt + (uint32_t)kown);
              integ = __dadd_rn(integ, __dmul_rn((double)a, tau));
            }
            while (tn >= tf) {
              const double frac = __ddiv_rn(__dsub_rn(tf, t), tau);
              for (int k = 0; k < kappa; ++k)
                if (m.out(k) == gl) {
                  const double inc = rint(__dmul_rn((double)d, frac));
                  store_sample(o, ita, k, f, x + (int)inc);
                }
              f++;
              if (f == ita) {
                done = true;
                break;
              }
              tf = m.time(f);
            }
            x = (int)((int64_t)x + d);
            events += fired;
            t = tn;
          }
#pragma unroll
          for (int q = 0; q < FC; ++q) {
            const int xs = gshfl(x, fsp[q] >= 0 ? fsp[q] : 0);
            if (lp && fsp[q] >= 0) xf[q] = xs;
          }
          advance();
        }
      }
    }

    // ---- finished trajectories -------------------------------------------
    if (active && done) {
      for (; f < ita; ++f)
        for (int k = 0; k < kappa; ++k)
          if (m.out(k) == gl)
            store_sample(o, ita, k, f, fill_state ? x : -1);
      if (gl == 0) {
        if (o.status) *o.status = (uint8_t)status;
        if (o.events) *o.events = events + nev;
        if (o.seqhash) *o.seqhash = h;
        if (o.t_final) *o.t_final = t;
      }
      if (SCORE && o.score && gl < Rm)
        o.score[gl] = __dsub_rn((double)cnt, integ);
      active = false;
      done = false;
    }
  }
}

}  // namespace pyst
