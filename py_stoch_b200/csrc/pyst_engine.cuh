// Per-trajectory simulation engines.
//
// Two mappings of one trajectory onto the GPU:
//   * run_thread<MAXR,...>: one trajectory per thread, for R <= MAXR <= 32.
//     The propensities a[MAXR] live in registers (loops unrolled over the
//     compile-time bound and guarded by j < R); species counts live in a
//     per-thread column of shared memory (element i*bs + lane-of-block).
//   * run_warp<...>: one trajectory per warp, for any R.  Lanes own
//     contiguous reaction slices; the total propensity is a Kogge-Stone
//     prefix sum over the lanes' FP64 partial sums (shuffles) and the firing
//     reaction is found with a ballot over the lane prefixes.
//
// Both restate the reference algorithms:
//   direct method   mod/simulator/cuGillespie/gillespie.py:70-146,
//                   mod/simulator/cuTauLeaping/P3.py:71-151
//   tau-leaping     mod/simulator/cuTauLeaping/P1_P2.py:96-297 with helpers
//                   299-584; the host rounds of cuTauLeaping.py:49-76 become
//                   one loop per trajectory (mode DECIDE = P1_P2, mode SSA =
//                   up to ssa_fallback_steps iterations of P3).
// Precision: propensities FP32; total propensity, clock, cumulative
// selection sums and score integrals FP64; tau selection and leap sampling
// FP32.  Every floating-point operation is explicitly rounded.
#pragma once
#include <stdint.h>

#include "pyst_math.cuh"
#include "pyst_model.cuh"

namespace pyst {

struct RunArgs {
  uint64_t seed;
  int64_t step_budget;
  int32_t ssa_fallback_steps;
  int32_t max_leap_retries;
  int32_t stage_polls;  // bound of the model-staging wait (stage_blob)
};

// Output pointers of one trajectory (already offset to it).
struct TrajOut {
  int32_t* samples;  // element (k*ita + f)*stride
  int64_t stride;
  uint8_t* status;
  int64_t* events;
  uint64_t* seqhash;
  double* t_final;
  double* score;  // [R]
};

#define PYST_I32MAX 2147483647ll
#define PYST_LEAP_TAG 0xFFFFFFFFull

__device__ __forceinline__ float gfun(uint32_t gw, int x) {
  const int H = (int)(gw & 0xFFu);
  const int Ht = (int)((gw >> 8) & 0xFFu);
  const float xf = (float)x;
  if (H == 1) return 1.0f;
  if (H == 2) {
    if (Ht == 2) return __fadd_rn(2.0f, __fdiv_rn(1.0f, __fsub_rn(xf, 1.0f)));
    return 2.0f;
  }
  if (H == 3) {
    if (Ht == 3) {
      const float t1 = __fdiv_rn(1.0f, __fsub_rn(xf, 1.0f));
      const float t2 = __fdiv_rn(2.0f, __fsub_rn(xf, 2.0f));
      return __fadd_rn(__fadd_rn(3.0f, t1), t2);
    }
    if (Ht == 2)
      return __fmul_rn(1.5f,
                       __fadd_rn(2.0f, __fdiv_rn(1.0f, __fsub_rn(xf, 1.0f))));
    return 3.0f;
  }
  if (H >= 4) {
    // Cao-Gillespie-Petzold's g generalised past third order (the
    // reference's CalculateG returns 0 there, P1_P2.py:480-485, which makes
    // tau infinite): g = (H/n) (n + sum_{k=1}^{n-1} k/(x-k)), n = H_type;
    // for H <= 3 this is exactly the table above.
    const int n = Ht < 1 ? 1 : Ht;
    float sm = (float)n;
    for (int k = 1; k < n; ++k)
      sm = __fadd_rn(sm, __fdiv_rn((float)k, __fsub_rn(xf, (float)k)));
    return __fmul_rn(__fdiv_rn((float)H, (float)n), sm);
  }
  return 0.0f;
}

// Candidate tau of one reactant species (P1_P2.py:421-426), FP32.
__device__ __forceinline__ float tau_candidate(float eta, uint32_t gw, int x,
                                               float mu, float s2) {
  const float g = gfun(gw, x);
  const float num = fmaxf(__fdiv_rn(__fmul_rn(eta, (float)x), g), 1.0f);
  const float lhs = __fdiv_rn(num, fabsf(mu));
  const float rhs = __fdiv_rn(__fmul_rn(num, num), s2);
  return fminf(lhs, rhs);
}

__device__ __forceinline__ PoissonKey leap_key(const Stream& s, uint32_t q,
                                               int j, int retry) {
  PoissonKey pk;
  pk.k0 = s.k0;
  pk.k1 = s.k1;
  pk.c0 = q;
  pk.c1 = 0x80000000u | ((uint32_t)j << 12) | ((uint32_t)retry << 6);
  pk.c2 = s.c2;
  pk.c3 = s.c3;
  return pk;
}

// C integer division of two integral FP64 values: the quotient truncated
// toward zero (exact for |a|, |b| < 2^53: a quotient rounded up onto an
// integer is stepped back by the sign of the exact remainder).
__device__ __forceinline__ double law_idiv(double a, double b) {
  if (b == 0.0) return __longlong_as_double(0x7ff8000000000000ll);
  double q = trunc(__ddiv_rn(a, b));
  const double rem = __fma_rn(-q, b, a);
  if (q != 0.0 && rem != 0.0 && ((rem < 0.0) != (a < 0.0)))
    q = __dsub_rn(q, copysign(1.0, q));
  return q;
}

__device__ __forceinline__ double law_exp(double a) {
  if (!(a == a)) return a;
  if (a > 709.0) return __longlong_as_double(0x7ff0000000000000ll);
  if (a < -708.0) return 0.0;
  return pyst_exp(a);
}

__device__ __forceinline__ double law_ln(double a) {
  if (!(a >= 0.0)) return __longlong_as_double(0x7ff8000000000000ll);
  if (a == 0.0) return __longlong_as_double((long long)0xfff0000000000000ull);
  if (a > 1.7976931348623157e308) return a;
  return pyst_log(a);
}

// General kinetic law of reaction j (pyst_model_desc: postfix program over
// the species counts x[i * xs] and FP64 constants), each operation
// explicitly rounded, the result rounded once to the FP32 propensity.  The
// packer checks the programs' stacks; a malformed one gives NaN here (and
// the trajectory the PYST_TRAJ_RATE status).  Out of line: one copy serves
// every call site.  Bound by the latency of its dependent operations: an
// operand followed by a binary operation is applied to the top of the stack
// at once, so that most operands are never pushed, the top of the stack and
// the next two program words are in registers, and program, constants and
// counts are read by their shared-memory addresses (all three are in shared
// memory in every kernel; passing the model view by reference put two
// dependent local-memory loads before each of them).  Saturating laws, direct
// method, 10,007 trajectories: 17.1 -> 12.9 ms.
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ double lds_f64(uint32_t addr) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
// law: address of the program's first word, n its words; lawc: of the
// constants; x, xs: of species 0's count and bytes between species.
__device__ __forceinline__ float law_program(uint32_t law, int n,
                                             uint32_t lawc, uint32_t x,
                                             uint32_t xs) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  double st[8];  // below the top: st[0 .. sp - 2]
  double top = 0.0;
  int sp = 0, c = 0;
  uint32_t w0 = c < n ? lds_u32(law) : 0u;
  uint32_t w1 = c + 1 < n ? lds_u32(law + 4u) : 0u;
  auto step = [&]() {
    ++c;
    w0 = w1;
    w1 = c + 1 < n ? lds_u32(law + 4u * (uint32_t)(c + 1)) : 0u;
  };
  while (c < n) {
    int op = (int)(w0 >> 24);
    const int arg = (int)(w0 & 0xFFFFFFu);
    step();
    double a, b;
    if (op == 1 || op == 2 || op == 16) {
      if (sp >= 8 || (op == 16 && sp < 1)) return (float)nan;
      double v = top;
      if (op == 1)
        // the exact conversion of an int, by placement in a double's fields
        v = __dsub_rn(
            __hiloint2double(0x43300000,
                             (int)(lds_u32(x + (uint32_t)arg * xs) ^
                                   0x80000000u)),
            0x1.0p52 + 0x1.0p31);
      else if (op == 2)
        v = lds_f64(lawc + 8u * (uint32_t)arg);
      const int nop = c < n ? (int)(w0 >> 24) : 0;
      if (nop < 3 || nop > 7 || sp < 1) {
        if (sp > 0) st[sp - 1] = top;
        ++sp;
        top = v;
        continue;
      }
      a = top;
      b = v;
      op = nop;
      step();
    } else if (op >= 3 && op <= 7) {
      if (sp < 2) return (float)nan;
      --sp;
      b = top;
      a = st[sp - 1];
    } else {
      if (sp < 1) return (float)nan;
      if (op == 8) top = -top;
      else if (op == 10) top = law_exp(top);
      else if (op == 11) top = law_ln(top);
      else if (op == 12) top = __dsqrt_rn(top);
      else if (op == 13) top = fabs(top);
      else if (op == 14) top = floor(top);
      else if (op == 15) top = ceil(top);
      else return (float)nan;
      continue;
    }
    if (op == 5) top = __dmul_rn(a, b);
    else if (op == 3) top = __dadd_rn(a, b);
    else if (op == 4) top = __dsub_rn(a, b);
    else if (op == 6) top = __ddiv_rn(a, b);
    else top = law_idiv(a, b);
  }
  return sp == 1 ? __double2float_rn(top) : (float)nan;
}

// A propensity a kinetic law may return: finite and non-negative.
__device__ __forceinline__ bool valid_rate(float a) {
  return a >= 0.0f && a <= 3.4028234663852886e38f;
}

// A law is called in two forms.  By addresses: the caller computes
// them, which costs it registers at every call site; by the model view, which
// then lives in local memory.  The register engine takes the second for more
// than 4 reactions, whose unrolled call sites spill otherwise (direct method,
// 30,000 trajectories without any law, ms: 12 reactions 7.6 -> 6.1, 32
// reactions 32.9 -> 22.4; with two laws among 23 reactions 10.1 -> 8.7), the
// first up to 4 (10,007 trajectories, two laws of 3 reactions: 2.63 against
// 2.80).
static __device__ __noinline__ float eval_law(uint32_t law, int n,
                                              uint32_t lawc, uint32_t x,
                                              uint32_t xs) {
  return law_program(law, n, lawc, x, xs);
}
static __device__ __noinline__ float eval_law_of(const ModelView& m, int j,
                                                 const int32_t* xc, int xs) {
  const int c0 = m.lawptr(j), n = m.lawptr(j + 1) - c0;
  return law_program(smem_u32(m.w + m.o_law + c0), n,
                     smem_u32(m.w + m.o_lawc), smem_u32(xc),
                     (uint32_t)xs * 4u);
}
// Propensity of reaction j in FP32: the reaction's kinetic-law program if
// it has one (LAWS: the caller supports them), else the rate, then factors
// in entry order.  Species counts are x[i * xs].
// VIEW: which form of the law evaluation.
template <bool LAWS = true, bool VIEW = false>
__device__ __forceinline__ float propensity(const ModelView& m, int j,
                                            const int32_t* xc, int xs) {
  if (LAWS && VIEW) {
    if (m.nlaw && m.lawptr(j + 1) > m.lawptr(j))
      return eval_law_of(m, j, xc, xs);
  } else if (LAWS && m.nlaw) {
    const int c0 = m.lawptr(j), n = m.lawptr(j + 1) - c0;
    if (n > 0)
      return eval_law(smem_u32(m.w + m.o_law + c0), n,
                      smem_u32(m.w + m.o_lawc), smem_u32(xc),
                      (uint32_t)xs * 4u);
  }
  float a = m.rate(j);
  const int e1 = m.facptr(j + 1);
  for (int e = m.facptr(j); e < e1; ++e) {
    const uint32_t fe = m.fac(e);
    const int x = xc[(int64_t)ent_lo(fe) * xs];
    const int n = fac_order(fe);
    const int fall = fac_falling(fe);
    for (int q = 0; q < n; ++q) a = __fmul_rn(a, (float)(x - q * fall));
  }
  return a;
}

// Packed reaction descriptors for small mass-action reactions, built in
// shared memory by each block after staging the model:
//   factors  pk[j]:     two slots of 13 bits, slot s at bit 13s:
//                       species (10 bits) | order 1..3 (2 bits) | falling
//                       (1 bit); order 0 = empty slot;
//   net      pk[R + j]: two slots of 15 bits, slot s at bit 15s: species
//                       (10 bits) | delta (5-bit two's complement), and the
//                       number of entries in bits 30-31.
// A reaction fits when it has at most two reactant entries of order <= 3
// and at most two net-change entries with |delta| <= 15 over species
// < 1024.  The packed forms take the same operations in the same order as
// the entry lists, so results are identical; they only remove the chains
// of dependent shared-memory loads (entry pointer -> entry -> species).
// Whether reaction j of the blob at `w` fits the packed descriptors: the
// host launchers' form of the conditions pack_reactions checks inline (its
// own form keeps the mode-sorted kernel's register allocation unchanged);
// tests check that both decide alike.
__host__ __device__ inline bool blob_reaction_packable(const uint32_t* w,
                                                       int j) {
  const int ofp = (int)w[PYST_H_OFF_FACPTR], of = (int)w[PYST_H_OFF_FAC];
  const int onp = (int)w[PYST_H_OFF_NETPTR], on = (int)w[PYST_H_OFF_NET];
  const int e0 = (int)w[ofp + j], e1 = (int)w[ofp + j + 1];
  if (e1 - e0 > 2) return false;
  for (int e = e0; e < e1; ++e) {
    const uint32_t fe = w[of + e];
    const int sp = (int)(fe & 0xFFFFu), n = (int)((fe >> 16) & 0xFFu);
    if (sp > 1023 || n < 1 || n > 3) return false;
  }
  const int n0 = (int)w[onp + j], n1 = (int)w[onp + j + 1];
  if (n1 - n0 > 2) return false;
  for (int e = n0; e < n1; ++e) {
    const uint32_t ne = w[on + e];
    const int sp = (int)(ne & 0xFFFFu);
    const int v = (int)(int16_t)(uint16_t)(ne >> 16);
    if (sp > 1023 || v < -16 || v > 15) return false;
  }
  return true;
}

// All threads of the block call this; true when every reaction fits (the
// conditions of blob_reaction_packable, checked inline).
__device__ __forceinline__ bool pack_reactions(const ModelView& m,
                                               uint32_t* pk) {
  bool ok = m.nlaw == 0;  // kinetic-law programs use the general path
  for (int j = threadIdx.x; j < m.R; j += blockDim.x) {
    const int e0 = m.facptr(j), e1 = m.facptr(j + 1);
    uint32_t d = 0;
    if (e1 - e0 > 2) ok = false;
    for (int e = e0; e < e1 && e < e0 + 2; ++e) {
      const uint32_t fe = m.fac(e);
      const int sp = ent_lo(fe), n = fac_order(fe);
      if (sp > 1023 || n < 1 || n > 3) ok = false;
      d |= ((uint32_t)(sp & 1023) | ((uint32_t)(n & 3) << 10) |
            ((uint32_t)fac_falling(fe) << 12))
           << (13 * (e - e0));
    }
    pk[j] = d;
    const int n0 = m.netptr(j), n1 = m.netptr(j + 1);
    uint32_t q = (uint32_t)(n1 - n0) << 30;
    if (n1 - n0 > 2) ok = false;
    for (int e = n0; e < n1 && e < n0 + 2; ++e) {
      const uint32_t ne = m.net(e);
      const int sp = ent_lo(ne), v = ent_hi_s16(ne);
      if (sp > 1023 || v < -16 || v > 15) ok = false;
      q |= ((uint32_t)(sp & 1023) | ((uint32_t)(v & 31) << 10))
           << (15 * (e - n0));
    }
    pk[m.R + j] = q;
  }
  return ok;
}

// propensity() from a packed factor descriptor and the rate.
template <class XGet>
__device__ __forceinline__ float propensity_packed(float rate, uint32_t d,
                                                   XGet xget) {
  float a = rate;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t f = d >> (13 * s);
    const int n = (int)((f >> 10) & 3u);
    if (n) {
      const int x = xget((int)(f & 1023u));
      const int fall = (int)((f >> 12) & 1u);
      a = __fmul_rn(a, (float)x);
      if (n > 1) a = __fmul_rn(a, (float)(x - fall));
      if (n > 2) a = __fmul_rn(a, (float)(x - 2 * fall));
    }
  }
  return a;
}

// ---- direct forms of small reactions ------------------------------------
// The packed descriptors still cost about 30 instructions per reaction and
// step to take apart, with branches that keep the compiler from overlapping
// a step's chains.  For models of at most 8 packable reactions with at most
// three reactant factors each, every block therefore also builds, per
// reaction, words that are used as they are:
//   fd[3j]     rate, byte offsets of the (up to) three factors' species in a
//              thread's column
//   fd[3j + 1] what the second and the third factor subtract (0, 1, 2)
//   fd[3j + 2] byte offset and change of the (up to) two species a firing
//              changes; fd[3R + 2]: of none (an unselected step)
// Slots a reaction does not use point to one extra element of the column,
// after the S species, that holds 1 (a factor 1, a change by 0), so there is
// nothing to test: with FC factor slots (1, 2 or 3, a template parameter: the
// most any reaction of the model has) a propensity is one load, FC species
// loads, conversions and multiplications, in entry order as before.
// Telegraph (R = 6, one factor) with scores, 1,048,576 trajectories: 158 ->
// 130 ms (423 thread instructions per event before); Schlogl direct, 50,000:
// 35.4 -> 32.2 ms with its copy to the host.
constexpr int kDirectMaxR = 8;
constexpr int kDirectMaxFactors = 3;

// The most reactant factors any reaction of a packable model has (1 to 6), 0
// for a model of more than 8 reactions: the launchers' choice of a kernel.
__host__ __device__ inline int blob_direct_factors(const uint32_t* w) {
  const int R = (int)w[PYST_H_R];
  if (R > kDirectMaxR) return 0;
  const int ofp = (int)w[PYST_H_OFF_FACPTR], of = (int)w[PYST_H_OFF_FAC];
  int most = 1;
  for (int j = 0; j < R; ++j) {
    int n = 0;
    for (int e = (int)w[ofp + j]; e < (int)w[ofp + j + 1]; ++e)
      n += (int)((w[of + e] >> 16) & 0xFFu);
    if (n > most) most = n;
  }
  return most;
}
// Whether such a model has direct forms, given that number.
__host__ __device__ inline bool has_direct_forms(int R, int factors) {
  return R >= 2 && factors > 0 && factors <= kDirectMaxFactors;
}

// Build the direct forms of a packable model for species columns of
// `stride` elements.  All threads of the block call this and synchronise
// before fd is read.
__device__ __forceinline__ void build_direct(const ModelView& m, uint4* fd,
                                             int stride) {
  const uint32_t one = (uint32_t)m.S * (uint32_t)stride * 4u;
  if (threadIdx.x == 0) fd[3 * m.R + 2] = make_uint4(one, 0u, one, 0u);
  for (int j = threadIdx.x; j < m.R; j += blockDim.x) {
    uint32_t off[kDirectMaxFactors] = {one, one, one};
    uint32_t sub[kDirectMaxFactors] = {0, 0, 0};
    int n = 0;
    for (int e = m.facptr(j); e < m.facptr(j + 1); ++e) {
      const uint32_t fe = m.fac(e);
      for (int q = 0; q < fac_order(fe); ++q)
        if (n < kDirectMaxFactors) {
          off[n] = (uint32_t)ent_lo(fe) * (uint32_t)stride * 4u;
          sub[n++] = (uint32_t)(q * fac_falling(fe));
        }
    }
    fd[3 * j] =
        make_uint4(__float_as_uint(m.rate(j)), off[0], off[1], off[2]);
    fd[3 * j + 1] = make_uint4(sub[1], sub[2], 0u, 0u);
    uint32_t noff[2] = {one, one}, nd[2] = {0, 0};
    for (int e = m.netptr(j), q = 0; e < m.netptr(j + 1) && q < 2; ++e, ++q) {
      noff[q] = (uint32_t)ent_lo(m.net(e)) * (uint32_t)stride * 4u;
      nd[q] = (uint32_t)ent_hi_s16(m.net(e));
    }
    fd[3 * j + 2] = make_uint4(noff[0], nd[0], noff[1], nd[1]);
  }
}

template <int FC>
__device__ __forceinline__ float propensity_direct(const uint4* fd, int j,
                                                   const int32_t* xc) {
  auto x = [&](uint32_t off) {
    return *reinterpret_cast<const int32_t*>(
        reinterpret_cast<const char*>(xc) + off);
  };
  const uint4 f = fd[3 * j];
  float a = __fmul_rn(__uint_as_float(f.x), (float)x(f.y));
  if (FC > 1) {
    const uint4 c = fd[3 * j + 1];
    a = __fmul_rn(a, (float)(x(f.z) - (int)c.x));
    if (FC > 2) a = __fmul_rn(a, (float)(x(f.w) - (int)c.y));
  }
  return a;
}

// ---- large networks ------------------------------------------------------
// Beyond the register arrays every step evaluates every propensity, so the
// chain of dependent loads per reaction (entry range, entry, count) and its
// loops are what a step consists of.  For mass-action models whose reactions
// have at most two reactant species of order 1 or 2, each block keeps one
// 16-byte word per reaction:
//   rate; per reactant species << 8 | 4 | falling << 1 | (order 2); 0: none
// -- one load, then the counts.  Same operations in the same order.
__device__ __forceinline__ size_t wide_bytes(int R) { return (size_t)R * 16; }

// All threads of the block call this; true (per thread) when every reaction
// this thread looked at fits.
__device__ __forceinline__ bool build_wide(const ModelView& m, uint4* fw) {
  bool ok = m.nlaw == 0;
  for (int j = threadIdx.x; j < m.R; j += blockDim.x) {
    uint32_t e2[2] = {0u, 0u};
    const int e0 = m.facptr(j), e1 = m.facptr(j + 1);
    if (e1 - e0 > 2) ok = false;
    for (int e = e0; e < e1 && e < e0 + 2; ++e) {
      const uint32_t fe = m.fac(e);
      const int n = fac_order(fe);
      if (n < 1 || n > 2) ok = false;
      e2[e - e0] = (uint32_t)ent_lo(fe) << 8 | 4u |
                   (uint32_t)fac_falling(fe) << 1 | (n == 2 ? 1u : 0u);
    }
    fw[j] = make_uint4(__float_as_uint(m.rate(j)), e2[0], e2[1], 0u);
  }
  return ok;
}

__device__ __forceinline__ float propensity_wide(const uint4 d,
                                                 const int32_t* xc, int xs) {
  float a = __uint_as_float(d.x);
  if (d.y) {
    const int x = xc[(int)(d.y >> 8) * xs];
    a = __fmul_rn(a, (float)x);
    if (d.y & 1u) a = __fmul_rn(a, (float)(x - (int)((d.y >> 1) & 1u)));
  }
  if (d.z) {
    const int x = xc[(int)(d.z >> 8) * xs];
    a = __fmul_rn(a, (float)x);
    if (d.z & 1u) a = __fmul_rn(a, (float)(x - (int)((d.z >> 1) & 1u)));
  }
  return a;
}

// The same with selects for the tests (a missing factor is an exact factor
// 1): for lanes that evaluate different reactions, which would diverge at
// every test.
__device__ __forceinline__ float propensity_wide_lanes(const uint4 d,
                                                       const int32_t* xc) {
  const int xa = xc[d.y >> 8], xb = xc[d.z >> 8];
  const float fa = d.y ? (float)xa : 1.0f;
  const float fb = d.z ? (float)xb : 1.0f;
  const float ga = d.y & 1u ? (float)(xa - (int)((d.y >> 1) & 1u)) : 1.0f;
  const float gb = d.z & 1u ? (float)(xb - (int)((d.z >> 1) & 1u)) : 1.0f;
  float a = __fmul_rn(__uint_as_float(d.x), fa);
  a = __fmul_rn(a, ga);
  a = __fmul_rn(a, fb);
  return __fmul_rn(a, gb);
}

// Entry q (< 2) of a packed net-change descriptor: species and delta.
__device__ __forceinline__ int pnet_species(uint32_t d, int q) {
  return (int)((d >> (15 * q)) & 1023u);
}
__device__ __forceinline__ int pnet_delta(uint32_t d, int q) {
  return ((int)((d >> (15 * q + 10)) & 31u) ^ 16) - 16;
}
__device__ __forceinline__ int pnet_count(uint32_t d) { return (int)(d >> 30); }

// acc + (double)a for a >= 0 (the sign of a zero is dropped: it does not
// change the sum).  The float's bits shifted into a double's fields are
// a 2^-896, subnormals and zero included, and the fused multiply-add scales
// them back exactly, so no conversion instruction (23 cycles of latency, an
// eighth of the issue rate) is on a step's dependent chain.  An infinite or
// NaN a adds 2^128 or more: callers test sums against PYST_RATE_BIG.
#define PYST_RATE_BIG 0x1.0p128
__device__ __forceinline__ double rate_bits(float a) {
  const uint32_t u = __float_as_uint(a) & 0x7FFFFFFFu;
  return __hiloint2double((int)(u >> 3), (int)(u << 29));
}
__device__ __forceinline__ double add_rate(double acc, float a) {
  return __fma_rn(rate_bits(a), 0x1.0p896, acc);
}
// Whether a sum of add_rate terms is neither zero nor at PYST_RATE_BIG
// (for a sum >= 0, by its high word).
__device__ __forceinline__ bool rate_sum_usable(double a0) {
  return (uint32_t)__double2hiint(a0) - 1u < 0x47F00000u - 1u;
}

__device__ __forceinline__ void store_sample(const TrajOut& o, int ita, int k,
                                             int f, int32_t v) {
  o.samples[((int64_t)k * ita + f) * o.stride] = v;
}

// ===================================================================
// one trajectory per thread
// ===================================================================
// Everything a thread-mapped trajectory carries between steps, apart from
// its species counts (shared-memory column) and score accumulators.  Split
// out so a block can park a trajectory between scheduling rounds.
struct TState {
  double t;
  uint64_t n;        // Philox block index of the main stream
  int64_t events;
  int64_t steps;
  uint64_t h;        // firing-sequence hash
  int32_t f;         // next sample index
  uint32_t leap_q;   // leaps taken (Poisson stream counter)
  int32_t ssa_left;  // SSA steps left in the current fallback round
  int32_t flags;     // TS_* bits, status in bits 8..15
};

enum {
  TS_SSA = 1,        // in an SSA fallback round (else DECIDE next)
  TS_LEAPGRP = 2,    // last DECIDE chose to leap
  TS_DONE = 4,       // trajectory finished
  TS_FILL = 8        // absorbed: remaining samples take the final state
};

__device__ __forceinline__ int ts_status(const TState& s) {
  return (s.flags >> 8) & 0xFF;
}

// ONE: the column has an element after the species that holds 1 (the
// direct forms').
template <bool TAU, bool ONE = false>
__device__ __forceinline__ void thread_init(const ModelView& m, int32_t* xcol,
                                            int bs, TState& s) {
  for (int i = 0; i < m.S; ++i) xcol[(int64_t)i * bs] = m.x0(i);
  if (ONE) xcol[(int64_t)m.S * bs] = 1;
  s.t = 0.0;
  s.n = 0;
  s.events = 0;
  s.steps = 0;
  s.h = PYST_FNV_OFFSET;
  s.f = 0;
  s.leap_q = 0;
  s.ssa_left = 0;
  s.flags = TAU ? TS_LEAPGRP : TS_SSA;
}

// Advance one trajectory.  Returns when it finishes, or -- for block
// scheduling -- when it has taken cap_ssa SSA steps or cap_leap leaps in
// this call, or when a DECIDE picks the other mode than the one the call
// started in (stop_on_switch).  Species counts are xcol[i*bs], the leap
// scratch of species i is slot[i*ss].  It stops only between steps, so the trajectory resumes
// exactly where it left off.  With unbounded caps this is the whole
// trajectory.
// PK: how reactions are read -- kPkLists (entry lists, general kinetic
// laws included), kPkPacked (packed descriptors, m.fast must hold) or
// kPkRuntime (whichever m.fast says; mass-action models only).
// The fixed forms carry only their own code and live registers (faster for
// the plain kernels); the mode-sorted kernel measured faster with one
// run-time form.
// LG > 1 (direct method only): LG adjacent lanes run the same trajectory
// in lockstep, each on its own species column, and lane g computes the
// Philox block and exponential variate of every LG-th step (g, g + LG, ...);
// a step takes its variates from the owning lane by shuffle.  The random
// numbers, and so the trajectory, are those of LG = 1; only the Philox and
// log work leaves the per-step dependent chain.  The caller lets one lane
// of the group write the outputs.
// GROUP (tau-leaping with stop_on_switch, the mode-sorted scheduler): 0
// any round; kGroupSsa / kGroupLeap when the caller knows the slot's group,
// which lets the compiler drop the code such a round never reaches (an SSA
// round stops when a DECIDE picks a leap, a leap round when it picks SSA
// steps) -- the same arithmetic, a smaller instruction footprint per warp.
enum { kPkLists = 0, kPkPacked = 1, kPkRuntime = 2 };
enum { kGroupAny = 0, kGroupSsa = 1, kGroupLeap = 2 };
// RX: the model's reaction count when the caller fixes it at compile time
// (the per-reaction loops then carry no run-time bound), else 0.
// FC: factor slots of the direct forms (build_direct; packed form only), or
// 0 to read the packed descriptors; the column then has S + 1 elements.
template <int MAXR, bool TAU, bool SCORE, int PK, int LG = 1,
          int GROUP = kGroupAny, int RX = 0, int FC = 0>
__device__ void thread_round(const ModelView& m, int32_t* xcol, int64_t* slot,
                             int bs, int ss, const RunArgs& ra,
                             uint64_t traj_id, TState& st, double* integ,
                             int* cnt, const TrajOut& o, int cap_ssa,
                             int cap_leap, bool stop_on_switch) {
  static_assert(RX == 0 || RX == MAXR, "an exact reaction count is MAXR");
  static_assert(FC == 0 || PK == kPkPacked, "direct forms: packed models");
  // The selection reads the prefix sums of the propensities where they stay
  // in registers: packable models of up to 8 reactions, others of up to 4.
  // Elsewhere they would be spilled, a store and a load per reaction and
  // step, and the selection adds up again until it reaches its reaction
  // (direct method, 30,000 trajectories, ms: packable, 12 reactions 4.43
  // with prefix sums, 3.82 without; 32 reactions with scores 35.7, 18.2;
  // 8 reactions, four factors 1.80, 2.06; lists, 8 reactions 4.21, 3.57).
  constexpr bool kPrefix = MAXR <= (PK == kPkPacked ? 8 : 4);
  const int S = m.S, R = RX ? RX : m.R, ita = m.ita, kappa = m.kappa;
  // the selection of a step that selects none (the direct forms have a
  // reaction without changes there, so that a step needs no test)
  const int kNone = FC > 0 ? R : -1;
  const bool pk = PK == kPkPacked || (PK == kPkRuntime && m.fast);
  // general kinetic laws: entry-list form only (a model with laws never
  // packs, and the sorted kernel's run-time form is not given such models)
  constexpr bool kLaws = PK == kPkLists;
#define XV(i) xcol[(int64_t)(i) * bs]
#define SL(i) slot[(int64_t)(i) * ss]
  Stream rs = make_stream(ra.seed, traj_id);
  rs.n = st.n;
  // The main stream is stateless, so its next block (and that block's
  // exponential variate) is computed one step ahead, off the dependent
  // chain of the current step; rs.n runs one block ahead of use.
  static_assert(LG == 1 || (!TAU && LG <= 32 && (LG & (LG - 1)) == 0),
                "lane groups: direct method, power of two up to 32 lanes");
  uint4 w_pf = make_uint4(0u, 0u, 0u, 0u);
  double e_pf = 0.0;
  // lane-group variates: block g_base + g_lane, consumed at step g_i
  const int g_lane = LG > 1 ? (int)(threadIdx.x & (LG - 1)) : 0;
  const unsigned g_mask =
      LG == 32 ? 0xffffffffu
      : LG > 1 ? ((1u << (LG & 31)) - 1u) << (threadIdx.x & 31 & ~(LG - 1))
               : 0u;
  uint64_t g_base = st.n;
  int g_i = 0;
  double g_e = 0.0, g_u = 0.0;
  if constexpr (LG > 1) {
    rs.n = g_base + (uint64_t)g_lane;
    const uint4 wg = next_block(rs);
    g_e = -pyst_log(u53(wg.x, wg.y));
    g_u = u53(wg.z, wg.w);
  } else {
    w_pf = next_block(rs);
    e_pf = -pyst_log(u53(w_pf.x, w_pf.y));
  }
  double t = st.t;
  int f = st.f;
  // steps and events of this call in 32 bits (nst; the events of its
  // direct-method steps are their number), folded into the 64-bit counts at
  // its end or when nst reaches `lim`, the step budget or 2^30
  int64_t events = st.events, steps = st.steps;
  int nst = 0, n_ssa = 0, n_leap = 0;
  auto steps_left = [&]() {
    const int64_t left = ra.step_budget - steps;
    return (int)(left < (1ll << 30) ? left : (1ll << 30));
  };
  int lim = steps_left();
  // out of steps?  (folds the counts when only the 32-bit range is used up)
  auto budget_spent = [&]() {
    steps += nst;
    events += n_ssa;
    nst = n_ssa = 0;
    lim = steps_left();
    return lim <= 0;
  };
  uint64_t h = st.h;
  const bool want_h = o.seqhash != nullptr;
  int status = PYST_TRAJ_DONE;
  bool fill_state = false, done = false;
  const double t_end = m.time(ita - 1);
  double tf = m.time(f);  // next sample time (f < ita while running)
  static_assert(GROUP == kGroupAny || TAU, "groups: tau-leaping only");
  // (a leap-group slot enters in DECIDE mode: the DECIDE that put it there
  // picked a leap)
  bool ssa_mode = GROUP == kGroupLeap ? false : (st.flags & TS_SSA) != 0;
  const bool group_leap = GROUP == kGroupAny ? (st.flags & TS_LEAPGRP) != 0
                                             : GROUP == kGroupLeap;
  bool leap_grp = group_leap;
  int ssa_left = st.ssa_left;
  uint32_t leap_q = st.leap_q;
  auto xget = [&](int i) { return XV(i); };
  // exponential variate and uniform of the main stream's next block
  auto take_variates = [&](double& e, double& u) {
    if constexpr (LG > 1) {
      e = __shfl_sync(g_mask, g_e, g_i, LG);
      u = __shfl_sync(g_mask, g_u, g_i, LG);
      if (++g_i == LG) {
        g_i = 0;
        g_base += LG;
        rs.n = g_base + (uint64_t)g_lane;
        const uint4 wg = next_block(rs);
        g_e = -pyst_log(u53(wg.x, wg.y));
        g_u = u53(wg.z, wg.w);
      }
    } else {
      e = e_pf;
      u = u53(w_pf.z, w_pf.w);
      w_pf = next_block(rs);
      e_pf = -pyst_log(u53(w_pf.x, w_pf.y));
    }
  };

  while (true) {
    // an SSA-group round whose cap falls where a DECIDE is due runs the
    // DECIDE before stopping, so the slot's next round is in the group of
    // its outcome (it would otherwise spend that round only switching).
    // (Leap-group rounds do not: their slots would run every continuing
    // leap's DECIDE twice.)  Whole-trajectory calls have no caps.
    const bool capped = GROUP == kGroupSsa ? n_ssa >= cap_ssa
                        : GROUP == kGroupLeap ? n_leap >= cap_leap : false;
    if (capped && !(GROUP == kGroupSsa && !ssa_mode)) break;
    float a[MAXR];
    double P[kPrefix ? MAXR : 1];  // prefix sums of the propensities
    double a0 = 0.0;
#pragma unroll
    for (int j = 0; j < MAXR; ++j) {
      if (j >= R) break;
      if constexpr (FC > 0)
        a[j] = propensity_direct<FC>(m.fd, j, xcol);
      else
        a[j] = pk ? propensity_packed(m.rate(j), m.pk[j], xget)
                  : propensity<kLaws, (MAXR > 4)>(m, j, xcol, bs);
      a0 = add_rate(a0, a[j]);
      if (kPrefix) P[j] = a0;
    }
    if (kLaws && m.nlaw) {
      bool bad = false;
#pragma unroll
      for (int j = 0; j < MAXR; ++j) {
        if (j >= R) break;
        bad |= !valid_rate(a[j]);
      }
      if (bad) {
        status = PYST_TRAJ_RATE;
        done = true;
        break;
      }
    }
    if (TAU && (GROUP == kGroupLeap || !ssa_mode)) {
      // ---------------- DECIDE: critical set, tau_1, SSA switch -------
      if (!rate_sum_usable(a0)) {
        if (a0 == 0.0) {
          status = PYST_TRAJ_ABSORBED;
          fill_state = true;
          done = true;
          break;
        }
        a0 = 0.0;  // an infinite or NaN propensity: plain conversions
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          a0 = __dadd_rn(a0, (double)a[j]);
        }
      }
      if (nst >= lim && budget_spent()) {
        status = PYST_TRAJ_STEP_BUDGET;
        done = true;
        break;
      }
      uint32_t crit = 0u;
#pragma unroll
      for (int j = 0; j < MAXR; ++j) {
        if (j >= R) break;
        if (pk) {
          // the negative entries of the net change (same test, any order)
          const uint32_t d = m.pk[R + j];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int v = pnet_delta(d, q);
            if (q < pnet_count(d) && v < 0 &&
                (int64_t)(-v) * m.n_c > (int64_t)XV(pnet_species(d, q)))
              crit |= 1u << j;
          }
        } else {
          const int e1 = m.critptr(j + 1);
          for (int e = m.critptr(j); e < e1; ++e) {
            const uint32_t ce = m.crit(e);
            if ((int64_t)(ce >> 16) * m.n_c > (int64_t)XV(ent_lo(ce)))
              crit |= 1u << j;
          }
        }
      }
      for (int i = 0; i < S; ++i) SL(i) = 0;
#pragma unroll
      for (int j = 0; j < MAXR; ++j) {
        if (j >= R) break;
        if (!((crit >> j) & 1u)) {
          auto acc = [&](int sp, int v) {
            float2 ms = *reinterpret_cast<float2*>(&SL(sp));
            ms.x = __fadd_rn(ms.x, __fmul_rn((float)v, a[j]));
            ms.y = __fadd_rn(ms.y, __fmul_rn((float)(v * v), a[j]));
            *reinterpret_cast<float2*>(&SL(sp)) = ms;
          };
          if (pk) {
            const uint32_t d = m.pk[R + j];
#pragma unroll
            for (int q = 0; q < 2; ++q)
              if (q < pnet_count(d)) acc(pnet_species(d, q), pnet_delta(d, q));
          } else {
            const int e1 = m.netptr(j + 1);
            for (int e = m.netptr(j); e < e1; ++e) {
              const uint32_t ne = m.net(e);
              acc(ent_lo(ne), ent_hi_s16(ne));
            }
          }
        }
      }
      float tau1 = __int_as_float(0x7f800000);
      for (int i = 0; i < S; ++i) {
        const uint32_t gw = m.g(i);
        if (!((gw >> 16) & 1u)) continue;
        const float2 ms = *reinterpret_cast<float2*>(&SL(i));
        const float c = tau_candidate(m.eta, gw, XV(i), ms.x, ms.y);
        if (c < tau1) tau1 = c;
      }
      if ((double)tau1 < __ddiv_rn(10.0, a0)) {
        ssa_mode = true;
        ssa_left = ra.ssa_fallback_steps;
        leap_grp = false;
        // regroup before stepping
        if (capped || GROUP == kGroupLeap || (stop_on_switch && group_leap))
          break;
        // fall through to the SSA step below with the same propensities
      } else {
        leap_grp = true;
        if (capped || GROUP == kGroupSsa || (stop_on_switch && !group_leap))
          break;
        // ---------------- leap ---------------------------------------
        nst++;
        n_leap++;
        double a0c = 0.0;
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          if ((crit >> j) & 1u) a0c = __dadd_rn(a0c, (double)a[j]);
        }
        double tau2 = __longlong_as_double(0x7ff0000000000000ll);
        double uc = 0.0;
        if (a0c > 0.0) {
          double ec;
          take_variates(ec, uc);
          tau2 = __ddiv_rn(ec, a0c);
        }
        const double tau1d = (double)tau1;
        double tau = (tau2 < tau1d) ? tau2 : tau1d;
        int kcrit = -1;
        if (tau1d > tau2) {
          const double r = __dmul_rn(uc, a0c);
          double cum = 0.0;
          int lastnz = -1;
#pragma unroll
          for (int j = 0; j < MAXR; ++j) {
            if (j >= R) break;
            if ((crit >> j) & 1u) {
              cum = __dadd_rn(cum, (double)a[j]);
              if (a[j] > 0.0f) lastnz = j;
              if (cum >= r) {
                kcrit = j;
                break;
              }
            }
          }
          if (kcrit < 0) kcrit = lastnz;
        }
        int K[MAXR];
        int retry = 0;
        bool ok = false;
        while (true) {
          bool bad = false;
          auto draw = [&](int j, float aj) {
            if ((crit >> j) & 1u) return (j == kcrit) ? 1 : 0;
            const float lam = __fmul_rn(aj, (float)tau);
            const int k = poisson(lam, leap_key(rs, leap_q, j, retry));
            if (k < 0) bad = true;
            return k < 0 ? 0 : k;
          };
          if constexpr (GROUP != kGroupAny && RX == 0) {
            // (the mode-sorted scheduler's leap rounds with a run-time
            // reaction count) one reaction per iteration, not unrolled: a
            // single inlined copy of the sampler's call sequence, a[j] and
            // K[j] by unrolled selects.  With the count fixed at compile
            // time the unrolled loop below measured as fast or faster
            // (6-reaction network 11.6 vs 12.0 ms).
#pragma unroll 1
            for (int j = 0; j < R; ++j) {
              float aj = a[0];
#pragma unroll
              for (int q = 1; q < MAXR; ++q) aj = (j == q) ? a[q] : aj;
              const int kj = draw(j, aj);
#pragma unroll
              for (int q = 0; q < MAXR; ++q)
                if (q == j) K[q] = kj;
            }
          } else {
#pragma unroll
            for (int j = 0; j < MAXR; ++j) {
              if (j >= R) break;
              K[j] = draw(j, a[j]);
            }
          }
          if (bad) {
            status = PYST_TRAJ_SAMPLER;
            break;
          }
          for (int i = 0; i < S; ++i) SL(i) = 0;
#pragma unroll
          for (int j = 0; j < MAXR; ++j) {
            if (j >= R) break;
            if (K[j] != 0) {
              if (pk) {
                const uint32_t d = m.pk[R + j];
#pragma unroll
                for (int q = 0; q < 2; ++q)
                  if (q < pnet_count(d))
                    SL(pnet_species(d, q)) += (int64_t)K[j] * pnet_delta(d, q);
              } else {
                const int e1 = m.netptr(j + 1);
                for (int e = m.netptr(j); e < e1; ++e) {
                  const uint32_t ne = m.net(e);
                  SL(ent_lo(ne)) += (int64_t)K[j] * ent_hi_s16(ne);
                }
              }
            }
          }
          bool neg = false, over = false;
          for (int i = 0; i < S; ++i) {
            const int64_t nx = (int64_t)XV(i) + SL(i);
            neg |= nx < 0;
            over |= nx > PYST_I32MAX;
          }
          if (over) {
            status = PYST_TRAJ_OVERFLOW;
            break;
          }
          if (!neg) {
            ok = true;
            break;
          }
          tau = __dmul_rn(tau, 0.5);
          retry++;
          if (retry > ra.max_leap_retries) {
            status = PYST_TRAJ_LEAP_RETRY;
            break;
          }
        }
        if (!ok) {
          done = true;
          break;
        }
        leap_q++;
        const double tn = __dadd_rn(t, tau);
        int64_t fired = 0;
        if (want_h) h = seq_mix(h, PYST_LEAP_TAG);
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          fired += K[j];
          if (want_h && K[j] != 0)
            h = seq_mix(h, ((uint64_t)j << 32) | (uint32_t)K[j]);
          if (SCORE) {
            cnt[j] += K[j];
            integ[j] = __dadd_rn(integ[j], __dmul_rn((double)a[j], tau));
          }
        }
        while (tn >= tf) {
          const double frac = __ddiv_rn(__dsub_rn(tf, t), tau);
          for (int k = 0; k < kappa; ++k) {
            const int i = m.out(k);
            const double inc = rint(__dmul_rn((double)SL(i), frac));
            store_sample(o, ita, k, f, XV(i) + (int)inc);
          }
          f++;
          if (f == ita) {
            done = true;
            break;
          }
          tf = m.time(f);
        }
        for (int i = 0; i < S; ++i) XV(i) = (int)((int64_t)XV(i) + SL(i));
        events += fired;
        t = tn;
        if (done) break;
        continue;
      }
    }
    // ------------------------ one direct-method step -------------------
    // The propensities above, the clock, the next step's random numbers
    // and the selection are one straight line of code, so that their
    // chains overlap; everything rare (a zero or infinite total, the step
    // budget, a sample time passed) is behind the one test at its end.
    double e, uu;
    take_variates(e, uu);
    double tau = ddiv_normal(e, a0);
    // the first j whose prefix sum reaches r: r <= a0, the last one (uu <=
    // 1), and the sums do not decrease, so it is the number of sums below
    // r, and a[sel] > 0
    const double r = __dmul_rn(uu, a0);
    int sel = 0;
    if constexpr (kPrefix) {
#pragma unroll
      for (int j = 0; j < MAXR - 1; ++j) {
        if (j >= R - 1) break;
        sel += P[j] < r ? 1 : 0;
      }
    } else {
      double cum = 0.0;
#pragma unroll
      for (int j = 0; j < MAXR - 1; ++j) {
        if (j >= R - 1) break;
        cum = add_rate(cum, a[j]);
        if (cum >= r) break;
        ++sel;
      }
    }
    double tn = __dadd_rn(t, tau);
    if (!rate_sum_usable(a0) || tn >= tf || nst >= lim) {
      if (a0 == 0.0) {
        status = PYST_TRAJ_ABSORBED;
        fill_state = true;
        done = true;
        break;
      }
      if (nst >= lim && budget_spent()) {
        status = PYST_TRAJ_STEP_BUDGET;
        done = true;
        break;
      }
      if (!rate_sum_usable(a0)) {
        // an infinite or NaN propensity: plain conversions and division
        a0 = 0.0;
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          a0 = __dadd_rn(a0, (double)a[j]);
        }
        tau = __ddiv_rn(e, a0);
        tn = __dadd_rn(t, tau);
        const double rx = __dmul_rn(uu, a0);
        double cum = 0.0;
        int lastnz = -1;
        sel = -1;
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          cum = __dadd_rn(cum, (double)a[j]);
          if (a[j] > 0.0f) lastnz = j;
          if (sel < 0 && cum >= rx) sel = j;
        }
        if (sel < 0) sel = lastnz < 0 ? kNone : lastnz;
      }
      while (tn >= tf) {
        if (LG == 1 || g_lane == 0)
          for (int k = 0; k < kappa; ++k)
            store_sample(o, ita, k, f, XV(m.out(k)));
        f++;
        if (f == ita) {
          done = true;
          break;
        }
        tf = m.time(f);
      }
    }
    nst++;
    if (SCORE) {
      const double dt = (tn >= t_end) ? __dsub_rn(t_end, t) : tau;
      if (rate_sum_usable(a0)) {
        // a dt by the shifted bits of add_rate: a 2^-896 x dt 2^896
        const double dts = __dmul_rn(dt, 0x1.0p896);
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          integ[j] = __dadd_rn(integ[j],
                               __dmul_rn(rate_bits(a[j]), dts));
        }
      } else {
#pragma unroll
        for (int j = 0; j < MAXR; ++j) {
          if (j >= R) break;
          integ[j] = __dadd_rn(integ[j], __dmul_rn((double)a[j], dt));
        }
      }
    }
    t = tn;
    if (done) break;
    // an unselected step (the total is NaN and no propensity is positive)
    // counts as a step and an event, and changes nothing
    if (FC > 0 || sel != kNone) {
      // counts stay in [0, 2^31): a step outside wraps to a negative number
      bool over = false;
      if constexpr (FC > 0) {
        const uint4 d = m.fd[3 * sel + 2];
        int32_t* xa = reinterpret_cast<int32_t*>(
            reinterpret_cast<char*>(xcol) + d.x);
        int32_t* xb = reinterpret_cast<int32_t*>(
            reinterpret_cast<char*>(xcol) + d.z);
        const int na = (int)((uint32_t)*xa + d.y);
        const int nb = (int)((uint32_t)*xb + d.w);
        *xa = na;
        *xb = nb;
        over = (na | nb) < 0;
      } else if (pk) {
        const uint32_t d = m.pk[R + sel];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q < pnet_count(d)) {
            const int sp = pnet_species(d, q);
            const int nx =
                (int)((uint32_t)XV(sp) + (uint32_t)pnet_delta(d, q));
            if (nx < 0) over = true;
            else XV(sp) = nx;
          }
        }
      } else {
        const int e1 = m.netptr(sel + 1);
        for (int e = m.netptr(sel); e < e1; ++e) {
          const uint32_t ne = m.net(e);
          const int sp = ent_lo(ne);
          const int nx = (int)((uint32_t)XV(sp) + (uint32_t)ent_hi_s16(ne));
          if (nx < 0) over = true;
          else XV(sp) = nx;
        }
      }
      if (over) {
        status = PYST_TRAJ_OVERFLOW;
        done = true;
        break;
      }
    }
    n_ssa++;  // (completed steps: each is one event)
    if (want_h) h = seq_mix(h, sel == kNone ? ~0ull : (uint64_t)sel);
    if (SCORE) {
#pragma unroll
      for (int j = 0; j < MAXR; ++j) cnt[j] += (j == sel) ? 1 : 0;
    }
    if (TAU) {
      if (--ssa_left <= 0) ssa_mode = false;
    }
  }
  events += n_ssa;
  steps += nst;
  st.t = t;
  // the prefetched block (LG = 1) was not used
  st.n = LG > 1 ? g_base + (uint64_t)g_i : rs.n - 1;
  st.events = events;
  st.steps = steps;
  st.h = h;
  st.f = f;
  st.leap_q = leap_q;
  st.ssa_left = ssa_left;
  st.flags = (ssa_mode ? TS_SSA : 0) | (leap_grp ? TS_LEAPGRP : 0) |
             (done ? TS_DONE : 0) | (fill_state ? TS_FILL : 0) |
             (status << 8);
#undef XV
#undef SL
}

// Write the remaining samples (state after absorption, -1 after an error)
// and the per-trajectory outputs of a finished trajectory.
template <int MAXR, bool SCORE>
__device__ void thread_finish(const ModelView& m, const int32_t* xcol, int bs,
                              const TState& st, const double* integ,
                              const int* cnt, const TrajOut& o) {
  const int ita = m.ita, kappa = m.kappa, R = m.R;
  const bool fill_state = (st.flags & TS_FILL) != 0;
  for (int f = st.f; f < ita; ++f)
    for (int k = 0; k < kappa; ++k)
      store_sample(o, ita, k, f,
                   fill_state ? xcol[(int64_t)m.out(k) * bs] : -1);
  if (o.status) *o.status = (uint8_t)ts_status(st);
  if (o.events) *o.events = st.events;
  if (o.seqhash) *o.seqhash = st.h;
  if (o.t_final) *o.t_final = st.t;
  if (SCORE && o.score) {
#pragma unroll
    for (int j = 0; j < MAXR; ++j) {
      if (j >= R) break;
      o.score[j] = __dsub_rn((double)cnt[j], integ[j]);
    }
  }
}

// One whole trajectory by the calling thread.  PK: kPkPacked or kPkLists
// when the caller knows the form (the host checks packability), -1 to
// choose by m.fast at run time (batched launches mix models).
// RX, FC as thread_round's.
template <int MAXR, bool TAU, bool SCORE, int PK = -1, int RX = 0, int FC = 0>
__device__ void run_thread(const ModelView& m, int32_t* xcol, int64_t* slot,
                           int bs, const RunArgs& ra, uint64_t traj_id,
                           const TrajOut& o) {
  TState st;
  thread_init<TAU, (FC > 0)>(m, xcol, bs, st);
  double integ[SCORE ? MAXR : 1];
  int cnt[SCORE ? MAXR : 1];
#pragma unroll
  for (int j = 0; j < (SCORE ? MAXR : 1); ++j) {
    integ[j] = 0.0;
    cnt[j] = 0;
  }
  if (PK == kPkPacked || (PK < 0 && m.fast))
    thread_round<MAXR, TAU, SCORE, kPkPacked, 1, kGroupAny, RX, FC>(
        m, xcol, slot, bs, bs, ra, traj_id, st, integ, cnt, o, 0x7fffffff,
        0x7fffffff, false);
  else if constexpr (PK == kPkLists) {
    thread_round<MAXR, TAU, SCORE, kPkLists, 1, kGroupAny, RX>(
        m, xcol, slot, bs, bs, ra, traj_id, st, integ, cnt, o, 0x7fffffff,
        0x7fffffff, false);
  } else if constexpr (PK < 0) {
    // a copy for the law evaluation by the model view: the view itself then
    // stays in registers for the other forms in the same kernel (batches, ms:
    // 40 packable models of 9 reactions with scores, 500 trajectories each
    // 5.4 -> 4.5; 500 Schlogl models beside a network of 1,000 reactions
    // 84 -> 69)
    const ModelView ml = m;
    thread_round<MAXR, TAU, SCORE, kPkLists, 1, kGroupAny, RX>(
        ml, xcol, slot, bs, bs, ra, traj_id, st, integ, cnt, o, 0x7fffffff,
        0x7fffffff, false);
  }
  thread_finish<MAXR, SCORE>(m, xcol, bs, st, integ, cnt, o);
}

// ===================================================================
// one trajectory per thread, any number of reactions
// ===================================================================
// Same steps and arithmetic as thread_round, for R beyond the register
// arrays: loops over reactions are not unrolled and propensities are
// recomputed where thread_round reads a[j] again (selection pass, critical
// sums, leap means), so nothing per reaction is stored.  The critical flag
// of a reaction is re-derived from the species counts when needed.
__device__ __forceinline__ bool is_critical(const ModelView& m, int j,
                                            const int32_t* xcol, int bs) {
  const int e1 = m.critptr(j + 1);
  for (int e = m.critptr(j); e < e1; ++e) {
    const uint32_t ce = m.crit(e);
    if ((int64_t)(ce >> 16) * m.n_c >
        (int64_t)xcol[(int64_t)ent_lo(ce) * bs])
      return true;
  }
  return false;
}

template <bool TAU, bool WIDE>
__device__ void thread_round_big(const ModelView& m, int32_t* xcol,
                                 int64_t* slot, int bs, int ss,
                                 const RunArgs& ra, uint64_t traj_id,
                                 TState& st, const TrajOut& o, int cap_ssa,
                                 int cap_leap, bool stop_on_switch) {
  const int S = m.S, R = m.R, ita = m.ita, kappa = m.kappa;
#define XV(i) xcol[(int64_t)(i) * bs]
#define SL(i) slot[(int64_t)(i) * ss]
  Stream rs = make_stream(ra.seed, traj_id);
  rs.n = st.n;
  double t = st.t;
  int f = st.f;
  int64_t events = st.events, steps = st.steps;
  uint64_t h = st.h;
  int status = PYST_TRAJ_DONE;
  bool fill_state = false, done = false;
  const int64_t budget = ra.step_budget;
  bool ssa_mode = (st.flags & TS_SSA) != 0;
  const bool group_leap = (st.flags & TS_LEAPGRP) != 0;
  bool leap_grp = group_leap;
  int ssa_left = st.ssa_left;
  uint32_t leap_q = st.leap_q;
  int n_ssa = 0, n_leap = 0;
  auto prop = [&](int j) {
    if constexpr (WIDE) return propensity_wide(m.fw[j], xcol, bs);
    else return propensity(m, j, xcol, bs);
  };
  // the sum of the propensities is kept at kSegs places, so that a
  // selection evaluates one segment again instead of half of all reactions
  constexpr int kSegs = 8;
  const int seg = (R + kSegs - 1) / kSegs;

  while (true) {
    if (n_ssa >= cap_ssa || n_leap >= cap_leap) break;
    double a0 = 0.0;
    bool bad_rate = false;
    double P[kSegs];
    if constexpr (WIDE) {
#pragma unroll
      for (int s = 0; s < kSegs; ++s) {
        const int j1 = (s + 1) * seg < R ? (s + 1) * seg : R;
#pragma unroll 4
        for (int j = s * seg; j < j1; ++j) a0 = add_rate(a0, prop(j));
        P[s] = a0;
      }
      if (!rate_sum_usable(a0)) {
        a0 = 0.0;  // zero, or an infinite or NaN propensity
        for (int j = 0; j < R; ++j) a0 = __dadd_rn(a0, (double)prop(j));
      }
    } else {
      for (int j = 0; j < R; ++j) {
        const float aj = prop(j);
        bad_rate |= !valid_rate(aj);
        a0 = __dadd_rn(a0, (double)aj);
      }
    }
    if (!WIDE && m.nlaw && bad_rate) {
      status = PYST_TRAJ_RATE;
      done = true;
      break;
    }
    if (a0 == 0.0) {
      status = PYST_TRAJ_ABSORBED;
      fill_state = true;
      done = true;
      break;
    }
    if (steps >= budget) {
      status = PYST_TRAJ_STEP_BUDGET;
      done = true;
      break;
    }
    if (TAU && !ssa_mode) {
      for (int i = 0; i < S; ++i) SL(i) = 0;
      for (int j = 0; j < R; ++j) {
        if (is_critical(m, j, xcol, bs)) continue;
        const float aj = prop(j);
        const int e1 = m.netptr(j + 1);
        for (int e = m.netptr(j); e < e1; ++e) {
          const uint32_t ne = m.net(e);
          const int sp = ent_lo(ne);
          const int v = ent_hi_s16(ne);
          float2 ms = *reinterpret_cast<float2*>(&SL(sp));
          ms.x = __fadd_rn(ms.x, __fmul_rn((float)v, aj));
          ms.y = __fadd_rn(ms.y, __fmul_rn((float)(v * v), aj));
          *reinterpret_cast<float2*>(&SL(sp)) = ms;
        }
      }
      float tau1 = __int_as_float(0x7f800000);
      for (int i = 0; i < S; ++i) {
        const uint32_t gw = m.g(i);
        if (!((gw >> 16) & 1u)) continue;
        const float2 ms = *reinterpret_cast<float2*>(&SL(i));
        const float c = tau_candidate(m.eta, gw, XV(i), ms.x, ms.y);
        if (c < tau1) tau1 = c;
      }
      if ((double)tau1 < __ddiv_rn(10.0, a0)) {
        ssa_mode = true;
        ssa_left = ra.ssa_fallback_steps;
        leap_grp = false;
        if (stop_on_switch && group_leap) break;
      } else {
        leap_grp = true;
        if (stop_on_switch && !group_leap) break;
        steps++;
        n_leap++;
        double a0c = 0.0;
        for (int j = 0; j < R; ++j)
          if (is_critical(m, j, xcol, bs))
            a0c = __dadd_rn(a0c, (double)prop(j));
        double tau2 = __longlong_as_double(0x7ff0000000000000ll);
        uint4 wc = make_uint4(0, 0, 0, 0);
        if (a0c > 0.0) {
          wc = next_block(rs);
          tau2 = __ddiv_rn(-pyst_log(u53(wc.x, wc.y)), a0c);
        }
        const double tau1d = (double)tau1;
        double tau = (tau2 < tau1d) ? tau2 : tau1d;
        int kcrit = -1;
        if (tau1d > tau2) {
          const double r = __dmul_rn(u53(wc.z, wc.w), a0c);
          double cum = 0.0;
          int lastnz = -1;
          for (int j = 0; j < R; ++j) {
            if (!is_critical(m, j, xcol, bs)) continue;
            const float aj = prop(j);
            cum = __dadd_rn(cum, (double)aj);
            if (aj > 0.0f) lastnz = j;
            if (cum >= r) {
              kcrit = j;
              break;
            }
          }
          if (kcrit < 0) kcrit = lastnz;
        }
        int retry = 0;
        bool ok = false;
        int64_t fired = 0;
        uint64_t hl = 0;
        while (true) {
          // Poisson firings, accumulated straight into the state change
          for (int i = 0; i < S; ++i) SL(i) = 0;
          bool bad = false;
          fired = 0;
          hl = seq_mix(h, PYST_LEAP_TAG);
          for (int j = 0; j < R; ++j) {
            int kj;
            if (is_critical(m, j, xcol, bs)) {
              kj = (j == kcrit) ? 1 : 0;
            } else {
              const float lam = __fmul_rn(prop(j), (float)tau);
              const int k = poisson(lam, leap_key(rs, leap_q, j, retry));
              if (k < 0) bad = true;
              kj = k < 0 ? 0 : k;
            }
            if (kj != 0) {
              fired += kj;
              hl = seq_mix(hl, ((uint64_t)j << 32) | (uint32_t)kj);
              const int e1 = m.netptr(j + 1);
              for (int e = m.netptr(j); e < e1; ++e) {
                const uint32_t ne = m.net(e);
                SL(ent_lo(ne)) += (int64_t)kj * ent_hi_s16(ne);
              }
            }
          }
          if (bad) {
            status = PYST_TRAJ_SAMPLER;
            break;
          }
          bool neg = false, over = false;
          for (int i = 0; i < S; ++i) {
            const int64_t nx = (int64_t)XV(i) + SL(i);
            neg |= nx < 0;
            over |= nx > PYST_I32MAX;
          }
          if (over) {
            status = PYST_TRAJ_OVERFLOW;
            break;
          }
          if (!neg) {
            ok = true;
            break;
          }
          tau = __dmul_rn(tau, 0.5);
          retry++;
          if (retry > ra.max_leap_retries) {
            status = PYST_TRAJ_LEAP_RETRY;
            break;
          }
        }
        if (!ok) {
          done = true;
          break;
        }
        leap_q++;
        h = hl;
        const double tn = __dadd_rn(t, tau);
        while (tn >= m.time(f)) {
          const double frac = __ddiv_rn(__dsub_rn(m.time(f), t), tau);
          for (int k = 0; k < kappa; ++k) {
            const int i = m.out(k);
            const double inc = rint(__dmul_rn((double)SL(i), frac));
            store_sample(o, ita, k, f, XV(i) + (int)inc);
          }
          f++;
          if (f == ita) {
            done = true;
            break;
          }
        }
        for (int i = 0; i < S; ++i) XV(i) = (int)((int64_t)XV(i) + SL(i));
        events += fired;
        t = tn;
        if (done) break;
        continue;
      }
    }
    // ------------------------ one direct-method step -------------------
    steps++;
    n_ssa++;
    const uint4 w = next_block(rs);
    const double tau = __ddiv_rn(-pyst_log(u53(w.x, w.y)), a0);
    const double r = __dmul_rn(u53(w.z, w.w), a0);
    int sel = -1;
    bool found = false;
    if constexpr (WIDE) {
      if (rate_sum_usable(a0)) {
        // the first segment whose end reaches r (r <= a0, the last end),
        // then the first reaction in it, from the sum at its start
        int s = 0;
        double cum = 0.0;
#pragma unroll
        for (int q = 0; q < kSegs - 1; ++q)
          if (P[q] < r) {
            s = q + 1;
            cum = P[q];
          }
        const int j1 = (s + 1) * seg < R ? (s + 1) * seg : R;
        for (int j = s * seg; j < j1; ++j) {
          cum = add_rate(cum, prop(j));
          if (cum >= r) {
            sel = j;
            break;
          }
        }
        found = true;
      }
    }
    if (!found) {
      double cum = 0.0;
      int lastnz = -1;
      for (int j = 0; j < R; ++j) {
        const float aj = prop(j);
        cum = __dadd_rn(cum, (double)aj);
        if (aj > 0.0f) lastnz = j;
        if (cum >= r) {
          sel = j;
          break;
        }
      }
      if (sel < 0) sel = lastnz;
    }
    const double tn = __dadd_rn(t, tau);
    while (tn >= m.time(f)) {
      for (int k = 0; k < kappa; ++k) store_sample(o, ita, k, f, XV(m.out(k)));
      f++;
      if (f == ita) {
        done = true;
        break;
      }
    }
    t = tn;
    if (done) break;
    if (sel >= 0) {  // (as thread_round's)
      const int e1 = m.netptr(sel + 1);
      bool over = false;
      for (int e = m.netptr(sel); e < e1; ++e) {
        const uint32_t ne = m.net(e);
        const int sp = ent_lo(ne);
        const int64_t nx = (int64_t)XV(sp) + ent_hi_s16(ne);
        if (nx < 0 || nx > PYST_I32MAX) over = true;
        else XV(sp) = (int)nx;
      }
      if (over) {
        status = PYST_TRAJ_OVERFLOW;
        done = true;
        break;
      }
    }
    events++;
    h = seq_mix(h, (uint64_t)sel);
    if (TAU) {
      if (--ssa_left <= 0) ssa_mode = false;
    }
  }
  st.t = t;
  st.n = rs.n;
  st.events = events;
  st.steps = steps;
  st.h = h;
  st.f = f;
  st.leap_q = leap_q;
  st.ssa_left = ssa_left;
  st.flags = (ssa_mode ? TS_SSA : 0) | (leap_grp ? TS_LEAPGRP : 0) |
             (done ? TS_DONE : 0) | (fill_state ? TS_FILL : 0) |
             (status << 8);
#undef XV
#undef SL
}

// thread_round for MAXR > 0 (register arrays), thread_round_big for 0; PK,
// GROUP and RX as thread_round's
template <int MAXR, bool TAU, bool SCORE, int PK = kPkRuntime,
          int GROUP = kGroupAny, int RX = 0, int FC = 0>
__device__ __forceinline__ void any_round(
    const ModelView& m, int32_t* xcol, int64_t* slot, int bs, int ss,
    const RunArgs& ra, uint64_t traj_id, TState& st, double* integ, int* cnt,
    const TrajOut& o, int cap_ssa, int cap_leap, bool stop_on_switch) {
  if constexpr (MAXR == 0) {
    static_assert(!SCORE, "the large-R thread engine keeps no scores");
    thread_round_big<TAU, false>(m, xcol, slot, bs, ss, ra, traj_id, st, o,
                                 cap_ssa, cap_leap, stop_on_switch);
  } else {
    thread_round<MAXR, TAU, SCORE, PK, 1, GROUP, RX, FC>(
        m, xcol, slot, bs, ss, ra, traj_id, st, integ, cnt, o, cap_ssa,
        cap_leap, stop_on_switch);
  }
}

template <bool TAU>
__device__ void run_thread_big(const ModelView& m, int32_t* xcol,
                               int64_t* slot, int bs, const RunArgs& ra,
                               uint64_t traj_id, const TrajOut& o) {
  TState st;
  thread_init<TAU>(m, xcol, bs, st);
  if (m.fw)
    thread_round_big<TAU, true>(m, xcol, slot, bs, bs, ra, traj_id, st, o,
                                0x7fffffff, 0x7fffffff, false);
  else
    thread_round_big<TAU, false>(m, xcol, slot, bs, bs, ra, traj_id, st, o,
                                 0x7fffffff, 0x7fffffff, false);
  thread_finish<1, false>(m, xcol, bs, st, nullptr, nullptr, o);
}

// ===================================================================
// one trajectory per warp
// ===================================================================
// Per-warp shared memory: x[S] int32, a[R] float, slot[S] 8 bytes,
// K[R] int32, crit[R] uint8 (rounded up to 4).  Lane l owns reactions
// [l*c, min(R,(l+1)*c)) with c = ceil(R/32); it owns species l, l+32, ...
struct WarpSmem {
  int32_t* x;
  float* a;
  int64_t* slot;
  int32_t* K;
  uint8_t* crit;
};

__device__ __forceinline__ size_t warp_smem_bytes(int S, int R) {
  size_t b = (size_t)S * 8 + (size_t)S * 4 + (size_t)R * 4 + (size_t)R * 4 +
             (((size_t)R + 3) & ~(size_t)3);
  return (b + 15) & ~(size_t)15;
}

__device__ __forceinline__ WarpSmem warp_smem(void* base, int S, int R) {
  WarpSmem w;
  char* p = (char*)base;
  w.slot = (int64_t*)p;
  p += (size_t)S * 8;
  w.x = (int32_t*)p;
  p += (size_t)S * 4;
  w.a = (float*)p;
  p += (size_t)R * 4;
  w.K = (int32_t*)p;
  p += (size_t)R * 4;
  w.crit = (uint8_t*)p;
  return w;
}

// Kogge-Stone inclusive scan of lane partial sums (FP64).  The oracle's
// warp mode repeats exactly these additions.
__device__ __forceinline__ double warp_incl_scan(double v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double n = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v = __dadd_rn(n, v);
  }
  return v;
}

// Select within lane prefixes: first lane L with p_L > 0 and incl_L >= r
// (fallback: last lane with p > 0); inside L, with r' = r - (incl_L - p_L),
// the first owned j whose running sum reaches r' (fallback: last owned j
// with a_j > 0).  Returns j on every lane.
__device__ __forceinline__ int warp_select(const float* a, double part,
                                          double incl, double r, int j0,
                                          int j1, int lane,
                                          const uint8_t* mask) {
  const unsigned hit = __ballot_sync(0xffffffffu, part > 0.0 && incl >= r);
  const unsigned nz = __ballot_sync(0xffffffffu, part > 0.0);
  const int L = hit ? (__ffs(hit) - 1) : (31 - __clz(nz));
  int sel = -1;
  if (lane == L) {
    const double rr = __dsub_rn(r, __dsub_rn(incl, part));
    double cum = 0.0;
    if (!mask && rate_sum_usable(part)) {
      // the sums do not decrease, so the first that reaches rr comes after
      // as many as do not reach it: no exit, the loads and sums overlap
      // (rr is NaN when another lane's sum is infinite or NaN: none reaches)
      int below = j0;
#pragma unroll 4
      for (int j = j0; j < j1; ++j) {
        cum = add_rate(cum, a[j]);
        below += cum >= rr ? 0 : 1;
      }
      if (below < j1) sel = below;
      cum = 0.0;
    }
    int lastnz = -1;
    if (sel < 0) for (int j = j0; j < j1; ++j) {
      if (mask && !mask[j]) continue;
      const float aj = a[j];
      cum = __dadd_rn(cum, (double)aj);
      if (aj > 0.0f) lastnz = j;
      if (cum >= rr) {
        sel = j;
        break;
      }
    }
    if (sel < 0) sel = lastnz;
  }
  return __shfl_sync(0xffffffffu, sel, L);
}

template <bool TAU, bool SCORE>
__device__ void run_warp(const ModelView& m, const WarpSmem& ws,
                         const RunArgs& ra, uint64_t traj_id, const TrajOut& o,
                         double* score_acc /* per-warp [R] or null */) {
  const int S = m.S, R = m.R, ita = m.ita, kappa = m.kappa;
  const int lane = threadIdx.x & 31;
  const int c = (R + 31) >> 5;
  const int j0 = min(R, lane * c), j1 = min(R, j0 + c);
  for (int i = lane; i < S; i += 32) ws.x[i] = m.x0(i);
  if (SCORE)
    for (int j = lane; j < 2 * R; j += 32) score_acc[j] = 0.0;
  __syncwarp();
  Stream rs = make_stream(ra.seed, traj_id);
  double t = 0.0;
  int f = 0;
  int64_t events = 0, steps = 0;
  uint64_t h = PYST_FNV_OFFSET;
  int status = PYST_TRAJ_DONE;
  bool fill_state = false;
  const double t_end = m.time(ita - 1);
  double tf = m.time(0);  // next sample time (f < ita while running)
  bool ssa_mode = !TAU;
  int ssa_left = 0;
  uint32_t leap_q = 0;
  // lane g holds the exponential variate and uniform of main-stream block
  // vb + g, so the random block and logarithm of a step (500 cycles) are not
  // on its chain; off is the next block's lane
  uint64_t vb = 0;
  int off = 0;
  double e_l = 0.0, u_l = 0.0;
  auto fill_variates = [&]() {
    rs.n = vb + (uint64_t)lane;
    const uint4 w = next_block(rs);
    e_l = -pyst_log(u53(w.x, w.y));
    u_l = u53(w.z, w.w);
  };
  fill_variates();
  auto take_variates = [&](double& e, double& u) {
    e = __shfl_sync(0xffffffffu, e_l, off);
    u = __shfl_sync(0xffffffffu, u_l, off);
    if (++off == 32) {
      off = 0;
      vb += 32;
      fill_variates();
    }
  };

  while (true) {
    double part = 0.0;
    bool bad_rate = false;
    if (m.fw) {  // (uniform)
#pragma unroll 4
      for (int j = j0; j < j1; ++j) {
        const float aj = propensity_wide_lanes(m.fw[j], ws.x);
        ws.a[j] = aj;
        part = add_rate(part, aj);
      }
      // an infinite or NaN propensity: plain conversions
      if (__any_sync(0xffffffffu, !(part < PYST_RATE_BIG))) {
        part = 0.0;
        for (int j = j0; j < j1; ++j)
          part = __dadd_rn(part, (double)ws.a[j]);
      }
    } else {
      for (int j = j0; j < j1; ++j) {
        const float aj = propensity(m, j, ws.x, 1);
        bad_rate |= !valid_rate(aj);
        ws.a[j] = aj;
        part = __dadd_rn(part, (double)aj);
      }
    }
    const double incl = warp_incl_scan(part, lane);
    const double a0 = __shfl_sync(0xffffffffu, incl, 31);
    __syncwarp();
    if (__any_sync(0xffffffffu, m.nlaw && bad_rate)) {
      status = PYST_TRAJ_RATE;
      break;
    }
    if (a0 == 0.0) {
      status = PYST_TRAJ_ABSORBED;
      fill_state = true;
      break;
    }
    if (steps >= ra.step_budget) {
      status = PYST_TRAJ_STEP_BUDGET;
      break;
    }
    if (TAU && !ssa_mode) {
      // critical flags for owned reactions
      for (int j = j0; j < j1; ++j) {
        uint8_t cf = 0;
        const int e1 = m.critptr(j + 1);
        for (int e = m.critptr(j); e < e1; ++e) {
          const uint32_t ce = m.crit(e);
          if ((int64_t)(ce >> 16) * m.n_c > (int64_t)ws.x[ent_lo(ce)]) cf = 1;
        }
        ws.crit[j] = cf;
      }
      __syncwarp();
      // mu, sigma^2 and the tau candidate per owned species
      float tmin = __int_as_float(0x7f800000);
      for (int i = lane; i < S; i += 32) {
        const uint32_t gw = m.g(i);
        if (!((gw >> 16) & 1u)) continue;
        float mu = 0.0f, s2 = 0.0f;
        const int e1 = m.spvptr(i + 1);
        for (int e = m.spvptr(i); e < e1; ++e) {
          const uint32_t se = m.spv(e);
          const int j = ent_lo(se);
          if (ws.crit[j]) continue;
          const int v = ent_hi_s16(se);
          mu = __fadd_rn(mu, __fmul_rn((float)v, ws.a[j]));
          s2 = __fadd_rn(s2, __fmul_rn((float)(v * v), ws.a[j]));
        }
        const float cnd = tau_candidate(m.eta, gw, ws.x[i], mu, s2);
        if (cnd < tmin) tmin = cnd;
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        tmin = fminf(tmin, __shfl_xor_sync(0xffffffffu, tmin, d));
      const float tau1 = tmin;
      if ((double)tau1 < __ddiv_rn(10.0, a0)) {
        ssa_mode = true;
        ssa_left = ra.ssa_fallback_steps;
      } else {
        steps++;
        double pc = 0.0;
        for (int j = j0; j < j1; ++j)
          if (ws.crit[j]) pc = __dadd_rn(pc, (double)ws.a[j]);
        const double inc_c = warp_incl_scan(pc, lane);
        const double a0c = __shfl_sync(0xffffffffu, inc_c, 31);
        double tau2 = __longlong_as_double(0x7ff0000000000000ll);
        double uc = 0.0;
        if (a0c > 0.0) {
          double ec;
          take_variates(ec, uc);
          tau2 = __ddiv_rn(ec, a0c);
        }
        const double tau1d = (double)tau1;
        double tau = (tau2 < tau1d) ? tau2 : tau1d;
        int kcrit = -1;
        if (tau1d > tau2) {
          const double r = __dmul_rn(uc, a0c);
          kcrit = warp_select(ws.a, pc, inc_c, r, j0, j1, lane, ws.crit);
        }
        int retry = 0;
        bool ok = false;
        while (true) {
          bool bad = false;
          for (int j = j0; j < j1; ++j) {
            int kj = 0;
            if (ws.crit[j]) {
              kj = (j == kcrit) ? 1 : 0;
            } else {
              const float lam = __fmul_rn(ws.a[j], (float)tau);
              const int k = poisson(lam, leap_key(rs, leap_q, j, retry));
              if (k < 0) bad = true;
              kj = k < 0 ? 0 : k;
            }
            ws.K[j] = kj;
          }
          for (int i = lane; i < S; i += 32) ws.slot[i] = 0;
          __syncwarp();
          if (__any_sync(0xffffffffu, bad)) {
            status = PYST_TRAJ_SAMPLER;
            break;
          }
          // species-major accumulation of V K (lane owns species)
          bool neg = false, over = false;
          for (int i = lane; i < S; i += 32) {
            int64_t d = 0;
            const int e1 = m.spvptr(i + 1);
            const uint32_t gw = m.g(i);
            (void)gw;
            for (int e = m.spvptr(i); e < e1; ++e) {
              const uint32_t se = m.spv(e);
              d += (int64_t)ws.K[ent_lo(se)] * ent_hi_s16(se);
            }
            ws.slot[i] = d;
            const int64_t nx = (int64_t)ws.x[i] + d;
            neg |= nx < 0;
            over |= nx > PYST_I32MAX;
          }
          __syncwarp();
          if (__any_sync(0xffffffffu, over)) {
            status = PYST_TRAJ_OVERFLOW;
            break;
          }
          if (!__any_sync(0xffffffffu, neg)) {
            ok = true;
            break;
          }
          tau = __dmul_rn(tau, 0.5);
          retry++;
          if (retry > ra.max_leap_retries) {
            status = PYST_TRAJ_LEAP_RETRY;
            break;
          }
        }
        if (!ok) break;
        leap_q++;
        const double tn = __dadd_rn(t, tau);
        // firing count and hash (lane 0 walks K in order)
        int64_t fired = 0;
        for (int j = j0; j < j1; ++j) {
          fired += ws.K[j];
          if (SCORE) {
            score_acc[j] = __dadd_rn(score_acc[j], (double)ws.K[j]);
          }
        }
        if (SCORE) {
          for (int j = j0; j < j1; ++j) {
            // integral term kept in a separate pass of the same slot
            score_acc[R + j] =
                __dadd_rn(score_acc[R + j], __dmul_rn((double)ws.a[j], tau));
          }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
          fired += __shfl_xor_sync(0xffffffffu, fired, d);
        if (lane == 0) {
          h = seq_mix(h, PYST_LEAP_TAG);
          for (int j = 0; j < R; ++j)
            if (ws.K[j] != 0)
              h = seq_mix(h, ((uint64_t)j << 32) | (uint32_t)ws.K[j]);
        }
        bool done = false;
        while (tn >= tf) {
          const double frac = __ddiv_rn(__dsub_rn(tf, t), tau);
          for (int k = lane; k < kappa; k += 32) {
            const int i = m.out(k);
            const double inc = rint(__dmul_rn((double)ws.slot[i], frac));
            store_sample(o, ita, k, f, ws.x[i] + (int)inc);
          }
          f++;
          if (f == ita) {
            done = true;
            break;
          }
          tf = m.time(f);
        }
        __syncwarp();
        for (int i = lane; i < S; i += 32)
          ws.x[i] = (int)((int64_t)ws.x[i] + ws.slot[i]);
        __syncwarp();
        events += fired;
        t = tn;
        if (done) break;
        continue;
      }
    }
    // ------------------------ one direct-method step -------------------
    steps++;
    double e, uu;
    take_variates(e, uu);
    const double tau = __ddiv_rn(e, a0);
    const double r = __dmul_rn(uu, a0);
    const int sel = warp_select(ws.a, part, incl, r, j0, j1, lane, nullptr);
    // (an unselected step changes nothing, as in thread_round)
    const int ne0 = sel >= 0 ? m.netptr(sel) : 0;
    const int ne1 = sel >= 0 ? m.netptr(sel + 1) : 0;
    const double tn = __dadd_rn(t, tau);
    if (SCORE) {
      const double dt = (tn >= t_end) ? __dsub_rn(t_end, t) : tau;
      for (int j = j0; j < j1; ++j)
        score_acc[R + j] =
            __dadd_rn(score_acc[R + j], __dmul_rn((double)ws.a[j], dt));
    }
    bool done = false;
    if (tn >= tf) {
      do {
        for (int k = lane; k < kappa; k += 32)
          store_sample(o, ita, k, f, ws.x[m.out(k)]);
        f++;
        if (f == ita) {
          done = true;
          break;
        }
        tf = m.time(f);
      } while (tn >= tf);
      __syncwarp();  // the counts are read before they change
    }
    t = tn;
    if (done) break;
    bool over = false;
    // a reaction changes each species once: one entry per lane
    for (int e = ne0 + lane; e < ne1; e += 32) {
      const uint32_t ne = m.net(e);
      const int sp = ent_lo(ne);
      const int nx = (int)((uint32_t)ws.x[sp] + (uint32_t)ent_hi_s16(ne));
      if (nx < 0) over = true;
      else ws.x[sp] = nx;
    }
    if (SCORE && lane == 0 && sel >= 0)
      score_acc[sel] = __dadd_rn(score_acc[sel], 1.0);
    __syncwarp();
    if (__any_sync(0xffffffffu, over)) {
      status = PYST_TRAJ_OVERFLOW;
      break;
    }
    events++;
    h = seq_mix(h, (uint64_t)sel);
    if (TAU) {
      if (--ssa_left <= 0) ssa_mode = false;
    }
  }
  __syncwarp();
  for (; f < ita; ++f)
    for (int k = lane; k < kappa; k += 32)
      store_sample(o, ita, k, f, fill_state ? ws.x[m.out(k)] : -1);
  if (lane == 0) {
    if (o.status) *o.status = (uint8_t)status;
    if (o.events) *o.events = events;
    if (o.seqhash) *o.seqhash = h;
    if (o.t_final) *o.t_final = t;
  }
  if (SCORE && o.score) {
    __syncwarp();
    for (int j = lane; j < R; j += 32)
      o.score[j] = __dsub_rn(score_acc[j], score_acc[R + j]);
  }
  __syncwarp();
}

}  // namespace pyst
