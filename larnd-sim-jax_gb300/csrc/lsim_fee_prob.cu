// Probabilistic self-trigger front end: the beam search of
// get_adc_values_average_noise_vmap (src/larndsim/fee_jax.py:386-461) with
// its step _find_one_hit_step (:334-384) and log_diff_ndtr (:33-53), plus
// the per-hit reductions of get_average_hit_values (:463-480).
//
// One 512-thread block per pixel (persistent over pixels).  The block keeps
// the pixel's cumulative charge q, its running maximum and its suffix
// maximum in shared memory; because max(x - c) = max(x) - c holds exactly
// in floating point, the per-path running maxima of q - c are read from the
// two shared arrays instead of being rescanned for each of the K paths.
// Ticks whose inputs are bit-identical to the previous tick's are grouped
// into classes (one evaluation per class; flat stretches of a waveform
// collapse).  For each of the H hit steps the block evaluates the paths whose
// charge is new and every thread folds its classes' values of the K paths
// into three online log-sum-exp accumulators (hit, total, selection).  A
// block top-K over the selection values (largest first, lower tick first on ties, as lax.top_k)
// gives the next K paths.  The reference stops the whole batch once no pixel
// keeps a total path probability above stop_threshold; the step kernel
// records per step whether any pixel stayed active and a second kernel
// blanks the steps the reference would not have run.
#include "lsim_internal.cuh"
#include "lsim_fee.cuh"

namespace lsim {
namespace {

constexpr int kProbThreads = 512;
constexpr int kProbTicks = 4;   // ticks per thread: up to 2048 ticks
constexpr int kProbMaxT = kProbThreads * kProbTicks;
constexpr int kProbMaxPaths = 32;
constexpr int kProbArrays = 10;  // q, running max, suffix max, esperance, soft-where weight, 3 class values, class, representative
// plus 6 partial sums per thread and the per-warp top-K candidates (value, index)
constexpr int kProbExtraFloats = 6 * kProbThreads + 2 * (kProbThreads / 32) * kProbMaxPaths + kProbMaxT;
static_assert(6 * kProbThreads >= kProbMaxT, "the path-group partials hold one tick array");
constexpr float kProbFloor = -1000.0f;

// ---------------------------------------------------------------- special functions
// jax.scipy.special.ndtr / log_ndtr in float32 (the published piecewise
// form: erf near zero and erfc in the tails for ndtr; -ndtr(-x) above 5,
// log(ndtr(x)) down to -10, the order-3 asymptotic series below).
// log_ndtr below 15 is called, not inlined: inlined at every call site of the
// per-path loops its erf/erfc/log body overflowed the instruction cache (the
// beam search ran 2.0x and its adjoint 2.2x slower, with identical results).
// What surrounds it is inlined: the largest arguments, which need nothing, do
// not pay for a call.  Lanes differ in their branches, so both signs share one
// ndtr and both directions of a log-sum-exp one exp.

__device__ __forceinline__ float ndtr_f(float x) {
  const float hs2 = 0.70710678118654752f;
  const float w = x * hs2;
  const float z = fabsf(w);
  const float y = z < hs2 ? 1.0f + erff(w) : (w > 0.0f ? 2.0f - erfcf(z) : erfcf(z));
  return 0.5f * y;
}

__device__ __noinline__ float log_ndtr_below_15(float x) {
  if (x > -10.0f) {
    const float n = ndtr_f(x > 5.0f ? -x : x);
    return x > 5.0f ? -n : logf(n);
  }
  const float x2 = x * x;
  const float log_scale = (-(x2 / 2.0f) - logf(-x)) - 0.918938533204672742f;   // 0.5 log(2 pi)
  const float x4 = x2 * x2;
  const float x6 = x4 * x2;
  const float odd = 1.0f / x2 + 15.0f / x6;
  const float even = 3.0f / x4;
  return log_scale + logf((1.0f + even) - odd);
}

// above 15, erfc(x / sqrt 2) < 1e-50 is 0 in float32: -ndtr(-x) = -0
__device__ __forceinline__ float log_ndtr_f(float x) { return x > 15.0f ? -0.0f : log_ndtr_below_15(x); }

// jax.nn.softplus = logaddexp(y, 0) = max(y, 0) + log1p(exp(-|y|)).  For
// |y| > 110 exp(-|y|) is 0 in float32, so the value is exactly max(y, 0).
__device__ __forceinline__ float softplus_f(float y) {
  if (fabsf(y) > 110.0f) return fmaxf(y, 0.0f);
  return fmaxf(y, 0.0f) + log1pf(expf(-fabsf(y)));
}

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// The clamped log(1 - exp(safe)) term of log_diff_ndtr.
__device__ __forceinline__ float ldn_log_term(float safe) {
  const float neg = -expm1f(safe);
  const float neg_safe = 1e-30f + softplus_f((neg - 1e-30f) * 1e10f) / 1e10f;
  // neg_safe >= 1e-30, so lt >= -69.1 and the clamp's softplus argument
  // (lt + 100) * 10 >= 309: softplus is the identity there
  const float lt = logf(neg_safe);
  return -100.0f + ((lt + 100.0f) * 10.0f) / 10.0f;
}

// log(Phi(a) - Phi(b)) with the reference's smooth clamps; la, lb =
// log_ndtr(a), log_ndtr(b); term_m1 = ldn_log_term(-1), the value every
// a <= b takes (safe = -1 there), so flat stretches (a == b, w = 1/2 exactly)
// need no transcendental function at all.
__device__ __forceinline__ float log_diff_ndtr_f(float a, float b, float la, float lb, float term_m1) {
  if (a == b) return 0.5f * (la + term_m1) + 0.5f * kProbFloor;
  const float lts = a > b ? ldn_log_term(lb - la) : term_m1;
  const float lp = la + lts;
  if ((a - b) * 1000.0f > 20.0f) return lp;     // the gate is 1 in float32 (1 + e^-20)
  const float w = sigmoid_f((a - b) * 1000.0f);
  return w * lp + (1.0f - w) * kProbFloor;
}

// online log-sum-exp: m = running maximum, s = sum of exp(x - m)
// (exp of arguments below -110 is 0 in float32)
__device__ __forceinline__ void lse_add(float &m, float &s, float x) {
  const float d = x - m;
  const float e = fabsf(d) < 110.0f ? expf(-fabsf(d)) : 0.0f;   // one for both directions: lanes differ
  if (d > 0.0f) {
    s = s * e + 1.0f;
    m = x;
  } else {
    s += e;
  }
}

__device__ __forceinline__ float lse_final(float m, float s) { return logf(s) + m; }

// merge a partial (m2, s2) into (m, s)
__device__ __forceinline__ void lse_merge(float &m, float &s, float m2, float s2) {
  if (!(s2 > 0.0f)) return;
  if (!(s > 0.0f)) {
    m = m2;
    s = s2;
    return;
  }
  if (m2 > m) {
    s = (m - m2 > -110.0f ? s * expf(m - m2) : 0.0f) + s2;
    m = m2;
  } else if (m2 - m > -110.0f) {
    s += s2 * expf(m2 - m);
  }
}

// floats (no NaN) as unsigned integers in the same order, 0 below them all
__device__ __forceinline__ unsigned order_key(float x) { return (unsigned)float_key(x) ^ 0x80000000u; }
__device__ __forceinline__ float key_order(unsigned k) { return key_float((int)(k ^ 0x80000000u)); }

// ---------------------------------------------------------------- block scans over a pixel row

// in-place inclusive scan of a[0..n) with op (sum, max) or a suffix max;
// each thread scans a contiguous chunk of kProbTicks, warps and the block
// combine the chunk totals.
enum ScanOp { kScanSum = 0, kScanMax = 1, kScanSuffixMax = 2, kScanSuffixSum = 3 };

template <int OP>
__device__ void block_scan_row(float *a, int n, float *red) {
  constexpr bool SUFFIX = OP == kScanSuffixMax || OP == kScanSuffixSum;
  constexpr bool SUM = OP == kScanSum || OP == kScanSuffixSum;
  const float ident = SUM ? 0.0f : -INFINITY;
  auto comb = [](float x, float y) { return SUM ? x + y : fmaxf(x, y); };
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  float v[kProbTicks];
  // suffix scans walk each thread's chunk from the right, thread 0 holding the last chunk
  const int base = SUFFIX ? n - (tid + 1) * kProbTicks : tid * kProbTicks;
  float run = ident;
#pragma unroll
  for (int i = 0; i < kProbTicks; ++i) {
    const int t = SUFFIX ? base + kProbTicks - 1 - i : base + i;
    const bool ok = t >= 0 && t < n;
    const float x = ok ? a[t] : ident;
    run = comb(run, x);
    v[i] = run;
  }
  // exclusive prefix of the chunk totals across the block
  float incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl = comb(incl, y);
  }
  if (lane == 31) red[wid] = incl;
  __syncthreads();
  float carry = ident;
  for (int w = 0; w < wid; ++w) carry = comb(carry, red[w]);
  float ex = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) ex = ident;
  const float pre = comb(carry, ex);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kProbTicks; ++i) {
    const int t = SUFFIX ? base + kProbTicks - 1 - i : base + i;
    if (t >= 0 && t < n) a[t] = comb(pre, v[i]);
  }
  __syncthreads();
}

__device__ __forceinline__ float block_sum(float v, float *red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  float t = 0.0f;
#pragma unroll
  for (int w = 0; w < kProbThreads / 32; ++w) t += red[w];
  return t;
}

// What a record was made from, kept with it: the adjoint compares it with its
// own call (on the device: the host does not wait for the forward).
struct ProbMark {
  int64_t n_pix;
  int32_t T, K, H;
  int32_t all_steps;      // every tick, path and step is in it: serves cotangents on the distributions
};

struct ProbArgs {
  LsimParams p;
  const float *wfs;
  int64_t n_pix;
  int T, K, interval;
  float z, thr, log_stop;
  float *log_prob, *charge, *e_tick, *e_adc, *lam;
  unsigned long long *work;   // pixels handed out beyond the blocks' first
  int32_t *step_active;   // [H]: some pixel kept a total path probability above the stop level after step h
  float *cache;           // [blocks][K][kCacheArrays][cache_row]: path values kept from step to step
  int cache_row;          // floats per row of the cache, at least T - 1
  bool all_steps;         // run every step even when nothing can come of it
  // record for the adjoint (all or none):
  ProbMark *mark;
  float *state;           // [n_pix][H][2][K]: each step's input path charges and log-probabilities
  int32_t *state_top;     // [n_pix][H][K]: each step's selected ticks
  uint32_t *live;         // [n_pix][H][kLiveWords]: ticks whose probability is not 0
  int32_t *n_run;         // [n_pix]: steps run, kWildRow added for a row that the adjoint takes apart
  float *red;             // [3][n_pix][H]: expected tick and ADC, total probability
};

constexpr int kCacheArrays = 3;               // per path: dist, selection and hit value of each class
constexpr float kNoHit = 2.0f;                // a hit value (never above 0) that has not been formed yet
constexpr int kLiveWords = kProbMaxT / 32;
// exp of anything below is 0 in float32 (half of the smallest denormal is e^-103.97)
constexpr float kProbDead = -104.0f;
// a path's hit term below this leaves a log-sum-exp above kProbDead as it is:
// 32 terms of e^-26 next to 1 are below its rounding
constexpr float kProbFar = kProbDead - 26.0f;
// The adjoint's partials are finite for arguments up to kWildArgument (the derivative of log_ndtr is exp of a difference
// that rounds by less than 10 there); rows beyond are marked.
constexpr float kWildArgument = 1e4f;
constexpr int32_t kWildRow = 1 << 16;
static_assert(LSIM_MAX_HITS < kWildRow, "steps and mark");
// log_diff_ndtr(a, b) <= -1000 sigmoid(-1000 (a - b)): below -1000 sigmoid(-1.4) = -197.8 for a - b < 1.4e-3
constexpr float kWeakRise = 1.4f, kWeakMost = -190.0f;

// The per-tick work of a step reads, for tick t, only the running maximum
// at t and t+1, q at t, t+1, s = shifted(t) and s+1, and the suffix maximum
// at the selection window end.  Ticks whose 7 values are bit-identical to
// those of the tick before give bit-identical results, so the block
// evaluates one representative per run of equal ticks (a "class") and
// expands the class values back to ticks; flat stretches of a waveform
// (no charge arriving) collapse to a handful of classes.
//
// What a path adds to a class depends on its charge alone (its probability
// enters the log-sum-exps), and two thirds of a pixel's paths carry a charge
// that a path of the step before carried (after the last real hit the top-K
// ticks hardly change).  So the values of a path are kept in the block's
// scratch for as long as some path has its charge: a step evaluates new
// charges only and then folds the K paths' kept values, in the order and with
// the operations of an evaluation in place.  The scratch is global memory:
// the values-only form uses 10 to 30 % of it, which stays in L2; with the
// distributions of dense 2000-tick rows it is 20 x 3 x 2000 floats a block,
// 146 MB over 304 blocks, and does not fit in the 129 MB.
//
// Without the distributions (kDist false) a value matters only where its
// probability does not underflow, and the rest is left out exactly:
// * a tick on which the running maximum rises by less than kWeakRise / 1000
//   noise widths has dist terms below kWeakMost for every path (the smooth
//   gate's floor), so only the classes of the other ticks, 10 to 30 % of them,
//   are evaluated; a path selected on such a tick could add nothing that
//   float32 keeps.  Where fewer than K ticks are left, the paths that are
//   missing repeat the best path's charge at the floor's probability, as the
//   first step's do, and are skipped.  Should a tick with a likely dist value
//   have to compete with the ticks left out (its own selection value is below
//   theirs could be), the pixel starts over with all classes;
// * hit <= dist, so the hit terms are formed only for the (class, path) pairs
//   whose dist term is above kProbFar;
// * a pixel whose paths have all become improbable beyond kProbDead stops.
// Bound by instruction issue in the special functions.  Values and gradient of
// 1500 dense rows: 42.4 -> 6.1 ms (10.1 before the adjoint below); distributions of 1000 rows: 8.8 -> 5.0 ms.
template <bool kDist>
__global__ void __launch_bounds__(kProbThreads, 2) k_fee_prob(ProbArgs a) {
  extern __shared__ __align__(16) float sm[];
  float *qs = sm, *cm = qs + kProbMaxT, *cr = cm + kProbMaxT, *esp = cr + kProbMaxT, *sw = esp + kProbMaxT;
  float *vh = sw + kProbMaxT, *vd = vh + kProbMaxT, *vs = vd + kProbMaxT;
  int *cls = reinterpret_cast<int *>(vs + kProbMaxT), *rep = cls + kProbMaxT;
  float *part = reinterpret_cast<float *>(rep + kProbMaxT);   // [kProbThreads][6] partial sums of path groups
  unsigned *cand_k = reinterpret_cast<unsigned *>(part + 6 * kProbThreads);   // [warps][K] per-warp top-K lists
  int *cand_i = reinterpret_cast<int *>(cand_k + (kProbThreads / 32) * kProbMaxPaths);
  // per-tick log_ndtr of the running maximum and of q for one path, shared by
  // neighbouring classes on dense pixels (the path-group partials, unused
  // then, hold the first)
  float *lmv = part, *lqv = reinterpret_cast<float *>(cand_i + (kProbThreads / 32) * kProbMaxPaths);
  __shared__ float red[kProbThreads / 32];
  __shared__ float pc[kProbMaxPaths], plp[kProbMaxPaths], nc[kProbMaxPaths], nlp[kProbMaxPaths];
  __shared__ int pskip[kProbMaxPaths];
  __shared__ float slot_c[kProbMaxPaths];       // charge whose values a slot of the scratch holds
  __shared__ int path_slot[kProbMaxPaths], fresh[kProbMaxPaths];
  __shared__ int n_cls, n_all, n_fresh, n_slots, stop, again;
  __shared__ int64_t next_pix;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;

  const LsimParams &p = a.p;
  const int T = a.T, K = a.K, H = p.max_adc_values, tid = threadIdx.x;
  const float z = a.z, thr = a.thr;
  const float term_m1 = ldn_log_term(-1.0f);
  const float log_k = logf((float)K) + 1e-3f;
  float *cache = a.cache + (size_t)blockIdx.x * K * kCacheArrays * a.cache_row;
  auto kept = [&](int slot, int what) { return cache + (size_t)(slot * kCacheArrays + what) * a.cache_row; };
  auto shifted = [&](int t) { return min(t + a.interval + 1, T - 1); };
  // the hit term of a path at tick t from its two log_ndtr values and its dist term
  auto hit_term = [&](int t, float zqs, float zq0, float LQs, float LQ0, float lg) {
    float le = log_diff_ndtr_f(zqs, zq0, LQs, LQ0, term_m1);
    le = fminf(le, lg);
    le = kProbFloor + softplus_f(le - kProbFloor);
    return sw[t] * le + (1.0f - sw[t]) * kProbFloor;
  };

  bool leave_out = !kDist && !a.all_steps;
  if (a.mark && blockIdx.x == 0 && tid == 0) *a.mark = ProbMark{a.n_pix, T, K, H, leave_out ? 0 : 1};
  for (int64_t pix = blockIdx.x; pix < a.n_pix;) {
    const float *w = a.wfs + pix * T;
    for (int t = tid; t < T; t += kProbThreads) qs[t] = w[t] * p.t_sampling;
    __syncthreads();
    block_scan_row<kScanSum>(qs, T, red);
    for (int t = tid; t < T; t += kProbThreads) cm[t] = cr[t] = qs[t];
    __syncthreads();
    block_scan_row<kScanMax>(cm, T, red);
    block_scan_row<kScanSuffixMax>(cr, T, red);
    // rounding of (cm - c) - thr, times z, on both sides of a rise
    float most = fabsf(thr);
    if (!kDist || a.n_run) {
      float m = 0.0f;
      for (int t = tid; t < T; t += kProbThreads) m = fmaxf(m, isfinite(qs[t]) ? fabsf(qs[t]) : INFINITY);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) red[wid] = m;
      __syncthreads();
      for (int w2 = 0; w2 < kProbThreads / 32; ++w2) m = fmaxf(m, red[w2]);
      most += m;
      __syncthreads();
    }
    const bool partial = leave_out && isfinite(most);
    const bool wild = !(most * z < kWildArgument / 2);   // arguments are up to (2 max |q| + |thr|) z
    const float rise = kWeakRise - most * z * (12000.0f / 16777216.0f);
    // esperance values, soft-where weights and the tick classes
    for (int t = tid; t < T - 1; t += kProbThreads) {
      const int s = shifted(t);
      const float e = (qs[s] + thr) - 0.5f * (qs[t + 1] + qs[t]);
      esp[t] = e;
      sw[t] = sigmoid_f((e - thr) * 10.0f);
      bool head = t == 0;
      if (!head) {
        const int sp = shifted(t - 1);
        const int s1 = min(s + 1, T - 1), sp1 = min(sp + 1, T - 1);
        const int fe = min(s + a.interval + 1, T - 1), fep = min(sp + a.interval + 1, T - 1);
        auto ne = [](float x, float y) { return __float_as_uint(x) != __float_as_uint(y); };
        head = ne(cm[t], cm[t - 1]) || ne(cm[t + 1], cm[t]) || ne(qs[t], qs[t - 1]) || ne(qs[t + 1], qs[t]) ||
               ne(qs[s], qs[sp]) || ne(qs[s1], qs[sp1]) || ne(cr[fe], cr[fep]);
      }
      vh[t] = head ? 1.0f : 0.0f;
      if (!kDist) {   // heads of the classes that count (a class's ticks have one rise)
        const bool weak = partial && (cm[t + 1] - cm[t]) * z * 1000.0f < rise;
        vd[t] = weak ? 1.0f : 0.0f;
        vs[t] = head && !weak ? 1.0f : 0.0f;
      }
    }
    __syncthreads();
    block_scan_row<kScanSum>(vh, T - 1, red);   // integer counts, exact in float32
    if (!kDist) block_scan_row<kScanSum>(vs, T - 1, red);
    for (int t = tid; t < T - 1; t += kProbThreads) {
      const bool first = t == 0 || vh[t - 1] != vh[t];
      const int u = (int)(kDist ? vh[t] : vs[t]) - 1;
      const bool weak = !kDist && vd[t] != 0.0f;
      cls[t] = weak ? -1 : u;
      if (first && !weak) rep[u] = t;
      if (t == T - 2) {
        n_cls = u + 1;
        n_all = (int)vh[t];
      }
    }
    if (tid < K) {
      pc[tid] = 0.0f;
      plp[tid] = tid == 0 ? 0.0f : kProbFloor;
    }
    if (tid == 0) {
      n_slots = 0;
      stop = 0;
      again = 0;
    }
    __syncthreads();
    const int U = n_cls;
    // with few classes, G groups of threads share a class and split the paths
    // (by all classes' number: the order of a class's sum does not depend on what is left out)
    const int G = n_all <= kProbThreads / 2 ? min(8, kProbThreads / n_all) : 1;
    const int grp = G > 1 && U > 0 ? tid / U : 0;
    const int n_own = G > 1 ? (grp < G ? 1 : 0) : kProbTicks;
    const int r0 = G > 1 ? tid - grp * U : tid;
    // dense pixels: per path, log_ndtr at every tick (2 T calls) instead of
    // four per class (the running maximum at t + 1 and q at the shifted tick
    // are other ticks' values at t)
    const bool tick_mode = kDist && G == 1 && 2 * U > T;

    int h = 0;
    for (; h < H; ++h) {
      // paths whose charge repeats that of a path more than 110 log units
      // likelier add exp(< -110) = 0 to every float32 log-sum-exp: skip them
      if (wid == 0) {
        const float c = lane < K ? pc[lane] : 0.0f;
        if (lane < K) {
          int sk = 0;
          for (int j = 0; j < K; ++j)
            if (j != lane && pc[j] == c && plp[j] > plp[lane] + 110.0f) sk = 1;
          pskip[lane] = sk;
          if (a.state) {
            float *st = a.state + ((pix * H + h) * 2) * (int64_t)K;
            st[lane] = c;
            st[K + lane] = plp[lane];
          }
        }
        // slots: a charge that a slot holds keeps it, the others (one per
        // distinct charge) take the slots that are free
        const unsigned key = __float_as_uint(c);
        int slot = -1;
        for (int j = 0; j < n_slots; ++j)
          if (lane < K && __float_as_uint(slot_c[j]) == key) slot = j;
        const unsigned same = __match_any_sync(0xffffffffu, lane < K ? (unsigned long long)key
                                                                     : (1ull << 32) + (unsigned)lane);
        const int leader = __ffs(same) - 1;
        const unsigned used = __reduce_or_sync(0xffffffffu, slot >= 0 ? 1u << slot : 0u);
        const unsigned need = __ballot_sync(0xffffffffu, lane < K && slot < 0 && leader == lane);
        const int rank = __popc(need & ((1u << lane) - 1u));
        if ((need >> lane) & 1u) {
          unsigned free_slots = ~used;
          for (int j = 0; j < rank; ++j) free_slots &= free_slots - 1;
          slot = __ffs(free_slots) - 1;
          fresh[rank] = lane;
        }
        slot = __shfl_sync(0xffffffffu, slot, leader);
        __syncwarp();
        if (lane < K) {
          path_slot[lane] = slot;
          slot_c[slot] = c;
        }
        const int top = __reduce_max_sync(0xffffffffu, lane < K ? slot + 1 : 0);
        if (lane == 0) {
          n_fresh = __popc(need);
          n_slots = max(n_slots, top);   // a slot that is not in use keeps its charge's values until it is taken
        }
      }
      __syncthreads();
      // ---- the values of the charges that are new
      const int nf = n_fresh;
      auto evaluate = [&](int r, float c, float *kd, float *ks, float *kh) {
        const int t = rep[r];
        const int s = shifted(t);
        const float zm0 = ((cm[t] - c) - thr) * z, zm1 = ((cm[t + 1] - c) - thr) * z;
        const float LM0 = tick_mode ? lmv[t] : log_ndtr_f(zm0);
        const float LM1 = tick_mode ? lmv[t + 1] : (zm1 == zm0 ? LM0 : log_ndtr_f(zm1));
        const float lg = log_diff_ndtr_f(zm1, zm0, LM1, LM0, term_m1);
        kd[r] = lg;
        const int fe = min(s + a.interval + 1, T - 1);
        const float x = (((cr[fe] - c) - (qs[min(s + 1, T - 1)] - c)) - thr) * z;
        ks[r] = lg + log_ndtr_f(x);
        if (kDist) {
          const float zq0 = ((qs[t] - c) - thr) * z, zqs = ((qs[s] - c) - thr) * z;
          const float LQ0 = tick_mode ? lqv[t] : log_ndtr_f(zq0);
          const float LQs = tick_mode ? lqv[s] : (zqs == zq0 ? LQ0 : log_ndtr_f(zqs));
          kh[r] = hit_term(t, zqs, zq0, LQs, LQ0, lg);
        } else {
          kh[r] = kNoHit;
        }
      };
      if (kDist) {
        for (int f = grp; n_own > 0 && f < nf; f += G) {
          const int k = fresh[f];
          const float c = pc[k];
          float *kd = kept(path_slot[k], 0), *ks = kept(path_slot[k], 1), *kh = kept(path_slot[k], 2);
          if (tick_mode) {
            __syncthreads();   // the previous path's reads are done
            for (int t = tid; t < T; t += kProbThreads) {
              lmv[t] = log_ndtr_f(((cm[t] - c) - thr) * z);
              lqv[t] = log_ndtr_f(((qs[t] - c) - thr) * z);
            }
            __syncthreads();
          }
#pragma unroll
          for (int i = 0; i < kProbTicks; ++i) {
            const int r = r0 + i * kProbThreads;
            if (i < n_own && r < U) evaluate(r, c, kd, ks, kh);
          }
        }
      } else {
        // (path, class) pairs dealt over all threads
        int f = 0, r = tid;
        for (;; r += kProbThreads) {
          while (r >= U && f < nf) r -= U, ++f;
          if (f >= nf) break;
          const int k = fresh[f], slot = path_slot[k];
          evaluate(r, pc[k], kept(slot, 0), kept(slot, 1), kept(slot, 2));
        }
      }
      __syncthreads();
      // ---- the log-sum-exps over the paths
      float hm[kProbTicks], hs[kProbTicks], dm[kProbTicks], ds[kProbTicks], sm_[kProbTicks], ss[kProbTicks];
#pragma unroll
      for (int i = 0; i < kProbTicks; ++i) {
        hm[i] = dm[i] = sm_[i] = -INFINITY;
        hs[i] = ds[i] = ss[i] = 0.0f;
      }
      for (int k = grp; n_own > 0 && k < K; k += G) {
        if (pskip[k]) continue;
        const float c = pc[k], lp = plp[k];
        const float *kd = kept(path_slot[k], 0), *ks = kept(path_slot[k], 1);
        float *kh = kept(path_slot[k], 2);
        float lg[kProbTicks], lsel[kProbTicks], le[kProbTicks];
#pragma unroll
        for (int i = 0; i < kProbTicks; ++i) {
          const int r = r0 + i * kProbThreads;
          const bool ok = i < n_own && r < U;
          lg[i] = ok ? kd[r] : 0.0f;
          lsel[i] = ok ? ks[r] : 0.0f;
          le[i] = ok ? kh[r] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kProbTicks; ++i) {
          const int r = r0 + i * kProbThreads;
          if (i < n_own && r < U) {
            if (kDist) {
              lse_add(hm[i], hs[i], le[i] + lp);
            } else if (!(lg[i] + lp < kProbFar)) {
              if (le[i] == kNoHit) {
                const int t = rep[r], s = shifted(t);
                const float zq0 = ((qs[t] - c) - thr) * z, zqs = ((qs[s] - c) - thr) * z;
                const float LQ0 = log_ndtr_f(zq0);
                const float LQs = zqs == zq0 ? LQ0 : log_ndtr_f(zqs);
                le[i] = hit_term(t, zqs, zq0, LQs, LQ0, lg[i]);
                kh[r] = le[i];
              }
              lse_add(hm[i], hs[i], le[i] + lp);
            }
            lse_add(dm[i], ds[i], lg[i] + lp);
            lse_add(sm_[i], ss[i], lsel[i] + lp);
          }
        }
      }
      if (G > 1) {
        // merge the path groups' partial log-sum-exps into group 0
        if (grp > 0 && grp < G) {
          float *q = part + 6 * tid;
          q[0] = hm[0], q[1] = hs[0], q[2] = dm[0], q[3] = ds[0], q[4] = sm_[0], q[5] = ss[0];
        }
        __syncthreads();
        if (grp == 0) {
          for (int g2 = 1; g2 < G; ++g2) {
            const float *q = part + 6 * (g2 * U + tid);
            lse_merge(hm[0], hs[0], q[0], q[1]);
            lse_merge(dm[0], ds[0], q[2], q[3]);
            lse_merge(sm_[0], ss[0], q[4], q[5]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kProbTicks; ++i) {
        const int r = r0 + i * kProbThreads;
        if (i < n_own && grp == 0 && r < U) {
          vh[r] = lse_final(hm[i], hs[i]);
          vd[r] = lse_final(dm[i], ds[i]);
          vs[r] = lse_final(sm_[i], ss[i]);
        }
      }
      __syncthreads();
      // step outputs and the per-hit reductions
      float l_sum = 0.0f, t_sum = 0.0f, a_sum = 0.0f;
      float selv[kProbTicks];
      unsigned left = 0u;     // this thread's ticks that are not in the selection
      const int64_t row = (pix * H + h) * (int64_t)(T - 1);
#pragma unroll
      for (int i = 0; i < kProbTicks; ++i) {
        const int t = tid + i * kProbThreads;
        selv[i] = -INFINITY;
        float pr = 0.0f;
        const int u = t < T - 1 ? cls[t] : -1;
        if (u < 0) left |= 1u << i;
        if (u >= 0) {
          const float hit = vh[u];
          selv[i] = vs[u];
          if (a.log_prob) a.log_prob[row + t] = hit;
          if (a.charge) a.charge[row + t] = esp[t];
          pr = expf(hit);
          l_sum += pr;
          t_sum += (float)t * pr;
          a_sum += digitize(p, esp[t]) * pr;
        }
        if (a.live) {   // NaN counts as live
          const unsigned bits = __ballot_sync(0xffffffffu, pr != 0.0f);
          if (lane == 0) a.live[(pix * H + h) * kLiveWords + i * (kProbThreads / 32) + wid] = bits;
        }
      }
      if (a.lam || a.red) {
        const float L = block_sum(l_sum, red);
        const float Ts = block_sum(t_sum, red);
        const float As = block_sum(a_sum, red);
        if (tid == 0) {
          const float den = fmaxf(L, 1e-10f), et = Ts / den, ea = As / den;
          const int64_t o = pix * H + h;
          if (a.lam) {
            a.lam[o] = L;
            a.e_tick[o] = et;
            a.e_adc[o] = ea;
          }
          if (a.red) {
            a.red[o] = et;
            a.red[a.n_pix * H + o] = ea;
            a.red[2 * a.n_pix * H + o] = L;
          }
        }
      }
      // top-K ticks by selection value -> next paths (largest first, lower tick
      // first on ties, NaN never): each warp lists the K best of its ticks,
      // then warp 0 merges the 16 lists.  The values are compared as ordered
      // integers, so a round is two warp reductions.
      {
        unsigned key[kProbTicks];
#pragma unroll
        for (int i = 0; i < kProbTicks; ++i)
          key[i] = (left >> i & 1u) || selv[i] != selv[i] ? 0u : order_key(selv[i]);
        unsigned mine_k = 0u;
        int mine_t = 0x7fffffff;
        for (int r = 0; r < K; ++r) {
          unsigned bk = 0u;
          int bi = 0;
#pragma unroll
          for (int i = 0; i < kProbTicks; ++i)
            if (key[i] > bk) {
              bk = key[i];
              bi = i;
            }
          const unsigned m = __reduce_max_sync(0xffffffffu, bk);
          if (m == 0u) break;
          const int t = tid + bi * kProbThreads;
          const int first = __reduce_min_sync(0xffffffffu, bk == m ? t : 0x7fffffff);
          if (t == first)
#pragma unroll
            for (int i = 0; i < kProbTicks; ++i)
              if (i == bi) key[i] = 0u;
          if (lane == r) {
            mine_k = m;
            mine_t = first;
          }
        }
        if (lane < K) {
          cand_k[wid * kProbMaxPaths + lane] = mine_k;
          cand_i[wid * kProbMaxPaths + lane] = mine_t;
        }
      }
      __syncthreads();
      if (wid == 0) {
        static_assert(kProbThreads / 32 <= 32, "a lane per list");
        const int base = lane * kProbMaxPaths;
        const bool list = lane < kProbThreads / 32;
        int at = 0, tt = 0x7fffffff;
        unsigned hk = list ? cand_k[base] : 0u, bv = 0u;
        int hi = list ? cand_i[base] : 0x7fffffff;
        for (int r = 0; r < K; ++r) {
          const unsigned m = __reduce_max_sync(0xffffffffu, hk);
          if (m == 0u) break;
          const int first = __reduce_min_sync(0xffffffffu, hk == m ? hi : 0x7fffffff);
          if (lane == r) {
            bv = m;
            tt = first;
          }
          if (hk == m && hi == first) {
            ++at;
            hk = at < K ? cand_k[base + at] : 0u;
            hi = at < K ? cand_i[base + at] : 0x7fffffff;
          }
        }
        // charge of the paths that are missing, and what a tick left out can at most be selected by
        const int best = __shfl_sync(0xffffffffu, tt, 0);
        const float miss_c = best < T - 1 ? qs[min(shifted(best) + 1, T - 1)] : 0.0f;
        float mp = lane < K ? plp[lane] : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, o));
        if (lane < K) {
          const bool have = tt < T - 1, real = have || !partial;
          if (!have) tt = T - 2;
          const float lp_new = real ? vd[cls[tt]] : kProbFloor;
          nlp[lane] = lp_new;
          nc[lane] = real ? qs[min(shifted(tt) + 1, T - 1)] : miss_c;
          if (partial && have && !(key_order(bv) > mp + log_k + kWeakMost) && !(lp_new < kProbFar)) again = 1;
          if (a.state_top) a.state_top[(pix * H + h) * (int64_t)K + lane] = tt;
        }
      }
      __syncthreads();
      if (tid < 32) {
        const float v = tid < K ? nlp[tid] : -INFINITY;
        float m = v;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float mm = isfinite(m) ? m : 0.0f;
        float sum = tid < K ? expf(v - mm) : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (tid < K) {
          pc[tid] = nc[tid];
          plp[tid] = nlp[tid];
        }
        if (tid == 0) {
          const float total = logf(sum) + mm;
          if (!again && total > a.log_stop && !*(volatile int32_t *)(a.step_active + h)) atomicOr(a.step_active + h, 1);
          // a step at most multiplies the total by K (its K ticks' dist values)
          stop = partial && total < kProbDead - 1.0f - log_k * (float)(H - 1 - h) ? 1 : 0;
        }
      }
      __syncthreads();
      if (again) break;
      if (stop) {
        ++h;
        break;
      }
    }
    if (again) {        // once more with every class
      leave_out = false;
      __syncthreads();
      continue;
    }
    if (a.n_run && tid == 0) a.n_run[pix] = h | (wild ? kWildRow : 0);
    // the steps that were not run: every probability is exactly 0
    for (int g = h + tid; g < H; g += kProbThreads)
      if (a.lam) {
        a.lam[pix * H + g] = 0.0f;
        a.e_tick[pix * H + g] = 0.0f;
        a.e_adc[pix * H + g] = 0.0f;
      }
    leave_out = !kDist && !a.all_steps;
    // pixels differ several times in cost: the next one by a counter
    if (tid == 0) next_pix = gridDim.x + (int64_t)atomicAdd(a.work, 1ull);
    __syncthreads();
    pix = next_pix;
  }
}

// Steps after the first one that left no pixel active were not run by the
// reference: their log-probabilities are -1000 and their charges 0, and so
// are the reductions (exp(-1000) = 0 in float32).
__global__ void k_fee_prob_mask(ProbArgs a, int H) {
  int first = H;
  for (int h = 1; h < H; ++h)
    if (!a.step_active[h - 1]) {
      first = h;
      break;
    }
  if (first >= H) return;
  const int64_t T1 = a.T - 1;
  const int64_t rows = a.n_pix * (int64_t)(H - first);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < rows * T1; e += stride) {
    const int64_t r = e / T1, t = e - r * T1;
    const int64_t pix = r / (H - first), h = first + r % (H - first);
    const int64_t o = (pix * H + h) * T1 + t;
    if (a.log_prob) a.log_prob[o] = kProbFloor;
    if (a.charge) a.charge[o] = 0.0f;
    if (t == 0 && a.lam) {
      a.lam[pix * H + h] = 0.0f;
      a.e_tick[pix * H + h] = 0.0f;
      a.e_adc[pix * H + h] = 0.0f;
    }
  }
}

// ---------------------------------------------------------------- adjoint
// Reverse mode through the beam search as jax.grad takes it: the top-K tick
// choices are held (lax.stop_gradient), jnp.where passes the cotangent to
// the selected branch, jnp.minimum to the smaller argument (half each at a
// tie), the running maximum to the tick where it was first attained, and
// softplus / sigmoid / log-sum-exp by their derivatives.

// d log_ndtr / dx as jax.scipy.special.log_ndtr defines it (a custom
// derivative, the same on every branch): exp(norm_logpdf(x) - log_ndtr(x))
__device__ __forceinline__ float dlog_ndtr_f(float x, float lx) {
  return expf((-0.5f * x * x - 0.918938533204672742f) - lx);
}

// log_diff_ndtr and its partials d/da, d/db (la = log_ndtr(a), lb = log_ndtr(b))
struct LogDiff {
  float lp, w, out;       // log term, gate, value
  float u, y, ns;         // of the log term where a > b
  __device__ __forceinline__ LogDiff(float a, float b, float la, float lb, float term_m1) {
    u = y = ns = 0.f;
    float lts = term_m1;
    if (a > b) {
      u = lb - la;
      const float neg = -expm1f(u);
      y = (neg - 1e-30f) * 1e10f;
      ns = 1e-30f + softplus_f(y) / 1e10f;
      const float lt = logf(ns);
      lts = -100.0f + ((lt + 100.0f) * 10.0f) / 10.0f;
    }
    lp = la + lts;
    w = sigmoid_f((a - b) * 1000.0f);
    out = w * lp + (1.0f - w) * kProbFloor;
  }
  __device__ __forceinline__ void partials(float a, float b, float la, float lb, float &ga, float &gb) const {
    const float dla = dlog_ndtr_f(a, la);
    const float gw = (lp - kProbFloor) * w * (1.0f - w) * 1000.0f;   // through the gate
    if (a > b) {
      // softplus' = sigmoid; d neg / du = -exp(u); the second clamp is the identity there
      const float dlts_du = (1.0f / ns) * sigmoid_f(y) * (-expf(u));
      ga = w * (dla - dlts_du * dla) + gw;
      gb = w * (dlts_du * dlog_ndtr_f(b, lb)) - gw;
    } else {
      ga = w * dla + gw;
      gb = -gw;
    }
  }
};

struct ProbVjpArgs {
  ProbArgs f;                  // the forward's arguments (its record, mark, step_active and reductions read)
  const float *g_log_prob;     // optional [n_pix][H][T-1]
  const float *g_charge;       // optional [n_pix][H][T-1]
  const float *g_e_tick, *g_e_adc, *g_lam;   // optional [n_pix][H] (all three or none)
  float *g_wfs;                // [n_pix][T]
};

// Ticks are grouped into classes as in the forward, here by the five
// values a tick's hit and dist terms read (the running maximum at t and
// t + 1, q at t, t + 1 and at the shifted tick; the selection value is not
// differentiated).  Within a class every per-path partial derivative is the
// same; the per-tick cotangents (on the hit log-probability and on the dist
// value) enter linearly, so the partials are evaluated once per class and
// path, folded into seven per-class coefficients, and spread back to the
// class's ticks with the ticks' own cotangents.  Classes are also cut at
// every kVjpSpan ticks, so a warp's lanes hold a class's ticks.
//
// Few classes of a step have a cotangent at all: those of the K selected
// ticks and those whose probability is not 0 (the forward's record says
// which), about 10 % of the ticks.  A step lists them and takes as many at a
// time as there are threads for their (class, path) pairs: a thread evaluates
// the special functions of one pair, with paths that repeat a likelier path's
// charge left out (the first step has one path).  The weights exp(x - max) of
// a class's log-sum-exp stay unnormalised until its sums are formed, so the
// sums over the paths are a thread per (class, quantity) adding what the
// pairs left in shared memory, without shuffles; four lanes per class spread
// them to its ticks.
// Bound by instruction issue in the special functions, of which each lane
// should have one to evaluate: adjoint of 1500 dense rows 16.1 ms with a
// thread per class walking the K paths, 5.6 ms with a warp per class (15.5 of
// 32 lanes had a path) and the rows dealt in turn, 2.6 ms so.
constexpr int kVjpSpan = 16;
constexpr int kVjpArrays = 9;      // q, running max, 5 accumulators, dist cotangents, scratch; the esperance and the
                                   // soft-where weight are recomputed from q, so two blocks fit on an SM
constexpr int kVjpShorts = 3;      // class, representative, list of live classes (16 bits: ticks < kProbMaxT)
// what the pairs leave for their class: hit and dist terms; the hit weight and five partials times it, the dist weight
// and two partials times it (a class's sums then replace its first pair's); the hit terms' maximum
enum PairValue { kPairHit, kPairDist, kPairSums, kPairDistSums = kPairSums + 6, kPairMax = kPairDistSums + 3, kPairValues };
constexpr int kPairStride = kProbThreads + 1;   // quantities of one pair in different banks
constexpr int kTickLanes = 4;                   // lanes that share a class's ticks
static_assert(kProbMaxT <= 65536, "16-bit tick indices");

// Rows whose partials may not be finite (kWildRow) have a launch of their own (kWild): what they need besides costs the
// others 1.5 % of the adjoint's call.
template <bool kWild>
__global__ void __launch_bounds__(kProbThreads, 2) k_fee_prob_vjp(ProbVjpArgs va) {
  extern __shared__ __align__(16) float sm[];
  const ProbArgs &a = va.f;
  float *qs = sm, *cm = qs + kProbMaxT;
  float *Aq0 = cm + kProbMaxT, *Aqs = Aq0 + kProbMaxT, *Am0 = Aqs + kProbMaxT, *Am1 = Am0 + kProbMaxT;
  float *Aesp = Am1 + kProbMaxT, *Gd = Aesp + kProbMaxT, *tmp = Gd + kProbMaxT;
  float *pair = tmp + kProbMaxT;                               // [kPairValues][kPairStride]
  uint16_t *cls = reinterpret_cast<uint16_t *>(pair + kPairValues * kPairStride);
  uint16_t *rep = cls + kProbMaxT, *list = rep + kProbMaxT;
  __shared__ float red[kProbThreads / 32];
  __shared__ float pc[kProbMaxPaths], plp[kProbMaxPaths], glp_n[kProbMaxPaths], gc_n[kProbMaxPaths];
  __shared__ int ptop[kProbMaxPaths], act[kProbMaxPaths];
  __shared__ int counts[kProbTicks * (kProbThreads / 32)];
  __shared__ int n_exec, n_cls, n_act;

  const LsimParams &p = a.p;
  const int T = a.T, K = a.K, H = p.max_adc_values, tid = threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5;
  const float z = a.z, thr = a.thr;
  const float term_m1 = ldn_log_term(-1.0f);
  auto shifted = [&](int t) { return min(t + a.interval + 1, T - 1); };
  // the esperance and the soft-where weight of tick t, recomputed from q
  auto esp_at = [&](int t) { return (qs[shifted(t)] + thr) - 0.5f * (qs[t + 1] + qs[t]); };
  auto sw_at = [&](float e) { return sigmoid_f((e - thr) * 10.0f); };
  // whether every tick's cotangent from the reductions' is finite
  auto finite_cotangents = [&](float gl, float gt, float ga, float den) {
    return isfinite(fabsf(gl) + fabsf(gt) * (float)T / den + fabsf(ga) * p.adc_counts / den);
  };
  if (tid == 0) {
    int first = H;
    for (int h = 1; h < H; ++h)
      if (!a.step_active[h - 1]) {
        first = h;
        break;
      }
    n_exec = first;
  }
  __syncthreads();

  // a record of another call, or one that leaves out what a cotangent on the
  // distributions needs, has no gradient to give (its ticks may not even fit)
  const ProbMark mk = *a.mark;
  if (mk.n_pix != a.n_pix || mk.T != T || mk.K != K || mk.H != H ||
      ((va.g_log_prob || va.g_charge) && !mk.all_steps)) {
    for (int64_t pix = blockIdx.x; pix < a.n_pix; pix += gridDim.x)
      for (int t = tid; t < T; t += kProbThreads) va.g_wfs[pix * T + t] = NAN;
    return;
  }
  // the record is only read here: backward passes may share it
  for (int64_t pix = blockIdx.x; pix < a.n_pix; pix += gridDim.x) {
    if (((a.n_run[pix] & kWildRow) != 0) != kWild) continue;
    const float *w = a.wfs + pix * T;
    for (int t = tid; t < T; t += kProbThreads) qs[t] = w[t] * p.t_sampling;
    __syncthreads();
    block_scan_row<kScanSum>(qs, T, red);
    for (int t = tid; t < T; t += kProbThreads) {
      cm[t] = qs[t];
      Aq0[t] = Aqs[t] = Am0[t] = Am1[t] = Aesp[t] = 0.f;
    }
    __syncthreads();
    block_scan_row<kScanMax>(cm, T, red);
    for (int t = tid; t < T - 1; t += kProbThreads) {
      const int s = shifted(t);
      bool head = t % kVjpSpan == 0;
      if (!head) {
        const int sp = shifted(t - 1);
        auto ne = [](float x, float y) { return __float_as_uint(x) != __float_as_uint(y); };
        head = ne(cm[t], cm[t - 1]) || ne(cm[t + 1], cm[t]) || ne(qs[t], qs[t - 1]) || ne(qs[t + 1], qs[t]) ||
               ne(qs[s], qs[sp]);
      }
      tmp[t] = head ? 1.0f : 0.0f;
    }
    __syncthreads();
    block_scan_row<kScanSum>(tmp, T - 1, red);   // integer counts, exact in float32
    for (int t = tid; t < T - 1; t += kProbThreads) {
      const int u = (int)tmp[t] - 1;
      cls[t] = (uint16_t)u;
      if (t == 0 || (int)tmp[t - 1] != u + 1) rep[u] = (uint16_t)t;
      if (t == T - 2) n_cls = u + 1;
    }
    if (tid < K) {
      glp_n[tid] = 0.f;
      gc_n[tid] = 0.f;
    }
    __syncthreads();
    const int U = n_cls;
    if (tid == 0) rep[U] = (uint16_t)(T - 1);     // end of the last class

    const int n_run = min(n_exec, a.n_run[pix] & (kWildRow - 1));
    if (va.g_lam && n_run < n_exec) {
      // steps left out, every probability of theirs 0: a cotangent that is not finite is NaN on every tick
      bool odd = false;
      for (int h = n_run + tid; h < n_exec; h += kProbThreads) {
        const int64_t o = pix * H + h;
        odd |= !finite_cotangents(va.g_lam[o], va.g_e_tick[o], va.g_e_adc[o], 1e-10f);
      }
      if (__syncthreads_or(odd)) {
        for (int t = tid; t < T; t += kProbThreads) va.g_wfs[pix * T + t] = NAN;
        continue;
      }
    }
    for (int h = n_run - 1; h >= 0; --h) {
      const int64_t o = pix * H + h;
      // step h's input paths and selected ticks, recorded by the forward
      if (tid < K) {
        const float *st = a.state + (o * 2) * (int64_t)K;
        pc[tid] = st[tid];
        plp[tid] = st[K + tid];
        ptop[tid] = a.state_top[o * (int64_t)K + tid];
      }
      for (int t = tid; t < T; t += kProbThreads) Gd[t] = tmp[t] = 0.f;
      __syncthreads();
      if (wid == 0) {
        // the paths that count, in order (a path whose charge repeats that of one more than 110 log units likelier
        // adds nothing)
        bool on = lane < K;
        for (int j = 0; j < K; ++j)
          if (lane < K && j != lane && pc[j] == pc[lane] && plp[j] > plp[lane] + 110.0f) on = false;
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        if (on) act[__popc(bal & ((1u << lane) - 1u))] = lane;
        if (lane == 0) n_act = __popc(bal);
        if (lane < K && glp_n[lane] != 0.f) tmp[cls[ptop[lane]]] = 1.f;   // the class has a dist cotangent
      }
      if (wid == 1) {
        // the next step's state cotangents: new lp_j = dist[top_j], new c_j = q[best_j].  The first lane of those with
        // the same tick adds them all, in order
        auto add_to = [&](float *dst, int t, float v) {
          const bool on = lane < K;
          float sum = on ? dst[t] : 0.f;
          bool first = on;
          for (int j = 0; j < K; ++j) {
            const int tj = __shfl_sync(0xffffffffu, t, j);
            const float vj = __shfl_sync(0xffffffffu, v, j);
            if (tj == t) {
              sum += vj;
              if (j < lane) first = false;
            }
          }
          if (first) dst[t] = sum;
        };
        const int tt = lane < K ? ptop[lane] : 0;
        add_to(Gd, tt, lane < K ? glp_n[lane] : 0.f);
        add_to(Aq0, min(shifted(tt) + 1, T - 1), lane < K ? gc_n[lane] : 0.f);
      }
      if (va.g_charge)
        for (int t = tid; t < T - 1; t += kProbThreads) Aesp[t] += va.g_charge[o * (int64_t)(T - 1) + t];
      __syncthreads();
      // the reductions' cotangents, common to the step's ticks
      float gl = 0.f, gt = 0.f, ga = 0.f, den = 1.f;
      bool odd = false;      // not finite: a tick without probability has a cotangent too (0 times infinity)
      bool none = true;      // all zero: no tick has a cotangent from them
      if (va.g_lam) {
        const float ET = a.red[o], EA = a.red[a.n_pix * H + o], L = a.red[2 * a.n_pix * H + o];
        den = fmaxf(L, 1e-10f);
        const float on = L > 1e-10f ? 1.f : (L == 1e-10f ? 0.5f : 0.f);   // jnp.maximum's share
        gt = va.g_e_tick[o];
        ga = va.g_e_adc[o];
        // the lambda cotangent also reaches ET and EA through the denominator
        gl = va.g_lam[o] + on * (-(gt * ET + ga * EA) / den);
        odd = !finite_cotangents(gl, gt, ga, den);
        none = gl == 0.f && gt == 0.f && ga == 0.f;
      }
      // ---- the classes with a cotangent, in order
      unsigned live_bits[kProbTicks];
#pragma unroll
      for (int i = 0; i < kProbTicks; ++i) {
        const int u = tid + i * kProbThreads;
        bool live = false;
        if (u < U) {
          const int t = rep[u];
          live = odd || tmp[u] != 0.f;
          if (!none && !live) live = (a.live[o * kLiveWords + (t >> 5)] >> (t & 31)) & 1u;
          if (va.g_log_prob)
            for (int tt = t; tt < rep[u + 1] && !live; ++tt) live = va.g_log_prob[o * (int64_t)(T - 1) + tt] != 0.f;
        }
        live_bits[i] = __ballot_sync(0xffffffffu, live);
        if (lane == 0) counts[i * (kProbThreads / 32) + wid] = __popc(live_bits[i]);
      }
      __syncthreads();
      int n_live;
      {
        static_assert(kProbTicks * (kProbThreads / 32) == 64, "two counts a lane");
        const int c0 = counts[2 * lane], c1 = counts[2 * lane + 1];
        int incl = c0 + c1;
#pragma unroll
        for (int o2 = 1; o2 < 32; o2 <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o2);
          if (lane >= o2) incl += y;
        }
        n_live = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for (int i = 0; i < kProbTicks; ++i) {
          const int at = i * (kProbThreads / 32) + wid;      // entry of the prefix sums
          const int ex = __shfl_sync(0xffffffffu, incl - c0 - c1, at >> 1);
          const int first = __shfl_sync(0xffffffffu, c0, at >> 1);
          if ((live_bits[i] >> lane) & 1u)
            list[ex + (at & 1 ? first : 0) + __popc(live_bits[i] & ((1u << lane) - 1u))] =
                (uint16_t)(tid + i * kProbThreads);
        }
      }
      __syncthreads();
      auto at = [&](int what, int i) -> float & { return pair[what * kPairStride + i]; };
      // cotangent of the hit log-probability at a tick of probability pr
      auto cotangent = [&](int tt, float pr) {
        float gh = 0.f;
        if (va.g_log_prob) gh = va.g_log_prob[o * (int64_t)(T - 1) + tt];
        if (va.g_lam) gh += (gl + gt * (float)tt / den + ga * digitize(p, esp_at(tt)) / den) * pr;
        return gh;
      };
      const int na = n_act, per_round = kProbThreads / na;   // classes per round of pairs
      const int my = tid / na;                                // this thread's class in a round
      float glp = 0.f, gc = 0.f;                              // cotangents of its path act[tid - my na]
      for (int e0 = 0; e0 < n_live; e0 += per_round) {
        const int n_round = min(per_round, n_live - e0);
        const bool on = my < n_round;
        // ---- a thread per (class, path): values and partials at the class
        float xh = 0.f, xd = 0.f, v_q0 = 0.f, v_qs = 0.f, r = 0.f, v_m0 = 0.f, v_m1 = 0.f, v_e = 0.f;
        bool dist = false;     // the class has a dist cotangent
        if (on) {
          const int u = list[e0 + my], k = act[tid - my * na], t = rep[u], sidx = shifted(t);
          dist = tmp[u] != 0.f;
          const float c = pc[k], lp = plp[k];
          const float zm0 = ((cm[t] - c) - thr) * z, zm1 = ((cm[t + 1] - c) - thr) * z;
          const float LM0 = log_ndtr_f(zm0), LM1 = log_ndtr_f(zm1);
          const LogDiff dm(zm1, zm0, LM1, LM0, term_m1);
          const float zq0 = ((qs[t] - c) - thr) * z, zqs = ((qs[sidx] - c) - thr) * z;
          const float LQ0 = log_ndtr_f(zq0), LQs = log_ndtr_f(zqs);
          const LogDiff dq(zqs, zq0, LQs, LQ0, term_m1);
          const float lg = dm.out, lep = dq.out;
          // the partials of the smaller term (both at a tie), and of the other where 0 times it may be NaN
          float g_m1 = 0.f, g_m0 = 0.f, g_qs = 0.f, g_q0 = 0.f;
          if (dist || kWild || !(lep < lg)) dm.partials(zm1, zm0, LM1, LM0, g_m1, g_m0);
          if (kWild || !(lep > lg)) dq.partials(zqs, zq0, LQs, LQ0, g_qs, g_q0);
          const float le1 = fminf(lep, lg);
          const float le2 = kProbFloor + softplus_f(le1 - kProbFloor);
          const float wt = sw_at(esp_at(t));
          const float le = wt * le2 + (1.0f - wt) * kProbFloor;
          // per unit hit cotangent: le = w le2 + (1 - w)(-1000), w = sigmoid((esp - thr) 10)
          const float gl1 = wt * sigmoid_f(le1 - kProbFloor);
          const float s_lep = lep < lg ? 1.f : (lep == lg ? 0.5f : 0.f);
          xh = le + lp;
          xd = lg + lp;
          v_q0 = gl1 * s_lep * g_q0 * z;
          v_qs = gl1 * s_lep * g_qs * z;
          r = gl1 * (1.f - s_lep);
          v_m0 = g_m0 * z;
          v_m1 = g_m1 * z;
          v_e = (le2 - kProbFloor) * wt * (1.0f - wt) * 10.0f;
          at(kPairHit, tid) = xh;
          at(kPairDist, tid) = xd;
        }
        __syncthreads();
        // ---- weights of the log-sum-exps and the partials times them
        auto highest = [&](const float *x) {
          float m = -INFINITY;
          for (int j = 0; j < na; ++j) m = fmaxf(m, x[j]);
          return m;
        };
        float wh = 0.f, wd = 0.f, gh_c = 0.f, gd_c = 0.f;   // weights; charge partials times them
        if (on) {
          const float m = highest(&at(kPairHit, my * na));
          wh = expf(xh - m);
          const float p0 = wh * v_q0, ps = wh * v_qs, pm0 = wh * (r * v_m0), pm1 = wh * (r * v_m1);
          gh_c = p0 + ps + pm0 + pm1;
          at(kPairSums, tid) = wh;
          at(kPairSums + 1, tid) = p0;
          at(kPairSums + 2, tid) = ps;
          at(kPairSums + 3, tid) = pm0;
          at(kPairSums + 4, tid) = pm1;
          at(kPairSums + 5, tid) = wh * v_e;
          if (tid == my * na) at(kPairMax, tid) = m;
          if (dist) {
            wd = expf(xd - highest(&at(kPairDist, my * na)));
            const float d0 = wd * v_m0, d1 = wd * v_m1;
            gd_c = d0 + d1;
            at(kPairDistSums, tid) = wd;
            at(kPairDistSums + 1, tid) = d0;
            at(kPairDistSums + 2, tid) = d1;
          }
        }
        __syncthreads();
        // ---- a thread per (class, quantity): the sums over the paths
        constexpr int kSums = kPairMax - kPairSums;
        for (int i = tid; i < n_round * kSums; i += kProbThreads) {
          const int e = i / kSums, what = kPairSums + i % kSums;
          if (what >= kPairDistSums && tmp[list[e0 + e]] == 0.f) continue;
          float *x = &at(what, e * na), sum = 0.f;
          for (int j = 0; j < na; ++j) sum += x[j];
          x[0] = sum;
        }
        __syncthreads();
        // ---- kTickLanes lanes per class: its ticks
        for (int i = tid; (i & ~31) < n_round * kTickLanes; i += kProbThreads) {
          const int e = i / kTickLanes;
          const bool mine = e < n_round;
          float Hs = 0.f, Ds = 0.f, inv = 0.f, inv_d = 0.f;
          // a class without a cotangent takes no part, which shows only where its sums are not finite
          bool takes_part = true;
          if (kWild) {
            bool any = false;
            if (mine) {
              const int u = list[e0 + e];
              const float pr = expf(logf(at(kPairSums, e * na)) + at(kPairMax, e * na));
              for (int tt = rep[u] + i % kTickLanes; tt < rep[u + 1]; tt += kTickLanes)
                any |= cotangent(tt, pr) != 0.f || Gd[tt] != 0.f;
            }
            takes_part = (__ballot_sync(0xffffffffu, any) >> (lane & ~(kTickLanes - 1))) & ((1u << kTickLanes) - 1u);
          }
          if (mine) {
            const int u = list[e0 + e], f = e * na;
            const bool with_d = tmp[u] != 0.f;
            const float S = at(kPairSums, f), pr = expf(logf(S) + at(kPairMax, f));
            inv = 1.0f / S;
            inv_d = with_d ? 1.0f / at(kPairDistSums, f) : 0.f;
            for (int tt = rep[u] + i % kTickLanes; tt < rep[u + 1]; tt += kTickLanes) {
              const float add_e = va.g_lam ? digitize_vjp(p, esp_at(tt), ga * pr / den) : 0.f;
              if (!takes_part) {
                Aesp[tt] += add_e;
                continue;
              }
              const float gh = cotangent(tt, pr), gd = Gd[tt];
              Hs += gh;
              Ds += gd;
              const float n = gh * inv, nd = gd * inv_d;
              Aq0[tt] += n * at(kPairSums + 1, f);
              Aqs[tt] += n * at(kPairSums + 2, f);
              Aesp[tt] += add_e + n * at(kPairSums + 5, f);
              float m0 = n * at(kPairSums + 3, f), m1 = n * at(kPairSums + 4, f);
              if (with_d) {
                m0 += nd * at(kPairDistSums + 1, f);
                m1 += nd * at(kPairDistSums + 2, f);
              }
              Am0[tt] += m0;
              Am1[tt] += m1;
            }
          }
#pragma unroll
          for (int s2 = kTickLanes / 2; s2 > 0; s2 >>= 1) {
            Hs += __shfl_xor_sync(0xffffffffu, Hs, s2);
            Ds += __shfl_xor_sync(0xffffffffu, Ds, s2);
          }
          if (mine && i % kTickLanes == 0) {
            at(kPairMax, e * na) = Hs != 0.f ? Hs * inv : 0.f;
            at(kPairDistSums, e * na) = Ds * inv_d;
          }
        }
        __syncthreads();
        // ---- the pair's path (the next round writes these two values only after its first barrier)
        if (on) {
          const float n = at(kPairMax, my * na), nd = dist ? at(kPairDistSums, my * na) : 0.f;
          if (!kWild || n != 0.f || nd != 0.f) {
            glp += wh * n;
            gc -= gh_c * n;
            if (dist) {
              glp += wd * nd;
              gc -= gd_c * nd;
            }
          }
        }
      }
      if (h > 0) {
        // cotangent of this step's input state = the previous step's output state
        at(kPairHit, tid) = glp;
        at(kPairDist, tid) = gc;
        if (tid < K) glp_n[tid] = gc_n[tid] = 0.f;    // paths that do not count have none
        __syncthreads();
        const int n_used = min(per_round, n_live);
        if (wid < 2 && lane < na) {
          float sum = 0.f;
          for (int j = 0; j < n_used; ++j) sum += at(wid == 0 ? kPairHit : kPairDist, j * na + lane);
          (wid == 0 ? glp_n : gc_n)[act[lane]] = sum;
        }
      }
      __syncthreads();
    }
    // ---- assemble dL/dq from the per-tick partials
    // running maximum: cm[t] (tick t's zm0) and cm[t] as tick t-1's cm[t+1]
    for (int t = tid; t < T; t += kProbThreads) tmp[t] = (t < T - 1 ? Am0[t] : 0.f) + (t > 0 ? Am1[t - 1] : 0.f);
    __syncthreads();
    block_scan_row<kScanSum>(tmp, T, red);   // prefix sums P of dL/dcm
    // each run of a constant running maximum routes its sum to the run's first tick
    for (int t = tid; t < T; t += kProbThreads) {
      float g = Aq0[t];
      const bool start = t == 0 || cm[t] != cm[t - 1];
      if (start) {
        int e = t, hi = T;        // last tick of the run: cm does not fall (and is never NaN)
        while (hi - e > 1) {
          const int mid = (e + hi) >> 1;
          if (cm[mid] == cm[t]) e = mid; else hi = mid;
        }
        g += tmp[e] - (t > 0 ? tmp[t - 1] : 0.f);
      }
      // shifted-tick role q[s_t] (s_t = min(t + interval + 1, T - 1)), with the esperance terms
      const int t0 = t - a.interval - 1;
      if (t < T - 1) {
        if (t0 >= 0) g += Aqs[t0] + Aesp[t0];
      } else {
        for (int u = max(t0, 0); u < T - 1; ++u) g += Aqs[u] + Aesp[u];
      }
      // esperance: - 0.5 (q[t + 1] + q[t])
      if (t < T - 1) g -= 0.5f * Aesp[t];
      if (t > 0) g -= 0.5f * Aesp[t - 1];
      Gd[t] = g;
    }
    __syncthreads();
    // q = cumsum(w * ts): dL/dw[i] = ts * sum_{j >= i} dL/dq[j]
    block_scan_row<kScanSuffixSum>(Gd, T, red);
    for (int t = tid; t < T; t += kProbThreads) va.g_wfs[pix * T + t] = Gd[t] * p.t_sampling;
    __syncthreads();
  }
}

}  // namespace

// Blocks of the forward kernel: two per SM.
static int64_t prob_blocks() { return (int64_t)device_sm_count() * 2; }

static size_t al256(size_t b) { return (b + 255) & ~size_t(255); }

// The steps' flags, a record's mark and, at the end of their 256 bytes, the forward's pixel counter.
constexpr size_t kFlagBytes = 256, kMarkAt = 64;
static_assert(sizeof(int32_t) * LSIM_MAX_HITS <= kMarkAt && kMarkAt % alignof(ProbMark) == 0 &&
              kMarkAt + sizeof(ProbMark) + sizeof(unsigned long long) <= kFlagBytes, "flags, mark and counter");
static unsigned long long *work_counter(int32_t *flags) {
  return reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(flags) + kFlagBytes) - 1;
}

static int cache_row(int32_t n_t) { return n_t < 32 ? 32 : n_t > kProbMaxT ? kProbMaxT : (n_t + 31) & ~31; }

// step_active, then the path values of the blocks that a call starts
size_t fee_prob_workspace_bytes(int64_t n_pix, int32_t n_t, int32_t n_paths) {
  const int64_t cap = prob_blocks(), blocks = n_pix < 0 ? 0 : n_pix < cap ? n_pix : cap;
  const int paths = n_paths < 1 ? 1 : n_paths > kProbMaxPaths ? kProbMaxPaths : n_paths;
  return al256(kFlagBytes + sizeof(float) * (size_t)blocks * paths * kCacheArrays * cache_row(n_t));
}

size_t fee_prob_workspace_bytes() { return fee_prob_workspace_bytes(INT64_MAX, kProbMaxT, kProbMaxPaths); }

struct ProbRecord {
  ProbMark *mark;
  int32_t *step_active, *n_run, *top;
  float *state, *red;
  uint32_t *live;
};

static size_t record_layout(int64_t n_pix, int32_t max_adc_values, int32_t n_paths, ProbRecord *r, char *base) {
  const size_t steps = (size_t)(n_pix > 0 ? n_pix : 0) * (size_t)max_adc_values;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += al256(bytes);
    return base ? base + at : nullptr;
  };
  char *active = take(kFlagBytes);
  char *state = take(sizeof(float) * 2 * steps * n_paths);
  char *top = take(sizeof(int32_t) * steps * n_paths);
  char *run = take(sizeof(int32_t) * (size_t)(n_pix > 0 ? n_pix : 0));
  char *live = take(sizeof(uint32_t) * steps * kLiveWords);
  char *red = take(sizeof(float) * 3 * steps);
  if (r)
    *r = ProbRecord{reinterpret_cast<ProbMark *>(active + kMarkAt), reinterpret_cast<int32_t *>(active), reinterpret_cast<int32_t *>(run),
                    reinterpret_cast<int32_t *>(top), reinterpret_cast<float *>(state),
                    reinterpret_cast<float *>(red), reinterpret_cast<uint32_t *>(live)};
  return off;
}

size_t fee_prob_record_bytes(int64_t n_pix, int32_t max_adc_values, int32_t n_paths) {
  return record_layout(n_pix, max_adc_values, n_paths, nullptr, nullptr);
}

static ProbArgs prob_args(const LsimParams &p, const float *wfs, int64_t n_pix, int32_t n_t, int32_t n_paths) {
  ProbArgs a{};
  a.p = p;
  a.wfs = wfs;
  a.n_pix = n_pix;
  a.T = n_t;
  a.K = n_paths;
  a.interval = p.fee_interval;
  a.z = (float)(1.0 / (double)p.reset_noise);
  a.thr = p.threshold;
  return a;
}

static int check_prob(const LsimParams &p, int32_t n_t, int32_t n_paths) {
  if (n_t < 3 || n_t > kProbMaxT) return set_error(LSIM_ERR_UNSUPPORTED, "probabilistic FEE: n_t must be in [3, 2048]");
  if (n_paths < 1 || n_paths > kProbMaxPaths || n_paths > n_t - 1)
    return set_error(LSIM_ERR_UNSUPPORTED, "probabilistic FEE: fee_paths_scaling must be in [1, min(32, n_t - 1)]");
  if (!(p.reset_noise > 0.0f)) return set_error(LSIM_ERR_INVALID, "probabilistic FEE: RESET_NOISE_CHARGE must be > 0");
  return LSIM_OK;
}

template <bool kDist>
static int launch_prob(const ProbArgs &a, cudaStream_t st) {
  const size_t smem = sizeof(float) * (kProbArrays * kProbMaxT + kProbExtraFloats);
  if (cudaFuncSetAttribute(k_fee_prob<kDist>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return LSIM_ERR_CUDA;
  const int64_t cap = prob_blocks();
  k_fee_prob<kDist><<<(unsigned)(a.n_pix < cap ? a.n_pix : cap), kProbThreads, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? LSIM_OK : LSIM_ERR_CUDA;
}

// record: null, or where the adjoint's record goes (fee_prob_record_bytes).
// all_steps: the record serves cotangents on the log-probabilities too.
static int run_fee_prob_impl(const LsimParams &p, const float *wfs, int64_t n_pix, int32_t n_t, int32_t n_paths,
                             float stop_threshold, float *log_prob, float *charge, float *e_tick, float *e_adc,
                             float *lam, void *record, bool all_steps, void *ws, cudaStream_t st) {
  int rc = check_prob(p, n_t, n_paths);
  if (rc != LSIM_OK) return rc;
  ProbArgs a = prob_args(p, wfs, n_pix, n_t, n_paths);
  a.log_stop = logf(stop_threshold);
  a.log_prob = log_prob;
  a.charge = charge;
  a.e_tick = e_tick;
  a.e_adc = e_adc;
  a.lam = lam;
  a.all_steps = all_steps || charge != nullptr;
  char *b = static_cast<char *>(ws);
  a.step_active = reinterpret_cast<int32_t *>(b);
  a.cache = reinterpret_cast<float *>(b + kFlagBytes);
  a.cache_row = cache_row(n_t);
  if (record) {
    ProbRecord r;
    record_layout(n_pix, p.max_adc_values, n_paths, &r, static_cast<char *>(record));
    a.mark = r.mark;
    a.step_active = r.step_active;
    a.state = r.state;
    a.state_top = r.top;
    a.live = r.live;
    a.n_run = r.n_run;
    a.red = r.red;
  }
  a.work = work_counter(a.step_active);
  if (cudaMemsetAsync(a.step_active, 0, kFlagBytes, st) != cudaSuccess) return LSIM_ERR_CUDA;
  if (n_pix == 0) return LSIM_OK;
  rc = log_prob ? launch_prob<true>(a, st) : launch_prob<false>(a, st);
  if (rc != LSIM_OK) return rc;
  if (log_prob || charge || lam)
    k_fee_prob_mask<<<(unsigned)device_sm_count() * 4, 256, 0, st>>>(a, p.max_adc_values);
  return cudaGetLastError() == cudaSuccess ? LSIM_OK : LSIM_ERR_CUDA;
}

template <bool kWild>
static int launch_vjp(const ProbVjpArgs &va, cudaStream_t st) {
  const size_t smem = sizeof(float) * (kVjpArrays * kProbMaxT + kPairValues * kPairStride) +
                      sizeof(uint16_t) * kVjpShorts * kProbMaxT;
  if (cudaFuncSetAttribute(k_fee_prob_vjp<kWild>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return LSIM_ERR_CUDA;
  constexpr int64_t cap = 1 << 30;
  k_fee_prob_vjp<kWild><<<(unsigned)(va.f.n_pix < cap ? va.f.n_pix : cap), kProbThreads, smem, st>>>(va);
  return cudaGetLastError() == cudaSuccess ? LSIM_OK : LSIM_ERR_CUDA;
}

// The reverse pass on a record.
int run_fee_prob_vjp_recorded(const LsimParams &p, const float *wfs, int64_t n_pix, int32_t n_t, int32_t n_paths,
                              const void *record, const float *g_log_prob, const float *g_charge, const float *g_e_tick,
                              const float *g_e_adc, const float *g_lam, float *g_wfs, cudaStream_t st) {
  int rc = check_prob(p, n_t, n_paths);
  if (rc != LSIM_OK || n_pix == 0) return rc;
  ProbRecord r;
  record_layout(n_pix, p.max_adc_values, n_paths, &r, const_cast<char *>(static_cast<const char *>(record)));
  ProbVjpArgs va{};
  va.f = prob_args(p, wfs, n_pix, n_t, n_paths);
  va.f.mark = r.mark;
  va.f.step_active = r.step_active;
  va.f.state = r.state;
  va.f.state_top = r.top;
  va.f.live = r.live;
  va.f.n_run = r.n_run;
  va.f.red = r.red;
  va.g_log_prob = g_log_prob;
  va.g_charge = g_charge;
  va.g_e_tick = g_e_tick;
  va.g_e_adc = g_e_adc;
  va.g_lam = g_lam;
  va.g_wfs = g_wfs;
  // a block per pixel: pixels differ several times in cost, and blocks start as
  // others end (the record is only read, so it has no place for a counter).
  // 1500 rows, with a warp per class: 5.6 ms with the rows dealt in turn to the
  // resident blocks, 4.8 ms so
  rc = launch_vjp<false>(va, st);
  return rc != LSIM_OK ? rc : launch_vjp<true>(va, st);
}

size_t fee_prob_vjp_workspace_bytes(int64_t n_pix, int32_t max_adc_values, int32_t n_paths) {
  return fee_prob_workspace_bytes(n_pix, kProbMaxT, n_paths) + fee_prob_record_bytes(n_pix, max_adc_values, n_paths);
}

int run_fee_prob_vjp(const LsimParams &p, const float *wfs, int64_t n_pix, int32_t n_t, int32_t n_paths,
                     float stop_threshold, const float *g_log_prob, const float *g_charge, const float *g_e_tick,
                     const float *g_e_adc, const float *g_lam, float *g_wfs, void *ws, cudaStream_t st) {
  // the record, then the forward's workspace
  char *record = static_cast<char *>(ws);
  ws = record + fee_prob_record_bytes(n_pix, p.max_adc_values, n_paths);
  // forward with the steps recorded, then the reverse pass
  const int rc = run_fee_prob_impl(p, wfs, n_pix, n_t, n_paths, stop_threshold, nullptr, nullptr, nullptr, nullptr,
                                   nullptr, record, g_log_prob != nullptr || g_charge != nullptr, ws, st);
  if (rc != LSIM_OK) return rc;
  return run_fee_prob_vjp_recorded(p, wfs, n_pix, n_t, n_paths, record, g_log_prob, g_charge, g_e_tick, g_e_adc,
                                   g_lam, g_wfs, st);
}

int run_fee_prob(const LsimParams &p, const float *wfs, int64_t n_pix, int32_t n_t, int32_t n_paths,
                 float stop_threshold, float *log_prob, float *charge, float *e_tick, float *e_adc, float *lam,
                 void *record, void *ws, cudaStream_t st) {
  return run_fee_prob_impl(p, wfs, n_pix, n_t, n_paths, stop_threshold, log_prob, charge, e_tick, e_adc, lam, record,
                           false, ws, st);
}

}  // namespace lsim
