// Warp-cooperative self-trigger front end on a waveform held in shared
// memory: cumulative charge, threshold crossing, integration window, reset,
// digitisation, and the adjoint of all of it.
//
// Reference: get_adc_values (fee_jax.py:168-279) and digitize
// (fee_jax.py:55-71).  Per hit h the reference finds the first i with
// Q[i] <= thr <= Q[i+1] (Q = base + C, C = cumsum(w * t_sampling)),
// integrates to e = min(i + 1 + interval, T-1), accepts the hit when
// C[e] >= thr and a crossing exists, and resets
// C <- max(C - C[min(i + 2 + interval, T-1)], 0).
#pragma once

#include "lsim_common.cuh"

namespace lsim {

constexpr int kMaskWords = 64;   // words per hit: 2 per lane, bit 4m + q for tick 128m + 4 lane + q (T <= 2048)
static_assert(kFeeMaskWords == LSIM_MAX_HITS * kMaskWords, "reset-mask scratch per warp");
constexpr int kFeePass = 4 * kWarp;   // ticks per warp pass: lane l holds ticks 4l .. 4l + 3

struct FeeState {
  int n_done;                  // hits evaluated before the early exit (the rest are empty)
  int e[LSIM_MAX_HITS];        // integration end index
  int e2[LSIM_MAX_HITS];       // reset index
  int cond[LSIM_MAX_HITS];     // 1 = rejected (adc forced to 0)
  float raw[LSIM_MAX_HITS];    // integrated charge before digitisation
  float R[LSIM_MAX_HITS];      // threshold path: charge subtracted by reset h
  uint32_t *mask;              // sweep path: [max_adc_values][kMaskWords], (C - R >= 0) per tick, per hit, lane-private
};

__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// digitize (fee_jax.py:68-69): continuous, clamped to [0, ADC_COUNTS].
__device__ __forceinline__ float digitize(const LsimParams &p, float q) {
  float x = (q * p.gain + p.v_pedestal) - p.v_cm;
  x = x < 0.f ? 0.f : x;
  float y = (x * p.adc_counts) / p.vref_minus_cm;
  return y > p.adc_counts ? p.adc_counts : y;
}

// d digitize / d q times g, with JAX's 0.5 rule at the clamp ties.
__device__ __forceinline__ float digitize_vjp(const LsimParams &p, float q, float g) {
  float x = (q * p.gain + p.v_pedestal) - p.v_cm;
  float gx = x > 0.f ? 1.f : (x == 0.f ? 0.5f : 0.f);
  float y = ((x < 0.f ? 0.f : x) * p.adc_counts) / p.vref_minus_cm;
  float gy = y < p.adc_counts ? 1.f : (y == p.adc_counts ? 0.5f : 0.f);
  return ((g * gy) * (p.adc_counts / p.vref_minus_cm)) * gx * p.gain;
}

// A row's cumulative charge is kept as its chunks' own prefix sums X (lane l:
// ticks l per .. l per + per - 1) and each chunk's offset: C[i] = offset + X[i].
// lo, hi: smallest and largest C of the lane's ticks (the largest with the
// next lane's first tick); fast: whether the row suits the threshold path.
struct RowStats {
  float lo, hi, offset;
  bool fast;
};
__device__ __forceinline__ int chunk_ticks(int T) { return (T + kWarp - 1) / kWarp; }
// i / per for i < 2048, the quotient's distance from an integer being at least 0.5 / per
__device__ __forceinline__ int chunk_of(int i, int per) { return (int)(((float)i + 0.5f) * (1.0f / (float)per)); }
// C[i], i possibly different in each lane (all lanes take part)
__device__ __forceinline__ float row_charge(const float *X, const RowStats &rs, int T, int i) {
  return __shfl_sync(0xffffffffu, rs.offset, chunk_of(i, chunk_ticks(T))) + X[i];
}

// Rows whose values stay below this (and are finite) take the threshold
// path: no intermediate of the resets can overflow there.
constexpr float kFeeFastMax = 1e30f;

// Cumulative charge C[i] = sum_{j<=i} X[j]*ts over T ticks: X becomes the
// chunks' prefix sums, the offsets (a warp scan of the chunks' totals) and the
// extremes of C are returned.  Adding an offset is monotone with its rounding,
// so a chunk's extremes are the offset plus those of its prefix sums, and the
// row is passed over once: a second pass that added the offsets took half of
// this function's instructions, and the threshold path reads a few C only.
__device__ __forceinline__ RowStats warp_cumsum_charge(float *X, int T, float ts, int lane) {
  const int per = chunk_ticks(T);
  const int b = min(lane * per, T);
  const int e = min(b + per, T);
  float s = 0.f, lo = INFINITY, hi = -INFINITY;
  int i = b;
#pragma unroll 1
  for (; i + 8 <= e; i += 8) {   // eight loads in flight ahead of the serial chain
    float x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = X[i + q];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      X[i + q] = s = fmaf(x[q], ts, s);
      lo = fminf(lo, s);
      hi = fmaxf(hi, s);
    }
  }
#pragma unroll 1
  for (; i < e; ++i) {
    X[i] = s = fmaf(X[i], ts, s);
    lo = fminf(lo, s);
    hi = fmaxf(hi, s);
  }
  float incl = s;
#pragma unroll 1
  for (int o = 1; o < kWarp; o <<= 1) {
    float y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  RowStats st;
  st.offset = lane > 0 ? incl - s : -0.f;     // -0 + x is x
  st.lo = st.offset + lo;
  st.hi = st.offset + hi;
  // a NaN in the row shows in its chunk's total or in the next chunks' offset
  const bool ok = b >= e || (isfinite(s) && isfinite(st.offset) && st.lo > -kFeeFastMax && st.hi < kFeeFastMax);
  const float nx = __shfl_down_sync(0xffffffffu, b < e ? st.offset + X[b] : 0.f, 1);
  if (lane < kWarp - 1 && e < T) st.hi = fmaxf(st.hi, nx);
  st.fast = __all_sync(0xffffffffu, ok);
  __syncwarp();
  return st;
}

// The cumulative charge itself, in place of the prefix sums.
__device__ __forceinline__ void add_offsets(float *X, int T, const RowStats &rs, int lane) {
  const int per = chunk_ticks(T), b = min(lane * per, T), e = min(b + per, T);
  for (int i = b; i < e; ++i) X[i] = rs.offset + X[i];
  __syncwarp();
}

// The noise draws of a row ([1 + 3H], or none), loaded once: lane l holds draws l and l + 32.
struct Draws {
  const float *src;
  float a, b;
  __device__ __forceinline__ Draws(const float *normals, int H, int lane) : src(normals), a(0.f), b(0.f) {
    if (normals) {
      if (lane < 1 + 3 * H) a = normals[lane];
      if (lane + kWarp < 1 + 3 * H) b = normals[lane + kWarp];
    }
  }
  __device__ __forceinline__ float operator[](int i) const {   // i the same in all lanes
    return i < kWarp ? __shfl_sync(0xffffffffu, a, i) : __shfl_sync(0xffffffffu, b, i - kWarp);
  }
};
static_assert(1 + 3 * LSIM_MAX_HITS <= 2 * kWarp, "two draws a lane");
// ... and their absence, known when compiling
struct NoDraws {
  static constexpr const float *src = nullptr;
  __device__ __forceinline__ float operator[](int) const { return 0.f; }
};

// C = cumsum(W * ts)  ->  dL/dW[i] = ts * sum_{j >= i} dL/dC[j], in place
// (lane-contiguous chunks + warp suffix scan of the chunk totals).
// kUnroll: 1 in the pixel kernels, whose instructions do not fit in the cache;
// k_fee_vjp takes 8 (212 us instead of 244 on 16 events' rows of 2000 ticks).
template <int kUnroll>
__device__ __forceinline__ void warp_suffix_charge(float *G, int T, float ts, int lane) {
  const int per = chunk_ticks(T);
  const int b = lane * per;
  const int e = min(b + per, T);
  float s = 0.f;
#pragma unroll kUnroll
  for (int i = e - 1; i >= b; --i) {
    s += G[i];
    G[i] = s;
  }
  float incl = s;   // suffix sums across lanes
#pragma unroll 1
  for (int o = 1; o < kWarp; o <<= 1) {
    float y = __shfl_down_sync(0xffffffffu, incl, o);
    if (lane + o < kWarp) incl += y;
  }
  const float offset = incl - s;
#pragma unroll kUnroll
  for (int i = b; i < e; ++i) G[i] = (offset + G[i]) * ts;
  __syncwarp();
}

// First q in 0..3 with Q[i0+q] <= thr <= Q[i0+q+1] (Q = base + value) over
// the ticks v0..v3 and the following tick nx, counting only pairs with
// i0 + q < lim - 1; 4 if none.
__device__ __forceinline__ int first_crossing(float v0, float v1, float v2, float v3, float nx, float base, float thr,
                                              int i0, int lim) {
  const float q0 = base + v0, q1 = base + v1, q2 = base + v2, q3 = base + v3, q4 = base + nx;
  int first = 4;
  if (i0 + 3 < lim - 1 && q4 >= thr && q3 <= thr) first = 3;
  if (i0 + 2 < lim - 1 && q3 >= thr && q2 <= thr) first = 2;
  if (i0 + 1 < lim - 1 && q2 >= thr && q1 <= thr) first = 1;
  if (i0 < lim - 1 && q1 >= thr && q0 <= thr) first = 0;
  return first;
}

// ---------------------------------------------------------------- sweep path
//
// The general path: resets applied to the row, crossings found by sweeping
// it.  It serves the rows that the threshold path below does not take
// (values that are not finite or beyond kFeeFastMax).

// Forward self-trigger on C (in place).  normals: per-pixel standard
// normals [1 + 3H] or null (noise off).  Writes adc (digitized) and tick
// per hit through lane 0; fills st when non-null.  C must be 16-byte
// aligned with room for whole 4-tick groups (T rounded up to 4).
//
// Lane l works on ticks 128m + 4l .. 128m + 4l + 3 of pass m (one float4).
//
// early_exit (noise off, threshold > 0): once a rejected hit leaves C all
// zero, every later hit is provably empty (no crossing of a positive
// threshold, C[e] = 0, reset by 0 keeps C zero), so the remaining hits are
// written as empty without sweeping the row again.
static __device__ __noinline__ void fee_forward_sweep(const LsimParams &p, float *C, int T, const float *normals,
                                               float *adc_out, float *tick_out, FeeState *st, float *raw_out,
                                               bool early_exit, int lane) {
  const float thr = p.threshold;
  const int H = p.max_adc_values;
  float base = normals ? normals[0] * p.reset_noise : 0.f;
  float4 *C4 = reinterpret_cast<float4 *>(C);
  // first i < T - 1 with Q[i] <= thr <= Q[i + 1], Q = base + C, for hit 0;
  // later hits' searches run inside the previous hit's reset sweep
  int idx = T - 2;
  for (int i0 = 4 * lane, m = 0; m * kFeePass < T - 1; ++m, i0 += kFeePass) {
    const float4 c = i0 < T ? C4[i0 / 4] : make_float4(0.f, 0.f, 0.f, 0.f);
    float nx = __shfl_down_sync(0xffffffffu, c.x, 1);
    if (lane == kWarp - 1) nx = i0 + 4 < T ? C[i0 + 4] : 0.f;
    const int first = first_crossing(c.x, c.y, c.z, c.w, nx, base, thr, i0, T);
    const unsigned bal = __ballot_sync(0xffffffffu, first < 4);
    if (bal) {
      const int ln = __ffs(bal) - 1;
      idx = m * kFeePass + 4 * ln + __shfl_sync(0xffffffffu, first, ln);
      break;
    }
  }
  for (int h = 0; h < H; ++h) {
    int e = idx + 1 + p.fee_interval;
    if (e >= T) e = T - 1;
    const float qvn = C[e];
    const float qv = base + qvn;
    const float extra = normals ? normals[1 + 3 * h] * p.uncorr_noise : 0.f;
    float adc = (qvn != 0.f) ? (qv + extra) : qvn;
    const bool cond = (adc < thr) || (idx == T - 2);
    if (cond) adc = 0.f;
    const float tick = cond ? (float)(T - 2) : (float)idx;
    if (normals) base = cond ? normals[3 + 3 * h] * p.uncorr_noise : normals[2 + 3 * h] * p.reset_noise;
    int e2 = idx + 2 + p.fee_interval;
    if (e2 >= T) e2 = T - 1;
    const float R = C[e2];
    __syncwarp();
    // reset: C <- where(C - R < 0, 0, C - R), keep bits per lane (bit 4m + q),
    // and the next hit's crossing search on the reset values: pairs inside a
    // lane's 4 ticks and with the next lane's first tick are tested in the
    // pass; lane 31's last pair waits for lane 0's first value of the next pass
    bool nz = false;
    uint64_t km = 0u;
    int nidx = T - 2;
    bool found = false;
    float carry = 0.f;          // lane 31's last reset value of the previous pass
    for (int i0 = 4 * lane, sh = 0, m = 0; i0 - 4 * lane < T; i0 += kFeePass, sh += 4, ++m) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (i0 < T) {
        const float4 c = C4[i0 / 4];
        v[0] = c.x; v[1] = c.y; v[2] = c.z; v[3] = c.w;
        uint32_t bits = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (i0 + q < T) {
            const float d = v[q] - R;
            const bool keep = !(d < 0.f);
            v[q] = keep ? d : 0.f;
            nz |= keep && d != 0.f;
            bits |= (keep ? 1u : 0u) << q;
          }
        }
        C4[i0 / 4] = make_float4(v[0], v[1], v[2], v[3]);
        km |= (uint64_t)bits << sh;
      }
      const float nx = __shfl_down_sync(0xffffffffu, v[0], 1);
      const float v0 = __shfl_sync(0xffffffffu, v[0], 0);
      if (!found) {
        // the pair (128m - 1, 128m) left over from the previous pass
        const int ip = m * kFeePass - 1;
        if (m > 0 && ip < T - 1 && base + v0 >= thr && base + carry <= thr) {
          nidx = ip;
          found = true;
        } else {
          const int first = lane < kWarp - 1 ? first_crossing(v[0], v[1], v[2], v[3], nx, base, thr, i0, T)
                                             : first_crossing(v[0], v[1], v[2], v[3], 0.f, base, thr, i0, min(T, i0 + 4));
          const unsigned bal = __ballot_sync(0xffffffffu, first < 4);
          if (bal) {
            const int ln = __ffs(bal) - 1;
            nidx = m * kFeePass + 4 * ln + __shfl_sync(0xffffffffu, first, ln);
            found = true;
          }
        }
      }
      carry = __shfl_sync(0xffffffffu, v[3], kWarp - 1);
    }
    idx = nidx;
    if (st) {
      st->mask[h * kMaskWords + 2 * lane] = (uint32_t)km;
      st->mask[h * kMaskWords + 2 * lane + 1] = (uint32_t)(km >> 32);
    }
    __syncwarp();
    if (lane == 0) {
      if (adc_out) adc_out[h] = digitize(p, adc);
      if (tick_out) tick_out[h] = tick;
      if (raw_out) raw_out[h] = adc;
      if (st) { st->e[h] = e; st->e2[h] = e2; st->cond[h] = cond ? 1 : 0; st->raw[h] = adc; }
    }
    if (early_exit && cond && !__any_sync(0xffffffffu, nz)) {
      if (lane == 0) {
        const float a0 = digitize(p, 0.f);
        for (int k = h + 1; k < H; ++k) {
          if (adc_out) adc_out[k] = a0;
          if (tick_out) tick_out[k] = (float)(T - 2);
          if (raw_out) raw_out[k] = 0.f;
          if (st) { st->e[k] = T - 1; st->e2[k] = T - 1; st->cond[k] = 1; st->raw[k] = 0.f; }
        }
        if (st) st->n_done = h + 1;
      }
      __syncwarp();
      return;
    }
  }
  if (st && lane == 0) st->n_done = H;
  __syncwarp();
}

// Adjoint of fee_forward_sweep + cumsum: from dL/d(integrated charge) per hit
// (gint, identical in all lanes) to dL/dW[i] over T ticks, written to G.
// T must be a multiple of 4 and G 16-byte aligned.
static __device__ __noinline__ void fee_backward_sweep(const LsimParams &p, float *G, int T, const FeeState *st,
                                                const float *gint, int lane) {
  float4 *G4 = reinterpret_cast<float4 *>(G);
  for (int i = 4 * lane; i < T; i += kFeePass) G4[i / 4] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  // Hits skipped by the early exit have all-true masks, reset index T-1 and
  // no charge: each maps G to G - e_{T-1} sum(G).  After the first of them
  // sum(G) is zero, so one application is the whole chain.
  if (st->n_done < p.max_adc_values) {
    float S = 0.f;
    for (int i = 4 * lane; i < T; i += kFeePass) {
      const float4 g = G4[i / 4];
      S += (g.x + g.y) + (g.z + g.w);
    }
    S = warp_sum(S);
    __syncwarp();
    if (lane == 0) G[T - 1] -= S;
    __syncwarp();
  }
  // this lane's 64 keep bits of hit h (the next hit's are loaded ahead)
  auto keep_bits = [&](int h) {
    const uint2 m = *reinterpret_cast<const uint2 *>(st->mask + h * kMaskWords + 2 * lane);
    return (uint64_t)m.x | ((uint64_t)m.y << 32);
  };
  uint64_t kn = st->n_done > 0 ? keep_bits(st->n_done - 1) : 0u;
  for (int h = st->n_done - 1; h >= 0; --h) {
    uint64_t km = kn;
    if (h > 0) kn = keep_bits(h - 1);
    float S = 0.f;
    for (int i0 = 4 * lane; i0 < T; i0 += kFeePass, km >>= 4) {
      const uint32_t bits = (uint32_t)km;
      float4 g = G4[i0 / 4];
      if (bits & 1u) S += g.x; else g.x = 0.f;
      if (bits & 2u) S += g.y; else g.y = 0.f;
      if (bits & 4u) S += g.z; else g.z = 0.f;
      if (bits & 8u) S += g.w; else g.w = 0.f;
      G4[i0 / 4] = g;
    }
    S = warp_sum(S);
    __syncwarp();
    if (lane == 0) {
      G[st->e2[h]] -= S;
      if (!st->cond[h]) G[st->e[h]] += gint[h];
    }
    __syncwarp();
  }
  warp_suffix_charge<1>(G, T, p.t_sampling, lane);
}

// ---------------------------------------------------------------- threshold path
//
// After h resets a tick's charge is f_h(C), f_h(c) = max(f_{h-1}(c) - R_{h-1}, 0),
// the same function of the unreset charge C for every tick, and monotone in
// c with its roundings.  So "base + f_h(C) <= thr" and "base + f_h(C) >= thr"
// are comparisons of C with two thresholds, found exactly by a search over
// float bit patterns (the warp tests 30 neighbours of the real-number
// inverse at once).  The row is never rewritten: a crossing is looked for
// only in lanes whose smallest and largest values allow one, and C[e], C[e2]
// are replayed through the h resets.  Ticks, integrals and the adjoint are
// bit for bit those of the sweep path, at a cost per hit of about 100
// instructions per warp where a sweep of 2000 ticks takes about 1300.
// simulate_stochastic on 30000 rows of 2000 ticks with noise, this change
// alone: 809 -> 316 us (228 with the one-pass sums above and the leaner calls);
// the 64-event gradient step, where it is one phase of the pixel kernel: 18.71
// -> 17.92 ms.
// (The loops here are kept rolled: the code is hot inside the pixel kernels,
// whose instructions do not fit in the cache.)

// Total order of the floats as signed integers (and back).
__device__ __forceinline__ int float_key(float x) {
  const int b = __float_as_int(x);
  return b >= 0 ? b : (int)(0x80000000u - (uint32_t)b);
}
__device__ __forceinline__ float key_float(int k) {
  return __int_as_float(k >= 0 ? k : (int)(0x80000000u - (uint32_t)k));
}

// Charge of a tick after the first h resets (R in shared memory).
__device__ __forceinline__ float replay_resets(float c, const float *R, int h) {
#pragma unroll 1
  for (int k = 0; k < h; ++k) c = fmaxf(c - R[k], 0.f);
  return c;
}

// The smallest c in (-kFeeFastMax, kFeeFastMax) with base + f_h(c) >= thr
// and the smallest with base + f_h(c) > thr (-kFeeFastMax: everywhere,
// +infinity: nowhere).  guess: where to look first.
struct Crossing {
  float from, above;
};

__device__ __forceinline__ Crossing crossing_thresholds(float guess, float base, float thr, const float *R, int h,
                                                        int lane) {
  const int kmin = float_key(-kFeeFastMax), kmax = float_key(kFeeFastMax);
  int k0 = float_key(guess);
  k0 = k0 < kmin + 64 ? kmin + 64 : (k0 > kmax - 64 ? kmax - 64 : k0);
  const int key = lane == 0 ? kmin : (lane == kWarp - 1 ? kmax : k0 + lane - kWarp / 2);
  const float v = base + replay_resets(key_float(key), R, h);
  const unsigned m_from = __ballot_sync(0xffffffffu, v >= thr), m_above = __ballot_sync(0xffffffffu, v > thr);
  Crossing x;
#pragma unroll 1
  for (int strict = 0; strict < 2; ++strict) {   // (rolled: the code is hot in a large kernel)
    const unsigned m = strict ? m_above : m_from;
    float found;
    if (m & 1u) {
      found = -kFeeFastMax;
    } else if (!(m >> 31)) {
      found = (float)INFINITY;
    } else {
      int j = __ffs(m) - 1;                      // first lane that holds
      int lo = __shfl_sync(0xffffffffu, key, j - 1), hi = __shfl_sync(0xffffffffu, key, j);
      while ((uint32_t)hi - (uint32_t)lo > 1u) { // false at lo, true at hi; the span shrinks 33 times a round
        const uint32_t span = (uint32_t)hi - (uint32_t)lo;
        const uint32_t step = (uint32_t)(((uint64_t)span * (uint32_t)(lane + 1)) / (kWarp + 1));
        const int kt = (int)((uint32_t)lo + (step > 0 ? step : 1u));
        const float vt = base + replay_resets(key_float(kt), R, h);
        const unsigned mt = __ballot_sync(0xffffffffu, strict ? vt > thr : vt >= thr);
        j = mt ? __ffs(mt) - 1 : kWarp;
        const int below = __shfl_sync(0xffffffffu, kt, j > 0 ? j - 1 : 0);
        const int at = __shfl_sync(0xffffffffu, kt, j < kWarp ? j : 0);
        if (j < kWarp) hi = at;
        if (j > 0) lo = below;
      }
      found = key_float(hi);
    }
    (strict ? x.above : x.from) = found;
  }
  return x;
}

// (C here and below: the chunks' prefix sums, RowStats.)
// First i < T - 1 with C[i] < above and C[i + 1] >= from; T - 2 if none.
__device__ __forceinline__ int warp_crossing(const float *C, int T, const RowStats &rs, const Crossing &x, int lane) {
  const int per = chunk_ticks(T);
  for (unsigned m = __ballot_sync(0xffffffffu, rs.lo < x.above && rs.hi >= x.from); m; m &= m - 1) {
    const int chunk = __ffs(m) - 1, b = chunk * per, n = min(per, T - 1 - b);
    const float own = __shfl_sync(0xffffffffu, rs.offset, chunk);
    const float next = __shfl_sync(0xffffffffu, rs.offset, (chunk + 1) & (kWarp - 1));
#pragma unroll 1
    for (int j0 = 0; j0 < n; j0 += kWarp) {
      const int j = j0 + lane;
      const bool hit = j < n && own + C[b + j] < x.above && (j + 1 < per ? own : next) + C[b + j + 1] >= x.from;
      const unsigned bal = __ballot_sync(0xffffffffu, hit);
      if (bal) return b + j0 + __ffs(bal) - 1;
    }
  }
  return T - 2;
}

// Forward self-trigger on C (left as it is); st: the hits' state (its R
// serves every mode).  Outputs as fee_forward_sweep.  False (st and the
// outputs hold nothing) when a noise draw is not finite.
template <typename Noise>
__device__ __forceinline__ bool fee_forward_threshold(const LsimParams &p, const float *C, int T, const RowStats &rs,
                                                      const Noise &normals, float *adc_out, float *tick_out,
                                                      FeeState *st, float *raw_out, bool early_exit, int lane) {
  const float thr = p.threshold;
  const int H = p.max_adc_values;
  const bool noise = normals.src != nullptr;
  float base = noise ? normals[0] * p.reset_noise : 0.f;
  float top = rs.hi;   // the row's largest value, and what the resets leave of it
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  float left = top, sum_r = 0.f;
  float my_raw = 0.f, my_tick = (float)(T - 2);   // lane h: hit h; the empty hit's values
  int my_e = T - 1, my_e2 = T - 1, my_cond = 1;
  int done = H;
  for (int h = 0; h < H; ++h) {
    if (!(fabsf(base) < kFeeFastMax)) return false;
    int idx = T - 2;
    if (base + left >= thr)   // f_h is monotone: no tick reaches the threshold if the largest does not
      idx = warp_crossing(C, T, rs, crossing_thresholds((thr - base) + sum_r, base, thr, st->R, h, lane), lane);
    const int e = min(idx + 1 + p.fee_interval, T - 1), e2 = min(idx + 2 + p.fee_interval, T - 1);
    const float c = replay_resets(row_charge(C, rs, T, lane & 1 ? e2 : e), st->R, h);
    const float qvn = __shfl_sync(0xffffffffu, c, 0), R = __shfl_sync(0xffffffffu, c, 1);
    const float qv = base + qvn;
    const float extra = noise ? normals[1 + 3 * h] * p.uncorr_noise : 0.f;
    float adc = (qvn != 0.f) ? (qv + extra) : qvn;
    const bool cond = (adc < thr) || (idx == T - 2);
    if (cond) adc = 0.f;
    if (noise) {
      const float d2 = normals[2 + 3 * h], d3 = normals[3 + 3 * h];
      base = cond ? d3 * p.uncorr_noise : d2 * p.reset_noise;
    }
    if (lane == h) {
      my_raw = adc;
      my_tick = cond ? (float)(T - 2) : (float)idx;
      my_e = e;
      my_e2 = e2;
      my_cond = cond ? 1 : 0;
      st->R[h] = R;
    }
    __syncwarp();
    sum_r += R;
    left -= R;
    // once a rejected hit leaves nothing in the row, the later hits are empty
    if (early_exit && cond && left <= 0.f) {
      done = h + 1;
      break;
    }
    left = fmaxf(left, 0.f);
  }
  if (lane < H) {
    if (adc_out) adc_out[lane] = digitize(p, my_raw);
    if (tick_out) tick_out[lane] = my_tick;
    if (raw_out) raw_out[lane] = my_raw;
    st->e[lane] = my_e;
    st->e2[lane] = my_e2;
    st->cond[lane] = my_cond;
    st->raw[lane] = my_raw;
  }
  if (lane == 0) st->n_done = done;
  __syncwarp();
  return true;
}

// Adjoint of fee_forward_threshold + cumsum: C is replaced by dL/dW.  The
// cotangent of C is non-zero only at the hits' integration and reset ticks,
// at most two per hit: lane 2h stands for tick e_h, lane 2h + 1 for e2_h, and
// the lowest lane of a tick holds its cotangent.  A tick survives reset h if
// its replayed charge does, so going back over a reset only drops values;
// their sum is formed in the order of the sweeps (per owner of a tick's
// 4-tick group in ascending order, then across the warp).
template <int kUnroll>
__device__ __forceinline__ void fee_backward_threshold(const LsimParams &p, float *C, int T, const RowStats &rs,
                                                       const FeeState *st, const float *gint, int lane) {
  static_assert(2 * LSIM_MAX_HITS <= kWarp, "two entries per hit");
  const int n_done = st->n_done, mine = lane >> 1;
  const bool used = mine < n_done;
  const int tick = used ? ((lane & 1) ? st->e2[mine] : st->e[mine]) : -1 - lane;
  const unsigned same = __match_any_sync(0xffffffffu, tick);   // every lane takes part
  const bool holds = used && lane == __ffs(same) - 1;
  uint32_t keep = 0u;      // bit h: the tick survives reset h
  float c = row_charge(C, rs, T, used ? tick : 0);
#pragma unroll 1
  for (int h = 0; h < n_done; ++h) {
    const float d = c - st->R[h];
    keep |= d < 0.f ? 0u : 1u << h;
    c = fmaxf(d, 0.f);
  }
  float g = 0.f;
#pragma unroll 1
  for (int h = n_done - 1; h >= 0; --h) {
    if (!((keep >> h) & 1u)) g = 0.f;
    float S = 0.f;
    for (unsigned live = __ballot_sync(0xffffffffu, g != 0.f); live;) {
      const unsigned t = (live >> lane) & 1u ? (unsigned)tick : 0xffffffffu;
      const unsigned first = __reduce_min_sync(0xffffffffu, t);
      const unsigned at = __ballot_sync(0xffffffffu, t == first);
      const float x = __shfl_sync(0xffffffffu, g, __ffs(at) - 1);
      if ((int)(first / 4) % kWarp == lane) S += x;
      live &= ~at;
    }
    S = warp_sum(S);
    const int t1 = st->e2[h], t0 = st->e[h];
    if (holds && tick == t1) g -= S;
    if (holds && tick == t0 && !st->cond[h]) g += gint[h];
  }
  __syncwarp();
  float4 *C4 = reinterpret_cast<float4 *>(C);
#pragma unroll 1
  for (int i = 4 * lane; i < T; i += kFeePass) C4[i / 4] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  if (holds) C[tick] = g;
  __syncwarp();
  warp_suffix_charge<kUnroll>(C, T, p.t_sampling, lane);
}

// The front end on a row of cumulative charge: the threshold path where it
// applies, else the sweeps (which use the row up).  `masks`: whether the
// sweeps record their reset masks for the adjoint.  Returns whether the row
// was swept, which fee_backward needs to know.
template <typename Noise>
__device__ __forceinline__ bool fee_forward(const LsimParams &p, float *C, int T, const RowStats &rs,
                                            const Noise &normals, float *adc_out, float *tick_out, FeeState *st,
                                            bool masks, float *raw_out, bool early_exit, int lane) {
  if (rs.fast && fabsf(p.threshold) < kFeeFastMax &&
      fee_forward_threshold(p, C, T, rs, normals, adc_out, tick_out, st, raw_out, early_exit, lane))
    return false;
  add_offsets(C, T, rs, lane);
  fee_forward_sweep(p, C, T, normals.src, adc_out, tick_out, masks ? st : nullptr, raw_out, early_exit, lane);
  return true;
}

template <int kUnroll>
__device__ __forceinline__ void fee_backward(const LsimParams &p, float *C, int T, const RowStats &rs,
                                             const FeeState *st,
                                             const float *gint, bool swept, int lane) {
  if (swept)
    fee_backward_sweep(p, C, T, st, gint, lane);
  else
    fee_backward_threshold<kUnroll>(p, C, T, rs, st, gint, lane);
}

}  // namespace lsim
