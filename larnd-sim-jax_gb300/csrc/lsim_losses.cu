// Hit-level fit loss mse_adc (src/larndsim/losses_jax.py:13-39 rbf_kernel and
// mmd, :60-79 mse_adc): a weighted maximum mean discrepancy between the
// predicted hits and the reference hits with a Gaussian (RBF) kernel on the
// stacked coordinates (x + event * 1e5, y, z), plus a squared relative
// difference of the total charges.  Also its gradient with respect to the
// predicted weights w = Q * hit_prob and hit z (the coordinates with a
// gradient path: z depends on the drift velocity).
//
// The pairwise sums are computed row-wise: for each row hit i of one set and
// all column hits j of another, s_i = sum_j v_j K_ij and, for the predicted
// rows, s'_i = sum_j v_j K_ij (z_i - z_j).  Hits of different events are at
// least 1e5 - (detector size) apart in x, so their kernel value
// exp(-d / (2 sigma^2)) is exactly 0 in float32: inputs ordered by event (as
// the hit compaction emits them) make the cost per-event quadratic.
#include <cmath>

#include "lsim_internal.cuh"

namespace lsim {
namespace {

constexpr int kRbfRows = 128;    // chamfer: row hits per block (one per thread)
constexpr int kRbfChunk = 256;   // chamfer: column hits staged per chunk
constexpr float kEventOffset = 1e5f;

struct HitSet {
  const float *x, *y, *z, *w;
  const int32_t *event;
  int64_t n;
};

// per chunk of kRbfChunk hits: the smallest and largest event id
__global__ void k_chunk_events(const int32_t *__restrict__ event, int64_t n, int2 *__restrict__ ranges) {
  __shared__ int lo[kRbfChunk / 32], hi[kRbfChunk / 32];
  const int64_t i = (int64_t)blockIdx.x * kRbfChunk + threadIdx.x;
  int a = 0x7fffffff, b = -0x7fffffff - 1;
  if (i < n) a = b = event[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    lo[threadIdx.x >> 5] = a;
    hi[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kRbfChunk / 32; ++k) {
      a = min(a, lo[k]);
      b = max(b, hi[k]);
    }
    ranges[blockIdx.x] = make_int2(min(a, lo[0]), max(b, hi[0]));
  }
}

// ---------------------------------------------------------------- Gaussian pair sums
//
// s_i = sum_j w_j K_ij, sz_i = sum_j w_j K_ij (z_i - z_j) and, for the 4-d
// kernel, sq_i = sum_j w_j K_ij (q_i - q_j), with K_ij = exp(-d_ij / (2 sigma^2))
// evaluated as 2^(-d_ij log2(e) / (2 sigma^2)).
//
// Split: one warp owns a tile of 64 row hits (two per lane, advanced
// together in packed f32x2 operations) and walks the columns in chunks of
// 32, each staged once per warp in shared memory with its values doubled up
// for the packed operands.  Chunks with no event in common are passed over
// (their K is exactly 0), found 32 at a time by the lanes over a two-level
// list of event ranges.  Hits come in pixel order, so a chunk is short in y
// and x: chunks whose bounding box lies so far from the tile's that every
// K_ij is below 2^-kCutMse (mse_adc, 9.4 sigma) or 2^-kCutNll (nll, 11.8
// sigma) are passed over as well, about half of them on the 64-event batch
// (a spatial sort of the hits does not lower that: 32 hits fill a box of some
// cm).  A chunk or tile that holds an infinity or a NaN has an infinite box
// and is never passed over.
//
// What is left out so is bounded as the tile goes along (weights of a chunk
// times the largest K its box allows; kernel values below 2^-126, which the
// exponential flushes, the same way).  Where a row's sums are not 2^26 times
// that bound - a hit far from all others - they are formed again with expf,
// over every chunk whose K is not 0 in float32.
//
// A row's sums are formed per 32 chunks and those added up: at 64 events the
// z gradient's error against float64 is 1.9e-7 of its size (8.4e-7 with one
// running sum, more than with the exponential's own function, 8.3e-7).
//
// Bound by float32 issue: 10 packed operations and 2 exponentials per
// column for two rows, against about 23 operations per pair before.
// mse_adc with its gradient on the hits of 64 events (0.7M x 0.7M): 34.9 ->
// 5.87 ms; nll_loss on those of 8 events: 1.78 -> 0.43 ms.
// Few rows leave the chip idle, so the columns are dealt to pair_slices()
// warps per tile, whose partial sums are added in slice order.
constexpr int kPairTile = 64;     // row hits per warp
constexpr int kPairChunk = 32;    // column hits per chunk
constexpr int kPairSuper = 32;    // chunks per entry of the upper event-range list
constexpr int kPairWarps = 4;     // warps per block
constexpr int kPairMaxSlices = 16;
// below this the columns are sliced: 152 SMs x 32 warps, a constant so that the
// slices, hence the bits and the workspace, follow the counts of hits alone
constexpr int kPairWantWarps = 4864;
constexpr float kCutMse = 64.f, kCutNll = 100.f;
constexpr float kCutZero = 150.f;      // 2^-150 and below round to 0
constexpr float kLeftOut = 67108864.f; // 2^26: a quarter of a float32's last place
constexpr float kTiny = 1.1754944e-38f; // 2^-126, the smallest kernel value the fast exponential forms

// One set of hits as the pair kernel reads it: stacked coordinates and
// weight per hit (rounded up to whole chunks, weight 0 past the end), per
// chunk the event range, the box and the sum of |w|, per 32 chunks the event range.
struct PairSet {
  float4 *h;          // (stacked x, y, z, w)
  float *q;           // 4th coordinate or null
  int2 *ev, *ev_up;
  float4 *lo, *hi;    // box of a chunk (x, y, z, q)
  float *wsum;
  int64_t n;
};

inline int64_t pair_chunks(int64_t n) { return (n + kPairChunk - 1) / kPairChunk; }
inline int64_t pair_tiles(int64_t n) { return (n + kPairTile - 1) / kPairTile; }

// Column slices per row tile for a launch of `tiles` row tiles.
inline int pair_slices(int64_t tiles) {
  if (tiles <= 0) return 1;
  const int64_t want = (kPairWantWarps + tiles - 1) / tiles;
  return (int)(want < 1 ? 1 : want > kPairMaxSlices ? kPairMaxSlices : want);
}

struct PairSource {
  const float *x, *y, *z, *w, *q;
  const int32_t *event;
  float offset;       // stacked x = x + event * offset, float32 as the reference forms it
};

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Fills both sets: blocks [0, blocks_a) of 32 chunks belong to a, the rest to
// b; clears the tiles' counters.
__global__ void __launch_bounds__(kPairSuper * kPairChunk) k_pair_prepare(PairSource sa, PairSet a, int64_t blocks_a,
                                                                          PairSource sb, PairSet b, int32_t *done,
                                                                          int64_t n_done) {
  __shared__ int2 ranges[kPairSuper];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_done; i += (int64_t)gridDim.x * blockDim.x)
    done[i] = 0;
  const bool first = blockIdx.x < blocks_a;
  const PairSource &src = first ? sa : sb;
  const PairSet &set = first ? a : b;
  const int64_t blk = first ? blockIdx.x : blockIdx.x - blocks_a;
  const int lane = threadIdx.x % kPairChunk, wid = threadIdx.x / kPairChunk;
  const int64_t chunk = blk * kPairSuper + wid, i = chunk * kPairChunk + lane;
  const bool ok = i < set.n;
  float x = 0.f, y = 0.f, z = 0.f, q = 0.f, w = 0.f;
  int elo = 0x7fffffff, ehi = -0x7fffffff - 1;
  if (ok) {
    elo = ehi = src.event[i];
    x = __fadd_rn(src.x[i], __fmul_rn((float)elo, src.offset));
    if (fabsf(src.x[i]) > kEventOffset / 4) {   // may reach, or swallow, another event's offset: told apart by distance alone
      elo = -0x7fffffff - 1;
      ehi = 0x7fffffff;
    }
    y = src.y[i];
    z = src.z[i];
    w = src.w[i];
    if (src.q) q = src.q[i];
  }
  const bool odd = ok && !(isfinite(x) && isfinite(y) && isfinite(z) && isfinite(q) && isfinite(w));
  const bool any_odd = __any_sync(0xffffffffu, odd);
  const float wsum = warp_sum(fabsf(w));
  elo = __reduce_min_sync(0xffffffffu, elo);
  ehi = __reduce_max_sync(0xffffffffu, ehi);
  const float inf = INFINITY;
  float4 lo = make_float4(ok ? x : inf, ok ? y : inf, ok ? z : inf, ok ? q : inf);
  float4 hi = make_float4(ok ? x : -inf, ok ? y : -inf, ok ? z : -inf, ok ? q : -inf);
  lo = make_float4(warp_min(lo.x), warp_min(lo.y), warp_min(lo.z), warp_min(lo.w));
  hi = make_float4(warp_max(hi.x), warp_max(hi.y), warp_max(hi.z), warp_max(hi.w));
  if (any_odd) {
    lo = make_float4(-inf, -inf, -inf, -inf);
    hi = make_float4(inf, inf, inf, inf);
  }
  if (chunk * kPairChunk < set.n) {
    set.h[i] = make_float4(x, y, z, w);
    if (set.q) set.q[i] = q;
    if (lane == 0) {
      set.ev[chunk] = make_int2(elo, ehi);
      set.lo[chunk] = lo;
      set.hi[chunk] = hi;
      set.wsum[chunk] = wsum;
    }
  }
  if (lane == 0) ranges[wid] = make_int2(elo, ehi);
  __syncthreads();
  if (wid == 0) {
    const int2 r = ranges[lane];
    const int l = __reduce_min_sync(0xffffffffu, r.x), h = __reduce_max_sync(0xffffffffu, r.y);
    if (lane == 0) set.ev_up[blk] = make_int2(l, h);
  }
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Gap between two intervals (0 where they touch).
__device__ __forceinline__ float gap(float alo, float ahi, float blo, float bhi) {
  return fmaxf(0.f, fmaxf(blo - ahi, alo - bhi));
}

// -1 / (2 sigma^2) as the kernels use it: the fast exponent's factor in units
// of log2, and the exact one's in two parts (both of its sign and not 0, so
// that an infinite distance stays infinite).  Kept finite, so that hits at the
// same place have the kernel value 1 however small sigma is.
struct PairScale {
  float log2, hi, lo;
};

inline PairScale pair_scale(float sigma) {
  const double s = fmin(1.0 / (2.0 * (double)sigma * (double)sigma), 2e38);
  float hi = (float)s;
  if ((double)hi > s) hi = nextafterf(hi, 0.f);
  return PairScale{(float)(-1.4426950408889634074 * s), -hi, -fmaxf((float)(s - (double)hi), 1e-42f)};
}

// One job of the pair kernel: row tiles of `rows` against `cols`.  With
// `symmetric` (rows and cols the same set, only the total sum_i w_i s_i
// wanted) a tile takes its own two chunks once and the later ones twice.
struct PairJob {
  PairSet rows, cols;
  float *s, *sz, *sq;       // [slices][rows.n]
  int32_t *done;            // per tile, for several slices: slices with rows in doubt
  int64_t tiles;
  int slices;
  int symmetric;
};

constexpr int kPairSums = 6;    // s, sz, sq of the two rows
struct PairSmem {
  float4 col[3 * kPairChunk];
  float tot[kPairSums][32];
};

// This slice's share of the tile's sums over the columns, in sm.tot; left[]:
// this lane's part of a bound on what is left out of s, sz and sq.
template <bool FOUR_D, bool MOMENTS>
__device__ __forceinline__ void pair_sums(const PairJob &jb, int64_t tile, int slice, const PairScale &ps, float cut,
                                          PairSmem &sm, float (&left)[3], int lane) {
  const PairSet &R = jb.rows, &C = jb.cols;
  const int64_t i0 = tile * kPairTile + lane, i1 = i0 + kPairChunk;
  const int64_t nch = (C.n + kPairChunk - 1) / kPairChunk, rch = (R.n + kPairChunk - 1) / kPairChunk;
  // the tile is the rows' chunks 2 tile and 2 tile + 1
  const int64_t c0 = 2 * tile, c1 = min(c0 + 1, rch - 1);
  const int2 e0 = R.ev[c0], e1 = R.ev[c1];
  const int elo = min(e0.x, e1.x), ehi = max(e0.y, e1.y);
  const float4 la = R.lo[c0], lb = R.lo[c1], ha = R.hi[c0], hb = R.hi[c1];
  const float4 lo = make_float4(fminf(la.x, lb.x), fminf(la.y, lb.y), fminf(la.z, lb.z), fminf(la.w, lb.w));
  const float4 hi = make_float4(fmaxf(ha.x, hb.x), fmaxf(ha.y, hb.y), fmaxf(ha.z, hb.z), fmaxf(ha.w, hb.w));
  const float4 p0 = i0 < R.n ? R.h[i0] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 p1 = i1 < R.n ? R.h[i1] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float2 X = make_float2(p0.x, p1.x), Y = make_float2(p0.y, p1.y), Z = make_float2(p0.z, p1.z);
  float2 Q = make_float2(0.f, 0.f);
  if (FOUR_D) Q = make_float2(i0 < R.n ? R.q[i0] : 0.f, i1 < R.n ? R.q[i1] : 0.f);
  const float2 sc = make_float2(ps.log2, ps.log2);
#pragma unroll
  for (int q = 0; q < kPairSums; ++q) sm.tot[q][lane] = 0.f;
  left[0] = left[1] = left[2] = 0.f;
  const int64_t first = jb.symmetric ? c0 : 0;
  int turn = 0;
  for (int64_t u0 = (first / kPairSuper) & ~int64_t(31); u0 * kPairSuper < nch; u0 += 32) {
    bool up = false;
    if ((u0 + lane) * kPairSuper < nch) {
      const int2 r = C.ev_up[u0 + lane];
      up = r.y >= elo && r.x <= ehi;
    }
    for (unsigned um = __ballot_sync(0xffffffffu, up); um; um &= um - 1) {
      const int64_t cb = (u0 + (__ffs(um) - 1)) * kPairSuper, ch = cb + lane;
      bool near = false;
      if (ch >= first && ch < nch) {
        const int2 r = C.ev[ch];
        if (r.y >= elo && r.x <= ehi) {
          const float4 cl = C.lo[ch], cu = C.hi[ch];
          const float gx = gap(lo.x, hi.x, cl.x, cu.x), gy = gap(lo.y, hi.y, cl.y, cu.y);
          const float gz = gap(lo.z, hi.z, cl.z, cu.z), gq = FOUR_D ? gap(lo.w, hi.w, cl.w, cu.w) : 0.f;
          const float e = (gx * gx + gy * gy + gz * gz + gq * gq) * -ps.log2;
          near = !(e > cut);
          if (!(e > kCutZero)) {
            const float out = C.wsum[ch] * (near ? kTiny : fmaxf(ex2_approx(-e), kTiny));
            left[0] += out;
            if (MOMENTS) left[1] = fmaf(out, fmaxf(hi.z - cl.z, cu.z - lo.z), left[1]);
            if (MOMENTS && FOUR_D) left[2] = fmaf(out, fmaxf(hi.w - cl.w, cu.w - lo.w), left[2]);
          }
        }
      }
      unsigned cm = __ballot_sync(0xffffffffu, near);
      if (jb.slices > 1) {   // this slice's share: every slices-th chunk of those that count
        unsigned mine = 0u;
        for (unsigned m = cm; m; m &= m - 1) {
          if (turn == slice) mine |= m & (0u - m);
          turn = turn + 1 == jb.slices ? 0 : turn + 1;
        }
        cm = mine;
      }
      if (!cm) continue;
      int k = __ffs(cm) - 1;
      float4 v = C.h[(cb + k) * kPairChunk + lane];
      float vq = FOUR_D ? C.q[(cb + k) * kPairChunk + lane] : 0.f;
      float2 acc = make_float2(0.f, 0.f), accz = acc, accq = acc;
      while (cm) {
        const float wv = jb.symmetric && cb + k > c0 + 1 ? 2.f * v.w : v.w;
        __syncwarp();
        sm.col[lane * 3 + 0] = make_float4(-v.x, -v.x, -v.y, -v.y);
        sm.col[lane * 3 + 1] = make_float4(-v.z, -v.z, wv, wv);
        if (FOUR_D) sm.col[lane * 3 + 2] = make_float4(-vq, -vq, 0.f, 0.f);
        __syncwarp();
        cm &= cm - 1;
        if (cm) {   // the next chunk is in flight while this one is summed
          k = __ffs(cm) - 1;
          v = C.h[(cb + k) * kPairChunk + lane];
          if (FOUR_D) vq = C.q[(cb + k) * kPairChunk + lane];
        }
#pragma unroll 8
        for (int j = 0; j < kPairChunk; ++j) {
          const float4 a = sm.col[3 * j], b = sm.col[3 * j + 1];
          const float2 dx = __fadd2_rn(X, make_float2(a.x, a.y)), dy = __fadd2_rn(Y, make_float2(a.z, a.w));
          const float2 dz = __fadd2_rn(Z, make_float2(b.x, b.y));
          float2 d = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
          float2 dq;
          if (FOUR_D) {
            const float4 c = sm.col[3 * j + 2];
            dq = __fadd2_rn(Q, make_float2(c.x, c.y));
            d = __ffma2_rn(dq, dq, d);
          }
          const float2 e = __fmul2_rn(d, sc);
          const float2 kw = __fmul2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), make_float2(b.z, b.w));
          acc = __fadd2_rn(acc, kw);
          if (MOMENTS) accz = __ffma2_rn(kw, dz, accz);
          if (MOMENTS && FOUR_D) accq = __ffma2_rn(kw, dq, accq);
        }
      }
      sm.tot[0][lane] += acc.x;
      sm.tot[1][lane] += acc.y;
      if (MOMENTS) {
        sm.tot[2][lane] += accz.x;
        sm.tot[3][lane] += accz.y;
      }
      if (MOMENTS && FOUR_D) {
        sm.tot[4][lane] += accq.x;
        sm.tot[5][lane] += accq.y;
      }
    }
  }
}

// One row's sums over all columns whose kernel value is not 0 in float32, with
// expf, by the whole warp; into the first slice's place, zeros into the others.
// (Few rows: kept out of line.)
template <bool FOUR_D, bool MOMENTS>
__device__ __noinline__ void pair_row_exact(const PairJob &jb, int64_t i, const PairScale &ps, int lane) {
  const PairSet &R = jb.rows, &C = jb.cols;
  const int64_t nch = (C.n + kPairChunk - 1) / kPairChunk, own = i / kPairTile * 2;   // own: the tile's first chunk
  const float4 p = R.h[i];
  const float pq = FOUR_D ? R.q[i] : 0.f;
  const int2 ev = R.ev[i / kPairChunk];
  const bool odd = !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(pq));
  float acc = 0.f, accz = 0.f, accq = 0.f;
  for (int64_t cb = jb.symmetric ? own : 0; cb < nch; cb += 32) {
    const int64_t ch = cb + lane;
    bool near = false;
    if (ch < nch) {
      const int2 r = C.ev[ch];
      if (r.y >= ev.x && r.x <= ev.y) {
        const float4 cl = C.lo[ch], cu = C.hi[ch];
        const float gx = gap(p.x, p.x, cl.x, cu.x), gy = gap(p.y, p.y, cl.y, cu.y), gz = gap(p.z, p.z, cl.z, cu.z);
        const float gq = FOUR_D ? gap(pq, pq, cl.w, cu.w) : 0.f;
        near = odd || !((gx * gx + gy * gy + gz * gz + gq * gq) * -ps.log2 > kCutZero);
      }
    }
    for (unsigned m = __ballot_sync(0xffffffffu, near); m; m &= m - 1) {
      const int64_t k = cb + __ffs(m) - 1, j = k * kPairChunk + lane;
      const float4 v = C.h[j];
      const float dx = p.x - v.x, dy = p.y - v.y, dz = p.z - v.z, dq = FOUR_D ? pq - C.q[j] : 0.f;
      float d = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      if (FOUR_D) d = fmaf(dq, dq, d);
      const float kw = expf(fmaf(d, ps.hi, d * ps.lo)) * (jb.symmetric && k > own + 1 ? 2.f * v.w : v.w);
      acc += kw;
      if (MOMENTS) accz = fmaf(kw, dz, accz);
      if (MOMENTS && FOUR_D) accq = fmaf(kw, dq, accq);
    }
  }
  acc = warp_sum(acc);
  if (MOMENTS) accz = warp_sum(accz);
  if (MOMENTS && FOUR_D) accq = warp_sum(accq);
  __syncwarp();            // after the tile's own stores
  if (lane < jb.slices) {
    const int64_t o = lane * R.n + i;
    jb.s[o] = lane == 0 ? acc : 0.f;
    if (MOMENTS) jb.sz[o] = lane == 0 ? accz : 0.f;
    if (MOMENTS && FOUR_D) jb.sq[o] = lane == 0 ? accq : 0.f;
  }
}
static_assert(kPairMaxSlices <= 32, "a lane per slice");

template <bool FOUR_D, bool MOMENTS>
__device__ __forceinline__ void pair_tile(const PairJob &jb, int64_t tile, int slice, const PairScale &ps, float cut,
                                          PairSmem &sm, int lane) {
  constexpr int N = MOMENTS ? (FOUR_D ? 3 : 2) : 1;
  float left[3];
  pair_sums<FOUR_D, MOMENTS>(jb, tile, slice, ps, cut, sm, left, lane);
#pragma unroll
  for (int q = 0; q < 2 * N; ++q) {
    const int64_t i = tile * kPairTile + (q & 1) * kPairChunk + lane;
    float *dst = q < 2 ? jb.s : q < 4 ? jb.sz : jb.sq;
    if (i < jb.rows.n) dst[(int64_t)slice * jb.rows.n + i] = sm.tot[q][lane];
  }
  // rows in doubt: what is left out may show in their sums' last place
  auto in_doubt = [&](auto &&sum_of, bool (&unsure)[2]) {
    unsure[0] = unsure[1] = false;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const float bound = warp_sum(left[q]) * kLeftOut;
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (tile * kPairTile + r * kPairChunk + lane < jb.rows.n)
          unsure[r] |= !(fabsf(sum_of(q, r)) >= bound);   // (a NaN too)
    }
    return __any_sync(0xffffffffu, unsure[0] || unsure[1]);
  };
  bool unsure[2];
  if (!in_doubt([&](int q, int r) { return sm.tot[2 * q + r][lane]; }, unsure)) return;
  if (jb.slices > 1) {     // none if a slice has none; the last slice looks at the totals
    __threadfence();
    __syncwarp();
    int before = 0;
    if (lane == 0) before = atomicAdd(jb.done + tile, 1);
    if (__shfl_sync(0xffffffffu, before, 0) != jb.slices - 1) return;
    __threadfence();
    in_doubt([&](int q, int r) {
      const float *src = (q == 0 ? jb.s : q == 1 ? jb.sz : jb.sq) + tile * kPairTile + r * kPairChunk + lane;
      float t = 0.f;
      for (int k = 0; k < jb.slices; ++k) t += __ldcg(src + k * jb.rows.n);
      return t;
    }, unsure);
  }
#pragma unroll 1
  for (int r = 0; r < 2; ++r)
    for (unsigned m = __ballot_sync(0xffffffffu, r ? unsure[1] : unsure[0]); m; m &= m - 1)
      pair_row_exact<FOUR_D, MOMENTS>(jb, tile * kPairTile + r * kPairChunk + __ffs(m) - 1, ps, lane);
}

// Up to three jobs in one launch (their warps follow one another, so one
// job's last warps run beside the next job's first).
struct PairJobs {
  PairJob job[3];
  int n;
};

template <bool FOUR_D>
__global__ void __launch_bounds__(kPairWarps * 32) k_pair_rows(PairJobs jobs, PairScale ps, float cut) {
  __shared__ PairSmem sm[kPairWarps];
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  int64_t t = (int64_t)blockIdx.x * kPairWarps + wid;
  for (int k = 0; k < jobs.n; ++k) {
    const PairJob &jb = jobs.job[k];
    const int64_t count = jb.tiles * jb.slices;
    if (t < count) {
      const int64_t tile = t / jb.slices;
      const int slice = (int)(t - tile * jb.slices);
      if (jb.sz)
        pair_tile<FOUR_D, true>(jb, tile, slice, ps, cut, sm[wid], lane);
      else
        pair_tile<FOUR_D, false>(jb, tile, slice, ps, cut, sm[wid], lane);
      return;
    }
    t -= count;
  }
}

// sum over the slices of a row's partial sums, in slice order
__device__ __forceinline__ float slice_sum(const float *__restrict__ s, int64_t n, int slices, int64_t i) {
  float v = s[i];
  for (int k = 1; k < slices; ++k) v += s[k * n + i];
  return v;
}

template <bool FOUR_D>
void launch_pair_rows(const PairJobs &jobs, float sigma, float cut, cudaStream_t st) {
  int64_t warps = 0;
  for (int k = 0; k < jobs.n; ++k) warps += jobs.job[k].tiles * jobs.job[k].slices;
  if (warps <= 0) return;
  k_pair_rows<FOUR_D><<<(unsigned)((warps + kPairWarps - 1) / kPairWarps), kPairWarps * 32, 0, st>>>(
      jobs, pair_scale(sigma), cut);
}

// workspace carving; base null: sizes only
struct Carver {
  char *base;
  size_t off;
  char *take(size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) & ~size_t(255);
    return base ? base + at : nullptr;
  }
  float *floats(int64_t n) { return reinterpret_cast<float *>(take(4 * (size_t)n)); }
};

PairSet take_pair_set(Carver &c, int64_t n, bool four_d) {
  const int64_t ch = pair_chunks(n), up = (ch + kPairSuper - 1) / kPairSuper;
  PairSet s;
  s.h = reinterpret_cast<float4 *>(c.take(sizeof(float4) * (size_t)(ch * kPairChunk)));
  s.q = four_d ? c.floats(ch * kPairChunk) : nullptr;
  s.ev = reinterpret_cast<int2 *>(c.take(sizeof(int2) * (size_t)ch));
  s.ev_up = reinterpret_cast<int2 *>(c.take(sizeof(int2) * (size_t)up));
  s.lo = reinterpret_cast<float4 *>(c.take(sizeof(float4) * (size_t)ch));
  s.hi = reinterpret_cast<float4 *>(c.take(sizeof(float4) * (size_t)ch));
  s.wsum = c.floats(ch);
  s.n = n;
  return s;
}

void launch_pair_prepare(const PairSource &sa, const PairSet &a, const PairSource &sb, const PairSet &b,
                         int32_t *done, int64_t n_done, cudaStream_t st) {
  auto blocks = [](int64_t n) { return (pair_chunks(n) + kPairSuper - 1) / kPairSuper; };
  const int64_t ba = blocks(a.n), bb = blocks(b.n);
  if (ba + bb > 0)
    k_pair_prepare<<<(unsigned)(ba + bb), kPairSuper * kPairChunk, 0, st>>>(sa, a, ba, sb, b, done, n_done);
}

struct MseAdcTotals {
  double sw, sv, A, B, C;
  double ga, gb, g0, za, zb;   // dL/dw_i = ga a_i + gb b_i + g0, dL/dz_i = w_i (za az_i + zb bz_i)
  float loss, mmd, charge;
};

// Block sums of up to kRedMax doubles per thread: warp sums, then a thread per
// sum adds the warps' in order into out[q].  (At most kRedBlocks blocks, a
// constant for the same reason as the slices.)
constexpr int kRedBlocks = 304, kRedThreads = 256, kRedMax = 5;

template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double (*red)[32], double *out) {
#pragma unroll
  for (int q = 0; q < N; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v[q];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[threadIdx.x][k];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// Per block the sums (sum w, sum v, sum w a, sum w b, sum v c) of its share
// of the hits, strided so that the shares depend only on the counts.  One
// block over all hits took 1.8 ms on the 64-event batch.
__global__ void __launch_bounds__(kRedThreads) k_mse_adc_sums(HitSet pred, HitSet ref, const float *__restrict__ a,
                                                              const float *__restrict__ b, int slices_p,
                                                              const float *__restrict__ c, int slices_r,
                                                              double *__restrict__ parts) {
  __shared__ double red[kRedMax][32];
  double v[kRedMax] = {0, 0, 0, 0, 0};
  const int64_t step = (int64_t)gridDim.x * kRedThreads, at = (int64_t)blockIdx.x * kRedThreads + threadIdx.x;
  for (int64_t i = at; i < pred.n; i += step) {
    const double w = pred.w[i];
    v[0] += w;
    v[2] += w * slice_sum(a, pred.n, slices_p, i);
    v[3] += w * slice_sum(b, pred.n, slices_p, i);
  }
  for (int64_t j = at; j < ref.n; j += step) {
    const double w = ref.w[j];
    v[1] += w;
    v[4] += w * slice_sum(c, ref.n, slices_r, j);
  }
  block_sums(v, red, parts + (size_t)blockIdx.x * kRedMax);
}

// one block: the totals, the loss and the gradients' coefficients
__global__ void __launch_bounds__(kRedThreads) k_mse_adc_reduce(const double *__restrict__ parts, int n_parts,
                                                                float lambda_q, float inv_sigma2, MseAdcTotals *tot,
                                                                float *out) {
  __shared__ double red[kRedMax][32];
  __shared__ double t[kRedMax];
  double v[kRedMax] = {0, 0, 0, 0, 0};
  for (int k = threadIdx.x; k < n_parts; k += kRedThreads)
#pragma unroll
    for (int q = 0; q < kRedMax; ++q) v[q] += parts[(size_t)k * kRedMax + q];
  block_sums(v, red, t);
  if (threadIdx.x == 0) {
    MseAdcTotals r;
    r.sw = t[0];
    r.sv = t[1];
    r.A = t[2];
    r.B = t[3];
    r.C = t[4];
    const double sw2 = r.sw * r.sw, swsv = r.sw * r.sv;
    const double mmd = r.A / sw2 + r.C / (r.sv * r.sv) - 2.0 * r.B / swsv;
    const double rel = (r.sw - r.sv) / (r.sv + 1e-6);
    const double dc = 2.0 * (r.sw - r.sv) / ((r.sv + 1e-6) * (r.sv + 1e-6));
    r.ga = 2.0 / sw2;
    r.gb = -2.0 / swsv;
    r.g0 = -2.0 * r.A / (sw2 * r.sw) + 2.0 * r.B / (sw2 * r.sv) + (double)lambda_q * dc;
    r.za = -2.0 * (double)inv_sigma2 / sw2;
    r.zb = 2.0 * (double)inv_sigma2 / swsv;
    r.mmd = (float)mmd;
    r.charge = (float)(rel * rel);
    r.loss = (float)(mmd + (double)lambda_q * rel * rel);
    *tot = r;
    out[0] = r.loss;
    out[1] = r.mmd;
    out[2] = r.charge;
  }
}

// dL/dw_i and dL/dz_i of L = mmd + lambda_q * charge
__global__ void k_mse_adc_grad(HitSet pred, const float *__restrict__ a, const float *__restrict__ b,
                               const float *__restrict__ az, const float *__restrict__ bz, int slices,
                               const MseAdcTotals *__restrict__ tot, float *__restrict__ gw, float *__restrict__ gz) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pred.n) return;
  if (gw)
    gw[i] = (float)(tot->ga * slice_sum(a, pred.n, slices, i) + tot->gb * slice_sum(b, pred.n, slices, i) + tot->g0);
  if (gz)
    gz[i] = (float)((double)pred.w[i] * (tot->za * slice_sum(az, pred.n, slices, i) +
                                         tot->zb * slice_sum(bz, pred.n, slices, i)));
}

// ---------------------------------------------------------------- nll_loss and chamfer_3d
// Both stack (x + event * 1e9, y, z[, Q / adc_norm]) (losses_jax.py:221-222,
// :337-338); hits of different events are 1e9 apart and never interact.

struct HitSet4 {
  const float *x, *y, *z, *q, *w;   // q: 4th coordinate (nll) or null
  const int32_t *event;
  int64_t n;
};

__device__ __forceinline__ float stacked_x9(const HitSet4 &h, int64_t i) {
  return __fadd_rn(h.x[i], __fmul_rn((float)h.event[i], 1e9f));
}

// block-wide event range of the row tile into (lo, hi)
__device__ __forceinline__ void tile_event_range(bool ok, int ev, int *lo_s, int *hi_s, int &lo, int &hi) {
  int a = ok ? ev : 0x7fffffff, b = ok ? ev : -0x7fffffff - 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  if (threadIdx.x == 0) {
    *lo_s = 0x7fffffff;
    *hi_s = -0x7fffffff - 1;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicMin(lo_s, a);
    atomicMax(hi_s, b);
  }
  __syncthreads();
  lo = *lo_s;
  hi = *hi_s;
}

// Weights of the second nll pass, (ref_hit_prob > 0.5) / (lambda + 1e-10),
// into the reference set, and per block (sum hit_prob, sum log(lambda + 1e-10)).
__global__ void __launch_bounds__(kRedThreads) k_nll_mid(const float *__restrict__ hp, int64_t n,
                                                         const float *__restrict__ ref_hp,
                                                         const float *__restrict__ lam, int slices, PairSet ref,
                                                         double *__restrict__ parts) {
  __shared__ double red[2][32];
  double v[2] = {0, 0};
  const int64_t step = (int64_t)gridDim.x * kRedThreads, at = (int64_t)blockIdx.x * kRedThreads + threadIdx.x;
  for (int64_t i = at; i < n; i += step) v[0] += hp[i];
  for (int64_t j0 = at & ~int64_t(31); j0 < ref.n; j0 += step) {   // a warp a chunk
    const int64_t j = j0 + threadIdx.x % 32;
    const bool in = j < ref.n;
    const float l = (in ? slice_sum(lam, ref.n, slices, j) : 0.f) + 1e-10f;
    const bool on = in && ref_hp[j] > 0.5f;
    const float w = on ? 1.0f / l : 0.0f;
    if (in) ref.h[j].w = w;
    if (on) v[1] += (double)logf(l);
    const float wsum = warp_sum(fabsf(w));
    const bool odd = __any_sync(0xffffffffu, !isfinite(w));
    if (threadIdx.x % 32 == 0) {
      ref.wsum[j / kPairChunk] = wsum;
      if (odd) {   // never passed over by its distance
        const float inf = INFINITY;
        ref.lo[j / kPairChunk] = make_float4(-inf, -inf, -inf, -inf);
        ref.hi[j / kPairChunk] = make_float4(inf, inf, inf, inf);
      }
    }
  }
  block_sums(v, red, parts + (size_t)blockIdx.x * 2);
}

__global__ void __launch_bounds__(kRedThreads) k_nll_reduce(const double *__restrict__ parts, int n_parts,
                                                            float *out) {
  __shared__ double red[2][32];
  __shared__ double t[2];
  double v[2] = {0, 0};
  for (int k = threadIdx.x; k < n_parts; k += kRedThreads) {
    v[0] += parts[2 * (size_t)k];
    v[1] += parts[2 * (size_t)k + 1];
  }
  block_sums(v, red, t);
  if (threadIdx.x == 0) {
    out[0] = (float)(t[0] - t[1]);
    out[1] = (float)t[0];
    out[2] = (float)t[1];
  }
}

__global__ void k_nll_grad(const float *__restrict__ hp, int64_t n, const float *__restrict__ s,
                           const float *__restrict__ sz, const float *__restrict__ sq, int slices, float inv_sigma2,
                           float *__restrict__ g_hp, float *__restrict__ g_z, float *__restrict__ g_q) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (g_hp) g_hp[i] = 1.0f - slice_sum(s, n, slices, i);
  if (g_z) g_z[i] = hp[i] * inv_sigma2 * slice_sum(sz, n, slices, i);
  if (g_q) g_q[i] = hp[i] * inv_sigma2 * slice_sum(sq, n, slices, i);
}

// chamfer: nearest column of every row (first index on ties) and its
// squared distance; rows with no column in their events get (inf, -1)
__global__ void __launch_bounds__(kRbfRows) k_nn_rows(HitSet4 rows, HitSet4 cols, const int2 *__restrict__ col_ranges,
                                                      float *__restrict__ dmin, int32_t *__restrict__ amin) {
  __shared__ float cx[kRbfChunk], cy[kRbfChunk], cz[kRbfChunk];
  __shared__ int lo_s, hi_s;
  const int64_t i = (int64_t)blockIdx.x * kRbfRows + threadIdx.x;
  const bool ok = i < rows.n;
  float xi = 0.f, yi = 0.f, zi = 0.f;
  int ev = 0;
  if (ok) {
    xi = stacked_x9(rows, i);
    yi = rows.y[i];
    zi = rows.z[i];
    ev = rows.event[i];
  }
  int lo, hi;
  tile_event_range(ok, ev, &lo_s, &hi_s, lo, hi);
  float best = INFINITY;
  int64_t arg = -1;
  const int64_t n_chunks = (cols.n + kRbfChunk - 1) / kRbfChunk;
  for (int64_t c = 0; c < n_chunks; ++c) {
    const int2 r = col_ranges[c];
    if (r.y < lo || r.x > hi) continue;   // 1e9 apart: never the nearest when the row's event has columns
    const int64_t j0 = c * kRbfChunk;
    const int cnt = cols.n - j0 < kRbfChunk ? (int)(cols.n - j0) : kRbfChunk;
    __syncthreads();
    for (int k = threadIdx.x; k < cnt; k += kRbfRows) {
      cx[k] = stacked_x9(cols, j0 + k);
      cy[k] = cols.y[j0 + k];
      cz[k] = cols.z[j0 + k];
    }
    __syncthreads();
    if (ok) {
      for (int k = 0; k < cnt; ++k) {
        const float dx = __fsub_rn(xi, cx[k]), dy = __fsub_rn(yi, cy[k]), dz = __fsub_rn(zi, cz[k]);
        const float d = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
        if (d < best) {
          best = d;
          arg = j0 + k;
        }
      }
    }
  }
  if (ok) {
    dmin[i] = best;
    amin[i] = (int32_t)arg;
  }
}

// chamfer gradient gathers for predicted row i over the reference hits j
// whose nearest predicted hit is i: sum of mb_j wb_j and of wb_j 2 (z_i - z_j)
__global__ void __launch_bounds__(kRbfRows) k_chamfer_back(HitSet4 rows, HitSet4 cols,
                                                           const int2 *__restrict__ col_ranges,
                                                           const float *__restrict__ col_dmin,
                                                           const int32_t *__restrict__ col_amin,
                                                           float *__restrict__ acc_w, float *__restrict__ acc_z) {
  __shared__ float cz[kRbfChunk], cw[kRbfChunk], cd[kRbfChunk];
  __shared__ int ca[kRbfChunk];
  __shared__ int lo_s, hi_s;
  const int64_t i = (int64_t)blockIdx.x * kRbfRows + threadIdx.x;
  const bool ok = i < rows.n;
  const int ev = ok ? rows.event[i] : 0;
  const float zi = ok ? rows.z[i] : 0.f;
  int lo, hi;
  tile_event_range(ok, ev, &lo_s, &hi_s, lo, hi);
  double aw = 0.0, az = 0.0;
  const int64_t n_chunks = (cols.n + kRbfChunk - 1) / kRbfChunk;
  for (int64_t c = 0; c < n_chunks; ++c) {
    const int2 r = col_ranges[c];
    if (r.y < lo || r.x > hi) continue;
    const int64_t j0 = c * kRbfChunk;
    const int cnt = cols.n - j0 < kRbfChunk ? (int)(cols.n - j0) : kRbfChunk;
    __syncthreads();
    for (int k = threadIdx.x; k < cnt; k += kRbfRows) {
      cz[k] = cols.z[j0 + k];
      cw[k] = cols.w[j0 + k];
      cd[k] = col_dmin[j0 + k];
      ca[k] = col_amin[j0 + k];
    }
    __syncthreads();
    if (ok) {
      for (int k = 0; k < cnt; ++k) {
        if (ca[k] == (int)i && cd[k] < 1e4f) {
          aw += (double)cd[k] * (double)cw[k];
          az += (double)cw[k] * 2.0 * (double)__fsub_rn(zi, cz[k]);
        }
      }
    }
  }
  if (ok) {
    acc_w[i] = (float)aw;
    acc_z[i] = (float)az;
  }
}

// loss and gradients of chamfer_distance_3d_og (losses_jax.py:181-211)
__global__ void k_chamfer_reduce(const float *__restrict__ wa, int64_t n, const float *__restrict__ wb, int64_t m,
                                 const float *__restrict__ ma, const int32_t *__restrict__ ia,
                                 const float *__restrict__ mb, const int32_t *__restrict__ ib, float *out) {
  __shared__ double red[32];
  double t = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    if (ma[i] < 1e4f) t += (double)ma[i] * wa[i] * wb[ia[i]];
  for (int64_t j = threadIdx.x; j < m; j += blockDim.x)
    if (mb[j] < 1e4f) t += (double)mb[j] * wb[j] * wa[ib[j]];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) a += red[k];
    out[0] = (float)a;
  }
}

__global__ void k_chamfer_grad(HitSet4 pred, HitSet4 ref, const float *__restrict__ ma,
                               const int32_t *__restrict__ ia, const float *__restrict__ acc_w,
                               const float *__restrict__ acc_z, float *__restrict__ g_w, float *__restrict__ g_z) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pred.n) return;
  double gw = acc_w[i], gz = (double)pred.w[i] * acc_z[i];
  if (ma[i] < 1e4f) {
    const int j = ia[i];
    gw += (double)ma[i] * ref.w[j];
    gz += (double)pred.w[i] * ref.w[j] * 2.0 * (double)__fsub_rn(pred.z[i], ref.z[j]);
  }
  if (g_w) g_w[i] = (float)gw;
  if (g_z) g_z[i] = (float)gz;
}

struct MseAdcWs {
  PairSet pred, ref;
  float *a, *az, *b, *bz, *c;
  int slices;      // column slices of every job
  int32_t *done;   // per tile of the three jobs
  double *parts;
  MseAdcTotals *tot;
};

size_t mse_adc_layout(int64_t n, int64_t m, MseAdcWs *w, char *base) {
  Carver c{base, 0};
  MseAdcWs s;
  s.slices = pair_slices(2 * pair_tiles(n) + pair_tiles(m));
  s.pred = take_pair_set(c, n, false);
  s.ref = take_pair_set(c, m, false);
  s.a = c.floats(n * s.slices);
  s.az = c.floats(n * s.slices);
  s.b = c.floats(n * s.slices);
  s.bz = c.floats(n * s.slices);
  s.c = c.floats(m * s.slices);
  s.done = reinterpret_cast<int32_t *>(c.floats(2 * pair_tiles(n) + pair_tiles(m)));
  s.parts = reinterpret_cast<double *>(c.take(sizeof(double) * kRedBlocks * kRedMax));
  s.tot = reinterpret_cast<MseAdcTotals *>(c.take(sizeof(MseAdcTotals)));
  if (w) *w = s;
  return c.off;
}

struct NllWs {
  PairSet pred, ref;
  float *s, *sz, *sq, *lam;
  int slices_p, slices_r;
  int32_t *done;   // per tile of the two jobs
  double *parts;
};

size_t nll_layout(int64_t n, int64_t m, NllWs *w, char *base) {
  Carver c{base, 0};
  NllWs s;
  s.slices_p = pair_slices(pair_tiles(n));
  s.slices_r = pair_slices(pair_tiles(m));
  s.pred = take_pair_set(c, n, true);
  s.ref = take_pair_set(c, m, true);
  s.s = c.floats(n * s.slices_p);
  s.sz = c.floats(n * s.slices_p);
  s.sq = c.floats(n * s.slices_p);
  s.lam = c.floats(m * s.slices_r);
  s.done = reinterpret_cast<int32_t *>(c.floats(pair_tiles(n) + pair_tiles(m)));
  s.parts = reinterpret_cast<double *>(c.take(sizeof(double) * kRedBlocks * 2));
  if (w) *w = s;
  return c.off;
}

// blocks of the partial-sum kernels for n hits
inline unsigned red_blocks(int64_t n) {
  const int64_t b = (n + kRedThreads - 1) / kRedThreads;
  return (unsigned)(b < 1 ? 1 : b > kRedBlocks ? kRedBlocks : b);
}

}  // namespace

size_t mse_adc_workspace_bytes(int64_t n, int64_t m) { return mse_adc_layout(n, m, nullptr, nullptr); }

int run_mse_adc(const float *x, const float *y, const float *z, const int32_t *event, const float *w, int64_t n,
                const float *rx, const float *ry, const float *rz, const int32_t *revent, const float *rw, int64_t m,
                float sigma, float lambda_q, float *out, float *grad_w, float *grad_z, void *ws, cudaStream_t st) {
  MseAdcWs s;
  mse_adc_layout(n, m, &s, static_cast<char *>(ws));
  const HitSet pred{x, y, z, w, event, n}, ref{rx, ry, rz, rw, revent, m};
  const int64_t tn = pair_tiles(n), tm = pair_tiles(m);
  launch_pair_prepare(PairSource{x, y, z, w, nullptr, event, kEventOffset}, s.pred,
                      PairSource{rx, ry, rz, rw, nullptr, revent, kEventOffset}, s.ref, s.done, 2 * tn + tm, st);
  PairJobs jobs;
  jobs.n = 3;
  jobs.job[0] = PairJob{s.pred, s.pred, s.a, s.az, nullptr, s.done, tn, s.slices, 0};
  jobs.job[1] = PairJob{s.pred, s.ref, s.b, s.bz, nullptr, s.done + tn, tn, s.slices, 0};
  jobs.job[2] = PairJob{s.ref, s.ref, s.c, nullptr, nullptr, s.done + 2 * tn, tm, s.slices, 1};
  launch_pair_rows<false>(jobs, sigma, kCutMse, st);
  const unsigned rb = red_blocks(n > m ? n : m);
  k_mse_adc_sums<<<rb, kRedThreads, 0, st>>>(pred, ref, s.a, s.b, s.slices, s.c, s.slices, s.parts);
  k_mse_adc_reduce<<<1, kRedThreads, 0, st>>>(s.parts, (int)rb, lambda_q,
                                              (float)(1.0 / ((double)sigma * (double)sigma)), s.tot, out);
  if (n > 0 && (grad_w || grad_z))
    k_mse_adc_grad<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(pred, s.a, s.b, s.az, s.bz, s.slices, s.tot, grad_w,
                                                                grad_z);
  return LSIM_OK;
}

// nll_loss: out[0..2] = loss, sum of hit_prob, sum of log(lambda + 1e-10)
size_t nll_workspace_bytes(int64_t n, int64_t m) { return nll_layout(n, m, nullptr, nullptr); }

int run_nll(const float *x, const float *y, const float *z, const float *q, const int32_t *event, const float *hp,
            int64_t n, const float *rx, const float *ry, const float *rz, const float *rq, const int32_t *revent,
            const float *rhp, int64_t m, float sigma, float *out, float *g_q, float *g_z, float *g_hp, void *ws,
            cudaStream_t st) {
  NllWs s;
  nll_layout(n, m, &s, static_cast<char *>(ws));
  const int64_t tn = pair_tiles(n), tm = pair_tiles(m);
  launch_pair_prepare(PairSource{x, y, z, hp, q, event, 1e9f}, s.pred, PairSource{rx, ry, rz, rhp, rq, revent, 1e9f},
                      s.ref, s.done, tn + tm, st);
  PairJobs jobs;
  jobs.n = 1;
  // lambda_j = sum_i hp_i K_ij, then the reference hits weigh 1 / lambda_j
  jobs.job[0] = PairJob{s.ref, s.pred, s.lam, nullptr, nullptr, s.done + tn, tm, s.slices_r, 0};
  launch_pair_rows<true>(jobs, sigma, kCutNll, st);
  const unsigned rb = red_blocks(n > m ? n : m);
  k_nll_mid<<<rb, kRedThreads, 0, st>>>(hp, n, rhp, s.lam, s.slices_r, s.ref, s.parts);
  k_nll_reduce<<<1, kRedThreads, 0, st>>>(s.parts, (int)rb, out);
  if (n > 0 && (g_q || g_z || g_hp)) {
    jobs.job[0] = PairJob{s.pred, s.ref, s.s, s.sz, s.sq, s.done, tn, s.slices_p, 0};
    launch_pair_rows<true>(jobs, sigma, kCutNll, st);
    k_nll_grad<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(hp, n, s.s, s.sz, s.sq, s.slices_p,
                                                            (float)(1.0 / ((double)sigma * (double)sigma)), g_hp,
                                                            g_z, g_q);
  }
  return LSIM_OK;
}

size_t chamfer_workspace_bytes(int64_t n, int64_t m) {
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  return 4 * al(4 * (size_t)n) + 2 * al(4 * (size_t)m) +
         al(sizeof(int2) * (size_t)((n + kRbfChunk - 1) / kRbfChunk + 1)) +
         al(sizeof(int2) * (size_t)((m + kRbfChunk - 1) / kRbfChunk + 1));
}

int run_chamfer(const float *x, const float *y, const float *z, const int32_t *event, const float *w, int64_t n,
                const float *rx, const float *ry, const float *rz, const int32_t *revent, const float *rw, int64_t m,
                float *out, float *g_w, float *g_z, void *ws, cudaStream_t st) {
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  char *b = static_cast<char *>(ws);
  float *ma = reinterpret_cast<float *>(b); b += al(4 * (size_t)n);
  int32_t *ia = reinterpret_cast<int32_t *>(b); b += al(4 * (size_t)n);
  float *aw = reinterpret_cast<float *>(b); b += al(4 * (size_t)n);
  float *az = reinterpret_cast<float *>(b); b += al(4 * (size_t)n);
  float *mb = reinterpret_cast<float *>(b); b += al(4 * (size_t)m);
  int32_t *ib = reinterpret_cast<int32_t *>(b); b += al(4 * (size_t)m);
  int2 *rng_pred = reinterpret_cast<int2 *>(b); b += al(sizeof(int2) * (size_t)((n + kRbfChunk - 1) / kRbfChunk + 1));
  int2 *rng_ref = reinterpret_cast<int2 *>(b);
  const HitSet4 pred{x, y, z, nullptr, w, event, n}, ref{rx, ry, rz, nullptr, rw, revent, m};
  if (n > 0) k_chunk_events<<<(unsigned)((n + kRbfChunk - 1) / kRbfChunk), kRbfChunk, 0, st>>>(event, n, rng_pred);
  if (m > 0) k_chunk_events<<<(unsigned)((m + kRbfChunk - 1) / kRbfChunk), kRbfChunk, 0, st>>>(revent, m, rng_ref);
  if (n > 0) k_nn_rows<<<(unsigned)((n + kRbfRows - 1) / kRbfRows), kRbfRows, 0, st>>>(pred, ref, rng_ref, ma, ia);
  if (m > 0) k_nn_rows<<<(unsigned)((m + kRbfRows - 1) / kRbfRows), kRbfRows, 0, st>>>(ref, pred, rng_pred, mb, ib);
  k_chamfer_reduce<<<1, 1024, 0, st>>>(w, n, rw, m, ma, ia, mb, ib, out);
  if (n > 0 && (g_w || g_z)) {
    k_chamfer_back<<<(unsigned)((n + kRbfRows - 1) / kRbfRows), kRbfRows, 0, st>>>(pred, ref, rng_ref, mb, ib, aw,
                                                                                   az);
    k_chamfer_grad<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(pred, ref, ma, ia, aw, az, g_w, g_z);
  }
  return LSIM_OK;
}

}  // namespace lsim
