// Track chopping on the device: every input track becomes
// max(ceil(length / precision), 1) steps of length `precision`, the last step
// taking the remainder (optimize/dataio.py:63-106, chop_tracks).
//
// Four launches: per-track step counts with per-block sums, one CTA scanning
// the block sums (total to the caller's counter), per-track output offsets
// and records, then a fill kernel whose warps assemble 32 output rows at a time
// in shared memory and write them with coalesced stores.  The
// arithmetic is the reference's under NumPy 2 promotion: length, direction,
// step count and the per-step dE in float32; step positions and the last
// step's dE and dx in float64, rounded once to float32; midpoints in float32.
// The explicit _rn intrinsics keep the compiler from contracting any of it
// into FMAs.
//
// Float64 runs at 1/64 of the float32 rate here, and was what bounded the
// fill (six positions a row: 1.39 ms for 20M rows, 22 % of the copy
// bandwidth).  So a position is formed as a pair of floats (relative error
// below 2^-44, like the float64 chain's 2^-52 far below float32's 2^-24) and
// rounded; only where the rounding could differ within that error, about once
// in 2^19, is the float64 chain evaluated.  A step's end is the next row's
// start (the same expression), and what is per track (geometry, the last
// step's dE and dx with their float64 division) is evaluated once per track.
// 200k segments into 20M steps (2.1 GB written), the whole call: 1.46 -> 0.54 ms,
// now bound by the shared-memory assembly of the rows (L1 90 % busy; 4.6 TB/s).
#include "lsim_internal.cuh"

namespace lsim {
namespace {

constexpr int kChopThreads = 256;   // tracks per block in the count/offset kernels
constexpr int kFillWarps = 4;        // warps per block of the fill kernel, 32 output rows each at a time
constexpr int kMaxChopFields = 96;  // columns: 128 * 96 * 4 B = 48 KiB of shared memory

struct TrackGeom {
  float s[3], e[3], d[3];
  float len, lpe;  // length and length + 1e-10 (float32, dataio.py:98-100)
};

__device__ __forceinline__ TrackGeom track_geom(const float *row, const LsimFieldMap &f) {
  TrackGeom g;
  g.s[0] = row[f.x_start];
  g.s[1] = row[f.y_start];
  g.s[2] = row[f.z_start];
  g.e[0] = row[f.x_end];
  g.e[1] = row[f.y_end];
  g.e[2] = row[f.z_end];
  float seg[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) seg[a] = __fsub_rn(g.e[a], g.s[a]);
  // np.sum over the 3 squared components: left to right in float32
  float l2 = __fadd_rn(__fadd_rn(__fmul_rn(seg[0], seg[0]), __fmul_rn(seg[1], seg[1])), __fmul_rn(seg[2], seg[2]));
  g.len = __fsqrt_rn(l2);
  g.lpe = __fadd_rn(g.len, (float)1e-10);
#pragma unroll
  for (int a = 0; a < 3; ++a) g.d[a] = __fdiv_rn(seg[a], g.lpe);
  return g;
}

// max(ceil(length / precision), 1) as an integer; -1 when the quotient is
// not finite or does not fit (the reference's int cast then fails).
__device__ __forceinline__ int64_t step_count(float len, float prec32) {
  float q = ceilf(__fdiv_rn(len, prec32));
  if (!(q <= 9.0e18f)) return -1;
  return q < 1.0f ? 1 : (int64_t)q;
}

__device__ __forceinline__ int64_t block_sum_i64(int64_t v, int64_t *red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  int64_t t = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;
}

__global__ void __launch_bounds__(kChopThreads) k_chop_count(const float *__restrict__ tracks, int64_t n_rows,
                                                             LsimFieldMap f, float prec32,
                                                             int64_t *__restrict__ row_n,
                                                             int64_t *__restrict__ blk_sum, int32_t *bad) {
  __shared__ int64_t red[kChopThreads / 32];
  const int64_t r = (int64_t)blockIdx.x * kChopThreads + threadIdx.x;
  int64_t n = 0;
  if (r < n_rows) {
    TrackGeom g = track_geom(tracks + r * f.n_fields, f);
    n = step_count(g.len, prec32);
    if (n < 0) {
      *bad = 1;
      n = 0;
    }
    row_n[r] = n;
  }
  int64_t t = block_sum_i64(n, red);
  if (threadIdx.x == 0) blk_sum[blockIdx.x] = t;
}

// One CTA: exclusive scan of the block sums in place; the total (or -1 on
// a bad track) to *n_out.
__global__ void __launch_bounds__(1024) k_chop_scan_blocks(int64_t *blk, int64_t nblk, const int32_t *bad,
                                                           int64_t *n_out) {
  __shared__ int64_t warp_tot[32];
  __shared__ int64_t chunk_total;
  int64_t carry = 0;
  for (int64_t base = 0; base < nblk; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t v = i < nblk ? blk[i] : 0;
    const int64_t inc = block_scan_i64(v, warp_tot, &chunk_total);
    if (i < nblk) blk[i] = carry + inc - v;
    __syncthreads();
    carry += chunk_total;
    __syncthreads();
  }
  if (threadIdx.x == 0) *n_out = *bad ? -1 : carry;
}

// What the fill needs of a track.
struct __align__(16) ChopTrack {
  float s[3], de_step;   // start, dE of a full step
  float d[3], de_last;   // direction, dE of the last step
  float e[3], dx_last;   // end, dx of the last step
};

__global__ void __launch_bounds__(kChopThreads) k_chop_offsets(const float *__restrict__ tracks, LsimFieldMap f,
                                                               double prec, float prec32,
                                                               const int64_t *__restrict__ row_n, int64_t n_rows,
                                                               const int64_t *__restrict__ blk_off,
                                                               int64_t *__restrict__ row_off,
                                                               ChopTrack *__restrict__ recs) {
  __shared__ int64_t warp_tot[kChopThreads / 32];
  __shared__ int64_t total;
  const int64_t r = (int64_t)blockIdx.x * kChopThreads + threadIdx.x;
  const int64_t v = r < n_rows ? row_n[r] : 0;
  const int64_t inc = block_scan_i64(v, warp_tot, &total);
  if (r >= n_rows) return;
  row_off[r] = blk_off[blockIdx.x] + inc - v;
  if (!recs) return;
  const float *row = tracks + r * f.n_fields;
  const TrackGeom g = track_geom(row, f);
  const float dE = row[f.dE];
  ChopTrack c;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    c.s[a] = g.s[a];
    c.d[a] = g.d[a];
    c.e[a] = g.e[a];
  }
  c.de_step = __fdiv_rn(__fmul_rn(dE, prec32), g.lpe);   // dataio.py:67
  const double m = __dmul_rn(prec, (double)(v - 1));
  c.de_last = (float)__dmul_rn((double)dE, __dsub_rn(1.0, __ddiv_rn(m, (double)g.lpe)));   // :83
  c.dx_last = (float)__dsub_rn((double)g.len, m);                                          // :84
  recs[r] = c;
}

// The track whose output rows contain row `o`: the last r with row_off[r] <= o
// (offsets are strictly increasing: every track has at least one step).  One
// warp, 32 tracks tested a round.
__device__ __forceinline__ int64_t source_track(const int64_t *__restrict__ row_off, int64_t n_rows, int64_t o,
                                                int lane) {
  int64_t lo = 0, hi = n_rows;   // row_off[lo] <= o < row_off[hi]
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t at = lo + (lane + 1) * step;
    const unsigned m = __ballot_sync(0xffffffffu, at < hi && __ldg(row_off + at) <= o);
    const int j = __popc(m);     // the first j candidates hold
    const int64_t up = lo + (j + 1) * step;
    lo += j * step;
    hi = up < hi ? up : hi;
  }
  return lo;
}

// Position s0 + (k prec) d of a step boundary as the reference forms it in
// float64 (dataio.py:70-76, :80-82), rounded to float32.
__device__ __noinline__ float step_position64(float s0, float d, int64_t k, double prec) {
  return (float)__dadd_rn((double)s0, __dmul_rn(__dmul_rn((double)k, prec), (double)d));
}

struct PrecPair {
  float hi, lo;   // prec = hi + lo to 2^-48
};

__device__ __forceinline__ float step_position(float s0, float d, int64_t k, double prec, PrecPair pp) {
  const float kf = (float)k;
  // k prec and its product with d, each as a high part and what it lacks
  const float h = __fmul_rn(kf, pp.hi);
  const float l = __fmaf_rn(kf, pp.lo, __fmaf_rn(kf, pp.hi, -h));
  const float H = __fmul_rn(h, d);
  const float L = __fmaf_rn(l, d, __fmaf_rn(h, d, -H));
  // s0 + H exactly as S + err (Knuth's two-sum)
  const float S = __fadd_rn(s0, H);
  const float b = __fsub_rn(S, s0);
  const float err = __fadd_rn(__fsub_rn(s0, __fsub_rn(S, b)), __fsub_rn(H, b));
  const float low = __fadd_rn(err, L);
  const float tol = __fmul_rn(__fadd_rn(fabsf(s0), fabsf(H)), 5.6843418860808015e-14f);   // 2^-44
  const float up = __fadd_rn(S, __fadd_rn(low, tol)), down = __fadd_rn(S, __fsub_rn(low, tol));
  // (k beyond 2^24 is not exact above; what is not finite or tiny goes the long way too)
  if (up == down && k < (1 << 24) && fabsf(up) > 1e-25f) return up;
  return step_position64(s0, d, k, prec);
}

// One warp fills 32 rows at a time, of a contiguous run of such tiles, so
// that a tile's first track follows from the tile before and the next tile's
// track offsets are loaded ahead; nothing waits for another warp.
__global__ void __launch_bounds__(kFillWarps * 32, 12) k_chop_fill(const float *__restrict__ tracks, int64_t n_rows,
                                                                  LsimFieldMap f, double prec, float prec32,
                                                                  PrecPair pp, const int64_t *__restrict__ row_off,
                                                                  const ChopTrack *__restrict__ recs,
                                                                  const int64_t *__restrict__ n_out,
                                                                  float *__restrict__ out, int64_t capacity) {
  extern __shared__ __align__(16) float tiles[];
  const int64_t total = *n_out;
  if (total <= 0) return;
  const int64_t lim = total < capacity ? total : capacity;
  const int F = f.n_fields, lane = threadIdx.x % 32;
  float *tile = tiles + (threadIdx.x / 32) * 32 * F, *dst = tile + lane * F;
  const int cs[3] = {f.x_start, f.y_start, f.z_start};
  const int ce[3] = {f.x_end, f.y_end, f.z_end};
  const int cm[3] = {f.x, f.y, f.z};
  const bool pairs = F % 2 == 0 && (reinterpret_cast<uintptr_t>(tracks) & 7) == 0;   // rows of whole float2
  const int64_t n_tiles = (lim + 31) / 32, n_warps = (int64_t)gridDim.x * kFillWarps;
  const int64_t per = (n_tiles + n_warps - 1) / n_warps;
  const int64_t w = (int64_t)blockIdx.x * kFillWarps + threadIdx.x / 32;
  const int64_t tile0 = w * per, tile1 = min(n_tiles, tile0 + per);
  if (tile0 >= tile1) return;
  // where track src0 starts, and (lane l) where track src0 + 1 + l does
  int64_t src0 = source_track(row_off, n_rows, tile0 * 32, lane), start0 = row_off[src0];
  auto start_of = [&](int64_t r) { return r < n_rows ? __ldg(row_off + r) : total; };
  int64_t next = start_of(src0 + 1 + lane);
  for (int64_t t = tile0; t < tile1; ++t) {
    const int64_t t0 = t * 32, o = t0 + lane;
    // bit p: a track starts at row t0 + p (every track has a row, so the lanes see all of the tile's)
    const int64_t at = next - t0;
    const unsigned starts = __reduce_or_sync(0xffffffffu, at > 0 && at < 32 ? 1u << (int)at : 0u);
    const int mine = __popc(starts & (0xffffffffu >> (31 - lane)));   // my row's track: src0 + mine
    const int64_t before = __shfl_sync(0xffffffffu, next, mine > 0 ? mine - 1 : 0);
    const int64_t after = __shfl_sync(0xffffffffu, next, mine < 31 ? mine : 31);
    const int64_t k = o - (mine > 0 ? before : start0);
    // (mine = 31 only if every row of the tile starts a track: the row after is the 32nd's, next of lane 31)
    const bool last = after == o + 1;
    const int64_t src = src0 + mine;
    // the next tile's first track and its offsets
    const int moved = __popc(__ballot_sync(0xffffffffu, at > 0 && at <= 32));
    if (moved > 0) start0 = __shfl_sync(0xffffffffu, next, moved - 1);
    src0 += moved;
    if (t + 1 < tile1) next = start_of(src0 + 1 + lane);
    const bool ok = o < lim;
    ChopTrack c;
    float st[3], en[3];
    if (ok) {
      const float *row = tracks + src * F;
      c = recs[src];
      if (pairs) {
        const float2 *r2 = reinterpret_cast<const float2 *>(row);
        float2 *d2 = reinterpret_cast<float2 *>(dst);
#pragma unroll 8
        for (int q = 0; q < F / 2; ++q) d2[q] = __ldg(r2 + q);
      } else {
        for (int q = 0; q < F; ++q) dst[q] = __ldg(row + q);
      }
      dst[f.dE] = last ? c.de_last : c.de_step;
      dst[f.dx] = last ? c.dx_last : prec32;   // dataio.py:77
#pragma unroll
      for (int a = 0; a < 3; ++a) dst[cs[a]] = st[a] = step_position(c.s[a], c.d[a], k, prec, pp);
    }
    // a step ends where the next row starts
#pragma unroll
    for (int a = 0; a < 3; ++a) en[a] = __shfl_down_sync(0xffffffffu, st[a], 1);
    if (ok) {
      const bool own = !last && (lane == 31 || o + 1 >= lim);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (last) en[a] = c.e[a];
        else if (own) en[a] = step_position(c.s[a], c.d[a], k + 1, prec, pp);
        dst[ce[a]] = en[a];
        dst[cm[a]] = __fmul_rn(0.5f, __fadd_rn(st[a], en[a]));   // :87-89
      }
    }
    __syncwarp();
    const int count = (int)min((int64_t)32, lim - t0) * F;
    float *base = out + t0 * F;   // a tile is a multiple of 128 bytes
    if ((reinterpret_cast<uintptr_t>(base) & 15) == 0 && (reinterpret_cast<uintptr_t>(tile) & 15) == 0) {
      const float4 *t4 = reinterpret_cast<const float4 *>(tile);
      float4 *b4 = reinterpret_cast<float4 *>(base);
      for (int e = lane; e < count / 4; e += 32) b4[e] = t4[e];
      for (int e = (count & ~3) + lane; e < count; e += 32) base[e] = tile[e];
    } else {
      for (int e = lane; e < count; e += 32) base[e] = tile[e];
    }
    __syncwarp();
  }
}

struct ChopWs {
  int64_t *row_n, *row_off, *blk;
  int32_t *bad;
  ChopTrack *recs;
};

size_t chop_layout(int64_t n_rows, ChopWs *w, char *base) {
  const int64_t nblk = (n_rows + kChopThreads - 1) / kChopThreads;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t at = off;
    off += (bytes + 255) & ~size_t(255);
    return base ? base + at : nullptr;
  };
  char *a = take(sizeof(int64_t) * (size_t)n_rows);
  char *b = take(sizeof(int64_t) * (size_t)n_rows);
  char *c = take(sizeof(int64_t) * (size_t)(nblk > 0 ? nblk : 1));
  char *d = take(sizeof(int32_t));
  char *e = take(sizeof(ChopTrack) * (size_t)n_rows);
  if (w) {
    w->recs = reinterpret_cast<ChopTrack *>(e);
    w->row_n = reinterpret_cast<int64_t *>(a);
    w->row_off = reinterpret_cast<int64_t *>(b);
    w->blk = reinterpret_cast<int64_t *>(c);
    w->bad = reinterpret_cast<int32_t *>(d);
  }
  return off;
}

}  // namespace

size_t chop_workspace_bytes(int64_t n_rows) { return chop_layout(n_rows, nullptr, nullptr); }

int run_chop(const LsimFieldMap &f, const float *tracks, int64_t n_rows, double precision, float *out,
             int64_t capacity, int64_t *n_out, void *ws, cudaStream_t st) {
  if (f.n_fields > kMaxChopFields) return set_error(LSIM_ERR_UNSUPPORTED, "chop: more than 96 columns");
  ChopWs w;
  chop_layout(n_rows, &w, static_cast<char *>(ws));
  const float prec32 = (float)precision;
  const int64_t nblk = (n_rows + kChopThreads - 1) / kChopThreads;
  if (cudaMemsetAsync(w.bad, 0, sizeof(int32_t), st) != cudaSuccess) return LSIM_ERR_CUDA;
  if (nblk > 0)
    k_chop_count<<<(unsigned)nblk, kChopThreads, 0, st>>>(tracks, n_rows, f, prec32, w.row_n, w.blk, w.bad);
  k_chop_scan_blocks<<<1, 1024, 0, st>>>(w.blk, nblk, w.bad, n_out);
  const bool fill = out && capacity > 0 && n_rows > 0;
  if (nblk > 0)
    k_chop_offsets<<<(unsigned)nblk, kChopThreads, 0, st>>>(tracks, f, precision, prec32, w.row_n, n_rows, w.blk,
                                                           w.row_off, fill ? w.recs : nullptr);
  if (fill) {
    const int64_t blocks = (capacity + 32 * kFillWarps - 1) / (32 * kFillWarps);
    const int64_t cap = (int64_t)device_sm_count() * 12;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    const size_t smem = sizeof(float) * 32 * kFillWarps * (size_t)f.n_fields;
    const PrecPair pp{prec32, (float)(precision - (double)prec32)};
    k_chop_fill<<<grid, kFillWarps * 32, smem, st>>>(tracks, n_rows, f, precision, prec32, pp, w.row_off, w.recs,
                                               n_out, out, capacity);
  }
  return LSIM_OK;
}

}  // namespace lsim
