// Main-bin parts of LUT mode, segment-major.
//
// A segment's 5 x 5 transverse-diffusion bins cover at most 2 x 2 pixels.
// For each covered pixel the window it adds is
//   V[k] = n_e * sum over the bins (i, j) on that pixel of
//          ex_i ey_j * (a T_{t-1} + b T_t + c T_{t+1})[cx_i, cy_j, Nt - L + k]
// (main_vals_2d, sim_jax.py:186-192) with the quadratic long-diffusion
// interpolation weights (a, b, c) (sim_jax.py:162-168) and the
// cumulative-sum boundary term (sim_jax.py:237-241).  Bins of one pixel that share a LUT sub-position
// (u, v) are grouped, W_uv = sum ex_i * sum ey_j, so each window reads at
// most 25 LUT rows.
//
// k_main_records computes V and the boundary term once per (segment,
// pixel) and stores them as a record; the pixel-major accumulation adds the
// record like a neighbour part.  After the pixel-major adjoint has replaced
// the record by its cotangent, k_main_adjoint projects it back onto n_e,
// sigma_T and (a, b, c) and writes dL/dtheta per segment (reduced later in
// segment order, so the result does not depend on the processing order).
// Both kernels take the segments grouped by template index, a block a
// contiguous range of that order, so that a block's segments share the 25 LUT
// window rows of a template (64 KB) in L1.  A warp takes two segments at a
// time and loads a row once for the records of both that use it; a segment's
// own sums keep their order.  Bound by latency (about 40 % of the issue slots
// used): the chain from the order's entry over the segment, its grid slot and
// the cumulative sums to the rows.
#include <type_traits>

#include "lsim_internal.cuh"
#include "lsim_bins.cuh"
#include "lsim_fee.cuh"

namespace lsim {


constexpr int kSub = kMainSub * kMainSub;   // LUT sub-positions (u, v), e = 5 u + v

// Weights of one (segment, pixel) pair: W and dW/dsigma_T by sub-position,
// and (adjoint) W, dW and the cumulative-sum term D of the used ones in order.
struct MainSmem {
  float W[kSub], dW[kSub];
  float cW[kSub], cdW[kSub], cD[kSub];
};

// LUT index per bin of one axis on the pixel at offset d, four bits a bin
// (15: the bin is on another pixel).  It depends on the bin's place in its
// pixel alone, so a nibble string per place serves: bin b + i - 2 of place
// m = b mod 10 is position m + i - 2 of the ten positions' indices
// 4 3 2 1 0 0 1 2 3 4, of the pixel before below 0 and of the one after from 10.
struct AxisBins {
  uint32_t nib;
  __device__ __forceinline__ int index(int i) const { return (nib >> (4 * i)) & 15u; }
  __device__ __forceinline__ unsigned used() const {
    unsigned m = 0u;
#pragma unroll
    for (int i = 0; i < kMaxTran; ++i) m |= 1u << index(i);
    return m & 31u;
  }
};

__device__ __forceinline__ AxisBins axis_bins(int b, int d) {
  static_assert(kBinsPerPixel == 10 && kMaxTran == 5, "nibble string of ten positions, five bins");
  const int pos = imod(b, kBinsPerPixel) - kMaxTran / 2 - kBinsPerPixel * d;   // first bin's position in pixel d
  // positions 0..9 as nibbles, 15 around them: (~0 below) pos (~0 above)
  const uint64_t string = 0x4321001234ull;
  const uint64_t ones = ~0ull;
  // nibbles pos .. pos + 4
  uint32_t nib;
  if (pos >= 0) nib = pos < 10 ? (uint32_t)((string | (ones << 40)) >> (4 * pos)) : 0xfffffu;
  else nib = pos > -5 ? (uint32_t)((string << (-4 * pos)) | ((1ull << (-4 * pos)) - 1)) : 0xfffffu;
  return AxisBins{nib & 0xfffffu};
}

// Lane l < 25 owns sub-position (u, v) = (l / 5, l % 5).  Returns the mask of
// sub-positions with bins on the pixel; *wd and *wdl are sum W D and sum
// W dD/dfrac (dD/dfrac the boundary term's derivative).
template <bool GRAD>
__device__ __forceinline__ unsigned main_weights(const LsimParams &p, const Tables &tab, const SegFwd &f,
                                                 const SegAdj *a, int dx, int dy, MainSmem &ms, float *wd, float *wdl,
                                                 int lane) {
  // this lane's sub-position (u, v): summed 1-D bin integrals of the bins of
  // each axis that fall on the pixel with that LUT index
  const int u = lane / kMainSub, v = lane % kMainSub;
  float xw = 0.f, yw = 0.f, dxw = 0.f, dyw = 0.f;
  const AxisBins ax = axis_bins(f.bx, dx), ay = axis_bins(f.by, dy);
  const unsigned um = ax.used(), vm = ay.used();
#pragma unroll
  for (int i = 0; i < kMaxTran; ++i) {
    const bool tx = ax.index(i) == u, ty = ay.index(i) == v;
    xw += tx ? f.ex[i] : 0.f;
    yw += ty ? f.ey[i] : 0.f;
    if (GRAD) {
      dxw += tx ? a->dex[i] : 0.f;
      dyw += ty ? a->dey[i] : 0.f;
    }
  }
  const bool mine = lane < kSub && ((um >> u) & 1u) && ((vm >> v) & 1u);
  const unsigned bal = __ballot_sync(0xffffffffu, mine);
  float s_wd = 0.f, s_wdl = 0.f;
  if (mine) {
    float dl;
    const float D = cum_terms(tab.cm + (size_t)(f.tidx * kSub + lane) * p.lut_nt, f.cath, p.lut_nt, p.signal_length,
                              f.frac, &dl);
    const float W = xw * yw;
    ms.W[lane] = W;
    if (GRAD) {
      const int pos = __popc(bal & ((1u << lane) - 1u));
      const float dW = dxw * yw + xw * dyw;
      ms.dW[lane] = dW;
      ms.cW[pos] = W;
      ms.cdW[pos] = dW;
      ms.cD[pos] = D;
    }
    s_wd = W * D;
    s_wdl = W * dl;
  }
  if (!GRAD) {
    *wd = warp_sum(s_wd);
    *wdl = warp_sum(s_wdl);
  }
  return bal;
}

// This block's contiguous chunk [i0, i1) of the template-ordered segments;
// its warps take kGroup entries at a time in turn.
__device__ __forceinline__ void block_chunk(int64_t n, int64_t *i0, int64_t *i1) {
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  *i0 = (int64_t)blockIdx.x * chunk;
  *i1 = min(n, *i0 + chunk);
}

// The leading entries of seg_order[i, end) with one template index, at most
// kGroup: lane q < count holds segment q in *seg.
template <int kGroup>
__device__ __forceinline__ int take_group(const Workspace &w, int64_t i, int64_t end, int lane, int *seg) {
  const bool have = lane < kGroup && i + lane < end;
  *seg = have ? w.seg_order[i + lane] : 0;
  const int tidx = have ? w.segf[*seg].tidx : -1;
  const int first = __shfl_sync(0xffffffffu, tidx, 0);
  const unsigned same = __ballot_sync(0xffffffffu, have && tidx == first);
  return __ffs(~same) - 1;
}

// Bit 4 q + slot: segment q (of n) has a record in that slot.  Records of
// pixels that are not simulated are never read (the reference drops main
// bins outside unique_pixels, sim_jax.py:152-154).
__device__ __forceinline__ unsigned record_mask(const Workspace &w, const Grid &g, int my_seg, int n, int lane) {
  const int q = lane / kRecPerSeg, slot = lane % kRecPerSeg;
  const int s = __shfl_sync(0xffffffffu, my_seg, q);
  bool have = false;
  if (q < n) {
    const SegFwd &f = w.segf[s];
    int lx, hx, ly, hy;
    axis_range(f.bx, kBinsPerPixel, &lx, &hx);
    axis_range(f.by, kBinsPerPixel, &ly, &hy);
    const int dx = lx + slot / 2, dy = ly + slot % 2;
    have = dx <= hx && dy <= hy && slot_is_pixel(g, w.cnt, (int64_t)w.key[s] + (int64_t)dy * g.nxe + dx);
  }
  return __ballot_sync(0xffffffffu, have);
}

// Pixel offset of a segment's record slot.
__device__ __forceinline__ void slot_offset(const SegFwd &f, int slot, int *dx, int *dy) {
  int hx, hy;
  axis_range(f.bx, kBinsPerPixel, dx, &hx);
  axis_range(f.by, kBinsPerPixel, dy, &hy);
  *dx += slot / 2;
  *dy += slot % 2;
}

// Launch shape of the main-bin kernels: one block of 24 warps per SM, or as
// tuned (blocks of 8 or 4 warps in any number).  One block walks one stretch
// of the template order, so an SM's L1 holds one template's rows (64 KB);
// two blocks per SM hold two, and 8-warp blocks in a grid of 1024 left L1
// thrashing and a last wave: 1.76 and 2.13 ms on the 64-event batch, against
// 1.25 and 1.46.  Measured there: 16 warps a block 1.37-1.65 / 1.60-1.91,
// 32 warps 1.31-1.35 / 1.53-1.56, segments per warp 1, 3, 4: 1.31, 1.43, 1.39.
constexpr int kMainSmWarps = 24;
constexpr int kMaxMainBlocks = 65536;    // of a tuned shape: more blocks than segments only cost their launch

template <typename F>
static void with_main_shape(F &&launch) {
  const LsimTuning tu = tuning();
  const int warps = tu.main_block_warps == 8 || tu.main_block_warps == 4 ? tu.main_block_warps : kMainSmWarps;
  const int blocks = tu.main_blocks > 0 ? min(tu.main_blocks, kMaxMainBlocks)
                                        : device_sm_count() * (kMainSmWarps / warps);
  if (warps == 4) launch(std::integral_constant<int, 4>(), blocks);
  else if (warps == 8) launch(std::integral_constant<int, 8>(), blocks);
  else launch(std::integral_constant<int, kMainSmWarps>(), blocks);
}

// ---------------------------------------------------------------- order

// Segments with main-bin records, grouped by template index with a counting
// sort (the order inside a group is arbitrary); the counts are made by
// k_pass_prepare (main_order_count).
__global__ void k_main_order_scan(Workspace w) {
  __shared__ int sh[kMaxTemplates];
  const int t = threadIdx.x;
  const int c = w.tidx_hist[t];
  sh[t] = c;
  __syncthreads();
  for (int o = 1; o < kMaxTemplates; o <<= 1) {
    const int v = t >= o ? sh[t - o] : 0;
    __syncthreads();
    sh[t] += v;
    __syncthreads();
  }
  w.tidx_hist[kMaxTemplates + t] = sh[t] - c;
  if (t == kMaxTemplates - 1) w.counts->n_main_seg = sh[t];
}

__global__ void k_main_order_scatter(Workspace w, int64_t n_rows) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x % kWarp;
  int bin = 0;
  const bool act = main_active(w, s, n_rows, &bin);
  const unsigned am = __ballot_sync(0xffffffffu, act);
  if (act) {
    const unsigned peers = __match_any_sync(am, bin);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&w.tidx_hist[kMaxTemplates + bin], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    w.seg_order[base + __popc(peers & ((1u << lane) - 1u))] = (int32_t)s;
  }
}

// ---------------------------------------------------------------- kernels

// L1 prefetch of the next segment's records (segments come in template
// order, so their records are scattered; the next one's lines are fetched
// while this one is processed).
__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

constexpr int kRecGroup = 2, kAdjGroup = 2;
static_assert(kRecGroup * kRecPerSeg <= kWarp, "a lane per (segment, slot)");

template <int kMainBlockWarps>
__global__ void __launch_bounds__(kMainBlockWarps * kWarp, kMainSmWarps / kMainBlockWarps)
    k_main_records(LsimParams p, Tables tab, Workspace w, Grid g) {
  __shared__ MainSmem sms[kMainBlockWarps][kRecGroup];
  const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
  MainSmem *ms = sms[wid];
  int n_rec = 0;
  int64_t i0, i1;
  block_chunk(w.counts->n_main_seg, &i0, &i1);
  for (int64_t i = i0 + wid * kRecGroup; i < i1; i += kMainBlockWarps * kRecGroup) {
    const int64_t ahead = i + kMainBlockWarps * kRecGroup + lane / 2;
    if (lane < 2 * kRecGroup && ahead < i1)
      prefetch_l1(reinterpret_cast<const char *>(w.segf + w.seg_order[ahead]) + 64 * (lane & 1));
    const int64_t end = min(i1, i + kRecGroup);
    int ng;
    for (int64_t j0 = i; j0 < end; j0 += ng) {
      int my_seg;
      ng = take_group<kRecGroup>(w, j0, end, lane, &my_seg);
      const unsigned have = record_mask(w, g, my_seg, ng, lane);
      int seg[kRecGroup];
      float qa[kRecGroup], qb[kRecGroup], qc[kRecGroup];
#pragma unroll
      for (int q = 0; q < kRecGroup; ++q) {
        seg[q] = __shfl_sync(0xffffffffu, my_seg, q);
        const SegFwd &f = w.segf[seg[q]];
        qa[q] = f.qa;
        qb[q] = f.qb;
        qc[q] = f.qc;
      }
      const float4 *rows = tab.wmp + (size_t)w.segf[seg[0]].tidx * kSub * kWinSamples + lane;
#pragma unroll 1
      for (int slot = 0; slot < kRecPerSeg; ++slot) {
        unsigned used[kRecGroup], any = 0u;
        float wd[kRecGroup], wdl[kRecGroup], acc[kRecGroup][kChunks];
#pragma unroll
        for (int q = 0; q < kRecGroup; ++q) {
          used[q] = 0u;
          wd[q] = wdl[q] = 0.f;
          if ((have >> (kRecPerSeg * q + slot)) & 1u) {
            const SegFwd &f = w.segf[seg[q]];
            int dx, dy;
            slot_offset(f, slot, &dx, &dy);
            used[q] = main_weights<false>(p, tab, f, nullptr, dx, dy, ms[q], &wd[q], &wdl[q], lane);
          }
          any |= used[q];
#pragma unroll
          for (int j = 0; j < kChunks; ++j) acc[q][j] = 0.f;
        }
        __syncwarp();
#pragma unroll 1
        for (; any; any &= any - 1) {
          const int e = __ffs(any) - 1;
          // padded rows: entry idx is sample idx - 1, matching the record layout
          const float4 *src = rows + (size_t)e * kWinSamples;
          float4 t[kChunks];
#pragma unroll
          for (int j = 0; j < kChunks; ++j) t[j] = __ldg(src + j * kWarp);
#pragma unroll
          for (int q = 0; q < kRecGroup; ++q) {
            if (!((used[q] >> e) & 1u)) continue;
            const float W = ms[q].W[e];
            const float wa = W * qa[q], wb = W * qb[q], wc = W * qc[q];
#pragma unroll
            for (int j = 0; j < kChunks; ++j)
              acc[q][j] = fmaf(t[j].z, wc, fmaf(t[j].x, wa, fmaf(t[j].y, wb, acc[q][j])));
          }
        }
#pragma unroll
        for (int q = 0; q < kRecGroup; ++q) {
          if (!((have >> (kRecPerSeg * q + slot)) & 1u)) continue;
          const float ne = w.segf[seg[q]].ne;
          float *rec = w.mrec + ((size_t)seg[q] * kRecPerSeg + slot) * kRecFloats;
#pragma unroll
          for (int j = 0; j < kChunks; ++j) {
            const int idx = lane + j * kWarp;
            rec[idx] = idx == 0 ? wd[q] * ne : acc[q][j] * ne;
          }
          if (lane == 0) rec[kRecDl] = wdl[q] * ne;
          ++n_rec;
        }
        __syncwarp();
      }
    }
  }
  if (lane == 0 && n_rec) atomicAdd(&w.counts->n_main_rec, n_rec);
}

template <int kMainBlockWarps>
__global__ void __launch_bounds__(kMainBlockWarps * kWarp, kMainSmWarps / kMainBlockWarps)
    k_main_adjoint(LsimParams p, Tables tab, Workspace w, Grid g) {
  __shared__ MainSmem sms[kMainBlockWarps][kAdjGroup];
  const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
  MainSmem *ms = sms[wid];
  int64_t i0, i1;
  block_chunk(w.counts->n_main_seg, &i0, &i1);
  for (int64_t i = i0 + wid * kAdjGroup; i < i1; i += kMainBlockWarps * kAdjGroup) {
    // the next group's records (segment, adjoint partials, main-bin records)
#pragma unroll
    for (int q = 0; q < kAdjGroup; ++q) {
      const int64_t ahead = i + kMainBlockWarps * kAdjGroup + q;
      if (ahead < i1) {
        const int64_t sn = w.seg_order[ahead];
        if (lane < 2) prefetch_l1(reinterpret_cast<const char *>(w.segf + sn) + 64 * lane);
        else if (lane < 4) prefetch_l1(reinterpret_cast<const char *>(w.sega + sn) + 64 * (lane - 2));
        else if (lane < 4 + 21) prefetch_l1(w.mrec + (size_t)sn * kRecPerSeg * kRecFloats + 32 * (lane - 4));
      }
    }
    const int64_t end = min(i1, i + kAdjGroup);
    int ng;
    for (int64_t j0 = i; j0 < end; j0 += ng) {
      int my_seg;
      ng = take_group<kAdjGroup>(w, j0, end, lane, &my_seg);
      const unsigned have = record_mask(w, g, my_seg, ng, lane);
      int seg[kAdjGroup];
      float qa[kAdjGroup], qb[kAdjGroup], qc[kAdjGroup];
      float acc_ne[kAdjGroup], acc_sig[kAdjGroup], acc_a[kAdjGroup], acc_b[kAdjGroup], acc_c[kAdjGroup];
#pragma unroll
      for (int q = 0; q < kAdjGroup; ++q) {
        seg[q] = __shfl_sync(0xffffffffu, my_seg, q);
        const SegFwd &f = w.segf[seg[q]];
        qa[q] = f.qa;
        qb[q] = f.qb;
        qc[q] = f.qc;
        acc_ne[q] = acc_sig[q] = acc_a[q] = acc_b[q] = acc_c[q] = 0.f;
      }
      const float4 *rows = tab.wmp + (size_t)w.segf[seg[0]].tidx * kSub * kWinSamples + lane;
#pragma unroll 1
      for (int slot = 0; slot < kRecPerSeg; ++slot) {
        unsigned used[kAdjGroup], any = 0u;
        float d[kAdjGroup][kChunks], dcorr[kAdjGroup];
#pragma unroll
        for (int q = 0; q < kAdjGroup; ++q) {
          used[q] = 0u;
          dcorr[q] = 0.f;
#pragma unroll
          for (int j = 0; j < kChunks; ++j) d[q][j] = 0.f;
          if ((have >> (kRecPerSeg * q + slot)) & 1u) {
            const SegFwd &f = w.segf[seg[q]];
            int dx, dy;
            slot_offset(f, slot, &dx, &dy);
            used[q] = main_weights<true>(p, tab, f, w.sega + seg[q], dx, dy, ms[q], nullptr, nullptr, lane);
            // cotangents of the samples (idx >= 1; the padded rows are zero at
            // idx = 0, where the record holds the boundary term's cotangent)
            const float *rec = w.mrec + ((size_t)seg[q] * kRecPerSeg + slot) * kRecFloats;
#pragma unroll
            for (int j = 0; j < kChunks; ++j) d[q][j] = rec[lane + j * kWarp];
            dcorr[q] = rec[0];
          }
          any |= used[q];
        }
        __syncwarp();
#pragma unroll 1
        for (; any; any &= any - 1) {
          const int e = __ffs(any) - 1;
          const float4 *src = rows + (size_t)e * kWinSamples;
          float4 t[kChunks];
#pragma unroll
          for (int j = 0; j < kChunks; ++j) t[j] = __ldg(src + j * kWarp);
#pragma unroll
          for (int q = 0; q < kAdjGroup; ++q) {
            if (!((used[q] >> e) & 1u)) continue;
            float2 sxy = make_float2(0.f, 0.f);
            float sz = 0.f;
#pragma unroll
            for (int j = 0; j < kChunks; ++j) {
              sxy = __ffma2_rn(make_float2(d[q][j], d[q][j]), make_float2(t[j].x, t[j].y), sxy);
              sz = fmaf(d[q][j], t[j].z, sz);
            }
            const float sx = sxy.x, sy = sxy.y;
            const float W = ms[q].W[e], dW = ms[q].dW[e];
            const float sB = (sy * qb[q] + sx * qa[q]) + sz * qc[q];
            acc_ne[q] = fmaf(W, sB, acc_ne[q]);
            acc_sig[q] = fmaf(dW, sB, acc_sig[q]);
            acc_a[q] = fmaf(W, sx, acc_a[q]);
            acc_b[q] = fmaf(W, sy, acc_b[q]);
            acc_c[q] = fmaf(W, sz, acc_c[q]);
          }
        }
#pragma unroll
        for (int q = 0; q < kAdjGroup; ++q)
          if (lane < __popc(used[q])) {
            acc_ne[q] += dcorr[q] * ms[q].cW[lane] * ms[q].cD[lane];
            acc_sig[q] += dcorr[q] * ms[q].cdW[lane] * ms[q].cD[lane];
          }
        __syncwarp();
      }
      // V and the boundary term carry n_e * W(sigma_T) * (a, b, c)(longdiff)
#pragma unroll
      for (int q = 0; q < kAdjGroup; ++q) {
        if (q >= ng) break;
        const SegAdj &a = w.sega[seg[q]];
        const float ne = w.segf[seg[q]].ne;
        const float sig = acc_sig[q] * ne;
        const float lsum = (acc_a[q] * a.dqa + acc_b[q] * a.dqb + acc_c[q] * a.dqc) * ne;
        float th[LSIM_NPARAM];
        th[0] = acc_ne[q] * a.dne[0];
        th[1] = acc_ne[q] * a.dne[1];
        th[2] = acc_ne[q] * a.dne[2] + sig * a.dsig[0] + lsum * a.dld[0];
        th[3] = acc_ne[q] * a.dne[3];
        th[4] = 0.f;
        th[5] = lsum * a.dld[1];
        th[6] = sig * a.dsig[1];
        th[7] = acc_ne[q] * a.dne[4];
#pragma unroll
        for (int k = 0; k < LSIM_NPARAM; ++k)
          if (k != 4) th[k] = warp_sum(th[k]);
        if (lane == 0) {
          float *dst = w.main_out + (size_t)seg[q] * kPixRec;
#pragma unroll
          for (int k = 0; k < LSIM_NPARAM; ++k) dst[1 + k] = th[k];
        }
      }
    }
  }
}

int run_main_records(const AccumArgs &a, cudaStream_t st) {
  if (a.n_rows <= 0) return LSIM_OK;
  const unsigned nb = (unsigned)((a.n_rows + 255) / 256);
  k_main_order_scan<<<1, kMaxTemplates, 0, st>>>(a.w);
  k_main_order_scatter<<<nb, 256, 0, st>>>(a.w, a.n_rows);
  with_main_shape([&](auto warps, int blocks) {
    k_main_records<warps.value><<<blocks, warps.value * kWarp, 0, st>>>(a.p, a.tab, a.w, a.g);
  });
  return cudaGetLastError() == cudaSuccess ? LSIM_OK : LSIM_ERR_CUDA;
}

int run_main_adjoint(const AccumArgs &a, cudaStream_t st) {
  // per-segment records; segments without main-bin records contribute zeros
  if (cudaMemsetAsync(a.w.main_out, 0, sizeof(float) * kPixRec * (size_t)a.n_rows, st) != cudaSuccess)
    return LSIM_ERR_CUDA;
  if (a.n_rows <= 0) return LSIM_OK;
  with_main_shape([&](auto warps, int blocks) {
    k_main_adjoint<warps.value><<<blocks, warps.value * kWarp, 0, st>>>(a.p, a.tab, a.w, a.g);
  });
  return cudaGetLastError() == cudaSuccess ? LSIM_OK : LSIM_ERR_CUDA;
}

}  // namespace lsim
