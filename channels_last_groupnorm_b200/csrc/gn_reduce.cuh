// Sums over a CTA (or a part of it with a barrier of its own) and over the CTAs of a sample, for the cooperative kernels.
//
// What bounds them is latency: the tensors rest meanwhile.  So all groups are reduced at once, 2^part_shift neighbouring
// threads to each, behind one barrier where a vector lies in one group.  Measured in gn_fwd_resident_kernel, from the
// CTA's last rows to its sums: 1.0 us against 1.9 with a warp per group and one group after the other (256@512^2, 32
// groups of 8 channels), 2.4 against 3.8 with groups of 4 channels (128@1024^2).
#pragma once
#include "gn_async.cuh"

namespace gnb200 {

// The threads that reduce and merge together: a CTA, or a part of it with a hardware barrier of its own.
struct Crew {
  int tid, threads, lane, warp, nwarps, bar;
  // (the thread-counting form: an aligned one may open early for a warp whose lanes come back from lane-0-only code)
  __device__ __forceinline__ void sync() const {
    __syncwarp();
    asm volatile("barrier.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory");
  }
};

__device__ __forceinline__ float part_sum(float v, int part_shift) {
  for (int b = (1 << part_shift) >> 1; b >= 1; b >>= 1) v += __shfl_xor_sync(0xffffffffu, v, b);
  return v;
}
// Column of channel c in a row of per-channel values: element e of neighbouring threads side by side, so that neither
// the stores nor the sums meet bank conflicts.
template <int VE>
__device__ __forceinline__ int chan_column(int c, int CV) {
  return (c & (VE - 1)) * CV + c / VE;
}

// Moments of every group over the crew's rows from the threads' (mean, M2) per lane of `cnt` rows each: the group's mean
// first, then the squared deviations around it.  publish(s, mean, M2) is called by one thread per group s.
//   red: TY * stride floats (UNI: twice), slot: G floats.  Rows ty, ty + TY, ... of the nrows belong to row lane ty.
template <int VE, bool UNI, typename Publish>
__device__ __forceinline__ void crew_moments(const Crew& cr, const Geom& g, const ReduceGeom& ex, const float (&mean)[VE],
                                             const float (&m2)[VE], float cnt, int tx, int ty, int nrows, float* red, float* slot,
                                             Publish publish) {
  const int s = cr.tid >> ex.part_shift, part = cr.tid & ((1 << ex.part_shift) - 1), parts = 1 << ex.part_shift;
  const int W = UNI ? g.D / VE : g.D, total = s < g.G ? g.TY * W : 0, lo = s * W;
  const float inv_n = 1.0f / ((float)nrows * (float)g.D);
  if constexpr (UNI) {
    const int rows_each = nrows / g.TY, more = nrows - rows_each * g.TY;  // row lanes below `more` have a row more
    float* red2 = red + g.TY * ex.stride;
    if (ty < g.TY) {
      float mt = 0.f, qt = 0.f, dev = 0.f;
#pragma unroll
      for (int e = 0; e < VE; ++e) mt += mean[e];
      mt *= 1.0f / VE;
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        const float d = mean[e] - mt;
        dev = fmaf(d, d, dev);
        qt += m2[e];
      }
      red[ty * ex.stride + tx] = mt;
      red2[ty * ex.stride + tx] = fmaf(cnt, dev, qt);
    }
    cr.sync();
    float acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = ex.div_W.div(i), c = i - j * W;
      acc = fmaf((float)(rows_each + (j < more ? 1 : 0)), red[j * ex.stride + lo + c], acc);
    }
    const float mu = part_sum(acc, ex.part_shift) * (VE * inv_n);
    acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = ex.div_W.div(i), c = i - j * W;
      const float d = red[j * ex.stride + lo + c] - mu;
      acc += fmaf((float)(VE * (rows_each + (j < more ? 1 : 0))) * d, d, red2[j * ex.stride + lo + c]);
    }
    acc = part_sum(acc, ex.part_shift);
    if (part == 0 && s < g.G) publish(s, mu, acc);
  } else {
    float* mine = red + ty * ex.stride + tx;
    if (ty < g.TY) {
#pragma unroll
      for (int e = 0; e < VE; ++e) mine[e * g.CV] = cnt * mean[e];
    }
    cr.sync();
    float acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = ex.div_W.div(i), c = lo + i - j * W;
      acc += red[j * ex.stride + chan_column<VE>(c, g.CV)];
    }
    const float mu = part_sum(acc, ex.part_shift) * inv_n;
    if (part == 0 && s < g.G) slot[s] = mu;
    cr.sync();
    if (ty < g.TY) {
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        const float d = mean[e] - slot[g.div_D.div(tx * VE + e)];
        mine[e * g.CV] = fmaf(cnt * d, d, m2[e]);
      }
    }
    cr.sync();
    acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = ex.div_W.div(i), c = lo + i - j * W;
      acc += red[j * ex.stride + chan_column<VE>(c, g.CV)];
    }
    acc = part_sum(acc, ex.part_shift);
    if (part == 0 && s < g.G) publish(s, mu, acc);
  }
}

// Per-channel sums over the row lanes of one value per lane: chan[c].  red: TY * stride floats, stride > C.  On return
// chan is not yet synchronised, and red may not be written before it is.
template <int VE>
__device__ __forceinline__ void crew_channel_sums(const Crew& cr, const Geom& g, const ReduceGeom& ex, const float (&v)[VE], int tx, int ty,
                                                  float* red, float* chan) {
  if (ty < g.TY) {
    float* mine = red + ty * ex.stride + tx;
#pragma unroll
    for (int e = 0; e < VE; ++e) mine[e * g.CV] = v[e];
  }
  cr.sync();
  for (int k = cr.tid; k < g.C; k += cr.threads) {  // k: column
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    const float* q = red + k;
    int r = 0;
    for (; r + 4 <= g.TY; r += 4, q += 4 * ex.stride) {
      a0 += q[0];
      a1 += q[ex.stride];
      a2 += q[2 * ex.stride];
      a3 += q[3 * ex.stride];
    }
    for (; r < g.TY; ++r, q += ex.stride) a0 += q[0];
    const int e = g.div_CV.div(k);
    chan[(k - e * g.CV) * VE + e] = (a0 + a1) + (a2 + a3);
  }
}

// gamma-weighted sums of every group over chan[0 .. C) and chan[C .. 2C); publish(s, w1, w2) by one thread per group
template <typename Publish>
__device__ __forceinline__ void crew_group_sums(const Crew& cr, const Geom& g, const ReduceGeom& ex, const float* gam, const float* chan,
                                                Publish publish) {
  const int s = cr.tid >> ex.part_shift, part = cr.tid & ((1 << ex.part_shift) - 1), parts = 1 << ex.part_shift;
  float w1 = 0.f, w2 = 0.f;
  const int end = s < g.G ? (s + 1) * g.D : 0;
  for (int c = s * g.D + part; c < end; c += parts) {
    w1 = fmaf(gam[c], chan[c], w1);
    w2 = fmaf(gam[c], chan[g.C + c], w2);
  }
  w1 = part_sum(w1, ex.part_shift);
  w2 = part_sum(w2, ex.part_shift);
  if (part == 0 && s < g.G) publish(s, w1, w2);
}

constexpr int kMergeRows = 10;  // partial rows a warp has in flight in a merge (148 CTAs / 16 warps)

// Sums over `rows` partial rows of G pairs each: warp w takes the rows w, w + nwarps, ..., lane l the groups l, l + 32, ...;
// acc[w * G + s], acc[(nwarps + w) * G + s] receive the warp's two sums of group s, formed in row order.  All CTAs of
// a sample read the same rows at the same moment, so what counts is the number of L2 requests: with one warp per
// group and a lane per row (32 requests of 8 or 16 bytes per load) a merge of 32 groups x 148 rows took 8.1 us.
// add(i, pair, K0, sum1, sum2) takes one pair of row i; K0 is the first value of the group's row 0.
template <typename Add>
__device__ __forceinline__ void merge_rows(const float2* p, int rows, int G, int warp, int nwarps, int lane, float* acc,
                                           Add add) {
  for (int s = lane; s < G; s += 32) {
    const float K0 = __ldcg(p + s).x;
    float a1 = 0.f, a2 = 0.f;
    for (int i0 = warp; i0 < rows; i0 += nwarps * kMergeRows) {
      float2 v[kMergeRows];
#pragma unroll
      for (int q = 0; q < kMergeRows; ++q) {
        const int i = i0 + nwarps * q;
        v[q] = i < rows ? __ldcg(p + (size_t)i * G + s) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < kMergeRows; ++q)
        if (i0 + nwarps * q < rows) add(i0 + nwarps * q, v[q], K0, a1, a2);
    }
    acc[warp * G + s] = a1;
    acc[(nwarps + warp) * G + s] = a2;
  }
}

}  // namespace gnb200
