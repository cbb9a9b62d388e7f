// Sums over a CTA (or a part of it with a barrier of its own) and over the CTAs of a sample, for the cooperative kernels.
//
// What bounds them is latency: the tensors rest meanwhile.  So all groups are reduced at once, 2^part_shift neighbouring
// threads to each, behind one barrier where a vector lies in one group.  Measured in gn_fwd_resident_kernel, from the
// CTA's last rows to its sums: 1.0 us against 1.9 with a warp per group and one group after the other (256@512^2, 32
// groups of 8 channels), 2.4 against 3.8 with groups of 4 channels (128@1024^2).  In the fused forward kernel, whose small
// maps with groups of 10, 20 or 30 channels are a chain of dependent instructions, device us per call, channel by channel / this way: 320@64^2
// 9.1 / 7.6, 640@32^2 9.2 / 5.8, 2 x 960@76^2 34.5 / 24.9.
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

// Moments of every group of the column block (`groups`, all whole) over the crew's rows from the threads' (mean, M2) per
// lane of `cnt` rows each: the group's mean first, then the squared deviations around it.  publish(s, mean, M2) is called by
// one thread per group s.
//   red: reduce_layout() floats, slot: one per group.  Rows ty, ty + TY, ... of the nrows belong to row lane ty.
template <int VE, bool UNI, typename Publish>
__device__ __forceinline__ void crew_moments(const Crew& cr, const Geom& g, int groups, const float (&mean)[VE],
                                             const float (&m2)[VE], float cnt, int tx, int ty, int nrows, float* red, float* slot,
                                             Publish publish) {
  const int s = cr.tid >> g.rd.part_shift, part = cr.tid & ((1 << g.rd.part_shift) - 1), parts = 1 << g.rd.part_shift;
  const int W = UNI ? g.D / VE : g.D, total = s < groups ? g.TY * W : 0, lo = s * W;  // (no more groups than threads if D >= VE)
  const float inv_n = 1.0f / ((float)nrows * (float)g.D);
  if constexpr (UNI) {
    const int rows_each = nrows / g.TY, more = nrows - rows_each * g.TY;  // row lanes below `more` have a row more
    float* red2 = red + g.TY * g.rd.stride;
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
      red[ty * g.rd.stride + tx] = mt;
      red2[ty * g.rd.stride + tx] = fmaf(cnt, dev, qt);
    }
    cr.sync();
    float acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = g.rd.div_W.div(i), c = i - j * W;
      acc = fmaf((float)(rows_each + (j < more ? 1 : 0)), red[j * g.rd.stride + lo + c], acc);
    }
    const float mu = part_sum(acc, g.rd.part_shift) * (VE * inv_n);
    acc = 0.f;
    for (int i = part; i < total; i += parts) {
      const int j = g.rd.div_W.div(i), c = i - j * W;
      const float d = red[j * g.rd.stride + lo + c] - mu;
      acc += fmaf((float)(VE * (rows_each + (j < more ? 1 : 0))) * d, d, red2[j * g.rd.stride + lo + c]);
    }
    acc = part_sum(acc, g.rd.part_shift);
    if (part == 0 && s < groups) publish(s, mu, acc);
  } else if (g.D >= VE) {
    // a vector touches two groups at most: the thread's lanes of either are a part with a mean and an M2 of their own
    const int rows_each = nrows / g.TY, more = nrows - rows_each * g.TY;
    const int W = (g.D + 2 * VE - 2) / VE, pitch = 2 * g.CV + 1;  // vectors that a group can touch; parts per row, odd
    float2* parts2 = reinterpret_cast<float2*>(red);
    if (ty < g.TY) {
      const int n0 = min(VE, (g.div_D.div(tx * VE) + 1) * g.D - tx * VE);  // lanes of the first part
      float a0 = 0.f, a1 = 0.f, q0 = 0.f, q1 = 0.f, d0 = 0.f, d1 = 0.f;
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        a0 += e < n0 ? mean[e] : 0.f;
        a1 += e < n0 ? 0.f : mean[e];
      }
      a0 = a0 / (float)n0;
      a1 = n0 < VE ? a1 / (float)(VE - n0) : 0.f;
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        const float d = mean[e] - (e < n0 ? a0 : a1);
        d0 = e < n0 ? fmaf(d, d, d0) : d0;  // (chosen, not multiplied by 0: the other part's d may be infinite or NaN)
        d1 = e < n0 ? d1 : fmaf(d, d, d1);
        q0 += e < n0 ? m2[e] : 0.f;
        q1 += e < n0 ? 0.f : m2[e];
      }
      parts2[ty * pitch + 2 * tx] = make_float2(a0, fmaf(cnt, d0, q0));
      parts2[ty * pitch + 2 * tx + 1] = make_float2(a1, fmaf(cnt, d1, q1));
    }
    cr.sync();
    const int c_lo = s * g.D, c_hi = c_lo + g.D, t_lo = c_lo / VE, entries = s < groups ? g.TY * W : 0;
    auto entry = [&](int i, float& n, float2& v) {
      const int j = g.rd.div_W.div(i), t = t_lo + i - j * W;
      const int lanes = min((t + 1) * VE, c_hi) - max(t * VE, c_lo);
      if (lanes <= 0) return false;
      n = (float)(lanes * (rows_each + (j < more ? 1 : 0)));
      v = parts2[j * pitch + 2 * t + (t * VE < c_lo ? 1 : 0)];
      return true;
    };
    float acc = 0.f, n = 0.f;
    float2 v = make_float2(0.f, 0.f);
    for (int i = part; i < entries; i += parts)
      if (entry(i, n, v)) acc = fmaf(n, v.x, acc);
    const float mu = part_sum(acc, g.rd.part_shift) * inv_n;
    acc = 0.f;
    for (int i = part; i < entries; i += parts) {
      if (!entry(i, n, v)) continue;
      const float d = v.x - mu;
      acc += fmaf(n * d, d, v.y);
    }
    acc = part_sum(acc, g.rd.part_shift);
    if (part == 0 && s < groups) publish(s, mu, acc);
  } else {
    float* mine = red + ty * g.rd.stride + tx;
    if (ty < g.TY) {
#pragma unroll
      for (int e = 0; e < VE; ++e) mine[e * g.CV] = cnt * mean[e];
    }
    cr.sync();
    // A CTA can have more of these groups than threads (64 samples of 25 rows x 1280 channels, one a group: 160 groups a block, 128
    // threads), so the threads walk over them; all make the same number of rounds, since part_sum wants whole warps.
    const int step = cr.threads >> g.rd.part_shift;
    auto group_sum = [&](int grp) {
      float acc = 0.f;
      for (int i = part; i < (grp < groups ? g.TY * W : 0); i += parts) {
        const int j = g.rd.div_W.div(i), c = grp * W + i - j * W;
        acc += red[j * g.rd.stride + chan_column<VE>(c, g.CV)];
      }
      return part_sum(acc, g.rd.part_shift);
    };
    for (int s0 = 0; s0 < groups; s0 += step) {
      const float mu = group_sum(s0 + s) * inv_n;
      if (part == 0 && s0 + s < groups) slot[s0 + s] = mu;
    }
    cr.sync();
    if (ty < g.TY) {
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        const float d = mean[e] - slot[g.div_D.div(tx * VE + e)];
        mine[e * g.CV] = fmaf(cnt * d, d, m2[e]);
      }
    }
    cr.sync();
    for (int s0 = 0; s0 < groups; s0 += step) {
      const float q = group_sum(s0 + s);
      if (part == 0 && s0 + s < groups) publish(s0 + s, slot[s0 + s], q);
    }
  }
}

// Per-channel sums over the row lanes of one value per lane: chan[c].  red: TY * stride floats, stride > C.  On return
// chan is not yet synchronised, and red may not be written before it is.
template <int VE>
__device__ __forceinline__ void crew_channel_sums(const Crew& cr, const Geom& g, const float (&v)[VE], int tx, int ty,
                                                  float* red, float* chan) {
  if (ty < g.TY) {
    float* mine = red + ty * g.rd.stride + tx;
#pragma unroll
    for (int e = 0; e < VE; ++e) mine[e * g.CV] = v[e];
  }
  cr.sync();
  for (int k = cr.tid; k < g.C; k += cr.threads) {  // k: column
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    const float* q = red + k;
    int r = 0;
    for (; r + 4 <= g.TY; r += 4, q += 4 * g.rd.stride) {
      a0 += q[0];
      a1 += q[g.rd.stride];
      a2 += q[2 * g.rd.stride];
      a3 += q[3 * g.rd.stride];
    }
    for (; r < g.TY; ++r, q += g.rd.stride) a0 += q[0];
    const int e = g.div_CV.div(k);
    chan[(k - e * g.CV) * VE + e] = (a0 + a1) + (a2 + a3);
  }
}

// gamma-weighted sums of every group over chan[0 .. C) and chan[C .. 2C); publish(s, w1, w2) by one thread per group
template <typename Publish>
__device__ __forceinline__ void crew_group_sums(const Crew& cr, const Geom& g, const float* gam, const float* chan,
                                                Publish publish) {
  const int s = cr.tid >> g.rd.part_shift, part = cr.tid & ((1 << g.rd.part_shift) - 1), parts = 1 << g.rd.part_shift;
  float w1 = 0.f, w2 = 0.f;
  const int end = s < g.G ? (s + 1) * g.D : 0;
  for (int c = s * g.D + part; c < end; c += parts) {
    w1 = fmaf(gam[c], chan[c], w1);
    w2 = fmaf(gam[c], chan[g.C + c], w2);
  }
  w1 = part_sum(w1, g.rd.part_shift);
  w2 = part_sum(w2, g.rd.part_shift);
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
