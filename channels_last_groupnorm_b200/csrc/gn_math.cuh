// Per-thread arithmetic shared by the forward / backward kernels of every launch plan: running
// moments, affine coefficients, and one row of the backward sums.
#pragma once
#include "gn_common.cuh"

namespace gnb200 {

template <int VE>
__device__ __forceinline__ void welford_step(const float (&f)[VE], float (&mean)[VE], float (&m2)[VE], float& cnt) {
  cnt += 1.0f;
  const float inv = __fdividef(1.0f, cnt);
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    const float d = f[e] - mean[e];
    mean[e] = fmaf(d, inv, mean[e]);
    m2[e] = fmaf(d, f[e] - mean[e], m2[e]);
  }
}

// 16-bit tensors accumulate shifted sums instead: with K a value of the thread's own data (its
// first row),  s += x - K,  q += (x - K)^2;  the subtraction converts the 16-bit element on the fly
// (mixed-precision sub), three instructions per element and no division in the loop.  KN = VE: every
// lane has a K of its own, one of its samples, so (K - mean)^2 <= M2, q <= (n + 1) M2 and the cancellation
// in M2 = q - s^2 / n multiplies the rounding of q and s (sqrt(n) ulp or so) by at most n + 1, where sums of raw
// squares would multiply it by mean^2 / var.  KN = 1 (the lanes lie in one group): all lanes use lane 0's value, and
// the same holds for the M2 of the thread's VE * n samples about their common mean, with VE * n in the place of
// n + 1.  The callers keep n, the rows of one such sum, to 128 at most.
template <typename T, int VE, int KN>
__device__ __forceinline__ void shifted_step(const uint4& w, const float (&K)[KN], float (&s)[VE], float (&q)[VE]) {
  static_assert(sizeof(T) == 2 && VE == 8, "16-bit elements, 16-byte vectors");
  const uint32_t r[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint16_t lo, hi;
    split_halves(r[e], lo, hi);
    const float d0 = mixed_sub<T>(lo, K[KN == 1 ? 0 : 2 * e]);
    const float d1 = mixed_sub<T>(hi, K[KN == 1 ? 0 : 2 * e + 1]);
    add2(s[2 * e], s[2 * e + 1], s[2 * e], s[2 * e + 1], d0, d1);
    fma2(q[2 * e], q[2 * e + 1], d0, d1, d0, d1, q[2 * e], q[2 * e + 1]);
  }
}

// (s, q) about K over `rows` rows  ->  per-lane (mean, M2); s and q are overwritten.
template <int VE, int KN>
__device__ __forceinline__ void shifted_finish(const float (&K)[KN], int rows, float (&mean)[VE], float (&m2)[VE],
                                               float& cnt) {
  cnt = (float)rows;
  const float inv = rows > 0 ? 1.0f / cnt : 0.f;
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    const float s = mean[e], q = m2[e];
    const float ds = s * inv;
    mean[e] = K[KN == 1 ? 0 : e] + ds;
    m2[e] = fmaxf(fmaf(-s, ds, q), 0.f);
  }
}

// (pm, pq) of pn rows merged into (mean, m2) of cnt rows, lane by lane.
template <int VE>
__device__ __forceinline__ void merge_moments(const float (&pm)[VE], const float (&pq)[VE], float pn, float (&mean)[VE],
                                              float (&m2)[VE], float& cnt) {
  const float all = cnt + pn;
  const float f = all > 0.f ? pn / all : 0.f, h = cnt * f;
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    const float d = pm[e] - mean[e];
    m2[e] += fmaf(d * h, d, pq[e]);
    mean[e] = fmaf(d, f, mean[e]);
  }
  cnt = all;
}

// Per-lane affine coefficients  a = rstd * gamma,  b = beta - mean * a  for the thread's channels.
// `stat_mean` / `stat_rstd` are indexed by group relative to g_base.  UNI: all VE channels of the
// thread belong to one group, so the statistics are looked up once.
template <typename T, int VE, bool UNI>
__device__ __forceinline__ void lane_affine(const T* gamma, const T* beta, const float* stat_mean,
                                            const float* stat_rstd, int g_base, int c_first, const FastDiv div_D,
                                            float (&a)[VE], float (&b)[VE]) {
  float ga[VE], be[VE];
  load_params<T, VE>(gamma, c_first, ga);
  load_params<T, VE>(beta, c_first, be);
  if constexpr (UNI) {
    const int s = div_D.div(c_first) - g_base;
    const float mu = stat_mean[s], rs = stat_rstd[s];
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      a[e] = rs * ga[e];
      b[e] = fmaf(-mu, a[e], be[e]);
    }
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const int s = div_D.div(c_first + e) - g_base;
      a[e] = stat_rstd[s] * ga[e];
      b[e] = fmaf(-stat_mean[s], a[e], be[e]);
    }
  }
}

// The same from parameter vectors fetched earlier (raw 16-byte loads issued before phase 1 so that
// their latency is off the critical path between the statistics and the output pass).
template <typename T, int VE, bool UNI>
__device__ __forceinline__ void lane_affine_raw(const uint4& ga_raw, const uint4& be_raw, const float* stat_mean,
                                                const float* stat_rstd, int g_base, int c_first, const FastDiv div_D,
                                                float (&a)[VE], float (&b)[VE]) {
  static_assert(sizeof(T) * VE == 16, "16-byte vectors only");
  float ga[VE], be[VE];
  unpack16<T, VE>(ga_raw, ga);
  unpack16<T, VE>(be_raw, be);
  if constexpr (UNI) {
    const int s = div_D.div(c_first) - g_base;
    const float mu = stat_mean[s], rs = stat_rstd[s];
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      a[e] = rs * ga[e];
      b[e] = fmaf(-mu, a[e], be[e]);
    }
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const int s = div_D.div(c_first + e) - g_base;
      a[e] = stat_rstd[s] * ga[e];
      b[e] = fmaf(-stat_mean[s], a[e], be[e]);
    }
  }
}

// CTA-local moments of every group slot of the column block from the per-thread Welford states:
// first the slot means (sum of cnt * mean / n), then the squared deviations around them.
//   slot[s]            = local mean      slot[slots + s] = local M2      slot[2 * slots + s] = local count
// scratch: red (TY * CW floats), tmp (slots floats).
template <int VE, bool UNI>
__device__ __forceinline__ void cta_slot_moments(const Geom& g, const float (&mean)[VE], const float (&m2)[VE],
                                                 float cnt, int tx, int ty, int c0, int nrows, int g_lo, int n_slots,
                                                 float* red, float* tmp, float* slot) {
  constexpr int NV = UNI ? 1 : VE;
  float val[NV];
  if constexpr (UNI) {
    float sm = 0.f;
#pragma unroll
    for (int e = 0; e < VE; ++e) sm += mean[e];
    val[0] = cnt * sm;
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) val[e] = cnt * mean[e];
  }
  cta_group_sum<VE, NV>(g, val, tx, ty, c0, g_lo, n_slots, red, tmp);
  const int c_end = min(c0 + g.CW, g.C);
  for (int s = threadIdx.x; s < n_slots; s += blockDim.x) {
    const int w = min((g_lo + s + 1) * g.D, c_end) - max((g_lo + s) * g.D, c0);
    const float n_loc = (float)nrows * (float)w;
    slot[s] = n_loc > 0.f ? tmp[s] / n_loc : 0.f;
    slot[2 * g.slots + s] = n_loc;
  }
  __syncthreads();
  if constexpr (UNI) {
    const float lm = slot[g.div_D.div(min(c0 + tx * VE, g.C - 1)) - g_lo];
    float acc = 0.f, dev = 0.f;
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const float d = mean[e] - lm;
      dev = fmaf(d, d, dev);
      acc += m2[e];
    }
    val[0] = fmaf(cnt, dev, acc);
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const int c = min(c0 + tx * VE + e, g.C - 1);
      const float d = mean[e] - slot[g.div_D.div(c) - g_lo];
      val[e] = fmaf(cnt * d, d, m2[e]);
    }
  }
  cta_group_sum<VE, NV>(g, val, tx, ty, c0, g_lo, n_slots, red, slot + g.slots);
}

template <typename T, int VE>
struct BwdLane {
  float r[VE];    // rstd of the lane's group
  float nmr[VE];  // -mean * rstd
  float ga[VE];   // gamma
  float be[VE];   // beta
};

// UNI: all VE channels of the thread belong to one group (one statistics lookup; the compiler
// then keeps a single register for each of r / nmr).
template <typename T, int VE, bool UNI>
__device__ __forceinline__ void lane_setup(const T* gamma, const T* beta, const float* mean_n, const float* rstd_n,
                                           int c_first, const FastDiv div_D, BwdLane<T, VE>& L) {
  load_params<T, VE>(gamma, c_first, L.ga);
  load_params<T, VE>(beta, c_first, L.be);
  if constexpr (UNI) {
    const int grp = div_D.div(c_first);
    const float rs = rstd_n[grp];
    const float nm = -mean_n[grp] * rs;
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      L.r[e] = rs;
      L.nmr[e] = nm;
    }
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const int grp = div_D.div(c_first + e);
      const float rs = rstd_n[grp];
      L.r[e] = rs;
      L.nmr[e] = -mean_n[grp] * rs;
    }
  }
}

// The same in two steps, loads and arithmetic, for kernels that have something to start in between.
template <typename T, int VE, bool UNI>
struct LaneParams {
  static_assert(sizeof(T) * VE == 16, "16-byte vectors only");
  static constexpr int NS = UNI ? 1 : VE;
  uint4 ga, be;
  float mean[NS], rstd[NS];
  __device__ __forceinline__ void load(const T* gamma, const T* beta, const float* mean_n, const float* rstd_n, int c_first,
                                       const FastDiv div_D) {
    ga = *reinterpret_cast<const uint4*>(gamma + c_first);
    be = *reinterpret_cast<const uint4*>(beta + c_first);
#pragma unroll
    for (int e = 0; e < NS; ++e) {
      const int grp = div_D.div(c_first + e);
      mean[e] = mean_n[grp];
      rstd[e] = rstd_n[grp];
    }
  }
  __device__ __forceinline__ void unpack(BwdLane<T, VE>& L) const {
    unpack16<T, VE>(ga, L.ga);
    unpack16<T, VE>(be, L.be);
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      L.r[e] = rstd[UNI ? 0 : e];
      L.nmr[e] = -mean[UNI ? 0 : e] * L.r[e];
    }
  }
};

// One row of phase 1: dyh = dy * act'(yh) for the thread's VE channels, sums updated.
template <typename T, int VE, int ACT>
__device__ __forceinline__ void bwd_row_sums(const float (&fx)[VE], float (&fd)[VE], const BwdLane<T, VE>& L,
                                             float (&s1)[VE], float (&s2)[VE]) {
  float xh[VE], yh[VE], gr[VE];
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    xh[e] = fmaf(fx[e], L.r[e], L.nmr[e]);
    yh[e] = fmaf(xh[e], L.ga[e], L.be[e]);
  }
  act_grad_vec<T, VE, ACT>(yh, gr);
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    fd[e] *= gr[e];
    s1[e] += fd[e];
    s2[e] = fmaf(fd[e], xh[e], s2[e]);
  }
}

// 16-bit tensors, fused path: yh straight from x (a = rstd * gamma, b = beta - mean * a) and S2
// accumulated against the raw x; the caller converts it with S2 = rstd * (S2raw - mean * S1).  One
// FMA per element less; the conversion's rounding (relative 1e-7 * |mean| * rstd) is far below a
// 16-bit result.
// It works on the packed 16-bit values: dyh = dy * act'(yh) is formed two channels at a time in the tensor's own 16-bit format - which is
// the format it is parked in anyway - and enters the fp32 sums through mixed-precision add / fma,
// so dy is never unpacked and dyh never packed.  act' is evaluated in f16x2; for bf16 tensors it
// is rounded to bf16 before the product.  Returns the packed dyh.
// PAIRS: packed fp32 instructions, which want their operands in register pairs.
template <typename T, int ACT, bool PAIRS = kPairs<T>>
__device__ __forceinline__ uint4 bwd_row_sums_packed(const uint4& xw, const uint4& dw, const float (&a)[8],
                                                     const float (&b)[8], float (&s1)[8], float (&s2)[8]) {
  static_assert(sizeof(T) == 2, "16-bit tensors only");
  const uint32_t xr[4] = {xw.x, xw.y, xw.z, xw.w}, dr[4] = {dw.x, dw.y, dw.z, dw.w};
  uint32_t out[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint16_t x0, x1;
    split_halves(xr[p], x0, x1);
    uint32_t dyh = dr[p];
    if constexpr (ACT != kActIdentity) {
      float yh0, yh1;
      if constexpr (PAIRS) {
        fma2(yh0, yh1, mixed_add<T>(x0, -0.0f), mixed_add<T>(x1, -0.0f), a[2 * p], a[2 * p + 1], b[2 * p], b[2 * p + 1]);
      } else {
        yh0 = fmaf(mixed_add<T>(x0, -0.0f), a[2 * p], b[2 * p]);
        yh1 = fmaf(mixed_add<T>(x1, -0.0f), a[2 * p + 1], b[2 * p + 1]);
      }
      const __half2 g = act_grad_pair<ACT>(yh0, yh1);
      if constexpr (std::is_same<T, __half>::value) {
        const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&dr[p]), g);
        dyh = *reinterpret_cast<const uint32_t*>(&r);
      } else {
        const float2 gf = __half22float2(g);
        const __nv_bfloat162 gb = __floats2bfloat162_rn(gf.x, gf.y);
        const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&dr[p]), gb);
        dyh = *reinterpret_cast<const uint32_t*>(&r);
      }
    }
    uint16_t d0, d1;
    split_halves(dyh, d0, d1);
    s1[2 * p] = mixed_add<T>(d0, s1[2 * p]);
    s1[2 * p + 1] = mixed_add<T>(d1, s1[2 * p + 1]);
    s2[2 * p] = mixed_fma<T>(d0, x0, s2[2 * p]);
    s2[2 * p + 1] = mixed_fma<T>(d1, x1, s2[2 * p + 1]);
    out[p] = dyh;
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}

}  // namespace gnb200
