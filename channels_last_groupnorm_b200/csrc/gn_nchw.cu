// GroupNorm (+activation) for channels-first (NCHW) tensors, forward and backward, sm_100a.
//
// The reference sends inputs whose channel stride is not 1 to torch's group_norm followed by the
// activation (src/gnnhwc/custom_gn.py:75-79); there is no permute here and no call into torch: in
// NCHW storage the slab of (sample n, group g) is one contiguous run of D * R elements, and the R
// pixels of a channel are contiguous inside it, so the statistics are plain contiguous reductions
// and gamma / beta are per-run scalars.
//
//   forward   stats kernel (partial moments per slab chunk) -> apply kernel (merges the slab's
//             partials in a fixed order, then y = act(x a_c + b_c))
//   backward  reduce kernel (one warp per piece of a channel row: S1, S2) -> finalize kernel
//             (per-channel sums, group sums A, B) -> parameter-gradient kernel -> dx kernel
//
// Vectors are 16 bytes when R is a multiple of the vector width and the pointers are aligned (every
// channel row then starts on a 16-byte boundary), single elements otherwise.  Sums are fp32, formed in
// an order fixed by the launch geometry: no atomics, bit-identical reruns.
#include "gn_async.cuh"
#include "gn_kernels.h"
#include "gn_math.cuh"

namespace gnb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 4;

struct NchwGeom {
  int N, C, G, D;
  long long R;
  long long slab_vecs;   // vectors per (n, g) slab: D * R / VE
  long long chunk_vecs;  // forward: vectors per CTA chunk
  int chunks;            // forward: chunks per slab
  long long row_vecs;    // backward: vectors per channel row: R / VE
  long long piece_vecs;  // backward: vectors per warp piece
  int ppr;               // backward: pieces per channel row
  FastDiv div_R;         // element offset inside a slab -> channel (R < 2^31)
  int evict;             // results leave with streaming stores
};

template <typename T, int VE>
__device__ __forceinline__ void load_vec(const T* p, float (&f)[VE]) {
  if constexpr (sizeof(T) * VE == 16) {
    unpack16<T, VE>(ldg128(p), f);
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) f[e] = load_param<T>(p, e);
  }
}
// 16 bytes of a result.  A tensor that L2 can hold besides the inputs is left to the kernel that reads it next
// (and streaming it measured 2 % slower); a larger one must not push out the inputs that are still to be read again.
__device__ __forceinline__ void store16(void* p, const uint4 v, int evict) {
  if (evict)
    stg128_stream(p, v);
  else
    stg128(p, v);
}
// The same without a branch, for the dx kernel, whose arithmetic for the four vectors in flight a branch would keep
// apart.  (The forward's output pass is the other way round: 8 x 256@64^2 bf16 11.9 us with the branch, 12.8 without, 4 x
// 320@48^2 8.2 and 9.3.)
__device__ __forceinline__ void store16_predicated(void* p, const uint4 v, int evict) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.s32 p, %5, 0;\n"
      "@p st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};\n"
      "@!p st.global.v4.u32 [%0], {%1, %2, %3, %4};\n"
      "}\n" ::"l"(p),
      "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(evict)
      : "memory");
}
template <typename T, int VE>
__device__ __forceinline__ void store_vec(T* p, const float (&f)[VE], int evict) {
  if constexpr (sizeof(T) * VE == 16) {
    store16_predicated(p, pack16<T, VE>(f), evict);
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) p[e] = store_param<T>(f[e]);
  }
}

// Moments of a batch of U vectors, all of one group, merged into the thread's running (mean, M2) of cnt elements.
// The batch is summed about the running mean and its squares are taken about the batch's own mean, so neither a
// large common offset nor an outlier cancels anything.  (Sums of squares about one fixed sample K lose precision when
// K is an outlier, and its square, counted once for every other element, overflows in bf16 where M2 does not.)  Four instructions per element like
// Welford's, but one division per batch instead of one per vector, and the vectors stay packed while in flight.
// Measured (forward, us, fixed sample -> batches): 512@256^2 fp16 39.8 -> 36.2, 64 x 256@64^2 bf16 74.7 -> 70.1,
// 8 x 256@64^2 bf16 13.8 -> 11.7, 32 x 64@56^2 fp16 17.3 -> 14.2; rstd within 3e-7 of fp64 in every case tried.
template <typename T, int U>
__device__ __forceinline__ void batch_moments(const uint4 (&w)[U], float& mean, float& m2, float& cnt) {
  constexpr float n = 8.f * U;
  float s[2] = {0.f, 0.f}, q[2] = {0.f, 0.f};
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t r[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint16_t lo, hi;
      split_halves(r[e], lo, hi);
      add2(s[0], s[1], s[0], s[1], mixed_sub<T>(lo, mean), mixed_sub<T>(hi, mean));
    }
  }
  const float d = (s[0] + s[1]) * (1.f / n), mb = mean + d;  // 1 / n is a power of two
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t r[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint16_t lo, hi;
      split_halves(r[e], lo, hi);
      const float d0 = mixed_sub<T>(lo, mb), d1 = mixed_sub<T>(hi, mb);
      fma2(q[0], q[1], d0, d1, d0, d1, q[0], q[1]);
    }
  }
  const float f = __fdividef(n, cnt + n);
  m2 += fmaf(d * (cnt * f), d, q[0] + q[1]);
  mean = fmaf(d, f, mean);
  cnt += n;
}

// ------------------------------------------------------------------------------------------------
// forward 1: partial moments of chunk `chunk` of slab `slab` -> part[slab * chunks + chunk] = (mean, M2, n, -)
// ------------------------------------------------------------------------------------------------
template <typename T, int VE>
__global__ void __launch_bounds__(kThreads)
    gn_nchw_stats_kernel(const T* __restrict__ x, float4* __restrict__ part, const NchwGeom g) {
  __shared__ float scratch[kThreads / 32];
  grid_dep_launch_dependents();  // the apply kernel may take its place; it waits for this grid's partials
  const long long slab = blockIdx.x / g.chunks;
  const int chunk = (int)(blockIdx.x - slab * g.chunks);
  const long long v0 = (long long)chunk * g.chunk_vecs;
  const long long v1 = min(g.slab_vecs, v0 + g.chunk_vecs);
  const T* base = x + slab * g.slab_vecs * VE;
  // 16-bit vectors: one running (mean, M2) per thread, fed by batches; else Welford, a state per lane of the vectors
  // (one count for all lanes)
  constexpr bool kBatched = sizeof(T) == 2 && VE == 8;
  constexpr int L = kBatched ? 1 : VE;
  float mean[L], m2[L], cnt = 0.f;
#pragma unroll
  for (int e = 0; e < L; ++e) mean[e] = 0.f, m2[e] = 0.f;
  long long v = v0 + threadIdx.x;
  if constexpr (kBatched) {
    if (v < v1) mean[0] = load_param<T>(base + v * VE, 0);  // where the first batch is summed about
    for (; v + (kUnroll - 1) * kThreads < v1; v += kUnroll * kThreads) {
      uint4 w[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) w[u] = ldg128(base + (v + u * kThreads) * VE);
      batch_moments<T>(w, mean[0], m2[0], cnt);
    }
    for (; v < v1; v += kThreads) {
      const uint4 w[1] = {ldg128(base + v * VE)};
      batch_moments<T>(w, mean[0], m2[0], cnt);
    }
  } else {
    for (; v + (kUnroll - 1) * kThreads < v1; v += kUnroll * kThreads) {
      float f[kUnroll][VE];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) load_vec<T, VE>(base + (v + u * kThreads) * VE, f[u]);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) welford_step<VE>(f[u], mean, m2, cnt);
    }
    for (; v < v1; v += kThreads) {
      float f[VE];
      load_vec<T, VE>(base + v * VE, f);
      welford_step<VE>(f, mean, m2, cnt);
    }
  }
  // lanes -> thread, then threads -> CTA: mean first, squared deviations about it second
  float tsum = 0.f;
#pragma unroll
  for (int e = 0; e < L; ++e) tsum += mean[e];
  const float n_cta = block_sum(cnt * (float)L, scratch);
  const float mu = block_sum(cnt * tsum, scratch) / n_cta;
  float dev = 0.f;
#pragma unroll
  for (int e = 0; e < L; ++e) {
    const float d = mean[e] - mu;
    dev += fmaf(cnt * d, d, m2[e]);
  }
  const float M2 = block_sum(dev, scratch);
  if (threadIdx.x == 0) part[blockIdx.x] = make_float4(mu, M2, n_cta, 0.f);
}

// Fixed-order merge of the `chunks` partials of a slab by one warp (sums about the first chunk's
// mean, so that nothing cancels for a large |mean|).  Every lane returns the result.
__device__ __forceinline__ void merge_partials(const float4* __restrict__ p, int chunks, float eps, float& mu, float& rs) {
  const int lane = threadIdx.x & 31;
  const float K0 = p[0].x;
  float an = 0.f, ad = 0.f, aq = 0.f;
  for (int i = lane; i < chunks; i += 32) {
    const float4 v = p[i];
    const float d = v.x - K0;
    an += v.z;
    ad = fmaf(v.z, d, ad);
    aq += fmaf(v.z * d, d, v.y);
  }
#pragma unroll
  for (int b = 16; b >= 1; b >>= 1) {
    an += __shfl_xor_sync(0xffffffffu, an, b);
    ad += __shfl_xor_sync(0xffffffffu, ad, b);
    aq += __shfl_xor_sync(0xffffffffu, aq, b);
  }
  const float dm = ad / an;
  mu = K0 + dm;
  rs = rsqrtf(fmaxf(fmaf(-ad, dm, aq) / an, 0.f) + eps);
}

// ------------------------------------------------------------------------------------------------
// forward 2: statistics of the slab, then y = act(x * a_c + b_c) over the chunk.  The chunks are visited in the
// reverse order of the statistics kernel and walked from their end, and y leaves with streaming stores: what that
// kernel read last is read first, while L2 still holds it.
// ------------------------------------------------------------------------------------------------
template <typename T, int VE, int ACT>
__global__ void __launch_bounds__(kThreads)
    gn_nchw_apply_kernel(const T* __restrict__ x, const T* __restrict__ gamma, const T* __restrict__ beta,
                         const float4* __restrict__ part, T* __restrict__ y, float* __restrict__ mean_out,
                         float* __restrict__ rstd_out, float eps, const NchwGeom g) {
  constexpr bool FAST = sizeof(T) == 2;
  __shared__ float s_stat[2];
  const unsigned id = gridDim.x - 1 - blockIdx.x;
  const long long slab = id / g.chunks;
  const int chunk = (int)(id - slab * g.chunks);
  grid_dep_wait();  // the statistics kernel's partials
  if (threadIdx.x < 32) {
    float mu, rs;
    merge_partials(part + slab * g.chunks, g.chunks, eps, mu, rs);
    if (threadIdx.x == 0) {
      s_stat[0] = mu;
      s_stat[1] = rs;
      if (chunk == 0) {
        mean_out[slab] = mu;
        rstd_out[slab] = rs;
      }
    }
  }
  __syncthreads();
  const float mu = s_stat[0], rs = s_stat[1];
  const int c_base = (int)(slab % g.G) * g.D;
  const long long v0 = (long long)chunk * g.chunk_vecs;
  const long long v1 = min(g.slab_vecs, v0 + g.chunk_vecs);
  const T* xs = x + slab * g.slab_vecs * VE;
  T* ys = y + slab * g.slab_vecs * VE;
  auto one = [&](long long v, const float (&f)[VE]) {
    // VE > 1: the vector lies inside one channel row (R is a multiple of VE)
    const int c = c_base + g.div_R.div((int)(v * VE));
    const float a = rs * load_param<T>(gamma, c);
    const float b = fmaf(-mu, a, load_param<T>(beta, c));
    float o[VE];
    if constexpr (VE % 2 == 0) {
#pragma unroll
      for (int e = 0; e < VE; e += 2) fma2(o[e], o[e + 1], f[e], f[e + 1], a, a, b, b);
    } else {
#pragma unroll
      for (int e = 0; e < VE; ++e) o[e] = fmaf(f[e], a, b);
    }
    if constexpr (sizeof(T) * VE == 16) {
      store16(ys + v * VE, act_pack16<T, VE, ACT>(o), g.evict);
    } else {
#pragma unroll
      for (int e = 0; e < VE; ++e) ys[v * VE + e] = store_param<T>(act_fwd<ACT, FAST>(o[e]));
    }
  };
  long long v = v1 - 1 - threadIdx.x;
  for (; v - (kUnroll - 1) * kThreads >= v0; v -= kUnroll * kThreads) {
    if constexpr (sizeof(T) * VE == 16) {  // packed while in flight
      uint4 w[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) w[u] = ldg128(xs + (v - u * kThreads) * VE);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        float f[VE];
        unpack16<T, VE>(w[u], f);
        one(v - u * kThreads, f);
      }
    } else {
      float f[kUnroll][VE];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) load_vec<T, VE>(xs + (v - u * kThreads) * VE, f[u]);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) one(v - u * kThreads, f[u]);
    }
  }
  for (; v >= v0; v -= kThreads) {
    float f[VE];
    load_vec<T, VE>(xs + v * VE, f);
    one(v, f);
  }
}

// ------------------------------------------------------------------------------------------------
// backward 1: one warp per piece of a channel row:  tp[(n * C + c) * ppr + j] = (S1, S2)
// Bound by instruction issue (about 100 instructions per pair of 16-byte vectors) before it is bound by HBM: so two lanes per
// instruction, and vectors that stay packed while in flight (four CTAs per SM); the kernels of the other passes likewise.  What that gives,
// device us of forward and backward, scalar and unpacked / so: 512@256^2 fp16 35.5 / 33.4, 68.1 / 65.9; 32 x 64@56^2 fp32 18.6 / 18.3, 34.5 / 31.5.
// Single elements (rows that are no multiple of a vector) are bound by latency instead: five CTAs, and a remainder loop that is not unrolled, since
// its registers would leave four: then backward calls with short rows take 1.09 (16 x 2048@7^2) and 1.05 (84 x 2048 x 221 rows) of the time, mean over
// types and activations; rows of 30159 and 65025 elements the same.
// ------------------------------------------------------------------------------------------------
// xh = x * rs + nmr and yh = xh * ga + be, lane by lane
template <int VE>
__device__ __forceinline__ void normalise(const float (&fx)[VE], float rs, float nmr, float ga, float be, float (&xh)[VE], float (&yh)[VE]) {
  if constexpr (VE % 2 == 0) {
#pragma unroll
    for (int e = 0; e < VE; e += 2) {
      fma2(xh[e], xh[e + 1], fx[e], fx[e + 1], rs, rs, nmr, nmr);
      fma2(yh[e], yh[e + 1], xh[e], xh[e + 1], ga, ga, be, be);
    }
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      xh[e] = fmaf(fx[e], rs, nmr);
      yh[e] = fmaf(xh[e], ga, be);
    }
  }
}
template <typename T, int VE, int ACT>
__global__ void __launch_bounds__(kThreads, VE > 1 ? 4 : 5)
    gn_nchw_reduce_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                          const T* __restrict__ beta, const float* __restrict__ mean_in,
                          const float* __restrict__ rstd_in, float2* __restrict__ tp, long long pieces,
                          const NchwGeom g) {
  grid_dep_launch_dependents();  // the kernels after this one wait for this grid before they read its sums
  const int lane = threadIdx.x & 31;
  const long long piece = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (piece >= pieces) return;
  const long long row = piece / g.ppr;  // n * C + c
  const int j = (int)(piece - row * g.ppr);
  const int n = (int)(row / g.C), c = (int)(row - (long long)n * g.C);
  const int grp = c / g.D;
  const float rs = rstd_in[(size_t)n * g.G + grp];
  const float nmr = -mean_in[(size_t)n * g.G + grp] * rs;
  const float ga = load_param<T>(gamma, c), be = load_param<T>(beta, c);
  const long long v0 = (long long)j * g.piece_vecs;
  const long long v1 = min(g.row_vecs, v0 + g.piece_vecs);
  const T* xs = x + row * g.R;
  const T* ds = dy + row * g.R;
  float s1 = 0.f, s2 = 0.f, t1 = 0.f, t2 = 0.f;  // even and odd lanes
  auto one = [&](const float (&fx)[VE], const float (&fd)[VE]) {
    float xh[VE], yh[VE], gr[VE];
    normalise<VE>(fx, rs, nmr, ga, be, xh, yh);
    act_grad_vec<T, VE, ACT>(yh, gr);
    if constexpr (VE % 2 == 0) {
#pragma unroll
      for (int e = 0; e < VE; e += 2) {
        float d0, d1;
        mul2(d0, d1, fd[e], fd[e + 1], gr[e], gr[e + 1]);
        add2(s1, t1, s1, t1, d0, d1);
        fma2(s2, t2, d0, d1, xh[e], xh[e + 1], s2, t2);
      }
    } else {
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        const float dyh = fd[e] * gr[e];
        s1 += dyh;
        s2 = fmaf(dyh, xh[e], s2);
      }
    }
  };
  long long v = v0 + lane;
  for (; v + (kUnroll - 1) * 32 < v1; v += kUnroll * 32) {
    if constexpr (sizeof(T) * VE == 16) {  // packed while in flight
      uint4 wx[kUnroll], wd[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        wx[u] = ldg128(xs + (v + u * 32) * VE);
        wd[u] = ldg128(ds + (v + u * 32) * VE);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        float fx[VE], fd[VE];
        unpack16<T, VE>(wx[u], fx);
        unpack16<T, VE>(wd[u], fd);
        one(fx, fd);
      }
    } else {
      float fx[kUnroll][VE], fd[kUnroll][VE];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        load_vec<T, VE>(xs + (v + u * 32) * VE, fx[u]);
        load_vec<T, VE>(ds + (v + u * 32) * VE, fd[u]);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) one(fx[u], fd[u]);
    }
  }
#pragma unroll 1
  for (; v < v1; v += 32) {
    float fx[VE], fd[VE];
    load_vec<T, VE>(xs + v * VE, fx);
    load_vec<T, VE>(ds + v * VE, fd);
    one(fx, fd);
  }
  s1 += t1;
  s2 += t2;
#pragma unroll
  for (int b = 16; b >= 1; b >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, b);
    s2 += __shfl_xor_sync(0xffffffffu, s2, b);
  }
  if (lane == 0) tp[piece] = make_float2(s1, s2);
}

// backward 2: one CTA per (n, g): channel sums over the pieces (a lane per piece, then the butterfly)
// -> sums[n * C + c], and the gamma-weighted group sums -> coef[(n * G + g) * 2] = A, B.  With one sample the channel
// sums are the parameter gradients, which are then stored here (dparam_f32 given): the kernel between this one and the dx
// kernel was 2 us of waiting in a chain of four (512 x 256^2 fp16 training step 106.8 -> 105.25 us).
template <typename T>
__global__ void __launch_bounds__(128)
    gn_nchw_finalize_kernel(const float2* __restrict__ tp, const T* __restrict__ gamma, float2* __restrict__ sums,
                            float* __restrict__ coef, float* __restrict__ dparam_f32, T* __restrict__ dgamma,
                            T* __restrict__ dbeta, const NchwGeom g) {
  __shared__ float scratch[4];
  grid_dep_launch_dependents();
  grid_dep_wait();  // the reduce kernel's sums
  const int n = blockIdx.x / g.G, grp = blockIdx.x - n * g.G;
  // W lanes per channel, W the smallest power of two that covers the pieces (at most a warp)
  int sh = 0;
  while ((1 << sh) < g.ppr && sh < 5) ++sh;
  const int W = 1 << sh, lx = threadIdx.x & (W - 1), per_cta = 128 >> sh;
  float w1 = 0.f, w2 = 0.f;  // gamma-weighted sums, held by the first lane of every W
  for (int c0 = 0; c0 < g.D; c0 += per_cta) {
    const int cl = c0 + ((int)threadIdx.x >> sh), c = grp * g.D + cl;
    float t1 = 0.f, t2 = 0.f;
    if (cl < g.D) {
      const float2* p = tp + ((size_t)n * g.C + c) * g.ppr;
#pragma unroll 4
      for (int j = lx; j < g.ppr; j += W) {
        const float2 v = p[j];
        t1 += v.x;
        t2 += v.y;
      }
    }
    for (int b = W >> 1; b >= 1; b >>= 1) {
      t1 += __shfl_xor_sync(0xffffffffu, t1, b);
      t2 += __shfl_xor_sync(0xffffffffu, t2, b);
    }
    if (cl < g.D && lx == 0) {
      if (dparam_f32) {
        dparam_f32[c] = t2;
        dparam_f32[g.C + c] = t1;
        if (dgamma) dgamma[c] = store_param<T>(t2);
        if (dbeta) dbeta[c] = store_param<T>(t1);
      } else {
        sums[(size_t)n * g.C + c] = make_float2(t1, t2);
      }
      const float ga = load_param<T>(gamma, c);
      w1 = fmaf(ga, t1, w1);
      w2 = fmaf(ga, t2, w2);
    }
  }
  w1 = block_sum(w1, scratch);
  w2 = block_sum(w2, scratch);
  if (threadIdx.x == 0) {
    const float inv_m = 1.0f / ((float)g.D * (float)g.R);
    coef[(size_t)blockIdx.x * 2] = w1 * inv_m;
    coef[(size_t)blockIdx.x * 2 + 1] = w2 * inv_m;
  }
}

// backward 4: dx = rstd * (gamma_c * dyh - A - xh * B), one warp per piece as in the reduce kernel, the pieces in
// reverse order and from their ends (see forward 2)
template <typename T, int VE, int ACT>
__global__ void __launch_bounds__(kThreads, 4)
    gn_nchw_dx_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                      const T* __restrict__ beta, const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                      const float* __restrict__ coef, T* __restrict__ dx, long long pieces, const NchwGeom g) {
  const int lane = threadIdx.x & 31;
  const long long piece = pieces - 1 - ((long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5));
  if (piece < 0) return;
  const long long row = piece / g.ppr;
  const int j = (int)(piece - row * g.ppr);
  const int n = (int)(row / g.C), c = (int)(row - (long long)n * g.C);
  const int grp = c / g.D;
  const float rs = rstd_in[(size_t)n * g.G + grp];
  const float nmr = -mean_in[(size_t)n * g.G + grp] * rs;
  const float ga = load_param<T>(gamma, c), be = load_param<T>(beta, c);
  const float ag = rs * ga;
  grid_dep_wait();  // the finalize kernel's coefficients (everything above is the caller's)
  const float nb = -rs * coef[((size_t)n * g.G + grp) * 2 + 1];
  const float na = -rs * coef[((size_t)n * g.G + grp) * 2];
  const long long v0 = (long long)j * g.piece_vecs;
  const long long v1 = min(g.row_vecs, v0 + g.piece_vecs);
  const T* xs = x + row * g.R;
  const T* ds = dy + row * g.R;
  T* os = dx + row * g.R;
  // x and dy are read-only, so the compiler may move the first loads in front of the wait above: then the CTAs that are
  // placed early read their rows while the reduce kernel still streams its own through L2.  With at least four CTAs per SM (three
  // without the bound) it measured, us, loads in front / behind / behind and four CTAs: 64 x 256@64^2 bf16 136 / 127 / 123,
  // 512@256^2 fp16 75 / 70 / 68, 8 x 256@64^2 bf16 22.3 / 22.0 / 21.3; five CTAs: 123 / 68.8 / 23.0 and spills in fp32.
  asm volatile("" : "+l"(xs), "+l"(ds));
  auto one = [&](T* out, const float (&fx)[VE], const float (&fd)[VE]) {
    float xh[VE], yh[VE], gr[VE], o[VE];
    normalise<VE>(fx, rs, nmr, ga, be, xh, yh);
    act_grad_vec<T, VE, ACT>(yh, gr);
    if constexpr (VE % 2 == 0) {
#pragma unroll
      for (int e = 0; e < VE; e += 2) {
        float d0, d1;
        mul2(d0, d1, fd[e], fd[e + 1], gr[e], gr[e + 1]);
        fma2(xh[e], xh[e + 1], nb, nb, xh[e], xh[e + 1], na, na);
        fma2(o[e], o[e + 1], ag, ag, d0, d1, xh[e], xh[e + 1]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < VE; ++e) o[e] = fmaf(ag, fd[e] * gr[e], fmaf(nb, xh[e], na));
    }
    store_vec<T, VE>(out, o, g.evict);
  };
  constexpr int kStep = 32 * VE;
  long long v = v1 - 1 - lane;
  for (; v - (kUnroll - 1) * 32 >= v0; v -= kUnroll * 32) {
    const T *px = xs + v * VE, *pd = ds + v * VE;
    T* po = os + v * VE;
    if constexpr (sizeof(T) * VE == 16) {  // packed while in flight
      uint4 wx[kUnroll], wd[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        wx[u] = ldg128(px - u * kStep);
        wd[u] = ldg128(pd - u * kStep);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        float fx[VE], fd[VE];
        unpack16<T, VE>(wx[u], fx);
        unpack16<T, VE>(wd[u], fd);
        one(po - u * kStep, fx, fd);
      }
    } else {
      float fx[kUnroll][VE], fd[kUnroll][VE];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        load_vec<T, VE>(px - u * kStep, fx[u]);
        load_vec<T, VE>(pd - u * kStep, fd[u]);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) one(po - u * kStep, fx[u], fd[u]);
    }
  }
  for (; v >= v0; v -= 32) {
    float fx[VE], fd[VE];
    load_vec<T, VE>(xs + v * VE, fx);
    load_vec<T, VE>(ds + v * VE, fd);
    one(os + v * VE, fx, fd);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
constexpr int kSmCount = 148;

// n / d for 0 <= n < 2^31 (same construction as the NHWC planner's)
FastDiv fast_div(long long d) {
  FastDiv f;
  if (d < 1) d = 1;
  uint32_t s = 0;
  while ((1ull << s) < (unsigned long long)d) ++s;
  f.mul = (uint32_t)(((1ull << 32) * ((1ull << s) - (unsigned long long)d)) / (unsigned long long)d + 1);
  f.shr = s;
  return f;
}

NchwGeom make_geom(long long N, long long R, long long C, long long G, int ve) {
  NchwGeom g = {};
  g.N = (int)N, g.C = (int)C, g.G = (int)G, g.D = (int)(C / G), g.R = R;
  g.slab_vecs = (long long)g.D * R / ve;
  g.row_vecs = R / ve;
  g.div_R = fast_div(R);
  g.evict = (double)N * C * R * (16 / ve) > 32.0 * 1024 * 1024;  // (single elements are stored plainly)
  // forward: sixteen chunks per SM, at least 2048 vectors (32 KB) each, or 4096 single elements where that still gives every
  // SM a chunk (3 x 40@17x33 fp32, 24 slabs of 2805: 5.8 us in two chunks each, 7.1 in one).  Several waves of CTAs
  // even out the SMs and let the reverse order of the output pass work across CTAs too: with four chunks per SM (all in
  // flight at once) 39.3 us at 512@256^2 fp16, 90 us at 2 x 256@256^2 fp32, 113 us at 3 x 128@300x301 bf16; with sixteen
  // 36.1, 75.9, 76.2.  What does not fill a batch of kUnroll vectors per thread goes vector by vector, so chunks are whole
  // batches where that saves steps (2 x 32@300x200 fp32 18.1 -> 15.5, 64 x 64@112^2 bf16 with chunks of 1568 vectors 61.9
  // -> 56.8, 4 x 512@33^2 12.3 -> 10.9 and with 4096 elements 10.5, 16 x 1024@14^2 18.4 -> 16.7 and 14.7) and of equal
  // length elsewhere (640@32^2: twice 1280 vectors 5.8, 2048 and 512 6.1).
  const long long slabs = N * G, fwd_batch = kUnroll * kThreads;
  const long long min_chunk = ve == 1 && slabs * ((g.slab_vecs + 4095) / 4096) >= kSmCount ? 4096 : 2048;
  long long chunks = (16LL * kSmCount + slabs - 1) / slabs;
  const long long max_chunks = (g.slab_vecs + min_chunk - 1) / min_chunk;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  if (chunks > 1024) chunks = 1024;
  g.chunk_vecs = (g.slab_vecs + chunks - 1) / chunks;
  const long long steps = g.chunk_vecs / fwd_batch + (g.chunk_vecs % fwd_batch + kThreads - 1) / kThreads;
  const long long batches = (g.chunk_vecs + fwd_batch - 1) / fwd_batch;
  if (batches < steps) g.chunk_vecs = batches * fwd_batch;
  g.chunks = (int)((g.slab_vecs + g.chunk_vecs - 1) / g.chunk_vecs);
  // backward: one warp per piece of a channel row; about 96 warps per SM for the same reason (512@256^2 fp16 93 us with
  // 16, 71.9 with 64, 70.8 with 96, 71.6 with 128: 320 CTAs of the first kind lie three on some SMs and two on the others;
  // 2 x 256@256^2 fp32 133 / 127 / 120 / 124), up to 2048 vectors per piece and at least 128, or 256 where that still makes 28
  // warps per SM: a piece of 128 is one batch of loads and nothing to hide them behind (8 x 256@64^2 bf16 22.5 / 21.3,
  // 8 x 256@48^2 17.8 / 16.8, but 4 x 320@96^2, 1280 rows, 28.4 / 32.3).  Of single elements such a batch is a few hundred
  // bytes, and 16 warps per SM of the longer pieces do (320@63^2 13.5 / 11.5, 640@31^2 9.9 / 9.2; not 128@33x31 7.7 / 9.1).
  const long long rows = N * C, bwd_batch = kUnroll * 32, twice = 2 * bwd_batch;
  const bool longer = rows >= 2048 || (ve == 1 && rows * ((g.row_vecs + twice - 1) / twice) >= 16 * kSmCount);
  const long long min_piece = longer ? twice : bwd_batch;
  long long ppr = (96LL * kSmCount + rows - 1) / rows;
  const long long max_ppr = (g.row_vecs + min_piece - 1) / min_piece;
  if (ppr > max_ppr) ppr = max_ppr;
  if (ppr < 1) ppr = 1;
  // as few pieces as whole batches of that length make, of equal length (8 x 256@64^2 fp32: four of 256 37.1, seven of 160
  // 41.7; 512@256^2 fp16: 22 of 384 68.9, 26 of 320 70.8)
  long long piece = ((g.row_vecs + ppr - 1) / ppr + bwd_batch - 1) / bwd_batch * bwd_batch;
  ppr = (g.row_vecs + piece - 1) / piece;
  piece = (g.row_vecs + ppr - 1) / ppr;
  if (piece > 2048) piece = 2048;
  piece = (piece + 31) / 32 * 32;
  g.piece_vecs = piece;
  g.ppr = (int)((g.row_vecs + piece - 1) / piece);
  return g;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

struct BwdScratch {
  size_t tp, sums, coef, total;
};
BwdScratch bwd_scratch(const NchwGeom& g) {
  BwdScratch s;
  s.tp = 0;
  s.sums = (size_t)g.N * g.C * g.ppr * sizeof(float2);
  s.coef = s.sums + (size_t)g.N * g.C * sizeof(float2);
  s.total = (s.coef + (size_t)g.N * g.G * 2 * sizeof(float) + 15) & ~(size_t)15;
  return s;
}

template <typename T, int VE, int ACT>
cudaError_t fwd_t(const FwdCall& c, const NchwGeom& g, cudaStream_t stream) {
  float4* part = static_cast<float4*>(c.workspace);
  const unsigned grid = (unsigned)((long long)g.N * g.G * g.chunks);
  gn_nchw_stats_kernel<T, VE><<<grid, kThreads, 0, stream>>>((const T*)c.x, part, g);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  return launch_chained(gn_nchw_apply_kernel<T, VE, ACT>, grid, dim3(kThreads), 0, stream, chain_enabled(), (const T*)c.x,
                        (const T*)c.gamma, (const T*)c.beta, part, (T*)c.y, c.mean, c.rstd, c.eps, g);
}

template <typename T, int VE, int ACT>
cudaError_t bwd_t(const BwdCall& c, const NchwGeom& g, cudaStream_t stream) {
  const BwdScratch s = bwd_scratch(g);
  char* ws = static_cast<char*>(c.workspace);
  float2* tp = reinterpret_cast<float2*>(ws + s.tp);
  float2* sums = reinterpret_cast<float2*>(ws + s.sums);
  float* coef = reinterpret_cast<float*>(ws + s.coef);
  const long long pieces = (long long)g.N * g.C * g.ppr;
  const unsigned grid = (unsigned)((pieces + kThreads / 32 - 1) / (kThreads / 32));
  gn_nchw_reduce_kernel<T, VE, ACT><<<grid, kThreads, 0, stream>>>((const T*)c.dy, (const T*)c.x, (const T*)c.gamma,
                                                                   (const T*)c.beta, c.mean, c.rstd, tp, pieces, g);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const bool chain = chain_enabled();
  const bool one = g.N == 1;
  err = launch_chained(gn_nchw_finalize_kernel<T>, (unsigned)(g.N * g.G), dim3(128), 0, stream, chain, tp, (const T*)c.gamma,
                       sums, coef, one ? c.dparam_f32 : nullptr, one ? (T*)c.dgamma : nullptr, one ? (T*)c.dbeta : nullptr, g);
  if (err != cudaSuccess) return err;
  if (!one) err = launch_param_grads(c, reinterpret_cast<const float*>(sums), g.N, g.C, stream, chain);
  if (err != cudaSuccess) return err;
  return launch_chained(gn_nchw_dx_kernel<T, VE, ACT>, grid, dim3(kThreads), 0, stream, chain, (const T*)c.dy, (const T*)c.x,
                        (const T*)c.gamma, (const T*)c.beta, c.mean, c.rstd, coef, (T*)c.dx, pieces, g);
}

template <typename T, int VE>
cudaError_t fwd_act(const FwdCall& c, const NchwGeom& g, cudaStream_t stream) {
  switch (c.act) {
    case kActIdentity: return fwd_t<T, VE, kActIdentity>(c, g, stream);
    case kActRelu: return fwd_t<T, VE, kActRelu>(c, g, stream);
    case kActSilu: return fwd_t<T, VE, kActSilu>(c, g, stream);
    case kActGelu: return fwd_t<T, VE, kActGelu>(c, g, stream);
    default: return fwd_t<T, VE, kActGeluTanh>(c, g, stream);
  }
}
template <typename T, int VE>
cudaError_t bwd_act(const BwdCall& c, const NchwGeom& g, cudaStream_t stream) {
  switch (c.act) {
    case kActIdentity: return bwd_t<T, VE, kActIdentity>(c, g, stream);
    case kActRelu: return bwd_t<T, VE, kActRelu>(c, g, stream);
    case kActSilu: return bwd_t<T, VE, kActSilu>(c, g, stream);
    case kActGelu: return bwd_t<T, VE, kActGelu>(c, g, stream);
    default: return bwd_t<T, VE, kActGeluTanh>(c, g, stream);
  }
}

int vector_width(long long R, int dtype, bool aligned) {
  const int vfull = dtype == 0 ? 4 : 8;
  return (aligned && R % vfull == 0) ? vfull : 1;
}

}  // namespace

bool nchw_shape_supported(int64_t N, int64_t R, int64_t C, int64_t G) {
  if (N < 1 || R < 1 || C < 1 || G < 1 || C % G != 0) return false;
  if (R > 0x7fffffffLL || C > (1 << 24) || N * G > 0x7fffffffLL || N * C > 0x7fffffffLL) return false;
  if ((C / G) * R > 0x7fffffffLL) return false;  // offsets inside a slab are 32-bit
  return (double)N * (double)R * (double)C <= 9.0e15;
}

size_t nchw_workspace_bytes(int64_t N, int64_t R, int64_t C, int64_t G, int dtype, int direction) {
  if (!nchw_shape_supported(N, R, C, G)) return 0;
  size_t best = 0;
  for (int aligned = 0; aligned < 2; ++aligned) {
    const NchwGeom g = make_geom(N, R, C, G, vector_width(R, dtype, aligned != 0));
    const size_t need = direction == 0 ? (((size_t)g.N * g.G * g.chunks * sizeof(float4) + 15) & ~(size_t)15)
                                       : bwd_scratch(g).total;
    if (need > best) best = need;
  }
  return best;
}

cudaError_t launch_forward_nchw(const FwdCall& c, int64_t N, int64_t R, int64_t C, int64_t G, cudaStream_t stream) {
  const bool al = aligned16(c.x) && aligned16(c.y);
  const int ve = vector_width(R, c.dtype, al);
  const NchwGeom g = make_geom(N, R, C, G, ve);
  switch (c.dtype) {
    case 0: return ve == 1 ? fwd_act<float, 1>(c, g, stream) : fwd_act<float, 4>(c, g, stream);
    case 1: return ve == 1 ? fwd_act<__half, 1>(c, g, stream) : fwd_act<__half, 8>(c, g, stream);
    default: return ve == 1 ? fwd_act<__nv_bfloat16, 1>(c, g, stream) : fwd_act<__nv_bfloat16, 8>(c, g, stream);
  }
}

cudaError_t launch_backward_nchw(const BwdCall& c, int64_t N, int64_t R, int64_t C, int64_t G, cudaStream_t stream) {
  const bool al = aligned16(c.x) && aligned16(c.dy) && aligned16(c.dx);
  const int ve = vector_width(R, c.dtype, al);
  const NchwGeom g = make_geom(N, R, C, G, ve);
  switch (c.dtype) {
    case 0: return ve == 1 ? bwd_act<float, 1>(c, g, stream) : bwd_act<float, 4>(c, g, stream);
    case 1: return ve == 1 ? bwd_act<__half, 1>(c, g, stream) : bwd_act<__half, 8>(c, g, stream);
    default: return ve == 1 ? bwd_act<__nv_bfloat16, 1>(c, g, stream) : bwd_act<__nv_bfloat16, 8>(c, g, stream);
  }
}

}  // namespace gnb200
