// "Resident" launch plan for slabs that do not fit a thread-block cluster: forward and backward GroupNorm (+activation)
// for NHWC tensors as ONE persistent cooperative kernel each, one CTA per SM, sm_100a.
//
// The statistics (backward: the sums of dyh and dyh * xh) need every row of a sample before the first result can be
// written, so these shapes take two passes over their rows.  What bounds them is HBM: how much of the second pass is
// read from there again, and what lies between the passes.  Here a CTA owns one contiguous range of a sample's rows:
//
//   pass 1   the range streams through a ring of shared-memory stages (untiled cp.async.bulk copies: whole rows are
//            one contiguous run, so no thread computes an address and no tensor map is needed); the last `stages`
//            tiles are not overwritten, and the eight before them are parked in tensor memory as they pass through:
//            148 x (192 + 256) KB, 67 MB, stay on chip
//   barrier  partial sums to scratch, one arrival per CTA, bounded wait; every CTA merges what it needs
//   pass 2   the resident tiles first - no read at all; those in the stages before those in tensor memory, so that the
//            stages fill again early - and then the tiles before them in reverse order, so that what was read last (and
//            L2 still holds) is read first; results leave with streaming (evict-first) stores
//
// Tensor memory and evict-first marks (Stream::issue) have their rules, with the figures on either side, in gn_plan.cu; the parameters
// are asked for before the ring's first copies and all groups reduced at once because the tensors rest meanwhile (gn_reduce.cuh).
//
// dgamma / dbeta are added up at the end by the grid's warps, without a launch of their own.
// Measured against the plans it replaces: see the rule in gn_plan.cu.
//
// Every sum is formed in an order fixed by the launch geometry: bit-identical reruns.
// The passes restate what src/gnnhwc/csrc/gn_kernel.cu:132-412 and 533-872 of the reference compute.
#include "gn_async.cuh"
#include "gn_kernels.h"
#include "gn_math.cuh"
#include "gn_reduce.cuh"

namespace gnb200 {

namespace {

constexpr int kMaxStages = 16;
constexpr int kMergeLoads = 5;   // channel-sum rows a lane has in flight in the dgamma / dbeta sums

// A thread's sums run over at most this many rows before they are merged into the totals: its whole range is
// R / 148 / TY rows - 111 at 256@512^2, 3543 at 128@4096^2 - where the multi-kernel plan has 55 to 128 per tile, and
// the rounding of the shifted sums grows with n^1.5.  rstd against fp64 with one pixel far from the rest (fp16),
// multi-kernel plan / whole range / pieces of 128 / of 32: 256@512^2 5e-6 / 1.9e-5 / 1.9e-5 / 2e-6, 128@1024^2 1.5e-5 /
// 6.6e-5 / 2.2e-5 / 3e-6, 128 x 2^23 rows 1.3e-5 / 9e-4 / 1.2e-5 / 1.7e-6; the time does not change (337 MB 175 us either way).
constexpr int kFoldRows = 32;

// tests only: this CTA is the one that goes wrong in that way
__device__ __forceinline__ bool test_at(const ResidentGeom& r, int what) {
  return r.test_what == what && (int)blockIdx.x == r.test_cta;
}

// Shared memory: [stages * NT tiles][full][empty][flags][reduction scratch]; NT tensors: x, or x and dy
struct Smem {
  uint32_t stage0;
  uint64_t* full;
  uint64_t* empty;
  int* flags;  // [0] a wait gave up, [1] tensor-memory address
  float* red;
};
template <int NT>
__device__ __forceinline__ Smem carve(const ResidentGeom& r, unsigned char* base) {
  Smem s;
  s.stage0 = smem_addr(base);
  unsigned char* p = base + (size_t)r.stages * NT * r.tile_bytes;  // tile_bytes is a multiple of 16
  s.full = reinterpret_cast<uint64_t*>(p);
  s.empty = s.full + kMaxStages;
  s.flags = reinterpret_cast<int*>(s.empty + kMaxStages);
  s.red = reinterpret_cast<float*>(s.flags + 4);
  return s;
}
constexpr size_t kControlBytes = 2 * kMaxStages * 8 + 16;

// The stage sequence of both passes, as thread 0 (which issues the copies) and all threads walk it.  Tile t
// lives in stage t % stages in both passes; the parity of a barrier's current phase is one bit per stage.
// HOLD: tiles are parked in tensor memory and copies carry the evict-first hint, as the geometry says; otherwise neither.
template <typename T, int NT, bool HOLD>
struct Stream {
  const T* src[NT];  // x (and dy): first element of the CTA's row range
  int tiles, nrows, BR, stages;
  uint32_t row_bytes, tile_bytes;
  uint64_t policy;  // evict-first; made by thread 0 for each of its copies it cost 2 us (128@1024^2 backward 227.7 -> 225.5)
  unsigned full_ph, empty_ph, last_ph;  // last_ph: the phase of each stage's last copy
  Smem sm;

  // `once`: the tile is not read from global memory again
  __device__ __forceinline__ void issue(int t, int stage, bool once) {  // thread 0
    const uint32_t bytes = (uint32_t)min(BR, nrows - t * BR) * row_bytes;
    last_ph ^= 1u << stage;
    mbar_arrive_expect_tx(&sm.full[stage], NT * bytes);
    const uint32_t dst = sm.stage0 + (uint32_t)(stage * NT) * tile_bytes;
    const size_t at = (size_t)t * tile_bytes;
    if (HOLD && once) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
        bulk_load_once(dst + i * tile_bytes, reinterpret_cast<const char*>(src[i]) + at, bytes, &sm.full[stage], policy);
    } else {
#pragma unroll
      for (int i = 0; i < NT; ++i)
        bulk_load(dst + i * tile_bytes, reinterpret_cast<const char*>(src[i]) + at, bytes, &sm.full[stage]);
    }
  }
  // thread 0: waits until every warp has handed the stage back, then refills it.  Without the hand-back
  // (its wait gave up) nothing is copied over a stage that may still be read.
  __device__ __forceinline__ void refill(int t, int stage, bool once, const WaitLimit& lim, bool withhold = false) {
    producer_wait(&sm.empty[stage], (empty_ph >> stage) & 1u, &sm.flags[0], lim);
    empty_ph ^= 1u << stage;
    if (*(volatile int*)&sm.flags[0] == 0 && !withhold) issue(t, stage, once);
  }
  __device__ __forceinline__ bool wait_full(int stage, const WaitLimit& lim) {
    const bool ok = consumer_wait(&sm.full[stage], (full_ph >> stage) & 1u, &sm.flags[0], lim);
    full_ph ^= 1u << stage;
    return ok;
  }
  // A wait that gave up leaves copies behind that nobody waited for: they must not land after the CTA has left.
  __device__ __forceinline__ void drain(const WaitLimit& lim) {  // thread 0
    if (*(volatile int*)&sm.flags[0] == 0) return;
    for (int s = 0; s < stages; ++s)
      if (!mbar_wait_bounded(&sm.full[s], (last_ph >> s) & 1u, lim)) return;
  }

  // Where the tiles of the range are between the passes: [0, held0) must be read again, [held0, held0 + parked) are in
  // tensor memory, the last `stages` of them in the stages.
  int parked, held0;
  uint32_t tmem;  // the thread's first word

  // Pass 2 takes the tiles that pass through the stages as items 0, 1, ...: those held there newest first, then the
  // others in reverse order.  Item i lies in the i-th stage before the last tile's.
  int next, next_stage;  // thread 0: the item to be copied next, and its stage
  __device__ __forceinline__ int items() const { return tiles - parked; }
  __device__ __forceinline__ int tile_of(int item) const { return tiles - 1 - item - (item < stages ? 0 : parked); }
  __device__ __forceinline__ void start_pass2(int last_stage) {
    next = stages;
    next_stage = last_stage;
  }
  // thread 0, once item `done` has been read: the item that takes its stage
  __device__ __forceinline__ void refill_behind(int done, const ResidentGeom& r) {
    if (done + stages < next || next >= items()) return;
    refill(tile_of(next), next_stage, r.evict, r.g.wait, next == stages && test_at(r, kDebugNoSecondCopy));
    ++next;
    next_stage = next_stage == 0 ? stages - 1 : next_stage - 1;
  }
};

template <typename T, int NT, bool HOLD>
__device__ __forceinline__ void stream_start(Stream<T, NT, HOLD>& st, const ResidentGeom& r, const Smem& sm, int nrows) {
  st.sm = sm;
  st.nrows = nrows;
  st.BR = r.BR;
  st.stages = r.stages;
  st.tiles = (nrows + r.BR - 1) / r.BR;
  st.row_bytes = (uint32_t)(r.g.C * (int)sizeof(T));
  st.tile_bytes = (uint32_t)r.tile_bytes;
  st.full_ph = st.empty_ph = 0;
  st.last_ph = ~0u;
  if constexpr (HOLD) st.policy = evict_first_policy();
  st.parked = HOLD ? max(0, min(r.park, st.tiles - r.stages)) : 0;
  st.held0 = max(0, st.tiles - r.stages - st.parked);
  const int alloc_warp = 1 % (int)(blockDim.x >> 5);  // not the one that issues the copies, where there is another
  if (HOLD && st.parked && (int)(threadIdx.x >> 5) == alloc_warp) tmem_alloc(reinterpret_cast<uint32_t*>(&sm.flags[1]));
  if (threadIdx.x == 0) {
    for (int s = 0; s < r.stages; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], blockDim.x >> 5);
    }
    sm.flags[0] = 0;
    fence_mbar_init_cluster();
    for (int t = test_at(r, kDebugNoFirstCopy) ? 1 : 0; t < min(r.stages, st.tiles); ++t) st.issue(t, t, r.evict && t >= st.held0);
  }
  __syncwarp();
  __syncthreads();
  st.tmem = st.parked ? tmem_own(*(volatile uint32_t*)&sm.flags[1], threadIdx.x >> 5) : 0u;
}
template <typename T, int NT, bool HOLD>
__device__ __forceinline__ void stream_end(Stream<T, NT, HOLD>& st, const WaitLimit& lim) {
  if (threadIdx.x == 0) st.drain(lim);
  if (!HOLD || !st.parked) return;
  __syncwarp();
  __syncthreads();
  if ((int)(threadIdx.x >> 5) == 1 % (int)(blockDim.x >> 5)) tmem_free(*(volatile uint32_t*)&st.sm.flags[1]);
}

// Grid barrier: every CTA has written its partial sums.  `count` starts at 0 (cleared in stream order before the
// launch); its low half counts the CTAs, its high half those whose partial sums are worthless, because a copy they
// needed did not arrive in time.  In every CTA that learns of one, or that gives up waiting here, flags[0] is set
// afterwards; the caller then writes NaN.
__device__ __forceinline__ void grid_barrier(unsigned int* count, int* flags, const ResidentGeom& r) {
  const WaitLimit& lim = r.g.wait;
  __syncwarp();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (!test_at(r, kDebugNoArrival)) atomicAdd(count, *(volatile int*)flags == 0 ? 1u : 0x10001u);
    const long long t0 = clock64();
    unsigned int polls = 0, seen;
    while (((seen = ld_acquire_u32(count)) & 0xffffu) < gridDim.x) {
      if (++polls > lim.polls && clock64() - t0 > lim.clocks) {
        wait_gave_up(lim);
        flags[0] = 1;
        break;
      }
    }
    if (seen >> 16) flags[0] = 1;
    __threadfence();
  }
  __syncthreads();
}

// The thread's rows among the first `rows` of the CTA's range, whose values are not known: all bits set is a NaN in
// every element type.  `first` is the thread's first row.
__device__ __forceinline__ void store_nan_rows(void* first, size_t row_bytes, int my_row, int TY, int rows) {
  for (int i = my_row; i < rows; i += TY)
    stg128_stream(static_cast<char*>(first) + (size_t)(i - my_row) * row_bytes, make_uint4(~0u, ~0u, ~0u, ~0u));
}

// ------------------------------------------------------------------------------------------------
// forward.  scratch: part[cta * G + s] = (mean, M2) of group s over the CTA's rows
// ------------------------------------------------------------------------------------------------
template <typename T, int ACT, bool UNI>
__global__ void __launch_bounds__(kResidentThreads, 1)
    gn_fwd_resident_kernel(const T* __restrict__ x, const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y,
                           float* __restrict__ mean_out, float* __restrict__ rstd_out, float eps, float2* part,
                           unsigned int* count, const ResidentGeom r) {
  constexpr int VE = 16 / sizeof(T);
  constexpr int KR = resident_rows(0);
  constexpr bool kShifted = sizeof(T) == 2;  // 16-bit tensors: shifted sums about the thread's first row
  constexpr int KN = UNI ? 1 : VE;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const Geom& g = r.g;
  const Smem sm = carve<1>(r, smem_raw);
  float* red = sm.red;
  float* slot = red + g.red_floats;
  float* stat = slot + g.slots;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)blockDim.x >> 5;
  const int n = g.div_chunks.div((int)blockIdx.x), j = (int)blockIdx.x - n * r.cps;
  const int r0 = j * g.rows_per_cta;
  const int nrows = min(g.rows_per_cta, g.R - r0);
  const int ty = g.div_CV.div(tid), tx = tid - ty * g.CV;
  const bool streaming = ty < g.TY;
  const size_t row0 = (size_t)n * g.R + r0;

  Stream<T, 1, true> st;
  st.src[0] = x + row0 * g.C;
  stream_start(st, r, sm, nrows);
  const int T_ = st.tiles, S = st.stages;
  const uint32_t my_off = sm.stage0 + (streaming ? (uint32_t)(ty * g.CV + tx) * 16u : 0u);
  const uint32_t step = (uint32_t)(g.TY * g.CV) * 16u;
  const int my_row = streaming ? ty : 0x40000000;  // no row of a tile for idle threads

  // ---- pass 1: moments of the thread's rows, closed every kFoldRows rows (the shift is the first row of each piece)
  float mean[VE], m2[VE], cnt = 0.f;  // of the closed pieces
#pragma unroll
  for (int e = 0; e < VE; ++e) mean[e] = m2[e] = 0.f;
  int stage = 0, prev = 0;
  for (int t0 = 0; t0 < T_; t0 += kFoldRows / KR) {
    const int t1 = min(T_, t0 + kFoldRows / KR);
    float pm[VE], pq[VE], K[KN], pn = 0.f;
#pragma unroll
    for (int e = 0; e < VE; ++e) pm[e] = pq[e] = 0.f;
#pragma unroll
    for (int e = 0; e < KN; ++e) K[e] = 0.f;
    for (int t = t0; t < t1; ++t) {
      st.wait_full(stage, g.wait);
      const uint32_t base = my_off + (uint32_t)stage * st.tile_bytes;
      const int here = nrows - t * st.BR;
      uint4 w[KR];
#pragma unroll
      for (int u = 0; u < KR; ++u) w[u] = lds128(base + u * step);
      if (t >= st.held0 && t < T_ - S) tmem_store16(st.tmem + (t - st.held0) * 16, w[0], w[1], w[2], w[3]);
      if constexpr (kShifted) {
        if (t == t0) {
          float f0[VE];
          unpack16<T, VE>(w[0], f0);
          if (my_row < here) {
#pragma unroll
            for (int e = 0; e < KN; ++e) K[e] = f0[e];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < KR; ++u) {
        if (my_row + u * g.TY < here) {
          if constexpr (kShifted) {
            shifted_step<T, VE, KN>(w[u], K, pm, pq);
          } else {
            float f[VE];
            unpack16<T, VE>(w[u], f);
            welford_step<VE>(f, pm, pq, pn);
          }
        }
      }
      pin_regs(pm);
      pin_regs(pq);
      if (t + S < T_) release_stage(&sm.empty[stage], lane);
      if (tid == 0 && t >= 1 && t - 1 + S < T_) st.refill(t - 1 + S, prev, r.evict && t - 1 + S >= st.held0, g.wait);
      prev = stage;
      if (++stage == S) stage = 0;
    }
    if constexpr (kShifted) {
      const int left = min(nrows - t0 * st.BR, (t1 - t0) * st.BR);
      shifted_finish<VE, KN>(K, my_row < left ? (left - my_row + g.TY - 1) / g.TY : 0, pm, pq, pn);
    }
    merge_moments<VE>(pm, pq, pn, mean, m2, cnt);
  }
  const Crew cr = {tid, (int)blockDim.x, lane, warp, nwarps, 0};
  crew_moments<VE, UNI>(cr, g, g.G, mean, m2, cnt, tx, ty, nrows, red, slot,
                        [&](int s, float mu, float q) { part[(size_t)blockIdx.x * g.G + s] = make_float2(mu, q); });
  uint4 ga_raw = make_uint4(0, 0, 0, 0), be_raw = ga_raw;
  if (streaming) {  // (they arrive during the wait)
    ga_raw = ldg128(gamma + tx * VE);
    be_raw = ldg128(beta + tx * VE);
  }
  if (st.parked) tmem_store_wait();  // also where the barrier gives up and pass 2 is left out: stream_end frees the words
  grid_barrier(count, sm.flags, r);

  // ---- statistics of the sample: sums about the first CTA's mean, the counts known from the geometry
  const bool ok = *(volatile int*)&sm.flags[0] == 0;
  {
    const float2* p = part + (size_t)n * r.cps * g.G;
    float* acc = red;  // [2][nwarps][G]
    merge_rows(p, r.cps, g.G, warp, nwarps, lane, acc, [&](int i, float2 v, float K0, float& a1, float& a2) {
      const float cnt_i = (float)min(g.rows_per_cta, g.R - i * g.rows_per_cta) * (float)g.D, d = v.x - K0;
      a1 = fmaf(cnt_i, d, a1);
      a2 += fmaf(cnt_i * d, d, v.y);
    });
    __syncthreads();
    for (int s = tid; s < g.G; s += blockDim.x) {
      float ad = 0.f, aq = 0.f;
      for (int w = 0; w < nwarps; ++w) {
        ad += acc[w * g.G + s];
        aq += acc[(nwarps + w) * g.G + s];
      }
      const float an = (float)g.R * (float)g.D, K0 = __ldcg(p + s).x, dm = ad / an;
      const float mu = ok ? K0 + dm : kNaN;
      const float rs = ok ? rsqrtf(fmaxf(fmaf(-ad, dm, aq) / an, 0.f) + eps) : kNaN;
      stat[s] = mu;
      stat[g.slots + s] = rs;
      if (j == 0) {
        mean_out[(size_t)n * g.G + s] = mu;
        rstd_out[(size_t)n * g.G + s] = rs;
      }
    }
  }
  __syncthreads();

  // ---- pass 2: y = act(x * a + b), the resident tiles first
  float a[VE], b[VE];
#pragma unroll
  for (int e = 0; e < VE; ++e) a[e] = b[e] = 0.f;
  if (streaming) lane_affine_raw<T, VE, UNI>(ga_raw, be_raw, stat, stat + g.slots, 0, tx * VE, g.div_D, a, b);
  T* out = y + (row0 + (streaming ? ty : 0)) * g.C + (streaming ? tx * VE : 0);
  const size_t ostep = (size_t)g.TY * g.C;
  // one tile's vectors of the thread, wherever they were kept
  auto emit = [&](int t, const uint4 (&w)[KR]) {
    const int here = nrows - t * st.BR;
    T* o = out + (size_t)t * st.BR * g.C;
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      if (my_row + u * g.TY < here) {
        float f[VE];
        unpack16<T, VE>(w[u], f);
        affine<VE>(f, a, b);
        stg128_stream(o + (size_t)u * ostep, act_pack16<T, VE, ACT>(f));
      }
    }
  };
  stage = prev;  // of the last tile
  st.start_pass2(stage);
  int lost = ok ? -1 : T_ - 1;  // the rows of the tiles up to this one are not known
  for (int i = 0; ok; ++i) {
    if (i == S && st.parked) {  // the stages fill again meanwhile
      for (int p = st.parked - 1; p >= 0; --p) {
        uint4 w[KR];
        tmem_load16(st.tmem + p * 16, w[0], w[1], w[2], w[3]);
        emit(st.held0 + p, w);
        if (tid == 0) st.refill_behind(S - 1, r);
      }
    }
    if (i >= st.items()) break;
    const int t = st.tile_of(i);
    if (i >= S && !st.wait_full(stage, g.wait)) {
      lost = t;
      break;
    }
    const uint32_t base = my_off + (uint32_t)stage * st.tile_bytes;
    uint4 w[KR];
#pragma unroll
    for (int u = 0; u < KR; ++u) w[u] = lds128(base + u * step);
    emit(t, w);
    if (i + S < st.items()) release_stage(&sm.empty[stage], lane);
    if (tid == 0 && i > 0) st.refill_behind(i - 1, r);
    stage = stage == 0 ? S - 1 : stage - 1;
  }
  store_nan_rows(out, (size_t)g.C * sizeof(T), my_row, g.TY, min(nrows, (lost + 1) * st.BR));  // none, unless a wait gave up
  stream_end(st, g.wait);
}

// ------------------------------------------------------------------------------------------------
// backward.  scratch: tpart[cta * C + c] = (S1, S2) of channel c over the CTA's rows,
//          gpart[cta * G + s] = gamma-weighted sums of group s over the CTA's rows.
// ------------------------------------------------------------------------------------------------
template <typename T, int ACT, bool UNI, bool HOLD>
__global__ void __launch_bounds__(kResidentThreads, 1)
    gn_bwd_resident_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                           const T* __restrict__ beta, const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                           T* __restrict__ dx, float2* tpart, float2* gpart, unsigned int* count,
                           float* __restrict__ dparam_f32, T* __restrict__ dgamma, T* __restrict__ dbeta,
                           const ResidentGeom r) {
  constexpr int VE = 16 / sizeof(T);
  constexpr int KR = resident_rows(1);
  // 16-bit tensors: packed arithmetic, S2 against the raw x.  Packed fp32 pairs only where a vector has one rstd and one mean: with
  // eight of each the registers are short (128@1024^2: 229.0 us with them, 227.7 without)
  constexpr bool kRaw = sizeof(T) == 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const Geom& g = r.g;
  const Smem sm = carve<2>(r, smem_raw);
  float* red = sm.red;
  float* chan = red + g.red_floats;  // S1[C], S2[C]
  float* gam = chan + 2 * g.C;       // gamma[C]
  float* coef = gam + g.C;           // A[G], B[G]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)blockDim.x >> 5;
  const int n = g.div_chunks.div((int)blockIdx.x), j = (int)blockIdx.x - n * r.cps;
  const int r0 = j * g.rows_per_cta;
  const int nrows = min(g.rows_per_cta, g.R - r0);
  const int ty = g.div_CV.div(tid), tx = tid - ty * g.CV;
  const bool streaming = ty < g.TY;
  const size_t row0 = (size_t)n * g.R + r0;

  // what the caller gave is asked for before the ring's copies: behind 28 MB of them it would arrive 3 us later
  LaneParams<T, VE, UNI> lp;
  if (streaming) lp.load(gamma, beta, mean_in + (size_t)n * g.G, rstd_in + (size_t)n * g.G, tx * VE, g.div_D);
  Stream<T, 2, HOLD> st;
  st.src[0] = x + row0 * g.C;
  st.src[1] = dy + row0 * g.C;
  stream_start(st, r, sm, nrows);
  const int T_ = st.tiles, S = st.stages;
  const uint32_t my_off = sm.stage0 + (streaming ? (uint32_t)(ty * g.CV + tx) * 16u : 0u);
  const uint32_t step = (uint32_t)(g.TY * g.CV) * 16u;
  const int my_row = streaming ? ty : 0x40000000;

  BwdLane<T, VE> L;
  float a[VE], b[VE];
#pragma unroll
  for (int e = 0; e < VE; ++e) L.r[e] = L.nmr[e] = L.ga[e] = L.be[e] = 0.f;
  if (streaming) {
    lp.unpack(L);
    if (ty == 0) {
#pragma unroll
      for (int e = 0; e < VE; ++e) gam[tx * VE + e] = L.ga[e];
    }
  }
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    a[e] = L.r[e] * L.ga[e];
    b[e] = fmaf(L.nmr[e], L.ga[e], L.be[e]);
  }

  // ---- pass 1: S1, S2 over the thread's rows, closed every kFoldRows rows
  float s1[VE], s2[VE];  // of the closed pieces
#pragma unroll
  for (int e = 0; e < VE; ++e) s1[e] = s2[e] = 0.f;
  int stage = 0, prev = 0;
  for (int t0 = 0; t0 < T_; t0 += kFoldRows / KR) {
    const int t1 = min(T_, t0 + kFoldRows / KR);
    float p1[VE], p2[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) p1[e] = p2[e] = 0.f;
    for (int t = t0; t < t1; ++t) {
      st.wait_full(stage, g.wait);
      const uint32_t base = my_off + (uint32_t)(2 * stage) * st.tile_bytes;
      const int here = nrows - t * st.BR;
      uint4 xw[KR], dw[KR];
#pragma unroll
      for (int u = 0; u < KR; ++u) {
        xw[u] = lds128(base + u * step);
        dw[u] = lds128(base + st.tile_bytes + u * step);
      }
      if (HOLD && t >= st.held0 && t < T_ - S) tmem_store16(st.tmem + (t - st.held0) * 16, xw[0], xw[1], dw[0], dw[1]);
#pragma unroll
      for (int u = 0; u < KR; ++u) {
        if (my_row + u * g.TY < here) {
          if constexpr (kRaw) {
            bwd_row_sums_packed<T, ACT, UNI && kPairs<T>>(xw[u], dw[u], a, b, p1, p2);
          } else {
            float fx[VE], fd[VE];
            unpack16<T, VE>(xw[u], fx);
            unpack16<T, VE>(dw[u], fd);
            bwd_row_sums<T, VE, ACT>(fx, fd, L, p1, p2);
          }
        }
      }
      pin_regs(p1);
      pin_regs(p2);
      if (t + S < T_) release_stage(&sm.empty[stage], lane);
      if (tid == 0 && t >= 1 && t - 1 + S < T_) st.refill(t - 1 + S, prev, r.evict && t - 1 + S >= st.held0, g.wait);
      prev = stage;
      if (++stage == S) stage = 0;
    }
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      s1[e] += p1[e];
      // packed: S2 = sum dyh * xh = rstd * (sum dyh * x - mean * sum dyh)
      s2[e] += kRaw ? fmaf(L.r[e], p2[e], L.nmr[e] * p1[e]) : p2[e];
    }
  }
  const Crew cr = {tid, (int)blockDim.x, lane, warp, nwarps, 0};
  crew_channel_sums<VE>(cr, g, s1, tx, ty, red, chan);
  cr.sync();
  crew_channel_sums<VE>(cr, g, s2, tx, ty, red, chan + g.C);
  cr.sync();
  crew_group_sums(cr, g, gam, chan,
                  [&](int s, float w1, float w2) { gpart[(size_t)blockIdx.x * g.G + s] = make_float2(w1, w2); });
  for (int c = tid; c < g.C; c += blockDim.x) tpart[(size_t)blockIdx.x * g.C + c] = make_float2(chan[c], chan[g.C + c]);
  if (HOLD && st.parked) tmem_store_wait();  // also where the barrier gives up and pass 2 is left out: stream_end frees the words
  grid_barrier(count, sm.flags, r);

  // ---- A, B of the sample's groups
  const bool ok = *(volatile int*)&sm.flags[0] == 0;
  const float inv_m = ok ? 1.0f / ((float)g.D * (float)g.R) : kNaN;
  {
    float* acc = red;  // [2][nwarps][G]
    merge_rows(gpart + (size_t)n * r.cps * g.G, r.cps, g.G, warp, nwarps, lane, acc,
               [](int, float2 v, float, float& a1, float& a2) { a1 += v.x, a2 += v.y; });
    __syncthreads();
    for (int s = tid; s < g.G; s += blockDim.x) {
      float w1 = 0.f, w2 = 0.f;
      for (int w = 0; w < nwarps; ++w) {
        w1 += acc[w * g.G + s];
        w2 += acc[(nwarps + w) * g.G + s];
      }
      coef[s] = w1 * inv_m;
      coef[g.G + s] = w2 * inv_m;
    }
  }
  __syncthreads();

  // ---- pass 2: dx = ag dyh - r (A + xh B), with xh = r x + nmr:  c1 x + c2 (16-bit) or c1 xh + c2 (fp32)
  float c1[VE], c2[VE];
#pragma unroll
  for (int e = 0; e < VE; ++e) c1[e] = c2[e] = 0.f;
  if (streaming) {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const int s = g.div_D.div(tx * VE + (UNI ? 0 : e));
      const float nb = -L.r[e] * coef[g.G + s], na = -L.r[e] * coef[s];
      c1[e] = kRaw ? nb * L.r[e] : nb;
      c2[e] = kRaw ? fmaf(nb, L.nmr[e], na) : na;
    }
  }
  T* out = dx + (row0 + (streaming ? ty : 0)) * g.C + (streaming ? tx * VE : 0);
  const size_t ostep = (size_t)g.TY * g.C;
  auto emit = [&](int t, const uint4 (&xw)[KR], const uint4 (&dw)[KR]) {
    const int here = nrows - t * st.BR;
    T* o = out + (size_t)t * st.BR * g.C;
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      if (my_row + u * g.TY < here) {
        if constexpr (kRaw) {
          stg128_stream(o + (size_t)u * ostep, bwd_dx_packed<T, ACT, UNI && kPairs<T>>(xw[u], dw[u], a, b, a, c1, c2));
        } else {
          float fx[VE], fd[VE], xh[VE], yh[VE], gr[VE];
          unpack16<T, VE>(xw[u], fx);
          unpack16<T, VE>(dw[u], fd);
#pragma unroll
          for (int e = 0; e < VE; ++e) {
            xh[e] = fmaf(fx[e], L.r[e], L.nmr[e]);
            yh[e] = fmaf(xh[e], L.ga[e], L.be[e]);
          }
          act_grad_vec<T, VE, ACT>(yh, gr);
#pragma unroll
          for (int e = 0; e < VE; ++e) fx[e] = fmaf(a[e], fd[e] * gr[e], fmaf(c1[e], xh[e], c2[e]));
          stg128_stream(o + (size_t)u * ostep, pack16<T, VE>(fx));
        }
      }
    }
  };
  stage = prev;
  st.start_pass2(stage);
  int lost = ok ? -1 : T_ - 1;
  for (int i = 0; ok; ++i) {
    if (HOLD && i == S && st.parked) {
      for (int p = st.parked - 1; p >= 0; --p) {
        uint4 xw[KR], dw[KR];
        tmem_load16(st.tmem + p * 16, xw[0], xw[1], dw[0], dw[1]);
        emit(st.held0 + p, xw, dw);
        if (tid == 0) st.refill_behind(S - 1, r);
      }
    }
    if (i >= st.items()) break;
    const int t = st.tile_of(i);
    if (i >= S && !st.wait_full(stage, g.wait)) {
      lost = t;
      break;
    }
    const uint32_t base = my_off + (uint32_t)(2 * stage) * st.tile_bytes;
    uint4 xw[KR], dw[KR];
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      xw[u] = lds128(base + u * step);
      dw[u] = lds128(base + st.tile_bytes + u * step);
    }
    emit(t, xw, dw);
    if (i + S < st.items()) release_stage(&sm.empty[stage], lane);
    if (tid == 0 && i > 0) st.refill_behind(i - 1, r);
    stage = stage == 0 ? S - 1 : stage - 1;
  }
  store_nan_rows(out, (size_t)g.C * sizeof(T), my_row, g.TY, min(nrows, (lost + 1) * st.BR));  // none, unless a wait gave up

  // ---- dgamma / dbeta: the grid's warps share the channels; all channel sums are visible since the barrier
  const int rows = g.N * r.cps;
  const bool bad = *(volatile int*)&sm.flags[0] != 0;
  for (int c = (int)blockIdx.x + (int)gridDim.x * warp; c < g.C; c += (int)gridDim.x * nwarps) {
    float t1 = 0.f, t2 = 0.f;
    for (int i0 = lane; i0 < rows + lane; i0 += 32 * kMergeLoads) {
      float2 v[kMergeLoads];
#pragma unroll
      for (int q = 0; q < kMergeLoads; ++q) {
        const int i = i0 + 32 * q;
        v[q] = i < rows ? __ldcg(tpart + (size_t)i * g.C + c) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < kMergeLoads; ++q) t1 += v[q].x, t2 += v[q].y;
    }
    t1 = warp_sum_all(t1);
    t2 = warp_sum_all(t2);
    if (lane == 0) {
      if (bad) t1 = t2 = kNaN;
      dparam_f32[c] = t2;
      dparam_f32[g.C + c] = t1;
      if (dgamma) dgamma[c] = store_param<T>(t2);
      if (dbeta) dbeta[c] = store_param<T>(t1);
    }
  }
  stream_end(st, g.wait);
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
struct Scratch {
  size_t pairs, count, total;  // backward: channel sums first
};
Scratch scratch_of(const ResidentGeom& r, int direction) {
  Scratch s;
  s.pairs = direction == 0 ? 0 : (size_t)r.grid * r.g.C * sizeof(float2);
  s.count = s.pairs + (size_t)r.grid * r.g.G * sizeof(float2);
  s.total = (s.count + 4 + 15) & ~(size_t)15;
  return s;
}

// tests (gnb200_debug_next_resident): what the calling thread's next launch meets
thread_local ResidentDebug t_debug = {};

__global__ void gn_resident_refused_kernel() {}

// What the runtime says to a cooperative grid that cannot be resident: a million CTAs of an empty kernel.
cudaError_t launch_too_large(cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1u << 20, 1, 1);
  cfg.blockDim = dim3(1024, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gn_resident_refused_kernel);
}

template <typename Kern, typename... Args>
cudaError_t launch(Kern kern, const ResidentGeom& r, unsigned int* count, cudaStream_t stream, Args... args) {
  cudaError_t err = ensure_kernel_attributes((const void*)kern, r.smem_bytes, false);
  if (err != cudaSuccess) return err;
  err = check_resident((const void*)kern, r.threads, r.smem_bytes, r.test_what == kDebugRefusedByCheck ? 1LL << 20 : r.grid);
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(count, 0, sizeof(unsigned int), stream);
  if (err != cudaSuccess) return err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)r.grid, 1, 1);
  cfg.blockDim = dim3((unsigned)r.threads, 1, 1);
  cfg.dynamicSmemBytes = r.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  err = r.test_what == kDebugRefusedByRuntime ? launch_too_large(stream) : cudaLaunchKernelEx(&cfg, kern, args...);
  // the runtime notes the refusal as its last error too, which the fall-back plan's launches would report as theirs
  if (err == cudaErrorCooperativeLaunchTooLarge) (void)cudaGetLastError();
  return err;
}

template <typename T, int ACT, bool UNI>
cudaError_t launch_u(const FwdCall& c, const ResidentGeom& r, cudaStream_t stream) {
  const Scratch s = scratch_of(r, 0);
  char* ws = static_cast<char*>(c.workspace);
  unsigned int* count = reinterpret_cast<unsigned int*>(ws + s.count);
  return launch(gn_fwd_resident_kernel<T, ACT, UNI>, r, count, stream, (const T*)c.x, (const T*)c.gamma, (const T*)c.beta,
                (T*)c.y, c.mean, c.rstd, c.eps, reinterpret_cast<float2*>(ws + s.pairs), count, r);
}
template <typename T, int ACT, bool UNI>
cudaError_t launch_u(const BwdCall& c, const ResidentGeom& r, cudaStream_t stream) {
  const Scratch s = scratch_of(r, 1);
  char* ws = static_cast<char*>(c.workspace);
  unsigned int* count = reinterpret_cast<unsigned int*>(ws + s.count);
  // HOLD is a kernel of its own.  Where nothing is parked, because x and dy are beyond what that is good for (gn_plan.cu), the code for it in the
  // loops alone costs issue slots: device us with it / without, 16 bits: 320 x 164062 rows, 105 MB 3 % slower, 1536 x 43619 133.5 / 129.2,
  // 1536 x 130208, 400 MB 4.5 % slower.  Full CTAs of 512 threads hide it, and beyond 165 MB they are the faster ones with it (not understood: 268 MB
  // 256 x 523437 217.5 / 219.7, 400 MB 2.4 %; 105 MB 0.983, 165 MB 1.00, 200 MB 1.012 without / with).
  const bool hold = r.park > 0 || (r.threads == kResidentThreads && (double)r.g.N * r.g.R * r.g.C * sizeof(T) > 165e6);
  const auto kern = hold ? gn_bwd_resident_kernel<T, ACT, UNI, true> : gn_bwd_resident_kernel<T, ACT, UNI, false>;
  return launch(kern, r, count, stream, (const T*)c.dy, (const T*)c.x, (const T*)c.gamma,
                (const T*)c.beta, c.mean, c.rstd, (T*)c.dx, reinterpret_cast<float2*>(ws),
                reinterpret_cast<float2*>(ws + s.pairs), count, c.dparam_f32, (T*)c.dgamma, (T*)c.dbeta, r);
}
template <typename T, int ACT, typename Call>
cudaError_t launch_t(const Call& c, const ResidentGeom& r, cudaStream_t stream) {
  constexpr int VE = 16 / sizeof(T);
  return r.g.D % VE == 0 ? launch_u<T, ACT, true>(c, r, stream) : launch_u<T, ACT, false>(c, r, stream);
}
template <typename T, typename Call>
cudaError_t launch_act(const Call& c, const ResidentGeom& r, cudaStream_t stream) {
  switch (c.act) {
    case kActIdentity: return launch_t<T, kActIdentity>(c, r, stream);
    case kActRelu: return launch_t<T, kActRelu>(c, r, stream);
    case kActSilu: return launch_t<T, kActSilu>(c, r, stream);
    case kActGelu: return launch_t<T, kActGelu>(c, r, stream);
    default: return launch_t<T, kActGeluTanh>(c, r, stream);
  }
}
template <typename Call>
cudaError_t launch_resident(const Call& c, ResidentGeom r, cudaStream_t stream) {
  const cudaError_t err = wait_limit_for_device(&r.g.wait);
  if (err != cudaSuccess) return err;
  r.test_what = t_debug.what;
  r.test_cta = t_debug.cta;
  t_debug = ResidentDebug{};
  if (r.test_what >= kDebugNoArrival) r.g.wait.clocks = 2000000, r.g.wait.polls = 256;  // about a millisecond
  switch (c.dtype) {
    case 0: return launch_act<float>(c, r, stream);
    case 1: return launch_act<__half>(c, r, stream);
    default: return launch_act<__nv_bfloat16>(c, r, stream);
  }
}

}  // namespace

void debug_next_resident(const ResidentDebug& d) { t_debug = d; }

size_t resident_workspace_bytes(const ResidentGeom& r, int direction) { return scratch_of(r, direction).total; }

size_t resident_fixed_smem(const ResidentGeom& r, int direction) {
  const Geom& g = r.g;
  const size_t floats = direction == 0 ? 3 * (size_t)g.slots : 3 * (size_t)g.C + 2 * (size_t)g.G;
  return kControlBytes + ((size_t)g.red_floats + floats) * 4 + 16;
}

cudaError_t launch_forward_resident(const FwdCall& c, const ResidentGeom& r, cudaStream_t stream) {
  return launch_resident(c, r, stream);
}
cudaError_t launch_backward_resident(const BwdCall& c, const ResidentGeom& r, cudaStream_t stream) {
  return launch_resident(c, r, stream);
}

}  // namespace gnb200
