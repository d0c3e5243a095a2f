// Fused sampling for the rollout engine: temperature, optional top-k / top-p,
// inverse-CDF sampling from one uniform per row, and the log-probability of the
// drawn token under the temperature-scaled (unfiltered) distribution, which is
// what the trainer later compares with its own recomputed logprob.
//
// One CTA per row of fp32 logits [B, V]; each warp owns a contiguous segment and reads it in coalesced 16-byte vectors.
//
//   1. One pass from HBM: maximum, its place, and the sum of exponentials, online in registers.
//   2. Without a filter: one pass over the row (now in L2) gives the mass of each segment; the owner of the target
//      walks its segment to the token.
//   3. With a filter: both thresholds are bounded from below by what pass 1 knows. Tokens below log((1 - p) Z / V) hold at
//      most (1 - p) Z together, so the top-p set lies above; the k-th largest of the threads' maxima is no larger than
//      the k-th largest logit. One pass collects the tokens above the bound, for a trained model a few dozen to a few thousand,
//      and the thresholds and the token are found among those in shared memory. Their masses are added in fixed point, so
//      that the order in which they were collected does not matter.
//   4. A row with more candidates than fit (flat distributions): the threshold comes from histograms of the row, each narrowing
//      the range a thousandfold, and the token as in 2.
//
// Bound by the read of the logits. Before, every thread walked a contiguous chunk of its own (uncoalesced), and each filter
// took 26 passes of a bisection over the whole row: 128 rows of 151936 took 964 us with top-p, now 64 us (the read alone: 12 us).
//
// Stands in for the sampler of the external inference server the reference
// drives (areal/engine/sglang_remote.py:43-127 sampling_params, return_logprob).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common/host_utils.h"

namespace b200 {

constexpr int kSampThreads = 512;
constexpr int kSampWarps = kSampThreads / 32;
constexpr int kSampCand = 4096;           // candidates that fit into shared memory, 8 per thread
constexpr int kSampOwn = kSampCand / kSampThreads;
constexpr int kSampBins = 1024;
constexpr float kSampFloor = -60.f;       // a filter never keeps what is less likely than e^-60 of the likeliest token
constexpr float kSampResolution = 1e-6f;  // to which a threshold (a logarithm) is found

using u64 = unsigned long long;

struct SampSmem {
  union {
    struct {
      float y[kSampCand];
      int idx[kSampCand];
    } cand;
    u64 bins[kSampBins];
    float maxima[kSampThreads];
  };
  u64 part[2][kSampWarps][2];
  float fpart[kSampWarps];
  int ipart[kSampWarps];
  int n;
  int pick;
  float bound;
  float range[2];
  u64 above;
};

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <class T>
__device__ __forceinline__ T warp_add(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide reductions, the result in every thread; in a fixed order.
__device__ __forceinline__ float block_max(float v, float* sm) {
  v = warp_max(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sm[0];
#pragma unroll
  for (int w = 1; w < kSampWarps; ++w) r = fmaxf(r, sm[w]);
  return r;
}
__device__ __forceinline__ float block_add(float v, float* sm) {
  v = warp_add(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
#pragma unroll
  for (int w = 0; w < kSampWarps; ++w) r += sm[w];
  return r;
}

// Sums of two counters; `turn` alternates between calls, so that one barrier is enough.
__device__ __forceinline__ void block_add2(u64& a, u64& b, SampSmem& s, int turn) {
  a = warp_add(a);
  b = warp_add(b);
  if ((threadIdx.x & 31) == 0) {
    s.part[turn & 1][threadIdx.x >> 5][0] = a;
    s.part[turn & 1][threadIdx.x >> 5][1] = b;
  }
  __syncthreads();
  a = b = 0;
#pragma unroll
  for (int w = 0; w < kSampWarps; ++w) {
    a += s.part[turn & 1][w][0];
    b += s.part[turn & 1][w][1];
  }
}

// A row, and this warp's segment of it.
template <bool VEC>
struct SampRow {
  const float* x;
  int V, begin, end;  // segment: multiples of 128 except for the end of the row

  __device__ __forceinline__ SampRow(const float* row, int V_) : x(row), V(V_) {
    const int seg = (V / (kSampWarps * 128) + 1) * 128;
    begin = min(V, static_cast<int>(threadIdx.x >> 5) * seg);
    end = min(V, begin + seg);
  }
  // elements i .. i + 3; -inf past the end
  __device__ __forceinline__ float4 load(int i) const {
    if (VEC && i + 3 < end) return *reinterpret_cast<const float4*>(x + i);
    float4 v;
    v.x = i < end ? x[i] : -INFINITY;
    v.y = i + 1 < end ? x[i + 1] : -INFINITY;
    v.z = i + 2 < end ? x[i + 2] : -INFINITY;
    v.w = i + 3 < end ? x[i + 3] : -INFINITY;
    return v;
  }
  // f(first index, four elements) over the segment, U vectors loaded ahead
  template <int U, class F>
  __device__ __forceinline__ void each(F&& f) const {
    const int lane = threadIdx.x & 31;
    for (int c = begin; c < end; c += U * 128) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = load(c + u * 128 + lane * 4);
#pragma unroll
      for (int u = 0; u < U; ++u) f(c + u * 128 + lane * 4, v[u]);
    }
  }
};

// Largest t in [lo, hi] (to kSampResolution) for which the row's tokens with y >= t weigh at least `need`: counts, or masses
// in fixed point. Histograms of what is left of the range.
template <bool VEC>
__device__ float histogram_threshold(const SampRow<VEC>& row, float inv_t, float M, float lo, bool mass, float unit,
                                     u64 need, SampSmem& s) {
  if (threadIdx.x == 0) {
    s.range[0] = lo;
    s.range[1] = 0.f;
    s.above = 0;
  }
  __syncthreads();
  while (true) {
    const float a = s.range[0], b = s.range[1], scale = kSampBins / (b - a);
    const bool top = b == 0.f;  // the first range includes its upper end
    const u64 above = s.above;
    if (b - a <= kSampResolution) return a;
    __syncthreads();
    for (int i = threadIdx.x; i < kSampBins; i += kSampThreads) s.bins[i] = 0;
    __syncthreads();
    row.template each<2>([&](int, float4 v) {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y = e[j] * inv_t - M;
        if (y >= a && (top || y < b)) {
          const int bin = min(kSampBins - 1, static_cast<int>((y - a) * scale));
          atomicAdd(&s.bins[bin], mass ? static_cast<u64>(__expf(y) * unit) : 1ull);
        }
      }
    });
    __syncthreads();
    if (threadIdx.x < 32) {
      // the highest bin at which the weight is reached: 32 bins a lane, then the lane's own
      const int lane = threadIdx.x;
      u64 mine = 0;
      for (int i = 0; i < kSampBins / 32; ++i) mine += s.bins[lane * (kSampBins / 32) + i];
      u64 sum = mine;  // of this lane and those above
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u64 t = __shfl_down_sync(0xffffffffu, sum, o);
        if (lane + o < 32) sum += t;
      }
      const unsigned reached = __ballot_sync(0xffffffffu, above + sum >= need);
      if (lane == (reached ? 31 - __clz(reached) : 0)) {
        u64 w = above + (sum - mine);
        int k = (lane + 1) * (kSampBins / 32) - 1;
        for (; k > lane * (kSampBins / 32) && w + s.bins[k] < need; --k) w += s.bins[k];
        const float width = (b - a) / kSampBins, nlo = a + k * width;
        s.range[0] = nlo;
        s.range[1] = k == kSampBins - 1 ? b : nlo + width;
        s.above = w;
      }
    }
    __syncthreads();
  }
}

// uniforms: [B] in (0,1). temperature <= 0 means greedy. top_k <= 0 or >= V
// disables top-k; top_p >= 1 disables top-p.
template <bool VEC>
__global__ void __launch_bounds__(kSampThreads, 2)
sample_kernel(const float* __restrict__ logits, long long ld, int V,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ uniforms,
              int* __restrict__ tokens, float* __restrict__ logprobs) {
  __shared__ SampSmem s;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SampRow<VEC> row(logits + static_cast<long long>(b) * ld, V);
  const float* x = row.x;
  const float temp = temperature[b];
  const bool greedy = !(temp > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / temp;

  // ---- pass 1: maximum, the first vector that holds it, sum of exponentials (relative to the thread's maximum)
  float mx = -INFINITY, se = 0.f;
  int at = 0;
  row.template each<8>([&](int i, float4 v) {
    const float a0 = v.x * inv_t, a1 = v.y * inv_t, a2 = v.z * inv_t, a3 = v.w * inv_t;
    const float m4 = fmaxf(fmaxf(a0, a1), fmaxf(a2, a3));  // NaN loses
    if (m4 > mx) {
      se = mx == -INFINITY ? se : se * __expf(mx - m4);
      mx = m4;
      at = i;
    }
    // nothing but -inf so far weighs nothing (and NaN still shows)
    const float m = mx == -INFINITY ? 0.f : mx;
    se += (__expf(a0 - m) + __expf(a1 - m)) + (__expf(a2 - m) + __expf(a3 - m));
  });
  const float M = block_max(mx, s.fpart);
  const float Z = block_add(mx == -INFINITY ? se : se * __expf(mx - M), s.fpart);
  const float logZ = logf(Z);  // of the shifted logits: near the maximum nothing cancels
  // the first index of the maximum: a thread's vectors come in rising order, the block's minimum decides
  int best = 0x7fffffff;
  if (mx == M && mx > -INFINITY)
    for (int j = 3; j >= 0; --j)
      if (at + j < V && x[at + j] * inv_t == mx) best = at + j;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
  if (lane == 0) s.ipart[warp] = best;
  if (tid == 0) {
    s.n = 0;
    s.pick = -1;
  }
  __syncthreads();
  best = s.ipart[0];
#pragma unroll
  for (int w = 1; w < kSampWarps; ++w) best = min(best, s.ipart[w]);
  if (best >= V) best = 0;  // a row without any maximum (all NaN): the NaN log-probability tells
  if (greedy) {
    if (tid == 0) {
      tokens[b] = best;
      logprobs[b] = (x[best] * inv_t - M) - logZ;
    }
    return;
  }

  // ---- thresholds, in the shifted domain y = x / T - M <= 0: keep y >= thr
  const int k = top_k ? top_k[b] : 0;
  const float p_in = top_p ? top_p[b] : 1.f, p = fmaxf(p_in, 0.f);
  const bool by_k = k > 0 && k < V, by_p = p_in < 1.f;
  float thr = -INFINITY;
  bool picked = false;
  if (by_k || by_p) {
    const float unit = exp2f(static_cast<float>(61 - (32 - __clz(V))));  // fixed point of a mass of 1; V of them stay below 2^62
    float cut = kSampFloor;
    if (by_p) {
      const float c = logf((1.f - p) * Z / V) - 1e-3f;  // a margin for the rounding of Z
      if (c > cut) cut = c;  // a NaN leaves the floor
    }
    if (by_k && k <= kSampThreads) {
      // rank of every thread's maximum
      s.maxima[tid] = mx;
      __syncthreads();
      int rank = 0;
      for (int j = 0; j < kSampThreads; j += 4) {
        const float4 o = *reinterpret_cast<const float4*>(&s.maxima[j]);
        rank += (o.x > mx || (o.x == mx && j < tid)) + (o.y > mx || (o.y == mx && j + 1 < tid)) +
                (o.z > mx || (o.z == mx && j + 2 < tid)) + (o.w > mx || (o.w == mx && j + 3 < tid));
      }
      if (rank == k - 1) s.bound = mx - M;
      __syncthreads();
      const float c = s.bound;
      if (c > cut) cut = c;
      __syncthreads();
    }
    const bool finite = Z < INFINITY;  // false for NaN
    if (finite) {
      // ---- pass 2: tokens above the bound
      row.template each<8>([&](int i, float4 v) {
        const float y[4] = {v.x * inv_t - M, v.y * inv_t - M, v.z * inv_t - M, v.w * inv_t - M};
        if (fmaxf(fmaxf(y[0], y[1]), fmaxf(y[2], y[3])) >= cut) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (y[j] >= cut) {
              const int o = atomicAdd(&s.n, 1);
              if (o < kSampCand) {
                s.cand.y[o] = y[j];
                s.cand.idx[o] = i + j;
              }
            }
        }
      });
      __syncthreads();
    }
    const int n = s.n;
    const u64 need = finite && by_p ? static_cast<u64>(static_cast<double>(p) * Z * unit) : 0;
    if (finite && n <= kSampCand) {
      float y[kSampOwn];
      int idx[kSampOwn];
      u64 w[kSampOwn];
#pragma unroll
      for (int j = 0; j < kSampOwn; ++j) {
        const int o = tid + j * kSampThreads;
        y[j] = o < n ? s.cand.y[o] : -INFINITY;
        idx[j] = o < n ? s.cand.idx[o] : 0x7fffffff;
        w[j] = o < n ? static_cast<u64>(__expf(y[j]) * unit) : 0;
      }
      // both thresholds at once by bisection: counts and masses of what lies above
      float klo = cut, khi = 0.f, plo = cut, phi = 0.f;
      int turn = 0;
      while (fmaxf(khi - klo, phi - plo) > kSampResolution && turn < 28) {
        const float km = 0.5f * (klo + khi), pm = 0.5f * (plo + phi);
        u64 c = 0, m = 0;
#pragma unroll
        for (int j = 0; j < kSampOwn; ++j) {
          c += y[j] >= km;
          m += y[j] >= pm ? w[j] : 0;
        }
        block_add2(c, m, s, turn++);
        if (c >= static_cast<u64>(k)) klo = km; else khi = km;
        if (m >= need) plo = pm; else phi = pm;
      }
      thr = fmaxf(by_k ? klo : cut, by_p ? plo : cut);
      // the token: in vocabulary order the first at which the mass passes the target
      u64 total = 0, none = 0;
#pragma unroll
      for (int j = 0; j < kSampOwn; ++j) {
        w[j] = y[j] >= thr ? w[j] : 0;
        total += w[j];
      }
      block_add2(total, none, s, turn++);
      const u64 target = static_cast<u64>(static_cast<double>(uniforms[b]) * static_cast<double>(total));
      int lo = 0, hi = V;  // the answer is in [lo, hi); hi: even the whole mass does not pass
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        u64 m = 0, last = 0;
#pragma unroll
        for (int j = 0; j < kSampOwn; ++j) m += idx[j] <= mid ? w[j] : 0;
        block_add2(m, last, s, turn++);
        if (m > target) hi = mid; else lo = mid + 1;
      }
      if (tid == 0) s.pick = lo < V ? lo : -1;
      picked = true;
    } else {
      if (!finite) {
        thr = kSampFloor;
      } else {
        thr = cut;
        if (by_k) thr = fmaxf(thr, histogram_threshold(row, inv_t, M, cut, false, unit, static_cast<u64>(k), s));
        if (by_p) thr = fmaxf(thr, histogram_threshold(row, inv_t, M, cut, true, unit, need, s));
      }
    }
  }

  if (!picked) {
    // ---- masses of the segments over the kept set, then the owner of the target walks to the token
    float cm = 0.f;
    row.template each<8>([&](int, float4 v) {
      const float y[4] = {v.x * inv_t - M, v.y * inv_t - M, v.z * inv_t - M, v.w * inv_t - M};
#pragma unroll
      for (int j = 0; j < 4; ++j) cm += y[j] >= thr ? __expf(y[j]) : 0.f;
    });
    cm = warp_add(cm);
    __syncthreads();
    if (lane == 0) s.fpart[warp] = cm;
    __syncthreads();
    float total = 0.f, before = 0.f;
#pragma unroll
    for (int w = 0; w < kSampWarps; ++w) {
      if (w == warp) before = total;
      total += s.fpart[w];
    }
    const float target = uniforms[b] * total;
    const float after = before + cm;
    if (cm > 0.f && before <= target && target < after) {  // one warp, as the sums rise in the same order everywhere
      float run = before;
      int pick = -1, last_kept = -1;
      constexpr int U = 4;
      for (int c = row.begin; c < row.end && pick < 0; c += U * 128) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = row.load(c + u * 128 + lane * 4);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
          float m[4], mine = 0.f;
          int kept = -1;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float y = e[j] * inv_t - M;
            m[j] = y >= thr && c + u * 128 + lane * 4 + j < row.end ? __expf(y) : 0.f;
            if (m[j] > 0.f) kept = c + u * 128 + lane * 4 + j;
            mine += m[j];
          }
          float scan = mine;  // inclusive over the lanes
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, scan, o);
            if (lane >= o) scan += t;
          }
          const unsigned hit = __ballot_sync(0xffffffffu, mine > 0.f && run + scan > target);
          if (pick < 0 && hit) {
            const int owner = __ffs(hit) - 1;
            float r = run + (scan - mine);
            int mypick = kept;
            for (int j = 0; j < 4; ++j) {
              r += m[j];
              if (m[j] > 0.f && r > target) {
                mypick = c + u * 128 + lane * 4 + j;
                break;
              }
            }
            pick = __shfl_sync(0xffffffffu, mypick, owner);
          }
          const int top = __reduce_max_sync(0xffffffffu, kept);
          if (top >= 0) last_kept = top;
          run += __shfl_sync(0xffffffffu, scan, 31);
        }
      }
      if (pick < 0) pick = last_kept;
      if (lane == 0) s.pick = pick;
    }
  }
  __syncthreads();
  if (tid == 0) {
    // numerical corner (target == total): the most likely token
    const int pick = s.pick >= 0 ? s.pick : best;
    tokens[b] = pick;
    logprobs[b] = (x[pick] * inv_t - M) - logZ;
  }
}

}  // namespace b200

extern "C" {

int b200_sample(const float* logits, long long ld, int B, int V, const float* temperature,
                const int* top_k, const float* top_p, const float* uniforms, int* tokens,
                float* logprobs, cudaStream_t stream) {
  if (B == 0) return 0;
  const bool vec = !(ld & 3) && !(reinterpret_cast<uintptr_t>(logits) & 15);
  auto kernel = vec ? b200::sample_kernel<true> : b200::sample_kernel<false>;
  kernel<<<B, b200::kSampThreads, 0, stream>>>(logits, ld, V, temperature, top_k, top_p, uniforms, tokens, logprobs);
  B200_CHECK(cudaGetLastError());
  return 0;
}

}  // extern "C"
