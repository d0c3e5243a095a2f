// Memory-bound transformer glue for sm_100a: RMSNorm (+ fused residual add),
// per-head q/k RMSNorm fused with rotary embedding, and SwiGLU, each with its
// backward. All kernels move 16-byte vectors, keep a row in registers between
// the reduction and the write, and accumulate in fp32.
//
// Replaces the eager / Inductor-fused RMSNorm, rotate_half RoPE and SiLU*mul of
// the reference models (areal/experimental/models/archon/qwen3/model/model.py:75-101,
// 103-293; qwen2/model/rope.py).
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "norm_static_scratch.h"
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/host_utils.h"
#include "common/ptx.cuh"
#include "common/rms_row.cuh"
#include "common/sigmoid.cuh"

namespace b200 {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct alignas(16) BF8 {
  __nv_bfloat162 v[4];
};
__device__ __forceinline__ void bf8_to_float(const BF8& b, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(b.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ BF8 float_to_bf8(const float* f) {
  BF8 b;
#pragma unroll
  for (int i = 0; i < 4; ++i) b.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return b;
}

// ------------------------------------------------------------------ RMSNorm --
// A group of threads per row (common/rms_row.cuh), blockDim = (group, groups of the block). Bound by memory: x, the residual
// and both results cross HBM once. With a warp a row and 64 columns a lane, 16384 x 2048 with residual took 64 us (4.2 TB/s);
// spread over 256 threads it takes as long with one row a group, which leaves memory idle between blocks, and 53 us (5.1
// TB/s) with two rows a group, loaded together (four: 53 us). 32768 x 4096: 359 us before, 196 us now.
template <int VPT, int ROWS>
__global__ void __launch_bounds__(512)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd, int T, int H, float eps) {
  __shared__ float part[8][ROWS][kRmsMaxWarps];
  const int tid = threadIdx.x, group = blockDim.x;
  const long long row0 = (static_cast<long long>(blockIdx.x) * blockDim.y + threadIdx.y) * ROWS;
  if (row0 >= T) return;  // the whole group
  const int nvec = H >> 3;
  BF8 h[ROWS][VPT], r[ROWS][VPT];
  float ss[ROWS];
#pragma unroll
  for (int k = 0; k < ROWS; ++k)
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = tid + group * i;
      if (c < nvec && row0 + k < T) {
        h[k][i] = reinterpret_cast<const BF8*>(x + (row0 + k) * H)[c];
        if (res) r[k][i] = reinterpret_cast<const BF8*>(res + (row0 + k) * H)[c];
      }
    }
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    ss[k] = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = tid + group * i;
      if (c < nvec && row0 + k < T) {
        float v[8];
        bf8_to_float(h[k][i], v);
        if (res) {
          float f[8];
          bf8_to_float(r[k][i], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] += f[j];
          // the residual stream is kept in bf16: normalise what is stored
          h[k][i] = float_to_bf8(v);
          reinterpret_cast<BF8*>(res_out + (row0 + k) * H)[c] = h[k][i];
          bf8_to_float(h[k][i], v);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[k] += v[j] * v[j];
      }
    }
  }
  rms_group_sums<ROWS>(ss, &part[threadIdx.y][0][0], tid, group, threadIdx.y);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = tid + group * i;
    if (c < nvec) {
      float f[8];
      bf8_to_float(reinterpret_cast<const BF8*>(w)[c], f);
#pragma unroll
      for (int k = 0; k < ROWS; ++k)
        if (row0 + k < T) {
          const float rs = rsqrtf(ss[k] / H + eps);
          if (tid == 0 && i == 0 && rstd) rstd[row0 + k] = rs;
          float v[8], o[8];
          bf8_to_float(h[k][i], v);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = v[j] * rs * f[j];
          reinterpret_cast<BF8*>(y + (row0 + k) * H)[c] = float_to_bf8(o);
        }
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres); one partial row of dw per block. A thread keeps its columns over all
// rows of its group, so dw accumulates in registers; the next row is loaded before the current one is reduced, so that
// the barrier of the sum does not leave memory idle. 16384 x 2048: 164 us with a warp a row (8 vectors a lane and no
// load ahead), 74 us so (80 when the converted numbers stay in registers across the sum); 32768 x 4096: 1050 us and 283 us.
template <int VPT>
__global__ void __launch_bounds__(512, VPT == 1 ? 2 : 1)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, int T, int H) {
  __shared__ float part[2][8][kRmsMaxWarps];
  extern __shared__ float sm[];  // [rows of the block - 1][H], only with more than one
  const int tid = threadIdx.x, group = blockDim.x, slot = threadIdx.y;
  const int nvec = H >> 3;
  const float inv_h = 1.f / H;
  float dwacc[VPT][8];
  BF8 wv[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = tid + group * i;
    if (c < nvec) wv[i] = reinterpret_cast<const BF8*>(w)[c];
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
  }
  struct Row {
    BF8 g[VPT], x[VPT], r[VPT];
    float rs;
  };
  auto load = [&](long long row, Row& o) {
    if (row >= T) return;
    o.rs = rstd[row];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = tid + group * i;
      if (c < nvec) {
        o.g[i] = reinterpret_cast<const BF8*>(dy + row * H)[c];
        o.x[i] = reinterpret_cast<const BF8*>(x + row * H)[c];
        if (dres) o.r[i] = reinterpret_cast<const BF8*>(dres + row * H)[c];
      }
    }
  };
  const long long step = static_cast<long long>(gridDim.x) * blockDim.y;
  long long row = static_cast<long long>(blockIdx.x) * blockDim.y + slot;
  Row next;
  load(row, next);
  for (int it = 0; row < T; row += step, ++it) {
    const Row cur = next;
    load(row + step, next);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (tid + group * i < nvec) {
        float g[8], xh[8], f[8];
        bf8_to_float(cur.g[i], g);
        bf8_to_float(cur.x[i], xh);
        bf8_to_float(wv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] *= cur.rs;
          dwacc[i][j] += g[j] * xh[j];
          dot += g[j] * f[j] * xh[j];
        }
      }
    }
    dot = rms_group_sum(dot, part[it & 1][slot], tid, group, slot) * inv_h;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = tid + group * i;
      if (c < nvec) {
        float g[8], xh[8], f[8], o[8];
        bf8_to_float(cur.g[i], g);
        bf8_to_float(cur.x[i], xh);
        bf8_to_float(wv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = cur.rs * (g[j] * f[j] - xh[j] * cur.rs * dot);
        if (dres) {
          float r[8];
          bf8_to_float(cur.r[i], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        reinterpret_cast<BF8*>(dx + row * H)[c] = float_to_bf8(o);
      }
    }
  }
  // the block's row groups meet in shared memory
  if (blockDim.y > 1) {
    if (slot) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int c = tid + group * i;
        if (c < nvec)
#pragma unroll
          for (int j = 0; j < 8; ++j) sm[(slot - 1) * H + c * 8 + j] = dwacc[i][j];
      }
    }
    __syncthreads();
  }
  if (slot) return;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = tid + group * i;
    if (c < nvec) {
      for (int s = 1; s < blockDim.y; ++s)
#pragma unroll
        for (int j = 0; j < 8; ++j) dwacc[i][j] += sm[(s - 1) * H + c * 8 + j];
      float4* out = reinterpret_cast<float4*>(dw_partial + static_cast<long long>(blockIdx.x) * H + c * 8);
      out[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
      out[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
    }
  }
}

// Column sums of the partial rows: 32 columns a block, its 16 warps take every 16th row. (With one thread a column
// walking all rows this took 12 us, with these 5 us.)
__global__ void __launch_bounds__(512)
colsum_partials_kernel(const float* __restrict__ partial, float* __restrict__ out, int nblocks, int H,
                       int accumulate) {
  __shared__ float sm[16][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < H)
#pragma unroll 4
    for (int b = warp; b < nblocks; b += 16) s += partial[static_cast<long long>(b) * H + c];
  sm[warp][lane] = s;
  __syncthreads();
  if (warp || c >= H) return;
#pragma unroll
  for (int i = 1; i < 16; ++i) s += sm[i][lane];
  out[c] = accumulate ? out[c] + s : s;
}

// ------------------------------------------------------- q/k norm + RoPE ----
// qkv: [T, (Hq + 2*Hkv) * D] bf16 (q heads, then k heads, then v heads), D == 128. Eight lanes share a head: a lane owns
// columns 8l..8l+7 and their partners 64 + 8l.. (16-byte vectors), so a warp works on four heads of a token at a time,
// the sum of squares takes three shuffles, and the token's angles are read once for all of them. With a warp a head and four columns
// a lane the kernels were bound by issue slots: 16384 tokens of 16 + 8 heads took 91 us forward and 172 us backward, now
// 51 and 119 us (the latter with the copy of dv, which was a launch of its own, and with the next token loaded ahead: 144 without).
constexpr int kRopeD = 128;
constexpr int kRopeHeads = 4;  // heads of a warp at a time

struct RopeVec {  // a lane's columns of one head
  float a[8], b[8];
  __device__ __forceinline__ void read(const __nv_bfloat16* p, int l) {
    bf8_to_float(reinterpret_cast<const BF8*>(p)[l], a);
    bf8_to_float(reinterpret_cast<const BF8*>(p + 64)[l], b);
  }
  __device__ __forceinline__ void write(__nv_bfloat16* p, int l) const {
    reinterpret_cast<BF8*>(p)[l] = float_to_bf8(a);
    reinterpret_cast<BF8*>(p + 64)[l] = float_to_bf8(b);
  }
};

struct RopeAngles {  // a lane's angles of one position
  float c[8], s[8];
  __device__ __forceinline__ void read(const float* __restrict__ cos_t, const float* __restrict__ sin_t, int p, int l) {
    const float4* pc = reinterpret_cast<const float4*>(cos_t + static_cast<long long>(p) * 64) + 2 * l;
    const float4* ps = reinterpret_cast<const float4*>(sin_t + static_cast<long long>(p) * 64) + 2 * l;
    *reinterpret_cast<float4*>(c) = pc[0];
    *reinterpret_cast<float4*>(c + 4) = pc[1];
    *reinterpret_cast<float4*>(s) = ps[0];
    *reinterpret_cast<float4*>(s + 4) = ps[1];
  }
};

__device__ __forceinline__ float rope_sum8(float v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Norm (when w is given) and rotation of one head in place; returns the head's 1 / rms. Every lane of the warp calls.
__device__ __forceinline__ float rope_head(RopeVec& v, const RopeAngles& r, const __nv_bfloat16* w, int l, float eps) {
  float rs = 1.f;
  if (w) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v.a[j] * v.a[j] + v.b[j] * v.b[j];
    rs = rsqrtf(rope_sum8(ss) / kRopeD + eps);
    RopeVec ww;
    ww.read(w, l);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // match the reference's rounding: the normalised value is cast to bf16 before RoPE
      v.a[j] = __bfloat162float(__float2bfloat16(v.a[j] * rs * ww.a[j]));
      v.b[j] = __bfloat162float(__float2bfloat16(v.b[j] * rs * ww.b[j]));
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float a = v.a[j], b = v.b[j];
    v.a[j] = a * r.c[j] - b * r.s[j];
    v.b[j] = b * r.c[j] + a * r.s[j];
  }
  return rs;
}

__global__ void __launch_bounds__(256)
qknorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ qw,
                       const __nv_bfloat16* __restrict__ kw, const float* __restrict__ cos_t,
                       const float* __restrict__ sin_t, const int* __restrict__ pos,
                       __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_out,
                       float* __restrict__ rstd_out, int T, int Hq, int Hkv, float eps, int has_norm) {
  constexpr int D = kRopeD, J = 2;  // a warp takes J rounds of kRopeHeads heads of one token
  const int lane = threadIdx.x & 31, l = lane & 7;
  const int heads = Hq + Hkv;
  const int groups = (heads + J * kRopeHeads - 1) / (J * kRopeHeads);
  const long long gw = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (gw >= static_cast<long long>(T) * groups) return;
  const int t = static_cast<int>(gw / groups);
  const int h0 = static_cast<int>(gw % groups) * J * kRopeHeads + (lane >> 3);
  const __nv_bfloat16* src = qkv + static_cast<long long>(t) * (Hq + 2 * Hkv) * D;
  RopeAngles ang;
  ang.read(cos_t, sin_t, pos[t], l);
  RopeVec v[J];
#pragma unroll
  for (int j = 0; j < J; ++j)  // lanes past the last head repeat it and write nothing
    v[j].read(src + static_cast<long long>(min(h0 + j * kRopeHeads, heads - 1)) * D, l);
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int h = h0 + j * kRopeHeads;
    const bool is_q = h < Hq;
    const float rs = rope_head(v[j], ang, has_norm ? (is_q ? qw : kw) : nullptr, l, eps);
    if (h >= heads) continue;
    if (has_norm && l == 0) rstd_out[static_cast<long long>(t) * heads + h] = rs;
    v[j].write(is_q ? q_out + (static_cast<long long>(t) * Hq + h) * D
                    : k_out + (static_cast<long long>(t) * Hkv + (h - Hq)) * D, l);
  }
}

// Decode / prefill form of the kernel above: q is written out as before, k goes straight into the
// paged K cache and v is copied into the paged V cache (`[page, kv head, slot in page, D]`), so the
// separate cache-write launch disappears. A warp takes four of a token's q, k AND v heads.
// slot_mapping[t] = page * block_size + offset, negative to skip the token's cache write.
__global__ void __launch_bounds__(128)
qknorm_rope_kvwrite_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ qw,
                           const __nv_bfloat16* __restrict__ kw, const float* __restrict__ cos_t,
                           const float* __restrict__ sin_t, const int* __restrict__ pos,
                           __nv_bfloat16* __restrict__ q_out, const long long* __restrict__ slot_mapping,
                           __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, int T,
                           int Hq, int Hkv, int block_size, float eps, int has_norm) {
  constexpr int D = kRopeD;
  const int lane = threadIdx.x & 31, l = lane & 7;
  const int heads = Hq + 2 * Hkv;
  const int groups = (heads + kRopeHeads - 1) / kRopeHeads;
  const long long gw = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (gw >= static_cast<long long>(T) * groups) return;
  const int t = static_cast<int>(gw / groups);
  const int h = static_cast<int>(gw % groups) * kRopeHeads + (lane >> 3);
  const int hs = min(h, heads - 1);
  pdl_wait();
  pdl_trigger();
  const long long slot = slot_mapping[t];
  const __nv_bfloat16* src = qkv + (static_cast<long long>(t) * heads + hs) * D;
  const BF8 raw_a = reinterpret_cast<const BF8*>(src)[l], raw_b = reinterpret_cast<const BF8*>(src + 64)[l];
  RopeAngles ang;
  ang.read(cos_t, sin_t, pos[t], l);
  RopeVec v;
  bf8_to_float(raw_a, v.a);
  bf8_to_float(raw_b, v.b);
  rope_head(v, ang, has_norm ? (hs < Hq ? qw : kw) : nullptr, l, eps);  // the result of a v head is not used
  if (h >= heads) return;
  if (h < Hq) {
    v.write(q_out + (static_cast<long long>(t) * Hq + h) * D, l);
    return;
  }
  if (slot < 0) return;
  const bool is_v = h >= Hq + Hkv;
  const int hk = is_v ? h - Hq - Hkv : h - Hq;
  __nv_bfloat16* dst = (is_v ? v_cache : k_cache) +
                       (((slot / block_size) * Hkv + hk) * block_size + slot % block_size) * D;
  if (is_v) {
    reinterpret_cast<BF8*>(dst)[l] = raw_a;
    reinterpret_cast<BF8*>(dst + 64)[l] = raw_b;
  } else {
    v.write(dst, l);
  }
}

// Backward: un-rotate dq/dk, then per-head RMSNorm backward; writes the q, k and (copied from dv) v slots of dqkv. A warp
// keeps its heads and walks over tokens, so dqw / dkw [D] accumulate in registers and reach memory with one atomic
// per column and block.
__global__ void __launch_bounds__(256)
qknorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                       const __nv_bfloat16* __restrict__ dv, const __nv_bfloat16* __restrict__ qkv,
                       const __nv_bfloat16* __restrict__ qw, const __nv_bfloat16* __restrict__ kw,
                       const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                       const int* __restrict__ pos, const float* __restrict__ rstd,
                       __nv_bfloat16* __restrict__ dqkv, float* __restrict__ dqw, float* __restrict__ dkw,
                       int T, int Hq, int Hkv, int has_norm) {
  constexpr int D = kRopeD;
  __shared__ float s_dw[2][D];
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) (&s_dw[0][0])[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, l = lane & 7;
  const int heads = Hq + Hkv, all = Hq + 2 * Hkv;
  const int groups = (all + kRopeHeads - 1) / kRopeHeads;
  const int gw = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int walkers = static_cast<int>((gridDim.x * blockDim.x) >> 5) / groups;  // warps that share a group of heads
  const int h = (gw % groups) * kRopeHeads + (lane >> 3);
  const bool is_q = h < Hq, is_v = h >= heads;
  const int hs = min(h, all - 1);
  const __nv_bfloat16* g0 = is_q ? dq + static_cast<long long>(h) * D
                                 : !is_v ? dk + static_cast<long long>(h - Hq) * D
                                         : dv + static_cast<long long>(hs - heads) * D;
  const long long gpitch = static_cast<long long>(is_q ? Hq : Hkv) * D;
  RopeVec acc;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc.a[j] = acc.b[j] = 0.f;
  RopeVec ww;
  if (has_norm) ww.read(is_q ? qw : kw, l);
  struct Token {
    BF8 ga, gb, xa, xb;
    float rs;
    int pos;
  };
  auto load = [&](int t, Token& o) {
    if (t >= T) return;
    const __nv_bfloat16* g = g0 + t * gpitch;
    o.ga = reinterpret_cast<const BF8*>(g)[l];
    o.gb = reinterpret_cast<const BF8*>(g + 64)[l];
    o.pos = pos[t];
    o.rs = 0.f;
    if (has_norm) {
      const __nv_bfloat16* xp = qkv + (static_cast<long long>(t) * all + hs) * D;
      o.xa = reinterpret_cast<const BF8*>(xp)[l];
      o.xb = reinterpret_cast<const BF8*>(xp + 64)[l];
      if (!is_v) o.rs = rstd[static_cast<long long>(t) * heads + h];
    }
  };
  Token next;
  if (gw < walkers * groups) {
    load(gw / groups, next);
    for (int t = gw / groups; t < T; t += walkers) {
      const Token cur = next;
      RopeAngles r;
      r.read(cos_t, sin_t, cur.pos, l);
      load(t + walkers, next);  // on its way while this token is worked on
      const BF8 raw_a = cur.ga, raw_b = cur.gb;
      const long long row = static_cast<long long>(t) * all;
      const float rs = cur.rs;
      RopeVec x;
      if (has_norm) {
        bf8_to_float(cur.xa, x.a);
        bf8_to_float(cur.xb, x.b);
      }
      RopeVec d;
      {
        float ga[8], gb[8];
        bf8_to_float(raw_a, ga);
        bf8_to_float(raw_b, gb);
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // transpose of the rotation
          d.a[j] = ga[j] * r.c[j] + gb[j] * r.s[j];
          d.b[j] = gb[j] * r.c[j] - ga[j] * r.s[j];
        }
      }
      if (has_norm) {
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x.a[j] *= rs;
          x.b[j] *= rs;
          acc.a[j] += d.a[j] * x.a[j];
          acc.b[j] += d.b[j] * x.b[j];
          d.a[j] *= ww.a[j];
          d.b[j] *= ww.b[j];
          dot += d.a[j] * x.a[j] + d.b[j] * x.b[j];
        }
        dot = rope_sum8(dot) / D;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          d.a[j] = rs * (d.a[j] - x.a[j] * dot);
          d.b[j] = rs * (d.b[j] - x.b[j] * dot);
        }
      }
      if (h >= all) continue;
      __nv_bfloat16* out = dqkv + (row + h) * D;
      if (is_v) {
        reinterpret_cast<BF8*>(out)[l] = raw_a;
        reinterpret_cast<BF8*>(out + 64)[l] = raw_b;
      } else {
        d.write(out, l);
      }
    }
  }
  if (!has_norm) return;
  if (!is_v) {
    float* sw = s_dw[is_q ? 0 : 1];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      atomicAdd(&sw[8 * l + j], acc.a[j]);
      atomicAdd(&sw[64 + 8 * l + j], acc.b[j]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    if (s_dw[0][i] != 0.f) atomicAdd(&dqw[i], s_dw[0][i]);
    if (s_dw[1][i] != 0.f) atomicAdd(&dkw[i], s_dw[1][i]);
  }
}

// ------------------------------------------------------------------- SwiGLU --
// gu: [T, 2*I] (gate = first I columns, up = last I columns); out: [T, I]. A thread takes the same vector of ROWS rows
// and loads all of them before it computes; rows and columns come from the grid, not from a 64-bit division per vector, and the
// sigmoid is one approximate reciprocal (1 ulp; the exponential before it is no better), because IEEE divisions alone kept
// the issue slots busy for most of the time that the memory needs. Two rows a thread; one is 4% slower, four 30%. 16384 x 6144:
// 129 us forward and 181 us backward before, 96 and 146 us (6.3 and 6.9 TB/s) now.
template <int ROWS>
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, long long T, int I) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= I >> 3) return;
  for (long long t0 = static_cast<long long>(blockIdx.y) * ROWS; t0 < T; t0 += static_cast<long long>(gridDim.y) * ROWS) {
    BF8 g[ROWS], u[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      if (t0 + r < T) {
        g[r] = reinterpret_cast<const BF8*>(gu + (t0 + r) * 2 * I)[c];
        u[r] = reinterpret_cast<const BF8*>(gu + (t0 + r) * 2 * I + I)[c];
      }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      if (t0 + r < T) {
        float fg[8], fu[8], o[8];
        bf8_to_float(g[r], fg);
        bf8_to_float(u[r], fu);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = fg[j] * sigmoid_rcp(fg[j]) * fu[j];
        reinterpret_cast<BF8*>(out + (t0 + r) * I)[c] = float_to_bf8(o);
      }
  }
}
template <int ROWS>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ gu,
                  __nv_bfloat16* __restrict__ dgu, long long T, int I) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= I >> 3) return;
  for (long long t0 = static_cast<long long>(blockIdx.y) * ROWS; t0 < T; t0 += static_cast<long long>(gridDim.y) * ROWS) {
    BF8 g[ROWS], u[ROWS], d[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      if (t0 + r < T) {
        g[r] = reinterpret_cast<const BF8*>(gu + (t0 + r) * 2 * I)[c];
        u[r] = reinterpret_cast<const BF8*>(gu + (t0 + r) * 2 * I + I)[c];
        d[r] = reinterpret_cast<const BF8*>(dy + (t0 + r) * I)[c];
      }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      if (t0 + r < T) {
        float fg[8], fu[8], fd[8], dg[8], du[8];
        bf8_to_float(g[r], fg);
        bf8_to_float(u[r], fu);
        bf8_to_float(d[r], fd);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float sg = sigmoid_rcp(fg[j]);
          const float silu = fg[j] * sg;
          du[j] = fd[j] * silu;
          dg[j] = fd[j] * fu[j] * (sg * (1.f + fg[j] * (1.f - sg)));
        }
        reinterpret_cast<BF8*>(dgu + (t0 + r) * 2 * I)[c] = float_to_bf8(dg);
        reinterpret_cast<BF8*>(dgu + (t0 + r) * 2 * I + I)[c] = float_to_bf8(du);
      }
  }
}

// (columns / 256, rows / ROWS) blocks; the kernels walk on where that is more than a grid holds
static dim3 swiglu_grid(long long T, int I, int rows, int& threads) {
  const int nvec = I >> 3;
  threads = nvec >= 256 ? 256 : (nvec + 31) / 32 * 32;
  const long long y = (T + rows - 1) / rows;
  return dim3((nvec + threads - 1) / threads, static_cast<unsigned>(y < 65535 ? y : 65535));
}

template <class F>
static int rms_dispatch(int H, F&& f) {
  const RmsShape s = rms_shape(H);
  if (s.group > 512) return -101;
  return s.vpt == 1 ? f(std::integral_constant<int, 1>{}, s.group) : f(std::integral_constant<int, 2>{}, s.group);
}

}  // namespace b200

extern "C" {

// H must be a multiple of 8 and at most 8192. res/res_out/rstd may be null.
int b200_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out,
                     float* rstd, int T, int H, float eps, cudaStream_t stream) {
  using namespace b200;
  if (T == 0) return 0;
  if (H % 8) return -100;
  int rc = rms_dispatch(H, [&](auto vpt, int group) {
    const int groups = 256 / group > 1 ? 256 / group : 1;
    constexpr int R = 2;
    rmsnorm_fwd_kernel<decltype(vpt)::value, R><<<(T + groups * R - 1) / (groups * R), dim3(group, groups), 0, stream>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
        (__nv_bfloat16*)y, (__nv_bfloat16*)res_out, rstd, T, H, eps);
    return 0;
  });
  if (rc) return rc;
  B200_CHECK(cudaGetLastError());
  return 0;
}

// dw_partial: scratch of at least b200_rmsnorm_bwd_blocks(T) * H floats.
int b200_rmsnorm_bwd_blocks(int T) {
  int grid = (T + 3) / 4;
  const int maxg = b200::sm_count() * 2;
  return grid > maxg ? maxg : grid;
}
int b200_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                     const void* dres, void* dx, float* dw_partial, float* dw, int dw_accumulate,
                     int T, int H, cudaStream_t stream) {
  using namespace b200;
  if (T == 0) return 0;
  if (H % 8) return -100;
  const int grid = b200_rmsnorm_bwd_blocks(T);
  int rc = rms_dispatch(H, [&](auto vpt, int group) {
    // 512 threads a block, two blocks an SM; at most 8 rows side by side (a named barrier each)
    const int rows = 512 / group > 8 ? 8 : 512 / group;
    rmsnorm_bwd_kernel<decltype(vpt)::value>
        <<<grid, dim3(group, rows), static_cast<size_t>(rows - 1) * H * sizeof(float), stream>>>(
            (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,
            (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dw_partial, T, H);
    return 0;
  });
  if (rc) return rc;
  B200_CHECK(cudaGetLastError());
  colsum_partials_kernel<<<(H + 31) / 32, 512, 0, stream>>>(dw_partial, dw, grid, H, dw_accumulate);
  B200_CHECK(cudaGetLastError());
  return 0;
}

int b200_qknorm_rope_fwd(const void* qkv, const void* qw, const void* kw, const float* cos_t,
                         const float* sin_t, const int* pos, void* q_out, void* k_out,
                         float* rstd, int T, int Hq, int Hkv, int D, float eps, int has_norm,
                         cudaStream_t stream) {
  using namespace b200;
  if (D != 128) return -100;
  if (T == 0) return 0;
  const long long warps = static_cast<long long>(T) * ((Hq + Hkv + 2 * kRopeHeads - 1) / (2 * kRopeHeads));
  const int tpb = 256;
  const long long grid = (warps * 32 + tpb - 1) / tpb;
  qknorm_rope_fwd_kernel<<<(unsigned)grid, tpb, 0, stream>>>(
      (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, cos_t, sin_t,
      pos, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, rstd, T, Hq, Hkv, eps, has_norm);
  B200_CHECK(cudaGetLastError());
  return 0;
}

// q/k norm + RoPE of a fused qkv projection whose k and v go straight into the paged KV caches
// ([num_blocks, Hkv, block_size, 128] bf16) at slot_mapping[t] (int64; negative = skip).
int b200_qknorm_rope_kvwrite(const void* qkv, const void* qw, const void* kw, const float* cos_t,
                             const float* sin_t, const int* pos, void* q_out, const long long* slot_mapping,
                             void* k_cache, void* v_cache, int T, int Hq, int Hkv, int D, int block_size,
                             float eps, int has_norm, int chained, cudaStream_t stream) {
  using namespace b200;
  if (D != 128) return -100;
  if (T == 0) return 0;
  const long long warps = static_cast<long long>(T) * ((Hq + 2 * Hkv + kRopeHeads - 1) / kRopeHeads);
  const int tpb = 128;
  const long long grid = (warps * 32 + tpb - 1) / tpb;
  B200_CHECK(launch_kernel(qknorm_rope_kvwrite_kernel, (unsigned)grid, tpb, 0, stream, chained, (const __nv_bfloat16*)qkv,
                           (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, cos_t, sin_t, pos, (__nv_bfloat16*)q_out,
                           slot_mapping, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, T, Hq, Hkv, block_size, eps,
                           has_norm));
  return 0;
}

// dqw/dkw are fp32 [D] accumulators (added to, not overwritten); dq [T, Hq, D], dk and dv [T, Hkv, D] contiguous.
int b200_qknorm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* qkv, const void* qw,
                         const void* kw, const float* cos_t, const float* sin_t, const int* pos,
                         const float* rstd, void* dqkv, float* dqw, float* dkw, int T, int Hq,
                         int Hkv, int D, int has_norm, cudaStream_t stream) {
  using namespace b200;
  if (D != 128) return -100;
  if (T == 0) return 0;
  const int groups = (Hq + 2 * Hkv + kRopeHeads - 1) / kRopeHeads;
  const long long warps = static_cast<long long>(T) * groups;
  const int tpb = 256;
  // three blocks an SM are resident; every group of heads needs a warp of its own
  long long grid = (warps * 32 + tpb - 1) / tpb;
  const long long least = (groups * 32 + tpb - 1) / tpb, most = static_cast<long long>(sm_count()) * 3;
  if (grid > most) grid = most;
  if (grid < least) grid = least;
  qknorm_rope_bwd_kernel<<<(unsigned)grid, tpb, 0, stream>>>(
      (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)qkv,
      (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, cos_t, sin_t, pos, rstd,
      (__nv_bfloat16*)dqkv, dqw, dkw, T, Hq, Hkv, has_norm);
  B200_CHECK(cudaGetLastError());
  return 0;
}

int b200_swiglu_fwd(const void* gu, void* out, long long T, int I, cudaStream_t stream) {
  using namespace b200;
  if (T == 0) return 0;
  if (I % 8) return -100;
  int threads;
  const dim3 grid = swiglu_grid(T, I, 2, threads);
  swiglu_fwd_kernel<2><<<grid, threads, 0, stream>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)out, T, I);
  B200_CHECK(cudaGetLastError());
  return 0;
}
int b200_swiglu_bwd(const void* dy, const void* gu, void* dgu, long long T, int I,
                    cudaStream_t stream) {
  using namespace b200;
  if (T == 0) return 0;
  if (I % 8) return -100;
  int threads;
  const dim3 grid = swiglu_grid(T, I, 2, threads);
  swiglu_bwd_kernel<2><<<grid, threads, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)gu,
                                                     (__nv_bfloat16*)dgu, T, I);
  B200_CHECK(cudaGetLastError());
  return 0;
}

}  // extern "C"

// ------------------------------------------ RMSNorm backward, built-in scratch ----
// See norm_static_scratch.h. The partial sums of dw go to a file-scope device array
// whose address is looked up once per device; nothing here allocates.
namespace b200 {
static __device__ __align__(256) float g_rmsnorm_bwd_scratch[static_cast<size_t>(B200_RMSNORM_STATIC_MAX_BLOCKS) *
                                                             B200_RMSNORM_STATIC_MAX_H];
constexpr int kMaxDevices = 64;
static std::mutex g_scratch_mu;
static float* g_scratch_ptr[kMaxDevices] = {};
}  // namespace b200

extern "C" int b200_rmsnorm_bwd_static(const void* dy, const void* x, const void* w, const float* rstd,
                                       const void* dres, void* dx, float* dw, int dw_accumulate, int T, int H,
                                       cudaStream_t stream) {
  using namespace b200;
  if (T == 0) return 0;
  if (H % 8) return -100;
  const int grid = b200_rmsnorm_bwd_blocks(T);
  if (H > B200_RMSNORM_STATIC_MAX_H || grid > B200_RMSNORM_STATIC_MAX_BLOCKS) {
    fprintf(stderr,
            "b200_rmsnorm_bwd_static: H=%d (max %d) or %d blocks (max %d) exceeds the built-in scratch; "
            "use b200_rmsnorm_bwd with a caller-provided buffer\n",
            H, B200_RMSNORM_STATIC_MAX_H, grid, B200_RMSNORM_STATIC_MAX_BLOCKS);
    return B200_ERR_STATIC_SCRATCH_TOO_SMALL;
  }
  int dev = 0;
  B200_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return -3;
  float* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
      // the array's name is only meaningful in device code; ask the runtime for its address on
      // the current device
      float* p = nullptr;
      B200_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_rmsnorm_bwd_scratch));
      g_scratch_ptr[dev] = p;
    }
    scratch = g_scratch_ptr[dev];
  }
  return b200_rmsnorm_bwd(dy, x, w, rstd, dres, dx, scratch, dw, dw_accumulate, T, H, stream);
}
