// Varlen packed causal FlashAttention backward for sm_100a (tcgen05 + TMEM).
//
// One CTA owns one (128-row key/value block of one sequence, kv head) pair. It
// keeps K_j and V_j resident in shared memory and dK_j / dV_j as fp32
// accumulators in TMEM (2 x 128 columns) while it walks every query block i on
// or below the causal diagonal, for every query head of the GQA group:
//
//   S^T   = K_j Q_i^T           (TMEM cols 256..383)
//   dP^T  = V_j dO_i^T          (TMEM cols 384..511)
//   P^T   = exp2(S^T*c - lse_i) (registers → bf16 → TMEM, over the S^T columns it came from)
//   dV   += P^T dO_i            (A operand from TMEM; dO_i read MN-major from the same tile)
//   dS^T  = P^T ∘ (dP^T - Δ_i)  (registers → bf16 → swizzled smem; the softmax scale is applied to dK and dQ)
//   dQ_i^T = K_j^T dS^T         (over the dP^T columns; both operands MN-major)
//   dK   += dS^T Q_i            (Q_i read MN-major)
//
// Working on the transposed score tile makes each compute thread own (part of)
// one key row, so P^T and dS^T are written row-per-thread as K-major A operands
// and no tile is ever transposed in memory. dQ is produced transposed as well: a lane of
// the warps that drain it owns a head dimension, so the 32 lanes of a reduction into the fp32 dQ buffer hit one
// 128-byte line (with a query row per lane every lane touched a line of its own).
//
// What bounds it: 5 products of 128^3 take 2550 cycles per tile pair at the tensor cores' rate, their operands 2300
// cycles of shared memory bandwidth (P^T from TMEM saves a write and a read of 32 KB), the exponentials 1024 cycles. In sequence these and
// their hand-offs take four times as long, so the roles overlap: S^T of the next block is issued as soon as P^T is
// consumed and is ready while the compute warps still work on dS^T; four warps of their own drain dQ while
// dK accumulates. Before, one warp set did everything in turn: 8 sequences of 8192, 16 / 8 heads: 11.6 ms (472
// TFLOP/s), now 6.5 ms (842 TFLOP/s). The tensor cores
// are busy 42% of the time: what is left is the chain from dS^T over dQ and its read-out to the next dP^T (taking dQ out by bulk
// copies from shared memory, or not at all, changes nothing).
//
// Replaces flash-attn's backward / aten._flash_attention_backward in the
// reference (areal/experimental/models/archon/attention/varlen.py:116).
#include "common/host_utils.h"
#include "common/ptx.cuh"

namespace b200 {

constexpr int kD = 128;
constexpr int kBT = 128;  // rows of every tile (q and kv)
constexpr int kBwdCompute = 8;  // compute warps: w and w + 4 share 32 TMEM lanes and take 64 columns each
constexpr int kBwdDrain = 4;    // warps that take dQ out of TMEM and stage the row statistics
constexpr int kBwdThreads = (kBwdCompute + kBwdDrain + 2) * 32;  // + TMA producer + MMA issuer

struct AttnBwdTile {
  int kv_start;   // first global token row of this kv block
  int kv_len;     // valid kv rows in the block (<= 128)
  int kv_off;     // offset of the block inside its sequence
  int seq_start;  // first global token row of the sequence
  int seq_len;    // end of the query range (sequence-relative); queries [max(kv_off, q_begin), seq_len) are visited
  int q_begin;    // first sequence position present in the query array (0 unless context-parallel)
  int pad1, pad2;
};

constexpr int kTileBytes = kBT * kD * 2;  // 32 KB
// K, V resident; (Q, dO) x 2 stages; dS^T.
constexpr int kAttnBwdSmem = 2 * kTileBytes + 4 * kTileBytes + kTileBytes;  // 224 KB

// Δ[h, t] = sum_d dO[t,h,d] * O[t,h,d]
__global__ void attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ o,
                                      const __nv_bfloat16* __restrict__ dout,
                                      float* __restrict__ delta, int T, int Hq) {
  const long long gw = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= static_cast<long long>(T) * Hq) return;
  const int t = static_cast<int>(gw / Hq), h = static_cast<int>(gw % Hq);
  const uint2 a = reinterpret_cast<const uint2*>(o + gw * kD)[lane];
  const uint2 b = reinterpret_cast<const uint2*>(dout + gw * kD)[lane];
  const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]);
    s += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int o2 = 16; o2 > 0; o2 >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o2);
  if (lane == 0) delta[static_cast<long long>(h) * T + t] = s;
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                   long long n) {
  for (long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x * 4) {
    const float4 v = *reinterpret_cast<const float4*>(in + i);
    uint2 pk;
    reinterpret_cast<__nv_bfloat162*>(&pk)[0] = __floats2bfloat162_rn(v.x, v.y);
    reinterpret_cast<__nv_bfloat162*>(&pk)[1] = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(out + i) = pk;
  }
}

__device__ __forceinline__ void red_add(float* addr, float a) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(a) : "memory");
}
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// D[tmem] (+)= A[tmem] * B[smem desc]: A holds two bf16 per 32-bit column, 8 columns per 16-wide reduction step
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One arrival for the warp: 32 lanes that arrive by themselves queue up at the barrier.
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// two fp32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)),
        "l"(reinterpret_cast<const uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return d;
}

// What a compute thread needs to know to mask its key row against a query block.
struct BwdMask {
  bool kv_valid, diag;
  int q0, q_rows, kv_pos, kv_exit;
  template <bool TREE>
  __device__ __forceinline__ bool valid(int col) const {
    bool v = kv_valid && (col < q_rows) && (!diag || (q0 + col >= kv_pos));
    if (TREE) v = v && (q0 + col < kv_exit);
    return v;
  }
};

// 32 columns of P^T: exp2(S^T * c - lse), packed to bf16.
template <bool MASK, bool TREE>
__device__ __forceinline__ void bwd_p32(const uint32_t (&raw)[32], const float* lse, int col0, float scale_log2,
                                        const BwdMask& m, uint32_t* packed) {
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    const float4 l = *reinterpret_cast<const float4*>(lse + e);
    const float2 sc = make_float2(scale_log2, scale_log2);
    const float2 a0 = fma2(make_float2(__uint_as_float(raw[e]), __uint_as_float(raw[e + 1])), sc, make_float2(l.x, l.y));
    const float2 a1 = fma2(make_float2(__uint_as_float(raw[e + 2]), __uint_as_float(raw[e + 3])), sc, make_float2(l.z, l.w));
    float p[4] = {exp2_ftz(a0.x), exp2_ftz(a0.y), exp2_ftz(a1.x), exp2_ftz(a1.y)};
    if (MASK) {
#pragma unroll
      for (int u = 0; u < 4; ++u) p[u] = m.valid<TREE>(col0 + e + u) ? p[u] : 0.f;
    }
    __nv_bfloat162 a = __floats2bfloat162_rn(p[0], p[1]), b = __floats2bfloat162_rn(p[2], p[3]);
    packed[e / 2] = *reinterpret_cast<uint32_t*>(&a);
    packed[e / 2 + 1] = *reinterpret_cast<uint32_t*>(&b);
  }
}

// TREE: keys carry a subtree end (`key_exit`) that bounds the queries they are visible to.
template <bool TREE>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const AttnBwdTile* __restrict__ tiles, const float* __restrict__ lse,
                const float* __restrict__ delta, float* __restrict__ dq_acc,
                __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, int T, int Hq,
                int Hkv, long long lddk, long long lddv, float scale, int* status,
                const int* __restrict__ key_exit) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bars[20];
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_word;
  __shared__ __align__(16) float s_lse[2][kBT];
  __shared__ __align__(16) float s_delta[2][kBT];
  volatile int* abort_flag = &abort_word;

  uint8_t* sK = smem;
  uint8_t* sV = smem + kTileBytes;
  uint8_t* sQ = smem + 2 * kTileBytes;   // [2 stages]
  uint8_t* sdO = smem + 4 * kTileBytes;  // [2 stages]
  uint8_t* sdS = smem + 6 * kTileBytes;  // dS^T
  uint64_t* kv_full = &bars[0];
  uint64_t* q_full = &bars[1];    // [2]
  uint64_t* q_empty = &bars[3];   // [2]
  uint64_t* do_full = &bars[5];   // [2]
  uint64_t* do_empty = &bars[7];  // [2]
  uint64_t* ls_full = &bars[9];   // [2] lse and delta of a block are staged
  uint64_t* s_full = &bars[11];
  uint64_t* dp_full = &bars[12];
  uint64_t* p_ready = &bars[13];
  uint64_t* ds_ready = &bars[14];
  uint64_t* ds_free = &bars[15];  // the products that read dS^T are done
  uint64_t* dq_full = &bars[16];
  uint64_t* dq_read = &bars[17];
  uint64_t* acc_done = &bars[18];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const AttnBwdTile tile = tiles[blockIdx.x];
  const int hk = blockIdx.y;
  const int group = Hq / Hkv;
  // query blocks i with rows >= kv_off (causal): first block index containing kv_off
  // q_begin (0 for ordinary batches): first sequence position held by the local query array
  // (context parallelism: this rank owns the positions [q_begin, seq_len) of the sequence)
  const int qb_first = max(tile.kv_off, tile.q_begin) / kBT;
  const int qb_count = (tile.seq_len + kBT - 1) / kBT - qb_first;
  const int n_iter = qb_count > 0 ? qb_count * group : 0;  // iteration it -> (head g = it / qb_count, block i = it % qb_count)
  const float scale_log2 = scale * 1.4426950408889634f;

  if (threadIdx.x == 0) {
    abort_word = (smem_u32(smem) & 1023) ? 1 : 0;
    if (abort_word) atomicCAS(status, 0, kErrBounds);
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
      mbar_init(&ls_full[i], kBwdDrain);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, kBwdCompute);
    mbar_init(ds_ready, kBwdCompute);
    mbar_init(ds_free, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, kBwdDrain);
    mbar_init(acc_done, 1);
    fence_mbar_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmdO);
  }
  constexpr int kTmaWarp = kBwdCompute + kBwdDrain, kMmaWarp = kTmaWarp + 1;
  if (warp == kMmaWarp) {
    tmem_alloc(&tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  const uint32_t tm_dK = tmem_base;
  const uint32_t tm_dV = tmem_base + 128;
  const uint32_t tm_S = tmem_base + 256;   // S^T, then P^T (its first and its third quarter)
  const uint32_t tm_dP = tmem_base + 384;  // dP^T, then dQ^T
  const bool bad_align = (abort_word != 0);

  if (bad_align) {
  } else if (warp == kTmaWarp) {
    // ------------------------------------------------------ TMA producer --
    if (elect_one_sync()) {
      mbar_arrive_expect_tx(kv_full, 2 * kTileBytes);
      tma_load_2d(sK, &tmK, kv_full, hk * kD, tile.kv_start);
      tma_load_2d(sK + kTileBytes / 2, &tmK, kv_full, hk * kD + 64, tile.kv_start);
      tma_load_2d(sV, &tmV, kv_full, hk * kD, tile.kv_start);
      tma_load_2d(sV + kTileBytes / 2, &tmV, kv_full, hk * kD + 64, tile.kv_start);
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        const int st = it & 1;
        const uint32_t ph = (it >> 1) & 1;
        const int g = it / qb_count, i = qb_first + it % qb_count;
        const int h = hk * group + g;
        const int row = tile.seq_start + i * kBT;
        if (!mbar_wait(&q_empty[st], ph ^ 1, abort_flag)) { ok = false; break; }
        mbar_arrive_expect_tx(&q_full[st], kTileBytes);
        tma_load_2d(sQ + st * kTileBytes, &tmQ, &q_full[st], h * kD, row);
        tma_load_2d(sQ + st * kTileBytes + kTileBytes / 2, &tmQ, &q_full[st], h * kD + 64, row);
        if (!mbar_wait(&do_empty[st], ph ^ 1, abort_flag)) { ok = false; break; }
        mbar_arrive_expect_tx(&do_full[st], kTileBytes);
        tma_load_2d(sdO + st * kTileBytes, &tmdO, &do_full[st], h * kD, row);
        tma_load_2d(sdO + st * kTileBytes + kTileBytes / 2, &tmdO, &do_full[st], h * kD + 64, row);
      }
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(status, 0, kErrMbarTimeoutProducer);
        unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == kMmaWarp) {
    // -------------------------------------------------------- MMA issuer --
    if (elect_one_sync()) {
      // all tiles are [128 rows][2 halves of 64 columns], 128B-swizzled.
      // K-major view of a tile (rows = M/N index, columns = reduction):
      //   half hh, k-step kk: base + hh*16K + kk*32, LBO 16, SBO 1024
      // MN-major view (columns = M/N index, rows = reduction):
      //   k-step k (16 rows): base + k*2048, LBO 16K (next 64 columns), SBO 1024
      constexpr uint32_t id_kk = make_idesc(1, 1, 0, 0, kBT, kBT);  // A K-major, B K-major
      constexpr uint32_t id_kmn = make_idesc(1, 1, 0, 1, kBT, kD);  // A K-major, B MN-major
      constexpr uint32_t id_mnmn = make_idesc(1, 1, 1, 1, kD, kBT); // both MN-major
      constexpr uint32_t HALF = kTileBytes / 2;
      // Descriptors of the tiles, once; a reduction step, the second half and the other stage are additions to the address
      // field. One thread issues 40 products a block, and building two descriptors for each held it up.
      constexpr uint32_t kStage = kTileBytes >> 4;
      auto k_major = [](const uint8_t* t) { return make_sdesc_sw128(smem_u32(t), 16, 1024); };
      auto mn_major = [](const uint8_t* t) { return make_sdesc_sw128(smem_u32(t), HALF, 1024); };
      const uint64_t dK_k = k_major(sK), dK_mn = mn_major(sK), dV_k = k_major(sV), dS_k = k_major(sdS), dS_mn = mn_major(sdS);
      const uint64_t dQ_k = k_major(sQ), dQ_mn = mn_major(sQ), dO_k = k_major(sdO), dO_mn = mn_major(sdO);
      // D[128 keys, 128 queries] = tile (K-major) * rows of stage (K-major)^T
      auto scores = [&](uint32_t d, uint64_t a, uint64_t b) {
#pragma unroll
        for (int k = 0; k < kD / 16; ++k) {
          const uint32_t off = ((k >> 2) * HALF + (k & 3) * 32) >> 4;
          umma_f16(d, a + off, b + off, id_kk, k > 0 ? 1u : 0u);
        }
      };
      bool ok = mbar_wait(kv_full, 0, abort_flag);
      if (ok && n_iter > 0) {
        ok = mbar_wait(&q_full[0], 0, abort_flag);
        tc_fence_after();
        if (ok) {
          scores(tm_S, dK_k, dQ_k);
          umma_commit(s_full);
          ok = mbar_wait(&do_full[0], 0, abort_flag);
          tc_fence_after();
        }
        if (ok) {
          scores(tm_dP, dV_k, dO_k);
          umma_commit(dp_full);
        }
      }
      for (int it = 0; it < n_iter && ok; ++it) {
        const int st = it & 1, nst = st ^ 1;
        const uint32_t nph = ((it + 1) >> 1) & 1;
        const uint32_t itp = it & 1;
        const bool more = it + 1 < n_iter;
        if (!mbar_wait(p_ready, itp, abort_flag)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kBT / 16; ++k)  // dV += P^T dO   (reduction over q rows)
          umma_f16_ts(tm_dV, tm_S + (k >> 2) * 64 + (k & 3) * 8, dO_mn + st * kStage + k * 128, id_kmn,
                      (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(&do_empty[st]);
        if (more) {
          // products run in the order of issue: S^T of the next block overwrites P^T when dV has read it
          if (!mbar_wait(&q_full[nst], nph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          scores(tm_S, dK_k, dQ_k + nst * kStage);
          umma_commit(s_full);
        }
        if (!mbar_wait(ds_ready, itp, abort_flag)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kBT / 16; ++k)  // dQ^T = K^T dS^T  (reduction over kv rows)
          umma_f16(tm_dP, dK_mn + k * 128, dS_mn + k * 128, id_mnmn, k > 0 ? 1u : 0u);
        umma_commit(dq_full);
#pragma unroll
        for (int k = 0; k < kBT / 16; ++k) {  // dK += dS^T Q
          const uint32_t aoff = ((k >> 2) * HALF + (k & 3) * 32) >> 4;
          umma_f16(tm_dK, dS_k + aoff, dQ_mn + st * kStage + k * 128, id_kmn, (it > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&q_empty[st]);
        umma_commit(ds_free);
        if (more) {
          if (!mbar_wait(&do_full[nst], nph, abort_flag)) { ok = false; break; }
          // the dP^T columns hold dQ^T until it has been read out
          if (!mbar_wait(dq_read, itp, abort_flag)) { ok = false; break; }
          tc_fence_after();
          scores(tm_dP, dV_k, dO_k + nst * kStage);
          umma_commit(dp_full);
        }
      }
      if (ok) umma_commit(acc_done);
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(status, 0, kErrMbarTimeoutMma);
      }
    }
  } else if (warp >= kBwdCompute) {
    // ------------------------------------- row statistics in, dQ^T out --
    const int d = (warp - kBwdCompute) * 32 + lane;  // TMEM lane: a head dimension of dQ^T, a query row of the statistics
    const uint32_t lane_addr = static_cast<uint32_t>((warp - kBwdCompute) * 32) << 16;
    auto stage = [&](int it) {  // log2 units for lse; rows past the sequence: probability zero
      const int g = it / qb_count, i = qb_first + it % qb_count;
      const int h = hk * group + g;
      const int qi = i * kBT + d;
      const long long idx = static_cast<long long>(h) * T + tile.seq_start + qi;
      const bool v = qi < tile.seq_len;
      s_lse[it & 1][d] = v ? lse[idx] * -1.4426950408889634f : -INFINITY;
      s_delta[it & 1][d] = v ? -delta[idx] : 0.f;
      warp_arrive(&ls_full[it & 1]);
    };
    bool ok = true;
    if (n_iter > 0) stage(0);
    for (int it = 0; it < n_iter && ok; ++it) {
      // dQ of block it - 1 was complete, so the compute warps are done with the buffer of it - 1
      if (it + 1 < n_iter) stage(it + 1);
      const int g = it / qb_count, i = qb_first + it % qb_count;
      const int h = hk * group + g;
      const int q0 = i * kBT;
      const int q_rows = min(kBT, tile.seq_len - q0);
      float* dst = dq_acc + (static_cast<long long>(tile.seq_start + q0) * Hq + h) * kD + d;
      const long long pitch = static_cast<long long>(Hq) * kD;
      if (!mbar_wait(dq_full, it & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < kBT; c += 64) {
        uint32_t raw[2][32];
        tmem_ld_32x32(tm_dP + lane_addr + c, raw[0]);
        tmem_ld_32x32(tm_dP + lane_addr + c + 32, raw[1]);
        tmem_ld_wait();
        if (c) {
          tc_fence_before();
          warp_arrive(dq_read);
        }
        if (q_rows == kBT) {
#pragma unroll
          for (int e = 0; e < 64; ++e) red_add(dst + (c + e) * pitch, __uint_as_float(raw[e >> 5][e & 31]) * scale);
        } else {
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (c + e < q_rows) red_add(dst + (c + e) * pitch, __uint_as_float(raw[e >> 5][e & 31]) * scale);
        }
      }
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicCAS(status, 0, kErrMbarTimeoutEpilogue);
    }
  } else {
    // ---------------------------------------------------- compute warps --
    const int quad = warp & 3;    // TMEM lane quarter this warp may read
    const int cpart = warp >> 2;  // which 64 columns of every 128-column tile this warp handles
    const int r = quad * 32 + lane;  // kv row inside the block == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t my_S = tm_S + lane_addr + cpart * 64, my_dP = tm_dP + lane_addr + cpart * 64;
    BwdMask m;
    m.kv_pos = tile.kv_off + r;
    m.kv_valid = r < tile.kv_len;
    // tree attention: this key is visible to the queries of its own subtree only
    m.kv_exit = (TREE && m.kv_valid) ? key_exit[tile.kv_start + r] : 0x7fffffff;
    uint8_t* dsrow = sdS + cpart * (kTileBytes / 2) + r * 128;
    bool ok = true;
    for (int it = 0; it < n_iter && ok; ++it) {
      const uint32_t itp = it & 1;
      const int i = qb_first + it % qb_count;
      m.q0 = i * kBT;  // offset of the q block inside the sequence
      m.q_rows = min(kBT, tile.seq_len - m.q0);
      m.diag = m.q0 < tile.kv_off + kBT;  // block touches the causal diagonal
      // whole blocks need no masks: the row statistics and every key row are in range
      const bool mask = TREE || m.diag || m.q_rows < kBT || tile.kv_len < kBT;
      if (!mbar_wait(&ls_full[itp], (it >> 1) & 1, abort_flag)) { ok = false; break; }
      if (!mbar_wait(s_full, itp, abort_flag)) { ok = false; break; }
      tc_fence_after();
      uint32_t p[32];  // this thread's 64 columns, two to a word
#pragma unroll
      for (int cl = 0; cl < 2; ++cl) {
        uint32_t raw[32];
        tmem_ld_32x32(my_S + cl * 32, raw);
        tmem_ld_wait();
        const int col = cpart * 64 + cl * 32;
        if (mask) bwd_p32<true, TREE>(raw, &s_lse[itp][col], col, scale_log2, m, p + cl * 16);
        else bwd_p32<false, TREE>(raw, &s_lse[itp][col], col, scale_log2, m, p + cl * 16);
      }
      tmem_st_32x32(my_S, p);
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(p_ready);
      if (!mbar_wait(dp_full, itp, abort_flag)) { ok = false; break; }
      tc_fence_after();
      // the buffer holds dS^T of the previous block until dQ and dK have read it
      if (it > 0 && !mbar_wait(ds_free, itp ^ 1, abort_flag)) { ok = false; break; }
#pragma unroll
      for (int cl = 0; cl < 2; ++cl) {
        uint32_t raw[32];
        tmem_ld_32x32(my_dP + cl * 32, raw);
        tmem_ld_wait();
        const float* dl = &s_delta[itp][cpart * 64 + cl * 32];
#pragma unroll
        for (int e = 0; e < 32; e += 8) {  // a 16-byte piece of the row
          const float4 d0 = *reinterpret_cast<const float4*>(dl + e), d1 = *reinterpret_cast<const float4*>(dl + e + 4);
          const float dd[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
          uint4 out;
          uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t w = p[cl * 16 + e / 2 + u];
            const float pa = __uint_as_float(w << 16), pb = __uint_as_float(w & 0xffff0000u);
            const float2 pp = make_float2(pa, pb);
            const float2 ds = mul2(pp, add2(make_float2(__uint_as_float(raw[e + 2 * u]), __uint_as_float(raw[e + 2 * u + 1])),
                                            make_float2(dd[2 * u], dd[2 * u + 1])));
            __nv_bfloat162 b = __floats2bfloat162_rn(ds.x, ds.y);
            o[u] = *reinterpret_cast<uint32_t*>(&b);
          }
          const int piece = cl * 4 + e / 8;
          *reinterpret_cast<uint4*>(dsrow + ((piece ^ (r & 7)) << 4)) = out;
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      warp_arrive(ds_ready);
    }
    // epilogue: dK, dV
    if (ok) ok = mbar_wait(acc_done, 0, abort_flag);
    if (ok) {
      tc_fence_after();
      __nv_bfloat16* dk_row = dk + static_cast<long long>(tile.kv_start + r) * lddk + hk * kD;
      __nv_bfloat16* dv_row = dv + static_cast<long long>(tile.kv_start + r) * lddv + hk * kD;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        __nv_bfloat16* dst = which ? dv_row : dk_row;
        const uint32_t tm = which ? tm_dV : tm_dK;
        const float f = which ? 1.f : scale;
#pragma unroll 1
        for (int cl = 0; cl < 2; ++cl) {
          const int c = cpart * 2 + cl;
          uint32_t raw[32];
          if (n_iter > 0) {
            tmem_ld_32x32(tm + lane_addr + c * 32, raw);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) raw[e] = 0;
          }
          if (m.kv_valid) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              uint4 pk;
              __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
              for (int u = 0; u < 4; ++u)
                pb[u] = __floats2bfloat162_rn(__uint_as_float(raw[e * 8 + 2 * u]) * f,
                                              __uint_as_float(raw[e * 8 + 2 * u + 1]) * f);
              reinterpret_cast<uint4*>(dst + c * 32)[e] = pk;
            }
          }
        }
      }
    } else if (lane == 0) {
      *abort_flag = 1;
      atomicCAS(status, 0, kErrMbarTimeoutEpilogue);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200

extern "C" {

// q, o, dout: [T, Hq*128] contiguous bf16; k, v with pitches ldk/ldv; lse and
// delta_ws are [Hq, T] fp32; dq_acc is a zero-initialised fp32 [T, Hq*128]
// workspace; dq (bf16, pitch lddq) receives its rounded value; dk/dv are bf16
// with pitches lddk/lddv (they may point into a fused dqkv buffer).
int b200_attn_bwd_ex(const void* q, const void* k, const void* v, const void* o, const void* dout,
                     const float* lse, float* delta_ws, float* dq_acc, void* dq, void* dk, void* dv,
                     const void* tiles, int n_tiles, int T, int Tkv, int Hq, int Hkv, long long ldk,
                     long long ldv, long long lddk, long long lddv, float softmax_scale,
                     const int* key_exit, cudaStream_t stream);

int b200_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                  const float* lse, float* delta_ws, float* dq_acc, void* dq, void* dk, void* dv,
                  const void* tiles, int n_tiles, int T, int Hq, int Hkv, long long ldk,
                  long long ldv, long long lddk, long long lddv, float softmax_scale,
                  cudaStream_t stream) {
  return b200_attn_bwd_ex(q, k, v, o, dout, lse, delta_ws, dq_acc, dq, dk, dv, tiles, n_tiles, T, 0, Hq, Hkv, ldk,
                          ldv, lddk, lddv, softmax_scale, nullptr, stream);
}

// Extended form, see b200_attn_fwd_ex: k, v, dk, dv have Tkv rows; key_exit enables the tree mask.
int b200_attn_bwd_ex(const void* q, const void* k, const void* v, const void* o, const void* dout,
                     const float* lse, float* delta_ws, float* dq_acc, void* dq, void* dk, void* dv,
                     const void* tiles, int n_tiles, int T, int Tkv, int Hq, int Hkv, long long ldk,
                     long long ldv, long long lddk, long long lddv, float softmax_scale,
                     const int* key_exit, cudaStream_t stream) {
  using namespace b200;
  if (n_tiles == 0 || T == 0) return 0;
  if (Tkv <= 0) Tkv = T;
  if (Hq % Hkv) return -100;
  {
    const long long warps = static_cast<long long>(T) * Hq;
    attn_bwd_delta_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, stream>>>(
        (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta_ws, T, Hq);
  }
  CUtensorMap tmQ, tmK, tmV, tmdO;
  int rc = make_tmap_2d(&tmQ, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)Hq * kD,
                        (uint64_t)Hq * kD * 2, kBT, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tmdO, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)Hq * kD,
                    (uint64_t)Hq * kD * 2, kBT, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tmK, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tkv, (uint64_t)Hkv * kD, ldk * 2,
                    kBT, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tmV, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tkv, (uint64_t)Hkv * kD, ldv * 2,
                    kBT, 64);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    B200_CHECK(cudaFuncSetAttribute(attn_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnBwdSmem));
    B200_CHECK(cudaFuncSetAttribute(attn_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnBwdSmem));
    attr_set = true;
  }
  int* status = device_status_word();
  if (!status) return -3;
  dim3 grid(n_tiles, Hkv);
  auto kernel = key_exit ? attn_bwd_kernel<true> : attn_bwd_kernel<false>;
  kernel<<<grid, kBwdThreads, kAttnBwdSmem, stream>>>(
      tmQ, tmK, tmV, tmdO, reinterpret_cast<const AttnBwdTile*>(tiles), lse, delta_ws, dq_acc, (__nv_bfloat16*)dk,
      (__nv_bfloat16*)dv, T, Hq, Hkv, lddk, lddv, softmax_scale, status, key_exit);
  B200_CHECK(cudaGetLastError());
  if (dq) {
    const long long n = static_cast<long long>(T) * Hq * kD;
    long long g = (n / 4 + 255) / 256;
    const long long maxg = static_cast<long long>(sm_count()) * 16;
    if (g > maxg) g = maxg;
    f32_to_bf16_kernel<<<(unsigned)g, 256, 0, stream>>>(dq_acc, (__nv_bfloat16*)dq, n);
    B200_CHECK(cudaGetLastError());
  }
  return 0;
}

}  // extern "C"
