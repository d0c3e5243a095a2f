// The GEMM of gemm_core.cuh with the two SMs of a TPC on one 256 x 256 tile (cta_group::2).
//
// A single CTA's 128 x 256 tile takes in 48 KB per 64-wide reduction block, 94 bytes per cycle of its products: more than L2
// hands an SM. Here each CTA of the pair loads its own 128 rows of A and half of B's 256 (32 KB), the even CTA issues
// products that read both, and each CTA's TMEM collects its own 128 rows. Policies, operand majors and epilogue are those of
// the single-CTA kernel (a policy sees 128-row blocks; the optional grouped members are not supported). 16384 x 12288 x 2048:
// 1519 TFLOP/s forward and 1540 dgrad, against 1102 to 1290 and 1307 to 1457 on single SMs.
//
// Barriers: `full` and `tempty` live in the even CTA (loads of both CTAs complete on it, epilogue warps of both arrive on it),
// `empty` and `tfull` in each CTA (the even CTA's commits arrive in both). Every wait is bounded, as in gemm_core.cuh. No load
// is multicast.
#pragma once
#include "gemm_core.cuh"
#include "host_utils.h"

namespace b200 {

struct PairCfg {
  static constexpr int kBN = 256;
  static constexpr int kStages = 6;
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = kBN / 2 * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;  // of one CTA
  static constexpr int kSmemBytes = kStages * kStageBytes + 256 + 1024;
  static constexpr int kTmemCols = 2 * kBN;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address, in the cluster's shared window, of what lies at `p` in CTA `rank`
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// into this CTA's shared memory, completing on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t bar_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the products issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

template <bool A_MN, bool B_MN, class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N, int K,
                 const __grid_constant__ Epi epi, int* status) {
  using Cfg = PairCfg;
  constexpr int STAGES = Cfg::kStages, BN = Cfg::kBN;
  extern __shared__ uint8_t smem_raw[];
  // the same offset in both CTAs: the dynamic segment starts alike, and products address both with one descriptor
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * Cfg::kABytes;
  uint8_t* smem_epi = smem + STAGES * Cfg::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_epi + 4 * epi_warp_smem<Epi>(0));
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = bars + 2 * STAGES + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int tiles_mp = (M + 2 * kBM - 1) / (2 * kBM);
  const int tiles_n = (N + BN - 1) / BN;
  const int kblocks = (K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 8);
    }
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"(Cfg::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer --
    if (elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        int mp, n_blk;
        if (!epi.tile(pair, npairs, it, tiles_mp, tiles_n, mp, n_blk)) break;
        const int m0 = (2 * mp + static_cast<int>(rank)) * kBM, n0 = n_blk * BN + static_cast<int>(rank) * (BN / 2);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          // the even CTA's barrier counts the bytes of both; the other's loads may be ahead of this
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * Cfg::kStageBytes);
          const uint32_t bar = map_to_cta(&full[stage], 0);
          uint8_t* a_dst = smem_a + stage * Cfg::kABytes;
          uint8_t* b_dst = smem_b + stage * Cfg::kBBytes;
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < kBM / 64; ++j) tma_load_2d_pair(a_dst + j * 8192, &tmA, bar, m0 + j * 64, kb * kBK);
          } else {
            tma_load_2d_pair(a_dst, &tmA, bar, kb * kBK, m0);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(b_dst + j * 8192, &tmB, bar, n0 + j * 64, kb * kBK);
          } else {
            tma_load_2d_pair(b_dst, &tmB, bar, kb * kBK, n0);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // the even CTA's last commits arrive here too: stay until they have
      for (int s = 0; s < STAGES && ok; ++s) {
        ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(status, 0, kErrMbarTimeoutProducer);
        // Give copies already in flight time to land before the CTA retires.
        unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------ MMA issuer (even CTA) --
    if (rank == 0 && elect_one_sync()) {
      constexpr uint32_t idesc = make_idesc(1, 1, A_MN ? 1 : 0, B_MN ? 1 : 0, 2 * kBM, BN);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        int mp, n_blk;
        if (!epi.tile(pair, npairs, it, tiles_mp, tiles_n, mp, n_blk)) break;
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem_a + stage * Cfg::kABytes);
          const uint32_t b_addr = smem_u32(smem_b + stage * Cfg::kBBytes);
          const uint64_t a_desc =
              A_MN ? make_sdesc_sw128(a_addr, 8192, 1024) : make_sdesc_sw128(a_addr, 16, 1024);
          const uint64_t b_desc =
              B_MN ? make_sdesc_sw128(b_addr, 8192, 1024) : make_sdesc_sw128(b_addr, 16, 1024);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            const uint64_t a_k = a_desc + static_cast<uint64_t>((A_MN ? 2048 : 32) * k >> 4);
            const uint64_t b_k = b_desc + static_cast<uint64_t>((B_MN ? 2048 : 32) * k >> 4);
            umma_f16_pair(d_tmem, a_k, b_k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(&tfull[acc]);
      }
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(status, 0, kErrMbarTimeoutMma);
      }
    }
  } else {
    // ---------------------------------------------------------- epilogue --
    const int quarter = warp & 3;  // TMEM lanes [32*quarter, 32*quarter+32)
    typename Epi::State st;
    if constexpr (epi_warp_smem<Epi>(0) > 0) epi.bind(st, smem_epi + quarter * epi_warp_smem<Epi>(0));
    bool ok = true;
    for (int it = 0; ok; ++it) {
      int mp, n_blk;
      if (!epi.tile(pair, npairs, it, tiles_mp, tiles_n, mp, n_blk)) break;
      const int m_blk = 2 * mp + static_cast<int>(rank);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait(&tfull[acc], acc_phase, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int row = m_blk * kBM + quarter * 32 + lane;
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(quarter * 32) << 16);
      epi.begin(st, m_blk, n_blk, row);
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c * 32, r);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
        epi.chunk(st, row, n_blk * BN + c * 32, v);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(&tempty[acc], 0));
      epi.end(st, m_blk, n_blk, row);
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicCAS(status, 0, kErrMbarTimeoutEpilogue);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still reach its memory or barriers
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::kTmemCols));
  }
  // A pair's allocation is given back in both SMs: a CTA that left first would let a kernel of another stream allocate on its
  // SM while the other CTA is still at it.
  __syncwarp();
  cluster_sync_all();
}

// Host side: tensor maps with boxes of 128 rows (K-major) or 64 x 64 (MN-major) of both operands.
template <bool A_MN, bool B_MN, class Epi>
int launch_pair_epi(const CUtensorMap& tmA, const CUtensorMap& tmB, int M, int N, int K, const Epi& epi,
                    cudaStream_t stream) {
  auto kern = gemm_pair_kernel<A_MN, B_MN, Epi>;
  constexpr int smem = PairCfg::kSmemBytes + 4 * epi_warp_smem<Epi>(0);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set = true;
  }
  const long long tiles = static_cast<long long>((M + 2 * kBM - 1) / (2 * kBM)) * ((N + PairCfg::kBN - 1) / PairCfg::kBN);
  const int pairs = sm_count() / 2;
  const int grid = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  if (grid <= 0) return 0;
  int* status = device_status_word();
  if (!status) return -3;
  kern<<<grid, kGemmThreads, smem, stream>>>(tmA, tmB, M, N, K, epi, status);
  B200_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace b200
