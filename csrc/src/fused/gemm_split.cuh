// The same product for few output tiles: C[128, BN] tiles whose K range is divided over the CTAs of a cluster.
//
// A decode batch (128 rows against a few thousand output features) has so few 128 x 256 tiles that most SMs would idle
// while a handful of them walk all of K.  Here a cluster of `splits` CTAs shares a tile: each multiplies its part of K into
// its own tensor memory, the partial sums meet in shared memory, and every CTA adds 128 / splits rows of them, read from its
// peers through distributed shared memory in a fixed order (fp32, one rounding at the end: the same precision and the same
// result on every call).  No workspace, no flags, no second kernel.
// Bound by the loads of an SM (about 70 bytes per clock) and by HBM.  Device time before (persistent kernel) and now, launches
// back to back: 128 x 3584 x 8192 52 -> 16 us (weights at 3.7 TB/s), 128 x 8192 x 3584 27.4 -> 13.7, 128 x 512 x 512 7.9 -> 3.6,
// 1024^3 11.4 -> 5.0, 256 x 512 x 8192 42.7 -> 10.0.
//   warp 0  TMA producer   warp 1  MMA issuer   warp 2  tensor memory   then all eight warps reduce and store
#pragma once
#include "gemm_fused_common.cuh"

namespace bshmem {

constexpr int SPLIT_THREADS = 256, SPLIT_RING = 192 * 1024;   // ring of 48 / 32 / 24 KB stages for BN = 256 / 128 / 64
constexpr int SPLIT_SMEM = SPLIT_RING + 1024 /*alignment slack*/ + 256 /*barriers*/;

struct alignas(64) SplitParams {
  CUtensorMap tmA, tmB;
  char* out;
  int* error_flag;
  uint64_t wait_limit_ns;
  int M, N, K, act, a_mn, b_mn;
  int first_tile;  // in the order of the persistent kernel: 128 x 256 tiles, m fastest
  int row_blocks;  // 128-row blocks of that order; the last may lie past M
  int follows;     // the persistent kernel of the same product runs before this one
  int splits;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// Adds this CTA's rows of the partial tiles of the cluster and stores them.
template <int N_TILE, int SPLITS>
__device__ __forceinline__ void split_reduce_store(const SplitParams& p, const float* part, int rank, int row0, int col0) {
  constexpr int PITCH = N_TILE + 4, C4 = N_TILE / 4, ITEMS = BM / SPLITS * C4;
  const uint32_t base = smem_u32(part);
  uint32_t peer[SPLITS];
#pragma unroll
  for (int s = 0; s < SPLITS; ++s) peer[s] = SPLITS == 1 ? base : mapa_u32(base, s);
#pragma unroll 2
  for (int i = threadIdx.x; i < ITEMS; i += SPLIT_THREADS) {
    const int r = rank * (BM / SPLITS) + i / C4, c = i % C4 * 4;
    const uint32_t off = (uint32_t)(r * PITCH + c) * 4;
    float4 v[SPLITS];
#pragma unroll
    for (int s = 0; s < SPLITS; ++s) v[s] = ld_cluster_f4(peer[s] + off);
    float4 a = v[0];
#pragma unroll
    for (int s = 1; s < SPLITS; ++s) {
      a.x += v[s].x;
      a.y += v[s].y;
      a.z += v[s].z;
      a.w += v[s].w;
    }
    if (p.act == BSHMEM_FUSED_ACT_GELU_TANH) {
      a.x = gelu_tanh(a.x);
      a.y = gelu_tanh(a.y);
      a.z = gelu_tanh(a.z);
      a.w = gelu_tanh(a.w);
    }
    uint2 o;
    __nv_bfloat162* h = (__nv_bfloat162*)&o;
    h[0] = __floats2bfloat162_rn(a.x, a.y);
    h[1] = __floats2bfloat162_rn(a.z, a.w);
    *(uint2*)(p.out + ((size_t)(row0 + r) * p.N + col0 + c) * 2) = o;
  }
}

template <int N_TILE, bool MN>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) gemm_split_kernel(const __grid_constant__ SplitParams p) {
  constexpr int B_BYTES = N_TILE * BK * 2, STAGES = SPLIT_RING / (A_STAGE + B_BYTES), MN_BLOCK = 64 * BK * 2;
  static_assert(BM * (N_TILE + 4) * 4 <= SPLIT_RING, "the partial tile reuses the ring");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_STAGE;
  uint64_t* full = (uint64_t*)(smem + SPLIT_RING);  // [STAGES]
  uint64_t* empty = full + STAGES;                  // [STAGES]
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int SUB = BN / N_TILE;  // tiles of this kernel per 128 x 256 tile
  const int u = (int)blockIdx.x / p.splits, t = p.first_tile + u / SUB;
  const int row0 = t % p.row_blocks * BM, col0 = t / p.row_blocks * BN + u % SUB * N_TILE;
  const int splits = p.splits, rank = (int)blockIdx.x % splits;
  if (row0 >= p.M) {  // the whole cluster has no rows
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, N_TILE);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // The launch may overlap the end of the kernel before it in the stream: nothing that it writes is touched before this.
  // After the persistent kernel of the same product there is nothing to wait for (that one started when its inputs were
  // complete, and writes other tiles) until the end, so that the end of this kernel is the end of both.
  if (!p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");

  const int kblocks = p.K / BK, kb0 = kblocks * rank / splits, kb1 = kblocks * (rank + 1) / splits;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&p.tmA);
      tma_prefetch_desc(&p.tmB);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, p.wait_limit_ns, abort_flag)) break;
        mbar_expect_tx(&full[stage], A_STAGE + B_BYTES);
        if (MN && p.a_mn) {
#pragma unroll
          for (int i = 0; i < BM / 64; ++i) tma_load_2d(sA + stage * A_STAGE + i * MN_BLOCK, &p.tmA, &full[stage], row0 + i * 64, kb * BK);
        } else {
          tma_load_2d(sA + stage * A_STAGE, &p.tmA, &full[stage], kb * BK, row0);
        }
        if (MN && p.b_mn) {
#pragma unroll
          for (int i = 0; i < N_TILE / 64; ++i) tma_load_2d(sB + stage * B_BYTES + i * MN_BLOCK, &p.tmB, &full[stage], col0 + i * 64, kb * BK);
        } else {
          tma_load_2d(sB + stage * B_BYTES, &p.tmB, &full[stage], kb * BK, col0);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16_f32(BM, N_TILE) | (MN && p.a_mn ? UMMA_A_MN_MAJOR : 0u) | (MN && p.b_mn ? UMMA_B_MN_MAJOR : 0u);
      const uint64_t a_step = MN && p.a_mn ? 128 : 2, b_step = MN && p.b_mn ? 128 : 2;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, p.wait_limit_ns, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(sA + stage * A_STAGE), b_addr = smem_u32(sB + stage * B_BYTES);
        const uint64_t da = MN && p.a_mn ? umma_desc_mn_sw128(a_addr, MN_BLOCK) : umma_desc_k_sw128(a_addr);
        const uint64_t db = MN && p.b_mn ? umma_desc_mn_sw128(b_addr, MN_BLOCK) : umma_desc_k_sw128(b_addr);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16(tmem, da + k * a_step, db + k * b_step, idesc, kb != kb0 || k != 0);
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      umma_commit(acc_full);
    }
  }
  __syncwarp();
  // Every MMA of this CTA is complete, so every load has been consumed and the ring is free for the partial tile.
  const bool ok = mbar_wait(acc_full, 0, p.wait_limit_ns, abort_flag) && !*abort_flag;
  if (!ok) {
    const uint64_t t0 = timer_ns();  // copies still in flight land before the shared memory is reused or goes away
    while (timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_after_sync();
  float* part = (float*)smem;
  {
    const int row = (warp & 3) * 32 + lane;
    float* mine = part + row * (N_TILE + 4);
#pragma unroll
    for (int c = (warp >> 2) * (N_TILE / 2); c < (warp >> 2) * (N_TILE / 2) + N_TILE / 2; c += 32) {
      float f[32];
      tmem_ld_32x32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, (uint32_t*)f);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; j += 4) *(float4*)(mine + c + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
    }
  }
  tc_fence_before_sync();
  if (splits == 1) __syncthreads();
  else cluster_sync_all();
  if (warp == 2) tmem_dealloc(tmem, N_TILE);
  if (splits == 1) split_reduce_store<N_TILE, 1>(p, part, rank, row0, col0);
  else if (splits == 2) split_reduce_store<N_TILE, 2>(p, part, rank, row0, col0);
  else if (splits == 4) split_reduce_store<N_TILE, 4>(p, part, rank, row0, col0);
  else split_reduce_store<N_TILE, 8>(p, part, rank, row0, col0);
  if (splits > 1) cluster_sync_all();  // the peers have read my partial tile
  if (p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x == 0 && *abort_flag) atomicOr(p.error_flag, 1);
}

}  // namespace bshmem
