// The same product for few output tiles: C[128, BN] tiles cut into narrower ones, so that they reach more SMs.
//
// A decode batch (128 rows against a few thousand output features) has so few 128 x 256 tiles that most SMs would idle
// while a handful of them walk all of K.  Every element is one chain of MMAs over all of K in one accumulator, as in the
// persistent kernel, so that a row's result has the same bits whatever the number of rows and columns of the call.  (K divided
// over a cluster takes 13.3 us in place of 19.0 at 128 x 3584 x 8192 and gives up just that: it was built and taken back.)
// A K step of four dependent MMAs takes 0.13 us however narrow the tile, which bounds a tile with warm operands; with cold ones
// the loads of an SM do.  Device time of the persistent kernel and of this one, back to back, weights warm / cold in L2, us:
// 128 x 512 x 512 6.9 / 6.7 -> 3.5 / 3.4, 128 x 3584 x 8192 40.4 / 50.9 -> 19.0 / 22.8, 128 x 8192 x 3584 21.3 / 26.3 -> 10.4 / 14.0,
// 256 x 512 x 8192 40.3 / 41.0 -> 18.8 / 20.9, 1024^3 9.5 / 9.6 -> 4.8 / 4.8.
// Pairs of CTAs that share the rows of x (64 each, tiles of 32 and 64 columns) measured 20.7 / 21.4 at 128 x 3584 x 8192 and 1.7 us
// more than single CTAs at short K: not kept.
//   warp 0  TMA producer   warp 1  MMA issuer   warp 2  tensor memory   then all eight warps store
#pragma once
#include "gemm_fused_common.cuh"

namespace bshmem {

constexpr int NARROW_THREADS = 256, NARROW_RING = 192 * 1024;   // ring of 48 / 32 / 24 KB stages for BN = 256 / 128 / 64
constexpr int NARROW_SMEM = NARROW_RING + 1024 /*alignment slack*/ + 256 /*barriers*/;

struct alignas(64) NarrowParams {
  CUtensorMap tmA, tmB;
  char* out;
  int* error_flag;
  uint64_t wait_limit_ns;
  int M, N, K, act, a_mn, b_mn;
  int first_tile;  // in the order of the persistent kernel: 128 x 256 tiles, m fastest
  int row_blocks;  // 128-row blocks of that order; the last may lie past M
  int follows;     // the persistent kernel of the same product runs before this one
};

template <int N_TILE, bool MN>
__global__ void __launch_bounds__(NARROW_THREADS, 1) gemm_narrow_kernel(const __grid_constant__ NarrowParams p) {
  constexpr int B_BYTES = N_TILE * BK * 2, STAGES = NARROW_RING / (A_STAGE + B_BYTES), MN_BLOCK = 64 * BK * 2;
  constexpr int PITCH = N_TILE + 4;
  static_assert(BM * PITCH * 4 <= NARROW_RING, "the finished tile reuses the ring");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_STAGE;
  uint64_t* full = (uint64_t*)(smem + NARROW_RING);  // [STAGES]
  uint64_t* empty = full + STAGES;                   // [STAGES]
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int SUB = BN / N_TILE;  // tiles of this kernel per 128 x 256 tile
  const int u = (int)blockIdx.x, t = p.first_tile + u / SUB;
  const int row0 = t % p.row_blocks * BM, col0 = t / p.row_blocks * BN + u % SUB * N_TILE;
  if (row0 >= p.M) {  // the block that an odd number of blocks was rounded up with
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

  const int kblocks = p.K / BK;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&p.tmA);
      tma_prefetch_desc(&p.tmB);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < kblocks; ++kb) {
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
      for (int kb = 0; kb < kblocks; ++kb) {
        if (!mbar_wait(&full[stage], phase, p.wait_limit_ns, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(sA + stage * A_STAGE), b_addr = smem_u32(sB + stage * B_BYTES);
        const uint64_t da = MN && p.a_mn ? umma_desc_mn_sw128(a_addr, MN_BLOCK) : umma_desc_k_sw128(a_addr);
        const uint64_t db = MN && p.b_mn ? umma_desc_mn_sw128(b_addr, MN_BLOCK) : umma_desc_k_sw128(b_addr);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16(tmem, da + k * a_step, db + k * b_step, idesc, (kb | k) != 0);
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      umma_commit(acc_full);
    }
  }
  __syncwarp();
  // Every MMA of this CTA is complete, so every load has been consumed and the ring is free for the finished tile.
  const bool ok = mbar_wait(acc_full, 0, p.wait_limit_ns, abort_flag) && !*abort_flag;
  if (!ok) {
    const uint64_t t0 = timer_ns();  // copies still in flight land before the shared memory is reused or goes away
    while (timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_after_sync();
  float* tile = (float*)smem;  // [BM][PITCH]
  {
    const int row = (warp & 3) * 32 + lane;
    float* mine = tile + row * PITCH;
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
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, N_TILE);
#pragma unroll 4
  for (int i = threadIdx.x; i < BM * (N_TILE / 4); i += NARROW_THREADS) {
    const int r = i / (N_TILE / 4), c = i % (N_TILE / 4) * 4;
    float4 a = *(const float4*)(tile + r * PITCH + c);
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
  if (p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x == 0 && *abort_flag) atomicOr(p.error_flag, 1);
}

}  // namespace bshmem
