// Grouped GEMM over ragged row groups (the experts of a mixture-of-experts layer) with the operands swapped.
//
//   out[r, :] = x[r, :] · w_g^T   for the rows r of group g, boundaries in device memory
//
// The tensor core multiplies 128 rows of its first operand (256 in a CTA pair) by N of its second, N any multiple of 16.
// The weights are the first operand here and the rows of the group the second, because the group is what is ragged: a group
// of 1030 rows is five column chunks of 208 (the last 198) instead of nine blocks of 128, and a decode batch's group of 15
// rows costs 16 columns instead of a block of 128, an eighth of whose result is kept.
//   warp 0  TMA producer: 128 weight rows and this CTA's part of the chunk's rows per 64-wide K step
//   warp 1  MMA issuer    (pair: the even CTA, 256 weight rows x N) into one of two accumulators in tensor memory
//   warp 2  tensor memory; warp 3 the tile list (no host round trip decides it)
//   warps 4-11 epilogue: lanes are output columns and registers are rows, so 32 rows at a time are transposed through shared
//             memory and stored as whole 128- or 256-byte pieces of output rows
// The ring's stages are as large as the largest chunk of the call needs: small groups leave room for more stages, which is
// what keeps enough weight bytes in flight when the weights' HBM traffic is the bound.
// Large groups are bound by the clock that the power limit leaves (K 7168, 1024 rows: 1.04 GHz in a loop of seconds, MMAs in 0.885 of the
// cycles), small ones by HBM.  Rows as the first operand in blocks of 128 (before) / weights first in CTA pairs (now), us, sizes within
// 10 % of the mean:
//   32 groups, N 4096, K 7168, gated   16 rows 328 / 272 (1.88 GB of weights: 6.9 TB/s)   256 631 / 505   1024 1741 / 1695
//   32 groups, N 7168, K 2048          16 rows 156 / 146 (0.94 GB)                        256 295 / 251   1024 1015 / 782
//   32 groups, N 2048, K 512           16 rows 12.4 / 12.3                                256 32.5 / 27.6  1024 88.9 / 69.9
//   256 groups, N 512, K 512           16 rows 40.6 / 30.0                                256 68.5 / 54.3
// These are short runs; a whole layer of 4096 tokens (1024 rows a group) gains nothing in a loop of seconds, at 512 to 2048 tokens 4 to 18 %.
// One epilogue warpgroup instead of two: 120 us in place of 69.9, and 27 % more than now at 16 x 1024 x 1024, 1024 rows.
#pragma once
#include "gemm_fused_common.cuh"

namespace bshmem {

constexpr int GRP_MAX_N = 256, GRP_STEP_N = 16, GRP_MAX_STAGES = 12, GRP_BOXES = GRP_MAX_N / GRP_STEP_N;
constexpr int GRP_EPI = 2, GRP_THREADS = 128 + GRP_EPI * EPI_THREADS;
constexpr int GRP_RING = 192 * 1024, GRP_STAGING = 16 * 1024;  // staging of one epilogue warpgroup
constexpr int GRP_SMEM = GRP_RING + GRP_EPI * GRP_STAGING + 1024 /*alignment slack*/ + 512 /*barriers*/ + (MAX_GROUPS + 4) * 4;

struct alignas(64) GroupedParams {
  CUtensorMap tmW;             // weights [groups * N][K], box 128 rows
  CUtensorMap tmX[GRP_BOXES];  // rows [M][K]; box i: the rows that a CTA loads for a chunk of GRP_STEP_N * (i + 1) columns
  char* out;
  const int* offsets;     // [groups + 1]
  int* error_flag;
  uint64_t wait_limit_ns;
  int groups, N, K, act;
};

struct GroupTile {
  int w_row;       // first weight row of the tile (a pair adds its half)
  int row0, rows;  // first row of the chunk and how many exist
  int n;           // columns of the MMA
  int col;         // first output column of the tile, before a gated activation
};

// A group of `rows` rows is cut into as few chunks of at most GRP_MAX_N as possible, of even size.
__host__ __device__ __forceinline__ int group_chunks(int rows) { return (rows + GRP_MAX_N - 1) / GRP_MAX_N; }
__host__ __device__ __forceinline__ int group_chunk_rows(int rows) {
  const int c = group_chunks(rows);
  return c ? ((rows + c - 1) / c + GRP_STEP_N - 1) / GRP_STEP_N * GRP_STEP_N : 0;
}

template <int W_ROWS>
__device__ __forceinline__ GroupTile group_tile(const GroupedParams& p, const int* prefix, int t) {
  int lo = 0, hi = p.groups;  // find g with prefix[g] <= t < prefix[g + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= t) lo = mid;
    else hi = mid;
  }
  const int local = t - prefix[lo], r0 = __ldcg(p.offsets + lo), total = __ldcg(p.offsets + lo + 1) - r0;
  // chunks run fastest: CTAs that run together share the weights through L2
  const int chunks = group_chunks(total), n = group_chunk_rows(total);
  const int c = local % chunks;
  GroupTile g;
  g.col = local / chunks * W_ROWS;
  g.w_row = lo * p.N + g.col;
  g.row0 = r0 + c * n;
  g.rows = min(n, total - c * n);
  g.n = (g.rows + GRP_STEP_N - 1) / GRP_STEP_N * GRP_STEP_N;
  return g;
}

template <bool PAIR, bool GATED>
__global__ void __launch_bounds__(GRP_THREADS, 1) gemm_grouped_kernel(const __grid_constant__ GroupedParams p) {
  constexpr int W_ROWS = PAIR ? 2 * BM : BM;  // weight rows per tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* staging = smem + GRP_RING;
  uint64_t* full = (uint64_t*)(staging + GRP_EPI * GRP_STAGING);
  uint64_t* empty = full + GRP_MAX_STAGES;
  uint64_t* acc_full = empty + GRP_MAX_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;           // [2]
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  int* s_max_n = (int*)(tmem_slot + 2);
  int* prefix = (int*)(full + 64);              // [groups + 1]: tiles before each group
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = PAIR ? cluster_ctarank() : 0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < GRP_MAX_STAGES; ++i) {
      mbar_init(&full[i], PAIR ? 2 : 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], (PAIR ? 2 : 1) * GRP_EPI * (EPI_THREADS / 32));  // one arrival per epilogue warp
    }
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc<PAIR ? 2 : 1>(tmem_slot, TMEM_COLS);
    tmem_relinquish<PAIR ? 2 : 1>();
  }
  // The launch may overlap the end of the kernel before it on the stream: what that one writes (the boundaries among it) is
  // read only after this.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == 3) {
    int tiles = 0, max_n = GRP_STEP_N;
    for (int base = 0; base < p.groups; base += 32) {
      const int g = base + lane;
      const int rows = g < p.groups ? max(0, __ldcg(p.offsets + g + 1) - __ldcg(p.offsets + g)) : 0;
      const int mine = group_chunks(rows) * (p.N / W_ROWS);
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      if (g < p.groups) prefix[g] = tiles + upto - mine;
      tiles += __shfl_sync(0xffffffffu, upto, 31);
      max_n = max(max_n, (int)__reduce_max_sync(0xffffffffu, (unsigned)group_chunk_rows(rows)));
    }
    if (lane == 0) {
      prefix[p.groups] = tiles;
      *s_max_n = max_n;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = prefix[p.groups], kblocks = p.K / BK;
  const int stage_bytes = A_STAGE + (PAIR ? *s_max_n / 2 : *s_max_n) * BK * 2;
  const int stages = min(GRP_MAX_STAGES, GRP_RING / stage_bytes);
  const int first = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, step = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&p.tmW);
      int stage = 0;
      uint32_t phase = 0;
      for (int t = first; t < total_tiles && !*abort_flag; t += step) {
        const GroupTile g = group_tile<W_ROWS>(p, prefix, t);
        const int rows = PAIR ? g.n / 2 : g.n, row0 = g.row0 + (int)cta_rank * rows;
        const CUtensorMap* tmX = &p.tmX[g.n / GRP_STEP_N - 1];  // one copy per step: cut into 16-row boxes it starved the tensor cores
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, p.wait_limit_ns, abort_flag)) break;
          uint8_t* w = smem + stage * stage_bytes;
          uint8_t* x = w + A_STAGE;
          const uint32_t lead = PAIR ? mapa_u32(smem_u32(&full[stage]), 0) : 0;
          const uint32_t bytes = A_STAGE + rows * BK * 2;
          if (PAIR) mbar_expect_tx_cluster(lead, bytes);
          else mbar_expect_tx(&full[stage], bytes);
          auto load = [&](uint8_t* dst, const CUtensorMap* map, int y) {
            if (PAIR) tma_load_2d_pair(dst, map, lead, kb * BK, y);
            else tma_load_2d(dst, map, &full[stage], kb * BK, y);
          };
          load(w, &p.tmW, g.w_row + (int)cta_rank * BM);
          load(x, tmX, row0);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
      // The arrivals of the last MMAs (in a pair from the other SM) must find this CTA still there.
      for (int i = 0; i < stages && !*abort_flag; ++i) {
        if (!mbar_wait(&empty[stage], phase ^ 1, p.wait_limit_ns, abort_flag)) break;
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if ((!PAIR || cta_rank == 0) && elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int t = first; t < total_tiles && !*abort_flag; t += step) {
        const uint32_t idesc = umma_idesc_bf16_f32(W_ROWS, group_tile<W_ROWS>(p, prefix, t).n);
        if (!mbar_wait(&acc_empty[acc], acc_phase ^ 1, p.wait_limit_ns, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * ACC_COLS);
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, p.wait_limit_ns, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t addr = smem_u32(smem + stage * stage_bytes);
          const uint64_t dw = umma_desc_k_sw128(addr), dx = umma_desc_k_sw128(addr + A_STAGE);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            if (PAIR) umma_bf16_pair(d_tmem, dw + (uint64_t)(k * 2), dx + (uint64_t)(k * 2), idesc, (kb | k) != 0);
            else umma_bf16(d_tmem, dw + (uint64_t)(k * 2), dx + (uint64_t)(k * 2), idesc, (kb | k) != 0);
          }
          if (PAIR) umma_commit_pair(&empty[stage]);
          else umma_commit(&empty[stage]);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (PAIR) umma_commit_pair(&acc_full[acc]);
        else umma_commit(&acc_full[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else if (warp >= EPI_WARP0) {
    // Two warpgroups take turns with the 32-row pieces of a tile, each with its own staging and barriers.
    const int team = (warp - EPI_WARP0) >> 2, ew = warp & 3, et = (int)threadIdx.x & (EPI_THREADS - 1);
    constexpr int OUT_COLS = GATED ? BM / 2 : BM, PER_ROW = OUT_COLS / 8;  // output columns of this CTA's half of a tile; 16-byte pieces of a row
    uint8_t* mine = staging + team * GRP_STAGING;           // two buffers [32 rows][OUT_COLS] bf16
    float* ex = (float*)(mine + 8192) + (ew >> 1) * 1024;   // gated: [32 rows][32 columns] fp32 between a gate warp and its up warp
    const size_t pitch = GATED ? (size_t)p.N / 2 : (size_t)p.N;
    int acc = 0, buf = 0;
    uint32_t acc_phase = 0;
    for (int t = first; t < total_tiles; t += step) {
      const GroupTile g = group_tile<W_ROWS>(p, prefix, t);
      const uint32_t ok = mbar_wait(&acc_full[acc], acc_phase, p.wait_limit_ns, abort_flag) ? 1u : 0u;
      if (!named_bar_and(1 + team, EPI_THREADS, ok)) break;  // all 128 threads go on or all leave
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + ((uint32_t)(ew * 32) << 16) + (uint32_t)(acc * ACC_COLS);
      auto release = [&] {  // this warp has its share of the accumulator in registers
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[acc]), 0));
          else mbar_arrive(&acc_empty[acc]);
        }
      };
      const int col = (g.col + (int)cta_rank * BM) / (GATED ? 2 : 1);
      if (team * 32 >= g.n) release();
#pragma unroll 1
      for (int c = team * 32; c < g.n; c += GRP_EPI * 32, buf ^= 1) {
        float f[32];
        tmem_ld_32x32(t_row + c, (uint32_t*)f);
        tmem_ld_wait();
        if (c + GRP_EPI * 32 >= g.n) release();
        if (p.act == BSHMEM_FUSED_ACT_GELU_TANH) {
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = gelu_tanh(f[j]);
        }
        __nv_bfloat16* tile = (__nv_bfloat16*)(mine + buf * (32 * OUT_COLS * 2));
        if (GATED) {
          // The weight rows are 32 gate rows followed by their 32 up rows: warps 0 and 2 hold gates, 1 and 3 the matching ups.
          // The gate warp finishes the first 16 rows and the up warp the others; each hands over what the other one needs.
          if (ew & 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) ex[j * 32 + lane] = f[j];
          } else {
#pragma unroll
            for (int j = 16; j < 32; ++j) ex[j * 32 + lane] = f[j];
          }
          named_bar_sync(1 + GRP_EPI + team * 2 + (ew >> 1), 64);
          __nv_bfloat16* to = tile + (ew >> 1) * 32 + lane;
          if (ew & 1) {
#pragma unroll
            for (int j = 16; j < 32; ++j) {
              const float gate = ex[j * 32 + lane];
              to[j * OUT_COLS] = __float2bfloat16_rn(gate / (1.0f + __expf(-gate)) * f[j]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) to[j * OUT_COLS] = __float2bfloat16_rn(f[j] / (1.0f + __expf(-f[j])) * ex[j * 32 + lane]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) tile[j * OUT_COLS + ew * 32 + lane] = __float2bfloat16_rn(f[j]);
        }
        // Whoever writes a buffer again has passed the barrier of the piece between, which its readers reach when they are
        // done: two buffers and one barrier per piece are enough.
        named_bar_sync(1 + team, EPI_THREADS);
        uint4 v[32 * PER_ROW / EPI_THREADS];
#pragma unroll
        for (int i = 0; i < 32 * PER_ROW / EPI_THREADS; ++i) v[i] = ((const uint4*)tile)[i * EPI_THREADS + et];
        char* dst = p.out + ((size_t)(g.row0 + c + et / PER_ROW) * pitch + col + et % PER_ROW * 8) * 2;
#pragma unroll
        for (int i = 0; i < 32 * PER_ROW / EPI_THREADS; ++i) {
          constexpr int ROWS = EPI_THREADS / PER_ROW;
          if (c + et / PER_ROW + i * ROWS < g.rows) *(uint4*)(dst + (size_t)i * ROWS * pitch * 2) = v[i];
        }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  if (*abort_flag) {
    const uint64_t t0 = timer_ns();  // copies that are still in flight land before the shared memory goes away
    while (timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  if (warp == 2) tmem_dealloc<PAIR ? 2 : 1>(tmem_base, TMEM_COLS);
  if (threadIdx.x == 0 && *abort_flag) atomicOr(p.error_flag, 1);
}

}  // namespace bshmem
