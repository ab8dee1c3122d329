// Expert-parallel MoE dispatch and combine for sm_100a over NVLink peer memory.  What follows is the form for several PEs; one
// PE has kernels without any barrier (see "dispatch on one PE" and combine_kernel with LOCAL).
//
// dispatch (one cooperative kernel, persistent CTAs of 256 threads):
//   A  histogram of the K expert ids of every token (shared-memory bins, then global atomics)
//   B  CTA 0 stores this PE's E counts into row `rank` of every PE's count matrix and runs a
//      cross-PE barrier; a grid barrier releases the other CTAs
//   C  every CTA derives, from the complete [npes, E] matrix, the first row of each expert's
//      segment that belongs to this PE as a source: rows of a receive buffer are ordered by
//      local expert, then by source PE, so the expert GEMMs read contiguous groups
//   D  one CTA per token: the row is staged in shared memory once (and quantised once to fp8 with
//      1x128 fp32 scales when asked), each of its K slots takes the next row of its segment with an
//      atomic cursor, and the row is pushed with 16-byte stores to the owning PE.  With `dup_src` a row
//      crosses NVLink once per destination PE: the first of the token's slots on a PE carries the payload,
//      the others only the number of that row
//   E  grid barrier, then a cross-PE barrier: every PE's rows have landed
//   F  (with `dup_src`) every PE copies the rows that arrived by number from their first row, locally
// combine (one cooperative kernel): cross-PE barrier on entry (expert outputs are final), then one CTA
// per token pulls its K rows with 16-byte loads from the owners, multiplies by the routing weights in
// fp32, rounds once to bf16; a cross-PE barrier on exit lets the owners reuse their buffers.
// All waits are bounded and report through `error_flag`; nothing traps.
// (reference for the capability: examples/moe_shuffle.cu, an fp32 dispatch-only all-to-all-v)
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <limits.h>
#include <string.h>

#include <map>
#include <mutex>
#include <tuple>

#include "../../include/bshmem/moe.h"
#include "../../include/bshmem/tcgen05.cuh"

namespace bshmem {
namespace moe {

constexpr int THREADS = 256;

struct Scratch {                 // local device memory, zeroed by the host before each dispatch
  unsigned int grid_bar;         // arrivals at grid barriers (monotonic within a launch)
  unsigned int pad[63];
  int send_count[BSHMEM_MOE_MAX_EXPERTS];   // pairs this PE sends to each expert
  int cursor[BSHMEM_MOE_MAX_EXPERTS];       // next free position inside my segment of each expert
};

struct DispatchParams {
  bshmem_moe_dispatch_args_t a;
  uint64_t wait_limit_ns;
  int split;  // one PE, small batches: column ranges that a token's row is cut into
};
struct CombineParams {
  bshmem_moe_combine_args_t a;
  uint64_t wait_limit_ns;
  int split;  // one PE: column ranges that a token's row is cut into
};

__device__ __forceinline__ uint64_t timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint64_t ld_acquire_sys_u64(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_acquire_gpu_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier over co-resident CTAs (cooperative launch).  `phase` counts barriers of this launch; the
// counter starts at zero.  Returns false after the wait bound.
__device__ bool grid_barrier(unsigned* counter, unsigned& phase, uint64_t limit_ns, int* error_flag) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++phase;
    __threadfence();
    atomicAdd(counter, 1u);
    const unsigned target = phase * gridDim.x;
    const uint64_t start = timer_ns();
    int ok = 1;
    unsigned spins = 0;
    while (ld_acquire_gpu_u32(counter) < target) {
      if ((++spins & 63) == 0 && timer_ns() - start > limit_ns) {
        atomicOr(error_flag, BSHMEM_MOE_ERRBIT_TIMEOUT);
        ok = 0;
        break;
      }
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// Cross-PE barrier run by the first `npes` threads of one CTA: store `value` into slot `rank` of row
// `row` of every PE's flag block, wait until every slot of my row holds at least `value`.
__device__ bool pe_barrier(uint64_t* const* flags, int row, int rank, int npes, uint64_t value, uint64_t limit_ns, int* error_flag) {
  __shared__ int ok_s;
  if (threadIdx.x == 0) ok_s = 1;
  __syncthreads();
  if ((int)threadIdx.x < npes) {
    const int q = threadIdx.x;
    __threadfence_system();
    if (q != rank) asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(flags[q] + row * npes + rank), "l"(value) : "memory");
    if (q != rank) {
      const uint64_t* mine = flags[rank] + row * npes + q;
      const uint64_t start = timer_ns();
      unsigned spins = 0;
      while (ld_acquire_sys_u64(mine) < value) {
        if ((++spins & 31) == 0) {
          if (timer_ns() - start > limit_ns) {
            atomicOr(error_flag, BSHMEM_MOE_ERRBIT_TIMEOUT);
            ok_s = 0;
            break;
          }
          __nanosleep(64);
        }
      }
    }
  }
  __syncthreads();
  return ok_s != 0;
}

__global__ void __launch_bounds__(THREADS) dispatch_kernel(const __grid_constant__ DispatchParams P) {
  const bshmem_moe_dispatch_args_t& a = P.a;
  extern __shared__ __align__(16) uint8_t smem[];
  const int T = a.T, H = a.H, K = a.K, E = a.E, npes = a.npes, rank = a.rank;
  const int EL = E / npes;
  Scratch* sc = (Scratch*)a.scratch;
  unsigned phase = 0;
  int* s_bins = (int*)smem;                     // [E] histogram bins, later my segment starts; [E] more for totals
  __shared__ int s_row[THREADS], s_dest[THREADS];  // slots of one chunk of tokens: [token in chunk][choice]
  __shared__ int s_first[THREADS];                 // -1: this slot carries the payload; else the row (same PE) that does
  const bool dedup = a.dup_src[rank] != nullptr;

  // ---- A: histogram
  for (int e = threadIdx.x; e < E; e += THREADS) s_bins[e] = 0;
  __syncthreads();
  for (long i = (long)blockIdx.x * THREADS + threadIdx.x; i < (long)T * K; i += (long)gridDim.x * THREADS) {
    const int e = a.topk_idx[i];
    if (e >= 0 && e < E) atomicAdd(&s_bins[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += THREADS)
    if (s_bins[e]) atomicAdd(&sc->send_count[e], s_bins[e]);
  if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;

  // ---- B: publish my counts to every PE, cross-PE barrier
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < E * npes; i += THREADS) {
      const int q = i / E, e = i % E;
      a.counts[q][rank * E + e] = sc->send_count[e];
    }
    __syncthreads();
    pe_barrier(a.flags, 0, rank, npes, a.epoch, P.wait_limit_ns, a.error_flag);
  }
  if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;

  // ---- C: where my rows start on each owner.  Rows of PE d's buffer: for le in [0, EL): for s in [0, npes): count[s][d*EL+le] rows.
  // Per expert: rows from all PEs (s_tot) and rows from the PEs before me (s_bins); then a prefix over
  // the experts of one owner, from shared memory.
  const int* cm = a.counts[rank];
  int* s_tot = s_bins + E;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += THREADS) {
    int tot = 0, pre = 0;
    for (int s = 0; s < npes; ++s) {
      const int c = __ldcg(&cm[s * E + e]);
      tot += c;
      if (s < rank) pre += c;
    }
    s_tot[e] = tot;
    s_bins[e] = pre;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += THREADS) {
    const int first = (e / EL) * EL;
    int start = s_bins[e];
    for (int l2 = first; l2 < e; ++l2) start += s_tot[l2];
    s_bins[e] = start;  // only this thread reads or writes s_bins[e] in this loop
  }
  if (blockIdx.x == 0) {  // receiver-side description of my own buffer
    for (int le = threadIdx.x; le <= EL; le += THREADS) {
      int start = 0;
      for (int l2 = 0; l2 < le; ++l2) start += s_tot[rank * EL + l2];
      a.expert_offsets[le] = start;
      if (le < EL && a.src_offsets) {
        int run = start;
        for (int s = 0; s < npes; ++s) {
          a.src_offsets[le * npes + s] = run;
          run += __ldcg(&cm[s * E + rank * EL + le]);
        }
      }
    }
  }

  // ---- D: push rows.  The slots of a whole chunk of this CTA's tokens are claimed first (one atomic per
  // (token, choice) pair, all in flight together); after that each token moves from global memory through
  // registers to its K destinations with no CTA-wide synchronisation, so that the loads of one token
  // overlap the stores of the one before.
  const int row_bytes = a.payload == BSHMEM_MOE_FP8_E4M3 ? H : H * 2;
  const int nscale = H / BSHMEM_MOE_QUANT_BLOCK;
  const int per_chunk = THREADS / K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int base = 0; (long)blockIdx.x + (long)base * gridDim.x < T; base += per_chunk) {
    __syncthreads();  // the previous chunk's slots are no longer read (and s_bins is final on the first pass)
    {
      const int i = threadIdx.x / K, k = threadIdx.x % K;
      const long t = (long)blockIdx.x + (long)(base + i) * gridDim.x;
      if (i < per_chunk && t < T) {
        const int e = a.topk_idx[(size_t)t * K + k];
        int row = -1, dest = 0;
        if (e >= 0 && e < E) {
          const int pos = atomicAdd(&sc->cursor[e], 1);
          row = s_bins[e] + pos;
          dest = e / EL;
          if (row >= a.cap_rows) {
            atomicOr(a.error_flag, BSHMEM_MOE_ERRBIT_OVERFLOW);
            row = -1;
          }
        }
        s_row[i * K + k] = row;
        s_dest[i * K + k] = dest;
        a.slot_map[(size_t)t * K + k] = row;
      }
    }
    __syncthreads();
    {
      // Which slot of the token carries the payload to each destination PE: the first valid one.
      const int i = threadIdx.x / K, k = threadIdx.x % K;
      const long t = (long)blockIdx.x + (long)(base + i) * gridDim.x;
      if (i < per_chunk && t < T) {
        int first = -1;
        const int row = s_row[i * K + k], dest = s_dest[i * K + k];
        if (dedup && row >= 0) {
          for (int j = 0; j < k; ++j)
            if (s_row[i * K + j] >= 0 && s_dest[i * K + j] == dest) { first = s_row[i * K + j]; break; }
          a.dup_src[dest][row] = first;  // every row is written by its sender: -1 = payload follows, else copy from `first`
        }
        s_first[i * K + k] = first;
      }
    }
    __syncthreads();
    for (int i = 0; i < per_chunk; ++i) {
      const long t = (long)blockIdx.x + (long)(base + i) * gridDim.x;
      if (t >= T) break;
      const int* rows = s_row + i * K;
      const int* dests = s_dest + i * K;
      const int* firsts = s_first + i * K;
      if (a.payload == BSHMEM_MOE_FP8_E4M3) {
        // Eight lanes per 128-value block, 16 values per lane: a warp quantises four blocks at a time and
        // stores 16 bytes per lane (512 contiguous bytes per warp and destination).  absmax over the eight
        // lanes by shuffles, scale = amax / 448.  Two rounds of loads are in flight before the first store.
        const uint4* xrow = (const uint4*)a.x + (size_t)t * (H / 8);
        constexpr int WARPS = THREADS / 32;
        const int sub = lane >> 3, part = lane & 7;  // block within the warp's four, 16-value piece within the block
        const int ngroups = (nscale + 3) / 4;
        for (int q0 = warp; q0 < ngroups; q0 += 2 * WARPS) {
          uint4 raw[2][2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int g = (q0 + u * WARPS) * 4 + sub;
            if (q0 + u * WARPS < ngroups && g < nscale) {
              raw[u][0] = xrow[g * 16 + part * 2];
              raw[u][1] = xrow[g * 16 + part * 2 + 1];
            } else {
              raw[u][0] = raw[u][1] = make_uint4(0u, 0u, 0u, 0u);
            }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (q0 + u * WARPS >= ngroups) break;  // uniform over the warp
            const int g = (q0 + u * WARPS) * 4 + sub;
            float f[16];
            const __nv_bfloat162* h = (const __nv_bfloat162*)raw[u];
            float amax = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float2 v = __bfloat1622float2(h[e]);
              f[2 * e] = v.x;
              f[2 * e + 1] = v.y;
              amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            const float scale = fmaxf(amax, 1e-10f) / 448.0f;
            const float inv = 1.0f / scale;
            uint4 q16;
            uint32_t* qw = (uint32_t*)&q16;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * e] * inv, f[4 * e + 1] * inv), __NV_SATFINITE, __NV_E4M3);
              const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * e + 2] * inv, f[4 * e + 3] * inv), __NV_SATFINITE, __NV_E4M3);
              qw[e] = (uint32_t)lo | ((uint32_t)hi << 16);
            }
            if (g < nscale) {
              for (int j = 0; j < K; ++j) {
                const int row = rows[j];
                if (row < 0 || firsts[j] >= 0) continue;
                ((uint4*)((uint8_t*)a.recv_x[dests[j]] + (size_t)row * row_bytes))[g * 8 + part] = q16;
                if (part == 0) a.recv_scale[dests[j]][(size_t)row * nscale + g] = scale;
              }
            }
          }
        }
      } else {
        const uint4* xrow = (const uint4*)a.x + (size_t)t * (H / 8);
        const int nvec = H / 8;
        for (int c0 = threadIdx.x; c0 < nvec; c0 += 4 * THREADS) {
          uint4 v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c0 + u * THREADS < nvec) v[u] = xrow[c0 + u * THREADS];
          for (int j = 0; j < K; ++j) {
            const int row = rows[j];
            if (row < 0 || firsts[j] >= 0) continue;
            uint4* dst = (uint4*)((uint8_t*)a.recv_x[dests[j]] + (size_t)row * row_bytes);
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (c0 + u * THREADS < nvec) dst[c0 + u * THREADS] = v[u];
          }
        }
      }
    }
  }

  // ---- E: all my rows are out; meet every PE
  if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;
  if (blockIdx.x == 0) pe_barrier(a.flags, 1, rank, npes, a.epoch, P.wait_limit_ns, a.error_flag);
  if (!dedup) return;

  // ---- F: rows that arrived as a row number are copied from that row (always a payload row), locally
  if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;
  int total = 0;
  for (int le = 0; le < EL; ++le) total += s_tot[rank * EL + le];
  if (total > a.cap_rows) total = a.cap_rows;
  const int* dup = a.dup_src[rank];
  uint8_t* mine = (uint8_t*)a.recv_x[rank];
  const int nvec = row_bytes / 16;
  for (int r = blockIdx.x; r < total; r += gridDim.x) {
    const int from = __ldcg(dup + r);
    if (from < 0 || from >= total) continue;
    const uint4* src = (const uint4*)(mine + (size_t)from * row_bytes);
    uint4* dst = (uint4*)(mine + (size_t)r * row_bytes);
    for (int c = threadIdx.x; c < nvec; c += THREADS) dst[c] = __ldcg(src + c);
    if (a.payload == BSHMEM_MOE_FP8_E4M3)
      for (int g = threadIdx.x; g < nscale; g += THREADS) a.recv_scale[rank][(size_t)r * nscale + g] = __ldcg(&a.recv_scale[rank][(size_t)from * nscale + g]);
  }
}

// Weighted sum of up to KT expert rows into one output row.  Row pointers and weights sit in registers;
// for every 16-byte column block the KT loads are issued before the first is consumed.
template <int KT>
__device__ __forceinline__ void combine_token(const uint8_t* const* src, const float* wt, int K, uint4* out_row, int c_first, int c_end, const int c_step) {
  const uint4* p[KT];
  float w[KT];
#pragma unroll
  for (int j = 0; j < KT; ++j) {
    const bool on = j < K && src[j] != nullptr;
    p[j] = on ? (const uint4*)src[j] : nullptr;
    w[j] = on ? wt[j] : 0.f;
  }
  for (int c = c_first; c < c_end; c += c_step) {
    uint4 v[KT];
#pragma unroll
    for (int j = 0; j < KT; ++j) v[j] = p[j] ? p[j][c] : make_uint4(0u, 0u, 0u, 0u);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < KT; ++j) {
      const __nv_bfloat162* h = (const __nv_bfloat162*)&v[j];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = __bfloat1622float2(h[q]);
        acc[2 * q] += w[j] * f.x;
        acc[2 * q + 1] += w[j] * f.y;
      }
    }
    uint4 o;
    __nv_bfloat162* oh = (__nv_bfloat162*)&o;
#pragma unroll
    for (int q = 0; q < 4; ++q) oh[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
    out_row[c] = o;
  }
}

// LOCAL (one PE): nobody to meet on entry or exit, so no barrier, no cooperative launch and no cleared counter; the work items
// are `split` column ranges of every token, so that a decode batch of few tokens still fills the SMs.  Bound by HBM reads.
// H 7168, top-8: 4096 tokens 88 -> 82 us (6.4 TB/s), 64 tokens 13 -> 6.7 us;
// H 128, top-4, 16364 tokens: 36.6 -> 6.7 us.
// NARROW: rows (or column ranges) of at most half as many 16-byte pieces as the CTA has threads are taken several at a time,
// a power of two of threads each; a build of its own because the variable stride costs wide rows 3 %.
// The bound of one CTA more per SM is for LOCAL alone, where it was measured; the others keep the registers that hold their loads in
// flight (62 and 85, against 54 and 79; 4096 tokens of 128 values, top-8, on one PE 24.5 us against 26.6).
template <int KT, bool LOCAL, bool NARROW>
__global__ void __launch_bounds__(THREADS, (KT <= 8 ? 3 : 2) + (LOCAL ? 1 : 0)) combine_kernel(const __grid_constant__ CombineParams P) {
  const bshmem_moe_combine_args_t& a = P.a;
  const int H = a.H, K = a.K, E = a.E, npes = a.npes, rank = a.rank;
  const int EL = E / npes;
  const int split = LOCAL ? P.split : 1, nvec = H / 8;
  const long items = (long)a.T * split;
  Scratch* sc = (Scratch*)a.scratch;
  unsigned phase = 0;
  __shared__ const uint8_t* s_src[THREADS];  // one chunk of this CTA's items: [item in chunk][choice]
  __shared__ float s_w[THREADS];
  if (!LOCAL) {
    if (blockIdx.x == 0) pe_barrier(a.flags, 2, rank, npes, a.epoch, P.wait_limit_ns, a.error_flag);
    if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;
  }
  const int per_chunk = THREADS / K;
  int lanes = THREADS;
  if (NARROW) {
    const int per_item = (nvec + split - 1) / split;
    lanes = 16;  // H is a multiple of 128: 16 pieces at least
    while (lanes < per_item) lanes *= 2;
  }
  for (int base = 0; (long)blockIdx.x + (long)base * gridDim.x < items; base += per_chunk) {
    __syncthreads();
    {
      // Sources and weights of a whole chunk of items are looked up at once, so that the loop below runs without
      // CTA-wide synchronisation.
      const int i = threadIdx.x / K, k = threadIdx.x % K;
      const long it = (long)blockIdx.x + (long)(base + i) * gridDim.x;
      if (i < per_chunk && it < items) {
        const size_t t = (size_t)(it / split);
        const int e = a.topk_idx[t * K + k];
        const int row = a.slot_map[t * K + k];
        const bool ok = e >= 0 && e < E && row >= 0;
        s_src[i * K + k] = ok ? (const uint8_t*)a.y[e / EL] + (size_t)row * H * 2 : nullptr;
        s_w[i * K + k] = ok ? a.topk_weight[t * K + k] : 0.f;
      }
    }
    __syncthreads();
    for (int i = NARROW ? (int)threadIdx.x / lanes : 0; i < per_chunk; i += NARROW ? THREADS / lanes : 1) {
      const long it = (long)blockIdx.x + (long)(base + i) * gridDim.x;
      if (it >= items) break;
      const long t = split == 1 ? it : it / split;
      const int part = (int)(it - t * split);
      uint4* out_row = (uint4*)a.out + (size_t)t * nvec;
      combine_token<KT>(s_src + i * K, s_w + i * K, K, out_row, nvec * part / split + (NARROW ? (int)threadIdx.x % lanes : (int)threadIdx.x), nvec * (part + 1) / split, NARROW ? lanes : THREADS);
    }
  }
  if (LOCAL) return;
  if (!grid_barrier(&sc->grid_bar, phase, P.wait_limit_ns, a.error_flag)) return;
  if (blockIdx.x == 0) pe_barrier(a.flags, 3, rank, npes, a.epoch, P.wait_limit_ns, a.error_flag);
}

// ------------------------------------------------------------------ dispatch on one PE
// With one PE there is nobody to exchange counts with, so the three grid barriers, the cleared counters and the cooperative
// launch of dispatch_kernel are pure latency (about 25 us of 112 for 4096 tokens, all of the 16 us for 64).  Two forms:
//  * up to LOCAL_SMALL_PAIRS (token, choice) pairs: one kernel; every CTA counts all pairs itself in shared memory (8 KB from
//    L2) and finds the place of its own token's rows by counting the equal ids before them;
//  * more: a routing kernel (one cluster of eight CTAs, counts met through distributed shared memory) writes the slot map and
//    the offsets, then a kernel that only moves rows.
// The line lies at 2048 pairs because every item of the one kernel scans the pairs before it.  One kernel / two, us: 7168 values, top-8 of
// 256, bf16: 1024 pairs 7.0 / 8.1, 2048 9.0 / 11.0, 4096 14.5 / 15.7, 8192 31.4 / 25.2; fp8: 2048 7.9 / 9.5, 4096 12.2 / 11.3; 1024 values:
// 2048 6.2 / 7.4, 4096 8.3 / 7.6; 512 values, top-16 of 64: 2048 5.5 / 7.2, 3072 7.7 / 7.0.
// Routing CTAs: eight is the largest cluster that needs no opt-in; 8192 tokens of 128 values, fp8, top-8: 11.7 us with eight, 16.4 with
// four, 26.0 with two.
// Device time, 64 tokens x 7168, top-8 of 256: 16.5 us before, 7 us now; 4096 tokens: bf16 112 us -> 6.3 (routing) + 91
// (529 MB, 5.8 TB/s), fp8 79.6 us -> 6.5 + 51.5 (5.8 TB/s), bound by HBM writes.  The row kernel is launched early and loads
// token rows while the routing runs (2.5 us less).
constexpr int LOCAL_SMALL_PAIRS = 2048, ROUTE_CTAS = 8, ROUTE_THREADS = 1024;

// Exclusive prefix sum of s_val[0, n) in place, n <= 4 * NT; all NT threads call it.  Returns the total.
template <int NT>
__device__ __forceinline__ int block_exclusive_scan(int* s_val, int n) {
  __shared__ int s_warp[NT / 32 + 1];
  const int per = (n + NT - 1) / NT, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = threadIdx.x * per;
  int sum = 0;
  for (int i = first; i < first + per && i < n; ++i) sum += s_val[i];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp + 1] = incl;
  if (threadIdx.x == 0) s_warp[0] = 0;
  __syncthreads();
  if (warp == 0) {
    int w = lane < NT / 32 ? s_warp[lane + 1] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    if (lane < NT / 32) s_warp[lane + 1] = w;
  }
  __syncthreads();
  int run = s_warp[warp] + incl - sum;
  for (int i = first; i < first + per && i < n; ++i) {
    const int v = s_val[i];
    s_val[i] = run;
    run += v;
  }
  __syncthreads();
  return s_warp[NT / 32];
}

__device__ __forceinline__ int local_row(const bshmem_moe_dispatch_args_t& a, int row) {
  if (row < a.cap_rows) return row;
  atomicOr(a.error_flag, BSHMEM_MOE_ERRBIT_OVERFLOW);
  return -1;
}
// Receiver-side description of the buffer and this PE's row of the count matrix; s_start[0, E) and the total are final.
__device__ __forceinline__ void local_offsets(const bshmem_moe_dispatch_args_t& a, const int* s_start, int total, int nthreads) {
  for (int e = threadIdx.x; e <= a.E; e += nthreads) {
    const int start = e < a.E ? s_start[e] : total;
    a.expert_offsets[e] = start;
    if (e < a.E) {
      if (a.src_offsets) a.src_offsets[e] = start;
      a.counts[0][e] = (e + 1 < a.E ? s_start[e + 1] : total) - start;
    }
  }
}

// A warp's share of a quantised row: 16 of the 512 values that start at value 512 * q (eight lanes per 128-value block).
struct Fp8Piece {
  uint4 raw[2];
  __device__ __forceinline__ void load(const bshmem_moe_dispatch_args_t& a, long t, int q, int lane) {
    const int g = q * 4 + (lane >> 3);
    const uint4* x = (const uint4*)a.x + (size_t)t * (a.H / 8) + g * 16 + (lane & 7) * 2;
    const bool in = g < a.H / BSHMEM_MOE_QUANT_BLOCK;
    raw[0] = in ? __ldg(x) : make_uint4(0u, 0u, 0u, 0u);
    raw[1] = in ? __ldg(x + 1) : make_uint4(0u, 0u, 0u, 0u);
  }
  // absmax over the eight lanes of a block, scale = amax / 448, values rounded to e4m3
  __device__ __forceinline__ uint4 quantise(float* scale_out) const {
    float f[16], amax = 0.f;
    const __nv_bfloat162* h = (const __nv_bfloat162*)raw;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float2 v = __bfloat1622float2(h[e]);
      f[2 * e] = v.x;
      f[2 * e + 1] = v.y;
      amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float scale = fmaxf(amax, 1e-10f) / 448.0f;
    const float inv = 1.0f / scale;
    uint4 q16;
    uint32_t* qw = (uint32_t*)&q16;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * e] * inv, f[4 * e + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * e + 2] * inv, f[4 * e + 3] * inv), __NV_SATFINITE, __NV_E4M3);
      qw[e] = (uint32_t)lo | ((uint32_t)hi << 16);
    }
    *scale_out = scale;
    return q16;
  }
  __device__ __forceinline__ void store(const bshmem_moe_dispatch_args_t& a, int row, int q, int lane, uint4 q16, float scale) const {
    const int g = q * 4 + (lane >> 3), nscale = a.H / BSHMEM_MOE_QUANT_BLOCK;
    if (row < 0 || g >= nscale) return;
    ((uint4*)((uint8_t*)a.recv_x[0] + (size_t)row * a.H))[g * 8 + (lane & 7)] = q16;
    if ((lane & 7) == 0) a.recv_scale[0][(size_t)row * nscale + g] = scale;
  }
};

// Small batches.  Work items are `split` column ranges (whole groups of 512 values) of every token.
template <bool FP8>
__global__ void __launch_bounds__(THREADS) dispatch_small_kernel(const __grid_constant__ DispatchParams P) {
  const bshmem_moe_dispatch_args_t& a = P.a;
  const int K = a.K, E = a.E, pairs = a.T * K, split = P.split;
  __shared__ short s_id[LOCAL_SMALL_PAIRS];
  __shared__ int s_start[BSHMEM_MOE_MAX_EXPERTS], s_row[BSHMEM_MOE_MAX_TOPK];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += THREADS) s_start[e] = 0;
  __syncthreads();
#pragma unroll 8
  for (int i = threadIdx.x; i < pairs; i += THREADS) {
    const int e = a.topk_idx[i];
    const bool ok = e >= 0 && e < E;
    s_id[i] = ok ? (short)e : (short)-1;
    if (ok) atomicAdd(&s_start[e], 1);
  }
  __syncthreads();
  const int total = block_exclusive_scan<THREADS>(s_start, E);
  if (blockIdx.x == 0) local_offsets(a, s_start, total, THREADS);
  const int groups = (a.H + 511) / 512;
  for (long item = blockIdx.x; item < (long)a.T * split; item += gridDim.x) {
    const int t = (int)(item / split), part = (int)(item - (long)t * split);
    const int g0 = (int)((long)groups * part / split), g1 = (int)((long)groups * (part + 1) / split);
    __syncthreads();  // the rows of the item before are no longer read
    for (int k = warp; k < K; k += THREADS / 32) {
      const int i = t * K + k, e = s_id[i];
      int before = 0;
      for (int j = lane; j < i; j += 32) before += s_id[j] == e;
      before = (int)__reduce_add_sync(0xffffffffu, (unsigned)before);
      if (lane == 0) {
        const int row = e < 0 ? -1 : local_row(a, s_start[e] + before);
        s_row[k] = row;
        if (part == 0) a.slot_map[i] = row;
      }
    }
    __syncthreads();
    if (FP8) {
      for (int q = g0 + warp; q < g1; q += THREADS / 32) {
        Fp8Piece piece;
        piece.load(a, t, q, lane);
        float scale;
        const uint4 q16 = piece.quantise(&scale);
        for (int k = 0; k < K; ++k) piece.store(a, s_row[k], q, lane, q16, scale);
      }
    } else {
      const int nvec = a.H / 8, c1 = min(nvec, g1 * 64);
      const uint4* x = (const uint4*)a.x + (size_t)t * nvec;
      for (int c = g0 * 64 + threadIdx.x; c < c1; c += THREADS) {
        const uint4 v = __ldg(x + c);
        for (int k = 0; k < K; ++k)
          if (s_row[k] >= 0) ((uint4*)a.recv_x[0])[(size_t)s_row[k] * nvec + c] = v;
      }
    }
  }
}

// Routing of a large batch: the CTAs of one cluster (ROUTE_CTAS, or fewer where the caller allows fewer) take contiguous parts of the
// pairs.  A pair's place among its CTA's pairs of the same expert comes from a shared-memory counter and waits in slot_map until the
// starts are known.
__global__ void __launch_bounds__(ROUTE_THREADS) route_kernel(const __grid_constant__ DispatchParams P) {
  namespace cg = cooperative_groups;
  const bshmem_moe_dispatch_args_t& a = P.a;
  cg::cluster_group cluster = cg::this_cluster();
  // The kernel that moves the rows may start now: it loads token rows (which nothing here writes) and waits for this grid
  // to end before it reads the slot map.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int me = (int)cluster.block_rank(), ctas = (int)cluster.num_blocks(), E = a.E;
  __shared__ int s_count[BSHMEM_MOE_MAX_EXPERTS], s_start[BSHMEM_MOE_MAX_EXPERTS];
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) s_count[e] = 0;
  __syncthreads();
  const long pairs = (long)a.T * a.K, per = (pairs + ctas - 1) >> (__ffs(ctas) - 1);  // a power of two
  const long lo = min(pairs, per * me), hi = min(pairs, per * (me + 1));
  // The first ROUTE_HELD pairs of a thread stay in registers (all of a batch of 8192 tokens x 8), the rest goes by way of slot_map.
  constexpr int ROUTE_HELD = 8;
  int held_e[ROUTE_HELD], held_pos[ROUTE_HELD];
#pragma unroll
  for (int h = 0; h < ROUTE_HELD; ++h) {
    const long i = lo + threadIdx.x + (long)h * ROUTE_THREADS;
    held_e[h] = i < hi ? a.topk_idx[i] : -1;
  }
#pragma unroll
  for (int h = 0; h < ROUTE_HELD; ++h) held_pos[h] = held_e[h] >= 0 && held_e[h] < E ? atomicAdd(&s_count[held_e[h]], 1) : -1;
  const long rest = lo + threadIdx.x + (long)ROUTE_HELD * ROUTE_THREADS;
#pragma unroll 4
  for (long i = rest; i < hi; i += ROUTE_THREADS) {
    const int e = a.topk_idx[i];
    a.slot_map[i] = e >= 0 && e < E ? atomicAdd(&s_count[e], 1) : -1;
  }
  cluster.sync();
  int before = 0, mine = 0;  // pairs of expert `threadIdx.x` (E <= ROUTE_THREADS) in the CTAs before me, and in all
  if ((int)threadIdx.x < E) {
#pragma unroll
    for (int c = 0; c < ROUTE_CTAS; ++c) {
      const int v = c < ctas ? *cluster.map_shared_rank(&s_count[threadIdx.x], c) : 0;
      if (c < me) before += v;
      mine += v;
    }
    s_start[threadIdx.x] = mine;
  }
  __syncthreads();
  const int total = block_exclusive_scan<ROUTE_THREADS>(s_start, E);
  if (me == 0) local_offsets(a, s_start, total, ROUTE_THREADS);
  cluster.sync();  // nobody reads the counts, or the starts, any more
  if ((int)threadIdx.x < E) s_start[threadIdx.x] += before;
  __syncthreads();
#pragma unroll
  for (int h = 0; h < ROUTE_HELD; ++h) {
    const long i = lo + threadIdx.x + (long)h * ROUTE_THREADS;
    if (i < hi) a.slot_map[i] = held_pos[h] >= 0 ? local_row(a, s_start[held_e[h]] + held_pos[h]) : -1;
  }
#pragma unroll 4
  for (long i = rest; i < hi; i += ROUTE_THREADS) {
    const int e = a.topk_idx[i];
    if (e >= 0 && e < E) a.slot_map[i] = local_row(a, s_start[e] + a.slot_map[i]);
  }
}
static_assert(BSHMEM_MOE_MAX_EXPERTS <= ROUTE_THREADS, "one thread per expert");

// Rows of a large batch, bf16: every warp runs a ring of PUSH_DEPTH shared-memory buffers that the bulk-copy engine fills
// from a piece of a token's row and empties into the K receive rows, lane k issuing the copy to row k: no register or
// load / store unit touches the data, and one load feeds K stores.
// 4096 tokens of 7168 / 512 values, top-8, us with the routing: 4 warps x 4 buffers of 4 KB 96.5 / 12.0, of 2 KB 97.1 / 11.8, of 8 KB
// 96.4 / 12.7, 8 warps of 2 KB 97.3 / 12.7.
constexpr int PUSH_WARPS = 4, PUSH_DEPTH = 4, PUSH_BYTES = 4096;
constexpr int PUSH_SMEM = PUSH_WARPS * PUSH_DEPTH * PUSH_BYTES;

__global__ void __launch_bounds__(PUSH_WARPS * 32) push_rows_kernel(const __grid_constant__ DispatchParams P) {
  using namespace sm100;
  const bshmem_moe_dispatch_args_t& a = P.a;
  extern __shared__ __align__(128) uint8_t ring_all[];
  __shared__ uint64_t s_full[PUSH_WARPS][PUSH_DEPTH];
  __shared__ int s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* ring = ring_all + warp * PUSH_DEPTH * PUSH_BYTES;
  uint64_t* full = s_full[warp];
  if (threadIdx.x == 0) s_abort = 0;
  if (lane == 0) {
    for (int d = 0; d < PUSH_DEPTH; ++d) mbar_init(&full[d], 1);
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  __syncthreads();
  const int row_bytes = a.H * 2, pieces = (row_bytes + PUSH_BYTES - 1) / PUSH_BYTES;
  // even pieces, a multiple of 16 bytes; rows of many pieces keep whole buffers, so that the last piece is never empty
  const int piece_bytes = pieces <= 64 ? ((row_bytes + pieces - 1) / pieces + 15) & ~15 : PUSH_BYTES;
  const long items = (long)a.T * pieces, step = (long)gridDim.x * PUSH_WARPS;
  const long first = (long)blockIdx.x * PUSH_WARPS + warp;
  int rows[PUSH_DEPTH];
  auto fill = [&](int d, long item) {  // starts the load of `item` into buffer d; find() fetches its receive rows
    if (item >= items) return;
    const long t = item / pieces;
    const int off = (int)(item - t * pieces) * piece_bytes, n = min(piece_bytes, row_bytes - off);
    if (lane == 0) {
      mbar_expect_tx(&full[d], n);
      bulk_load(ring + d * PUSH_BYTES, (const uint8_t*)a.x + (size_t)t * row_bytes + off, n, &full[d]);
    }
  };
  auto find = [&](int d, long item) { rows[d] = item < items && lane < a.K ? __ldcg(a.slot_map + item / pieces * a.K + lane) : -1; };
#pragma unroll
  for (int d = 0; d < PUSH_DEPTH - 1; ++d) fill(d, first + d * step);
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the slot map is complete
#pragma unroll
  for (int d = 0; d < PUSH_DEPTH - 1; ++d) find(d, first + d * step);
  uint32_t parity = 0;
  bool ok = true;
  for (long item = first; item < items && ok; parity ^= 1) {
#pragma unroll
    for (int d = 0; d < PUSH_DEPTH; ++d, item += step) {
      if (item >= items) break;
      ok = mbar_wait(&full[d], parity, P.wait_limit_ns, &s_abort);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const long t = item / pieces;
      const int off = (int)(item - t * pieces) * piece_bytes, n = min(piece_bytes, row_bytes - off);
      if (rows[d] >= 0) bulk_store((uint8_t*)a.recv_x[0] + (size_t)rows[d] * row_bytes + off, ring + d * PUSH_BYTES, n);
      bulk_commit();
      // The buffer before this one was emptied by the copies of the previous item: all but the newest group have been read.
      bulk_wait_read<1>();
      __syncwarp();
      fill((d + PUSH_DEPTH - 1) % PUSH_DEPTH, item + (PUSH_DEPTH - 1) * step);
      find((d + PUSH_DEPTH - 1) % PUSH_DEPTH, item + (PUSH_DEPTH - 1) * step);
    }
  }
  bulk_wait<0>();  // the sources stay in place until the copies are complete
  if (!ok) {
    if (lane == 0) atomicOr(a.error_flag, BSHMEM_MOE_ERRBIT_TIMEOUT);
    const uint64_t t0 = timer_ns();  // loads still in flight land before the shared memory goes away
    while (timer_ns() - t0 < 200000) __nanosleep(1000);
  }
}

// Rows of a large batch, fp8: a warp takes 512 values of a token, with the loads of the next item in flight.
__global__ void __launch_bounds__(THREADS) push_rows_fp8_kernel(const __grid_constant__ DispatchParams P) {
  const bshmem_moe_dispatch_args_t& a = P.a;
  const int groups = (a.H + 511) / 512, K = a.K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long items = (long)a.T * groups, step = (long)gridDim.x * (THREADS / 32);
  long item = (long)blockIdx.x * (THREADS / 32) + warp;
  if (item >= items) return;
  Fp8Piece next;
  int next_row;
  auto fetch = [&](long it) {
    const long t = it / groups;
    next.load(a, t, (int)(it - t * groups), lane);
  };
  auto find = [&](long it) { next_row = lane < K ? __ldcg(a.slot_map + it / groups * K + lane) : -1; };
  fetch(item);
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the slot map is complete
  find(item);
  for (; item < items; item += step) {
    const Fp8Piece piece = next;
    const int my_row = next_row, q = (int)(item % groups);
    if (item + step < items) {
      fetch(item + step);
      find(item + step);
    }
    float scale;
    const uint4 q16 = piece.quantise(&scale);
    for (int k = 0; k < K; ++k) piece.store(a, __shfl_sync(0xffffffffu, my_row, k), q, lane, q16, scale);
  }
}

static size_t dispatch_smem(int E, int) { return (size_t)E * 8 + 16; }  // two int arrays of E entries; rows go through registers

// CTAs of a kernel that are co-resident on the current GPU, 0 on an error.  Asked once per kernel, launch shape and GPU: the
// driver's answer takes longer than the rest of a small launch.
static int resident_ctas(const void* k, size_t smem, int threads) {
  static std::mutex mutex;
  static std::map<std::tuple<const void*, size_t, int, int>, int> known;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mutex);
  int& n = known[std::make_tuple(k, smem, threads, dev)];
  if (n) return n;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem) != cudaSuccess) return 0;
  return n = per_sm * sms;
}
// Grid: as many CTAs as are co-resident (what a cooperative launch allows), at most `want`.
template <class Kernel>
static int coop_grid(Kernel k, size_t smem, int want, int max_ctas, int* grid_out, int threads = THREADS) {
  int grid = resident_ctas((const void*)k, smem, threads);
  if (grid < 1) return BSHMEM_MOE_ERR_DRIVER;
  if (grid > want) grid = want;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  if (grid < 1) grid = 1;
  *grid_out = grid;
  return 0;
}

// Column ranges per token so that few tokens still give every SM about two CTAs; at most one per piece of the row.
static int column_split(int T, int pieces) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int want = (2 * sms + T - 1) / T;
  return want < 1 ? 1 : want > pieces ? pieces : want;
}
static int launched(const char* what, cudaError_t e) {
  if (e == cudaSuccess) return BSHMEM_MOE_OK;
  fprintf(stderr, "%s: launch failed: %s\n", what, cudaGetErrorString(e));
  return BSHMEM_MOE_ERR_DRIVER;
}
// P.a is checked; one PE, no dup_src.
static int dispatch_local(DispatchParams& P, cudaStream_t stream) {
  const bshmem_moe_dispatch_args_t& a = P.a;
  const bool fp8 = a.payload == BSHMEM_MOE_FP8_E4M3;
  const int groups = (a.H + 511) / 512;
  int grid = 0, st;
  if ((long)a.T * a.K <= LOCAL_SMALL_PAIRS) {
    P.split = column_split(a.T, groups);
    auto kernel = fp8 ? dispatch_small_kernel<true> : dispatch_small_kernel<false>;
    st = coop_grid(kernel, 0, a.T * P.split, a.max_ctas, &grid);
    if (st) return st;
    kernel<<<grid, THREADS, 0, stream>>>(P);
    return launched("bshmem_moe_dispatch", cudaGetLastError());
  }
  // `max_ctas` holds for the call: a smaller cluster routes, and the rows wait for it instead of running beside it.
  int ctas = ROUTE_CTAS;
  while (a.max_ctas > 0 && ctas > a.max_ctas) ctas /= 2;
  cudaLaunchConfig_t route = {};
  route.gridDim = dim3(ctas);
  route.blockDim = dim3(ROUTE_THREADS);
  route.stream = stream;
  cudaLaunchAttribute cluster[1];
  cluster[0].id = cudaLaunchAttributeClusterDimension;
  cluster[0].val.clusterDim.x = ctas;
  cluster[0].val.clusterDim.y = cluster[0].val.clusterDim.z = 1;
  route.attrs = cluster;
  route.numAttrs = 1;
  st = launched("bshmem_moe_dispatch", cudaLaunchKernelEx(&route, route_kernel, P));
  if (st) return st;
  const long pieces = (a.H * 2l + PUSH_BYTES - 1) / PUSH_BYTES;
  const int threads = fp8 ? THREADS : PUSH_WARPS * 32;
  const size_t smem = fp8 ? 0 : PUSH_SMEM;
  const long items = ((long)a.T * (fp8 ? groups : pieces) + threads / 32 - 1) / (threads / 32);
  auto kernel = fp8 ? push_rows_fp8_kernel : push_rows_kernel;
  st = coop_grid(kernel, smem, (int)(items < INT_MAX ? items : INT_MAX), a.max_ctas, &grid, threads);
  if (st) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.max_ctas > 0 ? 0 : 1;
  return launched("bshmem_moe_dispatch", cudaLaunchKernelEx(&cfg, kernel, P));
}

}  // namespace moe
}  // namespace bshmem

using namespace bshmem::moe;

extern "C" size_t bshmem_moe_scratch_bytes(int) { return sizeof(Scratch); }

static int check_common(int T, int H, int K, int E, int rank, int npes) {
  if (npes < 1 || npes > BSHMEM_MOE_MAX_PES || rank < 0 || rank >= npes) return BSHMEM_MOE_ERR_ARGS;
  if (T <= 0 || K < 1 || K > BSHMEM_MOE_MAX_TOPK || E < npes || E > BSHMEM_MOE_MAX_EXPERTS || E % npes) return BSHMEM_MOE_ERR_SHAPE;
  if (H <= 0 || H % BSHMEM_MOE_QUANT_BLOCK) return BSHMEM_MOE_ERR_SHAPE;  // rows are moved in 16-byte pieces and quantised in blocks of 128
  return 0;
}

// `general`: the kernel for several PEs also with one.
static int dispatch(const bshmem_moe_dispatch_args_t* a, bool general, cudaStream_t stream) {
  if (!a || !a->x || !a->topk_idx || !a->slot_map || !a->expert_offsets || !a->scratch || !a->error_flag) return BSHMEM_MOE_ERR_ARGS;
  int st = check_common(a->T, a->H, a->K, a->E, a->rank, a->npes);
  if (st) return st;
  for (int q = 0; q < a->npes; ++q)
    if (!a->recv_x[q] || !a->counts[q] || !a->flags[q] || (a->payload == BSHMEM_MOE_FP8_E4M3 && !a->recv_scale[q])) return BSHMEM_MOE_ERR_ARGS;
  DispatchParams P;
  P.a = *a;
  P.wait_limit_ns = a->wait_limit_ms ? (uint64_t)a->wait_limit_ms * 1000000ull : 10000000000ull;
  if (a->npes == 1 && !a->dup_src[0] && !general) return dispatch_local(P, stream);
  const size_t smem = dispatch_smem(a->E, a->H);
  int grid = 0;
  st = coop_grid(dispatch_kernel, smem, a->T, a->max_ctas, &grid);
  if (st) return st;
  if (cudaMemsetAsync(a->scratch, 0, sizeof(Scratch), stream) != cudaSuccess) return BSHMEM_MOE_ERR_DRIVER;
  void* params[] = {(void*)&P};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)dispatch_kernel, dim3(grid), dim3(THREADS), params, smem, stream);
  if (e != cudaSuccess) {
    fprintf(stderr, "bshmem_moe_dispatch: launch failed: %s\n", cudaGetErrorString(e));
    return BSHMEM_MOE_ERR_DRIVER;
  }
  return 0;
}

static int combine(const bshmem_moe_combine_args_t* a, bool general, cudaStream_t stream) {
  if (!a || !a->topk_idx || !a->topk_weight || !a->slot_map || !a->out || !a->scratch || !a->error_flag) return BSHMEM_MOE_ERR_ARGS;
  int st = check_common(a->T, a->H, a->K, a->E, a->rank, a->npes);
  if (st) return st;
  for (int q = 0; q < a->npes; ++q)
    if (!a->y[q] || !a->flags[q]) return BSHMEM_MOE_ERR_ARGS;
  CombineParams P;
  P.a = *a;
  P.wait_limit_ns = a->wait_limit_ms ? (uint64_t)a->wait_limit_ms * 1000000ull : 10000000000ull;
  int grid = 0;
  P.split = 1;
  if (a->npes == 1 && !general) {
    P.split = column_split(a->T, a->H / BSHMEM_MOE_QUANT_BLOCK);
    const bool narrow = (a->H / 8 + P.split - 1) / P.split <= THREADS / 2;
    auto kernel = a->K <= 8 ? (narrow ? combine_kernel<8, true, true> : combine_kernel<8, true, false>)
                            : (narrow ? combine_kernel<BSHMEM_MOE_MAX_TOPK, true, true> : combine_kernel<BSHMEM_MOE_MAX_TOPK, true, false>);
    st = coop_grid(kernel, 0, a->T * P.split, a->max_ctas, &grid);
    if (st) return st;
    kernel<<<grid, THREADS, 0, stream>>>(P);
    return launched("bshmem_moe_combine", cudaGetLastError());
  }
  // Two builds of the kernel: up to 8 choices per token (62 registers, four CTAs per SM) and up to 16 (85, two).
  const void* kernel = a->K <= 8 ? (const void*)combine_kernel<8, false, false> : (const void*)combine_kernel<BSHMEM_MOE_MAX_TOPK, false, false>;
  st = a->K <= 8 ? coop_grid(combine_kernel<8, false, false>, 0, a->T, a->max_ctas, &grid) : coop_grid(combine_kernel<BSHMEM_MOE_MAX_TOPK, false, false>, 0, a->T, a->max_ctas, &grid);
  if (st) return st;
  if (cudaMemsetAsync(a->scratch, 0, 256, stream) != cudaSuccess) return BSHMEM_MOE_ERR_DRIVER;  // the grid-barrier counter
  void* params[] = {(void*)&P};
  cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(THREADS), params, 0, stream);
  if (e != cudaSuccess) {
    fprintf(stderr, "bshmem_moe_combine: launch failed: %s\n", cudaGetErrorString(e));
    return BSHMEM_MOE_ERR_DRIVER;
  }
  return 0;
}

extern "C" int bshmem_moe_dispatch(const bshmem_moe_dispatch_args_t* a, cudaStream_t stream) { return dispatch(a, false, stream); }
extern "C" int bshmem_moe_combine(const bshmem_moe_combine_args_t* a, cudaStream_t stream) { return combine(a, false, stream); }
// Test hooks: the kernels for several PEs on one PE, which otherwise takes kernels of its own.
extern "C" int bshmem_moe_test_dispatch_general(const bshmem_moe_dispatch_args_t* a, cudaStream_t stream) { return dispatch(a, true, stream); }
extern "C" int bshmem_moe_test_combine_general(const bshmem_moe_combine_args_t* a, cudaStream_t stream) { return combine(a, true, stream); }

// ------------------------------------------------------------------ dispatch without any allocation
// Single-PE dispatch whose count matrix and error word are a fixed array inside this library (see
// bshmem/moe_noalloc.h for who needs that and the rules of use).  In host code the array's name is only a handle; the
// address a kernel can use comes from cudaGetSymbolAddress, looked up once per GPU.
#include <limits.h>

#include <atomic>

#include "../../include/bshmem/moe_noalloc.h"

namespace {

struct NoAllocBlock {
  int counts[BSHMEM_MOE_NOALLOC_MAX_EXPERTS];  // the 1 x E count matrix (the kernels write all E of them)
  int error_flag;                              // used when the caller passes none; cleared by every call
};
static_assert(sizeof(NoAllocBlock) <= BSHMEM_MOE_NOALLOC_SCRATCH_BYTES, "documented scratch size is too small");

static __device__ __align__(256) unsigned char g_noalloc_block[BSHMEM_MOE_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
static std::atomic<NoAllocBlock*> g_noalloc_addr[kMaxDevices];  // device address of the array, per GPU ordinal (any host thread may fill it)

// Device address of the array on the current GPU, looked up on first use.
static int noalloc_block(NoAllocBlock** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return BSHMEM_MOE_ERR_DRIVER;
  NoAllocBlock* blk = g_noalloc_addr[dev].load(std::memory_order_acquire);
  if (!blk) {  // first call on this GPU (it is the current device): resolve the array's device address
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_block);
    if (e != cudaSuccess || !p) {
      fprintf(stderr, "bshmem_moe_dispatch_local_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
      return BSHMEM_MOE_ERR_DRIVER;
    }
    blk = (NoAllocBlock*)p;
    g_noalloc_addr[dev].store(blk, std::memory_order_release);  // two threads racing here store the same address
  }
  *out = blk;
  return BSHMEM_MOE_OK;
}

}  // namespace

extern "C" int bshmem_moe_dispatch_local_noalloc(const void* x, const int* topk_idx, int T, int H, int K, int E, void* recv_x, int* slot_map, int* expert_offsets,
                                                 int* error_flag, cudaStream_t stream) {
  if (!x || !topk_idx || !recv_x || !slot_map || !expert_offsets) return BSHMEM_MOE_ERR_ARGS;
  if (E > BSHMEM_MOE_NOALLOC_MAX_EXPERTS || E < 1 || K < 1 || K > BSHMEM_MOE_MAX_TOPK || T < 1 || H < 1 || H % BSHMEM_MOE_QUANT_BLOCK) {
    fprintf(stderr, "bshmem_moe_dispatch_local_noalloc: unsupported size (T=%d H=%d K=%d E=%d): at most %d experts and top-%d, H a multiple of %d\n", T, H, K, E,
            BSHMEM_MOE_NOALLOC_MAX_EXPERTS, BSHMEM_MOE_MAX_TOPK, BSHMEM_MOE_QUANT_BLOCK);
    return BSHMEM_MOE_ERR_SHAPE;
  }
  if ((long long)T * K > INT_MAX) {  // row numbers are 32-bit
    fprintf(stderr, "bshmem_moe_dispatch_local_noalloc: T * K = %lld rows do not fit 32-bit row numbers\n", (long long)T * K);
    return BSHMEM_MOE_ERR_SHAPE;
  }
  NoAllocBlock* blk = nullptr;
  int bst = noalloc_block(&blk);
  if (bst) return bst;
  // Of what the previous call left, only the error word has to start at zero (a caller with a word of its own may still ask for it).
  if (cudaMemsetAsync(&blk->error_flag, 0, sizeof(int), stream) != cudaSuccess) return BSHMEM_MOE_ERR_DRIVER;

  DispatchParams P;
  memset(&P, 0, sizeof(P));
  bshmem_moe_dispatch_args_t& a = P.a;
  a.T = T; a.H = H; a.K = K; a.E = E; a.rank = 0; a.npes = 1;
  a.payload = BSHMEM_MOE_BF16;
  a.cap_rows = T * K;
  a.epoch = 1;
  a.error_flag = error_flag ? error_flag : &blk->error_flag;
  a.x = x;
  a.topk_idx = topk_idx;
  a.recv_x[0] = recv_x;
  a.slot_map = slot_map;
  a.expert_offsets = expert_offsets;
  a.src_offsets = nullptr;
  a.counts[0] = blk->counts;
  P.wait_limit_ns = 10000000000ull;
  return dispatch_local(P, stream);
}

extern "C" int bshmem_moe_noalloc_error_bits(cudaStream_t stream, int* bits) {
  if (!bits) return BSHMEM_MOE_ERR_ARGS;
  NoAllocBlock* blk = nullptr;
  int st = noalloc_block(&blk);
  if (st) return st;
  if (cudaMemcpyAsync(bits, &blk->error_flag, sizeof(int), cudaMemcpyDeviceToHost, stream) != cudaSuccess) return BSHMEM_MOE_ERR_DRIVER;
  return cudaStreamSynchronize(stream) == cudaSuccess ? BSHMEM_MOE_OK : BSHMEM_MOE_ERR_DRIVER;
}
