// Single-pass exclusive scan over tiles of SCAN_CHUNK items with decoupled
// look-back (D. Merrill and M. Garland, "Single-pass parallel prefix scan with
// decoupled look-back", NVIDIA NVR-2016-002), with the items produced and the
// sums consumed by functors: a compaction is one launch (flags made, counted
// and their places used in the same kernel) instead of three and two arrays.
// A tile publishes its total, then warp 0 reads the flags of the 32 preceding
// tiles at once and adds totals back to the nearest tile whose inclusive
// prefix is known.  Tiles take their index from a ticket counter in start
// order (a tile only waits for running tiles); every wait is bounded and
// records an error in *err when it gives up.
#pragma once

#include "vg_internal.h"

namespace vg {

constexpr int SCAN_TPB = 256;
constexpr int SCAN_IPT = 16;                     // items per thread
constexpr int SCAN_CHUNK = SCAN_TPB * SCAN_IPT;  // items per tile
constexpr uint32_t SCAN_SPIN_LIMIT = 1u << 21;
constexpr int SCAN_ERR_LOOKBACK = 0x5e02;

template <class T>
__device__ T block_exclusive_scan(T v, T *warp_sums, T *block_total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    T s = lane < nw ? warp_sums[lane] : T(0);
    T incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane < nw) warp_sums[lane] = incl - s;
    if (lane == 31 && block_total) *block_total = incl;
  }
  __syncthreads();
  T r = warp_sums[w] + x - v;
  __syncthreads();
  return r;
}

__device__ __forceinline__ void st_release_u32(uint32_t *a, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *a) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *a) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *a) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
  return v;
}

template <class T>
struct ScanState {
  uint32_t *flag;  // per tile: 0 nothing, 1 total in agg, 2 inclusive prefix in pre
  T *agg, *pre;
  uint32_t *ticket;
};

// in(i) gives item i; out(i, sum of the items before i, item i) takes its
// place; *total (may be null): the sum of all items
template <int IPT, class T, class In, class Out>
__global__ void __launch_bounds__(SCAN_TPB) k_scan_map(In in, Out out, uint64_t n, T *total,
                                                       ScanState<T> S, int *err) {
  constexpr int CHUNK = SCAN_TPB * IPT;
  __shared__ T ws[32];
  __shared__ T s_tot, s_excl;
  __shared__ uint32_t s_tile;
  // items pass through shared memory between the two orders: consecutive
  // threads take consecutive items where the functors touch memory, a thread
  // takes IPT consecutive ones where it sums (one pad per IPT)
  __shared__ T x[CHUNK + SCAN_TPB];
  if (threadIdx.x == 0) s_tile = atomicAdd(S.ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = (uint64_t)tile * CHUNK + threadIdx.x;
  T v[IPT], own[IPT];
  T sum = 0;
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    const uint64_t i = base + k * SCAN_TPB;
    own[k] = i < n ? in(i) : T(0);
  }
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    const uint32_t j = k * SCAN_TPB + threadIdx.x;
    x[j + j / IPT] = own[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    v[k] = x[threadIdx.x * (IPT + 1) + k];
    sum += v[k];
  }
  T run = block_exclusive_scan<T>(sum, ws, &s_tot);
  if (threadIdx.x < 32) {
    const uint32_t lane = threadIdx.x;
    const T tot = s_tot;
    T excl = 0;
    if (tile == 0) {
      if (lane == 0) {
        S.pre[0] = tot;
        st_release_u32(S.flag, 2u);
      }
    } else {
      if (lane == 0) {
        S.agg[tile] = tot;
        st_release_u32(S.flag + tile, 1u);
      }
      int64_t t = (int64_t)tile - 1;
      uint32_t spins = 0;
      for (;;) {
        const int64_t tt = t - (int64_t)lane;
        const uint32_t f = tt >= 0 ? ld_acquire_u32(S.flag + tt) : 2u;
        const unsigned pm = __ballot_sync(0xffffffffu, f == 2u);
        const unsigned zm = __ballot_sync(0xffffffffu, f == 0u);
        const int P = pm ? __ffs(pm) - 1 : 32;  // nearest predecessor with a prefix
        const unsigned need = P == 32 ? 0xffffffffu : (2u << P) - 1u;
        if (zm & need) {  // a tile in between has published nothing yet
          if (++spins > SCAN_SPIN_LIMIT) {
            if (lane == 0) report_status(err, SCAN_ERR_LOOKBACK);
            break;
          }
          if (spins > 16) __nanosleep(64);
          continue;
        }
        T part = 0;
        if ((int)lane < P) part = ld_relaxed(S.agg + tt);
        else if ((int)lane == P && tt >= 0) part = ld_relaxed(S.pre + tt);
#pragma unroll
        for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        excl += part;
        if (P < 32) break;
        t -= 32;
        spins = 0;
      }
      if (lane == 0) {
        S.pre[tile] = excl + tot;
        st_release_u32(S.flag + tile, 2u);
      }
    }
    if (lane == 0) {
      s_excl = excl;
      if (total && ((uint64_t)tile + 1) * CHUNK >= n) *total = excl + tot;
    }
  }
  __syncthreads();
  run += s_excl;
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    x[threadIdx.x * (IPT + 1) + k] = run;
    run += v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    const uint32_t j = k * SCAN_TPB + threadIdx.x;
    const uint64_t i = base + k * SCAN_TPB;
    if (i < n) out(i, x[j + j / IPT], own[k]);
  }
}

template <class T>
uint64_t scan_scratch_bytes(uint64_t n, int ipt = SCAN_IPT) {
  const uint64_t nt = (n + SCAN_TPB * ipt - 1) / (SCAN_TPB * ipt);
  return 64 + nt * 4 + 2 * nt * sizeof(T) + 64;
}

// the tiles' state in scan_scratch_bytes<T>(n, ipt) bytes (flags zeroed here)
template <class T>
ScanState<T> scan_state(void *scratch, uint64_t n, cudaStream_t st, int ipt = SCAN_IPT) {
  const uint64_t nt = (n + SCAN_TPB * ipt - 1) / (SCAN_TPB * ipt);
  if (nt >= (1ull << 31)) fail(VG_ERR_NOMEM, "scan: too many items");
  char *buf = (char *)scratch;
  ScanState<T> S;
  S.ticket = (uint32_t *)buf;
  S.flag = (uint32_t *)(buf + 64);
  S.agg = (T *)(buf + ((64 + nt * 4 + 15) & ~15ull));
  S.pre = S.agg + nt;
  VG_CUDA(cudaMemsetAsync(buf, 0, 64 + nt * 4, st));
  return S;
}

// IPT: items per thread.  A thread's items overlap little where the functors
// chase pointers or store, so those take small tiles: with 16, 8 and 4 items
// the callers of a spawn among 2.2*10^5 agents take 31.9, 22 and 15.8 us; plain
// columns of that length 5.5, 7 and 10.2 us (a longer chain of tiles).
template <int IPT, class T, class In, class Out>
void scan_map(Sim &s, uint64_t n, const In &in, const Out &out, T *total) {
  if (n == 0) return;
  const ScanState<T> S =
      scan_state<T>(s.work(Sim::WORK_SCAN, scan_scratch_bytes<T>(n, IPT)), n, s.stream, IPT);
  constexpr uint64_t chunk = SCAN_TPB * IPT;
  k_scan_map<IPT, T, In, Out><<<(unsigned)((n + chunk - 1) / chunk), SCAN_TPB, 0, s.stream>>>(
      in, out, n, total, S, s.d_status.as<int>());
  VG_CUDA(cudaGetLastError());
}

}  // namespace vg
