// The sequential Float64 sum reduced = f(x) + reduced of mapreduce, computed
// in parallel and bit-identical to the loop.
//
// While the running sum a stays inside one binade, a = m 2^e with an integer
// 2^52 <= m < 2^53, every addition of the loop adds an integer to m: x is
// q 2^e with a real q, and round-to-nearest-even of m + q is m plus the
// nearest integer to q, except that a q halfway between two integers rounds
// to the side that leaves m + d even.  So one element is a map m -> m + d
// that depends on m through its parity alone, a run of elements is such a
// map too, and maps compose associatively: (d for even m, d for odd m).
// A run also carries the least and largest prefix of its map (over both
// parities), which tells, for the m it meets, that no addition inside leaves
// the binade; the runs for which that does not hold are cut finer and, at
// the end, added one by one with the hardware's addition.
//
//   k_fold_sums   approximate sum of every tile of FOLD_TILE elements
//   k_fold_frames their prefixes predict the binade ("frame") of each tile
//   k_fold_tiles  the map of each tile in its predicted frame; for a tile
//                 that is predicted to cross into another binade, the maps
//                 of its chunks of 64 elements in both
//   k_fold_first  beside k_fold_tiles, the exact sum through the first tile
//   k_fold_chain  one block carries it through the other tiles: up to
//                 1024 maps are composed and checked per round; a predicted
//                 crossing goes through fold_cross (one warp, its chunks'
//                 maps up to the crossing and behind it), any other tile that
//                 does not pass through fold_hard
//
// A wrong prediction costs time and nothing else: every map is applied only
// after its frame and its prefixes were checked against the exact sum.  Sums
// of one sign cross about log2(n) powers of two; data whose sum keeps
// changing its binade falls back to the hardware additions, no slower than the
// plain loop.
//
// Bound: for a few million elements the chain (a round 2 us, a crossing 3.5),
// beyond that the two passes over the column (k_fold_sums 7 us and k_fold_tiles
// 19 us for 5e6).  FOLD_TILE:
// tiles of 1024, 2048 and 4096 elements took 242, 242 and 270 us for 5e6
// uniform values, and 15.3, 9.2 and 6.4 ms for 2e6 values whose exponents spread
// over e^+-300 (there the chain goes tile by tile); 2048 keeps both.  Measured at
// 5e6 Float64 agents: 181 ms for the plain chain (36 ns per addition), 253 us
// with every crossing through fold_hard (two attempts of the whole block, 7.5
// us) and all 1024 maps read and composed in each round (4.3 us), 145 us with the
// first tile in the chain, 132 here;
// a sum that cancels to zero at every second addition (2e6): 72.6 and 73.4 ms.
#pragma once

#include <cstdint>

namespace vg {
namespace {

constexpr int FOLD_TILE = 2048;
constexpr int FOLD_TPB = 256;                       // blocks of the tile kernels
constexpr int FOLD_PER = FOLD_TILE / FOLD_TPB;      // consecutive elements per thread
constexpr int FOLD_CHAIN_TPB = 1024;
constexpr int FOLD_CHUNK = FOLD_TILE / 32;          // elements per warp of the chain block
constexpr int FOLD_LANE = FOLD_CHUNK / 32;          // and per lane
constexpr int FOLD_FEW = 128;                       // hardware additions an attempt is worth
constexpr int FOLD_PLAIN_MAX = 63;                  // tiles added without an attempt
constexpr int64_t FOLD_FAR = 1ll << 61;
constexpr int FOLD_NO_FRAME = -1;
constexpr int FOLD_CROSS = 1 << 24;                 // a tile's frame: FOLD_CROSS | first << 12 | last
constexpr int FOLD_SLOTS = 64;                      // crossing tiles with chunk maps
constexpr int FOLD_TURNS = 2;                       // attempts of fold_cross per tile and chunk

// d0, d1: what an even and an odd m change by; lo, hi: bounds of every
// prefix's change (lo > hi for the empty run); ok: no element too large for
// the frame
struct FoldMap {
  int64_t d0, d1, lo, hi;
  int ok;
};

// a predicted crossing's chunk maps in its first and its last frame
struct FoldCross {
  FoldMap m[2][32];
};

__device__ __forceinline__ FoldMap fold_identity() { return {0, 0, FOLD_FAR, -FOLD_FAR, 1}; }

__device__ __forceinline__ FoldMap fold_then(const FoldMap &a, const FoldMap &b) {
  FoldMap c;
  c.d0 = a.d0 + ((a.d0 & 1) ? b.d1 : b.d0);
  c.d1 = a.d1 + ((a.d1 & 1) ? b.d0 : b.d1);  // an odd m: parity of 1 + d1
  c.lo = min(a.lo, min(a.d0, a.d1) + b.lo);
  c.hi = max(a.hi, max(a.d0, a.d1) + b.hi);
  c.ok = a.ok & b.ok;
  return c;
}

__device__ __forceinline__ FoldMap fold_shfl_down(const FoldMap &a, int o) {
  return {__shfl_down_sync(0xffffffffu, a.d0, o), __shfl_down_sync(0xffffffffu, a.d1, o),
          __shfl_down_sync(0xffffffffu, a.lo, o), __shfl_down_sync(0xffffffffu, a.hi, o),
          __shfl_down_sync(0xffffffffu, a.ok, o)};
}
__device__ __forceinline__ FoldMap fold_shfl_up(const FoldMap &a, int o) {
  return {__shfl_up_sync(0xffffffffu, a.d0, o), __shfl_up_sync(0xffffffffu, a.d1, o),
          __shfl_up_sync(0xffffffffu, a.lo, o), __shfl_up_sync(0xffffffffu, a.hi, o),
          __shfl_up_sync(0xffffffffu, a.ok, o)};
}

// the map of the warp's 32 maps in lane order, on lane 0
__device__ __forceinline__ FoldMap fold_warp(FoldMap v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) v = fold_then(v, fold_shfl_down(v, o));
  return v;
}
// inclusive scan in lane order
__device__ __forceinline__ FoldMap fold_warp_scan(FoldMap v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const FoldMap u = fold_shfl_up(v, o);
    if (lane >= o) v = fold_then(u, v);
  }
  return v;
}

// frame of a sum: its sign and biased exponent (bits 52..63), or none for
// zero, subnormal, infinite and NaN
__device__ __forceinline__ int fold_frame(double a) {
  const int h = (int)((unsigned long long)__double_as_longlong(a) >> 52);
  const int e = h & 0x7ff;
  return e == 0 || e == 0x7ff ? FOLD_NO_FRAME : h;
}
__device__ __forceinline__ int64_t fold_m(double a) {
  return (__double_as_longlong(a) & ((1ll << 52) - 1)) | (1ll << 52);
}
__device__ __forceinline__ double fold_value(int frame, int64_t m) {
  return __longlong_as_double((long long)(((unsigned long long)frame << 52) |
                                          ((unsigned long long)m & ((1ull << 52) - 1))));
}
// every prefix of the run stays inside the binade: the rounded prefixes lie
// two units inside its ends, so the exact sums before rounding do too
__device__ __forceinline__ bool fold_fits(const FoldMap &a, int64_t m) {
  return a.ok && (a.lo > a.hi || (m + a.lo >= (1ll << 52) + 2 && m + a.hi <= (1ll << 53) - 2));
}
// A run whose prefixes leave +-2^52 fits no m; dropping it here keeps the
// sums of up to 1024 maps inside 64 bits.
__device__ __forceinline__ FoldMap fold_clip(FoldMap a) {
  if (a.lo <= a.hi && (a.lo < -(1ll << 52) || a.hi > (1ll << 52))) a.ok = 0;
  if (!a.ok) a.d0 = a.d1 = a.lo = a.hi = 0;
  return a;
}
__device__ __forceinline__ int64_t fold_apply(const FoldMap &a, int64_t m) {
  return m + ((m & 1) ? a.d1 : a.d0);
}

// one element in a frame; |q| has to stay below 2^(53 - lead)
__device__ __forceinline__ FoldMap fold_element(double x, int frame, int lead) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(b >> 52) & 0x7ff;
  unsigned long long mx = b & ((1ull << 52) - 1);
  if (ex) mx |= 1ull << 52;
  const int sh = (frame & 0x7ff) - (ex ? ex : 1);
  FoldMap r;
  r.ok = sh >= lead;
  const int s = min(max(sh, 1), 60);
  const int64_t f = (int64_t)(mx >> s);
  const unsigned long long rem = mx & ((1ull << s) - 1), half = 1ull << (s - 1);
  const int64_t up = rem > half, tie = rem == half, odd = f & 1;
  int64_t d0 = f + (tie ? odd : up), d1 = f + (tie ? 1 - odd : up);
  if ((int)(b >> 63) != (frame >> 11)) {
    d0 = -d0;
    d1 = -d1;
  }
  r.d0 = d0;
  r.d1 = d1;
  r.lo = min(d0, d1);
  r.hi = max(d0, d1);
  return r;
}

// a float near x, for the predictions: sign, rebased exponent and the high
// mantissa bits (a 64-bit conversion would go to the FP64 pipe)
__device__ __forceinline__ float fold_approx(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  const int e = (int)((h >> 20) & 0x7ff) - 1023 + 127;
  const uint32_t bits = e <= 0 ? 0u : e >= 255 ? 0x7f000000u
                                               : ((uint32_t)e << 23) | ((h & 0xfffffu) << 3);
  return __uint_as_float(bits | (h & 0x80000000u));
}

// element i as the loop sees it; false: skipped (died, or past the end)
template <bool F64>
__device__ __forceinline__ bool fold_load(const RedArgs &a, uint64_t i, double *v) {
  *v = 0.0;
  if (i >= a.n || (a.died && a.died[i])) return false;
  if (F64) {
    *v = ((const double *)a.p)[i];
  } else {
    int64_t vi;
    map_val(a.kind, a.arg, a.p, a.dt, i, 1, &vi, v);
  }
  return true;
}

template <bool F64>
__global__ void __launch_bounds__(FOLD_TPB) k_fold_sums(RedArgs a, float *tsum) {
  __shared__ float ws[FOLD_TPB / 32];
  let_next_start();
  const uint64_t base = (uint64_t)blockIdx.x * FOLD_TILE;
  double v[FOLD_PER];
#pragma unroll
  for (int k = 0; k < FOLD_PER; k++) fold_load<F64>(a, base + k * FOLD_TPB + threadIdx.x, &v[k]);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < FOLD_PER; k++) s += fold_approx(v[k]);
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < FOLD_TPB / 32; w++) t += ws[w];
    tsum[blockIdx.x] = t;
  }
}

// predicted frame of each tile: the binade of the approximate sum at its
// start when its end has the same, else both of them, or none when either has none
__global__ void __launch_bounds__(FOLD_CHAIN_TPB) k_fold_frames(const float *tsum, uint64_t ntiles,
                                                                double init, int *frame,
                                                                int *slots) {
  __shared__ float ws[32];
  let_next_start();
  wait_for_previous();
  if (threadIdx.x == 0) *slots = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float carry = fold_approx(init);
  for (uint64_t t0 = 0; t0 < ntiles; t0 += FOLD_CHAIN_TPB) {
    const uint64_t t = t0 + threadIdx.x;
    const float v = t < ntiles ? tsum[t] : 0.f;
    float x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    float s = ws[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    const float before = __shfl_sync(0xffffffffu, s, (w + 31) & 31);
    const float total = __shfl_sync(0xffffffffu, s, 31);
    const float end = carry + (w ? before : 0.f) + x;
    const int f1 = fold_frame((double)end), f0 = fold_frame((double)(end - v));
    if (t < ntiles)
      frame[t] = f0 == f1 ? f0 : f0 < 0 || f1 < 0 ? FOLD_NO_FRAME : FOLD_CROSS | f0 << 12 | f1;
    carry += total;
    __syncthreads();
  }
}

// a tile without a map leaves NO_FRAME in its frame, a crossing with chunk maps
// its slot in its map's d0
template <bool F64>
__device__ __forceinline__ void fold_tile(const RedArgs &a, int *frame, FoldMap *maps,
                                          FoldCross *cross, int *slots, int nslots) {
  __shared__ double v[FOLD_TILE + FOLD_TPB];  // one pad per thread's elements
  __shared__ uint32_t live[FOLD_TILE / 32];
  __shared__ FoldMap ws[FOLD_TPB / 32];
  __shared__ int slot;
  const int f = frame[blockIdx.x];
  if (f == FOLD_NO_FRAME) return;  // the chain cuts this tile finer
  if (f >= FOLD_CROSS && threadIdx.x == 0) slot = atomicAdd(slots, 1);
  const uint64_t base = (uint64_t)blockIdx.x * FOLD_TILE;
  const int lane = threadIdx.x & 31;
  double x[FOLD_PER];
  unsigned on = 0;
#pragma unroll
  for (int k = 0; k < FOLD_PER; k++)
    on |= (unsigned)fold_load<F64>(a, base + k * FOLD_TPB + threadIdx.x, &x[k]) << k;
#pragma unroll
  for (int k = 0; k < FOLD_PER; k++) {
    const int j = k * FOLD_TPB + threadIdx.x;
    v[j + j / FOLD_PER] = x[k];
    const unsigned b = __ballot_sync(0xffffffffu, (on >> k) & 1u);
    if (lane == 0) live[j / 32] = b;
  }
  __syncthreads();
  const unsigned mask = live[threadIdx.x * FOLD_PER / 32] >> (threadIdx.x * FOLD_PER & 31);
  auto mine = [&](int in) {  // the map of this thread's elements
    // all of the frame's sign and none halfway between two integers, as most
    // are: their rounded values add up, and every prefix lies between the
    // first and the last
    int64_t sum = 0, first = 0;
    bool plain = mask & ((1u << FOLD_PER) - 1), fit = true;
#pragma unroll
    for (int k = FOLD_PER - 1; k >= 0; k--) {
      if (!((mask >> k) & 1u)) continue;
      const int64_t b = __double_as_longlong(v[threadIdx.x * (FOLD_PER + 1) + k]);
      const int ex = (int)(b >> 52) & 0x7ff, sh = (in & 0x7ff) - (ex ? ex : 1);
      const uint64_t mx = ((uint64_t)b & ((1ull << 52) - 1)) | (uint64_t)(ex ? 1 : 0) << 52;
      const int s = min(max(sh, 1), 60);
      first = (int64_t)((mx + (1ull << (s - 1))) >> s);
      sum += first;
      plain &= mx << (64 - s) != 1ull << 63 && (int)((uint64_t)b >> 63) == in >> 11;
      fit &= sh >= 4;
    }
    if (plain) return FoldMap{sum, sum, first, sum, fit};
    FoldMap r = fold_identity();
#pragma unroll
    for (int k = 0; k < FOLD_PER; k++)
      if ((mask >> k) & 1u)
        r = fold_then(r, fold_element(v[threadIdx.x * (FOLD_PER + 1) + k], in, 4));
    return r;
  };
  if (f >= FOLD_CROSS) {
    if (slot >= nslots) {
      if (threadIdx.x == 0) frame[blockIdx.x] = FOLD_NO_FRAME;
      return;
    }
    if (threadIdx.x == 0) maps[blockIdx.x].d0 = slot;
    for (int q = 0; q < 2; q++) {
      FoldMap r = mine((q ? f : f >> 12) & 0xfff);
#pragma unroll
      for (int o = 1; o < FOLD_CHUNK / FOLD_PER; o <<= 1) r = fold_then(r, fold_shfl_down(r, o));
      if (threadIdx.x % (FOLD_CHUNK / FOLD_PER) == 0)
        cross[slot].m[q][threadIdx.x / (FOLD_CHUNK / FOLD_PER)] = fold_clip(r);
    }
    return;
  }
  FoldMap r = fold_warp(mine(f));
  if (lane == 0) ws[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x < 32) {
    r = lane < FOLD_TPB / 32 ? ws[lane] : fold_identity();
    r = fold_clip(fold_warp(r));
    if (lane == 0) {
      maps[blockIdx.x] = r;
      if (!r.ok) frame[blockIdx.x] = FOLD_NO_FRAME;
    }
  }
}

// (started beside k_fold_first)
template <bool F64>
__global__ void __launch_bounds__(FOLD_TPB) k_fold_tiles(RedArgs a, int *frame, FoldMap *maps,
                                                         FoldCross *cross, int *slots,
                                                         int nslots) {
  let_next_start();
  fold_tile<F64>(a, frame, maps, cross, slots, nslots);
  end_after_previous();
}

struct FoldShared {
  double v[2][FOLD_TILE];  // (the second half: the next tile of a plain run)
  uint32_t live[FOLD_TILE / 32];
  FoldMap wmap[32];
  double a;       // the exact running sum
  uint64_t next;  // next tile
  int at;         // next element of the tile (a multiple of FOLD_LANE)
  int step;       // groups of 32 the hardware adds after an attempt that failed early
  int plain, wait;  // tiles left to add without an attempt; how many after the next failure
  unsigned first;
  int warps, slot;  // whole warps of a round that pass; chunk maps of the tile behind it
  int64_t m;        // the sum behind those warps
  bool stopped;     // a tile of the round did not pass
};

// the map of one lane's FOLD_LANE elements from j on, none before `from`
__device__ __forceinline__ FoldMap fold_lane(const FoldShared &S, int j, int from, int frame) {
  FoldMap r = fold_identity();
  const unsigned live = S.live[j / 32] >> (j & 31);
  if (j >= from) {
#pragma unroll
    for (int k = 0; k < FOLD_LANE; k++)
      if ((live >> k) & 1u) r = fold_then(r, fold_element(S.v[0][j + k], frame, 1));
  }
  return r;
}

// 32 elements added by the hardware in order
__device__ __forceinline__ double fold_plain_32(const double *v, int j, double a) {
  const int i = j + ((int)threadIdx.x & 31);
  const double y = i < FOLD_TILE ? v[i] : -0.0;
#pragma unroll
  for (int l = 0; l < 32; l++) a = __dadd_rn(__shfl_sync(0xffffffffu, y, l), a);
  return a;
}

// `run` tiles by the hardware's additions alone: the other warps stage the
// next tile while warp 0 adds the current one (-0.0 added to anything
// changes nothing: it stands for the elements that do not count)
template <bool F64>
__device__ void fold_plain(const RedArgs &a, uint64_t tile, uint64_t run, FoldShared &S) {
  auto stage = [&](uint64_t t, int b, int first) {
    for (int j = (int)threadIdx.x - first; j < FOLD_TILE; j += FOLD_CHAIN_TPB - first) {
      double x;
      S.v[b][j] = fold_load<F64>(a, t * FOLD_TILE + j, &x) ? x : -0.0;
    }
  };
  double cur = S.a;
  stage(tile, 0, 0);
  __syncthreads();
  for (uint64_t k = 0; k < run; k++) {
    const int b = (int)(k & 1);
    if (threadIdx.x >= 32) {
      if (k + 1 < run) stage(tile + k + 1, b ^ 1, 32);
    } else {
      const uint64_t left = a.n - (tile + k) * FOLD_TILE;
      const int end = left < (uint64_t)FOLD_TILE ? (int)left : FOLD_TILE;
      double y[32];
#pragma unroll
      for (int l = 0; l < 32; l++) y[l] = S.v[b][l];
      for (int j = 0; j < end; j += 32) {  // the next 32 are read under the chain
        double z[32];
#pragma unroll
        for (int l = 0; l < 32; l++) z[l] = S.v[b][(j + 32) % FOLD_TILE + l];
#pragma unroll
        for (int l = 0; l < 32; l++) cur = __dadd_rn(y[l], cur);
#pragma unroll
        for (int l = 0; l < 32; l++) y[l] = z[l];
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) S.a = cur;
  __syncthreads();
}

// One tile whose map does not apply.  An attempt maps the rest of the tile
// in the frame of the current sum, FOLD_CHUNK elements per warp; warp 0
// carries the sum up to the first lane's elements that may leave the binade,
// adds those with the hardware, and the next attempt starts behind them in
// the new frame.  An attempt costs about as much as FOLD_FEW hardware
// additions (36 ns each), so one that carried fewer elements is followed by
// 32, 64, 128, ... hardware additions before the next, and once that is a
// whole tile, by whole tiles without an attempt (1, 3, 7, .. 63): a sum that
// leaves its binade at every turn runs at the speed of the plain chain.
// A sum that starts at zero doubles within every few elements at first: there
// FOLD_FEW hardware additions precede the first attempt.
// start: elements of the tile that are in the sum already
template <bool F64>
__device__ void fold_hard(const RedArgs &a, uint64_t tile, int start, FoldShared &S) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t base = tile * FOLD_TILE;
#pragma unroll
  for (int k = 0; k < FOLD_TILE / FOLD_CHAIN_TPB; k++) {
    const int j = k * FOLD_CHAIN_TPB + threadIdx.x;
    double x;
    const bool on = fold_load<F64>(a, base + j, &x);
    S.v[0][j] = on ? x : -0.0;
    const unsigned b = __ballot_sync(0xffffffffu, on);
    if (lane == 0) S.live[j / 32] = b;
  }
  if (threadIdx.x == 0) S.at = start;
  __syncthreads();
  if (tile == 0 && start == 0 && fold_frame(S.a) == FOLD_NO_FRAME) {  // block-uniform
    double cur = S.a;
    __syncthreads();
    if (w == 0) {
      for (int j = 0; j < FOLD_FEW; j += 32) cur = fold_plain_32(S.v[0], j, cur);
      if (lane == 0) {
        S.a = cur;
        S.at = FOLD_FEW;
      }
    }
    __syncthreads();
  }
  const uint64_t left = a.n - base;
  const int end = left < (uint64_t)FOLD_TILE
                      ? (int)(left + FOLD_LANE - 1) / FOLD_LANE * FOLD_LANE : FOLD_TILE;
  while (S.at < end) {
    const int from = S.at;
    const double acc = S.a;
    const int f = fold_frame(acc);
    const int c0 = from / FOLD_CHUNK;
    if (f != FOLD_NO_FRAME && w >= c0) {
      const FoldMap r = fold_warp(fold_lane(S, w * FOLD_CHUNK + FOLD_LANE * lane, from, f));
      if (lane == 0) S.wmap[w] = fold_clip(r);
    }
    __syncthreads();
    if (w == 0) {
      double cur = acc;
      int at = from;
      if (f != FOLD_NO_FRAME) {
        int64_t m = fold_m(acc);
        FoldMap r = fold_warp_scan(lane >= c0 ? S.wmap[lane] : fold_identity());
        unsigned bad = __ballot_sync(0xffffffffu, !fold_fits(r, m));
        const int c = bad ? __ffs(bad) - 1 : 32;
        if (c > c0) {
          m = __shfl_sync(0xffffffffu, fold_apply(r, m), c - 1);
          at = c * FOLD_CHUNK;
        }
        if (c < 32) {
          r = fold_warp_scan(fold_lane(S, c * FOLD_CHUNK + FOLD_LANE * lane, at, f));
          bad = __ballot_sync(0xffffffffu, !fold_fits(r, m));
          const int l = bad ? __ffs(bad) - 1 : 32;
          if (l) m = __shfl_sync(0xffffffffu, fold_apply(r, m), l - 1);
          at = max(at, c * FOLD_CHUNK + FOLD_LANE * l);
        }
        cur = fold_value(f, m);
      }
      const int carried = at - from;
      if (at < end) {  // the elements that stopped the attempt
#pragma unroll
        for (int k = 0; k < FOLD_LANE; k++) cur = __dadd_rn(S.v[0][at + k], cur);
        at += FOLD_LANE;
      }
      int step = 0;
      if (carried < FOLD_FEW && at < end) {
        step = S.step ? min(2 * S.step, FOLD_TILE / 32) : 1;
        for (int g = 0; g < step && at < end; g++, at += 32) cur = fold_plain_32(S.v[0], at, cur);
      }
      __syncwarp();
      if (lane == 0) {
        S.a = cur;
        S.at = at;
        if (step || carried >= FOLD_FEW) {  // (cut short by the tile's end: says nothing)
          S.step = step;
          if (step == FOLD_TILE / 32) {
            S.plain = S.wait;
            S.wait = min(2 * S.wait + 1, FOLD_PLAIN_MAX);
          } else {
            S.wait = 1;
          }
        }
      }
    }
    __syncthreads();
  }
}

// The first tile, where a sum that starts at zero crosses a binade every few
// elements: its sum needs no prediction, so it is taken while the other
// tiles are mapped (30 us of one block beside 19 of the others).
struct FoldStart {
  double a;
  int step, plain, wait;
};
template <bool F64>
__global__ void __launch_bounds__(FOLD_CHAIN_TPB) k_fold_first(RedArgs a, FoldStart *start) {
  __shared__ FoldShared S;
  wait_for_previous();  // (before the mapping may start: it reads the frames)
  let_next_start();
  if (threadIdx.x == 0) {
    S.a = a.init_f;
    S.step = S.plain = 0;
    S.wait = 1;
  }
  __syncthreads();
  fold_hard<F64>(a, 0, 0, S);
  if (threadIdx.x == 0) *start = {S.a, S.step, S.plain, S.wait};
}

// A predicted crossing, by warp 0: the maps of the chunks in the sum's frame,
// one per lane, carry it to the chunk that leaves the binade; that chunk's
// elements are mapped two per lane, those of the lane that crosses are added by
// the hardware, and what is behind them goes on in the new frame.  Returns
// the elements done, on all lanes, and the sum: all of the tile, or less when
// the sum is in neither frame or crosses again (fold_hard does the rest).
template <bool F64>
__device__ int fold_cross(const RedArgs &a, uint64_t tile, int frames, const FoldCross *cross,
                          double &acc) {
  const int lane = threadIdx.x & 31;
  const FoldMap m0 = cross->m[0][lane], m1 = cross->m[1][lane];
  int c = 0;
  for (int turn = 0; turn < FOLD_TURNS; turn++) {
    int f = fold_frame(acc);
    const bool second = f != (frames >> 12 & 0xfff);
    if (f == FOLD_NO_FRAME || (second && f != (frames & 0xfff))) return c * FOLD_CHUNK;
    int64_t m = fold_m(acc);
    FoldMap r = fold_warp_scan(lane < c ? fold_identity() : second ? m1 : m0);
    unsigned bad = __ballot_sync(0xffffffffu, !fold_fits(r, m));
    const int b = bad ? __ffs(bad) - 1 : 32;
    if (b > c) {
      acc = fold_value(f, __shfl_sync(0xffffffffu, fold_apply(r, m), b - 1));
      c = b;
    }
    if (c == 32) return FOLD_TILE;
    double x[FOLD_LANE];
    bool on[FOLD_LANE];
    const int at = c * FOLD_CHUNK + FOLD_LANE * lane;
#pragma unroll
    for (int k = 0; k < FOLD_LANE; k++) {
      on[k] = fold_load<F64>(a, tile * FOLD_TILE + at + k, &x[k]);
      if (!on[k]) x[k] = -0.0;
    }
    int l = 0;  // lanes of the chunk that are in the sum
    for (int in = 0; l < 32; in++) {
      f = fold_frame(acc);
      if (in == FOLD_TURNS || f == FOLD_NO_FRAME) return c * FOLD_CHUNK + FOLD_LANE * l;
      m = fold_m(acc);
      r = fold_identity();
      if (lane >= l) {
#pragma unroll
        for (int k = 0; k < FOLD_LANE; k++)
          if (on[k]) r = fold_then(r, fold_element(x[k], f, 1));
      }
      r = fold_warp_scan(r);
      bad = __ballot_sync(0xffffffffu, !fold_fits(r, m));
      const int e = bad ? __ffs(bad) - 1 : 32;
      if (e > l) acc = fold_value(f, __shfl_sync(0xffffffffu, fold_apply(r, m), e - 1));
      l = e;
      if (l < 32) {
#pragma unroll
        for (int k = 0; k < FOLD_LANE; k++)
          acc = __dadd_rn(__shfl_sync(0xffffffffu, x[k], l), acc);
        l++;
      }
    }
    c++;
    if (c == 32) return FOLD_TILE;
  }
  return c * FOLD_CHUNK;
}

// the exact sum through all tiles; maps == null: every tile is cut finer
// (short columns, where predicting costs more than it saves)
template <bool F64>
__global__ void __launch_bounds__(FOLD_CHAIN_TPB) k_fold_chain(RedArgs a, uint64_t ntiles,
                                                               const int *frame,
                                                               const FoldMap *maps,
                                                               const FoldCross *cross,
                                                               const FoldStart *start,
                                                               int64_t *oi, double *of) {
  __shared__ FoldShared S;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  wait_for_previous();
  if (threadIdx.x == 0) {
    S.a = start ? start->a : a.init_f;
    S.next = start ? (isnan(start->a) ? ntiles : 1) : 0;
    S.step = start ? start->step : 0;
    S.plain = start ? start->plain : 0;
    S.wait = start ? start->wait : 1;
  }
  __syncthreads();
  while (S.next < ntiles) {
    const uint64_t t0 = S.next;
    const double acc = S.a;
    if (S.plain) {  // block-uniform
      const uint64_t run = min((unsigned long long)S.plain, (unsigned long long)(ntiles - t0));
      fold_plain<F64>(a, t0, run, S);
      if (threadIdx.x == 0) {
        S.next = t0 + run;
        S.plain = 0;
      }
      __syncthreads();
      continue;
    }
    if (threadIdx.x == 0) {
      S.first = FOLD_CHAIN_TPB;
      S.slot = -1;
      S.at = 0;
    }
    __syncthreads();
    bool hard = true;
    if (maps) {
      // thread k: tile t0 + k; the run ends at the first tile in another
      // frame than the sum's, and only the warps of the run read and compose
      // its maps
      const int f = fold_frame(acc);
      const uint64_t t = t0 + threadIdx.x;
      const int tf = t < ntiles ? frame[t] : FOLD_NO_FRAME;
      const unsigned other = __ballot_sync(0xffffffffu, tf != f || f == FOLD_NO_FRAME);
      if (lane == 0 && other) atomicMin(&S.first, (unsigned)(w * 32 + __ffs(other) - 1));
      __syncthreads();
      const unsigned run = S.first, nw = (run + 31) / 32;
      FoldMap r = fold_identity();
      if (threadIdx.x == run && t < ntiles && tf >= FOLD_CROSS) S.slot = (int)maps[t].d0;
      if ((unsigned)w < nw) {
        if (threadIdx.x < run) r = maps[t];
        r = fold_warp_scan(r);
        if (lane == 31) S.wmap[w] = r;
      }
      __syncthreads();
      if (w == 0) {
        const FoldMap p = fold_warp_scan((unsigned)lane < nw ? S.wmap[lane] : fold_identity());
        const int64_t m = fold_m(acc);
        const unsigned bad = __ballot_sync(0xffffffffu, (unsigned)lane < nw && !fold_fits(p, m));
        const int k = bad ? __ffs(bad) - 1 : (int)nw;
        const int64_t to = __shfl_sync(0xffffffffu, fold_apply(p, m), (k + 31) & 31);
        if (lane == 0) {
          S.warps = k;
          S.m = k ? to : m;
          if (k == (int)nw) {
            if (run) S.a = fold_value(f, to);
            S.next = t0 + run;
          }
        }
      }
      __syncthreads();
      const int k = S.warps;
      hard = t0 + run < ntiles && run < FOLD_CHAIN_TPB;
      if (k < (int)nw) {  // block-uniform: warp k has the first tile that does not pass
        if (w == k) {
          // (none, when the warp's own bounds are met and only the bounds of
          // all before it together, taken over both parities, were not)
          const unsigned bad = __ballot_sync(0xffffffffu, !fold_fits(r, S.m));
          const int l = bad ? __ffs(bad) - 1 : 32;
          const int64_t to = __shfl_sync(0xffffffffu, fold_apply(r, S.m), (l + 31) & 31);
          if (lane == 0) {
            S.a = fold_value(f, l ? to : S.m);
            S.next = min(t0 + k * 32 + l, t0 + run);
            S.slot = -1;
            S.stopped = bad != 0;
          }
        }
        __syncthreads();
        hard = S.stopped;
      }
      if (hard && S.slot >= 0) {  // block-uniform
        const uint64_t tile = S.next;
        __syncthreads();
        if (w == 0) {
          double cur = S.a;
          const int done = fold_cross<F64>(a, tile, frame[tile], cross + S.slot, cur);
          if (lane == 0) {
            S.a = cur;
            S.at = done;
            if (done == FOLD_TILE) S.next = tile + 1;
            if (done >= FOLD_FEW) {  // an attempt that was worth it
              S.step = 0;
              S.wait = 1;
            }
          }
        }
        __syncthreads();
        hard = S.at < FOLD_TILE;
      }
    }
    if (hard) {
      fold_hard<F64>(a, S.next, S.at, S);
      // NaN stays NaN whatever is added
      if (threadIdx.x == 0) S.next = isnan(S.a) ? ntiles : S.next + 1;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *oi = a.init_i;
    *of = S.a;
  }
}

}  // namespace
}  // namespace vg
