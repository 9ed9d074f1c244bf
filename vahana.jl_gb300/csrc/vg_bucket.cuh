// The per-step rebuild of an edge type's container from typed records.
//
// The records are slots 0 .. n-1 in call order (the order in which the
// sequential sweep calls add_edge!, src/EdgeMethods.jl:478-522), each a
// target row, a value (its source, or its slot when the edge type carries
// payload) or a hole.  The container's rows are cut into at most BK_MAX
// buckets of 2^shift consecutive rows:
//
//   k_bucket_tiles  a block sorts a tile of BK_TILE consecutive slots by
//                   bucket, stably, and writes the tile's sorted records
//                   (row in the bucket and slot in the tile packed in a
//                   word, and the value where it is not the slot) and the
//                   bucket offsets of the tile.  No tile waits for another.
//   k_bucket_build  a block per bucket gathers the bucket's piece of every
//                   tile, in tile order.  The sum over the tiles of the
//                   bucket's offset is the number of records of all earlier
//                   buckets, so the block knows its place without a scan
//                   over the launch.  It counts the records of its rows in
//                   shared memory, scans the counts into row pointers, and
//                   places the records in order.
//
// One pass over the records each instead of one per 8 bits of the row
// number, and two launches instead of eight.
#pragma once

#include "vg_internal.h"

namespace vg {

constexpr uint32_t BK_HOLE = 0xFFFFFFFFu;  // row of a slot without a record
constexpr int BK_MAX = 2048;
constexpr int BK_TPB = 512;
constexpr int BK_WARPS = BK_TPB / 32;
constexpr int BK_IPT = 8;
constexpr int BK_TILE = BK_TPB * BK_IPT;  // 4096 slots

// Where a tile's records come from: load() reads what slot i needs (all of a
// thread's slots before the first make(), so that their loads overlap),
// make() forms the record; false: none.
// slots as two columns, or one (the value is the slot)
template <bool VALS_>
struct SlotSource {
  static constexpr bool VALS = VALS_;
  const uint32_t *rows, *vals;
  struct Raw {
    uint32_t row, val;
  };
  __device__ __forceinline__ Raw load(uint64_t i) const { return {rows[i], VALS ? vals[i] : 0u}; }
  __device__ __forceinline__ bool make(uint64_t, const Raw &r, uint32_t &row, uint32_t &val) const {
    row = r.row;
    val = r.val;
    return row != BK_HOLE;
  }
};

inline size_t bucket_tile_smem(const BucketPlan &p) {
  const size_t nb4 = (p.nbuckets + 3) & ~3u;
  return BK_WARPS * nb4 * 2 + nb4 * 2 + BK_TILE * (p.vals ? 8 : 4) + 64;
}

template <class Source>
__global__ void __launch_bounds__(BK_TPB) k_bucket_tiles(Source source, BucketPlan p) {
  extern __shared__ __align__(16) unsigned char bk_smem[];
  let_next_start();
  const uint32_t nb4 = (p.nbuckets + 3) & ~3u;
  uint32_t *srec = (uint32_t *)bk_smem;              // [BK_TILE]
  uint32_t *sval = srec + BK_TILE;                   // [BK_TILE] with VALS
  uint16_t *wcnt = (uint16_t *)(srec + (Source::VALS ? 2 : 1) * BK_TILE);  // [BK_WARPS][nb4]
  uint16_t *start = wcnt + BK_WARPS * nb4;           // [nb4]
  uint32_t *ws = (uint32_t *)(start + nb4);          // [16]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t t0 = (uint64_t)blockIdx.x * BK_TILE + (uint64_t)w * (32 * BK_IPT) + lane;
  uint32_t row[BK_IPT], val[BK_IPT], rank[BK_IPT];
  uint2 *z = (uint2 *)wcnt;  // four 16-bit counters per word
  for (uint32_t i = threadIdx.x; i < BK_WARPS * nb4 / 4; i += BK_TPB) z[i] = make_uint2(0, 0);
  wait_for_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) *p.maxdeg = 0;
  unsigned have = 0;
  typename Source::Raw raw[BK_IPT];
#pragma unroll
  for (int k = 0; k < BK_IPT; k++)
    if (t0 + 32 * k < p.n) raw[k] = source.load(t0 + 32 * k);
#pragma unroll
  for (int k = 0; k < BK_IPT; k++) {
    const uint64_t i = t0 + 32 * k;
    row[k] = val[k] = 0;
    if (i < p.n && source.make(i, raw[k], row[k], val[k])) have |= 1u << k;
  }
  __syncthreads();
  // rank of each record among the warp's earlier records of its bucket: the
  // lanes with the same label (bucket, and whether there is a record) from
  // one ballot per label bit
  const int bits = 32 - __clz(p.nbuckets - 1);  // 0 for one bucket
  uint16_t *mine = wcnt + w * nb4;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < BK_IPT; k++) {
    const bool valid = have >> k & 1u;
    const uint32_t b = row[k] >> p.shift;
    unsigned peers = __ballot_sync(0xffffffffu, valid);
    if (!valid) peers = ~peers;
    for (int bit = 0; bit < bits; bit++) {
      const bool set = b >> bit & 1u;
      const unsigned v = __ballot_sync(0xffffffffu, set);
      peers &= set ? v : ~v;
    }
    const uint32_t before = valid ? mine[b] : 0u;
    rank[k] = before + __popc(peers & lt);
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) mine[b] = (uint16_t)(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  // thread g: buckets 4 g .. 4 g + 3; the warps' counters become exclusive
  // sums over the warps (four 16-bit sums in a word: none exceeds BK_TILE)
  const uint32_t g = threadIdx.x;
  unsigned long long sum = 0;
  if (4 * g < nb4) {
    unsigned long long *c = (unsigned long long *)wcnt + g;
#pragma unroll
    for (int w2 = 0; w2 < BK_WARPS; w2++) {
      const unsigned long long v = c[w2 * (nb4 / 4)];
      c[w2 * (nb4 / 4)] = sum;
      sum += v;
    }
  }
  const uint32_t c0 = sum & 0xffff, c1 = sum >> 16 & 0xffff, c2 = sum >> 32 & 0xffff,
                 c3 = (uint32_t)(sum >> 48);
  const uint32_t tot = c0 + c1 + c2 + c3;
  uint32_t x = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w2 = 0; w2 < BK_WARPS; w2++) {
    const uint32_t v = ws[w2];
    before += w2 < w ? v : 0u;
    all += v;
  }
  before += x - tot;
  uint16_t *offs = p.offs + (uint64_t)blockIdx.x * p.pitch;
  if (4 * g < nb4) {
    const uint2 s = make_uint2(before | (before + c0) << 16,
                               (before + c0 + c1) | (before + c0 + c1 + c2) << 16);
    ((uint2 *)start)[g] = s;
    ((uint2 *)offs)[g] = s;  // (entries from nbuckets on: all records)
  }
  if (threadIdx.x == 0) offs[p.nbuckets] = (uint16_t)all;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < BK_IPT; k++)
    if (have >> k & 1u) {
      const uint32_t b = row[k] >> p.shift;
      const uint32_t at = start[b] + mine[b] + rank[k];
      srec[at] = (row[k] & ((1u << p.shift) - 1u)) |
                 (uint32_t)(w * (32 * BK_IPT) + 32 * k + lane) << p.shift;
      if (Source::VALS) sval[at] = val[k];
    }
  __syncthreads();
  uint32_t *out = p.recs + (uint64_t)blockIdx.x * BK_TILE;
  uint32_t *vout = p.vals + (uint64_t)blockIdx.x * BK_TILE;
  for (uint32_t i = threadIdx.x; i < all; i += BK_TPB) {
    out[i] = srec[i];
    if (Source::VALS) vout[i] = sval[i];
  }
}

template <class Source>
void launch_bucket_tiles(const Source &src, const BucketPlan &p, cudaStream_t st) {
  if (!p.ntiles) return;
  static const bool ok = cudaFuncSetAttribute(k_bucket_tiles<Source>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              128 * 1024) == cudaSuccess;
  if (!ok) fail(VG_ERR_CUDA, "cannot reserve the rebuild's shared memory");
  launch_dependent(k_bucket_tiles<Source>, p.ntiles, BK_TPB, bucket_tile_smem(p), st, src, p);
}

}  // namespace vg
