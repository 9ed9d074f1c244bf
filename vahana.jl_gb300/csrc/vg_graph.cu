// CSR construction and maintenance.
//
// build_csr_from_records rebuilds an edge type's containers from a batch of
// edge records that are in Vahana's call order (or carry an order key):
// the per-target order that results is the one `push!` produces in
// add_edge! (src/EdgeMethods.jl:478-522).  With merge_existing the old
// edges of a row come first, as with add_existing (src/EdgeMethods.jl:
// 639-663, where the write container starts as a copy of the read one).
//
// remove_died_edges removes the edges of agents that died in a transition:
// rows of died targets (_remove_edges_agent_target!, src/EdgeMethods.jl:
// 897-920) and, for edge types that store the source, edges whose source
// died (_remove_edges_agent_source!, :606-631).
#include <algorithm>
#include <cstring>

#include "vg_bucket.cuh"
#include "vg_internal.h"
#include "vg_rows.cuh"
#include "vg_scan.cuh"

namespace vg {

namespace {

constexpr int TPB = 256;
inline unsigned nblk(uint64_t n, int tpb = TPB) {
  uint64_t b = (n + tpb - 1) / tpb;
  return (unsigned)std::max<uint64_t>(b, 1);
}

__global__ void k_type_hist(const uint64_t *to, const uint64_t *from, uint64_t n,
                            unsigned long long *counts, unsigned *srcmask) {
  __shared__ unsigned long long sc[MAX_AGENT_TYPES];
  __shared__ unsigned sm;
  if (threadIdx.x < MAX_AGENT_TYPES) sc[threadIdx.x] = 0;
  if (threadIdx.x == 0) sm = 0;
  __syncthreads();
  // records mostly share one target type: count runs of equal types in a
  // register and flush a run to shared memory when the type changes
  unsigned mymask = 0, run_t = 0xFFFFFFFFu;
  unsigned long long run_n = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    unsigned t = (unsigned)(to[i] >> SHIFT_TYPE);
    if (t != run_t) {
      if (run_n && run_t < MAX_AGENT_TYPES) atomicAdd(&sc[run_t], run_n);
      run_t = t;
      run_n = 0;
    }
    run_n++;
    if (from) {
      unsigned f = (unsigned)(from[i] >> SHIFT_TYPE);
      if (f < 32) mymask |= 1u << f;
    }
  }
  if (run_n && run_t < MAX_AGENT_TYPES) atomicAdd(&sc[run_t], run_n);
  if (mymask) atomicOr(&sm, mymask);
  __syncthreads();
  if (threadIdx.x < MAX_AGENT_TYPES && sc[threadIdx.x])
    atomicAdd(&counts[threadIdx.x], sc[threadIdx.x]);
  if (threadIdx.x == 0 && sm) atomicOr(srcmask, sm);
}

__global__ void k_iota(uint32_t *v, uint64_t n) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = (uint32_t)i;
}

__global__ void k_copy_u64(const uint64_t *a, uint64_t *b, uint64_t n) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}

__global__ void k_flag_type(const uint64_t *to, const uint32_t *ord, uint64_t n,
                            unsigned T, uint32_t *flags) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) flags[j] = ((unsigned)(to[ord[j]] >> SHIFT_TYPE) == T) ? 1u : 0u;
}

__global__ void k_compact_sel(const uint32_t *ord, const uint32_t *flags,
                              const uint32_t *pos, uint64_t n, uint32_t *out) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n && flags[j]) out[pos[j]] = ord[j];
}

__global__ void k_row_keys(const uint64_t *to, const uint32_t *sel, uint64_t m,
                           uint64_t nrows, uint32_t *keys, uint32_t *vals,
                           int *status) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t r = sel ? sel[j] : (uint32_t)j;
  uint64_t nr = to[r] & NR_MASK;
  if (nr == 0 || nr > nrows) {
    atomicExch(status, 101);  // edge to an agent number that does not exist
    nr = 1;
  }
  keys[j] = (uint32_t)(nr - 1);
  vals[j] = r;
}

__global__ void k_hist_rows(const uint32_t *keys, uint64_t m, uint32_t *cnt) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) atomicAdd(&cnt[keys[j]], 1u);
}

__global__ void k_add_old_counts(const uint32_t *old_rp, uint64_t old_nrows,
                                 const uint32_t *newcnt, uint32_t *tot,
                                 uint32_t *oldcnt, uint64_t nrows) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  uint32_t o = 0;
  if (old_rp && r < old_nrows) o = old_rp[r + 1] - old_rp[r];
  oldcnt[r] = o;
  tot[r] = o + newcnt[r];
}

__global__ void k_clamp1(uint32_t *cnt, uint64_t nrows) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < nrows && cnt[r] > 1) cnt[r] = 1;
}

__global__ void k_max_u32(const uint32_t *v, uint64_t n, unsigned *out) {
  unsigned m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    m = max(m, v[i]);
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// destination of old edge k: same offset inside its row of the new CSR
__global__ void k_old_dest(const uint32_t *old_rp, uint64_t old_nrows,
                           uint64_t old_ne, const uint32_t *new_rp,
                           uint32_t *dest) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= old_ne) return;
  // binary search: last r with old_rp[r] <= k
  uint64_t lo = 0, hi = old_nrows;  // old_rp[lo] <= k < old_rp[hi]
  while (hi - lo > 1) {
    uint64_t mid = (lo + hi) >> 1;
    if (old_rp[mid] <= k) lo = mid; else hi = mid;
  }
  dest[k] = new_rp[lo] + (uint32_t)(k - old_rp[lo]);
}

__global__ void k_new_dest(const uint32_t *keys, uint64_t m,
                           const uint32_t *new_rp, const uint32_t *oldcnt,
                           const uint32_t *seg, uint32_t *dest, int dedupe) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  uint32_t r = keys[j];
  uint32_t within = (uint32_t)j - seg[r];
  if (dedupe && (within + oldcnt[r]) > 0) {
    dest[j] = 0xffffffffu;  // HasEdgeOnly keeps a single `true`
    return;
  }
  dest[j] = new_rp[r] + oldcnt[r] + within;
}

__global__ void k_place_src(const uint64_t *from, const uint32_t *rec,
                            const uint32_t *dest, uint64_t m, uint32_t *src,
                            uint8_t *src_type) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t d = dest ? dest[j] : (uint32_t)j;  // no dest: in place order
  if (d == 0xffffffffu) return;
  uint64_t f = from[rec[j]];
  src[d] = (uint32_t)((f & NR_MASK) - 1);
  if (src_type) src_type[d] = (uint8_t)(f >> SHIFT_TYPE);
}

template <class E>
__global__ void k_scatter_col(const E *in, const uint32_t *rec,
                              const uint32_t *dest, uint64_t m, E *out) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t dj = dest ? dest[j] : (uint32_t)j;  // no dest: a gather in place order
  if (dj == 0xffffffffu) return;
  out[dj] = rec ? in[rec[j]] : in[j];
}

__global__ void k_fill_u8(uint8_t *p, uint8_t v, const uint32_t *dest,
                          uint64_t m) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) p[dest ? dest[j] : j] = v;
}

void scatter_column(int esz, const void *in, const uint32_t *rec,
                    const uint32_t *dest, uint64_t m, void *out,
                    cudaStream_t st) {
  if (m == 0) return;
  switch (esz) {
    case 1: k_scatter_col<uint8_t><<<nblk(m), TPB, 0, st>>>((const uint8_t *)in, rec, dest, m, (uint8_t *)out); break;
    case 2: k_scatter_col<uint16_t><<<nblk(m), TPB, 0, st>>>((const uint16_t *)in, rec, dest, m, (uint16_t *)out); break;
    case 4: k_scatter_col<uint32_t><<<nblk(m), TPB, 0, st>>>((const uint32_t *)in, rec, dest, m, (uint32_t *)out); break;
    case 8: k_scatter_col<uint64_t><<<nblk(m), TPB, 0, st>>>((const uint64_t *)in, rec, dest, m, (uint64_t *)out); break;
    default: fail(VG_ERR_ARG, "unsupported field size");
  }
  VG_CUDA(cudaGetLastError());
}

template <class T> struct Tmp {
  T *p = nullptr;
  cudaStream_t st;
  Tmp(uint64_t n, cudaStream_t s) : st(s) {
    VG_CUDA(cudaMallocAsync((void **)&p, std::max<uint64_t>(n, 1) * sizeof(T), st));
  }
  ~Tmp() { if (p) cudaFreeAsync(p, st); }
};

// ------------------------------------------------------ died-edge removal
// an edge stays unless its target or (where sources are kept) its source died
struct DiedView {
  const uint8_t *target, *source[MAX_AGENT_TYPES];  // died flags, null: none of them died
  uint64_t target_n, source_n[MAX_AGENT_TYPES];
};

__device__ __forceinline__ bool edge_stays(const DevCSRView &c, const DiedView &d, uint32_t e) {
  if (!c.src) return true;
  const int t = c.src_type ? (int)c.src_type[e] : c.src_type_const;
  if (t <= 0 || t >= MAX_AGENT_TYPES || !d.source[t]) return true;
  const uint32_t s = c.src[e];
  return s >= d.source_n[t] || !d.source[t][s];
}

// Edges kept in each row (counts; entry nrows: 0), or, with their exclusive
// sums new_rp, the kept edges' columns packed.  A warp takes 32 rows' edges as
// one run (warp_edges), and a group's kept edges by one ballot; they lie one
// behind the other in the packed container too.
struct KeptOut {
  uint32_t *src;
  uint8_t *src_type;
  int npay, psize[MAX_FIELDS];
  void *pay[MAX_FIELDS];
};

template <bool COPY>
__global__ void __launch_bounds__(TPB) k_kept_edges(DevCSRView c, DiedView d, uint32_t *counts,
                                                    const uint32_t *new_rp, KeptOut out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned lane = threadIdx.x & 31;
  uint32_t deg;
  const uint32_t b = row_run(c, i, deg);
  const bool dead = d.target && i < d.target_n && d.target[i];
  const unsigned live = __ballot_sync(0xffffffffu, !dead);
  uint32_t kept = 0;
  const uint64_t row0 = i - lane;
  uint32_t at = COPY && row0 <= c.nrows ? new_rp[row0] : 0u;
  warp_edges(b, deg, [&](uint32_t e, unsigned owner, bool has) {
    const bool keep = has && (live >> owner & 1u) && edge_stays(c, d, e);
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (COPY) {
      if (keep) {
        const uint32_t o = at + __popc(mask & ((1u << lane) - 1u));
        if (out.src) out.src[o] = c.src[e];
        if (out.src_type) out.src_type[o] = c.src_type[e];
        for (int f = 0; f < out.npay; f++) copy_elem(out.psize[f], c.payload[f], e, out.pay[f], o);
      }
      at += __popc(mask);
    } else {
      // this lane's row holds the lanes lo .. hi - 1 of the group
      const uint32_t e0 = e - lane;
      const uint32_t lo = b > e0 ? min(b - e0, 32u) : 0u;
      const uint32_t hi = b + deg > e0 ? min(b + deg - e0, 32u) : 0u;
      const unsigned below_hi = hi >= 32 ? 0xffffffffu : (1u << hi) - 1u;
      const unsigned below_lo = lo >= 32 ? 0xffffffffu : (1u << lo) - 1u;
      kept += __popc(mask & below_hi & ~below_lo);
    }
  });
  if (!COPY && i <= c.nrows) counts[i] = i < c.nrows ? kept : 0u;
}

__global__ void k_new_rowptr(const uint32_t *rp, uint64_t nrows,
                             const uint32_t *keep_scan, uint32_t *out) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r <= nrows) out[r] = keep_scan[rp[r]];
}

__global__ void k_compact_dest(const uint32_t *keep, const uint32_t *scan,
                               uint64_t n, uint32_t *dest) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) dest[k] = keep[k] ? scan[k] : 0xffffffffu;
}

}  // namespace

static void ensure_buf(Sim &s, DevBuf &b, uint64_t bytes, bool slack = false) {
  if (b.bytes < bytes || !b.p)
    b.alloc(std::max<uint64_t>(slack ? bytes + bytes / 8 : bytes, 16), &s.footprint);
}

namespace {
struct RowsFrom {
  const uint32_t *p;
  __device__ __forceinline__ uint32_t operator()(uint64_t i) const { return p[i]; }
};
struct RowsTo {
  uint32_t *p;
  __device__ __forceinline__ void operator()(uint64_t i, uint32_t before, uint32_t) const {
    p[i] = before;
  }
};
}  // namespace

uint64_t csr_edges_total(const EdgeStore &es) {
  uint64_t t = 0;
  for (auto &c : es.csr) t += c.nedges;
  return t;
}

// ---------------------------------------- rebuild from typed records
namespace {
constexpr int BB_TPB = 256;
constexpr uint32_t BB_SPAN = 8192;  // rows counted in shared memory at a time
constexpr uint32_t BB_TILES = 512;  // tiles whose pieces are listed at a time
constexpr uint32_t BB_NONE = 0xFFFFu;
constexpr uint32_t BB_U = 4;         // records per thread of a large span, staged once
constexpr uint32_t BB_FEW = 8;

struct BuildArgs {
  BucketPlan p;
  uint64_t nrows;
  uint32_t span, chunk;
  uint32_t *rp, *src;        // src null: sources are not kept
  const uint32_t *slot_src;  // null: a record's value is its source, else its slot
  int npay;
  int psize[MAX_FIELDS];
  const void *pin[MAX_FIELDS];  // by slot
  void *pout[MAX_FIELDS];
  // the container that add_existing carries over (null: none)
  const uint32_t *old_rp, *old_src;
  uint64_t old_nrows;
  uint32_t old_ne;
  const void *old_pay[MAX_FIELDS];
};

// Rows of the span in shared memory: thread t owns the 4 Q consecutive rows
// from 4 Q t on, as Q chunks of 16 bytes, chunk q of thread t at q ^ (t mod Q)
// so that both the per-thread and the consecutive accesses avoid bank
// conflicts.  Q = 8 for spans of 2048 rows and more, 1 below.
template <int Q>
__device__ __forceinline__ uint32_t bb_slot(uint32_t i) {
  if (Q == 1) return i;
  const uint32_t t = i / (4 * Q), q = (i >> 2) & (Q - 1);
  return t * 4 * Q | ((q ^ (t & (Q - 1))) << 2) | (i & 3u);
}

__device__ __forceinline__ uint32_t bb_reduce(uint32_t v, uint32_t *ws) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
#pragma unroll
  for (int w = 0; w < BB_TPB / 32; w++) t += ws[w];
  return t;
}

// exclusive sum over the block's threads; *total: of all
__device__ __forceinline__ uint32_t bb_scan(uint32_t v, uint32_t *ws, uint32_t *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) ws[w] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w2 = 0; w2 < BB_TPB / 32; w2++) {
    before += w2 < w ? ws[w2] : 0u;
    all += ws[w2];
  }
  *total = all;
  return before + x - v;
}

// the value of the record q at place i
__device__ __forceinline__ uint32_t bb_value(const BucketPlan &p, uint64_t i, uint32_t q) {
  return p.vals ? p.vals[i] : ((uint32_t)i & ~(uint32_t)(BK_TILE - 1)) + (q >> p.shift);
}

// lists the bucket's pieces of the tiles from t0 on (pre: records before each,
// first: its place in its tile); returns their records, *before: the records
// of earlier buckets in these tiles
__device__ __forceinline__ uint32_t bb_pieces(const BucketPlan &p, uint32_t b, uint32_t t0,
                                              uint32_t *pre, uint16_t *first, uint32_t *ws,
                                              uint32_t *before) {
  const uint32_t tid = threadIdx.x;
  uint32_t run = 0, bsum = 0;
#pragma unroll
  for (uint32_t r = 0; r < BB_TILES; r += BB_TPB) {
    const uint32_t t = t0 + r + tid;
    uint32_t len = 0;
    if (t < p.ntiles) {
      const uint16_t *o = p.offs + (uint64_t)t * p.pitch + b;
      const uint32_t o0 = o[0];
      first[r + tid] = (uint16_t)o0;
      len = o[1] - o0;
      bsum += o0;
    }
    uint32_t all;
    pre[r + tid] = run + bb_scan(len, ws, &all);
    run += all;
    if (r + BB_TPB < BB_TILES && t0 + r + BB_TPB >= p.ntiles) break;  // (the rest is not read)
  }
  if (tid == 0) pre[min(BB_TILES, p.ntiles - t0)] = run;
  if (before) *before = bb_reduce(bsum, ws);
  __syncthreads();
  return run;
}

// place of record j of the listed pieces among the tiles' records
__device__ __forceinline__ uint64_t bb_find(const BucketPlan &p, uint32_t t0, uint32_t j,
                                            const uint32_t *pre, const uint16_t *first) {
  uint32_t lo = 0, hi = min(BB_TILES, p.ntiles - t0);  // pre[lo] <= j < pre[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= j) lo = mid;
    else hi = mid;
  }
  return (uint64_t)(t0 + lo) * BK_TILE + first[lo] + (j - pre[lo]);
}

// One block per bucket (vg_bucket.cuh).  The bucket's records, in order, are
// its pieces of the tiles one after the other.  They are staged `chunk` at a
// time, once when all of them fit.
//   Small spans, staged once: each warp ranks its eighth of the records in
// order against counters of its own; the counters' sums over the warps are
// the rows' counts.
//   Large spans, staged once: each thread keeps its records in registers,
// counts them with atomics on 16-bit counters and takes the counters' sums
// as positions.  A row of several records (most of a sparse container's rows
// have at most one) orders them by comparing each with the row's others, up
// to BB_FEW; more are walked as below.
//   Otherwise the records are counted with atomics, in half the span (32-bit
// counters); ranks within 32 records come from match.any, and the first warp
// walks the 32s in order, keeping each row's next position.
// Old edges (add_existing) stay ahead of the new ones in their row.
// Bound: the row pointers' write for a sparse container (67 MB for 16.8 M
// cells), the latency of a block's steps for a dense one (pieces, records,
// ranks, payload: about ten dependent memory accesses).  A bucket of more
// records than a chunk takes 35 ns per 32 of them, one after the other:
// records that crowd into few buckets are placed at that rate.
// Measured, us per launch (and of the tile pass before it): 10^6 records into
// 16.8 M rows 27 (17; the sort by 8 bits of the row and the row pointers
// before it took 77 together), 10^6 and 2*10^6 records with payload into 10^5
// rows 30 on average (16; 64-bit order keys and rows sorted before: 165), 4*10^4
// new records among 10^6 old edges 19.  Blocks per SM: 4, 5, 6, 7, 8 took 28,
// 27, 29, 33, 33 (large spans), 2 to 6 took 58, 33, 33, 33, 30 (small).
template <bool MERGE, int Q>
__device__ __forceinline__ void bucket_build(const BuildArgs &a, uint32_t span, uint32_t chunk) {
  extern __shared__ __align__(16) unsigned char bb_smem[];
  constexpr int BB_WARPS = BB_TPB / 32;
  uint32_t *cnt = (uint32_t *)bb_smem;             // [span] counts, then positions
  uint32_t *val = cnt + max(span, 4u);           // [chunk]
  uint32_t *pos = val + chunk;                   // [chunk]
  uint32_t *pre = pos + chunk;                   // [BB_TILES + 1] records before a piece
  uint16_t *first = (uint16_t *)(pre + BB_TILES + 2);  // [BB_TILES] a piece's place in its tile
  uint16_t *rowl = first + BB_TILES;               // [chunk] row in the span
  uint16_t *rk = rowl + chunk;                   // [chunk] ranks
  uint16_t *wc = rk + chunk;                     // Q == 1: [BB_WARPS][span]
  __shared__ uint32_t ws[BB_WARPS];
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const BucketPlan &p = a.p;
  const uint32_t b = blockIdx.x;
  const uint64_t row0 = (uint64_t)b << p.shift;
  // stages records j0 .. of the listed pieces; returns how many
  auto stage = [&](uint32_t t0, uint32_t j0, uint32_t mr, uint64_t R0) {
    const uint32_t mc = min(chunk, mr - j0);
    for (uint32_t j = tid; j < mc; j += BB_TPB) {
      const uint64_t i = bb_find(p, t0, j0 + j, pre, first);
      const uint32_t q = p.recs[i];
      // (wraps when below the span)
      const uint32_t r = (q & ((1u << p.shift) - 1u)) - (uint32_t)(R0 - row0);
      rowl[j] = (uint16_t)(r < span ? r : BB_NONE);
      val[j] = bb_value(p, i, q);
    }
    __syncthreads();
    return mc;
  };
  uint32_t base = 0, m = 0;  // records of earlier buckets, of this one
  const bool one_list = p.ntiles <= BB_TILES;
  if (one_list) {
    if (p.ntiles) m = bb_pieces(p, b, 0, pre, first, ws, &base);
  } else {
    for (uint32_t t = tid; t < p.ntiles; t += BB_TPB) {
      const uint16_t *o = p.offs + (uint64_t)t * p.pitch + b;
      base += o[0];
      m += (uint32_t)o[1] - o[0];
    }
    base = bb_reduce(base, ws);
    m = bb_reduce(m, ws);
  }
  const uint64_t rows_end = min((unsigned long long)a.nrows,
                                (unsigned long long)(row0 + (1ull << p.shift)));
  const bool once = m <= chunk && one_list && (1ull << p.shift) <= span;
  const bool by_warps = Q == 1 && once;
  if (!once && tid == 0) *(volatile unsigned *)&p.report->crowded = 1;
  unsigned dmax = 0;
  for (uint64_t R0 = row0; R0 < rows_end || R0 == row0; R0 += span) {
    const uint64_t R1 = min((unsigned long long)(R0 + span), (unsigned long long)rows_end);
    const uint32_t nr = R1 > R0 ? (uint32_t)(R1 - R0) : 0u;
    uint32_t mc = 0;
    // warp w's records, by_warps: a whole number of 32s
    uint32_t share = 0;
    if (by_warps) {
      for (uint32_t i = tid; i < BB_WARPS * span / 2; i += BB_TPB) ((uint32_t *)wc)[i] = 0;
      mc = m ? stage(0, 0, m, R0) : 0u;
      __syncthreads();
      share = ((mc + 31) / 32 + BB_WARPS - 1) / BB_WARPS * 32;
      uint16_t *mine = wc + wid * span;
      const uint32_t j1 = min(mc, (wid + 1) * share);
      for (uint32_t j0 = wid * share; j0 < j1; j0 += 32) {
        const uint32_t j = j0 + lane;
        const uint32_t r = j < j1 ? rowl[j] : BB_NONE;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        uint32_t at = 0;
        if (j < j1) at = mine[r];
        __syncwarp();
        if (j < j1) {
          rk[j] = (uint16_t)(at + __popc(peers & lt));
          if ((peers & lt) == 0) mine[r] = (uint16_t)(at + __popc(peers));
        }
        __syncwarp();
      }
      __syncthreads();
      for (uint32_t i = tid; i < span; i += BB_TPB) {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < BB_WARPS; w++) {
          const uint32_t c = wc[w * span + i];
          wc[w * span + i] = (uint16_t)run;
          run += c;
        }
        cnt[i] = run;
      }
      if (span < 4 && tid < 4 && tid >= span) cnt[tid] = 0;
    } else {
      for (uint32_t i = tid; i < max(span, 4u) / 4; i += BB_TPB)
        ((uint4 *)cnt)[i] = make_uint4(0, 0, 0, 0);
      __syncthreads();
      for (uint32_t t0 = 0; t0 < p.ntiles && m; t0 += BB_TILES) {
        const uint32_t mr = one_list ? m : bb_pieces(p, b, t0, pre, first, ws, nullptr);
        for (uint32_t j0 = 0; j0 < mr; j0 += chunk) {
          mc = stage(t0, j0, mr, R0);
          for (uint32_t j = tid; j < mc; j += BB_TPB)
            if (rowl[j] != BB_NONE) atomicAdd(&cnt[bb_slot<Q>(rowl[j])], 1u);
          __syncthreads();
        }
      }
    }
    __syncthreads();
    // counts into exclusive sums
    const uint32_t r_lo = tid * 4 * Q;
    uint4 v[Q];
    uint32_t sum = 0, here;
    if (r_lo < span) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        v[q] = ((uint4 *)cnt)[tid * Q + (q ^ (tid & (Q - 1)))];
        if (MERGE) {
          const uint32_t c[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const uint64_t r = R0 + r_lo + 4 * q + k;
            const uint32_t old = r < a.old_nrows ? a.old_rp[r + 1] - a.old_rp[r] : 0u;
            dmax = max(dmax, r < a.nrows ? c[k] + old : 0u);
          }
        } else {
          dmax = max(dmax, max(max(v[q].x, v[q].y), max(v[q].z, v[q].w)));
        }
        sum += v[q].x + v[q].y + v[q].z + v[q].w;
      }
    }
    uint32_t run = bb_scan(sum, ws, &here);
    if (r_lo < span) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const uint4 c = v[q];
        uint4 e;
        e.x = run;
        e.y = e.x + c.x;
        e.z = e.y + c.y;
        e.w = e.z + c.z;
        run = e.w + c.w;
        ((uint4 *)cnt)[tid * Q + (q ^ (tid & (Q - 1)))] = e;
      }
    }
    __syncthreads();
    if (!MERGE && Q == 8 && nr == span && ((uintptr_t)(a.rp + R0) & 15) == 0) {
      uint4 *out = (uint4 *)(a.rp + R0);
      for (uint32_t c = tid; c < span / 4; c += BB_TPB) {
        uint4 e = ((const uint4 *)cnt)[bb_slot<Q>(4 * c) >> 2];
        e.x += base;
        e.y += base;
        e.z += base;
        e.w += base;
        out[c] = e;
      }
    } else {
      for (uint32_t i = tid; i < nr; i += BB_TPB) {
        uint32_t e = base + cnt[bb_slot<Q>(i)];
        if (MERGE) e += R0 + i < a.old_nrows ? a.old_rp[R0 + i] : a.old_ne;
        a.rp[R0 + i] = e;
      }
    }
    if (MERGE && R0 < a.old_nrows) {
      // old edge k of row r moves up by the new records of the rows before
      const uint64_t O1 = min((unsigned long long)R1, (unsigned long long)a.old_nrows);
      const uint32_t k0 = a.old_rp[R0], k1 = a.old_rp[O1];
      for (uint32_t k = k0 + tid; k < k1; k += BB_TPB) {
        uint32_t lo = 0, hi = (uint32_t)(O1 - R0);  // old_rp[R0 + lo] <= k < old_rp[R0 + hi]
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (a.old_rp[R0 + mid] <= k) lo = mid;
          else hi = mid;
        }
        const uint64_t o = (uint64_t)k + base + cnt[bb_slot<Q>(lo)];
        if (a.src) a.src[o] = a.old_src[k];
        for (int f = 0; f < a.npay; f++) copy_elem(a.psize[f], a.old_pay[f], k, a.pout[f], o);
      }
    }
    // one record into the container
    auto put = [&](uint32_t j, uint32_t at) {
      uint64_t o = (uint64_t)base + at;
      if (MERGE) {
        const uint64_t r = R0 + rowl[j];
        o += r < a.old_nrows ? a.old_rp[r + 1] : a.old_ne;
      }
      const uint32_t u = val[j];
      if (a.src) a.src[o] = a.slot_src ? a.slot_src[u] : u;
      for (int f = 0; f < a.npay; f++) copy_elem(a.psize[f], a.pin[f], u, a.pout[f], o);
    };
    if (by_warps) {
      // in place order, so that consecutive threads write consecutive edges
      for (uint32_t j = tid; j < mc; j += BB_TPB)
        pos[cnt[rowl[j]] + wc[j / share * span + rowl[j]] + rk[j]] = j;
      __syncthreads();
      for (uint32_t at = tid; at < mc; at += BB_TPB) put(pos[at], at);
    } else {
      __syncthreads();
      for (uint32_t t0 = 0; t0 < p.ntiles && m; t0 += BB_TILES) {
        const uint32_t mr = once || one_list ? m : bb_pieces(p, b, t0, pre, first, ws, nullptr);
        for (uint32_t j0 = 0; j0 < mr; j0 += chunk) {
          if (!once) mc = stage(t0, j0, mr, R0);
          const uint32_t groups = (mc + 31) / 32;
          for (uint32_t c = wid; c < groups; c += BB_WARPS) {
            const uint32_t j = c * 32 + lane;
            const uint32_t r = j < mc ? rowl[j] : BB_NONE;
            const unsigned peers = __match_any_sync(0xffffffffu, r);
            if (j < mc) rk[j] = (uint16_t)(__popc(peers & lt) | (__popc(peers) - 1) << 5);
          }
          __syncthreads();
          if (wid == 0) {
            for (uint32_t c = 0; c < groups; c++) {
              const uint32_t j = c * 32 + lane;
              const uint32_t r = j < mc ? rowl[j] : BB_NONE, q = j < mc ? rk[j] : 0u;
              if (__all_sync(0xffffffffu, r == BB_NONE)) continue;  // (other parts of the span)
              const uint32_t sl = r == BB_NONE ? 0u : bb_slot<Q>(r);
              const uint32_t at = cnt[sl];
              __syncwarp();
              if (r != BB_NONE) {
                if ((q & 31u) == 0) cnt[sl] = at + (q >> 5) + 1;
                pos[j] = at + (q & 31u);
              }
              __syncwarp();
            }
          }
          __syncthreads();
          for (uint32_t j = tid; j < mc; j += BB_TPB)
            if (rowl[j] != BB_NONE) put(j, pos[j]);
          __syncthreads();
        }
      }
    }
    base += here;
  }
  if (b + 1 == p.nbuckets && tid == 0) a.rp[a.nrows] = base + (MERGE ? a.old_ne : 0u);
#pragma unroll
  for (int o = 16; o; o >>= 1) dmax = max(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  if (lane == 0 && dmax) atomicMax(a.p.maxdeg, dmax);
}

template <bool MERGE, int Q>
__global__ void __launch_bounds__(BB_TPB, 6) k_bucket_build(const __grid_constant__ BuildArgs a) {
  let_next_start();
  wait_for_previous();
  bucket_build<MERGE, Q>(a, a.span, a.chunk);
}

// out of line: k_bucket_rows' own path keeps its registers
__device__ __noinline__ void bucket_build_apart(const BuildArgs &a, uint32_t span, uint32_t chunk) {
  bucket_build<false, 8>(a, span, chunk);
}

// A bucket of 2048 R rows whose records fit the threads' registers: 16-bit
// counters, the thread's 8 R rows as R chunks of 16 bytes (chunk q at an
// exclusive-or with the thread's number that keeps 16-byte accesses of eight
// threads apart).
template <int R>
__device__ __forceinline__ uint32_t br_chunk(uint32_t t, uint32_t q) {
  return t * R + (R == 1 ? 0u : q ^ (t / (8 / R) & (R - 1)));
}
template <int R>
__device__ __forceinline__ uint32_t br_slot(uint32_t row) {
  return br_chunk<R>(row / (8 * R), row / 8 & (R - 1)) * 8 + (row & 7u);
}

template <int R>
__global__ void __launch_bounds__(BB_TPB, 5) k_bucket_rows(const __grid_constant__ BuildArgs a) {
  constexpr uint32_t SPAN = 2048 * R;
  extern __shared__ __align__(16) unsigned char bb_smem[];
  uint4 *cnt4 = (uint4 *)bb_smem;                      // [BB_TPB R]
  uint16_t *cnt = (uint16_t *)cnt4;                    // [SPAN], by br_slot
  uint32_t *pre = (uint32_t *)(cnt4 + BB_TPB * R);     // [BB_TILES + 2]
  uint16_t *first = (uint16_t *)(pre + BB_TILES + 2);  // [BB_TILES]
  uint16_t *lst = first + BB_TILES;                    // [BB_U BB_TPB]
  uint16_t *pos = lst + BB_U * BB_TPB;                 // [BB_U BB_TPB]
  __shared__ uint32_t ws[BB_TPB / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, b = blockIdx.x;
  const BucketPlan &p = a.p;
  uint32_t base = 0, m = 0;
  let_next_start();
#pragma unroll
  for (int q = 0; q < R; q++) cnt4[tid + BB_TPB * q] = make_uint4(0, 0, 0, 0);
  wait_for_previous();  // (launched beside the end of k_bucket_tiles)
  if (p.ntiles && p.ntiles <= BB_TILES) m = bb_pieces(p, b, 0, pre, first, ws, &base);
  if (p.ntiles > BB_TILES || m > BB_U * BB_TPB || 1u << p.shift != SPAN) {
    __syncthreads();
    if (tid == 0) *(volatile unsigned *)&p.report->crowded = 1;
    bucket_build_apart(a, SPAN / 2, 512);
    return;
  }
  __syncthreads();
  const uint64_t R0 = (uint64_t)b << p.shift;
  uint32_t row[BB_U], val[BB_U], arr[BB_U];
#pragma unroll
  for (int u = 0; u < BB_U; u++) {
    const uint32_t j = tid + BB_TPB * u;
    row[u] = BB_NONE;
    if (j < m) {
      const uint64_t i = bb_find(p, 0, j, pre, first);
      const uint32_t q = p.recs[i];
      row[u] = q & (SPAN - 1);
      val[u] = bb_value(p, i, q);
    }
  }
#pragma unroll
  for (int u = 0; u < BB_U; u++)
    if (row[u] != BB_NONE) {
      const uint32_t sl = br_slot<R>(row[u]), sh = 16 * (sl & 1u);
      arr[u] = atomicAdd((uint32_t *)cnt + (sl >> 1), 1u << sh) >> sh & 0xffffu;
    }
  __syncthreads();
  // exclusive sums of the thread's 8 R counters, two to a word
  uint32_t c[4 * R], sum = 0, top = 0;
#pragma unroll
  for (int q = 0; q < R; q++) {
    const uint4 v = cnt4[br_chunk<R>(tid, q)];
    c[4 * q] = v.x;
    c[4 * q + 1] = v.y;
    c[4 * q + 2] = v.z;
    c[4 * q + 3] = v.w;
  }
#pragma unroll
  for (int k = 0; k < 4 * R; k++) {
    sum += c[k];  // (the two halves' sums stay below 2^16)
    top = __vmaxu2(top, c[k]);
  }
  const uint32_t dmax = max(top & 0xffffu, top >> 16);
  uint32_t all;
  uint32_t run = bb_scan((sum & 0xffffu) + (sum >> 16), ws, &all);
#pragma unroll
  for (int k = 0; k < 4 * R; k++) {
    const uint32_t lo = c[k] & 0xffffu, hi = c[k] >> 16;
    c[k] = run | (run + lo) << 16;
    run += lo + hi;
  }
#pragma unroll
  for (int q = 0; q < R; q++)
    cnt4[br_chunk<R>(tid, q)] = make_uint4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
  // 0: no row of two records, 1: none of more than BB_FEW, 2 or 3: some
  const int crowd = __syncthreads_or(dmax > BB_FEW ? 2 : dmax > 1 ? 1 : 0);
  const uint32_t nr = a.nrows > R0 ? (uint32_t)min((unsigned long long)SPAN,
                                                   (unsigned long long)(a.nrows - R0)) : 0u;
  // four rows per thread and round; a round's 1024 rows lie one behind the
  // other in either layout
  const uint2 *from = (const uint2 *)(cnt + br_slot<R>(4 * tid));
  uint32_t *out = a.rp + R0 + 4 * tid;
  auto sums = [&](int k) {
    const uint2 v = from[k * BB_TPB];
    return make_uint4(base + (v.x & 0xffffu), base + (v.x >> 16), base + (v.y & 0xffffu),
                      base + (v.y >> 16));
  };
  if (nr == SPAN) {
#pragma unroll
    for (int k = 0; k < 2 * R; k++) *(uint4 *)(out + k * 4 * BB_TPB) = sums(k);
  } else {
    for (int k = 0; k < 2 * R; k++) {
      const uint4 e = sums(k);
      const uint32_t r = 4 * (tid + BB_TPB * k);
      uint32_t *q = out + k * 4 * BB_TPB;
      if (r < nr) q[0] = e.x;
      if (r + 1 < nr) q[1] = e.y;
      if (r + 2 < nr) q[2] = e.z;
      if (r + 3 < nr) q[3] = e.w;
    }
  }
  if (b + 1 == p.nbuckets && tid == 0) a.rp[a.nrows] = base + m;
  uint32_t at[BB_U];
  if (crowd < 2) {
    if (crowd) {
#pragma unroll
      for (int u = 0; u < BB_U; u++)
        if (row[u] != BB_NONE) lst[cnt[br_slot<R>(row[u])] + arr[u]] = (uint16_t)(tid + BB_TPB * u);
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < BB_U; u++)
      if (row[u] != BB_NONE) {
        at[u] = cnt[br_slot<R>(row[u])];
        if (crowd) {
          const uint32_t end = row[u] + 1 < SPAN ? cnt[br_slot<R>(row[u] + 1)] : m;
          uint32_t rank = 0;
          for (uint32_t k = at[u]; k < end; k++) rank += lst[k] < tid + BB_TPB * u;
          at[u] += rank;
        }
      }
  } else {
#pragma unroll
    for (int u = 0; u < BB_U; u++) lst[tid + BB_TPB * u] = (uint16_t)row[u];
    __syncthreads();
    if (tid < 32) {
      const unsigned lt = (1u << lane) - 1u;
      for (uint32_t j = lane; j - lane < m; j += 32) {
        const uint32_t r = lst[j];
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        const uint32_t sl = r == BB_NONE ? 0u : br_slot<R>(r);
        const uint32_t first_at = cnt[sl];
        __syncwarp();
        if (r != BB_NONE) {
          pos[j] = (uint16_t)(first_at + __popc(peers & lt));
          if ((peers & lt) == 0) cnt[sl] = (uint16_t)(first_at + __popc(peers));
        }
        __syncwarp();
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < BB_U; u++)
      if (row[u] != BB_NONE) at[u] = pos[tid + BB_TPB * u];
  }
  // the values in place order (over the lists, which nobody reads any more),
  // so that consecutive threads write consecutive edges
  __syncthreads();
  uint32_t *byplace = pre;  // [BB_U BB_TPB] 32-bit words over pre, first and lst
#pragma unroll
  for (int u = 0; u < BB_U; u++)
    if (row[u] != BB_NONE) byplace[at[u]] = val[u];
  __syncthreads();
  for (uint32_t k = tid; k < m; k += BB_TPB) {
    const uint64_t o = (uint64_t)base + k;
    const uint32_t v = byplace[k];
    if (a.src) a.src[o] = a.slot_src ? a.slot_src[v] : v;
    for (int f = 0; f < a.npay; f++) copy_elem(a.psize[f], a.pin[f], v, a.pout[f], o);
  }
  unsigned d = dmax;
#pragma unroll
  for (int o = 16; o; o >>= 1) d = max(d, __shfl_xor_sync(0xffffffffu, d, o));
  if (lane == 0 && d) atomicMax(a.p.maxdeg, d);
}

// ------------------------------------- typed rebuild by a radix sort
// For records that crowd into few buckets, that are too many for the buckets'
// blocks, or of which it is not known yet (plan_buckets).
// Keys and values of the slots (holes: key nrows, behind every row); the
// kernel also counts the keys' 8-bit digits for the sort's passes (its
// upfront count: per block in shared memory, then added to
// digit_counts[256 p + digit]).
__global__ void k_typed_keys(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ in,
                             uint64_t n, uint64_t nrows, uint32_t *__restrict__ keys,
                             uint32_t *__restrict__ vals, uint32_t *digit_counts, int passes) {
  __shared__ uint32_t h[4 * 256];
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  // four records per thread and round, their loads issued before the
  // shared-memory counts (which would otherwise order each load after the
  // previous record's atomics)
  constexpr int U = 4;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k0 < n; k0 += U * stride) {
    uint32_t r[U], v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t k = k0 + u * stride;
      r[u] = k < n ? rows[k] : 0u;
      v[u] = k < n && in ? in[k] : (uint32_t)k;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t k = k0 + u * stride;
      if (k >= n) break;
      const uint32_t key = r[u] == BK_HOLE ? (uint32_t)nrows : r[u];
      keys[k] = key;
      vals[k] = v[u];
      for (int p = 0; p < passes; p++) atomicAdd(&h[p * 256 + ((key >> (8 * p)) & 255u)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
    if (h[i]) atomicAdd(digit_counts + i, h[i]);
}

// row_ptr of the rows 0..nrows from the sorted row keys: rp[r] = the
// number of keys below r.  Rows are cut into spans of RP_ROWS, one block
// each; a first pass over the records finds, for every span boundary
// j * RP_ROWS, the first record at or above it (record k owns the boundaries
// in (keys[k-1], keys[k]]).  In the block, the last record of each row's run
// stores its end position (relative to the span's first record) at the
// row's slot in shared memory -- one plain store per non-empty row, however
// long the run.  Since the ends grow with the row, rp of a row is the
// largest end stored before it: an exclusive max-scan (each thread 32
// consecutive rows, then across the threads), which also gives every
// non-empty row's length for the block's largest degree.  The rows leave
// shared memory as coalesced 16-byte stores.  Shared rows are swizzled in
// 16-byte chunks (chunk q of thread t at q ^ (t & 7)) so that both the
// per-thread and the per-warp access patterns avoid bank conflicts.
constexpr uint32_t RP_ROWS = 8192;
constexpr uint32_t RP_PER_THREAD = RP_ROWS / TPB;  // 32

__global__ void k_rp_bounds(const uint32_t *keys, uint64_t n, uint64_t nbr, uint32_t *bstart) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k > n) return;
  const uint64_t jlo = k == 0 ? 0 : (uint64_t)keys[k - 1] / RP_ROWS + 1;
  const uint64_t jhi = k == n ? nbr : (uint64_t)keys[k] / RP_ROWS;
  for (uint64_t j = jlo; j <= jhi; j++) bstart[j] = (uint32_t)k;
}

// shared word of row i of the span (32 rows per thread, 8 chunks of 4)
__device__ __forceinline__ uint32_t rp_slot(uint32_t i) {
  const uint32_t t = i >> 5, q = (i >> 2) & 7u;
  return (t << 5) | ((q ^ (t & 7u)) << 2) | (i & 3u);
}

__global__ void __launch_bounds__(TPB) k_rp_fill(const uint32_t *keys, uint64_t nrows,
                                                 const uint32_t *bstart, uint32_t *rp,
                                                 unsigned *maxdeg) {
  __shared__ __align__(16) uint32_t E[RP_ROWS];
  __shared__ uint32_t ws[32];
  const uint32_t tid = threadIdx.x;
  const uint64_t R0 = (uint64_t)blockIdx.x * RP_ROWS;
  const uint64_t R1 = R0 + RP_ROWS < nrows + 1 ? R0 + RP_ROWS : nrows + 1;
  const uint32_t k0 = bstart[blockIdx.x], k1 = bstart[blockIdx.x + 1];
  uint4 *E4 = reinterpret_cast<uint4 *>(E);
  for (uint32_t i = tid; i < RP_ROWS / 4; i += TPB) E4[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  // (eight records in flight per thread: a crowded span is one block's work,
  // and one at a time took 300 ns each round; keys from nrows on are slots
  // without a record, and no key of another span is stored whatever the order)
  constexpr int U = 8;
  const uint32_t rows = (uint32_t)(min((unsigned long long)R1, (unsigned long long)nrows) - R0);
  for (uint32_t kk = k0 + tid; kk < k1; kk += U * TPB) {
    uint32_t key[U], next[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k = kk + u * TPB;
      key[u] = k < k1 ? keys[k] : 0u;
      next[u] = k + 1 < k1 ? keys[k + 1] : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k = kk + u * TPB;
      const uint32_t row = key[u] - (uint32_t)R0;
      if (k < k1 && next[u] != key[u] && row < rows) E[rp_slot(row)] = k + 1 - k0;
    }
  }
  __syncthreads();
  // pass 1: the largest end in the thread's 32 rows (its last stored end)
  uint4 v[RP_PER_THREAD / 4];
  uint32_t m = 0;
#pragma unroll
  for (uint32_t q = 0; q < RP_PER_THREAD / 4; q++) {
    v[q] = E4[(tid << 3) | (q ^ (tid & 7u))];
    m = max(m, max(max(v[q].x, v[q].y), max(v[q].z, v[q].w)));
  }
  // exclusive max-scan over the threads
  const uint32_t lane = tid & 31, wid = tid >> 5;
  uint32_t incl = m;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl = max(incl, y);
  }
  if (lane == 31) ws[wid] = incl;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t w2 = 0; w2 < wid; w2++) before = max(before, ws[w2]);
  const uint32_t excl_lane = __shfl_up_sync(0xffffffffu, incl, 1);
  uint32_t run = max(before, lane ? excl_lane : 0u);
  // pass 2: rp of each row = the largest end before it; a row's length is
  // its end minus that (0 for rows without an end: max(e, run) = run);
  // rows at or beyond nrows hold no end
  unsigned dmax = 0;
#pragma unroll
  for (uint32_t q = 0; q < RP_PER_THREAD / 4; q++) {
    uint32_t o0, o1, o2, o3, t;
    t = max(v[q].x, run); dmax = max(dmax, t - run); o0 = k0 + run; run = t;
    t = max(v[q].y, run); dmax = max(dmax, t - run); o1 = k0 + run; run = t;
    t = max(v[q].z, run); dmax = max(dmax, t - run); o2 = k0 + run; run = t;
    t = max(v[q].w, run); dmax = max(dmax, t - run); o3 = k0 + run; run = t;
    v[q] = make_uint4(o0, o1, o2, o3);
  }
#pragma unroll
  for (uint32_t q = 0; q < RP_PER_THREAD / 4; q++) E4[(tid << 3) | (q ^ (tid & 7u))] = v[q];
  __syncthreads();
  const uint32_t nr = (uint32_t)(R1 - R0);
  if (nr == RP_ROWS && ((uintptr_t)(rp + R0) & 15) == 0) {
    uint4 *out = reinterpret_cast<uint4 *>(rp + R0);
    for (uint32_t c = tid; c < RP_ROWS / 4; c += TPB)
      out[c] = E4[((c >> 3) << 3) | ((c & 7u) ^ ((c >> 3) & 7u))];
  } else {
    for (uint32_t i = tid; i < nr; i += TPB) rp[R0 + i] = E[rp_slot(i)];
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) dmax = max(dmax, __shfl_xor_sync(0xffffffffu, dmax, off));
  if (lane == 0 && dmax) atomicMax(maxdeg, dmax);
}

// largest number of records in a bucket of 2^shift rows, reported to the host
__global__ void __launch_bounds__(1024) k_bucket_load(const uint32_t *rp, uint64_t nrows,
                                                      uint32_t shift, uint32_t nbuckets,
                                                      uint32_t gen, RebuildReport *report) {
  __shared__ unsigned top;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < nbuckets; b += 1024) {
    const uint64_t r0 = (uint64_t)b << shift, r1 = min((unsigned long long)nrows, (unsigned long long)(r0 + (1ull << shift)));
    atomicMax(&top, rp[r1] - rp[r0]);
  }
  __syncthreads();
  if (threadIdx.x == 0)
    *(volatile unsigned long long *)&report->load = (unsigned long long)gen << 32 | top;
}

// the sorted records into the container's columns (old edges stay ahead)
__global__ void k_place_sorted(const uint32_t *keys, const uint32_t *vals, uint64_t n, BuildArgs a) {
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n || keys[j] >= a.nrows) return;
  uint64_t o = j;
  if (a.old_rp) o += keys[j] < a.old_nrows ? a.old_rp[keys[j] + 1] : a.old_ne;
  const uint32_t v = vals[j];
  if (a.src) a.src[o] = a.slot_src ? a.slot_src[v] : v;
  for (int f = 0; f < a.npay; f++) copy_elem(a.psize[f], a.pin[f], v, a.pout[f], o);
}

// row pointers of old and new edges together
__global__ void k_merge_rows(const uint32_t *new_rp, BuildArgs a) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned deg = 0;
  if (r <= a.nrows) {
    const uint32_t o0 = r < a.old_nrows ? a.old_rp[r] : a.old_ne;
    a.rp[r] = o0 + new_rp[r];
    if (r < a.nrows) {
      const uint32_t o1 = r < a.old_nrows ? a.old_rp[r + 1] : a.old_ne;
      deg = o1 - o0 + new_rp[r + 1] - new_rp[r];
    }
  }
  deg = __reduce_max_sync(0xffffffffu, deg);
  if ((threadIdx.x & 31) == 0 && deg) atomicMax(a.p.maxdeg, deg);
}

__global__ void k_merge_old(const uint32_t *new_rp, BuildArgs a) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.old_ne) return;
  uint64_t lo = 0, hi = a.old_nrows;  // old_rp[lo] <= k < old_rp[hi]
  while (hi - lo > 1) {
    const uint64_t mid = (lo + hi) >> 1;
    if (a.old_rp[mid] <= k) lo = mid;
    else hi = mid;
  }
  const uint64_t o = k + new_rp[lo];
  if (a.src) a.src[o] = a.old_src[k];
  for (int f = 0; f < a.npay; f++) copy_elem(a.psize[f], a.old_pay[f], k, a.pout[f], o);
}

}  // namespace

uint32_t csr_max_degree(Sim &s, CSR &c) {
  if (c.max_degree_pending) {
    s.fetch(&c.max_degree, c.d_max_degree.p, 4);
    c.max_degree_pending = false;
  }
  return c.max_degree;
}

void forget_record_spread(Sim &s) {
  for (auto &es : s.edges)
    for (auto &c : es.csr)
      if (c.rebuild) c.rebuild->forget();
}

// Buckets of about 512 records, 1024 rows or 1024 old edges carried over,
// whichever asks for more of them, up to BK_MAX (the chip holds about 700
// blocks at a time: fewer buckets leave it idle), each of at most BB_SPAN
// rows.  The buckets take a rebuild when every bucket's records fit its
// block's stage: a bucket that does not is placed at 5 ns per record by that
// one block (10^6 records in one cell: 5.1 ms, the sort 0.33).  So the sort
// takes rebuilds of more rows or records than that, and every rebuild until
// one with the same sizes has reported its largest bucket; the buckets take
// the following ones until a block reports that its bucket did not fit, or
// the agents are written from outside.  The reports are read without waiting.
// Measured, us per walker step, buckets and sort: 10^6 walkers on 4096^2
// cells 49 and 94, on 1024^2 44 and 90, 10^5 on 1000 x 800 20 and 59, 10^4 on
// 4096^2 32 and 64; 10^6 on 9000^2 476 and 164, 9*10^6 on 3000^2 661 and 438;
// 10^6 on a tenth, a hundredth of 4096^2 148 and 98, 1060 and 143.
BucketPlan plan_buckets(Sim &s, int e, int T, uint64_t n, bool vals) {
  EdgeStore &es = s.edges[e];
  if (es.csr.size() < (size_t)MAX_AGENT_TYPES) es.csr.resize(MAX_AGENT_TYPES);
  CSR &c = es.csr[T];
  if (!c.rebuild) c.rebuild.reset(new RebuildCache());
  RebuildCache &rc = *c.rebuild;
  if (!s.reports_host) {
    const size_t bytes = MAX_EDGE_TYPES * MAX_AGENT_TYPES * sizeof(RebuildReport);
    void *h = nullptr, *d = nullptr;
    VG_CUDA(cudaHostAlloc(&h, bytes, cudaHostAllocMapped));
    std::memset(h, 0, bytes);
    s.reports_host = (RebuildReport *)h;
    VG_CUDA(cudaHostGetDevicePointer(&d, h, 0));
    s.reports_dev = (RebuildReport *)d;
  }
  const uint64_t nrows = std::max<uint64_t>(s.agents[T - 1].n, 1);
  auto buckets = [&](uint32_t shift) { return (nrows + (1ull << shift) - 1) >> shift; };
  const uint64_t load = std::max<uint64_t>({n / 512, nrows / 1024,
                                            es.add_existing ? c.nedges / 1024 : 0});
  const uint64_t want = std::min<uint64_t>(BK_MAX, std::max<uint64_t>(1, load));
  BucketPlan p;
  while (buckets(p.shift) > want) p.shift++;
  while (p.shift > 0 && (1u << p.shift) > BB_SPAN && buckets(p.shift - 1) <= BK_MAX) p.shift--;
  p.n = n;
  p.nbuckets = (uint32_t)buckets(p.shift);
  p.ntiles = (uint32_t)((n + BK_TILE - 1) / BK_TILE);
  p.pitch = (p.nbuckets + 4) & ~3u;
  // (small spans stage 2048 records, large ones keep BB_U per thread)
  p.limit = 1u << p.shift >= 2048 ? (es.add_existing ? 1024 : BB_U * BB_TPB) : 2048;
  ensure_buf(s, c.d_max_degree, 4);
  p.maxdeg = c.d_max_degree.as<unsigned>();
  p.report = s.reports_dev + e * MAX_AGENT_TYPES + T;
  volatile RebuildReport *rep = s.reports_host + e * MAX_AGENT_TYPES + T;
  const bool same = rc.known_rows == nrows && rc.known_buckets == p.nbuckets &&
                    n <= rc.known_n + rc.known_n / 16;
  if (!same) {
    rc.forget();
  } else if (rc.known) {
    if (rep->crowded) rc.forget();
  } else {
    const uint64_t load = rep->load;
    const uint32_t gen = (uint32_t)(load >> 32);
    if ((int32_t)(gen - rc.unknown_gen) > 0 && (int32_t)(rc.sort_gen - gen) >= 0 &&
        (uint32_t)load <= p.limit - p.limit / 8) {
      rc.known = true;
      rep->crowded = 0;
    }
  }
  p.fits = 1u << p.shift <= BB_SPAN && p.ntiles <= BB_TILES && n <= (uint64_t)p.nbuckets * p.limit;
  p.sorted = !rc.known || !p.fits;
  // (at most one bucket's records: nothing to be known)
  if (n <= p.limit && 1u << p.shift <= BB_SPAN) p.sorted = false;
  if (p.sorted) {
    rc.known_n = n;
    rc.known_rows = nrows;
    rc.known_buckets = p.nbuckets;
    return p;
  }
  ensure_buf(s, rc.recs, (uint64_t)p.ntiles * BK_TILE * 4, true);
  if (vals) ensure_buf(s, rc.vals, (uint64_t)p.ntiles * BK_TILE * 4, true);
  ensure_buf(s, rc.offs, (uint64_t)p.ntiles * p.pitch * 2, true);
  p.recs = rc.recs.as<uint32_t>();
  p.vals = vals ? rc.vals.as<uint32_t>() : nullptr;
  p.offs = rc.offs.as<uint16_t>();
  if (!p.ntiles) VG_CUDA(cudaMemsetAsync(p.maxdeg, 0, 4, s.stream));
  return p;
}

// The rows of the records sorted, row pointers from the sorted rows, then the
// records' columns; a plain container (sources only, nothing carried over)
// has its source column carried through the sort, and its launch sequence
// replayed from a recorded graph.
static void build_sorted(Sim &s, CSR &c, const EdgeAppend &ap, BuildArgs &a, bool merge) {
  cudaStream_t st = s.stream;
  RebuildCache &rc = *c.rebuild;
  const uint64_t n = a.p.n, nrows = a.nrows;
  const bool plain = !merge && a.npay == 0 && a.src && !ap.holes;
  const int bits = bits_for(ap.holes ? nrows : nrows ? nrows - 1 : 0);
  const uint64_t nbr = (nrows + 1 + RP_ROWS - 1) / RP_ROWS;
  const uint64_t sort_bytes = radix_sort_scratch_bytes(n, 4, bits);
  ensure_buf(s, rc.keys, std::max<uint64_t>(n, 1) * 4, true);
  if (!plain) ensure_buf(s, rc.vals, std::max<uint64_t>(n, 1) * 4, true);
  ensure_buf(s, rc.bstart, (nbr + 1) * 4, true);
  if (merge) ensure_buf(s, rc.new_rp, (nrows + 1) * 4, true);
  if (sort_bytes) ensure_buf(s, rc.sort, sort_bytes, true);
  uint32_t *keys = rc.keys.as<uint32_t>();
  uint32_t *vals = plain ? a.src : rc.vals.as<uint32_t>();
  uint32_t *rp = merge ? rc.new_rp.as<uint32_t>() : a.rp;
  const uint32_t *rows = ap.to.as<uint32_t>(), *in = a.slot_src ? nullptr : ap.from.as<uint32_t>();
  auto enqueue = [&]() {
    VG_CUDA(cudaMemsetAsync(a.p.maxdeg, 0, 4, st));
    if (n) {
      const int passes = sort_bytes ? std::min((bits + 7) / 8, 4) : 0;
      uint32_t *dc = radix_sort_digit_counts(rc.sort.p);
      if (passes) VG_CUDA(cudaMemsetAsync(dc, 0, (size_t)passes * 256 * 4, st));
      k_typed_keys<<<std::min<unsigned>(nblk(n), 152 * 4), TPB, 0, st>>>(rows, in, n, nrows, keys,
                                                                        vals, dc, passes);
      radix_sort_pairs_u32_in(keys, vals, n, bits, st, s.d_status.as<int>(), rc.sort.p, passes > 0);
    }
    k_rp_bounds<<<nblk(n + 1), TPB, 0, st>>>(keys, n, nbr, rc.bstart.as<uint32_t>());
    k_rp_fill<<<(unsigned)nbr, TPB, 0, st>>>(keys, nrows, rc.bstart.as<uint32_t>(), rp,
                                             a.p.maxdeg);
    VG_CUDA(cudaGetLastError());
  };
  // the launch sequence, a function of these arguments only
  const std::vector<uint64_t> args = {(uint64_t)rows, (uint64_t)in,   n,
                                      nrows,          (uint64_t)rp,   (uint64_t)vals,
                                      (uint64_t)keys, (uint64_t)rc.sort.p, (uint64_t)rc.bstart.p,
                                      (uint64_t)a.p.maxdeg, (uint64_t)s.d_status.p, (uint64_t)bits};
  const bool graphable = st != nullptr && st != cudaStreamLegacy && st != cudaStreamPerThread;
  if (rc.exec && args == rc.graph_args) {
    VG_CUDA(cudaGraphLaunch(rc.exec, st));
  } else if (graphable && args == rc.last) {
    // the same rebuild twice in a row: record it once, replay from now on
    if (rc.exec) {
      cudaGraphExecDestroy(rc.exec);
      rc.exec = nullptr;
      rc.graph_args.clear();
    }
    cudaGraph_t g = nullptr;
    VG_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    try {
      enqueue();
    } catch (...) {
      cudaStreamEndCapture(st, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    VG_CUDA(cudaStreamEndCapture(st, &g));
    const cudaError_t ie = cudaGraphInstantiate(&rc.exec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) rc.exec = nullptr;
    VG_CUDA(ie);
    rc.graph_args = args;
    VG_CUDA(cudaGraphLaunch(rc.exec, st));
  } else {
    enqueue();
  }
  rc.last = args;
  rc.sort_gen++;
  // (the first two rebuilds after what was known ended, then every eighth)
  const uint32_t since = rc.sort_gen - rc.unknown_gen;
  if (nrows && a.p.fits && (since <= 2 || since % 8 == 0))
    k_bucket_load<<<1, 1024, 0, st>>>(rp, nrows, a.p.shift, a.p.nbuckets, rc.sort_gen, a.p.report);
  if (merge) {
    VG_CUDA(cudaMemsetAsync(a.p.maxdeg, 0, 4, st));
    k_merge_rows<<<nblk(nrows + 1), TPB, 0, st>>>(rp, a);
    if (a.old_ne) k_merge_old<<<nblk(a.old_ne), TPB, 0, st>>>(rp, a);
  }
  if (!plain && n) k_place_sorted<<<nblk(n), TPB, 0, st>>>(keys, vals, n, a);
  VG_CUDA(cudaGetLastError());
}

static void launch_buckets(const BuildArgs &a, bool merge, cudaStream_t st) {
  // shared memory of bucket_build and of k_bucket_rows<rows / 2048>
  auto general = [](uint64_t span, uint64_t chunk, bool big) {
    return (size_t)((std::max<uint64_t>(span, 4) + 2 * chunk + BB_TILES + 2) * 4 +
                    (BB_TILES + 2 * chunk) * 2 + (big ? 0 : BB_TPB / 32 * span * 2) + 16);
  };
  const bool big = a.span >= 2048;
  size_t smem = general(a.span, a.chunk, big);
  void (*k)(const BuildArgs);
  if (merge) {
    k = big ? k_bucket_build<true, 8> : k_bucket_build<true, 1>;
  } else if (!big) {
    k = k_bucket_build<false, 1>;
  } else {
    k = a.span == 2048 ? k_bucket_rows<1> : a.span == 4096 ? k_bucket_rows<2> : k_bucket_rows<4>;
    smem = std::max<size_t>(general(a.span / 2, 512, true),
                            a.span * 2 + (BB_TILES + 2) * 4 + BB_TILES * 2 + 2 * BB_U * BB_TPB * 2);
  }
  static const bool ok = [] {
    bool r = true;
    for (auto f : {k_bucket_build<true, 8>, k_bucket_build<true, 1>, k_bucket_build<false, 1>,
                   k_bucket_rows<1>, k_bucket_rows<2>, k_bucket_rows<4>})
      r = r && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) ==
                   cudaSuccess;
    return r;
  }();
  if (!ok) fail(VG_ERR_CUDA, "cannot reserve the rebuild's shared memory");
  launch_dependent(k, a.p.nbuckets, BB_TPB, smem, st, a);
  VG_CUDA(cudaGetLastError());
}

void build_csr_typed(Sim &s, int e, EdgeAppend &ap) {
  s.csr_epoch++;
  const EdgeTypeDesc &ed = s.model->et(e);
  EdgeStore &es = s.edges[e];
  cudaStream_t st = s.stream;
  const int T = ap.target_type;
  const uint64_t n = ap.fixed_count, nrows = s.agents[T - 1].n;
  const int nf = ed.stores_payload() ? (int)ed.fields.size() : 0;
  BuildArgs a{};
  const bool vals = nf == 0 && ed.stores_src();  // (else a record's slot says where to look)
  a.p = ap.planned ? ap.plan : plan_buckets(s, e, T, n, vals);
  if (!es.add_existing)
    for (int U = 1; U < (int)es.csr.size(); U++)
      if (U != T && es.csr[U].row_ptr.p) es.csr[U] = CSR();
  CSR &c = es.csr[T];
  RebuildCache &rc = *c.rebuild;
  if (!ap.tiled) {
    if (a.p.sorted) {
      // (build_sorted)
    } else if (vals) {
      launch_bucket_tiles(SlotSource<true>{ap.to.as<uint32_t>(), ap.from.as<uint32_t>()}, a.p, st);
    } else {
      launch_bucket_tiles(SlotSource<false>{ap.to.as<uint32_t>(), nullptr}, a.p, st);
    }
    if (!vals) a.slot_src = ap.from.as<uint32_t>();
  }
  // without old edges to carry over, the previous container's buffers are
  // written in place (the stream orders its readers before); otherwise the
  // two containers take turns
  const bool merge = es.add_existing && c.row_ptr.p;
  const uint64_t old_ne = merge ? c.nedges : 0, ne_max = n + old_ne;
  DevBuf &rp = merge ? rc.row_ptr : c.row_ptr, &src = merge ? rc.src : c.src;
  std::vector<DevBuf> &pay = merge ? rc.payload : c.payload;
  ensure_buf(s, rp, (nrows + 1) * 4, merge);
  if (ed.stores_src()) ensure_buf(s, src, ne_max * 4, true);
  pay.resize(nf);
  for (int f = 0; f < nf; f++) ensure_buf(s, pay[f], ne_max * ed.fields[f].size, true);
  c.src_type.release();
  a.nrows = nrows;
  a.span = std::min<uint32_t>(1u << std::min(a.p.shift, 13u), BB_SPAN);
  a.chunk = a.span >= 2048 ? 1024 : 2048;
  a.rp = rp.as<uint32_t>();
  a.src = ed.stores_src() ? src.as<uint32_t>() : nullptr;
  a.npay = nf;
  for (int f = 0; f < nf; f++) {
    a.psize[f] = ed.fields[f].size;
    a.pin[f] = ap.payload[f].p;
    a.pout[f] = pay[f].p;
  }
  if (merge) {
    a.old_rp = c.row_ptr.as<uint32_t>();
    a.old_src = c.src.as<uint32_t>();
    a.old_nrows = c.nrows;
    a.old_ne = (uint32_t)old_ne;
    for (int f = 0; f < nf; f++) a.old_pay[f] = c.payload[f].p;
  }
  if (a.p.sorted) build_sorted(s, c, ap, a, merge);
  else launch_buckets(a, merge, st);
  uint64_t ne = ne_max;
  if (ap.holes) {
    uint32_t h = 0;
    s.fetch(&h, rp.as<uint32_t>() + nrows, 4);
    ne = h;
  }
  if (merge) {
    std::swap(c.row_ptr, rc.row_ptr);
    std::swap(c.src, rc.src);
    std::swap(c.payload, rc.payload);
  }
  if (!ed.stores_src()) c.src.release();
  c.nrows = nrows;
  c.nedges = ne;
  c.src_type_const = ed.stores_src() ? ap.src_type : 0;
  c.max_degree_pending = true;
  c.schedule_valid = false;
  c.unit_grid_weights = -1;
}

void build_csr_from_records(Sim &s, int e, const uint64_t *d_from,
                            const uint64_t *d_to,
                            const std::vector<const void *> &d_payload,
                            uint64_t n, bool records_sorted_by_key,
                            const uint64_t *d_key, bool merge_existing) {
  s.csr_epoch++;
  const EdgeTypeDesc &ed = s.model->et(e);
  EdgeStore &es = s.edges[e];
  cudaStream_t st = s.stream;
  if (n >= (1ull << 31)) fail(VG_ERR_NOMEM, "more than 2^31 edge records in one build");

  // 1. target types and source types of the records
  unsigned long long h_counts[MAX_AGENT_TYPES] = {0};
  unsigned h_srcmask = 0;
  if (n > 0) {
    Tmp<unsigned long long> counts(MAX_AGENT_TYPES + 1, st);
    VG_CUDA(cudaMemsetAsync(counts.p, 0, (MAX_AGENT_TYPES + 1) * 8, st));
    unsigned *d_mask = (unsigned *)(counts.p + MAX_AGENT_TYPES);
    k_type_hist<<<std::min<unsigned>(nblk(n), 1024), TPB, 0, st>>>(
        d_to, ed.stores_src() ? d_from : nullptr, n, counts.p, d_mask);
    VG_CUDA(cudaGetLastError());
    VG_CUDA(cudaMemcpyAsync(h_counts, counts.p, MAX_AGENT_TYPES * 8, cudaMemcpyDeviceToHost, st));
    VG_CUDA(cudaMemcpyAsync(&h_srcmask, d_mask, 4, cudaMemcpyDeviceToHost, st));
    VG_CUDA(cudaStreamSynchronize(st));
  }
  if (es.csr.size() < (size_t)MAX_AGENT_TYPES) es.csr.resize(MAX_AGENT_TYPES);
  int ntypes_present = 0;
  for (int T = 1; T < MAX_AGENT_TYPES; T++) ntypes_present += h_counts[T] > 0;
  if (h_counts[0] > 0) fail(VG_ERR_ASSERT, "edge target is not a valid agent id");
  for (int T = 1; T < MAX_AGENT_TYPES; T++) {
    if (h_counts[T] == 0) continue;
    if (T > (int)s.model->atypes.size())
      fail(VG_ERR_ASSERT, "edge target has an unknown agent type");
    if (ed.singletype() && T != ed.target)
      fail(VG_ERR_ASSERT, "The :SingleType hint is set for " + ed.name +
                              ", and the agent type is specified as " +
                              s.model->at(ed.target).name +
                              ". But the type for the given agent is " +
                              s.model->at(T).name + ".");
  }

  // 2. order permutation of the records (none: they are in order, of one type)
  const bool need_ord = n > 0 && ((d_key && !records_sorted_by_key) || ntypes_present > 1);
  Tmp<uint32_t> ord(need_ord ? n : 1, st);
  if (need_ord) {
    k_iota<<<nblk(n), TPB, 0, st>>>(ord.p, n);
    if (d_key && !records_sorted_by_key) {
      Tmp<uint64_t> kk(n, st);
      k_copy_u64<<<nblk(n), TPB, 0, st>>>(d_key, kk.p, n);
      radix_sort_pairs_u64(kk.p, ord.p, n, 64, st, s);
    }
  }

  // 3. per target type
  for (int T = 1; T < MAX_AGENT_TYPES; T++) {
    CSR &old = es.csr[T];
    bool has_old = merge_existing && old.nedges + old.nrows > 0 && old.row_ptr.p;
    if (h_counts[T] == 0 && !has_old) {
      if (!merge_existing) es.csr[T] = CSR();
      continue;
    }
    if (T > (int)s.model->atypes.size()) continue;
    uint64_t nrows = s.agents[T - 1].n;
    uint64_t m = h_counts[T];
    // select the records of this target type in order
    Tmp<uint32_t> sel(ntypes_present > 1 ? m : 1, st);
    const uint32_t *selp = need_ord ? ord.p : nullptr;
    if (m > 0 && ntypes_present > 1) {
      Tmp<uint32_t> flags(n + 1, st), pos(n + 1, st);
      k_flag_type<<<nblk(n), TPB, 0, st>>>(d_to, ord.p, n, (unsigned)T, flags.p);
      exclusive_scan_u32(flags.p, pos.p, n, st, s);
      k_compact_sel<<<nblk(n), TPB, 0, st>>>(ord.p, flags.p, pos.p, n, sel.p);
      selp = sel.p;
    }
    Tmp<uint32_t> keys(m, st), rec(m, st);
    Tmp<int> status(2, st);  // the error, the largest row
    VG_CUDA(cudaMemsetAsync(status.p, 0, 8, st));
    if (m > 0) {
      k_row_keys<<<nblk(m), TPB, 0, st>>>(d_to, selp, m, nrows, keys.p, rec.p, status.p);
      radix_sort_pairs_u32(keys.p, rec.p, m, bits_for(nrows ? nrows - 1 : 0), st, s);
    }
    // New containers without a hint that drops edges: the sorted records are
    // the edges, in place order, and the rows begin where the keys change --
    // no counts, scans and destinations, and one wait at the end.  Bound: the
    // sort.  Measured, finish_init! of 2*10^7 records with one payload column
    // over 10^6 agents: 10.3 ms with them, 9.4 here; all to one agent 22.5 and
    // 14.5; a burst of 24 served jobs 49.0 and 40.7 ms.
    if (!has_old && m > 0 && !ed.bool_only()) {
      CSR c;
      c.nrows = nrows;
      c.nedges = m;
      c.src_type_const = !ed.stores_src() ? 0 : __builtin_popcount(h_srcmask) == 1
                             ? __builtin_ctz(h_srcmask) : h_srcmask ? -1 : 0;
      c.row_ptr.alloc((nrows + 1) * 4, &s.footprint);
      const uint64_t nbr = (nrows + 1 + RP_ROWS - 1) / RP_ROWS;
      Tmp<uint32_t> bstart(nbr + 1, st);
      k_rp_bounds<<<nblk(m + 1), TPB, 0, st>>>(keys.p, m, nbr, bstart.p);
      k_rp_fill<<<(unsigned)nbr, TPB, 0, st>>>(keys.p, nrows, bstart.p, c.row_ptr.as<uint32_t>(),
                                               (unsigned *)status.p + 1);
      if (ed.stores_src()) {
        c.src.alloc(m * 4, &s.footprint);
        if (c.src_type_const < 0) c.src_type.alloc(m, &s.footprint);
        k_place_src<<<nblk(m), TPB, 0, st>>>(d_from, rec.p, nullptr, m, c.src.as<uint32_t>(),
                                             c.src_type_const < 0 ? c.src_type.as<uint8_t>() : nullptr);
      }
      c.payload.resize(ed.stores_payload() ? ed.fields.size() : 0);
      for (size_t f = 0; f < c.payload.size(); f++) {
        c.payload[f].alloc(m * ed.fields[f].size, &s.footprint);
        scatter_column(ed.fields[f].size, d_payload[f], rec.p, nullptr, m, c.payload[f].p, st);
      }
      VG_CUDA(cudaGetLastError());
      unsigned w[2];
      s.fetch(w, status.p, 8);
      if (w[0]) fail(VG_ERR_ASSERT, "an edge targets an agent that does not exist");
      c.max_degree = w[1];
      if (ed.singleedge() && c.max_degree > 1)
        fail(VG_ERR_ASSERT, "An edge has already been added to an agent of edge type " +
                                ed.name + " (which has the :SingleEdge hint).");
      es.csr[T] = std::move(c);
      continue;
    }
    int h_status = 0;
    VG_CUDA(cudaMemcpyAsync(&h_status, status.p, 4, cudaMemcpyDeviceToHost, st));
    // counts
    Tmp<uint32_t> newcnt(nrows + 1, st), oldcnt(nrows + 1, st),
        tot(nrows + 1, st), seg(nrows + 1, st);
    VG_CUDA(cudaMemsetAsync(newcnt.p, 0, (nrows + 1) * 4, st));
    if (m > 0) k_hist_rows<<<nblk(m), TPB, 0, st>>>(keys.p, m, newcnt.p);
    exclusive_scan_u32(newcnt.p, seg.p, nrows + 1, st, s);
    k_add_old_counts<<<nblk(nrows + 1), TPB, 0, st>>>(
        has_old ? old.row_ptr.as<uint32_t>() : nullptr, has_old ? old.nrows : 0,
        newcnt.p, tot.p, oldcnt.p, nrows);
    VG_CUDA(cudaMemsetAsync(tot.p + nrows, 0, 4, st));
    VG_CUDA(cudaMemsetAsync(oldcnt.p + nrows, 0, 4, st));
    bool dedupe = ed.bool_only();
    if (dedupe) k_clamp1<<<nblk(nrows + 1), TPB, 0, st>>>(tot.p, nrows);
    CSR c;
    c.nrows = nrows;
    c.row_ptr.alloc((nrows + 1) * 4, &s.footprint);
    exclusive_scan_u32(tot.p, c.row_ptr.as<uint32_t>(), nrows + 1, st, s);
    uint32_t h_total = 0;
    VG_CUDA(cudaMemcpyAsync(&h_total, c.row_ptr.as<uint32_t>() + nrows, 4, cudaMemcpyDeviceToHost, st));
    {
      Tmp<unsigned> mx(1, st);
      VG_CUDA(cudaMemsetAsync(mx.p, 0, 4, st));
      k_max_u32<<<std::min<unsigned>(nblk(nrows), 1024), TPB, 0, st>>>(tot.p, nrows, mx.p);
      VG_CUDA(cudaMemcpyAsync(&c.max_degree, mx.p, 4, cudaMemcpyDeviceToHost, st));
    }
    VG_CUDA(cudaStreamSynchronize(st));
    if (h_status) fail(VG_ERR_ASSERT, "an edge targets an agent that does not exist");
    if (ed.singleedge() && !dedupe && c.max_degree > 1)
      fail(VG_ERR_ASSERT, "An edge has already been added to an agent of edge type " +
                              ed.name + " (which has the :SingleEdge hint).");
    c.nedges = h_total;
    // source types
    unsigned mask = 0;
    if (ed.stores_src()) {
      mask = m > 0 ? h_srcmask : 0;  // conservative: mask of all records
      if (has_old) {
        if (old.src_type_const > 0) mask |= 1u << old.src_type_const;
        if (old.src_type_const < 0) mask |= 0xfffeu;  // mixed: keep mixed
      }
    }
    int npop = __builtin_popcount(mask);
    c.src_type_const = npop == 0 ? 0 : (npop == 1 ? __builtin_ctz(mask) : -1);
    uint64_t ne = c.nedges;
    if (ed.stores_src()) {
      c.src.alloc(std::max<uint64_t>(ne, 1) * 4, &s.footprint);
      if (c.src_type_const < 0) c.src_type.alloc(std::max<uint64_t>(ne, 1), &s.footprint);
    }
    int nf = ed.stores_payload() ? (int)ed.fields.size() : 0;
    c.payload.resize(nf);
    for (int f = 0; f < nf; f++)
      c.payload[f].alloc(std::max<uint64_t>(ne, 1) * ed.fields[f].size, &s.footprint);
    // old edges
    if (has_old && old.nedges > 0) {
      Tmp<uint32_t> dest(old.nedges, st);
      k_old_dest<<<nblk(old.nedges), TPB, 0, st>>>(old.row_ptr.as<uint32_t>(), old.nrows,
                                                   old.nedges, c.row_ptr.as<uint32_t>(), dest.p);
      if (dedupe) {
        // rows keep one entry; old rows already hold at most one
      }
      if (ed.stores_src()) {
        scatter_column(4, old.src.p, nullptr, dest.p, old.nedges, c.src.p, st);
        if (c.src_type_const < 0) {
          if (old.src_type.p)
            scatter_column(1, old.src_type.p, nullptr, dest.p, old.nedges, c.src_type.p, st);
          else
            k_fill_u8<<<nblk(old.nedges), TPB, 0, st>>>(c.src_type.as<uint8_t>(),
                                                        (uint8_t)old.src_type_const, dest.p, old.nedges);
        }
      }
      for (int f = 0; f < nf; f++)
        scatter_column(ed.fields[f].size, old.payload[f].p, nullptr, dest.p, old.nedges,
                       c.payload[f].p, st);
    }
    // new records
    if (m > 0) {
      Tmp<uint32_t> dest(m, st);
      k_new_dest<<<nblk(m), TPB, 0, st>>>(keys.p, m, c.row_ptr.as<uint32_t>(), oldcnt.p,
                                          seg.p, dest.p, dedupe ? 1 : 0);
      if (ed.stores_src())
        k_place_src<<<nblk(m), TPB, 0, st>>>(d_from, rec.p, dest.p, m, c.src.as<uint32_t>(),
                                             c.src_type_const < 0 ? c.src_type.as<uint8_t>() : nullptr);
      for (int f = 0; f < nf; f++)
        scatter_column(ed.fields[f].size, d_payload[f], rec.p, dest.p, m, c.payload[f].p, st);
    }
    VG_CUDA(cudaGetLastError());
    es.csr[T] = std::move(c);
  }
  VG_CUDA(cudaStreamSynchronize(st));
}

// Replace c by its edges with keep[k] = 1 (scan = exclusive scan of keep,
// newtotal = kept edges), rows and order unchanged.
static void compact_csr(Sim &s, const EdgeTypeDesc &ed, CSR &c, const uint32_t *keep,
                        const uint32_t *scan, uint32_t newtotal) {
  cudaStream_t st = s.stream;
  uint64_t ne = c.nedges;
  CSR n2;
  n2.nrows = c.nrows;
  n2.nedges = newtotal;
  n2.src_type_const = c.src_type_const;
  n2.row_ptr.alloc((c.nrows + 1) * 4, &s.footprint);
  k_new_rowptr<<<nblk(c.nrows + 1), TPB, 0, st>>>(c.row_ptr.as<uint32_t>(), c.nrows, scan,
                                                  n2.row_ptr.as<uint32_t>());
  Tmp<uint32_t> dest(ne, st);
  k_compact_dest<<<nblk(ne), TPB, 0, st>>>(keep, scan, ne, dest.p);
  uint64_t alloc_n = std::max<uint64_t>(newtotal, 1);
  if (c.src.p) {
    n2.src.alloc(alloc_n * 4, &s.footprint);
    scatter_column(4, c.src.p, nullptr, dest.p, ne, n2.src.p, st);
  }
  if (c.src_type.p) {
    n2.src_type.alloc(alloc_n, &s.footprint);
    scatter_column(1, c.src_type.p, nullptr, dest.p, ne, n2.src_type.p, st);
  }
  n2.payload.resize(c.payload.size());
  for (size_t f = 0; f < c.payload.size(); f++) {
    n2.payload[f].alloc(alloc_n * ed.fields[f].size, &s.footprint);
    scatter_column(ed.fields[f].size, c.payload[f].p, nullptr, dest.p, ne, n2.payload[f].p, st);
  }
  n2.max_degree = csr_max_degree(s, c);
  VG_CUDA(cudaGetLastError());
  VG_CUDA(cudaStreamSynchronize(st));
  c = std::move(n2);
}

// The rows' kept edges are counted for every affected container before the
// host learns any total (one wait); containers that lose edges are packed
// into the buffers of their previous packing, which change places.
void remove_died_edges(Sim &s, const std::vector<int> &died_types) {
  s.csr_epoch++;
  cudaStream_t st = s.stream;
  struct Affected {
    int e, T;
    DiedView d;
  };
  std::vector<Affected> list;
  for (size_t e = 0; e < s.edges.size(); e++) {
    EdgeStore &es = s.edges[e];
    const EdgeTypeDesc &ed = s.model->et((int)e);
    if (es.implicit) continue;
    for (int T = 1; T < (int)es.csr.size(); T++) {
      CSR &c = es.csr[T];
      if (c.nedges == 0) continue;
      Affected x{(int)e, T, DiedView{}};
      bool any = false;
      for (int D : died_types) {
        AgentStore &a = s.agents[D - 1];
        if (T == D) {
          x.d.target = a.died_rd.as<uint8_t>();
          x.d.target_n = a.n;
          any = true;
        }
        if (ed.stores_src() && D < MAX_AGENT_TYPES &&
            (c.src_type_const == D || c.src_type_const < 0)) {
          x.d.source[D] = a.died_rd.as<uint8_t>();
          x.d.source_n[D] = a.n;
          any = true;
        }
      }
      if (any) list.push_back(x);
    }
  }
  if (list.empty()) return;
  uint64_t rows = 0;
  for (auto &x : list) rows += s.edges[x.e].csr[x.T].nrows + 1;
  uint32_t *counts = (uint32_t *)s.work(Sim::WORK_ROWS, rows * 4);
  uint32_t *totals = (uint32_t *)s.results(list.size() * 4);
  uint64_t at = 0;
  for (size_t k = 0; k < list.size(); k++) {
    CSR &c = s.edges[list[k].e].csr[list[k].T];
    k_kept_edges<false><<<nblk(c.nrows + 1), TPB, 0, st>>>(csr_view(s, list[k].e, list[k].T),
                                                           list[k].d, counts + at, nullptr,
                                                           KeptOut{});
    VG_CUDA(cudaGetLastError());
    scan_map<SCAN_IPT, uint32_t>(s, c.nrows + 1, RowsFrom{counts + at}, RowsTo{counts + at}, totals + k);
    at += c.nrows + 1;
  }
  std::vector<uint32_t> kept(list.size());
  s.read_results(kept.data(), totals, kept.size() * 4);
  at = 0;
  for (size_t k = 0; k < list.size(); k++) {
    CSR &c = s.edges[list[k].e].csr[list[k].T];
    const EdgeTypeDesc &ed = s.model->et(list[k].e);
    const uint32_t *new_rp = counts + at;
    at += c.nrows + 1;
    if (kept[k] == c.nedges) continue;
    if (!c.rebuild) c.rebuild.reset(new RebuildCache());
    RebuildCache &rc = *c.rebuild;
    const uint64_t m = std::max<uint64_t>(kept[k], 1);
    ensure_buf(s, rc.row_ptr, (c.nrows + 1) * 4, true);
    VG_CUDA(cudaMemcpyAsync(rc.row_ptr.p, new_rp, (c.nrows + 1) * 4, cudaMemcpyDeviceToDevice, st));
    KeptOut out{};
    if (c.src.p) {
      ensure_buf(s, rc.src, m * 4, true);
      out.src = rc.src.as<uint32_t>();
    }
    DevBuf types;
    if (c.src_type.p) {
      types.alloc(m, &s.footprint);
      out.src_type = types.as<uint8_t>();
    }
    out.npay = (int)c.payload.size();
    rc.payload.resize(c.payload.size());
    for (size_t f = 0; f < c.payload.size(); f++) {
      out.psize[f] = ed.fields[f].size;
      ensure_buf(s, rc.payload[f], m * ed.fields[f].size, true);
      out.pay[f] = rc.payload[f].p;
    }
    k_kept_edges<true><<<nblk(c.nrows + 1), TPB, 0, st>>>(csr_view(s, list[k].e, list[k].T),
                                                          list[k].d, nullptr, new_rp, out);
    VG_CUDA(cudaGetLastError());
    std::swap(c.row_ptr, rc.row_ptr);
    if (c.src.p) std::swap(c.src, rc.src);
    if (c.src_type.p) {
      VG_CUDA(cudaStreamSynchronize(st));  // (the old column is freed here)
      c.src_type = std::move(types);
    }
    std::swap(c.payload, rc.payload);
    c.nedges = kept[k];
    c.schedule_valid = false;  // (the largest row length stays a bound)
    c.unit_grid_weights = -1;
  }
}

namespace {
// remove_edges! records sorted by (to, from); from = REMOVE_ALL sorts last
struct RemovalTable {
  const uint64_t *to, *from, *key;
  uint64_t n;
};

__device__ uint64_t removal_key(const RemovalTable &R, uint64_t to, uint64_t from) {
  uint64_t lo = 0, hi = R.n;
  while (lo < hi) {
    uint64_t mid = (lo + hi) >> 1;
    if (R.to[mid] < to || (R.to[mid] == to && R.from[mid] < from)) lo = mid + 1;
    else hi = mid;
  }
  uint64_t mx = 0;
  for (uint64_t k = lo; k < R.n && R.to[k] == to && R.from[k] == from; k++)
    mx = R.key[k] > mx ? R.key[k] : mx;
  return mx;
}

// an edge (to, from) added with key k is gone when a later removal hit it
__device__ __forceinline__ bool removed_edge(const RemovalTable &R, uint64_t to, uint64_t from,
                                             uint64_t k, bool has_from) {
  if (removal_key(R, to, REMOVE_ALL) > k) return true;
  return has_from && removal_key(R, to, from) > k;
}

__global__ void k_removal_keep_old(const uint32_t *rp, uint64_t nrows, const uint32_t *src,
                                   const uint8_t *src_type, int src_type_const, int target_type,
                                   RemovalTable R, uint32_t *keep) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  const uint64_t to = ((uint64_t)target_type << SHIFT_TYPE) | (r + 1);
  for (uint32_t k = rp[r]; k < rp[r + 1]; k++) {
    uint64_t from = REMOVE_ALL;
    if (src) {
      int ty = src_type ? (int)src_type[k] : src_type_const;
      from = ((uint64_t)ty << SHIFT_TYPE) | ((uint64_t)src[k] + 1);
    }
    keep[k] = removed_edge(R, to, from, 0, src != nullptr) ? 0u : 1u;
  }
}

__global__ void k_removal_keep_new(const uint64_t *to, const uint64_t *from, const uint64_t *key,
                                   uint64_t n, int has_from, RemovalTable R, uint32_t *keep) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keep[i] = removed_edge(R, to[i], from[i], key[i] + 1, has_from != 0) ? 0u : 1u;
}

__global__ void k_gather_u64(const uint64_t *in, const uint32_t *perm, uint64_t n, uint64_t *out) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[perm[i]];
}
}  // namespace

void apply_edge_removals(Sim &s, int e, EdgeRemoval &rm, EdgeAppend *ap, uint64_t &n_records,
                         bool merge_existing) {
  s.csr_epoch++;
  cudaStream_t st = s.stream;
  const EdgeTypeDesc &ed = s.model->et(e);
  EdgeStore &es = s.edges[e];
  uint64_t r = 0;
  VG_CUDA(cudaMemcpyAsync(&r, rm.counter.p, 8, cudaMemcpyDeviceToHost, st));
  VG_CUDA(cudaStreamSynchronize(st));
  if (r > rm.cap) fail(VG_ERR_DEVICE, "remove_edges! record buffer overflow");
  if (r == 0) return;
  if (r >= (1ull << 31)) fail(VG_ERR_NOMEM, "more than 2^31 remove_edges! calls in one apply!");
  // the table sorted by (to, from): stable LSD passes, from first
  Tmp<uint32_t> perm(r, st);
  k_iota<<<nblk(r), TPB, 0, st>>>(perm.p, r);
  Tmp<uint64_t> k1(r, st), tto(r, st), tfrom(r, st), tkey(r, st);
  k_copy_u64<<<nblk(r), TPB, 0, st>>>(rm.from.as<uint64_t>(), k1.p, r);
  radix_sort_pairs_u64(k1.p, perm.p, r, 64, st, s);
  k_gather_u64<<<nblk(r), TPB, 0, st>>>(rm.to.as<uint64_t>(), perm.p, r, tto.p);
  radix_sort_pairs_u64(tto.p, perm.p, r, 64, st, s);
  k_gather_u64<<<nblk(r), TPB, 0, st>>>(rm.from.as<uint64_t>(), perm.p, r, tfrom.p);
  k_gather_u64<<<nblk(r), TPB, 0, st>>>(rm.key.as<uint64_t>(), perm.p, r, tkey.p);
  VG_CUDA(cudaGetLastError());
  RemovalTable R{tto.p, tfrom.p, tkey.p, r};
  // the old edges that add_existing carries over
  if (merge_existing) {
    for (int T = 1; T < (int)es.csr.size(); T++) {
      CSR &c = es.csr[T];
      if (c.nedges == 0 || !c.row_ptr.p) continue;
      uint64_t ne = c.nedges;
      Tmp<uint32_t> keep(ne + 1, st), scan(ne + 1, st);
      VG_CUDA(cudaMemsetAsync(keep.p + ne, 0, 4, st));
      k_removal_keep_old<<<nblk(c.nrows), TPB, 0, st>>>(
          c.row_ptr.as<uint32_t>(), c.nrows, ed.stores_src() ? c.src.as<uint32_t>() : nullptr,
          c.src_type.as<uint8_t>(), c.src_type_const, T, R, keep.p);
      exclusive_scan_u32(keep.p, scan.p, ne + 1, st, s);
      uint32_t newtotal = 0;
      VG_CUDA(cudaMemcpyAsync(&newtotal, scan.p + ne, 4, cudaMemcpyDeviceToHost, st));
      VG_CUDA(cudaStreamSynchronize(st));
      if (newtotal != ne) compact_csr(s, ed, c, keep.p, scan.p, newtotal);
    }
  }
  // the edges appended in this transition
  if (ap && n_records > 0) {
    if (ap->key.p == nullptr)
      fail(VG_ERR_ARG, "remove_edges! with edges appended in a fixed order is not supported");
    uint64_t n = n_records;
    Tmp<uint32_t> keep(n + 1, st), scan(n + 1, st);
    VG_CUDA(cudaMemsetAsync(keep.p + n, 0, 4, st));
    k_removal_keep_new<<<nblk(n), TPB, 0, st>>>(ap->to.as<uint64_t>(), ap->from.as<uint64_t>(),
                                                ap->key.as<uint64_t>(), n,
                                                ed.stores_src() ? 1 : 0, R, keep.p);
    exclusive_scan_u32(keep.p, scan.p, n + 1, st, s);
    uint32_t kept = 0;
    VG_CUDA(cudaMemcpyAsync(&kept, scan.p + n, 4, cudaMemcpyDeviceToHost, st));
    VG_CUDA(cudaStreamSynchronize(st));
    if (kept != n) {
      Tmp<uint32_t> dest(n, st);
      k_compact_dest<<<nblk(n), TPB, 0, st>>>(keep.p, scan.p, n, dest.p);
      auto squeeze = [&](DevBuf &b, int esz) {
        DevBuf nb;
        nb.alloc(std::max<uint64_t>(kept, 1) * esz, &s.footprint);
        scatter_column(esz, b.p, nullptr, dest.p, n, nb.p, st);
        b = std::move(nb);
      };
      squeeze(ap->to, 8);
      squeeze(ap->from, 8);
      squeeze(ap->key, 8);
      for (size_t f = 0; f < ap->payload.size(); f++) squeeze(ap->payload[f], ed.fields[f].size);
      ap->cap = std::max<uint64_t>(kept, 1);
      VG_CUDA(cudaGetLastError());
      VG_CUDA(cudaStreamSynchronize(st));
      n_records = kept;
    }
  }
}

namespace {
__device__ __forceinline__ uint32_t row_degree(const uint32_t *rp, uint64_t nrows, uint64_t r) {
  return r < nrows ? rp[r + 1] - rp[r] : 0u;
}

// flag rows with lo < degree <= hi
__global__ void k_flag_degree(const uint32_t *rp, uint64_t nrows, uint64_t n, uint32_t lo,
                              uint32_t hi, uint32_t *flag) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  uint32_t d = row_degree(rp, nrows, r);
  flag[r] = (d > lo && d <= hi) ? 1u : 0u;
}

__global__ void k_compact_rows(const uint32_t *flag, const uint32_t *pos, uint64_t n,
                               uint32_t *rows) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n && flag[r]) rows[pos[r]] = (uint32_t)r;
}

// sort key of a hub row: descending degree
__global__ void k_count_above(const uint32_t *rp, const uint32_t *rows, uint64_t m,
                              uint32_t thr, unsigned *cnt) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m && rp[rows[k] + 1] - rp[rows[k]] > thr) atomicAdd(cnt, 1u);
}

__global__ void k_hub_keys(const uint32_t *rp, const uint32_t *rows, uint64_t m, uint32_t *keys) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) keys[k] = 0xFFFFFFFFu - (rp[rows[k] + 1] - rp[rows[k]]);
}

// order keys: rows with degree <= cap by window, then descending degree
// (stable sort: ties by index); the others sort last
__global__ void k_order_keys(const uint32_t *rp, uint64_t nrows, uint64_t n, uint32_t cap,
                             uint32_t wshift, uint32_t *keys, uint32_t *vals) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  uint32_t d = row_degree(rp, nrows, r);
  keys[r] = d > cap ? 0xFFFFFFFFu : (((uint32_t)(r >> wshift) << 16) | (0xFFFFu - min(d, 0xFFFFu)));
  vals[r] = (uint32_t)r;
}




// largest degree of each slice of 32 order positions
__global__ void k_slice_deg(const uint32_t *rp, uint64_t nrows, const uint32_t *order, uint64_t m,
                            uint64_t nslices, uint32_t *sdeg, uint64_t *slots) {
  uint64_t sl = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (sl >= nslices) return;
  uint32_t dm = 0;
  for (uint64_t k = sl * 32; k < min(m, sl * 32 + 32); k++)
    dm = max(dm, row_degree(rp, nrows, order[k]));
  sdeg[sl] = dm;
  slots[sl] = 32ull * dm;
}

// flag the slices of at least thr slots; *tail: the longest of the others from
// slice `from` on
__global__ void k_flag_long(const uint32_t *sdeg, uint64_t nslices, uint32_t thr, uint64_t from,
                            uint32_t *flag, uint32_t *tail) {
  uint64_t sl = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t d = sl < nslices ? sdeg[sl] : 0u;
  if (sl < nslices) flag[sl] = d >= thr ? 1u : 0u;
  const uint32_t m = __reduce_max_sync(0xffffffffu, sl >= from && d < thr ? d : 0u);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(tail, m);
}

// sort key of a listed slice: descending length
__global__ void k_long_keys(const uint32_t *sdeg, const uint32_t *list, uint64_t m,
                            uint32_t *keys) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) keys[k] = 0xFFFFFFFFu - sdeg[list[k]];
}

// copy each row's edges into its slice, column-major; padding source 0,
// weight 0
__global__ void k_sell_fill(const uint32_t *__restrict__ rp, uint64_t nrows,
                            const uint32_t *__restrict__ src, const double *__restrict__ w,
                            const uint32_t *__restrict__ order, uint64_t m,
                            const uint64_t *__restrict__ base, const uint32_t *__restrict__ sdeg,
                            uint32_t *__restrict__ ssrc, double *__restrict__ sw) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t nslices_pos = (m + 31) / 32 * 32;
  if (k >= nslices_pos) return;
  const uint64_t sl = k >> 5, lane = k & 31;
  uint32_t b = 0, d = 0;
  if (k < m) {
    uint32_t r = order[k];
    if (r < nrows) {
      b = rp[r];
      d = rp[r + 1] - b;
    }
  }
  const uint64_t o = base[sl] + lane;
  const uint32_t D = sdeg[sl];
  // (the columns do not overlap the CSR: each lane's loads of a round are
  // in flight together)
#pragma unroll 4
  for (uint32_t q = 0; q < D; q++) {
    ssrc[o + 32ull * q] = q < d ? src[b + q] : 0u;
    sw[o + 32ull * q] = q < d ? w[b + q] : 0.0;
  }
}

// rows with lo < degree <= hi, in index order
uint64_t select_rows(Sim &s, const CSR &c, uint64_t n, uint32_t lo, uint32_t hi, DevBuf &out) {
  cudaStream_t st = s.stream;
  Tmp<uint32_t> flag(n + 1, st), pos(n + 1, st);
  VG_CUDA(cudaMemsetAsync(flag.p + n, 0, 4, st));
  k_flag_degree<<<nblk(n), TPB, 0, st>>>(c.row_ptr.as<uint32_t>(), c.nrows, n, lo, hi, flag.p);
  exclusive_scan_u32(flag.p, pos.p, n + 1, st, s);
  uint32_t m = 0;
  VG_CUDA(cudaMemcpyAsync(&m, pos.p + n, 4, cudaMemcpyDeviceToHost, st));
  VG_CUDA(cudaStreamSynchronize(st));
  if (m) {
    out.alloc((uint64_t)m * 4, &s.footprint);
    k_compact_rows<<<nblk(n), TPB, 0, st>>>(flag.p, pos.p, n, out.as<uint32_t>());
    VG_CUDA(cudaGetLastError());
  }
  return m;
}
}  // namespace

// in-degree of the row at each position of the slice order
__global__ void k_order_deg(const uint32_t *rp, uint64_t nrows, const uint32_t *order,
                            uint64_t m, uint32_t *deg) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) deg[k] = row_degree(rp, nrows, order[k]);
}

void ensure_schedule(Sim &s, CSR &c, uint32_t thr, uint32_t big_thr, uint64_t n) {
  if (c.schedule_valid && c.hub_threshold == thr && c.block_threshold == big_thr &&
      c.sched_n == n)
    return;
  cudaStream_t st = s.stream;
  c.hub_rows.release();
  c.order.release();
  c.order_deg.release();
  c.slice_base.release();
  c.slice_deg.release();
  c.sell_src.release();
  c.sell_w.release();
  c.long_slices.release();
  c.long_slots.clear();
  c.long_hubs.clear();
  c.tail_slots = 0;
  c.nhub = c.norder = c.nslices = c.nbig = 0;
  c.range_block.clear();
  c.range_rows.clear();
  c.range_window.clear();
  c.hub_rows_sorted.clear();
  if (n > 0 && c.row_ptr.p) {
    const uint32_t *rp = c.row_ptr.as<uint32_t>();
    // (a launch that folds other graphs' edges too only takes longer slices)
    const uint32_t long_min = opinion_long_slots(c.nedges);
    // hub rows by descending degree
    c.nhub = select_rows(s, c, n, thr, 0xFFFFFFFFu, c.hub_rows);
    if (c.nhub) {
      const uint32_t *rows = c.hub_rows.as<uint32_t>();
      Tmp<uint32_t> keys(c.nhub, st);
      k_hub_keys<<<nblk(c.nhub), TPB, 0, st>>>(rp, rows, c.nhub, keys.p);
      radix_sort_pairs_u32(keys.p, c.hub_rows.as<uint32_t>(), c.nhub, 32, st, s);
      // the leading hubs above the block threshold, and those that may take
      // a block of the long launch
      Tmp<unsigned> cnt(2, st);
      VG_CUDA(cudaMemsetAsync(cnt.p, 0, 8, st));
      k_count_above<<<nblk(c.nhub), TPB, 0, st>>>(rp, rows, c.nhub, big_thr, cnt.p);
      k_count_above<<<nblk(c.nhub), TPB, 0, st>>>(rp, rows, c.nhub, 32 * long_min - 1,
                                                  cnt.p + 1);
      unsigned h[2] = {0, 0};
      VG_CUDA(cudaMemcpyAsync(h, cnt.p, 8, cudaMemcpyDeviceToHost, st));
      VG_CUDA(cudaStreamSynchronize(st));
      c.nbig = h[0];
      if (h[1]) {
        c.long_hubs.resize(h[1]);
        VG_CUDA(cudaMemcpyAsync(c.long_hubs.data(), keys.p, (uint64_t)h[1] * 4,
                                cudaMemcpyDeviceToHost, st));
        VG_CUDA(cudaStreamSynchronize(st));
        for (uint32_t &k : c.long_hubs) k = 0xFFFFFFFFu - k;  // the sort's keys
      }
    }
    // the other rows by descending degree in windows of 2^13 rows (or
    // more, so that the window number stays below the sentinel)
    uint32_t wshift = 13;
    while ((n >> wshift) >= 0xFFFFull) wshift++;
    c.wshift = wshift;
    Tmp<uint32_t> keys(n, st);
    c.order.alloc(n * 4, &s.footprint);
    k_order_keys<<<nblk(n), TPB, 0, st>>>(rp, c.nrows, n, thr, wshift, keys.p,
                                          c.order.as<uint32_t>());
    radix_sort_pairs_u32(keys.p, c.order.as<uint32_t>(), n, 32, st, s);
    const uint64_t m = n - c.nhub;
    c.norder = m;
    const uint64_t ns = (m + 31) / 32;
    c.nslices = ns;
    if (ns > 0) {
      c.slice_deg.alloc(ns * 4, &s.footprint);
      c.slice_base.alloc((ns + 1) * 8, &s.footprint);
      Tmp<uint64_t> slots(ns + 1, st);
      VG_CUDA(cudaMemsetAsync(slots.p + ns, 0, 8, st));
      k_slice_deg<<<nblk(ns), TPB, 0, st>>>(rp, c.nrows, c.order.as<uint32_t>(), m, ns,
                                            c.slice_deg.as<uint32_t>(), slots.p);
      exclusive_scan_u64(slots.p, c.slice_base.as<uint64_t>(), ns + 1, st, s);
      uint64_t total = 0;
      VG_CUDA(cudaMemcpyAsync(&total, c.slice_base.as<uint64_t>() + ns, 8, cudaMemcpyDeviceToHost,
                              st));
      // the long slices, listed longest first (no slice has more than thr slots)
      if (thr >= long_min) {
        Tmp<uint32_t> flag(ns + 1, st), pos(ns + 2, st);
        VG_CUDA(cudaMemsetAsync(flag.p + ns, 0, 4, st));
        VG_CUDA(cudaMemsetAsync(pos.p + ns + 1, 0, 4, st));
        // (two windows at least: the last full one's first slices among them)
        const uint64_t last = std::min(ns, std::max<uint64_t>(ns / 8, 2ull << (wshift - 5)));
        k_flag_long<<<nblk(ns), TPB, 0, st>>>(c.slice_deg.as<uint32_t>(), ns, long_min,
                                              ns - last, flag.p, pos.p + ns + 1);
        exclusive_scan_u32(flag.p, pos.p, ns + 1, st, s);
        uint32_t found[2] = {0, 0};
        VG_CUDA(cudaMemcpyAsync(found, pos.p + ns, 8, cudaMemcpyDeviceToHost, st));
        VG_CUDA(cudaStreamSynchronize(st));
        const uint32_t nlong = found[0];
        c.tail_slots = found[1];
        if (nlong) {
          Tmp<uint32_t> lkeys(nlong, st);
          c.long_slices.alloc((uint64_t)nlong * 4, &s.footprint);
          k_compact_rows<<<nblk(ns), TPB, 0, st>>>(flag.p, pos.p, ns,
                                                   c.long_slices.as<uint32_t>());
          k_long_keys<<<nblk(nlong), TPB, 0, st>>>(c.slice_deg.as<uint32_t>(),
                                                   c.long_slices.as<uint32_t>(), nlong, lkeys.p);
          radix_sort_pairs_u32(lkeys.p, c.long_slices.as<uint32_t>(), nlong, 32, st, s);
          c.long_slots.resize(nlong);
          VG_CUDA(cudaMemcpyAsync(c.long_slots.data(), lkeys.p, (uint64_t)nlong * 4,
                                  cudaMemcpyDeviceToHost, st));  // (read after the wait below)
        }
      } else {
        VG_CUDA(cudaStreamSynchronize(st));
      }
      c.sell_src.alloc(std::max<uint64_t>(total, 1) * 4, &s.footprint);
      c.sell_w.alloc(std::max<uint64_t>(total, 1) * 8, &s.footprint);
      k_sell_fill<<<nblk(ns * 32), TPB, 0, st>>>(
          rp, c.nrows, c.src.as<uint32_t>(), c.payload[0].as<double>(), c.order.as<uint32_t>(), m,
          c.slice_base.as<uint64_t>(), c.slice_deg.as<uint32_t>(), c.sell_src.as<uint32_t>(),
          c.sell_w.as<double>());
      c.order_deg.alloc(std::max<uint64_t>(m, 1) * 4, &s.footprint);
      k_order_deg<<<nblk(m), TPB, 0, st>>>(rp, c.nrows, c.order.as<uint32_t>(), m,
                                           c.order_deg.as<uint32_t>());
    }
    VG_CUDA(cudaGetLastError());
    VG_CUDA(cudaStreamSynchronize(st));
    for (uint32_t &k : c.long_slots) k = 0xFFFFFFFFu - k;  // the sort's keys
  }
  c.sched_n = n;
  c.hub_threshold = thr;
  c.block_threshold = big_thr;
  c.schedule_valid = true;
}

}  // namespace vg
