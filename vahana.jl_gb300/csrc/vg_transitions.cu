// Transition kernels bound by name (the `f` of apply!, src/Simulation.jl:
// 720-821).  Every kernel sweeps the agents of the called type in index
// order semantics (transition_with_read!, src/AgentMethods.jl:193-207):
// died agents are skipped, a returned state is written to the write buffer
// (transition_with_write!, :159-181) and `nothing` marks the agent died.
//
// Floating-point arithmetic on the ordered paths uses explicitly rounded
// intrinsics (__dadd_rn, __dmul_rn, __ddiv_rn) in the reference's
// left-to-right order, so results are bit-identical to the sequential CPU
// fold (the library is also compiled with -fmad=false).
#include <algorithm>
#include <array>
#include <cstring>
#include <map>
#include <vector>

#include "vg_bucket.cuh"
#include "vg_internal.h"
#include "vg_philox.cuh"
#include "vg_rows.cuh"
#include "vg_scan.cuh"

namespace vg {

namespace {

constexpr int TPB = 256;
inline unsigned nblk(uint64_t n, int tpb = TPB) {
  uint64_t b = (n + tpb - 1) / tpb;
  return (unsigned)std::max<uint64_t>(b, 1);
}

__device__ __forceinline__ void set_status(int *st, int code) {
  report_status(st, code);
}

// ----------------------------------------------------------- field access
__device__ __forceinline__ int64_t ld_i64(const void *p, int dt, uint64_t i) {
  switch (dt) {
    case VG_BOOL: case VG_U8: return ((const uint8_t *)p)[i];
    case VG_I8: return ((const int8_t *)p)[i];
    case VG_U16: return ((const uint16_t *)p)[i];
    case VG_I16: return ((const int16_t *)p)[i];
    case VG_U32: return ((const uint32_t *)p)[i];
    case VG_I32: return ((const int32_t *)p)[i];
    case VG_U64: case VG_I64: return ((const int64_t *)p)[i];
    case VG_F32: return (int64_t)((const float *)p)[i];
    case VG_F64: return (int64_t)((const double *)p)[i];
  }
  return 0;
}
__device__ __forceinline__ double ld_f64(const void *p, int dt, uint64_t i) {
  switch (dt) {
    case VG_F32: return (double)((const float *)p)[i];
    case VG_F64: return ((const double *)p)[i];
    case VG_U64: return (double)((const uint64_t *)p)[i];
  }
  return (double)ld_i64(p, dt, i);
}
__device__ __forceinline__ void st_i64(void *p, int dt, uint64_t i, int64_t v) {
  switch (dt) {
    case VG_BOOL: ((uint8_t *)p)[i] = v != 0; break;
    case VG_U8: case VG_I8: ((uint8_t *)p)[i] = (uint8_t)v; break;
    case VG_U16: case VG_I16: ((uint16_t *)p)[i] = (uint16_t)v; break;
    case VG_U32: case VG_I32: ((uint32_t *)p)[i] = (uint32_t)v; break;
    case VG_U64: case VG_I64: ((int64_t *)p)[i] = v; break;
    case VG_F32: ((float *)p)[i] = (float)v; break;
    case VG_F64: ((double *)p)[i] = (double)v; break;
  }
}
__device__ __forceinline__ void st_f64(void *p, int dt, uint64_t i, double v) {
  switch (dt) {
    case VG_F32: ((float *)p)[i] = (float)v; break;
    case VG_F64: ((double *)p)[i] = v; break;
    default: st_i64(p, dt, i, (int64_t)v);
  }
}
__device__ __forceinline__ bool is_float(int dt) { return dt == VG_F32 || dt == VG_F64; }

// ------------------------------------------------------------ sweep frame
struct Sweep {
  DevAgentView a;
  int nfields;
  int fsize[MAX_FIELDS];
  int fdt[MAX_FIELDS];
  int mortal;
  int writes;              // the called type is in `write`
  const uint32_t *with_rp; // with_edge: row_ptr of that edge type, or null
  uint64_t with_nrows;
  int type_nr;
  int *status;
};

__device__ void sw_copy(const Sweep &s, uint64_t i) {
  for (int f = 0; f < s.nfields; f++) {
    switch (s.fsize[f]) {
      case 1: ((uint8_t *)s.a.wr[f])[i] = ((const uint8_t *)s.a.rd[f])[i]; break;
      case 2: ((uint16_t *)s.a.wr[f])[i] = ((const uint16_t *)s.a.rd[f])[i]; break;
      case 4: ((uint32_t *)s.a.wr[f])[i] = ((const uint32_t *)s.a.rd[f])[i]; break;
      case 8: ((uint64_t *)s.a.wr[f])[i] = ((const uint64_t *)s.a.rd[f])[i]; break;
    }
  }
  if (s.mortal) s.a.died_wr[i] = 0;
}

// Returns true when agent i is swept.  Died agents stay died; with_edge
// restricts the sweep to targets of that edge type (src/AgentMethods.jl:
// 209-229), the others keep their state.
__device__ __forceinline__ bool sw_begin(const Sweep &s, uint64_t i) {
  if (s.mortal && s.a.died_rd[i]) {
    if (s.writes) s.a.died_wr[i] = 1;
    return false;
  }
  if (s.with_rp) {
    bool has = i < s.with_nrows && s.with_rp[i + 1] > s.with_rp[i];
    if (!has) {
      if (s.writes) sw_copy(s, i);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void sw_die(const Sweep &s, uint64_t i) {
  if (!s.mortal) {
    set_status(s.status, 201);  // `nothing` returned for an immortal agent
    sw_copy(s, i);
    return;
  }
  s.a.died_wr[i] = 1;
}

// source field of every agent type (flexible neighbour states)
struct SrcTable {
  const void *ptr[MAX_AGENT_TYPES];
  int dt[MAX_AGENT_TYPES];
  const uint8_t *died[MAX_AGENT_TYPES];
};

__device__ __forceinline__ int edge_src_type(const DevCSRView &c, uint64_t k) {
  return c.src_type ? (int)c.src_type[k] : c.src_type_const;
}

// --------------------------------------------------- generic neighbour ops
// mode 0: dst = sum of the neighbours' field (neighbor_sum)
// mode 1: dst = own dst || any neighbour field != 0 (neighbor_or)
// mode 2: dst = number of edges (count_edges)
__global__ void k_neighbor_op(Sweep s, DevCSRView c, SrcTable t, int dst,
                              int mode) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.a.n || !sw_begin(s, i)) return;
  int ddt = s.fdt[dst];
  int64_t si = 0;
  double sf = 0.0;
  bool anyv = false;
  uint32_t b = 0, e = 0;
  if (i < c.nrows) {
    b = c.row_ptr[i];
    e = c.row_ptr[i + 1];
  }
  for (uint32_t k = b; k < e && mode != 2; k++) {
    int ty = edge_src_type(c, k);
    uint32_t j = c.src[k];
    if (ty <= 0 || ty >= MAX_AGENT_TYPES || !t.ptr[ty]) {
      set_status(s.status, 202);  // source type not readable
      continue;
    }
    if (t.died[ty] && t.died[ty][j]) set_status(s.status, 203);
    if (mode == 0) {
      if (is_float(ddt)) sf = __dadd_rn(sf, ld_f64(t.ptr[ty], t.dt[ty], j));
      else si = (int64_t)((uint64_t)si + (uint64_t)ld_i64(t.ptr[ty], t.dt[ty], j));
    } else {
      anyv |= ld_i64(t.ptr[ty], t.dt[ty], j) != 0;
    }
  }
  if (!s.writes) return;
  sw_copy(s, i);
  if (mode == 0) {
    if (is_float(ddt)) st_f64(s.a.wr[dst], ddt, i, sf);
    else st_i64(s.a.wr[dst], ddt, i, si);
  } else if (mode == 1) {
    bool own = ld_i64(s.a.rd[dst], ddt, i) != 0;
    st_i64(s.a.wr[dst], ddt, i, (own || anyv) ? 1 : 0);
  } else {
    st_i64(s.a.wr[dst], ddt, i, (int64_t)(e - b));
  }
}

// modes 0 and 1 where all sources are of one type, its column of type E:
// U edges of a row in flight (sources, then values and died flags), folded in
// the row's order.  One edge at a time, its source's type and the column's
// looked up for each (k_neighbor_op), left one load in flight per lane.  Bound:
// the random reads; for short rows the rows' own words, for a row beyond the
// others the chain of its additions.
//
// Rows of few edges take 4, long ones 8.  The registers of 8 (40 and 48, of 4
// 32) leave fewer warps to hide a short row's reads, and what a lane adds beyond
// its row's end costs the binary64 pipe (additions, conversions) as much as an
// edge: with 4 the warp stops at its longest rest.  us, k_neighbor_op, 8 and 4
// edges in flight, f32 column into f64, then i32 column:
//   5*10^6 agents, 10^5 edges       65  122  64    65   96  64
//   10^6 agents, 5*10^5 edges       21   38  18    18   17  13
//   10^6 agents, 4*10^6 edges       46   55  42    33   27  25
//   10^6 agents, 1.4*10^7 edges    103  106  93    90   64  63
// and, f64 column and i32 column, where 8 are the better ones:
//   20000 agents, 6*10^5 edges      26   11  13    24    9  11
//   one row of 2*10^5 edges (ms)    70   19  22    67   14  16
// 6 in flight lie between the two.
constexpr int NB_SHORT = 4, NB_LONG = 8;

// NB_LONG: a container of 16 edges a row (f64 column, 20000 agents of 14
// edges, us: 9.0 and, with NB_SHORT, 9.2; of 20 edges 9.6 and 11.2), or one
// whose longest row is known to have 1024 and so outlasts the others
inline bool neighbor_rows_long(uint64_t nrows, uint64_t nedges, uint32_t longest) {
  return nedges / 16 >= nrows || longest >= 1024;
}

template <class E, int U>
__global__ void __launch_bounds__(256) k_neighbor_typed(Sweep s, DevCSRView c,
                                                        const E *__restrict__ val,
                                                        const uint8_t *died, int dst, int mode) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.a.n || !sw_begin(s, i)) return;
  const int ddt = s.fdt[dst];
  const bool sums = mode == 0 && is_float(ddt);
  int64_t si = 0;
  double sf = 0.0;
  bool gone = false;
  uint32_t b = 0, e = 0;
  if (i < c.nrows) {
    b = c.row_ptr[i];
    e = c.row_ptr[i + 1];
  }
  for (uint32_t k = b; k < e; k += U) {
    uint32_t j[U];
    E v[U];
#pragma unroll
    for (int u = 0; u < U; u++) j[u] = k + u < e ? c.src[k + u] : 0u;
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = k + u < e ? val[j[u]] : E(0);
    if (died) {
#pragma unroll
      for (int u = 0; u < U; u++) gone |= k + u < e && died[j[u]];
    }
    if constexpr (U == NB_SHORT) {
      const unsigned lanes = __activemask();
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (u && !__any_sync(lanes, k + u < e)) break;
        if (k + u < e) {
          if (sums) sf = __dadd_rn(sf, (double)v[u]);
          else if (mode == 0) si = (int64_t)((uint64_t)si + (uint64_t)(int64_t)v[u]);
          else si |= (int64_t)v[u];
        }
      }
    } else if (sums) {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k + u < e) sf = __dadd_rn(sf, (double)v[u]);
    } else if (mode == 0) {
#pragma unroll
      for (int u = 0; u < U; u++) si = (int64_t)((uint64_t)si + (uint64_t)(int64_t)v[u]);
    } else {
#pragma unroll
      for (int u = 0; u < U; u++) si |= (int64_t)v[u];
    }
  }
  if (gone) set_status(s.status, 203);
  if (!s.writes) return;
  sw_copy(s, i);
  if (sums) st_f64(s.a.wr[dst], ddt, i, sf);
  else if (mode == 0) st_i64(s.a.wr[dst], ddt, i, si);
  else st_i64(s.a.wr[dst], ddt, i, (ld_i64(s.a.rd[dst], ddt, i) != 0 || si != 0) ? 1 : 0);
}

// die_if: kind 0 always; 1 field >= arg; 2 field % arg != 0; 3 the agent has
// no edge of the given edge type (num_edges == 0)
__global__ void k_die_if(Sweep s, int kind, int field, double arg,
                         const uint32_t *rp2, uint64_t nrows2) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.a.n || !sw_begin(s, i)) return;
  bool die = false;
  if (kind == 0) die = true;
  else if (kind == 1) die = ld_f64(s.a.rd[field], s.fdt[field], i) >= arg;
  else if (kind == 2) die = (ld_i64(s.a.rd[field], s.fdt[field], i) % (int64_t)arg) != 0;
  else if (kind == 3) die = !(rp2 && i < nrows2 && rp2[i + 1] > rp2[i]);
  if (!s.writes) return;
  if (die) sw_die(s, i);
  else sw_copy(s, i);
}

// set_field: kind 0 constant; 1 (agent id mod 2 == 1)
__global__ void k_set_field(Sweep s, int field, int kind, double value) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.a.n || !sw_begin(s, i)) return;
  if (!s.writes) return;
  sw_copy(s, i);
  int dt = s.fdt[field];
  if (kind == 0) {
    if (is_float(dt)) st_f64(s.a.wr[field], dt, i, value);
    else st_i64(s.a.wr[field], dt, i, (int64_t)value);
  } else {
    uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
    st_i64(s.a.wr[field], dt, i, (id % 2) == 1 ? 1 : 0);
  }
}

__global__ void k_keep(Sweep s) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.a.n || !sw_begin(s, i)) return;
  if (s.writes) sw_copy(s, i);
}

// edge appends with an order key (call position, caller index, sequence):
// the order in which the reference's sequential sweep calls add_edge!.
// slots: the records' places are known instead (a prefix of the callers'
// records: all callers' records lie in call order), rows and srcs take the
// target row and the source, and nothing is counted or keyed.
struct Append {
  uint64_t *to, *from, *key;
  uint32_t *rows, *srcs;
  void *payload[MAX_FIELDS];
  int psize[MAX_FIELDS];
  int npayload;
  unsigned long long *counter;
  uint64_t cap;
};

__device__ __forceinline__ uint64_t order_key(int call_pos, uint64_t i,
                                              uint32_t seq) {
  return ((uint64_t)call_pos << 60) | ((i & ((1ull << 40) - 1)) << 20) | seq;
}

// Slots of the append and removal buffers are reserved per warp: the lanes
// that add a record in this round vote, the lowest of them reserves all of
// the warp's slots with one atomicAdd on the buffer's counter, and each lane
// takes the next slot by its rank among the voters.  Every lane of the warp
// must call it (full mask; lanes with nothing to add pass want = false).
// The slot is only a place in the buffer: the record's order key decides its
// position in the rebuilt container.  -1: nothing wanted, or the buffer is
// full (err is recorded in the status word).
constexpr unsigned FULL_WARP = 0xffffffffu;

__device__ __forceinline__ int64_t warp_slot(unsigned long long *counter, uint64_t cap, bool want,
                                             int *status, int err) {
  const unsigned voters = __ballot_sync(FULL_WARP, want);
  if (!voters) return -1;
  const unsigned lane = threadIdx.x & 31;
  const int leader = __ffs(voters) - 1;
  unsigned long long base = 0;
  if ((int)lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(voters));
  base = __shfl_sync(FULL_WARP, base, leader);
  if (!want) return -1;
  const unsigned long long k = base + __popc(voters & ((1u << lane) - 1u));
  if (k >= cap) {
    set_status(status, err);
    return -1;
  }
  return (int64_t)k;
}

// add_edge!(sim, id, id, state) for every swept agent
__global__ void k_self_edge(Sweep s, Append ap, int call_pos, const uint8_t *pl) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < s.a.n && sw_begin(s, i);
  if (live && s.writes) sw_copy(s, i);
  int64_t k;
  if (ap.rows) {
    if (i >= s.a.n) return;
    k = (int64_t)i;
    ap.rows[k] = live ? (uint32_t)i : BK_HOLE;
    if (!live) return;
    ap.srcs[k] = (uint32_t)i;
  } else {
    k = warp_slot(ap.counter, ap.cap, live, s.status, 301);
    if (k < 0) return;
    uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
    ap.to[k] = id;
    ap.from[k] = id;
    ap.key[k] = order_key(call_pos, i, 0);
  }
  int off = 0;
  for (int f = 0; f < ap.npayload; f++) {
    for (int b = 0; b < ap.psize[f]; b++)
      ((uint8_t *)ap.payload[f])[k * ap.psize[f] + b] = pl[off + b];
    off += ap.psize[f];
  }
}

// add_edges!(sim, id, edges(sim, id, ET)): re-add every in-edge of the agent
// (round q: the q-th in-edge of every lane that has one)
__global__ void k_readd_edges(Sweep s, DevCSRView c, Append ap, int call_pos) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < s.a.n && sw_begin(s, i);
  if (live && s.writes) sw_copy(s, i);
  const bool rows = live && i < c.nrows;
  const uint32_t b = rows ? c.row_ptr[i] : 0u;
  const uint32_t deg = rows ? c.row_ptr[i + 1] - b : 0u;
  const uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
  for (uint32_t q = 0; __any_sync(FULL_WARP, q < deg); q++) {
    const int64_t k = warp_slot(ap.counter, ap.cap, q < deg, s.status, 301);
    if (k < 0) continue;
    const uint32_t e = b + q;
    ap.to[k] = id;
    ap.from[k] = ((uint64_t)edge_src_type(c, e) << SHIFT_TYPE) | ((uint64_t)c.src[e] + 1);
    ap.key[k] = order_key(call_pos, i, q);
    for (int f = 0; f < ap.npayload; f++) {
      int sz = ap.psize[f];
      for (int bb = 0; bb < sz; bb++)
        ((uint8_t *)ap.payload[f])[k * sz + bb] = ((const uint8_t *)c.payload[f])[(uint64_t)e * sz + bb];
    }
  }
}

// k_readd_edges into slots: edge e of the read container is record e
__global__ void k_readd_slots(Sweep s, DevCSRView c, Append ap) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < s.a.n && sw_begin(s, i);
  if (live && s.writes) sw_copy(s, i);
  uint32_t deg;
  const uint32_t b = row_run(c, i, deg);
  const unsigned alive = __ballot_sync(FULL_WARP, live);
  const uint32_t r0 = (uint32_t)(i & ~31ull);
  warp_edges(b, deg, [&](uint32_t e, unsigned owner, bool has) {
    if (!has) return;
    const bool swept = alive >> owner & 1u;
    ap.rows[e] = swept ? r0 + owner : BK_HOLE;
    if (!swept) return;
    ap.srcs[e] = c.src[e];
    for (int f = 0; f < ap.npayload; f++)
      copy_elem(ap.psize[f], c.payload[f], e, ap.payload[f], e);
  });
}

// remove_edges!: a swept agent keeps its state; mode 0: when its field 0
// passes the test (kind 0 always, 1 field >= arg, 2 field % arg != 0) it
// calls remove_edges!(sim, id, E); mode 1: for every source nid of its
// in-edges of E (read container, insertion order) whose field 0 passes the
// test it calls remove_edges!(sim, nid, id, E).
struct Removal {
  uint64_t *to, *from, *key;
  unsigned long long *counter;
  uint64_t cap;
};

__device__ __forceinline__ bool field_test(int kind, double arg, const void *p, int dt,
                                           uint64_t i) {
  if (kind == 0) return true;
  if (kind == 1) return ld_f64(p, dt, i) >= arg;
  return (ld_i64(p, dt, i) % (int64_t)arg) != 0;
}

// one removal record per lane with want (every lane of the warp calls it)
__device__ __forceinline__ void push_removal(const Removal &r, bool want, uint64_t to,
                                             uint64_t from, uint64_t key, int *status) {
  const int64_t k = warp_slot(r.counter, r.cap, want, status, 302);
  if (k < 0) return;
  r.to[k] = to;
  r.from[k] = from;
  r.key[k] = key;
}

__global__ void k_remove_edges(Sweep s, DevCSRView c, SrcTable t, int kind, double arg, int mode,
                               Removal rm, int call_pos) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < s.a.n && sw_begin(s, i);
  if (live && s.writes) sw_copy(s, i);
  const uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
  if (mode == 0) {
    const bool want = live && (s.nfields == 0 || field_test(kind, arg, s.a.rd[0], s.fdt[0], i));
    push_removal(rm, want, id, REMOVE_ALL, order_key(call_pos, i, 0) + 1, s.status);
    return;
  }
  // round j: the j-th in-edge of every lane that has one; a lane's records
  // are numbered q in insertion order of the edges that pass the test
  const bool rows = live && i < c.nrows;
  const uint32_t b = rows ? c.row_ptr[i] : 0u;
  const uint32_t deg = rows ? c.row_ptr[i + 1] - b : 0u;
  uint32_t q = 0;
  for (uint32_t j = 0; __any_sync(FULL_WARP, j < deg); j++) {
    bool want = false;
    uint64_t nid = 0;
    if (j < deg) {
      const uint32_t e = b + j;
      const int ty = edge_src_type(c, e);
      const uint32_t src = c.src[e];
      if (ty <= 0 || ty >= MAX_AGENT_TYPES || !t.ptr[ty]) {
        set_status(s.status, 202);  // source type not readable
      } else if (field_test(kind, arg, t.ptr[ty], t.dt[ty], src)) {
        want = true;
        nid = ((uint64_t)ty << SHIFT_TYPE) | ((uint64_t)src + 1);
      }
    }
    push_removal(rm, want, id, nid, order_key(call_pos, i, q) + 1, s.status);
    q += want;
  }
}

// ------------------------------------------- add_agent! within a transition
// spawn: every swept agent keeps its state and calls add_agent! k times
// (src/AgentMethods.jl:37-89) with a copy of its state whose field 0 is
// increased by offset j; with a link edge type, after each add_agent! it
// adds the edges new -> caller and caller -> new, payload field 0 = the new
// agent's id.  Pass 1 keeps the callers and flags them; the callers' rank
// (an exclusive scan in index order) numbers the new agents in the order of
// the sequential sweep: new agent s takes the s-th slot popped from the
// reuse stack (LIFO) and, when the stack is empty, the next fresh number.
constexpr int SPAWN_MAX = 8;
struct SpawnArgs {
  int k;
  double off[SPAWN_MAX];
  const uint64_t *reuse;  // 1-based agent numbers, top at nreuse - 1
  uint64_t nreuse, take;  // stack height, slots taken from it
  uint64_t n_old;         // nextid - 1 before the transition
};

// item i: 1 for a caller, which keeps its state on the way; its rank is the
// callers before it (BK_HOLE for the others)
struct SpawnCallers {
  Sweep s;
  __device__ __forceinline__ uint32_t operator()(uint64_t i) const {
    const bool swept = sw_begin(s, i);
    if (swept && s.writes) sw_copy(s, i);
    return swept ? 1u : 0u;
  }
};
struct SpawnRanks {
  uint32_t *rank;
  __device__ __forceinline__ void operator()(uint64_t i, uint32_t before, uint32_t is) const {
    rank[i] = is ? before : BK_HOLE;
  }
};

__global__ void k_spawn_new(Sweep s, uint64_t n_callers_scope, const uint32_t *rank, SpawnArgs g,
                            Append ap, int link_dt, int call_pos) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t mine = i < n_callers_scope ? rank[i] : BK_HOLE;
  const bool caller = mine != BK_HOLE;
  const uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
  for (int j = 0; j < g.k; j++) {
    const uint64_t q = caller ? (uint64_t)mine * g.k + j : 0;
    const uint64_t nr = !caller ? 0
                        : q < g.take ? g.reuse[g.nreuse - 1 - q] : g.n_old + 1 + (q - g.take);
    const uint64_t t = nr - 1;
    if (caller) {
      for (int f = 0; f < s.nfields; f++) {
        switch (s.fsize[f]) {
          case 1: ((uint8_t *)s.a.wr[f])[t] = ((const uint8_t *)s.a.rd[f])[i]; break;
          case 2: ((uint16_t *)s.a.wr[f])[t] = ((const uint16_t *)s.a.rd[f])[i]; break;
          case 4: ((uint32_t *)s.a.wr[f])[t] = ((const uint32_t *)s.a.rd[f])[i]; break;
          case 8: ((uint64_t *)s.a.wr[f])[t] = ((const uint64_t *)s.a.rd[f])[i]; break;
        }
      }
      if (s.nfields > 0) {
        int dt = s.fdt[0];
        if (is_float(dt)) st_f64(s.a.wr[0], dt, t, ld_f64(s.a.rd[0], dt, i) + g.off[j]);
        else st_i64(s.a.wr[0], dt, t, ld_i64(s.a.rd[0], dt, i) + (int64_t)g.off[j]);
      }
      if (s.mortal) s.a.died_wr[t] = 0;
    }
    if (link_dt < 0) continue;
    const uint64_t nid = ((uint64_t)s.type_nr << SHIFT_TYPE) | nr;
    for (int d = 0; d < 2; d++) {
      int64_t k;
      if (ap.rows) {
        if (!caller) continue;
        k = (int64_t)(2 * q + d);
        ap.rows[k] = (uint32_t)(d == 0 ? i : t);
        ap.srcs[k] = (uint32_t)(d == 0 ? t : i);
      } else {
        k = warp_slot(ap.counter, ap.cap, caller, s.status, 301);
        if (k < 0) continue;
        ap.from[k] = d == 0 ? nid : id;
        ap.to[k] = d == 0 ? id : nid;
        ap.key[k] = order_key(call_pos, i, 2 * j + d);
      }
      if (ap.npayload > 0) st_i64(ap.payload[0], link_dt, k, (int64_t)nid);
    }
  }
}

// link_neighbors: an agent whose field 0 equals die_value returns nothing;
// every other agent keeps its state and, for each source nid of its
// in-edges of type E in insertion order, adds nid -> id and id -> nid of
// type F with payload field 0 = its own field 0.
__global__ void k_link_neighbors(Sweep s, DevCSRView c, Append ap, int pl_dt, int has_die,
                                 double die_value, int call_pos) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool live = i < s.a.n && sw_begin(s, i);
  const int dt0 = s.fdt[0];
  const double v = live && s.nfields > 0 ? ld_f64(s.a.rd[0], dt0, i) : 0.0;
  if (live && has_die && s.nfields > 0 && v == die_value) {
    if (s.writes) sw_die(s, i);
    live = false;
  } else if (live && s.writes) {
    sw_copy(s, i);
  }
  const bool rows = live && i < c.nrows;
  const uint32_t b = rows ? c.row_ptr[i] : 0u;
  const uint32_t deg = rows ? c.row_ptr[i + 1] - b : 0u;
  const uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
  const int64_t vi = live && s.nfields > 0 ? ld_i64(s.a.rd[0], dt0, i) : 0;
  for (uint32_t j = 0; __any_sync(FULL_WARP, j < deg); j++) {
    const bool has = j < deg;
    const uint32_t e = b + j;
    const uint64_t nid =
        has ? ((uint64_t)edge_src_type(c, e) << SHIFT_TYPE) | ((uint64_t)c.src[e] + 1) : 0;
    for (int d = 0; d < 2; d++) {
      const int64_t k = warp_slot(ap.counter, ap.cap, has, s.status, 301);
      if (k < 0) continue;
      ap.from[k] = d == 0 ? nid : id;
      ap.to[k] = d == 0 ? id : nid;
      ap.key[k] = order_key(call_pos, i, 2 * j + d);
      if (ap.npayload > 0) {
        if (is_float(pl_dt)) st_f64(ap.payload[0], pl_dt, k, v);
        else st_i64(ap.payload[0], pl_dt, k, vi);
      }
    }
  }
}

// k_link_neighbors into slots: in-edge e of E gives the records 2 e and 2 e + 1
__global__ void k_link_slots(Sweep s, DevCSRView c, Append ap, int pl_dt, int has_die,
                             double die_value) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool live = i < s.a.n && sw_begin(s, i);
  const int dt0 = s.fdt[0];
  const double v = live && s.nfields > 0 ? ld_f64(s.a.rd[0], dt0, i) : 0.0;
  if (live && has_die && s.nfields > 0 && v == die_value) {
    if (s.writes) sw_die(s, i);
    live = false;
  } else if (live && s.writes) {
    sw_copy(s, i);
  }
  const long long vi = live && s.nfields > 0 ? (long long)ld_i64(s.a.rd[0], dt0, i) : 0;
  uint32_t deg;
  const uint32_t b = row_run(c, i, deg);
  const unsigned alive = __ballot_sync(FULL_WARP, live);
  const uint32_t r0 = (uint32_t)(i & ~31ull);
  warp_edges(b, deg, [&](uint32_t e, unsigned owner, bool has) {
    const double ov = __shfl_sync(FULL_WARP, v, owner);
    const long long oi = __shfl_sync(FULL_WARP, vi, owner);
    if (!has) return;
    const bool swept = alive >> owner & 1u;
    const uint32_t id = r0 + owner;
    uint32_t nid = c.src[e];
    if (swept && nid >= s.a.n) {  // an edge from an agent that does not exist
      set_status(s.status, STATUS_NO_AGENT);
      nid = id;
    }
    ((uint2 *)ap.rows)[e] = swept ? make_uint2(id, nid) : make_uint2(BK_HOLE, BK_HOLE);
    if (!swept) return;
    ((uint2 *)ap.srcs)[e] = make_uint2(nid, id);
    if (ap.npayload > 0)
      for (int d = 0; d < 2; d++) {
        if (is_float(pl_dt)) st_f64(ap.payload[0], pl_dt, 2ull * e + d, ov);
        else st_i64(ap.payload[0], pl_dt, 2ull * e + d, oi);
      }
  });
}

// ----------------------------------------------- move_to! in a transition
// move_to!(sim, raster, id, pos, edge_from_raster, edge_to_raster; distance,
// metric, periodic, only_surrounding) -- src/Raster.jl:437-477 -- called by
// every swept agent: the cell at pos (unless only_surrounding), then the
// cells at the stencil offsets in the reference's order, each wrapped
// (periodic) or dropped when outside the raster (_checkpos,
// src/Raster.jl:479-499); per cell first the cell -> agent edge
// (edge_from_raster), then the agent -> cell edge (edge_to_raster).  The
// order key numbers the calls, so the rebuilt containers hold them in the
// order of the sequential sweep.  The new position: mode 0 the agent's
// fields 0..ndims-1 (1-based; the state is kept); mode 1 the Int field
// `nbr_field` of the agent's first in-neighbour along edge type `nbr_edge`
// in every dimension, which also becomes the agent's field 0 (the rule of
// test/raster.jl:309-314).
struct MoveArgs {
  int ndims;
  int64_t dims[MAX_DIMS];
  int cell_type;
  uint64_t first_nr;
  const int32_t *off;  // noff offsets, ndims each
  int noff;
  int periodic, only_surrounding;
  int mode;
  DevCSRView nbr;       // mode 1: the agent's in-edges
  SrcTable nbr_val;     // mode 1: the neighbours' field, per source type
  int has_from, has_to, same;  // same: one edge type, one buffer for both
  Append from, to;
};

// slot: the call's place among all agents' calls
__device__ __forceinline__ void move_emit(const MoveArgs &m, bool want, const int64_t *p,
                                          uint64_t id, uint64_t slot, uint64_t key, int *status) {
  uint64_t lin = 0, mul = 1;
  for (int d = 0; d < m.ndims; d++) {
    lin += (uint64_t)(p[d] - 1) * mul;
    mul *= (uint64_t)m.dims[d];
  }
  const uint64_t cell = ((uint64_t)m.cell_type << SHIFT_TYPE) | (m.first_nr + lin);
  for (int dir = 0; dir < 2; dir++) {
    if (dir == 0 ? !m.has_from : !m.has_to) continue;  // uniform over the launch
    const Append &ap = (dir == 1 && !m.same) ? m.to : m.from;
    int64_t k;
    if (ap.rows) {
      if (slot == ~0ull) continue;  // no agent
      k = (int64_t)slot;
      if (!want) {
        ap.rows[k] = BK_HOLE;
        continue;
      }
      const uint32_t c32 = (uint32_t)(m.first_nr + lin - 1), a32 = (uint32_t)((id & NR_MASK) - 1);
      ap.rows[k] = dir == 0 ? a32 : c32;
      ap.srcs[k] = dir == 0 ? c32 : a32;
    } else {
      k = warp_slot(ap.counter, ap.cap, want, status, 301);
      if (k < 0) continue;
      ap.to[k] = dir == 0 ? id : cell;
      ap.from[k] = dir == 0 ? cell : id;
      ap.key[k] = key + dir;
    }
    for (int f = 0; f < ap.npayload; f++)  // payload fields zero
      for (int b = 0; b < ap.psize[f]; b++) ((uint8_t *)ap.payload[f])[k * ap.psize[f] + b] = 0;
  }
}

__global__ void k_move_to(Sweep s, MoveArgs m, int call_pos) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < s.a.n && sw_begin(s, i);
  int64_t pos[MAX_DIMS] = {1, 1, 1, 1};
  bool ok = live;
  if (live) {
    if (m.mode == 0) {
      for (int d = 0; d < m.ndims; d++) pos[d] = ld_i64(s.a.rd[d], s.fdt[d], i);
    } else {
      int64_t v = 0;
      const int ty = i < m.nbr.nrows && m.nbr.row_ptr[i + 1] > m.nbr.row_ptr[i]
                         ? edge_src_type(m.nbr, m.nbr.row_ptr[i]) : 0;
      if (ty > 0 && ty < MAX_AGENT_TYPES && m.nbr_val.ptr[ty]) {
        v = ld_i64(m.nbr_val.ptr[ty], m.nbr_val.dt[ty], m.nbr.src[m.nbr.row_ptr[i]]);
      } else if (ty != 0) {
        set_status(s.status, 202);  // source type not readable, or without the field
        ok = false;
      } else {
        set_status(s.status, 203);  // first() of no neighbour
        ok = false;
      }
      for (int d = 0; d < m.ndims; d++) pos[d] = v;
    }
    for (int d = 0; d < m.ndims; d++)
      if (pos[d] < 1 || pos[d] > m.dims[d]) ok = false;
    if (!ok && m.mode == 0) set_status(s.status, 204);  // position outside the raster
    if (s.writes) {
      sw_copy(s, i);
      if (m.mode == 1 && ok) st_i64(s.a.wr[0], s.fdt[0], i, pos[0]);
    }
  }
  const uint64_t id = ((uint64_t)s.type_nr << SHIFT_TYPE) | (i + 1);
  const bool agent = i < s.a.n;
  uint64_t slot = i * (uint64_t)(m.noff + (m.only_surrounding ? 0 : 1));
  if (!m.only_surrounding) {
    move_emit(m, ok, pos, id, agent ? slot : ~0ull, order_key(call_pos, i, 0), s.status);
    slot++;
  }
  for (int k = 0; k < m.noff; k++) {
    int64_t q[MAX_DIMS] = {1, 1, 1, 1};
    bool in = ok;
    for (int d = 0; d < m.ndims; d++) {
      int64_t v = pos[d] + m.off[k * m.ndims + d];
      if (v < 1 || v > m.dims[d]) {
        if (!m.periodic) in = false;
        v = ((v - 1) % m.dims[d] + m.dims[d]) % m.dims[d] + 1;
      }
      q[d] = v;
    }
    move_emit(m, in, q, id, agent ? slot : ~0ull, order_key(call_pos, i, 2 * (uint32_t)(k + 1)),
              s.status);
    slot++;
  }
}

// ---------------------------------------------------------- SIR (cfg 0)
// Person{state::UInt8 (0 S, 1 I, 2 R), days::Int32}.  A susceptible agent
// with k infected in-neighbours is infected with p_k = 1 - (1 - beta)^k
// (p_k from the host table, built by the same repeated multiplication);
// an infected agent recovers when days reaches `recovery`.
constexpr int SIR_U = 16;
constexpr uint64_t SIR_EARLY_EDGES = 400000;

// One SIR step.  Launched with programmatic dependent launch when the
// contact rows cannot be written by the preceding kernel (Sim::csr_epoch):
// this grid lets the next step's grid be scheduled once all its blocks run,
// and each thread requests its row bounds, and with EARLY its first SIR_U
// sources, before griddepcontrol.wait; the states (written by the previous
// step) and every output are touched only after it.  Without the launch
// attribute the wait returns at once.  SIR_U sources are requested together,
// then what they name: for a row of up to SIR_U in-edges two memory round trips
// with EARLY (beside the agent's own state, and the neighbours), else three.
//
// A step that follows a step reads its neighbours from the mask that one left
// (MASK), an eighth of the state bytes: every SM fetches what its rows name once
// per step.  EARLY hides a round trip, but reads the rows of agents that turn
// out not to be susceptible: below SIR_EARLY_EDGES edges the round trip is the
// larger part.  Bound: latency there, else the random reads of the rows.
// Measured, us per step over the first 60 steps of an epidemic (agents x degree).
// Mask, with EARLY and without: 20 000 x 10 3.17 and 3.28; 40 000 x 7 3.84, 4.04;
// 10 000 x 30 2.82, 2.58; 40 000 x 10 3.90, 3.91; 20 000 x 20 3.80, 3.70; 50 000 x
// 10 4.92, 4.71; 25 000 x 20 3.99, 3.81; 100 000 x 5 5.39, 5.44; 24 000 x 30 3.32,
// 2.71; 40 000 x 20 4.73, 4.05; 100 000 x 10 5.30, 5.38; 50 000 x 20 5.49, 4.26;
// 100 000 x 25 6.89, 5.34; 10^6 x 10 19.2, 17.9; 10^6 x 30 35.5, 17.8: the two
// cross near 4*10^5 edges.  State bytes: 20 000 x 10 3.25, 3.35; 40 000 x 10 4.30,
// 4.03; 60 000 x 10 5.33, 4.95; 100 000 x 10 5.90, 5.50; 100 000 x 25 7.14, 5.50;
// 10^6 x 10 22.6, 20.8; 10^6 x 30 40.1, 22.3.
template <bool MASK, bool EARLY>
__global__ void k_sir(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ src,
                      const uint8_t *st_rd, const int32_t *d_rd, uint8_t *st_wr, int32_t *d_wr,
                      uint64_t n, uint64_t nrows, const double *__restrict__ ptab,
                      uint32_t ptab_n, uint64_t seed, uint32_t step, int32_t recovery,
                      int *status, const uint32_t *m_rd, uint32_t *m_wr) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool row = i < n && i < nrows;
  uint32_t q = row ? __ldg(rp + i) : 0u;
  const uint32_t e = row ? __ldg(rp + i + 1) : 0u;
  uint32_t sv[SIR_U];
  if (EARLY) {
#pragma unroll
    for (int u = 0; u < SIR_U; u++) sv[u] = q + u < e ? __ldg(src + q + u) : 0u;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint8_t s = i < n ? st_rd[i] : (uint8_t)3;
  int32_t d = i < n ? d_rd[i] : 0;
  if (s == 0) {
    uint32_t k = 0;
    if (!EARLY) {
#pragma unroll
      for (int u = 0; u < SIR_U; u++) sv[u] = q + u < e ? __ldg(src + q + u) : 0u;
    }
    while (q < e) {
#pragma unroll
      for (int u = 0; u < SIR_U; u++) {
        if (MASK) k += q + u < e ? (m_rd[sv[u] >> 5] >> (sv[u] & 31)) & 1u : 0u;
        else k += (q + u < e ? st_rd[sv[u]] : 0) == 1;
      }
      q += SIR_U;
#pragma unroll
      for (int u = 0; u < SIR_U; u++) sv[u] = q + u < e ? __ldg(src + q + u) : 0u;
    }
    if (k > 0) {
      if (k >= ptab_n) {
        set_status(status, 401);
      } else {
        if (unit_below(philox_u64(philox_draw(seed, i + 1, step, TAG_INFECT)), ptab[k])) {
          s = 1;
          d = 0;
        }
      }
    }
  } else if (s == 1) {
    d = d + 1;
    if (d >= recovery) s = 2;
  }
  if (i < n) {
    st_wr[i] = s;
    d_wr[i] = d;
  }
  const unsigned set = __ballot_sync(0xffffffffu, s == 1);
  if ((threadIdx.x & 31) == 0 && i < n) m_wr[i >> 5] = set;
}

// ------------------------------------------------ Life B3/S23 (cfg 2)
// Cells of a 2-D raster, implicit Moore stencil (chebyshev, distance 1).
// The count of alive neighbours does not depend on edge order.
// Four cells are the bytes of a 32-bit word (byte i = cell x + i): the
// sum of a row's three horizontally adjacent cells for all four bytes at
// once, three rows added and the centre subtracted; with cells of 0 and 1 no
// byte exceeds 8, so none carries into the next.  A warp holds 32 consecutive words of a row;
// the neighbouring words come from the adjacent lanes, and only the warp's
// edge lanes load them.
__device__ __forceinline__ uint32_t life_hsum(uint32_t c, uint32_t lw, uint32_t rw) {
  return __funnelshift_l(lw, c, 8) + c + __funnelshift_r(c, rw, 8);
}
// alive next: a count of three, or of two around a living cell.  For cells of
// 0 and 1 (UNIT) exactly when count | cell is 3: bytes below 16 are zero when
// adding 15 leaves bit 4 clear.  UInt8 cells may hold more, and three byte-wise
// comparisons stay: a cell of 2 beside one neighbour of 1 is not born.
template <bool UNIT>
__device__ __forceinline__ uint32_t life_rule(uint32_t cnt, uint32_t self) {
  if (UNIT) {
    const uint32_t t = (cnt | self) ^ 0x03030303u;
    return ~((t + 0x0f0f0f0fu) >> 4) & 0x01010101u;
  }
  const uint32_t born = __vcmpeq4(cnt, 0x03030303u);
  const uint32_t stay = __vcmpeq4(cnt, 0x02020202u) & __vcmpne4(self, 0u);
  return (born | stay) & 0x01010101u;
}

// blocks of 32 x 8 threads; each thread LIFE_ROWS consecutive rows of one
// word column.  All LIFE_ROWS + 2 rows it reads are requested before any
// is used (one memory latency per thread); rows outside a non-periodic
// raster read as 0, a periodic raster wraps (a compare, no modulo).
// Bound: instruction issue (the 33 MB of a 4096 x 4096 raster stay in L2).
// Measured at 4096 x 4096: 16.8 us per launch with three byte-wise
// comparisons per word and every row tested for the border, 9.9 now (half the
// instructions).
constexpr int LIFE_ROWS = 8;

template <bool UNIT>
__global__ void __launch_bounds__(256) k_life2d_x4(const uint32_t *a, uint32_t *o, int Wq,
                                                   int64_t H, int periodic) {
  let_next_start();
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  const int qx = (int)blockIdx.x * 32 + lane;
  const int64_t y0 = ((int64_t)blockIdx.y * blockDim.y + threadIdx.y) * LIFE_ROWS;
  if (y0 >= H) return;  // warp-uniform
  // each lane's own word; the lane behind the row's last word stands in for
  // the first (its neighbour on a periodic raster); lanes 0 and 31 also load
  // the word beyond theirs
  const int cx = qx < Wq ? qx : 0;
  const bool own = qx < Wq || (qx == Wq && periodic);
  int ex = 0;
  bool edge = false;
  if (lane == 0) {
    ex = qx > 0 ? qx - 1 : Wq - 1;
    edge = qx > 0 || periodic;
  } else if (lane == 31 && qx < Wq) {
    ex = qx + 1 < Wq ? qx + 1 : 0;
    edge = qx + 1 < Wq || periodic;
  }
  uint32_t c[LIFE_ROWS + 2], e[LIFE_ROWS + 2];
  const uint32_t *pc = a + (y0 - 1) * Wq + cx, *pe = a + (y0 - 1) * Wq + ex;
  if (y0 > 0 && y0 + LIFE_ROWS < H) {  // warp-uniform: every row read exists
#pragma unroll
    for (int i = 0; i < LIFE_ROWS + 2; i++) {
      c[i] = own ? pc[(int64_t)i * Wq] : 0u;
      e[i] = edge ? pe[(int64_t)i * Wq] : 0u;
    }
  } else {
#pragma unroll
    for (int i = 0; i < LIFE_ROWS + 2; i++) {
      const int64_t y = y0 - 1 + i;
      const bool use = (y >= 0 && y < H) || (periodic && y <= H);
      const int64_t row = (y < 0 ? H - 1 : y >= H ? 0 : y) * Wq;
      c[i] = use && own ? a[row + cx] : 0u;
      e[i] = use && edge ? a[row + ex] : 0u;
    }
  }
#pragma unroll
  for (int i = 0; i < LIFE_ROWS + 2; i++) {
    const uint32_t l = __shfl_up_sync(0xffffffffu, c[i], 1);
    const uint32_t r = __shfl_down_sync(0xffffffffu, c[i], 1);
    e[i] = life_hsum(c[i], lane == 0 ? e[i] : l, lane == 31 ? e[i] : r);
  }
  if (qx >= Wq) return;
  uint32_t *out = o + y0 * Wq + qx;
  if (y0 + LIFE_ROWS <= H) {
#pragma unroll
    for (int j = 0; j < LIFE_ROWS; j++)
      out[(int64_t)j * Wq] = life_rule<UNIT>(e[j] + e[j + 1] + e[j + 2] - c[j + 1], c[j + 1]);
  } else {
#pragma unroll
    for (int j = 0; j < LIFE_ROWS; j++)
      if (y0 + j < H)
        out[(int64_t)j * Wq] = life_rule<UNIT>(e[j] + e[j + 1] + e[j + 2] - c[j + 1], c[j + 1]);
  }
}

// Moore neighbourhood, one cell per thread: smaller rasters, and UInt8 cells,
// whose values are summed as they are.
__global__ void k_life2d(const uint8_t *__restrict__ a, uint8_t *__restrict__ o,
                         int64_t W, int64_t H, int periodic) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t y = (int64_t)blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  int cnt = 0;
#pragma unroll
  for (int dy = -1; dy <= 1; dy++) {
    int64_t yy = y + dy;
    if (yy < 0 || yy >= H) {
      if (!periodic) continue;
      yy = (yy + H) % H;
    }
#pragma unroll
    for (int dx = -1; dx <= 1; dx++) {
      if (!dx && !dy) continue;
      int64_t xx = x + dx;
      if (xx < 0 || xx >= W) {
        if (!periodic) continue;
        xx = (xx + W) % W;
      }
      cnt += __ldg(a + yy * W + xx);
    }
  }
  uint8_t alive = a[y * W + x];
  o[y * W + x] = (cnt == 3 || (alive && cnt == 2)) ? 1 : 0;
}

// Implicit stencils of any metric on Bool cells, distance up to ROW_D_MAX,
// 2 to 4 dimensions of any size.  A stencil of the reference's metrics is a
// set of rows along the first dimension, each an interval of cells [-r, r]
// around the centre (the centre's own row without the centre): the count is
// the sum of the rows' window sums minus the cell.  Four cells are the bytes
// of a 32-bit word (Bool cells are 0 or 1, and at most 128 offsets fit a
// byte); a window sum grows by two byte-shifted words per step of r.  A
// block of 32 x 8 threads takes a tile of 128 cells x 32 rows of one plane
// (third and fourth coordinate); for every plane the stencil touches it
// stages the tile and its halo in shared memory, wrapping or zeroing outside
// positions there, and each thread adds the rows to the four rows of its
// word column.
// Rows of any length: global words are read aligned and shifted into place,
// and results leave as aligned words put together from two lanes (lane 0
// computes the word before the tile for that), byte by byte only at a row's
// ends.
// Bound: instruction issue, about 50 per cell word of a thread's four and the
// set-up and loads of a tile (ncu: 2.5 instructions per cycle on the busy
// SMs, 55 % of the launch busy).  The kernel before took one cell per thread
// with a 64-bit division and modulo per dimension and a byte load per
// offset.  Measured, us per launch, 2047 x 1531 bounded, euclidean distance
// 2: 100 before, 9.3 now (2, 4, 8 rows per thread: 9.4, 9.3, 11.5).
constexpr int ROW_D_MAX = 4;
constexpr int ROW_RY = 4, ROW_TY = 8 * ROW_RY;
constexpr int ROW_TX = 124;      // cells of a tile: lanes 1 .. 31, lane 0 the word before
constexpr int ROW_WORDS = 34;    // the lanes' words and one on each side
constexpr int ROW_PLANES = 128;

struct RowStencil {
  int64_t dims[MAX_DIMS];  // 1 beyond the raster's dimensions
  uint32_t tx, ty;         // tiles along the first two
  int nplanes, periodic;
  uint32_t birth, survive;
  int noff;
  // the rules as bytes for counts 0 .. 31: entry 8 g + k in byte k of the
  // 64-bit word g (two registers of a byte permutation)
  uint32_t birth_tab[8], survive_tab[8];
  // the planes: offset in the third and fourth dimension, the window radii by
  // dy + D (-1: no row) and the same as row_code (-1: not expressible).  What
  // a launch over one plane reads fits the first lines of the constant bank:
  // each line is a miss of its own at every launch.
  struct Plane {
    int8_t z, v;
    int16_t code;
    int8_t rad[2 * ROW_D_MAX + 1];
  } plane[ROW_PLANES];
};

// radii of the rows dy = 0, +-1, +-2 (-1: no row) of a plane within that
// reach, symmetric in dy
__host__ __device__ constexpr int row_code(int r0, int r1, int r2) {
  return (r0 + 1) | (r1 + 1) << 4 | (r2 + 1) << 8;
}

// adds the plane's rows to the thread's ROW_RY words; CODE -1: radii from rad
template <int D, int CODE>
__device__ __forceinline__ void row_sums(const uint32_t *rows, const int8_t *rad,
                                         uint32_t (&acc)[ROW_RY]) {
  int r[2 * D + 1];
#pragma unroll
  for (int dy = -D; dy <= D; dy++) {
    const int ady = dy < 0 ? -dy : dy;
    r[dy + D] = CODE < 0 ? rad[dy + D] : ady > 2 ? -1 : ((CODE >> (4 * ady)) & 15) - 1;
  }
#pragma unroll
  for (int i = 0; i < ROW_RY + 2 * D; i++) {
    const uint32_t l = rows[i * ROW_WORDS], c = rows[i * ROW_WORDS + 1],
                   n = rows[i * ROW_WORDS + 2];
    uint32_t h[D + 1];
    h[0] = c;
#pragma unroll
    for (int k = 1; k <= D; k++)
      h[k] = h[k - 1] + (k < 4 ? __funnelshift_l(l, c, 8 * k) : l) +
             (k < 4 ? __funnelshift_r(c, n, 8 * k) : n);
#pragma unroll
    for (int j = 0; j < ROW_RY; j++) {
      const int dy = i - j;  // dy + D
      if (dy < 0 || dy > 2 * D) continue;
#pragma unroll
      for (int k = 0; k <= D; k++)
        if (r[dy] == k) acc[j] += h[k];
    }
  }
}

// the next state of a word's four cells: byte permutations look the four
// counts up in the rule's table, eight entries at a time
__device__ __forceinline__ uint32_t row_rule(const RowStencil &s, uint32_t self, uint32_t cnt) {
  if (s.noff > 31) {
    uint32_t w = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t rule = self & (1u << (8 * c)) ? s.survive : s.birth;
      w |= ((rule >> min((cnt >> (8 * c)) & 0xffu, 31u)) & 1u) << (8 * c);
    }
    return w;
  }
  const uint32_t k = cnt & 0x07070707u, pairs = k | (k >> 4);
  const uint32_t sel = __byte_perm(pairs, 0, 0x4420);  // the four counts' low bits as selectors
  const uint32_t alive = self * 0xffu;
  auto look = [&](int g) {
    const uint32_t b = __byte_perm(s.birth_tab[2 * g], s.birth_tab[2 * g + 1], sel);
    const uint32_t v = __byte_perm(s.survive_tab[2 * g], s.survive_tab[2 * g + 1], sel);
    return (v & alive) | (b & ~alive);
  };
  uint32_t w = look(0);
  if (s.noff > 7) {
    const uint32_t b3 = ((cnt >> 3) & 0x01010101u) * 0xffu;
    w = (w & ~b3) | (look(1) & b3);
    if (s.noff > 15) {
      const uint32_t b4 = ((cnt >> 4) & 0x01010101u) * 0xffu;
      w = (w & ~b4) | (((look(2) & ~b3) | (look(3) & b3)) & b4);
    }
  }
  return w;
}

// CODE: the row code of a stencil of one plane (rasters of up to two
// dimensions), -1: any planes
template <int D, int CODE>
__global__ void __launch_bounds__(256, 4) k_life_rows(const uint8_t *a, uint8_t *o,
                                                   const __grid_constant__ RowStencil s) {
  constexpr int ROWS = ROW_TY + 2 * D, LOADS = (ROWS + 7) / 8;
  __shared__ uint32_t t[ROWS * ROW_WORDS];
  const int lane = threadIdx.x;
  const int W = (int)s.dims[0], H = (int)s.dims[1], Z = (int)s.dims[2], V = (int)s.dims[3];
  uint32_t blk = blockIdx.x;
  const int x0 = (int)(blk % s.tx) * ROW_TX;
  blk /= s.tx;
  const int y0 = (int)(blk % s.ty) * ROW_TY;
  blk /= s.ty;
  const int z = (int)(blk % (uint32_t)Z), v = (int)(blk / (uint32_t)Z);
  let_next_start();
  wait_for_previous();
  uint32_t acc[ROW_RY], self[ROW_RY];
#pragma unroll
  for (int j = 0; j < ROW_RY; j++) acc[j] = self[j] = 0;
  const int nplanes = CODE >= 0 ? 1 : s.nplanes;
  for (int p = 0; p < nplanes; p++) {
    int pz = z + (CODE >= 0 ? 0 : s.plane[p].z), pv = v + (CODE >= 0 ? 0 : s.plane[p].v);
    if (pz < 0 || pz >= Z || pv < 0 || pv >= V) {
      if (!s.periodic) continue;  // (block-uniform)
      pz += pz < 0 ? Z : pz >= Z ? -Z : 0;
      pv += pv < 0 ? V : pv >= V ? -V : 0;
    }
    const uint8_t *base = a + (uint64_t)(pv * (int64_t)Z + pz) * ((uint64_t)H * W);
    if (p) __syncthreads();  // the previous plane is read
    // Warp y loads the rows y, y + 8, ..: lane l the word l, lanes 0 and 1
    // also the last two; every load is issued before the first is used.
    // Words not whole inside their row (and the array's last, whose second
    // aligned word would lie behind it) are left 0 here.
    const uint8_t *end = a + (uint64_t)V * Z * H * W;
    const bool xin = x0 >= 8 && x0 + ROW_TX + 8 <= W;  // (block-uniform) no such word
    uint32_t w0[LOADS][2], w1[LOADS][2], sh[LOADS];
#pragma unroll
    for (int u = 0; u < LOADS; u++) {
      const int r = u * 8 + (int)threadIdx.y;  // warp-uniform
      int y = y0 - D + r;
      const bool use = r < ROWS && ((y >= 0 && y < H) || (s.periodic && y < H + D));
      y += y < 0 ? H : y >= H ? -H : 0;
      const uint8_t *row = base + (uint64_t)(use ? y : 0) * W;
      sh[u] = 8 * ((uint32_t)(uint64_t)(row + x0) & 3u);
      const int x = x0 - 8 + 4 * lane;
      const uint32_t *q = (const uint32_t *)((uint64_t)(row + x) & ~3ull);
      const bool in = use && (xin || (x >= 0 && x + 4 <= W && row + x + 8 <= end));
      w0[u][0] = in ? q[0] : 0u;
      w1[u][0] = in ? q[1] : 0u;
      const bool in2 = use && lane < 2 &&
                       (xin || (x + 128 >= 0 && x + 132 <= W && row + x + 136 <= end));
      w0[u][1] = in2 ? q[32] : 0u;
      w1[u][1] = in2 ? q[33] : 0u;
    }
#pragma unroll
    for (int u = 0; u < LOADS; u++) {
      const int r = u * 8 + (int)threadIdx.y;
      if (r >= ROWS) continue;
      t[r * ROW_WORDS + lane] = __funnelshift_r(w0[u][0], w1[u][0], sh[u]);
      if (lane < 2) t[r * ROW_WORDS + lane + 32] = __funnelshift_r(w0[u][1], w1[u][1], sh[u]);
    }
    if (!xin) {
      // the words at the row's ends byte by byte, wrapped or zero outside:
      // the first two of the tile and those around cell W
      __syncthreads();
      const int jr = (W - (x0 - 8)) / 4;
      for (int i = threadIdx.y * 32 + lane; i < ROWS * 8; i += 256) {
        const int r = i / 8, k = i % 8, j = k < 2 ? k : jr + k - 4;
        const int x = x0 - 8 + 4 * j;
        int y = y0 - D + r;
        if (j >= ROW_WORDS || (k >= 2 && j < 2) || !((y >= 0 && y < H) || (s.periodic && y < H + D)))
          continue;
        y += y < 0 ? H : y >= H ? -H : 0;
        const uint8_t *row = base + (uint64_t)y * W;
        if (x >= 0 && x + 4 <= W && row + x + 8 <= end) continue;
        uint32_t w = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          int xc = x + c;
          const bool out = xc < 0 || xc >= W;
          const bool use = !out || (s.periodic && xc >= -D && xc < W + D);
          xc += xc < 0 ? W : out ? -W : 0;
          w |= (use ? (uint32_t)row[xc] : 0u) << (8 * c);
        }
        t[r * ROW_WORDS + j] = w;
      }
    }
    __syncthreads();
    const uint32_t *rows = t + threadIdx.y * ROW_RY * ROW_WORDS + lane;
    if (CODE >= 0) {
      row_sums<D, CODE>(rows, nullptr, acc);
    } else if (D <= 2) {
      switch (s.plane[p].code) {  // (uniform) the planes of the metrics at distance 1 and 2
        case row_code(1, 1, -1): row_sums<D, row_code(1, 1, -1)>(rows, nullptr, acc); break;
        case row_code(1, 0, -1): row_sums<D, row_code(1, 0, -1)>(rows, nullptr, acc); break;
        case row_code(0, -1, -1): row_sums<D, row_code(0, -1, -1)>(rows, nullptr, acc); break;
        default: row_sums<D, -1>(rows, s.plane[p].rad, acc);
      }
    } else {
      row_sums<D, -1>(rows, s.plane[p].rad, acc);
    }
    if (CODE >= 0 || (s.plane[p].z == 0 && s.plane[p].v == 0)) {
#pragma unroll
      for (int j = 0; j < ROW_RY; j++) self[j] = rows[(j + D) * ROW_WORDS + 1];
    }
  }
  const bool border = x0 == 0 || x0 + ROW_TX >= W;  // (block-uniform)
#pragma unroll
  for (int j = 0; j < ROW_RY; j++) {
    const int y = y0 + (int)threadIdx.y * ROW_RY + j;
    if (y >= H) break;  // warp-uniform
    const uint32_t w = row_rule(s, self[j], acc[j] - self[j]);  // (no byte is below its cell)
    // Cells x0 - 4 + 4 lane ..: shifted by the row's misalignment m, every
    // lane but 0 stores the aligned word of cells x0 - 4 + 4 lane - m ..;
    // a row's tiles are shifted alike, so its words are stored once.  At the
    // row's ends the words that are not all in the row go byte by byte.
    const uint64_t row = ((uint64_t)(v * (int64_t)Z + z) * H + y) * W;
    const int m = (int)(row + x0) & 3;
    const uint32_t prev = __shfl_up_sync(0xffffffffu, w, 1);
    const uint32_t u = __funnelshift_l(prev, w, 8 * m);
    const int x = x0 - 4 + 4 * lane - m;
    if (!border) {
      if (lane) *(uint32_t *)(o + row + x) = u;
    } else {
      // the last tile also stores the m cells its last word leaves over
      const bool last = x0 + ROW_TX >= W;
      if (lane && x >= 0 && x + 4 <= W) {
        *(uint32_t *)(o + row + x) = u;
      } else if (lane) {
        for (int c = max(0, -x); c < 4 && x + c < W; c++) o[row + x + c] = (uint8_t)(u >> (8 * c));
      }
      if (last && lane == 31)
        for (int c = 4 - m; c < 4 && x0 + 120 + c < W; c++)
          o[row + x0 + 120 + c] = (uint8_t)(w >> (8 * c));
    }
  }
}

// general implicit stencil (any dims, offsets): count of alive sources
struct StencilArgs {
  int ndims;
  int64_t dims[MAX_DIMS];
  int noff;
  int8_t off[128 * MAX_DIMS];
  int periodic;
};

__global__ void k_life_stencil(const uint8_t *__restrict__ a, uint8_t *__restrict__ o,
                               uint64_t ncells, StencilArgs st, int birth_mask,
                               int survive_mask) {
  uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  int64_t pos[MAX_DIMS];
  uint64_t t = c;
  for (int i = 0; i < st.ndims; i++) {
    pos[i] = (int64_t)(t % st.dims[i]);
    t /= st.dims[i];
  }
  int cnt = 0;
  for (int k = 0; k < st.noff; k++) {
    uint64_t lin = 0, m = 1;
    bool ok = true;
    for (int i = 0; i < st.ndims; i++) {
      int64_t q = pos[i] - st.off[k * st.ndims + i];
      if (q < 0 || q >= st.dims[i]) {
        if (!st.periodic) { ok = false; break; }
        q = ((q % st.dims[i]) + st.dims[i]) % st.dims[i];
      }
      lin += (uint64_t)q * m;
      m *= st.dims[i];
    }
    if (ok) cnt += a[lin];
  }
  uint8_t alive = a[c];
  int bit = cnt < 31 ? (1 << cnt) : 0;
  o[c] = alive ? ((survive_mask & bit) ? 1 : 0) : ((birth_mask & bit) ? 1 : 0);
}

// ------------------------------------------------- random walk (cfg 2)
// Walker{x::Int32, y::Int32} (1-based cell position).  Each step a walker
// moves by one of the 8 Moore offsets, drawn by Philox, wraps (mod1) and
// calls move_to!(sim, raster, id, (x', y'), nothing, OnCell()): one edge
// walker -> cell.  Record i belongs to walker i, so records come out in the
// reference's sweep order without atomics.
__global__ void k_random_walk(const int32_t *__restrict__ x, const int32_t *__restrict__ y,
                              int32_t *__restrict__ xo, int32_t *__restrict__ yo, uint64_t n,
                              int64_t W, int64_t H, uint64_t seed, uint32_t step,
                              uint64_t *__restrict__ to, uint64_t *__restrict__ from,
                              int walker_type, int cell_type, uint64_t cell_first_nr) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Philox4 r = philox_draw(seed, i + 1, step, TAG_MOVE);
  uint32_t k = bounded32(r.v[0], 8);
  // Moore offsets in stencil order (first dimension fastest, centre removed)
  uint32_t m = k < 4 ? k : k + 1;
  int64_t nx = (int64_t)x[i] + (int)(m % 3) - 1;
  int64_t ny = (int64_t)y[i] + (int)(m / 3) - 1;
  nx = ((nx - 1) % W + W) % W + 1;
  ny = ((ny - 1) % H + H) % H + 1;
  xo[i] = (int32_t)nx;
  yo[i] = (int32_t)ny;
  from[i] = ((uint64_t)walker_type << SHIFT_TYPE) | (i + 1);
  to[i] = ((uint64_t)cell_type << SHIFT_TYPE) |
          (cell_first_nr + (uint64_t)(nx - 1) + (uint64_t)(ny - 1) * (uint64_t)W);
}

// The same walk as the rebuild's tile pass: slot i is walker i, whose record
// goes from its registers into the tile's sort.
struct WalkSource {
  static constexpr bool VALS = false;  // the source is the walker, its slot
  const int32_t *__restrict__ x, *__restrict__ y;
  int32_t *__restrict__ xo, *__restrict__ yo;
  int32_t W, H;
  uint64_t seed;
  uint32_t step, cell0;  // row of the raster's first cell
  struct Raw {
    int32_t x, y;
  };
  __device__ __forceinline__ Raw load(uint64_t i) const { return {x[i], y[i]}; }
  __device__ __forceinline__ bool make(uint64_t i, const Raw &p, uint32_t &row,
                                       uint32_t &) const {
    const Philox4 r = philox_draw(seed, i + 1, step, TAG_MOVE);
    const uint32_t k = bounded32(r.v[0], 8), m = k < 4 ? k : k + 1;
    const int32_t nx = move1(p.x, (int)(m % 3) - 1, W), ny = move1(p.y, (int)(m / 3) - 1, H);
    xo[i] = nx;
    yo[i] = ny;
    row = cell0 + (uint32_t)(nx - 1) + (uint32_t)(ny - 1) * (uint32_t)W;
    return true;
  }
  // mod1(v + d, n); from a position inside without a division (out of line,
  // so that the unrolled tile loop stays short)
  static __device__ __noinline__ int32_t move_far(int32_t v, int d, int32_t n) {
    const int64_t w = (int64_t)v + d;
    return (int32_t)(((w - 1) % n + n) % n + 1);
  }
  static __device__ __forceinline__ int32_t move1(int32_t v, int d, int32_t n) {
    if (__builtin_expect((uint32_t)(v - 1) >= (uint32_t)n, 0)) return move_far(v, d, n);
    const uint32_t u = (uint32_t)(v + d);  // 0 .. n + 1
    return u == 0 ? n : u > (uint32_t)n ? 1 : (int32_t)u;
  }
};

__global__ void k_walk_slots(WalkSource w, uint64_t n, uint32_t *__restrict__ rows,
                             uint32_t *__restrict__ srcs) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t row = 0, unused = 0;
  w.make(i, w.load(i), row, unused);
  rows[i] = row;
  srcs[i] = (uint32_t)i;
}

// ------------------------------------------------------------- launchers
Sweep make_sweep(ApplyCtx &c) {
  Sim &s = *c.sim;
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  Sweep w{};
  w.a = agent_view(s, c.call_type);
  w.nfields = (int)ad.fields.size();
  for (int f = 0; f < w.nfields; f++) {
    w.fsize[f] = ad.fields[f].size;
    w.fdt[f] = ad.fields[f].dtype;
  }
  w.mortal = !ad.immortal();
  w.writes = c.writes_call() ? 1 : 0;
  w.type_nr = c.call_type;
  w.status = s.d_status.as<int>();
  if (c.with_edge >= 0) {
    EdgeStore &es = s.edges[c.with_edge];
    if (c.call_type < (int)es.csr.size() && es.csr[c.call_type].row_ptr.p) {
      w.with_rp = es.csr[c.call_type].row_ptr.as<uint32_t>();
      w.with_nrows = es.csr[c.call_type].nrows;
    } else {
      // no agent of this type is the target of such an edge: with_nrows = 0
      // makes every row empty (the pointer is never dereferenced)
      w.with_rp = (const uint32_t *)s.d_status.p;
      w.with_nrows = 0;
    }
  }
  return w;
}

int need_edge_param(ApplyCtx &c, int idx) {
  Sim &s = *c.sim;
  if (idx >= c.nparams) fail(VG_ERR_ARG, "transition parameter missing: edge type");
  int e = (int)c.params[idx];
  s.model->et(e);
  return e;
}

void require_read(ApplyCtx &c, int ref, const std::string &what) {
  if (!c.in_read(ref) && c.sim->check_readable) fail(VG_ERR_ASSERT, what);
}

void require_edge_read(ApplyCtx &c, int e) {
  require_read(c, VG_EDGE(e),
               "You try to access an edge of type " + c.sim->model->et(e).name +
                   " but the type is not in the `read` argument of the apply! function.");
}

void require_agent_read(ApplyCtx &c, int T) {
  require_read(c, T, c.sim->model->at(T).name +
                         " must be in the `read` argument of the transition function.");
}

// the source types present in a CSR must be readable
void require_sources_read(ApplyCtx &c, int e, int T) {
  Sim &s = *c.sim;
  EdgeStore &es = s.edges[e];
  if (T >= (int)es.csr.size()) return;
  CSR &cs = es.csr[T];
  if (cs.nedges == 0) return;
  std::vector<int> types;
  if (cs.src_type_const > 0) {
    types.push_back(cs.src_type_const);
  } else if (cs.src_type_const < 0) {
    std::vector<uint8_t> st(cs.nedges);
    VG_CUDA(cudaMemcpyAsync(st.data(), cs.src_type.p, cs.nedges, cudaMemcpyDeviceToHost, s.stream));
    VG_CUDA(cudaStreamSynchronize(s.stream));
    bool seen[256] = {false};
    for (auto t : st) seen[t] = true;
    for (int t = 1; t < 256; t++)
      if (seen[t]) types.push_back(t);
  }
  for (int t : types) require_agent_read(c, t);
}

SrcTable make_src_table(ApplyCtx &c, int field_index) {
  Sim &s = *c.sim;
  SrcTable t{};
  for (int T = 1; T <= (int)s.model->atypes.size() && T < MAX_AGENT_TYPES; T++) {
    const AgentTypeDesc &ad = s.model->at(T);
    if (field_index < (int)ad.fields.size() && !s.agents[T - 1].rd.empty()) {
      t.ptr[T] = s.agents[T - 1].rd[field_index].p;
      t.dt[T] = ad.fields[field_index].dtype;
    }
    t.died[T] = ad.immortal() ? nullptr : s.agents[T - 1].died_rd.as<uint8_t>();
  }
  return t;
}

void launch_neighbor_op(ApplyCtx &c, int mode) {
  Sim &s = *c.sim;
  int e = need_edge_param(c, 0);
  int sf = (int)c.param(1, 0), df = (int)c.param(2, 0);
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  if (df < 0 || df >= (int)ad.fields.size()) fail(VG_ERR_ARG, "destination field out of range");
  require_edge_read(c, e);
  if (mode != 2) require_sources_read(c, e, c.call_type);
  Sweep w = make_sweep(c);
  DevCSRView v = csr_view(s, e, c.call_type);
  SrcTable t = make_src_table(c, sf);
  if (w.a.n == 0) return;
  const int T = v.src_type || mode == 2 ? 0 : v.src_type_const;
  const unsigned g = nblk(w.a.n);
  const CSR *rows = c.call_type < (int)s.edges[e].csr.size() ? &s.edges[e].csr[c.call_type] : nullptr;
  const bool rows_long =
      neighbor_rows_long(w.a.n, v.nedges, rows && !rows->max_degree_pending ? rows->max_degree : 0);
  auto typed = [&](auto zero) {
    using E = decltype(zero);
    auto k = rows_long ? k_neighbor_typed<E, NB_LONG> : k_neighbor_typed<E, NB_SHORT>;
    k<<<g, TPB, 0, s.stream>>>(w, v, (const E *)t.ptr[T], t.died[T], df, mode);
  };
  // (the last rows' edge indices plus a batch stay below 2^32)
  if (T > 0 && T < MAX_AGENT_TYPES && t.ptr[T] && v.src && v.nedges < UINT32_MAX - NB_LONG) {
    switch (t.dt[T]) {
      case VG_BOOL: case VG_U8: typed(uint8_t()); break;
      case VG_I8: typed(int8_t()); break;
      case VG_U16: typed(uint16_t()); break;
      case VG_I16: typed(int16_t()); break;
      case VG_U32: typed(uint32_t()); break;
      case VG_I32: typed(int32_t()); break;
      case VG_U64: typed(uint64_t()); break;
      case VG_F32: typed(float()); break;
      case VG_F64: typed(double()); break;
      default: typed(int64_t());
    }
  } else {
    k_neighbor_op<<<g, TPB, 0, s.stream>>>(w, v, t, df, mode);
  }
  VG_CUDA(cudaGetLastError());
}

void tr_neighbor_sum(ApplyCtx &c) { launch_neighbor_op(c, 0); }
void tr_neighbor_or(ApplyCtx &c) { launch_neighbor_op(c, 1); }
void tr_count_edges(ApplyCtx &c) { launch_neighbor_op(c, 2); }

void tr_die_if(ApplyCtx &c) {
  Sim &s = *c.sim;
  int kind = (int)c.param(0, 0);
  int field = (int)c.param(1, 0);
  double arg = c.param(2, 0);
  const uint32_t *rp2 = nullptr;
  uint64_t n2 = 0;
  if (kind == 3) {
    int e = field;
    s.model->et(e);
    require_edge_read(c, e);
    DevCSRView v = csr_view(s, e, c.call_type);
    rp2 = v.row_ptr;
    n2 = v.nrows;
    field = 0;
  } else if (kind == 1 || kind == 2) {
    if (field < 0 || field >= (int)s.model->at(c.call_type).fields.size())
      fail(VG_ERR_ARG, "field out of range");
    require_agent_read(c, c.call_type);
  }
  Sweep w = make_sweep(c);
  if (w.a.n == 0) return;
  c.may_die = true;
  k_die_if<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, kind, field, arg, rp2, n2);
  VG_CUDA(cudaGetLastError());
}

void tr_set_field(ApplyCtx &c) {
  Sim &s = *c.sim;
  int field = (int)c.param(0, 0);
  if (field < 0 || field >= (int)s.model->at(c.call_type).fields.size())
    fail(VG_ERR_ARG, "field out of range");
  Sweep w = make_sweep(c);
  if (w.a.n == 0) return;
  k_set_field<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, field, (int)c.param(1, 0), c.param(2, 0));
  VG_CUDA(cudaGetLastError());
}

void tr_keep(ApplyCtx &c) {
  Sim &s = *c.sim;
  Sweep w = make_sweep(c);
  if (w.a.n == 0) return;
  k_keep<<<nblk(w.a.n), TPB, 0, s.stream>>>(w);
  VG_CUDA(cudaGetLastError());
}

// Whether a caller's slots may stay empty: agents that died and agents without
// a with_edge edge are not swept, and their rows may hold edges all the same (a
// dead agent loses its edges when it dies, but walkers move onto dead cells and
// add_edges! takes any target).
bool slots_may_be_empty(const Sweep &w) { return w.mortal || w.with_rp; }

// Whether every cell of a raster is an agent: cells of a mortal type are gone
// after a transition that writes their type anew (no add_existing).  Records onto
// such cells take the general build, which refuses them.
bool cells_exist(const Sim &s, const Raster &R) {
  return R.first_nr - 1 + R.ncells <= s.agents[R.type_nr - 1].n;
}

// T, S: target and source type of every record, when the call's records have
// known slots (0 .. cap - 1 in call order; holes: some may stay empty)
Append make_append(ApplyCtx &c, int e, uint64_t cap, int T = 0, int S = 0, bool holes = false) {
  Sim &s = *c.sim;
  const EdgeTypeDesc &ed = s.model->et(e);
  if (!c.in_write(VG_EDGE(e)) && s.check_readable)
    fail(VG_ERR_ASSERT, ed.name + " must be in the `write` argument of the transition function.");
  const bool typed = T > 0 && S > 0 && c.typed_ok(e, T, S, cap);
  EdgeAppend *a = typed ? c.append_typed(e, T, S, cap, holes, false) : c.append_for(e, cap, false);
  Append ap{};
  if (typed) {
    ap.rows = a->to.as<uint32_t>();
    ap.srcs = a->from.as<uint32_t>();
  } else {
    ap.to = a->to.as<uint64_t>();
    ap.from = a->from.as<uint64_t>();
    ap.key = a->key.as<uint64_t>();
  }
  ap.npayload = (int)a->payload.size();
  for (int f = 0; f < ap.npayload; f++) {
    ap.payload[f] = a->payload[f].p;
    ap.psize[f] = ed.fields[f].size;
  }
  ap.counter = a->counter.as<unsigned long long>();
  ap.cap = a->cap;
  return ap;
}

void tr_self_edge(ApplyCtx &c) {
  Sim &s = *c.sim;
  int e = need_edge_param(c, 0);
  const EdgeTypeDesc &ed = s.model->et(e);
  Sweep w = make_sweep(c);
  if (w.a.n == 0) return;
  Append ap = make_append(c, e, w.a.n, c.call_type, c.call_type, slots_may_be_empty(w));
  // constant payload from params[1..]: one value per field
  std::vector<uint8_t> pl;
  if (ed.stores_payload())
    for (size_t f = 0; f < ed.fields.size(); f++) {
      double v = c.param(1 + (int)f, 0);
      uint8_t buf[8] = {0};
      int dt = ed.fields[f].dtype;
      if (dt == VG_F64) std::memcpy(buf, &v, 8);
      else if (dt == VG_F32) { float x = (float)v; std::memcpy(buf, &x, 4); }
      else { int64_t x = (int64_t)v; std::memcpy(buf, &x, 8); }
      pl.insert(pl.end(), buf, buf + ed.fields[f].size);
    }
  uint8_t *d_pl = (uint8_t *)s.scratch(std::max<size_t>(pl.size(), 8));
  if (!pl.empty())
    VG_CUDA(cudaMemcpyAsync(d_pl, pl.data(), pl.size(), cudaMemcpyHostToDevice, s.stream));
  k_self_edge<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, ap, c.call_pos, d_pl);
  VG_CUDA(cudaGetLastError());
  VG_CUDA(cudaStreamSynchronize(s.stream));
}

void tr_readd_edges(ApplyCtx &c) {
  Sim &s = *c.sim;
  int e = need_edge_param(c, 0);
  const EdgeTypeDesc &ed = s.model->et(e);
  if (ed.stateless() || ed.ignorefrom())
    fail(VG_ERR_ASSERT, "edges is not defined for the hint combination of " + ed.name);
  require_edge_read(c, e);
  Sweep w = make_sweep(c);
  DevCSRView v = csr_view(s, e, c.call_type);
  if (w.a.n == 0) return;
  Append ap = v.nedges && v.nrows <= w.a.n
                  ? make_append(c, e, v.nedges, c.call_type, v.src_type_const,
                                slots_may_be_empty(w))
                  : make_append(c, e, std::max<uint64_t>(v.nedges, 1));
  if (ap.rows) k_readd_slots<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, v, ap);
  else k_readd_edges<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, v, ap, c.call_pos);
  VG_CUDA(cudaGetLastError());
}

void tr_remove_edges(ApplyCtx &c) {
  Sim &s = *c.sim;
  const int E = need_edge_param(c, 0);
  const EdgeTypeDesc &ed = s.model->et(E);
  const int kind = (int)c.param(1, 0);
  const double arg = c.param(2, 0);
  const int mode = (int)c.param(3, 0);
  if (kind < 0 || kind > 2 || mode < 0 || mode > 1) fail(VG_ERR_ARG, "remove_edges: kind 0..2, mode 0..1");
  if (kind == 2 && arg == 0) fail(VG_ERR_ARG, "remove_edges: modulus 0");
  if (!c.in_write(VG_EDGE(E)) && s.check_readable)
    fail(VG_ERR_ASSERT, ed.name + " must be in the `write` argument of the transition function.");
  Sweep w = make_sweep(c);
  DevCSRView v = csr_view(s, E, c.call_type);
  SrcTable t{};
  uint64_t cap = w.a.n;
  if (mode == 1) {
    if (ed.ignorefrom())
      fail(VG_ERR_ASSERT, "remove_edges! with a source agent is not defined for edgetypes "
                          "with the :IgnoreFrom hint.");
    require_edge_read(c, E);
    require_sources_read(c, E, c.call_type);
    t = make_src_table(c, 0);
    cap = v.nedges;
  } else if (kind != 0) {
    require_agent_read(c, c.call_type);
  }
  if (w.a.n == 0) return;
  EdgeRemoval *r = c.removal_for(E, std::max<uint64_t>(cap, 1));
  Removal rm{r->to.as<uint64_t>(), r->from.as<uint64_t>(), r->key.as<uint64_t>(),
             r->counter.as<unsigned long long>(), r->cap};
  k_remove_edges<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, v, t, kind, arg, mode, rm, c.call_pos);
  VG_CUDA(cudaGetLastError());
}

void tr_spawn(ApplyCtx &c) {
  Sim &s = *c.sim;
  const int T = c.call_type;
  const AgentTypeDesc &ad = s.model->at(T);
  const int k = (int)c.param(0, 1);
  if (k < 0 || k > SPAWN_MAX) fail(VG_ERR_ARG, "spawn: 0..8 new agents per caller");
  if (!c.writes_call())
    fail(VG_ERR_ASSERT, ad.name + " must be in the `write` argument of the transition function.");
  if (!ad.fields.empty()) require_agent_read(c, T);
  SpawnArgs g{};
  g.k = k;
  for (int j = 0; j < k; j++) g.off[j] = c.param(1 + j, 0);
  const int link = c.nparams > 1 + k ? (int)c.params[1 + k] : -1;
  int link_dt = -1;
  if (link >= 0) {
    const EdgeTypeDesc &ed = s.model->et(link);
    link_dt = ed.stores_payload() ? ed.fields[0].dtype : VG_I64;
    if (ed.stores_payload() && (link_dt == VG_F32 || link_dt == VG_F64))
      fail(VG_ERR_ARG, "spawn: the link edge's field 0 holds an agent id (an integer)");
  }
  Sweep w = make_sweep(c);
  const uint64_t n = w.a.n;
  if (n == 0) return;
  uint32_t *rank = (uint32_t *)s.work(Sim::WORK_PLACES, n * 4);
  uint32_t *callers = (uint32_t *)s.results(4);
  scan_map<4, uint32_t>(s, n, SpawnCallers{w}, SpawnRanks{rank}, callers);
  uint32_t m = 0;
  s.read_results(&m, callers, 4);
  AgentStore &a = s.agents[T - 1];
  const uint64_t total = (uint64_t)m * k;
  g.nreuse = ad.immortal() ? 0 : a.nreuse;
  g.take = std::min<uint64_t>(total, g.nreuse);
  g.reuse = a.reuse.as<uint64_t>();
  g.n_old = a.n;
  const uint64_t n_new = a.n + (total - g.take);
  agent_reserve(s, T, n_new);  // may move the columns: take the views after it
  Sweep w2 = make_sweep(c);
  Append ap{};
  if (link >= 0 && total > 0) ap = make_append(c, link, 2 * total, T, T);
  if (total > 0)
    k_spawn_new<<<nblk(n), TPB, 0, s.stream>>>(w2, n, rank, g, ap, link >= 0 ? link_dt : -1,
                                               c.call_pos);
  VG_CUDA(cudaGetLastError());
  a.nreuse = g.nreuse - g.take;
  a.n = n_new;
  a.nliving += total;
}

void tr_link_neighbors(ApplyCtx &c) {
  Sim &s = *c.sim;
  const int E = (int)c.param(0, -1), F = (int)c.param(1, -1);
  s.model->et(E);
  const EdgeTypeDesc &fd = s.model->et(F);
  require_edge_read(c, E);
  Sweep w = make_sweep(c);
  if (w.nfields > 0) require_agent_read(c, c.call_type);
  const int has_die = c.nparams > 2;
  c.may_die |= has_die != 0;
  const double die_value = c.param(2, 0);
  DevCSRView v = csr_view(s, E, c.call_type);
  if (w.a.n == 0) return;
  // (with neighbours of the called type every record links it with itself)
  Append ap = v.nedges && v.nrows <= w.a.n && v.src && v.src_type_const == c.call_type
                  ? make_append(c, F, 2 * v.nedges, c.call_type, c.call_type,
                                has_die || slots_may_be_empty(w))
                  : make_append(c, F, std::max<uint64_t>(2 * v.nedges, 1));
  const int pl_dt = fd.stores_payload() ? fd.fields[0].dtype : -1;
  if (ap.rows)
    k_link_slots<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, v, ap, pl_dt, has_die, die_value);
  else
    k_link_neighbors<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, v, ap, pl_dt, has_die, die_value,
                                                        c.call_pos);
  VG_CUDA(cudaGetLastError());
}

void tr_sir(ApplyCtx &c) {
  Sim &s = *c.sim;
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  if (ad.fields.size() < 2 || ad.fields[0].dtype != VG_U8 || ad.fields[1].dtype != VG_I32)
    fail(VG_ERR_ARG, "sir: agent type needs fields (state::UInt8, days::Int32)");
  if (!ad.immortal()) fail(VG_ERR_ARG, "sir: Person is :Immortal");
  int e = need_edge_param(c, 0);
  double beta = c.param(1, 0.05);
  int32_t rec = (int32_t)c.param(2, 7);
  uint64_t seed = (uint64_t)c.param(3, 0);
  require_edge_read(c, e);
  require_agent_read(c, c.call_type);
  if (!c.writes_call()) fail(VG_ERR_ARG, "sir: the called type must be in `write`");
  EdgeStore &es = s.edges[e];
  DevCSRView v = csr_view(s, e, c.call_type);
  if (v.nedges && v.src_type_const != c.call_type)
    fail(VG_ERR_ARG, "sir: contact sources must be of the called type");
  uint32_t maxdeg = c.call_type < (int)es.csr.size() ? csr_max_degree(s, es.csr[c.call_type]) : 0;
  // p_k = 1 - q^k by repeated multiplication, k = 0..maxdeg
  std::vector<double> ptab(maxdeg + 1);
  double q = 1.0, om = 1.0 - beta;
  ptab[0] = 0.0;
  for (uint32_t k = 1; k <= maxdeg; k++) {
    q = q * om;
    ptab[k] = 1.0 - q;
  }
  const double *d_ptab = (const double *)s.const_table("sir.p_infect", ptab.data(), ptab.size() * 8);
  DevAgentView a = agent_view(s, c.call_type);
  if (a.n == 0) return;
  // programmatic dependent launch only while no edge container was written
  // since the previous SIR step (the kernel reads its rows before waiting)
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nblk(a.n));
  cfg.blockDim = dim3(TPB);
  cfg.stream = s.stream;
  cfg.attrs = attr;
  cfg.numAttrs = s.sir_epoch == s.csr_epoch ? 1 : 0;
  Sim::InfectedMask &inf = s.infected;
  const size_t words = (a.n + 31) / 32 * 4;
  // (columns that may change without a call: the step reads the states, and
  // leaves no mask for the next)
  const bool direct = !s.columns_shared;
  const bool mask = direct && inf.call + 1 == s.calls && inf.type == c.call_type &&
                    inf.m[inf.cur].bytes >= words;
  const bool early = v.nedges < SIR_EARLY_EDGES;
  auto kernel = mask ? (early ? k_sir<true, true> : k_sir<true, false>)
                     : (early ? k_sir<false, true> : k_sir<false, false>);
  inf.call = ~1ull;  // (until this apply! has succeeded)
  for (auto &m : inf.m)
    if (m.bytes < words) m.alloc(words + words / 4, &s.footprint);
  VG_CUDA(cudaLaunchKernelEx(&cfg, kernel, v.row_ptr, v.src,
                             (const uint8_t *)a.rd[0], (const int32_t *)a.rd[1],
                             (uint8_t *)a.wr[0], (int32_t *)a.wr[1], a.n, v.nrows, d_ptab,
                             (uint32_t)ptab.size(), seed, (uint32_t)c.step, rec,
                             s.d_status.as<int>(), (const uint32_t *)inf.m[inf.cur].p,
                             inf.m[1 - inf.cur].as<uint32_t>()));
  inf.cur = 1 - inf.cur;
  inf.type = c.call_type;
  inf.pending = direct;
  s.sir_epoch = s.csr_epoch;
}

// Where k_life_rows is the faster form: estimates, in us per launch, of both
// forms, fitted to 2881 pairs of a raster and a stencil that were measured in both (2
// to 4 dimensions, 45 to 2.4*10^7 cells, rows of 2 to 10^6 cells, 1 to 10^6 rows, 4
// to 124 offsets, bounded and periodic).  A tile takes a pass per plane, longer for
// each of its up to 32 rows; four tiles run on an SM at once, so up to 608 tiles the
// launch takes what one SM's tiles take beside one another, beyond that the tiles'
// number times their share.  Whole tiles cost what they cost however few cells they
// hold.  A cell per thread costs each offset's index arithmetic, growing with the
// dimensions, and on a periodic raster a division per coordinate that leaves it, for
// the whole warp when one of its cells does; k_life2d (Moore neighbourhood) costs
// the lanes of its 32-cell blocks.  With these the chosen form is 0.3 % behind the
// faster one on average; at worst it is by rows and takes 21.3 us for 18.7 (27 x 195 x
// 25, 24 offsets), or is not and takes 127 for 95 (11 x 5 x 6 x 256, 88 offsets,
// periodic).  Measured, rows and a cell per thread: 4 offsets 400 x 64 4.2 and 6.3, 33
// x 121212 36 and 57, 1000001 x 2 33 and 29; 12 offsets 2001 x 1000 6.8 and 66; Moore
// 1001 x 1000 5.8 and 10.4, 9 x 111111 35 and 27, 300001 x 3 12.7 and 10.4; 6 offsets 20
// x 8 x 18750 238 and 74, 20 x 33 x 4545 144 and 74, 248 x 32 x 37 8.9 and 12.5, 62 x 24
// x 20 7.8 and 6.3; 26 offsets 9 x 8 x 41666 577 and 260, 300 x 100 x 10 10.4 and 33; 8
// offsets in four dimensions 20 x 32 x 10 x 46 22 and 17; 40 offsets, periodic, 4 x 3 x
// 3535 x 32 5493 and 385.
double rows_us(const RowStencil &rs) {
  const double tiles = (double)rs.tx * rs.ty * rs.dims[2] * rs.dims[3], planes = rs.nplanes;
  const double full = std::min<int64_t>(rs.dims[1], ROW_TY);      // rows of a whole tile
  const double mean = (double)rs.dims[1] / rs.ty;                 // and on average
  const double few = 1.3 + 1.43 * planes + (0.009 + 0.03 * planes) * full +
                     std::min(tiles, 608.0) / 152 *
                         (0.05 + 0.084 * planes + (0.005 + 0.0117 * planes) * full);
  const double many = 1.5 + 1.25 * planes +
                      tiles / 1e3 * (3.2 * planes + (0.08 + 0.09 * planes) * mean);
  return std::max(few, many);
}
double cells_us(const StencilDesc &st, int reach, uint64_t ncells, bool moore2d) {
  const double n = (double)ncells / 1e6;
  // periodic: coordinates of the offsets that may leave the raster, and the share
  // of the warps that hold a cell whose do
  int coords = 0;
  double share = 0;
  if (st.periodic) {
    for (int v : st.offsets) coords += v != 0;
    double before = (double)st.dims[0];
    share = (31 + reach) / before;
    for (int i = 1; i < st.ndims; i++) {
      share += std::min(1.0, reach / (double)st.dims[i] * std::max(1.0, 32 / before));
      before *= (double)st.dims[i];
    }
    share = std::min(share, 1.0);
  }
  if (moore2d)
    return std::max(4.0, 3.7 + n * (6.4 * ((st.dims[0] + 31) / 32 * 32) / st.dims[0] + 6 * share));
  return std::max(4.3 + 0.33 * st.noff + (0.12 * st.ndims - 0.03) * std::max(0, coords - st.noff),
                  3.5 + 0.19 * st.noff +
                      n * (5 + (0.5 + 0.83 * st.ndims) * st.noff + share * coords));
}

// The stencil as rows for k_life_rows; false when it is none (an offset
// beyond ROW_D_MAX, a dimension no larger than the reach, where a position
// can wrap more than once, or a row that is no interval).  Rasters of one
// dimension are one row of the 32 of a tile, and positions beside it lie
// outside the column: 1 000 003 cells at distance 1 and 4 took 38 and 74 us by
// rows, 10.4 and 18.6 a cell per thread.
bool row_stencil(const StencilDesc &st, int birth, int survive, RowStencil &rs, int &reach) {
  reach = 0;
  for (int v : st.offsets) reach = std::max(reach, std::abs(v));
  if (reach < 1 || reach > ROW_D_MAX || st.noff > 128 || st.ndims < 2) return false;
  for (int i = 0; i < MAX_DIMS; i++) {
    rs.dims[i] = i < st.ndims ? st.dims[i] : 1;
    if (i < st.ndims && (rs.dims[i] <= reach || rs.dims[i] >= 1 << 30)) return false;
  }
  // the cells of each (plane, dy) row as a bit set of dx
  std::map<std::array<int, 3>, uint32_t> rows;  // (dv, dz, dy)
  for (int k = 0; k < st.noff; k++) {
    int q[MAX_DIMS] = {0, 0, 0, 0};  // a source lies at minus the offset
    for (int i = 0; i < st.ndims; i++) q[i] = -st.offsets[k * st.ndims + i];
    rows[{q[3], q[2], q[1]}] |= 1u << (q[0] + reach);
  }
  rs.nplanes = 0;
  for (auto &r : rows) {
    const bool centre = r.first == std::array<int, 3>{0, 0, 0};
    const uint32_t bits = r.second | (centre ? 1u << reach : 0u);
    if (centre && (r.second >> reach & 1u)) return false;
    int rad = -1;
    for (int k = 0; k <= reach; k++) {
      uint32_t window = 0;
      for (int x = -k; x <= k; x++) window |= 1u << (x + reach);
      if (bits == window) rad = k;
    }
    if (rad < 0) return false;
    int p = 0;
    while (p < rs.nplanes && (rs.plane[p].z != r.first[1] || rs.plane[p].v != r.first[0])) p++;
    if (p == rs.nplanes) {
      if (p == ROW_PLANES) return false;
      rs.nplanes++;
      rs.plane[p].z = (int8_t)r.first[1];
      rs.plane[p].v = (int8_t)r.first[0];
      std::fill(rs.plane[p].rad, rs.plane[p].rad + 2 * ROW_D_MAX + 1, (int8_t)-1);
    }
    rs.plane[p].rad[r.first[2] + reach] = (int8_t)rad;
  }
  for (int p = 0; p < rs.nplanes; p++) {
    const int8_t *r = rs.plane[p].rad + reach;
    bool fits = true;
    for (int dy = 0; dy <= reach; dy++) fits = fits && r[dy] == r[-dy] && (dy <= 2 || r[dy] < 0);
    rs.plane[p].code = fits ? (int16_t)row_code(r[0], reach > 0 ? r[1] : -1, reach > 1 ? r[2] : -1) : -1;
  }
  if (!rows.count({0, 0, 0})) return false;  // (the kernel takes the cell out of its own row)
  rs.periodic = st.periodic;
  rs.birth = (uint32_t)birth & 0x7fffffffu;  // counts of 31 and more are no rule's
  rs.survive = (uint32_t)survive & 0x7fffffffu;
  rs.noff = st.noff;
  for (int k = 0; k < 8; k++) {
    rs.birth_tab[k] = rs.survive_tab[k] = 0;
    for (int c = 0; c < 4; c++) {
      rs.birth_tab[k] |= (rs.birth >> (4 * k + c) & 1u) << (8 * c);
      rs.survive_tab[k] |= (rs.survive >> (4 * k + c) & 1u) << (8 * c);
    }
  }
  const uint64_t tx = (rs.dims[0] + ROW_TX - 1) / ROW_TX, ty = (rs.dims[1] + ROW_TY - 1) / ROW_TY;
  if (tx * ty * rs.dims[2] * rs.dims[3] >= 1ull << 31) return false;
  rs.tx = (uint32_t)tx;
  rs.ty = (uint32_t)ty;
  return true;
}

void tr_life(ApplyCtx &c) {
  Sim &s = *c.sim;
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  if (ad.fields.empty() || (ad.fields[0].dtype != VG_BOOL && ad.fields[0].dtype != VG_U8))
    fail(VG_ERR_ARG, "life: cell field 0 must be Bool");
  int e = need_edge_param(c, 0);
  EdgeStore &es = s.edges[e];
  if (!es.implicit) fail(VG_ERR_ARG, "life: the neighbour edges must be implicit raster edges");
  require_edge_read(c, e);
  require_agent_read(c, c.call_type);
  if (!c.writes_call()) fail(VG_ERR_ARG, "life: the called type must be in `write`");
  const StencilDesc &st = es.st;
  const Raster &R = s.rasters[st.raster];
  if (R.type_nr != c.call_type) fail(VG_ERR_ARG, "life: raster cells must be the called type");
  AgentStore &A = s.agents[c.call_type - 1];
  if (R.first_nr != 1 || R.ncells != A.n)
    fail(VG_ERR_ARG, "life: the raster must hold all agents of its type");
  const uint8_t *in = A.rd[0].as<uint8_t>();
  uint8_t *out = A.wr[0].as<uint8_t>();
  int birth = (int)c.param(1, 8), survive = (int)c.param(2, 12);  // B3 = 1<<3, S23 = 1<<2|1<<3
  bool moore2d = st.ndims == 2 && st.noff == 8 && birth == 8 && survive == 12;
  if (moore2d) {
    for (int k = 0; k < 8; k++) {
      int ox = st.offsets[2 * k], oy = st.offsets[2 * k + 1];
      if (std::abs(ox) > 1 || std::abs(oy) > 1) moore2d = false;
    }
  }
  RowStencil rs;
  int reach = 0;
  if (moore2d && st.dims[0] % 4 == 0 && st.dims[0] < 1ll << 32) {
    const int64_t Wq = st.dims[0] / 4;
    dim3 blk(32, 8);
    dim3 grd((unsigned)((Wq + 31) / 32),
             (unsigned)((st.dims[1] + 8 * LIFE_ROWS - 1) / (8 * LIFE_ROWS)));
    launch_dependent(ad.fields[0].dtype == VG_BOOL ? k_life2d_x4<true> : k_life2d_x4<false>, grd,
                     blk, 0, s.stream, (const uint32_t *)in, (uint32_t *)out, (int)Wq, st.dims[1],
                     st.periodic);
  } else if (ad.fields[0].dtype == VG_BOOL && row_stencil(st, birth, survive, rs, reach) &&
             1.06 * rows_us(rs) < cells_us(st, reach, R.ncells, moore2d)) {
    const uint64_t blocks = (uint64_t)rs.tx * rs.ty * rs.dims[2] * rs.dims[3];
    dim3 blk(32, 8);
    const int code = rs.nplanes == 1 ? rs.plane[0].code : -1;
    auto k = reach == 1 ? k_life_rows<1, -1> : reach == 2 ? k_life_rows<2, -1>
             : reach == 3 ? k_life_rows<3, -1> : k_life_rows<4, -1>;
    if (reach == 1 && code == row_code(1, 1, -1)) k = k_life_rows<1, row_code(1, 1, -1)>;
    if (reach == 1 && code == row_code(1, 0, -1)) k = k_life_rows<1, row_code(1, 0, -1)>;
    if (reach == 2 && code == row_code(2, 2, 2)) k = k_life_rows<2, row_code(2, 2, 2)>;
    if (reach == 2 && code == row_code(2, 1, 0)) k = k_life_rows<2, row_code(2, 1, 0)>;
    launch_dependent(k, (unsigned)blocks, blk, 0, s.stream, in, out, rs);
  } else if (moore2d) {
    dim3 blk(32, 8);
    dim3 grd((unsigned)((st.dims[0] + 31) / 32), (unsigned)((st.dims[1] + 7) / 8));
    k_life2d<<<grd, blk, 0, s.stream>>>(in, out, st.dims[0], st.dims[1], st.periodic);
  } else {
    if (st.noff > 128) fail(VG_ERR_ARG, "life: at most 128 stencil offsets");
    StencilArgs sa{};
    sa.ndims = st.ndims;
    for (int i = 0; i < st.ndims; i++) sa.dims[i] = st.dims[i];
    sa.noff = st.noff;
    for (int k = 0; k < st.noff * st.ndims; k++) sa.off[k] = (int8_t)st.offsets[k];
    sa.periodic = st.periodic;
    k_life_stencil<<<nblk(R.ncells), TPB, 0, s.stream>>>(in, out, R.ncells, sa, birth, survive);
  }
  VG_CUDA(cudaGetLastError());
}

void tr_random_walk(ApplyCtx &c) {
  Sim &s = *c.sim;
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  if (ad.fields.size() < 2 || ad.fields[0].dtype != VG_I32 || ad.fields[1].dtype != VG_I32)
    fail(VG_ERR_ARG, "random_walk: walker fields (x::Int32, y::Int32)");
  if (!ad.immortal()) fail(VG_ERR_ARG, "random_walk: walkers are :Immortal");
  int e = need_edge_param(c, 0);
  int ri = (int)c.param(1, 0);
  uint64_t seed = (uint64_t)c.param(2, 0);
  if (ri < 0 || ri >= (int)s.rasters.size()) fail(VG_ERR_ARG, "random_walk: raster index");
  const Raster &R = s.rasters[ri];
  if (R.ndims != 2) fail(VG_ERR_ARG, "random_walk: 2-D raster");
  const EdgeTypeDesc &ed = s.model->et(e);
  if (ed.stores_payload()) fail(VG_ERR_ARG, "random_walk: OnCell edges are stateless");
  if (!c.writes_call()) fail(VG_ERR_ARG, "random_walk: the called type must be in `write`");
  if (!c.in_write(VG_EDGE(e)))
    fail(VG_ERR_ASSERT, ed.name + " must be in the `write` argument of the transition function.");
  require_agent_read(c, c.call_type);
  DevAgentView a = agent_view(s, c.call_type);
  if (a.n == 0) return;
  if (cells_exist(s, R) && c.typed_ok(e, R.type_nr, c.call_type, a.n) &&
      !s.edges[e].add_existing && R.dims[0] < (1ll << 31) && R.dims[1] < (1ll << 31)) {
    const BucketPlan plan = plan_buckets(s, e, R.type_nr, a.n, false);
    EdgeAppend *ap = c.append_typed(e, R.type_nr, c.call_type, a.n, false, !plan.sorted);
    ap->plan = plan;
    ap->planned = true;
    WalkSource src{(const int32_t *)a.rd[0], (const int32_t *)a.rd[1], (int32_t *)a.wr[0],
                   (int32_t *)a.wr[1], (int32_t)R.dims[0], (int32_t)R.dims[1], seed,
                   (uint32_t)c.step, (uint32_t)(R.first_nr - 1)};
    if (plan.sorted)
      k_walk_slots<<<nblk(a.n), TPB, 0, s.stream>>>(src, a.n, ap->to.as<uint32_t>(),
                                                    ap->from.as<uint32_t>());
    else
      launch_bucket_tiles(src, plan, s.stream);
    VG_CUDA(cudaGetLastError());
    return;
  }
  EdgeAppend *ap = c.append_for(e, a.n, true);
  ap->fixed_count = a.n;
  k_random_walk<<<nblk(a.n), TPB, 0, s.stream>>>(
      (const int32_t *)a.rd[0], (const int32_t *)a.rd[1], (int32_t *)a.wr[0],
      (int32_t *)a.wr[1], a.n, R.dims[0], R.dims[1], seed, (uint32_t)c.step,
      ap->to.as<uint64_t>(), ap->from.as<uint64_t>(), c.call_type, R.type_nr, R.first_nr);
  VG_CUDA(cudaGetLastError());
}

// apply!(sim, move_to, [T], read, write; params = [raster, edge_from
// (-1: nothing), edge_to (-1: nothing), distance, metric (0 chebyshev, 1
// euclidean, 2 manhatten), periodic, only_surrounding, mode, nbr_edge,
// nbr_field]); mode and the last two as in k_move_to.
void tr_move_to(ApplyCtx &c) {
  Sim &s = *c.sim;
  const AgentTypeDesc &ad = s.model->at(c.call_type);
  const int ri = (int)c.param(0, -1);
  if (ri < 0 || ri >= (int)s.rasters.size()) fail(VG_ERR_ARG, "move_to: raster index");
  const Raster &R = s.rasters[ri];
  const int ef = (int)c.param(1, -1), et = (int)c.param(2, -1);
  const double distance = c.param(3, 0);
  const int metric = (int)c.param(4, VG_METRIC_CHEBYSHEV);
  const int mode = (int)c.param(7, 0);
  if (metric < 0 || metric > 2) fail(VG_ERR_ARG, "move_to: metric 0..2");
  if (mode < 0 || mode > 1) fail(VG_ERR_ARG, "move_to: mode 0 (own fields) or 1 (neighbour)");
  MoveArgs m{};
  m.ndims = R.ndims;
  for (int d = 0; d < R.ndims; d++) m.dims[d] = R.dims[d];
  m.cell_type = R.type_nr;
  m.first_nr = R.first_nr;
  m.periodic = c.param(5, 1) != 0;
  m.only_surrounding = c.param(6, 0) != 0;
  m.mode = mode;
  if (mode == 0) {
    if ((int)ad.fields.size() < R.ndims) fail(VG_ERR_ARG, "move_to: one Int field per dimension");
    for (int d = 0; d < R.ndims; d++)
      if (ad.fields[d].dtype == VG_F32 || ad.fields[d].dtype == VG_F64)
        fail(VG_ERR_ARG, "move_to: the position fields are integers");
    require_agent_read(c, c.call_type);
  } else {
    const int ne = need_edge_param(c, 8);
    require_edge_read(c, ne);
    require_sources_read(c, ne, c.call_type);
    m.nbr = csr_view(s, ne, c.call_type);
    if (ad.fields.empty() || ad.fields[0].dtype == VG_F32 || ad.fields[0].dtype == VG_F64)
      fail(VG_ERR_ARG, "move_to: mode 1 writes the position to an Int field 0");
    const int nf = (int)c.param(9, 0);
    if (nf < 0) fail(VG_ERR_ARG, "move_to: neighbour field");
    m.nbr_val = make_src_table(c, nf);
  }
  Sweep w = make_sweep(c);
  if (w.a.n == 0) return;
  std::vector<int> off = distance >= 1 ? make_stencil(metric, R.ndims, distance) : std::vector<int>();
  m.noff = (int)(off.size() / std::max(1, R.ndims));
  if (m.noff > (1 << 18)) fail(VG_ERR_ARG, "move_to: stencil too large");
  std::vector<int32_t> off32(off.begin(), off.end());
  const std::string key = "move_to:" + std::to_string(metric) + ":" + std::to_string(R.ndims) +
                          ":" + std::to_string(distance);
  m.off = off32.empty() ? nullptr
                        : (const int32_t *)s.const_table(key, off32.data(), off32.size() * 4);
  const uint64_t per = (uint64_t)(m.only_surrounding ? 0 : 1) + (uint64_t)m.noff;
  m.has_from = ef >= 0;
  m.has_to = et >= 0;
  m.same = m.has_from && m.has_to && ef == et;
  // (positions beyond a bounded raster leave their slots empty; one outside a
  // periodic raster is an error, status 204, which is read before the rebuild
  // unless transitions are queued)
  const bool typed = per > 0 && !m.same && cells_exist(s, R);
  const bool holes = slots_may_be_empty(w) || !m.periodic || mode == 1 || s.async;
  const int T = typed ? c.call_type : 0, R_T = typed ? R.type_nr : 0;
  if (m.has_from)
    m.from = make_append(c, ef, std::max<uint64_t>(1, w.a.n * per * (m.same ? 2 : 1)), T, R_T, holes);
  if (m.has_to && !m.same)
    m.to = make_append(c, et, std::max<uint64_t>(1, w.a.n * per), R_T, T, holes);
  k_move_to<<<nblk(w.a.n), TPB, 0, s.stream>>>(w, m, c.call_pos);
  VG_CUDA(cudaGetLastError());
}

}  // namespace

const std::vector<TransitionDef> &transitions() {
  static const std::vector<TransitionDef> defs = {
      {"bounded_confidence", tr_bounded_confidence},
      {"sir", tr_sir},
      {"life", tr_life},
      {"random_walk", tr_random_walk},
      {"move_to", tr_move_to},
      {"neighbor_sum", tr_neighbor_sum},
      {"neighbor_or", tr_neighbor_or},
      {"count_edges", tr_count_edges},
      {"die_if", tr_die_if},
      {"set_field", tr_set_field},
      {"keep", tr_keep},
      {"self_edge", tr_self_edge},
      {"readd_edges", tr_readd_edges},
      {"spawn", tr_spawn},
      {"link_neighbors", tr_link_neighbors},
      {"remove_edges", tr_remove_edges},
  };
  return defs;
}

}  // namespace vg
