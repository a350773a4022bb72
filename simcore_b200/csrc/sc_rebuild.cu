// Pair-list rebuild of a context (InteractionManager::UpdateInteractions,
// src/interaction_manager.cpp:211-231, over CellList::MakePairs,
// src/cell_list.cpp:139-199, and Cell::MakePairs, src/cell.cpp:14-70).
//
// The bonds of the rebuilt systems are sorted by cell with a two-level
// (most-significant-digit first) radix sort on the cell key: a counting pass
// on the high digits -- the group of 32 consecutive cells, one occupancy word
// -- and then, inside every group, each bond's rank by (cell, bond id).  The
// ranking keeps every cell's bonds in bond order, the order in which
// Cell::AddObj appends them.  The counting pass scans one counter per group
// (n_cells / 32 of them), not the cell grid; cell ranges and occupancy bits
// are written where cells start and end in the sorted order.
//
//   k_rb_keys      ZeroDrTot and the rebuild counters; cell key of every
//                  bond, group counts; clears the occupancy words and the
//                  per-bond entry counts of the rebuilt systems
//   (scan)         group offsets
//   k_rb_scatter   bonds into their groups (counts back to zero)
//   k_rb_rank      stable order inside each group; cell ranges and bits
//   k_rb_count     each cell's pairs in the reference's order, as candidates
//                  (one reservation per block), their count at the cell's
//                  head entry, per-bond entry counts
//   (scan)         pair offsets and entry offsets, one scan of both
//   k_rb_place     candidates to their list slots, stored forces zeroed,
//                  per-bond entries (pair << 1 | role)
//   k_rb_csr_sort  entries in pair order, slots of both roles, ranges
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "sc_cells.cuh"
#include "sc_common.cuh"
#include "sc_kernels.h"
#include "sc_launch.h"

namespace sc {

// Bonds of the rebuilt systems: cell key (system's first cell + cell within
// it) and warp-aggregated group counts; others get the sentinel n_cells.  The
// bond's thread also does InteractionManager::ZeroDrTot (src/
// interaction_manager.cpp:316-321) for its first site, the last bond's of a
// filament for its last site too: nothing in the rebuild moves the sites, and
// the thread has both in hand.  Clears the occupancy words of the rebuilt
// systems (each system's cells start at a multiple of 32: a word, a group,
// belongs to one system, grp_rep's).
// Bound by memory latency: 71,758 filaments in 64 systems took 40 us with
// three dependent lookups a site for its system and every thread walking the
// systems one after another for their words, 8.9 us now.
__device__ __forceinline__ void rb_systems(const DevState &d, const RebuildBufs &rb, int tid,
                                           int nthreads) {
  if (tid == 0) {
    *d.n_rebuilds += 1;
    *rb.cand_n = 0;
  }
  for (int r = tid; r < d.nrep; r += nthreads) {
    if (!d.due[r]) continue;
    d.dr_max_bits[r] = 0ull;
    d.rep_rebuilds[r] += 1;
  }
  for (int w = tid; w < rb.n_groups; w += nthreads)
    if (d.nrep == 1 || d.due[rb.grp_rep[w]]) rb.occ[w] = 0u;
}

// (A whole warp's consecutive bonds; those past the last do nothing.)
template <int ND>
__device__ __forceinline__ void rb_key(const SysConst &k, const DevState &d, const RebuildBufs &rb,
                                       int b) {
  bool in = false;
  int g = 0;
  if (b < d.nb) {
    uint32_t c = (uint32_t)k.n_cells;
    const int r = rep_of_bond(d, b);
    if (d.due[r]) {
      rb.deg[b] = 0;
      const ReplicaConst &R = d.rep[r];
      const int f = d.bond_fil[b], s = b + f;
      const bool tail = b + 1 >= d.nb || d.bond_fil[b + 1] != f;
      double r1[3], r2[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        r1[i] = d.r[i][s];
        r2[i] = d.r[i][s + 1];
      }
      int xyz[3];
      c = (uint32_t)(R.cell0 + bond_cell_of<ND>(d, R, r1, r2, xyz));
      in = true;
      g = (int)(c >> 5);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        d.dz[i][s] = r1[i];
        if (tail) d.dz[i][s + 1] = r2[i];
      }
      d.dt[s] = 0.0;
      if (tail) d.dt[s + 1] = 0.0;
    }
    rb.key[b] = c;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, in);
  if (in) {
    const unsigned peers = __match_any_sync(mask, g);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&rb.gcount[g], __popc(peers));
  }
}

template <int ND>
__global__ void __launch_bounds__(256) k_rb_keys(SysConst k, DevState d, RebuildBufs rb) {
  grid_dep_sync();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  rb_systems(d, rb, tid, gridDim.x * blockDim.x);
  rb_key<ND>(k, d, rb, tid);
}

// Each rebuilt bond into its group's range of the scanned offsets (any
// order inside the group); decrements the counts back to zero, ready for
// the next rebuild.
__device__ __forceinline__ void rb_scatter(const DevState &d, const RebuildBufs &rb, int b) {
  if (b >= d.nb || !d.due[rep_of_bond(d, b)]) return;
  const int g = (int)(rb.key[b] >> 5);
  const int slot = atomicSub(&rb.gcount[g], 1) - 1;
  rb.tmp[rb.gstart[g] + slot] = b;
}

__global__ void k_rb_scatter(DevState d, RebuildBufs rb) {
  grid_dep_sync();
  rb_scatter(d, rb, blockIdx.x * blockDim.x + threadIdx.x);
}

// Sorted position of every rebuilt bond: its group's first entry plus the
// number of bonds of the group that come before it by (cell, bond id).  The
// first of a cell writes the cell's start and occupancy bit, the last its
// end.
__device__ __forceinline__ void rb_rank(const DevState &d, const RebuildBufs &rb, int q) {
  if (q >= rb.gstart[rb.n_groups]) return;
  const int b = rb.tmp[q];
  const uint32_t c = rb.key[b];
  const int g = (int)(c >> 5);
  const int s = rb.gstart[g], e = rb.gstart[g + 1];
  int rank = 0;
  bool first = true, last = true;
  for (int j = s; j < e; ++j) {
    const int bj = rb.tmp[j];
    const uint32_t cj = rb.key[bj];
    rank += (cj < c || (cj == c && bj < b)) ? 1 : 0;
    if (cj == c) {
      first = first && !(bj < b);
      last = last && !(bj > b);
    }
  }
  const int pos = s + rank;
  rb.skey[pos] = c;
  rb.sval[pos] = b;
  if (first) {
    rb.range[c].x = pos;
    atomicOr(&rb.occ[c >> 5], 1u << (c & 31));
  }
  if (last) rb.range[c].y = pos + 1;
}

__global__ void k_rb_rank(DevState d, RebuildBufs rb) {
  grid_dep_sync();
  rb_rank(d, rb, blockIdx.x * blockDim.x + threadIdx.x);
}

__device__ __forceinline__ bool occupied(const unsigned *occ, int c) {
  return (occ[c >> 5] >> (c & 31)) & 1u;
}

// Sorted span [lo, hi) of system R's bonds: its groups' entries.
__device__ __forceinline__ int sys_lo(const RebuildBufs &rb, const ReplicaConst &R) {
  return rb.gstart[R.cell0 >> 5];
}
__device__ __forceinline__ int sys_hi(const RebuildBufs &rb, const ReplicaConst &R) {
  return rb.gstart[(R.cell0 + R.n_cells + 31) >> 5];
}

// The cell whose head is sorted entry q: its m members, its half-shell
// neighbours (context cell indices; -1 where the wrap gives the cell itself
// or, in 2D, a third dimension) and their sorted ranges (empty where
// unoccupied), and the mask of non-empty neighbours.
struct CellHead {
  int c, m;
  const int *it;
  int nbr[13], s0[13], s1[13];
  unsigned busy;
};

__device__ __forceinline__ void cell_head(const SysConst &k, const RebuildBufs &rb,
                                          const ReplicaConst &R, int q, int c, CellHead &h) {
  h.c = c;
  h.m = rb.range[c].y - q;
  h.it = rb.sval + q;
  int x, y, z;
  cell_coords(R, c - R.cell0, x, y, z);
  const unsigned keep = half_shell_fixed(k, R, x, y, z, h.nbr);
  h.busy = 0;
#pragma unroll
  for (int kk = 0; kk < 13; ++kk) {  // all ranges loaded together
    h.s0[kk] = h.s1[kk] = 0;
    h.nbr[kk] += R.cell0;
    if ((keep >> kk) & 1u) {
      if (occupied(rb.occ, h.nbr[kk])) {
        const int2 g = rb.range[h.nbr[kk]];
        h.s0[kk] = g.x;
        h.s1[kk] = g.y;
        h.busy |= 1u << kk;
      }
    } else {
      h.nbr[kk] = -1;  // matches no cell key
    }
  }
}

// Calls f(a, b) for the cell's pairs in the reference's list order
// (Cell::MakePairs, src/cell.cpp:14-22): pairs inside the cell, then with
// each half-shell neighbour in order, less those pair_excluded drops.  Only
// the non-empty neighbours are visited (a warp steps through as many as its
// busiest lane has, not all 13).
template <class F>
__device__ __forceinline__ void cell_pairs_visit(const SysConst &k, const DevState &d,
                                                 const RebuildBufs &rb, const CellHead &h,
                                                 F &&f) {
  const int m = h.m;
  for (int i = 0; i < m - 1; ++i)
    for (int j = i + 1; j < m; ++j) {
      const int a = h.it[i], b = h.it[j];
      if (!pair_excluded(k, d, a, b)) f(a, b);
    }
  unsigned busy = h.busy;
  while (busy) {
    const int kk = __ffs(busy) - 1;
    busy &= busy - 1;
    int lo = 0, hi = 0;
#pragma unroll
    for (int q2 = 0; q2 < 13; ++q2)
      if (q2 == kk) {
        lo = h.s0[q2];
        hi = h.s1[q2];
      }
    for (int i = 0; i < m; ++i)
      for (int j = lo; j < hi; ++j) {
        const int a = h.it[i], b = rb.sval[j];
        if (!pair_excluded(k, d, a, b)) f(a, b);
      }
  }
}

// Each cell's pairs, found once: the head entry of a cell collects them (the
// first kHeadBuf in shared memory, all again in the rare longer case), takes
// a run of candidate slots from one reservation per block, and writes them
// there in order; it records their count (0 at the other entries) and adds
// each pair to both bonds' entry counts.  Candidates past cand_cap are
// dropped: their system's list then outgrows its segment, which k_rb_place
// reports.
constexpr int kCountBlock = 128;
constexpr int kHeadBuf = 8;

// (A block's consecutive entries; called by all of its BLOCK threads.)
template <int BLOCK>
__device__ __forceinline__ void rb_count(const SysConst &k, const DevState &d,
                                         const RebuildBufs &rb, int q, int2 (*sbuf)[kHeadBuf],
                                         int *swarp) {
  const int t = threadIdx.x, lane = t & 31;
  int cnt = 0;
  const ReplicaConst *R = nullptr;
  int c = 0;
  if (q < d.nb && q < rb.gstart[rb.n_groups] && k.like_like) {
    c = (int)rb.skey[q];
    if (q == 0 || (int)rb.skey[q - 1] != c) {
      R = &d.rep[d.nrep > 1 ? rep_of_bond(d, rb.sval[q]) : 0];
      CellHead h;
      cell_head(k, rb, *R, q, c, h);
      cell_pairs_visit(k, d, rb, h, [&](int a, int b) {
        if (cnt < kHeadBuf) sbuf[t][cnt] = make_int2(a, b);
        atomicAdd(&rb.deg[a], 1);
        atomicAdd(&rb.deg[b], 1);
        ++cnt;
      });
    }
  }
  // The block's candidate slots: a scan of the counts, one atomic.
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) swarp[t >> 5] = incl;
  __syncthreads();
  if (t == 0) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < BLOCK / 32; ++w) {
      const int v = swarp[w];
      swarp[w] = run;
      run += v;
    }
    const int base = run > 0 ? atomicAdd(rb.cand_n, run) : 0;
#pragma unroll
    for (int w = 0; w < BLOCK / 32; ++w) swarp[w] += base;
  }
  __syncthreads();
  const int t0 = swarp[t >> 5] + incl - cnt;
  if (cnt > 0 && cnt <= kHeadBuf) {
    for (int i = 0; i < cnt; ++i)
      if (t0 + i < rb.cand_cap) rb.cand[t0 + i] = make_int4(sbuf[t][i].x, sbuf[t][i].y, q, 0);
  } else if (cnt > kHeadBuf) {
    CellHead h;
    cell_head(k, rb, *R, q, c, h);
    int i = 0;
    cell_pairs_visit(k, d, rb, h, [&](int a, int b) {
      if (t0 + i < rb.cand_cap) rb.cand[t0 + i] = make_int4(a, b, q, 0);
      ++i;
    });
  }
  if (q < d.nb) {
    rb.pair_count[q] = cnt;
    rb.cand_start[q] = t0;
  }
}

__global__ void __launch_bounds__(kCountBlock) k_rb_count(SysConst k, DevState d, RebuildBufs rb) {
  __shared__ int2 sbuf[kCountBlock][kHeadBuf];
  __shared__ int swarp[kCountBlock / 32];
  grid_dep_sync();
  rb_count<kCountBlock>(k, d, rb, blockIdx.x * blockDim.x + threadIdx.x, sbuf, swarp);
}

// First entry slot of bond b (rebuilt system R): its system's slots start at
// 2 p0, its bonds' entries follow in bond order.
__device__ __forceinline__ int entry_first(const RebuildBufs &rb, const ReplicaConst &R, int b) {
  return 2 * R.p0 + (rb.deg_off[b] - rb.deg_off[R.b0]);
}

// Every candidate to its slot -- its cell's scanned offset in its system's
// pair segment plus its place among the cell's candidates (slots past the
// segment are not written) -- with the new pair's stored force (and virial
// record) zeroed and both of its per-bond entries (pair << 1 | role; role 0
// = obj1, 1 = obj2) in any order, the entry counts going back to zero.  A
// system whose list outgrew its segment gets no entries: its step stops on
// the overflow bit and is redone.  Threads u < nrep record their system's
// pair count (the count is kept so the host can size the segment).
__device__ __forceinline__ void rb_place(const DevState &d, const RebuildBufs &rb, int prec,
                                         int u) {
  if (u < d.nrep && d.due[u]) {
    const ReplicaConst &R = d.rep[u];
    const int np = rb.pair_off[sys_hi(rb, R)] - rb.pair_off[sys_lo(rb, R)];
    d.np_rep[u] = np;
    if (np > R.pcap) atomicOr(d.status, ST_LIST_OVERFLOW);
  }
  if (u >= min(*rb.cand_n, rb.cand_cap)) return;
  const int4 e = rb.cand[u];
  const int q = e.z;
  const ReplicaConst &R = d.rep[d.nrep > 1 ? rep_of_bond(d, e.x) : 0];
  const int lo = rb.pair_off[sys_lo(rb, R)];
  const bool fits = rb.pair_off[sys_hi(rb, R)] - lo <= R.pcap;
  const int p = rb.pair_off[q] - lo + (u - rb.cand_start[q]);
  if (p < R.pcap) {
    const int g = R.p0 + p;
    d.pa[g] = e.x;
    d.pb[g] = e.y;
    if (prec == 0) {
      double2 *st = reinterpret_cast<double2 *>(d.pf64) + 2 * (size_t)g;
      st[0] = make_double2(0.0, 0.0);
      st[1] = make_double2(0.0, 0.0);
      if (d.pv64) {  // a new Interaction's stress and potential are 0
        double2 *v = reinterpret_cast<double2 *>(d.pv64) + 2 * (size_t)g;
        v[0] = make_double2(0.0, 0.0);
        v[1] = make_double2(0.0, 0.0);
      }
    } else {
      reinterpret_cast<float4 *>(d.pf32)[g] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (d.pv32) reinterpret_cast<float4 *>(d.pv32)[g] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (fits) {
      const int sa = atomicSub(&rb.deg[e.x], 1) - 1;
      const int sb = atomicSub(&rb.deg[e.y], 1) - 1;
      d.e_ent[entry_first(rb, R, e.x) + sa] = g << 1;
      d.e_ent[entry_first(rb, R, e.y) + sb] = (g << 1) | 1;
    }
  }
}

__global__ void k_rb_place(DevState d, RebuildBufs rb, int prec) {
  grid_dep_sync();
  rb_place(d, rb, prec, blockIdx.x * blockDim.x + threadIdx.x);
}

// The wn entries at w0 sorted by the whole warp (`own`: the list's own lane).
// Each lane ranks up to four entries, read before any is written; lists beyond
// 128 entries, which no stable system has, are sorted by their lane in memory.
// A function of its own: a few bonds in a dense system reach it.
static __device__ __noinline__ void sort_long_list(int *e_ent, int *pos1, int *pos2, int w0, int wn,
                                                   bool own) {
  const int lane = threadIdx.x & 31;
  int *e = e_ent + w0;
  constexpr int PER = 4;
  if (wn <= 32 * PER) {
    int v[PER], rank[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = lane + 32 * i < wn ? e[lane + 32 * i] : 0x7fffffff;
      rank[i] = 0;
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int m = min(32, wn - 32 * q);
      for (int j = 0; j < m; ++j) {
        const int x = __shfl_sync(0xffffffffu, v[q], j);
#pragma unroll
        for (int i = 0; i < PER; ++i) rank[i] += x < v[i] ? 1 : 0;  // (entries are distinct)
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < wn) {
        const int at = w0 + rank[i];
        e_ent[at] = v[i];
        if (v[i] & 1) pos2[v[i] >> 1] = at;
        else pos1[v[i] >> 1] = at;
      }
  } else if (own) {
    for (int i = 1; i < wn; ++i) {
      const int v = e[i];
      int j = i - 1;
      while (j >= 0 && e[j] > v) {
        e[j + 1] = e[j];
        --j;
      }
      e[j + 1] = v;
    }
    for (int i = 0; i < wn; ++i) {
      const int ent = e[i];
      if (ent & 1) pos2[ent >> 1] = w0 + i;
      else pos1[ent >> 1] = w0 + i;
    }
  }
}

// Each bond's entries sorted by pair index -- the order in which the
// reference's serial ApplyPairInteractions adds them to the bond; the slot of
// each (pair, role) entry; the bond's entry range.  Up to kRegEntries entries
// are sorted in registers by the bond's thread; longer lists, a few bonds in a
// dense system, by the whole warp, one after another: every lane ranks its
// entries against all of them, read together.  (One thread's insertion sort in
// memory made the kernel wait for its longest list: 3,000 filaments of 50
// bonds, 388,000 pairs, 43 us, 22 us now.)
constexpr int kRegEntries = 16;

// (A whole warp's consecutive bonds.)
__device__ __forceinline__ void rb_csr_sort(const DevState &d, const RebuildBufs &rb, int b) {
  const int lane = threadIdx.x & 31;
  int e0 = 0, n = 0;
  if (b < d.nb) {
    const int r = rep_of_bond(d, b);
    const ReplicaConst &R = d.rep[r];
    // (A list that outgrew its segment gets no entries.)
    if (d.due[r] && d.np_rep[r] <= R.pcap) {
      e0 = entry_first(rb, R, b);
      n = rb.deg_off[b + 1] - rb.deg_off[b];
      d.e_off[b] = e0;
      d.e_cnt[b] = n;
    }
  }
  if (n > 0 && n <= kRegEntries) {
    int *e = d.e_ent + e0;
    int v[kRegEntries];
#pragma unroll
    for (int i = 0; i < kRegEntries; ++i) v[i] = i < n ? e[i] : 0x7fffffff;
    // Odd-even transposition sort: kRegEntries rounds sort kRegEntries keys.
#pragma unroll
    for (int round = 0; round < kRegEntries; ++round) {
#pragma unroll
      for (int i = round & 1; i + 1 < kRegEntries; i += 2) {
        const int lo = min(v[i], v[i + 1]), hi = max(v[i], v[i + 1]);
        v[i] = lo;
        v[i + 1] = hi;
      }
    }
#pragma unroll
    for (int i = 0; i < kRegEntries; ++i) {
      if (i < n) {
        e[i] = v[i];
        if (v[i] & 1) d.pos2[v[i] >> 1] = e0 + i;
        else d.pos1[v[i] >> 1] = e0 + i;
      }
    }
  }
  unsigned longer = __ballot_sync(0xffffffffu, n > kRegEntries);
  while (longer) {
    const int src = __ffs(longer) - 1;
    longer &= longer - 1;
    const int w0 = __shfl_sync(0xffffffffu, e0, src), wn = __shfl_sync(0xffffffffu, n, src);
    sort_long_list(d.e_ent, d.pos1, d.pos2, w0, wn, lane == src);
    __syncwarp();
  }
}

__global__ void k_rb_csr_sort(DevState d, RebuildBufs rb) {
  grid_dep_sync();
  rb_csr_sort(d, rb, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---- a chained step's control: bookkeeping, decision, rebuild in one kernel ---
// A graph's loop pays 9 us a BD step for its conditional nodes, a third of a
// small system's step.  Small contexts run without them: their steps are
// launched one after another, and one cluster of blocks between them ends a
// step, decides the next one's rebuild and does it when due, phase by phase
// over the hardware's cluster barrier (the kernels above, over all items in
// turn).  2,000 bonds, 10 BD steps: 320 us with the loop, 270 so.  Idle it is
// bound by its launch and three dependent round trips to L2 (4 us); a rebuild
// by the phases' latencies, 36 us at 2,000 bonds (as the ten kernels), 125 at
// 20,000.  A cluster and not the chip: its barrier needs no waiting loop and
// no cooperative launch.
constexpr int kCtlBlocks = 8;  // the portable cluster size
constexpr int kCtlThreads = 512;

// Exclusive prefix sums of in[0, n) into out[0, n], the total last, by the
// cluster: a run of entries per block.  tot: kCtlBlocks, part: one per warp.
static __device__ __noinline__ void cluster_scan(const int *in, int *out, int n, int *tot,
                                                 int *part) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int tiles = (n + kCtlThreads - 1) / kCtlThreads;
  const int run = (tiles + kCtlBlocks - 1) / kCtlBlocks * kCtlThreads;
  const int lo = min(rank * run, n), hi = min(lo + run, n);
  int sum = 0;
  for (int i = lo + t; i < hi; i += kCtlThreads) sum += in[i];
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if (lane == 0) part[w] = sum;
  __syncthreads();
  if (t < kCtlBlocks) {
    int all = 0;
    for (int i = 0; i < kCtlThreads / 32; ++i) all += part[i];
    cl.map_shared_rank(tot, t)[rank] = all;
  }
  cl.sync();
  int base = 0, total = 0;
  for (int i = 0; i < kCtlBlocks; ++i) {
    if (i < rank) base += tot[i];
    total += tot[i];
  }
  if (rank == 0 && t == 0) out[n] = total;
  for (int i0 = lo; i0 < hi; i0 += kCtlThreads) {
    const int i = i0 + t;
    const int v = i < hi ? in[i] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();  // the last tile's part is read
    if (lane == 31) part[w] = x;
    __syncthreads();
    int before = 0, tile = 0;
    for (int j = 0; j < kCtlThreads / 32; ++j) {
      if (j < w) before += part[j];
      tile += part[j];
    }
    if (i < hi) out[i] = base + before + x - v;
    base += tile;
  }
  cl.sync();
}

// first: the run's BD steps, at its start (else 0).  close: a BD step lies
// before.  more: another one follows.  A step whose rebuild overflowed its list
// did nothing past the rebuild and stays counted as remaining; after it, and
// after a step that recorded an error, the rest of the run does nothing.
template <int ND>
__global__ void __cluster_dims__(kCtlBlocks, 1, 1) __launch_bounds__(kCtlThreads)
    k_step_control(SysConst k, DevState d, RebuildBufs rb, int prec, int stoch, int first,
                   int close, int more, HostReport out) {
  namespace cg = cooperative_groups;
  __shared__ int2 sbuf[kCtlThreads][kHeadBuf];
  __shared__ int part[kCtlThreads / 32], tot[kCtlBlocks];
  __shared__ int go;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), t = threadIdx.x;
  cl.sync();  // every block has started: its shared memory may be written
  double limit = 0.0;  // (older than the kernel before)
  if (rank == 0 && t < d.nrep) limit = d.rep[t].dr_update;
  grid_dep_sync();
  if (rank == 0) {
    // The bookkeeping's operands and the first systems' maxima load together.
    const unsigned status = *d.status;  // the same word for every thread
    const unsigned long long mcount = *d.mcount;
    const int left = *d.loop_count;
    const bool halted = close && (status & ST_HALT), error = close && status != 0u;
    bool mine = false;
    unsigned bad = 0u;
    for (int r = t; r < d.nrep; r += kCtlThreads) {
      const double dr = __longlong_as_double((long long)d.dr_max_bits[r]);
      if (r != t) limit = d.rep[r].dr_update;
      int due = 0;
      if (dr > 10000.0 || !(dr == dr)) bad = ST_UNPHYSICAL;
      else due = dr > limit ? 1 : 0;
      if (!halted) d.due[r] = due;
      mine = mine || due;
    }
    const int any = __syncthreads_or(mine);  // and every thread has read the status
    if (t < kCtlBlocks) *cl.map_shared_rank(&go, t) = more && !halted && !error && any;
    if (bad && !halted) atomicOr(d.status, bad);
    if (t == 0) {
      if (first) {
        *d.loop_count = first;
        out.rebuilds[0] = *d.n_rebuilds;
      }
      if (close && !halted) {
        if (stoch) *d.mcount = mcount + 1ull;
        *d.loop_count = error ? 0 : left - 1;
        if (error && more) atomicOr(d.status, ST_STOP);
      }
      if (!more) atomicAnd(d.status, ~ST_STOP);
    }
  }
  cl.sync();
  if (!go) return;  // the same in every block
  const int step = kCtlBlocks * kCtlThreads, t0 = rank * kCtlThreads;
  rb_systems(d, rb, t0 + t, step);
  for (int i = t0; i < d.nb; i += step) rb_key<ND>(k, d, rb, i + t);
  cl.sync();
  cluster_scan(rb.gcount, rb.gstart, rb.n_groups, tot, part);
  for (int i = t0; i < d.nb; i += step) rb_scatter(d, rb, i + t);
  cl.sync();
  for (int i = t0; i < d.nb; i += step) rb_rank(d, rb, i + t);
  cl.sync();
  for (int i = t0; i < d.nb; i += step) {
    rb_count<kCtlThreads>(k, d, rb, i + t, sbuf, part);
    __syncthreads();  // (part is used again)
  }
  cl.sync();
  cluster_scan(rb.pair_count, rb.pair_off, 2 * d.nb, tot, part);
  const int cand = max(min(*rb.cand_n, rb.cand_cap), d.nrep);
  for (int i = t0; i < cand; i += step) rb_place(d, rb, prec, i + t);
  cl.sync();
  for (int i = t0; i < d.nb; i += step) rb_csr_sort(d, rb, i + t);
}

int launch_step_control(const SysConst &k, const DevState &d, const RebuildBufs &rb, int prec,
                        int stoch, int first, int close, int more, const HostReport &out,
                        cudaStream_t st) {
  if (k.n_dim == 3)
    launch_pdl(k_step_control<3>, dim3(kCtlBlocks), dim3(kCtlThreads), 0, st, k, d, rb, prec, stoch,
               first, close, more, out);
  else
    launch_pdl(k_step_control<2>, dim3(kCtlBlocks), dim3(kCtlThreads), 0, st, k, d, rb, prec, stoch,
               first, close, more, out);
  return 1;
}

int launch_rebuild(const SysConst &k, const DevState &d, const RebuildBufs &rb, int prec,
                   cudaStream_t st, bool first_in_graph) {
  int launched = 0;
  const int nb = d.nb > 0 ? d.nb : 1;
  const int g256 = (nb + 255) / 256;
  if (first_in_graph) {
    // Captured, the first kernel starts the conditional body: no kernel
    // before it to overlap.
    PdlOff off;
    if (k.n_dim == 3) launch_pdl(k_rb_keys<3>, dim3(g256), dim3(256), 0, st, k, d, rb);
    else launch_pdl(k_rb_keys<2>, dim3(g256), dim3(256), 0, st, k, d, rb);
  } else {
    if (k.n_dim == 3) launch_pdl(k_rb_keys<3>, dim3(g256), dim3(256), 0, st, k, d, rb);
    else launch_pdl(k_rb_keys<2>, dim3(g256), dim3(256), 0, st, k, d, rb);
  }
  ++launched;
  launched += launch_exclusive_scan(rb.gcount, rb.gstart, rb.n_groups, rb.scan_tmp, st);
  launch_pdl(k_rb_scatter, dim3(g256), dim3(256), 0, st, d, rb);
  launch_pdl(k_rb_rank, dim3(g256), dim3(256), 0, st, d, rb);
  const int gc = (nb + kCountBlock - 1) / kCountBlock;
  launch_pdl(k_rb_count, dim3(gc), dim3(kCountBlock), 0, st, k, d, rb);
  // pair_count and deg are one array of 2 nb (pair_off and deg_off alike).
  launched += 3 + launch_exclusive_scan(rb.pair_count, rb.pair_off, 2LL * d.nb, rb.scan_tmp, st);
  const int cap = rb.cand_cap > d.nrep ? rb.cand_cap : d.nrep;
  launch_pdl(k_rb_place, dim3((cap + 255) / 256), dim3(256), 0, st, d, rb, prec);
  launch_pdl(k_rb_csr_sort, dim3(g256), dim3(256), 0, st, d, rb);
  return launched + 2;
}

}  // namespace sc
