// Narrow supersteps: a CTA relaxes its share of a small frontier, and what
// that reaches below the bucket's end, on its own until nothing is left,
// instead of one grid barrier per hop.
//
// A traversal of a grid, a mesh or a road-like graph runs thousands of
// supersteps whose frontiers hold a few vertices per CTA.  Each of those
// costs a chain of dependent round trips (barrier, counts, queue entry, row,
// column, label, claim, append): 5.9 us a level for BFS and 10.6 us a
// superstep for SSSP on the 4096 x 4096 grid, whatever little it relaxes.
// Here the frontier stays in the CTA's shared memory as arc slots {arc,
// vertex, label}, one thread per slot, and a hop is two round trips (columns
// and weights; then label atomics with the targets' rows beside them) and
// one CTA barrier.
//
// Any order of relaxations reaches the same least labels: every strict
// improvement of a label makes slots (or a queue or pile mark) for its
// vertex, a slot whose label is no longer its vertex's is dropped (the later
// improvement has its own), and the grid barrier that ends the superstep
// comes when every CTA has run dry.  A CTA hands its vertices to the next
// superstep's frontier, for all CTAs to share, when a hop has more arcs
// than slots or after kDrainSteps hops (a barrier wait is bounded in time).
// Heavy vertices always go there: their arcs are walked in chunks by many
// warps.
//
// 4096 x 4096 grid, U[1,1000] weights, from the corner: SSSP 106.8 -> 21.2 ms
// (10,000 hops of 2.0 us; 1.4 us where the graph stays in L2), BFS 48.3 ->
// 12.2.  One warp group per 32 entries with an owner search per arc, instead
// of a slot per arc, took 27.7 ms: the search and the lanes' votes were 0.6 us
// of the hop's chain.  Prefetching the next lines of columns and rows into L2
// gained 2.5 % there and lost 1 % on small grids: left out.
#pragma once

#include "gdb_sweep.cuh"

namespace gdb {

constexpr uint32_t kDrainSteps = 128;

template <uint32_t Cap, uint32_t List>
struct DrainMem {
  static constexpr uint32_t kCap = Cap;   // arc slots per buffer
  static constexpr uint32_t kList = List;
  // pile entries per CTA up to which a phase change is narrow (Cap / 4, / 2 and
  // Cap itself are the same on grids of 4,096 to 16.8 M vertices and in mixed
  // batches, within 0.4 %)
  static constexpr uint32_t kPile = Cap / 2;
  uint32_t arc[2][Cap], v[2][Cap], d[2][Cap];
  uint32_t far[List];    // reached at or beyond the bucket's end
  uint32_t spill[List];  // handed to the next superstep's frontier
  uint32_t n[3];         // slots, by hop % 3
  uint32_t nfar, nspill;
};

// Vertices of a frontier per CTA up to which its superstep is narrow: those
// whose arcs fill three quarters of the slots.
__host__ __device__ inline uint32_t drain_share(uint64_t E, uint32_t V, uint32_t slots) {
  const uint32_t deg = (uint32_t)(E / (V ? V : 1u)) + 1u;
  const uint32_t s = slots / 4u * 3u / deg;
  return s < 4u ? 4u : s;
}

// Slots for the arcs [b, b + deg) of vertex v at label d; false when they do
// not fit (any slots reserved then hold no vertex).
template <class Mem>
__device__ __forceinline__ bool drain_add(Mem& m, uint32_t slot, uint32_t buf, uint32_t v, uint32_t d, uint32_t b,
                                          uint32_t deg) {
  const uint32_t at = atomicAdd(&m.n[slot], deg);
  const bool fits = at + deg <= Mem::kCap;
  for (uint32_t i = 0; i < deg && at + i < Mem::kCap; ++i) {
    m.arc[buf][at + i] = b + i;
    m.v[buf][at + i] = fits ? v : 0xFFFFFFFFu;
    m.d[buf][at + i] = d;
  }
  return fits;
}

template <class Mem>
__device__ __forceinline__ void drain_reset(Mem& m) {
  __syncthreads();
  if (threadIdx.x < 3) m.n[threadIdx.x] = 0;
  if (threadIdx.x == 0) m.nfar = m.nspill = 0;
  __syncthreads();
}

// Items [0, n) of a list go to the CTAs in turn: item k of this CTA, and the
// most a CTA gets.  One by one: what follows in a queue or pile was reached
// together, and runs of 64 to one CTA left others dry (4096^2 grid, SSSP at
// width 16,016: 28.8 ms one by one, 29.1 / 30.5 / 34.2 in runs of 4 / 16 / 64).
__device__ __forceinline__ uint32_t drain_item(uint32_t k, int id, int P) { return k * (uint32_t)P + (uint32_t)id; }
__device__ __forceinline__ uint32_t drain_items(uint32_t n, int P) { return (n + (uint32_t)P - 1) / (uint32_t)P; }

// Take this CTA's share of a light queue as hop 0 (label(v): the vertex's
// label); what does not fit goes to spill(want, v).
template <class Mem, class Label, class Spill>
__device__ __forceinline__ void drain_take(const GraphView& G, Mem& m, const uint32_t* q, uint32_t n, int id,
                                           int P, Label&& label, Spill&& spill) {
  const uint32_t have = drain_items(n, P);
  for (uint32_t base = threadIdx.x & ~31u; base < have; base += blockDim.x) {
    const uint32_t i = drain_item(base + lane_id(), id, P);
    uint32_t v = 0;
    bool over = false;
    if (base + lane_id() < have && i < n) {
      v = ld_cg(&q[i]);
      const uint32_t d = label(v), b = __ldg(&G.row[v]), deg = __ldg(&G.row[v + 1]) - b;
      over = !drain_add(m, 0, 0, v, d, b, deg);
    }
    if (__any_sync(kFull, over)) spill(over, v);
  }
}

// Relax hop 0's slots and everything they reach below `split`, hop by hop.
//   weight(arc): the arc's weight (kInf: no arc)
//   label(v), relax(v, d): the label now; lower it to d, returning what it was
//   far(want, v), spill(want, v): take the lanes' vertices when their list
//   is full or at the end (every lane of a warp calls them)
// On return the lists have been handed over; every CTA of the grid calls it
// in the same superstep.  Returns the hops made.
template <class Mem, class Weight, class Label, class Relax, class Far, class Spill>
__device__ __forceinline__ uint32_t drain_run(const GraphView& G, Mem& m, uint32_t split, uint32_t& fmin,
                                              unsigned long long& arcs, Weight&& weight, Label&& label,
                                              Relax&& relax, Far&& far, Spill&& spill) {
  const int lane = lane_id();
  uint32_t hop = 0;
  for (;; ++hop) {
    const uint32_t cur = hop % 3, nxt = (hop + 1) % 3, buf = hop & 1;
    __syncthreads();  // the hop's slots are in place
    const uint32_t all = m.n[cur], n = min(all, Mem::kCap);
    if (n == 0) break;
    // read by every thread at hop - 1, before the barrier just passed
    if (threadIdx.x == 0) m.n[(hop + 2) % 3] = 0;
    if ((hop > 0 && all > Mem::kCap) || hop == kDrainSteps) {
      for (uint32_t base = threadIdx.x & ~31u; base < n; base += blockDim.x) {
        const uint32_t v = base + lane < n ? m.v[buf][base + lane] : 0xFFFFFFFFu;
        spill(v != 0xFFFFFFFFu, v);
      }
      break;
    }
    for (uint32_t base = threadIdx.x & ~31u; base < n; base += 2 * blockDim.x) {
      // two slots per thread, their round trips together
      uint32_t u[2], v[2], nd[2], r0[2], r1[2], old[2];
      bool in[2], heavy[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t i = base + lane + j * blockDim.x;
        u[j] = i < n ? m.v[buf][i] : 0xFFFFFFFFu;
        v[j] = 0;
        nd[j] = kInf;
        in[j] = u[j] != 0xFFFFFFFFu;
        if (in[j]) {
          const uint32_t arc = m.arc[buf][i];
          v[j] = __ldg(&G.col[arc]);
          nd[j] = weight(arc);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t d = in[j] ? m.d[buf][base + lane + j * blockDim.x] : 0u;
        in[j] = in[j] && nd[j] < kInf && label(u[j]) == d;
        nd[j] += d;
        arcs += in[j];
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        old[j] = in[j] ? relax(v[j], nd[j]) : 0u;
        r0[j] = in[j] ? __ldg(&G.row[v[j]]) : 0u;
        r1[j] = in[j] ? __ldg(&G.row[v[j] + 1]) : 0u;
        heavy[j] = G.nheavy && in[j] && is_heavy(G, v[j]);
      }
      // one shared-memory counter add per vertex reached, with no vote
      // among the lanes (aggregated per warp, the adds cost 0.3 us on the
      // hop's chain)
      uint32_t lost = 0;  // bit j: slot j's vertex goes to spill, bit 2 + j: to far
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (in[j] && nd[j] < old[j]) {
          if (nd[j] >= split) {
            fmin = min(fmin, nd[j]);
            const uint32_t at = atomicAdd(&m.nfar, 1u);
            if (at < Mem::kList) m.far[at] = v[j];
            else lost |= 4u << j;
          } else if (heavy[j] || !drain_add(m, nxt, buf ^ 1, v[j], nd[j], r0[j], r1[j] - r0[j])) {
            const uint32_t at = atomicAdd(&m.nspill, 1u);
            if (at < Mem::kList) m.spill[at] = v[j];
            else lost |= 1u << j;
          }
        }
      }
      if (__any_sync(kFull, lost)) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          spill((lost >> j) & 1u, v[j]);
          far((lost >> (2 + j)) & 1u, v[j]);
        }
      }
    }
  }
  __syncthreads();
  const uint32_t nf = min(m.nfar, Mem::kList), ns = min(m.nspill, Mem::kList);
  for (uint32_t base = threadIdx.x & ~31u; base < nf; base += blockDim.x) {
    const bool act = base + lane < nf;
    far(act, act ? m.far[base + lane] : 0u);
  }
  for (uint32_t base = threadIdx.x & ~31u; base < ns; base += blockDim.x) {
    const bool act = base + lane < ns;
    spill(act, act ? m.spill[base + lane] : 0u);
  }
  return hop;
}

}  // namespace gdb
