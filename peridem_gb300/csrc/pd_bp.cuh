// pd_bp.cuh -- per-node bodies of the contact broad phase (pd_broadphase.cu): the rebuild
// decision, the cell count, the scatter into the cell list and the candidate search. The
// per-phase kernels of pd_broadphase.cu and the persistent step of pd_fp32c.cu call the same
// code, so both build the same lists.
#ifndef PD_BP_CUH
#define PD_BP_CUH

#include <cuda_runtime.h>
#include <math.h>

#include "pd_device.cuh"
#include "pd_engine.h"
#include "pd_math.cuh"

namespace pdg {

constexpr uint32_t kNoKey = 0xFFFFFFFFu;  // node not in the cell list

// Node n's record in the cell list, from its current position (a cell is wider than the candidate
// radius, so two nodes within it lie in the same or adjacent cells; CandWalk computes the cell the
// same way).
__device__ __forceinline__ CellRec node_cell(const DevView &v, uint64_t n, uint32_t sim) {
  const double inv = v.sp[sim].inv_cell;
  CellRec r;
  r.cx = cell_coord(v.pos[n] + v.disp[n], inv, r.fx);
  r.cy = cell_coord(v.pos[n + v.Ncap] + v.disp[n + v.Ncap], inv, r.fy);
  r.cz = cell_coord(v.pos[n + 2 * v.Ncap] + v.disp[n + 2 * v.Ncap], inv, r.fz);
  r.node = (uint32_t)n;
  r.sim = sim;
  return r;
}

// Whether this step rebuilds (one thread): the accumulated movement bound against half the
// skin; the per-step counters restart.
__device__ __forceinline__ uint32_t bp_decide(const DevView &v, double half_skin) {
  DevCounters &c = *v.cnt;
  const double stepmax = __longlong_as_double((long long)c.stepmax_bits);
  c.rebuild = (c.moved + stepmax > half_skin) ? 1u : 0u;
  c.contacts = 0;
  c.live_bonds = 0;
  return c.rebuild;
}

// Node n's cell bucket and its slot in it (count must be zeroed); its candidate list restarts
// empty (the search writes the lists that are not).
__device__ __forceinline__ void bp_count_node(const DevView &v, uint64_t n, uint32_t *count, uint32_t *key,
                                              uint32_t *slot, uint32_t mask, uint16_t *cand_n) {
  cand_n[n] = 0;
  const uint32_t sim = v.S == 1 ? 0u : v.parts[v.pid[n]].sim;
  if (!v.ss[sim].active) {  // finished simulations leave the cell list
    key[n] = kNoKey;
    return;
  }
  const CellRec r = node_cell(v, n, sim);
  const uint32_t kk = (cell_row(r.cy, r.cz, sim) + r.cx) & mask;
  key[n] = kk;
  slot[n] = atomicAdd(&count[kk], 1u);
}

__device__ __forceinline__ void bp_scatter_node(const DevView &v, uint64_t n, const uint32_t *start,
                                                const uint32_t *key, const uint32_t *slot, CellRec *rec) {
  if (key[n] == kNoKey) return;
  rec[start[key[n]] + slot[n]] = node_cell(v, n, v.S == 1 ? 0u : v.parts[v.pid[n]].sim);
}

// The records of one row's three buckets around cell me.cx: entries b .. b + len - 1 of the cell
// list, taken modulo its nact records (start[0] is 0, so a range that runs past the table's last
// bucket goes on at record 0).
__device__ __forceinline__ void row_range(const CellRec &me, int row, const uint32_t *start, uint32_t mask,
                                          uint32_t nact, uint32_t &b, uint32_t &len) {
  const int dy = row % 3 - 1, dz = row / 3 - 1;
  const uint32_t k = (cell_row(me.cy + dy, me.cz + dz, me.sim) + me.cx - 1u) & mask;
  b = start[k];
  len = (k + 3 <= mask + 1 ? start[k + 3] : nact + start[k + 2 - mask]) - b;
}

// Whether record q of that row holds a candidate of me: a node of the simulation in one of the
// row's three cells (buckets are shared by hash) within the candidate radius. Distances are taken
// in cell edges from the positions inside the cells: their rounding, a few 2^-24, is far below the
// 1e-5 the test is widened by, so a list holds every node within the candidate radius; the
// consumers' exact FP64 tests decide.
__device__ __forceinline__ bool row_hit(const CellRec &me, int row, const CellRec &q) {
  const uint32_t dy = row % 3 - 1, dz = row / 3 - 1;
  const int dx = (int)(q.cx - me.cx);
  if (q.node == me.node || dx < -1 || dx > 1 || q.cy != me.cy + dy || q.cz != me.cz + dz || q.sim != me.sim)
    return false;
  const float x = (float)dx + (q.fx - me.fx), y = (float)(int)dy + (q.fy - me.fy), z = (float)(int)dz + (q.fz - me.fz);
  return x * x + y * y + z * z <= 1.0f + 1e-5f;
}

// Candidate list of the node of record t: the nodes of its simulation within the candidate radius,
// ascending in file order, by one thread. Records are taken in the cell list's order, so the
// threads of a warp walk neighbouring cells of a row and share the sectors of the buckets and
// records they read. The list is kept sorted as it grows (few nodes have candidates, and few).
// Bound by the latency of the bucket loads. A whole rebuild with 27 separately hashed cells per
// node and FP64 positions gathered per entry took 8.0 ms on crush512_4m (3.98 M nodes) and 0.62 ms
// on a 363k-node plate; with rows of cells and 32-byte records 1.9 and 0.15 ms.
__device__ __forceinline__ void bp_candidates_node(const DevView &v, uint64_t t, const uint32_t *start,
                                                   const CellRec *rec, uint32_t mask, uint32_t *cand, uint16_t *cand_n,
                                                   uint32_t cap) {
  const uint32_t nact = start[(uint64_t)mask + 1];
  if (t >= nact) return;
  const CellRec me = rec[t];
  uint32_t b[9], len[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) row_range(me, r, start, mask, nact, b[r], len[r]);
  uint32_t *out = cand + (uint64_t)me.node * cap;
  uint32_t cnt = 0;
#pragma unroll
  for (int r = 0; r < 9; ++r)
    for (uint32_t i = 0; i < len[r]; ++i) {
      const uint32_t at = b[r] + i;
      const CellRec q = rec[at < nact ? at : at - nact];
      if (!row_hit(me, r, q)) continue;
      if (cnt < cap) {  // insert by file index
        const uint32_t fq = v.file_of[q.node];
        uint32_t pos = cnt;
        while (pos > 0 && v.file_of[out[pos - 1]] > fq) {
          out[pos] = out[pos - 1];
          --pos;
        }
        out[pos] = q.node;
      }
      ++cnt;
    }
  if (!cnt) return;
  if (cnt > cap) {
    // more partners than the list holds: the consumers walk the cell list for this node instead
    // (CandWalk), which gives the same partners in the same order; the host grows the lists
    cand_n[me.node] = kCandCells;
    atomicAdd(&v.cnt->cand_cells, 1u);
  } else {
    cand_n[me.node] = (uint16_t)cnt;
  }
  if (v.xnodes) v.xnodes[atomicAdd(&v.xcount[0], 1u)] = me.node;  // work list of the contact kernels
}

// Words of shared memory bp_candidates_quad takes per warp: four gather buffers of kMaxCandCap
// entries plus a count.
constexpr uint32_t kCandQuadWords = 4 * (kMaxCandCap + 1);

// The same lists built for four records per warp (t0 .. t0 + 3): lane g of a record's eight takes
// row g of its nine, lane 0 the ninth as well (a row holds one or two records; loading several
// ahead took registers from the persistent step's bond loop, cubes125 38.5 -> 39.8 us per step).
// The candidates' file indices are gathered in the record's shared buffer and ranked into ascending
// order. A small handle's search is a chain of dependent loads per node (its record, the buckets,
// their records); nine short chains side by side instead of one long one. All 32 lanes of the warp
// call it with the same t0; sh holds kCandQuadWords words.
__device__ __forceinline__ void bp_candidates_quad(const DevView &v, uint64_t t0, uint32_t lane, const uint32_t *start,
                                                   const CellRec *rec, uint32_t mask, uint32_t *cand, uint16_t *cand_n,
                                                   uint32_t cap, uint32_t *sh) {
  const uint32_t q = lane >> 3, g = lane & 7u;
  const uint32_t nact = start[(uint64_t)mask + 1];
  const uint64_t t = t0 + q;
  const bool run = t < nact;
  uint32_t *buf = sh + (kMaxCandCap + 1) * q;  // the record's candidates (file indices), their count last
  if (g == 0) buf[kMaxCandCap] = 0;
  const CellRec me = rec[run ? t : 0];
  __syncwarp();
  if (run) {
    uint32_t b0, len0, b1 = 0, len1 = 0;
    row_range(me, (int)g, start, mask, nact, b0, len0);
    if (g == 0) row_range(me, 8, start, mask, nact, b1, len1);
    for (uint32_t j = 0; j < len0 + len1; ++j) {
      const bool first = j < len0;
      const uint32_t at = first ? b0 + j : b1 + (j - len0);
      const CellRec c = rec[at < nact ? at : at - nact];
      if (!row_hit(me, first ? (int)g : 8, c)) continue;
      const uint32_t slot = atomicAdd(&buf[kMaxCandCap], 1u);
      if (slot < cap) buf[slot] = v.file_of[c.node];
    }
  }
  __syncwarp();
  const uint32_t total = run ? buf[kMaxCandCap] : 0u;
  if (total) {
    if (total > cap) {  // as bp_candidates_node
      if (g == 0) {
        cand_n[me.node] = kCandCells;
        atomicAdd(&v.cnt->cand_cells, 1u);
      }
    } else {
      uint32_t *out = cand + (uint64_t)me.node * cap;
      for (uint32_t i = g; i < total; i += 8) {
        const uint32_t fi = buf[i];
        uint32_t rk = 0;
        for (uint32_t j = 0; j < total; ++j) rk += buf[j] < fi;
        out[rk] = v.node_of[fi];
      }
      if (g == 0) cand_n[me.node] = (uint16_t)total;
    }
    if (g == 0 && v.xnodes) v.xnodes[atomicAdd(&v.xcount[0], 1u)] = me.node;
  }
  __syncwarp();
}

}  // namespace pdg
#endif
