// pd_pairs.cu -- bond lists on the GPU: for every particle, all node pairs (i, j), i < j, with
// |x_i - x_j| <= r, sorted by (i, j). This is the pair list the reference's setup scripts take
// from scipy's cKDTree.query_pairs(delta) and sort (exp_dict.py:542-567). The distance test is
// ((dx*dx + dy*dy) + dz*dz <= r*r in FP64, compiled without contraction), which is how x86
// builds of scipy evaluate it: the lists equal the sorted query_pairs output there. (aarch64
// builds of scipy contract the expression into fused multiply-adds, which can move pairs that
// lie within an ulp of r.)
//
// Method: per particle, a grid of cells slightly larger than r anchored at the particle's lower
// corner, hashed so that the cells of a row along x are consecutive buckets (nine ranges hold a node's
// 27 cells), built by a counting sort into 32-byte records with the position inside the cell in
// FP32. One thread per record scans the nine ranges -- records in cell order, so the threads of a
// warp read the same ranges -- and decides a pair in FP32 unless its distance lies within 4e-6 of r,
// then in FP64 from the positions as stated above: the FP32 distance is off by less than 1.2e-6 of r
// (in-cell positions rounded to 2^-25 of a cell, the sums to a few 2^-24). Pass 1 counts the partners
// j > i, pass 2 writes them after a device scan of the counts, pass 3 sorts each row, one warp per row.
// 182k nodes, 8.7e6 pairs: pass 1 10.2 ms with each candidate's cell from FP64 divisions and 27
// separate buckets, 0.24 ms now; the whole call 30 -> 1.6 ms (into memory already touched).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "peridem_gb300.h"

namespace {

constexpr int kThreads = 256;
constexpr unsigned kGrid = 152 * 8;  // blocks of the grid-stride kernels
constexpr int kScanThreads = 1024;
constexpr int kScanBlock = 4 * kScanThreads;  // entries per block of the scans

// A node in the cell list: position inside its cell (in cell edges), node, cell (modulo 2^32), particle.
struct __align__(32) Rec {
  float fx, fy, fz;
  uint32_t node;
  uint32_t cx, cy, cz, p;
};

struct PairsArgs {
  const double *pos;        // [N][3]
  uint32_t *pid;            // particle of each node
  const uint64_t *off;      // [P+1] first node of each particle
  const double *r;          // radius of each particle
  unsigned long long *lo, *hi;  // [P][3] ordered keys of each particle's box
  uint64_t N, T;
  uint32_t P, mask;         // hash table size T - 1
  uint32_t *count, *start, *key, *slot;  // start: [T + 1]
  Rec *rec;
  uint32_t *deg;            // partners j > i per node (pass 1)
  uint64_t *first;          // [N + 1] their exclusive scan
  uint64_t *sums;           // scan scratch
  uint32_t *bad;            // set by a non-finite position
  uint32_t *out;            // [M][2] local (i, j)
};

__device__ __forceinline__ unsigned long long key_of(double x) {  // orders as x does
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double val_of(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

__device__ __forceinline__ uint32_t row_hash(uint32_t p, uint32_t cy, uint32_t cz) {
  uint32_t h = cy * 0x9E3779B1u + cz * 0x85EBCA77u + p * 0xC2B2AE3Du;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  return h ^ (h >> 15);
}

// Particle of each node and the particles' boxes.
__global__ void k_boxes(PairsArgs a) {
  for (uint64_t n0 = (uint64_t)blockIdx.x * blockDim.x; n0 < a.N; n0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t n = n0 + threadIdx.x;
    const bool valid = n < a.N;
    uint32_t p = 0xFFFFFFFFu;
    unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
    if (valid) {
      uint32_t b = 0, e = a.P;  // the last p with off[p] <= n (particles may be empty)
      while (e - b > 1) {
        const uint32_t m = b + (e - b) / 2;
        if (a.off[m] <= n) b = m;
        else e = m;
      }
      p = b;
      a.pid[n] = p;
      bool fine = true;
      for (int c = 0; c < 3; ++c) {
        const double x = a.pos[3 * n + c];
        fine = fine && isfinite(x);
        lo[c] = hi[c] = key_of(x);
      }
      if (!fine) *a.bad = 1;
    }
    const uint32_t p0 = __shfl_sync(0xffffffffu, p, 0);
    if (__all_sync(0xffffffffu, !valid || p == p0)) {
      for (int o = 16; o > 0; o >>= 1)
        for (int c = 0; c < 3; ++c) {
          lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
          hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
      if ((threadIdx.x & 31) != 0 || p0 == 0xFFFFFFFFu) continue;
    } else if (!valid) {
      continue;
    }
    for (int c = 0; c < 3; ++c) {
      atomicMin(&a.lo[3 * (uint64_t)p + c], lo[c]);
      atomicMax(&a.hi[3 * (uint64_t)p + c], hi[c]);
    }
  }
}

// Cells a little larger than r, so that every pair within r lies in the same or adjacent cells.
__device__ __forceinline__ double cell_edge(double r) { return r * (1.0 + 1e-6); }

__device__ __forceinline__ Rec record(const PairsArgs &a, uint64_t n) {
  Rec q;
  q.p = a.pid[n];
  const double c = cell_edge(a.r[q.p]);
  float f[3];
  uint32_t k[3];
  for (int d = 0; d < 3; ++d) {
    const double s = (a.pos[3 * n + d] - val_of(a.lo[3 * (uint64_t)q.p + d])) / c, fl = floor(s);
    f[d] = (float)(s - fl);
    k[d] = (uint32_t)(long long)fl;
  }
  q.fx = f[0];
  q.fy = f[1];
  q.fz = f[2];
  q.node = (uint32_t)n;
  q.cx = k[0];
  q.cy = k[1];
  q.cz = k[2];
  return q;
}

__global__ void k_count(PairsArgs a) {
  for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < a.N; n += (uint64_t)gridDim.x * blockDim.x) {
    const Rec q = record(a, n);
    const uint32_t k = (row_hash(q.p, q.cy, q.cz) + q.cx) & a.mask;
    a.key[n] = k;
    a.slot[n] = atomicAdd(&a.count[k], 1u);
  }
}

__global__ void k_scatter(PairsArgs a) {
  for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < a.N; n += (uint64_t)gridDim.x * blockDim.x)
    a.rec[a.start[a.key[n]] + a.slot[n]] = record(a, n);
}

// Sum over the block's threads before this one; *total receives the block's sum.
__device__ __forceinline__ uint64_t block_excl(uint64_t x, uint64_t *total) {
  __shared__ uint64_t sh[kScanThreads / 32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t s = x;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= (uint32_t)o) s += y;
  }
  if (lane == 31) sh[w] = s;
  __syncthreads();
  if (w == 0) {
    uint64_t t = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= (uint32_t)o) t += y;
    }
    sh[lane] = t;
  }
  __syncthreads();
  *total = sh[kScanThreads / 32 - 1];
  return s - x + (w ? sh[w - 1] : 0);
}

// Exclusive scan of in[n] into out[n + 1] (out[n] the total): block totals, then every block scans its
// entries from the totals of the blocks before it.
__global__ void __launch_bounds__(kScanThreads) k_sum_blocks(const uint32_t *in, uint64_t *sums, uint64_t n) {
  uint64_t s = 0, total;
  for (int i = 0; i < 4; ++i) {
    const uint64_t k = (uint64_t)blockIdx.x * kScanBlock + 4ull * threadIdx.x + i;
    s += k < n ? in[k] : 0u;
  }
  block_excl(s, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
template <typename O>
__global__ void __launch_bounds__(kScanThreads) k_scan(const uint32_t *in, const uint64_t *sums, O *out, uint64_t n) {
  uint64_t before = 0, off, total, x[4], s = 0;
  for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kScanThreads) before += sums[i];
  block_excl(before, &off);
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kScanBlock + 4ull * threadIdx.x;
  for (int i = 0; i < 4; ++i) {
    x[i] = base + i < n ? in[base + i] : 0u;
    s += x[i];
  }
  uint64_t run = off + block_excl(s, &total);
  for (int i = 0; i < 4; ++i) {
    if (base + i < n) out[base + i] = (O)run;
    run += x[i];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = (O)(off + total);
}

// Calls f(record) for every other node of me's particle within its radius (in one of the nine
// ranges: its cell and adjacent ones), until f returns true. SQRT: the distance is compared as
// sqrt(d2) <= r instead of d2 <= r * r. Returns whether f did.
template <bool SQRT, class F>
__device__ __forceinline__ bool visit(const PairsArgs &a, const Rec &me, F &&f) {
  const double r = a.r[me.p], r2 = r * r, c = cell_edge(r);
  const float rc2 = (float)((r / c) * (r / c));
  float in2 = rc2 * (1.0f - 8e-6f), out2 = rc2 * (1.0f + 8e-6f);  // squared: within 4e-6 of r
  // FP64 decides everything where a box has more cells than FP32 in-cell positions are good for, or
  // where r * r is near the ends of the FP64 range (a box wider than that range has NaN in-cell
  // positions: the comparisons below let a NaN pass to FP64)
  bool wide = !(r2 > 1e-280 && r2 < 1e280);
  for (int d = 0; d < 3; ++d)
    wide = wide || !(val_of(a.hi[3 * (uint64_t)me.p + d]) - val_of(a.lo[3 * (uint64_t)me.p + d]) < 1e6 * c);
  if (wide) {
    in2 = -1.0f;
    out2 = INFINITY;
  }
  const uint32_t total = (uint32_t)a.N;
  for (int row = 0; row < 9; ++row) {
    const int dy = row % 3 - 1, dz = row / 3 - 1;
    const uint32_t cy = me.cy + dy, cz = me.cz + dz;
    const uint32_t k = (row_hash(me.p, cy, cz) + me.cx - 1u) & a.mask;
    // three buckets; a range past the table's end goes on at record 0 (start[0] is 0)
    const uint32_t b = a.start[k];
    const uint32_t e = k + 3 <= a.mask + 1 ? a.start[k + 3] : total + a.start[k + 2 - a.mask];
    const float by = (float)dy - me.fy, bz = (float)dz - me.fz;
    for (uint32_t i = b; i < e; ++i) {
      const Rec q = a.rec[i < total ? i : i - total];
      const int dx = (int)(q.cx - me.cx);
      if (q.cy != cy || q.cz != cz || q.p != me.p || dx < -1 || dx > 1 || q.node == me.node) continue;
      const float x = (float)dx + (q.fx - me.fx), y = q.fy + by, z = q.fz + bz;
      const float d2 = x * x + y * y + z * z;
      if (d2 > out2) continue;
      if (!(d2 < in2)) {  // too close to r for FP32
        const double *pi = a.pos + 3 * (uint64_t)me.node, *pj = a.pos + 3 * (uint64_t)q.node;
        const double ex = pj[0] - pi[0], ey = pj[1] - pi[1], ez = pj[2] - pi[2];
        const double s = (ex * ex + ey * ey) + ez * ez;
        if (!(SQRT ? sqrt(s) <= r : s <= r2)) continue;
      }
      if (f(q)) return true;
    }
  }
  return false;
}

// Every j > i of node i's particle within r; WRITE selects pass 1 (count) or 2 (write). A call with a
// non-finite position is refused and none of its nodes searched: the box of such a particle may have
// no finite corner, which puts all its nodes in one cell.
template <bool WRITE>
__global__ void k_pairs(PairsArgs a) {
  if (*a.bad) return;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.N; t += (uint64_t)gridDim.x * blockDim.x) {
    const Rec me = a.rec[t];
    const uint32_t base = (uint32_t)a.off[me.p];
    uint32_t c = 0;
    uint2 *row = WRITE ? reinterpret_cast<uint2 *>(a.out) + a.first[me.node] : nullptr;
    visit<false>(a, me, [&](const Rec &q) {
      if (q.node > me.node) {
        if (WRITE) row[c] = make_uint2(me.node - base, q.node - base);
        ++c;
      }
      return false;
    });
    if (!WRITE) a.deg[me.node] = c;
  }
}

// Flags every node q that lies within r of a marked node of its particle (itself included), with
// the reference's test: d = sqrt((dx*dx + dy*dy) + dz*dz), d <= r (gen_nonlocal_boundry_nodes,
// exp_dict.py:1231-1248, which scans every node for every edge node).
__global__ void k_near(PairsArgs a, const uint8_t *marked, uint8_t *near) {
  if (*a.bad) return;  // as k_pairs
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.N; t += (uint64_t)gridDim.x * blockDim.x) {
    const Rec me = a.rec[t];
    near[me.node] = marked[me.node] || visit<true>(a, me, [&](const Rec &q) { return marked[q.node] != 0; });
  }
}

// Sorts each node's row by j, one warp per row: a row of up to 128 partners is held in registers and
// each partner written at its rank (partners are distinct, so the ranks are a permutation); longer
// rows are left to k_sort_long.
__global__ void k_sort_rows(PairsArgs a) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t n = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; n < a.N; n += warps) {
    uint32_t *row = a.out + 2 * a.first[n];
    const uint64_t d = a.first[n + 1] - a.first[n];
    if (d > 128) continue;
    uint32_t x[4], rank[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = (lane + 32u * k < d) ? row[2 * (lane + 32 * k) + 1] : 0xFFFFFFFFu;
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      if (32u * k2 >= d) break;  // uniform across the warp
      for (uint32_t src = 0; src < 32; ++src) {
        const uint32_t y = __shfl_sync(0xffffffffu, x[k2], src);  // the largest value past the row's end
#pragma unroll
        for (int k = 0; k < 4; ++k) rank[k] += y < x[k] ? 1u : 0u;
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (lane + 32u * k < d) row[2 * rank[k] + 1] = x[k];
    __syncwarp();
  }
}
__global__ void k_sort_long(PairsArgs a) {
  for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < a.N; n += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = a.first[n], e = a.first[n + 1];
    if (e - b <= 128) continue;
    for (uint64_t x = b + 1; x < e; ++x) {
      const uint32_t v = a.out[2 * x + 1];
      uint64_t y = x;
      while (y > b && a.out[2 * (y - 1) + 1] > v) {
        a.out[2 * y + 1] = a.out[2 * (y - 1) + 1];
        --y;
      }
      a.out[2 * y + 1] = v;
    }
  }
}

// The pairs before each particle's first node.
__global__ void k_particle_pairs(PairsArgs a, uint64_t *pair_off) {
  const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p <= a.P) pair_off[p] = a.first[a.off[p]];
}

struct Dev {
  std::vector<void *> ptrs;
  cudaStream_t s = nullptr;
  ~Dev() {
    for (void *p : ptrs) cudaFreeAsync(p, s);
    if (s) {
      cudaStreamSynchronize(s);
      cudaStreamDestroy(s);
    }
  }
  template <typename T>
  cudaError_t alloc(T **p, size_t count) {
    void *q = nullptr;
    cudaError_t e = cudaMallocAsync(&q, (count ? count : 1) * sizeof(T), s);
    if (e == cudaSuccess) ptrs.push_back(q);
    *p = (T *)q;
    return e;
  }
};

thread_local std::string g_pairs_error;

int fail(int rc, const std::string &m) {
  g_pairs_error = m;
  return rc;
}

static int check_inputs(const double *pos, const uint64_t *node_offset, const double *radius, uint32_t n_particles) {
  if (!pos || !node_offset || !radius) return fail(PD_EINVAL, "null argument");
  if (node_offset[0] != 0) return fail(PD_EINVAL, "node_offset must start at 0");
  for (uint32_t p = 0; p < n_particles; ++p) {
    if (node_offset[p + 1] < node_offset[p]) return fail(PD_EINVAL, "node_offset not monotone");
    if (!(radius[p] > 0) || !std::isfinite(radius[p])) return fail(PD_EINVAL, "radius must be positive");
  }
  if (node_offset[n_particles] >= 0xFFFFFFF0ull) return fail(PD_EINVAL, "too many nodes");
  return PD_OK;
}

// The cell list of all nodes, on d's stream; a receives the device arrays. The device's verdict on the
// positions (a.bad) is read by the caller.
static int build_grid(const double *pos, const uint64_t *node_offset, const double *radius, uint32_t n_particles,
                      Dev &d, PairsArgs &a) {
  const uint64_t N = node_offset[n_particles];
  uint32_t bits = 10;
  while ((1ull << bits) < 2 * N) ++bits;
  if (bits > 31) return fail(PD_EINVAL, "too many nodes");
  const uint64_t T = 1ull << bits;
  if (cudaStreamCreateWithFlags(&d.s, cudaStreamNonBlocking) != cudaSuccess)
    return fail(PD_ECUDA, "stream create failed");
  a.N = N;
  a.T = T;
  a.P = n_particles;
  a.mask = (uint32_t)(T - 1);
  double *dpos, *dr;
  uint64_t *doff;
  cudaError_t e = cudaSuccess;
  auto ck = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  ck(d.alloc(&dpos, 3 * N));
  ck(d.alloc(&a.pid, N));
  ck(d.alloc(&doff, (size_t)n_particles + 1));
  ck(d.alloc(&dr, n_particles));
  ck(d.alloc(&a.lo, 3 * (size_t)n_particles));
  ck(d.alloc(&a.hi, 3 * (size_t)n_particles));
  ck(d.alloc(&a.count, T));
  ck(d.alloc(&a.start, T + 1));
  ck(d.alloc(&a.key, N));
  ck(d.alloc(&a.slot, N));
  ck(d.alloc(&a.rec, N));
  ck(d.alloc(&a.sums, (std::max(T, N) + kScanBlock - 1) / kScanBlock));
  ck(d.alloc(&a.bad, 1));
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? PD_ENOMEM : PD_ECUDA, cudaGetErrorString(e));
  ck(cudaMemcpyAsync(dpos, pos, 3 * N * 8, cudaMemcpyHostToDevice, d.s));
  ck(cudaMemcpyAsync(doff, node_offset, ((size_t)n_particles + 1) * 8, cudaMemcpyHostToDevice, d.s));
  ck(cudaMemcpyAsync(dr, radius, (size_t)n_particles * 8, cudaMemcpyHostToDevice, d.s));
  ck(cudaMemsetAsync(a.lo, 0xFF, 3 * (size_t)n_particles * 8, d.s));
  ck(cudaMemsetAsync(a.hi, 0, 3 * (size_t)n_particles * 8, d.s));
  ck(cudaMemsetAsync(a.count, 0, T * 4, d.s));
  ck(cudaMemsetAsync(a.bad, 0, 4, d.s));
  a.pos = dpos;
  a.off = doff;
  a.r = dr;
  a.out = nullptr;
  const unsigned nb = (unsigned)((T + kScanBlock - 1) / kScanBlock);
  k_boxes<<<kGrid, kThreads, 0, d.s>>>(a);
  k_count<<<kGrid, kThreads, 0, d.s>>>(a);
  k_sum_blocks<<<nb, kScanThreads, 0, d.s>>>(a.count, a.sums, T);
  k_scan<uint32_t><<<nb, kScanThreads, 0, d.s>>>(a.count, a.sums, a.start, T);
  k_scatter<<<kGrid, kThreads, 0, d.s>>>(a);
  ck(cudaGetLastError());
  if (e != cudaSuccess) return fail(PD_ECUDA, cudaGetErrorString(e));
  return PD_OK;
}

}  // namespace

extern "C" {

const char *pd_pairs_error(void) { return g_pairs_error.c_str(); }

int pd_query_pairs(const double *pos, const uint64_t *node_offset, const double *radius, uint32_t n_particles,
                   uint32_t *pairs, uint64_t cap, uint64_t *pair_offset) {
  if (!pair_offset) return fail(PD_EINVAL, "null argument");
  const int bad = check_inputs(pos, node_offset, radius, n_particles);
  if (bad != PD_OK) return bad;
  const uint64_t N = node_offset[n_particles];
  pair_offset[0] = 0;
  if (N == 0) {
    for (uint32_t p = 0; p < n_particles; ++p) pair_offset[p + 1] = 0;
    return PD_OK;
  }
  Dev d;
  PairsArgs a;
  const int rc = build_grid(pos, node_offset, radius, n_particles, d, a);
  if (rc != PD_OK) return rc;
  uint64_t *poff;
  cudaError_t e = cudaSuccess;
  auto ck = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  ck(d.alloc(&a.deg, N));
  ck(d.alloc(&a.first, N + 1));
  ck(d.alloc(&poff, (size_t)n_particles + 1));
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? PD_ENOMEM : PD_ECUDA, cudaGetErrorString(e));
  const unsigned nb = (unsigned)((N + kScanBlock - 1) / kScanBlock);
  k_pairs<false><<<(unsigned)((N + 127) / 128), 128, 0, d.s>>>(a);
  k_sum_blocks<<<nb, kScanThreads, 0, d.s>>>(a.deg, a.sums, N);
  k_scan<uint64_t><<<nb, kScanThreads, 0, d.s>>>(a.deg, a.sums, a.first, N);
  k_particle_pairs<<<n_particles / 256 + 1, 256, 0, d.s>>>(a, poff);
  uint32_t odd = 0;
  std::vector<uint64_t> po((size_t)n_particles + 1);
  ck(cudaGetLastError());
  ck(cudaMemcpyAsync(&odd, a.bad, 4, cudaMemcpyDeviceToHost, d.s));
  ck(cudaMemcpyAsync(po.data(), poff, po.size() * 8, cudaMemcpyDeviceToHost, d.s));
  ck(cudaStreamSynchronize(d.s));
  if (e != cudaSuccess) return fail(PD_ECUDA, cudaGetErrorString(e));
  if (odd) return fail(PD_EINVAL, "non-finite position");
  const uint64_t M = po[n_particles];
  for (uint32_t p = 0; p < n_particles; ++p) pair_offset[p + 1] = po[p + 1];
  if (!pairs) return PD_OK;  // counts only
  if (cap < M) return fail(PD_EINVAL, "pair buffer too small: " + std::to_string(M) + " pairs");
  ck(d.alloc(&a.out, 2 * M));
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? PD_ENOMEM : PD_ECUDA, cudaGetErrorString(e));
  k_pairs<true><<<(unsigned)((N + 127) / 128), 128, 0, d.s>>>(a);
  k_sort_rows<<<kGrid, kThreads, 0, d.s>>>(a);
  k_sort_long<<<kGrid, kThreads, 0, d.s>>>(a);
  ck(cudaGetLastError());
  ck(cudaMemcpyAsync(pairs, a.out, 2 * M * 4, cudaMemcpyDeviceToHost, d.s));
  ck(cudaStreamSynchronize(d.s));
  if (e != cudaSuccess) return fail(PD_ECUDA, cudaGetErrorString(e));
  return PD_OK;
}

int pd_query_near(const double *pos, const uint64_t *node_offset, const double *radius, uint32_t n_particles,
                  const uint8_t *marked, uint8_t *near) {
  if (!marked || !near) return fail(PD_EINVAL, "null argument");
  const int bad = check_inputs(pos, node_offset, radius, n_particles);
  if (bad != PD_OK) return bad;
  const uint64_t N = node_offset[n_particles];
  if (N == 0) return PD_OK;
  Dev d;
  PairsArgs a;
  const int rc = build_grid(pos, node_offset, radius, n_particles, d, a);
  if (rc != PD_OK) return rc;
  uint8_t *dmark, *dnear;
  uint32_t odd = 0;
  cudaError_t e = cudaSuccess;
  auto ck = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  ck(d.alloc(&dmark, N));
  ck(d.alloc(&dnear, N));
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? PD_ENOMEM : PD_ECUDA, cudaGetErrorString(e));
  ck(cudaMemcpyAsync(dmark, marked, N, cudaMemcpyHostToDevice, d.s));
  k_near<<<(unsigned)((N + 127) / 128), 128, 0, d.s>>>(a, dmark, dnear);
  ck(cudaGetLastError());
  ck(cudaMemcpyAsync(&odd, a.bad, 4, cudaMemcpyDeviceToHost, d.s));
  ck(cudaStreamSynchronize(d.s));
  if (e == cudaSuccess && odd) return fail(PD_EINVAL, "non-finite position");
  ck(cudaMemcpyAsync(near, dnear, N, cudaMemcpyDeviceToHost, d.s));
  ck(cudaStreamSynchronize(d.s));
  if (e != cudaSuccess) return fail(PD_ECUDA, cudaGetErrorString(e));
  return PD_OK;
}

}  // extern "C"
