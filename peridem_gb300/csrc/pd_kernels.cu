// pd_kernels.cu -- the per-step kernels (compiled with -fmad=false).
//
// One step (src/particle/timeloop.h:395-797) is:
//   k_predict        predictor for all nodes (timeloop.h:537-540), step-max displacement
//                    increment for the broad-phase rebuild test, FP32 local displacement
//   [broad phase]    pd_broadphase.cu, runs only when a rebuild is due
//   k_step           FP64 fused per-node force and corrector: PD bond sum with breaking
//                    (particle2.h:107-237), self-contact, walls, extforce, torque
//                    (timeloop.h:544-634), node-node contact of particle pairs in
//                    ascending partner order (timeloop.h:636-651, contact.h:744-942) and
//                    the velocity-Verlet corrector (timeloop.h:661-781)
//   k_end_step       AABB refresh, clamped nodes, anchors, per-particle toggles; its last
//                    block: wall motion (timeloop.h:784-797), scheduled toggles, step counter
// Each node's force is gathered by one thread in the reference's summation order, so the
// FP64 form reproduces the reference bit for bit without atomics on forces.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include "pd_device.cuh"
#include "pd_end.cuh"
#include "pd_engine.h"
#include "pd_extra.cuh"
#include "pd_math.cuh"

namespace pdg {

// ------------------------------------------------------------------------------------
// predictor

__global__ void k_predict(DevView v) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float inc2 = 0.f;
  if (n < v.N) {
    const uint32_t k = v.pid[n];
    const DevPart &P = v.parts[k];
    const DevSimParams &sp = v.sp[P.sim];
    if (v.ss[P.sim].active) {
      D3 d = ld3(v.disp, n, v.Ncap), ve = ld3(v.vel_in, n, v.Ncap), a = ld3(v.acc, n, v.Ncap);
      // disp += dt*vel + (dt*dt*0.5)*acc  (timeloop.h:538, overloads.h:129-159)
      D3 dv = sp.dt * ve;
      D3 da = sp.hdt2 * a;
      D3 in = dv + da;
      d = d + in;
      st3(v.disp, n, v.Ncap, d);
      // squared increment in FP32 (only bounds the broad-phase rebuild test)
      const float ix = (float)in.x, iy = (float)in.y, iz = (float)in.z;
      inc2 = ix * ix + iy * iy + iz * iz;
      if (v.rec) {
        const double *an = v.anchor + 3 * (uint64_t)k;
        set_rec_u(v.rec[n], (float)(d.x - an[0]), (float)(d.y - an[1]), (float)(d.z - an[2]));
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) inc2 = fmaxf(inc2, __shfl_xor_sync(0xffffffffu, inc2, o));
  if ((threadIdx.x & 31) == 0 && inc2 > 0.f) {
    const double inc = sqrt((double)inc2) * (1.0 + 1e-5);
    atomicMax(&v.cnt->stepmax_bits, (unsigned long long)__double_as_longlong(inc));
  }
}

void launch_predict(const DevView &v, int tpb, cudaStream_t s) {
  uint64_t blocks = (v.N + tpb - 1) / tpb;
  if (blocks) k_predict<<<(unsigned)blocks, tpb, 0, s>>>(v);
}

// ------------------------------------------------------------------------------------
// fused force + corrector

// A bond's terms are the same seen from both of its ends, but for the sign of the unit vector: every
// operation on eta = (d_q - d_i) + xi is odd or even in it, rounding included. So each bond is
// evaluated once (k_pair64), and k_step's rows add the terms in the reference's order: 27 FP64
// instructions per row entry instead of 46 on a pipe that was 88 % busy (an FP64 instruction holds
// it for 16 cycles of an SM a warp), and on small handles a bond per thread instead of a row's
// square roots and divisions one after another.
// 778k nodes, 7.0e7 row entries: 6.1 ms in one kernel; now 2.2 ms here (the FP64 pipe) and 1.25 ms in
// k_step. 8,338 nodes: 257 us; now 30 us here and 56 us in k_step (and 13-39 in
// k_contact64).
__global__ void __launch_bounds__(256) k_pair64(const __grid_constant__ DevView v) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= v.M) return;
  const uint2 e = v.pair_end[k];
  const DevPart &P = v.parts[v.pid[e.x]];
  if (!P.movable || !v.ss[P.sim].active) return;
  const D3 xi = ld3(v.pair_xi, k, v.M);
  const D3 eta = (ld3(v.disp, e.y, v.Ncap) - ld3(v.disp, e.x, v.Ncap)) + xi;  // particle2.h:139-157
  const double xn = v.pair_xi[k + 3 * v.M], rxn = v.pair_xi[k + 4 * v.M];
  const double en = norm3(eta);
  const double str = div_rcp(en - xn, xn, rxn);
  const double ren = __drcp_rn(en);
  const double ux = div_rcp(eta.x, en, ren), uy = div_rcp(eta.y, en, ren), uz = div_rcp(eta.z, en, ren);
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(v.pair + k), "d"(str), "d"(ux), "d"(uy), "d"(uz)
               : "memory");
}

// a > b for a positive finite b, by integer comparison (a NaN is not).
__device__ __forceinline__ bool above(double a, long long b_bits) {
  const long long x = __double_as_longlong(a);
  return x > b_bits && x <= 0x7FF0000000000000ll;
}

// Least and largest of a warp's 64-bit keys.
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32));
  const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xffffffffu);
  return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) { return ~warp_min_key(~k); }

// Velocity-Verlet corrector of a node, given its whole force density (timeloop.h:662-781).
__device__ __forceinline__ void correct64(const DevView &v, uint64_t nn, uint32_t k, const DevPart &P,
                                          const DevSimParams &sp, const DevSimState &st, D3 vi, D3 f) {
  const uint64_t C3 = v.Ncap;
  const D3 ao = ld3(v.acc, nn, C3);
  D3 vo = vi;
  st3(v.force, nn, C3, f);
  if (nonfinite(f.x) || nonfinite(f.y) || nonfinite(f.z)) atomicOr(&v.cnt->err, PD_DERR_NONFINITE);
  if (P.movable) {
    if (v.afd && st.vconstraint && (int32_t)(k - sp.p0) == sp.pv_particle) st3(v.afd, nn, C3, ao);
    const D3 an = P.irho * f;
    D3 tmp = ao + an;
    tmp = sp.hdt * tmp;
    vo = vi + tmp;
    st3(v.acc, nn, C3, an);
  }
  st3(v.vel_out, nn, C3, vo);
}

// Node-level inputs of the non-bond force in this form: every movable node takes the walls' exact
// tests and its external force.
__device__ __forceinline__ ExtraCtx ctx64(const DevView &v, uint64_t n, uint32_t k, const DevPart &P,
                                          const DevSimParams &sp, D3 pi, D3 di, D3 vi) {
  ExtraCtx c;
  c.k = k;
  c.nc = v.cand_n[n] != 0;
  c.mov = P.movable != 0;
  c.wall_near = P.stoppable && sp.allow_wall;
  c.ext = c.mov;
  c.di = di;
  c.pi = pi;
  c.vi = vi;
  c.voli = v.vol[n];
  c.bdry_i = v.bdry[n] != 0;
  return c;
}

__global__ void __launch_bounds__(128) k_step(DevView v) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = n < v.N;
  const uint64_t nn = valid ? n : 0;
  const uint32_t k = v.pid[nn];
  const DevPart &P = v.parts[k];
  const DevSimParams &sp = v.sp[P.sim];
  DevSimState &st = v.ss[P.sim];
  const bool run = valid && st.active;
  const uint64_t C3 = v.Ncap;

  D3 f = d3(0.0, 0.0, 0.0);
  D3 di = ld3(v.disp, nn, C3);
  const D3 pi = ld3(v.pos, nn, C3);
  const D3 vi = ld3(v.vel_in, nn, C3);
  unsigned long long live = 0;

  if (run && P.movable) {
    // ---- peridynamic bond force (particle2.h:117-157) and breaking (particle2.h:196-237)
    const uint64_t s = nn >> 5;
    const uint32_t lane = (uint32_t)(nn & 31);
    const uint64_t base = v.slice_ptr[s] + lane;
    const uint64_t mbase = v.slice_ptr[s] >> 5;
    const int dg = v.deg[nn];
    const bool brk = st.fracture && P.breakable && P.break_bonds;
    D3 acc = d3(0.0, 0.0, 0.0);
    const bool pos_snot = P.snot > 0 && isfinite(P.snot);
    const long long snot_bits = __double_as_longlong(P.snot);
    // four entries at a time, added in row order; the terms of the next four and the indices of the
    // four after them are requested before these are added
    struct Index {
      uint32_t mw, lw, id, q;
    };
    struct Terms {
      double s, x, y, z, vol;
    };
    auto index = [&](int j) {
      const bool in = j < dg;
      const uint64_t e = base + 32ull * j;
      return Index{in ? v.mask[mbase + j] : 0u, in ? v.plow[mbase + j] : 0u, in ? v.pidx[e] : 0u,
                   in ? v.col[e] : (uint32_t)nn};
    };
    auto terms = [&](const Index &i) {
      Terms t;
      asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
          : "=d"(t.s), "=d"(t.x), "=d"(t.y), "=d"(t.z)
          : "l"(v.pair + i.id));
      t.vol = v.vol[i.q];
      return t;
    };
    constexpr int U = 4;
    Index now[U], next[U];
    Terms tn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) now[u] = index(u);
#pragma unroll
    for (int u = 0; u < U; ++u) next[u] = index(U + u);
#pragma unroll
    for (int u = 0; u < U; ++u) tn[u] = terms(now[u]);
    for (int j0 = 0; j0 < dg; j0 += U) {
      Terms t[U];
      Index after[U];
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = tn[u];
#pragma unroll
      for (int u = 0; u < U; ++u) tn[u] = terms(next[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) after[u] = index(j0 + 2 * U + u);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!((now[u].mw >> lane) & 1u)) continue;
        ++live;
        double mag = (P.cnot * t[u].s) * t[u].vol;
        // the partner's side: the unit vector negated, here as the sign of its factor
        mag = __hiloint2double(__double2hiint(mag) ^ (int)(((now[u].lw >> lane) & 1u) << 31), __double2loint(mag));
        acc = acc + mag * d3(t[u].x, t[u].y, t[u].z);
        if (brk && (pos_snot ? above(t[u].s, snot_bits) : t[u].s > P.snot))
          atomicAnd(&v.mask[mbase + j0 + u], ~(1u << lane));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        now[u] = next[u];
        next[u] = after[u];
      }
    }
    f = d3(0.0, 0.0, 0.0) + acc;
  }

  // walls, external force and torque, then the corrector. A node with contact candidates leaves its
  // bond sum to k_contact64 instead: its pairs are chains of FP64 square roots and divisions, ~5 us
  // each, on which the node's whole warp and then the kernel would wait.
  if (run) {
    if (v.cand_n[nn] != 0) {
      st3(v.force, nn, C3, f);
    } else {
      extra_middle(v, nn, P, sp, st, ctx64(v, nn, k, P, sp, pi, di, vi), f);
      correct64(v, nn, k, P, sp, st, vi, f);
    }
  }

  // ---- AABB of CurrPos for the next step (timeloop.h:779), warp-reduced as ordered keys (integer
  // instructions: FP64 comparisons share the pipe with the bond terms); a NaN coordinate counts as
  // absent
  {
    const bool contrib = run && P.movable;
    const D3 cur = pi + di;
    unsigned long long lo[3], hi[3];
    for (int c = 0; c < 3; ++c) {
      const double x = comp(cur, c);
      const bool on = contrib && !((__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll) > 0x7FF0000000000000ll);
      lo[c] = ord_key(on ? x : INFINITY);
      hi[c] = ord_key(on ? x : -INFINITY);
    }
    const uint32_t k0 = __shfl_sync(0xffffffffu, k, 0);
    const bool uniform = __all_sync(0xffffffffu, k == k0);
    if (uniform) {
      for (int c = 0; c < 3; ++c) {
        lo[c] = warp_min_key(lo[c]);
        hi[c] = warp_max_key(hi[c]);
      }
    }
    const bool writer = uniform ? ((threadIdx.x & 31) == 0) : contrib;
    if (writer && lo[0] <= hi[0]) {
      unsigned long long *L = reinterpret_cast<unsigned long long *>(v.lrtb_next) + 6 * (uint64_t)k;
      for (int c = 0; c < 3; ++c) {
        atomicMin(&L[c], lo[c]);
        atomicMax(&L[3 + c], hi[c]);
      }
    }
  }

  if (v.stats) {
    for (int o = 16; o > 0; o >>= 1) live += __shfl_xor_sync(0xffffffffu, live, o);
    if ((threadIdx.x & 31) == 0 && live) atomicAdd(&v.cnt->live_bonds, live);
  }
}

// The nodes with contact candidates (listed when the lists are built): eight lanes each, sharing the
// listed candidates and adding their forces to the bond sum in the reference's order (extra_lanes). A
// warp's four groups start each round of nodes together: once apart they stay so, and the warp takes
// their nodes one after another (453k nodes with 29 candidates each: a few such warps 10 ms, all others 2).
// Then the nodes whose list overflowed, a thread each in the engine's order, so that the threads of a warp
// scan the same cells (453k nodes at a contact radius of 1.6 spacings, some of them: 26 ms a step with one of
// the eight lanes, 19 now; of 1.9, all of them: 3.9 s, 1.2 now).
__global__ void __launch_bounds__(128) k_contact64(const __grid_constant__ DevView v) {
  constexpr uint32_t L = 8, G = 32 / L;
  const uint32_t nx = v.xcount[0], lane = threadIdx.x & 31u, sub = lane & (L - 1);
  const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  auto node = [&](uint64_t n, bool writer, auto add) {
    const uint32_t k = v.pid[n];
    const DevPart &P = v.parts[k];
    const DevSimParams &sp = v.sp[P.sim];
    DevSimState &st = v.ss[P.sim];
    if (!st.active) return;
    const D3 vi = ld3(v.vel_in, n, v.Ncap);
    const ExtraCtx c = ctx64(v, n, k, P, sp, ld3(v.pos, n, v.Ncap), ld3(v.disp, n, v.Ncap), vi);
    const D3 f = add(P, sp, st, c, ld3(v.force, n, v.Ncap));
    if (writer) correct64(v, n, k, P, sp, st, vi, f);
  };
  for (uint32_t i0 = thread / 32 * G; i0 < nx; i0 += threads / 32 * G) {
    __syncwarp();
    const uint32_t i = i0 + lane / L;
    if (i >= nx) continue;  // the group's lanes together
    const uint64_t n = v.xnodes[i];
    if (v.cand_n[n] == kCandCells) continue;
    node(n, sub == 0, [&](const DevPart &P, const DevSimParams &sp, DevSimState &st, const ExtraCtx &c, D3 f) {
      return extra_lanes<L>(v, n, P, sp, st, c, f, sub, lane - sub);
    });
  }
  if (nx == 0) return;
  for (uint64_t n = thread; n < v.N; n += threads)
    if (v.cand_n[n] == kCandCells)
      node(n, true, [&](const DevPart &P, const DevSimParams &sp, DevSimState &st, const ExtraCtx &c, D3 f) {
        return extra_walk(v, n, P, sp, st, c, f);
      });
}

void launch_step_kernel(const DevView &v, int precision, int variant, cudaStream_t s) {
  uint64_t blocks = (v.N + 127) / 128;
  if (!blocks) return;
  if (precision == PD_FP32C) {
    launch_step_fp32c(v, variant, s);
    return;
  }
  if (v.M) k_pair64<<<(unsigned)((v.M + 255) / 256), 256, 0, s>>>(v);
  // a small handle's warps one to a block, so that they spread over every SM (8,338 nodes in blocks of
  // 128 threads would use 66 of 152)
  if (v.N < 152 * 512) k_step<<<(unsigned)((v.N + 31) / 32), 32, 0, s>>>(v);
  else k_step<<<(unsigned)blocks, 128, 0, s>>>(v);
  k_contact64<<<152 * 4, 128, 0, s>>>(v);
}

// ------------------------------------------------------------------------------------
// end of step

// Per-particle end of step, then (last block) the simulations' advance (pd_end.cuh). One kernel:
// the particles read their simulation's state of this step and derive the next step's wall
// planes and step index themselves, with the same arithmetic as the advance, which the last block
// to finish applies once every other block is done reading.
__global__ void k_end_step(DevView v, const uint32_t *clamped_ptr, const uint32_t *clamped, double *clamped_disp) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < v.P) end_step_particle(v, k, clamped_ptr, clamped, clamped_disp);
  // the last block to finish advances the simulations and the step counters
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&v.cnt->end_blocks, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  end_step_advance(v, threadIdx.x, blockDim.x);
}

// The FP32 form's end of step with one warp per particle (end_particle_warp), the last block
// advancing the simulations as in k_end_step.
__global__ void __launch_bounds__(128) k_end_step_w(DevView v) {
  const uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k < v.P) end_particle_warp(v, (uint32_t)k, threadIdx.x & 31);
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&v.cnt->end_blocks, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  end_step_advance(v, threadIdx.x, blockDim.x);
}

void launch_end_step(const DevView &v, const uint32_t *clamped, uint64_t n_clamped, double *clamped_disp,
                     cudaStream_t s) {
  if (v.rec && v.fused) {  // FP32 form (its clamped nodes are handled by the corrector)
    k_end_step_w<<<(v.P + 3) / 4, 128, 0, s>>>(v);
    return;
  }
  const uint32_t *cptr = n_clamped ? clamped : nullptr;
  const uint32_t *clist = n_clamped ? clamped + (v.P + 1) : nullptr;
  k_end_step<<<(v.P + 127) / 128, 128, 0, s>>>(v, cptr, clist, clamped_disp);
}

// ------------------------------------------------------------------------------------
// auxiliary kernels

// Component c of the sum of load(i), i = 0 .. n - 1, added in that order (a mean in file node order, like
// the reference's += loops), on thread c < 3 of a block of kSumThreads: all threads fetch a round of terms
// into shared memory while those three add the round before. Bound by the chain of FP64 additions; by one
// thread alone each term also waited for its gather, the longer the farther the engine's node order is
// from the file's: a step with torque on 64k nodes 7.9 ms in file order, 8.2 along the curve, now 2.7.
constexpr uint32_t kSumThreads = 256;
template <class F>
__device__ __forceinline__ double ordered_sum(uint32_t n, F load) {
  __shared__ double sh[2][3][kSumThreads + 1];
  const uint32_t t = threadIdx.x;
  double m = 0.0;
  D3 x = t < n ? load(t) : d3(0.0, 0.0, 0.0);
  for (uint32_t b = 0; b < n; b += kSumThreads) {
    double(*r)[kSumThreads + 1] = sh[(b / kSumThreads) & 1u];
    r[0][t] = x.x;
    r[1][t] = x.y;
    r[2][t] = x.z;
    __syncthreads();  // the adders are done with the round before the last, whose place this one took
    if (n - b > kSumThreads + t) x = load(b + kSumThreads + t);
    if (t < 3) {
      const uint32_t c = min(n - b, kSumThreads);
#pragma unroll 8
      for (uint32_t j = 0; j < c; ++j) m = m + r[t][j];
    }
  }
  return m;
}

// mean_CurrPos per particle (particle2.h:94-103).
__global__ void __launch_bounds__(kSumThreads) k_centroids(DevView v) {
  const uint32_t k = blockIdx.x;
  const DevPart &P = v.parts[k];
  if (!v.ss[P.sim].torque) return;
  const double m = ordered_sum(P.n, [&](uint32_t i) {
    const uint32_t g = v.node_of[P.g0 + i];
    return ld3(v.pos, g, v.Ncap) + ld3(v.disp, g, v.Ncap);
  });
  if (threadIdx.x < 3) const_cast<double *>(v.centroid)[3 * (uint64_t)k + threadIdx.x] = m / (double)P.n;
}

void launch_centroids(const DevView &v, cudaStream_t s) {
  if (v.P) k_centroids<<<v.P, kSumThreads, 0, s>>>(v);
}

// Prescribed velocity of one particle per simulation, after the corrector (timeloop.h:684-764):
// the particle's velocity is split into its mean and the rest; the mean's x component
// (fix_velocity_mean_x) and the rest (fix_velocity_angular: rotation about z at the
// prescribed rate, about mean_CurrPos) are replaced. applied_force_density =
// rho*((2/dt)*(pv - vel) - acc_old) - force, with vel already equal to pv (as in the
// reference). The means are sequential sums in file node order, like Eigen's += loop.
__global__ void __launch_bounds__(kSumThreads) k_prescribed(DevView v) {
  const uint32_t s = blockIdx.x;
  if (s >= v.S) return;
  const DevSimParams &sp = v.sp[s];
  const DevSimState &st = v.ss[s];
  if (!st.active || !st.vconstraint || sp.pv_particle < 0) return;
  const uint32_t k = sp.p0 + (uint32_t)sp.pv_particle;
  const DevPart &P = v.parts[k];
  if (!P.movable) return;
  const uint64_t C3 = v.Ncap;
  __shared__ double sh[6];
  const double mv = ordered_sum(P.n, [&](uint32_t i) { return ld3(v.vel_out, v.node_of[P.g0 + i], C3); });
  if (threadIdx.x < 3) sh[threadIdx.x] = mv / (double)P.n;
  if (sp.fix_angular) {  // mean_CurrPos (particle2.h:94-103)
    const double mp = ordered_sum(P.n, [&](uint32_t i) {
      const uint32_t g = v.node_of[P.g0 + i];
      return ld3(v.pos, g, C3) + ld3(v.disp, g, C3);
    });
    if (threadIdx.x < 3) sh[3 + threadIdx.x] = mp / (double)P.n;
  }
  __syncthreads();
  const double two_dt = 2 / sp.dt;
  float i2 = 0.f;
  for (uint32_t i = threadIdx.x; i < P.n; i += blockDim.x) {
    const uint64_t g = P.g0 + i;
    const D3 vel = ld3(v.vel_out, g, C3);
    D3 mean = d3(sh[0], sh[1], sh[2]);
    D3 vrot = vel - mean;
    if (sp.fix_mean_x) mean.x = sp.pv_mean_x;
    if (sp.fix_angular) {
      const D3 rv = (ld3(v.pos, g, C3) + ld3(v.disp, g, C3)) - d3(sh[3], sh[4], sh[5]);
      const double r = norm3(rv);
      D3 ru = d3(0.0, 0.0, 0.0);
      if (r > 0) ru = d3(rv.x / r, rv.y / r, rv.z / r);
      const double rw = r * sp.pv_angular;
      vrot = d3(-rw * ru.y, rw * ru.x, 0.0);
    }
    const D3 pv = vrot + mean;
    const bool clamped32 = v.fused && v.clamp_flag[g];  // FP32 form: clamped nodes already at rest
    if (!clamped32) st3(v.vel_out, g, C3, pv);
    const D3 dd = pv - pv;
    const D3 a = (two_dt * dd) - ld3(v.afd, g, C3);
    st3(v.afd, g, C3, (P.rho * a) - ld3(v.force, g, C3));
    if (v.fused && !clamped32) {
      // the fused predictor of the FP32 form ran with the velocity before the overwrite
      const D3 d = ld3(v.disp, g, C3);
      const D3 an = ld3(v.acc, g, C3);
      const D3 inc = sp.dt * pv + sp.hdt2 * an;
      const D3 dn = d + inc;
      st3(v.disp_next, g, C3, dn);
      const double *anx = v.anchor_next + 3 * (uint64_t)k;
      set_rec_u(v.rec_next[g], (float)(dn.x - anx[0]), (float)(dn.y - anx[1]), (float)(dn.z - anx[2]));
      const float ix = (float)(dn.x - d.x), iy = (float)(dn.y - d.y), iz = (float)(dn.z - d.z);
      i2 = fmaxf(i2, ix * ix + iy * iy + iz * iz);
    }
  }
  for (int o = 16; o > 0; o >>= 1) i2 = fmaxf(i2, __shfl_xor_sync(0xffffffffu, i2, o));
  if ((threadIdx.x & 31) == 0 && i2 > 0.f) {
    const double inc = sqrt((double)i2) * (1.0 + 1e-5);
    atomicMax(&v.cnt->stepmax_bits, (unsigned long long)__double_as_longlong(inc));
  }
}

void launch_prescribed(const DevView &v, cudaStream_t s) {
  if (v.S && v.afd) k_prescribed<<<v.S, kSumThreads, 0, s>>>(v);
}

// reset_partzero_y at the top of step t (timeloop.h:500-535): particle 0 is lifted so that its
// mean y sits wheel_rad + contact radius above the highest node of the other particles within
// wheel_rad (in x) of its mean x. The displacement read here is the one after the previous
// corrector (clamped nodes at zero).
__device__ __forceinline__ D3 disp_after_corrector(const DevView &v, uint64_t g, uint32_t t) {
  if (v.fused) {  // FP32 form: the previous step's buffer keeps clamped nodes' prediction
    if (t > 1 && v.clamp_flag[g]) return d3(0.0, 0.0, 0.0);
    return ld3(v.disp_next, g, v.Ncap);
  }
  return ld3(v.disp, g, v.Ncap);
}

__global__ void __launch_bounds__(kSumThreads) k_reset_y(DevView v) {
  const uint32_t s = blockIdx.x;
  if (s >= v.S) return;
  const DevSimParams &sp = v.sp[s];
  const DevSimState &st = v.ss[s];
  if (!st.active || !sp.reset_y || st.t != sp.reset_y_ts) return;
  const uint64_t C3 = v.Ncap;
  const DevPart &P0 = v.parts[sp.p0];
  const DevPart &P1 = v.parts[sp.p0 + 1];
  __shared__ double m0[3];
  __shared__ unsigned long long best;
  __shared__ int found;
  __shared__ double move;
  const double m = ordered_sum(P0.n, [&](uint32_t i) {
    const uint32_t g = v.node_of[P0.g0 + i];
    return ld3(v.pos, g, C3) + disp_after_corrector(v, g, st.t);
  });
  if (threadIdx.x < 3) m0[threadIdx.x] = m / (double)P0.n;
  if (threadIdx.x == 0) {
    best = ord_key(-INFINITY);
    found = 0;
  }
  __syncthreads();
  // highest y among the other particles' nodes near particle 0's mean x (an exact max)
  const uint64_t a = P1.g0, b = sp.node0 + sp.nnodes;
  double my = -INFINITY;
  int any = 0;
  for (uint64_t g = a + threadIdx.x; g < b; g += blockDim.x) {
    const D3 now = ld3(v.pos, g, C3) + disp_after_corrector(v, g, st.t);
    if (fabs(m0[0] - now.x) <= sp.wheel_rad) {
      any = 1;
      my = fmax(my, now.y);
    }
  }
  if (any) {
    atomicMax(&best, ord_key(my));
    found = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double max_bulk_y;
    if (found) {
      max_bulk_y = ord_val(best);
    } else {  // the reference's initial value: pos[0] of particle 1 plus disp[1] (file order)
      const uint64_t j = P1.n > 1 ? 1 : 0;
      max_bulk_y = v.pos[v.node_of[P1.g0] + C3] + disp_after_corrector(v, v.node_of[P1.g0 + j], st.t).y;
    }
    const double dest = (max_bulk_y + sp.wheel_rad) + sp.Rc;
    move = dest - m0[1];
    v.cnt->xall = 1;       // particle 0 moved: the non-bond work lists are stale for this step
    v.cnt->moved = 1e300;  // and so are the contact candidate lists: this step rebuilds them
    if (v.fused) {  // the FP32 form keeps positions relative to the particle's anchor
      DevPart &Pw = v.parts[sp.p0];
      Pw.anchor_pos[1] = Pw.anchor_pos[1] + move;
      float *wl = v.wall_local + 6 * (uint64_t)sp.p0;
      const double *an = v.anchor + 3 * (uint64_t)sp.p0;
      for (int f = 0; f < 6; ++f) {
        const int c = f % 3;
        wl[f] = (float)(st.wall[f] - (Pw.anchor_pos[c] + an[c]));
      }
    }
  }
  __syncthreads();
  double *py = const_cast<double *>(v.pos) + C3;
  for (uint32_t i = threadIdx.x; i < P0.n; i += blockDim.x) py[P0.g0 + i] = py[P0.g0 + i] + move;
}

void launch_reset_y(const DevView &v, cudaStream_t s) {
  if (v.S) k_reset_y<<<v.S, kSumThreads, 0, s>>>(v);
}

// The pairs of the FP64 form. The end with the lower file index owns a bond; of a bond of a node with
// itself, pushed twice onto its row, the first entry does. A node's pairs lie one after another in
// row order, the nodes of a block in order, the blocks in the order they finish counting (a pair's
// place does not matter to any result).
__global__ void __launch_bounds__(256) k_pair_count(const __grid_constant__ DevView v, uint32_t *first, uint32_t *low,
                                                    uint32_t *total) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t own = 0, other = 0;
  if (n < v.N) {
    const uint32_t *row = v.col + v.slice_ptr[n >> 5] + (n & 31);
    const uint32_t fn = v.file_of[n];
    const int dg = v.deg[n];
    bool again = false;
    for (int j = 0; j < dg; ++j) {
      const uint32_t q = row[32 * j];
      const bool mine = q == n ? !again : v.file_of[q] > fn;
      if (q == n) again = !again;
      mine ? ++own : ++other;
    }
  }
  __shared__ uint32_t warps[8], base;
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t s = own;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= (uint32_t)o) s += y;
  }
  if (lane == 31) warps[w] = s;
  __syncthreads();
  uint32_t before = 0, sum = 0;
  for (uint32_t i = 0; i < 8; ++i) {
    if (i < w) before += warps[i];
    sum += warps[i];
  }
  if (threadIdx.x == 0) base = atomicAdd(total, sum);
  __syncthreads();
  if (n < v.N) {
    first[n] = base + before + s - own;
    low[n] = other;
  }
}

// gen_xi (particle2.h:241-257) for the owned pairs: xi = pos[q] - pos[i], |xi| and RN(1/|xi|); every
// entry's pair: an owner's its own, another's the one its partner's row holds for it.
__global__ void __launch_bounds__(256) k_pair_fill(const __grid_constant__ DevView v, bool sorted,
                                                   const uint32_t *first, const uint32_t *low, uint2 *end, double *xi,
                                                   uint32_t *pidx, uint32_t *plow) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;  // whole warps: Ncap is a multiple of 32
  if (n >= v.Ncap) return;
  const uint32_t lane = (uint32_t)(n & 31);
  const uint64_t base = v.slice_ptr[n >> 5];
  const int dg = n < v.N ? v.deg[n] : 0, w = (int)((v.slice_ptr[(n >> 5) + 1] - base) >> 5);
  const uint32_t fn = n < v.N ? v.file_of[n] : 0u;
  const D3 pi = ld3(v.pos, n, v.Ncap);
  uint32_t k = n < v.N ? first[n] : 0u;
  uint32_t again = 0, self = 0;
  for (int j = 0; j < w; ++j) {
    const uint64_t e = base + 32ull * j + lane;
    bool theirs = false;
    if (j < dg) {
      const uint32_t q = v.col[e];
      const uint32_t fq = v.file_of[q];
      if (q == n ? !again : fq > fn) {
        const D3 x = ld3(v.pos, q, v.Ncap) - pi;
        const double xn = norm3(x);
        end[k] = make_uint2((uint32_t)n, q);
        xi[k] = x.x;
        xi[k + v.M] = x.y;
        xi[k + 2 * v.M] = x.z;
        xi[k + 3 * v.M] = xn;
        xi[k + 4 * v.M] = __drcp_rn(xn);
        if (q == n) self = k;
        pidx[e] = k++;
      } else if (q == n) {
        theirs = true;
        pidx[e] = self;
      } else {
        theirs = true;
        const uint32_t *row = v.col + v.slice_ptr[q >> 5] + (q & 31);
        const int dq = v.deg[q];
        uint32_t at = 0;
        if (sorted) {  // the row ascends by file index, the entries q owns last
          int a = 0, b = dq;
          while (b - a > 1) {
            const int m = (a + b) >> 1;
            if (v.file_of[row[32 * m]] <= fn) a = m;
            else b = m;
          }
          at = (uint32_t)a - low[q];
        } else {  // the owned entries before it
          bool twice = false;
          for (int m = 0; m < dq && row[32 * m] != n; ++m) {
            const uint32_t c = row[32 * m];
            at += (c == q ? !twice : v.file_of[c] > fq) ? 1u : 0u;
            if (c == q) twice = !twice;
          }
        }
        pidx[e] = first[q] + at;
      }
      if (q == n) again ^= 1u;
    } else {
      pidx[e] = 0;
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, theirs);
    if (lane == 0) plow[(base >> 5) + j] = bits;
  }
}

void launch_pair_build(const DevView &v, bool sorted, uint32_t *first, uint32_t *low, uint32_t *total, uint2 *end,
                       double *xi, uint32_t *pidx, uint32_t *plow, cudaStream_t s) {
  k_pair_count<<<(unsigned)((v.N + 255) / 256), 256, 0, s>>>(v, first, low, total);
  k_pair_fill<<<(unsigned)((v.Ncap + 255) / 256), 256, 0, s>>>(v, sorted, first, low, end, xi, pidx, plow);
}

// AABBs of all particles before the loop (timeloop.h:389-393). A warp whose nodes all belong to
// one particle reduces its keys with shuffles first (min/max are exact, so the result does not
// depend on how they are combined), which keeps the atomics on a particle's six keys few.
__global__ void k_init_lrtb_acc(DevView v) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = n < v.N;
  const uint32_t k = valid ? v.pid[n] : 0xFFFFFFFFu;
  unsigned long long lo[3], hi[3];
  if (valid) {
    const D3 cur = ld3(v.pos, n, v.Ncap) + ld3(v.disp, n, v.Ncap);
    lo[0] = hi[0] = ord_key(cur.x);
    lo[1] = hi[1] = ord_key(cur.y);
    lo[2] = hi[2] = ord_key(cur.z);
  } else {
    for (int c = 0; c < 3; ++c) {
      lo[c] = ord_key(INFINITY);
      hi[c] = ord_key(-INFINITY);
    }
  }
  const uint32_t k0 = __shfl_sync(0xffffffffu, k, 0);
  if (__all_sync(0xffffffffu, !valid || k == k0)) {  // lanes past N carry the identity keys
    if (k0 == 0xFFFFFFFFu) return;
    for (int o = 16; o > 0; o >>= 1)
      for (int c = 0; c < 3; ++c) {
        lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
        hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
      }
    if ((threadIdx.x & 31) != 0) return;
  } else if (!valid) {
    return;
  }
  const uint64_t kp = valid ? k : k0;
  unsigned long long *L = reinterpret_cast<unsigned long long *>(v.lrtb_next) + 6 * kp;
  for (int c = 0; c < 3; ++c) {
    atomicMin(&L[c], lo[c]);
    atomicMax(&L[3 + c], hi[c]);
  }
}
__global__ void k_init_lrtb_fin(DevView v) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= v.P) return;
  unsigned long long *L = reinterpret_cast<unsigned long long *>(v.lrtb_next) + 6 * (uint64_t)k;
  for (int c = 0; c < 6; ++c) v.lrtb[6 * (uint64_t)k + c] = ord_val(L[c]);
  for (int c = 0; c < 3; ++c) {
    L[c] = ord_key(INFINITY);
    L[3 + c] = ord_key(-INFINITY);
  }
  if (v.rec) {
    const DevPart &P = v.parts[k];
    const DevSimState &st = v.ss[P.sim];
    double *an = const_cast<double *>(v.anchor) + 3 * (uint64_t)k;
    an[0] = v.disp[P.anchor];
    an[1] = v.disp[P.anchor + v.Ncap];
    an[2] = v.disp[P.anchor + 2 * v.Ncap];
    // the breaking band from the anchor-relative extent of the current positions
    double ext = 0.0;
    for (int c = 0; c < 3; ++c) {
      const double A = P.anchor_pos[c] + an[c];
      ext = fmax(ext, fmax(fabs(v.lrtb[6 * (uint64_t)k + c] - A), fabs(v.lrtb[6 * (uint64_t)k + 3 + c] - A)));
    }
    set_break_band(v.parts[k], u_extent(P, ext * (1.0 + 1e-6)));
    unsigned int *Lf = v.lrtb_local_next + 6 * (uint64_t)k;
    float *wl = v.wall_local + 6 * (uint64_t)k;
    for (int c = 0; c < 3; ++c) {
      Lf[c] = fkey(INFINITY);
      Lf[3 + c] = fkey(-INFINITY);
    }
    for (int f = 0; f < 6; ++f) wl[f] = (float)(st.wall[f] - (P.anchor_pos[f % 3] + an[f % 3]));
  }
}
__global__ void k_reset_lrtb_next(DevView v) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= v.P) return;
  unsigned long long *L = reinterpret_cast<unsigned long long *>(v.lrtb_next) + 6 * (uint64_t)k;
  for (int c = 0; c < 3; ++c) {
    L[c] = ord_key(INFINITY);
    L[3 + c] = ord_key(-INFINITY);
  }
}

void launch_init_lrtb(const DevView &v, cudaStream_t s) {
  if (!v.P) return;
  k_reset_lrtb_next<<<(v.P + 127) / 128, 128, 0, s>>>(v);
  uint64_t blocks = (v.N + 127) / 128;
  if (blocks) k_init_lrtb_acc<<<(unsigned)blocks, 128, 0, s>>>(v);
  k_init_lrtb_fin<<<(v.P + 127) / 128, 128, 0, s>>>(v);
}

// Readback in file order: a [3][Ncap] engine-order array (plus `add` of the same layout,
// added as add + src, when given) -> N*3 rows in file order.
__global__ void k_rows_to_file(const double *src, const double *add, uint64_t Ncap, uint64_t N,
                               const uint32_t *file_of, double *dst) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const uint64_t f = file_of[n];
  for (int c = 0; c < 3; ++c) {
    const double x = src[c * Ncap + n];
    dst[3 * f + c] = add ? add[c * Ncap + n] + x : x;
  }
}

// The rows of the clamped nodes: zero (FP32 form's displacement after a step), or pos + the
// predicted displacement kept for them (FP64 form's CurrPos, timeloop.h:767-774).
__global__ void k_clamped_rows(const uint32_t *clamped, uint64_t n_clamped, const uint32_t *file_of,
                               const double *pos, const double *cdisp, uint64_t Ncap, double *dst) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_clamped) return;
  const uint64_t g = clamped[i], f = file_of[g];
  for (int c = 0; c < 3; ++c) dst[3 * f + c] = cdisp ? pos[c * Ncap + g] + cdisp[3 * i + c] : 0.0;
}

void launch_rows_to_file(const double *src, const double *add, uint64_t Ncap, uint64_t N, const uint32_t *file_of,
                         double *dst, cudaStream_t s) {
  if (N) k_rows_to_file<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(src, add, Ncap, N, file_of, dst);
}

void launch_clamped_rows(const uint32_t *clamped, uint64_t n_clamped, const uint32_t *file_of, const double *pos,
                         const double *cdisp, uint64_t Ncap, double *dst, cudaStream_t s) {
  if (n_clamped)
    k_clamped_rows<<<(unsigned)((n_clamped + 127) / 128), 128, 0, s>>>(clamped, n_clamped, file_of, pos, cdisp,
                                                                       Ncap, dst);
}

// Number of particle pairs the pair loop evaluates (timeloop.h:641-649), for the
// progress line's "#contacts" column.
__global__ void k_pairwise(DevView v) {
  const uint32_t s = blockIdx.y;
  if (s >= v.S) return;
  const DevSimParams &sp = v.sp[s];
  if (!v.ss[s].active) return;
  const uint64_t np = sp.np;
  const uint64_t total = np * (np - 1) / 2;
  unsigned long long cnt = 0;
  for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (uint64_t)gridDim.x * blockDim.x) {
    // invert idx -> (i, j), i < j, lexicographic
    uint64_t i = (uint64_t)((2.0 * np - 1 - sqrt((2.0 * np - 1) * (2.0 * np - 1) - 8.0 * idx)) / 2);
    while (i > 0 && i * (2 * np - i - 1) / 2 > idx) --i;
    while ((i + 1) * (2 * np - i - 2) / 2 <= idx) ++i;
    uint64_t j = idx - i * (2 * np - i - 1) / 2 + i + 1;
    const uint32_t a = sp.p0 + (uint32_t)i, b = sp.p0 + (uint32_t)j;
    if (!(v.parts[a].movable || v.parts[b].movable)) continue;
    if (intersects_fext(v.lrtb + 6 * (uint64_t)a, v.lrtb + 6 * (uint64_t)b, sp.Rc)) ++cnt;
  }
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&v.cnt->pairwise, cnt);
}

void launch_pairwise_count(const DevView &v, cudaStream_t s) {
  if (!v.S) return;
  dim3 grid(64, v.S);
  k_pairwise<<<grid, 256, 0, s>>>(v);
}

}  // namespace pdg

namespace pdg {

// Live directed bonds of movable particles: popcount of each node's live bits.
__global__ void k_count_live(DevView v, unsigned long long *out) {
  const uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long c = 0;
  if (n < v.N && v.parts[v.pid[n]].movable) {
    const uint64_t s = n >> 5;
    const uint32_t lane = (uint32_t)(n & 31);
    const uint64_t mbase = v.slice_ptr[s] >> 5;
    const int dg = v.deg[n];
    for (int j = 0; j < dg; ++j) c += (v.mask[mbase + j] >> lane) & 1u;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

void launch_count_live(const DevView &v, unsigned long long *out, cudaStream_t s) {
  uint64_t blocks = (v.N + 255) / 256;
  if (blocks) k_count_live<<<(unsigned)blocks, 256, 0, s>>>(v, out);
}

// Bonds of each node as a saved Connectivity counts them: NbdArr2conn (timeloop.h:20-44)
// keeps the live pair (i, q) for i < q only, and total_neighbors (plot3d_timestep.py:95-105)
// counts each kept pair at both ends. So row n adds every live partner above it in file
// order to both n and that partner. Nodes [n0, n0 + nn) are whole particles (the same range
// in engine and file order); now[] is indexed by file order - n0 and starts at zero.
__global__ void k_damage_count(DevView v, uint64_t n0, uint64_t nn, uint32_t *now) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nn) return;
  const uint64_t n = n0 + k;
  const uint64_t e0 = v.slice_ptr[n >> 5];
  const uint32_t lane = (uint32_t)(n & 31);
  const uint32_t fn = v.file_of[n];
  const int dg = v.deg[n];
  uint32_t own = 0;
  for (int j = 0; j < dg; ++j) {
    if (!((v.mask[(e0 >> 5) + j] >> lane) & 1u)) continue;
    const uint32_t fq = v.file_of[v.col[e0 + 32 * (uint64_t)j + lane] & kColIndex];
    if (fq > fn) {
      ++own;
      atomicAdd(&now[fq - n0], 1u);
    }
  }
  if (own) atomicAdd(&now[fn - n0], own);
}

// damage = (orig - now) / orig per node (plot3d_timestep.py:156-166), orig being the node's
// bond count in the setup's Connectivity (its row length); 0/0 gives NaN as it does there.
__global__ void k_damage_out(DevView v, uint64_t n0, uint64_t nn, const uint32_t *now, double *out) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nn) return;
  const uint64_t n = n0 + k;
  const uint64_t f = v.file_of[n] - n0;
  const double orig = (double)v.deg[n];
  out[f] = (orig - (double)now[f]) / orig;
}

void launch_damage(const DevView &v, uint64_t n0, uint64_t nn, uint32_t *now, double *out, cudaStream_t s) {
  const uint64_t blocks = (nn + 255) / 256;
  if (!blocks) return;
  k_damage_count<<<(unsigned)blocks, 256, 0, s>>>(v, n0, nn, now);
  k_damage_out<<<(unsigned)blocks, 256, 0, s>>>(v, n0, nn, now, out);
}

}  // namespace pdg
