// The dust photon loop (cmi_dust.cuh) by whole paths: one lane follows one source
// packet through all of its walks -- depth to the box edge, forced first scattering,
// and per scattering the peel-off copy to the image and the next walk -- with the
// FP64 geometry of cmi_path.cuh.  The passes of cmi_dust.cuh wrote every packet (80
// bytes and its status) after each walk and returned to the host after each
// generation; a warp there also waited for its longest packet.
//
// Lanes whose walk has ended wait until kDustRefill do: their draws and the series of
// the logarithm and the exponential cost several hundred instructions, one copy of
// which, out of line, serves every kind of lane (a copy each overflowed the
// instruction cache: 12.7 ms for 10.0 below).
//
// Bound by the two opacity loads of a crossing (L1 at 80% of its throughput) and by
// instruction issue (60% of slots, 15 of 32 lanes).  B200, one call, unit sphere with
// clumps, the passes against this kernel: 128^3, 4e6 packets, albedo 0.5 26.6 -> 10.0
// ms; 32^3, 1e6 2.85 -> 1.27 ms; 90^3, 1e4, albedo 0.8 2.23 -> 0.55 ms.
#pragma once

#include "cmi_dust.cuh"
#include "cmi_path.cuh"

namespace cmi {

struct DustPathParams {
  PathParams path;         // geo (the instance's), subs, nH, xH, table
  uint32_t n;              // source packets
  uint32_t *next;          // packets claimed
  uint64_t seed;
  uint32_t instance, iteration;
  uint32_t src_sub;        // of the instance
  double src[3];
  double albedo;
  double x0, wx, y0, wy;   // box of the image
  int32_t npx, npy;
  double *image;
  // [0] crossings, [1] transits, [2] walk-bound hits, [3] absorbed, [4] escaped,
  // [5] scattered, [6] off the image, [7] generations
  unsigned long long *counters;
};

// what a lane's packet is beyond its walk
struct DustLanes {
  double weight[32], depth[32];
  double at[3][32];        // last scattering: position, subgrid
  uint32_t ci[3][32], sub[32];
  uint32_t id[32], gen[32], type[32];
};

using DustWalk = PathF<false, false, false>;
constexpr uint32_t kDustMaxGenerations = 4096u;
// lanes whose walk has ended before the warp turns to them (B200, 128^3 / 32^3 above:
// 10 -> 11.1 / 1.66 ms, 16 -> 10.5 / 1.45, 24 -> 11.4 / 1.34, with 6 CTAs per SM)
constexpr uint32_t kDustRefill = 16u;
// lanes at a subgrid face, likewise (8 / 12 / 16 / 20: 9932 / 9735 / 9680 / 9685 us)
constexpr uint32_t kDustTransit = 16u;

__device__ __forceinline__ void dust_direct(const DustPathParams &prm, DustWalk &w,
                                            const DevGeo &g, const double dir[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) w.direction(g, a, dir[a], DustWalk::inverse(g, a, dir[a]));
}

// out of line: inlined, the series and draws overflow the instruction cache
__device__ __noinline__ double dust_exp_call(double x) { return dust_exp(x); }
__device__ __noinline__ double dust_neg_log_call(double u) { return dust_neg_log(u); }
__device__ __noinline__ void dust_direction_call(const DustPathParams &prm, uint32_t id,
                                                 uint32_t gen, uint32_t purpose, double dir[3],
                                                 uint32_t *w0, uint32_t *w3) {
  dust_direction(prm.seed, prm.instance, prm.iteration, id, gen, purpose, dir, w0, w3);
}

template <int kMinBlocks>
__global__ void __launch_bounds__(kPathThreads, kMinBlocks)
    k_dust_path(const __grid_constant__ DustPathParams prm) {
  extern __shared__ __align__(16) unsigned char path_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PathShared &sh = reinterpret_cast<PathShared *>(path_smem)[warp];
  DustLanes &dl =
      reinterpret_cast<DustLanes *>(path_smem + sizeof(PathShared) * kPathWarps)[warp];
  double *table = reinterpret_cast<double *>(path_smem + (sizeof(PathShared) + sizeof(DustLanes)) *
                                                             kPathWarps) +
                  (size_t)warp * prm.path.table;
  const uint32_t tab = smem_addr(table);
  for (int i = lane; i < (int)(sizeof(DevGeo) / 4); i += 32)
    reinterpret_cast<uint32_t *>(&sh.geo)[i] =
        reinterpret_cast<const uint32_t *>(prm.path.geo)[i];
  if (lane == 0) sh.job = sh.job_end = sh.q_at = sh.q_n = sh.exhausted = 0u;
  __syncwarp();
  path_table(table, sh, prm.path.subs, 0u, lane);
  __syncwarp();
  if (lane == 0) {
    sh.geo.sigma = 1.;  // the cross section of the dust packets
    DustWalk at;
    at.at_position(prm.path, sh, tab, prm.src, prm.src_sub);
  }
  __syncwarp();
  const double never = __longlong_as_double(0x7ff0000000000000ll);
  DustWalk w;
  w.steps = 0;
  int status = kPathFree;
  uint32_t cross = 0, trans = 0, bound = 0, absorbed = 0, escaped = 0, scattered = 0, off = 0,
           most = 0;

  for (;;) {
    // walks that have ended; kDrop: left the box (or the visits ran out)
    const unsigned done = __ballot_sync(kFull, status != kRun);
    uint32_t waiting = (uint32_t)__popc(done);
    if (waiting >= kDustRefill || done == kFull) {
      const bool stopped = status == kAbsorbed;
      if (stopped || status == kDrop) {
        const uint32_t id = dl.id[lane], type = dl.type[lane];
        const bool tau = !stopped && type == kDustTau, peel = !stopped && type == kDustPeeloff;
        const bool left = sh.again[lane] != 0u;  // through the box's edge
        uint32_t gen = dl.gen[lane];
        double q[3], dir[3], e = 0., u = 0.;
        bool on = tau;  // another walk follows
        if (stopped) {
          w.template absorb<true>(prm.path, sh.geo);
          cross += (uint32_t)w.steps;
          ++trans;
          ++gen;
        }
        // one copy of the costly draws and series for all kinds of lanes
        if (tau || peel) e = dust_exp_call(-dl.depth[lane]);
        if (!tau && (stopped || (peel && gen < kDustMaxGenerations))) {
          uint32_t w0 = 0, w3 = 0;
          dust_direction_call(prm, id, gen, kDustScatter, dir, &w0, &w3);
          u = dust_uniform(w3);
          on = peel || dust_uniform(w0) < prm.albedo;
        }
        if (tau) {  // forced first scattering: target depth within tau0
          uint32_t v[4];
          dust_words(prm.seed, prm.instance, prm.iteration, id, 0u, kDustRelaunch, 0u, v);
          const double weight = 1. - e;
          dl.weight[lane] = weight;
          u = 1. - dust_uniform(v[0]) * weight;
        } else if (peel) {
          if (left) {  // into the pixel under its exit point
            const double fx = ((w.pos[0] - prm.x0) / prm.wx) * (double)prm.npx;
            const double fy = ((w.pos[1] - prm.y0) / prm.wy) * (double)prm.npy;
            if (!(fx >= 0. && fx < (double)prm.npx && fy >= 0. && fy < (double)prm.npy))
              ++off;
            else
              atomicAdd(&prm.image[(size_t)(int)fx * prm.npy + (int)fy], dl.weight[lane] * e);
          }
        } else if (stopped) {
          if (on) {
            ++scattered;
            most = max(most, gen);
            dl.gen[lane] = gen;
            dl.weight[lane] = dl.weight[lane] * 0.25 * 0.318309886183790671538;  // 1 / (4 pi)
          } else {
            ++absorbed;
          }
        } else if (left) {
          ++escaped;
        }
        if (on) {
          dl.type[lane] = stopped ? kDustPeeloff : kDustDirect;
          dl.depth[lane] = 0.;
          sh.visits[lane] = 1u;
          if (stopped) {  // the peel-off copy along +z from here
            dir[0] = dir[1] = 0.;
            dir[2] = 1.;
            dl.sub[lane] = sh.sub[lane];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
              const uint32_t ci = sh.ci[a][lane];
              q[a] = __dadd_rn(w.pos[a], table_at(ci));
              dl.at[a][lane] = q[a];
              dl.ci[a][lane] = ci;
            }
            w.depth(never);
          } else {
            w.depth(dust_neg_log_call(u));
          }
          if (tau) {  // from the source again, in the same direction
            status = w.start(prm.path, sh, lane, tab);
          } else {
            if (peel) {  // on from the last scattering
              sh.sub[lane] = dl.sub[lane];
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                q[a] = dl.at[a][lane];
                sh.ci[a][lane] = dl.ci[a][lane];
              }
            }
            dust_direct(prm, w, sh.geo, dir);
            status = w.reenter(prm.path, sh, lane, tab, q, 0u);
          }
        } else {
          status = kPathFree;
        }
      }
      const unsigned idle = __ballot_sync(kFull, status == kPathFree);
      if (sh.exhausted) {
        if (idle == kFull) break;
      } else if (idle != 0u) {
        if (sh.q_at == sh.q_n) {  // the next packets of the warp
          uint32_t j0 = sh.job, j1 = sh.job_end;
          __syncwarp();
          if (j0 == j1) {
            if (lane == 0) {
              const uint32_t taken = *(volatile uint32_t *)prm.next;
              const uint32_t left = prm.n > taken ? prm.n - taken : 0u;
              const uint32_t jn =
                  min(256u, max(32u, (left / (2u * gridDim.x * kPathWarps)) & ~31u));
              j0 = atomicAdd(prm.next, jn);
              j1 = j0 + jn;
            }
            j0 = __shfl_sync(kFull, j0, 0);
            j1 = min(prm.n, __shfl_sync(kFull, j1, 0));
          }
          const uint32_t n = j0 < j1 ? min(32u, j1 - j0) : 0u;
          if ((uint32_t)lane < n) {
            double dir[3];
            uint32_t w0, w3;
            dust_direction_call(prm, j0 + (uint32_t)lane, 0u, kDustEmit, dir, &w0, &w3);
            for (int a = 0; a < 3; ++a) {
              sh.q_dir[a][lane] = dir[a];
              sh.q_inv[a][lane] = DustWalk::inverse(sh.geo, a, dir[a]);
            }
          }
          if (lane == 0) {
            sh.src_begin = j0;  // id of the queue's first packet
            sh.job = j0 + n;
            sh.job_end = n ? j1 : j0;
            sh.q_at = 0u;
            sh.q_n = n;
            sh.exhausted = n ? 0u : 1u;
          }
          __syncwarp();
        }
        const uint32_t q_at = sh.q_at, q_n = sh.q_n;
        const uint32_t r = q_at + (uint32_t)__popc(idle & ((1u << lane) - 1u));
        if (status == kPathFree && r < q_n) {
          for (int a = 0; a < 3; ++a) w.direction(sh.geo, a, sh.q_dir[a][r], sh.q_inv[a][r]);
          w.depth(never);
          dl.id[lane] = sh.src_begin + r;
          dl.gen[lane] = 0u;
          dl.type[lane] = kDustTau;
          dl.depth[lane] = 0.;
          sh.visits[lane] = 1u;
          status = w.start(prm.path, sh, lane, tab);
        }
        __syncwarp();
        if (lane == 0) sh.q_at = min(q_n, q_at + (uint32_t)__popc(idle));
        __syncwarp();
        if (sh.exhausted && __all_sync(kFull, status == kPathFree)) break;
      }
      waiting = (uint32_t)__popc(__ballot_sync(kFull, status != kRun && status != kExited));
    }
    // crossings, until enough more lanes wait (half of those left when they are few)
    const uint32_t enough =
        min(32u, waiting + max(1u, min(kDustTransit, (33u - waiting) / 2u)));
    bool over = true;
#pragma unroll 1
    for (int u = 0; u < kPathStretch; ++u) {
      if (status == kRun) status = w.step(prm.path, sh.geo, tab);
      if ((uint32_t)__popc(__ballot_sync(kFull, status != kRun)) >= enough) {
        over = false;
        break;
      }
    }
    if (over && status == kRun && w.steps > sh.geo.n[0] + sh.geo.n[1] + sh.geo.n[2] + 3) {
      ++bound;
      sh.again[lane] = 0u;
      status = kPathFree;
    }
    // lanes at a subgrid face
    if (status == kExited) {
      cross += (uint32_t)w.steps;
      ++trans;
      dl.depth[lane] = __dadd_rn(dl.depth[lane], w.done);
      const double ex = __dadd_rn(w.pos[0], table_at(sh.ci[0][lane]));
      const double ey = __dadd_rn(w.pos[1], table_at(sh.ci[1][lane]));
      status = w.transit(prm.path, sh, lane, tab);
      if (status == kPathFree) {  // out of the box
        w.pos[0] = ex;
        w.pos[1] = ey;
        sh.again[lane] = 1u;
        status = kDrop;
      } else if (++sh.visits[lane] > (uint32_t)kDustMaxVisits) {
        sh.again[lane] = 0u;
        status = kDrop;
      }
    }
  }
  const unsigned long long sums[7] = {cross, trans, bound, absorbed, escaped, scattered, off};
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    const unsigned long long v = warp_sum64(sums[k]);
    if (lane == 0 && v) atomicAdd(&prm.counters[k], v);
  }
  most = __reduce_max_sync(kFull, most);
  if (lane == 0 && most) atomicMax(&prm.counters[7], (unsigned long long)most);
}

}  // namespace cmi
