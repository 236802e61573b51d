// Whole-path transport: one lane follows one packet from its source through
// every subgrid it crosses to absorption or out of the box.
//
// The reference moves packets from subgrid to subgrid through buffers
// (do_photon_traversal, testDensitySubGrid_omp.cpp:607-666), and so does the
// wavefront of cmi_kernels.cuh.  On the workloads a packet crosses 7 to 13 cells per
// subgrid, so sorting, staging and appending it at every visit cost more than the
// crossings.  Here the packet stays in the lane's registers and only re-anchors at a
// subgrid face, with the reference's arithmetic (pos + anchor of the subgrid it
// leaves, - anchor of the one it enters, DensitySubGrid.hpp:1307-1309, 1186-1219):
// emission, walk and reemission are one launch, and no packet is ever written.
//
// * Opacity comes from the field through L1 and L2.  Where a packet goes does not
//   hang on it, so its load has a whole crossing to come back (kDefer).
// * Path lengths go to 64-bit tallies in L2 by reductions without return (fixed point,
//   the same units as the shared-memory tallies; FP64 in the FP64 walk).  The L2 takes
//   1.9e11 scattered reductions a second, but one cache line only 1.7e9, and the cells
//   around a source see every packet: subgrids within kHotCells cells of a source have
//   several copies of their tally, a warp adds to one, and the balance sums them.  The
//   packets are also cut into shares, and CTAs start on different ones, so that
//   several sources are worked on at once.
// * The cell faces and subgrid anchors of an instance sit in a shared-memory table;
//   the entry beyond the last face is a guard (a NaN), so leaving a subgrid is seen in
//   the face that is loaded anyway.
// * Lanes at a face, done and free ones wait until several do (kTransit and kRefill of
//   the lane state); packets are emitted 32 at a time into a queue.
//
// Bound by instruction issue and lane divergence (log-normal 128^3, mixed, 4e6 packets:
// 63% of issue slots, 19 of 32 lanes, L1 73% of peak, L2 48% and 95% in its busiest
// slice).  Against the wavefront, us per iteration: 32^3, 2e4 packets 214 -> 57;
// stromgren 64^3, 1e6 913 -> 329; log-normal 128^3, 1e7 3800 -> 2005; 256^3, 1e8
// 79100 -> 54300; 12 uneven instances 7170 -> 4200; FP64 walk, 64^3, 1e6 1561 -> 280.
#pragma once

#include "cmi_kernels.cuh"

namespace cmi {

// Geometry of one instance, as the path kernel reads it.
struct alignas(16) DevGeo {
  double cs[3], inv_cs[3];
  double sigma, reemission;
  float cs_f[3], inv_cs_f[3];
  int32_t n[3];            // cells per subgrid and axis
  int32_t ns[3];           // subgrids per axis
  int32_t stride[3];       // cells: to the next cell along an axis
  int32_t sub_stride[3];   // subgrids: to the next subgrid along an axis
  int32_t jump[3];         // cells: from just outside a subgrid to the next one's first
  uint32_t padded;         // cells from one subgrid's fields to the next's
  uint32_t first_cell;     // of the instance's first subgrid
  uint32_t first_sub;
  float tally_scale;       // 2^22 / lref
  int32_t face_off[3];     // table offsets: faces of axis a, a guard before and behind
  int32_t anchor_off[3];   // subgrid anchors of axis a, a guard before and behind
  int32_t inf_off;         // an entry +inf: the face ahead on an axis without motion
  int32_t table;           // doubles in the table
};

struct PathParams {
  const DevGeo *geo;
  const DevSubgrid *subs;
  const DevInstance *inst;
  const DevSource *src;
  int nsrc_total;
  const uint64_t *src_first;
  RoundState *st;
  DevStats *stats;
  const float *kappa;             // FP32 and mixed
  const double *nH, *xH;          // FP64
  const double2 *nx;              // dust: the same, side by side
  unsigned long long *tally;      // fixed-point path lengths (lref / 2^22); FP64: doubles
  const uint32_t *hot;            // per subgrid: first cell of its tally copies, 0: none
  uint32_t copies;                // tally copies of a subgrid next to a source
  int32_t table;                  // largest table (doubles)
  uint32_t round_cap;             // most subgrid visits of one packet
};

constexpr int kPathFree = 4;      // lane status beyond WalkStatus and kDrop
constexpr int kPathStretch = 32;  // looks between two checks of the step bound
// crossings between two looks at the warp (B200, us per iteration at 1 / 2 / 3: stromgren 64^3
// 349 / 340 / 354, log-normal 128^3 2136 / 2083 / 2151, reemission 687 / 649 / 662)
constexpr int kPathLook = 2;
// shared memory a CTA may take: six CTAs (the FP64-geometry build) fit an SM and leave
// its L1 most of the rest
constexpr size_t kPathSmemMost = 32768;
constexpr uint32_t kGuardHi = 0x7ff80000u;  // high word of the guard (a NaN)

// What the turn at a subgrid face needs of an axis.
struct alignas(16) PathAxis {
  double inv_cs;
  uint32_t low;   // address in the table of the face behind cell 0, 12 bytes on
  uint32_t span;  // cells of a subgrid
  int32_t sub_stride, jump;
};

// Per-warp shared memory: the instance's geometry, the state of a packet at the
// current source, a queue of up to 32 emitted packets, then the table.
struct PathShared {
  DevGeo geo;
  PathAxis axis[3];
  double q_dir[3][32], q_inv[3][32], q_tau[32];
  double src_pos[3];       // relative to the subgrid's anchor (FP32: in cells)
  int32_t src_idx[3];
  uint32_t src_c[3];
  uint32_t src_sub, src_cell, src_toff, src_out;
  uint32_t copy_base;      // tally word of a copied cell: field cell + first copied cell + this
  // per lane, what only the turn at a subgrid face needs
  uint32_t ci[3][32];      // subgrid anchors (FP64 geometry: table addresses; FP32: coordinates)
  uint32_t sub[32];        // subgrid of the instance
  uint32_t visits[32];     // subgrids entered
  uint32_t again[32];      // reemissions in this subgrid
  // the warp's work: claimed packets, end of the current source's, queue
  uint64_t inst_first;     // first packet of the current instance
  uint32_t inst, fresh, share, job, job_end, src_begin, src_end, q_at, q_n, exhausted;
  // per lane: packets absorbed, escaped and re-emitted, most subgrids entered
  uint32_t absorbed[32], escaped[32], reemitted[32], most[32];
};

// The face and anchor table of the warp's instance, and what follows from it for a warp
// that adds to tally copy `copy`; all lanes.
__device__ __forceinline__ void path_table(double *tab, PathShared &sh, const DevSubgrid *subs,
                                           uint32_t copy, int lane) {
  const DevGeo &g = sh.geo;
  if (lane < 3)
    sh.axis[lane] = {g.inv_cs[lane], smem_addr(tab) + 12u + 8u * (uint32_t)g.face_off[lane],
                     (uint32_t)g.n[lane], g.sub_stride[lane], g.jump[lane]};
  if (lane == 0) sh.copy_base = copy * g.padded - g.first_cell;
  const double guard = __hiloint2double((int)kGuardHi, 0);
  if (lane == 0) tab[g.inf_off] = __longlong_as_double(0x7ff0000000000000ll);
  for (int a = 0; a < 3; ++a) {
    for (int i = lane; i < g.n[a] + 3; i += 32)
      tab[g.face_off[a] + i] =
          (i == 0 || i == g.n[a] + 2) ? guard : __dmul_rn((double)(i - 1), g.cs[a]);
    for (int i = lane; i < g.ns[a] + 2; i += 32)
      tab[g.anchor_off[a] + i] =
          (i == 0 || i == g.ns[a] + 1)
              ? guard
              : subs[g.first_sub + (uint32_t)((i - 1) * g.sub_stride[a])].anchor[a];
  }
}

// offset of this warp's tally copy of a subgrid (0: no copies, the field itself)
__device__ __forceinline__ uint32_t tally_offset(const PathParams &prm, const PathShared &sh,
                                                 uint32_t sub) {
  const uint32_t hot = __ldg(prm.hot + sh.geo.first_sub + sub);
  return hot ? hot + (sh.copy_base - sub * sh.geo.padded) : 0u;
}

__device__ __forceinline__ double table_at(uint32_t byte) {
  double v;
  asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(byte));
  return v;
}

// If the axis with path length l is crossed (l == lmin): next face and cell.
// Predicated adds; written as C++ they become a branch per axis, and the lanes of a
// warp cross different axes.
__device__ __forceinline__ void cross_axis(double l, double lmin, double &pos, double moved,
                                           double &face, uint32_t &fi, int fstep,
                                           uint32_t &cell, int cstep) {
  asm("{\n\t.reg .pred p;\n\t"
      "setp.eq.f64 p, %4, %5;\n\t"
      "selp.f64 %0, %3, %6, p;\n\t"
      "@p add.s32 %1, %1, %7;\n\t"
      "@p ld.shared.f64 %3, [%1];\n\t"
      "@p add.s32 %2, %2, %8;\n\t}"
      : "=d"(pos), "+r"(fi), "+r"(cell), "+d"(face)
      : "d"(l), "d"(lmin), "d"(moved), "r"(fstep), "r"(cstep));
}
__device__ __forceinline__ void cross_axis(float l, float lmin, float &p, float moved,
                                           float &face, float fstep, float fexit, uint32_t &ex,
                                           uint32_t bit, uint32_t &cell, int cstep) {
  asm("{\n\t.reg .pred p, q;\n\t"
      "setp.eq.f32 p, %4, %5;\n\t"
      "setp.eq.and.f32 q, %1, %8, p;\n\t"
      "selp.f32 %0, %1, %6, p;\n\t"
      "@p add.rn.f32 %1, %1, %7;\n\t"
      "@q or.b32 %2, %2, %9;\n\t"
      "@p add.s32 %3, %3, %10;\n\t}"
      : "=f"(p), "+f"(face), "+r"(ex), "+r"(cell)
      : "f"(l), "f"(lmin), "f"(moved), "f"(fstep), "f"(fexit), "r"(bit), "r"(cstep));
}
// tally += v unless v is zero
__device__ __forceinline__ void add_tally(unsigned long long *tally, uint32_t v) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 w;\n\t"
               "setp.ne.u32 p, %1, 0;\n\t"
               "cvt.u64.u32 w, %1;\n\t"
               "@p red.global.add.u64 [%0], w;\n\t}" ::"l"(tally), "r"(v)
               : "memory");
}
__device__ __forceinline__ void add_tally(unsigned long long *tally, double v) {
  asm volatile("{\n\t.reg .pred p;\n\t"
               "setp.neu.f64 p, %1, 0d0000000000000000;\n\t"
               "@p red.global.add.f64 [%0], %1;\n\t}" ::"l"(tally), "d"(v)
               : "memory");
}

// exit code of a crossing: the axes in `out` with their sides (bit 3 + a: high)
__device__ __forceinline__ uint32_t exit_sides(uint32_t out, const float sg[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) out |= ((out >> a) & 1u) && sg[a] > 0 ? 8u << a : 0u;
  return out;
}

// Lane state of the FP64 geometry walks (mixed and FP64): the operations of
// WalkM / Walk64, with the cell as an index into the whole field and the face
// ahead read from the instance's table; the entry beyond the last face is a
// guard whose high word marks the exit.
template <bool kMixed, bool kDefer, bool kTally = true>
struct PathF {
  using Real = typename std::conditional<kMixed, float, double>::type;
  // A warp turns to its lanes at subgrid faces once kTransit more lanes wait than it
  // could not help, and absorbs and refills once kRefill lanes do not walk.  B200, us per
  // shoot with 12 and 12 / 16 and 6: stromgren 64^3, 1e6 packets 374 / 361, log-normal
  // 128^3, 1e7 1664 / 1630, 12 uneven instances 3340 / 3260; with reemission, where
  // more lanes wait for the draws, 644 / 697.
  static constexpr uint32_t kTransit = kDefer ? 16 : 12, kRefill = kDefer ? 6 : 12;
  double pos[3], d[3], inv[3], face[3];
  uint32_t fi[3];       // shared-memory address of the face ahead
  int sg[3];            // to the next face in bytes: +8 / -8, 0: no motion along the axis
  int cst[3];           // to the next cell
  float scale;          // tally units per metre
  uint32_t cell;        // in the whole field
  uint32_t toff;        // tally word of a cell: cell + toff
  Real done, target;
  int steps;
  uint32_t ex;          // exit: bit a axis a, bit 3 + a through the high face
  // kDefer: the last crossing, its opacity (FP64: n_H, x_H) still on the way; else the
  // opacity of the present cell
  double last;
  Real lk, lx;
  uint32_t lat;

  static __device__ __forceinline__ double inverse(const DevGeo &, int, double d) {
    return d > 0. || d < 0. ? __drcp_rn(d) : __longlong_as_double(0x7ff0000000000000ll);
  }
  __device__ __forceinline__ void direction(const DevGeo &g, int a, double dir, double i) {
    d[a] = dir;
    inv[a] = i;
    sg[a] = dir > 0. ? 8 : (dir < 0. ? -8 : 0);
    cst[a] = dir > 0. ? g.stride[a] : -g.stride[a];
    scale = g.tally_scale;
  }
  __device__ __forceinline__ void depth(double tau) {
    if (kMixed) target = (Real)tau32(tau); else target = (Real)tau;
    done = (Real)0;
    steps = 0;
    clear();
  }
  __device__ __forceinline__ void clear() {  // no crossing open
    last = 0.;
    lk = lx = (Real)0;
    lat = 0u;
  }

  // the face ahead of cell idx (tab: shared-memory address of the table)
  __device__ __forceinline__ void ahead(const DevGeo &g, uint32_t tab, int a, int idx) {
    fi[a] = tab + 8u * (uint32_t)(sg[a] ? g.face_off[a] + 1 + idx + (sg[a] > 0 ? 1 : 0)
                                        : g.inf_off);
    face[a] = table_at(fi[a]);
  }

  // Entry INSIDE the subgrid (ci, sub) at the absolute position q: the start indices
  // (get_start_index, DensitySubGrid.hpp:428-469) and the axes outside of it.
  __device__ __forceinline__ uint32_t locate(const DevGeo &g, const double anchor[3],
                                             const double q[3], uint32_t in, int idx[3]) {
    uint32_t out = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      pos[a] = __dsub_rn(q[a], anchor[a]);
      idx[a] = __double2int_rz(__dmul_rn(pos[a], g.inv_cs[a]));
      if ((in >> a) & 1u) idx[a] = ((in >> (3 + a)) & 1u) ? 0 : g.n[a] - 1;
      if (idx[a] < 0) out |= 1u << a;
      if (idx[a] >= g.n[a]) out |= 9u << a;
    }
    return out;
  }
  __device__ __forceinline__ int settle(const PathParams &prm, const PathShared &sh, int lane,
                                        uint32_t tab, const int idx[3], uint32_t out) {
    const DevGeo &g = sh.geo;
    const uint32_t sub = sh.sub[lane];
    if (!((Real)0 < target)) return kAbsorbed;
    ex = out;
    if (out) return kExited;
    cell = g.first_cell + sub * g.padded +
           (uint32_t)(idx[0] * g.stride[0] + idx[1] * g.stride[1] + idx[2]);
    toff = kTally ? tally_offset(prm, sh, sub) : 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) ahead(g, tab, a, idx[a]);
    if (!kDefer) opacity(prm, lk, lx);
    return kRun;
  }

  // the state of a packet at the source, shared by the warp
  __device__ __forceinline__ void at_source(const PathParams &prm, PathShared &sh,
                                            uint32_t tab, const DevSource &S) {
    at_position(prm, sh, tab, S.position, S.subgrid - sh.geo.first_sub);
  }
  __device__ __forceinline__ void at_position(const PathParams &prm, PathShared &sh, uint32_t tab,
                                              const double position[3], uint32_t sub) {
    const DevGeo &g = sh.geo;
    int idx[3];
    double anchor[3];
    for (int a = 0; a < 3; ++a) {
      sh.src_c[a] = tab + 8u * (uint32_t)(g.anchor_off[a] + 1 +
                                          (int)(sub / (uint32_t)g.sub_stride[a]) % g.ns[a]);
      anchor[a] = table_at(sh.src_c[a]);
    }
    const uint32_t out = locate(g, anchor, position, 0u, idx);
    for (int a = 0; a < 3; ++a) {
      sh.src_pos[a] = pos[a];
      sh.src_idx[a] = idx[a];
    }
    sh.src_sub = sub;
    sh.src_cell = g.first_cell + sub * g.padded +
                  (uint32_t)(idx[0] * g.stride[0] + idx[1] * g.stride[1] + idx[2]);
    sh.src_toff = kTally ? tally_offset(prm, sh, sub) : 0u;
    sh.src_out = out;
  }
  __device__ __forceinline__ int start(const PathParams &prm, PathShared &sh, int lane,
                                       uint32_t tab) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      pos[a] = sh.src_pos[a];
      sh.ci[a][lane] = sh.src_c[a];
      if (!sh.src_out) ahead(sh.geo, tab, a, sh.src_idx[a]);
    }
    sh.sub[lane] = sh.src_sub;
    cell = sh.src_cell;
    toff = sh.src_toff;
    if (!((Real)0 < target)) return kAbsorbed;
    ex = sh.src_out;
    if (ex) return kExited;
    if (!kDefer) opacity(prm, lk, lx);
    return kRun;
  }

  // Entry into the subgrid on the other side of the faces in `in` (bit a: axis a, bit
  // 3 + a: upwards) at the absolute position q, with every index found afresh.
  __device__ __forceinline__ int reenter(const PathParams &prm, PathShared &sh,
                                         int lane, uint32_t tab, const double q[3], uint32_t in) {
    double anchor[3];
    int idx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) anchor[a] = table_at(sh.ci[a][lane]);
    const uint32_t out = locate(sh.geo, anchor, q, in, idx);
    return settle(prm, sh, lane, tab, idx, out);
  }

  // a packet found outside the subgrid's index range at entry moves on at once
  __device__ __forceinline__ int pass_on(const PathParams &prm, PathShared &sh,
                                         int lane, uint32_t tab) {
    const DevGeo &g = sh.geo;
    double q[3];
    bool outside = false;
    for (int a = 0; a < 3; ++a) {
      const uint32_t ci = sh.ci[a][lane];
      q[a] = __dadd_rn(pos[a], table_at(ci));
      if (!((ex >> a) & 1u)) continue;
      const bool up = (ex >> (3 + a)) & 1u;
      sh.ci[a][lane] = ci + (up ? 8u : (uint32_t)-8);
      sh.sub[lane] += (uint32_t)(up ? g.sub_stride[a] : -g.sub_stride[a]);
      outside = outside || (uint32_t)__double2hiint(table_at(sh.ci[a][lane])) == kGuardHi;
    }
    if (outside) return kPathFree;
    return reenter(prm, sh, lane, tab, q, ex);
  }

  // Across the face(s) it left by into the next subgrid: pos + anchor of this one -
  // anchor of the next, remaining depth, start index.  kPathFree: out of the box.
  __device__ __forceinline__ int transit(const PathParams &prm, PathShared &sh,
                                         int lane, uint32_t tab) {
    target = kMixed ? (Real)__fsub_rn((float)target, (float)done)
                    : (Real)__dsub_rn((double)target, (double)done);
    done = (Real)0;
    if (steps == 0) return pass_on(prm, sh, lane, tab);
    steps = 0;
    double q[3], anchor[3];
    bool outside = false, same = true;
    uint32_t sub = sh.sub[lane], ci[3];
    int hop[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ci[a] = sh.ci[a][lane];
      q[a] = __dadd_rn(pos[a], table_at(ci[a]));
      hop[a] = (uint32_t)__double2hiint(face[a]) == kGuardHi ? sg[a] : 0;  // 8 bytes up or down
      ci[a] += (uint32_t)hop[a];
      anchor[a] = table_at(ci[a]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const PathAxis &A = sh.axis[a];
      sh.ci[a][lane] = ci[a];
      const int one = hop[a] >> 3;
      sub += (uint32_t)(one * A.sub_stride);
      cell += (uint32_t)(one * A.jump);
      fi[a] -= (uint32_t)hop[a] * A.span;
      outside = outside || (uint32_t)__double2hiint(anchor[a]) == kGuardHi;
      pos[a] = __dsub_rn(q[a], anchor[a]);
      // the start index of an axis it did not leave by is the present one but for
      // rounding; an axis it left by starts at the first cell behind the face.  The low
      // word of the sum is the index rounded down; below 0, where truncation
      // differs, it matches no cell and the entry is found afresh.
      const int idx = __double2loint(__dadd_rd(__dmul_rn(pos[a], A.inv_cs), 6755399441055744.));
      same = same && (hop[a] != 0 ||
                      fi[a] - (uint32_t)(sg[a] >> 1) == A.low + 8u * (uint32_t)idx);
    }
    if (outside) return kPathFree;
    sh.sub[lane] = sub;
    if (same) {
      if (kTally) toff = tally_offset(prm, sh, sub);
      // the guard on the axes it left by: read again
#pragma unroll
      for (int a = 0; a < 3; ++a) face[a] = table_at(fi[a]);
      if (!kDefer) opacity(prm, lk, lx);
      return (Real)0 < target ? kRun : kAbsorbed;
    }
    uint32_t in = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if ((uint32_t)__double2hiint(face[a]) == kGuardHi) in |= (sg[a] > 0 ? 9u : 1u) << a;
    return reenter(prm, sh, lane, tab, q, in);
  }

  // back to the absorption point with a new direction and depth
  __device__ __forceinline__ int reemit(const PathParams &prm, const PathShared &sh, int lane,
                                        uint32_t tab, const double rd[4]) {
    const DevGeo &g = sh.geo;
    double q[3], anchor[3];
    int idx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      anchor[a] = table_at(sh.ci[a][lane]);
      q[a] = __dadd_rn(pos[a], anchor[a]);
      direction(g, a, rd[a], inverse(g, a, rd[a]));
    }
    depth(rd[3]);
    const uint32_t out = locate(g, anchor, q, 0u, idx);
    return settle(prm, sh, lane, tab, idx, out);
  }
  __device__ __forceinline__ void reemit_counter(const PathShared &sh, int lane, uint32_t tab,
                                                 uint32_t h[3]) const {
#pragma unroll
    for (int a = 0; a < 3; ++a) h[a] = reemit_hash(__dadd_rn(pos[a], table_at(sh.ci[a][lane])));
  }

  // The optical depth of a crossing of length lmin in a cell of opacity k (FP64: n_H
  // and x_H) and its path length into the tally; false: the target depth lies in it
  // and nothing was done.
  __device__ __forceinline__ bool pass(const PathParams &prm, const DevGeo &g, double lmin, Real k,
                                       Real x, uint32_t at) {
    if (kMixed) {
      const float lf = __double2float_rn(lmin);
      const Real after = (Real)__fadd_rn((float)done, __fmul_rn(lf, (float)k));
      if (after >= target) return false;
      if (kTally) add_tally(prm.tally + at, Tally32<3>::fixed(lf, scale));
      done = after;
    } else {
      const double ls = __dmul_rn(lmin, g.sigma);
      const Real after = (Real)__dadd_rn((double)done, __dmul_rn(__dmul_rn(ls, (double)k), (double)x));
      if (after >= target) return false;
      if (kTally) add_tally(prm.tally + at, ls);
      done = after;
    }
    return true;
  }
  // the same for the part of the crossing up to the target depth; its length
  __device__ __forceinline__ double stop(const PathParams &prm, const DevGeo &g, double lmin,
                                         Real k, Real x, uint32_t at) {
    if (kMixed) {
      const float tau = __fmul_rn(__double2float_rn(lmin), (float)k);
      const float frac = fminf(__fdiv_rn(__fsub_rn((float)target, (float)done), tau), 1.f);
      lmin = __dmul_rn(lmin, (double)frac);
      if (kTally)
        add_tally(prm.tally + at, Tally32<3>::fixed(__double2float_rn(lmin), scale));
    } else {
      const double tau = __dmul_rn(__dmul_rn(__dmul_rn(lmin, g.sigma), (double)k), (double)x);
      const double after = __dadd_rn((double)done, tau);
      const double correction = __ddiv_rn(__dsub_rn(after, (double)target), tau);
      lmin = __dmul_rn(lmin, __dsub_rn(1., correction));
      if (kTally) add_tally(prm.tally + at, __dmul_rn(lmin, g.sigma));
    }
    return lmin;
  }
  __device__ __forceinline__ void opacity(const PathParams &prm, Real &k, Real &x) const {
    if (kMixed) {
      k = (Real)__ldg(prm.kappa + cell);
      x = (Real)0;
    } else if (kTally) {
      k = (Real)__ldg(prm.nH + cell);
      x = (Real)__ldg(prm.xH + cell);
    } else {
      const double2 v = __ldg(prm.nx + cell);
      k = (Real)v.x;
      x = (Real)v.y;
    }
  }

  // One crossing (one trip of the loop at DensitySubGrid.hpp:1221-1305).  A packet
  // that stops in a cell is left before it (kAbsorbed): absorb() finishes it.
  // kDefer: where a packet goes does not hang on the opacity until it is absorbed, so
  // the depth of a crossing is added after the geometry of the next one, when its
  // load has had a whole turn to come back.
  __device__ __forceinline__ int step(const PathParams &prm, const DevGeo &g, uint32_t tab) {
    Real k, x;
    if (kDefer) opacity(prm, k, x);
    double l[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) l[a] = __dmul_rn(__dsub_rn(face[a], pos[a]), inv[a]);
    const double lmin = min_ref(l[0], min_ref(l[1], l[2]));
    if (kDefer) {
      if (!pass(prm, g, last, lk, lx, lat)) return kAbsorbed;
      last = lmin;
      lk = k;
      lx = x;
      lat = cell + toff;
    } else {
      if (!pass(prm, g, lmin, lk, lx, cell + toff)) return kAbsorbed;
    }
    ++steps;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      cross_axis(l[a], lmin, pos[a], __dadd_rn(pos[a], __dmul_rn(lmin, d[a])), face[a], fi[a],
                 sg[a], cell, cst[a]);
    // faces are not negative, so their high words order like integers
    const int top = max(__double2hiint(face[0]),
                        max(__double2hiint(face[1]), __double2hiint(face[2])));
    if (top >= (int)kGuardHi) return kExited;
    if (!kDefer) opacity(prm, lk, lx);
    return kRun;
  }

  // at a subgrid face: the depth of the crossing that led there
  __device__ __forceinline__ bool settle_last(const PathParams &prm, const DevGeo &g) {
    if (!kDefer) return true;
    if (!pass(prm, g, last, lk, lx, lat)) return false;
    clear();
    return true;
  }

  // the crossing that step() left: the part of the cell up to the target depth
  template <bool kReemit>
  __device__ __forceinline__ void absorb(const PathParams &prm, const DevGeo &g) {
    static_assert(!(kReemit && kDefer), "reemission needs the position of the absorption");
    if (!((Real)0 < target)) return;  // stopped at entry: no cell crossed
    if constexpr (kDefer) {
      (void)stop(prm, g, last, lk, lx, lat);
    } else {
      double l[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) l[a] = __dmul_rn(__dsub_rn(face[a], pos[a]), inv[a]);
      const double lmin = stop(prm, g, min_ref(l[0], min_ref(l[1], l[2])), lk, lx, cell + toff);
      ++steps;
      if (kReemit) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          pos[a] = (l[a] == lmin) ? face[a] : __dadd_rn(pos[a], __dmul_rn(lmin, d[a]));
      }
    }
  }
};

// Lane state of the FP32 cell-unit walk: Walk32's operations.
template <bool kDefer>
struct Path32 {
  // as in PathF; 96 x 80 x 112, 4e6 packets, us per shoot with 12 and 12 / 16 and 6: 1981 / 2014
  static constexpr uint32_t kTransit = 12, kRefill = 12;
  float p[3], face[3], inv[3], dcs[3];
  float fexit[3];
  float sg[3];          // +1 / -1, 0: no motion along the axis
  int cst[3];
  float scale;
  uint32_t cell, toff;
  float done, target;
  int steps;
  uint32_t ex;
  float last, lk;       // kDefer: the last crossing, its opacity still on the way
  uint32_t lat;

  static __device__ __forceinline__ double inverse(const DevGeo &g, int a, double dir) {
    const float d = (float)dir;
    return (double)(d > 0.f || d < 0.f ? __fmul_rn(g.cs_f[a], __frcp_rn(d))
                                       : __int_as_float(0x7f800000));
  }
  __device__ __forceinline__ void direction(const DevGeo &g, int a, double dir, double i) {
    const float d = (float)dir;
    dcs[a] = __fmul_rn(d, g.inv_cs_f[a]);
    inv[a] = (float)i;
    sg[a] = d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f);
    cst[a] = d > 0.f ? g.stride[a] : -g.stride[a];
    scale = g.tally_scale;
    fexit[a] = d > 0.f ? (float)g.n[a] : 0.f;
  }
  __device__ __forceinline__ void depth(double tau) {
    target = (float)tau;
    done = 0.f;
    steps = 0;
    clear();
  }
  __device__ __forceinline__ void clear() {
    last = lk = 0.f;
    lat = 0u;
  }
  __device__ __forceinline__ void ahead(int a, int idx) {
    face[a] = sg[a] != 0.f ? (float)(sg[a] > 0.f ? idx + 1 : idx) : __int_as_float(0x7f800000);
  }
  __device__ __forceinline__ uint32_t locate(const DevGeo &g, uint32_t in, int idx[3]) {
    uint32_t out = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      idx[a] = __float2int_rz(p[a]);
      if ((in >> a) & 1u) idx[a] = ((in >> (3 + a)) & 1u) ? 0 : g.n[a] - 1;
      if (idx[a] < 0) out |= 1u << a;
      if (idx[a] >= g.n[a]) out |= 9u << a;
    }
    return out;
  }
  __device__ __forceinline__ int settle(const PathParams &prm, const PathShared &sh, int lane,
                                        const int idx[3], uint32_t out) {
    const DevGeo &g = sh.geo;
    const uint32_t sub = sh.sub[lane];
#pragma unroll
    for (int a = 0; a < 3; ++a) ahead(a, idx[a]);
    if (!(0.f < target)) return kAbsorbed;
    ex = out;
    if (out) return kExited;
    cell = g.first_cell + sub * g.padded +
           (uint32_t)(idx[0] * g.stride[0] + idx[1] * g.stride[1] + idx[2]);
    toff = tally_offset(prm, sh, sub);
    return kRun;
  }
  __device__ __forceinline__ void at_source(const PathParams &prm, PathShared &sh,
                                            uint32_t, const DevSource &S) {
    const DevGeo &g = sh.geo;
    const uint32_t sub = S.subgrid - g.first_sub;
    int idx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) p[a] = S.pos_cell[a];
    const uint32_t out = locate(g, 0u, idx);
    for (int a = 0; a < 3; ++a) {
      sh.src_pos[a] = (double)p[a];
      sh.src_idx[a] = idx[a];
      sh.src_c[a] = sub / (uint32_t)g.sub_stride[a] % (uint32_t)g.ns[a];
    }
    sh.src_sub = sub;
    sh.src_cell = g.first_cell + sub * g.padded +
                  (uint32_t)(idx[0] * g.stride[0] + idx[1] * g.stride[1] + idx[2]);
    sh.src_toff = tally_offset(prm, sh, sub);
    sh.src_out = out;
  }
  __device__ __forceinline__ int start(const PathParams &, PathShared &sh, int lane, uint32_t) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      p[a] = (float)sh.src_pos[a];
      sh.ci[a][lane] = sh.src_c[a];
      ahead(a, sh.src_idx[a]);
    }
    sh.sub[lane] = sh.src_sub;
    cell = sh.src_cell;
    toff = sh.src_toff;
    if (!(0.f < target)) return kAbsorbed;
    ex = sh.src_out;
    return ex ? kExited : kRun;
  }
  // the exit coordinate is 0 or n, so re-anchoring is exact
  __device__ __forceinline__ int transit(const PathParams &prm, PathShared &sh, int lane,
                                         uint32_t) {
    const DevGeo &g = sh.geo;
    const bool crossed = steps > 0;
    if (crossed) ex = exit_sides(ex, sg);
    uint32_t sub = sh.sub[lane];
    bool outside = false, same = crossed;
    int idx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const bool off = (ex >> a) & 1u;
      const int up = ((ex >> (3 + a)) & 1u) ? 1 : -1;
      const uint32_t ci = sh.ci[a][lane] + (uint32_t)(off ? up : 0);
      sh.ci[a][lane] = ci;
      sub += off ? (uint32_t)(up * g.sub_stride[a]) : 0u;
      outside = outside || ci >= (uint32_t)g.ns[a];
      p[a] = off ? __fsub_rn(p[a], __int2float_rn(up * g.n[a])) : p[a];
      same = same && (off || sg[a] == 0.f ||
                      truncf(p[a]) == (sg[a] > 0 ? __fsub_rn(face[a], 1.f) : face[a]));
    }
    if (outside) return kPathFree;
    sh.sub[lane] = sub;
    target = __fsub_rn(target, done);
    done = 0.f;
    steps = 0;
    if (same) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const bool off = (ex >> a) & 1u;
        // one cell beyond the face it left by: 1 upwards, n - 1 downwards
        face[a] = off ? (sg[a] > 0 ? 1.f : (float)(g.n[a] - 1)) : face[a];
        cell += off ? (uint32_t)(sg[a] > 0.f ? g.jump[a] : -g.jump[a]) : 0u;
      }
      toff = tally_offset(prm, sh, sub);
      return 0.f < target ? kRun : kAbsorbed;
    }
    const uint32_t out = locate(g, ex, idx);
    return settle(prm, sh, lane, idx, out);
  }
  __device__ __forceinline__ int reemit(const PathParams &prm, const PathShared &sh, int lane,
                                        uint32_t, const double rd[4]) {
    const DevGeo &g = sh.geo;
    int idx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) direction(g, a, rd[a], inverse(g, a, rd[a]));
    depth(rd[3]);
    const uint32_t out = locate(g, 0u, idx);
    return settle(prm, sh, lane, idx, out);
  }
  __device__ __forceinline__ void reemit_counter(const PathShared &sh, int lane, uint32_t,
                                                 uint32_t h[3]) const {
    const uint32_t s = sh.geo.first_sub + sh.sub[lane];
    h[0] = __float_as_uint(p[0]) ^ s;
    h[1] = __float_as_uint(p[1]) ^ (s * 0x9E3779B9u);
    h[2] = __float_as_uint(p[2]);
  }

  __device__ __forceinline__ bool pass(const PathParams &prm, float lmin, float k, uint32_t at) {
    const float after = __fadd_rn(done, __fmul_rn(lmin, k));
    if (after >= target) return false;
    add_tally(prm.tally + at, Tally32<3>::fixed(lmin, scale));
    done = after;
    return true;
  }
  __device__ __forceinline__ float stop(const PathParams &prm, float lmin, float k, uint32_t at) {
    const float tau = __fmul_rn(lmin, k);
    const float corr = __fdiv_rn(__fsub_rn(__fadd_rn(done, tau), target), tau);
    lmin = __fmul_rn(lmin, __fsub_rn(1.f, corr));
    add_tally(prm.tally + at, Tally32<3>::fixed(lmin, scale));
    return lmin;
  }

  __device__ __forceinline__ int step(const PathParams &prm, const DevGeo &, uint32_t) {
    const float k = __ldg(prm.kappa + cell);
    float l[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) l[a] = __fmul_rn(__fsub_rn(face[a], p[a]), inv[a]);
    const float lmin = min_ref(l[0], min_ref(l[1], l[2]));
    if (kDefer) {
      if (!pass(prm, last, lk, lat)) return kAbsorbed;
      last = lmin;
      lk = k;
      lat = cell + toff;
    } else {
      if (!pass(prm, lmin, k, cell + toff)) return kAbsorbed;
    }
    ++steps;
    ex = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      cross_axis(l[a], lmin, p[a], __fmaf_rn(lmin, dcs[a], p[a]), face[a], sg[a], fexit[a], ex,
                 1u << a, cell, cst[a]);
    return ex ? kExited : kRun;
  }

  __device__ __forceinline__ bool settle_last(const PathParams &prm, const DevGeo &) {
    if (!kDefer) return true;
    if (!pass(prm, last, lk, lat)) return false;
    clear();
    return true;
  }

  template <bool kReemit>
  __device__ __forceinline__ void absorb(const PathParams &prm, const DevGeo &) {
    static_assert(!(kReemit && kDefer), "reemission needs the position of the absorption");
    if (!(0.f < target)) return;
    if constexpr (kDefer) {
      (void)stop(prm, last, lk, lat);
    } else {
      float l[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) l[a] = __fmul_rn(__fsub_rn(face[a], p[a]), inv[a]);
      const float lmin =
          stop(prm, min_ref(l[0], min_ref(l[1], l[2])), __ldg(prm.kappa + cell), cell + toff);
      ++steps;
      if (kReemit) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          p[a] = (l[a] == lmin) ? face[a] : __fmaf_rn(lmin, dcs[a], p[a]);
      }
    }
  }
};

// counters of the warp -> statistics of its instance (all lanes)
__device__ __forceinline__ void path_counters(const PathParams &prm, PathShared &sh, int lane,
                                              uint32_t &cross, uint32_t &trans) {
  uint32_t a = sh.absorbed[lane], e = sh.escaped[lane], r = sh.reemitted[lane];
  flush_counters(prm.stats, sh.inst, cross, trans, a, e, r);
  sh.absorbed[lane] = sh.escaped[lane] = sh.reemitted[lane] = 0u;
}

// The next packets of the warp's share into its (empty) queue; all lanes.  none: no
// lane holds a packet.  Another instance's geometry waits until then.
template <class W>
__device__ __noinline__ void path_emit(const PathParams &prm, PathShared &sh, double *table,
                                       uint32_t copy, bool none, uint32_t *counts) {
  const int lane = threadIdx.x & 31;
  RoundState *st = prm.st;
  const uint32_t N = st->emit_total, it = st->iteration;
  const uint64_t seed = st->seed;
  uint32_t job = sh.job, job_end = sh.job_end, inst = sh.inst;
  __syncwarp();
  if (job == job_end) {
    // Guided claims, about half an even part of what is left of the share, then of the
    // next share with anything left.  CTAs start on different shares, so that they
    // spread over the sources: the cells around one take every packet it emits.
    uint32_t j0 = 0, j1 = 0, own = sh.share;
    if (sh.fresh) {
      // the first claim is the warp's by its place (k_begin_emission counts it)
      const PathShare mine(N, own);
      const uint32_t q = (blockIdx.x / kPathShares * kPathWarps + (threadIdx.x >> 5)) * 32u;
      j0 = mine.begin + min(q, mine.size);
      j1 = mine.begin + min(q + 32u, mine.size);
      __syncwarp();
      if (lane == 0) sh.fresh = 0u;
    }
    while (j0 >= j1) {
      // what is left of share (own + lane), seen by lane
      const uint32_t k = (own + (uint32_t)lane) % kPathShares;
      const PathShare there(N, k);
      const uint32_t size = there.size;
      const uint32_t taken =
          lane < kPathShares ? *(volatile uint32_t *)&st->share_next[k] : size;
      const unsigned open = __ballot_sync(kFull, taken < size);
      if (open == 0u) break;
      const int first = __ffs(open) - 1;
      if (lane == first) {
        const uint32_t jn = min(256u, max(32u, ((size - taken) * (uint32_t)kPathShares /
                                                (2u * gridDim.x * kPathWarps)) & ~31u));
        const uint32_t q = atomicAdd(&st->share_next[k], jn);
        j0 = there.begin + min(q, size);
        j1 = there.begin + min(q + jn, size);
      }
      j0 = __shfl_sync(kFull, j0, first);
      j1 = __shfl_sync(kFull, j1, first);
      own = (own + (uint32_t)first) % kPathShares;
    }
    if (lane == 0) sh.share = own;
    if (j0 >= j1) {
      if (lane == 0) sh.exhausted = 1u;
      __syncwarp();
      return;
    }
    job = j0;
    job_end = j1;
  }
  if (job < sh.src_begin) {  // a share of an earlier source
    if (lane == 0) sh.src_end = 0u;
    __syncwarp();
  }
  if (job >= sh.src_end) {
    const int s = find_bin(prm.src_first, prm.nsrc_total + 1, job);
    const uint32_t next = prm.src[s].instance;
    if (next != inst && !none) {
      if (lane == 0) {
        sh.job = job;
        sh.job_end = job_end;
      }
      __syncwarp();
      return;
    }
    if (next != inst) {
      if (inst != kNone) path_counters(prm, sh, lane, counts[0], counts[1]);
      __syncwarp();
      inst = next;
      for (int i = lane; i < (int)(sizeof(DevGeo) / 4); i += 32)
        reinterpret_cast<uint32_t *>(&sh.geo)[i] =
            reinterpret_cast<const uint32_t *>(prm.geo + inst)[i];
      __syncwarp();
      path_table(table, sh, prm.subs, copy, lane);
      __syncwarp();
    }
    if (lane == 0) {
      sh.inst = inst;
      sh.inst_first = prm.src_first[prm.inst[inst].first_source];
      sh.src_begin = (uint32_t)prm.src_first[s];
      sh.src_end = (uint32_t)prm.src_first[s + 1];
      W at;
      at.at_source(prm, sh, smem_addr(table), prm.src[s]);
    }
    __syncwarp();
  }
  const uint32_t n = min(32u, min(job_end, sh.src_end) - job);
  if ((uint32_t)lane < n) {
    double dir[3], tau;
    philox_packet(seed, inst, it, (uint64_t)(job + (uint32_t)lane) - sh.inst_first, dir, tau);
    for (int a = 0; a < 3; ++a) {
      sh.q_dir[a][lane] = dir[a];
      sh.q_inv[a][lane] = W::inverse(sh.geo, a, dir[a]);
    }
    sh.q_tau[lane] = tau;
  }
  if (lane == 0) {
    sh.job = job + n;
    sh.job_end = job_end;
    sh.q_at = 0u;
    sh.q_n = n;
  }
  __syncwarp();
}

template <class W, bool kReemit, int kMinBlocks>
__global__ void __launch_bounds__(kPathThreads, kMinBlocks) k_path(const __grid_constant__ PathParams prm) {
  extern __shared__ __align__(16) unsigned char path_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PathShared &sh = reinterpret_cast<PathShared *>(path_smem)[warp];
  double *table = reinterpret_cast<double *>(path_smem + sizeof(PathShared) * kPathWarps) +
                  (size_t)warp * prm.table;
  const uint32_t tab = smem_addr(table);
  const uint32_t copy = (blockIdx.x * kPathWarps + (uint32_t)warp) % prm.copies;
  if (lane == 0) {
    sh.inst = kNone;
    sh.fresh = 1u;
    sh.share = blockIdx.x % (uint32_t)kPathShares;
    sh.job = sh.job_end = sh.src_begin = sh.src_end = sh.q_at = sh.q_n = sh.exhausted = 0u;
  }
  sh.absorbed[lane] = sh.escaped[lane] = sh.reemitted[lane] = sh.most[lane] = 0u;
  __syncwarp();
  W w;
  w.steps = 0;
  int status = kPathFree;
  uint32_t cross = 0, trans = 0;  // cells crossed, subgrids entered

  for (;;) {
    // lanes that are done with their packet, and new packets for them
    const unsigned done = __ballot_sync(kFull, status != kRun);
    uint32_t waiting = (uint32_t)__popc(done);
    if (waiting >= W::kRefill || done == kFull) {
      if (status == kAbsorbed) {
        w.template absorb<kReemit>(prm, sh.geo);
        cross += (uint32_t)w.steps;
        ++trans;
        status = kPathFree;
        if (kReemit && sh.geo.reemission > 0.) {
          uint32_t h[3];
          double rd[4];
          w.reemit_counter(sh, lane, tab, h);
          if (reemit_draw_call(prm.st->seed, sh.inst, prm.st->iteration, h[0], h[1], h[2],
                               sh.again[lane], sh.geo.reemission, rd)) {
            ++sh.reemitted[lane];
            ++sh.again[lane];
            status = w.reemit(prm, sh, lane, tab, rd);
          }
        }
        if (status == kPathFree) {
          ++sh.absorbed[lane];
          sh.most[lane] = max(sh.most[lane], sh.visits[lane]);
        }
      }
      // well before a 32-bit counter or its sum over the warp could wrap
      if (__any_sync(kFull, cross > 0x04000000u)) path_counters(prm, sh, lane, cross, trans);
      const unsigned idle = __ballot_sync(kFull, status == kPathFree);
      if (sh.exhausted) {
        if (idle == kFull) break;
      } else if (idle != 0u) {
        if (sh.q_at == sh.q_n) {
          uint32_t counts[2] = {cross, trans};
          path_emit<W>(prm, sh, table, copy, idle == kFull, counts);
          cross = counts[0];
          trans = counts[1];
        }
        const uint32_t q_at = sh.q_at, q_n = sh.q_n;
        const uint32_t r = q_at + (uint32_t)__popc(idle & ((1u << lane) - 1u));
        if (status == kPathFree && r < q_n) {
          for (int a = 0; a < 3; ++a) w.direction(sh.geo, a, sh.q_dir[a][r], sh.q_inv[a][r]);
          w.depth(sh.q_tau[r]);
          status = w.start(prm, sh, lane, tab);
          sh.visits[lane] = 1u;
          if (kReemit) sh.again[lane] = 0u;
        }
        __syncwarp();
        if (lane == 0) sh.q_at = min(q_n, q_at + (uint32_t)__popc(idle));
        __syncwarp();
      }
      waiting = (uint32_t)__popc(__ballot_sync(kFull, status != kRun && status != kExited));
    }
    // crossings, until enough more lanes wait (half of those left when they are few)
    const uint32_t enough =
        min(32u, waiting + max(1u, min(W::kTransit, (33u - waiting) / 2u)));
    bool over = true;
#pragma unroll 1
    for (int u = 0; u < kPathStretch; ++u) {
#pragma unroll
      for (int k = 0; k < kPathLook; ++k)
        if (status == kRun) status = w.step(prm, sh.geo, tab);
      if ((uint32_t)__popc(__ballot_sync(kFull, status != kRun)) >= enough) {
        over = false;
        break;
      }
    }
    if (over && status == kRun && w.steps > sh.geo.n[0] + sh.geo.n[1] + sh.geo.n[2] + 3) {
      atomicOr(&prm.st->flags, kFlagWalkLimit);
      status = kPathFree;
    }
    // lanes at a subgrid face
    if (status == kExited && !w.settle_last(prm, sh.geo)) status = kAbsorbed;
    if (status == kExited) {
      cross += (uint32_t)w.steps;
      ++trans;
      status = w.transit(prm, sh, lane, tab);
      if (kReemit) sh.again[lane] = 0u;
      const uint32_t v = sh.visits[lane] + 1u;
      sh.visits[lane] = v;
      if (status == kPathFree) {
        ++sh.escaped[lane];
        sh.most[lane] = max(sh.most[lane], v - 1u);
      } else if (v > prm.round_cap) {
        atomicOr(&prm.st->flags, kFlagLeftover);
        status = kPathFree;
      }
    }
  }
  uint32_t most = __reduce_max_sync(kFull, sh.most[lane]);
  if (sh.inst != kNone) path_counters(prm, sh, lane, cross, trans);
  if (lane == 0 && most) atomicMax(&prm.st->rounds_active, most);
}

// n_H and x_H of an instance side by side for the dust walks, whose scattered loads
// then take one sector of a cell instead of two (128^3, 4e6 packets: 9735 -> 9200 us
// with this pass of 15 us; the ionizing FP64 walk, whose fields change with every
// iteration, lost: 64^3, 1e6 packets 238 -> 242).
__global__ void __launch_bounds__(256) k_pair(const DevSubgrid *subs, uint32_t first_sub,
                                              const double *nH, const double *xH, double2 *nx) {
  const DevSubgrid &S = subs[first_sub + blockIdx.x];
  const int end = min(S.ncells, (int)(blockIdx.y + 1) * kFieldCells);
  for (int c = (int)blockIdx.y * kFieldCells + threadIdx.x; c < end; c += blockDim.x) {
    const int64_t i = S.field_offset + c;
    nx[i] = make_double2(nH[i], xH[i]);
  }
}

// tallies of a transport without balance into J
__global__ void __launch_bounds__(256) k_merge_tally(const DevSubgrid *subs, const DevInstance *inst,
                              unsigned long long *tally, const uint32_t *hot, uint32_t copies,
                              bool fixed, double *J) {
  const DevSubgrid &S = subs[blockIdx.x];
  const DevInstance &I = inst[S.instance];
  const uint32_t h = hot[blockIdx.x];
  const int end = min(S.ncells, (int)(blockIdx.y + 1) * kBalanceCells);
  for (int c = (int)blockIdx.y * kBalanceCells + threadIdx.x; c < end; c += blockDim.x) {
    const int64_t i = S.field_offset + c;
    const double v = take_tally(tally, i, h, copies, (uint32_t)S.padded_cells, c, fixed, I);
    if (v != 0.) J[i] += v;
  }
}

}  // namespace cmi
