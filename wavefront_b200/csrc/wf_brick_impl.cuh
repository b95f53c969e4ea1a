// wf_brick_impl.cuh -- the one-shot fused H->E step: one CTA computes one
// brick of 32 x 8 x 4 cells and exits (wf_brick.cu and wf_brick16.cu
// instantiate it).
//
//  * The brick's E (with a one-cell halo) and old H (with the -x, -y and -z
//    faces) arrive in two TMA boxes; cells outside the domain arrive as zeros
//    (OUTER_ZERO_BLOCK, src/engine.rs:83), and on a periodic axis the wrapped
//    cells are then patched in with plain loads.
//  * Every thread updates H of one group of 4 cells in place in shared memory
//    (some also a group of a face), and after one barrier E of its group.  H
//    on the faces is recomputed, never exchanged between CTAs; the state is
//    double-buffered.
//  * CPML code is entered per axis where the brick meets that axis's slab; a
//    brick reads and writes psi only where its cells are graded, at any slab
//    width.
//  * Sources and probes are applied by the brick that holds their cell, so a
//    step with few of them is one launch (BrickTail).
//
// Per-cell arithmetic is wf_internal.cuh's: results are bit-identical to the
// marching and split kernels.
//
// What bounds it, and why this shape (B200, us a step):
//  * The marching tiles walk a z chunk plane by plane, 2 to 4 us a plane for a
//    CTA that holds CPML cells, so a small grid waits for one item's chain
//    (64^3 with 16 CPML cells: 51.9) and one launch per CPML class.  A brick's
//    chain is one load, two phases, one store: 6.8; 128^3 117 -> 40; 256^3
//    with 8 CPML cells 298 -> 233.
//  * Bound by latency inside the SM (24 warps in flight with CPML, 36
//    without), not by the loads: with everything after the boxes skipped the
//    same grids take half the time.  Halo groups have warps of their own: done
//    by the main warps in a second pass they cost 15-20 % (128^3: 48).  Four
//    planes a brick, two or three CTAs an SM, beat eight planes (128^3: 43.6)
//    and bricks of 32 x 4 x 4 at three or four CTAs (44.6, 42.4; 256^3 286,
//    275 for 250) and 32 x 4 x 8 at two (41.0, 260).
//    Forcing more CTAs an SM spills and loses (64 registers: 64^3 17 us), and
//    so does a persistent CTA that prefetches its next brick (128^3: 55).
#pragma once
#include <algorithm>
#include <type_traits>

#include "wf_internal.cuh"
#include "wf_launch.h"
#include "wf_store.cuh"

namespace wf {

namespace {

// main warps: one group of 4 cells per thread; halo warps: the groups of the
// -y rows, the -z plane, and the -x column (one cell per thread)
constexpr int kBrickMain = kBrickX / 4 * kBrickY * kBrickZ;
constexpr int kYh = 8 * kBrickZ, kZh = kYh + 64, kXh = kZh + 8 * kBrickZ;
constexpr int kBrickThreads = kBrickMain + kXh;

template <typename ST>
struct BrickL {
  static constexpr int PAD = Store<ST>::PAD;
  static constexpr int EW = kBrickX + 2 * PAD, EH = kBrickY + 2, ED = kBrickZ + 2;
  static constexpr int EP = EW * EH, EC = EP * ED;  // one plane, one component
  static constexpr int HW = kBrickX + PAD, HH = kBrickY + 1, HD = kBrickZ + 1;
  static constexpr int HP = HW * HH, HC = HP * HD;
  static constexpr int E_BYTES = 3 * EC * static_cast<int>(sizeof(ST));
  static constexpr int H_BYTES = 3 * HC * static_cast<int>(sizeof(ST));
  static constexpr int H_OFF = (E_BYTES + 127) / 128 * 128;
  static constexpr int BYTES = H_OFF + H_BYTES + 128;  // + base alignment slack
};

__device__ __forceinline__ float4 b_ldg4(const float *p) {
  return __ldg(reinterpret_cast<const float4 *>(p));
}
__device__ __forceinline__ void b_st4(float *p, const float v[4]) {
  *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void unpack(const float4 &v, float o[4]) {
  o[0] = v.x;
  o[1] = v.y;
  o[2] = v.z;
  o[3] = v.w;
}
__device__ __forceinline__ unsigned char id_of(uchar4 m, int q) {
  return q == 0 ? m.x : (q == 1 ? m.y : (q == 2 ? m.z : m.w));
}

// Computing units of a plane (16-bit storage; all 1 for FP32): fC and fN
// take the stored values of the plane and of the next one into units of 2^w;
// psi stays in field units, so a raw difference enters the recursion times
// su = 2^w and its result leaves it times iu = 2^-w.
struct PlaneUnits {
  float fC, fN, su, iu;
};

// Where one group's 4 cells meet the CPML slabs: flags (1 x, 2 y, 4 z), the
// slab positions, and for x whether the group moves as one vector.
struct GroupPml {
  int fl;
  unsigned xin;    // XS: bit k: cell k is in the x slab
  bool xvec;       // its x psi move as one vector
  int sx, sy, sz;  // sx: position cell 0 has, or would have, in the x slab
};

template <bool XS>
__device__ __forceinline__ GroupPml group_pml(const GridArgs &g, int fl, int x, int y, int z, bool ok) {
  GroupPml m{0, 0u, false, 0, 0, 0};
  if (!ok) return m;
  if (fl & 1) {
    const PmlAxis &P = g.pml[0];
    const int s0 = slab_pos(x, g.nx, P.T, P.W);
    m.sx = s0;
    if (!XS) {  // T and nx are multiples of 4: a group is all in or all out
      if (s0 >= 0) m.fl |= 1;
      m.xvec = true;
    } else {
      // (nx % 8 == 0: a group meets the low slab or the high one, never both
      // with a gap between, so its positions are consecutive)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (slab_pos(x + k, g.nx, P.T, P.W) >= 0) m.xin |= 1u << k;
      if (m.xin) m.fl |= 1;
      m.sx = x < P.T ? x : x - (g.nx - P.W);
      m.xvec = m.xin == 15u && (m.sx & 3) == 0;
    }
  }
  if (fl & 2) {
    m.sy = slab_pos(y, g.ny, g.pml[1].T, g.pml[1].W);
    if (m.sy >= 0) m.fl |= 2;
  }
  if (fl & 4) {
    m.sz = slab_pos(z, g.nz, g.pml[2].T, g.pml[2].W);
    if (m.sz >= 0) m.fl |= 4;
  }
  return m;
}

// psi index of the group's first cell on an axis (x: of its row, slab
// position 0).  Cell and psi indices stay below 2^31 here (brick_ok,
// wf_engine.cu), so an address is a uniform component base plus a 32-bit offset.
__device__ __forceinline__ unsigned psi_at(const GridArgs &g, const GroupPml &m, int axis, int x, int y,
                                           int z) {
  if (axis == 0) return static_cast<unsigned>((z * g.ny + y) * g.pml[0].pitch);
  if (axis == 1) return static_cast<unsigned>((z * g.pml[1].W + m.sy) * g.nx + x);
  return static_cast<unsigned>((m.sz * g.ny + y) * g.nx + x);
}

// One psi of one axis for 4 cells (slot: the component in the axis's array)
template <bool XS>
__device__ __forceinline__ void psi_load(const GridArgs &g, const GroupPml &m, int axis, int slot, int x,
                                         int y, int z, float q[4]) {
  if (!(m.fl & (1 << axis))) return;
  const PmlAxis &P = g.pml[axis];
  const float *c = P.psi_cur + slot * P.cells;
  const unsigned i = psi_at(g, m, axis, x, y, z) + (axis == 0 ? m.sx : 0);
  if (!XS || axis != 0 || m.xvec) {
    if (!idx_ok(g.err, static_cast<long long>(i) + 3, P.cells)) return;
    unpack(b_ldg4(c + i), q);
  } else {
    // (cell 0 of a group that only ends in the slab may lie before position 0,
    // so i + k is formed in 32 bits, where it wraps back, before the pointer)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned j = i + k;
      q[k] = (m.xin >> k & 1u) && idx_ok(g.err, j, P.cells) ? __ldg(c + j) : 0.0f;
    }
  }
}

// The psi recursion of one difference over 4 cells, the new psi stored when
// `store`.
template <bool FMA, bool U, bool XS>
__device__ __forceinline__ void psi_corr(const GridArgs &g, const GroupPml &m, int axis, int slot, int x,
                                         int y, int z, bool store, const PlaneUnits &u, float d[4],
                                         float p[4]) {
  if (!(m.fl & (1 << axis))) return;
  const PmlAxis &P = g.pml[axis];
  auto one = [&](float &v, float &ps, float b, float a, float ik) {
    v = U ? __fmul_rn(pml_corr<FMA>(__fmul_rn(v, u.su), b, a, ik, ps), u.iu)
          : pml_corr<FMA>(v, b, a, ik, ps);
  };
  const unsigned i = psi_at(g, m, axis, x, y, z) + (axis == 0 ? m.sx : 0);
  float *o = P.psi_nxt + slot * P.cells;
  if (axis != 0) {
    const int s = axis == 1 ? m.sy : m.sz;
    const float b = __ldg(P.prof + s), a = __ldg(P.prof + P.W + s), ik = __ldg(P.prof + 2 * P.W + s);
#pragma unroll
    for (int k = 0; k < 4; ++k) one(d[k], p[k], b, a, ik);
    if (store && idx_ok(g.err, static_cast<long long>(i) + 3, P.cells)) b_st4(o + i, p);
  } else {
    float b[4], a[4], ik[4];  // by x coordinate: aligned for every group
    unpack(b_ldg4(P.full + x), b);
    unpack(b_ldg4(P.full + g.nx + x), a);
    unpack(b_ldg4(P.full + 2 * g.nx + x), ik);
    if (!XS || m.xvec) {
#pragma unroll
      for (int k = 0; k < 4; ++k) one(d[k], p[k], b[k], a[k], ik[k]);
      if (store && idx_ok(g.err, static_cast<long long>(i) + 3, P.cells)) b_st4(o + i, p);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float v = d[k];
        one(v, p[k], b[k], a[k], ik[k]);
        const bool in = m.xin >> k & 1u;
        d[k] = in ? v : d[k];
        const unsigned j = i + k;  // as in psi_load
        if (store && in && idx_ok(g.err, j, P.cells)) o[j] = p[k];
      }
    }
  }
}

// The psi of a group's six differences: x (ez, ey), y (ez, ex), z (ey, ex)
// for H (term 0), x (hz, hy), y (hz, hx), z (hy, hx) for E (term 2).
struct Psi6 {
  float x0[4], x1[4], y0[4], y1[4], z0[4], z1[4];
};
template <bool XS>
__device__ __forceinline__ void psi_load6(const GridArgs &g, const GroupPml &m, int term, int x, int y,
                                          int z, Psi6 &q) {
  psi_load<XS>(g, m, 1, term, x, y, z, q.y0);
  psi_load<XS>(g, m, 2, term, x, y, z, q.z0);
  psi_load<XS>(g, m, 2, term + 1, x, y, z, q.z1);
  psi_load<XS>(g, m, 0, term, x, y, z, q.x0);
  psi_load<XS>(g, m, 0, term + 1, x, y, z, q.x1);
  psi_load<XS>(g, m, 1, term + 1, x, y, z, q.y1);
}

// New H of one group, in place in the H box (update_h_field[_pml],
// src/fdtd.rs:194-345): e and hb point at its first cell in the E and H
// boxes; MASK: the components wanted (1 hx, 2 hy, 4 hz); st: called with
// (component, stored word) of each.  Whole warp (the +x neighbours come by
// shuffle); a HALO group outside
// the domain (!ok) writes zeros (no E update reads the others beyond it).
template <bool FMA, bool PML, bool XS, int MASK, bool HALO, typename ST, typename F>
__device__ __forceinline__ void brick_h(const GridArgs &g, const ST *e, ST *hb, int col, const GroupPml &m,
                                        int x, int y, int z, bool ok, bool store, const PlaneUnits &u,
                                        Psi6 &ps, uchar4 id, F st) {
  using L = BrickL<ST>;
  using SD = Store<ST>;
  constexpr bool U = SD::k16;
  float ex[4], ey[4], ez[4];
  auto ld = [&](const ST *p, float f, float o[4]) {
    if (U && f != 1.0f)
      unpack(SD::template ld4<true>(p, f), o);
    else
      unpack(SD::template ld4<false>(p, f), o);
  };
  ld(e, u.fC, ex);
  ld(e + L::EC, u.fC, ey);
  ld(e + 2 * L::EC, u.fC, ez);
  float ezx = __shfl_down_sync(0xffffffffu, ez[0], 1);
  float eyx = __shfl_down_sync(0xffffffffu, ey[0], 1);
  if (col == kBrickX / 4 - 1) {
    ezx = SD::template ld1<U>(e + 2 * L::EC + 4, u.fC);
    eyx = SD::template ld1<U>(e + L::EC + 4, u.fC);
  }
  float2 cf[4];  // da, db
#pragma unroll
  for (int q = 0; q < 4; ++q) cf[q] = __ldg(reinterpret_cast<const float2 *>(g.coef + id_of(id, q)) + 1);
  auto finish = [&](int c, const float d0[4], const float d1[4]) {
    float o[4];
    ld(hb + c * L::HC, u.fC, o);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      o[q] = h_new<FMA>(cf[q].x, o[q], cf[q].y, sub(d0[q], d1[q]));
      if (HALO && !ok) o[q] = 0.0f;
    }
    const typename SD::Word w = SD::enc4(o);
    SD::st4(hb + c * L::HC, w);
    st(c, w);
  };
  float a[4], b[4];
  if (MASK & 1) {
    ld(e + 2 * L::EC + L::EW, u.fC, a);
    ld(e + L::EC + L::EP, u.fN, b);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = sub(a[q], ez[q]);
      b[q] = sub(b[q], ey[q]);
    }
    if (PML && m.fl) {
      psi_corr<FMA, U, XS>(g, m, 1, 0, x, y, z, store, u, a, ps.y0);
      psi_corr<FMA, U, XS>(g, m, 2, 0, x, y, z, store, u, b, ps.z0);
    }
    finish(0, a, b);
  }
  if (MASK & 2) {
    ld(e + L::EP, u.fN, a);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = sub(a[q], ex[q]);
      b[q] = sub(q < 3 ? ez[q + 1] : ezx, ez[q]);
    }
    if (PML && m.fl) {
      psi_corr<FMA, U, XS>(g, m, 2, 1, x, y, z, store, u, a, ps.z1);
      psi_corr<FMA, U, XS>(g, m, 0, 0, x, y, z, store, u, b, ps.x0);
    }
    finish(1, a, b);
  }
  if (MASK & 4) {
    ld(e + L::EW, u.fC, b);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = sub(q < 3 ? ey[q + 1] : eyx, ey[q]);
      b[q] = sub(b[q], ex[q]);
    }
    if (PML && m.fl) {
      psi_corr<FMA, U, XS>(g, m, 0, 1, x, y, z, store, u, a, ps.x1);
      psi_corr<FMA, U, XS>(g, m, 1, 1, x, y, z, store, u, b, ps.y1);
    }
    finish(2, a, b);
  }
}

// The wrapped cells of the periodic axes, where the boxes hold zeros: E on
// every face the brick shares with the domain's, H on the -x, -y, -z ones.
__device__ __forceinline__ void patch_periodic(const GridArgs &g, float *sE, float *sH, int x0, int y0,
                                               int z0) {
  using L = BrickL<float>;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int xe = min(x0 + kBrickX, nx), bw = xe - x0 + 2;  // box columns x0 - 1 .. xe
  auto patch = [&](int X, int Y, int Z) {
    int wx = X, wy = Y, wz = Z;
    if (wx < 0 || wx >= nx) {
      if (!g.periodic[0]) return;
      wx = wx < 0 ? wx + nx : wx - nx;
    }
    if (wy < 0 || wy >= ny) {
      if (!g.periodic[1]) return;
      wy = wy < 0 ? wy + ny : wy - ny;
    }
    if (wz < 0 || wz >= nz) {
      if (!g.periodic[2]) return;
      wz = wz < 0 ? wz + nz : wz - nz;
    }
    const long long i = (static_cast<long long>(wz) * ny + wy) * nx + wx;
    if (!idx_ok(g.err, i, g.N)) return;
    const int bx = X - x0, by = Y - y0 + 1, bz = Z - z0 + 1;
    const int o = (bz * L::EH + by) * L::EW + L::PAD + bx;
#pragma unroll
    for (int c = 0; c < 3; ++c) sE[o + c * L::EC] = __ldg(g.cur + c * g.N + i);
    if (bx < kBrickX && by <= kBrickY && bz <= kBrickZ) {
      const int k = (bz * L::HH + by) * L::HW + L::PAD + bx;
#pragma unroll
      for (int c = 0; c < 3; ++c) sH[k + c * L::HC] = __ldg(g.cur + (3 + c) * g.N + i);
    }
  };
  const int tid = threadIdx.x;
  for (int side = 0; side < 2; ++side) {
    if (g.periodic[0] && (side ? x0 + kBrickX >= nx : x0 == 0))
      for (int i = tid; i < L::EH * L::ED; i += kBrickThreads)
        patch(side ? xe : x0 - 1, y0 - 1 + i % L::EH, z0 - 1 + i / L::EH);
    if (g.periodic[1] && (side ? y0 + kBrickY >= ny : y0 == 0))
      for (int i = tid; i < bw * L::ED; i += kBrickThreads)
        patch(x0 - 1 + i % bw, side ? y0 + kBrickY : y0 - 1, z0 - 1 + i / bw);
    if (g.periodic[2] && (side ? z0 + kBrickZ >= nz : z0 == 0))
      for (int i = tid; i < bw * L::EH; i += kBrickThreads)
        patch(x0 - 1 + i % bw, y0 - 1 + i / bw, side ? z0 + kBrickZ : z0 - 1);
  }
}

// A brick's own sources (their cells, components and this step's values) and
// probes (cells and components, then samples): lists of hits by list index.
struct BrickTailSmem {
  unsigned src, prb;  // bit k: source / probe k has a cell in the brick
  struct Src {
    int comp, mode, x, y, z;
    float v;
  } s[kBrickTailMax];
  int4 p[kBrickTailMax];  // comp, x, y, z
  float raw[kBrickTailMax];
};

// Programmatic dependent launch: a brick launch may start while the step
// before is still running and waits here, its barrier and coordinates ready,
// until that step's results are visible; then it lets the next one start.
// (A launch without the attribute passes straight through.)
__device__ __forceinline__ void wait_previous_step() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// One brick.  smem: BrickL<ST>::BYTES, 128-byte aligned.
// ARGS: BrickArgs, or without TAIL BrickGrid
template <bool FMA, bool PML, bool XS, bool TAIL, typename ST, typename ARGS>
__device__ __forceinline__ void brick_body(const CUtensorMap *tmE, const CUtensorMap *tmH,
                                           const ARGS &a, unsigned char *smem, int x0, int y0,
                                           int z0) {
  using L = BrickL<ST>;
  using SD = Store<ST>;
  constexpr bool U = SD::k16;
  const GridArgs &g = a.g;
  __shared__ uint64_t s_bar;
  __shared__ unsigned s_max[2];
  __shared__ typename std::conditional<TAIL, BrickTailSmem, int>::type s_tail;
  (void)s_tail;
  const int tid = threadIdx.x;
  ST *sE = reinterpret_cast<ST *>(smem), *sH = reinterpret_cast<ST *>(smem + L::H_OFF);
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long N = g.N;
  if (tid == 0) {
    const uint32_t bar = smem_u32(&s_bar);
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmE)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmH)) : "memory");
    mbar_init(bar, 1);
    mbar_fence_init();
    s_max[0] = s_max[1] = 0u;
    wait_previous_step();
    // (a nonzero test_extra_tx leaves the phase incomplete after the copies
    // have landed, so the bounded wait runs out: the timeout path, tested)
    mbar_expect_tx(bar, L::E_BYTES + L::H_BYTES + static_cast<uint32_t>(a.test_extra_tx));
    tma_load_4d(smem_u32(sE), tmE, x0 - L::PAD, y0 - 1, z0 - 1, 0, bar);
    tma_load_4d(smem_u32(sH), tmH, x0 - L::PAD, y0 - 1, z0 - 1, 3, bar);
  }

  // CPML axes the brick's cells or its -x, -y, -z faces meet
  int fl = 0;
  if (PML && g.pml[0].T > 0 &&
      (x0 - 1 < g.pml[0].T || x0 + kBrickX > nx - g.pml[0].T || (x0 == 0 && g.periodic[0])))
    fl |= 1;
  if (PML && g.pml[1].T > 0 &&
      (y0 - 1 < g.pml[1].T || y0 + kBrickY > ny - g.pml[1].T || (y0 == 0 && g.periodic[1])))
    fl |= 2;
  if (PML && g.pml[2].T > 0 &&
      (z0 - 1 < g.pml[2].T || z0 + kBrickZ > nz - g.pml[2].T || (z0 == 0 && g.periodic[2])))
    fl |= 4;

  // this thread's group: 4 cells from (x, y, z), or one cell (-x column);
  // role 0 main, 1 the -y rows, 2 the -z plane, 3 the -x column
  const int ht = tid - kBrickMain;
  const int role = ht < 0 ? 0 : (ht < kYh ? 1 : (ht < kZh ? 2 : 3));
  const int col = tid & 7;
  int r = (tid >> 3) & 7, p = tid >> 6;  // row and plane in the brick
  if (role == 1) {
    r = -1;
    p = ht >> 3;
  } else if (role == 2) {
    r = (ht - kYh) >> 3;
    p = -1;
  } else if (role == 3) {
    r = tid & 7;
    p = (ht - kZh) >> 3;
  }
  int x = role == 3 ? x0 - 1 : x0 + 4 * col, y = y0 + r, z = z0 + p;
  bool in = x < nx;  // nx % 8 == 0: a group is all in or all out
  if (role) {        // the faces wrap on a periodic axis
    if (x < 0) {
      in = g.periodic[0];
      x += nx;
    }
    if (y < 0) {
      in = in && g.periodic[1];
      y += ny;
    }
    if (z < 0) {
      in = in && g.periodic[2];
      z += nz;
    }
  }
  const unsigned cell = static_cast<unsigned>((z * ny + y) * nx + x);
  ST *const nxt = reinterpret_cast<ST *>(g.nxt);
  in = in && idx_ok(g.err, static_cast<long long>(cell) + (role == 3 ? 0 : 3), N);
  // sources and probes with a cell in this brick: the first -x warp looks at
  // the sources, the first -y warp at the probes, and the sources' values are
  // loaded while the boxes arrive
  if constexpr (TAIL) {
    const int li = tid & 31;
    const bool src_warp = role == 3 && ht - kZh < 32;
    bool hit = false;
    if (src_warp) {
      if (li < a.tail.nsrc) {
        const SrcDev &q = a.tail.src[li];
        s_tail.s[li] = BrickTailSmem::Src{q.comp, q.mode, q.x, q.y, q.z, 0.0f};
        hit = q.x >= x0 && q.x < x0 + kBrickX &&
              (q.mode != 0 || (q.y >= y0 && q.y < y0 + kBrickY && q.z >= z0 && q.z < z0 + kBrickZ));
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (li == 0) s_tail.src = m;
    } else if (role == 1 && ht < 32) {
      bool at = false;
      if (li < a.tail.nprobe) {
        const ProbeDev &q = a.tail.probe[li];
        s_tail.p[li] = make_int4(q.comp, q.x, q.y, q.z);
        at = q.x >= x0 && q.x < x0 + kBrickX && q.y >= y0 && q.y < y0 + kBrickY && q.z >= z0 &&
             q.z < z0 + kBrickZ;
      }
      const unsigned m = __ballot_sync(0xffffffffu, at);
      if (li == 0) s_tail.prb = m;
    }
    wait_previous_step();
    const bool first = src_warp && li == 0 && x0 == 0 && y0 == 0 && z0 == 0;
    if (hit || first) {
      const long long st = __ldcg(a.tail.step);
      if (hit) {
        const SrcDev &q = a.tail.src[li];
        s_tail.s[li].v = st < q.nvals ? q.vals[st] : 0.0f;
      }
      if (first) *a.tail.step_next = st + 1;
    }
  } else {
    wait_previous_step();
  }
  uchar4 id = make_uchar4(0, 0, 0, 0);
  if (in) {
    const uint8_t *m = g.mat + static_cast<unsigned>((z * ny + y) * g.mat_pitch + x);
    if (role == 3)
      id.x = __ldg(m);
    else
      id = __ldg(reinterpret_cast<const uchar4 *>(m));
  }
  // the H terms' psi: in flight while the boxes arrive
  GroupPml gm{0, 0u, false, 0, 0, 0};
  Psi6 ps;
  if (PML && role < 3) {
    gm = group_pml<XS>(g, fl, x, y, z, in);
    if (gm.fl) psi_load6<XS>(g, gm, 0, x, y, z, ps);
  }

  // 16-bit units: of the brick's slab (a brick's planes lie in one slab) and
  // of the slab below (the -z plane)
  PlaneUnits u{1.0f, 1.0f, 1.0f, 1.0f}, ul = u;
  float f_top = 1.0f, f_down = 1.0f;
  const int sl = z0 / kSlabPlanes;
  if constexpr (U) {
    const int up = min((z0 + kBrickZ) / kSlabPlanes, g.nslab - 1);
    const int dn = max(z0 - 1, 0) / kSlabPlanes;
    const int w = __ldg(g.shift_wr + 2 * sl), wd = __ldg(g.shift_wr + 2 * dn);
    const int rd = __ldg(g.shift_rd + 2 * sl);
    u = PlaneUnits{pow2f(rd - w), pow2f(rd - w), pow2f(w), pow2f(-w)};
    f_top = pow2f(__ldg(g.shift_rd + 2 * up) - w);
    ul = PlaneUnits{pow2f(__ldg(g.shift_rd + 2 * dn) - wd), pow2f(rd - wd), pow2f(wd), pow2f(-wd)};
    f_down = pow2f(wd - w);
  }

  __syncthreads();  // the mbarrier is initialised
  bool ok = mbar_wait_or_error(smem_u32(&s_bar), 0, g.err);
  ok = __syncthreads_or(ok ? 0 : 1) == 0;
  if (!ok) {
    // the phase never completed within the limit: latch the error (without an
    // error word, the caller's own fields: the brick's new values become NaN);
    // one more bounded wait before this CTA's shared memory is released (short
    // when the error is latched: its copies have had the first wait)
    if (tid == 0) {
      if (g.err) atomicOr(g.err, kErrTimeout);
      mbar_wait_or_error(smem_u32(&s_bar), 0, g.err);
    }
    if (!g.err && role == 0 && in) {
      if constexpr (!U)
        for (int c = 0; c < 6; ++c)
          for (int q = 0; q < 4; ++q) nxt[c * N + cell + q] = __int_as_float(0x7fffffff);
    }
    return;
  }
  if constexpr (!U) {
    if (g.periodic[0] | g.periodic[1] | g.periodic[2]) {
      patch_periodic(g, sE, sH, x0, y0, z0);
      __syncthreads();
    }
  }

  // ---- H ----
  unsigned mxE = 0u, mxH = 0u;
  const ST *const e = sE + ((p + 1) * L::EH + r + 1) * L::EW + L::PAD + 4 * col;
  ST *const hb = sH + ((p + 1) * L::HH + r + 1) * L::HW + L::PAD + 4 * col;
  PlaneUnits v = role == 2 ? ul : u;
  if (U && p == kBrickZ - 1) v.fN = f_top;
  auto keep = [](int, const typename SD::Word &) {};
  if (role == 0) {
    brick_h<FMA, PML, XS, 7, false, ST>(g, e, hb, col, gm, x, y, z, in, true, v, ps, id,
                                        [&](int c, const typename SD::Word &w) {
                                          if (!in) return;
                                          SD::st4(nxt + (3 + c) * N + cell, w);
                                          if constexpr (U)
                                            mxH = __vmaxu2(mxH, __vmaxu2(SD::mag(w.x), SD::mag(w.y)));
                                        });
  } else if (role == 1) {
    brick_h<FMA, PML, XS, 5, true, ST>(g, e, hb, col, gm, x, y, z, in, false, v, ps, id, keep);
  } else if (role == 2) {
    brick_h<FMA, PML, XS, 3, true, ST>(g, e, hb, col, gm, x, y, z, in, false, v, ps, id, keep);
  } else {
    // hy, hz of the cell (x0 - 1, y, z) for the E update at x0
    ST *const ho = hb - 4 * col - 1;
    float hyv = 0.0f, hzv = 0.0f;
    if (in) {
      const ST *const q = e - 4 * col - 1;
      auto ev = [&](int o, float f) { return SD::template ld1<U>(q + o, f); };
      const float ex = ev(0, v.fC), ey = ev(L::EC, v.fC), ez = ev(2 * L::EC, v.fC);
      float d_ez_dx = sub(ev(2 * L::EC + 1, v.fC), ez), d_ey_dx = sub(ev(L::EC + 1, v.fC), ey);
      float d_ex_dy = sub(ev(L::EW, v.fC), ex), d_ex_dz = sub(ev(L::EP, v.fN), ex);
      auto one = [&](int axis, int s, unsigned i, int slot, float &d) {
        const PmlAxis &P = g.pml[axis];
        if (s < 0 || !idx_ok(g.err, i, P.cells)) return;
        float q_ = __ldg(P.psi_cur + slot * P.cells + i);
        const float b = __ldg(P.prof + s), c = __ldg(P.prof + P.W + s), ik = __ldg(P.prof + 2 * P.W + s);
        d = U ? __fmul_rn(pml_corr<FMA>(__fmul_rn(d, v.su), b, c, ik, q_), v.iu)
              : pml_corr<FMA>(d, b, c, ik, q_);
      };
      if (PML && (fl & 1)) {
        const PmlAxis &P = g.pml[0];
        const int s = slab_pos(x, nx, P.T, P.W);
        const unsigned i = static_cast<unsigned>((z * ny + y) * P.pitch + s);
        one(0, s, i, 0, d_ez_dx);
        one(0, s, i, 1, d_ey_dx);
      }
      if (PML && (fl & 2)) {
        const PmlAxis &P = g.pml[1];
        const int s = slab_pos(y, ny, P.T, P.W);
        one(1, s, static_cast<unsigned>((z * P.W + s) * nx + x), 1, d_ex_dy);
      }
      if (PML && (fl & 4)) {
        const PmlAxis &P = g.pml[2];
        const int s = slab_pos(z, nz, P.T, P.W);
        one(2, s, static_cast<unsigned>((s * ny + y) * nx + x), 1, d_ex_dz);
      }
      const float2 cf = __ldg(reinterpret_cast<const float2 *>(g.coef + id.x) + 1);
      hyv = h_new<FMA>(cf.x, SD::template ld1<U>(ho + L::HC, v.fC), cf.y, sub(d_ex_dz, d_ez_dx));
      hzv = h_new<FMA>(cf.x, SD::template ld1<U>(ho + 2 * L::HC, v.fC), cf.y, sub(d_ey_dx, d_ex_dy));
    }
    if constexpr (U) {
      *reinterpret_cast<unsigned short *>(ho + L::HC) = static_cast<unsigned short>(SD::enc2(hyv, hyv));
      *reinterpret_cast<unsigned short *>(ho + 2 * L::HC) = static_cast<unsigned short>(SD::enc2(hzv, hzv));
    } else {
      ho[L::HC] = hyv;
      ho[2 * L::HC] = hzv;
    }
  }
  // the E terms' psi: in flight across the barrier
  if (PML && role == 0 && gm.fl) psi_load6<XS>(g, gm, 2, x, y, z, ps);
  __syncthreads();

  // ---- E (update_e_field[_pml], src/fdtd.rs:369-509) ----
  if (role == 0) {
    float hx4[4], hy4[4], hz4[4], b4[4], a4[4];
    auto ldh = [&](const ST *q, float o[4]) { unpack(SD::template ld4<false>(q, 1.0f), o); };
    ldh(hb, hx4);
    ldh(hb + L::HC, hy4);
    ldh(hb + 2 * L::HC, hz4);
    float hzx = __shfl_up_sync(0xffffffffu, hz4[3], 1);
    float hyx = __shfl_up_sync(0xffffffffu, hy4[3], 1);
    if (col == 0) {
      hzx = SD::template ld1<false>(hb + 2 * L::HC - 1, 1.0f);
      hyx = SD::template ld1<false>(hb + L::HC - 1, 1.0f);
    }
    if (in) {
      float2 cf[4];  // ca, cb
#pragma unroll
      for (int q = 0; q < 4; ++q) cf[q] = __ldg(reinterpret_cast<const float2 *>(g.coef + id_of(id, q)));
      auto ldz = [&](const ST *q, float o[4]) {  // the plane below, in this slab's units
        ldh(q, o);
        if (U && p == 0 && f_down != 1.0f) {
#pragma unroll
          for (int k = 0; k < 4; ++k) o[k] = __fmul_rn(o[k], f_down);
        }
      };
      auto finish = [&](int c) {
        float o[4];
        if (U && u.fC != 1.0f)
          unpack(SD::template ld4<true>(e + c * L::EC, u.fC), o);
        else
          unpack(SD::template ld4<false>(e + c * L::EC, 1.0f), o);
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = e_new<FMA>(cf[q].x, o[q], cf[q].y, sub(a4[q], b4[q]));
        const typename SD::Word w = SD::enc4(o);
        SD::st4(nxt + c * N + cell, w);
        if constexpr (U) mxE = __vmaxu2(mxE, __vmaxu2(SD::mag(w.x), SD::mag(w.y)));
      };
      // ex: d_hz_dy - d_hy_dz
      ldh(hb + 2 * L::HC - L::HW, a4);
      ldz(hb + L::HC - L::HP, b4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a4[q] = sub(hz4[q], a4[q]);
        b4[q] = sub(hy4[q], b4[q]);
      }
      if (PML && gm.fl) {
        psi_corr<FMA, U, XS>(g, gm, 1, 2, x, y, z, true, u, a4, ps.y0);
        psi_corr<FMA, U, XS>(g, gm, 2, 2, x, y, z, true, u, b4, ps.z0);
      }
      finish(0);
      // ey: d_hx_dz - d_hz_dx
      ldz(hb - L::HP, a4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a4[q] = sub(hx4[q], a4[q]);
        b4[q] = sub(hz4[q], q == 0 ? hzx : hz4[q - 1]);
      }
      if (PML && gm.fl) {
        psi_corr<FMA, U, XS>(g, gm, 2, 3, x, y, z, true, u, a4, ps.z1);
        psi_corr<FMA, U, XS>(g, gm, 0, 2, x, y, z, true, u, b4, ps.x0);
      }
      finish(1);
      // ez: d_hy_dx - d_hx_dy
      ldh(hb - L::HW, b4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a4[q] = sub(hy4[q], q == 0 ? hyx : hy4[q - 1]);
        b4[q] = sub(hx4[q], b4[q]);
      }
      if (PML && gm.fl) {
        psi_corr<FMA, U, XS>(g, gm, 0, 3, x, y, z, true, u, a4, ps.x1);
        psi_corr<FMA, U, XS>(g, gm, 1, 3, x, y, z, true, u, b4, ps.y1);
      }
      finish(2);
    }
  }
  if constexpr (U) {  // the slab's largest stored magnitudes (one shift per slab)
    const unsigned e = __reduce_max_sync(0xffffffffu, max(mxE & 0xffffu, mxE >> 16));
    const unsigned hm = __reduce_max_sync(0xffffffffu, max(mxH & 0xffffu, mxH >> 16));
    if ((tid & 31) == 0) {
      atomicMax(&s_max[0], e);
      atomicMax(&s_max[1], hm);
    }
    __syncthreads();
    if (tid < 2 && s_max[tid])
      atomicMax(g.slab_max + 2 * sl + tid,
                __float_as_uint(__fmul_rn(SD::dec_lo(s_max[tid]), u.su)));
  }

  // ---- sources in list order, then probes (src/engine.rs:769-782) ----
  if constexpr (TAIL) {
    const unsigned mprb = s_tail.prb;
    if (s_tail.src | mprb) {
      if (role == 0 && in) {  // by the cell's own thread, on what it just stored
        for (unsigned m = s_tail.src; m; m &= m - 1) {
          const BrickTailSmem::Src s = s_tail.s[__ffs(m) - 1];
          if (s.x < x || s.x > x + 3 || (s.mode == 0 && (s.y != y || s.z != z))) continue;
          float *f = g.nxt + s.comp * N + cell + (s.x - x);
          if (idx_ok(g.err, s.comp * N + cell + (s.x - x), 6 * N))
            *f = s.mode == 0 ? __fadd_rn(*f, s.v) : s.v;
        }
        for (unsigned m = mprb; m; m &= m - 1) {
          const int4 s = s_tail.p[__ffs(m) - 1];
          if (s.y < x || s.y > x + 3 || s.z != y || s.w != z) continue;
          if (idx_ok(g.err, s.x * N + cell + (s.y - x), 6 * N))
            s_tail.raw[__ffs(m) - 1] = g.nxt[s.x * N + cell + (s.y - x)];
        }
      }
      if (mprb) {
        const bool mine = role == 1 && ht < 32 && (mprb >> ht & 1u);
        ProbeDev q;
        long long st = 0;
        if (mine) {
          q = a.tail.probe[ht];
          st = __ldcg(a.tail.step);
        }
        __syncthreads();  // the samples
        if (mine) {
          const float raw = s_tail.raw[ht];
          if (q.record && st < q.nsteps) q.trace[st] = raw;
          if (st >= q.first_step && st < q.nsteps) {
            const double v = static_cast<double>(raw);
            for (int f = 0; f < q.nfreq; ++f) {
              q.sc[f] = __dadd_rn(q.sc[f], __dmul_rn(v, q.cos_tab[st * q.nfreq + f]));
              q.ss[f] = __dadd_rn(q.ss[f], __dmul_rn(v, q.sin_tab[st * q.nfreq + f]));
            }
            q.n[0] += 1ull;
          }
        }
      }
    }
  }
}

// CTA (x + tiles_x * j, z, band): brick (x, 8 band + j, z).  CTAs run x
// fastest, then 8 rows of bricks in y, then z, then the next band of rows, so
// that a brick's z neighbour runs within a few MB of traffic of it and only
// every 8th y face is far away: halo planes and rows come from L2.
template <bool FMA, bool PML, bool XS, bool TAIL, typename ST>
__global__ void __launch_bounds__(kBrickThreads, PML ? 2 : 3)
    k_brick(const __grid_constant__ CUtensorMap tmE, const __grid_constant__ CUtensorMap tmH,
            const __grid_constant__ BrickArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  int x0, y0, z0;
  if (PML && !TAIL && a.shell.n) {  // around an interior of marching tiles
    int b = 0, first = 0;
#pragma unroll
    for (int k = 0; k < 5; ++k)
      if (static_cast<int>(blockIdx.x) >= a.shell.end[k]) {
        b = k + 1;
        first = a.shell.end[k];
      }
    const int3 lo = a.shell.lo[b];
    const unsigned sx = a.shell.nxy[b].x, sy = a.shell.nxy[b].y;
    const unsigned i = blockIdx.x - first, q = i / sx, z = q / sy;
    x0 = (lo.x + static_cast<int>(i - q * sx)) * kBrickX;
    y0 = (lo.y + static_cast<int>(q - z * sy)) * kBrickY;
    z0 = (lo.z + static_cast<int>(z)) * kBrickZ;
  } else {
    const unsigned j = a.x_magic ? __umulhi(blockIdx.x, a.x_magic) : blockIdx.x;  // / tiles_x
    y0 = (blockIdx.z * kBrickBand + j) * kBrickY;
    if (y0 >= a.g.ny) return;
    x0 = (blockIdx.x - j * a.tiles_x) * kBrickX;
    z0 = blockIdx.y * kBrickZ;
  }
  brick_body<FMA, PML, XS, TAIL, ST>(&tmE, &tmH, a, smem, x0, y0, z0);
}

// Batched step: CTA i computes brick items[i] = (scene, x0, y0, z0).  The
// scene's arguments are copied to shared memory first: constant-bank operands
// of k_brick become shared loads here.
template <bool XS>
__global__ void __launch_bounds__(kBrickThreads, 2)
    k_brick_batch(const BrickScene *scenes, const int4 *items, int parity) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  __shared__ BrickGrid s_args;
  const int4 it = __ldg(items + blockIdx.x);
  const BrickScene *sc = scenes + it.x;
  const int *src = reinterpret_cast<const int *>(&sc->args[parity]);
  for (int i = threadIdx.x; i < static_cast<int>(sizeof(BrickGrid) / 4); i += kBrickThreads)
    reinterpret_cast<int *>(&s_args)[i] = __ldg(src + i);
  __syncthreads();
  brick_body<false, true, XS, false, float>(&sc->maps[parity].e, &sc->maps[parity].h, s_args, smem, it.y, it.z,
                                     it.w);
}

// Instantiations of a storage type: no CPML; CPML with an x depth that is a
// multiple of 4; any CPML.  TAIL: FP32 only.
using BrickFn = void (*)(CUtensorMap, CUtensorMap, BrickArgs);

template <bool FMA, bool TAIL, typename ST>
BrickFn brick_fn(int variant) {
  return variant == 0   ? k_brick<FMA, false, false, TAIL, ST>
         : variant == 1 ? k_brick<FMA, true, false, TAIL, ST>
                        : k_brick<FMA, true, true, TAIL, ST>;
}

template <bool FMA, typename ST>
cudaError_t brick_prepare_t() {
  for (int v = 0; v < 3; ++v) {
    cudaError_t e = cudaFuncSetAttribute(brick_fn<FMA, false, ST>(v),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, BrickL<ST>::BYTES);
    if constexpr (!Store<ST>::k16)
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(brick_fn<FMA, true, ST>(v), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 BrickL<ST>::BYTES);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <bool FMA, typename ST>
cudaError_t brick_launch_t(const BrickMaps &m, const BrickArgs &a, cudaStream_t s) {
  const int tiles_y = a.g.ny / kBrickY;
  cudaLaunchConfig_t c{};
  c.gridDim = a.shell.n ? dim3(a.shell.n)
                        : dim3(a.tiles_x * std::min(tiles_y, kBrickBand), a.g.nz / kBrickZ,
                               (tiles_y + kBrickBand - 1) / kBrickBand);
  c.blockDim = dim3(kBrickThreads);
  c.dynamicSmemBytes = BrickL<ST>::BYTES;
  c.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr;
  c.numAttrs = a.shell.n ? 0 : 1;  // a shell launch joins the interior's stream instead
  const int T = a.g.pml[0].T;
  const int v = !(T | a.g.pml[1].T | a.g.pml[2].T) ? 0 : (T % 4 == 0 ? 1 : 2);
  BrickFn f = brick_fn<FMA, false, ST>(v);
  if constexpr (!Store<ST>::k16)
    if (a.tail.on) f = brick_fn<FMA, true, ST>(v);
  return cudaLaunchKernelEx(&c, f, m.e, m.h, a);
}

}  // namespace
}  // namespace wf
