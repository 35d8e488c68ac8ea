// Differentiable form: the forward step with per-particle weights and the
// discrete adjoint of the whole step.
//
// Forward step n -> n+1 (the plain push of kernels_push.cuh and the field
// solve of kernels_field.cuh):
//   G^n = N(E^n, B^n)                       node averages (linear)
//   (x, u)^{n+1}, J = Push((x, u)^n, G^n)   gather, Boris, move, zig-zag deposit
//   (E, B)^{n+1} = A (E, B)^n + C J         B half step, E full step, B half step
// The adjoint runs the steps backwards:
//   field adjoint: the transposed FDTD update (k_adj_bhalf, k_adj_efull), and
//                  the transposed node average (k_adj_nodes);
//   particle adjoint (k_dadjoint): recompute the push of each particle from its
//                  stored state, then the deposition adjoint as a gather of the
//                  current adjoint at the particle's stencil, the move adjoint,
//                  the reverse Boris rotation, and the field-gather adjoint as a
//                  scatter-add of the particle's field adjoint to its 4 nodes.
// Branch decisions (cell crossings, relay points, the jz quadrant, wall
// reflections) are piecewise constant and enter the adjoint as fixed.
// Adjoint quantities are accumulated in double precision.
//
// Order: a state's particles are read in the order of their cells, through a permutation
// that the step before left with it, and the step writes its results in that
// order; each particle carries its index in load order (species and sheet follow
// from it). Elements of one cell take their places in the order their atomics land, so a
// recomputed segment may end in another order than the forward run's checkpoint: the
// adjoint carried into it is read by particle there (remap). The lanes of a warp that share a cell then form a run, and what they
// add to the same nodes is summed in shared memory first (run_sums). Without that every
// particle added its 12 current terms and its 24 node adjoints to L2 on its
// own, from places all over the grid (load order): 4.19 M particles, 256x128 cells, FP32
// forward: k_dpush 299 us, k_dadjoint 782 us, bound by the rate of the atomics;
// now 152 us and 426 us, with 25 us for the order. What bounds them now: k_dpush instruction
// issue (70 %); k_dadjoint the latency of its chain of loads at 20 warps per SM (96
// registers; 3 blocks of 128 per SM without spills 547 us, 4 427 us, 6 at 80
// registers slower). Quotients by gamma are products with rsqrt(1 + u^2), and 2 / (1 + t^2) is
// push_two_over: against extended precision, 1 <= 1 + u^2 <= 2, rms error of c / gamma 5.9e-17 (7.4e-17 as a quotient by a
// square root), c / gamma^2 9.5e-17 (14.3e-17), c / gamma^3 13.3e-17 (20.2e-17), up to 1 + u^2 = 11 also smaller in each;
// largest errors 1.8, 3.5 and 4.8e-16 (2.2, 3.3, 5.4e-16), up to 11 2.1, 4.2 and 6.2e-16 (2.2, 3.3, 5.3e-16); those of
// 2 / (1 + t^2) are the same. The sums are FP64 as before;
// FP32 deposit terms are rounded to the fixed point of the accumulators before they are
// summed, which makes the sums exact, so the current has the same bits in any order.
#pragma once
#include "device_common.cuh"
#include "kernels_push.cuh"
#include "kernels_sort.cuh"
#include "pic_fields_init.h"

namespace pbd {

// The particles of one state.
template <class T>
struct DiffState {
  uint32_t* cell;
  Comps<T> c;      // dx dy ux uy as one record, uz
  int32_t* id;     // index in load order (pairs: 2k ion, 2k+1 electron)
  int32_t* perm;   // position in cell order -> element, bit 31 for a background particle (perm_entry)
};
constexpr int32_t PERM_ELEM = 0x7fffffff;
__device__ __forceinline__ int32_t perm_entry(int64_t e, int32_t id, int64_t nsheet) {
  return (int32_t)e | ((id >> 1) < nsheet ? 0 : (int32_t)0x80000000);
}

template <class T>
struct DiffParams {
  PushParams<T> push;     // constants, geometry, the node grid of step n and the current
  int64_t n;              // particles
  double omega_bg;        // weight of background particles (of the sheet's: 1)
  double in0;             // current normalisation
  DiffState<T> in, out;   // states before and after the step (out: forward only, cell null: not wanted)
  int32_t* rank;          // forward: each new element's rank in its cell
  int32_t* counts;        // and the cells' counts (0 on entry)
  Comps<T> lam_in;        // adjoint of the state after the step (null: zero)
  const int32_t* remap;   // null, or the element of each particle (by id) in lam_in's order
  Comps<T> lam_out;       // adjoint of the state before the step; may be in.c itself
  const double* jbar;     // adjoint of the normalised current, 3 planes of mx x S
  double* gbar;           // adjoint of the node fields (mx+1) x (my+1) x 8
  double* domega;         // d loss / d omega_bg (one double)
};

// Rank of this lane's element among those of its cell counted so far; key < 0: no element. In no
// particular order across warps.
__device__ __forceinline__ int32_t count_in_cell(int32_t* counts, int key) {
  const unsigned peers = __match_any_sync(FULL, key);
  const int leader = __ffs(peers) - 1;
  int32_t base = 0;
  if (key >= 0 && (int)lane_id() == leader) base = atomicAdd(&counts[key], __popc(peers));
  base = __shfl_sync(FULL, base, leader);
  return base + __popc(peers & lanemask_lt());
}

// Sums v[0..NV) (NV <= 16) over each run of lanes with the same key (the lanes of a run are
// adjacent); entry k of the run with that key goes to add(k, key, sum), by lane k.
// st: the warp's staging, [NV][33]. Lanes with key < 0 take no part.
template <int NV, class Add>
__device__ __forceinline__ void run_sums(const double (&v)[NV], int key, double* st, const Add& add) {
  const int lane = (int)lane_id(), k = lane & 15, half = lane >> 4;
  const int prev = __shfl_up_sync(FULL, key, 1);
  unsigned heads = __ballot_sync(FULL, lane == 0 || prev != key);
#pragma unroll
  for (int i = 0; i < NV; ++i) st[i * 33 + lane] = v[i];
  __syncwarp();
  while (heads) {
    const int start = __ffs(heads) - 1;
    heads &= heads - 1;
    const int end = heads ? __ffs(heads) - 1 : 32;
    const int rk = __shfl_sync(FULL, key, start);
    if (rk < 0) continue;
    double s = 0.0;
    if (k < NV)
      for (int l = start + half; l < end; l += 2) s += st[k * 33 + l];
    s += __shfl_xor_sync(FULL, s, 16);
    if (lane < NV) add(k, rk, s);
  }
  __syncwarp();
}

constexpr int DT = 128, DWARPS = DT / 32;  // threads of the particle kernels' blocks
#ifndef DADJ_MINBLOCKS
#define DADJ_MINBLOCKS 5
#endif

// A cell whose deposit stencil needs no wrap or wall image.
template <class T>
__device__ __forceinline__ bool inner_cell(const PushParams<T>& pp, int ix, int iy) {
  return ix >= 2 && ix < pp.mx - 2 && iy >= 2 && iy < pp.my - 2;
}

// Forward push with weights: the plain push, current (jx, jy, jz) deposited
// into double accumulators (FP64) or int64 fixed point (FP32, deterministic).
template <class T>
__global__ void __launch_bounds__(DT) k_dpush(DiffParams<T> a) {
  constexpr bool F32 = sizeof(T) == 4;
  __shared__ double stage[DWARPS][13 * 33];
  const PushParams<T>& pp = a.push;
  const int64_t j = (int64_t)blockIdx.x * DT + threadIdx.x;
  const bool ok = j < a.n;
  const int32_t pe = ok ? a.in.perm[j] : 0;
  const int e = pe & PERM_ELEM;
  const uint32_t w = a.in.cell[e];
  const int sp = cw_sp(w), ix = cw_ix(w), iy = cw_iy(w);
  const T* g00 = pp.ng + ((long long)ix * (pp.my + 1) + iy) * 8;
  const T* g10 = g00 + (long long)(pp.my + 1) * 8;
  const Node6<T> n00 = load_node(g00), n01 = load_node(g00 + 8), n10 = load_node(g10), n11 = load_node(g10 + 8);
  Pushed<T> o;
  const P5<T> q = ldg_part(a.in.c, e);
  push_one<T, false>(pp, sp, ix, iy, q.dx, q.dy, q.ux, q.uy, q.uz, n00, n01, n10, n11, o);
  const double om = !ok ? 0.0 : (pe >= 0 ? 1.0 : a.omega_bg);
  double t[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    t[k] = om * (double)o.e[k];
    if (F32) t[k] = rint(t[k] * (double)FIX_SCALE);  // whole steps of the fixed point: exact sums
  }
  auto put = [&](int c, int cx, int cy, int x, int y, double v) {  // at node (cx + x, cy + y) of cell (cx, cy)
    long long gi = ((long long)c * pp.mx + cx + x) * pp.S + cy + y;
    if (!inner_cell(pp, cx, cy)) {
      int sg;
      if (!map_current(c, cx + x, cy + y, pp.mx, pp.my, pp.S, pp.ybc, 0, &gi, &sg)) return;
      v = sg < 0 ? -v : v;
    }
    if (F32) atomicAdd(reinterpret_cast<unsigned long long*>(pp.jacc) + gi, (unsigned long long)__double2ll_rn(v));
    else atomicAdd(reinterpret_cast<double*>(pp.jacc) + gi, v);
  };
  const bool cross = o.dcx != 0 || o.dcy != 0;
  double v[13];
  v[0] = cross ? t[0] : t[0] + t[2];
  v[1] = cross ? t[1] : t[1] + t[3];
  v[2] = cross ? t[4] : t[4] + t[6];
  v[3] = cross ? t[5] : t[5] + t[7];
#pragma unroll
  for (int x = -1; x <= 1; ++x)
#pragma unroll
    for (int y = -1; y <= 1; ++y)
      v[4 + (x + 1) * 3 + y + 1] = (x == 0 || x == o.di) && (y == 0 || y == o.dj)
                                       ? (x == 0 ? (y == 0 ? t[8] : t[10]) : (y == 0 ? t[9] : t[11]))
                                       : 0.0;
  if (ok && cross) {  // the second segment, in the new cell
    put(JX, ix, iy, o.dcx, o.dcy, t[2]);
    put(JX, ix, iy, o.dcx, o.dcy + 1, t[3]);
    put(JY, ix, iy, o.dcx, o.dcy, t[6]);
    put(JY, ix, iy, o.dcx + 1, o.dcy, t[7]);
  }
  const int key = ok ? ix * pp.my + iy : -1;
  int kc, kx, ky;
  stencil_node((int)lane_id() & 15, &kc, &kx, &ky);
  run_sums<13>(v, key, stage[threadIdx.x >> 5], [&](int k, int rk, double sum) {
    if (sum == 0.0) return;
    const int cx = rk / pp.my, cy = rk - cx * pp.my;
    put(kc, cx, cy, kx, ky, sum);
  });
  if (!a.out.cell) return;  // (the whole grid)
  if (ok) {
    a.out.cell[j] = o.cw;
    put_part(a.out.c, j, P5<T>{o.dx, o.dy, o.ux, o.uy, o.uz});
    a.out.id[j] = a.in.id[e];
  }
  const int32_t r = count_in_cell(a.counts, ok ? cw_ix(o.cw) * pp.my + cw_iy(o.cw) : -1);
  if (ok) a.rank[j] = r;
}

struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 cross3(D3 a, D3 b) {
  return D3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ D3 add3(D3 a, D3 b) { return D3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 scale3(D3 a, double s) { return D3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ double dot3(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Particle adjoint of one step (see the file comment).
template <class T>
__global__ void __launch_bounds__(DT, DADJ_MINBLOCKS) k_dadjoint(DiffParams<T> a) {
  const PushParams<T>& pp = a.push;
  __shared__ double red[32];
  __shared__ double stage[DWARPS][12 * 33];
  double domega = 0.0;
  const int64_t j = (int64_t)blockIdx.x * DT + threadIdx.x;
  const bool ok = j < a.n;
  const int32_t pe = ok ? a.in.perm[j] : 0;
  const int e = pe & PERM_ELEM;
  const uint32_t w = a.in.cell[e];
  const int sp = cw_sp(w), ix = cw_ix(w), iy = cw_iy(w);
  const bool sheet = pe >= 0;
  const int64_t p = !ok ? 0 : (a.remap ? a.remap[a.in.id[e]] : j);  // the particle in the state after the step
  const T* g00 = pp.ng + ((long long)ix * (pp.my + 1) + iy) * 8;
  const T* g10 = g00 + (long long)(pp.my + 1) * 8;
  const Node6<T> n00 = load_node(g00), n01 = load_node(g00 + 8), n10 = load_node(g10), n11 = load_node(g10 + 8);
  // (in.c by plain loads, by the element's own thread only: lam_out may take its place)
  const P5<T> q = ok ? get_part(a.in.c, e) : P5<T>{}, l1 = a.lam_in.q ? ldg_part(a.lam_in, p) : P5<T>{};
  const T px = q.dx, py = q.dy, pux = q.ux, puy = q.uy, puz = q.uz;
  Pushed<T> o;  // the forward push, for the branch decisions and the deposit terms
  push_one<T, false>(pp, sp, ix, iy, px, py, pux, puy, puz, n00, n01, n10, n11, o);
  const double om = sheet ? 1.0 : a.omega_bg;
  // ---- forward quantities in double
  const double c0 = (double)(sp ? pp.c0[1] : pp.c0[0]), c1 = (double)(sp ? pp.c1[1] : pp.c1[0]);
  const double qx = (double)(sp ? pp.qx[1] : pp.qx[0]), qy = (double)(sp ? pp.qy[1] : pp.qy[0]);
  const double qq = (double)(sp ? pp.q[1] : pp.q[0]);
  const double ax = 0.5 + (double)px, ay = 0.5 + (double)py;
  const double W[4] = {(1 - ax) * (1 - ay), ax * (1 - ay), (1 - ax) * ay, ax * ay};  // n00 n10 n01 n11
  const Node6<T>* nodes[4] = {&n00, &n10, &n01, &n11};
  D3 E{0, 0, 0}, B{0, 0, 0};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    E = add3(E, scale3(D3{(double)nodes[k]->ex, (double)nodes[k]->ey, (double)nodes[k]->ez}, W[k]));
    B = add3(B, scale3(D3{(double)nodes[k]->bx, (double)nodes[k]->by, (double)nodes[k]->bz}, W[k]));
  }
  const D3 u{(double)pux, (double)puy, (double)puz};
  const D3 um = add3(u, scale3(E, c1));
  const double rgm = rsqrt(1.0 + dot3(um, um));  // 1 / gamma: every quotient by gamma is a product with it
  const double c2 = c0 * rgm;
  const D3 t = scale3(B, c2);
  const double t2 = push_two_over(1.0 + dot3(t, t));
  const D3 s = scale3(t, t2);
  const D3 u0 = add3(um, cross3(um, t));
  const D3 up = add3(um, cross3(u0, s));
  const D3 u1 = add3(up, scale3(E, c1));
  const double rg1 = rsqrt(1.0 + dot3(u1, u1));
  const double dtcva = (double)pp.dtcva, cva = (double)pp.cva;
  const double c3 = dtcva * rg1;
  const double idx = (double)pp.idx, idy = (double)pp.idy;
  const double x1 = (double)px + c3 * u1.x * idx, y1 = (double)py + c3 * u1.y * idy;
  const double vz = u1.z * cva * rg1;
  const int dcx = o.dcx, dcy = o.dcy;
  // ---- adjoint of the state after the step; undo the wall reflection
  const bool refl = pp.ybc == 1 && (iy + dcy < 0 || iy + dcy >= pp.my);
  double lx1 = (double)l1.dx;
  double ly1 = (double)l1.dy * (refl ? -1.0 : 1.0);
  D3 lu1{(double)l1.ux, (double)l1.uy * (refl ? -1.0 : 1.0), (double)l1.uz};
  double lpx = 0.0, lpy = 0.0, lvz = 0.0;
  // ---- deposition adjoint: gather the current adjoint at the 12 terms (no wrap or image inside the domain)
  const bool inner = inner_cell(pp, ix, iy);
  double tb[12];
  double dom = 0.0;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    int rx, ry;
    term_node(k, dcx, dcy, o.di, o.dj, &rx, &ry);
    double jb = 0.0;  // d loss / d (unweighted term k)
    if (inner) {
      jb = a.jbar[((long long)(k >> 2) * pp.mx + ix + rx) * pp.S + iy + ry] * a.in0;
    } else {
      long long gi;
      int sg;
      if (map_current(k >> 2, ix + rx, iy + ry, pp.mx, pp.my, pp.S, pp.ybc, 0, &gi, &sg)) jb = a.jbar[gi] * a.in0 * sg;
    }
    tb[k] = jb * om;
    dom += jb * (double)o.e[k];
  }
  if (ok && !sheet) domega += dom;
  {
    const double fdcx = dcx, fdcy = dcy;
    const double im = 0.5 * ((double)px + x1 + 1.0), jm = 0.5 * ((double)py + y1 + 1.0);
    const double ir = dcx == 0 ? im : (dcx > 0 ? 1.0 : 0.0);
    const double jr = dcy == 0 ? jm : (dcy > 0 ? 1.0 : 0.0);
    const double fx1 = qx * (ir - px - 0.5), fx2 = qx * (x1 + 0.5 - ir);
    const double fy1 = qy * (jr - py - 0.5), fy2 = qy * (y1 + 0.5 - jr);
    const double wx1 = 0.5 * (ir + px + 0.5), wy1 = 0.5 * (jr + py + 0.5);
    const double wx2 = 0.5 * (ir + x1 - 2 * fdcx + 0.5), wy2 = 0.5 * (jr + y1 - 2 * fdcy + 0.5);
    const double bfx1 = tb[0] * (1 - wy1) + tb[1] * wy1, bwy1 = (tb[1] - tb[0]) * fx1;
    const double bfx2 = tb[2] * (1 - wy2) + tb[3] * wy2, bwy2 = (tb[3] - tb[2]) * fx2;
    const double bfy1 = tb[4] * (1 - wx1) + tb[5] * wx1, bwx1 = (tb[5] - tb[4]) * fy1;
    const double bfy2 = tb[6] * (1 - wx2) + tb[7] * wx2, bwx2 = (tb[7] - tb[6]) * fy2;
    double bir = qx * bfx1 - qx * bfx2 + 0.5 * bwx1 + 0.5 * bwx2;
    double bjr = qy * bfy1 - qy * bfy2 + 0.5 * bwy1 + 0.5 * bwy2;
    lpx += -qx * bfx1 + 0.5 * bwx1;
    lx1 += qx * bfx2 + 0.5 * bwx2;
    lpy += -qy * bfy1 + 0.5 * bwy1;
    ly1 += qy * bfy2 + 0.5 * bwy2;
    double bim = dcx == 0 ? bir : 0.0;
    double bjm = dcy == 0 ? bjr : 0.0;
    // jz: CIC at the midpoint, z1 = ab, z2 = a(1-b), z3 = b(1-a), z4 = (1-a)(1-b)
    const double dmx = im - 0.5, dmy = jm - 0.5;
    const double av = fabs(dmx), bv = fabs(dmy);
    const double quz = qq * vz;
    const double z1 = av * bv, z2 = av * (1 - bv), z3 = bv * (1 - av), z4 = (1 - av) * (1 - bv);
    const double bquz = tb[8] * z4 + tb[9] * z2 + tb[10] * z3 + tb[11] * z1;
    const double bz1 = quz * tb[11], bz2 = quz * tb[9], bz3 = quz * tb[10], bz4 = quz * tb[8];
    const double ba = bz1 * bv + bz2 * (1 - bv) - bz3 * bv - bz4 * (1 - bv);
    const double bb = bz1 * av - bz2 * av + bz3 * (1 - av) - bz4 * (1 - av);
    bim += ba * (dmx >= 0 ? 1.0 : -1.0);
    bjm += bb * (dmy >= 0 ? 1.0 : -1.0);
    lpx += 0.5 * bim;
    lx1 += 0.5 * bim;
    lpy += 0.5 * bjm;
    ly1 += 0.5 * bjm;
    lvz += qq * bquz;
  }
  // ---- move adjoint: x1 = px + c3 ux idx, y1 = py + c3 uy idy, vz = uz cva / g1
  lpx += lx1;
  lpy += ly1;
  lu1.x += lx1 * c3 * idx;
  lu1.y += ly1 * c3 * idy;
  lu1.z += lvz * cva * rg1;
  const double bc3 = lx1 * u1.x * idx + ly1 * u1.y * idy;
  const double bg1 = -(bc3 * dtcva + lvz * u1.z * cva) * (rg1 * rg1);
  lu1 = add3(lu1, scale3(u1, bg1 * rg1));
  // ---- reverse Boris rotation
  D3 lE = scale3(lu1, c1);
  const D3 lup = lu1;
  D3 lum = lup;
  const D3 lu0 = cross3(s, lup);
  const D3 ls = cross3(lup, u0);
  lum = add3(lum, add3(lu0, cross3(t, lu0)));
  D3 lt = cross3(lu0, um);
  lt = add3(lt, scale3(ls, t2));
  const double lt2 = dot3(ls, t);
  lt = add3(lt, scale3(t, -lt2 * t2 * t2));
  const double lc2 = dot3(lt, B);
  const D3 lB = scale3(lt, c2);
  const double lgm = -lc2 * c0 * (rgm * rgm);
  lum = add3(lum, scale3(um, lgm * rgm));
  const D3 lu = lum;
  lE = add3(lE, scale3(lum, c1));
  // ---- field-gather adjoint: the weights' adjoint to the offsets ...
  double bW[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Node6<T>& nd = *nodes[k];
    bW[k] = lE.x * (double)nd.ex + lE.y * (double)nd.ey + lE.z * (double)nd.ez + lB.x * (double)nd.bx +
            lB.y * (double)nd.by + lB.z * (double)nd.bz;
  }
  // W = [(1-ax)(1-ay), ax(1-ay), (1-ax)ay, ax ay]
  lpx += -bW[0] * (1 - ay) + bW[1] * (1 - ay) - bW[2] * ay + bW[3] * ay;
  lpy += -bW[0] * (1 - ax) - bW[1] * ax + bW[2] * (1 - ax) + bW[3] * ax;
  if (ok) put_part(a.lam_out, e, P5<T>{(T)lpx, (T)lpy, (T)lu.x, (T)lu.y, (T)lu.z});
  // ... and to the 4 nodes, summed over the particles of a cell: two nodes at a time
  const int key = ok ? ix * pp.my + iy : -1;
  double* st = stage[threadIdx.x >> 5];
  const double f[6] = {lE.x, lE.y, lE.z, lB.x, lB.y, lB.z};
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // the nodes of rows iy + h
    double v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = W[2 * h + k / 6] * f[k % 6];
    run_sums<12>(v, key, st, [&](int k, int rk, double sum) {
      const int cx = rk / pp.my, cy = rk - cx * pp.my, c = k % 6;
      atomicAdd(a.gbar + ((long long)(cx + k / 6) * (pp.my + 1) + cy + h) * 8 + (c < 3 ? c : c + 1), sum);
    });
  }
  const double sum = block_sum(domega, red);
  if (threadIdx.x == 0 && sum != 0.0) atomicAdd(a.domega, sum);
}

// Exclusive scan of the cell counts by chunks of CS_TILE (off, chunk totals in sums), then each
// chunk's prefix added; clears the counts.
static __global__ void __launch_bounds__(CS_BT) k_diff_scan(int32_t* counts, int64_t ncells, int32_t* off, int32_t* sums) {
  __shared__ int32_t ws[CS_BT / 32];
  const int t = threadIdx.x;
  const int64_t c0 = (int64_t)blockIdx.x * CS_TILE + t * CS_IPT;
  int32_t v[CS_IPT], s = 0;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    v[k] = s;
    if (c0 + k < ncells) {
      s += counts[c0 + k];
      counts[c0 + k] = 0;
    }
  }
  int32_t inc = s;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t y = __shfl_up_sync(FULL, inc, d);
    if ((int)lane_id() >= d) inc += y;
  }
  if (lane_id() == 31) ws[t >> 5] = inc;
  __syncthreads();
  int32_t before = inc - s;
#pragma unroll
  for (int k = 0; k < CS_BT / 32; ++k) before += k < (t >> 5) ? ws[k] : 0;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k)
    if (c0 + k < ncells) off[c0 + k] = before + v[k];
  if (t == CS_BT - 1) sums[blockIdx.x] = before + s;
}
static __global__ void __launch_bounds__(CS_BT) k_diff_offsets(int32_t* off, const int32_t* sums, int64_t ncells) {
  __shared__ int32_t ws[CS_BT / 32];
  int32_t add = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += CS_BT) add += sums[k];
  add = __reduce_add_sync(FULL, add);
  if (lane_id() == 0) ws[threadIdx.x >> 5] = add;
  __syncthreads();
  add = 0;
#pragma unroll
  for (int k = 0; k < CS_BT / 32; ++k) add += ws[k];
  const int64_t base = (int64_t)blockIdx.x * CS_TILE;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    const int64_t c = base + k * CS_BT + threadIdx.x;
    if (c < ncells) off[c] += add;
  }
}
// Initial planes of the sheet, and the derivative of the loss by psi0 (the initial B is linear in
// it): sum of the B adjoint times B(psi0 = 1) - B(psi0 = 0). (On the host these cost
// 1.1 ms and 3.5 ms a gradient at 256x128 cells.)
template <class T>
__global__ void k_diff_fields(pic::FieldInit f, int S, T* planes) {
  const int64_t pl = (int64_t)f.mx * S;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < pl; k += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(k / S), j = (int)(k - (int64_t)i * S);
    planes[k] = planes[pl + k] = planes[2 * pl + k] = T(0);
    planes[3 * pl + k] = (T)pic::init_bx(f, i, j);
    planes[4 * pl + k] = (T)pic::init_by(f, i, j);
    planes[5 * pl + k] = (T)pic::init_bz(f, i, j);
  }
}
static __global__ void k_diff_psi(pic::FieldInit f, int S, const double* bx, const double* by, double* out) {
  __shared__ double red[32];
  pic::FieldInit f1 = f, f0 = f;
  f1.psi0 = 1.0;
  f0.psi0 = 0.0;
  const int64_t pl = (int64_t)f.mx * S;
  double s = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < pl; k += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(k / S), j = (int)(k - (int64_t)i * S);
    s += bx[k] * (pic::init_bx(f1, i, j) - pic::init_bx(f0, i, j));
    if (j < f.my) s += by[k] * (pic::init_by(f1, i, j) - pic::init_by(f0, i, j));
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}
// The permutation of a state from its elements' ranks in their cells.
static __global__ void k_diff_perm(const uint32_t* cell, const int32_t* id, int64_t nsheet, const int32_t* rank,
                                   const int32_t* off, int64_t n, int my, int32_t* perm) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t w = cell[e];
    perm[off[(int64_t)cw_ix(w) * my + cw_iy(w)] + rank[e]] = perm_entry(e, id[e], nsheet);
  }
}
// Element of each particle (by id).
static __global__ void k_diff_inverse(const int32_t* id, int64_t n, int32_t* inv) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    inv[id[e]] = (int32_t)e;
}
// Ranks of loaded particles (load order), and their move into cell order.
static __global__ void k_diff_rank(const uint32_t* cell, int64_t n, int my, int32_t* counts, int32_t* rank) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t w = e < n ? cell[e] : 0u;
  const int32_t r = count_in_cell(counts, e < n ? cw_ix(w) * my + cw_iy(w) : -1);
  if (e < n) rank[e] = r;
}
template <class T>
__global__ void k_diff_move(const uint32_t* cell, Comps<T> in, int64_t nsheet, const int32_t* rank, const int32_t* off,
                            int64_t n, int my, DiffState<T> out) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t w = cell[e];
    const int64_t d = (int64_t)off[(int64_t)cw_ix(w) * my + cw_iy(w)] + rank[e];
    out.cell[d] = w;
    put_part(out.c, d, get_part(in, e));
    out.id[d] = (int32_t)e;
    out.perm[d] = perm_entry(d, (int32_t)e, nsheet);
  }
}

// ------------------------------------------------------------ field adjoint
struct AdjField {
  int mx, my, S, ybc;
  double dth, cdt, idx, idy;
  double *ex, *ey, *ez, *bx, *by, *bz;  // adjoint planes (mx x S)
  double* jbar;                          // 3 planes: adjoint of the normalised current
};

__device__ __forceinline__ void adj_half(double* f, int i, int j, int my, int S, int ybc, double odd_sign, double v) {
  if (ybc == 0) {
    j = j < 0 ? j + my : (j >= my ? j - my : j);
    atomicAdd(&f[(long long)i * S + j], v);
    return;
  }
  if (j < 0) atomicAdd(&f[(long long)i * S], odd_sign * v);
  else if (j >= my) atomicAdd(&f[(long long)i * S + my - 1], odd_sign * v);
  else atomicAdd(&f[(long long)i * S + j], v);
}

__device__ __forceinline__ void adj_node(double* f, int i, int j, int my, int S, int ybc, double v) {
  if (ybc == 0 && j >= my) j -= my;
  atomicAdd(&f[(long long)i * S + j], v);
}

// Transposed B half step: the forward reads E and adds to B, so the adjoint
// adds the transposed curl of the B adjoint to the E adjoint.
static __global__ void k_adj_bhalf(AdjField a) {
  const int rows = a.ybc == 0 ? a.my : a.my + 1;
  const long long n = (long long)a.mx * rows;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / rows), j = (int)(k - (long long)i * rows);
    const long long o = (long long)i * a.S + j;
    const double bbx = a.bx[o];  // bx -= dth (ez(i,j) - ez(i,j-1)) idy
    adj_half(a.ez, i, j, a.my, a.S, a.ybc, -1.0, -a.dth * a.idy * bbx);
    adj_half(a.ez, i, j - 1, a.my, a.S, a.ybc, -1.0, a.dth * a.idy * bbx);
    if (j < a.my) {
      const int im = i == 0 ? a.mx - 1 : i - 1, ip = i + 1 == a.mx ? 0 : i + 1;
      const double bby = a.by[o];  // by += dth (ez(i,j) - ez(i-1,j)) idx
      atomicAdd(&a.ez[o], a.dth * a.idx * bby);
      atomicAdd(&a.ez[(long long)im * a.S + j], -a.dth * a.idx * bby);
      const double bbz = a.bz[o];  // bz += dth ((ex(i,j+1)-ex(i,j)) idy - (ey(i+1,j)-ey(i,j)) idx)
      adj_node(a.ex, i, j + 1, a.my, a.S, a.ybc, a.dth * a.idy * bbz);
      atomicAdd(&a.ex[o], -a.dth * a.idy * bbz);
      atomicAdd(&a.ey[(long long)ip * a.S + j], -a.dth * a.idx * bbz);
      atomicAdd(&a.ey[o], a.dth * a.idx * bbz);
    }
  }
}

// Transposed E full step: adds the transposed curl of the E adjoint to the B
// adjoint and sets the current adjoint; the wall rows of ex are set to zero
// by the forward step, so their adjoint does not flow back.
static __global__ void k_adj_efull(AdjField a) {
  const int rows = a.ybc == 0 ? a.my : a.my + 1;
  const long long n = (long long)a.mx * rows;
  const long long plane = (long long)a.mx * a.S;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / rows), j = (int)(k - (long long)i * rows);
    const long long o = (long long)i * a.S + j;
    if (a.ybc == 1 && (j == 0 || j == a.my)) {
      a.jbar[o] = 0.0;
      a.ex[o] = 0.0;  // (no other thread reads it)
    } else {
      const double bex = a.ex[o];  // ex += cdt ((bz(i,j) - bz(i,j-1)) idy - jx)
      adj_half(a.bz, i, j, a.my, a.S, a.ybc, 1.0, a.cdt * a.idy * bex);
      adj_half(a.bz, i, j - 1, a.my, a.S, a.ybc, 1.0, -a.cdt * a.idy * bex);
      a.jbar[o] = -a.cdt * bex;
    }
    if (j < a.my) {
      const int im = i == 0 ? a.mx - 1 : i - 1, ip = i + 1 == a.mx ? 0 : i + 1;
      const double bey = a.ey[o];  // ey -= cdt ((bz(i,j) - bz(i-1,j)) idx + jy)
      atomicAdd(&a.bz[o], -a.cdt * a.idx * bey);
      atomicAdd(&a.bz[(long long)im * a.S + j], a.cdt * a.idx * bey);
      a.jbar[plane + o] = -a.cdt * bey;
      const double bez = a.ez[o];  // ez += cdt ((by(i+1,j)-by(i,j)) idx - (bx(i,j+1)-bx(i,j)) idy - jz)
      atomicAdd(&a.by[(long long)ip * a.S + j], a.cdt * a.idx * bez);
      atomicAdd(&a.by[o], -a.cdt * a.idx * bez);
      adj_node(a.bx, i, j + 1, a.my, a.S, a.ybc, -a.cdt * a.idy * bez);
      atomicAdd(&a.bx[o], a.cdt * a.idy * bez);
      a.jbar[2 * plane + o] = -a.cdt * bez;
    } else {
      a.jbar[plane + o] = 0.0;
      a.jbar[2 * plane + o] = 0.0;
    }
  }
}

// Transposed node average: the node adjoint (mx+1) x (my+1) x 8 goes back to
// the Yee planes with the images and wraps of k_nodes, and is cleared for the next step.
static __global__ void k_adj_nodes(AdjField a, double* gbar) {
  const int NX = a.mx + 1, NY = a.my + 1;
  const long long n = (long long)NX * NY;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int ia = (int)(k / NY), b = (int)(k - (long long)ia * NY);
    const int i = ia == a.mx ? 0 : ia;
    const int im = i == 0 ? a.mx - 1 : i - 1;
    const int bn = (a.ybc == 0 && b == a.my) ? 0 : b;
    double g[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      g[c] = gbar[k * 8 + c];
      gbar[k * 8 + c] = 0.0;
    }
    if (g[0] != 0.0) {
      atomicAdd(&a.ex[(long long)i * a.S + bn], 0.5 * g[0]);
      atomicAdd(&a.ex[(long long)im * a.S + bn], 0.5 * g[0]);
    }
    if (g[4] != 0.0) {
      atomicAdd(&a.bx[(long long)i * a.S + bn], 0.5 * g[4]);
      atomicAdd(&a.bx[(long long)im * a.S + bn], 0.5 * g[4]);
    }
    if (g[1] != 0.0) {
      adj_half(a.ey, i, b, a.my, a.S, a.ybc, 1.0, 0.5 * g[1]);
      adj_half(a.ey, i, b - 1, a.my, a.S, a.ybc, 1.0, 0.5 * g[1]);
    }
    if (g[5] != 0.0) {
      adj_half(a.by, i, b, a.my, a.S, a.ybc, -1.0, 0.5 * g[5]);
      adj_half(a.by, i, b - 1, a.my, a.S, a.ybc, -1.0, 0.5 * g[5]);
    }
    if (g[2] != 0.0) {
      const double v = 0.25 * g[2];
      adj_half(a.ez, i, b, a.my, a.S, a.ybc, -1.0, v);
      adj_half(a.ez, im, b, a.my, a.S, a.ybc, -1.0, v);
      adj_half(a.ez, i, b - 1, a.my, a.S, a.ybc, -1.0, v);
      adj_half(a.ez, im, b - 1, a.my, a.S, a.ybc, -1.0, v);
    }
    if (g[6] != 0.0) {
      const double v = 0.25 * g[6];
      adj_half(a.bz, i, b, a.my, a.S, a.ybc, 1.0, v);
      adj_half(a.bz, im, b, a.my, a.S, a.ybc, 1.0, v);
      adj_half(a.bz, i, b - 1, a.my, a.S, a.ybc, 1.0, v);
      adj_half(a.bz, im, b - 1, a.my, a.S, a.ybc, 1.0, v);
    }
  }
}

// Magnetic-energy loss of one step, dt * 0.5 mime/(cva^2 in0) * sum w |B_node|^2
// over the energy nodes of k_nodes, and its seed for the node adjoint.
template <class T>
__global__ void k_loss_b(int mx, int my, int ybc, const T* ng, double scale, double* loss, double* gbar) {
  __shared__ double red[32];
  const int NX = mx + 1, NY = my + 1;
  const long long n = (long long)NX * NY;
  double s = 0.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int ia = (int)(k / NY), b = (int)(k - (long long)ia * NY);
    if (ia < mx && (ybc == 1 || b < my)) {
      const double wgt = (ybc == 1 && (b == 0 || b == my)) ? 0.5 : 1.0;
      const double bx = (double)ng[k * 8 + 4], by = (double)ng[k * 8 + 5], bz = (double)ng[k * 8 + 6];
      s += wgt * (bx * bx + by * by + bz * bz);
      if (gbar) {
        gbar[k * 8 + 4] += 2.0 * scale * wgt * bx;
        gbar[k * 8 + 5] += 2.0 * scale * wgt * by;
        gbar[k * 8 + 6] += 2.0 * scale * wgt * bz;
      }
    }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0 && loss) atomicAdd(loss, scale * s);
}

// The j.E loss of one step and its adjoint seeds: sum over the Yee entries
// (ex: node rows, off the walls; ey, ez: half rows) of J_k E_k, J the step's
// normalised current (jacc * jscale), E the fields the step starts from.
// With jbar/fbar_e, also adds scale * E to the current adjoint and scale * J to
// the E adjoint (3 planes each, mx x S).
template <class T, class Acc>
__global__ void k_loss_jdote(int mx, int my, int S, int ybc, const void* jacc, double jscale, const T* ex,
                             const T* ey, const T* ez, double scale, double* loss, double* jbar, double* fbar_e) {
  __shared__ double red[32];
  const Acc* J = reinterpret_cast<const Acc*>(jacc);
  const long long plane = (long long)mx * S;
  const int rows = ybc == 0 ? my : my + 1;
  const long long n = (long long)mx * rows;
  double s = 0.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / rows), j = (int)(k - (long long)i * rows);
    const long long o = (long long)i * S + j;
    if (!(ybc == 1 && (j == 0 || j == my))) {
      const double jx = (double)J[o] * jscale, e = (double)ex[o];
      s += jx * e;
      if (jbar) {
        jbar[o] += scale * e;
        fbar_e[o] += scale * jx;
      }
    }
    if (j < my) {
      const double jy = (double)J[plane + o] * jscale, ey_ = (double)ey[o];
      const double jz = (double)J[2 * plane + o] * jscale, ez_ = (double)ez[o];
      s += jy * ey_ + jz * ez_;
      if (jbar) {
        jbar[plane + o] += scale * ey_;
        jbar[2 * plane + o] += scale * ez_;
        fbar_e[plane + o] += scale * jy;
        fbar_e[2 * plane + o] += scale * jz;
      }
    }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0 && loss) atomicAdd(loss, scale * s);
}

// d loss / d (Ti/Te) through the loaded momenta. The loader sets
// u = g uth(tau) + U(tau) (U: the sheet drift along z), so with g recovered
// from the loaded u, du/dtau = g duth/dtau + dU/dtau, contracted here with the
// adjoint of the initial momenta. Pair k = id/2: ion id even, electron id odd.
template <class T>
__global__ void k_dtau(int64_t n, int64_t nsheet, const int32_t* id, Comps<T> u, Comps<T> lam,
                       double uthi, double uthe, double duthi, double duthe, double udi, double ude,
                       double dudi, double dude, double* out) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const bool el = (id[p] & 1) != 0, sheet = (id[p] >> 1) < nsheet;
    const double uth = el ? uthe : uthi, duth = el ? duthe : duthi;
    const double U = sheet ? (el ? ude : udi) : 0.0, dU = sheet ? (el ? dude : dudi) : 0.0;
    const P5<T> v = ldg_part(u, p), l = ldg_part(lam, p);
    const double gx = (double)v.ux / uth, gy = (double)v.uy / uth, gz = ((double)v.uz - U) / uth;
    acc += (double)l.ux * gx * duth + (double)l.uy * gy * duth + (double)l.uz * (gz * duth + dU);
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

}  // namespace pbd
