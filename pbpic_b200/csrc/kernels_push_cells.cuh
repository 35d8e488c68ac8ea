// Particle push over cell-sorted input, cell by cell (both forms; the exact order and the
// compat switches keep the tile push of kernels_push.cuh).
//
// A group of L lanes takes one cell of the tile at a time and walks its
// particles L at a time, so that everything a cell's particles share is read
// once per cell: the gather coefficients stay in registers, the cell word is not
// decoded, and the 17 deposit sums of the cell are kept in registers and
// reduced over the group once per 8 of its passes. Consecutive lanes work on
// consecutive positions. The permutation entries and the particles come through
// a ring of asynchronous copies, two passes ahead each.
//
// A particle that leaves its cell deposits its two zig-zag segments, and moves
// its count to its new cell's bin, from a per-warp queue that is emptied 32
// particles at a time: crossers are 2-10 % of the particles, so that in
// the main pass their branch would run almost every time for one or two lanes.
//
// Mixed form's window: every value v (FP32, |v| below 2^15) is added in fixed point as
// hi * 2^16 + lo to two signed 32-bit shared sums, which native shared atomics
// update; a tile of more than 32767 particles uses the same memory as 64-bit
// sums. hi = v 2^16 rounded to nearest, so that both parts are exact and lo, |lo| <= 2^15, has
// the rounding that the 64-bit sum would give v. With at most 32767 particles neither
// sum can overflow. A particle takes part in at most two additions to an entry: a crosser's two segments can share a
// node (jx when it leaves through a y face, jy through an x face), and a cell's
// sums, one addition a chunk of at least one particle, hold jx and jy of the others only and jz and rho of all. So
//   |sum of lo| <= 2 * 32767 * 2^15 < 2^31;
//   |sum of hi| <= 32767 * (2^16 + 1) + rounding < 2^31,
// since what a particle adds to an entry is at most 1 in all (a move of less than a cell, a speed below c, a
// charge, each times a weight), each addition rounds by 1/2, and 32767 steps are left for the FP32 rounding.
// (The split at 2^17 of kernels_push.cuh, with lo >= 0, holds for one addition a particle only.)
//
// What bounds it, and why this form (512x256 Harris sheet, 26.2 M particles): the tile
// push of kernels_push.cuh takes 575 us, 14.7 warp instructions a
// particle at 65 % issue, a third of them moving registers, decoding cells and running
// the crossers' branch for one or two lanes. This form takes 357 us with
// 10.0 warp instructions a particle at 72 % issue: bound by instruction issue.
// On the way there, each with those before it: particles loaded into registers one pass ahead, 540 us and 45 % of
// the warps' time waiting for loads (the permutation entry, one pass
// ahead, then the particle: two DRAM latencies in one pass's time); dx, dy, ux, uy as one
// 16-byte record in place of four arrays, 450 us; the particles by asynchronous
// copies, 435 us at any depth, because the permutation entries still came one
// pass ahead; those through the ring too, 370 us; the species table and the crossers' one record below, 357 us. Blocks of 4 warps, 5 per SM at 96
// registers (4 per SM: 385 us; 6 per SM spill: 500 us). A species' constants come from a
// table in shared memory, with zero charge and mass for lanes beyond the cell, and a
// crosser is queued as one 16-byte record: 10.7 -> 10.0 instructions, step 453 -> 442 us.
// Shared memory beyond this (buffers padded to a power of two: 207 KB an SM) takes the
// L1 lines that the 4-byte copies share: 410 us.
//
// Plain form: the same with the coefficients read from shared memory in every pass (24 more
// FP64 registers would cost a block per SM) and no window: a cell's 17 sums and
// the crossers' 8 values go straight to the global current as reductions in L2 (FP64
// atomics in shared memory are compare-and-swap loops, on which the crossers of one cell
// collide). Its step on the same sheet: 1230 -> 703 us (the tile push 1041 us of it
// before); 3 blocks per SM at 146 registers (4 at 128: 758 us, but 1.5 % slower at 128x128 cells).
#pragma once
#include "kernels_push.cuh"

namespace pbd {

constexpr int PC_THREADS = PushThreads<float>::value, PC_WARPS = PC_THREADS / 32;
constexpr int PC_QUEUE = 64;  // crossers a warp holds: up to 31 left over and 32 more
constexpr int PC_CHUNK = 8;   // passes whose sums are kept in FP32 before they go to the window (FP64: any number)

// Dynamic shared memory: the window (mixed form), the new-cell histogram, 24
// gather coefficients of each row's cell.
__host__ __device__ __forceinline__ size_t cells_rec_offset(int ty, bool mixed) {
  return ((mixed ? (size_t)16 * (ty + 3) * 8 : 0) + (size_t)3 * (ty + 2) * 4 + 15) & ~(size_t)15;
}
__host__ __device__ __forceinline__ size_t cells_smem_bytes(int ty, bool mixed) {
  return cells_rec_offset(ty, mixed) + (size_t)ty * 24 * (mixed ? 4 : 8);
}

// rsqrt and quotient of normal positive arguments (1 <= x): the hardware estimates
// without the subnormal scaling.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_normal(float a, float b) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ double rsqrt_normal(double x) { return push_rsqrt(x); }
__device__ __forceinline__ float two_over(float x) { return div_normal(2.0f, x); }
__device__ __forceinline__ double two_over(double x) { return push_two_over(x); }
__device__ __forceinline__ float positive(float x) { return fmaxf(x, 0.0f); }
__device__ __forceinline__ double positive(double x) { return x > 0.0 ? x : 0.0; }
__device__ __forceinline__ float max_nan(float a, float b) {  // a NaN stays
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Passes on their way, a ring of 4 per warp (pass j in buffer j mod 4). In pass i a lane starts the copies
// (cp.async) of its particle of pass i + 2, whose element it reads from the ring, and of the
// permutation entry of pass i + 4; it waits for those it started in pass
// i - 2. A lane reads only what it copied itself.
constexpr int PC_STAGES = 4;
template <class T>
struct alignas(16) PassBuf {
  T quad[32][4];
  T uz[32];
  uint32_t cw[32];
  int32_t elem[32];
};
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void copy_small(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}
template <class T>
__device__ __forceinline__ void start_pass(const PushParams<T>& a, PassBuf<T>* buf, int lane, int e) {
  const T* src = a.c.q + 4 * (int64_t)e;
  copy16(&buf->quad[lane][0], src);
  if (sizeof(T) == 8) copy16(&buf->quad[lane][2], src + 2);
  copy_small<(int)sizeof(T)>(&buf->uz[lane], a.c.z + e);
  copy_small<4>(&buf->cw[lane], a.cell + e);
}
// The element of position p: an entry of the permutation, or p itself.
template <bool GATHER, class T>
__device__ __forceinline__ void start_elem(const PushParams<T>& a, PassBuf<T>* buf, int lane, int p) {
  if (GATHER) copy_small<4>(&buf->elem[lane], a.src + p);
  else buf->elem[lane] = p;
}
__device__ __forceinline__ void end_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <class T>
struct CellsSmem {
  PassBuf<T> pass[PC_WARPS][PC_STAGES];
  alignas(16) T q[PC_WARPS][PC_QUEUE][4];  // crossers: x, y before, x, y after the move
  int2 qw[PC_WARPS][PC_QUEUE];             // and the old cell's word, the position
  alignas(16) T spc[3][8];                 // ion, electron, no particle: c0, c1, q, its mass as an electron, as an ion
  int32_t off[65];                 // positions of the tile's cells
  double red[32];
  uint64_t mbar;
};

// The window, the new-cell histogram (shared-memory addresses), the tile's place and, in the
// plain form, the global current with the factors of unit-charge jx, jy.
struct CellsWin {
  int WR, TY;
  unsigned lo, hi, hist;
  bool split;
  int ixt, y0, mx, my, S, walls;
  double* jacc;
  double fx, fy;
  uint32_t* cell;  // where the pushed particles go
  void* quad;
};

__device__ __forceinline__ void shared_add(unsigned addr, unsigned v) {
  asm volatile("red.shared.add.u32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void win_add(const CellsWin& w, int idx, float v) {
  if (w.split) {  // v 2^32 = h 2^16 + l, h = v 2^16 rounded; s - h and its product are exact
    const float s = __fmul_rn(v, 65536.0f);
    const float h = rintf(s);
    shared_add(w.hi + 4 * idx, (unsigned)(int)h);
    shared_add(w.lo + 4 * idx, (unsigned)__float2int_rn(__fmul_rn(__fsub_rn(s, h), 65536.0f)));
  } else {
    asm volatile("red.shared.add.u64 [%0], %1;\n" ::"r"(w.lo + 8 * idx), "l"(to_acc<float, true>(v)) : "memory");
  }
}

// Value v of component c at window place (wx, wy), the node (ixt - 1 + wx, y0 - 1 + wy): to the
// window (mixed), or times `scale` to the global current by one reduction in L2
// (plain: FP64 shared atomics are compare-and-swap loops, and the crossers of a cell meet on the
// same nodes).
__device__ __forceinline__ void deposit_at(const CellsWin& w, int c, int wx, int wy, float v, double) {
  win_add(w, (c * 4 + wx) * w.WR + wy, v);
}
__device__ __forceinline__ void deposit_at(const CellsWin& w, int c, int wx, int wy, double v, double scale) {
  long long gi;
  int sg;
  if (map_current(c, w.ixt - 1 + wx, w.y0 - 1 + wy, w.mx, w.my, w.S, w.walls, 0, &gi, &sg))
    atomicAdd(&w.jacc[gi], sg < 0 ? -v * scale : v * scale);
}

// Cell step along one axis.
template <class T>
__device__ __forceinline__ int cell_step(T x) { return x > T(0.5) ? 1 : (x < T(-0.5) ? -1 : 0); }

__device__ __forceinline__ void get_quad(const float* p, float& a, float& b, float& c, float& d) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = v.x, b = v.y, c = v.z, d = v.w;
}
__device__ __forceinline__ void get_quad(const double* p, double& a, double& b, double& c, double& d) {
  const double2 u = reinterpret_cast<const double2*>(p)[0], v = reinterpret_cast<const double2*>(p)[1];
  a = u.x, b = u.y, c = v.x, d = v.y;
}
__device__ __forceinline__ void set_quad(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void set_quad(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}
__device__ __forceinline__ void put_xy(float* p, float x, float y) { *reinterpret_cast<float2*>(p) = make_float2(x, y); }
__device__ __forceinline__ void put_xy(double* p, double x, double y) { *reinterpret_cast<double2*>(p) = make_double2(x, y); }

// Empties `n` (<= 32) queued crossers, those at [first, first + n): both zig-zag segments
// (pic2d.f90:1237-1272) to the window, the count from the old cell's bin to the new
// one's, and with RESOLVE the new cell and the offsets in it (kernels_push.cuh: push_core)
// over what the pass stored. Returns the status bits.
template <class T, bool RESOLVE>
__device__ __noinline__ int drain_crossers(const CellsWin w, const T (*q)[4], const int2* qw, int first, int n) {
  const int lane = (int)lane_id();
  int status = 0;
  __syncwarp();
  if (lane < n) {
    const int e = first + lane;
    T px, py, x1, y1;
    get_quad(q[e], px, py, x1, y1);
    const int2 wp = qw[e];
    const uint32_t wrd = (uint32_t)wp.x;
    const int iy = cw_iy(wrd), key = iy - w.y0, dcx = cell_step(x1), dcy = cell_step(y1);
    if (M<T, true>::abs(x1) > T(1.5) || M<T, true>::abs(y1) > T(1.5)) status = PBPIC_STATUS_CELL_JUMP;
    const bool refl = w.walls && (unsigned)(iy + dcy) >= (unsigned)w.my;
    if (RESOLVE) {
      int nix = w.ixt + dcx, niy = refl ? iy : iy + dcy;
      nix = nix < 0 ? nix + w.mx : (nix >= w.mx ? nix - w.mx : nix);
      niy = niy < 0 ? niy + w.my : (niy >= w.my ? niy - w.my : niy);
      T* out = static_cast<T*>(w.quad) + 4 * (int64_t)wp.y;
      const T ny = M<T, true>::sub(y1, (T)dcy);
      put_xy(out, M<T, true>::sub(x1, (T)dcx), refl ? -ny : ny);
      if (refl) out[3] = -out[3];
      w.cell[wp.y] = (wrd & 0x80000000u) | ((uint32_t)nix << 16) | (uint32_t)niy;
    }
    const int row1 = refl ? key : key + dcy;  // a reflected particle keeps its row
    const T qq = (int)wrd < 0 ? T(-1) : T(1), half = T(0.5), one = T(1);
    using A = M<T, true>;
    const T fdcx = (T)dcx, fdcy = (T)dcy;
    const T xs = A::add(px, half), xe = A::add(x1, half), ys = A::add(py, half), ye = A::add(y1, half);
    const T im = A::mul(A::add(xs, xe), half), jm = A::mul(A::add(ys, ye), half);
    const T ir = dcx == 0 ? im : (dcx > 0 ? one : T(0)), jr = dcy == 0 ? jm : (dcy > 0 ? one : T(0));
    const T fx1 = A::mul(qq, A::sub(ir, xs)), fx2 = A::mul(qq, A::sub(xe, ir));
    const T fy1 = A::mul(qq, A::sub(jr, ys)), fy2 = A::mul(qq, A::sub(ye, jr));
    const T wx1 = A::mul(A::add(ir, xs), half), wy1 = A::mul(A::add(jr, ys), half);
    const T wx2 = A::sub(A::mul(A::add(ir, xe), half), fdcx), wy2 = A::sub(A::mul(A::add(jr, ye), half), fdcy);
    const int k1 = key + 1, k2 = k1 + dcy;
    deposit_at(w, JX, 1, k1, A::mad(-fx1, wy1, fx1), w.fx);
    deposit_at(w, JX, 1, k1 + 1, A::mul(fx1, wy1), w.fx);
    deposit_at(w, JX, 1 + dcx, k2, A::mad(-fx2, wy2, fx2), w.fx);
    deposit_at(w, JX, 1 + dcx, k2 + 1, A::mul(fx2, wy2), w.fx);
    deposit_at(w, JY, 1, k1, A::mad(-fy1, wx1, fy1), w.fy);
    deposit_at(w, JY, 2, k1, A::mul(fy1, wx1), w.fy);
    deposit_at(w, JY, 1 + dcx, k2, A::mad(-fy2, wx2, fy2), w.fy);
    deposit_at(w, JY, 2 + dcx, k2, A::mul(fy2, wx2), w.fy);
    const int b0 = (w.TY + 2) + key + 1, b1 = (1 + dcx) * (w.TY + 2) + row1 + 1;
    if (b0 != b1) {
      shared_add(w.hist + 4 * b1, 1u);
      shared_add(w.hist + 4 * b0, (unsigned)-1);
    }
  }
  __syncwarp();
  return status;
}

// The 17 stencil entries (kernels_push.cuh: stencil_node) of the accumulated
// moments of the push's deposit: jx and jy with the midpoint's offset h/2 from
// the cell centre, jz with weights twice their size on either axis, rho
// from the moments of the charge. (200 particles summed so against extended precision, relative
// error in FP64: jx 1.5e-16, with its terms formed from x + 1/2 as in the tile
// push 9e-16; rho 1.0e-16 to 1.7e-16, its 4 products summed 0.7e-16 to 8.4e-16.)
template <class T>
__device__ __forceinline__ void cell_terms(const T (&m)[17], T (&v)[16], T& v16) {
  using A = M<T, true>;
  v[0] = A::mul(T(0.5), A::sub(m[0], m[1]));
  v[1] = A::mul(T(0.5), A::add(m[0], m[1]));
  v[2] = A::mul(T(0.5), A::sub(m[2], m[3]));
  v[3] = A::mul(T(0.5), A::add(m[2], m[3]));
#pragma unroll
  for (int k = 4; k < 13; ++k) v[k] = A::mul(T(0.25), m[k]);
  const T a = A::mad(T(0.25), m[13], m[16]), b = A::mad(T(0.25), m[13], -m[16]);
  const T c = A::mul(T(0.5), A::add(m[14], m[15])), d = A::mul(T(0.5), A::sub(m[14], m[15]));
  v[13] = A::sub(a, c);
  v[14] = A::add(b, d);
  v[15] = A::sub(b, d);
  v16 = A::add(a, c);
}

// Sums v[0..15] over the L lanes of a group by recursive halving: v[0] is then the total
// of entry (lane of the group) * 16 / L (L = 32: the same one in both lanes of a pair).
template <int L, class T>
__device__ __forceinline__ void group_sums(T (&v)[16]) {
  const unsigned lane = lane_id();
  int n = 16;
#pragma unroll
  for (int d = L / 2; d > 0; d >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = (lane & d) != 0;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n) {
          const T give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
          v[i] = add_rn(keep, __shfl_xor_sync(FULL, give, d));
        }
    } else {
      v[0] = add_rn(v[0], __shfl_xor_sync(FULL, v[0], d));
    }
  }
}

// Bilinear coefficients (A, B, C, D) of the 6 fields over a cell, from the node grid
// (kernels_field.cuh: cell_record). A is the correctly rounded mean (its sums' rounding errors are carried), and
// coef_at adds it last, so that the gather is no further off than the sum of four
// weighted nodes: rms error 6.9e-17 of the field against 7.4e-17 for nodes that differ by a tenth,
// 7.8e-17 against 7.9e-17 for uncorrelated Yee values averaged to nodes (9.9e-17 with a plain
// mean added first).
__device__ __forceinline__ void cell_coefs(const PushParams<double>& a, int ix, int iy, int f, double* r) {
  const double* g = a.ng + ((long long)ix * (a.my + 1) + iy) * 8 + (f < 3 ? f : f + 1);
  const double* h = g + (long long)(a.my + 1) * 8;
  const double n00 = __ldg(g), n01 = __ldg(g + 8), n10 = __ldg(h), n11 = __ldg(h + 8);
  auto err = [](double a, double b, double s) {  // a + b - s, s = a + b rounded (Knuth's two-sum)
    const double t = s - a;
    return (a - (s - t)) + (b - t);
  };
  const double s0 = n00 + n01, s1 = n10 + n11, s = s0 + s1;
  r[0] = 0.25 * (s + (err(s0, s1, s) + (err(n00, n01, s0) + err(n10, n11, s1))));
  r[1] = 0.5 * ((n10 - n00) + (n11 - n01));
  r[2] = 0.5 * ((n01 - n00) + (n11 - n10));
  r[3] = (n11 - n10) - (n01 - n00);
}
__device__ __forceinline__ double coef_at(const double* r, double x, double y) {
  const double2 ab = reinterpret_cast<const double2*>(r)[0], cd = reinterpret_cast<const double2*>(r)[1];
  return __dadd_rn(__fma_rn(__fma_rn(cd.y, x, cd.x), y, __dmul_rn(ab.y, x)), ab.x);
}

// Push of tile t by all threads of the block (kernels_push.cuh: push_tile).
template <class T, int L, bool GATHER, bool PID>
__device__ __forceinline__ void push_cells(const PushParams<T>& a, const int t, CellsSmem<T>& sm,
                                           unsigned char* smem_raw, unsigned parity) {
  using A = M<T, true>;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int GRP = 32 / L;
  // Where a crosser's new cell is found: in the queue, whose 32 lanes are all crossers, or in the pass, where one
  // or two lanes of 32 are. The first saves instructions (20 of 330 a pass) but writes a crosser twice. Step,
  // queue against pass: 64x64 cells 36.0/37.3 us, 193x131 74.4/77.8, FP64 128x128 80.7/82.3, 512x256 703/708; but
  // at 200 particles a cell, 512x256 FP32 455/444 us: there the extra writes cost more than the instructions.
  constexpr bool LATE = L == 16 || !F32;
  const T half = T(0.5), one = T(1);
  CellsWin w;
  w.TY = a.tile_rows;
  w.WR = w.TY + 3;
  unsigned* lo = reinterpret_cast<unsigned*>(smem_raw);
  int* hi = reinterpret_cast<int*>(lo + 16 * w.WR);
  int* hist = F32 ? hi + 16 * w.WR : reinterpret_cast<int*>(smem_raw);
  T* rec = reinterpret_cast<T*>(smem_raw + cells_rec_offset(w.TY, F32));
  const int ixt = t / a.tiles_per_col;
  const int y0 = (t - ixt * a.tiles_per_col) * w.TY, y1 = min(y0 + w.TY, a.my), nrow = y1 - y0;
  const long long cell0 = (long long)ixt * a.my + y0;
  w.lo = smem_addr(lo);
  w.hi = smem_addr(hi);
  w.hist = smem_addr(hist);
  w.ixt = ixt;
  w.y0 = y0;
  w.mx = a.mx;
  w.my = a.my;
  w.S = a.S;
  w.walls = a.ybc;
  w.jacc = reinterpret_cast<double*>(a.jacc);
  w.fx = F32 ? 1.0 : (double)a.qx[0];
  w.fy = F32 ? 1.0 : (double)a.qy[0];
  w.cell = GATHER ? a.cell_o : a.cell;
  w.quad = GATHER ? a.c_o.q : a.c.q;
  if constexpr (F32) {
    if (threadIdx.x == 0) {  // the records of the tile's cells: one bulk copy
      const unsigned bytes = (unsigned)nrow * 96u;
      bulk_expect(&sm.mbar, bytes);
      bulk_copy(rec, a.cg + cell0 * 24, bytes, &sm.mbar);
    }
    for (int e = threadIdx.x; e < 32 * w.WR; e += PC_THREADS) lo[e] = 0u;
  } else {
    for (int e = threadIdx.x; e < 6 * nrow; e += PC_THREADS) {
      const int f = e / nrow, r = e - f * nrow;
      cell_coefs(a, ixt, y0 + r, f, rec + r * 24 + f * 4);
    }
  }
  for (int e = threadIdx.x; e <= nrow; e += PC_THREADS) sm.off[e] = a.cell_off[cell0 + e];
  for (int e = threadIdx.x; e < 3 * (w.TY + 2); e += PC_THREADS) {  // the counts before any particle moved
    const int by = e - (w.TY + 2);
    hist[e] = by >= 1 && by <= nrow ? a.cell_off[cell0 + by] - a.cell_off[cell0 + by - 1] : 0;
  }
  if (threadIdx.x < 3) {
    T* sp = sm.spc[threadIdx.x];
    const int k = threadIdx.x;
    sp[0] = k == 2 ? T(0) : a.c0[k & 1];
    sp[1] = k == 2 ? T(0) : a.c1[k & 1];
    sp[2] = k == 2 ? T(0) : (k == 1 ? T(-1) : one);
    sp[3] = k == 1 ? a.ms[1] : T(0);
    sp[4] = k == 0 ? a.ms[0] : T(0);
  }
  __syncthreads();
  w.split = sm.off[nrow] - sm.off[0] <= 32767;
  const int plast = sm.off[nrow] - 1;
  [[maybe_unused]] const bool edge = ixt == 0 || ixt == a.mx - 1 || y0 == 0 || y1 == a.my;  // a step may leave the domain
  bool staged = true;
  if constexpr (F32) staged = mbar_wait(&sm.mbar, parity);
  const int lane = (int)lane_id(), wp = threadIdx.x >> 5;
  const int grp = lane / L, gl = lane % L;
  T(*q)[4] = sm.q[wp];
  int2* qw = sm.qw[wp];
  int nq = 0;
  // this lane's entry of the stencil once a group's sums are spread over its lanes (L = 32: a pair
  // of lanes holds the same sum, lane 1 takes the last entry)
  int sc, sx0, sy0;
  stencil_node(L == 32 && lane == 1 ? 16 : gl * 16 / L, &sc, &sx0, &sy0);
  const double sscale = F32 ? 1.0 : (sc == JX ? w.fx : (sc == JY ? w.fy : (sc == JZ ? (double)a.cva : 1.0)));
  double ke_e = 0.0, ke_i = 0.0;
  int status = staged ? 0 : PBPIC_STATUS_COPY_TIMEOUT;

  // Rounds: round r gives the warp the rows (4 r + wp) GRP + group; a pass takes L
  // particles of each. Cursor C is the pass at work, cursor A four passes ahead.
  const int nround = (nrow + PC_WARPS * GRP - 1) / (PC_WARPS * GRP);
  struct Cursor {
    int rd, left, row, p, end;
  };
  auto next_round = [&](Cursor& k) {  // to the next round with particles; left = 0 after the last
    k.left = 0;
    while (k.left == 0 && k.rd + 1 < nround) {
      ++k.rd;
      k.row = (PC_WARPS * k.rd + wp) * GRP + grp;
      k.p = k.end = 0;
      if (k.row < nrow) {
        k.p = sm.off[k.row];
        k.end = sm.off[k.row + 1];
      }
      k.left = (k.end - k.p + L - 1) / L;
      if (GRP > 1) k.left = __reduce_max_sync(FULL, k.left);
      k.p += gl;
    }
    if (k.left == 0) k.p = k.end = 0, k.left = 0x7fffffff;
  };
  // position of the cursor's pass (lanes beyond the cell: the particles after it), and the cursor moved on
  auto take = [&](Cursor& k) -> int {
    const int p = min(k.p, plast);
    k.p += L;
    if (--k.left == 0) next_round(k);
    return p;
  };
  Cursor kc{-1, 0, 0, 0, 0};
  next_round(kc);
  if (kc.left != 0x7fffffff) {
    Cursor ka = kc;
    PassBuf<T>* ring = &sm.pass[wp][0];
    {
      const int p0 = take(ka), p1 = take(ka);
      const int e0 = GATHER ? __ldg(a.src + p0) : p0, e1 = GATHER ? __ldg(a.src + p1) : p1;
      ring[0].elem[lane] = e0;  // (read again in the pass itself for tracked ids)
      ring[1].elem[lane] = e1;
      start_pass(a, ring, lane, e0);
      start_elem<GATHER>(a, ring + 2, lane, take(ka));
      end_group();
      start_pass(a, ring + 1, lane, e1);
      start_elem<GATHER>(a, ring + 3, lane, take(ka));
      end_group();
    }
    unsigned at = 0;  // the pass's buffer: a byte offset in the ring
    constexpr unsigned STRIDE = sizeof(PassBuf<T>);
    auto buf = [&](unsigned o) -> PassBuf<T>* {
      return reinterpret_cast<PassBuf<T>*>(reinterpret_cast<unsigned char*>(ring) + o);
    };
    T acc[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) acc[k] = T(0);
    T pke_e = T(0), pke_i = T(0);
    do {  // one round's cells
      float4 c[6];  // mixed: the cell's coefficients
      const T* rc = rec + min(kc.row, nrow - 1) * 24;  // plain: read from shared memory in every pass
      if constexpr (F32) {
        const int r = min(kc.row, nrow - 1);
        if (staged) {
          const float4* rp = reinterpret_cast<const float4*>(rec + r * 24);
#pragma unroll
          for (int k = 0; k < 6; ++k) c[k] = rp[k];
        } else {
          const float4* rp = reinterpret_cast<const float4*>(a.cg + (cell0 + r) * 24);
#pragma unroll
          for (int k = 0; k < 6; ++k) c[k] = __ldg(rp + k);
        }
      }
      const int row = kc.row, end = kc.end;
      int p = kc.p, left = kc.left;
      while (left > 0) {
        int chunk = F32 ? min(left, PC_CHUNK) : left;
        left -= chunk;
        do {
          asm volatile("cp.async.wait_group 1;\n" ::: "memory");
          const PassBuf<T>& in = *buf(at);
          T quad[4];
          get_quad(in.quad[lane], quad[0], quad[1], quad[2], quad[3]);
          const uint32_t wrd = in.cw[lane];
          const T px = quad[0], py = quad[1], uz_in = in.uz[lane];
          const int elem = in.elem[lane];  // (tracked ids)
          PassBuf<T>* ahead = buf(at >= 2 * STRIDE ? at - 2 * STRIDE : at + 2 * STRIDE);
          start_pass(a, ahead, lane, ahead->elem[lane]);
          start_elem<GATHER>(a, buf(at), lane, take(ka));
          end_group();
          at = at == 3 * STRIDE ? 0u : at + STRIDE;
          const bool valid = p < end;
          const T* sp = sm.spc[valid ? (int)(wrd >> 31) : 2];
          // gather and Boris rotation (kernels_push.cuh: push_core, the same operations)
          T ex, ey, ez, bx, by, bz;
          if constexpr (F32) {
            ex = coef_at(c[0], px, py), ey = coef_at(c[1], px, py), ez = coef_at(c[2], px, py);
            bx = coef_at(c[3], px, py), by = coef_at(c[4], px, py), bz = coef_at(c[5], px, py);
          } else {
            ex = coef_at(rc, px, py), ey = coef_at(rc + 4, px, py), ez = coef_at(rc + 8, px, py);
            bx = coef_at(rc + 12, px, py), by = coef_at(rc + 16, px, py), bz = coef_at(rc + 20, px, py);
          }
          T c0, c1, qv, me;
          get_quad(sp, c0, c1, qv, me);
          const T mi = sp[4];
          const T umx = A::mad(c1, ex, quad[2]), umy = A::mad(c1, ey, quad[3]), umz = A::mad(c1, ez, uz_in);
          const T g2m = A::mad(umz, umz, A::mad(umy, umy, A::mad(umx, umx, one)));
          const T c2 = A::mul(c0, rsqrt_normal(g2m));
          const T tx = A::mul(c2, bx), ty = A::mul(c2, by), tz = A::mul(c2, bz);
          const T t2 = two_over(A::mad(tz, tz, A::mad(ty, ty, A::mad(tx, tx, one))));
          const T sx = A::mul(t2, tx), sy = A::mul(t2, ty), sz = A::mul(t2, tz);
          const T u0x = A::mad(umy, tz, A::mad(-umz, ty, umx));
          const T u0y = A::mad(umz, tx, A::mad(-umx, tz, umy));
          const T u0z = A::mad(umx, ty, A::mad(-umy, tx, umz));
          const T upx = A::mad(u0y, sz, A::mad(-u0z, sy, umx));
          const T upy = A::mad(u0z, sx, A::mad(-u0x, sz, umy));
          const T upz = A::mad(u0x, sy, A::mad(-u0y, sx, umz));
          const T ux = A::mad(c1, ex, upx), uz = A::mad(c1, ez, upz); T uy = A::mad(c1, ey, upy);
          const T g2 = A::mad(uz, uz, A::mad(uy, uy, A::mad(ux, ux, one)));
          const T rg = rsqrt_normal(g2), gama = A::mul(g2, rg), c3 = A::mul(a.dtcva, rg);
          T x1 = A::mad(A::mul(c3, ux), a.idx, px), y1 = A::mad(A::mul(c3, uy), a.idy, py);
          // the cell is left when either offset passes 1/2 (a NaN counts as leaving)
          bool cross;
          if constexpr (F32) cross = valid && !(max_nan(fabsf(x1), fabsf(y1)) <= 0.5f);
          else cross = valid && !(fabs(x1) <= 0.5 && fabs(y1) <= 0.5);
          if constexpr (F32) {  // kinetic energy: (gamma - 1) m = u^2 m / (gamma + 1)
            const float usq = A::mad(uz, uz, A::mad(uy, uy, A::mul(ux, ux)));
            const float ke = div_normal(usq, A::add(gama, 1.0f));
            pke_e = A::mad(ke, me, pke_e);
            pke_i = A::mad(ke, mi, pke_i);
          } else {
            const T ke = A::sub(gama, one);
            pke_e = A::mad(ke, me, pke_e);
            pke_i = A::mad(ke, mi, pke_i);
          }
          {  // deposit (pic2d.f90:1237-1295), cell-relative and for unit charges: the whole move of a particle that stays
            const T qs = cross ? T(0) : qv;
            // twice the midpoint, from the cell centre; the factors 1/2 and the constant parts of the weights
            // enter with the cell's sums (cell_terms)
            const T hx = A::add(px, x1), hy = A::add(py, y1);
            const T ja = A::mul(qs, A::sub(x1, px)), jb = A::mul(qs, A::sub(y1, py));
            acc[0] = A::add(acc[0], ja);
            acc[1] = A::mad(ja, hy, acc[1]);
            acc[2] = A::add(acc[2], jb);
            acc[3] = A::mad(jb, hx, acc[3]);
            // jz: outer product of the weights of x and y = -1, 0, 1 about the cell
            const T quz = A::mul(qv, A::mul(uz, rg));
            const T ax = A::abs(hx), ay = A::abs(hy);
            const T xp = positive(hx), xm = A::sub(xp, hx), yp = positive(hy), ym = A::sub(yp, hy);
            const T y0w = A::sub(T(2), ay), x0w = A::sub(T(2), ax);
            const T qxm = A::mul(quz, xm), qxp = A::mul(quz, xp), qx0 = A::mul(quz, x0w);
            acc[4] = A::mad(qxm, ym, acc[4]);
            acc[5] = A::mad(qxm, y0w, acc[5]);
            acc[6] = A::mad(qxm, yp, acc[6]);
            acc[7] = A::mad(qx0, ym, acc[7]);
            acc[8] = A::mad(qx0, y0w, acc[8]);
            acc[9] = A::mad(qx0, yp, acc[9]);
            acc[10] = A::mad(qxp, ym, acc[10]);
            acc[11] = A::mad(qxp, y0w, acc[11]);
            acc[12] = A::mad(qxp, yp, acc[12]);
            // rho at the old position: the moments 1, x, y, x y of the charge
            const T qx = A::mul(qv, px);
            acc[13] = A::add(acc[13], qv);
            acc[14] = A::add(acc[14], qx);
            acc[15] = A::mad(qv, py, acc[15]);
            acc[16] = A::mad(qx, py, acc[16]);
          }
          const unsigned mc = __ballot_sync(FULL, cross);
          uint32_t cw = wrd;
          if (cross) {  // LATE: stored as it is, its new cell comes with the queue
            const int e = nq + __popc(mc & lanemask_lt());
            set_quad(q[e], px, py, x1, y1);
            qw[e] = make_int2((int)wrd, p);
            if constexpr (!LATE) {
              const int dcx = cell_step(x1), dcy = cell_step(y1);
              x1 = A::sub(x1, (T)dcx);
              y1 = A::sub(y1, (T)dcy);
              cw = wrd + (uint32_t)(dcx * 65536 + dcy);
              if (edge) {  // boundaries (kernels_push.cuh: push_core)
                int nix = ixt + dcx, niy = y0 + row + dcy;
                nix = nix < 0 ? nix + a.mx : (nix >= a.mx ? nix - a.mx : nix);
                if (a.ybc == 0) {
                  niy = niy < 0 ? niy + a.my : (niy >= a.my ? niy - a.my : niy);
                } else if (niy < 0 || niy >= a.my) {
                  niy = niy < 0 ? 0 : a.my - 1;
                  y1 = -y1;
                  uy = -uy;
                }
                cw = (wrd & 0x80000000u) | ((uint32_t)nix << 16) | (uint32_t)niy;
              }
            }
          }
          if (valid) {
            (GATHER ? a.cell_o : a.cell)[p] = cw;
            put_part(GATHER ? a.c_o : a.c, p, P5<T>{x1, y1, ux, uy, uz});
            if (PID && a.pid_o) a.pid_o[p] = __ldg(a.pid_i + elem);
          }
          p += L;
          nq += __popc(mc);
          if (nq >= 32) {
            nq -= 32;
            status |= drain_crossers<T, LATE>(w, q, qw, nq, 32);
          }
        } while (--chunk > 0);
        // the cell's sums so far to the window
        T v[16], v16;
        cell_terms(acc, v, v16);
        group_sums<L>(v);
#pragma unroll
        for (int d = L / 2; d > 0; d >>= 1) v16 = add_rn(v16, __shfl_xor_sync(FULL, v16, d));
        if (row < nrow) {
          if (L == 32) {
            const T x = lane == 1 ? v16 : v[0];
            if (((lane & 1) == 0 || lane == 1) && x != T(0)) deposit_at(w, sc, 1 + sx0, row + 1 + sy0, x, sscale);
          } else {
            if (v[0] != T(0)) deposit_at(w, sc, 1 + sx0, row + 1 + sy0, v[0], sscale);
            if (gl == 0 && v16 != T(0)) deposit_at(w, RHO, 2, row + 2, v16, 1.0);
          }
        }
#pragma unroll
        for (int k = 0; k < 17; ++k) acc[k] = T(0);
        if (!(pke_e + pke_i < T(3.0e38))) status |= PBPIC_STATUS_NAN;  // a momentum whose gamma is not finite
        ke_e += (double)pke_e;
        ke_i += (double)pke_i;
        pke_e = pke_i = T(0);
      }
      next_round(kc);
    } while (kc.left != 0x7fffffff);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  }
  if (nq) status |= drain_crossers<T, LATE>(w, q, qw, 0, nq);
  if (F32 && !staged) mbar_wait(&sm.mbar, parity);  // not in flight when the shared memory is reused

  // fold the window into the global current; the tile's counts and energies
  __syncthreads();
  if constexpr (F32) {
    long long* gacc = reinterpret_cast<long long*>(a.jacc);
    for (int e = threadIdx.x; e < 16 * w.WR; e += PC_THREADS) {
      const long long val = w.split ? (long long)hi[e] * 65536 + (int)lo[e] : reinterpret_cast<const long long*>(lo)[e];
      if (val == 0) continue;
      const int cmp = e / (4 * w.WR), r = e - cmp * 4 * w.WR, wx = r / w.WR, wy = r - wx * w.WR;
      long long gi;
      int sg;
      if (map_current(cmp, ixt - 1 + wx, y0 - 1 + wy, a.mx, a.my, a.S, a.ybc, a.compat, &gi, &sg))
        acc_add(&gacc[gi], sg < 0 ? -val : val);
    }
  }
  const int nb = 3 * (w.TY + 2);
  for (int e = threadIdx.x; e < nb; e += PC_THREADS) a.tilecnt[(long long)t * nb + e] = hist[e];
  const double se = block_sum(ke_e, sm.red), si = block_sum(ke_i, sm.red);
  if (threadIdx.x == 0) {
    a.ke_part[2 * t] = se;
    a.ke_part[2 * t + 1] = si;
  }
  status = __reduce_or_sync(FULL, status);
  if (lane == 0 && status) atomicOr(a.status, status);
}

// Resident blocks per SM the registers must allow.
#ifndef PBPIC_CELLS_MINBLOCKS
#define PBPIC_CELLS_MINBLOCKS 5
#endif
#ifndef PBPIC_CELLS_MINBLOCKS_FP64
#define PBPIC_CELLS_MINBLOCKS_FP64 3
#endif
constexpr int cells_minblocks(bool f32) { return f32 ? PBPIC_CELLS_MINBLOCKS : PBPIC_CELLS_MINBLOCKS_FP64; }

// Single domain: one block per tile.
template <class T, int L, bool GATHER, bool PID>
__global__ void __launch_bounds__(PC_THREADS, cells_minblocks(sizeof(T) == 4)) k_push_cells(PushParams<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ CellsSmem<T> sm;
  if (sizeof(T) == 4 && threadIdx.x == 0) mbar_init(&sm.mbar);
  cudaTriggerProgrammaticLaunchCompletion();  // (pbpic_api.cu: launch_early)
  push_cells<T, L, GATHER, PID>(a, blockIdx.x, sm, smem_raw, 0u);
}

// Batched domains: persistent blocks take (domain, tile) pairs from a global
// counter (reset to 0 before each launch) in the order of `tiles`.
template <bool PID>
__global__ void __launch_bounds__(PC_THREADS, PBPIC_CELLS_MINBLOCKS)
    k_push_cells_batched(const PushParams<float>* descs, const int2* tiles, int ntiles, int* counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ CellsSmem<float> sm;
  __shared__ PushParams<float> a;
  __shared__ int next;
  if (threadIdx.x == 0) mbar_init(&sm.mbar);
  unsigned parity = 0;
  while (true) {
    if (threadIdx.x == 0) next = atomicAdd(counter, 1);
    __syncthreads();
    const int t = next;
    if (t >= ntiles) break;
    const int2 it = tiles[t];
    if (threadIdx.x == 0) a = descs[it.x];
    __syncthreads();
    if (a.lanes == 32) push_cells<float, 32, true, PID>(a, it.y, sm, smem_raw, parity);
    else push_cells<float, 16, true, PID>(a, it.y, sm, smem_raw, parity);
    parity ^= 1u;
    __syncthreads();
  }
}

}  // namespace pbd
