// Differentiable form of the step (include/pbpic.h, pbpic_diff_*): a
// checkpointed forward run of the GEM Harris sheet and the discrete adjoint of
// every step (kernels_adjoint.cuh), giving d loss / d (psi0, nb, Ti/Te).
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/pbpic.h"
#include "api_internal.h"
#include "kernels_adjoint.cuh"
#include "kernels_field.cuh"
#include "kernels_misc.cuh"
#include "pic_common.h"
#include "pic_fields_init.h"

using namespace pbd;

namespace {

#define DCK(call)                                                                                       \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess)                                                                              \
      return pbpic_internal_fail(PBPIC_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
  } while (0)
#define DLAUNCH(what)                                                                                   \
  do {                                                                                                  \
    pbpic_internal_count_launch();                                                                      \
    cudaError_t e_ = cudaGetLastError();                                                                \
    if (e_ != cudaSuccess)                                                                              \
      return pbpic_internal_fail(PBPIC_ECUDA, std::string(what) + ": " + cudaGetErrorString(e_));       \
  } while (0)
#define DTRY(...)                  \
  do {                             \
    int r_ = (__VA_ARGS__);        \
    if (r_ != PBPIC_OK) return r_; \
  } while (0)

int grid_of(int64_t n, int maxblocks = 148 * 8) {
  int64_t g = (n + 255) / 256;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, maxblocks));
}

// One stored state: particles and Yee fields.
struct Slot {
  void* p = nullptr;  // records of 4 T and uz (T), cell words and ids (a checkpoint) or the permutation (4 B each)
  void* f = nullptr;  // 6 planes of T
};

}  // namespace

struct pbpic_diff {
  pbpic_diff_config cfg;
  bool f32 = false;
  size_t tsz = 8;
  int mx = 0, my = 0, S = 0;
  int64_t n = 0, npairs = 0, nsheet = 0;
  double dx = 0, dy = 0, dt = 0, cva = 0, in0 = 0;
  int nseg = 0;
  // The states that exist at once. What a state holds beside its particles and fields is kept only where
  // it cannot be had again: a checkpoint's permutation and every node grid are formed when the
  // state is opened, a state's ids only where the order is left (checkpoints; the two newest states), whether a
  // particle is background in its permutation entry, and a state's adjoint takes its particles' place.
  std::vector<Slot> ck;   // checkpoints: state at steps 0, K, 2K, ...
  std::vector<Slot> seg;  // [1..K-1]: the states between two checkpoints, of the segment at work
  Slot fin;               // magnetic loss: fields of the last state (no push reads its particles)
  int32_t* ckperm = nullptr;                // the open checkpoint's permutation
  int32_t* ids[2] = {nullptr, nullptr};     // ids of the newest even and odd state of the segment
  void* ng = nullptr;                       // node grid of the state before step ng_at
  int ng_at = -1;
  void* jacc[2] = {nullptr, nullptr};  // 4 planes of 8-byte accumulators; [0] is clear before a push
  double* fe_part = nullptr;
  int nfe = 0;
  int32_t *rank = nullptr, *counts = nullptr, *off = nullptr, *sums = nullptr;  // cell order of a new state
  bool last_seg = false;  // seg holds the states of the forward run's last segment
  void* lam[2] = {nullptr, nullptr};  // particle adjoints of a checkpoint (the second for K = 1): records of 4 T, then uz
  double* fbar = nullptr;  // 6 adjoint planes (ex ey ez bx by bz)
  double* jbar = nullptr;  // 3 planes
  double* gbar = nullptr;  // node adjoint
  double* scal = nullptr;  // [0] loss, [1] d loss / d omega, [2] d loss / d tau, [3] d loss / d psi0
  void* jseg = nullptr;    // j.E loss: the current of each step of the recomputed segment (3 planes each)
  pbpic_diff_params last{};
  bool have_forward = false;
  std::vector<void*> allocs;
};

namespace {

int dmalloc(pbpic_diff* d, void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, std::max<size_t>(bytes, 16));
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    pbpic_internal_trim();
    e = cudaMalloc(p, std::max<size_t>(bytes, 16));
  }
  if (e != cudaSuccess)
    return pbpic_internal_fail(PBPIC_ENOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  d->allocs.push_back(*p);
  return PBPIC_OK;
}

size_t part_bytes(const pbpic_diff* d) { return (size_t)d->n * (8 + 5 * d->tsz); }
size_t field_bytes(const pbpic_diff* d) { return (size_t)6 * d->mx * d->S * d->tsz; }
size_t node_bytes(const pbpic_diff* d) { return (size_t)(d->mx + 1) * (d->my + 1) * 8 * d->tsz; }
int64_t plane(const pbpic_diff* d) { return (int64_t)d->mx * d->S; }

template <class T>
struct View {
  DiffState<T> p;
  T* f[6];
};

template <class T>
Comps<T> comps(const pbpic_diff* d, void* p) {
  return Comps<T>{(T*)p, (T*)p + (size_t)4 * d->n};
}

// The state before step it (it = nsteps: the last state's fields).
template <class T>
View<T> state(const pbpic_diff* d, int it) {
  const int K = d->cfg.checkpoint_every;
  const bool final = it == d->cfg.nsteps, ck = !final && it % K == 0;
  const Slot& s = final ? d->fin : (ck ? d->ck[it / K] : d->seg[it % K]);
  View<T> v{};
  if (!final) {
    v.p.c = comps<T>(d, s.p);
    v.p.cell = (uint32_t*)((T*)s.p + (size_t)5 * d->n);
    int32_t* last = (int32_t*)(v.p.cell + d->n);
    v.p.id = ck ? last : d->ids[it & 1];
    v.p.perm = ck ? d->ckperm : last;
  }
  for (int k = 0; k < 6; ++k) v.f[k] = (T*)s.f + (size_t)k * plane(d);
  return v;
}

struct Harris {
  double vthe, vthi, ude, udi;  // thermal speeds and drifts (units of c)
};

Harris harris_speeds(const pbpic_diff* d, double tite) {
  const pbpic_diff_config& c = d->cfg;
  const double te = 1.0 / (2.0 * (1.0 + tite));
  Harris h;
  h.vthe = sqrt(c.mime * te) / d->cva;
  h.vthi = h.vthe * sqrt(tite / c.mime);
  const double du = -1.0 / (c.lambda * d->cva);
  h.udi = du * tite / (1.0 + tite);
  h.ude = -du / (1.0 + tite);
  return h;
}

double urel(double v) { return v / sqrt(1.0 - v * v); }
double durel(double v) { return 1.0 / pow(1.0 - v * v, 1.5); }

template <class T>
PushParams<T> push_params(const pbpic_diff* d) {
  PushParams<T> p;
  memset(&p, 0, sizeof(p));
  p.mx = d->mx;
  p.my = d->my;
  p.S = d->S;
  p.ybc = PBPIC_BC_CONDUCTING;
  p.compat = 0;
  p.ng = (const T*)d->ng;
  p.cg = nullptr;  // the adjoint kernels gather from the node grid
  p.jacc = d->jacc[0];
  const T dt = (T)d->dt, mime = (T)d->cfg.mime, cva = (T)d->cva, dx = (T)d->dx, dy = (T)d->dy;
  for (int sp = 0; sp < 2; ++sp) {
    const T q = sp == 0 ? T(1) : T(-1);
    const T ms = sp == 0 ? mime : T(1);
    p.c0[sp] = q * dt * mime / ms / T(2);
    p.c1[sp] = p.c0[sp] / cva;
    p.ms[sp] = ms;
    p.q[sp] = q;
    p.qx[sp] = q * dx / dt;
    p.qy[sp] = q * dy / dt;
  }
  p.dtcva = dt * cva;
  p.idx = T(1) / dx;
  p.idy = T(1) / dy;
  p.cva = cva;
  return p;
}

template <class T>
FieldParams<T> field_params(const pbpic_diff* d, const View<T>& v) {
  FieldParams<T> a{};
  a.mx = d->mx;
  a.my = d->my;
  a.S = d->S;
  a.ybc = PBPIC_BC_CONDUCTING;
  a.ex = v.f[0];
  a.ey = v.f[1];
  a.ez = v.f[2];
  a.bx = v.f[3];
  a.by = v.f[4];
  a.bz = v.f[5];
  const T dt = (T)d->dt, cva = (T)d->cva;
  a.dth = dt / T(2);
  a.cdt = dt * (cva * cva);
  a.idx = T(1) / (T)d->dx;
  a.idy = T(1) / (T)d->dy;
  a.jacc = d->jacc[0];
  for (int k = 0; k < 4; ++k) a.jscale[k] = d->f32 ? d->in0 * FIX_INV : d->in0;
  a.ng = (T*)d->ng;
  a.cg = nullptr;
  a.fe_part = d->fe_part;
  return a;
}

double loss_scale(const pbpic_diff* d) { return d->dt * 0.5 * d->cfg.mime / (d->cva * d->cva * d->in0); }

// j.E loss: dt * mime / (cva^2 in0) * sum J . E, the work done on the particles
// in the units of the field energy (the E update drains cva^2 J per unit time
// from fields whose energy is mime / (2 cva^4 in0) sum E^2).
double jdote_scale(const pbpic_diff* d) { return d->dt * d->cfg.mime / (d->cva * d->cva * d->in0); }
double jdote_jscale(const pbpic_diff* d) { return d->f32 ? d->in0 * FIX_INV : d->in0; }

// The j.E loss of the step whose current is in `jacc` and whose starting
// fields are the state's; with jbar/fbar_e, its adjoint seeds.
template <class T>
int loss_jdote(pbpic_diff* d, const View<T>& v, const void* jacc, double* loss, double* jbar, double* fbar_e) {
  const int g = grid_of((int64_t)d->mx * (d->my + 1));
  if (d->f32)
    k_loss_jdote<T, long long><<<g, 256>>>(d->mx, d->my, d->S, PBPIC_BC_CONDUCTING, jacc, jdote_jscale(d), v.f[0],
                                           v.f[1], v.f[2], jdote_scale(d), loss, jbar, fbar_e);
  else
    k_loss_jdote<T, double><<<g, 256>>>(d->mx, d->my, d->S, PBPIC_BC_CONDUCTING, jacc, jdote_jscale(d), v.f[0],
                                        v.f[1], v.f[2], jdote_scale(d), loss, jbar, fbar_e);
  DLAUNCH("k_loss_jdote");
  return PBPIC_OK;
}

// Node grid of the state before step it into d->ng.
template <class T>
int nodes(pbpic_diff* d, int it) {
  if (d->ng_at == it) return PBPIC_OK;
  FieldParams<T> a = field_params<T>(d, state<T>(d, it));
  k_nodes<T><<<d->nfe, 256>>>(a);
  DLAUNCH("k_nodes");
  d->ng_at = it;
  return PBPIC_OK;
}

// Permutation into cell order of a state whose elements' ranks and cell counts are in
// d->rank and d->counts; leaves the counts clear.
int cell_offsets(pbpic_diff* d) {
  const int64_t nc = (int64_t)d->mx * d->my;
  const unsigned nb = (unsigned)((nc + CS_TILE - 1) / CS_TILE);
  k_diff_scan<<<nb, CS_BT>>>(d->counts, nc, d->off, d->sums);
  DLAUNCH("k_diff_scan");
  k_diff_offsets<<<nb, CS_BT>>>(d->off, d->sums, nc);
  DLAUNCH("k_diff_offsets");
  return PBPIC_OK;
}

// Opens checkpoint `it`: its permutation and its node grid.
template <class T>
int open_checkpoint(pbpic_diff* d, int it) {
  const View<T> v = state<T>(d, it);
  k_diff_rank<<<(unsigned)((d->n + 255) / 256), 256>>>(v.p.cell, d->n, d->my, d->counts, d->rank);
  DLAUNCH("k_diff_rank");
  DTRY(cell_offsets(d));
  k_diff_perm<<<grid_of(d->n, 148 * 16), 256>>>(v.p.cell, v.p.id, d->nsheet, d->rank, d->off, d->n, d->my, v.p.perm);
  DLAUNCH("k_diff_perm");
  return nodes<T>(d, it);
}

// Step it, from the state before it (its node grid in d->ng) to o, whose node grid is then in d->ng; adds the
// step's loss to scal[0]. With the j.E loss and `jkeep`, also keeps the step's current (3 planes)
// there. An o without particles or without fields: those are not wanted.
template <class T>
int step(pbpic_diff* d, int it, const View<T>& o, double omega, void* jkeep = nullptr) {
  const View<T> s = state<T>(d, it);
  DiffParams<T> dp;
  memset(&dp, 0, sizeof(dp));
  dp.push = push_params<T>(d);
  dp.n = d->n;
  dp.omega_bg = omega;
  dp.in0 = d->in0;
  dp.in = s.p;
  dp.out = o.p;
  dp.rank = d->rank;
  dp.counts = d->counts;
  k_dpush<T><<<(unsigned)((d->n + DT - 1) / DT), DT>>>(dp);
  DLAUNCH("k_dpush");
  if (o.p.cell) {
    DTRY(cell_offsets(d));
    k_diff_perm<<<grid_of(d->n, 148 * 16), 256>>>(o.p.cell, o.p.id, d->nsheet, d->rank, d->off, d->n, d->my, o.p.perm);
    DLAUNCH("k_diff_perm");
  }
  const bool jdote = d->cfg.loss == PBPIC_LOSS_JDOTE;
  if (jdote) {
    DTRY(loss_jdote<T>(d, s, d->jacc[0], d->scal, nullptr, nullptr));
    if (jkeep) DCK(cudaMemcpyAsync(jkeep, d->jacc[0], (size_t)3 * plane(d) * 8, cudaMemcpyDeviceToDevice));
  }
  if (!o.f[0]) {  // (the field solve would have left a clear current)
    DCK(cudaMemsetAsync(d->jacc[0], 0, (size_t)4 * plane(d) * 8));
    return PBPIC_OK;
  }
  FieldParams<T> a = field_params<T>(d, s);
  a.nex = o.f[0];
  a.ney = o.f[1];
  a.nez = o.f[2];
  a.nbx = o.f[3];
  a.nby = o.f[4];
  a.nbz = o.f[5];
  a.jnext = d->jacc[1];
  if (d->f32) k_field_step<T, long long><<<field_tiles(d->mx, d->my), FT>>>(a);
  else k_field_step<T, double><<<field_tiles(d->mx, d->my), FT>>>(a);
  DLAUNCH("k_field_step");
  std::swap(d->jacc[0], d->jacc[1]);
  d->ng_at = it + 1;
  if (!jdote) {
    k_loss_b<T><<<grid_of((int64_t)(d->mx + 1) * (d->my + 1)), 256>>>(d->mx, d->my, 1, (const T*)d->ng,
                                                                       loss_scale(d), d->scal, nullptr);
    DLAUNCH("k_loss_b");
  }
  return PBPIC_OK;
}

pic::FieldInit field_init(const pbpic_diff* d, double psi0) {
  pic::FieldInit f;
  f.kind = pic::LOAD_HARRIS;
  f.mx = d->mx;
  f.my = d->my;
  f.dx = d->dx;
  f.dy = d->dy;
  f.lambda = d->cfg.lambda;
  f.psi0 = psi0;
  f.bguide = 0.0;
  f.b0z = 0.0;
  return f;
}

template <class T>
int load(pbpic_diff* d, const pbpic_diff_params* prm) {
  const pbpic_diff_config& c = d->cfg;
  Harris hs = harris_speeds(d, prm->ti_te);
  pic::LoadParams L;
  memset(&L, 0, sizeof(L));
  L.kind = pic::LOAD_HARRIS;
  L.mx = d->mx;
  L.my = d->my;
  L.dx = d->dx;
  L.dy = d->dy;
  L.ppc = c.ppc;
  L.npairs = d->npairs;
  L.nsheet = d->nsheet;
  L.uthe = urel(hs.vthe);
  L.uthi = urel(hs.vthi);
  L.uthe_perp = L.uthe;
  L.udrift_e = urel(hs.ude);
  L.udrift_i = urel(hs.udi);
  L.lambda = c.lambda;
  L.seed = c.seed;
  // loaded in load order (where the adjoint and a state's ids go later), then moved into cell order
  const Comps<T> c0 = comps<T>(d, d->lam[0]);
  uint32_t* cell0 = (uint32_t*)d->ids[0];
  const View<T> v = state<T>(d, 0);
  k_load<T><<<(unsigned)((d->npairs + 255) / 256), 256>>>(L, d->npairs, 0, cell0, c0, nullptr);
  DLAUNCH("k_load");
  DCK(cudaMemsetAsync(d->counts, 0, (size_t)d->mx * d->my * 4));
  DCK(cudaMemsetAsync(d->jacc[0], 0, (size_t)4 * plane(d) * 8));
  k_diff_rank<<<(unsigned)((d->n + 255) / 256), 256>>>(cell0, d->n, d->my, d->counts, d->rank);
  DLAUNCH("k_diff_rank");
  DTRY(cell_offsets(d));
  k_diff_move<T><<<grid_of(d->n, 148 * 16), 256>>>(cell0, c0, d->nsheet, d->rank, d->off, d->n, d->my, v.p);
  DLAUNCH("k_diff_move");
  k_diff_fields<T><<<grid_of(plane(d)), 256>>>(field_init(d, prm->psi0), d->S, v.f[0]);
  DLAUNCH("k_diff_fields");
  d->ng_at = -1;
  return nodes<T>(d, 0);
}

template <class T>
int forward(pbpic_diff* d, const pbpic_diff_params* prm, double* loss) {
  d->have_forward = d->last_seg = false;
  DTRY(load<T>(d, prm));
  DCK(cudaMemset(d->scal, 0, 4 * sizeof(double)));
  const int K = d->cfg.checkpoint_every, N = d->cfg.nsteps;
  const int last0 = (d->nseg - 1) * K;  // first step of the last segment, whose states stay for the adjoint
  const double omega = prm->nb / d->cfg.nb0;
  const size_t jbytes = (size_t)3 * plane(d) * 8;
  for (int it = 0; it < N; ++it) {
    const bool keep = it >= last0 && d->jseg;
    // (the j.E loss of the last step ends with its current)
    const View<T> o = it + 1 == N && d->jseg ? View<T>{} : state<T>(d, it + 1);
    DTRY(step<T>(d, it, o, omega, keep ? (char*)d->jseg + (it - last0) * jbytes : nullptr));
  }
  DCK(cudaMemcpy(loss, d->scal, sizeof(double), cudaMemcpyDeviceToHost));
  d->last = *prm;
  d->have_forward = d->last_seg = true;
  return PBPIC_OK;
}

AdjField adj_field(pbpic_diff* d) {
  AdjField a;
  a.mx = d->mx;
  a.my = d->my;
  a.S = d->S;
  a.ybc = PBPIC_BC_CONDUCTING;
  a.dth = (double)(d->f32 ? (double)((float)d->dt / 2.0f) : d->dt / 2.0);
  const double cva = d->f32 ? (double)(float)d->cva : d->cva;
  const double dt = d->f32 ? (double)(float)d->dt : d->dt;
  a.cdt = dt * cva * cva;
  a.idx = 1.0 / d->dx;
  a.idy = 1.0 / d->dy;
  const int64_t pl = plane(d);
  a.ex = d->fbar;
  a.ey = d->fbar + pl;
  a.ez = d->fbar + 2 * pl;
  a.bx = d->fbar + 3 * pl;
  a.by = d->fbar + 4 * pl;
  a.bz = d->fbar + 5 * pl;
  a.jbar = d->jbar;
  return a;
}

template <class T>
int backward(pbpic_diff* d, double grad[3]) {
  if (!d->have_forward) return pbpic_internal_fail(PBPIC_ESTATE, "pbpic_diff_backward needs a forward call first");
  const int K = d->cfg.checkpoint_every, N = d->cfg.nsteps;
  const double omega = d->last.nb / d->cfg.nb0;
  const int64_t pl = plane(d);
  const size_t nodes_bytes = (size_t)(d->mx + 1) * (d->my + 1) * 8 * sizeof(double);
  const bool jdote = d->cfg.loss == PBPIC_LOSS_JDOTE;
  const size_t jbytes = (size_t)3 * pl * 8;
  DCK(cudaMemset(d->fbar, 0, (size_t)6 * pl * sizeof(double)));
  DCK(cudaMemset(d->gbar, 0, nodes_bytes));
  DCK(cudaMemset(d->scal + 1, 0, 3 * sizeof(double)));
  Comps<T> lam{nullptr, nullptr};  // adjoint of the state after the step (none: zero), in its order
  int buf = 0;
  AdjField af = adj_field(d);
  const int gf = grid_of((int64_t)d->mx * (d->my + 1));
  const int gn = grid_of((int64_t)(d->mx + 1) * (d->my + 1));
  // magnetic loss of the state whose node grid is in d->ng: the seed of its node adjoint
  auto seed = [&]() -> int {
    k_loss_b<T><<<gn, 256>>>(d->mx, d->my, 1, (const T*)d->ng, loss_scale(d), nullptr, d->gbar);
    DLAUNCH("k_loss_b");
    return PBPIC_OK;
  };
  const bool resident = d->last_seg;
  d->last_seg = false;  // (the segments before it are recomputed into its place)
  for (int sg = d->nseg - 1; sg >= 0; --sg) {
    const int s0 = sg * K, s1 = std::min(N, s0 + K);
    const bool tail = sg == d->nseg - 1;
    if (!(resident && tail)) {  // recompute the segment, keeping every state
      DTRY(open_checkpoint<T>(d, s0));
      for (int it = s0; it < s1; ++it) {
        // the state after the segment is not needed, its adjoint comes by particle: of the last step
        // the j.E loss wants the current, the magnetic one the fields at the end of the run
        const bool end = it + 1 == s1;
        if (end && !tail && !jdote) break;
        const View<T> o = end && jdote ? View<T>{} : state<T>(d, it + 1);
        DTRY(step<T>(d, it, o, omega, jdote ? (char*)d->jseg + (it - s0) * jbytes : nullptr));
      }
    }
    if (tail && !jdote) {  // the last state's loss
      DTRY(seed());
      k_adj_nodes<<<gn, 256>>>(af, d->gbar);
      DLAUNCH("k_adj_nodes");
    }
    for (int it = s1 - 1; it >= s0; --it) {
      const View<T> v = state<T>(d, it);
      // transposed field solve: B half step, E full step, B half step in reverse
      k_adj_bhalf<<<gf, 256>>>(af);
      DLAUNCH("k_adj_bhalf");
      k_adj_efull<<<gf, 256>>>(af);
      DLAUNCH("k_adj_efull");
      // j.E loss of step it: E (the step's start) into the current adjoint, the
      // step's current into the adjoint of that E
      if (jdote)
        DTRY(loss_jdote<T>(d, v, (char*)d->jseg + (it - s0) * jbytes, nullptr, d->jbar, d->fbar));
      k_adj_bhalf<<<gf, 256>>>(af);
      DLAUNCH("k_adj_bhalf");
      // particle adjoint of the push of step it
      DTRY(nodes<T>(d, it));
      DiffParams<T> dp;
      memset(&dp, 0, sizeof(dp));
      dp.push = push_params<T>(d);
      dp.n = d->n;
      dp.omega_bg = omega;
      dp.in0 = d->in0;
      dp.in = v.p;
      if (it == s1 - 1 && !tail) {  // lam comes in the order of the next checkpoint
        k_diff_inverse<<<grid_of(d->n, 148 * 16), 256>>>(state<T>(d, s1).p.id, d->n, d->rank);
        DLAUNCH("k_diff_inverse");
        dp.remap = d->rank;
      }
      dp.lam_in = lam;
      if (it > s0) {  // the state's adjoint in its particles' place: nothing reads them after this
        dp.lam_out = v.p.c;
      } else {  // a checkpoint stays as it is
        dp.lam_out = comps<T>(d, d->lam[buf]);
        if (K == 1) buf = 1 - buf;  // (the next step reads from the buffer that this one wrote)
      }
      lam = dp.lam_out;
      dp.jbar = d->jbar;
      dp.gbar = d->gbar;
      dp.domega = d->scal + 1;
      k_dadjoint<T><<<(unsigned)((d->n + DT - 1) / DT), DT>>>(dp);
      DLAUNCH("k_dadjoint");
      // the state's own magnetic loss (none at the start), in the same transposed node average
      if (!jdote && it > 0) DTRY(seed());
      k_adj_nodes<<<gn, 256>>>(af, d->gbar);
      DLAUNCH("k_adj_nodes");
    }
  }
  // d loss / d tau through the loaded momenta (checkpoint 0 holds the initial state)
  {
    const double tite = d->last.ti_te;
    Harris hs = harris_speeds(d, tite);
    const double dvthe = -hs.vthe / (2.0 * (1.0 + tite));
    const double dvthi = dvthe * sqrt(tite / d->cfg.mime) + hs.vthe * 0.5 / sqrt(tite * d->cfg.mime);
    const double du = -1.0 / (d->cfg.lambda * d->cva);
    const double dudi_v = du / ((1.0 + tite) * (1.0 + tite)), dude_v = du / ((1.0 + tite) * (1.0 + tite));
    const View<T> v0 = state<T>(d, 0);
    k_dtau<T><<<grid_of(d->n, 148 * 16), 256>>>(
        d->n, d->nsheet, v0.p.id, v0.p.c, lam, urel(hs.vthi), urel(hs.vthe), durel(hs.vthi) * dvthi, durel(hs.vthe) * dvthe,
        urel(hs.udi), urel(hs.ude), durel(hs.udi) * dudi_v, durel(hs.ude) * dude_v, d->scal + 2);
    DLAUNCH("k_dtau");
  }
  k_diff_psi<<<grid_of(pl), 256>>>(field_init(d, 0.0), d->S, d->fbar + 3 * pl, d->fbar + 4 * pl, d->scal + 3);
  DLAUNCH("k_diff_psi");
  double sc[3];  // d loss / d omega, d tau, d psi0
  DCK(cudaMemcpy(sc, d->scal + 1, 3 * sizeof(double), cudaMemcpyDeviceToHost));
  grad[0] = sc[2];
  grad[1] = sc[0] / d->cfg.nb0;
  grad[2] = sc[1];
  return PBPIC_OK;
}

}  // namespace

extern "C" {

int pbpic_diff_create(const pbpic_diff_config* cfg, pbpic_diff** out) {
  if (!cfg || !out) return pbpic_internal_fail(PBPIC_EINVAL, "null argument");
  *out = nullptr;
  const pbpic_diff_config& c = *cfg;
  if (c.mx < 3 || c.my < 3 || c.mx > 32767 || c.my > 65535 || c.ppc <= 0)
    return pbpic_internal_fail(PBPIC_EINVAL, "bad grid or ppc");
  if (c.precision != PBPIC_FP64_PLAIN && c.precision != PBPIC_FP32_MIXED)
    return pbpic_internal_fail(PBPIC_EINVAL, "unknown precision");
  if (c.nsteps <= 0 || c.checkpoint_every <= 0) return pbpic_internal_fail(PBPIC_EINVAL, "nsteps and checkpoint_every must be positive");
  if (c.loss != PBPIC_LOSS_MAGNETIC && c.loss != PBPIC_LOSS_JDOTE) return pbpic_internal_fail(PBPIC_EINVAL, "unknown loss");
  if (!(c.dx > 0 && c.mime > 0 && c.wpe_wce > 0 && c.lambda > 0 && c.nb0 > 0 && c.cfl > 0 && c.cfl < 1))
    return pbpic_internal_fail(PBPIC_EINVAL, "dx, mime, wpe_wce, lambda, nb0 must be positive and 0 < cfl < 1");
  if ((int64_t)2 * c.ppc * c.mx * c.my > 0x7fffff00ll) return pbpic_internal_fail(PBPIC_EINVAL, "too many particles");
  pbpic_diff* d = new pbpic_diff();
  d->cfg = c;
  d->f32 = c.precision == PBPIC_FP32_MIXED;
  d->tsz = d->f32 ? 4 : 8;
  d->mx = c.mx;
  d->my = c.my;
  d->S = c.my + 1;
  d->dx = d->dy = c.dx;
  d->cva = c.wpe_wce * sqrt(c.mime);
  d->dt = c.cfl / (d->cva * sqrt(2.0) / c.dx);
  d->npairs = (int64_t)c.ppc * c.mx * c.my;
  d->n = 2 * d->npairs;
  const double ly = c.my * c.dx, lx = c.mx * c.dx;
  d->nsheet = (int64_t)llround((double)d->npairs * (2.0 * c.lambda / (2.0 * c.lambda + c.nb0 * ly)));
  d->in0 = lx * (2.0 * c.lambda + c.nb0 * ly) / (c.dx * c.dx) / (double)d->npairs;
  d->nseg = (c.nsteps + c.checkpoint_every - 1) / c.checkpoint_every;
  int r = PBPIC_OK;
  auto A = [&](void** p, size_t b) {
    if (r == PBPIC_OK) r = dmalloc(d, p, b);
  };
  d->ck.resize(d->nseg);
  const int K = std::min(c.checkpoint_every, c.nsteps);
  d->seg.resize(K);  // (a segment's first state is its checkpoint)
  auto slot = [&](Slot& s) {
    A(&s.p, part_bytes(d));
    A(&s.f, field_bytes(d));
  };
  for (auto& s : d->ck) slot(s);
  for (int k = 1; k < K; ++k) slot(d->seg[k]);
  if (c.loss == PBPIC_LOSS_MAGNETIC) A(&d->fin.f, field_bytes(d));
  A((void**)&d->ckperm, (size_t)d->n * 4);
  for (int b = 0; b < 2; ++b) A((void**)&d->ids[b], (size_t)d->n * 4);
  A(&d->ng, node_bytes(d));
  for (int k = 0; k < 2; ++k) A(&d->jacc[k], (size_t)4 * plane(d) * 8);
  const int64_t nc = (int64_t)c.mx * c.my;
  A((void**)&d->rank, (size_t)d->n * 4);
  A((void**)&d->counts, (size_t)nc * 4);
  A((void**)&d->off, (size_t)nc * 4);
  A((void**)&d->sums, (size_t)((nc + CS_TILE - 1) / CS_TILE + 1) * 4);
  d->nfe = grid_of((int64_t)(c.mx + 1) * (c.my + 1));
  A((void**)&d->fe_part, (size_t)std::max(d->nfe, field_tiles(c.mx, c.my)) * 2 * sizeof(double));
  for (int b = 0; b < (c.checkpoint_every == 1 ? 2 : 1); ++b) A(&d->lam[b], (size_t)5 * d->n * d->tsz);
  A((void**)&d->fbar, (size_t)6 * plane(d) * sizeof(double));
  A((void**)&d->jbar, (size_t)3 * plane(d) * sizeof(double));
  A((void**)&d->gbar, (size_t)(c.mx + 1) * (c.my + 1) * 8 * sizeof(double));
  A((void**)&d->scal, 4 * sizeof(double));
  if (c.loss == PBPIC_LOSS_JDOTE) A(&d->jseg, (size_t)K * 3 * plane(d) * 8);
  if (r != PBPIC_OK) {
    pbpic_diff_destroy(d);
    return r;
  }
  *out = d;
  return PBPIC_OK;
}

int pbpic_diff_destroy(pbpic_diff* d) {
  if (!d) return PBPIC_OK;
  cudaDeviceSynchronize();
  for (void* p : d->allocs) cudaFree(p);
  delete d;
  return PBPIC_OK;
}

int pbpic_diff_forward(pbpic_diff* d, const pbpic_diff_params* params, double* loss) {
  if (!d || !params || !loss) return pbpic_internal_fail(PBPIC_EINVAL, "null argument");
  if (!(params->nb > 0 && params->ti_te > 0)) return pbpic_internal_fail(PBPIC_EINVAL, "nb and ti_te must be positive");
  return d->f32 ? forward<float>(d, params, loss) : forward<double>(d, params, loss);
}

int pbpic_diff_backward(pbpic_diff* d, double grad[3]) {
  if (!d || !grad) return pbpic_internal_fail(PBPIC_EINVAL, "null argument");
  int r = d->f32 ? backward<float>(d, grad) : backward<double>(d, grad);
  if (r == PBPIC_OK && cudaDeviceSynchronize() != cudaSuccess)
    return pbpic_internal_fail(PBPIC_ECUDA, "device error in the adjoint");
  return r;
}

}  // extern "C"
