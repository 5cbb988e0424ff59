// Step kernels of the B200 RMHD advance, templated on the bulk type T.
//
// Data layout in HBM (structure of arrays, one contiguous array per component):
//   zone index z = (i*G1 + j)*G2 + k over the guarded grid (x slowest, as in the reference's
//   AoS layout, Mara/hydro.cpp:80-110), component c at base + c*cs.
//   "state" arrays (committed prims, conserved RK registers): components 0..4 in T,
//                 components 5..7 (the magnetic field) in double, always;
//   "face" arrays (stage prims PA, fluxes F/G/H): all 8 components in T.
// Guard zones of a state are never read: the c2p kernel writes each interior zone's
// primitives to the zone and to every periodic image of it in the guard layers, which gives
// exactly the arrays SimpleCartesianDomain::Synchronize (Mara/simple-cart.cpp:81-174) would.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "rmhd_face32.cuh"

// Minimum resident blocks of 128 threads per SM requested for the flux sweep (caps its
// registers at 65536 / (128 * MGPU_FLUX_MINB)).
#ifndef MGPU_FLUX_MINB
#define MGPU_FLUX_MINB 2
#endif
// The same for the HLLD sweeps.
#ifndef MGPU_HLLD_MINB
#define MGPU_HLLD_MINB MGPU_FLUX_MINB
#endif
// The same for the zone c2p kernel (5 blocks: chosen by a sweep of 3-5; its natural register
// count allows 3).
#ifndef MGPU_C2P_MINB
#define MGPU_C2P_MINB 5
#endif

namespace mgpu {

__device__ __forceinline__ bool stage_failed(const Ctl *ctl, int upto)
{
  int e = 0;
  for (int s = 0; s < upto && s < MAX_STAGES; ++s) e |= ctl->stage_err[s];
  return e != 0;
}

// Positions of zone m_d and its periodic guard images along one dimension.
__device__ __forceinline__ int images_1d(int m, int n, int ng, bool active, int *pos)
{
  pos[0] = m;
  if (!active) return 1;
  int c = 1;
  if (m - n >= 0 && m - n < ng) pos[c++] = m - n;
  if (m + n >= n + ng && m + n < n + 2 * ng) pos[c++] = m + n;
  return c;
}

// Whether dimension d (0-based) gets its guard layers from the periodic images of this
// grid's own zones (false for unused dimensions and for dimensions whose guards a halo
// exchange fills).
__device__ __forceinline__ bool self_periodic(const Grid &g, int d) { return g.nd > d && !g.ext[d]; }

// Number of guarded arrays holding zone (i, j, k) -- this grid's, counting the zone's
// periodic images, and on a decomposed domain its neighbours' -- which is how many times
// the reference's ConsToPrim over every guarded zone of every rank counts its failure
// (Mara/hydro.cpp:133-149,201).
__device__ __forceinline__ int multiplicity(const Grid &g, int i, int j, int k)
{
  int p[3];
  const int m[3] = {i, j, k};
  int c = 1;
  for (int d = 0; d < 3; ++d) {
    if (g.ext[d]) c *= g.mult[d][m[d] - g.ng];
    else c *= images_1d(m[d], g.n[d], g.ng, g.nd > d, p);
  }
  return c;
}

template <class T>
__device__ __forceinline__ void load_state(const Grid &g, StateCPtr<T> s, long long z, double *U)
{
#pragma unroll
  for (int c = 0; c < 5; ++c) U[c] = double(s.bulk[c * g.cs + z]);
#pragma unroll
  for (int c = 0; c < 3; ++c) U[5 + c] = s.B[c * g.cs + z];
}

// The statistics slot of the calling block.
__device__ __forceinline__ StatSlot &stat_slot(Ctl *ctl) { return ctl->stat[blockIdx.x % STAT_SLOTS]; }

// Zeroes the statistics slots (all threads of the calling block take part).
__device__ __forceinline__ void stat_reset(Ctl *ctl)
{
  for (int i = threadIdx.x; i < STAT_SLOTS * (int) (sizeof(StatSlot) / 8); i += blockDim.x)
    reinterpret_cast<unsigned long long *>(ctl->stat)[i] = 0ull;
}

// Warp-aggregated counter increment: every active lane must pass the same counter.
__device__ __forceinline__ void warp_add(unsigned long long *ctr, unsigned v)
{
  const unsigned mask = __activemask();
  const unsigned sum = __reduce_add_sync(mask, v);
  if ((threadIdx.x & 31) == __ffs(mask) - 1 && sum) atomicAdd(ctr, (unsigned long long) sum);
}

// Minimum resident blocks of the sweeps of Riemann solver RS.
template <int RS> __host__ __device__ constexpr int flux_minb()
{
  return RS == RIEMANN_HLLD ? MGPU_HLLD_MINB : MGPU_FLUX_MINB;
}

// ---- begin: dt and counters ----------------------------------------------------------------
// dt_mode 0: dt given by the host; 1: dt = cfl * min_dx / MaxLambda of the previous advance
// (luaC_Mara_get_timestep, Mara/mara.cpp:374-381), computed on the device.
static __global__ void k_begin(Ctl *ctl, int dt_mode, double dt, double cfl, double min_dx)
{
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    if (dt_mode == 1) dt = cfl * min_dx / __longlong_as_double((long long) ctl->max_lambda_bits);
    ctl->dt = dt;
    ctl->max_lambda_bits = 0ull;   // RiemannSolver::ResetMaxLambda
    for (int s = 0; s < MAX_STAGES; ++s) ctl->stage_err[s] = 0;
    ctl->final_err = 0;
    for (int s = 0; s < 4; ++s) ctl->ctu_err[s] = 0;
    ctl->ctu_c2p_err = ctl->ctu_reset = 0;
    ctl->committed = 0;
  }
  if (blockIdx.x == 0) stat_reset(ctl);
}

static __global__ void k_commit(Ctl *ctl, int nstages)
{
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int e = 0, first = 0;
    for (int s = 0; s < nstages; ++s) {
      e |= ctl->stage_err[s];
      if (!first) first = ctl->stage_err[s];
    }
    e |= ctl->final_err;
    if (!first) first = ctl->final_err;
    ctl->n_advances += 1;
    if (e == 0) {
      ctl->cur ^= 1;
      ctl->committed = 1;
    } else {
      ctl->n_failed += 1;
      ctl->n_failed_zones += (unsigned) first;
    }
  }
}

// ---- P -> U on interior zones (GodunovOperator::PrimToCons, Mara/hydro.cpp:112-123) ----------
template <class T>
__device__ __forceinline__ void p2c_zone(const Grid &g, StateCPtr<T> P, StatePtr<T> U, double gamma, long long t)
{
  int i, j, k;
  interior_coords(g, t, i, j, k);
  const long long z = ((long long) i * g.G[1] + j) * g.G[2] + k;
  double p[8], u[8];
  load_state(g, P, z, p);
  prim_to_cons(gamma, p, u);
#pragma unroll
  for (int c = 0; c < 5; ++c) U.bulk[c * g.cs + z] = T(u[c]);
#pragma unroll
  for (int c = 0; c < 3; ++c) U.B[c * g.cs + z] = u[5 + c];
}

template <class T>
__global__ void __launch_bounds__(256) k_prim_to_cons(Grid g, StateCPtr<T> P0, StateCPtr<T> P1, StatePtr<T> U,
                                                      double gamma, const Ctl *ctl)
{
  const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.ninterior) return;
  p2c_zone<T>(g, ctl->cur ? P1 : P0, U, gamma, t);
}

// ---- c2p with guard scatter (GodunovOperator::ConsToPrim, Mara/hydro.cpp:125-202) -----------
// Stage c2p (final == 0): guess from PA (or zeros on the first stage, as the reference's
// PrimitiveArray is zero-filled by every advance, Mara/mara.cpp:321); result into PA.
// Closing c2p (final == 1): guess from PA, result into the next committed state.
// CTU-Hancock stage c2p (final == 2): as a stage c2p, but its failures do not abort the stage
// (PlmCtuHancockOperator::dUdt ignores the count, Mara/ctu-hancock.cpp:61-66; a failed zone
// keeps its guess) and its emergency resets are recorded, because the reset also replaces the
// operator's conserved input by P->U of the repaired primitives (Mara/hydro.cpp:186-195).
// Counts a zone's c2p outcome and scatters its primitives to the zone and its guard images.
template <class T>
__device__ __forceinline__ void c2p_finish(const Grid &g, T *PA, StatePtr<T> Pn, Ctl *ctl, int stage, int final,
                                           int ereset, double preset, double dreset, int i, int j, int k,
                                           const double *u, double *p, int err, const C2PTally &tally)
{
  const bool counted = final != C2P_LEAN_RESTORE;
  if (counted && final != C2P_DIFFUSE) {
    StatSlot &st = stat_slot(ctl);
    warp_add(&st.c2p_calls, 1u);
    warp_add(&st.c2p_iters, (unsigned) tally.iters);
    if (tally.attempts != 1) {   // [1] is the rest
#pragma unroll 1
      for (int a = 0; a < 6; ++a)   // one counter at a time: warp_add sums over the active lanes
        if (tally.attempts == a) warp_add(&st.c2p_attempt[a], 1u);
    }
    if (err) warp_add(&st.c2p_failed, 1u);
  }
  if (err) {
    if (ereset) {   // emergency reset of the failed zone
      p[0] = dreset;
      p[1] = preset;
      p[2] = p[3] = p[4] = 0.0;
      p[5] = u[5];
      p[6] = u[6];
      p[7] = u[7];
      if (final == 2) atomicAdd(&ctl->ctu_reset, 1);
    } else if (final == C2P_DIFFUSE) {
      atomicAdd(&ctl->diffuse_err, multiplicity(g, i, j, k));
    } else if (counted) {
      const bool closing = final == C2P_CLOSING || final == C2P_LEAN_CLOSING;
      atomicAdd(closing ? &ctl->final_err : final == C2P_CTU_STAGE ? &ctl->ctu_c2p_err : &ctl->stage_err[stage],
                multiplicity(g, i, j, k));
    }
  }
  // the failure mask of this c2p at the zone and its images (an emergency reset clears it)
  unsigned char *const fm = counted ? ctl->fmask : nullptr;
  const unsigned char failed = (unsigned char) (err && !ereset);
  const auto store = [&](long long w) {
    if (fm) fm[w] = failed;
    if (final == C2P_CLOSING || final == C2P_DIFFUSE) {
#pragma unroll
      for (int q = 0; q < 5; ++q) Pn.bulk[q * g.cs + w] = T(p[q]);
#pragma unroll
      for (int q = 0; q < 3; ++q) Pn.B[q * g.cs + w] = p[5 + q];
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) PA[q * g.cs + w] = T(p[q]);
      if (final == C2P_LEAN_CLOSING) {   // the field of the register about to be committed
#pragma unroll
        for (int q = 0; q < 3; ++q) Pn.B[q * g.cs + w] = u[5 + q];
      }
    }
  };
  // a zone further than ng from every face has no image
  const int m[3] = {i, j, k};
  bool inside = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) inside = inside && (d >= g.nd || (m[d] >= 2 * g.ng && m[d] < g.n[d]));
  if (inside) {
    store(((long long) i * g.G[1] + j) * g.G[2] + k);
    return;
  }
  int pi[3], pj[3], pk[3];
  const int ni = images_1d(i, g.n[0], g.ng, self_periodic(g, 0), pi);
  const int nj = images_1d(j, g.n[1], g.ng, self_periodic(g, 1), pj);
  const int nk = images_1d(k, g.n[2], g.ng, self_periodic(g, 2), pk);
#pragma unroll 1
  for (int a = 0; a < ni; ++a)
#pragma unroll 1
    for (int b = 0; b < nj; ++b)
#pragma unroll 1
      for (int c = 0; c < nk; ++c) store(((long long) pi[a] * g.G[1] + pj[b]) * g.G[2] + pk[c]);
}

// The conserved input of a c2p launch: U, or in the lean layout one of the two conserved
// registers (Pn0 = U[0], Pn1 = U[1]) by the committed role bit ctl->cur -- U[cur] for the
// restore, U[!cur] (the RK register) otherwise.
template <class T>
__device__ __forceinline__ StateCPtr<T> c2p_input(const Ctl *ctl, int final, StateCPtr<T> U, StatePtr<T> Pn0,
                                                  StatePtr<T> Pn1)
{
  if (final < C2P_LEAN_STAGE || final == C2P_DIFFUSE) return U;
  const int r = final == C2P_LEAN_RESTORE ? ctl->cur : ctl->cur ^ 1;
  const StatePtr<T> R = r ? Pn1 : Pn0;
  return StateCPtr<T>{R.bulk, R.B};
}

// Whether a c2p launch has nothing to do: an earlier stage failed, or (restore) the advance
// committed.
__device__ __forceinline__ bool c2p_skip(const Ctl *ctl, int stage, int final)
{
  return final == C2P_LEAN_RESTORE ? ctl->committed != 0 : stage_failed(ctl, stage);
}

// One interior zone's c2p.  Guess: 0 compiles in the per-thread network guess (used when
// pp.learned), 2 leaves it out -- the network's activations would otherwise set the register
// and stack budget of every c2p launch.  PAg holds the previous primitives the ladder may start
// from (PA itself, except in the pipelined host advance, whose stages alternate two arrays).
template <class T, int Guess = 2>
__device__ __forceinline__ void c2p_zone(const Grid &g, StateCPtr<T> U, T *PA, const T *PAg, StatePtr<T> Pn,
                                         const PhysParams &pp,
                                         Ctl *ctl, int stage, int zero_guess, int final, int ereset, double preset,
                                         double dreset, long long t)
{
  int i, j, k;
  interior_coords(g, t, i, j, k);
  const long long z = ((long long) i * g.G[1] + j) * g.G[2] + k;
  double u[8], p[8];
  load_state(g, U, z, u);
  // the previous primitives are read only when the ladder needs them or a failure keeps them
  const auto prev = [&](double *q) {
#pragma unroll
    for (int c = 0; c < 8; ++c) q[c] = zero_guess ? 0.0 : double(PAg[c * g.cs + z]);
  };
  C2PTally tally;
  const int err = cons_to_prim<(sizeof(T) < sizeof(double)), Guess>(pp, u, p, &tally, 0.0, 0.0, true, prev) != 0;
  c2p_finish<T>(g, PA, Pn, ctl, stage, final, ereset, preset, dreset, i, j, k, u, p, err, tally);
}

template <class T, int Guess>
__global__ void __launch_bounds__(128, MGPU_C2P_MINB) k_cons_to_prim(Grid g, StateCPtr<T> U, T *PA, const T *PAg,
                                                      StatePtr<T> Pn0, StatePtr<T> Pn1,
                                                      PhysParams pp, Ctl *ctl, int stage, int zero_guess, int final,
                                                      int ereset, double preset, double dreset)
{
  if (c2p_skip(ctl, stage, final)) return;
  const long long t = win_tbeg(g) + (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= win_tend(g)) return;
  // the uncommitted buffer, or for Mara.diffuse the committed one (rewritten in place)
  const int target = final == C2P_DIFFUSE ? ctl->cur : ctl->cur ^ 1;
  c2p_zone<T, Guess>(g, c2p_input(ctl, final, U, Pn0, Pn1), PA, PAg, target ? Pn1 : Pn0, pp, ctl, stage, zero_guess,
                     final, ereset, preset, dreset, t);
}

// The boundary shell of a decomposed block: interior zones within Ng of a face whose guards a
// halo exchange fills (region 1), and the rest (region 2, the core).  The exchange reads only
// shell zones (and their periodic images along the unsplit dimensions), so the core's c2p can
// run while the slabs travel.
__device__ __forceinline__ bool in_shell(const Grid &g, int i, int j, int k)
{
  const int m[3] = {i, j, k};
  for (int d = 0; d < 3; ++d) {
    if (!g.ext[d]) continue;
    const int r = m[d] - g.ng;
    if (r < g.ng || r >= g.n[d] - g.ng) return true;
  }
  return false;
}

// The stage c2p of one region of the interior (1 shell, 2 core); zones of the other region
// exit at once.
template <class T>
__global__ void __launch_bounds__(128, MGPU_C2P_MINB) k_cons_to_prim_region(Grid g, StateCPtr<T> U, T *PA,
                                                                            StatePtr<T> Pn0, StatePtr<T> Pn1,
                                                                            PhysParams pp, Ctl *ctl, int stage,
                                                                            int zero_guess, int final, int ereset,
                                                                            double preset, double dreset, int region)
{
  if (c2p_skip(ctl, stage, final)) return;
  const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.ninterior) return;
  int i, j, k;
  interior_coords(g, t, i, j, k);
  if (in_shell(g, i, j, k) != (region == 1)) return;
  const int target = ctl->cur ^ 1;
  c2p_zone<T, 2>(g, c2p_input(ctl, final, U, Pn0, Pn1), PA, PA, target ? Pn1 : Pn0, pp, ctl, stage, zero_guess, final,
                 ereset, preset, dreset, t);
}

// ---- flux sweep (MethodOfLinesSplit::intercell_flux_sweep, Mara/plm-split.cpp:43-73) ---------
// One thread per face.  The face set is the reference's: every zone index f with
// 2*S <= f < nz - 3*S in the flattened guarded array (S the zone stride of `dim`), the face
// between zones f and f + S.  Faces that straddle a row end in the flattened array are
// evaluated too, because they enter MaxLambda in the reference.
// Per-thread flux statistics, summed per block.
struct FluxTally {
  int hlld_ok, hlld_hllc, pcm_retry, face_c2p_calls, face_c2p_iters;
};

// The component that slot q of a face's states and flux holds: the HLLD solvers and the FP32 HLLC
// work in the normal frame of the sweep direction, HLL and the FP64 HLLC in the reference's
// component order.
template <class T, int RS> __host__ __device__ constexpr int face_slot(int dim, int q)
{
  return RS == RIEMANN_HLLD || (RS == RIEMANN_HLLC && sizeof(T) < sizeof(double)) ? frame_slot(dim, q) : q;
}

// The slot that component c goes to: face_slot's inverse.
template <class T, int RS> __host__ __device__ constexpr int slot_of(int dim, int c)
{
  if (face_slot<T, RS>(2, 2) == 2) return c;
  return c < 2 ? c : c < 5 ? 2 + (c - 2 + 4 - dim) % 3 : 5 + (c - 5 + 4 - dim) % 3;
}

// The two states of one component of the face between zones a and a + S: reconstructed by
// `recon`.
template <class T>
__device__ __forceinline__ void face_component(const T *__restrict__ a, long long S, const PhysParams &pp, int recon,
                                               T theta, T &l, T &r)
{
  if (recon == RECON_PCM) {
    l = a[0];
    r = a[S];
  } else if (recon == RECON_PLM) {
    const T vm = a[-S], v0 = a[0], vp = a[S], vpp = a[2 * S];
    l = plm(theta, vm, v0, vp, T(+1));
    r = plm(theta, v0, vp, vpp, T(-1));
  } else {
    const T vm2 = a[-2 * S], vm1 = a[-S], v0 = a[0], vp1 = a[S], vp2 = a[2 * S], vp3 = a[3 * S];
    l = weno5(pp.is_mode, T(pp.sz10A), vm2, vm1, v0, vp1, vp2, true);
    r = weno5(pp.is_mode, T(pp.sz10A), vm1, v0, vp1, vp2, vp3, false);
  }
}

// The two states of the face between zones f and f + S of direction dim: reconstructed, or with
// retry the zone states themselves.  The reconstruction is chosen once, outside the component
// loops, so that each loop's loads are issued together.
template <class T, int RS>
__device__ __forceinline__ void face_states(const Grid &g, const T *__restrict__ PA, const PhysParams &pp, int dim,
                                            long long f, bool retry, T *Pl, T *Pr)
{
  const long long S = g.s[dim - 1];
  const T theta = T(pp.theta);
#define MGPU_FACE_LOOP(R)                                                                                   \
  _Pragma("unroll") for (int q = 0; q < 8; ++q)                                                             \
      face_component<T>(PA + face_slot<T, RS>(dim, q) * g.cs + f, S, pp, R, theta, Pl[q], Pr[q])
  if (retry || pp.recon == RECON_PCM) { MGPU_FACE_LOOP(RECON_PCM); }
  else if (pp.recon == RECON_PLM) { MGPU_FACE_LOOP(RECON_PLM); }
  else { MGPU_FACE_LOOP(RECON_WENO5); }
#undef MGPU_FACE_LOOP
}

// The same into this thread's column (left 0..7, right 8..15), one component at a time: an eighth
// of the code of the unrolled form, which in FP64 is long (WENO5 divides eight times per
// component).
template <class T, int RS>
__device__ __forceinline__ void face_states_column(const Grid &g, const T *__restrict__ PA, const PhysParams &pp,
                                                   int dim, long long f, bool retry, const Column<T> &col)
{
  const long long S = g.s[dim - 1];
  const T theta = T(pp.theta);
  const int recon = retry ? (int) RECON_PCM : pp.recon;
#pragma unroll 1
  for (int q = 0; q < 8; ++q)
    face_component<T>(PA + face_slot<T, RS>(dim, q) * g.cs + f, S, pp, recon, theta, col[q], col[8 + q]);
}

// Both face values of zone z along direction dim: lo toward z - S, hi toward z + S, which are
// face_states' Pr of the face below and Pl of the face above.  which: the reconstructions that
// pp may ask for, where the launch has chosen the kernel by them.
enum { ZONE_ANY, ZONE_WENO5, ZONE_NOT_WENO5 };
template <class T, int RS, int which = ZONE_ANY>
__device__ __forceinline__ void zone_states(const Grid &g, const T *__restrict__ PA, const PhysParams &pp, int dim,
                                            long long z, T *lo, T *hi)
{
  const long long S = g.s[dim - 1];
  const T *a = PA + z;
  // components in memory order, each into its slot of the normal frame
#define MGPU_ZONE_LOOP(expr)                             \
  _Pragma("unroll") for (int c = 0; c < 8; ++c, a += g.cs) { \
    const int q = slot_of<T, RS>(dim, c);                \
    expr;                                                \
  }
  if (which != ZONE_WENO5 && pp.recon == RECON_PCM) {
    MGPU_ZONE_LOOP(lo[q] = hi[q] = a[0])
  } else if (which == ZONE_NOT_WENO5 || (which == ZONE_ANY && pp.recon == RECON_PLM)) {
    const T theta = T(pp.theta);
    MGPU_ZONE_LOOP(plm_zone(theta, a[-S], a[0], a[S], lo[q], hi[q]))
  } else {
    MGPU_ZONE_LOOP(weno5_zone(pp.is_mode, T(pp.sz10A), a[-2 * S], a[-S], a[0], a[S], a[2 * S], lo[q], hi[q]))
  }
#undef MGPU_ZONE_LOOP
}

// A face's states (reference component order) fetched again on the rare paths of the HLLD
// solvers, out of line.
template <class T> struct FaceStates {
  T l[8], r[8];
};
template <class T>
static __device__ __noinline__ FaceStates<T> refetch_face(const T *PA, long long cs, long long S, PhysParams pp,
                                                          long long f, bool retry)
{
  FaceStates<T> o;
  const int recon = retry ? (int) RECON_PCM : pp.recon;
#pragma unroll 1
  for (int q = 0; q < 8; ++q) face_component<T>(PA + q * cs + f, S, pp, recon, T(pp.theta), o.l[q], o.r[q]);
  return o;
}

// Whether a sweep of Riemann solver RS keeps its states in columns of shared memory
// (riemann_hlld64), and the entries per thread.
template <class T, int RS> __host__ __device__ constexpr bool uses_column()
{
  return RS == RIEMANN_HLLD && sizeof(T) == sizeof(double);
}
template <class T, int RS> __host__ __device__ constexpr int column_entries() { return uses_column<T, RS>() ? 32 : 1; }

// The Riemann solver at one face of direction dim.
template <class T, int RS, class Src>
__device__ __forceinline__ int riemann_face(const PhysParams &pp, int dim, const T *Pl, const T *Pr, T *Fo, T &ml,
                                            int &used_hllc, C2PTally *t, const Column<T> &col, const Src &src)
{
  const T gamma = T(pp.gamma);
  if constexpr (RS == RIEMANN_HLLD) {
    if constexpr (sizeof(T) < sizeof(double)) return riemann_hlld32(pp, dim, Pl, Pr, Fo, ml, used_hllc, t, src);
    else return riemann_hlld64(pp, dim, col, Fo, ml, used_hllc, t, src);
  } else if constexpr (RS == RIEMANN_HLLC && sizeof(T) < sizeof(double)) {
    return riemann_hllc32(gamma, Pl, Pr, Fo, ml);
  } else if constexpr (RS == RIEMANN_HLLC) {
    if (dim == 1) return riemann_hllc<T, 1>(gamma, Pl, Pr, Fo, ml);
    if (dim == 2) return riemann_hllc<T, 2>(gamma, Pl, Pr, Fo, ml);
    return riemann_hllc<T, 3>(gamma, Pl, Pr, Fo, ml);
  } else {
    if (dim == 1) return riemann_hll<T, 1>(gamma, Pl, Pr, Fo, ml);
    if (dim == 2) return riemann_hll<T, 2>(gamma, Pl, Pr, Fo, ml);
    return riemann_hll<T, 3>(gamma, Pl, Pr, Fo, ml);
  }
}

// The flux of the face between zones f and f + S of direction dim, in Fo (face_slot's order; zero
// when both attempts fail); the face's |lambda| is folded into ml.  `given`: its states are in
// Pl, Pr (the marching sweeps); otherwise they are reconstructed here.  Attempt 1 takes the
// zone states themselves (the PCM retry).  colp: this thread's column (uses_column), 128 apart.
template <class T, int RS, bool given>
__device__ __forceinline__ void solve_face(const Grid &g, const T *__restrict__ PA, const PhysParams &pp, int dim,
                                           long long f, T *Pl, T *Pr, T &ml, FluxTally &ft, T *Fo, T *colp)
{
  const long long S = g.s[dim - 1];
  int err = 1, used_hllc = 0;
  C2PTally tally{0, 0};
  const Column<T> col{colp, 128};
  if constexpr (!given && !uses_column<T, RS>()) face_states<T, RS>(g, PA, pp, dim, f, false, Pl, Pr);
  if constexpr (given && uses_column<T, RS>()) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      col[q] = Pl[q];
      col[8 + q] = Pr[q];
    }
  }
  // One call site per solver keeps a single inlined copy of it.
#pragma unroll 1
  for (int attempt = 0; attempt < 2 && err; ++attempt) {
    if (attempt == 1) ft.pcm_retry += 1;
    if constexpr (uses_column<T, RS>()) {
      if (!given || attempt == 1) face_states_column<T, RS>(g, PA, pp, dim, f, attempt == 1, col);
    } else if (attempt == 1) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        Pl[q] = PA[face_slot<T, RS>(dim, q) * g.cs + f];
        Pr[q] = PA[face_slot<T, RS>(dim, q) * g.cs + f + S];
      }
    }
    C2PTally t{0, 0};
    const auto src = [&](T *l, T *r) {
      const FaceStates<T> o = refetch_face<T>(PA, g.cs, S, pp, f, attempt == 1);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        l[q] = o.l[q];
        r[q] = o.r[q];
      }
    };
    err = riemann_face<T, RS>(pp, dim, Pl, Pr, Fo, ml, used_hllc, &t, col, src);
    tally.iters += t.iters;
    tally.attempts += t.attempts;
  }
  if (err) {
#pragma unroll
    for (int q = 0; q < 8; ++q) Fo[q] = T(0);
  }
  if constexpr (RS == RIEMANN_HLLD) {
    ft.hlld_ok += 1 - used_hllc;
    ft.hlld_hllc += used_hllc;
  }
  ft.face_c2p_calls += tally.attempts > 0;
  ft.face_c2p_iters += tally.iters;
}

// One face, its flux stored in F.
template <class T, int RS>
__device__ __forceinline__ void flux_face(const Grid &g, const T *__restrict__ PA, T *__restrict__ F,
                                          const PhysParams &pp, int dim, long long f, T &ml, FluxTally &ft, T *colp)
{
  T Pl[8], Pr[8], Fo[8];
  solve_face<T, RS, false>(g, PA, pp, dim, f, Pl, Pr, ml, ft, Fo, colp);
#pragma unroll
  for (int q = 0; q < 8; ++q) F[face_slot<T, RS>(dim, q) * g.cs + f] = Fo[q];
}

// MaxLambda of a block: warp max -> block max -> one atomicMax (non-negative doubles order
// like their bit patterns); plus the block's flux statistics.  All threads must call.
__device__ __forceinline__ void flux_block_finish(double m, const FluxTally &ft, Ctl *ctl, bool hlld)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double wmax[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();   // wmax may still be read from a previous tile
  if (lane == 0) wmax[warp] = m;
  __syncthreads();
  if (warp == 0) {
    m = lane < (blockDim.x >> 5) ? wmax[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && m > 0.0) atomicMax(&ctl->max_lambda_bits, (unsigned long long) __double_as_longlong(m));
  }
  StatSlot &st = stat_slot(ctl);
  if (hlld) {
    warp_add(&st.hlld_ok, (unsigned) ft.hlld_ok);
    warp_add(&st.hlld_hllc, (unsigned) ft.hlld_hllc);
  }
  warp_add(&st.pcm_retry, (unsigned) ft.pcm_retry);
  warp_add(&st.face_c2p_calls, (unsigned) ft.face_c2p_calls);
  warp_add(&st.face_c2p_iters, (unsigned) ft.face_c2p_iters);
}

// The faces of every direction in one launch: blocks [0, n1) sweep x, [n1, n2) y, the rest z.  The
// sweeps are independent, a face's latency is some ten microseconds in FP32 and over fifty in
// FP64, and a small box fills less than one wave of blocks per direction, so one launch takes
// little more than one sweep where three took three: 16^3 FP64 flux 0.62 -> 0.24 ms per RK2
// step.  Large boxes gain the tails of two launches.
template <class T, int RS>
__global__ void __launch_bounds__(128, flux_minb<RS>()) k_flux(Grid g, const T *__restrict__ PA, T *__restrict__ F0,
                                                              T *__restrict__ F1, T *__restrict__ F2, unsigned n1,
                                                              unsigned n2, PhysParams pp, Ctl *ctl, int stage)
{
  if (stage_failed(ctl, stage + 1)) return;
  const int dim = blockIdx.x < n1 ? 1 : blockIdx.x < n2 ? 2 : 3;
  const unsigned b = blockIdx.x - (dim == 1 ? 0u : dim == 2 ? n1 : n2);
  T *F = dim == 1 ? F0 : dim == 2 ? F1 : F2;
  const long long S = g.s[dim - 1];
  const long long f = 2 * S + (long long) b * blockDim.x + threadIdx.x;
  T ml = T(0);
  FluxTally ft{0, 0, 0, 0, 0};
  __shared__ T cols[column_entries<T, RS>() * 128];
  if (f < g.nz - 3 * S) flux_face<T, RS>(g, PA, F, pp, dim, f, ml, ft, cols + threadIdx.x);
  flux_block_finish(double(ml), ft, ctl, RS == RIEMANN_HLLD);
}

// ---- CT + flux divergence + Runge-Kutta combine ---------------------------------------------
// Flux-CT (AdiabaticIdealRmhd::ConstrainedTransport3d/2d, Mara/rmhd.cpp:311-381), the
// divergence L = -(dF/dx + dG/dy + dH/dz) (Mara/plm-split.cpp:75-122) and the stage combine
// of Mara/runge-kutta.hpp:129-177, fused, on interior zones only.
struct UpdateArgs {
  int combine;
  double c;        // COMB_RK4_K coefficient
};

template <class T>
__device__ __forceinline__ double fval(const T *F, const Grid &g, int q, long long z)
{
  return double(F[q * g.cs + z]);
}

// Zone index of interior flat index t.
__device__ __forceinline__ long long interior_zone(const Grid &g, long long t)
{
  int i, j, k;
  interior_coords(g, t, i, j, k);
  return ((long long) i * g.G[1] + j) * g.G[2] + k;
}

// 8-point corner-EMF average for the B-flux component (normal dir a, field component b):
// (2 F0 + F[+b] + F[-b] - G0 - G[+a] - G[-b] - G[+a-b]) / 8 with F the a-flux of B_b and G
// the b-flux of B_a, strides sa (normal dir) and sb (field dir).
template <class T>
__device__ __forceinline__ double ct_emf(const T *Fa, const T *Fb, const Grid &g, int qb, int qa, long long z,
                                         long long sa, long long sb)
{
  const T *F = Fa + qb * g.cs + z;
  const T *G = Fb + qa * g.cs + z;
  return (2 * double(F[0]) + double(F[sb]) + double(F[-sb]) - double(G[0]) - double(G[sa]) - double(G[-sb]) -
          double(G[sa - sb])) * 0.125;
}

template <class T>
__device__ __forceinline__ T combine_bulk(const UpdateArgs &a, T un, T us, T dt, T L, T *K, T k1, T k2, T k3)
{
  switch (a.combine) {
  case COMB_EULER: return un + dt * L;
  case COMB_RK2_2: return T(0.5) * (un + us + dt * L);
  case COMB_RK3_2: return T(3. / 4) * un + T(1. / 4) * us + T(1. / 4) * dt * L;
  case COMB_RK3_3: return T(1. / 3) * un + T(2. / 3) * us + T(2. / 3) * dt * L;
  case COMB_RK4_K: { const T kk = dt * L; *K = kk; return un + T(a.c) * kk; }
  default: return un + (T(1.0) / T(6.0)) * (k1 + T(2.0) * k2 + T(2.0) * k3 + dt * L);
  }
}

// Zone z's bulk components 0..4: plain flux differences in T.  Here and in update_field everything
// is read before anything is written: the compiler cannot tell the stored component from the next
// one's operands, and would make the components' reads wait for one another, eight trips to
// memory in a row where one is enough.  Per step, the update's launches: 96^3 FP32 RK2
// 0.150 -> 0.117 ms, 160^3 FP32 RK3 0.92 -> 0.66, 96^3 FP64 RK3 0.367 -> 0.353.
template <class T, int ND>
__device__ __forceinline__ void update_bulk(const Grid &g, const UpdateArgs &a, StateCPtr<T> Un, StateCPtr<T> Us,
                                            const T *__restrict__ F, const T *__restrict__ G,
                                            const T *__restrict__ H, StatePtr<T> Uout, StatePtr<T> Kout,
                                            StateCPtr<T> K1, StateCPtr<T> K2, StateCPtr<T> K3, double dtd,
                                            long long z)
{
  const long long sx = g.s[0], sy = g.s[1], sz = g.s[2];
  const T dx = T(g.dx), dy = T(g.dy), dz = T(g.dz), dt = T(dtd);
  const bool two = a.combine == COMB_RK2_2 || a.combine == COMB_RK3_2 || a.combine == COMB_RK3_3;
  T un[5], us[5], L[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    un[q] = Un.bulk[q * g.cs + z];
    us[q] = two ? Us.bulk[q * g.cs + z] : T(0);
  }
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const T *f = F + q * g.cs + z, *h = G + q * g.cs + z, *k = H + q * g.cs + z;
    if (ND == 1) {
      L[q] = -(f[0] - f[-sx]) / dx;
    } else if (ND == 2) {
      L[q] = -(f[0] - f[-sx]) / dx - (h[0] - h[-sy]) / dy;
    } else {
      L[q] = -(f[0] - f[-sx]) / dx - (h[0] - h[-sy]) / dy - (k[0] - k[-sz]) / dz;
    }
  }
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    T k1 = T(0), k2 = T(0), k3 = T(0), kk = T(0);
    if (a.combine == COMB_RK4_4) { k1 = K1.bulk[q * g.cs + z]; k2 = K2.bulk[q * g.cs + z]; k3 = K3.bulk[q * g.cs + z]; }
    Uout.bulk[q * g.cs + z] = combine_bulk<T>(a, un[q], us[q], dt, L[q], &kk, k1, k2, k3);
    if (a.combine == COMB_RK4_K) Kout.bulk[q * g.cs + z] = kk;
  }
}

// Zone z's field components 5..7 in double, with the constrained-transport fluxes.  inv: 1/dx,
// 1/dy, 1/dz, for the FP32 bulk's form.
template <class T, int ND>
__device__ __forceinline__ void update_field(const Grid &g, const UpdateArgs &a, StateCPtr<T> Un, StateCPtr<T> Us,
                                             const T *__restrict__ F, const T *__restrict__ G,
                                             const T *__restrict__ H, StatePtr<T> Uout, StatePtr<T> Kout,
                                             StateCPtr<T> K1, StateCPtr<T> K2, StateCPtr<T> K3, double dtd,
                                             double3 inv, long long z)
{
  const long long sx = g.s[0], sy = g.s[1], sz = g.s[2];
  const double dx = g.dx, dy = g.dy, dz = g.dz;
  const bool two = a.combine == COMB_RK2_2 || a.combine == COMB_RK3_2 || a.combine == COMB_RK3_3;
  double bn[3], bs[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    bn[c] = Un.B[c * g.cs + z];
    bs[c] = two ? Us.B[c * g.cs + z] : 0.0;
  }
  double Lb[3];
  if (ND == 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) Lb[c] = -(fval(F, g, 5 + c, z) - fval(F, g, 5 + c, z - sx)) / dx;
  } else if (ND == 2) {
    // CT2d: Fx[Bx] = 0, Fx[By] = FxBy, Fy[Bx] = FyBx, Fy[By] = 0; Bz keeps its Godunov fluxes
    const double FxBy0 = ct_emf(F, G, g, By, Bx, z, sx, sy), FxBym = ct_emf(F, G, g, By, Bx, z - sx, sx, sy);
    const double FyBx0 = ct_emf(G, F, g, Bx, By, z, sy, sx), FyBxm = ct_emf(G, F, g, Bx, By, z - sy, sy, sx);
    if constexpr (sizeof(T) < sizeof(double)) {   // FP32 bulk: reciprocals, zeroed fluxes dropped
      Lb[0] = -(FyBx0 - FyBxm) * inv.y;
      Lb[1] = -(FxBy0 - FxBym) * inv.x;
      Lb[2] = -(fval(F, g, Bz, z) - fval(F, g, Bz, z - sx)) * inv.x - (fval(G, g, Bz, z) - fval(G, g, Bz, z - sy)) * inv.y;
    } else {   // the reference's expressions, bit for bit
      Lb[0] = -(0.0 - 0.0) / dx - (FyBx0 - FyBxm) / dy;
      Lb[1] = -(FxBy0 - FxBym) / dx - (0.0 - 0.0) / dy;
      Lb[2] = -(fval(F, g, Bz, z) - fval(F, g, Bz, z - sx)) / dx - (fval(G, g, Bz, z) - fval(G, g, Bz, z - sy)) / dy;
    }
  } else {
    const double FxBy0 = ct_emf(F, G, g, By, Bx, z, sx, sy), FxBym = ct_emf(F, G, g, By, Bx, z - sx, sx, sy);
    const double FyBx0 = ct_emf(G, F, g, Bx, By, z, sy, sx), FyBxm = ct_emf(G, F, g, Bx, By, z - sy, sy, sx);
    const double FyBz0 = ct_emf(G, H, g, Bz, By, z, sy, sz), FyBzm = ct_emf(G, H, g, Bz, By, z - sy, sy, sz);
    const double FzBy0 = ct_emf(H, G, g, By, Bz, z, sz, sy), FzBym = ct_emf(H, G, g, By, Bz, z - sz, sz, sy);
    const double FzBx0 = ct_emf(H, F, g, Bx, Bz, z, sz, sx), FzBxm = ct_emf(H, F, g, Bx, Bz, z - sz, sz, sx);
    const double FxBz0 = ct_emf(F, H, g, Bz, Bx, z, sx, sz), FxBzm = ct_emf(F, H, g, Bz, Bx, z - sx, sx, sz);
    if constexpr (sizeof(T) < sizeof(double)) {   // FP32 bulk: reciprocals, zeroed fluxes dropped
      Lb[0] = -(FyBx0 - FyBxm) * inv.y - (FzBx0 - FzBxm) * inv.z;
      Lb[1] = -(FxBy0 - FxBym) * inv.x - (FzBy0 - FzBym) * inv.z;
      Lb[2] = -(FxBz0 - FxBzm) * inv.x - (FyBz0 - FyBzm) * inv.y;
    } else {   // the reference's expressions, bit for bit
      Lb[0] = -(0.0 - 0.0) / dx - (FyBx0 - FyBxm) / dy - (FzBx0 - FzBxm) / dz;
      Lb[1] = -(FxBy0 - FxBym) / dx - (0.0 - 0.0) / dy - (FzBy0 - FzBym) / dz;
      Lb[2] = -(FxBz0 - FxBzm) / dx - (FyBz0 - FyBzm) / dy - (0.0 - 0.0) / dz;
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double un = bn[c], us = bs[c];
    const double L = Lb[c];
    double out;
    switch (a.combine) {
    case COMB_EULER: out = un + dtd * L; break;
    case COMB_RK2_2: out = 0.5 * (un + us + dtd * L); break;
    case COMB_RK3_2: out = 3. / 4 * un + 1. / 4 * us + 1. / 4 * dtd * L; break;
    case COMB_RK3_3: out = 1. / 3 * un + 2. / 3 * us + 2. / 3 * dtd * L; break;
    case COMB_RK4_K: { const double kk = dtd * L; Kout.B[c * g.cs + z] = kk; out = un + a.c * kk; } break;
    default:
      out = un + (1.0 / 6.0) * (K1.B[c * g.cs + z] + 2.0 * K2.B[c * g.cs + z] + 2.0 * K3.B[c * g.cs + z] + dtd * L);
      break;
    }
    Uout.B[c * g.cs + z] = out;
  }
}

template <class T, int ND>
__device__ __forceinline__ void update_zone(const Grid &g, const UpdateArgs &a, StateCPtr<T> Un, StateCPtr<T> Us,
                                            const T *__restrict__ F, const T *__restrict__ G,
                                            const T *__restrict__ H, StatePtr<T> Uout, StatePtr<T> Kout,
                                            StateCPtr<T> K1, StateCPtr<T> K2, StateCPtr<T> K3, double dtd,
                                            double3 inv, long long z)
{
  update_bulk<T, ND>(g, a, Un, Us, F, G, H, Uout, Kout, K1, K2, K3, dtd, z);
  update_field<T, ND>(g, a, Un, Us, F, G, H, Uout, Kout, K1, K2, K3, dtd, inv, z);
}

#ifndef MGPU_UPDATE_MINB
#define MGPU_UPDATE_MINB 4   // 64 registers: 96^3 FP32 RK2 with 4 blocks 0.117 ms, with 3 0.126
#endif

template <class T, int ND>
__global__ void __launch_bounds__(256, MGPU_UPDATE_MINB) k_update(Grid g, UpdateArgs a, StateCPtr<T> Un, StateCPtr<T> Us,
                                                const T *__restrict__ F, const T *__restrict__ G,
                                                const T *__restrict__ H, StatePtr<T> Uout, StatePtr<T> Kout,
                                                StateCPtr<T> K1, StateCPtr<T> K2, StateCPtr<T> K3,
                                                const Ctl *ctl, int stage, double3 inv)
{
  if (stage_failed(ctl, stage + 1)) return;
  const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.ninterior) return;
  update_zone<T, ND>(g, a, Un, Us, F, G, H, Uout, Kout, K1, K2, K3, ctl->dt, inv, interior_zone(g, t));
}

}  // namespace mgpu
