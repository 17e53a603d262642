// cav_drift.cuh -- the integrator's first stage of one slot (src/md_simulator.cpp:640-656,
// 748-837, 890-905): the drift kernels of cav_kernels.cu and the step kernel (cav_chunk.cu).
#pragma once

#include "cav_common.cuh"

namespace cav {

// Velocity-Verlet drift (src/md_simulator.cpp:640-656) with the NaN check of the
// acceleration and the half-skin test; the pair kernel fuses the same update into
// the step before when it can (FUSE_VV), so this runs at the start of a chunk.
template <bool MIXED>
__device__ __forceinline__ void drift_slot_vv(const Dev &d, const Box &b, const StepConsts &sc, int i) {
  const int rep = rep_of_slot(b, i);
  if (rep < 0) return;  // padding slot
  dbl4 x = d.pos[i];
  const dbl4 v = d.vel[i], a = d.acc[i];
  nan_check(d, i, a);
  drift_vv<MIXED>(x, v, a, sc);
  d.pos[i] = x;  // acc stays: the pair kernel's kick reads it as a_old
  if (MIXED) mixed_track(d, b, rep, i, x, d.ic);
  else half_skin_test(d, b, rep, i, x);
}

// Leap-frog first half (src/md_simulator.cpp:890-905): v += (0.5 dt) a ; r += dt v.
// The closing half, v += (0.5 dt) a(t + dt), is the velocity-Verlet kick of the pair
// kernel with a_old = 0: v + (a + 0)(0.5 dt) rounds exactly as v + (0.5 dt) a.
template <bool MIXED>
__device__ __forceinline__ void drift_slot_lf(const Dev &d, const Box &b, const StepConsts &sc, int i) {
  const int rep = rep_of_slot(b, i);
  if (rep < 0) return;  // padding slot
  dbl4 x = d.pos[i], v = d.vel[i];
  const dbl4 a = d.acc[i];
  nan_check(d, i, a);
  drift_lf<MIXED>(x, v, a, sc);
  d.pos[i] = x;
  d.vel[i] = v;
  d.acc[i] = make_dbl4(0.0, 0.0, 0.0, 0.0);  // a_old = 0 for the kick
  if (MIXED) mixed_track(d, b, rep, i, x, d.ic);
  else half_skin_test(d, b, rep, i, x);
}

// Langevin position update r += v*c (src/md_simulator.cpp:822-827) with the
// half-skin tracking; with THERMO the temperature sums of the velocities first.
template <bool MIXED, bool THERMO>
__device__ __forceinline__ void lang_position(const Dev &d, const Box &b, const StepConsts &sc, int rep, int i, dbl4 x,
                                              const dbl4 &v, double (&part)[4]) {
  if (THERMO) {
    const double m = d.tab->mass[type_of(x.w)];
    part[0] = twice_ke(m, v);
    part[1] = m * v.x; part[2] = m * v.y; part[3] = m * v.z;
  }
  lang_move<MIXED>(x, v, sc);
  d.pos[i] = x;
  if (MIXED) mixed_track(d, b, rep, i, x, d.ic);
  else half_skin_test(d, b, rep, i, x);
}

// Langevin first half (src/md_simulator.cpp:748-837):
//   v += (a*0.5)*dt + eta*b ; [temperature here] ; r += v*c
// POS false: the velocity half only; constraint::Nve then acts on the mid-step
// velocities (:784-791) and k_lang_pos takes the temperature and moves the atoms.
template <bool MIXED, bool THERMO, bool POS>
__device__ __forceinline__ void lang_slot(const Dev &d, const Box &b, const StepConsts &sc, long long step, int i,
                                          double (&part)[4]) {
  const int rep = rep_of_slot(b, i);
  if (rep < 0) return;
  dbl4 x = d.pos[i], v = d.vel[i];
  const dbl4 a = d.acc[i];
  nan_check(d, i, a);
  double e0 = 0.0, e1 = 0.0, e2 = 0.0;
  if (!sc.noise_off) {
    // replica r draws the noise stream of seed + r with its local ids
    if (MIXED) langevin_eta_f(sc.seed + rep, step, d.id[i], e0, e1, e2);
    else langevin_eta(sc.seed + rep, step, d.id[i], e0, e1, e2);
  }
  lang_half<MIXED>(v, a, e0, e1, e2, sc);
  d.vel[i] = v;
  if (POS) lang_position<MIXED, THERMO>(d, b, sc, rep, i, x, v, part);
}

}  // namespace cav
