// cav_pair.cuh -- what the pair kernels share (cav_force.cu, cav_exchange.cu): the pair
// tables in shared memory, the split of an atom's row over lanes, the closing update of a
// step and its end (status, conditional node, thermo fold).
#pragma once

#include <type_traits>

#include "cav_common.cuh"

namespace cav {

struct SmemTabD {
  double rc2[MAXT * MAXT], sig2[MAXT * MAXT], eps4[MAXT * MAXT], gc[MAXT * MAXT], uc[MAXT * MAXT];
  double e6[MAXT * MAXT], e12[MAXT * MAXT];  // 6 eps4 and 12 eps4 (exact: products by 6 and 12)
  double minv[MAXT], mass[MAXT];
};
struct SmemTabF {
  float4 c4[MAXT * MAXT];  // {rc2, sig2, eps4, gc} of a type pair: one 128-bit load per pair
  float rc2[MAXT * MAXT], sig2[MAXT * MAXT], eps4[MAXT * MAXT], gc[MAXT * MAXT];
  float pk[MAXT * MAXT];   // 0.5 gc rc2 - uc, rounded once from FP64: V = eps4 s6 (s6 - 1) - 0.5 gc r2 + pk
  double minv[MAXT], mass[MAXT];
};
// FP64 reciprocal by Newton-Raphson refinement of the hardware approximation
// (PTX rcp.approx.ftz.f64): each step y <- y + y (1 - x y) with two FMAs roughly
// doubles the correct bits (Markstein, "IA-64 and Elementary Functions", 2000), so
// two steps take the approximation to within an ulp or two of 1/x -- far inside the
// 1e-12 force tolerance -- at four FP64-pipe operations, the pipe this kernel is
// bound by.  Both orders of a pair see the same r^2, hence the same value.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// Loads the pair table into shared memory (FP32 copy for the mixed form).
template <class Tab>
__device__ inline void load_tab(const Dev &d, Tab &tab) {
  const PairTab &T = *d.tab;
  const int nt = T.nt;
  for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) {
    tab.rc2[k] = T.rc2[k]; tab.sig2[k] = T.sig2[k]; tab.eps4[k] = T.eps4[k]; tab.gc[k] = T.gc[k];
    if constexpr (std::is_same<Tab, SmemTabF>::value) {
      tab.c4[k] = make_float4(tab.rc2[k], tab.sig2[k], tab.eps4[k], tab.gc[k]);
      tab.pk[k] = (float)(0.5 * T.gc[k] * T.rc2[k] - T.uc[k]);
    } else {
      tab.uc[k] = T.uc[k];
      tab.e6[k] = 6.0 * T.eps4[k];
      tab.e12[k] = 12.0 * T.eps4[k];
    }
  }
  for (int k = threadIdx.x; k < nt; k += blockDim.x) { tab.minv[k] = T.minv[k]; tab.mass[k] = T.mass[k]; }
}

// masses alone, for the closing update (finish_atom)
struct MassTab {
  double minv[MAXT], mass[MAXT];
  __device__ __forceinline__ void load(const Dev &d) {
    if (threadIdx.x < MAXT) {
      minv[threadIdx.x] = d.tab->minv[threadIdx.x];
      mass[threadIdx.x] = d.tab->mass[threadIdx.x];
    }
  }
};

// How an atom's row is split over lanes in the FP64 form.  Entry e of the row adds to
// partial sum e mod 4, in row order; a lane holds all four sums (TPA 1), two of them (TPA
// 2) or one (TPA >= 4: t mod 4, of the chunks t / 4, t / 4 + TPA / 4, ...).  Sums 0 and 1, 2
// and 3 are added, then the two halves, then the lanes: 1, 2 and 4 lanes per atom give the
// same sums bit for bit, so that the lane count may follow the size of a whole batch and
// its replicas still equal their single-system runs.
template <int TPA>
struct RowSplit {
  static constexpr int PER = TPA == 1 ? 4 : TPA == 2 ? 2 : 1;  // entries of a chunk a lane takes
  static constexpr int STRIDE = TPA <= 4 ? 1 : TPA / 4;        // chunks a lane steps by
  static __device__ __forceinline__ int first_chunk(int t) { return TPA <= 4 ? 0 : t >> 2; }
  static __device__ __forceinline__ int first_entry(int t) { return TPA == 1 ? 0 : TPA == 2 ? 2 * t : t & 3; }
};

// Folds the TPA lanes of each atom (lanes a, a+A, a+2A, ...; every lane of the warp
// calls this).
template <int A, bool EV>
__device__ __forceinline__ void fold_lanes(double &fx, double &fy, double &fz, double &vir, double &pe) {
#pragma unroll
  for (int o = A; o < 32; o <<= 1) {
    fx += __shfl_xor_sync(FULL_MASK, fx, o);
    fy += __shfl_xor_sync(FULL_MASK, fy, o);
    fz += __shfl_xor_sync(FULL_MASK, fz, o);
    if (EV) {
      vir += __shfl_xor_sync(FULL_MASK, vir, o);
      pe += __shfl_xor_sync(FULL_MASK, pe, o);
    }
  }
}

// NaN for the acceleration of an atom that mixed_track marked, if it has neighbours (the
// integers of a position that is not a number give a finite force)
template <bool MIXED>
__device__ __forceinline__ void spread_nan(const Dev &d, int i, const dbl4 &v, dbl4 &a) {
  if (MIXED && __double2hiint(v.w) != 0 && d.nnbr[i] > 0) a.x = a.y = a.z = __longlong_as_double(0x7ff8000000000000ll);
}

// The closing update of the step of atom i, given its folded force sum.
// KICK: 0 = store the acceleration only; 1 = velocity-Verlet closing kick
// v += (a + a_old) * (0.5 dt) (src/md_simulator.cpp:672-679); 2 = Langevin closing
// update v = (v a_L + eta b) + (a*0.5) dt (src/md_simulator.cpp:853-862).
// EV: the atom's KE terms into `ke` (KICK == 2: that of the velocities at the end of the step, kept
// apart from the mid-step temperature's).
// fuse: then the first half of the next step, with the arithmetic of the drift
// kernels (k_drift_vv, k_drift_lf, k_lang_a): the NaN check of the new acceleration,
// the drift, the half-skin test; the new coordinates go to the alternate buffer
// (FP64: pos_alt, which the neighbours of this step no longer read; mixed: ic_alt,
// the FP64 positions being this atom's alone).  Leap-frog keeps a_old = 0 for the
// next kick, as its drift kernel does.
template <bool MIXED, int KICK, bool EV, class Tab>
__device__ __forceinline__ void finish_atom(const Dev &d, const Box &b, const StepConsts &sc, const Tab &tab, int i,
                                            int ti, int rep, long long step, int fuse, double fx, double fy,
                                            double fz, double (&ke)[4]) {
  const double mi = tab.minv[ti];
  dbl4 an = make_dbl4(fx * mi, fy * mi, fz * mi, 0.0);
  dbl4 v;
  if (KICK == 0) {
    d.acc[i] = an;
    if (EV) {
      v = d.vel[i];
      const double m = tab.mass[ti];
      ke[0] = twice_ke(m, v);
      ke[1] = m * v.x; ke[2] = m * v.y; ke[3] = m * v.z;
    }
  } else if (KICK == 1) {
    v = d.vel[i];
    spread_nan<MIXED>(d, i, v, an);
    const dbl4 ao = d.acc[i];  // a(t), still in place until the store below
    if (MIXED) {
      v.x = fma(an.x + ao.x, sc.hdt, v.x);
      v.y = fma(an.y + ao.y, sc.hdt, v.y);
      v.z = fma(an.z + ao.z, sc.hdt, v.z);
    } else {  // v += (a + a_old) * (0.5 dt), the reference's order
      v.x = __dadd_rn(v.x, __dmul_rn(__dadd_rn(an.x, ao.x), sc.hdt));
      v.y = __dadd_rn(v.y, __dmul_rn(__dadd_rn(an.y, ao.y), sc.hdt));
      v.z = __dadd_rn(v.z, __dmul_rn(__dadd_rn(an.z, ao.z), sc.hdt));
    }
    if (EV) {
      const double m = tab.mass[ti];
      ke[0] = twice_ke(m, v);
      ke[1] = m * v.x; ke[2] = m * v.y; ke[3] = m * v.z;
    }
  } else {
    v = d.vel[i];
    spread_nan<MIXED>(d, i, v, an);
    double e0 = 0.0, e1 = 0.0, e2 = 0.0;
    if (!sc.noise_off) {  // replica r draws the noise stream of seed + r with its local ids
      if (MIXED) langevin_eta_f(sc.seed + rep, step, d.id[i], e0, e1, e2);
      else langevin_eta(sc.seed + rep, step, d.id[i], e0, e1, e2);
    }
    if (MIXED) {
      v.x = fma(an.x, sc.hdt, fma(v.x, sc.la, e0 * sc.lb));
      v.y = fma(an.y, sc.hdt, fma(v.y, sc.la, e1 * sc.lb));
      v.z = fma(an.z, sc.hdt, fma(v.z, sc.la, e2 * sc.lb));
    } else {  // v = (v a + eta b) + (a*0.5) dt, the reference's order
      v.x = __dadd_rn(__dadd_rn(__dmul_rn(v.x, sc.la), __dmul_rn(e0, sc.lb)), __dmul_rn(an.x, sc.hdt));
      v.y = __dadd_rn(__dadd_rn(__dmul_rn(v.y, sc.la), __dmul_rn(e1, sc.lb)), __dmul_rn(an.y, sc.hdt));
      v.z = __dadd_rn(__dadd_rn(__dmul_rn(v.z, sc.la), __dmul_rn(e2, sc.lb)), __dmul_rn(an.z, sc.hdt));
    }
    if (EV) {  // Atom_data::kinetic_energy() read after the step (the temperature was taken mid-step)
      const double m = tab.mass[ti];
      ke[0] = twice_ke(m, v);
      ke[1] = m * v.x; ke[2] = m * v.y; ke[3] = m * v.z;
    }
  }
  if (KICK != 0) {
    if (fuse != FUSE_NONE) {  // the next step's first half (its drift kernel's arithmetic)
      nan_check(d, i, an);
      dbl4 x = d.pos[i];
      dbl4 ao = an;
      if (fuse == FUSE_VV) {
        drift_vv<MIXED>(x, v, an, sc);
      } else if (fuse == FUSE_LF) {
        drift_lf<MIXED>(x, v, an, sc);
        ao = make_dbl4(0.0, 0.0, 0.0, 0.0);  // a_old = 0 for the next kick
      } else {
        double e0 = 0.0, e1 = 0.0, e2 = 0.0;
        if (!sc.noise_off) {
          if (MIXED) langevin_eta_f(sc.seed + rep, step + 1, d.id[i], e0, e1, e2);
          else langevin_eta(sc.seed + rep, step + 1, d.id[i], e0, e1, e2);
        }
        lang_half<MIXED>(v, an, e0, e1, e2, sc);
        lang_move<MIXED>(x, v, sc);
      }
      d.acc[i] = ao;
      d.vel[i] = v;
      if (MIXED) {
        d.pos[i] = x;
        mixed_track(d, b, rep, i, x, d.ic_alt);
      } else {
        d.pos_alt[i] = x;
        half_skin_test(d, b, rep, i, x);
      }
    } else {
      d.acc[i] = an;
      d.vel[i] = v;
    }
  }
}

// virial and potential energy of atom i (both orders of its pairs are counted)
__device__ __forceinline__ void set_ev(const Dev &d, int i, double vir, double pe, double (&ev)[2]) {
  ev[0] = vir;
  ev[1] = pe;
  if (d.ev_atom) d.ev_atom[i] = make_double2(vir, pe);
}

// per-launch arguments of the pair kernels
struct ForceArgs {
  int k_in_chunk;                   // step index inside the chunk (Langevin noise counter)
  int fuse;                         // Fuse: the next step's drift in this launch
  int set_cond;                     // set `cond` at the end (inside a captured graph)
  cudaGraphConditionalHandle cond;  // the next step's rebuild node
  int fold;                         // the last block folds the thermo record (EV launches)
  FoldArgs fa;
};

// Sums of n blocks' partials of W doubles (W = 2 or 4) into v[0..W): thread t takes
// blocks t, t + B, t + 2B, ... in that order, four blocks' loads in flight at a time
// (L2 loads: other blocks wrote them).
template <int W>
__device__ __forceinline__ void fold_strided(const double *p, int n, double *v) {
  const int B = blockDim.x;
  for (int k0 = threadIdx.x; k0 < n; k0 += 4 * B) {
    double2 x[4][W / 2];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < W / 2; ++h)
        x[u][h] = k0 + u * B < n ? __ldcg(reinterpret_cast<const double2 *>(p + (size_t)(k0 + u * B) * W) + h)
                                 : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k0 + u * B < n)
#pragma unroll
        for (int h = 0; h < W / 2; ++h) {
          v[2 * h] += x[u][h].x;
          v[2 * h + 1] += x[u][h].y;
        }
  }
}

// The thermo fold in the last block: every thread sums a strided subset of the
// partials, the block folds the threads' sums in a fixed order, thread 0 finishes
// the record.  The sums do not depend on which block finished last.
static __device__ __noinline__ void fold_thermo(const Dev &d, const FoldArgs &fa) {
  double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  fold_strided<4>(d.partials_ke, fa.nb_ke, v);
  fold_strided<2>(d.partials_ev, fa.nb_ev, v + 4);
  fold_strided<4>(d.partials_ke_end, fa.nb_ke_end, v + 6);
  __shared__ double out[10];
  block_sum_store<10>(v, out);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const ThermoCfg &tc = fa.tc;
  double res[5];
  const double P3[3] = {out[1], out[2], out[3]};
  thermo_finish(out[0], P3, d.thermo[5], out[4], out[5], tc.n, tc.n_r_df, tc.k_b, tc.volume, tc.langevin, res);
  if (fa.nb_ke_end > 0) {  // KE as Atom_data::kinetic_energy() reads it after the step
    double e[5];
    const double Q3[3] = {out[7], out[8], out[9]};
    thermo_finish(out[6], Q3, d.thermo[5], 0.0, 0.0, tc.n, tc.n_r_df, tc.k_b, tc.volume, tc.langevin, e);
    res[0] = e[0];
  }
#pragma unroll
  for (int q = 0; q < 5; ++q) d.thermo[q] = res[q];
  if (fa.ring_slot >= 0) {
    double *r = d.thermo_ring + (size_t)fa.ring_slot * THERMO_REC;
#pragma unroll
    for (int q = 0; q < THERMO_REC; ++q) r[q] = res[q];
  }
}

// End of a pair-kernel launch, every block: the last block to finish counts the
// step, turns a NaN seen by the fused drift into a halt, -- inside a graph -- sets
// the conditional node of the next step's rebuild, and (EV, fold) folds the thermo
// record unless the chunk halted.  The flag and partial stores of this launch are
// ordered before the ticket by the fence.
template <bool EV>
__device__ __forceinline__ void end_of_step(const Dev &d, bool was_halted, const ForceArgs &fa) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(d.force_ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __shared__ int s_fold;
  if (threadIdx.x == 0) {
    __threadfence();
    volatile int *f = d.flags;
    if (!was_halted) {
      f[F_STEPS_OK] = f[F_STEPS_OK] + 1;
      if (f[F_NAN]) f[F_HALT] = 1;
    }
    if (fa.set_cond) cudaGraphSetConditional(fa.cond, (f[F_REBUILD] != 0 && f[F_HALT] == 0) ? 1u : 0u);
    *d.force_ticket = 0u;
    s_fold = EV && fa.fold && f[F_HALT] == 0;
  }
  __syncthreads();
  if constexpr (EV) {
    if (s_fold) fold_thermo(d, fa.fa);
  }
}

template <int KICK, bool EV>
__device__ inline void store_partials(const Dev &d, double (&ke_p)[4], double (&ev_p)[2]) {
  if (EV) {
    block_sum_store<2>(ev_p, &d.partials_ev[(size_t)blockIdx.x * 2]);
    __syncthreads();
    block_sum_store<4>(ke_p, &(KICK == 2 ? d.partials_ke_end : d.partials_ke)[(size_t)blockIdx.x * 4]);
  }
}

}  // namespace cav
