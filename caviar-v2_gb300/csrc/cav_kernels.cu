// cav_kernels.cu -- sm_103a kernels of the CAVIAR2 MD step (integrator stages,
// cell binning, Verlet-list build, thermo reductions, parity exports).  The
// pair-force kernels live in cav_force.cu.  Every kernel serves R >= 1 replicas
// (see cav_common.cuh); a single system is R = 1.
#include <algorithm>

#include "cav_drift.cuh"
#include "cav_rebuild.cuh"

namespace cav {

static inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

int num_sms() {
  static PerDevice sms;
  return sms.get([](int dev) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
  });
}

// ---------------------------------------------------------------------------
// integrator stage 1 -- src/md_simulator.cpp:640-656 (velocity Verlet) and
// :748-837 (Langevin first half); NaN check; half-skin test per replica
// ---------------------------------------------------------------------------
template <bool MIXED>
__global__ void __launch_bounds__(256) k_drift_vv(Dev d, Box b, StepConsts sc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < sc.n && !halted(d)) drift_slot_vv<MIXED>(d, b, sc, i);
}

template <bool MIXED>
__global__ void __launch_bounds__(256) k_drift_lf(Dev d, Box b, StepConsts sc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < sc.n && !halted(d)) drift_slot_lf<MIXED>(d, b, sc, i);
}

template <bool MIXED, bool THERMO, bool POS>
__global__ void __launch_bounds__(256) k_lang_a(Dev d, Box b, StepConsts sc, int k_in_chunk) {
  if (halted(d)) return;  // the same value for every block: no block reaches the reduction alone
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double part[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < sc.n) lang_slot<MIXED, THERMO, POS>(d, b, sc, *d.step_base + k_in_chunk, i, part);
  if (POS && THERMO) block_sum_store<4>(part, &d.partials_ke[(size_t)blockIdx.x * 4]);
}

template <bool MIXED, bool THERMO>
__global__ void __launch_bounds__(256) k_lang_pos(Dev d, Box b, StepConsts sc) {
  if (halted(d)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double part[4] = {0.0, 0.0, 0.0, 0.0};
  const int rep = i < sc.n ? rep_of_slot(b, i) : -1;
  if (rep >= 0) lang_position<MIXED, THERMO>(d, b, sc, rep, i, d.pos[i], d.vel[i], part);
  if (THERMO) block_sum_store<4>(part, &d.partials_ke[(size_t)blockIdx.x * 4]);
}

// ---------------------------------------------------------------------------
// list rebuild of the flagged replicas (cav_rebuild.cuh): wrap + bin -> per-replica scan ->
// scatter -> per-cell sort and gather -> build
// ---------------------------------------------------------------------------
constexpr int BUILD_WARPS = 8;  // warps per block

__global__ void __launch_bounds__(256) k_bin(Dev d, Box b, int forced) {
  rebuild_bin(d, b, forced, blockIdx.x * blockDim.x + threadIdx.x);
}

// Exclusive scan of each replica's cell counts, starting at the replica's first
// slot; the padding cell counts the replica's padding slots.  Block rep*P + p owns
// slice p of the replica's m counts (scan_slice(m, P, p); P > 1 only for a single
// system, whose slices start from the sums k_scan_part left in scan_part).
// Warp w owns the contiguous run [w*seg, (w+1)*seg) of its slice and walks it 32
// counts at a time with coalesced loads: a first pass sums the run, one scan of the
// 32 warp sums gives every run its start, and a second pass scans the run (warp
// shuffles, carry from lane 31) and writes the starts.  Zeroes the counts and
// cursors it read.
__device__ inline int2 scan_slice(int m, int P, int p) {
  const int len = ((m + P - 1) / P + 31) & ~31;
  const int s0 = min(m, p * len);
  return make_int2(s0, min(m, s0 + len));
}

// single system: the sum of each slice's counts (first level of the scan)
__global__ void __launch_bounds__(1024) k_scan_part(Dev d, Box b, int forced) {
  if (!rebuild_on(d, b, 0, forced)) return;
  const RepBox &rb = repbox(b, 0);
  const int m = rb.ncell + 1;
  const int2 sl = scan_slice(m, gridDim.x, blockIdx.x);
  int v = 0;
  for (int k = sl.x + (int)threadIdx.x; k < sl.y; k += blockDim.x) v += scan_count(d, rb, m, k);
  __shared__ int warp_tot[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
  if (lane == 0) warp_tot[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    if (lane == 0) d.scan_part[blockIdx.x] = v;
  }
}

__global__ void __launch_bounds__(1024) k_scan_rep(Dev d, Box b, int forced, int P) {
  const int rep = blockIdx.x / P, p = blockIdx.x - rep * P;
  if (!rebuild_on(d, b, rep, forced)) return;
  const RepBox &rb = repbox(b, rep);
  const int m = rb.ncell + 1, off = rb.cell_off;
  const int2 sl = scan_slice(m, P, p);
  __shared__ int warp_tot[32];
  __shared__ int slice_base;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (wid == 0) {  // counts before this slice: the first-level sums of slices 0 .. p-1
    int v = 0;
    for (int q = lane; q < p; q += 32) v += d.scan_part[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    if (lane == 0) slice_base = v;
  }
  const int seg = ((sl.y - sl.x + 31) / 32 + 31) & ~31;  // counts per warp, a multiple of 32
  const int k0 = min(sl.y, sl.x + wid * seg), k1 = min(sl.y, k0 + seg);
  auto count = [&](int k) { return k < k1 ? scan_count(d, rb, m, k) : 0; };
  int s = 0;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32) s += count(k);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
  if (lane == 0) warp_tot[wid] = s;
  __syncthreads();
  if (wid == 0) {
    int wv = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL_MASK, wv, o);
      if (lane >= o) wv += y;
    }
    warp_tot[lane] = wv;  // inclusive
  }
  __syncthreads();
  int carry = rb.slot_off + slice_base + (wid ? warp_tot[wid - 1] : 0);
  for (int base = k0; base < k1; base += 32) {
    const int k = base + lane;
    const int v = count(k);
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL_MASK, inc, o);
      if (lane >= o) inc += y;
    }
    if (k < k1) {
      d.cell_start[off + k] = carry + inc - v;
      d.cell_count[off + k] = 0;
      d.cell_cursor[off + k] = 0;
    }
    carry += __shfl_sync(FULL_MASK, inc, 31);
  }
}

__global__ void __launch_bounds__(256) k_scatter(Dev d, Box b, int forced) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.nslot) rebuild_scatter(d, b, forced, i);
}

__global__ void __launch_bounds__(256) k_sort_gather(Dev d, Box b, int forced) {
  const int cell = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);  // up to 2^30 cells
  if (cell < b.ncell_all) rebuild_sort_gather(d, b, forced, cell);
}

template <int MODE>
__global__ void __launch_bounds__(BUILD_WARPS * 32, 4) k_build_group(Dev d, Box b, int forced) {
  __shared__ BuildStage stage[BUILD_WARPS];
  rebuild_build<MODE, false>(d, b, forced, stage[threadIdx.x >> 5], (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                             (gridDim.x * blockDim.x) >> 5, nullptr);
}

// few windows: a block of four warps each (BuildShare)
constexpr int SHARED_WINDOWS = 8;  // per SM
// blocks per window of a batch: its replicas' rows of cells are short and a window meets one
// to three of them, each a group with a chain of its own (step of 56 replicas: 92 us with 1, 89
// with 2, 92 with 3; of 24 in FP64 182, 177, 177)
constexpr int BATCH_SPLIT = 2;
template <int MODE>
__global__ void __launch_bounds__(128) k_build_shared(Dev d, Box b, int forced, int split) {
  __shared__ BuildShare share;
  rebuild_build<MODE, true>(d, b, forced, share.stage[threadIdx.x >> 5], blockIdx.x, gridDim.x, &share, split);
}

// after the build: count the rebuilt replicas, clear their flags and the global one;
// a build that overflowed its rows halts the chunk (the host grows the list and
// completes the step)
__global__ void __launch_bounds__(256) k_finish_rebuild(Dev d, Box b, int forced) {
  if (halted(d)) return;
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  int n = 0;
  for (int r = threadIdx.x; r < b.nrep; r += blockDim.x) {
    n += (forced || b.rep_flag[r] != 0) ? 1 : 0;
    b.rep_flag[r] = 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(FULL_MASK, n, o);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd_block(&total, n);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (total) {
      d.flags[F_REBUILDS] += total;
      d.flags[F_PASSES] += 1;
    }
    d.flags[F_REBUILD] = 0;
    if (d.flags[F_OVERFLOW]) d.flags[F_HALT] = 1;
  }
}

// Inside a captured step that starts with a drift kernel: a NaN the drift saw halts
// the chunk, and the half-skin flag becomes the value of the graph's conditional
// node that wraps the rebuild kernels (when the pair kernel drifted the step, its
// last block does both).
__global__ void k_set_rebuild_cond(Dev d, cudaGraphConditionalHandle h) {
  if (d.flags[F_NAN]) d.flags[F_HALT] = 1;
  cudaGraphSetConditional(h, (d.flags[F_REBUILD] != 0 && d.flags[F_HALT] == 0) ? 1u : 0u);
}

// the same NaN check for steps launched from the host (no conditional node)
__global__ void k_halt_check(Dev d) {
  if (d.flags[F_NAN]) d.flags[F_HALT] = 1;
}

// ---------------------------------------------------------------------------
// thermo: fold the per-block partials (fixed order) into KE, T, P, virial, PE
// (Atom_data::kinetic_energy_mpi_domain / finalize_temperature / finalize_pressure,
//  src/atom_data/kinetic_energy.cpp:26-134, 189-198, 238-303)
// thermo[] = {KE, T, P, virial, PE, sum m, -, -}
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_thermo_final(Dev d, ThermoCfg tc, int nb_ke, int nb_ev, int nb_ke_end,
                                                      int ring_slot) {
  if (halted(d)) return;  // every block alike: the ticket is not taken
  // level 1: block g folds partials g*256 + tid, stepping by the grid's threads (one
  // round of independent loads for up to 8192 partials)
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
  double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int k = gt; k < nb_ke; k += gs)
    for (int q = 0; q < 4; ++q) v[q] += d.partials_ke[(size_t)k * 4 + q];
  const double *ev = d.partials_ev;
  for (int k = gt; k < nb_ev; k += gs) {
    v[4] += ev[(size_t)k * 2];
    v[5] += ev[(size_t)k * 2 + 1];
  }
  for (int k = gt; k < nb_ke_end; k += gs)
    for (int q = 0; q < 4; ++q) v[6 + q] += d.partials_ke_end[(size_t)k * 4 + q];
  __shared__ double out[10];
  __shared__ bool last;
  block_sum_store<10>(v, out);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < 10; ++q) d.fold[blockIdx.x * 10 + q] = out[q];
    __threadfence();
    last = atomicAdd(d.fold_ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  // level 2, in the last block: the blocks' sums in block order.  All loads first
  // (L2-coherent, independent of one another), then the adds in block order: a
  // volatile load per add waited a full L2 round trip 32 times in a row
  if (threadIdx.x < 10) {
    __threadfence();
    double v[THERMO_FOLD_BLOCKS];
#pragma unroll
    for (int g = 0; g < THERMO_FOLD_BLOCKS; ++g) v[g] = __ldcg(&d.fold[g * 10 + threadIdx.x]);
    double s = 0.0;
#pragma unroll
    for (int g = 0; g < THERMO_FOLD_BLOCKS; ++g) s += v[g];
    out[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *d.fold_ticket = 0u;
    double res[5];
    const double P3[3] = {out[1], out[2], out[3]};
    // total mass is fixed at upload (thermo[5])
    thermo_finish(out[0], P3, d.thermo[5], out[4], out[5], tc.n, tc.n_r_df, tc.k_b, tc.volume, tc.langevin, res);
    if (nb_ke_end > 0) {  // KE as Atom_data::kinetic_energy() reads it after the step
      double e[5];
      const double Q3[3] = {out[7], out[8], out[9]};
      thermo_finish(out[6], Q3, d.thermo[5], 0.0, 0.0, tc.n, tc.n_r_df, tc.k_b, tc.volume, tc.langevin, e);
      res[0] = e[0];
    }
    for (int q = 0; q < 5; ++q) d.thermo[q] = res[q];
    if (ring_slot >= 0) {
      double *r = d.thermo_ring + (size_t)ring_slot * THERMO_REC;
      for (int q = 0; q < THERMO_REC; ++q) r[q] = res[q];
    }
  }
}

// Batches: one block per replica folds its slots in a fixed order.  ke: KE/T/P
// from the current velocities; ev: virial and PE from the per-slot sums the
// force kernel wrote (VV: P gets the virial term).  thermo_rep[r*8 + 0..5].
__global__ void __launch_bounds__(256) k_thermo_rep(Dev d, Box b, ThermoCfg tc, int ke, int ev) {
  if (halted(d)) return;
  const int rep = blockIdx.x;
  const RepBox &rb = repbox(b, rep);
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int i = rb.slot_off + threadIdx.x; i < rb.slot_off + rb.natoms; i += blockDim.x) {
    if (ke) {
      const dbl4 vv = d.vel[i];
      const double m = d.tab->mass[d.type[i]];
      v[0] += twice_ke(m, vv);
      v[1] += m * vv.x; v[2] += m * vv.y; v[3] += m * vv.z;
      v[4] += m;
    }
    if (ev) {
      const double2 e = d.ev_atom[i];
      v[5] += e.x;
      v[6] += e.y;
    }
  }
  __shared__ double out[7];
  block_sum_store<7>(v, out);
  __syncthreads();
  if (threadIdx.x == 0) {
    double *o = d.thermo_rep + (size_t)rep * 8;
    const double volume = rb.L[0] * rb.L[1] * rb.L[2];
    if (ke) {
      double res[5];
      const double P3[3] = {out[1], out[2], out[3]};
      thermo_finish(out[0], P3, out[4], 0.0, 0.0, rb.natoms, tc.n_r_df, tc.k_b, volume, 1, res);
      o[0] = res[0]; o[1] = res[1]; o[2] = res[2]; o[5] = out[4];
    }
    if (ev) {
      o[3] = 0.5 * out[5];
      o[4] = 0.5 * out[6];
      if (!tc.langevin) o[2] += o[3] / (3.0 * volume);
    }
  }
}

// end of a chunk: the step counter advances by the steps whose pair kernel ran; a
// halted chunk records how many that were (the host completes the failed step)
__global__ void k_advance_step(Dev d) {
  const int ok = d.flags[F_STEPS_OK];
  *d.step_base += ok;
  if (d.flags[F_HALT]) d.flags[F_HALT_STEP] += ok;
  d.flags[F_STEPS_OK] = 0;
}

// ---------------------------------------------------------------------------
// constraint::Nve (src/constraint/nve.cpp:132-184), single system: on steps whose
// index is a multiple of `step`, lambda = sqrt(target / KE) with KE the kinetic
// energy of Atom_data::kinetic_energy (centre-of-mass part removed for n_r_df
// 1..3), velocities scaled by lambda, then the temperature and pressure of the
// step follow the scaled velocities (finalize_temperature / finalize_pressure).
// ---------------------------------------------------------------------------
__device__ inline bool nve_applies(const Dev &d, const NveCfg &c, int k) {
  return !halted(d) && (*d.step_base + k) % c.step == 0;
}

__global__ void __launch_bounds__(256) k_nve_ke(Dev d, int n, NveCfg c, int k) {
  if (!nve_applies(d, c, k)) return;
  double part[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const dbl4 v = d.vel[i];
    const double m = d.tab->mass[d.type[i]];
    part[0] += twice_ke(m, v);
    part[1] += m * v.x; part[2] += m * v.y; part[3] += m * v.z;
  }
  block_sum_store<4>(part, &d.nve_partials[(size_t)blockIdx.x * 4]);
}

__global__ void __launch_bounds__(256) k_nve_lambda(Dev d, ThermoCfg tc, NveCfg c, int k, int thermo, int ring_slot) {
  if (!nve_applies(d, c, k)) return;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < NVE_BLOCKS; b += blockDim.x)
    for (int q = 0; q < 4; ++q) v[q] += d.nve_partials[(size_t)b * 4 + q];
  __shared__ double s[4];
  block_sum_store<4>(v, s);
  __syncthreads();
  if (threadIdx.x != 0) return;
  double ke2 = s[0];
  const double msum = d.thermo[5];
  if (tc.n_r_df >= 1 && tc.n_r_df <= 3 && msum > 0) ke2 -= (s[1] * s[1] + s[2] * s[2] + s[3] * s[3]) / msum;
  const double ke = 0.5 * ke2;
  const double dof = (double)(3 * tc.n - tc.n_r_df);  // Atom_data::degree_of_freedoms
  double lambda = 1.0;
  if (c.mode == CAVGPU_NVE_ENERGY_PER_DOF) lambda = sqrt(c.value * dof / ke);
  else if (c.mode == CAVGPU_NVE_ENERGY_TOT) lambda = sqrt(c.value / ke);
  else if (c.mode == CAVGPU_NVE_KBT) lambda = sqrt(dof * c.value * 0.5 / ke);
  else lambda = sqrt(dof * c.kb * c.value * 0.5 / ke);
  *d.nve_lambda = lambda;
  if (thermo) {  // the thermo point of this step: KE and T of the scaled velocities, P from them
    const double l2 = lambda * lambda;
    double *o = d.thermo;
    o[0] *= l2;
    o[1] *= l2;
    o[2] = ((double)tc.n * tc.k_b * o[1]) / tc.volume + (tc.langevin ? 0.0 : o[3]) / (3.0 * tc.volume);
    if (ring_slot >= 0)
      for (int q = 0; q < 3; ++q) d.thermo_ring[(size_t)ring_slot * THERMO_REC + q] = o[q];
  }
}

__global__ void __launch_bounds__(256) k_nve_scale(Dev d, int n, NveCfg c, int k) {
  if (!nve_applies(d, c, k)) return;
  const double lambda = *d.nve_lambda;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    dbl4 v = d.vel[i];
    v.x *= lambda; v.y *= lambda; v.z *= lambda;
    d.vel[i] = v;
  }
}

// ---------------------------------------------------------------------------
// parity exports
// ---------------------------------------------------------------------------
// The state in host order: positions wrapped as Domain::fix_position, velocities,
// accelerations, each where asked for (one pass over the ids and one launch for all).
__global__ void __launch_bounds__(256) k_state_to_host(Dev d, Box b, double *pos3, double *vel3, double *acc3) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.nslot) return;
  const int rep = rep_of_slot(b, k);
  if (rep < 0) return;
  const RepBox &rb = repbox(b, rep);
  const size_t h = ((size_t)rb.id_off + d.id[k]) * 3;
  if (pos3) {
    dbl4 v = d.pos[k];
    if (v.x < rb.lo[0]) v.x += rb.L[0]; else if (v.x > rb.hi[0]) v.x -= rb.L[0];
    if (v.y < rb.lo[1]) v.y += rb.L[1]; else if (v.y > rb.hi[1]) v.y -= rb.L[1];
    if (v.z < rb.lo[2]) v.z += rb.L[2]; else if (v.z > rb.hi[2]) v.z -= rb.L[2];
    pos3[h] = v.x; pos3[h + 1] = v.y; pos3[h + 2] = v.z;
  }
  if (vel3) {
    const dbl4 v = d.vel[k];
    vel3[h] = v.x; vel3[h + 1] = v.y; vel3[h + 2] = v.z;
  }
  if (acc3) {
    const dbl4 v = d.acc[k];
    acc3[h] = v.x; acc3[h + 1] = v.y; acc3[h + 2] = v.z;
  }
}

// boundary crossings in host order: the stored counts plus the wrap the current
// position still owes (the reference wraps every step, the device at list builds)
__global__ void __launch_bounds__(256) k_images_to_host(Dev d, Box b) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.nslot) return;
  const int rep = rep_of_slot(b, k);
  if (rep < 0) return;
  const int3 w = wrap_shift(repbox(b, rep), d.pos[k]);
  const int4 m = d.img[k];
  const size_t h = ((size_t)repbox(b, rep).id_off + d.id[k]) * 3;
  d.hi3[h] = m.x + w.x; d.hi3[h + 1] = m.y + w.y; d.hi3[h + 2] = m.z + w.z;
}

// canonical rows (id_i, id_j, sx, sy, sz) of the current list (single system)
__global__ void __launch_bounds__(256) k_export_pairs(Dev d, Box b, int mode, int32_t *rows,
                                                      unsigned long long *counter, long long cap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.nslot) return;
  const RepBox &rb = b.r0;
  const int ci = d.cell_of[i] - rb.cell_off;
  const int c3[3] = {ci % rb.nc[0], (ci / rb.nc[0]) % rb.nc[1], ci / (rb.nc[0] * rb.nc[1])};
  const int nn = d.nnbr[i];
  for (int k = 0; k < nn; ++k) {
    const uint32_t e = d.nbr[nbr_index(i, k, d.cap, d.tpa)];
    const int j = (int)(e & IDX_MASK), code = (int)(e >> CODE_SHIFT);
    int s[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
    if (mode == 1)  // cell-offset code -> image shift
      for (int q = 0; q < 3; ++q) {
        const int c = c3[q] + s[q];
        s[q] = c < 0 ? -1 : (c >= rb.nc[q] ? 1 : 0);
      }
    const unsigned long long r = atomicAdd(counter, 1ull);
    if ((long long)r < cap) {
      int32_t *o = rows + r * 5;
      o[0] = (int32_t)d.id[i]; o[1] = (int32_t)d.id[j]; o[2] = s[0]; o[3] = s[1]; o[4] = s[2];
    }
  }
}

struct RefBins {
  double lo[3], inv;
  int nb[3];
};

__device__ inline void ref_bin(const RefBins &rb, double x, double y, double z, int32_t *o) {
  const double q[3] = {x, y, z};
  for (int a = 0; a < 3; ++a) {
    int v = (int)floor((q[a] - rb.lo[a]) * rb.inv);
    if (v < 0) v = 0;
    if (v >= rb.nb[a]) v = rb.nb[a] - 1;
    o[a] = v;
  }
}

// Neighborlist::binlist_index of each atom at its wrapped position (host order)
__global__ void __launch_bounds__(256) k_ref_bins(Dev d, int n, RefBins rb) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n) return;
  ref_bin(rb, d.h3[3 * (size_t)h], d.h3[3 * (size_t)h + 1], d.h3[3 * (size_t)h + 2], &d.hi3[3 * (size_t)h]);
}

struct GhostCfg {
  double llow[3], lupp[3], L[3];
};

__device__ inline int ghost_vals(const GhostCfg &g, const double *q, int v[3]) {
  for (int a = 0; a < 3; ++a) v[a] = q[a] < g.llow[a] ? -1 : (q[a] > g.lupp[a] ? 1 : 0);
  const int nx = v[0] != 0, ny = v[1] != 0, nz = v[2] != 0;
  return nx + ny + nz + (nx & ny) + (nx & nz) + (ny & nz) + (nx & ny & nz);
}

__global__ void __launch_bounds__(256) k_ghost_count(Dev d, int n, GhostCfg g, int *counts) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n) return;
  int v[3];
  counts[h] = ghost_vals(g, &d.h3[3 * (size_t)h], v);
}

// images in the order x, y, z, xy, xz, yz, xyz with coordinate pos - val*width
// (src/atom_data/exchange_ghost_single_md_domain.cpp:163-214)
__global__ void __launch_bounds__(256) k_ghost_emit(Dev d, int n, GhostCfg g, const int *starts, int32_t *src,
                                                    int32_t *shift3, double *pos3, int32_t *bins3, long long cap,
                                                    RefBins rb) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n) return;
  const double *q = &d.h3[3 * (size_t)h];
  int v[3];
  ghost_vals(g, q, v);
  const double gx = q[0] - v[0] * g.L[0], gy = q[1] - v[1] * g.L[1], gz = q[2] - v[2] * g.L[2];
  const int combos[7][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
  long long o = starts[h];
  for (int c = 0; c < 7; ++c) {
    const int ux = combos[c][0], uy = combos[c][1], uz = combos[c][2];
    if ((ux && !v[0]) || (uy && !v[1]) || (uz && !v[2])) continue;
    if (o < cap) {
      const double p[3] = {ux ? gx : q[0], uy ? gy : q[1], uz ? gz : q[2]};
      src[o] = h;
      shift3[3 * o] = ux ? -v[0] : 0; shift3[3 * o + 1] = uy ? -v[1] : 0; shift3[3 * o + 2] = uz ? -v[2] : 0;
      pos3[3 * o] = p[0]; pos3[3 * o + 1] = p[1]; pos3[3 * o + 2] = p[2];
      ref_bin(rb, p[0], p[1], p[2], &bins3[3 * o]);
    }
    ++o;
  }
}

// exclusive scan of counts[0..m) into starts[0..m] (ghost export; one block)
__global__ void __launch_bounds__(1024) k_scan_plain(const int *count, int *start, int m) {
  __shared__ int warp_tot[32];
  __shared__ int carry_s;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (t == 0) carry_s = 0;
  __syncthreads();
  for (int base = 0; base < m; base += 1024) {
    const int k = base + t;
    const int s = k < m ? count[k] : 0;
    int inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL_MASK, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
      int wv = warp_tot[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL_MASK, wv, o);
        if (lane >= o) wv += y;
      }
      warp_tot[lane] = wv;
    }
    __syncthreads();
    const int run = carry_s + inc - s + (wid ? warp_tot[wid - 1] : 0);
    if (k < m) start[k] = run;
    __syncthreads();
    if (t == 1023) carry_s = run + s;
    __syncthreads();
  }
  if (t == 0) start[m] = carry_s;
}

// ---------------------------------------------------------------------------
// upload of a single system (cavgpu_upload): host layouts to slot arrays on the device
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_upload_single(Dev d, Box b, int n, int ntypes, int has_vel, int has_id,
                                                       const double *raw_pos, const double *raw_vel,
                                                       const uint64_t *raw_type, const uint64_t *raw_id, int *seen,
                                                       int *type_count) {
  // per-type counts of the block in shared memory, one global atomic per type and
  // block (one per atom on a single address serialised the whole upload)
  __shared__ int s_count[CAVGPU_MAX_TYPES];
  if (threadIdx.x < CAVGPU_MAX_TYPES) s_count[threadIdx.x] = 0;
  __syncthreads();
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h < n) {
    const RepBox &rb = b.r0;
    const double x = raw_pos[3 * (size_t)h], y = raw_pos[3 * (size_t)h + 1], z = raw_pos[3 * (size_t)h + 2];
    // Atom_data::position_inside_global_domain (src/atom_data.cpp:548-559)
    bool bad = !(x >= rb.lo[0] && x < rb.hi[0] && y >= rb.lo[1] && y < rb.hi[1] && z >= rb.lo[2] && z < rb.hi[2]);
    const uint64_t t = raw_type[h];
    bad |= t >= (uint64_t)ntypes;
    const uint64_t id = has_id ? raw_id[h] : (uint64_t)h;
    if (id >= (uint64_t)n) bad = true;
    else if (atomicExch(&seen[id], 1) != 0) bad = true;  // ids: a permutation of 0..n-1
    if (bad) {
      d.flags[F_UPLOAD_BAD] = 1;
    } else {
      atomicAdd_block(&s_count[t], 1);
      d.pos[h] = make_dbl4(x, y, z, type_bits((int)t));
      d.vel[h] = has_vel ? make_dbl4(raw_vel[3 * (size_t)h], raw_vel[3 * (size_t)h + 1], raw_vel[3 * (size_t)h + 2],
                                     0.0)
                         : make_dbl4(0.0, 0.0, 0.0, 0.0);
      d.type[h] = (int)t;
      d.id[h] = (uint32_t)id;
    }
  }
  __syncthreads();
  if (threadIdx.x < CAVGPU_MAX_TYPES && s_count[threadIdx.x]) atomicAdd(&type_count[threadIdx.x], s_count[threadIdx.x]);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int chk() { return cudaPeekAtLastError() == cudaSuccess ? CAVGPU_OK : CAVGPU_E_CUDA; }

int drift_grid_blocks(const LaunchCfg &lc) { return ceil_div(lc.n, 256); }

int launch_drift(const Dev &d, const Box &b, const StepConsts &sc, const LaunchCfg &lc, int k, int thermo,
                 cudaStream_t st) {
  const int g = drift_grid_blocks(lc);
  const bool mixed = lc.precision == CAVGPU_MIXED;
  if (lc.integrator == CAVGPU_VELOCITY_VERLET) {
    if (mixed) k_drift_vv<true><<<g, 256, 0, st>>>(d, b, sc);
    else k_drift_vv<false><<<g, 256, 0, st>>>(d, b, sc);
  } else if (lc.integrator == CAVGPU_LEAP_FROG) {
    if (mixed) k_drift_lf<true><<<g, 256, 0, st>>>(d, b, sc);
    else k_drift_lf<false><<<g, 256, 0, st>>>(d, b, sc);
  } else if (thermo < 0) {  // the velocity half only (constraint::Nve acts next)
    if (mixed) k_lang_a<true, false, false><<<g, 256, 0, st>>>(d, b, sc, k);
    else k_lang_a<false, false, false><<<g, 256, 0, st>>>(d, b, sc, k);
  } else {
    if (mixed) {
      if (thermo) k_lang_a<true, true, true><<<g, 256, 0, st>>>(d, b, sc, k);
      else k_lang_a<true, false, true><<<g, 256, 0, st>>>(d, b, sc, k);
    } else {
      if (thermo) k_lang_a<false, true, true><<<g, 256, 0, st>>>(d, b, sc, k);
      else k_lang_a<false, false, true><<<g, 256, 0, st>>>(d, b, sc, k);
    }
  }
  return chk();
}

int launch_lang_pos(const Dev &d, const Box &b, const StepConsts &sc, const LaunchCfg &lc, int thermo,
                    cudaStream_t st) {
  const int g = drift_grid_blocks(lc);
  if (lc.precision == CAVGPU_MIXED) {
    if (thermo) k_lang_pos<true, true><<<g, 256, 0, st>>>(d, b, sc);
    else k_lang_pos<true, false><<<g, 256, 0, st>>>(d, b, sc);
  } else {
    if (thermo) k_lang_pos<false, true><<<g, 256, 0, st>>>(d, b, sc);
    else k_lang_pos<false, false><<<g, 256, 0, st>>>(d, b, sc);
  }
  return chk();
}

int launch_rebuild(const Dev &d, const Box &b, const LaunchCfg &lc, int forced, cudaStream_t st) {
  const int g = ceil_div(b.nslot, 256);
  k_bin<<<g, 256, 0, st>>>(d, b, forced);
  const int P = scan_slices(b);
  if (P > 1) k_scan_part<<<P, 1024, 0, st>>>(d, b, forced);
  k_scan_rep<<<b.nrep * P, 1024, 0, st>>>(d, b, forced, P);
  k_scatter<<<g, 256, 0, st>>>(d, b, forced);
  k_sort_gather<<<ceil_div((long long)b.ncell_all * 32, 256), 256, 0, st>>>(d, b, forced);
  const int windows = ceil_div(b.nslot, 32), build_grid = std::min(ceil_div(windows, BUILD_WARPS), num_sms() * 32);
  const bool batch = b.nrep > 1;
  const int split = batch ? BATCH_SPLIT : 1;
  // one window per warp up to 1.2 M slots: with 8 blocks per SM a warp had 3 or 4 of them at
  // 1,048,576 atoms and the build 30 us of tail; up to SHARED_WINDOWS windows per SM (38,912
  // atoms) a window's own chain of work is the time: 33 us with its four warps, 46 us with one,
  // at 32,000 atoms.  Of a batch some replicas rebuild in a step, about a sixth when each does
  // so every sixth, so the line lies further up: a step of 56 replicas (1,900 windows) takes 89
  // us with four warps per window and 138 with one, of 128 (4,900) 137 and 178, but of 256
  // large ones (34,900) 511 and 426.
  if (shared_windows(lc) && windows <= num_sms() * SHARED_WINDOWS * (batch && !forced ? 8 : 1)) {
    if (stencil_codes(lc)) k_build_shared<1><<<windows * split, 128, 0, st>>>(d, b, forced, split);
    else k_build_shared<0><<<windows * split, 128, 0, st>>>(d, b, forced, split);
  } else if (stencil_codes(lc)) k_build_group<1><<<build_grid, BUILD_WARPS * 32, 0, st>>>(d, b, forced);
  else k_build_group<0><<<build_grid, BUILD_WARPS * 32, 0, st>>>(d, b, forced);
  if (lc.exchange) {
    const int rc = launch_exchange_build(d, b, forced, st);
    if (rc) return rc;
  }
  k_finish_rebuild<<<1, 256, 0, st>>>(d, b, forced);
  return chk();
}

int launch_set_rebuild_cond(const Dev &d, cudaGraphConditionalHandle h, cudaStream_t st) {
  k_set_rebuild_cond<<<1, 1, 0, st>>>(d, h);
  return chk();
}

int launch_halt_check(const Dev &d, cudaStream_t st) {
  k_halt_check<<<1, 1, 0, st>>>(d);
  return chk();
}

int launch_thermo_final(const Dev &d, const ThermoCfg &tc, int nb_ke, int nb_ev, int nb_ke_end, int ring_slot,
                        cudaStream_t st) {
  k_thermo_final<<<THERMO_FOLD_BLOCKS, 256, 0, st>>>(d, tc, nb_ke, nb_ev, nb_ke_end, ring_slot);
  return chk();
}

int launch_thermo_replicas(const Dev &d, const Box &b, const ThermoCfg &tc, int ke, int ev, cudaStream_t st) {
  k_thermo_rep<<<b.nrep, 256, 0, st>>>(d, b, tc, ke, ev);
  return chk();
}

int launch_advance_step(const Dev &d, cudaStream_t st) {
  k_advance_step<<<1, 1, 0, st>>>(d);
  return chk();
}

int launch_nve(const Dev &d, const Box &b, const ThermoCfg &tc, const NveCfg &cfg, int k, int thermo, int ring_slot,
               cudaStream_t st) {
  if (b.nrep != 1 || cfg.step <= 0) return CAVGPU_E_ARG;
  const int n = b.nslot;
  k_nve_ke<<<NVE_BLOCKS, 256, 0, st>>>(d, n, cfg, k);
  k_nve_lambda<<<1, 256, 0, st>>>(d, tc, cfg, k, thermo, ring_slot);
  k_nve_scale<<<NVE_BLOCKS, 256, 0, st>>>(d, n, cfg, k);
  return chk();
}

int launch_state_to_host(const Dev &d, const Box &b, double *pos3, double *vel3, double *acc3, cudaStream_t st) {
  k_state_to_host<<<ceil_div(b.nslot, 256), 256, 0, st>>>(d, b, pos3, vel3, acc3);
  return chk();
}

int launch_to_host_order(const Dev &d, const Box &b, cudaStream_t st) {
  return launch_state_to_host(d, b, d.h3, nullptr, nullptr, st);
}

int launch_images_to_host(const Dev &d, const Box &b, cudaStream_t st) {
  if (!d.img || !d.hi3) return CAVGPU_E_STATE;
  k_images_to_host<<<ceil_div(b.nslot, 256), 256, 0, st>>>(d, b);
  return chk();
}

int launch_export_pairs(const Dev &d, const Box &b, int mode, int32_t *rows, unsigned long long *counter,
                        int64_t cap, cudaStream_t st) {
  k_export_pairs<<<ceil_div(b.nslot, 256), 256, 0, st>>>(d, b, mode, rows, counter, (long long)cap);
  return chk();
}

int launch_ref_bins(const Dev &d, int n, double cutoff_inv, const int nb[3], const double lo_local[3],
                    cudaStream_t st) {
  RefBins rb;
  for (int a = 0; a < 3; ++a) { rb.lo[a] = lo_local[a]; rb.nb[a] = nb[a]; }
  rb.inv = cutoff_inv;
  k_ref_bins<<<ceil_div(n, 256), 256, 0, st>>>(d, n, rb);
  return chk();
}

int launch_upload_single(const Dev &d, const Box &b, int n, int ntypes, bool has_vel, bool has_id,
                         const double *raw_pos, const double *raw_vel, const uint64_t *raw_type,
                         const uint64_t *raw_id, int *seen, int *type_count, cudaStream_t st) {
  k_upload_single<<<ceil_div(n, 256), 256, 0, st>>>(d, b, n, ntypes, has_vel, has_id, raw_pos, raw_vel, raw_type,
                                                     raw_id, seen, type_count);
  return chk();
}

int launch_ghosts(const Dev &d, const Box &b, int n, double gc, int *counts, int *starts, int32_t *src,
                  int32_t *shift3, double *pos3, int32_t *bins3, int64_t cap, double cutoff_inv, const int nb[3],
                  const double lo_local[3], cudaStream_t st) {
  GhostCfg g;
  RefBins rb;
  for (int a = 0; a < 3; ++a) {
    g.llow[a] = b.r0.lo[a] + gc;
    g.lupp[a] = b.r0.hi[a] - gc;
    g.L[a] = b.r0.L[a];
    rb.lo[a] = lo_local[a];
    rb.nb[a] = nb[a];
  }
  rb.inv = cutoff_inv;
  k_ghost_count<<<ceil_div(n, 256), 256, 0, st>>>(d, n, g, counts);
  k_scan_plain<<<1, 1024, 0, st>>>(counts, starts, n);
  k_ghost_emit<<<ceil_div(n, 256), 256, 0, st>>>(d, n, g, starts, src, shift3, pos3, bins3, (long long)cap, rb);
  return chk();
}

}  // namespace cav
