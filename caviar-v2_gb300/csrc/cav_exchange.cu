// cav_exchange.cu -- the FP64 form's pair force with every pair evaluated once
// (force_field::Lj::calculate_acceleration, src/force/lj.cpp:393-517).
//
// The FP64 pipe (2 thread instructions per SM and cycle) bounds the FP64 form, so the
// work taken off it counts and little else does.  A step is two kernels:
//   k_pairs64  every pair is claimed by one of its two atoms (claims()).  An atom walks the
//              entries it claimed, evaluates those inside the cutoff, adds the force to its
//              own sum and stores the opposite force in a slot of the other atom's (systems
//              of few atoms: k_atoms64, a warp per atom);
//   k_close64  every atom adds the forces it received to its own sum, in a fixed order,
//              then does the closing update of the step and the next drift.
// Which pairs are near the cutoff is decided off the FP64 pipe, on FP32 differences of
// fixed-point coordinates with a margin far above their error; entries that pass wait in a
// queue per lane until every lane has one, so that the lanes of a warp evaluate together.
// The sums do not depend on the lane count (1, 2 or 4 per atom), nor on the order in which
// the blocks of k_claim took receiving slots (k_rank sorts them): reruns, batches and
// launch shapes give the same bits.
//
// Against one kernel over the full list (19 FP64 instructions per entry once any lane of
// the warp is inside the cutoff): 20 per pair inside it, once per pair, plus 3 to add the
// received force.  LJ fluid, force of a step: 1,048,576 atoms 3.81 -> 1.87 ms, 131,072 atoms
// 0.52 -> 0.28 ms; of that k_pairs64 three quarters (FP64 pipe 80-85% busy, 691 FP64
// instructions per 32 atoms and warp against 557 that its lanes need) and k_close64 one (79%,
// 204 instructions, 1.6 KB read per atom, 1.2 of it received forces).  A build takes 1.2 ms longer at 1,048,576 atoms
// (k_claim 0.7: its atomics and scattered notes; k_rank 0.5: issue), 0.2 ms per step.
// Tried: all lanes of a warp on one atom after the other in step (1.0-1.05 of the time);
// each warp in a region of its own (1.5 times the time: the handed-over forces then go to
// the whole array at once).
#include <algorithm>

#include "cav_exchange.cuh"

namespace cav {

namespace {

constexpr int CLOSE_THREADS = 128;

// One warp per block.  A warp takes runs of RUN consecutive tasks (A slots each, one
// replica at a time), strided by the grid: the warps together move through the system, so
// that the forces they hand over go to a few MB of it.
template <int TPA, bool EV, bool ONE>
__global__ void __launch_bounds__(32, MINB) k_pairs64(Dev d, Box b, StepConsts sc, int RUN) {
  constexpr int A = 32 / TPA;
  __shared__ TabX<ONE ? 1 : MAXT * MAXT> tab;
  __shared__ PairWarp<EV ? 5 : 3> W;
  if (halted(d)) return;
  load_tabx<EV, ONE>(d, tab);
  const int nt = d.tab->nt, ntask = (sc.n + A - 1) / A;
  double ev_p[2] = {0.0, 0.0};
  for (int run = blockIdx.x; run * RUN < ntask; run += gridDim.x) {
    const int task_end = min(ntask, (run + 1) * RUN);
    for (int task = run * RUN; task < task_end;) {
      const int rep = rep_of_slot(b, task * A);
      task = rep < 0 ? task + 1  // padding slots
                     : pair_tasks<TPA, EV, ONE, false>(d, b, sc, tab, W, nt, rep, task, task_end, ev_p);
    }
  }
  if (EV) block_sum_store<2>(ev_p, &d.partials_ev[(size_t)blockIdx.x * 2]);
}

// Few atoms: a warp each, unless virial and energy are wanted.  A step as a graph of kernels
// (constraint::Nve) of 500 / 4,000 atoms: 39.8 / 54.7 us, with k_pairs64 54.9 / 59.0.
constexpr int ATOM_WARPS = 4;
template <bool ONE>
__global__ void __launch_bounds__(32 * ATOM_WARPS) k_atoms64(Dev d, Box b, StepConsts sc) {
  __shared__ TabX<ONE ? 1 : MAXT * MAXT> tab;
  __shared__ double share[ATOM_WARPS][32][3];
  if (halted(d)) return;
  load_tabx<false, ONE>(d, tab);
  __syncthreads();
  const int i = blockIdx.x * ATOM_WARPS + (threadIdx.x >> 5);
  if (i < sc.n) pair_atom<ONE>(d, b, sc, tab, share[threadIdx.x >> 5], d.tab->nt, i);
}

// Received forces, closing update, the end of the step.
template <int TPA, int KICK, bool EV>
__global__ void __launch_bounds__(CLOSE_THREADS) k_close64(Dev d, Box b, StepConsts sc, ForceArgs fa) {
  constexpr int A = 32 / TPA;
  __shared__ MassTab tab;
  __shared__ int s_halt;
  if (threadIdx.x == 0) s_halt = halted(d);
  tab.load(d);
  __syncthreads();
  const bool was_halted = s_halt != 0;  // a step after a halt does nothing
  const int lane = threadIdx.x & 31, a = lane % A, t = lane / A;
  const int n = sc.n, warps_total = (gridDim.x * blockDim.x) >> 5, ntask = was_halted ? 0 : (n + A - 1) / A;
  long long step = 0;
  if (KICK == 2) step = *d.step_base + fa.k_in_chunk;
  double ke_p[4] = {0.0, 0.0, 0.0, 0.0};
  for (int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < ntask; task += warps_total) {
    const int i = task * A + a;
    const int rep = i < n ? rep_of_slot(b, i) : -1;
    double F[3];
    close_sum<TPA, false>(d, rep >= 0, i, t, F);
    if (rep >= 0 && t == 0) {
      double ke[4];
      finish_atom<false, KICK, EV>(d, b, sc, tab, i, d.type[i], rep, step, fa.fuse, F[0], F[1], F[2], ke);
      if (EV)
#pragma unroll
        for (int q = 0; q < 4; ++q) ke_p[q] += ke[q];
      if (EV && d.ev_part) close_ev<TPA>(d, i);
    }
  }
  if (EV && !was_halted)
    block_sum_store<4>(ke_p, &(KICK == 2 ? d.partials_ke_end : d.partials_ke)[(size_t)blockIdx.x * 4]);
  if (KICK != 0) end_of_step<EV>(d, was_halted, fa);
}

__global__ void __launch_bounds__(256) k_claim(Dev d, Box b, int forced) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i < b.nslot) claim_slot(d, b, forced, i);
}

__global__ void __launch_bounds__(256) k_rank(Dev d, Box b, int forced) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j < b.nslot) rank_slot(d, b, forced, j);
}

int exchange_run(int ntask) { return ntask >= num_sms() * MINB * 8 ? 4 : 1; }

inline int chk() { return cudaPeekAtLastError() == cudaSuccess ? CAVGPU_OK : CAVGPU_E_CUDA; }

template <int TPA>
void pairs(bool ev, bool one, int grid, int run, const Dev &d, const Box &b, const StepConsts &sc, cudaStream_t st) {
  if (ev) {
    if (one) k_pairs64<TPA, true, true><<<grid, 32, 0, st>>>(d, b, sc, run);
    else k_pairs64<TPA, true, false><<<grid, 32, 0, st>>>(d, b, sc, run);
  } else {
    if (one) k_pairs64<TPA, false, true><<<grid, 32, 0, st>>>(d, b, sc, run);
    else k_pairs64<TPA, false, false><<<grid, 32, 0, st>>>(d, b, sc, run);
  }
}

template <int TPA, int KICK>
void close_kick(bool ev, int grid, const Dev &d, const Box &b, const StepConsts &sc, const ForceArgs &fa,
                cudaStream_t st) {
  if (ev) k_close64<TPA, KICK, true><<<grid, CLOSE_THREADS, 0, st>>>(d, b, sc, fa);
  else k_close64<TPA, KICK, false><<<grid, CLOSE_THREADS, 0, st>>>(d, b, sc, fa);
}

template <int TPA>
void both(int kick, bool ev, bool one, int grid, int grid_ev, const Dev &d, const Box &b, const StepConsts &sc,
          const ForceArgs &fa, cudaStream_t st) {
  constexpr int A = 32 / TPA;
  const int run = exchange_run((sc.n + A - 1) / A);
  if (!ev && sc.n <= BY_ATOM) {
    const int blocks = (sc.n + ATOM_WARPS - 1) / ATOM_WARPS;
    if (one) k_atoms64<true><<<blocks, 32 * ATOM_WARPS, 0, st>>>(d, b, sc);
    else k_atoms64<false><<<blocks, 32 * ATOM_WARPS, 0, st>>>(d, b, sc);
  } else {
    pairs<TPA>(ev, one, grid_ev, run, d, b, sc, st);
  }
  if (kick == 0) close_kick<TPA, 0>(ev, grid, d, b, sc, fa, st);
  else if (kick == 1) close_kick<TPA, 1>(ev, grid, d, b, sc, fa, st);
  else close_kick<TPA, 2>(ev, grid, d, b, sc, fa, st);
}

}  // namespace

// k_pairs64: one wave of resident warps.  Runs of four tasks (its lanes then evaluate 691
// instead of 731 FP64 instructions per task) once every warp has eight tasks; below that
// the longer runs leave too few warps in flight.  131,072 atoms: 283 us with runs of one,
// 293 with runs of four; 1,048,576 atoms: 1931 and 1867 (both kernels together).
int exchange_pair_blocks(int ntask) {
  const int run = exchange_run(ntask);
  return std::max(1, std::min((ntask + run - 1) / run, num_sms() * MINB));
}
int exchange_close_threads() { return CLOSE_THREADS; }

int launch_exchange_build(const Dev &d, const Box &b, int forced, cudaStream_t st) {
  const int grid = (int)(((long long)b.nslot * 32 + 255) / 256);  // a warp per atom
  k_claim<<<grid, 256, 0, st>>>(d, b, forced);
  k_rank<<<grid, 256, 0, st>>>(d, b, forced);
  return chk();
}

int launch_force_exchange(const Dev &dev, const Box &b, const StepConsts &sc, const LaunchCfg &lc, int kick, bool ev,
                          const ForceArgs &fa, int grid, int grid_ev, cudaStream_t st) {
  Dev d = dev;
  d.pos_alt = d.pos;  // the drift is a kernel of its own here: positions in place
  const bool one = lc.ntypes == 1;
  switch (lc.tpa) {
    case 1: both<1>(kick, ev, one, grid, grid_ev, d, b, sc, fa, st); break;
    case 2: both<2>(kick, ev, one, grid, grid_ev, d, b, sc, fa, st); break;
    case 4: both<4>(kick, ev, one, grid, grid_ev, d, b, sc, fa, st); break;
    default: return CAVGPU_E_ARG;
  }
  return chk();
}

}  // namespace cav
