// cav_chunk.cu -- the steps of a small system in one launch.
//
// A step of a captured graph costs about 28 us however small the system is (a conditional
// node and two or three kernels, each launched and drained; seven to nine more when the
// list is rebuilt), while the work of a few thousand atoms is done in a few microseconds.
// Here one cooperative launch runs all steps of a chunk: the blocks, all resident, go
// through the phases of a step with a grid barrier (0.3 us and the slowest block's wait)
// between -- mixed form: force with
// the closing update and the next drift; FP64 form: pairs, then the received forces with the
// same; and the phases of a rebuild when an atom has asked for one.  The phases are the
// device functions that the kernels run one each, with the same tasks, the same partial
// sums per (virtual) block and the same folds, so that the results equal those of the
// kernels bit for bit.
//
// Steps (LJ fluid, us, graph of kernels / here): mixed 4,000 atoms 23.3 / 12.4, 19,652 26.9 / 18.9,
// 32,000 31.0 / 22.6; FP64 500 atoms 29.8 / 19.9, 4,000 42.4 / 35.5.  Of 4,000 mixed atoms: force,
// kick and drift 4.7 (one walk through a list row, gather by gather, and ~45 FP64 instructions
// of 64 cycles per warp), barriers and phase starts 2, a rebuild every seventh step ~45 (build 17,
// bin, scan, scatter, sort and gather 13, barriers and the slowest blocks' waits the rest).
#include <algorithm>

#include "cav_drift.cuh"
#include "cav_exchange.cuh"
#include "cav_mixed.cuh"
#include "cav_rebuild.cuh"

namespace cav {

namespace {

constexpr int CHUNK_THREADS = 128;
constexpr int CHUNK_WARPS = CHUNK_THREADS / 32;
// FP64 form: the step kernel up to FP64_ATOMS (19,652 atoms: 102 us against 95 in a graph, whose
// pair kernel has more warps in flight)
constexpr int FP64_ATOMS = 12288;
// With more than a few replicas one rebuilds in nearly every step, and the kernels' rebuild,
// with more blocks than stay resident, takes less time: step of 4 replicas (4,900 slots) mixed
// 36.6 us here and 39.1 with kernels, FP64 67.2 and 69.4; of 8 (10,400) mixed 48.9 and 51.4,
// FP64 99.5 and 92.1; of 16 (5,200) mixed 73.9 and 66.6, FP64 120 and 101; of 36 (11,800)
// mixed 77.0 and 71.2.
constexpr int MAX_REPLICAS = 6;
// One block scans the cells of a replica while the others wait, at ~0.7 us per step and 1,000
// cells: step of a 4,000-atom droplet in boxes of 9,261, 42,875 and 1,225,043 cells mixed 22.7,
// 46.1 and 828 us here, 25.4, 26.3 and 59.4 with kernels, FP64 40.2, 63.2 and 836 against
// 47.8, 48.8 and 81.9; of 32,000 atoms mixed 32.8, 58.0 and 913 against 35.1, 36.0 and 71.2.  (The
// waits of boxes with 10^8 cells would run into the barrier's limit.)
constexpr int MAX_CELLS = 12288;
// And one warp sorts the n atoms of a cell, n^2 / 32 comparisons one after the other: rows of
// 2,048 words mean up to ~4,000 atoms in a cell and 10 ms, where 19,456 atoms in one cell (a box of
// two list cutoffs) would take most of the time a barrier waits.
constexpr int MAX_ROW = 2048;
// polls of a barrier before a block gives up (seconds): the launch is cooperative, so a block
// that never comes means a fault elsewhere.  The state is then half way through a step: the
// host reads F_STALL and the context does nothing more.  (No block goes on past a barrier
// that another gave up unless all had reached it.)
#ifndef CAV_BARRIER_POLLS
#define CAV_BARRIER_POLLS (1u << 21)
#endif
constexpr unsigned BARRIER_POLLS = CAV_BARRIER_POLLS;

struct ChunkArgs {
  Dev d;
  Box b;
  StepConsts sc;
  FoldArgs fa;
  int S, ev, fuse, drop;
  int nblk;        // virtual blocks of the force phase on recorded steps (the kernels' grid)
  int ncell, lang;
  int by_atom;     // FP64 form: a warp per atom evaluates the pairs (few atoms)
};

// Barrier of all blocks.  Block 0 adds what makes the word's top bit flip once the others
// have added one each (the construction of CUDA's cooperative groups); nothing has to be
// reset.  False when the barrier gave up.
__device__ __forceinline__ bool grid_barrier(const Dev &d) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned old = atomicAdd(d.barrier, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u);
    unsigned now, polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(d.barrier) : "memory");
    } while ((((old ^ now) & 0x80000000u) == 0u) && ++polls < BARRIER_POLLS);
    s_ok = polls < BARRIER_POLLS;
    if (!s_ok) d.flags[F_STALL] = 1;
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}

// the shared memory of a phase
template <bool MIXED>
union PhaseShared {
  BuildShare build;
  PairWarp<5> pairs[MIXED ? 1 : CHUNK_WARPS];
};

// exclusive scan of replica rep's cell counts by the block (k_scan_rep)
__device__ void scan_replica(const Dev &d, const RepBox &rb) {
  __shared__ int tot[CHUNK_WARPS];
  const int m = rb.ncell + 1, t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int seg = (m + CHUNK_THREADS - 1) / CHUNK_THREADS, k0 = min(m, t * seg), k1 = min(m, k0 + seg);
  int s = 0;
  for (int k = k0; k < k1; ++k) s += scan_count(d, rb, m, k);
  int inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) tot[wid] = inc;
  __syncthreads();
  int run = rb.slot_off + inc - s;
  for (int w = 0; w < wid; ++w) run += tot[w];
  for (int k = k0; k < k1; ++k) {
    const int v = scan_count(d, rb, m, k), c = rb.cell_off + k;
    d.cell_start[c] = run;
    d.cell_count[c] = 0;
    d.cell_cursor[c] = 0;
    run += v;
  }
  __syncthreads();
}

// A rebuild pass of the flagged replicas; `ic` = the coordinates current at this step.
// Not inlined: it runs once in several steps and would take the registers of the others.
// False when a barrier gave up.
template <bool MIXED, bool SHARED>
__device__ __noinline__ bool rebuild(const ChunkArgs &A, int4 *ic, PhaseShared<MIXED> &sh) {
  Dev d = A.d;
  d.ic = ic;
  const Box &b = A.b;
  const int nthr = gridDim.x * CHUNK_THREADS, wid = threadIdx.x >> 5, nwarp = gridDim.x * CHUNK_WARPS;
  const int thr = blockIdx.x * CHUNK_THREADS + threadIdx.x, warp = wid * gridDim.x + blockIdx.x;
  const int slots = (b.nslot + 31) & ~31;
  for (int i = thr; i < slots; i += nthr) rebuild_bin(d, b, 0, i);  // whole warps
  if (!grid_barrier(d)) return false;
  for (int r = blockIdx.x; r < b.nrep; r += gridDim.x)
    if (rebuild_on(d, b, r, 0)) scan_replica(d, repbox(b, r));
  if (!grid_barrier(d)) return false;
  for (int i = thr; i < b.nslot; i += nthr) rebuild_scatter(d, b, 0, i);
  if (!grid_barrier(d)) return false;
  for (int c = warp; c < A.ncell; c += nwarp) rebuild_sort_gather(d, b, 0, c);
  if (!grid_barrier(d)) return false;
  if constexpr (SHARED) rebuild_build<MIXED ? 1 : 0, true>(d, b, 0, sh.build.stage[wid], blockIdx.x, gridDim.x, &sh.build);
  else rebuild_build<MIXED ? 1 : 0, false>(d, b, 0, sh.build.stage[wid], warp, nwarp, nullptr);
  if (!grid_barrier(d)) return false;
  if (!MIXED) {
    for (int i = warp; i < b.nslot; i += nwarp) claim_slot(d, b, 0, i);
    if (!grid_barrier(d)) return false;
    for (int j = warp; j < b.nslot; j += nwarp) rank_slot(d, b, 0, j);
    if (!grid_barrier(d)) return false;
  }
  // count the rebuilt replicas and clear their flags before any block can raise one again
  if (blockIdx.x == 0) {
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    int n = 0;
    for (int r = threadIdx.x; r < b.nrep; r += CHUNK_THREADS) {
      n += b.rep_flag[r] != 0 ? 1 : 0;
      b.rep_flag[r] = 0;
    }
    if (n) atomicAdd_block(&total, n);
    __syncthreads();
    if (threadIdx.x == 0 && total) {
      d.flags[F_REBUILDS] += total;
      d.flags[F_PASSES] += 1;
    }
  }
  return grid_barrier(d);
}

// A phase of fewer blocks than the launch takes them from the end: of 608 blocks, four per SM, the
// first 16 sit on 4 SMs and the last 152 on as many.  (Langevin, a record every step, FP64,
// 4,000 atoms: 140 us a step with the drift's 16 blocks, 500 tasks and 125 closing blocks from the
// front, 74 from the end; 89 with kernels.  The steps between do not care.)
__device__ __forceinline__ int from_the_end() { return (int)(gridDim.x - 1 - blockIdx.x); }

// Drift at the start of a chunk, or of a step that the one before did not drift.  THERMO
// (Langevin): the mid-step sums per 256 slots, as the drift kernel's blocks leave them.
template <bool MIXED, bool LANG>
__device__ __forceinline__ void drift_phase(const Dev &d, const Box &b, const StepConsts &sc, int fuse, bool thermo,
                                            long long step) {
  if (LANG && thermo) {
    __shared__ double sh[8][4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int v = from_the_end(); v * 256 < sc.n; v += gridDim.x) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        double part[4] = {0.0, 0.0, 0.0, 0.0};
        const int i = v * 256 + half * CHUNK_THREADS + threadIdx.x;
        if (i < sc.n) lang_slot<MIXED, true, true>(d, b, sc, step, i, part);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) part[k] += __shfl_xor_sync(FULL_MASK, part[k], o);
        if (lane == 0)
#pragma unroll
          for (int k = 0; k < 4; ++k) sh[half * CHUNK_WARPS + wid][k] = part[k];
      }
      __syncthreads();
      if (threadIdx.x < 4) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += sh[w][threadIdx.x];
        d.partials_ke[(size_t)v * 4 + threadIdx.x] = s;
      }
      __syncthreads();
    }
    return;
  }
  const int nthr = gridDim.x * CHUNK_THREADS;
  for (int i = from_the_end() * CHUNK_THREADS + threadIdx.x; i < sc.n; i += nthr) {
    if (LANG) {
      double part[4];
      lang_slot<MIXED, false, true>(d, b, sc, step, i, part);
    } else if (fuse == FUSE_LF) {
      drift_slot_lf<MIXED>(d, b, sc, i);
    } else {
      drift_slot_vv<MIXED>(d, b, sc, i);
    }
  }
}

// force on the atoms of one task, their closing update and the next drift
template <int TPA, int KICK, bool EV, bool ONE>
__device__ __forceinline__ void mixed_task(const Dev &d, const Box &b, const StepConsts &sc, const SmemTabF &tab, int nt,
                                           int task, long long step, int fuse, double (&ke)[4], double (&ev)[2]) {
  constexpr int A = 32 / TPA;
  const int lane = threadIdx.x & 31, a = lane % A, t = lane / A;
  const int rep = rep_of_slot(b, task * A);
  if (rep < 0) return;  // a task of padding slots (uniform over the warp)
  const RepBox &rb = repbox(b, rep);
  const float4 uh = make_float4(rb.uh[0], rb.uh[1], rb.uh[2], 0.f), ul = make_float4(rb.ul[0], rb.ul[1], rb.ul[2], 0.f);
  const int i = task * A + a;
  const bool act = i < sc.n && rep_of_slot(b, i) >= 0;
  double fx = 0.0, fy = 0.0, fz = 0.0, vir = 0.0, pe = 0.0;
  int ti = 0;
  if (act) {
    const uint4 *row4 = reinterpret_cast<const uint4 *>(d.nbr + (size_t)task * d.cap * A) + (t * A + a);
    const int4 ri = d.ic[i];
    ti = ri.w;
    float ax = 0.f, ay = 0.f, az = 0.f;
    const int4 *ic = d.ic;
    mixed_pairs<TPA, EV, ONE, true>(row4, d.nnbr[i], t, ri, nt, tab, one_type(tab), uh, ul, sc.jump_tolf,
                                    [ic](uint32_t w) { return ic[w & IDX_MASK]; }, ax, ay, az, vir, pe);
    fx = ax; fy = ay; fz = az;
  }
  fold_lanes<A, EV>(fx, fy, fz, vir, pe);
  if (act && t == 0) {
    finish_atom<true, KICK, EV>(d, b, sc, tab, i, ti, rep, step, fuse, fx, fy, fz, ke);
    if (EV) set_ev(d, i, vir, pe, ev);
  }
}

// received forces of one task, the closing update and the next drift (FP64 form)
template <int TPA, int KICK, bool EV>
__device__ __forceinline__ void close_task(const Dev &d, const Box &b, const StepConsts &sc, const MassTab &tab, int task,
                                           long long step, int fuse, double (&ke)[4]) {
  constexpr int A = 32 / TPA;
  const int lane = threadIdx.x & 31, a = lane % A, t = lane / A, i = task * A + a;
  const int rep = i < sc.n ? rep_of_slot(b, i) : -1;
  double F[3];
  close_sum<TPA, true>(d, rep >= 0, i, t, F);
  if (rep >= 0 && t == 0) {
    finish_atom<false, KICK, EV>(d, b, sc, tab, i, d.type[i], rep, step, fuse, F[0], F[1], F[2], ke);
    if (EV && d.ev_part) close_ev<TPA>(d, i);
  }
}

// pair phase of the FP64 form: one task per warp, spread over the SMs first (the FP64 pipe
// is an SM's own); a recorded step leaves the partial sums of each task
template <int TPA, bool EV, bool ONE>
__device__ __forceinline__ void pair_phase(const Dev &d, const Box &b, const StepConsts &sc,
                                           const TabX<ONE ? 1 : MAXT * MAXT> &tab, PairWarp<5> &W5, int nt, int ntask) {
  PairWarp<EV ? 5 : 3> &W = reinterpret_cast<PairWarp<EV ? 5 : 3> &>(W5);
  const int nwarp = gridDim.x * CHUNK_WARPS;
  const int block = EV ? from_the_end() : (int)blockIdx.x;
  for (int task = (threadIdx.x >> 5) * gridDim.x + block; task < ntask; task += nwarp) {
    double ev[2] = {0.0, 0.0};
    const int rep = rep_of_slot(b, task * (32 / TPA));
    if (rep >= 0) pair_tasks<TPA, EV, ONE, true>(d, b, sc, tab, W, nt, rep, task, task + 1, ev);
    if (EV) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ev[k] += __shfl_xor_sync(FULL_MASK, ev[k], o);
      if ((threadIdx.x & 31) == 0) {
        d.partials_ev[(size_t)task * 2] = 0.0 + ev[0];
        d.partials_ev[(size_t)task * 2 + 1] = 0.0 + ev[1];
      }
    }
  }
}

// SHARED: windows of a list build shared by a block's warps (shared_windows; both builds in one
// kernel cost 0.3 us a step, in the instruction cache)
template <bool MIXED, int TPA, int KICK, bool ONE, bool SHARED>
__global__ void __launch_bounds__(CHUNK_THREADS, 4) k_chunk(const __grid_constant__ ChunkArgs A) {
  constexpr int ATOMS = 32 / TPA;
  __shared__ PhaseShared<MIXED> sh;
  __shared__ typename std::conditional<MIXED, SmemTabF, TabX<ONE ? 1 : MAXT * MAXT>>::type tab;
  __shared__ MassTab mtab;
  if (halted(A.d) || stalled(A.d)) return;  // a chunk after a halt does nothing (the same for every block)
  Dev d = A.d;
  const Box &b = A.b;
  const StepConsts &sc = A.sc;
  if (!MIXED) d.pos_alt = d.pos;  // the FP64 form drifts in place (the pairs are a phase of their own)
  if constexpr (MIXED) load_tab(d, tab);
  else load_tabx<true, ONE>(d, tab);
  mtab.load(d);
  __syncthreads();
  const int nt = d.tab->nt, wid = threadIdx.x >> 5, nwarp = gridDim.x * CHUNK_WARPS;
  const int warp = wid * gridDim.x + blockIdx.x, ntask = (sc.n + ATOMS - 1) / ATOMS;
  const long long step0 = *d.step_base;
  volatile int *const flags = d.flags;
  // Rebuild requests and NaNs go to the word of the phase in which a drift runs (phases
  // are counted modulo 3) and are read after the phase's barrier; the word of the phase
  // before is cleared by then, two barriers before it is used again.
  int q = flags[F_PHASE], done = 0, rec = 0;
  bool halt = false, nan = false, need = false, drifted = false;
  auto phase_end = [&]() -> bool {
    if (!grid_barrier(d)) return false;
    need = flags[F_PHASE_REQ + q] != 0;
    nan = flags[F_PHASE_NAN + q] != 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const int p = q == 0 ? 2 : q - 1;
      flags[F_PHASE_REQ + p] = 0;
      flags[F_PHASE_NAN + p] = 0;
    }
    q = q == 2 ? 0 : q + 1;
    return true;
  };
  auto recorded = [&](int k) { return A.ev > 0 && (k + 1) % A.ev == 0; };

  for (int k = 0; k < A.S; ++k) {
    const bool th = recorded(k);
    const long long step = step0 + k;
    // recorded steps alternate between two sets of partial sums: block 0 may fold one while
    // the others are already at the next recorded step
    const size_t alt = th && (rec & 1) ? (size_t)d.partials_alt : 0;
    Dev v = d;
    v.partials_ke += 4 * alt;
    v.partials_ke_end += 4 * alt;
    v.partials_ev += 2 * alt;
    if (!drifted) {
      v.req = A.d.flags + F_PHASE_REQ + q;
      v.nan = A.d.flags + F_PHASE_NAN + q;
      drift_phase<MIXED, KICK == 2>(v, b, sc, A.fuse, th, step);
      if (!phase_end()) return;
    }
    if (nan) {
      halt = true;
      break;
    }
    if (need) {
      if (!rebuild<MIXED, SHARED>(A, d.ic, sh)) return;
      if (flags[F_OVERFLOW]) {
        // the host completes the step and folds its record from the first set of sums: a
        // Langevin step's temperature sums, of its drift above, go there (block 0 has folded
        // the record before, if that was in it)
        if (KICK == 2 && alt && blockIdx.x == 0)
          for (int i = threadIdx.x; i < 4 * ((sc.n + 255) / 256); i += CHUNK_THREADS) d.partials_ke[i] = v.partials_ke[i];
        halt = true;
        break;
      }
    }
    const bool fuse = k + 1 < A.S && !(A.lang && recorded(k + 1)) && !(A.fuse == FUSE_LF && th) && k != A.drop;
    const int fuse_mode = fuse ? A.fuse : FUSE_NONE;
    v.req = A.d.flags + F_PHASE_REQ + q;
    v.nan = A.d.flags + F_PHASE_NAN + q;
    if constexpr (!MIXED) {
      if (th) {
        pair_phase<TPA, true, ONE>(v, b, sc, tab, sh.pairs[wid], nt, ntask);
      } else if (A.by_atom) {
        double(*const share)[3] = reinterpret_cast<double(*)[3]>(&sh.pairs[wid]);
        for (int i = warp; i < sc.n; i += nwarp) pair_atom<ONE>(v, b, sc, tab, share, nt, i);
      } else {
        pair_phase<TPA, false, ONE>(v, b, sc, tab, sh.pairs[wid], nt, ntask);
      }
      if (!grid_barrier(d)) return;
    }
    double ke[4] = {0.0, 0.0, 0.0, 0.0}, ev[2] = {0.0, 0.0};
    if (th) {  // four tasks to a virtual block, as the kernels' blocks hold them
      for (int vb = from_the_end(); vb < A.nblk; vb += gridDim.x) {
        const int task = vb * CHUNK_WARPS + wid;
        ke[0] = ke[1] = ke[2] = ke[3] = ev[0] = ev[1] = 0.0;
        if (task < ntask) {
          if constexpr (MIXED) mixed_task<TPA, KICK, true, ONE>(v, b, sc, tab, nt, task, step, fuse_mode, ke, ev);
          else close_task<TPA, KICK, true>(v, b, sc, mtab, task, step, fuse_mode, ke);
        }
        if constexpr (MIXED) {
          block_sum_store<2>(ev, &v.partials_ev[(size_t)vb * 2]);
          __syncthreads();
        }
        block_sum_store<4>(ke, &(KICK == 2 ? v.partials_ke_end : v.partials_ke)[(size_t)vb * 4]);
        __syncthreads();
      }
    } else {
      for (int task = warp; task < ntask; task += nwarp) {
        if constexpr (MIXED) mixed_task<TPA, KICK, false, ONE>(v, b, sc, tab, nt, task, step, fuse_mode, ke, ev);
        else close_task<TPA, KICK, false>(v, b, sc, mtab, task, step, fuse_mode, ke);
      }
    }
    need = nan = false;
    if (!phase_end()) return;
    ++done;
    if (MIXED && fuse) {
      int4 *const t = d.ic;
      d.ic = d.ic_alt;
      d.ic_alt = t;
    }
    drifted = fuse;
    if (nan) {
      halt = true;
      break;
    }
    if (th) {
      if (blockIdx.x == 0) {
        Dev w = A.d;  // (a copy in memory, for a function that is not inlined)
        w.partials_ke += 4 * alt;
        w.partials_ke_end += 4 * alt;
        w.partials_ev += 2 * alt;
        FoldArgs fa = A.fa;
        fa.ring_slot = (k + 1) / A.ev - 1;
        fold_thermo(w, fa);
        __syncthreads();
      }
      ++rec;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    flags[F_PHASE] = q;
    *d.step_base = step0 + done;
    if (nan) flags[F_NAN] = 1;
    if (halt) {
      flags[F_HALT] = 1;
      flags[F_HALT_STEP] = flags[F_HALT_STEP] + done;
    }
  }
}

template <bool MIXED, int TPA, int KICK, bool ONE, bool SHARED>
int go(const ChunkArgs &A, int want, int share, cudaStream_t st) {
  static PerDevice blocks_per_sm;  // resident
  const int per_sm = blocks_per_sm.get([](int) {
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_chunk<MIXED, TPA, KICK, ONE, SHARED>, CHUNK_THREADS, 0);
    return e == cudaSuccess && n > 0 ? n : -1;
  });
  if (per_sm < 1) return CAVGPU_E_CUDA;
  // Contexts stepped at the same time (threads) divide the blocks that can be resident: a
  // launch whose blocks do not fit beside the running ones waits for them to end.  Time per
  // step and context of 4 contexts of 4,000 atoms, each on its own / sharing / as graphs of
  // kernels, which overlap: mixed 14.8 / 3.9 / 8.0 us, FP64 35.5 / 19.6 / 20.8; of 19,652 atoms mixed
  // 18.7 / 10.3 / 11.7; of 8 contexts of 48,668 mixed 33.1 / 21.7 / 21.6.
  const int grid = std::max(1, std::min(want, num_sms() * per_sm / std::min(std::max(share, 1), 4)));
  void *args[] = {const_cast<ChunkArgs *>(&A)};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_chunk<MIXED, TPA, KICK, ONE, SHARED>), dim3(grid),
                                     dim3(CHUNK_THREADS), args, 0, st) == cudaSuccess
             ? CAVGPU_OK
             : CAVGPU_E_CUDA;
}

template <bool MIXED, int TPA, bool SHARED>
int pick_kick(const ChunkArgs &A, int kick, bool one, int want, int share, cudaStream_t st) {
  if (kick == 1)
    return one ? go<MIXED, TPA, 1, true, SHARED>(A, want, share, st) : go<MIXED, TPA, 1, false, SHARED>(A, want, share, st);
  return one ? go<MIXED, TPA, 2, true, SHARED>(A, want, share, st) : go<MIXED, TPA, 2, false, SHARED>(A, want, share, st);
}

template <bool MIXED, int TPA>
int pick(const ChunkArgs &A, const LaunchCfg &lc, int kick, int want, int share, cudaStream_t st) {
  const bool one = lc.ntypes == 1;
  return shared_windows(lc) ? pick_kick<MIXED, TPA, true>(A, kick, one, want, share, st)
                            : pick_kick<MIXED, TPA, false>(A, kick, one, want, share, st);
}

}  // namespace

// Sizes for which the kernels' blocks hold one task per warp (the partial sums are then
// those of the virtual blocks), at the lane counts small systems use.
bool chunk_fits(const Box &b, const LaunchCfg &lc) {
  if (b.nrep > MAX_REPLICAS || b.ncell_all > MAX_CELLS || lc.row > MAX_ROW) return false;
  if (lc.images) return false;  // (k_force alone applies image codes to fixed-point coordinates)
  if (lc.use_seg || lc.block != CHUNK_THREADS || (lc.tpa != 2 && lc.tpa != 4)) return false;
  if (lc.precision == CAVGPU_FP64 && (!lc.exchange || lc.tpa != 4 || lc.n > FP64_ATOMS)) return false;
  const int ntask = (lc.n + 32 / lc.tpa - 1) / (32 / lc.tpa);
  // Long rows: no more than a task per resident warp, 16 per SM; the kernels keep twice the warps
  // in flight.  Mixed, 281 words per row, 32,000 and 42,592 atoms 53.0 and 74.0 us here, 62.8 and
  // 70.8 with kernels; 526 words 85.7 and 140 against 95.9 and 118; 127 words 28.2 and 39.9
  // against 37.0 and 44.7.
  if (lc.precision == CAVGPU_MIXED && lc.row > LONG_ROW && ntask > num_sms() * 16) return false;
  if (force_grid_blocks(lc) * CHUNK_WARPS < ntask) return false;
  return !lc.exchange || ev_grid_blocks(lc) >= ntask;
}

int launch_chunk(const Dev &d, const Box &b, const StepConsts &sc, const LaunchCfg &lc, int S, int ev, int fuse, int drop,
                 const FoldArgs &fa, int share, cudaStream_t st) {
  if (lc.precision == CAVGPU_FP64 && (!lc.exchange || !d.recv)) return CAVGPU_E_ARG;
  ChunkArgs A{d, b, sc, fa, S, ev, fuse, drop, force_grid_blocks(lc), b.ncell_all, fuse == FUSE_LANG, lc.n <= BY_ATOM};
  A.d.step_kernel = 1;
  // Mixed: four lanes a task per warp, and a warp per atom (the rebuild's phases) up to a block per
  // multiprocessor (4,000 atoms 12.4 us a step, with a block per task 13.4, with a warp per atom
  // 14.9: more blocks to wait for at every barrier; 500 atoms 11.3, with a block per task 11.7,
  // which does where others are at work); two lanes, whose systems are larger, a block per task
  // (32,000 atoms 22.75 against 23.03).  FP64: a block per task, a warp per atom where those
  // evaluate the pairs (the FP64 pipe is an SM's own: 1,372 atoms 24.5 us, with a task per warp
  // 27.6).
  const int ntask = (lc.n + 32 / lc.tpa - 1) / (32 / lc.tpa);
  const int want = lc.precision == CAVGPU_FP64 ? std::max(ntask, A.by_atom ? lc.n / CHUNK_WARPS : 0)
                   : lc.tpa == 4 ? std::max((ntask + CHUNK_WARPS - 1) / CHUNK_WARPS,
                                                std::min(share > 1 ? ntask : lc.n / CHUNK_WARPS, num_sms()))
                                 : ntask;
  const int kick = fuse == FUSE_LANG ? 2 : 1;
  if (lc.precision == CAVGPU_MIXED)
    return lc.tpa == 2 ? pick<true, 2>(A, lc, kick, want, share, st) : pick<true, 4>(A, lc, kick, want, share, st);
  return pick<false, 4>(A, lc, kick, want, share, st);
}

}  // namespace cav
