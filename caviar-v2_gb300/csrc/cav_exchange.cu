// cav_exchange.cu -- the FP64 form's pair force with every pair evaluated once
// (force_field::Lj::calculate_acceleration, src/force/lj.cpp:393-517).
//
// The FP64 pipe (2 thread instructions per SM and cycle) bounds the FP64 form, so the
// work taken off it counts and little else does.  A step is two kernels:
//   k_pairs64  every pair is claimed by one of its two atoms (claims()).  An atom walks the
//              entries it claimed, evaluates those inside the cutoff, adds the force to its
//              own sum and stores the opposite force in a slot of the other atom's;
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
// 204 instructions, 1.6 KB read per atom).  A build takes 1.2 ms longer at 1,048,576 atoms
// (k_claim 0.7: its atomics and scattered notes; k_rank 0.5: issue), 0.2 ms per step.
// Tried: all lanes of a warp on one atom after the other in step (1.0-1.05 of the time);
// each warp in a region of its own (1.5 times the time: the handed-over forces then go to
// the whole array at once).
#include <algorithm>

#include "cav_pair.cuh"

namespace cav {

namespace {

constexpr int MINB = 20;        // resident warps per SM (one per block)
constexpr int RING = 16;        // queued entries per lane
constexpr int CLOSE_THREADS = 128;

// Which atom of a listed pair evaluates it.  By parity and order of the slots: either
// about half the time, and unchanged when a replica's slots are shifted by whole warps.
__device__ __forceinline__ bool claims(int i, int j) { return (((i ^ j) & 1) != 0) == (i < j); }

__device__ __forceinline__ size_t recv_index(int j, int r, int cap_h) {
  return ((size_t)(j >> 5) * cap_h + r) * 32 + (j & 31);
}

// 1 / x by one third-order step (Chebyshev's iteration) from the hardware approximation:
// e = 1 - x y, y (1 + e + e^2) leaves e^3, far below 2^-53 for an approximation to 20 bits.
// Three FP64 instructions; both orders of a pair use the one value.
__device__ __forceinline__ double rcp_cubic(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// Constants of the type pairs.  coef(r) = (w12 u^3 + w6) u^3 u - gc and
// V(r) = (l12 u^3 - l6) u^3 - uc - gc/2 (r^2 - rc2) with u = 1/r^2.
template <int N>
struct TabX {
  double rc2[N], w12[N], w6[N], gc[N], l12[N], l6[N], uc[N];
  float screen[N];
};

// A lane's queue and partial sums, its warp's image shifts.
template <int NV>
struct PairWarp {
  uint2 ring[RING][32];   // {list word, receiving slot | partial sum << 16}
  double sum[4][NV][32];  // {force, virial, potential energy} per partial sum (RowSplit)
  double3 img[27];
};

// the list words and receiving slots of a lane's entries of one chunk
template <int PER>
struct ChunkWords {
  uint32_t w[PER];
  uint32_t s[(PER + 1) / 2];  // two 16-bit slots a word
  __device__ __forceinline__ void load(const Dev &d, size_t at) {
    if constexpr (PER == 4) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(d.hw + at));
      const uint2 x = __ldg(reinterpret_cast<const uint2 *>(d.hslot + at));
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
      s[0] = x.x; s[1] = x.y;
    } else if constexpr (PER == 2) {
      const uint2 v = __ldg(reinterpret_cast<const uint2 *>(d.hw + at));
      w[0] = v.x; w[1] = v.y;
      s[0] = __ldg(reinterpret_cast<const uint32_t *>(d.hslot + at));
    } else {
      w[0] = __ldg(d.hw + at);
      s[0] = __ldg(d.hslot + at);
    }
  }
  __device__ __forceinline__ uint32_t word(int u) const { return w[u]; }
  __device__ __forceinline__ uint32_t slot(int u) const { return PER == 1 ? s[0] : (s[u >> 1] >> (16 * (u & 1))) & 0xffffu; }
};

// One warp per block.  A warp takes runs of RUN consecutive tasks (A slots each, one
// replica at a time), strided by the grid: the warps together move through the system, so
// that the forces they hand over go to a few MB of it.  A lane goes through its atoms of them at its own pace -- it queues and
// evaluates the entries of one atom and goes on to the next without waiting for the warp,
// whose lanes have 27 +- 3 pairs per atom to evaluate: one atom after the other in step,
// every atom would take the 33 of the longest lane.  The partial sums go to memory as they
// are (k_close64 adds them), so that the change of atom, which lanes make at different
// times, has no FP64 instructions.
// EV: also virial and potential energy, each pair counted for both orders at the atom
// that claimed it.
template <int TPA, bool EV, bool ONE>
__global__ void __launch_bounds__(32, MINB) k_pairs64(Dev d, Box b, StepConsts sc, int RUN) {
  using Split = RowSplit<TPA>;
  constexpr int A = 32 / TPA, PER = Split::PER, NV = EV ? 5 : 3;
  __shared__ TabX<ONE ? 1 : MAXT * MAXT> tab;
  __shared__ PairWarp<NV> W;
  if (halted(d)) return;
  const PairTab &T = *d.tab;
  const int nt = T.nt, lane = threadIdx.x;
  for (int k = lane; k < nt * nt; k += 32) {
    tab.rc2[k] = T.rc2[k]; tab.w12[k] = T.w12[k]; tab.w6[k] = T.w6[k]; tab.gc[k] = T.gc[k];
    if (EV) tab.l12[k] = T.l12[k], tab.l6[k] = T.l6[k], tab.uc[k] = T.uc[k];
    tab.screen[k] = T.screen[k];
  }
  const int a = lane % A, t = lane / A, e0 = Split::first_entry(t);
  const int n = sc.n, cap_h = d.cap_h, ntask = (n + A - 1) / A;
  const bool jump = sc.jump_tol > 0.0;
  double ev_p[2] = {0.0, 0.0};
  int run = blockIdx.x, task0 = run * RUN;

  while (task0 < ntask) {
    const int task_end = min(ntask, (run + 1) * RUN);
    if (task0 >= task_end) {
      run += gridDim.x;
      task0 = run * RUN;
      continue;
    }
    // the tasks of one replica in [task0, task_end)
    const int rep = rep_of_slot(b, task0 * A);
    if (rep < 0) {  // padding slots
      ++task0;
      continue;
    }
    const RepBox &rb = repbox(b, rep);
    const int slot_end = rb.slot_off + rb.natoms, run_end = min(task_end, (slot_end + A - 1) / A);
    __syncwarp();
    if (lane < 27) {
      const int sx = lane % 3 - 1, sy = (lane / 3) % 3 - 1, sz = lane / 9 - 1;
      W.img[lane] = make_double3(sx * rb.L[0], sy * rb.L[1], sz * rb.L[2]);
    }
    const float ux = rb.uh[0], uy = rb.uh[1], uz = rb.uh[2];
    __syncwarp();

    // the lane's atom: slot, position, coordinates, claimed entries and where they are
    int i = -1, task = task0 - 1, nh = 0, g = 0, head = 0, cnt = 0, t1 = 0;
    dbl4 xi = make_dbl4(0.0, 0.0, 0.0, 0.0);
    int4 ci = make_int4(0, 0, 0, 0);
    size_t row = 0;
    bool more = false, cur = false, atoms = true;  // entries left to screen; one being evaluated; atoms left
    uint2 w_cur = make_uint2(0u, 0u);
    dbl4 x_cur = xi;
    ChunkWords<PER> next = {};
    for (;;) {
      // a lane that has nothing to evaluate goes on to its next atom and screens its entries
      while (__any_sync(FULL_MASK, cnt == 0 && (more || (atoms && !cur)))) {
        if (cnt == 0 && !more && atoms && !cur) {
          if (i >= 0) {  // the sums of the atom it is done with
#pragma unroll
            for (int c = 0; c < PER; ++c)
              d.own[4 * (size_t)i + e0 + c] =
                  make_dbl4(W.sum[e0 + c][0][lane], W.sum[e0 + c][1][lane], W.sum[e0 + c][2][lane], 0.0);
            if (EV) {
              double e[2];  // both orders of the pairs
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                e[q] = W.sum[e0][3 + q][lane];
                if (PER > 1) e[q] += W.sum[(e0 + 1) & 3][3 + q][lane];
                if (PER > 2) e[q] += W.sum[(e0 + 2) & 3][3 + q][lane] + W.sum[(e0 + 3) & 3][3 + q][lane];
                e[q] *= 2.0;
              }
              const double vir = e[0], pe = e[1];
              ev_p[0] += vir;
              ev_p[1] += pe;
              if (d.ev_part) d.ev_part[(size_t)i * TPA + t] = make_double2(vir, pe);
            }
          }
          ++task;
          i = task * A + a;
          atoms = task < run_end && i < slot_end;
          if (atoms) {
            nh = d.nh[i];
            xi = d.pos[i];
            ci = d.ic[i];
            t1 = ci.w * nt;
            row = (size_t)task * cap_h * A + 4 * a + e0;
            g = Split::first_chunk(t);
            more = 4 * g + e0 < nh;
            if (more) next.load(d, row + (size_t)g * (4 * A));
#pragma unroll
            for (int c = 0; c < PER; ++c)
#pragma unroll
              for (int q = 0; q < NV; ++q) W.sum[e0 + c][q][lane] = 0.0;
          }
        }
        if (more && cnt <= RING - PER) {
          const ChunkWords<PER> now = next;
          int4 cj[PER];
#pragma unroll
          for (int u = 0; u < PER; ++u)
            if (4 * g + e0 + u < nh) cj[u] = __ldg(&d.ic[now.word(u) & IDX_MASK]);
          const int g_now = g;
          g += Split::STRIDE;
          more = 4 * g + e0 < nh;
          if (more) next.load(d, row + (size_t)g * (4 * A));  // in flight with the gathers
#pragma unroll
          for (int u = 0; u < PER; ++u) {
            if (4 * g_now + e0 + u >= nh) break;
            const float dx = (float)fixed_diff(cj[u].x, ci.x) * ux, dy = (float)fixed_diff(cj[u].y, ci.y) * uy,
                        dz = (float)fixed_diff(cj[u].z, ci.z) * uz;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 <= tab.screen[ONE ? t1 : t1 + cj[u].w]) {
              W.ring[(head + cnt) & (RING - 1)][lane] = make_uint2(now.word(u), now.slot(u) | (uint32_t)(e0 + u) << 16);
              ++cnt;
            } else {
              d.recv[recv_index((int)(now.word(u) & IDX_MASK), (int)now.slot(u), cap_h)] = make_dbl4(0.0, 0.0, 0.0, 0.0);
            }
          }
        }
      }
      // take the next entry and start on its position before the current one is evaluated
      const bool nxt = cnt > 0;
      if (!__any_sync(FULL_MASK, cur || nxt)) break;
      uint2 w_nxt = w_cur;
      dbl4 x_nxt = x_cur;
      if (nxt) {
        w_nxt = W.ring[head][lane];
        head = (head + 1) & (RING - 1);
        --cnt;
        x_nxt = ldg_dbl4(&d.pos[w_nxt.x & IDX_MASK]);
      }
      // image x_j + s L (the reference's ghost coordinate); s = 0 for most entries, where
      // x_j + 0 is x_j exactly and the three adds are skipped
      if (cur && (w_cur.x >> CODE_SHIFT) != CODE_ZERO) {
        const double3 s = W.img[w_cur.x >> CODE_SHIFT];
        x_cur.x += s.x; x_cur.y += s.y; x_cur.z += s.z;
      }
      __syncwarp();
      if (cur) {
        const int c = (int)(w_cur.y >> 16);
        const double dx = x_cur.x - xi.x, dy = x_cur.y - xi.y, dz = x_cur.z - xi.z;
        const double r2d = dx * dx + dy * dy + dz * dz;
        const int tt = ONE ? t1 : t1 + type_of(x_cur.w);
        dbl4 f = make_dbl4(0.0, 0.0, 0.0, 0.0);
        // the cutoff test compares bit patterns as integers (the same order for doubles
        // >= +0; rc^2 < 0, an eps == 0 pair, admits none)
        if (__double_as_longlong(r2d) <= __double_as_longlong(tab.rc2[tt])) {
          // Lj jump_fix (src/force/lj.cpp:459-468): r^2 floored after the cutoff test
          double r2 = r2d;
          if (jump) r2 = r2d < sc.jump_tol ? sc.jump_tol : r2d;
          const double u = rcp_cubic(r2), u3 = u * u * u;
          const double coef = fma(fma(tab.w12[tt], u3, tab.w6[tt]) * u3, u, -tab.gc[tt]);
          const double px = W.sum[c][0][lane], py = W.sum[c][1][lane], pz = W.sum[c][2][lane];
          W.sum[c][0][lane] = fma(coef, dx, px); W.sum[c][1][lane] = fma(coef, dy, py); W.sum[c][2][lane] = fma(coef, dz, pz);
          f.x = -coef * dx; f.y = -coef * dy; f.z = -coef * dz;
          if (EV) {
            W.sum[c][3][lane] -= coef * r2;
            W.sum[c][4][lane] += fma(tab.l12[tt], u3, -tab.l6[tt]) * u3 - tab.uc[tt] - 0.5 * tab.gc[tt] * (r2 - tab.rc2[tt]);
          }
        }
        d.recv[recv_index((int)(w_cur.x & IDX_MASK), (int)(w_cur.y & 0xffffu), cap_h)] = f;
      }
      __syncwarp();
      cur = nxt;
      w_cur = w_nxt;
      x_cur = x_nxt;
    }
    task0 = run_end;
  }
  if (EV) block_sum_store_f<2>(ev_p, &d.partials_ev[(size_t)blockIdx.x * 2]);
}

// Received forces, closing update, the end of the step.
template <int TPA, int KICK, bool EV>
__global__ void __launch_bounds__(CLOSE_THREADS) k_close64(Dev d, Box b, StepConsts sc, ForceArgs fa) {
  using Split = RowSplit<TPA>;
  constexpr int A = 32 / TPA, PER = Split::PER;
  __shared__ double s_minv[MAXT], s_mass[MAXT];
  __shared__ int s_halt;
  if (threadIdx.x == 0) s_halt = halted(d);
  if (threadIdx.x < MAXT) {
    s_minv[threadIdx.x] = d.tab->minv[threadIdx.x];
    s_mass[threadIdx.x] = d.tab->mass[threadIdx.x];
  }
  __syncthreads();
  const bool was_halted = s_halt != 0;  // a step after a halt does nothing
  struct {
    const double *minv, *mass;
  } const tab{s_minv, s_mass};
  const int lane = threadIdx.x & 31, a = lane % A, t = lane / A;
  const int n = sc.n, cap_h = d.cap_h, e0 = Split::first_entry(t);
  const int warps_total = (gridDim.x * blockDim.x) >> 5, ntask = was_halted ? 0 : (n + A - 1) / A;
  long long step = 0;
  if (KICK == 2) step = *d.step_base + fa.k_in_chunk;
  double ke_p[4] = {0.0, 0.0, 0.0, 0.0};
  for (int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < ntask; task += warps_total) {
    const int i = task * A + a;
    const int rep = i < n ? rep_of_slot(b, i) : -1;
    const bool act = rep >= 0;
    const int nr = act ? d.nr[i] : 0;
    double P[PER][3];
#pragma unroll
    for (int u = 0; u < PER; ++u) P[u][0] = P[u][1] = P[u][2] = 0.0;
    const dbl4 *const in = d.recv + recv_index(act ? i : 0, e0, cap_h);
#pragma unroll 2
    for (int g = Split::first_chunk(t); 4 * g + e0 < nr; g += Split::STRIDE) {
      dbl4 f[PER];
#pragma unroll
      for (int u = 0; u < PER; ++u)
        f[u] = 4 * g + e0 + u < nr ? ldg_dbl4(in + (size_t)(4 * g + u) * 32) : make_dbl4(0.0, 0.0, 0.0, 0.0);
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        P[u][0] += f[u].x; P[u][1] += f[u].y; P[u][2] += f[u].z;
      }
    }
    dbl4 own[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) own[u] = act ? d.own[4 * (size_t)i + e0 + u] : make_dbl4(0.0, 0.0, 0.0, 0.0);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      P[u][0] += own[u].x; P[u][1] += own[u].y; P[u][2] += own[u].z;
    }
    double F[3], none = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      F[q] = PER == 4   ? (P[0][q] + P[1 % PER][q]) + (P[2 % PER][q] + P[3 % PER][q])
             : PER == 2 ? P[0][q] + P[1 % PER][q]
                        : P[0][q];
    fold_lanes<A, false>(F[0], F[1], F[2], none, none);
    if (act && t == 0) {
      finish_atom<false, KICK, EV>(d, b, sc, tab, i, d.type[i], rep, step, fa.fuse, F[0], F[1], F[2], ke_p);
      if (EV && d.ev_part) {
        double2 e[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) e[q] = q < TPA ? d.ev_part[(size_t)i * TPA + q] : make_double2(0.0, 0.0);
        d.ev_atom[i] = make_double2((e[0].x + e[1].x) + (e[2].x + e[3].x), (e[0].y + e[1].y) + (e[2].y + e[3].y));
      }
    }
  }
  if (EV && !was_halted)
    block_sum_store_f<4>(ke_p, &(KICK == 2 ? d.partials_ke_end : d.partials_ke)[(size_t)blockIdx.x * 4]);
  if (KICK != 0) end_of_step<EV>(d, was_halted, fa);
}

// ---------------------------------------------------------------------------
// after a list build: the claimed entries of every atom and their receiving slots
// ---------------------------------------------------------------------------
__device__ inline bool exchange_on(const Dev &d, const Box &b, int rep, int forced) {
  return rep >= 0 && !halted(d) && (forced || b.rep_flag[rep] != 0);
}

// Thread per atom: copies the entries it claims out of its row, takes a receiving slot of
// the other atom for each and leaves {its slot, the entry} there.  A row that outgrows the
// space counts as an overflow of the list (which doubles as the room for it).
__global__ void __launch_bounds__(256) k_claim(Dev d, Box b, int forced) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.nslot || !exchange_on(d, b, rep_of_slot(b, i), forced)) return;
  const int as = 5 - log2_pow2(d.tpa);
  const uint4 *row = reinterpret_cast<const uint4 *>(d.nbr + nbr_block_base(i, d.cap, d.tpa));
  uint4 *const out = reinterpret_cast<uint4 *>(d.hw + nbr_block_base(i, d.cap_h, d.tpa));
  uint4 buf = make_uint4(0u, 0u, 0u, 0u);
  uint2 *const note = reinterpret_cast<uint2 *>(d.recv);
  const int nn = d.nnbr[i];
  int k = 0;
  for (int g = 0; 4 * g < nn; ++g) {
    const uint4 w4 = __ldg(row + ((size_t)g << as));
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
    bool mine[4];
    int p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) mine[u] = 4 * g + u < nn && claims(i, (int)(w[u] & IDX_MASK));
#pragma unroll
    for (int u = 0; u < 4; ++u)  // the four in flight together
      if (mine[u]) p[u] = atomicAdd(&d.nr[w[u] & IDX_MASK], 1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (!mine[u]) continue;
      const size_t j = w[u] & IDX_MASK;
      // claimed words go out four at a time (a partial chunk at the end)
      buf.x = (k & 3) == 0 ? w[u] : buf.x;
      buf.y = (k & 3) == 1 ? w[u] : buf.y;
      buf.z = (k & 3) == 2 ? w[u] : buf.z;
      buf.w = w[u];
      if ((k & 3) == 3 && k < d.cap_h) out[(size_t)(k >> 2) << as] = buf;
      if (p[u] < d.cap_h) note[j * d.cap_h + p[u]] = make_uint2((uint32_t)i, (uint32_t)k);
      ++k;
      if (p[u] >= d.cap_h) atomicMax(&d.flags[F_OVERFLOW], 2 * (p[u] + 1));
    }
  }
  if ((k & 3) != 0 && k < d.cap_h) out[(size_t)(k >> 2) << as] = buf;
  if (k > d.cap_h) atomicMax(&d.flags[F_OVERFLOW], 2 * k);
  d.nh[i] = min(k, d.cap_h);
}

// Warp per receiving atom: its notes in the order of the claiming slots; the rank is the
// receiving slot, so that sums do not depend on the order of the atomics.
__global__ void __launch_bounds__(256) k_rank(Dev d, Box b, int forced) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (j >= b.nslot || !exchange_on(d, b, rep_of_slot(b, j), forced)) return;
  const int n = min(d.nr[j], d.cap_h);
  const uint2 *const note = reinterpret_cast<const uint2 *>(d.recv) + (size_t)j * d.cap_h;
  for (int p0 = 0; p0 < n; p0 += 64) {  // two notes per lane
    const int pa = p0 + lane, pb = pa + 32;
    const uint2 none = make_uint2(0xffffffffu, 0xffffffffu), ma = pa < n ? note[pa] : none, mb = pb < n ? note[pb] : none;
    int ra = 0, rb = 0;
    for (int q0 = 0; q0 < n; q0 += 32) {
      const uint32_t other = q0 == p0 ? ma.x : q0 == p0 + 32 ? mb.x : (q0 + lane < n ? note[q0 + lane].x : 0xffffffffu);
      const int m = min(32, n - q0);
      if (n <= 32) {  // (one note per lane)
        for (int q = 0; q < m; q += 4)
#pragma unroll
          for (int v = 0; v < 4; ++v) ra += __shfl_sync(FULL_MASK, other, q + v) < ma.x;  // beyond n: never less
      } else {
        for (int q = 0; q < m; q += 4)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint32_t x = __shfl_sync(FULL_MASK, other, q + v);
            ra += x < ma.x;
            rb += x < mb.x;
          }
      }
    }
    if (ma.y < (uint32_t)d.cap_h) d.hslot[nbr_index((int)ma.x, (int)ma.y, d.cap_h, d.tpa)] = (uint16_t)ra;
    if (mb.y < (uint32_t)d.cap_h) d.hslot[nbr_index((int)mb.x, (int)mb.y, d.cap_h, d.tpa)] = (uint16_t)rb;
  }
  if (lane == 0) d.nr[j] = n;
}

int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
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
  pairs<TPA>(ev, one, grid_ev, run, d, b, sc, st);
  if (kick == 0) close_kick<TPA, 0>(ev, grid, d, b, sc, fa, st);
  else if (kick == 1) close_kick<TPA, 1>(ev, grid, d, b, sc, fa, st);
  else close_kick<TPA, 2>(ev, grid, d, b, sc, fa, st);
}

}  // namespace

// k_pairs64: one wave of resident warps.  Runs of four tasks (its lanes then evaluate 691
// instead of 731 FP64 instructions per task) once every warp has eight tasks; below that
// the longer runs leave too few warps in flight.  131,072 atoms: 283 us with runs of one,
// 293 with runs of four; 1,048,576 atoms: 1931 and 1867 (both kernels together).
int exchange_pair_blocks(int ntask, int sms) {
  const int run = exchange_run(ntask);
  return std::max(1, std::min((ntask + run - 1) / run, sms * MINB));
}
int exchange_close_threads() { return CLOSE_THREADS; }

int launch_exchange_build(const Dev &d, const Box &b, int forced, cudaStream_t st) {
  k_claim<<<(b.nslot + 255) / 256, 256, 0, st>>>(d, b, forced);
  k_rank<<<(int)(((long long)b.nslot * 32 + 255) / 256), 256, 0, st>>>(d, b, forced);
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
