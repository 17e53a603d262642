// cav_exchange.cuh -- device parts of the FP64 pair exchange (described in
// cav_exchange.cu, whose kernels run one each; the step kernel of cav_chunk.cu runs all).
#pragma once

#include "cav_pair.cuh"

namespace cav {

constexpr int MINB = 20;        // resident warps per SM (one per block)
constexpr int RING = 16;        // queued entries per lane
// a warp per atom (pair_atom) up to this many atoms; step of 500, 1,372, 4,000 and 8,788 atoms in
// the step kernel 24, 28, 39 and 59 us, with four lanes per atom 39, 39, 44 and 53
constexpr int BY_ATOM = 6144;

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
  template <bool COH>
  __device__ __forceinline__ void load(const Dev &d, size_t at) {
    if constexpr (PER == 4) {
      const uint4 v = ld_ro<COH>(reinterpret_cast<const uint4 *>(d.hw + at));
      const uint2 x = ld_ro<COH>(reinterpret_cast<const uint2 *>(d.hslot + at));
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
      s[0] = x.x; s[1] = x.y;
    } else if constexpr (PER == 2) {
      const uint2 v = ld_ro<COH>(reinterpret_cast<const uint2 *>(d.hw + at));
      w[0] = v.x; w[1] = v.y;
      s[0] = ld_ro<COH>(reinterpret_cast<const uint32_t *>(d.hslot + at));
    } else {
      w[0] = ld_ro<COH>(d.hw + at);
      s[0] = ld_ro<COH>(d.hslot + at);
    }
  }
  __device__ __forceinline__ uint32_t word(int u) const { return w[u]; }
  __device__ __forceinline__ uint32_t slot(int u) const { return PER == 1 ? s[0] : (s[u >> 1] >> (16 * (u & 1))) & 0xffffu; }
};

// The tasks [task0, run_end) (A slots each; all of one replica, none of padding alone) by
// one warp: a lane goes through its atoms of them at its own pace -- it queues and evaluates
// the entries of one atom and goes on to the next without waiting for the warp, whose lanes
// have 27 +- 3 pairs per atom to evaluate: one atom after the other in step, every atom would
// take the 33 of the longest lane.  The partial sums go to memory as they are (close_sum adds
// them), so that the change of atom, which lanes make at different times, has no FP64
// instructions.  EV: also virial and potential energy, each pair counted for both orders at
// the atom that claimed it.  Returns the first task not done (a replica ends early).
template <int TPA, bool EV, bool ONE, bool COH>
__device__ __forceinline__ int pair_tasks(const Dev &d, const Box &b, const StepConsts &sc,
                                          const TabX<ONE ? 1 : MAXT * MAXT> &tab, PairWarp<EV ? 5 : 3> &W, int nt,
                                          int rep, int task0, int task_end, double (&ev_p)[2]) {
  using Split = RowSplit<TPA>;
  constexpr int A = 32 / TPA, PER = Split::PER, NV = EV ? 5 : 3;
  const int lane = threadIdx.x & 31, a = lane % A, t = lane / A, e0 = Split::first_entry(t), cap_h = d.cap_h;
  const bool jump = sc.jump_tol > 0.0;
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
          if (more) next.template load<COH>(d, row + (size_t)g * (4 * A));
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
          if (4 * g + e0 + u < nh) cj[u] = ld_ro<COH>(&d.ic[now.word(u) & IDX_MASK]);
        const int g_now = g;
        g += Split::STRIDE;
        more = 4 * g + e0 < nh;
        if (more) next.template load<COH>(d, row + (size_t)g * (4 * A));  // in flight with the gathers
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
      x_nxt = ld_dbl4<COH>(&d.pos[w_nxt.x & IDX_MASK]);
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
      // (roundings spelled out: every kernel that holds this loop gives the same bits)
      const double r2d = fma(dz, dz, fma(dy, dy, __dmul_rn(dx, dx)));
      const int tt = ONE ? t1 : t1 + type_of(x_cur.w);
      dbl4 f = make_dbl4(0.0, 0.0, 0.0, 0.0);
      // the cutoff test compares bit patterns as integers (the same order for doubles
      // >= +0; rc^2 < 0, an eps == 0 pair, admits none)
      if (__double_as_longlong(r2d) <= __double_as_longlong(tab.rc2[tt])) {
        // Lj jump_fix (src/force/lj.cpp:459-468): r^2 floored after the cutoff test
        double r2 = r2d;
        if (jump) r2 = r2d < sc.jump_tol ? sc.jump_tol : r2d;
        const double u = rcp_cubic(r2), u3 = __dmul_rn(__dmul_rn(u, u), u);
        const double coef = fma(__dmul_rn(fma(tab.w12[tt], u3, tab.w6[tt]), u3), u, -tab.gc[tt]);
        f.x = __dmul_rn(-coef, dx); f.y = __dmul_rn(-coef, dy); f.z = __dmul_rn(-coef, dz);
        const double px = W.sum[c][0][lane], py = W.sum[c][1][lane], pz = W.sum[c][2][lane];
        W.sum[c][0][lane] = __dsub_rn(px, f.x); W.sum[c][1][lane] = __dsub_rn(py, f.y); W.sum[c][2][lane] = __dsub_rn(pz, f.z);
        if (EV) {
          W.sum[c][3][lane] = fma(-coef, r2, W.sum[c][3][lane]);
          const double pe = fma(fma(tab.l12[tt], u3, -tab.l6[tt]), u3, -tab.uc[tt]);
          W.sum[c][4][lane] += fma(__dmul_rn(-0.5, tab.gc[tt]), __dsub_rn(r2, tab.rc2[tt]), pe);
        }
      }
      d.recv[recv_index((int)(w_cur.x & IDX_MASK), (int)(w_cur.y & 0xffffu), cap_h)] = f;
    }
    __syncwarp();
    cur = nxt;
    w_cur = w_nxt;
    x_cur = x_nxt;
  }
  return run_end;
}

// The claimed pairs of one atom by a whole warp, an entry per lane: for systems with fewer
// atoms than the GPU has FP64 units to keep busy.  A warp's FP64 instructions take 64 cycles
// each, one after the other (measured: three independent chains as long as one three
// times), so that time goes with the pairs of the longest lane, not with their sum.  The
// forces meet in shared memory, where 12 lanes add the 4 partial sums' components in row
// order: the sums of pair_tasks bit for bit.
template <bool ONE>
__device__ __forceinline__ void pair_atom(const Dev &d, const Box &b, const StepConsts &sc,
                                          const TabX<ONE ? 1 : MAXT * MAXT> &tab, double (*share)[3], int nt, int i) {
  const int rep = rep_of_slot(b, i);
  if (rep < 0) return;  // padding slot
  const RepBox &rb = repbox(b, rep);
  const int lane = threadIdx.x & 31, cs = 7 - log2_pow2(d.tpa), nh = d.nh[i], cap_h = d.cap_h;
  const dbl4 xi = d.pos[i];
  const size_t row = nbr_block_base(i, cap_h, d.tpa);
  const int t1 = type_of(xi.w) * nt;
  double acc = 0.0;  // lane 3 c + q: component q of partial sum c
  for (int e0 = 0; e0 < nh; e0 += 32) {
    const int e = e0 + lane;
    dbl4 f = make_dbl4(0.0, 0.0, 0.0, 0.0);
    if (e < nh) {
      const size_t at = row + ((size_t)(e >> 2) << cs) + (e & 3);
      const uint32_t w = d.hw[at], slot = d.hslot[at];
      const int j = (int)(w & IDX_MASK), code = (int)(w >> CODE_SHIFT);
      dbl4 xj = ld_dbl4<true>(&d.pos[j]);
      if (code != CODE_ZERO) {
        xj.x += (code % 3 - 1) * rb.L[0];
        xj.y += ((code / 3) % 3 - 1) * rb.L[1];
        xj.z += (code / 9 - 1) * rb.L[2];
      }
      const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
      const double r2d = fma(dz, dz, fma(dy, dy, __dmul_rn(dx, dx)));
      const int tt = ONE ? t1 : t1 + type_of(xj.w);
      if (__double_as_longlong(r2d) <= __double_as_longlong(tab.rc2[tt])) {
        double r2 = r2d;
        if (sc.jump_tol > 0.0) r2 = r2d < sc.jump_tol ? sc.jump_tol : r2d;
        const double u = rcp_cubic(r2), u3 = __dmul_rn(__dmul_rn(u, u), u);
        const double coef = fma(__dmul_rn(fma(tab.w12[tt], u3, tab.w6[tt]), u3), u, -tab.gc[tt]);
        f.x = __dmul_rn(-coef, dx); f.y = __dmul_rn(-coef, dy); f.z = __dmul_rn(-coef, dz);
      }
      d.recv[recv_index(j, (int)slot, cap_h)] = f;
    }
    __syncwarp();
    share[lane][0] = f.x; share[lane][1] = f.y; share[lane][2] = f.z;
    __syncwarp();
    if (lane < 12) {
      const int c = lane / 3, q = lane - 3 * c, n = min(32, nh - e0);
      for (int m = c; m < n; m += 4) acc = __dsub_rn(acc, share[m][q]);
    }
  }
  if (lane < 12) reinterpret_cast<double *>(d.own)[(4 * (size_t)i + lane / 3) * 4 + lane % 3] = acc;
}

// the pair constants a warp or block needs in shared memory (synchronise afterwards)
template <bool EV, bool ONE>
__device__ __forceinline__ void load_tabx(const Dev &d, TabX<ONE ? 1 : MAXT * MAXT> &tab) {
  const PairTab &T = *d.tab;
  for (int k = threadIdx.x; k < T.nt * T.nt; k += blockDim.x) {
    tab.rc2[k] = T.rc2[k]; tab.w12[k] = T.w12[k]; tab.w6[k] = T.w6[k]; tab.gc[k] = T.gc[k];
    if (EV) tab.l12[k] = T.l12[k], tab.l6[k] = T.l6[k], tab.uc[k] = T.uc[k];
    tab.screen[k] = T.screen[k];
  }
}

// The force on atom i (any lane of the warp; act: it has an atom): what it received and its
// own partial sums, in the order of RowSplit.
template <int TPA, bool COH>
__device__ __forceinline__ void close_sum(const Dev &d, bool act, int i, int t, double (&F)[3]) {
  using Split = RowSplit<TPA>;
  constexpr int A = 32 / TPA, PER = Split::PER;
  const int cap_h = d.cap_h, e0 = Split::first_entry(t), nr = act ? d.nr[i] : 0;
  double P[PER][3];
#pragma unroll
  for (int u = 0; u < PER; ++u) P[u][0] = P[u][1] = P[u][2] = 0.0;
  const dbl4 *const in = d.recv + recv_index(act ? i : 0, e0, cap_h);
#pragma unroll 2
  for (int g = Split::first_chunk(t); 4 * g + e0 < nr; g += Split::STRIDE) {
    dbl4 f[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u)
      f[u] = 4 * g + e0 + u < nr ? ld_dbl4<COH>(in + (size_t)(4 * g + u) * 32) : make_dbl4(0.0, 0.0, 0.0, 0.0);
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
  double none = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q)
    F[q] = PER == 4   ? (P[0][q] + P[1 % PER][q]) + (P[2 % PER][q] + P[3 % PER][q])
           : PER == 2 ? P[0][q] + P[1 % PER][q]
                      : P[0][q];
  fold_lanes<A, false>(F[0], F[1], F[2], none, none);
}

// batches: virial and potential energy of atom i from its lanes
template <int TPA>
__device__ __forceinline__ void close_ev(const Dev &d, int i) {
  double2 e[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) e[q] = q < TPA ? d.ev_part[(size_t)i * TPA + q] : make_double2(0.0, 0.0);
  d.ev_atom[i] = make_double2((e[0].x + e[1].x) + (e[2].x + e[3].x), (e[0].y + e[1].y) + (e[2].y + e[3].y));
}

// ---------------------------------------------------------------------------
// after a list build: the claimed entries of every atom and their receiving slots
// ---------------------------------------------------------------------------
// Warp per atom: copies the entries it claims out of its row, takes a receiving slot of the
// other atom for each and leaves {its slot, the entry} there.  A row that outgrows the
// space counts as an overflow of the list (which doubles as the room for it).
__device__ __forceinline__ void claim_slot(const Dev &d, const Box &b, int forced, int i) {
  const int lane = threadIdx.x & 31;
  const int rep = rep_of_slot(b, i);
  if (rep < 0 || !rebuild_on(d, b, rep, forced)) return;
  const int cs = 7 - log2_pow2(d.tpa);  // chunk stride 4A words = 2^(log2 A + 2)
  const uint32_t *const row = d.nbr + nbr_block_base(i, d.cap, d.tpa);
  uint32_t *const out = d.hw + nbr_block_base(i, d.cap_h, d.tpa);
  uint2 *const note = reinterpret_cast<uint2 *>(d.recv);
  const int nn = d.nnbr[i];
  int claimed = 0;
  for (int e0 = 0; e0 < nn; e0 += 32) {
    const int e = e0 + lane;
    const uint32_t w = e < nn ? row[((size_t)(e >> 2) << cs) + (e & 3)] : 0u;
    const int j = (int)(w & IDX_MASK);
    const bool mine = e < nn && claims(i, j);
    const unsigned m = __ballot_sync(FULL_MASK, mine);
    if (mine) {
      const int k = claimed + __popc(m & ((1u << lane) - 1u)), p = atomicAdd(&d.nr[j], 1);
      if (k < d.cap_h) out[((size_t)(k >> 2) << cs) + (k & 3)] = w;
      if (p < d.cap_h) note[(size_t)j * d.cap_h + p] = make_uint2((uint32_t)i, (uint32_t)k);
      else atomicMax(&d.flags[F_OVERFLOW], 2 * (p + 1));
    }
    claimed += __popc(m);
  }
  if (lane == 0) {
    if (claimed > d.cap_h) atomicMax(&d.flags[F_OVERFLOW], 2 * claimed);
    d.nh[i] = min(claimed, d.cap_h);
  }
}

// Warp per receiving atom: its notes in the order of the claiming slots; the rank is the
// receiving slot, so that sums do not depend on the order of the atomics.
__device__ __forceinline__ void rank_slot(const Dev &d, const Box &b, int forced, int j) {
  const int lane = threadIdx.x & 31;
  const int rep = rep_of_slot(b, j);
  if (rep < 0 || !rebuild_on(d, b, rep, forced)) return;
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

}  // namespace cav
