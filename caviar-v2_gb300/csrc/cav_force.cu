// cav_force.cu -- the shifted-force LJ pair kernels (force_field::Lj::calculate_acceleration,
// src/force/lj.cpp:393-517), fused with the closing integrator update of the step.
//
// Full neighbour list, gather only (no atomics, deterministic): TPA lanes work on one
// atom, a warp on A = 32/TPA atoms, and the list layout (nbr_index) makes every
// iteration one coalesced 128-byte read of neighbour words.  Two precisions:
//   FP64  : image = x_j + s*L, all pair arithmetic in double;
//   MIXED : FP32 pair arithmetic on exact differences of fixed-point coordinates
//           (int4 x,y,z,type; to_fixed) and FP32 sums per lane, FP64 accumulation across
//           lanes, FP64 acceleration/velocity/reductions.
#include <algorithm>

#include "cav_mixed.cuh"

namespace cav {

// per warp: the 27 image shifts s*L (FP64) or the fixed-point units (mixed) of the
// replica the warp's current atoms belong to (a warp never straddles two)
template <bool MIXED>
struct WarpImages;
template <>
struct WarpImages<true> {
  float4 hi, lo;  // length of a coordinate unit per axis, as an FP32 pair hi + lo
  uint3 flip;     // IMG: what an image shift does to a coordinate
};

template <>
struct WarpImages<false> {
  double3 v[27];
};

// the coordinates of the image that a list word names (lists of image codes)
__device__ __forceinline__ int4 image_of(int4 q, uint32_t word, const uint3 &flip) {
  const int code = (int)(word >> CODE_SHIFT), sz = code / 9, sy = code / 3 - 3 * sz, sx = code % 3;
  if (sx != 1) q.x ^= (int)flip.x;
  if (sy != 1) q.y ^= (int)flip.y;
  if (sz != 1) q.z ^= (int)flip.z;
  return q;
}

// FP64 pair loop of one lane (the entries RowSplit gives it).  ONE: single type, the pair
// constants in registers, no table lookups; t1 = the atom's first table entry.  The
// cutoff test r^2 <= rc^2 compares the bit patterns as integers (the same order for
// doubles >= +0, and rc^2 < 0, an eps == 0 pair, admits none), off the FP64 pipe.
template <int TPA, bool EV, bool ONE>
__device__ __forceinline__ void fp64_pairs(const Dev &d, const uint4 *row4, int nn, int t, const dbl4 &xi, int t1,
                                           const SmemTabD &tab, const double3 *img, double jump_tol, double (&F)[5]) {
  using Split = RowSplit<TPA>;
  constexpr int A = 32 / TPA, NV = EV ? 5 : 3, PER = Split::PER;
  const bool jump = jump_tol > 0.0;
  const long long rc2b1 = __double_as_longlong(tab.rc2[t1]);
  const double sig21 = tab.sig2[t1], e61 = tab.e6[t1], e121 = tab.e12[t1], gc1 = tab.gc[t1];
  const int e0 = Split::first_entry(t);
  double P[PER][5];
#pragma unroll
  for (int u = 0; u < PER; ++u)
#pragma unroll
    for (int q = 0; q < 5; ++q) P[u][q] = 0.0;
  const uint32_t *row = reinterpret_cast<const uint32_t *>(row4) + e0;
  for (int g = Split::first_chunk(t); 4 * g + e0 < nn; g += Split::STRIDE) {
    uint32_t e[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) e[u] = __ldg(row + (size_t)g * (4 * A) + u);
    const int k0 = 4 * g + e0;
    dbl4 xj[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u)
      if (k0 + u < nn) xj[u] = ldg_dbl4(&d.pos[e[u] & IDX_MASK]);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (k0 + u >= nn) break;
      // image x_j + s L (the reference's ghost coordinate); s = 0 for most
      // entries, where x_j + 0 is x_j exactly and the three adds are skipped
      const int code = (int)(e[u] >> CODE_SHIFT);
      double jx = xj[u].x, jy = xj[u].y, jz = xj[u].z;
      if (code != CODE_ZERO) {
        const double3 s = img[code];
        jx += s.x; jy += s.y; jz += s.z;
      }
      const double dx = jx - xi.x, dy = jy - xi.y, dz = jz - xi.z;
      const double r2d = dx * dx + dy * dy + dz * dz;
      const int tt = ONE ? t1 : t1 + type_of(xj[u].w);
      const long long rc2b = ONE ? rc2b1 : __double_as_longlong(tab.rc2[tt]);
      if (__double_as_longlong(r2d) <= rc2b) {
        // Lj jump_fix (src/force/lj.cpp:459-468): r^2 floored at jump_tol after the
        // cutoff test (jump_tol = 0 when off); the direction stays dx, dy, dz
        double r2 = r2d;
        if (jump) r2 = r2d < jump_tol ? jump_tol : r2d;
        const double r2i = rcp_nr(r2);
        const double s2 = (ONE ? sig21 : tab.sig2[tt]) * r2i;
        const double s6 = s2 * s2 * s2;
        // eps4 s6 (6 - 12 s6) / r^2 - g(rc) as (s6 (e6 - e12 s6)) r2i - gc
        const double coef = ONE ? fma(s6 * fma(-e121, s6, e61), r2i, -gc1)
                                : fma(s6 * fma(-tab.e12[tt], s6, tab.e6[tt]), r2i, -tab.gc[tt]);
        P[u][0] = fma(coef, dx, P[u][0]); P[u][1] = fma(coef, dy, P[u][1]); P[u][2] = fma(coef, dz, P[u][2]);
        if (EV) {
          P[u][3] -= coef * r2;
          P[u][4] += tab.eps4[tt] * (s6 * s6 - s6) - tab.uc[tt] - 0.5 * tab.gc[tt] * (r2 - tab.rc2[tt]);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NV; ++q)
    F[q] = PER == 4   ? (P[0][q] + P[1 % PER][q]) + (P[2 % PER][q] + P[3 % PER][q])
           : PER == 2 ? P[0][q] + P[1 % PER][q]
                      : P[0][q];
}

// Grid-strided pair kernel over the full list (the mixed form when it has no segments; the FP64
// form with 8 or 16 lanes or without room for the pair exchange):
// warp-sized tasks of A consecutive slots, neighbour coordinates gathered from
// global memory.  IMG: the mixed form with image codes in the list.
template <int TPA, bool MIXED, int KICK, bool EV, bool ONE, bool IMG>
__global__ void __launch_bounds__(256, MIXED ? 4 : 1) k_force(Dev d, Box b, StepConsts sc, ForceArgs fa) {
  constexpr int A = 32 / TPA;
  __shared__ typename std::conditional<MIXED, SmemTabF, SmemTabD>::type tab;
  __shared__ WarpImages<MIXED> wimg[8];
  __shared__ int s_halt;
  if (threadIdx.x == 0) s_halt = halted(d);
  load_tab(d, tab);
  __syncthreads();
  const bool was_halted = s_halt != 0;  // a step after a halt does nothing
  const int nt = d.tab->nt;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int a = lane % A, t = lane / A;
  const int n = sc.n, cap = d.cap;
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  const int ntask = was_halted ? 0 : (n + A - 1) / A;
  // EV: each thread's KE / virial / PE sums live in shared memory between tasks;
  // six doubles held in registers across the pair loop spill at 64 registers (dynamic, no
  // larger than the block: what shared memory takes, the gathers miss in L1)
  extern __shared__ double s_sum[];
  const int nthr = blockDim.x;
  if (EV)
#pragma unroll
    for (int q = 0; q < 6; ++q) s_sum[q * nthr + threadIdx.x] = 0.0;
  long long step = 0;
  if (KICK == 2) step = *d.step_base + fa.k_in_chunk;
  int img_rep = -1;

  for (int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < ntask; task += warps_total) {
    const int rep = rep_of_slot(b, task * A);
    if (rep < 0) continue;  // a task of padding slots (uniform over the warp)
    if (rep != img_rep) {
      const RepBox &rb = repbox(b, rep);
      if constexpr (MIXED) {
        if (lane == 0) {
          wimg[wid].hi = make_float4(rb.uh[0], rb.uh[1], rb.uh[2], 0.f);
          wimg[wid].lo = make_float4(rb.ul[0], rb.ul[1], rb.ul[2], 0.f);
          if (IMG) wimg[wid].flip = make_uint3(rb.flip[0], rb.flip[1], rb.flip[2]);
        }
      } else if (lane < 27) {
        const int sx = lane % 3 - 1, sy = (lane / 3) % 3 - 1, sz = lane / 9 - 1;
        wimg[wid].v[lane] = make_double3(sx * rb.L[0], sy * rb.L[1], sz * rb.L[2]);
      }
      __syncwarp();
      img_rep = rep;
    }
    const int i = task * A + a;
    const bool act = i < n && rep_of_slot(b, i) >= 0;
    double fx = 0.0, fy = 0.0, fz = 0.0, vir = 0.0, pe = 0.0;
    int ti = 0;
    if (act) {
      const int nn = d.nnbr[i];
      // the atom's neighbour words: chunk g (entries 4g..4g+3) is row4[g * A] (nbr_index)
      const uint4 *row4 = reinterpret_cast<const uint4 *>(d.nbr + (size_t)task * cap * A) + a;
      if constexpr (MIXED) {
        const int4 ri = d.ic[i];
        ti = ri.w;
        float ax = 0.f, ay = 0.f, az = 0.f;
        const int4 *ic = d.ic;
        const uint3 flip = IMG ? wimg[wid].flip : make_uint3(0u, 0u, 0u);
        mixed_pairs<TPA, EV, ONE, false>(row4 + t * A, nn, t, ri, nt, tab, one_type(tab), wimg[wid].hi, wimg[wid].lo, sc.jump_tolf,
                                  [ic, flip](uint32_t w) {
                                    const int4 q = __ldg(&ic[w & IDX_MASK]);
                                    return IMG ? image_of(q, w, flip) : q;
                                  },
                                  ax, ay, az, vir, pe);
        fx = ax; fy = ay; fz = az;
      } else {
        const dbl4 xi = d.pos[i];
        ti = type_of(xi.w);
        double F[5];
        fp64_pairs<TPA, EV, ONE>(d, row4, nn, t, xi, ti * nt, tab, wimg[wid].v, sc.jump_tol, F);
        fx = F[0]; fy = F[1]; fz = F[2];
        if (EV) vir = F[3], pe = F[4];
      }
    }
    fold_lanes<A, EV>(fx, fy, fz, vir, pe);
    if (act && t == 0) {
      double ke[4], ev[2];
      finish_atom<MIXED, KICK, EV>(d, b, sc, tab, i, ti, rep, step, fa.fuse, fx, fy, fz, ke);
      if (EV) {
        set_ev(d, i, vir, pe, ev);
#pragma unroll
        for (int q = 0; q < 4; ++q) s_sum[q * nthr + threadIdx.x] += ke[q];
#pragma unroll
        for (int q = 0; q < 2; ++q) s_sum[(4 + q) * nthr + threadIdx.x] += ev[q];
      }
    }
  }
  double ke_p[4] = {0.0, 0.0, 0.0, 0.0}, ev_p[2] = {0.0, 0.0};
  if (EV) {
#pragma unroll
    for (int q = 0; q < 4; ++q) ke_p[q] = s_sum[q * nthr + threadIdx.x];
#pragma unroll
    for (int q = 0; q < 2; ++q) ev_p[q] = s_sum[(4 + q) * nthr + threadIdx.x];
  }
  if (!was_halted) store_partials<KICK, EV>(d, ke_p, ev_p);
  if (KICK != 0) end_of_step<EV>(d, was_halted, fa);
}

// Mixed-form pair kernel over row segments.  A block takes a segment -- up to
// seg_umax - 2 consecutive cells of one x-row of one replica -- and stages into
// shared memory the fixed-point coordinates of the atoms of the 9 neighbouring rows'
// cells x0-1 .. x0+len (periodic), so that every neighbour gather of the
// segment's atoms reads shared memory.  A list word (slot j, stencil index k)
// finds its copy through a table: row r = k / 3 of the stencil, staged cell
// u = (home cell - x0) + k % 3, index = j + (stage offset - first slot) of (r, u).
// The arithmetic is that of the grid-strided kernel, so results are the same bit
// for bit.  A segment whose stencil holds more atoms than the stage falls back to
// global gathers.  Warps take the segment's A-slot tasks; lanes whose atom lies
// outside the segment idle (their atoms belong to the adjacent segment).
template <int TPA, int KICK, bool EV, bool ONE>
__global__ void __launch_bounds__(256) k_force_seg(Dev d, Box b, StepConsts sc, ForceArgs fa) {
  constexpr int A = 32 / TPA;
  constexpr int AS = 5 - (TPA == 1 ? 0 : TPA == 2 ? 1 : TPA == 4 ? 2 : TPA == 8 ? 3 : 4);  // log2(A)
  __shared__ SmemTabF tab;
  __shared__ float4 s_uh, s_ul;
  __shared__ int s_total;
  extern __shared__ int4 stage[];
  const int umax = d.seg_umax;
  int *const toff = reinterpret_cast<int *>(stage + d.stage_cap);  // [9 * umax] stage offset - first slot
  int *const tcnt = toff + 9 * umax;                                 // [9 * umax] atoms, then exclusive scan
  __shared__ int s_halt;
  if (threadIdx.x == 0) s_halt = halted(d);
  load_tab(d, tab);
  __syncthreads();
  const bool was_halted = s_halt != 0;  // a step after a halt does nothing
  const int nt = d.tab->nt;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int a = lane % A, t = lane / A;
  const int cap = d.cap;
  double ke_p[4] = {0.0, 0.0, 0.0, 0.0};
  double ev_p[2] = {0.0, 0.0};
  long long step = 0;
  if (KICK == 2) step = *d.step_base + fa.k_in_chunk;
  int img_rep = -1;
  const int nseg = was_halted ? 0 : d.nseg;

  for (int sgi = blockIdx.x; sgi < nseg; sgi += gridDim.x) {
    const int4 sg = d.seg[sgi];
    const int rep = sg.x, cy = sg.y & 0xffff, cz = sg.y >> 16, x0 = sg.z, len = sg.w;
    const RepBox &rb = repbox(b, rep);
    const int U = len + 2, nq = 9 * U;
    __syncthreads();  // the previous segment's gathers are done with the stage and tables
    if (rep != img_rep) {
      if (threadIdx.x == 0) {
        s_uh = make_float4(rb.uh[0], rb.uh[1], rb.uh[2], 0.f);
        s_ul = make_float4(rb.ul[0], rb.ul[1], rb.ul[2], 0.f);
      }
      img_rep = rep;
    }
    // staged cells q = r * U + u: row r = (dy + 1) + 3 (dz + 1), x cell x0 - 1 + u (periodic)
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
      const int r = q / U, u = q - r * U;
      int ny = cy + r % 3 - 1, nz = cz + r / 3 - 1, nx = (x0 - 1 + u) % rb.nc[0];
      if (nx < 0) nx += rb.nc[0];
      if (ny < 0) ny += rb.nc[1]; else if (ny >= rb.nc[1]) ny -= rb.nc[1];
      if (nz < 0) nz += rb.nc[2]; else if (nz >= rb.nc[2]) nz -= rb.nc[2];
      const int c = rb.cell_off + nx + rb.nc[0] * (ny + rb.nc[1] * nz);
      const int st = d.cell_start[c];
      toff[q] = st;
      tcnt[q] = d.cell_start[c + 1] - st;
    }
    __syncthreads();
    // exclusive scan of the counts (nq <= 9 * umax) by warp 0, 32 entries at a time
    if (wid == 0) {
      int carry = 0;
      for (int base = 0; base < nq; base += 32) {
        const int q = base + lane;
        const int v = q < nq ? tcnt[q] : 0;
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL_MASK, inc, o);
          if (lane >= o) inc += y;
        }
        if (q < nq) tcnt[q] = carry + inc - v;
        carry += __shfl_sync(FULL_MASK, inc, 31);
      }
      if (lane == 0) s_total = carry;
    }
    __syncthreads();
    const bool staged = s_total <= d.stage_cap;
    if (staged) {
      // copy: warp w takes staged cells w, w + nwarp, ...; lanes copy the cell's atoms
      for (int q = wid; q < nq; q += nwarp) {
        const int st = toff[q], base = tcnt[q];
        const int cn = (q + 1 < nq ? tcnt[q + 1] : s_total) - base;
        for (int k = lane; k < cn; k += 32) stage[base + k] = __ldg(&d.ic[st + k]);
      }
      __syncthreads();
      for (int q = threadIdx.x; q < nq; q += blockDim.x) toff[q] = tcnt[q] - toff[q];
    }
    __syncthreads();
    // the segment's atoms: slots of its cells (consecutive cell indices, so one range)
    const int rowc = rb.cell_off + rb.nc[0] * (cy + rb.nc[1] * cz);
    const int hs = d.cell_start[rowc + x0], he = d.cell_start[rowc + x0 + len];
    if (he > hs) {
      const int t_first = hs >> AS, t_last = (he - 1) >> AS;
      for (int task = t_first + wid; task <= t_last; task += nwarp) {
        const int i = task * A + a;
        const bool act = i >= hs && i < he;
        double fx = 0.0, fy = 0.0, fz = 0.0, vir = 0.0, pe = 0.0;
        int ti = 0;
        if (act) {
          const int nn = d.nnbr[i];
          const uint4 *row4 = reinterpret_cast<const uint4 *>(d.nbr + (size_t)task * cap * A) + (t * A + a);
          const int4 ri = d.ic[i];
          ti = ri.w;
          float ax = 0.f, ay = 0.f, az = 0.f;
          if (staged) {
            const int hx = d.cell_of[i] - rowc - x0;  // home cell within the segment
            const int *tr = toff + hx;
            mixed_pairs<TPA, EV, ONE, false>(row4, nn, t, ri, nt, tab, one_type(tab), s_uh, s_ul, sc.jump_tolf,
                                 [tr, U](uint32_t w) {  // `stage` is the block's shared array
                                   const int k = (int)(w >> CODE_SHIFT), r = (k * 11) >> 5;  // k / 3 for k < 27
                                   return stage[(int)(w & IDX_MASK) + tr[r * U + (k - 3 * r)]];
                                 },
                                 ax, ay, az, vir, pe);
          } else {
            const int4 *ic = d.ic;
            mixed_pairs<TPA, EV, ONE, false>(row4, nn, t, ri, nt, tab, one_type(tab), s_uh, s_ul, sc.jump_tolf,
                                 [ic](uint32_t w) { return __ldg(&ic[w & IDX_MASK]); }, ax, ay, az, vir, pe);
          }
          fx = ax; fy = ay; fz = az;
        }
        fold_lanes<A, EV>(fx, fy, fz, vir, pe);
        if (act && t == 0) {
          double ke[4], ev[2];
          finish_atom<true, KICK, EV>(d, b, sc, tab, i, ti, rep, step, fa.fuse, fx, fy, fz, ke);
          if (EV) {
            set_ev(d, i, vir, pe, ev);
#pragma unroll
            for (int q = 0; q < 4; ++q) ke_p[q] += ke[q];
#pragma unroll
            for (int q = 0; q < 2; ++q) ev_p[q] += ev[q];
          }
        }
      }
    }
  }
  if (!was_halted) store_partials<KICK, EV>(d, ke_p, ev_p);
  if (KICK != 0) end_of_step<EV>(d, was_halted, fa);
}

template <int TPA, bool MIXED, int KICK>
static void launch_ev(bool ev, bool one, bool img, int grid, int block, const Dev &d, const Box &b,
                      const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  const size_t ev_smem = (size_t)6 * block * sizeof(double);
  if (img) {  // (rare: whatever the types)
    if (ev) k_force<TPA, MIXED, KICK, true, false, MIXED><<<grid, block, ev_smem, st>>>(d, b, sc, fa);
    else k_force<TPA, MIXED, KICK, false, false, MIXED><<<grid, block, 0, st>>>(d, b, sc, fa);
    return;
  }
  if (one) {  // single-type systems: pair constants in registers
    if (ev) k_force<TPA, MIXED, KICK, true, true, false><<<grid, block, ev_smem, st>>>(d, b, sc, fa);
    else k_force<TPA, MIXED, KICK, false, true, false><<<grid, block, 0, st>>>(d, b, sc, fa);
    return;
  }
  if (ev) k_force<TPA, MIXED, KICK, true, false, false><<<grid, block, ev_smem, st>>>(d, b, sc, fa);
  else k_force<TPA, MIXED, KICK, false, false, false><<<grid, block, 0, st>>>(d, b, sc, fa);
}

template <int TPA, bool MIXED>
static void launch_kick(int kick, bool ev, bool one, bool img, int grid, int block, const Dev &d, const Box &b,
                        const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  if (kick == 0) launch_ev<TPA, MIXED, 0>(ev, one, img, grid, block, d, b, sc, fa, st);
  else if (kick == 1) launch_ev<TPA, MIXED, 1>(ev, one, img, grid, block, d, b, sc, fa, st);
  else launch_ev<TPA, MIXED, 2>(ev, one, img, grid, block, d, b, sc, fa, st);
}

template <bool MIXED>
static int launch_tpa(int tpa, int kick, bool ev, bool one, bool img, int grid, int block, const Dev &d, const Box &b,
                      const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  switch (tpa) {
    case 1: launch_kick<1, MIXED>(kick, ev, one, img, grid, block, d, b, sc, fa, st); break;
    case 2: launch_kick<2, MIXED>(kick, ev, one, img, grid, block, d, b, sc, fa, st); break;
    case 4: launch_kick<4, MIXED>(kick, ev, one, img, grid, block, d, b, sc, fa, st); break;
    case 8: launch_kick<8, MIXED>(kick, ev, one, img, grid, block, d, b, sc, fa, st); break;
    case 16: launch_kick<16, MIXED>(kick, ev, one, img, grid, block, d, b, sc, fa, st); break;
    default: return CAVGPU_E_ARG;
  }
  return CAVGPU_OK;
}

// the segment kernel's variants, for launching and for their shared-memory attribute
template <int TPA, int KICK, bool EV>
static int seg_variant(bool launch, bool one, int grid, int block, size_t smem, const Dev &d, const Box &b,
                       const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  if (!launch) {
    if (cudaFuncSetAttribute(k_force_seg<TPA, KICK, EV, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(k_force_seg<TPA, KICK, EV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return CAVGPU_E_CUDA;
    return CAVGPU_OK;
  }
  if (one) k_force_seg<TPA, KICK, EV, true><<<grid, block, smem, st>>>(d, b, sc, fa);
  else k_force_seg<TPA, KICK, EV, false><<<grid, block, smem, st>>>(d, b, sc, fa);
  return CAVGPU_OK;
}
template <int TPA>
static int seg_kick(bool launch, int kick, bool ev, bool one, int grid, int block, size_t smem, const Dev &d,
                    const Box &b, const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  if (kick == 0) return ev ? seg_variant<TPA, 0, true>(launch, one, grid, block, smem, d, b, sc, fa, st)
                           : seg_variant<TPA, 0, false>(launch, one, grid, block, smem, d, b, sc, fa, st);
  if (kick == 1) return ev ? seg_variant<TPA, 1, true>(launch, one, grid, block, smem, d, b, sc, fa, st)
                           : seg_variant<TPA, 1, false>(launch, one, grid, block, smem, d, b, sc, fa, st);
  return ev ? seg_variant<TPA, 2, true>(launch, one, grid, block, smem, d, b, sc, fa, st)
            : seg_variant<TPA, 2, false>(launch, one, grid, block, smem, d, b, sc, fa, st);
}
static int seg_tpa(bool launch, int tpa, int kick, bool ev, bool one, int grid, int block, size_t smem,
                   const Dev &d, const Box &b, const StepConsts &sc, const ForceArgs &fa, cudaStream_t st) {
  switch (tpa) {
    case 1: return seg_kick<1>(launch, kick, ev, one, grid, block, smem, d, b, sc, fa, st);
    case 2: return seg_kick<2>(launch, kick, ev, one, grid, block, smem, d, b, sc, fa, st);
    case 4: return seg_kick<4>(launch, kick, ev, one, grid, block, smem, d, b, sc, fa, st);
    case 8: return seg_kick<8>(launch, kick, ev, one, grid, block, smem, d, b, sc, fa, st);
    case 16: return seg_kick<16>(launch, kick, ev, one, grid, block, smem, d, b, sc, fa, st);
    default: return CAVGPU_E_ARG;
  }
}

int prepare_force_seg(size_t smem_bytes) {
  Dev d{};
  Box b{};
  StepConsts sc{};
  for (int tpa = 1; tpa <= 16; tpa *= 2)
    for (int kick = 0; kick < 3; ++kick)
      for (int ev = 0; ev < 2; ++ev) {
        const int rc = seg_tpa(false, tpa, kick, ev != 0, false, 0, 0, smem_bytes, d, b, sc, ForceArgs{}, nullptr);
        if (rc) return rc;
      }
  return CAVGPU_OK;
}

int force_grid_blocks(const LaunchCfg &lc) {
  const int sms = num_sms();
  if (segments_on(lc))  // one segment per block at a time
    return lc.nseg < sms * 4 ? lc.nseg : sms * 4;
  const int A = 32 / lc.tpa, block = lc.exchange ? exchange_close_threads() : lc.block;
  const long long ntask = (lc.n + A - 1) / A;
  const long long warps_per_block = block / 32;
  long long need = (ntask + warps_per_block - 1) / warps_per_block;
  // the mixed kernels (64 registers) hold 32 warps per SM: one wave of resident blocks,
  // each warp walking its tasks grid-strided (fewer, longer-lived blocks: fewer block
  // reductions and tails; 5% less pair-kernel time and 16% less for the thermo
  // variant on the 1M-atom fluid than four waves); the FP64 kernels: four waves
  const long long cap = lc.precision == CAVGPU_MIXED ? (long long)sms * (1024 / block)
                                                     : (long long)sms * (2048 / block) * 4;
  if (need > cap) need = cap;
  return (int)(need < 1 ? 1 : need);
}

int ev_grid_blocks(const LaunchCfg &lc) {
  if (!lc.exchange) return force_grid_blocks(lc);
  const int A = 32 / lc.tpa;
  return exchange_pair_blocks((lc.n + A - 1) / A);
}

int launch_force(const Dev &d, const Box &b, const StepConsts &sc, const LaunchCfg &lc, int kick, int thermo,
                 int k, int fuse, int set_cond, cudaGraphConditionalHandle cond, cudaStream_t st,
                 const FoldArgs *fold) {
  const int grid = force_grid_blocks(lc);
  const int grid_ev = ev_grid_blocks(lc);
  if (std::max(grid, grid_ev) > d.partials_blocks) return CAVGPU_E_ARG;  // each block writes its own partial sums
  if (kick == 0 && (fuse || set_cond)) return CAVGPU_E_ARG;
  if (fold && (kick == 0 || !thermo)) return CAVGPU_E_ARG;  // the fold needs this launch's EV partials
  ForceArgs fa{k, fuse, set_cond, cond, fold ? 1 : 0, {}};
  if (fold) fa.fa = *fold;
  int rc;
  if (segments_on(lc)) {
    if (!d.seg || d.nseg != lc.nseg) return CAVGPU_E_ARG;
    rc = seg_tpa(true, lc.tpa, kick, thermo != 0, lc.ntypes == 1, grid, lc.block,
                 seg_smem_bytes(d.stage_cap, d.seg_umax), d, b, sc, fa, st);
  } else if (lc.exchange) {
    if (!d.recv) return CAVGPU_E_ARG;
    rc = launch_force_exchange(d, b, sc, lc, kick, thermo != 0, fa, grid, grid_ev, st);
  } else {
    const bool one = lc.ntypes == 1;
    rc = lc.precision == CAVGPU_MIXED
             ? launch_tpa<true>(lc.tpa, kick, thermo != 0, one, lc.images != 0, grid, lc.block, d, b, sc, fa, st)
             : launch_tpa<false>(lc.tpa, kick, thermo != 0, one, false, grid, lc.block, d, b, sc, fa, st);
  }
  if (rc) return rc;
  return cudaPeekAtLastError() == cudaSuccess ? CAVGPU_OK : CAVGPU_E_CUDA;
}

}  // namespace cav
