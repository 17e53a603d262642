// cav_rebuild.cuh -- the parts of a list rebuild as device functions: the kernels of
// cav_kernels.cu run one each, the step kernel of small systems (cav_chunk.cu) all of them
// with barriers between.
#pragma once

#include "cav_common.cuh"

namespace cav {

// ---------------------------------------------------------------------------
// list rebuild of the flagged replicas: wrap + bin -> per-replica scan ->
// scatter -> per-cell sort -> gather -> build
// (Neighborlist::update_cell_list + update_verlet_list_from_cell_list,
//  src/neighborlist.cpp:422-455, 496-553; Domain::fix_position, src/domain.cpp:443-493)
// ---------------------------------------------------------------------------
// Domain::fix_position's single-image test per axis (src/domain.cpp:443-493):
// -1 below the lower face (x += L), +1 above the upper face (x -= L), else 0
__device__ inline int3 wrap_shift(const RepBox &rb, const dbl4 &p) {
  return make_int3(p.x < rb.lo[0] ? -1 : (p.x > rb.hi[0] ? 1 : 0), p.y < rb.lo[1] ? -1 : (p.y > rb.hi[1] ? 1 : 0),
                   p.z < rb.lo[2] ? -1 : (p.z > rb.hi[2] ? 1 : 0));
}

// Search cell of an atom (clamped into the grid), its place in it: position relative to the
// cell's origin and Morton index of the 4x4x4 sub-cell.
struct CellPlace {
  int c[3];
  float rel[3];
  uint32_t morton;
};
__device__ __forceinline__ uint32_t spread_bits(int s) { return (s & 1) | ((s & 2) << 2); }

// The general case: any position.  Wraps p (single image, exactly as Domain::fix_position)
// and counts the crossings (+1 through the upper face) as exchange_owned adds them to
// msd_domain_cross.
static __device__ __noinline__ void place_general(const Dev &d, const RepBox &rb, int i, dbl4 &p, CellPlace &q) {
  const int3 w = wrap_shift(rb, p);
  if (w.x | w.y | w.z) {
    if (w.x) p.x += w.x > 0 ? -rb.L[0] : rb.L[0];
    if (w.y) p.y += w.y > 0 ? -rb.L[1] : rb.L[1];
    if (w.z) p.z += w.z > 0 ? -rb.L[2] : rb.L[2];
    d.pos[i] = p;
    if (d.img) {
      int4 m = d.img[i];
      m.x += w.x; m.y += w.y; m.z += w.z;
      d.img[i] = m;
    }
  }
  const double x[3] = {p.x, p.y, p.z};
  q.morton = 0;
  for (int a = 0; a < 3; ++a) {
    const double u = (x[a] - rb.lo[a]) * rb.inv_w[a];
    q.c[a] = min(max((int)floor(u), 0), rb.nc[a] - 1);
    q.rel[a] = (float)(x[a] - (rb.lo[a] + q.c[a] * rb.w[a]));
    q.morton |= spread_bits(min(max((int)((u - q.c[a]) * 4.0), 0), 3)) << a;
  }
}

// An atom inside the box, along one axis: the cell coordinate in fixed point with 34
// fractional bits (one subtraction and one FMA, which leaves the integer in the mantissa),
// the rest by integers.  The FP64 pipe bound the binning kernel (79% busy, 61 us for 1,048,576
// atoms: floors, conversions and compares, ~36 FP64 instructions per atom); 6 are left.  The
// rounding, 2^-35 of a cell, is below the 1e-10 by which cells are wider than the list
// cutoff at least.  False when the atom is not well inside, or the grid too long for this.
__device__ __forceinline__ bool place_axis(double x, double lo, double inv_w, int nc, float wf, int &c, float &rel,
                                           int &sub) {
  const long long t = __double_as_longlong(fma(x - lo, inv_w * 17179869184.0, 6755399441055744.0));  // 2^34, 1.5 * 2^52
  const long long n = t - 0x4338000000000000ll;
  c = (int)(n >> 34);
  sub = (int)(n >> 32) & 3;
  rel = (float)(unsigned)((unsigned long long)n >> 2) * (wf * 2.3283064365386963e-10f);  // 2^-32
  return (t >> 52) == 0x433 && n >= 1 && n < ((long long)nc << 34) - 1 && nc <= 65536;
}

// Thread of slot i (the whole warp calls this): wraps the atom, counts it in its cell and
// copies its state, which rebuild_sort_gather takes back in the new order.
__device__ __forceinline__ void rebuild_bin(const Dev &d, const Box &b, int forced, int i) {
  if (i == 0) d.flags[F_MAXNB] = 0;
  int rep = i < b.nslot ? rep_of_slot(b, i) : -1;
  const bool act = rep >= 0 && rebuild_on(d, b, rep, forced);
  int c = 0;
  if (act) {
    const RepBox &rb = repbox(b, rep);
    dbl4 p = d.pos[i];
    CellPlace q;
    int sx, sy, sz;
    const bool inside = place_axis(p.x, rb.lo[0], rb.inv_w[0], rb.nc[0], rb.wf[0], q.c[0], q.rel[0], sx) &
                        place_axis(p.y, rb.lo[1], rb.inv_w[1], rb.nc[1], rb.wf[1], q.c[1], q.rel[1], sy) &
                        place_axis(p.z, rb.lo[2], rb.inv_w[2], rb.nc[2], rb.wf[2], q.c[2], q.rel[2], sz);
    q.morton = spread_bits(sx) | (spread_bits(sy) << 1) | (spread_bits(sz) << 2);
    if (!inside) place_general(d, rb, i, p, q);
    c = rb.cell_off + q.c[0] + rb.nc[0] * (q.c[1] + rb.nc[1] * q.c[2]);
    d.atom_cell[i] = c;
    // order inside the cell: the sub-cell, then the id, so that consecutive slots (a warp's
    // lanes) sit close together and their neighbour lists run through the same candidates
    const uint32_t id = d.id[i];
    d.skey[i] = ((uint64_t)q.morton << 32) | id;
    d.t_pos[i] = p;
    d.t_vel[i] = d.vel[i];
    d.t_acc[i] = d.acc[i];  // a(t): the next kick reads it as a_old
    d.t_rel[i] = make_float4(q.rel[0], q.rel[1], q.rel[2], __int_as_float(type_of(p.w)));
    d.t_id[i] = id;
    if (d.img) d.t_img[i] = d.img[i];
    if (d.mol) d.t_mol[i] = d.mol[i];
  }
  // warp-aggregated counting: one atomic per distinct cell in the warp
  const unsigned m = __ballot_sync(FULL_MASK, act);
  if (act) {
    const unsigned peers = __match_any_sync(m, c);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&d.cell_count[c], __popc(peers));
  }
}

__device__ inline int scan_count(const Dev &d, const RepBox &rb, int m, int k) {
  return k == m - 1 ? rb.pad : d.cell_count[rb.cell_off + k];
}

__device__ __forceinline__ void rebuild_scatter(const Dev &d, const Box &b, int forced, int i) {
  const int rep = rep_of_slot(b, i);
  if (rep < 0 || !rebuild_on(d, b, rep, forced)) return;
  const int c = d.atom_cell[i];
  d.perm_tmp[d.cell_start[c] + atomicAdd(&d.cell_cursor[c], 1)] = i;
}

// slot k takes the state of old slot o
__device__ __forceinline__ void rebuild_gather(const Dev &d, const RepBox &rb, int k, int o) {
  const dbl4 x = d.t_pos[o];
  d.pos[k] = x;
  d.pos_ref[k] = x;
  d.vel[k] = d.t_vel[o];
  d.acc[k] = d.t_acc[o];
  const float4 rel = d.t_rel[o];
  d.rel[k] = rel;
  const int type = __float_as_int(rel.w);
  d.type[k] = type;
  d.id[k] = d.t_id[o];
  if (d.img) d.img[k] = d.t_img[o];
  if (d.mol) d.mol[k] = d.t_mol[o];
  d.cell_of[k] = d.atom_cell[o];
  if (d.ic) {
    int3 w;
    const int4 q = fixed_pos(rb, x, type, w);
    d.ic[k] = q;
    if (d.ic_ref) d.ic_ref[k] = fixed_ref(q, w);
  }
  if (d.nr) d.nr[k] = 0;
}

// Warp of a cell: orders its atoms by their sort key (sub-cell, then host index:
// deterministic lists) and moves their state to their slots; cells of up to 32 atoms rank
// in registers with warp shuffles.
__device__ __forceinline__ void rebuild_sort_gather(const Dev &d, const Box &b, int forced, int cell) {
  const int lane = threadIdx.x & 31;
  const int rep = rep_of_cell(b, cell);
  if (rep < 0 || !rebuild_on(d, b, rep, forced)) return;
  const RepBox &rb = repbox(b, rep);
  const int s = d.cell_start[cell], e = d.cell_start[cell + 1], n = e - s;
  if (n <= 32) {
    const int ia = lane < n ? d.perm_tmp[s + lane] : 0;
    const uint64_t ka = lane < n ? d.skey[ia] : ~0ull;
    int rank = 0;
    for (int q = 0; q < n; ++q) rank += __shfl_sync(FULL_MASK, ka, q) < ka;
    if (lane < n) rebuild_gather(d, rb, s + rank, ia);
    return;
  }
  for (int a = lane; a < n; a += 32) {
    const int ia = d.perm_tmp[s + a];
    const uint64_t ka = d.skey[ia];
    int rank = 0;
    for (int q = 0; q < n; ++q) rank += d.skey[d.perm_tmp[s + q]] < ka;
    rebuild_gather(d, rb, s + rank, ia);
  }
}

// Verlet-list build over the 27-cell stencil with periodic image shifts.
// Predicate: r^2 < cutoff_extra^2 evaluated in FP64 exactly as the reference
// evaluates it for a ghost image (image = x_j + s*L, then minus x_i, squares
// summed x, y, z; no FMA contraction), pre-screened in FP32 on cell-relative
// coordinates: only candidates inside a narrow band around the cutoff take
// the FP64 path.  mode 0 stores image codes (FP64 force), mode 1 cell-offset
// codes (mixed force).
static __device__ __noinline__ bool exact_pair(const Dev &d, const RepBox &rb, double ce2, int i, int j, int img) {
  const dbl4 xi = d.pos[i], xj = d.pos[j];
  const double shx = (img % 3 - 1) * rb.L[0], shy = ((img / 3) % 3 - 1) * rb.L[1], shz = (img / 9 - 1) * rb.L[2];
  const double ddx = __dsub_rn(__dadd_rn(xj.x, shx), xi.x);
  const double ddy = __dsub_rn(__dadd_rn(xj.y, shy), xi.y);
  const double ddz = __dsub_rn(__dadd_rn(xj.z, shz), xi.z);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
  return r2 < ce2;
}

// Home groups.  A warp takes a window of 32 consecutive slots; the window's atoms
// that lie in one x-row of search cells, within GROUP_SPAN + 1 consecutive cells of
// it, form a group (a window that crosses the end of a row, or a sparse row, takes
// two or more groups in turn).  Slots are sorted by cell, so a group is 32 (or
// fewer) atoms from 1-3 neighbouring cells.  Its candidates are the atoms of the
// cells cx_first - 1 .. cx_last + 1 of the 3 x 3 neighbouring rows, taken row by row,
// and of those only the ones within the list cutoff (plus the FP32 band) of the
// group's bounding box are staged: ~540 staged candidates per 32 atoms of the 1M-atom
// fluid, against 27 cells x 19 atoms = 516 per 19-atom cell when a warp took one cell.
//
// Order of an atom's row: the neighbouring rows of cells as ROW_ORDER has them, in a row
// the cells by their x index modulo 3, slot order inside a cell; it depends on the
// atom's cell alone, not on how slots fall into windows.  The order is chosen for the
// pair kernel's gathers, where the 32 lanes of a warp are 32 atoms that each read the
// k-th entry of their own row: they touch the fewest 128-byte lines when the lanes are
// at the same cell at the same k.  In stencil order (z, then y, then x) they are not --
// an atom at the bottom of its cell has half its neighbours in the lower layer, one at
// the top next to none -- so the rows alternate between opposite sides of the stencil,
// which keeps the running counts of the lanes close, and the x index modulo 3 makes
// atoms of adjacent cells take their common cells at the same time.  Distinct lines per
// gather in a melted fluid (counted on the host): 16.0 in stencil order, 10.6 in this one.
__constant__ const int8_t ROW_ORDER[9] = {4, 0, 8, 2, 6, 1, 7, 3, 5};  // (dy+1) + 3 (dz+1), nearest row first
// Which of the group's nu candidate cells of a row comes k-th: cells x0 + u by
// (x0 + u) mod 3, ascending inside a class (x0 >= -1).
__device__ __forceinline__ int class_cell(int x0, int nu, int k) {
  int u = 0;
  for (int c = 0; c < 3; ++c) {
    u = (c + 3 - (x0 + 3) % 3) % 3;  // first cell of class c
    const int n = (nu - u + 2) / 3;  // nu >= 3: every class has a cell
    if (k < n) break;
    k -= n;
  }
  return u + 3 * k;
}

// Staging: candidates u and u+1 (u even) interleaved as {x_u, x_u+1, y_u, y_u+1}
// and {z_u, z_u+1} in the warp's slice of shared memory (coordinates relative to
// the origin of the group's first cell), the words (j | code) in an array of their
// own, plus one byte per candidate: its cell's x index in the group's window of
// cells and its row (dy, dz).  The sweep takes 32 candidates at a time, two per
// packed FP32x2 distance evaluation: every pair of candidates is two shared-memory
// broadcasts tested by all group atoms, the results collect in a hit and a band bit
// mask per lane (one warp vote per 32 candidates for the rare exact FP64 test), and
// only then are the hits (~15% of the staged candidates) written, in candidate order.
constexpr int BUILD_STAGE = 256;  // staged candidates per warp and pass (4 KiB + 256 B)
// hits per lane that a part of a shared window holds: up to ~0.42 of an atom's, ~46 of 110 at
// density 1.2 (40: one warp did most dense windows again, a step of 24 replicas 101 us against
// 82; 64: a block fewer per SM)
constexpr int SEG_HITS = 56;
constexpr int GROUP_SPAN = 5;     // a group spans at most 6 cells: x index + 8 row < 256

// q_u, q_u+1 = |c - r|^2 of two candidates with packed FP32x2 arithmetic (sm_100+):
// (cx - rx)^2, then + (cy - ry)^2, then + (cz - rz)^2, each rounded once
__device__ __forceinline__ void dist2_pair(const float4 &xy, const float2 &z, unsigned long long rxx,
                                           unsigned long long ryy, unsigned long long rzz, float &q0, float &q1) {
  asm("{\n\t.reg .b64 c, dd, q;\n\t"
      "mov.b64 c, {%2, %3};\n\tsub.rn.f32x2 dd, c, %8;\n\tmul.rn.f32x2 q, dd, dd;\n\t"
      "mov.b64 c, {%4, %5};\n\tsub.rn.f32x2 dd, c, %9;\n\tfma.rn.f32x2 q, dd, dd, q;\n\t"
      "mov.b64 c, {%6, %7};\n\tsub.rn.f32x2 dd, c, %10;\n\tfma.rn.f32x2 q, dd, dd, q;\n\t"
      "mov.b64 {%0, %1}, q;\n\t}"
      : "=f"(q0), "=f"(q1)
      : "f"(xy.x), "f"(xy.y), "f"(xy.z), "f"(xy.w), "f"(z.x), "f"(z.y), "l"(rxx), "l"(ryy), "l"(rzz));
}

__device__ __forceinline__ unsigned long long pack2(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

// The lane's side of a group: its atom, where it sits in the group, its row.
struct BuildLane {
  int i;              // slot (valid when `me`)
  bool me;            // member of the current group
  int ci;             // x cell index within the group (0 .. span)
  int cx, cy, cz;     // cell of the atom
  int mol;            // molecule index (ignore_intra_molecule)
  unsigned long long rxx, ryy, rzz;  // the atom's coordinates in the group frame, packed twice
  float hi;           // upper end of the FP32 band (-1 for non-members: they never hit)
  uint32_t *row;      // the atom's list row
  int cnt;            // list words the atom has so far
  const int *selfpos; // shared: per lane, where its own atom sits in the current stage (-1: not in it)
};

// Sweep of nst staged candidates against every member of the group (see above).
// Staged words carry j and a code: the image code (MODE 0), or (MODE 1) the cell's
// x index in the group's window of cells plus 3 x its row, from which a member
// subtracts its own x index to get the stencil index of j's cell relative to its own.
template <int MODE>
__device__ __forceinline__ void build_sweep(const Dev &d, const Box &b, const RepBox &rb, int nst,
                                            const float4 *sxy, const float2 *sz, const uint32_t *sw,
                                            const uint8_t *su, BuildLane &L, int cshift, bool by_mol, uint32_t *seg) {
  const int lane = threadIdx.x & 31;
  float *pxy = const_cast<float *>(reinterpret_cast<const float *>(sxy));
  float *pz = const_cast<float *>(reinterpret_cast<const float *>(sz));
  const int npad32 = (nst + 31) & ~31;
  for (int t = nst + lane; t < npad32; t += 32) {  // far-away padding up to a whole 32
    const int e = (t >> 1) * 4 + (t & 1);
    pxy[e] = 1e18f;
    pxy[e + 2] = 1e18f;
    pz[t] = 1e18f;
    const_cast<uint32_t *>(sw)[t] = 0u;
  }
  __syncwarp();
  const float lo = b.ce2_lo;
  const int cap = d.cap;
  const int self = L.selfpos[lane];
  const uint32_t ci_code = (uint32_t)L.ci << CODE_SHIFT;
  for (int t0 = 0; t0 < npad32; t0 += 32) {
    // phase 1: bits of the sure hits (q < ce2_lo) and of everything up to ce2_hi
    uint32_t hm = 0u, am = 0u;
#pragma unroll
    for (int u = 0; u < 32; u += 2) {
      const int pr = (t0 + u) >> 1;
      const float4 xy = sxy[pr];  // broadcast
      const float2 z = sz[pr];    // broadcast
      float q0, q1;
      dist2_pair(xy, z, L.rxx, L.ryy, L.rzz, q0, q1);
      if (q0 < lo) hm |= 1u << u;
      if (q0 <= L.hi) am |= 1u << u;
      if (q1 < lo) hm |= 2u << u;
      if (q1 <= L.hi) am |= 2u << u;
    }
    const int ts = self - t0;  // the atom itself is no candidate
    if (ts >= 0 && ts < 32) am &= ~(1u << ts);
    hm &= am;
    uint32_t bm = am & ~hm;  // the band
    const uint32_t *swc = sw + t0;
    if (__any_sync(FULL_MASK, bm != 0u)) {  // rare: the exact FP64 predicate
      while (bm) {
        const int u = __ffs(bm) - 1;
        bm &= bm - 1u;
        const int t = t0 + u;
        const uint32_t w = swc[u];
        const int j = (int)(w & IDX_MASK);
        int img = (int)(w >> CODE_SHIFT);
        if (MODE != 0) {  // the image from the candidate cell's unwrapped index
          const int s = su[t], r = s >> 3;
          const int nx = L.cx + (s & 7) - 1 - L.ci, ny = L.cy + r % 3 - 1, nz = L.cz + r / 3 - 1;
          img = image_code(nx < 0 ? -1 : (nx >= rb.nc[0] ? 1 : 0), ny < 0 ? -1 : (ny >= rb.nc[1] ? 1 : 0),
                           nz < 0 ? -1 : (nz >= rb.nc[2] ? 1 : 0));
        }
        if (exact_pair(d, rb, b.ce2, L.i, j, img)) hm |= 1u << u;
      }
    }
    // phase 2: the hits, in candidate order (with ignore_intra_molecule none of the
    // atom's own molecule, as Lj::calculate_acceleration skips them, src/force/lj.cpp:446).
    // A warp takes as many turns as its lane with the most hits, twice the mean, so a turn is
    // kept short: the place moves by steps instead of being computed (forces() of 1,048,576
    // atoms 969 -> 950 us)
    if (by_mol)
      for (uint32_t m = hm; m; m &= m - 1u) {
        const int u = __ffs(m) - 1;
        if (d.mol[swc[u] & IDX_MASK] == L.mol) hm &= ~(1u << u);
      }
    int n = L.cnt;
    // seg: a part of the group's candidates, hits by number and lane
    uint32_t *p = seg ? seg + n * 32 + lane : L.row + ((n >> 2) << cshift) + (n & 3);
    const int room = seg ? SEG_HITS : cap, next = seg ? 32 : 1, next4 = seg ? 32 : (1 << cshift) - 3;
    while (hm) {
      const int u = __ffs(hm) - 1;
      hm &= hm - 1u;
      uint32_t w = swc[u];
      if (MODE != 0) w -= ci_code;  // stencil index of j's cell relative to the atom's
      if (n < room) *p = w;
      ++n;
      p += (n & 3) ? next : next4;
    }
    L.cnt = n;
  }
  __syncwarp();  // the stage is refilled next
}

__device__ inline float warp_minf(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(FULL_MASK, v, o));
  return v;
}
__device__ inline float warp_maxf(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL_MASK, v, o));
  return v;
}

// a warp's stage: pair p = candidates 2p, 2p+1: xy[p] = {x, x', y, y'}, z[p] = {z, z'}; w[t] =
// word of t, u[t] its cell in the group's window, self: where the lanes' own atoms are
struct BuildStage {
  float4 xy[BUILD_STAGE / 2];
  float2 z[BUILD_STAGE / 2];
  uint32_t w[BUILD_STAGE];
  uint8_t u[BUILD_STAGE];
  int self[32];
};

// The four warps of a block share a window (small systems: a window takes one warp some
// 38 us from end to end, whatever the rest of the GPU does): each takes a part of the
// candidates' rows, about balanced by the candidates that survive the culling; the first
// writes its hits straight to the list rows, the others keep theirs in shared memory and
// move them behind those of the parts before.  An atom with more hits in a part than fit
// there sends the window to one warp.  Not where rows are so long that every window would
// end there, after the four warps' work (shared_windows).
struct BuildShare {
  BuildStage stage[4];
  uint32_t hits[3][SEG_HITS * 32];
  int cnt[4][32];
};
__constant__ const int8_t PART_ROWS[5] = {0, 2, 5, 7, 9};  // of ROW_ORDER

// Step mixed, shared and not: rows of 127 words 4,000 atoms 14.5 and 19.8 us, 32,000 atoms 27.3 and
// 31.2; of 139 words 23.4 and 23.0, 42.1 and 34.3; of 179 words 28.4 and 25.0, 58.2 and 37.9.
constexpr int SHARED_ROW = 132;
inline bool shared_windows(const LaunchCfg &lc) { return lc.row <= SHARED_ROW; }

// SHARED false: warp gw of nw takes the windows gw, gw + nw, ...; true: block gw of nw, the
// warps of a block (four) the parts of its windows.  split > 1: the groups of a window are
// dealt to that many warps or blocks.
template <int MODE, bool SHARED>
__device__ __forceinline__ void rebuild_build(const Dev &d, const Box &b, int forced, BuildStage &stage, int gw, int nw,
                                              BuildShare *share, int split = 1) {
  const int part = SHARED ? threadIdx.x >> 5 : 0;
  const int lane = threadIdx.x & 31;
  float4 *sxy = stage.xy;
  float2 *sz = stage.z;
  uint32_t *sw = stage.w;
  float *fxy = reinterpret_cast<float *>(sxy), *fz = reinterpret_cast<float *>(sz);
  uint8_t *su = stage.u;
  const bool by_mol = d.mol != nullptr;
  const int cshift = 7 - log2_pow2(d.tpa);  // chunk stride 4A words = 2^(log2 A + 2)
  const unsigned lt_mask = (1u << lane) - 1u;
  const int nwin = (b.nslot + 31) >> 5;
  int wmax = 0;
  for (int task = gw; task < nwin * split; task += nw) {
    const int win = task / split, mine = task - win * split;
    int group = 0;
    BuildLane L;
    L.i = (win << 5) + lane;
    const int rep = L.i < b.nslot ? rep_of_slot(b, L.i) : -1;
    const bool act = rep >= 0 && rebuild_on(d, b, rep, forced);
    int rowkey = -1;  // global index of the first cell of the atom's row: one value per (replica, row)
    float4 ri = make_float4(0.f, 0.f, 0.f, 0.f);
    L.cx = L.cy = L.cz = 0;
    L.mol = 0;
    if (act) {
      const RepBox &rb = repbox(b, rep);
      const int c = d.cell_of[L.i], lc = c - rb.cell_off;
      L.cx = lc % rb.nc[0];
      L.cy = (lc / rb.nc[0]) % rb.nc[1];
      L.cz = lc / (rb.nc[0] * rb.nc[1]);
      rowkey = c - L.cx;
      ri = d.rel[L.i];
      if (d.mol) L.mol = d.mol[L.i];
    }
    L.row = d.nbr + nbr_block_base(act ? L.i : 0, d.cap, d.tpa);
    int *selfpos = stage.self;
    L.selfpos = selfpos;
    const int win0 = win << 5;
    unsigned pending = __ballot_sync(FULL_MASK, act);
    while (pending) {
      const int leader = __ffs(pending) - 1;
      const int rk = __shfl_sync(FULL_MASK, rowkey, leader);
      const int cx0 = __shfl_sync(FULL_MASK, L.cx, leader);  // slots sort by cell: the leader's is the lowest
      const int grep = __shfl_sync(FULL_MASK, rep, leader);
      const unsigned mem = __ballot_sync(FULL_MASK, ((pending >> lane) & 1u) && rowkey == rk && L.cx - cx0 <= GROUP_SPAN);
      pending &= ~mem;
      if (group++ % split != mine) continue;
      L.me = (mem >> lane) & 1u;
      const RepBox &rb = repbox(b, grep);
      const int span = __reduce_max_sync(FULL_MASK, L.me ? L.cx - cx0 : 0);
      L.ci = L.me ? L.cx - cx0 : 0;
      const int cy = __shfl_sync(FULL_MASK, L.cy, leader), cz = __shfl_sync(FULL_MASK, L.cz, leader);
      // the atom in the group frame (origin: the group's first cell), and the group's box
      const float gx = ri.x + (float)L.ci * rb.wf[0], gy = ri.y, gz = ri.z;
      const float bxl = warp_minf(L.me ? gx : 1e30f), bxh = warp_maxf(L.me ? gx : -1e30f);
      const float byl = warp_minf(L.me ? gy : 1e30f), byh = warp_maxf(L.me ? gy : -1e30f);
      const float bzl = warp_minf(L.me ? gz : 1e30f), bzh = warp_maxf(L.me ? gz : -1e30f);
      L.rxx = pack2(gx);
      L.ryy = pack2(gy);
      L.rzz = pack2(gz);
      L.hi = L.me ? b.ce2_hi : -1.0f;
      L.cnt = 0;
      // candidate cells, nu in each of the 9 rows r = (dy+1) + 3 (dz+1): x cell cx0 - 1 + u
      const int nu = span + 3;
      int q_first = SHARED ? PART_ROWS[part] * nu : 0, ncand = SHARED ? PART_ROWS[part + 1] * nu : 9 * nu;
      uint32_t *seg = SHARED && part > 0 ? share->hits[part - 1] : nullptr;
      bool parts = SHARED;
     again:
      int nst = 0;
      selfpos[lane] = -1;
      __syncwarp();
      for (int q0 = q_first; q0 < ncand; q0 += 32) {
        // lane q - q0: the candidate cell's first slot, count, image code, origin offset
        int kb = 0, kn = 0, ks = 0, kimg = 0;
        uint32_t kcode = 0u;
        float kox = 0.f, koy = 0.f, koz = 0.f;
        const int q = q0 + lane;
        if (q < ncand) {
          const int qr = q / nu, r = ROW_ORDER[qr], u = class_cell(cx0 - 1, nu, q - qr * nu);
          const int dy = r % 3 - 1, dz = r / 3 - 1;
          int nx = cx0 - 1 + u, ny = cy + dy, nz = cz + dz, sx = 0, sy = 0, sz = 0;
          if (nx < 0) { nx += rb.nc[0]; sx = -1; } else if (nx >= rb.nc[0]) { nx -= rb.nc[0]; sx = 1; }
          if (ny < 0) { ny += rb.nc[1]; sy = -1; } else if (ny >= rb.nc[1]) { ny -= rb.nc[1]; sy = 1; }
          if (nz < 0) { nz += rb.nc[2]; sz = -1; } else if (nz >= rb.nc[2]) { nz -= rb.nc[2]; sz = 1; }
          const int c2 = rb.cell_off + nx + rb.nc[0] * (ny + rb.nc[1] * nz);
          kb = d.cell_start[c2];
          kn = d.cell_start[c2 + 1] - kb;
          // mode 0: the image code; mode 1: x index + 3 x row (<= 7 + 24), from which a
          // member's stencil index follows by subtracting its own x index
          kimg = image_code(sx, sy, sz);
          kcode = (uint32_t)(MODE == 0 ? kimg : u + 3 * r) << CODE_SHIFT;
          ks = u | (r << 3);
          kox = (float)(u - 1) * rb.wf[0];
          koy = (float)dy * rb.wf[1];
          koz = (float)dz * rb.wf[2];
        }
        const int kend = min(32, ncand - q0);
        for (int k = 0; k < kend; ++k) {
          const int cn = __shfl_sync(FULL_MASK, kn, k);
          if (cn == 0) continue;
          const int jb = __shfl_sync(FULL_MASK, kb, k);
          const uint32_t code = __shfl_sync(FULL_MASK, kcode, k);
          const uint8_t sbyte = (uint8_t)__shfl_sync(FULL_MASK, ks, k);
          const bool zero_img = __shfl_sync(FULL_MASK, kimg, k) == CODE_ZERO;
          const float ox = __shfl_sync(FULL_MASK, kox, k), oy = __shfl_sync(FULL_MASK, koy, k),
                      oz = __shfl_sync(FULL_MASK, koz, k);
          for (int t0 = 0; t0 < cn; t0 += 32) {
            const int t = t0 + lane;
            bool keep = false;
            float X = 0.f, Y = 0.f, Z = 0.f;
            if (t < cn) {
              const float4 rj = d.rel[jb + t];
              X = rj.x + ox;
              Y = rj.y + oy;
              Z = rj.z + oz;
              // squared distance to the group's box; within the band's upper end: staged
              const float ex = fmaxf(fmaxf(bxl - X, X - bxh), 0.f), ey = fmaxf(fmaxf(byl - Y, Y - byh), 0.f),
                          ez = fmaxf(fmaxf(bzl - Z, Z - bzh), 0.f);
              keep = fmaf(ez, ez, fmaf(ey, ey, ex * ex)) <= b.ce2_hi;
            }
            const unsigned km = __ballot_sync(FULL_MASK, keep);
            if (keep) {
              const int s = nst + __popc(km & lt_mask);
              const int e = (s >> 1) * 4 + (s & 1);
              fxy[e] = X;
              fxy[e + 2] = Y;
              fz[s] = Z;
              sw[s] = (uint32_t)(jb + t) | code;
              su[s] = sbyte;
              // a window atom at its own cell and zero image: that lane's self position
              const unsigned l = (unsigned)(jb + t - win0);
              if (zero_img && l < 32u) selfpos[l] = s;
            }
            nst += __popc(km);
            if (nst > BUILD_STAGE - 32) {
              __syncwarp();
              build_sweep<MODE>(d, b, rb, nst, sxy, sz, sw, su, L, cshift, by_mol, seg);
              selfpos[lane] = -1;
              __syncwarp();
              nst = 0;
            }
          }
        }
      }
      if (nst > 0) {
        __syncwarp();
        build_sweep<MODE>(d, b, rb, nst, sxy, sz, sw, su, L, cshift, by_mol, seg);
      }
      if (parts) {
        share->cnt[part][lane] = L.cnt;
        __syncthreads();
        int before = 0, total = 0;
        bool fits = true;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int n = share->cnt[p][lane];
          if (p < part) before += n;
          total += n;
          fits = fits && (p == 0 || n <= SEG_HITS);
        }
        if (__syncthreads_and(fits)) {
          if (L.me && part > 0)
            for (int k = 0; k < L.cnt; ++k)
              if (before + k < d.cap) L.row[(((before + k) >> 2) << cshift) + ((before + k) & 3)] = seg[k * 32 + lane];
          L.cnt = total;
        } else {  // warp 0 takes all candidates, straight to the rows
          parts = false;
          seg = nullptr;
          q_first = 0;
          ncand = part == 0 ? 9 * nu : 0;
          L.cnt = 0;
          goto again;
        }
      }
      if (SHARED) __syncthreads();  // the counts are overwritten next
      if (L.me && part == 0) {
        d.nnbr[L.i] = min(L.cnt, d.cap);
        if (L.cnt > d.cap) atomicMax(&d.flags[F_OVERFLOW], L.cnt);
        wmax = max(wmax, L.cnt);
      }
    }
  }
  // one atomic per warp for the largest list length (not one per atom)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) wmax = max(wmax, __shfl_xor_sync(FULL_MASK, wmax, o));
  if (lane == 0 && wmax > 0) atomicMax(&d.flags[F_MAXNB], wmax);
}

}  // namespace cav
