// cav_mixed.cuh -- the mixed form's pair arithmetic and the walk of a lane through its
// part of an atom's list row (cav_force.cu, cav_chunk.cu).
#pragma once

#include "cav_pair.cuh"

namespace cav {

// Single-type systems keep the pair constants in registers (no table lookups).
struct OneType {
  float rc2, sig2, eps4, gc, pk;
};

// FP32 reciprocal from the hardware approximation (PTX rcp.approx.ftz.f32): one
// instruction instead of the correctly rounded sequence; it is a function of r^2
// alone, so both orders of a pair still see the same value.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two FP32 values in one 64-bit register for the packed FP32x2 arithmetic of sm_100+
// (add/sub/mul/fma .rn.f32x2: each half rounded exactly as the scalar instruction).
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unf2(F2 x, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// A list chunk: read once per step and larger than L1, so it is not allocated in L1
// (which keeps the neighbour coordinates the gathers reuse).
template <bool COH>
__device__ __forceinline__ uint4 ld_list(const uint4 *p) {
  uint4 v;
  if constexpr (COH)
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
  else
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p));
  return v;
}

// One pair evaluation of the mixed form, two list entries at a time in packed FP32x2
// arithmetic: sums of the even and of the odd entries of a lane's chunks.
struct PairSums {
  F2 ax, ay, az, vr, pp;  // vr: sum of +coef r^2
};

// Displacement r_j - r_i: the integer difference is exact, its conversion to FP32 and
// the product with the unit (an FP32 pair hi + lo) round once each.  The small product comes
// first, f hi + (f lo): the other way round f hi is rounded and f lo, no more than half an ulp
// of it, mostly lost, which leaves all distances of a system with one scale error of up to
// 2^-25 (virial of 4,000 atoms off by 2.9e-6, now 5e-8).  All of it is odd in the difference,
// so d_ji = -d_ij bit for bit and the FP32 pair forces obey Newton's third law exactly (each
// half of a packed operation rounds as the scalar one).
__device__ __forceinline__ F2 displacement2(int ja, int jb, int i, float hi, float lo) {
  const F2 f = f2((float)fixed_diff(ja, i), (float)fixed_diff(jb, i));
  return fma2(f, f2(hi, hi), mul2(f, f2(lo, lo)));
}

template <bool EV, bool ONE>
__device__ __forceinline__ void mixed_pair2(const int4 &ja, const int4 &jb, bool va, bool vb, const int4 &ri, int nt,
                                            const SmemTabF &tab, const OneType &c1, const float4 &uh,
                                            const float4 &ul, float jtol, PairSums &S) {
  const F2 dx = displacement2(ja.x, jb.x, ri.x, uh.x, ul.x), dy = displacement2(ja.y, jb.y, ri.y, uh.y, ul.y),
           dz = displacement2(ja.z, jb.z, ri.z, uh.z, ul.z);
  const F2 r2d = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
  float r2a, r2b;
  unf2(r2d, r2a, r2b);
  float rc2a, rc2b, sg2a, sg2b, e4a, e4b, gca, gcb, pka, pkb;
  if (ONE) {
    rc2a = rc2b = c1.rc2; sg2a = sg2b = c1.sig2; e4a = e4b = c1.eps4; gca = gcb = c1.gc; pka = pkb = c1.pk;
  } else {
    const int ta = ri.w * nt + ja.w, tb = ri.w * nt + jb.w;
    const float4 pa = tab.c4[ta], pb = tab.c4[tb];
    rc2a = pa.x; sg2a = pa.y; e4a = pa.z; gca = pa.w;
    rc2b = pb.x; sg2b = pb.y; e4b = pb.z; gcb = pb.w;
    pka = EV ? tab.pk[ta] : 0.0f;
    pkb = EV ? tab.pk[tb] : 0.0f;
  }
  const bool ina = va && r2a <= rc2a, inb = vb && r2b <= rc2b;
  if (!(ina || inb)) return;
  const float r2ca = fmaxf(r2a, jtol), r2cb = fmaxf(r2b, jtol);  // Lj jump_fix floor (0 when off)
  const F2 r2 = f2(r2ca, r2cb), r2i = f2(rcp_approx(r2ca), rcp_approx(r2cb));
  const F2 eps4 = f2(e4a, e4b);
  const F2 s2 = mul2(f2(sg2a, sg2b), r2i);
  const F2 s6 = mul2(mul2(s2, s2), s2);
  const F2 w = mul2(mul2(eps4, r2i), s6);
  F2 coef = fma2(w, fma2(f2(-12.0f, -12.0f), s6, f2(6.0f, 6.0f)), f2(-gca, -gcb));
  float ca, cb;
  unf2(coef, ca, cb);
  coef = f2(ina ? ca : 0.0f, inb ? cb : 0.0f);
  S.ax = fma2(coef, dx, S.ax);
  S.ay = fma2(coef, dy, S.ay);
  S.az = fma2(coef, dz, S.az);
  if (EV) {
    S.vr = fma2(coef, r2, S.vr);
    const F2 pe = fma2(mul2(eps4, s6), sub2(s6, f2(1.0f, 1.0f)), fma2(f2(-0.5f * gca, -0.5f * gcb), r2, f2(pka, pkb)));
    float pa, pb;
    unf2(pe, pa, pb);
    S.pp = add2(S.pp, f2(ina ? pa : 0.0f, inb ? pb : 0.0f));
  }
}

// Mixed-form pair loop of one lane: list chunks t, t+TPA, ... of atom i (four words
// per 128-bit load; the next chunk's load and four neighbour coordinates in
// flight); `gather(word)` returns the neighbour's int4 (global memory or a
// shared-memory stage).  Whole chunks run without tests of the entry number; the
// row's last, partial chunk follows, its missing entries stood in for by the first.
// What bounds it: the gathers (16 bytes per lane from some 10 lines: the LSU data path is
// busy 71% of the time) and their latency.  Against coordinates relative to each atom's
// cell, whose offsets had to be decoded from the list words and added (and lists in
// stencil order), the loop issues 99 M instead of 135 M instructions on the 1,048,576-atom
// fluid and a launch takes 160 us instead of 186 (one lane per atom); half or a quarter
// of the gathers through the texture path: 174 and 192 us; 40 or 48 warps per SM (48 and
// 40 registers): 240 and 320 us, the loop spills.
// Sums: a lane holds its even and its odd entries in one FP32 sum each.  One lane per atom
// thus has two sums of ~38 entries where four lanes have eight of ~10, whose pairs meet in
// FP64: force error 5.51e-7 and 5.45e-7 of the rms at 256,000 atoms (1.31e-6 on four lanes with
// cell-relative coordinates).  The two are joined in FP32 (in FP64: 5.50e-7, and 1.6% more
// time per step with one lane, 10% with four), virial and energy in FP64.
// ONE: single-type system, pair constants in registers; otherwise from the
// shared-memory table.
template <int TPA, bool EV, bool ONE, bool COH, class Gather>
__device__ __forceinline__ void mixed_pairs(const uint4 *row4, int nn, int t, const int4 ri, int nt,
                                            const SmemTabF &tab, const OneType c1, const float4 uh,
                                            const float4 ul, const float jtol, Gather gather, float &ax,
                                            float &ay, float &az, double &vr, double &pp) {
  PairSums S;
  S.ax = S.ay = S.az = S.vr = S.pp = f2(0.f, 0.f);
  const int nfull = nn >> 2;
  uint4 nxt = 4 * t < nn ? ld_list<COH>(row4) : make_uint4(0, 0, 0, 0);
  int g = t;
  for (; g < nfull; g += TPA) {
    const uint4 w4 = nxt;
    row4 += 32;
    if (4 * (g + TPA) < nn) nxt = ld_list<COH>(row4);  // the next list chunk in flight
    const int4 j0 = gather(w4.x), j1 = gather(w4.y), j2 = gather(w4.z), j3 = gather(w4.w);
    mixed_pair2<EV, ONE>(j0, j1, true, true, ri, nt, tab, c1, uh, ul, jtol, S);
    mixed_pair2<EV, ONE>(j2, j3, true, true, ri, nt, tab, c1, uh, ul, jtol, S);
  }
  const int rest = nn & 3;
  if (g == nfull && rest) {
    const int4 j0 = gather(nxt.x), j1 = rest > 1 ? gather(nxt.y) : j0;
    mixed_pair2<EV, ONE>(j0, j1, true, rest > 1, ri, nt, tab, c1, uh, ul, jtol, S);
    if (rest > 2) {
      const int4 j2 = gather(nxt.z);
      mixed_pair2<EV, ONE>(j2, j2, true, false, ri, nt, tab, c1, uh, ul, jtol, S);
    }
  }
  float lo, hi;
  unf2(S.ax, lo, hi); ax += lo + hi;
  unf2(S.ay, lo, hi); ay += lo + hi;
  unf2(S.az, lo, hi); az += lo + hi;
  if (EV) {
    unf2(S.vr, lo, hi); vr = -((double)lo + (double)hi);
    unf2(S.pp, lo, hi); pp = (double)lo + (double)hi;
  }
}

__device__ inline OneType one_type(const SmemTabF &tab) {
  return OneType{tab.rc2[0], tab.sig2[0], tab.eps4[0], tab.gc[0], tab.pk[0]};
}

}  // namespace cav
