// mcx_packed.cuh -- the update of a same-colour site pair in packed FP32
// arithmetic (two FP32 operations per instruction: fma / mul / add.rn.f32x2,
// sm_100 and later).  Site A of the pair is the low half of every 64-bit
// value, site B the high half.
//
// What bounds the plain pass is the instruction issue rate and the latency it
// leaves exposed, not DRAM (LL 128^3: 0.44 instructions per cycle and
// scheduler over the whole pass).  A pair's two sites run the same FP32 chain
// on different numbers, and the director rows hold them next to each other,
// so the bond sums, the rotation and the energy change take half the
// instructions.  Measured per pass, scalar -> packed: LL 128^3 10.0 -> 8.95 us
// (autotuned shape), 16 x LL 96^3 59.3 -> 55.8 us, 48 GHRL slabs of 16^3 to
// 64^3 35.2 -> 26.4 us, 8 droplets of 96^3 67.3 -> 61.4 us.
//
// Each half of a packed operation is rounded as the scalar operation (round to
// nearest even, denormals kept), so with the operations of site_update
// (mcx_pass.cuh) in their order the results are the same bits; the direct pass
// keeps the scalar form and the tests compare the two bit for
// bit.
#pragma once
#include <cuda_runtime.h>

#include "mcx_pass.cuh"

namespace mcx {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f32x2 pk(const float2 &v) { return pk(v.x, v.y); }
__device__ __forceinline__ f32x2 pk1(float v) { return pk(v, v); }
__device__ __forceinline__ float2 unpk(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a - b (a + b * -1 is rounded once, like the subtraction)
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, pk1(-1.f), a); }
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }

// Three components of a pair.
struct V2 {
  f32x2 x, y, z;
};

__device__ __forceinline__ f32x2 dot2(const V2 &a, const V2 &b) {
  return fma2(a.z, b.z, fma2(a.y, b.y, mul2(a.x, b.x)));
}

template <int AXIS>
__device__ __forceinline__ f32x2 axis_of(const V2 &v) {
  return AXIS == 0 ? v.x : (AXIS == 1 ? v.y : v.z);
}

// Couplings of the pair potential, both halves alike.
template <int POT>
struct PairConst {
  f32x2 ga, gb, gc, mu;      // GHRL
  float sigma;               // GHRL, chiral
  f32x2 mA, mB1, mC, one;    // Pear: -A, -B1, -C/4
  __device__ __forceinline__ explicit PairConst(const RepDev &R) {
    if (POT == POT_GHRL) {
      ga = pk1(R.ga);
      gb = pk1(R.gb);
      gc = pk1(R.gc);
      mu = pk1(R.mu);
      sigma = R.sigma;
    } else if (POT == POT_PEAR) {
      mA = pk1(-R.A);
      mB1 = pk1(-R.B1);
      mC = pk1(-0.25f * R.C);
    }
  }
};

// Per-director terms that the six bonds of one evaluation share.
template <int POT>
struct DirTerms {
  V2 n;
  V2 h;  // GHRL: 1.5 n
  V2 m;  // GHRL, chiral: -n
  __device__ __forceinline__ DirTerms(const V2 &d, bool chiral) {
    n = d;
    if (POT == POT_GHRL) {
      const f32x2 c = pk1(1.5f);
      h.x = mul2(c, d.x);
      h.y = mul2(c, d.y);
      h.z = mul2(c, d.z);
      if (chiral) {
        m.x = neg2(d.x);
        m.y = neg2(d.y);
        m.z = neg2(d.z);
      }
    }
  }
};

// The chiral part of the GHRL bond, added to v: sigma * (n.n' > 0 ? cr : -cr),
// cr the reference's cross-product component along the bond with the bond's
// sign (cross_ref_rn).  The sign goes to sigma: the sign bit of n.n' minus the
// smallest denormal is set exactly where n.n' > 0 does not hold.
template <int D>
__device__ __forceinline__ f32x2 add_chiral(float sigma, const V2 &n, const V2 &m, const V2 &b, f32x2 nij, f32x2 v) {
  constexpr int X = D >> 1;
  f32x2 cr;
  if (D & 1) {  // -(p q - r s) = (-p) q + r s
    if (X == 0) cr = fma2(m.z, b.y, mul2(n.y, b.z));
    else if (X == 1) cr = fma2(m.x, b.z, mul2(n.z, b.x));
    else cr = fma2(m.y, b.x, mul2(n.x, b.y));
  } else {
    if (X == 0) cr = fma2(n.z, b.y, mul2(m.y, b.z));
    else if (X == 1) cr = fma2(n.x, b.z, mul2(m.z, b.x));
    else cr = fma2(n.y, b.x, mul2(m.x, b.y));
  }
  const float2 t = unpk(add2(nij, pk1(-1.401298464324817e-45f)));
  const uint32_t s = __float_as_uint(sigma);
  const f32x2 sg = pk(__uint_as_float(s ^ (__float_as_uint(t.x) & 0x80000000u)),
                      __uint_as_float(s ^ (__float_as_uint(t.y) & 0x80000000u)));
  return fma2(sg, cr, v);
}

// Slot D's bond (bond<POT, D>) of the old and of the new directors, added to
// the running sums eo and en with weight w (W: some weights are not 1; they
// are 0 or 1), and with X to xo and xn with weight x (a measured masked pass:
// bonds to inactive neighbours).
template <int POT, int D, bool W, bool X_>
__device__ __forceinline__ void add_bonds(const PairConst<POT> &K, bool chiral, const DirTerms<POT> &o,
                                          const DirTerms<POT> &n, const V2 &b, f32x2 w, f32x2 &eo, f32x2 &en, f32x2 x,
                                          f32x2 &xo, f32x2 &xn) {
  constexpr int X = D >> 1;
  f32x2 no = dot2(o.n, b), nn = dot2(n.n, b);
  f32x2 vo, vn;
  if (POT == POT_LL) {
    if (D == 0 && !W) {
      eo = mul2(no, no);
      en = mul2(nn, nn);
    } else if (D == 0) {
      eo = mul2(mul2(no, w), no);
      en = mul2(mul2(nn, w), nn);
    } else {
      eo = fma2(W ? mul2(no, w) : no, no, eo);
      en = fma2(W ? mul2(nn, w) : nn, nn, en);
    }
    if (X_) {
      xo = D == 0 ? mul2(mul2(no, x), no) : fma2(mul2(no, x), no, xo);
      xn = D == 0 ? mul2(mul2(nn, x), nn) : fma2(mul2(nn, x), nn, xn);
    }
    return;
  } else if (POT == POT_PEAR) {
    const f32x2 bj = axis_of<X>(b), one = pk1(1.f), two = pk1(2.f);
    const f32x2 d_o = (D & 1) ? sub2(axis_of<X>(o.n), bj) : sub2(bj, axis_of<X>(o.n));
    const f32x2 d_n = (D & 1) ? sub2(axis_of<X>(n.n), bj) : sub2(bj, axis_of<X>(n.n));
    const f32x2 so = mul2(fma2(no, add2(no, two), one), d_o);
    const f32x2 sn = mul2(fma2(nn, add2(nn, two), one), d_n);
    vo = fma2(K.mA, mul2(no, no), fma2(K.mB1, no, mul2(K.mC, so)));
    vn = fma2(K.mA, mul2(nn, nn), fma2(K.mB1, nn, mul2(K.mC, sn)));
  } else {
    // the neighbour-only terms serve both directors
    const f32x2 bj = axis_of<X>(b);
    const f32x2 t = fma2(mul2(pk1(1.5f), bj), bj, pk1(-1.f)), mj = mul2(K.mu, bj);
    const f32x2 qo = mul2(no, no), qn = mul2(nn, nn);
    vo = fma2(fma2(axis_of<X>(o.h), axis_of<X>(o.n), t), fma2(K.ga, qo, K.gb),
              fma2(K.gc, qo, mul2(mj, mul2(axis_of<X>(o.n), no))));
    vn = fma2(fma2(axis_of<X>(n.h), axis_of<X>(n.n), t), fma2(K.ga, qn, K.gb),
              fma2(K.gc, qn, mul2(mj, mul2(axis_of<X>(n.n), nn))));
    if (chiral) {
      vo = add_chiral<D>(K.sigma, o.n, o.m, b, no, vo);
      vn = add_chiral<D>(K.sigma, n.n, n.m, b, nn, vn);
    }
  }
  if (D == 0) {
    eo = W ? mul2(w, vo) : vo;
    en = W ? mul2(w, vn) : vn;
  } else {
    eo = W ? fma2(w, vo, eo) : add2(vo, eo);
    en = W ? fma2(w, vn, en) : add2(vn, en);
  }
  if (X_) {
    xo = D == 0 ? mul2(x, vo) : fma2(x, vo, xo);
    xn = D == 0 ? mul2(x, vn) : fma2(x, vn, xn);
  }
}

// Bond sums of the old and the new directors over the six slots (X: also with
// the weights x, into xo and xn).
template <int POT, bool W, bool X>
__device__ __forceinline__ void bond_sums_c(const RepDev &R, bool chiral, const V2 &o, const V2 &n, const V2 nb[6],
                                            const f32x2 w[6], f32x2 &eo, f32x2 &en, const f32x2 x[6], f32x2 &xo,
                                            f32x2 &xn) {
  const PairConst<POT> K(R);
  const DirTerms<POT> O(o, chiral), N(n, chiral);
  add_bonds<POT, 0, W, X>(K, chiral, O, N, nb[0], w[0], eo, en, x[0], xo, xn);
  add_bonds<POT, 1, W, X>(K, chiral, O, N, nb[1], w[1], eo, en, x[1], xo, xn);
  add_bonds<POT, 2, W, X>(K, chiral, O, N, nb[2], w[2], eo, en, x[2], xo, xn);
  add_bonds<POT, 3, W, X>(K, chiral, O, N, nb[3], w[3], eo, en, x[3], xo, xn);
  add_bonds<POT, 4, W, X>(K, chiral, O, N, nb[4], w[4], eo, en, x[4], xo, xn);
  add_bonds<POT, 5, W, X>(K, chiral, O, N, nb[5], w[5], eo, en, x[5], xo, xn);
}

template <int POT, bool W, bool X>
__device__ __forceinline__ void bond_sums(const RepDev &R, const V2 &o, const V2 &n, const V2 nb[6], const f32x2 w[6],
                                          f32x2 &eo, f32x2 &en, const f32x2 x[6], f32x2 &xo, f32x2 &xn) {
  // uniform: a CTA serves one replica
  if (POT == POT_GHRL && R.sigma != 0.f) bond_sums_c<POT, W, X>(R, true, o, n, nb, w, eo, en, x, xo, xn);
  else bond_sums_c<POT, W, X>(R, false, o, n, nb, w, eo, en, x, xo, xn);
}

// The constant the GHRL bond leaves out (ghrl_bond_var), per weighted bond.
template <int POT, bool W>
__device__ __forceinline__ f32x2 add_bond_const(const RepDev &R, const f32x2 w[6], f32x2 e) {
  if (POT != POT_GHRL) return e;
  if (!W) return fma2(pk1(R.gconst), pk1(6.f), e);
  return fma2(pk1(R.gconst), add2(add2(add2(w[0], w[1]), add2(w[2], w[3])), add2(w[4], w[5])), e);
}

// The pair's uniforms (pair_uniforms) as the packed update uses them: f0 and
// f2 hold 1 + u0 and 1 + u2 (21 bits below a set exponent: exact, no integer
// conversion), ax the rotation axis from u1.
constexpr uint32_t kAxisX = 698352u, kAxisY = 1396704u;  // u1 < 0.333f, u1 < 0.666f as 21-bit integers
static_assert((double)(kAxisX - 1) < (double)0.333f * 2097152.0 && (double)kAxisX >= (double)0.333f * 2097152.0, "");
static_assert((double)(kAxisY - 1) < (double)0.666f * 2097152.0 && (double)kAxisY >= (double)0.666f * 2097152.0, "");

__device__ __forceinline__ float one_plus(uint32_t u21_shl2) { return __uint_as_float(u21_shl2 | 0x3F800000u); }

// Rotates both directors (propose): by pi va about the axis each site drew.
// The multiply-add fusions are the ones the compiler gives propose().
__device__ __forceinline__ V2 propose2(const V2 &n, const uint4 &w, float ang) {
  const f32x2 f0 = pk(one_plus((w.x >> 9) & 0x7FFFFCu), one_plus((w.w >> 9) & 0x7FFFFCu));
  // 2 u0 - 1 = 2 f0 - 3 exactly
  const f32x2 th2 = mul2(pk1(3.14159265358979f), mul2(fma2(pk1(2.f), f0, pk1(-3.f)), pk1(ang)));
  const float2 th = unpk(th2);
  const float aA = fabsf(th.x), aB = fabsf(th.y);
  const f32x2 sn = pk(copysignf(__sinf(aA), th.x), copysignf(__sinf(aB), th.y));
  const f32x2 cs = pk(__cosf(aA), __cosf(aB));
  const uint32_t b1 = ((w.x & 0x7FFu) << 10) | (w.y & 0x3FFu);
  const bool xA = w.y < (kAxisX << 11), yA = w.y < (kAxisY << 11);
  const bool xB = b1 < kAxisX, yB = b1 < kAxisY;
  const float2 x = unpk(n.x), y = unpk(n.y), z = unpk(n.z);
  const f32x2 u = pk(xA ? y.x : (yA ? z.x : x.x), xB ? y.y : (yB ? z.y : x.y));
  const f32x2 v = pk(xA ? z.x : (yA ? x.x : y.x), xB ? z.y : (yB ? x.y : y.y));
  const float2 up = unpk(fma2(u, cs, mul2(v, sn)));
  const float2 vp = unpk(fma2(v, cs, neg2(mul2(u, sn))));
  V2 p;
  p.x = pk(xA ? x.x : (yA ? vp.x : up.x), xB ? x.y : (yB ? vp.y : up.y));
  p.y = pk(xA ? up.x : (yA ? y.x : vp.x), xB ? up.y : (yB ? y.y : vp.y));
  p.z = pk(xA ? vp.x : (yA ? up.x : z.x), xB ? vp.y : (yB ? up.y : z.y));
  const float2 n2 = unpk(fma2(p.z, p.z, fma2(p.y, p.y, mul2(p.x, p.x))));
  const f32x2 inv = pk(rsqrtf(n2.x), rsqrtf(n2.y));
  p.x = mul2(p.x, inv);
  p.y = mul2(p.y, inv);
  p.z = mul2(p.z, inv);
  return p;
}

// u2 of both sites.
__device__ __forceinline__ float2 accept_uniforms(const uint4 &w) {
  const uint32_t a = (w.z >> 9) & 0x7FFFFCu, b = ((w.z & 0x7FFu) << 12) | ((w.w & 0x3FFu) << 2);
  return unpk(add2(pk(one_plus(a), one_plus(b)), pk1(-1.f)));
}

// Sums of a measured pass (kQ quantities) over a thread's pairs, in the scalar
// update's order: site A's terms, then site B's, one FP32 addition each (a
// packed accumulator per quantity would save some additions and give other last
// bits, which the statistics of lattices of some hundred sites show in their
// ninth digit).  MASKED: the energy of active sites is a sum of its own.
template <bool MASKED>
struct PairSums {
  static constexpr bool kMasked = MASKED;
  float v[kQ];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < kQ; q++) v[q] = 0.f;
  }
  __device__ __forceinline__ void site_q(float x, float y, float z, float xm, float ym, float zm) {
    v[2] = fmaf(xm, x, v[2]);
    v[3] = fmaf(xm, y, v[3]);
    v[4] = fmaf(xm, z, v[4]);
    v[5] = fmaf(ym, y, v[5]);
    v[6] = fmaf(zm, y, v[6]);
  }
  // Q-tensor products of a pair; nm: its directors, zero for a site that does not count
  __device__ __forceinline__ void tensor(const V2 &n, const V2 &nm) {
    const float2 x = unpk(n.x), y = unpk(n.y), z = unpk(n.z), xm = unpk(nm.x), ym = unpk(nm.y), zm = unpk(nm.z);
    site_q(x.x, y.x, z.x, xm.x, ym.x, zm.x);
    site_q(x.y, y.y, z.y, xm.y, ym.y, zm.y);
  }
  // energies: anchoring s, field (all sites f0, active ones f1), bonds (b0, b1)
  // and bonds to inactive sites x
  template <bool MASK, bool FIELD>
  __device__ __forceinline__ void energy(int c, f32x2 s, f32x2 f0, f32x2 f1, f32x2 b0, f32x2 b1, f32x2 x) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      auto of = [&](f32x2 t) { return h ? unpk(t).y : unpk(t).x; };
      if (MASK) v[0] += of(s);
      if (FIELD) v[0] += of(f0);
      if (c == 1) {
        v[0] += of(b0);
        if (MASK) v[0] += of(x);
      }
      if (MASKED) {
        if (MASK) v[1] += of(s);
        if (FIELD) v[1] += of(f1);
        if (c == 1) v[1] += of(b1);
      }
    }
  }
  __device__ __forceinline__ void fold(float out[kQ]) const {
#pragma unroll
    for (int q = 0; q < kQ; q++) out[q] = v[q];
  }
};

// A thread's sums over a chunk of many planes: every kLongPlanes the FP32 sums so
// far move into high and low parts, and the warp's and the CTA's
// sums keep both parts.  Chunks of the default shape are up to a whole lattice
// deep and 256 threads wide: with FP32 sums alone the energy of a sweep of 16 x
// LL 96^3 (46 planes to a chunk, 19 CTAs to a replica) was 1.3e-8 of itself off
// (rms), and 7e-9 on 8 x 64^3, against 2.2e-9 and 3.1e-9 in 128 threads x 8 planes;
// so 4e-10.  Chunks of at most 128 threads x 8 planes keep the plain sums.
// They lie in shared memory: stores to local or global memory would make the
// compiler read the replica's constants again after them.
constexpr int kLongPlanes = 8;
template <bool USED, int NT>
struct LongSums {
  float (*part)[NT];  // [2 kQ][NT]
  bool on;
  __device__ __forceinline__ LongSums(float (*p)[NT], bool deep) : part(p), on(USED && deep) {
    if (!on) return;
#pragma unroll
    for (int q = 0; q < 2 * kQ; q++) part[q][threadIdx.x] = 0.f;
  }
  // before plane `done` of the chunk
  template <class Q>
  __device__ __forceinline__ void plane(int done, Q &sums) {
    if (!USED || done == 0 || done % kLongPlanes != 0) return;
#pragma unroll
    for (int q = 0; q < kQ; q++) {
      float h = part[q][threadIdx.x], l = part[kQ + q][threadIdx.x];
      add_split(h, l, sums.v[q], 0.f);
      part[q][threadIdx.x] = h;
      part[kQ + q][threadIdx.x] = l;
    }
    sums.clear();
  }
  // after the last plane: all of the sums
  template <class Q>
  __device__ __forceinline__ void fold(const Q &sums, float qs[kQ], float low[kQ]) {
    sums.fold(qs);
    if (!on) return;
#pragma unroll
    for (int q = 0; q < kQ; q++) {
      const float v = qs[q];
      qs[q] = part[q][threadIdx.x];
      low[q] = part[kQ + q][threadIdx.x];
      add_split(qs[q], low[q], v, 0.f);
    }
  }
};

__device__ __forceinline__ V2 mul2(const V2 &n, f32x2 m) { return {mul2(n.x, m), mul2(n.y, m), mul2(n.z, m)}; }

// Electric term of both sites (field_energy).
__device__ __forceinline__ f32x2 field_energy2(const RepDev &R, const V2 &n) {
  const V2 e = {pk1(R.ex), pk1(R.ey), pk1(R.ez)};
  const f32x2 d = mul2(pk1(R.elecE), dot2(n, e));
  return mul2(mul2(pk1(-R.elecA), d), d);
}

__device__ __forceinline__ f32x2 pick2(bool a, bool b, f32x2 yes, f32x2 no) {
  const float2 y = unpk(yes), n = unpk(no);
  return pk(a ? y.x : n.x, b ? y.y : n.y);
}

}  // namespace mcx
