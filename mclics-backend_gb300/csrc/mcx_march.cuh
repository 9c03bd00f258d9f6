// mcx_march.cuh -- the per-thread state of the z-march passes (the plain
// pass in mcx_march.cu, the learned one in mcx_lmarch.cu): a thread owns one
// same-colour site pair of a row and marches it through a chunk of planes.
#pragma once
#include <cuda_runtime.h>

#include "mcx_packed.cuh"
#include "mcx_pass.cuh"

namespace mcx {

// Opposite-colour director loads of the z-march passes: L2 loads
// (ld.global.cg).  A pass starts under programmatic dependent launch while
// the previous pass, which writes these directors, drains; after
// griddepcontrol.wait, read-only-path loads (__ldg) were seen to return lines
// that an SM's L1 still held from before the previous pass's writes (the
// chain then differed from a launch-by-launch run), while L2 loads always
// see them.
#ifdef MCX_OPP_L1
__device__ __forceinline__ float2 ldo2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float ldo1(const float *p) { return *p; }
#else
__device__ __forceinline__ float2 ldo2(const float *p) { return __ldcg(reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ float ldo1(const float *p) { return __ldcg(p); }
#endif

// Programmatic dependent launch: wait until the preceding grid on the stream
// has completed and its memory is visible (returns at once when the launch
// had no programmatic dependency), and let the following grid be scheduled.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// What a measured pass adds for the opposite pair of an unmasked lattice: its
// Q-tensor products and field energy (its bonds are the own sites').
template <bool FIELD, bool PER, class Q>
__device__ __forceinline__ void measure_opposite(const RepDev &R, const float2 &x, const float2 &y, const float2 &z,
                                                 bool hasB, Q &sums) {
  const V2 n = {pk(x), pk(y), pk(z)};
  const f32x2 m = pk(1.f, hasB ? 1.f : 0.f);
  sums.tensor(n, PER ? n : mul2(n, m));
  if (FIELD) {
    f32x2 ef = field_energy2(R, n);
    if (!PER) ef = mul2(ef, m);
    sums.template energy<false, true>(0, 0ull, ef, ef, 0ull, 0ull, 0ull);
  }
}

// Opposite-colour pair of one row: 3 components (and point types).
struct OPair {
  float2 v[3];
  uint16_t pt;
};

// Per-thread state of the march.  Offsets are float offsets within a
// (colour, component) plane; the three component planes of a colour are
// reached through three base pointers.
struct March {
  float *A0, *A1, *A2;              // own colour, components x y z
  const float *O0, *O1, *O2;        // opposite colour
  const uint8_t *PA, *PO;           // point types of the two colours (MASK)
  int off, offp;                    // this plane's pair: row * hs + h0, row * hps + h0
  int dz, dzp;                      // one plane further: ny * hs, ny * hps
  int dyp, dym, dypp, dymp;         // rows y+1, y-1 relative to the pair's row
  int dx0, dx1;                     // the extra x neighbour for s = 0, 1
  uint32_t pid, dpid;               // Philox pair counter and its step per plane
  int s;                            // parity of the own sites in this plane
  int h0, row;                      // half-row index of site A; row j + ny * k of this plane
  bool hasB;
  uint8_t tail;                     // odd nx: 1 / 2 when site A / B sits in the row's last slot (0 otherwise)
  float ee0, ee1, eyp, eym;         // bond present: extra x (s = 0, 1), y+1, y-1
};

// griddepcontrol.wait for a march whose director pointers are in m.  The
// pointers pass through the asm as operands, so every director address is
// computed from values that exist only after the wait, and no load through
// them can be scheduled above it, whatever its cache path.
__device__ __forceinline__ void grid_dependency_wait(March &m) {
  asm volatile("griddepcontrol.wait;"
               : "+l"(m.A0), "+l"(m.A1), "+l"(m.A2), "+l"(m.O0), "+l"(m.O1), "+l"(m.O2)
               :
               : "memory");
}

// A unit without an active site in or next to it (kUnitDead) of an engine whose
// passes add inactive sites' field energy themselves (PassArgs::idle_in_pass).
template <bool FIELD, int MODE, class Q>
__device__ __forceinline__ void dead_unit(const RepDev &R, March &m, int kb, int ke, Q &sums) {
  if (!(FIELD && MODE == MODE_SWEEP_MEASURE)) return;
  int s = m.s;
#pragma unroll 1
  for (int k = kb; k < ke; k++) {
    const V2 n = {pk(*reinterpret_cast<const float2 *>(m.A0 + m.off)), pk(*reinterpret_cast<const float2 *>(m.A1 + m.off)),
                  pk(*reinterpret_cast<const float2 *>(m.A2 + m.off))};
    const bool hereA = !(s && m.tail == 1), hereB = m.hasB && !(s && m.tail == 2);
    const f32x2 f = mul2(field_energy2(R, n), pk(hereA ? 1.f : 0.f, hereB ? 1.f : 0.f));
    sums.template energy<false, true>(0, 0ull, f, 0ull, 0ull, 0ull, 0ull);
    m.off += m.dz;
    s ^= 1;
  }
}

template <bool MASK>
__device__ __forceinline__ void load_opair_at(const March &m, int off, int offp, bool on, OPair &o) {
  if (on) {
    o.v[0] = ldo2(m.O0 + off);
    o.v[1] = ldo2(m.O1 + off);
    o.v[2] = ldo2(m.O2 + off);
    if (MASK) o.pt = __ldg(reinterpret_cast<const uint16_t *>(m.PO + offp));
  } else {
    o.v[0] = o.v[1] = o.v[2] = make_float2(0.f, 0.f);
    if (MASK) o.pt = 0;
  }
}

// The constants an unmasked update reads, in registers.  A pass whose loop
// holds barriers or asynchronous copies reads global constants again after
// each of them (their memory clobbers), a load of some hundred cycles per
// plane.
__device__ __forceinline__ RepDev local_constants(const RepDev &R) {
  RepDev c;
  c.A = R.A;
  c.ga = R.ga;
  c.gb = R.gb;
  c.gc = R.gc;
  c.mu = R.mu;
  c.sigma = R.sigma;
  c.gconst = R.gconst;
  c.B1 = R.B1;
  c.C = R.C;
  c.elecA = R.elecA;
  c.elecE = R.elecE;
  c.ex = R.ex;
  c.ey = R.ey;
  c.ez = R.ez;
  return c;
}

// The thread's march state for pair p of the plane (p < hp * ny) of colour
// c, starting at plane kb: its geometry, y rows, x extras and the offsets of
// plane kb.  Constants only (no director or state reads).  ODD false: the
// batch has no odd nx, so no pair has a phantom slot (odd_tail).
template <bool MASK, bool ODD = true>
__device__ __forceinline__ void march_init(const PassArgs &a, const RepDev &R, int c, int p, int kb, March &m) {
    const int hs = R.hs, hps = R.hps, ny = R.ny, hx = R.hx;
    const int j = (int)fastdiv((uint32_t)p, R.hp_m, R.hp_p);
    const int h0 = 2 * (p - j * R.hp);
    m.hasB = h0 + 1 < hx;
    m.tail = odd_tail<MASK, ODD>(R, h0);
    // the x neighbour outside the opposite pair: x- of A when s = 0, x+ of B
    // (or of A when the pair has no B) when s = 1
    int ex0 = h0 - 1, ex1 = m.hasB ? h0 + 2 : h0 + 1;
    m.ee0 = m.ee1 = 1.f;
    if (ex0 < 0) { if (R.xb == BOUND_PERIODIC) ex0 = hx - 1; else { m.ee0 = 0.f; ex0 = h0; } }
    if (ex1 == hx) { if (R.xb == BOUND_PERIODIC) ex1 = 0; else { m.ee1 = 0.f; ex1 = h0; } }
    m.dx0 = ex0 - h0;
    m.dx1 = ex1 - h0;
    int jp = j + 1, jm = j - 1;
    m.eyp = m.eym = 1.f;
    if (jp == ny) { if (R.yb == BOUND_PERIODIC) jp = 0; else { m.eyp = 0.f; jp = j; } }
    if (jm < 0) { if (R.yb == BOUND_PERIODIC) jm = ny - 1; else { m.eym = 0.f; jm = j; } }
    m.dyp = (jp - j) * hs;
    m.dym = (jm - j) * hs;
    m.dypp = (jp - j) * hps;
    m.dymp = (jm - j) * hps;
    const int P = R.plane;
    m.A0 = a.dir + R.dir_off + (long long)(c * 3) * P;
    m.A1 = m.A0 + P;
    m.A2 = m.A1 + P;
    m.O0 = a.dir + R.dir_off + (long long)((c ^ 1) * 3) * P;
    m.O1 = m.O0 + P;
    m.O2 = m.O1 + P;
    m.PA = MASK ? a.pt + R.pt_off + (long long)c * R.pplane : nullptr;
    m.PO = MASK ? a.pt + R.pt_off + (long long)(c ^ 1) * R.pplane : nullptr;
    m.dz = ny * hs;
    m.dzp = ny * hps;
    m.off = (j + ny * kb) * hs + h0;
    m.offp = (j + ny * kb) * hps + h0;
    m.pid = (uint32_t)(j + ny * kb) * (uint32_t)R.hp + (uint32_t)(h0 >> 1);
    m.dpid = (uint32_t)ny * (uint32_t)R.hp;
    m.s = (c + j + kb) & 1;
    m.h0 = h0;
    m.row = j + ny * kb;
}

// Resident CTAs per SM the compiler is asked for (measured best): the
// unmasked Lebwohl-Lasher pass at 96 to 128 registers per thread (five CTAs of
// 128: at six, 80 registers, the packed update spills 48 to 132 bytes and a
// 16^3 block of 200 sweeps took 3.59 ms against 2.78); the GHRL and masked
// variants at 128 (they spill a little there, and still run 1.5x faster than
// unconstrained at 160-206 registers, from the doubled occupancy).
#ifndef MCX_MARCH_LL128_BLOCKS
#define MCX_MARCH_LL128_BLOCKS 5
#endif
#ifndef MCX_MARCH_LL256_BLOCKS
#define MCX_MARCH_LL256_BLOCKS 2
#endif
#ifndef MCX_MARCH_MASK_REGS
#define MCX_MARCH_MASK_REGS 128
#endif
template <int POT, bool MASK, int NT, int MODE = MODE_SWEEP>
constexpr int march_min_blocks() {
  // measured masked passes at 168 registers: at 128 they spill 460 to 540 bytes,
  // more than the L1 cache holds for 16 warps (8 droplets of 96^3: 65.7 us a
  // pass against 71.4; unmeasured ones spill 120 bytes and are slower at 144 or
  // 168, 52.6 and 55.0 against 51.8)
  // (LL in 256 threads at 128, two CTAs: 2 x 45x50x41 9.7 us a measured sweep
  // against 13.5 at 194 registers, 4 slabs of 48x48x40 16.3 against 18.7)
  if (POT == POT_LL && MASK && MODE == MODE_SWEEP_MEASURE && NT == 256) return 2;
  if (MASK && MODE == MODE_SWEEP_MEASURE) return 65536 / (NT * 168) > 0 ? 65536 / (NT * 168) : 1;
  // measured LL passes at 128 registers too: at 96 their seven sums leave too few
  // for loads ahead of the arithmetic (us a measured sweep, 128 against 96: 4 x 64^3
  // in 128 x 8 19.0, 23.7; 4 x 96^3 in 128 x 8 39.4, 48.1; 16^3 in 64 x 4 7.9, 10.0)
  if (POT == POT_LL && !MASK && MODE == MODE_SWEEP_MEASURE) return 65536 / (NT * 128);
  return POT == POT_LL && !MASK ? (NT == 64 ? 9 : (NT == 128 ? MCX_MARCH_LL128_BLOCKS : MCX_MARCH_LL256_BLOCKS))
                                : (MCX_MARCH_MASK_REGS > 0 ? 65536 / (NT * MCX_MARCH_MASK_REGS) : 1);
}

// The neighbourhood of a pair as the update uses it: the neighbours in slots
// x+ x- y+ y- z+ z- of both sites, which bonds exist (e) and exist to an active
// neighbour (w), and which of the two sites are there and active.
struct PairSlots {
  V2 nb[6];
  f32x2 w[6];
  float eA[6], eB[6], wA[6], wB[6];
  bool hereA, hereB, actA, actB;
  int psA, psB;
};

// Own parity s of the row; o0 the opposite pair of the same row, yp / ym those
// of rows y+1 / y-1, op / om those of the planes above / below (zp / zm: those
// bonds exist), exv the extra x neighbour.
template <bool MASK, bool PER>
__device__ __forceinline__ PairSlots pair_slots(int s, bool hasB_, float ee0, float ee1, float eyp, float eym,
                                                const OPair &o0, const OPair &yp, const OPair &ym, const OPair &op,
                                                const OPair &om, const float exv[3], uint16_t pself, uint8_t pex,
                                                bool zp, bool zm, int tail) {
  constexpr bool W = !PER;  // PER: every bond exists (all axes periodic, pairs always complete)
  const bool hasB = PER || hasB_;
  // neighbour slots x+ x- y+ y- z+ z- of both sites
  PairSlots S;
  {
    f32x2 q0[3], q1[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const float lo = o0.v[q].x, hi = o0.v[q].y, ex = exv[q];
      q0[q] = pk(s ? (hasB ? hi : ex) : lo, s ? ex : hi);
      q1[q] = pk(s ? lo : ex, s ? hi : lo);
    }
    S.nb[0] = {q0[0], q0[1], q0[2]};
    S.nb[1] = {q1[0], q1[1], q1[2]};
    S.nb[2] = {pk(yp.v[0]), pk(yp.v[1]), pk(yp.v[2])};
    S.nb[3] = {pk(ym.v[0]), pk(ym.v[1]), pk(ym.v[2])};
    S.nb[4] = {pk(op.v[0]), pk(op.v[1]), pk(op.v[2])};
    S.nb[5] = {pk(om.v[0]), pk(om.v[1]), pk(om.v[2])};
  }
  // bonds present (e) and present to an active neighbour (w), per site
  if (W) {
    const float exe = s ? ee1 : ee0;
    const float erz[4] = {eyp, eym, zp ? 1.f : 0.f, zm ? 1.f : 0.f};
    S.eA[0] = s && !hasB ? exe : 1.f;
    S.eB[0] = s ? exe : 1.f;
    S.eA[1] = s ? 1.f : exe;
    S.eB[1] = 1.f;
    // odd nx (masked only): the last site of an s = 0 row has no x+ bond
    if (MASK && s == 0 && tail == 1) S.eA[0] = 0.f;
    if (MASK && s == 0 && tail == 2) S.eB[0] = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) S.eA[2 + q] = S.eB[2 + q] = erz[q];
    if (MASK) {
      const uint8_t lo = (uint8_t)(o0.pt & 0xFF), hi = (uint8_t)(o0.pt >> 8);
      const uint16_t pr[4] = {yp.pt, ym.pt, op.pt, om.pt};
      auto wt = [](float e, uint8_t p) { return e != 0.f && p != 0 ? 1.f : 0.f; };
      S.wA[0] = wt(S.eA[0], s ? (hasB ? hi : pex) : lo);
      S.wB[0] = wt(S.eB[0], s ? pex : hi);
      S.wA[1] = wt(S.eA[1], s ? lo : pex);
      S.wB[1] = wt(S.eB[1], s ? hi : lo);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        S.wA[2 + q] = wt(erz[q], (uint8_t)(pr[q] & 0xFF));
        S.wB[2 + q] = wt(erz[q], (uint8_t)(pr[q] >> 8));
      }
    } else {
#pragma unroll
      for (int d = 0; d < 6; d++) {
        S.wA[d] = S.eA[d];
        S.wB[d] = S.eB[d];
      }
    }
#pragma unroll
    for (int d = 0; d < 6; d++) S.w[d] = pk(S.wA[d], S.wB[d]);
  } else {
#pragma unroll
    for (int d = 0; d < 6; d++) S.eA[d] = S.eB[d] = S.wA[d] = S.wB[d] = 1.f;
  }
  // odd nx (masked only): a phantom in the last slot of an s = 1 row is skipped
  S.hereA = !(MASK && s == 1 && tail == 1);
  S.hereB = hasB && !(MASK && s == 1 && tail == 2);
  S.psA = MASK ? (pself & 0xFF) : 1;
  S.psB = MASK ? (pself >> 8) : 1;
  S.actA = S.hereA && S.psA != 0;
  S.actB = S.hereB && S.psB != 0;
  return S;
}

// Energies of a pair's old and new directors: bond sums to active neighbours
// (e; unscaled for LL), for a measured masked pass to inactive ones (x, weights
// x[6]), anchoring (s) and field (f), and the energy change dE with every
// rounding the scalar update's (site_update).
struct PairEnergy {
  f32x2 dE, e_old, e_new, x[6], x_old, x_new, s_old, s_new, f_old, f_new;
};

template <int POT, bool MASK, bool FIELD, bool MEAS, bool PER>
__device__ __forceinline__ PairEnergy pair_energy(const PassArgs &a, const RepDev &R, int c, long long ns_at,
                                                  const PairSlots &S, const V2 &n, const V2 &p, const float2 &ax,
                                                  const float2 &ay, const float2 &az) {
  PairEnergy E;
  E.x_old = E.x_new = 0ull;
  if (MASK && MEAS) {  // bonds of active sites to inactive ones
#pragma unroll
    for (int d = 0; d < 6; d++) E.x[d] = pk(S.actA ? S.eA[d] - S.wA[d] : 0.f, S.actB ? S.eB[d] - S.wB[d] : 0.f);
  }
  bond_sums<POT, !PER, MASK && MEAS>(R, n, p, S.nb, S.w, E.e_old, E.e_new, E.x, E.x_old, E.x_new);
  // every rounding of dE is the scalar update's (site_update)
  E.dE = sub2(E.e_new, E.e_old);
  if (POT == POT_LL) E.dE = mul2(pk1(bond_scale<POT>(R)), E.dE);
  E.s_old = E.s_new = E.f_old = E.f_new = 0ull;
  if (MASK && (S.psA > 1 || S.psB > 1)) {  // surface sites
    const float *nsb = a.ns + R.ns_off + (long long)(c * 3) * R.plane + ns_at;
    // the quadratic anchorings W (n.v)^2 of both sites in packed arithmetic
    // (surface_energy's operations): v the surface normal or the easy axis, k
    // its signed strength, 0 for a site without one
    float sn[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}}, v[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    float k[2] = {0.f, 0.f};
    bool form[2] = {false, false};  // a GHRL-form anchoring: the general function
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const int sid = (b ? S.psB : S.psA) - 2;
      if (sid < 0) continue;
#pragma unroll
      for (int q = 0; q < 3; q++) sn[b][q] = __ldg(nsb + q * R.plane + b);
      if (sid >= R.nsurf) continue;
      const int kind = R.anch[sid];
      form[b] = kind == ANCH_HOMEOTROPIC_GHRL || kind == ANCH_FG_GHRL || kind == ANCH_RP_GHRL;
      if (form[b]) continue;
      const bool normal = kind == ANCH_HOMEOTROPIC || kind == ANCH_FG;
      k[b] = kind == ANCH_FG ? R.W[sid] : -R.W[sid];
      v[b][0] = normal ? sn[b][0] : R.dx[sid];
      v[b][1] = normal ? sn[b][1] : R.dy[sid];
      v[b][2] = normal ? sn[b][2] : R.dz[sid];
    }
    const V2 vv = {pk(v[0][0], v[1][0]), pk(v[0][1], v[1][1]), pk(v[0][2], v[1][2])};
    const f32x2 kk = pk(k[0], k[1]);
    // n.v with the fusions the compiler gives surface_energy: x fused onto y
    const f32x2 cn = fma2(p.z, vv.z, fma2(p.x, vv.x, mul2(p.y, vv.y)));
    const f32x2 co = fma2(n.z, vv.z, fma2(n.x, vv.x, mul2(n.y, vv.y)));
    E.s_new = mul2(mul2(kk, cn), cn);
    E.s_old = mul2(mul2(kk, co), co);
    if (form[0] || form[1]) {
      const float2 px = unpk(p.x), py = unpk(p.y), pz = unpk(p.z);
      float2 en = unpk(E.s_new), eo = unpk(E.s_old);
      if (form[0]) {
        en.x = surface_energy(R, S.psA - 2, px.x, py.x, pz.x, sn[0][0], sn[0][1], sn[0][2]);
        eo.x = surface_energy(R, S.psA - 2, ax.x, ay.x, az.x, sn[0][0], sn[0][1], sn[0][2]);
      }
      if (form[1]) {
        en.y = surface_energy(R, S.psB - 2, px.y, py.y, pz.y, sn[1][0], sn[1][1], sn[1][2]);
        eo.y = surface_energy(R, S.psB - 2, ax.y, ay.y, az.y, sn[1][0], sn[1][1], sn[1][2]);
      }
      E.s_new = pk(en);
      E.s_old = pk(eo);
    }
    E.dE = add2(E.dE, sub2(E.s_new, E.s_old));
  }
  if (FIELD) {
    E.f_new = field_energy2(R, p);
    E.f_old = field_energy2(R, n);
    E.dE = add2(E.dE, sub2(E.f_new, E.f_old));
  }
  return E;
}

// What a measured pass adds for a pair with its final directors (ax, ay, az).
// Each bond counts in the local energy of each active end, from the colour-1
// side; the all-site energy also counts inactive sites' bonds to active ones,
// and their field energy with idle (k_idle_field adds it otherwise).
template <int POT, bool MASK, bool FIELD, bool PER, class Q>
__device__ __forceinline__ void measure_pair(const RepDev &R, int c, const PairSlots &S, const PairEnergy &E, bool accA,
                                             bool accB, const float2 &ax, const float2 &ay, const float2 &az, Q &sums,
                                             bool idle) {
  constexpr bool ALL = PER;  // both sites count
  const V2 nf = {pk(ax), pk(ay), pk(az)};
  const f32x2 m = pk(S.actA ? 1.f : 0.f, S.actB ? 1.f : 0.f);
  sums.tensor(nf, ALL ? nf : mul2(nf, m));
  f32x2 s = 0ull, f0 = 0ull, f1 = 0ull, b0 = 0ull, b1 = 0ull, x = 0ull;
  if (MASK) s = mul2(pick2(accA, accB, E.s_new, E.s_old), m);
  if (FIELD) {
    const f32x2 f = pick2(accA, accB, E.f_new, E.f_old);
    f0 = f1 = ALL ? f : mul2(f, m);
    if (MASK && idle) f0 = mul2(f, pk(S.hereA ? 1.f : 0.f, S.hereB ? 1.f : 0.f));
  }
  if (c == 1) {
    f32x2 eb = pick2(accA, accB, E.e_new, E.e_old);
    if (POT == POT_LL) eb = mul2(pk1(bond_scale<POT>(R)), eb);
    eb = add_bond_const<POT, !PER>(R, S.w, eb);
    if (ALL) {
      b0 = b1 = add2(eb, eb);
    } else {
      b0 = mul2(pk(S.actA ? 2.f : (S.hereA ? 1.f : 0.f), S.actB ? 2.f : (S.hereB ? 1.f : 0.f)), eb);
      if (Q::kMasked) b1 = mul2(pk(S.actA ? 2.f : 0.f, S.actB ? 2.f : 0.f), eb);
      if (MASK) {
        x = pick2(accA, accB, E.x_new, E.x_old);
        if (POT == POT_LL) x = mul2(pk1(bond_scale<POT>(R)), x);
        x = add_bond_const<POT, true>(R, E.x, x);
      }
    }
  }
  sums.template energy<MASK, FIELD>(c, s, f0, f1, b0, b1, x);
}

__device__ __forceinline__ void accept_pair(bool accA, bool accB, const V2 &p, float2 &ax, float2 &ay, float2 &az) {
  const float2 px = unpk(p.x), py = unpk(p.y), pz = unpk(p.z);
  if (accA) {
    ax.x = px.x;
    ay.x = py.x;
    az.x = pz.x;
  }
  if (accB) {
    ax.y = px.y;
    ay.y = py.y;
    az.y = pz.y;
  }
}

// The update of one same-colour pair from its loaded neighbourhood (shared by
// the z-march, its staged and prefetching forms and the resident sweeps): own
// directors (ax, ay, az) in and out; the neighbourhood as in pair_slots; rw the
// pair's Philox draw (pair_draw below).  Both sites run in packed arithmetic
// (mcx_packed.cuh); a missing, phantom or inactive site's half is computed and
// dropped.
template <int POT, bool MASK, bool FIELD, int MODE, bool PER, class Q>
__device__ __forceinline__ void update_pair_draw(const PassArgs &a, const RepDev &R, int c, int s, bool hasB,
                                                 float ee0, float ee1, float eyp, float eym, const OPair &o0,
                                                 const OPair &yp, const OPair &ym, const OPair &op, const OPair &om,
                                                 const float exv[3], uint16_t pself, uint8_t pex, bool zp, bool zm,
                                                 const uint4 rw, long long ns_at, float ang, float invT, float2 &ax,
                                                 float2 &ay, float2 &az, unsigned &acc, Q &sums,
                                                 int tail = 0) {
  constexpr bool MEAS = MODE == MODE_SWEEP_MEASURE;
  const PairSlots S = pair_slots<MASK, PER>(s, hasB, ee0, ee1, eyp, eym, o0, yp, ym, op, om, exv, pself, pex, zp, zm,
                                            tail);
  const V2 n = {pk(ax), pk(ay), pk(az)};
  const V2 p = propose2(n, rw, ang);
  const PairEnergy E = pair_energy<POT, MASK, FIELD, MEAS, PER>(a, R, c, ns_at, S, n, p, ax, ay, az);
  // src/evolve.cpp:160: accept when u < exp(-(E_new - E_old)/T)
  const float2 arg = unpk(mul2(E.dE, pk1(-invT))), u2 = accept_uniforms(rw);
  const bool accA = S.actA && u2.x < __expf(arg.x), accB = S.actB && u2.y < __expf(arg.y);
  accept_pair(accA, accB, p, ax, ay, az);
  acc += (accA ? 1u : 0u) + (accB ? 1u : 0u);
  if (MEAS) measure_pair<POT, MASK, FIELD, PER>(R, c, S, E, accA, accB, ax, ay, az, sums, a.idle_in_pass != 0);
}

// The pair's Philox draw (counter: pair index, sweep, colour; key: seed,
// stream), and update_pair_draw with it.
__device__ __forceinline__ uint4 pair_draw(uint32_t pid, int c, unsigned long long sw, uint32_t seed, uint32_t stream) {
  return philox4x32_10(make_uint4(pid, (uint32_t)sw, (uint32_t)(sw >> 32), TAG_PLAIN | (uint32_t)c), seed, stream);
}

template <int POT, bool MASK, bool FIELD, int MODE, bool PER, class Q>
__device__ __forceinline__ void update_pair(const PassArgs &a, const RepDev &R, int c, int s, bool hasB_, float ee0,
                                            float ee1, float eyp, float eym, const OPair &o0, const OPair &yp,
                                            const OPair &ym, const OPair &op, const OPair &om, const float exv[3],
                                            uint16_t pself, uint8_t pex, bool zp, bool zm, uint32_t pid,
                                            long long ns_at, uint32_t seed, uint32_t stream, unsigned long long sw,
                                            float ang, float invT, float2 &ax, float2 &ay, float2 &az, unsigned &acc,
                                            Q &sums, int tail = 0) {
  update_pair_draw<POT, MASK, FIELD, MODE, PER>(a, R, c, s, hasB_, ee0, ee1, eyp, eym, o0, yp, ym, op, om, exv, pself,
                                                pex, zp, zm, pair_draw(pid, c, sw, seed, stream), ns_at, ang, invT, ax,
                                                ay, az, acc, sums, tail);
}

}  // namespace mcx
