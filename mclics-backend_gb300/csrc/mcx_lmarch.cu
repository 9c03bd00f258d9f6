// mcx_lmarch.cu -- the learned-proposal pass as a z-march (no counterpart in
// the reference).
//
//   k_lmarch  the z-march of mcx_march.cu with the learned proposal: per
//             plane every thread loads its pair's neighbourhood, writes the two
//             sites' network inputs as rows lane and lane+32 of its warp's
//             64-row tile, the warp evaluates the network on the tensor cores
//             (mlp_warp, mcx_mlp.cuh), and each thread loads the neighbourhood
//             again, draws and accepts its sites' moves
//             (update_pair_learned).  The network is warp-synchronous, so every
//             lane runs every plane: a thread past the end of the plane
//             contributes zero rows and updates nothing.  41 KB of shared memory
//             per CTA (weights and one input/output tile per warp), four CTAs of
//             128 threads per SM at 128 registers.
//
//             What bounded it: shared-memory wavefronts (60% of peak, the
//             network's weight fragments) and the issue of 44 warp instructions
//             per site.  Two row tiles now share each weight fragment; for their
//             registers the neighbourhood is not held across the network but
//             read a second time (L2, 7% busy).  Bonds and energies run packed
//             (mcx_packed.cuh).  4 x LL 96^3: 123.5 -> 112.4 us a pass (37
//             instructions per site, wavefronts 41%); 6 droplets of 64^3, whose
//             chunks of 8 planes also left the last wave idle (learn_depth,
//             mcx_engine.cu): 85 -> 50 us, measured 100 -> 55.
//
//             With TC the network runs on the 5th-generation tensor cores
//             instead (tc_mlp, mcx_tcmlp.cuh): per plane the CTA's 128
//             threads store their two sites' input rows as two M = 128 tiles
//             (thread t is row t of each: site A, site B), one thread issues
//             the tcgen05.mma of each layer, the accumulators sit in 128 TMEM
//             columns of the CTA and every thread reads back its own rows.
//             63 KB of shared memory per CTA (three CTAs per SM).
//
// It computes what the learned direct pass (k_pass<LEARN>) computes, bit for
// bit: the same rows reach the network, the same per-site Philox counters drive
// the draws, and the energies keep the scalar update's roundings.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mcx_march.cuh"
#include "mcx_mlp.cuh"
#include "mcx_tcmlp.cuh"

namespace mcx {

constexpr int kLPB = 128;  // threads per CTA (4 warps)
constexpr int kLmarchSmem = kMlpBytes + (kLPB / 32) * (64 * kXs * 2 + 64 * 4 * 4);
constexpr int kLmarchTcSmem = kTcWBytes + 2 * kTcXBytes + 2 * kTcHBytes + 64;
constexpr uint32_t kLmarchTcCols = 128;  // two tiles of 64 FP32 accumulator columns
#ifndef MCX_LMARCH_MIN_BLOCKS
#define MCX_LMARCH_MIN_BLOCKS 4
#endif

// A pair's neighbourhood as loaded for plane k.
struct Hood {
  OPair o0, yp, ym, op, om;
  float ex[3];
  uint8_t pex;
};

// CARRY: om and o0 are there already (the plane before's o0 and op).
template <bool MASK, bool CARRY = false>
__device__ __forceinline__ void load_hood(const March &m, int up, int down, bool zp, bool zm, Hood &h) {
  const int dx = m.s ? m.dx1 : m.dx0;
  if (!CARRY) load_opair_at<MASK>(m, m.off, m.offp, true, h.o0);
  load_opair_at<MASK>(m, m.off + m.dyp, m.offp + m.dypp, true, h.yp);
  load_opair_at<MASK>(m, m.off + m.dym, m.offp + m.dymp, true, h.ym);
  load_opair_at<MASK>(m, m.off + up * m.dz, m.offp + up * m.dzp, zp, h.op);
  if (!CARRY) load_opair_at<MASK>(m, m.off - down * m.dz, m.offp - down * m.dzp, zm, h.om);
  h.ex[0] = ldo1(m.O0 + m.off + dx);
  h.ex[1] = ldo1(m.O1 + m.off + dx);
  h.ex[2] = ldo1(m.O2 + m.off + dx);
  h.pex = 1;
  if (MASK) h.pex = __ldg(m.PO + m.offp + dx);
}

template <bool MASK, bool PER>
__device__ __forceinline__ PairSlots hood_slots(const March &m, const Hood &h, uint16_t pself, bool zp, bool zm) {
  return pair_slots<MASK, PER>(m.s, m.hasB, m.ee0, m.ee1, m.eyp, m.eym, h.o0, h.yp, h.ym, h.op, h.om, h.ex, pself,
                               h.pex, zp, zm, m.tail);
}

// The network input rows of both sites (feature_words): the six neighbours
// (absent or inactive ones as zero vectors), T and a zero, as BF16 pairs; zero
// rows for sites that are not there.
__device__ __forceinline__ void pair_features(const PairSlots &S, float T, bool liveA, bool liveB, uint32_t rA[16],
                                              uint32_t rB[16]) {
  float fA[20], fB[20];
  const f32x2 live = pk(liveA ? 1.f : 0.f, liveB ? 1.f : 0.f);
#pragma unroll
  for (int d = 0; d < 6; d++) {
    const f32x2 w = pk(liveA ? S.wA[d] : 0.f, liveB ? S.wB[d] : 0.f);
    const float2 x = unpk(mul2(S.nb[d].x, w)), y = unpk(mul2(S.nb[d].y, w)), z = unpk(mul2(S.nb[d].z, w));
    fA[3 * d] = x.x; fA[3 * d + 1] = y.x; fA[3 * d + 2] = z.x;
    fB[3 * d] = x.y; fB[3 * d + 1] = y.y; fB[3 * d + 2] = z.y;
  }
  const float2 t = unpk(mul2(live, pk1(T)));
  fA[18] = t.x;
  fB[18] = t.y;
  fA[19] = fB[19] = 0.f;
#pragma unroll
  for (int q = 0; q < 10; q++) {
    rA[q] = pack_bf16(fA[2 * q], fA[2 * q + 1]);
    rB[q] = pack_bf16(fB[2 * q], fB[2 * q + 1]);
  }
#pragma unroll
  for (int q = 10; q < 16; q++) rA[q] = rB[q] = 0u;
}

// One site's draw from the network's mixture.
struct Drawn {
  float mu[3], kappa, v[3], u;
};
__device__ __forceinline__ void draw_site(const RepDev &R, const float4 &y4, uint32_t nat, unsigned long long sw,
                                          Drawn &d) {
  const float y[4] = {y4.x, y4.y, y4.z, y4.w};
  const uint4 r = philox4x32_10(make_uint4(nat, (uint32_t)sw, (uint32_t)(sw >> 32), TAG_VMF), R.seed, R.stream);
  vmf_params(y, d.mu, d.kappa);
  vmf_sample(d.mu, d.kappa, u01(r.x), u01(r.y), u01(r.z), d.v);
  d.u = u01(r.w);
}

// The learned update of a pair (site_update_learned for both sites): the draws
// site by site, everything between them in packed arithmetic with the scalar
// update's roundings.
template <int POT, bool MASK, bool FIELD, int MODE, bool PER, class Q>
__device__ __forceinline__ void update_pair_learned(const PassArgs &a, const RepDev &R, int c, const PairSlots &S,
                                                    const float4 &yA, const float4 &yB, uint32_t nat, long long ns_at,
                                                    unsigned long long sw, float invT, float2 &ax, float2 &ay,
                                                    float2 &az, unsigned &acc, Q &sums) {
  constexpr bool MEAS = MODE == MODE_SWEEP_MEASURE;
  const V2 n = {pk(ax), pk(ay), pk(az)};
  Drawn A = {{0.f, 0.f, 1.f}, 0.f, {0.f, 0.f, 1.f}, 1.f}, B = A;
  if (!MASK || S.actA) draw_site(R, yA, nat, sw, A);
  if (!MASK || S.actB) draw_site(R, yB, nat + 2u, sw, B);
  const V2 p = {pk(A.v[0], B.v[0]), pk(A.v[1], B.v[1]), pk(A.v[2], B.v[2])};
  const V2 mu = {pk(A.mu[0], B.mu[0]), pk(A.mu[1], B.mu[1]), pk(A.mu[2], B.mu[2])};
  const PairEnergy E = pair_energy<POT, MASK, FIELD, MEAS, PER>(a, R, c, ns_at, S, n, p, ax, ay, az);
  const f32x2 kap = pk(A.kappa, B.kappa);
  const float2 co = unpk(mul2(kap, dot2(mu, n))), cn = unpk(mul2(kap, dot2(mu, p)));
  const f32x2 lo = pk(log_cosh_shift(co.x), log_cosh_shift(co.y));
  const f32x2 ln = pk(log_cosh_shift(cn.x), log_cosh_shift(cn.y));
  const float2 lr = unpk(sub2(fma2(E.dE, pk1(-invT), lo), ln));
  const bool accA = S.actA && A.u < __expf(lr.x), accB = S.actB && B.u < __expf(lr.y);
  accept_pair(accA, accB, p, ax, ay, az);
  acc += (accA ? 1u : 0u) + (accB ? 1u : 0u);
  if (MEAS) measure_pair<POT, MASK, FIELD, PER>(R, c, S, E, accA, accB, ax, ay, az, sums, a.idle_in_pass != 0);
}

// the tensor-core form holds 63 KB of shared memory: three CTAs per SM, so
// each thread may use up to 170 registers.  ODD: the batch holds an odd nx
// (phantom slots, odd_tail); built only for masked batches that need it.
template <int POT, bool MASK, bool FIELD, int MODE, bool TC, bool ODD, bool PER>
__global__ void __launch_bounds__(kLPB, TC ? 3 : MCX_LMARCH_MIN_BLOCKS) k_lmarch(PassArgs a) {
  static_assert(MODE == MODE_SWEEP || MODE == MODE_SWEEP_MEASURE, "sweep modes only");
  extern __shared__ __align__(1024) uint8_t dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t *W = dyn;
  __nv_bfloat16 *X = reinterpret_cast<__nv_bfloat16 *>(dyn + kMlpBytes) + (size_t)warp * 64 * kXs;
  float *Y = reinterpret_cast<float *>(dyn + kMlpBytes + (kLPB / 32) * 64 * kXs * 2) + (size_t)warp * 64 * 4;
  // tensor-core form: network image, two input tiles, two activation tiles,
  // the MMA mbarrier and the TMEM address
  uint8_t *TX = dyn + kTcWBytes, *TH = TX + 2 * kTcXBytes;
  uint64_t *tbar = reinterpret_cast<uint64_t *>(TH + 2 * kTcHBytes);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(tbar + 1);
  uint32_t tmem = 0, tphase = 0;
  // the weights are written only between launches (host copies on the stream)
  if (TC) {
    tc_load_weights(a.mlp, W, kLPB);
    if (threadIdx.x == 0) {
      mbar_init(tbar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc_alloc(tslot, kLmarchTcCols);
    fence_proxy_async();
    tc_fence_before();
  } else {
    for (int i = threadIdx.x; i < kMlpBytes / 16; i += kLPB)
      reinterpret_cast<int4 *>(W)[i] = reinterpret_cast<const int4 *>(a.mlp)[i];
    clear_row_tails(X, lane);
  }
  const int4 u = a.units[blockIdx.x];
  const int r = u.x, c = a.colour;
  const RepDev &R = a.reps[r];
  const RepState *S = a.st + r;
  const int npp = R.hp * R.ny;
  const bool valid = u.y + (int)threadIdx.x < npp;
  const int p = valid ? u.y + (int)threadIdx.x : npp - 1;  // lanes past the plane shadow the last pair
  March m;
  march_init<MASK, ODD>(a, R, c, p, u.z, m);
  const int nz = R.nz, nx = R.nx;
  const bool zper = R.zb == BOUND_PERIODIC;
  const int kb = u.z, ke = u.z + (u.w & kUnitPlanes);
  unsigned acc = 0;
  PairSums<MASK> sums;
  sums.clear();
  __syncthreads();  // weights in shared memory
  if (TC) {
    tc_fence_after();
    tmem = *tslot;
  }
  grid_dependency_wait(m);
  if (MASK && (u.w & kUnitDead)) {  // no active site in or next to it
    if (valid && a.idle_in_pass) dead_unit<FIELD, MODE>(R, m, kb, ke, sums);
  } else {
    const unsigned long long sw = S->sweep;
    const float T = S->T, invT = 1.0f / S->T;
    Hood h;
    if (TC) {
      const int down = kb > 0 ? 1 : 1 - nz;
      load_opair_at<MASK>(m, m.off - down * m.dz, m.offp - down * m.dzp, kb > 0 || zper, h.om);
      load_opair_at<MASK>(m, m.off, m.offp, true, h.o0);
    }
#pragma unroll 1
    for (int k = kb; k < ke; k++) {
      const bool zp = k + 1 < nz || zper, zm = k > 0 || zper;
      const int up = k + 1 < nz ? 1 : 1 - nz, down = k > 0 ? 1 : 1 - nz;
      uint16_t pself = 0x0101;
      if (MASK) pself = __ldg(reinterpret_cast<const uint16_t *>(m.PA + m.offp));
      // a warp whose 64 sites are all inactive: nothing moves, so it needs no
      // network, and only the colour-1 sites' bonds to active ones are measured
      // (the tensor-core form evaluates the network per CTA and does not skip)
      const bool idle = !TC && MASK && __all_sync(0xffffffffu, !valid || pself == 0);
      if (!(idle && (MODE == MODE_SWEEP || (c == 0 && !(FIELD && a.idle_in_pass))))) {
        float4 yA = make_float4(0.f, 0.f, 0.f, 0.f), yB = yA;
        if (!idle) {
          load_hood<MASK, TC>(m, up, down, zp, zm, h);
          const PairSlots sl = hood_slots<MASK, PER>(m, h, pself, zp, zm);
          uint32_t rA[16], rB[16];
          pair_features(sl, T, valid, valid && (PER || m.hasB), rA, rB);
          if (TC) {
            // the network for the CTA's 256 sites: two M = 128 tiles on the tensor cores
            tc_store_row32(TX, threadIdx.x, rA);
            tc_store_row32(TX + kTcXBytes, threadIdx.x, rB);
            fence_proxy_async();
            __syncthreads();
            float y[2][4];
            if (!tc_mlp(W, TX, TH, 2, tmem, tbar, tphase, y, a.err)) break;  // uniform: every thread saw the same waits
            yA = make_float4(y[0][0], y[0][1], y[0][2], y[0][3]);
            yB = make_float4(y[1][0], y[1][1], y[1][2], y[1][3]);
          } else {
            // the network for the warp's 64 sites
            __syncwarp();
            store_row(X, site_row(lane, 0), rA);  // words 10..15 are zeros that clear_row_tails wrote
            store_row(X, site_row(lane, 1), rB);
            __syncwarp();
            mlp_warp<2>(W, X, Y);
            __syncwarp();
            yA = reinterpret_cast<const float4 *>(Y)[site_row(lane, 0)];
            yB = reinterpret_cast<const float4 *>(Y)[site_row(lane, 1)];
          }
        }
        if (valid) {
          // the neighbourhood again: held in registers across the warp's network
          // it would cost the network its second row tile (spills).  The tensor
          // cores' network needs few registers, and its CTAs have 168 per thread:
          // held there, with the z reuse of the march (4 x LL 96^3 at one shape 259 us
          // a sweep; 317 with the second reading)
          if (!TC) load_hood<MASK>(m, up, down, zp, zm, h);
          float2 ax = *reinterpret_cast<const float2 *>(m.A0 + m.off);
          float2 ay = *reinterpret_cast<const float2 *>(m.A1 + m.off);
          float2 az = *reinterpret_cast<const float2 *>(m.A2 + m.off);
          const PairSlots sl = hood_slots<MASK, PER>(m, h, pself, zp, zm);
          const uint32_t nat = (uint32_t)(2 * m.h0 + m.s) + (uint32_t)nx * (uint32_t)m.row;
          update_pair_learned<POT, MASK, FIELD, MODE, PER>(a, R, c, sl, yA, yB, nat, m.off, sw, invT, ax, ay, az, acc,
                                                           sums);
          *reinterpret_cast<float2 *>(m.A0 + m.off) = ax;
          *reinterpret_cast<float2 *>(m.A1 + m.off) = ay;
          *reinterpret_cast<float2 *>(m.A2 + m.off) = az;
        }
      }
      if (TC) {
        h.om = h.o0;
        h.o0 = h.op;
      }
      m.off += m.dz;
      m.offp += m.dzp;
      m.row += R.ny;
      m.s ^= 1;
    }
  }
  grid_launch_dependents();
  // chunks deeper than 8 planes (32 at most, learn_depth): the warp's and the CTA's
  // sums in two parts, which makes up for the thread's longer ones (energy of a
  // sweep of 8 x LL 96^3, rms against FP64: 1.2e-9 of itself; 5.0e-9 with FP32
  // sums, 2.9e-9 in chunks of 8 planes)
  float qs[kQ], low[kQ];
  sums.fold(qs);
#pragma unroll
  for (int q = 0; q < kQ; q++) low[q] = 0.f;
  flush_replica<kLPB, MODE>(a, r, 1, (unsigned)R.lcta, acc, qs, MASK, -1, -1, ke - kb > kLongPlanes ? low : nullptr);
  if (TC) {  // every TMEM read is done (tc_mlp ends on a fenced barrier; flush_replica syncs again)
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, kLmarchTcCols);
  }
}

template <int POT, bool MASK, bool FIELD, bool TC, bool ODD, bool PER>
static const void *lmarch_fn(int mode) {
  return mode == MODE_SWEEP_MEASURE ? (const void *)k_lmarch<POT, MASK, FIELD, MODE_SWEEP_MEASURE, TC, ODD, PER>
                                    : (const void *)k_lmarch<POT, MASK, FIELD, MODE_SWEEP, TC, ODD, PER>;
}

template <int POT, bool FIELD, bool TC>
static const void *lmarch_fn_v(const Variant &v, int mode) {
  if (v.mask)
    return v.odd ? lmarch_fn<POT, true, FIELD, TC, true, false>(mode) : lmarch_fn<POT, true, FIELD, TC, false, false>(mode);
  return v.per ? lmarch_fn<POT, false, FIELD, TC, false, true>(mode) : lmarch_fn<POT, false, FIELD, TC, false, false>(mode);
}

template <bool TC>
static const void *lmarch_kernel_tc(const Variant &v, int mode) {
  if (v.pot == POT_LL) return v.field ? lmarch_fn_v<POT_LL, true, TC>(v, mode) : lmarch_fn_v<POT_LL, false, TC>(v, mode);
  return v.field ? lmarch_fn_v<POT_GHRL, true, TC>(v, mode) : lmarch_fn_v<POT_GHRL, false, TC>(v, mode);
}

static const void *lmarch_kernel(const Variant &v, int mode, bool tc) {
  return tc ? lmarch_kernel_tc<true>(v, mode) : lmarch_kernel_tc<false>(v, mode);
}

static int lmarch_smem(bool tc) { return tc ? kLmarchTcSmem : kLmarchSmem; }

int lmarch_block_threads() { return kLPB; }

int lmarch_blocks_per_sm(const Variant &v, bool tc) {
  int n = 0;
  if (tc) {
    // the occupancy call answers 1 for a kernel that allocates tensor memory;
    // registers, shared memory and TMEM columns hold three such CTAs
    cudaFuncAttributes f;
    int dev = 0, smem = 0, regs = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&f, lmarch_kernel(v, MODE_SWEEP, tc)) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&regs, cudaDevAttrMaxRegistersPerMultiprocessor, dev) != cudaSuccess)
      return 0;
    const int per_cta = (f.numRegs + 7) / 8 * 8 * kLPB;  // registers come in blocks of 8 a thread
    n = smem / (lmarch_smem(tc) + (int)f.sharedSizeBytes + 1024);  // 1 KB of each CTA's is the system's
    if (regs / per_cta < n) n = regs / per_cta;
    if (512 / (int)kLmarchTcCols < n) n = 512 / (int)kLmarchTcCols;
    return n;
  }
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, lmarch_kernel(v, MODE_SWEEP, tc), kLPB, lmarch_smem(tc)) !=
      cudaSuccess)
    return 0;
  return n;
}

bool lmarch_prepare(const Variant &v, bool tc) {
  if (v.pot == POT_PEAR) return false;
  for (int mode : {MODE_SWEEP, MODE_SWEEP_MEASURE})
    if (cudaFuncSetAttribute(lmarch_kernel(v, mode, tc), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             lmarch_smem(tc)) != cudaSuccess)
      return false;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, lmarch_kernel(v, MODE_SWEEP, tc), kLPB, lmarch_smem(tc)) !=
      cudaSuccess)
    return false;
  // the tensor-core form's CTAs must all find their TMEM columns (512 per SM)
  return n > 0 && (!tc || (uint32_t)n * kLmarchTcCols <= 512);
}

void launch_lmarch(const Variant &v, int mode, const PassArgs &a, bool pdl, bool tc, cudaStream_t st) {
  if (v.pot == POT_PEAR) return;  // the learned proposal is refused for Pear
  PassArgs args = a;
  void *params[] = {&args};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.nunits);
  cfg.blockDim = dim3(kLPB);
  cfg.dynamicSmemBytes = lmarch_smem(tc);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelExC(&cfg, lmarch_kernel(v, mode, tc), params);
}

}  // namespace mcx
