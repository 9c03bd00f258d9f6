// mcx_resident.cu -- the plain-proposal sweeps of small lattices, resident in
// shared memory (k_resident), and their launchers.
//
// What bounds a small lattice is the launch and the latency chain of a pass,
// not work: a 16^3 pass is 32 warps of work and took 7 us (launch, unit and
// replica loads, directors from L2, and the atomic that ends the sweep), twice
// per sweep.  Here a cluster of CTAs holds one replica for a whole run of
// sweeps: each CTA keeps a run of its rows of both colours in shared memory
// with one plane of rows on either side, a pass reads shared memory only, the
// sites next to another CTA's rows are also sent into that CTA's copy
// (distributed shared memory), and every thread applies the step-size rule by
// itself from the sweep's acceptances, which each warp adds into every CTA's
// counter.  Directors are read from and written to HBM once per run.
//
// Halo rows and acceptances travel as asynchronous stores (st.async, red.async)
// that count their bytes on the receiving CTA's mbarrier, so a CTA waits for
// its neighbours' rows only and no store is fenced: with a cluster barrier per
// pass, 30% of a 16^3 pass was the barrier's release fence.  mcx_phase.h says
// which barrier counts what.  Who may overwrite what, and what orders it:
//   - a CTA's halo rows of colour c are read by its own rows next to them, in
//     its pass of the other colour, and rewritten by the neighbour's next pass
//     of colour c.  For c = 1 that pass starts after the neighbour has received
//     the new directors of every pair that read the halo (in a pass of colour 0
//     only pairs with an active site do, and those are sent); a pair's director
//     depends on what it read.  For c = 0 it starts after the neighbour has
//     received every warp's acceptances of that pass, which depend on what the
//     warp's pairs read: on active pairs' by their decisions, on those of two
//     inactive sites, which a measured pass of colour 1 reads for their bonds,
//     by a bit of the energy sum (a fence there cost 1.5 us a sweep).
//   - nobody clears the acceptance counters: they grow, and a thread subtracts
//     what it read two sweeps before.  They are added to again after every
//     warp's acceptances of the next sweep, so after its read.
// Every wait has a limit in time.  A CTA one of whose waits ran out leaves the
// run at the end of that sweep; the others, which then miss its acceptances, in
// the next.  They tell each other at the cluster barrier after the run, after
// which nobody sends: then all wait for a millisecond, so that no row or count on
// its way (a microsecond at most) meets a CTA that has ended, set the error flag
// and leave the replica as it was before the run.
//
// Same Philox counters and pair update as k_march (mcx_march.cuh), so the chain
// is the same bit for bit.
#include <cuda_runtime.h>

#include "mcx_march.cuh"
#include "mcx_phase.h"
#include "mcx_step.h"
#include "mcx_tma.cuh"

namespace mcx {

// Most threads per CTA: measured masked builds take up to 168 registers per
// thread (at 128 they spill 260 bytes; 16 droplets of 25^3: 6.9 us a pass
// against 7.9; unmeasured ones fit 128, and at 168 fewer CTAs share an SM, 5.2
// against 4.3)
constexpr int kResThreads = 512, kResMaskThreads = 384;

// A pair of the CTA's rows: offsets (floats) into a (colour, component) plane
// of shared memory, and which of its bonds exist.
struct __align__(16) ResPair {
  uint16_t off, yp, ym, ex0, ex1, flags;
  uint32_t zero;
};
enum : int {
  RF_ODD = 1,      // (j + k) & 1
  RF_HASB = 2,
  RF_ZP = 4,
  RF_ZM = 8,
  RF_YP = 16,
  RF_YM = 32,
  RF_EX0 = 64,
  RF_EX1 = 128,
  RF_TAIL = 8,     // shift of the two tail bits (odd_tail)
  RF_PREV = 1024,  // in a row the previous / next CTA also holds
  RF_NEXT = 2048
};

// Shared-memory layout of a CTA for a replica whose largest share is n rows:
// those rows plus one plane of rows on either side.
struct ResLayout {
  int fl;     // floats per (colour, component)
  int pt;     // bytes per colour of point types (masked)
  int pairs;  // pairs of the largest share
};
__host__ __device__ __forceinline__ ResLayout res_layout(const RepDev &R, int n) {
  ResLayout L;
  L.fl = (n + 2 * R.ny) * R.hs;
  L.pt = (L.fl + 15) / 16 * 16;
  L.pairs = n * R.hp;
  return L;
}

// Sums of a measured sweep over a thread's pairs, each term split so that the
// result does not depend on how the pairs fall to threads and CTAs (a batch is
// cut by its own sizes, and a replica measures the same in any batch): the
// Q-tensor products, below 1, into multiples of 2^-17, which add exactly up to
// 2^7, and a remainder; the energies with the rounding error of each addition.
template <bool MASKED>
struct SplitSums {
  static constexpr bool kMasked = MASKED;
  f32x2 hi[kQ], lo[kQ];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < kQ; q++) hi[q] = lo[q] = 0ull;
  }
  __device__ __forceinline__ void add(int q, f32x2 t) {
    if (q >= 2) {
      const f32x2 h = add2(add2(t, pk1(96.f)), pk1(-96.f));
      hi[q] = add2(hi[q], h);
      lo[q] = add2(lo[q], sub2(t, h));
    } else {
      const f32x2 s = add2(hi[q], t), b = sub2(s, hi[q]);
      lo[q] = add2(lo[q], add2(sub2(hi[q], sub2(s, b)), sub2(t, b)));
      hi[q] = s;
    }
  }
  __device__ __forceinline__ void tensor(const V2 &n, const V2 &nm) {
    add(2, mul2(nm.x, n.x));
    add(3, mul2(nm.x, n.y));
    add(4, mul2(nm.x, n.z));
    add(5, mul2(nm.y, n.y));
    add(6, mul2(nm.z, n.y));
  }
  template <bool MASK, bool FIELD>
  __device__ __forceinline__ void energy(int c, f32x2 s, f32x2 f0, f32x2 f1, f32x2 b0, f32x2 b1, f32x2 x) {
    if (!MASK && !FIELD && c != 1) return;
    f32x2 all = b0, valid = b1;
    if (FIELD) {
      all = add2(all, f0);
      valid = add2(valid, f1);
    }
    if (MASK) {
      all = add2(all, add2(s, x));
      valid = add2(valid, s);
    }
    add(0, all);
    if (MASKED) add(1, valid);
  }
};

// The warp's sums (warp_sums): quantity q in lane 4 q.
template <bool MASKED>
__device__ __forceinline__ double warp_split_sums(const SplitSums<MASKED> &t) {
  float h[kQ], l[kQ];
#pragma unroll
  for (int q = 0; q < kQ; q++) {
    const float2 a = unpk(t.hi[q]), b = unpk(t.lo[q]);
    h[q] = a.x;
    l[q] = b.x;
    add_split(h[q], l[q], a.y, b.y);
  }
  return warp_sums(h, l);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
// 8 bytes to another CTA's shared memory, counted on its mbarrier
__device__ __forceinline__ void st_remote(uint32_t addr, const float2 &v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void red_remote(uint32_t addr, unsigned v, uint32_t bar) {
  asm volatile("red.async.relaxed.cluster.shared::cluster.mbarrier::complete_tx::bytes.add.u32 [%0], %1, [%2];" ::"r"(
                   addr),
               "r"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void set_remote(uint32_t addr, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool res_try(uint32_t b, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(b), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits for a phase of a barrier that other CTAs complete; false when `limit`
// nanoseconds (or some seconds of polls, should the timer not run) are over.
__device__ __forceinline__ bool res_wait(uint64_t *bar, uint32_t parity, unsigned long long limit) {
  const uint32_t b = smem_u32(bar);
  if (res_try(b, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (unsigned i = 0; i < (1u << 25); i++) {
    if (res_try(b, parity)) return true;
    if (now_ns() - t0 > limit) return false;
  }
  return false;
}
// After a run that was given up: rows and counts on their way land.
__device__ __forceinline__ void let_land() {
  const unsigned long long t0 = now_ns();
  for (unsigned i = 0; i < (1u << 20) && now_ns() - t0 < 1000000ull; i++) __nanosleep(1000);
}

template <int POT, bool MASK, bool FIELD, int MODE, bool PER>
__global__ void __launch_bounds__(MASK && MODE == MODE_SWEEP_MEASURE ? kResMaskThreads : kResThreads, 1)
    k_resident(PassArgs a, const int *cut, int nsweeps, int C, unsigned long long limit, unsigned extra) {
  constexpr bool MEAS = MODE == MODE_SWEEP_MEASURE;
  extern __shared__ __align__(16) uint8_t res_smem[];
  __shared__ unsigned s_cnt[2];            // accepted moves of the even and of the odd sweeps, every CTA's
  __shared__ __align__(8) uint64_t bars[kResBars];  // halo_bar, count_bar (mcx_phase.h)
  __shared__ unsigned s_bad;               // a CTA of the cluster gave up
  __shared__ unsigned s_tx[2];             // pairs that arrive per pass of each colour
  __shared__ __align__(16) RepDev sR;      // the replica's constants: read in every pass
  const int rank = (int)cluster_rank(), r = blockIdx.x / C;
  RepState *S = a.st + r;
  const int NT = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < (int)(sizeof(RepDev) / 4); i += NT)
    reinterpret_cast<uint32_t *>(&sR)[i] = reinterpret_cast<const uint32_t *>(a.reps + r)[i];
  if (tid < 2) s_cnt[tid] = 0;
  if (tid == 0) s_bad = 0;
  if (tid < 2) s_tx[tid] = 0;
  if (tid == 0) {
    for (int q = 0; q < kResBars; q++) mbar_init(&bars[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const RepDev &R = sR;
  const int hs = R.hs, hp = R.hp, ny = R.ny, nz = R.nz, rows_all = ny * nz;
  cut += (size_t)r * (C + 2);  // the first row of each CTA, the row count, the largest share
  const ResLayout L = res_layout(R, cut[C + 1]);
  const int r0 = cut[rank], n = cut[rank + 1] - r0;
  const int np = n * hp, dz = ny * hs;
  const bool zper = R.zb == BOUND_PERIODIC;
  float *D = reinterpret_cast<float *>(res_smem);  // [2][3][L.fl]
  ResPair *pairs = reinterpret_cast<ResPair *>(res_smem + (size_t)6 * 4 * L.fl);
  uint8_t *PT = res_smem + (size_t)6 * 4 * L.fl + (size_t)sizeof(ResPair) * L.pairs;  // [2][L.pt]
  // masked: per colour the pairs to update, those of bulk sites with all bonds
  // to bulk sites from the front, the others from the back
  uint16_t *lists = reinterpret_cast<uint16_t *>(PT + 2 * L.pt);  // [2][L.pairs]
  // neighbouring CTAs (the CTA itself when C = 1): their rows end where this
  // CTA's begin, and begin where this one's end
  const int prev = rank > 0 ? rank - 1 : C - 1, next = rank + 1 < C ? rank + 1 : 0;
  const int n_prev = cut[prev + 1] - cut[prev];
  const bool to_prev = rank > 0 || zper, to_next = rank + 1 < C || zper;
  const uint32_t base = smem_u32(D);
  const uint32_t rprev = map_rank(base, prev) + 4u * (uint32_t)(n_prev * hs);
  const uint32_t rnext = map_rank(base, next) - 4u * (uint32_t)(n * hs);
  const uint32_t bprev = map_rank(smem_u32(bars), prev), bnext = map_rank(smem_u32(bars), next);
  const uint32_t rcnt = map_rank(smem_u32(s_cnt), lane < C ? lane : 0);
  const uint32_t rcntb = map_rank(smem_u32(bars), lane < C ? lane : 0);
  // both colours of rows r0 - ny .. r0 + n + ny - 1 (zeros where z ends)
  for (int q = 0; q < 6; q++) {
    const float *g = a.dir + R.dir_off + (long long)q * R.plane;
    for (int i = tid; i < (n + 2 * ny) * (hs / 4); i += NT) {
      const int lr = i / (hs / 4), x = 4 * (i - lr * (hs / 4));
      int row = r0 - ny + lr;
      bool on = true;
      if (row < 0) { on = zper; row += rows_all; }
      if (row >= rows_all) { on = zper; row -= rows_all; }
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on) v = __ldcg(reinterpret_cast<const float4 *>(g + (long long)row * hs + x));
      *reinterpret_cast<float4 *>(D + (size_t)q * L.fl + lr * hs + x) = v;
    }
  }
  if (MASK) {
    for (int q = 0; q < 2; q++)
      for (int i = tid; i < (n + 2 * ny) * (hs / 4); i += NT) {
        const int lr = i / (hs / 4), x = 4 * (i - lr * (hs / 4));
        int row = r0 - ny + lr;
        bool on = true;
        if (row < 0) { on = zper; row += rows_all; }
        if (row >= rows_all) { on = zper; row -= rows_all; }
        uint32_t v = 0;
        if (on)
          v = *reinterpret_cast<const uint32_t *>(a.pt + R.pt_off + (long long)q * R.pplane + (long long)row * R.hps + x);
        *reinterpret_cast<uint32_t *>(PT + (size_t)q * L.pt + lr * hs + x) = v;
      }
  }
  for (int p = tid; p < np; p += NT) {
    const int l = (int)fastdiv((uint32_t)p, R.hp_m, R.hp_p), h0 = 2 * (p - l * hp), row = r0 + l;
    const int k = (int)fastdiv((uint32_t)row, R.ny_m, R.ny_p), j = row - k * ny;
    const int at = (ny + l) * hs;
    const bool hasB = h0 + 1 < R.hx;
    int f = ((j + k) & 1) | (hasB ? RF_HASB : 0);
    f |= (k + 1 < nz || zper ? RF_ZP : 0) | (k > 0 || zper ? RF_ZM : 0);
    int ex0 = h0 - 1, ex1 = hasB ? h0 + 2 : h0 + 1, jp = j + 1, jm = j - 1;
    f |= RF_EX0 | RF_EX1 | RF_YP | RF_YM;
    if (ex0 < 0) { if (R.xb == BOUND_PERIODIC) ex0 = R.hx - 1; else { f &= ~RF_EX0; ex0 = h0; } }
    if (ex1 == R.hx) { if (R.xb == BOUND_PERIODIC) ex1 = 0; else { f &= ~RF_EX1; ex1 = h0; } }
    if (jp == ny) { if (R.yb == BOUND_PERIODIC) jp = 0; else { f &= ~RF_YP; jp = j; } }
    if (jm < 0) { if (R.yb == BOUND_PERIODIC) jm = ny - 1; else { f &= ~RF_YM; jm = j; } }
    f |= (int)odd_tail<MASK>(R, h0) << RF_TAIL;
    if (to_prev && l < ny) f |= RF_PREV;
    if (to_next && l >= n - ny) f |= RF_NEXT;
    ResPair d;
    d.off = (uint16_t)(at + h0);
    d.yp = (uint16_t)(at + (jp - j) * hs + h0);
    d.ym = (uint16_t)(at + (jm - j) * hs + h0);
    d.ex0 = (uint16_t)(at + ex0);
    d.ex1 = (uint16_t)(at + ex1);
    d.flags = (uint16_t)f;
    d.zero = 0;
    pairs[p] = d;
  }
  int nb[2] = {0, 0}, nm[2] = {0, 0};  // masked: the lists' lengths
  if (MASK) {
    __shared__ unsigned s_w[2][kResThreads / 32];
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < 2; c++) {
      const uint8_t *Pc = PT + (size_t)c * L.pt, *Po = PT + (size_t)(1 - c) * L.pt;
      uint16_t *list = lists + (size_t)c * L.pairs;
#pragma unroll 1
      for (int q = 0; q < np; q += NT) {
        const int p = q + tid;
        int cls = 0;  // 1 bulk, 2 other
        if (p < np) {
          const ResPair d = pairs[p];
          const int f = d.flags, off = d.off, sl = (f ^ c) & 1, tail = (f >> RF_TAIL) & 3;
          const uint16_t ps = *reinterpret_cast<const uint16_t *>(Pc + off);
          const uint16_t t[5] = {*reinterpret_cast<const uint16_t *>(Po + off),
                                 *reinterpret_cast<const uint16_t *>(Po + d.yp),
                                 *reinterpret_cast<const uint16_t *>(Po + d.ym),
                                 *reinterpret_cast<const uint16_t *>(Po + off + dz),
                                 *reinterpret_cast<const uint16_t *>(Po + off - dz)};
          const uint8_t ex = Po[sl ? d.ex1 : d.ex0];
          bool any = ex != 0, bulk = ps == 0x0101 && tail == 0 && (f & RF_HASB) && (f & (sl ? RF_EX1 : RF_EX0)) &&
                                     (f & RF_ZP) && (f & RF_ZM) && (f & RF_YP) && (f & RF_YM) && ex != 0;
#pragma unroll
          for (int w = 0; w < 5; w++) {
            any = any || t[w] != 0;
            bulk = bulk && (t[w] & 0xFF) != 0 && (t[w] >> 8) != 0;
          }
          // a pair of two inactive sites: only the bonds of colour 1 to active
          // sites vary, and only a measured sweep counts them
          cls = bulk ? 1 : (ps != 0 || (MEAS && c == 1 && any) ? 2 : 0);
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, cls == 1), m2 = __ballot_sync(0xffffffffu, cls == 2);
        if (lane == 0) {
          s_w[0][tid >> 5] = __popc(m1);
          s_w[1][tid >> 5] = __popc(m2);
        }
        __syncthreads();
        int at1 = nb[c], at2 = nm[c], all1 = 0, all2 = 0;
        for (int w = 0; w < NT / 32; w++) {
          if (w < (tid >> 5)) {
            at1 += s_w[0][w];
            at2 += s_w[1][w];
          }
          all1 += s_w[0][w];
          all2 += s_w[1][w];
        }
        const unsigned below = (1u << lane) - 1u;
        if (cls == 1) list[at1 + __popc(m1 & below)] = (uint16_t)p;
        if (cls == 2) list[L.pairs - 1 - (at2 + __popc(m2 & below))] = (uint16_t)p;
        nb[c] += all1;
        nm[c] += all2;
        __syncthreads();
      }
    }
  }
  // pairs each pass receives: the ny rows on either side that another CTA (or,
  // across a periodic z, this one) owns, pairs of two inactive sites apart.
  __syncthreads();
  for (int q = tid; q < 4 * ny * hp; q += NT) {
    const int c = q & 1, lr = (q >> 1) / hp, h0 = 2 * ((q >> 1) - lr * hp);
    const bool low = lr < ny;
    const int at = (low ? lr : lr + n) * hs + h0;
    bool on = low ? to_prev : to_next;
    if (MASK) on = on && *reinterpret_cast<const uint16_t *>(PT + (size_t)c * L.pt + at) != 0;
    if (on) atomicAdd(&s_tx[c], 1u);
  }
  const uint32_t seed = R.seed, stream = R.stream, pid0 = (uint32_t)r0 * (uint32_t)hp;
  const unsigned long long sw0 = S->sweep, meas0 = S->meas;
  const unsigned frozen = S->frozen;
  const float invT = 1.0f / S->T;
  float ang = S->ang_var;
  unsigned long long total = 0;
  unsigned seen0 = 0, seen1 = 0;  // the counters two sweeps before
  cluster_arrive();
  cluster_wait();
  const uint32_t tx[2] = {24u * s_tx[0], 24u * s_tx[1]}, tx_cnt = 4u * (uint32_t)(NT / 32) * (uint32_t)C + extra;
  bool ok = true, gave_up = false;  // whether a wait of this thread, of any thread of the CTA ran out
  // the thread's first pair of each colour: its draw is made before the waits.
  // Masked: indices below nb32 are bulk pairs, so that a warp runs one kind
  const int nb32[2] = {(nb[0] + 31) & ~31, (nb[1] + 31) & ~31};
  auto pair_at = [&](int c, int q) {
    if (!MASK) return q < np ? q : -1;
    const uint16_t *list = lists + (size_t)c * L.pairs;
    if (q < nb32[c]) return q < nb[c] ? (int)list[q] : -1;
    return q - nb32[c] < nm[c] ? (int)list[L.pairs - 1 - (q - nb32[c])] : -1;
  };
  const int first[2] = {pair_at(0, tid), pair_at(1, tid)};
  const int count[2] = {MASK ? nb32[0] + nm[0] : np, MASK ? nb32[1] + nm[1] : np};
  uint4 rw0 = pair_draw(pid0 + (uint32_t)first[0], 0, sw0, seed, stream);
#pragma unroll 1
  for (int i = 0; i < nsweeps; i++) {
    const unsigned long long sw = sw0 + (unsigned long long)i;
    const uint32_t odd = (uint32_t)i & 1u;
    if (tid == 0) mbar_arrive_expect_tx(&bars[count_bar(i)], tx_cnt);
    unsigned acc = 0;
    SplitSums<MASK> sums;
    if (MEAS) sums.clear();
#pragma unroll 1
    for (int c = 0; c < 2; c++) {
      if (tid == 0) mbar_arrive_expect_tx(&bars[halo_bar(c, i)], tx[c]);
      float *Dc = D + (size_t)(3 * c) * L.fl;
      const float *Do = D + (size_t)(3 - 3 * c) * L.fl;
      const uint8_t *Pc = PT + (size_t)c * L.pt, *Po = PT + (size_t)(1 - c) * L.pt;
      const uint32_t rc = 4u * (uint32_t)(3 * c * L.fl);
      // the other colour's halo rows (colour 1's of the sweep before were
      // waited for at that sweep's end)
      if (c == 1 && ok) ok = res_wait(&bars[halo_bar(0, i)], halo_parity(0, i), limit);
      const uint32_t hb = 8u * (uint32_t)halo_bar(c, i);
#pragma unroll 1
      for (int q0 = tid; q0 < count[c]; q0 += NT) {
        const int p = q0 == tid ? first[c] : pair_at(c, q0);
        if (MASK && p < 0) continue;
        const bool bulk = !MASK || q0 < nb32[c];
        const ResPair d = pairs[p];
        const int f = d.flags, off = d.off, s = (f ^ c) & 1;
        uint16_t pself = 0x0101;
        uint8_t pex = 1;
        const int ex = s ? d.ex1 : d.ex0;
        OPair o0, yp, ym, op, om;
        if (MASK && !bulk) {
          pself = *reinterpret_cast<const uint16_t *>(Pc + off);
          pex = Po[ex];
          o0.pt = *reinterpret_cast<const uint16_t *>(Po + off);
          yp.pt = *reinterpret_cast<const uint16_t *>(Po + d.yp);
          ym.pt = *reinterpret_cast<const uint16_t *>(Po + d.ym);
          op.pt = *reinterpret_cast<const uint16_t *>(Po + off + dz);
          om.pt = *reinterpret_cast<const uint16_t *>(Po + off - dz);
        }
        float exv[3];
        float2 ax, ay, az;
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const float *o = Do + (size_t)q * L.fl;
          o0.v[q] = *reinterpret_cast<const float2 *>(o + off);
          yp.v[q] = *reinterpret_cast<const float2 *>(o + d.yp);
          ym.v[q] = *reinterpret_cast<const float2 *>(o + d.ym);
          op.v[q] = *reinterpret_cast<const float2 *>(o + off + dz);
          om.v[q] = *reinterpret_cast<const float2 *>(o + off - dz);
          exv[q] = o[ex];
        }
        ax = *reinterpret_cast<const float2 *>(Dc + off);
        ay = *reinterpret_cast<const float2 *>(Dc + L.fl + off);
        az = *reinterpret_cast<const float2 *>(Dc + 2 * L.fl + off);
        const uint4 rw = q0 == tid ? rw0 : pair_draw(pid0 + (uint32_t)p, c, sw, seed, stream);
        if (MASK && bulk)
          update_pair_draw<POT, false, FIELD, MODE, true>(a, R, c, s, true, 1.f, 1.f, 1.f, 1.f, o0, yp, ym, op, om, exv,
                                                          0x0101, 1, true, true, rw, 0, ang, invT, ax, ay, az, acc,
                                                          sums);
        else
          update_pair_draw<POT, MASK, FIELD, MODE, PER>(
              a, R, c, s, (f & RF_HASB) != 0, f & RF_EX0 ? 1.f : 0.f, f & RF_EX1 ? 1.f : 0.f, f & RF_YP ? 1.f : 0.f,
              f & RF_YM ? 1.f : 0.f, o0, yp, ym, op, om, exv, pself, pex, (f & RF_ZP) != 0, (f & RF_ZM) != 0, rw,
              (long long)off + (long long)(r0 - ny) * hs, ang, invT, ax, ay, az, acc, sums, (f >> RF_TAIL) & 3);
        *reinterpret_cast<float2 *>(Dc + off) = ax;
        *reinterpret_cast<float2 *>(Dc + L.fl + off) = ay;
        *reinterpret_cast<float2 *>(Dc + 2 * L.fl + off) = az;
        if (MASK && pself == 0) continue;  // measured only
        if (f & RF_PREV) {
          const uint32_t t = rprev + rc + 4u * (uint32_t)off, b = bprev + hb;
          st_remote(t, ax, b);
          st_remote(t + 4u * (uint32_t)L.fl, ay, b);
          st_remote(t + 8u * (uint32_t)L.fl, az, b);
        }
        if (f & RF_NEXT) {
          const uint32_t t = rnext + rc + 4u * (uint32_t)off, b = bnext + hb;
          st_remote(t, ax, b);
          st_remote(t + 4u * (uint32_t)L.fl, ay, b);
          st_remote(t + 8u * (uint32_t)L.fl, az, b);
        }
      }
      if (c == 0) {
        rw0 = pair_draw(pid0 + (uint32_t)first[1], 1, sw, seed, stream);
        __syncthreads();  // this CTA's rows of colour 0
      }
    }
    // the sweep's acceptances to every CTA's counter
    if (MASK && MEAS) {  // never true (no FP32 operation gives this NaN): a dependence on every pair's bonds
      const float2 e = unpk(sums.hi[0]);
      acc += (__float_as_uint(e.x) & __float_as_uint(e.y)) == 0xFFFFFFFFu;
    }
    const unsigned wa = __reduce_add_sync(0xffffffffu, acc);
    if (lane < C) red_remote(rcnt + 4u * odd, wa, rcntb + 8u * (uint32_t)count_bar(i));
    if (MEAS) {
      const double v = warp_split_sums(sums);
      double *ring = a.ring + (((size_t)r * (a.ring_cap + 1) +
                                (size_t)((meas0 + (unsigned long long)i) % (unsigned long long)a.ring_cap)) *
                                   kLanes +
                               (rank + (tid >> 5)) % kLanes) * kQ;
      if ((lane & 3) == 0 && lane < 4 * kQ && (MASK || lane != 4)) atomicAdd(ring + (lane >> 2), v);
      if (!MASK && lane == 1) atomicAdd(ring + 1, v);  // lane 1 holds lane 0's: with every site active, E of active sites is E
    }
    rw0 = pair_draw(pid0 + (uint32_t)first[0], 0, sw + 1, seed, stream);
    // this CTA's rows of colour 1, and whether a wait ran out since this barrier of the sweep before
    if (__syncthreads_or(!ok)) {
      gave_up = true;
      break;
    }
    ok = res_wait(&bars[halo_bar(1, i)], halo_parity(1, i), limit) &&
         res_wait(&bars[count_bar(i)], count_parity(i), limit);
    const unsigned sum = *(volatile unsigned *)&s_cnt[odd], sweep_acc = sum - (odd ? seen1 : seen0);
    if (odd) seen1 = sum;
    else seen0 = sum;
    total += sweep_acc;
    if (!frozen) ang = next_step(ang, sweep_acc, (unsigned)R.valid);
  }
  gave_up = __syncthreads_or(gave_up || !ok);
  if (gave_up && tid < C) set_remote(map_rank(smem_u32(&s_bad), tid), 1u);
  cluster_arrive();  // nobody sends any more, and unless one gave up every store to this CTA has landed: it may end
  cluster_wait();
  if (*(volatile unsigned *)&s_bad) {
    let_land();
    cluster_arrive();
    cluster_wait();
    if (tid == 0) atomicOr(a.err, 8u);
    if (MEAS && rank == 0 && tid == 0) S->meas = meas0 + (unsigned long long)nsweeps;  // the ring's slots are counted on the host too
    return;
  }
  // directors back (own rows), and the replica's state
  for (int q = 0; q < 6; q++) {
    float *g = a.dir + R.dir_off + (long long)q * R.plane + (long long)r0 * hs;
    const float *d = D + (size_t)q * L.fl + ny * hs;
    for (int i = tid; i < n * hs / 4; i += NT)
      reinterpret_cast<float4 *>(g)[i] = reinterpret_cast<const float4 *>(d)[i];
  }
  if (rank == 0 && tid == 0) {
    S->ang_var = ang;
    S->sweep = sw0 + (unsigned long long)nsweeps;
    if (MEAS) S->meas = meas0 + (unsigned long long)nsweeps;
    double *st = a.stats + (size_t)r * kStats;
    st[7] += (double)total;
    st[8] += (double)nsweeps;
    st[11] = (double)ang;
    st[12] = (double)(sw0 + (unsigned long long)nsweeps);
  }
}

template <int POT, bool MASK, bool FIELD, bool PER>
static const void *res_fn(int mode) {
  return mode == MODE_SWEEP_MEASURE ? (const void *)k_resident<POT, MASK, FIELD, MODE_SWEEP_MEASURE, PER>
                                    : (const void *)k_resident<POT, MASK, FIELD, MODE_SWEEP, PER>;
}

template <int POT>
static const void *res_fn_p(const Variant &v, int mode) {
  if (v.mask) return v.field ? res_fn<POT, true, true, false>(mode) : res_fn<POT, true, false, false>(mode);
  if (v.per) return v.field ? res_fn<POT, false, true, true>(mode) : res_fn<POT, false, false, true>(mode);
  return v.field ? res_fn<POT, false, true, false>(mode) : res_fn<POT, false, false, false>(mode);
}

static const void *res_kernel(const Variant &v, int mode) {
  return v.pot == POT_LL ? res_fn_p<POT_LL>(v, mode)
                         : (v.pot == POT_PEAR ? res_fn_p<POT_PEAR>(v, mode) : res_fn_p<POT_GHRL>(v, mode));
}

// Shared memory of a CTA when the largest share is n rows, and its pairs.
long long resident_smem_bytes(const RepDev &R, bool mask, int n) {
  const ResLayout L = res_layout(R, n);
  if (L.fl > 65535 || L.pairs > 65535) return 1ll << 40;  // offsets and lists are 16 bits
  return 24ll * L.fl + (long long)sizeof(ResPair) * L.pairs + (mask ? 2ll * L.pt + 4ll * L.pairs : 0);
}

int resident_max_threads(bool mask, int mode) {
  return mask && mode == MODE_SWEEP_MEASURE ? kResMaskThreads : kResThreads;
}

static void res_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at, int nrep, int C, int nt, int smem,
                       cudaStream_t st) {
  cfg.gridDim = dim3(nrep * C);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
}

// Sets the kernels' attributes: the largest values any engine uses, because they
// belong to the kernel.
bool resident_prepare(const Variant &v) {
  for (int mode : {MODE_SWEEP, MODE_SWEEP_MEASURE}) {
    const void *fn = res_kernel(v, mode);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

// Clusters of C CTAs of nt threads with smem bytes the GPU holds at once (0:
// the shape cannot run).
int resident_clusters(const Variant &v, int mode, int C, int nt, int smem) {
  const void *fn = res_kernel(v, mode);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  res_config(cfg, at, 1, C, nt, smem, nullptr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_resident(const Variant &v, int mode, const PassArgs &a, const int *cut, int nrep, int nsweeps,
                            int C, int nt, int smem, cudaStream_t st, unsigned long long limit, unsigned extra) {
  PassArgs args = a;
  int ns = nsweeps, cc = C;
  const int *ct = cut;
  void *params[] = {&args, &ct, &ns, &cc, &limit, &extra};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  res_config(cfg, at, nrep, C, nt, smem, st);
  return cudaLaunchKernelExC(&cfg, res_kernel(v, mode), params);
}

}  // namespace mcx
