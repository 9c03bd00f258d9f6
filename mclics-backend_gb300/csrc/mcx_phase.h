// mcx_phase.h -- which mbarrier of a CTA counts what in the resident sweeps
// (mcx_resident.cu), and the phase parity to wait for.
//
// Each barrier is armed once per use with the bytes of that use.  Bytes of a
// later use must not reach a barrier whose phase of an earlier use is still
// short of bytes, or they complete it in the missing ones' place:
//   - halo rows of colour 0: a CTA sends those of sweep i + 1 after it has the
//     acceptances of sweep i from every warp, and a warp sends its acceptances
//     after its waits for the halo rows of colour 0 of sweep i: one barrier;
//   - halo rows of colour 1: a CTA sends those of sweep i + 1 after it has the
//     rows of colour 0 of sweep i + 1 that others send it.  That says something
//     about a neighbour only if the neighbour sends it a row: where a mask has
//     active sites of one colour only next to a cut, it may send none, and may
//     still be waiting for a third CTA's rows of sweep i.  So even and odd sweeps
//     have barriers of their own; rows of sweep i + 2 follow every warp's
//     acceptances of sweep i + 1, which follow its waits at the end of sweep i;
//   - acceptances: even and odd sweeps, for the same reason.
#pragma once

#if defined(__CUDACC__)
#define MCX_PHASE __host__ __device__ __forceinline__
#else
#define MCX_PHASE static inline
#endif

namespace mcx {

constexpr int kResBars = 5;
MCX_PHASE int halo_bar(int colour, int sweep) { return colour == 0 ? 0 : 1 + (sweep & 1); }
MCX_PHASE unsigned halo_parity(int colour, int sweep) { return (unsigned)(colour == 0 ? sweep : sweep >> 1) & 1u; }
MCX_PHASE int count_bar(int sweep) { return 3 + (sweep & 1); }
MCX_PHASE unsigned count_parity(int sweep) { return (unsigned)(sweep >> 1) & 1u; }

}  // namespace mcx
