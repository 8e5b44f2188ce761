// bpx_ring.h -- the order of copies, products and bounded waits in the operand rings of the tcgen05 kernels
// (bpx_gemm.cu).  Ops does the steps; tests/c_host/ring_check.cpp runs the same order on the host with each
// wait in turn giving up.
//
// A copy into shared memory must not outlive its CTA nor land in memory that has been given another use.  So
// whichever wait gives up, every copy issued is waited for (again with a limit) before the order returns:
// of `issued` copies, piece p into place p % ring, those before the last `ring` have been consumed.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define BPX_RING_FN __device__ __forceinline__
#else
#define BPX_RING_FN inline
#endif

namespace bpx {
namespace gemm {

template <class Ops>
BPX_RING_FN void ring_drain(Ops& ops, int issued, int ring) {
  for (int p = issued > ring ? issued - ring : 0; p < issued; ++p) ops.drain(p % ring, (uint32_t)(p / ring) & 1u);
}

// One thread copies and multiplies `chunks` chunks through `stages` places.  Ops: copy(chunk, place),
// wait_full(place, phase), multiply(chunk, place), which frees the place when it has completed,
// wait_empty(place, phase), finish() after the last product, drain(place, phase).
template <class Ops>
BPX_RING_FN bool ring_contract(Ops& ops, int chunks, int stages) {
  int issued = 0, s = 0;
  uint32_t ph = 0;
  bool ok = true;
  for (; issued < stages && issued < chunks; ++issued) ops.copy(issued, issued);
  for (int c = 0; c < chunks; ++c) {
    ok = ops.wait_full(s, ph);
    if (!ok) break;
    ops.multiply(c, s);
    if (issued < chunks) {
      ok = ops.wait_empty(s, ph);
      if (!ok) break;
      ops.copy(issued++, s);
    }
    if (++s == stages) {
      s = 0;
      ph ^= 1;
    }
  }
  ops.finish();
  if (!ok) ring_drain(ops, issued, stages);
  return ok;
}

// The pieces of a chain of layers, in order of use: layer, chunk of K, half of the columns (the last layer
// has one half).  The first layer has nk0 chunks of inputs, which come with its first halves through
// `spans` places of their own; the other layers have `spans` chunks.
template <int LAYERS, int SPANS, int RING, int HALVES>
struct RingChain {
  static BPX_RING_FN int chunks(int layer, int nk0) { return layer == 0 ? nk0 : SPANS; }
  static BPX_RING_FN int halves(int layer) { return layer == LAYERS - 1 ? 1 : HALVES; }

  // The copying thread.  Ops: wait_empty(place, phase), copy(layer, chunk, half, place), drain(place, phase).
  // Another thread multiplies and can give up after the last copy has been issued, so this one ends with the
  // pieces in flight in any case.
  template <class Ops>
  static BPX_RING_FN bool copy(Ops& ops, int nk0) {
    int p = 0, slot = 0;
    uint32_t ph = 1;  // of the slot's previous piece; the first round finds its slots empty
    bool ok = true;
    for (int layer = 0; layer < LAYERS && ok; ++layer) {
      const int nh = halves(layer), nk = chunks(layer, nk0);
      for (int kc = 0; kc < nk && ok; ++kc)
        for (int half = 0; half < nh; ++half) {
          ok = p < RING || ops.wait_empty(slot, ph);
          if (ok && layer == 0 && half == 0 && kc >= SPANS) {  // the chunk that was in this span
            const int q = p - HALVES * SPANS + HALVES - 1;
            ok = ops.wait_empty(q % RING, (uint32_t)(q / RING) & 1u);
          }
          if (!ok) break;
          ops.copy(layer, kc, half, slot);
          ++p;
          if (++slot == RING) {
            slot = 0;
            ph ^= 1;
          }
        }
    }
    ring_drain(ops, p, RING);
    return ok;
  }
};

}  // namespace gemm
}  // namespace bpx
