// Runs the operand rings' order of copies, products and waits (bpx_ring.h) on the host, for every size and
// with each wait in turn giving up, and checks that a place is refilled only when its copy has been
// consumed, that waits name the right phase, and that no copy is in flight when the order returns.
#include <cstdio>
#include <cstdlib>

#include "bpx_ring.h"

static int g_runs = 0;
#define CHECK(x)                                                            \
  do {                                                                      \
    if (!(x)) {                                                             \
      std::printf("%s:%d: %s (run %d)\n", __FILE__, __LINE__, #x, g_runs);  \
      std::exit(1);                                                         \
    }                                                                       \
  } while (0)

constexpr int kPlaces = 16;

struct Places {
  int copies[kPlaces] = {}, products[kPlaces] = {};
  bool in_flight[kPlaces] = {}, consumed[kPlaces] = {};
  int waits = 0, give_up = -1;

  bool wait() { return waits++ != give_up; }
  void land(int s, uint32_t ph) {
    CHECK(copies[s] > 0 && ph == (uint32_t)((copies[s] - 1) & 1));
    in_flight[s] = false;
  }
  void issue(int s) {
    CHECK(copies[s] == 0 || consumed[s]);
    CHECK(!in_flight[s]);
    ++copies[s];
    in_flight[s] = true;
    consumed[s] = false;
  }
  void drain(int s, uint32_t ph) { land(s, ph); }
  void at_rest() const {
    for (int s = 0; s < kPlaces; ++s) CHECK(!in_flight[s]);
  }
};

struct Contract : Places {
  int next_copy = 0, next_product = 0, finished = 0;
  void copy(int c, int s) {
    CHECK(c == next_copy++);
    issue(s);
  }
  bool wait_full(int s, uint32_t ph) {
    if (!wait()) return false;
    land(s, ph);
    return true;
  }
  void multiply(int c, int s) {
    CHECK(c == next_product++ && !in_flight[s] && !finished);
    ++products[s];
  }
  bool wait_empty(int s, uint32_t ph) {
    if (!wait()) return false;
    CHECK(products[s] > 0 && ph == (uint32_t)((products[s] - 1) & 1));
    consumed[s] = true;
    return true;
  }
  void finish() { ++finished; }
};

constexpr int kLayers = 5, kSpans = 4, kRing = 10, kHalves = 2;
using Ring = bpx::gemm::RingChain<kLayers, kSpans, kRing, kHalves>;

// the copying thread alone: the pieces that the multiplying thread has not reached stay in flight
struct Chain : Places {
  int issued = 0, layer_ = 0, chunk_ = 0, half_ = 0, span_piece[kSpans], nk0;
  bool free_piece[512] = {};
  explicit Chain(int n) : nk0(n) {}
  bool wait_empty(int s, uint32_t ph) {
    CHECK(copies[s] > 0 && ph == (uint32_t)((copies[s] - 1) & 1));
    if (!wait()) return false;
    in_flight[s] = false;  // the product that frees the place has waited for its copy
    consumed[s] = true;
    free_piece[(copies[s] - 1) * kRing + s] = true;
    return true;
  }
  void copy(int layer, int kc, int half, int s) {
    CHECK(layer == layer_ && kc == chunk_ && half == half_ && s == issued % kRing);
    if (layer == 0 && half == 0) {
      if (kc >= kSpans) CHECK(free_piece[span_piece[kc % kSpans]]);
    }
    if (layer == 0) span_piece[kc % kSpans] = issued;  // its last half, in the end
    issue(s);
    ++issued;
    if (++half_ == Ring::halves(layer_)) {
      half_ = 0;
      if (++chunk_ == Ring::chunks(layer_, nk0)) {
        chunk_ = 0;
        ++layer_;
      }
    }
  }
};

int main() {
  for (int stages = 2; stages <= 4; ++stages)
    for (int chunks = 1; chunks <= 14; ++chunks) {
      int waits = 0;
      for (int give_up = -1; give_up < waits; ++give_up, ++g_runs) {
        Contract c;
        c.give_up = give_up;
        const bool ok = bpx::gemm::ring_contract(c, chunks, stages);
        CHECK(ok == (give_up < 0) && c.finished == 1);
        CHECK(!ok || c.next_product == chunks);
        c.at_rest();
        if (give_up < 0) waits = c.waits;
      }
    }
  for (int nk0 = 1; nk0 <= 12; ++nk0) {
    int waits = 0;
    for (int give_up = -1; give_up < waits; ++give_up, ++g_runs) {
      Chain c(nk0);
      c.give_up = give_up;
      const bool ok = Ring::copy(c, nk0);
      CHECK(ok == (give_up < 0));
      CHECK(!ok || c.issued == kHalves * (nk0 + (kLayers - 2) * kSpans) + kSpans);
      c.at_rest();
      if (give_up < 0) waits = c.waits;
    }
  }
  std::printf("%d runs\n", g_runs);
  return 0;
}
