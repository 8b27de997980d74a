// Test-only program: prints the rings that the CTA-pair kernel is compiled with, one "key=value ..." line per configuration.
// Host code only (nothing is launched).  Built by __graft_entry__.build(); read by tests/test_pair_waits.py.
#include <cstdio>

#include "../../awesome-cute_b200/csrc/w4a16_kernel_2sm.cuh"

template <int TM, int KS, int OUT, int P>
void row() {
  using C = w4a16::Config2<TM, KS, OUT, P>;
  std::printf("tm=%d out=%d p=%d w_slots=%d a_slots=%d bufs=%d sets=%d\n", TM, OUT, P, C::W_SLOTS, C::A_SLOTS, C::WBUFS, C::NSETS);
}
template <int OUT, int P>
void rows() {
  row<32, 256, OUT, P>(), row<64, 256, OUT, P>(), row<128, 128, OUT, P>(), row<192, 128, OUT, P>();
}

int main() {
  using namespace w4a16;
  rows<OUT_PLAIN, 1>(), rows<OUT_GATHER, 1>(), rows<OUT_TMA, 1>(), rows<OUT_DUAL, 1>();
  rows<OUT_PLAIN, 2>(), rows<OUT_PLAIN, 3>(), rows<OUT_PLAIN, 4>();
  return 0;
}
