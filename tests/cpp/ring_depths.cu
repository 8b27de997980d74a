// Test-only program: prints the ring depths that the kernels are compiled with, one "kernel key=value ..." line per
// configuration.  Host code only (nothing is launched).  Built by __graft_entry__.build(); read by tests/test_ring_waits.py.
#include <cstdio>

#include "../../awesome-cute_b200/csrc/w4a16_kernel_decode.cuh"

template <int OUT, int CL>
void decode() {
  using C = w4a16::DecodeConfig<OUT, CL>;
  std::printf("decode out=%d cl=%d stages=%d sets=%d bufs=%d accs=%d buf_first=%d\n", OUT, CL, C::STAGES, C::NSETS, C::WBUFS, C::NACC,
              (int)C::BUF_FIRST);
}

int main() {
  using namespace w4a16;
  decode<OUT_PLAIN, 1>();
  decode<OUT_GATHER, 1>();
  decode<OUT_TMA, 1>();
  decode<OUT_DUAL, 1>();
  decode<OUT_PLAIN, 2>();
  decode<OUT_PLAIN, 4>();
  decode<OUT_PLAIN, 8>();
  decode<OUT_DUAL, 2>();
  decode<OUT_DUAL, 4>();
  decode<OUT_DUAL, 8>();
  return 0;
}
