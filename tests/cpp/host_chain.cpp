// Test-only library: the ordering rules of host-buffer calls behind a C interface (loaded by tests/test_host_chain.py).
#include "../../awesome-cute_b200/csrc/w4a16_host_chain.h"

using w4a16::HostBuffers;
using w4a16::HostChain;
using w4a16::Place;

extern "C" {
void *chain_new() { return new HostChain; }
void chain_delete(void *c) { delete static_cast<HostChain *>(c); }
int chain_order(void *c, const Place *p, uint64_t count, const HostBuffers *b) {
  return static_cast<HostChain *>(c)->order(*p, count, *b);
}
void chain_record(void *c, const Place *p, uint64_t seen, uint64_t now, int how, const HostBuffers *b) {
  static_cast<HostChain *>(c)->record(*p, seen, now, static_cast<w4a16::CopyIn>(how), *b);
}
void chain_forget(void *c, const Place *p) { static_cast<HostChain *>(c)->forget(*p); }
}
