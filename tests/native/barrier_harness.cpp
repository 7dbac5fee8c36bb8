// Host build of pointvortex_b200/csrc/pv_barrier.cuh for the CPU tests (tests/test_barrier_word.py).
#include "../../pointvortex_b200/csrc/pv_barrier.cuh"

using namespace pvb;

extern "C" {
unsigned pvl_max_ctas() { return barrier::kMaxCtas; }
unsigned long long pvl_arrival(int error, unsigned parity) { return barrier::arrival(error != 0, parity); }
unsigned long long pvl_arrivals(unsigned ctas) { return barrier::arrivals(ctas); }
int pvl_open(unsigned long long word, unsigned long long open_at) { return barrier::open(word, open_at); }
int pvl_errors(unsigned long long word, unsigned parity) { return barrier::errors(word, parity); }
unsigned long long pvl_broken(unsigned parity) { return barrier::broken(parity); }
}
