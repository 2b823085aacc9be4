// A scan whose wait ran past its bound, for the entries that report it: the
// engine's scan and then, when told to, the error bit that a wait sets when it
// gives up.  Linked in place of lc_scan.cu (tests/test_scan_timeout_gpu.py).
#include "../../licenta_gb300/csrc/lc_internal.cuh"

#include <string>

#define scan_u32 scan_u32_engine
#include "../../licenta_gb300/csrc/lc_scan.cu"
#undef scan_u32

namespace lc {

static int g_give_up = 0;
static __global__ void k_gave_up(uint32_t *err) { atomicOr(err, ERR_SORT); }

void scan_u32(const ScanJob &a, const ScanJob *b, uint32_t *scratch, uint32_t *err, cudaStream_t st) {
    scan_u32_engine(a, b, scratch, err, st);
    if (err && g_give_up) k_gave_up<<<1, 1, 0, st>>>(err);
}

void set_last_error(const std::string &) {}

}  // namespace lc

extern "C" void set_give_up(int on) { lc::g_give_up = on; }
