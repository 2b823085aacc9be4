// lc_scan.cu — device-wide exclusive scans of u32 counts whose length may live
// in device memory (so a captured step needs no host round trip).  Replaces
// the host-synchronous CubWrap::ExclusiveSumInPlace / SelectFlagged count
// read-backs of Core/CubWrappers.cuh:26-50, 77-89.
//
// One launch, one or two independent scans (blockIdx.y).  Block b (blocks take
// their index by ticket) owns the contiguous range [b chunk, (b + 1) chunk),
// chunk a whole number of tiles: it sums its range, publishes the sum, adds up
// the sums of all blocks before it, and writes its range out.  Every sum is
// published before its block waits and a block only waits on blocks that
// started before it, so the wait always ends; it is bounded all the same (a
// wait that gives up is reported and goes on with the sums it saw, so offsets
// never exceed the true total).  A range of one tile stays in registers between
// the two halves.  The last block to finish clears the published sums for the
// next launch.  Integer sums: the result does not depend on the schedule.
//
// What bounds it is launches, not bytes.  A scan was three launches (reduce,
// scan of the 1024 sums, write), and a step has five scans: three launches now.
// One 32x32 cloth's step 293 -> 281 us; a hash broadphase of 20,011 objects
// (three scans) 380 -> 358; a million counts take as long as before.
#include <cuda/atomic>

#include "lc_internal.cuh"

namespace lc {

namespace {

constexpr int kScanItems = 16;  // per thread per tile
constexpr uint32_t kScanTile = kThreads * kScanItems;
constexpr uint32_t kScanSpins = 1u << 22;  // bound on the wait for one published sum
constexpr unsigned long long kScanValid = 1ull << 32;

struct ScanState {
    unsigned long long sum[kScanBlocks];  // kScanValid | sum of the block's range; 0: not published
    uint32_t ticket, done;
};
static_assert(2 * sizeof(ScanState) <= kScanScratch * sizeof(uint32_t), "scan scratch");

__device__ __forceinline__ uint32_t block_sum(uint32_t v) {
    __shared__ uint32_t s[kThreads / 32];
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) t += s[w];
    return t;
}

// Exclusive scan of one value per thread; total: the block's sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t &total) {
    __shared__ uint32_t s[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) s[wid] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        if (w < wid) before += s[w];
        total += s[w];
    }
    return before + incl - v;
}

// A thread's 16 consecutive values of the tile at base (zeros past end);
// vec: the arrays start on 16-byte boundaries, as cudaMalloc's do, and so does
// every thread's run of a tile.
__device__ __forceinline__ void load_tile(const uint32_t *__restrict__ in, uint64_t base, uint64_t end, bool vec,
                                          uint32_t v[kScanItems]) {
    const uint64_t mine = base + (uint64_t)threadIdx.x * kScanItems;
    if (vec && mine + kScanItems <= end) {
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            const uint4 a = *reinterpret_cast<const uint4 *>(in + mine + 4 * q);
            v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = a.z; v[4 * q + 3] = a.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = mine + k < end ? in[mine + k] : 0u;
    }
}

__device__ __forceinline__ uint32_t sum_of(const uint32_t v[kScanItems]) {
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    return s;
}

// Writes the tile's exclusive sums from carry on; returns the next carry.
__device__ __forceinline__ uint32_t store_tile(uint32_t *__restrict__ out, uint64_t base, uint64_t end, bool vec,
                                               const uint32_t v[kScanItems], uint32_t carry) {
    uint32_t total;
    uint32_t ex = carry + block_scan(sum_of(v), total);
    const uint64_t mine = base + (uint64_t)threadIdx.x * kScanItems;
    uint32_t o[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        o[k] = ex;
        ex += v[k];
    }
    if (vec && mine + kScanItems <= end) {
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q)
            *reinterpret_cast<uint4 *>(out + mine + 4 * q) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (mine + k < end) out[mine + k] = o[k];
    }
    return carry + total;
}

__global__ void __launch_bounds__(kThreads) k_scan(ScanJob j0, ScanJob j1, ScanState *states, uint32_t *err) {
    const ScanJob j = blockIdx.y ? j1 : j0;
    ScanState &st = states[blockIdx.y];
    __shared__ uint32_t s_block, s_last;
    if (threadIdx.x == 0) s_block = atomicAdd(&st.ticket, 1u);
    __syncthreads();
    const uint32_t b = s_block, G = gridDim.x;
    const uint32_t n = min(j.n_dev ? *j.n_dev : j.n_static, j.n_cap);
    const uint64_t chunk = (((uint64_t)n + G - 1) / G + kScanTile - 1) / kScanTile * kScanTile;
    const uint64_t b0 = min((uint64_t)n, b * chunk), b1 = min((uint64_t)n, b0 + chunk);
    const bool vec = ((reinterpret_cast<uintptr_t>(j.in) | reinterpret_cast<uintptr_t>(j.out)) & 15u) == 0;
    const bool one = b1 - b0 <= kScanTile;
    uint32_t v[kScanItems];
    uint32_t own = 0;
    if (b0 < b1) {
        for (uint64_t base = b0; base < b1; base += kScanTile) {
            load_tile(j.in, base, b1, vec, v);
            own += sum_of(v);
        }
        own = block_sum(own);
    }
    using Word = cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>;
    if (threadIdx.x == 0) Word(st.sum[b]).store(kScanValid | own, cuda::memory_order_relaxed);
    if (b0 < b1 || b == G - 1) {  // the last block also reports the total
        uint32_t before = 0;
        for (uint32_t k = threadIdx.x; k < b; k += kThreads) {
            unsigned long long w;
            uint32_t spins = 0;
            while (!((w = Word(st.sum[k]).load(cuda::memory_order_relaxed)) & kScanValid)) {
                if (++spins > kScanSpins) {
                    if (err) atomicOr(err, ERR_SORT);
                    break;
                }
                if (spins > 8) __nanosleep(20);
            }
            before += (uint32_t)w;
        }
        uint32_t carry = block_sum(before);
        if (one && b0 < b1) {
            carry = store_tile(j.out, b0, b1, vec, v, carry);
        } else {
            for (uint64_t base = b0; base < b1; base += kScanTile) {
                load_tile(j.in, base, b1, vec, v);
                carry = store_tile(j.out, base, b1, vec, v, carry);
            }
        }
        if (b == G - 1 && threadIdx.x == 0) {
            j.out[n] = carry;
            if (j.total) *j.total = carry;
            if (j.total64) *j.total64 = carry;
        }
    }
    __syncthreads();  // every wait of this block is over
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&st.done, 1u) == G - 1;
    }
    __syncthreads();
    if (s_last) {
        for (uint32_t k = threadIdx.x; k < G; k += kThreads) st.sum[k] = 0ull;
        if (threadIdx.x == 0) st.ticket = st.done = 0u;
    }
}

}  // namespace

// Each out holds n + 1 entries; out[n] = total.  scratch: kScanScratch u32,
// zero before the first scan that uses it and left zero by each; scans that
// share it are ordered on one stream.  b may be null.
void scan_u32(const ScanJob &a, const ScanJob *b, uint32_t *scratch, uint32_t *err, cudaStream_t st) {
    const uint32_t cap = b && b->n_cap > a.n_cap ? b->n_cap : a.n_cap;
    // one tile per block up to two blocks per SM, then more tiles each
    uint32_t g = (cap + kScanTile - 1) / kScanTile;
    g = g < 1 ? 1 : g > kScanBlocks ? kScanBlocks : g;
    k_scan<<<dim3(g, b ? 2 : 1), kThreads, 0, st>>>(a, b ? *b : a, reinterpret_cast<ScanState *>(scratch), err);
}

}  // namespace lc
