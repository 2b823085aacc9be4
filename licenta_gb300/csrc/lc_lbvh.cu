// lc_lbvh.cu — triangle boxes + Morton codes, segmented stable radix sort,
// Karras hierarchy, bottom-up refit, leaf-vs-tree traversal, pair
// compaction and the VF/EE narrowphase (feature AABB cull + CCD).
//
// Compiled with -fmad=false: every float expression here keeps the separate
// roundings of the reference kernels, so Morton codes, tree topology, pair
// lists and contact lists are bit-exact against the FP32 oracle for the
// same input positions.
#include <algorithm>
#include <cooperative_groups.h>
#include <cuda/atomic>

#include "lc_internal.cuh"

namespace cg = cooperative_groups;

namespace lc {

// ---------------------------------------------------------------------------
// Morton encoding: Core/CudaUtils.cu:278-325 (REF63) and the commented 30-bit
// variant at :289-308 (K30).  Bit k of an axis goes to bit 3k.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ unsigned long long spread21(unsigned long long v) {
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}
__host__ __device__ __forceinline__ unsigned long long spread10(unsigned long long v) {
    v &= 0x3ffull;
    v = (v | (v << 16)) & 0x30000ffull;
    v = (v | (v << 8)) & 0x300f00full;
    v = (v | (v << 4)) & 0x30c30c3ull;
    v = (v | (v << 2)) & 0x9249249ull;
    return v;
}
__host__ __device__ __forceinline__ unsigned long long morton3(float x, float y, float z, int mode) {
    if (mode == LC_MORTON_K30) {
        unsigned long long qx = (unsigned long long)fminf(fmaxf(x * 1024.f, 0.0f), 1023.0f);
        unsigned long long qy = (unsigned long long)fminf(fmaxf(y * 1024.f, 0.0f), 1023.0f);
        unsigned long long qz = (unsigned long long)fminf(fmaxf(z * 1024.f, 0.0f), 1023.0f);
        return (spread10(qx) << 2) + (spread10(qy) << 1) + spread10(qz);
    }
    unsigned long long qx = (unsigned long long)fminf(fmaxf(x * 2097152.f, 0.0f), 2097151.0f);
    unsigned long long qy = (unsigned long long)fminf(fmaxf(y * 2097152.f, 0.0f), 2097151.0f);
    unsigned long long qz = (unsigned long long)fminf(fmaxf(z * 2097152.f, 0.0f), 2097151.0f);
    return (spread21(qx) << 2) + (spread21(qy) << 1) + spread21(qz);
}

unsigned long long morton3_host(float x, float y, float z, int mode) { return morton3(x, y, z, mode); }

// ---------------------------------------------------------------------------
// Triangle update: Physics/CudaDeformableUtils.cu:120-151.  One thread per
// slot; the swept, thickness-inflated box goes to leaf (T-1+slot) — the
// pre-sort slot, which is the reference's leaf-AABB quirk — or to a
// temporary, by original triangle, that the post-sort gather places under the
// sorted leaf.  The keys, with the original triangle as payload, start in the
// alternate buffers: after an even number of passes they are there again, and
// the post-sort writes the final order to keys and perm.
// ---------------------------------------------------------------------------
__global__ void k_triangles(DevPtrs d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.Ttot) return;
    const int c = d.tcloth[s];
    const ClothDev &cd = d.cloth[c];
    const int local = s - cd.t_off;
    const uint32_t orig = d.perm[s];
    const int4 t = d.tri[orig];
    const float3 a = xyz(d.x[t.x]), b = xyz(d.x[t.y]), cc = xyz(d.x[t.z]);
    const float3 pa = xyz(d.xp[t.x]), pb = xyz(d.xp[t.y]), pc = xyz(d.xp[t.z]);
    const float h = cd.h;
    d.fn[orig] = f4(normalize(cross(sub(b, a), sub(cc, a))), 0.f);
    const float3 mn = subc(min3(a, b, cc), h), mx = addc(max3(a, b, cc), h);
    const float3 pmn = subc(min3(pa, pb, pc), h), pmx = addc(max3(pa, pb, pc), h);
    const float3 smn = vmin(mn, pmn), smx = vmax(mx, pmx);
    if (cd.leaf_quirk) {
        const int node = cd.n_off + (cd.T - 1) + local;
        d.nmin[node] = f4(smn, 0.f);
        d.nmax[node] = f4(smx, 0.f);
    } else {
        d.leaf_tmp_min[orig] = f4(smn, 0.f);
        d.leaf_tmp_max[orig] = f4(smx, 0.f);
    }
    if (local == 0 && d.eq3) d.eq3[c] = 0;
    if (s == 0) *d.nfar = 0;
    const float3 mid = add(smn, dvs(sub(smx, smn), 2.f));
    const float qx = (mid.x - cd.morton_origin[0]) * cd.morton_scale;
    const float qy = (mid.y - cd.morton_origin[1]) * cd.morton_scale;
    const float qz = (mid.z - cd.morton_origin[2]) * cd.morton_scale;
    d.keys_alt[s] = morton3(qx, qy, qz, cd.morton_mode);
    d.payload_alt[s] = orig;
}

// Standalone LBVH: leaf boxes supplied by the caller (one cloth, T slots).
__global__ void k_leaves_from_boxes(DevPtrs d, const float *__restrict__ bmin, const float *__restrict__ bmax,
                                    int T, int mode) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= T) return;
    const float3 mn = f3(bmin[3 * s], bmin[3 * s + 1], bmin[3 * s + 2]);
    const float3 mx = f3(bmax[3 * s], bmax[3 * s + 1], bmax[3 * s + 2]);
    d.leaf_tmp_min[s] = f4(mn, 0.f);
    d.leaf_tmp_max[s] = f4(mx, 0.f);
    const float3 mid = add(mn, dvs(sub(mx, mn), 2.f));
    d.keys_alt[s] = morton3(mid.x, mid.y, mid.z, mode);
    d.payload_alt[s] = (uint32_t)s;
    if (s == 0 && d.eq3) d.eq3[0] = 0;
    if (s == 0) *d.nfar = 0;
}

// ---------------------------------------------------------------------------
// Segmented stable LSD radix sort of (u64 key, u32 payload), 8-bit digits.
// Tiles never straddle cloths, so every pass ranks keys within their own
// cloth: the result equals a stable sort of each cloth's slots by key, the
// order CUB's SortPairs gives at Physics/CudaDeformableUtils.cu:346-349.
// ---------------------------------------------------------------------------
__global__ void k_sort_hist(DevPtrs d, const unsigned long long *__restrict__ keys, int shift) {
    __shared__ uint32_t hist[kSortBuckets];
    const int tile = blockIdx.x;
    for (int i = threadIdx.x; i < kSortBuckets; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int c = d.stile_cloth[tile];
    const int start = d.stile_start[tile];
    const ClothDev &cd = d.cloth[c];
    const int end = min(start + kSortTile, cd.t_off + cd.T);
    for (int i = start + threadIdx.x; i < end; i += blockDim.x) {
        const uint32_t dig = (uint32_t)(keys[i] >> shift) & (kSortBuckets - 1);
        atomicAdd(&hist[dig], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortBuckets; i += blockDim.x) d.shist[(size_t)tile * kSortBuckets + i] = hist[i];
}

// One block per cloth: turns the per-tile digit counts into global scatter
// offsets (digit-major, tile-minor within the cloth).  kOffsetsSplit threads
// per digit each take a contiguous quarter of the cloth's tiles, with their
// loads unrolled, so a cloth of hundreds of tiles (one segment of a million
// keys) is not one serial chain of loads per digit.
constexpr int kOffsetsSplit = 4;
__global__ void __launch_bounds__(kSortBuckets * kOffsetsSplit) k_sort_offsets(DevPtrs d,
                                                                               const int *__restrict__ tile_first) {
    const int c = blockIdx.x;
    const int d0 = threadIdx.x % kSortBuckets, q = threadIdx.x / kSortBuckets;
    const int t0 = tile_first[c], t1 = tile_first[c + 1];
    const int per = (t1 - t0 + kOffsetsSplit - 1) / kOffsetsSplit;
    const int a = min(t1, t0 + q * per), e = min(t1, a + per);
    uint32_t part = 0;
#pragma unroll 8
    for (int t = a; t < e; ++t) part += d.shist[(size_t)t * kSortBuckets + d0];
    __shared__ uint32_t qs[kOffsetsSplit][kSortBuckets];
    __shared__ uint32_t s[kSortBuckets];
    qs[q][d0] = part;
    __syncthreads();
    // digit totals, then their exclusive scan (threads of quarter 0)
    uint32_t tot = 0;
    if (q == 0) {
#pragma unroll
        for (int k = 0; k < kOffsetsSplit; ++k) tot += qs[k][d0];
        s[d0] = tot;
    }
    __syncthreads();
    for (int o = 1; o < kSortBuckets; o <<= 1) {
        const uint32_t v = (q == 0 && d0 >= o) ? s[d0 - o] : 0u;
        __syncthreads();
        if (q == 0) s[d0] += v;
        __syncthreads();
    }
    if (q == 0) s[d0] -= tot;  // exclusive
    __syncthreads();
    uint32_t run = (uint32_t)d.cloth[c].t_off + s[d0];
    for (int k = 0; k < q; ++k) run += qs[k][d0];
#pragma unroll 8
    for (int t = a; t < e; ++t) {
        const size_t k = (size_t)t * kSortBuckets + d0;
        const uint32_t n = d.shist[k];
        d.shist[k] = run;
        run += n;
    }
}

// One-sweep offsets (every sort of up to 2^30 keys; beyond, which only the
// object broadphase's grid and hash entries can reach, the per-pass histogram
// above).  k_sort_hist_all reads each
// tile's keys once and adds the digit counts of every pass to its segment's
// totals, so the digits' first positions in the segment are known before
// the first pass; the scatter of a pass then finds a tile's place among its
// segment's earlier tiles by a decoupled look-back over per-tile, per-digit
// status words (flag in the top two bits: aggregate of the tile alone, or
// inclusive prefix from the segment's first tile).  Tiles take their
// position from a ticket counter, so a block only ever waits on blocks that
// started before it.  The offsets are the numbers k_sort_offsets gives.
constexpr uint32_t kStatAgg = 1u << 30, kStatPre = 2u << 30, kStatCount = kStatAgg - 1;
constexpr uint32_t kLookbackSpins = 1u << 22;  // bound on the status waits of one look-back (then ERR_SORT)
constexpr int kLookbackWindow = 8;               // earlier tiles' statuses read per look-back step
__global__ void __launch_bounds__(kThreads) k_sort_hist_all(DevPtrs d, const unsigned long long *__restrict__ keys,
                                                            int shift0, int passes) {
    static_assert(kThreads == kSortBuckets, "one thread per digit");
    constexpr int R = kSortTile / kThreads;
    __shared__ uint32_t h[kSortPassesMax][kSortBuckets];
    const int tile = blockIdx.x, t = threadIdx.x, lane = t & 31;
    const int c = d.stile_cloth[tile];
    const int start = d.stile_start[tile];
    const ClothDev &cd = d.cloth[c];
    const int n = min(kSortTile, cd.t_off + cd.T - start);
    for (int p = 0; p < passes; ++p) {
        h[p][t] = 0;
        d.sstat[((size_t)p * d.nstiles + tile) * kSortBuckets + t] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int li = r * kThreads + t;
        const bool valid = li < n;
        const unsigned long long key = valid ? keys[start + li] : 0ull;
        for (int p = 0; p < passes; ++p) {
            // a digit common to the whole warp (the high digits of nearby
            // Morton codes) is one atomic; otherwise one per lane
            const uint32_t dig = valid ? (uint32_t)(key >> (shift0 + p * kSortBits)) & (kSortBuckets - 1) : kSortBuckets;
            const uint32_t d0 = __shfl_sync(0xffffffffu, dig, 0);
            if (__all_sync(0xffffffffu, dig == d0)) {
                if (lane == 0 && d0 < kSortBuckets) atomicAdd(&h[p][d0], 32u);
            } else if (valid) {
                atomicAdd(&h[p][dig], 1u);
            }
        }
    }
    __syncthreads();
    uint32_t *seg = d.sseg + kSortHead + (size_t)c * kSortPassesMax * kSortBuckets;
    for (int p = 0; p < passes; ++p)
        if (h[p][t]) atomicAdd(&seg[p * kSortBuckets + t], h[p][t]);
}

// Lanes of the warp whose digit equals this one's: eight votes, one per bit of
// the digit.  __match_any_sync gives the same mask in one instruction, but a
// sort pass is bound by its rate: a sort in one launch of 1922, 7938 or 20 k
// keys took 19, 46 and 44 us with it, 17, 42 and 40 us so.
__device__ __forceinline__ uint32_t digit_peers(uint32_t dig) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < kSortBits; ++b) {
        const bool bit = (dig >> b) & 1u;
        const uint32_t v = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? v : ~v;
    }
    return peers;
}

// One tile per block, ranked without block-wide rounds: warp w takes the
// tile's keys [256 w, 256 w + 256) in 8 steps of 32 and ranks each key among
// the warp's earlier keys of its digit (warp-private counts, no block
// barrier); one scan per digit over the warps then gives every key its slot
// in the tile sorted by digit, stable because index order is (warp, step,
// lane).  The sorted tile is staged in shared memory and written out with
// consecutive threads on consecutive slots of each digit's run.
struct SortTile {
    int start, n;           // the tile's first key and number of keys
    uint32_t lo, hi;        // its segment
    int tile, first;        // the tile and its segment's first one, numbered as their status words
    uint32_t *stat;         // kLookback: the pass's status words
    const uint32_t *total;  // kLookback: the segment's digit totals in this pass
};
struct SortShared {
    unsigned long long key[kSortTile];
    uint32_t pay[kSortTile];
    uint32_t wcnt[kThreads / 32][kSortBuckets];  // per warp: keys of each digit (then: first tile slot)
    uint32_t lbase[kSortBuckets];                // first tile slot per digit
    uint32_t gbase[kSortBuckets];                // first global slot per digit
    uint32_t wsum[kThreads / 32], wseg[kThreads / 32];
    int bad;
};
enum SortPlace {
    kOffsets,   // a tile's global slots are in d.shist (k_sort_offsets)
    kLookback,  // they come from the one-sweep look-back (tiles in ticket order)
    kAlone,     // the tile is its segment
};
// False: a wait ran past its bound.  kFresh: the keys were written in this launch.
template <SortPlace kPlace, bool kFresh>
__device__ __forceinline__ bool sort_tile(const DevPtrs &d, SortShared &sh, const SortTile &T,
                                          const unsigned long long *__restrict__ kin, const uint32_t *__restrict__ pin,
                                          unsigned long long *__restrict__ kout, uint32_t *__restrict__ pout, int shift) {
    constexpr int W = kThreads / 32;
    constexpr int R = kSortTile / kThreads;  // keys per lane
    static_assert(kThreads == kSortBuckets && kSortTile == W * 32 * R, "one thread per digit, 32 R keys per warp");
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int n = T.n, start = T.start;
    auto &wcnt = sh.wcnt;
    if (kPlace == kOffsets) sh.gbase[t] = d.shist[(size_t)T.tile * kSortBuckets + t];
    if (kPlace == kLookback && t == 0) sh.bad = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) wcnt[w][t] = 0;
    __syncthreads();
    const uint32_t lt_mask = (1u << lane) - 1u;
    unsigned long long kr[R];
    uint32_t pr[R], rk[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int li = wid * 32 * R + r * 32 + lane;
        const bool valid = li < n;
        kr[r] = valid ? (kFresh ? __ldcg(&kin[start + li]) : kin[start + li]) : 0ull;
        pr[r] = valid ? (kFresh ? __ldcg(&pin[start + li]) : pin[start + li]) : 0u;
        const uint32_t dig = (uint32_t)(kr[r] >> shift) & (kSortBuckets - 1);
        const uint32_t peers = digit_peers(dig) & __ballot_sync(0xffffffffu, valid);
        const uint32_t before = valid ? wcnt[wid][dig] : 0u;
        rk[r] = before + __popc(peers & lt_mask);
        __syncwarp();
        if (valid && (peers & lt_mask) == 0) wcnt[wid][dig] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread t owns digit t: its tile total, then the exclusive scan of the
    // totals over the digits (first slot of the digit) and over the warps
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) tot += wcnt[w][t];
    // one-sweep: publish the tile's count of digit t, and scan the segment's
    // digit totals (the digits' first positions in the segment)
    uint32_t segtot = 0, segincl = 0;
    if (kPlace == kLookback) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(T.stat[(size_t)T.tile * kSortBuckets + t])
            .store((T.tile == T.first ? kStatPre : kStatAgg) | tot, cuda::memory_order_relaxed);
        segtot = segincl = kFresh ? __ldcg(&T.total[t]) : T.total[t];
    }
    uint32_t incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
        if (kPlace == kLookback) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, segincl, o);
            if (lane >= o) segincl += u;
        }
    }
    if (lane == 31) {
        sh.wsum[wid] = incl;
        if (kPlace == kLookback) sh.wseg[wid] = segincl;
    }
    __syncthreads();
    uint32_t run = incl - tot;
    for (int w = 0; w < wid; ++w) run += sh.wsum[w];
    sh.lbase[t] = run;
    if (kPlace == kAlone) sh.gbase[t] = T.lo + run;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const uint32_t v = wcnt[w][t];
        wcnt[w][t] = run;
        run += v;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int li = wid * 32 * R + r * 32 + lane;
        if (li < n) {
            const uint32_t dig = (uint32_t)(kr[r] >> shift) & (kSortBuckets - 1);
            const uint32_t pos = wcnt[wid][dig] + rk[r];
            sh.key[pos] = kr[r];
            sh.pay[pos] = pr[r];
        }
    }
    if (kPlace == kLookback) {
        // the tile's place among the segment's earlier tiles, digit t: sum
        // the aggregates back to the first inclusive prefix
        // A window of kLookbackWindow earlier tiles is read at once (the
        // segment's first tile always holds its inclusive prefix, so the
        // walk never passes it); a window that meets an unpublished tile
        // resumes there.
        uint32_t excl = 0;
        if (T.tile != T.first) {
            uint32_t spins = 0;
            for (int j = T.tile - 1;;) {
                uint32_t sv[kLookbackWindow];
#pragma unroll
                for (int k = 0; k < kLookbackWindow; ++k)
                    sv[k] = j - k >= T.first ? cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(
                                                   T.stat[(size_t)(j - k) * kSortBuckets + t])
                                                   .load(cuda::memory_order_relaxed)
                                             : kStatPre;
                bool done = false;
                int k = 0;
                for (; k < kLookbackWindow; ++k) {
                    if (sv[k] == 0) break;  // not published yet
                    excl += sv[k] & kStatCount;
                    if ((sv[k] & ~kStatCount) == kStatPre || j - k == T.first) {
                        done = true;
                        break;
                    }
                }
                if (done) break;
                j -= k;
                if (k == 0) {
                    if (++spins > kLookbackSpins) {
                        sh.bad = 1;
                        atomicOr(d.err, ERR_SORT);
                        break;
                    }
                    __nanosleep(32);
                }
            }
            // published even after a failed wait, so that later tiles end
            cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(T.stat[(size_t)T.tile * kSortBuckets + t])
                .store(kStatPre | (excl + tot), cuda::memory_order_relaxed);
        }
        uint32_t dbase = segincl - segtot;
        for (int w = 0; w < wid; ++w) dbase += sh.wseg[w];
        sh.gbase[t] = T.lo + dbase + excl;
    }
    __syncthreads();
    if (kPlace == kLookback && sh.bad) return false;
    for (int i = t; i < n; i += kThreads) {
        const unsigned long long key = sh.key[i];
        const uint32_t dig = (uint32_t)(key >> shift) & (kSortBuckets - 1);
        const uint32_t g = sh.gbase[dig] + (uint32_t)i - sh.lbase[dig];
        if (kPlace == kLookback && (g < T.lo || g >= T.hi)) {  // only after a failed wait elsewhere
            atomicOr(d.err, ERR_SORT);
            continue;
        }
        kout[g] = key;
        pout[g] = sh.pay[i];
    }
    return true;
}

template <SortPlace kPlace>
__global__ void __launch_bounds__(kThreads, 4) k_sort_scatter(DevPtrs d, const unsigned long long *__restrict__ kin,
                                                           const uint32_t *__restrict__ pin,
                                                           unsigned long long *__restrict__ kout,
                                                           uint32_t *__restrict__ pout, int shift, int pass,
                                                           const int *__restrict__ tile_first) {
    __shared__ SortShared sh;
    __shared__ int s_tile;
    if (kPlace == kLookback) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(&d.sseg[pass], 1u);
        __syncthreads();
    }
    SortTile T;
    T.tile = kPlace == kLookback ? s_tile : (int)blockIdx.x;
    const int c = d.stile_cloth[T.tile];
    const ClothDev &cd = d.cloth[c];
    T.start = d.stile_start[T.tile];
    T.n = min(kSortTile, cd.t_off + cd.T - T.start);
    T.lo = (uint32_t)cd.t_off;
    T.hi = (uint32_t)(cd.t_off + cd.T);
    if (kPlace == kLookback) {
        T.first = tile_first[c];
        T.stat = d.sstat + (size_t)pass * d.nstiles * kSortBuckets;
        T.total = d.sseg + kSortHead + ((size_t)c * kSortPassesMax + pass) * kSortBuckets;
    }
    sort_tile<kPlace, false>(d, sh, T, kin, pin, kout, pout, shift);
}

// ---------------------------------------------------------------------------
// The low half of 63-bit keys.  The passes above sort such keys by their top
// half only (bits 32..62, about a millimetre of a metre per axis): half the
// passes.  Keys that share it stay in their order before the sort, in runs
// that are almost always of one or two keys; the post-sort ranks the keys of
// a run of at most kTieRun by (low half, position), which completes the stable
// sort, and longer runs (codes clamped at the frame's faces, scenes of about a
// millimetre) are sorted in place after it.
// A sort of a million keys: 8 passes and the histogram 178 us, 4 passes and the
// ranks 100 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t top_half(unsigned long long k) { return (uint32_t)(k >> 32); }

// A sorted slot's outputs: key, triangle order and record, (fixed mode) the
// leaf box, and no parents yet.
__device__ __forceinline__ void put_slot(const DevPtrs &d, const ClothDev &cd, int s, unsigned long long key,
                                         uint32_t orig) {
    d.keys[s] = key;
    d.perm[s] = orig;
    if (d.tri_slot) d.tri_slot[s] = d.tri[orig];  // one gather per slot instead of two per pair
    const int local = s - cd.t_off, leaf = cd.n_off + (cd.T - 1) + local;
    if (!cd.leaf_quirk) {
        d.nmin[leaf] = d.leaf_tmp_min[orig];
        d.nmax[leaf] = d.leaf_tmp_max[orig];
    }
    d.parent[leaf] = -1;
    if (local < cd.T - 1) d.parent[cd.n_off + local] = -1;
}

// The final place of slot s's key in its run of equal top halves (keys in
// [first, end), sorted by top half), and whether three equal keys meet in it;
// -1 in a run of more than kTieRun.
template <class Keys>
__device__ __forceinline__ int tie_place(const Keys &keys, int s, int first, int end, unsigned long long key,
                                         bool &three) {
    const uint32_t top = top_half(key);
    if ((s + kTieRun < end && top_half(keys[s + kTieRun]) == top) ||
        (s - kTieRun >= first && top_half(keys[s - kTieRun]) == top))
        return -1;
    int a = s, e = s + 1;
    while (a > first && s - a < kTieRun && top_half(keys[a - 1]) == top) --a;
    while (e < end && e - s <= kTieRun && top_half(keys[e]) == top) ++e;
    if (e - a > kTieRun) return -1;
    int r = a, same = 0;
    for (int j = a; j < e; ++j) {
        const unsigned long long q = keys[j];
        r += q < key || (q == key && j < s);
        same += q == key;
    }
    three = same >= 3;
    return r;
}

// After the sort: the low halves (halves != 0), the new triangle order and the
// cloths in which three equal codes meet (their hierarchy may be malformed).
// Runs longer than kTieRun are left, by the thread of their first slot, to
// k_sort_long_runs.
__global__ void __launch_bounds__(kThreads) k_post_sort(DevPtrs d, int halves) {
    __shared__ int q_first[kThreads / kTieRun + 1], q_end[kThreads / kTieRun + 1], s_n, s_at, s_tile;
    const int s = blockIdx.x * kThreads + threadIdx.x;
    bool starts = false;  // a longer run
    int end = 0;
    uint32_t top = 0;
    if (s < d.Ttot) {
        const int c = d.tcloth[s];
        const ClothDev &cd = d.cloth[c];
        const int first = cd.t_off;
        end = cd.t_off + cd.T;
        const unsigned long long key = d.keys_alt[s];
        const unsigned long long prev = s > first ? d.keys_alt[s - 1] : ~key, next = s + 1 < end ? d.keys_alt[s + 1] : ~key;
        int place = s;
        bool three = prev == key && next == key;
        top = top_half(key);
        if (halves && (top_half(prev) == top || top_half(next) == top))
            place = tie_place(d.keys_alt, s, first, end, key, three);
        if (place >= 0) {
            if (three && d.eq3) d.eq3[c] = 1;
            put_slot(d, cd, place, key, d.payload_alt[s]);
        } else {
            starts = top_half(prev) != top;
        }
    }
    if (threadIdx.x == 0) s_n = 0;
    if (!halves || !__syncthreads_or(starts)) return;
    if (starts) {
        int lo = s + kTieRun, hi = end;  // keys [s, lo] have this top half, hi has not (or is the end)
        while (hi - lo > 1) {
            const int m = lo + (hi - lo) / 2;
            if (top_half(d.keys_alt[m]) == top) lo = m;
            else hi = m;
        }
        const int k = atomicAdd(&s_n, 1);
        q_first[k] = s;
        q_end[k] = hi;
    }
    __syncthreads();
    for (int k = 0; k < s_n; ++k) {
        const int n = q_end[k] - q_first[k], nt = (n + kSortTile - 1) / kSortTile;
        if (threadIdx.x == 0) {
            s_at = (int)atomicAdd(&d.sseg[nt > 1 ? kRunsTiled : kRunsSmall], 1u);
            if (nt > 1) s_tile = (int)atomicAdd(&d.sseg[kRunsTiles], (uint32_t)nt);
        }
        __syncthreads();
        if (nt == 1) {
            if (threadIdx.x == 0) d.run_small[s_at] = make_int2(q_first[k], q_end[k]);
        } else {
            if (threadIdx.x == 0) d.run_tiled[s_at] = make_int4(q_first[k], q_end[k], s_tile, 0);
            for (int i = threadIdx.x; i < nt; i += kThreads) d.run_of_tile[s_tile + i] = s_at;
            for (int i = threadIdx.x; i < 4 * kSortBuckets; i += kThreads)
                d.run_total[(size_t)s_at * 4 * kSortBuckets + i] = 0;
        }
        __syncthreads();
    }
}

// The outputs of the sorted run r's slots [a, e), by one block.
__device__ __forceinline__ void put_run(const DevPtrs &d, int first, int end, int a, int e) {
    const int c = d.tcloth[first];
    const ClothDev &cd = d.cloth[c];
    for (int s = a + threadIdx.x; s < e; s += kThreads) {
        const unsigned long long key = __ldcg(&d.keys_alt[s]);
        if (s > first && s + 1 < end && __ldcg(&d.keys_alt[s - 1]) == key && __ldcg(&d.keys_alt[s + 1]) == key && d.eq3)
            d.eq3[c] = 1;
        put_slot(d, cd, s, key, __ldcg(&d.payload_alt[s]));
    }
}

// The long runs sorted by their low halves, in place.  Work items are taken by
// ticket: every tile's digit counts of the runs of several tiles (and whether
// the run is in order already, as equal codes are); their four passes, tile by
// tile, with the one-sweep's look-back within the run; their outputs; then the
// runs of one tile.  An item of a pass waits until every item before it is done.
// It waits on smaller tickets only, which blocks that run hold, and the
// smallest one in work waits for nothing: the wait ends without the blocks
// having to be resident together, and it is bounded all the same.
// Runs of up to kRankRun keys are ranked by counting in shared memory.
// So the sort's time is bounded by its passes, whatever the codes.  Bound by the
// passes, as they are by ranking; with few runs, by the chain of items.  A
// million boxes' build (ms) with one block per run / so: spread over the cube
// 0.271 / 0.271, in one cell of the top half 17.3 / 0.36, two codes in turn
// 10.1 / 0.40, half of each axis clamped 1.83 / 0.42, runs of 300 0.40 / 0.35,
// a 1 m cloth around the origin 0.44 / 0.40.
constexpr int kRankRun = 512;
constexpr int kRunBlocks = 608;  // four on each of 152 SMs
__global__ void __launch_bounds__(kThreads, 4) k_sort_long_runs(DevPtrs d) {
    __shared__ SortShared sh;
    __shared__ uint32_t s_item;
    __shared__ int s_ok;
    const uint32_t nsmall = d.sseg[kRunsSmall], ntiles = d.sseg[kRunsTiles], total = nsmall + 6 * ntiles;
    const int t = threadIdx.x, lane = t & 31;
    bool gave_up = false;  // block-uniform: it waits no more, and its passes are left out
    if (total == 0) return;
    for (;;) {
        if (t == 0) s_item = atomicAdd(&d.sseg[kRunsTicket], 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total) return;
        if (item >= 6 * ntiles) {
            const int2 r = d.run_small[item - 6 * ntiles];
            const int n = r.y - r.x;
            if (n <= kRankRun) {
                constexpr int R = kRankRun / kThreads;
                uint32_t *low = sh.pay;
                const uint4 *low4 = reinterpret_cast<const uint4 *>(sh.pay);
                unsigned long long key[R];
                uint32_t pay[R];
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const int i = k * kThreads + t;
                    key[k] = i < n ? d.keys_alt[r.x + i] : ~0ull;
                    pay[k] = i < n ? d.payload_alt[r.x + i] : 0u;
                    low[i] = (uint32_t)key[k];  // (past the run: above every key, or not below it)
                }
                __syncthreads();
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const int w0 = k * kThreads + (t & ~31);  // the warp's first position
                    if (w0 >= n) break;
                    const uint32_t mine = (uint32_t)key[k];
                    int place = 0, j = 0;
                    for (; j < w0; j += 4) {  // earlier positions: equal keys come first
                        const uint4 q = low4[j / 4];
                        place += (q.x <= mine) + (q.y <= mine) + (q.z <= mine) + (q.w <= mine);
                    }
                    for (int o = 0; o < 32; ++o, ++j) place += low[j] < mine || (low[j] == mine && o < lane);
                    for (; j < n; j += 4) {
                        const uint4 q = low4[j / 4];
                        place += (q.x < mine) + (q.y < mine) + (q.z < mine) + (q.w < mine);
                    }
                    if (w0 + lane < n) {
                        d.keys_alt[r.x + place] = key[k];
                        d.payload_alt[r.x + place] = pay[k];
                    }
                }
            } else {
                bool wrong = false;
                for (int i = r.x + t; i + 1 < r.y; i += kThreads) wrong = wrong || d.keys_alt[i] > d.keys_alt[i + 1];
                if (__syncthreads_or(wrong)) {
                    const SortTile T{r.x, n, (uint32_t)r.x, (uint32_t)r.y, 0, 0, nullptr, nullptr};
                    unsigned long long *k0 = d.keys_alt, *k1 = d.keys;
                    uint32_t *p0 = d.payload_alt, *p1 = d.payload;
#pragma unroll 1
                    for (int p = 0; p < 4; ++p) {
                        sort_tile<kAlone, true>(d, sh, T, k0, p0, k1, p1, p * kSortBits);
                        __syncthreads();
                        unsigned long long *tk = k0; k0 = k1; k1 = tk;
                        uint32_t *tp = p0; p0 = p1; p1 = tp;
                    }
                }
            }
            __syncthreads();
            put_run(d, r.x, r.y, r.x, r.y);
        } else {
            const uint32_t phase = item / ntiles;
            const int tile = (int)(item % ntiles), run = d.run_of_tile[tile];
            const int4 r = __ldcg(&d.run_tiled[run]);
            const int start = r.x + (tile - r.z) * kSortTile, n = min(kSortTile, r.y - start);
            if (phase == 0) {
                for (int p = 0; p < 4; ++p) {
                    sh.wcnt[p][t] = 0;
                    d.sstat[((size_t)p * ntiles + tile) * kSortBuckets + t] = 0;
                }
                __syncthreads();
                bool wrong = false;
                for (int i0 = 0; i0 < n; i0 += kThreads) {
                    const int i = i0 + t;
                    const bool valid = i < n;
                    const unsigned long long key = valid ? d.keys_alt[start + i] : 0ull;
                    wrong = wrong || (valid && start + i + 1 < r.y && key > d.keys_alt[start + i + 1]);
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const uint32_t dig = valid ? (uint32_t)(key >> (p * kSortBits)) & (kSortBuckets - 1) : kSortBuckets;
                        const uint32_t d0 = __shfl_sync(0xffffffffu, dig, 0);
                        if (__all_sync(0xffffffffu, dig == d0)) {
                            if (lane == 0 && d0 < kSortBuckets) atomicAdd(&sh.wcnt[p][d0], 32u);
                        } else if (valid) {
                            atomicAdd(&sh.wcnt[p][dig], 1u);
                        }
                    }
                }
                if (__syncthreads_or(wrong) && t == 0) d.run_tiled[run].w = 1;
                for (int p = 0; p < 4; ++p)
                    if (sh.wcnt[p][t]) atomicAdd(&d.run_total[((size_t)run * 4 + p) * kSortBuckets + t], sh.wcnt[p][t]);
            } else {
                if (t == 0 && !gave_up) {
                    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> done(d.sseg[kRunsDone]);
                    uint32_t spins = 0;
                    s_ok = 1;
                    while (done.load(cuda::memory_order_acquire) < phase * ntiles) {
                        if (++spins > kLookbackSpins) {
                            atomicOr(d.err, ERR_SORT);
                            s_ok = 0;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
                __syncthreads();
                gave_up = gave_up || !s_ok;
                if (phase == 5) {
                    put_run(d, r.x, r.y, start, start + n);  // (also after a failed wait: every slot gets a triangle)
                } else if (!gave_up && __ldcg(&d.run_tiled[run].w)) {
                    const int p = (int)phase - 1;
                    const SortTile T{start, n, (uint32_t)r.x, (uint32_t)r.y, tile, r.z,
                                     d.sstat + (size_t)p * ntiles * kSortBuckets,
                                     d.run_total + ((size_t)run * 4 + p) * kSortBuckets};
                    const bool odd = p & 1;
                    if (!sort_tile<kLookback, true>(d, sh, T, odd ? d.keys : d.keys_alt, odd ? d.payload : d.payload_alt,
                                                    odd ? d.keys_alt : d.keys, odd ? d.payload_alt : d.payload,
                                                    p * kSortBits))
                        gave_up = true;
                }
            }
        }
        __syncthreads();
        if (t == 0 && item < 5 * ntiles && !gave_up) {
            __threadfence();
            atomicAdd(&d.sseg[kRunsDone], 1u);
        }
    }
}

// Segments of at most CS R 1024 keys: sort and post-sort in one launch, one
// cluster of CS CTAs per segment, every key in a register or in shared memory
// throughout.  A key moves as one word, the 32 bits sorted by over its position
// before the sort; a pass ranks the CTA's keys per warp, exchanges the CTAs'
// digit counts and stores each key straight into the shared memory of the CTA
// that holds its place.  The full keys and payloads are fetched by position at
// the end.  Bound by barriers and by one SM's rate of ranking (5 us per 1024
// keys and four passes in one CTA), hence CTAs rather than keys per thread
// where few segments leave SMs idle.
constexpr int kSmallThreads = 1024;
constexpr int kSmallCtas = 8;
template <int CS, int R>
struct SegmentSort {
    static constexpr int W = kSmallThreads / 32, N = R * kSmallThreads;  // warps and keys per CTA
    static constexpr size_t kSmem = (size_t)N * 8 + (size_t)W * kSortBuckets * 4;
};
__device__ __forceinline__ uint32_t shared_of(const void *p, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
template <int CS, int R>
__global__ void __launch_bounds__(kSmallThreads) k_sort_segment(DevPtrs d, int halves) {
    using S = SegmentSort<CS, R>;
    constexpr int W = S::W, N = S::N;
    extern __shared__ unsigned long long s_key[];                                               // N
    uint32_t(*wcnt)[kSortBuckets] = reinterpret_cast<uint32_t(*)[kSortBuckets]>(s_key + N);    // per warp and digit
    __shared__ uint32_t qsum[4][kSortBuckets], ctot[kSortBuckets], s_base[kSortBuckets], wsum[kSortBuckets / 32];
    __shared__ int s_long;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = CS > 1 ? (int)cluster.block_rank() : 0;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int dig0 = t & (kSortBuckets - 1), q0 = t / kSortBuckets;  // digit and quarter of the warps
    const int c = blockIdx.x / CS;
    const ClothDev &cd = d.cloth[c];
    const int n = cd.T, off = cd.t_off, first = rank * N;            // this CTA's first place
    auto barrier = [&]() {
        if (CS > 1) cluster.sync();
        else __syncthreads();
    };
    auto place_of = [&](int r) { return wid * 32 * R + r * 32 + lane; };  // index order is (warp, step, lane)
    unsigned long long w[R];
    uint32_t rk[R];
    // bits sorted by (the top or the low half) over the position
    auto word = [&](int pos, bool top) {
        const unsigned long long k = d.keys_alt[off + pos];
        return (top ? k & 0xffffffff00000000ull : k << 32) | (unsigned)pos;
    };
    auto pass = [&](int shift) {
        for (int k = t; k < W * kSortBuckets; k += kSmallThreads) (&wcnt[0][0])[k] = 0;
        __syncthreads();
        const uint32_t below = (1u << lane) - 1u;
#pragma unroll
        for (int r = 0; r < R; ++r) {  // ranks among the warp's earlier keys of the digit
            const uint32_t dig = (uint32_t)(w[r] >> shift) & (kSortBuckets - 1);
            const uint32_t peers = digit_peers(dig);
            const uint32_t before = wcnt[wid][dig];
            rk[r] = before + __popc(peers & below);
            __syncwarp();
            if ((peers & below) == 0) wcnt[wid][dig] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t part = 0;
#pragma unroll
        for (int k = 0; k < W / 4; ++k) part += wcnt[q0 * (W / 4) + k][dig0];
        qsum[q0][dig0] = part;
        __syncthreads();
        uint32_t mine = 0, all = 0, before = 0;
        if (q0 == 0) ctot[dig0] = mine = qsum[0][dig0] + qsum[1][dig0] + qsum[2][dig0] + qsum[3][dig0];
        barrier();  // counts published, and every CTA's keys are in registers
        if (q0 == 0) {
            all = mine;
            if (CS > 1) {
                all = 0;
#pragma unroll
                for (int k = 0; k < CS; ++k) {
                    uint32_t v;
                    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(shared_of(&ctot[dig0], k)) : "memory");
                    before += k < rank ? v : 0u;
                    all += v;
                }
            }
            uint32_t incl = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) wsum[dig0 / 32] = incl;
            s_base[dig0] = incl - all + before;
        }
        __syncthreads();
        uint32_t run = s_base[dig0];
#pragma unroll
        for (int k = 0; k < kSortBuckets / 32; ++k) run += k < dig0 / 32 ? wsum[k] : 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) run += k < q0 ? qsum[k][dig0] : 0u;
#pragma unroll
        for (int k = 0; k < W / 4; ++k) {
            uint32_t &slot = wcnt[q0 * (W / 4) + k][dig0];
            const uint32_t v = slot;
            slot = run;
            run += v;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t pos = wcnt[wid][(uint32_t)(w[r] >> shift) & (kSortBuckets - 1)] + rk[r];
            if (CS > 1)
                asm volatile("st.shared::cluster.u64 [%0], %1;"
                             : : "r"(shared_of(s_key, (int)(pos / N)) + 8u * (pos % N)), "l"(w[r]) : "memory");
            else
                s_key[pos] = w[r];
        }
        barrier();
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = s_key[place_of(r)];
    };
    // places past the segment hold words above every key of it: they stay last
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = first + place_of(r) < n ? word(first + place_of(r), halves != 0) : ~0ull;
    for (int p = 0; p < 4; ++p) pass(32 + p * kSortBits);
    bool any = false;  // the keys are in the order of the whole code
    if (halves) {  // a long run of equal top halves: by low half first, then by top half again
        if (t == 0) s_long = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = place_of(r);  // a run longer than kTieRun has over half of that in one CTA
            if (i + kTieRun / 2 < N && first + i + kTieRun / 2 < n && top_half(s_key[i]) == top_half(s_key[i + kTieRun / 2])) s_long = 1;
        }
        barrier();
        any = s_long != 0;
        if (CS > 1) {
#pragma unroll
            for (int k = 0; k < CS; ++k) {
                int v;
                asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(shared_of(&s_long, k)) : "memory");
                any = any || v != 0;
            }
        }
        if (any)
            for (int half = 0; half < 2; ++half) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int i = first + place_of(r);
                    const int pos = half ? (int)(uint32_t)w[r] : i;
                    w[r] = i < n ? word(pos, half != 0) : ~0ull;
                }
                for (int p = 0; p < 4; ++p) pass(32 + p * kSortBits);
            }
    }
    barrier();
    // full keys by place, for the runs of equal top halves
    unsigned long long key[R];
    uint32_t pay[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool have = first + place_of(r) < n;
        const int pos = (int)(uint32_t)w[r];
        key[r] = have ? d.keys_alt[off + pos] : ~0ull;
        pay[r] = have ? d.payload_alt[off + pos] : 0u;
        s_key[place_of(r)] = key[r];
    }
    barrier();
    struct Keys {  // by place in the segment
        const unsigned long long *own;
        int rank;
        __device__ __forceinline__ unsigned long long operator[](int i) const {
            if (CS == 1 || i / N == rank) return own[i % N];
            unsigned long long v;
            asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(shared_of(own, i / N) + 8u * (i % N)) : "memory");
            return v;
        }
    };
    const Keys keys{s_key, rank};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = first + place_of(r);
        if (i >= n) continue;
        const unsigned long long prev = i > 0 ? keys[i - 1] : ~key[r], next = i + 1 < n ? keys[i + 1] : ~key[r];
        int place = i;
        bool three = prev == key[r] && next == key[r];
        if (halves && !any && (top_half(prev) == top_half(key[r]) || top_half(next) == top_half(key[r])))
            place = tie_place(keys, i, 0, n, key[r], three);
        if (three && d.eq3) d.eq3[c] = 1;
        put_slot(d, cd, off + place, key[r], pay[r]);
    }
    barrier();  // no CTA leaves while another reads its keys
}

// ---------------------------------------------------------------------------
// Karras hierarchy: Collision/CudaBVH.cu:163-242, Core/CudaUtils.cu:338-362.
// ---------------------------------------------------------------------------
// A cloth's sorted keys by local index, as far as the block's own slots and one
// on each side go; an access beyond them only sets `out`.
struct BlockKeys {
    const unsigned long long *own;  // shared: slots [b0 - 1, b0 + n]
    int b0, n;                      // local index of the block's first slot (negative: it begins in an earlier cloth), slots
    mutable bool out;
    __device__ __forceinline__ unsigned long long operator[](int i) const {
        const unsigned k = (unsigned)(i - b0 + 1);
        if (k < (unsigned)n + 2u) return own[k];
        out = true;
        return 0ull;
    }
};
template <class Keys>
__device__ __forceinline__ int delta(const Keys &m, int i, int j, int maxi) {
    if (j < 0 || j > maxi) return -1;
    const unsigned long long x = m[i] ^ m[j];
    return x ? __clzll((long long)x) : __clzll((long long)((unsigned long long)i ^ (unsigned long long)j)) + 64;
}
__device__ __forceinline__ int sgn_ref(int a) { return signbit((float)a) ? -1 : 1; }

// ---------------------------------------------------------------------------
// Node boxes without a climb.  A node's box is the union of the leaf boxes in
// its range, and min / max are exact, so any grouping gives the bits of the
// bottom-up refit: a binary tree over aligned runs of leaves (level k's entry j
// holds the union of the leaves [j 2^k, (j + 1) 2^k)) answers every range with
// at most two entries per level, and half of the nodes need two or three leaf
// boxes.  k_range_tree builds it with one block per 2048 leaves (levels 1..11)
// and the last block of a cloth the levels above; k_karras then writes every
// node complete, the traversal's record included.  The climb was bound by its
// chain of arrivals to the root, 31 us for 1922 triangles as for a million.
// From codes to records (us; cloths of 1922, 20 k and 522 k triangles, 30 cloths
// of 620 k, 64 of 1.92 M, a million random boxes): 60, 74, 124, 143, 272, 179
// with the climb, 28, 54, 93, 102, 219, 173 so.
// Cloths in which three equal codes meet keep the climb (below): there the
// reference's hierarchy may not be a tree, and which nodes it reaches counts.
// ---------------------------------------------------------------------------
constexpr int kTreeTop = 512;  // nodes of a level that one block combines in shared memory
__device__ __forceinline__ int half_up(int n) { return (n + 1) >> 1; }
constexpr int kTreeThreads = 512;
__global__ void __launch_bounds__(kTreeThreads) k_range_tree(DevPtrs d) {
    static_assert(kSortTile == 4 * kTreeThreads, "levels 1..5 per warp, 6..11 over 64 warp results");
    __shared__ float4 s_min[kTreeTop], s_max[kTreeTop];
    __shared__ int s_last;
    const int c = d.stile_cloth[blockIdx.x];
    const ClothDev &cd = d.cloth[c];
    if (d.eq3[c]) return;
    const int T = cd.T, first = d.stile_start[blockIdx.x] - cd.t_off;  // local first leaf of the tile
    const int t = threadIdx.x, lane = t & 31;
    const float4 *lmin = d.nmin + cd.n_off + (T - 1), *lmax = d.nmax + cd.n_off + (T - 1);
    float4 *rmin = d.rmin + cd.t_off + kRangePad * c, *rmax = d.rmax + cd.t_off + kRangePad * c;
    for (int q = 0; q < 4; ++q) {
        const int li = first + q * kTreeThreads + t;
        if (first + q * kTreeThreads >= T) break;
        float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
        if (li < T) { mn = xyz(lmin[li]); mx = xyz(lmax[li]); }
        int off = 0, n = T;
#pragma unroll
        for (int k = 1; k <= 5; ++k) {
            const int o = 1 << (k - 1);
            const float3 a = f3(__shfl_down_sync(0xffffffffu, mn.x, o), __shfl_down_sync(0xffffffffu, mn.y, o),
                                __shfl_down_sync(0xffffffffu, mn.z, o));
            const float3 b = f3(__shfl_down_sync(0xffffffffu, mx.x, o), __shfl_down_sync(0xffffffffu, mx.y, o),
                                __shfl_down_sync(0xffffffffu, mx.z, o));
            if ((lane & (2 * o - 1)) == 0 && li < T) {
                if (li + o < T) { mn = vmin(mn, a); mx = vmax(mx, b); }
                rmin[off + (li >> k)] = f4(mn, 0.f);
                rmax[off + (li >> k)] = f4(mx, 0.f);
            }
            n = half_up(n);
            off += n;
        }
        if (lane == 0 && li < T) { s_min[q * 16 + (t >> 5)] = f4(mn, 0.f); s_max[q * 16 + (t >> 5)] = f4(mx, 0.f); }
    }
    int off = 0, n = T;  // after level k: off = where level k + 1 starts, n = level k's entries
    for (int k = 1; k <= 5; ++k) { n = half_up(n); off += n; }
    __syncthreads();
    if (t < 32) {
        for (int k = 6; k <= 11; ++k) {
            const int j = t, per = 1 << k;
            const bool mine = j < (kSortTile >> k) && first + j * per < T;
            float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
            if (mine) {
                mn = xyz(s_min[2 * j]); mx = xyz(s_max[2 * j]);
                if (first + j * per + per / 2 < T) { mn = vmin(mn, xyz(s_min[2 * j + 1])); mx = vmax(mx, xyz(s_max[2 * j + 1])); }
                rmin[off + (first >> k) + j] = f4(mn, 0.f);
                rmax[off + (first >> k) + j] = f4(mx, 0.f);
            }
            __syncwarp();
            if (mine) { s_min[j] = f4(mn, 0.f); s_max[j] = f4(mx, 0.f); }
            __syncwarp();
            n = half_up(n);
            off += n;
        }
    }
    if (T <= kSortTile) return;
    // the last of the cloth's blocks to finish builds the levels above
    if (t == 0) {
        __threadfence();
        s_last = atomicAdd(&d.tree_done[c], 1) == (T + kSortTile - 1) / kSortTile - 1;
        if (s_last) d.tree_done[c] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    off = 0;
    n = T;
    int prev = 0;
    for (int k = 1; k <= 11; ++k) { prev = off; n = half_up(n); off += n; }  // prev: where level 11 starts
    while (n > kTreeTop) {  // more than a million leaves: level by level through memory
        const int m = half_up(n);
        for (int j = t; j < m; j += kTreeThreads) {
            float3 mn = xyz(__ldcg(&rmin[prev + 2 * j])), mx = xyz(__ldcg(&rmax[prev + 2 * j]));
            if (2 * j + 1 < n) {
                mn = vmin(mn, xyz(__ldcg(&rmin[prev + 2 * j + 1])));
                mx = vmax(mx, xyz(__ldcg(&rmax[prev + 2 * j + 1])));
            }
            rmin[off + j] = f4(mn, 0.f);
            rmax[off + j] = f4(mx, 0.f);
        }
        __threadfence();
        __syncthreads();
        prev = off;
        off += m;
        n = m;
    }
    for (int j = t; j < n; j += kTreeThreads) { s_min[j] = __ldcg(&rmin[prev + j]); s_max[j] = __ldcg(&rmax[prev + j]); }
    __syncthreads();
    while (n > 1) {
        const int m = half_up(n);
        float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
        const int j = t;  // m <= kTreeTop / 2 = one entry per thread
        if (j < m) {
            mn = xyz(s_min[2 * j]); mx = xyz(s_max[2 * j]);
            if (2 * j + 1 < n) { mn = vmin(mn, xyz(s_min[2 * j + 1])); mx = vmax(mx, xyz(s_max[2 * j + 1])); }
            rmin[off + j] = f4(mn, 0.f);
            rmax[off + j] = f4(mx, 0.f);
        }
        __syncthreads();
        if (j < m) { s_min[j] = f4(mn, 0.f); s_max[j] = f4(mx, 0.f); }
        __syncthreads();
        off += m;
        n = m;
    }
}

// Union of the leaf boxes [a, b]: each level takes the range's first and last
// entry, whether or not the level above covers them (taking a box twice
// changes nothing), so there is no branch on them.  n leaves at lmin / lmax,
// the levels above at rmin / rmax.
__device__ __forceinline__ void range_box(const float4 *lmin, const float4 *lmax, const float4 *rmin, const float4 *rmax,
                                          int n, int a, int b, float3 &mn, float3 &mx) {
    mn = vmin(xyz(lmin[a]), xyz(lmin[b]));
    mx = vmax(xyz(lmax[a]), xyz(lmax[b]));
    int l = a, r = b;  // this level's entries l .. r
    while (r - l > 1) {
        l = (l + 1) >> 1;
        r = (r - 1) >> 1;
        if (l > r) break;
        mn = vmin(mn, vmin(xyz(rmin[l]), xyz(rmin[r])));
        mx = vmax(mx, vmax(xyz(rmax[l]), xyz(rmax[r])));
        n = half_up(n);
        rmin += n;
        rmax += n;
    }
}

__device__ __forceinline__ void put_wnode(const DevPtrs &d, size_t node, float3 lmn, float3 lmx, float3 rmn, float3 rmx,
                                          int2 ch, int2 rm) {
    float4 *w = d.wnode + 4 * node;
    w[0] = f4(lmn, __int_as_float(ch.x));
    w[1] = f4(lmx, __int_as_float(rm.x));
    w[2] = f4(rmn, __int_as_float(ch.y));
    w[3] = f4(rmx, __int_as_float(rm.y));
}

// Range and split of internal node id (FindRange, FindSplit): the range's far
// end j and the last leaf of the left child.
template <class Keys>
__device__ __forceinline__ void karras_range(const Keys &m, int id, int In, int &j, int &split) {
    const int dd = sgn_ref(delta(m, id, id + 1, In) - delta(m, id, id - 1, In));
    const int delmin = delta(m, id, id - dd, In);
    int lmax = 2;
    while (delta(m, id, id + lmax * dd, In) > delmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(m, id, id + (l + t) * dd, In) > delmin) l += t;
    j = id + l * dd;
    const int first = min(id, j), last = max(id, j);
    // FindSplit (code-only prefix)
    const unsigned long long fc = m[first], lc = m[last];
    if (fc == lc) {
        split = (first + last) >> 1;
    } else {
        const int com = __clzll((long long)(fc ^ lc));
        split = first;
        int step = last - first;
        do {
            step = (step + 1) >> 1;
            const int ns = split + step;
            if (ns < last) {
                if (__clzll((long long)(fc ^ m[ns])) > com) split = ns;
            }
        } while (step > 1);
    }
}

// Writes node `id` of a cloth; where the hierarchy is a tree (boxes), with
// everything the refit and the record pass would write, from its children's
// boxes.
__device__ __forceinline__ void put_node(const DevPtrs &d, const ClothDev &cd, int id, int j, int split, bool boxes,
                                         float3 amn, float3 amx, float3 bmn, float3 bmx) {
    const int In = cd.T - 1, first = min(id, j), last = max(id, j);
    const int left = split == first ? In + split : split;
    const int right = split + 1 == last ? In + split + 1 : split + 1;
    d.child[cd.i_off + id] = make_int2(left, right);
    if (boxes) {
        const int2 rm = make_int2(In + split, In + last);
        d.nmin[cd.n_off + id] = f4(vmin(amn, bmn), 0.f);
        d.nmax[cd.n_off + id] = f4(vmax(amx, bmx), 0.f);
        d.rml[cd.i_off + id] = rm;
        d.parent[cd.n_off + left] = id;
        d.parent[cd.n_off + right] = id;
        put_wnode(d, (size_t)(cd.i_off + id), amn, amx, bmn, bmx, make_int2(left, right), rm);
        return;
    }
    if (d.nend) d.nend[cd.i_off + id] = j;
    // An internal node that the refit never reaches (possible only when a run
    // of >= 3 equal codes makes two nodes claim one child) keeps stale data in
    // the reference; here it keeps zeros, deterministically.
    d.nmin[cd.n_off + id] = make_float4(0.f, 0.f, 0.f, 0.f);
    d.nmax[cd.n_off + id] = make_float4(0.f, 0.f, 0.f, 0.f);
    d.rml[cd.i_off + id] = make_int2(0, 0);
    // The reference's parents[] write race resolved as "largest parent wins".
    atomicMax(&d.parent[cd.n_off + left], id);
    atomicMax(&d.parent[cd.n_off + right], id);
    d.visit[cd.i_off + id] = 0;
}

// One thread per internal node.  A block takes SPAN slots; nodes whose search
// stays in them take their keys, and the boxes of their children (from a small
// range tree over the block's leaves), from shared memory.  The few others,
// whose searches go through memory for a dozen dependent loads or more, are
// queued for k_karras_far: a lane in such a search holds up its warp, and
// nearly every warp would have one.  SPAN = kSortTile: blocks are the sort's
// tiles, for cloths of one tile, which have no such nodes (and need no range
// tree in memory); SPAN = 256: any.
template <int BS, int SPAN>
struct KarrasBlock {
    static constexpr bool kWhole = SPAN == kSortTile;  // a block holds a whole cloth
    static constexpr size_t kSmem = (size_t)4 * SPAN * sizeof(float4) + (size_t)(SPAN + 2) * 8 + (size_t)SPAN * 4;
};
template <int BS, int SPAN>
__global__ void __launch_bounds__(BS) k_karras(DevPtrs d) {
    constexpr bool kWhole = KarrasBlock<BS, SPAN>::kWhole;
    extern __shared__ float4 s_min[];                                     // leaves, then the levels above
    float4 *s_max = s_min + 2 * SPAN;
    unsigned long long *s_key = reinterpret_cast<unsigned long long *>(s_max + 2 * SPAN);
    int *s_far = reinterpret_cast<int *>(s_key + SPAN + 2);
    __shared__ int s_nfar;
    __shared__ uint32_t s_base;
    const int t = threadIdx.x;
    const int B0 = kWhole ? d.stile_start[blockIdx.x] : blockIdx.x * SPAN;
    const int B1 = kWhole ? B0 + d.cloth[d.stile_cloth[blockIdx.x]].T : min(B0 + SPAN, d.Ttot);
    if (blockIdx.x == 0 && t == 0 && d.nrexit) *d.nrexit = 0;  // k_refit_local appends to it
    if (t == 0) {
        s_nfar = 0;
        s_key[0] = B0 > 0 ? d.keys[B0 - 1] : 0ull;
        s_key[B1 - B0 + 1] = B1 < d.Ttot ? d.keys[B1] : 0ull;
    }
    // (block-uniform: flagged cloths take their boxes from the climb, so the
    // leaves are of no use only where every cloth of the block is flagged)
    bool tree = false;
    if (d.eq3)
        for (int c = d.tcloth[B0], c1 = d.tcloth[B1 - 1]; c <= c1 && !tree; ++c) tree = !d.eq3[c];
#pragma unroll
    for (int q = 0; q < SPAN / BS; ++q) {
        const int k = q * BS + t;
        if (k >= B1 - B0) break;
        s_key[k + 1] = d.keys[B0 + k];
        if (tree) {
            const ClothDev &cd = d.cloth[d.tcloth[B0 + k]];
            const int leaf = cd.n_off + (cd.T - 1) + B0 + k - cd.t_off;
            s_min[k] = d.nmin[leaf];
            s_max[k] = d.nmax[leaf];
        }
    }
    __syncthreads();
    if (tree) {  // levels over the block's slots: level k's entry e covers slots [e 2^k, (e + 1) 2^k)
        int from = 0;
        for (int n = SPAN / 2; n >= 1; n >>= 1) {
            const int to = from + 2 * n;
            if (t < n && (t + 1) * (SPAN / n) <= B1 - B0) {
                s_min[to + t] = f4(vmin(xyz(s_min[from + 2 * t]), xyz(s_min[from + 2 * t + 1])), 0.f);
                s_max[to + t] = f4(vmax(xyz(s_max[from + 2 * t]), xyz(s_max[from + 2 * t + 1])), 0.f);
            }
            __syncthreads();
            from = to;
        }
    }
#pragma unroll 1
    for (int q = 0; q < SPAN / BS; ++q) {
        const int s = B0 + q * BS + t;
        if (s >= B1) break;
        const int c = d.tcloth[s];
        const ClothDev &cd = d.cloth[c];
        const int id = s - cd.t_off, In = cd.T - 1;
        if (id >= In) continue;
        const BlockKeys m{s_key, B0 - cd.t_off, B1 - B0, false};
        int j, split;
        karras_range(m, id, In, j, split);
        const int first = min(id, j) + cd.t_off - B0, last = max(id, j) + cd.t_off - B0, mid = split + cd.t_off - B0;
        // (a range may end on the neighbouring slot without a search past it, at the cloth's end)
        if (!kWhole && (m.out || first < 0 || last >= B1 - B0)) {
            s_far[atomicAdd(&s_nfar, 1)] = s;
            continue;
        }
        const bool boxes = tree && !d.eq3[c];
        float3 amn, amx, bmn, bmx;
        if (boxes) {
            range_box(s_min, s_max, s_min + SPAN, s_max + SPAN, SPAN, first, mid, amn, amx);
            range_box(s_min, s_max, s_min + SPAN, s_max + SPAN, SPAN, mid + 1, last, bmn, bmx);
        }
        put_node(d, cd, id, j, split, boxes, amn, amx, bmn, bmx);
    }
    if (kWhole) return;
    __syncthreads();
    if (t == 0) s_base = s_nfar ? atomicAdd(d.nfar, (uint32_t)s_nfar) : 0u;
    __syncthreads();
    for (int k = t; k < s_nfar; k += BS) d.far[s_base + k] = s_far[k];
}

// The queued nodes, searched through memory, with the cloth's range tree for
// the boxes: two lanes per node, one for each child's box.
__global__ void __launch_bounds__(kThreads) k_karras_far(DevPtrs d) {
    const uint32_t n = *d.nfar;
    const bool tree = d.eq3 != nullptr;
    const uint32_t lane2 = threadIdx.x & 1u;
    const uint32_t stride = gridDim.x * (kThreads / 2);
    for (uint32_t e0 = (blockIdx.x * kThreads + (threadIdx.x & ~31u)) / 2; e0 < n; e0 += stride) {  // warp-uniform
        const uint32_t e = e0 + (threadIdx.x & 31u) / 2;
        const bool valid = e < n;
        const int s = d.far[valid ? e : e0], c = d.tcloth[s];
        const ClothDev &cd = d.cloth[c];
        const int id = s - cd.t_off, In = cd.T - 1;
        const unsigned long long *m = d.keys + cd.t_off;
        int j, split;
        karras_range(m, id, In, j, split);
        const bool boxes = tree && !d.eq3[c];
        float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
        if (boxes) {
            const float4 *lmin = d.nmin + cd.n_off + In, *lmax = d.nmax + cd.n_off + In;
            const float4 *rmin = d.rmin + cd.t_off + kRangePad * c, *rmax = d.rmax + cd.t_off + kRangePad * c;
            range_box(lmin, lmax, rmin, rmax, cd.T, lane2 ? split + 1 : min(id, j), lane2 ? max(id, j) : split, mn, mx);
        }
        __syncwarp();
        const float3 omn = f3(__shfl_xor_sync(0xffffffffu, mn.x, 1), __shfl_xor_sync(0xffffffffu, mn.y, 1),
                              __shfl_xor_sync(0xffffffffu, mn.z, 1));
        const float3 omx = f3(__shfl_xor_sync(0xffffffffu, mx.x, 1), __shfl_xor_sync(0xffffffffu, mx.y, 1),
                              __shfl_xor_sync(0xffffffffu, mx.z, 1));
        if (valid && lane2 == 0) put_node(d, cd, id, j, split, boxes, mn, mx, omn, omx);
    }
}

// Bottom-up refit: Collision/CudaBVH.cu:128-149.  The second arrival at a
// node unions its children; the arrival counter is an acq_rel atomic, which
// orders the child writes before it, and the children are re-read from L2.
// refit_climb starts at node pid, arriving from a child whose box is written.
__device__ __forceinline__ void refit_climb(const DevPtrs &d, const ClothDev &cd, int pid) {
    const int In = cd.T - 1;
    for (int guard = 0; guard <= cd.T; ++guard) {
        if (pid < 0 || pid >= In) {
            if (pid != 0) atomicOr(d.err, ERR_TREE);
            return;
        }
        // child ids and parent links come from k_karras (an earlier launch):
        // they are read ahead of the counter, so their round trip overlaps
        // the release below instead of following the acquire
        const int2 ch = __ldg(&d.child[cd.i_off + pid]);
        const int up = pid ? __ldg(&d.parent[cd.n_off + pid]) : 0;
        // acq_rel at device scope: releases this thread's writes of the child
        // it came from, and the second arrival acquires the first one's
        // (the reference's arrival counter has no ordering at all)
        cuda::atomic_ref<int, cuda::thread_scope_device> visit(d.visit[cd.i_off + pid]);
        if (visit.fetch_add(1, cuda::memory_order_acq_rel) == 0) return;
        const float4 lmn = __ldcg(&d.nmin[cd.n_off + ch.x]), lmx = __ldcg(&d.nmax[cd.n_off + ch.x]);
        const float4 rmn = __ldcg(&d.nmin[cd.n_off + ch.y]), rmx = __ldcg(&d.nmax[cd.n_off + ch.y]);
        d.nmin[cd.n_off + pid] = f4(vmin(xyz(lmn), xyz(rmn)), 0.f);
        d.nmax[cd.n_off + pid] = f4(vmax(xyz(lmx), xyz(rmx)), 0.f);
        int rl, rr;
        if (ch.x >= In) rl = ch.x;
        else { const int2 q = __ldcg(&d.rml[cd.i_off + ch.x]); rl = max(q.x, q.y); }
        if (ch.y >= In) rr = ch.y;
        else { const int2 q = __ldcg(&d.rml[cd.i_off + ch.y]); rr = max(q.x, q.y); }
        d.rml[cd.i_off + pid] = make_int2(rl, rr);
        if (pid == 0) return;
        pid = up;
    }
    atomicOr(d.err, ERR_TREE);
}

constexpr int kRefitBlock = 1024;
// One thread per leaf, the whole climb in L2 (the allocation-free entry).
__global__ void k_refit(DevPtrs d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.Ttot) return;
    const ClothDev &cd = d.cloth[d.tcloth[s]];
    const int id = s - cd.t_off;
    const int In = cd.T - 1;
    if (In <= 0) return;
    refit_climb(d, cd, d.parent[cd.n_off + In + id]);
}

// The same refit in two launches.  k_refit_local: block b owns the slots
// [256 b, 256 b + 256); an internal node whose leaf range [min(i, j),
// max(i, j)] lies inside one block (node i sits at one end of its range, so
// its slot is inside too) is "local": its arrival counter, box and rightmost
// leaves live in that block's shared memory (block-scope acq_rel counter),
// and its box is also written out.  A thread that reaches a node whose
// range crosses a block boundary stops there and leaves the arrival to
// k_refit_upper (each thread leaves at most one); the block writes its
// arrivals out densely, one global atomic per block.  k_refit_upper then
// climbs from the few left arrivals in L2 as k_refit does, so no block of
// the launch over all leaves waits on a climb to the root.
// Every arrival at a local node comes from inside its block: the ranges
// come from the index-tiebroken prefix (unique keys), so any two ranges are
// nested or disjoint, and an internal child is strictly inside its
// parent's range (a child at the range's end is a leaf), so its own range
// lies inside too -- also where equal codes make two nodes claim one child.
// Shared boxes start at zero, like the global ones k_karras clears.
__global__ void __launch_bounds__(kThreads) k_refit_local(DevPtrs d) {
    __shared__ float4 s_lmin[kThreads], s_lmax[kThreads];  // the block's leaves
    __shared__ float4 s_min[kThreads], s_max[kThreads];    // local internal nodes, by slot
    __shared__ int2 s_rml[kThreads];
    __shared__ int s_visit[kThreads];
    __shared__ int2 s_exit[kThreads];
    __shared__ uint32_t s_nexit, s_base;
    const int tid = threadIdx.x;
    const int B0 = blockIdx.x * kThreads, B1 = min(B0 + kThreads, d.Ttot);
    const int s = B0 + tid;
    const bool valid = s < d.Ttot && d.eq3[d.tcloth[s]];  // the other cloths' nodes are complete
    if (!__syncthreads_or(valid)) return;
    int c = 0, id = 0, In = 0;
    const ClothDev *cdp = nullptr;
    s_visit[tid] = 0;
    s_min[tid] = s_max[tid] = make_float4(0.f, 0.f, 0.f, 0.f);
    s_rml[tid] = make_int2(0, 0);
    if (tid == 0) s_nexit = 0;
    if (valid) {
        c = d.tcloth[s];
        cdp = &d.cloth[c];
        id = s - cdp->t_off;
        In = cdp->T - 1;
        s_lmin[tid] = __ldg(&d.nmin[cdp->n_off + In + id]);
        s_lmax[tid] = __ldg(&d.nmax[cdp->n_off + In + id]);
    }
    __syncthreads();
    if (valid && In > 0) {
        const ClothDev &cd = *cdp;
        const int base = cd.t_off - B0;  // cloth-local index -> block slot
        int pid = d.parent[cd.n_off + In + id];
        for (int guard = 0;; ++guard) {
            if (guard > cd.T) {
                atomicOr(d.err, ERR_TREE);
                break;
            }
            if (pid < 0 || pid >= In) {
                if (pid != 0) atomicOr(d.err, ERR_TREE);
                break;
            }
            const int je = __ldg(&d.nend[cd.i_off + pid]);
            const int lo = min(pid, je) + base, hi = max(pid, je) + base;
            if (lo < 0 || hi >= B1 - B0) {  // crosses a block boundary: the upper pass arrives
                const uint32_t e = atomicAdd(&s_nexit, 1u);
                s_exit[e] = make_int2(c, pid);
                break;
            }
            const int2 ch = __ldg(&d.child[cd.i_off + pid]);
            const int up = pid ? __ldg(&d.parent[cd.n_off + pid]) : 0;
            cuda::atomic_ref<int, cuda::thread_scope_block> visit(s_visit[pid + base]);
            if (visit.fetch_add(1, cuda::memory_order_acq_rel) == 0) break;
            const bool la = ch.x >= In, lb = ch.y >= In;
            const int ia = (la ? ch.x - In : ch.x) + base, ib = (lb ? ch.y - In : ch.y) + base;
            if (ia < 0 || ia >= B1 - B0 || ib < 0 || ib >= B1 - B0) {  // children outside the range: not a tree
                atomicOr(d.err, ERR_TREE);
                break;
            }
            const float4 amn = la ? s_lmin[ia] : s_min[ia], amx = la ? s_lmax[ia] : s_max[ia];
            const float4 bmn = lb ? s_lmin[ib] : s_min[ib], bmx = lb ? s_lmax[ib] : s_max[ib];
            const float4 mn = f4(vmin(xyz(amn), xyz(bmn)), 0.f), mx = f4(vmax(xyz(amx), xyz(bmx)), 0.f);
            int rl, rr;
            if (la) rl = ch.x;
            else { const int2 q = s_rml[ia]; rl = max(q.x, q.y); }
            if (lb) rr = ch.y;
            else { const int2 q = s_rml[ib]; rr = max(q.x, q.y); }
            s_min[pid + base] = mn;
            s_max[pid + base] = mx;
            s_rml[pid + base] = make_int2(rl, rr);
            d.nmin[cd.n_off + pid] = mn;
            d.nmax[cd.n_off + pid] = mx;
            d.rml[cd.i_off + pid] = make_int2(rl, rr);
            if (pid == 0) break;
            pid = up;
        }
    }
    __syncthreads();
    if (tid == 0) s_base = s_nexit ? atomicAdd(d.nrexit, s_nexit) : 0u;
    __syncthreads();
    if ((uint32_t)tid < s_nexit) d.rexit[s_base + tid] = s_exit[tid];
}
__global__ void k_refit_upper(DevPtrs d) {
    const uint32_t n = *d.nrexit;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int2 x = d.rexit[e];
        refit_climb(d, d.cloth[x.x], x.y);
    }
}

// Wide node records for the traversal: per internal node both children's
// boxes, with the child ids and rightmost leaves in the w lanes, so that one
// node visit is one contiguous 64-byte read instead of six dependent ones.
// For the cloths that took the climb, and after it, not part of it: a node
// the refit never reaches (a run of >= 3 equal codes, see k_karras) still gets
// its record from its children's boxes, as the per-node reads of the traversal
// see them.
__global__ void k_pack_nodes(DevPtrs d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.Ttot || !d.eq3[d.tcloth[s]]) return;
    const ClothDev &cd = d.cloth[d.tcloth[s]];
    const int k = s - cd.t_off;
    if (k >= cd.T - 1) return;
    const int2 ch = d.child[cd.i_off + k];
    const float4 *nmin = d.nmin + cd.n_off, *nmax = d.nmax + cd.n_off;
    put_wnode(d, (size_t)(cd.i_off + k), xyz(nmin[ch.x]), xyz(nmax[ch.x]), xyz(nmin[ch.y]), xyz(nmax[ch.y]), ch,
              d.rml[cd.i_off + k]);
}

// Climb and records of flagged cloths in one launch, `per` blocks per cloth, the
// last of which to arrive writes the records: where the three launches above cost
// more than they do.
__global__ void __launch_bounds__(kRefitBlock) k_refit_block(DevPtrs d, int per) {
    __shared__ int s_last;
    const int c = blockIdx.x / per;
    if (!d.eq3[c]) return;
    const ClothDev &cd = d.cloth[c];
    const int In = cd.T - 1;
    for (int id = (blockIdx.x % per) * kRefitBlock + threadIdx.x; id <= In && In > 0; id += per * kRefitBlock)
        refit_climb(d, cd, d.parent[cd.n_off + In + id]);
    __threadfence();
    __syncthreads();
    if (per > 1) {
        if (threadIdx.x == 0) {
            s_last = atomicAdd(&d.tree_done[c], 1) == per - 1;
            if (s_last) d.tree_done[c] = 0;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
    }
    const float4 *nmin = d.nmin + cd.n_off, *nmax = d.nmax + cd.n_off;
    for (int k = threadIdx.x; k < In; k += kRefitBlock) {
        const int2 ch = d.child[cd.i_off + k];
        put_wnode(d, (size_t)(cd.i_off + k), xyz(__ldcg(&nmin[ch.x])), xyz(__ldcg(&nmax[ch.x])), xyz(__ldcg(&nmin[ch.y])),
                  xyz(__ldcg(&nmax[ch.y])), ch, __ldcg(&d.rml[cd.i_off + k]));
    }
}

// Leaf-vs-tree traversal: Collision/CudaBVH.cu:23-113.  Pairs (i, j>i) in
// left-first DFS order, at most `chunk` per leaf, the rest counted as dropped.
__global__ void k_traverse(DevPtrs d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.Ttot) return;
    const int c = d.tcloth[s];
    const ClothDev &cd = d.cloth[c];
    const int id = s - cd.t_off;
    const int In = cd.T - 1;
    if (In <= 0) { d.pair_cnt[s] = 0; return; }
    const int me = In + id;
    const int chunk = cd.chunk;
    uint32_t *out = d.pair_chunk + cd.pc_off + (int64_t)id * chunk;
    const float4 *nmin = d.nmin + cd.n_off, *nmax = d.nmax + cd.n_off;
    const int2 *child = d.child + cd.i_off, *rml = d.rml + cd.i_off;
    const float3 amin = xyz(nmin[me]), amax = xyz(nmax[me]);
    int stack[kTraverseStack];
    stack[0] = -1;
    int top = 1, node = 0, got = 0;
    uint32_t dropped = 0;
    const int guard_max = 4 * cd.T + 64;
    for (int guard = 0; guard < guard_max; ++guard) {
        const int2 ch = __ldg(&child[node]);
        const int2 rm = __ldg(&rml[node]);
        bool ol = false, orr = false;
        if (rm.x > me && overlap(amin, amax, xyz(__ldg(&nmin[ch.x])), xyz(__ldg(&nmax[ch.x])))) ol = true;
        if (rm.y > me && overlap(amin, amax, xyz(__ldg(&nmin[ch.y])), xyz(__ldg(&nmax[ch.y])))) orr = true;
        if (ol && ch.x >= In) {
            if (got < chunk) out[got++] = (uint32_t)(ch.x - In);
            else ++dropped;
        }
        if (orr && ch.y >= In) {
            if (got < chunk) out[got++] = (uint32_t)(ch.y - In);
            else ++dropped;
        }
        const bool tl = ol && ch.x < In, tr = orr && ch.y < In;
        if (!tl && !tr) {
            node = stack[--top];
        } else {
            node = tl ? ch.x : ch.y;
            if (tl && tr) {
                if (top >= kTraverseStack) { atomicOr(d.err, ERR_STACK); break; }
                stack[top++] = ch.y;
            }
        }
        if (top == 0) break;
    }
    d.pair_cnt[s] = (uint32_t)got;
    if (dropped) atomicAdd(&d.counters[3], (unsigned long long)dropped);
}

// The single-leaf traversal over the records, one thread per leaf; a record is
// two 32-byte loads.  Bound by the latency of the walk in a small batch, by the
// records' L1 traffic in a large one.  A walk per 32 leaves, which read each
// record once for all, was slower from the smallest batch (43 us against 24 for
// 1922 leaves) to the largest (987 against 917 for 1.92 million, 1568 against
// 1509 for 3.3 million): every leaf then waits for the records of all.  With
// four 16-byte loads 442 us for 619 k leaves, 383 so; a million random boxes 95.
__global__ void __launch_bounds__(kTraverseBlockMax) k_traverse_leaf(DevPtrs d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.Ttot) return;
    const ClothDev &cd = d.cloth[d.tcloth[s]];
    const int id = s - cd.t_off;
    const int In = cd.T - 1;
    if (In <= 0) { d.pair_cnt[s] = 0; return; }
    const int me = In + id;
    const int chunk = cd.chunk;
    uint32_t *out = d.pair_chunk + cd.pc_off + (int64_t)id * chunk;
    const float3 amin = xyz(d.nmin[cd.n_off + me]), amax = xyz(d.nmax[cd.n_off + me]);
    const float4 *W = d.wnode + 4 * (size_t)cd.i_off;
    int stack[kTraverseStack];
    int top = 0, node = 0, got = 0;
    uint32_t dropped = 0;
    const int guard_max = 4 * cd.T + 64;
    for (int guard = 0; guard < guard_max; ++guard) {
        const float4 *r = W + 4 * (size_t)node;
        float4 l0, l1, r0, r1;
        ld_pair(r, l0, l1);
        ld_pair(r + 2, r0, r1);
        const int chx = __float_as_int(l0.w), rmx = __float_as_int(l1.w);
        const int chy = __float_as_int(r0.w), rmy = __float_as_int(r1.w);
        const bool ol = rmx > me && overlap(amin, amax, xyz(l0), xyz(l1));
        const bool orr = rmy > me && overlap(amin, amax, xyz(r0), xyz(r1));
        if (ol && chx >= In) {
            if (got < chunk) out[got++] = (uint32_t)(chx - In);
            else ++dropped;
        }
        if (orr && chy >= In) {
            if (got < chunk) out[got++] = (uint32_t)(chy - In);
            else ++dropped;
        }
        const bool tl = ol && chx < In, tr = orr && chy < In;
        if (tl) {
            node = chx;
            if (tr) {
                if (top >= kTraverseStack - 1) { atomicOr(d.err, ERR_STACK); break; }
                stack[top++] = chy;
            }
        } else if (tr) {
            node = chy;
        } else {
            if (top == 0) break;
            node = stack[--top];
        }
    }
    d.pair_cnt[s] = (uint32_t)got;
    if (dropped) atomicAdd(&d.counters[3], (unsigned long long)dropped);
}

// Order-preserving compaction of the per-leaf chunks into the pair list: a
// warp takes `per` leaves and copies those with pairs four at a time, eight lanes
// each (a leaf of a cloth at rest has ten pairs).  Four leaves per warp while the
// latency of one copy is what a launch takes, 32 when it is the number of
// warps (us, 4 / 32: 1922 leaves 6 / 16, 20 k 7 / 22, 130 k 12 / 12, 522 k 35 / 24, a million of cloths in
// contact 166 / 150, a million with a pair in 15 31 / 11; with lanes that look
// up their leaf for every output 18, 33, -, 181, 11).
constexpr int kCompactLanes = 8, kCompactManyLeaves = 1 << 17;
__global__ void k_pair_compact(DevPtrs d, int per) {
    const int lane = threadIdx.x & 31;
    const int64_t base = (int64_t)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5) * per;
    const uint32_t n = lane < per && base + lane < d.Ttot ? d.pair_cnt[base + lane] : 0u;
    const unsigned some = __ballot_sync(0xffffffffu, n != 0u);
    const int nsome = __popc(some), sub = lane / kCompactLanes;
    for (int r = 0; r < nsome; r += 32 / kCompactLanes) {
        const int pick = r + sub;
        const int L = pick < nsome ? (int)__fns(some, 0, pick + 1) : 0;
        const uint32_t nL = __shfl_sync(0xffffffffu, n, L);
        if (pick >= nsome) continue;
        const int leaf = (int)base + L;
        const uint32_t o = d.pair_off[leaf];
        const ClothDev &cd = d.cloth[d.tcloth[leaf]];
        const uint32_t *src = d.pair_chunk + cd.pc_off + (int64_t)(leaf - cd.t_off) * cd.chunk;
        for (uint32_t k = lane & (kCompactLanes - 1); k < nL; k += kCompactLanes)
            d.pairs[o + k] = make_uint2((uint32_t)leaf, (uint32_t)cd.t_off + src[k]);
    }
}

// ---------------------------------------------------------------------------
// Narrowphase.  Candidate slots of Collision/CudaCollisionDetection.cu:53-189,
// feature AABB cull of Collision/CudaPrimitiveTests.cu:427-490, CCD of
// :109-238 with Physics/CudaCubicSolver.cu:5-153 and the tests at :252-425.
// ---------------------------------------------------------------------------
// A hit's weights, normal and time (Physics::PrimitiveContact w1..w4, n, t).
// The tests write t where the reference's do (TestVF: 0; TestEE outside the
// segments: 0); the caller starts it at the candidate's -1.
struct Wts { float w0, w1, w2, w3; float3 n; float t; };

__device__ __forceinline__ float triple(float3 x21, float3 x31, float3 x41, float3 v21, float3 v31, float3 v41,
                                        float t) {
    return dot(cross(add(x21, mul(v21, t)), add(x31, mul(v31, t))), add(x41, mul(v41, t)));
}
// Physics/CudaCubicSolver.cu:131-153.  The reference evaluates f at both
// ends every iteration; f(x0) of an iteration is f(x1) of the previous one
// (same arguments, same bits), so it is carried over instead of recomputed.
// fa, fb: f(a), f(b) as the caller evaluated them (the same arguments, so
// the same bits as the reference's first-iteration evaluations).
__device__ float secant(float3 x21, float3 x31, float3 x41, float3 v21, float3 v31, float3 v41, float a, float b,
                        float fa, float fb) {
    float x0 = a, x1 = b;
    float f0 = fa;
    for (int i = 0; i < 20; ++i) {
        const float f1 = i == 0 ? fb : triple(x21, x31, x41, v21, v31, v41, x1);
        const float xc = (x0 * f1 - x1 * f0) / (f1 - f0);
        if (fabsf(xc - x1) < kEpsCubic) return xc;
        x0 = x1;
        f0 = f1;
        x1 = xc;
    }
    return -15.f;
}
__device__ __forceinline__ float3 project_on_line(float3 p, float3 e1, float3 e2) {
    const float3 ab = sub(e2, e1), ap = sub(p, e1);
    return add(e1, mul(ab, dot(ap, ab) / dot(ab, ab)));
}
__device__ __forceinline__ float3 clamp_on_line(float3 p, float3 e1, float3 e2) {
    const float d1 = dist(p, e1), d2 = dist(p, e2);
    if (fabsf(d1 + d2 - dist(e1, e2)) < kEpsPbd) return p;
    return d1 < d2 ? e1 : e2;
}

__device__ bool test_vf(float3 x4, float3 x1, float3 x2, float3 x3, float th, Wts &w) {
    const float3 x13 = sub(x1, x3), x23 = sub(x2, x3), x43 = sub(x4, x3);
    const float3 crs = cross(sub(x2, x1), sub(x3, x1));
    const float3 n = normalize(crs);
    if (fabsf(dot(x43, n)) <= th) {
        const float dt = dot(x13, x23);
        const float m11 = dot(x13, x13), m12 = dt, m21 = dt, m22 = dot(x23, x23);
        const float vr1 = dot(x13, x43), vr2 = dot(x23, x43);
        const float w2 = (m11 * vr2 - m21 * vr1) / (m11 * m22 - m21 * m12);
        const float w1 = (vr1 - m12 * w2) / m11;
        const float w3 = 1.f - w1 - w2;
        const float del = th / (len(x13) + len(x23) + len(sub(x1, x2)));
        const float lo = 0.f, hi = 1.f + del;
        if (between(w1, lo, hi) && between(w2, lo, hi) && between(w3, lo, hi)) {
            w.w0 = 1.f; w.w1 = -w1; w.w2 = -w2; w.w3 = -w3;
            w.n = n;
            w.t = 0.f;
            return true;
        }
    }
    return false;
}

__device__ bool test_ee(float3 x1, float3 x2, float3 x3, float3 x4, float th, Wts &w) {
    const float3 x21 = sub(x2, x1), x31 = sub(x3, x1), x43 = sub(x4, x3);
    const float3 crs = cross(x21, x43);
    if (len(crs) < kEpsEE) {
        const float3 m1 = add(x1, dvs(x21, 2.f)), m2 = add(x3, dvs(x43, 2.f));
        if (dist(m1, m2) <= th) {
            w.w0 = w.w1 = w.w2 = w.w3 = 0.5f;
            w.n = normalize(sub(m1, m2));
            return true;
        }
        return false;
    }
    if (is_zero(crs)) return false;
    const float dt = dot(neg(x21), x43);
    const float m11 = dot(x21, x21), m12 = dt, m21 = dt, m22 = dot(x43, x43);
    const float vr1 = dot(x21, x31), vr2 = dot(neg(x43), x31);
    float b = (m11 * vr2 - m21 * vr1) / (m11 * m22 - m21 * m12);
    float a = (vr1 - m12 * b) / m11;
    if (between(a, 0.f, 1.f) && between(b, 0.f, 1.f)) {
        const float3 cp1 = add(x1, mul(x21, a)), cp2 = add(x3, mul(x43, a));
        if (dist(cp1, cp2) <= th) {
            w.w0 = 1.f - a; w.w1 = a; w.w2 = -(1.f - b); w.w3 = -b;
            // the normal measures the second point with b (Collision/CudaPrimitiveTests.cu:305-307)
            const float3 dir = sub(add(x1, mul(x21, a)), add(x3, mul(x43, b)));
            w.n = normalize(is_zero(dir) ? crs : dir);
            return true;
        }
    } else {
        const float ac = clampf(a, 0.f, 1.f), bc = clampf(b, 0.f, 1.f);
        const float d1 = fabsf(a - ac) * len(x21), d2 = fabsf(b - bc) * len(x43);
        a = ac;
        b = bc;
        float3 cp1, cp2;
        if (d1 > d2) {
            cp1 = add(x1, mul(x21, a));
            cp2 = clamp_on_line(project_on_line(cp1, x3, x4), x3, x4);
        } else {
            cp2 = add(x3, mul(x43, b));
            cp1 = clamp_on_line(project_on_line(cp2, x1, x2), x1, x2);
        }
        if (dist(cp1, cp2) <= th) {
            w.w0 = 1.f - a; w.w1 = a; w.w2 = -(1.f - b); w.w3 = -b;
            w.n = normalize(sub(cp1, cp2));
            w.t = 0.f;
            return true;
        }
    }
    return false;
}

// A test_ee hit places both closest points on their segments (the parallel
// case uses the midpoints, the others clamp the parameters to [0,1]), up to
// a few float roundings of the coordinates, and needs their distance <= th.
// So edges whose boxes are apart by more than th plus a margin far above
// those roundings (1e-5 m + th/1000) cannot hit, and the test is skipped:
// the decision and the weights are the reference's bits either way.
__device__ __forceinline__ bool ee_far(float3 a, float3 b, float3 c, float3 d, float th) {
    const float m = th + 1e-5f + 1e-3f * th;
    return fminf(a.x, b.x) - fmaxf(c.x, d.x) > m || fminf(c.x, d.x) - fmaxf(a.x, b.x) > m ||
           fminf(a.y, b.y) - fmaxf(c.y, d.y) > m || fminf(c.y, d.y) - fmaxf(a.y, b.y) > m ||
           fminf(a.z, b.z) - fmaxf(c.z, d.z) > m || fminf(c.z, d.z) - fmaxf(a.z, b.z) > m;
}

// Whether two edges moving with constant velocities are further apart than a
// test_ee hit allows at every advance T of [lo, hi]: their projections on one
// axis, the line through their midpoints halfway, are apart by more than th
// plus the margin at both ends (the gap, a minimum of linear functions of T less
// a maximum of such, is concave, so nowhere between the ends is it smaller).  The margin
// also covers what roundings add at the size S of the coordinates, the largest
// over the vertices of |x| + T |v|: a vertex advanced six times at most is off
// by 13 u S (u = 2^-24, half a spacing), so two edges by 26 u S; the gap as
// computed here by 53 u S; the test's closest points by less than 20 u S:
// below 6e-6 S = 100 u S together.  NaN anywhere: not apart.
__device__ __forceinline__ bool ee_apart(float3 x1, float3 x2, float3 x3, float3 x4, float3 v1, float3 v2, float3 v3,
                                         float3 v4, float lo, float hi, float th) {
    const float3 u = sub(x2, x1), v = sub(x3, x1), w = sub(x4, x1);
    const float3 du = sub(v2, v1), dv = sub(v3, v1), dw = sub(v4, v1);
    const float mid = 0.5f * (lo + hi);
    const float3 m = add(sub(add(v, w), u), mul(sub(add(dv, dw), du), mid));
    const float pu = dot(u, m), pv = dot(v, m), pw = dot(w, m);
    const float qu = dot(du, m), qv = dot(dv, m), qw = dot(dw, m);
    const float gl = fminf(pv + qv * lo, pw + qw * lo) - fmaxf(pu + qu * lo, 0.f);
    const float gh = fminf(pv + qv * hi, pw + qw * hi) - fmaxf(pu + qu * hi, 0.f);
    const float T = fmaxf(fabsf(lo), fabsf(hi));
    auto reach = [&](float3 x, float3 vel) {
        return fabsf(x.x) + fabsf(x.y) + fabsf(x.z) + T * (fabsf(vel.x) + fabsf(vel.y) + fabsf(vel.z));
    };
    const float size = fmaxf(fmaxf(reach(x1, v1), reach(x2, v2)), fmaxf(reach(x3, v3), reach(x4, v4)));
    const float t = 1.001f * th + 1e-5f + 6e-6f * size;
    return fminf(gl, gh) > 0.f && gl * gl > t * t * dot(m, m) && gh * gh > t * t * dot(m, m);
}

// Particle swept box of Collision/FeatureList.cu:134-148, recomputed from
// x and x_prev (min/max are exact, so this equals the stored boxes).
struct Box { float3 lo, hi; };
__device__ __forceinline__ Box pbox(const DevPtrs &d, int v, float h) {
    if (d.vbox) {  // the same operations, once per vertex
        float4 lo, hi;
        ld_pair(d.vbox + 2 * (size_t)v, lo, hi);
        return Box{xyz(lo), xyz(hi)};
    }
    const float3 p = xyz(d.x[v]), q = xyz(d.xp[v]);
    return Box{subc(vmin(p, q), h), addc(vmax(p, q), h)};
}

// EE slot s: edge (s%3) of A x edge (s/3) of B; edge k of a triangle is
// (v1,v2 | bit 2), (v1,v3 | bit 0), (v2,v3 | bit 1).
__device__ __forceinline__ void edge_of(int k, int &a, int &b, int &bit) {
    if (k == 0) { a = 0; b = 1; bit = 2; }
    else if (k == 1) { a = 0; b = 2; bit = 0; }
    else { a = 1; b = 2; bit = 1; }
}

// Vertex ids of candidate slot s of a pair (A, B): VF slots 0..5 are
// (vertex s of A | face B) then (vertex s-3 of B | face A); EE slots 6..14 are
// edge (s-6)%3 of A x edge (s-6)/3 of B (Collision/CudaCollisionDetection.cu:101-187).
__device__ __forceinline__ int4 candidate_ids(const int vid[6], int s) {
    if (s < 6) {
        const int o = s < 3 ? 3 : 0;
        return make_int4(vid[s], vid[o], vid[o + 1], vid[o + 2]);
    }
    int a0, a1, ab, b0, b1, bb;
    edge_of((s - 6) % 3, a0, a1, ab);
    edge_of((s - 6) / 3, b0, b1, bb);
    return make_int4(vid[a0], vid[a1], vid[3 + b0], vid[3 + b1]);
}

// Stage 1 of the narrowphase: the candidates of one broadphase pair that
// survive feature ownership, the shared-vertex sanity checks and the feature
// AABB cull (Collision/CudaPrimitiveTests.cu:240-248, 427-490).  The checks
// commute, so the surviving set is the reference's; the six vertex boxes are
// built once per pair.  Bound by the gathers of boxes out of L1 and by issue
// slots: the ownership and shared-vertex checks as bit sets instead of one by
// one 204 -> 178 us for 9.7 million pairs, a box in one load 172; without
// branches in the overlap tests 183, more blocks per SM (spills) 218.
__device__ __forceinline__ uint16_t pair_filter(const DevPtrs &d, uint2 pr, bool cull) {
    const float h = d.vbox ? 0.f : d.cloth[d.tcloth[pr.x]].h;
    const int4 A = d.tri_slot[pr.x], B = d.tri_slot[pr.y];
    const unsigned fa = (unsigned)A.w, fb = (unsigned)B.w;
    const int vid[6] = {A.x, A.y, A.z, B.x, B.y, B.z};
    // Row i: which vertices of B vertex i of A is.  A vertex of one triangle that
    // is a vertex of the other makes no VF candidate, edges with a vertex in
    // common no EE candidate.
    unsigned row[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        row[k] = (vid[k] == B.x ? 1u : 0u) | (vid[k] == B.y ? 2u : 0u) | (vid[k] == B.z ? 4u : 0u);
    // ownership: vertex k of a triangle by bit 5 - k, edges 0, 1, 2 by bits 2, 0, 1
    const unsigned va = (__brev(fa) >> 26) & 7u, vb = (__brev(fb) >> 26) & 7u;
    const unsigned ea = ((fa << 1) & 6u) | ((fa >> 2) & 1u), eb = ((fb << 1) & 6u) | ((fb >> 2) & 1u);
    const unsigned sa = (row[0] ? 1u : 0u) | (row[1] ? 2u : 0u) | (row[2] ? 4u : 0u), sb = row[0] | row[1] | row[2];
    auto spread = [](unsigned b) { return (b & 1u) | (b & 2u) << 2 | (b & 4u) << 4; };  // bit k to bit 3 k
    // the edges of B that have one of the vertices r (bits): 0 0 1, 0 2, 1 2
    auto touched = [](unsigned r) { return (077767530u >> (3 * r)) & 7u; };
    const unsigned shared = spread(touched(row[0] | row[1])) | spread(touched(row[0] | row[2])) << 1 |
                            spread(touched(row[1] | row[2])) << 2;
    const uint32_t want = (va & ~sa) | (vb & ~sb) << 3 | ((ea * spread(eb)) & ~shared) << 6;
    if (!want || !cull) return (uint16_t)want;
    // the six vertex boxes, the two face boxes and the six edge boxes once
    // (min / max are exact, so any grouping gives the reference's boxes)
    Box bx[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) bx[k] = pbox(d, vid[k], h);
    Box face[2], edge[6];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        face[t] = Box{min3(bx[3 * t].lo, bx[3 * t + 1].lo, bx[3 * t + 2].lo),
                      max3(bx[3 * t].hi, bx[3 * t + 1].hi, bx[3 * t + 2].hi)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            int a0, a1, ab;
            edge_of(k, a0, a1, ab);
            edge[3 * t + k] = Box{vmin(bx[3 * t + a0].lo, bx[3 * t + a1].lo), vmax(bx[3 * t + a0].hi, bx[3 * t + a1].hi)};
        }
    }
    uint32_t mask = 0;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        const Box &f = face[s < 3 ? 1 : 0];
        if (((want >> s) & 1) && overlap(bx[s].lo, bx[s].hi, f.lo, f.hi)) mask |= 1u << s;
    }
#pragma unroll
    for (int s = 0; s < 9; ++s) {
        const Box &ea = edge[s % 3], &eb = edge[3 + s / 3];
        if (((want >> (6 + s)) & 1) && overlap(ea.lo, ea.hi, eb.lo, eb.hi)) mask |= 1u << (6 + s);
    }
    return (uint16_t)mask;
}


// Stage 1 for every pair, one thread per pair: its candidate mask, and per
// group of kPairGroup consecutive pairs (one warp iteration: the stride is a
// whole number of warps) the group's VF and EE candidate counts, whose scans
// give every group its first candidate; the number of groups at ngroups.
// cull = 0 keeps the candidates the ownership bits and the sanity checks
// leave, without the feature AABB cull (the discrete tests of
// Collision/CudaCollisionDetection.cu:191-221 apply none).
__global__ void __launch_bounds__(kThreads, 4) k_narrow_filter(DevPtrs d, const uint32_t *__restrict__ npairs,
                                                               int cull) {
    static_assert(kPairGroup == 32, "a group is one warp iteration");
    const uint32_t n = *npairs, G = (n + kPairGroup - 1) / kPairGroup;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *d.ngroups = G;
        d.hit_n[0] = d.hit_n[1] = 0;
    }
    const int lane = threadIdx.x & 31;
    const uint32_t end = G * kPairGroup;  // whole warps stay in the loop together (pair counts stay below 2^31)
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < end; p += gridDim.x * blockDim.x) {
        const uint16_t m = p < n ? pair_filter(d, d.pairs[p], cull != 0) : (uint16_t)0;
        if (p < n) d.pair_mask[p] = m;
        const uint32_t vf = __reduce_add_sync(0xffffffffu, (unsigned)__popc((unsigned)(m & 0x3Fu)));
        const uint32_t ee = __reduce_add_sync(0xffffffffu, (unsigned)__popc((unsigned)(m >> 6)));
        if (lane == 0) { d.grp_vf_cnt[p / kPairGroup] = vf; d.grp_ee_cnt[p / kPairGroup] = ee; }
    }
}

// First VF (or EE) candidate of pair p <= npairs: its group's offset plus the
// candidates of the pairs before it in the group; total when p starts a
// group past the last.
template <bool VF>
__device__ __forceinline__ uint32_t pair_cand_off(const DevPtrs &d, uint32_t p, uint32_t total) {
    const uint32_t g = p / kPairGroup;
    if (g >= *d.ngroups) return total;
    uint32_t o = VF ? d.grp_vf_off[g] : d.grp_ee_off[g];
    for (uint32_t q = g * kPairGroup; q < p; ++q) {
        const unsigned m = d.pair_mask[q];
        o += (uint32_t)__popc(VF ? (m & 0x3Fu) : (m >> 6));
    }
    return o;
}

// Stage 2: the surviving candidates written in the reference's order (pair,
// then slot) as the four vertex ids the CCD needs.  A warp takes 32
// consecutive pairs, whose outputs are contiguous.  Each lane lists its
// pair's candidates (pair, slot) in shared memory at their places; then every
// lane writes, coalesced, what the list says.  Bound by the writes and by
// issue slots.  12 cloths up to 160 squared, 12 million candidates: 101 us when
// every output looked its pair and slot up among the lanes, 63 so.
constexpr int kExpandWarps = kThreads / 32;
__global__ void __launch_bounds__(kThreads) k_narrow_expand(DevPtrs d, const uint32_t *__restrict__ npairs) {
    __shared__ int s_vid[kExpandWarps][32][7];        // padded: lanes of one pair and of its neighbours in other banks
    __shared__ uint16_t s_code[kExpandWarps][32 * 15];  // lane | slot << 5, the warp's VF then its EE candidates
    __shared__ uint32_t s_slot[16];                   // the vertices of a slot (0..5), four bits each
    const uint32_t n = *npairs;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < 15) {
        const int self[6] = {0, 1, 2, 3, 4, 5};
        const int4 v = candidate_ids(self, threadIdx.x);
        s_slot[threadIdx.x] = (uint32_t)(v.x | v.y << 4 | v.z << 8 | v.w << 12);
    }
    __syncthreads();
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp0 * 32u; base < n; base += nwarps * 32u) {
        const uint32_t p = base + lane;
        const uint32_t m = p < n ? d.pair_mask[p] : 0u;
        if (m) {
            const uint2 pr = d.pairs[p];
            const int4 A = d.tri_slot[pr.x], B = d.tri_slot[pr.y];
            int *v = s_vid[w][lane];
            v[0] = A.x; v[1] = A.y; v[2] = A.z; v[3] = B.x; v[4] = B.y; v[5] = B.z;
        }
        // both kinds' counts in one scan
        const uint32_t cnt = (uint32_t)__popc(m & 0x3Fu) | (uint32_t)__popc(m >> 6) << 16;
        uint32_t ex = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(full, ex, o);
            if (lane >= o) ex += t;
        }
        const uint32_t total = __shfl_sync(full, ex, 31), nvf = total & 0xffffu, nee = total >> 16;
        if (!total) continue;
        ex -= cnt;
        uint32_t at = ex & 0xffffu;
        for (uint32_t b = m & 0x3Fu; b; b &= b - 1u) s_code[w][at++] = (uint16_t)(lane | (__ffs(b) - 1) << 5);
        at = nvf + (ex >> 16);
        for (uint32_t b = m & ~0x3Fu; b; b &= b - 1u) s_code[w][at++] = (uint16_t)(lane | (__ffs(b) - 1) << 5);
        __syncwarp();
        const uint64_t vf0 = d.grp_vf_off[base / kPairGroup], ee0 = d.grp_ee_off[base / kPairGroup];
        for (uint32_t j = lane; j < nvf + nee; j += 32) {
            const uint32_t code = s_code[w][j], slot = s_slot[code >> 5];
            const int *v = s_vid[w][code & 31u];
            const int4 ids = make_int4(v[slot & 15u], v[(slot >> 4) & 15u], v[(slot >> 8) & 15u], v[slot >> 12]);
            const bool vf = j < nvf;
            const uint64_t o = vf ? vf0 + j : ee0 + (j - nvf);
            if (o < d.cand_cap) (vf ? d.cand : d.cand_e)[o] = ids;
            else atomicOr(d.err, ERR_CAND_OVERFLOW);
        }
        __syncwarp();
    }
}

// Stage 3: CCD of every candidate of one kind on x_prev and v
// (Collision/CudaPrimitiveTests.cu:109-238, Physics/CudaCubicSolver.cu:5-153).
// VF: vertex x4 against the face x1 x2 x3; EE: edges x1 x2 and x3 x4.  The
// reference collects every coplanarity time of [0,1] (the ends of the
// intervals cut at the derivative's roots where |f| < eps, and the secant
// root of every interval whose ends differ in sign), then advances the four
// positions by v t dt for each time in turn and tests after each advance
// until one test hits.  Here each warp takes 32 candidates at a time:
// (1) every lane sets up its candidate's cubic, evaluates f at the interval
// ends and queues the intervals that need a secant solve; (2) the warp runs
// the queued solves, one per lane; (3) VF: the tests of all candidates and
// times are spread over the lanes; EE: a candidate whose edges stay apart at all
// of its times (ee_apart: 19 in 20 of those of a batch in contact) is done, and
// the others are queued until 32 are together, whose tests one call runs.
// The operands and operations of every piece are the reference's, so the
// decisions are the same bits; only the assignment of work to lanes, and
// which tests that cannot hit are run, differs.  Bound by issue slots, for EE 30%
// set-up and 45% secant solves, with half of the lanes on (22 of 32 have a
// solve, and they end after 7 iterations on average and 16 at the latest).
// 17 million candidates of 24 cloths up to 160 squared, half of them: EE 199 us
// with the tests spread as for VF (47% of the time), 134 so; VF 80.
constexpr int kCcdWarps = 8;
constexpr int kNearCap = 64;  // 31 left over and 32 more

// A hit: its contact's weights, placed at their final index by k_ccd_emit.
template <bool VF>
__device__ __forceinline__ void record_hit(const DevPtrs &d, uint32_t q, const Wts &wt) {
    const uint64_t cap = VF ? d.vf_cap : d.ee_cap;
    const uint32_t slot = atomicAdd(&d.hit_n[VF ? 0 : 1], 1u);
    if (slot < cap) {
        d.hit_q[VF ? 0 : 1][slot] = q;
        d.hit_w[VF ? 0 : 1][slot] = make_float4(wt.w0, wt.w1, wt.w2, wt.w3);
        if (VF && d.hit_nrm) d.hit_nrm[slot] = make_float4(wt.n.x, wt.n.y, wt.n.z, 0.f);
        if (d.hit_tn[VF ? 0 : 1]) d.hit_tn[VF ? 0 : 1][slot] = make_float4(wt.n.x, wt.n.y, wt.n.z, wt.t);
    } else {
        atomicOr(d.err, VF ? ERR_VF_OVERFLOW : ERR_EE_OVERFLOW);
    }
}

// The ordered tests of queued EE candidate q, whose times are t[kNearCap k]:
// the same advances and tests, up to a hit.  A call, not inlined: the loop over
// the candidates then fits the instruction cache (EE 190 -> 171 us).
__device__ __noinline__ void test_near(const DevPtrs &d, uint32_t q, int nt, const float *t) {
    const int4 ids = d.cand_e[q];
    const ClothDev &cd = d.cloth[d.vcloth[ids.x]];
    const float h = cd.h, dt = cd.dt;
    float3 x1 = xyz(d.xp[ids.x]), x2 = xyz(d.xp[ids.y]), x3 = xyz(d.xp[ids.z]), x4 = xyz(d.xp[ids.w]);
    const float3 v1 = xyz(d.v[ids.x]), v2 = xyz(d.v[ids.y]), v3 = xyz(d.v[ids.z]), v4 = xyz(d.v[ids.w]);
    for (int k = 0; k < nt; ++k) {
        const float tt = t[k * kNearCap] * dt;
        x1 = add(x1, mul(v1, tt));
        x2 = add(x2, mul(v2, tt));
        x3 = add(x3, mul(v3, tt));
        x4 = add(x4, mul(v4, tt));
        Wts wt;
        if (ee_far(x1, x2, x3, x4, h) || !test_ee(x1, x2, x3, x4, h, wt)) continue;
        wt.t = tt;  // the contact's time (Collision/CudaPrimitiveTests.cu:174, 228)
        record_hit<false>(d, q, wt);
        atomicOr(&d.hitg_mask[1][q / 32], 1u << (q & 31u));
        atomicAdd(&d.hitg_cnt[1][q / 32], 1u);
        return;
    }
}

template <bool VF>
struct CcdShared {
    float4 geom[kCcdWarps][6][32];     // x1..x4 then v1..v4 (test order) per lane
    float fval[kCcdWarps][4][32];      // f at the interval ends
    float ends[kCcdWarps][2][32];      // the inner ends
    // each lane's times to test, in the reference's order: interval i's start
    // (if f is 0 there) at 2 i, its root at 2 i + 1
    float tq[kCcdWarps][6][32];
    int cloth_of[kCcdWarps][32];
    int best[VF ? kCcdWarps : 1][32];  // VF: each lane's first hitting test (6: none)
    // EE: candidates not apart, until 32 are together
    uint32_t near_q[VF ? 1 : kCcdWarps][kNearCap];
    float near_t[VF ? 1 : kCcdWarps][6][kNearCap];
    uint8_t near_n[VF ? 1 : kCcdWarps][kNearCap];
    uint8_t job_owner[kCcdWarps][96];  // queued secant solves: lane << 2 | interval
};
// Block `block` of nblocks.
template <bool VF>
__device__ __forceinline__ void ccd_run(const DevPtrs &d, const uint32_t *__restrict__ ncand, CcdShared<VF> &sh,
                                        uint32_t block, uint32_t nblocks) {
    auto &geom = sh.geom;
    auto &fval = sh.fval;
    auto &ends = sh.ends;
    auto &tq = sh.tq;
    auto &cloth_of = sh.cloth_of;
    auto &best = sh.best;
    auto &near_q = sh.near_q;
    auto &near_t = sh.near_t;
    auto &near_n = sh.near_n;
    auto &job_owner = sh.job_owner;
    int nnear = 0;
    const uint32_t n = (uint32_t)min((uint64_t)*ncand, d.cand_cap);
    const int4 *list = VF ? d.cand : d.cand_e;
    // hit bits per group of 32 candidates (one warp iteration: base is a
    // multiple of 32); the scan of their counts orders the contacts
    uint32_t *hmask = d.hitg_mask[VF ? 0 : 1], *hcnt = d.hitg_cnt[VF ? 0 : 1];
    if (block == 0 && threadIdx.x == 0) d.hitg_n[VF ? 0 : 1] = (n + 31) / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    const uint32_t nwarps = nblocks * kCcdWarps;
    for (uint32_t base = (block * kCcdWarps + w) * 32u; base < n; base += nwarps * 32u) {
        const uint32_t q = base + lane;
        const bool valid = q < n;
        int4 ids = make_int4(0, 0, 0, 0);
        int ncp = -1;
        float e1 = 1.f, e2 = 1.f;
        unsigned imm = 0, sec = 0;
        if (valid) {
            ids = list[q];
            // VF: face ids.y ids.z ids.w, vertex ids.x (x4); EE: x1..x4 = ids
            const int i1 = VF ? ids.y : ids.x, i2 = VF ? ids.z : ids.y, i3 = VF ? ids.w : ids.z, i4 = VF ? ids.x : ids.w;
            cloth_of[w][lane] = d.vcloth[ids.x];
            const float3 x1 = xyz(d.xp[i1]), x2 = xyz(d.xp[i2]), x3 = xyz(d.xp[i3]), x4 = xyz(d.xp[i4]);
            const float3 v1 = xyz(d.v[i1]), v2 = xyz(d.v[i2]), v3 = xyz(d.v[i3]), v4 = xyz(d.v[i4]);
            const float3 x21 = sub(x2, x1), x31 = sub(x3, x1), x41 = sub(x4, x1);
            const float3 v21 = sub(v2, v1), v31 = sub(v3, v1), v41 = sub(v4, v1);
            geom[w][0][lane] = make_float4(x1.x, x1.y, x1.z, x2.x);
            geom[w][1][lane] = make_float4(x2.y, x2.z, x3.x, x3.y);
            geom[w][2][lane] = make_float4(x3.z, x4.x, x4.y, x4.z);
            geom[w][3][lane] = make_float4(v1.x, v1.y, v1.z, v2.x);
            geom[w][4][lane] = make_float4(v2.y, v2.z, v3.x, v3.y);
            geom[w][5][lane] = make_float4(v3.z, v4.x, v4.y, v4.z);
            const float3 v21v31 = cross(v21, v31), x21v31 = cross(x21, v31), v21x31 = cross(v21, x31),
                         x21x31 = cross(x21, x31);
            const float v1v2v3 = dot(v21v31, v41), x1v2v3 = dot(x21v31, v41), v1x2v3 = dot(v21x31, v41),
                        v1v2x3 = dot(v21v31, x41), x1x2v3 = dot(x21x31, v41), x1v2x3 = dot(x21v31, x41),
                        v1x2x3 = dot(v21x31, x41);
            const float a3 = v1v2v3, b3 = x1v2v3 + v1x2v3 + v1v2x3, c3 = x1x2v3 + x1v2x3 + v1x2x3;
            const float ad = 3.f * a3, bd = 2.f * b3;
            const float disc = 4.f * (b3 * b3 - ad * c3);
            const float sq = sqrtf(disc);
            const float da = 2.f * ad;
            const float t1 = (-bd + sq) / da, t2 = (-bd - sq) / da;
            ncp = 0;
            if (disc >= kEpsCubic) {
                const bool in1 = between(t1, 0.f, 1.f), in2 = between(t2, 0.f, 1.f);
                ncp = (in1 || in2) ? ((in1 && in2) ? 2 : 1) : 0;
            } else if (fabsf(disc) < kEpsCubic) {
                ncp = between(t1, 0.f, 1.f) ? 1 : 0;
            }
            e1 = ncp >= 1 ? t1 : 1.f;
            e2 = ncp == 2 ? t2 : 1.f;
            ends[w][0][lane] = e1;
            ends[w][1][lane] = e2;
            tq[w][0][lane] = 0.f;
            tq[w][2][lane] = e1;
            tq[w][4][lane] = e2;
            float fa = triple(x21, x31, x41, v21, v31, v41, 0.f);
            fval[w][0][lane] = fa;
#pragma unroll 1
            for (int i = 0; i <= ncp; ++i) {
                const float fb = triple(x21, x31, x41, v21, v31, v41, i == ncp ? 1.f : (i == 0 ? e1 : e2));
                fval[w][i + 1][lane] = fb;
                if (fabsf(fa) < kEpsCubic) imm |= 1u << i;
                if (fa * fb < 0.f) sec |= 1u << i;
                fa = fb;
            }
        }
        // the four vertices of lane L's candidate in test order (VF: face x1 x2 x3,
        // vertex x4), as its set-up loaded them
        auto corners = [&](int L, float3 &x1, float3 &x2, float3 &x3, float3 &x4, float3 &v1, float3 &v2,
                           float3 &v3, float3 &v4) {
            const float4(*gm)[32] = geom[w];
            const float4 a = gm[0][L], b = gm[1][L], c = gm[2][L], e = gm[3][L], f = gm[4][L], g = gm[5][L];
            x1 = f3(a.x, a.y, a.z); x2 = f3(a.w, b.x, b.y); x3 = f3(b.z, b.w, c.x); x4 = f3(c.y, c.z, c.w);
            v1 = f3(e.x, e.y, e.z); v2 = f3(e.w, f.x, f.y); v3 = f3(f.z, f.w, g.x); v4 = f3(g.y, g.z, g.w);
        };
        // queue the secant solves of the warp
        int njobs = 0;
#pragma unroll
        for (int i = 0; i <= 2; ++i) {
            const bool want = (sec >> i) & 1u;
            const unsigned m = __ballot_sync(full, want);
            if (want) {
                const int pos = njobs + __popc(m & ((1u << lane) - 1u));
                job_owner[w][pos] = (uint8_t)(lane << 2 | i);
            }
            njobs += __popc(m);
        }
        __syncwarp();
        for (int j = lane; j < njobs; j += 32) {
            const int own = job_owner[w][j] >> 2, iv = job_owner[w][j] & 3;
            float3 x1, x2, x3, x4, v1, v2, v3, v4;
            corners(own, x1, x2, x3, x4, v1, v2, v3, v4);
            // (an outer end's place holds 1 where there are fewer intervals)
            const float a = iv == 0 ? 0.f : ends[w][iv - 1][own], b = iv == 2 ? 1.f : ends[w][iv][own];
            // the set-up's differences, from the same operands
            tq[w][2 * iv + 1][own] = secant(sub(x2, x1), sub(x3, x1), sub(x4, x1), sub(v2, v1), sub(v3, v1), sub(v4, v1), a, b,
                                          fval[w][iv][own], fval[w][iv + 1][own]);
        }
        __syncwarp();
        unsigned times = (imm & 1u) | (imm & 2u) << 1 | (imm & 4u) << 2;
#pragma unroll
        for (int i = 0; i <= 2; ++i)
            if (((sec >> i) & 1u) && tq[w][2 * i + 1][lane] != -15.f) times |= 2u << (2 * i);
        if constexpr (VF) {
            // The ordered tests of every candidate (the reference advances the
            // four positions by v t dt for each time in turn and tests after each
            // advance, stopping at the first hit).  Every (candidate, time) test
            // of the warp is a job of its own, spread evenly over the lanes: a
            // job rebuilds its positions by the same sequence of advances and
            // runs the same test, so it decides the same bits.  A candidate's
            // first hit is its smallest hitting test index; its owner lane then
            // runs that test once more for the weights.
            int nt = 0;
            float hq = 0.f, dtq = 0.f;
            if (valid) {
                for (; times; times &= times - 1u) tq[w][nt++][lane] = tq[w][__ffs(times) - 1][lane];
                hq = d.cloth[cloth_of[w][lane]].h;
                dtq = d.cloth[cloth_of[w][lane]].dt;
            }
            best[w][lane] = 6;
            uint32_t ex = (uint32_t)nt;  // inclusive scan of the test counts
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(full, ex, o);
                if (lane >= o) ex += t;
            }
            const uint32_t ntests = __shfl_sync(full, ex, 31);
            ex -= (uint32_t)nt;
            __syncwarp();
            // test m of lane L's candidate: the advances by its times 0..m, then the test
            auto run_test = [&](int L, int m, float h, float dt, Wts &wt) {
                float3 x1, x2, x3, x4, v1, v2, v3, v4;
                corners(L, x1, x2, x3, x4, v1, v2, v3, v4);
                float tt = 0.f;
                for (int k = 0; k <= m; ++k) {
                    tt = tq[w][k][L] * dt;
                    x1 = add(x1, mul(v1, tt));
                    x2 = add(x2, mul(v2, tt));
                    x3 = add(x3, mul(v3, tt));
                    x4 = add(x4, mul(v4, tt));
                }
                const bool r = test_vf(x4, x1, x2, x3, h, wt);
                wt.t = tt;  // the contact's time (Collision/CudaPrimitiveTests.cu:174, 228)
                return r;
            };
            for (uint32_t j0 = 0; j0 < ntests; j0 += 32) {
                const uint32_t j = j0 + lane;
                int L = 0;  // owner: the last lane whose first test is <= j
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int cand = L + step;
                    const uint32_t e = __shfl_sync(full, ex, cand & 31);
                    if (cand < 32 && e <= j) L = cand;
                }
                const uint32_t exL = __shfl_sync(full, ex, L);
                const float h = __shfl_sync(full, hq, L), dt = __shfl_sync(full, dtq, L);
                if (j < ntests) {
                    const int m = (int)(j - exL);
                    Wts wt;
                    if (run_test(L, m, h, dt, wt)) atomicMin(&best[w][L], m);
                }
            }
            __syncwarp();
            bool found = false;
            Wts wt;
            if (valid && best[w][lane] < 6) found = run_test(lane, best[w][lane], hq, dtq, wt);
            if (found) record_hit<VF>(d, q, wt);
            const unsigned hb = __ballot_sync(full, found);
            if (lane == 0) {
                hmask[base / 32] = hb;
                hcnt[base / 32] = (uint32_t)__popc(hb);
            }
            __syncwarp();
            continue;
        }
        // EE: the few candidates whose edges are not apart throughout their
        // times' advances go on to the tests, 32 of them at a time.
        bool is_near = false;
        if (valid && times) {
            const float h = d.cloth[cloth_of[w][lane]].h, dt = d.cloth[cloth_of[w][lane]].dt;
            float T = 0.f, lo = 3.4e38f, hi = -3.4e38f;
            for (unsigned m = times; m; m &= m - 1u) {
                T += tq[w][__ffs(m) - 1][lane] * dt;
                lo = fminf(lo, T);
                hi = fmaxf(hi, T);
            }
            float3 x1, x2, x3, x4, v1, v2, v3, v4;
            corners(lane, x1, x2, x3, x4, v1, v2, v3, v4);
            is_near = !(T == T && ee_apart(x1, x2, x3, x4, v1, v2, v3, v4, lo, hi, h));  // (NaN times: T is NaN)
        }
        const unsigned nb = __ballot_sync(full, is_near);
        if (is_near) {
            const int at = nnear + __popc(nb & ((1u << lane) - 1u));
            near_q[w][at] = q;
            near_n[w][at] = (uint8_t)__popc(times);
            int k = 0;
            for (unsigned m = times; m; m &= m - 1u) near_t[w][k++][at] = tq[w][__ffs(m) - 1][lane];
        }
        nnear += __popc(nb);
        if (lane == 0) hmask[base / 32] = hcnt[base / 32] = 0u;
        __syncwarp();
        if (nnear >= 32) {
            nnear -= 32;
            const int at = nnear + lane;
            test_near(d, near_q[w][at], near_n[w][at], &near_t[w][0][at]);
            __syncwarp();
        }
    }
    if (!VF && lane < nnear)
        test_near(d, near_q[w][lane], near_n[w][lane], &near_t[w][0][lane]);
}

// One kind, or both in one launch (the first half of the blocks takes the EE
// candidates): the two wait for nothing of each other, and in a small step
// each leaves most of the chip idle; in a large one the two codes evict each
// other from the instruction cache.  Us per step, one by one / both, folded
// cloths of 16, 32, 64, 101, 140 and 192 squared: 183, 238, 311, 455, 853, 955 /
// 176, 230, 306, 449, 850, 971; 24 cloths up to 128 squared 1255 / 1271.
// At most 64 registers, for 4 resident blocks per SM instead of 3: EE 134 us
// against 150.
template <bool VF>
__global__ void __launch_bounds__(kCcdWarps * 32, 4) k_ccd_warp(const __grid_constant__ DevPtrs d,
                                                                const uint32_t *__restrict__ ncand) {
    __shared__ CcdShared<VF> sh;
    ccd_run<VF>(d, ncand, sh, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kCcdWarps * 32, 4) k_ccd_both(const __grid_constant__ DevPtrs d,
                                                                const uint32_t *__restrict__ ncv,
                                                                const uint32_t *__restrict__ nce) {
    __shared__ union {
        CcdShared<true> vf;
        CcdShared<false> ee;
    } sh;
    const uint32_t half = gridDim.x / 2;
    if (blockIdx.x < half) ccd_run<false>(d, nce, sh.ee, blockIdx.x, half);
    else ccd_run<true>(d, ncv, sh.vf, blockIdx.x - half, half);
}

// The discrete tests (CudaPrimitiveTests::DCDTriangleTests,
// Collision/CudaPrimitiveTests.cu:21-94): one TestVF / TestEE of every
// candidate at x_prev, as HandleCollisionsDiscrete passes the previous
// positions (Physics/CudaDeformableBody.cpp:428).  Hits are recorded as the
// continuous kernel records them (per group of 32 candidates: the hit bits;
// k_ccd_emit places them), with t as the tests leave it.
template <bool VF>
__global__ void __launch_bounds__(kThreads) k_dcd_warp(DevPtrs d, const uint32_t *__restrict__ ncand) {
    const uint32_t n = (uint32_t)min((uint64_t)*ncand, d.cand_cap);
    const int4 *list = VF ? d.cand : d.cand_e;
    uint32_t *hmask = d.hitg_mask[VF ? 0 : 1], *hcnt = d.hitg_cnt[VF ? 0 : 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) d.hitg_n[VF ? 0 : 1] = (n + 31) / 32;
    const int lane = threadIdx.x & 31;
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp0 * 32u; base < n; base += nwarps * 32u) {
        const uint32_t q = base + lane;
        bool found = false;
        if (q < n) {
            const int4 ids = list[q];
            const float h = d.cloth[d.vcloth[ids.x]].h;
            Wts wt;
            wt.t = -1.f;  // the candidate's initial time (Physics/Structs.h:122-124)
            found = VF ? test_vf(xyz(d.xp[ids.x]), xyz(d.xp[ids.y]), xyz(d.xp[ids.z]), xyz(d.xp[ids.w]), h, wt)
                       : test_ee(xyz(d.xp[ids.x]), xyz(d.xp[ids.y]), xyz(d.xp[ids.z]), xyz(d.xp[ids.w]), h, wt);
            if (found) {
                const uint64_t cap = VF ? d.vf_cap : d.ee_cap;
                const uint32_t slot = atomicAdd(&d.hit_n[VF ? 0 : 1], 1u);
                if (slot < cap) {
                    d.hit_q[VF ? 0 : 1][slot] = q;
                    d.hit_w[VF ? 0 : 1][slot] = make_float4(wt.w0, wt.w1, wt.w2, wt.w3);
                    if (d.hit_tn[VF ? 0 : 1])
                        d.hit_tn[VF ? 0 : 1][slot] = make_float4(wt.n.x, wt.n.y, wt.n.z, wt.t);
                } else {
                    atomicOr(d.err, VF ? ERR_VF_OVERFLOW : ERR_EE_OVERFLOW);
                }
            }
        }
        const unsigned hb = __ballot_sync(0xffffffffu, found);
        if (lane == 0) {
            hmask[base / 32] = hb;
            hcnt[base / 32] = (uint32_t)__popc(hb);
        }
    }
}

// Contacts of the candidates before candidate q <= n (n the kind's
// candidate count): its group's first contact plus the hits before it in
// the group.
template <bool VF>
__device__ __forceinline__ uint32_t hit_index(const DevPtrs &d, uint32_t q) {
    const int k = VF ? 0 : 1;
    const uint32_t g = q / 32, r = q % 32;
    if (g >= d.hitg_n[k]) return d.hitg_off[k][d.hitg_n[k]];
    return d.hitg_off[k][g] + (uint32_t)__popc(d.hitg_mask[k][g] & ((1u << r) - 1u));
}

// Stage 4 after k_ccd_warp: every hit written at its index in candidate order
// (the exclusive scan of the hit flags), ids from the candidate list.
template <bool VF>
__device__ __forceinline__ void emit_hits(const DevPtrs &d, uint32_t first, uint32_t stride) {
    const uint64_t cap = VF ? d.vf_cap : d.ee_cap;
    const uint32_t n = (uint32_t)min((uint64_t)d.hit_n[VF ? 0 : 1], cap);
    const int4 *list = VF ? d.cand : d.cand_e;
    for (uint32_t k = first; k < n; k += stride) {
        const uint32_t q = d.hit_q[VF ? 0 : 1][k];
        const uint32_t o = hit_index<VF>(d, q);
        if (o < cap) {
            if (VF) {
                d.vf_v[o] = list[q];
                d.vf_w[o] = d.hit_w[0][k];
                if (d.vf_n) d.vf_n[o] = d.hit_nrm[k];
                if (d.vf_tn) d.vf_tn[o] = d.hit_tn[0][k];
            } else {
                d.ee_v[o] = list[q];
                d.ee_w[o] = d.hit_w[1][k];
                if (d.ee_tn) d.ee_tn[o] = d.hit_tn[1][k];
            }
        } else {
            atomicOr(d.err, VF ? ERR_VF_OVERFLOW : ERR_EE_OVERFLOW);
        }
    }
}

// Per-cloth contact ranges (the VF and the EE contacts of one cloth are
// contiguous).
__device__ __forceinline__ void contact_range(const DevPtrs &d, int c, const uint32_t *__restrict__ ncv,
                                              const uint32_t *__restrict__ nce) {
    const ClothDev &cd = d.cloth[c];
    const uint32_t nv = (uint32_t)min((uint64_t)*ncv, d.cand_cap), ne = (uint32_t)min((uint64_t)*nce, d.cand_cap);
    const uint32_t p0 = d.pair_off[cd.t_off], p1 = d.pair_off[cd.t_off + cd.T];
    const uint32_t v0 = min(pair_cand_off<true>(d, p0, nv), nv), v1 = min(pair_cand_off<true>(d, p1, nv), nv);
    const uint32_t e0 = min(pair_cand_off<false>(d, p0, ne), ne), e1 = min(pair_cand_off<false>(d, p1, ne), ne);
    d.crange[c] = make_uint4((uint32_t)min((uint64_t)hit_index<true>(d, v0), d.vf_cap),
                             (uint32_t)min((uint64_t)hit_index<true>(d, v1), d.vf_cap),
                             (uint32_t)min((uint64_t)hit_index<false>(d, e0), d.ee_cap),
                             (uint32_t)min((uint64_t)hit_index<false>(d, e1), d.ee_cap));
}

// Both kinds' hits and the ranges in one launch: none needs another's output,
// and each takes longer to launch than to run.  The first `ranges` blocks
// take the cloths, the others every hit.
__global__ void __launch_bounds__(kThreads) k_ccd_emit(DevPtrs d, const uint32_t *__restrict__ ncv,
                                                       const uint32_t *__restrict__ nce, int ranges) {
    if ((int)blockIdx.x < ranges) {
        const int c = blockIdx.x * kThreads + threadIdx.x;
        if (c < d.C) contact_range(d, c, ncv, nce);
        return;
    }
    const uint32_t first = (blockIdx.x - ranges) * kThreads + threadIdx.x, stride = (gridDim.x - ranges) * kThreads;
    emit_hits<true>(d, first, stride);
    emit_hits<false>(d, first, stride);
}

// ---------------------------------------------------------------------------
// Static triangle colliders (lc_batch_set_collider; no counterpart in the
// reference, whose sphere is analytic).  One thread per cloth vertex walks
// its cloth's collider BVH with the vertex's swept box inflated by h + m
// (m = kColliderMargin h).  For a face with unit normal n towards the free
// side (the winding given to lc_batch_set_collider) and d0 = n . a, the
// vertex's signed heights s0 = n . x_prev - d0 and s1 = n . x - d0 (x the
// prediction) make it a contact when it ends within reach of the face's
// layer (s1 < h + m) without having started far behind it (s0 > -m), and the
// point where it crosses the plane (without a crossing, its prediction) lies
// on the triangle: barycentric coordinates >= -h / perimeter, the tolerance
// of the reference's TestVF (Collision/CudaPrimitiveTests.cu:348-406).  The
// motion is the prediction's straight line, so the test is exact.  The reach
// lets the constraint act on a vertex that the solver iterations drag
// towards the face after this test, and brings back one that ended a step
// behind it; a contact above its layer is inactive, the constraint being
// one-sided.  A contact records the face and its plane (n, d0): the
// constraint n . x >= d0 + h, onto which the vertex is projected here, in
// slot order, and again at the end of every solver iteration.  The
// kColliderSlots lowest faces are kept, ascending, so the result does not
// depend on the traversal order.
// ---------------------------------------------------------------------------
// The per-face part of the test, computed once per lc_batch_set_collider
// (the same operations in the same order as a per-test evaluation, so the
// same bits): plane (n towards the free side, d0 = n . a), corner a and the
// perimeter, the edges and their dot products.
__global__ void k_collider_faces(DevPtrs d, int ntri) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const int4 tv = d.ct[t];
    const float3 a = xyz(d.cv[tv.x]), b = xyz(d.cv[tv.y]), c = xyz(d.cv[tv.z]);
    float3 nf = normalize(cross(sub(b, a), sub(c, a)));
    if (d.cloth[tv.w].coll_cw) nf = mul(nf, -1.f);
    const float3 e1 = sub(b, a), e2 = sub(c, a), e3 = sub(c, b);
    const float d00 = dot(e1, e1), d01 = dot(e1, e2), d11 = dot(e2, e2);
    float4 *g = d.cface_geo + (size_t)5 * t;
    g[0] = f4(nf, dot(nf, a));
    g[1] = f4(a, len(e1) + len(e2) + len(e3));
    g[2] = f4(e1, d00);
    g[3] = f4(e2, d11);
    g[4] = make_float4(d01, d00 * d11 - d01 * d01, 0.f, 0.f);
}
void launch_collider_faces(const DevPtrs &d, int ntri, cudaStream_t st) {
    if (ntri) k_collider_faces<<<(ntri + kThreads - 1) / kThreads, kThreads, 0, st>>>(d, ntri);
}

__device__ bool collider_hit(float3 xp, float3 x, const float4 *__restrict__ g, float h, float m) {
    const float4 pl = g[0];
    const float3 n = xyz(pl);
    const float d0 = pl.w;
    const float s0 = dot(n, xp) - d0, s1 = dot(n, x) - d0;
    if (!(s1 < h + m) || !(s0 > -m)) return false;
    const float4 ga = g[1], g1 = g[2], g2 = g[3], g3 = g[4];
    const float3 q = (s0 > 0.f && s1 < 0.f) ? add(xp, mul(sub(x, xp), s0 / (s0 - s1))) : x;
    const float3 r = sub(q, xyz(ga));
    const float d00 = g1.w, d01 = g3.x, d11 = g2.w, d20 = dot(r, xyz(g1)), d21 = dot(r, xyz(g2));
    const float den = g3.y;
    if (!(den > 0.f)) return false;
    const float wb = (d11 * d20 - d01 * d21) / den, wc = (d00 * d21 - d01 * d20) / den;
    const float wa = 1.f - wb - wc;
    const float del = h / ga.w;
    return wa >= -del && wb >= -del && wc >= -del;
}

__global__ void k_collider_query(DevPtrs d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.Vtot; i += gridDim.x * blockDim.x) {
        const ClothDev &cd = d.cloth[d.vcloth[i]];
        int n = 0;
        int face[kColliderSlots];
        float4 pln[kColliderSlots];
        const float4 x4 = d.x[i];
        const float h = cd.h;
        if (cd.coll_root >= 0) {
            const float m = kColliderMargin * h, hm = h + m;
            const float3 xi = xyz(x4), xpi = xyz(d.xp[i]);
            const float3 lo = subc(vmin(xi, xpi), hm), hi = addc(vmax(xi, xpi), hm);
            int stack[kColliderStack];
            int top = 0;
            stack[top++] = cd.coll_root;
            while (top > 0) {
                const int node = stack[--top];
                if (!overlap(lo, hi, xyz(d.cnmin[node]), xyz(d.cnmax[node]))) continue;
                const int2 ch = d.cnchild[node];
                if (ch.x >= 0) {
                    if (top + 2 > kColliderStack) { atomicOr(d.err, ERR_STACK); break; }
                    stack[top++] = ch.y;
                    stack[top++] = ch.x;
                    continue;
                }
                const int tri = -(ch.x + 1);
                const float4 *g = d.cface_geo + (size_t)5 * tri;
                if (!collider_hit(xpi, xi, g, h, m)) continue;
                // keep the kColliderSlots lowest faces, ascending
                if (n == kColliderSlots && tri > face[n - 1]) { atomicOr(d.err, ERR_COLL_OVERFLOW); continue; }
                if (n == kColliderSlots) atomicOr(d.err, ERR_COLL_OVERFLOW);
                int k = n < kColliderSlots ? n++ : kColliderSlots - 1;
                while (k > 0 && face[k - 1] > tri) {
                    face[k] = face[k - 1];
                    pln[k] = pln[k - 1];
                    --k;
                }
                face[k] = tri;
                pln[k] = g[0];
            }
        }
        d.ccnt[i] = n;
        float3 xn = xyz(x4);
        uint32_t act = 0;
        for (int k = 0; k < n; ++k) {
            d.cface[(size_t)i * kColliderSlots + k] = face[k];
            d.cw[(size_t)i * kColliderSlots + k] = pln[k];
            const float c = dot(xyz(pln[k]), xn) - pln[k].w - h;
            if (c < 0.f) {
                xn = add(xn, mul(xyz(pln[k]), -c));
                act |= 1u << k;
            }
        }
        if (x4.w == 0.f) act = 0;                  // pinned vertices do not move
        else if (n) d.x[i] = f4(xn, x4.w);
        if (d.coll_act) d.coll_act[i] = (uint8_t)act;  // the adjoint's record of the projection
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static inline int nblk(int64_t n, int b = kThreads) { return (int)((n + b - 1) / b); }

void launch_collider(const DevPtrs &d, int grid, cudaStream_t st) {
    if (d.Vtot && d.any_collider) k_collider_query<<<grid, kThreads, 0, st>>>(d);
}
void launch_triangles(const DevPtrs &d, cudaStream_t st) {
    if (d.Ttot) k_triangles<<<nblk(d.Ttot), kThreads, 0, st>>>(d);
}
void launch_leaves_from_boxes(const DevPtrs &d, const float *bmin, const float *bmax, int T, int mode,
                              cudaStream_t st) {
    if (T) k_leaves_from_boxes<<<nblk(T), kThreads, 0, st>>>(d, bmin, bmax, T, mode);
}
// Sorts by `passes` 8-bit digits from bit shift0 up (an even number: the result
// is where the keys were).  alt: the keys start in keys_alt / payload_alt.
void launch_sort(const DevPtrs &d, const int *tile_first, int shift0, int passes, bool alt, cudaStream_t st) {
    if (!d.nstiles) return;
    unsigned long long *k0 = alt ? d.keys_alt : d.keys, *k1 = alt ? d.keys : d.keys_alt;
    uint32_t *p0 = alt ? d.payload_alt : d.payload, *p1 = alt ? d.payload : d.payload_alt;
    // One-sweep wherever the digit counts fit the status word's 30 bits; the
    // per-pass histogram and per-segment offsets block remain for the rest.
    const bool sweep = d.sstat && d.sseg && d.Ttot <= (int64_t)kStatCount && passes <= kSortPassesMax;
    if (sweep) {
        cudaMemsetAsync(d.sseg, 0, sizeof(uint32_t) * (kSortHead + (size_t)d.C * kSortPassesMax * kSortBuckets), st);
        k_sort_hist_all<<<d.nstiles, kThreads, 0, st>>>(d, k0, shift0, passes);
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = shift0 + p * kSortBits;
        if (sweep) {
            k_sort_scatter<kLookback><<<d.nstiles, kThreads, 0, st>>>(d, k0, p0, k1, p1, shift, p, tile_first);
        } else {
            k_sort_hist<<<d.nstiles, kThreads, 0, st>>>(d, k0, shift);
            k_sort_offsets<<<d.C, kSortBuckets * kOffsetsSplit, 0, st>>>(d, tile_first);
            k_sort_scatter<kOffsets><<<d.nstiles, kThreads, 0, st>>>(d, k0, p0, k1, p1, shift, p, tile_first);
        }
        std::swap(k0, k1);
        std::swap(p0, p1);
    }
}

template <int CS, int R>
static cudaError_t sort_segments(const DevPtrs &d, int halves, cudaStream_t st) {
    const size_t smem = SegmentSort<CS, R>::kSmem;
    const cudaError_t e =
        cudaFuncSetAttribute(k_sort_segment<CS, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.C * CS);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CS > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_sort_segment<CS, R>, d, halves);
}

// Sort by Morton code and its outputs (keys, perm, tri_slot, fixed-mode leaf
// boxes) from the codes in keys_alt.  max_T: the largest segment.  Measured (us,
// the launches of one step timed together) one CTA per segment / eight / the
// general passes: one segment of 1922 17 / 21 / 54, of 7938 42 / 23 / 54, of
// 15842 - / 30 / 56, of 31752 - / 42 / 59, of 64082 - / 67 / 64; 8 segments up
// to 32258 - / 41 / 58; 16 up to 6498 39 / 36 / 54; 64 up to 7938 41 / 82 / 58;
// 64 up to 31752 - / 178 / 110.  So one CTA up to 2048 keys, eight for at most
// eight segments of up to 32768, one up to 8192, and the passes beyond.
void launch_morton_sort(const DevPtrs &d, const int *tile_first, int mode, int max_T, cudaStream_t st) {
    if (!d.Ttot) return;
    const int halves = mode == LC_MORTON_K30 ? 0 : 1, shift0 = halves ? 32 : 0;
    cudaError_t e = cudaErrorNotSupported;
    if (max_T <= kSmallThreads) e = sort_segments<1, 1>(d, halves, st);
    else if (max_T <= 2 * kSmallThreads) e = sort_segments<1, 2>(d, halves, st);
    else if (d.C <= kSmallCtas) {
        if (max_T <= kSmallCtas * kSmallThreads) e = sort_segments<kSmallCtas, 1>(d, halves, st);
        else if (max_T <= 2 * kSmallCtas * kSmallThreads) e = sort_segments<kSmallCtas, 2>(d, halves, st);
        else if (max_T <= 4 * kSmallCtas * kSmallThreads) e = sort_segments<kSmallCtas, 4>(d, halves, st);
    }
    else if (max_T <= 4 * kSmallThreads) e = sort_segments<1, 4>(d, halves, st);
    else if (max_T <= 8 * kSmallThreads) e = sort_segments<1, 8>(d, halves, st);
    if (e == cudaSuccess) return;
    cudaGetLastError();
    if (halves && !d.run_small) {  // (the allocation-free entry, should the launch above fail: the whole key)
        launch_sort(d, tile_first, 0, 8, true, st);
        k_post_sort<<<nblk(d.Ttot), kThreads, 0, st>>>(d, 0);
        return;
    }
    launch_sort(d, tile_first, shift0, 4, true, st);
    k_post_sort<<<nblk(d.Ttot), kThreads, 0, st>>>(d, halves);
    if (halves) k_sort_long_runs<<<kRunBlocks, kThreads, 0, st>>>(d);
}
// The hierarchy with its boxes and records.
void launch_hierarchy(const DevPtrs &d, int max_T, cudaStream_t st) {
    if (!d.Ttot) return;
    using Any = KarrasBlock<kThreads, kThreads>;
    using Whole = KarrasBlock<1024, kSortTile>;
    const int far_blocks = std::min(nblk(d.Ttot, 2 * kThreads), 1024);
    if (!d.eq3) {  // the allocation-free entry: no range tree, the climb for all
        k_karras<kThreads, kThreads><<<nblk(d.Ttot), kThreads, Any::kSmem, st>>>(d);
        k_karras_far<<<far_blocks, kThreads, 0, st>>>(d);
        k_refit<<<nblk(d.Ttot), kThreads, 0, st>>>(d);
        return;
    }
    if (max_T <= kSortTile && cudaFuncSetAttribute(k_karras<1024, kSortTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)Whole::kSmem) == cudaSuccess) {
        k_karras<1024, kSortTile><<<d.nstiles, 1024, Whole::kSmem, st>>>(d);
    } else {
        cudaGetLastError();
        k_range_tree<<<d.nstiles, kTreeThreads, 0, st>>>(d);
        k_karras<kThreads, kThreads><<<nblk(d.Ttot), kThreads, Any::kSmem, st>>>(d);
        k_karras_far<<<far_blocks, kThreads, 0, st>>>(d);
    }
    // Cloths in which three equal codes meet: one launch where they are small, or
    // few of up to 8192 triangles.  A flagged cloth of 8192 (mostly clamped at the
    // frame's faces): its one block took 180 us, the three launches 54 and 5 more
    // for every other cloth, eight blocks 58 and none.
    if (max_T <= kSortTile || (max_T <= 4 * kSortTile && d.C <= kSmallCtas)) {
        const int per = max_T <= kSortTile ? 1 : 8;
        k_refit_block<<<per * d.C, kRefitBlock, 0, st>>>(d, per);
        return;
    }
    // the upper pass: a grid-stride loop over the arrivals left, sized to be
    // resident at once
    k_refit_local<<<nblk(d.Ttot), kThreads, 0, st>>>(d);
    k_refit_upper<<<std::min(nblk(2 * (int64_t)std::max(d.Itot, 1)), 1024), kThreads, 0, st>>>(d);
    k_pack_nodes<<<nblk(d.Ttot), kThreads, 0, st>>>(d);
}
void launch_traverse(const DevPtrs &d, int block, cudaStream_t st) {
    if (!d.Ttot) return;
    if (d.wnode) {
        k_traverse_leaf<<<nblk(d.Ttot, block), block, 0, st>>>(d);
    } else {
        k_traverse<<<nblk(d.Ttot, block), block, 0, st>>>(d);
    }
}
void launch_pair_compact(const DevPtrs &d, cudaStream_t st) {
    if (!d.Ttot) return;
    const int per = d.Ttot > kCompactManyLeaves ? 32 : 4;
    k_pair_compact<<<nblk(((int64_t)d.Ttot + per - 1) / per * 32), kThreads, 0, st>>>(d, per);
}
void launch_narrow(const DevPtrs &d, const uint32_t *npairs, const uint32_t *ncv, const uint32_t *nce, int grid,
                   int stage, cudaStream_t st) {
    if (stage == 0) k_narrow_filter<<<grid, kThreads, 0, st>>>(d, npairs, 1);
    else if (stage == 6) k_narrow_filter<<<grid, kThreads, 0, st>>>(d, npairs, 0);  // no feature AABB cull
    else if (stage == 7) {
        k_dcd_warp<true><<<grid, kThreads, 0, st>>>(d, ncv);
    } else if (stage == 8) {
        k_dcd_warp<false><<<grid, kThreads, 0, st>>>(d, nce);
    }
    else if (stage == 1) k_narrow_expand<<<grid, kThreads, 0, st>>>(d, npairs);
    else if (stage == 2) {
        k_ccd_warp<true><<<grid, kCcdWarps * 32, 0, st>>>(d, ncv);
    } else if (stage == 9) {
        k_ccd_both<<<2 * grid, kCcdWarps * 32, 0, st>>>(d, ncv, nce);
    } else if (stage == 5) {
        k_ccd_warp<false><<<grid, kCcdWarps * 32, 0, st>>>(d, nce);
    } else if (stage == 3) {
        k_ccd_emit<<<grid, kThreads, 0, st>>>(d, ncv, nce, 0);
    } else {
        const int ranges = nblk(d.C);
        k_ccd_emit<<<grid + ranges, kThreads, 0, st>>>(d, ncv, nce, ranges);
    }
}

}  // namespace lc
