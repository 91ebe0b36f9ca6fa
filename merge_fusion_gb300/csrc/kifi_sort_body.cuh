// kifi_sort_body.cuh -- the device bodies of the onesweep radix sort
// (kifi_sort.cu): digit histograms, the pass set-up and one digit pass.
// Their shared memory is passed in, so that a kernel running several stages
// (the batched fusion queue, kifi_integrate.cu) can overlay it.
#pragma once

#include "kifi_api_util.h"

namespace kifi {
namespace sort_detail {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kKeysPerThread = 8;
constexpr int kTile = kThreads * kKeysPerThread;  // 2048
constexpr int kRadix = 256;
constexpr unsigned long long kSpinLimit = 1ull << 22;
constexpr int kLookAhead = 8;  // predecessor look-back words fetched per round
constexpr unsigned int kGroup = 16;  // tiles whose sum the look-back takes at once
__host__ __device__ constexpr size_t lookback_rows(size_t max_tiles) { return max_tiles + max_tiles / kGroup + 1; }
// Every scratch's sizes: tiles of up to max_n keys, and the look-back words of `digits` counters (passes x radix).
constexpr size_t tiles_of(size_t max_n) { return (max_n + kTile - 1) / kTile + 1; }
constexpr size_t lookback_bytes(size_t max_tiles, size_t digits) {
    return digits * lookback_rows(max_tiles) * sizeof(unsigned long long);
}

constexpr unsigned long long kFlagAggregate = 1ull << 30;
constexpr unsigned long long kFlagInclusive = 2ull << 30;
constexpr unsigned long long kCountMask = (1ull << 30) - 1;

__device__ __forceinline__ void sort_prepare_body(const SortScratch& s, int passes) {
    for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) s.hist[i] = 0u;
    if (threadIdx.x < passes) s.tile_counter[threadIdx.x] = s.first_tile;
    if (threadIdx.x == 0) *s.epoch += 1ull;
}

// all `passes` digit histograms in one read of the keys
struct SortHistSmem {
    unsigned int h[kSortMaxPasses][kRadix];
};
template <typename K>
__device__ __forceinline__ void sort_histogram_body(const K* __restrict__ keys, const unsigned int* __restrict__ n_ptr,
                                                    const SortScratch& s, int passes, unsigned int blk,
                                                    unsigned int nblk, SortHistSmem& sm) {
    auto& h = sm.h;
    for (int i = threadIdx.x; i < passes * kRadix; i += kThreads) (&h[0][0])[i] = 0u;
    __syncthreads();
    const size_t n = min((size_t)*n_ptr, s.max_n);
    for (size_t i = (size_t)blk * kThreads + threadIdx.x; i < n;
         i += (size_t)nblk * kThreads) {
        const K k = keys[i];
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(unsigned int)(k >> (8 * p)) & 0xffu], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kRadix; i += kThreads) {
        unsigned int c = (&h[0][0])[i];
        if (c) atomicAdd(&s.hist[i], c);
    }
}

__device__ __forceinline__ unsigned int lanemask_lt() {
    unsigned int m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Reads of what the kernels before wrote go to L2: a chained kernel's life
// begins before those writes, so they are no read-only data to it and L1 may
// hold older lines.
__device__ __forceinline__ uint32_t ld_l2(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ uint64_t ld_l2(const uint64_t* p) { return __ldcg((const unsigned long long*)p); }
__device__ __forceinline__ unsigned long long ld_volatile_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_volatile_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One digit pass of kBits bits (radix R = 2^kBits, R / kThreads digits per
// thread in the scans and the look-back: one for 8-bit digits, four for the
// frame keys' 10-bit digits).
template <int kBits, int kT = kThreads>
struct SortPassSmem {
    uint16_t warp_hist[kT / 32][(1 << kBits) + 2];  // last columns: out-of-range keys
    unsigned int digit_base[1 << kBits];
    unsigned int pass_offset[1 << kBits];
    unsigned int wsum[kT / 32];
    unsigned int tile_id;
};
template <bool kWithValues, typename K, int kBits, int kT = kThreads>
__device__ __forceinline__ void sort_pass_body(const K* keys_in, K* __restrict__ keys_out,
                                               const uint32_t* vals_in, uint32_t* __restrict__ vals_out,
                                               const unsigned int* n_ptr, const SortScratch& s,
                                               int pass, unsigned int blk, unsigned int nblk,
                                               SortPassSmem<kBits, kT>& sm) {
    constexpr int R = 1 << kBits;
    constexpr int D = R > kT ? R / kT : 1;         // digits per thread (of the first R threads)
    constexpr int kLA = D == 1 ? kLookAhead : kLookAhead / 2;  // look-back words per digit and round
    constexpr int kWarps = kT / 32, kTile = kT * kKeysPerThread;
    static_assert(D * kT == R || kT > R, "whole digits per thread");
    const bool digits = kT <= R || threadIdx.x < R;  // this thread has digits
    auto& warp_hist = sm.warp_hist;
    auto& digit_base = sm.digit_base;
    auto& pass_offset = sm.pass_offset;
    auto& wsum = sm.wsum;
    auto& tile_id = sm.tile_id;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Tiles come from a counter, so that every tile a CTA waits for has been
    // taken by a CTA that runs, in whatever order the CTAs start (their order
    // is not promised, and beside other work not all are resident).
    auto take_tile = [&] {
        if (threadIdx.x == 0) tile_id = atomicAdd(&s.tile_counter[pass], 1u);
        for (int i = threadIdx.x; i < kWarps * (R + 2) / 2; i += kT)
            reinterpret_cast<unsigned int*>(&warp_hist[0][0])[i] = 0u;
    };
    // Grids are sized before the key count exists.  CTAs beyond the tile count
    // leave before the counter, at which they would queue; of a frame's alone
    // (kT > kThreads: four CTAs per SM) the first quarter take a ticket while the
    // count is read.  Ten 320x240 frames at 8 mm, 640x480 at 4 mm and 512x424 with
    // 64-bit keys, us: tiles by block index 512, 2732, 2214; every ticket behind
    // the count 520, 2733, 2272; the first quarter ahead of it 506, 2707, 2244; the
    // first half 509, 2712, 2310.
    const bool early = kT > kThreads && blk < nblk / 4;
    if (early) take_tile();
    const unsigned int n = (unsigned int)min((size_t)*n_ptr, s.max_n);
    const unsigned int n_tiles = (n + kTile - 1) / kTile;
    if (!early) {
        if (blk >= n_tiles) return;
        take_tile();
    }
    const int shift = pass * kBits;
    const unsigned long long gen = (*s.epoch & 0xffffffffull) << 32;
    unsigned long long* lb = s.lookback + (size_t)pass * lookback_rows(s.max_tiles) * R;  // tiles, then groups
    unsigned int c[D];
#pragma unroll
    for (int q = 0; q < D; ++q) c[q] = digits ? __ldcg(s.hist + pass * R + threadIdx.x * D + q) : 0u;
    __syncthreads();
    unsigned int tile = tile_id;
    for (bool first = true; tile < n_tiles; first = false) {
        const unsigned int base = tile * kTile + warp * (32 * kKeysPerThread);
        K k[kKeysPerThread];
        uint32_t v[kKeysPerThread];
        unsigned int rank[kKeysPerThread];
        int dig[kKeysPerThread];
#pragma unroll
        for (int j = 0; j < kKeysPerThread; ++j) {
            unsigned int i = base + j * 32 + lane;
            bool ok = i < n;
            k[j] = ok ? ld_l2(keys_in + i) : (K)0;
            if (kWithValues) v[j] = ok ? __ldcg(vals_in + i) : 0u;
        }
        if (first) {
            // exclusive scan of this pass's global digit histogram: thread t
            // holds digits t*D .. t*D + D - 1
            unsigned int sum = 0;
#pragma unroll
            for (int q = 0; q < D; ++q) sum += c[q];
            unsigned int x = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) wsum[warp] = x;
            __syncthreads();
            unsigned int run = x - sum;
            for (int w = 0; w < warp; ++w) run += wsum[w];
#pragma unroll
            for (int q = 0; q < D; ++q) {
                if (digits) pass_offset[threadIdx.x * D + q] = run;  // read behind later barriers
                run += c[q];
            }
        }
        // stable warp-local ranks: lanes with equal digits, in (j, lane) order
        unsigned int peers[kKeysPerThread];
#pragma unroll
        for (int j = 0; j < kKeysPerThread; ++j) {
            dig[j] = base + j * 32 + lane < n ? (int)((unsigned int)(k[j] >> shift) & (unsigned int)(R - 1)) : R;
            peers[j] = __match_any_sync(0xffffffffu, dig[j]);
        }
#pragma unroll
        for (int j = 0; j < kKeysPerThread; ++j) {
            unsigned int before = warp_hist[warp][dig[j]];
            rank[j] = before + __popc(peers[j] & lanemask_lt());
            __syncwarp();
            if (lane == __ffs(peers[j]) - 1) warp_hist[warp][dig[j]] = (uint16_t)(before + __popc(peers[j]));
            __syncwarp();
        }
        __syncthreads();
        // per digit d = threadIdx.x + q * kT: counts across warps ->
        // exclusive prefix over warps
        unsigned int tile_count[D];
#pragma unroll
        for (int q = 0; q < D; ++q) {
            const int d = threadIdx.x + q * kT;
            unsigned int tc = 0;
            for (int w = 0; digits && w < kWarps; ++w) {
                const unsigned int c = warp_hist[w][d];
                warp_hist[w][d] = (uint16_t)tc;
                tc += c;
            }
            tile_count[q] = tc;
        }
        // Decoupled look-back for the thread's digits, in two levels, as a walk
        // over all predecessors costs a memory latency per kLA of them (13 of
        // 20 us at 250 tiles): a tile sums up its predecessors within its
        // group of kGroup, whose last tile publishes the group's sum, and walks
        // the groups before.
        unsigned int excl[D];
#pragma unroll
        for (int q = 0; q < D; ++q) excl[q] = 0;
        if (digits) {
#pragma unroll
            for (int q = 0; q < D; ++q)
                st_volatile_u64(lb + (size_t)tile * R + threadIdx.x + q * kT, gen | kFlagAggregate | tile_count[q]);
            const unsigned int group = tile / kGroup;
            unsigned long long spins = 0;
            // words first - i, i in [0, count): waits for each (independent loads, kLA at a time) and adds
            // them to excl; with `incl` up to the first inclusive one
            auto look_back = [&](const unsigned long long* words, int first, int count, bool incl) {
                int t[D];  // words left
                unsigned int pending = 0;
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    t[q] = count;
                    if (count > 0) pending |= 1u << q;
                }
                while (pending) {
                    unsigned long long w[D][kLA];
#pragma unroll
                    for (int q = 0; q < D; ++q) {
                        const unsigned long long* at =
                            words + (size_t)(first - (count - t[q])) * R + threadIdx.x + q * kT;
#pragma unroll
                        for (int i = 0; i < kLA; ++i)
                            w[q][i] = ((pending >> q) & 1u) && i < t[q] ? ld_volatile_u64(at - (size_t)i * R) : 0ull;
                    }
                    // consume each digit's words in order, up to the first inclusive
                    // one or the first one not yet published
                    bool stalled_any = false;
#pragma unroll
                    for (int q = 0; q < D; ++q) {
                        if (!((pending >> q) & 1u)) continue;
                        int used = 0;
                        bool done = false, stalled = false;
#pragma unroll
                        for (int i = 0; i < kLA; ++i) {
                            if (done || stalled || i >= t[q]) continue;
                            const unsigned long long x = w[q][i];
                            if ((x & 0xffffffff00000000ull) != gen || (x & (3ull << 30)) == 0) {
                                stalled = true;
                                continue;
                            }
                            excl[q] += (unsigned int)(x & kCountMask);
                            ++used;
                            done = incl && (x & kFlagInclusive) != 0;
                        }
                        t[q] -= used;
                        if (done || t[q] == 0) pending &= ~(1u << q);
                        else if (stalled) stalled_any = true;
                    }
                    if (stalled_any && ++spins > s.spin_limit) {
                        atomicOr(s.status, KIFI_DEV_ERR_TIMEOUT);
                        break;
                    }
                }
            };
            unsigned long long* groups = lb + (size_t)s.max_tiles * R;
            look_back(lb, (int)tile - 1, (int)(tile % kGroup), false);
            const bool last = tile % kGroup == kGroup - 1;
#pragma unroll
            for (int q = 0; q < D; ++q) {
                if (last && group)
                    st_volatile_u64(groups + (size_t)group * R + threadIdx.x + q * kT,
                                    gen | kFlagAggregate | ((excl[q] + tile_count[q]) & kCountMask));
            }
            look_back(groups, (int)group - 1, (int)group, true);
#pragma unroll
            for (int q = 0; q < D; ++q) {
                const int d = threadIdx.x + q * kT;
                if (last)
                    st_volatile_u64(groups + (size_t)group * R + d,
                                    gen | kFlagInclusive | ((excl[q] + tile_count[q]) & kCountMask));
                digit_base[d] = pass_offset[d] + excl[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kKeysPerThread; ++j) {
            if (dig[j] == R) continue;
            unsigned int pos = digit_base[dig[j]] + warp_hist[warp][dig[j]] + rank[j];
            if (pos >= n) {  // only reachable after a timed-out look-back
                atomicOr(s.status, KIFI_DEV_ERR_TIMEOUT);
                continue;
            }
            keys_out[pos] = k[j];
            if (kWithValues) vals_out[pos] = v[j];
        }
        if (n_tiles <= nblk) break;  // a CTA per tile: this was its only one
        __syncthreads();
        take_tile();
        __syncthreads();
        tile = tile_id;
    }
}

}  // namespace sort_detail
}  // namespace kifi
