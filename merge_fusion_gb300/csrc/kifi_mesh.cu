// kifi_mesh.cu -- sparse marching cubes over the sorted voxel keys on
// sm_103a: kifi::Mesher::Mesh (KinectFission/kifi/Mesher.cpp:14-45) and
// Mesher::Generate<bool> (:85-229).
//
// The reference walks the sorted volume backwards (voxels n-2 .. 0) with
// three neighbour pointers (+y, +z, +yz) that start at n-2 and only move down.
// After the walk for voxel i each pointer sits at
//     min(n-2, upper_bound(keys, key_i + delta) - 1),
// a closed form that depends on voxel i alone: the voxel at key_i + delta when
// it is resident and not the last one, else a voxel of another key; and the
// pointer plus one is the voxel at key_i + delta + 1 exactly when that is
// resident.  So what a cube reads is decided by which keys are resident, and
// 32 voxels are handled at once: a word is a run of 32 consecutive keys (key >>
// 5; the bits per axis are at least 10, so +y and +z move by whole words) of
// which at least one is resident, with a bit per key in a few masks.  Sorted
// keys give sorted words, and there are 10 to 20 times fewer of them.
//
//  k_word_count     counts the words that start in each of kVoxelRuns runs of voxels.
//  k_word_build     writes the words: first voxel, masks (resident, weight != 0,
//                   weight > 0, Distance() < 0, operands in the sign rule's
//                   range), and the first word of every (y, z) key row.
//  k_word_classify  a word per thread: finds the +y, +z and +yz words through
//                   the row table, and from the masks which +x/+y/+z edges
//                   carry a vertex (Mesher.cpp:140-168) and which cubes have
//                   triangles (:172-226), 32 at a time.  Lists the voxels with
//                   output, and totals vertices and indices per run of words.
//  k_mesh_emit      over the listed voxels: writes the vertices (by the voxel's
//                   lane) and the triangle indices (spread over the warp's lanes).
//
// (14.6 M voxels of a 640 x 480 room scan at 4 mm in 1.36 M words, 4.6 M
// vertices and 21 M indices: a mesh call 440 us, of it count and build 100,
// classification 107, emission 139.  A thread per voxel that searched among
// staged keys and a second emission for the stop rule: 728.)
//
// Output order equals the reference's:
//  * Mesh(verts): vertices in generation order -- voxels descending, axes
//    x, y, z -- so voxel i's vertices start after those of all voxels j > i.
//  * Mesh(verts, indices): vertices sorted by id 3*key+axis (Mesher.cpp:25-26),
//    which is ascending voxel order; triangles in generation order (voxels
//    descending, table order), each index mapped to its vertex's rank
//    (:28-44).  That mapping walk stops at the first index id that has no
//    vertex; every index id at or above it keeps its raw id.  The smallest
//    such id is found by the classification, so one emission writes the
//    indices as they end up.
#include "kifi_internal.h"
#include "mc_table.cuh"

namespace kifi {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float vdist(float2 v) { return fdiv(v.x, v.y); }  // Voxel::Distance

// exclusive scan of one 64-bit value per thread over a CTA of kT threads;
// the CTA's total to *total
template <int kT, bool kTrailingSync = true>
__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long x,
                                                                   unsigned long long* total) {
    __shared__ unsigned long long warp_sums[kT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    unsigned long long before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kT / 32; ++w) {
        if (w < warp) before += warp_sums[w];
        all += warp_sums[w];
    }
    if (kTrailingSync) __syncthreads();  // warp_sums may be rewritten next
    *total = all;
    return before + inc - x;
}

// Mesher.cpp:140-168's test Distance(self) * Distance(neighbour) <= 0
// without the divisions where its outcome is certain: for 2^-30 <= |x|, |w|
// <= 2^30 (both voxels) each quotient x / w is a float of magnitude in
// [2^-60, 2^60], so their product is a normal non-zero float (magnitude in
// [2^-120, 2^120]) whose sign is the product of the four operand signs; it
// is <= 0 exactly when the two quotients differ in sign.  Zeros, NaNs,
// infinities and the rest of the range take the reference's divisions.
__device__ __forceinline__ bool in_sign_range(float2 v) {
    const float ax = fabsf(v.x), aw = fabsf(v.y);
    return ax >= 0x1p-30f && ax <= 0x1p30f && aw >= 0x1p-30f && aw <= 0x1p30f;
}
// Voxel::Distance(v) < 0 without the division where its sign is certain:
// for 2^-100 <= |x| and 2^-100 <= |w| <= 2^24 the quotient x / w is a
// normal non-zero float (|x / w| >= 2^-124), so it is negative exactly when
// x and w differ in sign.  Zeros, NaNs, infinities and the rest of the
// range take the reference's division.
__device__ __forceinline__ bool dist_negative(float2 v) {
    const float ax = fabsf(v.x), aw = fabsf(v.y);
    if (ax >= 0x1p-100f && aw >= 0x1p-100f && aw <= 0x1p24f) return (v.x < 0.0f) != (v.y < 0.0f);
    return vdist(v) < 0.0f;
}

// edge e of the cube -> (corner, axis), from localToGlobal (Mesher.cpp:206-218):
// corners {4, 0, 0, 1, 6, 2, 2, 3, 5, 4, 0, 1} (4 bits each) and axes
// {0, 2, 0, 2, 0, 2, 0, 2, 1, 1, 1, 1} (2 bits each), decoded in registers
constexpr unsigned long long kEdgeCorners = 0x104532261004ull;
constexpr unsigned int kEdgeAxes = 0x558888u;
__device__ __forceinline__ int edge_corner(int e) { return (int)((kEdgeCorners >> (4 * e)) & 15u); }
__device__ __forceinline__ int edge_axis(int e) { return (int)((kEdgeAxes >> (2 * e)) & 3u); }


// Distance(a) * Distance(b) <= 0 with the reference's divisions
__device__ __noinline__ bool cross_exact(const float2* vals, unsigned int a, unsigned int b) {
    return fmul(vdist(vals[a]), vdist(vals[b])) <= 0.0f;
}

// Voxels, and then words, are cut into contiguous runs, one per CTA (2048
// voxels or more to a run of either).  Of voxels, the runs' counts are summed up by every
// CTA of the next kernel for itself; of words, the last CTA to finish turns the
// runs' totals into offsets.  Up to 4 and 3 rounds of resident CTAs: runs differ
// in what they hold, and in one round the longest sets the time (at the size
// above, build 98 us in one round, 82 in four; classification 130 and 107): 16 and
// 24 runs for each of the GPU's 152 SMs.
constexpr unsigned int kVoxelRuns = 2432, kWordRuns = 3648;
constexpr int kClassThreads = 128;
constexpr unsigned int kNoWord = 0xffffffffu;
constexpr unsigned int kBuildGroups = 64, kBuildTile = 32 * kBuildGroups;  // voxels taken at a time
__device__ __forceinline__ unsigned int run_length(unsigned int n, unsigned int runs, unsigned int whole) {
    return ((n + runs - 1) / runs + whole - 1u) / whole * whole;
}

// words that start in each run of voxels; and the row table cleared, for which
// there are more CTAs than runs where the volume is small (a table is 4 MB at 10
// bits per axis and 268 MB at 13, which one CTA took 35 and 4000 us to clear: a mesh
// of 30 voxels at 1024 and 8192 voxels per axis 115 -> 54, 4107 -> 93 us)
template <typename K>
__global__ void __launch_bounds__(kThreads) k_word_count(const K* __restrict__ keys,
                                                         const unsigned int* __restrict__ n_dev,
                                                         unsigned int* __restrict__ run_words, unsigned int runs,
                                                         uint4* __restrict__ rows, unsigned int row_vecs,
                                                         MeshCounts* __restrict__ mc) {
    const unsigned int n = *n_dev;
    for (unsigned int r = blockIdx.x * kThreads + threadIdx.x; r < row_vecs; r += gridDim.x * kThreads)
        rows[r] = make_uint4(kNoWord, kNoWord, kNoWord, kNoWord);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        mc->missing_min = ~0ull;
        mc->runs_done = 0u;
    }
    if (blockIdx.x >= runs) return;
    const unsigned int len = run_length(n, runs, kBuildTile);
    const unsigned int lo = min(blockIdx.x * len, n), hi = min(lo + len, n);
    const unsigned int lane = threadIdx.x & 31u;
    unsigned int cnt = 0;
#pragma unroll 4
    for (unsigned int i0 = lo; i0 < hi; i0 += 4 * kThreads) {
        const unsigned int i = i0 + 4 * threadIdx.x;
        K k[4] = {};
        if (i < hi) {  // (reads up to 3 keys past the run: the buffers are padded)
            const uint4* p = reinterpret_cast<const uint4*>(keys + i);
#pragma unroll
            for (int q = 0; q < (int)sizeof(K) / 4; ++q) reinterpret_cast<uint4*>(k)[q] = __ldg(p + q);
        }
        K before = __shfl_up_sync(0xffffffffu, k[3], 1);
        if (lane == 0 && i < hi && i > 0) before = keys[i - 1];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const K b = q ? k[q - 1] : before;
            if (i + q < hi && (i + q == 0 || (k[q] ^ b) >> 5)) ++cnt;
        }
    }
    __shared__ unsigned int s_cnt[kThreads / 32];
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) s_cnt[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int all = 0;
        for (int w = 0; w < kThreads / 32; ++w) all += s_cnt[w];
        run_words[blockIdx.x] = all;
    }
}

// Tiles of 2048 voxels (and the 32 after them, where the last word may end),
// 4 consecutive voxels per thread and load: bits for "a word starts", "keys
// leave a gap" and the voxel's state, in the order of position, 32 to a group;
// then a thread per word moves its stretch of those to the keys' bits, one
// shift per gap-free run of keys.  Reads 12 B
// per voxel; bound by instructions (100 per 32 voxels) more than by memory: 82
// us at the size above, of which the reads take 26.
template <typename K>
__global__ void __launch_bounds__(kThreads, 4) k_word_build(const K* __restrict__ keys, int kb,
                                                            const float2* __restrict__ vals,
                                                            const unsigned int* __restrict__ n_dev,
                                                            const unsigned int* __restrict__ run_words,
                                                            unsigned int* __restrict__ rows, MeshWords words,
                                                            unsigned int words_cap, MeshCounts* __restrict__ mc) {
    constexpr unsigned int kWarps = kThreads / 32, kSteps = kBuildTile / (4 * kThreads);  // 128 voxels per warp step
    __shared__ __align__(16) K s_key[kBuildTile + 32];
    __shared__ unsigned short s_list[kBuildTile + 1];  // positions where words start, then the last one's end
    __shared__ unsigned int s_gap[kBuildGroups + 2], s_neg[kBuildGroups + 2];
    __shared__ unsigned int s_e[kBuildGroups + 2], s_p[kBuildGroups + 2], s_r[kBuildGroups + 2];
    __shared__ unsigned int s_cnt[kWarps];
    __shared__ K s_before;
    const unsigned int n = *n_dev;
    const Codec<K> cd(kb);
    const unsigned int len = run_length(n, gridDim.x, kBuildTile);
    const unsigned int lo = min(blockIdx.x * len, n), hi = min(lo + len, n);
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // words before this run, and all of them
    unsigned int base;
    {
        unsigned int before = 0, all = 0;
        for (unsigned int c = threadIdx.x; c < gridDim.x; c += kThreads) {
            const unsigned int w = run_words[c];
            all += w;
            if (c < blockIdx.x) before += w;
        }
        unsigned long long total;
        block_exclusive_scan<kThreads>((unsigned long long)all << 32 | before, &total);
        base = (unsigned int)total;
        const unsigned int n_words = (unsigned int)(total >> 32);
        const bool fit = n_words <= words_cap;  // else none is written (every CTA alike), and the emission says so
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *words.count = fit ? n_words : 0u;
            mc->n_words = n_words;
        }
        if (!fit) return;
    }
    K* wkey = (K*)words.key;
    // four bits per lane, eight lanes to a group's 32: to every lane of the group
    auto join = [&](unsigned int nibble) {
        unsigned int m = nibble << (4u * (lane & 7u));
        m |= __shfl_xor_sync(0xffffffffu, m, 1);
        m |= __shfl_xor_sync(0xffffffffu, m, 2);
        m |= __shfl_xor_sync(0xffffffffu, m, 4);
        return m;
    };
    const unsigned int p0 = warp * (kSteps * 128u) + 4u * lane;  // this thread's first position in a tile
    // a tile's loads, issued while the tile before is turned into words
    K key[kSteps][4], carry = 0, tail_key = 0, tail_prev = 0;
    float2 v[kSteps][4], tail_val = make_float2(0.0f, 0.0f);
    auto load = [&](unsigned int t0) {
#pragma unroll
        for (int u = 0; u < (int)kSteps; ++u) {
            const unsigned int i = t0 + p0 + 128u * u;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                key[u][q] = 0;
                v[u][q] = make_float2(0.0f, 0.0f);
            }
            if (i < n) {  // (reads up to 3 voxels past the last: the buffers are padded)
                const uint4* kp = reinterpret_cast<const uint4*>(keys + i);
#pragma unroll
                for (int q = 0; q < (int)sizeof(K) / 4; ++q) reinterpret_cast<uint4*>(key[u])[q] = __ldg(kp + q);
                const float4* vp = reinterpret_cast<const float4*>(vals + i);
#pragma unroll
                for (int q = 0; q < 2; ++q) reinterpret_cast<float4*>(v[u])[q] = __ldg(vp + q);
            }
        }
        carry = 0;  // the key before the warp's first
        const unsigned int i0 = t0 + warp * (kSteps * 128u);
        if (lane == 0 && i0 > 0 && i0 < n) carry = keys[i0 - 1];
        if (warp == 0) {  // the group after the tile, a voxel per lane
            const unsigned int i = t0 + (min(kBuildTile, hi - t0) + 31u) / 32u * 32u + lane;
            tail_key = tail_prev = 0;
            tail_val = make_float2(0.0f, 0.0f);
            if (i < n) {
                tail_key = keys[i];
                tail_prev = keys[i - 1];
                tail_val = vals[i];
            }
        }
    };
    if (lo < hi) load(lo);
    for (unsigned int t0 = lo; t0 < hi; t0 += kBuildTile) {
        const unsigned int t1 = min(t0 + kBuildTile, hi);
        const unsigned int ng = (t1 - t0 + 31u) / 32u;  // the tile's groups; group ng is the one after
        if (threadIdx.x == 0) s_before = carry;
        unsigned int starts[kSteps], gmask[kSteps], words_here = 0;
#pragma unroll
        for (int u = 0; u < (int)kSteps; ++u) {
            const unsigned int pos = p0 + 128u * u, i = t0 + pos;
            K prev = __shfl_up_sync(0xffffffffu, key[u][3], 1);
            if (lane == 0) prev = carry;
            carry = __shfl_sync(0xffffffffu, key[u][3], 31);
            unsigned int st = 0, gp = 0, ng_ = 0;
            bool plain = true;  // both operands in the sign rule's range and the weight positive: the usual case
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const K b = q ? key[u][q - 1] : prev;
                const unsigned int xb = __float_as_uint(v[u][q].x), wb = __float_as_uint(v[u][q].y);
                st |= (key[u][q] ^ b) >> 5 ? 1u << q : 0u;
                gp |= key[u][q] != b + 1 ? 1u << q : 0u;
                ng_ |= xb >> 31 << q;
                const bool r = (xb & 0x7fffffffu) - 0x30800000u <= 0x4e800000u - 0x30800000u &&
                               wb - 0x30800000u <= 0x4e800000u - 0x30800000u;
                plain = plain && (r || i + q >= n);
            }
            if (i == 0) st |= 1u;
            const unsigned int left = i < t1 ? min(t1 - i, 4u) : 0u;  // the tile's voxels among the four
            starts[u] = st & ((1u << left) - 1u);
            words_here += __popc(starts[u]);
            gmask[u] = join(starts[u]);
            const unsigned int g = pos >> 5;
            const bool put = (lane & 7u) == 0u && g < ng;
            const unsigned int gpm = join(gp);
            unsigned int e = ~0u, p = ~0u, r = ~0u;  // (positions past the last voxel are not read)
            if (!__all_sync(0xffffffffu, plain)) {
                unsigned int eb = 0, pb = 0, rb = 0;
                ng_ = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    eb |= v[u][q].y != 0.0f ? 1u << q : 0u;
                    pb |= v[u][q].y > 0.0f ? 1u << q : 0u;
                    rb |= in_sign_range(v[u][q]) ? 1u << q : 0u;
                    ng_ |= dist_negative(v[u][q]) ? 1u << q : 0u;
                }
                e = join(eb);
                p = join(pb);
                r = join(rb);
            }
            const unsigned int nm = join(ng_);
            if (put) {
                s_gap[g] = gpm;
                s_neg[g] = nm;
                s_e[g] = e;
                s_p[g] = p;
                s_r[g] = r;
            }
            if (g < ng)
#pragma unroll
                for (int q = 0; q < (int)sizeof(K) / 4; ++q)
                    reinterpret_cast<uint4*>(s_key + pos)[q] = reinterpret_cast<const uint4*>(key[u])[q];
        }
        words_here = __reduce_add_sync(0xffffffffu, words_here);
        if (lane == 0) s_cnt[warp] = words_here;
        unsigned int tail_start = 0;  // warp 0: where words start in the group after the tile
        if (warp == 0) {
            tail_start = __ballot_sync(0xffffffffu, t0 + 32u * ng + lane >= n || (tail_key ^ tail_prev) >> 5);
            const unsigned int gp = __ballot_sync(0xffffffffu, tail_key != tail_prev + 1);
            const unsigned int e = __ballot_sync(0xffffffffu, tail_val.y != 0.0f);
            const unsigned int p = __ballot_sync(0xffffffffu, tail_val.y > 0.0f);
            const unsigned int r = __ballot_sync(0xffffffffu, in_sign_range(tail_val));
            const unsigned int nm = __ballot_sync(0xffffffffu, dist_negative(tail_val));
            s_key[32u * ng + lane] = tail_key;
            if (lane == 0) {
                s_gap[ng] = gp;
                s_neg[ng] = nm;
                s_e[ng] = e;
                s_p[ng] = p;
                s_r[ng] = r;
            }
        }
        if (t0 + kBuildTile < hi) load(t0 + kBuildTile);
        __syncthreads();
        unsigned int slot0 = 0, total = 0;  // words of the warps before; of the tile
#pragma unroll
        for (unsigned int w = 0; w < kWarps; ++w) {
            const unsigned int c = s_cnt[w];
            if (w < warp) slot0 += c;
            total += c;
        }
#pragma unroll
        for (int u = 0; u < (int)kSteps; ++u) {
            const unsigned int gc = __popc(gmask[u]);
            unsigned int slot = slot0 + __popc(gmask[u] & ((1u << (4u * (lane & 7u))) - 1u));
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const unsigned int c = __shfl_sync(0xffffffffu, gc, 8 * o);
                if (o < (int)(lane >> 3)) slot += c;
                slot0 += c;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (starts[u] >> q & 1u) s_list[slot++] = (unsigned short)(p0 + 128u * u + q);
        }
        if (threadIdx.x == 0)  // where the last word ends: the first start after the tile
            s_list[total] = (unsigned short)(t1 == n ? n - t0 : t1 - t0 + (unsigned int)__ffs(tail_start) - 1u);
        __syncthreads();
        for (unsigned int w = threadIdx.x; w < total; w += kThreads) {
            const unsigned int pos = s_list[w], cnt = s_list[w + 1] - pos;
            const unsigned int g = pos >> 5, sh = pos & 31u;
            const unsigned int ones = 0xffffffffu >> (32u - cnt);
            auto stretch = [&](const unsigned int* s) { return __funnelshift_r(s[g], s[g + 1], sh) & ones; };
            unsigned int gap = stretch(s_gap) | 1u;
            const unsigned int e = stretch(s_e), p = stretch(s_p), ng_ = stretch(s_neg), r = stretch(s_r);
            unsigned int M = 0, E = 0, P = 0, N = 0, R = 0;
            while (gap) {
                const unsigned int a = __ffs(gap) - 1u;  // the run [a, next gap) of positions
                gap &= gap - 1u;
                const unsigned int run = ones & (0xffffffffu << a) & (gap ? (gap & (0u - gap)) - 1u : 0xffffffffu);
                const unsigned int up = ((unsigned int)s_key[pos + a] & 31u) - a;
                M |= run << up;
                E |= (e & run) << up;
                P |= (p & run) << up;
                N |= (ng_ & run) << up;
                R |= (r & run) << up;
            }
            const unsigned int j = base + w;
            const K k = s_key[pos], before = pos ? s_key[pos - 1] : s_before;
            // beside the word's number, the state of its key 0, which the word before looks at
            wkey[j] = (k >> 5) << 4 | (K)((E & 1u) | (P & 1u) << 1 | (N & 1u) << 2 | (R & 1u) << 3);
            words.a[j] = make_uint4(t0 + pos, M, E, P);
            words.b[j] = make_uint2(N, R);
            if (t0 + pos == 0 || cd.row(k) != cd.row(before)) rows[cd.row(k)] = j;
        }
        base += total;
        __syncthreads();  // the staging is rewritten by the next tile
    }
}

// The position in the sorted words of word `t` (a key >> 5), where it is or
// would be.  `s` is the first word of its row, of which four words from the
// guess g on (w[], loaded by the caller beside other lookups') mostly settle it.
template <typename K>
__device__ __forceinline__ unsigned int find_word(const K* __restrict__ wkey, K t, unsigned int s, unsigned int g,
                                                  const K (&w)[4], unsigned int n_words, int kb) {
    unsigned int c = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) c += w[q] < t ? 1u : 0u;
    if (c < 4u && (c > 0u || g == s)) return g + c;
    unsigned int lo = c ? g + 4u : s, hi = c ? min(s + (1u << (kb - 5)), n_words) : g;  // a row's words: 2^(kb - 5)
    while (lo < hi) {
        const unsigned int mid = (lo + hi) >> 1;
        if ((wkey[mid] >> 4) < t) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// A row of cubes' corners: a word's masks, and those at key + 1
struct CornerRow {
    unsigned int start, M, E, P, N, R;  // the word (0 when it is not resident)
    unsigned int En, Pn, Nn, Rn;
};
template <typename K>
__device__ __forceinline__ CornerRow corner_row(const MeshWords& words, K t, unsigned int q, bool found,
                                                unsigned int n_words) {
    CornerRow c = {};
    const unsigned int q1 = found ? q + 1u : q;
    K next = 0;
    if (q1 < n_words) next = ((const K*)words.key)[q1];
    if (found) {
        const uint4 a = words.a[q];
        const uint2 b = words.b[q];
        c.start = a.x;
        c.M = a.y;
        c.E = a.z;
        c.P = a.w;
        c.N = b.x;
        c.R = b.y;
    }
    const unsigned int low = next >> 4 == t + 1 ? (unsigned int)next : 0u;  // the next word's key 0
    c.En = __funnelshift_r(c.E, low, 1u);
    c.Pn = __funnelshift_r(c.P, low >> 1, 1u);
    c.Nn = __funnelshift_r(c.N, low >> 2, 1u);
    c.Rn = __funnelshift_r(c.R, low >> 3, 1u);
    return c;
}
__device__ __forceinline__ unsigned int top_bit(unsigned int m) { return 0x80000000u >> __clz(m); }  // m != 0

// One cube's triangle edges without a vertex: the smallest of their ids into *missing.  Corner c =
// (c&1, c>>1&1, c>>2), Distance() < 0 in bit c of `neg`; its row is c >> 1, at words q[row].  All
// corners are resident, and the triangles use the edges whose corners differ in sign.  An edge
// carries a vertex when its corner is not the last voxel (the walk starts at n - 2), the
// neighbour has weight > 0 and is not the last voxel unless along +x, and the distances do not
// have the same sign.
__device__ __noinline__ void missing_edges(const MeshWords words, const float2* vals, unsigned int n, uint4 q,
                                           unsigned int bit, unsigned int neg, unsigned long long key,
                                           unsigned long long dy, unsigned long long dz,
                                           unsigned long long* missing) {
    const unsigned int qs[4] = {q.x, q.y, q.z, q.w};
    unsigned int idx[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const unsigned int b = bit + (c & 1);
        const uint4 a = words.a[qs[c >> 1] + (b >> 5)];
        idx[c] = a.x + __popc(a.y & ((1u << (b & 31u)) - 1u));
    }
    float d[8], w[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float2 v = vals[idx[c]];
        d[c] = vdist(v);
        w[c] = v.y;
    }
    unsigned long long first = ~0ull;
#pragma unroll
    for (int e = 0; e < 12; ++e) {
        const int c = edge_corner(e), axis = edge_axis(e), o = c | 1 << axis;
        if (!((neg >> c ^ neg >> o) & 1u)) continue;
        const bool has = idx[c] != n - 1u && w[o] > 0.0f && (axis == 0 || idx[o] != n - 1u) &&
                         fmul(d[c], d[o]) <= 0.0f;
        if (!has)
            first = min(first, 3ull * (key + (c & 1) + (c & 2 ? dy : 0ull) + (c & 4 ? dz : 0ull)) +
                                   (unsigned long long)axis);
    }
    if (first != ~0ull) atomicMin(missing, first);
}

// the reference's corner bit order (Mesher.cpp:191-199), from bit 0 of each corner's mask
__device__ __forceinline__ unsigned int lut_of(unsigned int c0, unsigned int c1, unsigned int c2, unsigned int c3,
                                               unsigned int c4, unsigned int c5, unsigned int c6, unsigned int c7) {
    return (c0 & 1u) << 2 | (c1 & 1u) << 3 | (c2 & 1u) << 6 | (c3 & 1u) << 7 | (c4 & 1u) << 1 | (c5 & 1u) |
           (c6 & 1u) << 5 | (c7 & 1u) << 4;
}

// A word per thread.  Of a corner looked up as "at the pointer" the last voxel
// is never found (the pointers stay at or below n - 2); of one looked up as
// "pointer plus one" it is.  Bound by latency and by
// instructions (1000 per 32 words): 107 us at the size above; the voxel per
// thread before it took 330, with 79 for the passes that prepared it.
template <bool kTris, typename K>
__global__ void __launch_bounds__(kClassThreads, 8) k_word_classify(int kb, const float2* __restrict__ vals,
                                                               const unsigned int* __restrict__ n_dev,
                                                               const unsigned int* __restrict__ rows, MeshWords words,
                                                               uint4* __restrict__ run_out,
                                                               uint2* __restrict__ flagged,
                                                               MeshCounts* __restrict__ mc) {
    constexpr int kWarps = kClassThreads / 32;
    __shared__ uint64_t s_mc[256];
    __shared__ unsigned int s_nx[kWarps][8][32], s_tri[kWarps][32];
    __shared__ unsigned int s_sum[kWarps], s_ind[kWarps];
    __shared__ unsigned short s_item[kWarps][1024];  // lane << 5 | bit
    if (kTris) mc_table_to_shared(s_mc);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int n = *n_dev, n_words = *words.count;
    const K* wkey = (const K*)words.key;
    const unsigned int len = run_length(n_words, gridDim.x, 32u);
    const unsigned int lo = min(blockIdx.x * len, n_words), hi = min(lo + len, n_words);
    const K dy = (K)1 << (kb - 5), dz = (K)1 << (2 * kb - 5);
    unsigned int verts = 0, inds = 0, flags = 0;  // this run's so far
    // the run's list of voxels with output starts at its first voxel's slot
    const unsigned int list0 = lo < hi ? words.a[lo].x : 0u;
    for (unsigned int j0 = lo; j0 < hi; j0 += kClassThreads) {
        const unsigned int j = j0 + threadIdx.x;
        unsigned int vx = 0, vy = 0, vz = 0, tri = 0;
        unsigned int q2 = 0, q4 = 0, q6 = 0;
        unsigned int nx[8] = {};  // Distance() < 0 of the eight corners
        K key = 0;
        if (j < hi) {
            key = wkey[j] >> 4;
            constexpr int kD = kTris ? 3 : 2;  // +y, +z (and +yz)
            const K t[3] = {key + dy, key + dz, key + dy + dz};
            // every row's first word, then every row's four words about the guess -- this word's offset
            // in its own row, as neighbouring rows of a surface hold similar runs -- at once
            const unsigned int own = rows[key >> (kb - 5)];
            unsigned int s[kD], g[kD], q[kD];
            bool f[3] = {};
            K w[kD][4];
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                const K r = t[d] >> (kb - 5);
                s[d] = r >> (2 * kb) ? kNoWord : rows[r];
            }
            const unsigned int back = j - own > 1u ? j - own - 1u : 0u;
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                g[d] = s[d] == kNoWord ? 0u : min(s[d] + back, n_words - 1u);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    w[d][k] = s[d] != kNoWord && g[d] + k < n_words ? wkey[g[d] + k] >> 4 : ~(K)0;
            }
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                if (s[d] == kNoWord) {
                    // an empty row: after it only the next row's first key matters, to the row's last key
                    const K r1 = (t[d] >> (kb - 5)) + 1;
                    const bool last = ((t[d] + 1) & (((K)1 << (kb - 5)) - 1)) == 0;
                    q[d] = last && !(r1 >> (2 * kb)) ? min(rows[r1], n_words) : n_words;
                } else {
                    q[d] = find_word<K>(wkey, t[d], s[d], g[d], w[d], n_words, kb);
                    // (a word beyond the window: looked at again)
                    f[d] = q[d] < n_words && wkey[q[d]] >> 4 == t[d];
                }
            }
            q2 = q[0];
            q4 = q[1];
            if (kTris) q6 = q[kD - 1];
            const bool f2 = f[0], f4 = f[1], f6 = kTris && f[kD - 1];
            const CornerRow c0 = corner_row<K>(words, key, j, true, n_words);
            CornerRow c2 = corner_row<K>(words, key + dy, q2, f2, n_words);
            CornerRow c4 = corner_row<K>(words, key + dz, q4, f4, n_words);
            CornerRow c6 = {};
            if (kTris) c6 = corner_row<K>(words, key + dy + dz, q6, f6, n_words);
            unsigned int live = c0.E;
            if (j + 1 == n_words) live &= ~top_bit(c0.M);
            auto no_last = [&](CornerRow& c, unsigned int q, bool f) {
                if (f && q + 1 == n_words) {
                    const unsigned int m = ~top_bit(c.M);
                    c.E &= m;
                    c.P &= m;
                }
            };
            no_last(c2, q2, f2);
            no_last(c4, q4, f4);
            if (kTris) no_last(c6, q6, f6);
            // vertices: neighbour weight > 0 and a change of sign; by the divisions where an
            // operand is out of the sign rule's range
            auto axis = [&](unsigned int P, unsigned int N, unsigned int R, unsigned int start, unsigned int M,
                            bool self) {
                const unsigned int may = live & P;
                unsigned int v = may & c0.R & R & (c0.N ^ N);
                unsigned int slow = may & ~(c0.R & R);
                while (slow) {
                    const unsigned int b = __ffs(slow) - 1u;
                    slow &= slow - 1u;
                    const unsigned int i = c0.start + __popc(c0.M & ((1u << b) - 1u));
                    const unsigned int o = self ? i + 1u : start + __popc(M & ((1u << b) - 1u));
                    if (cross_exact(vals, i, o)) v |= 1u << b;
                }
                return v;
            };
            vx = axis(c0.Pn, c0.Nn, c0.Rn, 0u, 0u, true);
            vy = axis(c2.P, c2.N, c2.R, c2.start, c2.M, false);
            vz = axis(c4.P, c4.N, c4.R, c4.start, c4.M, false);
            if (kTris) {
                nx[0] = c0.N;
                nx[1] = c0.Nn;
                nx[2] = c2.N;
                nx[3] = c2.Nn;
                nx[4] = c4.N;
                nx[5] = c4.Nn;
                nx[6] = c6.N;
                nx[7] = c6.Nn;
                const unsigned int all = live & c0.En & c2.E & c2.En & c4.E & c4.En & c6.E & c6.En;
                const unsigned int any = nx[0] | nx[1] | nx[2] | nx[3] | nx[4] | nx[5] | nx[6] | nx[7];
                const unsigned int every = nx[0] & nx[1] & nx[2] & nx[3] & nx[4] & nx[5] & nx[6] & nx[7];
                tri = all & any & ~every;
                // A cube whose corners all have weight > 0 and operands in range, and whose last corner
                // is not the last voxel, has a vertex on every edge its triangles use (the table uses
                // exactly the edges whose corners differ in sign); the others are looked at edge by edge.
                const unsigned int good = c0.Pn & c2.P & c2.Pn & c4.P & c4.Pn & c6.P & c6.Pn & c0.R & c0.Rn & c2.R &
                                          c2.Rn & c4.R & c4.Rn & c6.R & c6.Rn;
                unsigned int odd = tri & ~good;
                if (f6 && q6 + 1 == n_words) odd |= tri & top_bit(c6.M) >> 1;
                if (f6 && q6 + 2 == n_words) odd |= tri & 0x80000000u;  // key + 1 may be the last word's only voxel
                while (odd) {
                    const unsigned int b = __ffs(odd) - 1u;
                    odd &= odd - 1u;
                    unsigned int neg = 0;
#pragma unroll
                    for (int c = 0; c < 8; ++c) neg |= (nx[c] >> b & 1u) << c;
                    missing_edges(words, vals, n, make_uint4(j, q2, q4, q6), b, neg,
                                  (unsigned long long)key << 5 | b, (unsigned long long)dy << 5,
                                  (unsigned long long)dz << 5, &mc->missing_min);
                }
            }
        }
        unsigned int out = vx | vy | vz | tri;  // voxels with output
        const bool any_out = out != 0u;
        const unsigned int nv = __popc(vx) + __popc(vy) + __popc(vz);
        // the run's positions: vertices and listed voxels before this word (both below 2^16 here)
        const unsigned int mine = (unsigned int)__popc(out) << 16 | nv;
        unsigned int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s_sum[warp] = inc;
        __syncthreads();
        unsigned int ex = inc - mine, total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const unsigned int c = s_sum[w];
            if (w < warp) ex += c;
            total += c;
        }
        // The warp's voxels with output are listed in shared memory and then taken 32 at a time: a
        // loop over each word's own would wait on the word with the most.
        const unsigned int at = ex >> 16, at0 = __shfl_sync(0xffffffffu, at, 0);
        const unsigned int items = __shfl_sync(0xffffffffu, at + __popc(out), 31) - at0;
        if (kTris) {
#pragma unroll
            for (int c = 0; c < 8; ++c) s_nx[warp][c][lane] = nx[c];
            s_tri[warp][lane] = tri;
        }
        for (unsigned int o = at - at0; out; ++o) {
            s_item[warp][o] = (unsigned short)(lane << 5 | (__ffs(out) - 1u));
            out &= out - 1u;
        }
        __syncwarp();
        unsigned int n_ind = 0;  // the warp's indices so far
        uint2* list = flagged + list0 + flags + at0;
        for (unsigned int k0 = 0; k0 < items; k0 += 32u) {
            const bool valid = k0 + lane < items;
            const unsigned int it = valid ? s_item[warp][k0 + lane] : 0u, w = it >> 5, b = it & 31u;
            unsigned int lut = 0, ni = 0;
            if (kTris) {
                if (valid && (s_tri[warp][w] >> b & 1u)) {
                    lut = lut_of(s_nx[warp][0][w] >> b, s_nx[warp][1][w] >> b, s_nx[warp][2][w] >> b,
                                 s_nx[warp][3][w] >> b, s_nx[warp][4][w] >> b, s_nx[warp][5][w] >> b,
                                 s_nx[warp][6][w] >> b, s_nx[warp][7][w] >> b);
                    ni = 3u * mc_tri_count_of(s_mc[lut]);
                }
                unsigned int inc = ni;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += y;
                }
                ni = n_ind + inc - ni;  // the voxel's first index, from the warp's first
                n_ind += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (valid) list[k0 + lane] = make_uint2((j0 + 32u * warp + w - lo) << 13 | b << 8 | lut, ni);
        }
        if (j < hi) words.v[j] = make_uint4(vx, vy, vz, verts + (ex & 0xffffu));
        verts += total & 0xffffu;
        flags += total >> 16;
        if (kTris) {
            if (lane == 0) s_ind[warp] = n_ind;
            __syncthreads();
            unsigned int before = inds;
#pragma unroll
            for (int w = 0; w < kClassThreads / 32; ++w) {
                const unsigned int c = s_ind[w];
                if (w < warp) before += c;
                inds += c;
            }
            if (any_out) words.link[j] = make_uint4(q2, q4, q6, before);
        } else {
            if (vy | vz) words.link[j] = make_uint4(q2, q4, 0u, 0u);
            __syncthreads();  // s_sum is rewritten by the next step
        }
    }
    __shared__ bool s_last;
    if (threadIdx.x == 0) {
        run_out[blockIdx.x] = make_uint4(verts, inds, flags, list0);
        __threadfence();
        s_last = atomicAdd(&mc->runs_done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    // totals to offsets, in place; the sums after the last (the loads of a thread's stretch all in flight)
    __threadfence();
    constexpr unsigned int kEach = (kWordRuns + kClassThreads - 1) / kClassThreads;
    const unsigned int each = (gridDim.x + kClassThreads - 1u) / kClassThreads, k0 = each * threadIdx.x;
    const unsigned int mine = k0 < gridDim.x ? min(each, gridDim.x - k0) : 0u;
    unsigned long long vi = 0, f = 0, vi_all, f_all;  // indices << 32 | vertices: each below 2^32 under 2^28 voxels
#pragma unroll
    for (unsigned int k = 0; k < kEach; ++k) {
        const uint4 c = k < mine ? __ldcg(run_out + k0 + k) : make_uint4(0u, 0u, 0u, 0u);
        vi += (unsigned long long)c.y << 32 | c.x;
        f += c.z;
    }
    vi = block_exclusive_scan<kClassThreads>(vi, &vi_all);
    f = block_exclusive_scan<kClassThreads>(f, &f_all);
#pragma unroll 8
    for (unsigned int k = 0; k < mine; ++k) {
        const uint4 c = __ldcg(run_out + k0 + k);
        __stcg(run_out + k0 + k, make_uint4((unsigned int)vi, (unsigned int)(vi >> 32), (unsigned int)f, c.w));
        vi += (unsigned long long)c.y << 32 | c.x;
        f += c.z;
    }
    if (threadIdx.x == 0)
        run_out[gridDim.x] = make_uint4((unsigned int)vi_all, (unsigned int)(vi_all >> 32), (unsigned int)f_all, 0u);
}

// Emission over the voxels with output in ascending order (the runs' lists
// end to end), 32 per warp step.  A voxel's first vertex, and that of each
// corner of its cube, is counted from the corner's word: the word's first
// vertex plus the set bits below in its three vertex masks.  139 us at the size
// above, of it 43 for the bytes; bound by instructions (560 per 32 voxels).  With
// flags and lookups kept per voxel: 103 us, but run twice for the stop rule.
template <bool kTris, typename K>
__global__ void __launch_bounds__(kThreads) k_mesh_emit(int kb, const float2* __restrict__ vals, Geom g,
                                                        MeshWords words, const uint4* __restrict__ run_out,
                                                        unsigned int runs,
                                                        const uint2* __restrict__ flagged,
                                                        MeshCounts* __restrict__ mc, unsigned int words_cap,
                                                        unsigned long long vert_cap,
                                                        unsigned long long idx_cap, float* __restrict__ verts,
                                                        uint32_t* __restrict__ idx) {
    __shared__ uint64_t s_mc[256];
    if (kTris) mc_table_to_shared(s_mc);
    __shared__ unsigned int s_cf[kWordRuns + 1];  // the runs' first listed voxels
    for (unsigned int k = threadIdx.x; k <= runs; k += kThreads) s_cf[k] = run_out[k].z;
    __syncthreads();
    const unsigned int n_verts = run_out[runs].x, n_idx = run_out[runs].y, n_out = s_cf[runs];
    // outputs that do not fit are not written (every CTA returns alike; the host grows and re-emits)
    const bool too_many = mc->n_words > words_cap;
    const bool overflow = too_many || n_verts > vert_cap || (kTris && n_idx > idx_cap);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        mc->n_verts = n_verts;
        mc->n_idx = n_idx;
        mc->overflow = too_many ? kMeshWords : overflow ? kMeshBuffers : 0ull;
    }
    if (overflow) return;
    const unsigned long long bound = kTris ? mc->missing_min : ~0ull;  // ids from here on stay ids
    // Triangles are emitted warp-cooperatively: the warp's 32 voxels stage their
    // case word, the vertices of their cubes' 12 edges, their first output slot
    // and a list of their triangles in shared memory, and all lanes walk the
    // triangles together, so a warp does not wait on its lane with the most.
    constexpr int kWarps = kThreads / 32;
    __shared__ unsigned int s_vert[kWarps][12][32];  // each edge's vertex
    __shared__ uint64_t s_mcw[kWarps][32];
    __shared__ unsigned int s_first[kWarps][32];
    __shared__ unsigned char s_map[kWarps][160];  // voxel's lane << 3 | triangle (at most 5)
    const Codec<K> cd(kb);
    const K* wkey = (const K*)words.key;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned int warps = gridDim.x * kWarps;
    const unsigned int len = run_length(*words.count, runs, 32u);
    const unsigned int inv = len > 1u ? (unsigned int)(0x100000000ull / len) : 0xffffffffu;
    auto run_of = [&](unsigned int j) {  // j / len: the estimate is at most one short
        unsigned int c = __umulhi(j, inv);
        if (j - c * len >= len) ++c;
        return c;
    };
    // the listed voxels are cut into steps of 32; each warp takes a contiguous run of steps
    const unsigned int steps = (n_out + 31u) / 32u;
    const unsigned int wid = blockIdx.x * kWarps + warp;
    const unsigned int cbeg = (unsigned int)((unsigned long long)steps * wid / warps);
    const unsigned int cend = (unsigned int)((unsigned long long)steps * (wid + 1) / warps);
    unsigned int run = 0;
    if (cbeg < cend) {  // the warp's first run of words: the last with a first position <= 32 cbeg
        unsigned int a = 0, b = runs;
        while (a + 1 < b) {
            const unsigned int mid = (a + b) >> 1;
            if (s_cf[mid] <= 32u * cbeg) a = mid;
            else b = mid;
        }
        run = a;
    }
    // a step's listed voxels, loaded a step ahead
    unsigned int rl_next = 0;
    uint2 item_next = make_uint2(0u, 0u);
    auto next_items = [&](unsigned int ch) {
        const unsigned int gpos = 32u * ch + lane;
        const bool valid = ch < cend && gpos < n_out;
        rl_next = run;
        if (valid) {
            while (s_cf[rl_next + 1] <= gpos) ++rl_next;  // s_cf[runs] = n_out > gpos
            item_next = flagged[run_out[rl_next].w + (gpos - s_cf[rl_next])];
        }
        run = __shfl_sync(0xffffffffu, rl_next, 31);  // positions only move forward
    };
    next_items(cbeg);
    for (unsigned int ch = cbeg; ch < cend; ++ch) {
        const bool valid = 32u * ch + lane < n_out;
        const unsigned int rl = rl_next;
        const uint2 item = valid ? item_next : make_uint2(0u, 0u);
        next_items(ch + 1u);
        const unsigned int j = rl * len + (item.x >> 13), bit = item.x >> 8 & 31u, lut = item.x & 0xffu;
        const unsigned int lt = (1u << bit) - 1u;
        uint4 v0 = make_uint4(0u, 0u, 0u, 0u), a0 = v0, link = v0;
        K key = 0;
        uint4 ofs = make_uint4(0u, 0u, 0u, 0u);
        if (valid) {
            ofs = run_out[rl];
            v0 = words.v[j];
            a0 = words.a[j];
            key = wkey[j] >> 4 << 5 | (K)bit;
            link = words.link[j];
        }
        const unsigned int axes = (v0.x >> bit & 1u) | (v0.y >> bit & 1u) << 1 | (v0.z >> bit & 1u) << 2;
        // a voxel's first vertex: its word's, plus those of the word's voxels below
        auto rank = [](const uint4& v, unsigned int below) {
            return v.w + __popc(v.x & below) + __popc(v.y & below) + __popc(v.z & below);
        };
        // vertices (Mesher.cpp:134-168): at most three per voxel, by the voxel's lane
        if (axes) {
            const unsigned int vbase = ofs.x + rank(v0, lt);
            const unsigned int nv = __popc(axes);
            const unsigned int first = kTris ? vbase : n_verts - vbase - nv;  // ascending ids / generation order
            const float cx = fadd(fmul((float)(int)cd.x(key), g.vlen), g.center_off);
            const float cy = fadd(fmul((float)(int)cd.y(key), g.vlen), g.center_off);
            const float cz = fadd(fmul((float)(int)cd.z(key), g.vlen), g.center_off);
            const unsigned int self = a0.x + __popc(a0.y & lt);
            unsigned int nb[3];  // the neighbours' voxels (a flagged axis: the neighbour exists)
            nb[0] = self + 1u;
            uint4 ay = make_uint4(0u, 0u, 0u, 0u), az = ay;
            if (axes & 2u) ay = words.a[link.x];
            if (axes & 4u) az = words.a[link.y];
            nb[1] = ay.x + __popc(ay.y & lt);
            nb[2] = az.x + __popc(az.y & lt);
            const float dself = vdist(vals[self]);
            float2 vn[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if (axes >> a & 1u) vn[a] = vals[nb[a]];
            unsigned int r = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (!(axes >> a & 1u)) continue;
                const float dn = vdist(vn[a]);
                const float t = fmul(fdiv(fabsf(dself), fadd(fabsf(dself), fabsf(dn))), g.vlen);
                float p[3] = {cx, cy, cz};
                p[a] = fadd(p[a], t);
                float* o = verts + 3 * (unsigned long long)(first + r);
                o[0] = p[0];
                o[1] = p[1];
                o[2] = p[2];
                ++r;
            }
        }
        if constexpr (kTris) {
            const uint64_t mcw = s_mc[lut];
            const unsigned int nt = valid ? mc_tri_count_of(mcw) : 0u;
            unsigned int inc = nt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            const unsigned int total = __shfl_sync(0xffffffffu, inc, 31);
            if (total == 0u) continue;  // warp-uniform
            __syncwarp();  // the previous round's readers are done with the staging
            if (nt) {
                for (unsigned int t = 0; t < nt; ++t) s_map[warp][inc - nt + t] = (unsigned char)(lane << 3 | t);
                s_mcw[warp][lane] = mcw;  // the case's triangle edges
                // generation order: voxels descending
                s_first[warp][lane] = n_idx - (ofs.y + link.w + item.y) - 3u * nt;
                // The corners' first vertices and axes, by rows along x: corner 2k and, along x from it,
                // 2k + 1 (in the next word when the voxel is its word's last key)
                const unsigned int q[4] = {j, link.x, link.y, link.z};
                uint4 v[4];
                unsigned int first[8], ax[8];
                v[0] = v0;
#pragma unroll
                for (int k = 1; k < 4; ++k) v[k] = words.v[q[k]];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    ax[2 * k] = (v[k].x >> bit & 1u) | (v[k].y >> bit & 1u) << 1 | (v[k].z >> bit & 1u) << 2;
                    first[2 * k] = (k ? run_out[run_of(q[k])].x : ofs.x) + rank(v[k], lt);
                    if (bit == 31u) {
                        const uint4 w = words.v[q[k] + 1u];
                        ax[2 * k + 1] = (w.x & 1u) | (w.y & 1u) << 1;
                        first[2 * k + 1] = run_out[run_of(q[k] + 1u)].x + w.w;
                    } else {
                        ax[2 * k + 1] = (v[k].x >> bit >> 1 & 1u) | (v[k].y >> bit >> 1 & 1u) << 1;
                        first[2 * k + 1] = first[2 * k] + __popc(ax[2 * k]);
                    }
                }
                // each edge's vertex: its corner's first, plus the corner's axes before the edge's
#pragma unroll
                for (int e = 0; e < 12; ++e)
                    s_vert[warp][e][lane] =
                        first[edge_corner(e)] + __popc(ax[edge_corner(e)] & ((1u << edge_axis(e)) - 1u));
                // edge ids 3 * key + axis from the stop rule's bound on stay ids: 32 bits wide for
                // 30-bit keys (as in the reference); for 64-bit keys the rule compares full ids and
                // an id written in place of a missing vertex keeps its low 32 bits
                if (3ull * (unsigned long long)(key + cd.pack(1, 1, 1)) + 2ull >= bound) {
#pragma unroll
                    for (int e = 0; e < 12; ++e) {
                        const int c = edge_corner(e);
                        const unsigned long long id = 3ull * (unsigned long long)(key + cd.pack(c & 1, c >> 1 & 1, c >> 2)) +
                                                      (unsigned long long)edge_axis(e);
                        if (id >= bound) s_vert[warp][e][lane] = (unsigned int)id;
                    }
                }
            }
            __syncwarp();
            for (unsigned int o = lane; o < total; o += 32u) {
                const unsigned int u = s_map[warp][o] >> 3, t = s_map[warp][o] & 7u;
                const unsigned int e3 = (unsigned int)(s_mcw[warp][u] >> (12u * t));
                uint32_t* d = idx + (unsigned long long)(s_first[warp][u] + 3u * t);
                d[0] = s_vert[warp][e3 & 15u][u];
                d[1] = s_vert[warp][e3 >> 4 & 15u][u];
                d[2] = s_vert[warp][e3 >> 8 & 15u][u];
            }
        }
    }
}

}  // namespace

namespace {

// one allocation, cut into 256-byte aligned arrays
struct Cut {
    size_t size = 0;
    size_t take(size_t bytes) {
        const size_t at = size;
        size += (bytes + 255) / 256 * 256;
        return at;
    }
};

// The words to expect of `cap` voxels: scans have 10 to 20 voxels to a word.  A
// word takes 64 B, so one per voxel (any volume fits then) is for small ones only;
// 16 B per voxel in all for the others, unless their words turn out to be more (of
// 14.6 M voxels in 1.36 M words 292 MB with headroom, where one per voxel took 1.3 GB).
size_t likely_words(size_t cap) {
    const size_t small = cap < 65536 ? cap : 65536;
    return cap / 8 > small ? cap / 8 : small;
}

cudaError_t alloc_block(MeshScratch* m, size_t cap, size_t words) {
    cudaFree(m->block);
    m->block = nullptr;
    m->cap = m->words_cap = 0;
    Cut c;
    ++words;  // reads go to the word behind the last
    const size_t key = c.take(words * sizeof(uint64_t)), a = c.take(words * sizeof(uint4)),
                 b = c.take(words * sizeof(uint2)), v = c.take(words * sizeof(uint4)),
                 link = c.take(words * sizeof(uint4)), flagged = c.take(cap * sizeof(uint2));
    const cudaError_t e = cudaMalloc(&m->block, c.size);
    if (e) {
        cudaGetLastError();
        return e;
    }
    unsigned char* p = (unsigned char*)m->block;
    m->words.key = p + key;
    m->words.a = (uint4*)(p + a);
    m->words.b = (uint2*)(p + b);
    m->words.v = (uint4*)(p + v);
    m->words.link = (uint4*)(p + link);
    m->flagged = (uint2*)(p + flagged);
    m->cap = cap;
    m->words_cap = words - 1;
    return cudaSuccess;
}

// The voxel count is read on the device from ms.n_dev (<= n_cap, which sizes
// the grids), so the passes can be enqueued before the count is known.
unsigned int mesh_runs(size_t n_cap, unsigned int most) {
    const size_t r = (n_cap + kBuildTile - 1) / kBuildTile;
    return (unsigned int)(r < 1 ? 1 : (r < most ? r : most));
}

template <typename K>
void count_words(const K* keys, size_t n_cap, int kb, const MeshScratch& ms, cudaStream_t st) {
    const unsigned int vruns = mesh_runs(n_cap, kVoxelRuns);
    const unsigned int row_vecs = (unsigned int)(((size_t)1 << (2 * kb)) / 4);
    // four vectors of the row table per thread, eight CTAs per SM of the 152 at most
    const unsigned int clear = row_vecs / (4 * kThreads) < kVoxelRuns / 2 ? row_vecs / (4 * kThreads) : kVoxelRuns / 2;
    k_word_count<K><<<vruns > clear ? vruns : clear, kThreads, 0, st>>>(keys, ms.n_dev, ms.run_words, vruns,
                                                                        (uint4*)ms.rows, row_vecs, ms.counts);
}

cudaError_t alloc_tables(MeshScratch* m, int kb) {
    const size_t rows = (size_t)1 << (2 * kb);
    if (m->tables && m->rows_cap >= rows) return cudaSuccess;
    cudaFree(m->tables);
    m->tables = nullptr;
    m->rows_cap = 0;
    Cut c;
    const size_t run_words = c.take(kVoxelRuns * sizeof(unsigned int)), run_out = c.take((kWordRuns + 1) * sizeof(uint4)),
                 row = c.take(rows * sizeof(unsigned int)), counts = c.take(sizeof(MeshCounts)),
                 single = c.take(2 * sizeof(unsigned int));
    const cudaError_t e = cudaMalloc(&m->tables, c.size);
    if (e) {
        cudaGetLastError();
        return e;
    }
    unsigned char* p = (unsigned char*)m->tables;
    m->words.count = (unsigned int*)(p + single) + 1;
    m->run_words = (unsigned int*)(p + run_words);
    m->run_out = (uint4*)(p + run_out);
    m->rows = (unsigned int*)(p + row);
    m->counts = (MeshCounts*)(p + counts);
    m->n_dev = (unsigned int*)(p + single);
    m->rows_cap = rows;
    return cudaSuccess;
}

}  // namespace

cudaError_t mesh_scratch_reserve(MeshScratch* m, size_t n, size_t want, size_t n_words, int kb) {
    cudaError_t e = alloc_tables(m, kb);
    if (e || (m->block && m->cap >= n && m->words_cap >= n_words)) return e;
    if (want < m->cap) want = m->cap;
    if (want < 1024) want = 1024;
    const size_t likely = likely_words(want), ahead = n_words + n_words / 4;
    e = alloc_block(m, want, likely > ahead ? likely : ahead);
    if (e == cudaErrorMemoryAllocation) {
        const size_t words = likely_words(n);
        e = alloc_block(m, n, words > n_words ? words : n_words);
    }
    return e;
}

void mesh_scratch_free(MeshScratch* m) {
    cudaFree(m->tables);
    cudaFree(m->block);
    *m = MeshScratch{};
}

template <typename K>
static void mesh_count_t(const K* keys, const float2* vals, size_t n_cap, int kb, int with_indices, MeshScratch& ms,
                         cudaStream_t st, cudaEvent_t* stage_events) {
    const unsigned int vruns = mesh_runs(n_cap, kVoxelRuns), wruns = mesh_runs(n_cap, kWordRuns);
    count_words<K>(keys, n_cap, kb, ms, st);
    k_word_build<K><<<vruns, kThreads, 0, st>>>(keys, kb, vals, ms.n_dev, ms.run_words, ms.rows, ms.words,
                                                  (unsigned int)ms.words_cap, ms.counts);
    if (stage_events) cudaEventRecord(stage_events[0], st);
    if (with_indices)
        k_word_classify<true, K><<<wruns, kClassThreads, 0, st>>>(kb, vals, ms.n_dev, ms.rows, ms.words, ms.run_out,
                                                              ms.flagged, ms.counts);
    else
        k_word_classify<false, K><<<wruns, kClassThreads, 0, st>>>(kb, vals, ms.n_dev, ms.rows, ms.words, ms.run_out,
                                                               ms.flagged, ms.counts);
    if (stage_events) cudaEventRecord(stage_events[1], st);
}

cudaError_t mesh_count_enqueue(const void* keys, int key_bytes, const float2* vals, size_t n_cap, int kb, int with_indices,
                               MeshScratch& ms, cudaStream_t st, cudaEvent_t* stage_events) {
    if (key_bytes == 8)
        mesh_count_t<uint64_t>((const uint64_t*)keys, vals, n_cap, kb, with_indices, ms, st, stage_events);
    else mesh_count_t<uint32_t>((const uint32_t*)keys, vals, n_cap, 10, with_indices, ms, st, stage_events);
    return cudaGetLastError();
}

// up to 4 CTAs per SM (all resident), each with 2048 voxels of the volume or more
template <typename K>
static void mesh_emit_t(const Geom& g, const float2* vals, size_t n_cap, int with_indices, MeshScratch& ms,
                        size_t vert_cap, size_t idx_cap, float* verts_dev, uint32_t* idx_dev, int sms,
                        cudaStream_t st) {
    const int kb = sizeof(K) == 4 ? 10 : g.kb;
    const size_t want = (n_cap + 2047) / 2048;
    const unsigned int runs = mesh_runs(n_cap, kWordRuns);  // as the classification's
    const int grid = (int)(want < 1 ? 1 : (want > (size_t)sms * 4 ? (size_t)sms * 4 : want));
    if (with_indices)
        k_mesh_emit<true, K><<<grid, kThreads, 0, st>>>(kb, vals, g, ms.words, ms.run_out, runs, ms.flagged, ms.counts,
                                                       (unsigned int)ms.words_cap, vert_cap, idx_cap, verts_dev, idx_dev);
    else
        k_mesh_emit<false, K><<<grid, kThreads, 0, st>>>(kb, vals, g, ms.words, ms.run_out, runs, ms.flagged, ms.counts,
                                                        (unsigned int)ms.words_cap, vert_cap, idx_cap, verts_dev, idx_dev);
}

cudaError_t mesh_emit_enqueue(const Geom& g, int key_bytes, const float2* vals, size_t n_cap, int with_indices,
                              MeshScratch& ms, size_t vert_cap, size_t idx_cap, float* verts_dev, uint32_t* idx_dev,
                              int sms, cudaStream_t st) {
    if (key_bytes == 8)
        mesh_emit_t<uint64_t>(g, vals, n_cap, with_indices, ms, vert_cap, idx_cap, verts_dev, idx_dev, sms, st);
    else
        mesh_emit_t<uint32_t>(g, vals, n_cap, with_indices, ms, vert_cap, idx_cap, verts_dev, idx_dev, sms, st);
    return cudaGetLastError();
}

// Copy of the resident voxels (buffer ctl->cur, ctl->n[cur] of them) for a
// mesh that runs while fusion goes on; the count goes to *n_dev.  16-byte
// loads (four 32-bit or two 64-bit keys, two voxels), four in flight per
// thread, streaming past L1; the buffers are cudaMalloc'd (256-byte aligned).
template <typename K>
__global__ void __launch_bounds__(256) k_mesh_snapshot(const DeviceCtl* __restrict__ ctl, VolumeBuffers vb,
                                                       K* __restrict__ keys, float2* __restrict__ vals,
                                                       unsigned long long cap, unsigned int* __restrict__ n_dev) {
    constexpr unsigned int kPerVec = 16 / sizeof(K);  // keys per 16 bytes
    const unsigned int cur = ctl->cur;
    unsigned long long n = ctl->n[cur];
    if (n > cap) n = cap;
    const K* sk = (const K*)(cur ? vb.keys[1] : vb.keys[0]);
    const float2* sv = cur ? vb.vals[1] : vb.vals[0];
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned long long t0 = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    // keys: n / kPerVec vectors, then the tail
    const unsigned long long nk = n / kPerVec;
    const uint4* ks = reinterpret_cast<const uint4*>(sk);
    uint4* kd = reinterpret_cast<uint4*>(keys);
    for (unsigned long long i = t0; i < nk; i += 4 * stride) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < nk) v[u] = __ldcs(ks + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < nk) kd[i + u * stride] = v[u];
    }
    for (unsigned long long i = nk * kPerVec + t0; i < n; i += stride) keys[i] = __ldcs(sk + i);
    // voxels: two per vector
    const unsigned long long nv = n / 2;
    const float4* vs = reinterpret_cast<const float4*>(sv);
    float4* vd = reinterpret_cast<float4*>(vals);
    for (unsigned long long i = t0; i < nv; i += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < nv) v[u] = __ldcs(vs + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < nv) vd[i + u * stride] = v[u];
    }
    if ((n & 1) && t0 == 0) vals[n - 1] = __ldcs(sv + n - 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_dev = (unsigned int)n;
}

cudaError_t mesh_snapshot_enqueue(const DeviceCtl* ctl, const VolumeBuffers& vb, void* keys, float2* vals,
                                  size_t cap, unsigned int* n_dev, int sms, cudaStream_t st) {
    if (vb.key_bytes == 8)
        k_mesh_snapshot<uint64_t><<<sms * 4, 256, 0, st>>>(ctl, vb, (uint64_t*)keys, vals, cap, n_dev);
    else
        k_mesh_snapshot<uint32_t><<<sms * 4, 256, 0, st>>>(ctl, vb, (uint32_t*)keys, vals, cap, n_dev);
    return cudaGetLastError();
}

}  // namespace kifi
