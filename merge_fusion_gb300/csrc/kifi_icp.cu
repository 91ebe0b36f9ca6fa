// kifi_icp.cu -- projective ICP on sm_103a: kifi::ICP::Align / AlignStep
// (KinectFission/kifi/ICP.cpp:9-265) and its target producers,
// Renderer::Bin (Renderer.cpp:39-80) and a depth back-projection.
//
// One AlignStep is one kernel, k_icp_step, ending in a last-CTA-done
// finisher, so a whole Align (any iteration count) is a fixed launch sequence
// with no host round trip:
//
//  association   every row and every 4th column (ICP.cpp:66-67) is a source
//                pixel: back-project it with the current pose estimate,
//                project into the target camera, search the 21x21 window for
//                the nearest valid target point within len^2 < 0.01
//                (:100-131; the first minimum in scan order wins).  Only the
//                candidates that can win are read: a bound on the distance
//                (the last step's winner, or a few probes) cuts the window to
//                a rectangle, see Prune.  Where that is much of the window
//                (the first step, fast motion, targets of which nothing is
//                known) a tile scans its windows whole, two candidates at a
//                time.  CTAs own tiles of sources and stage the part of the
//                target they will read in shared memory.
//  moments       the associated pairs are not stored: count, sum p, sum q,
//                sum p q^T and the squared distances are accumulated per
//                CTA in float-float, each product split exactly by an FMA.
//  finisher      the last CTA totals the per-CTA partials, and one warp
//                forms the centroids and the centred cross-covariance
//                (:166-197), Horn's matrix (:199-213), its dominant
//                eigenvector (:215-231), R and t (:233-261) and the pose
//                update (:20-28), without double precision (see the Horn
//                solve below).
//
// Consecutive steps are programmatic dependent launches: the next step's
// grid is scheduled once every CTA has finished its association, and waits
// (griddepcontrol.wait) for the finisher before it reads the pose.
//
// The per-point arithmetic follows the reference's float expression order
// and x86 float-to-int conversion (CVTTSS2SI: truncation, INT_MIN for NaN or
// out-of-range); the reference's 640x480 window clamp (:108-109) is kept,
// with reads past the end of a smaller target buffer treated as invalid
// points.
#include <type_traits>

#include "kifi_internal.h"

namespace kifi {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ int cvt_i32_x86(float f) {
    if (f >= -2147483648.0f && f < 2147483648.0f) return __float2int_rz(f);
    return INT_MIN;
}
__device__ __forceinline__ int wrap_sub(int a, int b) { return (int)((unsigned int)a - (unsigned int)b); }

// Float-float (double-single) arithmetic: a value is hi + lo with |lo| about
// ulp(hi)/2 or less -- a 48-bit significand.  GB300 issues double precision
// at a small fraction of the float rate, so every compensated sum and the
// Horn solve's precise steps use float pairs instead.
struct FF {
    float hi, lo;
};
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = fadd(a, b);
    float bb = fsub(s, a);
    e = fadd(fsub(a, fsub(s, bb)), fsub(b, bb));
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
    float s, e;
    two_sum(a.hi, b.hi, s, e);
    e = fadd(e, fadd(a.lo, b.lo));
    const float hi = fadd(s, e);
    return FF{hi, fsub(e, fsub(hi, s))};
}
__device__ __forceinline__ FF ff_norm(float hi, float lo) {  // |lo| may exceed ulp(hi)/2
    const float s = fadd(hi, lo);
    return FF{s, fsub(lo, fsub(s, hi))};
}
__device__ __forceinline__ FF operator+(FF a, FF b) { return ff_add(a, b); }
__device__ __forceinline__ FF operator-(FF a, FF b) { return ff_add(a, FF{-b.hi, -b.lo}); }
__device__ __forceinline__ FF operator-(FF a) { return FF{-a.hi, -a.lo}; }
__device__ __forceinline__ FF operator*(FF a, FF b) {
    const float p = fmul(a.hi, b.hi);
    const float e = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p)));
    return ff_norm(p, e);
}
__device__ __forceinline__ FF operator*(FF a, float b) {
    const float p = fmul(a.hi, b);
    return ff_norm(p, __fmaf_rn(a.lo, b, __fmaf_rn(a.hi, b, -p)));
}
__device__ __forceinline__ FF ff_div(FF a, FF b) {  // a / b, b != 0
    const float q1 = fdiv(a.hi, b.hi);
    const FF r = a - b * q1;
    return ff_norm(q1, fdiv(r.hi, b.hi));
}
__device__ __forceinline__ float load_depth(const void* depth, size_t i, bool u16) {
    if (u16) return fmul((float)(unsigned int)__ldg((const unsigned short*)depth + i), 0.001f);
    return __ldg((const float*)depth + i);
}

// Last CTA to arrive returns true and gets the grid's total of `mine` (an
// association count, read after the barrier); resets the counter.  The
// counter holds finished CTAs in its high 32 bits and the running total in
// its low 32 bits, so one atomic does both.  Thread 0's atomic orders the
// whole CTA's earlier stores (the barrier makes them visible to it) before
// the count, and the count before the last CTA's reads.
__device__ __forceinline__ bool last_cta(unsigned long long* counter, const unsigned int& mine,
                                         unsigned int* total, unsigned int nblk) {
    __shared__ bool last;
    __shared__ unsigned int s_total;
    __syncthreads();
    if (threadIdx.x == 0) {
        // one acquire-release atomic at gpu scope: the release (cumulative
        // over the CTA's writes ordered before it by the barrier) publishes
        // this CTA's partials; the acquire lets the last CTA read everyone's
        const unsigned long long add = (1ull << 32) | mine;
        unsigned long long prev;
        asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;"
                     : "=l"(prev) : "l"(counter), "l"(add) : "memory");
        last = (unsigned int)(prev >> 32) == nblk - 1;
        s_total = (unsigned int)prev + mine;
        if (last) *counter = 0ull;  // read again only by the next launch
    }
    __syncthreads();
    *total = s_total;
    return last;
}

// Totals of the per-CTA float-float partials, by the whole (last) CTA.  The
// partials are stored component-major (hi row, then lo row, each
// kIcpMaxCtas long), so warp w (of 8) reduces components w + 1 and w + 9 (the count,
// component 0, comes with the last-CTA counter) with coalesced loads: lane l adds CTAs
// l, l + 32, ... in float-float -- all of a lane's loads (up to 320 CTAs)
// issued in one round -- then a shuffle tree.
// Fixed order: independent of scheduling.  The loads bypass L1 (the partials
// were written by other SMs during this launch).
constexpr int kTotalsPerLane = 10;
__device__ __forceinline__ FF lane_partials(const float* ph, int b0, int n) {
    float h[kTotalsPerLane], l[kTotalsPerLane];
#pragma unroll
    for (int k = 0; k < kTotalsPerLane; ++k) {
        const int b = b0 + 32 * k;
        h[k] = b < n ? __ldcg(ph + b) : 0.0f;
        l[k] = b < n ? __ldcg(ph + kIcpMaxCtas + b) : 0.0f;
    }
    FF acc{h[0], l[0]};
#pragma unroll
    for (int k = 1; k < kTotalsPerLane; ++k) acc = ff_add(acc, FF{h[k], l[k]});
    return acc;
}
template <int NV, int kWarps>
__device__ __forceinline__ void moments_total(const IcpState* st, unsigned int count, FF* out, int n) {
    constexpr int kPer = 16 / kWarps;  // moments w + 1 and, with 8 warps, w + 9 side by side
    const int lane = threadIdx.x & 31, c0 = (threadIdx.x >> 5) + 1;
    static_assert(NV == 17, "16 moments after the count");
    if (threadIdx.x == 0) out[0] = FF{(float)count, 0.0f};  // exact: at most 2^24 sources
    FF a[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) a[h] = FF{0.0f, 0.0f};
    for (int b0 = lane; b0 < n; b0 += 32 * kTotalsPerLane)
#pragma unroll
        for (int h = 0; h < kPer; ++h)
            a[h] = ff_add(a[h], lane_partials(st->part + (size_t)(2 * (c0 + kWarps * h)) * kIcpMaxCtas, b0, n));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const FF x{__shfl_xor_sync(0xffffffffu, a[h].hi, o), __shfl_xor_sync(0xffffffffu, a[h].lo, o)};
            a[h] = ff_add(a[h], x);
        }
    if (lane < kPer) out[c0 + kWarps * lane] = lane ? a[kPer - 1] : a[0];
    __syncthreads();
}

constexpr int kTileCols = 8, kTileRows = 32;
constexpr int kBlockW = 8, kBlockH = 4;  // target pixels per bounding box, a warp's worth
constexpr int kTileThreads = kTileCols * kTileRows;  // one source per thread
static_assert(kTileThreads == kIcpTileSources, "a winner per source");
constexpr int kPredMargin = 4;  // pixels added around the rectangles that a tile searched in the last step,
constexpr int kUseMargin = 4;   // and that the region so staged must leave around the projections to be used
// The step's builds.  Build kWhole scans whole windows only; the others scan
// windows or search rectangles, tile by tile (whole_next), and differ in how
// many tiles share an SM.  One: launches of no more tiles than SMs, with two
// threads per source.  Two: 80 KB of target and 128 registers a thread, for
// launches that fill no more than that in one round, where a tile's own time
// counts.  Three: 52 KB and 80 registers (a few spilled words) for more tiles: a
// tile takes longer, but 24 warps hide more of the waits (tracking at 1024x848,
// 864 tiles, ten frames 6140 -> 5817 us; at 640x480, 300 tiles, 327 against 333).
// 52 KB hold a tile's rectangles (32 pixels and up to 20 around) while the target's
// pixels are no finer than 1 / 1.15 of the source's; for finer ones the 80 KB stay
// (a 1024x768 target for 640x480 frames, the closed loop: 2100 us against 2365).
constexpr int kWhole = 0;
// Two halves of the CTA per source search half of the rows each: whole windows
// in 19 us a step at 640x480 (with one thread per source 21 to 26), and in small
// launches, where 8 warps would have an SM to themselves.
template <int kS>
constexpr int kHalves = kS <= 1 ? 2 : 1;
template <int kS>
constexpr int kResident = kS == kWhole ? 2 : kS;  // CTAs per SM
// Target points (float4) staged per tile.
template <int kS>
constexpr int kStagePixels = kS == kWhole ? 0 : kS == 3 ? 3328 : 5120;
constexpr int kWindowMargin = 5;  // pixels added around the windows that a tile scanned

// Row pitch of a staged region `w` pixels wide: odd, so that the 16-byte
// loads of eight lanes one row apart cover all banks.
__host__ __device__ constexpr int stage_pitch(int w) { return w | 1; }

// The target pixels [x0, x0 + w) x [y0, y0 + h) (linear index y * synth_w + x,
// as the reference reads them) into `stage` with row pitch `pitch`, by the
// CTA's warps, as 16-byte asynchronous copies (stage_wait, then a
// barrier, before they are read).  Points that are none (ICP.cpp:112) hold NaN in the
// target buffer; indices past the buffer's end are none too.
template <int kWarps>
__device__ __forceinline__ void stage_region(float4* stage, const float4* __restrict__ synth, size_t n_synth,
                                             int synth_w, int x0, int y0, int w, int h, int pitch) {
    // warps take rows, lanes take columns
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int ry = warp; ry < h; ry += kWarps) {
        for (int rx = lane; rx < w; rx += 32) {
            const size_t at = (size_t)(y0 + ry) * synth_w + (x0 + rx);
            float4* dst = stage + ry * pitch + rx;
            if (at < n_synth) {
                const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(synth + at) : "memory");
            } else {
                *dst = make_float4(__int_as_float(0x7fffffff), 0.f, 0.f, 0.f);
            }
        }
    }
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The same region as three float planes (x, y, z), for the whole-window scan:
// two adjacent candidates are one 64-bit load per plane.  The pitch is even, so
// that such pairs are aligned, with pitch / 2 odd, so that the 64-bit loads of
// lanes whose windows lie one row apart hit distinct banks.  Asynchronous copies
// (stage_wait) of 4 bytes: they take no registers, and the planes of a region
// staged ahead arrive while the step before finishes.
__host__ __device__ constexpr int plane_pitch(int w) {
    return ((w + 1) & ~1) + ((((w + 1) & ~1) >> 1) & 1 ? 0 : 2);
}
struct Planes {
    float *x, *y, *z;
};
template <int kWarps>
__device__ __forceinline__ void stage_planes(const Planes& stage, const float4* __restrict__ synth, size_t n_synth,
                                             int synth_w, int x0, int y0, int w, int h, int pitch) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned int dx = (unsigned int)__cvta_generic_to_shared(stage.x), dy = (unsigned int)__cvta_generic_to_shared(stage.y),
                       dz = (unsigned int)__cvta_generic_to_shared(stage.z);
    for (int ry = warp; ry < h; ry += kWarps) {
        for (int rx = lane; rx < w; rx += 32) {
            const size_t at = (size_t)(y0 + ry) * synth_w + (x0 + rx);
            const int to = ry * pitch + rx;
            if (at < n_synth && x0 + rx < 640) {  // (the reference's windows end at column 640)
                const float* q = reinterpret_cast<const float*>(synth + at);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dx + 4u * to), "l"(q) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dy + 4u * to), "l"(q + 1) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dz + 4u * to), "l"(q + 2) : "memory");
            } else {
                stage.x[to] = __int_as_float(0x7fffffff);
                stage.y[to] = stage.z[to] = 0.0f;
            }
        }
    }
}

// Which candidates of a source's window can win.
//
// A target point q at pixel x has a projected column X(q) in [x + lo, x + hi]
// (lo = hi = 1/2 for a back-projected frame, [0, 1] for a binned cloud), and
// the points whose column is X lie in a plane through the eye.  A source p at
// distance |n . p + n3| / |n| from that plane -- |X(p) - X| w / (W/2) over at
// most max |n| -- cannot be nearer than that to q, nor to a point whose
// column lies further out.  So once some candidate of the window is at
// distance r, only candidates within
//     m = r (W/2) max|n| / w
// columns of X(p) can be as near; likewise for rows.  The first strict
// minimum of that rectangle is the first strict minimum of the window: the
// candidates left out are strictly further away.  kx, ky hold (W/2) max|n| and
// (H/2) max|n| over the target's columns and rows; r is widened by 1e-5 (the
// rounding of len^2) and by eps |p|_1 + eps0 (metres: the roundings of the
// target's points, of proj and of p's projection), m by 0.1% and a fiftieth of
// a pixel.  Sources nearer than w_min to the eye plane (points behind the eye
// project too), windows that wrap past the target's width into the next row
// (:110) and targets without the property search the whole window.
struct Prune {
    float kx, ky, eps, eps0, w_min;
    float lo_x, hi_x, lo_y, hi_y;
    bool on;
};

// A point as two packed float pairs (x, y), (z, w); target points have w = 1.
struct alignas(16) Packed {
    unsigned long long xy, zw;
};
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// Squared distance of a candidate and a source in the reference's order,
// (dx^2 + dy^2) + (dz^2 + dw^2): two packed subtractions and two packed
// squares (f32x2: each half rounded as the scalar operation), three adds.  A
// square is fma(d, d, -0) with the -0 a kernel parameter: the rounded product
// for every input (x + -0 = x, also for x = -0), which unlike a packed
// multiply ptxas does not fuse into the add that consumes it.
__device__ __forceinline__ float len2(const Packed& q, const Packed& p, unsigned long long nz) {
    unsigned long long a, b;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(a) : "l"(q.xy), "l"(p.xy));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(b) : "l"(q.zw), "l"(p.zw));
    asm("fma.rn.f32x2 %0, %0, %0, %1;" : "+l"(a) : "l"(nz));
    asm("fma.rn.f32x2 %0, %0, %0, %1;" : "+l"(b) : "l"(nz));
    float xx, yy, zz, ww;
    f2_unpack(a, xx, yy);
    f2_unpack(b, zz, ww);
    return fadd(fadd(xx, yy), fadd(zz, ww));
}

// A tile while its sources' windows are searched: the sources whose rectangles
// are searched by all threads, and their rows.
struct Rect {
    long long first;  // its first candidate's index in the staging buffer or the target
    int stride;       // of its rows there; negative in the target
    int number;       // the first candidate's number r * 32 + c << 8 | columns
};
constexpr int kItems = 21 * kTileThreads;  // every row of every window
template <int kS>
struct TileList {  // per thread: kHalves to a source
    static constexpr int kThreads = kTileThreads * kHalves<kS>;
    Packed p[kThreads];               // world point
    Rect rect[kThreads];
    unsigned short item[kItems];      // rows to search: thread << 5 | row
    unsigned long long key[kThreads]; // best so far: len^2 bits << 32 | candidate number
};
template <>
struct TileList<kWhole> {
    float rec[7][kTileThreads];
    unsigned long long key[2 * kTileThreads];
};
// The tile's dynamic shared memory: the staged float4s and the list, whose start
// the sources' records take after the search -- per source p xyz, q xyz, len^2
// (zeros when no pair).  Planes of a whole-window scan reach over both, up to
// the keys.
template <int kS>
constexpr size_t kStageBytes = kS == kWhole ? 5120 * 12 : kStagePixels<kS> * sizeof(float4);
template <int kS>
constexpr size_t kTileBytes = kStageBytes<kS> + sizeof(TileList<kS>);
template <int kS>
constexpr int kPlanePixels =
    (int)((kStageBytes<kS> + (kS == kWhole ? 0 : offsetof(TileList<kS>, key))) / 12) & ~1;
struct SearchSmem {
    unsigned int n_items;
    int box[4];      // the tile's rectangles: x0, y0, x1, y1
    int cbox[4];     // and projections (or windows)
    int pred[4];     // the region staged ahead: x0, y0, w, h
    int ahead_whole; // as planes, for a whole-window scan
    unsigned int area;  // the cost of the rectangles, in candidates, of the warp that has the most
    FF acc[17];      // the CTA's moments (index 0 unused: count)
    unsigned int count;
};
// Whether the tile's next step scans whole windows: where the rectangles of one of
// its warps hold more than 5/16 of the windows' candidates (a step is as long as
// the slowest warp, not as the average).  The whole-window scan reads two
// candidates at a time with no bounds or boxes before it, and all of a warp's
// lanes alike; with fast motion a tile of large rectangles holds up its whole step.
// The share is the step's own after a search, and after a scan what the distances
// to the winners would leave.  Times, us, of 15 steps, windows only where a
// launch's shape says so / by tile: 640x480, frames one apart 423 / 345, three
// apart 461 / 422; 512x424 411 / 315, 452 / 395; 1024x848 626 / 459, 724 / 576;
// tracking at 640x480, ten frames 5290 / 4990.  4/16: the closed loop 2130 ->
// 2170 us; 6/16 and 8/16: three apart 459 and more.
constexpr unsigned int kWholeShare = 5;  // sixteenths
__device__ __forceinline__ int whole_next(const SearchSmem& ss) { return ss.area > 441u * 32u * kWholeShare / 16u; }
// What part of the target a tile has staged: pixels [x0, x1) x [y0, y1).
struct Region {
    int buf;  // its first pixel's index in the CTA's staging buffer
    int x0, y0, x1, y1, pitch;
    __device__ __forceinline__ int at(int x, int y) const { return buf + (y - y0) * pitch + (x - x0); }
    __device__ __forceinline__ bool holds(int x, int y, int cols, int rows) const {
        return x >= x0 && y >= y0 && x + cols <= x1 && y + rows <= y1;
    }
};

constexpr unsigned long long kNoPair = (unsigned long long)0x3c23d70au << 32;  // len^2 = 0.01f, candidate 0

// The tile's staged region (dynamic shared memory).
extern __shared__ float4 stage_all[];

// A target point in the staging buffer or in the target itself.
template <bool kStaged>
__device__ __forceinline__ Packed target_at(const float4* __restrict__ synth, long long i) {
    if (kStaged) return *reinterpret_cast<const Packed*>(stage_all + (int)i);
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(synth + i));
    return Packed{v.x, v.y};
}

// The first strict minimum of `cols` candidates from index i on: four at a
// time, then the rest three at a time (past the row's end its last one again,
// which cannot win).
template <bool kStaged>
__device__ __forceinline__ void scan_row(const float4* __restrict__ synth, long long i, int cols, const Packed& p,
                                         unsigned long long nz, float& best, int& at, int number) {
    int c = 0;
    for (; c + 8 <= cols; c += 4) {
        float l2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) l2[k] = len2(target_at<kStaged>(synth, i + c + k), p, nz);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (l2[k] < best) {
                best = l2[k];
                at = number + c + k;
            }
    }
    for (; c < cols; c += 3) {
        float l2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) l2[k] = len2(target_at<kStaged>(synth, i + min(c + k, cols - 1)), p, nz);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (l2[k] < best) {
                best = l2[k];
                at = number + c + k;
            }
    }
}

__device__ __forceinline__ unsigned long long f2_sub(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2_sq(unsigned long long a, unsigned long long neg_zero) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(a), "l"(neg_zero));
    return d;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The whole-window scan of a thread's rows (`base`: its first candidate's plane
// index).  A row is 21 wide (past the window's clamp at 640 columns the planes
// hold no points): ten aligned pairs of adjacent candidates, whose
// squared distances are formed two at a time (each half with the reference's
// operations and rounding), plus the one left over: the first when the window
// starts on an odd plane index, else the last.  Three chains -- the pairs' first
// halves, their second halves and the left-over ones -- keep their own first
// strict minimum; the lexicographic (len^2, candidate) minimum of the chains is
// the first strict minimum of the row-major scan.  Returns the best squared
// distance (0.01 when none) and its candidate number r * 32 + c (-1 when none).
// For sources with w = 1 (dz^2 + dw^2 == dz^2 exactly when dw == 0, as dz^2 >= 0).
__device__ __forceinline__ float scan_planes(const Planes& sp, int base, int pitch, int nr, float px, float py, float pz,
                                             float neg_zero, int* best_rc) {
    float b0 = 0.01f, b1 = 0.01f, b2 = 0.01f;
    int i0 = 0x7fffffff, i1 = 0x7fffffff, i2 = 0x7fffffff;
    const int o = base & 1;     // the pairs start at an even plane index
    const int cs = o ? 0 : 20;  // the left-over candidate's column
    const unsigned long long PX = f2_pack(px, px), PY = f2_pack(py, py), PZ = f2_pack(pz, pz);
    const unsigned long long NZ = f2_pack(neg_zero, neg_zero);
    for (int r = 0; r < nr; ++r, base += pitch) {
        // a candidate records only its pair number (a constant of the
        // unrolled row); the row and the parity are folded in once per row
        int c0 = -1, c1 = -1;
        const int pb = base + o;
#pragma unroll
        for (int k = 0; k < 10; ++k) {
            const int at = pb + 2 * k;
            const unsigned long long X = *(const unsigned long long*)(sp.x + at);
            const unsigned long long Y = *(const unsigned long long*)(sp.y + at);
            const unsigned long long Z = *(const unsigned long long*)(sp.z + at);
            const unsigned long long dx = f2_sub(X, PX), dy = f2_sub(Y, PY), dz = f2_sub(Z, PZ);
            const unsigned long long l2 = f2_add(f2_add(f2_sq(dx, NZ), f2_sq(dy, NZ)), f2_sq(dz, NZ));
            float lo, hi;
            f2_unpack(l2, lo, hi);
            if (lo < b0) {
                b0 = lo;
                c0 = 2 * k;
            }
            if (hi < b1) {
                b1 = hi;
                c1 = 2 * k;
            }
        }
        const int r32 = r * 32;
        {  // one candidate in scalar float, the reference's order: (dx^2 + dy^2) + dz^2
            const int at = base + cs;
            const float dx = fsub(sp.x[at], px), dy = fsub(sp.y[at], py), dz = fsub(sp.z[at], pz);
            const float l2 = fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz));
            if (l2 < b2) {
                b2 = l2;
                i2 = r32 + cs;
            }
        }
        if (c0 >= 0) i0 = r32 + o + c0;
        if (c1 >= 0) i1 = r32 + o + c1 + 1;
    }
    if (b1 < b0 || (b1 == b0 && i1 < i0)) {
        b0 = b1;
        i0 = i1;
    }
    if (b2 < b0 || (b2 == b0 && i2 < i0)) {
        b0 = b2;
        i0 = i2;
    }
    *best_rc = i0 == 0x7fffffff ? -1 : i0;
    return b0;
}

// Any rows of a window in the target itself, one candidate at a time: where the
// windows are not staged (they span too much), and for sources with w != 1.
__device__ __noinline__ unsigned long long scan_target(const float4* __restrict__ synth, long long n_synth, int synth_w,
                                                       int u, int v, int r0, int r1, int nc, float px, float py, float pz,
                                                       float pw) {
    const float dw = fsub(1.0f, pw), dw2 = fmul(dw, dw);
    float best = 0.01f;
    int rc = -1;
    for (int r = r0; r < r1; ++r)
#pragma unroll 3
        for (int c = 0; c < nc; ++c) {
            const long long at = (long long)(v + r) * synth_w + (u + c);
            if (at >= n_synth) break;
            const float4 q = __ldg(synth + at);
            const float dx = fsub(q.x, px), dy = fsub(q.y, py), dz = fsub(q.z, pz);
            const float l2 = fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fadd(fmul(dz, dz), dw2));
            if (l2 < best) {
                best = l2;
                rc = r * 32 + c;
            }
        }
    return rc < 0 ? kNoPair : (unsigned long long)__float_as_uint(best) << 32 | (unsigned int)rc;
}

// A thread's rows of its window, all candidates, in the staged planes (whose pitch
// is 0 where they are not staged; `base`: its first candidate's plane index).
constexpr int kSplitRow = 10;  // of two threads, the first takes window rows [0, 10)
template <int kH>
__device__ __forceinline__ unsigned long long search_whole(const IcpArgs& a, const Planes& planes, int pitch, int base,
                                                           int nr, int nc, int u, int v, const float (&p)[4], int half) {
    const int r0 = kH == 2 && half ? kSplitRow : 0, r1 = kH == 2 && !half ? min(nr, kSplitRow) : nr;
    if (r1 <= r0) return kNoPair;
    if (!pitch || p[3] != 1.0f)
        return scan_target(a.synth, (long long)a.synth_w * a.synth_h, a.synth_w, u, v, r0, r1, nc, p[0], p[1], p[2], p[3]);
    int rc = -1;
    const float best = scan_planes(planes, base + r0 * pitch, pitch, r1 - r0, p[0], p[1], p[2], a.neg_zero, &rc);
    return rc < 0 ? kNoPair : (unsigned long long)__float_as_uint(best) << 32 | (unsigned int)(rc + r0 * 32);
}

// The search of a source's window [nr x nc] (first candidate: target pixel
// (u, v)) by its own thread.  It bounds the distance to the nearest candidate,
// cuts the window down to the rectangle that can win and, where that is still
// large (fast motion, a depth edge), to the blocks of 8 x 4 target pixels
// whose bounding boxes are near enough (bound_own); it scans the rectangle in the
// reference's row-major order, in the staged region where that holds it, else
// in the target itself (scan_own).  A rectangle far above its warp's average goes onto
// the tile's list row by row, for all threads (search_items).  (cr, cc): the
// candidate the source projects to; X, Y, w: its projected column and row
// coordinate (upwards) and clip w; (hr, hc): a candidate likely to be near
// (-1: none), the last winner or the pixel nearest to it in a window that has
// moved past it.  Where the rectangles leave the staged region, all of a tile's
// are staged instead, if they fit (from global memory a few dozen of them take
// longer than the step: 15 steps at 640x480 with frames three apart 446 -> 422 us).
// Returns the best key so far; by whole warps.  Measured at
// 640x480: 10-40 candidates per source instead of 441 after the first two
// steps, an alignment of 15 steps 334 us (433 us with the whole windows); the
// step is then held by its serial parts -- the projection, the moments, the
// last CTA's totals and Horn solve, about 11 of 16 us -- and by the tile with
// the most candidates.
constexpr int kOwnArea = 32;    // rectangles up to this, and up to 1.5 times the warp's average, are scanned by their thread
constexpr int kBoxArea = 72;    // rectangles above this are cut down by the blocks' boxes,
constexpr int kBoxCost = 4;     // of which one takes about as long as this many candidates
struct OwnRect {
    int r0, rows, c0, cols;
    bool wraps;  // reads on in the next row of the target
};
template <int kS, bool kRects>
__device__ __forceinline__ OwnRect bound_own(const IcpArgs& a, const Region& reg, int nr, int nc, int cr, int cc, int hr,
                                             int hc, bool first, int u, int v, float X, float Y, float w,
                                             const Prune& pr, const float (&p)[4], int half, SearchSmem& ss) {
    constexpr int kH = kHalves<kS>;
    const int W = a.synth_w, H = a.synth_h;
    const Packed pp{f2_pack(p[0], p[1]), f2_pack(p[2], p[3])};
    const unsigned long long nz = f2_pack(a.neg_zero, a.neg_zero);
    auto pixel_len2 = [&](int x, int y) {
        const Packed q = reg.holds(x, y, 1, 1) ? target_at<true>(nullptr, reg.at(x, y))
                                               : target_at<false>(a.synth, (long long)y * W + x);
        return len2(q, pp, nz);
    };
    // the distance bound.  From the second step on the pixel that won the
    // step before is usually within a pixel of the new winner; in the first
    // one, the 3 x 3 candidates around the projection and, when the source is
    // still five pixels' distance and more from them, every fifth candidate of
    // the window's rows and columns.
    const int nrt = min(nr, H - v), nct = min(nc, W - u);  // the window's part inside the target
    float b = 0.01f;
    if (hr >= 0 && hr < nrt && hc < nct) {
        const float l2 = pixel_len2(u + hc, v + hr);
        if (l2 < b) b = l2;
    }
    if (first) {
        float l2[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int r = cr + k / 3 - 1, c = cc + k % 3 - 1;
            l2[k] = 1.0f;
            if (r >= 0 && c >= 0 && r < nrt && c < nct) l2[k] = pixel_len2(u + c, v + r);
        }
#pragma unroll
        for (int k = 0; k < 9; ++k)
            if (l2[k] < b) b = l2[k];
        if (b * pr.kx * pr.kx > 25.0f * w * w) {
            const int rs = cr >= 10 ? cr - 10 : 0, cs = cc >= 10 ? cc - 10 : 0;
            const bool all = reg.holds(u + cs, v + rs, max(nct - cs, 0), max(nrt - rs, 0));
            for (int r = rs; r < nrt; r += 5)
                for (int c = cs; c < nct; c += 5) {
                    const float g = all ? len2(target_at<true>(nullptr, reg.at(u + c, v + r)), pp, nz)
                                        : pixel_len2(u + c, v + r);
                    if (g < b) b = g;
                }
        }
    }
    int r0 = 0, rows = nr, c0 = 0, cols = nc;
    if (pr.on && w > pr.w_min && nr > 0) {
        const float r = sqrtf(b) * 1.00001f + (pr.eps * (fabsf(p[0]) + fabsf(p[1]) + fabsf(p[2])) + pr.eps0);
        const float s = __fdividef(r * 1.001f, w);
        const float mx = fmaf(pr.kx, s, 0.02f + 1e-5f * fabsf(X)), my = fmaf(pr.ky, s, 0.02f + 1e-5f * fabsf(Y));
        // a window past the target's width reads on in the next row, whose
        // first columns are the ones to exclude then
        const int wrap = u + nc - W;
        if (wrap <= 0 || X - mx - pr.hi_x > (float)wrap) {
            const int nc1 = wrap > 0 ? nc - wrap : nc;
            // columns x + lo <= X + mx, x + hi >= X - mx; column 0 also takes what truncates to it from below
            const int x0 = (int)ceilf(fminf(fmaxf(X - mx - pr.hi_x, (float)u), (float)(u + nc)));
            const int x1 = max((int)floorf(fmaxf(fminf(X + mx - pr.lo_x, (float)(u + nc1 - 1)), (float)u - 1.0f)), 0);
            // rows count downwards: row y has coordinate t = H - 1 - y
            const float tv0 = (float)(H - 1 - (v + nr - 1)), tv1 = (float)(H - 1 - v);
            const int t0 = (int)ceilf(fminf(fmaxf(Y - my - pr.hi_y, tv0), tv1 + 1.0f));
            const int t1 = max((int)floorf(fmaxf(fminf(Y + my - pr.lo_y, tv1), tv0 - 1.0f)), 0);
            c0 = x0 - u;
            cols = min(x1 - u, nc1 - 1) - c0 + 1;
            r0 = max(H - 1 - t1 - v, 0);
            rows = min(H - 1 - t0 - v, nr - 1) - r0 + 1;
        }
    }
    rows = min(rows, H - v - r0);  // past the target's last row there is nothing
    if (kH == 2 && rows > 0) {     // this half's rows
        const int mid = (rows + 1) >> 1;
        r0 += half ? mid : 0;
        rows = half ? rows - mid : mid;
    }
    if (rows <= 0 || cols <= 0) rows = cols = 0;
    const bool wraps = u + c0 + cols > W;
    int boxes = 0;  // looked at
    if (rows * cols > kBoxArea && !wraps) {  // (blocks do not follow a window into the next row)
        // the rectangle of the blocks no further than the bound (with the roundings covered)
        const int nbx = (W + kBlockW - 1) / kBlockW;
        const int x0 = u + c0, y0 = v + r0, bx1 = (x0 + cols - 1) >> 3, by1 = (y0 + rows - 1) >> 2;
        const float far = b * 1.00001f;
        boxes = (bx1 - (x0 >> 3) + 1) * (by1 - (y0 >> 2) + 1);
        int mx0 = bx1 + 1, mx1 = -1, my0 = by1 + 1, my1 = -1;
        for (int by = y0 >> 2; by <= by1; ++by)
            for (int bx = x0 >> 3; bx <= bx1; ++bx) {
                const float4* q = a.boxes + 2 * ((size_t)by * nbx + bx);
                const float4 lo = __ldg(q), hi = __ldg(q + 1);
                const float dx = fmaxf(fmaxf(lo.x - p[0], p[0] - hi.x), 0.0f);
                const float dy = fmaxf(fmaxf(lo.y - p[1], p[1] - hi.y), 0.0f);
                const float dz = fmaxf(fmaxf(lo.z - p[2], p[2] - hi.z), 0.0f);
                if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= far) {
                    mx0 = min(mx0, bx);
                    mx1 = max(mx1, bx);
                    my0 = min(my0, by);
                    my1 = max(my1, by);
                }
            }
        const int nx0 = max(x0, mx0 * kBlockW), nx1 = min(x0 + cols, (mx1 + 1) * kBlockW);
        const int ny0 = max(y0, my0 * kBlockH), ny1 = min(y0 + rows, (my1 + 1) * kBlockH);
        c0 = nx0 - u;
        cols = nx1 - nx0;
        r0 = ny0 - v;
        rows = ny1 - ny0;
        if (rows <= 0 || cols <= 0) rows = cols = 0;  // no block near enough
    }
    const int n = rows * cols, x0 = u + c0, y0 = v + r0;
    {  // the region the next step will want
        const int bx0 = (int)__reduce_min_sync(0xffffffffu, n ? (unsigned)x0 : 0x7fffffffu);
        const int by0 = (int)__reduce_min_sync(0xffffffffu, n ? (unsigned)y0 : 0x7fffffffu);
        const int bx1 = __reduce_max_sync(0xffffffffu, n ? x0 + cols : -1);
        const int by1 = __reduce_max_sync(0xffffffffu, n ? y0 + rows : -1);
        if ((threadIdx.x & 31) == 0 && bx1 >= 0) {
            atomicMin(&ss.box[0], bx0);
            atomicMin(&ss.box[1], by0);
            atomicMax(&ss.box[2], bx1);
            atomicMax(&ss.box[3], by1);
        }
    }
    if constexpr (!kRects) {  // for whole_next
        const unsigned int cost = __reduce_add_sync(0xffffffffu, (unsigned int)(n + kBoxCost * boxes));
        if ((threadIdx.x & 31) == 0) atomicMax(&ss.area, cost * kH);
    }
    return OwnRect{r0, rows, c0, cols, wraps};
}
template <int kS>
__device__ __forceinline__ unsigned long long scan_own(const IcpArgs& a, const Region& reg, const OwnRect& own, int u,
                                                       int v, const float (&p)[4], SearchSmem& ss, TileList<kS>& list,
                                                       bool& listed) {
    const int W = a.synth_w, H = a.synth_h;
    const Packed pp{f2_pack(p[0], p[1]), f2_pack(p[2], p[3])};
    const unsigned long long nz = f2_pack(a.neg_zero, a.neg_zero);
    const int r0 = own.r0, rows = own.rows, c0 = own.c0, cols = own.cols, n = rows * cols, x0 = u + c0, y0 = v + r0;
    const bool wraps = own.wraps;
    // (a warp's own rectangles, of vertical neighbours, read shared memory
    // without conflicts; the list's rows do not)
    const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned int)n);
    const int most = max(kOwnArea, total * 3 >> 6);
    const bool in = reg.holds(x0, y0, cols, rows);
    const int number = r0 * 32 + c0;
    if (n > most && !wraps) {
        listed = true;
        const int me = threadIdx.x;
        list.p[me] = pp;
        list.rect[me] = in ? Rect{reg.at(x0, y0), reg.pitch, number << 8 | cols}
                              : Rect{(long long)y0 * W + x0, -W, number << 8 | cols};
        list.key[me] = kNoPair;
        const unsigned int i0 = atomicAdd(&ss.n_items, (unsigned int)rows);
        for (int r = 0; r < rows; ++r) list.item[i0 + r] = (unsigned short)(me << 5 | r);
        return kNoPair;
    }
    float best = 0.01f;
    int brc = -1;
    if (in) {  // (a staged region has no points past the target's end)
        int i = reg.at(x0, y0);
        for (int r = 0; r < rows; ++r, i += reg.pitch) scan_row<true>(nullptr, i, cols, pp, nz, best, brc, number + r * 32);
    } else {  // (a wrapped window's last columns may lie past the target's end)
        long long i = (long long)y0 * W + x0;
        for (int r = 0; r < rows; ++r, i += W)
            scan_row<false>(a.synth, i, (int)min((long long)cols, (long long)W * H - i), pp, nz, best, brc,
                            number + r * 32);
    }
    return brc < 0 ? kNoPair : (unsigned long long)__float_as_uint(best) << 32 | (unsigned int)brc;
}

// The listed rows, dealt out to the CTA's threads; a source's key takes the
// lexicographic (len^2, candidate number) minimum, the first strict minimum
// in row-major order.
template <int kS>
__device__ __forceinline__ void search_items(const float4* __restrict__ synth, unsigned int n_items, float neg_zero,
                                             TileList<kS>& list) {
    const unsigned long long nz = f2_pack(neg_zero, neg_zero);
    for (unsigned int i = threadIdx.x; i < n_items; i += TileList<kS>::kThreads) {
        const int it = list.item[i], s = it >> 5, row = it & 31;
        const Packed p = list.p[s];
        const Rect rect = list.rect[s];
        float best = 0.01f;
        int at = -1;
        const int cols = rect.number & 0xff, number = (rect.number >> 8) + row * 32;
        if (rect.stride > 0)
            scan_row<true>(nullptr, (int)rect.first + row * rect.stride, cols, p, nz, best, at, number);
        else
            scan_row<false>(synth, rect.first - (long long)row * rect.stride, cols, p, nz, best, at, number);
        if (at >= 0) atomicMin(&list.key[s], (unsigned long long)__float_as_uint(best) << 32 | (unsigned int)at);
    }
}

__device__ __noinline__ void finish_step(IcpState* __restrict__ st, const FF* __restrict__ tot,
                                        IcpPoseMail* mail, unsigned long long mail_seq);

// One ICP::AlignStep (ICP.cpp:35-265) as one kernel.
//
// Association (:66-131): a CTA owns a tile of 8 source columns x 32 source
// rows, a thread one source (two threads where kHalves is 2), a warp 32 vertically adjacent ones.  Each thread
// back-projects and projects its source, the CTA stages the part of the
// target that the tile's searches will mostly read in shared memory, and
// bound_own, scan_own and search_items find each source's nearest candidate, the
// reference's first strict minimum.  Target pixel (y1, x1) is linear index y1 * synth_w + x1 as
// in the reference; indices past the buffer's end are invalid points.
//
// Horn's sums: instead of a second pass over the pairs for the centred
// cross-covariance (:169-197), the kernel accumulates the raw moments --
// count, sum p, sum q, sum p_r q_c (each product split exactly into a
// float-float pair by an FMA) and the squared distances -- in float-float
// per warp and CTA; the last CTA to finish totals them, forms the centroids
// and S = sum p q^T - (sum p) mu_q^T in float-float, and runs the Horn
// solve.  Algebraically this is the reference's two-pass sum; numerically it
// is more accurate than the reference's float Kahan sums.
constexpr int kMoments = 17;  // n, p xyz, q xyz, p q^T (9), len^2

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// floats as integers of the same order (atomicMin / atomicMax of any sign)
__device__ __forceinline__ int to_ordered(float f) {
    const int b = __float_as_int(f);
    return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }
constexpr float kMaxRange = 4.0f;  // pixels: a target whose points scatter further is searched whole

__device__ __forceinline__ FF two_prod(float a, float b) {
    const float p = fmul(a, b);
    return FF{p, __fmaf_rn(a, b, -p)};  // exact remainder of the product
}

// One AlignStep of one frame pair; `blk` / `nblk`: this CTA's index among
// the nblk CTAs that work on the pair (the launch's own grid, or a share of
// a batched launch over several pairs).
// kRects: rectangles only (a batch has tiles enough to hide a slow one).
template <int kS, bool kRects = false>
__device__ __forceinline__ void icp_step_body(const IcpArgs& a, IcpState* __restrict__ st, bool first,
                                              unsigned int blk, unsigned int nblk) {
    constexpr int kH = kHalves<kS>, kWarps = kH * kTileThreads / 32;
    static_assert(16 % kWarps == 0 && kMoments == 17, "one or two moments after the count per warp");
    static_assert(offsetof(TileList<kS>, key) >= 7 * kTileThreads * sizeof(float), "keys outlive the records' start");
    __shared__ SearchSmem ss;
    TileList<kS>& list = *reinterpret_cast<TileList<kS>*>(reinterpret_cast<unsigned char*>(stage_all) + kStageBytes<kS>);
    float(*const rec)[kTileThreads] = reinterpret_cast<float(*)[kTileThreads]>(&list);
    __shared__ unsigned int s_hint[kH == 2 ? kTileThreads : 1];  // the halves' common hints
    const int lane = threadIdx.x & 31, half = kH == 2 ? threadIdx.x / kTileThreads : 0;
    const int source = threadIdx.x % kTileThreads, warp = source >> 5;  // the tile's source, its column
    // Steps are launched programmatically behind one another: this grid may
    // start while the previous step's last CTA still updates the pose.  Wait
    // for that grid (and its memory) before touching the ICP state.
    const int n_cols = (a.width + 3) / 4;
    const int tiles_x = (n_cols + kTileCols - 1) / kTileCols;
    const int tiles = tiles_x * ((a.height + kTileRows - 1) / kTileRows);
    const size_t n_synth = (size_t)a.synth_w * a.synth_h;
    // While the previous step may still be finishing: stage the box that the
    // tile searched then, plus a margin -- little moves between steps.  The
    // box is read by one thread (it may be stale or half-updated; any box is
    // only a guess) and shared, so every thread stages the same region; after
    // the wait the guess is used if it holds every projection with a margin.
    const int tile0 = (int)blk;
    // this thread's depth and last winner (a hint: it may be older, any pixel will do)
    float pre_d = 0.0f;
    unsigned int pre_hint = ~0u;
    if (tile0 < tiles) {
        const int col = (tile0 % tiles_x) * kTileCols + warp, y = (tile0 / tiles_x) * kTileRows + lane;
        if (col < n_cols && y < a.height) {
            pre_d = load_depth(a.depth, (size_t)y * a.width + col * 4, a.depth_u16);
            if (!first && tile0 < kIcpMaxCtas) pre_hint = __ldcg(st->winner + tile0 * kTileThreads + source);
        }
    }
    const Planes planes{(float*)stage_all, (float*)stage_all + kPlanePixels<kS>,
                        (float*)stage_all + 2 * kPlanePixels<kS>};
    if (threadIdx.x == 0) {
        int p[4] = {0, 0, 0, 0};
        bool guess = !kRects;
        if (tile0 < tiles && tile0 < kIcpMaxCtas && (!kRects || !first)) {
            // (independent reads: one memory latency)
            const volatile IcpTile* t = st->tile + tile0;
            const int next_whole = t->whole;
            const int c0 = t->near[0], c1 = t->near[1], c2 = t->near[2], c3 = t->near[3];
            const int r0 = t->rect[0], r1 = t->rect[1], r2 = t->rect[2], r3 = t->rect[3];
            guess = kRects ? false : kS == kWhole || first || next_whole != 0;
            const int b0 = guess ? c0 : r0, b1 = guess ? c1 : r1, b2 = guess ? c2 : r2, b3 = guess ? c3 : r3;
            if (b2 > b0 && b3 > b1 && b0 >= 0 && b1 >= 0) {
                const int m = guess ? 10 + kWindowMargin : kPredMargin;
                const int x0 = max(b0 - m, 0), y0 = max(b1 - m, 0);
                const int w = b2 + m - x0, h = b3 + m - y0;
                const int most = guess ? kPlanePixels<kS> : kStagePixels<kS>;
                if (w <= most && h <= most && (guess ? plane_pitch(w) : stage_pitch(w)) * h <= most) {
                    p[0] = x0;
                    p[1] = y0;
                    p[2] = w;
                    p[3] = h;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ss.pred[k] = p[k];
            ss.box[k] = ss.cbox[k] = k < 2 ? 0x7fffffff : -1;
        }
        ss.ahead_whole = guess;
        ss.n_items = ss.count = ss.area = 0u;
    }
    if (threadIdx.x < kMoments) ss.acc[threadIdx.x] = FF{0.0f, 0.0f};
    __syncthreads();
    const int px0 = ss.pred[0], py0 = ss.pred[1], pw = ss.pred[2], ph = ss.pred[3];
    const bool ahead_whole = ss.ahead_whole != 0;
    if (pw > 0) {
        if (!kRects && (kS == kWhole || ahead_whole))
            stage_planes<kWarps>(planes, a.synth, n_synth, a.synth_w, px0, py0, pw, ph, plane_pitch(pw));
        else stage_region<kWarps>(stage_all, a.synth, n_synth, a.synth_w, px0, py0, pw, ph, stage_pitch(pw));
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float half_w = fmul((float)a.synth_w, 0.5f), half_h = fmul((float)a.synth_h, 0.5f);
    Prune pr;
    pr.kx = a.kx;
    pr.ky = a.ky;
    pr.eps = a.eps;
    pr.eps0 = a.eps0;
    pr.w_min = a.w_min;
    pr.lo_x = a.lo[0];
    pr.hi_x = a.hi[0];
    pr.lo_y = a.lo[1];
    pr.hi_y = a.hi[1];
    pr.on = a.prune != kPruneOff;
    if (a.prune == kPruneMeasured) {  // measured by k_target_range before the first step
        pr.lo_x = from_ordered(st->range[0]);
        pr.hi_x = from_ordered(st->range[1]);
        pr.lo_y = from_ordered(st->range[2]);
        pr.hi_y = from_ordered(st->range[3]);
        // (an empty target leaves lo > hi: nothing to find either way); within 2% of
        // their pixels, so that kx and ky, taken over 105% of the image, hold
        pr.on = pr.hi_x - pr.lo_x <= kMaxRange && pr.hi_y - pr.lo_y <= kMaxRange &&
                pr.lo_x >= -0.02f * a.synth_w && pr.hi_x <= 1.0f + 0.02f * a.synth_w &&
                pr.lo_y >= -0.02f * a.synth_h && pr.hi_y <= 1.0f + 0.02f * a.synth_h;
    }
    if (threadIdx.x == 0) atomicMin(&st->t_start, global_ns());
    float pose[16];  // four 16-byte loads of the new pose
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 c = reinterpret_cast<const float4*>(st->pose_f)[i];
        pose[4 * i] = c.x; pose[4 * i + 1] = c.y; pose[4 * i + 2] = c.z; pose[4 * i + 3] = c.w;
    }
    for (int tile = (int)blk; tile < tiles; tile += (int)nblk) {
        const bool ahead = tile == tile0;  // its region, depths and hints were loaded above
        // the tile's scan, as it found it best in the last step
        const bool whole = kRects ? false
                                  : kS == kWhole || first || !pr.on || tile >= kIcpMaxCtas ||
                                        (ahead ? ahead_whole : st->tile[tile].whole != 0);
        const int col = (tile % tiles_x) * kTileCols + warp, y = (tile / tiles_x) * kTileRows + lane;
        const bool mine = col < n_cols && y < a.height;
        float wp[4] = {0.f, 0.f, 0.f, 0.f};
        float X = 0.f, Y = 0.f, w = 0.f;
        unsigned int hint = ~0u;
        if (ahead) hint = pre_hint;
        else if (mine && !first && tile < kIcpMaxCtas) hint = st->winner[tile * kTileThreads + source];
        if (kH == 2 && half == 0) s_hint[source] = hint;  // (two reads of it may differ)
        int u = 0, v = 0, nr = 0, nc = 0, cc = 0, cr = 0;
        if (mine) {
            const int x = col * 4;
            const float d = ahead ? pre_d : load_depth(a.depth, (size_t)y * a.width + x, a.depth_u16);
            if (0.0f != d) {
                float pt[4], cl[4];
                pt[0] = fmul(fadd(fmul((float)x, a.fl_inv_x), a.pp_x), d);
                pt[1] = fmul(fadd(fmul(-(float)y, a.fl_inv_y), a.pp_y), d);
                pt[2] = fmul(fadd(fmul(-1.0f, 1.0f), 0.0f), d);
                pt[3] = 1.0f;
                mat_vec(pose, pt, wp);
                mat_vec(a.proj, wp, cl);
                const float ux = fdiv(cl[0], cl[3]), uy = fdiv(cl[1], cl[3]);
                X = fadd(fmul(ux, half_w), half_w);
                Y = fadd(fmul(uy, half_h), half_h);
                w = cl[3];
                const int cx = cvt_i32_x86(X), cy = wrap_sub(a.synth_h - 1, cvt_i32_x86(Y));
                u = max(0, wrap_sub(cx, 10));
                v = max(0, wrap_sub(cy, 10));
                nr = (int)min(480ll, (long long)v + 21) - v;
                nc = (int)min(640ll, (long long)u + 21) - u;
                if (nr <= 0 || nc <= 0) nr = nc = 0;
                cc = wrap_sub(cx, u);
                cr = wrap_sub(cy, v);
            }
        }
        stage_wait();  // the region staged ahead
        {  // the windows, or the projections inside them; one shared atomic per warp and bound
            const bool has = nr > 0;
            const int px = min(max(cc, 0), nc - 1) + u, py = min(max(cr, 0), nr - 1) + v;
            const int mu0 = (int)__reduce_min_sync(0xffffffffu, has ? (unsigned)(whole ? u : px) : 0x7fffffffu);
            const int mv0 = (int)__reduce_min_sync(0xffffffffu, has ? (unsigned)(whole ? v : py) : 0x7fffffffu);
            const int mu1 = __reduce_max_sync(0xffffffffu, has ? (whole ? u + 21 : px + 1) : -1);
            const int mv1 = __reduce_max_sync(0xffffffffu, has ? (whole ? v + nr : py + 1) : -1);
            if (lane == 0 && mu1 >= 0 && half == 0) {
                atomicMin(&ss.cbox[0], mu0);
                atomicMin(&ss.cbox[1], mv0);
                atomicMax(&ss.cbox[2], mu1);
                atomicMax(&ss.cbox[3], mv1);
            }
        }
        __syncthreads();
        const int ax0 = ss.cbox[0], ay0 = ss.cbox[1], ax1 = ss.cbox[2], ay1 = ss.cbox[3];
        // a tile whose windows are all empty (most of a frame wider than the
        // reference's 640 columns projects past them) has no pairs to search or sum
        if (ax1 < 0) {
            if (a.pairs && mine) {
                const size_t k = (size_t)y * n_cols + col;
                a.pairs[k] = -1ll;
                a.pairs_len2[k] = 0.01f;
            }
            __syncthreads();  // every thread has read the box before the next tile writes it
            continue;
        }
        Region reg{0, 0, 0, 0, 0, 1};  // the staged part of the target, for the search by rectangles
        unsigned long long key;
        int wx0 = ax0, wy0 = ay0, wpitch = 0;  // and for the scan of whole windows: its corner, its pitch (0: not staged)
        if (whole) {
            if (ahead && ahead_whole && pw > 0 && ax0 >= px0 && ay0 >= py0 && ax1 <= px0 + pw && ay1 <= py0 + ph) {
                wx0 = px0;
                wy0 = py0;
                wpitch = plane_pitch(pw);
            } else if (plane_pitch(ax1 - ax0) * (ay1 - ay0) <= kPlanePixels<kS>) {
                wpitch = plane_pitch(ax1 - ax0);
                stage_planes<kWarps>(planes, a.synth, n_synth, a.synth_w, ax0, ay0, ax1 - ax0, ay1 - ay0, wpitch);
                stage_wait();
                __syncthreads();
            }
            key = search_whole<kH>(a, planes, wpitch, (v - wy0) * wpitch + (u - wx0), nr, nc, u, v, wp, half);
            if (half) list.key[threadIdx.x] = key;
            if (threadIdx.x == 0 && tile < kIcpMaxCtas) {
                // where the projections lie in windows of 21, and a little more for the next step's rectangles
                IcpTile& t = st->tile[tile];
                const int b[4] = {ax0 + 10, ay0 + 10, max(ax1 - 10, ax0 + 11), max(ay1 - 10, ay0 + 11)};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t.near[k] = b[k];
                    t.rect[k] = b[k] + (k < 2 ? -kUseMargin : kUseMargin);
                }
            }
            __syncthreads();
        } else if constexpr (kS != kWhole) {
            // the region staged ahead if it holds every projection of the tile with a
            // margin, else the projections with as much of the windows around them as
            // fits; where the target's points are off their pixels' centres, as far off
            // (in a batch, whose 80 registers that would spill, at the projections)
            const int sx = kRects ? 0 : __float2int_rn(0.5f * (pr.lo_x + pr.hi_x) - 0.5f);
            const int sy = kRects ? 0 : __float2int_rn(0.5f * (pr.lo_y + pr.hi_y) - 0.5f);
            const int bx0 = ax0 - sx, by0 = ay0 + sy, bx1 = ax1 - sx, by1 = ay1 + sy;
            if (ahead && !ahead_whole && pw > 0 && max(bx0 - kUseMargin, 0) >= px0 && max(by0 - kUseMargin, 0) >= py0 &&
                min(bx1 + kUseMargin, 640) <= px0 + pw && min(by1 + kUseMargin, 480) <= py0 + ph) {
                reg = Region{0, px0, py0, px0 + pw, py0 + ph, stage_pitch(pw)};
            } else {
                for (int m = 10; m >= 0; m -= m > 4 ? 3 : 1) {
                    const int x0 = max(bx0 - m, 0), y0 = max(by0 - m, 0);
                    const int w0 = min(bx1 + m, 640) - x0, h0 = min(by1 + m, 480) - y0;
                    if (w0 <= 0 || h0 <= 0 || stage_pitch(w0) * h0 > kStagePixels<kS>) continue;
                    reg = Region{0, x0, y0, x0 + w0, y0 + h0, stage_pitch(w0)};
                    stage_region<kWarps>(stage_all, a.synth, n_synth, a.synth_w, x0, y0, w0, h0, reg.pitch);
                    stage_wait();
                    __syncthreads();
                    break;
                }
            }
            if (kH == 2) hint = s_hint[source];
            // (where the window has moved past it, the window's nearest pixel)
            const int hr = hint == ~0u ? -1 : min(max((int)(hint >> 16) - v, 0), nr - 1);
            const int hc = hint == ~0u ? -1 : min(max((int)(hint & 0xffffu) - u, 0), nc - 1);
            const OwnRect own = bound_own<kS, kRects>(a, reg, nr, nc, cr, cc, hr, hc, first || tile >= kIcpMaxCtas, u, v,
                                                      X, Y, w, pr, wp, half, ss);
            if constexpr (!kRects) {  // rectangles beyond the staged region: those of all sources, if they fit
                __syncthreads();
                const int x0 = ss.box[0], y0 = ss.box[1], w0 = ss.box[2] - x0, h0 = ss.box[3] - y0;
                if (ss.box[2] >= 0 && !reg.holds(x0, y0, w0, h0) && stage_pitch(w0) * h0 <= kStagePixels<kS>) {
                    reg = Region{0, x0, y0, x0 + w0, y0 + h0, stage_pitch(w0)};
                    stage_region<kWarps>(stage_all, a.synth, n_synth, a.synth_w, x0, y0, w0, h0, reg.pitch);
                    stage_wait();
                    __syncthreads();
                }
            }
            bool listed = false;
            key = scan_own<kS>(a, reg, own, u, v, wp, ss, list, listed);
            if (half && !listed) list.key[threadIdx.x] = key;  // for the source's first thread
            __syncthreads();
            const unsigned int n_items = ss.n_items;
            if (threadIdx.x == 0 && tile < kIcpMaxCtas && ss.box[2] >= 0) {
                IcpTile& t = st->tile[tile];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t.near[k] = k == 0 ? ax0 : k == 1 ? ay0 : k == 2 ? ax1 : ay1;
                    t.rect[k] = ss.box[k];
                }
                if constexpr (!kRects) t.whole = whole_next(ss);
            }
            if (n_items) {
                search_items<kS>(a.synth, n_items, a.neg_zero, list);
                __syncthreads();
                if (listed) key = list.key[threadIdx.x];
                __syncthreads();  // the records take the list's place
            }
        }
        if (kH == 2 && !half) key = min(key, list.key[threadIdx.x + kTileThreads]);
        const bool out = mine && half == 0;  // the source's pair is its first thread's
        const bool hit = out && key < kNoPair;
        const float best = __uint_as_float((unsigned int)(key >> 32));
        const int rc = (int)(unsigned int)key;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (hit) {
            const int x = u + (rc & 31), yy = v + (rc >> 5);
            if (wpitch) {
                const int at = (yy - wy0) * wpitch + (x - wx0);
                q = make_float4(planes.x[at], planes.y[at], planes.z[at], 1.0f);
            } else q = reg.holds(x, yy, 1, 1) ? stage_all[reg.at(x, yy)] : __ldg(a.synth + (size_t)yy * a.synth_w + x);
        }
        if (out && tile < kIcpMaxCtas)
            st->winner[tile * kTileThreads + source] = hit ? (unsigned int)(v + (rc >> 5)) << 16 | (u + (rc & 31)) : ~0u;
        if (kS != kWhole && whole && pr.on) {  // what the next step's rectangles may hold, from the distance now
            unsigned int n = nr * nc;
            if (hit && w > pr.w_min) {
                const float r = __fdividef(sqrtf(best), w);
                n = (unsigned int)(fminf(fmaf(2.0f * pr.kx, r, 1.5f), (float)nc) * fminf(fmaf(2.0f * pr.ky, r, 1.5f), (float)nr));
            }
            const unsigned int total = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0 && half == 0) atomicMax(&ss.area, total);
        }
        if (a.pairs && out) {
            const size_t k = (size_t)y * n_cols + col;
            a.pairs[k] = hit ? (long long)(v + (rc >> 5)) * a.synth_w + (u + (rc & 31)) : -1ll;
            a.pairs_len2[k] = hit ? best : 0.01f;
        }
        if (kS != kWhole && whole) {
            __syncthreads();  // the records take the planes' end
            if (threadIdx.x == 0 && tile < kIcpMaxCtas) st->tile[tile].whole = !pr.on || whole_next(ss);
        }
        // this source's pair for the tile's moments (zeros when none)
        if (half == 0) {
            const int sidx = source;
            rec[0][sidx] = hit ? wp[0] : 0.f;
            rec[1][sidx] = hit ? wp[1] : 0.f;
            rec[2][sidx] = hit ? wp[2] : 0.f;
            rec[3][sidx] = q.x;
            rec[4][sidx] = q.y;
            rec[5][sidx] = q.z;
            rec[6][sidx] = hit ? best : 0.f;
            const unsigned int nh = __popc(__ballot_sync(0xffffffffu, hit));
            if (lane == 0 && nh) atomicAdd(&ss.count, nh);
        }
        __syncthreads();
        if (threadIdx.x == 0) {  // for the next tile
#pragma unroll
            for (int k = 0; k < 4; ++k) ss.box[k] = ss.cbox[k] = k < 2 ? 0x7fffffff : -1;
            ss.n_items = ss.area = 0u;
        }
        // the tile's raw moments: each warp reduces two of the 16 over all
        // sources (lane l takes sources l, l + 32, ...), in float-float
        {
            constexpr int kPer = 16 / kWarps;
            const int w0 = threadIdx.x >> 5;
            FF acc[kPer];
#pragma unroll
            for (int h = 0; h < kPer; ++h) {
                const int c = w0 + 1 + kWarps * h;
                acc[h] = FF{0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < kTileCols; ++k) {
                    const int sidx = lane + 32 * k;
                    FF m;
                    if (c < 7) m = FF{rec[c - 1][sidx], 0.0f};
                    else if (c < 16) m = two_prod(rec[(c - 7) / 3][sidx], rec[3 + (c - 7) % 3][sidx]);
                    else m = FF{rec[6][sidx], 0.0f};
                    acc[h] = ff_add(acc[h], m);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)  // the trees side by side
#pragma unroll
                for (int h = 0; h < kPer; ++h) {
                    const FF x{__shfl_xor_sync(0xffffffffu, acc[h].hi, o), __shfl_xor_sync(0xffffffffu, acc[h].lo, o)};
                    acc[h] = ff_add(acc[h], x);
                }
            if (lane < kPer) {
                const int c = w0 + 1 + kWarps * lane;
                ss.acc[c] = ff_add(ss.acc[c], lane ? acc[kPer - 1] : acc[0]);
            }
        }
        __syncthreads();  // staging buffer and records are reused by the next tile
    }
    // association done: the next step's grid may be scheduled (it waits above)
    asm volatile("griddepcontrol.launch_dependents;");
    if (threadIdx.x >= 1 && threadIdx.x < kMoments) {
        const FF t = ss.acc[threadIdx.x];
        st->part[(size_t)(2 * threadIdx.x) * kIcpMaxCtas + blk] = t.hi;
        st->part[(size_t)(2 * threadIdx.x + 1) * kIcpMaxCtas + blk] = t.lo;
    }
    if (threadIdx.x == 0) atomicMax(&st->t_body, global_ns());
    unsigned int n_total;
    if (!last_cta(&st->done, ss.count, &n_total, nblk)) return;
    __shared__ FF tot[kMoments];
    moments_total<kMoments, kWarps>(st, n_total, tot, (int)nblk);
    if (threadIdx.x < 32) finish_step(st, tot, a.mail, a.mail_seq);
}

template <int kS>
__global__ void __launch_bounds__(kTileThreads * kHalves<kS>, kResident<kS>) k_icp_step(IcpArgs a, IcpState* __restrict__ st, bool first) {
    icp_step_body<kS>(a, st, first, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------- Horn solve
// Cyclic Jacobi on a symmetric 4x4 (row-major) in double; V accumulates the
// rotations (columns are eigenvectors), the eigenvalues end in A[0..3].  The
// fallback for spectra whose largest eigenvalue is (nearly) repeated.
__device__ __noinline__ void jacobi4(double* A, double* V) {
    double a[16];
    for (int i = 0; i < 16; ++i) {
        a[i] = A[i];
        V[i] = (i % 5 == 0) ? 1.0 : 0.0;
    }
    double scale = 0.0;
    for (int i = 0; i < 16; ++i) scale += a[i] * a[i];
    // converged once the off-diagonal mass is below (1e-13)^2 of the total:
    // tighter bounds sit at double rounding noise and never terminate early
    for (int sweep = 0; sweep < 32; ++sweep) {
        double off = 0.0;
        for (int p = 0; p < 4; ++p)
            for (int q = p + 1; q < 4; ++q) off += a[4 * p + q] * a[4 * p + q];
        if (!(off > 1e-26 * scale)) break;
        for (int p = 0; p < 3; ++p)
            for (int q = p + 1; q < 4; ++q) {
                const double apq = a[4 * p + q];
                if (apq == 0.0) continue;
                const double theta = (a[4 * q + q] - a[4 * p + p]) / (2.0 * apq);
                const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < 4; ++k) {
                    const double akp = a[4 * k + p], akq = a[4 * k + q];
                    a[4 * k + p] = c * akp - s * akq;
                    a[4 * k + q] = s * akp + c * akq;
                }
                for (int k = 0; k < 4; ++k) {
                    const double apk = a[4 * p + k], aqk = a[4 * q + k];
                    a[4 * p + k] = c * apk - s * aqk;
                    a[4 * q + k] = s * apk + c * aqk;
                }
                for (int k = 0; k < 4; ++k) {
                    const double vkp = V[4 * k + p], vkq = V[4 * k + q];
                    V[4 * k + p] = c * vkp - s * vkq;
                    V[4 * k + q] = s * vkp + c * vkq;
                }
            }
    }
    for (int i = 0; i < 4; ++i) A[i] = a[5 * i];
}

// Horn's closed form (B. K. P. Horn, "Closed-form solution of absolute
// orientation using unit quaternions", JOSA A 4(4), 1987), written for one
// thread and without double precision: GB300 issues a double instruction
// (conversions included) at about one per 64 cycles per SM sub-partition,
// even for a single thread, and this tail runs on one SM while the others
// wait.  Precision comes from float-float (FF) arithmetic where it matters.
//
//  1. FF: centroids, the centred cross-covariance S = sum p q^T - (sum p)
//     mu_q^T (the raw moments cancel heavily) and Horn's symmetric N, scaled
//     by a power of two to unit size (exact).
//  2. float: the characteristic polynomial of N by the Faddeev-LeVerrier
//     recursion, its largest root by Newton's method from an upper bound of
//     the spectrum (Gershgorin or the Frobenius norm; right of the largest
//     root the polynomial is increasing and convex, so the iterates fall
//     monotonically onto it), and the largest diagonal entry j of
//     adj(N - lambda I), whose column j is then proportional to the
//     eigenvector.
//  3. FF: one step of Rayleigh-quotient inverse iteration -- rho = q'Nq / q'q,
//     q <- column j of adj(N - rho I) -- which converges cubically, so the
//     float-accurate start lands well below float rounding (two steps when
//     the eigen-gaps are small).
//  4. A spectrum whose gap product (the adjugate diagonal above) is tiny --
//     a nearly repeated largest eigenvalue -- goes to the double Jacobi
//     solver instead.
//
// R, t and the accumulated pose are FF as well; the float pose the next
// association uses is the FF pose rounded (its high part).
//
// Symmetric 4x4 matrices are held as their upper triangle, row by row.
__host__ __device__ constexpr int sym(int i, int j) {
    return i <= j ? (i * (7 - i)) / 2 + j : (j * (7 - j)) / 2 + i;
}
template <typename T>
__device__ __forceinline__ T shifted(const T* n, T s, int i, int j) {
    return i == j ? n[sym(i, i)] - s : n[sym(i, j)];
}
// determinant of rows r0..r2 and columns k0..k2 of N - s I
template <typename T>
__device__ __forceinline__ T minor3(const T* n, T s, int r0, int r1, int r2, int k0, int k1, int k2) {
    const T a00 = shifted(n, s, r0, k0), a01 = shifted(n, s, r0, k1), a02 = shifted(n, s, r0, k2);
    const T a10 = shifted(n, s, r1, k0), a11 = shifted(n, s, r1, k1), a12 = shifted(n, s, r1, k2);
    const T a20 = shifted(n, s, r2, k0), a21 = shifted(n, s, r2, k1), a22 = shifted(n, s, r2, k2);
    return a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) + a02 * (a10 * a21 - a11 * a20);
}
// column j of adj(N - s I) (the matrix is symmetric, so cofactor (i, j))
template <typename T>
__device__ __forceinline__ void adj_column(const T* n, T s, int j, T* q) {
    switch (j) {
        case 0:
            q[0] = minor3(n, s, 1, 2, 3, 1, 2, 3);
            q[1] = -minor3(n, s, 1, 2, 3, 0, 2, 3);
            q[2] = minor3(n, s, 1, 2, 3, 0, 1, 3);
            q[3] = -minor3(n, s, 1, 2, 3, 0, 1, 2);
            break;
        case 1:
            q[0] = -minor3(n, s, 0, 2, 3, 1, 2, 3);
            q[1] = minor3(n, s, 0, 2, 3, 0, 2, 3);
            q[2] = -minor3(n, s, 0, 2, 3, 0, 1, 3);
            q[3] = minor3(n, s, 0, 2, 3, 0, 1, 2);
            break;
        case 2:
            q[0] = minor3(n, s, 0, 1, 3, 1, 2, 3);
            q[1] = -minor3(n, s, 0, 1, 3, 0, 2, 3);
            q[2] = minor3(n, s, 0, 1, 3, 0, 1, 3);
            q[3] = -minor3(n, s, 0, 1, 3, 0, 1, 2);
            break;
        default:
            q[0] = -minor3(n, s, 0, 1, 2, 1, 2, 3);
            q[1] = minor3(n, s, 0, 1, 2, 0, 2, 3);
            q[2] = -minor3(n, s, 0, 1, 2, 0, 1, 3);
            q[3] = minor3(n, s, 0, 1, 2, 0, 1, 2);
            break;
    }
}
// out = n (p + c I); symmetric because p is a polynomial in n
__device__ __forceinline__ void sym_mul_shift(const float* n, const float* p, float c, float* out) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i; j < 4; ++j) {
            float t = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k) t = fmaf(n[sym(i, k)], k == j ? p[sym(k, j)] + c : p[sym(k, j)], t);
            out[sym(i, j)] = t;
        }
}

// Warp 0 of the last CTA of an AlignStep: from the totals of the raw
// moments, the centroids and S (ICP.cpp:166-197), N (:199-213), its dominant
// eigenvector (above), R and t (:215-256) and pose <- (T R) pose (:20-28).
// The work is spread over the lanes entry by entry -- centroids, S, N,
// the four minors and cofactors, R, t and the twelve pose entries -- and
// joined by shuffles; the float characteristic polynomial and its Newton
// search run on every lane alike.  Symmetric matrices indexed by a lane go
// through shared memory (a register array indexed by a lane would live in
// local memory).
__device__ __forceinline__ FF shfl_ff(FF v, int src) {
    return FF{__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src)};
}
// minor3 of rows {0..3} \ {rx} and columns {0..3} \ {cx} of n - s I, n in
// shared memory (upper triangle), for lane-dependent rx, cx
template <typename T>
__device__ __forceinline__ T minor_excl(const T* n, T s, int rx, int cx) {
    const int r0 = rx == 0 ? 1 : 0, r1 = rx <= 1 ? 2 : 1, r2 = rx <= 2 ? 3 : 2;
    const int k0 = cx == 0 ? 1 : 0, k1 = cx <= 1 ? 2 : 1, k2 = cx <= 2 ? 3 : 2;
    return minor3(n, s, r0, r1, r2, k0, k1, k2);
}
// N's entry k (upper triangle, row by row) as (S[i1] s2 S[i2]) s3 S[i3]:
// N = [[Sxx+Syy+Szz, Syz-Szy, Szx-Sxz, Sxy-Syx], [., Sxx-Syy-Szz, Sxy+Syx,
// Szx+Sxz], [., ., Syy-Sxx-Szz, Syz+Szy], [., ., ., Szz-Sxx-Syy]] (:199-213)
__device__ __forceinline__ void n_terms(int k, int& i1, int& i2, int& i3, bool& m2, bool& m3, bool& t3) {
    // per k (4 bits each): i1, i2, i3; flags: minus second, minus third, has third
    constexpr unsigned long long kI1 = 0x8546101650ull, kI2 = 0x0702343274ull, kI3 = 0x4080080008ull;
    constexpr unsigned int kM2 = 0x29e, kM3 = 0x290, kT3 = 0x291;
    i1 = (int)(kI1 >> (4 * k)) & 15;
    i2 = (int)(kI2 >> (4 * k)) & 15;
    i3 = (int)(kI3 >> (4 * k)) & 15;
    m2 = (kM2 >> k) & 1u;
    m3 = (kM3 >> k) & 1u;
    t3 = (kT3 >> k) & 1u;
}

__device__ __noinline__ void finish_step(IcpState* __restrict__ st, const FF* __restrict__ tot,
                                        IcpPoseMail* mail, unsigned long long mail_seq) {
    __shared__ float s_f[10];
    __shared__ FF s_nf[10];
    const int lane = threadIdx.x & 31;
    // the step's counters for the statistics, read now so that no load is
    // left behind the pose update (final: every CTA wrote them before its
    // release of the last-CTA counter)
    int step = 0;
    unsigned long long t_start = 0ull, t_body = 0ull;
    if (lane == 0) {
        step = __ldcg(&st->iter);
        t_start = __ldcg(&st->t_start);
        t_body = __ldcg(&st->t_body);
    }
    const int pk = lane < 12 ? lane : 0, pc = pk / 3, pr = pk - 3 * pc;  // the pose entry it will update ...
    FF P[4];                                                            // ... and its column, likewise read now
    {
        const float4 hi = __ldcg(reinterpret_cast<const float4*>(st->pose_f) + pc);
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(st->pose_lo) + pc);
        P[0] = FF{hi.x, lo.x};
        P[1] = FF{hi.y, lo.y};
        P[2] = FF{hi.z, lo.z};
        P[3] = FF{hi.w, lo.w};
    }
    // 1. centroids (lanes 0-5), S (lanes 0-8), N (lanes 0-9) in FF
    const float n = fadd(tot[0].hi, tot[0].lo);  // an exact count below 2^24
    FF my_mu{0.0f, 0.0f};
    if (lane < 6) {
        const float h = fdiv(tot[1 + lane].hi, n);
        const float r = fadd(__fmaf_rn(-h, n, tot[1 + lane].hi), tot[1 + lane].lo);  // exact remainder + lo
        my_mu = ff_norm(h, fdiv(r, n));
    }
    const int sl = lane < 9 ? lane : 0;
    const FF mu_c = shfl_ff(my_mu, 3 + sl % 3);
    const FF my_s = tot[7 + sl] - tot[1 + sl / 3] * mu_c;
    int i1, i2, i3;
    bool m2, m3, t3;
    n_terms(lane < 10 ? lane : 0, i1, i2, i3, m2, m3, t3);
    const FF a1 = shfl_ff(my_s, i1), a2 = shfl_ff(my_s, i2), a3 = shfl_ff(my_s, i3);
    FF my_n = m2 ? a1 - a2 : a1 + a2;
    if (t3) my_n = m3 ? my_n - a3 : my_n + a3;
    const bool diag = lane == 0 || lane == 4 || lane == 7 || lane == 9;
    float f2 = lane < 10 ? fmul(diag ? my_n.hi : 2.0f * my_n.hi, my_n.hi) : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f2 = fadd(f2, __shfl_xor_sync(0xffffffffu, f2, o));
    // power-of-two scale 2^-e/2 with f2 = m 2^e: N's Frobenius norm lands in [0.5, 1.5)
    const int e = ((__float_as_int(f2) >> 23) & 0xff) - 127;
    const float sc = __int_as_float((127 - (e >> 1)) << 23);
    const bool finite = f2 > 1e-30f && f2 < 1e30f;
    if (lane < 10) {
        s_nf[lane] = FF{my_n.hi * sc, my_n.lo * sc};
        s_f[lane] = my_n.hi * sc;
    }
    __syncwarp();
    float f[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) f[i] = s_f[i];
    // 2. float search (every lane)
    float gmax = -1e30f;  // Gershgorin: the largest row bound
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float t = f[sym(i, i)];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j != i) t += fabsf(f[sym(i, j)]);
        gmax = fmaxf(gmax, t);
    }
    // start just above the smaller of the Gershgorin and Frobenius bounds
    float l = fminf(gmax, sqrtf(f2 * sc * sc)) * 1.00001f + 1e-6f;
    float m[10], w[10];
    const float c3 = -(f[0] + f[4] + f[7] + f[9]);
    sym_mul_shift(f, f, c3, m);
    const float c2 = -0.5f * (m[0] + m[4] + m[7] + m[9]);
    sym_mul_shift(f, m, c2, w);
    const float c1 = -(w[0] + w[4] + w[7] + w[9]) * (1.0f / 3.0f);
    float tr = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) tr = fmaf(f[sym(i, k)], k == i ? w[sym(k, i)] + c1 : w[sym(k, i)], tr);
    const float c0 = -0.25f * tr;
    for (int it = 0; it < 32; ++it) {
        const float p = fmaf(fmaf(fmaf(l + c3, l, c2), l, c1), l, c0);
        const float dp = fmaf(fmaf(fmaf(4.0f, l, 3.0f * c3), l, 2.0f * c2), l, c1);
        if (!(dp > 0.0f)) break;
        const float step = __fdividef(p, dp);
        if (!(step > 0.0f)) break;
        l -= step;
        if (step <= 1e-7f * fabsf(l)) break;
    }
    // the principal minors (lanes 0-3); j = the first largest
    const int q4 = lane & 3;
    const float my_d = fabsf(minor_excl(s_f, l, q4, q4));
    int j = 0;
    float dj = __shfl_sync(0xffffffffu, my_d, 0);
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        const float di = __shfl_sync(0xffffffffu, my_d, i);
        if (di > dj) {
            j = i;
            dj = di;
        }
    }
    // cofactor (i, j) of a symmetric matrix: lane i takes q[i] = (-1)^(i+j) minor(rows != j, cols != i)
    const bool neg = ((q4 + j) & 1) != 0;
    FF my_q{0.0f, 0.0f};
    int solver = 0;
    if (finite && dj > 1e-4f) {
        // 3. Rayleigh-quotient inverse iteration in FF
        float my_qf = minor_excl(s_f, l, j, q4);
        if (neg) my_qf = -my_qf;
        const int steps = dj < 1e-2f ? 2 : 1;
        for (int s = 0; s < steps; ++s) {
            // lane r: row r of N times qf, then the Rayleigh quotient num / qq over lanes 0-3
            FF t{0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 4; ++c) t = t + s_nf[sym(q4, c)] * __shfl_sync(0xffffffffu, my_qf, c);
            FF num = lane < 4 ? t * my_qf : FF{0.0f, 0.0f};
            FF qq = lane < 4 ? FF{my_qf, 0.0f} * my_qf : FF{0.0f, 0.0f};
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                num = num + shfl_ff(num, lane ^ o);
                qq = qq + shfl_ff(qq, lane ^ o);
            }
            num = shfl_ff(num, 0);
            qq = shfl_ff(qq, 0);
            my_q = minor_excl(s_nf, ff_div(num, qq), j, q4);
            if (neg) my_q = -my_q;
            my_qf = my_q.hi;
        }
    } else {
        // 4. nearly repeated largest eigenvalue (or no finite solution)
        solver = 1;
        if (lane == 0) {
            double A[16], V[16];
            for (int r = 0; r < 4; ++r)
                for (int c = 0; c < 4; ++c) A[4 * r + c] = (double)s_nf[sym(r, c)].hi + (double)s_nf[sym(r, c)].lo;
            jacobi4(A, V);
            int imax = 0;
            for (int i = 1; i < 4; ++i)
                if (A[i] > A[imax]) imax = i;
            for (int i = 0; i < 4; ++i) {
                const double vi = V[4 * i + imax];
                s_nf[i] = FF{(float)vi, (float)(vi - (double)(float)vi)};  // N is not needed any more
            }
        }
        __syncwarp();
        my_q = s_nf[q4];
    }
    // q = normalize(q) (:231): 1/sqrt(q'q) from a float estimate and one FF Newton step
    FF qq = lane < 4 ? my_q * my_q : FF{0.0f, 0.0f};
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) qq = qq + shfl_ff(qq, lane ^ o);
    qq = shfl_ff(qq, 0);
    const float r0 = rsqrtf(qq.hi);
    const FF corr = (FF{1.0f, 0.0f} - qq * r0 * r0) * (0.5f * r0);
    my_q = my_q * (FF{r0, 0.0f} + corr);
    // R from the quaternion, x = scalar part (:233-254), in FF: lane k < 9 takes entry k
    //   diagonal k = 0, 4, 8:  1 - 2 (q_a q_a + q_b q_b)
    //   off-diagonal:          2 (q_a q_b +- q_c q_d)
    const int rk = lane < 9 ? lane : 0;
    // (a, b, c, d) per entry, 4 bits each: (2,2,3,3) (1,2,0,3) (1,3,0,2) (1,2,0,3) (1,1,3,3)
    // (2,3,0,1) (1,3,0,2) (2,3,0,1) (1,1,2,2)
    constexpr unsigned long long kA = 0x121211112ull, kB = 0x133312322ull, kC = 0x200030003ull,
                                 kD = 0x212133233ull;
    const int ia = (int)(kA >> (4 * rk)) & 15, ib = (int)(kB >> (4 * rk)) & 15;
    const int ic = (int)(kC >> (4 * rk)) & 15, id = (int)(kD >> (4 * rk)) & 15;
    const FF qa = shfl_ff(my_q, ia), qb = shfl_ff(my_q, ib), qc = shfl_ff(my_q, ic), qd = shfl_ff(my_q, id);
    const FF pab = qa * qb, pcd = qc * qd;
    const bool rdiag = rk == 0 || rk == 4 || rk == 8;
    const bool rminus = rk == 1 || rk == 5 || rk == 6;
    const FF my_r = rdiag ? FF{1.0f, 0.0f} - (pab + pcd) * 2.0f : (rminus ? pab - pcd : pab + pcd) * 2.0f;
    // t = dstMedian - R srcMedian (:256): lane r < 3
    const int tr3 = lane < 3 ? lane : 0;
    const FF mu0 = shfl_ff(my_mu, 0), mu1 = shfl_ff(my_mu, 1), mu2 = shfl_ff(my_mu, 2);
    const FF mud = shfl_ff(my_mu, 3 + tr3);
    const FF my_t = mud - (shfl_ff(my_r, 3 * tr3) * mu0 + shfl_ff(my_r, 3 * tr3 + 1) * mu1 +
                           shfl_ff(my_r, 3 * tr3 + 2) * mu2);
    // pose <- [R t; 0 1] pose (:259-263, :20-28): lane k < 12 takes row r = k % 3 of column c = k / 3
    const FF v = shfl_ff(my_r, 3 * pr) * P[0] + shfl_ff(my_r, 3 * pr + 1) * P[1] + shfl_ff(my_r, 3 * pr + 2) * P[2] +
                 shfl_ff(my_t, pr) * P[3];
    __syncwarp();  // every lane has read its column before any entry is replaced
    if (lane < 12) {
        st->pose_f[4 * pc + pr] = v.hi;
        st->pose_lo[4 * pc + pr] = v.lo;
    }
    const FF md0 = shfl_ff(my_mu, 3), md1 = shfl_ff(my_mu, 4), md2 = shfl_ff(my_mu, 5);
    // the alignment's last step publishes the pose to the host's mailbox (a
    // launch argument, null in the other steps): lanes 0-11 their new entries,
    // lanes 0, 3, 6, 9 their column's unchanged bottom entry, then lane 0 the number
    if (mail) {
        if (lane < 12) {
            mail->pose[4 * pc + pr] = v.hi;
            if (pr == 0) mail->pose[4 * pc + 3] = P[3].hi;
        }
        __threadfence_system();
        __syncwarp();
        if (lane == 0) *(volatile unsigned long long*)&mail->seq = mail_seq;
    }
    if (lane != 0) return;
    st->n_assoc = (int)n;
    st->mu_s[0] = fadd(mu0.hi, mu0.lo);
    st->mu_s[1] = fadd(mu1.hi, mu1.lo);
    st->mu_s[2] = fadd(mu2.hi, mu2.lo);
    st->mu_d[0] = fadd(md0.hi, md0.lo);
    st->mu_d[1] = fadd(md1.hi, md1.lo);
    st->mu_d[2] = fadd(md2.hi, md2.lo);
    if (step < kIcpMaxStats) {
        st->stats[step].n_assoc = (int)n;
        st->stats[step].solver = solver;
        st->stats[step].sum_l2 = fadd(tot[16].hi, tot[16].lo);
        const unsigned long long t_end = global_ns();
        // spans below 2^32 ns: the 32-bit conversions round as the 64-bit ones
        st->stats[step].body_us = (float)(unsigned int)(t_body - t_start) * 1e-3f;
        st->stats[step].tail_us = (float)(unsigned int)(t_end - t_body) * 1e-3f;
    }
    st->t_start = ~0ull;
    st->t_body = 0ull;
    st->iter = step + 1;
}

__device__ __forceinline__ void icp_begin_body(IcpState* st, const Mat4& guess) {
    for (int i = 0; i < 16; ++i) {
        st->pose_f[i] = guess.m[i];
        st->pose_lo[i] = 0.0f;
    }
    st->iter = 0;
    st->range[0] = st->range[2] = to_ordered(INFINITY);
    st->range[1] = st->range[3] = to_ordered(-INFINITY);
    st->done = 0ull;
    st->t_start = ~0ull;
    st->t_body = 0ull;
}

__global__ void k_icp_begin(IcpState* st, Mat4 guess) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    icp_begin_body(st, guess);
}

// Where the points of a caller's target project within their pixels: the
// smallest and largest X(q) - x and Y(q) - (H - 1 - y) over the points in
// front of the eye (a point nearer than w_far to the eye plane, or behind
// it, is further than 0.1 m from every source that prunes).  A CTA joins its
// threads' bounds first: one atomic per warp and bound queued at four words (18
// us of a 1024x848 target, now 5, and 4 at 320x240).
constexpr int kRangeThreads = 512;
__global__ void __launch_bounds__(kRangeThreads) k_target_range(IcpArgs a, float w_far, IcpState* __restrict__ st) {
    __shared__ int s_range[4];
    if (threadIdx.x < 4) s_range[threadIdx.x] = threadIdx.x & 1 ? to_ordered(-INFINITY) : to_ordered(INFINITY);
    __syncthreads();
    const int n = a.synth_w * a.synth_h;
    const float hw = fmul((float)a.synth_w, 0.5f), hh = fmul((float)a.synth_h, 0.5f);
    float lx = INFINITY, hx = -INFINITY, ly = INFINITY, hy = -INFINITY;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 q = __ldg(a.synth + i);
        const float p[4] = {q.x, q.y, q.z, 1.0f};
        float c[4];
        mat_vec(a.proj, p, c);
        if (!(isfinite(q.x) && isfinite(q.y) && isfinite(q.z)) || !(c[3] > w_far)) continue;
        const int y = (int)i / a.synth_w, x = (int)i - y * a.synth_w;
        const float dx = c[0] / c[3] * hw + hw - (float)x;
        const float dy = c[1] / c[3] * hh + hh - (float)(a.synth_h - 1 - y);
        lx = fminf(lx, dx);
        hx = fmaxf(hx, dx);
        ly = fminf(ly, dy);
        hy = fmaxf(hy, dy);
    }
    const int r0 = __reduce_min_sync(0xffffffffu, to_ordered(lx)), r1 = __reduce_max_sync(0xffffffffu, to_ordered(hx));
    const int r2 = __reduce_min_sync(0xffffffffu, to_ordered(ly)), r3 = __reduce_max_sync(0xffffffffu, to_ordered(hy));
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_range[0], r0);
        atomicMax(&s_range[1], r1);
        atomicMin(&s_range[2], r2);
        atomicMax(&s_range[3], r3);
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        if (threadIdx.x & 1) atomicMax(&st->range[threadIdx.x], s_range[threadIdx.x]);
        else atomicMin(&st->range[threadIdx.x], s_range[threadIdx.x]);
    }
}

// The target's producers walk it in blocks of 8 x 4 pixels, a warp each (lane
// 8 r + c: the block's row r and column c), so that a block's bounding box is
// six warp reductions.
struct TargetPixel {
    int x, y, block;
    bool in;  // inside the target (blocks at its edges stick out)
};
__device__ __forceinline__ TargetPixel target_pixel(int block, int width, int height) {
    const int nbx = (width + kBlockW - 1) / kBlockW, by = block / nbx, lane = threadIdx.x & 31;
    TargetPixel t;
    t.x = (block - by * nbx) * kBlockW + (lane & 7);
    t.y = by * kBlockH + (lane >> 3);
    t.block = block;
    t.in = t.x < width && t.y < height;
    return t;
}
__device__ __forceinline__ int target_blocks(int width, int height) {
    return ((width + kBlockW - 1) / kBlockW) * ((height + kBlockH - 1) / kBlockH);
}

// Writes a target point as the association reads it -- (0,0,0) is no point
// (ICP.cpp:112) and gets x = NaN, which no distance test passes -- and, by
// the whole warp, its block's bounding box (inverted where there is no point).
__device__ __forceinline__ void put_target(const TargetPixel& t, float x, float y, float z, int width,
                                           float4* __restrict__ out, float4* __restrict__ boxes) {
    const bool point = t.in && !(x == 0.0f && y == 0.0f && z == 0.0f);
    if (t.in) out[(size_t)t.y * width + t.x] = make_float4(point ? x : __int_as_float(0x7fffffff), y, z, 1.0f);
    // a point with a NaN is nearest to nothing; infinite ones leave a box that excludes nothing wrongly
    const bool use = point && x == x && y == y && z == z;
    const float big = INFINITY;
    const float lx = from_ordered(__reduce_min_sync(0xffffffffu, to_ordered(use ? x : big)));
    const float ly = from_ordered(__reduce_min_sync(0xffffffffu, to_ordered(use ? y : big)));
    const float lz = from_ordered(__reduce_min_sync(0xffffffffu, to_ordered(use ? z : big)));
    const float hx = from_ordered(__reduce_max_sync(0xffffffffu, to_ordered(use ? x : -big)));
    const float hy = from_ordered(__reduce_max_sync(0xffffffffu, to_ordered(use ? y : -big)));
    const float hz = from_ordered(__reduce_max_sync(0xffffffffu, to_ordered(use ? z : -big)));
    if ((threadIdx.x & 31) == 0) {
        boxes[2 * (size_t)t.block] = make_float4(lx, ly, lz, 0.0f);
        boxes[2 * (size_t)t.block + 1] = make_float4(hx, hy, hz, 0.0f);
    }
}

// World points of a depth frame: the back-projection of
// DepthMap2PointCloud (Integrator.cpp:121-144) without the voxel step;
// pixels without depth get (0,0,0), the reference's "invalid" target value.
__device__ __forceinline__ void backproject_body(const void* __restrict__ depth, int u16, int width, int height,
                                                 float fl_inv_x, float fl_inv_y, float pp_x, float pp_y,
                                                 const Mat4& e2w, float4* __restrict__ out,
                                                 float4* __restrict__ boxes, unsigned int blk, unsigned int nblk) {
    const int n = target_blocks(width, height), warps = blockDim.x >> 5;
    for (int b = blk * warps + (threadIdx.x >> 5); b < n; b += nblk * warps) {
        const TargetPixel t = target_pixel(b, width, height);
        const float d = t.in ? load_depth(depth, (size_t)t.y * width + t.x, u16 != 0) : 0.0f;
        float w[4] = {0.f, 0.f, 0.f, 0.f};
        if (d > 0.0f) {
            float p[4];
            p[0] = fadd(fmul(fadd(fmul((float)t.x, fl_inv_x), pp_x), d), 0.0f);
            p[1] = fadd(fmul(fadd(fmul(fadd(0.0f, -(float)t.y), fl_inv_y), pp_y), d), 0.0f);
            p[2] = fadd(fmul(fadd(fmul(-1.0f, 1.0f), 0.0f), d), 0.0f);
            p[3] = fadd(fmul(fadd(fmul(0.0f, 1.0f), 0.0f), d), 1.0f);
            mat_vec(e2w.m, p, w);
        }
        put_target(t, w[0], w[1], w[2], width, out, boxes);
    }
}

__global__ void k_backproject(const void* __restrict__ depth, int u16, int width, int height,
                              float fl_inv_x, float fl_inv_y, float pp_x, float pp_y, Mat4 e2w,
                              float4* __restrict__ out, float4* __restrict__ boxes) {
    backproject_body(depth, u16, width, height, fl_inv_x, fl_inv_y, pp_x, pp_y, e2w, out, boxes, blockIdx.x,
                     gridDim.x);
}

// host float3 target -> the float4 layout the association reads (one
// 16-byte load per candidate)
__global__ void k_expand_target(const float* __restrict__ in, int width, int height, float4* __restrict__ out,
                                float4* __restrict__ boxes) {
    const int n = target_blocks(width, height), warps = blockDim.x >> 5;
    for (int b = blockIdx.x * warps + (threadIdx.x >> 5); b < n; b += gridDim.x * warps) {
        const TargetPixel t = target_pixel(b, width, height);
        const size_t i = t.in ? (size_t)t.y * width + t.x : 0;
        put_target(t, in[3 * i], in[3 * i + 1], in[3 * i + 2], width, out, boxes);
    }
}

// Renderer::Bin: a z-buffered splat.  The first point (in input order) with
// the smallest clip-space z wins a pixel, as the reference's sequential
// strict "<" test does; a 64-bit atomicMin over (ordered z, point index)
// gives the same winner in parallel.
__device__ __forceinline__ unsigned int ordered_bits(float z) {
    if (z == 0.0f) z = 0.0f;  // -0 and +0 compare equal
    unsigned int b = __float_as_uint(z);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__global__ void k_bin_splat(const float* __restrict__ pts, unsigned int n, Mat4 w2c, int width,
                            int height, unsigned long long* __restrict__ zbuf) {
    const float hw = fmul((float)width, 0.5f), hh = fmul((float)height, 0.5f);
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float p[4] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], 1.0f}, c[4];
        mat_vec(w2c.m, p, c);
        const float x = fdiv(c[0], c[3]), y = fdiv(c[1], c[3]), z = fdiv(c[2], c[3]);
        const int u = cvt_i32_x86(fadd(fmul(x, hw), hw));
        const int v = wrap_sub(height - 1, cvt_i32_x86(fadd(fmul(y, hh), hh)));
        if (u >= 0 && u < width && v >= 0 && v < height && z >= -1.0f && z <= 1.0f)
            atomicMin(zbuf + (size_t)v * width + u, (unsigned long long)ordered_bits(z) << 32 | i);
    }
}

__global__ void k_bin_resolve(const float* __restrict__ pts, const unsigned long long* __restrict__ zbuf,
                              int n_pix, float* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pix; i += gridDim.x * blockDim.x) {
        const unsigned long long z = zbuf[i];
        float x = 0.f, y = 0.f, w = 0.f;
        if (z != ~0ull) {
            const unsigned int j = (unsigned int)(z & 0xffffffffu);
            x = pts[3 * j];
            y = pts[3 * j + 1];
            w = pts[3 * j + 2];
        }
        out[3 * i] = x;
        out[3 * i + 1] = y;
        out[3 * i + 2] = w;
    }
}

// ---- batched: several frame pairs per launch, each pair's CTAs running the
// single-pair body on its arguments
__global__ void k_icp_begin_batch(const IcpJob* __restrict__ jobs, int n) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) icp_begin_body(jobs[v].st, jobs[v].guess);
}

// A batch's tiles search rectangles throughout (unless a target of the batch
// allows none): they are many rounds of CTAs, so that their work counts and not the
// slowest tile (8 sequences, 4 steps of 15: 10314 us, with windows by tile 10899,
// with windows only 17463; frames three apart 11729, 12421, 18189).
template <int kS>
__global__ void __launch_bounds__(kTileThreads * kHalves<kS>, kResident<kS>) k_icp_step_batch(const IcpJob* __restrict__ jobs, BlockMap m,
                                                                        bool first) {
    const int v = block_owner(m, blockIdx.x);
    const unsigned int b0 = m.first[v];
    icp_step_body<kS, kS != kWhole>(jobs[v].a, jobs[v].st, first, blockIdx.x - b0, m.first[v + 1] - b0);
}

__global__ void k_backproject_batch(const BackprojectJob* __restrict__ jobs, BlockMap m) {
    const int v = block_owner(m, blockIdx.x);
    const BackprojectJob& j = jobs[v];
    const unsigned int b0 = m.first[v];
    backproject_body(j.depth, 1, j.width, j.height, j.fl_inv_x, j.fl_inv_y, j.pp_x, j.pp_y, j.e2w, j.out, j.boxes,
                     blockIdx.x - b0, m.first[v + 1] - b0);
}

// the same resolve into the association's float4 target layout
__global__ void k_bin_resolve_target(const float* __restrict__ pts, const unsigned long long* __restrict__ zbuf,
                                     int width, int height, float4* __restrict__ out, float4* __restrict__ boxes) {
    const int n = target_blocks(width, height), warps = blockDim.x >> 5;
    for (int b = blockIdx.x * warps + (threadIdx.x >> 5); b < n; b += gridDim.x * warps) {
        const TargetPixel t = target_pixel(b, width, height);
        const unsigned long long z = t.in ? zbuf[(size_t)t.y * width + t.x] : ~0ull;
        float x = 0.f, y = 0.f, w = 0.f;
        if (z != ~0ull) {
            const unsigned int j = (unsigned int)(z & 0xffffffffu);
            x = pts[3 * (size_t)j];
            y = pts[3 * (size_t)j + 1];
            w = pts[3 * (size_t)j + 2];
        }
        put_target(t, x, y, w, width, out, boxes);
    }
}

}  // namespace

// CTAs of one pair's association (its tiles, at most kIcpMaxCtas)
int icp_tiles(int width, int height) {
    const int n_cols = (width + 3) / 4;
    const int tiles = ((n_cols + kTileCols - 1) / kTileCols) * ((height + kTileRows - 1) / kTileRows);
    return tiles < kIcpMaxCtas ? tiles : kIcpMaxCtas;
}

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Which build an alignment's steps take, all of them the same: the first steps
// after a change of kernels wait for the finisher's instructions, 2 us each.
// Whole windows only where nothing is known of the target, and where there are too
// few steps to win by rectangles: a 640x480 pair wins from the fifth step on and
// loses a little before (4 steps 133 us against 127), one of 320x240 wins at once (4
// steps 84 against 91).  A finer target's windows take more than that build stages.
struct StepShape {
    int shape;
    template <typename F>
    auto with(F f) const {
        switch (shape) {
            case kWhole: return f(std::integral_constant<int, kWhole>{});
            case 1: return f(std::integral_constant<int, 1>{});
            case 2: return f(std::integral_constant<int, 2>{});
            default: return f(std::integral_constant<int, 3>{});
        }
    }
};
// fine: the target's pixels are finer than 1 / 1.15 of the source's
static StepShape tile_shape(int ctas, bool fine) {
    const int sms = sm_count();
    return {ctas <= sms ? 1 : ctas > 2 * sms && !fine ? 3 : 2};
}
static StepShape step_shape(int ctas, int iterations, int prune, bool fine) {
    const StepShape s = tile_shape(ctas, fine);
    return prune == kPruneOff || (iterations < (s.shape == 2 ? 8 : 4) && !fine) ? StepShape{kWhole} : s;
}

// programmatic dependent launch: each step's grid is scheduled as soon as
// every CTA of the one before has finished its association, overlapping
// its launch with the previous finisher (k_icp_step waits for it)
template <int kS, typename Kernel, typename... Args>
static cudaError_t launch_step(Kernel kernel, int ctas, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kTileThreads * kHalves<kS>);
    cfg.dynamicSmemBytes = kTileBytes<kS>;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t icp_align_enqueue(const IcpArgs& a, IcpState* st, const Mat4& guess, int iterations,
                              int /*ctas*/, cudaStream_t stream, IcpPoseMail* mail, unsigned long long seq) {
    k_icp_begin<<<1, 32, 0, stream>>>(st, guess);
    const int ctas = icp_tiles(a.width, a.height);
    const bool fine = 20 * a.synth_w > 23 * a.width || 20 * a.synth_h > 23 * a.height;
    IcpArgs other = a;
    other.mail = nullptr;
    const StepShape shape = step_shape(ctas, iterations, a.prune, fine);
    if (shape.shape == kWhole) other.prune = kPruneOff;
    if (other.prune == kPruneMeasured)
        k_target_range<<<sm_count(), kRangeThreads, 0, stream>>>(a, a.w_min * 0.125f, st);
    IcpArgs last = other;  // the last step publishes the pose
    last.mail = mail;
    last.mail_seq = seq;
    for (int it = 0; it < iterations; ++it) {
        const cudaError_t e =
            shape.with([&](auto s) {
                return launch_step<s.value>(k_icp_step<s.value>, ctas, stream, it + 1 == iterations ? last : other, st,
                                            it == 0);
            });
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

// The association's dynamic shared memory above the default 48 KB limit; set
// with every context, outside any stream capture.
cudaError_t icp_init_device() {
    cudaError_t e = cudaSuccess;
    for (int shape = 0; shape < 4 && !e; ++shape)
        e = StepShape{shape}.with([](auto s) {
            const cudaError_t x = cudaFuncSetAttribute(k_icp_step<s.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)kTileBytes<s.value>);
            return x ? x
                     : cudaFuncSetAttribute(k_icp_step_batch<s.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kTileBytes<s.value>);
        });
    return e;
}

cudaError_t icp_align_batch_enqueue(const IcpJob* jobs, int n, const BlockMap& map, int iterations, bool prune,
                                    cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    k_icp_begin_batch<<<(n + 63) / 64, 64, 0, stream>>>(jobs, n);
    const StepShape shape = prune ? tile_shape((int)map.grid, false) : StepShape{kWhole};  // (targets have their sources' sizes)
    for (int it = 0; it < iterations; ++it) {
        const cudaError_t e = shape.with([&](auto s) {
            return launch_step<s.value>(k_icp_step_batch<s.value>, (int)map.grid, stream, jobs, map, it == 0);
        });
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t backproject_batch_enqueue(const BackprojectJob* jobs, int n, const BlockMap& map, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_backproject_batch<<<map.grid, kThreads, 0, st>>>(jobs, map);
    return cudaGetLastError();
}

// float4s of a target's block boxes
size_t icp_box_count(int width, int height) {
    return 2 * (size_t)((width + kBlockW - 1) / kBlockW) * ((height + kBlockH - 1) / kBlockH);
}

cudaError_t expand_target_enqueue(const float* in, int width, int height, float4* out, float4* boxes, int ctas,
                                  cudaStream_t st) {
    k_expand_target<<<ctas, kThreads, 0, st>>>(in, width, height, out, boxes);
    return cudaGetLastError();
}

cudaError_t backproject_enqueue(const void* depth, bool u16, const kifi_camera& cam,
                                const Mat4& eye_to_world, float4* out, float4* boxes, int ctas, cudaStream_t st) {
    const float fix = fdiv(1.0f, cam.fx), fiy = fdiv(1.0f, cam.fy);
    const float ppx = fmul(fsub(0.5f, cam.cx), fix), ppy = fmul(fsub(cam.cy, 0.5f), fiy);
    k_backproject<<<ctas, kThreads, 0, st>>>(depth, u16 ? 1 : 0, cam.width, cam.height, fix, fiy,
                                             ppx, ppy, eye_to_world, out, boxes);
    return cudaGetLastError();
}

cudaError_t bin_enqueue(const float* pts, unsigned int n, const Mat4& w2c, int width, int height,
                        unsigned long long* zbuf, float* out, int ctas, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(zbuf, 0xff, (size_t)width * height * 8, st);
    if (e) return e;
    if (n) k_bin_splat<<<ctas, kThreads, 0, st>>>(pts, n, w2c, width, height, zbuf);
    k_bin_resolve<<<ctas, kThreads, 0, st>>>(pts, zbuf, width * height, out);
    return cudaGetLastError();
}

cudaError_t bin_target_enqueue(const float* pts, unsigned int n, const Mat4& w2c, int width, int height,
                               unsigned long long* zbuf, float4* out, float4* boxes, int ctas, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(zbuf, 0xff, (size_t)width * height * 8, st);
    if (e) return e;
    if (n) k_bin_splat<<<ctas, kThreads, 0, st>>>(pts, n, w2c, width, height, zbuf);
    k_bin_resolve_target<<<ctas, kThreads, 0, st>>>(pts, zbuf, width, height, out, boxes);
    return cudaGetLastError();
}

}  // namespace kifi
