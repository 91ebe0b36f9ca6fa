// kifi_internal.h -- declarations shared between the library's translation
// units (not part of the public ABI).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "kifi_common.cuh"

namespace kifi {

// ------------------------------------------------- chained launches
// The kernels of a frame's fusion follow one another on one stream, each a
// few microseconds long.  Launched as programmatic dependents (chained), a
// kernel's CTAs are placed as the last CTAs of the one before leave, and wait
// (chain_begin, the first thing they do) for its memory to be visible: the
// launch no longer stands between them (a 320x240 frame 75 -> 59 us; letting
// them in when the kernel before had started, so that they held SM slots while
// it ran, gave 65).  Beside a tracking stream launches are plain: waiting CTAs
// would hold the SMs that tracking's next step needs.  To a chained kernel,
// what the ones before write is not read-only data (ld.global.nc, which const
// __restrict__ pointers invite, may find stale lines): such pointers are not
// restrict, and the arrays are read in L2.  The few words that every CTA
// starts with are plain loads: every warp of a grid reading them in L2 queues
// at one slice (7 us of a 320x240 frame's merge).
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
inline cudaError_t chain_launch(bool chained, dim3 grid, dim3 block, cudaStream_t st, void (*kernel)(Params...),
                                Args&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// ------------------------------------------------------------ radix sort
// up to 8 digit passes: keys of up to 64 bits
constexpr int kSortMaxPasses = 8;
// A frame's 30-bit new keys sort in three 10-bit digit passes, 64-bit ones in
// as many 8-bit passes as their bits need (five beyond 10 bits per axis: their
// frames have more tiles, and 10-bit digits' look-back words, 8 KB a tile, would
// be half the traffic).  The frame's set-up kernel zeroes the passes' histograms
// and tile counters, and the splat counts the digits of every key it stores,
// so the sort itself is its passes (after an odd number the result lies in
// SortScratch::alt_keys).
template <typename K>
constexpr int kFrameDigitBits = sizeof(K) == 4 ? 10 : 8;
template <typename K>
__host__ __device__ constexpr int frame_sort_passes(int kb) {
    return (3 * kb + kFrameDigitBits<K> - 1) / kFrameDigitBits<K>;
}
constexpr int kFrameMaxPasses = 5;
// counters of the largest digit set: 3 x 1024 (30-bit frame keys) or 8 x 256
constexpr int kSortHistWords = 3 * 1024;
static_assert(kSortHistWords >= kSortMaxPasses * 256, "histogram sized for both digit sets");
struct SortScratch {
    unsigned int* hist = nullptr;           // [passes][radix] digit counts
    unsigned int* tile_counter = nullptr;   // [passes] dynamic tile ids per pass
    unsigned long long* epoch = nullptr;    // look-back generation tag
    unsigned long long* lookback = nullptr; // [passes][tiles, then groups of tiles][radix]
    void* alt_keys = nullptr;               // ping-pong buffers, max_n (+pad), 8 bytes per key
    uint32_t* alt_vals = nullptr;
    unsigned int* status = nullptr;         // where timeouts are reported
    size_t max_tiles = 0, max_n = 0;
    // polls of a predecessor's look-back word before a pass gives up, and the
    // first tile id the passes hand out (0; a test sets both through
    // kifi_sort_set_fault_injection to make a look-back wait run out)
    unsigned long long spin_limit = 0;
    unsigned int first_tile = 0;
};

size_t sort_max_tiles(size_t max_n);
// zeroes its look-back words on `st`: the sorts that use it must run on st
// (or after it)
cudaError_t sort_scratch_alloc(SortScratch* s, size_t max_n, cudaStream_t st);
void sort_scratch_free(SortScratch* s);
cudaError_t sort_u32(uint32_t* keys, uint32_t* vals, const unsigned int* n_dev, SortScratch& s,
                     unsigned int* status, int grid_ctas, cudaStream_t st);
// keys of key_bytes (4 or 8) bytes holding key_bits significant bits: one
// stable 8-bit digit pass per byte of significant bits, rounded up to an
// even count so the result lands back in `keys`
cudaError_t sort_keys(void* keys, int key_bytes, int key_bits, uint32_t* vals, const unsigned int* n_dev,
                      SortScratch& s, unsigned int* status, int grid_ctas, cudaStream_t st);
// the frame path's passes (three of 10 bits over 30-bit keys, up to five of 8 bits
// over 64-bit ones) over keys whose histograms and pass counters are already set
// (see kFrameDigitBits); *sorted receives the buffer holding the result
cudaError_t sort_frame_keys(void* keys, int key_bytes, int kb, const unsigned int* n_dev, SortScratch& s,
                            unsigned int* status, int grid_ctas, bool alone, bool chained, cudaStream_t st, const void** sorted);

// ------------------------------------------------------------- integrate
struct VolumeBuffers {
    int key_bytes = 4;              // 4: 30-bit keys (uint32_t), 8: 64-bit keys (uint64_t)
    void* keys[2] = {nullptr, nullptr};
    float2* vals[2] = {nullptr, nullptr};
    size_t cap = 0;                 // voxels per buffer (arrays hold cap + pad)
    uint32_t* bitmap = nullptr;     // res^3 occupancy bits
    size_t bitmap_words = 0;
    void* new_keys = nullptr;       // keys new to the volume in this frame
    uint32_t* new_idx = nullptr;    // insert path: source position of each new key
    size_t new_cap = 0;
    unsigned long long* splits = nullptr;  // merge-path split of every output tile
};

struct LaunchShape {
    int sms = 0;          // multiprocessors of the device
    int sort_ctas = 0;    // persistent CTAs of the sort passes
    int merge_ctas = 0;   // persistent CTAs of the merge/update kernel
    int splat_ctas = 0;
    // beside tracking (a pipeline's volume): short-lived CTAs and the merge
    // variant that leaves room on the SMs (3 CTAs of 256 threads per SM);
    // alone: persistent CTAs and the merge variant capped at 64 registers
    // (4 CTAs per SM)
    bool beside_tracking = false;
};

// Enqueues one Integrator::Integrate on `st`.  depth_dev holds the frame
// (float metres, or uint16 millimetres when depth_u16).
// `events` (optional, 4 entries) are recorded before the frame set-up, after
// splat+emit, after the sort and after merge+update.
cudaError_t integrate_enqueue(DeviceCtl* ctl, const Geom& g, VolumeBuffers& vb, SortScratch& ss,
                              const void* depth_dev, bool depth_u16, const kifi_camera& cam,
                              const Mat4& world_to_eye, const LaunchShape& ls, cudaStream_t st,
                              cudaEvent_t* events);

// resident CTAs per SM of the merge/update kernel (occupancy API)
int merge_blocks_per_sm();

// flat_map::insert of n sorted unique device keys: filter out resident keys
// (their values win) and collect (key, index) of the rest in new_keys /
// new_idx; the caller sorts those pairs and then merges.
// merge-path split slots a volume of `cap` voxels needs
size_t merge_max_tiles(const VolumeBuffers& vb, size_t cap);
cudaError_t insert_filter_enqueue(DeviceCtl* ctl, const Geom& g, VolumeBuffers& vb,
                                  const void* keys_dev, const unsigned int* n_dev,
                                  const LaunchShape& ls, cudaStream_t st);
cudaError_t insert_merge_enqueue(DeviceCtl* ctl, const Geom& g, VolumeBuffers& vb,
                                 const float2* vals_dev, const LaunchShape& ls, cudaStream_t st);
// clears the occupancy bitmap and sets the bits of the resident keys
cudaError_t bitmap_rebuild_enqueue(const DeviceCtl* ctl, const Geom& g, const VolumeBuffers& vb,
                                   const LaunchShape& ls, cudaStream_t st);

// ------------------------------------------------------------- batches
// A batched launch runs one stage for several volumes (or ICP frame pairs)
// at once: volume v owns the CTAs [first[v], first[v+1]) of the grid and
// reads its arguments from a device table.
struct BlockMap {
    const unsigned int* first;  // device, n + 1 entries; first[n] = grid
    int n;
    unsigned int grid;          // the launch's CTAs (known on the host)
};

// One volume's frame in a batched fusion launch: the arguments of the
// single-volume kernels.  Depth frames are uint16 millimetres.
struct FuseJob {
    DeviceCtl* ctl;
    Geom g;
    VolumeBuffers vb;
    SortScratch ss;
    const void* depth;
    FrameConst fc;
    unsigned int max_tiles;  // merge-path split slots of the volume
};

#ifdef __CUDACC__
// the volume that owns CTA b of a batched launch
__device__ __forceinline__ int block_owner(const BlockMap& m, unsigned int b) {
    int lo = 0, hi = m.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (m.first[mid] <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}
#endif

// The CTA shares of one batched fusion step, one map per stage; every
// volume of the batch has the same key width.
struct FuseMaps {
    BlockMap splat, hist, pass, partition, merge;
};

// The batched fusion of a step as one persistent launch over a device work
// queue (integrate_queue_enqueue): stages 0 set-up, 1 splat, 2 histogram,
// 3 .. 2 + passes the digit passes, then the partition and the merge; first[k]
// is the number of stage k's first item, first[stages] the item count.
constexpr int kQueueMaxStages = 5 + kSortMaxPasses;
struct FuseQueuePlan {
    int n = 0;       // scenes
    int passes = 0;  // digit passes
    int stages = 0;  // 5 + passes
    unsigned int first[kQueueMaxStages + 1] = {};
    BlockMap maps[5] = {};  // splat, histogram, pass, partition, merge
};
// the block map of stage k (k >= 1)
KIFI_HD int fuse_stage_map(int k, int passes) {
    return k == 1 ? 0 : k == 2 ? 1 : k < 3 + passes ? 2 : k == 3 + passes ? 3 : 4;
}

// Enqueues Integrator::Integrate of one frame for each of the n volumes of
// `jobs` (a device table) on `st`: one launch per stage for all of them.
// key_bytes: the volumes' key width; passes: digit passes of the sort.
// the sort of every volume's new keys (FuseJob::vb.new_keys, count in ctl->n_new)
cudaError_t sort_batch_enqueue(const FuseJob* jobs, int n, int key_bytes, int passes, const BlockMap& hist,
                               const BlockMap& pass, cudaStream_t st);
// the look-back limits every sort applies (kifi_sort_set_fault_injection)
void sort_limits(SortScratch* s);
cudaError_t integrate_batch_enqueue(const FuseJob* jobs, int n, int key_bytes, int passes, const FuseMaps& maps,
                                    cudaStream_t st);
// the same as one persistent launch of `ctas` CTAs; next (1 word) and done
// (plan.n x plan.stages words) must be zero
cudaError_t integrate_queue_enqueue(const FuseJob* jobs, int key_bytes, const FuseQueuePlan& plan,
                                    unsigned int* next, unsigned int* done, int ctas, cudaStream_t st);

// ---------------------------------------------------------------- mesher
struct MeshCounts {
    unsigned long long n_verts;
    unsigned long long n_idx;
    unsigned long long missing_min;  // smallest triangle edge id without a vertex (or ~0)
    unsigned long long overflow;     // emission skipped: kMeshBuffers or kMeshWords were too small
    unsigned int runs_done;          // classification CTAs that have finished
    unsigned int n_words;
};
constexpr unsigned long long kMeshBuffers = 1, kMeshWords = 2;  // the output buffers, the scratch's words

// The volume as words: runs of 32 consecutive keys (key >> 5) with at least
// one resident voxel, ascending; at most one per voxel.
struct MeshWords {
    void* key = nullptr;           // key >> 5 << 4 | the state of its key 0 (bits of the four masks below)
    uint4* a = nullptr;            // first voxel; masks: resident, weight != 0, weight > 0
    uint2* b = nullptr;            // masks: Distance() < 0, operands in the sign rule's range
    uint4* v = nullptr;            // vertex masks of the +x, +y and +z edges; the first vertex within the run
    uint4* link = nullptr;         // words with output: the +y, +z and +yz words; an index offset within the run
    unsigned int* count = nullptr;
};

struct MeshScratch {
    void* tables = nullptr;  // the allocation that holds the arrays whose sizes the volume does not change
    void* block = nullptr;   // and the one for the words and the list
    MeshWords words;
    uint2* flagged = nullptr;            // a slot per voxel: those with output, run by run, ascending --
                                         // word within the run << 13 | bit << 8 | case; first index, from the word's link
    unsigned int* run_words = nullptr;  // per run of voxels: words that start in it
    uint4* run_out = nullptr;           // per run of words: vertices, indices and voxels with output before it, their list
    unsigned int* rows = nullptr;         // first word of each (z, y) key row
    MeshCounts* counts = nullptr;
    unsigned int* n_dev = nullptr;        // the voxel count the passes read
    size_t cap = 0, words_cap = 0, rows_cap = 0;
};

// Scratch for a mesh of up to n voxels: room for `want` (>= n) where it can be
// had.  Its words are an estimate until a mesh has asked for more: a mesh with
// more words than they hold is not emitted (MeshCounts::overflow kMeshWords), and
// is to be counted again after a call with its n_words.
cudaError_t mesh_scratch_reserve(MeshScratch* m, size_t n, size_t want, size_t n_words, int kb);
void mesh_scratch_free(MeshScratch* m);
// stage_events (optional, 2 entries): recorded after the words are built and
// after the classification
cudaError_t mesh_count_enqueue(const void* keys, int key_bytes, const float2* vals, size_t n_cap, int kb,
                               int with_indices, MeshScratch& ms, cudaStream_t st, cudaEvent_t* stage_events = nullptr);
// Emission sums up the counting passes' totals on the device and writes them
// to ms.counts, so it can be enqueued right behind them.  The buffers
// hold vert_cap vertices and idx_cap indices; when the mesh needs more, the
// emission writes nothing else and sets ms.counts->overflow.
cudaError_t mesh_emit_enqueue(const Geom& g, int key_bytes, const float2* vals, size_t n_cap, int with_indices,
                              MeshScratch& ms, size_t vert_cap, size_t idx_cap, float* verts_dev, uint32_t* idx_dev,
                              int sms, cudaStream_t st);
cudaError_t mesh_snapshot_enqueue(const DeviceCtl* ctl, const VolumeBuffers& vb, void* keys, float2* vals,
                                  size_t cap, unsigned int* n_dev, int sms, cudaStream_t st);

// ------------------------------------------------------------------ ICP
constexpr int kIcpMaxStats = 64;
constexpr int kIcpMaxCtas = 2048;
constexpr int kIcpTileSources = 256;  // sources per association tile

// Where the last step of an alignment publishes its pose for a host that
// polls instead of synchronising (page-locked, mapped host memory): the pose
// (kifi order), then the alignment's sequence number, written after it.
struct IcpPoseMail {
    float pose[16];
    unsigned long long seq;
};

constexpr int kPruneOff = 0, kPruneKnown = 1, kPruneMeasured = 2;

struct IcpArgs {
    const void* depth;      // source frame (float metres or uint16 mm)
    int depth_u16;
    int width, height;
    float fl_inv_x, fl_inv_y, pp_x, pp_y;
    float proj[16];         // EyeToClipRH * inverse(synth eye-to-world), kifi order
    const float4* synth;    // target world points (x = NaN: none; w = 1), synth_w * synth_h
    int synth_w, synth_h;
    const float4* boxes;    // per block of 8 x 4 target pixels (row-major): its points' bounds, lower then upper
    // which candidates of a window can win (kifi_icp.cu, Prune)
    int prune;              // kPruneOff, kPruneKnown (lo, hi below) or kPruneMeasured (IcpState::range)
    float kx, ky, eps, eps0, w_min;
    float lo[2], hi[2];
    long long* pairs;       // optional: per source the winner's target index (-1: none) ...
    float* pairs_len2;      // ... and its len^2, overwritten by every iteration
    float neg_zero;         // -0.0f, a value the device code cannot see at compile time
    IcpPoseMail* mail;      // the step that publishes the final pose (the last): its
    unsigned long long mail_seq;  // mailbox and the alignment's number; null otherwise
};

struct IcpIterStats {
    int n_assoc;
    int solver;       // Horn's eigenvector: 0 closed form, 1 Jacobi fallback
    float sum_l2;     // the associated squared distances' sum (the host forms the RMS)
    float body_us;    // first CTA start to last CTA end of the association
    float tail_us;    // last CTA end to the updated pose
};

// What an association tile leaves for its next step.
struct IcpTile {
    int near[4];  // where its sources project: x0, y0, x1, y1
    int rect[4];  // the part of the target that it searched, likewise
    int whole;    // scan whole windows (else the rectangles that can win)
    int pad[3];
};

struct IcpState {
    alignas(16) float pose_f[16];   // eye-to-world estimate, kifi order (float-float high part)
    float pose_lo[16];  // and its low part
    unsigned long long done;  // CTAs finished (high 32 bits) and their associations (low 32 bits)
    float mu_s[4], mu_d[4];
    int n_assoc;
    int iter;
    int range[4];  // kPruneMeasured: the target's lo x, hi x, lo y, hi y as ordered integers
    unsigned long long t_start, t_body;  // globaltimer stamps of the running step
    IcpIterStats stats[kIcpMaxStats];
    float part[34 * kIcpMaxCtas];   // per-CTA float-float partials: hi, lo rows of 17 components
    IcpTile tile[kIcpMaxCtas];
    // per tile and source: the pixel that won the last step (row << 16 | column), or ~0; here, so that
    // an alignment allocates nothing, whatever its frame's size (tiles from kIcpMaxCtas on keep none)
    unsigned int winner[kIcpTileSources * kIcpMaxCtas];
};

cudaError_t icp_init_device();
// One ICP frame pair of a batched alignment: the arguments of the
// single-pair kernels.
struct IcpJob {
    IcpArgs a;
    IcpState* st;
    Mat4 guess;
};
// `iterations` AlignSteps of the n pairs of `jobs` (a device table), one
// launch per step for all of them; pair v's CTAs are map.first[v] ..
// map.first[v+1] - 1, one per association tile.
// prune: every pair's (IcpArgs::prune is not kPruneOff)
cudaError_t icp_align_batch_enqueue(const IcpJob* jobs, int n, const BlockMap& map, int iterations, bool prune,
                                    cudaStream_t stream);
// Back-projection of one frame per pair into its target (the next frame's
// ICP target), for the n entries of `jobs` (device table).
struct BackprojectJob {
    const void* depth;  // uint16 millimetres
    int width, height;
    float fl_inv_x, fl_inv_y, pp_x, pp_y;
    Mat4 e2w;
    float4* out;
    float4* boxes;
};
cudaError_t backproject_batch_enqueue(const BackprojectJob* jobs, int n, const BlockMap& map, cudaStream_t st);
// CTAs of one frame pair's association (one per tile)
int icp_tiles(int width, int height);
// mail (device address of mapped host memory, or null): the last step
// publishes the final pose there with sequence number `seq`
cudaError_t icp_align_enqueue(const IcpArgs& a, IcpState* st, const Mat4& guess, int iterations,
                              int ctas, cudaStream_t stream, IcpPoseMail* mail = nullptr,
                              unsigned long long seq = 0);
cudaError_t backproject_enqueue(const void* depth, bool u16, const kifi_camera& cam,
                                const Mat4& eye_to_world, float4* out, float4* boxes, int ctas, cudaStream_t st);
// float4s of a width x height target's block boxes (IcpArgs::boxes)
size_t icp_box_count(int width, int height);
cudaError_t expand_target_enqueue(const float* in, int width, int height, float4* out, float4* boxes, int ctas,
                                  cudaStream_t st);

cudaError_t bin_enqueue(const float* pts, unsigned int n, const Mat4& w2c, int width, int height,
                        unsigned long long* zbuf, float* out, int ctas, cudaStream_t st);
// Bin straight into an ICP target (a float4 per pixel: w = 1, which the distances take in; x = NaN: no point)
cudaError_t bin_target_enqueue(const float* pts, unsigned int n, const Mat4& w2c, int width, int height,
                               unsigned long long* zbuf, float4* out, float4* boxes, int ctas, cudaStream_t st);

// Optional epilogue of gemm_bf16_enqueue: C = acc + bias[n] (FP32), or with
// out_bf16 set, out_bf16 = bf16(relu?(acc + bias[n])) (row stride ldc) in
// place of C.
struct GemmEpilogue {
    const float* bias = nullptr;
    bool relu = false;
    void* out_bf16 = nullptr;
};

// C[M x N] (+)= A[M x K] * B[N x K]^T, BF16 in, FP32 out, on tcgen05 tensor
// cores with TMA-fed operands (kifi_tc_gemm.cu).  k_split > 0 splits K
// across tiles that add into C atomically (atomic must then be true and C
// pre-initialised; the split is rounded up to a multiple of 64).
cudaError_t gemm_bf16_enqueue(const void* A, const void* B, float* C, int M, int N, int K, int lda, int ldb,
                              int ldc, int k_split, bool atomic, unsigned int* status, cudaStream_t st,
                              const GemmEpilogue* epi = nullptr);

// 3x3 / stride 2 / pad 1 convolution of an NHWC BF16 input [batch][H][W][Cin]
// (Cin 32 or 64) with weights [Co][Kp] (k = (ky * 3 + kx) * Cin + c, Co 64 or
// 128) as an implicit GEMM on the tensor cores: out_bf16 [batch][Ho][Wo][Co]
// = bf16(relu?(conv + bias)), Ho = (H + 1) / 2, Wo = (W + 1) / 2.
cudaError_t conv3x3s2_bf16_enqueue(const void* x, int batch, int H, int W, int Cin, const void* Wt, int Co, int Kp,
                                   const float* bias, bool relu, void* out_bf16, unsigned int* status,
                                   cudaStream_t st);

}  // namespace kifi
