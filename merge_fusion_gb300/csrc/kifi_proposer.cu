// kifi_proposer.cu -- the learned ICP pose proposer: a small convolutional
// network that maps two box-downsampled depth frames (2 x 60 x 80, FP16,
// metres, 0 = no depth) to a 6-DoF twist that warm-starts ICP.  No
// counterpart in the reference.
//
//   conv 3x3/2 2->32, ReLU     60x80 -> 30x40
//   conv 3x3/2 32->64, ReLU    -> 15x20
//   conv 3x3/2 64->64, ReLU    -> 8x10
//   conv 3x3/2 64->128, ReLU   -> 4x5
//   global average pool        -> 128
//   fc 128->64, ReLU; fc 64->6
//
// Activations are NHWC BF16; every product -- convolutions 2-4 as implicit
// GEMMs whose A tiles TMA gathers straight from the previous activation,
// convolution 1 through its im2col matrix, the fully connected layers, and
// all the backward products -- runs on the TMA-fed tcgen05 GEMM
// (kifi_tc_gemm.cu) with FP32 accumulation; forward products add the bias
// and apply the ReLU in the GEMM epilogue.  Parameters keep an
// FP32 master copy updated by Adam, which also writes the BF16 copies the
// GEMMs read.  Padded parameter entries (conv 1's K = 18 padded to 32, the
// output layer's 6 rows padded to 16) stay zero.
//
// Backward products, with col the im2col matrix [M x Kp] and dY the
// pre-activation gradient [M x Cout]:
//   dW    [Cout x Kp] = dY^T col      A = dY^T, B = col^T (inner M, split K)
//   dcol  [M x Kp]    = dY W          A = dY,   B = W^T
//   dX                = col2im(dcol)  a gather over the <= 4 taps per input, in
//                                     the pass that forms the next dY (k_grad)
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "kifi_api_util.h"

using namespace kifi;

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kInH = 60, kInW = 80, kInC = 2;
constexpr int kConvs = 4;
constexpr int kCin[kConvs] = {2, 32, 64, 64};
constexpr int kCout[kConvs] = {32, 64, 64, 128};
constexpr int kHin[kConvs] = {60, 30, 15, 8};
constexpr int kWin[kConvs] = {80, 40, 20, 10};
constexpr int kHout[kConvs] = {30, 15, 8, 4};
constexpr int kWout[kConvs] = {40, 20, 10, 5};
constexpr int kKp[kConvs] = {32, 288, 576, 576};  // 9 * Cin, padded to a multiple of 16
constexpr int kFc1 = 64, kOut = 6, kOutPad = 16;
constexpr int kThreads = 256;

// parameter tensors, in order: conv W/b x 4, fc1 W/b, fc2 W/b
struct Layout {
    size_t off[12], size[12], total;
    Layout() {
        const size_t sz[12] = {32 * 32, 32, 64 * 288, 64, 64 * 576, 64, 128 * 576, 128, 64 * 128, 64,
                               16 * 64, 16};
        total = 0;
        for (int i = 0; i < 12; ++i) {
            off[i] = total;
            size[i] = sz[i];
            total += (sz[i] + 7) / 8 * 8;  // 16-byte aligned BF16 copies
        }
    }
};
const Layout kLayout;

int blocks(size_t n) { return (int)((n + kThreads - 1) / kThreads); }

// ------------------------------------------------------------------ kernels

// Box mean of the valid (non-zero) depth of each 8x8 block of two frames ->
// NHWC FP16 [60][80][2]; 0 where a block has no depth.
__global__ void k_downsample(const void* __restrict__ da, const void* __restrict__ db, int u16, int width,
                             int height, __half* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kInH * kInW * 2) return;
    const int f = i & 1, px = (i >> 1) % kInW, py = (i >> 1) / kInW;
    const void* d = f ? db : da;
    const int bw = width / kInW, bh = height / kInH;
    float sum = 0.0f;
    int n = 0;
    for (int y = py * bh; y < (py + 1) * bh; ++y)
        for (int x = px * bw; x < (px + 1) * bw; ++x) {
            const size_t at = (size_t)y * width + x;
            const float z = u16 ? fmul((float)((const unsigned short*)d)[at], 0.001f) : ((const float*)d)[at];
            if (z > 0.0f) {
                sum += z;
                ++n;
            }
        }
    out[i] = __float2half_rn(n ? sum / (float)n : 0.0f);
}

// im2col of the first convolution (3x3, stride 2, pad 1, C = 2): col[m][k],
// m = (b, oy, ox), k = (ky * 3 + kx) * 2 + c, zero outside the input and for
// k >= 18; with kTrain its transpose colT[k][m] too, which the weight
// gradient reads.  A thread takes one m: nine 4-byte loads, one 64-byte row,
// and 32 columns that its warp writes as 64-byte runs.  Bound by its bytes
// (20 MB read and written per 256 inputs): 11 us, 80 with a thread per element
// and a transpose pass after it before.
template <bool kTrain>
__global__ void __launch_bounds__(kThreads) k_im2col_first(const __half* __restrict__ x, int batch,
                                                           bf16* __restrict__ col, bf16* __restrict__ colT) {
    constexpr int H = kHin[0], W = kWin[0], Ho = kHout[0], Wo = kWout[0], Kp = kKp[0];
    const int M = batch * Ho * Wo;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const int ox = m % Wo, oy = m / Wo % Ho, b = m / (Wo * Ho);
        __align__(16) bf16 v[Kp];
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const int iy = 2 * oy - 1 + t / 3, ix = 2 * ox - 1 + t % 3;
            __half2 h = __floats2half2_rn(0.0f, 0.0f);
            if (iy >= 0 && iy < H && ix >= 0 && ix < W)
                h = reinterpret_cast<const __half2*>(x)[((size_t)b * H + iy) * W + ix];
            v[2 * t] = __float2bfloat16_rn(__low2float(h));
            v[2 * t + 1] = __float2bfloat16_rn(__high2float(h));
        }
#pragma unroll
        for (int k = 18; k < Kp; ++k) v[k] = __float2bfloat16_rn(0.0f);
        uint4* row = reinterpret_cast<uint4*>(col + (size_t)m * Kp);
#pragma unroll
        for (int q = 0; q < Kp / 8; ++q) row[q] = reinterpret_cast<const uint4*>(v)[q];
        if (kTrain)
#pragma unroll
            for (int k = 0; k < Kp; ++k) colT[(size_t)k * M + m] = v[k];
    }
}

constexpr int kTileM = 64;        // rows of a transposing tile
constexpr int kTileP = kTileM + 8;  // its pitch: 16-byte vectors, a quarter of the banks apart

// A [rows of C][kTileM] tile in shared memory out to out[c][m0 ..], 16 bytes
// at a time (M is a multiple of 8: batches are).
template <int C>
__device__ __forceinline__ void put_transposed(const bf16 (*t)[kTileP], int m0, int M, bf16* __restrict__ out) {
    for (int i = threadIdx.x; i < C * (kTileM / 8); i += kThreads) {
        const int c = i / (kTileM / 8), q = i % (kTileM / 8) * 8;
        if (m0 + q < M)
            *reinterpret_cast<uint4*>(out + (size_t)c * M + m0 + q) = *reinterpret_cast<const uint4*>(&t[c][q]);
    }
}

// The transposed im2col matrix colT[k][m] of convolution L > 0, straight from
// the activation x [b][H][W][C] it convolves: per tap a tile of 64 output
// pixels' channel vectors goes through shared memory.  The matrix itself is
// not formed (the forward pass gathers its windows by TMA).  Bound by its
// writes: 74 MB for the three layers at batch 256, where the im2col matrix was
// written, read and written transposed (about 420 us, now 40).
template <int L>
__global__ void __launch_bounds__(kThreads) k_im2col_t(const bf16* __restrict__ x, int batch,
                                                       bf16* __restrict__ colT) {
    constexpr int H = kHin[L], W = kWin[L], C = kCin[L], Ho = kHout[L], Wo = kWout[L];
    constexpr int kVec = C / 8;  // 16-byte vectors per pixel
    __shared__ __align__(16) bf16 t[C][kTileP];
    const int M = batch * Ho * Wo, tap = blockIdx.y, ky = tap / 3, kx = tap % 3;
    for (int m0 = blockIdx.x * kTileM; m0 < M; m0 += gridDim.x * kTileM) {
        for (int i = threadIdx.x; i < kTileM * kVec; i += kThreads) {
            const int r = i / kVec, q = i % kVec, m = m0 + r;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (m < M) {
                const int ox = m % Wo, oy = m / Wo % Ho, b = m / (Wo * Ho);
                const int iy = 2 * oy - 1 + ky, ix = 2 * ox - 1 + kx;
                if (iy >= 0 && iy < H && ix >= 0 && ix < W)
                    v = *reinterpret_cast<const uint4*>(x + (((size_t)b * H + iy) * W + ix) * C + q * 8);
            }
            const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
            for (int k = 0; k < 8; ++k) t[q * 8 + k][r] = e[k];
        }
        __syncthreads();
        put_transposed<C>(t, m0, M, colT + (size_t)tap * C * M);
        __syncthreads();
    }
}

// out[c][r] = in[r][c] for several small matrices in one launch, 32x32 tiles
// through shared memory
struct TransposeJob {
    const bf16* in;
    bf16* out;
    int R, C, first;  // first: the launch's first tile of this matrix
};
constexpr int kMaxTransposes = 7;
struct TransposeJobs {
    TransposeJob j[kMaxTransposes];
    int n;
};
__global__ void k_transpose(TransposeJobs jobs) {
    __shared__ bf16 t[32][33];
    int k = 0;
    while (k + 1 < jobs.n && (int)blockIdx.x >= jobs.j[k + 1].first) ++k;
    const TransposeJob& q = jobs.j[k];
    const int tile = (int)blockIdx.x - q.first, tc = (q.C + 31) / 32;
    const int c0 = tile % tc * 32, r0 = tile / tc * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        if (r < q.R && c < q.C) t[j][threadIdx.x] = q.in[(size_t)r * q.C + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (r < q.R && c < q.C) q.out[(size_t)c * q.R + r] = t[threadIdx.x][j];
    }
}

// global average pool: [B][P][C] -> [B][C]
__global__ void k_gap(const bf16* __restrict__ act, int batch, int P, int C, bf16* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= batch * C) return;
    const int b = i / C, c = i % C;
    float s = 0.0f;
    for (int p = 0; p < P; ++p) s += __bfloat162float(act[((size_t)b * P + p) * C + c]);
    out[i] = __float2bfloat16_rn(s / (float)P);
}

// mean squared error over batch x 6; d = dL/dpred into dpred[B][16] (FP32
// and BF16), columns 6..15 zero; the summed loss is added to *loss
__global__ void k_mse(const float* __restrict__ pred, const float* __restrict__ target, int batch,
                      float* __restrict__ dpred, bf16* __restrict__ dpred_bf, float* __restrict__ loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < batch * kOutPad) {
        const int b = i / kOutPad, j = i % kOutPad;
        float d = 0.0f;
        if (j < kOut) {
            const float e = pred[i] - target[b * kOut + j];
            l = e * e;
            d = 2.0f * e / (float)(batch * kOut);
        }
        dpred[i] = d;
        dpred_bf[i] = __float2bfloat16_rn(d);
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.0f) atomicAdd(loss, l / (float)(batch * kOut));
}

// The gradient of a layer's pre-activation, in one pass: its value from the
// layer above, through the ReLU (act > 0, where there is one), as BF16 [M][C]
// and its transpose [C][M] for the two products that read it, and its column
// sums per CTA (part[c][CTA], which k_bias_sum turns into the bias gradient in a
// fixed order: it repeats bit for bit).  A thread keeps one column; a tile of 64
// rows is transposed in shared memory.  Values:
//   kPlain   src[m][c]
//   kPool    src[b][c] / P: the global average pool's gradient
//   kConv    the gather form of col2im over src = dcol [M'][Kp] of the
//            convolution above (3x3, stride 2, pad 1; taps in order): input
//            pixel (iy, ix) collects the outputs with iy = 2 oy - 1 + ky,
//            ix = 2 ox - 1 + kx
// Bound by its bytes and the gathers' latency: the lowest layer's pass moves
// 150 MB in 61 us.  Before, col2im, the ReLU, the column sums (one strided
// column per CTA, 830 of 2080 us at batch 256) and the transpose were passes of
// their own; a gradient step 1750 -> 678 us.
// L is the convolution above for kConv.
enum class GradSrc { kPlain, kPool, kConv };
template <int C, GradSrc kSrc, int L = 0>
__global__ void __launch_bounds__(kThreads) k_grad(const float* __restrict__ src, const bf16* __restrict__ act, int M,
                                                   bf16* __restrict__ gb, bf16* __restrict__ gbT,
                                                   float* __restrict__ part) {
    constexpr int H = kHin[L], W = kWin[L], Ho = kHout[L], Wo = kWout[L], Kp = kKp[L], P = kHout[3] * kWout[3];
    constexpr int kGroups = kThreads / C;  // rows taken side by side
    __shared__ __align__(16) bf16 t[C][kTileP];
    __shared__ float red[kGroups][C];
    const int c = threadIdx.x % C, rg = threadIdx.x / C;
    float sum = 0.0f;
    for (int m0 = blockIdx.x * kTileM; m0 < M; m0 += gridDim.x * kTileM) {
#pragma unroll 8
        for (int r = rg; r < kTileM; r += kGroups) {
            const int m = m0 + r;
            bf16 o = __float2bfloat16_rn(0.0f);
            if (m < M) {
                float v;
                if (kSrc == GradSrc::kPlain) {
                    v = src[(size_t)m * C + c];
                } else if (kSrc == GradSrc::kPool) {
                    v = src[(size_t)(m / P) * C + c] / (float)P;
                } else {
                    const int ix = m % W, iy = m / W % H, b = m / (W * H);
                    v = 0.0f;
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky) {
                        const int ty = iy + 1 - ky;
                        if (ty < 0 || (ty & 1) || (ty >> 1) >= Ho) continue;
#pragma unroll
                        for (int kx = 0; kx < 3; ++kx) {
                            const int tx = ix + 1 - kx;
                            if (tx < 0 || (tx & 1) || (tx >> 1) >= Wo) continue;
                            const size_t q = ((size_t)b * Ho + (ty >> 1)) * Wo + (tx >> 1);
                            v += src[q * Kp + (ky * 3 + kx) * C + c];
                        }
                    }
                }
                if (act && !(__bfloat162float(act[(size_t)m * C + c]) > 0.0f)) v = 0.0f;
                sum += v;
                o = __float2bfloat16_rn(v);
                if (gb) gb[(size_t)m * C + c] = o;
            }
            t[c][r] = o;
        }
        __syncthreads();
        put_transposed<C>(t, m0, M, gbT);
        __syncthreads();
    }
    red[rg][c] = sum;
    __syncthreads();
    if (rg == 0) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < kGroups; ++k) s += red[k][c];
        part[(size_t)c * gridDim.x + blockIdx.x] = s;
    }
}

// The bias gradients of all layers from k_grad's sums per CTA: a CTA per
// column, whose threads take every 256th sum and join in a tree.  Latency-bound,
// 4.7 us: a gradient step at batch 256 takes 678 us, and 672 with one atomic per
// CTA and column, whose order changes from run to run.
struct BiasJob {
    const float* part;
    float* db;
    int ctas, cols;
};
constexpr int kBiases = kConvs + 2;
struct BiasJobs {
    BiasJob j[kBiases];
    int n, cols;  // cols: of all of them, a CTA each
};
__global__ void __launch_bounds__(kThreads) k_bias_sum(BiasJobs jobs) {
    chain_begin();
    int c = (int)blockIdx.x, k = 0;
    while (c >= jobs.j[k].cols) c -= jobs.j[k++].cols;
    const BiasJob& q = jobs.j[k];
    float s = 0.0f;
#pragma unroll 5
    for (int b = threadIdx.x; b < q.ctas; b += kThreads) s += q.part[(size_t)c * q.ctas + b];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ float red[kThreads / 32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0.0f;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) s += red[w];
        q.db[c] = s;
    }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; masked entries stay
// zero; writes the BF16 copies
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, const unsigned char* __restrict__ mask, size_t n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2, bf16* __restrict__ pb) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (mask[i]) {
            const float gi = g[i];
            const float a = b1 * m1[i] + (1.0f - b1) * gi;
            const float s = b2 * m2[i] + (1.0f - b2) * gi * gi;
            m1[i] = a;
            m2[i] = s;
            v = p[i] - lr * (a / bc1) / (sqrtf(s / bc2) + eps);
        }
        p[i] = v;
        pb[i] = __float2bfloat16_rn(v);
    }
}

__global__ void k_to_bf16(const float* __restrict__ p, size_t n, bf16* __restrict__ pb) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        pb[i] = __float2bfloat16_rn(p[i]);
}

}  // namespace

struct kifi_proposer {
    int device = 0, max_batch = 0;
    cudaStream_t stream = nullptr;
    unsigned int* status = nullptr;  // GEMM wait status
    float* loss = nullptr;
    // parameters (FP32 master, gradients, Adam moments), BF16 copies, trainable mask
    float *p = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;
    bf16* pb = nullptr;
    unsigned char* mask = nullptr;
    long long step = 0;
    // activations and scratch
    __half* x = nullptr;                 // the network input [B][60][80][2]
    bf16* col = nullptr;                 // convolution 1's im2col [M][Kp]
    bf16* colT[kConvs] = {};             // transposed im2col matrices [Kp][M] (training)
    float* y = nullptr;                  // the hidden layer's gradient, FP32 [B][64]
    float* y2 = nullptr;                 // FP32 scratch: dout, dgap, dcol
    bf16* act[kConvs] = {};              // conv activations [M][Cout]
    bf16 *gap = nullptr, *gapT = nullptr;   // [B][128], [128][B]
    bf16 *h1 = nullptr, *h1T = nullptr;     // [B][64], [64][B]
    float* out = nullptr;                   // [B][16]
    bf16 *dbf = nullptr, *dbfT = nullptr;   // BF16 gradient [M][C] and transpose
    float* bias_part = nullptr;             // column sums per CTA of the gradient passes
    bf16* wT[12] = {};                      // transposed weights (those whose layer passes a gradient on)
};

namespace {

size_t conv_m(int l, int batch) { return (size_t)batch * kHout[l] * kWout[l]; }

kifi_status gemm(kifi_proposer* pr, const void* A, const void* B, float* C, int M, int N, int K, int lda, int ldb,
                 int ldc, int k_split, bool acc, const GemmEpilogue* epi = nullptr) {
    KIFI_CUDA(gemm_bf16_enqueue(A, B, C, M, N, K, lda, ldb, ldc, k_split, acc, pr->status, pr->stream, epi));
    return KIFI_OK;
}
// CTAs of a gradient pass, 64 rows a tile, at most eight on each of the GPU's 152 SMs
int tile_grid(int M) { return std::min((M + kTileM - 1) / kTileM, 8 * 152); }
// floats of the gradient passes' column sums
size_t bias_part_size(int batch) {
    size_t n = (size_t)tile_grid(batch) * (kOutPad + kFc1);
    for (int l = 0; l < kConvs; ++l) n += (size_t)tile_grid((int)conv_m(l, batch)) * kCout[l];
    return n;
}

const bf16* wb(const kifi_proposer* pr, int t) { return pr->pb + kLayout.off[t]; }
const float* pf(const kifi_proposer* pr, int t) { return pr->p + kLayout.off[t]; }
float* gf(kifi_proposer* pr, int t) { return pr->g + kLayout.off[t]; }

// forward pass; with `train` the transposed im2col matrices are written for
// the weight gradients.  Convolutions 2-4 run as implicit GEMMs over the previous
// activation; convolution 1 (Cin = 2) through its im2col matrix.  Bias and
// ReLU are applied in the GEMM epilogue, which writes the BF16 activation.
kifi_status forward(kifi_proposer* pr, int batch, bool train) {
    kifi_status s;
    cudaStream_t st = pr->stream;
    for (int l = 0; l < kConvs; ++l) {
        const int M = (int)conv_m(l, batch);
        if (l == 0) {
            if (train) k_im2col_first<true><<<blocks(M), kThreads, 0, st>>>(pr->x, batch, pr->col, pr->colT[0]);
            else k_im2col_first<false><<<blocks(M), kThreads, 0, st>>>(pr->x, batch, pr->col, nullptr);
        } else if (train) {
            const dim3 tiles((M + kTileM - 1) / kTileM, 9);
            if (l == 1) k_im2col_t<1><<<tiles, kThreads, 0, st>>>(pr->act[0], batch, pr->colT[1]);
            else if (l == 2) k_im2col_t<2><<<tiles, kThreads, 0, st>>>(pr->act[1], batch, pr->colT[2]);
            else k_im2col_t<3><<<tiles, kThreads, 0, st>>>(pr->act[2], batch, pr->colT[3]);
        }
        KIFI_CUDA(cudaGetLastError());
        GemmEpilogue epi;
        epi.bias = pf(pr, 2 * l + 1);
        epi.relu = true;
        epi.out_bf16 = pr->act[l];
        if (l == 0) {
            if ((s = gemm(pr, pr->col, wb(pr, 0), nullptr, M, kCout[0], kKp[0], kKp[0], kKp[0], kCout[0], 0, false,
                          &epi)))
                return s;
        } else {
            KIFI_CUDA(conv3x3s2_bf16_enqueue(pr->act[l - 1], batch, kHin[l], kWin[l], kCin[l], wb(pr, 2 * l),
                                             kCout[l], kKp[l], epi.bias, true, pr->act[l], pr->status, st));
        }
    }
    k_gap<<<blocks((size_t)batch * 128), kThreads, 0, st>>>(pr->act[3], batch, kHout[3] * kWout[3], 128, pr->gap);
    GemmEpilogue e1;
    e1.bias = pf(pr, 9);
    e1.relu = true;
    e1.out_bf16 = pr->h1;
    if ((s = gemm(pr, pr->gap, wb(pr, 8), nullptr, batch, kFc1, 128, 128, 128, kFc1, 0, false, &e1))) return s;
    GemmEpilogue e2;
    e2.bias = pf(pr, 11);
    if ((s = gemm(pr, pr->h1, wb(pr, 10), pr->out, batch, kOutPad, kFc1, kFc1, kFc1, kOutPad, 0, false, &e2)))
        return s;
    KIFI_CUDA(cudaGetLastError());
    return KIFI_OK;
}

// backward pass from dL/dout (FP32 in pr->y2 [B][16], BF16 in pr->dbf) into pr->g
kifi_status backward(kifi_proposer* pr, int batch) {
    kifi_status s;
    cudaStream_t st = pr->stream;
    KIFI_CUDA(cudaMemsetAsync(pr->g, 0, kLayout.total * sizeof(float), st));
    {  // every transpose that waits for nothing of the backward pass
        TransposeJobs tj{};
        int tiles = 0;
        auto add = [&](const bf16* in, int R, int C, bf16* out) {
            tj.j[tj.n++] = TransposeJob{in, out, R, C, tiles};
            tiles += ((R + 31) / 32) * ((C + 31) / 32);
        };
        add(pr->h1, batch, kFc1, pr->h1T);
        add(pr->gap, batch, 128, pr->gapT);
        add(wb(pr, 10), kOutPad, kFc1, pr->wT[10]);
        add(wb(pr, 8), kFc1, 128, pr->wT[8]);
        for (int l = 1; l < kConvs; ++l) add(wb(pr, 2 * l), kCout[l], kKp[l], pr->wT[2 * l]);
        k_transpose<<<tiles, dim3(32, 8), 0, st>>>(tj);
    }
    BiasJobs bj{};
    float* next = pr->bias_part;
    // the place of a pass's column sums, whose total goes to parameter t's gradient
    auto sums = [&](int t, int ctas, int cols) {
        bj.j[bj.n++] = BiasJob{next, gf(pr, t), ctas, cols};
        bj.cols += cols;
        float* const at = next;
        next += (size_t)ctas * cols;
        return at;
    };
    // fc2: db2 = colsum(dout), dW2 [16 x 64] = dout^T h1, dh1 = dout W2
    k_grad<kOutPad, GradSrc::kPlain><<<tile_grid(batch), kThreads, 0, st>>>(pr->y2, nullptr, batch, nullptr,
                                                                          pr->dbfT, sums(11, tile_grid(batch), kOutPad));
    if ((s = gemm(pr, pr->dbfT, pr->h1T, gf(pr, 10), kOutPad, kFc1, batch, batch, batch, kFc1, batch, true)))
        return s;
    if ((s = gemm(pr, pr->dbf, pr->wT[10], pr->y, batch, kFc1, kOutPad, kOutPad, kOutPad, kFc1, 0, false))) return s;
    // fc1: through its ReLU; db1, dW1 [64 x 128] = dh^T gap, dgap = dh W1
    k_grad<kFc1, GradSrc::kPlain><<<tile_grid(batch), kThreads, 0, st>>>(pr->y, pr->h1, batch, pr->dbf,
                                                                       pr->dbfT, sums(9, tile_grid(batch), kFc1));
    if ((s = gemm(pr, pr->dbfT, pr->gapT, gf(pr, 8), kFc1, 128, batch, batch, batch, 128, batch, true))) return s;
    if ((s = gemm(pr, pr->dbf, pr->wT[8], pr->y2, batch, 128, kFc1, kFc1, kFc1, 128, 0, false))) return s;
    for (int l = kConvs - 1; l >= 0; --l) {
        const int M = (int)conv_m(l, batch), Co = kCout[l], Kp = kKp[l], grid = tile_grid(M);
        // the pre-activation's gradient, from the pool (y2 [B][128]) or from
        // the convolution above (y2 = its dcol)
        bf16* const db = pr->dbf;
        bf16* const dt = pr->dbfT;
        float* const bias = sums(2 * l + 1, grid, kCout[l]);
        if (l == 3) k_grad<128, GradSrc::kPool><<<grid, kThreads, 0, st>>>(pr->y2, pr->act[3], M, db, dt, bias);
        else if (l == 2) k_grad<64, GradSrc::kConv, 3><<<grid, kThreads, 0, st>>>(pr->y2, pr->act[2], M, db, dt, bias);
        else if (l == 1) k_grad<64, GradSrc::kConv, 2><<<grid, kThreads, 0, st>>>(pr->y2, pr->act[1], M, db, dt, bias);
        else k_grad<32, GradSrc::kConv, 1><<<grid, kThreads, 0, st>>>(pr->y2, pr->act[0], M, nullptr, dt, bias);
        // dW [Co x Kp] = dY^T col, inner M split across CTAs
        if ((s = gemm(pr, pr->dbfT, pr->colT[l], gf(pr, 2 * l), Co, Kp, M, M, M, Kp, 4096, true))) return s;
        if (l == 0) break;
        // dcol = dY W for the layer below
        if ((s = gemm(pr, pr->dbf, pr->wT[2 * l], pr->y2, M, Kp, Co, Co, Co, Kp, 0, false))) return s;
    }
    KIFI_CUDA(chain_launch(true, dim3(bj.cols), dim3(kThreads), st, k_bias_sum, bj));
    KIFI_CUDA(cudaGetLastError());
    return KIFI_OK;
}

kifi_status take_status(kifi_proposer* pr) {
    unsigned int h = 0;
    KIFI_CUDA(cudaMemcpyAsync(&h, pr->status, sizeof h, cudaMemcpyDeviceToHost, pr->stream));
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    if (h) {
        KIFI_CUDA(cudaMemsetAsync(pr->status, 0, sizeof(unsigned int), pr->stream));
        return fail(KIFI_ERR_TIMEOUT, "proposer: a bounded device wait gave up");
    }
    return KIFI_OK;
}

kifi_status check_batch(kifi_proposer* pr, int batch) {
    if (batch <= 0 || batch > pr->max_batch || batch % 8)
        return fail(KIFI_ERR_INVALID_ARGUMENT, "proposer batch must be a positive multiple of 8 up to max_batch");
    return KIFI_OK;
}

}  // namespace

extern "C" {

kifi_status kifi_proposer_destroy(kifi_proposer* pr) {
    if (!pr) return KIFI_OK;
    if (pr->stream) cudaStreamSynchronize(pr->stream);
    void* bufs[] = {pr->status, pr->loss, pr->p, pr->g, pr->m1, pr->m2, pr->pb, pr->mask, pr->x, pr->y, pr->y2,
                    pr->gap, pr->gapT, pr->h1, pr->h1T, pr->out, pr->dbf, pr->dbfT, pr->col, pr->bias_part};
    for (void* b : bufs) cudaFree(b);
    for (int l = 0; l < kConvs; ++l) {
        cudaFree(pr->colT[l]);
        cudaFree(pr->act[l]);
    }
    for (bf16* w : pr->wT) cudaFree(w);
    if (pr->stream) cudaStreamDestroy(pr->stream);
    delete pr;
    return KIFI_OK;
}

kifi_status kifi_proposer_create(int device, int max_batch, kifi_proposer** out) {
    if (!out || max_batch <= 0 || max_batch % 8) return fail(KIFI_ERR_INVALID_ARGUMENT, "bad argument");
    *out = nullptr;
    kifi_proposer* pr = new (std::nothrow) kifi_proposer();
    if (!pr) return fail(KIFI_ERR_OUT_OF_MEMORY, "host allocation");
    pr->device = device;
    pr->max_batch = max_batch;
    const size_t B = (size_t)max_batch, P = kLayout.total;
    cudaError_t e = cudaSetDevice(device);
    if (!e) e = cudaStreamCreateWithFlags(&pr->stream, cudaStreamNonBlocking);
    auto alloc = [&](auto** ptr, size_t bytes) {
        if (!e) e = cudaMalloc((void**)ptr, bytes);
    };
    alloc(&pr->status, 16);
    alloc(&pr->loss, 16);
    alloc(&pr->p, P * 4);
    alloc(&pr->g, P * 4);
    alloc(&pr->m1, P * 4);
    alloc(&pr->m2, P * 4);
    alloc(&pr->pb, P * 2);
    alloc(&pr->mask, P);
    alloc(&pr->x, B * kInH * kInW * kInC * 2);
    size_t colmax = 0, dmax = 0;
    for (int l = 0; l < kConvs; ++l) {
        const size_t M = conv_m(l, max_batch);
        if (l == 0) alloc(&pr->col, M * kKp[0] * 2);
        alloc(&pr->colT[l], M * kKp[l] * 2);
        alloc(&pr->act[l], M * kCout[l] * 2);
        colmax = std::max(colmax, M * (size_t)kKp[l]);
        dmax = std::max(dmax, M * (size_t)kCout[l]);
    }
    alloc(&pr->y, B * kFc1 * 4);
    alloc(&pr->y2, std::max(colmax, B * 128) * 4);
    alloc(&pr->gap, B * 128 * 2);
    alloc(&pr->gapT, B * 128 * 2);
    alloc(&pr->h1, B * kFc1 * 2);
    alloc(&pr->h1T, B * kFc1 * 2);
    alloc(&pr->out, B * kOutPad * 4);
    alloc(&pr->dbf, dmax * 2);
    alloc(&pr->dbfT, dmax * 2);
    alloc(&pr->bias_part, bias_part_size(max_batch) * 4);
    for (int t = 2; t <= 10; t += 2) alloc(&pr->wT[t], kLayout.size[t] * 2);
    if (!e) e = cudaMemsetAsync(pr->status, 0, 16, pr->stream);
    if (!e) e = cudaMemsetAsync(pr->p, 0, P * 4, pr->stream);
    if (!e) e = cudaMemsetAsync(pr->m1, 0, P * 4, pr->stream);
    if (!e) e = cudaMemsetAsync(pr->m2, 0, P * 4, pr->stream);
    if (!e) e = cudaMemsetAsync(pr->pb, 0, P * 2, pr->stream);
    if (!e) {  // trainable mask: everything but the padding
        std::vector<unsigned char> m(P, 0);
        for (int t = 0; t < 12; ++t)
            for (size_t i = 0; i < kLayout.size[t]; ++i) {
                bool on = true;
                if (t == 0) on = (i % 32) < 18;         // conv 1: K = 18 of 32
                if (t == 10) on = (i / kFc1) < kOut;    // output rows 0..5
                if (t == 11) on = i < (size_t)kOut;
                m[kLayout.off[t] + i] = on ? 1 : 0;
            }
        // on the proposer's stream (non-blocking: it would not wait for the legacy default stream)
        e = cudaMemcpyAsync(pr->mask, m.data(), P, cudaMemcpyHostToDevice, pr->stream);
        if (!e) e = cudaStreamSynchronize(pr->stream);
    }
    if (e) {
        kifi_proposer_destroy(pr);
        return cuda_fail(e, "proposer allocation");
    }
    *out = pr;
    return KIFI_OK;
}

kifi_status kifi_proposer_param_count(kifi_proposer* pr, size_t* n) {
    if (!pr || !n) return fail(KIFI_ERR_INVALID_ARGUMENT, "null argument");
    *n = kLayout.total;
    return KIFI_OK;
}

kifi_status kifi_proposer_set_params(kifi_proposer* pr, const float* host, size_t n) {
    if (!pr || !host || n != kLayout.total) return fail(KIFI_ERR_INVALID_ARGUMENT, "bad parameter vector");
    KIFI_CUDA(cudaSetDevice(pr->device));
    KIFI_CUDA(cudaMemcpyAsync(pr->p, host, n * 4, cudaMemcpyHostToDevice, pr->stream));
    k_to_bf16<<<blocks(n), kThreads, 0, pr->stream>>>(pr->p, n, pr->pb);
    KIFI_CUDA(cudaMemsetAsync(pr->m1, 0, n * 4, pr->stream));
    KIFI_CUDA(cudaMemsetAsync(pr->m2, 0, n * 4, pr->stream));
    pr->step = 0;
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    return KIFI_OK;
}

kifi_status kifi_proposer_get_params(kifi_proposer* pr, float* host, size_t n) {
    if (!pr || !host || n != kLayout.total) return fail(KIFI_ERR_INVALID_ARGUMENT, "bad parameter vector");
    KIFI_CUDA(cudaSetDevice(pr->device));
    KIFI_CUDA(cudaMemcpyAsync(host, pr->p, n * 4, cudaMemcpyDeviceToHost, pr->stream));
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    return KIFI_OK;
}

kifi_status kifi_proposer_make_input(kifi_proposer* pr, const void* depth_a_dev, const void* depth_b_dev,
                                     int depth_is_u16, int width, int height, void* out_fp16_dev) {
    if (!pr || !depth_a_dev || !depth_b_dev || !out_fp16_dev || width % kInW || height % kInH || width <= 0 ||
        height <= 0)
        return fail(KIFI_ERR_INVALID_ARGUMENT, "bad argument (frames must be multiples of 80 x 60)");
    KIFI_CUDA(cudaSetDevice(pr->device));
    k_downsample<<<blocks(kInH * kInW * 2), kThreads, 0, pr->stream>>>(depth_a_dev, depth_b_dev, depth_is_u16,
                                                                       width, height, (__half*)out_fp16_dev);
    KIFI_CUDA(cudaGetLastError());
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    return KIFI_OK;
}

kifi_status kifi_proposer_set_inputs(kifi_proposer* pr, const void* inputs_fp16_dev, int batch) {
    if (!pr || !inputs_fp16_dev) return fail(KIFI_ERR_INVALID_ARGUMENT, "null argument");
    kifi_status s = check_batch(pr, batch);
    if (s) return s;
    KIFI_CUDA(cudaSetDevice(pr->device));
    KIFI_CUDA(cudaMemcpyAsync(pr->x, inputs_fp16_dev, (size_t)batch * kInH * kInW * kInC * 2,
                              cudaMemcpyDeviceToDevice, pr->stream));
    return KIFI_OK;
}

kifi_status kifi_proposer_get_inputs(kifi_proposer* pr, void* out_fp16_dev, int batch) {
    if (!pr || !out_fp16_dev) return fail(KIFI_ERR_INVALID_ARGUMENT, "null argument");
    kifi_status s = check_batch(pr, batch);
    if (s) return s;
    KIFI_CUDA(cudaSetDevice(pr->device));
    KIFI_CUDA(cudaMemcpyAsync(out_fp16_dev, pr->x, (size_t)batch * kInH * kInW * kInC * 2,
                              cudaMemcpyDeviceToDevice, pr->stream));
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    return KIFI_OK;
}

kifi_status kifi_proposer_predict(kifi_proposer* pr, int batch, float* out_twists_host) {
    if (!pr || !out_twists_host) return fail(KIFI_ERR_INVALID_ARGUMENT, "null argument");
    kifi_status s = check_batch(pr, batch);
    if (s) return s;
    KIFI_CUDA(cudaSetDevice(pr->device));
    if ((s = forward(pr, batch, false))) return s;
    std::vector<float> o((size_t)batch * kOutPad);
    KIFI_CUDA(cudaMemcpyAsync(o.data(), pr->out, o.size() * 4, cudaMemcpyDeviceToHost, pr->stream));
    if ((s = take_status(pr))) return s;
    for (int b = 0; b < batch; ++b)
        for (int j = 0; j < kOut; ++j) out_twists_host[b * kOut + j] = o[(size_t)b * kOutPad + j];
    return KIFI_OK;
}

kifi_status kifi_proposer_gradients(kifi_proposer* pr, const float* targets_dev, int batch, float* out_loss,
                                    float* out_grads_host) {
    if (!pr || !targets_dev) return fail(KIFI_ERR_INVALID_ARGUMENT, "null argument");
    kifi_status s = check_batch(pr, batch);
    if (s) return s;
    KIFI_CUDA(cudaSetDevice(pr->device));
    if ((s = forward(pr, batch, true))) return s;
    KIFI_CUDA(cudaMemsetAsync(pr->loss, 0, 4, pr->stream));
    k_mse<<<blocks((size_t)batch * kOutPad), kThreads, 0, pr->stream>>>(pr->out, targets_dev, batch, pr->y2,
                                                                        pr->dbf, pr->loss);
    if ((s = backward(pr, batch))) return s;
    if (out_loss) KIFI_CUDA(cudaMemcpyAsync(out_loss, pr->loss, 4, cudaMemcpyDeviceToHost, pr->stream));
    if (out_grads_host)
        KIFI_CUDA(cudaMemcpyAsync(out_grads_host, pr->g, kLayout.total * 4, cudaMemcpyDeviceToHost, pr->stream));
    return take_status(pr);
}

kifi_status kifi_proposer_train_step(kifi_proposer* pr, const float* targets_dev, int batch, float lr,
                                     float* out_loss) {
    kifi_status s = kifi_proposer_gradients(pr, targets_dev, batch, out_loss, nullptr);
    if (s) return s;
    ++pr->step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.0f - (float)std::pow(b1, (double)pr->step), bc2 = 1.0f - (float)std::pow(b2, (double)pr->step);
    k_adam<<<blocks(kLayout.total), kThreads, 0, pr->stream>>>(pr->p, pr->g, pr->m1, pr->m2, pr->mask,
                                                              kLayout.total, lr, b1, b2, 1e-8f, bc1, bc2, pr->pb);
    KIFI_CUDA(cudaGetLastError());
    KIFI_CUDA(cudaStreamSynchronize(pr->stream));
    return KIFI_OK;
}

}  // extern "C"
