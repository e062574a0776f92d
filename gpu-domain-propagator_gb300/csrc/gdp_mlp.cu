// gdp_mlp.cu -- training and inference kernels of the row-marking MLP
// (16 -> 64 -> 64 -> 1, ReLU, BF16 weights/activations, FP32 accumulation)
// and its C-ABI (gdp_mlp_*).
//
// Training minimises the weighted binary cross-entropy of sigmoid(z) against
// the label "processing this row tightened a bound" with Adam on FP32 master
// weights; BF16 copies are refreshed after every step.
//
// Backward of one 16-sample tile (one warp), in the forward's fragment layout:
//   dz      = w (sigmoid(z) - y) / sum(w)
//   g_w3   += dz relu(a2),            g_b3 += dz
//   da2     = dz w3 [a2 > 0]          (FP32)
//   g_W2   += da2^T bf16(relu(a1)),   g_b2 += da2        (FP32, CUDA cores)
//   dh1     = bf16(da2) @ W2          (tensor cores, W2^T as the B operand)
//   da1     = dh1 [a1 > 0]
//   g_W1   += da1^T x,                g_b1 += da1        (FP32, CUDA cores)
// Each warp adds its tiles' weight gradients to sums of its own in shared
// memory, a CTA writes the sum over its warps to its row of a partial array, and
// the optimizer step (or the gradient call) adds up the rows: no atomics, and
// every sum in a fixed order, so equal calls give equal bits.
#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "gdp_context.h"
#include "gdp_mlp.h"
#include "gdp_pages.h"

namespace gdp {

namespace {

constexpr int kMlpWarps = 4;
constexpr int kMlpThreads = 32 * kMlpWarps;

// Per-warp scratch of a tile (FP32) and the warp's gradient sums. da holds da2
// and then da1, transposed: the 16 samples of a column are 64 consecutive bytes,
// four 16-byte loads that every lane of the warp shares (rows of 20 floats:
// aligned, and the stores of a fragment's columns fall in different banks).
constexpr int kTileLd = kMlpH + 8;
struct TileSmem {
    float da[kMlpH][20];
    float h1[16][kTileLd];
    float x[16][kMlpIn];
    float sum[(kMlpParams + 4) & ~3];  // parameters, then the loss
};
constexpr int kPartLd = kMlpParams + 1;  // a CTA's row of the partial sums: gradient, loss
constexpr int kGradWarpsFew = 4, kGradWarpsMany = 7;  // 32 KB of shared memory per warp

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Samples [r0, r0 + 16) of [0, n), sample r being number perm[r] (perm null: r)
// of a row-major BF16 [.][16] array: A registers, labels and weights of rows g
// and g + 8, zero past n.
__device__ __forceinline__ void load_samples(const __nv_bfloat16 *X, const int *perm, const float *y, const float *w,
                                             int n, int r0, int lane, unsigned (&a)[4], float (&yy)[2],
                                             float (&ww)[2]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = r0 + g + 8 * h;
        a[h] = a[2 + h] = 0u;
        yy[h] = ww[h] = 0.f;
        if (r < n) {
            const int k = perm ? __ldg(perm + r) : r;
            const unsigned *x = reinterpret_cast<const unsigned *>(X + (size_t)k * kMlpIn) + t;
            a[h] = __ldg(x);
            a[2 + h] = __ldg(x + 4);
            yy[h] = __ldg(y + k);
            ww[h] = __ldg(w + k);
        }
    }
}

// Logits of n rows of FP32 features. X and z may be host memory that the device
// reaches directly: the features are read once, where they are, 1 KB per warp
// and tile in whole lines with the next tile in flight, rounded to BF16 on the
// way and passed to the fragment layout through shared memory; a copy to the
// device and a conversion pass are left out. What bounds it is
// the rate of those reads over NVLink-C2C (1M rows, 64 MB: 0.41 ms, 165 GB/s,
// against 0.93 ms with the copies).
__global__ void __launch_bounds__(kMlpThreads) k_mlp_forward(MlpDev M, const float *__restrict__ X, int n, float *z) {
    __shared__ __align__(16) __nv_bfloat16 tile[kMlpWarps][16][kMlpIn];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int tiles = (n - 1) / 16 + 1;
    const float4 *X4 = reinterpret_cast<const float4 *>(X);
    const long long have = (long long)n * (kMlpIn / 4);  // float4s of X
    auto load = [&](int t, float4 (&v)[2]) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const long long at = (long long)t * 64 + 32 * i + lane;
            v[i] = t < tiles && at < have ? __ldcs(X4 + at) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    float4 v[2];
    load(warp, v);
    for (int t = warp; t < tiles; t += nwarps) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; i++)
            *(reinterpret_cast<uint2 *>(&tile[wid][0][0]) + 32 * i + lane) =
                    make_uint2(pack_bf16(v[i].x, v[i].y), pack_bf16(v[i].z, v[i].w));
        __syncwarp();
        load(t + nwarps, v);
        unsigned a[4];
        load_a_smem(&tile[wid][0][0], lane, a);
        float z0, z1;
        mlp_infer_tile(M, a, lane, z0, z1);
        const int r = 16 * t + (lane >> 2);
        if ((lane & 3) == 0) {
            if (r < n) z[r] = z0;
            if (r + 8 < n) z[r + 8] = z1;
        }
    }
}

// Gradient of the weighted BCE over samples [0, n) (sample r is perm[r], or r):
// row blockIdx.x of part receives the CTA's sums and its loss. W warps per CTA,
// one CTA per SM. A minibatch of 8,192 is 512 tiles, one per warp of 128 CTAs:
// what bounds it is the time of one tile on one warp -- forward, 64 x 64 and
// 64 x 16 FP32 outer products of 16 samples -- 11 us, of which the FP32
// multiply-adds need 1.4. The outer products keep four rows in flight, and their
// row values come four to a load. Gradients added by shared and global atomics
// took 24 us and 19 on clearing them, the Adam step and the BF16 copies; a step
// of this kernel and k_mlp_step is 16 us (46 before).
template <int W>
__global__ void __launch_bounds__(32 * W) k_mlp_grad(MlpDev M, const __nv_bfloat16 *X, const int *perm, const float *y,
                                                     const float *w, int n, float inv_wsum, float *part) {
    extern __shared__ float4 smem_raw[];
    TileSmem *tiles = reinterpret_cast<TileSmem *>(smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    TileSmem &S = tiles[wid];
    for (int i = lane; i < kPartLd; i += 32) S.sum[i] = 0.f;
    float *gW1 = S.sum + kOffW1, *gb1 = S.sum + kOffB1, *gW2 = S.sum + kOffW2, *gb2 = S.sum + kOffB2,
          *gw3 = S.sum + kOffW3;
    const int g = lane >> 2, t = lane & 3;
    const int ntiles = (n - 1) / 16 + 1;
    float lsum = 0.f, b3sum = 0.f;
    __syncwarp();
    int tile = blockIdx.x * W + wid;
    unsigned an[4];  // the next tile's samples
    float yn[2], wn[2];
    load_samples(X, perm, y, w, tile < ntiles ? n : 0, 16 * (tile < ntiles ? tile : 0), lane, an, yn, wn);
    // up to here the kernel may run while the optimizer step before it ends
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    while (tile < ntiles) {
        const int r0 = 16 * tile;
        unsigned a[4];
        float yy[2], ww[2];
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = an[q];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            yy[h] = yn[h];
            ww[h] = wn[h];
        }
        tile = ntiles - tile > gridDim.x * W ? tile + gridDim.x * W : ntiles;
        if (tile < ntiles) load_samples(X, perm, y, w, n, 16 * tile, lane, an, yn, wn);
        MlpTile T;
        mlp_forward_tile(M, a, lane, T);
        // the tile's inputs (FP32 copy of the A registers)
        {
            const __nv_bfloat162 *v = reinterpret_cast<const __nv_bfloat162 *>(a);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 f = __bfloat1622float2(v[q]);
                *reinterpret_cast<float2 *>(&S.x[g + 8 * (q & 1)][2 * t + 8 * (q >> 1)]) = f;
            }
        }
        // per-row dz (rows g and g + 8)
        float dz[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            dz[h] = 0.f;
            if (r0 + g + 8 * h < n) {
                const float zz = T.z[h], p = 1.f / (1.f + __expf(-zz));
                dz[h] = ww[h] * (p - yy[h]) * inv_wsum;
                // BCE with logits: max(z, 0) - z y + log(1 + exp(-|z|))
                if (t == 0) lsum += ww[h] * (fmaxf(zz, 0.f) - zz * yy[h] + log1pf(__expf(-fabsf(zz)))) * inv_wsum;
            }
        }
        if (t == 0) b3sum += dz[0] + dz[1];
        // layer 3, da2 and the layer-1 activations; da2's A registers for dh1
        unsigned da[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
            float d[4];
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int col = nt * 8 + 2 * t + c;
                const float w3 = __bfloat162float(M.w3[col]);
                const float h0 = fmaxf(T.a2[nt][c], 0.f), h8 = fmaxf(T.a2[nt][2 + c], 0.f);
                float gw = dz[0] * h0 + dz[1] * h8;
                gw += __shfl_xor_sync(0xffffffffu, gw, 4);
                gw += __shfl_xor_sync(0xffffffffu, gw, 8);
                gw += __shfl_xor_sync(0xffffffffu, gw, 16);
                if (g == 0) gw3[col] += gw;
                d[c] = T.a2[nt][c] > 0.f ? dz[0] * w3 : 0.f;
                d[2 + c] = T.a2[nt][2 + c] > 0.f ? dz[1] * w3 : 0.f;
                S.da[col][g] = d[c];
                S.da[col][g + 8] = d[2 + c];
                S.h1[g][col] = bf16r(fmaxf(T.a1[nt][c], 0.f));
                S.h1[g + 8][col] = bf16r(fmaxf(T.a1[nt][2 + c], 0.f));
            }
            da[nt >> 1][2 * (nt & 1)] = pack_bf16(d[0], d[1]);
            da[nt >> 1][2 * (nt & 1) + 1] = pack_bf16(d[2], d[3]);
        }
        __syncwarp();
        // weight gradients of the tile, each a sum over its 16 samples in
        // sample order: column `row` of da against the samples' inputs
        auto column = [&](int row, float (&d)[16]) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 v = *reinterpret_cast<const float4 *>(&S.da[row][4 * q]);
                d[4 * q] = v.x; d[4 * q + 1] = v.y; d[4 * q + 2] = v.z; d[4 * q + 3] = v.w;
            }
        };
        {  // W2: lane owns columns lane and lane + 32 of every row; b2: rows lane and lane + 32
            float hl[16], hh[16];
#pragma unroll
            for (int s = 0; s < 16; s++) {
                hl[s] = S.h1[s][lane];
                hh[s] = S.h1[s][lane + 32];
            }
            for (int row = 0; row < kMlpH; row += 4) {  // four rows' chains in flight
                float d[4][16], vl[4], vh[4], ol[4], oh[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    column(row + u, d[u]);
                    ol[u] = gW2[(row + u) * kMlpH + lane];
                    oh[u] = gW2[(row + u) * kMlpH + lane + 32];
                    vl[u] = vh[u] = 0.f;
                }
#pragma unroll
                for (int s = 0; s < 16; s++)
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        vl[u] = fmaf(d[u][s], hl[s], vl[u]);
                        vh[u] = fmaf(d[u][s], hh[s], vh[u]);
                    }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    gW2[(row + u) * kMlpH + lane] = ol[u] + vl[u];
                    gW2[(row + u) * kMlpH + lane + 32] = oh[u] + vh[u];
                }
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                float d[16], v = 0.f;
                column(lane + 32 * q, d);
#pragma unroll
                for (int s = 0; s < 16; s++) v += d[s];
                gb2[lane + 32 * q] += v;
            }
        }
        // dh1 = bf16(da2) @ W2 on the tensor cores; da1 takes da2's place
        __syncwarp();
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kt = 0; kt < 4; kt++) {
                unsigned b0, b1;
                load_bfrag(M.w2t, 4, nt, kt, lane, b0, b1);
                mma_bf16(c, da[kt], b0, b1);
            }
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const int col = nt * 8 + 2 * t + cc;
                S.da[col][g] = T.a1[nt][cc] > 0.f ? c[cc] : 0.f;
                S.da[col][g + 8] = T.a1[nt][2 + cc] > 0.f ? c[2 + cc] : 0.f;
            }
        }
        __syncwarp();
        {  // W1: lane owns column lane & 15 of the rows of parity lane >> 4; b1 as b2
            const int k = lane & 15;
            float xs[16];
#pragma unroll
            for (int s = 0; s < 16; s++) xs[s] = S.x[s][k];
            for (int r = lane >> 4; r < kMlpH; r += 8) {
                float d[4][16], v[4], o[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    column(r + 2 * u, d[u]);
                    o[u] = gW1[(r + 2 * u) * kMlpIn + k];
                    v[u] = 0.f;
                }
#pragma unroll
                for (int s = 0; s < 16; s++)
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = fmaf(d[u][s], xs[s], v[u]);
#pragma unroll
                for (int u = 0; u < 4; u++) gW1[(r + 2 * u) * kMlpIn + k] = o[u] + v[u];
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                float d[16], v = 0.f;
                column(lane + 32 * q, d);
#pragma unroll
                for (int s = 0; s < 16; s++) v += d[s];
                gb1[lane + 32 * q] += v;
            }
        }
        __syncwarp();
    }
    for (int off = 16; off > 0; off >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        b3sum += __shfl_xor_sync(0xffffffffu, b3sum, off);
    }
    if (lane == 0) {
        S.sum[kOffB3] = b3sum;
        S.sum[kMlpParams] = lsum;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPartLd; i += 32 * W) {
        float v = tiles[0].sum[i];
#pragma unroll
        for (int q = 1; q < W; q++) v += tiles[q].sum[i];
        part[(size_t)blockIdx.x * kPartLd + i] = v;
    }
}

// Adds up column i of the `rows` partial rows, in order within 8 interleaved
// groups of rows and over the groups: 8 threads per column (threadIdx.y), whose
// loads are coalesced across columns. Every thread of threadIdx.y == 0 returns
// the sum.
constexpr int kSumCols = 32, kSumGroups = 8;
__device__ __forceinline__ float sum_partials(const float *part, int rows, int i, float (&sh)[kSumGroups][kSumCols]) {
    float v = 0.f;
    if (i < kPartLd) {
#pragma unroll 8
        for (int r = threadIdx.y; r < rows; r += kSumGroups) v += __ldcg(part + (size_t)r * kPartLd + i);
    }
    sh[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0) {
        v = sh[0][threadIdx.x];
#pragma unroll
        for (int q = 1; q < kSumGroups; q++) v += sh[q][threadIdx.x];
    }
    return v;
}

__global__ void __launch_bounds__(kSumCols *kSumGroups) k_mlp_sum(const float *part, int rows, float *grad, float *loss) {
    __shared__ float sh[kSumGroups][kSumCols];
    const int i = blockIdx.x * kSumCols + threadIdx.x;
    const float v = sum_partials(part, rows, i, sh);
    if (threadIdx.y == 0 && i < kMlpParams) grad[i] = v;
    if (threadIdx.y == 0 && i == kMlpParams) *loss = v;
}

// BF16 copies of master parameter i: W1, W2, W2 transposed in fragment order
// (frag_index), w3.
__device__ __forceinline__ void cast_param(int i, float v, __nv_bfloat16 *w1, __nv_bfloat16 *w2, __nv_bfloat16 *w2t,
                                           __nv_bfloat16 *w3) {
    static_assert(kMlpIn == 16 && kMlpH % 16 == 0, "one k-tile for layer 1, whole k-tiles for layer 2");
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    if (i < kOffB1) {
        w1[frag_index(i / kMlpIn, i % kMlpIn, 1)] = b;
    } else if (i >= kOffW2 && i < kOffB2) {
        const int r = (i - kOffW2) / kMlpH, c = (i - kOffW2) % kMlpH;
        w2[frag_index(r, c, kMlpH / 16)] = b;
        w2t[frag_index(c, r, kMlpH / 16)] = b;
    } else if (i >= kOffW3 && i < kOffB3) {
        w3[i - kOffW3] = b;
    }
}

// One optimizer step from the partial rows: gradient sums, Adam on the FP32
// master parameters, their BF16 copies, the minibatch's loss. Bound by its chain
// of loads from L2 (4.5 us for 152 rows, 3.2 MB); a last CTA of the gradient
// kernel doing this would read them through one SM.
__global__ void __launch_bounds__(kSumCols *kSumGroups)
        k_mlp_step(const float *part, int rows, float *p, float *m1, float *m2, int step, float lr, float beta1,
                   float beta2, float eps, __nv_bfloat16 *w1, __nv_bfloat16 *w2, __nv_bfloat16 *w2t,
                   __nv_bfloat16 *w3, float *loss) {
    __shared__ float sh[kSumGroups][kSumCols];
    const int i = blockIdx.x * kSumCols + threadIdx.x;
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const float gr = sum_partials(part, rows, i, sh);
    if (threadIdx.y != 0) return;
    if (i == kMlpParams) *loss = gr;
    if (i >= kMlpParams) return;
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    const float a = beta1 * m1[i] + (1.f - beta1) * gr;
    const float b = beta2 * m2[i] + (1.f - beta2) * gr * gr;
    m1[i] = a;
    m2[i] = b;
    const float v = p[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[i] = v;
    cast_param(i, v, w1, w2, w2t, w3);
}

__global__ void k_mlp_cast(const float *p, __nv_bfloat16 *w1, __nv_bfloat16 *w2, __nv_bfloat16 *w2t,
                           __nv_bfloat16 *w3) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x)
        cast_param(i, p[i], w1, w2, w2t, w3);
}

__global__ void k_copy(const float *x, float *y, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = x[i];
}

__global__ void k_to_bf16(const float *x, __nv_bfloat16 *y, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16_rn(x[i]);
}

}  // namespace

// ---- host ---------------------------------------------------------------------
#define GDP_MCUDA(call)                                                                          \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            set_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #call);      \
            return GDP_ERROR;                                                                    \
        }                                                                                        \
    } while (0)

namespace {

unsigned long long splitmix(unsigned long long &s) {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
double uniform01(unsigned long long &s) { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }

int device_sms() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

constexpr int kSumBlocks = (kPartLd + kSumCols - 1) / kSumCols;

// A launch whose blocks may become resident, and run up to their grid
// dependency, while the kernel before it ends (early): the two kernels of a
// training step alternate, each reads what the other wrote only after that.
struct LaunchNext {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    LaunchNext(int grid, dim3 block, size_t smem, bool early, cudaStream_t s) {
        cfg.gridDim = dim3(grid);
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = early;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// Rows of the partial array: at most one CTA per SM.
int grad_rows_max() { return device_sms(); }

// Enqueues the gradient of samples [0, n): one CTA per SM, 4 warps while that
// gives every tile a warp of its own, else 7, what the shared memory holds (most
// warps then have a second one on their SM quarter to overlap with: 2M samples
// take 1.1 ms instead of 1.8).
cudaError_t launch_grad(const MlpDev &M, const __nv_bfloat16 *X, const int *perm, const float *y, const float *w, int n,
                        float inv_wsum, float *part, int *rows, bool early, cudaStream_t s) {
    const int tiles = (n - 1) / 16 + 1, sms = device_sms();
    const bool few = tiles <= sms * kGradWarpsFew;
    const int warps = few ? kGradWarpsFew : kGradWarpsMany;
    *rows = std::min(sms, (tiles + warps - 1) / warps);
    LaunchNext L(*rows, 32 * warps, sizeof(TileSmem) * warps, early, s);
    return few ? cudaLaunchKernelEx(&L.cfg, k_mlp_grad<kGradWarpsFew>, M, X, perm, y, w, n, inv_wsum, part)
               : cudaLaunchKernelEx(&L.cfg, k_mlp_grad<kGradWarpsMany>, M, X, perm, y, w, n, inv_wsum, part);
}

// Forward: every CTA that fits on an SM (the loop waits on its loads, and more
// warps hide them), at most one per 4 tiles.
int forward_grid(int n) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mlp_forward, kMlpThreads, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 2;
    const int tiles = (n - 1) / 16 + 1;
    return std::max(1, std::min(per_sm * device_sms(), (tiles + kMlpWarps - 1) / kMlpWarps));
}
}  // namespace

Mlp::~Mlp() {
    if (stream) cudaStreamSynchronize(stream);
    for (void *q : {(void *)p, (void *)m1, (void *)m2, (void *)grad, (void *)loss, (void *)w1, (void *)w2,
                    (void *)w2t, (void *)w3})
        if (q) cudaFree(q);
    if (stream) cudaStreamDestroy(stream);
}

MlpDev Mlp::dev() const {
    MlpDev d;
    d.w1 = w1; d.w2 = w2; d.w2t = w2t; d.w3 = w3;
    d.b1 = p + kOffB1; d.b2 = p + kOffB2; d.b3 = p + kOffB3;
    return d;
}

GDP_RETCODE Mlp::refresh_bf16() {
    k_mlp_cast<<<16, 256, 0, stream>>>(p, w1, w2, w2t, w3);
    GDP_MCUDA(cudaGetLastError());
    return GDP_OKAY;
}

GDP_RETCODE Mlp::init(unsigned long long seed, int dev_index) {
    device = dev_index;
    GDP_MCUDA(cudaSetDevice(device));
    GDP_MCUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    int pageable = 0;
    GDP_MCUDA(cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device));
    host_direct = pageable == 1;
    const size_t pb = sizeof(float) * kMlpParams;
    GDP_MCUDA(cudaMalloc(&p, pb));
    GDP_MCUDA(cudaMalloc(&m1, pb));
    GDP_MCUDA(cudaMalloc(&m2, pb));
    GDP_MCUDA(cudaMalloc(&grad, pb));
    GDP_MCUDA(cudaMalloc(&loss, sizeof(float)));
    GDP_MCUDA(cudaMalloc(&w1, sizeof(__nv_bfloat16) * kMlpH * kMlpIn));
    GDP_MCUDA(cudaMalloc(&w2, sizeof(__nv_bfloat16) * kMlpH * kMlpH));
    GDP_MCUDA(cudaMalloc(&w2t, sizeof(__nv_bfloat16) * kMlpH * kMlpH));
    GDP_MCUDA(cudaMalloc(&w3, sizeof(__nv_bfloat16) * kMlpH));
    GDP_MCUDA(cudaFuncSetAttribute(k_mlp_grad<kGradWarpsFew>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(TileSmem) * kGradWarpsFew));
    GDP_MCUDA(cudaFuncSetAttribute(k_mlp_grad<kGradWarpsMany>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(TileSmem) * kGradWarpsMany));
    // He-uniform weights, zero biases
    std::vector<float> h(kMlpParams, 0.f);
    unsigned long long s = seed;
    auto fill = [&](int off, int count, int fan_in) {
        const double a = std::sqrt(6.0 / fan_in);
        for (int i = 0; i < count; i++) h[off + i] = (float)((2.0 * uniform01(s) - 1.0) * a);
    };
    fill(kOffW1, kMlpH * kMlpIn, kMlpIn);
    fill(kOffW2, kMlpH * kMlpH, kMlpH);
    fill(kOffW3, kMlpH, kMlpH);
    return set(h.data());
}

GDP_RETCODE Mlp::set(const float *params) {
    if (!params) { set_error("null parameters"); return GDP_ERROR; }
    GDP_MCUDA(cudaMemcpyAsync(p, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, stream));
    GDP_MCUDA(cudaMemsetAsync(m1, 0, sizeof(float) * kMlpParams, stream));
    GDP_MCUDA(cudaMemsetAsync(m2, 0, sizeof(float) * kMlpParams, stream));
    step = 0;
    if (refresh_bf16() != GDP_OKAY) return GDP_ERROR;
    GDP_MCUDA(cudaStreamSynchronize(stream));
    return GDP_OKAY;
}

GDP_RETCODE Mlp::get(float *params) const {
    if (!params) { set_error("null parameters"); return GDP_ERROR; }
    GDP_MCUDA(cudaMemcpyAsync(params, p, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, stream));
    GDP_MCUDA(cudaStreamSynchronize(stream));
    return GDP_OKAY;
}

namespace {
// A call's kernels and copies use its host memory: one that fails waits for
// them before its buffers are given back.
struct Drained {
    cudaStream_t s;
    ~Drained() { cudaStreamSynchronize(s); }
};
}  // namespace

// Samples on the device: features as BF16, labels, weights (device memory of
// `mem`). With coherent access the features are read from host memory by the
// conversion kernel, which does not hold up the calling thread.
GDP_RETCODE Mlp::upload(Arena &mem, int n, const float *x, const float *y, const float *w, __nv_bfloat16 **xb,
                        float **dy, float **dw) {
    const size_t cnt = (size_t)n * kMlpIn;
    *xb = (__nv_bfloat16 *)mem.alloc_bytes(sizeof(__nv_bfloat16) * cnt);
    *dy = (float *)mem.alloc_bytes(sizeof(float) * (size_t)n);
    *dw = (float *)mem.alloc_bytes(sizeof(float) * (size_t)n);
    const float *src = x;
    if (!host_direct || reinterpret_cast<uintptr_t>(x) % alignof(float)) {
        float *up = (float *)mem.alloc_bytes(sizeof(float) * cnt);
        if (up) GDP_MCUDA(cudaMemcpyAsync(up, x, sizeof(float) * cnt, cudaMemcpyHostToDevice, stream));
        src = up;
    }
    if (!*xb || !*dy || !*dw || !src) { set_error("device allocation failed (samples)"); return GDP_ERROR; }
    GDP_MCUDA(cudaMemcpyAsync(*dy, y, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, stream));
    GDP_MCUDA(cudaMemcpyAsync(*dw, w, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, stream));
    k_to_bf16<<<4 * device_sms(), 256, 0, stream>>>(src, *xb, (long long)cnt);
    GDP_MCUDA(cudaGetLastError());
    return GDP_OKAY;
}

// Host threads that touch the pages of `bytes` bytes: one per MB.
static int touch_threads(size_t bytes) {
    return (int)std::max(1LL, std::min<long long>((long long)(bytes >> 20), omp_get_max_threads() - 1));
}

GDP_RETCODE Mlp::forward(int n, const float *x, float *z) {
    if (n < 0 || (n && (!x || !z))) { set_error("bad forward arguments"); return GDP_ERROR; }
    if (!n) return GDP_OKAY;
    GDP_MCUDA(cudaSetDevice(device));
    const size_t xb = sizeof(float) * (size_t)n * kMlpIn, zb = sizeof(float) * (size_t)n;
    // 16-byte loads need an aligned array (numpy's are), and logits may be written
    // while features are still read: other features are copied first
    const uintptr_t xa = reinterpret_cast<uintptr_t>(x), za = reinterpret_cast<uintptr_t>(z);
    const bool overlap = xa < za + zb && za < xa + xb;
    const bool direct = host_direct && xa % 16 == 0 && !overlap;
    const bool z_direct = host_direct && za % alignof(float) == 0;
    // The logits go straight to host memory. The GPU's first write to a page that
    // nothing has touched yet is a fault of many microseconds, and a new array has new
    // pages, so the host touches them: up to 1 MB before the launch, of more while the
    // first quarter of the rows runs, whose logits go by way of device memory (2M rows
    // into a new array: 3.6 ms written untouched, 0.77 with all of them by way of
    // device memory, 0.72 so, 1.9 with the features copied too).
    constexpr size_t kTouchFirst = 1 << 20;
    // rows by way of device memory
    const int early = !direct || !z_direct ? n : zb > kTouchFirst ? n / 4 / 16 * 16 : 0;
    Arena tmp;
    const Drained drained{stream};
    const float *dx = x;
    float *dz = nullptr;
    if (!direct) {
        float *up = (float *)tmp.alloc_bytes(xb);
        if (!up) { set_error("device allocation failed (forward)"); return GDP_ERROR; }
        GDP_MCUDA(cudaMemcpyAsync(up, x, xb, cudaMemcpyHostToDevice, stream));
        dx = up;
    }
    if (early) {
        dz = (float *)tmp.alloc_bytes(sizeof(float) * (size_t)early);
        if (!dz) { set_error("device allocation failed (forward)"); return GDP_ERROR; }
        k_mlp_forward<<<forward_grid(early), kMlpThreads, 0, stream>>>(dev(), dx, early, dz);
        GDP_MCUDA(cudaGetLastError());
    }
    if (z_direct) touch_pages(z, zb, touch_threads(zb));
    if (early < n) {
        k_mlp_forward<<<forward_grid(n - early), kMlpThreads, 0, stream>>>(dev(), dx + (size_t)early * kMlpIn, n - early,
                                                                          z + early);
        GDP_MCUDA(cudaGetLastError());
    }
    if (early && z_direct) {
        k_copy<<<2 * device_sms(), 256, 0, stream>>>(dz, z, early);
        GDP_MCUDA(cudaGetLastError());
    } else if (early) {
        GDP_MCUDA(cudaMemcpyAsync(z, dz, sizeof(float) * (size_t)early, cudaMemcpyDeviceToHost, stream));
    }
    GDP_MCUDA(cudaStreamSynchronize(stream));
    return GDP_OKAY;
}

GDP_RETCODE Mlp::gradient(int n, const float *x, const float *y, const float *w, float *g, float *lossv) {
    if (n <= 0 || !x || !y || !w || !g) { set_error("bad gradient arguments"); return GDP_ERROR; }
    GDP_MCUDA(cudaSetDevice(device));
    Arena mem;
    const Drained drained{stream};
    __nv_bfloat16 *xb;
    float *dy, *dw;
    if (upload(mem, n, x, y, w, &xb, &dy, &dw) != GDP_OKAY) return GDP_ERROR;
    float *part = (float *)mem.alloc_bytes(sizeof(float) * kPartLd * (size_t)grad_rows_max());
    if (!part) { set_error("device allocation failed (gradient)"); return GDP_ERROR; }
    double ws = 0.0;
    for (int i = 0; i < n; i++) ws += w[i];
    int rows = 0;
    GDP_MCUDA(launch_grad(dev(), xb, nullptr, dy, dw, n, ws > 0 ? (float)(1.0 / ws) : 0.f, part, &rows, false,
                          stream));
    k_mlp_sum<<<kSumBlocks, dim3(kSumCols, kSumGroups), 0, stream>>>(part, rows, grad, loss);
    GDP_MCUDA(cudaGetLastError());
    GDP_MCUDA(cudaMemcpyAsync(g, grad, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, stream));
    float l = 0.f;
    GDP_MCUDA(cudaMemcpyAsync(&l, loss, sizeof(float), cudaMemcpyDeviceToHost, stream));
    GDP_MCUDA(cudaStreamSynchronize(stream));
    if (lossv) *lossv = l;
    return GDP_OKAY;
}

GDP_RETCODE Mlp::train(int n, const float *x, const float *y, const float *w, int epochs, int batch, float lr,
                       unsigned long long seed, float *final_loss) {
    if (n <= 0 || !x || !y || !w || epochs <= 0 || batch <= 0 || !(lr > 0.f)) {
        set_error("bad training arguments");
        return GDP_ERROR;
    }
    GDP_MCUDA(cudaSetDevice(device));
    // one shuffle of the samples; epochs walk contiguous minibatches from a
    // rotating start. The samples go up in their order while the shuffle is
    // drawn; the gradient kernel reads them through it.
    std::vector<int> perm(n);
    std::vector<double> wpre(n + 1, 0.0);
    Arena mem;
    const Drained drained{stream};
    __nv_bfloat16 *xb;
    float *dy, *dw;
    if (upload(mem, n, x, y, w, &xb, &dy, &dw) != GDP_OKAY) return GDP_ERROR;
    for (int i = 0; i < n; i++) perm[i] = i;
    unsigned long long s = seed;
    for (int i = n - 1; i > 0; i--) std::swap(perm[i], perm[(int)(splitmix(s) % (unsigned long long)(i + 1))]);
    const int nb = (n - 1) / batch + 1;
    int *dperm = (int *)mem.alloc_bytes(sizeof(int) * (size_t)n);
    float *part = (float *)mem.alloc_bytes(sizeof(float) * kPartLd * (size_t)grad_rows_max());
    float *d_losses = (float *)mem.alloc_bytes(sizeof(float) * (size_t)nb);
    if (!dperm || !part || !d_losses) { set_error("device allocation failed (training)"); return GDP_ERROR; }
    GDP_MCUDA(cudaMemcpyAsync(dperm, perm.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, stream));
    for (int i = 0; i < n; i++) wpre[i + 1] = wpre[i] + w[perm[i]];
    double last = 0.0;
    std::vector<float> lh(nb);
    const int step0 = step;
    for (int e = 0; e < epochs; e++) {
        const int rot = (int)(splitmix(s) % (unsigned long long)nb);
        for (int b = 0; b < nb; b++) {
            const int bi = (b + rot) % nb;
            const int r0 = bi * batch, cnt = std::min(batch, n - r0);
            const double ws = wpre[r0 + cnt] - wpre[r0];
            int rows = 0;
            GDP_MCUDA(launch_grad(dev(), xb, dperm + r0, dy, dw, cnt, ws > 0 ? (float)(1.0 / ws) : 0.f, part, &rows,
                                  step0 != step, stream));
            step++;
            LaunchNext L(kSumBlocks, dim3(kSumCols, kSumGroups), 0, true, stream);
            GDP_MCUDA(cudaLaunchKernelEx(&L.cfg, k_mlp_step, (const float *)part, rows, p, m1, m2, step, lr, 0.9f,
                                         0.999f, 1e-8f, w1, w2, w2t, w3, d_losses + bi));
        }
    }
    GDP_MCUDA(cudaMemcpyAsync(lh.data(), d_losses, sizeof(float) * (size_t)nb, cudaMemcpyDeviceToHost, stream));
    GDP_MCUDA(cudaStreamSynchronize(stream));
    for (int b = 0; b < nb; b++) {
        const int r0 = b * batch, cnt = std::min(batch, n - r0);
        last += lh[b] * (wpre[r0 + cnt] - wpre[r0]);
    }
    if (final_loss) *final_loss = wpre[n] > 0 ? (float)(last / wpre[n]) : 0.f;
    return GDP_OKAY;
}

}  // namespace gdp

// ---- C-ABI ----------------------------------------------------------------------

#pragma GCC visibility push(default)
extern "C" {

GDP_RETCODE gdp_mlp_create(unsigned long long seed, int device, gdp_mlp **out) {
    if (!out) { gdp::set_error("null output pointer"); return GDP_ERROR; }
    *out = nullptr;
    gdp_mlp *m = new (std::nothrow) gdp_mlp();
    if (!m) { gdp::set_error("host allocation failed"); return GDP_ERROR; }
    if (gdp::guarded([&]() -> GDP_RETCODE { return m->impl.init(seed, device); }) != GDP_OKAY) {
        delete m;
        return GDP_ERROR;
    }
    *out = m;
    return GDP_OKAY;
}

GDP_RETCODE gdp_mlp_destroy(gdp_mlp *m) {
    delete m;
    return GDP_OKAY;
}

GDP_RETCODE gdp_mlp_get_params(const gdp_mlp *m, float *params) {
    if (!m) { gdp::set_error("null model"); return GDP_ERROR; }
    return gdp::guarded([&]() -> GDP_RETCODE { return m->impl.get(params); });
}

GDP_RETCODE gdp_mlp_set_params(gdp_mlp *m, const float *params) {
    if (!m) { gdp::set_error("null model"); return GDP_ERROR; }
    return gdp::guarded([&]() -> GDP_RETCODE { return m->impl.set(params); });
}

GDP_RETCODE gdp_mlp_forward(gdp_mlp *m, int n, const float *x, float *logits) {
    if (!m) { gdp::set_error("null model"); return GDP_ERROR; }
    return gdp::guarded([&]() -> GDP_RETCODE { return m->impl.forward(n, x, logits); });
}

GDP_RETCODE gdp_mlp_gradient(gdp_mlp *m, int n, const float *x, const float *y, const float *w, float *grad,
                             float *loss) {
    if (!m) { gdp::set_error("null model"); return GDP_ERROR; }
    return gdp::guarded([&]() -> GDP_RETCODE { return m->impl.gradient(n, x, y, w, grad, loss); });
}

GDP_RETCODE gdp_mlp_train(gdp_mlp *m, int n, const float *x, const float *y, const float *w, int epochs, int batch,
                          float lr, unsigned long long seed, float *final_loss) {
    if (!m) { gdp::set_error("null model"); return GDP_ERROR; }
    return gdp::guarded([&]() -> GDP_RETCODE { return m->impl.train(n, x, y, w, epochs, batch, lr, seed, final_loss); });
}

}  // extern "C"
#pragma GCC visibility pop
