// Surrogate MLP on the tensor cores: training (forward, backward, Adam) and inference of a fully
// connected network with SiLU hidden layers, BF16 weights and activations and FP32 accumulation,
// built on the tcgen05 GEMM of tc_gemm.cuh. No counterpart in the reference; the network maps the
// optical properties of a layered model to its ring- and time-resolved reflectance and is
// trained on tallies of the batched Monte Carlo (batch.cu).
//
// Layer l computes Z_l = A_{l-1} W_l^T + b_l with A_{-1} = X (inputs zero-padded to 64 columns)
// and A_l = SiLU(Z_l) for hidden layers; the last layer is linear (outputs padded to a multiple of
// 256 with zero weights). Every GEMM is D = A . B^T with both operands K-major:
//   forward            A = A_{l-1} [rows x in]     B = W_l   [out x in]
//   backward (data)    A = dZ_l    [rows x out]    B = W_l^T [in x out]      -> dA_{l-1}, x SiLU'(Z_{l-1})
//   backward (weights) A = dZ_l^T  [out x rows]    B = A_{l-1}^T [in x rows] -> dW_l (split over rows)
// so the forward epilogues also write A_l^T and the backward epilogues dZ^T (coalesced: the 32
// lanes of a warp hold 32 consecutive rows), and each Adam step refreshes W_l and W_l^T in BF16
// from the FP32 master weights. Loss: mean squared error over rows x n_out.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include <cudaTypedefs.h>

#include "mlp_fused.cuh"
#include "photon.cuh"
#include "tc_gemm.cuh"
#include "xmc_internal.h"

using bf16 = __nv_bfloat16;

namespace xmc {
namespace {

constexpr int kInPad = 64;
constexpr int kMaxLayers = 9;

__device__ __forceinline__ float f32(uint32_t r) { return __uint_as_float(r); }

__device__ __forceinline__ void load_bf16x32(const bf16* p, float (&v)[32]) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 u = q[j];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
            const float2 f = __bfloat1622float2(h);
            v[8 * j + 2 * i] = f.x;
            v[8 * j + 2 * i + 1] = f.y;
        }
    }
}

// The warp's 32 rows x 32 columns (lane t holds row row0 + t) to a row-major matrix through the
// warp's shared-memory tile: 32 stores, each one row segment of 32 consecutive elements.
__device__ __forceinline__ void warp_rows_f32(float* sw, const float (&v)[32], float* dst, size_t ld, int row0, int col0,
                                              int ncols, int lane) {
#pragma unroll
    for (int j = 0; j < 32; ++j) sw[lane * 33 + j] = v[j];
    __syncwarp();
    if (col0 + lane < ncols) {
#pragma unroll 4
        for (int k = 0; k < 32; ++k) dst[(size_t)(row0 + k) * ld + col0 + lane] = sw[k * 33 + lane];
    }
    __syncwarp();
}
// The lane's 32 columns of its own row: four 16-byte stores, which fill whole 32-byte sectors. (Through the
// shared-memory tile, 32 stores of 64 bytes per warp, the epilogue took three times the instructions.)
__device__ __forceinline__ void lane_row_bf16(const float (&v)[32], bf16* dst) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        reinterpret_cast<uint4*>(dst)[j] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// r[] plus the bias of its 32 columns (the same for every lane).
__device__ __forceinline__ void add_bias(const uint32_t (&r)[32], const float* __restrict__ bias, float (&v)[32]) {
    const float4* b4 = reinterpret_cast<const float4*>(bias);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float4 b = __ldg(&b4[q]);
        v[4 * q] = f32(r[4 * q]) + b.x;
        v[4 * q + 1] = f32(r[4 * q + 1]) + b.y;
        v[4 * q + 2] = f32(r[4 * q + 2]) + b.z;
        v[4 * q + 3] = f32(r[4 * q + 3]) + b.w;
    }
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// ---------------------------------------------------------------- epilogues

// Plain FP32 store of the accumulator (split-K partials at blockIdx.z * split_stride).
struct EpiF32 {
    float* d;
    int ld;
    size_t split_stride;
    __device__ void apply(int row, int col0, const uint32_t (&r)[32], int lane, float* sw) const {
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = f32(r[j]);
        warp_rows_f32(sw, v, d + blockIdx.z * split_stride, (size_t)ld, row - lane, col0, col0 + 32, lane);
    }
};

// Hidden layer: Z = acc + b, A = SiLU(Z); A row-major always, Z and A^T when training.
struct EpiHidden {
    const float* bias;
    bf16* a;
    int lda;
    bf16* z;    // nullable
    bf16* at;   // nullable, [cols x ldt]
    int ldt;
    __device__ void apply(int row, int col0, const uint32_t (&r)[32], int lane, float* sw) const {
        float v[32];
        add_bias(r, bias + col0, v);
        if (z) lane_row_bf16(v, z + (size_t)row * lda + col0);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
        lane_row_bf16(v, a + (size_t)row * lda + col0);
        if (at) {
#pragma unroll
            for (int j = 0; j < 32; ++j) at[(size_t)(col0 + j) * ldt + row] = __float2bfloat16_rn(v[j]);
        }
    }
};

// Output layer: Y = acc + b for the first n_out columns. Training (t != nullptr): the gradient of
// the (optionally per-output weighted) mean squared error dY = scale w (Y - T) (0 in the padding
// columns), row-major and transposed, and the sum of w (Y - T)^2 added to loss[*step + step_add]. The targets
// of row i are row src[i] of t (row i without src): they are read where the data set holds them.
struct EpiOut {
    const float* bias;
    float* y;  // nullable, [rows x ldy]
    int ldy;
    int n_out;
    const float* t;  // nullable, [. x ldtg]
    int ldtg;
    const int* src;  // nullable
    bf16* dy;
    int lddy;
    bf16* dyt;
    int lddyt;
    float scale;
    const float* colw;  // nullable: per-output weight of the squared error
    float* loss;
    const int* step;
    int step_add;
    __device__ void apply(int row, int col0, const uint32_t (&r)[32], int lane, float* sw) const {
        float v[32];
        add_bias(r, bias + col0, v);
        if (y && col0 < n_out) warp_rows_f32(sw, v, y, (size_t)ldy, row - lane, col0, n_out, lane);
        if (t) {
            const int own = src ? __ldg(&src[row]) : row;
            if ((ldtg & 3) == 0 && col0 + 32 <= n_out && (reinterpret_cast<uintptr_t>(t) & 15) == 0) {
                // the lane's own row, eight 16-byte loads in flight (33 -> 17 us of the layer at 4,096 rows x 1,000)
                const float4* tp = reinterpret_cast<const float4*>(t + (size_t)own * ldtg + col0);
                float4 q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) q[j] = __ldg(&tp[j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    sw[lane * 33 + 4 * j] = q[j].x;
                    sw[lane * 33 + 4 * j + 1] = q[j].y;
                    sw[lane * 33 + 4 * j + 2] = q[j].z;
                    sw[lane * 33 + 4 * j + 3] = q[j].w;
                }
            } else {
                // rows of any alignment, through the warp's tile along their columns
                const bool col = col0 + lane < n_out;
#pragma unroll 8
                for (int k = 0; k < 32; ++k) {
                    const float* tp = t + (size_t)__shfl_sync(0xffffffffu, own, k) * ldtg + col0 + lane;
                    sw[k * 33 + lane] = col ? __ldg(tp) : 0.0f;
                }
            }
            __syncwarp();
            float se = 0.0f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const int c = col0 + j;
                const float d = c < n_out ? v[j] - sw[lane * 33 + j] : 0.0f;
                const float wd = (colw && c < n_out) ? d * __ldg(&colw[c]) : d;
                se = fmaf(wd, d, se);
                v[j] = wd * scale;
            }
            __syncwarp();
            lane_row_bf16(v, dy + (size_t)row * lddy + col0);
#pragma unroll
            for (int j = 0; j < 32; ++j) dyt[(size_t)(col0 + j) * lddyt + row] = __float2bfloat16_rn(v[j]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
            if (lane == 0) atomicAdd(loss + *step + step_add, se);
        }
    }
};

// Backward through SiLU: dZ = acc * SiLU'(Z), row-major and transposed.
struct EpiBwd {
    const bf16* z;
    int ldz;
    bf16* dz;
    bf16* dzt;
    int ldt;
    __device__ void apply(int row, int col0, const uint32_t (&r)[32], int lane, float* sw) const {
        float zv[32], v[32];
        load_bf16x32(z + (size_t)row * ldz + col0, zv);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = f32(r[j]) * dsilu(zv[j]);
        lane_row_bf16(v, dz + (size_t)row * ldz + col0);
#pragma unroll
        for (int j = 0; j < 32; ++j) dzt[(size_t)(col0 + j) * ldt + row] = __float2bfloat16_rn(v[j]);
    }
};

// ---------------------------------------------------------------- small kernels

// FP32 host inputs [valid x n_in] -> bf16 [rows x 64] (zero padded both ways), and optionally transposed.
__global__ void pack_inputs_kernel(const float* __restrict__ x, int rows, int valid, int n_in, bf16* __restrict__ xb,
                                   bf16* __restrict__ xt, int ldt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * kInPad) return;
    const int r = i / kInPad, c = i % kInPad;
    const bf16 v = __float2bfloat16_rn(c < n_in && r < valid ? x[(size_t)r * n_in + c] : 0.0f);
    xb[i] = v;
    if (xt) xt[(size_t)c * ldt + r] = v;
}

// Minibatch of `rows` rows drawn with replacement from the device data set (Philox keyed by seed, counter
// (step, row)) for step *step + 1: inputs (bf16, padded, and transposed) and the rows' places in the data
// set, where the output layer reads their targets. 32 rows per block, a warp per four.
__global__ void gather_kernel(const bf16* __restrict__ ds_x, int ds_rows, int rows, uint32_t k0, uint32_t k1,
                              const int* __restrict__ step, float* __restrict__ loss, bf16* __restrict__ xb,
                              bf16* __restrict__ xt, int* __restrict__ src, const float* __restrict__ ds_t, int n_out) {
    __shared__ bf16 tile[32][kInPad + 2];
    const int r0 = blockIdx.x * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = *step + 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) loss[t] = 0.0f;
    const uint4 u = philox4x32_10(make_uint4((uint32_t)(r0 + lane), (uint32_t)t, 0x6d6c70u, 0u), k0, k1);
    const int own = (int)(((unsigned long long)u.x * (unsigned long long)ds_rows) >> 32);
    if (warp == 0) src[r0 + lane] = own;
    // the targets come into L2 while the hidden layers run; the output layer's epilogue, which would wait for
    // DRAM at every line, then finds them there (42 -> 20 us of that layer at 4,096 rows)
    for (int k = warp; k < 32; k += 8) {
        const float* tp = ds_t + (size_t)__shfl_sync(0xffffffffu, own, k) * n_out;
        for (int c = 32 * lane; c < n_out; c += 32 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(tp + c));
        if (lane == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(tp + n_out - 1));
    }
    for (int k = warp; k < 32; k += 8) {
        const int s = __shfl_sync(0xffffffffu, own, k);
        const uint32_t v = reinterpret_cast<const uint32_t*>(ds_x + (size_t)s * kInPad)[lane];
        reinterpret_cast<uint32_t*>(xb + (size_t)(r0 + k) * kInPad)[lane] = v;
        *reinterpret_cast<uint32_t*>(&tile[k][2 * lane]) = v;
    }
    __syncthreads();
    for (int c = warp; c < kInPad; c += 8) xt[(size_t)c * rows + r0 + lane] = tile[lane][c];
}

// db of one unit: the sum over the rows of dZ^T, by a warp. 256 running sums (eight per lane, row r in sum
// r % 256), then their pairwise tree: a fixed order, whatever the launch.
__device__ __forceinline__ float bias_grad(const bf16* __restrict__ dzt_row, int rows, int lane) {
    float s[8] = {};
#pragma unroll 4
    for (int i = 0; i < rows; i += 256) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (i + 32 * k < rows) s[k] += __bfloat162float(dzt_row[i + 32 * k + lane]);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) s[k] += s[k + o];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[0] += __shfl_down_sync(0xffffffffu, s[0], o);
    return s[0];  // lane 0's
}
__global__ void bias_grad_kernel(const bf16* __restrict__ dzt, int rows, float* __restrict__ db) {
    const int n = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const float s = bias_grad(dzt + (size_t)n * rows, rows, lane);
    if (lane == 0) db[n] = s;
}

// g[i] = sum over splits of part[s][i] (fixed order)
__global__ void split_sum_kernel(const float* __restrict__ part, int splits, size_t n, float* __restrict__ g) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float s = 0.0f;
        for (int k = 0; k < splits; ++k) s += part[(size_t)k * n + i];
        g[i] = s;
    }
}

// One Adam step (Kingma & Ba, 2015) on one FP32 master parameter and its moments, bias correction in alpha.
__device__ __forceinline__ float adam(float w, float g, float& m, float& v, float alpha, float b1, float b2, float eps) {
    m = b1 * m + (1.0f - b1) * g;
    v = b2 * v + (1.0f - b2) * g * g;
    return w - alpha * m / (sqrtf(v) + eps);
}

struct UpdateLayer {
    float *w, *m, *v, *b, *mb, *vb;  // masters and moments of the weights [rows x cols] and biases [rows]
    const float* part;               // [splits][rows x cols] partial weight gradients
    const float* gb;                 // [rows] bias gradients
    bf16 *w16, *w16t;
    int rows, cols, valid_rows, splits;
    int first_tile, first_bias;      // its first block of weights and of biases in the launch
};  // (blocks of 256 biases)
struct UpdateParams {
    UpdateLayer layer[kMaxLayers];
    int layers, biases;              // the first `biases` blocks take biases, the others weights
    float lr, b1, b2, eps;
    int *step, *ticket;
};

// Gradient sums and Adam of every parameter of the network in one launch: blocks of 32 x 32 weights sum their
// split-K partials in split order, step, and write the bf16 copies both ways through a shared tile; the
// last block to finish counts the step. As four launches per layer (split sums, bias sums, two Adam launches
// with strided transposed stores) this took 130 us of a 296 us step on a 15-256x4-1000 network at 4,096 rows;
// now 44 us, bound by the partials (71 MB, written and read back), with the bias sums beside the backward
// chain. Folding the splits in one CTA per tile instead, in the same order, moved no time: 64 dependent
// k-blocks took 36 us per layer and what they saved here (144 us per step against 150, slower at 8,192 rows).
__global__ void __launch_bounds__(256) update_kernel(const __grid_constant__ UpdateParams P) {
    const int t = *P.step + 1;
    const float c1 = 1.0f - __powf(P.b1, (float)t), c2 = 1.0f - __powf(P.b2, (float)t);
    const float alpha = P.lr * sqrtf(c2) / c1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int l = P.layers - 1;
    if ((int)blockIdx.x >= P.biases) {
        const int blk = (int)blockIdx.x - P.biases;
        while (blk < P.layer[l].first_tile) --l;
        const UpdateLayer& L = P.layer[l];
        const int tile = blk - L.first_tile, tc = L.cols / 32;
        const int r0 = tile / tc * 32, c0 = tile % tc * 32;
        const size_t n = (size_t)L.rows * L.cols;
        __shared__ bf16 s[32][33];
        // every load of the thread's four weights before the first store
        const size_t i0 = (size_t)(r0 + warp) * L.cols + c0 + lane, di = 8 * (size_t)L.cols;
        float w[4], m[4], v[4], g[4] = {};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[k] = L.w[i0 + k * di];
            m[k] = L.m[i0 + k * di];
            v[k] = L.v[i0 + k * di];
        }
#pragma unroll 8
        for (int q = 0; q < L.splits; ++q)
#pragma unroll
            for (int k = 0; k < 4; ++k) g[k] += __ldg(&L.part[(size_t)q * n + i0 + k * di]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (r0 + warp + 8 * k < L.valid_rows) {
                w[k] = adam(w[k], g[k], m[k], v[k], alpha, P.b1, P.b2, P.eps);
                L.m[i0 + k * di] = m[k];
                L.v[i0 + k * di] = v[k];
                L.w[i0 + k * di] = w[k];
            }
            const bf16 h = __float2bfloat16_rn(w[k]);
            L.w16[i0 + k * di] = h;
            s[warp + 8 * k][lane] = h;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) L.w16t[(size_t)(c0 + warp + 8 * k) * L.rows + r0 + lane] = s[lane][warp + 8 * k];
    } else {
        const int blk = (int)blockIdx.x;
        while (blk < P.layer[l].first_bias) --l;
        const UpdateLayer& L = P.layer[l];
        const int r = (blk - L.first_bias) * 256 + threadIdx.x;
        if (r < L.valid_rows) L.b[r] = adam(L.b[r], L.gb[r], L.mb[r], L.vb[r], alpha, P.b1, P.b2, P.eps);
    }
    // every block has read *step before it takes its ticket
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(P.ticket, 1) == (int)gridDim.x - 1) {
        *P.ticket = 0;
        *P.step = t;
    }
}

// FP32 master -> bf16 copy and transpose (after set_params)
__global__ void refresh_kernel(const float* __restrict__ p, int rows, int cols, bf16* __restrict__ w16, bf16* __restrict__ w16t) {
    const size_t n = (size_t)rows * cols;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / cols), c = (int)(i % cols);
        const bf16 h = __float2bfloat16_rn(p[i]);
        w16[i] = h;
        w16t[(size_t)c * rows + r] = h;
    }
}

// ---------------------------------------------------------------- host helpers

int mfail(int status, const std::string& msg) {
    set_error(msg);
    return status;
}

#define XM_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return mfail(XMC_ERR_DEVICE, std::string(#call) + ": " + cudaGetErrorString(e_));      \
    } while (0)

std::mutex g_encode_mutex;
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

int get_encoder() {
    std::lock_guard<std::mutex> lock(g_encode_mutex);
    if (g_encode) return XMC_OK;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || !fn || q != cudaDriverEntryPointSuccess)
        return mfail(XMC_ERR_DEVICE, "cuTensorMapEncodeTiled is not available from the driver");
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return XMC_OK;
}

// Tensor map of a row-major bf16 matrix [rows x cols] read in boxes of box_rows x 64 with the
// 128-byte swizzle (the layout the GEMM's shared-memory descriptors describe).
int make_map(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    int st = get_encoder();
    if (st) return st;
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols * 2) % 16 || cols % tc::kBK || box_rows > 256)
        return mfail(XMC_ERR_INVALID_INPUT, "tensor map: misaligned operand");
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)tc::kBK, box_rows};
    const cuuint32_t es[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return mfail(XMC_ERR_DEVICE, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return XMC_OK;
}

// Tensor map of the FP32 output [rows x n_out] stored in boxes of 32 rows x 16 columns with the
// 64-byte swizzle (the fused forward's staging layout); columns past n_out are clipped by the store.
int make_out_map(CUtensorMap* map, float* y, uint64_t rows, uint64_t n_out) {
    int st = get_encoder();
    if (st) return st;
    if ((reinterpret_cast<uintptr_t>(y) & 15) || (n_out * 4) % 16)
        return mfail(XMC_ERR_INVALID_INPUT, "tensor map: misaligned output");
    const cuuint64_t dims[2] = {n_out, rows};
    const cuuint64_t strides[1] = {n_out * 4};
    const cuuint32_t box[2] = {(cuuint32_t)fused::kOutCols, 32};
    const cuuint32_t es[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, y, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return mfail(XMC_ERR_DEVICE, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return XMC_OK;
}

// Lets `kernel` take `bytes` of dynamic shared memory on the current device. `done`: one for each kernel.
template <class F>
int allow_smem(F kernel, int bytes, OncePerDevice& done) {
    int device = 0;
    XM_CUDA(cudaGetDevice(&device));
    if (!done.pending(device)) return XMC_OK;
    XM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done.set(device);
    return XMC_OK;
}

// D = A[rows_a x k] . B[n x k]^T with A, B device bf16 row-major; grid (n / BN, rows_a / 128, splits).
template <int BN, class Epi>
int launch_gemm(const void* a, int rows_a, const void* b, int n, int k, int splits, const Epi& epi, int* err,
                cudaStream_t stream) {
    if (rows_a % tc::kBM || n % BN || k % (tc::kBK * splits) || splits < 1)
        return mfail(XMC_ERR_INVALID_INPUT, "gemm: shape not a multiple of the tile");
    static OncePerDevice smem_set;
    int st = allow_smem(tc::gemm_kernel<BN, Epi>, tc::smem_bytes(BN), smem_set);
    if (st) return st;
    CUtensorMap ma, mb;
    st = make_map(&ma, a, (uint64_t)rows_a, (uint64_t)k, tc::kBM);
    if (st) return st;
    st = make_map(&mb, b, (uint64_t)n, (uint64_t)k, BN);
    if (st) return st;
    const dim3 grid(n / BN, rows_a / tc::kBM, splits);
    tc::gemm_kernel<BN, Epi><<<grid, tc::kThreads, tc::smem_bytes(BN), stream>>>(ma, mb, k / tc::kBK / splits, err, epi);
    XM_CUDA(cudaGetLastError());
    return XMC_OK;
}

int round_up(int x, int m) { return (x + m - 1) / m * m; }

}  // namespace
}  // namespace xmc

using namespace xmc;

// ---------------------------------------------------------------- model

struct xmc_mlp {
    xmc_mlp_spec spec{};
    int L = 0;                      // layers (hidden + 1)
    int in[kMaxLayers], out[kMaxLayers];   // padded dimensions
    int valid_out[kMaxLayers];             // rows of W that are real (n_out for the last layer)
    int cap = 0;                    // row capacity
    int sms = 0;                    // of its device
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    int* d_err = nullptr;
    int* d_step = nullptr;
    float* d_loss = nullptr;        // [max_steps + 1]
    int loss_cap = 0;
    float *w32[kMaxLayers] = {}, *b32[kMaxLayers] = {};
    float *mw[kMaxLayers] = {}, *vw[kMaxLayers] = {}, *mb[kMaxLayers] = {}, *vb[kMaxLayers] = {};
    float *gw[kMaxLayers] = {}, *gb[kMaxLayers] = {};
    bf16 *w16[kMaxLayers] = {}, *w16t[kMaxLayers] = {};
    // activations [cap x width] (and transposes [width x cap])
    bf16 *x = nullptr, *xt = nullptr;
    bf16 *a[kMaxLayers] = {}, *at[kMaxLayers] = {}, *z[kMaxLayers] = {};
    bf16 *dz[kMaxLayers] = {}, *dzt[kMaxLayers] = {};
    float *y = nullptr, *t = nullptr, *xin = nullptr;
    float* colw = nullptr;          // per-output loss weights, or null
    float* part[kMaxLayers] = {};   // split-K partials of each layer's weight gradient (one allocation, part[0])
    int* src = nullptr;             // minibatch rows' places in the data set
    cudaStream_t side[2] = {};      // weight gradients beside the data gradients, layers in turn
    cudaEvent_t ev_dz[kMaxLayers] = {}, ev_side[2] = {};
    // data set
    bf16* ds_x = nullptr;
    float* ds_t = nullptr;
    int ds_rows = 0;
    std::map<int, cudaGraphExec_t> train_graphs;  // by batch rows (hyper-parameters in key below)
    std::map<int, cudaGraphExec_t> fwd_graphs;
    float g_lr = 0, g_b1 = 0, g_b2 = 0, g_eps = 0;
    uint64_t g_seed = 0;
    float* h_y = nullptr;           // pinned staging of the outputs read back by xmc_mlp_forward (lazy)
    size_t h_y_floats = 0;
    cudaEvent_t ev_chunk[8] = {};   // completion of each chunk of that read-back (lazy)
};

namespace xmc {
namespace {

void free_mlp(xmc_mlp* m) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m) return;
    cudaSetDevice(m->spec.device);
    for (auto& kv : m->train_graphs) cudaGraphExecDestroy(kv.second);
    for (auto& kv : m->fwd_graphs) cudaGraphExecDestroy(kv.second);
    std::vector<void*> d = {m->d_err, m->d_step, m->d_loss, m->x, m->xt, m->y, m->t, m->xin, m->src, m->part[0], m->ds_x, m->ds_t,
                            m->colw};
    for (int l = 0; l < kMaxLayers; ++l)
        for (void* p : {(void*)m->w32[l], (void*)m->b32[l], (void*)m->mw[l], (void*)m->vw[l], (void*)m->mb[l],
                        (void*)m->vb[l], (void*)m->gw[l], (void*)m->gb[l], (void*)m->w16[l], (void*)m->w16t[l],
                        (void*)m->a[l], (void*)m->at[l], (void*)m->z[l], (void*)m->dz[l], (void*)m->dzt[l]})
            d.push_back(p);
    for (void* p : d)
        if (p) cudaFree(p);
    for (cudaEvent_t e : m->ev)
        if (e) cudaEventDestroy(e);
    if (m->h_y) cudaFreeHost(m->h_y);
    for (cudaEvent_t e : m->ev_chunk)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : m->ev_dz)
        if (e) cudaEventDestroy(e);
    for (int k = 0; k < 2; ++k) {
        if (m->ev_side[k]) cudaEventDestroy(m->ev_side[k]);
        if (m->side[k]) cudaStreamDestroy(m->side[k]);
    }
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

// Widest tile that still gives the device's `sms` SMs a CTA each, else the narrowest: the tile width changes no sum.
int tile_width(int rows_a, int n, int splits, int sms) {
    for (int bn = 256; bn > 64; bn /= 2)
        if (n % bn == 0 && (rows_a / tc::kBM) * (n / bn) * splits >= sms) return bn;
    return 64;
}

// split-K factor of the weight-gradient GEMM of layer l for `rows` rows: about 128 CTAs of full width
int wgrad_splits(const xmc_mlp* m, int l, int rows) {
    const int tiles = m->out[l] / tc::kBM;
    const int kblocks = rows / tc::kBK;
    int s = std::max(1, 128 / tiles);
    while (s > 1 && (kblocks % s)) --s;
    return std::min(s, kblocks);
}

bool fused_forward_ok(const xmc_mlp* m) {
    return m->spec.forward_kernel == 0 && m->spec.n_out % 4 == 0 && m->L <= fused::kMaxL && m->in[0] == kInPad;
}

// Inference forward over `rows` rows of m->x into m->y with the fused kernel (mlp_fused.cuh).
int enqueue_fused_forward(xmc_mlp* m, int rows) {
    static OncePerDevice smem_set[2];
    int st = allow_smem(fused::mlp_forward_kernel<1>, fused::kSmemBytes, smem_set[0]);
    if (!st) st = allow_smem(fused::mlp_forward_kernel<2>, fused::kSmemBytes, smem_set[1]);
    if (st) return st;
    fused::Params p;
    std::memset(&p, 0, sizeof(p));
    st = make_map(&p.x, m->x, (uint64_t)rows, (uint64_t)kInPad, tc::kBM);
    for (int l = 0; !st && l < m->L; ++l) {
        st = make_map(&p.w[l], m->w16[l], (uint64_t)m->out[l], (uint64_t)m->in[l], l < m->L - 1 ? m->spec.hidden : 256);
        p.bias[l] = m->b32[l];
    }
    if (!st) st = make_out_map(&p.y, m->y, (uint64_t)rows, (uint64_t)m->spec.n_out);
    if (st) return st;
    p.L = m->L;
    p.hidden = m->spec.hidden;
    p.out_chunks = m->out[m->L - 1] / 256;
    p.n_tiles = rows / tc::kBM;
    p.n_out = m->spec.n_out;
    p.err = m->d_err;
    const int sms = m->sms;
    // no more tiles than SMs: one tile per CTA; where the SMs also suffice for every output chunk of every tile, a
    // CTA takes one of those
    p.split = p.n_tiles * p.out_chunks <= sms;
    if (p.n_tiles <= sms)
        fused::mlp_forward_kernel<1><<<p.split ? p.n_tiles * p.out_chunks : p.n_tiles, fused::kThreads, fused::kSmemBytes,
                                       m->stream>>>(p);
    else fused::mlp_forward_kernel<2><<<sms, fused::kThreads, fused::kSmemBytes, m->stream>>>(p);
    XM_CUDA(cudaGetLastError());
    return XMC_OK;
}

// D = A . B^T with the widest tile that fills the chip.
template <class Epi>
int launch_gemm_wide(const xmc_mlp* m, const void* a, int rows_a, const void* b, int n, int k, int splits, const Epi& epi,
                     cudaStream_t stream) {
    switch (tile_width(rows_a, n, splits, m->sms)) {
        case 256: return launch_gemm<256>(a, rows_a, b, n, k, splits, epi, m->d_err, stream);
        case 128: return launch_gemm<128>(a, rows_a, b, n, k, splits, epi, m->d_err, stream);
        default: return launch_gemm<64>(a, rows_a, b, n, k, splits, epi, m->d_err, stream);
    }
}

// Forward pass over `rows` rows of m->x (bf16, padded). Training: also Z, A^T, dY, loss, with the targets from
// m->t or, for a minibatch, from the data set.
int enqueue_forward(xmc_mlp* m, int rows, bool train, bool from_data_set = false) {
    if (!train && fused_forward_ok(m)) return enqueue_fused_forward(m, rows);
    const cudaStream_t st = m->stream;
    for (int l = 0; l < m->L; ++l) {
        const bf16* a_in = l == 0 ? m->x : m->a[l - 1];
        const int k = m->in[l];
        int s;
        if (l < m->L - 1) {
            EpiHidden e{m->b32[l], m->a[l], m->out[l], train ? m->z[l] : nullptr, train ? m->at[l] : nullptr, rows};
            s = launch_gemm_wide(m, a_in, rows, m->w16[l], m->out[l], k, 1, e, st);
        } else {
            EpiOut e{};
            e.bias = m->b32[l];
            e.n_out = m->spec.n_out;
            if (train) {
                e.y = nullptr;
                e.t = from_data_set ? m->ds_t : m->t;
                e.src = from_data_set ? m->src : nullptr;
                e.step_add = from_data_set ? 1 : 0;  // the step under way is counted when it is done
                e.ldtg = m->spec.n_out;
                e.dy = m->dz[l];
                e.lddy = m->out[l];
                e.dyt = m->dzt[l];
                e.lddyt = rows;
                e.scale = 2.0f / ((float)rows * (float)m->spec.n_out);
                e.colw = m->colw;
                e.loss = m->d_loss;
                e.step = m->d_step;
            } else {
                e.y = m->y;
                e.ldy = m->spec.n_out;
            }
            s = launch_gemm_wide(m, a_in, rows, m->w16[l], m->out[l], k, 1, e, st);
        }
        if (s) return s;
    }
    return XMC_OK;
}

// Backward pass after enqueue_forward(train): per-layer partial weight gradients into m->part, bias gradients
// into m->gb. The data gradients are one chain; each layer's weight and bias gradients hang off it and run on
// a stream of their own.
int enqueue_backward(xmc_mlp* m, int rows) {
    const cudaStream_t st = m->stream;
    for (int l = m->L - 1; l >= 0; --l) {
        XM_CUDA(cudaEventRecord(m->ev_dz[l], st));  // dZ_l is ready
        if (l > 0) {
            EpiBwd e{m->z[l - 1], m->out[l - 1], m->dz[l - 1], m->dzt[l - 1], rows};
            const int s = launch_gemm_wide(m, m->dz[l], rows, m->w16t[l], m->in[l], m->out[l], 1, e, st);
            if (s) return s;
        }
        // bias gradient, then the weight gradient dW = dZ^T . A_{l-1}, split over rows. The first layer's, the last
        // to start, run side by side.
        XM_CUDA(cudaStreamWaitEvent(m->side[l & 1], m->ev_dz[l], 0));
        bias_grad_kernel<<<m->out[l] / 8, 256, 0, l > 0 ? m->side[l & 1] : st>>>(m->dzt[l], rows, m->gb[l]);
        XM_CUDA(cudaGetLastError());
        const bf16* bt = l == 0 ? m->xt : m->at[l - 1];
        EpiF32 e{m->part[l], m->in[l], (size_t)m->out[l] * m->in[l]};
        const int s = launch_gemm_wide(m, m->dzt[l], m->out[l], bt, m->in[l], rows, wgrad_splits(m, l, rows), e, m->side[l & 1]);
        if (s) return s;
    }
    for (int k = 0; k < std::min(2, m->L); ++k) {
        XM_CUDA(cudaEventRecord(m->ev_side[k], m->side[k]));
        XM_CUDA(cudaStreamWaitEvent(st, m->ev_side[k], 0));
    }
    return XMC_OK;
}

// Sums of the weight gradients after enqueue_backward, into gw.
int enqueue_gradient_sums(xmc_mlp* m, int rows) {
    for (int l = 0; l < m->L; ++l) {
        split_sum_kernel<<<296, 256, 0, m->stream>>>(m->part[l], wgrad_splits(m, l, rows), (size_t)m->out[l] * m->in[l], m->gw[l]);
    }
    XM_CUDA(cudaGetLastError());
    return XMC_OK;
}

// Gradient sums and Adam after enqueue_backward.
int enqueue_update(xmc_mlp* m, int rows, float lr, float b1, float b2, float eps) {
    UpdateParams p;
    std::memset(&p, 0, sizeof(p));
    int tiles = 0;
    for (int l = 0; l < m->L; ++l) {
        UpdateLayer& U = p.layer[l];
        U = {m->w32[l], m->mw[l], m->vw[l], m->b32[l], m->mb[l], m->vb[l], m->part[l], m->gb[l], m->w16[l], m->w16t[l],
             m->out[l], m->in[l], m->valid_out[l], wgrad_splits(m, l, rows), tiles, p.biases};
        tiles += m->out[l] / 32 * (m->in[l] / 32);
        p.biases += (m->out[l] + 255) / 256;
    }
    p.layers = m->L;
    p.lr = lr; p.b1 = b1; p.b2 = b2; p.eps = eps;
    p.step = m->d_step;
    p.ticket = m->d_step + 1;
    update_kernel<<<tiles + p.biases, 256, 0, m->stream>>>(p);
    XM_CUDA(cudaGetLastError());
    return XMC_OK;
}

int check_err(xmc_mlp* m) {
    int e = 0;
    XM_CUDA(cudaMemcpy(&e, m->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
        cudaMemset(m->d_err, 0, sizeof(int));
        return mfail(XMC_ERR_DEVICE, "tensor-core GEMM: a pipeline wait timed out");
    }
    return XMC_OK;
}

int upload_inputs(xmc_mlp* m, const float* x, int rows, int valid, bool transposed) {
    XM_CUDA(cudaMemcpyAsync(m->xin, x, sizeof(float) * (size_t)valid * m->spec.n_in, cudaMemcpyHostToDevice, m->stream));
    pack_inputs_kernel<<<(rows * kInPad + 255) / 256, 256, 0, m->stream>>>(m->xin, rows, valid, m->spec.n_in, m->x,
                                                                           transposed ? m->xt : nullptr, rows);
    XM_CUDA(cudaGetLastError());
    return XMC_OK;
}

int check_rows(const xmc_mlp* m, int rows) {
    if (rows <= 0 || rows % tc::kBM || rows > m->cap)
        return mfail(XMC_ERR_RANGE, "rows must be a positive multiple of 128 up to max_rows");
    return XMC_OK;
}

}  // namespace
}  // namespace xmc

extern "C" int xmc_mlp_create(const xmc_mlp_spec* spec, xmc_mlp** out) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!spec || !out) return mfail(XMC_ERR_INVALID_INPUT, "spec or out is NULL");
    *out = nullptr;
    xmc_mlp_spec s{};
    std::memcpy(&s, spec, std::min((size_t)spec->struct_size, sizeof(s)));
    s.struct_size = sizeof(s);
    if (s.n_in < 1 || s.n_in > kInPad) return mfail(XMC_ERR_RANGE, "n_in must be in [1, 64]");
    if (s.hidden != 128 && s.hidden != 256) return mfail(XMC_ERR_RANGE, "hidden must be 128 or 256");
    if (s.n_hidden < 1 || s.n_hidden > kMaxLayers - 1) return mfail(XMC_ERR_RANGE, "n_hidden must be in [1, 8]");
    if (s.n_out < 1 || s.n_out > 4096) return mfail(XMC_ERR_RANGE, "n_out must be in [1, 4096]");
    if (s.max_rows < tc::kBM || s.max_rows % tc::kBM || s.max_rows > (1 << 20))
        return mfail(XMC_ERR_RANGE, "max_rows must be a multiple of 128 in [128, 2^20]");
    xmc_mlp* m = new (std::nothrow) xmc_mlp;
    if (!m) return mfail(XMC_ERR_DEVICE, "out of host memory");
    m->spec = s;
    m->L = s.n_hidden + 1;
    m->cap = s.max_rows;
    for (int l = 0; l < m->L; ++l) {
        m->in[l] = l == 0 ? kInPad : s.hidden;
        m->out[l] = l == m->L - 1 ? round_up(s.n_out, 256) : s.hidden;
        m->valid_out[l] = l == m->L - 1 ? s.n_out : s.hidden;
    }
#define XM_TRY(call)                                                                             \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));                      \
            free_mlp(m);                                                                         \
            return XMC_ERR_DEVICE;                                                               \
        }                                                                                        \
    } while (0)
    XM_TRY(cudaSetDevice(s.device));
    XM_TRY(cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, s.device));
    XM_TRY(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    XM_TRY(cudaEventCreate(&m->ev[0]));
    XM_TRY(cudaEventCreate(&m->ev[1]));
    XM_TRY(cudaMalloc(&m->d_err, sizeof(int)));
    XM_TRY(cudaMalloc(&m->d_step, 2 * sizeof(int)));  // steps taken, tickets of the step under way
    m->loss_cap = 1 << 20;
    XM_TRY(cudaMalloc(&m->d_loss, sizeof(float) * (m->loss_cap + 1)));
    XM_TRY(cudaMemset(m->d_err, 0, sizeof(int)));
    XM_TRY(cudaMemset(m->d_step, 0, 2 * sizeof(int)));
    // Training's buffers too, so that no training call of a model that was made fails for want of memory: streams and
    // events of the backward pass, the minibatch's row numbers, and the split-K partials of every layer at the
    // largest split any batch takes.
    for (int k = 0; k < 2; ++k) {
        XM_TRY(cudaStreamCreateWithFlags(&m->side[k], cudaStreamNonBlocking));
        XM_TRY(cudaEventCreateWithFlags(&m->ev_side[k], cudaEventDisableTiming));
    }
    size_t part_at[kMaxLayers + 1] = {};
    for (int l = 0; l < m->L; ++l) {
        XM_TRY(cudaEventCreateWithFlags(&m->ev_dz[l], cudaEventDisableTiming));
        part_at[l + 1] = part_at[l] + (size_t)m->out[l] * m->in[l] * std::max(1, 128 / (m->out[l] / tc::kBM));
    }
    XM_TRY(cudaMalloc(&m->part[0], sizeof(float) * part_at[m->L]));
    for (int l = 1; l < m->L; ++l) m->part[l] = m->part[0] + part_at[l];
    const size_t R = (size_t)m->cap;
    XM_TRY(cudaMalloc(&m->src, sizeof(int) * R));
    for (int l = 0; l < m->L; ++l) {
        const size_t n = (size_t)m->out[l] * m->in[l];
        XM_TRY(cudaMalloc(&m->w32[l], sizeof(float) * n));
        XM_TRY(cudaMalloc(&m->mw[l], sizeof(float) * n));
        XM_TRY(cudaMalloc(&m->vw[l], sizeof(float) * n));
        XM_TRY(cudaMalloc(&m->gw[l], sizeof(float) * n));
        XM_TRY(cudaMalloc(&m->w16[l], sizeof(bf16) * n));
        XM_TRY(cudaMalloc(&m->w16t[l], sizeof(bf16) * n));
        XM_TRY(cudaMalloc(&m->b32[l], sizeof(float) * m->out[l]));
        XM_TRY(cudaMalloc(&m->mb[l], sizeof(float) * m->out[l]));
        XM_TRY(cudaMalloc(&m->vb[l], sizeof(float) * m->out[l]));
        XM_TRY(cudaMalloc(&m->gb[l], sizeof(float) * m->out[l]));
        for (float* p : {m->w32[l], m->mw[l], m->vw[l], m->gw[l]}) XM_TRY(cudaMemset(p, 0, sizeof(float) * n));
        for (float* p : {m->b32[l], m->mb[l], m->vb[l], m->gb[l]}) XM_TRY(cudaMemset(p, 0, sizeof(float) * m->out[l]));
        XM_TRY(cudaMemset(m->w16[l], 0, sizeof(bf16) * n));
        XM_TRY(cudaMemset(m->w16t[l], 0, sizeof(bf16) * n));
        XM_TRY(cudaMalloc(&m->a[l], sizeof(bf16) * R * m->out[l]));
        XM_TRY(cudaMalloc(&m->at[l], sizeof(bf16) * R * m->out[l]));
        XM_TRY(cudaMalloc(&m->z[l], sizeof(bf16) * R * m->out[l]));
        XM_TRY(cudaMalloc(&m->dz[l], sizeof(bf16) * R * m->out[l]));
        XM_TRY(cudaMalloc(&m->dzt[l], sizeof(bf16) * R * m->out[l]));
    }
    XM_TRY(cudaMalloc(&m->x, sizeof(bf16) * R * kInPad));
    XM_TRY(cudaMalloc(&m->xt, sizeof(bf16) * R * kInPad));
    XM_TRY(cudaMalloc(&m->xin, sizeof(float) * R * s.n_in));
    XM_TRY(cudaMalloc(&m->y, sizeof(float) * R * s.n_out));
    XM_TRY(cudaMalloc(&m->t, sizeof(float) * R * s.n_out));
#undef XM_TRY
    *out = m;
    return XMC_OK;
}

extern "C" int64_t xmc_mlp_param_count(const xmc_mlp* m) {
    if (!m) return -1;
    int64_t n = 0;
    int in = m->spec.n_in;
    for (int l = 0; l < m->L; ++l) {
        n += (int64_t)m->valid_out[l] * in + m->valid_out[l];
        in = m->valid_out[l];
    }
    return n;
}

// Flat parameter layout: for each layer W_l [out_l][in_l] row-major, then b_l [out_l], with
// in_0 = n_in, out_{L-1} = n_out (no padding).
extern "C" int xmc_mlp_set_params(xmc_mlp* m, const float* p) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !p) return mfail(XMC_ERR_INVALID_INPUT, "model or params is NULL");
    XM_CUDA(cudaSetDevice(m->spec.device));
    int in = m->spec.n_in;
    const float* q = p;
    for (int l = 0; l < m->L; ++l) {
        const int vo = m->valid_out[l];
        std::vector<float> w((size_t)m->out[l] * m->in[l], 0.0f), b(m->out[l], 0.0f);
        for (int r = 0; r < vo; ++r)
            for (int c = 0; c < in; ++c) w[(size_t)r * m->in[l] + c] = q[(size_t)r * in + c];
        q += (size_t)vo * in;
        for (int r = 0; r < vo; ++r) b[r] = q[r];
        q += vo;
        XM_CUDA(cudaMemcpy(m->w32[l], w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice));
        XM_CUDA(cudaMemcpy(m->b32[l], b.data(), sizeof(float) * b.size(), cudaMemcpyHostToDevice));
        XM_CUDA(cudaMemset(m->mw[l], 0, sizeof(float) * w.size()));
        XM_CUDA(cudaMemset(m->vw[l], 0, sizeof(float) * w.size()));
        XM_CUDA(cudaMemset(m->mb[l], 0, sizeof(float) * b.size()));
        XM_CUDA(cudaMemset(m->vb[l], 0, sizeof(float) * b.size()));
        refresh_kernel<<<m->sms, 256, 0, m->stream>>>(m->w32[l], m->out[l], m->in[l], m->w16[l], m->w16t[l]);
        XM_CUDA(cudaGetLastError());
        in = vo;
    }
    XM_CUDA(cudaMemsetAsync(m->d_step, 0, sizeof(int), m->stream));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    return XMC_OK;
}

static int copy_layers_out(const xmc_mlp* m, float* const* wsrc, float* const* bsrc, float* p) {
    int in = m->spec.n_in;
    float* q = p;
    for (int l = 0; l < m->L; ++l) {
        const int vo = m->valid_out[l];
        std::vector<float> w((size_t)m->out[l] * m->in[l]), b(m->out[l]);
        XM_CUDA(cudaMemcpy(w.data(), wsrc[l], sizeof(float) * w.size(), cudaMemcpyDeviceToHost));
        XM_CUDA(cudaMemcpy(b.data(), bsrc[l], sizeof(float) * b.size(), cudaMemcpyDeviceToHost));
        for (int r = 0; r < vo; ++r)
            for (int c = 0; c < in; ++c) q[(size_t)r * in + c] = w[(size_t)r * m->in[l] + c];
        q += (size_t)vo * in;
        for (int r = 0; r < vo; ++r) q[r] = b[r];
        q += vo;
        in = vo;
    }
    return XMC_OK;
}

extern "C" int xmc_mlp_get_params(const xmc_mlp* m, float* p) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !p) return mfail(XMC_ERR_INVALID_INPUT, "model or params is NULL");
    XM_CUDA(cudaSetDevice(m->spec.device));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    return copy_layers_out(m, m->w32, m->b32, p);
}

// Forward pass of `valid` host rows as `rows` rows (a multiple of 128; the others are zero), the outputs of the
// valid ones into y.
static int forward_host(xmc_mlp* m, const float* x, int rows, int valid, float* y, double* ms) {
    XM_CUDA(cudaSetDevice(m->spec.device));
    int st = upload_inputs(m, x, rows, valid, false);
    if (st) return st;
    XM_CUDA(cudaEventRecord(m->ev[0], m->stream));
    st = enqueue_forward(m, rows, false);
    if (st) return st;
    XM_CUDA(cudaEventRecord(m->ev[1], m->stream));
    // outputs through pinned staging (kept by the model, sized for its row capacity), then into the
    // caller's array on up to 8 host threads. Large outputs go back in 8 chunks of rows, each with
    // its own event, and every thread copies its share of a chunk as soon as that chunk has landed,
    // so the host copies overlap the device-to-host transfer of the later chunks.
    const size_t nf = (size_t)valid * m->spec.n_out;
    if (m->h_y_floats < nf) {
        if (m->h_y) cudaFreeHost(m->h_y);
        m->h_y = nullptr;
        m->h_y_floats = 0;
        XM_CUDA(cudaHostAlloc((void**)&m->h_y, sizeof(float) * ((size_t)m->cap * m->spec.n_out + 1), cudaHostAllocDefault));
        m->h_y_floats = (size_t)m->cap * m->spec.n_out;
    }
    // the kernels' error word travels with the outputs, behind them in the staging buffer
    const int* const h_err = reinterpret_cast<const int*>(m->h_y + m->h_y_floats);
    XM_CUDA(cudaMemcpyAsync(m->h_y + m->h_y_floats, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    const int chunks = nf < ((size_t)1 << 22) ? 1 : 8;
    const size_t cf = ((size_t)(valid + chunks - 1) / chunks) * m->spec.n_out;  // floats per chunk (whole rows)
    for (int k = 0; k < chunks; ++k) {
        if (!m->ev_chunk[k]) XM_CUDA(cudaEventCreateWithFlags(&m->ev_chunk[k], cudaEventDisableTiming));
        const size_t a = std::min(nf, k * cf), b = std::min(nf, a + cf);
        if (a < b)
            XM_CUDA(cudaMemcpyAsync(m->h_y + a, m->y + a, sizeof(float) * (b - a), cudaMemcpyDeviceToHost, m->stream));
        XM_CUDA(cudaEventRecord(m->ev_chunk[k], m->stream));
    }
    const unsigned parts = nf < ((size_t)1 << 20) ? 1u : std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
    std::atomic<int> copy_err{0};
    auto copy_part = [&](unsigned p) {
        for (int k = 0; k < chunks; ++k) {
            if (cudaEventSynchronize(m->ev_chunk[k]) != cudaSuccess) {
                copy_err = 1;
                return;
            }
            const size_t a = std::min(nf, k * cf), b = std::min(nf, a + cf);
            const size_t per = (b - a + parts - 1) / parts;
            const size_t pa = std::min(b, a + p * per), pb = std::min(b, pa + per);
            if (pa < pb) std::memcpy(y + pa, m->h_y + pa, sizeof(float) * (pb - pa));
        }
    };
    std::vector<std::thread> pool;
    unsigned started = 1;
    try {
        for (; started < parts; ++started) pool.emplace_back(copy_part, started);
    } catch (...) {
    }
    copy_part(0);
    for (unsigned p = started; p < parts; ++p) copy_part(p);
    for (auto& th : pool) th.join();
    if (copy_err) {
        const cudaError_t e = cudaStreamSynchronize(m->stream);
        return mfail(XMC_ERR_DEVICE, std::string("reading the outputs back failed: ") +
                                         cudaGetErrorString(e != cudaSuccess ? e : cudaErrorUnknown));
    }
    float t = 0.0f;
    XM_CUDA(cudaEventElapsedTime(&t, m->ev[0], m->ev[1]));
    if (ms) *ms = t;
    return *h_err ? check_err(m) : XMC_OK;
}

extern "C" int xmc_mlp_forward(xmc_mlp* m, const float* x, int rows, float* y, double* ms) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !x || !y) return mfail(XMC_ERR_INVALID_INPUT, "model, x or y is NULL");
    const int st = check_rows(m, rows);
    return st ? st : forward_host(m, x, rows, rows, y, ms);
}

// The same for any number of rows in [1, max_rows]: a query of one row does not send its tile's other 127 to
// the host and copy them there (15-256x4-1000, one row: 131 -> 65 us per call, half of it by this and the error word that travels with the outputs).
extern "C" int xmc_mlp_forward_rows(xmc_mlp* m, const float* x, int n, float* y, double* ms) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !x || !y) return mfail(XMC_ERR_INVALID_INPUT, "model, x or y is NULL");
    if (n < 1 || n > m->cap) return mfail(XMC_ERR_RANGE, "rows must be in [1, max_rows]");
    return forward_host(m, x, round_up(n, tc::kBM), n, y, ms);
}

// Times `reps` forward passes of the inputs already on the device (the last xmc_mlp_forward's),
// replayed from a CUDA graph; *ms gets the mean device time of one pass.
extern "C" int xmc_mlp_forward_timed(xmc_mlp* m, int rows, int reps, double* ms) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || reps < 1) return mfail(XMC_ERR_INVALID_INPUT, "model is NULL or reps < 1");
    int st = check_rows(m, rows);
    if (st) return st;
    XM_CUDA(cudaSetDevice(m->spec.device));
    cudaGraphExec_t ex = nullptr;
    auto it = m->fwd_graphs.find(rows);
    if (it != m->fwd_graphs.end()) {
        ex = it->second;
    } else {
        XM_CUDA(cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
        st = enqueue_forward(m, rows, false);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(m->stream, &g);
        if (st) {
            if (g) cudaGraphDestroy(g);
            return st;
        }
        if (e != cudaSuccess) return mfail(XMC_ERR_DEVICE, std::string("capture: ") + cudaGetErrorString(e));
        e = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return mfail(XMC_ERR_DEVICE, std::string("instantiate: ") + cudaGetErrorString(e));
        m->fwd_graphs[rows] = ex;
    }
    XM_CUDA(cudaGraphLaunch(ex, m->stream));  // warm
    XM_CUDA(cudaEventRecord(m->ev[0], m->stream));
    for (int i = 0; i < reps; ++i) XM_CUDA(cudaGraphLaunch(ex, m->stream));
    XM_CUDA(cudaEventRecord(m->ev[1], m->stream));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    float t = 0.0f;
    XM_CUDA(cudaEventElapsedTime(&t, m->ev[0], m->ev[1]));
    if (ms) *ms = t / reps;
    return check_err(m);
}

// Gradients of the mean squared error over `rows` rows at the current parameters (no update), in
// the flat parameter layout; *loss gets the mean squared error.
extern "C" int xmc_mlp_gradients(xmc_mlp* m, const float* x, const float* t, int rows, float* grads, float* loss) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !x || !t || !grads) return mfail(XMC_ERR_INVALID_INPUT, "NULL argument");
    int st = check_rows(m, rows);
    if (st) return st;
    XM_CUDA(cudaSetDevice(m->spec.device));
    st = upload_inputs(m, x, rows, rows, true);
    if (st) return st;
    XM_CUDA(cudaMemcpyAsync(m->t, t, sizeof(float) * (size_t)rows * m->spec.n_out, cudaMemcpyHostToDevice, m->stream));
    // loss slot: loss[step + ... ] uses *d_step; use slot (current step) after zeroing it
    int step = 0;
    XM_CUDA(cudaMemcpyAsync(&step, m->d_step, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    XM_CUDA(cudaMemsetAsync(m->d_loss + step, 0, sizeof(float), m->stream));
    st = enqueue_forward(m, rows, true);
    if (st) return st;
    st = enqueue_backward(m, rows);
    if (!st) st = enqueue_gradient_sums(m, rows);
    if (st) return st;
    float l = 0.0f;
    XM_CUDA(cudaMemcpyAsync(&l, m->d_loss + step, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    if (loss) *loss = l / ((float)rows * (float)m->spec.n_out);
    st = check_err(m);
    if (st) return st;
    return copy_layers_out(m, m->gw, m->gb, grads);
}

extern "C" int xmc_mlp_set_dataset(xmc_mlp* m, const float* x, const float* t, int rows) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || !x || !t || rows < 1) return mfail(XMC_ERR_INVALID_INPUT, "NULL argument or empty data set");
    XM_CUDA(cudaSetDevice(m->spec.device));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    for (auto& kv : m->train_graphs) cudaGraphExecDestroy(kv.second);  // they hold the old data set's addresses
    m->train_graphs.clear();
    if (m->ds_x) cudaFree(m->ds_x);
    if (m->ds_t) cudaFree(m->ds_t);
    m->ds_x = nullptr;
    m->ds_t = nullptr;
    m->ds_rows = 0;
    XM_CUDA(cudaMalloc(&m->ds_x, sizeof(bf16) * (size_t)rows * kInPad));
    XM_CUDA(cudaMalloc(&m->ds_t, sizeof(float) * (size_t)rows * m->spec.n_out));
    float* xin = nullptr;
    XM_CUDA(cudaMalloc(&xin, sizeof(float) * (size_t)rows * m->spec.n_in));
    cudaError_t e = cudaMemcpy(xin, x, sizeof(float) * (size_t)rows * m->spec.n_in, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        pack_inputs_kernel<<<(int)(((size_t)rows * kInPad + 255) / 256), 256>>>(xin, rows, rows, m->spec.n_in, m->ds_x, nullptr, 0);
        e = cudaDeviceSynchronize();
    }
    cudaFree(xin);
    if (e != cudaSuccess) return mfail(XMC_ERR_DEVICE, std::string("set_dataset: ") + cudaGetErrorString(e));
    XM_CUDA(cudaMemcpy(m->ds_t, t, sizeof(float) * (size_t)rows * m->spec.n_out, cudaMemcpyHostToDevice));
    m->ds_rows = rows;
    return XMC_OK;
}

// `steps` Adam steps on minibatches of `batch` rows drawn (with replacement, Philox keyed by seed)
// from the device data set; each step is one replay of a CUDA graph (gather, forward, backward,
// Adam). losses[i] (may be NULL) gets the mean squared error of step i's minibatch.
extern "C" int xmc_mlp_train(xmc_mlp* m, int steps, int batch, float lr, float beta1, float beta2, float eps,
                             uint64_t seed, float* losses, double* ms) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m || steps < 0) return mfail(XMC_ERR_INVALID_INPUT, "model is NULL or steps < 0");
    if (!m->ds_rows) return mfail(XMC_ERR_INVALID_INPUT, "no data set (xmc_mlp_set_dataset)");
    int st = check_rows(m, batch);
    if (st) return st;
    XM_CUDA(cudaSetDevice(m->spec.device));
    int step0 = 0;
    XM_CUDA(cudaMemcpy(&step0, m->d_step, sizeof(int), cudaMemcpyDeviceToHost));
    if (step0 + steps >= m->loss_cap) return mfail(XMC_ERR_RANGE, "too many training steps for the loss log");
    if (lr != m->g_lr || beta1 != m->g_b1 || beta2 != m->g_b2 || eps != m->g_eps || seed != m->g_seed) {
        for (auto& kv : m->train_graphs) cudaGraphExecDestroy(kv.second);
        m->train_graphs.clear();
        m->g_lr = lr; m->g_b1 = beta1; m->g_b2 = beta2; m->g_eps = eps; m->g_seed = seed;
    }
    cudaGraphExec_t ex = nullptr;
    auto it = m->train_graphs.find(batch);
    if (it != m->train_graphs.end()) {
        ex = it->second;
    } else {
        XM_CUDA(cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
        gather_kernel<<<batch / 32, 256, 0, m->stream>>>(m->ds_x, m->ds_rows, batch, (uint32_t)seed, (uint32_t)(seed >> 32),
                                                         m->d_step, m->d_loss, m->x, m->xt, m->src, m->ds_t,
                                                         m->spec.n_out);
        st = enqueue_forward(m, batch, true, true);
        if (!st) st = enqueue_backward(m, batch);
        if (!st) st = enqueue_update(m, batch, lr, beta1, beta2, eps);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(m->stream, &g);
        if (st) {
            if (g) cudaGraphDestroy(g);
            return st;
        }
        if (e != cudaSuccess) return mfail(XMC_ERR_DEVICE, std::string("capture: ") + cudaGetErrorString(e));
        e = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return mfail(XMC_ERR_DEVICE, std::string("instantiate: ") + cudaGetErrorString(e));
        m->train_graphs[batch] = ex;
    }
    XM_CUDA(cudaEventRecord(m->ev[0], m->stream));
    for (int i = 0; i < steps; ++i) XM_CUDA(cudaGraphLaunch(ex, m->stream));
    XM_CUDA(cudaEventRecord(m->ev[1], m->stream));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    float t = 0.0f;
    XM_CUDA(cudaEventElapsedTime(&t, m->ev[0], m->ev[1]));
    if (ms) *ms = t;
    st = check_err(m);
    if (st) return st;
    if (losses && steps > 0) {
        XM_CUDA(cudaMemcpy(losses, m->d_loss + step0 + 1, sizeof(float) * steps, cudaMemcpyDeviceToHost));
        const float inv = 1.0f / ((float)batch * (float)m->spec.n_out);
        for (int i = 0; i < steps; ++i) losses[i] *= inv;
    }
    return XMC_OK;
}

// Per-output weights of the squared error in training and in xmc_mlp_gradients (NULL: all 1).
extern "C" int xmc_mlp_set_output_weights(xmc_mlp* m, const float* w) {
    xmc::DeviceGuard device_guard;  // the caller's current device is restored on return
    if (!m) return mfail(XMC_ERR_INVALID_INPUT, "model is NULL");
    XM_CUDA(cudaSetDevice(m->spec.device));
    XM_CUDA(cudaStreamSynchronize(m->stream));
    if (!w) {
        if (m->colw) cudaFree(m->colw);
        m->colw = nullptr;
    } else {
        for (int j = 0; j < m->spec.n_out; ++j)
            if (!(w[j] >= 0.0f) || !std::isfinite(w[j])) return mfail(XMC_ERR_INVALID_INPUT, "weights must be finite and >= 0");
        if (!m->colw) XM_CUDA(cudaMalloc(&m->colw, sizeof(float) * m->spec.n_out));
        XM_CUDA(cudaMemcpy(m->colw, w, sizeof(float) * m->spec.n_out, cudaMemcpyHostToDevice));
    }
    // the training graphs hold the old pointer
    for (auto& kv : m->train_graphs) cudaGraphExecDestroy(kv.second);
    m->train_graphs.clear();
    return XMC_OK;
}

extern "C" int xmc_mlp_destroy(xmc_mlp* m) {
    free_mlp(m);
    return XMC_OK;
}

// Plain GEMM through the same kernel, for tests: D[M x N] = A[M x K] . B[N x K]^T with bf16 inputs
// given as raw 16-bit patterns; split-K partials are summed on the host in split order.
extern "C" int xmc_gemm_bf16(const uint16_t* a, const uint16_t* b, int M, int N, int K, int bn, int splits, float* d) {
    if (!a || !b || !d) return mfail(XMC_ERR_INVALID_INPUT, "NULL argument");
    if (M <= 0 || N <= 0 || K <= 0 || splits < 1 || (bn != 64 && bn != 128 && bn != 256) || M % tc::kBM || N % bn ||
        K % (tc::kBK * splits))
        return mfail(XMC_ERR_INVALID_INPUT, "gemm: M % 128, N % bn, K % (64 splits) must be 0");
    void *da = nullptr, *db = nullptr;
    float* dd = nullptr;
    int* derr = nullptr;
    int st = XMC_OK;
    const size_t nd = (size_t)splits * M * N;
    cudaError_t e = cudaMalloc(&da, sizeof(uint16_t) * (size_t)M * K);
    if (e == cudaSuccess) e = cudaMalloc(&db, sizeof(uint16_t) * (size_t)N * K);
    if (e == cudaSuccess) e = cudaMalloc(&dd, sizeof(float) * nd);
    if (e == cudaSuccess) e = cudaMalloc(&derr, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(derr, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(da, a, sizeof(uint16_t) * (size_t)M * K, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, sizeof(uint16_t) * (size_t)N * K, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) st = mfail(XMC_ERR_DEVICE, std::string("gemm setup: ") + cudaGetErrorString(e));
    if (!st) {
        EpiF32 epi{dd, N, (size_t)M * N};
        if (bn == 256) st = launch_gemm<256>(da, M, db, N, K, splits, epi, derr, 0);
        else if (bn == 128) st = launch_gemm<128>(da, M, db, N, K, splits, epi, derr, 0);
        else st = launch_gemm<64>(da, M, db, N, K, splits, epi, derr, 0);
    }
    if (!st) {
        e = cudaDeviceSynchronize();
        if (e != cudaSuccess) st = mfail(XMC_ERR_DEVICE, std::string("gemm: ") + cudaGetErrorString(e));
    }
    int herr = 0;
    if (!st && cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && herr)
        st = mfail(XMC_ERR_DEVICE, "gemm: a pipeline wait timed out");
    if (!st) {
        std::vector<float> part(nd);
        e = cudaMemcpy(part.data(), dd, sizeof(float) * nd, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            st = mfail(XMC_ERR_DEVICE, std::string("gemm read-back: ") + cudaGetErrorString(e));
        } else {
            for (size_t i = 0; i < (size_t)M * N; ++i) {
                float s = 0.0f;
                for (int k = 0; k < splits; ++k) s += part[(size_t)k * M * N + i];
                d[i] = s;
            }
        }
    }
    cudaFree(da);
    cudaFree(db);
    cudaFree(dd);
    cudaFree(derr);
    return st;
}
