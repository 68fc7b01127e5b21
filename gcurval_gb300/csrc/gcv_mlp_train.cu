// Training of the learned form's MLP on the GPU with the project's own FP32
// kernels: tiled SGEMM (forward and both backward products), bias + GELU
// and its derivative, the three-part loss with its gradient, column sums for
// the bias gradients, and Adam.  Also the FP32 forward pass used as the
// reference of the BF16 tensor-core inference.
#include "gcurval_gb300_learned.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "gcv_learned.cuh"

using namespace gcv;

extern "C" void gcv_internal_device_free(void* p);

namespace {

thread_local std::string g_err_train;

// ---------------------------------------------------------------- kernels
__device__ __forceinline__ float gelu(float x, float& t)
{
    t = tanhf(GELU_C * (x + GELU_A * x * x * x));
    return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ float gelu_grad(float x)
{
    float t;
    gelu(x, t);
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * GELU_C * (1.0f + 3.0f * GELU_A * x * x);
}

// SGEMM tile: 64 x 64 outputs, K step 16, 256 threads of 4 x 4 outputs; the next
// step's operands are loaded into registers while the current one is summed.
constexpr int GB = 64, GK = 16;

// what happens to an output tile
enum Epilogue {
    EP_BIAS,       // C = AB + bias
    EP_BIAS_GELU,  // C = AB + bias, H = GELU(C)
    EP_ACT_GRAD,   // C = AB * GELU'(Z)
    EP_PARTIAL     // split K: chunk z's sums to C + z * stride, and below the last row the column sums of B
};

struct GemmArgs {
    int M, N, K;
    const float *A, *B;
    int lda, ldb;
    float* C;  // row-major, N columns
    const float* aux;  // EP_BIAS*: bias [N]; EP_ACT_GRAD: Z [M x N]
    float* H;
    int chunk;      // EP_PARTIAL: rows of K per chunk (a multiple of GK)
    size_t stride;  // EP_PARTIAL: floats between the chunks' results
};

// 4 consecutive floats; vec: p is 16-byte aligned
__device__ __forceinline__ float4 load4(const float* __restrict__ p, bool vec)
{
    return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

// C[M x N] = op(A)[M x K] op(B)[K x N], row-major storage:
// op(A)[m][k] = TA ? A[k * lda + m] : A[m * lda + k]; likewise B with TB.
// The contiguous extents (K of a plain A or transposed B, M and N otherwise)
// are multiples of 4.
//
// What bounds it: latency and the number of blocks, not FP32 throughput.  The
// weight gradients sum over the batch's rows into 16 x 128 .. 128 x 128 outputs,
// one to four tiles: split over K they fill the GPU, and a plain operand is read
// 16 bytes a lane along its rows (it was read column by column).  A batch
// of 8,192 rows: weight gradients 4 x 1,350 us -> 4 x 9-13 us, bias gradients (one block,
// one thread per column) 4 x 460 us -> part of the same pass; bias, GELU and its
// derivative in the epilogues instead of passes of their own (all under ncu; a call
// of gcv_mlp_trainer_gradients 4.21 -> 0.20 ms).
template <bool TA, bool TB, Epilogue EP>
__global__ void __launch_bounds__(256) k_sgemm(GemmArgs g)
{
    __shared__ __align__(16) float As[GK][GB + 4];
    __shared__ __align__(16) float Bs[GK][GB + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GB, n0 = blockIdx.x * GB;
    const int k_begin = EP == EP_PARTIAL ? blockIdx.z * g.chunk : 0;
    const int k_end = EP == EP_PARTIAL ? min(g.K, k_begin + g.chunk) : g.K;
    const bool vec_a = ((reinterpret_cast<size_t>(g.A) | (size_t)g.lda * 4) & 15) == 0;
    const bool vec_b = ((reinterpret_cast<size_t>(g.B) | (size_t)g.ldb * 4) & 15) == 0;
    // an operand stored along k: thread -> row tid % 64, k quad tid / 64;
    // stored across k: k row tid / 16, quad tid % 16
    auto fetch = [&](const float* X, int ld, bool along_k, int row0, int rows, int k0, bool vec) {
        const int r = row0 + (along_k ? tid & 63 : 4 * (tid & 15)), k = k0 + (along_k ? 4 * (tid >> 6) : tid >> 4);
        if (r >= rows || k >= k_end) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return load4(along_k ? X + (size_t)r * ld + k : X + (size_t)k * ld + r, vec);
    };
    auto stage = [&](float (*S)[GB + 4], bool along_k, float4 v) {
        if (along_k) {
            const int r = tid & 63, k = 4 * (tid >> 6);
            S[k][r] = v.x;
            S[k + 1][r] = v.y;
            S[k + 2][r] = v.z;
            S[k + 3][r] = v.w;
        } else {
            *reinterpret_cast<float4*>(&S[tid >> 4][4 * (tid & 15)]) = v;
        }
    };
    float acc[4][4] = {};
    float col[4] = {};  // EP_PARTIAL: column sums of B over this thread's share of k (k % 16 == ty)
    float4 a4 = fetch(g.A, g.lda, !TA, m0, g.M, k_begin, vec_a);
    float4 b4 = fetch(g.B, g.ldb, TB, n0, g.N, k_begin, vec_b);
    for (int k0 = k_begin; k0 < k_end; k0 += GK) {
        stage(As, !TA, a4);
        stage(Bs, TB, b4);
        __syncthreads();
        if (k0 + GK < k_end) {
            a4 = fetch(g.A, g.lda, !TA, m0, g.M, k0 + GK, vec_a);
            b4 = fetch(g.B, g.ldb, TB, n0, g.N, k0 + GK, vec_b);
        }
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) {
            const float4 av = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 bv = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float a[4] = {av.x, av.y, av.z, av.w}, bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], bb[j], acc[i][j]);
        }
        if constexpr (EP == EP_PARTIAL) {
#pragma unroll
            for (int j = 0; j < 4; ++j) col[j] += Bs[ty][tx * 4 + j];
        }
        __syncthreads();
    }
    float* C = EP == EP_PARTIAL ? g.C + blockIdx.z * g.stride : g.C;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m >= g.M || n >= g.N) continue;
            const size_t at = (size_t)m * g.N + n;
            float v = acc[i][j];
            if constexpr (EP == EP_BIAS || EP == EP_BIAS_GELU) v += g.aux[n];
            if constexpr (EP == EP_ACT_GRAD) v *= gelu_grad(g.aux[at]);
            C[at] = v;
            if constexpr (EP == EP_BIAS_GELU) {
                float t;
                g.H[at] = gelu(v, t);
            }
        }
    if constexpr (EP == EP_PARTIAL) {
        if (blockIdx.y == 0) {  // the 16 threads of a column, added in a fixed order
#pragma unroll
            for (int j = 0; j < 4; ++j) As[ty][tx * 4 + j] = col[j];
            __syncthreads();
            if (tid < GB && n0 + tid < g.N) {
                float s = 0.0f;
#pragma unroll
                for (int k = 0; k < GK; ++k) s += As[k][tid];
                C[(size_t)g.M * g.N + n0 + tid] = s;
            }
        }
    }
}

constexpr int SUM_THREADS = 128;
constexpr int LOSS_THREADS = 64;  // rows per block of k_loss
constexpr int LOSS_BLOCKS = 152 * 32;
int loss_blocks(int n) { return (int)std::min<int64_t>(((int64_t)n + LOSS_THREADS - 1) / LOSS_THREADS, LOSS_BLOCKS); }

// g[i] = the sum of the chunks' partial gradients, in chunk order; the last block adds
// up the loss of k_loss's blocks, in a fixed order and in FP64 (added by FP32 atomics,
// the loss of 8,192 rows differed by 2e-7 from call to call)
__global__ void __launch_bounds__(SUM_THREADS) k_sum_partials(const float* __restrict__ part, int chunks, int count,
                                                              float* __restrict__ g, const float* __restrict__ loss_part,
                                                              int n_loss, float* __restrict__ loss3)
{
    if (blockIdx.x + 1 == gridDim.x) {
        __shared__ double s_l[SUM_THREADS];
        for (int k = 0; k < 3; ++k) {
            double l = 0.0;
            for (int b = threadIdx.x; b < n_loss; b += SUM_THREADS) l += (double)loss_part[3 * b + k];
            s_l[threadIdx.x] = l;
            __syncthreads();
            for (int o = SUM_THREADS / 2; o > 0; o >>= 1) {
                if (threadIdx.x < o) s_l[threadIdx.x] += s_l[threadIdx.x + o];
                __syncthreads();
            }
            if (threadIdx.x == 0) loss3[k] = (float)s_l[0];
            __syncthreads();
        }
        return;
    }
    const int i = blockIdx.x * SUM_THREADS + threadIdx.x;
    if (i >= count) return;
    float s = 0.0f;
#pragma unroll 8
    for (int c = 0; c < chunks; ++c) s += part[(size_t)c * count + i];
    g[i] = s;
}

// loss parts (sums over the block's rows) and dOut = d(mean loss) / d out
__global__ void __launch_bounds__(LOSS_THREADS) k_loss(const float* out, const int* depth, const float* share,
                                                       const float* tg, int n, float* dOut, float* loss_part)
{
    __shared__ float s_l[LOSS_THREADS / 32][3];
    float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f;
    const float inv = 1.0f / (float)n;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const float* o = out + (size_t)r * MLP_OUT;
        float* g = dOut + (size_t)r * MLP_OUT;
        // depth: softmax cross-entropy
        float mx = o[0];
        for (int i = 1; i < MLP_DEPTHS; ++i) mx = fmaxf(mx, o[i]);
        float z = 0.0f;
        for (int i = 0; i < MLP_DEPTHS; ++i) z += expf(o[i] - mx);
        const int d = depth[r];
        l0 += logf(z) + mx - o[d];
        for (int i = 0; i < MLP_DEPTHS; ++i) g[i] = (expf(o[i] - mx) / z - (i == d ? 1.0f : 0.0f)) * inv;
        // split: soft cross-entropy against the leaf shares
        mx = o[MLP_O_SPLIT];
        for (int q = 1; q < 4; ++q) mx = fmaxf(mx, o[MLP_O_SPLIT + q]);
        z = 0.0f;
        for (int q = 0; q < 4; ++q) z += expf(o[MLP_O_SPLIT + q] - mx);
        const float lz = logf(z) + mx;
        for (int q = 0; q < 4; ++q) {
            const float s = share[(size_t)r * 4 + q];
            l1 += s * (lz - o[MLP_O_SPLIT + q]);
            g[MLP_O_SPLIT + q] = (expf(o[MLP_O_SPLIT + q] - mx) / z - s) * inv;
        }
        // t guesses: squared error
        for (int j = 0; j < 8; ++j) {
            const float e = o[MLP_O_T + j] - tg[(size_t)r * 8 + j];
            l2 += 0.5f * e * e;
            g[MLP_O_T + j] = e * inv;
        }
        for (int i = MLP_O_T + 8; i < MLP_OUT; ++i) g[i] = 0.0f;
    }
    for (int o = 16; o > 0; o >>= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        l2 += __shfl_xor_sync(0xffffffffu, l2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_l[threadIdx.x >> 5][0] = l0;
        s_l[threadIdx.x >> 5][1] = l1;
        s_l[threadIdx.x >> 5][2] = l2;
    }
    __syncthreads();
    static_assert(LOSS_THREADS == 64, "two warps' sums");
    if (threadIdx.x < 3) loss_part[3 * blockIdx.x + threadIdx.x] = s_l[0][threadIdx.x] + s_l[1][threadIdx.x];
}

__global__ void k_adam(float* w, const float* g, float* m, float* v, int count, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

template <bool TA, bool TB, Epilogue EP>
void sgemm(const GemmArgs& g, int chunks, cudaStream_t st)
{
    dim3 grid((g.N + GB - 1) / GB, (g.M + GB - 1) / GB, chunks);
    k_sgemm<TA, TB, EP><<<grid, 256, 0, st>>>(g);
}

// chunks of rows the weight gradients are summed in: up to GRAD_CHUNKS, of at
// least 64 rows (with two to four tiles each, 64 chunks fill 152 SMs)
constexpr int GRAD_CHUNKS = 64;
int grad_chunk_rows(int n)
{
    const int rows = std::max(64, (n + GRAD_CHUNKS - 1) / GRAD_CHUNKS);
    return (rows + GK - 1) / GK * GK;
}

// the most chunks of any batch up to max_batch rows (a larger batch may take fewer, longer ones)
int grad_chunks_max(int max_batch) { return (int)std::min<int64_t>(GRAD_CHUNKS, ((int64_t)max_batch + 63) / 64); }

unsigned blocks_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 152 * 32); }

}  // namespace

struct gcv_mlp_trainer {
    int max_batch = 0;
    cudaStream_t st = nullptr;
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    float *Z[3] = {}, *H[3] = {}, *out = nullptr, *dOut = nullptr, *dA = nullptr, *dB = nullptr, *loss3 = nullptr;
    float* part = nullptr;  // grad_chunks_max(max_batch) partial gradients, each packed like w
    float* loss_part = nullptr;  // the loss parts of k_loss's blocks
    long long step = 0;
};

namespace {

gcv_status tfail(gcv_status s, const std::string& m)
{
    g_err_train = m;
    return s;
}

#define TCU(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return tfail(GCV_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

constexpr int OFF_W[4] = {MLP_OFF_W1, MLP_OFF_W2, MLP_OFF_W3, MLP_OFF_W4};
constexpr int OFF_B[4] = {MLP_OFF_B1, MLP_OFF_B2, MLP_OFF_B3, MLP_OFF_B4};
static_assert(MLP_OFF_B1 == MLP_OFF_W1 + MLP_IN * MLP_H && MLP_OFF_B4 == MLP_OFF_W4 + MLP_H * MLP_OUT,
              "a layer's bias gradient follows its weights' like a last row");

// forward pass of n rows of X into tr->Z / H / out
void forward(gcv_mlp_trainer* tr, const float* X, int n)
{
    const float* in = X;
    int fan = MLP_IN;
    for (int l = 0; l < 3; ++l) {
        sgemm<false, false, EP_BIAS_GELU>(GemmArgs{n, MLP_H, fan, in, tr->w + OFF_W[l], fan, MLP_H, tr->Z[l],
                                                   tr->w + OFF_B[l], tr->H[l]}, 1, tr->st);
        in = tr->H[l];
        fan = MLP_H;
    }
    sgemm<false, false, EP_BIAS>(GemmArgs{n, MLP_OUT, MLP_H, in, tr->w + OFF_W[3], MLP_H, MLP_OUT, tr->out,
                                          tr->w + OFF_B[3]}, 1, tr->st);
}

// loss and gradients of the mean loss into tr->g
void backward(gcv_mlp_trainer* tr, const float* X, const int* depth, const float* share, const float* tg, int n)
{
    k_loss<<<loss_blocks(n), LOSS_THREADS, 0, tr->st>>>(tr->out, depth, share, tg, n, tr->dOut, tr->loss_part);
    const int rows = grad_chunk_rows(n), chunks = (n + rows - 1) / rows;
    const float* dz = tr->dOut;  // d loss / d (layer l's output before its activation)
    float* bufs[2] = {tr->dA, tr->dB};
    for (int l = 3; l >= 0; --l) {
        const float* in = l ? tr->H[l - 1] : X;
        const int fan = l ? MLP_H : MLP_IN, cols = l == 3 ? MLP_OUT : MLP_H;
        sgemm<true, false, EP_PARTIAL>(GemmArgs{fan, cols, n, in, dz, fan, cols, tr->part + OFF_W[l], nullptr, nullptr,
                                                rows, MLP_NPARAM}, chunks, tr->st);
        if (l) {
            float* next = bufs[l & 1];
            sgemm<false, true, EP_ACT_GRAD>(GemmArgs{n, MLP_H, cols, dz, tr->w + OFF_W[l], cols, cols, next, tr->Z[l - 1]},
                                            1, tr->st);
            dz = next;
        }
    }
    k_sum_partials<<<(MLP_NPARAM + SUM_THREADS - 1) / SUM_THREADS + 1, SUM_THREADS, 0, tr->st>>>(
        tr->part, chunks, MLP_NPARAM, tr->g, tr->loss_part, loss_blocks(n), tr->loss3);
}

}  // namespace

extern "C" {

const char* gcv_mlp_last_error(void) { return g_err_train.c_str(); }

int gcv_mlp_param_count(void) { return MLP_NPARAM; }

gcv_status gcv_mlp_trainer_create(gcv_mlp_trainer** out, int max_batch, unsigned long long seed)
{
    if (!out || max_batch < 1) return tfail(GCV_ERR_INVALID, "bad trainer arguments");
    *out = nullptr;
    gcv_mlp_trainer* tr = new gcv_mlp_trainer();
    tr->max_batch = max_batch;
    const size_t P = MLP_NPARAM * sizeof(float);
    const size_t A = (size_t)max_batch * MLP_H * sizeof(float), O = (size_t)max_batch * MLP_OUT * sizeof(float);
    cudaError_t e = cudaSuccess;
    float** bufs[] = {&tr->w, &tr->g, &tr->m, &tr->v};
    for (float** b : bufs)
        if (e == cudaSuccess) e = cudaMalloc(b, P);
    for (int l = 0; l < 3 && e == cudaSuccess; ++l) {
        e = cudaMalloc(&tr->Z[l], A);
        if (e == cudaSuccess) e = cudaMalloc(&tr->H[l], A);
    }
    if (e == cudaSuccess) e = cudaMalloc(&tr->out, O);
    if (e == cudaSuccess) e = cudaMalloc(&tr->dOut, O);
    if (e == cudaSuccess) e = cudaMalloc(&tr->dA, A);
    if (e == cudaSuccess) e = cudaMalloc(&tr->dB, A);
    if (e == cudaSuccess) e = cudaMalloc(&tr->loss3, 3 * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&tr->loss_part, (size_t)loss_blocks(max_batch) * 3 * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&tr->part, (size_t)grad_chunks_max(max_batch) * P);
    if (e != cudaSuccess) {
        gcv_mlp_trainer_destroy(tr);
        return tfail(GCV_ERR_OUT_OF_MEMORY, std::string("trainer buffers: ") + cudaGetErrorString(e));
    }
    // He initialisation (normal, variance 2 / fan_in), zero biases
    std::vector<float> h(MLP_NPARAM, 0.0f);
    std::mt19937_64 rng(seed);
    auto init = [&](int off, int fan_in, int count) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / fan_in));
        for (int i = 0; i < count; ++i) h[(size_t)off + i] = nd(rng);
    };
    init(MLP_OFF_W1, MLP_IN, MLP_IN * MLP_H);
    init(MLP_OFF_W2, MLP_H, MLP_H * MLP_H);
    init(MLP_OFF_W3, MLP_H, MLP_H * MLP_H);
    init(MLP_OFF_W4, MLP_H, MLP_H * MLP_OUT);
    if (cudaMemcpy(tr->w, h.data(), P, cudaMemcpyHostToDevice) != cudaSuccess || cudaMemset(tr->m, 0, P) != cudaSuccess ||
        cudaMemset(tr->v, 0, P) != cudaSuccess) {
        gcv_mlp_trainer_destroy(tr);
        return tfail(GCV_ERR_CUDA, "trainer initialisation");
    }
    *out = tr;
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_destroy(gcv_mlp_trainer* tr)
{
    if (!tr) return GCV_OK;
    float* bufs[] = {tr->w, tr->g, tr->m, tr->v, tr->Z[0], tr->Z[1], tr->Z[2], tr->H[0], tr->H[1], tr->H[2],
                     tr->out, tr->dOut, tr->dA, tr->dB, tr->loss3, tr->part, tr->loss_part};
    for (float* b : bufs)
        if (b) gcv_internal_device_free(b);
    delete tr;
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_set_weights(gcv_mlp_trainer* tr, const float* host_w)
{
    if (!tr || !host_w) return tfail(GCV_ERR_INVALID, "NULL argument");
    TCU(cudaMemcpy(tr->w, host_w, MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_get_weights(gcv_mlp_trainer* tr, float* host_w)
{
    if (!tr || !host_w) return tfail(GCV_ERR_INVALID, "NULL argument");
    TCU(cudaMemcpy(host_w, tr->w, MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_forward(gcv_mlp_trainer* tr, const float* d_X, int n, float* d_out)
{
    if (!tr || !d_X || !d_out || n < 0 || n > tr->max_batch) return tfail(GCV_ERR_INVALID, "bad forward arguments");
    if (n == 0) return GCV_OK;
    forward(tr, d_X, n);
    TCU(cudaMemcpyAsync(d_out, tr->out, (size_t)n * MLP_OUT * sizeof(float), cudaMemcpyDeviceToDevice, tr->st));
    TCU(cudaStreamSynchronize(tr->st));
    TCU(cudaGetLastError());
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_gradients(gcv_mlp_trainer* tr, const float* d_X, const int* d_depth, const float* d_share,
                                     const float* d_tguess, int n, float* host_grad, float* host_loss3)
{
    if (!tr || !d_X || !d_depth || !d_share || !d_tguess || n < 1 || n > tr->max_batch)
        return tfail(GCV_ERR_INVALID, "bad gradient arguments");
    forward(tr, d_X, n);
    backward(tr, d_X, d_depth, d_share, d_tguess, n);
    TCU(cudaStreamSynchronize(tr->st));
    TCU(cudaGetLastError());
    if (host_grad) TCU(cudaMemcpy(host_grad, tr->g, MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    if (host_loss3) {
        TCU(cudaMemcpy(host_loss3, tr->loss3, 3 * sizeof(float), cudaMemcpyDeviceToHost));
        for (int i = 0; i < 3; ++i) host_loss3[i] /= (float)n;
    }
    return GCV_OK;
}

gcv_status gcv_mlp_trainer_step(gcv_mlp_trainer* tr, const float* d_X, const int* d_depth, const float* d_share,
                                const float* d_tguess, int n, float lr, float* host_loss3)
{
    gcv_status s = gcv_mlp_trainer_gradients(tr, d_X, d_depth, d_share, d_tguess, n, nullptr, host_loss3);
    if (s != GCV_OK) return s;
    tr->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)tr->step), c2 = 1.0f - std::pow(b2, (float)tr->step);
    k_adam<<<blocks_for(MLP_NPARAM), 256, 0, tr->st>>>(tr->w, tr->g, tr->m, tr->v, MLP_NPARAM, lr, b1, b2, 1e-8f, c1, c2);
    TCU(cudaGetLastError());
    return GCV_OK;
}

}  // extern "C"
