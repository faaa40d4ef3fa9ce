// A small multilayer perceptron with hand-written FP32 CUDA training and
// inference kernels: the learned warm start for DI calibration (this project's
// addition; mwa_hyperdrive has no counterpart).
//
// Layers: y_0 = x; y_l = relu(y_{l-1} W_l^T + b_l) for hidden layers; the
// output layer is linear; if `residual_dim` > 0 the output adds the input
// slice x[:, residual_offset : residual_offset + out_dim] (the net predicts a
// correction to the centre input).  Training minimises the mean squared error
// with Adam.
//
// Kernels: one tiled SGEMM body (64x64 output tile per 256-thread CTA, 4x4
// per thread, K staged through shared memory 16 at a time, the next stage
// read into registers meanwhile) with transpose flags and a fused epilogue
// (bias, ReLU, the residual slice, or the ReLU backward mask), the MSE
// gradient, every layer's weight and bias gradient in one launch split over
// the batch, the sum of those splits and the Adam update.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "common.cuh"

namespace hdc {
namespace mlp {

constexpr int TM = 64, TN = 64, TK = 16;

// What a GEMM adds to or does with its sums.
struct Epilogue {
    const float* bias = nullptr;      // [N], added
    const float* residual = nullptr;  // [M][residual_ld], added after the bias
    int residual_ld = 0;
    const float* mask = nullptr;      // [M][N]: 0 where mask <= 0 (ReLU backward)
    bool relu = false;
};

// Four consecutive elements of a row of n from column j (zero past its end);
// VEC: rows start 16-byte aligned and n is a multiple of 4.
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* __restrict__ row, int j, int n) {
    if (VEC) return j < n ? __ldg(reinterpret_cast<const float4*>(row + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(j < n ? row[j] : 0.f, j + 1 < n ? row[j + 1] : 0.f, j + 2 < n ? row[j + 2] : 0.f,
                       j + 3 < n ? row[j + 3] : 0.f);
}

struct Tiles {
    alignas(16) float a[TK][TM + 4];
    alignas(16) float b[TK][TN + 4];
};

// One 64 x 64 tile at (m0, n0) of C[M][N] = op(A) op(B) over k in [k0, k1)
// (k0 a multiple of TK), op(A)[m][k] = TA ? A[k][m] : A[m][k], op(B)[k][n] =
// TB ? B[n][k] : B[k][n]; the sums run over k in order.  colsum (TA only,
// may be null): colsum[m] = sum_k A[k][m], by the tiles of column n0 = 0.
template <bool TA, bool TB, bool VEC>
__device__ __forceinline__ void gemm_tile(Tiles& t, int M, int N, int m0, int n0, int k0, int k1,
                                          const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb,
                                          float* __restrict__ C, int ldc, const Epilogue& ep,
                                          float* __restrict__ colsum) {
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    // this thread's four elements of a stage: along m (n) at one k when the
    // operand is stored that way round, else along k at one m (n)
    const int ka = TA ? tid / 16 : (tid % 4) * 4, ma = TA ? (tid % 16) * 4 : tid / 4;
    const int kb = TB ? (tid % 4) * 4 : tid / 16, nb = TB ? tid / 4 : (tid % 16) * 4;
    float4 ra, rb;
    auto fetch = [&](int k) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (TA)
            ra = k + ka < k1 ? load4<VEC>(A + (size_t)(k + ka) * lda, m0 + ma, M) : zero;
        else
            ra = m0 + ma < M ? load4<VEC>(A + (size_t)(m0 + ma) * lda, k + ka, k1) : zero;
        if (TB)
            rb = n0 + nb < N ? load4<VEC>(B + (size_t)(n0 + nb) * ldb, k + kb, k1) : zero;
        else
            rb = k + kb < k1 ? load4<VEC>(B + (size_t)(k + kb) * ldb, n0 + nb, N) : zero;
    };
    float acc[4][4] = {};
    float cs = 0.f;
    fetch(k0);
    for (int k = k0; k < k1; k += TK) {
        __syncthreads();  // the previous stage has been read
        if (TA) {
            *reinterpret_cast<float4*>(&t.a[ka][ma]) = ra;
        } else {
            t.a[ka][ma] = ra.x, t.a[ka + 1][ma] = ra.y, t.a[ka + 2][ma] = ra.z, t.a[ka + 3][ma] = ra.w;
        }
        if (TB) {
            t.b[kb][nb] = rb.x, t.b[kb + 1][nb] = rb.y, t.b[kb + 2][nb] = rb.z, t.b[kb + 3][nb] = rb.w;
        } else {
            *reinterpret_cast<float4*>(&t.b[kb][nb]) = rb;
        }
        __syncthreads();
        if (k + TK < k1) fetch(k + TK);
        if (TA && colsum && n0 == 0 && tid < TM)
#pragma unroll
            for (int kk = 0; kk < TK; kk++) cs += t.a[kk][tid];
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            const float4 av = *reinterpret_cast<const float4*>(&t.a[kk][ty * 4]);
            const float4 bv = *reinterpret_cast<const float4*>(&t.b[kk][tx * 4]);
            const float a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
    }
    if (TA && colsum && n0 == 0 && tid < TM && m0 + tid < M) colsum[m0 + tid] = cs;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (ep.bias) v += ep.bias[n];
            if (ep.residual) v += ep.residual[(size_t)m * ep.residual_ld + n];
            if (ep.relu) v = fmaxf(v, 0.f);
            if (ep.mask && ep.mask[(size_t)m * N + n] <= 0.f) v = 0.f;
            C[(size_t)m * ldc + n] = v;
        }
    }
}

template <bool TB, bool VEC>
__global__ void __launch_bounds__(256) sgemm_kernel(int M, int N, int K, const float* __restrict__ A, int lda,
                                                    const float* __restrict__ B, int ldb, float* __restrict__ C,
                                                    int ldc, const Epilogue ep) {
    __shared__ Tiles t;
    gemm_tile<false, TB, VEC>(t, M, N, blockIdx.y * TM, blockIdx.x * TN, 0, K, A, lda, B, ldb, C, ldc, ep, nullptr);
}

// Rows of both operands can be read as 16-byte vectors.
static bool vec_ok(const float* A, int lda, const float* B, int ldb) {
    return ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0 && lda % 4 == 0 && ldb % 4 == 0;
}

// C = A op(B) with the epilogue; the rows of op(B)'s storage and of A are
// their leading dimensions long.
template <bool TB>
static cudaError_t sgemm(int M, int N, int K, const float* A, const float* B, float* C, const Epilogue& ep,
                         cudaStream_t s) {
    const int lda = K, ldb = TB ? K : N;
    dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
    if (vec_ok(A, lda, B, ldb))
        sgemm_kernel<TB, true><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, N, ep);
    else
        sgemm_kernel<TB, false><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, N, ep);
    count_launches(1);
    return cudaGetLastError();
}

// Weight and bias gradients of every layer in one launch: layer l's tiles of
// dW_l = delta_{l+1}^T y_l ([out][in], over the batch) start at tile0; grid
// (tiles of all layers, splits), split z sums rows [z rows, (z + 1) rows) of
// the batch into part[z][parameter].  A layer's own 4 to 16 tiles would leave
// most SMs idle over a batch of thousands (one launch per layer, no splits:
// 1.1 ms each at a batch of 4096 with 256 hidden units).
constexpr int MAXL = 8;  // layers per launch
struct GradLayer {
    const float *delta, *y;  // [batch][out], [batch][in]
    int out, in, tile0, vec;
    size_t w_off, b_off;
};
struct GradArgs {
    GradLayer l[MAXL];
    int nl, batch, rows;
    float* part;
    size_t nparams;
};
__global__ void __launch_bounds__(256) grad_kernel(const __grid_constant__ GradArgs G) {
    __shared__ Tiles t;
    int l = 0;
    while (l + 1 < G.nl && (int)blockIdx.x >= G.l[l + 1].tile0) l++;
    const GradLayer& L = G.l[l];
    const int tile = blockIdx.x - L.tile0, ncol = (L.in + TN - 1) / TN;
    const int m0 = tile / ncol * TM, n0 = tile % ncol * TN;
    const int k0 = blockIdx.y * G.rows, k1 = min(G.batch, k0 + G.rows);
    float* out = G.part + (size_t)blockIdx.y * G.nparams;
    if (L.vec)
        gemm_tile<true, false, true>(t, L.out, L.in, m0, n0, k0, k1, L.delta, L.out, L.y, L.in, out + L.w_off, L.in,
                                     Epilogue{}, out + L.b_off);
    else
        gemm_tile<true, false, false>(t, L.out, L.in, m0, n0, k0, k1, L.delta, L.out, L.y, L.in, out + L.w_off, L.in,
                                      Epilogue{}, out + L.b_off);
}

// g[i] = sum of the splits' parts, in order
__global__ void grad_sum_kernel(const float* __restrict__ part, int splits, size_t n, float* __restrict__ g) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v = 0.f;
    for (int z = 0; z < splits; z++) v += part[z * n + i];
    g[i] = v;
}

// d = 2 (y - t) / (batch * out_dim); loss partial sums per block
__global__ void mse_grad_kernel(const float* y, const float* t, float* d, int n, float scale, double* loss) {
    __shared__ double red[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (i < n) {
        const float e = y[i] - t[i];
        d[i] = 2.f * e * scale;
        l = (double)e * e;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0]);
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

struct Net {
    std::vector<int> dims;  // n_layers + 1
    int residual_offset = -1;
    float *d_params = nullptr, *d_grads = nullptr, *d_m = nullptr, *d_v = nullptr;
    size_t nparams = 0;
    std::vector<size_t> w_off, b_off;
    // activations for training (acts[0] is unused: layer 0 reads the caller's
    // input), and the gradient's parts per batch split
    std::vector<float*> acts, deltas;
    int cap_batch = 0;
    float* d_part = nullptr;
    int cap_splits = 0;
    double* d_loss = nullptr;
    long long step = 0;

    int layers() const { return (int)dims.size() - 1; }

    // Batch splits of the weight gradients: 256 rows each, at most 32 (a batch
    // of 4096 fills the SMs twice over with 16; more parts cost more traffic
    // than they save).
    static int splits(int batch) { return std::min(32, (batch + 255) / 256); }

    void free_acts() {
        for (float* p : acts) cudaFree(p);
        for (float* p : deltas) cudaFree(p);
        acts.clear();
        deltas.clear();
        cap_batch = 0;
    }

    int ensure(int batch) {
        if (batch <= cap_batch) return HDC_OK;
        free_acts();
        bool ok = true;
        for (int l = 0; l <= layers(); l++) {
            float *a = nullptr, *d = nullptr;
            if (l > 0) {
                ok = ok && cudaMalloc(&a, sizeof(float) * (size_t)batch * dims[l]) == cudaSuccess;
                ok = ok && cudaMalloc(&d, sizeof(float) * (size_t)batch * dims[l]) == cudaSuccess;
            }
            acts.push_back(a);
            deltas.push_back(d);
        }
        if (!ok) {
            free_acts();
            cudaGetLastError();
            set_error("mlp: activation allocation failed");
            return HDC_ERR_ALLOC;
        }
        cap_batch = batch;
        return HDC_OK;
    }

    // the gradient's parts, which a network that only predicts does without
    int ensure_parts(int batch) {
        const int n = splits(batch);
        if (n <= cap_splits) return HDC_OK;
        cudaFree(d_part);
        d_part = nullptr;
        cap_splits = 0;
        if (cudaMalloc(&d_part, sizeof(float) * nparams * n) != cudaSuccess) {
            cudaGetLastError();
            d_part = nullptr;
            set_error("mlp: gradient allocation failed");
            return HDC_ERR_ALLOC;
        }
        cap_splits = n;
        return HDC_OK;
    }

    ~Net() {
        free_acts();
        cudaFree(d_part);
        cudaFree(d_params);
        cudaFree(d_grads);
        cudaFree(d_m);
        cudaFree(d_v);
        cudaFree(d_loss);
    }

    // forward through acts[1..L]; the output into d_y (acts[L] when NULL)
    int forward(const float* d_x, int batch, float* d_y, cudaStream_t s) {
        int rc = ensure(batch);
        if (rc) return rc;
        for (int l = 0; l < layers(); l++) {
            const bool last = l == layers() - 1;
            Epilogue ep;
            ep.bias = d_params + b_off[l];
            ep.relu = !last;
            if (last && residual_offset >= 0) {
                ep.residual = d_x + residual_offset;
                ep.residual_ld = dims[0];
            }
            HDC_CUDA_RET_INT((sgemm<true>(batch, dims[l + 1], dims[l], l == 0 ? d_x : acts[l], d_params + w_off[l],
                                          last && d_y ? d_y : acts[l + 1], ep, s)));
        }
        return HDC_OK;
    }

    // gradients of the mean squared error into d_grads after ensure_parts() and
    // forward() of the same d_x; loss (sum of squares / n) to *loss
    int backward(const float* d_x, const float* d_target, int batch, double* h_loss, cudaStream_t s) {
        const int L = layers();
        const int n = batch * dims[L];
        HDC_CUDA_RET_INT(cudaMemsetAsync(d_loss, 0, sizeof(double), s));
        mse_grad_kernel<<<(n + 255) / 256, 256, 0, s>>>(acts[L], d_target, deltas[L], n, 1.f / (float)n, d_loss);
        count_launches(1);
        // delta_l = (delta_{l+1} W_l) * relu'(y_l)
        for (int l = L - 1; l > 0; l--) {
            Epilogue ep;
            ep.mask = acts[l];
            HDC_CUDA_RET_INT((sgemm<false>(batch, dims[l], dims[l + 1], deltas[l + 1], d_params + w_off[l], deltas[l],
                                           ep, s)));
        }
        const int ns = splits(batch);
        for (int l0 = 0; l0 < L; l0 += MAXL) {
            GradArgs G;
            G.nl = std::min(MAXL, L - l0);
            G.batch = batch;
            G.rows = ((batch + ns - 1) / ns + TK - 1) / TK * TK;
            G.part = d_part;
            G.nparams = nparams;
            int tiles = 0;
            for (int i = 0; i < G.nl; i++) {
                const int l = l0 + i;
                const float* y = l == 0 ? d_x : acts[l];
                G.l[i] = GradLayer{deltas[l + 1], y, dims[l + 1], dims[l], tiles, vec_ok(deltas[l + 1], dims[l + 1], y, dims[l]),
                                   w_off[l], b_off[l]};
                tiles += ((dims[l + 1] + TM - 1) / TM) * ((dims[l] + TN - 1) / TN);
            }
            grad_kernel<<<dim3(tiles, ns), 256, 0, s>>>(G);
            count_launches(1);
        }
        grad_sum_kernel<<<(unsigned)((nparams + 255) / 256), 256, 0, s>>>(d_part, ns, nparams, d_grads);
        count_launches(1);
        HDC_CUDA_RET_INT(cudaGetLastError());
        if (h_loss) {
            double l = 0.0;
            HDC_CUDA_RET_INT(cudaMemcpyAsync(&l, d_loss, sizeof(double), cudaMemcpyDeviceToHost, s));
            HDC_CUDA_RET_INT(cudaStreamSynchronize(s));
            *h_loss = l / (double)n;
        }
        return HDC_OK;
    }
};

}  // namespace mlp
}  // namespace hdc

using hdc::mlp::Net;

extern "C" int hdc_mlp_new(int num_layers, const int* dims, int residual_offset, unsigned long long seed,
                           HdcMlp** out) {
    if (num_layers < 1 || !dims || !out) return HDC_ERR_ARG;
    Net* n = new Net();
    n->dims.assign(dims, dims + num_layers + 1);
    n->residual_offset = residual_offset;
    if (residual_offset >= 0 && residual_offset + dims[num_layers] > dims[0]) {
        delete n;
        hdc::set_error("mlp: residual slice outside the input");
        return HDC_ERR_ARG;
    }
    size_t off = 0;
    for (int l = 0; l < num_layers; l++) {
        n->w_off.push_back(off);
        off += (size_t)dims[l] * dims[l + 1];
        n->b_off.push_back(off);
        off += dims[l + 1];
    }
    n->nparams = off;
    // He initialisation for hidden layers; the output layer starts at zero so
    // that a residual net begins as the identity map of its centre input.
    std::vector<float> h(off, 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < num_layers; l++) {
        const bool last = l == num_layers - 1;
        std::normal_distribution<float> nd(0.f, std::sqrt(2.f / dims[l]));
        for (size_t i = 0; i < (size_t)dims[l] * dims[l + 1]; i++) h[n->w_off[l] + i] = last ? 0.f : nd(rng);
    }
    if (cudaMalloc(&n->d_params, sizeof(float) * off) != cudaSuccess ||
        cudaMalloc(&n->d_grads, sizeof(float) * off) != cudaSuccess ||
        cudaMalloc(&n->d_m, sizeof(float) * off) != cudaSuccess || cudaMalloc(&n->d_v, sizeof(float) * off) != cudaSuccess ||
        cudaMalloc(&n->d_loss, sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        delete n;
        hdc::set_error("mlp: parameter allocation failed");
        return HDC_ERR_ALLOC;
    }
    cudaMemcpy(n->d_params, h.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
    cudaMemset(n->d_m, 0, sizeof(float) * off);
    cudaMemset(n->d_v, 0, sizeof(float) * off);
    cudaMemset(n->d_grads, 0, sizeof(float) * off);
    *out = reinterpret_cast<HdcMlp*>(n);
    return HDC_OK;
}

extern "C" void hdc_mlp_free(HdcMlp* m) { delete reinterpret_cast<Net*>(m); }

namespace hdc {
// input and output widths of a network (for callers that build its inputs)
int mlp_io_dims(HdcMlp* m, int* in, int* out) {
    if (!m) return HDC_ERR_ARG;
    const Net* n = reinterpret_cast<const Net*>(m);
    *in = n->dims.front();
    *out = n->dims.back();
    return HDC_OK;
}
}  // namespace hdc

extern "C" long long hdc_mlp_num_params(HdcMlp* m) { return (long long)reinterpret_cast<Net*>(m)->nparams; }

extern "C" int hdc_mlp_get_params(HdcMlp* hm, float* h_out) {
    Net* n = reinterpret_cast<Net*>(hm);
    HDC_CUDA_RET_INT(cudaMemcpy(h_out, n->d_params, sizeof(float) * n->nparams, cudaMemcpyDeviceToHost));
    return HDC_OK;
}

extern "C" int hdc_mlp_set_params(HdcMlp* hm, const float* h_in) {
    Net* n = reinterpret_cast<Net*>(hm);
    HDC_CUDA_RET_INT(cudaMemcpy(n->d_params, h_in, sizeof(float) * n->nparams, cudaMemcpyHostToDevice));
    return HDC_OK;
}

extern "C" int hdc_mlp_forward(HdcMlp* hm, const float* d_x, int batch, float* d_y, hdcStream_t stream) {
    Net* n = reinterpret_cast<Net*>(hm);
    cudaStream_t s = (cudaStream_t)stream;
    // an output that overlaps the input is written once the input has been read
    const size_t nx = (size_t)batch * n->dims.front(), ny = (size_t)batch * n->dims.back();
    const bool overlap = d_y < d_x + nx && d_x < d_y + ny;
    int rc = n->forward(d_x, batch, overlap ? nullptr : d_y, s);
    if (rc || !overlap) return rc;
    HDC_CUDA_RET_INT(cudaMemcpyAsync(d_y, n->acts.back(), sizeof(float) * ny, cudaMemcpyDeviceToDevice, s));
    return HDC_OK;
}

extern "C" int hdc_mlp_gradients(HdcMlp* hm, const float* d_x, const float* d_target, int batch, float* h_grads,
                                 double* h_loss, hdcStream_t stream) {
    Net* n = reinterpret_cast<Net*>(hm);
    cudaStream_t s = (cudaStream_t)stream;
    int rc = n->ensure_parts(batch);
    if (rc) return rc;
    rc = n->forward(d_x, batch, nullptr, s);
    if (rc) return rc;
    rc = n->backward(d_x, d_target, batch, h_loss, s);
    if (rc) return rc;
    if (h_grads) {
        HDC_CUDA_RET_INT(cudaMemcpyAsync(h_grads, n->d_grads, sizeof(float) * n->nparams, cudaMemcpyDeviceToHost, s));
        HDC_CUDA_RET_INT(cudaStreamSynchronize(s));
    }
    return HDC_OK;
}

extern "C" int hdc_mlp_train_step(HdcMlp* hm, const float* d_x, const float* d_target, int batch, float lr,
                                  double* h_loss, hdcStream_t stream) {
    Net* n = reinterpret_cast<Net*>(hm);
    cudaStream_t s = (cudaStream_t)stream;
    int rc = n->ensure_parts(batch);
    if (rc) return rc;
    rc = n->forward(d_x, batch, nullptr, s);
    if (rc) return rc;
    rc = n->backward(d_x, d_target, batch, h_loss, s);
    if (rc) return rc;
    n->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)n->step), c2 = 1.f - std::pow(b2, (float)n->step);
    const int np = (int)n->nparams;
    hdc::mlp::adam_kernel<<<(np + 255) / 256, 256, 0, s>>>(n->d_params, n->d_grads, n->d_m, n->d_v, np, lr, b1, b2,
                                                           1e-8f, c1, c2);
    hdc::count_launches(1);
    HDC_CUDA_RET_INT(cudaGetLastError());
    return HDC_OK;
}
