// Tomography model update on the device: the Gaussian smoothing of
// Inversion::model_smoothing / smooth_matrix (src/inversion/inversion.cpp:
// 347-447) and the slowness update of Tomography_ISO::model_update
// (src/inversion/tomography_iso.cpp:77-92), with the reference's arithmetic.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "sf_engine.h"

using namespace sf;

#define CK(call)                                                          \
    do {                                                                  \
        int _st = sf_cuda_check(c, (call), #call);                        \
        if (_st != SF_OK) return _st;                                     \
    } while (0)

namespace {

// Output cell (i, j) of the model (nz x nx, z fastest): the reference pads the
// model with `samples` zero cells on every side, then sums samples x samples taps
// (tap (zk, xk) of the kernel on cell (i - mid + zk, j - mid + xk) of the padded
// grid) in FP32, xk outer, zk inner, product then sum. Every model cell lies
// at least mid = samples/2 cells inside the padded grid, so every model cell
// is smoothed.
//
// A CTA smooths a tile of 32 x 32 cells: a lane owns a column, a warp four
// rows of it, and a thread slides down its column of the input tile, where each
// value and each tap (both read once from shared memory) serve four cells. The
// kernel's columns come in groups of xc, so that the tile and the taps fit in
// shared memory for any kernel size.
// On a grid with fewer tiles than SMs a thread has one cell instead: the rest of
// the chip is idle, and the tile is done in a quarter of the steps (307 x 75
// cells, 9 samples: 7.6 us, 9.0 with four; 1701 x 351, 11 samples, where a
// thread's four cells share their reads: 19 us with four, 26 with one).
constexpr int kTile = 32;

// Kernels of up to 31 x 31 taps go along as an argument of the launch instead of
// a copy before it (update of 307 x 75 cells, 9 samples: 64.7 -> 62.2 us).
constexpr int kInlineTaps = 31 * 31;
struct Taps {
    float k[kInlineTaps];
    __device__ float operator[](size_t q) const { return k[q]; }
};

template <int kRows, class K_t>
__global__ void __launch_bounds__(kTile / kRows * 32) k_smooth(const float* __restrict__ in, int nx, int nz, int n, int xc,
                                                               const __grid_constant__ K_t K, float* __restrict__ out)
{
    extern __shared__ float sm_smooth[];
    const int mid = n / 2, rows = kTile + n - 1, pitch = rows | 1;
    float* tile = sm_smooth;                                     // kTile + xc - 1 columns of `rows` rows
    float* taps = sm_smooth + (size_t)(kTile + xc - 1) * pitch;  // xc x n
    const int lane = threadIdx.x & 31, row0 = (threadIdx.x >> 5) * kRows;
    const int ntz = (nz + kTile - 1) / kTile;
    const int i0 = (blockIdx.x % ntz) * kTile, j0 = (blockIdx.x / ntz) * kTile;
    float acc[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) acc[r] = 0.0f;
    for (int x0 = 0; x0 < n; x0 += xc) {
        const int nxk = min(xc, n - x0);
        __syncthreads();
        for (int cj = threadIdx.x >> 5; cj < kTile + nxk - 1; cj += kTile / kRows) {
            const int mj = j0 - mid + x0 + cj;
            for (int ci = lane; ci < rows; ci += 32) {
                const int mi = i0 - mid + ci;
                tile[cj * pitch + ci] = (mi >= 0 && mi < nz && mj >= 0 && mj < nx) ? in[mi + (size_t)mj * nz] : 0.0f;
            }
        }
        for (int q = threadIdx.x; q < nxk * n; q += blockDim.x) taps[q] = K[(size_t)x0 * n + q];
        __syncthreads();
        for (int xk = 0; xk < nxk; xk++) {
            const float* col = tile + (lane + xk) * pitch + row0;
            const float* k = taps + xk * n;
            float kk[kRows];  // tap t at t mod kRows
            // input row t serves cell r with tap t - r; the first and the last rows
            // serve fewer cells
            auto rows_from = [&](int tb, auto all) {
#pragma unroll
                for (int u = 0; u < kRows; u++) {
                    const int t = tb + u;
                    const float v = col[t];
                    kk[u] = (all.value || t < n) ? k[t] : 0.0f;
#pragma unroll
                    for (int r = 0; r < kRows; r++)
                        if (all.value || (t - r >= 0 && t - r < n))
                            acc[r] = __fadd_rn(acc[r], __fmul_rn(v, kk[(u - r) & (kRows - 1)]));
                }
            };
            int tb = 0;
            rows_from(tb, std::false_type{});
#pragma unroll 2
            for (tb = kRows; tb + kRows <= n; tb += kRows) rows_from(tb, std::true_type{});
            for (; tb < n + kRows - 1; tb += kRows) rows_from(tb, std::false_type{});
        }
    }
    const int j = j0 + lane;
    if (j < nx)
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            const int i = i0 + row0 + r;
            if (i < nz) out[i + (size_t)j * nz] = acc[r];
        }
}

// dS = scale * grad over the model interior of the padded gradient.
__global__ void k_scale_interior(const float* __restrict__ g, int nx, int nz, int nb, int nzz, float scale,
                                 float* __restrict__ dS)
{
    const size_t np = (size_t)nx * nz;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < np;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % nz), j = (int)(idx / nz);
        dS[idx] = __fmul_rn(scale, g[(i + nb) + (size_t)(j + nb) * nzz]);
    }
}

}  // namespace

// The reference's normalised Gaussian: weight 1/(pi stdv) exp(-r^2/(2 stdv^2))
// computed as its source does (the prefactor in double, expf in float, the
// product rounded once to float), summed in FP32 (x outer, z inner) and
// divided by the sum; stdv == 0 gives the unit tap at the centre.
void sf_smooth_kernel(float stdv, int n, std::vector<float>& k)
{
    k.assign((size_t)n * n, 0.0f);
    const int mid = n / 2;
    k[mid + (size_t)mid * n] = 1.0f;
    if (stdv == 0.0f) return;
    float sum = 0.0f;
    for (int x = -mid; x <= mid; x++)
        for (int z = -mid; z <= mid; z++) {
            const int index = (z + mid) + (x + mid) * n;
            const float r = std::sqrt((float)(x * x + z * z));
            k[index] = (float)(1.0f / (M_PI * stdv) * (double)std::exp(-((r * r) / (2.0f * stdv * stdv))));
            sum += k[index];
        }
    for (auto& v : k) v /= sum;
}

static int smooth_on_device(sf_ctx* c, const float* d_in, float* d_out, float stdv, int samples, cudaStream_t st)
{
    std::vector<float> k;
    sf_smooth_kernel(stdv, samples, k);
    const bool along = k.size() <= (size_t)kInlineTaps;
    Taps taps;
    if (along) {
        std::memcpy(taps.k, k.data(), k.size() * sizeof(float));
    } else {
        int rc = sf_dev_reserve(c, (void**)&c->d_skern, &c->cap_skern, k.size() * sizeof(float));
        if (rc) return rc;
        c->h_skern.swap(k);
        CK(cudaMemcpyAsync(c->d_skern, c->h_skern.data(), c->h_skern.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    }
    // as many kernel columns at a time as fit in shared memory
    int xc = std::min(samples, 16);
    auto smem = [&](int x) {
        return ((size_t)(kTile + x - 1) * ((kTile + samples - 1) | 1) + 4 + (size_t)x * samples) * sizeof(float);
    };
    while (xc > 1 && smem(xc) > (size_t)200 * 1024) xc /= 2;
    const unsigned grid = (unsigned)((c->nz + kTile - 1) / kTile) * (unsigned)((c->nx + kTile - 1) / kTile);
    const int rows = (int)grid < c->sms ? 1 : 4;
    auto launch = [&](auto kern, const auto& K) {
        if (smem(xc) > size_t(48) * 1024)  // more than a kernel has without asking
            CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem(xc)));
        kern<<<grid, kTile / rows * 32, smem(xc), st>>>(d_in, c->nx, c->nz, samples, xc, K, d_out);
        return (int)SF_OK;
    };
    const float* dk = c->d_skern;
    const int rc = along ? (rows == 1 ? launch(k_smooth<1, Taps>, taps) : launch(k_smooth<4, Taps>, taps))
                         : (rows == 1 ? launch(k_smooth<1, const float*>, dk) : launch(k_smooth<4, const float*>, dk));
    if (rc) return rc;
    CK(cudaGetLastError());
    return SF_OK;
}

static int check_samples(sf_ctx* c, int samples)
{
    if (samples < 1 || samples % 2 == 0 || samples > 1001)
        return sf_fail(c, SF_ERR_ARG, "gaussian_filter_samples must be an odd number in 1..1001");
    return SF_OK;
}

extern "C" int sf_smooth_model(sf_ctx* c, const float* in, float* out, float stdv, int samples, int mem,
                               void* stream)
{
    if (!c || !in || !out) return sf_fail(c, SF_ERR_ARG, "null argument");
    int rc = check_samples(c, samples);
    if (rc) return rc;
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    const size_t nb = (size_t)c->nx * c->nz * sizeof(float);
    const float* d_in = in;
    float* d_out = out;
    if (mem == SF_MEM_HOST) {
        rc = sf_dev_reserve(c, (void**)&c->d_upd, &c->cap_upd, 2 * nb);
        if (rc) return rc;
        CK(cudaMemcpyAsync(c->d_upd, in, nb, cudaMemcpyHostToDevice, st));
        d_in = c->d_upd;
        d_out = c->d_upd + (size_t)c->nx * c->nz;
    }
    rc = smooth_on_device(c, d_in, d_out, stdv, samples, st);
    if (rc) return rc;
    if (mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(out, d_out, nb, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

extern "C" int sf_update_slowness(sf_ctx* c, const float* grad, int grad_mem, float scale, float stdv, int samples,
                                  float* dS, int dS_mem, void* stream)
{
    if (!c || !grad) return sf_fail(c, SF_ERR_ARG, "null argument");
    if (samples != 0) {
        int rc = check_samples(c, samples);
        if (rc) return rc;
    }
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    const size_t np = (size_t)c->nx * c->nz, npad = (size_t)c->nxx * c->nzz;
    int rc = sf_dev_reserve(c, (void**)&c->d_upd, &c->cap_upd, (2 * np + npad) * sizeof(float));
    if (rc) return rc;
    float* d_a = c->d_upd;
    float* d_b = c->d_upd + np;
    const float* d_g = grad;
    if (grad_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(c->d_upd + 2 * np, grad, npad * sizeof(float), cudaMemcpyHostToDevice, st));
        d_g = c->d_upd + 2 * np;
    }
    const unsigned grid = (unsigned)std::min<size_t>((np + 255) / 256, (size_t)c->sms * 8);
    k_scale_interior<<<grid, 256, 0, st>>>(d_g, c->nx, c->nz, c->nb, c->nzz, scale, d_a);
    CK(cudaGetLastError());
    float* d_dS = d_a;
    if (samples != 0) {
        rc = smooth_on_device(c, d_a, d_b, stdv, samples, st);
        if (rc) return rc;
        d_dS = d_b;
    }
    rc = sf_wait_slowness(c, st);
    if (!rc) rc = sf_solver_slowness(c, nullptr, d_dS, st);
    if (rc) return rc;
    if (dS) CK(cudaMemcpyAsync(dS, d_dS, np * sizeof(float),
                               dS_mem == SF_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));  // the slowness is read by calls on any stream
    return SF_OK;
}
