// Host side of the persistent solve kernels (persist.cuh): the inverse of the
// coarsest operator and the cooperative launch.
#include <algorithm>
#include <cmath>
#include <vector>

#include "persist.cuh"

namespace f2d {

// Columns of the inverse of H = L L^T (bandwidth bw), a warp per column in
// shared memory: both substitutions in axpy form, a step's bw updates across
// the lanes. lc: columns of L below the diagonal, lr: its rows left of it (bw
// each), id: 1 / diagonal. Bound by the chain of 2 n dependent steps (about
// 200 cycles each): 0.4 ms at n = 1600, bw = 40, where one launch per pivot
// of a Gauss-Jordan elimination of the full matrix took 34 ms.
constexpr int BI_W = 8;  // warps (columns) per block, at most
__global__ void __launch_bounds__(32 * BI_W)
k_band_inverse(const double* __restrict__ lc, const double* __restrict__ lr,
               const double* __restrict__ id, int n, int bw, double* __restrict__ out)
{
    extern __shared__ double cols[];
    const int lane = threadIdx.x & 31, j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= n) return;
    double* x = cols + (size_t)(threadIdx.x >> 5) * n;
    for (int i = lane; i < n; i += 32) x[i] = i == j ? 1.0 : 0.0;
    __syncwarp();
    for (int i = j; i < n; ++i) {
        const double xi = x[i] * id[i];
        __syncwarp();
        if (lane == 0) x[i] = xi;
        for (int k = lane; k < bw && i + 1 + k < n; k += 32)
            x[i + 1 + k] -= lc[(size_t)i * bw + k] * xi;
        __syncwarp();
    }
    for (int i = n - 1; i >= 0; --i) {
        const double xi = x[i] * id[i];
        __syncwarp();
        if (lane == 0) x[i] = xi;
        for (int k = lane; k < bw && i - 1 - k >= 0; k += 32)
            x[i - 1 - k] -= lr[(size_t)i * bw + k] * xi;
        __syncwarp();
    }
    for (int i = lane; i < n; i += 32) out[(size_t)j * n + i] = x[i];
}

// mean of row i over its part; one warp per row
__global__ void k_row_means(const double* __restrict__ X, const int* __restrict__ part,
                            const double* __restrict__ isize, int n, double* __restrict__ r)
{
    const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;
    double a = 0.0;
    if (part[i] >= 0)
        for (int j = lane; j < n; j += 32)
            if (part[j] == part[i]) a += X[(size_t)i * n + j];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) r[i] = a * isize[i];
}

// out = scale (X - row mean - column mean + mean) inside a part (X symmetric:
// its column means are the row means), 0 between parts and in dead rows
template <typename S>
__global__ void k_inverse_out(const double* __restrict__ X, const int* __restrict__ part,
                              const double* __restrict__ r, const double* __restrict__ mean,
                              int n, double scale, S* __restrict__ out)
{
    const int np = ps_pitch<S>(n);
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)n * np) return;
    const int i = (int)(e / np), j = (int)(e % np);
    if (j >= n) {
        out[e] = S(0);
        return;
    }
    // the mean of the two triangles: exactly symmetric
    double v = 0.5 * (X[(size_t)i * n + j] + X[(size_t)j * n + i]);
    if (part) v = part[i] >= 0 && part[i] == part[j] ? v - (r[i] + r[j]) + mean[i] : 0.0;
    out[e] = (S)(scale * v);
}

static_assert(PS_NDENSE32 <= 2 * PS_NDENSE, "shared memory of k_band_inverse");

int ps_invert(const std::vector<double>& band, int n, int bw, const std::vector<int>& part,
              double scale, int prec, void* out)
{
    const int w1 = bw + 1;
    // L, row i: l[i w1 + k] = L(i, i - k)
    std::vector<double> l((size_t)n * w1, 0.0), lc((size_t)n * bw, 0.0), lr((size_t)n * bw, 0.0),
        id(n);
    for (int i = 0; i < n; ++i) {
        const int j0 = std::max(0, i - bw);
        // (rows reversed: L(i, j) = row[i - j], so the products of rows i and
        // j run over m = j - 1 .. as row_i[i - m] row_j[j - m])
        double* li = &l[(size_t)i * w1];
        for (int j = j0; j <= i; ++j) {
            const double* lj = &l[(size_t)j * w1];
            const int m0 = std::max(j0, j - bw);
            double s = band[(size_t)i * w1 + i - j];
            const double *pi = li + (i - j) + 1, *pj = lj + 1;
            for (int m = 0; m < j - m0; ++m) s -= pi[m] * pj[m];
            if (j < i) li[i - j] = s * id[j];
            else {
                if (!(s > 0.0)) return 5;
                li[0] = std::sqrt(s);
                id[i] = 1.0 / li[0];
            }
        }
        for (int k = 0; k < bw && i - 1 - k >= 0; ++k) {
            lr[(size_t)i * bw + k] = li[k + 1];
            lc[(size_t)(i - 1 - k) * bw + k] = li[k + 1];
        }
    }
    std::vector<void*> tmp;
    auto dal = [&](size_t bytes, const void* src) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
        tmp.push_back(p);
        if (src && cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
        return p;
    };
    auto run = [&]() -> int {
        double* dlc = (double*)dal(lc.size() * 8, lc.data());
        double* dlr = (double*)dal(lr.size() * 8, lr.data());
        double* did = (double*)dal(id.size() * 8, id.data());
        double* X = (double*)dal((size_t)n * n * 8, nullptr);
        if (!dlc || !dlr || !did || !X) return 2;
        const int w = n <= PS_NDENSE ? BI_W : BI_W / 2;
        const size_t smem = (size_t)w * n * sizeof(double);
        if (cudaFuncSetAttribute(k_band_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 BI_W * PS_NDENSE * (int)sizeof(double)) != cudaSuccess)
            return 3;
        k_band_inverse<<<(n + w - 1) / w, 32 * w, smem>>>(dlc, dlr, did, n, bw, X);
        int* dpart = nullptr;
        double *dr = nullptr, *dm = nullptr;
        if (!part.empty()) {
            std::vector<double> isize(n, 0.0), cnt(n, 0.0), r(n), sum(n, 0.0), mean(n, 0.0);
            for (int i = 0; i < n; ++i)
                if (part[i] >= 0) cnt[part[i]] += 1.0;
            for (int i = 0; i < n; ++i)
                if (part[i] >= 0) isize[i] = 1.0 / cnt[part[i]];
            dpart = (int*)dal((size_t)n * 4, part.data());
            double* dsz = (double*)dal((size_t)n * 8, isize.data());
            dr = (double*)dal((size_t)n * 8, nullptr);
            if (!dpart || !dsz || !dr) return 2;
            k_row_means<<<(n + 7) / 8, 256>>>(X, dpart, dsz, n, dr);
            if (cudaMemcpy(r.data(), dr, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
                return 2;
            for (int i = 0; i < n; ++i)
                if (part[i] >= 0) sum[part[i]] += r[i] * isize[i];
            for (int i = 0; i < n; ++i)
                if (part[i] >= 0) mean[i] = sum[part[i]];
            dm = (double*)dal((size_t)n * 8, mean.data());
            if (!dm) return 2;
        }
        const unsigned ng = (unsigned)(((size_t)n * (n + 4) + 255) / 256);
        if (prec == 0)
            k_inverse_out<double><<<ng, 256>>>(X, dpart, dr, dm, n, scale, (double*)out);
        else
            k_inverse_out<float><<<ng, 256>>>(X, dpart, dr, dm, n, scale, (float*)out);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 3;
    };
    const int rc = run();
    for (void* p : tmp) cudaFree(p);
    return rc;
}

int ps_launch(const void* kern, int grid, size_t smem, void** args, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(PS_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelExC(&cfg, kern, args);
}

int ps_sms()
{
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return n;
}

}  // namespace f2d
