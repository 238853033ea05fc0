// Host side of the persistent solve kernels (persist.cuh): the inverse of the
// coarsest operator and the cooperative launch.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "persist.cuh"

namespace f2d {

// Columns of the inverse of H = L L^T (bandwidth bw), a warp per column in
// shared memory: both substitutions in axpy form, a step's bw updates across
// the lanes, down to the diagonal only (the rest is the transpose's). lc:
// columns of L below the diagonal, lr: its rows left of it (bw each), id:
// 1 / diagonal. Bound by the chain of 2 (n - j) dependent steps, so the next
// step's row (its first 64 entries) and 1 / diagonal are loaded a step ahead:
// n = 2976, bw = 62: 7.9 -> 2.4 ms with the allocations and copies around it.
constexpr int BI_W = 8;  // warps (columns) per block, at most
__device__ __forceinline__ void band_step(double* x, const double* __restrict__ row, int lane,
                                          int bw, int room, int dir, double xi, double r0,
                                          double r1)
{
    const int m = min(bw, room);
    if (lane < m) x[dir * (1 + lane)] -= r0 * xi;
    if (lane + 32 < m) x[dir * (33 + lane)] -= r1 * xi;
    for (int k = lane + 64; k < m; k += 32) x[dir * (1 + k)] -= row[k] * xi;
    __syncwarp();
}

__global__ void __launch_bounds__(32 * BI_W)
k_band_inverse(const double* __restrict__ lc, const double* __restrict__ lr,
               const double* __restrict__ id, int n, int bw, double* __restrict__ out)
{
    extern __shared__ double cols[];
    const int lane = threadIdx.x & 31, j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= n) return;
    double* x = cols + (size_t)(threadIdx.x >> 5) * n;
    for (int i = j + lane; i < n; i += 32) x[i] = i == j ? 1.0 : 0.0;
    __syncwarp();
    auto first = [&](const double* l, int i) { return lane < bw ? l[(size_t)i * bw + lane] : 0.0; };
    auto second = [&](const double* l, int i) {
        return lane + 32 < bw ? l[(size_t)i * bw + lane + 32] : 0.0;
    };
    double r0 = first(lc, j), r1 = second(lc, j), d = id[j];
    for (int i = j; i < n; ++i) {
        const int q = min(i + 1, n - 1);
        const double n0 = first(lc, q), n1 = second(lc, q), nd = id[q];
        const double xi = x[i] * d;
        __syncwarp();
        if (lane == 0) x[i] = xi;
        band_step(x + i, lc + (size_t)i * bw, lane, bw, n - 1 - i, 1, xi, r0, r1);
        r0 = n0;
        r1 = n1;
        d = nd;
    }
    r0 = first(lr, n - 1);
    r1 = second(lr, n - 1);
    d = id[n - 1];
    for (int i = n - 1; i >= j; --i) {
        const int q = max(i - 1, 0);
        const double n0 = first(lr, q), n1 = second(lr, q), nd = id[q];
        const double xi = x[i] * d;
        __syncwarp();
        if (lane == 0) x[i] = xi;
        band_step(x + i, lr + (size_t)i * bw, lane, bw, i - j, -1, xi, r0, r1);
        r0 = n0;
        r1 = n1;
        d = nd;
    }
    for (int i = j + lane; i < n; i += 32) out[(size_t)j * n + i] = x[i];
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
            if (part[j] == part[i]) a += X[(size_t)min(i, j) * n + max(i, j)];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) r[i] = a * isize[i];
}

// out = scale (X - row mean - column mean + mean) inside a part (X symmetric,
// its rows from the diagonal on:
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
    double v = X[(size_t)min(i, j) * n + max(i, j)];
    if (part) v = part[i] >= 0 && part[i] == part[j] ? v - (r[i] + r[j]) + mean[i] : 0.0;
    out[e] = (S)(scale * v);
}

static_assert(PS_NDENSE32 <= 2 * PS_NDENSE, "shared memory of k_band_inverse");

int ps_invert(const std::vector<double>& band, int n, int bw, const std::vector<int>& part,
              double scale, int prec, void* out, PSScratch& scratch)
{
    // Right-looking Cholesky in column bands, c[j w1 + k] = H(j + k, j), B
    // columns at a time: one update of the columns after them costs a load and
    // a store for B products (a product a time: n = 2976, bw = 62: 4.5 ms; this:
    // 1.1 ms)
    constexpr int B = 4;
    const int w1 = bw + 1, np = (n + B - 1) / B * B, cp = w1 + bw + B;
    std::vector<double> c((size_t)(np + bw + B) * w1, 0.0), col((size_t)B * cp, 0.0);
    std::vector<double> lc((size_t)n * bw, 0.0), lr((size_t)n * bw, 0.0), id(n);
    for (int i = 0; i < n; ++i)
        for (int k = 0; k <= std::min(bw, i); ++k)
            c[(size_t)(i - k) * w1 + k] = band[(size_t)i * w1 + k];
    for (int i = n; i < np; ++i) c[(size_t)i * w1] = 1.0;  // (padding)
    for (int j = 0; j < np; j += B) {
        // columns j .. j + B - 1 of L (col, zero past the band)
        for (int q = 0; q < B; ++q) {
            double *cj = &c[(size_t)(j + q) * w1], *L = &col[(size_t)q * cp];
            for (int p = 0; p < q; ++p) {
                const double* P = &col[(size_t)p * cp] + (q - p);
                const double f = P[0];
                for (int k = 0; k <= bw; ++k) cj[k] -= f * P[k];
            }
            if (!(cj[0] > 0.0)) return 5;
            L[0] = std::sqrt(cj[0]);
            const double r = 1.0 / L[0];
            for (int k = 1; k <= bw; ++k) L[k] = cj[k] * r;
            if (j + q >= n) continue;
            id[j + q] = r;
            for (int k = 0; k < bw && j + q + 1 + k < n; ++k) {
                lc[(size_t)(j + q) * bw + k] = L[k + 1];
                lr[(size_t)(j + q + 1 + k) * bw + k] = L[k + 1];
            }
        }
        // their products off the columns j + B .. of the band
        for (int m = B; m < bw + B; ++m) {
            double* __restrict__ t = &c[(size_t)(j + m) * w1];
            const double* __restrict__ s0 = &col[m];
            const double* __restrict__ s1 = &col[cp + m - 1];
            const double* __restrict__ s2 = &col[2 * cp + m - 2];
            const double* __restrict__ s3 = &col[3 * cp + m - 3];
            const double f0 = s0[0], f1 = s1[0], f2 = s2[0], f3 = s3[0];
            const int e = std::min(bw, bw - m + B - 1);
            for (int k = 0; k <= e; ++k)
                t[k] -= (f0 * s0[k] + f1 * s1[k]) + (f2 * s2[k] + f3 * s3[k]);
        }
    }
    // one allocation, one copy (an allocation per array and a synchronisation per
    // member were half of the set-up of an ensemble of small members)
    const size_t nb = (size_t)n * bw, nn = (size_t)n * n;
    std::vector<double> host(2 * nb + 4 * (size_t)n, 0.0);
    std::copy(lc.begin(), lc.end(), host.begin());
    std::copy(lr.begin(), lr.end(), host.begin() + nb);
    std::copy(id.begin(), id.end(), host.begin() + 2 * nb);
    double* isize = &host[2 * nb + n];
    if (!part.empty()) {
        std::vector<double> cnt(n, 0.0);
        for (int i = 0; i < n; ++i)
            if (part[i] >= 0) cnt[part[i]] += 1.0;
        for (int i = 0; i < n; ++i)
            if (part[i] >= 0) isize[i] = 1.0 / cnt[part[i]];
        memcpy(&host[2 * nb + 2 * (size_t)n], part.data(), (size_t)n * sizeof(int));
    }
    double* d = (double*)scratch.get((host.size() + nn) * 8);
    if (!d) return 2;
    if (cudaMemcpy(d, host.data(), host.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
        return 2;
    double *dlr = d + nb, *did = d + 2 * nb, *dsz = did + n, *dr = dsz + 2 * n;
    int* dpart = part.empty() ? nullptr : (int*)(dsz + n);
    double* X = d + host.size();
    const int w = n <= PS_NDENSE ? BI_W : BI_W / 2;
    const size_t smem = (size_t)w * n * sizeof(double);
    if (cudaFuncSetAttribute(k_band_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             BI_W * PS_NDENSE * (int)sizeof(double)) != cudaSuccess)
        return 3;
    k_band_inverse<<<(n + w - 1) / w, 32 * w, smem>>>(d, dlr, did, n, bw, X);
    double* dm = nullptr;
    if (dpart) {
        k_row_means<<<(n + 7) / 8, 256>>>(X, dpart, dsz, n, dr);
        std::vector<double> r(n), sum(n, 0.0), mean(n, 0.0);
        if (cudaMemcpy(r.data(), dr, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
            return 2;
        for (int i = 0; i < n; ++i)
            if (part[i] >= 0) sum[part[i]] += r[i] * isize[i];
        for (int i = 0; i < n; ++i)
            if (part[i] >= 0) mean[i] = sum[part[i]];
        dm = dsz;  // (the sizes are not needed any more)
        if (cudaMemcpy(dm, mean.data(), (size_t)n * 8, cudaMemcpyHostToDevice) != cudaSuccess)
            return 2;
    }
    const unsigned ng = (unsigned)(((size_t)n * (n + 4) + 255) / 256);
    if (prec == 0)
        k_inverse_out<double><<<ng, 256>>>(X, dpart, dr, dm, n, scale, (double*)out);
    else
        k_inverse_out<float><<<ng, 256>>>(X, dpart, dr, dm, n, scale, (float*)out);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int ps_test_wait(PSBar* bar, unsigned int limit_us)
{
    if (!bar) return 0;
    const unsigned int v[2] = {limit_us ? 1u : 0u, limit_us};
    return (int)cudaMemcpy(&bar->hold, v, sizeof(v), cudaMemcpyHostToDevice);
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
