// Building blocks of the persistent solve kernels (nsolver.cu, psolver.cu): a
// whole multigrid-preconditioned CG solve is one cooperative launch of one
// block per SM, whose phases are separated by grid barriers instead of kernel
// boundaries.
//
// Why: a CG iteration of a 256^2 .. 1024^2 model is a chain of 10 to 70 short
// dependent steps. As kernels in a graph each costs its launch gap, the
// dependent loads of its descriptors and the drain of its last blocks (5 to
// 8 us for a few hundred ns of work); a grid barrier on GB300 costs about
// 1.3 us (2.7k cycles) and the descriptors stay in the kernel's parameters.
#pragma once
#include <vector>

#include "common.cuh"

namespace f2d {

constexpr int PS_NT = 512;  // threads of a block (one block per SM)

// ---- grid barrier ------------------------------------------------------------
// Four counters on lines of their own, zeroed before the launch; a block
// increments one of them once per barrier, and the k-th barrier is passed when
// each reaches k times its number of blocks. (One counter for all 152 blocks:
// 2840 cycles with writes in flight, four: 2660. A flag per block that all
// blocks poll: 5000 to 8500; clusters with one arrival each: 3500 and more.) The wait
// is bounded: after 2 s without progress the block sets the abort word
// and the kernel's status, and every block returns from the kernel.
struct PSBar {
    unsigned int count[4][32];  // arrivals
    int abort;                  // a wait ran out
    unsigned int base;          // barriers passed by the launches before (k_ps_cycle)
    // test hook (f2d_test_grid_wait): one arrival more than there are blocks
    // (hold = 1), and the limit of the wait (0: 2 s). Never reset by a solve
    unsigned int hold;
    unsigned int limit_us;
};

struct PSGrid {
    PSBar* bar;
    int* status;
    unsigned int round, hold, limit_us;
};

__device__ __forceinline__ PSGrid ps_grid(PSBar* bar, int* status, unsigned int round)
{
    return {bar, status, round, bar->hold, bar->limit_us};
}

// zero the counters (before the launch)
__device__ __forceinline__ void ps_reset(PSBar* b)
{
    for (int k = 0; k < 4; ++k) b->count[k][0] = 0u;
    b->abort = 0;
    b->base = 0u;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Returns false when the kernel must return. Writes of all threads of all
// blocks before the barrier are visible to all threads after it: the CTA
// barrier orders them before thread 0's release, and warp 0's acquires before
// the second CTA barrier. (Data written in the kernel is read with plain loads,
// never through the read-only path.) While warp 0 waits, the other warps
// run idle(): work that needs nothing of this phase and is over in less time
// than the barrier takes.
template <typename F>
__device__ __forceinline__ bool ps_sync(PSGrid& g, F idle)
{
    __shared__ int s_dead;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned lane = threadIdx.x;
        int dead = 0;
        g.round += 1;
        if (lane == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(
                             g.bar->count[blockIdx.x & 3])
                         : "memory");
        if (lane < 4) {
            // blocks of counter `lane`
            const unsigned target = g.round * ((gridDim.x + 3 - lane) / 4) + g.hold;
            uint64_t t0 = 0;
            for (unsigned spin = 0; (int)(ld_acquire(g.bar->count[lane]) - target) < 0; ++spin) {
                if ((spin & 255u) != 255u) continue;
                const uint64_t t = globaltimer_ns();
                if (t0 == 0) t0 = t;
                // (here: used any earlier, the loads would hold the kernel's start up)
                const uint64_t limit = g.limit_us ? g.limit_us * 1000ull : 2000000000ull;
                if (t - t0 > limit || *(volatile int*)&g.bar->abort) {
                    *(volatile int*)&g.bar->abort = 1;
                    atomicOr(g.status, ST_GRID_TIMEOUT);
                    dead = 1;
                    break;
                }
            }
        }
        dead = __any_sync(0xffffffffu, dead);
        if (lane == 0) s_dead = dead;
    } else {
        idle();
    }
    __syncthreads();
    return s_dead == 0;
}

__device__ __forceinline__ bool ps_sync(PSGrid& g)
{
    return ps_sync(g, [] {});
}

// ---- deterministic sums over the blocks --------------------------------------
// The block's totals of N <= 4 per-thread values into part[k * stride]; after
// the next barrier every block adds all blocks' totals in one fixed order, so
// all blocks hold the same bits and take the same decisions
// without a broadcast. An FP64 instruction of a warp occupies its SM
// partition's pipe for 64 cycles, so sums and scalar arithmetic are kept to
// few warps: a shuffle tree in all 16 warps, or three divisions in all
// threads, cost 1.3 us and 4.6 us of a phase of 5.
template <int N>
__device__ __forceinline__ void ps_block_total(const double (&v)[N], double* part, int stride)
{
    static_assert(N <= 4, "two values per half warp of four warps");
    __shared__ double sh[N][PS_NT];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) sh[k][threadIdx.x] = v[k];
    __syncthreads();
    // warps 0 .. 3 values 0 and 1, warps 4 .. 7 values 2 and 3, each a quarter
    // of the threads' values; the second value goes to the upper half warp at
    // the first step, so the two share the rest of the tree
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, k = (w >> 2) * 2;
    if (k < N) {
        const int q = (w & 3) * (PS_NT / 4);
        const double* s = &sh[k][q + lane];
        double a = 0.0;
#pragma unroll
        for (int i = 0; i < PS_NT / 4; i += 128)
            a += (s[i] + s[i + 32]) + (s[i + 64] + s[i + 96]);
        if (k + 1 < N) {
            const double* u = &sh[k + 1 < N ? k + 1 : k][q + lane];
            double b = 0.0;
#pragma unroll
            for (int i = 0; i < PS_NT / 4; i += 128)
                b += (u[i] + u[i + 32]) + (u[i + 64] + u[i + 96]);
            const double o = __shfl_xor_sync(0xffffffffu, lane < 16 ? b : a, 16);
            a = (lane < 16 ? a : b) + o;
        } else {
            a += __shfl_xor_sync(0xffffffffu, a, 16);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        __syncwarp();
        if (lane == 0) sh[k][q] = a;
        if (lane == 16 && k + 1 < N) sh[k + 1 < N ? k + 1 : k][q] = a;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        const double* s = sh[threadIdx.x];
        part[(size_t)threadIdx.x * stride] =
            (s[0] + s[PS_NT / 4]) + (s[PS_NT / 2] + s[3 * (PS_NT / 4)]);
    }
}

// The total of p[0 .. n) in a fixed order, by one whole warp (all lanes hold it)
__device__ __forceinline__ double ps_total(const double* p, int n)
{
    const int lane = threadIdx.x & 31;
    double a = 0.0, b = 0.0;
    int i = lane;
    for (; i + 32 < n; i += 64) {
        a += __ldcg(&p[i]);
        b += __ldcg(&p[i + 32]);
    }
    if (i < n) a += __ldcg(&p[i]);
    a += b;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Two of them at once
__device__ __forceinline__ void ps_total2(const double* p, const double* q, int n, double& tp,
                                          double& tq)
{
    const int lane = threadIdx.x & 31;
    double a = 0.0, b = 0.0;
    for (int i = lane; i < n; i += 32) {
        a += __ldcg(&p[i]);
        b += __ldcg(&q[i]);
    }
    const double o = __shfl_xor_sync(0xffffffffu, lane < 16 ? b : a, 16);
    a = (lane < 16 ? a : b) + o;
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) a += __shfl_xor_sync(0xffffffffu, a, s);
    tp = __shfl_sync(0xffffffffu, a, 0);
    tq = __shfl_sync(0xffffffffu, a, 16);
}

// The grid's totals of N values, then f(totals) in thread 0, whose results
// (shared variables) all threads may read on return.
template <int N, typename F>
__device__ __forceinline__ void ps_grid_total(const double* part, F f)
{
    __shared__ double tot[N];
    const int w = threadIdx.x >> 5;
    if (w < N) {
        const double a = ps_total(part + (size_t)w * gridDim.x, gridDim.x);
        if ((threadIdx.x & 31) == 0) tot[w] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) f(tot);
    __syncthreads();
}

// quotient of a non-negative index by a positive width through an FP32
// reciprocal rw = 1/w: exact for indices below 2^20 (the fractional part of
// (k + 0.5)/w is at least 0.5/w away from an integer)
__device__ __forceinline__ int fdiv(int k, float rw) { return __float2int_rz((k + 0.5f) * rw); }

// ---- dense coarsest level -----------------------------------------------------
// x = M b for the n x n inverse M of the coarsest operator, its rows dealt to
// the blocks. The coarse correction is exact, and one more grid level would
// cost two legs and barriers, about 17k cycles. M is stored with rows of
// ps_pitch(n) elements and read 16 bytes per lane; a block whose rows fit
// beside its tiles keeps them in shared memory for the whole solve. In FP64
// n = 1024 costs 3.4k cycles of the FP64 pipe and n = 2048 14k; in FP32 the
// reads of M from L2 count (n = 3000, 37 MB: 19k cycles with 4-byte loads,
// too few bytes in flight).
constexpr int PS_NDENSE = 2048, PS_NDENSE32 = 4096;

template <typename S>
__host__ __device__ constexpr int ps_pitch(int n)
{
    constexpr int V = 16 / (int)sizeof(S);
    return (n + V - 1) / V * V;
}
// shared memory of ps_dense for `rows` rows, in elements
template <typename S>
__host__ __device__ constexpr size_t ps_dense_elems(int n, int rows)
{
    return (size_t)ps_pitch<S>(n) + 128 * (size_t)rows;
}

template <typename S> struct Vec16;
template <> struct Vec16<float> {
    using T = float4;
    static __device__ __forceinline__ float dot(float4 m, float4 b, float a)
    {
        a = fmaf(m.x, b.x, a);
        a = fmaf(m.y, b.y, a);
        a = fmaf(m.z, b.z, a);
        return fmaf(m.w, b.w, a);
    }
};
template <> struct Vec16<double> {
    using T = double2;
    static __device__ __forceinline__ double dot(double2 m, double2 b, double a)
    {
        return fma(m.y, b.y, fma(m.x, b.x, a));
    }
};

// The unknowns of a dense level in its arrays (rows of ld elements): unknown e
// is column e mod w of row e / w of the box that starts at element o.
struct PSBox {
    int w, ld, o;
    float rw;  // 1 / w
};

// rows r0 .. r1 - 1 of x = M b, row r at M + (r - r0) pitch (global or shared
// memory), the chunks of a row dealt to four warps; sb: ps_dense_elems. The
// lanes' sums of a row's quarters meet in shared memory (a shuffle tree per
// quarter would cost as many FP64 instructions as the row's products).
template <typename S>
__device__ __forceinline__ void ps_dense(const S* M, const S* b, S* x, int n, int r0, int r1,
                                         S* sb, const PSBox& box)
{
    using V = typename Vec16<S>::T;
    constexpr int NW = PS_NT / 32, U = 4, VN = 16 / (int)sizeof(S), CH = 32 * VN;
    const int np = ps_pitch<S>(n);
    S* part = sb + np;  // 128 per row
    if (r1 <= r0) return;
    auto at = [&](int e) {
        const int r = fdiv(e, box.rw);
        return box.o + r * box.ld + e - r * box.w;
    };
    for (int e0 = threadIdx.x; e0 < np; e0 += 4 * PS_NT) {
        S v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * PS_NT;
            v[u] = e < n ? __ldcg(&b[at(e)]) : S(0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e0 + u * PS_NT < np) sb[e0 + u * PS_NT] = v[u];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < 4 * (r1 - r0); t += NW) {
        const S* m = M + (size_t)(t >> 2) * np;
        S a = S(0);
        for (int e = (t & 3) * CH + lane * VN; e < np; e += 4 * CH * U) {
            V v[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (e + 4 * CH * u < np) v[u] = *(const V*)(m + e + 4 * CH * u);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (e + 4 * CH * u < np)
                    a = Vec16<S>::dot(v[u], *(const V*)(sb + e + 4 * CH * u), a);
        }
        part[32 * t + lane] = a;
    }
    __syncthreads();
    // 8 lanes per row add 16 values each, then a tree over the 8
    for (int t0 = 0; t0 < 8 * (r1 - r0); t0 += PS_NT) {
        const int t = t0 + threadIdx.x;
        const bool in = t < 8 * (r1 - r0);
        S a = S(0);
        if (in) {
            // (stride 8: consecutive lanes read consecutive elements)
            const S* p = part + 128 * (t >> 3) + (t & 7);
#pragma unroll
            for (int u = 0; u < 16; ++u) a += p[8 * u];
        }
        if (__any_sync(0xffffffffu, in)) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (in && (t & 7) == 0) x[at(r0 + (t >> 3))] = a;
        }
    }
}

// copy `bytes` (a multiple of 16) of global memory to shared memory
__device__ __forceinline__ void ps_copy16(void* dst, const void* src, size_t bytes)
{
    const int4* g = (const int4*)src;
    int4* d = (int4*)dst;
    for (int k = threadIdx.x; k < (int)(bytes / 16); k += PS_NT) d[k] = __ldg(&g[k]);
}

// Host: the inverse of a symmetric positive definite banded matrix H of n
// rows, band[i (bw + 1) + k] = H(i, i - k), times `scale`, as n rows of
// ps_pitch(n) doubles (prec 0) or floats on the device (zeros behind column
// n). Cholesky on the host (ps_band_ok
// bounds its n bw^2 operations), the columns of the inverse on the GPU. part:
// empty, or a part number per row: the constants of a part are projected out
// of the result from both sides, and rows of part -1 become 0. 0 on success: the
// work is on the default stream, which the caller synchronises before the
// scratch goes or another stream reads the result.
struct PSScratch {  // device memory of the inversions of one set-up
    void* p = nullptr;
    size_t bytes = 0;
    PSScratch() = default;
    PSScratch(const PSScratch&) = delete;
    PSScratch& operator=(const PSScratch&) = delete;
    ~PSScratch() { cudaFree(p); }
    void* get(size_t n)
    {
        if (n > bytes) {
            cudaFree(p);  // (waits for its readers)
            p = nullptr;
            bytes = cudaMalloc(&p, n) == cudaSuccess ? n : 0;
        }
        return bytes ? p : nullptr;
    }
};
int ps_invert(const std::vector<double>& band, int n, int bw, const std::vector<int>& part,
              double scale, int prec, void* out, PSScratch& scratch);
// whether a level of n cells in rows of bw may be the dense one
inline bool ps_band_ok(long long n, long long bw, int prec)
{
    return n <= (prec == 0 ? PS_NDENSE : PS_NDENSE32) && n * bw * bw <= 50000000ll;
}
// The test hook of the barrier's wait: limit_us > 0 makes every one run out
// after it, 0 ends that.
int ps_test_wait(PSBar* bar, unsigned int limit_us);
// Launch a cooperative kernel of PS_NT threads per block.
int ps_launch(const void* kern, int grid, size_t smem, void** args, cudaStream_t st);
// SMs of the current device.
int ps_sms();

}  // namespace f2d
