// Multigrid-preconditioned CG for the masked cell-centred Poisson operator
// with Neumann walls: Poisson2D(mesh, "c") of the reference (elliptic.py:
// 71-87, 114-195), the pressure solve of pressure_projection
// (operators.py:114-119). The reference factorises the singular matrix with
// SuperLU; here it is solved matrix-free.
//
// Operator at a fluid cell c, with face couplings f (dy/dx across x-faces,
// dx/dy across y-faces, 0 where either side is not fluid):
//     (A x)_c = sum_faces f (x_n - x_c)
// which is the reference's matrix (off-diagonals for present neighbours,
// diagonal minus their sum), in difference form. A is singular (constants),
// so the right-hand side is projected to zero mean over the fluid cells (the
// compatibility condition; for a divergence it is zero up to rounding) and
// the solution is returned with zero mean: the pressure is defined up to a
// constant, and only its gradient enters the model. One connected fluid region
// is assumed: the mean is that of all fluid cells. Unconnected basins are
// solvable where each one's sum of b is 0 to rounding by itself (the divergence
// of an FP64 velocity); an FP32 velocity leaves 1e-7 of it in each, that system
// has no solution, and the solve reports its iteration limit.
//
// Preconditioner: cell-centred V-cycle with red-black Gauss-Seidel (2 sweeps
// per leg, symmetric order), coarse cells = 2x2 agglomerates (fluid if any
// child is), restriction = sum of the children's residuals, prolongation =
// the parent's value, coarse couplings = half the sum of the fine face
// couplings a coarse face contains. (The sum itself is the Galerkin operator
// R A P for this R and P; with piecewise-constant P it is twice too stiff for
// smooth errors, and the coarse correction comes out halved - half the sum is
// the re-discretised coupling where the face is fully open and keeps the
// partial openings of masked faces.) The first level of at most 2048 cells is
// solved exactly with its precomputed dense pseudo-inverse (the FP32 form: 4096
// cells and the matrix of the V-cycle from it on, coarse_map). The FP32 form
// runs the cycle in FP32 (levels, couplings and smoothing in float; its
// right-hand side is the FP64 Krylov residual rounded, its result converted
// back), while the Krylov vectors, the operator products, the dot products and
// the zero-mean projections stay FP64.
//
// The solve is one cooperative kernel (persist.cuh), one block per SM. CG in
// the form of Chronopoulos and Gear (s-step methods for symmetric linear
// systems, J. Comput. Appl. Math. 25, 1989; here s = 1): with w = A z the two
// inner products <r, z> and <z, w> come from one pass, s = A p by the same
// recurrence as p, so an iteration has 2 (grid levels) + 1 barriers:
//   A   update s, r, p, x (r also on the tile's halo, recomputed), <r, r>,
//       and the pre-smoothing, residual and restriction of level 0
//   D_l the down legs of the other grid levels
//   the dense level
//   U_l the up legs
//   B   the up leg of level 0 with z one cell past the tile, w = A z, the
//       two inner products
// A leg works on a tile and a halo of the 4 (B: 5) cells its half sweeps
// reach over, in shared memory, so a leg needs one barrier; tile sizes are
// chosen per level so that the chip is filled (pick_tile).
// What bounds it: at 40^2 (one iteration on the dense level, 42 us) the latency
// of its phases and barriers; at 512^2 FP64 (75 us an iteration) the FP64 pipe,
// 40 % busy, and between its bursts the loads of a phase and the barriers (2.6k
// cycles each). One launch per sweep and level before it: 11.8 ms a step of
// euler 512^2, now 1.84 with the warm start.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <numeric>

#include "nsolver.cuh"
#include "persist.cuh"

namespace f2d {

constexpr int NS_H = 5;  // halo of the widest leg

// A staged region of a tile: rows J0 - h .. J0 + th + h - 1, columns alike
template <typename S>
struct NReg {
    S *x, *b, *fx, *fy, *inv;
    uint8_t* code;
    int J0, I0, h, W, RH;
    float rW;
};

// level-0 tables in the cycle's precision (shared memory)
template <typename S>
struct NTab {
    S cxi[9], cyi[9], inv[9], cs[9];
};

__device__ __forceinline__ int n_open(uint8_t c)
{
    return 3 * (((c >> 1) & 1) + ((c >> 2) & 1)) + ((c >> 3) & 1) + ((c >> 4) & 1);
}

// wrapped column of a region cell; false outside the level
__device__ __forceinline__ bool n_cell(const NLevel& L, int J, int& I)
{
    if (J < 0 || J >= L.nyn) return false;
    if (L.per) {
        // a tile wider than the level wraps more than once
        while (I < 0) I += L.nxn;
        while (I >= L.nxn) I -= L.nxn;
        return true;
    }
    return I >= 0 && I < L.nxn;
}

// the Gauss-Seidel value of region cell e (0 at cells without couplings)
template <typename S, bool L0>
__device__ __forceinline__ S n_gs(const NReg<S>& R, const NTab<S>& T, int e)
{
    if constexpr (L0) {
        const uint8_t c = R.code[e];
        const int k = n_open(c);
        const S xw = c & 2 ? R.x[e - 1] : S(0), xe = c & 4 ? R.x[e + 1] : S(0);
        const S xs = c & 8 ? R.x[e - R.W] : S(0), xn = c & 16 ? R.x[e + R.W] : S(0);
        // b holds b / (coupling sum)
        return T.cxi[k] * (xw + xe) + (T.cyi[k] * (xs + xn) - R.b[e]);
    } else {
        S v = R.fx[e] * R.x[e - 1] - R.b[e];
        v = R.fx[e + 1] * R.x[e + 1] + v;
        v = R.fy[e] * R.x[e - R.W] + v;
        v = R.fy[e + R.W] * R.x[e + R.W] + v;
        return v * R.inv[e];
    }
}

// residual b - A x at region cell e = (coupling sum) (x - Gauss-Seidel value)
template <typename S, bool L0>
__device__ __forceinline__ S n_res(const NReg<S>& R, const NTab<S>& T, int e)
{
    if constexpr (L0) {
        return T.cs[n_open(R.code[e])] * (R.x[e] - n_gs<S, true>(R, T, e));
    } else {
        S v = R.fx[e] * R.x[e - 1] - R.b[e];
        v = R.fx[e + 1] * R.x[e + 1] + v;
        v = R.fy[e] * R.x[e - R.W] + v;
        v = R.fy[e + R.W] * R.x[e + R.W] + v;
        const S cs = (R.fx[e] + R.fx[e + 1]) + (R.fy[e] + R.fy[e + R.W]);
        return cs * R.x[e] - v;
    }
}

// Half sweep of one colour over the cells within rad of the tile, next to a
// seam (a periodic level of odd width: the cells at both ends of the wrap are
// of one colour). Every value is formed before any is written, which is
// Jacobi across the seam and keeps the cycle symmetric.
constexpr int NS_SEAM_T = 32;  // tile rows and columns of such a level, at most
template <typename S, bool L0>
__device__ __noinline__ void n_half_seam(NReg<S> R, const NTab<S>& T, const NLevel& L, int color,
                                         int rad)
{
    constexpr int N = NS_SEAM_T + 2 * (NS_H - 1), MAXC = (N * N + PS_NT - 1) / PS_NT;
    const int o = R.h - rad, nr = L.th + 2 * rad;
    const int wc = L.tw + 2 * rad;
    const float rw = 1.0f / (float)wc;
    S v[MAXC];
#pragma unroll
    for (int q = 0; q < MAXC; ++q) {
        const int k = threadIdx.x + q * PS_NT;
        v[q] = S(0);
        if (k < nr * wc) {
            const int a = fdiv(k, rw);
            v[q] = n_gs<S, L0>(R, T, (o + a) * R.W + o + k - a * wc);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < MAXC; ++q) {
        const int k = threadIdx.x + q * PS_NT;
        if (k >= nr * wc) continue;
        const int a = fdiv(k, rw), r = o + a, c = o + k - a * wc;
        int I = R.I0 - R.h + c;
        const int J = R.J0 - R.h + r;
        if (n_cell(L, J, I) && ((J + I) & 1) == color) R.x[r * R.W + c] = v[q];
    }
    __syncthreads();
}

// Half sweep of one colour over the cells within rad of the tile
template <typename S, bool L0>
__device__ __forceinline__ void n_half(const NReg<S>& R, const NTab<S>& T, const NLevel& L,
                                       int color, int rad)
{
    if (L.seam) {
        n_half_seam<S, L0>(R, T, L, color, rad);
        return;
    }
    const int o = R.h - rad, nr = L.th + 2 * rad;
    const int wc = L.tw / 2 + rad;
    const float rw = 1.0f / (float)wc;
    for (int k = threadIdx.x; k < nr * wc; k += PS_NT) {
        const int a = fdiv(k, rw), r = o + a;
        // J0, I0 are even: the colour of region cell (r, c) is r + c
        const int c = o + 2 * (k - a * wc) + ((r + o + color) & 1);
        const int e = r * R.W + c;
        R.x[e] = n_gs<S, L0>(R, T, e);
    }
    __syncthreads();
}

// whether region cell (r, c) is red (the colour of the wrapped cell)
template <typename S>
__device__ __forceinline__ bool n_red(const NReg<S>& R, const NLevel& L, int r, int c)
{
    if (!L.seam) return ((r + c) & 1) == 0;
    int I = R.I0 - R.h + c;
    const int J = R.J0 - R.h + r;
    return n_cell(L, J, I) && ((J + I) & 1) == 0;
}

template <typename S>
__device__ __forceinline__ void n_region(NReg<S>& R, const NLevel& L, int tile, int h,
                                         unsigned char* smem, bool l0)
{
    const int ty = tile / L.ntx, tx = tile - ty * L.ntx;
    R.J0 = ty * L.th;
    R.I0 = tx * L.tw;
    R.h = h;
    R.W = L.tw + 2 * h;
    R.RH = L.th + 2 * h;
    R.rW = 1.0f / (float)R.W;
    const int n = R.W * R.RH;
    S* p = (S*)smem;
    R.x = p;
    R.b = p + n;
    if (l0) {
        R.code = (uint8_t*)(p + 2 * n);
        R.fx = R.fy = R.inv = nullptr;
    } else {
        R.fx = p + 2 * n;
        R.fy = p + 3 * n;
        R.inv = p + 4 * n;
        R.code = nullptr;
    }
}

// The cells of a region in batches of NB per thread: load(q, in, k, r, c) for
// the NB cells (k: the element of cell (r, c) if it lies in the level; the
// loads of a batch are in flight together), then use(q, e, in, k, r, c).
constexpr int NB = 2;
template <typename S, typename FL, typename FU>
__device__ __forceinline__ void n_load(const NReg<S>& R, const NLevel& L, FL load, FU use)
{
    const int n = R.W * R.RH;
    for (int e0 = threadIdx.x; e0 < n; e0 += NB * PS_NT) {
        int rc[NB];
        long long k[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int e = e0 + q * PS_NT;
            const int r = fdiv(e, R.rW), c = e - r * R.W;
            int I = R.I0 - R.h + c;
            const int J = R.J0 - R.h + r;
            const bool in = e < n && n_cell(L, J, I);
            rc[q] = (r << 16) | c;
            k[q] = in ? L.off + (long long)J * L.pitch + I : -1;
            // (the wrapped cell's colour and column are needed below)
            load(q, in, k[q], J, I);
        }
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int e = e0 + q * PS_NT;
            if (e < n) use(q, e, k[q] >= 0, k[q], rc[q] >> 16, rc[q] & 0xffff);
        }
    }
}

// coarse b of the agglomerates of the tile: the sum of the children's
// residuals. After a black half sweep the black residuals are zero and only
// the two red children contribute (all four next to a seam).
template <typename S, bool L0>
__device__ __forceinline__ void n_restrict(const NReg<S>& R, const NTab<S>& T, const NLevel& F,
                                           const NLevel& C)
{
    const int wc = F.tw / 2, nc = wc * (F.th / 2);
    const float rw = 1.0f / (float)wc;
    for (int k = threadIdx.x; k < nc; k += PS_NT) {
        const int a = fdiv(k, rw), c = k - a * wc;
        const int J = R.J0 / 2 + a, I = R.I0 / 2 + c;
        if (J >= C.nyn || I >= C.nxn) continue;
        const int e = (R.h + 2 * a) * R.W + R.h + 2 * c;
        S v = n_res<S, L0>(R, T, e);
        if (!F.seam) v += n_res<S, L0>(R, T, e + R.W + 1);
        else {
            v += n_res<S, L0>(R, T, e + R.W);
            // the last agglomerate of an odd count has one column (the next
            // one of the region is the wrapped first)
            if (2 * I + 1 < F.nxn)
                v += n_res<S, L0>(R, T, e + 1) + n_res<S, L0>(R, T, e + R.W + 1);
        }
        ((S*)C.b)[C.off + (long long)J * C.pitch + I] = v;
    }
}

// The tile's cells in batches, as n_load: load(q, in, k, e), use(q, k, e) with
// k the element and e the region index of a cell of the level
template <typename S, typename FL, typename FU>
__device__ __forceinline__ void n_tile(const NReg<S>& R, const NLevel& L, FL load, FU use)
{
    const int n = L.tw * L.th;
    const float rw = 1.0f / (float)L.tw;
    for (int e0 = threadIdx.x; e0 < n; e0 += NB * PS_NT) {
        int e[NB];
        long long k[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int i = e0 + q * PS_NT;
            const int a = fdiv(i, rw), c = i - a * L.tw;
            const int J = R.J0 + a, I = R.I0 + c;
            const bool in = i < n && J < L.nyn && I < L.nxn;
            k[q] = in ? L.off + (long long)J * L.pitch + I : -1;
            e[q] = (R.h + a) * R.W + R.h + c;
            load(q, in, k[q], e[q]);
        }
#pragma unroll
        for (int q = 0; q < NB; ++q)
            if (k[q] >= 0) use(q, k[q], e[q]);
    }
}

// x of the tile's cells
template <typename S>
__device__ __forceinline__ void n_store(const NReg<S>& R, const NLevel& L, S* y)
{
    n_tile(R, L, [](int, bool, long long, int) {}, [&](int, long long k, int e) { y[k] = R.x[e]; });
}

// down leg of a coarse grid level
template <typename S>
__device__ __forceinline__ void n_down(const NSArgs& A, int l, unsigned char* smem,
                                       const NTab<S>& T)
{
    const NLevel& L = A.lev[l];
    for (int tile = blockIdx.x; tile < L.nt; tile += gridDim.x) {
        NReg<S> R;
        n_region<S>(R, L, tile, 4, smem, false);
        const S* B = (const S*)L.b;
        const S* FX = (const S*)L.fx;
        const S* FY = (const S*)L.fy;
        const S* IV = (const S*)L.inv;
        S b[NB], fx[NB], fy[NB], iv[NB];
        n_load(
            R, L,
            [&](int q, bool in, long long k, int, int) {
                b[q] = in ? B[k] : S(0);
                fx[q] = in ? FX[k] : S(0);
                fy[q] = in ? FY[k] : S(0);
                iv[q] = in ? IV[k] : S(0);
            },
            [&](int q, int e, bool, long long, int r, int c) {
                R.b[e] = b[q];
                R.fx[e] = fx[q];
                R.fy[e] = fy[q];
                R.inv[e] = iv[q];
                R.x[e] = n_red(R, L, r, c) ? -b[q] * iv[q] : S(0);
            });
        __syncthreads();
#pragma unroll 1
        for (int rad = 3; rad >= 1; --rad) n_half<S, false>(R, T, L, rad & 1, rad);
        n_restrict<S, false>(R, T, L, A.lev[l + 1]);
        n_store<S>(R, L, (S*)L.xa);
        __syncthreads();
    }
}

// up leg of a coarse grid level: the black cells' own values do not enter
// (the first half sweep overwrites them from the red ones), so only red
// cells are prolongated (all next to a seam)
template <typename S>
__device__ __forceinline__ void n_up(const NSArgs& A, int l, unsigned char* smem,
                                     const NTab<S>& T)
{
    const NLevel& L = A.lev[l];
    const NLevel& C = A.lev[l + 1];
    for (int tile = blockIdx.x; tile < L.nt; tile += gridDim.x) {
        NReg<S> R;
        n_region<S>(R, L, tile, 4, smem, false);
        const S* B = (const S*)L.b;
        const S* XA = (const S*)L.xa;
        const S* XC = (const S*)C.x;
        const S* FX = (const S*)L.fx;
        const S* FY = (const S*)L.fy;
        const S* IV = (const S*)L.inv;
        S b[NB], fx[NB], fy[NB], iv[NB], xa[NB], xc[NB];
        n_load(
            R, L,
            [&](int q, bool in, long long k, int J, int I) {
                const bool use = in && (L.seam || ((J + I) & 1) == 0);
                b[q] = in ? B[k] : S(0);
                fx[q] = in ? FX[k] : S(0);
                fy[q] = in ? FY[k] : S(0);
                iv[q] = in ? IV[k] : S(0);
                xa[q] = use ? XA[k] : S(0);
                xc[q] = use ? XC[C.off + (long long)(J >> 1) * C.pitch + (I >> 1)] : S(0);
            },
            [&](int q, int e, bool, long long, int, int) {
                R.b[e] = b[q];
                R.fx[e] = fx[q];
                R.fy[e] = fy[q];
                R.inv[e] = iv[q];
                R.x[e] = iv[q] != S(0) ? xa[q] + xc[q] : S(0);
            });
        __syncthreads();
#pragma unroll 1
        for (int rad = 3; rad >= 0; --rad) n_half<S, false>(R, T, L, rad & 1, rad);
        n_store<S>(R, L, (S*)L.x);
        __syncthreads();
    }
}

// phase A: with it > 0 the CG update of the previous iteration (s, p, x of
// the tile; r of the tile and its halo), the block's <r, r> and sum of x,
// then the down leg of level 0 on the new residual
template <typename S>
__device__ __forceinline__ void n_phase_a(const NSArgs& A, int it, double alpha, double beta,
                                          double (&tot)[2], unsigned char* smem,
                                          const NTab<S>& T)
{
    const NLevel& L = A.lev[0];
    const int par = it & 1;
    const double* r0 = A.r[it > 0 ? 1 - par : 0];
    const double* s0 = A.s[1 - par];
    double* r1 = A.r[par];
    double* s1 = A.s[par];
    const S* z = (const S*)A.z;
    for (int tile = blockIdx.x; tile < L.nt; tile += gridDim.x) {
        NReg<S> R;
        n_region<S>(R, L, tile, 4, smem, true);
        uint8_t code[NB];
        double rv[NB], sv[NB], wv[NB], xv[NB], pv[NB];
        S zv[NB];
        n_load(
            R, L,
            [&](int q, bool in, long long k, int, int) {
                code[q] = in ? L.code[k] : 0;
                rv[q] = in ? r0[k] : 0.0;
                wv[q] = in && it > 0 ? A.w[k] : 0.0;
                sv[q] = in && it > 1 ? s0[k] : 0.0;
            },
            [&](int q, int e, bool in, long long k, int r, int c) {
                double rn = rv[q];
                if (it > 0) {
                    const double sn = wv[q] + beta * sv[q];
                    rn -= alpha * sn;
                    if (in && r >= 4 && r < 4 + L.th && c >= 4 && c < 4 + L.tw &&
                        R.I0 - 4 + c < L.nxn) {
                        s1[k] = sn;
                        r1[k] = rn;
                        tot[0] += rn * rn;  // (0 at dry cells)
                    }
                }
                const S bi = conv<S>(rn) * T.inv[n_open(code[q])];
                R.code[e] = code[q];
                R.b[e] = bi;
                R.x[e] = n_red(R, L, r, c) ? -bi : S(0);
            });
        __syncthreads();
#pragma unroll 1
        for (int rad = 3; rad >= 1; --rad) n_half<S, true>(R, T, L, rad & 1, rad);
        n_restrict<S, true>(R, T, L, A.lev[1]);
        // xa, and p and x of the tile
        n_tile(
            R, L,
            [&](int q, bool in, long long k, int) {
                xv[q] = in && it > 0 ? A.x[k] : 0.0;
                pv[q] = in && it > 1 ? A.p[k] : 0.0;
                zv[q] = in && it > 0 ? z[k] : S(0);
            },
            [&](int q, long long k, int e) {
                ((S*)L.xa)[k] = R.x[e];
                if (it == 0) return;
                const double pn = conv<double>(zv[q]) + beta * pv[q];
                A.p[k] = pn;
                if (R.code[e]) {
                    const double xn = xv[q] + alpha * pn;
                    A.x[k] = xn;
                    tot[1] += xn;
                }
            });
        __syncthreads();
    }
}

// phase B: up leg of level 0 (z), w = A z in FP64, <r, z> and <z, w>
template <typename S>
__device__ __forceinline__ void n_phase_b(const NSArgs& A, int it, double (&tot)[2],
                                          unsigned char* smem, const NTab<S>& T)
{
    const NLevel& L = A.lev[0];
    const NLevel& C = A.lev[1];
    const double* rr = A.r[it & 1];
    const S* XA = (const S*)L.xa;
    const S* XC = (const S*)C.x;
    const double cx = A.cx, cy = A.cy;
    for (int tile = blockIdx.x; tile < L.nt; tile += gridDim.x) {
        NReg<S> R;
        n_region<S>(R, L, tile, NS_H, smem, true);
        uint8_t code[NB];
        double rv[NB];
        S xa[NB], xc[NB];
        n_load(
            R, L,
            [&](int q, bool in, long long k, int J, int I) {
                const bool use = in && (L.seam || ((J + I) & 1) == 0);
                code[q] = in ? L.code[k] : 0;
                rv[q] = in ? rr[k] : 0.0;
                xa[q] = use ? XA[k] : S(0);
                xc[q] = use ? XC[C.off + (long long)(J >> 1) * C.pitch + (I >> 1)] : S(0);
            },
            [&](int q, int e, bool, long long, int, int) {
                R.code[e] = code[q];
                R.b[e] = conv<S>(rv[q]) * T.inv[n_open(code[q])];
                R.x[e] = code[q] & 30 ? xa[q] + xc[q] : S(0);
            });
        __syncthreads();
#pragma unroll 1
        for (int rad = 4; rad >= 1; --rad) n_half<S, true>(R, T, L, 1 - (rad & 1), rad);
        n_tile(
            R, L, [&](int q, bool in, long long k, int) { rv[q] = in ? rr[k] : 0.0; },
            [&](int q, long long k, int e) {
                const uint8_t cd = R.code[e];
                const double zc = conv<double>(R.x[e]);
                // differences to the centre across open faces
                const double dw = cd & 2 ? conv<double>(R.x[e - 1]) - zc : 0.0;
                const double de = cd & 4 ? conv<double>(R.x[e + 1]) - zc : 0.0;
                const double ds = cd & 8 ? conv<double>(R.x[e - R.W]) - zc : 0.0;
                const double dn = cd & 16 ? conv<double>(R.x[e + R.W]) - zc : 0.0;
                const double wv = cx * (dw + de) + cy * (ds + dn);
                ((S*)A.z)[k] = R.x[e];
                A.w[k] = wv;
                tot[0] += rv[q] * zc;
                tot[1] += zc * wv;
            });
        __syncthreads();
    }
}

// cells of level 0, dealt to all threads of the grid by rows of 512 cells
template <typename F>
__device__ __forceinline__ void n_cells(const NLevel& L, F f)
{
    const int nseg = (L.nxn + PS_NT - 1) / PS_NT;
    for (int q = blockIdx.x; q < L.nyn * nseg; q += gridDim.x) {
        const int J = q / nseg, I = (q - J * nseg) * PS_NT + threadIdx.x;
        if (I < L.nxn) f(J, I, L.off + (long long)J * L.pitch + I);
    }
}

// Phases A and B when level 0 itself is the dense level (D: its x = z and
// its b in the cycle's precision, without the halo)
template <typename S>
__device__ __forceinline__ void n_dense_a(const NSArgs& A, int it, double alpha, double beta,
                                          double (&tot)[2])
{
    const NLevel& L = A.lev[0];
    n_cells(L, [&](int J, int I, long long k) {
        const int d = J * L.nxn + I;
        double rv = A.r[0][k];
        if (it > 0) {
            double sv = A.w[k], pv = conv<double>(((const S*)L.x)[d]);
            if (it > 1) {
                sv += beta * A.s[0][k];
                pv += beta * A.p[k];
            }
            rv -= alpha * sv;
            A.s[0][k] = sv;
            A.r[0][k] = rv;
            A.p[k] = pv;
            if (L.code[k]) {
                const double xn = A.x[k] + alpha * pv;
                A.x[k] = xn;
                tot[0] += rv * rv;
                tot[1] += xn;
            }
        }
        ((S*)L.b)[d] = conv<S>(rv);
    });
}

template <typename S>
__device__ __forceinline__ void n_dense_b(const NSArgs& A, double (&tot)[2])
{
    const NLevel& L = A.lev[0];
    const S* z = (const S*)L.x;
    n_cells(L, [&](int J, int I, long long k) {
        const int d = J * L.nxn + I;
        const uint8_t c = L.code[k];
        double wv = 0.0;
        if (c) {
            const double zc = conv<double>(z[d]);
            const int dw_ = I > 0 ? d - 1 : d + L.nxn - 1, de_ = I + 1 < L.nxn ? d + 1 : d - I;
            const double dw = c & 2 ? conv<double>(z[dw_]) - zc : 0.0;
            const double de = c & 4 ? conv<double>(z[de_]) - zc : 0.0;
            const double ds = c & 8 ? conv<double>(z[d - L.nxn]) - zc : 0.0;
            const double dn = c & 16 ? conv<double>(z[d + L.nxn]) - zc : 0.0;
            wv = A.cx * (dw + de) + A.cy * (ds + dn);
            tot[0] += A.r[0][k] * zc;
            tot[1] += zc * wv;
        }
        A.w[k] = wv;
    });
}

template <typename S>
__global__ void __launch_bounds__(PS_NT, 1) k_ns_solve(const __grid_constant__ NSArgs A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ NTab<S> T;
    if (threadIdx.x < 9) {
        const int k = threadIdx.x;
        T.inv[k] = conv<S>(A.inv[k]);
        T.cs[k] = conv<S>(A.cs[k]);
        T.cxi[k] = conv<S>(A.cx * A.inv[k]);
        T.cyi[k] = conv<S>(A.cy * A.inv[k]);
    }
    __shared__ struct {
        double mean, bb, goal, rr, xsum, rz, irz, d, alpha, beta;
        int done, status;
    } c;
    DevScalars* sc = (DevScalars*)A.sc;
    PSGrid g = ps_grid((PSBar*)A.bar, &A.eg->status, 0u);
    const NLevel& L = A.lev[0];
    const unsigned G = gridDim.x;
    // the block's rows of the dense level, kept in shared memory if they fit
    const int d0 = A.nd * blockIdx.x / G, d1 = A.nd * (blockIdx.x + 1) / G;
    const PSBox box = {A.nd, A.nd, 0, 1.0f / (float)A.nd};
    const S* mrows = (const S*)A.minv + (size_t)d0 * ps_pitch<S>(A.nd);
    if (A.mkeep) {
        ps_copy16(smem + A.mkeep, mrows, (size_t)(d1 - d0) * ps_pitch<S>(A.nd) * sizeof(S));
        mrows = (const S*)(smem + A.mkeep);
    }
    // totals: <r, z>, <z, w> | <r, r>, sum x | sum b | <b, b>, <r, r>, sum x
    double *pz = A.part, *pr = A.part + 2 * G, *pi = A.part + 4 * G, *pb = A.part + 5 * G;
    // b -= mean(b)
    double vb[1] = {0.0};
    n_cells(L, [&](int, int, long long k) { if (L.code[k]) vb[0] += A.b[k]; });
    ps_block_total<1>(vb, pi + blockIdx.x, G);
    if (!ps_sync(g)) return;
    ps_grid_total<1>(pi, [&](const double* t) { c.mean = t[0] / A.nfluid; });
    // r = b - A x
    double v[3] = {0.0, 0.0, 0.0};
    n_cells(L, [&](int J, int I, long long k) {
        const uint8_t cd = L.code[k];
        double rv = 0.0;
        if (cd) {
            const double bv = A.b[k] - c.mean, xc = A.x[k];
            const long long kw = I > 0 ? k - 1 : k + L.nxn - 1;
            const long long ke = I + 1 < L.nxn ? k + 1 : k - I;
            const double dw = cd & 2 ? A.x[kw] - xc : 0.0, de = cd & 4 ? A.x[ke] - xc : 0.0;
            const double ds = cd & 8 ? A.x[k - L.pitch] - xc : 0.0;
            const double dn = cd & 16 ? A.x[k + L.pitch] - xc : 0.0;
            rv = bv - (A.cx * (dw + de) + A.cy * (ds + dn));
            A.b[k] = bv;
            v[0] += bv * bv;
            v[1] += rv * rv;
            v[2] += xc;
        }
        A.r[0][k] = rv;
    });
    ps_block_total<3>(v, pb + blockIdx.x, G);
    if (!ps_sync(g)) return;
    ps_grid_total<3>(pb, [&](const double* t) {
        c.bb = t[0];
        c.rr = t[1];
        c.xsum = t[2];
        c.goal = sc->tol2 * t[0];
        c.done = t[0] == 0.0 || t[1] <= c.goal;
        c.status = 0;
        c.alpha = c.beta = c.irz = c.d = 0.0;
    });
    const int maxit = sc->maxit;
    int it = 0;
    // the decision after the update of iteration it: warps 1 and 2, while
    // warp 0 waits at the next barrier (the phase before it is lost when
    // the solve is over, but its totals cost no time)
    auto decide = [&] {
        const int w = threadIdx.x >> 5;
        if (it == 0 || w > 2) return;
        const double a = ps_total(pr + (w - 1) * G, G);
        if (threadIdx.x & 31) return;
        if (w == 2) {
            c.xsum = a;
            return;
        }
        c.rr = a;
        if (!(a == a)) c.status = ST_NONFINITE;
        else if (a > c.goal && it >= maxit) c.status = ST_PCG_MAXIT;
        c.done = c.status || a <= c.goal;
    };
    while (!c.done) {
        double t[2] = {0.0, 0.0};
        if (A.ng > 0) n_phase_a<S>(A, it, c.alpha, c.beta, t, smem, T);
        else n_dense_a<S>(A, it, c.alpha, c.beta, t);
        if (it > 0) ps_block_total<2>(t, pr + blockIdx.x, G);
        if (!ps_sync(g)) return;
        if (A.ng == 0 && it > 0) {
            // no level leg to hide the decision behind, and the phase that
            // would be lost is the whole solve: decide first
            if (threadIdx.x >= 32) decide();
            __syncthreads();
            if (c.done) break;
        }
        for (int l = 1; l < A.ng; ++l) {
            n_down<S>(A, l, smem, T);
            if (!(l == 1 ? ps_sync(g, decide) : ps_sync(g))) return;
            if (l == 1 && c.done) break;
        }
        if (c.done) break;
        const NLevel& D = A.lev[A.ng];
        ps_dense<S>(mrows, (const S*)D.b, (S*)D.x, A.nd, d0, d1, (S*)smem, box);
        if (!(A.ng == 1 ? ps_sync(g, decide) : ps_sync(g))) return;
        if (c.done) break;
        for (int l = A.ng - 1; l >= 1; --l) {
            n_up<S>(A, l, smem, T);
            if (!ps_sync(g)) return;
        }
        t[0] = t[1] = 0.0;
        if (A.ng > 0) n_phase_b<S>(A, it, t, smem, T);
        else n_dense_b<S>(A, t);
        ps_block_total<2>(t, pz + blockIdx.x, G);
        if (!ps_sync(g)) return;
        ps_grid_total<2>(pz, [&](const double* u) {
            // beta = rz / rz_old and <p, A p> = <z, w> - beta^2 <p, A p>_old,
            // alpha = rz / <p, A p>
            c.beta = u[0] * c.irz;
            c.d = u[1] - c.beta * c.beta * c.d;
            c.alpha = u[0] / c.d;
            c.rz = u[0];
        });
        if (threadIdx.x == 0) c.irz = 1.0 / c.rz;  // for the next beta
        ++it;
    }
    // zero-mean solution (its sum was formed with the last update); 0 for a zero
    // right-hand side, whatever x was on entry
    const double xm = c.xsum / A.nfluid;
    const bool zero = c.bb == 0.0;
    n_cells(L, [&](int, int, long long k) {
        if (L.code[k]) A.x[k] = zero ? 0.0 : A.x[k] - xm;
    });
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->bb = c.bb;
        sc->rr = c.rr;
        sc->iter = it;
        sc->converged = 1;
        sc->total_iters += it;
        A.eg->iters += it;
        if (c.status) A.eg->status |= c.status;
    }
}

__global__ void k_ns_setup(DevScalars* sc, double tol2, int maxit, PSBar* bar)
{
    sc->tol2 = tol2;
    sc->maxit = maxit;
    sc->converged = 0;
    sc->iter = 0;
    ps_reset(bar);
}

// ---- host ----------------------------------------------------------------------
int ns_record(NSolver& s, cudaStream_t st, int* launches)
{
    k_ns_setup<<<1, 1, 0, st>>>(s.sc, s.tol * s.tol, s.maxit, (PSBar*)s.a.bar);
    void* args[1] = {&s.a};
    const void* kern = s.prec == 0 ? (const void*)k_ns_solve<double>
                                   : (const void*)k_ns_solve<float>;
    int e = (int)cudaGetLastError();
    if (!e) e = ps_launch(kern, s.grid, s.smem, args, st);
    if (launches) *launches = 2;
    return e;
}

// Tiles of a level: of the partitions into even widths and heights that fit
// the shared memory, the one with the smallest estimate of the busiest
// block's time, (its tiles) x (a fixed cost + the FP64 or FP32 cycles of the
// cells its leg visits, the halo among them). Up to about 1300^2 cells that
// is one tile per block: its halo is small, and nothing is left over.
constexpr size_t NS_SMEM = 200 * 1024;
static void pick_tile(NLevel& L, int sms, int prec, int h, size_t cell_bytes)
{
    const double per = prec == 0 ? 2.5 : 0.5;  // cycles of a visited cell
    const int cap = L.seam ? NS_SEAM_T : 1 << 20;
    double best = 0.0;
    for (int ntx = 1; ntx <= (L.nxn + 7) / 8 || ntx == 1; ++ntx) {
        const int tw = ((L.nxn + ntx - 1) / ntx + 1) / 2 * 2;
        if (tw > cap || (L.nxn + tw - 1) / tw != ntx) continue;
        for (int nty = 1; nty <= (L.nyn + 7) / 8 || nty == 1; ++nty) {
            const int th = ((L.nyn + nty - 1) / nty + 1) / 2 * 2;
            if (th > cap || (L.nyn + th - 1) / th != nty) continue;
            const size_t n = (size_t)(tw + 2 * h) * (th + 2 * h);
            if (n * cell_bytes > NS_SMEM) continue;
            double cells = (double)n + (double)tw * th;
            for (int q = 0; q < 4; ++q) cells += 0.5 * (tw + 2 * q) * (th + 2 * q);
            const long long nt = (long long)ntx * nty;
            const double cost = (double)((nt + sms - 1) / sms) * (1500.0 + per * cells);
            if (best == 0.0 || cost < best) {
                best = cost;
                L.tw = tw;
                L.th = th;
                L.ntx = ntx;
                L.nt = (int)nt;
            }
        }
    }
}

// The dense level's inverse: of -A with one cell of every connected part
// grounded, the parts' constants projected out of it (its pseudo-inverse);
// dry cells and cells without couplings keep x = 0.
static int dense_inverse(const std::vector<double>& fx, const std::vector<double>& fy, int nyn,
                         int nxn, int per, double cx, double cy, int prec, void* out)
{
    const int n = nyn * nxn, bw = nxn, w1 = bw + 1;
    std::vector<double> h((size_t)n * w1, 0.0);  // h[i w1 + k] = H(i, i - k)
    std::vector<int> part(n);
    std::iota(part.begin(), part.end(), 0);
    auto root = [&](int k) {
        while (part[k] != k) k = part[k] = part[part[k]];
        return k;
    };
    auto link = [&](int a, int b, double c) {
        if (c == 0.0) return;
        h[(size_t)a * w1] += c;
        h[(size_t)b * w1] += c;
        h[(size_t)std::max(a, b) * w1 + std::abs(a - b)] -= c;
        part[root(a)] = root(b);
    };
    for (int J = 0; J < nyn; ++J)
        for (int I = 0; I < nxn; ++I) {
            const int k = J * nxn + I;
            if (I > 0) link(k, k - 1, fx[k]);
            else if (per && nxn > 1) link(k, k + nxn - 1, fx[k]);
            if (J > 0) link(k, k - nxn, fy[k]);
        }
    for (int k = 0; k < n; ++k) part[k] = root(k);
    std::vector<int> size(n, 0);
    for (int k = 0; k < n; ++k) size[part[k]] += 1;
    for (int k = 0; k < n; ++k) {
        if (size[part[k]] == 1) {
            h[(size_t)k * w1] = 1.0;
            part[k] = -1;
        } else if (part[k] == k) {
            h[(size_t)k * w1] += cx + cy;
        }
    }
    PSScratch scratch;
    const int rc = ps_invert(h, n, bw, part, -1.0, prec, out, scratch);
    if (rc) return rc;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 3;
}

// The FP32 form's dense level: not the inverse but the V-cycle on the levels
// from it on (2 sweeps per leg, (R,B)^k (B,R)^k on the first level of at most
// 8 cells in a direction), as the matrix of that linear map, column by column
// in FP64. The euler models' FP32 velocities round differently wherever the
// pressure moves by its tolerance, so this form keeps the cycle, and with it
// the CG iterates, of the level-by-level form it replaced: the velocities and
// the pressure stay the same to the last bits.
constexpr int NC_LMAX = 12;
struct NCoarse {
    int nl, ksweeps;
    int nyn[NC_LMAX], nxn[NC_LMAX], off[NC_LMAX], per;
};

__device__ __forceinline__ double nc_ax(const NCoarse& C, int l, const double* x,
                                        const double* fx, const double* fy, int J, int I,
                                        double& cs)
{
    const int nx = C.nxn[l], ny = C.nyn[l], o = C.off[l], k = o + J * nx + I;
    const double cw = fx[k], so = fy[k];
    const int ke = I + 1 < nx ? k + 1 : k - I;
    const double ce = I + 1 < nx || C.per ? fx[ke] : 0.0;
    const double cn = J + 1 < ny ? fy[k + nx] : 0.0;
    double v = -((cw + ce) + (so + cn)) * x[k];
    cs = (cw + ce) + (so + cn);
    if (cw != 0.0) v += cw * x[I > 0 ? k - 1 : k + nx - 1];
    if (ce != 0.0) v += ce * x[ke];
    if (so != 0.0) v += so * x[k - nx];
    if (cn != 0.0) v += cn * x[k + nx];
    return v;
}

__device__ __forceinline__ void nc_half(const NCoarse& C, int l, double* x, const double* b,
                                        const double* fx, const double* fy, int color)
{
    // (the colour's cells only: an FP64 instruction takes as long for half a warp)
    const int nx = C.nxn[l], wc = (nx + 1) / 2, n = wc * C.nyn[l], o = C.off[l];
    // On an x-periodic level of odd width the cells at both ends of a row are
    // neighbours of one colour: one thread forms both values before it writes
    // either, which is Jacobi across the seam as in n_half_seam.
    const bool seam = C.per && nx > 1 && nx % 2;
    auto value = [&](int J, int I) {
        const int k = o + J * nx + I;
        double cs;
        const double ax = nc_ax(C, l, x, fx, fy, J, I, cs);
        return cs > 0.0 ? x[k] + (ax - b[k]) / cs : x[k];
    };
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int J = i / wc, I = 2 * (i - J * wc) + ((J + color) & 1), k = o + J * nx + I;
        if (I >= nx || (seam && I == nx - 1)) continue;
        const double v = value(J, I);
        if (seam && I == 0) x[k + nx - 1] = value(J, nx - 1);
        x[k] = v;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256)
k_ns_coarse_map(const __grid_constant__ NCoarse C, const double* __restrict__ fx,
                const double* __restrict__ fy, float* __restrict__ out)
{
    extern __shared__ double sm[];
    const int nl = C.nl, tot = C.off[nl - 1] + C.nyn[nl - 1] * C.nxn[nl - 1];
    double *x = sm, *b = sm + tot;
    const int n = C.nyn[0] * C.nxn[0], col = blockIdx.x;
    for (int k = threadIdx.x; k < tot; k += blockDim.x) {
        x[k] = 0.0;
        b[k] = k == col ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int l = 0; l + 1 < nl; ++l) {
        for (int s = 0; s < 4; ++s) nc_half(C, l, x, b, fx, fy, s & 1);
        const int cx = C.nxn[l + 1];
        for (int k = threadIdx.x; k < cx * C.nyn[l + 1]; k += blockDim.x) {
            double v = 0.0, cs;
            for (int q = 0; q < 4; ++q) {
                const int J = 2 * (k / cx) + (q >> 1), I = 2 * (k % cx) + (q & 1);
                if (J < C.nyn[l] && I < C.nxn[l])
                    v += b[C.off[l] + J * C.nxn[l] + I] - nc_ax(C, l, x, fx, fy, J, I, cs);
            }
            b[C.off[l + 1] + k] = v;
        }
        __syncthreads();
    }
    for (int s = 0; s < 2 * C.ksweeps; ++s)
        for (int h = 0; h < 2; ++h)
            nc_half(C, nl - 1, x, b, fx, fy, s < C.ksweeps ? h : 1 - h);
    for (int l = nl - 2; l >= 0; --l) {
        const int nx = C.nxn[l], cx = C.nxn[l + 1];
        for (int k = threadIdx.x; k < nx * C.nyn[l]; k += blockDim.x)
            x[C.off[l] + k] += x[C.off[l + 1] + (k / nx / 2) * cx + k % nx / 2];
        __syncthreads();
        for (int s = 0; s < 4; ++s) nc_half(C, l, x, b, fx, fy, (s + 1) & 1);
    }
    // column col = row col (the cycle is symmetric)
    const int np = ps_pitch<float>(n);
    for (int k = threadIdx.x; k < np; k += blockDim.x)
        out[(size_t)col * np + k] = k < n ? (float)x[k] : 0.f;
}

static void coarsen(std::vector<double>& fx, std::vector<double>& fy, int& ny, int& nx, int per)
{
    const int cyn = (ny + 1) / 2, cxn = (nx + 1) / 2;
    std::vector<double> cfx((size_t)cyn * cxn, 0.0), cfy((size_t)cyn * cxn, 0.0);
    for (int J = 0; J < cyn; ++J)
        for (int I = 0; I < cxn; ++I) {
            double sx = 0.0, sy = 0.0;
            // fine x-faces at column 2I, y-faces at row 2J
            for (int q = 0; q < 2; ++q) {
                if (2 * J + q < ny) sx += fx[(size_t)(2 * J + q) * nx + 2 * I];
                if (2 * I + q < nx) sy += fy[(size_t)(2 * J) * nx + 2 * I + q];
            }
            cfx[(size_t)J * cxn + I] = 0.5 * sx;
            cfy[(size_t)J * cxn + I] = 0.5 * sy;
        }
    // one coarse column: the wrap face joins the cell to itself
    if (per && cxn == 1) std::fill(cfx.begin(), cfx.end(), 0.0);
    fx.swap(cfx);
    fy.swap(cfy);
    ny = cyn;
    nx = cxn;
}

static int coarse_map(std::vector<double> fx, std::vector<double> fy, int ny, int nx, int per,
                      float* out)
{
    NCoarse C = {};
    C.per = per;
    const int n = ny * nx;
    std::vector<double> ax, ay;
    for (;;) {
        C.nyn[C.nl] = ny;
        C.nxn[C.nl] = nx;
        C.off[C.nl] = (int)ax.size();
        C.nl += 1;
        ax.insert(ax.end(), fx.begin(), fx.end());
        ay.insert(ay.end(), fy.begin(), fy.end());
        if (!(ny > 8 && nx > 8 && (!per || nx % 2 == 0)) || C.nl == NC_LMAX) break;
        coarsen(fx, fy, ny, nx, per);
    }
    C.ksweeps = std::min(64, std::max(4, std::max(ny, nx)));
    double *dx = nullptr, *dy = nullptr;
    const size_t bytes = ax.size() * 8;
    int rc = 0;
    if (cudaMalloc(&dx, bytes) != cudaSuccess || cudaMalloc(&dy, bytes) != cudaSuccess ||
        cudaMemcpy(dx, ax.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dy, ay.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess)
        rc = 2;
    // (4096 cells and their coarser levels: 88 KB)
    if (!rc && (2 * bytes > 128 * 1024 ||
                cudaFuncSetAttribute(k_ns_coarse_map, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     128 * 1024) != cudaSuccess))
        rc = 3;
    if (!rc) {
        k_ns_coarse_map<<<n, 256, 2 * bytes>>>(C, dx, dy, out);
        if (cudaDeviceSynchronize() != cudaSuccess) rc = 3;
    }
    cudaFree(dx);
    cudaFree(dy);
    return rc;
}

int ns_build(NSolver& s, int nyn, int nxn, long long pitch, long long off, int per,
             const uint8_t* hmask, double* x, double* b, double cx, double cy, int prec)
{
    ns_free(s);
    s.prec = prec;
    const size_t es = prec == 0 ? 8 : 4;
    auto dal = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
        cudaMemset(p, 0, bytes);
        s.owned.push_back(p);
        return p;
    };
    // a device array of n host values in the cycle's precision
    auto up = [&](const std::vector<double>& v) -> void* {
        void* p = dal(v.size() * es);
        if (!p) return nullptr;
        std::vector<float> f;
        const void* src = v.data();
        if (prec) {
            f.assign(v.begin(), v.end());
            src = f.data();
        }
        return cudaMemcpy(p, src, v.size() * es, cudaMemcpyHostToDevice) == cudaSuccess ? p
                                                                                       : nullptr;
    };
    const int sms = ps_sms();
    if (sms < 1) return 3;
    std::vector<uint8_t> m((size_t)nyn * nxn);
    long long nf = 0;
    for (int J = 0; J < nyn; ++J)
        for (int I = 0; I < nxn; ++I) {
            m[(size_t)J * nxn + I] = hmask[off + (long long)J * pitch + I] ? 1 : 0;
            nf += m[(size_t)J * nxn + I];
        }
    if (nf == 0) return 6;
    std::vector<double> fx((size_t)nyn * nxn, 0.0), fy((size_t)nyn * nxn, 0.0);
    const size_t n0 = (size_t)(off + (long long)nyn * pitch);
    std::vector<uint8_t> code(n0, 0);
    for (int J = 0; J < nyn; ++J)
        for (int I = 0; I < nxn; ++I) {
            const size_t k = (size_t)J * nxn + I;
            if (!m[k]) continue;
            const bool w = I > 0 ? m[k - 1] : per && nxn > 1 && m[k + nxn - 1];
            const bool e = I + 1 < nxn ? m[k + 1] : per && nxn > 1 && m[k - I];
            const bool so = J > 0 && m[k - nxn];
            const bool no = J + 1 < nyn && m[k + nxn];
            if (w) fx[k] = cx;
            if (so) fy[k] = cy;
            code[off + (size_t)J * pitch + I] =
                (uint8_t)(1 | (w ? 2 : 0) | (e ? 4 : 0) | (so ? 8 : 0) | (no ? 16 : 0));
        }
    NSArgs& a = s.a;
    memset(&a, 0, sizeof(a));
    a.cx = cx;
    a.cy = cy;
    a.nfluid = (double)nf;
    for (int k = 0; k < 9; ++k) {
        a.cs[k] = (k / 3) * cx + (k % 3) * cy;
        a.inv[k] = a.cs[k] > 0.0 ? 1.0 / a.cs[k] : 0.0;
    }
    a.x = x;
    a.b = b;
    double* vec[6];
    for (auto& p : vec)
        if (!(p = (double*)dal(n0 * 8))) return 2;
    a.r[0] = vec[0];
    a.r[1] = vec[1];
    a.s[0] = vec[2];
    a.s[1] = vec[3];
    a.p = vec[4];
    a.w = vec[5];
    NLevel& L0 = a.lev[0];
    uint8_t* dc = (uint8_t*)dal(n0);
    if (!dc) return 2;
    if (cudaMemcpy(dc, code.data(), n0, cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    L0.code = dc;
    L0.pitch = pitch;
    L0.off = off;
    L0.nyn = nyn;
    L0.nxn = nxn;
    L0.per = per;
    L0.seam = per && (nxn % 2);
    // coarse levels (2x2 agglomerates) down to the dense one, which is level 0
    // when that is small enough: then the preconditioner is the inverse and
    // CG ends after one or two iterations (40^2: 1.6 instead of 9)
    int ny = nyn, nx = nxn, l = 0;
    bool dense = ps_band_ok((long long)nyn * nxn, nxn, 0);
    if (dense) {
        L0.x = dal((size_t)nyn * nxn * es);
        L0.b = dal((size_t)nyn * nxn * es);
        if (!L0.x || !L0.b) return 2;
    } else {
        a.z = dal(n0 * es);
        L0.xa = dal(n0 * es);
        if (!a.z || !L0.xa) return 2;
        pick_tile(L0, sms, prec, NS_H, 2 * es + 1);
    }
    while (!dense) {
        if (l + 1 >= NS_LMAX) return 3;
        coarsen(fx, fy, ny, nx, per);
        const int cyn = ny, cxn = nx;
        ++l;
        NLevel& C = a.lev[l];
        dense = ps_band_ok((long long)cyn * cxn, cxn, prec);
        C.nyn = cyn;
        C.nxn = cxn;
        C.pitch = dense ? cxn : (cxn + 31) / 32 * 32;
        C.off = 0;
        C.per = per;
        C.seam = per && (cxn % 2);
        const size_t n = (size_t)C.pitch * cyn;
        C.x = dal(n * es);
        C.b = dal(n * es);
        if (!C.x || !C.b) return 2;
        if (dense) continue;  // (the last)
        C.xa = dal(n * es);
        std::vector<double> hx(n, 0.0), hy(n, 0.0), hi(n, 0.0);
        for (int J = 0; J < cyn; ++J)
            for (int I = 0; I < cxn; ++I) {
                const size_t k = (size_t)J * cxn + I, g = (size_t)J * C.pitch + I;
                const double fe = I + 1 < cxn ? fx[k + 1] : (per ? fx[k - I] : 0.0);
                const double fn = J + 1 < cyn ? fy[k + cxn] : 0.0;
                const double cs = (fx[k] + fe) + (fy[k] + fn);
                hx[g] = fx[k];
                hy[g] = fy[k];
                hi[g] = cs > 0.0 ? 1.0 / cs : 0.0;
            }
        C.fx = up(hx);
        C.fy = up(hy);
        C.inv = up(hi);
        if (!C.xa || !C.fx || !C.fy || !C.inv) return 2;
        pick_tile(C, sms, prec, 4, 5 * es);
    }
    a.ng = l;
    a.nd = ny * nx;
    const int np = prec == 0 ? ps_pitch<double>(a.nd) : ps_pitch<float>(a.nd);
    void* minv = dal((size_t)a.nd * np * es);
    if (!minv) return 2;
    int rc = prec == 1 && a.ng > 0 ? coarse_map(fx, fy, ny, nx, per, (float*)minv)
                                   : dense_inverse(fx, fy, ny, nx, per, cx, cy, prec, minv);
    if (rc) return rc;
    a.minv = minv;
    // every SM also for small problems: the rows of the dense level are dealt
    // to all blocks, and a barrier of 152 blocks costs hardly more than one of 25
    // (1.36 us and 1.28, timed by barriers alone)
    s.grid = sms;
    const int rows = (a.nd + sms - 1) / sms;  // of a block, at most
    s.smem = (prec == 0 ? ps_dense_elems<double>(a.nd, rows) : ps_dense_elems<float>(a.nd, rows)) *
             es;
    for (int q = 0; q < a.ng; ++q) {
        const int h = q == 0 ? NS_H : 4;
        const size_t n = (size_t)(a.lev[q].tw + 2 * h) * (a.lev[q].th + 2 * h);
        s.smem = std::max(s.smem, q == 0 ? n * (2 * es + 1) : n * 5 * es);
    }
    s.smem = (s.smem + 15) / 16 * 16;
    if (s.smem + (size_t)rows * np * es <= NS_SMEM) {
        a.mkeep = (int)s.smem;
        s.smem += (size_t)rows * np * es;
    }
    const void* kern = prec == 0 ? (const void*)k_ns_solve<double> : (const void*)k_ns_solve<float>;
    // (the attribute is per kernel: never lowered below another solver's need)
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NS_SMEM) !=
        cudaSuccess)
        return 3;
    s.eg = (NGlobals*)dal(sizeof(NGlobals));
    s.sc = (DevScalars*)dal(sizeof(DevScalars));
    a.part = (double*)dal((size_t)8 * sms * sizeof(double));
    a.bar = dal(sizeof(PSBar));
    if (!s.eg || !s.sc || !a.part || !a.bar) return 2;
    a.eg = s.eg;
    a.sc = s.sc;
    return 0;
}

void ns_free(NSolver& s)
{
    for (void* p : s.owned) cudaFree(p);
    s.owned.clear();
    s.a = NSArgs{};
    s.eg = nullptr;
    s.sc = nullptr;
}

}  // namespace f2d
