// Persistent solve kernel of the masked vertex Poisson/Helmholtz operator
// (the reference factorises it with SuperLU: elliptic.py:71-87, 114-195) for
// a batch of one or many members: a whole multigrid-preconditioned CG solve
// of every member in one cooperative launch of one block per SM
// (persist.cuh), the CG iterations inside, its phases separated by grid
// barriers.
//
// Operator, hierarchy and cycle are mg.cu's: red-black Gauss-Seidel with nu
// sweeps per leg, bilinear prolongation and its transpose, coarse masks by
// injection, re-discretised coarse operators. The first level with few enough
// unknowns (nodes off the closed edges) is solved exactly with its dense inverse
// (a single model: up to 2048 unknowns, FP32 4096, level 0 itself if it is that
// small). S is the cycle's precision;
// the CG vectors, the operator product and the inner products are FP64 in
// both forms (FP32 form: the cycle's right-hand side is the FP64 residual
// rounded).
//
// CG in the form of Chronopoulos and Gear (J. Comput. Appl. Math. 25, 1989):
// w = A z and the two inner products <r, z>, <z, w> come from one pass, s =
// A p by recurrence. Phases of an iteration, a barrier after each:
//   A   update s, r, p, x (r on the tile and its halo, recomputed), <r, r>,
//       pre-smoothing, residual and restriction of level 0
//   D_l the same legs of the coarser grid levels;  the dense level
//   U_l the up legs
//   B   up leg of level 0 with z one node past the tile, w = A z, the two
//       inner products
// A leg works in shared memory on a tile and the halo its half sweeps reach
// over (5 nodes at nu = 2); nodes within s of the region's edge are inexact
// after half sweep s and only reach halo nodes. After the last black half
// sweep the black residuals are zero and the black values do not enter the
// up leg (its first half sweep overwrites them from the red ones), so only
// red residuals are formed and only red nodes are prolongated.
//
// What it replaced, FP64: one launch per level and leg on 54 x 70-node tiles,
// each bound by the FP64 pipe of the few SMs that had a tile (36 to 42 us a
// launch for 40 to 400 ns of work on the whole chip).
#include <algorithm>
#include <cstring>
#include <functional>
#include <queue>

#include "psolver.cuh"
#include "solver.cuh"

namespace f2d {

template <typename S>
struct PReg {
    S *x, *b;  // b: right-hand side / diagonal, then the residual
    uint8_t* m;
    int J0, I0, h, W, RH, tw, th;
    float rW;
    S cxi, cyi, dg;
};

template <typename S>
__device__ __forceinline__ PReg<S> p_region(const PTile& t, int h, unsigned char* smem)
{
    PReg<S> R;
    R.J0 = t.J0;
    R.I0 = t.I0;
    R.tw = t.tw;
    R.th = t.th;
    R.h = h;
    R.W = t.tw + 2 * h;
    R.RH = t.th + 2 * h;
    R.rW = 1.0f / (float)R.W;
    const int n = R.W * R.RH;
    R.x = (S*)smem;
    R.b = R.x + n;
    R.m = (uint8_t*)(R.b + n);
    R.cxi = conv<S>(t.cxi);
    R.cyi = conv<S>(t.cyi);
    R.dg = conv<S>(t.dg);
    return R;
}

__device__ __forceinline__ bool p_node(const PTile& t, int J, int& I)
{
    if (J < 0 || J >= t.nyn) return false;
    if (t.per) {
        while (I < 0) I += t.nxn;
        while (I >= t.nxn) I -= t.nxn;
        return true;
    }
    return I >= 0 && I < t.nxn;
}

// Gauss-Seidel value of region node e (non-fluid nodes hold x = 0)
template <typename S>
__device__ __forceinline__ S p_gs(const PReg<S>& R, int e)
{
    return fma(-R.cxi, R.x[e - 1] + R.x[e + 1],
               fma(-R.cyi, R.x[e - R.W] + R.x[e + R.W], R.b[e]));
}

// half sweep of a colour over the nodes within rad of the tile
template <typename S>
__device__ __forceinline__ void p_half(const PReg<S>& R, int color, int rad)
{
    const int o = R.h - rad, nr = R.th + 2 * rad, wc = R.tw / 2 + rad;
    const float rw = 1.0f / (float)wc;
    for (int k = threadIdx.x; k < nr * wc; k += PS_NT) {
        const int a = fdiv(k, rw), r = o + a;
        // J0 and I0 are even: the colour of region node (r, c) is r + c
        const int c = o + 2 * (k - a * wc) + ((r + o + color) & 1);
        const int e = r * R.W + c;
        if (R.m[e]) R.x[e] = p_gs(R, e);
    }
    __syncthreads();
}

constexpr int PB = 2;  // nodes per thread and batch

// The region's nodes in batches of PB per thread: load(q, in, k, J, I) for the
// batch (its loads in flight together), then use(q, e, in, k, r, c)
template <typename S, typename FL, typename FU>
__device__ __forceinline__ void p_load(const PReg<S>& R, const PTile& t, FL load, FU use)
{
    const int n = R.W * R.RH;
    for (int e0 = threadIdx.x; e0 < n; e0 += PB * PS_NT) {
        int rc[PB];
        long long k[PB];
#pragma unroll
        for (int q = 0; q < PB; ++q) {
            const int e = e0 + q * PS_NT;
            const int r = fdiv(e, R.rW), c = e - r * R.W;
            int I = R.I0 - R.h + c;
            const int J = R.J0 - R.h + r;
            const bool in = e < n && p_node(t, J, I);
            rc[q] = (r << 16) | c;
            k[q] = in ? t.off + (long long)J * t.pitch + I : -1;
            load(q, in, k[q], J, I);
        }
#pragma unroll
        for (int q = 0; q < PB; ++q) {
            const int e = e0 + q * PS_NT;
            if (e < n) use(q, e, k[q] >= 0, k[q], rc[q] >> 16, rc[q] & 0xffff);
        }
    }
}

// the tile's nodes of the level, in batches: load(q, in, k), use(q, k, e)
template <typename S, typename FL, typename FU>
__device__ __forceinline__ void p_tile(const PReg<S>& R, const PTile& t, FL load, FU use)
{
    const int n = R.tw * R.th;
    const float rw = 1.0f / (float)R.tw;
    for (int e0 = threadIdx.x; e0 < n; e0 += PB * PS_NT) {
        int e[PB];
        long long k[PB];
#pragma unroll
        for (int q = 0; q < PB; ++q) {
            const int i = e0 + q * PS_NT;
            const int a = fdiv(i, rw), c = i - a * R.tw;
            const int J = R.J0 + a, I = R.I0 + c;
            const bool in = i < n && J < t.nyn && I < t.nxn;
            k[q] = in ? t.off + (long long)J * t.pitch + I : -1;
            e[q] = (R.h + a) * R.W + R.h + c;
            load(q, in, k[q]);
        }
#pragma unroll
        for (int q = 0; q < PB; ++q)
            if (k[q] >= 0) use(q, k[q], e[q]);
    }
}

// From the region with b and the red x = b / diagonal: the rest of the
// pre-smoothing, the red residuals, their restriction to the coarse nodes
// whose centre lies in the tile (weight 1 at the centre, 1/4 at the corners).
template <typename S>
__device__ __forceinline__ void p_down_leg(const PReg<S>& R, const PTile& t, int nu)
{
#pragma unroll 1
    for (int q = 1; q < 2 * nu; ++q) p_half(R, q & 1, 2 * nu + 1 - q);
    {
        // residual / diagonal = Gauss-Seidel value - x of the red nodes within
        // 1 of the tile, into b
        const int o = R.h - 1, nr = R.th + 2, wc = R.tw / 2 + 1;
        const float rw = 1.0f / (float)wc;
        for (int k = threadIdx.x; k < nr * wc; k += PS_NT) {
            const int a = fdiv(k, rw), r = o + a;
            const int e = r * R.W + o + 2 * (k - a * wc) + ((r + o) & 1);
            R.b[e] = R.m[e] ? p_gs(R, e) - R.x[e] : S(0);
        }
        __syncthreads();
    }
    const int wc = R.tw / 2, nc = wc * (R.th / 2);
    const float rw = 1.0f / (float)wc;
    for (int k = threadIdx.x; k < nc; k += PS_NT) {
        const int a = fdiv(k, rw), c = k - a * wc;
        const int J = R.J0 / 2 + a, I = R.I0 / 2 + c;
        if (J >= t.cyn || I >= t.cxn) continue;
        const int e = (R.h + 2 * a) * R.W + R.h + 2 * c;
        S v = S(0);
        if (t.cm[t.cmoff + (long long)J * t.cmpitch + I])
            v = R.dg * fma(S(0.25), (R.b[e - R.W - 1] + R.b[e - R.W + 1]) +
                                        (R.b[e + R.W - 1] + R.b[e + R.W + 1]),
                           R.b[e]);
        ((S*)t.cb)[t.coff + (long long)J * t.cpitch + I] = v;
    }
}

// P (coarse x) at the red node (J, I) is the coarse node v[0], or (odd rows)
// the mean of the four v. use: whether to load at all. (The level has no fluid
// node on a closed edge: those rows and columns of the coarse level are 0.)
template <typename S>
__device__ __forceinline__ void p_coarse(const PTile& t, bool use, int J, int I, S (&v)[4])
{
    const int cj = J >> 1, ci = I >> 1;
    const S* xc = (const S*)t.cx_ + t.coff + (long long)cj * t.cpitch;
    const bool odd = use && (J & 1), up = odd && cj + 1 < t.cyn;
    const int c1 = ci + 1 < t.cxn ? ci + 1 : (t.per ? 0 : -1);
    v[0] = use ? xc[ci] : S(0);
    v[1] = odd && c1 >= 0 ? xc[c1] : S(0);
    v[2] = up ? xc[t.cpitch + ci] : S(0);
    v[3] = up && c1 >= 0 ? xc[t.cpitch + c1] : S(0);
}

// x = xa + P (coarse x) at the region's red nodes, 0 at its black ones. FP64:
// the nodes of even rows of the level and those of odd rows are dealt to
// different warps, so only the latter average and no lane idles on black
// nodes (in the region's own order a warp spent five FP64 instructions on
// every pair of rows, a sixth of phase B at 1024^2). FP32, where the indexing
// costs more than the arithmetic: in the region's own order (p_load's use).
template <typename S>
__device__ __forceinline__ void p_prolong(const PReg<S>& R, const PTile& t)
{
    const S* XA = (const S*)t.xa;
    const int wc = R.W / 2, n2 = wc * (R.RH / 2);
    const float rw = 1.0f / (float)wc;
    for (int i = threadIdx.x; i < 2 * n2; i += PS_NT) {
        const bool odd = i >= n2;  // odd row of the level
        const int a = fdiv(odd ? i - n2 : i, rw);
        const int r = 2 * a + ((R.h & 1) != (int)odd);
        const int c = 2 * ((odd ? i - n2 : i) - a * wc) + (r & 1);
        const int J = R.J0 - R.h + r, e = r * R.W + c;
        int I = R.I0 - R.h + c;
        S x = S(0);
        if (p_node(t, J, I)) {
            const long long k = t.off + (long long)J * t.pitch + I;
            const S xa = XA[k];
            S v[4];
            p_coarse<S>(t, true, J, I, v);
            const S pc = odd ? S(0.25) * ((v[0] + v[1]) + (v[2] + v[3])) : v[0];
            if (t.m[k]) x = xa + pc;
        }
        R.x[e] = x;
        R.x[r * R.W + (c ^ 1)] = S(0);
    }
}

template <typename S>
__device__ __forceinline__ void p_down(const PTile& t, int nu, unsigned char* smem)
{
    const PReg<S> R = p_region<S>(t, 2 * nu + 1, smem);
    const S* B = (const S*)t.b;
    const S id = conv<S>(t.id);
    S b[PB];
    uint8_t m[PB];
    p_load(
        R, t,
        [&](int q, bool in, long long k, int, int) {
            m[q] = in ? t.m[k] : 0;
            b[q] = in ? B[k] : S(0);
        },
        [&](int q, int e, bool, long long, int r, int c) {
            const S bi = m[q] ? b[q] * id : S(0);
            R.m[e] = m[q];
            R.b[e] = bi;
            R.x[e] = (r + c) & 1 ? S(0) : bi;
        });
    __syncthreads();
    p_down_leg(R, t, nu);
    S* XA = (S*)t.xa;
    p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int e) { XA[k] = R.x[e]; });
    __syncthreads();
}

template <typename S>
__device__ __forceinline__ void p_up(const PTile& t, int nu, unsigned char* smem)
{
    const PReg<S> R = p_region<S>(t, 2 * nu, smem);
    const S* B = (const S*)t.b;
    const S id = conv<S>(t.id);
    S b[PB];
    uint8_t m[PB];
    const S* XA = (const S*)t.xa;
    S xr[PB], cv[PB][4];
    int oj[PB];
    p_load(
        R, t,
        [&](int q, bool in, long long k, int J, int I) {
            m[q] = in ? t.m[k] : 0;
            if constexpr (sizeof(S) == 4) {
                const bool red = in && ((J + I) & 1) == 0;
                xr[q] = red ? XA[k] : S(0);
                p_coarse<S>(t, red, J, I, cv[q]);
                oj[q] = J & 1;
            }
            b[q] = in ? B[k] : S(0);
        },
        [&](int q, int e, bool, long long, int, int) {
            R.m[e] = m[q];
            R.b[e] = m[q] ? b[q] * id : S(0);
            if constexpr (sizeof(S) == 4)
                R.x[e] = m[q] ? xr[q] + (oj[q] ? S(0.25) * ((cv[q][0] + cv[q][1]) +
                                                            (cv[q][2] + cv[q][3]))
                                               : cv[q][0])
                              : S(0);
        });
    if constexpr (sizeof(S) == 8) p_prolong(R, t);
    __syncthreads();
#pragma unroll 1
    for (int q = 1; q <= 2 * nu; ++q) p_half(R, q & 1, 2 * nu - q);
    S* X = (S*)t.x;
    p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int e) { X[k] = R.x[e]; });
    __syncthreads();
}

// phase A of a level-0 tile (it > 0: with the CG update of the previous
// iteration): tot = <r, r>
template <typename S>
__device__ __forceinline__ void p_phase_a(const PSArgs& A, const PTile& t, int it, double alpha,
                                          double beta, double (&tot)[1], unsigned char* smem)
{
    const int nu = A.nu, h = 2 * nu + 1, par = it & 1;
    const PReg<S> R = p_region<S>(t, h, smem);
    const double* r0 = A.r[it > 0 ? 1 - par : 0];
    const double* s0 = A.s[1 - par];
    double* r1 = A.r[par];
    double* s1 = A.s[par];
    const S* Z = (const S*)t.x;
    S* B32 = (S*)t.b;  // the FP32 form's copy of r for phase B
    const S id = conv<S>(t.id);
    uint8_t m[PB];
    double rv[PB], sv[PB], wv[PB], xv[PB], pv[PB];
    S zv[PB];
    p_load(
        R, t,
        [&](int q, bool in, long long k, int, int) {
            m[q] = in ? t.m[k] : 0;
            rv[q] = in ? r0[k] : 0.0;
            wv[q] = in && it > 0 ? A.w[k] : 0.0;
            sv[q] = in && it > 1 ? s0[k] : 0.0;
        },
        [&](int q, int e, bool in, long long k, int r, int c) {
            double rn = rv[q];
            const bool own = in && r >= h && r < h + R.th && c >= h && c < h + R.tw &&
                             R.I0 - h + c < t.nxn;
            if (it > 0) {
                const double sn = wv[q] + beta * sv[q];
                rn -= alpha * sn;
                if (own) {
                    s1[k] = sn;
                    r1[k] = rn;
                    tot[0] += rn * rn;  // (0 at non-fluid nodes)
                }
            }
            const S rs = m[q] ? conv<S>(rn) : S(0);
            if constexpr (sizeof(S) == 4)
                if (own) B32[k] = rs;
            const S bi = rs * id;
            R.m[e] = m[q];
            R.b[e] = bi;
            R.x[e] = (r + c) & 1 ? S(0) : bi;
        });
    __syncthreads();
    p_down_leg(R, t, nu);
    S* XA = (S*)t.xa;
    p_tile(
        R, t,
        [&](int q, bool in, long long k) {
            xv[q] = in && it > 0 ? A.x[k] : 0.0;
            pv[q] = in && it > 1 ? A.p[k] : 0.0;
            zv[q] = in && it > 0 ? Z[k] : S(0);
        },
        [&](int q, long long k, int e) {
            XA[k] = R.x[e];
            if (it == 0) return;
            const double pn = conv<double>(zv[q]) + beta * pv[q];
            A.p[k] = pn;
            if (R.m[e]) A.x[k] = xv[q] + alpha * pn;
        });
    __syncthreads();
}

// phase B of a level-0 tile: tot = <r, z>, <z, A z>
template <typename S>
__device__ __forceinline__ void p_phase_b(const PSArgs& A, const PTile& t, int it,
                                          double (&tot)[2], unsigned char* smem)
{
    const int nu = A.nu, h = 2 * nu + 1;
    const PReg<S> R = p_region<S>(t, h, smem);
    const double* rr = A.r[it & 1];
    // the cycle's right-hand side: r, or the FP32 copy of it
    const S* bb = sizeof(S) == 8 ? (const S*)rr : (const S*)t.b;
    const S id = conv<S>(t.id);
    uint8_t m[PB];
    double rv[PB];
    S bv[PB];
    const S* XA = (const S*)t.xa;
    S xr[PB], cv[PB][4];
    int oj[PB];
    p_load(
        R, t,
        [&](int q, bool in, long long k, int J, int I) {
            m[q] = in ? t.m[k] : 0;
            if constexpr (sizeof(S) == 4) {
                const bool red = in && ((J + I) & 1) == 0;
                xr[q] = red ? XA[k] : S(0);
                p_coarse<S>(t, red, J, I, cv[q]);
                oj[q] = J & 1;
            }
            bv[q] = in ? bb[k] : S(0);
        },
        [&](int q, int e, bool, long long, int, int) {
            R.m[e] = m[q];
            R.b[e] = m[q] ? bv[q] * id : S(0);
            if constexpr (sizeof(S) == 4)
                R.x[e] = m[q] ? xr[q] + (oj[q] ? S(0.25) * ((cv[q][0] + cv[q][1]) +
                                                            (cv[q][2] + cv[q][3]))
                                               : cv[q][0])
                              : S(0);
        });
    if constexpr (sizeof(S) == 8) p_prolong(R, t);
    __syncthreads();
#pragma unroll 1
    for (int q = 1; q <= 2 * nu; ++q) p_half(R, q & 1, h - q);
    S* Z = (S*)t.x;
    const double cx = t.cx, cy = t.cy, md = t.md, dg = t.dg;
    p_tile(
        R, t, [&](int q, bool in, long long k) { rv[q] = in ? rr[k] : 0.0; },
        [&](int q, long long k, int e) {
            const double c = conv<double>(R.x[e]);
            double wv = 0.0;
            if (R.m[e]) {
                const double w = conv<double>(R.x[e - 1]), ea = conv<double>(R.x[e + 1]);
                const double so = conv<double>(R.x[e - R.W]), no = conv<double>(R.x[e + R.W]);
                if constexpr (sizeof(S) == 4) {
                    // sums of two floats are exact in FP64; the rest rounds
                    // at 1e-16 |z|, 1e-11 of w and less than z's own rounding
                    wv = cx * (w + ea) + (cy * (so + no) + dg * c);
                } else {
                    // differences to the centre (apply_diff): the same
                    // operator, but far less cancellation for smooth z
                    wv = (cx * ((w - c) + (ea - c)) + cy * ((so - c) + (no - c))) - md * c;
                }
                tot[0] += rv[q] * c;
                tot[1] += c * wv;
            }
            Z[k] = R.x[e];
            A.w[k] = wv;
        });
    __syncthreads();
}

// Level 0 as the dense level (one member): phases A and B without smoothing;
// z and the cycle's b in the compact layout of the dense level
template <typename S>
__device__ __forceinline__ void p_dense_a(const PSArgs& A, const PTile& t, const PDense& D, int it,
                                          double alpha, double beta, double (&tot)[1],
                                          unsigned char* smem)
{
    const PReg<S> R = p_region<S>(t, 0, smem);
    p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int e) {
        const int a = fdiv(e, R.rW);
        const int d = (t.J0 + a) * t.nxn + t.I0 + e - a * R.W;
        double rv = A.r[0][k];
        if (it > 0) {
            double sv = A.w[k], pv = conv<double>(((const S*)D.x)[d]);
            if (it > 1) {
                sv += beta * A.s[0][k];
                pv += beta * A.p[k];
            }
            rv -= alpha * sv;
            A.s[0][k] = sv;
            A.r[0][k] = rv;
            A.p[k] = pv;
            tot[0] += rv * rv;
            if (t.m[k]) A.x[k] += alpha * pv;
        }
        ((S*)D.b)[d] = conv<S>(rv);
    });
}

template <typename S>
__device__ __forceinline__ void p_dense_b(const PSArgs& A, const PTile& t, const PDense& D,
                                          double (&tot)[2], unsigned char* smem)
{
    const PReg<S> R = p_region<S>(t, 0, smem);
    const S* z = (const S*)D.x;
    p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int e) {
        const int a = fdiv(e, R.rW), J = t.J0 + a, I = t.I0 + e - a * R.W;
        const int d = J * t.nxn + I;
        double wv = 0.0;
        if (t.m[k]) {
            const int w = I > 0 ? d - 1 : t.per ? d + t.nxn - 1 : -1;
            const int ea = I + 1 < t.nxn ? d + 1 : t.per ? d - I : -1;
            const double c = conv<double>(z[d]);
            // (non-fluid nodes hold z = 0)
            const double zw = w >= 0 ? conv<double>(z[w]) : 0.0;
            const double ze = ea >= 0 ? conv<double>(z[ea]) : 0.0;
            const double zs = J > 0 ? conv<double>(z[d - t.nxn]) : 0.0;
            const double zn = J + 1 < t.nyn ? conv<double>(z[d + t.nxn]) : 0.0;
            wv = (t.cx * ((zw - c) + (ze - c)) + t.cy * ((zs - c) + (zn - c))) - t.md * c;
            tot[0] += A.r[0][k] * c;
            tot[1] += c * wv;
        }
        A.w[k] = wv;
    });
}

// The dense level of every member: the rows of all members dealt to the blocks.
// A block finds the members that its rows belong to once per solve and keeps
// the first of them in shared memory; a walk over all members' records every
// iteration, a load each, cost the 24-member ensemble 2 % of its step (2.97 ->
// 2.91 ms).
constexpr int PS_SEGS = 8;
struct PSegs {
    PDense D[PS_SEGS];
    int a[PS_SEGS], b[PS_SEGS];  // the block's rows a .. b - 1 of the member
    int n, first;
};

__device__ __forceinline__ bool p_rows(const PSArgs& A, const PDense& D, int& a, int& b)
{
    const int r0 = (int)((long long)A.nrows * blockIdx.x / gridDim.x);
    const int r1 = (int)((long long)A.nrows * (blockIdx.x + 1) / gridDim.x);
    a = max(r0 - D.row0, 0);
    b = min(r1 - D.row0, D.n);
    return a < b;
}

// (all threads; ends with a barrier)
__device__ __forceinline__ void p_find_rows(const PSArgs& A, PSegs& s)
{
    if (threadIdx.x == 0) {
        s.n = 0;
        s.first = A.nmem;
    }
    __syncthreads();
    int a, b;
    for (int m = threadIdx.x; m < A.nmem; m += PS_NT)
        if (p_rows(A, A.dense[m], a, b)) {
            atomicMin(&s.first, m);
            atomicAdd(&s.n, 1);
        }
    __syncthreads();
    if (threadIdx.x < min(s.n, PS_SEGS)) {  // (they follow one another)
        const PDense D = A.dense[s.first + threadIdx.x];
        p_rows(A, D, a, b);
        s.D[threadIdx.x] = D;
        s.a[threadIdx.x] = a;
        s.b[threadIdx.x] = b;
    }
    __syncthreads();
}

// f(D, a, b) for the block's rows of each member
template <typename F>
__device__ __forceinline__ void p_dense_rows(const PSArgs& A, const PSegs& s, F f)
{
    for (int i = 0; i < s.n; ++i) {
        if (i < PS_SEGS) {
            f(s.D[i], s.a[i], s.b[i]);
        } else {
            const PDense D = A.dense[s.first + i];
            int a, b;
            p_rows(A, D, a, b);
            f(D, a, b);
        }
    }
}

template <typename S>
__device__ __forceinline__ void p_dense(const PSArgs& A, const PSegs& segs, unsigned char* smem)
{
    const S* kept = (const S*)(smem + A.mkeep);
    p_dense_rows(A, segs, [&](const PDense& D, int a, int b) {
        const size_t np = ps_pitch<S>(D.n);
        ps_dense<S>(A.mkeep ? kept : (const S*)D.minv + a * np, (const S*)D.b, (S*)D.x, D.n, a, b,
                    (S*)smem, D.box);
        kept += (b - a) * np;
        __syncthreads();
    });
}

// r = b - A x of a tile; tot = <b, b>, <r, r>. CHECK: r is not stored, tot[0] =
// <x, x>
template <bool CHECK>
__device__ __forceinline__ void p_init(const PSArgs& A, const PTile& t, double (&tot)[2],
                                       unsigned char* smem)
{
    const PReg<double> R = p_region<double>(t, 0, smem);
    p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int e) {
        const int a = fdiv(e, R.rW), J = t.J0 + a, I = t.I0 + e - a * R.W;
        double rv = 0.0;
        if (t.m[k]) {
            const long long kw = I > 0 ? k - 1 : t.per ? k + t.nxn - 1 : -1;
            const long long ke = I + 1 < t.nxn ? k + 1 : t.per ? k - I : -1;
            const bool s = J > 0 && t.m[k - t.pitch], n = J + 1 < t.nyn && t.m[k + t.pitch];
            const double c = A.x[k], b = A.b[k];
            const double xw = kw >= 0 && t.m[kw] ? A.x[kw] : 0.0;
            const double xe = ke >= 0 && t.m[ke] ? A.x[ke] : 0.0;
            const double xs = s ? A.x[k - t.pitch] : 0.0, xn = n ? A.x[k + t.pitch] : 0.0;
            rv = b - ((t.cx * ((xw - c) + (xe - c)) + t.cy * ((xs - c) + (xn - c))) - t.md * c);
            tot[0] += CHECK ? c * c : b * b;
            tot[1] += rv * rv;
        }
        if constexpr (!CHECK) A.r[0][k] = rv;
    });
}

// State of a level-0 tile's member, kept by every block that has one of its
// tiles (a single member: one slot in every block), from the same totals in
// the same order: the same bits.
struct PSlot {
    double alpha, beta, d, rz, irz, goal, bb, rr;
    double checked;  // <r, r> of the last true residual, 0: none yet
    double floor;    // (8 eps diagonal)^2
    int conv, zero, status;
    int far;         // the start was worse than 0: <r, r> above <b, b>
    int verify;      // the recurrence has ended, the true residual is to be formed
    int member, n0, nn, owner;  // owner: this block writes the member's state
};

template <typename S>
__global__ void __launch_bounds__(PS_NT, 1) k_ps_solve(const __grid_constant__ PSArgs A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ PTile rec[PS_RECS];
    __shared__ PSlot slot[PS_SLOTS];
    __shared__ int rconv[PS_RECS];
    __shared__ PSegs segs;
    __shared__ int lev0[PS_LMAX + 1];
    const int nl = A.ng + 1;
    if (threadIdx.x < nl) lev0[threadIdx.x] = A.rec0[blockIdx.x * nl + threadIdx.x];
    __syncthreads();
    const int base = lev0[0], nrec = lev0[A.ng] - base;
    {
        constexpr int W = sizeof(PTile) / 16;
        const int4* src = (const int4*)(A.recs + base);
        for (int k = threadIdx.x; k < nrec * W; k += PS_NT) ((int4*)rec)[k] = src[k];
        for (int k = threadIdx.x; k < nrec; k += PS_NT) rconv[k] = 0;
    }
    p_find_rows(A, segs);
    if (A.mkeep) {
        unsigned char* kept = smem + A.mkeep;
        p_dense_rows(A, segs, [&](const PDense& D, int a, int b) {
            const size_t np = ps_pitch<S>(D.n) * sizeof(S), bytes = (b - a) * np;
            ps_copy16(kept, (const unsigned char*)D.minv + a * np, bytes);
            kept += bytes;
        });
    }
    __syncthreads();
    const int ns = lev0[1] - base;  // level-0 tiles of the block
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool single = A.nmem == 1;
    const int nt = A.ntiles;
    // totals per tile: <r, z>, <z, w> | <r, r> | <b, b>, <r, r>
    double *pz = A.part, *pr = A.part + 2 * nt, *pb = A.part + 3 * nt;
    PSGrid g = ps_grid(A.bar, A.status, 0u);
    const double tol2 = A.scs[0].tol2;
    const int maxit = A.scs[0].maxit;
    // r = b - A x, <b, b>, <r, r>
    for (int i = 0; i < ns; ++i) {
        double v[2] = {0.0, 0.0};
        p_init<false>(A, rec[i], v, smem);
        ps_block_total<2>(v, pb + rec[i].tile, nt);
    }
    const int nslot = single ? 1 : ns;
    if (!ps_sync(g)) return;
    for (int i = w; i < nslot; i += PS_NT / 32) {
        const int n0 = single ? 0 : rec[i].n0, nn = single ? nt : rec[i].nn;
        double bb, rr;
        ps_total2(pb + n0, pb + nt + n0, nn, bb, rr);
        if (lane) continue;
        PSlot& c = slot[i];
        c.member = single ? 0 : rec[i].member;
        c.n0 = n0;
        c.nn = nn;
        c.owner = single ? blockIdx.x == 0 : rec[i].tile == n0;
        c.bb = bb;
        c.rr = rr;
        c.goal = tol2 * bb;
        c.alpha = c.beta = c.d = c.rz = c.irz = 0.0;
        c.zero = bb == 0.0;
        c.conv = c.zero || rr <= c.goal;
        c.status = 0;
        c.far = rr > bb;
        c.verify = 0;
        c.checked = 0.0;
        // (one member: also in the blocks without a level-0 tile)
        const double e8 = 8.0 * 2.220446049250313e-16 * (single ? A.dg : rec[i].dg);
        c.floor = e8 * e8;
        if (c.owner && !single) {
            A.conv[c.member] = c.conv;
            if (!c.conv) atomicAdd(A.active, 1);
            if (c.far) atomicAdd(A.active + 1, 1);
        }
    }
    __syncthreads();
    for (int i = 0; i < ns; ++i)  // a zero right-hand side: x = 0
        if (slot[single ? 0 : i].zero) {
            const PTile& t = rec[i];
            const PReg<double> R = p_region<double>(t, 0, smem);
            p_tile(R, t, [](int, bool, long long) {}, [&](int, long long k, int) {
                if (t.m[k]) A.x[k] = 0.0;
            });
        }
    if (!ps_sync(g)) return;
    int it = 0, before = 0;  // iterations since and before the last start
    // The decision after the update of iteration `it`, by the idle warps of
    // the next barrier: the tiles' <r, r> are complete, the phase before that
    // barrier is lost when a solve is over, but the totals cost no time.
    auto decide = [&] {
        if (it == 0) return;
        for (int i = w - 1; i < nslot; i += PS_NT / 32 - 1) {
            PSlot& c = slot[i];
            if (c.conv) continue;
            const double rr = ps_total(pr + c.n0, c.nn);
            if (lane) continue;
            c.rr = rr;
            c.irz = 1.0 / c.rz;  // for the next beta
            if (!(rr == rr)) c.status = ST_NONFINITE;
            else if (rr > c.goal && before + it >= maxit) c.status = ST_PCG_MAXIT;
            c.conv = c.status || rr <= c.goal;
            c.verify = sizeof(S) == 4 && c.far && c.conv && c.status != ST_NONFINITE;
            if (!c.owner) continue;
            if (c.conv) {
                if (!single) {
                    A.conv[c.member] = 1;
                    atomicSub(A.active, 1);
                }
                if (c.status && !c.verify) atomicOr(A.status, c.status);
            }
            DevScalars& sc = A.scs[c.member];
            sc.iter = before + it;
            sc.total_iters += 1;
        }
    };
    // the converged members' flags for the tiles of the coarser levels (a
    // flag seen early or late only skips or repeats work that is not used)
    auto refresh = [&] {
        if (single) return;
        for (int k = threadIdx.x - 32; k < nrec; k += PS_NT - 32)
            rconv[k] = *(volatile int*)&A.conv[rec[k].member];
    };
    // Members still iterating. Of a batch: the counter, which changes only
    // while blocks wait at the barrier after phase A, so it reads the same in
    // every block here.
    __shared__ int s_go;
    auto go_on = [&] {
        if (single) return slot[0].conv == 0;
        if (threadIdx.x == 0) s_go = *(volatile int*)A.active;
        __syncthreads();
        const int v = s_go;
        __syncthreads();
        return v > 0;
    };
    // The FP32 form's true residual, once the recurrences have ended: x is
    // rounded with every update, so the two differ by a few eps |diagonal| |x| of
    // the largest iterate (0.7 to 4 on 256^2 .. 2000 x 40 from zero), and a start
    // 1e10 times the solution left 2e-5 to 1e-4 |b| unseen. So where a start was
    // worse than 0, b - A x is formed: within 8 eps |diagonal| |x| the solve is
    // done, beyond, CG starts again from it, as long as that reduces it 10x (as
    // the refinement rounds of the larger problems). False (in all blocks) when
    // no member goes on. (For every solve the pass cost 2 to 5 % of a step.)
    auto again = [&] {
        if (single && !slot[0].verify) return false;
        for (int i = 0; i < ns; ++i) {
            if (!slot[single ? 0 : i].verify) continue;
            double v[2] = {0.0, 0.0};
            p_init<true>(A, rec[i], v, smem);
            ps_block_total<2>(v, pb + rec[i].tile, nt);
        }
        if (!ps_sync(g)) return false;
        for (int i = w; i < nslot; i += PS_NT / 32) {
            PSlot& c = slot[i];
            if (!c.verify) continue;
            double xx, rr;
            ps_total2(pb + c.n0, pb + nt + c.n0, c.nn, xx, rr);
            if (lane) continue;
            const bool slow = c.checked > 0.0 && rr > 0.01 * c.checked;
            const bool done = rr <= 4.0 * c.goal || rr <= c.floor * xx || slow;
            c.verify = 0;
            c.rr = rr;
            c.checked = rr;
            if (done) c.status = 0;
            if (done || c.status) {
                if (c.status && c.owner) atomicOr(A.status, c.status);
                continue;
            }
            c.conv = 0;
            c.alpha = c.beta = c.d = c.rz = c.irz = 0.0;
            if (!c.owner) continue;
            A.scs[c.member].total_outer += 1;
            if (!single) {
                A.conv[c.member] = 0;
                atomicAdd(A.active, 1);
            }
        }
        before += it;
        it = 0;
        __syncthreads();
        if (single && slot[0].conv) return false;
        for (int i = 0; i < ns; ++i) {
            if (slot[single ? 0 : i].conv) continue;
            double v[2] = {0.0, 0.0};
            p_init<false>(A, rec[i], v, smem);
        }
        if (!ps_sync(g)) return false;
        for (int k = threadIdx.x; k < nrec; k += PS_NT)
            if (!single) rconv[k] = *(volatile int*)&A.conv[rec[k].member];
        return go_on();
    };
    __shared__ int s_far;
    if (threadIdx.x == 0) s_far = single ? slot[0].far : *(volatile int*)(A.active + 1);
    __syncthreads();
    while (go_on() || (sizeof(S) == 4 && s_far && again())) {
        for (int i = 0; i < ns; ++i) {
            const PSlot& c = slot[single ? 0 : i];
            if (c.conv) continue;
            double t[1] = {0.0};
            if (A.dense0) p_dense_a<S>(A, rec[i], A.dense[0], it, c.alpha, c.beta, t, smem);
            else p_phase_a<S>(A, rec[i], it, c.alpha, c.beta, t, smem);
            if (it > 0) ps_block_total<1>(t, pr + rec[i].tile, nt);
        }
        if (!ps_sync(g)) return;
        bool told = false;
        for (int l = 1; l < A.ng; ++l) {
            for (int i = lev0[l] - base; i < lev0[l + 1] - base; ++i)
                if (!rconv[i]) p_down<S>(rec[i], A.nu, smem);
            if (!(told ? ps_sync(g, refresh) : ps_sync(g, decide))) return;
            told = true;
            if (single && slot[0].conv) break;
        }
        if (single && slot[0].conv) continue;
        if (A.dense0 && single && it > 0) {
            // no level leg to hide the decision behind, and the phase that
            // would be lost is the whole solve: decide first
            if (w > 0) decide();
            __syncthreads();
            if (slot[0].conv) continue;
            told = true;
        }
        p_dense<S>(A, segs, smem);
        if (!(told ? ps_sync(g, refresh) : ps_sync(g, decide))) return;
        if (single && slot[0].conv) continue;
        for (int l = A.ng - 1; l >= 1; --l) {
            for (int i = lev0[l] - base; i < lev0[l + 1] - base; ++i)
                if (!rconv[i]) p_up<S>(rec[i], A.nu, smem);
            if (!ps_sync(g)) return;
        }
        for (int i = 0; i < ns; ++i) {
            if (slot[single ? 0 : i].conv) continue;
            double t[2] = {0.0, 0.0};
            if (A.dense0) p_dense_b<S>(A, rec[i], A.dense[0], t, smem);
            else p_phase_b<S>(A, rec[i], it, t, smem);
            ps_block_total<2>(t, pz + rec[i].tile, nt);
        }
        if (!ps_sync(g)) return;
        for (int i = w; i < nslot; i += PS_NT / 32) {
            PSlot& c = slot[i];
            if (c.conv) continue;
            double rz, zw;
            ps_total2(pz + c.n0, pz + nt + c.n0, c.nn, rz, zw);
            if (lane) continue;
            // beta = rz / rz_old, <p, A p> = <z, w> - beta^2 <p, A p>_old,
            // alpha = rz / <p, A p>
            c.beta = rz * c.irz;
            c.d = zw - c.beta * c.beta * c.d;
            c.alpha = rz / c.d;
            c.rz = rz;
        }
        __syncthreads();
        ++it;
    }
    if (threadIdx.x == 0)
        for (int i = 0; i < nslot; ++i)
            if (slot[i].owner) {
                DevScalars& sc = A.scs[slot[i].member];
                sc.bb = slot[i].bb;
                sc.rr = slot[i].rr;
                sc.converged = 1;
            }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.eg->loops_out += 1;
        A.eg->loops_in += before + it;
    }
}

// the level-0 down leg of every member by itself (a measurement)
template <typename S>
__global__ void __launch_bounds__(PS_NT, 1) k_ps_down0(const __grid_constant__ PSArgs A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int* l0 = A.rec0 + blockIdx.x * (A.ng + 1);
    double t[1] = {0.0};
    for (int i = l0[0]; i < l0[1]; ++i) p_phase_a<S>(A, A.recs[i], 0, 0.0, 0.0, t, smem);
}

// The V-cycle of one member on the levels from A.l0 on, for the FP32 form's
// level kernels of the grids that do not take the whole solve: a launch per
// level and leg took 8 to 9 us, whatever the level's size (its chain of
// dependent loads, tile record, flags, tensor map, tile, starts over with
// each), and the one-block kernel of the coarsest levels 23 us. Here a leg is
// a barrier and a tile, and the coarsest level is the dense one.
// qg 4096^2, the five levels from 512^2 on: 45 us; its step 14.28 -> 13.41 ms.
template <typename S>
__global__ void __launch_bounds__(PS_NT, 1) k_ps_cycle(const __grid_constant__ PSArgs A, int ir)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ PTile rec[PS_RECS];
    __shared__ int lev0[PS_LMAX + 1];
    __shared__ PSegs segs;
    const DevScalars& sc = A.scs[0];
    const int skip = sc.converged | (ir ? sc.conv_in : 0);
    PSGrid g = ps_grid(A.bar, A.status, A.bar->base);
    const int nl = A.ng + 1;
    if (threadIdx.x < nl) lev0[threadIdx.x] = A.rec0[blockIdx.x * nl + threadIdx.x];
    if (skip) return;  // (the same in every block: no barrier is left waiting)
    __syncthreads();
    const int base = lev0[0], nrec = lev0[A.ng] - base;
    {
        constexpr int W = sizeof(PTile) / 16;
        const int4* src = (const int4*)(A.recs + base);
        for (int k = threadIdx.x; k < nrec * W; k += PS_NT) ((int4*)rec)[k] = src[k];
    }
    p_find_rows(A, segs);  // (with a barrier after the copies above)
    for (int l = A.l0; l < A.ng; ++l) {
        for (int i = lev0[l] - base; i < lev0[l + 1] - base; ++i) p_down<S>(rec[i], A.nu, smem);
        if (!ps_sync(g)) return;
    }
    p_dense<S>(A, segs, smem);
    for (int l = A.ng - 1; l >= A.l0; --l) {
        if (!ps_sync(g)) return;
        for (int i = lev0[l] - base; i < lev0[l + 1] - base; ++i) p_up<S>(rec[i], A.nu, smem);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.bar->base = g.round;
}

__global__ void k_ps_cycle_reset(PSBar* bar) { ps_reset(bar); }

__global__ void k_ps_setup(const __grid_constant__ PSArgs A, double tol2, int maxit)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b == 0) {
        ps_reset(A.bar);
        A.active[0] = A.active[1] = 0;
    }
    if (b < A.nmem) {
        A.scs[b].tol2 = tol2;
        A.scs[b].bb_last = A.scs[b].bb;
        A.scs[b].bb = 0.0;  // (of a solve that does not finish, too)
        A.scs[b].maxit = maxit;
        A.scs[b].converged = 0;
        A.scs[b].iter = 0;
    }
}

// ---- host ----------------------------------------------------------------------
constexpr size_t PS_SMEM = 180 * 1024;

// Cycles of phases A and B for a tile of tw x th nodes: a fixed cost (the
// chain of loads, half sweeps and sums) and one per cell that the legs visit.
// Fitted to FP64 tiles of 26 x 18 (28.5k) and 52 x 52 (84k) and FP32 tiles of
// 34 x 40 (37k).
static double tile_cost(int tw, int th, int prec)
{
    const double n = (double)(tw + 10) * (th + 10);
    double cells = 2.0 * n + 3.0 * tw * th;
    for (int q = 0; q < 5; ++q) cells += (double)(tw + 2 * q) * (th + 2 * q);
    return 13400.0 + (prec == 0 ? 2.24 : 1.45) * cells;
}

struct TileDim {
    int tw, th, ntx, nty;
};

// dimensions of a level's tiles: nx x ny nodes in ntx x nty tiles, even sizes
static TileDim tile_dim(int nx, int ny, int ntx, int nty)
{
    TileDim d;
    d.tw = std::max(2, ((nx + ntx - 1) / ntx + 1) / 2 * 2);
    d.th = std::max(2, ((ny + nty - 1) / nty + 1) / 2 * 2);
    d.ntx = (nx + d.tw - 1) / d.tw;
    d.nty = (ny + d.th - 1) / d.th;
    return d;
}

static size_t region_bytes(int tw, int th, int prec)
{
    return (size_t)(tw + 10) * (th + 10) * (prec == 0 ? 17 : 9);
}

// Longest tiles first, each to the block with the least work: the block of
// every tile and the load of the busiest block
static double deal(const std::vector<double>& cost, int blocks, std::vector<int>* where)
{
    std::vector<int> order(cost.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>,
                        std::greater<std::pair<double, int>>> q;
    for (int g = 0; g < blocks; ++g) q.push({0.0, g});
    if (where) where->assign(cost.size(), 0);
    double worst = 0.0;
    for (int i : order) {
        std::pair<double, int> t = q.top();
        q.pop();
        t.first += cost[i];
        worst = std::max(worst, t.first);
        if (where) (*where)[i] = t.second;
        q.push(t);
    }
    return worst;
}

// Tiles of one level of all members. One member: of all partitions the one
// with the smallest estimate of the busiest block's time; up to about 1300^2
// nodes that is one tile per block. A batch: one tile per block, the members
// cut in turn, or tiles of at most T x T nodes for all members, whichever has
// the smallest estimate for the busiest block.
static std::vector<TileDim> pick_tiles(const std::vector<std::pair<int, int>>& nxny, int sms,
                                       int prec)
{
    std::vector<TileDim> best(nxny.size(), TileDim{0, 0, 0, 0}), cur(nxny.size());
    double bc = 0.0;
    if (nxny.size() == 1) {
        const int nx = nxny[0].first, ny = nxny[0].second;
        if (nx <= 0) return best;
        for (int ntx = 1; ntx <= (nx + 7) / 8; ++ntx)
            for (int nty = 1; nty <= (ny + 7) / 8; ++nty) {
                const TileDim d = tile_dim(nx, ny, ntx, nty);
                if (region_bytes(d.tw, d.th, prec) > PS_SMEM) continue;
                const long long nt = (long long)d.ntx * d.nty;
                const double c = (double)((nt + sms - 1) / sms) * tile_cost(d.tw, d.th, prec);
                if (bc == 0.0 || c < bc) {
                    bc = c;
                    best[0] = d;
                }
            }
        return best;
    }
    // one tile per block at most: the member with the costliest tiles is cut
    // once more, in the direction that helps it more, while blocks are left
    {
        std::vector<std::pair<int, int>> cut(nxny.size(), {1, 1});
        std::vector<double> cost(nxny.size(), 0.0);
        auto dim = [&](size_t b, int x, int y) {
            return tile_dim(nxny[b].first, nxny[b].second, x, y);
        };
        auto price = [&](const TileDim& d) {
            return region_bytes(d.tw, d.th, prec) > PS_SMEM ? 1e12 * d.tw * d.th
                                                            : tile_cost(d.tw, d.th, prec);
        };
        int total = 0;
        for (size_t b = 0; b < nxny.size(); ++b) {
            if (nxny[b].first <= 0) continue;
            cur[b] = dim(b, 1, 1);
            cost[b] = price(cur[b]);
            ++total;
        }
        while (total <= sms) {
            const size_t b = std::max_element(cost.begin(), cost.end()) - cost.begin();
            const TileDim x = dim(b, cut[b].first + 1, cut[b].second);
            const TileDim y = dim(b, cut[b].first, cut[b].second + 1);
            const bool wide = price(x) <= price(y);
            const TileDim& d = wide ? x : y;
            const int more = d.ntx * d.nty - cur[b].ntx * cur[b].nty;
            if (total + more > sms || price(d) >= cost[b]) break;
            total += more;
            cur[b] = d;
            cost[b] = price(d);
            (wide ? cut[b].first : cut[b].second) += 1;
        }
        const double worst = *std::max_element(cost.begin(), cost.end());
        if (total <= sms && worst < 1e9) {
            bc = worst;
            best = cur;
        }
    }
    for (int T = 8; T <= 128; T += 4) {
        if (region_bytes(T, T, prec) > PS_SMEM) break;
        std::vector<double> cost;
        for (size_t b = 0; b < nxny.size(); ++b) {
            const int nx = nxny[b].first, ny = nxny[b].second;
            cur[b] = TileDim{0, 0, 0, 0};
            if (nx <= 0) continue;
            cur[b] = tile_dim(nx, ny, (nx + T - 1) / T, (ny + T - 1) / T);
            cost.insert(cost.end(), (size_t)cur[b].ntx * cur[b].nty,
                        tile_cost(cur[b].tw, cur[b].th, prec));
        }
        const double c = deal(cost, sms, nullptr);
        if (bc == 0.0 || c < bc) {
            bc = c;
            best = cur;
        }
    }
    return best;
}

static int ps_try(PSolver& s, const std::vector<PSMember>& mem, int prec, long long nelem,
                  double* const (&work)[4], DevScalars* scs, BSGlobals* eg, int* status, int l0)
{
    const int n = (int)mem.size(), sms = ps_sms();
    if (n < 1 || sms < 1 || (l0 == 0 && nelem <= 0) || (l0 > 0 && n > 1)) return 0;
    const size_t es = prec == 0 ? 8 : 4;
    auto dal = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
        cudaMemset(p, 0, bytes);
        s.owned.push_back(p);
        return p;
    };
    // grid levels of every member: down to its dense level
    std::vector<int> ng(n);
    int maxg = 0, nrows = 0;
    auto unknowns = [](const MGLevel& L) {
        return (long long)(L.per ? L.nxn : std::max(0, L.nxn - 2)) * std::max(0, L.nyn - 2);
    };
    for (int b = 0; b < n; ++b) {
        const std::vector<MGLevel>& lev = mem[b].mg->lev;
        int l = l0 > 0 ? l0 + 1 : n == 1 ? 0 : 1;  // (a cycle: one grid level at least)
        for (; l < (int)lev.size(); ++l) {
            const long long k = unknowns(lev[l]);
            if (k <= mem[b].ndense_cap && ps_band_ok(k, lev[l].nxn, prec)) break;
        }
        if (l >= (int)lev.size() || l >= PS_LMAX || unknowns(lev[l]) < 1) return 0;
        for (int q = l0; q < l; ++q)  // colours and the coarse grid wrap only over an even count
            if (lev[q].per && lev[q].nxn % 2) return 0;
        // the unknowns leave the closed edges out: they must be dry
        const std::vector<uint8_t>& hm = mem[b].mg->hmask[l];
        for (int J = 0; J < lev[l].nyn; ++J)
            for (int I = 0; I < lev[l].nxn; ++I)
                if ((J == 0 || J == lev[l].nyn - 1 ||
                     (!lev[l].per && (I == 0 || I == lev[l].nxn - 1))) &&
                    hm[(size_t)J * lev[l].nxn + I])
                    return 0;
        ng[b] = l;
        maxg = std::max(maxg, l);
        nrows += (int)unknowns(lev[l]);
    }
    PSArgs& a = s.a;
    memset(&a, 0, sizeof(a));
    a.dense0 = maxg == 0;
    a.l0 = l0;
    a.ng = std::max(1, maxg);
    a.nmem = n;
    a.nrows = nrows;
    // tiles, level by level
    std::vector<std::vector<PTile>> tl(a.ng);
    std::vector<PDense> dense(n);
    size_t smem = 0, maxrow = 0;
    PSScratch scratch;
    // b, x and the inverse of every dense level, in one allocation
    auto align = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    size_t dbytes = 0;
    auto sizes = [&](int b, size_t& nv, size_t& ni) {
        const MGLevel& D = mem[b].mg->lev[ng[b]];
        const int nd = (int)unknowns(D);
        nv = align((size_t)D.nyn * D.nxn * es);
        ni = align((size_t)nd * (prec == 0 ? ps_pitch<double>(nd) : ps_pitch<float>(nd)) * es);
        return 2 * nv + ni;
    };
    size_t nv, ni;
    for (int b = 0; b < n; ++b) dbytes += sizes(b, nv, ni);
    char* dmem = (char*)dal(dbytes);
    if (!dmem) return 2;
    for (int b = 0; b < n; ++b) {
        const MGLevel& D = mem[b].mg->lev[ng[b]];
        // the unknowns: all nodes but the closed edges' (no fluid node there)
        const int e0 = D.per ? 0 : 1, w = D.nxn - 2 * e0, nd = w * (D.nyn - 2);
        dense[b].n = nd;
        dense[b].row0 = b ? dense[b - 1].row0 + dense[b - 1].n : 0;
        dense[b].box = PSBox{w, D.nxn, D.nxn + e0, 1.0f / (float)w};
        const size_t member = sizes(b, nv, ni);
        dense[b].b = dmem;
        dense[b].x = dmem + nv;
        void* minv = dmem + 2 * nv;
        dmem += member;
        const int np = prec == 0 ? ps_pitch<double>(nd) : ps_pitch<float>(nd);
        maxrow = std::max(maxrow, np * es);
        dense[b].minv = minv;
        // -A of the dense level (identity rows at non-fluid nodes: their b is 0)
        const std::vector<uint8_t>& hm = mem[b].mg->hmask[ng[b]];
        const int w1 = w + 1;
        std::vector<double> h((size_t)nd * w1, 0.0);
        auto fluid = [&](int J, int I) {
            return J >= 0 && J < D.nyn && I >= 0 && I < D.nxn && hm[(size_t)J * D.nxn + I] != 0;
        };
        for (int k = 0; k < nd; ++k) {
            const int J = 1 + k / w, I = e0 + k % w;
            double* r = &h[(size_t)k * w1];
            r[0] = fluid(J, I) ? -D.diag : 1.0;
            if (!fluid(J, I)) continue;
            if (k % w > 0 && fluid(J, I - 1)) r[1] -= D.cx;
            if (J > 1 && fluid(J - 1, I)) r[w] -= D.cy;
            if (D.per && I == D.nxn - 1 && D.nxn > 1 && fluid(J, 0)) r[I] -= D.cx;
        }
        const int rc = ps_invert(h, nd, w, {}, -1.0, prec, minv, scratch);
        if (rc == 5) return 0;
        if (rc) return rc;
        const int rows = (nrows + sms - 1) / sms;  // of a block, at most
        smem = std::max(smem, es * (prec == 0 ? ps_dense_elems<double>(nd, rows)
                                              : ps_dense_elems<float>(nd, rows)));
    }
    for (int l = l0; l < a.ng; ++l) {
        std::vector<std::pair<int, int>> dims(n);
        for (int b = 0; b < n; ++b) {
            const MGLevel& L = mem[b].mg->lev[l];
            dims[b] = l < ng[b] || (l == 0 && a.dense0) ? std::make_pair(L.nxn, L.nyn)
                                                        : std::make_pair(0, 0);
        }
        const std::vector<TileDim> td = pick_tiles(dims, sms, prec);
        for (int b = 0; b < n; ++b) {
            if (dims[b].first <= 0) continue;
            if (td[b].tw <= 0) return 0;
            const std::vector<MGLevel>& lev = mem[b].mg->lev;
            const MGLevel& L = lev[l];
            PTile t;
            memset(&t, 0, sizeof(t));
            t.m = L.m;
            t.x = L.x;
            t.xa = L.xa;
            t.b = L.b;
            t.off = L.off;
            t.pitch = (int)L.pitch;
            t.nyn = L.nyn;
            t.nxn = L.nxn;
            t.per = L.per;
            t.member = b;
            t.tw = td[b].tw;
            t.th = td[b].th;
            t.cx = L.cx;
            t.cy = L.cy;
            t.md = L.md;
            t.id = L.idiag;
            t.dg = L.diag;
            t.cxi = L.cx * L.idiag;
            t.cyi = L.cy * L.idiag;
            if (l < ng[b]) {
                const MGLevel& C = lev[l + 1];
                const bool d = l + 1 == ng[b];
                t.cx_ = d ? dense[b].x : C.x;
                t.cb = d ? dense[b].b : C.b;
                t.coff = d ? 0 : C.off;
                t.cpitch = d ? C.nxn : (int)C.pitch;
                t.cm = C.m;
                t.cmoff = C.off;
                t.cmpitch = (int)C.pitch;
                t.cyn = C.nyn;
                t.cxn = C.nxn;
            }
            t.n0 = (int)tl[l].size();
            t.nn = td[b].ntx * td[b].nty;
            for (int y = 0; y < td[b].nty; ++y)
                for (int x = 0; x < td[b].ntx; ++x) {
                    t.J0 = y * t.th;
                    t.I0 = x * t.tw;
                    t.tile = (int)tl[l].size();
                    tl[l].push_back(t);
                }
            smem = std::max(smem, region_bytes(t.tw, t.th, prec));
        }
    }
    a.ntiles = (int)tl[0].size();
    smem = (smem + 15) / 16 * 16;
    const size_t keep = maxrow * ((nrows + sms - 1) / sms);
    if (l0 == 0 && smem + keep <= PS_SMEM) {  // (a cycle reads them once)
        a.mkeep = (int)smem;
        smem += keep;
    }
    std::vector<std::vector<std::vector<int>>> of(sms, std::vector<std::vector<int>>(a.ng));
    for (int l = 0; l < a.ng; ++l) {
        std::vector<double> cost;
        std::vector<int> where;
        for (const PTile& t : tl[l]) cost.push_back(tile_cost(t.tw, t.th, prec));
        deal(cost, sms, &where);
        for (size_t t = 0; t < where.size(); ++t) of[where[t]][l].push_back((int)t);
    }
    std::vector<PTile> recs;
    std::vector<int> rec0;
    for (int g = 0; g < sms; ++g) {
        const size_t first = recs.size();
        for (int l = 0; l < a.ng; ++l) {
            rec0.push_back((int)recs.size());
            for (int t : of[g][l]) recs.push_back(tl[l][t]);
            if (l == 0 && recs.size() - first > PS_SLOTS) return 0;
        }
        rec0.push_back((int)recs.size());
        if (recs.size() - first > PS_RECS) return 0;
    }
    PTile* drec = (PTile*)dal(recs.size() * sizeof(PTile));
    int* d0 = (int*)dal(rec0.size() * sizeof(int));
    PDense* dd = (PDense*)dal(n * sizeof(PDense));
    // r and s in the caller's vectors (no value is read before it is written)
    double* vec[6] = {work[0], work[1], work[2], work[3], nullptr, nullptr};
    for (double*& p : vec)
        if (l0 == 0 && !p && !(p = (double*)dal((size_t)nelem * 8))) return 2;
    a.part = (double*)dal((size_t)5 * std::max(1, a.ntiles) * sizeof(double));
    a.conv = (int*)dal(n * sizeof(int));
    a.active = (int*)dal(2 * sizeof(int));
    a.bar = (PSBar*)dal(sizeof(PSBar));
    if (!drec || !d0 || !dd || !a.part || !a.conv || !a.active || !a.bar) return 2;
    if (cudaMemcpy(drec, recs.data(), recs.size() * sizeof(PTile), cudaMemcpyHostToDevice) !=
            cudaSuccess ||
        cudaMemcpy(d0, rec0.data(), rec0.size() * sizeof(int), cudaMemcpyHostToDevice) !=
            cudaSuccess ||
        cudaMemcpy(dd, dense.data(), n * sizeof(PDense), cudaMemcpyHostToDevice) != cudaSuccess)
        return 2;
    a.recs = drec;
    a.rec0 = d0;
    a.dense = dd;
    a.r[0] = vec[0];
    a.r[1] = vec[1];
    a.s[0] = vec[2];
    a.s[1] = vec[3];
    a.p = vec[4];
    a.w = vec[5];
    a.scs = scs;
    a.eg = eg;
    a.status = status;
    s.prec = prec;
    a.dg = mem[0].mg->lev[0].diag;
    s.grid = sms;
    s.smem = smem;
    for (const void* k : {(const void*)k_ps_solve<double>, (const void*)k_ps_solve<float>,
                          (const void*)k_ps_down0<double>, (const void*)k_ps_down0<float>,
                          (const void*)k_ps_cycle<float>})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PS_SMEM) !=
            cudaSuccess)
            return 3;
    if (smem > PS_SMEM) return 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    s.on = true;
    return 0;
}

int ps_build(PSolver& s, const std::vector<PSMember>& mem, int prec, long long nelem,
             double* const (&work)[4], DevScalars* scs, BSGlobals* eg, int* status, int l0)
{
    ps_free(s);
    const int rc = ps_try(s, mem, prec, nelem, work, scs, eg, status, l0);
    if (s.on) return 0;
    ps_free(s);
    if (rc != 2) return rc;
    cudaGetLastError();  // out of memory: the level kernels need less
    return 0;
}

void ps_free(PSolver& s)
{
    for (void* p : s.owned) cudaFree(p);
    s.owned.clear();
    s.on = false;
    s.a = PSArgs{};
}

int ps_record(PSolver& s, double* x, double* b, int nu, double tol, int maxit, cudaStream_t st)
{
    s.a.x = x;
    s.a.b = b;
    s.a.nu = nu;
    k_ps_setup<<<(s.a.nmem + 127) / 128, 128, 0, st>>>(s.a, tol * tol, maxit);
    const int e = (int)cudaGetLastError();
    if (e) return e;
    void* args[1] = {&s.a};
    return ps_launch(s.prec == 0 ? (const void*)k_ps_solve<double>
                                 : (const void*)k_ps_solve<float>,
                     s.grid, s.smem, args, st);
}

int ps_record_cycle_reset(PSolver& s, cudaStream_t st)
{
    k_ps_cycle_reset<<<1, 1, 0, st>>>(s.a.bar);
    return (int)cudaGetLastError();
}

int ps_record_cycle(PSolver& s, int nu, int ir, cudaStream_t st)
{
    s.a.nu = nu;
    void* args[2] = {&s.a, &ir};
    return ps_launch((const void*)k_ps_cycle<float>, s.grid, s.smem, args, st);
}

int ps_time_down(PSolver& s, int nu, cudaStream_t st)
{
    s.a.nu = nu;
    if (s.prec == 0) k_ps_down0<double><<<s.grid, PS_NT, s.smem, st>>>(s.a);
    else k_ps_down0<float><<<s.grid, PS_NT, s.smem, st>>>(s.a);
    return (int)cudaGetLastError();
}

}  // namespace f2d
