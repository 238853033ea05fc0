// Launchers of the fused stage and diagnostic kernels (stage.cu).
#pragma once
#include "common.cuh"

namespace f2d {

struct RswIn {
    const void *ux, *uy, *h;        // prognostic, stage input
    const void* w;                  // omega (qgrsw: the wrap of the edge tiles)
    void *uxo, *uyo, *ho;           // prognostic, stage output
    const void *Ux, *Uy, *ke, *p;   // diagnostics of the stage input
    void *dux, *duy, *dh;           // this stage's tendencies (stored if != 0)
    const void *dux1, *duy1, *dh1;  // earlier tendencies
    const void *dux2, *duy2, *dh2;
    const void *fx, *fy, *fh;       // forcing terms added to the tendencies (or null)
    double fc;                      // f0 * area * 0.25 (operators.py:33)
    double bdy;                     // 0.5 * dy (addbuoyancy, operators.py:152-153)
    float fbdy;                     // the same in FP32 (set by the launcher)
    // 0 rsw; 1 euler (vortex force + grad ke only); 2 boussinesq (euler +
    // buoyancy, with the buoyancy b advected in place of h); 3 qgrsw (the
    // raw tendency of vortex force, Coriolis and mass flux into dux/duy/dh,
    // no update)
    int euler;
};

struct RswDiag {
    const void *ux, *uy, *h;
    void *Ux, *Uy, *omega, *ke, *p;
    double rdx2, rdy2;  // 1/dx**2, 1/dy**2 (operators.py:62-63)
    double goa;         // g/area (operators.py:111)
    float frdx2, frdy2, fgoa;  // the same in FP32 (set by the launcher)
    int euler;          // euler model: no pressure from h
    int noke;           // qgrsw: no kinetic energy (equations.py:127-133)
    int maxu;           // max |U.x|, |U.y| into the scalars (zeroed before)
};

int launch_fluxform_stage(int method, int prec, const CUtensorMap* tq,
                          const void* qin, void* qout, const void* Ux,
                          const void* Uy, const uint32_t* code, void* ds_out,
                          const void* ds1, const void* ds2, const void* frc, int stage,
                          const Geom& g, DevScalars* sc, cudaStream_t s);
int launch_rsw_stage(int method, int prec, const CUtensorMap* th,
                     const CUtensorMap* tw, const RswIn& a, const uint32_t* code,
                     int stage, const Geom& g, DevScalars* sc, cudaStream_t s);
int launch_rsw_diag(int method, int prec, const CUtensorMap* tux,
                    const CUtensorMap* tuy, const RswDiag& a, const uint32_t* code,
                    const Geom& g, DevScalars* sc, cudaStream_t s);
int launch_c2v(int prec_in, int prec_out, const void* q, void* v, const uint32_t* code,
               const void* fv, const Geom& g, cudaStream_t s);
int launch_perpgrad(int prec_psi, int prec_U, const void* psi, void* Ux, void* Uy,
                    const uint32_t* code, double rdy2, double rdx2, int fillU,
                    const Geom& g, DevScalars* sc, double* partials, cudaStream_t s);
int launch_convert(int prec_in, int prec_out, const void* in, void* out, const Geom& g,
                   cudaStream_t s);
int launch_maxabs2(int prec, const void* Ux, const void* Uy, const Geom& g,
                   DevScalars* sc, double* partials, cudaStream_t s);
int launch_fill_periodic(int prec, void* a, const Geom& g, cudaStream_t s);
int launch_set_dt(DevScalars* sc, cudaStream_t s);
// Warm start of the Poisson solve of SSP-RK3 stage mode+1. The stage states
// are y1 = y0 + dt L1, y2 = y0 + dt/4 (L1 + L2), y3 = y0 + dt/6 (L1 + L2) +
// 2dt/3 L3 (integrators.py:92-107, L_k the tendency at the stage's input),
// and psi solves a linear problem in y, so with S_k = dt A^-1 B(L_k):
// psi1 = psi0 + S1, psi2 = psi0 + (S1 + S2)/4. The guesses extrapolate the
// S_k, not psi, from the relations of the previous step (primes: its values,
// scaled by dt / dt_warm when the step size changed):
//   S1 (the tendency at t)       ~ S2' + (S1' - S2'')          (S2' at y1' ~ y(t))
//   S2 (at y1 ~ t + dt)          ~ S1 + D' + (D' - D''), D = S2 - S1
//   S3 (at y2 ~ t + dt/2)        ~ (S1 + S2)/2 + (S3' - (S1' + S2')/2)
// with S3 = 1.5 (psi3 - psi0) - (S1 + S2)/4. The terms in brackets, kept as
// e1, e2, e3 (0 until the steps they need are there), change slowly: on
// eulerpsi 128^2 they cut the starting relative residuals from 1.3e-5, 7e-6
// and 4.4e-6 to 1.7e-6, 9e-7 and 5.5e-7, on qg 128^2 turbulence from 1.3e-3,
// 7.5e-4 and 4.7e-4 to 5.6e-4, 5.6e-4 and 3.2e-4. Where the increments of a
// step come down to the FP32 rounding of the state (psi_warm_brackets) the
// brackets are noise and left out. A guess moves the solve's starting point, and
// the residual that its recurrence can attain by about eps times the largest
// iterate: it must not be larger than the solution (no history across a diag of another
// state).
struct WarmArrays {
    double* psi;  // in: the last solution; out: the guess
    double* s0;   // psi at the step start
    double* p1;   // psi of stage 1
    double* d1;   // the previous step's S2
    double* d2;   // the previous step's D = S2 - S1
    double *e1, *e2, *e3;  // the brackets, or null
};
// whether a model keeps the brackets: FP64 states always, FP32 ones up to 3M
// points. (A CFL step's change shrinks with the grid spacing, its rounding
// does not. FP32 CG iterations per solve without and with them: 9.67 and 8.36
// on the 256-member ensemble of 64^2 .. 512^2, 8.33 and 8.64 on qg 4096^2;
// 2048^2 gains what the extra arrays cost.) Beyond 1e8 points a model is to fit
// the memory as it did without them: 2.4 GB and more of arrays (the pressure's
// whole history, 4.8 GB), which only shorten the solves.
constexpr long long WARM_POINTS = 100000000ll;
inline bool psi_warm_brackets(int prec, long long points)
{
    return points <= (prec == 0 ? WARM_POINTS : 3000000ll);
}

// U pairs of elements (k, k + 1), k even and every array 16-byte aligned
// there: 16-byte loads and stores, all the loads of the U pairs before any
// store (the arrays do not overlap, but a store ahead of a load through
// another pointer would hold the load back). ok[u] false skips pair u. The
// brackets are 0 without ws.hist. The large grids are bound by the FP64
// pipe here too, so the mode and the brackets (EXT) are compile-time.
// e3 holds t3 = 1.5 psi0 + 0.75 (S1 + S2) of the step between its stages 2
// and 3 (S3 - (S1 + S2)/2 = 1.5 psi3 - t3).
template <int MODE, bool EXT, int U>
__device__ __forceinline__ void psi_warm_pairs(const WarmArrays& w, const long long (&k)[U],
                                               const bool (&ok)[U], const WarmState& ws)
{
    const bool hist = ws.hist;
    const double rho = ws.rho;
    double2 a[U], s0[U], p1[U], d1[U], d2[U], e[U], t3[U];
    const double* ein = MODE == 0 ? w.e1 : MODE == 1 ? w.e2 : w.e3;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const double2 z = make_double2(0.0, 0.0);
        const bool h = ok[u] && hist;
        a[u] = ok[u] ? *(const double2*)(w.psi + k[u]) : z;
        s0[u] = MODE >= 1 && ok[u] ? *(const double2*)(w.s0 + k[u]) : z;
        p1[u] = MODE == 2 && ok[u] ? *(const double2*)(w.p1 + k[u]) : z;
        d1[u] = (MODE == 0 || (MODE == 1 && EXT)) && h ? *(const double2*)(w.d1 + k[u]) : z;
        d2[u] = (MODE == 1 || (MODE == 2 && EXT)) && h ? *(const double2*)(w.d2 + k[u]) : z;
        e[u] = EXT && h ? *(const double2*)(ein + k[u]) : z;
        t3[u] = EXT && MODE == 0 && h ? *(const double2*)(w.e3 + k[u]) : z;
    }
    const double rq = 0.25 * rho, r23 = rho * (2.0 / 3.0);
    // one element: the guess g, the bracket en, mode 2: S2, D and t3
    auto one = [&](double A, double S, double P, double D1, double D2, double E, double T3,
                   double& g, double& en, double& n1, double& n2, double& n3) {
        if constexpr (MODE == 0) {  // A = psi0, psi3 of the previous step
            if constexpr (EXT) {
                en = fma(1.5, A, -T3);
                D1 += E;
            }
            g = fma(rho, D1, A);
        } else if constexpr (MODE == 1) {  // A = psi1
            const double S1 = A - S;
            if constexpr (EXT) {
                en = fma(-rho, D1, S1);
                D2 += E;
            }
            g = S + fma(rq, D2, 0.5 * S1);
        } else {  // A = psi2
            const double t = A - S, S1 = P - S;
            n1 = fma(4.0, t, -S1);
            n2 = n1 - S1;
            g = A + t;
            if constexpr (EXT) {
                en = fma(-rho, D2, n2);
                g = fma(r23, E, g);
                n3 = fma(1.5, S, 0.75 * (S1 + n1));
            }
        }
    };
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        double2 g, en, n1, n2, n3;
        one(a[u].x, s0[u].x, p1[u].x, d1[u].x, d2[u].x, e[u].x, t3[u].x, g.x, en.x, n1.x, n2.x,
            n3.x);
        one(a[u].y, s0[u].y, p1[u].y, d1[u].y, d2[u].y, e[u].y, t3[u].y, g.y, en.y, n1.y, n2.y,
            n3.y);
        if (!hist) en = make_double2(0.0, 0.0);
        if constexpr (MODE == 0) {
            *(double2*)(w.s0 + k[u]) = a[u];
            if (hist) *(double2*)(w.psi + k[u]) = g;
            if constexpr (EXT) *(double2*)(w.e3 + k[u]) = en;
        } else if constexpr (MODE == 1) {
            *(double2*)(w.p1 + k[u]) = a[u];
            *(double2*)(w.psi + k[u]) = g;
            if constexpr (EXT) *(double2*)(w.e1 + k[u]) = en;
        } else {
            *(double2*)(w.d1 + k[u]) = n1;
            *(double2*)(w.d2 + k[u]) = n2;
            *(double2*)(w.psi + k[u]) = g;
            if constexpr (EXT) {
                *(double2*)(w.e2 + k[u]) = en;
                *(double2*)(w.e3 + k[u]) = n3;
            }
        }
    }
}

// the single-model form over n elements, n even (every point; non-fluid points
// stay 0)
int launch_psi_warm(int mode, const WarmArrays& w, long long n, DevScalars* sc,
                    cudaStream_t s);

// after a diag: keep the history of n models only where the state is still the
// last step's (warm_check)
int launch_warm_check(DevScalars* scs, int n, cudaStream_t s);

// Warm start of the pressure solve of RK3 stage mode+1 (euler and boussinesq,
// FP64 states). The stages add -3/4 L1 + 1/4 L2 and so on of the unprojected
// tendencies, so with Q_k the pressure of L_k and S_k = dt Q_k the three solves
// give p1 = S1, p2 = (S2 - 3 S1)/4 and p3 = 2/3 S3 - (S1 + S2)/12, whose signs
// alternate: the previous solution is no better a start than zero. The S_k are
// extrapolated like those of psi above (s0 holds S1, d1 S2, d2 S2 - S1, e1 to
// e3 the brackets, p1 is not used). CG iterations per solve, euler 512^2 with
// the previous solution and with this: 9.0 and 6.9. FP32 states keep the
// former: their velocities round differently wherever the pressure moves by
// the solve's tolerance.
int launch_p_warm(int mode, const WarmArrays& w, const uint32_t* code, long long n,
                  DevScalars* sc, cudaStream_t s);
// the failure-detection test switch of the stage kernels' TMA waits, one per
// translation unit (stage.cu, ensemble.cu)
int tma_wait_test_set_stage(int enabled, unsigned long long limit_ns);
int tma_wait_test_set_ensemble(int enabled, unsigned long long limit_ns);
int launch_pushforward(DevScalars* sc, cudaStream_t s);
size_t pt_grid_blocks(const Geom& g);
// euler pressure projection around the Neumann solve
int launch_euler_div(int prec, const void* ux, const void* uy, void* dv, double* rhs,
                     const uint32_t* code, double rdx2, double rdy2, double area,
                     const Geom& g, cudaStream_t s);
// qgrsw: the QG projection of a tendency (or of the state) around the
// Helmholtz solve (qg_projection, operators.py:176-211)
struct QgProj {
    const void *ux, *uy, *h;        // state in (the update's base)
    void *uxo, *uyo, *ho;           // state out
    void *cx, *cy, *ch;             // raw tendency (state form: the state, in place)
    void *sx, *sy, *sh;             // projected tendency out (if store)
    const void *d1x, *d1y, *d1h;    // earlier projected tendencies (RK) or the
    const void *d2x, *d2y, *d2h;    //   filtered previous state (LFRA, d1)
    void *px, *py, *ph;             // LFRA: filtered state out
    const void *fx, *fy, *fh;       // forcing terms added to the projected tendency
    double c2;                      // f0 * area / g (thickness_from_psi)
    double h0;                      // state mode: H * area - hb, else 0
    int mode;                       // 0: tendency + integrator update;
                                    // 1: project the state (cx.. in place);
                                    // 2: the projected tendency into sx.. only
    int store;                      // keep the projected tendency in sx..
};
int launch_qgrsw_pv(int prec, const void* ux, const void* uy, const void* h, double* pv,
                    const uint32_t* code, double cs, double h0, const Geom& g,
                    cudaStream_t s);
int launch_qgrsw_update(int prec, const QgProj& a, const double* psi, const uint32_t* code,
                        int stage, const Geom& g, DevScalars* sc, cudaStream_t s);
// Bulk diagnostics (diagnostics.py:39-57) appended to a device ring
struct BulkArgs {
    const void *ke, *omega, *Ux, *Uy;
    double* ring;      // records of {t, ke, ens, vort, angular}
    int* count;        // records in the ring
    int cap;
    double summsk, area, dx, dy;
};
int launch_bulk(int prec, const BulkArgs& a, const Geom& g, DevScalars* sc, double* partials,
                cudaStream_t s);
// a field as packed (NY, NX) float32 (the history's dtype "f", io.py:71)
int launch_to_f32(int prec, const void* in, float* out, const Geom& g, cudaStream_t s);
int launch_euler_project(int prec, void* ux, void* uy, const double* p, const uint32_t* code,
                         const Geom& g, DevScalars* sc, cudaStream_t s);

}  // namespace f2d
