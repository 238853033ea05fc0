// Multigrid-preconditioned CG for the masked cell-centred Poisson operator
// with Neumann walls (the pressure projection of the euler model). See
// nsolver.cu.
#pragma once
#include <vector>

#include "common.cuh"

namespace f2d {

constexpr int NS_LMAX = 16;  // levels, the dense one included

// One grid level: cells (J, I) of nyn x nxn at off + J*pitch + I; face
// couplings fx(J, I) between cells (J, I-1) and (J, I) (column 0: the
// periodic wrap face, else 0), fy(J, I) between (J-1, I) and (J, I) (row 0:
// 0), inv = 1 / (sum of a cell's four couplings), 0 where that sum is 0.
// Level 0 has a code byte per cell instead (its couplings are cx, cy or 0).
struct NLevel {
    void* x;           // the level's unknown (the cycle's precision)
    void* xa;          // x after the pre-smoothing
    void* b;
    const void* fx;
    const void* fy;
    const void* inv;
    const uint8_t* code;  // level 0: bit 0 fluid, bits 1-4 open west, east, south, north
    long long pitch, off;
    int nyn, nxn, per;
    int seam;          // x-periodic over an odd count: same-colour neighbours across the wrap
    int tw, th, ntx, nt;  // tiles of tw x th cells (both even)
};

struct NGlobals {
    int status, pad;
    long long iters;
};

// everything the solve kernel reads, in its parameter bank
struct NSArgs {
    NLevel lev[NS_LMAX];
    int ng;                // grid levels; level ng is the dense one
    int nd;                // cells of the dense level
    const void* minv;      // its inverse
    int mkeep;             // offset in shared memory of the block's rows of it (0: not kept)
    double cx, cy;
    double cs[9], inv[9];  // by 3 (open x-faces) + (open y-faces): coupling sum, its inverse
    // FP64 vectors in the level-0 layout: solution, right-hand side, residual
    // and s = A p (two buffers each, by the parity of the iteration), p, z, A z
    double *x, *b, *r[2], *s[2], *p, *w;
    void* z;               // the cycle's precision
    double* part;          // block totals
    void* bar;             // PSBar
    void* sc;              // DevScalars
    NGlobals* eg;
    double nfluid;
};

struct NSolver {
    NSArgs a = {};
    NGlobals* eg = nullptr;
    DevScalars* sc = nullptr;     // iteration state (own)
    int prec = 0;                 // 0: FP64 cycle; 1: FP32 cycle
    int grid = 0;                 // blocks of the solve kernel
    size_t smem = 0;
    double tol = 1e-12;
    int maxit = 200;
    std::vector<void*> owned;
};

// Build from the level-0 fluid mask (host, (J, I) at hoff + J*pitch + I) for
// the cells of the model layout: x = the pressure field, b = the right-hand
// side (both FP64, level-0 layout). cx = dy/dx (E-W), cy = dx/dy (N-S).
int ns_build(NSolver& s, int nyn, int nxn, long long pitch, long long off, int per,
             const uint8_t* hmask, double* x, double* b, double cx, double cy, int prec);
void ns_free(NSolver& s);
// Record a solve on `st` (two launches, eager or captured): b is made
// zero-mean over the fluid cells (the compatibility projection of the
// singular problem), x (warm start) is iterated to |r| <= tol |b| and
// finally made zero-mean.
int ns_record(NSolver& s, cudaStream_t st, int* launches);

}  // namespace f2d
