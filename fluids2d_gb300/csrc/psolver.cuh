// Persistent solve kernel for the masked vertex Poisson/Helmholtz operator of
// one or many models: the FP64 form of the batched solver, and its FP32 form
// for problems that do not fill the GPU. See psolver.cu.
#pragma once
#include <vector>

#include "mg.cuh"
#include "persist.cuh"

namespace f2d {

struct BSGlobals;

// One tile of one level of one member: everything a block reads about it
struct alignas(16) PTile {
    const uint8_t* m;   // fluid mask of the level; node (J, I) at off + J pitch + I
    void *x, *xa, *b;   // level arrays (level 0: z, xa, the FP32 copy of r)
    void *cx_, *cb;     // the next coarser level's x and b, node at coff + J cpitch + I
    const uint8_t* cm;  // its mask, at cmoff + J cmpitch + I
    long long off, coff, cmoff;
    int pitch, cpitch, cmpitch;
    int nyn, nxn, cyn, cxn, per;
    int J0, I0, tw, th;
    int member, tile;   // tile: index in the level's table
    int n0, nn;         // the member's tiles in the level-0 table
    int pad[2];
    double cx, cy, md;              // the operator
    double cxi, cyi, id, dg;        // couplings / diagonal, 1 / diagonal, diagonal
};

struct PDense {
    const void* minv;  // inverse of the member's dense level (n unknowns)
    void *b, *x;       // compact: rows of nxn nodes
    int n, row0;       // unknowns; those of the members before it
    PSBox box;         // the unknowns: the nodes off the closed edges
};

constexpr int PS_LMAX = 14;
constexpr int PS_RECS = 96;  // tile records of a block, all levels
constexpr int PS_SLOTS = 64; // of these, on level 0

struct PSArgs {
    const PTile* recs;   // block b's records: rec0[b (ng + 1) + l] .. for level l
    const int* rec0;
    const PDense* dense;
    int nmem, ng, nu;    // members, grid levels (of the deepest member)
    int l0;              // first level: 0, or that of the cycle alone
    int nrows;           // dense rows of all members
    int dense0;          // one member whose level 0 is the dense level
    int ntiles;          // level-0 tiles
    int mkeep;           // offset in shared memory of the block's dense rows (0: not kept)
    double dg;           // level-0 diagonal of the first member
    double *x, *b, *r[2], *s[2], *p, *w;  // arenas, FP64
    double* part;        // tile totals, 2 x 2 ntiles
    int* conv;           // per member
    int* active;         // members still iterating, members whose start was worse than 0
    DevScalars* scs;
    BSGlobals* eg;
    int* status;
    PSBar* bar;
};

struct PSolver {
    bool on = false;
    PSArgs a = {};
    int prec = 0, grid = 0;
    size_t smem = 0;
    std::vector<void*> owned;
};

struct PSMember {
    const MGHost* mg;   // its hierarchy (mg_build)
    int ndense_cap;     // nodes of its dense level, at most
};

// Build for the members' hierarchies: on = false (and no error) where the
// kernel does not apply (no level small enough for the dense inverse, more
// tiles than a block has records) or its memory is not to be had. work: FP64
// vectors of nelem elements that the solves may use. l0 > 0: one member, for
// ps_record_cycle alone, on the levels from l0 on (nelem and work are not used).
int ps_build(PSolver& s, const std::vector<PSMember>& mem, int prec, long long nelem,
             double* const (&work)[4], DevScalars* scs, BSGlobals* eg, int* status, int l0 = 0);
void ps_free(PSolver& s);
// Record one solve of every member on `st`: x and b are the arenas (FP64). It
// ends at |r| <= tol |b|, r the recurrence residual (FP32 form from a start worse
// than 0: b - A x to within its rounding, see k_ps_solve), or after maxit
// iterations.
int ps_record(PSolver& s, double* x, double* b, int nu, double tol, int maxit, cudaStream_t st);
// Record the V-cycle on the levels from l0 on (from its b to its x), skipped
// when the member is not iterating (ir: its inner loop); ps_record_cycle_reset
// before the first of a solve.
int ps_record_cycle(PSolver& s, int nu, int ir, cudaStream_t st);
int ps_record_cycle_reset(PSolver& s, cudaStream_t st);
// Measurement hook: one launch of the level-0 down leg of every member.
int ps_time_down(PSolver& s, int nu, cudaStream_t st);

}  // namespace f2d
