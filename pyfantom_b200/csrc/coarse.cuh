// Element-level operator of multigrid level 1 (coarse.cu).
#pragma once

#include "common.cuh"
#include "elemop.cuh"

namespace pf {

struct CoarseOp {
    Grid fine, g;                 // fine grid and level-1 grid
    int tsize = 8;                // bytes per value of the V-cycle precision
    double coef[150];             // the distinct nonzeros of B0 (Walsh-basis child-0 matrix)
    void* Eh = nullptr;           // Ehat [8][coarse elements], V-cycle precision
    int* count = nullptr;         // device: number of dirty elements, of listed nodes
    int* h_count = nullptr;       // pinned copy
    int* bcount = nullptr;        // per-block counts of the flag compactions
    int ndirty = 0;               // elements that touch a constraint
    // their corner nodes: flag per node, list, and assembled stencil rows [cap][243]
    uint8_t* nflag = nullptr;
    int* nlist = nullptr;
    void* S = nullptr;
    int cap = 0, nrows = 0;
};

// PF_OK if K0 has the structure of an isotropic box element (coefficients in coef[150])
int coarse_factorise(const Op* op, double* coef);
int coarse_create(const Op* op, int fp32, CoarseOp** out);
void coarse_destroy(CoarseOp* c);
// Ehat for E and the rows of the constrained elements' corners from the level-1 stencil A64;
// *realloc set when their storage moved, or when the first such node came or the last one went
int coarse_setup(CoarseOp* c, const double* E, const uint8_t* mask, const uint8_t* elem_flag, const double* A64,
                 cudaStream_t st, bool* realloc);
template <typename T>
int launch_coarse_matvec(const CoarseOp* c, const Grid& g, const T* u, const Epi<T>& epi, cudaStream_t st);

}  // namespace pf
