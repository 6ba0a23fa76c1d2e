// Direct solve of K(E) u = b for small structured problems: the drop-in for the reference's
// SPSOLVE (pyFANTOM/solvers/CUDA/_solvers.py:245-328), which assembles K in CSR
// (StructuredStiffnessKernel.construct, stiffness/CUDA/_FEA.py:484-516), keeps the free
// rows and columns and calls a sparse direct solver; constrained entries of the solution
// are the right-hand side's.
//
// Long thin grids (a half bandwidth of at most 96 with the nodes numbered along the shorter
// axis first; 2D grids up to 45 elements across) are solved by a banded Cholesky factorisation
// in 32 x 32 tiles that works inwards from both ends, k_band_solve: the constrained DOFs are
// kept as identity rows, the band holds the free-DOF block of K.  Elimination along a beam
// loses more digits than across it, so the solution is corrected once with its residual in
// pairs of doubles.
// Other problems assemble the free-DOF matrix dense (one thread per free row gathers its
// entries from the row node's adjacent elements, so every entry is written by one thread in a
// fixed order), factor it by the tiled Cholesky of the coarse solver (L L^T, inverse factor
// L^-1), and the solution is x = L^-T (L^-1 b) by two dense matvecs.  Meant for problems
// up to kDirectMaxFree free DOFs (the matrix and its inverse factor held dense).
#include <vector>

#include "common.cuh"
#include "elemop.cuh"
#include "mgkern.cuh"

constexpr int kDirectMaxFree = 20480;

struct pf_direct {
    const pf::Op* op = nullptr;
    pf::Dense dense;
    double* K0 = nullptr;  // device copy of the element matrix
    double* bf = nullptr;  // free right-hand side / intermediate
    double* xf = nullptr;
    int n = 0;
    double* band = nullptr;  // tiles of the two halves, then their right-hand sides and the window
    int* fail = nullptr;     // inside `band`
};

namespace pf {

// row thread: free DOF r = global DOF g; M[r][f(gc)] += E_e K0[a*dof + comp][b*dof + c]
template <int DIM>
__global__ void k_direct_assemble(Grid g, const double* __restrict__ E, const double* __restrict__ K0,
                                  const int* __restrict__ free_dofs, const int* __restrict__ dof_to_free, int n,
                                  int np, double* __restrict__ M) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    constexpr int NC = DIM == 3 ? 8 : 4, ND = NC * DIM;
    const int gdof = free_dofs[r];
    const int node = gdof / DIM, comp = gdof - node * DIM;
    int i, j, k = 0;
    if (DIM == 3) {
        const int t = node / g.nn[2];
        k = node - t * g.nn[2];
        j = t / g.nn[0];
        i = t - j * g.nn[0];
    } else {
        j = node / g.nn[0];
        i = node - j * g.nn[0];
    }
    double* row = M + (long long)r * np;
    for (int a = 0; a < NC; a++) {  // the row node is corner a of element (i, j, k) - corner(a)
        const int ei = i - kCXd(a), ej = j - kCYd(a), ek = DIM == 3 ? k - kCZd(a) : 0;
        if (ei < 0 || ej < 0 || ei >= g.nel[0] || ej >= g.nel[1]) continue;
        if (DIM == 3 && (ek < 0 || ek >= g.nel[2])) continue;
        const long long e = DIM == 3 ? ((long long)ei * g.nel[1] + ej) * g.nel[2] + ek : (long long)ei * g.nel[1] + ej;
        const double w = E[e];
        const double* Kr = K0 + (a * DIM + comp) * ND;
        for (int b = 0; b < NC; b++) {
            const int bi = ei + kCXd(b), bj = ej + kCYd(b), bk = DIM == 3 ? ek + kCZd(b) : 0;
            const long long bn = DIM == 3 ? (long long)bk + (long long)g.nn[2] * (bi + (long long)g.nn[0] * bj)
                                           : (long long)bi + (long long)g.nn[0] * bj;
            for (int c = 0; c < DIM; c++) {
                const int fc = dof_to_free[bn * DIM + c];
                if (fc >= 0) row[fc] += w * Kr[b * DIM + c];
            }
        }
    }
}

__global__ void k_gather(int n, const int* __restrict__ idx, const double* __restrict__ src, double* __restrict__ dst) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) dst[r] = src[idx[r]];
}
__global__ void k_scatter(int n, const int* __restrict__ idx, const double* __restrict__ src, double* __restrict__ dst) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) dst[idx[r]] = src[r];
}

// y = L^-1 b: warp per row, lower triangle only
__global__ void __launch_bounds__(256) k_lower_matvec(const double* __restrict__ Li, int np, int n,
                                                      const double* __restrict__ b, double* __restrict__ y) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), l = threadIdx.x & 31;
    if (row >= n) return;
    const double* Lr = Li + (long long)row * np;
    double s = 0.0;
    for (int c = l; c <= row; c += 32) s += Lr[c] * b[c];
    s = warp_sum(s);
    if (l == 0) y[row] = s;
}

// x = L^-T y: warp per group of 32 columns, coalesced rows i >= column
__global__ void __launch_bounds__(256) k_lower_tmatvec(const double* __restrict__ Li, int np, int n,
                                                       const double* __restrict__ y, double* __restrict__ x) {
    const int grp = blockIdx.x * 8 + (threadIdx.x >> 5), l = threadIdx.x & 31;
    const int col = grp * 32 + l;
    if (grp * 32 >= n) return;
    double s = 0.0;
    for (int i = grp * 32; i < n; i++)
        if (col < n && i >= col) s += Li[(long long)i * np + col] * y[i];
    if (col < n) x[col] = s;
}

// ---------------------------------------------------------------------------------------
// banded solve
// ---------------------------------------------------------------------------------------
// Positions: node (i, j[, k]) numbered with the longest axis slowest, DOF = position * dim +
// component; N positions padded to nt tiles of 32.  Tiles [0, c) are half 0, tiles
// [c + BW, nt) half 1, whose local order is reversed (position N' - 1 - g), and the BW tiles
// between them are the window that both halves' eliminations reach: the two CTAs of a cluster
// eliminate their halves at the same time, CTA 0 adds the two Schur complements, factors the
// window and solves it, and both substitute back.  Local block row i of a half holds the
// tiles (i, i - d), d = 0 .. BW.
struct BandGeom {
    int nt, c, BW;
    int nn[3], ord[3];  // nodes per axis; axes from the slowest to the fastest
    int dim, ndof;
    long long half1;    // tile offset of half 1
};

__host__ __device__ inline int band_rows(const BandGeom& g, int h) { return (h ? g.nt - g.c : g.c + g.BW); }
// node indices at[] of position p (node position * dim + component), and its DOF
__device__ __forceinline__ int band_dof(const BandGeom& g, int p, int (&at)[3]) {
    int rem = p / g.dim;
    for (int a = g.dim - 1; a >= 0; a--) {
        at[g.ord[a]] = rem % g.nn[g.ord[a]];
        rem /= g.nn[g.ord[a]];
    }
    const int node = g.dim == 3 ? at[2] + g.nn[2] * (at[0] + g.nn[0] * at[1]) : at[0] + g.nn[0] * at[1];
    return node * g.dim + p % g.dim;
}
// position of component 0 of the node at m[]
__device__ __forceinline__ int band_pos(const BandGeom& g, const int (&m)[3]) {
    int node = 0;
    for (int a = 0; a < g.dim; a++) node = node * g.nn[g.ord[a]] + m[g.ord[a]];
    return node * g.dim;
}
// entry of a right-hand side (half 0, then half 1) that holds the solution at a position
__device__ __forceinline__ int band_at(const BandGeom& g, int gp) {
    return gp < (g.c + g.BW) * 32 ? gp : band_rows(g, 0) * 32 + g.nt * 32 - 1 - gp;
}

// one thread per (half, local row, neighbour node): the dim entries of that row's DOF
template <int DIM>
__global__ void k_band_assemble(BandGeom g, Grid gr, const double* __restrict__ E, const double* __restrict__ K0,
                                const int* __restrict__ dof_to_free, const double* __restrict__ b, double* __restrict__ band,
                                double* __restrict__ rhs) {
    constexpr int NC = DIM == 3 ? 8 : 4, ND = NC * DIM, NB = DIM == 3 ? 27 : 9;
    const int r0 = band_rows(g, 0) * 32, r1 = band_rows(g, 1) * 32;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nb = (int)(t % NB);
    int q = (int)(t / NB);
    if (q >= r0 + r1) return;
    const int h = q >= r0;
    q -= h * r0;
    const int gp = h ? g.nt * 32 - 1 - q : q;  // global position
    const bool window = gp >= g.c * 32 && gp < (g.c + g.BW) * 32;
    double* tiles = band + (h ? g.half1 : 0) * 1024;
    auto put = [&](int ql, double v) {  // entry (q, ql), ql <= q
        const int i = q >> 5, d = i - (ql >> 5);
        tiles[((long long)i * (g.BW + 1) + d) * 1024 + (q & 31) * 32 + (ql & 31)] = v;
    };
    int at[3] = {0, 0, 0};
    const int dof = gp < g.ndof ? band_dof(g, gp, at) : -1;
    const bool free = dof >= 0 && dof_to_free[dof] >= 0;
    if (nb == NB / 2) rhs[h * r0 + q] = (free && !(window && h)) ? b[dof] : 0.0;
    if (!free) {
        if (nb == NB / 2) put(q, (window && h) ? 0.0 : 1.0);
        return;
    }
    const int o[3] = {nb % 3 - 1, (nb / 3) % 3 - 1, DIM == 3 ? nb / 9 - 1 : 0};
    int m[3];
    for (int a = 0; a < DIM; a++) {
        m[a] = at[a] + o[a];
        if (m[a] < 0 || m[a] >= g.nn[a]) return;
    }
    const int comp = gp % DIM;
    double v[3] = {0.0, 0.0, 0.0};
    for (int ca = 0; ca < NC; ca++) {  // the row node is corner ca of element at - corner(ca)
        const int cx[3] = {kCXd(ca), kCYd(ca), DIM == 3 ? kCZd(ca) : 0};
        int e[3];
        bool in = true;
        int cb = -1;
        for (int a = 0; a < DIM; a++) {
            e[a] = at[a] - cx[a];
            if (e[a] < 0 || e[a] >= gr.nel[a]) in = false;
            const int l = cx[a] + o[a];
            if (l < 0 || l > 1) in = false;
        }
        if (!in) continue;
        for (int k = 0; k < NC; k++)
            if (kCXd(k) == cx[0] + o[0] && kCYd(k) == cx[1] + o[1] && (DIM == 2 || kCZd(k) == cx[2] + o[2])) cb = k;
        const long long ei = DIM == 3 ? ((long long)e[0] * gr.nel[1] + e[1]) * gr.nel[2] + e[2] : (long long)e[0] * gr.nel[1] + e[1];
        const double w = E[ei];
        for (int k = 0; k < DIM; k++) v[k] += w * K0[(ca * DIM + comp) * ND + cb * DIM + k];
    }
    const int p0 = band_pos(g, m);
    for (int k = 0; k < DIM; k++) {
        const int gc = p0 + k;
        if (dof_to_free[band_dof(g, gc, m)] < 0) continue;
        const int ql = h ? g.nt * 32 - 1 - gc : gc;
        if (ql > q || ql < 0) continue;
        if (window && h && gc >= g.c * 32 && gc < (g.c + g.BW) * 32) continue;  // the window's own entries: half 0
        put(ql, v[k]);
    }
}

constexpr int kBP = 36;             // row pitch of a tile in shared memory (conflict-free MMA fragments)
constexpr int kBTile = 32 * kBP;
constexpr int kLP = 34;             // column pitch of the diagonal factor

// C (32 x 32) -= A B^T on the 8 rows of strip s and columns [8 n0, 8 (n0 + NB)): one warp,
// 8 x 8 x 4 FP64 MMAs
template <int NB>
__device__ __forceinline__ void band_strip(double* C, const double* A, const double* B, int s, int n0) {
    const int l = threadIdx.x & 31, r = l >> 2, k = l & 3;
    C += (8 * s + r) * kBP + 8 * n0 + 2 * k;
    A += (8 * s + r) * kBP + k;
    B += (8 * n0 + r) * kBP + k;
    double c[NB][2];
#pragma unroll
    for (int n = 0; n < NB; n++) {
        const double2 v = *reinterpret_cast<const double2*>(C + 8 * n);
        c[n][0] = v.x, c[n][1] = v.y;
    }
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
        const double a = -A[kk];
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const double b = B[8 * n * kBP + kk];
            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                : "+d"(c[n][0]), "+d"(c[n][1])
                : "d"(a), "d"(b));
        }
    }
#pragma unroll
    for (int n = 0; n < NB; n++) *reinterpret_cast<double2*>(C + 8 * n) = make_double2(c[n][0], c[n][1]);
}

// 1 / sqrt(v) without branches, for 1e-280 < v < 1e280: the hardware's estimate (about 2^-22)
// and two Newton steps y += y/2 (1 - v y^2)
__device__ __forceinline__ double band_rsqrt(double v) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
#pragma unroll
    for (int i = 0; i < 2; i++) y = fma(0.5 * y, fma(-v * y, y, 1.0), y);
    return y;
}

// diagonal tile by the plain column loop in shared memory (one warp; D is overwritten): pivots
// out of band_rsqrt's range, and the report of one that is not positive
__device__ __noinline__ void band_potrf_careful(double* D, double* L, double* ri, int* first_bad) {
    const int l = threadIdx.x & 31;
    int bad = -1;
    for (int j = 0; j < 32; j++) {
        double piv = D[j * kBP + j];
        if (!(piv > 0.0)) {
            if (bad < 0) bad = j;
            piv = 1.0;
        }
        const double s = sqrt(piv), lj = l == j ? s : l > j ? D[l * kBP + j] / s : 0.0;
        __syncwarp();
        if (l >= j) L[j * kLP + l] = lj;
        if (l == j) ri[j] = 1.0 / s;
        __syncwarp();
        for (int k = j + 1; k < 32; k++) D[l * kBP + k] -= lj * L[j * kLP + k];
        __syncwarp();
    }
    *first_bad = bad;
}

// Bound by the chain over the columns: one reciprocal square root, shuffle and FMA per column
// of the longer half, about 7,500 cycles per block column (a diagonal tile with the library's
// branching rsqrt took 12,000).  60x20 elements (2562 DOFs, 40 block columns a half): 310 us in
// this kernel, 508 us per solve with the host's preparation, against 10,870 us for the dense
// factor and its inverse.  8 warps; per block column: warp 0 factors the diagonal tile while the
// others finish the previous column's updates, then warp w solves the tile below by w + 1
// (and one warp the right-hand side), then all update the next diagonal tile.
// FACTORED: the band holds the factor, and only the two substitutions run (65 us, bound by the loads
// of each step's tiles from L2; two steps ahead instead of one 53 us, but 324 us in the other form).
// The correction with it: 60 problems of 24x8 to 120x40 elements, contrast up to 1e9, error of the
// solution against long double 3.3e-12 -> 4e-16 (geometric mean; the dense form 1.9e-12), 446 -> 508 us.
template <int BW, bool FACTORED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, 1)
    k_band_solve(BandGeom g, double* __restrict__ band, double* __restrict__ rhs, double* __restrict__ win,
                 const int* __restrict__ dof_to_free, int* fail) {
    extern __shared__ __align__(16) double s_t[];  // (BW + 1)^2 tiles: ring of block rows
    __shared__ __align__(16) double s_L[2][32 * kLP];
    __shared__ double s_ri[2][32], s_b[BW + 1][32], s_z[2][32], s_red[8][32], s_x[BW + 1][32];
    constexpr int R = BW + 1;
    const int h = blockIdx.x, tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int rows = band_rows(g, h), nf = rows - BW;  // block rows; block columns of this half alone
    double* tiles = band + (h ? g.half1 : 0) * 1024;
    double* b = rhs + (h ? band_rows(g, 0) * 32 : 0);
    auto slot = [&](int i, int d) { return s_t + ((i % R) * R + d) * kBTile; };
    double pre[4 * R];  // block row on its way to shared memory: 4 values of each tile
    double preb = 0.0;
    auto fetch = [&](int i) {
        if (i >= rows) return;
#pragma unroll
        for (int d = 0; d < R; d++)
            if (d <= i) {
#pragma unroll
                for (int q = 0; q < 4; q++) pre[d * 4 + q] = tiles[((long long)i * R + d) * 1024 + q * 256 + tid];
            }
        if (tid < 32) preb = b[i * 32 + tid];
    };
    auto place = [&](int i) {
        if (i >= rows) return;
#pragma unroll
        for (int d = 0; d < R; d++)
            if (d <= i) {
#pragma unroll
                for (int q = 0; q < 4; q++) slot(i, d)[(q * 8 + w) * kBP + l] = pre[d * 4 + q];
            }
        if (tid < 32) s_b[i % R][tid] = preb;
    };
    // updates of block column p other than that of tile (p + 1, p + 1), by warps w0 .. 7
    auto rest = [&](int p, int last) {
        int job = 0;
        for (int i = p + 1; i <= p + BW && i < last; i++) {
            for (int k = p + 1; k <= i; k++) {
                if (i == p + 1) continue;
                for (int s = 0; s < 4; s++, job++)
                    if (job % 7 == w - 1) band_strip<4>(slot(i, i - k), slot(i, i - p), slot(k, k - p), s, 0);
            }
            if (job++ % 7 == w - 1) {  // right-hand side
                const double* L = slot(i, i - p) + l * kBP;
                double v = s_b[i % R][l];
#pragma unroll 8
                for (int q = 0; q < 32; q++) v = fma(-L[q], s_z[p & 1][q], v);
                s_b[i % R][l] = v;
            }
        }
    };
    // inverse of the diagonal factor of column p into its place in the band (lane: column)
    auto invert = [&](int p) {
        const double* L = s_L[p & 1];
        double x[32];
#pragma unroll
        for (int r = 0; r < 32; r++) x[r] = r == l ? 1.0 : 0.0;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            x[j] *= s_ri[p & 1][j];
#pragma unroll
            for (int r = j + 1; r < 32; r++) x[r] = fma(-L[j * kLP + r], x[j], x[r]);
        }
        double* out = tiles + (long long)p * R * 1024;
#pragma unroll
        for (int r = 0; r < 32; r++) out[r * 32 + l] = x[r];
    };
    // one block column; `last`: end of the block rows that exist for it
    auto column = [&](int p, int last, bool deferred) {
        if (w == 0) {
            double* D = slot(p, 0);
            double v[32];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const double2 t = *reinterpret_cast<const double2*>(D + l * kBP + j);
                v[j] = t.x, v[j + 1] = t.y;
            }
            double* L = s_L[p & 1];
            double own = 1.0, rown = 1.0, piv = __shfl_sync(0xffffffffu, v[0], 0);
#pragma unroll
            for (int j = 0; j < 32; j++) {
                const double ri = band_rsqrt(piv), lj = v[j] * ri;
                if (l == j) own = piv, rown = ri;
                // the next pivot is complete in lane j + 1: its reciprocal root overlaps the updates
                if (j < 31) piv = __shfl_sync(0xffffffffu, fma(-lj, lj, v[j < 31 ? j + 1 : 31]), j + 1);
                if (l >= j) L[j * kLP + l] = lj;
                __syncwarp();
#pragma unroll
                for (int k = j + 1; k < 32; k++) v[k] = fma(-lj, L[j * kLP + k], v[k]);
            }
            s_ri[p & 1][l] = rown;
            if (!__all_sync(0xffffffffu, own > 1e-280 && own < 1e280)) {
                __syncwarp();
                int bad;
                band_potrf_careful(D, L, s_ri[p & 1], &bad);
                if (bad >= 0 && l == 0) {  // the failing free DOF (1-based)
                    const int gp = h ? g.nt * 32 - 1 - (p * 32 + bad) : p * 32 + bad;
                    int at[3];
                    atomicCAS(fail, 0, gp < g.ndof ? dof_to_free[band_dof(g, gp, at)] + 1 : 1);
                }
            }
        } else if (deferred) {
            rest(p - 1, last);
        }
        __syncthreads();
        // the tiles below, and the right-hand side as one more row
        if (w < BW && p + 1 + w < last) {
            double* X = slot(p + 1 + w, 1 + w) + l * kBP;
            double v[32];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const double2 t = *reinterpret_cast<const double2*>(X + j);
                v[j] = t.x, v[j + 1] = t.y;
            }
            const double* L = s_L[p & 1];
#pragma unroll
            for (int j = 0; j < 32; j++) {
                v[j] *= s_ri[p & 1][j];
#pragma unroll
                for (int k = j + 1; k < 32; k++) v[k] = fma(-v[j], L[j * kLP + k], v[k]);
            }
            double* out = tiles + ((long long)(p + 1 + w) * R + 1 + w) * 1024 + l * 32;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const double2 t = make_double2(v[j], v[j + 1]);
                *reinterpret_cast<double2*>(X + j) = t;
                *reinterpret_cast<double2*>(out + j) = t;
            }
        } else if (w == BW) {
            // lane j holds entry j; the solved entries come by shuffle
            const double* L = s_L[p & 1];
            double v = s_b[p % R][l], z = 0.0;
#pragma unroll 8
            for (int j = 0; j < 32; j++) {
                const double zj = __shfl_sync(0xffffffffu, v, j) * s_ri[p & 1][j];
                if (l == j) z = zj;
                if (l > j) v = fma(-L[j * kLP + l], zj, v);
            }
            s_z[p & 1][l] = z;
            b[p * 32 + l] = z;
        } else if (w == 7) {
            invert(p);
        }
        __syncthreads();
        if (p + R < rows) place(p + R);  // into the ring row of block row p, which is finished
        if (p + 1 < last) band_strip<2>(slot(p + 1, 0), slot(p + 1, 1), slot(p + 1, 1), w >> 1, 2 * (w & 1));
        fetch(p + R + 1);
        __syncthreads();
    };
    auto cluster_sync = [&]() {
        __threadfence();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    };
    double tl[BW][4], li[4], zl = 0.0;  // tiles of the substitutions' next step, loaded one step ahead
    if constexpr (FACTORED) {
        // forward: z_p = L_pp^-1 (r_p - sum_d L_p,(p-d) z_(p-d)); warp w takes rows 4 w .. 4 w + 3, its lanes the
        // columns
        double* part = win + BW * R * 1024;  // half 1's share of the window, reversed order
        auto row_sums = [&](const double (&v)[4]) {  // valid for row 4 w + ((l >> 3) & 3) of the warp
            const bool h16 = l & 16, h8 = l & 8;
            const double a = (h16 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16);
            const double c = (h16 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16);
            double t = (h8 ? c : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : c, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            return t;
        };
        const int row = w * 4 + ((l >> 3) & 3);
        auto ahead = [&](int p, int end) {
            if (p >= end) return;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                li[q] = tiles[(long long)p * R * 1024 + (w * 4 + q) * 32 + l];
#pragma unroll
                for (int d = 1; d <= BW; d++)
                    tl[d - 1][q] = p >= d ? tiles[((long long)p * R + d) * 1024 + (w * 4 + q) * 32 + l] : 0.0;
            }
            zl = b[p * 32 + row];
            if (h == 0 && p >= nf) zl += __ldcg(part + BW * 32 - 1 - ((p - nf) * 32 + row));
        };
        auto known = [&](int p, int dmin) {  // sum over d >= dmin of this lane's column
            double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int d = 1; d <= BW; d++)
                if (d >= dmin && p >= d) {
                    const double z = s_x[(p - d) % R][l];
#pragma unroll
                    for (int q = 0; q < 4; q++) v[q] = fma(tl[d - 1][q], z, v[q]);
                }
            return row_sums(v);
        };
        auto forward = [&](int p, int end) {
            const double r = zl - known(p, 1);
            double v[4];
            if ((l & 7) == 0) s_z[0][row] = r;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = li[q] * s_z[0][l];
            ahead(p + 1, end);
            const double z = row_sums(v);
            if ((l & 7) == 0) s_x[p % R][row] = z, b[p * 32 + row] = z;
            __syncthreads();
        };
        ahead(0, nf);
        for (int p = 0; p < nf; p++) forward(p, nf);
        if (h == 1) {
            for (int i = 0; i < BW; i++) {
                const int p = nf + i;
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int d = 1; d <= BW; d++)
                        tl[d - 1][q] = p >= d ? tiles[((long long)p * R + d) * 1024 + (w * 4 + q) * 32 + l] : 0.0;
                const double v = known(p, i + 1);
                if ((l & 7) == 0) part[i * 32 + row] = -v;
            }
        }
        cluster_sync();
        if (h == 0) {
            ahead(nf, rows);
            for (int p = nf; p < rows; p++) forward(p, rows);
        }
        __syncthreads();
    } else {
    for (int i = 0; i < R; i++) {
        fetch(i);
        place(i);
    }
    fetch(R);
    __syncthreads();
    for (int p = 0; p < nf; p++) column(p, rows, p > 0);
    if (nf > 0) {
        if (w > 0) rest(nf - 1, rows);
        __syncthreads();
    }
    // half 1 hands its window over (lower triangle and right-hand side, reversed order)
    if (h == 1) {
        for (int i = 0; i < BW; i++) {
            for (int d = 0; d <= i; d++)
                for (int q = 0; q < 4; q++)
                    win[(i * R + d) * 1024 + q * 256 + tid] = slot(nf + i, d)[(q * 8 + w) * kBP + l];
            if (tid < 32) win[BW * R * 1024 + i * 32 + tid] = s_b[(nf + i) % R][tid];
        }
    }
    cluster_sync();
    if (h == 0) {
        constexpr int NW = BW * 32;
        for (int i = 0; i < BW; i++) {
            for (int d = 0; d <= i; d++)
                for (int q = 0; q < 4; q++) {
                    const int r = q * 8 + w, ra = i * 32 + r, ca = (i - d) * 32 + l;
                    if (ca > ra) continue;
                    // reversed: row NW - 1 - ca >= column NW - 1 - ra
                    const int rr = NW - 1 - ca, cr = NW - 1 - ra;
                    slot(nf + i, d)[r * kBP + l] += __ldcg(win + ((rr >> 5) * R + (rr >> 5) - (cr >> 5)) * 1024 + (rr & 31) * 32 + (cr & 31));
                }
            if (tid < 32) {
                const int rr = NW - 1 - (i * 32 + tid);
                s_b[(nf + i) % R][tid] += __ldcg(win + BW * R * 1024 + rr);
            }
        }
        __syncthreads();
        for (int p = nf; p < rows; p++) column(p, rows, p > nf);
    }
    }  // factorisation
    // back substitution: x_p = L_pp^-T (z_p - sum_d L_(p+d),p^T x_(p+d))
    auto ahead = [&](int p) {
        if (p < 0) return;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            li[q] = __ldcg(tiles + (long long)p * R * 1024 + (w * 4 + q) * 32 + l);
#pragma unroll
            for (int d = 1; d <= BW; d++)
                tl[d - 1][q] = p + d < rows ? __ldcg(tiles + ((long long)(p + d) * R + d) * 1024 + (w * 4 + q) * 32 + l) : 0.0;
        }
        if (w == 0) zl = __ldcg(b + p * 32 + l);
    };
    auto back = [&](int p) {
        double s = 0.0, lc[4];
#pragma unroll
        for (int d = 1; d <= BW; d++)
            if (p + d < rows) {
#pragma unroll
                for (int q = 0; q < 4; q++) s = fma(tl[d - 1][q], s_x[(p + d) % R][w * 4 + q], s);
            }
        double z = zl;
#pragma unroll
        for (int q = 0; q < 4; q++) lc[q] = li[q];
        s_red[w][l] = s;
        ahead(p - 1);
        __syncthreads();
        if (w == 0) {
#pragma unroll
            for (int q = 0; q < 8; q++) z -= s_red[q][l];
            s_z[0][l] = z;
        }
        __syncthreads();
        s = 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) s = fma(lc[q], s_z[0][w * 4 + q], s);
        s_red[w][l] = s;
        __syncthreads();
        if (w == 0) {
            double x = 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++) x += s_red[q][l];
            s_x[p % R][l] = x;
            b[p * 32 + l] = x;
        }
        __syncthreads();
    };
    if (h == 0) {
        ahead(rows - 1);
        for (int p = rows - 1; p >= nf; p--) back(p);
        for (int i = tid; i < BW * 32; i += 256) win[i] = s_x[(nf + (i >> 5)) % R][i & 31];
    }
    cluster_sync();
    if (h == 1) {
        for (int i = tid; i < BW * 32; i += 256) s_x[(nf + (i >> 5)) % R][i & 31] = __ldcg(win + BW * 32 - 1 - i);
        ahead(nf - 1);
        __syncthreads();
    }
    for (int p = nf - 1; p >= 0; p--) back(p);
}

// r = b - K x over the free DOFs for the solution x = sol, in pairs of doubles (error-free products and sums), so
// that r is exact to its own last bits; zero for the rows that half 0 or nothing holds.  NC consecutive threads
// share a row, one element each (one thread per row, with the positions by division, took 25 us at 60x20).
template <int DIM>
__global__ void __launch_bounds__(128) k_band_residual(BandGeom g, Grid gr, const double* __restrict__ E, const double* __restrict__ K0,
                                                       const int* __restrict__ dof_to_free, const double* __restrict__ b,
                                                       const double* __restrict__ sol, double* __restrict__ res) {
    constexpr int NC = DIM == 3 ? 8 : 4, ND = NC * DIM;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, q = t / NC, ca = t % NC;
    const int r0 = band_rows(g, 0) * 32, nrow = r0 + band_rows(g, 1) * 32;
    const int gp = q < r0 ? q : g.nt * 32 - 1 - (q - r0);
    int at[3] = {0, 0, 0};
    const int dof = q < nrow && gp < g.ndof ? band_dof(g, gp, at) : -1;
    const bool row = dof >= 0 && dof_to_free[dof] >= 0 && band_at(g, gp) == q;
    auto add = [](double& h, double& l, double v, double ve) {  // (h, l) += (v, ve)
        const double t = __dadd_rn(h, v), z = __dsub_rn(t, h);
        l += __dadd_rn(__dsub_rn(h, __dsub_rn(t, z)), __dsub_rn(v, z)) + ve;
        h = t;
    };
    double hi = row && ca == 0 ? b[dof] : 0.0, lo = 0.0;
    const int e[3] = {at[0] - kCXd(ca), at[1] - kCYd(ca), DIM == 3 ? at[2] - kCZd(ca) : 0};  // the row node is its corner ca
    bool in = row;
    for (int a = 0; a < DIM; a++) in = in && e[a] >= 0 && e[a] < gr.nel[a];
    if (in) {
        int ps[3], m[3] = {1, 1, 1};  // a step along an axis in positions and in DOFs
        for (int a = DIM - 1, st = DIM; a >= 0; a--) {
            ps[g.ord[a]] = st;
            st *= g.nn[g.ord[a]];
        }
        const int ds[3] = {DIM == 3 ? DIM * g.nn[2] : DIM, DIM == 3 ? DIM * g.nn[2] * g.nn[0] : DIM * g.nn[0], DIM};
        const int comp = gp % DIM;
        double sh = 0.0, sl = 0.0;
        for (int cb = 0; cb < NC; cb++) {
            m[0] = kCXd(cb) - kCXd(ca), m[1] = kCYd(cb) - kCYd(ca), m[2] = DIM == 3 ? kCZd(cb) - kCZd(ca) : 0;
            int p0 = gp - comp, d0 = dof - comp;
            for (int a = 0; a < DIM; a++) p0 += m[a] * ps[a], d0 += m[a] * ds[a];
            for (int k = 0; k < DIM; k++) {
                if (dof_to_free[d0 + k] < 0) continue;
                const double kv = K0[(ca * DIM + comp) * ND + cb * DIM + k], xv = sol[band_at(g, p0 + k)], v = __dmul_rn(kv, xv);
                add(sh, sl, v, fma(kv, xv, -v));
            }
        }
        const double w = -E[DIM == 3 ? ((long long)e[0] * gr.nel[1] + e[1]) * gr.nel[2] + e[2] : (long long)e[0] * gr.nel[1] + e[1]];
        const double v = __dmul_rn(w, sh);
        add(hi, lo, v, fma(w, sh, -v) + w * sl);
    }
#pragma unroll
    for (int o = 1; o < NC; o <<= 1) {
        const double h2 = __shfl_xor_sync(0xffffffffu, hi, o), l2 = __shfl_xor_sync(0xffffffffu, lo, o);
        add(hi, lo, h2, l2);
    }
    if (q < nrow && ca == 0) res[q] = hi + lo;
}

// x: free entries from the halves' solutions and their corrections, constrained entries the right-hand side's
__global__ void k_band_scatter(BandGeom g, const int* __restrict__ dof_to_free, const double* __restrict__ sol,
                               const double* __restrict__ cor, const double* b, double* x) {
    const int gp = blockIdx.x * blockDim.x + threadIdx.x;
    if (gp >= g.ndof) return;
    int at[3];
    const int dof = band_dof(g, gp, at), i = band_at(g, gp);
    x[dof] = dof_to_free[dof] >= 0 ? sol[i] + cor[i] : b[dof];
}

// band geometry of a grid; false where the dense solve serves (bandwidth, or a grid that is
// mostly constrained, whose free DOFs alone are the smaller problem)
static bool band_geometry(const Grid& g, int n_free, BandGeom* o) {
    o->dim = g.dim;
    const long long nd = g.n_nodes * g.dof;
    if (nd > 4LL * n_free + 1024) return false;
    o->ndof = (int)nd;
    for (int a = 0; a < 3; a++) o->nn[a] = g.nn[a], o->ord[a] = a;
    for (int i = 0; i < g.dim; i++)
        for (int j = i + 1; j < g.dim; j++)
            if (g.nn[o->ord[j]] > g.nn[o->ord[i]]) {
                const int t = o->ord[i];
                o->ord[i] = o->ord[j];
                o->ord[j] = t;
            }
    long long stride = 1, reach = 0;  // largest position difference of neighbouring nodes
    for (int a = g.dim - 1; a >= 0; a--) {
        reach += stride;
        stride *= g.nn[o->ord[a]];
    }
    const long long hb = reach * g.dim + g.dim - 1;
    const long long bw = (hb + 31) / 32;
    if (bw > 3) return false;
    o->BW = (int)bw;
    o->nt = (o->ndof + 31) / 32;
    if (o->nt < o->BW) o->nt = o->BW;
    o->c = (o->nt - o->BW) / 2;
    o->half1 = (long long)band_rows(*o, 0) * (o->BW + 1);
    return true;
}

static int band_solve(pf_direct* d, const BandGeom& g, const double* E, const int* dof_to_free, const double* b, double* x,
                      cudaStream_t st) {
    const Grid& gr = d->op->grid;
    const long long brows = band_rows(g, 0) + band_rows(g, 1), R = g.BW + 1;
    const long long nt = brows * R * 1024;
    const long long nwin = (g.BW * R * 1024 + g.BW * 32), nrhs = brows * 32;
    // the geometry is the grid's: one allocation for the object's life
    if (!d->band && cudaMalloc(&d->band, sizeof(double) * (nt + 2 * nrhs + nwin + 1)) != cudaSuccess) {
        cudaGetLastError();
        d->band = nullptr;
        return fail(PF_NO_MEMORY, "pf_direct_solve_f64: allocation failed");
    }
    d->fail = reinterpret_cast<int*>(d->band + nt + 2 * nrhs + nwin);
    double *rhs = d->band + nt, *cor = rhs + nrhs, *win = cor + nrhs;
    PF_CUDA(cudaMemsetAsync(d->band, 0, sizeof(double) * nt, st));
    PF_CUDA(cudaMemsetAsync(d->fail, 0, sizeof(int), st));
    count_launch(5);
    const int nb = gr.dim == 3 ? 27 : 9;
    const unsigned blocks = (unsigned)((brows * 32 * nb + 255) / 256);
    if (gr.dim == 3)
        k_band_assemble<3><<<blocks, 256, 0, st>>>(g, gr, E, d->K0, dof_to_free, b, d->band, rhs);
    else
        k_band_assemble<2><<<blocks, 256, 0, st>>>(g, gr, E, d->K0, dof_to_free, b, d->band, rhs);
    PF_LAUNCH_CHECK("band assembly launch");
    auto solve = [&](auto kernel, size_t sm, double* v) {
        if (sm) PF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        kernel<<<2, 256, sm, st>>>(g, d->band, v, win, dof_to_free, d->fail);
        PF_LAUNCH_CHECK("band solve launch");
        return (int)PF_OK;
    };
    const size_t sm = (size_t)R * R * kBTile * sizeof(double);
    int s = g.BW == 1 ? solve(k_band_solve<1, false>, sm, rhs)
          : g.BW == 2 ? solve(k_band_solve<2, false>, sm, rhs) : solve(k_band_solve<3, false>, sm, rhs);
    if (s) return s;
    const unsigned rblocks = (unsigned)((nrhs * (gr.dim == 3 ? 8 : 4) + 127) / 128);
    if (gr.dim == 3)
        k_band_residual<3><<<rblocks, 128, 0, st>>>(g, gr, E, d->K0, dof_to_free, b, rhs, cor);
    else
        k_band_residual<2><<<rblocks, 128, 0, st>>>(g, gr, E, d->K0, dof_to_free, b, rhs, cor);
    PF_LAUNCH_CHECK("band residual launch");
    s = g.BW == 1 ? solve(k_band_solve<1, true>, 0, cor)
      : g.BW == 2 ? solve(k_band_solve<2, true>, 0, cor) : solve(k_band_solve<3, true>, 0, cor);
    if (s) return s;
    k_band_scatter<<<(unsigned)((g.ndof + 255) / 256), 256, 0, st>>>(g, dof_to_free, rhs, cor, b, x);
    PF_LAUNCH_CHECK("direct solve launch");
    return PF_OK;
}

}  // namespace pf

using namespace pf;

extern "C" int pf_direct_create(const pf_op* op, pf_direct** out) {
    if (!op || !out) return fail(PF_BAD_ARG, "pf_direct_create: NULL argument");
    auto* d = new pf_direct();
    d->op = op;
    const int nd = (op->grid.dim == 3 ? 8 : 4) * op->grid.dim;
    if (cudaMalloc(&d->K0, sizeof(double) * nd * nd) != cudaSuccess) {
        delete d;
        return fail(PF_NO_MEMORY, "pf_direct_create: allocation failed");
    }
    if (cudaMemcpy(d->K0, op->K0, sizeof(double) * nd * nd, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(d->K0);
        delete d;
        return fail(PF_CUDA_ERROR, "pf_direct_create: copy of K0 failed");
    }
    *out = d;
    return PF_OK;
}

extern "C" int pf_direct_destroy(pf_direct* d) {
    if (!d) return PF_OK;
    dense_free(&d->dense);
    for (void* p : {(void*)d->K0, (void*)d->bf, (void*)d->xf, (void*)d->band})
        if (p) cudaFree(p);
    delete d;
    return PF_OK;
}

static int direct_reserve(pf_direct* d, int n) {
    if (d->n == n && d->dense.M) return PF_OK;
    dense_free(&d->dense);
    if (d->bf) cudaFree(d->bf);
    if (d->xf) cudaFree(d->xf);
    d->bf = d->xf = nullptr;
    d->n = 0;
    int s = dense_alloc(&d->dense, n);
    if (s) return s;
    if (cudaMalloc(&d->bf, sizeof(double) * n) != cudaSuccess || cudaMalloc(&d->xf, sizeof(double) * n) != cudaSuccess)
        return fail(PF_NO_MEMORY, "pf_direct_solve_f64: allocation failed");
    d->n = n;
    return PF_OK;
}

extern "C" int pf_direct_solve_f64(pf_direct* d, const double* E, const int* free_dofs, const int* dof_to_free,
                                   int n_free, const double* b, double* x, void* stream) {
    if (!d || !E || !free_dofs || !dof_to_free || !b || !x || n_free < 1)
        return fail(PF_BAD_ARG, "pf_direct_solve_f64: bad argument");
    if (n_free > kDirectMaxFree)
        return fail(PF_BAD_ARG, "pf_direct_solve_f64: %d free DOFs exceed the dense direct solver's limit of %d",
                    n_free, kDirectMaxFree);
    cudaStream_t st = as_stream(stream);
    int s;
    BandGeom bg;
    if (band_geometry(d->op->grid, n_free, &bg)) {
        if ((s = band_solve(d, bg, E, dof_to_free, b, x, st))) return s;
        int fpiv = 0;
        PF_CUDA(cudaMemcpyAsync(&fpiv, d->fail, sizeof(int), cudaMemcpyDeviceToHost, st));
        PF_CUDA(cudaStreamSynchronize(st));
        if (fpiv) return fail(PF_FACTOR_FAILED, "pf_direct_solve_f64: matrix not positive definite (pivot %d)", fpiv - 1);
        return PF_OK;
    }
    if ((s = direct_reserve(d, n_free))) return s;
    Dense& D = d->dense;
    const Grid& g = d->op->grid;
    const long long ndof = g.n_nodes * g.dof;
    PF_CUDA(cudaMemsetAsync(D.M, 0, (size_t)D.np * D.np * sizeof(double), st));
    count_launch();
    if (g.dim == 3)
        k_direct_assemble<3><<<(n_free + 127) / 128, 128, 0, st>>>(g, E, d->K0, free_dofs, dof_to_free, n_free, D.np,
                                                                   D.M);
    else
        k_direct_assemble<2><<<(n_free + 127) / 128, 128, 0, st>>>(g, E, d->K0, free_dofs, dof_to_free, n_free, D.np,
                                                                   D.M);
    PF_LAUNCH_CHECK("direct assembly launch");
    if ((s = dense_factor_linv(&D, 0.0, st))) return s;
    // x = b (constrained entries keep the right-hand side), then the free entries
    PF_CUDA(cudaMemcpyAsync(x, b, sizeof(double) * ndof, cudaMemcpyDeviceToDevice, st));
    count_launch(4);
    k_gather<<<(n_free + 255) / 256, 256, 0, st>>>(n_free, free_dofs, b, d->bf);
    k_lower_matvec<<<(n_free + 7) / 8, 256, 0, st>>>(D.Linv, D.np, n_free, d->bf, d->xf);
    k_lower_tmatvec<<<((n_free + 31) / 32 + 7) / 8, 256, 0, st>>>(D.Linv, D.np, n_free, d->xf, d->bf);
    k_scatter<<<(n_free + 255) / 256, 256, 0, st>>>(n_free, free_dofs, d->bf, x);
    PF_LAUNCH_CHECK("direct solve launch");
    int fpiv = 0;
    PF_CUDA(cudaMemcpyAsync(&fpiv, D.fail, sizeof(int), cudaMemcpyDeviceToHost, st));
    PF_CUDA(cudaStreamSynchronize(st));
    if (fpiv) return fail(PF_FACTOR_FAILED, "pf_direct_solve_f64: matrix not positive definite (pivot %d)", fpiv - 1);
    return PF_OK;
}
