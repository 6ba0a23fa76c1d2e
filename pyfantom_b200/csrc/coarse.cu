// Level-1 coarse operator applied element by element (no assembled coefficients).
//
// With trilinear interpolation Phat and the reference's normalised transfers
// R = D Phat^T, P = Phat D, D = diag(1/tw) (pyFANTOM/core/CUDA/Kernels/mgm.cu:1-244), the
// level-1 Galerkin operator is A1 = R (Z K Z + I - Z) P = D A^ D with
//   A^ = sum over coarse elements C of M_C,
//   M_C = sum_c E_{C,c} Kc[c],  Kc[c] = Phat_c^T K0 Phat_c   (C touches no constraint),
// where c runs over the 8 children of C.  Child c is child 0 reflected along the axes of
// its bits, and K0 of a box element is invariant under those reflections, so in the Walsh
// basis of C's corners (v = T u, the basis the fine matvec uses, T K0 T^T / 64 block
// diagonal)
//   T M_C T^T / 64 = B0 o Ehat[p(i) ^ p(j)],   Ehat_k = sum_c E_{C,c} (-1)^{popcount(c & k)},
// with B0 = T Kc[0] T^T / 64 and p(i) the reflection-parity class of Walsh slot i (mode m,
// component a: p = m ^ (1 << a)).  For isotropic box elements B0 has 279 nonzeros (150
// distinct by symmetry) in a fixed pattern, and the rows of the rigid translations (mode 0)
// vanish: one coarse element costs 279 + 150 multiply-adds on 8 precomputed Ehat values
// and no coefficient traffic, where the assembled stencil streams 126 coefficients per
// coarse node.
//
// Coarse elements with a constrained fine node ("dirty") have Z-masked children, and the
// identity rows Phat^T (I - Z) Phat reach the same elements' corners: the rows of these corner
// nodes are taken from the assembled level-1 stencil (which the setup forms for the deeper
// levels) into a compact table.  The march skips them, so what it computes for dirty elements
// (from their unmasked children) is never used, and the warps of all blocks share them out:
// a clamped face puts thousands of them into a few tile columns.  (Explicit 24 x 24 matrices
// inside the march held those columns' blocks back: 53.9 us per FP32 level-1 product of
// 256x128x128 with a clamped face, 30.0 us without one.)  The stiffness rows stay in the
// physical basis, where FP32 resolves the O(E_min) stiffness of void children beside the O(1)
// identity rows to the same relative error as the stencil; in the Walsh basis they would mix.
// Largest FP32 row error over |A1| |u|, contrast 1e9, a clamped face, two pinned lines, random DOFs:
// 1.6e-7 to 2.7e-7 (explicit matrices with the identity rows apart: 2.8e-7 to 7.0e-7).
//
// The matvec is an x-march like the fine one (csrc/elemop.cu): warps cover element rows in
// y, lanes element columns in z, the element's Walsh transform is formed from the two
// faces, D is applied to u on load and to y at the owner, rows are exchanged through
// shared memory once per step; owner computes, no atomics, fixed summation order.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "coarse.cuh"
#include "common.cuh"
#include "elemop.cuh"
#include "mgkern.cuh"

namespace pf {

// coefficient index (0..149) of Walsh entry (i, j), i = m*3 + a, or -1 for a structural zero
// of B0 for isotropic box elements (rows and columns 0..2 are the rigid translations)
__host__ __device__ constexpr int coarse_pat(int i, int j) {
    constexpr int t[24][24] = {
        {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {-1, -1, -1, 0, -1, -1, -1, 1, -1, 2, 3, -1, -1, -1, 4, 5, -1, 6, -1, 7, 8, 9, 10, 11},
        {-1, -1, -1, -1, 12, -1, 13, -1, -1, 14, 15, -1, -1, -1, -1, -1, 16, -1, 17, -1, -1, 18, 19, -1},
        {-1, -1, -1, -1, -1, 20, -1, -1, -1, -1, -1, 21, 22, -1, -1, 23, -1, 24, 25, -1, -1, 26, -1, 27},
        {-1, -1, -1, -1, 13, -1, 28, -1, -1, 29, 30, -1, -1, -1, -1, -1, 31, -1, 32, -1, -1, 33, 34, -1},
        {-1, -1, -1, 1, -1, -1, -1, 35, -1, 36, 37, -1, -1, -1, 38, 39, -1, 40, -1, 41, 42, 43, 44, 45},
        {-1, -1, -1, -1, -1, -1, -1, -1, 46, -1, -1, 47, -1, 48, -1, -1, 49, -1, -1, 50, 51, -1, 52, 53},
        {-1, -1, -1, 2, 14, -1, 29, 36, -1, 54, 55, -1, -1, -1, 56, 57, 58, 59, 60, 61, 62, 63, 64, 65},
        {-1, -1, -1, 3, 15, -1, 30, 37, -1, 55, 66, -1, -1, -1, 67, 68, 69, 70, 71, 72, 73, 74, 75, 76},
        {-1, -1, -1, -1, -1, 21, -1, -1, 47, -1, -1, 77, 78, 79, -1, 80, 81, 82, 83, 84, 85, 86, 87, 88},
        {-1, -1, -1, -1, -1, 22, -1, -1, -1, -1, -1, 78, 89, -1, -1, 90, -1, 91, 92, -1, -1, 93, -1, 94},
        {-1, -1, -1, -1, -1, -1, -1, -1, 48, -1, -1, 79, -1, 95, -1, -1, 96, -1, -1, 97, 98, -1, 99, 100},
        {-1, -1, -1, 4, -1, -1, -1, 38, -1, 56, 67, -1, -1, -1, 101, 102, -1, 103, -1, 104, 105, 106, 107, 108},
        {-1, -1, -1, 5, -1, 23, -1, 39, -1, 57, 68, 80, 90, -1, 102, 109, -1, 110, 111, 112, 113, 114, 115, 116},
        {-1, -1, -1, -1, 16, -1, 31, -1, 49, 58, 69, 81, -1, 96, -1, -1, 117, -1, 118, 119, 120, 121, 122, 123},
        {-1, -1, -1, 6, -1, 24, -1, 40, -1, 59, 70, 82, 91, -1, 103, 110, -1, 124, 125, 126, 127, 128, 129, 130},
        {-1, -1, -1, -1, 17, 25, 32, -1, -1, 60, 71, 83, 92, -1, -1, 111, 118, 125, 131, -1, -1, 132, 133, 134},
        {-1, -1, -1, 7, -1, -1, -1, 41, 50, 61, 72, 84, -1, 97, 104, 112, 119, 126, -1, 135, 136, 137, 138, 139},
        {-1, -1, -1, 8, -1, -1, -1, 42, 51, 62, 73, 85, -1, 98, 105, 113, 120, 127, -1, 136, 140, 141, 142, 143},
        {-1, -1, -1, 9, 18, 26, 33, 43, -1, 63, 74, 86, 93, -1, 106, 114, 121, 128, 132, 137, 141, 144, 145, 146},
        {-1, -1, -1, 10, 19, -1, 34, 44, 52, 64, 75, 87, -1, 99, 107, 115, 122, 129, 133, 138, 142, 145, 147, 148},
        {-1, -1, -1, 11, -1, 27, -1, 45, 53, 65, 76, 88, 94, 100, 108, 116, 123, 130, 134, 139, 143, 146, 148, 149},
    };
    return t[i][j];
}
constexpr int kCoarseCoefs = 150;
// reflection-parity class of Walsh slot i = m*3 + a
__host__ __device__ constexpr int wclass(int i) { return (i / 3) ^ (1 << (i % 3)); }
// Walsh slot of component a in class q
__host__ __device__ constexpr int wslot(int q, int a) { return (q ^ (1 << a)) * 3 + a; }

template <typename T>
struct CoarseCoef {
    T b[kCoarseCoefs];
};

// compile-time unrolled loop: f(std::integral_constant<int, 0>) ... f(<N-1>)
template <int N>
struct Unroll {
    template <typename F>
    __device__ __forceinline__ static void run(F&& f) {
        Unroll<N - 1>::run(f);
        f(std::integral_constant<int, N - 1>{});
    }
};
template <>
struct Unroll<0> {
    template <typename F>
    __device__ __forceinline__ static void run(F&&) {}
};

static int host_walsh(int m, int l) {
    const int pos[3] = {kCXd(l), kCYd(l), kCZd(l)};
    int s = 1;
    for (int a = 0; a < 3; a++)
        if ((m >> a) & 1) s *= pos[a] ? 1 : -1;
    return s;
}

// B0 = T Kc[0] T^T / 64 checked against the pattern; PF_UNSUPPORTED if K0 does not have it
int coarse_factorise(const Op* op, double* coef /* [150] */) {
    if (op->grid.dim != 3) return fail(PF_UNSUPPORTED, "element-level coarse operator: 3D only");
    std::vector<double> Kc(8 * 24 * 24);
    galerkin_child_matrices(3, op->K0, Kc.data());
    const double* K = Kc.data();  // child 0 (lowest corner)
    double B[24][24], tmp[24][24];
    for (int i = 0; i < 24; i++)
        for (int j = 0; j < 24; j++) {
            double s = 0.0;
            for (int l = 0; l < 8; l++) s += host_walsh(i / 3, l) * K[(l * 3 + i % 3) * 24 + j];
            tmp[i][j] = s;
        }
    double bmax = 0.0;
    for (int i = 0; i < 24; i++)
        for (int j = 0; j < 24; j++) {
            double s = 0.0;
            for (int l = 0; l < 8; l++) s += tmp[i][l * 3 + j % 3] * host_walsh(j / 3, l);
            B[i][j] = s / 64.0;
            bmax = fmax(bmax, fabs(B[i][j]));
        }
    const double tol = 1e-12 * bmax;
    for (int q = 0; q < kCoarseCoefs; q++) coef[q] = 0.0;
    for (int i = 0; i < 24; i++)
        for (int j = 0; j < 24; j++) {
            const int q = coarse_pat(i, j);
            if (q < 0) {
                if (fabs(B[i][j]) > tol)
                    return fail(PF_UNSUPPORTED, "coarse operator: K0 lacks the isotropic-box structure (%d,%d)", i, j);
            } else {
                if (fabs(B[i][j] - B[j][i]) > tol) return fail(PF_UNSUPPORTED, "coarse operator: B0 not symmetric");
                coef[q] = B[i][j];
            }
        }
    return PF_OK;
}

// ---------------------------------------------------------------------------------------
// setup: Ehat, rows of the nodes next to constraints
// ---------------------------------------------------------------------------------------
constexpr int kScanThreads = 1024;  // flags per block of the compaction

// Stream compaction of a flag array in index order, in two passes: block b counts the
// flags of items [1024 b, 1024 (b + 1)); then every block adds the counts of the blocks
// before it and places its items with a ballot scan.  list[rank] = i (rank < cap; list may be
// NULL), *count = number of flagged items.
__global__ void __launch_bounds__(kScanThreads) k_flag_count(long long n, const uint8_t* __restrict__ flag,
                                                             int* __restrict__ bcount) {
    const long long i = (long long)blockIdx.x * kScanThreads + threadIdx.x;
    const int c = __syncthreads_count(i < n && flag[i]);
    if (threadIdx.x == 0) bcount[blockIdx.x] = c;
}

__global__ void __launch_bounds__(kScanThreads) k_flag_compact(long long n, const uint8_t* __restrict__ flag,
                                                               const int* __restrict__ bcount, int* __restrict__ list,
                                                               int cap, int* __restrict__ count) {
    __shared__ int s_w[kScanThreads / 32];
    __shared__ int s_base;
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    // base: the flagged items of all earlier blocks
    int acc = 0;
    for (int b = t; b < (int)blockIdx.x; b += kScanThreads) acc += bcount[b];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (l == 0) s_w[w] = acc;
    __syncthreads();
    if (t == 0) {
        int sum = 0;
        for (int q = 0; q < kScanThreads / 32; q++) sum += s_w[q];
        s_base = sum;
    }
    __syncthreads();
    const long long i = (long long)blockIdx.x * kScanThreads + t;
    const bool f = i < n && flag[i];
    const unsigned m = __ballot_sync(0xffffffffu, f);
    s_w[w] = __popc(m);  // s_w is free again after the barrier above
    __syncthreads();
    int before = 0;
    for (int q = 0; q < w; q++) before += s_w[q];
    const int r = s_base + before + __popc(m & ((1u << l) - 1u));
    if (i < n && list && f && r < cap) list[r] = (int)i;
    if (blockIdx.x == gridDim.x - 1 && t == kScanThreads - 1) {
        int tot = 0;
        for (int q = 0; q < kScanThreads / 32; q++) tot += s_w[q];
        *count = s_base + tot;
    }
}

static int flag_compact(long long n, const uint8_t* flag, int* bcount, int* list, int cap, int* count, cudaStream_t st) {
    const unsigned nb = (unsigned)((n + kScanThreads - 1) / kScanThreads);
    pf::count_launch(2);
    k_flag_count<<<nb, kScanThreads, 0, st>>>(n, flag, bcount);
    k_flag_compact<<<nb, kScanThreads, 0, st>>>(n, flag, bcount, list, cap, count);
    PF_LAUNCH_CHECK("flag compaction launch");
    return PF_OK;
}

// Ehat of every coarse element, element-major Eh[e * 8 + k] (one 32-byte (FP32) or 64-byte
// (FP64) run per element, read with vector loads)
template <typename T>
__global__ void k_coarse_ehat(int NXc, int NYc, int NZc, const double* __restrict__ E, T* __restrict__ Eh) {
    const long long ne = (long long)NXc * NYc * NZc;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int ez = (int)(e % NZc), ey = (int)((e / NZc) % NYc), ex = (int)(e / ((long long)NZc * NYc));
    const int NYf = 2 * NYc, NZf = 2 * NZc;
    double c[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int fx = 2 * ex + (q & 1), fy = 2 * ey + ((q >> 1) & 1), fz = 2 * ez + ((q >> 2) & 1);
        c[q] = E[((long long)fx * NYf + fy) * NZf + fz];
    }
    // 8-point Walsh-Hadamard transform over the child bits (x = bit 0)
#pragma unroll
    for (int b = 1; b < 8; b <<= 1)
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (!(q & b)) {
                const double lo = c[q], hi = c[q | b];
                c[q] = lo + hi;
                c[q | b] = lo - hi;
            }
#pragma unroll
    for (int q = 0; q < 8; q++) Eh[e * 8 + q] = (T)c[q];
}

// coarse nodes that are corners of a dirty element
__global__ void k_corner_flags(int NXc, int NYc, int NZc, const uint8_t* __restrict__ elem_flag,
                               uint8_t* __restrict__ nflag) {
    const int nx = NXc + 1, nz = NZc + 1;
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (long long)nx * (NYc + 1) * nz) return;
    const unsigned t = (unsigned)n / nz;
    const int k = (int)((unsigned)n - t * nz), j = (int)(t / nx), i = (int)(t - (unsigned)j * nx);
    uint8_t f = 0;
    for (int q = 0; q < 8; q++) {
        const int ex = i - kCXd(q), ey = j - kCYd(q), ez = k - kCZd(q);
        if (ex >= 0 && ey >= 0 && ez >= 0 && ex < NXc && ey < NYc && ez < NZc)
            f |= elem_flag[((long long)ex * NYc + ey) * NZc + ez];
    }
    nflag[n] = f;
}

// S[q * 243 + e] = stencil entry e (neighbour, row, column component) of node nlist[q]
template <typename T>
__global__ void __launch_bounds__(256) k_flag_rows(long long N, const double* __restrict__ A, const int* __restrict__ nlist,
                                                   int nq, T* __restrict__ S) {
    // threads along q: reads of consecutive nodes coalesce; written through shared memory
    __shared__ T s_v[27][33];
    const int q0 = blockIdx.x * 32, l = threadIdx.x & 31, w = threadIdx.x >> 5, e0 = blockIdx.y * 27;
    const long long n = q0 + l < nq ? nlist[q0 + l] : -1;
    for (int e = w; e < 27; e += 8) s_v[e][l] = n >= 0 ? (T)A[(long long)(e0 + e) * N + n] : T(0);
    __syncthreads();
    for (int q = w; q < 32; q += 8)
        if (q0 + q < nq && l < 27) S[(long long)(q0 + q) * 243 + e0 + l] = s_v[l][q];
}

// ---------------------------------------------------------------------------------------
// matvec: register x-march over coarse elements
// ---------------------------------------------------------------------------------------

template <typename T>
__device__ __forceinline__ T inv_tw(int n, int nn) {
    return (n == 0 || n == nn - 1) ? T(1.0 / 1.5) : T(0.5);
}

// Element operator in the Walsh basis.  glo / ghi: transformed lower / upper faces; eh: the
// element's Ehat.  G receives the lower-face outputs plus the carry of the previous element;
// carry the upper-face outputs.
template <typename T>
__device__ __forceinline__ void coarse_element(const T (&glo)[3][2][2], const T (&ghi)[3][2][2], const T (&eh)[8],
                                               const CoarseCoef<T>& cf, T (&carry)[3][2][2], T (&G)[3][2][2]) {
    T v[24];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int ym = 0; ym < 2; ym++)
#pragma unroll
            for (int zm = 0; zm < 2; zm++) {
                v[((0 | (ym << 1) | (zm << 2)) * 3) + a] = ghi[a][ym][zm] + glo[a][ym][zm];
                v[((1 | (ym << 1) | (zm << 2)) * 3) + a] = ghi[a][ym][zm] - glo[a][ym][zm];
            }
    // outputs slot by slot (component a, y-mode, z-mode; x-modes 0 and 1), folded into G
    Unroll<12>::run([&](auto S) {
        constexpr int slot = decltype(S)::value;
        constexpr int a = slot / 4, ym = (slot >> 1) & 1, zm = slot & 1;
        T zx[2];
        Unroll<2>::run([&](auto X) {
            constexpr int xm = decltype(X)::value;
            constexpr int i = ((xm | (ym << 1) | (zm << 2)) * 3) + a;
            T acc = T(0);
            if constexpr (i >= 3) {
                Unroll<8>::run([&](auto K) {
                    constexpr int k = decltype(K)::value;
                    constexpr int q = wclass(i) ^ k;
                    constexpr int j0 = wslot(q, 0), j1 = wslot(q, 1), j2 = wslot(q, 2);
                    constexpr int c0 = coarse_pat(i, j0), c1 = coarse_pat(i, j1), c2 = coarse_pat(i, j2);
                    if constexpr (c0 >= 0 || c1 >= 0 || c2 >= 0) {
                        T t = T(0);
                        if constexpr (c0 >= 0) t = fma(cf.b[c0 < 0 ? 0 : c0], v[j0], t);
                        if constexpr (c1 >= 0) t = fma(cf.b[c1 < 0 ? 0 : c1], v[j1], t);
                        if constexpr (c2 >= 0) t = fma(cf.b[c2 < 0 ? 0 : c2], v[j2], t);
                        acc = fma(eh[k], t, acc);
                    }
                });
            }
            zx[xm] = acc;
        });
        G[a][ym][zm] = (zx[0] - zx[1]) + carry[a][ym][zm];
        carry[a][ym][zm] = zx[0] + zx[1];
    });
}

// RW element rows per warp: lanes are RW segments of L = 32 / RW along z (shuffles of width L),
// so a z-tile owns L - 2 node columns; RW = 2 wastes fewer lanes when the level's z extent
// is just above a multiple of 30 (level 1 of a 256x128x128 grid: 65 node columns).
template <typename T, int NW, int MINB, int MODE, int RW>
__global__ void __launch_bounds__(NW * 32, MINB)
    k_coarse_matvec(int NX, int NY, int NZ, int CXc, const T* __restrict__ u, const T* __restrict__ Eh,
                    const CoarseCoef<T> cf, Epi<T> epi, const uint8_t* __restrict__ nflag,
                    const int* __restrict__ nlist, const int* __restrict__ nlisted, const T* __restrict__ S) {
    pdl_wait();
    pdl_trigger();
    constexpr int L = 32 / RW, NR = NW * RW, TY = NR - 1;  // lanes per row, rows, owned rows
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ T s_q[2][3][NR][L];
    const int nq = nflag ? *nlisted : 0, done = epi.skip ? *epi.skip : 0;
    if (done) return;
    constexpr bool need_b = MODE != PF_EPI_STORE, need_x = MODE == PF_EPI_JACOBI || MODE == PF_EPI_JACOBI_ADD;
    constexpr bool need_xa = MODE == PF_EPI_JACOBI_ADD;
    const int nx = NX + 1, ny = NY + 1, nz = NZ + 1;
    const int tid = threadIdx.x, w = (tid >> 5) * RW + (tid & 31) / L, l = tid % L;  // w: row, l: lane in row
    const int kz0 = blockIdx.x * (L - 2), jy0 = blockIdx.y * TY, ix0 = blockIdx.z * CXc;
    const int je = jy0 - 1 + w, kc = kz0 - 1 + l;
    const bool col_ok = kc >= 0 && kc < nz;
    const bool ok0 = col_ok && je >= 0 && je < ny, ok1 = col_ok && je + 1 < ny;
    const bool elem_ok = l < L - 1 && je >= 0 && je < NY && kc >= 0 && kc < NZ;
    const bool owner = w < TY && l < L - 2 && je + 1 < ny && kc + 1 < nz;
    const int rows = nz * nx;
    const int n0 = kc + rows * je;
    const int n1 = n0 + rows;
    const int eplane = NY * NZ;
    const int e0 = je * NZ + kc;
    // D = diag(1/tw): per-axis factors of this lane's node column and the two node rows
    const T sz = inv_tw<T>(kc, nz), sy0 = inv_tw<T>(je, ny), sy1 = inv_tw<T>(je + 1, ny);
    const T s0 = sz * sy0, s1 = sz * sy1;
    const T so = inv_tw<T>(kc + 1, nz) * sy1;  // owned node (je + 1, kc + 1), without x
    const T wgt = epi_omega(epi);

    // rows of the nodes next to constraints, one warp each: lane o < 27 takes neighbour o
    if (nflag) {
        const int gl = tid & 31;
        const int nwarp = gridDim.x * gridDim.y * gridDim.z * NW;
        for (int q = (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)) * NW + (tid >> 5); q < nq; q += nwarp) {
            const int n = nlist[q];
            const unsigned tz = (unsigned)n / nz;
            const int k = (int)((unsigned)n - tz * nz), j = (int)(tz / nx), i = (int)(tz - (unsigned)j * nx);
            const int mi = i + gl % 3 - 1, mj = j + (gl / 3) % 3 - 1, mk = k + gl / 9 - 1;
            T acc[3] = {T(0), T(0), T(0)};
            if (gl < 27 && mi >= 0 && mj >= 0 && mk >= 0 && mi < nx && mj < ny && mk < nz) {
                const T* um = u + 3 * ((long long)mk + (long long)nz * (mi + (long long)nx * mj));
                const T* Sq = S + (long long)q * 243 + gl * 9;
                const T u0 = um[0], u1 = um[1], u2 = um[2];
#pragma unroll
                for (int c = 0; c < 3; c++) acc[c] = fma(Sq[3 * c], u0, fma(Sq[3 * c + 1], u1, Sq[3 * c + 2] * u2));
            }
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(FULL, acc[c], o);
            if (gl < 3) epi.out[3 * n + gl] = epi_apply(epi, 3 * n + gl, gl == 0 ? acc[0] : gl == 1 ? acc[1] : acc[2], wgt);
        }
    }

    auto load = [&](int p, T (&v)[2][3]) {
        const bool pok = p >= 0 && p < nx;
        const int a0 = n0 + nz * p, a1 = n1 + nz * p;
        const T sx = pok ? inv_tw<T>(p, nx) : T(0);
        if (pok && ok0) {
#pragma unroll
            for (int c = 0; c < 3; c++) v[0][c] = u[3 * a0 + c] * (sx * s0);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) v[0][c] = T(0);
        }
        if (pok && ok1) {
#pragma unroll
            for (int c = 0; c < 3; c++) v[1][c] = u[3 * a1 + c] * (sx * s1);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) v[1][c] = T(0);
        }
    };
    auto face = [&](const T (&v)[2][3], T (&g)[3][2][2]) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const T s = v[1][c] + v[0][c], dd = v[1][c] - v[0][c];
            const T sn = __shfl_down_sync(FULL, s, 1, L), dn = __shfl_down_sync(FULL, dd, 1, L);
            g[c][0][0] = s + sn;
            g[c][0][1] = sn - s;
            g[c][1][0] = dd + dn;
            g[c][1][1] = dn - dd;
        }
    };
    auto eload = [&](int ie, T (&eh)[8]) {
        const bool ok = elem_ok && ie >= 0 && ie < NX;
        const long long e = (long long)e0 + (long long)eplane * ie;
        if (ok) {
            if constexpr (sizeof(T) == 4) {
                const float4* p = reinterpret_cast<const float4*>(Eh + e * 8);
                const float4 a = p[0], b = p[1];
                eh[0] = a.x, eh[1] = a.y, eh[2] = a.z, eh[3] = a.w;
                eh[4] = b.x, eh[5] = b.y, eh[6] = b.z, eh[7] = b.w;
            } else {
                const double2* p = reinterpret_cast<const double2*>(Eh + e * 8);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double2 a = p[k];
                    eh[2 * k] = a.x, eh[2 * k + 1] = a.y;
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) eh[k] = T(0);
        }
    };

    T carry[3][2][2];
    auto step = [&](int s, T (&gl)[3][2][2], T (&gh)[3][2][2], T (&v)[2][3], T (&eh)[8]) {
        const int ie = ix0 - 1 + s;
        face(v, gh);
        if (s < CXc) load(ie + 2, v);
        const int no = n1 + 1 + nz * ie;
        bool out_now = owner && s >= 1 && ie < nx;
        T G[3][2][2];
        coarse_element<T>(gl, gh, eh, cf, carry, G);
        if (s < CXc) eload(ie + 1, eh);
        T pb[3], px[3], pd[3], pa[3];
        uint8_t nf = 0;
        if (out_now) {
            if (nflag) nf = nflag[no];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                if constexpr (need_b) pb[c] = epi.b[3 * no + c];
                if constexpr (need_x) px[c] = epi.x[3 * no + c];
                if constexpr (need_x) pd[c] = epi.dinv[3 * no + c];
                if constexpr (need_xa) pa[c] = epi.xadd[3 * no + c];
            }
        }
        T P1[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const T r0a = G[c][0][0] - G[c][1][0], r0b = G[c][0][1] - G[c][1][1];
            const T r1a = G[c][0][0] + G[c][1][0], r1b = G[c][0][1] + G[c][1][1];
            const T lo0 = r0a - r0b, up0 = r0a + r0b, lo1 = r1a - r1b, up1 = r1a + r1b;
            P1[c] = up1 + __shfl_down_sync(FULL, lo1, 1, L);
            s_q[s & 1][c][w][l] = up0 + __shfl_down_sync(FULL, lo0, 1, L);
        }
        __syncthreads();
        if (out_now && !nf) {
            const T sc = so * inv_tw<T>(ie, nx);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const T y = (P1[c] + s_q[s & 1][c][w + 1][l]) * sc;
                T o = y;
                if constexpr (MODE == PF_EPI_RESID) {
                    o = pb[c] - y;
                } else if constexpr (MODE == PF_EPI_JACOBI) {
                    o = px[c] + wgt * pd[c] * (pb[c] - y);
                } else if constexpr (MODE == PF_EPI_JACOBI_ADD) {
                    o = pa[c] + px[c] + wgt * pd[c] * (pb[c] - y);
                }
                epi.out[3 * no + c] = o;
            }
        }
    };

    T gA[3][2][2], gB[3][2][2];
    T vA[2][3];
    T eh[8];
    load(ix0 - 1, vA);
    face(vA, gA);
    load(ix0, vA);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++) carry[c][a][b] = T(0);
    eload(ix0 - 1, eh);
    for (int s = 0; s <= CXc; s++) {
        step(s, gA, gB, vA, eh);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int b = 0; b < 2; b++) gA[c][a][b] = gB[c][a][b];
    }
}

// FP64: 8 warps, 1 block per SM (the operator holds 24 Walsh values and 8 Ehat in
// registers); FP32: 8 warps, 2 blocks per SM (measured: 74.7 us per 256x128x128 level-1
// launch against 81.9 us for one block of 16 warps, whose halo rows are fewer but whose
// step barrier holds all 16 warps)
template <typename T>
struct CoarseShape {  // warps per block (NW - 1 owned element rows) and blocks per SM
    static constexpr int NW = 8;
    static constexpr int MINB = sizeof(T) == 4 ? 2 : 1;
};

// element rows per warp (1 or 2): the one with fewer warp-rows of lanes per x-plane
template <typename T>
static int coarse_rows_per_warp(const Grid& g) {
    if (sizeof(T) != 4) return 1;
    constexpr int NW = CoarseShape<T>::NW;
    long long best = -1;
    int pick = 1;
    for (int rw = 1; rw <= 2; rw++) {
        const int L = 32 / rw, nr = NW * rw;
        const long long cost = (long long)((g.nn[2] + L - 3) / (L - 2)) * ((g.nn[1] + nr - 2) / (nr - 1)) * NW;
        if (best < 0 || cost < best) {
            best = cost;
            pick = rw;
        }
    }
    return pick;
}

template <typename T>
static void coarse_launch_dims(const Grid& g, dim3* grid, int* CXc, int rw) {
    constexpr int NW = CoarseShape<T>::NW;
    const int ny = g.nn[1], nz = g.nn[2], nx = g.nn[0];
    const int L = 32 / rw, nr = NW * rw;
    const int tz = (nz + L - 3) / (L - 2), ty = (ny + nr - 2) / (nr - 1);
    const long long slots = (long long)kNumSM * CoarseShape<T>::MINB;
    const long long cols = (long long)tz * ty;
    int best = 2;
    long long best_cost = -1;
    for (int cx = 2; cx <= 64; cx++) {
        const long long nb = cols * ((nx + cx - 1) / cx);
        const long long cost = ((nb + slots - 1) / slots) * (cx + 1);
        if (best_cost < 0 || cost <= best_cost) {
            best_cost = cost;
            best = cx;
        }
    }
    *CXc = best;
    *grid = dim3(tz, ty, (nx + best - 1) / best);
}

template <typename T, int MODE, int RW>
static int coarse_launch(dim3 grid, int cx, const Grid& g, const T* u, const CoarseOp* c, const CoarseCoef<T>& cf,
                         const Epi<T>& epi, cudaStream_t st) {
    constexpr int NW = CoarseShape<T>::NW, MINB = CoarseShape<T>::MINB;
    const uint8_t* nflag = c->nrows > 0 ? c->nflag : nullptr;
    PF_CUDA(launch_pdl(k_coarse_matvec<T, NW, MINB, MODE, RW>, grid, dim3(NW * 32), 0, st, g.nel[0], g.nel[1],
                       g.nel[2], cx, u, (const T*)c->Eh, cf, epi, nflag, (const int*)c->nlist,
                       (const int*)(c->count + 1), (const T*)c->S));
    return PF_OK;
}

template <typename T>
int launch_coarse_matvec(const CoarseOp* c, const Grid& g, const T* u, const Epi<T>& epi, cudaStream_t st) {
    if (epi.dot_partial) return fail(PF_UNSUPPORTED, "coarse element matvec: no fused dot");
    CoarseCoef<T> cf;
    for (int q = 0; q < kCoarseCoefs; q++) cf.b[q] = (T)c->coef[q];
    const int rw = coarse_rows_per_warp<T>(g);
    dim3 grid;
    int cx;
    coarse_launch_dims<T>(g, &grid, &cx, rw);
    pf::count_launch();
#define PF_COARSE(M)                                                               \
    return rw == 2 ? coarse_launch<T, M, sizeof(T) == 4 ? 2 : 1>(grid, cx, g, u, c, cf, epi, st) \
                   : coarse_launch<T, M, 1>(grid, cx, g, u, c, cf, epi, st)
    switch (epi.mode) {
        case PF_EPI_STORE:
            PF_COARSE(PF_EPI_STORE);
        case PF_EPI_RESID:
            PF_COARSE(PF_EPI_RESID);
        case PF_EPI_JACOBI:
            PF_COARSE(PF_EPI_JACOBI);
        default:
            PF_COARSE(PF_EPI_JACOBI_ADD);
    }
#undef PF_COARSE
}
template int launch_coarse_matvec<double>(const CoarseOp*, const Grid&, const double*, const Epi<double>&,
                                          cudaStream_t);
template int launch_coarse_matvec<float>(const CoarseOp*, const Grid&, const float*, const Epi<float>&,
                                         cudaStream_t);

// ---------------------------------------------------------------------------------------
// object lifetime and setup
// ---------------------------------------------------------------------------------------
static int calloc_dev(void** p, size_t bytes) {
    if (cudaMalloc(p, bytes ? bytes : 8) != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return fail(PF_NO_MEMORY, "device allocation of %zu bytes failed", bytes);
    }
    return PF_OK;
}

int coarse_create(const Op* op, int fp32, CoarseOp** out) {
    *out = nullptr;
    CoarseOp* c = new CoarseOp();
    int s = coarse_factorise(op, c->coef);
    if (s) {
        cudaGetLastError();
        delete c;
        return s;
    }
    c->fine = op->grid;
    c->g = coarse_grid(op->grid);
    c->tsize = fp32 ? 4 : 8;
    const long long ne = c->g.n_elem;
    s = calloc_dev(&c->Eh, (size_t)ne * 8 * c->tsize);
    s = s ? s : calloc_dev((void**)&c->nflag, (size_t)c->g.n_nodes);
    s = s ? s : calloc_dev((void**)&c->count, 2 * sizeof(int));
    {
        const long long nmax = ne > c->g.n_nodes ? ne : c->g.n_nodes;
        s = s ? s : calloc_dev((void**)&c->bcount, (size_t)((nmax + kScanThreads - 1) / kScanThreads) * sizeof(int));
    }
    if (!s && cudaMallocHost((void**)&c->h_count, 2 * sizeof(int)) != cudaSuccess) s = fail(PF_NO_MEMORY, "pinned alloc");
    if (s) {
        coarse_destroy(c);
        return s;
    }
    *out = c;
    return PF_OK;
}

void coarse_destroy(CoarseOp* c) {
    if (!c) return;
    for (void* p : {c->Eh, (void*)c->count, (void*)c->nflag, (void*)c->nlist, c->S, (void*)c->bcount})
        if (p) cudaFree(p);
    if (c->h_count) cudaFreeHost(c->h_count);
    delete c;
}

// Ehat for densities E (FP64), and the assembled rows (level-1 stencil A64) of the nodes next to
// constraints.  These are recounted on every call; the host waits for the counts (two ints) and
// grows the rows' storage when they no longer fit.  *realloc: launches captured before are stale.
int coarse_setup(CoarseOp* c, const double* E, const uint8_t* mask, const uint8_t* elem_flag, const double* A64,
                 cudaStream_t st, bool* realloc) {
    *realloc = false;
    const Grid& gc = c->g;
    const long long ne = gc.n_elem;
    if (ne >= (1LL << 31) || gc.n_nodes >= (1LL << 31)) return fail(PF_BAD_ARG, "coarse grid too large");
    int nd = 0, ni = 0;
    if (mask) {
        pf::count_launch();
        k_corner_flags<<<(unsigned)((gc.n_nodes + 255) / 256), 256, 0, st>>>(gc.nel[0], gc.nel[1], gc.nel[2], elem_flag,
                                                                           c->nflag);
        for (int pass = 0; pass < 2; pass++) {
            int s = pass ? (int)PF_OK : flag_compact(ne, elem_flag, c->bcount, nullptr, 0, c->count, st);
            s = s ? s : flag_compact(gc.n_nodes, c->nflag, c->bcount, c->nlist, c->cap, c->count + 1, st);
            if (s) return s;
            PF_CUDA(cudaMemcpyAsync(c->h_count, c->count, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
            PF_CUDA(cudaStreamSynchronize(st));
            nd = c->h_count[0];
            ni = c->h_count[1];
            if (nd >= (1 << 24)) return fail(PF_UNSUPPORTED, "coarse operator: %d dirty elements (limit 2^24)", nd);
            if (ni <= c->cap) break;
            for (void* p : {(void*)c->nlist, c->S})
                if (p) cudaFree(p);
            c->nlist = nullptr;
            c->S = nullptr;
            c->cap = 0;
            const int cap = ni + ni / 4 + 32;
            s = calloc_dev((void**)&c->nlist, (size_t)cap * sizeof(int));
            s = s ? s : calloc_dev(&c->S, (size_t)cap * 243 * c->tsize);
            if (s) return s;
            c->cap = cap;
            *realloc = true;
        }
    }
    if ((ni > 0) != (c->nrows > 0)) *realloc = true;  // a launch bakes in whether there are such rows
    c->nrows = ni;
    c->ndirty = nd;
    const unsigned nb = (unsigned)((ne + 255) / 256);
    pf::count_launch();
    if (c->tsize == 4)
        k_coarse_ehat<float><<<nb, 256, 0, st>>>(gc.nel[0], gc.nel[1], gc.nel[2], E, (float*)c->Eh);
    else
        k_coarse_ehat<double><<<nb, 256, 0, st>>>(gc.nel[0], gc.nel[1], gc.nel[2], E, (double*)c->Eh);
    PF_LAUNCH_CHECK("coarse ehat launch");
    if (ni > 0) {
        pf::count_launch();
        const dim3 gr((unsigned)((ni + 31) / 32), 9);
        if (c->tsize == 4)
            k_flag_rows<float><<<gr, 256, 0, st>>>(gc.n_nodes, A64, c->nlist, ni, (float*)c->S);
        else
            k_flag_rows<double><<<gr, 256, 0, st>>>(gc.n_nodes, A64, c->nlist, ni, (double*)c->S);
        PF_LAUNCH_CHECK("constrained rows launch");
    }
    return PF_OK;
}

}  // namespace pf
