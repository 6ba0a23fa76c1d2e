// Cone density filter on a structured element grid (forward H x and exact adjoint H^T v).
//
// Reference: apply_filter_2D/3D_kernel, get_filter_2D/3D_weights_kernel and
// apply_filter_2D/3D_transpose_kernel (pyFANTOM/core/CUDA/Kernels/filters.cu:1-154):
//   forward  y_e = sum_k w_k x_{e+o_k} / sum_k w_k      (sums over in-bounds taps only)
//   norm_e   = sum over in-bounds taps of w_k
//   adjoint  s_e = sum_k (w_k / norm_{e+o_k}) v_{e+o_k} (the offset set is symmetric)
//
// k_filter_tile serves the cone filters (every column of taps along x is an unbroken,
// symmetric run): a block stages its tile and halo in shared memory (zeros outside the
// mesh) and each thread computes RI outputs along x, so a staged value read into a register
// serves up to 2m + 1 taps.  Away from the mesh faces the normaliser is one constant, which
// is divided into the weights once; only elements next to a face divide by their own (the
// adjoint when they are staged), instead of one division per tap.  k_filter
// (one thread per element, taps read from global memory, in the reference order) forms the
// normaliser and serves any other set of taps.
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace pf {
// the tap columns as kernel parameters (uniform loads): cone filters up to rmin 3
constexpr int kTapCols = 32, kTapWeights = 128;
struct FilterTaps {
    int4 col[kTapCols];
    double w[kTapWeights];
};
}  // namespace pf

struct pf_filter {
    pf::Grid grid;
    int n_taps;
    void* d_mem;       // the allocation that holds the arrays below
    int* d_off;        // n_taps x dim
    double* d_w;       // n_taps
    double* d_norm;    // n_elem normaliser
    // tap columns of k_filter_tile (ncol = 0: the taps are not columns; k_filter)
    int ncol;
    int* d_col;        // ncol x 4: dj, dk, half length along x, first weight
    double* d_cw;      // weights over norm_in, column by column
    int rad[3];        // largest offset along x, y, z (2D: 0, x, y)
    double norm_in;    // normaliser of an element all of whose taps are inside
    pf::FilterTaps taps;
};

namespace pf {

constexpr int kMaxTaps = 2048;  // keeps the staged tap table under 48 KB of shared memory

template <int DIM, int MODE>  // MODE 0 forward, 1 adjoint, 2 normaliser
__global__ void __launch_bounds__(256) k_filter(int nelx, int nely, int nelz, int K, const int* __restrict__ off,
                                                const double* __restrict__ w, const double* __restrict__ norm,
                                                const double* __restrict__ x, double* __restrict__ y) {
    extern __shared__ unsigned char smem[];
    double* s_w = reinterpret_cast<double*>(smem);
    int* s_o = reinterpret_cast<int*>(s_w + K);
    for (int t = threadIdx.x; t < K; t += blockDim.x) {
        s_w[t] = w[t];
        for (int a = 0; a < DIM; a++) s_o[t * DIM + a] = off[t * DIM + a];
    }
    __syncthreads();
    const long long ne = DIM == 3 ? (long long)nelx * nely * nelz : (long long)nelx * nely;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    int i, j, k = 0;
    const unsigned ue = (unsigned)e;  // element counts stay below 2^31 (validate_grid)
    if (DIM == 3) {
        const unsigned t = ue / (unsigned)nelz;
        k = (int)(ue - t * (unsigned)nelz);
        i = (int)(t / (unsigned)nely);
        j = (int)(t - (unsigned)i * (unsigned)nely);
    } else {
        i = (int)(ue / (unsigned)nely);
        j = (int)(ue - (unsigned)i * (unsigned)nely);
    }
    double sv = 0.0, sw = 0.0;
    for (int t = 0; t < K; t++) {
        const int a = i + s_o[t * DIM], b = j + s_o[t * DIM + 1], c = DIM == 3 ? k + s_o[t * DIM + 2] : 0;
        if (a < 0 || a >= nelx || b < 0 || b >= nely) continue;
        if (DIM == 3 && (c < 0 || c >= nelz)) continue;
        const long long jd = DIM == 3 ? ((long long)a * nely + b) * nelz + c : (long long)a * nely + b;
        if (MODE == 0) {
            sv += s_w[t] * x[jd];
            sw += s_w[t];
        } else if (MODE == 1) {
            sv += (s_w[t] / norm[jd]) * x[jd];
        } else {
            sw += s_w[t];
        }
    }
    if (MODE == 0)
        y[e] = sw > 0 ? sv / sw : 0.0;
    else if (MODE == 1)
        y[e] = sv;
    else
        y[e] = sw;
}

// ---------------------------------------------------------------------------------------
// tiled filter
// ---------------------------------------------------------------------------------------
struct FilterTile {
    int nx, ny, nz;     // elements (2D: nx = 1)
    int ri, rj, rk;     // radii
    int tj, tk;         // tiles along y and z
    int ncol, nw;
    double norm_in;
};

// one column of taps (2m + 1 along x) applied to RI consecutive outputs
template <int RI, int M>
__device__ __forceinline__ void filter_column(const double* s, int plane, const double* w, double (&acc)[RI]) {
    double v[RI + 2 * M];
#pragma unroll
    for (int r = 0; r < RI + 2 * M; r++) v[r] = s[r * plane];
#pragma unroll
    for (int t = 0; t <= 2 * M; t++) {
        const double wt = w[t];
#pragma unroll
        for (int r = 0; r < RI; r++) acc[r] = fma(wt, v[r + t], acc[r]);
    }
}

// Block: 256 threads, TK columns along z by 256 / TK along y, RI elements along x each.
// With 27 taps an output costs 9 (RI + 2) / RI shared-memory reads and 27 FMAs.  No unit is at its
// limit (ncu, 256x128x128, rmin 2: issue 61 to 63 % of the cycles, shared memory 41 %, FP64 pipe 22 %,
// DRAM 12 %); the warps, 34 to 40 per SM, mostly wait for the loads that stage the tile, which nothing
// but other blocks' arithmetic covers.  256x128x128, rmin 2, forward and adjoint together:
// 76.4 us against 367 us for k_filter; 96x48x48: 14.2 against 29.7 us.  Staging by division-free
// rows rather than by a flat index took 108 to 97 us, the constant normaliser in the weights 97 to
// 90 us, the tap table in the kernel's parameters (uniform loads instead of shared-memory ones)
// and eight staging loads in flight 90 to 76 us.
template <int RI, int MI, int TK, bool ADJ>
__global__ void __launch_bounds__(256) k_filter_tile(const FilterTile t, const __grid_constant__ FilterTaps tap,
                                                     const int4* __restrict__ col, const double* __restrict__ cw,
                                                     const double* __restrict__ norm, const double* __restrict__ x,
                                                     double* __restrict__ y) {
    pdl_wait();
    pdl_trigger();
    constexpr bool TAB = MI > 2;  // tap table in shared memory instead of the kernel's parameters
    constexpr int TJ = 256 / TK;
    extern __shared__ __align__(16) double s_f[];
    const int SJ = TJ + 2 * t.rj, SK = TK + 2 * t.rk, plane = SJ * SK, SI = RI + 2 * t.ri;
    double* s_w = s_f + SI * plane;
    int4* s_c = reinterpret_cast<int4*>(s_w + ((t.nw + 1) & ~1));
    const int tid = threadIdx.x, tk = tid % TK, tj = tid / TK;
    const unsigned b = blockIdx.x, bt = b / t.tk;
    const int k0 = (int)(b - bt * t.tk) * TK, j0 = (int)(bt % t.tj) * TJ, i0 = (int)(bt / t.tj) * RI;
    if constexpr (TAB) {
        for (int q = tid; q < t.nw; q += 256) s_w[q] = cw[q];
        for (int q = tid; q < t.ncol; q += 256) s_c[q] = col[q];
    }
    // elements with the interior normaliser (already in the weights); `inner`: all staged ones
    auto is_in = [&](int i, int j, int k) {
        return i >= t.ri && i < t.nx - t.ri && j >= t.rj && j < t.ny - t.rj && k >= t.rk && k < t.nz - t.rk;
    };
    const bool inner = i0 >= 2 * t.ri && i0 + RI + 2 * t.ri <= t.nx && j0 >= 2 * t.rj && j0 + TJ + 2 * t.rj <= t.ny &&
                       k0 >= 2 * t.rk && k0 + TK + 2 * t.rk <= t.nz;
    // stage: thread (tj, tk) takes column tk of every TJ-th row of the tile, then the last
    // 2 rk columns of all rows are shared out
    auto stage = [&](int a, int bj, int c) {
        const int i = i0 + a - t.ri, j = j0 + bj - t.rj, k = k0 + c - t.rk;
        double v = 0.0;
        if ((unsigned)i < (unsigned)t.nx && (unsigned)j < (unsigned)t.ny && (unsigned)k < (unsigned)t.nz) {
            const int e = (i * t.ny + j) * t.nz + k;  // fewer than 2^31 elements (validate_grid)
            v = x[e];
            if (ADJ && !inner && !is_in(i, j, k)) v = v * t.norm_in / norm[e];
        }
        s_f[(a * SJ + bj) * SK + c] = v;
    };
    const int rows = SI * SJ;
    {
        int a = 0, bj = tj;
#pragma unroll 8
        for (int r = tj; r < rows; r += TJ) {
            stage(a, bj, tk);
            bj += TJ;
            if (bj >= SJ) bj -= SJ, a++;
        }
    }
    for (int q = tid; q < rows * 2 * t.rk; q += 256) {
        const int r = q / (2 * t.rk), a = r / SJ;
        stage(a, r - a * SJ, TK + q - r * 2 * t.rk);
    }
    __syncthreads();
    const int j = j0 + tj, k = k0 + tk;
    if (j >= t.ny || k >= t.nz) return;
    double acc[RI];
#pragma unroll
    for (int r = 0; r < RI; r++) acc[r] = 0.0;
    const double* base = s_f + (tj + t.rj) * SK + tk + t.rk;
    for (int c = 0; c < t.ncol; c++) {
        const int4 cc = TAB ? s_c[c] : tap.col[c];
        const double* sc = base + (t.ri - cc.z) * plane + cc.x * SK + cc.y;
        const double* wc = TAB ? s_w + cc.w : tap.w + cc.w;
        if (cc.z == 0) filter_column<RI, 0>(sc, plane, wc, acc);
        if constexpr (RI > 1 && MI >= 1)
            if (cc.z == 1) filter_column<RI, 1>(sc, plane, wc, acc);
        if constexpr (RI > 1 && MI >= 2)
            if (cc.z == 2) filter_column<RI, 2>(sc, plane, wc, acc);
        if constexpr (RI > 1 && MI >= 4) {
            if (cc.z == 3) filter_column<RI, 3>(sc, plane, wc, acc);
            if (cc.z == 4) filter_column<RI, 4>(sc, plane, wc, acc);
        }
    }
#pragma unroll
    for (int r = 0; r < RI; r++) {
        const int i = i0 + r;
        if (i >= t.nx) break;
        const int e = (i * t.ny + j) * t.nz + k;
        double v = acc[r];
        if (!ADJ && !is_in(i, j, k)) {
            const double nv = norm[e];
            v = nv > 0 ? v * t.norm_in / nv : 0.0;
        }
        y[e] = v;
    }
}

constexpr size_t kFilterMaxSmem = 160 * 1024;
static size_t filter_tile_smem(const FilterTile& t, int RI, int TK) {
    return ((size_t)(RI + 2 * t.ri) * (256 / TK + 2 * t.rj) * (TK + 2 * t.rk) + ((t.nw + 1) & ~1)) * sizeof(double) +
           (size_t)t.ncol * sizeof(int4);
}

template <int RI, int MI, int TK, bool ADJ>
static int launch_filter_tile(const pf_filter* f, FilterTile t, const double* x, double* y, cudaStream_t st) {
    constexpr int TJ = 256 / TK;
    t.tk = (t.nz + TK - 1) / TK;
    t.tj = (t.ny + TJ - 1) / TJ;
    const long long nb = (long long)t.tk * t.tj * ((t.nx + RI - 1) / RI);
    const size_t sm = filter_tile_smem(t, RI, TK);
    if (sm > 48 * 1024)
        PF_CUDA(cudaFuncSetAttribute(k_filter_tile<RI, MI, TK, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kFilterMaxSmem));
    count_launch();
    PF_CUDA(launch_pdl(k_filter_tile<RI, MI, TK, ADJ>, dim3((unsigned)nb), dim3(256), sm, st, t, f->taps,
                       reinterpret_cast<const int4*>(f->d_col), (const double*)f->d_cw, (const double*)f->d_norm, x, y));
    PF_LAUNCH_CHECK("filter launch");
    return PF_OK;
}

// Tile shape: 32 columns along z unless 16 by 16 covers the y-z cross-section with fewer
// padded elements; 8 outputs per thread along x when that still gives every SM two blocks,
// else 4.
template <bool ADJ>
static int dispatch_filter_tile(const pf_filter* f, const double* x, double* y, cudaStream_t st) {
    const Grid& g = f->grid;
    FilterTile t;
    t.nx = g.dim == 3 ? g.nel[0] : 1;
    t.ny = g.dim == 3 ? g.nel[1] : g.nel[0];
    t.nz = g.dim == 3 ? g.nel[2] : g.nel[1];
    t.ri = f->rad[0];
    t.rj = f->rad[1];
    t.rk = f->rad[2];
    t.ncol = f->ncol;
    t.nw = f->n_taps;
    t.norm_in = f->norm_in;
    t.tj = t.tk = 0;
    auto cover = [&](int TK) {
        const int TJ = 256 / TK;
        return (long long)((t.nz + TK - 1) / TK) * ((t.ny + TJ - 1) / TJ);
    };
    const bool k16 = cover(16) < cover(32);
    const bool long_run = cover(k16 ? 16 : 32) * ((t.nx + 7) / 8) >= 2 * kNumSM;
#define PF_FT(RI, MI) \
    return k16 ? launch_filter_tile<RI, MI, 16, ADJ>(f, t, x, y, st) : launch_filter_tile<RI, MI, 32, ADJ>(f, t, x, y, st)
    if (g.dim == 2 && f->ncol <= kTapCols && f->n_taps <= kTapWeights) PF_FT(1, 0);
    const bool table = f->ncol > kTapCols || f->n_taps > kTapWeights;
    if (t.ri <= 1 && !table) {
        if (long_run) PF_FT(8, 1);
        PF_FT(4, 1);
    }
    if (t.ri == 2 && !table) {
        if (long_run) PF_FT(8, 2);
        PF_FT(4, 2);
    }
    if (g.dim == 2) PF_FT(1, 3);
    if (long_run) PF_FT(8, 4);
    PF_FT(4, 4);
#undef PF_FT
}

// Tap columns: taps grouped by their y-z offset (2D: every tap a column of one along the
// absent x axis).  Left empty (k_filter serves) unless each column is an unbroken symmetric
// run of distinct offsets along x, at most 9 long, and the largest tile fits in shared memory.
// h_col and h_cw hold 4 and 1 entries per tap.
static void filter_columns(pf_filter* f, const int* off, const double* w, int* h_col, double* h_cw) {
    const Grid& g = f->grid;
    const int dim = g.dim, K = f->n_taps;
    f->ncol = 0;
    for (int a = 0; a < 3; a++) f->rad[a] = 0;
    constexpr int kRad = 64;
    f->norm_in = 0.0;
    for (int t = 0; t < K; t++) {
        f->norm_in += w[t];
        for (int a = 0; a < dim; a++) {
            const int r = off[t * dim + a] < 0 ? -off[t * dim + a] : off[t * dim + a];
            if (r > kRad || r < 0) return;
            int& m = f->rad[a + 3 - dim];
            if (r > m) m = r;
        }
    }
    if (f->rad[0] > 4 || !(f->norm_in > 0.0) || !std::isfinite(f->norm_in)) return;
    const int W = 2 * f->rad[0] + 1, nk = 2 * f->rad[2] + 1, nc = (2 * f->rad[1] + 1) * nk;
    std::vector<int> at((size_t)nc * W, -1);
    for (int t = 0; t < K; t++) {
        const int di = dim == 3 ? off[t * 3] : 0, dj = off[t * dim + dim - 2], dk = off[t * dim + dim - 1];
        int& p = at[(size_t)((dj + f->rad[1]) * nk + dk + f->rad[2]) * W + di + f->rad[0]];
        if (p >= 0) return;  // an offset twice
        p = t;
    }
    std::vector<int> col;
    std::vector<double> cw;
    for (int c = 0; c < nc; c++) {
        int m = -1;
        for (int d = 0; d <= f->rad[0]; d++)
            if (at[(size_t)c * W + f->rad[0] + d] >= 0 || at[(size_t)c * W + f->rad[0] - d] >= 0) m = d;
        if (m < 0) continue;
        col.insert(col.end(), {c / nk - f->rad[1], c % nk - f->rad[2], m, (int)cw.size()});
        for (int d = -m; d <= m; d++) {
            const int t = at[(size_t)c * W + f->rad[0] + d];
            if (t < 0) return;
            cw.push_back(w[t] / f->norm_in);
        }
    }
    FilterTile t{};
    t.ri = f->rad[0];
    t.rj = f->rad[1];
    t.rk = f->rad[2];
    t.ncol = (int)col.size() / 4;
    t.nw = K;
    if (filter_tile_smem(t, 8, 16) > kFilterMaxSmem || filter_tile_smem(t, 8, 32) > kFilterMaxSmem) return;
    f->ncol = t.ncol;
    memcpy(h_col, col.data(), sizeof(int) * col.size());
    memcpy(h_cw, cw.data(), sizeof(double) * cw.size());
    if (f->ncol <= kTapCols && K <= kTapWeights) {
        memcpy(f->taps.col, col.data(), sizeof(int) * col.size());
        memcpy(f->taps.w, cw.data(), sizeof(double) * cw.size());
    }
}

static int launch_filter(const pf_filter* f, int mode, const double* x, double* y, cudaStream_t st) {
    const Grid& g = f->grid;
    if (f->ncol > 0 && mode == 0) return dispatch_filter_tile<false>(f, x, y, st);
    if (f->ncol > 0 && mode == 1) return dispatch_filter_tile<true>(f, x, y, st);
    const unsigned nb = (unsigned)((g.n_elem + 255) / 256);
    const size_t sm = (size_t)f->n_taps * (sizeof(double) + g.dim * sizeof(int));
    const int nz = g.dim == 3 ? g.nel[2] : 1;
    count_launch();
#define PF_FILTER_CASE(D, M) \
    k_filter<D, M><<<nb, 256, sm, st>>>(g.nel[0], g.nel[1], nz, f->n_taps, f->d_off, f->d_w, f->d_norm, x, y)
    if (g.dim == 3) {
        if (mode == 0) PF_FILTER_CASE(3, 0);
        else if (mode == 1) PF_FILTER_CASE(3, 1);
        else PF_FILTER_CASE(3, 2);
    } else {
        if (mode == 0) PF_FILTER_CASE(2, 0);
        else if (mode == 1) PF_FILTER_CASE(2, 1);
        else PF_FILTER_CASE(2, 2);
    }
#undef PF_FILTER_CASE
    PF_LAUNCH_CHECK("filter launch");
    return PF_OK;
}

}  // namespace pf

using namespace pf;

extern "C" int pf_filter_create(const pf_grid* grid, int n_taps, const int* h_offsets, const double* h_weights,
                                pf_filter** out) {
    if (!out || !h_offsets || !h_weights) return fail(PF_BAD_ARG, "pf_filter_create: NULL argument");
    *out = nullptr;
    Grid g;
    int s = validate_grid(grid, &g);
    if (s) return s;
    if (n_taps < 1 || n_taps > kMaxTaps) return fail(PF_BAD_ARG, "n_taps must be in [1, %d]", kMaxTaps);
    pf_filter* f = new pf_filter();
    f->grid = g;
    f->n_taps = n_taps;
    // one block holds the tap tables (uploaded together) and the normaliser
    const size_t nt = (size_t)n_taps, head = (2 * nt + 2 * nt + (nt * (g.dim + 1)) / 2 + 2) * sizeof(double);
    std::vector<unsigned char> h(head, 0);
    int* h_col = reinterpret_cast<int*>(h.data());
    double* h_w = reinterpret_cast<double*>(h_col + 4 * nt);
    double* h_cw = h_w + nt;
    int* h_off = reinterpret_cast<int*>(h_cw + nt);
    memcpy(h_w, h_weights, nt * sizeof(double));
    memcpy(h_off, h_offsets, nt * g.dim * sizeof(int));
    filter_columns(f, h_offsets, h_weights, h_col, h_cw);
    if (cudaMalloc(&f->d_mem, head + sizeof(double) * g.n_elem) != cudaSuccess) {
        cudaGetLastError();
        pf_filter_destroy(f);
        return fail(PF_NO_MEMORY, "filter allocation failed");
    }
    auto dev = [&](const void* p) { return static_cast<unsigned char*>(f->d_mem) + (static_cast<const unsigned char*>(p) - h.data()); };
    f->d_col = reinterpret_cast<int*>(dev(h_col));
    f->d_w = reinterpret_cast<double*>(dev(h_w));
    f->d_cw = reinterpret_cast<double*>(dev(h_cw));
    f->d_off = reinterpret_cast<int*>(dev(h_off));
    f->d_norm = reinterpret_cast<double*>(static_cast<unsigned char*>(f->d_mem) + head);
    if (cudaMemcpy(f->d_mem, h.data(), head, cudaMemcpyHostToDevice) != cudaSuccess) {
        pf_filter_destroy(f);
        return fail(PF_CUDA_ERROR, "filter upload failed");
    }
    if ((s = launch_filter(f, 2, nullptr, f->d_norm, nullptr)) || (s = check_cuda(cudaDeviceSynchronize(), "filter normaliser"))) {
        pf_filter_destroy(f);
        return s;
    }
    *out = f;
    return PF_OK;
}

extern "C" int pf_filter_destroy(pf_filter* f) {
    if (!f) return PF_OK;
    if (f->d_mem) cudaFree(f->d_mem);
    delete f;
    return PF_OK;
}

extern "C" int pf_filter_normalizer_f64(const pf_filter* f, double* out, void* stream) {
    if (!f || !out) return fail(PF_BAD_ARG, "pf_filter_normalizer_f64: NULL argument");
    PF_CUDA(cudaMemcpyAsync(out, f->d_norm, sizeof(double) * f->grid.n_elem, cudaMemcpyDeviceToDevice, as_stream(stream)));
    return PF_OK;
}

extern "C" int pf_filter_fwd_f64(const pf_filter* f, const double* x, double* y, void* stream) {
    if (!f || !x || !y) return fail(PF_BAD_ARG, "pf_filter_fwd_f64: NULL argument");
    return launch_filter(f, 0, x, y, as_stream(stream));
}

extern "C" int pf_filter_adj_f64(const pf_filter* f, const double* x, double* y, void* stream) {
    if (!f || !x || !y) return fail(PF_BAD_ARG, "pf_filter_adj_f64: NULL argument");
    return launch_filter(f, 1, x, y, as_stream(stream));
}
