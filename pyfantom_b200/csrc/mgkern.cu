// Multigrid level kernels: grid transfers, Galerkin coarse operators, block-stencil
// matvec with the shared epilogues, stencil diagonal and dense export of the coarsest
// operator.  All kernels are generic over the dimension (DIM = 2 or 3, dof = DIM).
//
// Transfer operators follow the reference (pyFANTOM/core/CUDA/Kernels/mgm.cu:1-244):
// restriction R = diag(1/tw) Phat^T and prolongation P = Phat diag(1/tw) = R^T, where Phat
// is trilinear (bilinear) interpolation (weights 0.5^{|d|_1} on the 3^DIM fine nodes
// around an even fine node) and tw(c) = prod over axes of (1.5 on a boundary, else 2).
// Coarse grids floor nel / 2; along an axis with an odd element count the last fine node
// has one coarse parent, which the prolongation copies (there P differs from R^T, while
// the Galerkin product uses R^T throughout, as the reference).
// Coarse operators are Galerkin R A P with A_fine = Z K Z + I - Z on level 0
// (mgm.cu:247-447) and R A_l P on deeper levels (mgm.cu:449-590).
#include "common.cuh"
#include "elemop.cuh"
#include "mgkern.cuh"

namespace pf {

template <int DIM>
struct GridDev {
    int nel[3];
    int nn[3];
    long long n_nodes;
};

template <int DIM>
__host__ __device__ __forceinline__ long long nidx(const GridDev<DIM>& g, int i, int j, int k) {
    if (DIM == 3) return (long long)k + (long long)g.nn[2] * (i + (long long)g.nn[0] * j);
    return (long long)i + (long long)g.nn[0] * j;
}
// node index -> (i, j, k); 32-bit unsigned division (grids hold fewer than 2^31 DOFs,
// checked by validate_grid), far cheaper than the emulated 64-bit one
template <int DIM>
__device__ __forceinline__ void ndec(const GridDev<DIM>& g, long long n, int& i, int& j, int& k) {
    const unsigned un = (unsigned)n;
    if (DIM == 3) {
        const unsigned nz = (unsigned)g.nn[2], nx = (unsigned)g.nn[0];
        const unsigned t = un / nz;
        k = (int)(un - t * nz);
        j = (int)(t / nx);
        i = (int)(t - (unsigned)j * nx);
    } else {
        const unsigned nx = (unsigned)g.nn[0];
        j = (int)(un / nx);
        i = (int)(un - (unsigned)j * nx);
        k = 0;
    }
}
template <int DIM>
__device__ __forceinline__ bool nok(const GridDev<DIM>& g, int i, int j, int k) {
    if (i < 0 || j < 0 || i >= g.nn[0] || j >= g.nn[1]) return false;
    if (DIM == 3 && (k < 0 || k >= g.nn[2])) return false;
    return true;
}
template <int DIM>
__device__ __forceinline__ double total_weight(const GridDev<DIM>& gc, int i, int j, int k) {
    double t = ((i == 0 || i == gc.nn[0] - 1) ? 1.5 : 2.0) * ((j == 0 || j == gc.nn[1] - 1) ? 1.5 : 2.0);
    if (DIM == 3) t *= (k == 0 || k == gc.nn[2] - 1) ? 1.5 : 2.0;
    return t;
}
__device__ __forceinline__ double half_pow(int d) { return d == 0 ? 1.0 : d == 1 ? 0.5 : d == 2 ? 0.25 : 0.125; }

template <int DIM>
static GridDev<DIM> gdev(const Grid& g) {
    GridDev<DIM> d;
    for (int a = 0; a < 3; a++) {
        d.nel[a] = g.nel[a];
        d.nn[a] = g.nn[a];
    }
    d.n_nodes = g.n_nodes;
    return d;
}

// ---------------------------------------------------------------------------------------
// transfers
// ---------------------------------------------------------------------------------------
// 2D restriction, one thread per (coarse node, component): the 9 weighted fine values of that
// component, accumulated in the output precision.  Per axis the weights are 0.5 / 1 / 0.5
// and 1/tw factorises into 1/1.5 (boundary node) or 1/2.
template <typename TI, typename TO>
__global__ void k_restrict_q(GridDev<2> gf, GridDev<2> gc, const TI* __restrict__ vf, TO* __restrict__ vc,
                             const int* skip, Jacobi0<TO> j0) {
    pdl_wait();
    pdl_trigger();
    const int done = skip ? *skip : 0;  // looked at only once the values are on their way
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= gc.n_nodes * 2) return;
    const long long c = (unsigned)t / 2;
    const int d = (int)(t - c * 2);
    TO jw = TO(0);
    if (j0.x) jw = (TO)((*j0.omega) * j0.scale) * j0.dinv[t];
    int ic, jc, kc;
    ndec(gc, c, ic, jc, kc);
    const int fi = 2 * ic, fj = 2 * jc;
    const TO ti = (ic == 0 || ic == gc.nn[0] - 1) ? TO(1.0 / 1.5) : TO(0.5);
    const TO tj = (jc == 0 || jc == gc.nn[1] - 1) ? TO(1.0 / 1.5) : TO(0.5);
    // values outside the grid are not read but their place in the sums is kept, so that the loads
    // need no branches and are all in flight together
    TO v[9];
    const bool ok_i[3] = {fi > 0, true, fi + 1 < gf.nn[0]}, ok_j[3] = {fj > 0, true, fj + 1 < gf.nn[1]};
    const TI* base = vf + nidx(gf, fi, fj, 0) * 2 + d;
    const int sj = 2 * gf.nn[0];
#pragma unroll
    for (int dj = -1; dj <= 1; dj++)
#pragma unroll
        for (int di = -1; di <= 1; di++)
            v[(dj + 1) * 3 + di + 1] = ok_j[dj + 1] && ok_i[di + 1] ? (TO)base[dj * sj + di * 2] : TO(0);
    TO acc = TO(0);
#pragma unroll
    for (int dj = -1; dj <= 1; dj++) {
        TO accj = TO(0);
#pragma unroll
        for (int di = -1; di <= 1; di++) {
            const TO q = v[(dj + 1) * 3 + di + 1];
            accj += di == 0 ? q : TO(0.5) * q;
        }
        acc += dj == 0 ? accj : TO(0.5) * accj;
    }
    if (done) return;
    const TO bc = (TO)(acc * ti * tj);
    vc[t] = bc;
    // first smoothing sweep of the coarse level from x = 0: x = omega * scale / diag * b
    if (j0.x) j0.x[t] = jw * bc;
}

// 3D restriction by rows: the block of coarse rows (ic0 .. ic0 + NI - 1, jc), or of a chunk of KCB <=
// kRestrictKC coarse nodes of them along z.  Thread s takes component s % 3 of fine node s / 3 along
// z, in the 3 x (2 NI + 1) fine rows that those coarse rows read: loads consecutive across the warp,
// the x and y stages in registers; the z stage goes through shared memory, where the two threads of a
// coarse node share its NI rows.  Per axis the weights are 0.5 / 1 / 0.5 and 1/tw factorises into
// 1/1.5 (boundary node) or 1/2.
// Bound by the loads on the fine levels and by latency on the others.  One thread per coarse value
// reading its 27 fine ones every other node took 2.06 us from 24x12x12 (now 1.55) and 12.6 us from
// 192x96x96 (11.3) in FP64, and 25.7 us of the 256x128x128 FP32 V-cycle, now 6 us less.  Blocks of
// up to 256 threads: with whole rows of 416 only one fits an SM beside the 27 loads in flight (FP64
// 45 us from 256x128x128 instead of 35).
constexpr int kRestrictKC = 42;
template <int NI, typename TI, typename TO>
__global__ void __launch_bounds__((6 * kRestrictKC + 3 + 31) / 32 * 32) k_restrict_rows(GridDev<3> gf, GridDev<3> gc, int chunks, int KCB, const TI* __restrict__ vf,
                                                       TO* __restrict__ vc, const int* skip, Jacobi0<TO> j0) {
    pdl_wait();
    pdl_trigger();
    __shared__ TO s_a[NI][3 * (2 * kRestrictKC + 1)];
    const int done = skip ? *skip : 0;  // looked at only once the values are on their way
    const unsigned row = blockIdx.x / (unsigned)chunks;
    const int kc0 = (int)(blockIdx.x - row * (unsigned)chunks) * KCB;
    const int nxb = (gc.nn[0] + NI - 1) / NI;
    const int jc = (int)(row / (unsigned)nxb), ic0 = (int)(row - (unsigned)jc * (unsigned)nxb) * NI;
    const int s = (int)threadIdx.x, f = s / 3, d = s - 3 * f;
    const int KC = min(KCB, gc.nn[2] - kc0);  // coarse nodes of this block
    const int k = 2 * kc0 - 1 + f;                    // fine node
    const bool in_k = f <= 2 * KC && k >= 0 && k < gf.nn[2];
    // values outside the grid are not read but their place in the sums is kept
    TO v[3][2 * NI + 1];
    const int si = gf.nn[2] * 3;
    const long long sj = (long long)si * gf.nn[0];
    const TI* base = vf + (2 * jc - 1) * sj + (long long)(2 * ic0 - 1) * si + 3 * k + d;
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 2 * NI + 1; a++) {
            const int j = 2 * jc - 1 + b, i = 2 * ic0 - 1 + a;
            v[b][a] = in_k && j >= 0 && j < gf.nn[1] && i >= 0 && i < gf.nn[0] ? (TO)base[b * sj + a * si] : TO(0);
        }
    const int q = f >> 1, kc = kc0 + q;  // this thread's coarse node: rows ic0 + (f & 1), + 2, ..
    const bool out = q < KC;
    const long long c0 = nidx(gc, ic0, jc, kc) * 3 + d;
    TO jw[(NI + 1) / 2];
#pragma unroll
    for (int m = 0; m < (NI + 1) / 2; m++) {
        const int a = 2 * m + (f & 1);
        jw[m] = TO(0);
        if (j0.x && out && a < NI && ic0 + a < gc.nn[0])
            jw[m] = (TO)((*j0.omega) * j0.scale) * j0.dinv[c0 + (long long)a * gc.nn[2] * 3];
    }
    if (f <= 2 * KC) {
#pragma unroll
        for (int a = 0; a < NI; a++) {
            TO y[3];
#pragma unroll
            for (int b = 0; b < 3; b++) y[b] = v[b][2 * a + 1] + TO(0.5) * (v[b][2 * a] + v[b][2 * a + 2]);
            s_a[a][s] = y[1] + TO(0.5) * (y[0] + y[2]);
        }
    }
    __syncthreads();
    if (done || !out) return;
    auto itw = [](int c, int n) { return (c == 0 || c == n - 1) ? TO(1.0 / 1.5) : TO(0.5); };
    const TO tjk = itw(jc, gc.nn[1]) * itw(kc, gc.nn[2]);
#pragma unroll
    for (int m = 0; m < (NI + 1) / 2; m++) {
        const int a = 2 * m + (f & 1);
        if (a >= NI || ic0 + a >= gc.nn[0]) continue;
        const TO* z = s_a[a] + 6 * q + d;
        const TO bc = (z[3] + TO(0.5) * (z[0] + z[6])) * (tjk * itw(ic0 + a, gc.nn[0]));
        const long long c = c0 + (long long)a * gc.nn[2] * 3;
        vc[c] = bc;
        // first smoothing sweep of the coarse level from x = 0: x = omega * scale / diag * b
        if (j0.x) j0.x[c] = jw[m] * bc;
    }
}

// One thread per fine node (all DIM components, contiguous loads of each parent): P =
// Phat diag(1/tw), the mean of the 1, 2, 4 or 8 parent values divided by their tw.  With an
// odd element count the last fine node along that axis has a single parent and takes its
// value (mgm.cu:198-244 averages over the parents that exist), so there P is not R^T.
template <int DIM, typename T>
__global__ void k_prolong(GridDev<DIM> gf, GridDev<DIM> gc, const T* __restrict__ vc, T* __restrict__ vf,
                          const int* skip) {
    pdl_wait();
    pdl_trigger();
    if (skip && *skip) return;
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= gf.n_nodes) return;
    int i, j, k;
    ndec(gf, f, i, j, k);
    const int i0 = i >> 1, j0 = j >> 1, k0 = DIM == 3 ? k >> 1 : 0;
    // an odd fine node past the last coarse node (odd element count) has one parent
    const int i1 = min(i0 + (i & 1), gc.nn[0] - 1), j1 = min(j0 + (j & 1), gc.nn[1] - 1);
    const int k1 = DIM == 3 ? min(k0 + (k & 1), gc.nn[2] - 1) : 0;
    auto itw = [&](int c, int n) { return (c == 0 || c == n - 1) ? T(1.0 / 1.5) : T(0.5); };
    T acc[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) acc[d] = T(0);
    for (int cj = j0; cj <= j1; cj++) {
        const T wj = itw(cj, gc.nn[1]);
        for (int ci = i0; ci <= i1; ci++) {
            const T wij = wj * itw(ci, gc.nn[0]);
            for (int ck = k0; ck <= k1; ck++) {
                const T w = DIM == 3 ? wij * itw(ck, gc.nn[2]) : wij;
                const T* v = vc + nidx(gc, ci, cj, ck) * DIM;
#pragma unroll
                for (int d = 0; d < DIM; d++) acc[d] += w * v[d];
            }
        }
    }
    const int npar = (i1 - i0 + 1) * (j1 - j0 + 1) * (k1 - k0 + 1);  // the mean over the parents
    const T scale = npar == 1 ? T(1) : npar == 2 ? T(0.5) : npar == 4 ? T(0.25) : T(0.125);
#pragma unroll
    for (int d = 0; d < DIM; d++) vf[f * DIM + d] = acc[d] * scale;
}

// 3D prolongation by rows: the block of coarse row (ic, jc) (or a chunk of it along z) writes the
// up-to-4 fine rows (2ic + di, 2jc + dj), di, dj in {0, 1}.  Thread s takes component s % 3 of fine
// node s / 3 along z in each: it forms the z stage in the up-to-4 coarse rows (ic + a, jc + b), then
// the y and x stages, and its stores are consecutive across the warp.  Per axis a fine node at 2c
// takes parent c, one at 2c + 1 the mean of c and c + 1, or c alone past the last coarse node
// (odd count): the same values as k_prolong.
// Bound by its stores on the fine levels and by latency on the others: one thread per coarse node
// writing its 2x2x2 children left 24 dependent loads and 24 strided stores to each thread (FP64:
// 51 -> 28 us onto 256x128x128, 5.6 -> 3.4 us onto 96x48x48, 4.6 -> 1.75 us onto 24x12x12).
// NI coarse rows along x per thread (4 on the fine levels: consecutive rows share their parents, and
// 16 stores are in flight; one row per thread took 33.6 us onto 256x128x128 in FP32).
template <typename T, int NI>
__global__ void __launch_bounds__(512) k_prolong_rows(GridDev<3> gf, GridDev<3> gc, int chunks, const T* __restrict__ vc,
                                                      T* __restrict__ vf, const int* skip) {
    pdl_wait();
    pdl_trigger();
    const int done = skip ? *skip : 0;  // looked at only once the values are on their way
    const unsigned row = blockIdx.x / (unsigned)chunks;
    const int s = (int)(blockIdx.x - row * (unsigned)chunks) * (int)blockDim.x + (int)threadIdx.x;
    if (s >= 3 * gf.nn[2]) return;
    const int nxb = (gc.nn[0] + NI - 1) / NI;
    const int jc = (int)(row / (unsigned)nxb), ic0 = (int)(row - (unsigned)jc * (unsigned)nxb) * NI;
    const int k = s / 3, d = s - 3 * k, kc = k >> 1;
    auto itw = [](int v, int n) { return (v == 0 || v == n - 1) ? T(1.0 / 1.5) : T(0.5); };
    const bool hy = jc + 1 < gc.nn[1];  // upper parent along y
    const bool up = (k & 1) && kc + 1 < gc.nn[2];
    const T wk0 = itw(kc, gc.nn[2]), wk1 = itw(kc + 1, gc.nn[2]);
    T z[NI + 1][2];  // z stage in row (ic0 + a, jc + b); a row outside is not used
#pragma unroll
    for (int a = 0; a <= NI; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int pi = min(ic0 + a, gc.nn[0] - 1), pj = jc + (hy ? b : 0);
            const T wab = itw(pi, gc.nn[0]) * itw(pj, gc.nn[1]);
            const T* v = vc + nidx(gc, pi, pj, kc) * 3 + d;
            const T lo = wab * wk0 * v[0];
            z[a][b] = up ? T(0.5) * (lo + wab * wk1 * v[3]) : lo;
        }
    if (done) return;
    const bool fy = 2 * jc + 1 < gf.nn[1];  // odd child along y
    T* out = vf + nidx(gf, 2 * ic0, 2 * jc, 0) * 3 + s;
    const long long si = (long long)gf.nn[2] * 3, sj = si * gf.nn[0];
#pragma unroll
    for (int a = 0; a < NI; a++, out += 2 * si) {
        const int ic = ic0 + a;
        if (ic >= gc.nn[0]) break;
        const bool hx = ic + 1 < gc.nn[0], fx = 2 * ic + 1 < gf.nn[0];
        const T y0 = hy ? T(0.5) * (z[a][0] + z[a][1]) : z[a][0];
        const T y1 = hy ? T(0.5) * (z[a + 1][0] + z[a + 1][1]) : z[a + 1][0];
        out[0] = z[a][0];
        if (fx) out[si] = hx ? T(0.5) * (z[a][0] + z[a + 1][0]) : z[a][0];
        if (fy) out[sj] = y0;
        if (fx && fy) out[sj + si] = hx ? T(0.5) * (y0 + y1) : y0;
    }
}

template <typename TI, typename TO>
int launch_restrict(const Grid& gf, const TI* vf, TO* vc, const int* skip, cudaStream_t st, Jacobi0<TO> j0) {
    const Grid gc = coarse_grid(gf);
    const unsigned nb = (unsigned)((gc.n_nodes * gf.dim + 255) / 256);
    pf::count_launch();
    if (gf.dim == 3) {
        const int chunks = (gc.nn[2] + kRestrictKC - 1) / kRestrictKC;
        const int kc = (gc.nn[2] + chunks - 1) / chunks, th = (3 * (2 * kc + 1) + 31) / 32 * 32;
        // four rows per thread once that still gives every SM three blocks (from 128x64x64 FP64 5.2 us;
        // one row 6.2; from 96x48x48 3.4 against 3.7 the other way round)
        const bool four = (long long)((gc.nn[0] + 3) / 4) * gc.nn[1] * chunks >= 3LL * kNumSM;
        const long long rows = (long long)(four ? (gc.nn[0] + 3) / 4 : gc.nn[0]) * gc.nn[1];
        PF_CUDA(launch_pdl(four ? k_restrict_rows<4, TI, TO> : k_restrict_rows<1, TI, TO>, dim3((unsigned)(rows * chunks)),
                           dim3(th), 0, st, gdev<3>(gf), gdev<3>(gc), chunks, kc, vf, vc, skip, j0));
    } else
        PF_CUDA(launch_pdl(k_restrict_q<TI, TO>, dim3(nb), dim3(256), 0, st, gdev<2>(gf), gdev<2>(gc), vf, vc, skip, j0));
    PF_LAUNCH_CHECK("restrict launch");
    return PF_OK;
}
template <typename T>
int launch_prolong(const Grid& gf, const T* vc, T* vf, const int* skip, cudaStream_t st) {
    const Grid gc = coarse_grid(gf);
    const unsigned nb = (unsigned)((gf.n_nodes + 255) / 256);
    pf::count_launch();
    if (gf.dim == 3) {
        const int n = 3 * gf.nn[2], chunks = (n + 511) / 512, th = ((n + chunks - 1) / chunks + 31) / 32 * 32;
        // four rows per thread once that still gives every SM eight blocks
        const bool four = (long long)((gc.nn[0] + 3) / 4) * gc.nn[1] * chunks >= 8LL * kNumSM;
        const long long rows = (long long)(four ? (gc.nn[0] + 3) / 4 : gc.nn[0]) * gc.nn[1];
        PF_CUDA(launch_pdl(four ? k_prolong_rows<T, 4> : k_prolong_rows<T, 1>, dim3((unsigned)(rows * chunks)), dim3(th), 0,
                           st, gdev<3>(gf), gdev<3>(gc), chunks, vc, vf, skip));
    } else
        PF_CUDA(launch_pdl(k_prolong<2, T>, dim3(nb), dim3(256), 0, st, gdev<2>(gf), gdev<2>(gc), vc, vf, skip));
    PF_LAUNCH_CHECK("prolong launch");
    return PF_OK;
}
template int launch_restrict<double, double>(const Grid&, const double*, double*, const int*, cudaStream_t,
                                            Jacobi0<double>);
template int launch_restrict<float, float>(const Grid&, const float*, float*, const int*, cudaStream_t,
                                          Jacobi0<float>);
template int launch_prolong<double>(const Grid&, const double*, double*, const int*, cudaStream_t);
template int launch_prolong<float>(const Grid&, const float*, float*, const int*, cudaStream_t);

// ---------------------------------------------------------------------------------------
// bottom of the V-cycle: the last smoothed level and the dense solve below it in one launch
// ---------------------------------------------------------------------------------------
// A cluster of kBottomCTAs blocks.  Block r owns nodes [r npc, (r + 1) npc); thread (node n, group
// grp < 9) keeps the 27 stencil values of offsets 3 grp .. 3 grp + 2 in registers through the
// 2 n_smooth products.  A product's result is stored into every block's copy of the level vector, so
// that one cluster barrier separates two steps; the restricted residual and the prolonged correction
// are formed by every block for itself.
// Bound by latency: 13x7x7 nodes over 336 coarse values, n_smooth 2, FP64: 2 us to read the operators
// (beside the launch before), 1.4 to 2.3 us per product, of which 1 us for its distribution and the
// barrier, 2.1 us for the coarse inverse.  Level by level it was seven launches and 16 us: FP64
// V-cycle of 96x48x48 140.8 -> 133.5 us, mixed of 192x96x96 352.8 -> 339.2 us.  With the stencil in
// shared memory and read again for each product, and the inverse read from L2, it was 36 us.
constexpr int kBottomCTAs = 16;

template <typename T>
struct BottomArgs {
    GridDev<3> g, gc;
    const T* H;  // half storage of the level's stencil
    const T *b, *x0, *dinv;
    T* out;
    const double* Ainv;
    int np, ns, npc;
    int inv_off, inv_rows;  // rows of Ainv held in shared memory (per block), at this byte offset
    const double* omega;
    double scale;
    const int* skip;
};

template <typename T>
struct BottomSmem {  // offsets in values of T
    int u, b, d, x, r, part, bc, xc, end;
    __host__ __device__ BottomSmem(int npc, int N, int Nc) {
        u = 0, b = 6 * N, d = b + 3 * npc, x = d + 3 * npc, r = x + 3 * npc, part = r + 3 * npc;
        bc = part + 27 * npc, xc = bc + 3 * Nc, end = xc + 3 * Nc;
    }
};

template <typename T>
__device__ __forceinline__ void st_rank(T* p, int rank, T v) {  // *p of block `rank`
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    if constexpr (sizeof(T) == 8)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
    else
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

template <typename T, int NT>
__global__ void __launch_bounds__(NT, 1) k_mg_bottom(const BottomArgs<T> p) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int N = (int)p.g.n_nodes, Nc = (int)p.gc.n_nodes, npc = p.npc, rank = blockIdx.x, tid = threadIdx.x;
    cluster_arrive();  // every block has started: before the first store into another one
    const BottomSmem<T> so(npc, N, Nc);
    T* const sm = reinterpret_cast<T*>(s_raw);
    T *const sb = sm + so.b, *const sd = sm + so.d, *const sx = sm + so.x, *const sr = sm + so.r;
    T *const part = sm + so.part, *const sbc = sm + so.bc, *const sxc = sm + so.xc;
    const int n0 = rank * npc, nloc = max(0, min(npc, N - n0));
    const int sj = p.g.nn[2] * p.g.nn[0], si = p.g.nn[2];
    // The stencil and the coarse inverse are written by the setup, several launches back: they are
    // read (the inverse into L2) while the launch before this one still runs.
    const int grp = (unsigned)tid / (unsigned)npc, n = tid - grp * npc;
    const bool item = grp < 9 && n < nloc;
    T A[27];
    int m[3];  // the neighbours' places in a level vector
    {
        int i = 0, j = 0, k = 0;
        if (item) ndec(p.g, n0 + n, i, j, k);
        const int oy = grp % 3 - 1, oz = grp / 3 - 1;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const bool ok = item && nok(p.g, i + q - 1, j + oy, k + oz);
            m[q] = 3 * (ok ? n0 + n + oz + (q - 1) * si + oy * sj : item ? n0 + n : 0);
            // as in k_stencil_matvec: a lower offset is its neighbour's opposite block, transposed
            constexpr int C = 13;
            const int o = 3 * grp + q, t = o >= C ? n0 + n : m[q] / 3, sa = o >= C ? 96 : 32;
            const T* Ho = p.H + ((long long)(t >> 5) * (C + 1) + abs(o - C)) * 9 * 32 + (t & 31);
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) A[9 * q + 3 * a + b] = ok ? __ldcg(Ho + a * sa + b * (128 - sa)) : T(0);
        }
    }
    const int nrow = (3 * Nc - rank + kBottomCTAs - 1) / kBottomCTAs;  // rows rank, rank + kBottomCTAs, ..
    double* const s_inv = reinterpret_cast<double*>(s_raw + p.inv_off);
    const int c2 = (3 * Nc + 1) / 2, ld = 2 * c2;  // pairs per row; a row is padded to pairs (np is even)
    for (int t = tid; t < min(nrow, p.inv_rows) * c2; t += NT) {
        const int r = (unsigned)t / (unsigned)c2, c = 2 * (t - r * c2);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(s_inv + r * ld + c)),
                     "l"(p.Ainv + (long long)(rank + r * kBottomCTAs) * p.np + c)
                     : "memory");
    }
    pdl_wait();
    pdl_trigger();
    const int done = p.skip ? *p.skip : 0;  // the same for all blocks
    const T w = (T)((*p.omega) * p.scale);
    T* u = sm + so.u;  // the current level vector (all nodes)
    T* v = u + 3 * N;  // the next one
#pragma unroll 4
    for (int t = tid; t < 3 * N; t += NT) u[t] = p.x0[t];
    for (int t = tid; t < 3 * nloc; t += NT) {
        sb[t] = p.b[3 * n0 + t];
        sd[t] = p.dinv[3 * n0 + t];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_wait();
    if (done) return;
    __syncthreads();
    // f(own DOF, (A u) there)
    auto product = [&](auto f) {
        if (item) {
            T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const T u0 = u[m[q]], u1 = u[m[q] + 1], u2 = u[m[q] + 2];
#pragma unroll
                for (int a = 0; a < 3; a++)
                    acc[a] = fma(A[9 * q + 3 * a], u0, fma(A[9 * q + 3 * a + 1], u1, fma(A[9 * q + 3 * a + 2], u2, acc[a])));
            }
#pragma unroll
            for (int a = 0; a < 3; a++) part[(grp * npc + n) * 3 + a] = acc[a];
        }
        __syncthreads();
        if (tid < 3 * nloc) {
            T y = part[tid];
#pragma unroll
            for (int q = 1; q < 9; q++) y += part[q * 3 * npc + tid];
            f(tid, y);
        }
    };
    auto share = [&](int t, T val) {
#pragma unroll
        for (int r = 0; r < kBottomCTAs; r++) st_rank(v + 3 * n0 + t, r, val);
    };
    auto next = [&]() {  // everybody's values are in v
        cluster_arrive();
        cluster_wait();
        T* q = u;
        u = v;
        v = q;
    };
    for (int k = 1; k < p.ns; k++) {
        product([&](int t, T y) { share(t, u[3 * n0 + t] + w * sd[t] * (sb[t] - y)); });
        next();
    }
    product([&](int t, T y) {
        sx[t] = u[3 * n0 + t];
        sr[t] = sb[t] - y;
        share(t, sr[t]);
    });
    next();
    // restriction (the values of k_restrict_rows)
    auto itw = [](int c, int nn) { return (c == 0 || c == nn - 1) ? T(1.0 / 1.5) : T(0.5); };
    for (int t = tid; t < 3 * Nc; t += NT) {
        const int c = (unsigned)t / 3u, d = t - 3 * c;
        int i, j, k;
        ndec(p.gc, c, i, j, k);
        const T* uc = u + 3 * (2 * k + si * 2 * i + sj * 2 * j) + d;
        T acc = T(0);
#pragma unroll
        for (int b = -1; b <= 1; b++)
#pragma unroll
            for (int a = -1; a <= 1; a++)
#pragma unroll
                for (int q = -1; q <= 1; q++)
                    acc += T((a ? 0.5 : 1.0) * (b ? 0.5 : 1.0) * (q ? 0.5 : 1.0)) *
                           (nok(p.g, 2 * i + a, 2 * j + b, 2 * k + q) ? uc[3 * (q + a * si + b * sj)] : T(0));
        sbc[t] = acc * (itw(i, p.gc.nn[0]) * itw(j, p.gc.nn[1]) * itw(k, p.gc.nn[2]));
    }
    __syncthreads();
    // x_c = A_c^-1 b_c, accumulation in FP64, a row per warp; the loads of 12 x 32 columns are in
    // flight together.  Stored divided by tw, so that the prolongation takes plain means.
    const int l = tid & 31;
    for (int r = tid >> 5; r < nrow; r += NT / 32) {
        const int row = rank + r * kBottomCTAs;
        const double* Ar = r < p.inv_rows ? s_inv + r * ld : p.Ainv + (long long)row * p.np;
        double s = 0.0;
        for (int c0 = l; c0 < 3 * Nc; c0 += 12 * 32) {
            double a[12];
#pragma unroll
            for (int q = 0; q < 12; q++) a[q] = c0 + 32 * q < 3 * Nc ? Ar[c0 + 32 * q] : 0.0;
#pragma unroll
            for (int q = 0; q < 12; q++)
                if (c0 + 32 * q < 3 * Nc) s += a[q] * (double)sbc[c0 + 32 * q];
        }
        s = __shfl_sync(0xffffffffu, warp_sum(s), 0);
        int i, j, k;
        ndec(p.gc, row / 3, i, j, k);
        const T x = (T)s * (itw(i, p.gc.nn[0]) * itw(j, p.gc.nn[1]) * itw(k, p.gc.nn[2]));
        if (l < kBottomCTAs) st_rank(sxc + row, l, x);
    }
    cluster_arrive();
    cluster_wait();
    // prolongation (the values of k_prolong): the mean over the parents, one that is alone along an
    // axis taken twice
#pragma unroll 4
    for (int t = tid; t < 3 * N; t += NT) {
        const int f = (unsigned)t / 3u, d = t - 3 * f;
        int i, j, k;
        ndec(p.g, f, i, j, k);
        const int ck = p.gc.nn[2], ci = p.gc.nn[0];
        const int k1 = (k >> 1) + (k & 1) < ck ? 3 * (k & 1) : 0, i1 = (i >> 1) + (i & 1) < ci ? 3 * ck * (i & 1) : 0;
        const int j1 = (j >> 1) + (j & 1) < p.gc.nn[1] ? 3 * ck * ci * (j & 1) : 0;
        const T* x = sxc + 3 * ((k >> 1) + ck * ((i >> 1) + ci * (j >> 1))) + d;
        v[t] = T(0.125) * (((x[0] + x[k1]) + (x[i1] + x[i1 + k1])) + ((x[j1] + x[j1 + k1]) + (x[j1 + i1] + x[j1 + i1 + k1])));
    }
    {
        T* q = u;
        u = v;
        v = q;
    }
    __syncthreads();
    for (int k = 1; k < p.ns; k++) {
        product([&](int t, T y) { share(t, u[3 * n0 + t] + w * sd[t] * (sr[t] - y)); });
        next();
    }
    product([&](int t, T y) { p.out[3 * n0 + t] = sx[t] + u[3 * n0 + t] + w * sd[t] * (sr[t] - y); });
}

// A level fits when the stencil goes into the cluster's registers, 27 values per thread: 512 threads
// per block in FP64 (896 nodes), 1024 in FP32 (1808).  Only 16 SMs read the coarse inverse: 675 values
// take 6.6 us of the kernel where a launch over all SMs takes 4, and the 256x128x128 V-cycle still
// gained 13 us (699 -> 686); the line is drawn a little above.
constexpr int kBottomCoarse = 768;

static int bottom_npc(const Grid& g) { return (int)((g.n_nodes + kBottomCTAs - 1) / kBottomCTAs); }
// shared memory: the vectors, then as many of the block's rows of the coarse inverse as fit
constexpr int kBottomSmem = 200 * 1024;
template <typename T>
static size_t bottom_smem(const Grid& g, int* inv_off, int* inv_rows) {
    const int nc = 3 * (int)coarse_grid(g).n_nodes, row = (nc + 1) / 2 * 16, rows = (nc + kBottomCTAs - 1) / kBottomCTAs;
    const int off = (int)(sizeof(T) * BottomSmem<T>(bottom_npc(g), (int)g.n_nodes, nc / 3).end + 15) / 16 * 16;
    const int fit = (kBottomSmem - off) / row;
    *inv_off = off;
    *inv_rows = fit < rows ? fit : rows;
    return off + (size_t)*inv_rows * row;
}
template <typename T>
static cudaLaunchConfig_t bottom_config(const Grid& g, int threads, cudaLaunchAttribute* attr, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    int off, rows;
    cfg.gridDim = dim3(kBottomCTAs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bottom_smem<T>(g, &off, &rows);
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kBottomCTAs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}
template <typename T>
static auto bottom_kernel(const Grid& g, int* threads) {
    *threads = sizeof(T) == 8 || 9 * bottom_npc(g) <= 512 ? 512 : 1024;
    return *threads == 512 ? k_mg_bottom<T, 512> : k_mg_bottom<T, sizeof(T) == 8 ? 512 : 1024>;
}

template <typename T>
bool bottom_fits(const Grid& g) {
    if (g.dim != 3 || g.n_nodes > kBottomCTAs * 113) return false;
    int threads, n = 0;
    auto kernel = bottom_kernel<T>(g, &threads);
    if (9 * bottom_npc(g) > threads || coarse_grid(g).n_nodes * 3 > kBottomCoarse) return false;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = bottom_config<T>(g, threads, attr, nullptr);
    cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBottomSmem) == cudaSuccess &&
                    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
    cudaGetLastError();
    return ok;
}

template <typename T>
int launch_bottom(const Grid& g, const T* H, const T* b, const T* x0, const T* dinv, T* out, const Dense* d, int ns,
                  const double* omega, double scale, const int* skip, cudaStream_t st) {
    int threads;
    auto kernel = bottom_kernel<T>(g, &threads);
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = bottom_config<T>(g, threads, attr, st);
    int off, rows;
    bottom_smem<T>(g, &off, &rows);
    const BottomArgs<T> a{gdev<3>(g), gdev<3>(coarse_grid(g)), H, b, x0, dinv, out, d->Ainv, d->np, ns, bottom_npc(g),
                          off, rows, omega, scale, skip};
    pf::count_launch();
    PF_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    PF_LAUNCH_CHECK("V-cycle bottom launch");
    return PF_OK;
}
template bool bottom_fits<double>(const Grid&);
template bool bottom_fits<float>(const Grid&);
template int launch_bottom<double>(const Grid&, const double*, const double*, const double*, const double*, double*, const Dense*,
                                   int, const double*, double, const int*, cudaStream_t);
template int launch_bottom<float>(const Grid&, const float*, const float*, const float*, const float*, float*, const Dense*,
                                  int, const double*, double, const int*, cudaStream_t);

// ---------------------------------------------------------------------------------------
// block-stencil matvec (levels >= 1): y_n = sum_o A[n,o] u_{n+o}
// A block covers 32 consecutive nodes; warp w gathers the neighbour offsets 3w..3w+2 for
// all 32 nodes (coalesced reads of the structure-of-arrays coefficients), the per-warp
// partial sums meet in shared memory and warp a adds those of component a in a fixed order and
// applies the epilogue.  3D: 9 warps x 3 offsets, 2D: 3 warps x 3 offsets.
// HALF: A holds only the centre and the upper offsets o > c (c = NB/2 the centre, stored
// block q = o - c); a lower offset o < c uses the symmetry of the level operator,
// A[n, o] = A[n+o, -o]^T, i.e. block q = c - o of the neighbour n+o, transposed.  The
// neighbour's coefficients are read again by another block shortly after (from L2), so
// DRAM carries each coefficient once: (NB+1)/2 blocks per node instead of NB.  The half
// copy is tiled by 32 nodes, A[((n >> 5) * NH*BS + q*BS + a*DIM + b) * 32 + (n & 31)]:
// each tile's (NB+1)/2 * DIM^2 coefficient rows are one contiguous run (16 KB in 3D FP32),
// so DRAM streams through it instead of jumping between NH*BS planes of N values.
// ---------------------------------------------------------------------------------------
// Launch bounds: FP32 keeps 7 blocks per SM (32 registers), FP64 4 (56 registers; the 40 that the
// compiler took by itself measured slower).
// On the small levels a launch is a chain of latencies: the completion flag, the Jacobi weight
// and the epilogue's operands (component a by warp a) are loaded before the coefficients, and the
// flag is looked at when these have arrived.
template <int DIM, typename T, bool HALF>
__global__ void __launch_bounds__(DIM == 3 ? 288 : 96, DIM == 3 ? (sizeof(T) == 4 ? 7 : 4) : 1)
    k_stencil_matvec(GridDev<DIM> g, const T* __restrict__ A, const T* __restrict__ u, Epi<T> epi) {
    pdl_wait();
    pdl_trigger();
    constexpr int NB = DIM == 3 ? 27 : 9, BS = DIM * DIM, NG = NB / 3, C = NB / 2;
    constexpr long long TS = (long long)(C + 1) * BS * 32;  // values per tile of the half copy
    __shared__ T s_part[NG][DIM][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const long long n = (long long)blockIdx.x * 32 + l;
    const long long N = g.n_nodes;
    const bool valid = n < N;
    const int done = epi.skip ? *epi.skip : 0;
    T pb = T(0), px = T(0), pd = T(0), wgt = T(0);
    const long long gi = n * DIM + w;
    if (w < DIM && valid) {
        if (epi.mode != PF_EPI_STORE) pb = epi.b[gi];
        if (epi.mode == PF_EPI_JACOBI || epi.mode == PF_EPI_JACOBI_ADD) {
            wgt = epi_omega(epi);
            pd = epi.dinv[gi];
            px = epi.x[gi];
            if (epi.mode == PF_EPI_JACOBI_ADD) px = epi.xadd[gi] + px;
        }
    }
    T acc[DIM];
#pragma unroll
    for (int a = 0; a < DIM; a++) acc[a] = T(0);
    if (valid) {
        int i, j, k;
        ndec(g, n, i, j, k);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int o = 3 * w + q;
            const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = DIM == 3 ? o / 9 - 1 : 0;
            if (!nok(g, i + ox, j + oy, k + oz)) continue;
            const long long m = nidx(g, i + ox, j + oy, k + oz);
            T um[DIM];
#pragma unroll
            for (int b = 0; b < DIM; b++) um[b] = u[m * DIM + b];
            if (!HALF) {
#pragma unroll
                for (int a = 0; a < DIM; a++)
#pragma unroll
                    for (int b = 0; b < DIM; b++)
                        acc[a] = fma(A[((long long)(o * BS + a * DIM + b)) * N + n], um[b], acc[a]);
            } else if (o >= C) {
                const T* Aq = A + (n >> 5) * TS + (o - C) * BS * 32 + (n & 31);
#pragma unroll
                for (int a = 0; a < DIM; a++)
#pragma unroll
                    for (int b = 0; b < DIM; b++) acc[a] = fma(Aq[(a * DIM + b) * 32], um[b], acc[a]);
            } else {
                const T* Aq = A + (m >> 5) * TS + (C - o) * BS * 32 + (m & 31);
#pragma unroll
                for (int a = 0; a < DIM; a++)
#pragma unroll
                    for (int b = 0; b < DIM; b++) acc[a] = fma(Aq[(b * DIM + a) * 32], um[b], acc[a]);
            }
        }
    }
    if (done) return;
#pragma unroll
    for (int a = 0; a < DIM; a++) s_part[w][a][l] = acc[a];
    __syncthreads();
    if (w >= DIM || !valid) return;
    T y = s_part[0][w][l];
#pragma unroll
    for (int v = 1; v < NG; v++) y += s_part[v][w][l];
    T o = y;
    if (epi.mode == PF_EPI_RESID)
        o = pb - y;
    else if (epi.mode != PF_EPI_STORE)
        o = px + wgt * pd * (pb - y);
    epi.out[gi] = o;
}

template <typename T>
int launch_stencil_matvec(const Grid& g, const T* A, const T* u, const Epi<T>& epi, cudaStream_t st, bool half) {
    if (epi.dot_partial) return fail(PF_UNSUPPORTED, "stencil matvec: no fused dot");
    const unsigned nb = (unsigned)((g.n_nodes + 31) / 32);
    pf::count_launch();
    if (g.dim == 3) {
        if (half)
            PF_CUDA(launch_pdl(k_stencil_matvec<3, T, true>, dim3(nb), dim3(288), 0, st, gdev<3>(g), A, u, epi));
        else
            PF_CUDA(launch_pdl(k_stencil_matvec<3, T, false>, dim3(nb), dim3(288), 0, st, gdev<3>(g), A, u, epi));
    } else {
        if (half)
            PF_CUDA(launch_pdl(k_stencil_matvec<2, T, true>, dim3(nb), dim3(96), 0, st, gdev<2>(g), A, u, epi));
        else
            PF_CUDA(launch_pdl(k_stencil_matvec<2, T, false>, dim3(nb), dim3(96), 0, st, gdev<2>(g), A, u, epi));
    }
    PF_LAUNCH_CHECK("stencil matvec launch");
    return PF_OK;
}
long long stencil_matvec_num_blocks(const Grid& g) { return (g.n_nodes + 31) / 32; }
template int launch_stencil_matvec<double>(const Grid&, const double*, const double*, const Epi<double>&,
                                           cudaStream_t, bool);
template int launch_stencil_matvec<float>(const Grid&, const float*, const float*, const Epi<float>&, cudaStream_t,
                                          bool);

// half storage for the V-cycle: the centre and upper-offset blocks of the full FP64 stencil,
// converted to the V-cycle precision
template <typename T>
__global__ void k_stencil_half(long long N, int nh, int bs, int c, const double* __restrict__ A, T* __restrict__ H) {
    // tiles of 32 nodes (the last one zero-padded): H[(t * nh*bs + qab) * 32 + lane]
    const long long per_tile = (long long)nh * bs * 32;
    const long long total = ((N + 31) / 32) * per_tile;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long t = i / per_tile;
        const int r = (int)(i - t * per_tile), qab = r >> 5;
        const long long n = t * 32 + (r & 31);
        H[i] = n < N ? (T)A[(long long)(c * bs + qab) * N + n] : T(0);
    }
}
long long stencil_half_size(const Grid& g) {
    const int nb = g.dim == 3 ? 27 : 9;
    return ((g.n_nodes + 31) / 32) * 32 * ((nb + 1) / 2) * g.dof * g.dof;
}
template <typename T>
int launch_stencil_half(const Grid& g, const double* A, T* H, cudaStream_t st) {
    const int nb = g.dim == 3 ? 27 : 9, bs = g.dof * g.dof;
    const long long total = stencil_half_size(g);
    long long blocks = (total + 255) / 256;
    if (blocks > 8LL * kNumSM * 4) blocks = 8LL * kNumSM * 4;
    pf::count_launch();
    k_stencil_half<T><<<(unsigned)blocks, 256, 0, st>>>(g.n_nodes, (nb + 1) / 2, bs, nb / 2, A, H);
    PF_LAUNCH_CHECK("stencil half launch");
    return PF_OK;
}
template int launch_stencil_half<double>(const Grid&, const double*, double*, cudaStream_t);
template int launch_stencil_half<float>(const Grid&, const double*, float*, cudaStream_t);

// ---------------------------------------------------------------------------------------
// Galerkin level 1 from the element operator.
// With Phat_c the local interpolation from a coarse element's corners to its child c,
//   Phat^T (Z K Z) Phat = sum_C sum_c E_{C,c} (Z Phat_c)^T K0 (Z Phat_c)
// which for a coarse element C whose 3^DIM fine nodes carry no constraint is
// sum_c E_{C,c} Kc[c] with the fixed child matrices Kc[c] = Phat_c^T K0 Phat_c.  The
// identity rows of constrained DOFs add Phat^T (I - Z) Phat.  Each thread produces one
// dof x dof block (coarse node I, neighbour o) by gathering the coarse elements that
// contain I and I+o (owner computes, no atomics), then scales by 1/(tw_I tw_J).  Bound by writing
// the 27 blocks (1944 bytes per node) and by FP64 FMAs; with the child matrices read from global
// memory entry by entry it took 1580 us at 256x128x128.
// ---------------------------------------------------------------------------------------
template <int DIM>
__device__ __forceinline__ int ccx(int l) {
    return kCXd(l);
}

// flags: per coarse element, 1 if any of its fine nodes has a constraint;
//        per coarse node, 1 if any fine node within distance 1 of 2I has a constraint.
template <int DIM>
__global__ void k_coarse_flags(GridDev<DIM> gf, GridDev<DIM> gc, const uint8_t* __restrict__ mask,
                               uint8_t* __restrict__ elem_flag, uint8_t* __restrict__ node_flag) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= gc.n_nodes) return;
    int ic, jc, kc;
    ndec(gc, c, ic, jc, kc);
    constexpr int KR = DIM == 3 ? 1 : 0;
    uint8_t nf = 0;
    for (int di = -1; di <= 1; di++)
        for (int dj = -1; dj <= 1; dj++)
            for (int dk = -KR; dk <= KR; dk++) {
                const int fi = 2 * ic + di, fj = 2 * jc + dj, fk = 2 * kc + dk;
                if (nok(gf, fi, fj, fk) && mask[nidx(gf, fi, fj, fk)]) nf = 1;
            }
    node_flag[c] = nf;
    // coarse element with lower corner (ic, jc, kc)
    const bool has_elem = ic < gc.nel[0] && jc < gc.nel[1] && (DIM == 2 || kc < gc.nel[2]);
    if (has_elem) {
        uint8_t ef = 0;
        for (int di = 0; di <= 2; di++)
            for (int dj = 0; dj <= 2; dj++)
                for (int dk = 0; dk <= 2 * KR; dk++)
                    if (mask[nidx(gf, 2 * ic + di, 2 * jc + dj, 2 * kc + dk)]) ef = 1;
        const long long e = DIM == 3 ? ((long long)ic * gc.nel[1] + jc) * gc.nel[2] + kc : (long long)ic * gc.nel[1] + jc;
        elem_flag[e] = ef;
    }
}

template <int DIM>
__global__ void __launch_bounds__(128) k_galerkin_l0(GridDev<DIM> gf, GridDev<DIM> gc, const double* __restrict__ E,
                                                      const uint8_t* __restrict__ mask,
                                                      const uint8_t* __restrict__ elem_flag,
                                                      const uint8_t* __restrict__ node_flag,
                                                      const double* __restrict__ K0,  // (NC*DIM)^2
                                                      const double* __restrict__ Kc,  // NC x (NC*DIM)^2
                                                      double* __restrict__ A) {
    constexpr int NC = DIM == 3 ? 8 : 4, ND = NC * DIM, BS = DIM * DIM, KP = DIM == 3 ? 10 : 4;
    // the neighbour offset is the block's: the corner pairs (LI, LJ = LI + offset) and their child
    // blocks are the same for all its nodes and are staged in shared memory (padded to pairs)
    __shared__ __align__(16) double s_k[NC * NC * KP];
    __shared__ int s_li[NC], s_lj[NC], s_np;
    const long long Nc = gc.n_nodes;
    const int o = blockIdx.y;
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = DIM == 3 ? o / 9 - 1 : 0;
    if (threadIdx.x == 0) {
        int np = 0;
        for (int LI = 0; LI < NC; LI++) {
            const int lx = kCXd(LI) + ox, ly = kCYd(LI) + oy, lz = DIM == 3 ? kCZd(LI) + oz : 0;
            if (lx < 0 || lx > 1 || ly < 0 || ly > 1 || lz < 0 || lz > 1) continue;
            for (int q = 0; q < NC; q++)
                if (kCXd(q) == lx && kCYd(q) == ly && (DIM == 2 || kCZd(q) == lz)) s_lj[np] = q;
            s_li[np++] = LI;
        }
        s_np = np;
    }
    __syncthreads();
    const int npair = s_np;
    for (int q = threadIdx.x; q < npair * NC * BS; q += blockDim.x) {
        const int ab = q % BS, c = (q / BS) % NC, p = q / (BS * NC);
        s_k[(p * NC + c) * KP + ab] =
            Kc[(long long)c * ND * ND + (s_li[p] * DIM + ab / DIM) * ND + s_lj[p] * DIM + ab % DIM];
    }
    __syncthreads();
    const long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= Nc) return;
    int ic, jc, kc;
    ndec(gc, I, ic, jc, kc);
    double blk[BS];
#pragma unroll
    for (int a = 0; a < BS; a++) blk[a] = 0.0;
    const int ti = ic + ox, tj = jc + oy, tk = kc + oz;
    if (nok(gc, ti, tj, tk)) {
        // coarse elements containing I as local corner LI and its neighbour as corner LJ
        for (int p = 0; p < npair; p++) {
            const int LI = s_li[p], LJ = s_lj[p];
            const int ex = ic - kCXd(LI), ey = jc - kCYd(LI), ez = DIM == 3 ? kc - kCZd(LI) : 0;
            // past the last coarse node of an axis with an odd element count lies a virtual
            // coarse element: its far corners do not exist and only its near children do
            const bool vx = ex == gc.nel[0] && gf.nel[0] > 2 * gc.nel[0];
            const bool vy = ey == gc.nel[1] && gf.nel[1] > 2 * gc.nel[1];
            const bool vz = DIM == 3 && ez == gc.nel[2] && gf.nel[2] > 2 * gc.nel[2];
            if (ex < 0 || ey < 0 || (ex >= gc.nel[0] && !vx) || (ey >= gc.nel[1] && !vy)) continue;
            if (DIM == 3 && (ez < 0 || (ez >= gc.nel[2] && !vz))) continue;
            if ((vx && (kCXd(LI) || kCXd(LJ))) || (vy && (kCYd(LI) || kCYd(LJ))) || (vz && (kCZd(LI) || kCZd(LJ)))) continue;
            const bool virt = vx || vy || vz;
            const long long ce = DIM == 3 ? ((long long)ex * gc.nel[1] + ey) * gc.nel[2] + ez : (long long)ex * gc.nel[1] + ey;
            const bool dirty = virt || elem_flag[ce] != 0;  // virtual elements check their masks
            if (!dirty) {
                double we[NC];
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const int fx = 2 * ex + kCXd(c), fy = 2 * ey + kCYd(c), fz = DIM == 3 ? 2 * ez + kCZd(c) : 0;
                    we[c] = E[DIM == 3 ? (fx * gf.nel[1] + fy) * gf.nel[2] + fz : fx * gf.nel[1] + fy];
                }
                const double* kp = s_k + p * NC * KP;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    double kv[KP];
#pragma unroll
                    for (int a = 0; a < KP; a += 2) {
                        const double2 t = *reinterpret_cast<const double2*>(kp + c * KP + a);
                        kv[a] = t.x, kv[a + 1] = t.y;
                    }
#pragma unroll
                    for (int a = 0; a < BS; a++) blk[a] = fma(we[c], kv[a], blk[a]);
                }
                continue;
            }
            for (int c = 0; c < NC; c++) {
                const int fx = 2 * ex + kCXd(c), fy = 2 * ey + kCYd(c), fz = DIM == 3 ? 2 * ez + kCZd(c) : 0;
                if (fx >= gf.nel[0] || fy >= gf.nel[1] || (DIM == 3 && fz >= gf.nel[2])) continue;
                const long long fe = DIM == 3 ? ((long long)fx * gf.nel[1] + fy) * gf.nel[2] + fz : (long long)fx * gf.nel[1] + fy;
                const double we = E[fe];
                {
                    // masked child: sum_{l,l2} Phat_c[l][LI] z(l,a) K0[(l,a),(l2,b)] z(l2,b) Phat_c[l2][LJ]
                    for (int l = 0; l < NC; l++) {
                        const int nxl = kCXd(c) + kCXd(l), nyl = kCYd(c) + kCYd(l), nzl = DIM == 3 ? kCZd(c) + kCZd(l) : 0;
                        double pl = (1.0 - 0.5 * abs(nxl - 2 * kCXd(LI))) * (1.0 - 0.5 * abs(nyl - 2 * kCYd(LI)));
                        if (DIM == 3) pl *= 1.0 - 0.5 * abs(nzl - 2 * kCZd(LI));
                        if (pl == 0.0) continue;
                        const uint8_t ml = mask ? mask[nidx(gf, 2 * ex + nxl, 2 * ey + nyl, 2 * ez + nzl)] : 0;
                        for (int l2 = 0; l2 < NC; l2++) {
                            const int nx2 = kCXd(c) + kCXd(l2), ny2 = kCYd(c) + kCYd(l2), nz2 = DIM == 3 ? kCZd(c) + kCZd(l2) : 0;
                            double p2 = (1.0 - 0.5 * abs(nx2 - 2 * kCXd(LJ))) * (1.0 - 0.5 * abs(ny2 - 2 * kCYd(LJ)));
                            if (DIM == 3) p2 *= 1.0 - 0.5 * abs(nz2 - 2 * kCZd(LJ));
                            if (p2 == 0.0) continue;
                            const uint8_t m2 = mask ? mask[nidx(gf, 2 * ex + nx2, 2 * ey + ny2, 2 * ez + nz2)] : 0;
                            const double f = we * pl * p2;
                            for (int a = 0; a < DIM; a++) {
                                if (ml & (1 << a)) continue;
                                for (int b = 0; b < DIM; b++) {
                                    if (m2 & (1 << b)) continue;
                                    blk[a * DIM + b] += f * K0[(l * DIM + a) * ND + l2 * DIM + b];
                                }
                            }
                        }
                    }
                }
            }
        }
        // identity rows of constrained fine DOFs: sum_n Phat[n,I] Phat[n,J] on the diagonal
        if (node_flag[I]) {
            constexpr int KR = DIM == 3 ? 1 : 0;
            for (int di = -1; di <= 1; di++)
                for (int dj = -1; dj <= 1; dj++)
                    for (int dk = -KR; dk <= KR; dk++) {
                        const int fi = 2 * ic + di, fj = 2 * jc + dj, fk = 2 * kc + dk;
                        if (!nok(gf, fi, fj, fk)) continue;
                        const int ei = fi - 2 * ti, ej = fj - 2 * tj, ek = fk - 2 * tk;
                        if (ei < -1 || ei > 1 || ej < -1 || ej > 1 || ek < -1 || ek > 1) continue;
                        const uint8_t m = mask[nidx(gf, fi, fj, fk)];
                        if (!m) continue;
                        const double w = half_pow((di != 0) + (dj != 0) + (dk != 0)) *
                                         half_pow((ei != 0) + (ej != 0) + (ek != 0));
                        for (int a = 0; a < DIM; a++)
                            if (m & (1 << a)) blk[a * DIM + a] += w;
                    }
        }
        const double s = 1.0 / (total_weight(gc, ic, jc, kc) * total_weight(gc, ti, tj, tk));
#pragma unroll
        for (int a = 0; a < BS; a++) blk[a] *= s;
    }
#pragma unroll
    for (int a = 0; a < BS; a++) A[((long long)(o * BS + a)) * Nc + I] = blk[a];
}

// child matrices Kc[c] = Phat_c^T K0 Phat_c (host)
void galerkin_child_matrices(int dim, const double* K0, double* Kc) {
    const int NC = dim == 3 ? 8 : 4, ND = NC * dim;
    for (int c = 0; c < NC; c++) {
        double P[8][8];  // P[l][L]: weight of coarse corner L at child corner l
        for (int l = 0; l < NC; l++)
            for (int L = 0; L < NC; L++) {
                const int fx = kCXd(c) + kCXd(l), fy = kCYd(c) + kCYd(l), fz = dim == 3 ? kCZd(c) + kCZd(l) : 0;
                double w = (1.0 - 0.5 * abs(fx - 2 * kCXd(L))) * (1.0 - 0.5 * abs(fy - 2 * kCYd(L)));
                if (dim == 3) w *= 1.0 - 0.5 * abs(fz - 2 * kCZd(L));
                P[l][L] = w;
            }
        double* out = Kc + (long long)c * ND * ND;
        for (int L = 0; L < NC; L++)
            for (int a = 0; a < dim; a++)
                for (int L2 = 0; L2 < NC; L2++)
                    for (int b = 0; b < dim; b++) {
                        double s = 0.0;
                        for (int l = 0; l < NC; l++) {
                            if (P[l][L] == 0.0) continue;
                            for (int l2 = 0; l2 < NC; l2++) {
                                if (P[l2][L2] == 0.0) continue;
                                s += P[l][L] * K0[(l * dim + a) * ND + l2 * dim + b] * P[l2][L2];
                            }
                        }
                        out[(L * dim + a) * ND + L2 * dim + b] = s;
                    }
    }
}

int launch_coarse_flags(const Grid& gf, const uint8_t* mask, uint8_t* elem_flag, uint8_t* node_flag, cudaStream_t st) {
    const Grid gc = coarse_grid(gf);
    const unsigned nb = (unsigned)((gc.n_nodes + 255) / 256);
    pf::count_launch();
    if (gf.dim == 3)
        k_coarse_flags<3><<<nb, 256, 0, st>>>(gdev<3>(gf), gdev<3>(gc), mask, elem_flag, node_flag);
    else
        k_coarse_flags<2><<<nb, 256, 0, st>>>(gdev<2>(gf), gdev<2>(gc), mask, elem_flag, node_flag);
    PF_LAUNCH_CHECK("coarse flags launch");
    return PF_OK;
}

int launch_galerkin_l0(const Grid& gf, const double* E, const uint8_t* mask, const uint8_t* elem_flag,
                       const uint8_t* node_flag, const double* K0_dev, const double* Kc_dev, double* A, cudaStream_t st) {
    const Grid gc = coarse_grid(gf);
    const int NB = gf.dim == 3 ? 27 : 9;
    const dim3 nb((unsigned)((gc.n_nodes + 127) / 128), (unsigned)NB);
    pf::count_launch();
    if (gf.dim == 3)
        k_galerkin_l0<3><<<nb, 128, 0, st>>>(gdev<3>(gf), gdev<3>(gc), E, mask, elem_flag, node_flag, K0_dev, Kc_dev, A);
    else
        k_galerkin_l0<2><<<nb, 128, 0, st>>>(gdev<2>(gf), gdev<2>(gc), E, mask, elem_flag, node_flag, K0_dev, Kc_dev, A);
    PF_LAUNCH_CHECK("galerkin l0 launch");
    return PF_OK;
}

// ---------------------------------------------------------------------------------------
// Galerkin level l+1 from the level-l block stencil:
//   A_c[I,J] = sum_{n in supp I} sum_{m in supp J, |m-n|<=1} Phat[n,I] A[n, m-n] Phat[m,J] / (tw_I tw_J)
// Per axis, the admissible (dn, dm) offset pairs depend only on the neighbour offset o.
// ---------------------------------------------------------------------------------------
__constant__ int c_pairs[3][7][2];  // [o+1][pair][dn, dm]
__constant__ int c_npairs[3];

template <int DIM>
__global__ void __launch_bounds__(128) k_galerkin_l1p(GridDev<DIM> gf, GridDev<DIM> gc, const double* __restrict__ Af,
                                                       double* __restrict__ Ac) {
    constexpr int NB = DIM == 3 ? 27 : 9, BS = DIM * DIM;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long Nc = gc.n_nodes, Nf = gf.n_nodes;
    if (tid >= Nc * NB) return;
    const int o = (int)(tid / Nc);
    const long long I = tid - (long long)o * Nc;
    int ic, jc, kc;
    ndec(gc, I, ic, jc, kc);
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = DIM == 3 ? o / 9 - 1 : 0;
    double blk[BS];
#pragma unroll
    for (int a = 0; a < BS; a++) blk[a] = 0.0;
    const int ti = ic + ox, tj = jc + oy, tk = kc + oz;
    if (nok(gc, ti, tj, tk)) {
        const int npx = c_npairs[ox + 1], npy = c_npairs[oy + 1], npz = DIM == 3 ? c_npairs[oz + 1] : 1;
        for (int px = 0; px < npx; px++) {
            const int dnx = c_pairs[ox + 1][px][0], dmx = c_pairs[ox + 1][px][1];
            const int nx_ = 2 * ic + dnx, mx = 2 * ti + dmx;
            if (nx_ < 0 || nx_ >= gf.nn[0] || mx < 0 || mx >= gf.nn[0]) continue;
            for (int py = 0; py < npy; py++) {
                const int dny = c_pairs[oy + 1][py][0], dmy = c_pairs[oy + 1][py][1];
                const int ny_ = 2 * jc + dny, my = 2 * tj + dmy;
                if (ny_ < 0 || ny_ >= gf.nn[1] || my < 0 || my >= gf.nn[1]) continue;
                for (int pz = 0; pz < npz; pz++) {
                    int dnz = 0, dmz = 0, nz_ = 0, mz = 0;
                    if (DIM == 3) {
                        dnz = c_pairs[oz + 1][pz][0];
                        dmz = c_pairs[oz + 1][pz][1];
                        nz_ = 2 * kc + dnz;
                        mz = 2 * tk + dmz;
                        if (nz_ < 0 || nz_ >= gf.nn[2] || mz < 0 || mz >= gf.nn[2]) continue;
                    }
                    const double w = half_pow((dnx != 0) + (dny != 0) + (dnz != 0)) *
                                     half_pow((dmx != 0) + (dmy != 0) + (dmz != 0));
                    const long long n = nidx(gf, nx_, ny_, nz_);
                    const int rx = mx - nx_, ry = my - ny_, rz = DIM == 3 ? mz - nz_ : 0;
                    const int on = (rx + 1) + 3 * (ry + 1) + (DIM == 3 ? 9 * (rz + 1) : 0);
#pragma unroll
                    for (int a = 0; a < BS; a++) blk[a] += w * Af[((long long)(on * BS + a)) * Nf + n];
                }
            }
        }
        const double s = 1.0 / (total_weight(gc, ic, jc, kc) * total_weight(gc, ti, tj, tk));
#pragma unroll
        for (int a = 0; a < BS; a++) blk[a] *= s;
    }
#pragma unroll
    for (int a = 0; a < BS; a++) Ac[((long long)(o * BS + a)) * Nc + I] = blk[a];
}

// One axis of the Galerkin product of a 3D level >= 2.  R = D Phat^T and P = Phat D are
// tensor products of per-axis factors (linear-interpolation weights 0.5^|d|, the per-axis
// part 1/1.5 or 1/2 of 1/tw, the bounds of each axis), so A_c = R A P is three one-axis
// products, x, then y, then z, each on a grid coarsened along the axes already done.  An
// output entry (node I, offset O) sums over the admissible (dn, dm) pairs of its axis only
// (at most 7, against up to 343 triples in k_galerkin_l1p): 2197 instead of 5 x 13^3 terms per
// coarse node summed over its 27 offsets, with the first pass on the fine grid coalesced.  Same
// operator, other rounding order.
template <int AX>
__global__ void __launch_bounds__(128) k_galerkin_axis(GridDev<3> gi, GridDev<3> go, const double* __restrict__ Si,
                                                       double* __restrict__ So) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long No = go.n_nodes, Ni = gi.n_nodes;
    if (tid >= No * 27) return;
    const int o = (int)(tid / No);
    const long long I = tid - (long long)o * No;
    int c[3];
    ndec(go, I, c[0], c[1], c[2]);
    const int oo[3] = {o % 3 - 1, (o / 3) % 3 - 1, o / 9 - 1};
    const int Ia = c[AX], Ta = Ia + oo[AX];
    double blk[9];
#pragma unroll
    for (int a = 0; a < 9; a++) blk[a] = 0.0;
    if (Ta >= 0 && Ta < go.nn[AX]) {
        const int np = c_npairs[oo[AX] + 1];
        for (int p = 0; p < np; p++) {
            const int dn = c_pairs[oo[AX] + 1][p][0], dm = c_pairs[oo[AX] + 1][p][1];
            const int na = 2 * Ia + dn, ma = 2 * Ta + dm;
            if (na < 0 || na >= gi.nn[AX] || ma < 0 || ma >= gi.nn[AX]) continue;
            const double w = (dn != 0 ? 0.5 : 1.0) * (dm != 0 ? 0.5 : 1.0);
            int ci[3] = {c[0], c[1], c[2]}, ri[3] = {oo[0], oo[1], oo[2]};
            ci[AX] = na;
            ri[AX] = ma - na;
            const long long n = nidx(gi, ci[0], ci[1], ci[2]);
            const int on = (ri[0] + 1) + 3 * (ri[1] + 1) + 9 * (ri[2] + 1);
#pragma unroll
            for (int a = 0; a < 9; a++) blk[a] += w * Si[((long long)(on * 9 + a)) * Ni + n];
        }
        const int nn = go.nn[AX];
        const double s = 1.0 / (((Ia == 0 || Ia == nn - 1) ? 1.5 : 2.0) * ((Ta == 0 || Ta == nn - 1) ? 1.5 : 2.0));
#pragma unroll
        for (int a = 0; a < 9; a++) blk[a] *= s;
    }
#pragma unroll
    for (int a = 0; a < 9; a++) So[((long long)(o * 9 + a)) * No + I] = blk[a];
}

static bool g_pairs_ready = false;
static int init_pairs() {
    if (g_pairs_ready) return PF_OK;
    int pairs[3][7][2] = {};
    int np[3] = {0, 0, 0};
    for (int o = -1; o <= 1; o++)
        for (int dn = -1; dn <= 1; dn++)
            for (int dm = -1; dm <= 1; dm++) {
                const int r = 2 * o + dm - dn;
                if (r < -1 || r > 1) continue;
                pairs[o + 1][np[o + 1]][0] = dn;
                pairs[o + 1][np[o + 1]][1] = dm;
                np[o + 1]++;
            }
    PF_CUDA(cudaMemcpyToSymbol(c_pairs, pairs, sizeof(pairs)));
    PF_CUDA(cudaMemcpyToSymbol(c_npairs, np, sizeof(np)));
    g_pairs_ready = true;
    return PF_OK;
}

int launch_galerkin_l1p(const Grid& gf, const double* Af, double* Ac, cudaStream_t st) {
    int s = init_pairs();
    if (s) return s;
    const Grid gc = coarse_grid(gf);
    const int NB = gf.dim == 3 ? 27 : 9;
    const unsigned nb = (unsigned)((gc.n_nodes * NB + 127) / 128);
    pf::count_launch();
    if (gf.dim == 3)
        k_galerkin_l1p<3><<<nb, 128, 0, st>>>(gdev<3>(gf), gdev<3>(gc), Af, Ac);
    else
        k_galerkin_l1p<2><<<nb, 128, 0, st>>>(gdev<2>(gf), gdev<2>(gc), Af, Ac);
    PF_LAUNCH_CHECK("galerkin l1p launch");
    return PF_OK;
}

// the fine grid with one axis coarsened (element count halved, floored)
static Grid coarsen_axis(const Grid& g, int ax) {
    int nel[3] = {g.nel[0], g.nel[1], g.nel[2]};
    nel[ax] /= 2;
    return make_grid(g.dim, nel);
}

long long galerkin_sep_scratch(const Grid& gf) {
    if (gf.dim != 3) return 0;
    const Grid g1 = coarsen_axis(gf, 0), g2 = coarsen_axis(g1, 1);
    return 243LL * (g1.n_nodes + g2.n_nodes);
}

int launch_galerkin_sep(const Grid& gf, const double* Af, double* Ac, double* scratch, cudaStream_t st) {
    if (gf.dim != 3) return launch_galerkin_l1p(gf, Af, Ac, st);
    int s = init_pairs();
    if (s) return s;
    const Grid g1 = coarsen_axis(gf, 0), g2 = coarsen_axis(g1, 1), gc = coarsen_axis(g2, 2);
    double* S1 = scratch;
    double* S2 = scratch + 243LL * g1.n_nodes;
    auto nb = [](const Grid& g) { return (unsigned)((g.n_nodes * 27 + 127) / 128); };
    pf::count_launch(3);
    k_galerkin_axis<0><<<nb(g1), 128, 0, st>>>(gdev<3>(gf), gdev<3>(g1), Af, S1);
    k_galerkin_axis<1><<<nb(g2), 128, 0, st>>>(gdev<3>(g1), gdev<3>(g2), S1, S2);
    k_galerkin_axis<2><<<nb(gc), 128, 0, st>>>(gdev<3>(g2), gdev<3>(gc), S2, Ac);
    PF_LAUNCH_CHECK("separable galerkin launch");
    return PF_OK;
}

// ---------------------------------------------------------------------------------------
// stencil diagonal -> inverse diagonal, precision conversion, dense export
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void k_stencil_dinv(long long N, int dim, const double* __restrict__ A, T* __restrict__ dinv) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * dim) return;
    const long long n = t / dim;
    const int a = (int)(t - n * dim);
    const int oc = dim == 3 ? 13 : 4, BS = dim * dim;
    dinv[t] = (T)(1.0 / A[((long long)(oc * BS + a * dim + a)) * N + n]);
}

template <typename T>
int launch_stencil_dinv(const Grid& g, const double* A, T* dinv, cudaStream_t st) {
    const long long n = g.n_nodes * g.dim;
    pf::count_launch();
    k_stencil_dinv<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g.n_nodes, g.dim, A, dinv);
    PF_LAUNCH_CHECK("stencil dinv launch");
    return PF_OK;
}
template int launch_stencil_dinv<double>(const Grid&, const double*, double*, cudaStream_t);
template int launch_stencil_dinv<float>(const Grid&, const double*, float*, cudaStream_t);

template <int DIM>
__global__ void k_stencil_to_dense(GridDev<DIM> g, const double* __restrict__ A, double* __restrict__ M, long long ld) {
    constexpr int NB = DIM == 3 ? 27 : 9, BS = DIM * DIM;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long N = g.n_nodes;
    if (t >= N * NB * BS) return;
    const long long n = t % N;
    const int ob = (int)(t / N);
    const int o = ob / BS, ab = ob % BS, a = ab / DIM, b = ab % DIM;
    int i, j, k;
    ndec(g, n, i, j, k);
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = DIM == 3 ? o / 9 - 1 : 0;
    if (!nok(g, i + ox, j + oy, k + oz)) return;
    const long long m = nidx(g, i + ox, j + oy, k + oz);
    M[(n * DIM + a) * ld + m * DIM + b] = A[t];
}

int launch_stencil_to_dense(const Grid& g, const double* A, double* M, long long ld, cudaStream_t st) {
    const int NB = g.dim == 3 ? 27 : 9;
    const long long n = g.n_nodes * NB * g.dim * g.dim;
    pf::count_launch();
    if (g.dim == 3)
        k_stencil_to_dense<3><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(gdev<3>(g), A, M, ld);
    else
        k_stencil_to_dense<2><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(gdev<2>(g), A, M, ld);
    PF_LAUNCH_CHECK("stencil to dense launch");
    return PF_OK;
}

__global__ void k_d2f(long long n, const double* __restrict__ a, float* __restrict__ b) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}
int launch_d2f(long long n, const double* a, float* b, cudaStream_t st) {
    long long nb = (n + 255) / 256;
    if (nb > 4 * kNumSM * 8) nb = 4 * kNumSM * 8;
    if (nb < 1) nb = 1;
    pf::count_launch();
    k_d2f<<<(unsigned)nb, 256, 0, st>>>(n, a, b);
    PF_LAUNCH_CHECK("d2f launch");
    return PF_OK;
}

__global__ void k_d2bf(long long n, const double* __restrict__ a, __nv_bfloat16* __restrict__ b) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = __double2bfloat16(a[i]);
}
int launch_d2bf(long long n, const double* a, __nv_bfloat16* b, cudaStream_t st) {
    long long nb = (n + 255) / 256;
    if (nb > 4 * kNumSM * 8) nb = 4 * kNumSM * 8;
    if (nb < 1) nb = 1;
    pf::count_launch();
    k_d2bf<<<(unsigned)nb, 256, 0, st>>>(n, a, b);
    PF_LAUNCH_CHECK("d2bf launch");
    return PF_OK;
}

}  // namespace pf
