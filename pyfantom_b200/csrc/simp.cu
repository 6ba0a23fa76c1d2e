// SIMP element-wise steps, deterministic reductions and the OC update.
//
// penalize / penalize_grad follow pyFANTOM/Problem/CUDA/MinimumCompliance.py:305-324 and
// :351-367 (single material): optional Heaviside projection
//   H(r) = (tanh(b eta) + tanh(b (r - eta))) / (tanh(b eta) + tanh(b (1 - eta))),
//   E = clip(clip(H^p, void, 1) * E_mul, void, inf),   dE = p H^(p-1) H'(r) E_mul.
//
// OC (pyFANTOM/Optimizers/CUDA/OC.py:67-129) bisects the Lagrange multiplier with the host
// testing g(x_new) after every step.  Here a pass evaluates the constraint at many midpoints
// in one sweep over the elements (one partial sum per midpoint and block); its last block
// adds the partial sums and replays the sequential decisions with the reference's stopping
// rule; the midpoints are formed exactly as the sequential loop forms them, so the sequence
// of (l1, l2) is the same.  See k_oc_pass for the single constraint; with several constraints
// (k_oc_eval, k_oc_step_multi) each pass covers the 31 midpoints of five bisection levels.
#include <cmath>
#include <cstddef>

#include <type_traits>
#include <vector>

#include "common.cuh"

namespace pf {

constexpr int kRT = 256;

__device__ __forceinline__ void heavy(double r, double beta, double eta, double* h, double* dh) {
    const double den = tanh(beta * eta) + tanh(beta * (1.0 - eta));
    const double t = tanh(beta * (r - eta));
    *h = (tanh(beta * eta) + t) / den;
    *dh = beta * (1.0 - t * t) / den;
}

// r^e: pow, but for the exponents 0 .. 3 of a penalty of 1, 2 or 3 and its derivative, products
// (at most two roundings, within pow's own error; pow costs some hundred instructions)
template <int EXP>
__device__ __forceinline__ double simp_pow(double r, double e) {
    if (EXP == 0) return 1.0;
    if (EXP == 1) return r;
    if (EXP == 2) return r * r;
    if (EXP == 3) return r * r * r;
    return pow(r, e);
}

// PEN: the penalty if it is 1, 2 or 3, else 0.  Bound by FP64 arithmetic: 128x64x64 elements with
// projection 6.5 us against 12.3 us with pow and three tanh for each element.  The two constant
// tanh are formed here, once per block, and not on the host: at rho = 0 the projection is
// tanh(beta eta) + tanh(-beta eta), which cancels to 0 only if both come from one function.
template <int PEN>
__global__ void k_penalize(long long n, const double* __restrict__ rho, pf_simp_params P, double* __restrict__ E,
                           double* __restrict__ dE) {
    pdl_wait();
    pdl_trigger();
    __shared__ double s_th, s_den;
    if (P.heavyside) {
        if (threadIdx.x == 0) {
            s_th = tanh(P.beta * P.eta);
            s_den = s_th + tanh(P.beta * (1.0 - P.eta));
        }
        __syncthreads();
    }
    const double th = P.heavyside ? s_th : 0.0, den = P.heavyside ? s_den : 1.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double r = rho[i], dh = 1.0;
        if (P.heavyside) {
            const double t = tanh(P.beta * (r - P.eta));
            r = (th + t) / den;
            dh = P.beta * (1.0 - t * t) / den;
        }
        if (E) {
            double e = simp_pow<PEN ? PEN : 9>(r, P.penalty);
            e = fmin(fmax(e, P.void_value), 1.0) * P.E_mul;
            E[i] = fmax(e, P.void_value);
        }
        if (dE) dE[i] = P.penalty * simp_pow<PEN ? PEN - 1 : 9>(r, P.penalty - 1.0) * dh * P.E_mul;
    }
}

// Multi-material SIMP (pyFANTOM/Problem/CUDA/MinimumCompliance.py:326-349, 369-411): with
// a_i = H(rho_i)^p and b_i = 1 - a_i,
//   E = max(sum_i E_mul_i a_i prod_{j != i} b_j, void)
//   dE/drho_k = H'(rho_k) sum_i E_mul_i { p H^(p-1)(rho_k) prod_{j != k} b_j            (i = k)
//                                         -p H^(p-1)(rho_k) a_i prod_{j != i, k} b_j     (i != k) }
// rho and dE are material-major [n_material][n_elements] (the design-variable order).
constexpr int kMaxMaterials = 8;
struct MultiEmul {
    double v[kMaxMaterials];
};
__global__ void k_penalize_multi(long long ne, int nm, const double* __restrict__ rho, pf_simp_params P, MultiEmul em,
                                 double* __restrict__ E, double* __restrict__ dE) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
        double a[kMaxMaterials], b[kMaxMaterials], da[kMaxMaterials];
        for (int k = 0; k < nm; k++) {
            double r = rho[k * ne + e], dh = 1.0;
            if (P.heavyside) heavy(rho[k * ne + e], P.beta, P.eta, &r, &dh);
            a[k] = pow(r, P.penalty);
            b[k] = 1.0 - a[k];
            da[k] = P.penalty * pow(r, P.penalty - 1.0) * dh;
        }
        if (E) {
            double s = 0.0;
            for (int i = 0; i < nm; i++) {
                double t = a[i];
                for (int j = 0; j < nm; j++)
                    if (j != i) t *= b[j];
                s += em.v[i] * t;
            }
            E[e] = fmax(s, P.void_value);
        }
        if (dE) {
            for (int k = 0; k < nm; k++) {
                double s = 0.0;
                for (int i = 0; i < nm; i++) {
                    double t = i == k ? da[k] : -da[k] * a[i];
                    for (int j = 0; j < nm; j++)
                        if (j != i && j != k) t *= b[j];
                    s += em.v[i] * t;
                }
                dE[k * ne + e] = s;
            }
        }
    }
}

__global__ void k_mul(long long n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = a[i] * b[i];
}

static unsigned grid_for(long long n) {
    long long nb = (n + kRT - 1) / kRT;
    if (nb > 8LL * kNumSM) nb = 8LL * kNumSM;
    return (unsigned)(nb < 1 ? 1 : nb);
}

__global__ void __launch_bounds__(kRT) k_dot_part(long long n, const double* __restrict__ a, const double* __restrict__ b,
                                                  double* partials) {
    __shared__ double s_red[kRT / 32];
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        s += a[i] * b[i];
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kRT) k_sum_to(const double* partials, int np, double* out) {
    __shared__ double s_red[kRT / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) s += partials[i];
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) *out = s;
}

// ---------------------------------------------------------------------------------------
// OC
// ---------------------------------------------------------------------------------------
constexpr int kOcTree = 31;  // midpoints of 5 bisection levels
constexpr int kOcPasses = 24;

struct OcState {
    double l1, l2, lmid, abs_sum, change2, g[kOcTree], lam[kOcTree];
    int done, steps, allzero, pad;
};

__global__ void __launch_bounds__(kRT) k_oc_prep(long long n, const double* __restrict__ x, const double* __restrict__ df,
                                                 const double* __restrict__ dg, double* __restrict__ ocp,
                                                 double* partials) {
    __shared__ double s_red[kRT / 32];
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double t = fmax(-df[i] / dg[i], 0.0);
        double q = sqrt(t);
        if (q != q) q = 0.0;
        const double v = x[i] * q;
        ocp[i] = v;
        s += fabs(v);
    }
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

__device__ void oc_tree(OcState* S) {
    // heap layout: node t covers (a_t, b_t); its midpoint is (a_t + b_t) / 2; the left
    // child (a_t, m_t) follows g(m_t) <= 0 (l2 = m_t), the right child (m_t, b_t) otherwise
    double a[kOcTree], b[kOcTree];
    a[0] = S->l1;
    b[0] = S->l2;
    for (int t = 0; t < kOcTree; t++) {
        const double m = (a[t] + b[t]) / 2.0;
        S->lam[t] = m;
        if (2 * t + 2 < kOcTree) {
            a[2 * t + 1] = a[t];
            b[2 * t + 1] = m;
            a[2 * t + 2] = m;
            b[2 * t + 2] = b[t];
        }
    }
}

__device__ __forceinline__ double oc_xnew(double xi, double oc, double lam, double move) {
    const double xu = fmin(fmax(xi + move, 0.0), 1.0), xl = fmin(fmax(xi - move, 0.0), 1.0);
    return fmax(0.0, fmax(xl, fmin(1.0, fmin(xu, oc / lam))));
}

__global__ void __launch_bounds__(kRT) k_oc_eval(long long n, const double* __restrict__ x, const double* __restrict__ ocp,
                                                 const double* __restrict__ dg, double move, const OcState* S,
                                                 double* partials) {
    __shared__ double s_lam[kOcTree];
    __shared__ double s_part[kRT / 32][kOcTree];
    if (S->done) return;
    if (threadIdx.x < kOcTree) s_lam[threadIdx.x] = S->lam[threadIdx.x];
    __syncthreads();
    const bool allzero = S->allzero;
    double acc[kOcTree];
#pragma unroll
    for (int t = 0; t < kOcTree; t++) acc[t] = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double xi = x[i], oc = allzero ? 1e-3 : ocp[i], d = dg[i];
#pragma unroll
        for (int t = 0; t < kOcTree; t++) acc[t] += d * oc_xnew(xi, oc, s_lam[t], move);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int t = 0; t < kOcTree; t++) {
        const double v = warp_sum(acc[t]);
        if (l == 0) s_part[w][t] = v;
    }
    __syncthreads();
    if (threadIdx.x < kOcTree) {
        double s = 0.0;
        for (int k = 0; k < kRT / 32; k++) s += s_part[k][threadIdx.x];
        partials[(long long)blockIdx.x * kOcTree + threadIdx.x] = s;
    }
}

__global__ void __launch_bounds__(kRT) k_oc_write(long long n, const double* __restrict__ x, const double* __restrict__ ocp,
                                                  double move, const OcState* S, double* __restrict__ xnew,
                                                  double* partials) {
    __shared__ double s_red[kRT / 32];
    const double lam = S->lmid;
    const bool allzero = S->allzero;
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double v = oc_xnew(x[i], allzero ? 1e-3 : ocp[i], lam, move);
        xnew[i] = v;
        const double d = x[i] - v;
        s += d * d;
    }
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// Several volume constraints (one per material, variables material-major): the reference
// bisects all multipliers in lockstep while any of them is unconverged (OC.py:111-127),
// so every multiplier takes the same number of steps.  One OcState per material; the
// evaluation pass runs per material segment, this kernel replays the lockstep decisions.
struct MultiVf {
    double v[kMaxMaterials];
};
__global__ void __launch_bounds__(32) k_oc_step_multi(const double* partials, int np, int nm, MultiVf vf, OcState* S) {
    if (S[0].done) return;
    const int t = threadIdx.x;
    for (int k = 0; k < nm; k++) {
        if (t < kOcTree) {
            double s = 0.0;
            const double* pk = partials + (size_t)k * np * kOcTree;
            for (int b = 0; b < np; b++) s += pk[(long long)b * kOcTree + t];
            S[k].g[t] = s - vf.v[k];
        }
    }
    __syncwarp();
    if (t == 0) {
        int node[kMaxMaterials];
        for (int k = 0; k < nm; k++) node[k] = 0;
        bool done = false;
        for (int d = 0; d < 5 && !done; d++) {
            bool any = false;
            for (int k = 0; k < nm; k++) any |= (S[k].l2 - S[k].l1) / (S[k].l2 + S[k].l1) > 1e-8;
            if (!any) {
                done = true;
                break;
            }
            for (int k = 0; k < nm; k++) {
                const double lmid = S[k].lam[node[k]];
                S[k].lmid = lmid;
                S[k].steps += 1;
                if (S[k].g[node[k]] <= 0.0) {
                    S[k].l2 = lmid;
                    node[k] = 2 * node[k] + 1;
                } else {
                    S[k].l1 = lmid;
                    node[k] = 2 * node[k] + 2;
                }
            }
        }
        if (!done) {
            bool any = false;
            for (int k = 0; k < nm; k++) any |= (S[k].l2 - S[k].l1) / (S[k].l2 + S[k].l1) > 1e-8;
            done = !any;
        }
        for (int k = 0; k < nm; k++) {
            S[k].done = done;
            if (!done) oc_tree(&S[k]);
        }
    }
}

__global__ void __launch_bounds__(kRT) k_oc_init_multi(const double* partials, int np, int nm, OcState* S) {
    __shared__ double s_red[kRT / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) s += partials[i];
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) {
        for (int k = 0; k < nm; k++) {
            S[k].abs_sum = s;
            S[k].allzero = s == 0.0;
            S[k].l1 = 1e-9;
            S[k].l2 = 1e9;
            S[k].lmid = 0.0;
            S[k].done = 0;
            S[k].steps = 0;
            S[k].change2 = 0.0;
            oc_tree(&S[k]);
        }
    }
}

// ---------------------------------------------------------------------------------------
// OC with one constraint
// ---------------------------------------------------------------------------------------
// The sequential loop starts with the bracket [1e-9, 1e9]; as long as g(mid) <= 0 the next
// midpoint is (1e-9 + mid) / 2.  These midpoints (the spine) are known in advance.  For
// dg >= 0 the volume g falls with the multiplier, so the first spine point with g > 0 is found
// in two passes: every 11th spine point (fused with the computation of ocP), then the ten
// between two of them.  The bracket then spans a factor of two, and each further pass covers
// the 15 midpoints of four bisection levels (31 of five need more registers than two blocks
// per SM leave): 9 passes in all.  Within a pass an element whose x_new sits on the same
// bound (or on neither) for the whole bracket adds one term instead of 15; after the first
// pass or two of the tree almost every element does.  Where dg is not a finite number >= 0,
// or ocP vanishes everywhere (x_new = 1e-3 / lambda), every pass covers four levels from the
// start: more passes, the same sequence.
// In the sums the reciprocal of the midpoint replaces the division (x_new itself is divided): two
// roundings per term instead of one, but x_new, lambda and the steps of 100 runs over 16 to 126
// elements across are bitwise those of the division.
// No unit is at its limit (ncu, 192x96x96): the first two passes issue in 53 % of the cycles with 16
// warps per SM (ALU pipe 41 and 48 %: the selects of the two comparisons; FP64 pipe 37 and 34 %; DRAM
// 19 %), the next two wait for x, ocP and dg (24 B per element, from L2 up to about 4 M elements), the
// list passes are a chain of latencies (issue 19 %, 12 us cold).  1720 -> 168 us.
constexpr int kOcStride = 11;
constexpr int kOcMid = 15;  // midpoints of four bisection levels

struct OcSpine {
    int n;
    double m[96];
};

struct OcRun {
    double change2, lmid;
    int steps, done;
    double l1, l2, blo, bhi;  // bracket; smallest and largest midpoint of the pass
    int mode;                 // 0 four levels of the tree, 1 coarse spine, 2 fine spine
    int ne, base, hipos;      // midpoints of the pass; fine spine: its first index, g > 0 behind it
    int allzero, flags;       // flags: 1 some dg not finite >= 0, 2 some ocP != 0
    int listed;               // 1: the warps hold lists of the elements still undecided
    unsigned count;           // blocks of the running pass that have finished
    double lam[kOcMid];
};
static_assert(sizeof(OcRun) <= sizeof(OcState), "OcRun shares the workspace of OcState");

// one element's terms of the constraint at NE midpoints; true if they differ by more than a
// common constant (cst) or a common constant over the multiplier (lin)
template <int NE>
__device__ __forceinline__ bool oc_accumulate(double xi, double oc, double d, double move, const double* s_r, double rlo,
                                              double rhi, double& cst, double& lin, double (&acc)[kOcMid]) {
    const double xu = fmin(fmax(xi + move, 0.0), 1.0), xl = fmin(fmax(xi - move, 0.0), 1.0);
    const double vmax = oc * rlo, vmin = oc * rhi;  // oc over the smallest and largest midpoint
    const bool up = vmin >= xu, low = vmax <= xl, mid = vmin >= xl && vmax <= xu;
    if (up || low) {
        cst += d * (up ? xu : xl);
        return false;
    }
    if (mid) {
        lin += d * oc;
        return false;
    }
#pragma unroll
    for (int t = 0; t < NE; t++) {
        double v = oc * s_r[t];
        v = v < xu ? v : xu;  // as fmin and fmax, a NaN gives the bound
        v = v > xl ? v : xl;
        acc[t] += d * v;
    }
    return true;
}

// decisions after a pass (one block; g[0..ne) in shared memory); writes the next midpoints
__device__ void oc_decide(OcRun* S, const OcSpine& sp, const double* g, int mode, int ne, int base, int hipos, int flags,
                          const double* s_lam) {
    __shared__ int s_next;  // next mode, -1: done
    if (threadIdx.x == 0) {
        int next = 0;
        if (mode == 1) {
            S->allzero = !(flags & 2);
            if ((flags & 1) || !(flags & 2)) {
                S->l1 = 1e-9, S->l2 = 1e9, S->lmid = 0.0, S->steps = 0;
            } else {
                int j = 0;
                while (j < ne && g[j] <= 0.0) j++;
                S->base = j * kOcStride;
                S->hipos = j < ne;
                S->ne = j < ne ? kOcStride - 1 : sp.n - j * kOcStride;
                next = 2;
            }
        } else if (mode == 2) {
            int q = 0;
            while (q < ne && g[q] <= 0.0) q++;
            if (q == ne && !hipos) {  // g <= 0 down to the end of the bisection
                S->l1 = 1e-9, S->l2 = S->lmid = sp.m[sp.n - 1], S->steps = sp.n;
            } else {
                const int k = base + q;
                S->l1 = S->lmid = sp.m[k];
                S->l2 = k > 0 ? sp.m[k - 1] : 1e9;
                S->steps = k + 1;
            }
        } else {
            int node = 0;
            double l1 = S->l1, l2 = S->l2, lmid = S->lmid;
            int steps = S->steps;
            for (int d = 0; d < 4; d++) {
                if (!((l2 - l1) / (l2 + l1) > 1e-8)) break;
                lmid = s_lam[node];
                steps++;
                if (g[node] <= 0.0) {
                    l2 = lmid;
                    node = 2 * node + 1;
                } else {
                    l1 = lmid;
                    node = 2 * node + 2;
                }
            }
            S->l1 = l1, S->l2 = l2, S->lmid = lmid, S->steps = steps;
        }
        if (next == 0) {
            const double l1 = S->l1, l2 = S->l2;
            S->done = !((l2 - l1) / (l2 + l1) > 1e-8);
            S->ne = kOcMid;
            S->blo = l1, S->bhi = l2;
        } else {
            S->blo = sp.m[S->base + S->ne - 1 + (S->ne == 0)], S->bhi = sp.m[S->base];
        }
        S->mode = next;
        S->count = 0;
        s_next = next;
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= kOcMid) return;
    if (s_next == 2) {
        if (t < S->ne) S->lam[t] = sp.m[S->base + t];
        return;
    }
    // heap layout: node t covers (a, b), its midpoint is (a + b) / 2; the left child (a, mid)
    // follows g(mid) <= 0 (l2 = mid), the right child (mid, b) otherwise
    double a = S->l1, b = S->l2, m = (a + b) / 2.0;
    const int depth = 31 - __clz(t + 1);
    for (int d = depth - 1; d >= 0; d--) {
        if (((t + 1) >> d) & 1)
            a = m;
        else
            b = m;
        m = (a + b) / 2.0;
    }
    S->lam[t] = m;
}

// ints of x_new for each warp's list (even: the list starts with two sums)
__host__ __device__ inline int oc_list_room(long long n, unsigned nb) { return (int)(2 * n / ((long long)nb * (kRT / 32))) & ~1; }

// KIND 0: the first pass; 1: any later pass over all elements; 2: a pass over the warps' lists
// (does nothing before they are built), a kernel of its own so that its few instructions are
// not fetched between the unrolled sweeps of the others
template <int KIND>
__global__ void __launch_bounds__(kRT, 2) k_oc_pass(long long n, const double* __restrict__ x, const double* __restrict__ df,
                                                 const double* __restrict__ dg, double* __restrict__ ocp, double move,
                                                 double vf, const __grid_constant__ OcSpine sp, OcRun* S,
                                                 double* partials, int* lists) {
    pdl_wait();
    pdl_trigger();
    constexpr bool FIRST = KIND == 0;
    constexpr int NWp = kRT / 32;
    __shared__ double s_lam[kOcMid], s_r[kOcMid], s_g[kOcMid];
    __shared__ double s_part[NWp][kOcMid + 2];
    __shared__ int s_last;
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    // the state in one round of loads
    const int done = FIRST ? 0 : S->done, mode = FIRST ? 1 : S->mode, ne = FIRST ? sp.n / kOcStride : S->ne;
    const int base = FIRST ? 0 : S->base, hipos = FIRST ? 0 : S->hipos, inlist = FIRST ? 0 : S->listed;
    const double lam = FIRST ? (tid < ne ? sp.m[kOcStride * tid + kOcStride - 1] : 1.0) : S->lam[tid < kOcMid ? tid : 0];
    const double blo0 = FIRST ? 1.0 : S->blo, bhi0 = FIRST ? 1.0 : S->bhi;
    const bool allzero = FIRST ? false : S->allzero != 0;
    if (done || (KIND == 2 && !inlist)) return;
    if (tid < ne) {
        const double v = lam;
        s_lam[tid] = v;
        s_r[tid] = 1.0 / v;
    } else if (tid < kOcMid) {
        s_lam[tid] = 1.0;
        s_r[tid] = 1.0;
    }
    __syncthreads();
    const double blo = FIRST ? s_lam[ne - 1] : blo0, bhi = FIRST ? s_lam[0] : bhi0;
    const double rlo = 1.0 / blo, rhi = 1.0 / bhi;
    double acc[kOcMid], cst = 0.0, lin = 0.0;
#pragma unroll
    for (int t = 0; t < kOcMid; t++) acc[t] = 0.0;
    int flags = 0;
    // warp-uniform loop over runs of 32 elements, several of them loaded ahead of their use
    const long long wstep = (long long)gridDim.x * kRT, w0 = (long long)blockIdx.x * kRT + w * 32;
    int listed = 0;  // entries of this warp's list of undecided elements
    const int lcap = oc_list_room(n, gridDim.x);
    int* seg = lists ? lists + ((long long)blockIdx.x * NWp + w) * lcap : nullptr;
    auto sweep = [&](auto NEc, bool build) {
        constexpr int NE = decltype(NEc)::value, kOcBatch = 4;
        for (long long k0 = w0; k0 < n; k0 += kOcBatch * wstep) {
            double xv[kOcBatch], ov[kOcBatch], dv[kOcBatch];
#pragma unroll
            for (int q = 0; q < kOcBatch; q++) {
                const long long i = k0 + q * wstep + l;
                const bool ok = i < n;
                xv[q] = ok ? x[i] : 0.0;
                dv[q] = ok ? dg[i] : 0.0;
                ov[q] = ok ? (FIRST ? df[i] : ocp[i]) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < kOcBatch; q++) {
                const long long i = k0 + q * wstep + l;
                const bool ok = i < n;
                double oc = ov[q];
                if constexpr (FIRST) {
                    double r = sqrt(fmax(-oc / dv[q], 0.0));
                    if (r != r) r = 0.0;
                    oc = ok ? xv[q] * r : 0.0;
                    if (ok) ocp[i] = oc;
                    if (!(dv[q] >= 0.0) || isinf(dv[q])) flags |= 1;
                    if (oc != 0.0) flags |= 2;
                } else if (allzero && ok) {
                    oc = 1e-3;
                }
                const bool act = oc_accumulate<NE>(xv[q], oc, dv[q], move, s_r, rlo, rhi, cst, lin, acc);
                if (build) {
                    const unsigned m = __ballot_sync(0xffffffffu, act);
                    if (act) seg[6 + listed + __popc(m & ((1u << l) - 1u))] = (int)i;
                    listed += __popc(m);
                }
            }
        }
    };
    const bool build = KIND == 1 && lists && mode == 0 && !inlist && bhi < 1.5 * blo;
    if constexpr (FIRST) {
        sweep(std::integral_constant<int, kOcStride - 1>{}, false);
    } else if constexpr (KIND == 2) {
        // the sums of the elements decided for the bracket of the building pass, then the others
        double* head = reinterpret_cast<double*>(seg);
        const int cnt = seg[4];
        int next = 6 + l < lcap ? seg[6 + l] : 0;  // the first entry beside the count
        if (l == 0) cst = head[0], lin = head[1];
        for (int q = l; q < cnt; q += 32) {
            const int i = next;
            if (q + 32 < cnt) next = seg[6 + q + 32];
            oc_accumulate<kOcMid>(x[i], allzero ? 1e-3 : ocp[i], dg[i], move, s_r, rlo, rhi, cst, lin, acc);
        }
    } else if (mode == 2) {
        sweep(std::integral_constant<int, kOcStride - 1>{}, false);
    } else {
        sweep(std::integral_constant<int, kOcMid>{}, build);
    }
    cst = warp_sum(cst);
    lin = warp_sum(lin);
    if (l == 0) s_part[w][kOcMid] = cst, s_part[w][kOcMid + 1] = lin;
    if (build && l == 0) {
        double* head = reinterpret_cast<double*>(seg);
        head[0] = cst, head[1] = lin;
        seg[4] = listed;
    }
#pragma unroll
    for (int t = 0; t < kOcMid; t++) {
        if (t < ne) {  // uniform over the grid
            const double v = warp_sum(acc[t]);
            if (l == 0) s_part[w][t] = v;
        }
    }
    if (FIRST) flags = __reduce_or_sync(0xffffffffu, flags);
    if (FIRST && l == 0 && flags) atomicOr(&S->flags, flags);
    __syncthreads();
    if (tid < ne) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NWp; k++) s += s_part[k][tid] + s_part[k][kOcMid] + s_part[k][kOcMid + 1] * s_r[tid];
        partials[(long long)blockIdx.x * kOcMid + tid] = s;
    }
    // the last block to get here adds the partial sums (in block order) and decides
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&S->count, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    {  // thread (t, group): every 16th block's sum for midpoint t
        constexpr int G = kRT / 16, NL = (2 * kNumSM + G - 1) / G;  // at most 2 blocks per SM (oc_blocks)
        const int t = tid & 15, tc = t < ne ? t : 0, nbk = (int)gridDim.x;
        double part[NL], s = 0.0;  // all loads in flight together
#pragma unroll
        for (int q = 0; q < NL; q++) part[q] = __ldcg(partials + (long long)min((tid >> 4) + q * G, nbk - 1) * kOcMid + tc);
#pragma unroll
        for (int q = 0; q < NL; q++)
            if ((tid >> 4) + q * G < nbk) s += part[q];
        s += __shfl_xor_sync(0xffffffffu, s, 16);
        if (l < 16) s_part[w][t] = s;  // 17 columns a row
    }
    __syncthreads();
    if (tid < ne) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NWp; k++) s += s_part[k][tid];
        s_g[tid] = s - vf;
    }
    __syncthreads();
    if (build && tid == 0) S->listed = 1;
    oc_decide(S, sp, s_g, mode, ne, base, hipos, FIRST ? *(volatile int*)&S->flags : 0, s_lam);
}

// x_new and ||x_new - x||^2 (partial sums, added by the last block); without `force` only once
// the bisection has ended
__global__ void __launch_bounds__(kRT) k_oc_final(long long n, const double* x, const double* __restrict__ ocp, double move,
                                                  OcRun* S, int force, double* xnew, double* partials) {
    pdl_wait();
    pdl_trigger();
    __shared__ double s_red[kRT / 32];
    __shared__ int s_last;
    if (!force && !S->done) return;
    const double lam = S->lmid;
    const bool allzero = S->allzero != 0;
    double s = 0.0;
#pragma unroll 4
    for (long long i = (long long)blockIdx.x * kRT + threadIdx.x; i < n; i += (long long)gridDim.x * kRT) {
        const double xi = x[i], v = oc_xnew(xi, allzero ? 1e-3 : ocp[i], lam, move);
        xnew[i] = v;
        s += (xi - v) * (xi - v);
    }
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s;
        __threadfence();
        s_last = atomicAdd(&S->count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    s = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kRT) s += __ldcg(partials + b);
    s = block_sum<kRT>(s, s_red);
    if (threadIdx.x == 0) S->change2 = s, S->count = 0;
}

static OcSpine oc_spine() {
    OcSpine sp;
    sp.n = 0;
    const double l1 = 1e-9;
    for (double l2 = 1e9; (l2 - l1) / (l2 + l1) > 1e-8; l2 = sp.m[sp.n++]) sp.m[sp.n] = (l1 + l2) / 2.0;
    return sp;
}

static unsigned oc_blocks(long long n) {
    long long nb = (n + kRT - 1) / kRT;
    if (nb > 2LL * kNumSM) nb = 2LL * kNumSM;
    return (unsigned)(nb < 1 ? 1 : nb);
}

size_t oc_workspace(long long n) {
    return (size_t)n + (size_t)oc_blocks(n) * kOcTree + (sizeof(OcState) + 7) / 8 + 8;
}

int oc_update(long long n, const double* x, const double* df, const double* dg, double vf, double move,
              double* x_new, double* work, double* h_out, cudaStream_t st) {
    const unsigned nb = oc_blocks(n);
    double* ocp = work;
    double* partials = work + n;
    OcRun* S = reinterpret_cast<OcRun*>(partials + (size_t)nb * kOcTree);
    static const OcSpine sp = oc_spine();
    // until it is written, x_new holds the lists of undecided elements (unless it shares memory with x or
    // dg, which every pass reads, or is too short for each warp's whole share and the list's head)
    const long long share = 32 * ((n + (long long)nb * kRT - 1) / ((long long)nb * kRT));
    auto apart = [&](const double* a) { return (size_t)a + n * sizeof(double) <= (size_t)x_new || (size_t)x_new + n * sizeof(double) <= (size_t)a; };
    const bool own = apart(x) && apart(dg);
    int* lists = n < (1LL << 31) && own && share + 6 <= oc_list_room(n, nb) ? reinterpret_cast<int*>(x_new) : nullptr;
    PF_CUDA(cudaMemsetAsync(S, 0, sizeof(OcRun), st));
    auto passes = [&](int count, int list_passes) {
        for (int p = 0; p < count + list_passes; p++) {
            pf::count_launch();
            PF_CUDA(launch_pdl(p < count ? k_oc_pass<1> : k_oc_pass<2>, dim3(nb), dim3(kRT), 0, st, n, x, df, dg, ocp, move, vf, sp, S, partials, lists));
        }
        return (int)PF_OK;
    };
    auto final = [&](int force) {
        pf::count_launch();
        PF_CUDA(launch_pdl(k_oc_final, dim3(nb), dim3(kRT), 0, st, n, x, (const double*)ocp, move, S, force, x_new, partials));
        PF_LAUNCH_CHECK("oc launch");
        return (int)PF_OK;
    };
    int s;
    pf::count_launch();
    PF_CUDA(launch_pdl(k_oc_pass<0>, dim3(nb), dim3(kRT), 0, st, n, x, df, dg, ocp, move, vf, sp, S, partials, lists));
    // fine spine, then the 25 levels below a bracket of a factor of two, the first eight of them
    // over all elements; a caller that does not wait for the result gets the passes of the
    // general sequence (86 levels) too
    if ((s = lists ? passes(3, 5) : passes(8, 0)) || (!h_out && (s = passes(kOcPasses - 3, 0)))) return s;
    if ((s = final(h_out ? 0 : 1))) return s;
    if (h_out) {
        OcRun h;
        constexpr size_t head = offsetof(OcRun, l1);  // the results come first
        PF_CUDA(cudaMemcpyAsync(&h, S, head, cudaMemcpyDeviceToHost, st));
        PF_CUDA(cudaStreamSynchronize(st));
        if (!h.done) {
            if ((s = passes(kOcPasses - 3, 0)) || (s = final(1))) return s;
            PF_CUDA(cudaMemcpyAsync(&h, S, head, cudaMemcpyDeviceToHost, st));
            PF_CUDA(cudaStreamSynchronize(st));
        }
        h_out[0] = sqrt(h.change2);
        h_out[1] = h.lmid;
        h_out[2] = (double)h.steps;
        if (!h.done) return fail(PF_NOT_CONVERGED, "OC bisection did not terminate in %d steps", h.steps);
    }
    return PF_OK;
}

size_t oc_multi_workspace(long long ne, int nm) {
    const long long n = ne * nm;
    return (size_t)n + (size_t)oc_blocks(ne) * kOcTree * nm + (size_t)oc_blocks(n) +
           (sizeof(OcState) * nm + 7) / 8 + 8;
}

int oc_update_multi(long long ne, int nm, const double* x, const double* df, const double* dg, const double* vf,
                    double move, double* x_new, double* work, double* h_out, cudaStream_t st) {
    const long long n = ne * nm;
    const unsigned nb = oc_blocks(ne), nbn = oc_blocks(n);
    double* ocp = work;
    double* partials = work + n;                               // nm segments of nb * kOcTree
    double* sums = partials + (size_t)nb * kOcTree * nm;        // nbn
    OcState* S = reinterpret_cast<OcState*>(sums + nbn);
    MultiVf mv;
    for (int k = 0; k < nm; k++) mv.v[k] = vf[k];
    pf::count_launch(2);
    k_oc_prep<<<nbn, kRT, 0, st>>>(n, x, df, dg, ocp, sums);
    k_oc_init_multi<<<1, kRT, 0, st>>>(sums, nbn, nm, S);
    for (int p = 0; p < kOcPasses; p++) {
        for (int k = 0; k < nm; k++) {
            pf::count_launch();
            k_oc_eval<<<nb, kRT, 0, st>>>(ne, x + k * ne, ocp + k * ne, dg + k * ne, move, &S[k],
                                          partials + (size_t)k * nb * kOcTree);
        }
        pf::count_launch();
        k_oc_step_multi<<<1, 32, 0, st>>>(partials, nb, nm, mv, S);
    }
    for (int k = 0; k < nm; k++) {
        pf::count_launch();
        k_oc_write<<<nb, kRT, 0, st>>>(ne, x + k * ne, ocp + k * ne, move, &S[k], x_new + k * ne,
                                       partials + (size_t)k * nb * kOcTree);
    }
    PF_LAUNCH_CHECK("oc multi launch");
    if (h_out) {  // change^2: the per-block sums k_oc_write left in each material's segment
        std::vector<OcState> h(nm);
        std::vector<double> part((size_t)nb * kOcTree * nm);
        PF_CUDA(cudaMemcpyAsync(h.data(), S, sizeof(OcState) * nm, cudaMemcpyDeviceToHost, st));
        PF_CUDA(cudaMemcpyAsync(part.data(), partials, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, st));
        PF_CUDA(cudaStreamSynchronize(st));
        double c2 = 0.0;
        for (int k = 0; k < nm; k++)
            for (unsigned b = 0; b < nb; b++) c2 += part[(size_t)k * nb * kOcTree + b];
        h_out[0] = sqrt(c2);
        h_out[1] = h[0].lmid;
        h_out[2] = (double)h[0].steps;
        if (!h[0].done) return fail(PF_NOT_CONVERGED, "OC bisection did not terminate in %d steps", h[0].steps);
    }
    return PF_OK;
}

}  // namespace pf

using namespace pf;

extern "C" int pf_penalize_multi_f64(long long ne, int nm, const double* rho, const pf_simp_params* p,
                                     const double* h_E_mul, double* E, double* dE, void* stream) {
    if (ne < 0 || nm < 2 || nm > kMaxMaterials || !rho || !p || !h_E_mul || (!E && !dE))
        return fail(PF_BAD_ARG, "pf_penalize_multi_f64: bad argument (2..%d materials)", kMaxMaterials);
    MultiEmul em;
    for (int k = 0; k < nm; k++) em.v[k] = h_E_mul[k];
    count_launch();
    k_penalize_multi<<<grid_for(ne < 1 ? 1 : ne), kRT, 0, as_stream(stream)>>>(ne, nm, rho, *p, em, E, dE);
    PF_LAUNCH_CHECK("penalize multi launch");
    return PF_OK;
}

extern "C" size_t pf_oc_multi_workspace_size(long long ne, int nm) { return oc_multi_workspace(ne < 1 ? 1 : ne, nm); }

extern "C" int pf_oc_update_multi_f64(long long ne, int nm, const double* x, const double* df, const double* dg,
                                      const double* h_vf, double move, double* x_new, double* work, double* h_out,
                                      void* stream) {
    if (ne < 1 || nm < 1 || nm > kMaxMaterials || !x || !df || !dg || !h_vf || !x_new || !work)
        return fail(PF_BAD_ARG, "pf_oc_update_multi_f64: bad argument (1..%d materials)", kMaxMaterials);
    return oc_update_multi(ne, nm, x, df, dg, h_vf, move, x_new, work, h_out, as_stream(stream));
}

extern "C" int pf_penalize_f64(long long n, const double* rho, const pf_simp_params* p, double* E, double* dE,
                               void* stream) {
    if (n < 0 || !rho || !p || (!E && !dE)) return fail(PF_BAD_ARG, "pf_penalize_f64: bad argument");
    if (n == 0) return PF_OK;
    pf::count_launch();
    const double e = p->penalty;
    auto kernel = e == 1.0 ? k_penalize<1> : e == 2.0 ? k_penalize<2> : e == 3.0 ? k_penalize<3> : k_penalize<0>;
    PF_CUDA(launch_pdl(kernel, dim3(grid_for(n)), dim3(kRT), 0, as_stream(stream), n, rho, *p, E, dE));
    PF_LAUNCH_CHECK("penalize launch");
    return PF_OK;
}

extern "C" int pf_mul_f64(long long n, const double* a, const double* b, double* out, void* stream) {
    if (n < 0 || !a || !b || !out) return fail(PF_BAD_ARG, "pf_mul_f64: bad argument");
    if (n == 0) return PF_OK;
    pf::count_launch();
    k_mul<<<grid_for(n), kRT, 0, as_stream(stream)>>>(n, a, b, out);
    PF_LAUNCH_CHECK("mul launch");
    return PF_OK;
}

extern "C" size_t pf_dot_workspace_size(long long n) { return (size_t)grid_for(n < 1 ? 1 : n) + 1; }

extern "C" int pf_dot_f64(long long n, const double* a, const double* b, double* result, double* work, void* stream) {
    if (n < 0 || !a || !b || !result || !work) return fail(PF_BAD_ARG, "pf_dot_f64: bad argument");
    cudaStream_t st = as_stream(stream);
    const unsigned nb = grid_for(n < 1 ? 1 : n);
    pf::count_launch();
    k_dot_part<<<nb, kRT, 0, st>>>(n, a, b, work);
    pf::count_launch();
    k_sum_to<<<1, kRT, 0, st>>>(work, (int)nb, result);
    PF_LAUNCH_CHECK("dot launch");
    return PF_OK;
}

extern "C" size_t pf_oc_workspace_size(long long n) { return oc_workspace(n < 1 ? 1 : n); }

extern "C" int pf_oc_update_f64(long long n, const double* x, const double* df, const double* dg, double vf, double move,
                                double* x_new, double* work, double* h_out, void* stream) {
    if (n < 1 || !x || !df || !dg || !x_new || !work) return fail(PF_BAD_ARG, "pf_oc_update_f64: bad argument");
    if (!(move >= 0.0)) return fail(PF_BAD_ARG, "move must be >= 0");
    return oc_update(n, x, df, dg, vf, move, x_new, work, h_out, as_stream(stream));
}
