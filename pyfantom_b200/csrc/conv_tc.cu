// 3x3x3 convolution (forward, input gradient, weight gradient) on the tensor cores:
// implicit GEMM with tcgen05.mma, BF16 operands staged in shared memory from the FP32
// tensors, FP32 accumulation in tensor memory.
//
//   forward     D[o, co] = sum_k A[o, k] B[k, co],  k = ci*27 + t,
//               A[o, k] = x[n, ci, s*o + t - 1] (zero outside), B[k, co] = w[co, ci, t]
//               y[n, co, o] = D[o, co] + b[co] (ReLU optional)
//   input grad  D[v, ci] = sum_k A[v, k] B[k, ci],  k = co*27 + t,
//               A[v, k] = dy[n, co, (v - t + 1) / s] (where divisible and inside), B[k, ci] = w[co, ci, t]
//               dx[n, ci, v] = D[v, ci] (+= with accumulate)
//   weight grad D[m, co] = sum_k A[m, k] B[co, k] over k = (n, o), m = ci*27 + t plus a row of
//               ones (the bias gradient): A[m, k] = x[n, ci, s*o + t - 1], B[co, k] = dy[n, co, o]
// Layouts are those of the FP32 kernels (cnn.cu): [N][C][X][Y][Z], weights [Cout][Cin][27].
//
// The im2col matrix is never formed.  A CTA stages the source voxels of its output tile with
// their halo once per 16 reduction channels, as BF16 in groups of 8 channels (16 bytes per
// voxel and group, voxels consecutive along z).  In that layout 8 z-neighbours are one core
// matrix of the tensor cores' no-swizzle layouts, and moving by a voxel moves the start
// address by 16 bytes: the operand of each of the 27 taps is the same staged tile read from
// another start address.  In the weight gradient the reduction runs over voxels, so the same
// layout is the MN-major form of both operands (channels contiguous).  With stride 2 the
// voxels of a row are stored even ones first, so that a tap's voxels stay consecutive; the
// input gradient with stride 2 runs as eight kernels' worth of CTAs, one per parity of the
// input voxel, each with the one to eight taps that reach it.
// Producer warps gather (8 coalesced loads per 16 staged bytes), convert and store; one warp
// issues the MMAs; two buffers alternate, handed over by mbarriers.  Every wait on an mbarrier
// is bounded: past the limit the kernel records an error in `err`, skips the epilogue, and
// releases its tensor memory.
#include <cuda_bf16.h>

#include <cstdint>

#include "common.cuh"

#if __has_include(<cute/arch/mma_sm100_desc.hpp>)
#include <cute/arch/mma_sm100_desc.hpp>
#define PF_HAVE_CUTE_DESC 1
#endif

namespace pf {

constexpr long long kTcSpin = 1LL << 20;  // try_wait polls before giving up

// ---- descriptors -----------------------------------------------------------------------
// shared-memory matrix descriptor, K-major, no swizzle: start address, leading byte offset
// (between the two 8-element K halves of a 16-wide slice), stride byte offset (between
// 8-row groups), all in 16-byte units; version 1 (sm_100).
__host__ __device__ constexpr uint64_t umma_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
// (MN-major, no swizzle: the leading offset is between groups of 8 along K, the stride offset
// between groups of 8 along M or N)
// instruction descriptor of kind::f16: BF16 A and B, FP32 accumulator, M x N
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, bool mn_major = false) {
    return (1u << 4)                       // D format F32
           | (1u << 7) | (1u << 10)        // A, B format BF16
           | (mn_major ? 3u << 15 : 0u)    // A and B MN-major instead of K-major
           | ((uint32_t)(N >> 3) << 17)    // N / 8
           | ((uint32_t)(M >> 4) << 24);   // M / 16
}

// The encodings above against CuTe's bit-field definitions of the same descriptors (when
// its headers are on the include path): checked once on the host before the first launch.
static bool tc_encodings_match() {
#ifdef PF_HAVE_CUTE_DESC
    const uint32_t i64 = uint32_t(cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, 128, 64,
                                                              cute::UMMA::Major::K, cute::UMMA::Major::K>());
    const uint32_t i16 = uint32_t(cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, 128, 16,
                                                              cute::UMMA::Major::K, cute::UMMA::Major::K>());
    const uint32_t mn = uint32_t(cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, 64, 32,
                                                             cute::UMMA::Major::MN, cute::UMMA::Major::MN>());
    cute::UMMA::SmemDescriptor d;
    d.desc_ = 0;
    d.start_address_ = (uint16_t)(0x1230 >> 4);
    d.leading_byte_offset_ = (uint16_t)(2048 >> 4);
    d.stride_byte_offset_ = (uint16_t)(128 >> 4);
    d.version_ = 1;
    d.lbo_mode_ = 0;
    d.base_offset_ = 0;
    d.layout_type_ = uint8_t(cute::UMMA::LayoutType::SWIZZLE_NONE);
    return mn == umma_idesc_bf16(64, 32, true) && i64 == umma_idesc_bf16(128, 64) && i16 == umma_idesc_bf16(128, 16) &&
           uint64_t(d) == umma_smem_desc(0x1230, 2048, 128);
#else
    return true;
#endif
}

// ---- PTX wrappers ------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (long long i = 0; i < kTcSpin; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tc_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

struct ConvTcArgs {
    const float* src;  // forward, weight grad: x; input gradient: dy
    const float* w;    // forward, input gradient: weights; weight grad: dy
    const float* b;    // forward bias
    float* dst;        // forward: y, input gradient: dx
    int* err;
    int N, Cin, Cout, s, relu, accumulate;
    int X, Y, Z, Xo, Yo, Zo;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

constexpr size_t kTcMaxSmem = 220 * 1024;
constexpr size_t kTcHalfSmem = 113 * 1024 - 512;  // with the static shared memory, two CTAs per SM

// Tile of one CTA: rows of the product are the voxels q of a TX x 16 x 8 ZH box of the row
// grid, T = TX ZH accumulators of 128 rows; staged source: LX x LY x LZ voxels from
// q0 * step + org.
struct ConvTile {
    int QX, QY, QZ;            // row grid (largest parity class)
    int SX, SY, SZ;            // source grid
    int TX, ZH, ntx, nty, ntz;
    int LX, LY, LZ, even;      // even: z positions of even offset (0: stored in order)
    int step, org, ost;        // source step per row voxel, origin; row voxel q is output ost * q + parity
    int NT, ncols, nsplit;     // columns per CTA, tensor memory columns, column splits
    int nbuf;                  // staging buffers (1 when one chunk holds all reduction channels)
};

// shared-memory position of raw z offset r
__device__ __forceinline__ int tc_zpos(int r, int even) { return even ? (r & 1 ? even + (r >> 1) : r >> 1) : r; }

// 8 values at p, p + stride, ... as BF16 (zeros where !in; the first `cnt` of them): the loads
// are unconditional (an excluded voxel reads a valid address), so that all are in flight together
__device__ __forceinline__ uint4 tc_gather8(const float* __restrict__ p, long long stride, bool in, int cnt) {
    float v[8];
    if (cnt >= 8) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            v[j] = __ldg(p);
            p += stride;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = j < cnt ? __ldg(p + j * stride) : 0.f;
    }
    uint4 q;
    q.x = in ? pack_bf16(v[0], v[1]) : 0u;
    q.y = in ? pack_bf16(v[2], v[3]) : 0u;
    q.z = in ? pack_bf16(v[4], v[5]) : 0u;
    q.w = in ? pack_bf16(v[6], v[7]) : 0u;
    return q;
}

constexpr int kTcProd = 256;  // producer threads of the forward / input gradient (8 warps)

constexpr int kTcIssue = 4;    // issuing warps (one thread each; an accumulator has one issuer)

// MODE 0: forward, MODE 1: input gradient.  Warps 0..7 stage and run the epilogue, warps 8..11
// issue: a single thread needed about 400 cycles per MMA beside the producers, six times what the
// MMA itself takes.
template <int MODE>
__global__ void __launch_bounds__(kTcProd + 32 * kTcIssue, 2) k_conv_tc(ConvTcArgs a, ConvTile t) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t s_full[2], s_empty[2], s_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_ntap, s_tw[27], s_ts[27];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NCH = MODE == 0 ? a.Cout : a.Cin, KCH = MODE == 0 ? a.Cin : a.Cout;
    const int nvox = t.LX * t.LY * t.LZ;
    const size_t a_bytes = (size_t)nvox * 32, b_bytes = (size_t)27 * 32 * t.NT;
    uint8_t* sA = smem;
    uint8_t* sB = smem + t.nbuf * a_bytes;
    int* s_off = reinterpret_cast<int*>(sB + t.nbuf * b_bytes);
    // tile fastest, then column split, then sample (in one dimension: N * nsplit may exceed 65,535)
    const unsigned ntile = (unsigned)(t.ntx * t.nty * t.ntz), bt = blockIdx.x % ntile, bs = blockIdx.x / ntile;
    const int n = (int)(bs / t.nsplit), j0 = (int)(bs % t.nsplit) * t.NT;
    const int par = blockIdx.z, px = par & 1, py = (par >> 1) & 1, pz = par >> 2;  // parity class (stride-2 input gradient)
    const int bz = bt % t.ntz, by = (bt / t.ntz) % t.nty, bx = bt / (t.ntz * t.nty);
    const int q0x = bx * t.TX, q0y = by * 16, q0z = bz * 8 * t.ZH;
    const int nchunk = (KCH + 15) / 16, T = t.TX * t.ZH, nis = min(kTcIssue, T);
    if (warp == 8) {
        tc_alloc(&s_tmem, (uint32_t)t.ncols);
        tc_relinquish();
    }
    if (tid == 0) {
        for (int b = 0; b < 2; b++) {
            mbar_init(&s_full[b], kTcProd);
            mbar_init(&s_empty[b], nis);
        }
        mbar_init(&s_done, nis);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid == 32) {  // taps: weight index and start offset in the staged tile
        int k = 0;
        for (int w = 0; w < 27; w++) {
            const int tx = w / 9, ty = (w / 3) % 3, tz = w % 3;
            int dx, dy, dz;
            if (MODE == 0) {
                dx = tx, dy = ty, dz = tz;
            } else if (a.s == 1) {
                dx = 2 - tx, dy = 2 - ty, dz = 2 - tz;
            } else {  // input voxel 2q + p takes the taps t with t = p + 1 (mod 2), from q + (p + 1 - t) / 2
                if (((px + 1 - tx) & 1) || ((py + 1 - ty) & 1) || ((pz + 1 - tz) & 1)) continue;
                dx = (px + 1 - tx) >> 1, dy = (py + 1 - ty) >> 1, dz = (pz + 1 - tz) >> 1;
            }
            s_tw[k] = w;
            s_ts[k] = (dx * t.LY + dy) * t.LZ + tc_zpos(dz, t.even);
            k++;
        }
        s_ntap = k;
    }
    // first voxel of the tile inside the source; staged voxels by their offset from it (a source may hold more
    // than 2^31 voxels)
    const int g0x = max(q0x * t.step + t.org, 0), g0y = max(q0y * t.step + t.org, 0), g0z = max(q0z * t.step + t.org, 0);
    if (tid < kTcProd) {  // offset of every staged voxel (-1 outside)
        for (int v = tid; v < nvox; v += kTcProd) {
            const int row = v / t.LZ, lx = row / t.LY;
            const int p = v - row * t.LZ, ly = row - lx * t.LY;
            const int lz = t.even ? (p < t.even ? 2 * p : 2 * (p - t.even) + 1) : p;
            const int gx = q0x * t.step + t.org + lx, gy = q0y * t.step + t.org + ly, gz = q0z * t.step + t.org + lz;
            const bool in = gx >= 0 && gy >= 0 && gz >= 0 && gx < t.SX && gy < t.SY && gz < t.SZ;
            s_off[v] = in ? ((gx - g0x) * t.SY + gy - g0y) * t.SZ + gz - g0z : -1;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int ntap = s_ntap;
    bool ok = true;
    if (warp < 8) {
        const long long V = (long long)t.SX * t.SY * t.SZ;
        const float* src = a.src + (long long)n * KCH * V + ((long long)g0x * t.SY + g0y) * t.SZ + g0z;
        for (int c = 0; c < nchunk; c++) {
            const int b = c & 1;
            if (c >= 2 && !mbar_wait(&s_empty[b], ((c >> 1) - 1) & 1)) ok = false;
            uint4* dA = reinterpret_cast<uint4*>(sA + b * a_bytes);
            for (int h = 0; h < 2; h++) {
                const int ch0 = c * 16 + h * 8, cnt = KCH - ch0;
                const float* sc = src + (long long)(cnt > 0 ? ch0 : 0) * V;
#pragma unroll 2
                for (int v = tid; v < nvox; v += kTcProd) {
                    const int off = s_off[v];
                    dA[h * nvox + v] = tc_gather8(sc + max(off, 0), V, off >= 0, cnt);
                }
            }
            // weights of the chunk, lanes over the taps: (tap, half, column) -> 8 reduction channels
            uint4* dB = reinterpret_cast<uint4*>(sB + b * b_bytes);
            if (lane < ntap) {
                const int wt = s_tw[lane];
#pragma unroll 2
                for (int r = warp; r < 2 * t.NT; r += kTcProd / 32) {
                    const int h = r & 1, j = r >> 1, ch0 = c * 16 + h * 8, cnt = KCH - ch0;
                    const bool in = j0 + j < NCH;
                    const int jc = in ? j0 + j : 0, chc = cnt > 0 ? ch0 : 0;
                    const long long at = MODE == 0 ? (long long)jc * KCH + chc : (long long)chc * a.Cin + jc;
                    dB[(lane * 2 + h) * t.NT + j] = tc_gather8(a.w + at * 27 + wt, MODE == 0 ? 27 : 27 * a.Cin, in, cnt);
                }
            }
            fence_async_smem();  // the generic-proxy stores become visible to the tensor cores
            mbar_arrive(&s_full[b]);
        }
    } else if (lane == 0 && warp - 8 < nis) {
        const uint32_t idesc = umma_idesc_bf16(128, t.NT);
        // this issuer's accumulators: tiles m0 and m0 + 4
        const int m0 = warp - 8, m1 = m0 + kTcIssue;
        auto tile_at = [&](int m) { return (uint64_t)((m / t.ZH) * t.step * t.LY * t.LZ + (m % t.ZH) * 8); };
        const uint64_t at0 = tile_at(m0), at1 = tile_at(m1) - at0;
        const uint32_t d0 = tmem + (uint32_t)(m0 * t.NT), d1 = tmem + (uint32_t)(m1 * t.NT);
        const bool second = m1 < T;
        for (int c = 0; c < nchunk && ok; c++) {
            const int b = c & 1;
            ok = mbar_wait(&s_full[b], (c >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint64_t da0 =
                umma_smem_desc(smem_u32(sA + b * a_bytes), (uint32_t)nvox * 16, (uint32_t)(t.step * t.LZ * 16)) + at0;
            uint64_t db = umma_smem_desc(smem_u32(sB + b * b_bytes), (uint32_t)t.NT * 16, 128);
            uint32_t accum = c ? 1u : 0u;
#pragma unroll 3
            for (int k = 0; k < ntap; k++) {
                const uint64_t da = da0 + (uint64_t)s_ts[k];
                tc_mma(d0, da, db, idesc, accum);
                if (second) tc_mma(d1, da + at1, db, idesc, accum);
                db += (uint64_t)(2 * t.NT);
                accum = 1u;
            }
            tc_commit(&s_empty[b]);
        }
        if (ok) tc_commit(&s_done);
    }
    __syncwarp();
    if (!mbar_wait(&s_done, 0)) ok = false;
    tc_fence_after();
    // tcgen05.ld is warp-collective: decide the epilogue for the whole block
    if (__syncthreads_and(ok ? 1 : 0)) {
        if (warp < 8) {
            const int y = t.ost * (q0y + (warp & 3) * 4 + (lane >> 3)) + py;
            const int RX = MODE == 0 ? a.Xo : a.X, RY = MODE == 0 ? a.Yo : a.Y, RZ = MODE == 0 ? a.Zo : a.Z;
            const long long Vr = (long long)RX * RY * RZ;
            for (int m = warp >> 2; m < T; m += 2) {
                const int x = t.ost * (q0x + m / t.ZH) + px, z = t.ost * (q0z + (m % t.ZH) * 8 + (lane & 7)) + pz;
                const bool rv = x < RX && y < RY && z < RZ;
                float* dst = a.dst + (long long)n * NCH * Vr + ((long long)x * RY + y) * RZ + z;
                for (int c0 = 0; c0 < t.NT; c0 += 16) {
                    float v[16];
                    tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(m * t.NT + c0), v);
                    if (rv) {
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const int ch = j0 + c0 + i;
                            if (ch >= NCH) break;
                            float* d = dst + (long long)ch * Vr;
                            if constexpr (MODE == 0) {
                                float yv = v[i] + __ldg(a.b + ch);
                                if (a.relu) yv = fmaxf(yv, 0.f);
                                *d = yv;
                            } else {
                                *d = a.accumulate ? *d + v[i] : v[i];
                            }
                        }
                    }
                }
            }
        }
    } else if (tid == 0) {
        atomicExch(a.err, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tc_dealloc(tmem, (uint32_t)t.ncols);
}

// Weight gradient.  The output voxels are cut into tiles of TX x 16 x 8, the tiles into `nsplit`
// ranges; CTA (range, tap group, input-channel tile, column split) accumulates its taps'
// 64 x NT products (row: input channel, after them one row of ones that gives the bias
// gradient; column: output channel) over its range in tensor memory and writes them to
// part[range][co][ci * 27 + t]; k_conv_tc_wsum adds the ranges in order.
constexpr int kTcWSplit = 4096;  // voxels per range (sets the workspace)
constexpr int kTcWProd = 512;

struct ConvWTile {
    int TX, ntx, nty, ntz;
    int LX, LY, LZ, even;
    int np;                // planes of 8 input channels per CTA (the plane of ones follows)
    int nci;               // input-channel tiles
    int NT, nco, TG, ntg;  // columns per CTA and splits, taps per CTA and groups
    int ncols, nsplit;
};

constexpr int kTcWTaps = 7;  // taps of one issuing thread: ceil(27 / 4)

__global__ void __launch_bounds__(kTcWProd + 32 * kTcIssue, 1) k_conv_tc_wgrad(ConvTcArgs a, ConvWTile t, float* __restrict__ part) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t s_full[2], s_empty[2], s_done;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nrow = t.LX * t.LY, nvox = nrow * t.LZ, np1 = t.np + 1, RP = np1 * t.LZ;  // row pitch, 16-byte units
    const int nvd = t.TX * 128;
    const size_t a_bytes = (size_t)nrow * RP * 16, b_bytes = (size_t)(t.NT / 8) * nvd * 16;
    uint8_t* sA = smem;
    uint8_t* sB = smem + 2 * a_bytes;
    int2* s_tab = reinterpret_cast<int2*>(sB + 2 * b_bytes);  // two tables of nvox
    const int range = blockIdx.x, tg = blockIdx.y % t.ntg, cot = blockIdx.y / t.ntg;
    const int co0 = cot * t.NT, ci0 = blockIdx.z * t.np * 8;
    const int tap0 = tg * t.TG, ntap = min(t.TG, 27 - tap0);
    const long long ntile = (long long)a.N * t.ntx * t.nty * t.ntz;
    const long long tb = ntile * range / t.nsplit, te = ntile * (range + 1) / t.nsplit;
    if (warp == 16) {
        tc_alloc(&s_tmem, (uint32_t)t.ncols);
        tc_relinquish();
    }
    if (tid == 0) {
        for (int b = 0; b < 2; b++) {
            mbar_init(&s_full[b], kTcWProd);
            mbar_init(&s_empty[b], kTcIssue);
        }
        mbar_init(&s_done, kTcIssue);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kTcWProd) {  // the planes of ones stay as they are
        const uint4 one = {0x3f80u, 0u, 0u, 0u};
        for (int v = tid; v < 2 * nvox; v += kTcWProd) {
            const int b = v >= nvox, q = v - b * nvox, row = q / t.LZ;
            *reinterpret_cast<uint4*>(sA + b * a_bytes + ((size_t)row * RP + t.np * t.LZ + q - row * t.LZ) * 16) = one;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    bool ok = true;
    if (warp < 16) {
        const long long Vi = (long long)a.X * a.Y * a.Z, Vo = (long long)a.Xo * a.Yo * a.Zo;
        int c = 0;
        for (long long tl = tb; tl < te; tl++, c++) {
            const int b = c & 1;
            int r = (int)(tl % (t.ntx * t.nty * t.ntz));
            const int n = (int)(tl / (t.ntx * t.nty * t.ntz));
            const int oz0 = (r % t.ntz) * 8, oy0 = (r / t.ntz) % t.nty * 16, ox0 = r / (t.ntz * t.nty) * t.TX;
            // the tile's first voxel inside x: offsets from there
            const int g0x = max(ox0 * a.s - 1, 0), g0y = max(oy0 * a.s - 1, 0), g0z = max(oz0 * a.s - 1, 0);
            int2* tab = s_tab + b * nvox;
            for (int v = tid; v < nvox; v += kTcWProd) {
                const int row = v / t.LZ, lx = row / t.LY;
                const int p = v - row * t.LZ, ly = row - lx * t.LY;
                const int lz = t.even ? (p < t.even ? 2 * p : 2 * (p - t.even) + 1) : p;
                const int gx = ox0 * a.s - 1 + lx, gy = oy0 * a.s - 1 + ly, gz = oz0 * a.s - 1 + lz;
                const bool in = gx >= 0 && gy >= 0 && gz >= 0 && gx < a.X && gy < a.Y && gz < a.Z;
                tab[v] = make_int2(in ? ((gx - g0x) * a.Y + gy - g0y) * a.Z + gz - g0z : -1, row * RP + p);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kTcWProd) : "memory");  // the table, among the producers
            if (c >= 2 && !mbar_wait(&s_empty[b], ((c >> 1) - 1) & 1)) ok = false;
            uint8_t* dA = sA + b * a_bytes;
            const float* x = a.src + (long long)n * a.Cin * Vi + ((long long)g0x * a.Y + g0y) * a.Z + g0z;
            int h = 0, v = tid;
            while (v >= nvox) v -= nvox, h++;
#pragma unroll 2
            for (int it = tid; it < t.np * nvox; it += kTcWProd) {
                const int2 e = tab[v];
                const int ch0 = ci0 + h * 8, cnt = a.Cin - ch0;
                *reinterpret_cast<uint4*>(dA + ((size_t)e.y + h * t.LZ) * 16) =
                    tc_gather8(x + (long long)(cnt > 0 ? ch0 : 0) * Vi + max(e.x, 0), Vi, e.x >= 0, cnt);
                v += kTcWProd;
                while (v >= nvox) v -= nvox, h++;
            }
            uint8_t* dB = sB + b * b_bytes;
            const float* dy = a.w + (long long)n * a.Cout * Vo + ((long long)ox0 * a.Yo + oy0) * a.Zo + oz0;
            for (int it = tid; it < (t.NT / 8) * nvd; it += kTcWProd) {
                const int g = it / nvd, q = it - g * nvd;
                const int ox = q >> 7, oy = (q >> 3) & 15, oz = q & 7;
                const bool in = ox0 + ox < a.Xo && oy0 + oy < a.Yo && oz0 + oz < a.Zo;
                const int ch0 = co0 + g * 8, cnt = a.Cout - ch0;
                *reinterpret_cast<uint4*>(dB + (size_t)it * 16) = tc_gather8(
                    dy + (long long)(cnt > 0 ? ch0 : 0) * Vo + (in ? (ox * a.Yo + oy) * a.Zo + oz : 0), Vo, in, cnt);
            }
            fence_async_smem();
            mbar_arrive(&s_full[b]);
        }
    } else if (lane == 0) {
        const uint32_t idesc = umma_idesc_bf16(64, t.NT, true);
        // this issuer's taps: every fourth; their start offsets and accumulators
        const int is = warp - kTcWProd / 32;
        uint32_t off[kTcWTaps];
        int nk = 0;
#pragma unroll
        for (int i = 0; i < kTcWTaps; i++) {
            const int k = is + i * kTcIssue, w = tap0 + k, tx = w / 9, ty = (w / 3) % 3, tz = w % 3;
            off[i] = (uint32_t)((tx * t.LY + ty) * RP + tc_zpos(tz, t.even));
            if (k < ntap) nk++;
        }
        const uint32_t d0 = tmem + (uint32_t)(is * t.NT), dstep = (uint32_t)(kTcIssue * t.NT);
        int c = 0;
        for (long long tl = tb; tl < te && ok; tl++, c++) {
            const int b = c & 1;
            ok = mbar_wait(&s_full[b], (c >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint64_t da0 = umma_smem_desc(smem_u32(sA + b * a_bytes), (uint32_t)(a.s * RP * 16), (uint32_t)(t.LZ * 16));
            uint64_t db = umma_smem_desc(smem_u32(sB + b * b_bytes), 128, (uint32_t)(nvd * 16));
            uint32_t accum = c ? 1u : 0u;
            for (int x = 0; x < t.TX; x++) {
                uint64_t da = da0 + (uint64_t)(x * a.s * t.LY * RP);
                for (int y = 0; y < 16; y += 2) {  // 16 voxels: two rows of 8
                    uint32_t d = d0;
#pragma unroll
                    for (int i = 0; i < kTcWTaps; i++) {
                        if (i < nk) tc_mma(d, da + off[i], db, idesc, accum);
                        d += dstep;
                    }
                    da += (uint64_t)(2 * a.s * RP);
                    db += 16;
                    accum = 1u;
                }
            }
            tc_commit(&s_empty[b]);
        }
        if (ok) tc_commit(&s_done);
    }
    __syncwarp();
    if (te > tb && !mbar_wait(&s_done, 0)) ok = false;
    tc_fence_after();
    const int Mtot = 27 * a.Cin + 1;
    if (__syncthreads_and(ok ? 1 : 0)) {
        // 64-row accumulators: rows 16 q .. 16 q + 15 lie in lanes 32 q .. 32 q + 15
        if (warp < 16) {
            const int q = warp & 3, row = q * 16 + lane, ci = ci0 + row;
            for (int k = warp >> 2; k < ntap; k += 4) {
                const int tap = tap0 + k;
                for (int c0 = 0; c0 < t.NT; c0 += 16) {
                    float v[16];
                    tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(k * t.NT + c0), v);
                    int m = -1;
                    if (lane < 16) {
                        if (row < t.np * 8 && ci < a.Cin) m = ci * 27 + tap;
                        if (row == t.np * 8 && tap == 13 && blockIdx.z == 0) m = Mtot - 1;
                    }
                    if (m >= 0) {
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const int co = co0 + c0 + i;
                            if (co >= a.Cout) break;
                            part[((long long)range * a.Cout + co) * Mtot + m] = te > tb ? v[i] : 0.f;
                        }
                    }
                }
            }
        }
    } else if (tid == 0) {
        atomicExch(a.err, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) tc_dealloc(tmem, (uint32_t)t.ncols);
}

// dw[co, ci, t] = sum over ranges of part[range][co][ci*27 + t]; db[co] from the ones row.
// Warp g of a block adds every eighth range for 32 outputs, then the eight sums in order (one
// thread per output over all ranges waited on 16 rounds of loads: 35 us for 128 ranges).
// An output voxel that only pads a tile has dy = 0, but for a tap that lies one voxel below it (offset 0 along
// an axis where `pad` is set) its x is the upper face of the grid: an infinity or NaN there gave 0 * inf in a tap
// that never meets that voxel.  Such a tap whose sum is not finite is formed again from the valid outputs
// alone (about one multiply-add per voxel and tap; nothing of it runs on finite sums).
struct ConvPad {
    int x, y, z;
};
__global__ void __launch_bounds__(256) k_conv_tc_wsum(ConvTcArgs a, ConvPad pad, const float* __restrict__ part, int nsplit,
                                                      float* __restrict__ dw, float* __restrict__ db) {
    __shared__ float s_p[8][32];
    __shared__ double s_red[8];
    __shared__ unsigned s_again;
    const int Cout = a.Cout, Mtot = 27 * a.Cin + 1;
    const int g = threadIdx.x >> 5, l = threadIdx.x & 31;
    const long long tot = (long long)Cout * Mtot, i0 = (long long)blockIdx.x * 32, i = i0 + l;
    float s = 0.f;
    if (i < tot) {
#pragma unroll 8
        for (int r = g; r < nsplit; r += 8) s += part[r * tot + i];
    }
    s_p[g][l] = s;
    __syncthreads();
    if (g == 0) {
#pragma unroll
        for (int q = 1; q < 8; q++) s += s_p[q][l];
        const int co = (int)(i / Mtot), m = (int)(i - (long long)co * Mtot), t = m % 27;
        if (i < tot) {
            if (m < Mtot - 1)
                dw[(long long)co * (Mtot - 1) + m] = s;
            else if (db)
                db[co] = s;
        }
        const bool touched = (pad.x && t / 9 == 0) || (pad.y && (t / 3) % 3 == 0) || (pad.z && t % 3 == 0);
        const unsigned again = __ballot_sync(0xffffffffu, i < tot && m < Mtot - 1 && touched && !isfinite(s));
        if (l == 0) s_again = again;
    }
    __syncthreads();
    const long long Vi = (long long)a.X * a.Y * a.Z, Vo = (long long)a.Xo * a.Yo * a.Zo;
    for (unsigned again = s_again; again; again &= again - 1) {
        const long long o = i0 + __ffs(again) - 1;
        const int co = (int)(o / Mtot), m = (int)(o - (long long)co * Mtot), ci = m / 27, t = m - 27 * ci;
        double sum = 0.0;
        for (long long v = threadIdx.x; v < a.N * Vo && sum == sum; v += 256) {
            const long long n = v / Vo, q = v - n * Vo;
            const int oz = (int)(q % a.Zo), oy = (int)(q / a.Zo % a.Yo), ox = (int)(q / a.Zo / a.Yo);
            const int gx = a.s * ox + t / 9 - 1, gy = a.s * oy + (t / 3) % 3 - 1, gz = a.s * oz + t % 3 - 1;
            const bool in = gx >= 0 && gy >= 0 && gz >= 0 && gx < a.X && gy < a.Y && gz < a.Z;
            const float x = in ? a.src[(n * a.Cin + ci) * Vi + ((long long)gx * a.Y + gy) * a.Z + gz] : 0.f;
            const float d = a.w[(n * Cout + co) * Vo + q];
            sum += (double)(__bfloat162float(__float2bfloat16_rn(x)) * __bfloat162float(__float2bfloat16_rn(d)));
        }
        sum = block_sum<256>(sum, s_red);
        if (threadIdx.x == 0) dw[(long long)co * (Mtot - 1) + m] = (float)sum;
        __syncthreads();
    }
}

static int tc_ncols(int NP) {
    int c = 32;
    while (c < NP) c <<= 1;
    return c;
}

static int tc_check() {
    static const bool enc_ok = tc_encodings_match();
    if (!enc_ok) return fail(PF_UNSUPPORTED, "tensor-core conv: descriptor encoding check failed");
    return PF_OK;
}

// staged extent along an axis for n row voxels
static int tc_extent(int mode, int s, int n) { return mode == 0 ? s * (n - 1) + 3 : s == 1 ? n + 2 : n + 1; }

static size_t tc_conv_smem(const ConvTile& t) {
    const size_t nvox = (size_t)t.LX * t.LY * t.LZ;
    return t.nbuf * (nvox * 32 + (size_t)27 * 32 * t.NT) + nvox * sizeof(int);
}

// offsets within a tile of lx planes of an sx x sy x sz grid fit 32 bits
static bool tc_span(int lx, int sx, int sy, int sz) { return (long long)(lx < sx ? lx : sx) * sy * sz < (1LL << 31); }

template <int MODE>
static int launch_conv_tc(const ConvTcArgs& a, cudaStream_t st) {
    const int NCH = MODE == 0 ? a.Cout : a.Cin;
    const int NP = (NCH + 15) / 16 * 16;
    if (NP > 256) return fail(PF_UNSUPPORTED, "tensor-core conv: at most 256 output channels");
    int s = tc_check();
    if (s) return s;
    ConvTile t;
    const bool half = MODE == 1 && a.s == 2;  // one CTA class per parity of the input voxel
    t.QX = MODE == 0 ? a.Xo : half ? (a.X + 1) / 2 : a.X;
    t.QY = MODE == 0 ? a.Yo : half ? (a.Y + 1) / 2 : a.Y;
    t.QZ = MODE == 0 ? a.Zo : half ? (a.Z + 1) / 2 : a.Z;
    t.SX = MODE == 0 ? a.X : a.Xo;
    t.SY = MODE == 0 ? a.Y : a.Yo;
    t.SZ = MODE == 0 ? a.Z : a.Zo;
    t.step = MODE == 0 ? a.s : 1;
    t.org = half ? 0 : -1;
    t.ost = half ? 2 : 1;
    // columns: equal splits of at most 64, so that the weights of a chunk fit beside the voxels
    t.nsplit = (NP + 63) / 64;
    t.NT = (NP / 16 + t.nsplit - 1) / t.nsplit * 16;
    t.nbuf = (MODE == 0 ? a.Cin : a.Cout) > 16 ? 2 : 1;
    // tile: the largest of up to 8 accumulators that leaves two CTAs per SM (tensor memory,
    // shared memory) and at least two CTAs for every SM; else the smallest
    long long best = -1;
    ConvTile pick = t;
    for (int TX = 1; TX <= 4; TX *= 2)
        for (int ZH = 1; ZH <= 2; ZH++) {
            ConvTile c = t;
            c.TX = TX;
            c.ZH = ZH;
            c.LX = tc_extent(MODE, a.s, TX);
            c.LY = tc_extent(MODE, a.s, 16);
            c.LZ = tc_extent(MODE, a.s, 8 * ZH);
            c.even = t.step == 2 ? (c.LZ + 1) / 2 : 0;
            c.ntx = (t.QX + TX - 1) / TX;
            c.nty = (t.QY + 15) / 16;
            c.ntz = (t.QZ + 8 * ZH - 1) / (8 * ZH);
            const long long ctas = (long long)c.ntx * c.nty * c.ntz * a.N * t.nsplit * (half ? 8 : 1);
            const bool two = TX * ZH * t.NT <= 256 && tc_conv_smem(c) <= kTcHalfSmem;
            const bool fits = TX * ZH * t.NT <= 512 && tc_conv_smem(c) <= kTcMaxSmem && tc_span(c.LX, t.SX, t.SY, t.SZ);
            const long long score = !fits ? -2 : ctas >= 2 * kNumSM ? (two ? 100 : 0) + TX * ZH * 4 + ZH : 0;
            if (score > best) best = score, pick = c;
        }
    if (best < 0) return fail(PF_UNSUPPORTED, "tensor-core conv: no tile fits");
    t = pick;
    t.ncols = tc_ncols(t.TX * t.ZH * t.NT);
    const size_t smem = tc_conv_smem(t);
    PF_CUDA(cudaFuncSetAttribute(k_conv_tc<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcMaxSmem));
    const long long blocks = (long long)t.ntx * t.nty * t.ntz * a.N * t.nsplit;
    if (blocks >= (1LL << 31)) return fail(PF_UNSUPPORTED, "tensor-core conv: %lld tiles", blocks);
    const dim3 grid((unsigned)blocks, 1, half ? 8u : 1u);
    pf::count_launch();
    k_conv_tc<MODE><<<grid, kTcProd + 32 * kTcIssue, smem, st>>>(a, t);
    PF_LAUNCH_CHECK("tensor-core conv launch");
    return PF_OK;
}

static inline int out_ext(int n, int s) { return (n - 1) / s + 1; }

}  // namespace pf

using namespace pf;

extern "C" int pf_cnn_conv3d_fwd_tc(const float* x, int N, int Cin, int X, int Y, int Z, const float* w, const float* b,
                                    int Cout, int stride, int relu, float* y, int* err, void* stream) {
    if (!x || !w || !b || !y || !err || N < 1 || Cin < 1 || Cout < 1 || X < 1 || Y < 1 || Z < 1 ||
        (stride != 1 && stride != 2))
        return fail(PF_BAD_ARG, "pf_cnn_conv3d_fwd_tc: bad argument");
    ConvTcArgs a = {x, w, b, y, err, N, Cin, Cout, stride, relu, 0, X, Y, Z,
                    out_ext(X, stride), out_ext(Y, stride), out_ext(Z, stride)};
    return launch_conv_tc<0>(a, as_stream(stream));
}

extern "C" int pf_cnn_conv3d_bwd_data_tc(const float* dy, int N, int Cin, int X, int Y, int Z, const float* w,
                                         int Cout, int stride, int accumulate, float* dx, int* err, void* stream) {
    if (!dy || !w || !dx || !err || N < 1 || Cin < 1 || Cout < 1 || X < 1 || Y < 1 || Z < 1 ||
        (stride != 1 && stride != 2))
        return fail(PF_BAD_ARG, "pf_cnn_conv3d_bwd_data_tc: bad argument");
    ConvTcArgs a = {dy, w, nullptr, dx, err, N, Cin, Cout, stride, 0, accumulate, X, Y, Z,
                    out_ext(X, stride), out_ext(Y, stride), out_ext(Z, stride)};
    return launch_conv_tc<1>(a, as_stream(stream));
}

extern "C" size_t pf_cnn_conv3d_bwd_weight_tc_workspace(int N, int Cin, int X, int Y, int Z, int Cout, int stride) {
    if (N < 1 || Cin < 1 || Cout < 1 || X < 1 || Y < 1 || Z < 1 || (stride != 1 && stride != 2)) return 0;
    const long long Ktot = (long long)N * out_ext(X, stride) * out_ext(Y, stride) * out_ext(Z, stride);
    const long long nsplit = (Ktot + kTcWSplit - 1) / kTcWSplit;
    return (size_t)(nsplit * Cout * (27LL * Cin + 1));
}

extern "C" int pf_cnn_conv3d_bwd_weight_tc(const float* x, const float* dy, int N, int Cin, int X, int Y, int Z,
                                           int Cout, int stride, float* dw, float* db, float* work, int* err,
                                           void* stream) {
    if (!x || !dy || !dw || !work || !err || N < 1 || Cin < 1 || Cout < 1 || X < 1 || Y < 1 || Z < 1 ||
        (stride != 1 && stride != 2))
        return fail(PF_BAD_ARG, "pf_cnn_conv3d_bwd_weight_tc: bad argument");
    const int NP = (Cout + 15) / 16 * 16;
    if (NP > 256) return fail(PF_UNSUPPORTED, "tensor-core conv: at most 256 output channels");
    int s = tc_check();
    if (s) return s;
    ConvTcArgs a = {x, dy, nullptr, dw, err, N, Cin, Cout, stride, 0, 0, X, Y, Z,
                    out_ext(X, stride), out_ext(Y, stride), out_ext(Z, stride)};
    const long long Ktot = (long long)N * a.Xo * a.Yo * a.Zo;
    const int nsplit = (int)((Ktot + kTcWSplit - 1) / kTcWSplit);
    // input-channel tiles of at most 56 (7 planes and the ones: 64 rows), the largest with which
    // two buffers of a tile of two or one x planes fit
    ConvWTile t;
    t.nco = (NP + 63) / 64;
    t.NT = (NP / 16 + t.nco - 1) / t.nco * 16;
    t.TG = 512 / t.NT < 27 ? 512 / t.NT : 27;
    t.ntg = (27 + t.TG - 1) / t.TG;
    t.ncols = tc_ncols((t.TG < 27 ? t.TG : 27) * t.NT);
    t.nsplit = nsplit;
    t.LY = stride * 15 + 3;
    t.LZ = stride * 7 + 3;
    t.even = stride == 2 ? 9 : 0;
    const int planes = (Cin + 7) / 8;
    size_t smem = 0;
    bool found = false;
    for (int parts = 1; parts <= planes && !found; parts++) {
        t.np = (planes + parts - 1) / parts;
        if (t.np > 7) continue;
        for (int TX = 2; TX >= 1 && !found; TX--) {
            t.TX = TX;
            t.LX = stride * (TX - 1) + 3;
            const size_t vox = (size_t)t.LX * t.LY * t.LZ;
            smem = 2 * (vox * (t.np + 1) * 16 + (size_t)(t.NT / 8) * TX * 128 * 16 + vox * sizeof(int2));
            found = smem <= kTcMaxSmem && tc_span(t.LX, X, Y, Z);
        }
    }
    if (!found) return fail(PF_UNSUPPORTED, "tensor-core conv: no tile fits");
    t.nci = (planes + t.np - 1) / t.np;
    t.ntx = (a.Xo + t.TX - 1) / t.TX;
    t.nty = (a.Yo + 15) / 16;
    t.ntz = (a.Zo + 7) / 8;
    cudaStream_t st = as_stream(stream);
    PF_CUDA(cudaFuncSetAttribute(k_conv_tc_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcMaxSmem));
    pf::count_launch(2);
    k_conv_tc_wgrad<<<dim3((unsigned)nsplit, (unsigned)(t.ntg * t.nco), (unsigned)t.nci), kTcWProd + 32 * kTcIssue, smem, st>>>(a, t,
                                                                                                                   work);
    const long long nt = (long long)Cout * (27 * Cin + 1);
    // padded outputs along an axis, the first of which reads the upper face (stride 2: if its extent is even)
    auto reach = [&](int n, int no, int tile) { return no % tile != 0 && stride * no <= n; };
    const ConvPad pad = {reach(X, a.Xo, t.TX), reach(Y, a.Yo, 16), reach(Z, a.Zo, 8)};
    k_conv_tc_wsum<<<(unsigned)((nt + 31) / 32), 256, 0, st>>>(a, pad, work, nsplit, dw, db);
    PF_LAUNCH_CHECK("tensor-core conv weight gradient launch");
    return PF_OK;
}
