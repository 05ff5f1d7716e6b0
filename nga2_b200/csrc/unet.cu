// unet.cu -- kernels of the learned initial guess (a small 3-D U-Net).
//
// No counterpart in the reference (NGA2 starts each pressure solve from the
// previous pressure).  The 3x3x3 convolutions (forward and data gradient) are
// implicit GEMMs on the tensor cores: M = voxels, N = output channels, K = 27
// taps x input channels, BF16 operands, FP32 accumulation.  They run on tcgen05
// (k_conv3_zm: a column of voxel tiles per CTA, its accumulators in TMEM, input
// planes staged once for all their taps); views that are not 16-byte aligned and
// other output widths on mma.sync m16n8k16 (k_conv3: a warp owns 16 consecutive
// voxels and all output channels, its A fragments the tap-shifted input rows
// with periodic wrap, its B fragments the
// packed weights).  The weight gradient, a contraction over voxels, runs on
// mma.sync with ldmatrix.trans fragments (k_wgrad_mma); everything else is
// elementwise.
#include <cuda_bf16.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "../../include/bbmg_b200.h"
#include "../../include/bbmg_learned.h"

namespace {

typedef __nv_bfloat16 bf16;

struct Act {
    bf16 *p;
    int n, d, h, w, c, ld;
    int nvox;
};

Act act_of(const nn_act *a) {
    Act r;
    r.p = (bf16 *)a->data;
    r.n = a->n; r.d = a->d; r.h = a->h; r.w = a->w; r.c = a->c; r.ld = a->ld;
    r.nvox = a->n * a->d * a->h * a->w;
    return r;
}

bool bad_act(const nn_act *a) {
    return !a || !a->data || a->n < 1 || a->d < 1 || a->h < 1 || a->w < 1 || a->c < 1 || a->ld < a->c ||
           (a->ld & 1) || (long long)a->n * a->d * a->h * a->w * a->ld >= (1LL << 31);
}

int done(cudaError_t e) { return e == cudaSuccess ? BBMG_OK : BBMG_CUDA; }

__device__ __forceinline__ void decode(const Act &a, int v, int &n, int &d, int &h, int &w) {
    w = v % a.w;
    int r = v / a.w;
    h = r % a.h;
    r /= a.h;
    d = r % a.d;
    n = r / a.d;
}
__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
__device__ __forceinline__ int vox(const Act &a, int n, int d, int h, int w) {
    return ((n * a.d + d) * a.h + h) * a.w + w;
}

__device__ __forceinline__ uint32_t ld32(const bf16 *p) { return *reinterpret_cast<const uint32_t *>(p); }

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------
// Convolution as implicit GEMM.  wt is [27][cout][cin] (K contiguous per
// output channel, the layout of the mma B operand).  NT = cout / 8.
template <int NT>
__global__ void __launch_bounds__(128) k_conv3(Act x, const bf16 *__restrict__ wt, const float *__restrict__ bias,
                                                Act y, int relu) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int v0 = (blockIdx.x * 4 + warp) * 16;
    if (v0 >= x.nvox) return;
    const int cin = x.c;
    const int r0 = v0 + g, r1 = v0 + g + 8;
    const int q0 = min(r0, x.nvox - 1), q1 = min(r1, x.nvox - 1);
    int n0, d0, h0, w0, n1, d1, h1, w1;
    decode(x, q0, n0, d0, h0, w0);
    decode(x, q1, n1, d1, h1, w1);
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int tap = 0; tap < 27; tap++) {
        const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
        const int s0 = vox(x, n0, wrapi(d0 + dz, x.d), wrapi(h0 + dy, x.h), wrapi(w0 + dx, x.w));
        const int s1 = vox(x, n1, wrapi(d1 + dz, x.d), wrapi(h1 + dy, x.h), wrapi(w1 + dx, x.w));
        const bf16 *xa = x.p + (long long)s0 * x.ld + 2 * t;
        const bf16 *xb = x.p + (long long)s1 * x.ld + 2 * t;
        const bf16 *wtap = wt + (long long)tap * (NT * 8) * cin + (long long)g * cin + 2 * t;
        for (int c0 = 0; c0 < cin; c0 += 16) {
            const uint32_t a0 = ld32(xa + c0), a1 = ld32(xb + c0), a2 = ld32(xa + c0 + 8), a3 = ld32(xb + c0 + 8);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const bf16 *wp = wtap + (long long)nt * 8 * cin + c0;
                mma16816(acc[nt], a0, a1, a2, a3, __ldg(reinterpret_cast<const unsigned int *>(wp)),
                         __ldg(reinterpret_cast<const unsigned int *>(wp + 8)));
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        const int col = nt * 8 + 2 * t;
        const float b0 = bias ? bias[col] : 0.f, b1 = bias ? bias[col + 1] : 0.f;
        float o0 = acc[nt][0] + b0, o1 = acc[nt][1] + b1, o2 = acc[nt][2] + b0, o3 = acc[nt][3] + b1;
        if (relu) {
            o0 = fmaxf(o0, 0.f); o1 = fmaxf(o1, 0.f); o2 = fmaxf(o2, 0.f); o3 = fmaxf(o3, 0.f);
        }
        if (r0 < y.nvox)
            *reinterpret_cast<__nv_bfloat162 *>(y.p + (long long)r0 * y.ld + col) = __floats2bfloat162_rn(o0, o1);
        if (r1 < y.nvox)
            *reinterpret_cast<__nv_bfloat162 *>(y.p + (long long)r1 * y.ld + col) = __floats2bfloat162_rn(o2, o3);
    }
}

// ---------------------------------------------------------------------------
// Convolution as implicit GEMM on the fifth-generation tensor cores (tcgen05).
// A CTA owns a column of 8 (w) x 16 (h) voxels (M = 128) over up to DZ output
// planes and N output channels (all of them, or one of G groups: with_width); its FP32
// accumulators, DZ x N columns, stay in TMEM.
//   * K is walked in chunks of 16 input channels; a chunk marches over the
//     DZ + 2 input planes.  A stage is one plane of one chunk: its 10 x 18
//     voxels with the halo (periodic wrap), as [8-channel group][voxel][16 B],
//     the K-major no-swizzle layout of the MMA with 160 bytes from one h row to
//     the next.  Each of the nine (dy, dx) taps is then a descriptor shifted by
//     whole 16-byte rows: every input element is read from global memory 1.4
//     times per plane instead of once per tap.
//   * Input plane p contributes to the output planes p-1, p, p+1 through the
//     taps dz = +1, 0, -1.  Their accumulators are neighbouring TMEM columns and
//     the chunk's weights are stored [dy, dx][group][dz][cout], so one MMA of
//     up to 3 N columns does all three: with 16 output channels an MMA's time is
//     the reading of A (128 rows of 32 bytes at 128 B per cycle), whatever N.
//   * A planes sit in a ring of S slots filled with cp.async S - 1 stages ahead;
//     one thread issues a stage's MMAs and commits them to the slot's mbarrier,
//     which gates its refill.  The weights of a chunk have NB buffers; with one,
//     the next chunk's load waits for the MMAs before it.  A tile of one output
//     plane has the weights of each stage's dz in its slot.
//   * The epilogue reads the four warps' 32 TMEM lanes, adds the bias, applies
//     the ReLU and stores BF16.
// Measured at 128^3 (the whole forward pass of the U-Net with its guess assembly):
// 3.55 ms with one CTA per 128-voxel row tile that staged an input row for each
// (dz, dy) and issued 27 MMAs of N = cout per tile, 1.32 ms with this kernel.  The
// nine MMAs of a tile of one plane are unrolled: one thread issues them, and on
// 8^3 64->64 takes 25 us with a loop and 20 without.
// Every mbarrier wait is bounded: a wait that runs out raises g_tc_err (read by
// nn_tc_error), and the CTA then drains its copies, frees its TMEM and returns
// without writing.
__device__ int g_tc_err;  // each device's own, there without an allocation: a first call may be captured
constexpr unsigned kTcSpinLimit = 1u << 22;
constexpr int kZmA = 4;                     // A slots, or 2 (conv_geo)
constexpr int kZmVox = 10 * 18;             // voxels of a halo plane
constexpr int kZmPlane = kZmVox * 32;       // bytes of a stage's A

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cpa16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// shared-memory matrix descriptor: K-major, no swizzle (addresses and offsets in bytes)
__device__ __forceinline__ uint64_t umma_desc(unsigned saddr, unsigned lbo, unsigned sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of sm_100
    return d;                // base offset 0, layout type 0 (no swizzle)
}

// instruction descriptor, kind::f16: D FP32, A and B BF16, both K-major, M = 128
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(unsigned tmem, uint64_t ad, uint64_t bd, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
        ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(1), "r"(0));
}

// bounded wait for the completion of phase `parity` of an mbarrier
__device__ __forceinline__ bool mbar_wait(const uint64_t *mb, unsigned parity) {
    for (unsigned spins = 0; spins < kTcSpinLimit; spins++) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done) : "r"(smem_u32(mb)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

struct ZmGeo {
    int tw, th, tz;  // tiles along w, h, d
    int dz;          // output planes per tile
    int cols;        // TMEM columns
    int nb;          // weight buffers; 0: with one output plane per tile, weights in the plane's stage
    int slots;       // A slots
};

__device__ __forceinline__ int wrapn(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

template <int N, int G, int S>
__global__ void __launch_bounds__(128) k_conv3_zm(Act x, const bf16 *__restrict__ wt, const float *__restrict__ bias,
                                                   Act y, int relu, ZmGeo geo) {
    static_assert(3 * N <= 256 && S >= 2 && S <= 4, "one MMA for three planes; the first S - 1 stages in one chunk");
    constexpr int kB = 27 * N * 32;  // bytes of a chunk's weights
    constexpr int kB3 = kB / 3;      // of one dz of it
    extern __shared__ __align__(128) unsigned char smtc[];
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(smtc);
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smtc + 16);  // S barriers
    unsigned char *A = smtc + 128;
    unsigned char *B = A + (size_t)S * kZmPlane;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int cin = x.c, nchunk = cin >> 4;
    constexpr int cout = G * N;
    const int co0 = G == 1 ? 0 : blockIdx.y * N;  // this CTA's output channels
    if (G > 1) wt += (long long)co0 * cin;
    if (G > 1 && bias) bias += co0;
    int t = blockIdx.x;
    const int w0 = (t % geo.tw) * 8;
    t /= geo.tw;
    const int h0 = (t % geo.th) * 16;
    t /= geo.th;
    const int z0 = (t % geo.tz) * geo.dz, n = t / geo.tz;
    const int nq = min(geo.dz, x.d - z0);  // output planes of this tile
    const int npl = nq + 2, nst = nchunk * npl;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(geo.cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0)
        for (int s = 0; s < S; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + s)));

    // this thread's copies of a plane: chunk e = tid + 128 u is group e & 1 of voxel e >> 1
    int src[3];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const int hv = min((tid + 128 * u) >> 1, kZmVox - 1);
        src[u] = (wrapn(h0 - 1 + hv / 10, x.h) * x.w + wrapn(w0 - 1 + hv % 10, x.w)) * x.ld + (tid & 1) * 8;
    }
    const int zstride = x.h * x.w * x.ld;
    const bf16 *xn = x.p + (long long)n * x.d * zstride;
    auto load_a = [&](int st) {
        const int c = st / npl, r = st - c * npl;
        const bf16 *p = xn + (long long)wrapn(z0 - 1 + r, x.d) * zstride + c * 16;
        unsigned char *As = A + (size_t)(st % S) * kZmPlane;
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const int e = tid + 128 * u;
            if (e < 2 * kZmVox) cpa16(As + (e & 1) * (kZmVox * 16) + (e >> 1) * 16, p + src[u]);
        }
    };
    // weights of chunk c: [dy, dx][group][dz = +1, 0, -1][cout][16 B]
    auto load_b = [&](int c) {
        unsigned char *Bs = B + (size_t)(c % geo.nb) * kB;  // nb >= 1
        for (int e = tid; e < 54 * N; e += 128) {
            const int g = e & 1, o = (e >> 1) % N, tap = (e >> 1) / N;  // tap = 9 dz + 3 dy + dx
            const int dzi = tap / 9, t9 = tap - 9 * dzi;
            cpa16(Bs + (((t9 * 2 + g) * 3 + 2 - dzi) * N + o) * 16, wt + ((long long)tap * cout + o) * cin + c * 16 + g * 8);
        }
    };
    // one output plane: stage st (input plane st % 3 of chunk st / 3) has only the
    // taps of one dz, and they come with it: [dy, dx][group][cout][16 B]
    const bool third = geo.nb == 0;
    auto load_b3 = [&](int st) {
        const int c = st / 3, r = st - 3 * c;
        unsigned char *Bs = B + (size_t)(st % S) * kB3;
        for (int e = tid; e < 18 * N; e += 128) {
            const int g = e & 1, o = (e >> 1) % N, t9 = (e >> 1) / N;
            cpa16(Bs + ((t9 * 2 + g) * N + o) * 16, wt + ((long long)(9 * r + t9) * cout + o) * cin + c * 16 + g * 8);
        }
    };
    auto commit_group = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };

    if (!third) load_b(0);
#pragma unroll 1
    for (int p = 0; p < S - 1; p++) {
        if (p < nst) {
            if (third) load_b3(p);
            load_a(p);  // S - 1 <= npl: of the first chunk
        }
        commit_group();
    }
    __syncthreads();  // barrier inits and the TMEM address are visible
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *reinterpret_cast<volatile unsigned *>(tmem_slot);
    // the accumulators start at zero
    for (int c0 = 0; c0 < nq * N; c0 += 16)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(
                tmem + ((unsigned)(warp * 32) << 16) + (unsigned)c0), "r"(0));
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    bool ok = true;
#pragma unroll 1
    for (int st = 0; st < nst; st++) {
        const int c = st / npl, r = st - c * npl;
        if (st && r == 0 && geo.nb == 1) {
            // one weight buffer: the MMAs of the chunk before have to be done
            const bool done = mbar_wait(mbar + (st - 1) % S, ((st - 1) / S) & 1);
            if (__syncthreads_or(!done)) {
                ok = false;
                break;
            }
            load_b(c);
            commit_group();
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");  // stage st has landed
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the tensor core
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned as = smem_u32(A + (size_t)(st % S) * kZmPlane), bs = smem_u32(third ? B + (size_t)(st % S) * kB3 : B + (size_t)(c % geo.nb) * kB);
            // output planes lo .. hi (tile-local) of input plane r - 1
            const int lo = max(0, r - 2), hi = min(nq - 1, r), b0 = lo - (r - 2);
            const auto tap = [&](int t9) { return umma_desc(as + ((t9 / 3) * 10 + t9 % 3) * 16, kZmVox * 16, 160); };
            if (third) {
#pragma unroll
                for (int t9 = 0; t9 < 9; t9++)
                    umma_bf16(tmem, tap(t9), umma_desc(bs + t9 * 2 * N * 16, N * 16, 128), umma_idesc_bf16(N));
            } else {
                const uint32_t idesc = umma_idesc_bf16((hi - lo + 1) * N);
#pragma unroll 1
                for (int t9 = 0; t9 < 9; t9++)
                    umma_bf16(tmem + lo * N, tap(t9), umma_desc(bs + (t9 * 6 + b0) * N * 16, 3 * N * 16, 128), idesc);
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(mbar + st % S)) : "memory");
        }
        const int nx = st + S - 1;  // the stage to fill next, in the slot stage st-1 used
        if (nx < nst) {
            if (st >= 1) {
                const bool done = mbar_wait(mbar + nx % S, ((st - 1) / S) & 1);
                if (__syncthreads_or(!done)) {
                    ok = false;
                    break;
                }
            }
            if (third) load_b3(nx);
            else if (nx % npl == 0 && geo.nb > 1) load_b(nx / npl);
            load_a(nx);
        }
        commit_group();
    }
    bool done = false;
    if (ok) done = mbar_wait(mbar + (nst - 1) % S, ((nst - 1) / S) & 1);
    if (__syncthreads_or(!done)) {
        done = false;
        if (tid == 0) atomicExch(&g_tc_err, 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (done) {
        // TMEM lane = tile row = voxel (h0 + tid / 8, w0 + tid % 8)
        const int h = h0 + (tid >> 3), w = w0 + (tid & 7);
        const bool in = h < x.h && w < x.w;
        for (int q = 0; q < nq; q++) {
            bf16 *dst = y.p + ((((long long)n * x.d + z0 + q) * x.h + h) * x.w + w) * y.ld + co0;
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 16) {
                unsigned v[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                    : "r"(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(q * N + c0)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                alignas(16) __nv_bfloat162 o2[8];
#pragma unroll
                for (int m = 0; m < 8; m++) {
                    float a = __uint_as_float(v[2 * m]) + (bias ? bias[c0 + 2 * m] : 0.f);
                    float b = __uint_as_float(v[2 * m + 1]) + (bias ? bias[c0 + 2 * m + 1] : 0.f);
                    if (relu) { a = fmaxf(a, 0.f); b = fmaxf(b, 0.f); }
                    o2[m] = __floats2bfloat162_rn(a, b);
                }
                if (in) {
                    uint4 *d4 = reinterpret_cast<uint4 *>(dst + c0);
                    d4[0] = *reinterpret_cast<uint4 *>(&o2[0]);
                    d4[1] = *reinterpret_cast<uint4 *>(&o2[4]);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(geo.cols));
}

// dynamic shared memory above 48 KB, asked for once per kernel and device
// (`seen` holds the devices that granted it)
template <typename K> bool allow_smem(K kern, int bytes, std::atomic<uint64_t> &seen) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (seen.load(std::memory_order_relaxed) & bit) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    seen.fetch_or(bit, std::memory_order_relaxed);
    return true;
}

// the tcgen05 path: 16-byte aligned channel rows and weights (all three are
// copied 16 bytes at a time) and an output width the kernel is instantiated for
bool tc_eligible(const Act &x, const bf16 *wt, const Act &y) {
    static const bool off = getenv("BBMG_NO_TCGEN05") != nullptr;
    if (off || x.c % 16) return false;
    if (y.c != 16 && y.c != 32 && y.c != 48 && y.c != 64 && y.c != 96 && y.c != 128 && y.c != 192) return false;
    const auto off16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    return !(x.ld % 8 || y.ld % 8 || off16(x.p) || off16(wt) || off16(y.p));
}

// Wide outputs go in groups of 64 or 32 channels (with_width): with 96, 128 or 192
// at once the weights of a tile of one plane fill an SM, whose copies then wait for
// its MMAs.  At 128^3 64->128, 128->128, 32->96 and 64->192 take 3.84, 7.23, 1.79
// and 5.77 ms so, 1.95, 3.67, 0.88 and 3.06 in groups; at 8^3, where more CTAs
// cover more SMs, 35, 66, 17 and 52 us and 20, 37, 9 and 20.
constexpr int zm_smem(int n, int slots, int nb) {
    return 128 + slots * kZmPlane + (nb ? nb * 27 * n * 32 : slots * 9 * n * 32);
}

constexpr int kZmMost = 226 * 1024;
static_assert(zm_smem(64, kZmA, 2) <= kZmMost, "the widest group has to fit");

template <int N>
ZmGeo conv_geo(const Act &x, int groups) {
    constexpr int kTwoPerSm = 112 * 1024;
    ZmGeo g;
    g.tw = (x.w + 7) / 8;
    g.th = (x.h + 15) / 16;
    // output planes per tile: as many as 128 TMEM columns hold (four CTAs share
    // an SM's 512), fewer where that would leave SMs idle
    const long long cols = (long long)g.tw * g.th * x.n * groups;
    g.dz = min(x.d, 128 / N);
    while (g.dz > 1 && cols * ((x.d + g.dz - 1) / g.dz) < 2 * 148) g.dz = (g.dz + 1) / 2;
    g.tz = (x.d + g.dz - 1) / g.dz;
    for (g.cols = 32; g.cols < g.dz * N;) g.cols *= 2;
    // One plane per tile (the deep levels: few tiles, long K): each stage brings
    // the weights of its own dz, so that no load waits for a whole chunk's MMAs.
    // Otherwise two weight buffers where two CTAs per SM still fit with them.
    g.nb = g.dz == 1 ? 0 : (x.c > 16 && zm_smem(N, kZmA, 2) <= kTwoPerSm ? 2 : 1);
    // Two slots where that lets more CTAs share an SM and so ends in fewer waves.
    // A wave of o2 CTAs per SM takes about (o2 + o4) / (2 o4) of the time of one
    // of o4 (64->64: 45 us with 2, 56 with 3).  At 128^3 64->64 takes 1.24 ms with
    // four slots and 1.04 with two; on 8x128x128 (1.7 against 1.2 waves, two of
    // either) 95 and 99 us.
    const long long ctas = cols * g.tz;
    const auto per_sm = [&](int slots) { return min(512 / g.cols, 228 * 1024 / (zm_smem(N, slots, g.nb) + 1024)); };
    const auto waves = [&](int o) { return (ctas + 148 * o - 1) / (148 * o); };
    const int o2 = per_sm(2), o4 = per_sm(kZmA);
    g.slots = o2 > o4 && waves(o2) * (o2 + o4) < waves(o4) * 2 * o4 ? 2 : kZmA;
    return g;
}

template <int N, int G, int S>
int launch_zm(const Act &x, const bf16 *wt, const float *bias, const Act &y, int relu, const ZmGeo &g, cudaStream_t s) {
    static std::atomic<uint64_t> seen{0};
    if (!allow_smem(k_conv3_zm<N, G, S>, kZmMost, seen)) return BBMG_CUDA;
    const long long grid = (long long)g.tw * g.th * x.n * g.tz;
    if (grid >= (1LL << 31)) return BBMG_BAD_ARGS;
    k_conv3_zm<N, G, S><<<dim3((unsigned)grid, G), 128, zm_smem(N, S, g.nb), s>>>(x, wt, bias, y, relu, g);
    return done(cudaGetLastError());
}

// f(output channels of a CTA, groups) as constants, for the widths of tc_eligible
template <typename F>
int with_width(int cout, F f) {
    using std::integral_constant;
    switch (cout) {
    case 16: return f(integral_constant<int, 16>{}, integral_constant<int, 1>{});
    case 32: return f(integral_constant<int, 32>{}, integral_constant<int, 1>{});
    case 48: return f(integral_constant<int, 48>{}, integral_constant<int, 1>{});
    case 64: return f(integral_constant<int, 64>{}, integral_constant<int, 1>{});
    case 96: return f(integral_constant<int, 32>{}, integral_constant<int, 3>{});
    case 128: return f(integral_constant<int, 64>{}, integral_constant<int, 2>{});
    case 192: return f(integral_constant<int, 64>{}, integral_constant<int, 3>{});
    }
    return BBMG_BAD_ARGS;
}

int launch_conv(const Act &x, const bf16 *wt, const float *bias, const Act &y, int relu, cudaStream_t s) {
    const int blocks = (x.nvox + 63) / 64;
    if (tc_eligible(x, wt, y))
        return with_width(y.c, [&](auto width, auto groups) {
            constexpr int N = decltype(width)::value, G = decltype(groups)::value;
            const ZmGeo g = conv_geo<N>(x, G);
            return g.slots == 2 ? launch_zm<N, G, 2>(x, wt, bias, y, relu, g, s)
                                : launch_zm<N, G, kZmA>(x, wt, bias, y, relu, g, s);
        });
    // output widths of the U-Net: 16/32/64/128 forward; the data gradients
    // of the concatenated decoder inputs add 48/96/192
    if (y.c % 8) return BBMG_BAD_ARGS;
    switch (y.c / 8) {
    case 2: k_conv3<2><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 4: k_conv3<4><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 6: k_conv3<6><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 8: k_conv3<8><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 12: k_conv3<12><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 16: k_conv3<16><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    case 24: k_conv3<24><<<blocks, 128, 0, s>>>(x, wt, bias, y, relu); break;
    default: return BBMG_BAD_ARGS;
    }
    return done(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Weight gradient: dw[tap][ci][co] += sum_v x(v + tap, ci) dy(v, co).  Block
// (tap, voxel chunk); each step stages VB voxels of dy and of the tap-shifted
// x in shared memory, every thread accumulates its (ci, co) pairs.
constexpr int kWgVB = 16;
__global__ void __launch_bounds__(256) k_wgrad(Act x, Act gy, float *__restrict__ dw, float *__restrict__ db,
                                                int vchunk) {
    extern __shared__ float sm[];
    const int cin = x.c, cout = gy.c, tap = blockIdx.y;
    float *sx = sm;                      // [kWgVB][cin]
    float *sg = sm + kWgVB * cin;        // [kWgVB][cout]
    const int npair = cin * cout;
    constexpr int kMaxPairs = 24;        // pairs per thread; blockIdx.z selects a range of 24*256 pairs
    const int pbase = blockIdx.z * kMaxPairs * 256;
    float acc[kMaxPairs];
#pragma unroll
    for (int q = 0; q < kMaxPairs; q++) acc[q] = 0.f;
    float accb = 0.f;
    const int dz = tap / 9 - 1, dyy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
    const int vbeg = blockIdx.x * vchunk, vend = min(vbeg + vchunk, gy.nvox);
    for (int vb = vbeg; vb < vend; vb += kWgVB) {
        __syncthreads();
        for (int e = threadIdx.x; e < kWgVB * cin; e += blockDim.x) {
            const int k = e / cin, c = e % cin, v = vb + k;
            float val = 0.f;
            if (v < vend) {
                int n, d, h, w;
                decode(gy, v, n, d, h, w);
                const int s = vox(x, n, wrapi(d + dz, x.d), wrapi(h + dyy, x.h), wrapi(w + dx, x.w));
                val = __bfloat162float(x.p[(long long)s * x.ld + c]);
            }
            sx[e] = val;
        }
        for (int e = threadIdx.x; e < kWgVB * cout; e += blockDim.x) {
            const int k = e / cout, c = e % cout, v = vb + k;
            sg[e] = v < vend ? __bfloat162float(gy.p[(long long)v * gy.ld + c]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kMaxPairs; q++) {
            const int p = pbase + threadIdx.x + q * blockDim.x;
            if (p < npair) {
                const int ci = p / cout, co = p % cout;
                float a = acc[q];
#pragma unroll
                for (int k = 0; k < kWgVB; k++) a = fmaf(sx[k * cin + ci], sg[k * cout + co], a);
                acc[q] = a;
            }
        }
        if (db && tap == 13 && blockIdx.z == 0 && threadIdx.x < cout)
            for (int k = 0; k < kWgVB; k++) accb += sg[k * cout + threadIdx.x];
    }
#pragma unroll
    for (int q = 0; q < kMaxPairs; q++) {
        const int p = pbase + threadIdx.x + q * blockDim.x;
        if (p < npair) atomicAdd(&dw[(long long)tap * npair + p], acc[q]);
    }
    if (db && tap == 13 && blockIdx.z == 0 && threadIdx.x < cout) atomicAdd(&db[threadIdx.x], accb);
}

// Weight gradient on the tensor cores: dW[tap][ci][co] = sum over voxels v of
// x(v + tap, ci) dy(v, co) is, per tap, a GEMM with M = ci, N = co and the voxels
// as K (mma.sync m16n8k16, BF16 products, FP32 accumulation).
//   * A CTA takes one block of 16 ci x 16 co for all 27 taps, on a tile of 16 (h)
//     x 16 (w) voxels marching along d: each plane of dy is staged once and each
//     plane of x (with its halo, periodic wrap) once for the three dz that use it,
//     instead of once per tap.  Planes are [8-channel group][voxel][16 B] in a
//     ring of four (x) and two (dy) slots filled with cp.async a plane ahead.
//   * Nine warps, one per (dz, dy); a K step is one row of 16 voxels.  Its B
//     fragments (dy) serve the warp's three dx taps, whose A fragments are the
//     x row shifted by a voxel; ldmatrix.trans turns the channels-last rows into
//     both (eight consecutive 16-byte rows: no bank conflicts).  Four ldmatrix
//     feed six MMAs, 24 accumulators per lane.
//   * The CTA's 27 x 256 sums go to dw with one atomicAdd each; the bias
//     gradient is an MMA of dy with a matrix of ones.  Voxels beyond the grid and
//     channels beyond cout are staged as zeros of dy, and the x that only those
//     would meet as zeros too: a tile on 1^3 that fetched its 972 wrapped images
//     of the one voxel took 37 us for 128->128 (all CTAs on the same lines),
//     5.5 us with the 27 that are needed.
// Measured at 64^3 (the 14 layers of the U-Net): 1.85 ms with one tap per CTA,
// which read both operands 27 times, 0.30 ms with this kernel.
constexpr int kWgThreads = 288;
constexpr int kWgXV = 18 * 18, kWgGV = 16 * 16;         // staged voxels of an x and a dy plane
constexpr int kWgXB = kWgXV * 32, kWgGB = kWgGV * 32;   // bytes
constexpr size_t kWgSmem = 4 * kWgXB + 2 * kWgGB;

__device__ __forceinline__ void ldsm_x4_t(unsigned &r0, unsigned &r1, unsigned &r2, unsigned &r3, unsigned p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(p));
}

__global__ void __launch_bounds__(kWgThreads) k_wgrad_mma(Act x, Act gy, float *__restrict__ dw,
                                                           float *__restrict__ db, int tw, int th, int tz, int nz) {
    extern __shared__ __align__(128) unsigned char smw[];
    unsigned char *SX = smw, *SG = smw + 4 * kWgXB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cin = x.c, cout = gy.c, nbo = (cout + 15) >> 4;
    const int ci0 = (blockIdx.y / nbo) * 16, co0 = (blockIdx.y % nbo) * 16;
    int t = blockIdx.x;
    const int w0 = (t % tw) * 16;
    t /= tw;
    const int h0 = (t % th) * 16;
    t /= th;
    const int z0 = (t % tz) * nz, n = t / tz, z1 = min(z0 + nz, x.d);
    const bf16 *xn = x.p + (long long)n * x.d * x.h * x.w * x.ld + ci0;
    const bf16 *gn = gy.p + (long long)n * x.d * x.h * x.w * gy.ld + co0;
    const int xz = x.h * x.w * x.ld, gz = x.h * x.w * gy.ld;
    // this thread's copies of a plane: chunk e = tid + kWgThreads u is group e & 1 of voxel e >> 1
    // -1: only products with the dy beyond the grid need it, a zero there
    int xo[3], go[2];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const int e = tid + kWgThreads * u, v = e >> 1, vh = v / 18, vw = v % 18;
        const bool need = e < 2 * kWgXV && vh <= min(16, x.h - h0) + 1 && vw <= min(16, x.w - w0) + 1;
        xo[u] = need ? (wrapn(h0 - 1 + vh, x.h) * x.w + wrapn(w0 - 1 + vw, x.w)) * x.ld + (e & 1) * 8 : -1;
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int e = tid + kWgThreads * u, h = h0 + (e >> 5), w = w0 + ((e >> 1) & 15);
        go[u] = e < 2 * kWgGV && h < x.h && w < x.w && co0 + (e & 1) * 8 < cout ? (h * x.w + w) * gy.ld + (e & 1) * 8 : -1;
    }
    auto load_x = [&](int p) {  // plane p of d, in [z0 - 1, z1]
        const bf16 *src = xn + (long long)wrapn(p, x.d) * xz;
        unsigned char *dst = SX + (size_t)((p - z0 + 1) & 3) * kWgXB;
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const int e = tid + kWgThreads * u;
            if (e >= 2 * kWgXV) continue;
            unsigned char *d = dst + (e & 1) * (kWgXV * 16) + (e >> 1) * 16;
            if (xo[u] >= 0) cpa16(d, src + xo[u]);
            else *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
        }
    };
    auto load_g = [&](int z) {
        const bf16 *src = gn + (long long)z * gz;
        unsigned char *dst = SG + (size_t)((z - z0) & 1) * kWgGB;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int e = tid + kWgThreads * u;
            if (e >= 2 * kWgGV) continue;
            unsigned char *d = dst + (e & 1) * (kWgGV * 16) + (e >> 1) * 16;
            if (go[u] >= 0) cpa16(d, src + go[u]);
            else *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
        }
    };
    load_x(z0 - 1);
    load_x(z0);
    load_x(z0 + 1);
    load_g(z0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float acc[3][2][4] = {}, accb[2][4] = {};
    const bool bias = db && warp == 4 && ci0 == 0;
    const int dz = warp / 3, dy = warp % 3;
    // ldmatrix: lane L gives the row (L & 7) of matrix L >> 3
    const int mi = lane >> 3, r8 = lane & 7;
    const unsigned xa = smem_u32(SX) + ((mi & 1) * kWgXV + (mi >> 1) * 8 + r8 + dy * 18) * 16;  // (ci half, voxel half)
    const unsigned ga = smem_u32(SG) + ((mi >> 1) * kWgGV + (mi & 1) * 8 + r8) * 16;            // (co half, voxel half)
    for (int z = z0; z < z1; z++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // plane z + 1 of x and z of dy are there, the slots of z - 2 and z - 1 free
        if (z + 1 < z1) {
            load_x(z + 2);
            load_g(z + 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const unsigned xs = xa + ((z - z0 + dz) & 3) * kWgXB, gs = ga + ((z - z0) & 1) * kWgGB;
#pragma unroll 4
        for (int row = 0; row < 16; row++) {
            unsigned b0, b1, b2, b3;
            ldsm_x4_t(b0, b1, b2, b3, gs + row * 256);
            if (bias) {
                mma16816(accb[0], 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, b0, b1);
                mma16816(accb[1], 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, b2, b3);
            }
#pragma unroll
            for (int dx = 0; dx < 3; dx++) {
                unsigned a0, a1, a2, a3;
                ldsm_x4_t(a0, a1, a2, a3, xs + (row * 18 + dx) * 16);
                mma16816(acc[dx][0], a0, a1, a2, a3, b0, b1);
                mma16816(acc[dx][1], a0, a1, a2, a3, b2, b3);
            }
        }
    }
    // D fragment: rows g, g + 8 (ci), columns 2 t4, 2 t4 + 1 of each co half
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
        const int co = co0 + hf * 8 + 2 * t4;
        if (co >= cout) continue;
#pragma unroll
        for (int dx = 0; dx < 3; dx++) {
            float *o = dw + ((long long)(dz * 9 + dy * 3 + dx) * cin + ci0 + g) * cout + co;
            atomicAdd(o, acc[dx][hf][0]);
            atomicAdd(o + 1, acc[dx][hf][1]);
            atomicAdd(o + 8LL * cout, acc[dx][hf][2]);
            atomicAdd(o + 8LL * cout + 1, acc[dx][hf][3]);
        }
        if (bias && g == 0) {
            atomicAdd(db + co, accb[hf][0]);
            atomicAdd(db + co + 1, accb[hf][1]);
        }
    }
}

// tensor cores: channel counts in whole tiles and 16-byte aligned channel rows
bool wgrad_mma(const Act &x, const Act &gy) {
    static const bool off = getenv("BBMG_NO_WGRAD_MMA") != nullptr;
    return !off && x.c % 16 == 0 && gy.c % 8 == 0 && x.ld % 8 == 0 && gy.ld % 8 == 0 &&
           !(reinterpret_cast<uintptr_t>(x.p) & 15) && !(reinterpret_cast<uintptr_t>(gy.p) & 15);
}

// planes per CTA: a CTA ends with 27 x 256 atomic additions, so as many planes
// as leave two CTAs per SM
int wgrad_planes(const Act &x, const Act &gy) {
    const int blocks = (x.c / 16) * ((gy.c + 15) / 16);
    const long long cols = (long long)((x.w + 15) / 16) * ((x.h + 15) / 16) * x.n;
    int nz = x.d;
    while (nz > 1 && cols * blocks * ((x.d + nz - 1) / nz) < 2 * 148) nz = (nz + 1) / 2;
    return nz;
}

// ---------------------------------------------------------------------------
__global__ void k_pack(const float *__restrict__ w, int cin, int cout, bf16 *__restrict__ wt, bf16 *__restrict__ wd) {
    const long long n = 27LL * cin * cout;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int tap = (int)(e / (cin * cout)), r = (int)(e % (cin * cout)), ci = r / cout, co = r % cout;
        const bf16 v = __float2bfloat16(w[e]);
        wt[((long long)tap * cout + co) * cin + ci] = v;               // forward: [tap][co][ci]
        wd[((long long)(26 - tap) * cin + ci) * cout + co] = v;        // backward: [26-tap][ci][co]
    }
}

// The elementwise kernels take V channels per thread: V = 8 (one 16-byte access)
// on views whose rows are 16-byte aligned, else 1.  Ch is aligned as its access is.
template <int V> struct alignas(V == 8 ? 16 : 2) Ch {
    bf16 v[V];
};
static_assert(alignof(Ch<8>) == 16 && sizeof(Ch<8>) == 16 && sizeof(Ch<1>) == 2, "accessed as one vector");
template <int V> __device__ __forceinline__ Ch<V> ldc(const Act &a, int v, int c) {
    Ch<V> r;
    const bf16 *p = a.p + (long long)v * a.ld + c;
    if (V == 8) *reinterpret_cast<uint4 *>(r.v) = *reinterpret_cast<const uint4 *>(p);
    else r.v[0] = p[0];
    return r;
}
template <int V> __device__ __forceinline__ void stc(const Act &a, int v, int c, const Ch<V> &r) {
    bf16 *p = a.p + (long long)v * a.ld + c;
    if (V == 8) *reinterpret_cast<uint4 *>(p) = *reinterpret_cast<const uint4 *>(r.v);
    else p[0] = r.v[0];
}
#define FOR_CHANNELS(a)                                                                                              \
    const int cg_ = (a).c / V;                                                                                       \
    const long long n_ = (long long)(a).nvox * cg_;                                                                  \
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n_; e += (long long)gridDim.x * blockDim.x)

template <int V> __global__ void k_relu_bwd(Act dy, Act y) {
    FOR_CHANNELS(dy) {
        const int v = (int)(e / cg_), c = V * (int)(e - (long long)v * cg_);
        const Ch<V> a = ldc<V>(y, v, c);
        Ch<V> g = ldc<V>(dy, v, c);
#pragma unroll
        for (int q = 0; q < V; q++)
            if (!(__bfloat162float(a.v[q]) > 0.f)) g.v[q] = __float2bfloat16(0.f);
        stc<V>(dy, v, c, g);
    }
}

// y (half size) = mean of the 8 children of x
template <int V> __global__ void k_pool2(Act x, Act y) {
    FOR_CHANNELS(y) {
        const int v = (int)(e / cg_), c = V * (int)(e - (long long)v * cg_);
        int nn, d, h, w;
        decode(y, v, nn, d, h, w);
        Ch<V> in[8];
#pragma unroll
        for (int q = 0; q < 8; q++) in[q] = ldc<V>(x, vox(x, nn, 2 * d + (q >> 2), 2 * h + ((q >> 1) & 1), 2 * w + (q & 1)), c);
        Ch<V> o;
#pragma unroll
        for (int m = 0; m < V; m++) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) s += __bfloat162float(in[q].v[m]);
            o.v[m] = __float2bfloat16(0.125f * s);
        }
        stc<V>(y, v, c, o);
    }
}
// dx (twice the size of dy) = dy(parent) / 8, or dx += that (accumulate: the
// pooled tensor is also a skip connection whose gradient is already in dx)
template <int V> __global__ void k_pool2_bwd(Act dy, Act dx, int accumulate) {
    FOR_CHANNELS(dx) {
        const int v = (int)(e / cg_), c = V * (int)(e - (long long)v * cg_);
        int nn, d, h, w;
        decode(dx, v, nn, d, h, w);
        const Ch<V> p = ldc<V>(dy, vox(dy, nn, d >> 1, h >> 1, w >> 1), c);
        Ch<V> o;
        if (accumulate) o = ldc<V>(dx, v, c);
#pragma unroll
        for (int m = 0; m < V; m++) {
            float g = 0.125f * __bfloat162float(p.v[m]);
            if (accumulate) g += __bfloat162float(o.v[m]);
            o.v[m] = __float2bfloat16(g);
        }
        stc<V>(dx, v, c, o);
    }
}
// y (twice the size of x) = x(parent)
template <int V> __global__ void k_up2(Act x, Act y) {
    FOR_CHANNELS(y) {
        const int v = (int)(e / cg_), c = V * (int)(e - (long long)v * cg_);
        int nn, d, h, w;
        decode(y, v, nn, d, h, w);
        stc<V>(y, v, c, ldc<V>(x, vox(x, nn, d >> 1, h >> 1, w >> 1), c));
    }
}
// dx (half the size of dy) = sum of the 8 children of dy
template <int V> __global__ void k_up2_bwd(Act dy, Act dx) {
    FOR_CHANNELS(dx) {
        const int v = (int)(e / cg_), c = V * (int)(e - (long long)v * cg_);
        int nn, d, h, w;
        decode(dx, v, nn, d, h, w);
        Ch<V> in[8];
#pragma unroll
        for (int q = 0; q < 8; q++) in[q] = ldc<V>(dy, vox(dy, nn, 2 * d + (q >> 2), 2 * h + ((q >> 1) & 1), 2 * w + (q & 1)), c);
        Ch<V> o;
#pragma unroll
        for (int m = 0; m < V; m++) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) s += __bfloat162float(in[q].v[m]);
            o.v[m] = __float2bfloat16(s);
        }
        stc<V>(dx, v, c, o);
    }
}

struct Fields {
    const double *f[NN_MAX_FIELDS];
    double s[NN_MAX_FIELDS];
    int nf;
};

// pool = 1: the fields are on x's grid.  pool = 2: they are on the grid twice
// as fine and each voxel gets the mean of its 8 children (FP64 sum).
template <int V> __global__ void k_embed(Fields fs, Act x, int pool) {
    FOR_CHANNELS(x) {
        const int v = (int)(e / cg_), c0 = V * (int)(e - (long long)v * cg_);
        Ch<V> o;
#pragma unroll
        for (int m = 0; m < V; m++) o.v[m] = __float2bfloat16(0.f);
        if (c0 < fs.nf) {
            int nn, d, h, w;
            if (pool == 2) decode(x, v, nn, d, h, w);
#pragma unroll
            for (int m = 0; m < (V < NN_MAX_FIELDS ? V : NN_MAX_FIELDS); m++) {
                const int c = c0 + m;
                if (c >= fs.nf) continue;
                if (pool == 1) {
                    o.v[m] = __float2bfloat16((float)(fs.s[c] * fs.f[c][v]));
                } else {
                    const int D = 2 * x.d, H = 2 * x.h, W = 2 * x.w;
                    const double *f = fs.f[c] + (long long)nn * D * H * W;
                    double sum = 0.0;
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        sum += f[((long long)(2 * d + (q >> 2)) * H + (2 * h + ((q >> 1) & 1))) * W + 2 * w + (q & 1)];
                    o.v[m] = __float2bfloat16((float)(fs.s[c] * 0.125 * sum));
                }
            }
        }
        stc<V>(x, v, c0, o);
    }
}

template <int V> __global__ void k_head(Act x, const float *__restrict__ w, const float *__restrict__ b, float *__restrict__ out) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < x.nvox; v += gridDim.x * blockDim.x) {
        float s = b[0];
        for (int c = 0; c < x.c; c += V) {
            const Ch<V> a = ldc<V>(x, v, c);
#pragma unroll
            for (int m = 0; m < V; m++) s = fmaf(__bfloat162float(a.v[m]), w[c + m], s);
        }
        out[v] = s;
    }
}

// one group of V channels per blockIdx.y: the sums stay in registers until the
// grid-stride loop ends, then go over the warp and the block
template <int V>
__global__ void __launch_bounds__(256) k_head_bwd(Act x, const float *__restrict__ w, const float *__restrict__ dout,
                                                   Act dx, float *__restrict__ dw, float *__restrict__ db) {
    __shared__ float sh[8][V + 1];
    const int c = blockIdx.y * V, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float acc[V + 1], wc[V];
#pragma unroll
    for (int m = 0; m <= V; m++) acc[m] = 0.f;
#pragma unroll
    for (int m = 0; m < V; m++) wc[m] = w[c + m];
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < x.nvox; v += gridDim.x * blockDim.x) {
        const float g = dout[v];
        const Ch<V> a = ldc<V>(x, v, c);
        Ch<V> o;
#pragma unroll
        for (int m = 0; m < V; m++) {
            o.v[m] = __float2bfloat16(g * wc[m]);
            acc[m] += g * __bfloat162float(a.v[m]);
        }
        acc[V] += g;
        stc<V>(dx, v, c, o);
    }
#pragma unroll
    for (int m = 0; m <= V; m++) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc[m] += __shfl_down_sync(0xffffffffu, acc[m], s);
        if (lane == 0) sh[warp][m] = acc[m];
    }
    __syncthreads();
    if (threadIdx.x <= V) {
        float s = 0.f;
        for (int q = 0; q < 8; q++) s += sh[q][threadIdx.x];
        if (threadIdx.x < V) atomicAdd(dw + c + threadIdx.x, s);
        else if (blockIdx.y == 0) atomicAdd(db, s);
    }
}

__global__ void k_mse(const float *__restrict__ pred, const double *__restrict__ tgt, double scale, long long n,
                      float *__restrict__ grad, double *loss) {
    __shared__ double sh[256];
    double s = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const double d = (double)pred[v] - scale * tgt[v];
        grad[v] = (float)(2.0 * d / (double)n);
        s += d * d;
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, sh[0]);
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       long long n, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float gg = g[e];
        const float mm = b1 * m[e] + (1.f - b1) * gg;
        const float vv = b2 * v[e] + (1.f - b2) * gg * gg;
        m[e] = mm;
        v[e] = vv;
        w[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    }
}

// out = base + scale * pred, pred given on the same grid (up = 1) or on a grid
// half as fine (up = 2), then interpolated trilinearly between cell centres
// (weights 3/4 and 1/4 per direction, periodic wrap).
__global__ void k_apply(const double *__restrict__ base, const float *__restrict__ pred, double scale, int nb, int d,
                        int h, int w, int up, double *__restrict__ out) {
    const int D = d * up, H = h * up, W = w * up;
    const long long n = (long long)nb * D * H * W;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        double v;
        if (up == 1) {
            v = (double)pred[e];
        } else {
            const int i = (int)(e % W), j = (int)((e / W) % H), k = (int)((e / ((long long)W * H)) % D);
            const int b = (int)(e / ((long long)W * H * D));
            const int i0 = i >> 1, j0 = j >> 1, k0 = k >> 1;
            const int i1 = wrapi(i0 + ((i & 1) ? 1 : -1), w), j1 = wrapi(j0 + ((j & 1) ? 1 : -1), h),
                      k1 = wrapi(k0 + ((k & 1) ? 1 : -1), d);
            const float *pb = pred + (long long)b * d * h * w;
            float acc = 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int kk = (q & 4) ? k1 : k0, jj = (q & 2) ? j1 : j0, ii = (q & 1) ? i1 : i0;
                const float wq = ((q & 4) ? 0.25f : 0.75f) * ((q & 2) ? 0.25f : 0.75f) * ((q & 1) ? 0.25f : 0.75f);
                acc = fmaf(wq, pb[((long long)kk * h + jj) * w + ii], acc);
            }
            v = (double)acc;
        }
        out[e] = (base ? base[e] : 0.0) + scale * v;
    }
}

int grid_elems(long long n) {
    long long g = (n + 255) / 256;
    if (g > 148 * 32) g = 148 * 32;
    return (int)(g < 1 ? 1 : g);
}

// views the elementwise kernels take eight channels at a time
bool vec8(const Act &a) { return a.c % 8 == 0 && a.ld % 8 == 0 && !(reinterpret_cast<uintptr_t>(a.p) & 15); }
// Means and sums of eight children keep one channel per thread while the outputs
// are few: there a thread's eight sums one after the other take longer than the
// loads.  8192 outputs take 1.8 us with one channel per thread and 2.2 with eight,
// 65536 2.05 and 2.3, 110592 2.37 and 2.31, 262144 3.5 and 2.4.
bool small(const Act &a) { return (long long)a.nvox * a.c <= 148 * 640; }
#define BB_CHANNELS(eight, view, kern, ...)                                                                          \
    do {                                                                                                             \
        if (eight)                                                                                                   \
            kern<8><<<grid_elems((long long)(view).nvox * (view).c / 8), 256, 0, (cudaStream_t)stream>>>(__VA_ARGS__); \
        else                                                                                                         \
            kern<1><<<grid_elems((long long)(view).nvox * (view).c), 256, 0, (cudaStream_t)stream>>>(__VA_ARGS__);   \
    } while (0)

}  // namespace

// ===========================================================================
extern "C" {

int nn_conv3(const nn_act *x, const void *wt, const float *bias, const nn_act *y, int relu, void *stream) {
    if (bad_act(x) || bad_act(y) || !wt || x->c % 16 || y->c % 16 || x->n != y->n || x->d != y->d ||
        x->h != y->h || x->w != y->w)
        return BBMG_BAD_ARGS;
    return launch_conv(act_of(x), (const bf16 *)wt, bias, act_of(y), relu, (cudaStream_t)stream);
}

int nn_conv3_dgrad(const nn_act *dy, const void *wd, const nn_act *dx, void *stream) {
    // conv of dy with the [tap'][ci][co] packing: input channels = cout of the
    // forward, output channels = its cin; with taps mirrored this is the
    // transposed convolution.
    if (bad_act(dy) || bad_act(dx) || !wd || dy->c % 16 || dx->c % 16 || dy->n != dx->n || dy->d != dx->d ||
        dy->h != dx->h || dy->w != dx->w)
        return BBMG_BAD_ARGS;
    return launch_conv(act_of(dy), (const bf16 *)wd, nullptr, act_of(dx), 0, (cudaStream_t)stream);
}

int bbmg_debug_conv3(const nn_act *x, const void *wt, const nn_act *y, int *tcgen05, int *planes, int *buffers,
                     int *slots) {
    if (bad_act(x) || bad_act(y) || !wt || !tcgen05 || !planes || !buffers || !slots) return BBMG_BAD_ARGS;
    const Act ax = act_of(x), ay = act_of(y);
    *tcgen05 = tc_eligible(ax, (const bf16 *)wt, ay);
    *planes = *buffers = *slots = 0;
    if (!*tcgen05) return BBMG_OK;
    return with_width(ay.c, [&](auto width, auto groups) {
        const ZmGeo g = conv_geo<decltype(width)::value>(ax, decltype(groups)::value);
        *planes = g.dz;
        *buffers = g.nb;
        *slots = g.slots;
        return BBMG_OK;
    });
}

int bbmg_debug_conv3_wgrad(const nn_act *x, const nn_act *dy, int *tensor, int *planes) {
    if (bad_act(x) || bad_act(dy) || !tensor || !planes) return BBMG_BAD_ARGS;
    const Act ax = act_of(x), ag = act_of(dy);
    *tensor = wgrad_mma(ax, ag);
    *planes = *tensor ? wgrad_planes(ax, ag) : 0;
    return BBMG_OK;
}

int nn_conv3_wgrad(const nn_act *x, const nn_act *dy, float *dw, float *db, void *stream) {
    if (bad_act(x) || bad_act(dy) || !dw || x->n != dy->n || x->d != dy->d || x->h != dy->h || x->w != dy->w ||
        dy->c > 256)
        return BBMG_BAD_ARGS;
    const Act ax = act_of(x), ag = act_of(dy);
    if (wgrad_mma(ax, ag)) {
        static std::atomic<uint64_t> seen{0};
        if (!allow_smem(k_wgrad_mma, (int)kWgSmem, seen)) return BBMG_CUDA;
        const int tw = (ax.w + 15) / 16, th = (ax.h + 15) / 16, blocks = (ax.c / 16) * ((ag.c + 15) / 16);
        const long long cols = (long long)tw * th * ax.n;
        if (blocks > 65535 || cols * ax.d >= (1LL << 31)) return BBMG_BAD_ARGS;
        const int nz = wgrad_planes(ax, ag), tz = (ax.d + nz - 1) / nz;
        k_wgrad_mma<<<dim3((unsigned)(cols * tz), blocks), kWgThreads, kWgSmem, (cudaStream_t)stream>>>(ax, ag, dw, db, tw, th, tz, nz);
        return done(cudaGetLastError());
    }
    const int chunks = 148 * 4 / 27 + 1;
    int vchunk = (ag.nvox + chunks - 1) / chunks;
    vchunk = (vchunk + kWgVB - 1) / kWgVB * kWgVB;
    const int nchunk = (ag.nvox + vchunk - 1) / vchunk;
    const size_t shm = sizeof(float) * kWgVB * (ax.c + ag.c);
    const int nz = (ax.c * ag.c + 24 * 256 - 1) / (24 * 256);
    k_wgrad<<<dim3(nchunk, 27, nz), 256, shm, (cudaStream_t)stream>>>(ax, ag, dw, db, vchunk);
    return done(cudaGetLastError());
}

int nn_tc_error(void) {
    int v = 0;
    const int none = 0;
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(&v, g_tc_err, sizeof(int)) != cudaSuccess)
        return BBMG_CUDA;
    if (v && cudaMemcpyToSymbol(g_tc_err, &none, sizeof(int)) != cudaSuccess) return BBMG_CUDA;
    return v ? BBMG_CUDA : BBMG_OK;
}

int nn_pack_weights(const float *w, int cin, int cout, void *wt, void *wd, void *stream) {
    if (!w || !wt || !wd || cin < 1 || cout < 1) return BBMG_BAD_ARGS;
    k_pack<<<grid_elems(27LL * cin * cout), 256, 0, (cudaStream_t)stream>>>(w, cin, cout, (bf16 *)wt, (bf16 *)wd);
    return done(cudaGetLastError());
}

int nn_relu_bwd(const nn_act *dy, const nn_act *y, void *stream) {
    if (bad_act(dy) || bad_act(y) || dy->c != y->c) return BBMG_BAD_ARGS;
    const Act a = act_of(dy), b = act_of(y);
    BB_CHANNELS(vec8(a) && vec8(b), a, k_relu_bwd, a, b);
    return done(cudaGetLastError());
}

static bool halves(const nn_act *big, const nn_act *small) {
    return big->n == small->n && big->d == 2 * small->d && big->h == 2 * small->h && big->w == 2 * small->w &&
           big->c == small->c;
}

int nn_pool2(const nn_act *x, const nn_act *y, void *stream) {
    if (bad_act(x) || bad_act(y) || !halves(x, y)) return BBMG_BAD_ARGS;
    const Act a = act_of(x), b = act_of(y);
    BB_CHANNELS(vec8(a) && vec8(b) && !small(b), b, k_pool2, a, b);
    return done(cudaGetLastError());
}
int nn_pool2_bwd(const nn_act *dy, const nn_act *dx, int accumulate, void *stream) {
    if (bad_act(dy) || bad_act(dx) || !halves(dx, dy)) return BBMG_BAD_ARGS;
    const Act a = act_of(dy), b = act_of(dx);
    BB_CHANNELS(vec8(a) && vec8(b), b, k_pool2_bwd, a, b, accumulate);
    return done(cudaGetLastError());
}
int nn_up2(const nn_act *x, const nn_act *y, void *stream) {
    if (bad_act(x) || bad_act(y) || !halves(y, x)) return BBMG_BAD_ARGS;
    const Act a = act_of(x), b = act_of(y);
    BB_CHANNELS(vec8(a) && vec8(b), b, k_up2, a, b);
    return done(cudaGetLastError());
}
int nn_up2_bwd(const nn_act *dy, const nn_act *dx, void *stream) {
    if (bad_act(dy) || bad_act(dx) || !halves(dy, dx)) return BBMG_BAD_ARGS;
    const Act a = act_of(dy), b = act_of(dx);
    BB_CHANNELS(vec8(a) && vec8(b) && !small(b), b, k_up2_bwd, a, b);
    return done(cudaGetLastError());
}

int nn_embed(int nf, const double *const *fields, const double *scales, int pool, const nn_act *x, void *stream) {
    if (bad_act(x) || nf < 1 || nf > NN_MAX_FIELDS || nf > x->c || !fields || !scales || (pool != 1 && pool != 2))
        return BBMG_BAD_ARGS;
    Fields fs{};
    fs.nf = nf;
    for (int i = 0; i < nf; i++) {
        if (!fields[i]) return BBMG_BAD_ARGS;
        fs.f[i] = fields[i];
        fs.s[i] = scales[i];
    }
    const Act a = act_of(x);
    BB_CHANNELS(vec8(a), a, k_embed, fs, a, pool);
    return done(cudaGetLastError());
}

int nn_head(const nn_act *x, const float *w, const float *b, float *out, void *stream) {
    if (bad_act(x) || !w || !b || !out) return BBMG_BAD_ARGS;
    const Act a = act_of(x);
    if (vec8(a)) k_head<8><<<grid_elems(a.nvox), 256, 0, (cudaStream_t)stream>>>(a, w, b, out);
    else k_head<1><<<grid_elems(a.nvox), 256, 0, (cudaStream_t)stream>>>(a, w, b, out);
    return done(cudaGetLastError());
}

int nn_head_bwd(const nn_act *x, const float *w, const float *dout, const nn_act *dx, float *dw, float *db,
                void *stream) {
    if (bad_act(x) || bad_act(dx) || !w || !dout || !dw || !db || x->c > 128 || dx->c != x->c) return BBMG_BAD_ARGS;
    const Act a = act_of(x), d = act_of(dx);
    const unsigned gx = (unsigned)std::min(grid_elems(a.nvox), 148 * 4);
    if (vec8(a) && vec8(d))
        k_head_bwd<8><<<dim3(gx, a.c / 8), 256, 0, (cudaStream_t)stream>>>(a, w, dout, d, dw, db);
    else
        k_head_bwd<1><<<dim3(gx, a.c), 256, 0, (cudaStream_t)stream>>>(a, w, dout, d, dw, db);
    return done(cudaGetLastError());
}

int nn_mse(const float *pred, const double *target, double scale, long long nvox, float *grad, double *loss,
           void *stream) {
    if (!pred || !target || !grad || !loss || nvox < 1) return BBMG_BAD_ARGS;
    k_mse<<<grid_elems(nvox), 256, 0, (cudaStream_t)stream>>>(pred, target, scale, nvox, grad, loss);
    return done(cudaGetLastError());
}

int nn_adam(float *w, const float *g, float *m, float *v, long long n, float lr, float b1, float b2, float eps,
            int t, void *stream) {
    if (!w || !g || !m || !v || n < 1 || t < 1) return BBMG_BAD_ARGS;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    k_adam<<<grid_elems(n), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, b1, b2, eps, c1, c2);
    return done(cudaGetLastError());
}

int nn_apply(const double *base, const float *pred, double scale, int nb, int d, int h, int w, int up, double *out,
             void *stream) {
    if (!pred || !out || nb < 1 || d < 1 || h < 1 || w < 1 || (up != 1 && up != 2) ||
        (long long)nb * d * h * w * up * up * up >= (1LL << 40))
        return BBMG_BAD_ARGS;
    const long long n = (long long)nb * d * h * w * up * up * up;
    k_apply<<<grid_elems(n), 256, 0, (cudaStream_t)stream>>>(base, pred, scale, nb, d, h, w, up, out);
    return done(cudaGetLastError());
}

}  // extern "C"
