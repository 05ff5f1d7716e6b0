// vtail.cu -- the coarse levels of the V-cycle in one launch, and the coarsest solve.
//
// cycle(n) (src/solver/bbmg_class.f90:732-776) for every level n0..nlvl inside
// one thread-block cluster.  A level's k-planes are dealt out in slabs, one per
// block; v, f and r live in the blocks' shared memory, each block also holding
// the planes just below and above its slab.  A pass (a Gauss-Seidel colour,
// residual, restriction, prolongation) reads v from the block's own shared
// memory, writes each new value there and, at a slab face or a periodic face,
// straight into the neighbour's copy (distributed shared memory); the cluster's
// hardware barrier ends the pass.  The operator does not depend on the pass
// before: the coefficients of the coarser levels are staged in shared memory
// before the wait for the predecessor, as many levels as fit, and those of the
// others are loaded from L2 into registers between arriving at a barrier and
// waiting for it.  Levels of at most kTailSingle cells, and always the coarsest,
// run inside block 0 with block-wide barriers while the others wait.
//
// What bounds it: a pass is a chain of latencies (barrier 0.4e3 cycles, shared
// memory loads, a sum in the reference's order, a division) of a few warps, no
// longer a kernel launch or an L2 round trip for v; FP64 levels of 16^3 and 32^3
// wait for their coefficients from L2, and with a 4- or 7-plane first level their
// kernel spills (255 registers, 3.8 KB of stores and 1.3 KB of loads; 0.8 and 0.3
// KB with 27 planes, FP32 none to speak of).  With the levels below 8^3 fused and
// the others one launch per colour, a 32^3 mixed solve took 3.13 ms and a 64^3 FP64
// one 4.19; fused from 32^3 they take 1.62 and 2.75 ms.  A cluster is scheduled
// as a unit, so no block can wait on one that is not running, and no barrier
// outlives its kernel.
//
// Arithmetic and term order are those of the single-pass kernels (solve.cu):
// FP64 results are the oracle's bits.
#include <algorithm>
#include <mutex>

#include "ops.cuh"

namespace bbmg {

namespace {

// ---------------------------------------------------------------------------
// coarsest level (bbmg_class.f90:891-927): the stored LU, FP64 always

// The factors as the solve reads them, column major: staged in shared memory
// with ld a multiple of 8, the rows and columns beyond np those of a unit
// matrix, or as they lie in global memory, where reads beyond np give that.
template <bool STAGED> struct Factors {
    const double *A;
    int np, ld;
    __device__ __forceinline__ double at(int r, int c) const {
        if (STAGED) return A[c * ld + r];
        return r < np && c < np ? __ldg(A + c * np + r) : (r == c ? 1.0 : 0.0);
    }
};

// x(i) of lane i % 32, register i / 32.
// Eight unknowns at a time: every lane solves their small triangle itself (the
// values come by eight independent shuffles), then updates its own rows with
// them.  Each x(i) still loses its terms one by one in increasing (backward:
// decreasing) order, so the values are those of the column-by-column solve;
// the chain per unknown is a product and a difference instead of a shuffle,
// a load and a store as well.  From global memory a block of eight costs one L2
// round trip (its coefficients do not depend on x) instead of eight.
template <int M, bool STAGED>
__device__ __forceinline__ void lu_solve_warp(const Factors<STAGED> &F, const int *__restrict__ pinned, int lane,
                                              double (&x)[M]) {
    const int np = F.np, rows = STAGED ? F.ld : np;
    unsigned pin[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int i = lane + 32 * m;
        pin[m] = __ballot_sync(0xffffffffu, i < np && pinned[i] != 0);
    }
#pragma unroll
    for (int mk = 0; mk < M; mk++) {
#pragma unroll 1
        for (int l0 = 0; l0 < 32; l0 += 8) {
            const int k0 = 32 * mk + l0;
            if (k0 >= np) break;
            double xb[8];
#pragma unroll
            for (int j = 0; j < 8; j++) xb[j] = __shfl_sync(0xffffffffu, x[mk], l0 + j);
#pragma unroll
            for (int j = 0; j < 7; j++)
#pragma unroll
                for (int i = j + 1; i < 8; i++) xb[i] = __dsub_rn(xb[i], __dmul_rn(xb[j], F.at(k0 + i, k0 + j)));
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (lane == l0 + j) x[mk] = xb[j];
#pragma unroll
            for (int m = mk; m < M; m++) {
                const int i = lane + 32 * m;
                if (i >= k0 + 8 && i < rows) {
#pragma unroll
                    for (int j = 0; j < 8; j++) x[m] = __dsub_rn(x[m], __dmul_rn(xb[j], F.at(i, k0 + j)));
                }
            }
        }
    }
#pragma unroll
    for (int mk = M - 1; mk >= 0; mk--) {
#pragma unroll 1
        for (int l0 = 24; l0 >= 0; l0 -= 8) {
            const int k0 = 32 * mk + l0;
            if (k0 >= np) continue;
            double xb[8];
#pragma unroll
            for (int j = 0; j < 8; j++) xb[j] = __shfl_sync(0xffffffffu, x[mk], l0 + j);
#pragma unroll
            for (int j = 7; j >= 0; j--) {
                // a pinned unknown is zero whatever its pivot
                xb[j] = (pin[mk] >> (l0 + j)) & 1u ? 0.0 : __ddiv_rn(xb[j], F.at(k0 + j, k0 + j));
#pragma unroll
                for (int i = 0; i < j; i++) xb[i] = __dsub_rn(xb[i], __dmul_rn(xb[j], F.at(k0 + i, k0 + j)));
            }
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (lane == l0 + j) x[mk] = xb[j];
#pragma unroll
            for (int m = 0; m <= mk; m++) {
                const int i = lane + 32 * m;
                if (i < k0) {
#pragma unroll
                    for (int j = 7; j >= 0; j--) x[m] = __dsub_rn(x[m], __dmul_rn(xb[j], F.at(i, k0 + j)));
                }
            }
        }
    }
}

// leading dimension of the factors in shared memory, and their copy there
__host__ __device__ constexpr int lu_ld(int np) { return (np + 7) / 8 * 8; }
__device__ __forceinline__ void lu_stage(const double *__restrict__ LU, int np, double *A) {
    const int ld = lu_ld(np);
    for (int e = threadIdx.x; e < ld * ld; e += blockDim.x) {
        const int c = e / ld, r = e - c * ld;
        A[e] = r < np && c < np ? LU[(long long)c * np + r] : (r == c ? 1.0 : 0.0);
    }
}

// factors left in global memory: column by column, x in shared memory
__device__ __noinline__ void lu_solve_mem(const double *__restrict__ A, const int *__restrict__ pinned, int np,
                                          int lane, double *x) {
    for (int kk = 0; kk < np; kk++) {
        const double xk = x[kk];
        if (xk != 0.0)
            for (int i = kk + 1 + lane; i < np; i += 32)
                x[i] = __dsub_rn(x[i], __dmul_rn(xk, A[(long long)kk * np + i]));
        __syncwarp();
    }
    for (int kk = np - 1; kk >= 0; kk--) {
        if (pinned[kk]) {
            if (lane == 0) x[kk] = 0.0;
            __syncwarp();
            continue;
        }
        double xk = x[kk];
        __syncwarp();
        if (xk != 0.0) {
            xk = __ddiv_rn(xk, A[(long long)kk * np + kk]);
            if (lane == 0) x[kk] = xk;
            for (int i = lane; i < kk; i += 32) x[i] = __dsub_rn(x[i], __dmul_rn(xk, A[(long long)kk * np + i]));
        }
        __syncwarp();
    }
}

template <int M, bool STAGED>
__device__ __forceinline__ void lu_solve_regs(const Factors<STAGED> &F, const int *__restrict__ pinned, int lane,
                                              double *xs) {
    double x[M];
#pragma unroll
    for (int m = 0; m < M; m++) x[m] = lane + 32 * m < F.np ? xs[lane + 32 * m] : 0.0;
    lu_solve_warp<M, STAGED>(F, pinned, lane, x);
#pragma unroll
    for (int m = 0; m < M; m++)
        if (lane + 32 * m < F.np) xs[lane + 32 * m] = x[m];
}
__device__ __noinline__ void lu_solve_l2(const double *__restrict__ LU, const int *__restrict__ pinned, int np,
                                         int lane, double *xs) {
    lu_solve_regs<5, false>(Factors<false>{LU, np, np}, pinned, lane, xs);
}

// xs: the row-permuted right-hand side in shared memory, replaced by the
// solution; one warp.  Factors staged in shared memory at A (up to 131 unknowns
// in the cluster, 160 in a launch of its own), or LU in global memory: eight
// columns at a time while x fits five registers a lane, else column by column.
// One cycle with 157 unknowns in the cluster: 203 us column by column, 136 us so.
__device__ __forceinline__ void lu_solve(const double *A, const double *__restrict__ LU, bool staged,
                                         const int *__restrict__ pinned, int np, int lane, double *xs) {
    if (!staged && np > 160) lu_solve_mem(LU, pinned, np, lane, xs);
    else if (!staged) lu_solve_l2(LU, pinned, np, lane, xs);
    else if (np <= 64) lu_solve_regs<2, true>(Factors<true>{A, np, lu_ld(np)}, pinned, lane, xs);
    else lu_solve_regs<5, true>(Factors<true>{A, np, lu_ld(np)}, pinned, lane, xs);
}

// The coarsest solve as a launch of its own (levels that are not fused): one
// block, the factors in shared memory when they fit.
template <typename T>
__global__ void __launch_bounds__(256) k_coarse_solve(Lay L, const double *__restrict__ LU,
                                                       const int *__restrict__ perm,
                                                       const int *__restrict__ pinned, const T *__restrict__ f,
                                                       T *__restrict__ v, int mat_in_smem) {
    pdl_launch();
    extern __shared__ double sd[];
    const int np = L.nx * L.ny * L.nz;
    double *x = sd;
    if (mat_in_smem) lu_stage(LU, np, sd + np);
    pdl_wait();
    for (int ind = threadIdx.x; ind < np; ind += blockDim.x) {
        const int p = perm[ind];
        x[ind] = (double)f[L.idx(p % L.nx, (p / L.nx) % L.ny, p / (L.nx * L.ny))];
    }
    __syncthreads();
    if (threadIdx.x < 32) lu_solve(sd + np, LU, mat_in_smem, pinned, np, threadIdx.x, x);
    __syncthreads();
    for (int ind = threadIdx.x; ind < np; ind += blockDim.x) {
        const int i = ind % L.nx, j = (ind / L.nx) % L.ny, k = ind / (L.nx * L.ny);
        const T val = (T)x[ind];
        v[L.idx(i, j, k)] = val;
        if (on_periodic_face(L, i, j, k)) write_images(L, v, i, j, k, val);
    }
}

// ---------------------------------------------------------------------------
// the cluster

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// A stage waits for the one before it at its start and arrives at its end, so
// that loads which do not depend on it go in between.  CL: levels dealt out
// over the cluster; otherwise block 0 alone.
template <bool CL> __device__ __forceinline__ void stage_wait() {
    if (CL) cl_wait();
    else __syncthreads();
}
template <bool CL> __device__ __forceinline__ void stage_arrive() {
    if (CL) cl_arrive();
}

// generic address of block `rank`'s copy of a shared variable
template <typename T> __device__ __forceinline__ T *in_block(T *p, int rank) {
    unsigned long long r;
    asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return reinterpret_cast<T *>(r);
}

// it / n for 0 <= it < 2^20, inv = 1.0f / n: the quotient's distance to the
// next integer is at least 0.5 / n, the rounding errors stay below it * 2^-22 / n
__device__ __forceinline__ int qdiv(int it, float inv) { return (int)(((float)it + 0.5f) * inv); }

template <typename T> __device__ __forceinline__ int slot_x(const TailLvl<T> &l, int i) {
    return (i & 1) ? (i + 1) >> 1 : l.E0 + (i >> 1);
}
template <typename T> __device__ __forceinline__ int owner(const TailLvl<T> &l, int k) { return l.single ? 0 : qdiv(k, l.iH); }
// plane k within its owner's slab
template <typename T> __device__ __forceinline__ int plane_in(const TailLvl<T> &l, int k, int o) { return k - o * l.H; }

// store to a neighbour block's shared memory (CL: a cluster address) or our own
template <bool CL> __device__ __forceinline__ void put(unsigned a, float v) {
    if (CL) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
    else asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
template <bool CL> __device__ __forceinline__ void put(unsigned a, double v) {
    if (CL) asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
    else asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// A block's part of a level.  V: planes k0-1 .. k0+nk in slots 0 .. nk+1, each
// plane rows j = -1 .. ny of PX elements, odd x first (i = -1 at 0), even x from
// E0; F, R: the own planes, rows 0 .. ny-1; C: the coefficients, one point's
// after the other.  prev / next: shared-memory address of the slot that holds
// the block's first / last plane as a neighbour's upper / lower plane (0 at a
// wall).
template <typename T> struct Blk {
    int k0, nk;
    T *V, *F, *R, *C;
    unsigned prev, next;
};

template <typename T, bool CL> __device__ __forceinline__ Blk<T> part(const TailLvl<T> &l, int rank, T *sm) {
    Blk<T> b;
    const int nz = l.L.nz;
    b.k0 = l.single ? (rank ? nz : 0) : min(nz, rank * l.H);
    b.nk = min(nz, b.k0 + l.H) - b.k0;
    b.V = sm + l.sv;
    b.F = sm + l.sf;
    b.R = sm + l.sr;
    b.C = sm + l.sc;
    b.prev = b.next = 0;
    if (b.nk > 0) {
        const unsigned v = (unsigned)__cvta_generic_to_shared(b.V);
        auto slot = [&](int k, int up) {
            const int o = owner(l, k);
            unsigned a = v + (unsigned)((plane_in(l, k, o) + up) * l.PP) * (unsigned)sizeof(T);
            if (CL) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(o));
            return a;
        };
        int k = b.k0 - 1;
        if (k < 0 && l.L.zper) k = nz - 1;
        if (k >= 0) b.prev = slot(k, 2);
        k = b.k0 + b.nk;
        if (k == nz && l.L.zper) k = 0;
        if (k < nz) b.next = slot(k, 0);
    }
    return b;
}

// the neighbours' copies of interior value val of own plane kl, held at element
// e of V, at the slab's faces
template <typename T, bool CL>
__device__ __forceinline__ void push_faces(const TailLvl<T> &l, const Blk<T> &b, int kl, int e, T val) {
    if (!CL) return;
    const unsigned o = (unsigned)(e - (kl + 1) * l.PP) * (unsigned)sizeof(T);
    if (kl == 0 && b.prev) put<CL>(b.prev + o, val);
    if (kl == b.nk - 1 && b.next) put<CL>(b.next + o, val);
}

// the same with the x and y periodic images in every copy, for levels whose
// reads do not wrap (an odd periodic size); block 0 alone copies its own faces
template <typename T, bool CL>
__device__ __forceinline__ void push(const TailLvl<T> &l, const Blk<T> &b, int i, int j, int kl, int e, T val) {
    const Lay &L = l.L;
    const bool lo = kl == 0 && b.prev, hi = kl == b.nk - 1 && b.next;
    const bool xb = L.xper && (i == 0 || i == L.nx - 1), yb = L.yper && (j == 0 || j == L.ny - 1);
    if (!(lo || hi || xb || yb)) return;
    const int in = e - (kl + 1) * l.PP;  // element within the plane
    auto copies = [&](int d, bool image) {
        if (image) b.V[e + d] = val;
        const unsigned o = (unsigned)(in + d) * (unsigned)sizeof(T);
        if (lo) put<CL>(b.prev + o, val);
        if (hi) put<CL>(b.next + o, val);
    };
    // a direction of one cell has two images, any other at most one
    const int dx = i == 0 ? slot_x(l, L.nx) - l.E0 : -((L.nx & 1) ? l.E0 + (L.nx >> 1) : L.nx >> 1);
    const int dy = j == 0 ? L.ny * l.PX : -L.ny * l.PX;
    copies(0, false);
    if (xb) copies(dx, true);
    if (yb) copies(dy, true);
    if (xb && yb) copies(dx + dy, true);
    if ((xb && L.nx == 1) || (yb && L.ny == 1)) {
        const int d2 = -l.E0, e2 = -L.ny * l.PX;
        const bool x2 = xb && L.nx == 1, y2 = yb && L.ny == 1;
        if (x2) copies(d2, true);
        if (x2 && yb) copies(d2 + dy, true);
        if (y2) copies(e2, true);
        if (y2 && xb) copies(dx + e2, true);
        if (x2 && y2) copies(d2 + e2, true);
    }
}

// coefficients of one point, the terms in the reference's order
template <typename T, int NPT> struct Coef {
    static constexpr int terms = Lay7<NPT>::terms;
    T c[terms];  // the centre at its own place
    T f;         // the right-hand side, where it stays in global memory
};

template <typename T, int NPT>
__device__ __forceinline__ T ld_coef(const TailLvl<T> &l, int q, long long id, int px) {
    const Lay &L = l.L;
    long long o = id;
    if (Lay7<NPT>::at_nbr(q))  // terms 0, 1, 2: the top, north, east coefficient of the z-, y-, x-neighbour
        o += q == 0 ? -(long long)(L.ny + 2) * L.P : (q == 1 ? -(long long)L.P : (px ? L.B0 : -L.B0 - 1));
    return __ldg(l.opr + (long long)Lay7<NPT>::plane(q) * L.plane + o);
}

// the point's coefficients and f: from global memory ahead of their use
// (fetch), or from shared memory where they are staged (use)
template <typename T, int NPT>
__device__ __forceinline__ void fetch(const TailLvl<T> &l, const Blk<T> &b, int i, int j, int kl, Coef<T, NPT> &c) {
    if (l.sc >= 0 && l.sf >= 0) return;
    const long long id = l.L.idx(i, j, b.k0 + kl);
    if (l.sc < 0) {
#pragma unroll
        for (int q = 0; q < Coef<T, NPT>::terms; q++) c.c[q] = ld_coef<T, NPT>(l, q, id, i & 1);
    }
    if (l.sf < 0) c.f = l.f[id];
}
template <typename T, int NPT>
__device__ __forceinline__ void use(const TailLvl<T> &l, const Blk<T> &b, int eF, Coef<T, NPT> &c) {
    if (l.sc >= 0) {
        // one point's coefficients in a row: constant offsets, and an odd
        // stride from lane to lane (no bank conflicts)
        const T *C = b.C + eF * Coef<T, NPT>::terms;
#pragma unroll
        for (int q = 0; q < Coef<T, NPT>::terms; q++) c.c[q] = C[q];
    }
    if (l.sf >= 0) c.f = b.F[eF];
}

// V element offsets of a cell's six neighbours.  Where the periodic images are
// kept up with each pass (fuse) nothing but a wall lies beyond the level: reads
// wrap instead, and no image is stored; along z only inside block 0.
struct Off6 {
    int xm, xp, ym, yp, zm, zp;
};
template <typename T, bool CL> struct Reach {
    int nx, ny, nz, PX, PP, E0, wx, wy, wz;
    __device__ __forceinline__ explicit Reach(const TailLvl<T> &l)
        : nx(l.L.nx), ny(l.L.ny), nz(l.L.nz), PX(l.PX), PP(l.PP), E0(l.E0), wx(l.fuse && l.L.xper ? l.L.nx >> 1 : 0),
          wy(l.fuse && l.L.yper ? l.L.ny * l.PX : 0), wz(!CL && l.fuse && l.L.zper ? l.L.nz * l.PP : 0) {}
    __device__ __forceinline__ Off6 at(int i, int j, int kl) const {
        Off6 o;
        o.xm = (i & 1 ? E0 - 1 : -E0);
        o.xp = o.xm + 1;
        if (i == 0) o.xm += wx;
        if (i == nx - 1) o.xp -= wx;
        o.ym = -PX + (j == 0 ? wy : 0);
        o.yp = PX - (j == ny - 1 ? wy : 0);
        o.zm = -PP;
        o.zp = PP;
        if (!CL) {
            if (kl == 0) o.zm += wz;
            if (kl == nz - 1) o.zp -= wz;
        }
        return o;
    }
};

// sum over the terms (the centre too with CENTRE) at V element e
template <typename T, int NPT, bool CENTRE>
__device__ __forceinline__ T terms_of(const T *V, int e, const Off6 &o, const Coef<T, NPT> &c) {
    using O = Ops<T, ExactOf<T>::value>;
    using S = Sten<NPT == 27 ? 27 : 7>;
    T s = T(0);
#pragma unroll
    for (int q = 0; q < Coef<T, NPT>::terms; q++) {
        if (!CENTRE && q == Lay7<NPT>::centre) continue;
        const int z = S::dz(q) < 0 ? o.zm : (S::dz(q) > 0 ? o.zp : 0), y = S::dy(q) < 0 ? o.ym : (S::dy(q) > 0 ? o.yp : 0),
                  x = S::dx(q) < 0 ? o.xm : (S::dx(q) > 0 ? o.xp : 0);
        s = O::mac(s, c.c[q], V[e + z + y + x]);
    }
    return s;
}

// One smoothing call: nsweeps alternating Gauss-Seidel sweeps (bbmg_class.f90:
// 872-885).  27-point levels go colour by colour; 7-point ones by phases of
// colours that do not read each other (k_relax_phase7).  A colour or phase
// that the opposite sweep before ended with is left out (same bits).  With an
// odd periodic size two cells of one colour meet across the wrap: there the
// images are written after the pass, as the reference's overlap copy does.
//
// A thread keeps its place (a, b, c) among the colour's points for the whole
// call: point (px + 2a, py + 2b, first plane of parity pz + 2c).
template <typename T, int NPT, bool CL>
__device__ __forceinline__ void tail_relax(const TailLvl<T> &lvl, const Blk<T> &b, int dir, int nsweeps) {
    using O = Ops<T, ExactOf<T>::value>;
    // a copy in registers, here and in the other passes: read as a kernel
    // parameter its fields are loaded again after every barrier and remote store
    // (a 15-colour smoothing call of 8^3 cells: 33.0e3 cycles, with copies 19.8e3)
    const TailLvl<T> l = lvl;
    constexpr int NPASS = NPT == 27 ? 8 : 4;
    const Lay &L = l.L;
    const int nx = L.nx, ny = L.ny, nk = b.nk, PX = l.PX, PP = l.PP, E0 = l.E0;
    const int na = (nx + 1) >> 1, nb = (ny + 1) >> 1, npt = na * nb * ((nk + 1) >> 1);
    const Reach<T, CL> reach(l);
    auto place = [&](int it, int &a, int &bb, int &c) {
        const int row = qdiv(it, l.ia);
        a = it - row * na;
        c = qdiv(row, l.ib);
        bb = row - c * nb;
    };
    int a0, b0, c0;
    place(threadIdx.x, a0, b0, c0);
#pragma unroll 1
    for (int s = 0; s < nsweeps; s++, dir = -dir) {
#pragma unroll 1
        for (int ps = 0; ps < NPASS; ps++) {
            // a backward sweep starts with the all-odd colour, which has no
            // cell on a periodic face of odd size
            if (ps == 0 && s > 0 && (l.fuse || dir < 0)) continue;
            const int pass = dir > 0 ? ps : NPASS - 1 - ps;
            // the pass's colours px + 2 py + 4 pz, four bits each (15: none)
            const unsigned cols = NPT == 27 ? 0xF0u | pass
                                            : (pass == 0 ? 0xF0u : (pass == 1 ? 0xF421u : (pass == 2 ? 0xF653u : 0xF7u)));
            if (NPT == 27 && l.fuse && npt <= kTailThreads) {
                // every thread at most one point: no loops
                const int px = pass & 1, py = (pass >> 1) & 1, ks = (b.k0 ^ (pass >> 2)) & 1;
                if (nx <= px || ny <= py || L.nz <= (pass >> 2)) continue;
                const int i = px + 2 * a0, j = py + 2 * b0, kl = ks + 2 * c0;
                const int x = px ? a0 + 1 : E0 + a0, e = (kl + 1) * PP + (j + 1) * PX + x;
                const bool on = (int)threadIdx.x < npt && i < nx && j < ny && kl < nk;
                Coef<T, NPT> c;
                if (on) fetch<T, NPT>(l, b, i, j, kl, c);
                const Off6 o = reach.at(i, j, kl);
                stage_wait<CL>();
                if (on) {
                    use<T, NPT>(l, b, (kl * ny + j) * PX + x, c);
                    const T val = O::div(O::sub(c.f, terms_of<T, NPT, false>(b.V, e, o, c)),
                                         O::add(c.c[Lay7<NPT>::centre], T(kEps)));
                    b.V[e] = val;
                    push_faces<T, CL>(l, b, kl, e, val);
                }
                stage_arrive<CL>();
                continue;
            }
            bool any = false;
            for (unsigned cs = cols; (cs & 15u) != 15u; cs >>= 4)
                any = any || (nx > (int)(cs & 1u) && ny > (int)((cs >> 1) & 1u) && L.nz > (int)((cs >> 2) & 1u));
            if (!any) continue;
            Coef<T, NPT> c;
            int a = a0, bb = b0, cc = c0;
            auto inside = [&](int it, int px, int py, int ks) {
                return it < npt && px + 2 * a < nx && py + 2 * bb < ny && ks + 2 * cc < nk;
            };
            {
                const int px = cols & 1, py = (cols >> 1) & 1, ks = (b.k0 ^ (cols >> 2)) & 1;
                if (inside(threadIdx.x, px, py, ks)) fetch<T, NPT>(l, b, px + 2 * a, py + 2 * bb, ks + 2 * cc, c);
            }
            stage_wait<CL>();
            bool fetched = true;
#pragma unroll 1
            for (unsigned cs = cols; (cs & 15u) != 15u; cs >>= 4) {
                const int px = cs & 1, py = (cs >> 1) & 1, ks = (b.k0 ^ (cs >> 2)) & 1;
                a = a0, bb = b0, cc = c0;
#pragma unroll 1
                for (int it = threadIdx.x; it < npt; it += kTailThreads) {
                    if (it != threadIdx.x) place(it, a, bb, cc);
                    if (inside(it, px, py, ks)) {
                        const int i = px + 2 * a, j = py + 2 * bb, kl = ks + 2 * cc;
                        if (!fetched) fetch<T, NPT>(l, b, i, j, kl, c);
                        const int x = px ? a + 1 : E0 + a, e = (kl + 1) * PP + (j + 1) * PX + x;
                        use<T, NPT>(l, b, (kl * ny + j) * PX + x, c);
                        const T sum = terms_of<T, NPT, false>(b.V, e, reach.at(i, j, kl), c);
                        const T val = O::div(O::sub(c.f, sum), O::add(c.c[Lay7<NPT>::centre], T(kEps)));
                        b.V[e] = val;
                        if (l.fuse) push_faces<T, CL>(l, b, kl, e, val);
                    }
                    fetched = false;
                }
            }
            if (!l.fuse) {
                stage_arrive<CL>();
                stage_wait<CL>();
                for (unsigned cs = cols; (cs & 15u) != 15u; cs >>= 4) {
                    const int px = cs & 1, py = (cs >> 1) & 1, ks = (b.k0 ^ (cs >> 2)) & 1;
                    for (int it = threadIdx.x; it < npt; it += kTailThreads) {
                        place(it, a, bb, cc);
                        if (!inside(it, px, py, ks)) continue;
                        const int i = px + 2 * a, j = py + 2 * bb, kl = ks + 2 * cc;
                        const int e = (kl + 1) * PP + (j + 1) * PX + (px ? a + 1 : E0 + a);
                        push<T, CL>(l, b, i, j, kl, e, b.V[e]);
                    }
                }
            }
            stage_arrive<CL>();
        }
    }
}

// cells of nk planes of a level in storage order: it -> (i, j, plane)
template <typename T> struct Cells {
    int n, nx, ny, nodd;
    float inx, iny;
    __device__ __forceinline__ Cells(const TailLvl<T> &l, int nk)
        : n(l.L.nx * l.L.ny * nk), nx(l.L.nx), ny(l.L.ny), nodd(l.L.nx >> 1), inx(l.inx), iny(l.iny) {}
    __device__ __forceinline__ void at(int it, int &i, int &j, int &kl) const {
        const int row = qdiv(it, inx), t = it - row * nx;
        kl = qdiv(row, iny);
        j = row - kl * ny;
        i = t < nodd ? 2 * t + 1 : 2 * (t - nodd);
    }
};

// residual of level l (bbmg_class.f90:831-844) into R
template <typename T, int NPT, bool CL>
__device__ __forceinline__ void tail_residual(const TailLvl<T> &lvl, const Blk<T> &b) {
    using O = Ops<T, ExactOf<T>::value>;
    const TailLvl<T> l = lvl;
    const Cells<T> cells(l, b.nk);
    const Reach<T, CL> reach(l);
    int it = threadIdx.x, i, j, kl;
    Coef<T, NPT> c;
    if (it < cells.n) {
        cells.at(it, i, j, kl);
        fetch<T, NPT>(l, b, i, j, kl, c);
    }
    stage_wait<CL>();
#pragma unroll 1
    while (it < cells.n) {
        const int x = slot_x(l, i), eF = (kl * l.L.ny + j) * l.PX + x;
        use<T, NPT>(l, b, eF, c);
        b.R[eF] = O::sub(c.f, terms_of<T, NPT, true>(b.V, (kl + 1) * l.PP + (j + 1) * l.PX + x, reach.at(i, j, kl), c));
        it += kTailThreads;
        if (it < cells.n) {
            cells.at(it, i, j, kl);
            fetch<T, NPT>(l, b, i, j, kl, c);
        }
    }
    stage_arrive<CL>();
}

// parity of fine index i in [-1, n]: pmod without its remainders
__device__ __forceinline__ int par_of(int per, int i, int n) { return wrap(per, i, n) & 1; }

// Restriction of R(l) into F(c) (bbmg_class.f90:805-827, weights as in
// restrict_point).  A block takes the coarse planes over its own fine ones, so
// that only the plane below its slab is read from another block, and hands each
// value to the coarse plane's owner.  Terms outside the stencil's reach and
// beyond a wall, where the residual is zero, enter as 0 * 0.
template <typename T, bool CL>
__device__ __forceinline__ void tail_restrict(const TailLvl<T> &fine, const TailLvl<T> &coarse, const Blk<T> &bl, T *Fc) {
    const TailLvl<T> l = fine, c = coarse;
    using O = Ops<T, ExactOf<T>::value>;
    const Lay &F = l.L;
    const int kc0 = (bl.k0 + 1) >> 1;  // coarse planes kc0 .. : fine planes 2 kc in [k0, k0 + nk)
    const Cells<T> cells(c, bl.nk > 0 ? ((bl.k0 + bl.nk + 1) >> 1) - kc0 : 0);
    int it = threadIdx.x;
    int i, j, kc;
    unsigned in = 0;  // terms taken
    T w[27];
    auto next = [&]() {
        cells.at(it, i, j, kc);
        kc += kc0;
        const int fi = 2 * i, fj = 2 * j, fk = 2 * kc;
        const bool x0 = par_of(F.xper, fi - 1, F.nx), x1 = par_of(F.xper, fi + 1, F.nx);
        const bool y0 = par_of(F.yper, fj - 1, F.ny), y1 = par_of(F.yper, fj + 1, F.ny);
        const bool z0 = par_of(F.zper, fk - 1, F.nz), z1 = par_of(F.zper, fk + 1, F.nz);
        in = 0;
#pragma unroll
        for (int q = 0; q < 27; q++) {
            const int ri = q % 3 - 1, rj = (q / 3) % 3 - 1, rk = q / 9 - 1;
            const bool t = (ri == 0 || (ri < 0 ? x0 : x1)) && (rj == 0 || (rj < 0 ? y0 : y1)) &&
                           (rk == 0 || (rk < 0 ? z0 : z1));
            w[q] = T(0);
            if (t) w[q] = __ldg(l.c2f + (long long)q8((1 - ri) / 2, (1 - rj) / 2, (1 - rk) / 2) * F.plane +
                                F.idx(fi + ri, fj + rj, fk + rk));
            in |= t ? 1u << q : 0u;
        }
    };
    if (it < cells.n) next();
    stage_wait<CL>();
#pragma unroll 1
    while (it < cells.n) {
        const T *Rk[3];
        int yj[3], xi[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const int kf = wrap(F.zper, 2 * kc + r - 1, F.nz), jf = wrap(F.yper, 2 * j + r - 1, F.ny),
                      xf = wrap(F.xper, 2 * i + r - 1, F.nx);
            const int ko = kf < 0 || kf >= F.nz ? 2 * kc : kf, o = owner(l, ko);
            Rk[r] = (CL ? in_block(bl.R, o) : bl.R) + plane_in(l, ko, o) * F.ny * l.PX;
            yj[r] = jf * l.PX;
            xi[r] = slot_x(l, xf);
            // a wall: no residual beyond it
            constexpr unsigned kX = 0x01249249u, kY = 0x001C0E07u, kZ = 0x000001FFu;
            if (kf < 0 || kf >= F.nz) in &= ~(kZ << (9 * r));
            if (jf < 0 || jf >= F.ny) in &= ~(kY << (3 * r));
            if (xf < 0 || xf >= F.nx) in &= ~(kX << r);
        }
        T rv[27];
#pragma unroll
        for (int q = 0; q < 27; q++) {
            rv[q] = T(0);
            if (in >> q & 1u) rv[q] = Rk[q / 9][yj[(q / 3) % 3] + xi[q % 3]];
        }
        T s = T(0);
#pragma unroll
        for (int q = 0; q < 27; q++) s = O::mac(s, w[q], rv[q]);
        const int o = owner(c, kc);
        (CL ? in_block(Fc, o) : Fc)[(plane_in(c, kc, o) * c.L.ny + j) * c.PX + slot_x(c, i)] = s;
        it += kTailThreads;
        if (it < cells.n) next();
    }
    stage_arrive<CL>();
}

// prolongation and correction of V(l) from V(c) (bbmg_class.f90:779-801, 770);
// beyond a wall the coarse correction is zero, and terms of the other parity
// classes enter as 0 * 0
template <typename T, bool CL>
__device__ __forceinline__ void tail_prolong(const TailLvl<T> &fine, const TailLvl<T> &coarse, const Blk<T> &bl, T *Vc) {
    const TailLvl<T> l = fine, c = coarse;
    using O = Ops<T, ExactOf<T>::value>;
    const Lay &F = l.L, &C = c.L;
    const Cells<T> cells(l, bl.nk);
    int it = threadIdx.x;
    int i, j, kl;
    T w[8];
    auto next = [&]() {
        cells.at(it, i, j, kl);
        const long long id = F.idx(i, j, bl.k0 + kl);
        const int k = bl.k0 + kl;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            w[q] = T(0);
            if ((q & 1) <= (i & 1) && ((q >> 1) & 1) <= (j & 1) && (q >> 2) <= (k & 1))
                w[q] = __ldg(l.c2f + (long long)q * F.plane + id);
        }
    };
    if (it < cells.n) next();
    stage_wait<CL>();
#pragma unroll 1
    while (it < cells.n) {
        const int i1 = i, j1 = j, kl1 = kl, k = bl.k0 + kl1, ci = i1 >> 1, cj = j1 >> 1, ck = k >> 1;
        T w1[8], cv[8];
#pragma unroll
        for (int q = 0; q < 8; q++) w1[q] = w[q];
        it += kTailThreads;
        if (it < cells.n) next();  // the next cell's weights are on their way
#pragma unroll
        for (int pk = 0; pk <= 1; pk++) {
            const int kc = wrap(C.zper, ck + pk, C.nz);
            const bool inz = pk <= (k & 1) && kc < C.nz;
            const int ko = inz ? kc : ck, o = owner(c, ko);
            const T *V = (CL ? in_block(Vc, o) : Vc) + (plane_in(c, ko, o) + 1) * c.PP + c.PX;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                int xi = ci + (q & 1), yj = cj + (q >> 1);
                if (c.fuse && C.xper && xi == C.nx) xi = 0;  // no images there
                if (c.fuse && C.yper && yj == C.ny) yj = 0;
                cv[4 * pk + q] = T(0);
                if (inz && (q >> 1) <= (j1 & 1) && (q & 1) <= (i1 & 1)) cv[4 * pk + q] = V[yj * c.PX + slot_x(c, xi)];
            }
        }
        T e = T(0);
#pragma unroll
        for (int q = 0; q < 8; q++) e = O::mac(e, w1[q], cv[q]);
        const int ev = (kl1 + 1) * l.PP + (j1 + 1) * l.PX + slot_x(l, i1);
        const T val = O::add(bl.V[ev], e);
        bl.V[ev] = val;
        if (l.fuse) push_faces<T, CL>(l, bl, kl1, ev, val);
        else push<T, CL>(l, bl, i1, j1, kl1, ev, val);
    }
    stage_arrive<CL>();
}

// coarsest level, inside block 0 (bbmg_class.f90:741-748)
template <typename T>
__device__ __forceinline__ void tail_coarsest(const TailArgs<T> &A, const TailLvl<T> &l, const Blk<T> &b, double *sd) {
    if (!A.direct) {
        tail_relax<T, 27, false>(l, b, 1, A.pre + A.post);
        return;
    }
    const Lay &L = l.L;
    const int np = L.nx * L.ny * L.nz;
    __syncthreads();
    for (int ind = threadIdx.x; ind < np; ind += kTailThreads) {
        const int p = A.perm[ind], row = qdiv(p, l.inx), i = p - row * L.nx, k = qdiv(row, l.iny), j = row - k * L.ny;
        sd[ind] = (double)b.F[(k * L.ny + j) * l.PX + slot_x(l, i)];
    }
    __syncthreads();
    if (threadIdx.x < 32) lu_solve(sd + np, A.LU, A.mat_in_smem, A.pinned, np, threadIdx.x, sd);
    __syncthreads();
    for (int ind = threadIdx.x; ind < np; ind += kTailThreads) {
        const int row = qdiv(ind, l.inx), i = ind - row * L.nx, k = qdiv(row, l.iny), j = row - k * L.ny;
        const T val = (T)sd[ind];
        const int e = (k + 1) * l.PP + (j + 1) * l.PX + slot_x(l, i);
        b.V[e] = val;
        if (!l.fuse) push<T, false>(l, b, i, j, k, e, val);
    }
}

template <typename T, int NPT, bool CL>
__device__ __forceinline__ void tail_down(const TailArgs<T> &A, int n, int rank, T *sm) {
    const TailLvl<T> &l = A.lv[n], &c = A.lv[n + 1];
    const Blk<T> b = part<T, CL>(l, rank, sm);
    tail_relax<T, NPT, CL>(l, b, 1, A.pre);
    tail_residual<T, NPT, CL>(l, b);
    tail_restrict<T, CL>(l, c, b, sm + c.sf);
}

template <typename T, int NPT, bool CL>
__device__ __forceinline__ void tail_up(const TailArgs<T> &A, int n, int rank, T *sm) {
    const TailLvl<T> &l = A.lv[n], &c = A.lv[n + 1];
    const Blk<T> b = part<T, CL>(l, rank, sm);
    tail_prolong<T, CL>(l, c, b, sm + c.sv);
    tail_relax<T, NPT, CL>(l, b, (A.pre & 1) ? -1 : 1, A.post);
}

// the block's coefficients of a level into shared memory, where they have a place
template <typename T, int NPT>
__device__ __forceinline__ void stage_coef(const TailLvl<T> &l, int rank, T *sm) {
    if (l.sc < 0) return;
    const Blk<T> b = part<T, true>(l, rank, sm);
    const Cells<T> cells(l, b.nk);
#pragma unroll 1
    for (int it = threadIdx.x; it < cells.n; it += kTailThreads) {
        int i, j, kl;
        cells.at(it, i, j, kl);
        const long long id = l.L.idx(i, j, b.k0 + kl);
        T *C = b.C + ((kl * l.L.ny + j) * l.PX + slot_x(l, i)) * Coef<T, NPT>::terms;
#pragma unroll
        for (int q = 0; q < Coef<T, NPT>::terms; q++) C[q] = ld_coef<T, NPT>(l, q, id, i & 1);
    }
}

template <typename T, int NPT1>
__global__ void __launch_bounds__(kTailThreads) k_vtail(const __grid_constant__ TailArgs<T> A) {
    extern __shared__ __align__(16) unsigned char raw[];
    double *sd = reinterpret_cast<double *>(raw);
    T *sm = reinterpret_cast<T *>(raw + A.solve_bytes);
    pdl_launch();
    const int rank = blockIdx.x, tid = threadIdx.x;
    for (int e = tid; e < A.zeroed; e += kTailThreads) sm[e] = T(0);
    // what only the setup writes comes in before the wait for the predecessor
    if (rank == 0 && A.mat_in_smem) lu_stage(A.LU, A.np, sd + A.np);
    for (int n = 0; n < A.n; n++) {
        if (NPT1 != 27 && n == 0) stage_coef<T, NPT1>(A.lv[n], rank, sm);
        else stage_coef<T, 27>(A.lv[n], rank, sm);
    }
    pdl_wait();
    __syncthreads();
    {  // the finest fused level's v, overlap included (its f stays in global memory)
        const TailLvl<T> &l = A.lv[0];
        const Lay &L = l.L;
        const Blk<T> b = part<T, true>(l, rank, sm);
        if (b.nk > 0) {
            const int w = L.nx + 2, h = L.ny + 2, total = w * h * (b.nk + 2);
            const float iw = 1.f / (float)w, ih = 1.f / (float)h;
#pragma unroll 4
            for (int it = tid; it < total; it += kTailThreads) {
                const int row = qdiv(it, iw), i = it - row * w - 1, kl = qdiv(row, ih), j = row - kl * h - 1;
                b.V[kl * l.PP + (j + 1) * l.PX + slot_x(l, i)] = l.v[L.idx(i, j, b.k0 + kl - 1)];
            }
        }
    }
    cl_arrive();
    const int ns = A.split;  // levels [0, ns) over the cluster
#pragma unroll 1
    for (int n = 0; n < ns; n++) {
        if (NPT1 != 27 && n == 0) tail_down<T, NPT1, true>(A, n, rank, sm);
        else tail_down<T, 27, true>(A, n, rank, sm);
    }
    cl_wait();
    if (rank == 0) {
#pragma unroll 1
        for (int n = ns; n + 1 < A.n; n++) {
            if (NPT1 != 27 && n == 0) tail_down<T, NPT1, false>(A, n, 0, sm);
            else tail_down<T, 27, false>(A, n, 0, sm);
        }
        tail_coarsest<T>(A, A.lv[A.n - 1], part<T, false>(A.lv[A.n - 1], 0, sm), sd);
#pragma unroll 1
        for (int n = A.n - 2; n >= ns; n--) {
            if (NPT1 != 27 && n == 0) tail_up<T, NPT1, false>(A, n, 0, sm);
            else tail_up<T, 27, false>(A, n, 0, sm);
        }
    }
    cl_arrive();
#pragma unroll 1
    for (int n = ns - 1; n >= 0; n--) {
        if (NPT1 != 27 && n == 0) tail_up<T, NPT1, true>(A, n, rank, sm);
        else tail_up<T, 27, true>(A, n, rank, sm);
    }
    cl_wait();
    {  // v and its overlap back
        const TailLvl<T> &l = A.lv[0];
        const Lay &L = l.L;
        const Blk<T> b = part<T, true>(l, rank, sm);
        const int w = L.nx + 2, h = L.ny + 2, total = w * h * b.nk;
        const float iw_ = 1.f / (float)w, ih = 1.f / (float)h;
        for (int it = tid; it < total; it += kTailThreads) {
            const int row = qdiv(it, iw_), i = it - row * w - 1, kl = qdiv(row, ih), j = row - kl * h - 1;
            const int k = b.k0 + kl;
            const int iw = l.fuse ? wrap(L.xper, i, L.nx) : i, jw = l.fuse ? wrap(L.yper, j, L.ny) : j;
            const T val = b.V[(kl + 1) * l.PP + (jw + 1) * l.PX + slot_x(l, iw)];
            l.v[L.idx(i, j, k)] = val;
            if (L.zper && k == 0) l.v[L.idx(i, j, L.nz)] = val;
            if (L.zper && k == L.nz - 1) l.v[L.idx(i, j, -1)] = val;
        }
    }
}

cudaLaunchConfig_t tail_cfg(int cl, size_t smem, cudaStream_t s, cudaLaunchAttribute *at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

template <typename T, int NPT1> bool tail_kernel_fits(int blocks, size_t smem) {
    auto kern = k_vtail<T, NPT1>;
    int nc = 0;
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = tail_cfg(blocks, smem, nullptr, at);
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmemMax) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc >= 1;
    if (!ok) cudaGetLastError();
    return ok;
}

}  // namespace

// ---------------------------------------------------------------------------
template <typename T>
bool tail_plan(const Lay *lay, const bool *fuse, int n, int npt1, int np, bool direct, int blocks, TailArgs<T> *A,
               size_t *smem) {
    if (n < 2 || n > kTailMax) return false;
    A->n = n;
    A->np = np;
    A->split = 0;
    A->direct = direct;
    const size_t mat = sizeof(double) * ((size_t)np + (size_t)lu_ld(np) * lu_ld(np));
    A->mat_in_smem = direct && mat <= kTailMatMax ? 1 : 0;
    A->solve_bytes = (int)(((A->mat_in_smem ? mat : sizeof(double) * (size_t)np) + 15) / 16 * 16);
    long long e = 0, rmax = 0;
    bool single = false;
    for (int m = 0; m < n; m++) {
        TailLvl<T> &t = A->lv[m];
        const Lay &L = lay[m];
        t.L = L;
        t.fuse = fuse[m];
        single = single || (long long)L.nx * L.ny * L.nz <= kTailSingle || m == n - 1;
        t.single = single;
        if (!single) A->split = m + 1;
        t.H = single ? L.nz : (L.nz + blocks - 1) / blocks;
        if (!single && (long long)t.H * L.nx * L.ny > kTailBlockCells) return false;
        t.E0 = (L.nx + 1) / 2 + 1;
        t.PX = L.nx + 2;
        t.PP = t.PX * (L.ny + 2);
        t.iH = 1.f / (float)t.H;
        t.inx = 1.f / (float)L.nx;
        t.iny = 1.f / (float)L.ny;
        t.ia = 1.f / (float)((L.nx + 1) / 2);
        t.ib = 1.f / (float)((L.ny + 1) / 2);
        t.sv = (int)e;
        e += (long long)t.PP * (t.H + 2);
        t.ncf = t.PX * L.ny * t.H;
        t.sf = m ? (int)e : -1;  // the first level's f is read where it is
        if (m) e += t.ncf;
        rmax = std::max(rmax, (long long)t.ncf);
        t.sc = -1;
        if ((e + rmax) * (long long)sizeof(T) > (long long)kTailSmemMax) return false;
    }
    // one residual at a time: every level's R is the same place
    for (int m = 0; m < n; m++) A->lv[m].sr = (int)e;
    e += rmax;
    A->zeroed = (int)e;
    if (A->solve_bytes + e * (long long)sizeof(T) > (long long)kTailSmemMax) return false;
    // coefficients, from the coarsest smoothed level up while they fit
    for (int m = direct ? n - 2 : n - 1; m >= 0; m--) {
        TailLvl<T> &t = A->lv[m];
        const long long c = (long long)t.ncf * (m == 0 && npt1 < 27 ? 7 : 27);
        if (A->solve_bytes + (e + c) * (long long)sizeof(T) > (long long)kTailSmemMax) break;
        t.sc = (int)e;
        e += c;
    }
    *smem = A->solve_bytes + (size_t)e * sizeof(T);
    return true;
}

// asked once per device, type and cluster size: the queries take milliseconds
template <typename T>
bool tail_fits(int blocks) {
    constexpr int kDev = 64;
    static std::mutex mu;
    static signed char known[kDev][2] = {};  // 1 it can, -1 it cannot
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lock(mu);
    signed char once = 0, &k = dev < kDev ? known[dev][blocks == kTailClusterMax] : once;
    if (!k)
        k = tail_kernel_fits<T, 27>(blocks, kTailSmemMax) && tail_kernel_fits<T, 7>(blocks, kTailSmemMax) &&
                    tail_kernel_fits<T, 4>(blocks, kTailSmemMax)
                ? 1
                : -1;
    return k > 0;
}

template <typename T>
cudaError_t launch_vtail(const TailArgs<T> &A, int npt1, int blocks, size_t smem, cudaStream_t s) {
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = tail_cfg(blocks, smem, s, at);
    if (npt1 == 4) BB_CHECK_LAUNCH((cudaLaunchKernelEx(&cfg, k_vtail<T, 4>, A)));
    else if (npt1 == 7) BB_CHECK_LAUNCH((cudaLaunchKernelEx(&cfg, k_vtail<T, 7>, A)));
    else BB_CHECK_LAUNCH((cudaLaunchKernelEx(&cfg, k_vtail<T, 27>, A)));
    return cudaSuccess;
}

template <typename T>
cudaError_t launch_coarse_solve(const Lay &L, const double *LU, const int *perm, const int *pinned, const T *f, T *v,
                                cudaStream_t s) {
    int np = L.nx * L.ny * L.nz;
    size_t mat = (size_t)lu_ld(np) * lu_ld(np) * sizeof(double), vec = (size_t)np * sizeof(double);
    int in_smem = (mat + vec) <= kCoarseSmem;
    size_t shm = vec + (in_smem ? mat : 0);
    BB_CHECK_LAUNCH((launch_k(k_coarse_solve<T>, dim3(1), dim3(256), shm, s, L, LU, perm, pinned, f, v, in_smem)));
    return cudaSuccess;
}

cudaError_t coarse_solve_prepare() {
    cudaError_t e = cudaFuncSetAttribute(k_coarse_solve<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kCoarseSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_coarse_solve<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseSmem);
}

#define BB_TAIL_INST(T)                                                                                           \
    template bool tail_plan<T>(const Lay *, const bool *, int, int, int, bool, int, TailArgs<T> *, size_t *);     \
    template bool tail_fits<T>(int);                                                                      \
    template cudaError_t launch_vtail<T>(const TailArgs<T> &, int, int, size_t, cudaStream_t);                    \
    template cudaError_t launch_coarse_solve<T>(const Lay &, const double *, const int *, const int *, const T *, \
                                                T *, cudaStream_t);
BB_TAIL_INST(double)
BB_TAIL_INST(float)

}  // namespace bbmg
