// setup.cuh -- launchers of the setup and solve kernels.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace bbmg {

// setup.cu (FP64)
// `wmask`/`mask`: 27-bit sets of operator planes (q27 slots); the scatter
// writes only the planes in wmask (the others hold zeros already), the
// prolongation and A*P skip planes outside mask (known to be all zero);
// the scatter's stc is the caller's stencil in host memory
cudaError_t setup_scatter(const Lay &L, const double *src, int nst, int g, const int *stc, double *opr, unsigned wmask,
                          cudaStream_t s);
cudaError_t wrap_planes(const Lay &L, double *a, int nplanes, cudaStream_t s);
cudaError_t wrap_planes_mask(const Lay &L, double *a, unsigned mask, cudaStream_t s);
cudaError_t wrap_planes(const Lay &L, float *a, int nplanes, cudaStream_t s);
// c2f32 / oprC32, if given, receive the FP32 copies of the prolongation
// weights and of the coarse operator (the mixed-precision V-cycle's arrays)
cudaError_t setup_prolongation(const Lay &L, const double *opr, double *c2f, unsigned mask, cudaStream_t s,
                               float *c2f32 = nullptr);
cudaError_t setup_restriction(const Lay &F, const Lay &C, const double *c2f, double *f2c, cudaStream_t s);
cudaError_t setup_operator(const Lay &F, const Lay &C, const double *oprF, const double *c2f, const double *f2c,
                           double *oprc2f, double *oprC, unsigned mask, cudaStream_t s, float *oprC32 = nullptr);
// the overlap of f2c and of A P (oprc2f) as the reference holds it (zero in
// non-periodic directions, the periodic image otherwise); the setup leaves it
// unfilled where nothing reads it, so it is filled before a read-out
cudaError_t fill_overlap_f2c(const Lay &C, double *f2c, cudaStream_t s);
cudaError_t fill_overlap_oprc2f(const Lay &F, double *oprc2f, cudaStream_t s);
// plane q of oprS (and of oprS32, if given) = plane slots[q] of the 27-plane opr, npt <= 7
cudaError_t setup_solve_planes(const Lay &L, const double *opr, int npt, const int *slots, double *oprS,
                               float *oprS32, cudaStream_t s);
cudaError_t check_symmetric7(const Lay &L, const double *opr, int *flag, cudaStream_t s);
cudaError_t setup_direct(const Lay &L, const double *opr, double *OP, double *LU, int *piv, int *perm, int *pinned,
                         int *info, cudaStream_t s);

// solve.cu
struct Off27 {
    int o[27];
};
template <typename T>
cudaError_t launch_relax(const Lay &L, const NbrOff &nb, int npt, bool fuse, const T *opr, T *v, const T *f, int dir,
                         cudaStream_t s, bool skip_first = false);
// `nsweeps` alternating sweeps starting with `first_dir` (the relax loops of
// cycle, bbmg_class.f90:754-758 and 772-775)
template <typename T>
cudaError_t launch_relax_sweeps(const Lay &L, const NbrOff &nb, int npt, bool fuse, const T *opr, T *v, const T *f,
                                int first_dir, int nsweeps, cudaStream_t s);
template <typename T>
cudaError_t launch_residual(const Lay &L, const NbrOff &nb, int npt, const T *opr, const T *v, const T *f, T *r,
                            cudaStream_t s);
template <typename T>
cudaError_t launch_restrict(const Lay &F, const Lay &C, const T *c2f, const T *rF, T *fC, T *vC, cudaStream_t s);
template <typename T>
cudaError_t launch_prolong(const Lay &F, const Lay &C, const T *c2f, const T *vC, T *vF, cudaStream_t s);
// vtail.cu: the coarsest solve; perm is the row permutation of the stored LU
constexpr size_t kCoarseSmem = 202 * 1024;  // factors of up to 160 unknowns stay on chip
cudaError_t coarse_solve_prepare();  // per device, before the first coarse solve
template <typename T>
cudaError_t launch_coarse_solve(const Lay &L, const double *LU, const int *perm, const int *pinned, const T *f, T *v,
                                cudaStream_t s);

// vtail.cu: levels n0..nlvl of the V-cycle in one launch of one thread-block
// cluster (ncycle = 1; the first level may hold a 4- or 7-plane operator)
template <typename T>
struct TailLvl {
    Lay L;
    const T *opr;          // coefficient planes
    T *v;                  // global v and f: the first level's are read and written
    const T *f;
    const T *c2f;          // prolongation weights of this level (to the next coarser one)
    int fuse;              // periodic images may be written inside a colour
    int single;            // inside block 0
    int H;                 // k-planes per block
    int PX, E0, PP;        // shared memory: row pitch, offset of the even x, plane pitch
    int sv, sf, sr, sc;    // first elements of V, F, R and the coefficients (-1: in global memory)
    int ncf;               // elements of F, of R and of one coefficient
    float iH, inx, iny, ia, ib;  // reciprocals of H, nx, ny and of a colour's points per row and rows
};
constexpr int kTailMax = 8;            // levels in one launch (kernel parameters stay under 4 KB)
constexpr int kTailThreads = 256;
constexpr int kTailClusterMax = 16;    // blocks of the cluster (non-portable size; 8 if refused)
// most cells of the first fused level: a 64^3 FP64 solve takes 4.19 ms with none
// fused, 3.04 from 16^3 and 2.75 ms from 32^3.  64x32x32 still fits the slabs of 16
// blocks, in FP32 (208 KB a block) though not in FP64 beside the staged factors of
// 128 unknowns; fused there a 64x32x32 cycle takes 0.184 instead of 0.197 ms, but a
// 256x128x128 mixed solve 12.86 instead of 12.39
constexpr long long kTailCells = 36864;
constexpr long long kTailBlockCells = 4096;  // most cells of a block's slab
// levels this small run inside block 0: a pass over 8^3 cells takes 0.65e3 cycles
// there, a barrier of the whole cluster alone 0.39e3
constexpr long long kTailSingle = 1024;
constexpr size_t kTailMatMax = 136 * 1024;   // LU factors held in shared memory
constexpr size_t kTailSmemMax = 226 * 1024;
template <typename T>
struct TailArgs {
    TailLvl<T> lv[kTailMax];
    int n;                 // levels in lv; lv[n-1] is the coarsest
    int split;             // levels below it are dealt out over the cluster
    int pre, post, direct, np, mat_in_smem;
    int solve_bytes, zeroed;  // shared memory: bytes of the coarsest solve, then values that start at zero
    const double *LU;
    const int *perm, *pinned;
};
// sizes and shared-memory layout of the n levels lay[0..n) for a cluster of
// `blocks`, the first with npt1 planes; false if they do not fit.  tail_fits:
// the device can run it.
template <typename T>
bool tail_plan(const Lay *lay, const bool *fuse, int n, int npt1, int np, bool direct, int blocks, TailArgs<T> *A,
               size_t *smem);
template <typename T>
bool tail_fits(int blocks);
template <typename T>
cudaError_t launch_vtail(const TailArgs<T> &A, int npt1, int blocks, size_t smem, cudaStream_t s);
// reductions (deterministic two-pass) into a device double
constexpr int kRedBlocks = 1184;  // 8 blocks of 256 threads per SM on 148 SMs
template <typename T>
cudaError_t launch_maxabs(const Lay &L, const T *x, double *part, double *out, cudaStream_t s);
template <typename T>
cudaError_t launch_dot(const Lay &L, const T *a, const T *b, double *part, double *out, cudaStream_t s);

// PCG scalars (device resident)
struct CgScal {
    double rho1, rho2, pap, alpha, beta;
    int iter, pad;
};
template <typename TZ>
cudaError_t launch_cg_rho(const Lay &L, const TZ *zz, const double *res, double *part, CgScal *sc, cudaStream_t s);
template <typename TZ>
cudaError_t launch_fcg_rho(const Lay &L, const TZ *zz, const double *res, const double *Ap, double *part, CgScal *sc,
                           cudaStream_t s);
template <typename TZ>
cudaError_t launch_cg_pap_fused(const Lay &L, const NbrOff &nb, int npt, const double *opr, const TZ *zz,
                                const double *pp_old, double *pp_new, double *Ap, double *part, CgScal *sc,
                                cudaStream_t s);
template <typename TV>
cudaError_t launch_cg_xr_fused(const Lay &L, double *sol, const double *pp, double *res, const double *Ap,
                               const CgScal *sc, float *f32, TV *vzero, double *part, double *out, cudaStream_t s);
cudaError_t launch_defect_fused(const Lay &L, const NbrOff &nb, int npt, const double *opr, const double *x_old,
                                const float *e, const double *b, double *x_new, float *f32, double *part,
                                double *out, cudaStream_t s);
cudaError_t launch_round_f32(const Lay &L, const double *r, float *f, cudaStream_t s);
// flexible CG: zz = z1 + e (z1 may be null), rho = zz.res, beta = -zz.Ap_old / pap_old
cudaError_t launch_fcg_z(const Lay &L, const double *z1, const float *e, const double *res, const double *Ap,
                         double *zz, double *part, CgScal *sc, cudaStream_t s);

// caller I/O: Fortran arrays with g overlap layers <-> level interior
template <typename T>
cudaError_t launch_from_caller(const Lay &L, const double *src, int g, T *dst, cudaStream_t s);
cudaError_t launch_to_caller(const Lay &L, const double *src, int g, double *dst, cudaStream_t s);
// FP64 level arrays <-> FP32 copies (planes)
cudaError_t launch_to_f32(const double *src, float *dst, long long n, cudaStream_t s);

}  // namespace bbmg
