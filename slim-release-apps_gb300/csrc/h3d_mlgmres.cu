// FGMRES preconditioned by the ML_GMRES multigrid V-cycle: the 3D applications' default
// Helmholtz solver (linearsolve.m:139-141 with SOLVE_FGMRES, discrete_helmholtz.m:349-350 with
// PREC_MLGMRES).
//
//   FGMRES        FGMRES.m:33-129: restarted flexible GMRES; classical Gram-Schmidt, the
//                 (k+1) x k least-squares problem solved after every step, the quasi-residual
//                 norm(beta e1 - H y) / normr0 as the inner stopping test, the true residual
//                 b - A x after every cycle as the outer one
//   ML_GMRES      ML_GMRES.m:36-72: smoother = FGMRES, 3 cycles of 5 steps to 1e-6, no
//                 preconditioner; coarse solver = FGMRES, 3 x 5 to 0.5 (opts.k overrides)
//   V-cycle       opMultigrid.m with recursive_v_cycle, GMG_V.m: smooth from zero, residual,
//                 restrict, coarse solve (preconditioned by the next level's V-cycle; on the
//                 last level by an unpreconditioned coarse-solver FGMRES), prolongate and add,
//                 smooth again from there
//
// GB300 layout of the work.  Every vector of every level stays on the device.  Each FGMRES
// instance (the outer solve, the smoother and coarse solver of every level, the last level's
// inner solver) owns its Krylov basis, a partial-sum buffer and a small state block
// (FgState) in device memory.  An Arnoldi step is three launches: the matvec, the k inner
// products V^H w (per-CTA partial sums), and the orthogonalisation w -= V h fused with the final
// sum of those partials and with ||w||^2 partials.  The step's Givens update (the previous rotations
// on the new Hessenberg column, the next rotation, the rotated right-hand side and the
// quasi-residual: a dependent chain of FP64 instructions, about 3 us) runs beside the next step's inner
// products, in a CTA of its own; after a cycle's last step, and in the preconditioned instances, whose next
// step the host decides on, in the last CTA of the orthogonalisation, at the end of a cycle followed by the
// back substitution.  The basis is kept unnormalised with a scale per
// vector in the unpreconditioned instances; the preconditioned ones (whose basis vectors feed
// the V-cycle) add a fourth launch, the scaling V(:,k+1) = w / ||w||.  The Givens update gives
// the least-squares residual norm of FGMRES.m:111-113 without a host round trip; the solution y
// is back-substituted once per cycle.  Every kernel after the matvec reads
// a flag of the state block (the step runs / the cycle runs) and returns at once when it is
// clear, the matvecs of the unpreconditioned instances too, so the host enqueues unpreconditioned cycles without waiting: it synchronises once per
// cycle of a coarse solve there, after every fourth cycle of a smoother (every one with a loose tolerance), and before each step of
// a preconditioned instance (to decide whether the expensive preconditioner runs at all).  Sums are deterministic: fixed
// per-thread and per-warp sums in the field's precision, then per-CTA partials and their
// totals in FP64 in a fixed order.
//
// The mixed precision of the Python front end carries over: the outer FGMRES in complex128,
// the V-cycle (all levels, smoothers and coarse solves) in complex64 with FP64 inner products.
#include <cfloat>
#include <chrono>
#include <cmath>
#include <functional>

#include <cooperative_groups.h>

#include "h3d_kernels.cuh"
#include "h3d_vec.cuh"

namespace h3d {
namespace cg = cooperative_groups;
namespace {

constexpr int kMaxM = 16;       // steps per cycle the state block holds
constexpr int kMaxLevels = 8;
constexpr int kThr = 256;
constexpr int kCluster = 8;     // CTAs of a cluster in the inner products of the larger levels

struct FgHead {                 // the part of the state the host reads
    int live;                   // the cycle loop goes on (FGMRES.m:88 and :125)
    int go;                     // the next Arnoldi step runs (FGMRES.m:97)
    int k;                      // steps done in the current cycle
    int it;                     // it_counter (FGMRES.m:74)
    int nhst;                   // quasi-residuals recorded (the leading 1 not counted)
    int conv;                   // stopped on the tolerance (quasi- or true residual)
    double normr0, beta, hst, rn;
};

struct FgState {
    FgHead hd;
    double hn;                  // ||w|| of the current step = H(k+1,k)
    double rhn, rbeta;          // 1 / hn and 1 / beta (0 when the norm is 0)
    double rnormr0;             // 1 / normr0
    double sv[kMaxM];           // basis vector j = sv[j] x stored vector j (1 when stored normalised)
    int ticket;                 // CTAs of the current orthogonalisation launch that have finished
    int pend;                   // steps orthogonalised whose Givens update is outstanding: j + 1, or 0
    double gres;                // |g(k+1)|: the current quasi-residual norm (before / normr0)
    double cs[kMaxM];           // Givens rotations: cosines (real) ...
    cplx<double> sn[kMaxM];     // ... and sines
    cplx<double> g[kMaxM + 1];  // rotated beta e1
    cplx<double> R[kMaxM * kMaxM];  // rotated Hessenberg, column j at R + j * kMaxM
    cplx<double> h[kMaxM];      // V^H w of the current step
    cplx<double> y[kMaxM];      // least-squares solution of the current cycle
};

__device__ __forceinline__ bool closed(const int *gate) { return gate && *gate == 0; }

// First thing in every kernel here: let the next launch set up early, and wait for the launch before
// (both do nothing in an ordinary launch).
__device__ __forceinline__ void fg_begin()
{
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Sum over the block's warps of one FP64 value per warp and index: lane w of eight holds warp w's.
__device__ __forceinline__ double warps_sum8(double v)
{
    for (int o = kThr / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide sum of one per-thread value kept in precision T (valid in every thread of warp 0): warp
// shuffles in T, the per-warp results added in FP64 in a fixed order.  GB300 executes FP64 at a small
// fraction of its FP32 rate (a warp's FP64 instruction holds its scheduler's pipe for 64 cycles, however
// few of its lanes are active), so the complex64 cycle's vector kernels form products and per-thread sums
// in FP32 (as a complex64 BLAS would), leave FP64 to the few values per CTA, and add those as a tree
// across lanes; the complex128 instances stay FP64 throughout.
template <typename T>
__device__ __forceinline__ double block_sum(T a)
{
    __shared__ double sa[kThr / 32];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sa[threadIdx.x >> 5] = (double)a;
    __syncthreads();
    return threadIdx.x < 32 ? warps_sum8(sa[threadIdx.x & (kThr / 32 - 1)]) : 0.0;
}

// ---- element kernels ----------------------------------------------------------------------

// r = b (x = 0 when given); per-CTA partials of ||r||^2.
template <typename T>
__global__ void __launch_bounds__(kThr) fg_copy_kernel(const cplx<T> *__restrict__ b, cplx<T> *__restrict__ r,
                                                       cplx<T> *__restrict__ x, long long n, double *part)
{
    fg_begin();
    T s = 0;
    for (long long e = blockIdx.x * (long long)kThr + threadIdx.x; e < n; e += (long long)gridDim.x * kThr) {
        const cplx<T> v = b[e];
        r[e] = v;
        if (x) x[e] = mk<T>(0, 0);
        s = fma(v.re, v.re, fma(v.im, v.im, s));
    }
    const double t = block_sum<T>(s);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// dst = src * (*rcp): V(:,k) = w / ||w|| with the reciprocal formed once per step.
template <typename T>
__global__ void __launch_bounds__(kThr) fg_scale_kernel(const cplx<T> *__restrict__ src, cplx<T> *__restrict__ dst,
                                                        long long n, const double *rcp, const int *gate)
{
    fg_begin();
    if (closed(gate)) return;
    const T d = (T)*rcp;
    for (long long e = blockIdx.x * (long long)kThr + threadIdx.x; e < n; e += (long long)gridDim.x * kThr) {
        const cplx<T> v = src[e];
        dst[e] = mk<T>(v.re * d, v.im * d);
    }
}

// Element loops take kU elements per thread per pass (stride apart, each coalesced across the
// warp) so that kU x (vectors) independent loads are in flight before the arithmetic.
constexpr int kU = 4;

// Vectors of a kernel that goes over the basis: MV of them where the number is known at compile time
// (kExact of them and fewer: one instance each, whose loads the compiler can all issue first), at most MV
// otherwise.
constexpr int kExact = 5;
template <int MV>
__device__ __forceinline__ int vectors(int nv)
{
    return MV <= kExact ? MV : nv;
}

__device__ void givens_step(FgState *st, const double *part, int nparts, int j, int m, double tol, double *hist,
                            int lazy);

// Partials of h_j = V_j^H w, j < nv: part[j * groups + group], a group being the CTAs of a cluster (or one
// CTA, in a launch without clusters): every CTA of the orthogonalisation adds all the partials up in FP64,
// which at 509 partials per vector took 5 (nv = 2 or 3) to 10 us (nv = 5) of its 12 and 20, so the eight
// CTAs of a cluster add theirs first, over distributed shared memory.
// Stored vector 0 is u0, vector j >= 1 is V + j n (the unpreconditioned instances keep vector 0
// in their residual buffer).
// The last cluster's first CTA runs the Givens update of the step before instead, when it is
// outstanding: the inner products do not need it, the orthogonalisation after them does.  While it is
// outstanding the gate may close under this launch, so the gate is read only when it is not (every CTA
// of a cluster has to take the same way).
template <typename T, int MV>
__global__ void __launch_bounds__(kThr) fg_dots_kernel(const cplx<T> *__restrict__ u0, const cplx<T> *__restrict__ V,
                                                       int nvec, const cplx<T> *__restrict__ w, long long n,
                                                       double2 *__restrict__ part, const int *gate, FgState *st,
                                                       const double *npart, int nparts, int m, double tol, double *hist)
{
    fg_begin();
    const int nv = vectors<MV>(nvec);
    const cg::cluster_group cl = cg::this_cluster();
    const int gs = (int)cl.num_blocks(), nd = (int)gridDim.x - gs, ng = nd / gs;
    const int pend = st->pend;
    if ((int)blockIdx.x >= nd) {
        if (pend && (int)blockIdx.x == nd) givens_step(st, npart, nparts, pend - 1, m, tol, hist, 1);
        return;
    }
    if (pend == 0 && closed(gate)) return;
    if (gs > 1) cl.barrier_arrive();  // started: its shared memory may be written
    cplx<T> acc[MV];
#pragma unroll
    for (int j = 0; j < MV; ++j) acc[j] = mk<T>(0, 0);
    const long long stride = (long long)nd * kThr;
    long long e = blockIdx.x * (long long)kThr + threadIdx.x;
    for (; e + (kU - 1) * stride < n; e += kU * stride) {
        cplx<T> wv[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) wv[u] = w[e + u * stride];
#pragma unroll
        for (int j = 0; j < MV; ++j) {
            if (j < nv) {
                const cplx<T> *vj = j == 0 ? u0 : V + (long long)j * n;
                cplx<T> v[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) v[u] = vj[e + u * stride];
#pragma unroll
                for (int u = 0; u < kU; ++u) cmac_cb(acc[j], wv[u], v[u]);  // conj(v) * w
            }
        }
    }
    for (; e < n; e += stride) {
        const cplx<T> wv = w[e];
#pragma unroll
        for (int j = 0; j < MV; ++j)
            if (j < nv) cmac_cb(acc[j], wv, (j == 0 ? u0 : V + (long long)j * n)[e]);
    }
    // all the sums at once: warp sums in T, then eight lanes add each part's warp results
    __shared__ double sw[MV * 2 * (kThr / 32)];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int j = 0; j < MV; ++j) {
            if (j < nv) {
                acc[j].re += __shfl_down_sync(0xffffffffu, acc[j].re, o);
                acc[j].im += __shfl_down_sync(0xffffffffu, acc[j].im, o);
            }
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < MV; ++j) {
            if (j < nv) {
                sw[(2 * j) * (kThr / 32) + wid] = (double)acc[j].re;
                sw[(2 * j + 1) * (kThr / 32) + wid] = (double)acc[j].im;
            }
        }
    }
    __syncthreads();
    static_assert(MV * 2 * (kThr / 32) <= kThr, "one thread per warp result");
    // thread 8 c + w: warp w's result of sum c (vector c / 2; real or imaginary part)
    __shared__ double scl[kCluster * kMaxM * 2];
    const int c = threadIdx.x / (kThr / 32);
    const bool mine = c < 2 * nv;
    double v = warps_sum8(mine ? sw[threadIdx.x] : 0.0);
    const bool first = mine && (threadIdx.x & (kThr / 32 - 1)) == 0;
    if (gs > 1) {
        static_assert(kCluster == kThr / 32, "the leader adds a cluster's CTAs as a CTA adds its warps");
        cl.barrier_wait();
        if (first) cl.map_shared_rank(scl, 0)[c * kCluster + cl.block_rank()] = v;
        cl.sync();
        if (cl.block_rank() != 0) return;
        v = warps_sum8(mine ? scl[threadIdx.x] : 0.0);
    }
    if (first) reinterpret_cast<double *>(part + (long long)(c >> 1) * ng + blockIdx.x / gs)[c & 1] = v;
}

// Sum of per-CTA partials written by other CTAs of the same launch (read through L2).
__device__ double sum_parts_cg(const double *part, int nparts)
{
    double s = 0.0;
    for (int p = threadIdx.x; p < nparts; p += kThr) s += __ldcg(part + p);
    return block_sum<double>(s);
}

// Publish this CTA's partial t (valid in thread 0); true in the CTA of the launch that does so last.
__device__ bool last_cta(FgState *st, double *part, double t)
{
    __shared__ int last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(&st->ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ bool cycles_left(int it, int m, long long maxit)
{
    return (long long)(it / m) < maxit;  // floor(it_counter / maxinnerit) < maxit
}

// INIT (first = 1): normr0 = beta = ||r||, hst = 1, it = 1 (FGMRES.m:62-76).
// END OF CYCLE (first = 0, while live): the true residual's norm decides the break of
// FGMRES.m:125, then the loop condition of FGMRES.m:88.  Either way the next cycle starts
// from beta = ||r|| (FGMRES.m:92).
// lazy: the cycle keeps its basis unnormalised (vector 0 = r itself, scale 1 / beta).
// Run by every thread of one CTA.
__device__ void norm_update(FgState *st, const double *part, int nparts, int first, double tol, int m, long long maxit,
                            int lazy)
{
    const double rnormr0 = st->rnormr0;
    const double s = sum_parts_cg(part, nparts);
    if (threadIdx.x != 0) return;
    FgHead &h = st->hd;
    // one reciprocal square root in place of a root and its reciprocals
    const bool plain = s > 0.0 && s <= DBL_MAX;
    const double rnr = plain ? rsqrt(s) : (s != 0.0 ? 1.0 / sqrt(s) : 0.0);
    const double nr = plain ? s * rnr : sqrt(s);
    if (first) {
        h.normr0 = nr;
        h.hst = 1.0;
        h.it = 1;
        h.nhst = 0;
        h.conv = nr == 0.0 ? 1 : 0;
        h.rn = nr;
        h.live = (nr != 0.0 && h.hst > tol && cycles_left(h.it, m, maxit)) ? 1 : 0;
    } else {
        h.rn = nr;
        if (nr * rnormr0 < tol) {
            h.live = 0;
            h.conv = 1;
        } else {
            if (h.hst <= tol) h.conv = 1;  // (a NaN quasi-residual stops the loop unconverged)
            h.live = (h.hst > tol && cycles_left(h.it, m, maxit)) ? 1 : 0;
        }
    }
    h.beta = nr;
    st->rbeta = rnr;
    st->gres = nr;
    st->sv[0] = lazy ? rnr : 1.0;
    if (first) st->rnormr0 = rnr;
    st->ticket = 0;
    st->pend = 0;
    h.k = 0;
    h.go = h.live;
    st->g[0] = mk<double>(nr, 0.0);
}

__global__ void __launch_bounds__(kThr) fg_norm_kernel(FgState *st, const double *part, int nparts, double tol, int m,
                                                       long long maxit, int lazy)
{
    fg_begin();
    norm_update(st, part, nparts, 1, tol, m, maxit, lazy);
}

// r = b - ax (r may alias ax).  While the instance is live (gate) and per-CTA partials of ||r||^2 in part; with
// st the CTA that finishes last updates the state at the end of a cycle (norm_update: the launch that
// would do it took 3.5 us on every level).
template <typename T>
__global__ void __launch_bounds__(kThr) fg_sub_kernel(const cplx<T> *__restrict__ b, const cplx<T> *ax, cplx<T> *r,
                                                      long long n, double *part, const int *gate, FgState *st,
                                                      double tol, int m, long long maxit, int lazy)
{
    fg_begin();
    if (closed(gate)) return;
    T s = 0;
    for (long long e = blockIdx.x * (long long)kThr + threadIdx.x; e < n; e += (long long)gridDim.x * kThr) {
        const cplx<T> v = b[e] - ax[e];
        r[e] = v;
        s = fma(v.re, v.re, fma(v.im, v.im, s));
    }
    const double t = block_sum<T>(s);
    if (!st) {
        if (threadIdx.x == 0) part[blockIdx.x] = t;
        return;
    }
    if (last_cta(st, part, t)) norm_update(st, part, gridDim.x, 0, tol, m, maxit, lazy);
}

// Step j of the cycle (0-based): H(1:j+1, j+1) = h, H(j+2, j+1) = ||w||; Givens rotations
// replace the least-squares solve of FGMRES.m:111 (same solution and residual norm; y itself
// is back-substituted once per cycle, by back_substitute).  With H(j+2, j+1) = ||w|| real the
// new rotation needs only reciprocal square roots (FP64 divisions and square roots are long
// dependent sequences on this GPU): c = |a| / r, s = (a / |a|) ||w|| / r, r = sqrt(|a|^2 +
// ||w||^2), and the quasi-residual |g(j+2)| = |s| |g(j+1)| follows without a square root.
// Run by every thread of one CTA: the one that finishes the orthogonalisation last (preconditioned
// instances, whose next step the host decides on), an extra one of the next step's inner products, or
// the one that finishes a cycle's last orthogonalisation.  One warp does the arithmetic, lane 2 i + p on part p
// (real, imaginary) of row i: what bounds it is the number of FP64 instructions one after the other
// (see block_sum), 2 per earlier rotation here against 12 with a thread doing them all, and one reciprocal
// square root for the three values that need one.
// hist (optional): the quasi-residual history, hist[nhst] written after each step.
// lazy: the next basis vector is kept as w itself with scale 1 / ||w||.
__device__ void givens_step(FgState *st, const double *part, int nparts, int j, int m, double tol, double *hist,
                            int lazy)
{
    static_assert(kMaxM == 16, "one warp: two lanes per row of the column");
    constexpr unsigned kAll = 0xffffffffu;
    const int row = (threadIdx.x & 31) >> 1, p = threadIdx.x & 1;
    double d = 0.0, cs = 0.0, sr = 0.0, si = 0.0, gp = 0.0, go = 0.0, gres = 0.0, rnormr0 = 0.0;
    int nhst = 0, it = 0;
    if (threadIdx.x < 32) {
        if (row <= j) d = __ldcg(reinterpret_cast<const double *>(st->h) + threadIdx.x);  // written by the orthogonalisation's CTA 0, maybe in this launch
        if (row < j) {
            cs = st->cs[row];
            sr = st->sn[row].re;
            si = st->sn[row].im;
        }
        const double *g = reinterpret_cast<const double *>(st->g + j);
        gp = g[p];
        go = g[p ^ 1];
        gres = st->gres;
        rnormr0 = st->rnormr0;
        nhst = st->hd.nhst;
        it = st->hd.it;
    }
    const double w2 = sum_parts_cg(part, nparts);  // ||w||^2 (synchronises the block)
    if (threadIdx.x >= 32) return;
    const double sg = p ? 1.0 : -1.0;
    // rotations 0..j-1 on the column: row i + 1 becomes cs d_(i+1) - conj(sn) c_i, row i cs c_i + sn d_(i+1)
    const double dn = __shfl_down_sync(kAll, d, 2), dno = __shfl_xor_sync(kAll, dn, 1);
    const double pn = cs * dn, ssi = sg * si;
    double c = __shfl_sync(kAll, d, p), mine = c;
    for (int i = 0; i < j; ++i) {
        const double q = __shfl_sync(kAll, pn, 2 * i + p), ri = __shfl_sync(kAll, sr, 2 * i + p);
        const double ii = __shfl_sync(kAll, ssi, 2 * i + p), co = __shfl_xor_sync(kAll, c, 1);
        c = fma(ii, co, fma(-ri, c, q));
        if (row == i + 1) mine = c;
    }
    double r = fma(ssi, dno, fma(sr, dn, cs * mine));  // row i < j
    // the new rotation, from a = c_j and ||w||
    const double c2 = c * c, na2 = c2 + __shfl_xor_sync(kAll, c2, 1), r2 = na2 + w2;
    const double rs = rsqrt(row == 0 ? w2 : (row == 1 ? r2 : na2));
    const double rw = __shfl_sync(kAll, rs, 0), rr = __shfl_sync(kAll, rs, 2), rna = __shfl_sync(kAll, rs, 4);
    const double rhn = w2 > 0.0 ? rw : 0.0;
    const double hn = w2 * rhn;
    double cj, sabs, sj, rjj;
    if (w2 == 0.0) {
        cj = 1.0;
        sj = 0.0;
        sabs = 0.0;
        rjj = c;
    } else if (na2 == 0.0) {
        cj = 0.0;
        sj = p ? 0.0 : 1.0;
        sabs = 1.0;
        rjj = p ? 0.0 : hn;
    } else {
        const double ph = rna * c;
        cj = na2 * rna * rr;
        sabs = hn * rr;
        sj = sabs * ph;
        rjj = (r2 * rr) * ph;
    }
    const double so = __shfl_xor_sync(kAll, sj, 1);
    if (row < j) reinterpret_cast<double *>(st->R + j * kMaxM)[threadIdx.x] = r;
    if (row == j) {
        reinterpret_cast<double *>(st->R + j * kMaxM)[threadIdx.x] = rjj;
        reinterpret_cast<double *>(st->sn)[threadIdx.x] = sj;
        // g(j+1) = -conj(sn) g(j), g(j) = cs g(j): the imaginary part of sn is the odd lane's
        const double sre = p ? so : sj, sim = p ? sj : so;
        reinterpret_cast<double *>(st->g + j + 1)[p] = fma(sg * sim, go, -(sre * gp));
        reinterpret_cast<double *>(st->g + j)[p] = cj * gp;
    }
    if (threadIdx.x != 0) return;
    FgHead &h = st->hd;
    st->cs[j] = cj;
    const double gnew = sabs * gres;
    st->gres = gnew;
    const double q = gnew * rnormr0;
    h.hst = q;
    st->hn = hn;
    st->rhn = rhn;
    if (j + 1 < kMaxM) st->sv[j + 1] = lazy ? rhn : 1.0;
    const int nh = nhst + 1;
    h.nhst = nh;
    if (hist) hist[nh] = q;
    h.it = it + 1;
    h.k = j + 1;
    h.go = (q > tol && j + 1 < m) ? 1 : 0;
}

// y = R \ g, the least-squares solution of FGMRES.m:111 after the last step, back-substituted from the
// rotated Hessenberg matrix.  Run by every thread of one CTA.
__device__ void back_substitute(FgState *st, int m)
{
    // lane 2 l + p: part p of row l; a row's diagonal enters as its reciprocal, formed for all rows at once
    __shared__ double sR[2 * kMaxM * kMaxM];
    const int kk = st->hd.k;
    for (int q = threadIdx.x; q < 2 * m * kMaxM; q += kThr) sR[q] = reinterpret_cast<const double *>(st->R)[q];
    constexpr unsigned kAll = 0xffffffffu;
    const int row = (threadIdx.x & 31) >> 1, p = threadIdx.x & 1;
    double t = threadIdx.x < 32 && row < kk ? reinterpret_cast<const double *>(st->g)[threadIdx.x] : 0.0;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const double sg = p ? 1.0 : -1.0;
    const double x = row < kk ? sR[2 * (row * kMaxM + row) + p] : 0.0, x2 = x * x;
    const double dd = x2 + __shfl_xor_sync(kAll, x2, 1);
    const double qp = -sg * x * (dd == 0.0 ? 0.0 : 1.0 / dd), qo = __shfl_xor_sync(kAll, qp, 1);
    const double qr = p ? qo : qp, qi = sg * (p ? qp : qo);
    for (int i = kk - 1; i >= 0; --i) {
        const double y = fma(t, qr, __shfl_xor_sync(kAll, t, 1) * qi);
        const double yp = __shfl_sync(kAll, y, 2 * i + p), yo = __shfl_sync(kAll, y, 2 * i + (p ^ 1));
        if (row == i) reinterpret_cast<double *>(st->y)[threadIdx.x] = y;
        if (row < i) {
            const double *e = sR + 2 * (i * kMaxM + row);
            t = fma(-e[0], yp, fma(-sg * e[1], yo, t));
        }
    }
}

// a -= v * h
template <typename T>
__device__ __forceinline__ void csub_mul(cplx<T> &a, cplx<T> v, cplx<T> h)
{
    a.re -= v.re * h.re;
    a.re += v.im * h.im;
    a.im -= v.re * h.im;
    a.im -= v.im * h.re;
}

// wout = sv[k] win - sum_j V_j h_j, k = nv - 1, with h summed here from the dots' partials (every
// CTA in the same fixed order, so all agree; CTA 0 stores h in the state) and scaled by the
// stored vectors' factors: the basis vector j is sv[j] times stored vector j, win = A (stored
// vector k).  Per-CTA partials of ||wout||^2.  wout may be win, or null (a cycle's last vector, of which
// only the norm is needed).  In complex64 the first elements are loaded before the sums, whose latency
// they cover (6.7 us for 1-4 vectors on an 81x71x51 level without).
// tail: with kTailStep and kTailCycle the CTA that finishes last (a ticket counter in the state: every CTA
// publishes its partial, fences, then takes a ticket; no CTA waits for another) runs the step's Givens
// update (givens_step) for step j = nv - 1, and with kTailCycle the back substitution that ends a cycle (as
// CTA 0 does when the cycle's steps have stopped before), and resets the counter.  With kTailNone the
// update is left outstanding.
enum FgStepTail { kTailNone, kTailStep, kTailCycle };
template <typename T, int MV>
__global__ void __launch_bounds__(kThr, sizeof(T) == 4 && MV <= 8 ? 4 : 1) fg_orth_kernel(const cplx<T> *__restrict__ u0, const cplx<T> *__restrict__ V,
                                                       int nvec, const cplx<T> *win, cplx<T> *wout, long long n,
                                                       const double2 *__restrict__ dpart, int ng, FgState *st,
                                                       double *part, int m, double tol, double *hist, int tail,
                                                       const int *gate)
{
    fg_begin();
    if (closed(gate)) {
        if (blockIdx.x == 0) {
            if (threadIdx.x == 0) st->pend = 0;
            if (tail == kTailCycle && st->hd.live) back_substitute(st, m);
        }
        return;
    }
    const int nv = vectors<MV>(nvec);
    // vectors whose elements are loaded ahead (registers for four CTAs per SM)
    constexpr int kAhead = sizeof(T) == 4 && MV <= kExact ? (MV < 3 ? MV : MV < 5 ? 3 : 2) : 0;
    const long long stride = (long long)gridDim.x * kThr;
    long long e = blockIdx.x * (long long)kThr + threadIdx.x;
    cplx<T> a[kU], vv[kAhead ? kAhead : 1][kU];
    auto ahead = [&]() -> bool {
        if (e + (kU - 1) * stride >= n) return false;
#pragma unroll
        for (int u = 0; u < kU; ++u) a[u] = win[e + u * stride];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const cplx<T> *vj = j == 0 ? u0 : V + (long long)j * n;
#pragma unroll
            for (int u = 0; u < kU; ++u) vv[j][u] = vj[e + u * stride];
        }
        return true;
    };
    bool have = false;
    if constexpr (kAhead > 0) have = ahead();
    __shared__ cplx<T> sh[kMaxM];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int j = wid; j < nv; j += kThr / 32) {
        const double svj = st->sv[j], svk = st->sv[nv - 1];
        double re = 0.0, im = 0.0;
        for (int p = lane; p < ng; p += 32) {
            const double2 v = dpart[(long long)j * ng + p];
            re += v.x;
            im += v.y;
        }
        // lanes 0-15 sum the real parts, 16-31 the imaginary ones: half the FP64 additions
        {
            const bool hi = lane & 16;
            double t = (hi ? im : re) + __shfl_xor_sync(0xffffffffu, hi ? re : im, 16);
            for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            re = t;
            im = __shfl_xor_sync(0xffffffffu, t, 16);
        }
        if (lane == 0) {
            const double f = svj * svk;
            const cplx<double> hj = mk<double>(f * re, f * im);      // H(j+1, k+1)
            sh[j] = mk<T>((T)(svj * hj.re), (T)(svj * hj.im));  // applied to stored vector j
            if (blockIdx.x == 0) st->h[j] = hj;
        }
    }
    const T sk = (T)st->sv[nv - 1];
    __syncthreads();
    T s = 0;
    auto put = [&]() {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (wout) wout[e + u * stride] = a[u];
            s = fma(a[u].re, a[u].re, fma(a[u].im, a[u].im, s));
        }
    };
    if constexpr (kAhead > 0) {
        while (have) {
#pragma unroll
            for (int u = 0; u < kU; ++u) a[u] = mk<T>(sk * a[u].re, sk * a[u].im);
#pragma unroll
            for (int j = 0; j < MV; ++j) {
                const cplx<T> *vj = j == 0 ? u0 : V + (long long)j * n;
                const cplx<T> hj = sh[j];
#pragma unroll
                for (int u = 0; u < kU; ++u) csub_mul(a[u], j < kAhead ? vv[j < kAhead ? j : 0][u] : vj[e + u * stride], hj);
            }
            put();
            e += kU * stride;
            have = ahead();
        }
    } else {
        for (; e + (kU - 1) * stride < n; e += kU * stride) {
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const cplx<T> t = win[e + u * stride];
                a[u] = mk<T>(sk * t.re, sk * t.im);
            }
#pragma unroll
            for (int j = 0; j < MV; ++j) {
                if (j < nv) {
                    const cplx<T> *vj = j == 0 ? u0 : V + (long long)j * n;
                    cplx<T> v[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) v[u] = vj[e + u * stride];
                    const cplx<T> hj = sh[j];
#pragma unroll
                    for (int u = 0; u < kU; ++u) csub_mul(a[u], v[u], hj);
                }
            }
            put();
        }
    }
    for (; e < n; e += stride) {
        const cplx<T> t = win[e];
        cplx<T> b = mk<T>(sk * t.re, sk * t.im);
#pragma unroll
        for (int j = 0; j < MV; ++j)
            if (j < nv) csub_mul(b, (j == 0 ? u0 : V + (long long)j * n)[e], sh[j]);
        if (wout) wout[e] = b;
        s = fma(b.re, b.re, fma(b.im, b.im, s));
    }
    const double t = block_sum<T>(s);
    if (tail == kTailNone) {
        if (threadIdx.x == 0) {
            part[blockIdx.x] = t;
            if (blockIdx.x == 0) st->pend = nv;
        }
        return;
    }
    if (!last_cta(st, part, t)) return;
    givens_step(st, part, gridDim.x, nv - 1, m, tol, hist, tail == kTailCycle ? 1 : 0);
    if (threadIdx.x == 0) {
        st->ticket = 0;
        st->pend = 0;
    }
    if (tail == kTailCycle) {
        __syncthreads();
        back_substitute(st, m);
    }
}

// End of a preconditioned instance's cycle, one CTA (the host may have ended it before its last step).
__global__ void __launch_bounds__(kThr) fg_finish_kernel(FgState *st, int m)
{
    fg_begin();
    if (st->hd.live) back_substitute(st, m);
}

// x += sum_{j < k} B_j y_j over the steps of the cycle (FGMRES.m:117-121), y from back_substitute.
// Stored vector 0 is u0, vector j >= 1 is B + j n; with scaled != 0 the basis vector j is sv[j]
// times the stored one.  MV: the steps of a full cycle where those are kExact or fewer, whose loads then
// all go first (a cycle cut short takes the loop over its k steps), else 0.
template <typename T, int MV>
__global__ void __launch_bounds__(kThr) fg_xupd_kernel(cplx<T> *__restrict__ x, const cplx<T> *__restrict__ u0,
                                                       const cplx<T> *__restrict__ B, long long n, const FgState *st,
                                                       int scaled, const int *gate)
{
    fg_begin();
    __shared__ cplx<T> syt[kMaxM];
    const int kk = st->hd.k;
    if (threadIdx.x < kk) {
        const double f = scaled ? st->sv[threadIdx.x] : 1.0;
        const cplx<double> yv = st->y[threadIdx.x];
        syt[threadIdx.x] = mk<T>((T)(f * yv.re), (T)(f * yv.im));
    }
    if (closed(gate)) return;
    __syncthreads();
    const long long stride = (long long)gridDim.x * kThr;
    long long e = blockIdx.x * (long long)kThr + threadIdx.x;
    if (MV > 0 && kk == MV) {
        constexpr int kX = sizeof(T) == 4 ? kU : kU / 2;
        for (; e + (kX - 1) * stride < n; e += kX * stride) {
            cplx<T> a[kX], v[MV + 1][kX];
#pragma unroll
            for (int j = 0; j < MV; ++j)
#pragma unroll
                for (int u = 0; u < kX; ++u) v[j][u] = (j == 0 ? u0 : B + (long long)j * n)[e + u * stride];
#pragma unroll
            for (int u = 0; u < kX; ++u) a[u] = mk<T>(0, 0), v[MV][u] = x[e + u * stride];
#pragma unroll
            for (int j = 0; j < MV; ++j) {
                const cplx<T> yj = syt[j];
#pragma unroll
                for (int u = 0; u < kX; ++u) cmac(a[u], v[j][u], yj);
            }
#pragma unroll
            for (int u = 0; u < kX; ++u) x[e + u * stride] = v[MV][u] + a[u];
        }
    } else {
        for (; e + (kU - 1) * stride < n; e += kU * stride) {
            cplx<T> a[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) a[u] = mk<T>(0, 0);
            for (int j = 0; j < kk; ++j) {
                const cplx<T> *bj = j == 0 ? u0 : B + (long long)j * n;
                cplx<T> v[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) v[u] = bj[e + u * stride];
                const cplx<T> yj = syt[j];
#pragma unroll
                for (int u = 0; u < kU; ++u) cmac(a[u], v[u], yj);
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) x[e + u * stride] = x[e + u * stride] + a[u];
        }
    }
    for (; e < n; e += stride) {
        cplx<T> a = mk<T>(0, 0);
        for (int j = 0; j < kk; ++j) cmac(a, (j == 0 ? u0 : B + (long long)j * n)[e], syt[j]);
        x[e] = x[e] + a;
    }
}

// complex128 <-> complex64 copies of a field (the mixed-precision preconditioner's edges)
template <typename S, typename D>
__global__ void __launch_bounds__(kThr) fg_cast_kernel(const cplx<S> *__restrict__ a, cplx<D> *__restrict__ b,
                                                       long long n)
{
    for (long long e = blockIdx.x * (long long)kThr + threadIdx.x; e < n; e += (long long)gridDim.x * kThr)
        b[e] = mk<D>((D)a[e].re, (D)a[e].im);
}

// ---- host side -------------------------------------------------------------------------------

int device_sms()
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0)
            sms = v;
        else {
            cudaGetLastError();
            sms = 148;
        }
    }
    return sms;
}

// CTAs of the reduction kernels (and entries of the partial-sum buffers): one pass of kU
// elements per thread on the coarse levels (latency-bound there: more CTAs in flight), at most
// four CTAs per SM.
int parts_for(long long n)
{
    const long long p = (n + kU * kThr - 1) / (kU * kThr);
    const long long cap = 4LL * device_sms();
    return (int)(p < 1 ? 1 : (p > cap ? cap : p));
}

// Sub-allocations of one device arena, 256-byte aligned.
struct Arena {
    size_t used = 0;
    char *base = nullptr;
    template <typename U>
    U *take(size_t count)
    {
        const size_t off = (used + 255) & ~(size_t)255;
        used = off + sizeof(U) * count;
        return base ? reinterpret_cast<U *>(base + off) : nullptr;
    }
};

template <typename T>
struct Fg {                     // one FGMRES instance
    long long n = 0;
    int m = 0;
    bool pre = false;
    // cycles enqueued between two reads of the state by the host (unpreconditioned instances): an
    // instance that has stopped leaves x and r as they are, its further launches return at once
    int ahead = 1;
    int nparts = 1;
    cplx<T> *V = nullptr, *Z = nullptr, *w = nullptr, *r = nullptr;
    double2 *dpart = nullptr;
    double *part = nullptr;
    FgState *st = nullptr;
    long long nhist = 0;        // history entries to keep (the outer solve), else 0
    double *hist = nullptr;
    void carve(Arena &a)
    {
        hist = nhist ? a.take<double>(nhist) : nullptr;
        V = a.take<cplx<T>>((size_t)m * n);
        Z = pre ? a.take<cplx<T>>((size_t)m * n) : nullptr;
        w = a.take<cplx<T>>(n);
        r = a.take<cplx<T>>(n);
        dpart = a.take<double2>((size_t)kMaxM * nparts);  // (fewer where clusters add first)
        part = a.take<double>(nparts);
        st = a.take<FgState>(1);
    }
};

template <typename T>
using Pre = std::function<int(const cplx<T> *, cplx<T> *)>;

struct Run {                    // per-call context
    cudaStream_t s = nullptr;
    bool adj = false;
    int64_t launches = 0, syncs = 0;
    long long before = -1;      // CTAs of the launch before on the stream, -1: not one to overlap with
    FgHead *hh = nullptr;       // pinned copy of a state head

    int fetch(const FgState *st)
    {
        H3D_CUDA_TRY(cudaMemcpyAsync(hh, &st->hd, sizeof(FgHead), cudaMemcpyDeviceToHost, s));
        H3D_CUDA_TRY(cudaStreamSynchronize(s));
        ++syncs;
        before = -1;
        return H3D_OK;
    }
    unsigned blocks(long long n) const
    {
        const long long b = (n + kThr - 1) / kThr, cap = 8LL * device_sms();
        return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
    }
};

#define H3D_ML_LAUNCH(...)                   \
    do {                                     \
        __VA_ARGS__;                         \
        ++R.launches;                        \
        R.before = -1;                       \
        H3D_CUDA_TRY(cudaGetLastError());    \
    } while (0)

// A launch of a kernel that begins with fg_begin: set up while the launch before still runs, where the
// two together leave every CTA an SM of its own (the coarse levels, whose launches take a few
// microseconds each; larger grids would crowd the SMs that free up first).
template <typename... KA, typename... A>
int fg_launch(Run &R, unsigned grid, unsigned cluster, void (*kern)(KA...), A... args)
{
    cudaLaunchAttribute attr[2]{};
    int na = 0;
    if (R.before > 0 && R.before + (long long)grid <= device_sms()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = cluster;
        attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThr);
    cfg.stream = R.s;
    cfg.attrs = attr;
    cfg.numAttrs = na;
    H3D_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...));
    R.before = grid;
    ++R.launches;
    return H3D_OK;
}
#define H3D_FG(...)                                        \
    do {                                                   \
        if ((rc = fg_launch(R, __VA_ARGS__))) return rc;   \
    } while (0)

// What a caller needs beside x: the state's head back on the host (the outer solve), the residual b - A x
// in I.r, or nothing (then the residual after the last cycle, which decides nothing, is left out).
enum FgTail { kFgHead, kFgResidual, kFgNone };

// FGMRES.m on one instance: x (in/out; zero_x = the initial guess is zero, FGMRES.m:65-67).
// pre: the flexible preconditioner z = P v (null = identity, the basis itself updates x).
// tail: see FgTail (kFgHead reads the state head back at the end, into R.hh).
template <typename T>
int fgmres(Run &R, Fg<T> &I, const Op<T> &op, const cplx<T> *b, cplx<T> *x, bool zero_x, double tol,
           long long maxit, const Pre<T> *pre, FgTail tail)
{
    const long long n = I.n;
    const int m = I.m;
    const unsigned nb = (unsigned)I.nparts;
    // the inner products' CTAs, in clusters where more than two per SM each have that many partials to add
    // (287 CTAs: an FWI gradient on 81x71x51 grids 116 ms without clusters, 119 with)
    const unsigned gs = nb > 2u * device_sms() ? kCluster : 1u, nd = (nb + gs - 1) / gs * gs;
    int rc;
    // gate: as the kernels after it have it.  A step's matvec runs before the Givens update that may stop the
    // instance, so it sees the flag one step late: one matvec more than needed at most.
    auto matvec = [&](const cplx<T> *in, cplx<T> *out, const int *gate) -> int {
        ++R.launches;
        return launch_mvp<T>(op, in, out, 1, R.adj, false, R.s, &R.before, gate);
    };
    // Unpreconditioned instances keep their basis unnormalised (each stored vector with its scale
    // in the state): no separate scaling pass per step; vector 0 is the residual buffer itself.
    const int lazy = pre ? 0 : 1;
    if (zero_x) {
        H3D_FG(nb, 1u, fg_copy_kernel<T>, b, I.r, x, n, I.part);
    } else {
        if ((rc = matvec(x, I.w, nullptr))) return rc;
        H3D_FG(nb, 1u, fg_sub_kernel<T>, b, I.w, I.r, n, I.part, nullptr, nullptr, tol, m, maxit, lazy);
    }
    H3D_FG(1u, 1u, fg_norm_kernel, I.st, I.part, I.nparts, tol, m, maxit, lazy);
    int *live = &I.st->hd.live, *go = &I.st->hd.go;
    const cplx<T> *u0 = lazy ? I.r : I.V;
    cplx<T> *basis = pre ? I.Z : I.V;
    for (long long c = 0; c < maxit; ++c) {
        if (pre || (c > 0 && c % I.ahead == 0)) {
            if ((rc = R.fetch(I.st))) return rc;
            if (!R.hh->live) break;
        }
        if (!lazy) H3D_FG(nb, 1u, fg_scale_kernel<T>, I.r, I.V, n, &I.st->rbeta, live);
        bool stopped = false;  // on the quasi-residual, as read by the host: no further cycle (FGMRES.m:88)
        for (int j = 0; j < m; ++j) {
            const cplx<T> *vj = j == 0 ? u0 : I.V + (long long)j * n;
            if (pre) {
                if (j > 0) {
                    if ((rc = R.fetch(I.st))) return rc;
                    if (!R.hh->go) {
                        stopped = R.hh->hst <= tol;
                        break;
                    }
                }
                cplx<T> *zj = I.Z + (long long)j * n;
                if ((rc = (*pre)(vj, zj))) return rc;
                vj = zj;
            }
            if ((rc = matvec(vj, I.w, pre ? nullptr : go))) return rc;
            // the orthogonalised vector: straight into the next basis slot (lazy), else into w; nowhere after
            // the last step
            cplx<T> *wout = j + 1 == m ? nullptr : (lazy ? I.V + (long long)(j + 1) * n : I.w);
            auto step = [&](auto dots, auto orth) -> int {
                H3D_FG(nd + gs, gs, dots, u0, I.V, j + 1, I.w, n, I.dpart, go, I.st, I.part, I.nparts, m, tol, I.hist);
                H3D_FG(nb, 1u, orth, u0, I.V, j + 1, I.w, wout, n, I.dpart, (int)(nd / gs), I.st, I.part, m, tol,
                       I.hist, pre ? kTailStep : j + 1 == m ? kTailCycle : kTailNone, go);
                return H3D_OK;
            };
            switch (j) {
                case 0: rc = step(fg_dots_kernel<T, 1>, fg_orth_kernel<T, 1>); break;
                case 1: rc = step(fg_dots_kernel<T, 2>, fg_orth_kernel<T, 2>); break;
                case 2: rc = step(fg_dots_kernel<T, 3>, fg_orth_kernel<T, 3>); break;
                case 3: rc = step(fg_dots_kernel<T, 4>, fg_orth_kernel<T, 4>); break;
                case 4: rc = step(fg_dots_kernel<T, 5>, fg_orth_kernel<T, 5>); break;
                case 5: case 6: case 7: rc = step(fg_dots_kernel<T, 8>, fg_orth_kernel<T, 8>); break;
                default: rc = step(fg_dots_kernel<T, kMaxM>, fg_orth_kernel<T, kMaxM>);
            }
            if (rc) return rc;
            if (!lazy && j + 1 < m) H3D_FG(nb, 1u, fg_scale_kernel<T>, I.w, I.V + (long long)(j + 1) * n, n, &I.st->rhn, go);
        }
        if (pre) H3D_FG(1u, 1u, fg_finish_kernel, I.st, m);
        auto update = [&](auto kern) -> int {
            H3D_FG(nb, 1u, kern, x, pre ? I.Z : u0, basis, n, I.st, lazy, live);
            return H3D_OK;
        };
        switch (m) {
            case 1: rc = update(fg_xupd_kernel<T, 1>); break;
            case 2: rc = update(fg_xupd_kernel<T, 2>); break;
            case 3: rc = update(fg_xupd_kernel<T, 3>); break;
            case 4: rc = update(fg_xupd_kernel<T, 4>); break;
            case 5: rc = update(fg_xupd_kernel<T, 5>); break;
            default: rc = update(fg_xupd_kernel<T, 0>);
        }
        if (rc) return rc;
        if (tail == kFgNone && (stopped || c == maxit - 1)) break;
        if ((rc = matvec(x, I.w, live))) return rc;
        const bool end = tail == kFgResidual && c == maxit - 1;
        H3D_FG(nb, 1u, fg_sub_kernel<T>, b, I.w, I.r, n, I.part, live, end ? nullptr : I.st, tol, m, maxit, lazy);
    }
    if (tail == kFgHead) return R.fetch(I.st);
    return H3D_OK;
}

// The V-cycle hierarchy in one precision.
template <typename T>
struct Cycle {
    int nl = 0;
    Op<T> op[kMaxLevels];
    long long n[kMaxLevels] = {};
    const h3d_ml_transfer *Rt = nullptr, *Pt = nullptr;
    Fg<T> smooth[kMaxLevels], coarse[kMaxLevels], bottom;
    cplx<T> *rc[kMaxLevels] = {}, *xc[kMaxLevels] = {};
    cplx<T> *t1 = nullptr, *t2 = nullptr;
    long long t1n = 0, t2n = 0;
    double stol = 1e-6, ctol = 0.5;
    int sk = 3, ck = 3;

    void size(const int k[4], long long tmp1, long long tmp2)
    {
        t1n = tmp1;
        t2n = tmp2;
        sk = k[0];
        ck = k[2];
        for (int i = 0; i < nl; ++i) {
            if (i < nl - 1) {
                smooth[i].n = n[i];
                smooth[i].m = k[1];
                smooth[i].nparts = parts_for(n[i]);
                // A tight tolerance is seldom met: the stream is not drained after each cycle (ms per solve,
                // read every cycle -> every fourth, tolerance 1e-6: mixed 41 x 41 x 35 7.4 -> 7.0, 121 x 101 x
                // 81 26.0 -> 25.3; 0.1: 8.3 -> 8.2, 25.4 -> 25.3).  A loose one is, and the launches of the
                // cycles that are left, though they return at once, cost more than the wait (0.3: 8.3 -> 8.7,
                // 25.6 -> 26.6; 0.5: 8.4 -> 10.4, 26.1 -> 30.2).
                smooth[i].ahead = stol < 0.2 ? 4 : 1;
            }
            if (i >= 1) {
                coarse[i].n = n[i];
                coarse[i].m = k[3];
                coarse[i].pre = true;
                coarse[i].nparts = parts_for(n[i]);
            }
        }
        bottom.n = n[nl - 1];
        bottom.m = k[3];
        bottom.nparts = parts_for(n[nl - 1]);
    }
    void carve(Arena &a)
    {
        for (int i = 0; i < nl; ++i) {
            if (i < nl - 1) {
                smooth[i].carve(a);
            }
            if (i >= 1) {
                coarse[i].carve(a);
                rc[i] = a.take<cplx<T>>(n[i]);
                xc[i] = a.take<cplx<T>>(n[i]);
            }
        }
        bottom.carve(a);
        t1 = a.take<cplx<T>>(t1n);
        t2 = a.take<cplx<T>>(t2n);
    }

    int transfer(Run &R, const h3d_ml_transfer &t, const cplx<T> *x, cplx<T> *y, bool accum)
    {
        int d[3] = {t.n_in[0], t.n_in[1], t.n_in[2]};
        int rcode;
        if ((rcode = launch_axis<T>(t.rowptr[0], t.col[0], t.val[0], t.n_out[0], 0, d, x, t1, 1, 1.0, false, R.s)))
            return rcode;
        d[0] = t.n_out[0];
        if ((rcode = launch_axis<T>(t.rowptr[1], t.col[1], t.val[1], t.n_out[1], 1, d, t1, t2, 1, 1.0, false, R.s)))
            return rcode;
        d[1] = t.n_out[1];
        if ((rcode = launch_axis<T>(t.rowptr[2], t.col[2], t.val[2], t.n_out[2], 2, d, t2, y, 1, t.scale, accum,
                                    R.s)))
            return rcode;
        R.launches += 3;
        R.before = -1;
        return H3D_OK;
    }

    // x = V-cycle(i) b (GMG_V.m; x is overwritten)
    int vcycle(Run &R, int i, const cplx<T> *b, cplx<T> *x)
    {
        int rcode;
        if ((rcode = fgmres<T>(R, smooth[i], op[i], b, x, true, stol, sk, nullptr, kFgResidual))) return rcode;
        if ((rcode = transfer(R, Rt[i], smooth[i].r, rc[i + 1], false))) return rcode;  // b - A x
        Pre<T> pre;
        if (i + 1 == nl - 1)
            pre = [this, &R](const cplx<T> *v, cplx<T> *z) {
                return fgmres<T>(R, bottom, op[nl - 1], v, z, true, ctol, ck, nullptr, kFgNone);
            };
        else
            pre = [this, &R, i](const cplx<T> *v, cplx<T> *z) { return vcycle(R, i + 1, v, z); };
        if ((rcode = fgmres<T>(R, coarse[i + 1], op[i + 1], rc[i + 1], xc[i + 1], true, ctol, ck, &pre, kFgNone)))
            return rcode;
        if ((rcode = transfer(R, Pt[i], xc[i + 1], x, true))) return rcode;
        return fgmres<T>(R, smooth[i], op[i], b, x, false, stol, sk, nullptr, kFgNone);
    }
};

long long npts(const h3d_grid &g) { return (long long)g.n[0] * g.n[1] * g.n[2]; }

bool same3(const int32_t *a, const int32_t *b) { return a[0] == b[0] && a[1] == b[1] && a[2] == b[2]; }

}  // namespace
}  // namespace h3d

using namespace h3d;

extern "C" void h3d_ml_default_opts(h3d_ml_opts *o)
{
    if (!o) return;
    o->tol = 1e-6;
    o->maxit = 10000;
    o->maxinnerit = 5;
    o->precond = H3D_ML_PREC_MLGMRES;
    o->precision = H3D_PREC_FP64;
    o->k[0] = 3;
    o->k[1] = 5;
    o->k[2] = 3;
    o->k[3] = 5;
    o->smooth_tol = 1e-6;
    o->coarse_tol = 0.5;
}

extern "C" int h3d_mlgmres_solve(const h3d_ml_level *levels, int nlevels, const h3d_ml_transfer *restrict_ops,
                                 const h3d_ml_transfer *prolong_ops, const void *b, void *x, int mode,
                                 const h3d_ml_opts *opts, double *hst, int hst_cap, h3d_ml_info *info, void *stream)
{
    const auto t0 = std::chrono::steady_clock::now();
    h3d_ml_opts o;
    h3d_ml_default_opts(&o);
    if (opts) o = *opts;
    const bool ml = o.precond == H3D_ML_PREC_MLGMRES;
    if (!levels || !b || !x || nlevels < 1 || nlevels > kMaxLevels || (mode != H3D_FORWARD && mode != H3D_ADJOINT) ||
        (o.precond != H3D_ML_PREC_NONE && !ml) || (o.precision != H3D_PREC_FP64 && o.precision != H3D_PREC_MIXED) ||
        !(o.tol >= 0.0) || o.maxit < 1 || o.maxinnerit < 1 || o.maxinnerit > kMaxM) {
        set_error("h3d_mlgmres_solve: bad argument");
        return H3D_ERR_BAD_ARG;
    }
    if (ml) {
        if (nlevels < 2 || !restrict_ops || !prolong_ops || o.k[0] < 1 || o.k[1] < 1 || o.k[1] > kMaxM || o.k[2] < 1 ||
            o.k[3] < 1 || o.k[3] > kMaxM || !(o.smooth_tol >= 0.0) || !(o.coarse_tol >= 0.0)) {
            set_error("h3d_mlgmres_solve: the multigrid preconditioner needs 2 or more levels, their transfers, "
                      "and 1-%d steps per smoother / coarse cycle", kMaxM);
            return H3D_ERR_BAD_ARG;
        }
        for (int i = 0; i < nlevels; ++i)
            if (!levels[i].wn || (o.precision == H3D_PREC_MIXED && !levels[i].wn32)) {
                set_error("h3d_mlgmres_solve: level %d has no wavenumber of the precision asked for", i);
                return H3D_ERR_BAD_ARG;
            }
        for (int i = 0; i + 1 < nlevels; ++i) {
            const h3d_ml_transfer &r = restrict_ops[i], &p = prolong_ops[i];
            if (!same3(r.n_in, levels[i].grid.n) || !same3(r.n_out, levels[i + 1].grid.n) ||
                !same3(p.n_in, levels[i + 1].grid.n) || !same3(p.n_out, levels[i].grid.n)) {
                set_error("h3d_mlgmres_solve: transfer %d does not connect the grids of levels %d and %d", i, i,
                          i + 1);
                return H3D_ERR_BAD_ARG;
            }
            for (int a = 0; a < 3; ++a)
                if (!r.rowptr[a] || !r.col[a] || !r.val[a] || !p.rowptr[a] || !p.col[a] || !p.val[a]) {
                    set_error("h3d_mlgmres_solve: transfer %d has a null axis operator", i);
                    return H3D_ERR_BAD_ARG;
                }
        }
    } else if (!levels[0].wn) {
        set_error("h3d_mlgmres_solve: level 0 has no wavenumber");
        return H3D_ERR_BAD_ARG;
    }
    const long long cap_needed = 1 + (long long)o.maxit * o.maxinnerit;
    if (hst && hst_cap < cap_needed) {
        set_error("h3d_mlgmres_solve: hst holds %d values, the solve may record %lld", hst_cap, cap_needed);
        return H3D_ERR_BAD_ARG;
    }
    const int nl = ml ? nlevels : 1;
    for (int i = 0; i < nl; ++i) {
        const int rc = check_grid(&levels[i].grid);
        if (rc) return rc;
    }

    Run R;
    R.s = (cudaStream_t)stream;
    R.adj = mode == H3D_ADJOINT;
    static thread_local FgHead *pinned = nullptr;
    if (!pinned) H3D_CUDA_TRY(cudaMallocHost(&pinned, sizeof(FgHead)));
    R.hh = pinned;

    // operators and sizes
    Cycle<double> c64;
    Cycle<float> c32;
    const bool mixed = o.precision == H3D_PREC_MIXED;
    Op<double> op0;
    int rc = make_op_f64(&levels[0].grid, levels[0].wn, nullptr, &op0);
    if (rc) return rc;
    const long long n0 = npts(levels[0].grid);
    long long tmp1 = 1, tmp2 = 1;
    if (ml) {
        for (int i = 0; i + 1 < nl; ++i) {
            const h3d_ml_transfer *ts[2] = {&restrict_ops[i], &prolong_ops[i]};
            for (const h3d_ml_transfer *t : ts) {
                const long long a = (long long)t->n_out[0] * t->n_in[1] * t->n_in[2];
                const long long bq = (long long)t->n_out[0] * t->n_out[1] * t->n_in[2];
                tmp1 = a > tmp1 ? a : tmp1;
                tmp2 = bq > tmp2 ? bq : tmp2;
            }
        }
        auto setup = [&](auto &cy, auto make) -> int {
            cy.nl = nl;
            cy.Rt = restrict_ops;
            cy.Pt = prolong_ops;
            cy.stol = o.smooth_tol;
            cy.ctol = o.coarse_tol;
            for (int i = 0; i < nl; ++i) {
                cy.n[i] = npts(levels[i].grid);
                const int r2 = make(i, &cy.op[i]);
                if (r2) return r2;
            }
            cy.size(o.k, tmp1, tmp2);
            return H3D_OK;
        };
        if (mixed)
            rc = setup(c32, [&](int i, Op<float> *op) { return make_op_f32(&levels[i].grid, levels[i].wn32, nullptr, op); });
        else
            rc = setup(c64, [&](int i, Op<double> *op) { return make_op_f64(&levels[i].grid, levels[i].wn, nullptr, op); });
        if (rc) return rc;
    }
    Fg<double> outer;
    outer.n = n0;
    outer.m = o.maxinnerit;
    outer.pre = ml;
    outer.nparts = parts_for(n0);
    outer.nhist = hst ? cap_needed : 0;

    // one arena for every vector of the call
    Arena a;
    auto carve_all = [&](Arena &ar, cplx<float> **b32, cplx<float> **x32) {
        outer.carve(ar);
        if (ml) {
            if (mixed) {
                c32.carve(ar);
                *b32 = ar.take<cplx<float>>(n0);
                *x32 = ar.take<cplx<float>>(n0);
            } else
                c64.carve(ar);
        }
    };
    cplx<float> *b32 = nullptr, *x32 = nullptr;
    carve_all(a, &b32, &x32);
    DevBuf arena;
    if ((rc = arena.alloc(a.used, R.s))) return rc;
    Arena a2;
    a2.base = arena.as<char>();
    carve_all(a2, &b32, &x32);

    Pre<double> pre;
    if (ml && mixed)
        pre = [&](const cplx<double> *v, cplx<double> *z) -> int {
            const unsigned nb = R.blocks(n0);
            H3D_ML_LAUNCH((fg_cast_kernel<double, float><<<nb, kThr, 0, R.s>>>(v, b32, n0)));
            const int r2 = c32.vcycle(R, 0, b32, x32);
            if (r2) return r2;
            H3D_ML_LAUNCH((fg_cast_kernel<float, double><<<nb, kThr, 0, R.s>>>(x32, z, n0)));
            return H3D_OK;
        };
    else if (ml)
        pre = [&](const cplx<double> *v, cplx<double> *z) -> int { return c64.vcycle(R, 0, v, z); };

    rc = fgmres<double>(R, outer, op0, (const cplx<double> *)b, (cplx<double> *)x, false, o.tol, o.maxit,
                        ml ? &pre : nullptr, kFgHead);
    if (rc) return rc;
    if (hst) {
        hst[0] = 1.0;
        if (R.hh->nhst > 0)
            H3D_CUDA_TRY(cudaMemcpyAsync(hst + 1, outer.hist + 1, sizeof(double) * R.hh->nhst, cudaMemcpyDeviceToHost,
                                         R.s));
    }
    H3D_CUDA_TRY(cudaStreamSynchronize(R.s));
    if (info) {
        info->iters = R.hh->nhst;
        info->converged = R.hh->conv;
        info->rel_res = R.hh->hst;
        info->kernel_launches = R.launches;
        info->host_syncs = R.syncs;
        info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    if (!std::isfinite(R.hh->hst) || !std::isfinite(R.hh->rn)) {
        set_error("h3d_mlgmres_solve: non-finite residual (NaN or Inf in b, x or the wavenumbers)");
        return H3D_ERR_NONFINITE;
    }
    return H3D_OK;
}
