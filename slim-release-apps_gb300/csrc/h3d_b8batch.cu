// Batched BLOCK8 Kaczmarz double sweep: one launch per block parity, or one in all, over a table of problems
// of any sizes, the stored coefficients of each colour staged by bulk copies into a ring of
// shared-memory buffers that complete on mbarriers.
//
// This file: the work list, the tuner, and the complex128 kernel on stored coefficients; the
// complex64 kernel, which forms its coefficients, is in h3d_b8slab.cu.
//
// Row order and arithmetic are those of the BLOCK8 sweep (h3d_block8.cu, h3d_blockrow.cuh):
// 12^3 blocks in eight parity classes, 27 colours inside a block, forward then backward
// (Helm3dkaczswp_mex.c:60-120 with another row order).  What changes is how work and data
// reach a CTA:
//
//  * Work list.  A launch of parity p runs sum over problems of (blocks of parity p) x
//    (groups of R right-hand sides) CTAs, problem-major, block-major, group fastest (the CTAs
//    of one block sit side by side and share its coefficient slabs through L2).  A CTA finds
//    its problem by a binary search over the per-parity prefix counts.
//  * Staging.  Thread 0 issues, per colour step, one cp.async.bulk of the colour's 27.6 KB
//    coefficient slab and one of its 64 inverse row norms,
//    both completing on the step's mbarrier, S steps ahead into an S-deep ring; no other
//    thread spends instructions on the copies.  Interior blocks (all PML values 1, real
//    wavenumber) form their real coefficients from the staged wavenumber box instead and
//    fetch only the row norms; the wavenumber box shares its space with the ring.
//  * Bounded waits.  Every mbarrier wait gives up after wait_limit_ns (globaltimer); the CTA
//    then records H3D_ERR_TIMEOUT in the status word, waits (bounded again) for the copies
//    it still has in flight, and returns without writing its box back.  The host reads the
//    status word and fails the call; the context stays usable.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "h3d_b8.cuh"
#include "h3d_b8slab.cuh"
#include "h3d_blockrow.cuh"
#include "h3d_kernels.cuh"

namespace h3d {

namespace {

constexpr int kBS = 12;                 // block side
constexpr int kNR = 64;                 // rows per colour and block (4 x 4 x 4)
constexpr int kPX = kBS + 2, kPY = kBS + 2;
constexpr int kNB = kPX * kPY * (kBS + 2);  // halo'd box points

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// Global -> shared bulk copy (16-byte aligned ends, size a multiple of 16) completing on bar.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for the completion of the phase with the given parity; false after limit_ns.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns)
{
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ int ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int *p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
constexpr uint32_t slab_bytes() { return 27u * kNR * sizeof(cplx<T>); }
template <typename T>
constexpr uint32_t rinv_bytes() { return kNR * sizeof(T); }
template <typename T, int S>
constexpr size_t ring_bytes()
{
    return std::max((size_t)kNB * sizeof(T), (size_t)S * slab_bytes<T>());
}
// [S mbarriers, padded to 128 B] [R x-boxes] [ring, or the wavenumber box] [S row-norm buffers]
template <typename T, int R, int S>
constexpr size_t b8_smem() { return 128 + (size_t)R * kNB * sizeof(cplx<T>) + ring_bytes<T, S>() + S * rinv_bytes<T>(); }

// selftest (h3d_check_wait_timeout only) 1: the first step's copies are announced on its mbarrier but
// never issued, so that every wait of the first colour step expires.  2 (FLOW): the block at the origin does
// not publish its passes, so that the waits of the blocks around it expire.
//
// R right-hand sides per CTA; two lanes project one row of every colour for RPT of them, from one
// load of the row's coefficients (128 R / RPT threads).  Two lanes, so that one right-hand side
// runs four warps, one per SM sub-partition: each sub-partition has a quarter of the SM's FP64 unit (a
// warp's FP64 instruction takes it 64 cycles), and with a lane per row the two warps of a
// block left half of it idle (us per double sweep, one column, a lane per row -> two: 61^3 3450 ->
// 2110, 161 x 161 x 81 3760 -> 2910).
//
// FLOW: the whole double sweep in one launch of a CTA per SM.  A CTA draws the next block of the order
// "parities up, then down" (a ticket counter, flow[0]), starts its copies, and waits until the blocks
// around it have finished the passes that come before (flow[1 + ..]: passes finished per block and group, the
// passes of the middle parity counting as two); the blocks it waits for have smaller tickets, so each of
// them is done or in the hands of a running CTA.  The wait is bounded like the others.
template <typename T, int R, int RPT, int S, bool FLOW>
__global__ void __launch_bounds__(2 * kNR *R / RPT) sweep_b8_kernel(const B8Prob<T> *__restrict__ probs,
                                                                const int *__restrict__ starts, int nprob, cplx<T> *x,
                                                                const cplx<T> *b, T w, const int *active, int par,
                                                                int backward, int nsteps, int *err, int *flow,
                                                                unsigned long long limit_ns, int selftest)
{
    static_assert(R % RPT == 0, "RPT must divide R");
    constexpr int NT = 2 * kNR * R / RPT, SLAB = 27 * kNR;
    constexpr uint32_t SLABB = slab_bytes<T>(), RVB = rinv_bytes<T>();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ B8Prob<T> sp;
    __shared__ int s_pi;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    cplx<T> *sx = reinterpret_cast<cplx<T> *>(smem + 128);
    unsigned char *ring = smem + 128 + (size_t)R * kNB * sizeof(cplx<T>);
    T *rv = reinterpret_cast<T *>(ring + ring_bytes<T, S>());
    const int tid = threadIdx.x;

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < S; ++s) mbar_init(smem_u32(bars + s), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    int steps0 = 0;  // colour steps of this CTA's blocks before
    for (;;) {
        int cta = (int)blockIdx.x;
        if constexpr (FLOW) {
            __shared__ int s_cta;
            if (tid == 0) s_cta = atomicAdd(flow, 1);
            __syncthreads();
            cta = s_cta;
            int pp = 0;  // parity step: 0-7 up (7: both passes), 8-14 down
            for (; pp < 15; ++pp) {
                par = pp < 8 ? pp : 14 - pp;
                const int n = starts[par * (nprob + 1) + nprob];
                if (cta < n) break;
                cta -= n;
            }
            if (pp == 15) return;
            backward = pp > 7;
            nsteps = pp == 7 ? 54 : 27;
        }
        const int *st0 = starts + par * (nprob + 1);
        if (tid == 0) {  // the problem whose CTA range holds this CTA
            int lo = 0, hi = nprob - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (st0[mid] <= cta) lo = mid;
                else hi = mid - 1;
            }
            s_pi = lo;
        }
        __syncthreads();
        {
            const int *src = reinterpret_cast<const int *>(probs + s_pi);
            int *dst = reinterpret_cast<int *>(&sp);
            for (int e = tid; e < (int)(sizeof(B8Prob<T>) / sizeof(int)); e += NT) dst[e] = src[e];
        }
        __syncthreads();
        const Op<T> &op = sp.op;
        const int local = cta - st0[s_pi];
        const int blk = local / sp.ngrp, grp = local - blk * sp.ngrp;
        const int nI = (sp.NI - (par & 1) + 1) >> 1, nJ = (sp.NJ - ((par >> 1) & 1) + 1) >> 1;
        const int Ib = (par & 1) + 2 * (blk % nI);
        const int Jb = ((par >> 1) & 1) + 2 * ((blk / nI) % nJ);
        const int Kb = (par >> 2) + 2 * (blk / (nI * nJ));
        const int bi0 = Ib * kBS, bj0 = Jb * kBS, bk0 = Kb * kBS;
        const int s0 = grp * R;
        unsigned act = 0;  // bit r: column s0 + r of the problem takes part
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (s0 + r < sp.nrhs && (!active || active[sp.c0 + s0 + r])) act |= 1u << r;
        const long long bid = Ib + (long long)sp.NI * (Jb + (long long)sp.NJ * Kb);
        int *done = FLOW ? flow + 1 + sp.done0 : nullptr;
        const int passes = backward || nsteps == 54 ? 2 : 1;  // of this block, once it is finished
        if (!act) {  // uniform over the CTA, before any copy
            if constexpr (!FLOW) return;
            // (its neighbours' columns are the same ones: none of them waits for data)
            __syncthreads();
            if (tid == 0) st_release(done + bid * sp.ngrp + grp, passes);
            continue;
        }

        const int *ilo = sp.adj ? op.int_lo_a : op.int_lo_f, *ihi = sp.adj ? op.int_hi_a : op.int_hi_f;
        const bool interior = !sp.wnc && bi0 >= ilo[0] && min(bi0 + kBS, op.nx) <= ihi[0] && bj0 >= ilo[1] &&
                              min(bj0 + kBS, op.ny) <= ihi[1] && bk0 >= ilo[2] && min(bk0 + kBS, op.nz) <= ihi[2];
        const bool edge_block = bi0 == 0 || bj0 == 0 || bk0 == 0 || bi0 + kBS >= op.nx || bj0 + kBS >= op.ny ||
                                bk0 + kBS >= op.nz;
        const cplx<T> *slab0 = sp.coef + bid * 27 * SLAB;
        const T *rv0 = sp.rinv8 + bid * 27 * kNR;
        auto colour_of = [&](int st) { return st < 27 ? (backward ? 26 - st : st) : 53 - st; };
        auto issue = [&](int st) {  // thread 0: step st's slab and row norms -> its ring buffer
            const int q = colour_of(st), buf = (steps0 + st) % S;
            const uint32_t bar = smem_u32(bars + buf);
            mbar_expect_tx(bar, (interior ? 0u : SLABB) + RVB);
            if (selftest == 1 && st == 0) return;
            if (!interior) bulk_g2s(smem_u32(ring + (size_t)buf * SLABB), slab0 + (size_t)q * SLAB, SLABB, bar);
            bulk_g2s(smem_u32(rv + buf * kNR), rv0 + q * kNR, RVB, bar);
        };

        __syncthreads();
        if (tid == 0)
            for (int st = 0; st < S && st < nsteps; ++st) issue(st);
        auto land = [&](int st0, int st1) {  // thread 0: wait for the copies of steps st0 .. st1 - 1
            for (int st = st0; st < st1 && st < nsteps; ++st)
                if (!(selftest == 1 && st == 0))
                    (void)mbar_wait(smem_u32(bars + (steps0 + st) % S), (uint32_t)(((steps0 + st) / S) & 1), limit_ns);
        };
        if constexpr (FLOW) {
            // thread t < 27: the block at offset t of this one; up, lower parities must have passed once, down,
            // higher ones twice and this one once
            bool ready = true;
            if (tid < 27) {
                const int I = Ib + tid % 3 - 1, J = Jb + (tid / 3) % 3 - 1, K = Kb + tid / 9 - 1;
                const int q = (I & 1) | (J & 1) << 1 | (K & 1) << 2;
                const int need = !backward ? (q < par ? 1 : 0) : q > par ? 2 : q == par && tid == 13 ? 1 : 0;
                if (need && I >= 0 && I < sp.NI && J >= 0 && J < sp.NJ && K >= 0 && K < sp.NK) {
                    const int *d = done + (I + (long long)sp.NI * (J + (long long)sp.NJ * K)) * sp.ngrp + grp;
                    const unsigned long long t0 = global_ns();
                    while (ld_acquire(d) < need) {
                        if (ld_acquire(err) != 0 || global_ns() - t0 > limit_ns) {
                            ready = false;
                            break;
                        }
                        __nanosleep(200);
                    }
                }
            }
            if (__syncthreads_or(!ready)) {  // report it, let the copies in flight land, leave x alone
                if (tid == 0) {
                    atomicCAS(err, 0, (int)H3D_ERR_TIMEOUT);
                    land(0, S);
                }
                __syncthreads();
                return;
            }
        }

        // the halo'd boxes of x (and the wavenumber box of an interior block), zero outside the grid,
        // one box row (14 points along x) at a time.  One right-hand side: a thread per row, its 14
        // points unrolled (fewest instructions).  Several: a
        // half-warp per row, lane l on point l (the copies of a warp stay contiguous).
        const int i0 = bi0 - 1, j0 = bj0 - 1, k0 = bk0 - 1;
        constexpr int kRows = kPY * (kBS + 2);
        T *swr = reinterpret_cast<T *>(ring);
        const int li_lo = max(0, -i0), li_hi = min(kPX, op.nx - i0);  // box columns inside the grid
        if constexpr (R == 1) {
            for (int rw = tid; rw < kRows; rw += NT) {
                const int lj = rw % kPY, lk = rw / kPY;
                const int gj = j0 + lj, gk = k0 + lk;
                const bool rin = gj >= 0 && gj < op.ny && gk >= 0 && gk < op.nz;
                const long long g0 = rin ? (long long)i0 + op.sy * gj + op.sz * gk : 0;
                const cplx<T> *xr = x + sp.col0 + s0 * sp.cstride + g0;
#pragma unroll
                for (int li = 0; li < kPX; ++li) {
                    const bool in = rin && li >= li_lo && li < li_hi;
                    if (interior) blk_cp_async<sizeof(T)>(swr + rw * kPX + li, op.wn + (in ? g0 + li : 0), in);
                    blk_cp_async<sizeof(cplx<T>)>(sx + rw * kPX + li, in ? xr + li : x, in);
                }
            }
        } else {
            constexpr int kSlots = NT / 16;
            const int li = tid & 15, slot = tid >> 4;
            const bool lin = li >= li_lo && li < li_hi;
            const cplx<T> *xcol = x + sp.col0 + s0 * sp.cstride;
            for (int rw = slot; rw < kRows; rw += kSlots) {
                if (li >= kPX) continue;
                const int lj = rw % kPY, lk = rw / kPY;
                const int gj = j0 + lj, gk = k0 + lk;
                const bool in = lin && gj >= 0 && gj < op.ny && gk >= 0 && gk < op.nz;
                const long long g = in ? (long long)(i0 + li) + op.sy * gj + op.sz * gk : 0;
                const int e = rw * kPX + li;
                if (interior) blk_cp_async<sizeof(T)>(swr + e, op.wn + g, in);
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (act & (1u << r))
                        blk_cp_async<sizeof(cplx<T>)>(sx + (size_t)r * kNB + e, xcol + r * sp.cstride + g, in);
            }
        }
        blk_cp_async_wait_all();
        __syncthreads();

        // thread slot: half h of row (u, v, w) of every colour, right-hand sides s0 + r0 .. s0 + r0 + RPT - 1
        // (a half-warp spans (u, w): conflict-free box offsets)
        const int r0 = (tid / (2 * kNR)) * RPT, lane = tid & 31;
        const int u = lane & 3, ww = (lane >> 2) & 3, v = (tid % (2 * kNR)) >> 5, row = u + 4 * ww + 16 * v;
        const bool centre = lane < 16;
        const int sg = centre ? 1 : -1;
        const unsigned mine = (act >> r0) & ((1u << RPT) - 1u);
        cplx<T> bv_n[RPT];
#pragma unroll
        for (int kk = 0; kk < RPT; ++kk) bv_n[kk] = mk<T>(T(0), T(0));
        auto fetch_b = [&](int q) {  // b_i of the next colour's row, one step ahead
            const int i = bi0 + q % 3 + 3 * u, j = bj0 + (q / 3) % 3 + 3 * v, k = bk0 + q / 9 + 3 * ww;
            if (i < op.nx && j < op.ny && k < op.nz) {
                const long long ctr = i + op.sy * j + op.sz * k;
#pragma unroll
                for (int kk = 0; kk < RPT; ++kk)
                    if (mine & (1u << kk)) bv_n[kk] = b[sp.col0 + (s0 + r0 + kk) * sp.cstride + ctr];
            }
        };
        if (b) fetch_b(colour_of(0));
        for (int qq = 0; qq < nsteps; ++qq) {
            const int q = colour_of(qq), buf = (steps0 + qq) % S;
            cplx<T> bv[RPT];
#pragma unroll
            for (int kk = 0; kk < RPT; ++kk) bv[kk] = bv_n[kk];
            if (b && qq + 1 < nsteps) fetch_b(colour_of(qq + 1));
            const bool ok = mbar_wait(smem_u32(bars + buf), (uint32_t)(((steps0 + qq) / S) & 1), limit_ns);
            const int a = q % 3, bq = (q / 3) % 3, cq = q / 9;
            const int i = bi0 + a + 3 * u, j = bj0 + bq + 3 * v, k = bk0 + cq + 3 * ww;
            // the two halves of a row agree on `run`; every lane takes part in the exchange
            const bool run = ok && mine && i < op.nx && j < op.ny && k < op.nz;
            const int lc = (1 + a + 3 * u) + kPX * ((1 + bq + 3 * v) + kPY * (1 + cq + 3 * ww));
            const T inv = run ? rv[buf * kNR + row] : T(0);
            cplx<T> xv[RPT][14], part[RPT];
#pragma unroll
            for (int kk = 0; kk < RPT; ++kk) part[kk] = mk<T>(T(0), T(0));
            auto project = [&](int kk) {  // d of right-hand side kk from both halves' sums
                cplx<T> t = part[kk];
                t.re += __shfl_xor_sync(0xffffffffu, t.re, 16);
                t.im += __shfl_xor_sync(0xffffffffu, t.im, 16);
                return (w * inv) * (bv[kk] - t);
            };
            if (!interior) {
                const cplx<T> *sc = reinterpret_cast<const cplx<T> *>(ring + (size_t)buf * SLABB) + (centre ? 0 : 26 * kNR) + row;
                cplx<T> c[14];
                if (run) {
#pragma unroll
                    for (int t = 0; t < 14; ++t) c[t] = sc[sg * t * kNR];
                    if (!centre) c[13] = mk<T>(T(0), T(0));
#pragma unroll
                    for (int kk = 0; kk < RPT; ++kk)
                        if (mine & (1u << kk))
                            part[kk] = half_gather<T, kPX, kPY>(sx + (size_t)(r0 + kk) * kNB, c, xv[kk], lc, sg);
                }
                // neighbours outside the grid keep reading zero: a row on a face of the grid scatters to its
                // inside neighbours only
                uint32_t m = 0x7ffffffu;
                if (edge_block && (i == 0 || j == 0 || k == 0 || i == op.nx - 1 || j == op.ny - 1 || k == op.nz - 1))
                    m = inside_mask(i, j, k, op.nx, op.ny, op.nz);
                if (!centre) m = (__brev(m) >> 5) & 0x1fffu;  // bit t: offset 26 - t, no centre
#pragma unroll
                for (int kk = 0; kk < RPT; ++kk) {
                    const cplx<T> d = project(kk);
                    if (run && (mine & (1u << kk)))
                        half_scatter<T, kPX, kPY>(sx + (size_t)(r0 + kk) * kNB, c, xv[kk], d, m, lc, sg);
                }
            } else {
                T cr[14];
                if (run) {
                    if (sp.adj) half_interior_coefs<T, true, kPX, kPY>(op, swr, lc, sg, centre, cr);
                    else half_interior_coefs<T, false, kPX, kPY>(op, swr, lc, sg, centre, cr);
#pragma unroll
                    for (int kk = 0; kk < RPT; ++kk)
                        if (mine & (1u << kk))
                            part[kk] = half_gather_r<T, kPX, kPY>(sx + (size_t)(r0 + kk) * kNB, cr, xv[kk], lc, sg);
                }
#pragma unroll
                for (int kk = 0; kk < RPT; ++kk) {
                    const cplx<T> d = project(kk);
                    if (run && (mine & (1u << kk)))
                        half_scatter_r<T, kPX, kPY>(sx + (size_t)(r0 + kk) * kNB, cr, xv[kk], d, centre, lc, sg);
                }
            }
            if (__syncthreads_or(!ok)) {
                // a wait expired: report it, let the copies still in flight land, leave x alone
                if (tid == 0) {
                    atomicCAS(err, 0, (int)H3D_ERR_TIMEOUT);
                    land(qq, qq + S);
                }
                __syncthreads();
                return;
            }
            if (tid == 0 && qq + S < nsteps) issue(qq + S);  // the buffer this step used is free
        }
        // write the box back (halo included), points inside the grid only, as staged
        cplx<T> *xw = x + sp.col0 + s0 * sp.cstride;
        if constexpr (R == 1) {
            for (int rw = tid; rw < kRows; rw += NT) {
                const int lj = rw % kPY, lk = rw / kPY;
                const int gj = j0 + lj, gk = k0 + lk;
                if (gj < 0 || gj >= op.ny || gk < 0 || gk >= op.nz) continue;
                cplx<T> *xr = xw + (long long)i0 + op.sy * gj + op.sz * gk;
#pragma unroll
                for (int li = 0; li < kPX; ++li)
                    if (li >= li_lo && li < li_hi) xr[li] = sx[rw * kPX + li];
            }
        } else {
            constexpr int kSlots = NT / 16;
            const int li = tid & 15, slot = tid >> 4;
            if (li < kPX && li >= li_lo && li < li_hi) {
                for (int rw = slot; rw < kRows; rw += kSlots) {
                    const int lj = rw % kPY, lk = rw / kPY;
                    const int gj = j0 + lj, gk = k0 + lk;
                    if (gj < 0 || gj >= op.ny || gk < 0 || gk >= op.nz) continue;
                    const long long g = (long long)(i0 + li) + op.sy * gj + op.sz * gk;
                    const int e = rw * kPX + li;
#pragma unroll
                    for (int rr = 0; rr < R; ++rr)
                        if (act & (1u << rr)) xw[rr * sp.cstride + g] = sx[(size_t)rr * kNB + e];
                }
            }
        }
        if constexpr (!FLOW) return;
        steps0 += nsteps;
        // (the ring may have held an interior block's wavenumbers: plain writes before the next bulk copies)
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();  // every thread's part of the box is written, and the boxes are free
        if (tid == 0 && !(selftest == 2 && bid == 0)) {
            __threadfence();
            st_release(done + bid * sp.ngrp + grp, passes);
        }
    }
}

// 1/||a_i||^2 from the grid layout into the block- and colour-major layout of the slabs
// (0 for the slots of rows outside the grid).
template <typename T>
__global__ void rinv8_kernel(const T *__restrict__ rinv, T *__restrict__ rinv8, int nx, int ny, int nz,
                             long long sy, long long sz, int NI, int NJ, long long nslab)
{
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= nslab * kNR) return;
    const long long bq = e / kNR;
    const int row = (int)(e % kNR);
    const long long bid = bq / 27;
    const int q = (int)(bq % 27);
    const int Ib = (int)(bid % NI), Jb = (int)((bid / NI) % NJ), Kb = (int)(bid / ((long long)NI * NJ));
    const int u = row % 4, w = (row / 4) % 4, v = row / 16;
    const int i = Ib * kBS + q % 3 + 3 * u, j = Jb * kBS + (q / 3) % 3 + 3 * v, k = Kb * kBS + q / 9 + 3 * w;
    rinv8[e] = (i < nx && j < ny && k < nz) ? rinv[i + sy * j + sz * k] : T(0);
}

// Compiled configurations (R right-hand sides per CTA, RPT per thread, ring depth S):
// complex64 on the slab kernel (no ring); complex128 with a 2-deep ring (its R = 4 boxes would
// exceed a CTA's 227 KB of shared memory).
const B8Cfg kCfgF32[] = {{1, 1, 0}, {2, 2, 0}};
const B8Cfg kCfgF64[] = {{1, 1, 2}, {2, 1, 2}, {2, 2, 2}};

// flow: the counters of a sweep in one launch (nctas: its CTAs), or null.
template <typename T, int R, int RPT, int S>
int launch_b8(const B8Prob<T> *probs, const int *starts, int nprob, long long nctas, cplx<T> *x, const cplx<T> *b,
              T w, const int *active, int par, int backward, int nsteps, int *err, int *flow,
              unsigned long long limit_ns, int selftest, cudaStream_t st)
{
    constexpr size_t smem = b8_smem<T, R, S>();
    static_assert(smem + sizeof(B8Prob<T>) + 16 <= 232448, "batched BLOCK8 configuration exceeds shared memory");
    static std::atomic<unsigned long long> attr_set{0};  // bit per device
    int dev = 0;
    H3D_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev > 63 || !(attr_set.load() & bit)) {
        H3D_CUDA_TRY(cudaFuncSetAttribute(sweep_b8_kernel<T, R, RPT, S, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        H3D_CUDA_TRY(cudaFuncSetAttribute(sweep_b8_kernel<T, R, RPT, S, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        attr_set.fetch_or(bit);
    }
    auto *kern = flow ? sweep_b8_kernel<T, R, RPT, S, true> : sweep_b8_kernel<T, R, RPT, S, false>;
    kern<<<(unsigned)nctas, 2 * kNR * R / RPT, smem, st>>>(probs, starts, nprob, x, b, w, active, par, backward, nsteps, err,
                                                           flow, limit_ns, selftest);
    return H3D_OK;
}

template <typename T>
int launch_b8_cfg(int cfg, bool wnc, const B8Prob<T> &one, const B8Prob<T> *probs, const int *starts, int nprob, long long nctas, cplx<T> *x,
                  const cplx<T> *b, T w, const int *active, int par, int pass, bool chained, int *err, int *flow,
                  unsigned long long limit_ns, int selftest, cudaStream_t st)
{
    if constexpr (sizeof(T) == 4) {
        return launch_slab(kCfgF32[cfg].r, wnc, one, probs, starts, nprob, nctas, x, b, w, active, par, pass,
                           chained, st);
    } else {
#define H3D_B8_ARGS probs, starts, nprob, nctas, x, b, w, active, par, pass == 1, pass == 2 ? 54 : 27, err, flow, limit_ns, selftest, st
        switch (cfg) {
        case 0: return launch_b8<T, 1, 1, 2>(H3D_B8_ARGS);
        case 1: return launch_b8<T, 2, 1, 2>(H3D_B8_ARGS);
        case 2: return launch_b8<T, 2, 2, 2>(H3D_B8_ARGS);
        default: break;
        }
#undef H3D_B8_ARGS
    }
    set_error("batched BLOCK8 configuration %d out of range", cfg);
    return H3D_ERR_BAD_ARG;
}

// Tuner cache: device and batch shape (grid sizes, columns, precision, mode, kind of wavenumber) -> configuration.
std::mutex g_b8_mutex;
std::map<std::vector<long long>, int> g_b8_cache;

}  // namespace

int b8_num_cfgs(bool fp64) { return fp64 ? (int)(sizeof(kCfgF64) / sizeof(B8Cfg)) : (int)(sizeof(kCfgF32) / sizeof(B8Cfg)); }
B8Cfg b8_cfg(bool fp64, int c) { return fp64 ? kCfgF64[c] : kCfgF32[c]; }

template <typename T>
static void block_counts(const Op<T> &op, int *NI, int *NJ, int *NK)
{
    *NI = (op.nx + kBS - 1) / kBS;
    *NJ = (op.ny + kBS - 1) / kBS;
    *NK = (op.nz + kBS - 1) / kBS;
}

template <typename T>
size_t B8Batch<T>::bytes_needed() const
{
    size_t tot = 0;
    for (const Item &it : items) {
        int NI, NJ, NK;
        block_counts(it.op, &NI, &NJ, &NK);
        const size_t nslab = (size_t)NI * NJ * NK * 27;
        if (sizeof(T) == 8) tot += nslab * 27 * kNR * sizeof(cplx<T>) + nslab * kNR * sizeof(T) + (size_t)it.op.N * sizeof(T);
        else tot += slab_record_bytes(NI, NJ, NK, any_wnc());
    }
    return tot;
}

template <typename T>
int B8Batch<T>::setup(cudaStream_t st)
{
    int rc;
    if (items.empty()) {
        set_error("batched BLOCK8 sweep without problems");
        return H3D_ERR_BAD_ARG;
    }
    coefs.clear();
    rinvs.clear();
    for (const Item &it : items) {
        int NI, NJ, NK;
        block_counts(it.op, &NI, &NJ, &NK);
        const long long nslab = (long long)NI * NJ * NK * 27;
        if (nslab * kNR > 0x7fffffffLL * 64LL) {
            set_error("grid too large for the batched BLOCK8 sweep");
            return H3D_ERR_NSIZE;
        }
        if constexpr (sizeof(T) == 4) {  // the slab kernel forms its coefficients: block records only
            auto rb = std::make_unique<DevBuf>();
            if ((rc = rb->alloc(slab_record_bytes(NI, NJ, NK, any_wnc()), st))) return rc;
            if ((rc = launch_slab_pack(it.op, it.adj, NI, NJ, NK, any_wnc(), rb->as<T>(), st))) return rc;
            rinvs.push_back(std::move(rb));
            continue;
        }
        auto cb = std::make_unique<DevBuf>();
        auto rb = std::make_unique<DevBuf>();
        if ((rc = cb->alloc(sizeof(cplx<T>) * block8_coef_count(it.op.nx, it.op.ny, it.op.nz), st))) return rc;
        if ((rc = rb->alloc(sizeof(T) * (size_t)nslab * kNR, st))) return rc;
        if ((rc = store_block8_coefs<T>(it.op, it.adj, cb->as<cplx<T>>(), st))) return rc;
        DevBuf grid_rinv;
        if ((rc = grid_rinv.alloc(sizeof(T) * (size_t)it.op.N, st))) return rc;
        if ((rc = row_inv_norms<T>(it.op, it.adj, grid_rinv.as<T>(), st))) return rc;
        const long long n = nslab * kNR;
        rinv8_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(grid_rinv.as<T>(), rb->as<T>(), it.op.nx, it.op.ny,
                                                                       it.op.nz, it.op.sy, it.op.sz, NI, NJ, nslab);
        H3D_CUDA_TRY(cudaGetLastError());
        coefs.push_back(std::move(cb));
        rinvs.push_back(std::move(rb));
    }
    if (!errb.p && (rc = errb.alloc(sizeof(int), st))) return rc;
    err = errb.as<int>();
    H3D_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
    return H3D_OK;
}

template <typename T>
int B8Batch<T>::configure(int c, cudaStream_t st)
{
    const bool fp64 = sizeof(T) == 8;
    if (c < 0 || c >= b8_num_cfgs(fp64)) {
        set_error("batched BLOCK8 configuration %d out of range", c);
        return H3D_ERR_BAD_ARG;
    }
    const int R = b8_cfg(fp64, c).r;
    const int np = (int)items.size();
    std::vector<B8Prob<T>> h(np);
    std::vector<int> hs(8 * (np + 1), 0);
    long long tot[8] = {0, 0, 0, 0, 0, 0, 0, 0}, counters = 0;
    for (int i = 0; i < np; ++i) {
        const Item &it = items[i];
        B8Prob<T> &d = h[i];
        std::memset(&d, 0, sizeof d);
        d.op = it.op;
        if (sizeof(T) == 8) {
            d.coef = coefs[i]->as<cplx<T>>();
            d.rinv8 = rinvs[i]->as<T>();
        } else {
            d.rec = rinvs[i]->as<T>();
        }
        d.col0 = it.col0;
        d.cstride = it.op.N;
        d.c0 = it.c0;
        d.nrhs = it.nrhs;
        d.ngrp = (it.nrhs + R - 1) / R;
        d.adj = it.adj ? 1 : 0;
        d.wnc = it.op.wni != nullptr;
        block_counts(it.op, &d.NI, &d.NJ, &d.NK);
        d.done0 = (int)counters;
        counters += (long long)d.NI * d.NJ * d.NK * d.ngrp;
        for (int p = 0; p < 8; ++p) {
            const long long nI = (d.NI - (p & 1) + 1) / 2, nJ = (d.NJ - ((p >> 1) & 1) + 1) / 2,
                            nK = (d.NK - (p >> 2) + 1) / 2;
            hs[p * (np + 1) + i] = (int)tot[p];
            tot[p] += nI * nJ * nK * d.ngrp;
        }
    }
    for (int p = 0; p < 8; ++p) {
        if (tot[p] > 0x7fffffffLL) {
            set_error("batched BLOCK8 launch too large (%lld CTAs)", tot[p]);
            return H3D_ERR_BAD_ARG;
        }
        hs[p * (np + 1) + np] = (int)tot[p];
        nctas[p] = tot[p];
    }
    int rc;
    desc.release();
    starts.release();
    // A single complex64 problem's descriptor goes with each launch and it needs no tables.  (Nor copies of
    // h and hs, which a stream capture would record to be read at each replay, when they are gone; in
    // complex128 the call's status read refuses a capture.)
    if (sizeof(T) == 8 || np > 1) {
        if ((rc = desc.alloc(sizeof(B8Prob<T>) * np, st)) || (rc = starts.alloc(sizeof(int) * hs.size(), st))) return rc;
        // pageable sources: staged before the calls return
        H3D_CUDA_TRY(cudaMemcpyAsync(desc.p, h.data(), sizeof(B8Prob<T>) * np, cudaMemcpyHostToDevice, st));
        H3D_CUDA_TRY(cudaMemcpyAsync(starts.p, hs.data(), sizeof(int) * hs.size(), cudaMemcpyHostToDevice, st));
    }
    first = h[0];
    cfg = c;
    nflow = counters;
    flow.release();
    if (in_one_launch() && (rc = flow.alloc(sizeof(int) * (size_t)(1 + nflow), st))) return rc;
    return H3D_OK;
}

static int device_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return sms;
}

// One launch where a parity's blocks do not fill the SMs evenly.  Up to a block per SM nothing is gained
// (a block waits for its neighbours either way, and the launches are chained).  Beyond, a launch per parity
// lasts as long as the SMs with a block more than the rest: 161 x 161 x 81, 196 blocks on 152 SMs, an FP64
// CGMN iteration 3.56 -> 3.05 ms; whole sweep calls (which store the coefficients first) with 250, 343, 405
// and 588 blocks 5.83 -> 5.82, 11.7 -> 10.3, 10.5 -> 9.8 and 11.9 -> 9.8 ms.  Four rounds and more are even
// enough, and keep two CTAs per SM.
template <typename T>
bool B8Batch<T>::in_one_launch() const
{
    if (sizeof(T) == 4 || nflow > 0x3fffffffLL) return false;
    if (force_one_launch) return true;
    const long long most = *std::max_element(nctas, nctas + 8), sms = device_sms();
    return most > sms && most <= 4 * sms;
}

template <typename T>
int B8Batch<T>::launches() const
{
    if (in_one_launch()) return 1;
    int n = 0;
    for (int pp = 0; pp < 15; ++pp) n += nctas[pp < 8 ? pp : 14 - pp] > 0;
    return n;
}

template <typename T>
int B8Batch<T>::dsweep(cplx<T> *x, const cplx<T> *b, T w, const int *active, cudaStream_t st, int selftest)
{
    if (cfg < 0) {
        set_error("batched BLOCK8 sweep used before configure()");
        return H3D_ERR_BAD_ARG;
    }
    const int np = (int)items.size();
    const bool wnc = any_wnc();
    // Overlapping a launch's prologue with the one before pays while both fit the device at one CTA
    // per SM (61^3: 212 -> 189 us per double sweep); beyond that the early CTAs crowd the SMs that
    // free up first (161 x 161 x 81, 147-196 CTAs a launch: 259 -> 311 us).
    const int sms = device_sms();
    if (in_one_launch()) {
        H3D_CUDA_TRY(cudaMemsetAsync(flow.p, 0, sizeof(int) * (size_t)(1 + nflow), st));
        int rc = launch_b8_cfg<T>(cfg, wnc, first, desc.as<B8Prob<T>>(), starts.as<int>(), np, sms, x, b, w, active, 0, 0,
                                  false, err, flow.as<int>(), wait_limit_ns, selftest, st);
        if (rc) return rc;
        H3D_CUDA_TRY(cudaGetLastError());
        return H3D_OK;
    }
    // forward parities 0..6, parity 7 up and down in one launch, backward parities 6..0
    long long before = -1;  // CTAs of the launch before, while this sweep has one
    for (int pp = 0; pp < 15; ++pp) {
        const int par = pp < 8 ? pp : 14 - pp;
        if (!nctas[par]) continue;
        int rc = launch_b8_cfg<T>(cfg, wnc, first, desc.as<B8Prob<T>>(), starts.as<int>(), np, nctas[par], x, b, w, active,
                                  par, pp < 7 ? 0 : pp == 7 ? 2 : 1, before >= 0 && before + nctas[par] <= sms, err, nullptr, wait_limit_ns, selftest, st);
        if (rc) return rc;
        before = nctas[par];
    }
    H3D_CUDA_TRY(cudaGetLastError());
    return H3D_OK;
}

template <typename T>
int B8Batch<T>::max_nrhs() const
{
    int m = 0;
    for (const Item &it : items) m = std::max(m, it.nrhs);
    return m;
}

template <typename T>
int B8Batch<T>::tune(cplx<T> *y, long long len, cudaStream_t st)
{
    const bool fp64 = sizeof(T) == 8;
    int dev = 0;
    H3D_CUDA_TRY(cudaGetDevice(&dev));
    std::vector<long long> key{dev, (long long)sizeof(T)};
    for (const Item &it : items) {
        key.push_back(it.op.nx);
        key.push_back(it.op.ny);
        key.push_back(it.op.nz);
        key.push_back(it.nrhs);
        key.push_back(it.adj);
        key.push_back(it.op.wni != nullptr);
    }
    {
        std::lock_guard<std::mutex> lk(g_b8_mutex);
        auto f = g_b8_cache.find(key);
        if (f != g_b8_cache.end()) return configure(f->second, st);
    }
    const int mx = max_nrhs();
    int best = -1;
    float best_ms = 1e30f;
    cudaEvent_t e0, e1;
    H3D_CUDA_TRY(cudaEventCreate(&e0));
    H3D_CUDA_TRY(cudaEventCreate(&e1));
    int rc = H3D_OK;
    for (int c = 0; c < b8_num_cfgs(fp64) && !rc; ++c) {
        if (c > 0 && b8_cfg(fp64, c).r > mx) break;  // only groups the columns fill
        if ((rc = configure(c, st))) break;
        H3D_CUDA_TRY(cudaMemsetAsync(y, 0, sizeof(cplx<T>) * (size_t)len, st));
        if ((rc = dsweep(y, nullptr, T(1.5), nullptr, st))) break;  // warm-up
        cudaEventRecord(e0, st);
        for (int rep = 0; rep < 2 && !rc; ++rep) rc = dsweep(y, nullptr, T(1.5), nullptr, st);
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (verbose) fprintf(stderr, "[h3d] tune batched BLOCK8 R=%d: %.3f ms per double sweep\n", b8_cfg(fp64, c).r, 0.5 * ms);
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    {
        std::lock_guard<std::mutex> lk(g_b8_mutex);
        g_b8_cache[key] = best;
    }
    return configure(best, st);
}

template struct B8Batch<float>;
template struct B8Batch<double>;

}  // namespace h3d
