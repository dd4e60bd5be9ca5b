// Matrix-free matvec y = H x (and H^H x, dH x, dH^H x) as a z-marching stencil.
//
// A CTA owns a 32 x 4 (complex128: 32 x 8) column of rows and marches a chunk of planes in z.  Each plane of
// x (and, forward, of the wavenumber) is staged in shared memory with its one-point xy
// halo by asynchronous copies (three buffers: planes p+1 and p+2 stream in while plane p is
// used).  From a plane every thread forms the partial sums of its 3 x 3 in-plane
// neighbourhood that the stencil needs -- centre, the two x-faces, the two y-faces and
// the corner pairs grouped by the sign of dx and of dy -- and keeps the last three planes
// in registers (a register queue along z).  One output row then combines planes k-1,
// k, k+1 with its own PML values: the 27 coefficients of Helm3d_27pt.h:676-825 regroup
// into 9 complex factors (xi_lo / xi_hi per axis and the per-axis sums S) multiplying
// real-weighted brackets of plane sums, plus the wavenumber (mass) part.  The adjoint
// uses the same algebra with the neighbour-shifted, conjugated PML values and the
// centre wavenumber; the derivative variants keep only the mass part.
//
// The same kernel produces the FP64 residual r = b - A x with per-block partial sums of
// ||r||^2 and ||b||^2 (RESID).
#include "h3d_internal.cuh"
#include "h3d_kernels.cuh"
#include "h3d_mvpflat.cuh"
#include "h3d_reduce.cuh"
#include "h3d_planes.cuh"

namespace h3d {

// CTA columns: kMX x tile_rows.  What the complex64 kernel lacks is instructions to choose from (128
// registers a thread: 16 warps per SM), and four small CTAs wait at their barriers less than two large
// ones: 201 x 201 x 101 51.0 us with 32 x 8, 44.4 with 32 x 4 (46.2 with 32 x 2, whose halo is as large as
// its tile); 81 x 71 x 51 10.0, 9.0 (9.2); 22 x 19 x 14 3.5, 3.1 (3.2).  More registers' worth of CTAs per SM
// spill (five of 32 x 4: 50.0 us).  The residual kernels and complex128 keep the larger tile, and with it the
// number of their partial sums.
constexpr int kMX = 32;
template <typename T, bool RESID>
__host__ __device__ constexpr int tile_rows()
{
    return sizeof(T) == 4 && !RESID ? 4 : 8;
}
constexpr int kPX = kMX + 2;                     // row of a staged plane with its halo
constexpr int kBufs = 3;                         // staged planes: one in use, two on their way

template <int BYTES>
__device__ __forceinline__ void mv_cp_async(void *sdst, const void *gsrc, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    const int n = valid ? BYTES : 0;
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gsrc), "n"(BYTES), "r"(n) : "memory");
}

// Origin shift of the column tiling along one axis: with tiles of t columns starting at
// -shift, a tile boundary falls on the first row whose forward PML values are all 1 (lo), so
// the interior columns fill whole tiles and take the folded-bracket path.
__host__ __device__ inline int tile_shift(int lo, int hi, int t)
{
    return (lo > 0 && lo < hi && lo % t != 0) ? t - lo % t : 0;
}

template <typename T, bool ADJ, bool DERIV, bool WNC, bool RESID>
__global__ void __launch_bounds__(kMX *tile_rows<T, RESID>(), sizeof(T) == 8 ? 1 : (RESID ? 2 : 3)) mvp_zmarch_kernel(Op<T> op, const cplx<T> *__restrict__ x,
                                                              cplx<T> *__restrict__ y,
                                                              const cplx<T> *__restrict__ b, int kz,
                                                              int nchunks, double *part, const int *gate)
{
    constexpr int kMY = tile_rows<T, RESID>(), kPN = kPX * (kMY + 2);
    constexpr bool NEED_WN = !ADJ;  // forward: neighbour wavenumbers; adjoint: centre only
    __shared__ __align__(16) cplx<T> sx[kBufs][kPN];
    __shared__ T swr[NEED_WN ? kBufs : 1][NEED_WN ? kPN : 1];
    __shared__ T swi[NEED_WN && WNC ? kBufs : 1][NEED_WN && WNC ? kPN : 1];

    // the next launch may set up early; wait for the launch before (nothing in an ordinary launch)
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (gate && *gate == 0) return;
    const int tid = threadIdx.x + kMX * threadIdx.y;
    const int s = blockIdx.z / nchunks, chunk = blockIdx.z % nchunks;
    const int kb = chunk * kz, ke = min(op.nz, kb + kz);
    const int sx0 = tile_shift(op.int_lo_f[0], op.int_hi_f[0], kMX);
    const unsigned gx = (unsigned)(op.nx + sx0 + kMX - 1) / kMX;  // tiles side by side in x
    const int i0 = (int)(blockIdx.x % gx) * kMX - sx0;
    const int j0 = (int)(blockIdx.x / gx) * kMY - tile_shift(op.int_lo_f[1], op.int_hi_f[1], kMY);
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
    const bool valid = i >= 0 && i < op.nx && j >= 0 && j < op.ny;
    const cplx<T> *xs = x + (long long)s * op.N;

    // Staging: the CTA's halo'd plane has kPN points; thread tid copies points tid and
    // tid + kMX*kMY.  Their in-plane offsets (32-bit: the host refuses nx*ny >= 2^31) and
    // x/y bounds are fixed for the march; per plane only the plane's base pointers change
    // (the same for every thread).  Points outside the grid copy nothing (zero fill) from a
    // valid address: the plane base, or plane 0 for planes outside the grid.
    constexpr int kNT = kMX * kMY;
    constexpr int kSlots = (kPN + kNT - 1) / kNT;
    int goff[kSlots];
    bool gin[kSlots];
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        const int e = tid + q * kNT;
        const int li = e % kPX, lj = e / kPX;
        const int gi = i0 - 1 + li, gj = j0 - 1 + lj;
        gin[q] = e < kPN && gi >= 0 && gi < op.nx && gj >= 0 && gj < op.ny;
        goff[q] = gin[q] ? gi + op.nx * gj : 0;
    }
    auto stage = [&](int buf, int pk) {
        const bool kin = pk >= 0 && pk < op.nz;
        const long long zo = kin ? op.sz * pk : 0;
        const cplx<T> *xp = xs + zo;
        const T *wp = op.wn + zo;
        const T *wip = WNC ? op.wni + zo : nullptr;
#pragma unroll
        for (int q = 0; q < kSlots; ++q) {
            const int e = tid + q * kNT;
            if (e < kPN) {
                const bool in = kin && gin[q];
                const int g = in ? goff[q] : 0;
                mv_cp_async<sizeof(cplx<T>)>(&sx[buf][e], xp + g, in);
                if constexpr (NEED_WN) {
                    mv_cp_async<sizeof(T)>(&swr[buf][e], wp + g, in);
                    if constexpr (WNC) mv_cp_async<sizeof(T)>(&swi[buf][e], wip + g, in);
                }
            }
        }
    };

    RowPml<T> pml{};
    if (valid && !DERIV) pml = load_row_pml<T, ADJ>(op, i, j, 0);
    // Columns whose x and y PML values are all 1 across the CTA (uniform): folded brackets;
    // rows inside the z interior as well: the interior class constants.
    const int *ilo = ADJ ? op.int_lo_a : op.int_lo_f, *ihi = ADJ ? op.int_hi_a : op.int_hi_f;
    const bool xyint = !DERIV && !WNC && i0 >= ilo[0] && i0 + kMX <= ihi[0] && j0 >= ilo[1] &&
                       j0 + kMY <= ihi[1];
    auto zint = [&](int k) { return k >= ilo[2] && k < ihi[2]; };
    const int l = (threadIdx.x + 1) + kPX * (threadIdx.y + 1);
    const long long col = i + op.sy * j;  // the thread's column: row k at col + k sz
    double rr = 0.0, bb = 0.0;

    // One plane pk: add it to the pending rows pk-1 (lo), pk (mid) and pk+1 (hi) and finish
    // row pk-1, whose accumulator then serves row pk+2 (its first plane sets every bracket,
    // so nothing is cleared).  The caller rotates the three accumulators' roles, so no
    // accumulator is ever copied.
    // The plane after next is copied into the buffer that the barrier shows to be read to its end:
    // one barrier a plane, and two planes of time for a copy.
    auto step = [&](int pk, int buf, RowAcc<T> &lo, RowAcc<T> &mid, RowAcc<T> &hi) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        if (pk + 2 <= ke) stage(buf == 0 ? 2 : buf - 1, pk + 2);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        {
            const PlaneSums<T> P = plane_sums<T, ADJ, WNC, kPX>(sx[buf], NEED_WN ? swr[buf] : nullptr,
                                                                NEED_WN && WNC ? swi[buf] : nullptr, l);
            if (xyint) {
                if (zint(pk - 1)) acc_plane_xy<2, T, true>(lo, P, op);
                else acc_plane_xy<2, T, false>(lo, P, op);
                if (zint(pk)) acc_plane_xy<1, T, true>(mid, P, op);
                else acc_plane_xy<1, T, false>(mid, P, op);
                if (zint(pk + 1)) acc_plane_xy<0, T, true>(hi, P, op);
                else acc_plane_xy<0, T, false>(hi, P, op);
            } else {
                acc_plane<2, T, DERIV>(lo, P, op);
                acc_plane<1, T, DERIV>(mid, P, op);
                acc_plane<0, T, DERIV>(hi, P, op);
            }
        }
        const int k = pk - 1;  // row completed by this plane
        if (k >= kb && valid) {
            RowPml<T> p = pml;
            if constexpr (!DERIV) {
                // only the z values change along the march
                const cplx<T> *t = op.tab;
                p.Sz = t[op.sum[2] + k + 1];
                if constexpr (!ADJ) {
                    p.Azm = t[op.lo[2] + k + 1];
                    p.Azp = t[op.hi[2] + k + 1];
                } else {
                    p.Azm = t[op.hi[2] + k];
                    p.Azp = t[op.lo[2] + k + 2];
                }
            }
            const long long ctr = col + op.sz * k;
            cplx<T> wc = mk<T>(T(0), T(0));
            if constexpr (ADJ) wc = load_wn<T, WNC>(op, ctr);
            const cplx<T> v = !xyint     ? acc_finish<T, ADJ, DERIV, WNC>(lo, p, wc)
                              : zint(k) ? acc_finish_xy<T, ADJ, true>(lo, p, wc)
                                        : acc_finish_xy<T, ADJ, false>(lo, p, wc);
            if constexpr (RESID) {
                const cplx<T> bv = b[(long long)s * op.N + ctr];
                const cplx<T> r = bv - v;
                y[(long long)s * op.N + ctr] = r;
                rr += (double)cabs2(r);
                bb += (double)cabs2(bv);
            } else {
                y[(long long)s * op.N + ctr] = v;
            }
        }
    };

    RowAcc<T> Q0, Q1, Q2;  // rows pk-1, pk, pk+1 at the top of the loop
    acc_zero(Q0);
    acc_zero(Q1);
    acc_zero(Q2);
    stage(0, kb - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    stage(1, kb);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int pk = kb - 1; pk <= ke; pk += 3) {
        step(pk, 0, Q0, Q1, Q2);
        if (pk + 1 <= ke) step(pk + 1, 1, Q1, Q2, Q0);
        if (pk + 2 <= ke) step(pk + 2, 2, Q2, Q0, Q1);
    }
    if constexpr (RESID) {
        const double2 t = block_sum2_r(rr, bb);
        if (tid == 0) {
            const long long G = (long long)gridDim.x * nchunks;
            const long long blin = blockIdx.x + (long long)gridDim.x * chunk;
            part[2 * (s * G + blin)] = t.x;
            part[2 * (s * G + blin) + 1] = t.y;
        }
    }
}

// CTAs of the z-march kernel resident on the whole device (occupancy of the forward
// variant of the precision and mode), queried once per device and kept for the process:
// the residual's partial-sum buffer is sized from the same grid as the launch, so the
// answer never changes (a failed query is remembered as "unknown").  make_op primes it,
// outside any stream capture.
template <typename T, bool RESID>
static int zmarch_slots()
{
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 0;
    }
    if (cache[dev] == 0) {
        int per_sm = 0, sms = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mvp_zmarch_kernel<T, false, false, false, RESID>,
                                                          kMX * tile_rows<T, RESID>(), 0) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 0;
        }
        cache[dev] = per_sm * sms > 0 ? per_sm * sms : -1;
    }
    return cache[dev] > 0 ? cache[dev] : 0;
}

void mvp_prime_occupancy()
{
    zmarch_slots<float, false>();
    zmarch_slots<double, false>();
    zmarch_slots<float, true>();
    zmarch_slots<double, true>();
}

// Split of the z axis into marching chunks.  A CTA's time grows with the planes it marches
// (its rows plus the two halo planes), and the launch takes as many rounds of resident CTAs
// as the grid needs: the split minimises rounds x (chunk + 2), which balances the halo
// overhead of short chunks against the partly empty last round of a grid that does not fill
// the device (201 x 201 x 101 in complex64: 5 chunks of 21 planes, 1785 CTAs in 3 rounds of
// 608).  Without an occupancy figure, chunks of 16 planes.
template <typename T, bool RESID>
static dim3 zmarch_grid(const Op<T> &op, int nrhs, int *kz, int *nchunks)
{
    const long long gx = (op.nx + tile_shift(op.int_lo_f[0], op.int_hi_f[0], kMX) + kMX - 1) / kMX;
    constexpr int kMY = tile_rows<T, RESID>();
    const long long gy = (op.ny + tile_shift(op.int_lo_f[1], op.int_hi_f[1], kMY) + kMY - 1) / kMY;
    const int slots = zmarch_slots<T, RESID>();
    int best_kz = op.nz < 32 ? op.nz : 16;
    if (slots > 0) {
        long long best = -1;
        const int nmax = op.nz < 64 ? op.nz : 64;
        for (int n = 1; n <= nmax; ++n) {
            const int k = (op.nz + n - 1) / n;
            const long long ctas = gx * gy * (long long)((op.nz + k - 1) / k) * nrhs;
            const long long cost = ((ctas + slots - 1) / slots) * (k + 2);
            if (best < 0 || cost < best) {
                best = cost;
                best_kz = k;
            }
        }
    }
    *kz = best_kz;
    *nchunks = (op.nz + *kz - 1) / *kz;
    return dim3((unsigned)(gx * gy), 1, *nchunks * nrhs);  // all tiles along x: no limit on ny
}

// The flat kernel's z split: an SM works off its CTAs at a fixed rate whatever runs side by side,
// but the last one alone keeps the FP64 unit only 70% busy; a CTA's time grows with the planes it
// marches (its own, and about half the work for either halo plane): the split minimises
// (CTAs of the fullest SM + 0.4) x (chunk + 1).
static int device_sms()
{
    static int cache[64] = {0};
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 1;
    }
    if (cache[dev] == 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) {
            cudaGetLastError();
            v = 1;
        }
        cache[dev] = v;
    }
    return cache[dev];
}

// RESID: a split in z takes at most the partial sums per right-hand side of the tiled kernel's grid. One
// chunk may take more (a tile is 128 points here, 256 there): mvp_residual_parts turns to the tiled kernel
// where a caller's buffer is too small for that.
template <typename T, bool RESID>
static dim3 flat_grid(const Op<T> &op, int nrhs, int *kz, int *nchunks)
{
    const long long gx = ((long long)op.nx * op.ny + kFT - 1) / kFT, sms = device_sms();
    long long most = 65535LL * gx;
    if (RESID) {
        const dim3 g = zmarch_grid<T, RESID>(op, nrhs, kz, nchunks);
        most = (long long)g.x * g.y * *nchunks;
    }
    int best_kz = op.nz;
    long long best = -1;
    const int nmax = op.nz < 64 ? op.nz : 64;
    for (int n = 1; n <= nmax; ++n) {
        const int k = (op.nz + n - 1) / n;
        const long long nch = (op.nz + k - 1) / k, ctas = gx * nch * nrhs;
        if (nch > 1 && (nch * nrhs > 65535 || nch * gx > most)) break;
        const long long cost = (5 * ((ctas + sms - 1) / sms) + 2) * (k + 1);
        if (best < 0 || cost < best) {
            best = cost;
            best_kz = k;
        }
    }
    *kz = best_kz;
    *nchunks = (op.nz + best_kz - 1) / best_kz;
    return dim3((unsigned)gx, (unsigned)(*nchunks * nrhs));
}

// Whether the flat kernel takes a grid: complex128 (bound by the FP64 unit), and staged planes (one
// row more on either side of 128 points) that leave room for two CTAs per SM.  In complex64 the
// column tiles are faster (201 x 201 x 101: 44 us against 89): what counts there is instructions, and
// a row more on either side of 128 points is many times the copies of a 34 x 6 tile.
template <typename T>
static bool use_flat(const Op<T> &op)
{
    return sizeof(T) == 8 && flat_smem<double, false, true>(op.nx) <= 96 * 1024;
}

// early: set up while the launch before still runs (it must let this one, and fill no SM it needs).
template <typename... KA, typename... A>
static int mvp_start(void (*kern)(KA...), dim3 grd, dim3 blk, size_t smem, bool early, cudaStream_t st, const A &...args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grd;
    cfg.blockDim = blk;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    H3D_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...));
    return H3D_OK;
}

template <typename T, bool ADJ, bool DERIV, bool WNC, bool RESID>
static int flat_launch(const Op<T> &op, const cplx<T> *x, cplx<T> *y, const cplx<T> *b, dim3 grd, int kz, int nch,
                       double *part, const int *gate, bool early, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8) {
        const size_t smem = flat_smem<T, ADJ, WNC>(op.nx);
        auto *kern = mvp_flat_kernel<T, ADJ, DERIV, WNC, RESID>;
        if (smem > 48 * 1024)
            H3D_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        auto aligned = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
        const int vec = aligned(x) && aligned(op.wn) && (!WNC || aligned(op.wni));
        return mvp_start(kern, grd, dim3(kFT), smem, early, st, op, x, y, b, kz, nch, vec, part, gate);
    }
    return H3D_OK;
}

template <typename T, bool RESID>
static int zmarch_dispatch(const Op<T> &op, const cplx<T> *x, cplx<T> *y, const cplx<T> *b, int nrhs,
                           bool adj, bool deriv, double *part, int parts, cudaStream_t st,
                           long long *before = nullptr, const int *gate = nullptr)
{
    if ((long long)op.nx * op.ny >= (1LL << 31)) {
        set_error("a z plane of more than 2^31 - 1 points is not supported by the matvec");
        return H3D_ERR_NSIZE;
    }
    int kz, nch;
    bool flat = use_flat(op);
    dim3 grd;
    if (flat) {
        grd = flat_grid<T, RESID>(op, nrhs, &kz, &nch);
        if (RESID && (long long)grd.x * nch != parts) flat = false;  // sized for the tiled kernel
    }
    if (!flat) grd = zmarch_grid<T, RESID>(op, nrhs, &kz, &nch);
    if ((long long)nch * nrhs > 65535) {
        set_error("too many right-hand sides for one launch");
        return H3D_ERR_BAD_ARG;
    }
    const long long have = flat ? (long long)grd.x * nch : (long long)grd.x * grd.y * nch;
    if (RESID && have != parts) {
        // the partial-sum buffer was sized for another grid: refuse rather than overrun it
        set_error("residual: %lld column blocks per right-hand side, buffer sized for %d",
                  have, parts);
        return H3D_ERR_BAD_ARG;
    }
    const dim3 blk(kMX, tile_rows<T, RESID>());
    const bool wnc = op.wni != nullptr;
    int rc = H3D_OK;
    const long long ctas = (long long)grd.x * grd.y * grd.z;
    const bool early = before && *before > 0 && *before + ctas <= device_sms();
    if (before) *before = ctas;
#define H3D_ZM(A, D, W)                                                                                   \
    if (flat) rc = flat_launch<T, A, D, W, RESID>(op, x, y, b, grd, kz, nch, part, gate, early, st);        \
    else rc = mvp_start(mvp_zmarch_kernel<T, A, D, W, RESID>, grd, blk, 0, early, st, op, x, y, b, kz, nch, part, gate)
    switch ((adj ? 4 : 0) + (deriv ? 2 : 0) + (wnc ? 1 : 0)) {
    case 0: H3D_ZM(false, false, false); break;
    case 1: H3D_ZM(false, false, true); break;
    case 2: H3D_ZM(false, true, false); break;
    case 3: H3D_ZM(false, true, true); break;
    case 4: H3D_ZM(true, false, false); break;
    case 5: H3D_ZM(true, false, true); break;
    case 6: H3D_ZM(true, true, false); break;
    default: H3D_ZM(true, true, true); break;
    }
#undef H3D_ZM
    if (rc) return rc;
    H3D_CUDA_TRY(cudaGetLastError());
    return H3D_OK;
}

template <typename T>
int launch_mvp(const Op<T> &op, const cplx<T> *x, cplx<T> *y, int nrhs, bool adj, bool deriv,
               cudaStream_t st, long long *before, const int *gate)
{
    return zmarch_dispatch<T, false>(op, x, y, nullptr, nrhs, adj, deriv, nullptr, 0, st, before, gate);
}

int mvp_residual_parts(const Op<double> &op, int nrhs, long long most)
{
    int kz, nch;
    if (use_flat(op)) {
        const dim3 g = flat_grid<double, true>(op, nrhs, &kz, &nch);
        if (most < 0 || (long long)g.x * nch * nrhs <= most) return (int)(g.x * nch);
    }
    const dim3 g = zmarch_grid<double, true>(op, nrhs, &kz, &nch);
    return (int)(g.x * g.y * nch);
}

int launch_residual(const Op<double> &op, const cplx<double> *b, const cplx<double> *x, cplx<double> *r,
                    int nrhs, bool adj, double *part, int parts, cudaStream_t st)
{
    return zmarch_dispatch<double, true>(op, x, r, b, nrhs, adj, false, part, parts, st);
}

template int launch_mvp<double>(const Op<double> &, const cplx<double> *, cplx<double> *, int, bool, bool, cudaStream_t, long long *, const int *);
template int launch_mvp<float>(const Op<float> &, const cplx<float> *, cplx<float> *, int, bool, bool, cudaStream_t, long long *, const int *);

}  // namespace h3d
