// The lexicographic Kaczmarz double sweep on stored row coefficients: hyperplane launches with a
// warp per row, chained so that a launch's reads of coefficients run under the launch before.
//
// Rows of a plane t = i + 3j + 9k are independent (see h3d_stencil.cu).  With q = j + 3k a plane's
// rows are i = t - 3q for about nx / 3 values of q and, for each, about ny / 3 values of k: a
// rectangle of at most a few hundred rows, 2 (nx + 3 ny + 9 nz) planes one after another.  What a
// plane takes is therefore latency, not work:
//
//  * A warp projects one row, lane t on offset t: 15 dependent-issue FP64 instructions (a
//    32-lane FP64 instruction takes 16 cycles of the SM's unit, so a thread that forms and
//    projects a whole row by itself, about 600 of them, held every plane for 26 us).
//  * The coefficients, formed once for both passes, lie row by row (27 values side by side): one
//    coalesced read.  They, the norm and b are read before the wait for the launch before
//    (programmatic dependent launch); after it come one gather of x through L2, the reduction
//    and one scatter.
//
// Measured on 61^3, complex128, one right-hand side with b: 41.7 -> 4.6 ms per double sweep (1562
// planes at 2.7 us each: launch rate and the latency of x through L2 bound it now; 0.4 ms of it
// forms the coefficients), against the kernel that forms each row in one thread (h3d_stencil.cu),
// which stays for grids whose 27 N coefficients would take more than half of the free memory.
#include "h3d_internal.cuh"
#include "h3d_kernels.cuh"

namespace h3d {
namespace {

constexpr int kWarps = 4;  // rows per CTA: one per SM sub-partition

struct LexOffsets {
    unsigned char t[32];   // grid direction (dx + 1) + 3 (dy + 1) + 9 (dz + 1) of coefficient column l
};

// INV: scale holds 1/||a_i||^2, else ||a_i||^2 (null: the sum over the row's coefficients).
template <typename T, bool INV>
__global__ void __launch_bounds__(32 * kWarps) lex_row_kernel(int nx, int ny, int nz, long long N,
                                                              const cplx<T> *__restrict__ coef,
                                                              const __grid_constant__ LexOffsets offs,
                                                              const T *__restrict__ scale, cplx<T> *x,
                                                              const cplx<T> *__restrict__ b, int nrhs, int t, int q0,
                                                              T w, const int *active)
{
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int q = q0 + blockIdx.x, i = t - 3 * q;
    const int klo = q < ny ? 0 : (q - ny + 3) / 3;  // j = q - 3k < ny
    const int k = klo + blockIdx.y * kWarps + (threadIdx.x >> 5), j = q - 3 * k;
    if (k >= nz || j < 0 || i < 0 || i >= nx) {
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // a launch completes after the one before it
        return;
    }
    const int dir = lane < 27 ? offs.t[lane] : 13;
    const int dx = dir % 3 - 1, dy = (dir / 3) % 3 - 1, dz = dir / 9 - 1;
    const long long row = i + (long long)nx * (j + (long long)ny * k);
    const bool in = lane < 27 && i + dx >= 0 && i + dx < nx && j + dy >= 0 && j + dy < ny && k + dz >= 0 && k + dz < nz;
    const long long nb = in ? row + dx + (long long)nx * (dy + (long long)ny * dz) : row;
    const bool hi = lane & 16;  // sums: lanes 0-15 carry the real part, 16-31 the imaginary one
    cplx<T> c = mk<T>(T(0), T(0));
    if (lane < 27) c = coef[27 * row + lane];
    T ws;
    if (INV) {
        ws = w * scale[row];
    } else {
        T n2;
        if (scale) {
            n2 = scale[row];
        } else {
            n2 = cabs2(c);
            for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
        }
        ws = w / n2;
    }
    if (!in) c = mk<T>(T(0), T(0));  // couplings that leave the grid meet x = 0 and write nothing
    T bv = T(0);
    if (b) bv = hi ? b[row].im : b[row].re;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    for (int s = 0; s < nrhs; ++s) {
        if (active && !active[s]) continue;
        cplx<T> *xp = x + (long long)s * N + nb;
        cplx<T> v = mk<T>(T(0), T(0));
        if (in) v = load_cg(xp);
        if (s > 0 && b) bv = hi ? b[(long long)s * N + row].im : b[(long long)s * N + row].re;
        T re = c.re * v.re, im = c.re * v.im;
        re -= c.im * v.im;
        im += c.im * v.re;
        T sum = (hi ? im : re) + __shfl_xor_sync(0xffffffffu, hi ? re : im, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const T d = ws * (bv - sum), e = __shfl_xor_sync(0xffffffffu, d, 16);
        const T dr = hi ? e : d, di = hi ? d : e;
        if (in) {  // x += d conj(c)
            v.re += dr * c.re;
            v.re += di * c.im;
            v.im += di * c.re;
            v.im -= dr * c.im;
            *xp = v;
        }
    }
}

// Row coefficients [row][27] (t = (dx + 1) + 3 (dy + 1) + 9 (dz + 1)) and 1/||a_i||^2 (forward: the
// neighbours inside the grid; adjoint: all 27); rows go to memory through shared memory, 27 values
// side by side.
constexpr int kStoreT = 64;
template <typename T, bool ADJ, bool WNC>
__global__ void __launch_bounds__(kStoreT) lex_store_kernel(Op<T> op, cplx<T> *__restrict__ coef, T *__restrict__ rinv)
{
    __shared__ cplx<T> sc[kStoreT * 27];
    const long long r0 = blockIdx.x * (long long)kStoreT, row = r0 + threadIdx.x;
    if (row < op.N) {
        const int i = (int)(row % op.nx), j = (int)((row / op.nx) % op.ny), k = (int)(row / op.sz);
        const uint32_t m = inside_mask(i, j, k, op.nx, op.ny, op.nz);
        cplx<T> c[27];
        const long long ctr = row;
        row_coefs_with<T, ADJ, false, WNC>(op, i, j, k, ADJ ? 0x7ffffffu : m,
                                           [&](int dx, int dy, int dz) {
                                               return load_wn<T, WNC>(op, ctr + dx + op.sy * dy + op.sz * dz);
                                           },
                                           c);
        T nrm = T(0);
#pragma unroll
        for (int t = 0; t < 27; ++t) {
            nrm += cabs2(c[t]);
            sc[27 * threadIdx.x + t] = c[t];
        }
        rinv[row] = T(1) / nrm;
    }
    __syncthreads();
    const long long left = op.N - r0;
    const int n = 27 * (int)(left < kStoreT ? left : kStoreT);
    for (int e = threadIdx.x; e < n; e += kStoreT) coef[27 * r0 + e] = sc[e];
}

template <typename T, bool INV>
int lex_passes(int nx, int ny, int nz, const cplx<T> *coef, const LexOffsets &offs, const T *scale, cplx<T> *x,
               const cplx<T> *b, int nrhs, T w, const int *active, cudaStream_t st)
{
    const long long N = (long long)nx * ny * nz;
    const int tmax = (nx - 1) + 3 * (ny - 1) + 9 * (nz - 1);
    const int qmax = (ny - 1) + 3 * (nz - 1);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(32 * kWarps);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 0;  // the first launch waits for whatever came before in the ordinary way
    const int kext = (ny + 2) / 3 < nz ? (ny + 2) / 3 : nz;  // k values of one q, at most
    for (int pass = 0; pass < 2; ++pass)
        for (int tt = 0; tt <= tmax; ++tt) {
            const int t = pass ? tmax - tt : tt;
            const int lo = t - (nx - 1) <= 0 ? 0 : (t - (nx - 1) + 2) / 3;
            const int hi = t / 3 < qmax ? t / 3 : qmax;
            if (hi < lo) continue;  // no rows (axes below 3 points)
            cfg.gridDim = dim3((unsigned)(hi - lo + 1), (unsigned)((kext + kWarps - 1) / kWarps));
            H3D_CUDA_TRY(cudaLaunchKernelEx(&cfg, lex_row_kernel<T, INV>, nx, ny, nz, N, coef, offs, scale, x, b, nrhs,
                                            t, lo, w, active));
            cfg.numAttrs = 1;
        }
    return H3D_OK;
}

}  // namespace

template <typename T>
bool lex_coefs_fit(long long N)
{
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return sizeof(cplx<T>) * 27 * (size_t)N <= fr / 2;
}

template <typename T>
int store_lex_coefs(const Op<T> &op, bool adj, cplx<T> *coef, T *rinv, cudaStream_t st)
{
    const long long blocks = (op.N + kStoreT - 1) / kStoreT;
    if (blocks > 0x7fffffffLL) {
        set_error("grid too large for stored lexicographic coefficients");
        return H3D_ERR_NSIZE;
    }
    const bool wnc = op.wni != nullptr;
#define H3D_LS(A, W) lex_store_kernel<T, A, W><<<(unsigned)blocks, kStoreT, 0, st>>>(op, coef, rinv)
    if (!adj && !wnc) H3D_LS(false, false);
    else if (!adj && wnc) H3D_LS(false, true);
    else if (adj && !wnc) H3D_LS(true, false);
    else H3D_LS(true, true);
#undef H3D_LS
    H3D_CUDA_TRY(cudaGetLastError());
    return H3D_OK;
}

template <typename T>
int sweep_lex_stored(int nx, int ny, int nz, const cplx<T> *coef, const unsigned char dirs[27], const T *scale,
                     bool inverse, cplx<T> *x, const cplx<T> *b, int nrhs, T w, const int *active, cudaStream_t st)
{
    LexOffsets offs{};
    for (int l = 0; l < 27; ++l) offs.t[l] = dirs ? dirs[l] : (unsigned char)l;
    if (inverse) return lex_passes<T, true>(nx, ny, nz, coef, offs, scale, x, b, nrhs, w, active, st);
    return lex_passes<T, false>(nx, ny, nz, coef, offs, scale, x, b, nrhs, w, active, st);
}

template bool lex_coefs_fit<double>(long long);
template bool lex_coefs_fit<float>(long long);
template int store_lex_coefs<double>(const Op<double> &, bool, cplx<double> *, double *, cudaStream_t);
template int store_lex_coefs<float>(const Op<float> &, bool, cplx<float> *, float *, cudaStream_t);
template int sweep_lex_stored<double>(int, int, int, const cplx<double> *, const unsigned char[27], const double *, bool,
                                      cplx<double> *, const cplx<double> *, int, double, const int *, cudaStream_t);
template int sweep_lex_stored<float>(int, int, int, const cplx<float> *, const unsigned char[27], const float *, bool,
                                     cplx<float> *, const cplx<float> *, int, float, const int *, cudaStream_t);

}  // namespace h3d
