// Matvec kernel over flattened planes (included by h3d_mvp.cu).
//
// A CTA owns 128 consecutive points of a z plane (x fastest, rows running on into one another)
// and marches a chunk of planes.  A plane's stretch, with one row and one point more on either
// side, is staged in shared memory in 16-byte pieces, three planes deep, one barrier per plane.  A thread
// forms from its 3 x 3 neighbourhood the plane's contribution to the row in the plane (A), to the rows
// above and below (B, the same for both) and, where the z PML values are not 1, the two sums its
// z factors multiply (Z1: the rows above and below, Z2: the row in the plane):
//
//   y(k) = A(k) + B(k-1) + B(k+1) + Azm(k) Z1(k-1) + Azp(k) Z1(k+1) + Sz(k) Z2(k)
//
// (the 27 coefficients of Helm3d_27pt.h:676-825 sorted by plane; the x and y factors do not depend on
// z, so a thread outside the x/y interior keeps its nine complex in-plane coefficients for A and
// for B in registers, one inside
// uses real constants on the sums of faces and corners, one with a single axis in the PML the six sums
// that axis leaves).  Where the
// z values are 1 around a plane, Z1 and Z2 join A and B.  Interior or not is decided per warp.
//
// Why: FP64 matvecs are bound by the FP64 unit (2 multiply-adds per clock and SM), so what counts is
// operations per grid point: 60 (interior), 86 (z PML), 88-144 (x or y PML), against 80, 106 and 186
// with nine brackets per pending row, and no lanes on points outside the grid: a 61^3 grid on 32 x 8
// column tiles ran half of its lanes there.  100 operations per point on 201 x 201 x 101 (198 before),
// 71% of the unit's peak over the launch.  us per launch, forward, one column, against the column tiles: 17^3 36 -> 21,
// 31^3 61 -> 27, 61^3 186 -> 83, 101 x 101 x 51 308 -> 172, 161 x 161 x 81 842 -> 505, 201 x 201 x 101
// 1374 -> 915.
#pragma once

#include "h3d_internal.cuh"
#include "h3d_planes.cuh"
#include "h3d_reduce.cuh"

namespace h3d {

constexpr int kFT = 128;   // points (threads) per CTA
constexpr int kFB = 3;     // staged planes

// Points of a staged plane, with room for the alignment shift of its first 16-byte piece.
__host__ __device__ inline int flat_points(int nx) { return (kFT + 2 * nx + 2 + 3 + 7) & ~7; }

template <typename T, bool ADJ, bool WNC>
__host__ __device__ inline size_t flat_smem(int nx)
{
    return (size_t)kFB * flat_points(nx) * (sizeof(cplx<T>) + (ADJ ? 0 : sizeof(T) * (WNC ? 2 : 1)));
}

template <int BYTES>
__device__ __forceinline__ void fl_cp_async(void *sdst, const void *gsrc, int n)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gsrc), "n"(BYTES), "r"(n) : "memory");
}

// Elements [e0, e0 + m) of the array a[0, n) into dst; what lies outside the array is not touched.
// vec: 16-byte pieces (a is 16-byte aligned or a column behind an aligned one); element e0 then lands
// at dst[flat_shift(a, e0)].
template <typename E>
__device__ __forceinline__ int flat_shift(const E *a, long long e0, bool vec)
{
    return vec ? (int)(((unsigned long long)a + (unsigned long long)(e0 * (long long)sizeof(E))) & 15) / (int)sizeof(E) : 0;
}
template <typename E>
__device__ __forceinline__ void flat_stage(E *dst, const E *a, long long n, long long e0, int m, bool vec)
{
    if (vec) {
        const int sh = flat_shift(a, e0, true);
        const long long end = n * (long long)sizeof(E);
        const long long o0 = (e0 - sh) * (long long)sizeof(E);  // byte offset of the first piece
        const int pieces = ((sh + m) * (int)sizeof(E) + 15) / 16;
        for (int c = threadIdx.x; c < pieces; c += kFT) {
            const long long o = o0 + 16 * c;
            if (o + 16 > 0 && o < end)
                fl_cp_async<16>((char *)dst + 16 * c, (const char *)a + o, (int)(end - o < 16 ? end - o : 16));
        }
    } else {
        for (int c = threadIdx.x; c < m; c += kFT) {
            const long long e = e0 + c;
            if (e >= 0 && e < n) fl_cp_async<sizeof(E)>(dst + c, a + e, sizeof(E));
        }
    }
}

template <typename T, bool ADJ, bool DERIV, bool WNC, bool RESID>
__global__ void __launch_bounds__(kFT)
    mvp_flat_kernel(const __grid_constant__ Op<T> op, const cplx<T> *__restrict__ x, cplx<T> *__restrict__ y,
                    const cplx<T> *__restrict__ b, int kz, int nchunks, int vec, double *part, const int *gate)
{
    using C = cplx<T>;
    constexpr bool NEED_WN = !ADJ;   // forward: neighbour wavenumbers; adjoint: the centre's, at the end
    extern __shared__ __align__(16) unsigned char fl_smem[];
    const int mp = flat_points(op.nx);
    C *sx = reinterpret_cast<C *>(fl_smem);
    T *sw = reinterpret_cast<T *>(sx + kFB * mp), *swi = sw + kFB * mp;

    // the next launch may set up early; wait for the launch before (nothing in an ordinary launch)
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (gate && *gate == 0) return;
    const int tid = threadIdx.x;
    const int s = blockIdx.y / nchunks, chunk = (int)outside_in(blockIdx.y % nchunks, nchunks);
    const unsigned tile = outside_in(blockIdx.x, gridDim.x);
    const int kb = chunk * kz, ke = min(op.nz, kb + kz);
    const int nx = op.nx;
    const long long P0 = (long long)tile * kFT, p = P0 + tid;
    const bool valid = p < op.sz;
    const int j = valid ? (int)(p / nx) : 0, i = valid ? (int)(p - (long long)j * nx) : 0;
    const C *xs = x + (long long)s * op.N;
    const int m = kFT + 2 * nx + 2;
    const long long first = P0 - nx - 1;  // of plane 0

    auto stage = [&](int pk) {
        if (pk >= 0 && pk < op.nz && pk <= ke) {
            const int buf = (pk - kb + 1) % kFB;
            const long long e0 = first + op.sz * pk;
            flat_stage(sx + buf * mp, xs, op.N, e0, m, vec);
            if constexpr (NEED_WN) {
                flat_stage(sw + buf * mp, op.wn, op.N, e0, m, vec);
                if constexpr (WNC) flat_stage(swi + buf * mp, op.wni, op.N, e0, m, vec);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    stage(kb - 1);
    stage(kb);

    // Neighbours inside the plane: bit (dx + 1) + 3 (dy + 1).
    const bool xl = i > 0, xr = i < nx - 1, yl = j > 0, yr = j < op.ny - 1;
    const bool edge = __any_sync(0xffffffffu, !(xl && xr && yl && yr));
    const int *ilo = ADJ ? op.int_lo_a : op.int_lo_f, *ihi = ADJ ? op.int_hi_a : op.int_hi_f;
    const bool xint = !DERIV && __all_sync(0xffffffffu, !valid || (i >= ilo[0] && i < ihi[0]));
    const bool yint = !DERIV && __all_sync(0xffffffffu, !valid || (j >= ilo[1] && j < ihi[1]));
    const bool xyint = xint && yint;
    auto zrow = [&](int k) { return k < 0 || k >= op.nz || (k >= ilo[2] && k < ihi[2]); };

    // In-plane coefficients of a row outside the x/y interior, for A and for B; zf: the z parts of a row
    // whose z values are 1 included.
    C c1[9], c0[9];
    auto build = [&](bool zf) {
        RowPml<T> q = load_row_pml<T, ADJ>(op, i, j, 0);
        const T z = zf ? T(1) : T(0);
        const C one = mk<T>(z, T(0)), two = mk<T>(z + z, T(0));
        const C Ax[3] = {q.Axm, q.Sx, q.Axp}, Ay[3] = {q.Aym, q.Sy, q.Ayp};
#define H3D_FL(t, dx, dy, dz)                                                                          \
    if constexpr (dz == 0) {                                                                            \
        c1[(dx + 1) + 3 * (dy + 1)] = pml_term<dx, dy, 0, T>(op, Ax[dx + 1], Ay[dy + 1], one, q.Sx, q.Sy, two); \
        c0[(dx + 1) + 3 * (dy + 1)] = pml_term<dx, dy, 1, T>(op, Ax[dx + 1], Ay[dy + 1], one, q.Sx, q.Sy, two); \
    }
        H3D_FOR_27(H3D_FL)
#undef H3D_FL
        if constexpr (ADJ) {
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                c1[t] = cconj(c1[t]);
                c0[t] = cconj(c0[t]);
            }
        }
    };
    const C zero = mk<T>(T(0), T(0));
#pragma unroll
    for (int t = 0; t < 9; ++t) c1[t] = c0[t] = zero;
    int built = -1;

    C R = zero, Bp = zero, Z1p = zero;          // row pk's sum so far; B and Z1 of the plane before
    C Rm = zero, Bmp = zero;                    // adjoint: the mass sums, multiplied by conj(wn) at the end
    double rr = 0.0, bb = 0.0;
    for (int pk = kb - 1; pk <= ke; ++pk) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        stage(pk + 2);  // into the buffer of plane pk - 1, which every thread has left
        C Aq = zero, Bq = zero, Z1 = zero, Z2 = zero, Am = zero, Bm = zero;
        const bool mine = pk >= kb && pk < ke;  // halo planes contribute B and Z1 only
        if (pk >= 0 && pk < op.nz) {
            const int buf = (pk - kb + 1) % kFB;
            const long long e0 = first + op.sz * pk;
            const C *xp = sx + buf * mp + flat_shift(xs, e0, vec) + nx + 1 + tid;
            C v[9];  // (dx + 1) + 3 (dy + 1)
#pragma unroll
            for (int t = 0; t < 9; ++t) v[t] = xp[(t % 3 - 1) + nx * (t / 3 - 1)];
            if (edge) {
#pragma unroll
                for (int t = 0; t < 9; ++t)
                    if (!((t % 3 != 0 || xl) && (t % 3 != 2 || xr) && (t / 3 != 0 || yl) && (t / 3 != 2 || yr))) v[t] = zero;
            }
            // sums over faces and corners
            const C fx = cadd<true>(v[3], v[5]), fy = cadd<true>(v[1], v[7]);
            const C c4 = cadd<true>(cadd<true>(v[0], v[2]), cadd<true>(v[6], v[8]));
            C qm, qf, qc;  // mass sums: centre, faces, corners (forward: weighted by the wavenumber)
            if constexpr (NEED_WN) {
                const T *wp = sw + buf * mp + flat_shift(op.wn, e0, vec) + nx + 1 + tid;
                const T *wip = WNC ? swi + buf * mp + flat_shift(op.wni, e0, vec) + nx + 1 + tid : nullptr;
                auto w = [&](int t) {
                    const int o = (t % 3 - 1) + nx * (t / 3 - 1);
                    return mk<T>(wp[o], WNC ? wip[o] : T(0));
                };
                // a neighbour outside the plane has x = 0, its wavenumber may be anything: drop it too
                auto wok = [&](int t) {
                    C r = w(t);
                    if (edge && !((t % 3 != 0 || xl) && (t % 3 != 2 || xr) && (t / 3 != 0 || yl) && (t / 3 != 2 || yr)))
                        r = zero;
                    return r;
                };
                auto mac = [&](C &a, int t, bool set) {
                    const C wt = wok(t);
                    if constexpr (WNC) {
                        if (set) a = wt * v[t];
                        else cmac(a, wt, v[t]);
                    } else {
                        if (set) a = cscale<true>(wt.re, v[t]);
                        else fma_rc<true>(a, wt.re, v[t]);
                    }
                };
                mac(qm, 4, true);
                mac(qf, 1, true);
                mac(qf, 3, false);
                mac(qf, 5, false);
                mac(qf, 7, false);
                mac(qc, 0, true);
                mac(qc, 2, false);
                mac(qc, 6, false);
                mac(qc, 8, false);
            } else {
                qm = v[4];
                qf = cadd<true>(fx, fy);
                qc = c4;
            }
            C ma = zero, mb = cscale<true>(T(-kWM2), qm);
            fma_rc<true>(mb, T(-kWM3), qf);
            fma_rc<true>(mb, T(-kWM4), qc);
            if (mine) {
                ma = cscale<true>(op.wn_c, qm);
                fma_rc<true>(ma, T(-kWM2), qf);
                fma_rc<true>(ma, T(-kWM3), qc);
            }
            if constexpr (ADJ) {
                Am = ma;
                Bm = mb;
            } else {
                Aq = ma;
                Bq = mb;
            }
            if constexpr (!DERIV) {
                const bool zf = zrow(pk - 1) && zrow(pk) && zrow(pk + 1);
                if (xyint) {
                    if (zf) {
                        if (mine) {
                            fma_rc<true>(Aq, op.kint[0], v[4]);
                            fma_rc<true>(Aq, op.kint[1], fx);
                            fma_rc<true>(Aq, op.kint[2], fy);
                            fma_rc<true>(Aq, op.kint[4], c4);
                        }
                        fma_rc<true>(Bq, op.kint[3], v[4]);
                        fma_rc<true>(Bq, op.kint[5], fx);
                        fma_rc<true>(Bq, op.kint[6], fy);
                        fma_rc<true>(Bq, op.kint[7], c4);
                    } else {
                        if (mine) {
                            fma_rc<true>(Aq, op.kxy[3], v[4]);
                            fma_rc<true>(Aq, op.kxy[0], fx);
                            fma_rc<true>(Aq, op.kxy[1], fy);
                            fma_rc<true>(Aq, op.kxy[2], c4);
                        }
                        fma_rc<true>(Bq, op.kxy[7], v[4]);
                        fma_rc<true>(Bq, op.kxy[4], fx);
                        fma_rc<true>(Bq, op.kxy[5], fy);
                        fma_rc<true>(Bq, op.kxy[6], c4);
                    }
                } else {
                    if (built != (int)zf) {
                        build(zf);
                        built = (int)zf;
                    }
                    if (xint || yint) {
                        // coefficients symmetric about the interior axis: six sums instead of nine points
                        // (the axis in the PML: a, b its faces, f the other's, ca, cb its corner pairs)
                        C a = v[3], bq = v[5], f = fy, ca = cadd<true>(v[0], v[6]), cb = cadd<true>(v[2], v[8]);
                        C k1[6] = {c1[4], c1[3], c1[5], c1[1], c1[0], c1[2]}, k0[6] = {c0[4], c0[3], c0[5], c0[1], c0[0], c0[2]};
                        if (xint) {
                            a = v[1], bq = v[7], f = fx, ca = cadd<true>(v[0], v[2]), cb = cadd<true>(v[6], v[8]);
                            k1[1] = c1[1], k1[2] = c1[7], k1[3] = c1[3], k1[5] = c1[6];
                            k0[1] = c0[1], k0[2] = c0[7], k0[3] = c0[3], k0[5] = c0[6];
                        }
                        const C sv[6] = {v[4], a, bq, f, ca, cb};
                        if (mine) {
                            CSum<T> as = csum_init(Aq);
#pragma unroll
                            for (int t = 0; t < 6; ++t) csum_mac<true>(as, k1[t], sv[t]);
                            Aq = csum_value(as);
                        }
                        CSum<T> bs = csum_init(Bq);
#pragma unroll
                        for (int t = 0; t < 6; ++t) csum_mac<true>(bs, k0[t], sv[t]);
                        Bq = csum_value(bs);
                    } else {
                        if (mine) {
                            CSum<T> a = csum_init(Aq);
#pragma unroll
                            for (int t = 0; t < 9; ++t) csum_mac<true>(a, c1[t], v[t]);
                            Aq = csum_value(a);
                        }
                        CSum<T> bs = csum_init(Bq);
#pragma unroll
                        for (int t = 0; t < 9; ++t) csum_mac<true>(bs, c0[t], v[t]);
                        Bq = csum_value(bs);
                    }
                }
                if (!zf) {
                    Z1 = cscale<true>(op.pml_z, v[4]);
                    fma_rc<true>(Z1, -op.xz, fx);
                    fma_rc<true>(Z1, -op.yz, fy);
                    fma_rc<true>(Z1, -op.w3a2, c4);
                    if (mine) {
                        Z2 = cscale<true>(op.wn_z, v[4]);
                        fma_rc<true>(Z2, op.xz, fx);
                        fma_rc<true>(Z2, op.yz, fy);
                        fma_rc<true>(Z2, op.w3a2, c4);
                    }
                }
            }
        }
        // z factors of row k (adjoint: the conjugated, neighbour-shifted values)
        auto zfac = [&](int table, int at) {
            const C t = op.tab[table + at];
            return ADJ ? cconj(t) : t;
        };
        auto add_z = [&](C &o, C f, C v) {
            CSum<T> a = csum_init(o);
            csum_mac<true>(a, f, v);
            o = csum_value(a);
        };
        // plane pk completes row pk - 1
        const int k = pk - 1;
        if (k >= kb) {
            C o = cadd<true>(R, Bq);
            if constexpr (!DERIV) {
                if (!(zrow(k) && zrow(k + 1) && zrow(k + 2)) && pk < op.nz)
                    add_z(o, ADJ ? zfac(op.lo[2], k + 2) : zfac(op.hi[2], k + 1), Z1);
            }
            if (valid) {
                const long long ctr = p + op.sz * k;
                if constexpr (ADJ) {
                    const C mass = cadd<true>(Rm, Bm);
                    const C wc = load_wn<T, WNC>(op, ctr);
                    if constexpr (WNC) o = o + cconj(wc) * mass;
                    else fma_rc<true>(o, wc.re, mass);
                }
                if constexpr (RESID) {
                    const C bv = b[(long long)s * op.N + ctr];
                    const C r = bv - o;
                    y[(long long)s * op.N + ctr] = r;
                    rr += (double)cabs2(r);
                    bb += (double)cabs2(bv);
                } else {
                    y[(long long)s * op.N + ctr] = o;
                }
            }
        }
        // row pk so far
        if (mine) R = cadd<true>(Aq, Bp);
        if constexpr (!DERIV) {
            if (mine) {
                if (!(zrow(pk - 2) && zrow(pk - 1) && zrow(pk)))  // the plane before kept its Z1
                    add_z(R, ADJ ? zfac(op.hi[2], pk) : zfac(op.lo[2], pk + 1), Z1p);
                if (!(zrow(pk - 1) && zrow(pk) && zrow(pk + 1))) add_z(R, zfac(op.sum[2], pk + 1), Z2);
            }
        }
        Bp = Bq;
        Z1p = Z1;
        if constexpr (ADJ) {
            if (mine) Rm = cadd<true>(Am, Bmp);
            Bmp = Bm;
        }
    }
    if constexpr (RESID) {
        const double2 t = block_sum2_r(rr, bb);
        if (tid == 0) {
            const long long G = (long long)gridDim.x * nchunks;
            const long long blin = tile + (long long)gridDim.x * chunk;
            part[2 * (s * G + blin)] = t.x;
            part[2 * (s * G + blin) + 1] = t.y;
        }
    }
}

}  // namespace h3d
