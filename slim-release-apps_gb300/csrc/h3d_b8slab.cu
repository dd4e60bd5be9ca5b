// BLOCK8 Kaczmarz double sweep in complex64: one CTA per 12^3 block, one warp per z slab, the
// x window of every row kept in registers.
//
// Row order as in the other BLOCK8 kernels (h3d_b8batch.cu): 12^3 blocks in eight parity
// classes, 27 colours q = a + 3b + 9c inside a block, forward then backward.  Two facts about
// that order shape the kernel:
//
//  * While c stands still, the rows of slab w (local z = c + 3w) touch box planes 3w + c ..
//    3w + c + 2 and nothing else, so the four slabs of a block are independent for nine
//    colours.  A warp owns a slab and needs only __syncwarp there; the CTA meets three times per
//    pass, when c changes (a kernel with coefficients in a ring needs 27 CTA barriers and waits).
//  * While b and c stand still, the rows of a pencil along x (local y = b + 3v) have footprints
//    that shift by one point per colour a.  A row's three columns stay in registers: after a colour
//    a lane hands the column it leaves to the neighbour whose row enters it (one shuffle per
//    line), so a (b, c) step reads and writes the shared box once instead of three times.
//
// Lanes: u = lane & 3 and v = (lane >> 2) & 3 select the row, h = lane >> 4 which half of its
// nine (dy, dz) lines the lane holds: z - 1 lines with the centre line, z + 1 lines with the
// other y face (five slots, the fifth empty for h = 1; the two halves of a slot belong to the
// same offset class, so all lanes use the same constants).  The sum a.x takes one exchange between
// the halves.  The box rows are pitched 14, with 2 extra points after every third row, so that
// the 16 rows of a half-warp fall on 16 different 8-byte banks.
//
// Coefficients are formed from three 1D tables per block,
//   c_t = kx X[dx](i) + ky Y[dy](j) + kz Z[dz](k) - WM_t wn
// (the closed form of every offset class of Helm3d_27pt.h:676-825, X[0] = xi_lo + xi_hi and
// X[-1], X[+1] the directional values), the y and z parts once per (b, c) step: nothing is
// stored per row but 1/||a_i||^2, against 216 B of stored coefficients per row and pass.
//
// What bounds it: one warp's instruction stream (about 2.6 cycles per instruction at one warp per
// scheduler; about 680 cycles per colour of a PML block, 415 of an interior one).  Measured against
// the ring kernel it replaces, us per double sweep: 61^3 405 -> 201, 161 x 161 x 81 420 -> 255,
// 201 x 201 x 101 500 -> 350; eight right-hand sides on 161 x 161 x 81 1460 -> 950.  Forms that
// measured slower on 61^3: four lanes per row with two warps per slab 258, the three
// colours of a pencil as one forward substitution on precomputed row products with two lanes per
// row 208-227, four lanes 213, one lane 432 (its straight-line code outruns the instruction cache).
#include "h3d_b8slab.cuh"

#include <atomic>

#include "h3d_blockrow.cuh"
#include "h3d_kernels.cuh"

namespace h3d {
namespace {

using C = cplx<float>;

constexpr int kBS = 12, kBP = kBS + 2;               // block side, box side
constexpr int kOwn = kBS * kBS * kBS;
constexpr int kPlane = kBP * kBP + 2 * 4, kBox = kBP * kPlane;  // pitched box plane, box
__host__ __device__ constexpr int row_off(int y) { return kBP * y + 2 * (y / 3); }
constexpr int kNT = 128, kNS = 5;                    // threads; (dy, dz) lines per lane
constexpr bool kPK = true;                           // packed FP32 pairs

// Block record in device memory (slab_pack_kernel), copied to shared memory as it stands:
// [1/||a||^2 of the block's rows, z, y, x | wavenumber box in the box layout], zero outside the grid.
template <bool WNC>
constexpr int rec_floats() { return kOwn + kBox * (WNC ? 2 : 1); }
static_assert(rec_floats<false>() % 4 == 0 && rec_floats<true>() % 4 == 0 && kOwn % 4 == 0, "16-byte copies");

// [x boxes | record | tables | b boxes]
template <int R, bool WNC, bool HASB>
constexpr size_t slab_smem()
{
    return sizeof(float2) * kBox * R + sizeof(float) * rec_floats<WNC>() + sizeof(float2) * 9 * kBS +
           (HASB ? sizeof(float2) * kOwn * R : 0);
}

struct SlabArgs {  // shared-memory pointers and block facts, the same for the whole CTA
    C *sx;
    const float *inv;      // [z][y][x]
    const float *sw;       // wavenumber box (complex pairs when WNC)
    const C *tab;          // [axis][d + 1][12]
    const C *sb;           // b boxes, 12^3 each
    int vx, vy, vz;        // rows of the block inside the grid
    unsigned edge;         // bit 2a: block starts at the grid's low face of axis a, 2a + 1: holds the high face
    bool adj;
    float w;
};

// What a block's coefficients need: all PML values 1 (kReal: real coefficients), those of x only
// (kXint: the x part joins the y and z parts, and the imaginary parts stand still along x), or
// the general form.
enum Mode { kFull, kXint, kReal };

// One pass (forward: a, b, c ascending; backward: descending) over the block.
template <int R, bool WNC, bool HASB, Mode M, bool BACK>
__device__ __forceinline__ void slab_pass(const SlabArgs &A, const Op<float> &op)
{
    constexpr bool REAL = M == kReal;
    const int lane = threadIdx.x & 31, wz = threadIdx.x >> 5;
    const int u = lane & 3, v = (lane >> 2) & 3, h = lane >> 4;
    const bool own_c = h == 0;       // the centre line belongs to half 0
    const float hz = own_c ? 1.f : 0.f;
    // slots: 0, 2 corner lines, 1 z face, 3 y face, 4 centre line; index 0 for dx = 0, 1 for dx = +-1
    const int dzh = h ? 1 : -1;
    const int dy[kNS] = {-1, 0, 1, dzh, 0}, dz[kNS] = {dzh, dzh, dzh, 0, 0};
    const float kx0[kNS] = {op.w3a2, op.xz, op.w3a2, op.xy, hz * op.wn_x};
    const float kx1[kNS] = {-op.w3a2, -op.xz, -op.w3a2, -op.xy, hz * op.pml_x};
    const float ky0[kNS] = {-op.yz, op.yz, -op.yz, op.pml_y, hz * op.wn_y};
    const float ky1[kNS] = {-op.w3a2, op.w3a2, -op.w3a2, -op.xy, hz * op.xy};
    const float kz0[kNS] = {-op.yz, op.pml_z, -op.yz, op.yz, hz * op.wn_z};
    const float kz1[kNS] = {-op.w3a2, -op.xz, -op.w3a2, op.w3a2, hz * op.xz};
    const float wm0[kNS] = {-(float)kWM3, -(float)kWM2, -(float)kWM3, -(float)kWM2, hz * op.wn_c};
    const float wm1[kNS] = {-(float)kWM4, -(float)kWM3, -(float)kWM4, -(float)kWM3, -hz * (float)kWM2};
    const float ki0[kNS] = {op.kint[6], op.kint[3], op.kint[6], op.kint[2], hz * op.kint[0]};
    const float ki1[kNS] = {op.kint[7], op.kint[5], op.kint[7], op.kint[4], hz * op.kint[1]};
    auto wn_at = [&](int e) {
        if constexpr (WNC) return reinterpret_cast<const C *>(A.sw)[e];
        else return mk<float>(A.sw[e], 0.f);
    };

#pragma unroll 1
    for (int cc = 0; cc < 3; ++cc) {
        const int c = BACK ? 2 - cc : cc;
        const int lz = c + 3 * wz;
#pragma unroll 1
        for (int bb = 0; bb < 3; ++bb) {
            const int b = BACK ? 2 - bb : bb;
            const int ly = b + 3 * v;
            // lines: offsets in the box of the point at box column 0
            int lo[kNS];
#pragma unroll
            for (int s = 0; s < kNS; ++s) lo[s] = kPlane * (1 + lz + dz[s]) + row_off(1 + b + dy[s]) + 44 * v;
            const bool vrow = ly < A.vy && lz < A.vz;
            C yz0[kNS], yz1[kNS];  // y and z parts of the coefficients
            if constexpr (!REAL) {
                const C *ty = A.tab + 4 * kBS + ly, *tz = A.tab + 7 * kBS + lz;
#pragma unroll
                for (int s = 0; s < kNS; ++s) {
                    const C yv = ty[kBS * dy[s]], zv = tz[kBS * dz[s]];
                    yz0[s] = cscale<kPK>(ky0[s], yv);
                    fma_rc<kPK>(yz0[s], kz0[s], zv);
                    yz1[s] = cscale<kPK>(ky1[s], yv);
                    fma_rc<kPK>(yz1[s], kz1[s], zv);
                    if constexpr (M == kXint) {  // X = 1, 2, 1
                        yz0[s].re = fmaf(2.f, kx0[s], yz0[s].re);
                        yz1[s].re += kx1[s];
                    }
                }
            }
            float ml[kNS];  // edge blocks: 0 for lines outside the grid
            if (A.edge) {
                const bool jl = (A.edge & 4u) && ly == 0, jh = (A.edge & 8u) && ly == A.vy - 1;
                const bool kl = (A.edge & 16u) && lz == 0, kh = (A.edge & 32u) && lz == A.vz - 1;
#pragma unroll
                for (int s = 0; s < kNS; ++s)
                    ml[s] = (dy[s] < 0 && jl) || (dy[s] > 0 && jh) || (dz[s] < 0 && kl) || (dz[s] > 0 && kh) ? 0.f : 1.f;
            }
            // the window: box columns 3u + a .. 3u + a + 2 of every line, and its wavenumbers
            C W[R][kNS][3], wv[kNS][3];
            const int col0 = 3 * u + (BACK ? 2 : 0);
#pragma unroll
            for (int s = 0; s < kNS; ++s)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
#pragma unroll
                    for (int r = 0; r < R; ++r) W[r][s][d] = A.sx[r * kBox + lo[s] + col0 + d];
                    if (!A.adj) wv[s][d] = wn_at(lo[s] + col0 + d);
                }
#pragma unroll
            for (int aa = 0; aa < 3; ++aa) {
                const int a = BACK ? 2 - aa : aa;
                const int lx = a + 3 * u;
                const int re = lx + kBS * (ly + kBS * lz);
                const float winv = A.w * A.inv[re];
                if (A.adj) {  // the row's own wavenumber for every offset
                    const C wc = wn_at(lo[kNS - 1] + 1 + lx);
#pragma unroll
                    for (int s = 0; s < kNS; ++s)
#pragma unroll
                        for (int d = 0; d < 3; ++d) wv[s][d] = wc;
                }
                const bool valid = vrow && lx < A.vx;
                C cf[kNS][3];
                if constexpr (REAL) {
#pragma unroll
                    for (int s = 0; s < kNS; ++s)
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                            cf[s][d].re = d == 1 ? fmaf(wm0[s], wv[s][d].re, ki0[s]) : fmaf(wm1[s], wv[s][d].re, ki1[s]);
                } else {
                    C X[3];
                    if constexpr (M == kFull) {
#pragma unroll
                        for (int d = 0; d < 3; ++d) X[d] = A.tab[kBS * d + lx];
                    }
#pragma unroll
                    for (int s = 0; s < kNS; ++s)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            C t = d == 1 ? yz0[s] : yz1[s];
                            if constexpr (M == kFull) fma_rc<kPK>(t, d == 1 ? kx0[s] : kx1[s], X[d]);
                            const float wm = d == 1 ? wm0[s] : wm1[s];
                            if constexpr (WNC) fma_rc<kPK>(t, wm, wv[s][d]);
                            else t.re = fmaf(wm, wv[s][d].re, t.re);
                            cf[s][d] = t;
                        }
                    if (A.edge) {
                        const float mxl = (A.edge & 1u) && lx == 0 ? 0.f : 1.f;
                        const float mxh = (A.edge & 2u) && lx == A.vx - 1 ? 0.f : 1.f;
#pragma unroll
                        for (int s = 0; s < kNS; ++s) {
                            cf[s][0] = cscale<kPK>(ml[s] * mxl, cf[s][0]);
                            cf[s][1] = cscale<kPK>(ml[s], cf[s][1]);
                            cf[s][2] = cscale<kPK>(ml[s] * mxh, cf[s][2]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    // a.x over the lane's lines: one partial sum per column
                    C p[3], q[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        p[d] = cscale<kPK>(cf[0][d].re, W[r][0][d]);
                        if constexpr (!REAL) q[d] = cscale<kPK>(cf[0][d].im, W[r][0][d]);
                    }
#pragma unroll
                    for (int s = 1; s < kNS; ++s)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            fma_rc<kPK>(p[d], cf[s][d].re, W[r][s][d]);
                            if constexpr (!REAL) fma_rc<kPK>(q[d], cf[s][d].im, W[r][s][d]);
                        }
                    C t = cadd<kPK>(cadd<kPK>(p[0], p[1]), p[2]);
                    if constexpr (!REAL) {
                        const C qs = cadd<kPK>(cadd<kPK>(q[0], q[1]), q[2]);
                        t = mk<float>(t.re - qs.im, t.im + qs.re);
                    }
                    t.re += __shfl_xor_sync(0xffffffffu, t.re, 16);
                    t.im += __shfl_xor_sync(0xffffffffu, t.im, 16);
                    C bv = mk<float>(0.f, 0.f);
                    if constexpr (HASB) bv = A.sb[r * kOwn + re];
                    C d1 = winv * (bv - t);
                    if (!valid) d1 = mk<float>(0.f, 0.f);
                    const C d2 = mk<float>(d1.im, -d1.re);
#pragma unroll
                    for (int s = 0; s < kNS; ++s)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            fma_rc<kPK>(W[r][s][d], cf[s][d].re, d1);
                            if constexpr (!REAL) fma_rc<kPK>(W[r][s][d], cf[s][d].im, d2);
                        }
                }
                if (aa < 2) {
                    // shift the window by one column: the column left goes to the neighbour in u; at the
                    // pencil's ends it goes to the box, and the entering one comes from it
                    const bool in_end = u == (BACK ? 0 : 3), out_end = u == (BACK ? 3 : 0);
                    const int cin = BACK ? 1 - aa : 12 + aa;
                    const int cout = BACK ? 13 - aa : aa;
#pragma unroll
                    for (int s = 0; s < kNS; ++s) {
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            C *row = A.sx + r * kBox + lo[s];
                            const C leave = W[r][s][BACK ? 2 : 0];
                            if (out_end && (s < kNS - 1 || own_c)) row[cout] = leave;
                            C in;
                            if constexpr (BACK) {
                                in.re = __shfl_up_sync(0xffffffffu, leave.re, 1);
                                in.im = __shfl_up_sync(0xffffffffu, leave.im, 1);
                            } else {
                                in.re = __shfl_down_sync(0xffffffffu, leave.re, 1);
                                in.im = __shfl_down_sync(0xffffffffu, leave.im, 1);
                            }
                            if (in_end) in = row[cin];
                            if constexpr (BACK) {
                                W[r][s][2] = W[r][s][1];
                                W[r][s][1] = W[r][s][0];
                                W[r][s][0] = in;
                            } else {
                                W[r][s][0] = W[r][s][1];
                                W[r][s][1] = W[r][s][2];
                                W[r][s][2] = in;
                            }
                        }
                        if (!A.adj) {
                            if constexpr (BACK) {
                                wv[s][2] = wv[s][1];
                                wv[s][1] = wv[s][0];
                                wv[s][0] = wn_at(lo[s] + lx - 1);
                            } else {
                                wv[s][0] = wv[s][1];
                                wv[s][1] = wv[s][2];
                                wv[s][2] = wn_at(lo[s] + lx + 3);
                            }
                        }
                    }
                }
            }
            // back to the box (the pencils' columns tile the lines; the ends were stored above)
            const int colw = 3 * u + (BACK ? 0 : 2);
#pragma unroll
            for (int s = 0; s < kNS; ++s)
                if (s < kNS - 1 || own_c) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int d = 0; d < 3; ++d) A.sx[r * kBox + lo[s] + colw + d] = W[r][s][d];
                }
            __syncwarp();
        }
        __syncthreads();  // the slabs meet
    }
}

// Entry e of a block's tables [axis][d + 1][12]: X[d], Y[d], Z[d] of the block's rows (forward:
// xi_lo, sum, xi_hi at the row; adjoint: the conjugated xi_hi of the row before, sum, xi_lo of the
// row after), zero outside the grid.
__device__ __forceinline__ C table_value(const Op<float> &op, bool adj, int bi0, int bj0, int bk0, int e)
{
    const int p = e % kBS, d = (e / kBS) % 3, ax = e / (3 * kBS);
    const int pos = (ax == 0 ? bi0 : ax == 1 ? bj0 : bk0) + p;
    const int n = ax == 0 ? op.nx : ax == 1 ? op.ny : op.nz;
    if (pos >= n) return mk<float>(0.f, 0.f);
    C t;
    if (d == 1) t = op.tab[op.sum[ax] + pos + 1];
    else if (!adj) t = op.tab[(d == 0 ? op.lo[ax] : op.hi[ax]) + pos + 1];
    else t = d == 0 ? op.tab[op.hi[ax] + pos] : op.tab[op.lo[ax] + pos + 2];
    return adj ? cconj(t) : t;
}

// The records of all blocks: 1/||a_i||^2 from the rows' coefficients (forward: of the neighbours
// inside the grid; adjoint: of all 27), and the wavenumber box (adjoint with a complex
// wavenumber: conjugated).  One CTA per block, once per operator; three threads per x line of rows,
// one per dz: the coefficients of one (dy, dz) line at a time, the partial sums of the 12 rows in
// registers, the three parts added in shared memory.
constexpr int kPackT = 448;
template <bool WNC>
__global__ void __launch_bounds__(kPackT) slab_pack_kernel(const __grid_constant__ Op<float> op, int adj, int NI, int NJ,
                                                           float *__restrict__ out)
{
    constexpr int kRec = rec_floats<WNC>(), W = WNC ? 2 : 1;
    __shared__ __align__(16) float sw[kBox * W];
    __shared__ C tab[9 * kBS];
    __shared__ float part[2][kBS][kBS * kBS];
    const int tid = threadIdx.x;
    const int Ib = blockIdx.x % NI, Jb = (blockIdx.x / NI) % NJ, Kb = blockIdx.x / (NI * NJ);
    const int bi0 = kBS * Ib, bj0 = kBS * Jb, bk0 = kBS * Kb;
    float *rec = out + (long long)blockIdx.x * kRec;
    if (tid < 9 * kBS) tab[tid] = table_value(op, adj != 0, bi0, bj0, bk0, tid);
    for (int e = tid; e < kBox * W; e += kPackT) sw[e] = 0.f;
    __syncthreads();
    {
        const int l = tid & 15, gi = bi0 - 1 + l;
        for (int rw = tid >> 4; rw < kBP * kBP; rw += kPackT / 16) {
            const int lj = rw % kBP, lk = rw / kBP, gj = bj0 - 1 + lj, gk = bk0 - 1 + lk;
            if (l < kBP && gi >= 0 && gi < op.nx && gj >= 0 && gj < op.ny && gk >= 0 && gk < op.nz) {
                const long long g = gi + op.sy * gj + op.sz * gk;
                const int e = kPlane * lk + row_off(lj) + l;
                sw[W * e] = op.wn[g];
                if constexpr (WNC) sw[W * e + 1] = op.wni ? (adj ? -op.wni[g] : op.wni[g]) : 0.f;
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < kBox * W; e += kPackT) rec[kOwn + e] = sw[e];
    const int third = tid / (kBS * kBS), line0 = tid % (kBS * kBS);
    const int ly = line0 % kBS, lz = line0 / kBS, j = bj0 + ly, k = bk0 + lz;
    const bool vrow = j < op.ny && k < op.nz;
    const int vx = min(kBS, op.nx - bi0);
    float nrm[kBS];
#pragma unroll
    for (int i = 0; i < kBS; ++i) nrm[i] = 0.f;
    if (vrow && third < 3) {
        const int ctr = kPlane * (lz + 1) + row_off(ly + 1) + 1;
#pragma unroll 1
        for (int dy = -1; dy <= 1; ++dy) {
            const int dz = third - 1;
            const bool in = j + dy >= 0 && j + dy < op.ny && k + dz >= 0 && k + dz < op.nz;
            if (!in && !adj) continue;
            // class constants of the line: index 0 for dx = 0, 1 for dx = +-1
            float kx0, kx1, ky0, ky1, kz0, kz1, w0, w1;
            if (dy != 0 && dz != 0) {
                kx0 = op.w3a2, ky0 = kz0 = -op.yz, w0 = -(float)kWM3;
                kx1 = ky1 = kz1 = -op.w3a2, w1 = -(float)kWM4;
            } else if (dy != 0) {
                kx0 = op.xy, ky0 = op.pml_y, kz0 = op.yz, w0 = -(float)kWM2;
                kx1 = ky1 = -op.xy, kz1 = op.w3a2, w1 = -(float)kWM3;
            } else if (dz != 0) {
                kx0 = op.xz, ky0 = op.yz, kz0 = op.pml_z, w0 = -(float)kWM2;
                kx1 = kz1 = -op.xz, ky1 = op.w3a2, w1 = -(float)kWM3;
            } else {
                kx0 = op.wn_x, ky0 = op.wn_y, kz0 = op.wn_z, w0 = op.wn_c;
                kx1 = op.pml_x, ky1 = op.xy, kz1 = op.xz, w1 = -(float)kWM2;
            }
            const C yv = tab[(4 + dy) * kBS + ly], zv = tab[(7 + dz) * kBS + lz];
            const C e0 = ky0 * yv + kz0 * zv, e1 = ky1 * yv + kz1 * zv;
            const int line = kPlane * (lz + 1 + dz) + row_off(ly + 1 + dy) + 1;
#pragma unroll
            for (int i = 0; i < kBS; ++i) {
                if (i < vx) {
#pragma unroll
                    for (int dd = 0; dd < 3; ++dd) {
                        const int e = adj ? ctr + i : line + i + dd - 1;
                        const C x = tab[dd * kBS + i];
                        C t = dd == 1 ? e0 : e1;
                        const float kx = dd == 1 ? kx0 : kx1, wm = dd == 1 ? w0 : w1;
                        fma_rc<kPK>(t, kx, x);
                        t.re = fmaf(wm, sw[W * e], t.re);
                        if constexpr (WNC) t.im = fmaf(wm, sw[W * e + 1], t.im);
                        const int gx = bi0 + i + dd - 1;
                        if (adj || (gx >= 0 && gx < op.nx)) nrm[i] += cabs2(t);
                    }
                }
            }
        }
    }
    if (third == 0 || third == 2) {
#pragma unroll
        for (int i = 0; i < kBS; ++i) part[third / 2][i][line0] = nrm[i];
    }
    __syncthreads();
    if (third != 1) return;
#pragma unroll
    for (int i = 0; i < kBS; ++i)
        rec[kBS * line0 + i] = vrow && i < vx ? 1.f / (part[0][i][line0] + nrm[i] + part[1][i][line0]) : 0.f;
}

// One block parity: dir 0 forward, 1 backward, 2 both passes.  R right-hand sides per CTA.
// SINGLE: the one problem's descriptor comes as a kernel parameter (one); otherwise a CTA finds
// its problem by a binary search over the per-parity prefix counts.
template <int R, bool WNC, bool HASB, bool SINGLE>
__global__ void __launch_bounds__(kNT, R == 1 ? 3 : 2) sweep_slab_kernel(const __grid_constant__ B8Prob<float> one,
                                                         const B8Prob<float> *__restrict__ probs,
                                                         const int *__restrict__ starts, int nprob, C *x,
                                                         const C *b, float w, const int *active, int par, int dir)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ B8Prob<float> ssp;
    __shared__ int s_pi;
    constexpr int kRec = rec_floats<WNC>();
    C *sx = reinterpret_cast<C *>(smem);
    float *srec = reinterpret_cast<float *>(sx + (size_t)R * kBox);
    C *tab = reinterpret_cast<C *>(srec + kRec);
    C *sb = tab + 9 * kBS;
    const int tid = threadIdx.x;

    int local = (int)blockIdx.x;
    if constexpr (!SINGLE) {
        const int *st0 = starts + par * (nprob + 1);
        if (tid == 0) {  // the problem whose CTA range holds this CTA
            int lo = 0, hi = nprob - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (st0[mid] <= (int)blockIdx.x) lo = mid;
                else hi = mid - 1;
            }
            s_pi = lo;
        }
        __syncthreads();
        const int *src = reinterpret_cast<const int *>(probs + s_pi);
        int *dst = reinterpret_cast<int *>(&ssp);
        for (int e = tid; e < (int)(sizeof(B8Prob<float>) / sizeof(int)); e += kNT) dst[e] = src[e];
        local -= st0[s_pi];
        __syncthreads();
    }
    const B8Prob<float> &sp = SINGLE ? one : ssp;
    const Op<float> &op = sp.op;
    const int blk = local / sp.ngrp, grp = local - blk * sp.ngrp;
    const int nI = (sp.NI - (par & 1) + 1) >> 1, nJ = (sp.NJ - ((par >> 1) & 1) + 1) >> 1;
    const int Ib = (par & 1) + 2 * (blk % nI), Jb = ((par >> 1) & 1) + 2 * ((blk / nI) % nJ);
    const int Kb = (par >> 2) + 2 * (blk / (nI * nJ));
    const int bi0 = kBS * Ib, bj0 = kBS * Jb, bk0 = kBS * Kb;
    const int s0 = grp * R;
    const int *ilo = sp.adj ? op.int_lo_a : op.int_lo_f, *ihi = sp.adj ? op.int_hi_a : op.int_hi_f;
    SlabArgs A;
    A.vx = min(kBS, op.nx - bi0);
    A.vy = min(kBS, op.ny - bj0);
    A.vz = min(kBS, op.nz - bk0);
    const bool xint = bi0 >= ilo[0] && bi0 + A.vx <= ihi[0];
    const bool yzint = bj0 >= ilo[1] && bj0 + A.vy <= ihi[1] && bk0 >= ilo[2] && bk0 + A.vz <= ihi[2];
    A.edge = (bi0 == 0 ? 1u : 0u) | (bi0 + kBS >= op.nx ? 2u : 0u) | (bj0 == 0 ? 4u : 0u) |
             (bj0 + kBS >= op.ny ? 8u : 0u) | (bk0 == 0 ? 16u : 0u) | (bk0 + kBS >= op.nz ? 32u : 0u);
    A.adj = sp.adj != 0;
    A.w = w;
    const float *rec = sp.rec + (long long)(Ib + sp.NI * (Jb + (long long)sp.NJ * Kb)) * kRec;
    A.sx = sx;
    A.inv = srec;
    A.sw = srec + kOwn;
    A.tab = tab;
    A.sb = sb;

    // The block's record and tables do not depend on the launch before.
    for (int e = tid; e < kRec / 4; e += kNT) blk_cp_async<16>(srec + 4 * e, rec + 4 * e, true);
    for (int e = tid; e < 9 * kBS; e += kNT) tab[e] = table_value(op, A.adj, bi0, bj0, bk0, e);
    // The next launch may start its own record copies; x, b and the flags wait for the launch before.
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    unsigned act = 0;  // bit r: column s0 + r of the problem takes part
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (s0 + r < sp.nrhs && (!active || active[sp.c0 + s0 + r])) act |= 1u << r;
    if (!act) {  // uniform over the CTA
        blk_cp_async_wait_all();
        return;
    }
    // x (and b of the block's own rows), zero outside the grid: half-warp q copies box rows q,
    // q + kNT / 16, .. of every plane, lane l point l of the row.  The offsets inside a plane are fixed per
    // thread, so a plane costs a few instructions per copy.
    constexpr int kT = (kBP * 16 + kNT - 1) / kNT;  // box rows per half-warp and plane
    const int l = tid & 15, q8 = tid >> 4;
    const int gi = bi0 - 1 + l;
    const bool lin = l < kBP && gi >= 0 && gi < op.nx, own_x = l >= 1 && l <= kBS;
    const long long xcol = sp.col0 + s0 * sp.cstride;
    long long goff[kT];  // offset of the thread's point inside a grid plane
    int soff[kT], ioff[kT];
    bool rin[kT], own[kT];
#pragma unroll
    for (int t = 0; t < kT; ++t) {
        const int lj = q8 + (kNT / 16) * t, gj = bj0 - 1 + lj;
        rin[t] = lin && lj < kBP && gj >= 0 && gj < op.ny;
        goff[t] = rin[t] ? gi + op.sy * gj : 0;
        soff[t] = row_off(lj) + l;
        own[t] = own_x && lj >= 1 && lj <= kBS;
        ioff[t] = (l - 1) + kBS * (lj - 1);
    }
    if (l < kBP) {
        for (int lk = 0; lk < kBP; ++lk) {
            const int gk = bk0 - 1 + lk;
            const bool kin = gk >= 0 && gk < op.nz, own_z = lk >= 1 && lk <= kBS;
            const long long zo = xcol + (kin ? op.sz * gk : 0);
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                if (q8 + (kNT / 16) * t >= kBP) break;
                const bool in = kin && rin[t];
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (act & (1u << r)) {
                        blk_cp_async<8>(sx + r * kBox + kPlane * lk + soff[t], x + zo + r * sp.cstride + goff[t], in);
                        if constexpr (HASB) {
                            if (own[t] && own_z)
                                blk_cp_async<8>(sb + r * kOwn + kBS * kBS * (lk - 1) + ioff[t],
                                                b + zo + r * sp.cstride + goff[t], in);
                        }
                    }
            }
        }
    }
    blk_cp_async_wait_all();
    __syncthreads();

    auto both = [&](auto fwd, auto bwd) {
        if (dir != 1) fwd();
        if (dir != 0) bwd();
    };
    if (!WNC && xint && yzint)
        both([&] { slab_pass<R, WNC, HASB, kReal, false>(A, op); }, [&] { slab_pass<R, WNC, HASB, kReal, true>(A, op); });
    else if (xint)
        both([&] { slab_pass<R, WNC, HASB, kXint, false>(A, op); }, [&] { slab_pass<R, WNC, HASB, kXint, true>(A, op); });
    else
        both([&] { slab_pass<R, WNC, HASB, kFull, false>(A, op); }, [&] { slab_pass<R, WNC, HASB, kFull, true>(A, op); });

    // write the boxes back (halo included), points inside the grid only, as staged
    if (lin) {
        const int k0 = bk0 == 0 ? 1 : 0, k1 = min(kBP, op.nz - bk0 + 1);
        C *xw = x + xcol + op.sz * (bk0 - 1);
#pragma unroll 2
        for (int lk = k0; lk < k1; ++lk) {
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                if (!rin[t]) continue;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (act & (1u << r))
                        xw[op.sz * lk + r * sp.cstride + goff[t]] = sx[r * kBox + kPlane * lk + soff[t]];
            }
        }
    }
}

template <int R, bool WNC, bool HASB, bool SINGLE>
int launch_one(const B8Prob<float> &one, const B8Prob<float> *probs, const int *starts, int nprob, long long nctas,
               C *x, const C *b, float w, const int *active, int par, int dir, bool chained, cudaStream_t st)
{
    constexpr size_t smem = slab_smem<R, WNC, HASB>();
    static_assert(smem + sizeof(B8Prob<float>) + 16 <= 232448, "slab sweep configuration exceeds shared memory");
    auto *kern = sweep_slab_kernel<R, WNC, HASB, SINGLE>;
    static std::atomic<unsigned long long> attr_set{0};  // bit per device
    int dev = 0;
    H3D_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev > 63 || !(attr_set.load() & bit)) {
        H3D_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set.fetch_or(bit);
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nctas);
    cfg.blockDim = dim3(kNT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    H3D_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, one, probs, starts, nprob, x, b, w, active, par, dir));
    return H3D_OK;
}

template <int R, bool WNC, bool HASB, typename... Args>
int launch_s(bool single, const Args &...a)
{
    return single ? launch_one<R, WNC, HASB, true>(a...) : launch_one<R, WNC, HASB, false>(a...);
}

template <int R, typename... Args>
int launch_r(bool wnc, bool hasb, bool single, const Args &...a)
{
    if (wnc) return hasb ? launch_s<R, true, true>(single, a...) : launch_s<R, true, false>(single, a...);
    return hasb ? launch_s<R, false, true>(single, a...) : launch_s<R, false, false>(single, a...);
}

}  // namespace

size_t slab_record_bytes(int NI, int NJ, int NK, bool wnc)
{
    return sizeof(float) * (size_t)NI * NJ * NK * (wnc ? rec_floats<true>() : rec_floats<false>());
}

int launch_slab_pack(const Op<float> &op, bool adj, int NI, int NJ, int NK, bool wnc, float *rec, cudaStream_t st)
{
    const unsigned nb = (unsigned)(NI * NJ * NK);
    if (wnc) slab_pack_kernel<true><<<nb, kPackT, 0, st>>>(op, adj ? 1 : 0, NI, NJ, rec);
    else slab_pack_kernel<false><<<nb, kPackT, 0, st>>>(op, adj ? 1 : 0, NI, NJ, rec);
    H3D_CUDA_TRY(cudaGetLastError());
    return H3D_OK;
}

int launch_slab(int r, bool wnc, const B8Prob<float> &one, const B8Prob<float> *probs, const int *starts, int nprob,
                long long nctas, C *x, const C *b, float w, const int *active, int par, int dir, bool chained,
                cudaStream_t st)
{
    const bool single = nprob == 1, hasb = b != nullptr;
#define H3D_SLAB(R) launch_r<R>(wnc, hasb, single, one, probs, starts, nprob, nctas, x, b, w, active, par, dir, chained, st)
    if (r == 1) return H3D_SLAB(1);
    if (r == 2) return H3D_SLAB(2);
#undef H3D_SLAB
    set_error("slab sweep with %d right-hand sides per CTA is not built", r);
    return H3D_ERR_BAD_ARG;
}

}  // namespace h3d
