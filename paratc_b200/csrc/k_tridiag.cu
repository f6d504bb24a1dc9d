// k_tridiag.cu -- wall-normal tridiagonal solves on B200.
//
// Both the implicit Helmholtz systems (I - beta*Lyy) du = Rhs of clcU1Hat /
// clcU2Hat / clcU3Hat / clcScalar (src/m_TScheme.f90:365-506) and the
// spectral Poisson systems (Lyy + lambda_x + lambda_z) phi = f of clcPPE
// (src/m_Poisson.f90:383-430) are many independent tridiagonal systems along
// y, one per (x, z) column.  The reference sweeps them with the serial Thomas
// algorithm InverseTridiagonal (src/m_Tools.f90:224-251), and across ranks
// with the reduced-system ("PaScaL") Thomas of clcPPE_x1_reduce
// (src/m_Poisson.f90:457-695).
//
// The matrices never depend on the column's data, only on the row (the
// Helmholtz systems, per step) or on the row and the wavenumber pair (the
// Poisson systems, per context).  So the Thomas pivots are computed apart
// from the solves, and a solve is a chain of multiply-adds per column with
// its loads issued ahead: k_helm (pivots per step, k_helm_factors) and
// k_ys_pair (pivots per context, k_pois_factors).  The
// partitioned reduced-system solver (part_eliminate / part_reduced /
// k_ysolve) computes its pivots in place; the allocation-free Poisson entry
// point uses it because it has no room to keep pivots between calls.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace ptc {

// local elimination of one partition of MR rows (MR >= 3), the modified
// Thomas sweep of src/m_Poisson.f90:496-537 in registers.  On exit row 0 reads
// a0*x_prev + x0 + c0*x_last = f0, row r (1..MR-2) a_r*x0 + x_r + c_r*x_last
// = f_r, row MR-1 a*x0 + x_last + c*x_next = f.  MR is a compile-time
// constant so that every register array index is static; rows past ny are
// identity rows (a = c = f = 0, b = 1), decoupled from the system.
template <int MAXM, int NC, class GetB>
__device__ __forceinline__ void part_eliminate(double (&a)[MAXM], double (&c)[MAXM], double (&f)[MAXM][NC],
                                               const GetB& getb) {
    {
        const double b0 = getb(0), b1 = getb(1);
        a[0] = a[0] / b0;
        c[0] = c[0] / b0;
        a[1] = a[1] / b1;
        c[1] = c[1] / b1;
#pragma unroll
        for (int q = 0; q < NC; q++) {
            f[0][q] = f[0][q] / b0;
            f[1][q] = f[1][q] / b1;
        }
    }
#pragma unroll
    for (int r = 2; r < MAXM; r++) {
        const double rr = 1.0 / (getb(r) - a[r] * c[r - 1]);
#pragma unroll
        for (int q = 0; q < NC; q++) f[r][q] = rr * (f[r][q] - a[r] * f[r - 1][q]);
        c[r] = rr * c[r];
        a[r] = -(rr * a[r] * a[r - 1]);
    }
#pragma unroll
    for (int r = MAXM - 3; r >= 1; r--) {
#pragma unroll
        for (int q = 0; q < NC; q++) f[r][q] = f[r][q] - c[r] * f[r + 1][q];
        a[r] = a[r] - c[r] * a[r + 1];
        c[r] = -(c[r] * c[r + 1]);
    }
    {
        const double rr = 1.0 / (1.0 - a[1] * c[0]);
#pragma unroll
        for (int q = 0; q < NC; q++) f[0][q] = rr * (f[0][q] - c[0] * f[1][q]);
        a[0] = rr * a[0];
        c[0] = -(rr * c[0] * c[1]);
    }
}

// writes the two reduced rows of this partition, solves the reduced systems
// (one column per lane of warp 0), returns x_first / x_last of the partition
template <int MAXM, int NC>
__device__ __forceinline__ void part_reduced(int P, int w, int lane, const double (&a)[MAXM], const double (&c)[MAXM],
                                             const double (&f)[MAXM][NC], double* sm, double (&xf)[NC], double (&xl)[NC]) {
    const int n2 = 2 * P;
    double* RA = sm;                          // [n2][32]
    double* RC = RA + n2 * 32;                // [n2][32]
    double* RW = RC + n2 * 32;                // [n2][32] Thomas factors
    double* RF = RW + n2 * 32;                // [n2][NC][32]
    const double al = a[MAXM - 1], cl = c[MAXM - 1];
    double fl[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) fl[q] = f[MAXM - 1][q];
    const int r0 = 2 * w, r1 = 2 * w + 1;
    RA[r0 * 32 + lane] = a[0];
    RC[r0 * 32 + lane] = c[0];
    RA[r1 * 32 + lane] = al;
    RC[r1 * 32 + lane] = cl;
#pragma unroll
    for (int q = 0; q < NC; q++) {
        RF[(r0 * NC + q) * 32 + lane] = f[0][q];
        RF[(r1 * NC + q) * 32 + lane] = fl[q];
    }
    __syncthreads();
    if (w == 0) {
        // unit-diagonal Thomas (InverseTridiagonal, src/m_Tools.f90:224-251)
        double vecm = 1.0;
        double fp[NC];
#pragma unroll
        for (int q = 0; q < NC; q++) fp[q] = RF[(0 * NC + q) * 32 + lane];
        for (int r = 1; r < n2; r++) {
            const double arr = RC[(r - 1) * 32 + lane] / vecm;
            const double ar = RA[r * 32 + lane];
            RW[r * 32 + lane] = arr;
            vecm = 1.0 - ar * arr;
#pragma unroll
            for (int q = 0; q < NC; q++) {
                const double v = (RF[(r * NC + q) * 32 + lane] - ar * fp[q]) / vecm;
                RF[(r * NC + q) * 32 + lane] = v;
                fp[q] = v;
            }
        }
        for (int r = n2 - 2; r >= 0; r--) {
            const double arr = RW[(r + 1) * 32 + lane];
#pragma unroll
            for (int q = 0; q < NC; q++) {
                const double v = RF[(r * NC + q) * 32 + lane] - arr * fp[q];
                RF[(r * NC + q) * 32 + lane] = v;
                fp[q] = v;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NC; q++) {
        xf[q] = RF[(r0 * NC + q) * 32 + lane];
        xl[q] = RF[(r1 * NC + q) * 32 + lane];
    }
}

// diagonal of row r of a partition starting at Fortran row s
struct PoisDiag {
    const double* ac2ph;
    double lam;
    int s, ny;
    bool dc;  // kx = kz = 0: row 1 is the identity
    __device__ __forceinline__ double operator()(int r) const {
        const int jc = s + r;
        if (jc > ny || (dc && jc == 1)) return 1.0;
        return __ldg(&ac2ph[jc]) + lam;
    }
};

// ---------------------------------------------------------------------------
// Helmholtz: comp 0 ux (clcU1Hat), 1 uy (clcU2Hat), 2 uz (clcU3Hat),
// 3 scalar (clcScalar); u(jc) += du(jc) with (I - beta*Lyy) du = Rhs
// (src/m_TScheme.f90:365-506).  The matrices depend on the row only, so
// their pivots are computed once per step by k_helm_factors.  Every column is
// eliminated from both walls at once, as in the spectral solve below: rows
// 1 .. h = ny/2 upwards, rows ny .. h+1 downwards, and for row j of either
// half the table holds r = 1 / pivot, MP = r times the coupling to the row
// swept before, MN = r times the coupling to the row after, so that a row's
// link of the chain is one FMA:
//   F(j) = r (Rhs + add) - MP F(before),   x(j) = F(j) - MN x(after).
// A work item is 32 adjacent columns of one component; a CTA is two warps,
// one per wall, and walks items with a stride of its grid.  A warp's half of
// the right-hand sides sits in its part of shared memory in sweep order
// (copied there with cp.async; F replaces it row by row, so no forward-swept
// value goes through memory), the sweep back reads u one chunk ahead, writes
// u + x, and copies the next item's rows into the slots it has read.  The
// columns are numbered through the planes (k nx + i), so that no lane idles
// on a narrow or ragged nx.
// uy and the scalar also get the ghost values that
// SetBC_and_UpdateHaloForPrSrc / _scalar give them.
// ---------------------------------------------------------------------------
namespace {
constexpr int HY_U = 8;  // rows a sweep reads ahead of its chain; 4 in the tuner's second variant
constexpr int HELM_NVAR = 2;
__host__ __device__ inline int helm_stride(int ny) { return 3 * (ny + 2); }
// shared memory of one wall's half of an item, hm rows: the columns, (r, MP)
// pairs, MN
__host__ __device__ inline int helm_half(int hm, int vsize, int wsize) {
    const int b = hm * 32 * vsize + 3 * ((hm + 1) & ~1) * wsize;
    return (b + 127) & ~127;
}
template <class W>
struct W2;
template <>
struct W2<double> {
    using T = double2;
};
template <>
struct W2<float> {
    using T = float2;
};
}  // namespace

// 16-byte copy that bypasses registers
__device__ __forceinline__ void cpa16(void* sdst, const void* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}

// V: storage of the fields.  W: the sweeps' arithmetic, double (FP64 in every
// form), or float for the FP32 storage form's third launch shape, whose rows
// are stored in float anyway.  G: the block this CTA works as (OwnGrid, or
// SubGrid in a grouped launch).
template <class V, int U, class W, class G>
__device__ __forceinline__ void helm_body(const G& grid, const DConst& cst, const DCoef* __restrict__ coef, int ncomp,
                                          const FieldSet<V>& fl, const double* __restrict__ duy_ym,
                                          const double* __restrict__ uy_ym, const double* __restrict__ facs) {
    using WP = typename W2<W>::T;
    constexpr int VL = 16 / (int)sizeof(V), LPR = 32 / VL, RPW = 32 / LPR;  // a copy's columns, lanes per row, rows per pass
    extern __shared__ __align__(128) unsigned char hm_raw[];
    __shared__ WP xch[2][2][32];  // [item parity][wall][lane]: the last row's F and MN
    const int nx = cst.nx, ny = cst.ny, nz = cst.nz;
    const int end = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = ny >> 1, nt = end ? ny - h : h, hm = ny - h;
    unsigned char* my = hm_raw + (size_t)end * helm_half(hm, sizeof(V), sizeof(W));
    V* const sd = reinterpret_cast<V*>(my);
    WP* const srp = reinterpret_cast<WP*>(my + (size_t)hm * 32 * sizeof(V));
    W* const smn = reinterpret_cast<W*>(srp + ((hm + 1) & ~1));
    const int dj = end ? -1 : 1, jw = end ? ny : 1;  // row i of the sweep is row jw + dj i
    const ptrdiff_t gstep = (ptrdiff_t)dj * nx;
    const int ncols = nx * nz, nct = (ncols + 31) / 32, nitems = nct * ncomp;
    const int stride = (int)grid.gx();
    const size_t pl = (size_t)cst.nyt * nx;
    auto rhs_of = [&](int comp) { return comp == 0 ? fl.rx : comp == 1 ? fl.ry : comp == 2 ? fl.rz : fl.rc; };
    auto u_of = [&](int comp) { return comp == 0 ? fl.ux : comp == 1 ? fl.uy : comp == 2 ? fl.uz : fl.sc; };
    // copies: lane = (row of a pass, VL adjacent columns)
    const int lr = lane / LPR, lc = (lane % LPR) * VL;
    V* const cdst = sd + lr * 32 + lc;
    const V* csrc = nullptr;  // row lr of the item's columns lc ..
    bool cval = false;
    auto aim = [&](int item) {
        const int c = item / nct, q = (item - c * nct) * 32 + lc;
        cval = q < ncols;
        const int k = q / nx;
        csrc = rhs_of(c) + (size_t)k * pl + (q - k * nx) + (size_t)jw * nx + lr * gstep;
    };
    auto copy_rows = [&](int i0, int n) {  // rows i0 .. i0 + n - 1, n <= U
        const V* src = csrc + i0 * gstep;
#pragma unroll
        for (int u = 0; u < U; u += RPW) {
            if (cval && u + lr < n) cpa16(cdst + (i0 + u) * 32, src);
            src += RPW * gstep;
        }
    };
    int item = (int)grid.x();
    if (item < nitems) aim(item);
    pdl_wait();
    if (item < nitems)
        for (int i0 = 0; i0 < nt; i0 += U) copy_rows(i0, min(U, nt - i0));
    const int nb = nt - 1, nf = nt / U * U, nbf = nb / U * U;
    int type = -1;
    for (int it = 0; item < nitems; item += stride, it++) {
        const int next = item + stride;
        if (next >= nitems) pdl_trigger();
        const int comp = item / nct;
        const int t = comp == 1 ? 1 : (comp == 3 ? 2 : 0);
        if (t != type) {  // this matrix's table, in sweep order
            type = t;
            const double* F = facs + (size_t)((coef->ns - 1) * 3 + t) * helm_stride(ny);
            for (int i = lane; i < nt; i += 32) {
                const int j = jw + dj * i;
                WP p;
                p.x = (W)F[(ny + 2) + j];
                p.y = (W)F[j];
                srp[i] = p;
                smn[i] = (W)F[2 * (ny + 2) + j];
            }
        }
        const int q = (item % nct) * 32 + lane, k = q / nx;
        const bool valid = q < ncols;
        const size_t col = (size_t)k * pl + (q - k * nx);
        V* const uc = u_of(comp) + col;
        const W add = comp == 0 ? (W)coef->rhsx_add : (W)0;
        // clcU2Hat: the row-1 value is the wall increment (kept in FP64)
        const bool v1 = comp == 1 && end == 0;
        const W a0 = v1 && valid ? (W)duy_ym[q] : (W)0;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncwarp();
        V* const s = sd + lane;
        W f = 0;
        // u is read on the way back: brought into L2 meanwhile
        const V* pf = uc + (ptrdiff_t)jw * nx;
        for (int i0 = 0; i0 < nf; i0 += U) {
            if (valid) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(pf));
                    pf += gstep;
                }
            }
            W g[U], mm[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const WP p = srp[i0 + u];
                g[u] = ((W)s[(i0 + u) * 32] + add) * p.x;
                mm[u] = p.y;
            }
            if (v1 && i0 == 0) g[0] = a0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                f = g[u] - mm[u] * f;
                s[(i0 + u) * 32] = (V)f;
            }
        }
        for (int i = nf; i < nt; i++) {
            const WP p = srp[i];
            f = (v1 && i == 0 ? a0 : ((W)s[i * 32] + add) * p.x) - p.y * f;
            s[i * 32] = (V)f;
        }
        WP mine;
        mine.x = f;
        mine.y = smn[nb];
        xch[it & 1][end][lane] = mine;
        __syncthreads();
        const WP o = xch[it & 1][end ^ 1][lane];
        W x = (f - mine.y * o.x) / ((W)1 - mine.y * o.y);
        // back to the wall: x(i) = F(i) - MN x(i+1), u += x
        V* up = uc + (ptrdiff_t)(jw + dj * nb) * nx;
        W un = 0;
        if (valid) {
            un = (W)*up + x;
            *up = (V)un;
        }
        for (int i = nb - 1; i >= nbf; i--) {
            x = (W)s[i * 32] - smn[i] * x;
            up -= gstep;
            if (valid) {
                un = (W)*up + x;
                *up = (V)un;
            }
        }
        V un0[U], un1[U];  // u of the chunk at hand and the one after it, in storage type
        auto ldu = [&](V (&X)[U], const V* p) {
#pragma unroll
            for (int u = U - 1; u >= 0; u--) {
                p -= gstep;
                if (valid) X[u] = *p;
            }
        };
        if (nbf > 0) ldu(un0, up);
        __syncwarp();
        if (next < nitems) {
            aim(next);
            copy_rows(nbf, nt - nbf);
        }
        for (int i0 = nbf - U; i0 >= 0; i0 -= U) {
            if (i0 > 0) ldu(un1, up - U * gstep);
            W d[U], mm[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                d[u] = (W)s[(i0 + u) * 32];
                mm[u] = smn[i0 + u];
            }
            __syncwarp();
            if (next < nitems) copy_rows(i0, U);
#pragma unroll
            for (int u = U - 1; u >= 0; u--) {
                x = d[u] - mm[u] * x;
                up -= gstep;
                un = (W)un0[u] + x;
                if (valid) *up = (V)un;
            }
#pragma unroll
            for (int u = 0; u < U; u++) un0[u] = un1[u];
        }
        // the wall rows: un holds u(1) or u(ny)
        if (comp == 1 && valid) {
            if (end == 0) uc[nx] = (V)uy_ym[q];
            else uc[(size_t)(ny + 1) * nx] = (V)((cst.flow_type == 1) ? cst.uybc_yp : 0.0);
        } else if (comp == 3 && valid) {
            if (end == 0) uc[0] = (V)(cst.sc_r1b * (double)un + cst.sc_r2b);
            else uc[(size_t)(ny + 1) * nx] = (V)(cst.sc_r1t * (double)un + cst.sc_r2t);
        }
    }
}

template <class V, int U, class W = double>
__global__ void __launch_bounds__(64, 8) k_helm(DConst cst, const DCoef* __restrict__ coef, int ncomp, FieldSet<V> fl,
                                                const double* __restrict__ duy_ym,
                                                const double* __restrict__ uy_ym, const double* __restrict__ facs) {
    helm_body<V, U, W>(OwnGrid{}, cst, coef, ncomp, fl, duy_ym, uy_ym, facs);
}

template <class V, int U, class W = double>
__global__ void __launch_bounds__(64, 8) k_helm_grp(const GrpTab<HelmArgs<V>>* __restrict__ t) {
    SubGrid g;
    const HelmArgs<V>& a = t->e[grp_member(t, g)];
    helm_body<V, U, W>(g, a.c, a.coef, a.ncomp, a.fl, a.duy_ym, a.uy_ym, a.fac);
}

// ---------------------------------------------------------------------------
// spectral y-solve of clcPPE_x1 (src/m_Poisson.f90:383-430) on the complex
// coefficients spec[(k*ny + j)*(nx/2+1) + kx].  The real and imaginary parts
// are two real right-hand sides of the same real matrix, so the array is
// treated as 2*(nx/2+1) real columns: lane pairs share kx and a warp reads
// 256 contiguous bytes per row.  The kx = kz = 0 system has its first row
// replaced by phi = 0 (src/m_Poisson.f90:399-404).
// ---------------------------------------------------------------------------
template <int MR>
__global__ void __launch_bounds__(512) k_ysolve(DConst cst, DMetric m, double* __restrict__ specd) {
    extern __shared__ double sm[];
    const int lane = threadIdx.x, w = threadIdx.y, P = blockDim.y;
    const int ny = cst.ny, ncol = 2 * (cst.nx / 2 + 1);
    const int cr = blockIdx.x * 32 + lane;
    const int kx = cr >> 1;
    const int k = blockIdx.y;
    const bool act = cr < ncol;
    const int s = w * MR + 1;
    const double lam = act ? __ldg(&m.wnx[kx]) + __ldg(&m.wnz[k]) : 0.0;
    const bool dc = (kx == 0 && k == 0);
    double* col = specd + (size_t)k * ny * ncol + (act ? cr : 0);
    double a[MR], c[MR], f[MR][1];
#pragma unroll
    for (int r = 0; r < MR; r++) {
        a[r] = 0.0; c[r] = 0.0; f[r][0] = 0.0;
        const int jc = s + r;
        if (jc <= ny && !(dc && jc == 1)) {
            a[r] = (jc == 1) ? 0.0 : __ldg(&m.am2ph[jc]);
            c[r] = (jc == ny) ? 0.0 : __ldg(&m.ap2ph[jc]);
            if (act) f[r][0] = col[(size_t)(jc - 1) * ncol];
        }
    }
    part_eliminate<MR, 1>(a, c, f, PoisDiag{m.ac2ph, lam, s, ny, dc});
    double xf[1], xl[1];
    part_reduced<MR, 1>(P, w, lane, a, c, f, sm, xf, xl);
    if (!act) return;
#pragma unroll
    for (int r = 0; r < MR; r++) {
        const int jc = s + r;
        if (jc <= ny) {
            double x;
            if (r == 0) x = xf[0];
            else if (r == MR - 1) x = xl[0];
            else x = f[r][0] - a[r] * xf[0] - c[r] * xl[0];
            col[(size_t)(jc - 1) * ncol] = x;
        }
    }
}

// ---------------------------------------------------------------------------
// Spectral y-solve with the factors computed once.  The Poisson matrices
// (am2ph, ac2ph + lambda_x(kx) + lambda_z(kz), ap2ph) depend on the mesh and
// the wavenumbers only, so their pivots are computed once per context.  Every
// system is eliminated from both walls at once: rows 1 .. h = ny/2 downwards
// from the lower wall, rows ny .. h+1 from the upper one,
//   lower:  x(j) = F(j) - c(j) r(j) x(j+1),  F(j) = r(j) (f(j) - a(j) F(j-1)),
//           r(j) = 1 / (b(j) - a(j) c(j-1) r(j-1)),
//   upper:  the same with a and c exchanged and the rows reversed,
// so that the two dependent chains of a column are half as long as the one
// of InverseTridiagonal (src/m_Tools.f90:224-251) and run side by side; the
// two equations that meet at rows h, h+1 give both unknowns, and the sweeps
// return to the walls.  Only r is kept: the multipliers a r and c r are one
// multiply off the chain.  lambda_z is even in kz, so the columns kz and
// nz - kz share their pivots: the table holds kz = 0 .. nz/2, blocks of YP_C
// modes kx, [kz][block][row][YP_C] -- a quarter of one FP64 factor pair per
// spectrum value.  The kx = kz = 0 system has row 1 replaced by phi = 0
// (b = 1, c = 0, f = 0; src/m_Poisson.f90:399-404).
// ---------------------------------------------------------------------------
namespace {
constexpr int YP_C = 8;  // complex columns of one kz in a work item: 128 bytes of a spectrum row
constexpr int YP_U = 8;  // rows a sweep reads ahead of its chain
__host__ __device__ inline int yp_blocks(int M1) { return (M1 + YP_C - 1) / YP_C; }

// esize-byte copy that bypasses registers (16: double2, 8: float2)
template <int N>
__device__ __forceinline__ void cpa(void* sdst, const void* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}

// shared memory of one wall's half of an item, hm rows: the two planes' boxes
// (with a float2 spectrum, whose rows are 64 bytes, the second box starts half
// a bank cycle after the first, so that a warp's two half-rows fall into
// different banks), the pivots, the two couplings
__host__ __device__ inline int yp_box(int hm, int esize) {
    const int b = hm * YP_C * esize;
    return esize == 8 && b % 128 == 0 ? b + 64 : b;
}
__host__ __device__ inline int yp_half(int hm, int esize) {
    const int b = 2 * yp_box(hm, esize) + (hm * YP_C + 2 * ((hm + 1) & ~1)) * (int)sizeof(double);
    return (b + 127) & ~127;
}
}  // namespace

// dc_here: column 0 is the kx = kz = 0 system (false for a z-slab rank
// whose modes start above kx = 0; m.wnx then starts at its first mode)
__global__ void k_pois_factors(int ny, int M1, int nz, DMetric m, double* __restrict__ fac, int dc_here) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= M1 * (nz / 2 + 1)) return;
    const int kz = q / M1, kx = q - kz * M1;
    const double wx = m.wnx[kx], wz = m.wnz[kz];
    const bool dc = dc_here && q == 0;
    double* r = fac + (size_t)(kz * yp_blocks(M1) + kx / YP_C) * ny * YP_C + kx % YP_C;
    const int h = ny >> 1;
    double vecm = dc ? 1.0 : __dadd_rn(__dadd_rn(m.ac2ph[1], wx), wz);
    // a pivot of 0 makes both sweeps leave phi = 0 in the pinned row
    r[0] = dc ? 0.0 : 1.0 / vecm;
    for (int jc = 2; jc <= h; jc++) {
        const double arr = ((dc && jc == 2) ? 0.0 : m.ap2ph[jc - 1]) / vecm;
        const double b = __dadd_rn(__dadd_rn(m.ac2ph[jc], wx), wz);
        vecm = __dsub_rn(b, __dmul_rn(m.am2ph[jc], arr));
        r[(size_t)(jc - 1) * YP_C] = 1.0 / vecm;
    }
    vecm = __dadd_rn(__dadd_rn(m.ac2ph[ny], wx), wz);
    r[(size_t)(ny - 1) * YP_C] = 1.0 / vecm;
    for (int jc = ny - 1; jc > h; jc--) {
        const double arr = m.am2ph[jc + 1] / vecm;
        const double b = __dadd_rn(__dadd_rn(m.ac2ph[jc], wx), wz);
        vecm = __dsub_rn(b, __dmul_rn(m.ap2ph[jc], arr));
        r[(size_t)(jc - 1) * YP_C] = 1.0 / vecm;
    }
}

// A work item is YP_C modes kx of the planes kz and nz - kz: 32 real columns
// (lane = plane, mode, real or imaginary part).  A CTA is two warps, one per
// wall, and walks items with a stride of its grid.  A warp's half of the
// columns and their pivots sits in its own part of shared memory in the order
// it sweeps them, copied there row by row with cp.async; while the sweep back
// leaves a row (the solution goes straight to memory) the next item's row is
// copied into the slot.  So a column crosses memory once each way, a row's
// link of the chain is a single FMA, and the warps of an SM's CTAs keep
// copies in flight all the time.
template <class S, class G>
__device__ __forceinline__ void ys_pair_body(const G& grid, int ny, int M1, int nz, const double* __restrict__ am2ph,
                                             const double* __restrict__ ap2ph, S* __restrict__ spec,
                                             const double* __restrict__ fac) {
    using R = decltype(S::x);
    constexpr int ES = (int)sizeof(S), ROW = YP_C * ES;  // bytes of a row of one plane
    extern __shared__ __align__(128) unsigned char yp_raw[];
    __shared__ double2 xch[2][2][32];  // [item parity][wall][lane]: the last row's F and its coupling
    const int end = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = ny >> 1, nt = end ? ny - h : h, hm = ny - h;
    const int box = yp_box(hm, ES);
    unsigned char* my = yp_raw + (size_t)end * yp_half(hm, ES);
    double* sr = reinterpret_cast<double*>(my + 2 * box);  // [hm][YP_C] pivots
    double* cp = sr + (size_t)hm * YP_C;                   // couplings to the row before, to the row after
    double* cn = cp + ((hm + 1) & ~1);
    for (int i = lane; i < nt; i += 32) {
        cp[i] = end ? ap2ph[ny - i] : am2ph[i + 1];
        cn[i] = end ? am2ph[ny - i] : ap2ph[i + 1];
    }
    const int nkb = yp_blocks(M1), nitems = (nz / 2 + 1) * nkb;
    const int stride = (int)grid.gx();
    const int dj = end ? -1 : 1, jw = end ? ny - 1 : 0;  // row i of the sweep is memory row jw + dj i
    const ptrdiff_t gstep = (ptrdiff_t)dj * M1;
    // copies: lane = (row of a pair, plane, mode)
    const int lc = lane & 7, lz = (lane >> 3) & 1, lr = lane >> 4;
    unsigned char* const cdst = my + lz * box + lr * ROW + lc * ES;
    double* const fdst = sr + 2 * lane;
    const S* csrc = nullptr;       // row lr of the next item's column
    const double* fsrc = nullptr;  // pivots of row lane / 4
    bool cval = false;
    auto aim = [&](int item) {
        const int kz = item / nkb, kx = (item - kz * nkb) * YP_C + lc, kp = lz ? (kz ? nz - kz : 0) : kz;
        cval = item < nitems && kx < M1 && (lz == 0 || kp != kz);
        csrc = spec + (size_t)kp * ny * M1 + kx + jw * M1 + lr * gstep;
        fsrc = fac + ((size_t)item * ny + jw + dj * (lane >> 2)) * YP_C + 2 * (lane & 3);
    };
    auto copy_fac = [&](int i0, int n) {  // rows i0 .. i0 + n - 1, n <= 8
        if ((lane >> 2) < n) cpa<16>(fdst + i0 * YP_C, fsrc + (ptrdiff_t)dj * i0 * YP_C);
    };
    auto copy_rows = [&](int i0, int n) {
        const S* src = csrc + i0 * gstep;
        unsigned char* dst = cdst + i0 * ROW;
#pragma unroll
        for (int u = 0; u < YP_U / 2; u++) {
            if (cval && 2 * u + lr < n) cpa<ES>(dst + 2 * u * ROW, src);
            src += 2 * gstep;
        }
    };
    int item = (int)grid.x();
    if (item < nitems) {
        aim(item);
        for (int i0 = 0; i0 < nt; i0 += YP_U) copy_fac(i0, nt - i0);
    }
    pdl_wait();  // the spectrum is written by the kernel before this one
    if (item < nitems)
        for (int i0 = 0; i0 < nt; i0 += YP_U) copy_rows(i0, nt - i0);
    // sweeps: lane = (plane, mode, part)
    const int pz = lane >> 4, col = (lane >> 1) & 7, part = lane & 1;
    R* const sd = reinterpret_cast<R*>(my + pz * box) + col * 2 + part;
    const double* const srl = sr + col;
    const int nb = nt - 1, nf = nt & ~(YP_U - 1), nbf = nb & ~(YP_U - 1);
    for (int it = 0; item < nitems; item += stride, it++) {
        const int next = item + stride;
        if (next >= nitems) pdl_trigger();
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncwarp();
        // to the junction: F(i) = r (f - cp F(i-1)), kept in the row's slot
        double f = 0.0;
        for (int i0 = 0; i0 < nf; i0 += YP_U) {
            double g[YP_U], mm[YP_U];
#pragma unroll
            for (int u = 0; u < YP_U; u++) {
                const double r = srl[(i0 + u) * YP_C];
                g[u] = (double)sd[(i0 + u) * 2 * YP_C] * r;
                mm[u] = cp[i0 + u] * r;
            }
#pragma unroll
            for (int u = 0; u < YP_U; u++) {
                f = fma(-mm[u], f, g[u]);
                sd[(i0 + u) * 2 * YP_C] = (R)f;
            }
        }
        for (int i = nf; i < nt; i++) {
            const double r = srl[i * YP_C];
            f = fma(-(cp[i] * r), f, (double)sd[i * 2 * YP_C] * r);
            sd[i * 2 * YP_C] = (R)f;
        }
        const double cu = cn[nb] * srl[nb * YP_C];
        xch[it & 1][end][lane] = make_double2(f, cu);
        __syncthreads();
        const double2 o = xch[it & 1][end ^ 1][lane];
        double x = (f - cu * o.x) / (1.0 - cu * o.y);
        // back to the wall: x(i) = F(i) - cn r x(i+1), out to memory; the
        // next item's rows follow into the slots just read
        const int kz = item / nkb, kx = (item - kz * nkb) * YP_C + col, kp = pz ? (kz ? nz - kz : 0) : kz;
        const bool valid = kx < M1 && (pz == 0 || kp != kz);
        R* out = reinterpret_cast<R*>(spec + (size_t)kp * ny * M1 + kx + jw * M1 + nb * gstep) + part;
        if (valid) *out = (R)x;
        for (int i = nb - 1; i >= nbf; i--) {
            x = fma(-(cn[i] * srl[i * YP_C]), x, (double)sd[i * 2 * YP_C]);
            out -= 2 * gstep;
            if (valid) *out = (R)x;
        }
        __syncwarp();
        if (next < nitems) {
            aim(next);
            copy_fac(nbf, nt - nbf);
            copy_rows(nbf, nt - nbf);
        }
        for (int i0 = nbf - YP_U; i0 >= 0; i0 -= YP_U) {
            double d[YP_U], mm[YP_U];
#pragma unroll
            for (int u = 0; u < YP_U; u++) {
                d[u] = (double)sd[(i0 + u) * 2 * YP_C];
                mm[u] = cn[i0 + u] * srl[(i0 + u) * YP_C];
            }
            __syncwarp();
            if (next < nitems) {
                copy_fac(i0, YP_U);
                copy_rows(i0, YP_U);
            }
#pragma unroll
            for (int u = YP_U - 1; u >= 0; u--) {
                x = fma(-mm[u], x, d[u]);
                out -= 2 * gstep;
                if (valid) *out = (R)x;
            }
        }
    }
}

template <class S>
__global__ void __launch_bounds__(64, 8) k_ys_pair(int ny, int M1, int nz, const double* __restrict__ am2ph,
                                                   const double* __restrict__ ap2ph, S* __restrict__ spec,
                                                   const double* __restrict__ fac) {
    ys_pair_body(OwnGrid{}, ny, M1, nz, am2ph, ap2ph, spec, fac);
}
template <class S>
__global__ void __launch_bounds__(64, 8) k_ys_pair_grp(const GrpTab<YsArgs<S>>* __restrict__ t) {
    SubGrid g;
    const YsArgs<S>& a = t->e[grp_member(t, g)];
    ys_pair_body(g, a.ny, a.M1, a.nz, a.am2ph, a.ap2ph, a.spec, a.fac);
}

size_t pois_fac_doubles(const DConst& c) {
    return (size_t)(c.nz / 2 + 1) * yp_blocks(c.nx / 2 + 1) * YP_C * c.ny;
}
void launch_pois_factors(cudaStream_t st, const DConst& c, const DMetric& m, double* fac, int dc_here) {
    const int M1 = c.nx / 2 + 1, n = M1 * (c.nz / 2 + 1);
    k_pois_factors<<<(n + 127) / 128, 128, 0, st>>>(c.ny, M1, c.nz, m, fac, dc_here);
}

static size_t yp_smem(int ny, int esize) { return 2 * (size_t)yp_half(ny - ny / 2, esize); }
size_t ys_smem(const DConst& c, int esize) { return yp_smem(c.ny, esize); }
// a CTA per work item up to the CTAs the device holds at once (8 per SM by
// registers, fewer by shared memory), which then walk the items
dim3 ys_member_grid(const DConst& c, int esize) {
    const int items = (c.nz / 2 + 1) * yp_blocks(c.nx / 2 + 1);
    const int per_sm = (int)std::min<size_t>(8, (size_t)(224 * 1024) / (yp_smem(c.ny, esize) + 3072));
    return dim3((unsigned)std::min(items, std::max(1, per_sm) * (c.nsm > 0 ? c.nsm : 148)));
}

template <class S>
static void ysolve_fac_t(cudaStream_t st, const DConst& c, const DMetric& m, S* spec, const double* fac) {
    launch_pdl(k_ys_pair<S>, ys_member_grid(c, sizeof(S)), dim3(64), yp_smem(c.ny, sizeof(S)), st, c.ny, c.nx / 2 + 1,
               c.nz, m.am2ph, m.ap2ph, spec, fac);
}
void launch_ysolve_fac(cudaStream_t st, const DConst& c, const DMetric& m, double2* spec, const double* fac) {
    ysolve_fac_t(st, c, m, spec, fac);
}
void launch_ysolve_fac(cudaStream_t st, const DConst& c, const DMetric& m, float2* spec, const double* fac) {
    ysolve_fac_t(st, c, m, spec, fac);
}
void launch_ys_grp(cudaStream_t st, const GrpTab<YsArgs<double2>>* t, int nblk, size_t smem) {
    launch_pdl(k_ys_pair_grp<double2>, dim3((unsigned)nblk), dim3(64), smem, st, t);
}
void launch_ys_grp(cudaStream_t st, const GrpTab<YsArgs<float2>>* t, int nblk, size_t smem) {
    launch_pdl(k_ys_pair_grp<float2>, dim3((unsigned)nblk), dim3(64), smem, st, t);
}

// ---------------------------------------------------------------------------
// launchers: partition length MR in {8, 12, 16}, P = ceil(ny/MR) <= 16 warps
// ---------------------------------------------------------------------------
__host__ __device__ inline int part_len_dev(int ny) { return ny <= 64 ? 8 : (ny <= 192 ? 12 : 16); }
__host__ __device__ inline int tridiag_partitions_dev(int ny) {
    const int mr = part_len_dev(ny);
    return (ny + mr - 1) / mr;
}
static int part_len(int ny) { return part_len_dev(ny); }

int tridiag_partitions(int ny) { return tridiag_partitions_dev(ny); }

bool tridiag_supported(int ny) { return ny >= 3 && ny <= 256; }

static size_t red_smem(int P, int nc) { return (size_t)2 * P * 32 * (3 + nc) * sizeof(double); }

__global__ void k_helm_factors(DConst cst, DMetric m, const DCoef* __restrict__ coef, int ns0, int nsub, double a1,
                               double a2, double a3, double* __restrict__ facs);

void tridiag_init() {
    cudaFuncSetAttribute(k_ysolve<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    cudaFuncSetAttribute(k_ysolve<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    cudaFuncSetAttribute(k_ysolve<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    for (auto* k : {(const void*)k_helm<double, HY_U>, (const void*)k_helm<double, HY_U / 2>,
                    (const void*)k_helm<float, HY_U>, (const void*)k_helm<float, HY_U / 2>,
                    (const void*)k_helm<float, HY_U, float>, (const void*)k_helm_grp<double, HY_U>,
                    (const void*)k_helm_grp<double, HY_U / 2>, (const void*)k_helm_grp<float, HY_U>,
                    (const void*)k_helm_grp<float, HY_U / 2>, (const void*)k_helm_grp<float, HY_U, float>})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 80 * 1024);
    for (auto* k : {(const void*)k_ys_pair<double2>, (const void*)k_ys_pair<float2>,
                    (const void*)k_ys_pair_grp<double2>, (const void*)k_ys_pair_grp<float2>})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024);
    cudaFuncSetAttribute(k_helm_factors, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
}

int tridiag_part_len(int ny) { return part_len(ny); }

size_t helm_fac_doubles(int ny) { return (size_t)9 * helm_stride(ny); }
int helm_variants() { return HELM_NVAR; }
// the Helmholtz launch shapes of precision form prec: FP32 storage adds
// float-arithmetic sweeps (helm_var 2)
int helm_variants(int prec) { return prec == 2 ? HELM_NVAR + 1 : HELM_NVAR; }

// pivots of the Helmholtz matrices of substeps ns0..ns0+nsub-1 for the
// current dt (coef->dt): one thread per (substep, type, wall) eliminates its
// half of the rows, in the order of InverseTridiagonal, on the coefficients of
// clcU1Hat / clcU2Hat / clcScalar (src/m_TScheme.f90:374-380,409-420,486-492)
__global__ void __launch_bounds__(32) k_helm_factors(DConst cst, DMetric m, const DCoef* __restrict__ coef, int ns0,
                                                     int nsub, double a1, double a2, double a3,
                                                     double* __restrict__ facs) {
    extern __shared__ double shm[];  // ap, ac, am of the three types, rows 0..ny+1
    const int ny = cst.ny, L = ny + 2;
    const double* srcs[9] = {m.ap2cCN, m.ac2cCN, m.am2cCN, m.ap2p, m.ac2p, m.am2p, m.ap2cScCN, m.ac2cScCN, m.am2cScCN};
    for (int a = 0; a < 9; a++)
        for (int j = threadIdx.x; j < L; j += blockDim.x) shm[a * L + j] = srcs[a][j];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const int q = threadIdx.x >> 1, w = threadIdx.x & 1;
    if (q >= 3 * nsub) return;
    const int ns = ns0 + q / 3, t = q % 3;
    const double alp = ns == 1 ? a1 : (ns == 2 ? a2 : a3);
    const double dt = coef->dt;
    const double beta = (t == 2) ? 0.5 * alp * cst.sdiff * dt : 0.5 * alp * cst.xnu * dt;
    const double* ap = shm + (3 * t) * L;
    const double* ac = ap + L;
    const double* am = ac + L;
    // from wall `w` (0 the lower) to the row before the junction: r, MP, MN of
    // helm_body; the other wall's first row couples to no wall of the table
    double* F = facs + (size_t)((ns - 1) * 3 + t) * helm_stride(ny);
    double* FP = F;                  // MP
    double* FR = F + (ny + 2);       // r
    double* FN = F + 2 * (ny + 2);   // MN
    const int h = ny >> 1, dj = w ? -1 : 1, n = w ? ny - h : h;
    const double* ab = w ? ap : am;  // to the row before, to the row after
    const double* an = w ? am : ap;
    int jc = w ? ny : 1;
    double cprev = 0.0, vecm = 1.0;
    for (int i = 0; i < n; i++, jc += dj) {
        const bool one = t == 1 && jc == 1;  // clcU2Hat: row 1 is the identity
        const double arr = i ? cprev / vecm : 0.0;
        const double a = one ? 0.0 : -__dmul_rn(beta, ab[jc]);
        const double b = one ? 1.0 : __dadd_rn(-__dmul_rn(beta, ac[jc]), 1.0);
        vecm = i ? __dsub_rn(b, __dmul_rn(a, arr)) : b;
        cprev = one ? 0.0 : -__dmul_rn(beta, an[jc]);
        FR[jc] = 1.0 / vecm;
        FP[jc] = i ? a / vecm : 0.0;
        FN[jc] = cprev / vecm;
    }
}

void launch_helm_factors(cudaStream_t st, const DConst& c, const DMetric& m, const DCoef* coef, int ns0, int nsub,
                         const double* alp, double* fac) {
    launch_pdl(k_helm_factors, dim3(1), dim3(32), (size_t)9 * (c.ny + 2) * sizeof(double), st, c, m, coef, ns0, nsub,
               alp[0], alp[1], alp[2], fac);
}

// the launch shapes by helm_var: rows per chunk HY_U, half of that, or (FP32
// storage) HY_U with float sweeps
static bool helm_float(const DConst& c, int vsize) { return c.helm_var == 2 && vsize == 4; }
size_t helm_smem(const DConst& c, int vsize) {
    return 2 * (size_t)helm_half(c.ny - c.ny / 2, vsize, helm_float(c, vsize) ? 4 : 8);
}
// a CTA per work item up to the CTAs the device holds at once (8 per SM by
// registers, fewer by shared memory), which then walk the items
dim3 helm_member_grid(const DConst& c, int ncomp, int vsize) {
    const long long items = ((long long)c.nx * c.nz + 31) / 32 * ncomp;
    const int per_sm = (int)std::min<size_t>(8, (size_t)(224 * 1024) / (helm_smem(c, vsize) + 3072));
    return dim3((unsigned)std::min<long long>(items, (long long)std::max(1, per_sm) * (c.nsm > 0 ? c.nsm : 148)));
}

template <class V>
static void helm_grp_t(cudaStream_t st, const DConst& key, const GrpTab<HelmArgs<V>>* t, int nblk, size_t smem) {
    using WF = std::conditional_t<sizeof(V) == 4, float, double>;
    const dim3 g((unsigned)nblk), b(64);
    if (key.helm_var == 1) launch_pdl(k_helm_grp<V, HY_U / 2>, g, b, smem, st, t);
    else if (helm_float(key, sizeof(V))) launch_pdl(k_helm_grp<V, HY_U, WF>, g, b, smem, st, t);
    else launch_pdl(k_helm_grp<V, HY_U>, g, b, smem, st, t);
}
void launch_helm_grp(cudaStream_t st, const DConst& key, const GrpTab<HelmArgs<double>>* t, int nblk, size_t smem) {
    helm_grp_t(st, key, t, nblk, smem);
}
void launch_helm_grp(cudaStream_t st, const DConst& key, const GrpTab<HelmArgs<float>>* t, int nblk, size_t smem) {
    helm_grp_t(st, key, t, nblk, smem);
}

template <class V>
static void helm_dispatch(cudaStream_t st, const DConst& c, const DCoef* coef, const FieldSet<V>& f,
                          const double* duy_ym, const double* uy_ym, const double* fac) {
    using WF = std::conditional_t<sizeof(V) == 4, float, double>;
    const int ncomp = c.scalar_on ? 4 : 3;
    const dim3 g = helm_member_grid(c, ncomp, sizeof(V)), b(64);
    const size_t smem = helm_smem(c, sizeof(V));
    if (c.helm_var == 1)
        launch_pdl(k_helm<V, HY_U / 2>, g, b, smem, st, c, coef, ncomp, f, duy_ym, uy_ym, fac);
    else if (helm_float(c, sizeof(V)))
        launch_pdl(k_helm<V, HY_U, WF>, g, b, smem, st, c, coef, ncomp, f, duy_ym, uy_ym, fac);
    else
        launch_pdl(k_helm<V, HY_U>, g, b, smem, st, c, coef, ncomp, f, duy_ym, uy_ym, fac);
}

void launch_helm(cudaStream_t st, const DConst& c, const DCoef* coef, const Fields& f, const double* duy_ym,
                 const double* uy_ym, const double* fac) {
    helm_dispatch(st, c, coef, f, duy_ym, uy_ym, fac);
}
void launch_helm(cudaStream_t st, const DConst& c, const DCoef* coef, const Fields32& f, const double* duy_ym,
                 const double* uy_ym, const double* fac) {
    helm_dispatch(st, c, coef, f, duy_ym, uy_ym, fac);
}

void launch_ysolve(cudaStream_t st, const DConst& c, const DMetric& m, double2* spec) {
    const int mr = part_len(c.ny), P = tridiag_partitions(c.ny);
    dim3 blk(32, P);
    dim3 grd((2 * (c.nx / 2 + 1) + 31) / 32, c.nz);
    const size_t sm = red_smem(P, 1);
    double* sd = reinterpret_cast<double*>(spec);
    if (mr == 8) k_ysolve<8><<<grd, blk, sm, st>>>(c, m, sd);
    else if (mr == 12) k_ysolve<12><<<grd, blk, sm, st>>>(c, m, sd);
    else k_ysolve<16><<<grd, blk, sm, st>>>(c, m, sd);
}

}  // namespace ptc
