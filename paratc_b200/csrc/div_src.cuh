// div_src.cuh -- the source of the pressure Poisson equation, computed where
// the forward x transform consumes it: the divergence of u* at the two x
// points 2e, 2e+1 of row g = k*ny + (jc-1) (clcPrSrc, src/m_TScheme.f90:
// 48-77: 4th-order staggered differences in x and z, 2nd-order in y).  The
// loads of a point pair are separated from its arithmetic so that a thread
// can put the loads of several pairs in flight before it uses any of them.
#pragma once
#include "common.cuh"

namespace ptc {

struct DivTaps {
    double2 u01, u23, v0, v1, w0, w1, w2, w3;
    double um, rdyp;
};

template <class V>
__device__ __forceinline__ void div_load(DivTaps& t, const DConst& c, const DMetric& m, const V* __restrict__ ux,
                                         const V* __restrict__ uy, const V* __restrict__ uz, int g, int e) {
    const int nx = c.nx, ny = c.ny, nz = c.nz;
    const size_t pl = (size_t)c.nyt * nx;
    const int k = g / ny, jc = g - k * ny + 1;
    const int km = k == 0 ? nz - 1 : k - 1, kp = k == nz - 1 ? 0 : k + 1, ku = kp == nz - 1 ? 0 : kp + 1;
    const int i0 = 2 * e, im = i0 == 0 ? nx - 1 : i0 - 1, i2 = i0 + 2 == nx ? 0 : i0 + 2;
    const size_t r0 = (size_t)jc * nx;
    const V* ur = ux + (size_t)k * pl + r0;
    const V* vr = uy + (size_t)k * pl + r0;
    t.u01 = ld_pair(ur + i0);
    t.u23 = ld_pair(ur + i2);
    t.um = (double)__ldg(ur + im);
    t.v0 = ld_pair(vr + i0);
    t.v1 = ld_pair(vr + nx + i0);
    t.w0 = ld_pair(uz + (size_t)km * pl + r0 + i0);
    t.w1 = ld_pair(uz + (size_t)k * pl + r0 + i0);
    t.w2 = ld_pair(uz + (size_t)kp * pl + r0 + i0);
    t.w3 = ld_pair(uz + (size_t)ku * pl + r0 + i0);
    t.rdyp = __ldg(&m.rdyp[jc]);
}

// (div at 2e, div at 2e+1)
__device__ __forceinline__ double2 div_eval(const DivTaps& t, const DConst& c) {
    const double dudx0 = c.dxC[0] * t.um + c.dxC[1] * t.u01.x + c.dxC[2] * t.u01.y + c.dxC[3] * t.u23.x;
    const double dudx1 = c.dxC[0] * t.u01.x + c.dxC[1] * t.u01.y + c.dxC[2] * t.u23.x + c.dxC[3] * t.u23.y;
    const double dvdy0 = (t.v1.x - t.v0.x) * t.rdyp, dvdy1 = (t.v1.y - t.v0.y) * t.rdyp;
    const double dwdz0 = c.dzC[0] * t.w0.x + c.dzC[1] * t.w1.x + c.dzC[2] * t.w2.x + c.dzC[3] * t.w3.x;
    const double dwdz1 = c.dzC[0] * t.w0.y + c.dzC[1] * t.w1.y + c.dzC[2] * t.w2.y + c.dzC[3] * t.w3.y;
    return make_double2(dudx0 + dvdy0 + dwdz0, dudx1 + dvdy1 + dwdz1);
}

// the source of every point pair f = start, start + STRIDE, ... < B*N of a
// batch of B rows from g0 (pair e of row b = f / N), U pairs in flight per
// thread: st(b, e, value) stores it, the running max|div| goes to dm
template <int N, int B, int STRIDE, int U, class V, class ST>
__device__ __forceinline__ void div_batch(const DConst& c, const DMetric& m, const V* __restrict__ ux,
                                          const V* __restrict__ uy, const V* __restrict__ uz, int g0,
                                          int nrows, double sudtal, int start, double& dm, const ST& st) {
    for (int f0 = start; f0 < B * N; f0 += U * STRIDE) {
        DivTaps tp[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int f = f0 + u * STRIDE;
            const int b = f / N, e = f - b * N;
            ok[u] = f < B * N && g0 + b < nrows;
            if (ok[u]) div_load(tp[u], c, m, ux, uy, uz, g0 + b, e);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int f = f0 + u * STRIDE;
            if (f >= B * N) continue;
            const int b = f / N, e = f - b * N;
            double2 val = make_double2(0.0, 0.0);
            if (ok[u]) {
                const double2 d = div_eval(tp[u], c);
                dm = nmax(dm, nmax(fabs(d.x), fabs(d.y)));
                val = make_double2(sudtal * d.x, sudtal * d.y);
            }
            st(b, e, val);
        }
    }
}

// The same sources with a thread marching through k: it owns NPT point pairs
// (e0, e0 + Q, ...) of one row jc and, plane by plane, takes one new pair of w
// (the other three taps stay in registers), u01 and the two v pairs; the x
// neighbours of u01 come from the neighbouring lanes.  So a pair of points
// costs four 16-byte loads instead of nine.  They go to slots of the thread's
// own in shared memory (cp.async, D planes ahead, no barrier), which keeps
// more of them in flight than registers could: the nine-load form was bound
// by that.
template <class V>
struct MarchPair;
template <>
struct MarchPair<double> {
    using T = double2;
};
template <>
struct MarchPair<float> {
    using T = float2;
};
template <int BYTES>
__device__ __forceinline__ void march_copy(void* sdst, const void* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}

// planes k0 .. k1-1 of row j (0-based; on: the thread has a pair and its row
// lies inside the grid); ring: [D][NPT][4][Q] pairs.  begin(k) runs before
// plane k's values are stored, st(k, e, value) stores them, done(k) runs after
// them; all threads of the group take every step.  begin returns false to stop.
template <int N, int Q, int NPT, int D, class V, class BEG, class ST, class DONE>
__device__ __forceinline__ bool div_march(const DConst& c, const DMetric& m, const V* __restrict__ ux,
                                          const V* __restrict__ uy, const V* __restrict__ uz, int j, int e0, bool on,
                                          int k0, int k1, double sudtal, double& dm,
                                          typename MarchPair<V>::T* __restrict__ ring, int tp, const BEG& begin,
                                          const ST& st, const DONE& done) {
    using P2 = typename MarchPair<V>::T;
    const int nx = c.nx, nz = c.nz, lane = threadIdx.x & 31;
    const unsigned pl = (unsigned)c.nyt * nx, r0 = (unsigned)(on ? j + 1 : 1) * nx, off = r0 + 2 * e0;
    const double rdyp = on ? __ldg(&m.rdyp[j + 1]) : 0.0;
    auto pair = [](const V* p) { return __ldg(reinterpret_cast<const P2*>(p)); };
    auto has = [&](int p) { return N % Q == 0 || p + 1 < NPT || e0 + p * Q < N; };
    auto el = [&](int p) { return lane == 0 || e0 + p * Q == 0; };
    auto er = [&](int p) { return lane == 31 || e0 + p * Q == N - 1; };
    auto plane = [&](int k) { return (unsigned)(k < 0 ? k + nz : (k >= nz ? k - nz : k)) * pl; };
    P2* const my = ring + tp;
    auto copy = [&](int k, int d) {  // plane k's pairs into ring slot d
        const unsigned a = (unsigned)k * pl;
        const V *ru = ux + a + off, *rv = uy + a + off, *rw = uz + plane(k + 2) + off;
#pragma unroll
        for (int p = 0; p < NPT; p++) {
            if (!on || !has(p)) continue;
            P2* s = my + (d * NPT + p) * 4 * Q;
            march_copy<sizeof(P2)>(s, ru + 2 * p * Q);
            march_copy<sizeof(P2)>(s + Q, rv + 2 * p * Q);
            march_copy<sizeof(P2)>(s + 2 * Q, rv + 2 * p * Q + nx);
            march_copy<sizeof(P2)>(s + 3 * Q, rw + 2 * p * Q);
        }
    };
    P2 w[3][NPT], ur[NPT];
    V ul[NPT];
    auto edges = [&](int k) {  // the neighbours that no lane of the warp holds
        const V* ru = ux + (unsigned)k * pl + off;
#pragma unroll
        for (int p = 0; p < NPT; p++) {
            if (!on || !has(p)) continue;
            if (el(p)) ul[p] = __ldg(e0 + p * Q == 0 ? ru + nx - 1 : ru + 2 * p * Q - 1);
            if (er(p)) ur[p] = pair(e0 + p * Q == N - 1 ? ru + 2 * p * Q + 2 - nx : ru + 2 * p * Q + 2);
        }
    };
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
        for (int p = 0; p < NPT; p++)
            if (on && has(p)) w[q][p] = pair(uz + plane(k0 - 1 + q) + off + 2 * p * Q);
    for (int d = 0; d < D; d++) {
        if (k0 + d < k1) copy(k0 + d, d);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    edges(k0);
    int d = 0;
    for (int k = k0; k < k1; k++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(D - 1) : "memory");
        double2 val[NPT];
#pragma unroll
        for (int p = 0; p < NPT; p++) {
            const P2* s = my + (d * NPT + p) * 4 * Q;
            const P2 u01 = s[0], v0 = s[Q], v1 = s[2 * Q], w3 = s[3 * Q];
            // (lanes without a pair take part in the exchange)
            const V lx = __shfl_up_sync(0xffffffffu, u01.y, 1);
            const V rx = __shfl_down_sync(0xffffffffu, u01.x, 1);
            const V ry = __shfl_down_sync(0xffffffffu, u01.y, 1);
            DivTaps q;
            q.u01 = make_double2(u01.x, u01.y);
            q.um = el(p) ? ul[p] : lx;
            q.u23 = er(p) ? make_double2(ur[p].x, ur[p].y) : make_double2(rx, ry);
            q.v0 = make_double2(v0.x, v0.y);
            q.v1 = make_double2(v1.x, v1.y);
            q.w0 = make_double2(w[0][p].x, w[0][p].y);
            q.w1 = make_double2(w[1][p].x, w[1][p].y);
            q.w2 = make_double2(w[2][p].x, w[2][p].y);
            q.w3 = make_double2(w3.x, w3.y);
            q.rdyp = rdyp;
            const double2 dv = div_eval(q, c);
            const bool act = on && has(p);
            if (act) dm = nmax(dm, nmax(fabs(dv.x), fabs(dv.y)));
            val[p] = act ? make_double2(sudtal * dv.x, sudtal * dv.y) : make_double2(0.0, 0.0);
            w[0][p] = w[1][p];
            w[1][p] = w[2][p];
            w[2][p] = w3;
        }
        if (k + 1 < k1) edges(k + 1);
        if (k + D < k1) copy(k + D, d);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        d = d + 1 == D ? 0 : d + 1;
        if (!begin(k)) {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            return false;
        }
#pragma unroll
        for (int p = 0; p < NPT; p++)
            if (has(p)) st(k, e0 + p * Q, val[p]);
        done(k);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    return true;
}

}  // namespace ptc
