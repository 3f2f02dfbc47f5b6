// k_momadj.cu -- tangent linear of the momentum advection operator
// qnadv_uvw (src/INTEG/windadv.f90:46-79 with uadv_fd :82-220, vadv_fd :223-357,
// wadv_fd :360-492 and the stencils :494-1127), FD4/FD2 with the artificial viscosity.
//
// The operator is evaluated per cell in gather form: each output (au, av or aw at one
// cell) recomputes the face fluxes it differences, with the advective velocities
// m/rho0 - shift formed from the same momentum loads.  The code keeps the reference's
// expressions and the direction order of ntime's parity, so its FP64 instance equals
// the K2 momentum advection bit for bit (a test checks it).
//   TL: the per-cell form on dual numbers with one partial (tangent = dm).
//   AD: k_momad.cu.
#include "dual.cuh"
#include "mg_common.cuh"
#include "mimica_gpu.h"

namespace {

constexpr double AVISC = 1. / 16.;   // windadv.f90:39


// advective velocity of momentum component f at level k (funcpack.f90:65-94)
template <typename T>
__device__ __forceinline__ T adv_vel(const DevGrid &G, int f, int k, const T &m)
{
    if (f == 0) return m / T(__ldg(G.den0 + k - 1)) - T(G.u0shift);
    if (f == 1) return m / T(__ldg(G.den0 + k - 1)) - T(G.v0shift);
    return m / T(__ldg(G.avden0 + k - 1));
}

// ---------------- the nine direction terms (oracle and K2 order of operations) ----------------
template <typename T, class L>
__device__ __forceinline__ T u_x(const DevGrid &G, const L &ld, int i, int j, int k, T ua)
{
    const bool fd4 = G.mom_ord == 4;
    const double dx1 = 1. / G.dx, dx2 = 1. / (2. * G.dx);
    const double c1 = fd4 ? 4. / 3. : 1., c2 = fd4 ? 1. / 3. : 0.;
    auto U = [&](int p) { return ld.m(0, p, j, k); };
    auto UT = [&](int p) { return ld.t(0, p, j, k); };
    auto F = [&](int p) { return ((UT(p + 1) + UT(p)) * T(0.5)) * ((U(p + 1) + U(p)) * T(0.5)); };
    auto A = [&](int p) { return ((UT(p + 2) + UT(p)) * T(0.5)) * ((U(p + 2) + U(p)) * T(0.5)); };
    ua = ua + T(c1) * (F(i) - F(i - 1)) * T(dx1) - T(c2) * (A(i) - A(i - 2)) * T(dx2);
    if (G.lavisc) {
        const T mu = dabs(UT(i)) * T(dx1);
        ua = ua - T(AVISC) * mu * (-U(i + 2) + T(4.) * U(i + 1) - T(6.) * U(i) + T(4.) * U(i - 1) - U(i - 2));
    }
    return ua;
}

template <typename T, class L>
__device__ __forceinline__ T u_y(const DevGrid &G, const L &ld, int i, int j, int k, T ua)
{
    const bool fd4 = G.mom_ord == 4;
    const double dy1 = 1. / G.dy, dy3 = 1. / (3. * G.dy);
    const double c1 = fd4 ? 9. / 8. : 1., c2 = fd4 ? 1. / 8. : 0.;
    auto U = [&](int q) { return ld.m(0, i, q, k); };
    auto V = [&](int di, int q) { return ld.t(1, i + di, q, k); };
    auto F = [&](int q) {
        const T vv = T(c1) * (V(-1, q + 1) + V(0, q + 1)) * T(0.5) - T(c2) * (V(-2, q + 1) + V(1, q + 1)) * T(0.5);
        const T fr = (U(q + 1) + U(q)) * T(0.5);
        return vv * fr;
    };
    ua = ua + T(c1) * (F(j) - F(j - 1)) * T(dy1) - T(c2) * (F(j + 1) - F(j - 2)) * T(dy3);
    if (G.lavisc) {
        const T mu = T(0.25) * dabs(V(-1, j) + V(0, j) + V(-1, j + 1) + V(0, j + 1)) * T(dy1);
        ua = ua - T(AVISC) * mu * (-U(j + 2) + T(4.) * U(j + 1) - T(6.) * U(j) + T(4.) * U(j - 1) - U(j - 2));
    }
    return ua;
}

// advuz_fd / advvz_fd (advhz): f = 0 (u, w at i-1, i, i-2, i+1) or 1 (v, w at j-1, j, j-2, j+1)
template <typename T, class L>
__device__ __forceinline__ T h_z(const DevGrid &G, const L &ld, int f, int i, int j, int k, T ua)
{
    const int nz = G.nz;
    const bool fd4 = G.mom_ord == 4;
    const double c1 = fd4 ? 9. / 8. : 1., c2 = fd4 ? 1. / 8. : 0.;
    auto dzw = [&](int q) { return __ldg(G.dzw + q - 1); };
    auto dz1w = [&](int q) { return __ldg(G.dz1w + q - 1); };
    auto U = [&](int q) { return ld.m(f, i, j, q); };
    auto W = [&](int d, int q) { return f == 0 ? ld.t(2, i + d, j, q) : ld.t(2, i, j + d, q); };
    auto F = [&](int q) -> T {
        if (q >= nz) return T(0.);
        const T ww = T(c1) * (W(-1, q + 1) + W(0, q + 1)) * T(0.5) - T(c2) * (W(-2, q + 1) + W(1, q + 1)) * T(0.5);
        const T fr = (T(dzw(q + 1)) * U(q + 1) + T(dzw(q)) * U(q)) / T(dzw(q + 1) + dzw(q));
        return ww * fr;
    };
    if (k >= 3 && k <= nz - 1)
        ua = ua + T(c1) * (F(k) - F(k - 1)) * T(dz1w(k)) - T(c2) * (F(k + 1) - F(k - 2)) / T(dzw(k - 1) + dzw(k) + dzw(k + 1));
    else if (k == 1)
        ua = ua + (F(1) - T(0.)) * T(dz1w(1));
    else if (k == 2)
        ua = ua + T(c1) * (F(2) - F(1)) * T(dz1w(f == 1 ? 2 : 1)) - T(c2) * (F(3) - T(0.)) / T(dzw(1) + dzw(2) + dzw(3));
    else   // k == nz
        ua = ua + (T(0.) - F(nz - 1)) * T(dz1w(nz));
    if (G.lavisc && k >= 3 && k <= nz - 2) {
        const T mu = T(0.25) * dabs(W(-1, k) + W(0, k) + W(-1, k + 1) + W(0, k + 1)) * T(dz1w(k));
        ua = ua - T(AVISC) * mu * (-U(k + 2) + T(4.) * U(k + 1) - T(6.) * U(k) + T(4.) * U(k - 1) - U(k - 2));
    }
    return ua;
}

template <typename T, class L>
__device__ __forceinline__ T v_x(const DevGrid &G, const L &ld, int i, int j, int k, T va)
{
    const bool fd4 = G.mom_ord == 4;
    const double dx1 = 1. / G.dx, dx3 = 1. / (3. * G.dx);
    const double c1 = fd4 ? 9. / 8. : 1., c2 = fd4 ? 1. / 8. : 0.;
    auto V = [&](int p) { return ld.m(1, p, j, k); };
    auto UT = [&](int p, int dj) { return ld.t(0, p, j + dj, k); };
    auto F = [&](int p) {
        const T uu = T(c1) * (UT(p + 1, -1) + UT(p + 1, 0)) * T(0.5) - T(c2) * (UT(p + 1, -2) + UT(p + 1, 1)) * T(0.5);
        const T fr = (V(p + 1) + V(p)) * T(0.5);
        return uu * fr;
    };
    va = va + T(c1) * (F(i) - F(i - 1)) * T(dx1) - T(c2) * (F(i + 1) - F(i - 2)) * T(dx3);
    if (G.lavisc) {
        const T mu = T(0.25) * dabs(UT(i, -1) + UT(i, 0) + UT(i + 1, -1) + UT(i + 1, 0)) * T(dx1);
        va = va - T(AVISC) * mu * (-V(i + 2) + T(4.) * V(i + 1) - T(6.) * V(i) + T(4.) * V(i - 1) - V(i - 2));
    }
    return va;
}

template <typename T, class L>
__device__ __forceinline__ T v_y(const DevGrid &G, const L &ld, int i, int j, int k, T va)
{
    const bool fd4 = G.mom_ord == 4;
    const double dy1 = 1. / G.dy, dy2 = 1. / (2. * G.dy);
    const double c1 = fd4 ? 4. / 3. : 1., c2 = fd4 ? 1. / 3. : 0.;
    auto V = [&](int q) { return ld.m(1, i, q, k); };
    auto VT = [&](int q) { return ld.t(1, i, q, k); };
    auto F = [&](int q) { return ((VT(q + 1) + VT(q)) * T(0.5)) * ((V(q + 1) + V(q)) * T(0.5)); };
    auto A = [&](int q) { return ((VT(q + 2) + VT(q)) * T(0.5)) * ((V(q + 2) + V(q)) * T(0.5)); };
    va = va + T(c1) * (F(j) - F(j - 1)) * T(dy1) - T(c2) * (A(j) - A(j - 2)) * T(dy2);
    if (G.lavisc) {
        const T mu = dabs(VT(j)) * T(dy1);
        va = va - T(AVISC) * mu * (-V(j + 2) + T(4.) * V(j + 1) - T(6.) * V(j) + T(4.) * V(j - 1) - V(j - 2));
    }
    return va;
}

// advwx_fd / advwy_fd (advwh): dir 0 (x, velocity ua) or 1 (y, velocity va); levels 2..nz
template <typename T, class L>
__device__ __forceinline__ T w_h(const DevGrid &G, const L &ld, int dir, int i, int j, int k, T wa)
{
    const int nz = G.nz;
    const bool fd4 = G.mom_ord == 4;
    const double d = dir == 0 ? G.dx : G.dy;
    const double d1 = 1. / d, d3 = 1. / (3. * d);
    const double c1 = fd4 ? 9. / 8. : 1., c2 = fd4 ? 1. / 8. : 0.;
    auto HT = [&](int p, int q) { return dir == 0 ? ld.t(0, p, j, q) : ld.t(1, i, p, q); };
    auto Wm = [&](int p, int q) { return dir == 0 ? ld.m(2, p, j, q) : ld.m(2, i, p, q); };
    const int s = dir == 0 ? i : j;
    auto FF = [&](int p) -> T {
        T uu;
        if (k == 2) uu = (HT(p + 1, 2) + HT(p + 1, 1)) * T(0.5);
        else if (k == nz) uu = (HT(p + 1, nz) + HT(p + 1, nz - 1)) * T(0.5);
        else uu = T(c1) * (HT(p + 1, k) + HT(p + 1, k - 1)) * T(0.5) - T(c2) * (HT(p + 1, k + 1) + HT(p + 1, k - 2)) * T(0.5);
        const T fr = (Wm(p + 1, k) + Wm(p, k)) * T(0.5);
        return uu * fr;
    };
    wa = wa + T(c1) * (FF(s) - FF(s - 1)) * T(d1) - T(c2) * (FF(s + 1) - FF(s - 2)) * T(d3);
    if (G.lavisc) {
        const T mu = T(0.25) * dabs(HT(s, k) + HT(s, k - 1) + HT(s + 1, k) + HT(s + 1, k - 1)) * T(d1);
        wa = wa - T(AVISC) * mu * (-Wm(s + 2, k) + T(4.) * Wm(s + 1, k) - T(6.) * Wm(s, k) + T(4.) * Wm(s - 1, k) - Wm(s - 2, k));
    }
    return wa;
}

template <typename T, class L>
__device__ __forceinline__ T w_z(const DevGrid &G, const L &ld, int i, int j, int k, T wa)
{
    const int nz = G.nz;
    const bool fd4 = G.mom_ord == 4;
    const double c1 = fd4 ? 4. / 3. : 1., c2 = fd4 ? 1. / 3. : 0.;
    auto dzw = [&](int q) { return __ldg(G.dzw + q - 1); };
    auto dz1 = [&](int q) { return __ldg(G.dz1 + q - 1); };
    auto W = [&](int q) { return ld.m(2, i, j, q); };
    auto WT = [&](int q) { return ld.t(2, i, j, q); };
    auto F = [&](int q) -> T {
        if (q == nz - 1) return T(0.25) * (WT(nz) + WT(nz - 1)) * (W(nz) + W(nz - 1));
        return ((WT(q + 1) + WT(q)) * T(0.5)) * ((W(q + 1) + W(q)) * T(0.5));
    };
    auto A = [&](int q) -> T {
        if (q == nz - 1) {
            const double s = dzw(nz) + dzw(nz - 1);
            return (T(0.) + T(dzw(nz - 1)) * WT(nz - 1)) * (T(0.) + T(dzw(nz - 1)) * W(nz - 1)) / T(s * s);
        }
        const T ww2 = (T(dzw(q + 1)) * WT(q + 2) + T(dzw(q)) * WT(q)) / T(dzw(q + 1) + dzw(q));
        const T fr2 = (T(dzw(q + 1)) * W(q + 2) + T(dzw(q)) * W(q)) / T(dzw(q + 1) + dzw(q));
        return ww2 * fr2;
    };
    if (k >= 3 && k <= nz - 1)
        wa = wa + T(c1) * (F(k) - F(k - 1)) * T(dz1(k - 1)) - T(c2) * (A(k) - A(k - 2)) / T(dzw(k) + dzw(k - 1));
    else if (k == 2)
        wa = wa + T(c1) * (F(2) - F(1)) * T(dz1(1)) - T(c2) * (A(2) - T(0.)) / T(dzw(2) + dzw(1));
    else if (k == nz)
        wa = wa + (T(0.) - F(nz - 1)) * T(dz1(nz - 1));
    if (G.lavisc && k >= 3 && k <= nz - 2) {
        const T mu = dabs(WT(k)) * T(dz1(k - 1));
        wa = wa - T(AVISC) * mu * (-W(k + 2) + T(4.) * W(k + 1) - T(6.) * W(k) + T(4.) * W(k - 1) - W(k - 2));
    }
    return wa;
}

// component c (0 u, 1 v, 2 w) of qnadv_uvw at interior cell (i,j,k): even ntime x, y, z;
// odd ntime z, y, x (windadv.f90:58-76)
template <typename T, class L>
__device__ __forceinline__ T adv_comp(const DevGrid &G, const L &ld, int c, int ntime, int i, int j, int k)
{
    T a = T(0.);
    if (c == 2 && k == 1) return a;   // w(1): the surface, no advective tendency
    const bool even = (ntime % 2) == 0;
    for (int pass = 0; pass < 3; pass++) {
        const int dir = even ? pass : 2 - pass;
        if (c == 0) a = dir == 0 ? u_x(G, ld, i, j, k, a) : (dir == 1 ? u_y(G, ld, i, j, k, a) : h_z(G, ld, 0, i, j, k, a));
        else if (c == 1) a = dir == 0 ? v_x(G, ld, i, j, k, a) : (dir == 1 ? v_y(G, ld, i, j, k, a) : h_z(G, ld, 1, i, j, k, a));
        else a = dir == 0 ? w_h(G, ld, 0, i, j, k, a) : (dir == 1 ? w_h(G, ld, 1, i, j, k, a) : w_z(G, ld, i, j, k, a));
    }
    return a;
}

// ---------------- loaders ----------------
struct Mom3 {
    const double *m[3];
};

// values and one tangent
struct LoadTL {
    const DevGrid &G;
    Mom3 v, d;
    __device__ D<1> m(int f, int i, int j, int k) const
    {
        const long long q = gidx(G, i, j, k);
        D<1> r(__ldg(v.m[f] + q));
        r.d[0] = __ldg(d.m[f] + q);
        return r;
    }
    __device__ D<1> t(int f, int i, int j, int k) const { return adv_vel(G, f, k, m(f, i, j, k)); }
};

// ---------------- kernels ----------------
__global__ void __launch_bounds__(128) mom_tl_kernel(DevGrid G, int ntime, Mom3 v, Mom3 d, Mom3 val, Mom3 tan)
{
    const int i = 4 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 4 + blockIdx.y;
    const int k = 1 + blockIdx.z;
    if (i > G.nx - 2) return;
    const LoadTL ld{G, v, d};
    const long long q = gidx(G, i, j, k);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const D<1> a = adv_comp<D<1>>(G, ld, c, ntime, i, j, k);
        if (val.m[c]) const_cast<double *>(val.m[c])[q] = a.v;
        const_cast<double *>(tan.m[c])[q] = a.d[0];
    }
}

}  // namespace

// val (optional) := qnadv_uvw(m) (positive convention), tan := its derivative along dm
cudaError_t launch_qnadv_tl(const DevGrid &g, int ntime, const double *mu, const double *mv, const double *mw,
                            const double *dmu, const double *dmv, const double *dmw, double *au, double *av, double *aw,
                            double *dau, double *dav, double *daw, cudaStream_t s)
{
    const dim3 grid((g.maxx + 127) / 128, g.maxy, g.nz);
    mom_tl_kernel<<<grid, 128, 0, s>>>(g, ntime, Mom3{{mu, mv, mw}}, Mom3{{dmu, dmv, dmw}}, Mom3{{au, av, aw}},
                                       Mom3{{dau, dav, daw}});
    return cudaGetLastError();
}
