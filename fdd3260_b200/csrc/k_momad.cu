// k_momad.cu -- adjoint of the momentum advection operator qnadv_uvw
// (src/INTEG/windadv.f90:46-79 with uadv_fd :82-220, vadv_fd :223-357, wadv_fd :360-492 and
// the stencils :494-1127), FD4/FD2 with the artificial viscosity; its tangent linear is in
// k_momadj.cu.
//   The transposed stencils, hand-written in gather form (one thread per input cell sums what
//   every face flux and viscosity term that reads the cell passes back); no atomics.  What the
//   forward reads through periodic ghost images lands on the interior cells they copy, so the
//   ghosts of the result stay 0.
// Unlike the tangent, nothing here has to equal another evaluation bit for bit: the file is
// compiled with contraction, and the level and grid constants are divided by through their
// reciprocals.
#include "mg_common.cuh"

namespace {

constexpr double AVISC = 1. / 16.;   // windadv.f90:39

struct Mom3 {
    const double *m[3];
};

// ---------------- adjoint: the transposed stencils in gather form ----------------
// Each direction term is a sum of face fluxes Phi = a * b with constant coefficients
// (a: an average of advective velocities, b: an average of the advected momentum; the
// coefficients of the vertical terms depend on the level, as the forward's branches at
// the surface and the lid), plus the artificial viscosity mu |velocity| D4(momentum).
// The adjoint at an input cell sums, over every face that reads the cell, Phi-bar (the
// coefficient-weighted adjoints of the outputs that difference the face) times the
// partial of Phi, and likewise over the viscosity terms.  Positions wrap periodically in
// x and y, so what the forward reads through a ghost image is gathered by the interior
// cell it copies; outputs outside 1..nz (and w at the surface) do not exist.

// 1/dx, 1/(2 dx), 1/(3 dx) of x and y
struct RSpace {
    double h1[2], h2[2], h3[2];
};

__device__ __forceinline__ double sgnd(double x) { return x < 0. ? -1. : 1.; }   // d|x|/dx as dabs takes it
__device__ __forceinline__ double w4(int d) { return d == 0 ? -6. : ((d == 1 || d == -1) ? 4. : -1.); }

template <bool CORE> struct Gath {
    const DevGrid &G;
    const RSpace &H;
    Mom3 m, ab;
    double c1s, c2s, c1c, c2c;
    int i0, j0, k0;   // the thread's cell: every position is addressed from its index
    long long q0;
    __device__ Gath(const DevGrid &g, const RSpace &h, Mom3 m_, Mom3 ab_, int i, int j, int k)
        : G(g), H(h), m(m_), ab(ab_), i0(i), j0(j), k0(k)
    {
        const bool fd4 = g.mom_ord == 4;
        c1s = fd4 ? 4. / 3. : 1.; c2s = fd4 ? 1. / 3. : 0.;
        c1c = fd4 ? 9. / 8. : 1.; c2c = fd4 ? 1. / 8. : 0.;
        q0 = gidx(g, i, j, k);
    }
    // (along, transverse) -> (i, j): direction 0 is x, 1 is y
    __device__ static int ci(int dir, int a, int t) { return dir == 0 ? a : t; }
    __device__ static int cj(int dir, int a, int t) { return dir == 0 ? t : a; }
    // the positions visited lie within 2 cells of the thread's (outputs) or 3 (momenta);
    // only a viscosity term three cells along reads past the last ghost, and is moved to
    // its periodic image
    __device__ int img_a(int dir, int a) const
    {
        return dir == 0 ? (a + 1 > G.nx ? a - G.maxx : a) : (a + 1 > G.ny ? a - G.maxy : a);
    }
    __device__ long long idx(int i, int j, int k) const
    {
        return q0 + (i - i0) + (long long)(j - j0) * G.px + (long long)(k - k0) * G.ps;
    }
    __device__ double M(int f, int i, int j, int k) const { return __ldg(m.m[f] + idx(i, j, k)); }
    // advective velocity with the reciprocal profiles (its partial is the same factor)
    __device__ double T(int f, int i, int j, int k) const
    {
        const double x = M(f, i, j, k) * rden(f, k);
        return f == 0 ? x - G.u0shift : (f == 1 ? x - G.v0shift : x);
    }
    // output adjoints, halo-filled: the ghost cells hold the periodic images
    __device__ double A(int c, int i, int j, int k) const
    {
        if (!CORE && (k < 1 || k > G.nz || (c == 2 && k == 1))) return 0.;
        return __ldg(ab.m[c] + idx(i, j, k));
    }
    __device__ double Ma(int f, int dir, int a, int t, int k) const { return M(f, ci(dir, a, t), cj(dir, a, t), k); }
    __device__ double Ta(int f, int dir, int a, int t, int k) const { return T(f, ci(dir, a, t), cj(dir, a, t), k); }
    __device__ double Aa(int c, int dir, int a, int t, int k) const { return A(c, ci(dir, a, t), cj(dir, a, t), k); }
    __device__ double rden(int f, int k) const { return __ldg((f == 2 ? G.ravden0 : G.rden0) + k - 1); }
    __device__ double dzw(int q) const { return __ldg(G.dzw + q - 1); }
    __device__ double dz1w(int q) const { return __ldg(G.dz1w + q - 1); }
    __device__ double dz1(int q) const { return __ldg(G.dz1 + q - 1); }
    // 1 / (dzw(q) + dzw(q+1)) and 1 / (dzw(q-1) + dzw(q) + dzw(q+1))
    __device__ double rzs(int q) const { return __ldg(&reinterpret_cast<const K2Coef<double> *>(G.k2tab)[q - 1].rzs); }
    __device__ double rs3(int q) const { return __ldg(&reinterpret_cast<const K2Coef<double> *>(G.k2tab)[q - 1].rs3); }
    // level k lies outside lo..hi (from a core level nothing does)
    __device__ bool off(int k, int lo, int hi) const { return !CORE && (k < lo || k > hi); }
    __device__ double d1(int dir) const { return H.h1[dir]; }

    // ---- u_x (f 0, dir x) and v_y (f 1, dir y): the advected field is its own velocity ----
    __device__ double self_h(int f, int i, int j, int k) const
    {
        const int dir = f, a0 = dir == 0 ? i : j, t = dir == 0 ? j : i;
        const double h1 = d1(dir), h2 = H.h2[dir], rd = rden(f, k);
        double r = 0.;
        for (int p = a0 - 1; p <= a0; p++) {   // F(p) = avg T(p, p+1) * avg m(p, p+1)
            const double fb = c1s * h1 * (Aa(f, dir, p, t, k) - Aa(f, dir, p + 1, t, k));
            r += fb * 0.5 * (0.5 * (Ma(f, dir, p + 1, t, k) + Ma(f, dir, p, t, k)) * rd +
                             0.5 * (Ta(f, dir, p + 1, t, k) + Ta(f, dir, p, t, k)));
        }
        for (int p = a0 - 2; p <= a0; p += 2) {   // A(p) = avg T(p, p+2) * avg m(p, p+2)
            const double gb = c2s * h2 * (Aa(f, dir, p + 2, t, k) - Aa(f, dir, p, t, k));
            r += gb * 0.5 * (0.5 * (Ma(f, dir, p + 2, t, k) + Ma(f, dir, p, t, k)) * rd +
                             0.5 * (Ta(f, dir, p + 2, t, k) + Ta(f, dir, p, t, k)));
        }
        if (G.lavisc) {
            for (int o = a0 - 2; o <= a0 + 2; o++) r -= AVISC * h1 * Aa(f, dir, o, t, k) * fabs(Ta(f, dir, o, t, k)) * w4(a0 - o);
            const double d4 = -Ma(f, dir, a0 + 2, t, k) + 4. * Ma(f, dir, a0 + 1, t, k) - 6. * Ma(f, dir, a0, t, k) +
                              4. * Ma(f, dir, a0 - 1, t, k) - Ma(f, dir, a0 - 2, t, k);
            r -= AVISC * h1 * Aa(f, dir, a0, t, k) * sgnd(Ta(f, dir, a0, t, k)) * rd * d4;
        }
        return r;
    }

    // ---- u_y (c 0: dir y, velocity v) and v_x (c 1: dir x, velocity u) ----
    // face bar at along-position q of line t
    __device__ double cross_fbar(int c, int dir, int q, int t, int k) const
    {
        const double h1 = d1(dir), h3 = H.h3[dir];
        return c1c * h1 * (Aa(c, dir, q, t, k) - Aa(c, dir, q + 1, t, k)) - c2c * h3 * Aa(c, dir, q - 1, t, k) +
               c2c * h3 * Aa(c, dir, q + 2, t, k);
    }
    // partial wrt the advected momentum c at its own cell
    __device__ double cross_adv(int c, int i, int j, int k) const
    {
        const int dir = 1 - c, g = 1 - c;
        const int a0 = dir == 0 ? i : j, t = dir == 0 ? j : i;
        double r = 0.;
        for (int q = a0 - 1; q <= a0; q++) {
            const double vel = c1c * (Ta(g, dir, q + 1, t - 1, k) + Ta(g, dir, q + 1, t, k)) * 0.5 -
                               c2c * (Ta(g, dir, q + 1, t - 2, k) + Ta(g, dir, q + 1, t + 1, k)) * 0.5;
            r += cross_fbar(c, dir, q, t, k) * 0.5 * vel;
        }
        if (G.lavisc)
            for (int o = a0 - 2; o <= a0 + 2; o++) {
                const int ob = img_a(dir, o);
                const double mu = 0.25 * fabs(Ta(g, dir, ob, t - 1, k) + Ta(g, dir, ob, t, k) + Ta(g, dir, ob + 1, t - 1, k) +
                                              Ta(g, dir, ob + 1, t, k)) * d1(dir);
                r -= AVISC * Aa(c, dir, ob, t, k) * mu * w4(a0 - o);
            }
        return r;
    }
    // partial wrt the advecting momentum g = 1 - c at its own cell
    __device__ double cross_vel(int c, int i, int j, int k) const
    {
        const int dir = 1 - c, g = 1 - c;
        const int a0 = dir == 0 ? i : j, t0 = dir == 0 ? j : i;
        const double rd = rden(g, k);
        double r = 0.;
        const int ds[4] = {-1, 0, -2, 1};
        for (int n = 0; n < 4; n++) {   // the velocity at transverse offset d of line t = t0 - d, face q = a0 - 1
            const int t = t0 - ds[n];
            const double gam = n < 2 ? 0.5 * c1c : -0.5 * c2c;
            const double fr = 0.5 * (Ma(c, dir, a0, t, k) + Ma(c, dir, a0 - 1, t, k));
            r += cross_fbar(c, dir, a0 - 1, t, k) * fr * gam * rd;
        }
        if (G.lavisc)
            for (int t = t0; t <= t0 + 1; t++)
                for (int o = a0 - 1; o <= a0; o++) {
                    const double s = Ta(g, dir, o, t - 1, k) + Ta(g, dir, o, t, k) + Ta(g, dir, o + 1, t - 1, k) +
                                     Ta(g, dir, o + 1, t, k);
                    const double d4 = -Ma(c, dir, o + 2, t, k) + 4. * Ma(c, dir, o + 1, t, k) - 6. * Ma(c, dir, o, t, k) +
                                      4. * Ma(c, dir, o - 1, t, k) - Ma(c, dir, o - 2, t, k);
                    r -= AVISC * Aa(c, dir, o, t, k) * d4 * 0.25 * d1(dir) * sgnd(s) * rd;
                }
        return r;
    }

    // ---- h_z (f 0: u with w at x offsets; f 1: v with w at y offsets) ----
    // coefficient of face flux F(q) in the output at level ko (advhz's branches)
    __device__ double hz_coef(int f, int ko, int q) const
    {
        const int nz = G.nz;
        if (!off(ko, 3, nz - 1)) {
            if (q == ko) return c1c * dz1w(ko);
            if (q == ko - 1) return -c1c * dz1w(ko);
            if (q == ko + 1) return -c2c * rs3(ko);
            if (q == ko - 2) return c2c * rs3(ko);
            return 0.;
        }
        if (ko == 1) return q == 1 ? dz1w(1) : 0.;
        if (ko == 2) {
            const double mz = dz1w(f == 1 ? 2 : 1);
            if (q == 2) return c1c * mz;
            if (q == 1) return -c1c * mz;
            if (q == 3) return -c2c * rs3(2);
            return 0.;
        }
        return q == nz - 1 ? -dz1w(nz) : 0.;   // ko == nz
    }
    __device__ double hz_fbar(int f, int i, int j, int q) const
    {
        double r = 0.;
        for (int ko = q - 1; ko <= q + 2; ko++)
            if (!off(ko, 1, G.nz)) r += A(f, i, j, ko) * hz_coef(f, ko, q);
        return r;
    }
    __device__ double WTo(int f, int i, int j, int d, int q) const { return f == 0 ? T(2, i + d, j, q) : T(2, i, j + d, q); }
    __device__ double hz_adv(int f, int i, int j, int k) const
    {
        const int nz = G.nz;
        double r = 0.;
        for (int q = k - 1; q <= k; q++) {
            if (off(q, 1, nz - 1)) continue;
            const double ww = c1c * (WTo(f, i, j, -1, q + 1) + WTo(f, i, j, 0, q + 1)) * 0.5 -
                              c2c * (WTo(f, i, j, -2, q + 1) + WTo(f, i, j, 1, q + 1)) * 0.5;
            const double wgt = (q == k ? dzw(q) : dzw(q + 1)) * rzs(q);
            r += hz_fbar(f, i, j, q) * ww * wgt;
        }
        if (G.lavisc)
            for (int ko = k - 2; ko <= k + 2; ko++) {
                if (off(ko, 3, nz - 2)) continue;
                const double mu = 0.25 * fabs(WTo(f, i, j, -1, ko) + WTo(f, i, j, 0, ko) + WTo(f, i, j, -1, ko + 1) +
                                              WTo(f, i, j, 0, ko + 1)) * dz1w(ko);
                r -= AVISC * A(f, i, j, ko) * mu * w4(k - ko);
            }
        return r;
    }
    __device__ double hz_w(int f, int i, int j, int k) const   // partial wrt w at (i, j, k)
    {
        const int nz = G.nz;
        const double ra = rden(2, k);
        double r = 0.;
        const int q = k - 1;
        if (!off(q, 1, nz - 1)) {
            const int ds[4] = {-1, 0, -2, 1};
            for (int n = 0; n < 4; n++) {
                const int ii = f == 0 ? i - ds[n] : i, jj = f == 0 ? j : j - ds[n];
                const double gam = n < 2 ? 0.5 * c1c : -0.5 * c2c;
                const double fr = (dzw(q + 1) * M(f, ii, jj, q + 1) + dzw(q) * M(f, ii, jj, q)) * rzs(q);
                r += hz_fbar(f, ii, jj, q) * fr * gam * ra;
            }
        }
        if (G.lavisc)
            for (int s = 0; s <= 1; s++) {   // outputs at the column itself and one further along
                const int ii = f == 0 ? i + s : i, jj = f == 0 ? j : j + s;
                for (int ko = k - 1; ko <= k; ko++) {
                    if (off(ko, 3, nz - 2)) continue;
                    const double sw = WTo(f, ii, jj, -1, ko) + WTo(f, ii, jj, 0, ko) + WTo(f, ii, jj, -1, ko + 1) +
                                      WTo(f, ii, jj, 0, ko + 1);
                    const double d4 = -M(f, ii, jj, ko + 2) + 4. * M(f, ii, jj, ko + 1) - 6. * M(f, ii, jj, ko) +
                                      4. * M(f, ii, jj, ko - 1) - M(f, ii, jj, ko - 2);
                    r -= AVISC * A(f, ii, jj, ko) * d4 * 0.25 * dz1w(ko) * sgnd(sw) * ra;
                }
            }
        return r;
    }

    // ---- w_h (dir 0: velocity u along x; dir 1: v along y), outputs w at levels 2..nz ----
    // weight of the velocity at level q in uu of the output at level kw
    __device__ double wh_lam(int kw, int q) const
    {
        const int nz = G.nz;
        if (!CORE && kw == 2) return (q == 2 || q == 1) ? 0.5 : 0.;
        if (!CORE && kw == nz) return (q == nz || q == nz - 1) ? 0.5 : 0.;
        if (q == kw || q == kw - 1) return 0.5 * c1c;
        if (q == kw + 1 || q == kw - 2) return -0.5 * c2c;
        return 0.;
    }
    __device__ double wh_fbar(int dir, int p, int t, int kw) const { return cross_fbar(2, dir, p, t, kw); }
    __device__ double wh_w(int dir, int i, int j, int k) const   // partial wrt w (advected) at (i, j, k)
    {
        if (off(k, 2, G.nz)) return 0.;
        const int a0 = dir == 0 ? i : j, t = dir == 0 ? j : i;
        double r = 0.;
        for (int p = a0 - 1; p <= a0; p++) {
            double uu = 0.;
            for (int q = k - 2; q <= k + 1; q++) {
                const double l = wh_lam(k, q);
                if (CORE || l != 0.) uu += l * Ta(dir, dir, p + 1, t, q);
            }
            r += wh_fbar(dir, p, t, k) * 0.5 * uu;
        }
        if (G.lavisc)
            for (int o = a0 - 2; o <= a0 + 2; o++) {
                const int ob = img_a(dir, o);
                const double mu = 0.25 * fabs(Ta(dir, dir, ob, t, k) + Ta(dir, dir, ob, t, k - 1) + Ta(dir, dir, ob + 1, t, k) +
                                              Ta(dir, dir, ob + 1, t, k - 1)) * d1(dir);
                r -= AVISC * Aa(2, dir, ob, t, k) * mu * w4(a0 - o);
            }
        return r;
    }
    __device__ double wh_vel(int dir, int i, int j, int k) const   // partial wrt the velocity momentum (u or v)
    {
        const int nz = G.nz;
        const int a0 = dir == 0 ? i : j, t = dir == 0 ? j : i;
        const double rd = rden(dir, k);
        double r = 0.;
        for (int kw = k - 1; kw <= k + 2; kw++) {
            if (off(kw, 2, nz)) continue;
            const double l = wh_lam(kw, k);
            if (!CORE && l == 0.) continue;
            const double fr = 0.5 * (Ma(2, dir, a0, t, kw) + Ma(2, dir, a0 - 1, t, kw));
            r += wh_fbar(dir, a0 - 1, t, kw) * fr * l * rd;
        }
        if (G.lavisc)
            for (int kw = k; kw <= k + 1; kw++) {
                if (off(kw, 2, nz)) continue;
                for (int o = a0 - 1; o <= a0; o++) {
                    const double s = Ta(dir, dir, o, t, kw) + Ta(dir, dir, o, t, kw - 1) + Ta(dir, dir, o + 1, t, kw) +
                                     Ta(dir, dir, o + 1, t, kw - 1);
                    const double d4 = -Ma(2, dir, o + 2, t, kw) + 4. * Ma(2, dir, o + 1, t, kw) - 6. * Ma(2, dir, o, t, kw) +
                                      4. * Ma(2, dir, o - 1, t, kw) - Ma(2, dir, o - 2, t, kw);
                    r -= AVISC * Aa(2, dir, o, t, kw) * d4 * 0.25 * d1(dir) * sgnd(s) * rd;
                }
            }
        return r;
    }

    // ---- w_z, outputs w at levels 2..nz ----
    __device__ double wz_fcoef(int ko, int q) const
    {
        const int nz = G.nz;
        if (!off(ko, 3, nz - 1)) return q == ko ? c1s * dz1(ko - 1) : (q == ko - 1 ? -c1s * dz1(ko - 1) : 0.);
        if (ko == 2) return q == 2 ? c1s * dz1(1) : (q == 1 ? -c1s * dz1(1) : 0.);
        if (ko == nz) return q == nz - 1 ? -dz1(nz - 1) : 0.;
        return 0.;
    }
    __device__ double wz_acoef(int ko, int q) const
    {
        const int nz = G.nz;
        if (!off(ko, 3, nz - 1)) return q == ko ? -c2s * rzs(ko - 1) : (q == ko - 2 ? c2s * rzs(ko - 1) : 0.);
        if (ko == 2) return q == 2 ? -c2s * rzs(1) : 0.;
        return 0.;
    }
    __device__ double wz_w(int i, int j, int k) const
    {
        const int nz = G.nz;
        const double ra = rden(2, k);
        auto W = [&](int q) { return M(2, i, j, q); };
        auto WT = [&](int q) { return T(2, i, j, q); };
        double r = 0.;
        for (int q = k - 1; q <= k; q++) {   // F(q) = avg WT(q, q+1) * avg W(q, q+1)
            if (off(q, 1, nz - 1)) continue;
            const double fb = A(2, i, j, q) * wz_fcoef(q, q) + A(2, i, j, q + 1) * wz_fcoef(q + 1, q);
            r += fb * 0.25 * ((W(q + 1) + W(q)) * ra + (WT(q + 1) + WT(q)));
        }
        for (int q = k - 2; q <= k; q += 2) {   // A(q): W(q) and W(q+2), or W(nz-1) alone at q = nz-1
            if (off(q, 1, nz - 1)) continue;
            const double gb = A(2, i, j, q) * wz_acoef(q, q) + A(2, i, j, q + 2) * wz_acoef(q + 2, q);
            if (!CORE && gb == 0.) continue;
            if (!CORE && q == nz - 1) {
                if (k != q) continue;
                const double dl = dzw(nz - 1) * rzs(nz - 1);
                r += gb * dl * dl * (W(q) * ra + WT(q));
            } else {
                const double al = dzw(q + 1) * rzs(q), be = dzw(q) * rzs(q);
                const double ww2 = al * WT(q + 2) + be * WT(q), fr2 = al * W(q + 2) + be * W(q);
                r += gb * (k == q + 2 ? al : be) * (fr2 * ra + ww2);
            }
        }
        if (G.lavisc) {
            for (int ko = k - 2; ko <= k + 2; ko++) {
                if (off(ko, 3, nz - 2)) continue;
                r -= AVISC * A(2, i, j, ko) * fabs(WT(ko)) * dz1(ko - 1) * w4(k - ko);
            }
            if (!off(k, 3, nz - 2)) {
                const double d4 = -W(k + 2) + 4. * W(k + 1) - 6. * W(k) + 4. * W(k - 1) - W(k - 2);
                r -= AVISC * A(2, i, j, k) * dz1(k - 1) * sgnd(WT(k)) * ra * d4;
            }
        }
        return r;
    }
};

// component C of the result at one cell
template <int C, bool CORE>
__device__ __forceinline__ void gather_cell(const DevGrid &G, const RSpace &H, const Mom3 &v, const Mom3 &ab, const Mom3 &bar,
                                            int i, int j, int k)
{
    const Gath<CORE> g(G, H, v, ab, i, j, k);
    double r;
    if constexpr (C == 0)   // u: u_x, u_y (advected), h_z (f 0, advected), v_x (velocity), w_h x (velocity)
        r = g.self_h(0, i, j, k) + g.cross_adv(0, i, j, k) + g.hz_adv(0, i, j, k) + g.cross_vel(1, i, j, k) +
            g.wh_vel(0, i, j, k);
    else if constexpr (C == 1)   // v: v_y, v_x (advected), h_z (f 1, advected), u_y (velocity), w_h y (velocity)
        r = g.self_h(1, i, j, k) + g.cross_adv(1, i, j, k) + g.hz_adv(1, i, j, k) + g.cross_vel(0, i, j, k) +
            g.wh_vel(1, i, j, k);
    else   // w: w_z, w_h x and y (advected), h_z f 0 and f 1 (velocity)
        r = g.wz_w(i, j, k) + g.wh_w(0, i, j, k) + g.wh_w(1, i, j, k) + g.hz_w(0, i, j, k) + g.hz_w(1, i, j, k);
    const_cast<double *>(bar.m[C])[g.q0] += r;
}

// one output component per launch (C: 0 u, 1 v, 2 w): a third of the code each.  Bound by the
// instructions issued and the L1 wavefronts of ~100 double loads a cell; levels away from the surface
// and the lid take a straight-line instance, whose loads the compiler can share between the terms.
// u / v / w at 128 x 128 x 96: 168 / 199 / 293 us with divisions, level branches and no contraction,
// 119 / 116 / 144 us now.
template <int C>
__global__ void __launch_bounds__(128) mom_ad_gather_kernel(const __grid_constant__ DevGrid G, const __grid_constant__ RSpace H,
                                                            Mom3 v, Mom3 ab, Mom3 bar)
{
    const int i = 4 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 4 + blockIdx.y;
    const int k = 1 + blockIdx.z;
    if (i > G.nx - 2) return;
    if (k >= 5 && k <= G.nz - 4) gather_cell<C, true>(G, H, v, ab, bar, i, j, k);
    else gather_cell<C, false>(G, H, v, ab, bar, i, j, k);
}

}  // namespace

// bar += (d qnadv / d m)^T abar (bar arrays must be zeroed by the caller for a plain adjoint);
// abar is read on the interior (its ghost cells are overwritten with periodic images),
// the ghost entries of bar are left as they are
cudaError_t launch_qnadv_ad(const DevGrid &g, const double *mu, const double *mv, const double *mw, double *aubar,
                            double *avbar, double *awbar, double *mubar, double *mvbar, double *mwbar, cudaStream_t s)
{
    double *ab[3] = {aubar, avbar, awbar};
    cudaError_t e = launch_halo_fill(g, ab, 3, s);
    if (e != cudaSuccess) return e;
    const dim3 grid((g.maxx + 127) / 128, g.maxy, g.nz);
    const Mom3 v{{mu, mv, mw}}, ab3{{aubar, avbar, awbar}}, bar{{mubar, mvbar, mwbar}};
    const RSpace h{{1. / g.dx, 1. / g.dy}, {1. / (2. * g.dx), 1. / (2. * g.dy)}, {1. / (3. * g.dx), 1. / (3. * g.dy)}};
    mom_ad_gather_kernel<0><<<grid, 128, 0, s>>>(g, h, v, ab3, bar);
    mom_ad_gather_kernel<1><<<grid, 128, 0, s>>>(g, h, v, ab3, bar);
    mom_ad_gather_kernel<2><<<grid, 128, 0, s>>>(g, h, v, ab3, bar);
    return cudaGetLastError();
}
