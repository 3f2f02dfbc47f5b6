// k1_body.cuh -- body of the K1 kernel (scalar advection + stage update), templated
// on the scheme, the arithmetic form and the stage; instantiated by k_scalar.cu (plain
// FP64, compiled without FMA contraction) and k_scalar_mixed.cu (FP32 scheme logic on
// differences, FP64 fluxes and state).
//
// One CTA (8 warps) owns a 32 x 8 column tile and a segment [kb, ke] of its levels (ColSplit:
// small grids fill the GPU and the last wave of CTAs is short).
// It takes the fields in groups of PF (2 for WENO, MUSCL, lw and QUICK, 1 for PPM, whose
// per-field reconstruction arrays are large) and marches each group up the segment in a pass
// of its own: what the column carries (the vertical window x(k-1..k+L), the flux below) is
// then a few registers of two fields, and the shared memory does not grow with the field
// count.  (Marching all fields together kept the windows of every field in shared memory,
// 110 KB at 6 fields and more than one CTA's share beyond, read and written on every level.)
//
// A segment above the surface starts with NPRO prologue levels that compute only vertical
// faces: the flux that the first level differences is the same arithmetic on the same values
// as in the segment below, so the result does not depend on the split.  PPM needs three such
// levels, for the reconstruction carried up the column.
//
// Per level: the group's haloed planes arrive by TMA, L+1 levels ahead of the level whose
// faces read them, in a ring of L+2 slots, since the own column's newest window value is
// taken from the plane as it arrives (stage 1 forms psi = s * rho there, in place); the x/y
// faces of level k are computed as independent chains, one barrier publishes them (into two
// buffers in turn), then each thread finishes the vertical face and the stage update.
//
// Stage 2 divides every scalar by the cell's new density, which the first pass computes: it
// is kept in the density's tendency accumulator (read for the last time by that pass), and
// the level-n density, which the later passes weigh the old values with, is overwritten by
// the last pass.
//
// Bound by the latency of dependent FP64 (mixed: FP32 and conversion) operations at the 16 warps
// that two CTAs hold: issue 54-62 % active in the mixed form, no memory unit above 30 %.  Per launch
// at 512x512x256 with 6 fields, averaged over the stages: FP64 14.83 -> 9.43 ms, mixed 7.35 -> 6.76
// ms against the marching of all fields together; PPM at 160x128x64 1.53 -> 0.42 ms.
#pragma once
#include <algorithm>
#include <type_traits>
#include "mg_common.cuh"
#include "schemes.cuh"
#include "tma.cuh"

namespace {

constexpr int TX = 32, TY = 8, H = 3;
constexpr int SW = TX + 2 * H, SH = TY + 2 * H;   // haloed plane box 38 x 14
constexpr int NTH = TX * TY;                      // 256 threads
constexpr int PLANE_BYTES = SW * SH * 8;          // 4256
constexpr int PLANE_SLOT = 4352;                  // 128-byte multiple
constexpr int VW = 34, VH = 9;                    // momentum box (x from i0-1, y from j0)
constexpr int VBOX_BYTES = VW * VH * 8;           // 2448
constexpr int VBOX_SLOT = 2560;
constexpr int NCELL = TX * TY;
constexpr int FXN = TY * (TX + 1), FYN = (TY + 1) * TX;   // x faces, y faces of one field
constexpr int XE = FXN - NCELL;                   // x faces beyond the cell threads' own
constexpr int NHALO = SW * SH - TX * TY;          // 276 plane elements outside the cells
// per-level coefficients in shared memory, written two levels ahead by the last warp: the
// shared memory of two CTAs leaves next to no L1, so every profile load was an L2
// round trip in front of a level's first faces
constexpr int NCS = 4;                            // level slots
__host__ __device__ constexpr int k1_ncoef(int scheme) { return scheme == MG_PPM ? 24 : 16; }   // doubles per level
enum { C_D0, C_RD0, C_AW, C_RAW, C_DZW, C_RDZW, C_D1M, C_D10, C_D1P, C_FM, C_FP, C_N };   // then PPM's face-value coefficients (FP64)
static_assert(C_N <= 16 && C_N + PPM_NC <= 24, "one lane of a warp each");

// fields per group: three where the registers allow, since a level of a pass costs about half
// of its instructions whatever the group (velocities, waits, halo products, loop)
__host__ __device__ constexpr int k1_pf(int scheme, bool mixed) { return scheme == MG_PPM ? 1 : (mixed && scheme == MG_WENO ? 3 : 2); }
__host__ __device__ constexpr int k1_win(int scheme) { return scheme == MG_PPM ? 3 : 2; }   // L: window x(k-1 .. k+L)
__host__ __device__ constexpr int k1_nrho(int scheme) { return k1_win(scheme) + 1; }        // density planes in flight (stage 1)
// CTAs per SM: two of 128 registers a thread in both forms (FP64 at 96 registers spilled to an
// L1 that hardly exists; the mixed form at 80, three CTAs, was slower)
constexpr int K1_CTAS = 2;

// Stage 2's pointwise operands (level-n values, accumulators, level-n density) wait in shared
// memory, copied asynchronously by the thread that uses them, while the faces are computed: in
// registers they made the FP64 kernels spill.  512x512x256 WENO 9.60 -> 9.43 ms a launch, 150x90x71
// MUSCL 158 -> 156 us; PPM (416 -> 420 us) and the mixed form (6.75 -> 6.82 ms) do not spill and lose.
__host__ __device__ constexpr bool k1_ops(int scheme, int stage, bool mixed) { return stage == 2 && !mixed && scheme != MG_PPM; }

struct Layout {
    size_t planes, rho, vbu, vbv, fx, fy, ops, mbar, coef, crx, cry, total;
};

// stage: 1, 2, or 0 (unit mode); only stage 1 keeps density planes
__host__ __device__ constexpr Layout make_layout(int scheme, bool mixed, int stage)
{
    Layout Ly{};
    const int PF = k1_pf(scheme, mixed), NR = k1_win(scheme) + 2;
    size_t o = 0;
    Ly.planes = o; o += (size_t)NR * PF * PLANE_SLOT;
    Ly.rho = o;
    if (stage == 1) o += (size_t)k1_nrho(scheme) * PLANE_SLOT;
    Ly.vbu = o; o += VBOX_SLOT;
    Ly.vbv = o; o += VBOX_SLOT;
    Ly.fx = o; o += (size_t)2 * PF * FXN * 8;
    Ly.fy = o; o += (size_t)2 * PF * FYN * 8;
    Ly.ops = o;
    if (k1_ops(scheme, stage, mixed)) o += (size_t)(2 * PF + 1) * NCELL * 8;
    o = (o + 127) / 128 * 128;
    Ly.mbar = o; o += 128;
    Ly.coef = o; o += (size_t)NCS * k1_ncoef(scheme) * 8;
    Ly.crx = o;
    Ly.cry = o;
    if (scheme == MG_PPM) {
        o += (size_t)2 * 4 * TY * (TX + 2) * 8;
        Ly.cry = o; o += (size_t)2 * 4 * (TY + 2) * TX * 8;
    }
    Ly.total = o + 128;   // slack for 128-byte alignment of the base
    return Ly;
}

// the fields one launch takes (PPM: the limit of the layout that kept every field's window in
// shared memory, which callers know as an error)
inline int k1_max_fields(int scheme) { return scheme == MG_PPM ? 8 : MG_MAXF; }

// the split of a column tile along k (column_split); a segment's lead is its prologue (three levels
// for PPM) and the pipeline fill
inline ColSplit k1_split(const DevGrid &g, int scheme)
{
    return column_split((long long)((g.maxx + TX - 1) / TX) * ((g.maxy + TY - 1) / TY), g.nz, K1_CTAS,
                           scheme == MG_PPM ? 2.5 : 1.5);
}

__device__ __forceinline__ double ldg(const double *p, long long i) { return __ldg(p + i); }

// plane element of halo index h in [0, NHALO): rows 0..2 and 11..13, then the halo
// columns of the cell rows
__device__ __forceinline__ int halo_elem(int h)
{
    if (h < 2 * H * SW) {
        const int r = h / SW, c = h - r * SW;
        return (r < H ? r : r + TY) * SW + c;
    }
    const int h2 = h - 2 * H * SW, r = h2 / (2 * H), cc = h2 - r * (2 * H);
    return (r + H) * SW + (cc < H ? cc : cc + TX);
}

// ((x - Tx) - Ty) - Tz from the flux differences.  The mixed form's roundings are written out
// (Tx and Ty rounded, Tz contracted), as are those of its stage update below: that translation
// unit is compiled with contraction, and which product a sum absorbs would otherwise change
// with the code around it, which the scheme's switch amplifies.
template <bool MIXED>
__device__ __forceinline__ double k1_tendency(double x, double dFx, double dx1, double dFy, double dy1, double dFz, double dzw1)
{
    if constexpr (MIXED) return __fma_rn(-dFz, dzw1, __dsub_rn(__dsub_rn(x, __dmul_rn(dFx, dx1)), __dmul_rn(dFy, dy1)));
    else return ((x - dFx * dx1) - dFy * dy1) - dFz * dzw1;
}

// N WENO faces in the form's arithmetic
template <bool MIXED, int N>
__device__ __forceinline__ void weno_faces(const double (&xm)[N], const double (&x0)[N], const double (&xp)[N],
                                           const double (&xq)[N], const double (&vel)[N], bool full, double (&Fo)[N])
{
    if constexpr (MIXED) weno_faces_up_mixed<N>(xm, x0, xp, xq, vel, full, Fo);
    else weno_faces_up<N>(xm, x0, xp, xq, vel, full, Fo);
}

// STAGE 1, 2: Heun stage update of density + density-weighted scalars (field 0 is the
// density); STAGE 0: unit mode (advection_ac of one field, xout := ((xout-Tx)-Ty)-Tz)
// SGS: the stage adds stored SGS tendencies (A.sgs); a variant of its own so that the kernels
// without SGS keep their register budget
// bid: the block's index in the domain's own grid of tiles x segments
template <int SCHEME, bool MIXED, int STAGE, bool SGS>
__device__ __forceinline__ void k1_run(const DevGrid &G, const K1Args &A, const K1Maps &M, const int bid)
{
    constexpr int PF = k1_pf(SCHEME, MIXED), L = k1_win(SCHEME), NR = L + 2, NRHO = k1_nrho(SCHEME), NCOEF = k1_ncoef(SCHEME);
    constexpr bool CONV1 = STAGE == 1;   // stage-1 inputs are natural: psi = s * rho
    constexpr bool PAIR = SCHEME == MG_WENO;   // a field's x and y faces as interleaved chains (weno_faces_up*)
    constexpr int NPRO = SCHEME == MG_PPM ? 3 : 1;       // prologue levels of a segment above the surface
    extern __shared__ unsigned char smraw[];
    // 128-byte alignment by an offset from the shared array itself, so that every pointer
    // derived from it stays a shared-memory pointer
    unsigned char *sm = smraw + ((128u - (smem_u32(smraw) & 127u)) & 127u);
    constexpr Layout Ly = make_layout(SCHEME, MIXED, STAGE);
    double *planes = (double *)(sm + Ly.planes), *rhop = (double *)(sm + Ly.rho);
    double *vbu = (double *)(sm + Ly.vbu), *vbv = (double *)(sm + Ly.vbv);
    double *fx = (double *)(sm + Ly.fx), *fy = (double *)(sm + Ly.fy);
    uint64_t *mb = (uint64_t *)(sm + Ly.mbar);    // [0, NR) plane slots, [NR] momentum boxes
    constexpr bool OPS = k1_ops(SCHEME, STAGE, MIXED);
    double *ops = (double *)(sm + Ly.ops) + threadIdx.y * TX + threadIdx.x;   // own operands: [2u] level n, [2u+1] accumulator, [2PF] density
    double *coef = (double *)(sm + Ly.coef);      // [level % NCS][NCOEF]
    double *crx = (double *)(sm + Ly.crx), *cry = (double *)(sm + Ly.cry);   // PPM reconstructions, two buffers

    const int F = A.nf;
    const int ntx = (G.maxx + TX - 1) / TX, nty = (G.maxy + TY - 1) / TY;
    const int tile = bid % (ntx * nty), seg = bid / (ntx * nty);
    const int ti = tile % ntx, tj = tile / ntx;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
    const int i0 = 4 + ti * TX, j0 = 4 + tj * TY;
    const int nx = G.nx, ny = G.ny, nz = G.nz;
    const int i = i0 + tx, j = j0 + ty;
    const bool act = (i <= nx - 2) && (j <= ny - 2);
    const int own_e = (ty + H) * SW + tx + H;   // own cell in a plane
    const double dx1 = 1. / G.dx, dy1 = 1. / G.dy, dt0 = G.dt0;
    // RN(1/lim_tol) for MUSCL's exact quotients (0: lim_tol outside their range)
    const double rlt = SCHEME == MG_MUSCL && G.lim_tol > 0x1p-900 && G.lim_tol < 0x1p900 ? 1. / G.lim_tol : 0.;
    const int NP = (F + PF - 1) / PF;      // passes (field groups)
    // this CTA's levels [kb, ke], the first prologue level kp (above the surface), and the
    // levels [l0, lmax] whose planes a pass takes; item n = pass * nlev + (level - l0)
    int kb, ke;
    segment_levels(nz, A.nseg, A.ns, A.ls, seg, kb, ke);
    const int kp = kb > NPRO ? kb - NPRO : 1;
    const int l0 = max(1, kp - 1), lmax = min(nz, ke + L), nlev = lmax - l0 + 1;
    const int NI = NP * nlev;

    // the extra faces of a group: a warp per field for the last y row, another for the last x
    // faces (8 of each field); the warps alternate with the block over the schedulers
    int ex = -1, ex_q = 0, ex_u = 0;
    bool ex_x = false;
    {
        const int wq = ty - ((bid & 1) ? TY - 1 - PF : 0);
        if (wq >= 0 && wq <= PF && (wq < PF || tx < PF * XE)) {
            ex_x = wq == PF;
            ex = wq * TX + tx;
            ex_u = ex_x ? tx / XE : wq;
            ex_q = NCELL + (ex_x ? tx % XE : tx);
        }
    }
    // where this thread's faces read: momentum boxes (uo, vo, eo) and planes (x(i-1) of x face
    // tid, x(j-1) of y face tid, likewise the extra face); its plane elements outside the cells
    const int uo = (tid / (TX + 1)) * VW + tid % (TX + 1) + 1, vo = ty * VW + tx + 1;
    const int eo = ex_x ? (ex_q / (TX + 1)) * VW + ex_q % (TX + 1) + 1 : (ex_q / TX) * VW + ex_q % TX + 1;
    const int bx = (tid / (TX + 1) + H) * SW + H + tid % (TX + 1) - 1, by = (ty - 1 + H) * SW + H + tx;
    const int eb = ex_x ? (ex_q / (TX + 1) + H) * SW + H + ex_q % (TX + 1) - 1 : (ex_q / TX - 1 + H) * SW + H + ex_q % TX;
    static_assert(NHALO > NTH && NHALO <= 2 * NTH, "one or two halo elements per thread");
    const int he0 = halo_elem(tid), he1 = tid + NTH < NHALO ? halo_elem(tid + NTH) : -1;
    if (tid == 0) {
        for (int b = 0; b <= NR; b++) mbar_init(&mb[b], 1);
        fence_mbar_init();
    }
    __syncthreads();

    int nxt = 0;   // thread 0: the next item to request
    // request items up to NR beyond n_free (the last item whose slot is free again) and, for
    // the density planes of stage 1, NRHO beyond n_conv (the last item multiplied by its own)
    auto issue_to = [&](int n_free, int n_conv) {
        while (nxt < NI && nxt <= n_free + NR && (!CONV1 || nxt <= n_conv + NRHO)) {
            const int p = nxt / nlev, l = l0 + nxt - p * nlev, slot = nxt % NR;
            const int nfg = min(PF, F - p * PF);
            const bool rho = CONV1 && p > 0;   // the first pass has the density as its first field
            fence_proxy_async_shared();
            mbar_arrive_expect_tx(&mb[slot], (nfg + (rho ? 1 : 0)) * PLANE_BYTES);
            for (int u = 0; u < nfg; u++)
                tma_load_3d(planes + (size_t)(slot * PF + u) * (PLANE_SLOT / 8), &M.x[p * PF + u], i0 - 4, j0 - 4, l - 1,
                            &mb[slot]);
            if (rho) tma_load_3d(rhop + (size_t)(nxt % NRHO) * (PLANE_SLOT / 8), &M.x[0], i0 - 4, j0 - 4, l - 1, &mb[slot]);
            nxt++;
        }
    };
    auto issue_vel = [&](int k) {
        fence_proxy_async_shared();
        mbar_arrive_expect_tx(&mb[NR], 2 * VBOX_BYTES);
        tma_load_3d(vbu, &M.mu, i0 - 2, j0 - 1, k - 1, &mb[NR]);
        tma_load_3d(vbv, &M.mv, i0 - 2, j0 - 1, k - 1, &mb[NR]);
    };
    // coefficient q of level l (avden0 and dz1 above it included), by the last warp
    auto fill_coef = [&](int l) {
        const int q = tid - (NTH - TX);
        if (q < 0 || q >= C_N + (SCHEME == MG_PPM && !MIXED ? PPM_NC : 0) || l > (SCHEME == MG_PPM ? min(ke + 1, nz) : ke)) return;
        if (SCHEME == MG_PPM && q >= C_N) {
            coef[(l % NCS) * NCOEF + q] = ldg(G.ppmtab, (long long)(l - 1) * 16 + q - C_N);
            return;
        }
        const double *src = q <= C_RD0 ? (q == C_D0 ? G.den0 : G.rden0) : q <= C_RAW ? (q == C_AW ? G.avden0 : G.ravden0)
                          : q <= C_RDZW ? G.dz1w : q <= C_D1P ? G.dz1 : G.fdz0;
        const int o = q == C_AW || q == C_RAW || q == C_D1P || q == C_FP ? l : (q == C_D1M || q == C_FM ? l - 2 : l - 1);
        double v = o >= 0 && o < nz ? ldg(src, o) : (q == C_AW || q == C_RAW ? 1. : 0.);
        if (q == C_RDZW) v = 1. / v;
        coef[(l % NCS) * NCOEF + q] = v;
    };
    // pointwise operands are read at the own cell (inactive threads: a cell of the domain)
    const long long idx0 = gidx(G, min(i, nx - 2), min(j, ny - 2), 1);

    if (tid == 0) {
        issue_to(-1, -1);
        issue_vel(kb);
    }
    int qv = 0;   // momentum boxes converted so far
#pragma unroll 1
    for (int p = 0; p < NP; p++) {
        const int gb = p * PF;
        const int nfg = min(PF, F - gb);   // fields of this pass
        double win[PF][L + 2];   // x(k-1 .. k+L) of the own column; stage 1: psi = s * rho
        double zf[PF];           // the flux through the face below
        double prfr = 0., prxp = 0.;   // PPM: Fr of the cell below, its xplus (relative in the mixed form)
        // wait for level l's planes, form psi in place (stage 1), take the own column's values
        auto take = [&](int l) {
            const int n = p * nlev + l - l0, slot = n % NR;
            mbar_wait_bounded(&mb[slot], (uint32_t)((n / NR) & 1), A.err);
            double *plq = planes + (size_t)slot * PF * (PLANE_SLOT / 8);
            if constexpr (CONV1) {
                // psi = s * rho, once per element: each thread its own, the halo shared out.  The
                // first pass has the density as field 0, unweighted
                const double *dsrc = p == 0 ? plq : rhop + (size_t)(n % NRHO) * (PLANE_SLOT / 8);
                const double dn = dsrc[own_e];
#pragma unroll
                for (int u = 0; u < PF; u++) {
                    if (u > 0 && u >= nfg) continue;
                    if (u == 0 && p == 0) {
                        win[0][L + 1] = dn;
                        continue;
                    }
                    double *plw = plq + u * (PLANE_SLOT / 8);
                    win[u][L + 1] = plw[own_e] * dn;
                    plw[own_e] = win[u][L + 1];
                }
                auto halo = [&](int e) {
                    const double d = dsrc[e];
#pragma unroll
                    for (int u = 0; u < PF; u++)
                        if (u < nfg && (u > 0 || p > 0)) plq[u * (PLANE_SLOT / 8) + e] = plq[u * (PLANE_SLOT / 8) + e] * d;
                };
                halo(he0);
                if (he1 >= 0) halo(he1);
            } else {
#pragma unroll
                for (int u = 0; u < PF; u++)
                    if (u < nfg) win[u][L + 1] = plq[u * (PLANE_SLOT / 8) + own_e];
            }
        };
        auto shift = [&]() {
#pragma unroll
            for (int u = 0; u < PF; u++)
#pragma unroll
                for (int m = 0; m <= L; m++) win[u][m] = win[u][m + 1];
        };
#pragma unroll
        for (int u = 0; u < PF; u++) {
            zf[u] = 0.;
#pragma unroll
            for (int m = 0; m < L + 2; m++) win[u][m] = 0.;
        }
        // w at levels k+1 and (PPM) k+2 of the own column, loaded a level ahead
        double wr1 = ldg(A.mw, idx0 + (long long)(min(kp + 1, nz) - 1) * G.ps);
        double wr2 = SCHEME == MG_PPM ? ldg(A.mw, idx0 + (long long)(min(kp + 2, nz) - 1) * G.ps) : 0.;
        __syncthreads();   // the previous pass's last level is done with the coefficients
        fill_coef(kp);
        fill_coef(kp + 1);
        for (int l = l0; l < kp + L && l <= lmax; l++) {
            take(l);
            shift();
        }
        __syncthreads();
        if (tid == 0) issue_to(p * nlev - 1, p * nlev + min(kp + L - 1, lmax) - l0);

#pragma unroll 1
        for (int k = kp; k <= ke; k++) {
            const bool pro = k < kb;   // prologue level: its vertical face only
            const double *ck = coef + (k % NCS) * NCOEF;   // this level's coefficients
            const long long idx = idx0 + (long long)(k - 1) * G.ps;
            // the level's pointwise operands, loaded before the faces, which cover their latency
            double c_xold[PF], c_tend[PF], c_sgs[PF], c_d0 = 0., c_dn = 0.;
            double c_xo[PF];   // mixed stage 1: the odd fields' natural values
            if (!pro && act) {
#pragma unroll
                for (int u = 0; u < PF; u++)
                    if (u == 0 || u < nfg) {
                        if (OPS) {
                            cp_async_8(ops + (2 * u) * NCELL, A.xold[gb + u] + idx);
                            cp_async_8(ops + (2 * u + 1) * NCELL, A.tend[gb + u] + idx);
                        } else if (STAGE == 2) {
                            c_xold[u] = ldg_stream(A.xold[gb + u] + idx);
                            c_tend[u] = ld_stream(A.tend[gb + u] + idx);
                        }
                        if (SGS) c_sgs[u] = A.sgs[gb + u] ? ldg_stream(A.sgs[gb + u] + idx) : 0.;
                    }
                if (STAGE == 2 && p > 0) {   // the cell's density: level n, new
                    if (OPS) cp_async_8(ops + 2 * PF * NCELL, A.xold[0] + idx);
                    else c_d0 = ldg_stream(A.xold[0] + idx);
                    c_dn = ld_stream(A.tend[0] + idx);
                }
                if (OPS) cp_async_commit();
                if (MIXED && STAGE == 1 && PF > 1) {
#pragma unroll
                    for (int u = 0; u < PF; u++)
                        if (u < nfg && ((gb + u) & 1)) c_xo[u] = ldg_stream(A.xin[gb + u] + idx);
                    c_d0 = ldg_stream(A.xin[0] + idx);
                }
            }
            if (k + L <= lmax) {
                take(k + L);
            } else {
#pragma unroll
                for (int u = 0; u < PF; u++) win[u][L + 1] = 0.;
            }
            double *fxb = fx + (k & 1) * PF * FXN, *fyb = fy + (k & 1) * PF * FYN;
            if (!pro) {
                const double *plq = planes + (size_t)((p * nlev + k - l0) % NR) * PF * (PLANE_SLOT / 8);
                // momentum boxes of level k -> face velocities: each thread converts those of its
                // own faces.
                // RN(1/rho0): the mixed form multiplies by it, the FP64 form divides exactly with it
                const double d0 = ck[C_D0], rd0 = ck[C_RD0];
                mbar_wait_bounded(&mb[NR], (uint32_t)(qv & 1), A.err);
                auto velocity = [&](double m, double shift) {
                    if (CONV1) m = m * d0;
                    return (MIXED ? m * rd0 : div_known(m, d0, rd0)) - shift;
                };
                const double uu = velocity(vbu[uo], G.u0shift), vv = velocity(vbv[vo], G.v0shift);
                const double ee = ex < 0 ? 0. : velocity(ex_x ? vbu[eo] : vbv[eo], ex_x ? G.u0shift : G.v0shift);
                double *crxq = crx + (k & 1) * 4 * TY * (TX + 2);
                double *cryq = cry + (k & 1) * 4 * (TY + 2) * TX;
                if constexpr (SCHEME == MG_PPM) {
                    const double *pl = plq;
                    auto V = [&](int e) -> double { return pl[e]; };
                    for (int qq = tid; qq < TY * (TX + 2) + (TY + 2) * TX; qq += NTH) {
                        double xv[5], pr = 0., pL = 0., p1 = 0., p2 = 0.;
                        if (qq < TY * (TX + 2)) {
                            int r = qq / (TX + 2), c = qq - r * (TX + 2);
                            int cell = i0 - 1 + c;
                            for (int m = 0; m < 5; m++) xv[m] = V((r + H) * SW + c + m);
                            int kind = cell == 3 ? 1 : (cell == 4 ? 2 : (cell == nx - 1 ? 3 : 0));
                            if (cell <= nx - 1) {
                                if constexpr (MIXED) {
                                    float a_, b_, c_, d_;
                                    ppm_cell_h_mixed(kind, xv, a_, b_, c_, d_);
                                    pr = a_; pL = b_; p1 = c_; p2 = d_;
                                } else {
                                    ppm_cell_h(kind, xv, pr, pL, p1, p2);
                                }
                            }
                            const int o = r * (TX + 2) + c, S = TY * (TX + 2);
                            crxq[o] = pr; crxq[S + o] = pL; crxq[2 * S + o] = p1; crxq[3 * S + o] = p2;
                        } else {
                            int q2 = qq - TY * (TX + 2);
                            int r = q2 / TX, c = q2 - r * TX;
                            int cell = j0 - 1 + r;
                            for (int m = 0; m < 5; m++) xv[m] = V((r + m) * SW + c + H);
                            int kind = cell == 3 ? 1 : (cell == 4 ? 2 : (cell == ny - 1 ? 3 : 0));
                            if (cell <= ny - 1) {
                                if constexpr (MIXED) {
                                    float a_, b_, c_, d_;
                                    ppm_cell_h_mixed(kind, xv, a_, b_, c_, d_);
                                    pr = a_; pL = b_; p1 = c_; p2 = d_;
                                } else {
                                    ppm_cell_h(kind, xv, pr, pL, p1, p2);
                                }
                            }
                            const int o = r * TX + c, S = (TY + 2) * TX;
                            cryq[o] = pr; cryq[S + o] = pL; cryq[2 * S + o] = p1; cryq[3 * S + o] = p2;
                        }
                    }
                __syncthreads();
                }
                if constexpr (PAIR) {   // x and y faces of a field as interleaved chains
#pragma unroll (MIXED ? PF : 1)
                    for (int u = 0; u < PF; u++) {
                        if (u > 0 && u >= nfg) continue;
                        const double *px = plq + u * (PLANE_SLOT / 8) + bx, *py = plq + u * (PLANE_SLOT / 8) + by;
                        const double xm[2] = {px[-1], py[-SW]}, x0[2] = {px[0], py[0]}, xp[2] = {px[1], py[SW]},
                                     xq[2] = {px[2], py[2 * SW]}, vel[2] = {uu, vv};
                        double Fo[2];
                        weno_faces<MIXED, 2>(xm, x0, xp, xq, vel, true, Fo);
                        fxb[u * FXN + tid] = Fo[0];
                        fyb[u * FYN + tid] = Fo[1];
                    }
                    if (ex >= 0 && ex_u < nfg) {
                        const int st = ex_x ? 1 : SW;
                        const double *pl = plq + ex_u * (PLANE_SLOT / 8) + eb;
                        const double xm[1] = {pl[-st]}, x0[1] = {pl[0]}, xp[1] = {pl[st]}, xq[1] = {pl[2 * st]}, vel[1] = {ee};
                        double Fo[1];
                        weno_faces<MIXED, 1>(xm, x0, xp, xq, vel, true, Fo);
                        (ex_x ? fxb + ex_u * FXN : fyb + ex_u * FYN)[ex_q] = Fo[0];
                    }
                } else {
                    // flux through x face q (isx) or y face q of field u
                    auto face = [&](int u, bool isx, int q, double vel) -> double {
                        const int r = isx ? q / (TX + 1) : q / TX, c = isx ? q - r * (TX + 1) : q - r * TX;
                        // x(i0 + c - 1) in row r; x(j0 + r - 1) in column c
                        const double *pl = plq + u * (PLANE_SLOT / 8) + (isx ? (r + H) * SW + H + c - 1 : (r - 1 + H) * SW + H + c);
                        const int st = isx ? 1 : SW;
                        const double d = isx ? G.dx : G.dy, d1 = isx ? dx1 : dy1;
                        if constexpr (SCHEME == MG_MUSCL) {
                            if constexpr (MIXED)
                                return muscl_face_h_mixed(G.muscl_lim, (float)G.lim_tol, (float)d, (float)d1, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                            else
                                return muscl_face_h(G.muscl_lim, G.lim_tol, rlt, d, d1, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                        } else if constexpr (SCHEME == MG_LW) {
                            if constexpr (MIXED)
                                return lw_face_h_mixed((float)G.lim_tol, (float)dt0, (float)d1, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                            else
                                return lw_face_h(G.lim_tol, dt0, d1, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                        } else if constexpr (SCHEME == MG_QUICK) {
                            if constexpr (MIXED) return quick_face_h_mixed((float)G.lim_tol, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                            else return quick_face_h(G.lim_tol, pl[-st], pl[0], pl[st], pl[2 * st], vel);
                        } else {   // PPM: from the cell reconstructions (relative to the cell's value in the mixed form)
                            const double mu = fabs(vel) * dt0 * d1;
                            const double *cr = isx ? crxq : cryq;
                            const int S = isx ? TY * (TX + 2) : (TY + 2) * TX;
                            const int o0 = isx ? r * (TX + 2) + c : q, o1 = isx ? o0 + 1 : q + TX;
                            if constexpr (MIXED) {
                                const float fr = ppm_fr((float)cr[o0], (float)mu, (float)cr[2 * S + o0], (float)cr[3 * S + o0]);
                                const float fl = ppm_fl((float)cr[S + o1], (float)mu, (float)cr[2 * S + o1], (float)cr[3 * S + o1]);
                                return vel > 0. ? vel * (pl[0] + (double)fr) : (vel < 0. ? vel * (pl[st] + (double)fl) : 0.);
                            } else {
                                const double fr = ppm_fr(cr[o0], mu, cr[2 * S + o0], cr[3 * S + o0]);
                                const double fl = ppm_fl(cr[S + o1], mu, cr[2 * S + o1], cr[3 * S + o1]);
                                return 0.5 * fr * (vel + fabs(vel)) + 0.5 * fl * (vel - fabs(vel));
                            }
                        }
                    };
#pragma unroll
                    for (int u = 0; u < PF; u++) {
                        if (u > 0 && u >= nfg) continue;
                        const double Fx = face(u, true, tid, uu), Fy = face(u, false, tid, vv);   // independent chains
                        fxb[u * FXN + tid] = Fx;
                        fyb[u * FYN + tid] = Fy;
                    }
                    if (ex >= 0 && ex_u < nfg) {
                        if (ex_x) fxb[ex_u * FXN + ex_q] = face(ex_u, true, ex_q, ee);
                        else fyb[ex_u * FYN + ex_q] = face(ex_u, false, ex_q, ee);
                    }
                }
            }
            // the faces of level k are complete; every thread is done with plane k and the boxes
            __syncthreads();
            if (tid == 0) {
                issue_to(p * nlev + (k < ke ? k - l0 : nlev - 1), p * nlev + min(k + L, lmax) - l0);
                if (!pro && (k < ke || p + 1 < NP)) issue_vel(k < ke ? k + 1 : kb);
            }
            if (!pro) qv++;
            // slot (k+2) % NCS last held level k-2; the barrier of level k+1 publishes it
            fill_coef(k + 2);
            if (OPS) cp_async_wait_group<0>();   // the thread's own operands

            // ---- vertical faces k+1/2 of the own column ----
            double wz2 = 0., wz3 = 0.;   // w_adv at levels k+1 and (PPM) k+2
            if (k <= nz - 1) {
                const double a0 = ck[C_AW], ra0 = ck[C_RAW];
                double x = wr1;
                if (CONV1) x = x * a0;
                wz2 = MIXED ? x * ra0 : div_known(x, a0, ra0);
            }
            if (SCHEME == MG_PPM && k + 2 <= nz) {
                const double *cn = coef + ((k + 1) % NCS) * NCOEF;
                double x = wr2;
                if (CONV1) x = x * cn[C_AW];
                wz3 = MIXED ? x / cn[C_AW] : div_known(x, cn[C_AW], cn[C_RAW]);
            }
            if (SCHEME == MG_PPM) {
                wr1 = wr2;
                wr2 = ldg(A.mw, idx0 + (long long)(min(k + 3, nz) - 1) * G.ps);
            } else {
                wr1 = ldg(A.mw, idx0 + (long long)(min(k + 2, nz) - 1) * G.ps);
            }
            double Fzp[PF];   // the group's vertical faces, evaluated together
            if constexpr (PAIR) {
                double xm[PF], x0[PF], xp[PF], xq[PF], vel[PF];
#pragma unroll
                for (int u = 0; u < PF; u++) {
                    // an absent second field repeats the first
                    const bool own = u < nfg;
                    xm[u] = own ? win[u][0] : win[0][0]; x0[u] = own ? win[u][1] : win[0][1];
                    xp[u] = own ? win[u][2] : win[0][2]; xq[u] = own ? win[u][3] : win[0][3];
                    vel[u] = wz2;
                    Fzp[u] = 0.;
                }
                if (k == 1) {
#pragma unroll
                    for (int u = 0; u < PF; u++) Fzp[u] = MIXED ? weno_face_bottom_mixed(x0[u], xp[u], xq[u], wz2) : weno_face_bottom(x0[u], xp[u], xq[u], wz2);
                } else if (k == nz - 1) {
#pragma unroll
                    for (int u = 0; u < PF; u++) Fzp[u] = MIXED ? weno_face_top_mixed(xm[u], x0[u], xp[u], wz2) : weno_face_top(xm[u], x0[u], xp[u], wz2);
                } else if (k < nz - 1) {
                    weno_faces<MIXED, PF>(xm, x0, xp, xq, vel, k >= 3 && k <= nz - 3, Fzp);
                }
            }
            double rdn = 0.;
#pragma unroll
            for (int u = 0; u < PF; u++) {
                const int f = gb + u;
                if (u > 0 && u >= nfg) continue;
                const double *fxq = fxb + u * FXN, *fyq = fyb + u * FYN;
                const double dFx = pro ? 0. : fxq[ty * (TX + 1) + tx + 1] - fxq[ty * (TX + 1) + tx];
                const double dFy = pro ? 0. : fyq[(ty + 1) * TX + tx] - fyq[ty * TX + tx];
                    const double dzw1 = ck[C_DZW];
                    double Fzn = 0.;
                    if (k <= nz - 1) {
                        const double ww = wz2;
                        if (SCHEME == MG_WENO) {
                            Fzn = Fzp[u];
                        } else if (SCHEME == MG_MUSCL) {
                            const int kind = k == 1 ? 1 : (k == nz - 1 ? 2 : 0);
                            const double d1m = ck[C_D1M], d10 = ck[C_D10], d1p = ck[C_D1P];
                            const double fm = ck[C_FM], fp = ck[C_FP];
                            const double xm1 = k >= 2 ? win[u][0] : 0.;
                            const double xp2 = k + 2 <= nz ? win[u][3] : 0.;
                            if constexpr (MIXED)
                                Fzn = muscl_face_z_mixed(kind, G.muscl_lim, (float)G.lim_tol, (float)G.dz, xm1, win[u][1], win[u][2], xp2,
                                                         (float)d1m, (float)d10, (float)d1p, (float)fm, (float)fp, (float)dzw1, ww);
                            else
                                Fzn = muscl_face_z(kind, G.muscl_lim, G.lim_tol, rlt, G.dz, xm1, win[u][1], win[u][2], xp2, d1m, d10,
                                                   d1p, fm, fp, dzw1, ck[C_RDZW], ww);
                        } else if (SCHEME == MG_LW || SCHEME == MG_QUICK) {
                            const int kind = k == 1 ? 1 : (k == nz - 1 ? 2 : 0);
                            const double d1m = ck[C_D1M], d10 = ck[C_D10], d1p = ck[C_D1P];
                            const double xm1 = k >= 2 ? win[u][0] : 0.;
                            const double xp2 = k + 2 <= nz ? win[u][3] : 0.;
                            if constexpr (MIXED) {
                                if constexpr (SCHEME == MG_LW)
                                    Fzn = lw_face_z_mixed(kind, (float)G.lim_tol, (float)G.dz, (float)dt0, xm1, win[u][1], win[u][2], xp2,
                                                          (float)d1m, (float)d10, (float)d1p, (float)dzw1, ww);
                                else
                                    Fzn = quick_face_z_mixed(kind, (float)G.lim_tol, (float)G.dz, xm1, win[u][1], win[u][2], xp2,
                                                             (float)d1m, (float)d10, (float)d1p, (float)dzw1, ww);
                            } else {
                                if constexpr (SCHEME == MG_LW)
                                    Fzn = lw_face_z(kind, G.lim_tol, G.dz, dt0, xm1, win[u][1], win[u][2], xp2, d1m, d10, d1p, dzw1, ww);
                                else
                                    Fzn = quick_face_z(kind, G.lim_tol, G.dz, xm1, win[u][1], win[u][2], xp2, d1m, d10, d1p, dzw1, ww);
                            }
                        } else if constexpr (MIXED) {
                            // chain values relative: prfr = Fr(k) - x(k), prxp = xplus(k) - x(k)
                            if (k == 1) {
                                const double x1 = win[u][1];
                                const float b1 = (float)(win[u][2] - x1), b2 = (float)(win[u][3] - x1);
                                const float mup = (float)(fabs(wz2) * dt0 * ck[C_D10]);
                                const float ffip1 = b1, ffip2 = b2 - b1;
                                float dr, dl, phi1, phi2;
                                ppm_limiter_rel((float)x1, b1, b1, 0.5f * ffip1, -0.5f * ffip1, ffip1, ffip2, 0.f, 0.f, dr, dl, phi1, phi2);
                                prfr = ppm_fr(dr, mup, phi1, phi2);
                                prxp = 0.5f * ffip1;
                            }
                            const int c = k + 1;
                            const double x0 = win[u][2], xkm = win[u][1];
                            const float m1 = (float)(xkm - x0);
                            const float m2 = k >= 2 ? (float)(win[u][0] - x0) : 0.f;
                            const float p1 = c + 1 <= nz ? (float)(win[u][3] - x0) : 0.f;
                            const float p2 = c + 2 <= nz ? (float)(win[u][4] - x0) : 0.f;
                            const double d1c = ck[C_D1P];   // dz1(c)
                            const float muc = (float)(fabs(ww) * dt0 * d1c);
                            float dfl;
                            if (c == nz) {
                                dfl = 0.5f * (-m1) * (1.f - muc);
                            } else {
                                const float mup = (float)(fabs(wz3) * dt0 * d1c);
                                float ffip1, ffip2, ffim1, ffim2, dplus;
                                const float dmin = (float)prxp + m1;   // xplus(k) - x(k+1)
                                if (c == 2) {
                                    ffip1 = p1; ffip2 = p2 - p1; ffim1 = -m1; ffim2 = 0.f;
                                    dplus = 0.5f * ffip1;
                                } else if (c == nz - 1) {
                                    ffip1 = p1; ffim1 = -m1; ffim2 = m1 - m2; ffip2 = ffip1;
                                    dplus = 0.5f * ffip1;
                                } else {
                                    ffip1 = p1; ffip2 = p2 - p1; ffim1 = -m1; ffim2 = m1 - m2;
                                    dplus = ppm_xplus_z(0.f, ffip1, ffip2, ffim1, (float)ldg(G.dz1w, c - 2), (float)ldg(G.dz1w, c - 1),
                                                        (float)ldg(G.dz1w, c), (float)ldg(G.dz1w, c + 1));
                                }
                                float dr, dl, phi1, phi2;
                                ppm_limiter_rel((float)x0, p1, m1, dplus, dmin, ffip1, ffip2, ffim1, ffim2, dr, dl, phi1, phi2);
                                dfl = ppm_fl(dl, muc, phi1, phi2);
                                const double fzn_up = ww > 0. ? ww * (xkm + prfr) : (ww < 0. ? ww * (x0 + (double)dfl) : 0.);
                                prfr = ppm_fr(dr, mup, phi1, phi2);
                                prxp = dplus;
                                Fzn = fzn_up;
                            }
                            if (c == nz) Fzn = ww > 0. ? ww * (xkm + prfr) : (ww < 0. ? ww * (x0 + (double)dfl) : 0.);
                        } else {
                            if (k == 1) {
                                // cell 1 (advq_ppm.f90:328-343): bottom special, bc51 = 0
                                const double x1 = win[u][1], x2 = win[u][2], x3 = win[u][3];
                                const double mup = fabs(wz2) * dt0 * ck[C_D10];   // w(2) at k = 1
                                const double ffip1 = x2 - x1, ffip2 = x3 - x2;
                                const double xmin = x1 - 0.5 * ffip1, xplus = x1 + 0.5 * ffip1;
                                double phir, phil, phi1, phi2;
                                ppm_limiter(x1, x2, x2, xplus, xmin, ffip1, ffip2, 0., 0., phir, phil, phi1, phi2);
                                prfr = ppm_fr(phir, mup, phi1, phi2);
                                prxp = xplus;
                            }
                            // reconstruction of cell c = k+1 (:345-414)
                            const int c = k + 1;
                            const double xm2 = k >= 2 ? win[u][0] : 0., xm1 = win[u][1], x0 = win[u][2];
                            const double xp1 = c + 1 <= nz ? win[u][3] : 0., xp2 = c + 2 <= nz ? win[u][4] : 0.;
                            const double d1c = ck[C_D1P];   // dz1(c)
                            const double muc = fabs(ww) * dt0 * d1c;
                            if (c == nz) {
                                const double fl = x0 + 0.5 * (x0 - xm1) * (1. - muc);
                                Fzn = 0.5 * prfr * (ww + fabs(ww)) + 0.5 * fl * (ww - fabs(ww));
                            } else {
                                const double mup = fabs(wz3) * dt0 * d1c;
                                double ffip1, ffip2, ffim1, ffim2, xplus;
                                const double xmin = prxp;
                                if (c == 2) {
                                    ffip1 = xp1 - x0; ffip2 = xp2 - xp1; ffim1 = (x0 - xm1); ffim2 = 0.;
                                    xplus = x0 + 0.5 * ffip1;
                                } else if (c == nz - 1) {
                                    ffip1 = xp1 - x0; ffim1 = x0 - xm1; ffim2 = xm1 - xm2; ffip2 = ffip1;
                                    xplus = x0 + 0.5 * ffip1;
                                } else {
                                    ffip1 = (xp1 - x0); ffip2 = (xp2 - xp1); ffim1 = (x0 - xm1); ffim2 = (xm1 - xm2);
                                    xplus = ppm_xplus_tab(x0, ffip1, ffip2, ffim1, ck + C_N);
                                }
                                double phir, phil, phi1, phi2;
                                ppm_limiter(x0, xp1, xm1, xplus, xmin, ffip1, ffip2, ffim1, ffim2, phir, phil, phi1, phi2);
                                const double fl = ppm_fl(phil, muc, phi1, phi2);
                                Fzn = 0.5 * prfr * (ww + fabs(ww)) + 0.5 * fl * (ww - fabs(ww));
                                prfr = ppm_fr(phir, mup, phi1, phi2);
                                prxp = xplus;
                            }
                        }
                    }
                    const double dFz = k == 1 ? Fzn - 0. : (k == nz ? 0. - zf[u] : Fzn - zf[u]);
                    zf[u] = Fzn;

                // ---- epilogue ----
                if (act && !pro) {
                    if constexpr (STAGE == 0) {
                        double *xs = A.xout[f];
                        xs[idx] = k1_tendency<MIXED>(xs[idx], dFx, dx1, dFy, dy1, dFz, dzw1);
                    } else {
                        double T;
                        if constexpr (SGS) {
                            const bool has = A.sgs[f] != nullptr, spost = (A.sgs_post >> f) & 1u;
                            const double sgv = c_sgs[u];
                            T = k1_tendency<MIXED>(has && !spost ? 0. + sgv : 0., dFx, dx1, dFy, dy1, dFz, dzw1);
                            if (has && spost) T = T + sgv;
                        } else {
                            T = k1_tendency<MIXED>(0., dFx, dx1, dFy, dy1, dFz, dzw1);
                        }
                        if (OPS) {
                            c_xold[u] = ops[2 * u * NCELL];
                            c_tend[u] = ops[(2 * u + 1) * NCELL];
                            if (u == 0 && p > 0) c_d0 = ops[2 * PF * NCELL];
                        }
                        const double told = STAGE == 1 ? 0. : c_tend[u];
                        const double tn = T + A.b * told;
                        // level n: stage 1 has psi = s * rho (density: rho) in the window; stage 2
                        // weighs the natural value, which it overwrites in place
                        if (f == 0) c_d0 = STAGE == 1 ? win[0][1] : c_xold[u];
                        double old;
                        if constexpr (STAGE == 1) old = win[u][1];
                        else old = f > 0 ? c_xold[u] * c_d0 : c_xold[u];
                        double xnew;
                        if constexpr (MIXED) {
                            if (PF > 1 && (f & 1)) xnew = __fma_rn(STAGE == 1 ? c_xo[u] : c_xold[u], c_d0, __dmul_rn(A.a_dt, tn));
                            else xnew = __fma_rn(A.a_dt, tn, old);
                        } else {
                            xnew = old + A.a_dt * tn;
                        }
                        if constexpr (STAGE == 2) {
                            // get_scalars (funcpack.f90:488-542): natural value with the new density,
                            // one reciprocal per cell and pass
                            if (f == 0) c_dn = xnew;
                            if (u == 0) rdn = MIXED ? rcp_nr(c_dn) : 1. / c_dn;
                            if (f == 0) {
                                if (NP > 1) A.tend[0][idx] = xnew;   // for the later passes
                                else A.xout[0][idx] = xnew;
                            } else {
                                A.xout[f][idx] = MIXED ? xnew * rdn : div_known(xnew, c_dn, rdn);
                            }
                            if (p > 0 && p == NP - 1 && u == 0) A.xout[0][idx] = c_dn;
                        } else {
                            A.xout[f][idx] = xnew;
                            A.tend[f][idx] = tn;
                        }
                        if (A.fst[f]) A.fst[f][idx] = T;
                    }
                }
            }
            shift();
        }
    }
}

template <int SCHEME, bool MIXED, int STAGE, bool SGS>
__global__ void __launch_bounds__(NTH, K1_CTAS)
    k1_kernel(const __grid_constant__ DevGrid G, const __grid_constant__ K1Args A, const __grid_constant__ K1Maps M)
{
    k1_run<SCHEME, MIXED, STAGE, SGS>(G, A, M, blockIdx.x);
}

// One launch over the blocks of several domains (an ensemble stage): block b of the
// launch runs block items[b].b of domain items[b].m, whose grid, arguments and tensor
// maps (in global memory, written before the launch and never changed while it runs)
// are mem[items[b].m].
template <int SCHEME, bool MIXED, int STAGE>
__global__ void __launch_bounds__(NTH, K1_CTAS) k1_group_kernel(const K1Member *__restrict__ mem, const GItem *__restrict__ items)
{
    const GItem it = items[blockIdx.x];
    const K1Member &m = mem[it.m];
    if (threadIdx.x == 0 && threadIdx.y == 0) {   // the thread that issues the bulk copies
        for (int f = 0; f < m.A.nf; f++) tensormap_acquire(&m.M.x[f]);
        tensormap_acquire(&m.M.mu);
        tensormap_acquire(&m.M.mv);
    }
    k1_run<SCHEME, MIXED, STAGE, false>(m.G, m.A, m.M, it.b);
}

}  // namespace
