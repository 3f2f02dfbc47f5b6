// k_scalar.cu -- K1 (scalar advection fused with the Heun stage update), plain FP64
// form.  The kernel body is in k1_body.cuh.  This translation unit is compiled
// with -fmad=false: bit-identical to the CPU restatement.
#include "k1_body.cuh"


namespace {
template <int SCHEME, int STAGE>
cudaError_t launch_one(const DevGrid &g, const K1Args &a, const K1Maps &maps, cudaStream_t s)
{
    const size_t sm = make_layout(SCHEME, false, STAGE).total;
    const int ntx = (g.maxx + TX - 1) / TX, nty = (g.maxy + TY - 1) / TY;
    K1Args as = a;
    ColSplit cut{as.nseg, 0, 0};
    if (as.nseg < 1 || as.nseg > g.nz) cut = k1_split(g, SCHEME);
    as.nseg = cut.nseg; as.ns = cut.ns; as.ls = cut.ls;
    const unsigned nblk = (unsigned)(ntx * nty) * (unsigned)(cut.nseg + cut.ns);
    bool sgs = false;
    for (int f = 0; f < a.nf; f++) sgs = sgs || a.sgs[f] != nullptr;
    if (STAGE != 0 && sgs)
        k1_kernel<SCHEME, false, STAGE, true><<<nblk, dim3(TX, TY), sm, s>>>(g, as, maps);
    else
        k1_kernel<SCHEME, false, STAGE, false><<<nblk, dim3(TX, TY), sm, s>>>(g, as, maps);
    return cudaGetLastError();
}
template <int SCHEME>
cudaError_t launch_scheme(const DevGrid &g, const K1Args &a, const K1Maps &maps, cudaStream_t s)
{
    if (a.mode == 1) return launch_one<SCHEME, 0>(g, a, maps, s);
    if (a.stage == 1) return launch_one<SCHEME, 1>(g, a, maps, s);
    return launch_one<SCHEME, 2>(g, a, maps, s);
}
template <int SCHEME>
cudaError_t init_scheme()
{
    cudaError_t e;
    const int mx = 232448;
    if ((e = cudaFuncSetAttribute(k1_kernel<SCHEME, false, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k1_kernel<SCHEME, false, 1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k1_kernel<SCHEME, false, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k1_kernel<SCHEME, false, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx)) != cudaSuccess) return e;
    return cudaFuncSetAttribute(k1_kernel<SCHEME, false, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
}
template <int SCHEME, int STAGE>
cudaError_t group_one(int nf, const K1Member *mem, const GItem *items, int nitems, cudaStream_t s)
{
    const size_t sm = make_layout(SCHEME, false, STAGE).total;
    cudaError_t e = cudaFuncSetAttribute(k1_group_kernel<SCHEME, false, STAGE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k1_group_kernel<SCHEME, false, STAGE><<<nitems, dim3(TX, TY), sm, s>>>(mem, items);
    return cudaGetLastError();
}
template <int SCHEME>
cudaError_t group_scheme(int stage, int nf, const K1Member *mem, const GItem *items, int nitems, cudaStream_t s)
{
    return stage == 1 ? group_one<SCHEME, 1>(nf, mem, items, nitems, s) : group_one<SCHEME, 2>(nf, mem, items, nitems, s);
}
}  // namespace

cudaError_t launch_k1(const DevGrid &g, const K1Args &a, const K1Maps &maps, cudaStream_t s)
{
    if (a.nf <= 0 || a.nf > MG_MAXF) return cudaErrorInvalidValue;
    if (a.mode != 1 && a.stage != 1 && a.stage != 2) return cudaErrorInvalidValue;
    if (a.nf > k1_max_fields(g.scal_adv)) return cudaErrorInvalidValue;
    switch (g.scal_adv) {
    case MG_WENO: return launch_scheme<MG_WENO>(g, a, maps, s);
    case MG_PPM: return launch_scheme<MG_PPM>(g, a, maps, s);
    case MG_LW: return launch_scheme<MG_LW>(g, a, maps, s);
    case MG_QUICK: return launch_scheme<MG_QUICK>(g, a, maps, s);
    default: return launch_scheme<MG_MUSCL>(g, a, maps, s);
    }
}

cudaError_t k1_init()
{
    cudaError_t e;
    if ((e = init_scheme<MG_WENO>()) != cudaSuccess) return e;
    if ((e = init_scheme<MG_PPM>()) != cudaSuccess) return e;
    if ((e = init_scheme<MG_LW>()) != cudaSuccess) return e;
    if ((e = init_scheme<MG_QUICK>()) != cudaSuccess) return e;
    return init_scheme<MG_MUSCL>();
}

// K1 over the blocks of several members (same scheme, stage and field count; no SGS)
cudaError_t launch_k1_group(int scheme, int stage, int nf, const K1Member *mem, const GItem *items, int nitems, cudaStream_t s)
{
    if (nf <= 0 || nf > MG_MAXF || (stage != 1 && stage != 2) || nitems < 1) return cudaErrorInvalidValue;
    if (nf > k1_max_fields(scheme)) return cudaErrorInvalidValue;
    switch (scheme) {
    case MG_WENO: return group_scheme<MG_WENO>(stage, nf, mem, items, nitems, s);
    case MG_PPM: return group_scheme<MG_PPM>(stage, nf, mem, items, nitems, s);
    case MG_LW: return group_scheme<MG_LW>(stage, nf, mem, items, nitems, s);
    case MG_QUICK: return group_scheme<MG_QUICK>(stage, nf, mem, items, nitems, s);
    default: return group_scheme<MG_MUSCL>(stage, nf, mem, items, nitems, s);
    }
}
