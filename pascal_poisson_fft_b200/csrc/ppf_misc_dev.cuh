// ppf_misc_dev.cuh -- device bodies of the small solve steps, shared by
// their kernels (ppf_ghost.cu, ppf_tdma.cu) and the persistent batch kernel
// (ppf_batch.cu): the ghost-cell update of one axis, the refinement gate and
// the z coefficients.
//
// The reference fills the ghost cells in a fixed order: quadratic Neumann
// extrapolation along every non-periodic axis (apply_bc_on_direction,
// 01_Fortran/src/fft_3d_poisson.f90:798-852, x then y then z), then the
// periodic copies along every periodic axis (ghostcell_update_on_direction
// at one rank, :709-796, x then y then z).  Each step covers the whole face
// including the other axes' ghost lines, so later steps read values written
// by earlier ones; the same order is kept, one step per axis.
#pragma once
#include "ppf_kernels.cuh"

#include <math.h>

namespace ppf {

// face elements idx0, idx0 + stride, ... of axis dir
__device__ __forceinline__ void ghost_axis(double* __restrict__ P, int dir, int neumann, int n1m, int n2m, int n3m,
                                           long sy, long sz, const double* __restrict__ dmx, int faces, long idx0,
                                           long stride)
{
    const int N1 = n1m + 2, N2 = n2m + 2, N3 = n3m + 2;
    int nb, nm;
    long sa, sb, sc;
    if (dir == 0)      { nb = N2; sa = 1;  sb = sy; sc = sz; nm = n1m; }
    else if (dir == 1) { nb = N1; sa = sy; sb = 1;  sc = sz; nm = n2m; }
    else               { nb = N1; sa = sz; sb = 1;  sc = sy; nm = n3m; }
    const int nc = (dir == 2) ? N2 : N3;
    const int na = nm + 1;  // upper ghost index
    double alo = 0, blo = 0, ahi = 0, bhi = 0;
    if (neumann) {
        const double d1 = dmx[1], d2 = dmx[2], dn = dmx[na], dn1 = dmx[nm];
        const double sl = d1 + d2, su = dn + dn1;
        alo = (sl * sl) / ((sl * sl) - d1 * d1);
        blo = (d1 * d1) / ((sl * sl) - d1 * d1);
        ahi = (su * su) / ((su * su) - dn * dn);
        bhi = (dn * dn) / ((su * su) - dn * dn);
    }
    const long total = (long)nb * nc;
    for (long idx = idx0; idx < total; idx += stride) {
        const long ib = idx % nb, ic = idx / nb;
        const long base = ib * sb + ic * sc;
        if (neumann) {
            if (faces & 1) P[base] = alo * P[base + sa] - blo * P[base + 2 * sa];
            if (faces & 2) P[base + na * sa] = ahi * P[base + nm * sa] - bhi * P[base + (na - 2) * sa];
        } else {
            const double v0 = P[base + sa], v1 = P[base + nm * sa];
            P[base] = v1;
            P[base + na * sa] = v0;
        }
    }
}

// After an x-inverse pass that wrote per-block partial sums: reduce them in
// a fixed order (deterministic), keep mean(u) for the next accumulate pass,
// and after a refinement sweep count it, record ||du||/||u|| and close the
// gate for the remaining sweeps once it is below tol.  A sweep that was
// skipped (gate already closed) leaves everything unchanged.
// (one CTA of a power-of-two size up to 512 threads)
__device__ __forceinline__ void sweep_gate(const double* partials, long nblocks, double ncell,
                                           double* mean_prev, int* skip, int* sweeps_done, double* last_rel,
                                           double tol, int initial)
{
    __shared__ double red[3][512];
    if (*skip) return;
    double a = 0.0, b = 0.0, c = 0.0;
    for (long i = threadIdx.x; i < nblocks; i += blockDim.x) {
        a += partials[3 * i + 0];
        b += partials[3 * i + 1];
        c += partials[3 * i + 2];
    }
    red[0][threadIdx.x] = a; red[1][threadIdx.x] = b; red[2][threadIdx.x] = c;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            red[0][threadIdx.x] += red[0][threadIdx.x + o];
            red[1][threadIdx.x] += red[1][threadIdx.x + o];
            red[2][threadIdx.x] += red[2][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    *mean_prev = red[2][0] / ncell;
    if (initial) return;
    *sweeps_done += 1;
    const double du = red[0][0], u = red[1][0];
    const double rel = (u > 0.0) ? sqrt(du / u) : (du > 0.0 ? INFINITY : 0.0);
    *last_rel = rel;
    if (tol > 0.0 && rel < tol) *skip = 1;
}

// z coefficients of cuda_Poisson_TDMA_z_* (fft_3d_poisson.f90:1139-1142):
// am_k = 1/dx3_k/dmx3_k, ap_k = 1/dx3_k/dmx3_{k+1}, am_1 = ap_n3m = 0; plus
// min_k dx3_k^2 for the low-wavenumber precision switch (a system is
// near-singular when lam dz^2 << 1 at the finest spacing).  One CTA.
__device__ __forceinline__ void zcoef(const double* __restrict__ dx3, const double* __restrict__ dmx3, int nz,
                                      double* __restrict__ am, double* __restrict__ ap, double* __restrict__ dzmin2)
{
    __shared__ double red[512];   // one CTA of a power-of-two size up to 512 threads
    double mn = INFINITY;
    for (int k = threadIdx.x; k < nz; k += blockDim.x) {
        const int kk = k + 1;
        double av = __ddiv_rn(__ddiv_rn(1.0, dx3[kk]), dmx3[kk]);
        double cv = __ddiv_rn(__ddiv_rn(1.0, dx3[kk]), dmx3[kk + 1]);
        if (k == 0) av = 0.0;
        if (k == nz - 1) cv = 0.0;
        am[k] = av;
        ap[k] = cv;
        mn = fmin(mn, dx3[kk] * dx3[kk]);
    }
    red[threadIdx.x] = mn;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] = fmin(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *dzmin2 = red[0];
}

// The preparation blocks of a solve (ZPrep): block `blk` of any number of
// warps, sm: zprep_smem bytes of shared memory.  The coefficients are formed
// as in zcoef, the table entries by the reference's Thomas operations in
// their order (thomas_poisson<Exact>; FP32: k_thomas_fast's).  Bound by the
// latency of its reciprocal chains (about 0.06 us a row), which the transform
// tiles running beside it hide.
static __device__ __noinline__ void zprep(const ZPrep& q, unsigned blk, double* sm)
{
    const int nz = q.nz, tid = threadIdx.x, nt = blockDim.x;
    double* const zl = sm;               // am, ap, -am - ap
    double* const red = sm + 3 * nz;     // 32
    double mn = INFINITY;
    for (int k = tid; k < nz; k += nt) {
        const int kk = k + 1;
        const double d = q.dx3[kk], inv = __ddiv_rn(1.0, d);
        double av = __ddiv_rn(inv, q.dmx3[kk]);
        double cv = __ddiv_rn(inv, q.dmx3[kk + 1]);
        if (k == 0) av = 0.0;
        if (k == nz - 1) cv = 0.0;
        zl[k] = av;
        zl[nz + k] = cv;
        zl[2 * nz + k] = __dsub_rn(-av, cv);
        if (blk == 0) { q.am[k] = av; q.ap[k] = cv; }
        mn = fmin(mn, d * d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    if ((tid & 31) == 0) red[tid >> 5] = mn;
    __syncthreads();
    for (int w = 0; w < (nt >> 5); ++w) mn = fmin(mn, red[w]);
    if (blk == 0) {
        if (tid < 8) q.scal[tid] = tid == 0 ? mn : 0.0;
        if (tid < 4) q.flags[tid] = 0;
    }
    if (!q.tab) return;
    const long idx = (long)blk * nt + tid;
    const int kx = (int)(idx % q.pitch), ky = (int)(idx / q.pitch);
    if (kx >= q.mx || ky >= q.rows) return;
    const double lx = q.lamx[kx], ly = q.lamy[ky];
    const bool pin = (kx == 0 && ky == 0);
    auto diag = [&](int k) { return __dsub_rn(__dsub_rn(zl[2 * nz + k], lx), ly); };
    // The reciprocal chains below form the next row's diagonal ahead of this
    // row's reciprocal, whose rare-case branch the scheduler does not move
    // loads and arithmetic across.
    if (q.f32 && !((lx + ly) * mn < q.lowk)) {
        float* tab = reinterpret_cast<float*>(q.tab + (size_t)nz * q.tplane) + idx;
        const float lam = (float)(lx + ly);
        float cp = __fdividef((float)zl[nz], (float)zl[2 * nz] - lam);
        tab[0] = cp;
#pragma unroll 4
        for (int k = 1; k < nz; ++k) {
            const float r = __fdividef(1.0f, ((float)zl[2 * nz + k] - lam) - (float)zl[k] * cp);
            cp = r * (float)zl[nz + k];
            tab[(size_t)k * q.tplane] = r;
        }
        return;
    }
    double* tab = q.tab + idx;
    if (!q.cyclic) {
        double cp = pin ? 0.0 : __ddiv_rn(zl[nz], diag(0));
        tab[0] = cp;
        double a = zl[1], c = zl[nz + 1], b = diag(1);
#pragma unroll 2
        for (int k = 1; k < nz; ++k) {
            const double p = __dsub_rn(b, __dmul_rn(a, cp)), ck = c;
            const int kn = min(k + 1, nz - 1);
            a = zl[kn];
            c = zl[nz + kn];
            b = diag(kn);
            const double r = __drcp_rn(p);
            cp = __dmul_rn(r, ck);
            tab += q.tplane;
            *tab = r;
        }
        return;
    }
    // rows 1 .. nz-1: r and e' (e_1 = -a_1, e_{nz-1} = -c_{nz-1}, the last
    // one set after the first), then e back-substituted in place
    double* tabe = tab + (size_t)nz * q.tplane;
    const double e_last = -zl[nz + nz - 1];
    double cp = __ddiv_rn(zl[nz + 1], diag(1));
    double e = __ddiv_rn(nz == 2 ? e_last : -zl[1], diag(1));
    tab[q.tplane] = cp;
    tabe[q.tplane] = e;
    {
        double a = zl[min(2, nz - 1)], c = zl[nz + min(2, nz - 1)], b = diag(min(2, nz - 1));
        double *t = tab + q.tplane, *te = tabe + q.tplane;
#pragma unroll 2
        for (int k = 2; k < nz; ++k) {
            const double p = __dsub_rn(b, __dmul_rn(a, cp)), ck = c;
            const double ei = __dsub_rn(k == nz - 1 ? e_last : 0.0, __dmul_rn(a, e));
            const int kn = min(k + 1, nz - 1);
            a = zl[kn];
            c = zl[nz + kn];
            b = diag(kn);
            const double r = __drcp_rn(p);
            e = __dmul_rn(r, ei);
            cp = __dmul_rn(r, ck);
            t += q.tplane;
            te += q.tplane;
            *t = r;
            *te = e;
        }
    }
    for (int k0 = nz - 2; k0 >= 1; k0 -= 8) {
        double rv[8], ev[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const int k = k0 - p;
            rv[p] = ev[p] = 0.0;
            if (k >= 1) { rv[p] = tab[(size_t)k * q.tplane]; ev[p] = tabe[(size_t)k * q.tplane]; }
        }
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const int k = k0 - p;
            if (k < 1) break;
            const double c = (k == 1) ? rv[p] : __dmul_rn(rv[p], zl[nz + k]);   // row 1 holds c' itself
            e = __dsub_rn(ev[p], __dmul_rn(c, e));
            tabe[(size_t)k * q.tplane] = e;
        }
    }
}

}  // namespace ppf
