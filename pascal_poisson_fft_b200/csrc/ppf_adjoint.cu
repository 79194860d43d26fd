// ppf_adjoint.cu -- transpose of the solve map and the z-metric gradient
// (sm_100a).  The reference has no adjoint; this is the differentiation
// addition to its solve path.
//
// The solve is u = P0 M' f (transforms in x and y, one z system per
// (kx, ky) with the zero mode pinned, inverse transforms, arithmetic-mean
// removal P0).  The x and y operators are symmetric (uniform 3-point,
// periodic or mirror-Neumann); the z operator T = V^-1 S (V = diag(dx3),
// S symmetric: S_{k,k+1} = 1/dmx3_{k+1}), so T^-T = V T^-1 V^-1 for every
// system but the pinned zero mode.  The transpose is therefore
//     M^T g = V M (V^-1 g) + c(z),
// one ordinary solve (any precision, refinement included) between two
// diagonal scalings, plus a per-level constant c that replaces the zero
// mode of V M V^-1 by the transposed pinned system, solved here in FP64
// from the plane sums of g.  Each level's plane mean is removed from g
// before the scaling: that changes only the zero mode (replaced anyway) and
// makes the scaled right-hand side compatible, so the FP64 residual of a
// mixed-precision solve can converge.  With the forward solution u given, the
// gradient of J = <g, u> (g = dJ/du) with respect to the z coefficients is
//     dJ/dam_k = -sum_xy df_k (u_{k-1} - u_k),  dJ/dap_k = -sum_xy df_k (u_{k+1} - u_k),
// with df = M^T g, minus the zero-mode part of the pinned row
// (+ sum_xy df_0 * (sum_xy u_1 - sum_xy u_0) / (nx ny) on ap_0), chained
// to dx3 and dmx3 through am_k = 1/dx3_k/dmx3_k, ap_k = 1/dx3_k/dmx3_{k+1}
// (fft_3d_poisson.f90:1139-1144).  Every reduction is per block in a fixed
// order, then across blocks in a fixed order: the results are deterministic.
#include "ppf_kernels.cuh"

namespace ppf {

namespace {

constexpr int ADJ_TPB = 256;

__device__ __forceinline__ double block_sum(double v, double* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
    __syncthreads();
    return s;  // valid in thread 0
}

// per-(chunk, level) partial sums of g
__global__ void __launch_bounds__(ADJ_TPB) k_adj_sum(const double* __restrict__ g, long plane, long chunk,
                                                      int nchunk, double* __restrict__ colpart)
{
    __shared__ double red[ADJ_TPB / 32];
    const int k = blockIdx.y;
    const long i0 = (long)blockIdx.x * chunk;
    const long i1 = min(plane, i0 + chunk);
    const double* gk = g + (long)k * plane;
    double s = 0.0;
#pragma unroll 8
    for (long i = i0 + threadIdx.x; i < i1; i += ADJ_TPB) s += gk[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) colpart[(long)k * nchunk + blockIdx.x] = s;
}

// sum over the chunks of level k, by one warp (valid in every lane)
__device__ __forceinline__ double chunk_sum(const double* part, int k, int nchunk)
{
    double s = 0.0;
    for (int c = threadIdx.x & 31; c < nchunk; c += 32) s += part[(long)k * nchunk + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Zero-mode correction c(z): the transposed pinned system of the plane sums
// (one block, sm: 4 nz doubles).  One thread's serial sweep, out of shared
// memory so that a row costs its divide and not a round trip to L2; it runs
// as one more block of k_adj_rhs, beside the scaling, instead of alone after
// the solve (38 us at 128 levels).
__device__ __forceinline__ void adj_corr(const double* __restrict__ colpart, int nchunk, int nz,
                                         const double* __restrict__ dx3, const double* __restrict__ dmx3, double nxy,
                                         double* __restrict__ corr, double* sm)
{
    double* const cs = sm;           // plane sums, then d'
    double* const cp = sm + nz;      // c'
    double* const am = sm + 2 * nz;  // am_k = 1/dx3_k/dmx3_k, ap_k = 1/dx3_k/dmx3_{k+1}
    double* const ap = sm + 3 * nz;
    for (int k = threadIdx.x >> 5; k < nz; k += ADJ_TPB / 32) {
        const double s = chunk_sum(colpart, k, nchunk);
        if ((threadIdx.x & 31) == 0) cs[k] = s;
    }
    for (int k = threadIdx.x; k < nz; k += ADJ_TPB) {
        const double inv = __ddiv_rn(1.0, dx3[k + 1]);
        am[k] = k == 0 ? 0.0 : __ddiv_rn(inv, dmx3[k + 1]);
        ap[k] = k == nz - 1 ? 0.0 : __ddiv_rn(inv, dmx3[k + 2]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int k = 0; k < nz; ++k) tot += cs[k];
        // zero mode of M^T g: T00^T x = cs - mean, T00^T having sub-diagonal
        // c_{k-1} (c_0 = 0 at the pin), super-diagonal a_{k+1}, diagonal b_k (b_0 = 1);
        // the scaled right-hand side has no zero mode, so nothing is subtracted
        const double mean = tot / (double)nz;
        double cprev = 0.0, dprev = 0.0;
        for (int k = 0; k < nz; ++k) {
            const double a = (k >= 2) ? ap[k - 1] : 0.0;
            const double c = (k + 1 < nz) ? am[k + 1] : 0.0;
            const double b = (k == 0) ? 1.0 : (-am[k] - ap[k]);
            const double r = 1.0 / (b - a * cprev);
            cprev = c * r;
            dprev = ((cs[k] - mean) - a * dprev) * r;
            cp[k] = cprev;
            cs[k] = dprev;
        }
        for (int k = nz - 2; k >= 0; --k) cs[k] -= cp[k] * cs[k + 1];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nz; k += ADJ_TPB) corr[k] = cs[k] / nxy;
}

// h = (g - plane mean of g) / dx3_k (dense; h may alias g); block (0, 0) of
// the extra column of blocks forms the zero-mode correction
__global__ void __launch_bounds__(ADJ_TPB) k_adj_rhs(const double* g, double* h, const double* __restrict__ dx3,
                                                      const double* __restrict__ dmx3, long plane, long chunk,
                                                      int nchunk, const double* __restrict__ colpart,
                                                      double* __restrict__ corr)
{
    extern __shared__ double adj_sm[];
    __shared__ double mean;
    if (blockIdx.x == 0) {
        if (blockIdx.y == 0) adj_corr(colpart, nchunk, gridDim.y, dx3, dmx3, (double)plane, corr, adj_sm);
        return;
    }
    const int k = blockIdx.y;
    if (threadIdx.x < 32) {
        const double s = chunk_sum(colpart, k, nchunk);
        if (threadIdx.x == 0) mean = s / (double)plane;
    }
    __syncthreads();
    const long i0 = (long)(blockIdx.x - 1) * chunk;
    const long i1 = min(plane, i0 + chunk);
    const double inv = 1.0 / dx3[k + 1], m = mean;
    const long base = (long)k * plane;
    // loads of several rows in flight (g and h may be the same array: each
    // element is read before it is written, by the same thread)
    long i = i0 + threadIdx.x;
    for (; i + 7 * ADJ_TPB < i1; i += 8 * ADJ_TPB) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = g[base + i + q * ADJ_TPB];
#pragma unroll
        for (int q = 0; q < 8; ++q) h[base + i + q * ADJ_TPB] = (v[q] - m) * inv;
    }
    for (; i < i1; i += ADJ_TPB) h[base + i] = (g[base + i] - m) * inv;
}

// df = dx3_k * W + c_k (W: ghosted solution of the scaled right-hand side);
// with u: per-(block, level) partial sums of df (u_{k-1} - u_k),
// df (u_{k+1} - u_k), df and u.  The row and column of an element advance by
// the blocks' stride without a division (a 64-bit one per element made this
// kernel issue-bound: 58 us at 256 x 256 x 128).  The blocks of a level take
// its rows of 256 elements in turn, so that each thread's and each block's
// partial sum runs over the whole plane: the terms of a smooth field cancel
// there, where sums over contiguous pieces grow large before they cancel
// across the pieces (ddmx3 of 70 problems 10 % further from 64 bits with
// 4096-cell pieces than with 16384-cell ones; in turn as near as the latter,
// at the same 540 us a gradient of 256 x 256 x 128).  A thread's last elements
// load together as the others do: one by one 162 x 300 x 120 takes 553 us
// instead of 547.
template <bool GRAD>
__global__ void __launch_bounds__(ADJ_TPB) k_adj_out(const double* __restrict__ W, double* __restrict__ df,
                                                      const double* __restrict__ dx3, const double* __restrict__ corr,
                                                      const double* __restrict__ u, int nx, int ny, int nz, long sy,
                                                      long sz, int nchunk, double* __restrict__ mpart)
{
    __shared__ double red[ADJ_TPB / 32];
    const int k = blockIdx.y;
    const int plane = nx * ny, step = nchunk * ADJ_TPB;
    const double s3 = dx3[k + 1], ck = corr[k];
    const int dj = step / nx, di = step - dj * nx;
    const double* const Wk = W + (long)(k + 1) * sz + sy + 1;
    const double* const uk = GRAD ? u + (long)(k + 1) * sz + sy + 1 : nullptr;
    double* const dk = df + (long)k * plane;
    const long lo = k > 0 ? -sz : 0, hi = k < nz - 1 ? sz : 0;   // the walls' terms are zero
    double sm = 0.0, sp = 0.0, sd = 0.0, su = 0.0;
    int e = blockIdx.x * ADJ_TPB + (int)threadIdx.x;
    int j = e / nx, i = e - j * nx;
    auto next = [&]() -> int {
        const int o = i + j * (int)sy;
        i += di;
        j += dj;
        if (i >= nx) { i -= nx; ++j; }
        return o;
    };
    auto one = [&](double w, int at, double uc, double um, double up) {
        const double v = s3 * w + ck;
        dk[at] = v;
        if constexpr (GRAD) {
            sm += v * (um - uc);
            sp += v * (up - uc);
            sd += v;
            su += uc;
        }
    };
    constexpr int Q = 4;   // elements in flight
    for (; e + (Q - 1) * step < plane; e += Q * step) {
        double w[Q], uc[Q], um[Q], up[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int o = next();
            w[q] = Wk[o];
            if constexpr (GRAD) { uc[q] = uk[o]; um[q] = uk[o + lo]; up[q] = uk[o + hi]; }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) one(w[q], e + q * step, uc[q], um[q], up[q]);
    }
    if (e < plane) {
        // the last elements, their loads in flight as well
        double w[Q - 1], uc[Q - 1], um[Q - 1], up[Q - 1];
#pragma unroll
        for (int q = 0; q < Q - 1; ++q) {
            const int o = next();
            if (e + q * step < plane) {
                w[q] = Wk[o];
                if constexpr (GRAD) { uc[q] = uk[o]; um[q] = uk[o + lo]; up[q] = uk[o + hi]; }
            }
        }
#pragma unroll
        for (int q = 0; q < Q - 1; ++q)
            if (e + q * step < plane) one(w[q], e + q * step, uc[q], um[q], up[q]);
    }
    if constexpr (GRAD) {
        sm = block_sum(sm, red);
        sp = block_sum(sp, red);
        sd = block_sum(sd, red);
        su = block_sum(su, red);
        if (threadIdx.x == 0) {
            const long q = (long)nz * nchunk, at = (long)k * nchunk + blockIdx.x;
            mpart[at] = sm;
            mpart[q + at] = sp;
            mpart[2 * q + at] = sd;
            mpart[3 * q + at] = su;
        }
    }
}

// reduce the partials per level and chain dJ/dam, dJ/dap to dx3, dmx3
// (Fortran index j = 0..nz+1; cell k is j = k+1)
__global__ void __launch_bounds__(ADJ_TPB) k_adj_metric(const double* __restrict__ mpart, int nchunk, int nz,
                                                         double nxy, const double* __restrict__ am,
                                                         const double* __restrict__ ap, const double* __restrict__ dx3,
                                                         const double* __restrict__ dmx3, double* __restrict__ ddx3,
                                                         double* __restrict__ ddmx3, double* __restrict__ wk)
{
    double* dam = wk;
    double* dap = wk + nz;
    double* sdu = wk + 2 * nz;  // [0] sum df_0, [1] sum u_0, [2] sum u_1
    const long q = (long)nz * nchunk;
    for (int k = threadIdx.x; k < nz; k += blockDim.x) {
        double a = 0.0, b = 0.0, d = 0.0, s = 0.0;
        for (int c = 0; c < nchunk; ++c) {
            const long at = (long)k * nchunk + c;
            a += mpart[at];
            b += mpart[q + at];
            d += mpart[2 * q + at];
            s += mpart[3 * q + at];
        }
        dam[k] = (k == 0) ? 0.0 : -a;
        dap[k] = (k == nz - 1) ? 0.0 : -b;
        if (k == 0) { sdu[0] = d; sdu[1] = s; }
        if (k == 1) sdu[2] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0 && nz > 1) dap[0] += sdu[0] * (sdu[2] - sdu[1]) / nxy;
    __syncthreads();
    for (int j = threadIdx.x; j < nz + 2; j += blockDim.x) {
        double gx = 0.0, gm = 0.0;
        if (j >= 1 && j <= nz) {
            const int k = j - 1;
            gx = -(dam[k] * am[k] + dap[k] * ap[k]) / dx3[j];
            gm -= dam[k] * am[k] / dmx3[j];
        }
        if (j >= 2 && j <= nz + 1) {
            const int k = j - 2;
            gm -= dap[k] * ap[k] / dmx3[j];
        }
        if (ddx3) ddx3[j] = gx;
        if (ddmx3) ddmx3[j] = gm;
    }
}

}  // namespace

int adjoint_chunks(long plane, long* chunk)
{
    // 4096 cells a block: enough blocks and loads in flight to stream a plane
    const long target = 4096;
    int n = (int)((plane + target - 1) / target);
    if (n < 1) n = 1;
    if (n > 64) n = 64;
    long c = (plane + n - 1) / n;
    c = (c + ADJ_TPB - 1) / ADJ_TPB * ADJ_TPB;
    *chunk = c;
    return (int)((plane + c - 1) / c);
}

cudaError_t launch_adj_rhs(const double* g, double* h, const double* dx3, const double* dmx3, const Geom& gm,
                           long chunk, int nchunk, double* colpart, double* corr, cudaStream_t st)
{
    const long plane = (long)gm.nx * gm.ny;
    k_adj_sum<<<dim3(nchunk, gm.nz), ADJ_TPB, 0, st>>>(g, plane, chunk, nchunk, colpart);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // 32 KB of shared memory at the tallest column (1024 levels)
    k_adj_rhs<<<dim3(nchunk + 1, gm.nz), ADJ_TPB, 4 * sizeof(double) * gm.nz, st>>>(g, h, dx3, dmx3, plane, chunk,
                                                                                  nchunk, colpart, corr);
    return cudaGetLastError();
}

cudaError_t launch_adj_out(const double* W, double* df, const double* dx3, const double* corr, const double* u,
                           const Geom& gm, int nchunk, double* mpart, cudaStream_t st)
{
    auto kern = u ? k_adj_out<true> : k_adj_out<false>;
    kern<<<dim3(nchunk, gm.nz), ADJ_TPB, 0, st>>>(W, df, dx3, corr, u, gm.nx, gm.ny, gm.nz, gm.pstride_y, gm.pstride_z,
                                                 nchunk, mpart);
    return cudaGetLastError();
}

cudaError_t launch_adj_metric(const double* mpart, int nchunk, const Geom& gm, const double* am, const double* ap,
                              const double* dx3, const double* dmx3, double* ddx3, double* ddmx3, double* wk,
                              cudaStream_t st)
{
    k_adj_metric<<<1, ADJ_TPB, 0, st>>>(mpart, nchunk, gm.nz, (double)gm.nx * gm.ny, am, ap, dx3, dmx3, ddx3,
                                        ddmx3, wk);
    return cudaGetLastError();
}

}  // namespace ppf
