// ppf_y_dev.cuh -- device bodies of the y-direction transforms, shared by
// the y kernels (ppf_y.cu) and the persistent batch kernel (ppf_batch.cu).
// One call transforms column block `cblk` (W consecutive spectral columns)
// of z-plane `z`, all ny rows, in shared memory (ppf_fft.cuh); the spectral
// rows stay in the [z][ky][kx] order the z solve reads, so no transpose pass
// exists (the reference transposes before and after every y transform,
// 01_Fortran/src/fft_3d_poisson.f90:421-559, 1035-1119).
//   Y_C2C  : complex FFT along y (periodic y on complex x-spectra)
//   Y_CDCT : DCT-II of real and imaginary parts at once (Neumann y; also the
//            real N-N case with adjacent kx columns packed as complex)
//   Y_RPAIR: real FFT of two packed real columns (DCT-x data, periodic y);
//            ny/2+1 rows of two complex columns per packed pair
#pragma once
#include "ppf_xy_common.cuh"

namespace ppf {

constexpr int ct_log2y(int w) { return w <= 1 ? 0 : 1 + ct_log2y(w / 2); }

template <typename T, int KIND, typename SH>
__device__ __forceinline__ void yfwd(const cx<T>* in, long in_pitch, cx<T>* __restrict__ out,
                                     long out_pitch, int ncols, const Geom& g, const FftSched& sch, int Wrt, int lgWrt,
                                     const cx<T>* __restrict__ tw_ny, const cx<T>* __restrict__ tw_dct,
                                     const int* skip, int cblk, int z)
{
    if (skip && *skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* s = reinterpret_cast<cx<T>*>(smem_raw);
    constexpr bool CT = SH::CT;
    const int W = CT ? SH::W : Wrt;
    const int lgW = CT ? ct_log2y(SH::W) : lgWrt;
    const int NTH = CT ? SH::NT : (int)blockDim.x;
    const int ny = CT ? SH::N : g.ny;
    const int col0 = cblk * W;
    const int nc = ncols - col0 < W ? ncols - col0 : W;   // columns of the tile
    const cx<T>* inp = in + (long)z * ny * in_pitch + col0;
    const int ip = (int)in_pitch, op = (int)out_pitch;
    const int E = ny << lgW;

    // run-time tiles: eight elements a thread at most, the loads of four issued together
#pragma unroll (CT ? 1 : 4)
    for (int e = threadIdx.x; e < E; e += NTH) {
        const int l = e & (W - 1), y = e >> lgW;
        cx<T> v = mk<T>((T)0, (T)0);
        if (l < nc) v = inp[y * ip + l];
        int row = y;
        if (KIND == Y_CDCT) row = (y & 1) ? (ny - 1 - (y >> 1)) : (y >> 1);
        s[tidx<T, SH>(row, l, W)] = v;
    }
    __syncthreads();
    tile_fft<T, false, SH>(s, sch, W, lgW, tw_ny);

    if (KIND == Y_C2C) {
        cx<T>* outp = out + (long)z * ny * out_pitch + col0;
        for (int e = threadIdx.x; e < E; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            if (l < nc) outp[k * op + l] = s[tidx<T, SH>(k, l, W)];
        }
    } else if (KIND == Y_CDCT) {
        // X_k and X_{n-k} from one read of V_k, V_{n-k}: with p = w V_k, q =
        // conj(w) V_{n-k}, w = e^{-i pi k/(2n)}, X_k = p + q and, as the
        // twiddle of n - k is -i conj(w), X_{n-k} = i (p - q)
        cx<T>* outp = out + (long)z * ny * out_pitch + col0;
        const int Eh = (ny / 2 + 1) << lgW;
        for (int e = threadIdx.x; e < Eh; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            if (l >= nc) continue;
            const cx<T> V = s[tidx<T, SH>(k, l, W)];
            const cx<T> Vp = s[tidx<T, SH>(k == 0 ? 0 : ny - k, l, W)];
            const cx<T> w = ldg(tw_dct + k);
            if constexpr (sizeof(T) == 8) {
                const cx<T> p = cmul(w, V), q = cmul(conj(w), Vp);
                outp[k * op + l] = p + q;
                if (k > 0 && 2 * k < ny) outp[(ny - k) * op + l] = mk<T>(q.y - p.y, p.x - q.x);
            } else {
                // (FP32 results stay as they are to the bit)
                auto one = [&](cx<T> a, cx<T> b, cx<T> t) {
                    cx<T> X;
                    X.x = t.x * (a.x + b.x) - t.y * (a.y - b.y);
                    X.y = t.x * (a.y + b.y) + t.y * (a.x - b.x);
                    return X;
                };
                outp[k * op + l] = one(V, Vp, w);
                if (k > 0 && 2 * k < ny) outp[(ny - k) * op + l] = one(Vp, V, ldg(tw_dct + (ny - k)));
            }
        }
    } else {
        const int my = ny / 2 + 1;
        cx<T>* outp = out + (long)z * my * out_pitch + 2 * col0;
        const int Eo = my << lgW;
        for (int e = threadIdx.x; e < Eo; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            if (l >= nc) continue;
            const cx<T> zk = s[tidx<T, SH>(k, l, W)];
            const cx<T> zc = conj(s[tidx<T, SH>(k == 0 ? 0 : ny - k, l, W)]);
            const cx<T> X1 = (zk + zc) * (T)0.5;
            const cx<T> D = zk - zc;
            const cx<T> X2 = mk<T>(D.y * (T)0.5, -D.x * (T)0.5);
            outp[k * op + 2 * l] = X1;
            outp[k * op + 2 * l + 1] = X2;
        }
    }
}

template <typename T, int KIND, typename SH>
__device__ __forceinline__ void yinv(const cx<T>* in, long in_pitch, cx<T>* __restrict__ out,
                                     long out_pitch, int ncols, const Geom& g, const FftSched& sch, int Wrt, int lgWrt,
                                     const cx<T>* __restrict__ tw_ny, const cx<T>* __restrict__ tw_dct,
                                     const double* dc_shift, const int* skip, int cblk,
                                     int z)
{
    if (skip && *skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* s = reinterpret_cast<cx<T>*>(smem_raw);
    constexpr bool CT = SH::CT;
    const int W = CT ? SH::W : Wrt;
    const int lgW = CT ? ct_log2y(SH::W) : lgWrt;
    const int NTH = CT ? SH::NT : (int)blockDim.x;
    const int ny = CT ? SH::N : g.ny;
    const int col0 = cblk * W;
    const int E = ny << lgW;
    // the zero mode's z-average, removed from the (kx,ky) = (0,0) coefficient
    const T shift = (col0 == 0 && dc_shift) ? (T)*dc_shift : (T)0;

    const int nc = ncols - col0 < W ? ncols - col0 : W;   // columns of the tile
    const int ip = (int)in_pitch, op = (int)out_pitch;
    if (KIND == Y_C2C) {
        const cx<T>* inp = in + (long)z * ny * in_pitch + col0;
#pragma unroll (CT ? 1 : 4)
        for (int e = threadIdx.x; e < E; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            cx<T> v = mk<T>((T)0, (T)0);
            if (l < nc) v = inp[k * ip + l];
            if (e == 0) v.x -= shift;
            s[tidx<T, SH>(k, l, W)] = v;
        }
    } else if (KIND == Y_CDCT) {
        // Z_k = e^{i pi k/(2n)} (X_k - i X_{n-k}), X_n = 0, per real component
        // (cuda_Poisson_DCT_b_pre, fft_3d_poisson.f90:971-1011), both
        // components packed into one complex inverse FFT: Z_k = conj(w) (X_k -
        // i X_{n-k}), Z_{n-k} = w (X_k + i X_{n-k}) from one read of the pair
        const cx<T>* inp = in + (long)z * ny * in_pitch + col0;
        const int Eh = (ny / 2 + 1) << lgW;
#pragma unroll (CT ? 1 : 2)
        for (int e = threadIdx.x; e < Eh; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            cx<T> Z = mk<T>((T)0, (T)0), Zp = Z;
            if (l < nc) {
                cx<T> X = inp[k * ip + l];
                if (e == 0) X.x -= shift;
                const cx<T> Xp = (k == 0) ? mk<T>((T)0, (T)0) : inp[(ny - k) * ip + l];
                const cx<T> w = ldg(tw_dct + k);
                if constexpr (sizeof(T) == 8) {
                    Z = cmul(conj(w), mk<T>(X.x + Xp.y, X.y - Xp.x));
                    Zp = cmul(w, mk<T>(X.x - Xp.y, X.y + Xp.x));
                } else {
                    // (FP32 results stay as they are to the bit)
                    auto one = [&](cx<T> a, cx<T> b, cx<T> t) {
                        const T c = t.x, sn = -t.y;
                        const T zax = c * a.x + sn * b.x, zay = sn * a.x - c * b.x;
                        const T zbx = c * a.y + sn * b.y, zby = sn * a.y - c * b.y;
                        return mk<T>(zax - zby, zay + zbx);
                    };
                    Z = one(X, Xp, w);
                    if (k > 0) Zp = one(Xp, X, ldg(tw_dct + (ny - k)));
                }
            }
            s[tidx<T, SH>(k, l, W)] = Z;
            if (k > 0 && 2 * k < ny) s[tidx<T, SH>(ny - k, l, W)] = Zp;
        }
    } else {
        // Z_k = X1_k + i X2_k of the two real columns, Z_{n-k} from the same
        // pair (both columns' spectra are Hermitian)
        const int my = ny / 2 + 1;
        const cx<T>* inp = in + (long)z * my * in_pitch + 2 * col0;
        const int Eh = my << lgW;
#pragma unroll (CT ? 1 : 2)
        for (int e = threadIdx.x; e < Eh; e += NTH) {
            const int l = e & (W - 1), k = e >> lgW;
            cx<T> Z = mk<T>((T)0, (T)0), Zp = Z;
            if (l < nc) {
                cx<T> X1 = inp[k * ip + 2 * l];
                cx<T> X2 = inp[k * ip + 2 * l + 1];
                if (k == 0 || 2 * k == ny) { X1.y = (T)0; X2.y = (T)0; }
                if (e == 0) X1.x -= shift;
                Z = mk<T>(X1.x - X2.y, X1.y + X2.x);
                Zp = mk<T>(X1.x + X2.y, X2.x - X1.y);
            }
            s[tidx<T, SH>(k, l, W)] = Z;
            if (k > 0 && 2 * k < ny) s[tidx<T, SH>(ny - k, l, W)] = Zp;
        }
    }
    __syncthreads();
    tile_fft<T, true, SH>(s, sch, W, lgW, tw_ny);

    cx<T>* outp = out + (long)z * ny * out_pitch + col0;
    for (int e = threadIdx.x; e < E; e += NTH) {
        const int l = e & (W - 1), i = e >> lgW;
        if (l >= nc) continue;
        int n = i;
        // inverse Makhoul order (cuda_Poisson_DCT_b_post, :1013-1033)
        if (KIND == Y_CDCT) n = (i & 1) ? (ny / 2 + ((ny - 1 - i) >> 1)) : (i >> 1);
        outp[i * op + l] = s[tidx<T, SH>(n, l, W)];
    }
}

}  // namespace ppf
