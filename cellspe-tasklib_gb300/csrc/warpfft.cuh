// Complex FFTs of 64 to 1024 points in the registers of 8, 16 or 32 lanes,
// shared by the batched transforms and the spectrometer.
//
// M = L R points by L lanes (L divides R): lane l holds z[l + L j], j < R, in
// v[j].  DFT-R over j, twiddle W_M^(l k1), one transpose through the group's
// tile in shared memory, and R/L DFT-Ls, after which lane l holds
//     v[c L + k2] = Z[(l + L c) + R k2],   c < R/L, k2 < L.
// No barrier wider than a warp: groups never wait on one another.
#pragma once
#include "common.cuh"

// PK: packed sums, FINE: eighth turns with cos(pi/4) as two terms (common.cuh).
template <int L, int R, bool PK = true, bool FINE = false> struct WarpFft {
    static_assert(R % L == 0 && L >= 8 && L <= 32 && R <= 32, "lanes and points per lane");
    static constexpr int M = L * R, CPL = R / L;
    static constexpr int TILE = R * (L + 1);         // float2 per group; the odd row keeps both passes conflict-free
    static constexpr int TWIDDLES = R * L;           // float2 per CTA

    // The CTA's twiddle table [R][L] from tw = exp(-2 pi i m / (M tws)).
    static CS_DEV void fill(float2* tab, const float2* __restrict__ tw, int tws)
    {
        for (int i = threadIdx.x; i < TWIDDLES; i += blockDim.x) tab[i] = __ldg(tw + (i / L) * (i % L) * tws);
    }

    static CS_DEV void run(float2 (&v)[R], float2* tile, int lane, const float2* tab)
    {
        Dft<R, PK, FINE>::run(v);
#pragma unroll
        for (int e = 1; e < R; e++) v[e] = cmul(v[e], tab[e * L + lane]);
#pragma unroll
        for (int e = 0; e < R; e++) tile[e * (L + 1) + lane] = v[e];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < CPL; c++)
#pragma unroll
            for (int n = 0; n < L; n++) v[c * L + n] = tile[(lane + L * c) * (L + 1) + n];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < CPL; c++) Dft<L, PK, FINE>::run(v + c * L);
    }

    // Real-FFT split of the result (z[n] = x[2n] + i x[2n+1], N = 2 M): calls
    // f(i, k, X[k], X[M - k]) for this lane's pairs, i = 0 .. R/2 - 1 a constant of the unrolled
    // code, and g(X[M/2]) on lane 0.  With s = Z[k] + conj(Z[M-k]), d = Z[k] -
    // conj(Z[M-k]) and t = (W_N^k / 2) d: X[k] = s/2 - i t, X[M-k] = conj(s/2 + i t).
    // wh(c, k2) = W_N^k / 2.  Z[M - k] of k = k1 + R k2 lies in lane L - l,
    // column R/L - 1 - c, register L - 1 - k2 (lane 0: its own column R/L - c,
    // column 0 in register (L - k2) mod L).
    template <class T, class F, class G> static CS_DEV void split(const float2 (&v)[R], int lane, T wh, F f, G g)
    {
        const int src = (L - lane) & (L - 1);
#pragma unroll
        for (int c = 0; c < CPL; c++)
#pragma unroll
            for (int k2 = 0; k2 < L / 2; k2++) {
                float2 zb;
                zb.x = __shfl_sync(0xffffffffu, v[(CPL - 1 - c) * L + L - 1 - k2].x, src, L);
                zb.y = __shfl_sync(0xffffffffu, v[(CPL - 1 - c) * L + L - 1 - k2].y, src, L);
                if (lane == 0) zb = c == 0 ? v[(L - k2) % L] : v[(CPL - c) * L + L - 1 - k2];
                float2 X1, X2;
                pair(v[c * L + k2], zb, wh(c, k2), X1, X2);
                f(c * (L / 2) + k2, lane + L * c + R * k2, X1, X2);
            }
        if (lane == 0) {
            // k = M/2 pairs with itself: W_N^(M/2) = -i
            const float2 z = v[L / 2];
            g(make_float2(z.x, -z.y));
        }
    }

    // w W_(2L)^k2, k2 < L/2 a constant: wh(c, k2) from w = W_N^(lane + L c) / 2, by a product
    static CS_DEV float2 rot_half(float2 w, int k2)
    {
        if (k2 == 0) return w;
        return cmul(w, L == 32 ? w64c(k2) : w32((32 / (2 * L)) * k2));
    }

private:
    static CS_DEV void pair(float2 za, float2 zb, float2 w, float2& X1, float2& X2)
    {
        const float2 s = make_float2(za.x + zb.x, za.y - zb.y);
        const float2 d = make_float2(za.x - zb.x, za.y + zb.y);
        const float2 t = cmul(w, d);
        X1 = make_float2(fmaf(0.5f, s.x, t.y), fmaf(0.5f, s.y, -t.x));
        X2 = make_float2(fmaf(0.5f, s.x, -t.y), -fmaf(0.5f, s.y, t.x));
    }
};
