// band.cuh — SymmetricBandMatrix.Factorize + Solve (Solver/SymmetricBandMatrix.cs:60-111) in one CTA: the plan, the kernel
// of the bands too wide for band_tri.cuh's shared-memory triangle, and the launch.
//
// The band is stored row-major, row i holding L[i][i-b .. i] at offsets 0 .. b (diagonal last). The reference's
// factorisation subtracts, for every entry (i, j), the products L_ik L_jk in ascending k, each product rounded
// before the subtraction, then divides by L_jj (or takes the square root on the diagonal); its solves subtract
// in ascending k (forward) and descending i (backward). Any schedule that keeps that order per entry gives the
// same bits. The wide kernel factorises in place in global memory, by panels of 32 columns:
//
//   A  panel factorisation: column by column inside the panel (scale, update of the panel's later columns,
//      pivot), two barriers per column;
//   B  trailing update of the rows below the panel by the whole panel: 4 x 4 register tiles, each entry's
//      products subtracted in ascending k (one load per two multiplies);
//   C  the forward substitution of the panel's rows and its update of the b rows below, by one warp, while the
//      other warps run B.
//
// The backward substitution then walks the rows in blocks of 32 from the bottom: one warp solves the block's
// triangle, all threads update the b rows above it (products in descending i).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "band_tri.cuh"

namespace ifea {
namespace band {

constexpr int kThreads = 512;
constexpr int kPanel = 32;

struct Plan {
    bool tri = true;   // the triangle kernel, wherever its window fits shared memory (half-bandwidth up to 188; at 185
                       // it takes 16 ms where the in-place kernel takes 46); else in place in global memory
    size_t bytes = 0;  // dynamic shared memory of the launch
};

inline Plan plan(int, int b)
{
    Plan p;
    p.tri = tri_fits(b);
    p.bytes = p.tri ? tri_bytes(b) : (size_t)(2 * kPanel + b) * sizeof(int64_t);
    return p;
}

// err_row[0] = -1 on success, else the first row whose pivot was not positive; pivot[0] that pivot.
static __global__ void __launch_bounds__(kThreads) k_band_wide(int n, int b, double *__restrict__ a, double *__restrict__ rhs,
                                                               int32_t *err_row, double *pivot)
{
    extern __shared__ __align__(16) unsigned char band_smem[];
    __shared__ int s_bad;
    __shared__ double xs[kPanel];
    __shared__ int64_t brow[kPanel];  // row offsets of a backward block
    const int w = b + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    int64_t *rowoff = (int64_t *)band_smem;  // rowoff[t]: offset of entry (k0 + t, 0) in the band (may be negative)
    auto entry = [&](int i, int j) -> double & { return a[(int64_t)i * w + (j - i + b)]; };
    auto do_pivot = [&](int k) {
        double s = entry(k, k);
        if (!(s > 0) || isnan(s)) {
            s_bad = k;
            *pivot = s;
        } else {
            entry(k, k) = sqrt(s);
        }
    };
    if (tid == 0) {
        s_bad = -1;
        *pivot = 0.0;
    }
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += kPanel) {
        const int k1 = min(n, k0 + kPanel);
        const int last = min(n - 1, k1 - 1 + b);  // last row the panel's columns reach
        for (int t = tid; t <= last - k0; t += kThreads) {
            int i = k0 + t;
            rowoff[t] = (int64_t)i * w - i + b;
        }
        if (tid == 0) do_pivot(k0);
        __syncthreads();
        if (s_bad >= 0) break;
        auto P = [&](int i, int j) -> double & { return a[rowoff[i - k0] + j]; };
        // A
        for (int k = k0; k < k1; k++) {
            const double lkk = P(k, k);
            const int r = min(n - 1, k + b);
            for (int i = k + 1 + tid; i <= r; i += kThreads) P(i, k) = P(i, k) / lkk;
            __syncthreads();
            const int c = k1 - 1 - k, rows = r - k;
            for (int idx = tid; idx < c * rows; idx += kThreads) {
                int di = idx / c, dj = idx - di * c;
                int i = k + 1 + di, j = k + 1 + dj;
                if (j <= i) {
                    double &e = P(i, j);
                    e = e - P(i, k) * P(j, k);
                    if (idx == 0) do_pivot(k + 1);  // (k + 1, k + 1) is final now
                }
            }
            __syncthreads();
            if (s_bad >= 0) break;
        }
        if (s_bad >= 0) break;
        // B on all warps but the last, C on the last warp (when there is a right-hand side)
        const int nbw = rhs ? kThreads - 32 : kThreads;
        if (tid < nbw) {
            const int m = last - k1 + 1;  // rows below the panel
            const int T = (m + 3) >> 2;
            const int pairs = ((T + 1) >> 1) * (T + 1);
            for (int idx = tid; idx < pairs; idx += nbw) {
                int q = idx / (T + 1), cc = idx - q * (T + 1);
                int ti, tj;
                if (cc <= q) {
                    ti = q;
                    tj = cc;
                } else {
                    ti = T - 1 - q;
                    tj = cc - q - 1;
                    if (ti == q) continue;  // the middle tile row of an odd count is covered by the first branch
                }
                const int ib = k1 + 4 * ti, jb = k1 + 4 * tj;
                // rows past the panel's reach borrow row ib's (or jb's) entries: computed, never stored
                int64_t pi[4], pj[4];
                int kf[4];
                bool iv[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    int i = ib + u, j = jb + u;
                    iv[u] = i <= last;
                    pi[u] = rowoff[(iv[u] ? i : ib) - k0];
                    pj[u] = rowoff[(j <= last ? j : jb) - k0];
                    kf[u] = max(k0, i - b);
                }
                double s[4][4];
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int v = 0; v < 4; v++) s[u][v] = (iv[u] && jb + v <= ib + u) ? a[pi[u] + jb + v] : 0.0;
                // the first rows' earliest columns lie outside the later rows' band: those few steps are masked
                const int kfull = min(k1, kf[3]);
                for (int k = kf[0]; k < kfull; k++) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (k < kf[u]) continue;
                        double li = a[pi[u] + k];
#pragma unroll
                        for (int v = 0; v < 4; v++)
                            if (jb + v <= ib + u) s[u][v] = s[u][v] - li * a[pj[v] + k];
                    }
                }
                // every entry of the tile takes every remaining step: loads one step ahead
                if (kfull < k1) {
                    double li[4], lj[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        li[u] = a[pi[u] + kfull];
                        lj[u] = a[pj[u] + kfull];
                    }
                    for (int k = kfull; k < k1; k++) {
                        double ni[4], nj[4];
                        const int kn = min(k + 1, k1 - 1);
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            ni[u] = a[pi[u] + kn];
                            nj[u] = a[pj[u] + kn];
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++)
#pragma unroll
                            for (int v = 0; v < 4; v++) s[u][v] = s[u][v] - li[u] * lj[v];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            li[u] = ni[u];
                            lj[u] = nj[u];
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int v = 0; v < 4; v++)
                        if (iv[u] && jb + v <= ib + u) a[pi[u] + jb + v] = s[u][v];
            }
        } else {
            // C: forward substitution of rows [k0, k1), then their products out of the rows below
            const int np = k1 - k0;
            double y = lane < np ? rhs[k0 + lane] : 0.0;
            for (int kk = 0; kk < np; kk++) {
                const double yd = y / P(k0 + kk, k0 + kk);  // every lane divides; lane kk keeps it
                if (lane == kk) y = yd;
                double xk = __shfl_sync(FULL, y, kk);
                if (lane > kk && lane < np && lane - kk <= b) y = y - P(k0 + lane, k0 + kk) * xk;
            }
            if (lane < np) {
                rhs[k0 + lane] = y;
                xs[lane] = y;
            }
            __syncwarp();
            for (int i = k1 + lane; i <= last; i += 32) {
                double rr = rhs[i];
                for (int k = max(k0, i - b); k < k1; k++) rr = rr - P(i, k) * xs[k - k0];
                rhs[i] = rr;
            }
        }
        __syncthreads();
    }
    __syncthreads();
    if (s_bad >= 0) {
        if (tid == 0) *err_row = s_bad;
        return;
    }
    if (tid == 0) *err_row = -1;
    if (!rhs) return;

    // backward substitution, blocks of 32 rows from the bottom
    for (int i1 = n; i1 > 0;) {
        const int i0 = max(0, i1 - kPanel);
        const int np = i1 - i0;
        if (warp == 0) {
            // lane l: row i0 + l; the block's row offsets go to brow[] for the update of the rows above
            int64_t ro = lane < np ? (int64_t)(i0 + lane) * w - (i0 + lane) + b : 0;
            brow[lane] = ro;
            double y = lane < np ? rhs[i0 + lane] : 0.0, d = lane < np ? a[ro + i0 + lane] : 1.0;
            __syncwarp();
            double e = 0.0;  // L(i, i0 + lane) of the current step's row i, loaded one step ahead
            if (np >= 1 && lane < np - 1 && np - 1 - lane <= b) e = a[brow[np - 1] + i0 + lane];
            for (int kk = np - 1; kk >= 0; kk--) {
                double en = 0.0;
                if (kk >= 1 && lane < kk - 1 && kk - 1 - lane <= b) en = a[brow[kk - 1] + i0 + lane];
                const double yd = y / d;  // every lane divides; lane kk keeps it
                if (lane == kk) y = yd;
                const double xi = __shfl_sync(FULL, y, kk);
                if (lane < kk && kk - lane <= b) y = y - e * xi;
                e = en;
            }
            if (lane < np) {
                rhs[i0 + lane] = y;
                xs[lane] = y;
            }
        }
        __syncthreads();
        for (int k = max(0, i0 - b) + tid; k < i0; k += kThreads) {
            double rr = rhs[k];
            for (int i = min(i1 - 1, k + b); i >= i0; i--) rr = rr - a[brow[i - i0] + k] * xs[i - i0];
            rhs[k] = rr;
        }
        __syncthreads();
        i1 = i0;
    }
}

inline const void *kernel_of(const Plan &p) { return p.tri ? (const void *)k_band_tri : (const void *)k_band_wide; }

// Launch on `st` with the plan for (n, b); the caller has raised the kernel's shared-memory limit to plan.bytes.
inline void launch(const Plan &p, int n, int b, double *a, double *rhs, int32_t *err_row, double *pivot,
                   cudaStream_t st)
{
    void *args[] = {&n, &b, &a, &rhs, &err_row, &pivot};
    cudaLaunchKernel(kernel_of(p), dim3(1), dim3(p.tri ? kTriThreads : kThreads), args, p.bytes, st);
}

}  // namespace band
}  // namespace ifea
