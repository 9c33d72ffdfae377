// band_tri.cuh — SymmetricBandMatrix.Factorize + Solve (Solver/SymmetricBandMatrix.cs:60-111) in one CTA for bands whose
// active triangle fits shared memory (half-bandwidth up to about 190).
//
// The reference subtracts, for every entry (i, j), the products L_ik L_jk in ascending k, each rounded before the
// subtraction, then divides by L_jj (or takes the square root on the diagonal); its solves subtract in ascending k
// (forward) and descending i (backward). Any schedule that keeps that order per entry gives the same bits. What
// bounds it is the chain from one pivot to the next (root, quotient, one product, one subtraction), and for wide bands
// the products themselves (a multiplication and a subtraction each: contraction would change the bits). Per block
// of eight columns, two barriers apart:
//   A   the first warps factor the block, a row a lane (the right-hand side is one more row: its forward substitution
//       is the same arithmetic), every lane along with the whole 8 x 8 diagonal block in registers: no exchange lies
//       on the pivot chain. The other warps subtract the block before from the columns beyond this one, write that
//       block's rows of L back and fetch the rows that enter the window;
//   B   the next block's columns, less this block's products, into the buffer that A starts from.
// The window holds the pairs of b + 16 consecutive indices, taken modulo b + 16, packed as a triangle: the pair {i, j}
// has one place whichever index is the row, and the place of a retired column is that of the row that enters, so
// nothing moves. The triangle's rows are padded to 1 modulo 16 entries, so that a warp's 32 consecutive rows (or columns)
// of one column (row) lie on distinct banks.
//
// Root and quotients: the correctly rounded root and reciprocal of a pivot by Goldschmidt's iteration and one exact
// residual correction each (Markstein, "Computation of elementary functions on the IBM RISC System/6000", 1990), both
// verified by their exact residuals; a quotient is then two residual corrections with that reciprocal, correctly
// rounded by Markstein's theorem: five dependent operations instead of a division. A warp runs a block without a
// branch and does it over with sqrt() and / when anything in it lay outside the conditions (exponents, a residual out of
// bounds, a significand of all ones, a pivot that is not positive).
//
// Measured (B200, factor and solve): 2,562 equations, half-bandwidth 85 (20 x 60 quads) 5.1 -> 1.74 ms; 3,001 x 141
// 8.3 -> 2.8 ms; 12,144 x 185 (45 x 131 quads) 46.3 -> 16.2 ms; 1,000 x 31 2.1 -> 0.52 ms, against the kernel with a panel
// chain of divisions and two barriers per eight columns (the third with the band in global memory). Of a block's 9,000
// cycles at half-bandwidth 85, 4,000 are the factoring warps' chain, at 185 16,000 of 19,000 the update's FP64 operations.
// Pivots and column entries exchanged by shuffles cost 470-660 cycles a column instead of about 400; 512 threads spill.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace ifea {
namespace band {

constexpr int kTriThreads = 384;     // 168 registers a thread: the diagonal block and a row, or a 4 x 4 tile, without spills
constexpr int kTriWorkers = kTriThreads - 32;
constexpr int kTriPitch = 10;      // doubles per row of the eight-column buffers (16-byte rows on distinct banks)
constexpr int kTriMaxSmem = 226 * 1024;
constexpr int kBackRows = 32;      // rows of a block of the backward substitution

// First entry of row p of the packed triangle: rows of p + 1 entries, padded to 1 modulo 16.
__host__ __device__ inline int tri_row(int p)
{
    const int t = (p - 1) >> 4, r = (p - 1) & 15;
    return p == 0 ? 0 : p + 16 * (8 * t * (t + 1) + r * (t + 1));
}
// Shared memory of the factorisation (window, the block to come, two factored blocks, right-hand side) and of the backward substitution
// (two blocks of rows, the circular solution), whichever is larger.
__host__ __device__ inline size_t tri_bytes(int b)
{
    const size_t W = b + 16, R = b + 8, w = b + 1;
    const size_t fwd = (size_t)tri_row((int)W) + 1 + 3 * (R + 1) * kTriPitch + W;
    const size_t bwd = 2 * kBackRows * (w | 1) + b + 4 * kBackRows;
    return (fwd > bwd ? fwd : bwd) * sizeof(double);
}
inline bool tri_fits(int b) { return tri_bytes(b) <= (size_t)kTriMaxSmem; }

// A pivot's root l and what its column's quotients need: y0 about 1 / l, y = 1 / l correctly rounded.
struct PivotRoot {
    double l, y0, y;
};
__device__ __forceinline__ double ulp_of(double v)
{
    return __hiloint2double((__double2hiint(v) & 0x7ff00000) - (52 << 20), 0);
}
__device__ __forceinline__ bool significand(double v, int hi_bits, int lo_bits)
{
    return (__double2hiint(v) & 0xfffff) == hi_bits && __double2loint(v) == lo_bits;
}
__device__ __forceinline__ PivotRoot pivot_root(double p)
{
    PivotRoot q;
    double s;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(s) : "d"(p));
    double g = p * s, h = 0.5 * s;
    double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    q.l = fma(fma(-g, g, p), h, g);
    q.y0 = h + h;
    q.y = fma(q.y0, fma(-q.l, q.y0, 1.0), q.y0);
    return q;
}
// whether l = RN(sqrt(p)) and quotient() by it is a correctly rounded division: l is RN(sqrt(p)) exactly when p lies within
// half a unit of l's last place squared, -l u < p - l^2 <= l u (p - l^2 is exact, and a multiple of u^2); y = RN(1 / l)
// when |1 - l y| <= l u_y / 2. Significands of 1 have a smaller unit below: accepted only where the residual is zero.
__device__ __forceinline__ bool pivot_ok(double p, const PivotRoot &q)
{
    const double e = fma(-q.l, q.l, p), lu = q.l * ulp_of(q.l);
    const double f = fma(-q.l, q.y, 1.0), hy = 0.5 * q.l * ulp_of(q.y);
    const bool exact = e == 0.0 && f == 0.0;
    const bool plain = !significand(q.l, 0, 0) && !significand(q.y, 0, 0) && !significand(q.l, 0xfffff, -1);
    return p > 1e-30 && p < 1e30 && ((e <= lu && e > -lu && fabs(f) <= hy && plain) || exact);
}
// a / l; ok is cleared when a's exponent is outside the range in which no operation underflows or overflows (a zero
// is fine; a negative zero keeps its sign only with SIGN, else it clears ok)
template <bool SIGN>
__device__ __forceinline__ double quotient(double a, const PivotRoot &q, bool &ok)
{
    const int hi = __double2hiint(a), lo = __double2loint(a);
    const double z = a * q.y0;
    double v = fma(fma(-z, q.l, a), q.y0, z);
    v = fma(fma(-v, q.l, a), q.y, v);
    const bool zero = ((SIGN ? hi & 0x7fffffff : hi) | lo) == 0;
    ok = ok && ((unsigned)((hi & 0x7fffffff) - 0x0df00000) < 0x64100000u || zero);
    return SIGN && zero ? a : v;
}

__device__ __forceinline__ void tri_cp8(double *dst, const double *src)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
}
__device__ __forceinline__ void tri_cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ int tri_at(int p, int q)  // the place of the pair of window indices p, q
{
    return tri_row(max(p, q)) + min(p, q);
}
__device__ __forceinline__ void tri_row8(const double *row, double (&v)[8])
{
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const double2 d = *reinterpret_cast<const double2 *>(row + k);
        v[k] = d.x, v[k + 1] = d.y;
    }
}
__device__ __forceinline__ void tri_put8(double *row, const double (&v)[8])
{
#pragma unroll
    for (int k = 0; k < 8; k += 2) *reinterpret_cast<double2 *>(row + k) = make_double2(v[k], v[k + 1]);
}

// One lane's share of a block by plain roots and divisions: the diagonal block's rows (in: their values, out: L) and its
// own row r. The column of the first pivot that is not positive, or 8; *value that pivot.
static __device__ __noinline__ int tri_plain(const double *in, int pitch, int nc, int b, int r, bool rhs_row, const double *row_in,
                                             double *diag, double *row, double *value)
{
    for (int i = 0; i < 8; i++)
        for (int j = 0; j <= i; j++) diag[8 * i + j] = in[i * pitch + j];
    for (int j = 0; j < 8; j++) row[j] = row_in[j];
    const int c0 = rhs_row ? 0 : max(0, r - b);
    for (int c = 0; c < nc; c++) {
        const double p = diag[9 * c];
        if (!(p > 0) || isnan(p)) {
            *value = p;
            return c;
        }
        const double l = sqrt(p);
        diag[9 * c] = l;
        for (int i = c + 1; i < 8 && i - c <= b; i++) diag[8 * i + c] = diag[8 * i + c] / l;
        if (c >= c0) row[c] = row[c] / l;
        for (int j = c + 1; j < 8 && j - c <= b; j++) {
            for (int i = j; i < 8 && i - c <= b; i++) diag[8 * i + j] = diag[8 * i + j] - diag[8 * i + c] * diag[8 * j + c];
            if (c >= c0) row[j] = row[j] - row[c] * diag[8 * j + c];
        }
    }
    return 8;
}

// A warp's share of a block (in nb, out l): the diagonal block, along in every lane, and the lane's row rr. MASK: rows whose
// first columns (before c0) lie outside the band. Returns whether every value is what sqrt() and / would give.
template <bool MASK>
__device__ __forceinline__ bool tri_factor(const double *nb, double *l, int rr, int c0, int lane, bool first)
{
    double d[8][8], u[8], mine = 1.0;
    PivotRoot keep = {1.0, 1.0, 1.0};
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) d[i][j] = nb[i * kTriPitch + j];
    tri_row8(nb + rr * kTriPitch, u);
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const PivotRoot q = pivot_root(d[c][c]);
        if (lane == c) {
            mine = d[c][c];
            keep = q;
        }
        d[c][c] = q.l;
#pragma unroll
        for (int i = c + 1; i < 8; i++) {
            d[i][c] = quotient<false>(d[i][c], q, ok);
#pragma unroll
            for (int j = c + 1; j <= i; j++) d[i][j] = d[i][j] - d[i][c] * d[j][c];
        }
        const double v = quotient<true>(u[c], q, ok);
        u[c] = !MASK || c >= c0 ? v : u[c];
#pragma unroll
        for (int j = c + 1; j < 8; j++) {
            const double s = u[j] - u[c] * d[j][c];
            u[j] = !MASK || c >= c0 ? s : u[j];
        }
    }
    if (lane < 8) ok = ok && pivot_ok(mine, keep);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
        tri_put8(l + rr * kTriPitch, u);
        if (first && lane == 0) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j <= i; j++) l[i * kTriPitch + j] = d[i][j];
        }
    }
    return ok;
}

// err_row[0] = -1 on success, else the first row whose pivot was not positive; pivot[0] that pivot.
static __global__ void __launch_bounds__(kTriThreads, 1) k_band_tri(int n, int b, double *__restrict__ a, double *__restrict__ rhs,
                                                                    int32_t *err_row, double *pivot)
{
    extern __shared__ __align__(16) unsigned char band_smem[];
    __shared__ int s_bad;   // a failed pivot's row
    __shared__ int s_tile;  // the next tile of the update in progress
    __shared__ double xs[kBackRows];
    const int w = b + 1, W = b + 16, R = b + 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    double *win = (double *)band_smem;                                    // packed window
    double *nb = win + (tri_row(W) + 1) / 2 * 2;                          // the block to factor: rows 0 .. R - 1, right-hand side
    double *pb = nb + (R + 1) * kTriPitch;                                // two factored blocks of the same form
    double *rv = pb + 2 * (R + 1) * kTriPitch;                            // right-hand side, by window index
    const int nrw = (max(b - 6, 1) + 31) / 32 + 1, nwork = kTriThreads / 32 - nrw;  // warps that factor, the others
    auto wrap = [&](int p) { return p >= W ? p - W : p; };

    // rows [i0, i1) of the band, the first at window index p0, into the window
    auto fetch = [&](int i0, int i1, int p0, int t, int nt) {
        i1 = min(i1, n);
        for (int i = i0 + t / 32; i < i1; i += nt / 32) {
            const int pi = wrap(p0 + i - i0), ps = wrap(pi + 16);  // i - b = i + 16 - W
            const double *g = a + (size_t)i * w;
            for (int c = max(t & 31, ((b - i + 31) & ~31) + (t & 31) - 32); c < w; c += 32)
                if (i - b + c >= 0) tri_cp8(win + tri_at(pi, wrap(ps + c)), g + c);
        }
        if (rhs)
            for (int i = i0 + t; i < i1; i += nt) tri_cp8(rv + wrap(p0 + i - i0), rhs + i);
    };
    // the block that starts at k0 (window index p0) into nb, less the products of the block `l` before it (null: none)
    auto stage = [&](int k0, int p0, const double *l) {
        double *o = nb;
        for (int t = tid; t < 2 * R; t += kTriThreads) {  // two threads a row, four columns each
            const int r = t < R ? t : t - R, cb = t < R ? 0 : 4, i = k0 + r, pi = wrap(p0 + r);
            double li[8];
            const bool upd = l && r + 8 < R && i < n;  // the rows that the block before reaches
            if (upd) tri_row8(l + (r + 8) * kTriPitch, li);
            const int ks = max(0, r + 8 - b);  // the first of its columns in row i's band
            int pj = wrap(p0 + cb), tj = tri_row(pj);
            const int ti = tri_row(pi);
#pragma unroll 1
            for (int cc = cb; cc < cb + 4; cc += 2) {
                double v[2];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    v[c] = r >= cc + c && r - cc - c <= b && i < n ? win[pj <= pi ? ti + pj : tj + pi] : 0.0;
                    tj += ((pj + 15) & ~15) + 1;
                    if (++pj == W) pj = tj = 0;
                }
                if (upd) {  // (what comes of entries above the diagonal is never used)
                    double lj[2][8];
#pragma unroll
                    for (int c = 0; c < 2; c++) tri_row8(l + min(cc + c + 8, R) * kTriPitch, lj[c]);  // (past R: unused, r < b)
                    if (ks == 0) {
#pragma unroll
                        for (int k = 0; k < 8; k++)
#pragma unroll
                            for (int c = 0; c < 2; c++) v[c] = v[c] - li[k] * lj[c][k];
                    } else {
#pragma unroll
                        for (int k = 1; k < 8; k++)
#pragma unroll
                            for (int c = 0; c < 2; c++) {
                                const double s = v[c] - li[k] * lj[c][k];
                                v[c] = k >= ks ? s : v[c];
                            }
                    }
                }
                *reinterpret_cast<double2 *>(o + r * kTriPitch + cc) = make_double2(v[0], v[1]);
            }
        }
        if (tid >= kTriThreads - 8) {  // the block's right-hand side
            const int r = tid - (kTriThreads - 8);
            double v = 0.0;
            if (rhs && k0 + r < n) {
                v = rv[wrap(p0 + r)];
                if (l && r + 8 < R) {
                    double lr[8], y[8];
                    tri_row8(l + (r + 8) * kTriPitch, lr);
                    tri_row8(l + R * kTriPitch, y);
                    const int ks = max(0, r + 8 - b);
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const double s = v - lr[k] * y[k];
                        v = k >= ks ? s : v;
                    }
                }
            }
            o[R * kTriPitch + r] = v;
        }
    };
    // the block at k0, factored in l: its rows of L and its solution entries to global memory
    auto retire = [&](int k0, const double *l, int t, int nt) {
        const int nc = min(8, n - k0), rows = min(R, n - k0);
        double *g = a + (size_t)k0 * w + b;  // entry (k0 + r, k0 + c): g[r * b + c]
        for (int q = t; q < 8 * rows; q += nt) {
            const int r = q >> 3, c = q & 7;
            if (c < nc && r >= c && r - c <= b) g[r * b + c] = l[r * kTriPitch + c];
        }
        if (rhs && t < nc) rhs[k0 + t] = l[R * kTriPitch + t];
    };

    if (tid == 0) {
        s_bad = -1;
        s_tile = 0;
        *pivot = 0.0;
    }
    fetch(0, W, 0, tid, kTriThreads);
    tri_cp_wait();
    __syncthreads();
    stage(0, 0, nullptr);
    __syncthreads();

    for (int k0 = 0, p0 = 0, J = 0;; k0 += 8, J++) {
        double *l = pb + (J & 1) * (R + 1) * kTriPitch, *lo = pb + (1 - (J & 1)) * (R + 1) * kTriPitch;
        if (warp < nrw) {
            // A: rows 8 .. b and the right-hand side, a row a lane; the last of these warps the seven rows that lack the
            // block's first columns
            const bool tail = warp == nrw - 1;
            const int q = 32 * warp + lane, rr = tail ? b + 1 + min(lane, 6) : 8 + q <= b ? 8 + q : R;
            const int c0 = tail ? rr - b : 0, nc = min(8, n - k0);
            // (bands narrower than the block, and the last block, go the plain way)
            bool ok = nc == 8 && b >= 7;
            if (ok) ok = tail ? tri_factor<true>(nb, l, rr, c0, lane, false) : tri_factor<false>(nb, l, rr, 0, lane, warp == 0);
            if (!ok) {
                double pd[64], pu[8], value = 0.0;
                const int rp = rr < 8 ? 8 : rr;  // (rows below 8 of a narrow band belong to the diagonal block)
                const int bad = tri_plain(nb, kTriPitch, nc, b, rp, rp == R, nb + rp * kTriPitch, pd, pu, &value);
                if (bad < 8 && tid == 0) {
                    s_bad = k0 + bad;
                    *pivot = value;
                }
                for (int k = 0; k < 8; k++) l[rp * kTriPitch + k] = pu[k];
                if (tid < 8)
                    for (int k = 0; k < 8; k++) l[tid * kTriPitch + k] = k <= tid ? pd[8 * tid + k] : 0.0;
            }
        } else if (J > 0) {
            const int t = tid - 32 * nrw, nt = 32 * nwork;
            fetch(k0 + 8 + b, k0 + 16 + b, wrap(p0 + 8 + b), t, nt);
            const int q0 = k0 - 8, last = min(R, n - q0);
            const int pq = wrap(p0 + W - 8);  // window index of q0
            // the last seven rows lack the block's first columns: a column a lane
            for (int c = 16 + t; c < min(last, b + 8); c += nt) {
                double lj[8];
                tri_row8(lo + c * kTriPitch, lj);
                const int pj = wrap(pq + c), tj = tri_row(pj);
#pragma unroll 1
                for (int m = 0; m < 7; m++) {
                    const int r = b + 1 + m;
                    if (r >= last || r < c || r < 16) continue;
                    const int pi = wrap(pq + r);
                    double &e = win[pj <= pi ? tri_row(pi) + pj : tj + pi];
                    double v = e;
#pragma unroll
                    for (int k = 1; k < 8; k++)
                        if (k > m) v = v - lo[r * kTriPitch + k] * lj[k];
                    e = v;
                }
            }
            if (rhs) {
                double y[8], row[8];
                tri_row8(lo + R * kTriPitch, y);
                for (int r = 16 + t; r < last; r += nt) {
                    tri_row8(lo + r * kTriPitch, row);
                    double &e = rv[wrap(pq + r)];
                    double s = e;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const double v = s - row[k] * y[k];
                        s = k >= r - b ? v : s;
                    }
                    e = s;
                }
            }
            retire(q0, lo, t, nt);
        }
        if (J > 0) {
            // the block before this one: rows and columns from k0 + 8 on (16 .. R - 1 of its own). Rows up to b have all
            // eight of its columns in their band: 32 x 16 tiles, drawn by whichever warp is free, a lane four rows by
            // four columns of one (rows lr + 8 u, columns from lc on, so that a half-warp's accesses lie on distinct banks)
            const int q0 = k0 - 8, last = min(R, n - q0), whole = min(last, b + 1);
            const int pq = wrap(p0 + W - 8);  // window index of q0
            const int lr = lane & 7, lc = 8 * (lane >> 3 & 1) + 4 * (lane >> 4);
            for (;;) {
                int tile = 0;
                if (lane == 0) tile = atomicAdd(&s_tile, 1);
                tile = __shfl_sync(FULL, tile, 0);
                int rb = 16, re = 0;
                for (; rb < whole; rb += 32) {
                    re = min(whole, rb + 32);
                    const int nct = (re - 1) >> 4;
                    if (tile < nct) break;
                    tile -= nct;
                }
                if (rb >= whole) break;
                const int cb = 16 + 16 * tile + lc;
                double li[4][8];
                int ti[4], pi[4], lim[4];  // lim: the last column of a row to store
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int r = min(rb + lr + 8 * u, re - 1);
                    tri_row8(lo + r * kTriPitch, li[u]);
                    pi[u] = wrap(pq + r);
                    ti[u] = tri_row(pi[u]);
                    lim[u] = rb + lr + 8 * u < re ? r : 0;
                }
                int pj = wrap(wrap(pq + min(cb, re))), tj = tri_row(pj);
#pragma unroll 1
                for (int c = cb; c < min(cb + 4, re); c++) {
                    double v[4], lj[8];
                    int at[4];
                    tri_row8(lo + c * kTriPitch, lj);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        at[u] = pj <= pi[u] ? ti[u] + pj : tj + pi[u];
                        v[u] = win[at[u]];
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++)
#pragma unroll
                        for (int u = 0; u < 4; u++) v[u] = v[u] - li[u][k] * lj[k];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (c <= lim[u]) win[at[u]] = v[u];
                    tj += ((pj + 15) & ~15) + 1;
                    if (++pj == W) pj = tj = 0;
                }
            }
            tri_cp_wait();
        }
        __syncthreads();
        if (s_bad >= 0) {
            if (tid == 0) *err_row = s_bad;
            return;
        }
        if (k0 + 8 >= n) {
            retire(k0, l, tid, kTriThreads);
            break;
        }
        // B: the next block
        if (tid == 0) s_tile = 0;
        p0 = wrap(p0 + 8);
        stage(k0 + 8, p0, l);
        __syncthreads();
    }
    if (tid == 0) *err_row = -1;
    if (!rhs) return;
    __syncthreads();

    // backward substitution, blocks of 32 rows from the bottom: warp 0 solves a block's triangle while the others fetch the
    // rows of the next one; then all threads subtract the block from the b rows above it (products in descending row)
    const int ws = w | 1, XW = b + 4 * kBackRows;
    double *br = (double *)band_smem, *xv = br + 2 * kBackRows * ws;
    auto fetch_rows = [&](int i0, int i1, int buf, int t, int nt) {
        for (int i = i0 + t / 32; i < i1; i += nt / 32)
            for (int c = t & 31; c < w; c += 32)
                if (i - b + c >= 0) tri_cp8(br + ((size_t)buf * kBackRows + (i - i0)) * ws + c, a + (size_t)i * w + c);
    };
    auto fetch_x = [&](int i0, int i1, int t, int nt) {
        for (int i = max(i0, 0) + t; i < i1; i += nt) tri_cp8(xv + i % XW, rhs + i);
    };
    {
        const int i0 = max(0, n - kBackRows);
        fetch_rows(i0, n, 0, tid, kTriThreads);
        fetch_x(i0 - b, n, tid, kTriThreads);
        tri_cp_wait();
        __syncthreads();
    }
    for (int i1 = n, buf = 0; i1 > 0; buf ^= 1) {
        const int i0 = max(0, i1 - kBackRows), np = i1 - i0;
        const double *rows = br + (size_t)buf * kBackRows * ws;
        if (warp == 0) {
            double y0 = 0.0;
            PivotRoot pr;
            pr.l = 1.0;
            if (lane < np) {
                y0 = xv[(i0 + lane) % XW];
                pr.l = rows[lane * ws + b];
            }
            // the diagonal's reciprocal is correctly rounded: quotient() is, too
            pr.y0 = pr.y = 1.0 / pr.l;
            bool ok = pr.l > 1e-15 && pr.l < 1e15 && !significand(pr.l, 0xfffff, -1);
            double y = y0;
#pragma unroll 1
            for (int k0 = (np - 1) / 8 * 8; k0 >= 0; k0 -= 8) {
                double e[8];  // L(i0 + k0 + u, i0 + lane)
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int kk = k0 + u;
                    e[u] = kk < np && lane < kk && kk - lane <= b ? rows[kk * ws + lane - kk + b] : 0.0;
                }
#pragma unroll
                for (int u = 7; u >= 0; u--) {
                    const int kk = k0 + u;
                    bool good = true;
                    const double q = quotient<true>(y, pr, good);
                    ok = ok && (good || lane != kk);
                    const double x = __shfl_sync(FULL, q, kk), t = e[u] * x;
                    if (lane == kk) y = x;
                    if (kk < np && lane < kk && kk - lane <= b) y = y - t;
                }
            }
            if (__any_sync(FULL, !ok)) {
                y = y0;
                for (int kk = np - 1; kk >= 0; kk--) {
                    const double x = __shfl_sync(FULL, y / pr.l, kk);
                    if (lane == kk) y = x;
                    if (lane < kk && kk - lane <= b) y = y - rows[kk * ws + lane - kk + b] * x;
                }
            }
            if (lane < np) {
                xs[lane] = y;
                rhs[i0 + lane] = y;
            }
        } else {
            const int j0 = max(0, i0 - kBackRows);
            fetch_rows(j0, i0, buf ^ 1, tid - 32, kTriWorkers);
            fetch_x(j0 - b, i0 - b, tid - 32, kTriWorkers);
            tri_cp_wait();
        }
        __syncthreads();
        for (int k = max(0, i0 - b) + tid; k < i0; k += kTriThreads) {
            double v = xv[k % XW];
            const double *col = rows + k - i0 + b;  // row i0 + u: col[u * (ws - 1)]
            const int top = min(np - 1, k + b - i0);
            if (top == kBackRows - 1) {
#pragma unroll 8
                for (int u = kBackRows - 1; u >= 0; u--) v = v - col[u * (ws - 1)] * xs[u];
            } else {
                for (int u = top; u >= 0; u--) v = v - col[u * (ws - 1)] * xs[u];
            }
            xv[k % XW] = v;
        }
        __syncthreads();
        i1 = i0;
    }
}

}  // namespace band
}  // namespace ifea
