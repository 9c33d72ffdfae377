// sweep.cuh — the forward and backward sweeps of the multifrontal solve as ONE persistent kernel.
//
// A solve reads the whole factor twice and computes almost nothing, along the elimination tree: up (each front's
// right-hand side is what its children leave over), then down. Launched level by level it was bound by the level
// barriers (60 dependent launches on the closed-die factor, most of them too small to fill the chip). Here the
// sweeps are a list of tile tasks in an order in which every task comes after those it needs; CTAs draw tasks by an
// atomic ticket, and a task waits for its inputs on per-front completion counters, so subtrees overlap freely and
// only the path to the root is serial. A CTA is eight computing warps and a scheduling warp that runs one task
// ahead: it draws the next ticket, asks L2 for that task's part of the factor (bulk prefetch) and polls its
// counters while the current task is computed; the computing warps issue a task's first factor loads before its
// inputs are complete. (Streaming the factor through a shared-memory ring by bulk copies measured slower: a stage's
// hand-over costs a CTA about half a microsecond, which plain loads of 24 or more warps hide.)
//
// Progress needs no co-residency: tickets are drawn in list order by running CTAs, so the lowest unfinished task
// always has its inputs complete. Every wait is bounded all the same (two seconds unless the host sets another limit);
// one that gives up sets a sticky error word, every CTA leaves, and what was not computed of the solution is NaN (tasks
// still at work may store their part of it). The host clears the word with the counters when it reads it. Counters
// are monotonic over the solves of an analysis (targets scale with the solve's number), so nothing is cleared between
// solves. Every sum has a fixed order: solves are bit-reproducible.
//
// What bounds it: the bytes of the factor on the large levels (3.3 TB/s over a whole solve of 308 M FP32 entries),
// the chain of dependent phases towards the root on small factors (two going up and two coming down per level, each
// about 2.2 us: a counter seen 0.5 us after it was raised, the operand vector from L2, the dot products, the release).
// Device time of one solve, launched level by level before / as one kernel now (B200, upsetting billets):
//   206k tets FP32 1.02 / 0.75 ms; 104k tets FP64 0.84 / 0.53; 62k tets FP32 0.42 / 0.27; 33k tets FP64 0.45 / 0.23;
//   5.6k tets FP64 0.141 / 0.092; 2.3k tets FP64 0.103 / 0.066.
#pragma once

namespace ifea {
namespace mf {

enum SweepKind : int32_t {
    kSwEnd = -1,
    kSwFS = 0,  // small front, forward: whole front
    kSwFA = 1,  // wide front: rows [r0, r1) of the assembled right-hand side (fronts of many y tiles only)
    kSwFY = 2,  // wide front: rows [r0, r1) of y1 = X acc1 (flag 1: acc1 gathered here, not read from kSwFA's)
    kSwFT = 3,  // wide front: rows [r0, r1) of the update vector, L21 y1 - acc2
    kSwBZ = 4,  // wide front: entries [r0, r1) of z = y1 - L21^T x2
    kSwBS = 5,  // small front, backward: whole front
    kSwBX = 6   // wide front: entries [r0, r1) of x1 = X^T z
};

// Everything a task needs to address its data, so that nothing is looked up once its inputs are complete.
struct __align__(16) SweepTask {
    int32_t kind, flag, r0, r1;
    int32_t wait, target;  // counter and its value per solve (wait < 0: none)
    int32_t done;          // counter to raise (< 0: none)
    int32_t is;            // first entry in the per-row arrays
    int32_t nc, ms, c0;    // pivots, rows, first pivot (new numbering)
    int64_t off;             // the front (small fronts, kSwFT, kSwBZ) or its pivot-block inverse (kSwFY, kSwBX)
    int64_t aux;             // the update vector (kSwFT, kSwFS); the panel inverses (kSwBS)
    int64_t inv;             // the panel inverses (kSwFS)
};
static_assert(sizeof(SweepTask) % 16 == 0, "tasks are read 16 bytes at a time");

constexpr int kSwCtas = 4;                    // CTAs per SM (three or two measured the same or slower)
constexpr int kSwWarps = 8;                   // computing warps
constexpr int kSwCompute = 32 * kSwWarps;     // 256
constexpr int kSwThreads = kSwCompute + 32;   // + the scheduling warp
constexpr int kSwGather = 1024;               // pivots from which a front's right-hand side is assembled once
constexpr int kSwPre = 4;                     // operand entries per thread whose indices are fetched ahead
// completion counters per front
enum { kCntUpd = 0, kCntA = 1, kCntY = 2, kCntZ = 3, kCntX = 4, kCntN = 5 };

template <typename T>
constexpr int kDotU = sizeof(T) == 4 ? 16 : 8;  // factor loads in flight per lane

// Lanes per row (or column) of a dot product of at most `len` entries.
__host__ __device__ inline int sweep_group(int len) { return len <= 96 ? 8 : len <= 224 ? 16 : 32; }

__device__ __forceinline__ void sweep_bar()  // a barrier of the computing warps
{
    asm volatile("bar.sync 7, %0;" ::"n"(kSwCompute) : "memory");
}
// hand-over between the scheduling warp and the computing warps: one side arrives, the other waits
__device__ __forceinline__ void sweep_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kSwThreads) : "memory"); }
__device__ __forceinline__ void sweep_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kSwThreads) : "memory"); }
enum { kBarDesc = 1, kBarReady = 3, kBarFree = 5 };  // one per task slot

__device__ __forceinline__ float ld_factor(const float *p)
{
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_factor(const double *p)
{
    double v;
    asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes)
{
    // bulk prefetches take 16-byte aligned addresses and sizes; the rounding stays inside the buffer's own granules
    const size_t a = (size_t)p & ~(size_t)15, e = ((size_t)p + (bytes < 131072 ? bytes : 131072) + 15) & ~(size_t)15;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global((void *)a)), "r"((uint32_t)(e - a)) : "memory");
}

// Order of sums. In single precision a dot product is summed as VG lanes of a warp would: VG partial sums of every VG-th
// product, added as a tree of halves (VG / 2 apart, VG / 4, .. 1). VG belongs to the front and the kind of product, not
// to the tile: G lanes (G <= VG, as many as the tile's rows can use) hold VG / G of the partial sums each. So a solve does
// not depend on how the tiles are cut: the single-precision factor is a preconditioner, and what its conjugate
// gradients return within their tolerance follows the last bits of a solve. A double-precision solve is taken as
// it is, and sums by its tile's own lanes (with fixed VG its solves measured 1 to 3 % slower).
template <typename T>
constexpr bool kFixedSums = sizeof(T) == 4;

template <int G, int NA, typename T>
__device__ __forceinline__ T group_sum(T (&p)[NA])
{
#pragma unroll
    for (int h = NA / 2; h > 0; h >>= 1)
#pragma unroll
        for (int k = 0; k < h; k++) p[k] += p[k + h];
    T v = p[0];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Sum of fa(c) fb(c) over c = first - lane .. len - 1 (VG = 32) by eight lanes, `first` being a lane's own first entry. The
// factor entries are loaded U at a time before any is used, so a lane keeps U loads in flight however short the run.
template <int U, typename T, typename FA, typename FB>
__device__ __forceinline__ T dot8(int first, int len, FA fa, FB fb)
{
    T p[4] = {T(0), T(0), T(0), T(0)};
    for (int c0 = first; c0 < len; c0 += 8 * U) {
        T a[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = c0 + 8 * u;
            a[u] = c < len ? fa(c) : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + 8 * u < len) p[u % 4] = fma(a[u], fb(c0 + 8 * u), p[u % 4]);
    }
    return group_sum<8, 4>(p);
}

template <typename T>
struct SweepArgs {
    Dev<T> D;
    const SweepTask *tasks;
    int ntasks;
    uint32_t *cnt;      // kCntN per front
    uint32_t *ticket;   // the next task, zero between solves; then the solves since the counters were cleared
    const int32_t *skip;  // nothing to do when *skip (null: never)
    const int32_t *perm;
    const int2 *pair;   // per front row: the children's update entries that land on it (see sweep_pairs)
    const double *b;
    double *x;
    T *A1, *Y, *Z, *X;  // assembled right-hand sides (per front row); y, z and x in the new numbering
    int *err;
    uint64_t wait_ns;   // a wait's limit; zero: a counter is looked at once
    int n;
};

// v minus the children's contributions to a front row, in child order. q.x, q.y: the first and the only other
// update entry (-1: none); q.y < -1: two or more others, listed at gat_src[-2 - q.y ...] after their number.
template <typename T>
__device__ __forceinline__ T sweep_gather(const Dev<T> &D, int2 q, T v)
{
    if (q.x >= 0) v -= __ldcg(D.U + q.x);
    if (q.y >= 0) v -= __ldcg(D.U + q.y);
    if (q.y < -1) {
        const int32_t *l = D.gat_src + (-2 - q.y);
        for (int k = 1, n = __ldg(l); k <= n; k++) v -= __ldcg(D.U + __ldg(l + k));
    }
    return v;
}

// Entries [k0, k1) of the operand vector into shared memory, eight loads of a thread in flight.
template <typename T, typename FFetch>
__device__ __forceinline__ void sweep_stage(T *vs, int k0, int k1, FFetch fetch)
{
    for (int k = k0 + threadIdx.x; k < k1; k += 8 * kSwCompute) {
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = k + u * kSwCompute < k1 ? fetch(k + u * kSwCompute) : T(0);
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (k + u * kSwCompute < k1) vs[k + u * kSwCompute - k0] = v[u];
    }
}

// A tile: rows (or columns) [r0, r1) of the factor against an operand vector over [v0, v1) (in vs[] from v0 on). Row r holds
// base[r * ld + c] for c in [v0, v1), but in [r, v1) for X's columns and in [0, r + 1) for its rows. Its sum has VG
// partial sums (see above), vg of them; G lanes a row.
template <typename T, int KIND>
struct SweepRows {
    const T *base;
    int64_t ld;
    int r0, r1, v0, v1, vg;
    __device__ __forceinline__ int start(int r) const { return KIND == kSwBX ? r : v0; }
    __device__ __forceinline__ int length(int r) const
    {
        return r >= r1 ? 0 : KIND == kSwBX ? v1 - r : KIND == kSwFY ? r + 1 : v1 - v0;
    }
    // one lane's share of a batch of a row's entries: c, c + G, ... from the row's start
    template <int G>
    __device__ __forceinline__ void load(T (&a)[kDotU<T>], int r, int c) const
    {
        const T *p = base + (int64_t)r * ld + start(r) + c;
        const int n = length(r);
#pragma unroll
        for (int u = 0; u < kDotU<T>; u++) a[u] = c + G * u < n ? ld_factor(p + G * u) : T(0);
    }
    template <int G>
    __device__ __forceinline__ void first(T (&a)[kDotU<T>]) const
    {
        const int lane = threadIdx.x & 31;
        load<G>(a, r0 + (threadIdx.x >> 5) * (32 / G) + lane / G, lane % G);
    }
    // every row's dot product; a[] holds the first batch already
    template <int G, int NA, typename FOut>
    __device__ __forceinline__ void dots(T (&a)[kDotU<T>], const T *vs, FOut out) const
    {
        constexpr int U = kDotU<T>, RP = 32 / G;
        const int lane = threadIdx.x & 31;
        for (int w0 = r0 + (threadIdx.x >> 5) * RP; w0 < r1; w0 += kSwWarps * RP) {
            const int r = w0 + lane / G, n = length(r);
            if (w0 >= r0 + kSwWarps * RP) load<G>(a, r, lane % G);
            T p[NA];
#pragma unroll
            for (int k = 0; k < NA; k++) p[k] = T(0);
            for (int c = lane % G;;) {
                const T *x = vs + (start(r) - v0) + c;
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (c + G * u < n) p[u % NA] = fma(a[u], x[G * u], p[u % NA]);
                c += G * U;
                if (c - lane % G >= n) break;
                load<G>(a, r, c);
            }
            const T v = group_sum<G, NA>(p);
            if (r < r1 && lane % G == 0) out(r, v);
        }
    }
    // ready() returns once the task's inputs are complete and the operand vector is in place (false: leave); the
    // first factor loads are in flight before that
    template <typename FReady, typename FOut>
    __device__ __forceinline__ bool run(const T *vs, FReady ready, FOut out) const
    {
        T a[kDotU<T>];
        const int g = sweep_group(v1 - v0);
        if (g == 8) first<8>(a);
        else if (g == 16) first<16>(a);
        else first<32>(a);
        if (!ready()) return false;
        const int na = vg / g;
        if constexpr (kFixedSums<T>) {
            if (g == 16 && na == 2) return dots<16, 2>(a, vs, out), true;
            if (g == 8 && na == 2) return dots<8, 2>(a, vs, out), true;
            if (g == 8 && na == 4) return dots<8, 4>(a, vs, out), true;
        }
        if (g == 32) dots<32, 1>(a, vs, out);
        else if (g == 16) dots<16, 1>(a, vs, out);
        else dots<8, 1>(a, vs, out);
        return true;
    }
};

// A small front's forward elimination by one CTA. Each 64-pivot block is applied through its stored inverse.
template <typename T, typename FWait>
__device__ __forceinline__ bool sweep_small_fwd(const SweepArgs<T> &A, const SweepTask &t, T *acc, T *part, T *yb, FWait wait)
{
    const Dev<T> &D = A.D;
    const int ms = t.ms, nc = t.nc, c0 = t.c0, tid = threadIdx.x;
    const T *F = D.F + t.off, *Inv = D.Inv + t.inv;
    {
        int2 q = make_int2(-1, -1);
        T b = T(0);
        if (tid < ms) q = __ldg(A.pair + t.is + tid);
        if (tid < nc) b = (T)A.b[__ldg(A.perm + c0 + tid)];
        if (!wait()) return false;
        if (tid < ms) acc[tid] = sweep_gather(D, q, b);
        for (int k = tid + kSwCompute; k < ms; k += kSwCompute)
            acc[k] = sweep_gather(D, __ldg(A.pair + t.is + k), k < nc ? (T)A.b[A.perm[c0 + k]] : T(0));
    }
    sweep_bar();
    for (int kb = 0; kb < nc; kb += PW) {
        const int w = min(PW, nc - kb);
        const T *I = Inv + (int64_t)(kb / PW) * PW * PW;
        {
            // y_blk = Linv acc_blk (VG = 32): four threads per row, every fourth column each (the upper part is
            // stored as zeros)
            const int i = tid & 63, g = tid >> 6;
            T f[16], p[8];
#pragma unroll
            for (int u = 0; u < 16; u++) f[u] = (i < w && g + 4 * u < w) ? ld_factor(I + (g + 4 * u) * PW + i) : T(0);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                p[u] = g + 4 * u < w ? f[u] * acc[kb + g + 4 * u] : T(0);
                if (g + 4 * u + 32 < w) p[u] = fma(f[u + 8], acc[kb + g + 4 * u + 32], p[u]);
            }
#pragma unroll
            for (int h = 4; h > 0; h >>= 1)
#pragma unroll
                for (int k = 0; k < h; k++) p[k] += p[k + h];
            part[tid] = p[0];
        }
        sweep_bar();
        if (tid < w) {
            const T v = (part[tid] + part[128 + tid]) + (part[64 + tid] + part[192 + tid]);
            yb[tid] = v;
            A.Y[c0 + kb + tid] = v;
        }
        sweep_bar();
        // rows below the block (in double precision two threads a row when one pass covers them)
        const int rb = kb + w, nrow = ms - rb, H = !kFixedSums<T> && nrow <= 128 ? 2 : 1, per = kSwCompute / H, h = tid / per;
        const int k0 = h * (PW / H), k1 = min(w, k0 + PW / H);
        for (int r = tid % per; r < nrow; r += per) {
            T v = H == 1 ? acc[rb + r] : T(0);
            const T *col = F + (int64_t)kb * ms + rb + r;
            for (int k = k0; k < k1; k += 16) {
                T f[16];
#pragma unroll
                for (int u = 0; u < 16; u++) f[u] = k + u < k1 ? ld_factor(col + (int64_t)(k + u) * ms) : T(0);
#pragma unroll
                for (int u = 0; u < 16; u++)
                    if (k + u < k1) v = fma(-f[u], yb[k + u], v);
            }
            if (H == 1) acc[rb + r] = v;
            else part[tid] = v;
        }
        sweep_bar();
        if (H == 2) {
            if (tid < nrow) acc[rb + tid] += part[tid] + part[128 + tid];
            sweep_bar();
        }
    }
    T *u = D.U + t.aux;
    for (int i = tid; i < ms - nc; i += kSwCompute) u[i] = -acc[nc + i];
    return true;
}

// A small front's back substitution by one CTA, eight lanes a column.
template <typename T, typename FWait>
__device__ __forceinline__ bool sweep_small_bwd(const SweepArgs<T> &A, const SweepTask &t, T *sm, T *xb, FWait wait)
{
    const Dev<T> &D = A.D;
    const int ms = t.ms, nc = t.nc, c0 = t.c0, nr = ms - nc;
    const T *F = D.F + t.off, *Inv = D.Inv + t.aux;
    const int32_t *ix = D.idx + t.is + nc;
    T *acc = sm, *xs = sm + nc;
    const int tid = threadIdx.x, lane = tid & 31, gl = lane & 7, grp = tid >> 3, ng = kSwCompute / 8;
    const int i0 = tid < nr ? __ldg(ix + tid) : 0;
    if (!wait()) return false;
    if (tid < nr) xs[tid] = __ldcg(A.X + i0);
    for (int i = tid + kSwCompute; i < nr; i += kSwCompute) xs[i] = __ldcg(A.X + __ldg(ix + i));
    for (int k = tid; k < nc; k += kSwCompute) acc[k] = __ldcg(A.Y + c0 + k);
    sweep_bar();
    for (int k0 = 0; k0 < nc; k0 += ng) {
        const int k = k0 + grp;
        const bool ok = k < nc;
        const T *col = F + (int64_t)(ok ? k : 0) * ms + nc;
        const T v = dot8<kDotU<T>, T>(gl, ok ? nr : 0, [&](int i) { return ld_factor(col + i); }, [&](int i) { return xs[i]; });
        if (ok && gl == 0) acc[k] -= v;
    }
    sweep_bar();
    for (int bi = (nc + PW - 1) / PW - 1; bi >= 0; bi--) {
        const int kb = bi * PW, w = min(PW, nc - kb), ke = kb + w;
        if (ke < nc) {
            for (int j0 = kb; j0 < ke; j0 += ng) {
                const int j = j0 + grp;
                const bool ok = j < ke;
                const T *col = F + (int64_t)(ok ? j : 0) * ms;
                const T v = dot8<kDotU<T>, T>(ke + gl, ok ? nc : 0, [&](int k) { return ld_factor(col + k); }, [&](int k) { return acc[k]; });
                if (ok && gl == 0) acc[j] -= v;
            }
            sweep_bar();
        }
        // x_blk = Linv^T acc_blk: x_j = sum_{i >= j} Linv[i][j] acc_i (column j of the inverse is contiguous)
        const T *I = Inv + (int64_t)bi * PW * PW;
        for (int j0 = 0; j0 < w; j0 += ng) {
            const int j = j0 + grp;
            const bool ok = j < w;
            const T v = dot8<8, T>((ok ? j : w) + gl, w, [&](int i) { return ld_factor(I + j * PW + i); }, [&](int i) { return acc[kb + i]; });
            if (ok && gl == 0) xb[j] = v;
        }
        sweep_bar();
        for (int j = tid; j < w; j += kSwCompute) acc[kb + j] = xb[j];
        sweep_bar();
    }
    for (int k = tid; k < nc; k += kSwCompute) {
        A.X[c0 + k] = acc[k];
        A.x[A.perm[c0 + k]] = (double)acc[k];
    }
    return true;
}

// One task by the computing warps: wait() returns when the task's inputs are complete (false: the solve is being
// abandoned); what does not depend on them (indices, right-hand side, the first factor loads) is fetched before.
// sa: the rows' own starting values (at most one row per thread in a tile).
template <typename T, typename FWait>
__device__ __forceinline__ bool sweep_task(const SweepArgs<T> &A, const SweepTask &t, T *vs, T *sa, T *yb, FWait wait)
{
    const Dev<T> &D = A.D;
    const int r0 = t.r0, r1 = t.r1, tid = threadIdx.x, nc = t.nc, ms = t.ms, c0 = t.c0;
    switch (t.kind) {
    case kSwFS: return sweep_small_fwd(A, t, vs, sa, yb, wait);
    case kSwBS: return sweep_small_bwd(A, t, vs, yb, wait);
    case kSwFA: {
        // two rows a thread
        const int k0 = r0 + tid, k1 = k0 + kSwCompute;
        int2 q0 = make_int2(-1, -1), q1 = q0;
        T b0 = T(0), b1 = T(0);
        if (k0 < r1) q0 = __ldg(A.pair + t.is + k0), b0 = (T)A.b[__ldg(A.perm + c0 + k0)];
        if (k1 < r1) q1 = __ldg(A.pair + t.is + k1), b1 = (T)A.b[__ldg(A.perm + c0 + k1)];
        if (!wait()) return false;
        if (k0 < r1) A.A1[t.is + k0] = sweep_gather(D, q0, b0);
        if (k1 < r1) A.A1[t.is + k1] = sweep_gather(D, q1, b1);
        return true;
    }
    case kSwFY: {
        // row r of X (read through its mirror: contiguous) against acc1
        const SweepRows<T, kSwFY> w = {D.Xinv + t.off, nc, r0, r1, 0, r1, sweep_group(nc)};
        int2 q[kSwPre];
        T b[kSwPre];
        if (t.flag)
#pragma unroll
            for (int u = 0; u < kSwPre; u++) {
                const int k = tid + u * kSwCompute;
                q[u] = k < r1 ? __ldg(A.pair + t.is + k) : make_int2(-1, -1);
                b[u] = k < r1 ? (T)A.b[__ldg(A.perm + c0 + k)] : T(0);
            }
        return w.run(
            vs,
            [&] {
                if (!wait()) return false;
                if (t.flag) {  // (at most kSwGather = kSwPre * kSwCompute pivots)
#pragma unroll
                    for (int u = 0; u < kSwPre; u++)
                        if (tid + u * kSwCompute < r1) vs[tid + u * kSwCompute] = sweep_gather(D, q[u], b[u]);
                } else {
                    sweep_stage(vs, 0, r1, [&](int k) { return __ldcg(A.A1 + t.is + k); });
                }
                sweep_bar();
                return true;
            },
            [&](int r, T v) {
                A.Y[c0 + r] = v;
                if (ms == nc) A.Z[c0 + r] = v;  // a root has nothing below: z = y1
            });
    }
    case kSwFT: {
        // row i of L21 (its mirror in the front's upper right block: contiguous) against y1
        const SweepRows<T, kSwFT> w = {D.F + t.off + (int64_t)nc * ms, ms, r0, r1, 0, nc, sweep_group(nc)};
        const bool own = tid < r1 - r0;
        const int2 q = own ? __ldg(A.pair + t.is + nc + r0 + tid) : make_int2(-1, -1);
        T *u = D.U + t.aux;
        return w.run(
            vs,
            [&] {
                if (!wait()) return false;
                if (own) sa[tid] = sweep_gather(D, q, T(0));
                sweep_stage(vs, 0, nc, [&](int k) { return __ldcg(A.Y + c0 + k); });
                sweep_bar();
                return true;
            },
            [&](int i, T v) { u[i] = v - sa[i - r0]; });
    }
    case kSwBZ: {
        // column k of L21 against x2; the operand's place holds the entries' indices until their values are known
        const int nr = ms - nc;
        const SweepRows<T, kSwBZ> w = {D.F + t.off + nc, ms, r0, r1, 0, nr, 32};
        const int32_t *ix = D.idx + t.is + nc;
        int *vi = reinterpret_cast<int *>(vs);
        constexpr int W = sizeof(T) / sizeof(int);
        return w.run(
            vs,
            [&] {
#pragma unroll 4
                for (int k = tid; k < nr; k += kSwCompute) vi[W * k] = __ldg(ix + k);
                if (!wait()) return false;
                if (tid < r1 - r0) sa[tid] = __ldcg(A.Y + c0 + r0 + tid);
                sweep_stage(vs, 0, nr, [&](int k) { return __ldcg(A.X + vi[W * k]); });
                sweep_bar();
                return true;
            },
            [&](int k, T v) { A.Z[c0 + k] = sa[k - r0] - v; });
    }
    default: {
        // kSwBX: column j of X against z
        const SweepRows<T, kSwBX> w = {D.Xinv + t.off, nc, r0, r1, r0, nc, sweep_group(nc)};
        return w.run(
            vs,
            [&] {
                if (!wait()) return false;
                sweep_stage(vs, r0, nc, [&](int k) { return __ldcg(A.Z + c0 + k); });
                sweep_bar();
                return true;
            },
            [&](int j, T v) {
                A.X[c0 + j] = v;
                A.x[__ldg(A.perm + c0 + j)] = (double)v;
            });
    }
    }
}

// The scheduling warp asks L2 for a task's part of the factor.
template <typename T>
__device__ __forceinline__ void sweep_prefetch(const Dev<T> &D, const SweepTask &t, int lane)
{
    const int ms = t.ms, nc = t.nc;
    switch (t.kind) {
    case kSwFS:
    case kSwBS:
        if (lane == 0) l2_prefetch(D.F + t.off, (size_t)ms * nc * sizeof(T));
        if (lane == 1) l2_prefetch(D.Inv + (t.kind == kSwFS ? t.inv : t.aux), (size_t)((nc + PW - 1) / PW) * PW * PW * sizeof(T));
        break;
    case kSwFY:
        for (int r = t.r0 + lane; r < t.r1; r += 32) l2_prefetch(D.Xinv + t.off + (int64_t)r * nc, (size_t)(r + 1) * sizeof(T));
        break;
    case kSwFT:
        for (int i = t.r0 + lane; i < t.r1; i += 32) l2_prefetch(D.F + t.off + (int64_t)(nc + i) * ms, (size_t)nc * sizeof(T));
        break;
    case kSwBZ:
        for (int k = t.r0 + lane; k < t.r1; k += 32) l2_prefetch(D.F + t.off + (int64_t)k * ms + nc, (size_t)(ms - nc) * sizeof(T));
        break;
    case kSwBX:
        for (int j = t.r0 + lane; j < t.r1; j += 32) l2_prefetch(D.Xinv + t.off + (int64_t)j * nc + j, (size_t)(nc - j) * sizeof(T));
        break;
    default: break;
    }
}

// Bounded wait until a counter has reached its target: false when another CTA gave up or the limit has passed.
__device__ __forceinline__ bool sweep_poll(const uint32_t *c, uint32_t target, uint64_t wait_ns, const int *err)
{
    uint64_t t0 = 0;
    for (uint32_t it = 0;; it++) {
        uint32_t v;
        // relaxed while it waits (an acquiring load drops the SM's L1 every time), one fence at the end
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
        if ((int32_t)(v - target) >= 0) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            return true;
        }
        if (wait_ns == 0) return false;
        if ((it & 255) == 255) {
            uint64_t now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (now - t0 > wait_ns || *(volatile const int *)err) return false;
        }
    }
}

template <typename T>
static __global__ void __launch_bounds__(kSwThreads, kSwCtas) k_sweep(const SweepArgs<T> A)
{
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ SweepTask desc[2];
    __shared__ int go[2];  // the task's inputs are complete; 0: a wait gave up
    __shared__ T sa[kSwCompute], yb[PW];
    const int tid = threadIdx.x, lane = tid & 31;
    if (A.skip && *A.skip) return;
    if (tid >= kSwCompute) {
        const uint32_t solves = *(volatile uint32_t *)(A.ticket + 1) + 1;
        for (uint32_t i = 0;; i++) {
            const int p = i & 1;
            uint32_t tk = 0;
            if (lane == 0) tk = atomicAdd(A.ticket, 1u);
            tk = __shfl_sync(0xffffffffu, tk, 0);
            if (i >= 2) sweep_sync(kBarFree + p);  // the computing warps are done with this slot
            const bool have = tk < (uint32_t)A.ntasks;
            if (lane < (int)(sizeof(SweepTask) / 16) && have)
                reinterpret_cast<int4 *>(&desc[p])[lane] = __ldg(reinterpret_cast<const int4 *>(A.tasks + tk) + lane);
            if (lane == 0 && !have) desc[p].kind = kSwEnd;
            __syncwarp();
            sweep_arrive(kBarDesc + p);
            if (!have) {
                // every CTA draws one ticket past the list: the last of them leaves the counters to the next solve
                if (lane == 0 && tk == (uint32_t)A.ntasks + gridDim.x - 1) {
                    A.ticket[0] = 0;
                    A.ticket[1] = solves;
                }
                return;
            }
            sweep_prefetch(A.D, desc[p], lane);
            int ok = 1;
            if (lane == 0) {
                const int w = desc[p].wait;
                ok = w < 0 || sweep_poll(A.cnt + w, solves * (uint32_t)desc[p].target, A.wait_ns, A.err);
                if (!ok) atomicExch(A.err, 1);
                go[p] = ok;
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            sweep_arrive(kBarReady + p);
            if (!ok) {  // given up, here or in another CTA: no result is to be taken for one
                for (int k = lane; k < A.n; k += 32) A.x[k] = nan("");
                return;
            }
        }
    }
    T *vs = (T *)sweep_smem;
    for (uint32_t i = 0;; i++) {
        const int p = i & 1;
        sweep_sync(kBarDesc + p);
        const SweepTask &t = desc[p];
        if (t.kind == kSwEnd) return;
        const bool ok = sweep_task(A, t, vs, sa, yb, [&] {
            sweep_sync(kBarReady + p);
            return go[p] != 0;
        });
        if (!ok) return;
        const int done = t.done;
        sweep_bar();  // all of the task's stores precede the count, all its reads the slot's reuse
        if (tid == 0 && done >= 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.cnt + done) : "memory");
        sweep_arrive(kBarFree + p);
    }
}

// The per-row form of the gather lists (gst: first list entry of each front row, src: the update entries in child
// order): two entries inline, longer lists appended to `src` as a number and its entries.
inline void sweep_pairs(const std::vector<int32_t> &gst, std::vector<int32_t> &src, std::vector<int2> &pair)
{
    const size_t rows = gst.size() - 1;
    pair.resize(std::max<size_t>(rows, 1));
    size_t more = 0;
    for (size_t k = 0; k < rows; k++)
        if (gst[k + 1] - gst[k] > 2) more += gst[k + 1] - gst[k];
    src.reserve(src.size() + more);
    for (size_t k = 0; k < rows; k++) {
        const int32_t a = gst[k], n = gst[k + 1] - a;
        int2 q = make_int2(n > 0 ? src[a] : -1, n == 2 ? src[a + 1] : -1);
        if (n > 2) {
            q.y = -2 - (int32_t)src.size();
            src.push_back(n - 1);
            for (int32_t u = 1; u < n; u++) {
                const int32_t e = src[a + u];
                src.push_back(e);
            }
        }
        pair[k] = q;
    }
}

// The task list of one analysis. Level by level up, then down; within a level a kind's longest tiles first.
// Expected counts per front and kind are filled on the way; a task's target is known once its producers are listed.
// vec: the longest operand vector (entries); width: the most tasks of one phase.
template <typename T>
inline void sweep_tasks(const MfSymbolic &S, const std::vector<int32_t> &small_start, const std::vector<int32_t> &small_list,
                        const std::vector<int32_t> &big_start, const std::vector<int32_t> &big_list,
                        const std::vector<int64_t> &inv_off, const std::vector<int64_t> &xinv_off,
                        std::vector<SweepTask> &out, int &vec, int &width)
{
    std::vector<int32_t> exp((size_t)kCntN * S.nsuper, 0);
    out.clear();
    vec = width = 1;
    int64_t bytes = 0;  // a tile's share of the factor in the phase at hand
    auto rows_for = [&](int len) {  // rows of `len` entries per tile
        const int rpc = kSwWarps * (32 / sweep_group(len));
        vec = std::max(vec, len);
        return (int)std::min<int64_t>(kSwCompute, std::max<int64_t>(rpc, bytes / ((int64_t)len * sizeof(T)) / rpc * rpc));
    };
    // a phase in about one wave of tiles, so that a tile's fixed cost (some two microseconds) is paid once, but no tile
    // below 16 KB (the fixed cost would dominate) or above 64 KB (the waves balance; 32 KB measured 1-3 % slower)
    auto set_tile = [&](double entries) {
        bytes = (int64_t)std::min(64.0 * 1024, std::max(16.0 * 1024, entries * sizeof(T) / (0.75 * kSwCtas * 148)));
    };
    auto add = [&](SweepKind kind, int s, int r0, int r1, int wait, int target, int done, int flag) {
        SweepTask t = {};
        t.kind = kind, t.r0 = r0, t.r1 = r1, t.wait = target ? wait : -1, t.target = target, t.done = done, t.flag = flag;
        t.nc = S.ncol[s], t.ms = S.m[s], t.c0 = S.c0[s], t.is = S.idx_start[s];
        t.off = kind == kSwFY || kind == kSwBX ? xinv_off[s] : S.front_off[s];
        t.aux = kind == kSwBS ? inv_off[s] : S.uvec_start[s];
        t.inv = inv_off[s];
        out.push_back(t);
        if (done >= 0) exp[done]++;
    };
    size_t phase0 = 0;
    auto close_phase = [&] {
        width = std::max(width, (int)(out.size() - phase0));
        phase0 = out.size();
    };
    for (int l = 0; l < S.nlevels; l++) {
        double e_x = 0, e_l = 0;
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const double nc = S.ncol[big_list[q]], nr = S.m[big_list[q]] - nc;
            e_x += 0.5 * nc * nc, e_l += nc * nr;
        }
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const int s = big_list[q], nc = S.ncol[s], upd = kCntN * s + kCntUpd;
            if (nc <= kSwGather) continue;
            for (int r0 = 0; r0 < nc; r0 += 2 * kSwCompute)
                add(kSwFA, s, r0, std::min(nc, r0 + 2 * kSwCompute), upd, exp[upd], kCntN * s + kCntA, 0);
        }
        for (int q = small_start[l]; q < small_start[l + 1]; q++) {
            // a root's own sweep down waits for it, else the parent does
            const int s = small_list[q], p = S.parent[s], upd = kCntN * s + kCntUpd;
            add(kSwFS, s, 0, 0, upd, exp[upd], p >= 0 ? kCntN * p + kCntUpd : kCntN * s + kCntY, 0);
        }
        close_phase();
        set_tile(e_x);
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const int s = big_list[q], nc = S.ncol[s];
            const bool own = nc <= kSwGather;
            const int wait = kCntN * s + (own ? kCntUpd : kCntA), target = exp[wait];
            for (int r1 = nc; r1 > 0;) {
                const int r0 = r1 - std::min(r1, rows_for(r1));
                add(kSwFY, s, r0, r1, wait, target, kCntN * s + kCntY, own);
                r1 = r0;
            }
        }
        close_phase();
        set_tile(e_l);
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const int s = big_list[q], nc = S.ncol[s], nr = S.m[s] - nc, p = S.parent[s], y = kCntN * s + kCntY, target = exp[y];
            const int step = rows_for(nc);
            for (int r0 = 0; r0 < nr; r0 += step)
                add(kSwFT, s, r0, std::min(nr, r0 + step), y, target, p >= 0 ? kCntN * p + kCntUpd : -1, 0);
        }
        close_phase();
    }
    auto down_wait = [&](int s) {  // the parent's solution, or a root's own y
        const int p = S.parent[s];
        return p >= 0 ? kCntN * p + kCntX : kCntN * s + kCntY;
    };
    for (int l = S.nlevels - 1; l >= 0; l--) {
        double e_x = 0, e_l = 0;
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const double nc = S.ncol[big_list[q]], nr = S.m[big_list[q]] - nc;
            e_x += 0.5 * nc * nc, e_l += nc * nr;
        }
        set_tile(e_l);
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const int s = big_list[q], nc = S.ncol[s], nr = S.m[s] - nc, wait = down_wait(s), target = exp[wait];
            if (nr == 0) continue;
            const int step = rows_for(nr);
            for (int r0 = 0; r0 < nc; r0 += step) add(kSwBZ, s, r0, std::min(nc, r0 + step), wait, target, kCntN * s + kCntZ, 0);
        }
        for (int q = small_start[l]; q < small_start[l + 1]; q++) {
            const int s = small_list[q], wait = down_wait(s);
            add(kSwBS, s, 0, 0, wait, exp[wait], kCntN * s + kCntX, 0);
        }
        close_phase();
        set_tile(e_x);
        for (int q = big_start[l]; q < big_start[l + 1]; q++) {
            const int s = big_list[q], nc = S.ncol[s], nr = S.m[s] - nc, wait = kCntN * s + (nr ? kCntZ : kCntY), target = exp[wait];
            for (int r0 = 0; r0 < nc;) {
                const int r1 = std::min(nc, r0 + rows_for(nc - r0));
                add(kSwBX, s, r0, r1, wait, target, kCntN * s + kCntX, 0);
                r0 = r1;
            }
        }
        close_phase();
    }
}

}  // namespace mf
}  // namespace ifea
