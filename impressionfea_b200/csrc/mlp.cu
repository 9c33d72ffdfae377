// mlp.cu — the learned warm start's network on the tensor cores: a per-node MLP 16 -> 128 -> 128 -> 128 -> 3 with
// GELU, BF16 weights and activations, FP32 accumulation, trained by Adam on FP32 master weights.
//
// A training step is three launches:
//   k_tile    per 128 rows of the batch, one CTA takes them through the whole network: gather and normalise, three hidden
//             layers, output layer, loss, and back to the first layer's gradient. Activations and layer gradients stay
//             in shared memory as the next product's operand (K-major core matrices without swizzle: 8 rows x 16 B, one
//             16-byte K chunk of all rows after another), pre-activations and then GELU' in tensor memory (three
//             accumulators of 128 columns, a fourth for the backward products); products are tcgen05.mma kind::f16 issued by one
//             thread. Only what the weight gradients need leaves the CTA: activations and layer gradients, transposed.
//   k_wgrad   the weight gradients: partial sums over slices of 512 batch rows (FP32, summed in order by k_update), a
//             slice's operands for 128 x 64 of a gradient all in shared memory, multiplied as they land;
//   k_update  sums the partial sums, the bias gradients and Adam, and the BF16 copies of the new weights.
// Inference is k_tile without the backward half, over all rows in one launch. Every sum runs in a fixed order, so
// training is bit-reproducible run to run.
//
// What bounds a step of 8,192 rows (B200): the chain inside k_tile, 27 us of the step's 47 on the device. It starts
// with 5 us of dependent loads (index, row, normalisation); an epilogue of 128 x 128 GELUs and their derivatives is
// 6,100 cycles of issue on one SM, 8,000 with the transposed stores, a product with its wait 300 - 800. k_wgrad takes
// 11.5 us (16 with a ring of four stages over slices of the whole width), k_update 5.6. A step through the public class
// takes 53 us; with a kernel for each layer and each sum, 21 launches a step with pre-activations, activations and
// transposes through global memory and a wait for the device in every step, it took 336.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <future>
#include <numeric>
#include <random>
#include <system_error>

#include "warmstart.h"

namespace ifea {
namespace wsm {

constexpr int BM = 128, BK = 64, SPLIT_K = 512;
constexpr int kTileThreads = 512, kGradN = 64, kGradStages = SPLIT_K / BK;
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major, no swizzle: core matrices of 8 rows x 16 B (rows 16 B apart, 8-row groups 128 B apart: stride
// offset), the two 16-byte K chunks of one MMA a whole chunk of all rows apart (leading offset); version 1
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t chunk_bytes)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((chunk_bytes >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((128 >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1), both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24
template <int N>
__host__ __device__ constexpr uint32_t idesc() { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); }

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t id, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
        "l"(da), "l"(db), "r"(id), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}

// bounded wait on an mbarrier phase: false if it gave up (an MMA of a few microseconds ends far sooner)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t it = 0; it < (1u << 20); it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// until at most `left` of this thread's groups of copies are in flight (left is known at compile time: one case stays)
__device__ __forceinline__ void cp_async_wait(int left)
{
    switch (left) {
    case 7: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
    case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
    case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
}

#define WSM_TMEM_ST16(taddr, r)                                                                                      \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "                                                     \
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"((r)[0]), "r"((r)[1]), "r"((r)[2]),   \
                 "r"((r)[3]), "r"((r)[4]), "r"((r)[5]), "r"((r)[6]), "r"((r)[7]), "r"((r)[8]), "r"((r)[9]),            \
                 "r"((r)[10]), "r"((r)[11]), "r"((r)[12]), "r"((r)[13]), "r"((r)[14]), "r"((r)[15]), "r"(taddr)        \
                 : "memory")

#define WSM_TMEM_LD16(taddr, r)                                                                                      \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "  \
                 "[%16];"                                                                                            \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),   \
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),           \
                   "=r"(r[15])                                                                                       \
                 : "r"(taddr))

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float z)
{
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

constexpr uint32_t kChunk = BM * 16;             // one 8-column chunk of 128 rows in shared memory
constexpr int kMat = BM * HID * 2;                // a 128 x 128 operand, 32 KB
// element (r, k) of an operand of 128 rows
__host__ __device__ constexpr int core(int r, int k) { return ((k >> 3) * BM + r) * 8 + (k & 7); }

struct Tile {
    const float *x, *t;      // raw inputs [.][16] and targets [.][3]
    const int32_t *idx;      // the rows of the batch (null: 0, 1, ..)
    int64_t n;               // rows of x
    int M;                   // rows of the batch (training: a multiple of 128)
    const float *norm, *par;
    const bf16 *w1, *w2, *w3, *w2t, *w3t;  // weights as operands
    float *y;                // inference: raw outputs [M][3]
    bf16 *xbt, *h1t, *h2t, *dz1t, *dz2t, *dz3t;  // training: [feature][M]
    float *hpart;            // per tile: dW4, db4, the loss
    int *err;
};

// shared memory: weights, activations, (training) transposed weights and layer gradient; inputs, W1; small vectors
template <bool TRAIN>
constexpr int tile_smem() { return (TRAIN ? 6 : 3) * kMat + 2 * BM * NIN * 2 + (3 * HID + NOUT * HID + NOUT + 1) * 4 + 128 * 4 * 4 + 64; }

template <bool TRAIN>
__global__ void __launch_bounds__(kTileThreads, 1) k_tile(Tile g)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    constexpr int TCOLS = TRAIN ? 512 : 128;
    bf16 *sw2 = (bf16 *)sm, *sw3 = sw2 + kMat / 2, *sh = sw3 + kMat / 2;  // sh: the activations
    bf16 *sw2t = sh + kMat / 2, *sw3t = sw2t + kMat / 2, *sdz = sw3t + kMat / 2;
    bf16 *sx = TRAIN ? sdz + kMat / 2 : sw2t, *sw1 = sx + BM * NIN;
    float *sbias = (float *)(sw1 + BM * NIN), *sw4 = sbias + 3 * HID;  // b1, b2, b3; W4, b4
    float *dys = sw4 + NOUT * HID + NOUT + 1, *red = dys + 128 * NOUT;
    uint64_t *bar = (uint64_t *)(((uintptr_t)(red + 128) + 15) & ~(uintptr_t)15);
    uint32_t *tslot = (uint32_t *)(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(TCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
    }
    // weights (already in operand form) asynchronously, behind the first layer
    auto load = [&](bf16 *dst, const bf16 *src, int bytes) {
        for (int q = tid; q < bytes / 16; q += kTileThreads) cp_async16(smem_u32(dst) + 16 * q, (const uint4 *)src + q, 16);
    };
    load(sw1, g.w1, BM * NIN * 2);
    asm volatile("cp.async.commit_group;" ::: "memory");
    load(sw2, g.w2, kMat);
    load(sw3, g.w3, kMat);
    if (TRAIN) {
        load(sw2t, g.w2t, kMat);
        load(sw3t, g.w3t, kMat);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = tid; i < HID; i += kTileThreads) {
        sbias[i] = g.par[OFF_B1 + i];
        sbias[HID + i] = g.par[OFF_B2 + i];
        sbias[2 * HID + i] = g.par[OFF_B3 + i];
    }
    for (int i = tid; i < NOUT * HID + NOUT; i += kTileThreads) sw4[i] = g.par[OFF_W4 + i];
    // normalised inputs, four columns a thread; rows past the data are zero. Threads 0 .. 127 keep their row's targets
    float tgt[NOUT];
    {
        const int r = tid & 127, c0 = 4 * (tid >> 7), row = m0 + r;
        int64_t src = row < g.M ? (int64_t)row : g.n;
        if (TRAIN && g.idx) {  // (host memory: each index is read once)
            if (tid < BM) ((int32_t *)dys)[tid] = g.idx[row];
            __syncthreads();
            src = ((int32_t *)dys)[r];
        }
        float v[4] = {0, 0, 0, 0};
        if (src < g.n) {
            const float4 q = *(const float4 *)(g.x + src * NIN + c0);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = (v[j] - g.norm[c0 + j]) / g.norm[NIN + c0 + j];
        }
        __align__(8) bf16 hb[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            hb[j] = __float2bfloat16_rn(v[j]);
            if (TRAIN) g.xbt[(int64_t)(c0 + j) * g.M + row] = hb[j];
        }
        *(uint2 *)(sx + core(r, c0)) = *(const uint2 *)hb;
        if (TRAIN && tid < BM)
#pragma unroll
            for (int o = 0; o < NOUT; o++)
                tgt[o] = src < g.n ? (g.t[src * NOUT + o] - g.norm[2 * NIN + o]) / g.norm[2 * NIN + NOUT + o] : 0.0f;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::);
    const uint32_t tmem = *tslot;
    uint32_t phase = 0;
    bool ok = true;
    // D(columns col ..) = A B^T over K columns; every thread sees the result when it returns
    auto product = [&](const bf16 *A, const bf16 *B, int K, uint32_t col) {
        if (tid == 0) {
            const uint32_t sa = smem_u32(A), sb = smem_u32(B);
            for (int j = 0; j < K / 16; j++)
                mma_bf16(tmem + col, sdesc(sa + j * 2 * kChunk, kChunk), sdesc(sb + j * 2 * kChunk, kChunk), idesc<HID>(), j > 0);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)));
        }
        ok = mbar_wait(smem_u32(bar), phase) && ok;
        phase ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::);
    };
    // before a product: this CTA's writes to shared memory and reads of tensor memory are done
    auto settle = [&]() {
        asm volatile("tcgen05.fence::before_thread_sync;" ::);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::);
    };
    // a thread's part of an epilogue: row r, columns cb .. cb + 31. Training leaves GELU'(z) where z was, for the way
    // back: the two share the error function, which is what an epilogue spends its time on
    const int r = 32 * (warp & 3) + lane, cb = 32 * (warp >> 2), row = m0 + r;
    const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cb;
    auto hidden = [&](uint32_t col, const float *bias, bf16 *ht) {
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            uint32_t v[16];
            WSM_TMEM_LD16(tl + col + 16 * h, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            __align__(16) bf16 hb[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float z = __uint_as_float(v[j]) + bias[cb + 16 * h + j];
                hb[j] = __float2bfloat16_rn(gelu(z));
                if (TRAIN) v[j] = __float_as_uint(gelu_d(z));
            }
            if (TRAIN) WSM_TMEM_ST16(tl + col + 16 * h, v);
            *(uint4 *)(sh + core(r, cb + 16 * h)) = ((const uint4 *)hb)[0];
            *(uint4 *)(sh + core(r, cb + 16 * h + 8)) = ((const uint4 *)hb)[1];
            if (TRAIN && ht)
#pragma unroll
                for (int j = 0; j < 16; j++) ht[(int64_t)(cb + 16 * h + j) * g.M + row] = hb[j];
        }
        if (TRAIN) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    };
    product(sx, sw1, NIN, 0);
    hidden(0, sbias, g.h1t);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    settle();
    product(sh, sw2, HID, TRAIN ? HID : 0);
    hidden(TRAIN ? HID : 0, sbias + HID, g.h2t);
    settle();
    product(sh, sw3, HID, TRAIN ? 2 * HID : 0);
    hidden(TRAIN ? 2 * HID : 0, sbias + 2 * HID, nullptr);
    __syncthreads();
    // output layer (FP32 over the BF16 activations), a row a thread
    if (tid < BM) {
        float acc[NOUT];
#pragma unroll
        for (int o = 0; o < NOUT; o++) acc[o] = sw4[NOUT * HID + o];
#pragma unroll 4
        for (int q = 0; q < HID / 8; q++) {
            const uint4 u = *(const uint4 *)(sh + core(tid, 8 * q));
            const bf16 *hv = (const bf16 *)&u;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float hf = __bfloat162float(hv[j]);
#pragma unroll
                for (int o = 0; o < NOUT; o++) acc[o] += sw4[o * HID + 8 * q + j] * hf;
            }
        }
        const int mr = m0 + tid;
        if (!TRAIN) {
            if (mr < g.M)
                for (int o = 0; o < NOUT; o++) g.y[(int64_t)mr * NOUT + o] = g.norm[2 * NIN + o] + g.norm[2 * NIN + NOUT + o] * acc[o];
        } else {
            // the loss and its gradient at the output
            const float scale = 2.0f / (float)(g.M * NOUT);
            float l = 0;
#pragma unroll
            for (int o = 0; o < NOUT; o++) {
                const float e = acc[o] - tgt[o];
                l += e * e;
                dys[tid * NOUT + o] = scale * e;
            }
            red[tid] = l;
        }
    }
    if (TRAIN) {
        __syncthreads();
        // dz3 = (dy W4) * GELU'(z3)
        float dy[NOUT];
#pragma unroll
        for (int o = 0; o < NOUT; o++) dy[o] = dys[r * NOUT + o];
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            uint32_t v[16];
            WSM_TMEM_LD16(tl + 2 * HID + 16 * h, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            __align__(16) bf16 hb[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int i = cb + 16 * h + j;
                float dh = 0;
#pragma unroll
                for (int o = 0; o < NOUT; o++) dh += dy[o] * sw4[o * HID + i];
                hb[j] = __float2bfloat16_rn(dh * __uint_as_float(v[j]));
                g.dz3t[(int64_t)i * g.M + row] = hb[j];
            }
            *(uint4 *)(sdz + core(r, cb + 16 * h)) = ((const uint4 *)hb)[0];
            *(uint4 *)(sdz + core(r, cb + 16 * h + 8)) = ((const uint4 *)hb)[1];
        }
        settle();
        if (warp >= 12) {
            // dW4[o][i] = sum over the tile's rows of dy[o] h3[row][i]: a thread owns column i; then db4
            float *out = g.hpart + (int64_t)blockIdx.x * (NOUT * HID + NOUT + 1);
            const int i = tid - 384;
            float acc[NOUT] = {0, 0, 0};
#pragma unroll 8
            for (int k = 0; k < BM; k++) {
                const float hv = __bfloat162float(sh[core(k, i)]);
#pragma unroll
                for (int o = 0; o < NOUT; o++) acc[o] += dys[k * NOUT + o] * hv;
            }
            for (int o = 0; o < NOUT; o++) out[o * HID + i] = acc[o];
            if (i < NOUT) {
                float s = 0;
                for (int k = 0; k < BM; k++) s += dys[k * NOUT + i];
                out[NOUT * HID + i] = s;
            }
        } else if (warp == 11) {
            // the loss: the 128 rows' squares by a tree of halves (64, 32, .. apart)
            float q[4];
            for (int k = 0; k < 4; k++) q[k] = red[lane + 32 * k];
            float s = (q[0] + q[2]) + (q[1] + q[3]);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) g.hpart[(int64_t)blockIdx.x * (NOUT * HID + NOUT + 1) + NOUT * HID + NOUT] = s;
        }
        // back through the hidden layers: dz = (dz above W) * GELU'(z)
        auto back = [&](uint32_t zcol, bf16 *dzt, bool keep) {
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                uint32_t v[16], z[16];
                WSM_TMEM_LD16(tl + 3 * HID + 16 * h, v);
                WSM_TMEM_LD16(tl + zcol + 16 * h, z);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                __align__(16) bf16 hb[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int i = cb + 16 * h + j;
                    hb[j] = __float2bfloat16_rn(__uint_as_float(v[j]) * __uint_as_float(z[j]));
                    dzt[(int64_t)i * g.M + row] = hb[j];
                }
                if (keep) {
                    *(uint4 *)(sdz + core(r, cb + 16 * h)) = ((const uint4 *)hb)[0];
                    *(uint4 *)(sdz + core(r, cb + 16 * h + 8)) = ((const uint4 *)hb)[1];
                }
            }
        };
        product(sdz, sw3t, HID, 3 * HID);
        back(HID, g.dz2t, true);
        settle();
        product(sdz, sw2t, HID, 3 * HID);
        back(0, g.dz1t, false);
    }
    if (__syncthreads_or(!ok) && tid == 0) atomicExch(g.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
}

// Partial weight gradients: part[split][layer] = dz^T h over a slice of 512 batch rows (operands [feature][batch], K-major).
struct Grad {
    const bf16 *A[3], *B[3];  // dz3^T h2^T, dz2^T h1^T, dz1^T x^T
    float *part[3];           // [split][128][128], the last [split][128][16]
    int M;                    // the batch
    int *err;
};
constexpr int grad_smem() { return kGradStages * (BM + kGradN) * BK * 2 + 64; }

// columns n0 .. n0 + N - 1 of slice `split` of a gradient [128][ldp]
template <int N>
__device__ __forceinline__ void grad_slice(const bf16 *A, const bf16 *B, int ld, float *part, int ldp, int n0, int split, int *err)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    constexpr int A_BYTES = BM * BK * 2, STAGE = A_BYTES + kGradN * BK * 2;
    constexpr uint32_t CHUNK_B = N * 16;
    constexpr int TCOLS = N < 32 ? 32 : N;
    uint64_t *bar = (uint64_t *)(sm + kGradStages * STAGE);
    uint32_t *tslot = (uint32_t *)(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k0 = split * SPLIT_K, nblk = (min(ld, k0 + SPLIT_K) - k0) / BK;  // (ld: a multiple of 128)
    const uint32_t sbase = smem_u32(sm);
    for (int b = 0; b < kGradStages; b++) {  // 64 batch rows a stage: 8 chunks of 8, lanes over 16 features x 2 chunks
        if (b < nblk) {
            const int kb = k0 + b * BK;
            const uint32_t sa = sbase + b * STAGE, sb = sa + A_BYTES;
            for (int q = tid; q < BM * 8; q += 256) {
                const int c = 2 * (q / (2 * BM)) + (q & 1), r = (q >> 1) % BM;
                cp_async16(sa + (uint32_t)(c * BM + r) * 16, A + (int64_t)r * ld + kb + 8 * c, 16);
            }
            for (int q = tid; q < N * 8; q += 256) {
                const int c = 2 * (q / (2 * N)) + (q & 1), r = (q >> 1) % N;
                cp_async16(sb + (uint32_t)(c * N + r) * 16, B + (int64_t)(n0 + r) * ld + kb + 8 * c, 16);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(TCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::);
    const uint32_t tmem = *tslot;
#pragma unroll
    for (int b = 0; b < kGradStages; b++) {
        cp_async_wait(kGradStages - 1 - b);  // block b has landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0 && b < nblk) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::);
            const uint32_t sa = sbase + b * STAGE, sb = sa + A_BYTES;
            for (int j = 0; j < BK / 16; j++)
                mma_bf16(tmem, sdesc(sa + j * 2 * kChunk, kChunk), sdesc(sb + j * 2 * CHUNK_B, CHUNK_B), idesc<N>(), (b > 0 || j > 0) ? 1u : 0u);
        }
    }
    if (tid == 0) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)));
    const bool ok = mbar_wait(smem_u32(bar), 0);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        asm volatile("tcgen05.fence::after_thread_sync;" ::);
        const int r = 32 * (warp & 3) + lane;
#pragma unroll 1
        for (int c0 = 16 * (warp >> 2); c0 < N; c0 += 32) {
            uint32_t v[16];
            WSM_TMEM_LD16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float4 *dst = (float4 *)(part + ((int64_t)split * BM + r) * ldp + n0 + c0);
#pragma unroll
            for (int j = 0; j < 4; j++)
                dst[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
}
__global__ void __launch_bounds__(256) k_wgrad(Grad g)
{
    constexpr int PER = HID / kGradN;
    if (blockIdx.y < 2 * PER) {
        const int n0 = kGradN * (blockIdx.y % PER);
        if (blockIdx.y < PER) grad_slice<kGradN>(g.A[0], g.B[0], g.M, g.part[0], HID, n0, blockIdx.x, g.err);
        else grad_slice<kGradN>(g.A[1], g.B[1], g.M, g.part[1], HID, n0, blockIdx.x, g.err);
    } else {
        grad_slice<NIN>(g.A[2], g.B[2], g.M, g.part[2], NIN, 0, blockIdx.x, g.err);
    }
}

// BF16 copies of a hidden weight as operands: W by rows of outputs for the forward products, W^T for the backward ones
struct Weights {
    bf16 *w1, *w2, *w3, *w2t, *w3t;
    __device__ __forceinline__ void publish(int p, float v) const
    {
        const bf16 a = __float2bfloat16_rn(v);
        if (p >= OFF_W1 && p < OFF_W1 + HID * NIN) {
            w1[core((p - OFF_W1) / NIN, (p - OFF_W1) % NIN)] = a;
        } else if (p >= OFF_W2 && p < OFF_W2 + HID * HID) {
            w2[core((p - OFF_W2) / HID, (p - OFF_W2) % HID)] = a;
            w2t[core((p - OFF_W2) % HID, (p - OFF_W2) / HID)] = a;
        } else if (p >= OFF_W3 && p < OFF_W3 + HID * HID) {
            w3[core((p - OFF_W3) / HID, (p - OFF_W3) % HID)] = a;
            w3t[core((p - OFF_W3) % HID, (p - OFF_W3) / HID)] = a;
        }
    }
};
__global__ void k_publish(const float *__restrict__ par, Weights w)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < NPAR; p += gridDim.x * blockDim.x) w.publish(p, par[p]);
}

// The gradient of every parameter from the partial sums (in order), and with lr != 0 one Adam step and the new
// weights' copies. Blocks 0 .. 3 HID - 1: a bias each, its layer gradient's row [HID][M] summed (fixed order); then a
// weight (or an output bias) a thread; the last thread the batch loss, when wanted.
struct Update {
    const bf16 *dzt[3];   // layers 3, 2, 1
    const float *part[3], *hpart;
    int M, splits, nblk;
    float *grad, *par, *m, *v, *loss;
    float lr, bc1, bc2;
    Weights w;
};
__device__ __forceinline__ void adam(const Update &u, int p, float gi)
{
    u.grad[p] = gi;
    if (u.lr == 0.0f) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * u.m[p] + (1 - b1) * gi, vi = b2 * u.v[p] + (1 - b2) * gi * gi;
    u.m[p] = mi;
    u.v[p] = vi;
    const float w = u.par[p] - u.lr * (mi / u.bc1) / (sqrtf(vi / u.bc2) + eps);
    u.par[p] = w;
    u.w.publish(p, w);
}
// sum over the parts j (in order) of p[j * stride]
__device__ __forceinline__ float sum_parts(const float *__restrict__ p, int n, int stride)
{
    float acc = 0;
    for (int j0 = 0; j0 < n; j0 += 16) {
        float q[16];
#pragma unroll
        for (int j = 0; j < 16; j++) q[j] = j0 + j < n ? p[(int64_t)(j0 + j) * stride] : 0.0f;
#pragma unroll
        for (int j = 0; j < 16; j++)
            if (j0 + j < n) acc += q[j];
    }
    return acc;
}
__global__ void __launch_bounds__(256) k_update(Update u)
{
    constexpr int HSTRIDE = NOUT * HID + NOUT + 1;
    if (blockIdx.x < 3 * HID) {
        __shared__ float red[256];
        const int l = blockIdx.x / HID, f = blockIdx.x % HID;
        const bf16 *row = u.dzt[l] + (int64_t)f * u.M;
        float acc = 0;
        for (int i0 = threadIdx.x; i0 < u.M; i0 += 8 * 256) {
            float q[8];
#pragma unroll
            for (int j = 0; j < 8; j++) q[j] = i0 + 256 * j < u.M ? __bfloat162float(row[i0 + 256 * j]) : 0.0f;
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (i0 + 256 * j < u.M) acc += q[j];
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        for (int s = 128; s > 0; s >>= 1) {
            if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
            __syncthreads();
        }
        if (threadIdx.x == 0) adam(u, (l == 0 ? OFF_B3 : l == 1 ? OFF_B2 : OFF_B1) + f, red[0]);
        return;
    }
    int q = (blockIdx.x - 3 * HID) * 256 + threadIdx.x;
    if (q < 2 * HID * HID) {
        const int l = q / (HID * HID), i = q % (HID * HID);
        adam(u, (l == 0 ? OFF_W3 : OFF_W2) + i, sum_parts(u.part[l] + i, u.splits, HID * HID));
        return;
    }
    q -= 2 * HID * HID;
    if (q < HID * NIN) {
        adam(u, OFF_W1 + q, sum_parts(u.part[2] + q, u.splits, HID * NIN));
        return;
    }
    q -= HID * NIN;
    if (q < NOUT * HID + NOUT) adam(u, OFF_W4 + q, sum_parts(u.hpart + q, u.nblk, HSTRIDE));
    else if (q == NOUT * HID + NOUT && u.loss) *u.loss = sum_parts(u.hpart + q, u.nblk, HSTRIDE);
}
constexpr int kUpdateBlocks = 3 * HID + (2 * HID * HID + HID * NIN + NOUT * HID + NOUT + 1 + 255) / 256;

// column sums and sums of squares of an [n][w] FP32 array, per block (double, fixed order)
__global__ void k_moments(const float *__restrict__ x, int64_t n, int w, double *__restrict__ part)
{
    __shared__ double red[2][256];
    for (int c = 0; c < w; c++) {
        double s = 0, q = 0;
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
            double a = x[r * w + c];
            s += a;
            q += a * a;
        }
        red[0][threadIdx.x] = s;
        red[1][threadIdx.x] = q;
        __syncthreads();
        for (int k = 128; k > 0; k >>= 1) {
            if (threadIdx.x < k) {
                red[0][threadIdx.x] += red[0][threadIdx.x + k];
                red[1][threadIdx.x] += red[1][threadIdx.x + k];
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            part[((int64_t)blockIdx.x * w + c) * 2] = red[0][0];
            part[((int64_t)blockIdx.x * w + c) * 2 + 1] = red[1][0];
        }
        __syncthreads();
    }
}

__global__ void k_read_err(int *err, int *out) { *out = *err; *err = 0; }

}  // namespace wsm

using namespace wsm;

WarmStartNet::WarmStartNet(uint64_t seed)
{
    cuda_check(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking), "cudaStreamCreate");
    par_.resize(NPAR); grad_.resize(NPAR); m_.resize(NPAR); v_.resize(NPAR); norm_.resize(NNORM);
    w1_.resize(HID * NIN); w2_.resize(HID * HID); w3_.resize(HID * HID); w2t_.resize(HID * HID); w3t_.resize(HID * HID);
    loss_.resize(4);
    loss_.zero(st_);  // slots 2-3 are the tensor-core error flag and its copy: they must start at zero
    // He-uniform initial weights, zero biases (seeded)
    std::vector<float> p(NPAR, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fan_in, int count) {
        float a = std::sqrt(6.0f / (float)fan_in);
        std::uniform_real_distribution<float> u(-a, a);
        for (int i = 0; i < count; i++) p[off + i] = u(rng);
    };
    fill(OFF_W1, NIN, HID * NIN);
    fill(OFF_W2, HID, HID * HID);
    fill(OFF_W3, HID, HID * HID);
    fill(OFF_W4, HID, NOUT * HID);
    for (int i = 0; i < NOUT * HID; i++) p[OFF_W4 + i] *= 0.1f;  // a small output layer: the first guess stays near zero
    set_params(p.data());
    norm_host_.assign(NNORM, 0.0f);
    for (int c = 0; c < NIN; c++) norm_host_[NIN + c] = 1.0f;
    for (int o = 0; o < NOUT; o++) norm_host_[2 * NIN + NOUT + o] = 1.0f;
    set_norm(norm_host_.data());
}

WarmStartNet::~WarmStartNet()
{
    if (st_) {
        cudaStreamSynchronize(st_);
        cudaStreamDestroy(st_);
    }
}

void WarmStartNet::get_params(float *host) const
{
    cuda_check(cudaMemcpyAsync(host, par_.p, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, st_), "D2H");
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
}

void WarmStartNet::set_params(const float *host)
{
    cuda_check(cudaMemcpyAsync(par_.p, host, sizeof(float) * NPAR, cudaMemcpyHostToDevice, st_), "H2D");
    m_.zero(st_);
    v_.zero(st_);
    adam_t_ = 0;
    publish(st_);
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
}

void WarmStartNet::get_norm(float *host) const { std::memcpy(host, norm_host_.data(), sizeof(float) * NNORM); }

void WarmStartNet::set_norm(const float *host)
{
    norm_host_.assign(host, host + NNORM);
    cuda_check(cudaMemcpyAsync(norm_.p, norm_host_.data(), sizeof(float) * NNORM, cudaMemcpyHostToDevice, st_), "H2D");
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
}

void WarmStartNet::publish(cudaStream_t s)
{
    k_publish<<<(NPAR + 255) / 256, 256, 0, s>>>(par_.p, Weights{w1_.p, w2_.p, w3_.p, w2t_.p, w3t_.p});
}

void WarmStartNet::add_samples_device(const float *d_x, const float *d_t, int64_t n, cudaStream_t s)
{
    if (n <= 0) return;
    if (count_ + n > cap_) {
        int64_t cap = std::max<int64_t>(2 * cap_, std::max<int64_t>(count_ + n, 1 << 16));
        DBuf<float> nx, nt;
        nx.resize((size_t)cap * NIN);
        nt.resize((size_t)cap * NOUT);
        if (count_) {
            cuda_check(cudaMemcpyAsync(nx.p, dx_.p, sizeof(float) * count_ * NIN, cudaMemcpyDeviceToDevice, s), "D2D");
            cuda_check(cudaMemcpyAsync(nt.p, dt_.p, sizeof(float) * count_ * NOUT, cudaMemcpyDeviceToDevice, s), "D2D");
        }
        cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        swap_buf(dx_, nx);
        swap_buf(dt_, nt);
        cap_ = cap;
    }
    cuda_check(cudaMemcpyAsync(dx_.p + count_ * NIN, d_x, sizeof(float) * n * NIN, cudaMemcpyDeviceToDevice, s), "D2D");
    cuda_check(cudaMemcpyAsync(dt_.p + count_ * NOUT, d_t, sizeof(float) * n * NOUT, cudaMemcpyDeviceToDevice, s), "D2D");
    count_ += n;
}

void WarmStartNet::add_samples_host(const float *x, const float *t, int64_t n)
{
    DBuf<float> a, b;
    a.upload(x, (size_t)n * NIN, st_);
    b.upload(t, (size_t)n * NOUT, st_);
    add_samples_device(a.p, b.p, n, st_);
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
}

void WarmStartNet::fit_normalisation()
{
    if (count_ < 2) throw Failure(IFEA_BAD_STATE, "The warm-start network has fewer than two training samples.");
    const int blocks = 148;
    DBuf<double> part;
    part.resize((size_t)blocks * NIN * 2);
    std::vector<double> h((size_t)blocks * NIN * 2);
    for (int pass = 0; pass < 2; pass++) {
        int w = pass == 0 ? NIN : NOUT;
        const float *src = pass == 0 ? dx_.p : dt_.p;
        k_moments<<<blocks, 256, 0, st_>>>(src, count_, w, part.p);
        cuda_check(cudaMemcpyAsync(h.data(), part.p, sizeof(double) * blocks * w * 2, cudaMemcpyDeviceToHost, st_), "D2H");
        cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
        for (int c = 0; c < w; c++) {
            double s = 0, q = 0;
            for (int b = 0; b < blocks; b++) {
                s += h[((size_t)b * w + c) * 2];
                q += h[((size_t)b * w + c) * 2 + 1];
            }
            double mean = s / count_, var = std::max(0.0, q / count_ - mean * mean);
            double sd = std::sqrt(var);
            int off = pass == 0 ? 0 : 2 * NIN;
            norm_host_[off + c] = (float)mean;
            norm_host_[off + w + c] = (float)(sd > 1e-6 ? sd : 1.0);
        }
    }
    set_norm(norm_host_.data());
}

void WarmStartNet::ensure_batch(int B)
{
    if (B <= bcap_) return;
    size_t b = (size_t)B;
    xbt_.resize(b * NIN);
    h1t_.resize(b * HID); h2t_.resize(b * HID);
    dz1t_.resize(b * HID); dz2t_.resize(b * HID); dz3t_.resize(b * HID);
    int splits = (B + SPLIT_K - 1) / SPLIT_K;
    part_.resize((size_t)splits * (2 * HID * HID + HID * NIN));
    hpart_.resize((size_t)((B + 127) / 128) * (NOUT * HID + NOUT + 1));
    bcap_ = B;
}

// One step on a batch of B rows (a multiple of 128; rows idx of the n rows x, t): gradients into grad_, and with lr != 0
// one Adam step; with loss the sum of the batch's squared errors.
void WarmStartNet::step(const float *x, const float *t, const int32_t *idx, int64_t n, int B, float lr, float *loss, cudaStream_t s)
{
    int *err = (int *)loss_.p + 2;
    const int splits = (B + SPLIT_K - 1) / SPLIT_K, nblk = B / BM;
    Tile g{};
    g.x = x; g.t = t; g.idx = idx; g.n = n; g.M = B; g.norm = norm_.p; g.par = par_.p;
    g.w1 = w1_.p; g.w2 = w2_.p; g.w3 = w3_.p; g.w2t = w2t_.p; g.w3t = w3t_.p;
    g.xbt = xbt_.p; g.h1t = h1t_.p; g.h2t = h2t_.p; g.dz1t = dz1t_.p; g.dz2t = dz2t_.p; g.dz3t = dz3t_.p;
    g.hpart = hpart_.p; g.err = err;
    ensure_dynamic_smem((const void *)k_tile<true>, tile_smem<true>());
    k_tile<true><<<nblk, kTileThreads, tile_smem<true>(), s>>>(g);
    float *p3 = part_.p, *p2 = p3 + (size_t)splits * HID * HID, *p1 = p2 + (size_t)splits * HID * HID;
    Grad w{{dz3t_.p, dz2t_.p, dz1t_.p}, {h2t_.p, h1t_.p, xbt_.p}, {p3, p2, p1}, B, err};
    ensure_dynamic_smem((const void *)k_wgrad, grad_smem());
    k_wgrad<<<dim3(splits, 2 * (HID / kGradN) + 1), 256, grad_smem(), s>>>(w);
    Update u{};
    u.dzt[0] = dz3t_.p; u.dzt[1] = dz2t_.p; u.dzt[2] = dz1t_.p;
    u.part[0] = p3; u.part[1] = p2; u.part[2] = p1; u.hpart = hpart_.p;
    u.M = B; u.splits = splits; u.nblk = nblk;
    u.grad = grad_.p; u.par = par_.p; u.m = m_.p; u.v = v_.p; u.loss = loss; u.lr = lr;
    u.w = Weights{w1_.p, w2_.p, w3_.p, w2t_.p, w3t_.p};
    if (lr != 0.0f) {
        adam_t_++;
        u.bc1 = 1.0f - std::pow(0.9f, (float)adam_t_);
        u.bc2 = 1.0f - std::pow(0.999f, (float)adam_t_);
    }
    k_update<<<kUpdateBlocks, 256, 0, s>>>(u);
    cuda_check(cudaGetLastError(), "warm-start training launch");
}

void WarmStartNet::infer_device(const float *d_x, int64_t n, float *d_y, cudaStream_t s)
{
    if (n <= 0) return;
    ensure_dynamic_smem((const void *)k_tile<false>, tile_smem<false>());
    for (int64_t done = 0; done < n;) {  // (one launch up to a thousand million rows)
        const int M = (int)std::min<int64_t>(n - done, 1 << 30);
        Tile g{};
        g.x = d_x + done * NIN; g.n = M; g.M = M; g.norm = norm_.p; g.par = par_.p; g.w1 = w1_.p; g.w2 = w2_.p; g.w3 = w3_.p;
        g.y = d_y + done * NOUT; g.err = (int *)loss_.p + 2;
        k_tile<false><<<(M + BM - 1) / BM, kTileThreads, tile_smem<false>(), s>>>(g);
        cuda_check(cudaGetLastError(), "warm-start inference launch");
        done += M;
    }
    int e = 0;
    k_read_err<<<1, 1, 0, s>>>((int *)loss_.p + 2, (int *)loss_.p + 3);
    cuda_check(cudaMemcpyAsync(&e, (int *)loss_.p + 3, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    if (e) throw Failure(IFEA_CUDA_ERROR, "Warm-start network: a tensor-core wait timed out.");
}

void WarmStartNet::infer_host(const float *x, int64_t n, float *y)
{
    DBuf<float> a, b;
    a.upload(x, (size_t)n * NIN, st_);
    b.resize((size_t)n * NOUT);
    infer_device(a.p, n, b.p, st_);
    b.download(y, (size_t)n * NOUT, st_);
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
}

float WarmStartNet::gradients_host(const float *x, const float *t, int64_t n, float *grad_host)
{
    if (n <= 0 || n % 128 || n > BMAX) throw Failure(IFEA_INPUT_INVALID, "Gradient rows must be a positive multiple of 128, at most 8192.");
    int B = (int)n;
    ensure_batch(B);
    DBuf<float> a, b;
    a.upload(x, (size_t)n * NIN, st_);
    b.upload(t, (size_t)n * NOUT, st_);
    step(a.p, b.p, nullptr, n, B, 0.0f, nullptr, st_);
    std::vector<float> g(NPAR + 1);
    cuda_check(cudaMemcpyAsync(g.data(), grad_.p, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, st_), "D2H");
    int e = 0;
    k_read_err<<<1, 1, 0, st_>>>((int *)loss_.p + 2, (int *)loss_.p + 3);
    cuda_check(cudaMemcpyAsync(&e, (int *)loss_.p + 3, sizeof(int), cudaMemcpyDeviceToHost, st_), "D2H");
    // the loss: the last per-block slot of the head partials, summed on the host
    int nblk = (B + 127) / 128, hstride = NOUT * HID + NOUT + 1;
    std::vector<float> hp((size_t)nblk * hstride);
    cuda_check(cudaMemcpyAsync(hp.data(), hpart_.p, sizeof(float) * hp.size(), cudaMemcpyDeviceToHost, st_), "D2H");
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
    if (e) throw Failure(IFEA_CUDA_ERROR, "Warm-start network: a tensor-core wait timed out.");
    std::memcpy(grad_host, g.data(), sizeof(float) * NPAR);
    double l = 0;
    for (int k = 0; k < nblk; k++) l += hp[(size_t)k * hstride + hstride - 1];
    return (float)(l / ((double)n * NOUT));
}

float WarmStartNet::train(int steps, int batch, float lr, uint64_t seed)
{
    if (count_ < 1) throw Failure(IFEA_BAD_STATE, "The warm-start network has no training samples.");
    int B = std::max(128, std::min(BMAX, batch / 128 * 128));
    ensure_batch(B);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st_);
    std::mt19937_64 rng(seed);
    // The next order of the samples is shuffled by a second thread while batches of the current one are launched
    // (below kShuffleAhead samples shuffling takes less than starting a thread).
    std::vector<int32_t> perm((size_t)count_), ahead;
    std::iota(perm.begin(), perm.end(), 0);
    int64_t pos = count_, shuffles = ((int64_t)steps * B + count_ - 1) / count_;
    std::future<void> busy;
    auto next_order = [&]() {
        if (busy.valid()) {
            busy.get();
            perm.swap(ahead);
        } else {
            std::shuffle(perm.begin(), perm.end(), rng);
        }
        pos = 0;
        if (--shuffles <= 0 || count_ < kShuffleAhead) return;
        ahead = perm;
        try {
            busy = std::async(std::launch::async, [&] { std::shuffle(ahead.begin(), ahead.end(), rng); });
        } catch (const std::system_error &) {  // (no thread to be had: shuffled above when its turn comes)
        }
    };
    // The device reads a batch's indices from pinned host memory, out of a ring of slots, so that the host runs ahead.
    HostPinned<int32_t> hidx;
    hidx.resize((size_t)B * kIdxSlots);
    struct Drain {  // (an error leaves no kernel behind that reads a slot)
        cudaStream_t s;
        ~Drain() { cudaStreamSynchronize(s); }
    } drain{st_};
    cudaEvent_t free_ev[kIdxSlots];
    for (auto &e : free_ev) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    DBuf<float> losses;
    int tail = std::max(1, steps / 10);
    losses.resize((size_t)tail);
    losses.zero(st_);
    for (int it = 0; it < steps; it++) {
        const int slot = it % kIdxSlots;
        int32_t *hb = hidx.p + (size_t)slot * B;
        if (it >= kIdxSlots) cuda_check(cudaEventSynchronize(free_ev[slot]), "cudaEventSynchronize");
        for (int r = 0; r < B;) {
            if (pos >= count_) next_order();
            const int take = (int)std::min<int64_t>(B - r, count_ - pos);
            std::memcpy(hb + r, perm.data() + pos, sizeof(int32_t) * take);
            r += take;
            pos += take;
        }
        step(dx_.p, dt_.p, hb, count_, B, lr, it >= steps - tail ? losses.p + (it - (steps - tail)) : nullptr, st_);
        cuda_check(cudaEventRecord(free_ev[slot], st_), "cudaEventRecord");
    }
    std::vector<float> hl((size_t)tail);
    losses.download(hl.data(), (size_t)tail, st_);
    cudaEventRecord(e1, st_);
    int e = 0;
    k_read_err<<<1, 1, 0, st_>>>((int *)loss_.p + 2, (int *)loss_.p + 3);
    cuda_check(cudaMemcpyAsync(&e, (int *)loss_.p + 3, sizeof(int), cudaMemcpyDeviceToHost, st_), "D2H");
    cuda_check(cudaStreamSynchronize(st_), "cudaStreamSynchronize");
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    train_ms += ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (auto &q : free_ev) cudaEventDestroy(q);
    if (e) throw Failure(IFEA_CUDA_ERROR, "Warm-start network: a tensor-core wait timed out.");
    double l = 0;
    for (float v : hl) l += v;
    return (float)(l / tail / ((double)B * NOUT));
}

}  // namespace ifea

// ------------------------------------------------------------------ C ABI

namespace {
template <class F>
ifea_status guard_mlp(ifea_mlp *m, F &&f)
{
    if (!m || !m->net) return IFEA_INPUT_INVALID;
    try {
        f(*m->net);
        return IFEA_OK;
    } catch (const ifea::Failure &e) {
        m->err = e.what();
        return e.status;
    } catch (const std::exception &e) {
        m->err = e.what();
        return IFEA_CUDA_ERROR;
    }
}
}  // namespace

extern "C" {

ifea_status ifea_mlp_create(uint64_t seed, ifea_mlp **out)
{
    if (!out) return IFEA_INPUT_INVALID;
    *out = nullptr;
    auto *m = new ifea_mlp;
    try {
        m->net = new ifea::WarmStartNet(seed);
    } catch (const std::exception &e) {
        delete m;
        return IFEA_CUDA_ERROR;
    }
    *out = m;
    return IFEA_OK;
}

void ifea_mlp_destroy(ifea_mlp *m)
{
    if (!m) return;
    delete m->net;
    delete m;
}

const char *ifea_mlp_last_error(const ifea_mlp *m) { return m ? m->err.c_str() : "null network"; }

int64_t ifea_mlp_param_count(void) { return ifea::wsm::NPAR; }

ifea_status ifea_mlp_get_params(ifea_mlp *m, float *host, int64_t count)
{
    if (count != ifea::wsm::NPAR || !host) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.get_params(host); });
}

ifea_status ifea_mlp_set_params(ifea_mlp *m, const float *host, int64_t count)
{
    if (count != ifea::wsm::NPAR || !host) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.set_params(host); });
}

ifea_status ifea_mlp_get_normalisation(ifea_mlp *m, float *host)
{
    if (!host) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.get_norm(host); });
}

ifea_status ifea_mlp_set_normalisation(ifea_mlp *m, const float *host)
{
    if (!host) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.set_norm(host); });
}

ifea_status ifea_mlp_add_samples(ifea_mlp *m, const float *features, const float *targets, int64_t n)
{
    if (n < 0 || (n > 0 && (!features || !targets))) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &net) { net.add_samples_host(features, targets, n); });
}

int64_t ifea_mlp_samples(const ifea_mlp *m) { return m && m->net ? m->net->samples() : 0; }

ifea_status ifea_mlp_clear_samples(ifea_mlp *m)
{
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.clear_samples(); });
}

ifea_status ifea_mlp_fit_normalisation(ifea_mlp *m)
{
    return guard_mlp(m, [&](ifea::WarmStartNet &n) { n.fit_normalisation(); });
}

ifea_status ifea_mlp_forward(ifea_mlp *m, const float *x, int64_t n, float *y)
{
    if (n < 0 || (n > 0 && (!x || !y))) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &net) { net.infer_host(x, n, y); });
}

ifea_status ifea_mlp_gradients(ifea_mlp *m, const float *x, const float *t, int64_t n, float *grad, float *loss)
{
    if (!x || !t || !grad) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &net) {
        float l = net.gradients_host(x, t, n, grad);
        if (loss) *loss = l;
    });
}

ifea_status ifea_mlp_train(ifea_mlp *m, int32_t steps, int32_t batch, float lr, uint64_t seed, float *final_loss,
                           double *gpu_ms)
{
    if (steps <= 0 || batch <= 0 || !(lr > 0)) return IFEA_INPUT_INVALID;
    return guard_mlp(m, [&](ifea::WarmStartNet &net) {
        double before = net.train_ms;
        float l = net.train(steps, batch, lr, seed);
        if (final_loss) *final_loss = l;
        if (gpu_ms) *gpu_ms = net.train_ms - before;
    });
}

}  // extern "C"
