// Learned face-flux surrogate: a 17 -> kHid x kNHid -> 8 SmeLU MLP (17-64-64-8 by default)
// trained and run on sm_100a.  Every matrix product is a BF16 tcgen05 MMA with an FP32 accumulator in
// tensor memory; operands are staged into shared memory by bulk copies from the blocked
// K-major layout of nn_umma.cuh.  The forward products write the next layer's operands
// (normal and transposed) and the activation derivative from their epilogues; the backward
// products fold that derivative and the bias-gradient sums into theirs; weight gradients
// are batch-split products reduced by the Adam kernel.  No counterpart exists in the
// reference, whose face solver is always exact (src/modules/solvers/solver.f90:163-187).
#include <chrono>
#include <cstdlib>
#include <thread>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "dumses_gpu.h"
#include "mhd_kernels.cuh"
#include "nn_features.cuh"
#include "nn_host.h"
#include "nn_umma.cuh"

namespace dg {
namespace nn {

using bf16 = __nv_bfloat16;

__host__ __device__ constexpr int layer_k(int l) { return l == 0 ? kInPad : kHid; }
__host__ __device__ constexpr int layer_n(int l) { return l == kNHid ? kOutPad : kHid; }
__host__ __device__ constexpr int real_k(int l) { return l == 0 ? kIn : kHid; }
__host__ __device__ constexpr int real_n(int l) { return l == kNHid ? kOut : kHid; }
// row length of the weight-gradient partials of hidden layer l: its B operand is the
// transposed input (kInPad rows) or the transposed, zero-padded activations (kHidT rows)
__host__ __device__ constexpr int dw_cols(int l) { return l == 0 ? kInPad : kHidT; }

__host__ __device__ constexpr int param_count() {
    int n = 0;
    for (int l = 0; l < kNL; l++) n += real_k(l) * real_n(l) + real_n(l);
    return n;
}

enum { M_FWD_HID = 0, M_FWD_OUT = 1, M_BWD_HID = 2, M_DW = 3 };

constexpr int kGemmSmem = 65536 + 1024;  // A tile, B tile, barriers, bias sums (caps residency at 3 CTAs/SM)

struct GemmArgs {
    const bf16 *A, *B;
    int C;             // reduction columns per CTA
    const float *bias; // forward
    bf16 *Hn, *Ht;     // outputs: blocked normal [rows][kHid] and transposed [kHidT][rows]
    float *G;          // activation derivative [rows][kHid]: written forward, read backward
    float *Y;          // network output [rows][8]
    float *part;       // weight-gradient partials [split][128][N] or bias partials [tile][128]
    long long rows;    // batch rows (row tiles x 128)
    int *err;
};

__device__ __forceinline__ void store_bf16x8(bf16 *dst, const float *v) {
    __align__(16) bf16 h[8];
#pragma unroll
    for (int q = 0; q < 8; q++) h[q] = __float2bfloat16_rn(v[q]);
    *(uint4 *)dst = *(const uint4 *)h;
}

template <int MODE, int N>
__device__ __forceinline__ void epilogue(const GemmArgs &g, uint32_t tmem, long long tile, int warp, int lane,
                                         float *sred) {
    const int rl = warp * 32 + lane;
    const long long row = tile * kTileRows + rl;
    const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
    if constexpr (MODE == M_DW) {
#pragma unroll
        for (int cc = 0; cc < N / 16; cc++) {
            float v[16];
            tmem_ld16(taddr + cc * 16, v);
            float4 *o = (float4 *)(g.part + ((long long)tile * kTileRows + rl) * N + cc * 16);
#pragma unroll
            for (int q = 0; q < 4; q++) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
    } else if constexpr (MODE == M_FWD_OUT) {
        float v[16];
        tmem_ld16(taddr, v);
        float4 *o = (float4 *)(g.Y + row * kOut);
        o[0] = make_float4(v[0] + g.bias[0], v[1] + g.bias[1], v[2] + g.bias[2], v[3] + g.bias[3]);
        o[1] = make_float4(v[4] + g.bias[4], v[5] + g.bias[5], v[6] + g.bias[6], v[7] + g.bias[7]);
    } else {
        for (int cc = 0; cc < kHid / 16; cc++) {
            float v[16];
            tmem_ld16(taddr + cc * 16, v);
            float *gp = g.G + row * kHid + cc * 16;
            if constexpr (MODE == M_FWD_HID) {
                float gd[16];
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const float z = v[q] + g.bias[cc * 16 + q];
                    v[q] = smelu(z);
                    gd[q] = smelu_d(z);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) ((float4 *)gp)[q] = make_float4(gd[4 * q], gd[4 * q + 1], gd[4 * q + 2], gd[4 * q + 3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 d = ((const float4 *)gp)[q];
                    v[4 * q] *= d.x; v[4 * q + 1] *= d.y; v[4 * q + 2] *= d.z; v[4 * q + 3] *= d.w;
                }
#pragma unroll
                for (int q = 0; q < 16; q++) {  // bias gradient: column sums over the tile
                    float s = v[q];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                    if (lane == 0) atomicAdd(&sred[cc * 16 + q], s);
                }
            }
            // normal blocked layout [rows/128][kHid/8][128][8]
            store_bf16x8(g.Hn + ((tile * (kHid / 8) + cc * 2) * kTileRows + rl) * 8, v);
            store_bf16x8(g.Hn + ((tile * (kHid / 8) + cc * 2 + 1) * kTileRows + rl) * 8, v + 8);
            // transposed blocked layout [rows/8][kHidT][8] (rows kHid.. are never written: zero)
            bf16 *t = g.Ht + (row >> 3) * (kHidT * 8) + (row & 7);
#pragma unroll
            for (int q = 0; q < 16; q++) t[(cc * 16 + q) * 8] = __float2bfloat16_rn(v[q]);
        }
    }
}

// one 128-row tile (forward / backward modes) or one batch split (weight-gradient mode)
template <int MODE, int N>
__global__ void __launch_bounds__(128) k_gemm(GemmArgs g) {
    extern __shared__ __align__(1024) unsigned char sm[];
    bf16 *As = (bf16 *)sm;
    bf16 *Bs = (bf16 *)(sm + 32768);
    uint64_t *bar = (uint64_t *)(sm + 65536);
    uint32_t *tslot = (uint32_t *)(sm + 65536 + 16);
    int *sflag = (int *)(sm + 65536 + 32);
    float *sred = (float *)(sm + 65536 + 64);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
        *sflag = 1;
    }
    sred[tid] = 0.0f;
    if (warp == 0) tmem_alloc(tslot, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const long long tile = blockIdx.x;
    if (tid == 0) {
        bool ok = true;
        if constexpr (MODE != M_DW) {
            const unsigned abytes = kTileRows * g.C * 2, bbytes = N * g.C * 2;
            mbar_expect_tx(&bar[0], abytes + bbytes);
            bulk_g2s(As, g.A + tile * (long long)g.C * kTileRows, abytes, &bar[0]);
            bulk_g2s(Bs, g.B, bbytes, &bar[0]);
            ok = mbar_wait(&bar[0], 0);
            if (ok) {
                tc_fence_after();
                mma_tiles(tmem, As, Bs, N, g.C / 16, 0);
                mma_commit(&bar[1]);
                ok = mbar_wait(&bar[1], 0);
                if (!ok) mbar_wait(&bar[1], 0);
            } else {
                mbar_wait(&bar[0], 0);  // let the copies land before the block leaves
            }
        } else {
            const int nch = g.C / 128;
            for (int c = 0; c < nch; c++) {
                const long long k0 = tile * (long long)g.C + c * 128;
                const unsigned abytes = kTileRows * 128 * 2, bbytes = N * 128 * 2;
                mbar_expect_tx(&bar[0], abytes + bbytes);
                bulk_g2s(As, g.A + (k0 / 8) * kTileRows * 8, abytes, &bar[0]);
                bulk_g2s(Bs, g.B + (k0 / 8) * N * 8, bbytes, &bar[0]);
                ok = mbar_wait(&bar[0], c & 1);
                if (!ok) { mbar_wait(&bar[0], c & 1); break; }
                tc_fence_after();
                mma_tiles(tmem, As, Bs, N, 8, c > 0);
                mma_commit(&bar[1]);
                ok = mbar_wait(&bar[1], c & 1);
                if (!ok) { mbar_wait(&bar[1], c & 1); break; }
            }
        }
        if (!ok) {
            *sflag = 0;
            atomicOr(g.err, NN_ERR_WAIT);
        }
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const bool ok = *sflag != 0;
    if (ok) epilogue<MODE, N>(g, tmem, tile, warp, lane, sred);
    tc_fence_before();
    __syncthreads();
    if (MODE == M_BWD_HID && ok) g.part[tile * kTileRows + tid] = sred[tid];
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {  // splitmix64 finaliser
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// batch assembly: rows drawn at random (with replacement) or in order from `first`;
// rows past the end of the sample set are zero
__global__ void k_gather(const float *__restrict__ xs, const float *__restrict__ ts, long long ns, long long rows,
                         int random, unsigned long long seed, long long first, const Scaling *__restrict__ sc,
                         bf16 *__restrict__ Xn, bf16 *__restrict__ Xt, float *__restrict__ Tb) {
    const long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (b >= rows) return;
    long long idx = random ? (long long)(mix64(seed ^ (unsigned long long)b * 0xD1B54A32D192ED03ull) % (unsigned long long)ns)
                           : first + b;
    float x[kInPad], t[kOut];
#pragma unroll
    for (int n = 0; n < kInPad; n++) x[n] = 0.0f;
#pragma unroll
    for (int n = 0; n < kOut; n++) t[n] = 0.0f;
    if (idx < ns) {
#pragma unroll
        for (int n = 0; n < kIn; n++) x[n] = (xs[idx * kIn + n] - sc->xmu[n]) * sc->xisd[n];
        if (ts) {
#pragma unroll
            for (int n = 0; n < kOut; n++) t[n] = ts[idx * kOut + n] / sc->ysd[n];
        }
    }
    const long long tile = b / kTileRows, rl = b % kTileRows;
#pragma unroll
    for (int cg = 0; cg < kInPad / 8; cg++) store_bf16x8(Xn + ((tile * (kInPad / 8) + cg) * kTileRows + rl) * 8, x + cg * 8);
    bf16 *xt = Xt + (b >> 3) * (kInPad * 8) + (b & 7);
#pragma unroll
    for (int n = 0; n < kInPad; n++) xt[n * 8] = __float2bfloat16_rn(x[n]);
    float4 *tb = (float4 *)(Tb + b * kOut);
    tb[0] = make_float4(t[0], t[1], t[2], t[3]);
    tb[1] = make_float4(t[4], t[5], t[6], t[7]);
}

// mean-squared-error gradient of the outputs, its transposed copy, and per-tile sums of
// the loss and of the output-bias gradient
__global__ void __launch_bounds__(128) k_loss(const float *__restrict__ Y, const float *__restrict__ Tb, long long rows,
                                              long long valid, bf16 *__restrict__ Dn, bf16 *__restrict__ Dt,
                                              float *__restrict__ lpart, float *__restrict__ bpart) {
    const long long b = blockIdx.x * (long long)kTileRows + threadIdx.x;
    const int rl = threadIdx.x;
    const float sc = 2.0f / (float)(valid * kOut);
    float d[16], l = 0.0f;
#pragma unroll
    for (int n = 0; n < 16; n++) d[n] = 0.0f;
    if (b < valid) {
#pragma unroll
        for (int n = 0; n < kOut; n++) {
            const float e = Y[b * kOut + n] - Tb[b * kOut + n];
            d[n] = sc * e;
            l += e * e;
        }
    }
    store_bf16x8(Dn + ((blockIdx.x * 2LL + 0) * kTileRows + rl) * 8, d);
    store_bf16x8(Dn + ((blockIdx.x * 2LL + 1) * kTileRows + rl) * 8, d + 8);
    bf16 *t = Dt + (b >> 3) * (kOutPad * 8) + (b & 7);
#pragma unroll
    for (int n = 0; n < kOutPad; n++) t[n * 8] = __float2bfloat16_rn(d[n]);
    __shared__ float s[kOut + 1][4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n <= kOut; n++) {
        float v = (n < kOut) ? d[n] : l;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) s[n][w] = v;
    }
    __syncthreads();
    if (threadIdx.x <= kOut) {
        const float v = s[threadIdx.x][0] + s[threadIdx.x][1] + s[threadIdx.x][2] + s[threadIdx.x][3];
        if (threadIdx.x < kOut) bpart[blockIdx.x * (long long)kOut + threadIdx.x] = v;
        else lpart[blockIdx.x] = v;
    }
}

// ---------------------------------------------------------------------------
// One training pass (gather, forward, loss, backward, weight gradients) in one kernel.
//
// The pass was a chain of 10 kernels that handed BF16 operands, their transposed copies and the
// activation derivatives to each other through HBM and spent their time in the epilogues' 2-byte and
// strided stores and per-column shuffle sums: 156 us for a batch of 65536 (17-64-64-8), where the
// products themselves are a few microseconds of tensor time (batch of 65536: an Adam step 206 us then,
// 52 us now, 41 of them in this kernel).  Here a persistent block takes
// 128-row tiles through the whole pass: the activations stay in shared memory as the operands of the
// next product, the pre-activations stay in tensor memory for the backward pass, and the weight
// gradients accumulate in tensor memory over a split of the batch.  Only the sampled rows are read and
// one weight gradient per split and the bias and loss sums of each tile are written.  Bound by the
// latency of its chain of products and epilogues: four warpgroups share a tile, each with 16 of its
// columns, and the next tile's rows are in flight.
//
// The order of the FP32 sums is the kernel chain's, so that a training run gives the same numbers by
// either: through the rounding of the weights to BF16 another grouping (every 148th tile in a block)
// moved the loss of 40 steps by 2.9e-5.  A split is split_rows() consecutive rows, one accumulation in the tensor core;
// k_adam adds the splits in order; bias and loss sums are per tile (32 rows by a fixed tree, then the
// four warps in order) and added in tile order.
//
// Shared-memory operands are blocked K-major as in nn_umma.cuh.  The transposed operands (reduction
// over the tile's 128 rows) hold kHid rows; as the A operand of an M = 128 product their rows kHid..127
// are whatever follows in shared memory, and so are the tensor-memory lanes that no one reads.
constexpr int kTrainBlocks = 148;
constexpr int kTrainThreads = 512, kParts = kTrainThreads / kTileRows;
constexpr int kTrainX = kInPad * kTileRows * 2, kTrainH = kHid * kTileRows * 2, kTrainD = kOutPad * kTileRows * 2;
constexpr int train_weights() {  // bytes of the forward and backward weight operands
    int b = 0;
    for (int l = 0; l < kNL; l++) b += layer_k(l) * layer_n(l) * 2 * (l > 0 ? 2 : 1);
    return b;
}
constexpr int kTrainRed = kNL * (kTrainThreads / 32) * 16 * 4;  // column sums: [layer][warp][16]
constexpr int kTrainSmem = 2 * kTrainX + (2 + kNHid) * kTrainH + 2 * kTrainD + train_weights() + kTrainRed + 1024;
constexpr int kTrainCols = (kNHid + 1) * kHid + kOutPad + kOutPad + (kNHid - 1) * kHid + kInPad;  // tensor-memory columns
// the shapes it is built for (default 17-64-64-8: 114 KB, 320 columns); others train by the kernel chain
constexpr bool kTrainFused = kHid <= 64 && kTrainSmem <= 227 * 1024 && kTrainCols <= 512;

struct TrainArgs {
    const float *xs, *ts;
    long long ns, rows, first;
    int random;
    unsigned long long seed;
    const Scaling *sc;
    const bf16 *Wt[kNL], *Wn[kNL];
    const float *b[kNL];
    int split_tiles;  // row tiles of a split: 4 or 1
    float *part;      // [split][parameters] weight gradients (the biases' places stay unused)
    float *db[kNL];   // [tile] bias gradients, kTileRows apart (kOut: output layer)
    float *lpart;     // [tile] loss sums
    int *err;
    unsigned long long wait_ns;  // bound of a wait
};

// column sums over a warp: lane L returns the sum over all lanes of v[L >> 1] (each exchange
// halves the columns a lane still carries)
__device__ __forceinline__ float warp_column_sum16(float v[16], int lane) {
#pragma unroll
    for (int w = 8, o = 16; w > 0; w >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < w; q++) {
            const float keep = up ? v[q + w] : v[q], send = up ? v[q] : v[q + w];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// D (+)= A B^T over ksteps K = 16 steps; A's row count fixes its chunk stride
__device__ __forceinline__ void mma_run(uint32_t d, const void *a, int arows, const void *b, int n, int ksteps, int acc) {
    const unsigned al = arows * 16, bl = n * 16;
    for (int s = 0; s < ksteps; s++)
        mma_bf16(d, sdesc((const char *)a + (size_t)s * 2 * al, al, 128), sdesc((const char *)b + (size_t)s * 2 * bl, bl, 128),
                 idesc_bf16(kTileRows, n), s > 0 || acc);
}

// the second wait of a block whose wait ran out: out of line, it is 1% of the kernel's time otherwise
__device__ __noinline__ void drain(uint64_t *bar, unsigned parity) { mbar_wait(bar, parity); }

__global__ void __launch_bounds__(kTrainThreads, 1) k_train(const __grid_constant__ TrainArgs g) {
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char *at = sm;
    auto take = [&](int bytes) { unsigned char *p = at; at += bytes; return (bf16 *)p; };
    bf16 *Xn = take(kTrainX), *Xt = take(kTrainX);
    bf16 *Hn = take(kTrainH), *Dt = take(kTrainH), *Ht[kNHid];  // Hn also holds the backward pass's deltas
    for (int l = 0; l < kNHid; l++) Ht[l] = take(kTrainH);
    bf16 *On = take(kTrainD), *Ot = take(kTrainD), *Wt[kNL], *Wn[kNL];
    for (int l = 0; l < kNL; l++) {
        Wt[l] = take(layer_k(l) * layer_n(l) * 2);
        Wn[l] = l > 0 ? take(layer_k(l) * layer_n(l) * 2) : nullptr;
    }
    float *red = (float *)take(kTrainRed);  // [layer][16 warps][16 columns], past the operands for M = 128 reads
    uint64_t *bar = (uint64_t *)take(1024);
    uint32_t *tslot = (uint32_t *)(bar + 1);
    int *stop = (int *)(bar + 2);  // [phase]: a wait ran out in the product before one of this phase
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rl = tid & (kTileRows - 1), part = tid / kTileRows;  // row of the tile, and 16 columns of a layer
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        stop[0] = stop[1] = 0;
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    for (int l = 0; l < kNL; l++) {
        const int n16 = layer_k(l) * layer_n(l) / 8;
        for (int q = tid; q < n16; q += kTrainThreads) {
            ((uint4 *)Wt[l])[q] = ((const uint4 *)g.Wt[l])[q];
            if (l > 0) ((uint4 *)Wn[l])[q] = ((const uint4 *)g.Wn[l])[q];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *tslot;
    // tensor-memory columns: pre-activations, outputs, backward accumulator, weight gradients
    const uint32_t zcol = tm, ocol = tm + kNHid * kHid, acol = ocol + kOutPad, gout = acol + kHid, ghid = gout + kOutPad;
    auto gcol = [&](int l) { return l == kNHid ? gout : l == 0 ? ghid + (kNHid - 1) * kHid : ghid + (l - 1) * kHid; };
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;

    unsigned phase = 0;
    bool late = false;  // a wait of this thread ran out
    // Make this tile's operands visible, have thread 0 issue the products, and wait for them.  Once a wait
    // has run out in any thread, all of them get false here and nothing more is issued; that thread waits a
    // second time first, so that no product outlives the operands, the tensor memory or the block.  The
    // word they read was written before the barrier and is not written again before the next one.
    auto products = [&](auto issue) {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (*(volatile int *)(stop + phase)) return false;
        if (tid == 0) {
            tc_fence_after();
            issue();
            mma_commit(bar);
        }
        if (!mbar_wait(bar, phase, g.wait_ns)) {
            late = true;
            stop[phase ^ 1] = 1;
            drain(bar, phase);
        }
        phase ^= 1;
        tc_fence_after();
        return true;
    };
    const long long tiles = g.rows / kTileRows;
    // this thread's 8 of the 32 padded input columns; the last part has only padding and takes the targets
    const int x0 = part * 8;
    float mu[8], isd[8], px[8], pt[kOut];
    const bool targets = part == kParts - 1;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        mu[q] = x0 + q < kIn ? g.sc->xmu[x0 + q] : 0.0f;
        isd[q] = x0 + q < kIn ? g.sc->xisd[x0 + q] : 0.0f;
    }
    auto fetch = [&](long long tile) {
        const long long b = tile * kTileRows + rl;
        const long long idx = g.random ? (long long)(mix64(g.seed ^ (unsigned long long)b * 0xD1B54A32D192ED03ull) % (unsigned long long)g.ns)
                                       : g.first + b;
        const bool in = idx < g.ns;
#pragma unroll
        for (int q = 0; q < 8; q++) px[q] = in && x0 + q < kIn ? g.xs[idx * kIn + x0 + q] : 0.0f;
#pragma unroll
        for (int q = 0; q < kOut; q++) pt[q] = in && targets ? g.ts[idx * kOut + q] : 0.0f;
    };
    // the block's tiles: those of the splits blockIdx.x, blockIdx.x + gridDim.x, ..., each split's in order
    long long tile = blockIdx.x * (long long)g.split_tiles;
    const int last = g.split_tiles - 1;
    fetch(tile);
    // this warp's sums of 16 columns of layer l (a bias's gradient; in the output layer also the loss)
    auto put_sums = [&](int l, float v[16]) {
        const float s = warp_column_sum16(v, lane);
        if (!(lane & 1)) red[(l * (kTrainThreads / 32) + warp) * 16 + (lane >> 1)] = s;
    };
    // 16 values of this row (columns 16 part ..) as operands of the next product and, transposed, of a gradient
    auto put = [&](const float v[16], bf16 *normal, bf16 *transposed) {
        if (normal) {
            store_bf16x8(normal + ((part * 2) * kTileRows + rl) * 8, v);
            store_bf16x8(normal + ((part * 2 + 1) * kTileRows + rl) * 8, v + 8);
        }
        bf16 *t = transposed + ((rl >> 3) * kHid + part * 16) * 8 + (rl & 7);
#pragma unroll
        for (int q = 0; q < 16; q++) t[q * 8] = __float2bfloat16_rn(v[q]);
    };
    const bool hidden = part * 16 < kHid;  // this part has columns of a hidden layer
    bool begun = false;  // the accumulators hold earlier tiles of this split
    auto pass = [&]() {  // this tile; false, to all threads alike, when a wait ran out
        const bool ends = (tile & last) == last;
        const long long next = tile + 1 + (ends ? (long long)(gridDim.x - 1) * g.split_tiles : 0);
        {   // standardised inputs; zero columns past kIn
            float x[8];
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = (px[q] - mu[q]) * isd[q];
            store_bf16x8(Xn + (part * kTileRows + rl) * 8, x);
            bf16 *t = Xt + ((rl >> 3) * kInPad + x0) * 8 + (rl & 7);
#pragma unroll
            for (int q = 0; q < 8; q++) t[q * 8] = __float2bfloat16_rn(x[q]);
        }
        float tgt[kOut];
#pragma unroll
        for (int q = 0; q < kOut; q++) tgt[q] = targets ? pt[q] / g.sc->ysd[q] : 0.0f;
        if (next < tiles) fetch(next);
        // forward
#pragma unroll
        for (int l = 0; l < kNHid; l++) {
            if (!products([&] { mma_run(zcol + l * kHid, l == 0 ? Xn : Hn, kTileRows, Wt[l], kHid, layer_k(l) / 16, 0); })) return false;
            if (hidden) {
                float v[16];
                tmem_ld16(zcol + l * kHid + part * 16 + lanes, v);
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] = smelu(v[q] + __ldg(g.b[l] + part * 16 + q));
                put(v, Hn, Ht[l]);
            }
        }
        if (!products([&] { mma_run(ocol, Hn, kTileRows, Wt[kNHid], kOutPad, kHid / 16, 0); })) return false;
        if (targets) {  // mean-squared-error gradient of the outputs, sums of the loss and the output biases
            float v[16];
            tmem_ld16(ocol + lanes, v);
            const float sc = 2.0f / (float)(g.rows * kOut);
            float l = 0.0f;
#pragma unroll
            for (int q = 0; q < kOut; q++) {
                const float e = v[q] + __ldg(g.b[kNHid] + q) - tgt[q];
                v[q] = sc * e;
                l += e * e;
            }
#pragma unroll
            for (int q = kOut; q < 16; q++) v[q] = 0.0f;
            store_bf16x8(On + rl * 8, v);
            store_bf16x8(On + (kTileRows + rl) * 8, v + 8);
            bf16 *t = Ot + ((rl >> 3) * kOutPad) * 8 + (rl & 7);
#pragma unroll
            for (int q = 0; q < kOutPad; q++) t[q * 8] = __float2bfloat16_rn(v[q]);
            v[kOut] = l;
            put_sums(kNHid, v);
        }
        // backward: deltas of layer l from those of layer l + 1, and the gradient of layer l + 1's weights
#pragma unroll
        for (int l = kNHid - 1; l >= 0; l--) {
            if (!products([&] {
                if (l == kNHid - 1) {
                    mma_run(acol, On, kTileRows, Wn[l + 1], kHid, kOutPad / 16, 0);
                    mma_run(gcol(l + 1), Ht[l], kHid, Ot, kOutPad, kTileRows / 16, begun);
                } else {
                    mma_run(acol, Hn, kTileRows, Wn[l + 1], kHid, kHid / 16, 0);
                    mma_run(gcol(l + 1), Dt, kHid, Ht[l], kHid, kTileRows / 16, begun);
                }
            })) return false;
            if (hidden) {
                float v[16], z[16];
                tmem_ld16(acol + part * 16 + lanes, v);
                tmem_ld16(zcol + l * kHid + part * 16 + lanes, z);
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] *= smelu_d(z[q] + __ldg(g.b[l] + part * 16 + q));
                put(v, l > 0 ? Hn : nullptr, Dt);
                put_sums(l, v);
            }
        }
        if (!products([&] { mma_run(gcol(0), Dt, kHid, Xt, kInPad, kTileRows / 16, begun); })) return false;
        // the tile's bias gradients and loss: column sums of the four warps that hold a column
        if (tid < kNHid * kHid + kOut + 1) {
            const int l = min(tid / kHid, kNHid), n = tid - l * kHid;
            const int w0 = l == kNHid ? 4 * (kParts - 1) : (n >> 4) * 4;
            const float *r = red + (l * (kTrainThreads / 32) + w0) * 16 + (n & 15);
            const float v = r[0] + r[16] + r[32] + r[48];
            if (l < kNHid) g.db[l][tile * kTileRows + n] = v;
            else if (n < kOut) g.db[l][tile * kOut + n] = v;
            else g.lpart[tile] = v;
        }
        // the split's weight gradients in parameter order: [n][k] for the hidden layers (lane n, column
        // k) and [k][n] for the output layer
        if (ends) {
            float *out = g.part + (tile / g.split_tiles) * (long long)param_count();
            const int n = rl;
#pragma unroll
            for (int l = 0; l < kNL; l++) {
                const int cols = l == kNHid ? kOutPad : l == 0 ? kInPad : kHid;
                if (part * 16 < cols) {
                    float v[16];
                    tmem_ld16(gcol(l) + part * 16 + lanes, v);
                    if (n < kHid) {
#pragma unroll
                        for (int q = 0; q < 16; q++) {
                            const int k = part * 16 + q;
                            if (l == kNHid) {
                                if (k < kOut) out[n * kOut + k] = v[q];
                            } else if (k < real_k(l)) {
                                out[k * kHid + n] = v[q];
                            }
                        }
                    }
                }
                out += real_k(l) * real_n(l) + real_n(l);
            }
        }
        begun = !ends;
        tile = next;
        return true;
    };
    while (tile < tiles && pass()) {}
    if (late) atomicOr(g.err, NN_ERR_WAIT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tm, 512);
    }
}

struct AdamArgs {
    float *W[kNL], *b[kNL], *mW[kNL], *vW[kNL], *mb[kNL], *vb[kNL];
    const float *dw[kNL];  // weight-gradient partials
    const float *db[kNL];  // bias-gradient partials
    const float *part;     // or (not null) weight-gradient partials in parameter order
    bf16 *Wt[kNL], *Wn[kNL], *Bt[kNHid];
    int splits, tiles;
    float lr, beta1, beta2, eps, c1, c2;  // c1 = 1 - beta1^t, c2 = 1 - beta2^t
    int apply;                             // 1: Adam step; 0: only reduce the gradient; 2: only pack BF16 copies
    float *gout;                           // reduced gradients in parameter order (or null)
    const int *err;                        // the gradient pass's error word: no step from an invalid gradient
};

__host__ __device__ constexpr long long layer_params(int l) { return (long long)real_k(l) * real_n(l) + real_n(l); }

// kAdamGroup threads per real parameter load its gradient partials (kAdamStage at a time, coalesced over
// the 32 parameters of a block); the first of them adds them in order, does the Adam step on the FP32
// master and writes the BF16 copies in both operand layouts.  Bound by the 512 ordered additions of a
// bias at 65536 rows: 8 us (23 with the next stage's loads behind the additions instead of before them).
// One thread per parameter that loaded its partials itself took 41 us: a serial chain of loads on 23 blocks.
constexpr int kAdamGroup = 8, kAdamParams = 32, kAdamStage = 128;
__global__ void __launch_bounds__(kAdamGroup * kAdamParams) k_adam(AdamArgs a) {
    const int col = threadIdx.x % kAdamParams, grp = threadIdx.x / kAdamParams;
    long long t = blockIdx.x * (long long)kAdamParams + col;
    int l = 0;
    while (l < kNL && t >= layer_params(l)) { t -= layer_params(l); l++; }
    const bool have = l < kNL;
    if (!have) l = kNL - 1;
    long long off = 0;
    for (int q = 0; q < l; q++) off += layer_params(q);
    const int K = layer_k(l), N = layer_n(l), kr = real_k(l), nr = real_n(l);
    const bool is_w = t < (long long)kr * nr;
    if (a.apply == 1 && *a.err) return;
    float g = 0.0f;
    int k = 0, n = 0;
    // the face kernel's bias operand of hidden layer l < kNHid (its columns 2.. stay zero)
    auto pack_bias = [&](int nb, float b) {
        if (l < kNHid) {
            bf16 hi, lo;
            bias_split(b, hi, lo);
            a.Bt[l][blk_off(nb, 0, kBiasK, kHid)] = hi;
            a.Bt[l][blk_off(nb, 1, kBiasK, kHid)] = lo;
        }
    };
    if (a.apply == 2) {  // pack only: BF16 copies of the current masters
        if (!have || grp) return;
        if (is_w) {
            k = (int)(t / nr);
            n = (int)(t % nr);
            const float w = a.W[l][k * N + n];
            a.Wt[l][blk_off(n, k, K, N < kTileRows ? N : kTileRows)] = __float2bfloat16_rn(w);
            if (l > 0) a.Wn[l][blk_off(k, n, N, K < kTileRows ? K : kTileRows)] = __float2bfloat16_rn(w);
        } else {
            n = (int)(t - (long long)kr * nr);
            pack_bias(n, a.b[l][n]);
        }
        return;
    }
    if (is_w) {
        k = (int)(t / nr);
        n = (int)(t % nr);
    } else {
        n = (int)(t - (long long)kr * nr);
    }
    // this parameter's partials: the weight-gradient product of the chain is [n][k] for the hidden layers
    // and [k][n] for the output layer
    const float *src;
    long long step;
    if (!is_w) {
        src = a.db[l] + n;
        step = l < kNHid ? kTileRows : kOut;
    } else if (a.part) {
        src = a.part + off + t;
        step = param_count();
    } else {
        src = a.dw[l] + (l < kNHid ? n * dw_cols(l) + k : k * N + n);
        step = kTileRows * (l < kNHid ? dw_cols(l) : N);
    }
    const int count = !have ? 0 : is_w ? a.splits : a.tiles;
    const int most = __syncthreads_or(have && !is_w) ? a.tiles : a.splits;  // a batch has no more splits than tiles
    __shared__ float stage[kAdamStage][kAdamParams];
    float in[kAdamStage / kAdamGroup];  // the stage after the one that is added: in flight meanwhile
    auto load = [&](int s0) {
#pragma unroll
        for (int q = 0; q < kAdamStage / kAdamGroup; q++) {
            const int s = s0 + grp + q * kAdamGroup;
            in[q] = s < count ? src[s * step] : 0.0f;  // past the end a zero: it changes no sum that began at +0
        }
    };
    load(0);
    for (int s0 = 0; s0 < most; s0 += kAdamStage) {
#pragma unroll
        for (int q = 0; q < kAdamStage / kAdamGroup; q++) stage[grp + q * kAdamGroup][col] = in[q];
        __syncthreads();
        load(s0 + kAdamStage);
        if (grp == 0) {
#pragma unroll 32
            for (int s = 0; s < kAdamStage; s++) g += stage[s][col];
        }
        __syncthreads();
    }
    if (grp || !have) return;
    if (a.gout) a.gout[off + t] = g;
    if (!a.apply) return;
    float *p = is_w ? &a.W[l][k * N + n] : &a.b[l][n];
    float *m = is_w ? &a.mW[l][k * N + n] : &a.mb[l][n];
    float *v = is_w ? &a.vW[l][k * N + n] : &a.vb[l][n];
    const float mm = a.beta1 * *m + (1.0f - a.beta1) * g;
    const float vv = a.beta2 * *v + (1.0f - a.beta2) * g * g;
    *m = mm;
    *v = vv;
    const float w = *p - a.lr * (mm / a.c1) / (sqrtf(vv / a.c2) + a.eps);
    *p = w;
    if (is_w) {
        a.Wt[l][blk_off(n, k, K, N < kTileRows ? N : kTileRows)] = __float2bfloat16_rn(w);
        if (l > 0) a.Wn[l][blk_off(k, n, N, K < kTileRows ? K : kTileRows)] = __float2bfloat16_rn(w);
    } else {
        pack_bias(n, w);
    }
}

// input envelope and largest |target| of the sample set (ordered-integer min/max)
__device__ __forceinline__ int f2o(float f) { int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7FFFFFFF; }
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }
__global__ void k_envelope(const float *__restrict__ xs, const float *__restrict__ ts, long long ns, int *mn_, int *mx_,
                           int *ymax) {
    int lo[kIn], hi[kIn], ym = 0;
#pragma unroll
    for (int n = 0; n < kIn; n++) { lo[n] = 0x7FFFFFFF; hi[n] = (int)0x80000000; }
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < ns; s += (long long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int n = 0; n < kIn; n++) {
            const int o = f2o(xs[s * kIn + n]);
            lo[n] = min(lo[n], o);
            hi[n] = max(hi[n], o);
        }
#pragma unroll
        for (int n = 0; n < kOut; n++) ym = max(ym, f2o(fabsf(ts[s * kOut + n])));
    }
#pragma unroll
    for (int n = 0; n < kIn; n++) {
        atomicMin(&mn_[n], lo[n]);
        atomicMax(&mx_[n], hi[n]);
    }
    atomicMax(ymax, ym);
}

// sums and sums of squares of every input and output over the sample set (FP64)
__global__ void k_moments(const float *__restrict__ xs, const float *__restrict__ ts, long long ns, double *acc) {
    double a[2 * (kIn + kOut)];
#pragma unroll
    for (int n = 0; n < 2 * (kIn + kOut); n++) a[n] = 0.0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < ns; s += (long long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int n = 0; n < kIn; n++) {
            const double v = xs[s * kIn + n];
            a[n] += v;
            a[kIn + kOut + n] += v * v;
        }
#pragma unroll
        for (int n = 0; n < kOut; n++) {
            const double v = ts[s * kOut + n];
            a[kIn + n] += v;
            a[2 * kIn + kOut + n] += v * v;
        }
    }
#pragma unroll
    for (int n = 0; n < 2 * (kIn + kOut); n++) {
        double v = a[n];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(&acc[n], v);
    }
}

}  // namespace nn
}  // namespace dg

using namespace dg::nn;

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct dg_nn {
    int device = 0;
    cudaStream_t stream = nullptr;
    int *d_err = nullptr, *h_err = nullptr;  // device error word and its pinned read-back
    float *W[kNL] = {}, *b[kNL] = {}, *mW[kNL] = {}, *vW[kNL] = {}, *mb[kNL] = {}, *vb[kNL] = {};
    bf16 *Wt[kNL] = {}, *Wn[kNL] = {}, *Bt[kNHid] = {};
    float *xs = nullptr, *ts = nullptr;  // samples
    long long ns = 0, cap = 0;
    float *gx = nullptr, *gt = nullptr;  // a caller's batch of dg_nn_gradients (gcap rows, kept between calls)
    float *gh = nullptr;                 // pinned read-back of its gradient and loss sums
    long long gcap = 0;
    // batch scratch
    long long bcap = 0;
    bf16 *Xn = nullptr, *Xt = nullptr, *Hn[kNHid] = {}, *Ht[kNHid] = {}, *Dn[2] = {}, *Dt[2] = {}, *D3n = nullptr,
         *D3t = nullptr;
    float *Tb = nullptr, *Y = nullptr, *G[kNHid] = {}, *dw[kNL] = {}, *db[kNL] = {}, *lpart = nullptr, *gout = nullptr;
    float *part = nullptr;       // weight gradients of the one-kernel pass by split (param_count() each)
    long long scap = 0;          // splits that the gradient scratch holds
    long long step = 0;
    unsigned long long seed = 1;
    unsigned long long wait_ns = kWaitNs;  // bound of a wait in the one-kernel pass
    float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    Gates gates{};
    Scaling sc{};              // host copy of the standardisation
    Scaling *d_sc = nullptr;   // device copy read by the batch gather
    int trained = 0;
    std::vector<void *> allocs, scratch;
};

namespace {
int nn_fail(int code, const std::string &m) { return dg::set_error(code, m.c_str()); }
#define NN_CUDA(x)                                                                                       \
    do {                                                                                                 \
        cudaError_t e_ = (x);                                                                            \
        if (e_ != cudaSuccess) return nn_fail(DG_ERR_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
    } while (0)

int nn_alloc(dg_nn *n, void **p, size_t bytes) {
    NN_CUDA(cudaMalloc(p, bytes));
    NN_CUDA(cudaMemsetAsync(*p, 0, bytes, n->stream));
    n->allocs.push_back(*p);
    return 0;
}
template <typename X> int nn_alloc_t(dg_nn *n, X **p, size_t count) { return nn_alloc(n, (void **)p, count * sizeof(X)); }

// wait for a stream with a wall-clock bound (DG_SYNC_TIMEOUT_S, default 300 s)
int nn_bounded_sync(cudaStream_t st) {
    const char *e = std::getenv("DG_SYNC_TIMEOUT_S");
    const double limit = (e && std::atof(e) > 0) ? std::atof(e) : 300.0;
    const auto t0 = std::chrono::steady_clock::now();
    for (;;) {
        const cudaError_t q = cudaStreamQuery(st);
        if (q == cudaSuccess) return 0;
        if (q != cudaErrorNotReady) return nn_fail(DG_ERR_CUDA, std::string("stream: ") + cudaGetErrorString(q));
        const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (el > limit) return nn_fail(DG_ERR_TIMEOUT, "device work did not finish within DG_SYNC_TIMEOUT_S");
        if (el > 0.002)  // poll without a sleep at first: a sleep of any length takes about 55 us
            std::this_thread::sleep_for(std::chrono::microseconds(el < 0.01 ? 5 : 100));
    }
}

int nn_sync(dg_nn *n) {
    NN_CUDA(cudaMemcpyAsync(n->h_err, n->d_err, sizeof(int), cudaMemcpyDeviceToHost, n->stream));
    if (int rc = nn_bounded_sync(n->stream)) return rc;
    const int err = *n->h_err;
    if (err) return nn_fail(DG_ERR_STATE, "network kernel gave up waiting on a tensor-core transfer (error bits " +
                                              std::to_string(err) + ")");
    return 0;
}

int scratch_alloc(dg_nn *n, void **p, size_t bytes) {
    NN_CUDA(cudaMalloc(p, bytes));
    NN_CUDA(cudaMemsetAsync(*p, 0, bytes, n->stream));
    n->scratch.push_back(*p);
    return 0;
}
template <typename X> int scratch_t(dg_nn *n, X **p, size_t count) { return scratch_alloc(n, (void **)p, count * sizeof(X)); }

// rows of one weight-gradient partial: 512 where they divide the batch, else one row tile
long long split_rows(long long rows) { return rows % 512 == 0 ? 512 : kTileRows; }

// batch work arrays for `rows` rows (reallocated when a larger batch, or one of more splits, comes)
int ensure_batch(dg_nn *n, long long rows) {
    const long long R = std::max(rows, n->bcap), tiles = R / kTileRows;
    const long long splits = std::max(rows / split_rows(rows), n->scap);
    if (R <= n->bcap && splits <= n->scap) return 0;
    NN_CUDA(cudaStreamSynchronize(n->stream));
    for (void *p : n->scratch) cudaFree(p);
    n->scratch.clear();
    n->bcap = n->scap = 0;
    int rc;
    if ((rc = scratch_t(n, &n->Xn, R * kInPad)) || (rc = scratch_t(n, &n->Xt, R * kInPad)) ||
        (rc = scratch_t(n, &n->Tb, R * kOut)) || (rc = scratch_t(n, &n->Y, R * kOut)) ||
        (rc = scratch_t(n, &n->lpart, tiles)) || (rc = scratch_t(n, &n->gout, dg_nn_param_count())))
        return rc;
    for (int l = 0; l < kNL; l++)
        if ((rc = scratch_t(n, &n->db[l], tiles * kTileRows))) return rc;
    for (int l = 0; l < kNHid; l++)
        if ((rc = scratch_t(n, &n->Hn[l], R * kHid)) || (rc = scratch_t(n, &n->Ht[l], R * kHidT)) ||
            (rc = scratch_t(n, &n->G[l], R * kHid)))
            return rc;
    if constexpr (kTrainFused) {
        if ((rc = scratch_t(n, &n->part, splits * param_count()))) return rc;
    } else {  // the gradient operands of the kernel chain
        if ((rc = scratch_t(n, &n->D3n, R * kOutPad)) || (rc = scratch_t(n, &n->D3t, R * kOutPad))) return rc;
        for (int q = 0; q < 2; q++)
            if ((rc = scratch_t(n, &n->Dn[q], R * kHid)) || (rc = scratch_t(n, &n->Dt[q], R * kHidT))) return rc;
        for (int l = 0; l < kNL; l++)
            if ((rc = scratch_t(n, &n->dw[l], splits * kTileRows * kHidT))) return rc;
    }
    n->bcap = R;
    n->scap = splits;
    return 0;
}

template <int MODE, int N>
int launch_gemm(dg_nn *n, const GemmArgs &g, long long grid) {
    NN_CUDA(cudaFuncSetAttribute(k_gemm<MODE, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
    k_gemm<MODE, N><<<(unsigned)grid, 128, kGemmSmem, n->stream>>>(g);
    NN_CUDA(cudaGetLastError());
    return 0;
}

// forward pass over `rows` gathered rows (a multiple of 128)
int forward(dg_nn *n, long long rows) {
    const long long tiles = rows / kTileRows;
    int rc;
    for (int l = 0; l < kNHid; l++) {
        GemmArgs g{};
        g.A = (l == 0) ? n->Xn : n->Hn[l - 1];
        g.B = n->Wt[l];
        g.C = layer_k(l);
        g.bias = n->b[l];
        g.Hn = n->Hn[l];
        g.Ht = n->Ht[l];
        g.G = n->G[l];
        g.rows = rows;
        g.err = n->d_err;
        if ((rc = launch_gemm<M_FWD_HID, kHid>(n, g, tiles))) return rc;
    }
    GemmArgs g{};
    g.A = n->Hn[kNHid - 1];
    g.B = n->Wt[kNHid];
    g.C = kHid;
    g.bias = n->b[kNHid];
    g.Y = n->Y;
    g.rows = rows;
    g.err = n->d_err;
    return launch_gemm<M_FWD_OUT, kOutPad>(n, g, tiles);
}

// loss gradient and backward pass; leaves weight/bias gradient partials in dw/db (a template: the
// kernels of the chain are built only for the shapes that use it)
template <int = 0>
int backward(dg_nn *n, long long rows, long long valid) {
    const long long tiles = rows / kTileRows;
    const int csplit = (int)split_rows(rows);
    const long long splits = rows / csplit;
    k_loss<<<(unsigned)tiles, 128, 0, n->stream>>>(n->Y, n->Tb, rows, valid, n->D3n, n->D3t, n->lpart, n->db[kNHid]);
    NN_CUDA(cudaGetLastError());
    int rc;
    {   // output layer: dW[k][n] = sum_b Ht[k][b] Dt[n][b] over the last hidden layer's activations
        GemmArgs g{};
        g.A = n->Ht[kNHid - 1]; g.B = n->D3t; g.C = csplit; g.part = n->dw[kNHid]; g.rows = rows; g.err = n->d_err;
        if ((rc = launch_gemm<M_DW, kOutPad>(n, g, splits))) return rc;
    }
    const bf16 *dn = n->D3n;
    int cdn = kOutPad;
    for (int l = kNHid - 1; l >= 0; l--) {
        bf16 *on = n->Dn[l & 1], *ot = n->Dt[l & 1];
        {   // dZ_l = (dZ_{l+1} W_{l+1}^T) * f'(Z_l), bias partials of layer l
            GemmArgs g{};
            g.A = dn; g.B = n->Wn[l + 1]; g.C = cdn; g.G = n->G[l]; g.Hn = on; g.Ht = ot; g.part = n->db[l];
            g.rows = rows; g.err = n->d_err;
            if ((rc = launch_gemm<M_BWD_HID, kHid>(n, g, tiles))) return rc;
        }
        {   // dW_l[n][k] = sum_b dZt_l[n][b] Ht_{l-1}[k][b]
            GemmArgs g{};
            g.A = ot; g.B = (l == 0) ? n->Xt : n->Ht[l - 1]; g.C = csplit; g.part = n->dw[l]; g.rows = rows; g.err = n->d_err;
            if (l == 0) rc = launch_gemm<M_DW, kInPad>(n, g, splits);
            else rc = launch_gemm<M_DW, kHidT>(n, g, splits);
            if (rc) return rc;
        }
        dn = on;
        cdn = kHid;
    }
    return 0;
}

int adam(dg_nn *n, long long rows, float lr, int apply, float *gout) {
    AdamArgs a{};
    for (int l = 0; l < kNL; l++) {
        a.W[l] = n->W[l]; a.b[l] = n->b[l]; a.mW[l] = n->mW[l]; a.vW[l] = n->vW[l]; a.mb[l] = n->mb[l];
        a.vb[l] = n->vb[l]; a.dw[l] = n->dw[l]; a.db[l] = n->db[l]; a.Wt[l] = n->Wt[l]; a.Wn[l] = n->Wn[l];
        if (l < kNHid) a.Bt[l] = n->Bt[l];
    }
    a.splits = (int)(rows / split_rows(rows));
    a.tiles = (int)(rows / kTileRows);
    if (kTrainFused) a.part = n->part;
    a.lr = lr; a.beta1 = n->beta1; a.beta2 = n->beta2; a.eps = n->eps;
    if (apply == 1) n->step++;
    const double t = (double)(n->step > 0 ? n->step : 1);
    a.c1 = (float)(1.0 - std::pow((double)n->beta1, t));
    a.c2 = (float)(1.0 - std::pow((double)n->beta2, t));
    a.apply = apply;
    a.gout = gout;
    a.err = n->d_err;
    const long long np = dg_nn_param_count();
    k_adam<<<(unsigned)((np + kAdamParams - 1) / kAdamParams), kAdamGroup * kAdamParams, 0, n->stream>>>(a);
    NN_CUDA(cudaGetLastError());
    return 0;
}

int gather(dg_nn *n, long long rows, int random, long long first) {
    k_gather<<<(unsigned)((rows + 127) / 128), 128, 0, n->stream>>>(n->xs, n->ts, n->ns, rows, random,
                                                                      n->seed + 0x9E37ull * (unsigned long long)n->step,
                                                                      first, n->d_sc, n->Xn, n->Xt, n->Tb);
    NN_CUDA(cudaGetLastError());
    return 0;
}

// gradient and loss sums of one batch (rows drawn at random, or in order from the first sample)
int gradient_pass(dg_nn *n, long long rows, int random) {
    if constexpr (kTrainFused) {
        TrainArgs g{};
        g.xs = n->xs; g.ts = n->ts; g.ns = n->ns; g.rows = rows; g.first = 0; g.random = random;
        g.seed = n->seed + 0x9E37ull * (unsigned long long)n->step;
        g.sc = n->d_sc;
        for (int l = 0; l < kNL; l++) { g.Wt[l] = n->Wt[l]; g.Wn[l] = n->Wn[l]; g.b[l] = n->b[l]; }
        for (int l = 0; l < kNL; l++) g.db[l] = n->db[l];
        g.split_tiles = (int)(split_rows(rows) / kTileRows);
        g.part = n->part; g.lpart = n->lpart; g.err = n->d_err; g.wait_ns = n->wait_ns;
        NN_CUDA(cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem));
        // a block per split, at most one per SM (its tensor memory)
        const long long splits = rows / split_rows(rows);
        k_train<<<(unsigned)std::min<long long>(splits, kTrainBlocks), kTrainThreads, kTrainSmem, n->stream>>>(g);
        NN_CUDA(cudaGetLastError());
        return 0;
    } else {
        int rc;
        if ((rc = gather(n, rows, random, 0)) || (rc = forward(n, rows))) return rc;
        return backward<>(n, rows, rows);
    }
}

// write the BF16 operand copies of the FP32 masters
int pack_weights(dg_nn *n) {
    return adam(n, kTileRows, 0.0f, 2, nullptr);
}

int check_batch(long long batch) {
    if (batch < kTileRows || batch % kTileRows) return nn_fail(DG_ERR_ARG, "batch must be a positive multiple of 128");
    return 0;
}
}  // namespace

namespace {
// one block waiting on an mbarrier with the library's bounded wait; one thread arrives on it
// (arrive = 1) or nothing does (arrive = 0), so the wait completes or runs out its time
__global__ void k_wait_selftest(int arrive, int *err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (arrive && threadIdx.x == 0) mbar_arrive(&bar);
    if (!mbar_wait(&bar, 0)) atomicOr(err, NN_ERR_WAIT);
}
}  // namespace

extern "C" {

int dg_wait_selftest(int device, int arrive, double *seconds) {
    if (cudaSetDevice(device) != cudaSuccess) return nn_fail(DG_ERR_NODEVICE, "no CUDA device");
    int *d_err = nullptr;
    NN_CUDA(cudaMalloc(&d_err, sizeof(int)));
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
        cudaFree(d_err);
        return nn_fail(DG_ERR_CUDA, "cudaStreamCreate failed");
    }
    int rc = 0, err = 0;
    const auto t0 = std::chrono::steady_clock::now();
    if (cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess) rc = nn_fail(DG_ERR_CUDA, "cudaMemsetAsync failed");
    if (!rc) {
        k_wait_selftest<<<1, 32, 0, st>>>(arrive, d_err);
        const cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) rc = nn_fail(DG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(le));
    }
    if (!rc) rc = nn_bounded_sync(st);
    if (!rc && cudaMemcpy(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = nn_fail(DG_ERR_CUDA, "cudaMemcpy failed");
    if (seconds) *seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    cudaStreamDestroy(st);
    cudaFree(d_err);
    if (rc) return rc;
    if (err) return nn_fail(DG_ERR_TIMEOUT, "an mbarrier wait ran out of its time bound");
    return DG_OK;
}

long long dg_nn_param_count(void) {
    long long n = 0;
    for (int l = 0; l < kNL; l++) n += layer_params(l);
    return n;
}

int dg_nn_shape(int *width, int *depth) {
    if (width) *width = kHid;
    if (depth) *depth = kNHid;
    return DG_OK;
}

int dg_nn_create(int device, unsigned long long seed, dg_nn **out) {
    if (!out) return nn_fail(DG_ERR_ARG, "null output pointer");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return nn_fail(DG_ERR_NODEVICE, "no CUDA device");
    if (device < 0 || device >= ndev) return nn_fail(DG_ERR_ARG, "device index out of range");
    NN_CUDA(cudaSetDevice(device));
    dg_nn *n = new dg_nn();
    n->device = device;
    n->seed = seed;
    int rc = 0;
    auto bail = [&](int code) { dg_nn_destroy(n); return code; };
    if (cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(nn_fail(DG_ERR_CUDA, "stream creation failed"));
    if ((rc = nn_alloc_t(n, &n->d_err, 1))) return bail(rc);
    if (cudaMallocHost((void **)&n->h_err, sizeof(int)) != cudaSuccess) return bail(nn_fail(DG_ERR_NOMEM, "cudaMallocHost failed"));
    // He-normal initial weights on the host from the seed (Box-Muller over splitmix64)
    unsigned long long st = seed * 0x9E3779B97F4A7C15ull + 12345u;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        unsigned long long z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    for (int l = 0; l < kNL; l++) {
        const int K = layer_k(l), N = layer_n(l);
        if ((rc = nn_alloc_t(n, &n->W[l], (size_t)K * N)) || (rc = nn_alloc_t(n, &n->b[l], N)) ||
            (rc = nn_alloc_t(n, &n->mW[l], (size_t)K * N)) || (rc = nn_alloc_t(n, &n->vW[l], (size_t)K * N)) ||
            (rc = nn_alloc_t(n, &n->mb[l], N)) || (rc = nn_alloc_t(n, &n->vb[l], N)) ||
            (rc = nn_alloc_t(n, &n->Wt[l], (size_t)K * N)) || (rc = nn_alloc_t(n, &n->Wn[l], (size_t)K * N)) ||
            (l < kNHid && (rc = nn_alloc_t(n, &n->Bt[l], (size_t)kBiasK * kHid))))
            return bail(rc);
        std::vector<float> w((size_t)K * N, 0.0f);
        const double sd = std::sqrt(2.0 / real_k(l)) * (l == kNHid ? 0.1 : 1.0);
        for (int k = 0; k < real_k(l); k++)
            for (int j = 0; j < real_n(l); j++) {
                const double u1 = next(), u2 = next();
                w[(size_t)k * N + j] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
            }
        if (cudaMemcpyAsync(n->W[l], w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice, n->stream) != cudaSuccess)
            return bail(nn_fail(DG_ERR_CUDA, "weight upload failed"));
    }
    for (int q = 0; q < kIn; q++) { n->sc.xmu[q] = 0.0f; n->sc.xsd[q] = 1.0f; n->sc.xisd[q] = 1.0f; }
    for (int q = 0; q < kOut; q++) n->sc.ysd[q] = 1.0f;
    if ((rc = nn_alloc_t(n, &n->d_sc, 1))) return bail(rc);
    if (cudaMemcpyAsync(n->d_sc, &n->sc, sizeof(Scaling), cudaMemcpyHostToDevice, n->stream) != cudaSuccess)
        return bail(nn_fail(DG_ERR_CUDA, "scaling upload failed"));
    for (int q = 0; q < kIn; q++) { n->gates.xmin[q] = -1e30f; n->gates.xmax[q] = 1e30f; }
    n->gates.ymax = 1e30f;
    n->gates.jump = 0.1f;
    n->gates.compress = 0.1f;
    n->gates.margin = 0.0f;
    if ((rc = pack_weights(n)) || (rc = nn_sync(n))) return bail(rc);
    *out = n;
    return DG_OK;
}

int dg_nn_destroy(dg_nn *n) {
    if (!n) return DG_OK;
    cudaSetDevice(n->device);
    if (n->stream) cudaStreamSynchronize(n->stream);
    for (void *p : n->allocs) cudaFree(p);
    for (void *p : n->scratch) cudaFree(p);
    if (n->xs) cudaFree(n->xs);
    if (n->ts) cudaFree(n->ts);
    if (n->gx) cudaFree(n->gx);
    if (n->gt) cudaFree(n->gt);
    if (n->gh) cudaFreeHost(n->gh);
    if (n->h_err) cudaFreeHost(n->h_err);
    if (n->stream) cudaStreamDestroy(n->stream);
    delete n;
    return DG_OK;
}

int dg_nn_set_samples(dg_nn *n, const float *x, const float *t, long long count) {
    if (!n || !x || !t || count <= 0) return nn_fail(DG_ERR_ARG, "bad sample arguments");
    NN_CUDA(cudaSetDevice(n->device));
    int rc;
    if ((rc = dg_nn_reserve_samples(n, count))) return rc;
    NN_CUDA(cudaMemcpyAsync(n->xs, x, (size_t)count * kIn * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    NN_CUDA(cudaMemcpyAsync(n->ts, t, (size_t)count * kOut * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    n->ns = count;
    return nn_sync(n);
}

int dg_nn_reserve_samples(dg_nn *n, long long count) {
    if (!n || count <= 0) return nn_fail(DG_ERR_ARG, "bad sample count");
    if (count <= n->cap) return DG_OK;
    NN_CUDA(cudaSetDevice(n->device));
    NN_CUDA(cudaStreamSynchronize(n->stream));
    float *xs = nullptr, *ts = nullptr;
    NN_CUDA(cudaMalloc(&xs, (size_t)count * kIn * sizeof(float)));
    if (cudaMalloc(&ts, (size_t)count * kOut * sizeof(float)) != cudaSuccess) {
        cudaFree(xs);
        return nn_fail(DG_ERR_CUDA, "out of device memory for samples");
    }
    if (n->ns) {
        cudaMemcpyAsync(xs, n->xs, (size_t)n->ns * kIn * sizeof(float), cudaMemcpyDeviceToDevice, n->stream);
        cudaMemcpyAsync(ts, n->ts, (size_t)n->ns * kOut * sizeof(float), cudaMemcpyDeviceToDevice, n->stream);
        NN_CUDA(cudaStreamSynchronize(n->stream));
    }
    if (n->xs) cudaFree(n->xs);
    if (n->ts) cudaFree(n->ts);
    n->xs = xs;
    n->ts = ts;
    n->cap = count;
    return DG_OK;
}

long long dg_nn_sample_count(const dg_nn *n) { return n ? n->ns : 0; }

int dg_nn_samples_copy(dg_nn *n, long long first, long long count, float *x, float *t) {
    if (!n || first < 0 || count < 0 || first + count > n->ns || (!x && !t)) return nn_fail(DG_ERR_ARG, "bad sample range");
    NN_CUDA(cudaSetDevice(n->device));
    if (x) NN_CUDA(cudaMemcpyAsync(x, n->xs + first * kIn, (size_t)count * kIn * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    if (t) NN_CUDA(cudaMemcpyAsync(t, n->ts + first * kOut, (size_t)count * kOut * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    return nn_sync(n);
}

int dg_nn_train(dg_nn *n, int steps, int batch, float lr, float *loss_out) {
    if (!n || steps < 0) return nn_fail(DG_ERR_ARG, "bad training arguments");
    if (n->ns <= 0) return nn_fail(DG_ERR_ARG, "no samples");
    int rc;
    if ((rc = check_batch(batch))) return rc;
    NN_CUDA(cudaSetDevice(n->device));
    if ((rc = ensure_batch(n, batch))) return rc;
    for (int s = 0; s < steps; s++) {
        if ((rc = gradient_pass(n, batch, 1)) || (rc = adam(n, batch, lr, 1, nullptr))) return rc;
    }
    if (loss_out) {
        std::vector<float> lp((size_t)batch / kTileRows);
        NN_CUDA(cudaMemcpyAsync(lp.data(), n->lpart, lp.size() * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
        if ((rc = nn_sync(n))) return rc;
        double l = 0.0;
        for (float v : lp) l += v;
        *loss_out = (float)(l / ((double)batch * kOut));
    }
    n->trained = 1;
    return nn_sync(n);
}

int dg_nn_gradients(dg_nn *n, const float *x, const float *t, int batch, float *loss, float *grad) {
    if (!n || !x || !t || !grad) return nn_fail(DG_ERR_ARG, "bad gradient arguments");
    int rc;
    if ((rc = check_batch(batch))) return rc;
    NN_CUDA(cudaSetDevice(n->device));
    if ((rc = ensure_batch(n, batch))) return rc;
    // a private sample set holding exactly this batch, in order, in buffers kept for the next call
    // (allocating and freeing them was two thirds of a call on 16384 rows)
    const long long np = dg_nn_param_count(), nl = batch / kTileRows;
    if (batch > n->gcap) {
        NN_CUDA(cudaStreamSynchronize(n->stream));
        if (n->gx) cudaFree(n->gx);
        if (n->gt) cudaFree(n->gt);
        if (n->gh) cudaFreeHost(n->gh);
        n->gx = n->gt = n->gh = nullptr;
        n->gcap = 0;
        if (cudaMalloc(&n->gx, (size_t)batch * kIn * sizeof(float)) != cudaSuccess ||
            cudaMalloc(&n->gt, (size_t)batch * kOut * sizeof(float)) != cudaSuccess ||
            cudaMallocHost(&n->gh, (size_t)(np + nl) * sizeof(float)) != cudaSuccess) {
            cudaGetLastError();
            return nn_fail(DG_ERR_CUDA, "out of memory for the gradient batch");
        }
        n->gcap = batch;
    }
    NN_CUDA(cudaMemcpyAsync(n->gx, x, (size_t)batch * kIn * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    NN_CUDA(cudaMemcpyAsync(n->gt, t, (size_t)batch * kOut * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    float *xs = n->xs, *ts = n->ts;
    const long long ns = n->ns;
    n->xs = n->gx; n->ts = n->gt; n->ns = batch;
    rc = gradient_pass(n, batch, 0);
    if (!rc) rc = adam(n, batch, 0.0f, 0, n->gout);
    n->xs = xs; n->ts = ts; n->ns = ns;
    if (rc) {
        nn_bounded_sync(n->stream);
        return rc;
    }
    NN_CUDA(cudaMemcpyAsync(n->gh, n->gout, (size_t)np * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    NN_CUDA(cudaMemcpyAsync(n->gh + np, n->lpart, (size_t)nl * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    if ((rc = nn_sync(n))) return rc;
    std::memcpy(grad, n->gh, (size_t)np * sizeof(float));
    if (loss) {
        double l = 0.0;
        for (long long q = 0; q < nl; q++) l += n->gh[np + q];
        *loss = (float)(l / ((double)batch * kOut));
    }
    return DG_OK;
}

int dg_nn_forward(dg_nn *n, const float *x, long long count, float *y) {
    if (!n || !x || !y || count <= 0) return nn_fail(DG_ERR_ARG, "bad forward arguments");
    NN_CUDA(cudaSetDevice(n->device));
    const long long rows = n->bcap ? n->bcap : 16384;
    int rc;
    if ((rc = ensure_batch(n, rows))) return rc;
    float *xs = n->xs, *ts = n->ts;
    const long long ns = n->ns, cap = n->cap;
    n->xs = nullptr; n->ts = nullptr; n->ns = 0; n->cap = 0;
    std::vector<float> zeros((size_t)count * kOut, 0.0f);
    rc = dg_nn_set_samples(n, x, zeros.data(), count);
    for (long long first = 0; !rc && first < count; first += rows) {
        const long long m = std::min(rows, count - first);
        const long long r = (m + kTileRows - 1) / kTileRows * kTileRows;
        if (!rc) rc = gather(n, r, 0, first);
        if (!rc) rc = forward(n, r);
        if (!rc && cudaMemcpyAsync(y + first * kOut, n->Y, (size_t)m * kOut * sizeof(float), cudaMemcpyDeviceToHost,
                                   n->stream) != cudaSuccess)
            rc = nn_fail(DG_ERR_CUDA, "output read-back failed");
        if (!rc) rc = nn_sync(n);
        for (long long r2 = 0; !rc && r2 < m; r2++)
            for (int c = 0; c < kOut; c++) y[(first + r2) * kOut + c] *= n->sc.ysd[c];
    }
    if (n->xs) cudaFree(n->xs);
    if (n->ts) cudaFree(n->ts);
    n->xs = xs; n->ts = ts; n->ns = ns; n->cap = cap;
    return rc;
}

int dg_nn_get_params(dg_nn *n, float *host, long long count) {
    if (!n || !host || count < dg_nn_param_count()) return nn_fail(DG_ERR_ARG, "bad parameter buffer");
    NN_CUDA(cudaSetDevice(n->device));
    long long off = 0;
    for (int l = 0; l < kNL; l++) {
        const int K = layer_k(l), N = layer_n(l);
        std::vector<float> w((size_t)K * N), b(N);
        NN_CUDA(cudaMemcpyAsync(w.data(), n->W[l], w.size() * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
        NN_CUDA(cudaMemcpyAsync(b.data(), n->b[l], b.size() * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
        NN_CUDA(cudaStreamSynchronize(n->stream));
        for (int k = 0; k < real_k(l); k++)
            for (int j = 0; j < real_n(l); j++) host[off++] = w[(size_t)k * N + j];
        for (int j = 0; j < real_n(l); j++) host[off++] = b[j];
    }
    return DG_OK;
}

int dg_nn_set_params(dg_nn *n, const float *host, long long count) {
    if (!n || !host || count < dg_nn_param_count()) return nn_fail(DG_ERR_ARG, "bad parameter buffer");
    NN_CUDA(cudaSetDevice(n->device));
    long long off = 0;
    for (int l = 0; l < kNL; l++) {
        const int K = layer_k(l), N = layer_n(l);
        std::vector<float> w((size_t)K * N, 0.0f), b(N, 0.0f);
        for (int k = 0; k < real_k(l); k++)
            for (int j = 0; j < real_n(l); j++) w[(size_t)k * N + j] = host[off++];
        for (int j = 0; j < real_n(l); j++) b[j] = host[off++];
        NN_CUDA(cudaMemcpyAsync(n->W[l], w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice, n->stream));
        NN_CUDA(cudaMemcpyAsync(n->b[l], b.data(), b.size() * sizeof(float), cudaMemcpyHostToDevice, n->stream));
        NN_CUDA(cudaStreamSynchronize(n->stream));
    }
    int rc = pack_weights(n);
    return rc ? rc : nn_sync(n);
}

// input envelope and output bound of the current samples become the confidence gate
int dg_nn_fit_envelope(dg_nn *n, float margin) {
    if (!n || n->ns <= 0) return nn_fail(DG_ERR_ARG, "no samples");
    NN_CUDA(cudaSetDevice(n->device));
    int *d = nullptr;
    NN_CUDA(cudaMalloc(&d, (2 * kIn + 1) * sizeof(int)));
    std::vector<int> init(2 * kIn + 1);
    for (int q = 0; q < kIn; q++) { init[q] = 0x7FFFFFFF; init[kIn + q] = (int)0x80000000; }
    init[2 * kIn] = 0;
    cudaMemcpyAsync(d, init.data(), init.size() * sizeof(int), cudaMemcpyHostToDevice, n->stream);
    k_envelope<<<296, 256, 0, n->stream>>>(n->xs, n->ts, n->ns, d, d + kIn, d + 2 * kIn);
    std::vector<int> h(2 * kIn + 1);
    cudaMemcpyAsync(h.data(), d, h.size() * sizeof(int), cudaMemcpyDeviceToHost, n->stream);
    const cudaError_t e = cudaStreamSynchronize(n->stream);
    cudaFree(d);
    if (e != cudaSuccess) return nn_fail(DG_ERR_CUDA, cudaGetErrorString(e));
    auto o2f_h = [](int i) { int j = i >= 0 ? i : i ^ 0x7FFFFFFF; float f; std::memcpy(&f, &j, 4); return f; };
    for (int q = 0; q < kIn; q++) { n->gates.xmin[q] = o2f_h(h[q]); n->gates.xmax[q] = o2f_h(h[kIn + q]); }
    n->gates.ymax = o2f_h(h[2 * kIn]);
    n->gates.margin = margin;
    return DG_OK;
}

int dg_nn_fit_scaling(dg_nn *n) {
    if (!n || n->ns <= 0) return nn_fail(DG_ERR_ARG, "no samples");
    NN_CUDA(cudaSetDevice(n->device));
    const int na = 2 * (kIn + kOut);
    double *d = nullptr;
    NN_CUDA(cudaMalloc(&d, na * sizeof(double)));
    cudaMemsetAsync(d, 0, na * sizeof(double), n->stream);
    k_moments<<<296, 128, 0, n->stream>>>(n->xs, n->ts, n->ns, d);
    std::vector<double> h(na);
    cudaMemcpyAsync(h.data(), d, na * sizeof(double), cudaMemcpyDeviceToHost, n->stream);
    const cudaError_t e = cudaStreamSynchronize(n->stream);
    cudaFree(d);
    if (e != cudaSuccess) return nn_fail(DG_ERR_CUDA, cudaGetErrorString(e));
    const double N = (double)n->ns;
    for (int q = 0; q < kIn; q++) {
        const double mu = h[q] / N, var = std::max(h[kIn + kOut + q] / N - mu * mu, 0.0);
        n->sc.xmu[q] = (float)mu;
        n->sc.xsd[q] = var > 1e-12 ? (float)std::sqrt(var) : 1.0f;  // a constant input stays at zero
        n->sc.xisd[q] = 1.0f / n->sc.xsd[q];
    }
    for (int q = 0; q < kOut; q++) {
        const double rms = std::sqrt(h[2 * kIn + kOut + q] / N);
        n->sc.ysd[q] = rms > 1e-30 ? (float)rms : 1.0f;
    }
    NN_CUDA(cudaMemcpyAsync(n->d_sc, &n->sc, sizeof(Scaling), cudaMemcpyHostToDevice, n->stream));
    return nn_sync(n);
}

int dg_nn_wait_bound(dg_nn *n, double seconds) {
    if (!n || !(seconds >= 0.0) || seconds > 60.0) return nn_fail(DG_ERR_ARG, "bad wait bound");
    n->wait_ns = (unsigned long long)(seconds * 1e9);
    return DG_OK;
}

int dg_nn_set_gates(dg_nn *n, float jump, float compress) {
    if (!n || !(jump >= 0.0f) || !(compress >= 0.0f)) return nn_fail(DG_ERR_ARG, "bad gate thresholds");
    n->gates.jump = jump;
    n->gates.compress = compress;
    return DG_OK;
}

}  // extern "C"

// ---- internal accessors for the step kernels (nn_host.h) ---------------------------
int dg_nn_view(const dg_nn *n, dg::nn::NetView *v) {
    if (!n) return DG_ERR_ARG;
    for (int l = 0; l < kNL; l++) { v->wt[l] = n->Wt[l]; v->b[l] = n->b[l]; }
    for (int l = 0; l < kNHid; l++) v->bt[l] = n->Bt[l];
    v->gates = n->gates;
    for (int q = 0; q < kIn; q++) {
        const float w = n->gates.margin * (n->gates.xmax[q] - n->gates.xmin[q]);
        v->xlo[q] = n->gates.xmin[q] - w;
        v->xhi[q] = n->gates.xmax[q] + w;
    }
    v->sc = n->sc;
    return DG_OK;
}
int dg_nn_device(const dg_nn *n) { return n ? n->device : -1; }
float *dg_nn_sample_x(dg_nn *n) { return n->xs; }
float *dg_nn_sample_t(dg_nn *n) { return n->ts; }
void dg_nn_set_count(dg_nn *n, long long c) { n->ns = c; }
