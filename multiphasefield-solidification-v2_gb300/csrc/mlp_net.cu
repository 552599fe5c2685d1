// mlp_net.cu -- the surrogate network as three kernels: the forward pass, the
// chain of input gradients, and all weight gradients.
//
// The network is 16 -> 256 -> 256 -> 256 -> 2 with SiLU (surrogate.py).  A
// row of its input needs no other row until the weight gradients, so a CTA
// takes 128 rows through all layers: the activations stay in shared memory as
// the next layer's A operand, the accumulator in tensor memory, and only the
// weights stream in from L2.  One launch per layer kept every activation going
// through L2 and HBM and, in the backward pass, gathered transposed operands
// element by element; here the transposed operands are MN-major tiles of the
// arrays as they lie in memory.
//
// Rounding points are those of the layer-by-layer GEMMs (mlp.cu): BF16
// activations and output gradients, FP32 accumulation with the reduction in
// ascending order, FP32 bias, SiLU and its derivative.
//
// CTA of the two chains, 320 threads:
//   warps 0-7  epilogue: tcgen05.ld of 32 rows x 128 columns each, bias and
//              SiLU (or the derivative), BF16 back into the A tile
//   warp 8     one lane loads the weights by TMA, 16 KB a chunk (64 of the
//              reduction x 128 outputs), into a ring of two
//   warp 9     one lane issues tcgen05.mma
// Two CTAs share an SM (256 tensor-memory columns and 110 KB each): the
// epilogue of one runs under the loads and MMAs of the other.  The epilogue's
// exponentials and reciprocals (2 per value, 16 a clock per SM) would take 21
// us for 65,536 rows; the weights' way from L2, 128 KB per tile and layer with
// 64 KB in flight per SM, adds the rest.  Measured on GB300: forward of 65,536
// rows 125 -> 41 us (one CTA per SM with a ring of 8 chunks: 66 us); an
// optimiser step on 512 rows, call to call, 843 -> 83 to 91 us (each kernel by itself
// with cold caches: forward 24 us, gradient chain 36, weight gradients 9).  For few rows the time is that of one tile, about 5
// us a layer, and the ring of 8 hides the weights.
// Every wait is bounded; a wait that runs out ends the CTA's work as in mlp.cu:
// the issued MMAs and copies are waited for (bounded), the outputs of the
// CTA's rows become NaN, MPF3D_DEV_GEMM_ABORT is set, and tensor memory is
// freed unless an MMA may still run.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "mpf3d.h"
#include "mpf3d_internal.h"
#include "tcgen05.cuh"

namespace mpf3d {
namespace mlp {
namespace net {

using namespace tc5;
using namespace tc5::tma;

constexpr int ROWS = 128, HID = 256, IN = 16, OUT = 2;
constexpr int EPI_WARPS = 8, THREADS = 32 * (EPI_WARPS + 2);
// parameter offsets (FP32 master copy and BF16 copy alike): W0 b0 W1 b1 W2 b2 W3 b3
__host__ __device__ constexpr int off_w(int l) { return l == 0 ? 0 : HID * IN + HID + (l - 1) * (HID * HID + HID); }
__host__ __device__ constexpr int off_b(int l) {
    return off_w(l) + (l == 0 ? HID * IN : (l < 3 ? HID * HID : OUT * HID));
}

constexpr int CHUNK = 128 * 128;  // 128 rows of 128 bytes
constexpr int ATOM = ROWS * 128;  // 64 columns of the A tile
constexpr int SM_A = 0, SM_X = 4 * ATOM, SM_B0 = SM_X + ROWS * IN * 2, SM_RING = SM_B0 + HID * IN * 2;
template <int STAGES>
constexpr int SM_BARS = SM_RING + STAGES * CHUNK;
template <int STAGES>
constexpr int SMEM = SM_BARS<STAGES> + 256 + 1024;  // and the alignment to 1024
enum { A_READY = 0, ACC_FULL, DRAIN, FULL };        // then EMPTY = FULL + STAGES

struct Abort {
    int flag, undrained;
};

// bounded wait that stops once any role of the CTA gave up
struct Waiter {
    uint64_t *bars;
    volatile Abort *ab;
    __device__ __forceinline__ uint32_t bar(int i) const { return smem_addr(bars + i); }
    __device__ __forceinline__ bool operator()(int i, uint32_t count) const {
        if (ab->flag) return false;
        if (mbar_wait(bar(i), count & 1u)) return true;
        ab->flag = 1;
        return false;
    }
};

__device__ __forceinline__ void bar_init(uint64_t *b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// silu_grad without the division's branch per value: 1 / d for d >= 1 by one
// Newton step from the approximate reciprocal (FMA residual), within one unit in the
// last place; near overflow of d the approximation itself
__device__ __forceinline__ float silu_slope(float z) {
    const float d = 1.0f + __expf(-z);
    const float r = __fdividef(1.0f, d);
    const float newton = fmaf(r, fmaf(-d, r, 1.0f), r);
    const float s = d < 1e37f ? newton : r;
    return s * (1.0f + z * (1.0f - s));
}

// 16 consecutive BF16 columns of row r into the swizzled A tile
__device__ __forceinline__ void store_a(uint8_t *sA, int r, int col, const uint32_t (&w)[8]) {
    uint8_t *row = sA + (col >> 6) * ATOM + r * 128;
    const int ch = (col & 63) >> 3;
    *reinterpret_cast<uint4 *>(row + ((ch ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4 *>(row + (((ch + 1) ^ (r & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
}

// 16 columns x 32 lanes: the column sums, column (lane >> 1) on lane pairs
__device__ __forceinline__ float column_sums(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1) {
        const bool up = (lane & (2 * n)) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

struct Args {
    const uint16_t *__restrict__ x;     // forward: input rows
    const uint16_t *__restrict__ w0;    // BF16 W0 (forward) or W3 (backward)
    const float *__restrict__ w;        // forward: FP32 parameters (biases)
    const float *__restrict__ dout;     // backward: gradient of the outputs
    // pre-activations [3][64][M][4]: four columns of consecutive rows are
    // consecutive, as the lanes of a warp write and read them
    float *__restrict__ Z;
    float *__restrict__ out;            // forward: outputs
    uint16_t *__restrict__ dz3;         // backward: dZ3 [M][8]
    float *__restrict__ partial;        // backward: [4 tiles][3][256] column sums
};
struct Maps {
    // forward W1, W2 (boxes of 64 x 128, K-major), W3 (64 x 16); backward W2,
    // W1 (boxes of 64 x 64, read as MN-major B)
    CUtensorMap w[3];
    CUtensorMap keep[3];  // A tiles to memory by layer: Y (forward) or dZ (backward), boxes of 64 x 128
};

// The two chains.  BACK false: layers 0..3 forward, KEEP: with what the
// backward pass needs.  BACK true: dZ3 -> dZ2 -> dZ1 -> dZ0.  The A tiles go to
// memory by TMA store.
template <bool BACK, bool KEEP, int STAGES>
__global__ void __launch_bounds__(THREADS, STAGES == 2 ? 2 : 1) chain_kernel(const __grid_constant__ Maps maps, int M,
                                                                             const Args G,
                                                                             int32_t *__restrict__ err) {
    constexpr int EMPTY = FULL + STAGES, BARS = FULL + 2 * STAGES;
    extern __shared__ uint8_t raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + SM_BARS<STAGES>);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + BARS);
    Abort *ab = reinterpret_cast<Abort *>(tslot + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = (M + ROWS - 1) / ROWS;
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            bar_init(bars + FULL + i, 1);
            bar_init(bars + EMPTY + i, 1);
        }
        bar_init(bars + A_READY, EPI_WARPS);
        bar_init(bars + ACC_FULL, 1);
        bar_init(bars + DRAIN, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        ab->flag = ab->undrained = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;\n" ::"r"(smem_addr(tslot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // B of the first product, 256 x 16 in K-major core matrices: W0, or W3
    // transposed with its two rows padded to 16
    if (threadIdx.x < HID) {
        const int r = threadIdx.x;
        uint4 v[2];
        if (BACK) {
            v[0] = make_uint4((uint32_t)__ldg(G.w0 + r) | ((uint32_t)__ldg(G.w0 + HID + r) << 16), 0u, 0u, 0u);
            v[1] = make_uint4(0u, 0u, 0u, 0u);
        } else {
            v[0] = __ldg(reinterpret_cast<const uint4 *>(G.w0 + r * IN));
            v[1] = __ldg(reinterpret_cast<const uint4 *>(G.w0 + r * IN) + 1);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
            *reinterpret_cast<uint4 *>(smem + SM_B0 + (r >> 3) * 256 + c * 128 + (r & 7) * 16) = v[c];
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const Waiter wait{bars, ab};
    constexpr int PER_TILE = BACK ? 16 : 17;  // chunks
    const uint32_t mine = blockIdx.x < tiles ? (uint32_t)((tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) : 0u;

    if (warp == EPI_WARPS) {
        if (lane == 0) {
            uint32_t c = 0;
            for (const uint32_t end = mine * PER_TILE; c < end; ++c) {
                const int s = c % STAGES, i = c % PER_TILE;
                if (!wait(EMPTY + s, c / STAGES + 1u)) break;
                const uint32_t dst = smem_addr(smem + SM_RING + s * CHUNK), full = wait.bar(FULL + s);
                const CUtensorMap *map = &maps.w[i >> 3];
                const int nh = (i & 7) >> 2, j = i & 3;
                if (i == 16) {
                    arrive_expect(full, 4 * 16 * 128);
                    for (int q = 0; q < 4; ++q) tma_load(dst + q * 16 * 128, map, q * 64, 0, full);
                } else {
                    arrive_expect(full, CHUNK);
                    if (BACK) {
                        tma_load(dst, map, nh * 128, j * 64, full);
                        tma_load(dst + CHUNK / 2, map, nh * 128 + 64, j * 64, full);
                    } else {
                        tma_load(dst, map, j * 64, nh * 128, full);
                    }
                }
            }
            if (ab->flag) {  // the copies in flight must land before the CTA can go away
                bool landed = true;
                for (uint32_t q = c > STAGES ? c - STAGES : 0; q < c; ++q)
                    landed = mbar_wait(wait.bar(FULL + q % STAGES), (q / STAGES) & 1u) && landed;
                if (!landed) atomicExch(&ab->undrained, 1);
            }
        }
    } else if (warp == EPI_WARPS + 1) {
        if (lane == 0) {
            const uint32_t a0 = smem_addr(smem + SM_A);
            uint32_t c = 0, ready = 0;
            bool issued = false;
            for (uint32_t t = 0; t < mine; ++t) {
                if (!wait(A_READY, ready++)) break;
                fence_after();
                umma(tmem, smem_desc(smem_addr(smem + SM_X), 128u, 256u), smem_desc(smem_addr(smem + SM_B0), 128u, 256u),
                     instr_desc(ROWS, HID), 0u);
                issued = true;
                commit(wait.bar(ACC_FULL));
                bool ok = true;
                for (int layer = 0; layer < 3 && ok; ++layer) {
                    ok = wait(A_READY, ready++);
                    if (!ok) break;
                    fence_after();
                    if (KEEP) {
                        const int m0 = ((int)blockIdx.x + (int)t * (int)gridDim.x) * ROWS;
                        for (int q = 0; q < 4; ++q)
                            tma_store(&maps.keep[BACK ? 2 - layer : layer], a0 + q * ATOM, q * 64, m0);
                        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                    }
                    for (int i = 0; i < (layer < 2 ? 8 : (BACK ? 0 : 1)) && ok; ++i, ++c) {
                        const int s = c % STAGES, nh = i >> 2, j = i & 3;
                        ok = wait(FULL + s, c / STAGES);
                        if (!ok) break;
                        fence_after();
                        const uint32_t b0 = smem_addr(smem + SM_RING + s * CHUNK);
                        if (layer == 2) {
                            for (int q = 0; q < 4; ++q)
                                for (int ks = 0; ks < 4; ++ks)
                                    umma(tmem, sw128_desc(a0 + q * ATOM + 32u * ks),
                                         sw128_desc(b0 + q * 16 * 128 + 32u * ks), instr_desc(ROWS, 16),
                                         q > 0 || ks > 0);
                        } else {
                            for (int ks = 0; ks < 4; ++ks) {
                                const uint64_t bd = BACK ? sw128_desc_mn(b0 + 2048u * ks, CHUNK / 2)
                                                         : sw128_desc(b0 + 32u * ks);
                                umma(tmem + nh * 128, sw128_desc(a0 + j * ATOM + 32u * ks), bd,
                                     instr_desc(ROWS, 128) | (BACK ? B_MN : 0u), j > 0 || ks > 0);
                            }
                        }
                        commit(wait.bar(EMPTY + s));
                    }
                    // the tile may be written again once it has been read
                    if (KEEP) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    if (ok) commit(wait.bar(ACC_FULL));
                }
                if (!ok) break;
            }
            if (KEEP) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
            if (ab->flag && issued) {
                // the MMAs issued before the abort must finish before the
                // tensor memory is freed and the CTA leaves
                commit(wait.bar(DRAIN));
                if (!mbar_wait(wait.bar(DRAIN), 0)) atomicExch(&ab->undrained, 1);
            }
        }
    } else {
        const int q = warp & 3, half = warp >> 2, r = q * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        uint32_t full = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int m0 = tile * ROWS, m = m0 + r;
            {  // A of the first product: 8 of a row's 16 columns per thread
                const int xr = threadIdx.x >> 1, c = threadIdx.x & 1;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (m0 + xr < M) {
                    if (!BACK) {
                        v = __ldg(reinterpret_cast<const uint4 *>(G.x + (int64_t)(m0 + xr) * IN) + c);
                    } else if (c == 0) {
                        const float2 d = __ldg(reinterpret_cast<const float2 *>(G.dout) + m0 + xr);
                        v.x = pack_bf16(d.x, d.y);
                        reinterpret_cast<uint4 *>(G.dz3)[m0 + xr] = v;
                    }
                }
                *reinterpret_cast<uint4 *>(smem + SM_X + (xr >> 3) * 256 + c * 128 + (xr & 7) * 16) = v;
            }
            auto ready = [&] {  // this warp's part of A is written, its accumulator columns are read
                fence_before();
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive(wait.bar(A_READY));
            };
            ready();
            bool ok = true;
            for (int st = 0; st < 3 && ok; ++st) {
                const int layer = BACK ? 2 - st : st;
                // backward: pre-activations are loaded one block of columns
                // ahead, the first under the product that is waited for
                float4 zn[4];
                auto load_z = [&](int col) {
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        zn[v] = m < M ? __ldg(reinterpret_cast<const float4 *>(G.Z) +
                                              ((int64_t)layer * (HID / 4) + col / 4 + v) * M + m)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                };
                if (BACK) load_z(half * 128);
                ok = __all_sync(0xffffffffu, wait(ACC_FULL, full++));
                if (!ok) break;
                fence_after();
                const float4 *bias = BACK ? nullptr : reinterpret_cast<const float4 *>(G.w + off_b(layer));
                float4 *zq = reinterpret_cast<float4 *>(G.Z) + (int64_t)layer * (HID / 4) * M + m;
                const int c0 = half * 128;
                uint32_t acc[2][16];
                tmem_ld16_async(lanes + (uint32_t)c0, acc[0]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // the next columns' load runs under these columns' arithmetic
                    const int col = c0 + 16 * i;
                    float z[16], y[16];
                    if (BACK) {
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            z[4 * v] = zn[v].x; z[4 * v + 1] = zn[v].y; z[4 * v + 2] = zn[v].z; z[4 * v + 3] = zn[v].w;
                        }
                        if (i < 7) load_z(col + 16);
                    }
                    uint32_t (&r16)[16] = acc[i & 1];
                    tmem_ld_wait(r16);
                    if (i < 7) tmem_ld16_async(lanes + (uint32_t)(col + 16), acc[(i + 1) & 1]);
                    if (BACK) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)  // 0 in rows past the end: their accumulators are 0
                            y[j] = __uint_as_float(r16[j]) * silu_slope(z[j]);
                    } else {
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            const float4 f = __ldg(bias + col / 4 + v);
                            z[4 * v] = __uint_as_float(r16[4 * v]) + f.x;
                            z[4 * v + 1] = __uint_as_float(r16[4 * v + 1]) + f.y;
                            z[4 * v + 2] = __uint_as_float(r16[4 * v + 2]) + f.z;
                            z[4 * v + 3] = __uint_as_float(r16[4 * v + 3]) + f.w;
                            if (KEEP && m < M)
                                zq[(int64_t)(col / 4 + v) * M] = make_float4(z[4 * v], z[4 * v + 1], z[4 * v + 2], z[4 * v + 3]);
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) y[j] = silu(z[j]);
                    }
                    uint32_t w[8];
#pragma unroll
                    for (int v = 0; v < 8; ++v) w[v] = pack_bf16(y[2 * v], y[2 * v + 1]);
                    store_a(smem + SM_A, r, col, w);
                    if (BACK) {
                        const float s = column_sums(y);
                        if ((lane & 1) == 0)
                            G.partial[((int64_t)(4 * tile + q) * 3 + layer) * HID + col + (lane >> 1)] = s;
                    }
                }
                ready();
            }
            if (ok) {  // the output layer: 2 of 16 accumulator columns; the backward chain's last tile is stored
                ok = __all_sync(0xffffffffu, wait(ACC_FULL, full++));
                if (ok) {
                    fence_after();
                    if (!BACK && half == 0) {
                        uint32_t acc[16];
                        tmem_ld16(lanes, acc);
                        if (m < M)
                            reinterpret_cast<float2 *>(G.out)[m] =
                                make_float2(__uint_as_float(acc[0]) + __ldg(G.w + off_b(3)),
                                            __uint_as_float(acc[1]) + __ldg(G.w + off_b(3) + 1));
                    }
                }
            }
            if (!ok) break;
        }
    }
    fence_before();
    __syncwarp();  // the single-lane roles rejoin their warps before the block barrier
    __syncthreads();
    fence_after();
    if (ab->flag) {
        if (threadIdx.x == 0 && err) atomicOr(err, MPF3D_DEV_GEMM_ABORT);
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int m = tile * ROWS + (int)threadIdx.x;
            if (threadIdx.x >= ROWS || m >= M) continue;
            if (!BACK) reinterpret_cast<float2 *>(G.out)[m] = make_float2(NAN, NAN);
            else G.dz3[8 * (int64_t)m] = G.dz3[8 * (int64_t)m + 1] = 0x7fc0;
        }
    }
    if (warp == 0 && !*(volatile int *)&ab->undrained)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;\n" ::"r"(tmem) : "memory");
}

// All weight gradients dW[n][k] = sum_m dZ[m][n] H[m][k] and bias gradients.
// One CTA per tile of 128 n x 64 k of one layer: layers 1 and 2 have 2 x 4
// tiles, layer 0 two (its 16 columns), layer 3 four (its 2 rows).  dZ and H are
// read as they lie in memory: boxes of 64 columns x 64 rows m are MN-major
// operands of a reduction over m.
namespace grad {

constexpr int TILES = 22, STAGES = 4, BOX = 64 * 128, CHUNK = 3 * BOX, THREADS = 192;
constexpr int SMEM = STAGES * CHUNK + 256 + 1024;
enum { FULL = 0, EMPTY = STAGES, ACC_FULL = 2 * STAGES, DRAIN, BARS };

struct GradMaps {
    CUtensorMap dz[4], h[4];
};

__global__ void __launch_bounds__(THREADS) grad_kernel(const __grid_constant__ GradMaps maps, int M, int partials,
                                                       const float *__restrict__ partial,
                                                       const float *__restrict__ dout, float *__restrict__ g,
                                                       int live_inputs, int32_t *__restrict__ err) {
    extern __shared__ uint8_t raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * CHUNK);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + BARS);
    Abort *ab = reinterpret_cast<Abort *>(tslot + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int layer = t < 8 ? 1 : (t < 16 ? 2 : (t < 18 ? 0 : 3));
    const int nb = t < 16 ? (t & 7) >> 2 : (t < 18 ? t - 16 : 0);
    const int kb = t < 16 ? t & 3 : (t < 18 ? 0 : t - 18);
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            bar_init(bars + FULL + i, 1);
            bar_init(bars + EMPTY + i, 1);
        }
        bar_init(bars + ACC_FULL, 1);
        bar_init(bars + DRAIN, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        ab->flag = ab->undrained = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;\n" ::"r"(smem_addr(tslot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const Waiter wait{bars, ab};
    const uint32_t chunks = (uint32_t)(M + 63) / 64;
    if (warp == 4) {
        if (lane == 0) {
            uint32_t c = 0;
            for (; c < chunks; ++c) {
                const int s = c % STAGES;
                if (!wait(EMPTY + s, c / STAGES + 1u)) break;
                const uint32_t dst = smem_addr(smem + s * CHUNK), full = wait.bar(FULL + s);
                arrive_expect(full, CHUNK);
                tma_load(dst, &maps.dz[layer], nb * 128, (int)c * 64, full);
                tma_load(dst + BOX, &maps.dz[layer], nb * 128 + 64, (int)c * 64, full);
                tma_load(dst + 2 * BOX, &maps.h[layer], kb * 64, (int)c * 64, full);
            }
            if (ab->flag) {
                bool landed = true;
                for (uint32_t q = c > STAGES ? c - STAGES : 0; q < c; ++q)
                    landed = mbar_wait(wait.bar(FULL + q % STAGES), (q / STAGES) & 1u) && landed;
                if (!landed) atomicExch(&ab->undrained, 1);
            }
        }
    } else if (warp == 5) {
        if (lane == 0) {
            bool issued = false;
            uint32_t c = 0;
            for (; c < chunks; ++c) {
                const int s = c % STAGES;
                if (!wait(FULL + s, c / STAGES)) break;
                fence_after();
                const uint32_t a = smem_addr(smem + s * CHUNK);
                for (int ks = 0; ks < 4; ++ks)
                    umma(tmem, sw128_desc_mn(a + 2048u * ks, BOX), sw128_desc_mn(a + 2 * BOX + 2048u * ks, BOX),
                         instr_desc(128, 64) | A_MN | B_MN, c > 0 || ks > 0);
                issued = true;
                commit(wait.bar(EMPTY + s));
            }
            if (c == chunks) commit(wait.bar(ACC_FULL));
            if (ab->flag && issued) {
                commit(wait.bar(DRAIN));
                if (!mbar_wait(wait.bar(DRAIN), 0)) atomicExch(&ab->undrained, 1);
            }
        }
    } else {
        // bias gradients meanwhile: the chain's column sums, tile by tile
        const int n = nb * 128 + warp * 32 + lane;
        if (kb == 0 && layer < 3) {
            float s = 0.0f;
            for (int p = 0; p < partials; ++p) s += __ldg(partial + ((int64_t)p * 3 + layer) * HID + n);
            g[off_b(layer) + n] = s;
        } else if (kb == 0 && warp < OUT) {
            float s = 0.0f;
            for (int m = lane; m < M; m += 32) s += __ldg(dout + (int64_t)m * OUT + warp);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) g[off_b(3) + warp] = s;
        }
        const bool ok = __all_sync(0xffffffffu, wait(ACC_FULL, 0u));
        fence_after();
        const int K = layer == 0 ? IN : HID, rows = layer == 3 ? OUT : HID;
        float *o = g + off_w(layer) + (int64_t)n * K + kb * 64;
        for (int c0 = 0; c0 < (K < 64 ? K : 64); c0 += 16) {
            uint32_t acc[16];
            if (ok) tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
            if (n >= rows) continue;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                float f[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    f[j] = ok ? __uint_as_float(acc[4 * v + j]) : NAN;
                    // the padded input columns carry no parameters
                    if (layer == 0 && c0 + 4 * v + j >= live_inputs) f[j] = 0.0f;
                }
                reinterpret_cast<float4 *>(o + c0)[v] = make_float4(f[0], f[1], f[2], f[3]);
            }
        }
    }
    fence_before();
    __syncwarp();
    __syncthreads();
    fence_after();
    if (ab->flag && threadIdx.x == 0 && err) atomicOr(err, MPF3D_DEV_GEMM_ABORT);
    if (warp == 0 && !*(volatile int *)&ab->undrained)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;\n" ::"r"(tmem) : "memory");
}

}  // namespace grad

}  // namespace net
}  // namespace mlp
}  // namespace mpf3d

using namespace mpf3d::mlp;

namespace {

int sms() {
    int dev = 0, n = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

// Two CTAs per SM with a ring of 2 chunks; where the rows make at most one tile
// per SM, one CTA with a ring of 8, a layer's whole weights, which then load
// under the previous epilogue.
template <bool BACK, bool KEEP>
int launch_chain(const net::Maps &maps, int M, const net::Args &G, int32_t *err, cudaStream_t s) {
    using namespace net;
    const int tiles = (M + ROWS - 1) / ROWS, n = sms();
    const bool deep = tiles <= n;
    const int smem = deep ? SMEM<8> : SMEM<2>;
    const auto kernel = deep ? chain_kernel<BACK, KEEP, 8> : chain_kernel<BACK, KEEP, 2>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return MPF3D_ERR_CUDA;
    kernel<<<tiles < 2 * n ? tiles : 2 * n, THREADS, smem, s>>>(maps, M, G, err);
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

}  // namespace

extern "C" int mpf3d_mlp_forward(int M, const uint16_t *x, const uint16_t *w16, const float *w, float *Z, uint16_t *Y,
                                 float *out, int32_t *err, void *stream) {
    using namespace net;
    if (M <= 0 || !x || !w16 || !w || !out || (Z == nullptr) != (Y == nullptr) || !aligned16(x) || !aligned16(w16) ||
        !aligned16(w) || !aligned16(Z) || !aligned16(Y) || ((uintptr_t)out & 7u) != 0)
        return MPF3D_ERR_ARG;
    Maps maps;
    bool ok = make_map(&maps.w[0], w16 + off_w(1), HID, HID, HID, 128) &&
              make_map(&maps.w[1], w16 + off_w(2), HID, HID, HID, 128) &&
              make_map(&maps.w[2], w16 + off_w(3), OUT, HID, HID, 16);
    for (int l = 0; l < 3 && ok && Y; ++l) ok = make_map(&maps.keep[l], Y + (int64_t)l * M * HID, M, HID, HID, ROWS);
    if (!ok) return MPF3D_ERR_CUDA;
    const Args A{x, w16, w, nullptr, Z, out, nullptr, nullptr};
    return Y ? launch_chain<false, true>(maps, M, A, err, (cudaStream_t)stream)
             : launch_chain<false, false>(maps, M, A, err, (cudaStream_t)stream);
}

extern "C" int mpf3d_mlp_backward(int M, const uint16_t *x, const uint16_t *w16, const float *Z, const uint16_t *Y,
                                  const float *dout, uint16_t *dz, float *partial, float *g, int live_inputs,
                                  int32_t *err, void *stream) {
    using namespace net;
    if (M <= 0 || !x || !w16 || !Z || !Y || !dout || !dz || !partial || !g || live_inputs < 0 || live_inputs > IN ||
        !aligned16(x) || !aligned16(w16) || !aligned16(Z) || !aligned16(Y) || !aligned16(dz) || !aligned16(g) ||
        ((uintptr_t)dout & 7u) != 0)
        return MPF3D_ERR_ARG;
    const int64_t layer = (int64_t)M * HID;
    uint16_t *dz3 = dz + 3 * layer;
    Maps chain;
    grad::GradMaps maps;
    bool ok = make_map(&chain.w[0], w16 + off_w(2), HID, HID, HID, 64) &&
              make_map(&chain.w[1], w16 + off_w(1), HID, HID, HID, 64);
    for (int l = 0; l < 3 && ok; ++l) ok = make_map(&chain.keep[l], dz + l * layer, M, HID, HID, ROWS);
    for (int l = 0; l < 4 && ok; ++l) {
        ok = l < 3 ? make_map(&maps.dz[l], dz + l * layer, M, HID, HID, 64) : make_map(&maps.dz[l], dz3, M, 8, 8, 64);
        ok = ok && (l == 0 ? make_map(&maps.h[l], x, M, IN, IN, 64)
                           : make_map(&maps.h[l], Y + (l - 1) * layer, M, HID, HID, 64));
    }
    if (!ok) return MPF3D_ERR_CUDA;
    const Args A{nullptr, w16 + off_w(3), nullptr, dout, const_cast<float *>(Z), nullptr, dz3, partial};
    const int rc = launch_chain<true, true>(chain, M, A, err, (cudaStream_t)stream);
    if (rc != MPF3D_OK) return rc;
    if (cudaFuncSetAttribute(grad::grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, grad::SMEM) != cudaSuccess)
        return MPF3D_ERR_CUDA;
    grad::grad_kernel<<<grad::TILES, grad::THREADS, grad::SMEM, (cudaStream_t)stream>>>(
        maps, M, 4 * ((M + ROWS - 1) / ROWS), partial, dout, g, live_inputs, err);
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}
