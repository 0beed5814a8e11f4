// The surrogate network's kernels (include/pacuda_surrogate.h): BF16 tensor-core products on
// tcgen05 with FP32 accumulators in tensor memory, operands streamed into shared memory by bulk
// copies, training by hand-written forward/backward/Adam kernels, and a fused inference kernel.
//
// Data in global memory are kept as "tile images" (umma.cuh): an A image (the M side of a
// product) is row tiles of 128 rows, each as K/64 tiles of 128 x 64 BF16 values, 16 KB each; a B
// image (the N side) is one row tile of N rows (64 or 256) as K/64 tiles of N x 64 values. One
// bulk copy moves one tile into shared memory in the layout the tensor cores read.
//
// Training (one batch of B points, B a multiple of 128), three launches:
//   chain_kernel   per 128 points, the forward products H_l = silu(H_{l-1} W_l^T + b_l), the output
//                  layer and dZ4, then the backward products dZ_{l-1} = (dZ_l W_l) silu'(Z_{l-1}),
//                  each layer's operand in shared memory; it writes X, H_l and dZ_l as A images
//   dw_kernel      dW_l = dZ_l^T H_{l-1}, split over the batch: the same images with K along the
//                  points (MN-major operands, so no transposed copy of them is written or read)
//   update_kernel  the sums of the partials in a fixed order, Adam and the weight images
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/pacuda_surrogate.h"
#include "phase.cuh"
#include "umma.cuh"

using namespace pacuda::umma;

namespace {

constexpr int WIDTH = PACUDA_SG_WIDTH;  // hidden width
constexpr int IN = PACUDA_SG_MAX_INPUTS;  // the first layer's K (inputs padded with zeros)
constexpr uint32_t TILE_A = 128 * 128;    // bytes of a 128-row x 64 BF16 tile
constexpr long long WAIT_CYCLES = 2000000000LL;  // a bounded wait gives up after about a second

// parameter offsets (FP32 vector)
constexpr size_t P_W1 = 0, P_B1 = P_W1 + (size_t)WIDTH * IN, P_W2 = P_B1 + WIDTH, P_B2 = P_W2 + (size_t)WIDTH * WIDTH,
                 P_W3 = P_B2 + WIDTH, P_B3 = P_W3 + (size_t)WIDTH * WIDTH, P_W4 = P_B3 + WIDTH,
                 P_B4 = P_W4 + (size_t)WIDTH * WIDTH, P_W5 = P_B4 + WIDTH, P_B5 = P_W5 + WIDTH, P_COUNT = P_B5 + 1;
__host__ __device__ constexpr size_t bias_at(int layer) {
    return layer == 0 ? P_B1 : layer == 1 ? P_B2 : layer == 2 ? P_B3 : layer == 3 ? P_B4 : P_B5;
}

// the forward weight images: W1 (1 tile of 256 x 64), W2..W4 (4 tiles each), contiguous
constexpr size_t WIMG_L1 = 0, WIMG_L2 = WIMG_L1 + 1 * 256 * 128, WIMG_L3 = WIMG_L2 + 4 * 256 * 128,
                 WIMG_L4 = WIMG_L3 + 4 * 256 * 128, WIMG_BYTES = WIMG_L4 + 4 * 256 * 128;
__host__ __device__ constexpr size_t wimg_at(int layer) {
    return layer == 0 ? WIMG_L1 : layer == 1 ? WIMG_L2 : layer == 2 ? WIMG_L3 : WIMG_L4;
}

enum Status { ST_OK = 0, ST_INVALID = 2, ST_DEVICE = 3 };

// ---- arithmetic shared by every kernel --------------------------------------------------------

__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// silu(z) = z (1 + tanh(z / 2)) / 2 = hz + hz tanh(hz) with hz = z / 2 (one MUFU, one FMA)
__device__ __forceinline__ float silu_of_half(float hz) { return fmaf(hz, tanh_fast(hz), hz); }
__device__ __forceinline__ float silu(float z) { return silu_of_half(0.5f * z); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = 0.5f + 0.5f * tanh_fast(0.5f * z);
    return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}
// byte offset of element (r, k) in a B image of `rows` rows
__device__ __forceinline__ size_t b_img(uint32_t r, uint32_t k, uint32_t rows) {
    return (size_t)(k >> 6) * rows * 128u + sw128_offset(r, k & 63u);
}

// lane j of the warp gets the sum over the warp's lanes of v[j] (v is consumed)
__device__ __forceinline__ float warp_column_sum(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int j = 0; j < off; j++) {
            const float send = upper ? v[j] : v[j + off];
            const float keep = upper ? v[j + off] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    return v[0];
}

__device__ __forceinline__ void flag_error(int *error, int code, volatile int *abort_flag) {
    if (error) atomicCAS(error, 0, code);
    *abort_flag = 1;
}

// ---- the forward and backward chain -------------------------------------------------------------
//
// One block per 128 points at a time: seven products (four layers forward, three back) one after the
// other, each on the operand that the epilogue before it left in shared memory. Warps 0-15 run the
// epilogues: thread (quarter, lane, c) owns point r = 32 quarter + lane, tensor-memory lane r, and
// columns [32 c, 32 c + 32) of each half of 128 columns; warp 16 streams the weight images (32 KB
// chunks: a k tile of all 256 rows), warp 17 issues the products (M = 128, N = 128 per half). Z
// stays with the thread that made it: it goes to global memory and back in the order of the threads.
//
// The halves overlap a layer with the next one. A product's k tiles 0 and 1 (of both column halves)
// need only the operand's first half, and go under the epilogue of its second half; k tiles 2 and 3
// of the first column half follow, are committed, and the next epilogue starts on them while those
// of the second column half run. Consecutive products use the two accumulators of 256 columns in
// turn. The operand is replaced in place: the commit of a column half tracks every product issued
// before it, which for the first are all those that read the operand's first half.
//
// At the training batch (16 384 points, 128 blocks) the chain of products and epilogues is what
// bounds it: a product is 2 048 cycles of the tensor pipe, an epilogue as many of the MUFU (a tanh
// per value). As seven launches, each with its operands read from and written to global memory, its
// transposed copies stored in 2-byte pieces and four epilogue warps, this part took 127 us of a
// step's 206. In one launch with whole layers one after the other: 68 thousand cycles per tile (35 us,
// a step 70.5 us); with the overlapping halves, the columns' sums behind the hand-overs and Z asked
// for ahead: 59 thousand (a step 65.5 us): a half's wait for its products 1.2 or 0.25 thousand
// forward, 2.2 or 1.5 back (the columns' sums in it), its epilogue 2 to 2.9, the output layer's 11.

constexpr int CH_EPI = 512, CH_THREADS = CH_EPI + 64, CH_STAGES = 4;
constexpr uint32_t CH_CHUNK = 256 * 128;  // 32 KB
constexpr uint32_t CH_SMEM = 4 * TILE_A + CH_STAGES * CH_CHUNK + 1024;
constexpr int CH_CHUNKS = 1 + 6 * 4;  // per tile: layer 1 (1 k tile), layers 2-4 and back (4 each)

struct ChainArgs {
    const uint8_t *wimg, *wtimg;
    const float *params, *x, *y;
    uint32_t inputs, tiles;
    float inv_batch;
    uint8_t *x_img, *h_img[3], *dz_img[4];
    uint4 *z[3];             // [tile][8][thread]: 8 BF16 values each
    float *db[4];            // [tile][256]
    float *dw5;              // [tile][256]
    float *scalars;          // [tile][2]: sum dout, sum (out - y)^2
    int *error;
};

// A training step's three kernels are launched ahead of their turn (launch_early): a block sets up
// its barriers and tensor memory while the kernel before runs out. grid_wait: until that kernel is
// complete and its writes, and those of every kernel before it, are seen; all that another kernel
// writes or reads is touched behind it. grid_trigger, behind the block's own wait: the next kernel's
// blocks may be placed, so a placed kernel has at most one unfinished kernel before it.
// 16 steps of 16 384 points: 1264 -> 1135 us (8 us of a step's 79 were the three kernels' ends and starts); the
// update's own loads of the parameters ahead of the wait gave none of it (1043 us with and without).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// row r of one A tile from 32 packed pairs
__device__ __forceinline__ void store_row(uint8_t *tile, uint32_t r, const uint32_t (&ph)[32]) {
#pragma unroll
    for (int q = 0; q < 8; q++)
        *reinterpret_cast<uint4 *>(tile + sw128_offset(r, 8 * q)) =
            make_uint4(ph[4 * q], ph[4 * q + 1], ph[4 * q + 2], ph[4 * q + 3]);
}

__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

__global__ void __launch_bounds__(CH_THREADS, 1) chain_kernel(ChainArgs g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[CH_STAGES], empty[CH_STAGES], act_ready[2], acc_ready[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ __align__(16) float bias[4][WIDTH], w5[WIDTH + 4];
    __shared__ float part_a[4][WIDTH], part_b[4][WIDTH], dot[4][128], scal[4][2];
    const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
    uint8_t *act = smem_raw + pad, *ring = act + 4 * TILE_A;
    const int warp = (int)uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t turns = blockIdx.x < g.tiles ? (g.tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < CH_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int h = 0; h < 2; h++) {
            mbar_init(&act_ready[h], 1);
            mbar_init(&acc_ready[h], 1);
        }
        abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&tmem_base, 512);
    grid_wait();
    grid_trigger();
    for (int i = threadIdx.x; i < 4 * WIDTH; i += CH_THREADS) bias[i / WIDTH][i % WIDTH] = g.params[bias_at(i / WIDTH) + i % WIDTH];
    for (int i = threadIdx.x; i <= WIDTH; i += CH_THREADS) w5[i] = g.params[P_W5 + i];  // (then b5)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (warp == 16) {
        if (lane == 0) {
            const uint32_t total = turns * CH_CHUNKS;
            uint32_t issued = 0;
            for (uint32_t i = 0; i < total && !abort_flag; i++) {
                const int s = i % CH_STAGES;
                if (i >= (uint32_t)CH_STAGES && !mbar_wait(&empty[s], ((i / CH_STAGES) - 1) & 1, WAIT_CYCLES)) {
                    flag_error(g.error, 101, &abort_flag);
                    break;
                }
                const uint32_t c = i % CH_CHUNKS;
                // forward: W1, W2, W3, W4; back: the transposes of W4, W3, W2
                const uint8_t *src = c < 13 ? g.wimg + (size_t)c * CH_CHUNK
                                            : g.wtimg + (size_t)(2 - (c - 13) / 4) * 4 * CH_CHUNK + (c - 13) % 4 * CH_CHUNK;
                mbar_expect_tx(&full[s], CH_CHUNK);
                bulk_load(ring + (size_t)s * CH_CHUNK, src, CH_CHUNK, &full[s]);
                issued = i + 1;
            }
            // the copies still in flight end before the block does
            for (uint32_t i = issued > (uint32_t)CH_STAGES ? issued - CH_STAGES : 0; i < issued; i++)
                if (!mbar_wait(&full[i % CH_STAGES], (i / CH_STAGES) & 1, WAIT_CYCLES)) flag_error(g.error, 102, &abort_flag);
        }
    } else if (warp == 17) {
        constexpr uint32_t idesc = idesc_bf16(128, 128);
        const bool leader = elect_one();
        const uint32_t act_addr = smem_u32(act), ring_addr = smem_u32(ring);
        uint32_t chunk = 0, seconds = 0;  // seconds: products so far that wait for the operand's second half
        bool ok = true;
        auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
            if (ok && !__all_sync(0xffffffffu, mbar_wait(bar, parity, WAIT_CYCLES))) {
                flag_error(g.error, code, &abort_flag);
                ok = false;
            }
        };
        // one k tile of one column half of product n
        auto issue = [&](uint32_t n, int kt, int h) {
            const uint32_t a_addr = act_addr + kt * TILE_A, b_addr = ring_addr + (chunk + kt) % CH_STAGES * CH_CHUNK + h * TILE_A;
            if (leader)
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    mma_bf16(tmem + (n & 1) * 256 + h * 128, sw128_desc(a_addr + 32 * k), sw128_desc(b_addr + 32 * k), idesc,
                             (kt | k) != 0);
        };
        auto commit = [&](uint64_t *bar) {
            if (leader) mma_commit(bar);
        };
        for (uint32_t n = 0; n < 7 * turns && ok; n++) {
            const int kts = n % 7 == 0 ? 1 : 4;
            auto arrived = [&](int kt) {
                wait(&full[(chunk + kt) % CH_STAGES], ((chunk + kt) / CH_STAGES) & 1, 104);
                tc_fence_after();
            };
            wait(&act_ready[0], n & 1, 103);
            if (kts == 4) {
                for (int kt = 0; kt < 2 && ok; kt++) {
                    arrived(kt);
                    if (!ok) break;
                    issue(n, kt, 0);
                    issue(n, kt, 1);
                    commit(&empty[(chunk + kt) % CH_STAGES]);
                }
                wait(&act_ready[1], seconds++ & 1, 103);
            }
            for (int kt = kts == 4 ? 2 : 0; kt < kts && ok; kt++) {
                arrived(kt);
                if (ok) issue(n, kt, 0);
            }
            if (!ok) break;
            if (kts == 1) issue(n, 0, 1);  // (it reads the half that the first epilogue replaces)
            commit(&acc_ready[0]);
            for (int kt = kts == 4 ? 2 : 0; kt < kts; kt++) {
                if (kts == 4) issue(n, kt, 1);
                commit(&empty[(chunk + kt) % CH_STAGES]);
            }
            commit(&acc_ready[1]);
            __syncwarp();
            chunk += kts;
        }
    } else {
        const uint32_t c = warp >> 2, quarter = warp & 3, r = 32 * quarter + lane, col = 32 * c;
        const uint32_t acc0 = tmem + ((uint32_t)(32 * quarter) << 16) + col;
        const bool first = threadIdx.x == 0;
        uint32_t n = 0, acc = acc0;  // the product, and this thread's columns of its accumulator's first half
        // After a given-up wait the threads go on without waiting (every barrier is met; the outputs
        // are not used: the error is flagged).
        auto wait_acc = [&](int h) {
            if (!abort_flag && !mbar_wait(&acc_ready[h], n & 1, WAIT_CYCLES)) flag_error(g.error, 105, &abort_flag);
            acc = acc0 + (n & 1) * 256;
            __syncwarp();
            tc_fence_after();
        };
        // Half h of the written operand is stored to `image` and, with `next`, handed to the next
        // product. The store before it, of the other half, has read its shared memory when the barrier
        // is passed: that half may be replaced.
        auto hand_over = [&](uint8_t *image, uint32_t bytes, int h, bool next) {
            fence_async_shared();
            tc_fence_before();
            if (first) bulk_store_read();
            epilogue_barrier();
            if (first) {
                if (next) mbar_arrive(&act_ready[h]);
                bulk_store(image + h * 2 * TILE_A, act + h * 2 * TILE_A, bytes);
            }
        };
        // 32 columns of half h of row r
        auto store_columns = [&](int h, const uint32_t (&ph)[16]) {
            uint8_t *tile = act + (2 * h + (c >> 1)) * TILE_A;
#pragma unroll
            for (uint32_t q = 0; q < 4; q++)
                *reinterpret_cast<uint4 *>(tile + sw128_offset(r, 32 * (c & 1) + 8 * q)) =
                    make_uint4(ph[4 * q], ph[4 * q + 1], ph[4 * q + 2], ph[4 * q + 3]);
        };
        // The sums over the 128 points of half h's columns, from the quarters' sums, into `out`
        // [tile][256]. The quarters' sums are taken behind the operand's hand-over, under the next
        // product, and added up behind the hand-over after that.
        auto column_sums = [&](float (*part)[WIDTH], float *out, uint32_t tile, int h) {
            const uint32_t k = (threadIdx.x & 127) + 128 * h;
            if (c == 3) out[(size_t)tile * WIDTH + k] = part[0][k] + part[1][k] + part[2][k] + part[3][k];
        };
        // this thread's Z of a layer's half h, asked for one half's epilogue ahead of its use
        uint4 zs[4];
        auto load_z = [&](int layer, uint32_t tile, int h) {
            const uint4 *zt = g.z[layer] + ((size_t)tile * 8 + 4 * h) * CH_EPI + threadIdx.x;
#pragma unroll
            for (int q = 0; q < 4; q++) zs[q] = zt[q * CH_EPI];
        };
        for (uint32_t i = 0; i < turns; i++) {
            const uint32_t tile = blockIdx.x + i * gridDim.x, m = tile * 128 + r;
            uint32_t ph[16];
            // the inputs: features [16 c, 16 c + 16) of row r (K = 64)
            {
                uint32_t p[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const uint32_t k = 16 * c + 2 * e;
                    const float lo = k < g.inputs ? g.x[(size_t)m * g.inputs + k] : 0.0f;
                    const float hi = k + 1 < g.inputs ? g.x[(size_t)m * g.inputs + k + 1] : 0.0f;
                    p[e] = pack_bf16(lo, hi);
                }
#pragma unroll
                for (int q = 0; q < 2; q++)
                    *reinterpret_cast<uint4 *>(act + sw128_offset(r, 16 * c + 8 * q)) =
                        make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
                hand_over(g.x_img + (size_t)tile * TILE_A, TILE_A, 0, true);
            }
            // layers 1-3 forward
            for (int layer = 0; layer < 3; layer++, n++) {
                uint4 *zt = g.z[layer] + (size_t)tile * 8 * CH_EPI + threadIdx.x;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float v[32];
                    uint32_t pz[16];
                    wait_acc(h);
                    tmem_load32(acc + 128 * h, v);
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const int k = 128 * h + col + j;
                        const float z0 = v[j] + bias[layer][k], z1 = v[j + 1] + bias[layer][k + 1];
                        pz[j / 2] = pack_bf16(z0, z1);
                        ph[j / 2] = pack_bf16(silu(z0), silu(z1));
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        zt[(4 * h + q) * CH_EPI] = make_uint4(pz[4 * q], pz[4 * q + 1], pz[4 * q + 2], pz[4 * q + 3]);
                    if (layer == 0 && h == 0) {  // X's store was the last one, and of the same half
                        if (first) bulk_store_read();
                        epilogue_barrier();
                    }
                    store_columns(h, ph);
                    hand_over(g.h_img[layer] + (size_t)tile * 4 * TILE_A, 2 * TILE_A, h, true);
                }
            }
            // layer 4 and the output layer: out, dout, dZ4 = dout w5 silu'(z4)
            {
                float out = 0.0f;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float v[32];
                    wait_acc(h);
                    tmem_load32(acc + 128 * h, v);
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const int k = 128 * h + col + j;
                        const uint32_t w = pack_bf16(silu(v[j] + bias[3][k]), silu(v[j + 1] + bias[3][k + 1]));
                        out += __uint_as_float(w << 16) * w5[k];
                        out += __uint_as_float(w & 0xffff0000u) * w5[k + 1];
                    }
                }
                dot[c][r] = out;
                epilogue_barrier();
                out = dot[0][r] + dot[1][r] + dot[2][r] + dot[3][r] + w5[WIDTH];
                const float err = out - g.y[m], dout = 2.0f * err * g.inv_batch;
                if (c == 0) {
                    float a = dout, b = err * err;
#pragma unroll
                    for (int off = 16; off >= 1; off >>= 1) {
                        a += __shfl_xor_sync(0xffffffffu, a, off);
                        b += __shfl_xor_sync(0xffffffffu, b, off);
                    }
                    if (lane == 0) {
                        scal[quarter][0] = a;
                        scal[quarter][1] = b;
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float v[32], hw[32];
                    tmem_load32(acc + 128 * h, v);
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const int k = 128 * h + col + j;
                        const float z = v[j] + bias[3][k], t = tanh_fast(0.5f * z), s = 0.5f + 0.5f * t;
                        hw[j] = fmaf(0.5f * z, t, 0.5f * z);
                        v[j] = dout * w5[k] * (s * (1.0f + z * (1.0f - s)));
                    }
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        ph[j / 2] = pack_bf16(v[j], v[j + 1]);
                        const uint32_t w = pack_bf16(hw[j], hw[j + 1]);
                        hw[j] = dout * __uint_as_float(w << 16);
                        hw[j + 1] = dout * __uint_as_float(w & 0xffff0000u);
                    }
                    store_columns(h, ph);
                    hand_over(g.dz_img[3] + (size_t)tile * 4 * TILE_A, 2 * TILE_A, h, true);
                    if (h == 1) {
                        load_z(2, tile, 0);
                        column_sums(part_a, g.db[3], tile, 0);
                        column_sums(part_b, g.dw5, tile, 0);
                    }
                    part_a[quarter][128 * h + col + lane] = warp_column_sum(v);
                    part_b[quarter][128 * h + col + lane] = warp_column_sum(hw);
                }
                if (threadIdx.x < 2)
                    g.scalars[2 * tile + threadIdx.x] =
                        scal[0][threadIdx.x] + scal[1][threadIdx.x] + scal[2][threadIdx.x] + scal[3][threadIdx.x];
                n++;
            }
            // back: dZ3, dZ2, dZ1
            for (int layer = 2; layer >= 0; layer--, n++) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float v[32];
                    uint4 z[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) z[q] = zs[q];
                    if (h == 0) load_z(layer, tile, 1);
                    else if (layer > 0) load_z(layer - 1, tile, 0);
                    wait_acc(h);
                    tmem_load32(acc + 128 * h, v);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t ws[4] = {z[q].x, z[q].y, z[q].z, z[q].w};
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            v[8 * q + 2 * e] *= silu_grad(__uint_as_float(ws[e] << 16));
                            v[8 * q + 2 * e + 1] *= silu_grad(__uint_as_float(ws[e] & 0xffff0000u));
                            ph[4 * q + e] = pack_bf16(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
                        }
                    }
                    store_columns(h, ph);
                    hand_over(g.dz_img[layer] + (size_t)tile * 4 * TILE_A, 2 * TILE_A, h, layer > 0);
                    column_sums(part_a, g.db[h ? layer : layer + 1], tile, 1 - h);
                    if (layer == 2 && h == 0) column_sums(part_b, g.dw5, tile, 1);
                    part_a[quarter][128 * h + col + lane] = warp_column_sum(v);
                }
            }
            epilogue_barrier();
            column_sums(part_a, g.db[0], tile, 1);
        }
        if (first) bulk_store_done();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- the weight gradients -------------------------------------------------------------------------
//
// dW_l = dZ_l^T H_{l-1}: a block takes one layer's upper or lower 128 rows over a part of the batch,
// 128 points per stage, A = dZ's tiles of those rows and B = H's (X's) tiles, K along the points. The
// parts fill the chip once (148 blocks for more than 20 tiles of points); FP32 partials go out as
// [part][column / 4][row][4], so that a warp writes whole lines.

constexpr uint32_t DW_PARTS = 21, DW_PARTS_X = 11;  // parts of the batch, layers 2-4 and layer 1
constexpr uint32_t DW_STAGE = 6 * TILE_A, DW_SMEM = 2 * DW_STAGE + 1024;
inline __host__ __device__ uint32_t dw_parts(int layer, uint32_t tiles) {
    const uint32_t most = layer == 0 ? DW_PARTS_X : DW_PARTS;
    return tiles < most ? tiles : most;
}

struct DwArgs {
    const uint8_t *x_img, *h_img[3], *dz_img[4];
    float *partial[4];
    uint32_t tiles;
    int *error;
};

__global__ void __launch_bounds__(256, 1) dw_kernel(DwArgs g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[2], empty[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
    uint8_t *smem = smem_raw + pad;
    const int warp = (int)uniform_warp(), lane = threadIdx.x & 31;
    // the block's layer, rows and part: layers 2-4 first
    const uint32_t parts = dw_parts(1, g.tiles), parts_x = dw_parts(0, g.tiles);
    uint32_t b = blockIdx.x;
    const int layer = b < 6 * parts ? 1 + (int)(b / (2 * parts)) : 0;
    b = layer ? b % (2 * parts) : b - 6 * parts;
    const uint32_t mine = layer ? parts : parts_x, half = b / mine, part = b % mine;
    const uint32_t t0 = g.tiles * part / mine, t1 = g.tiles * (part + 1) / mine;
    const uint32_t width = layer ? WIDTH : IN, b_bytes = width / 64 * TILE_A, bytes = 2 * TILE_A + b_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&done, 1);
        abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&tmem_base, 256);
    grid_wait();
    grid_trigger();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (warp == 0) {
        if (lane == 0) {
            const uint8_t *a = g.dz_img[layer] + 2 * half * TILE_A, *h = layer ? g.h_img[layer - 1] : g.x_img;
            uint32_t issued = 0;
            for (uint32_t i = 0; i < t1 - t0 && !abort_flag; i++) {
                const int s = i & 1;
                if (i >= 2 && !mbar_wait(&empty[s], ((i >> 1) - 1) & 1, WAIT_CYCLES)) {
                    flag_error(g.error, 111, &abort_flag);
                    break;
                }
                uint8_t *st = smem + s * DW_STAGE;
                mbar_expect_tx(&full[s], bytes);
                bulk_load(st, a + (size_t)(t0 + i) * 4 * TILE_A, 2 * TILE_A, &full[s]);
                bulk_load(st + 2 * TILE_A, h + (size_t)(t0 + i) * b_bytes, b_bytes, &full[s]);
                issued = i + 1;
            }
            for (uint32_t i = issued > 2 ? issued - 2 : 0; i < issued; i++)
                if (!mbar_wait(&full[i & 1], (i >> 1) & 1, WAIT_CYCLES)) flag_error(g.error, 112, &abort_flag);
        }
    } else if (warp == 1) {
        const uint32_t idesc = (layer ? idesc_bf16(128, WIDTH) : idesc_bf16(128, IN)) | IDESC_MN;
        const bool leader = elect_one();
        for (uint32_t i = 0; i < t1 - t0; i++) {
            const int s = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (i >> 1) & 1, WAIT_CYCLES))) {
                flag_error(g.error, 113, &abort_flag);
                break;
            }
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem) + s * DW_STAGE, b_addr = a_addr + 2 * TILE_A;
            if (leader) {
#pragma unroll
                for (uint32_t k = 0; k < 8; k++)  // 16 points each
                    mma_bf16(tmem, sw128_mn_desc(a_addr + 2048 * k, TILE_A), sw128_mn_desc(b_addr + 2048 * k, TILE_A), idesc,
                             (i | k) != 0);
                mma_commit(&empty[s]);
            }
            __syncwarp();
        }
        if (leader) mma_commit(&done);
    }
    __syncwarp();
    bool ready = mbar_wait(&done, 0, WAIT_CYCLES);
    tc_fence_after();
    if (!ready) flag_error(g.error, 114, &abort_flag);
    ready = __all_sync(0xffffffffu, ready && !abort_flag);
    if (ready) {
        const uint32_t quarter = warp & 3, m = 128 * half + 32 * quarter + lane;
        const uint32_t columns = width / 2, col = columns * (warp >> 2);  // this warp's columns
        float4 *out = reinterpret_cast<float4 *>(g.partial[layer]) + (size_t)part * width / 4 * WIDTH + m;
        for (uint32_t c = col; c < col + columns; c += 32) {
            float v[32];
            tmem_load32(tmem + ((32 * quarter) << 16) + c, v);
#pragma unroll
            for (int q = 0; q < 8; q++)
                out[(size_t)(c / 4 + q) * WIDTH] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 256);
}

// ---- parameters into weight images -----------------------------------------------------------

// one thread per weight of W1..W4: its BF16 value into the forward image (rows = outputs, K =
// inputs) and, for W2..W4, the transposed image (rows = inputs, K = outputs) the backward reads
__global__ void images_kernel(const float *params, uint8_t *wimg, uint8_t *wtimg) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t first = WIDTH * IN, per = WIDTH * WIDTH;
    if (t >= first + 3 * per) return;
    uint32_t layer, o, i;
    float w;
    if (t < first) {
        layer = 0;
        o = t / IN;
        i = t % IN;
        w = params[P_W1 + t];
    } else {
        const uint32_t u = t - first;
        layer = 1 + u / per;
        o = (u % per) / WIDTH;
        i = u % WIDTH;
        w = params[(layer == 1 ? P_W2 : layer == 2 ? P_W3 : P_W4) + (u % per)];
    }
    const __nv_bfloat16 b = __float2bfloat16_rn(w);
    const size_t at = wimg_at((int)layer);
    *reinterpret_cast<__nv_bfloat16 *>(wimg + at + b_img(o, i, WIDTH)) = b;
    if (layer > 0)
        *reinterpret_cast<__nv_bfloat16 *>(wtimg + (size_t)(layer - 1) * 4 * 256 * 128 + b_img(i, o, WIDTH)) = b;
}

// ---- gradients and Adam ----------------------------------------------------------------------------
//
// One launch sums the partials (each sum in a fixed order: the result does not depend on the launch),
// and writes the gradient, or takes the Adam step with the weights' BF16 images: blocks 0 .. 207 a
// piece of 16 rows x 64 columns of a layer's weights each, then 40 blocks of 32 bias or output weights
// (eight segments of the tiles' sums side by side) and one of the scalars. The partials come by
// (column / 4, row), the parameters, moments and images by rows, the transposed image by columns: a
// piece turns between them in shared memory, so that every access is of whole sectors.

enum UpdateMode { UP_GRADIENT, UP_TRAIN, UP_APPLY };
constexpr uint32_t UP_W = WIDTH / 16 * (1 + 3 * 4), UP_COLS = 5 * WIDTH / 32, UP_BLOCKS = UP_W + UP_COLS + 1;

struct UpdateArgs {
    const float *dw[4];   // [part][column / 4][row][4]
    const float *db[4];   // [tile][256]
    const float *dw5;     // [tile][256]
    const float *scalars; // [tile][2]
    uint32_t tiles;
    float *grad;          // UP_GRADIENT: written; UP_APPLY: read (param order)
    float *loss;          // one float (set), or null
    float *loss_sum;      // one float (added), or null
    float *params, *m1, *m2;
    uint8_t *wimg, *wtimg;
    float lr, c1, c2;
    uint32_t inputs;
};

// the Adam step of one value w with moments a and b on its gradient
__device__ __forceinline__ void adam_value(const UpdateArgs &u, float &w, float &a, float &b, float g) {
    a = 0.9f * a + 0.1f * g;
    b = 0.999f * b + 0.001f * g * g;
    w -= u.lr * (a * u.c1) / (sqrtf(b * u.c2) + 1e-8f);
}

template <int MODE> __device__ __forceinline__ void finish(const UpdateArgs &u, size_t t, float g) {
    if (MODE == UP_GRADIENT) u.grad[t] = g;
    else adam_value(u, u.params[t], u.m1[t], u.m2[t], MODE == UP_APPLY ? u.grad[t] : g);
}

template <int MODE>
__global__ void __launch_bounds__(256) update_kernel(UpdateArgs u) {
    __shared__ float red[8][33];
    if (blockIdx.x < UP_W) {
        __shared__ float4 piece[16][17];  // [row][column / 4]
        const int layer = blockIdx.x < WIDTH / 16 ? 0 : 1 + (int)((blockIdx.x - WIDTH / 16) / (WIDTH / 16 * 4));
        const uint32_t n = layer ? (blockIdx.x - WIDTH / 16) % (WIDTH / 16 * 4) : 4 * blockIdx.x;
        const uint32_t row0 = 16 * (n / 4), first4 = 16 * (n % 4), fan = layer ? WIDTH : IN;
        const uint32_t x = threadIdx.x & 15, y = threadIdx.x >> 4;
        // by rows: this thread's row and columns
        const uint32_t o = row0 + y, c4 = first4 + x;
        const size_t t = (layer == 0 ? P_W1 : layer == 1 ? P_W2 : layer == 2 ? P_W3 : P_W4) + (size_t)o * fan + 4 * c4;
        float4 w, a, b;
        grid_wait();
        grid_trigger();
        if (MODE != UP_GRADIENT) {  // (the network's own arrays: aligned; they come while the partials are summed)
            w = *reinterpret_cast<const float4 *>(u.params + t);
            a = *reinterpret_cast<const float4 *>(u.m1 + t);
            b = *reinterpret_cast<const float4 *>(u.m2 + t);
        }
        float4 g;
        if (MODE != UP_APPLY) {
            const float4 *p = reinterpret_cast<const float4 *>(u.dw[layer]) + (size_t)(first4 + y) * WIDTH + row0 + x;
            const uint32_t parts = dw_parts(layer, u.tiles);
            g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 11
            for (uint32_t k = 0; k < parts; k++) {
                const float4 v = p[(size_t)k * fan / 4 * WIDTH];
                g.x += v.x;
                g.y += v.y;
                g.z += v.z;
                g.w += v.w;
            }
            piece[x][y] = g;
            __syncthreads();
            g = piece[y][x];
        } else {  // (the caller's array, of any alignment)
            g = make_float4(u.grad[t], u.grad[t + 1], u.grad[t + 2], u.grad[t + 3]);
        }
        if constexpr (MODE == UP_GRADIENT) {
            u.grad[t] = g.x;
            u.grad[t + 1] = g.y;
            u.grad[t + 2] = g.z;
            u.grad[t + 3] = g.w;
        } else {
            float *wv = &w.x, *av = &a.x, *bv = &b.x;
            const float *gv = &g.x;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (layer > 0 || 4 * c4 + j < u.inputs) adam_value(u, wv[j], av[j], bv[j], gv[j]);  // (W1's padding columns stay zero)
            *reinterpret_cast<float4 *>(u.params + t) = w;
            *reinterpret_cast<float4 *>(u.m1 + t) = a;
            *reinterpret_cast<float4 *>(u.m2 + t) = b;
            *reinterpret_cast<uint2 *>(u.wimg + wimg_at(layer) + b_img(o, 4 * c4, WIDTH)) =
                make_uint2(pack_bf16(w.x, w.y), pack_bf16(w.z, w.w));
            if (layer > 0) {
                __syncthreads();
                piece[y][x] = w;
                __syncthreads();
                // by columns: eight rows of one column
                if (threadIdx.x < 128) {
                    const uint32_t c = threadIdx.x >> 1, r0 = 8 * (threadIdx.x & 1);
                    const float *col = &piece[0][c / 4].x + c % 4;
                    uint32_t q[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) q[j] = pack_bf16(col[(r0 + 2 * j) * 17 * 4], col[(r0 + 2 * j + 1) * 17 * 4]);
                    *reinterpret_cast<uint4 *>(u.wtimg + (size_t)(layer - 1) * 4 * 256 * 128 + b_img(4 * first4 + c, row0 + r0, WIDTH)) =
                        make_uint4(q[0], q[1], q[2], q[3]);
                }
            }
        }
    } else if (blockIdx.x < UP_W + UP_COLS) {
        const uint32_t n = 32 * (blockIdx.x - UP_W) + (threadIdx.x & 31), layer = n / WIDTH, seg = threadIdx.x >> 5;
        const float *src = (layer < 4 ? u.db[layer] : u.dw5) + n % WIDTH;
        float s = 0.0f;
        grid_wait();
        grid_trigger();
        if (MODE != UP_APPLY) {
#pragma unroll 8
            for (uint32_t k = seg; k < u.tiles; k += 8) s += src[(size_t)k * WIDTH];
            red[seg][threadIdx.x & 31] = s;
            __syncthreads();
            s = 0.0f;
            for (int k = 0; k < 8; k++) s += red[k][threadIdx.x & 31];
        }
        if (seg == 0) finish<MODE>(u, (layer < 4 ? bias_at((int)layer) : P_W5) + n % WIDTH, s);
    } else {
        // the sum of dout (b5's gradient) and the loss: 128 strided sums each, then in order
        __shared__ float sums[2][128];
        const uint32_t which = threadIdx.x & 1, k0 = threadIdx.x >> 1;
        float s = 0.0f;
        grid_wait();
        grid_trigger();
        if (MODE != UP_APPLY)
            for (uint32_t k = k0; k < u.tiles; k += 128) s += u.scalars[2 * k + which];
        sums[which][k0] = s;
        __syncthreads();
        if (threadIdx.x < 2) {
            s = 0.0f;
            for (int k = 0; k < 128; k++) s += sums[threadIdx.x][k];
            if (threadIdx.x == 0) finish<MODE>(u, P_B5, s);
            else if (MODE != UP_APPLY) {
                if (u.loss) *u.loss = s;
                if (u.loss_sum) *u.loss_sum += s;
            }
        }
    }
}

// ---- fused inference ------------------------------------------------------------------------------
//
// One persistent block per SM with two tiles of 128 points in flight. Warps 0-15 (eight per tile)
// build the inputs and run the epilogues: thread (quarter, lane, c) owns point r = 32 quarter + lane,
// tensor-memory lane r, and in each 128-column half of a layer the 64 columns of quarter c. Warp 16
// streams the weight images through a ring of 16 KB chunks (half, k tile: 128 output rows x 64
// values), each used by both tiles; warps 17 and 18 issue the tiles' products (M = 128, N = 128)
// into 256 FP32 columns of tensor memory per tile. A tile's activations stay in one 64 KB A tile set.
//
// What bounds it is the activations: 1024 tanh per point on 16 MUFU lanes per SM are 64 cycles, the
// products 52; so the products have to run behind the epilogues. A layer's products go half by half:
// the first half's epilogue runs while the second half is computed (its results wait packed in 32
// registers, since the products still read the activations they replace), and the next layer's
// products start on the first half's k tiles while the second half's epilogue runs. Each tile has its
// own issuing warp (one issues while the other waits), and the tiles' epilogues take turns, so that
// one tile's activations run while the other's stores, barriers and products do; a warp loads its
// accumulators before its turn. Sharing each chunk between two tiles halves the weights' L2 traffic.
// Measured on B200, 2^21 points: 0.83 ms (115 cycles per point and SM, 1077 TFLOP/s, 0.65 of the
// measured BF16 peak); 0.846 with the accumulators loaded inside the turns, 0.903 without turns, 1.25
// with one issuing warp for both tiles, 1.44 with that warp's loop on one lane (umma.cuh elect_one).
// The form before (two blocks per SM, a tile each, a layer's products and its epilogue one after the
// other): 1.31 ms. 300 007 points: 192 -> 131 us.
// Each output's sums keep their order (k tiles 0 .. 3; the output layer's 128 columns of a half one
// after the other): the bits do not depend on the split.

constexpr int FWD_TILE_THREADS = 256;
constexpr int FWD_THREADS = 2 * FWD_TILE_THREADS + 96;
constexpr uint32_t FWD_CHUNK = 128 * 128;  // 16 KB
constexpr int FWD_STAGES = 5;
constexpr uint32_t FWD_SMEM = 8 * TILE_A + FWD_STAGES * FWD_CHUNK + 1024;
constexpr int FWD_CHUNKS = 2 + 3 * 8;  // per tile: layer 1 (2 halves x 1 k tile), layers 2-4 (2 x 4)
constexpr int FWD_PARAMS = 5 * WIDTH + 1;  // b1..b4, w5, b5

struct ForwardArgs {
    const uint8_t *wimg;
    const float *params;
    const float *x;
    uint32_t inputs, count, tiles;
    uint32_t per;  // tiles in flight per block: 2 or 1
    float *out;
    int *error;
    // candidates (stage 1 of two-stage unweighting): segments of candidates, one per subprocess;
    // tile t belongs to the segment whose tiles [tile_first, next tile_first) hold it
    pacuda_uw_segment seg[PACUDA_UW_MAX_SEGMENTS];
    uint32_t tile_first[PACUDA_UW_MAX_SEGMENTS + 1];
    uint32_t segments;
    double mu, sigma;  // s = exp(mu + sigma out); kept when (first decision uniform) s_max < s
    uint32_t capacity;
    uint32_t numbers;  // the candidates' phase-space numbers: 5 (2 -> 3) or 8 (2 -> 4)
};

// the segment of tile t (segments are few: a linear scan)
__device__ __forceinline__ uint32_t segment_of(const ForwardArgs &g, uint32_t t) {
    uint32_t k = 0;
    while (k + 1 < g.segments && t >= g.tile_first[k + 1]) k++;
    return k;
}

enum { FWD_FROM_X = 0, FWD_CANDIDATES = 1 };

// the byte offset of chunk c of a tile's stream in the weight images (layer by layer, half by half,
// its k tiles in order)
__device__ __forceinline__ size_t fwd_chunk(uint32_t c) {
    if (c < 2) return wimg_at(0) + (size_t)c * FWD_CHUNK;
    const uint32_t layer = 1 + (c - 2) / 8, half = (c - 2) % 8 / 4, kt = (c - 2) % 4;
    return wimg_at((int)layer) + (size_t)kt * 256 * 128 + (size_t)half * FWD_CHUNK;
}

// 64 columns of tensor memory from `taddr` (loaded while the warp waits for its turn)
__device__ __forceinline__ void fwd_load(uint32_t taddr, uint32_t (&z)[4][16]) {
#pragma unroll
    for (int k = 0; k < 4; k++) tmem_load16_async(taddr + 16 * k, z[k]);
#pragma unroll
    for (int k = 0; k < 4; k++) tmem_wait16(z[k]);
}

// four values through the activation, as two packed BF16 pairs; halved biases: the epilogue works on
// z / 2 (in pairs: the single conversion shares the MUFU's pipe)
__device__ __forceinline__ void fwd_activate4(const uint32_t *z, float4 b, uint32_t &lo, uint32_t &hi) {
    lo = pack_bf16(silu_of_half(fmaf(__uint_as_float(z[0]), 0.5f, b.x)), silu_of_half(fmaf(__uint_as_float(z[1]), 0.5f, b.y)));
    hi = pack_bf16(silu_of_half(fmaf(__uint_as_float(z[2]), 0.5f, b.z)), silu_of_half(fmaf(__uint_as_float(z[3]), 0.5f, b.w)));
}

__device__ __forceinline__ void fwd_activate(const uint32_t (&z)[4][16], const float *bias, uint32_t (&ph)[32]) {
    const float4 *b4 = reinterpret_cast<const float4 *>(bias);
#pragma unroll
    for (int q = 0; q < 16; q++) fwd_activate4(&z[q / 4][4 * (q % 4)], b4[q], ph[2 * q], ph[2 * q + 1]);
}

template <int MODE>
__global__ void __launch_bounds__(FWD_THREADS, 1) forward_kernel(ForwardArgs g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[FWD_STAGES], empty[FWD_STAGES];
    // per tile: the activations' first and second 128 columns are written (the inputs are the first),
    // a layer's first and second half of products is done, the output layer's second half is summed
    __shared__ uint64_t act_ready[2][2], acc_ready[2][2], dot_ready[2];
    __shared__ uint64_t turn[2];  // the other tile's warps have finished an epilogue
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ __align__(16) float prm[FWD_PARAMS];
    __shared__ float dot_hi[2][128];
    const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
    uint8_t *act = smem_raw + pad;         // per tile 4 A tiles: its activations (K = 256)
    uint8_t *ring = act + 8 * TILE_A;      // weight chunks
    const int warp = (int)uniform_warp(), lane = threadIdx.x & 31;
    // the block's turns: turn i takes tiles per x (blockIdx + i gridDim) + 0 .. per - 1
    const uint32_t pairs = (g.tiles + g.per - 1) / g.per;
    const uint32_t turns = blockIdx.x < pairs ? (pairs - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < FWD_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], g.per);
        }
        for (int t = 0; t < 2; t++) {
            for (int h = 0; h < 2; h++) {
                mbar_init(&act_ready[t][h], FWD_TILE_THREADS);
                mbar_init(&acc_ready[t][h], 1);
            }
            mbar_init(&dot_ready[t], FWD_TILE_THREADS / 2);
            mbar_init(&turn[t], FWD_TILE_THREADS / 32);
        }
        abort_flag = 0;
        fence_mbar_init();
    }
    // b1..b4 halved (the epilogue computes z / 2 = acc / 2 + b / 2 in one FMA), then w5 and b5
    // (P_W5, P_B5 follow each other)
    for (int i = threadIdx.x; i < FWD_PARAMS; i += FWD_THREADS)
        prm[i] = i < 4 * WIDTH ? 0.5f * g.params[bias_at(i / WIDTH) + i % WIDTH] : g.params[P_W5 + (i - 4 * WIDTH)];
    if (warp == 0) tmem_alloc(&tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (warp == 16) {
        if (lane == 0) {
            const uint32_t total = turns * FWD_CHUNKS;
            uint32_t issued = 0;
            for (uint32_t i = 0; i < total && !abort_flag; i++) {
                const int s = i % FWD_STAGES;
                if (i >= (uint32_t)FWD_STAGES && !mbar_wait(&empty[s], ((i / FWD_STAGES) - 1) & 1, WAIT_CYCLES)) {
                    flag_error(g.error, 201, &abort_flag);
                    break;
                }
                mbar_expect_tx(&full[s], FWD_CHUNK);
                bulk_load(ring + (size_t)s * FWD_CHUNK, g.wimg + fwd_chunk(i % FWD_CHUNKS), FWD_CHUNK, &full[s]);
                issued = i + 1;
            }
            for (uint32_t i = issued > (uint32_t)FWD_STAGES ? issued - FWD_STAGES : 0; i < issued; i++)
                if (!mbar_wait(&full[i % FWD_STAGES], (i / FWD_STAGES) & 1, WAIT_CYCLES))
                    flag_error(g.error, 202, &abort_flag);
        }
    } else if (warp >= 17) {
        // the products of tile t; the two tiles' issuers share the chunks and the tensor pipe, one
        // issuing while the other waits
        constexpr uint32_t idesc = idesc_bf16(128, 128);
        const uint32_t t = warp - 17;
        const bool leader = elect_one();
        const uint32_t act_addr = smem_u32(act) + 4 * t * TILE_A, ring_addr = smem_u32(ring), acc = tmem + 256 * t;
        uint32_t chunk = 0, acts[2] = {0, 0};  // completed waits of act_ready[t][h]
        bool ok = t < g.per;
        for (uint32_t i = 0; i < turns && ok; i++) {
            const bool mine = g.per * (blockIdx.x + i * gridDim.x) + t < g.tiles;  // (else: the chunks pass by)
            for (int layer = 0; layer < 4 && ok; layer++) {
                const int kts = layer == 0 ? 1 : 4;
                for (int c = 0; c < 2 * kts && ok; c++, chunk++) {
                    const int half = c / kts, kt = c % kts, s = chunk % FWD_STAGES;
                    if (mine && half == 0 && (kt == 0 || kt == 2)) {  // the activations this k tile begins
                        ok = __all_sync(0xffffffffu, mbar_wait(&act_ready[t][kt / 2], acts[kt / 2] & 1, WAIT_CYCLES));
                        acts[kt / 2]++;
                        if (!ok) {
                            flag_error(g.error, 203, &abort_flag);
                            break;
                        }
                    }
                    ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (chunk / FWD_STAGES) & 1, WAIT_CYCLES));
                    if (!ok) {
                        flag_error(g.error, 204, &abort_flag);
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = act_addr + kt * TILE_A, b_addr = ring_addr + s * FWD_CHUNK;
                    if (leader) {
                        if (mine) {
#pragma unroll
                            for (uint32_t k = 0; k < 4; k++)
                                mma_bf16(acc + 128 * half, sw128_desc(a_addr + 32 * k), sw128_desc(b_addr + 32 * k), idesc, (kt | k) != 0);
                            if (kt == kts - 1) mma_commit(&acc_ready[t][half]);
                        }
                        mma_commit(&empty[s]);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // the tiles' warps: inputs, epilogues, outputs
        const uint32_t t = warp >> 3, c = (warp >> 2) & 1, r = 32 * (warp & 3) + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 256 * t;
        uint8_t *mine = act + 4 * t * TILE_A;
        uint32_t accs = 0, dots = 0, epilogues = 0;  // layers, tiles and epilogues so far
        // the two tiles' epilogues take turns (tile 0's n-th, tile 1's n-th, tile 0's next, ...); a tile
        // alone in the block's last turn does not wait
        bool paired = false;
        auto take_turn = [&]() -> bool {
            const uint32_t n = epilogues++;
            if (!paired || (t == 0 && n == 0)) return true;
            return __all_sync(0xffffffffu, mbar_wait(&turn[t], (t == 0 ? n - 1 : n) & 1, WAIT_CYCLES));
        };
        auto pass_turn = [&]() {
            __syncwarp();
            if (paired && lane == 0) mbar_arrive(&turn[t ^ 1]);
        };
        for (uint32_t i = 0; i < turns && !__any_sync(0xffffffffu, abort_flag != 0); i++) {
            const uint32_t tile = g.per * (blockIdx.x + i * gridDim.x) + t;
            if (t >= g.per || tile >= g.tiles) break;  // (only the last turn misses a tile)
            paired = g.per == 2 && tile - t + 1 < g.tiles;
            // candidates: the tile's segment and the point's place in it
            const uint32_t sg = MODE == FWD_CANDIDATES ? segment_of(g, tile) : 0;
            const uint32_t m = MODE == FWD_CANDIDATES ? (tile - g.tile_first[sg]) * 128 + r : tile * 128 + r;
            const uint32_t m_count = MODE == FWD_CANDIDATES ? g.seg[sg].count : g.count;
            // the inputs: features [32 c, 32 c + 32) of row r of A tile 0 (K = 64)
            uint32_t p[16];
            double u_keep = 1.0;
            uint64_t cand = 0;
            if (MODE == FWD_FROM_X) {
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    const uint32_t k = 32 * c + 2 * e;
                    const float lo = (m < g.count && k < g.inputs) ? g.x[(size_t)m * g.inputs + k] : 0.0f;
                    const float hi = (m < g.count && k + 1 < g.inputs) ? g.x[(size_t)m * g.inputs + k + 1] : 0.0f;
                    p[e] = pack_bf16(lo, hi);
                }
            } else {
                // the candidate's phase-space numbers (the first 32 features have them all) and the
                // subprocess one-hot (the listed candidates are inside the cuts)
                constexpr int MAXU = pacuda::phase::MAX_UNIFORMS;
                double u[MAXU];
#pragma unroll
                for (int k = 0; k < MAXU; k++) u[k] = 0.0;
                const uint32_t nx = g.numbers;
                const bool real = m < m_count;
                if (real && c == 0) {
                    cand = g.seg[sg].index[m];
                    if (nx == 8) {
                        pacuda::phase::uniforms(g.seg[sg].seed, cand, u);
                    } else {
                        double v[pacuda::phase::Space<3>::UNIFORMS];
                        pacuda::phase::uniforms(g.seg[sg].seed, cand, v);
#pragma unroll
                        for (int k = 0; k < pacuda::phase::Space<3>::UNIFORMS; k++) u[k] = v[k];
                    }
                }
                u_keep = nx == 8 ? u[8] : u[5];
                const uint32_t family = g.seg[sg].family;
                float f[32];  // this half's 32 features (constant indices only)
#pragma unroll
                for (int k = 0; k < 32; k++) f[k] = 0.0f;
                if (c == 0 && real) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        if ((uint32_t)k < nx) f[k] = (float)u[k];
                }
#pragma unroll
                for (int k = 0; k < 32; k++)
                    if (real && 32 * c + k == nx + family) f[k] = 1.0f;
#pragma unroll
                for (int e = 0; e < 16; e++) p[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                *reinterpret_cast<uint4 *>(mine + sw128_offset(r, 32 * c + 8 * q)) =
                    make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
            fence_async_shared();
            tc_fence_before();
            mbar_arrive(&act_ready[t][0]);
            bool got = true;
            for (int layer = 0; layer < 3 && got; layer++, accs++) {
                const float *bias = prm + layer * WIDTH + 64 * c;
                uint32_t z[4][16], ph[32];
                got = __all_sync(0xffffffffu, mbar_wait(&acc_ready[t][0], accs & 1, WAIT_CYCLES));
                if (!got) break;
                tc_fence_after();
                fwd_load(lane_addr + 64 * c, z);
                if (!(got = take_turn())) break;
                fwd_activate(z, bias, ph);
                pass_turn();
                // (the second half's products have read the activations when they are done)
                got = __all_sync(0xffffffffu, mbar_wait(&acc_ready[t][1], accs & 1, WAIT_CYCLES));
                if (!got) break;
                store_row(mine + c * TILE_A, r, ph);
                fence_async_shared();
                tc_fence_before();
                mbar_arrive(&act_ready[t][0]);
                tc_fence_after();
                fwd_load(lane_addr + 128 + 64 * c, z);
                if (!(got = take_turn())) break;
                fwd_activate(z, bias + 128, ph);
                pass_turn();
                store_row(mine + (2 + c) * TILE_A, r, ph);
                fence_async_shared();
                tc_fence_before();
                mbar_arrive(&act_ready[t][1]);
            }
            // layer 4 and the output: this thread's half c, its 128 columns in order
            float out = 0.0f;
            if (got) got = __all_sync(0xffffffffu, mbar_wait(&acc_ready[t][0], accs & 1, WAIT_CYCLES));
            if (got && c == 1) got = __all_sync(0xffffffffu, mbar_wait(&acc_ready[t][1], accs & 1, WAIT_CYCLES));
            uint32_t z[4][16];
            if (got) {
                tc_fence_after();
                fwd_load(lane_addr + 128 * c, z);
                got = take_turn();
            }
            accs++;  // (the first half's threads learn of the second's products from dot_ready)
            if (!got) {
                flag_error(g.error, 205, &abort_flag);
                break;
            }
#pragma unroll
            for (int part = 0; part < 2; part++) {
                if (part == 1) fwd_load(lane_addr + 128 * c + 64, z);
                const float4 *b4 = reinterpret_cast<const float4 *>(prm + 3 * WIDTH + 128 * c + 64 * part);
                const float4 *w4 = reinterpret_cast<const float4 *>(prm + 4 * WIDTH + 128 * c + 64 * part);
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    uint32_t lo, hi;
                    fwd_activate4(&z[q / 4][4 * (q % 4)], b4[q], lo, hi);
                    const float4 ww = w4[q];
                    out = fmaf(__uint_as_float(lo << 16), ww.x, out);
                    out = fmaf(__uint_as_float(lo & 0xffff0000u), ww.y, out);
                    out = fmaf(__uint_as_float(hi << 16), ww.z, out);
                    out = fmaf(__uint_as_float(hi & 0xffff0000u), ww.w, out);
                }
            }
            pass_turn();
            // (the next tile's inputs are written after both halves of this layer's products: the first
            // half's threads wait for the second's, which have waited for them)
            tc_fence_before();
            // the two column halves' dot products meet in shared memory: the upper half's threads
            // write theirs and arrive; the lower half's wait (bounded) and finish the point. The
            // next write of dot_hi comes after this tile's reads: it needs the next tile's inputs,
            // which the lower half writes after them.
            if (c == 1) {
                dot_hi[t][r] = out;
                mbar_arrive(&dot_ready[t]);
                continue;
            }
            const bool have = __all_sync(0xffffffffu, mbar_wait(&dot_ready[t], dots & 1, WAIT_CYCLES));
            dots++;
            if (!have) {
                flag_error(g.error, 206, &abort_flag);
                break;
            }
            out += dot_hi[t][r] + prm[5 * WIDTH];
            if (MODE == FWD_FROM_X) {
                if (m < g.count) g.out[m] = out;
            } else {
                // stage 1: s = exp(mu + sigma out), the network's estimate of the weight w = |M|^2 J;
                // kept when u5 s_max < s (warp-aggregated appends)
                const pacuda_uw_segment &sgm = g.seg[sg];
                const bool real = m < m_count;
                const double sv = real ? exp(g.mu + g.sigma * (double)out) : 0.0;
                const bool keep = real && u_keep * sgm.s_max < sv;
                const unsigned ballot = __ballot_sync(0xffffffffu, keep);
                unsigned long long base = 0;
                if (lane == 0 && ballot) base = atomicAdd(sgm.kept_count, (unsigned long long)__popc(ballot));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (keep) {
                    const unsigned long long slot = base + __popc(ballot & ((1u << lane) - 1u));
                    if (slot < g.capacity) {
                        sgm.kept_index[slot] = cand;
                        sgm.kept_s[slot] = sv;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- host ---------------------------------------------------------------------------------------

const char *kTag = "pacuda surrogate";
thread_local uint32_t g_last_launches = 0;

bool failed(cudaError_t e, const char *step) {
    if (e == cudaSuccess) return false;
    fprintf(stderr, "%s: %s: %s\n", kTag, step, cudaGetErrorString(e));
    return true;
}

// tiles in flight per SM of the inference kernel: 2 or 1
int g_forward_tiles = 2;

template <int MODE>
bool launch_forward(ForwardArgs &g, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        if (failed(cudaFuncSetAttribute(forward_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM),
                   "inference kernel attributes"))
            return false;
        configured = true;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // pairs of tiles once there are more tiles than SMs (a pair takes less than two turns of one)
    g.per = g_forward_tiles == 2 && g.tiles > (uint32_t)sms ? 2 : 1;
    const uint32_t grid = std::min<uint32_t>((g.tiles + g.per - 1) / g.per, (uint32_t)sms);
    forward_kernel<MODE><<<grid, FWD_THREADS, FWD_SMEM, s>>>(g);
    g_last_launches++;
    return !failed(cudaGetLastError(), "inference launch");
}

}  // namespace

struct pacuda_sg_net {
    uint32_t inputs = 0, max_batch = 0;
    uint64_t step = 0;
    float *params = nullptr, *m1 = nullptr, *m2 = nullptr;
    uint8_t *wimg = nullptr, *wtimg = nullptr;
    // workspace for a batch
    uint8_t *x_img = nullptr, *h_img[3] = {}, *dz_img[4] = {};
    uint4 *z[3] = {};
    float *dw_part[4] = {}, *db_part[4] = {}, *dw5_part = nullptr, *scal_part = nullptr;
    int *error = nullptr;
    void *slab = nullptr;  // one allocation for all of them
};

namespace {

int refresh_images(pacuda_sg_net *n, cudaStream_t s) {
    const uint32_t count = WIDTH * IN + 3 * WIDTH * WIDTH;
    images_kernel<<<(count + 255) / 256, 256, 0, s>>>(n->params, n->wimg, n->wtimg);
    g_last_launches++;
    return failed(cudaGetLastError(), "weight images") ? ST_DEVICE : ST_OK;
}

}  // namespace

// ---- the C ABI -------------------------------------------------------------------------------------

extern "C" size_t pacuda_sg_param_count(void) { return P_COUNT; }

extern "C" uint32_t pacuda_sg_last_launches(void) { return g_last_launches; }

extern "C" int pacuda_sg_set_inference_blocks(uint32_t blocks) {
    if (blocks != 1 && blocks != 2) return ST_INVALID;
    g_forward_tiles = (int)blocks;
    return ST_OK;
}

extern "C" void pacuda_sg_destroy(pacuda_sg_net *n) {
    if (!n) return;
    cudaFree(n->slab);
    delete n;
}

extern "C" pacuda_sg_net *pacuda_sg_create(uint32_t inputs, uint32_t max_batch, uint64_t seed) {
    if (inputs == 0 || inputs > IN || max_batch == 0 || max_batch % 128) {
        fprintf(stderr, "%s: create: %u inputs (1..%d), batches of %u points (a multiple of 128)\n", kTag, inputs, IN,
                max_batch);
        return nullptr;
    }
    pacuda_sg_net *n = new pacuda_sg_net;
    n->inputs = inputs;
    n->max_batch = max_batch;
    const size_t B = max_batch, tiles = B / 128;
    std::vector<std::pair<void **, size_t>> arrays;
    size_t total = 0;
    auto array = [&](auto **p, size_t bytes) {
        arrays.push_back({(void **)p, total});
        total += (bytes + 255) / 256 * 256;
    };
    for (float **p : {&n->params, &n->m1, &n->m2}) array(p, P_COUNT * 4);
    array(&n->error, 16);
    array(&n->wimg, WIMG_BYTES);
    array(&n->wtimg, 3 * 4 * 256 * 128);
    array(&n->x_img, B * IN * 2);
    array(&n->dw5_part, tiles * WIDTH * 4);
    array(&n->scal_part, tiles * 2 * 4);
    for (int l = 0; l < 3; l++) {
        array(&n->h_img[l], B * WIDTH * 2);
        array(&n->z[l], B * WIDTH * 2);
    }
    for (int l = 0; l < 4; l++) {
        array(&n->dz_img[l], B * WIDTH * 2);
        array(&n->db_part[l], tiles * WIDTH * 4);
        array(&n->dw_part[l], (size_t)dw_parts(l, (uint32_t)tiles) * WIDTH * (l == 0 ? IN : WIDTH) * 4);
    }
    if (failed(cudaMalloc(&n->slab, total), "allocation")) {
        pacuda_sg_destroy(n);
        return nullptr;
    }
    for (auto &a : arrays) *a.first = (uint8_t *)n->slab + a.second;
    // weights uniform in +-sqrt(6 / fan_in) from a splitmix64 stream, biases zero
    std::vector<float> p(P_COUNT, 0.0f);
    uint64_t state = seed;
    auto next = [&]() {
        uint64_t z = (state += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return ((z >> 11) + 0.5) / 9007199254740992.0;
    };
    for (int l = 0; l < 5; l++) {
        const size_t at = l == 0 ? P_W1 : l == 1 ? P_W2 : l == 2 ? P_W3 : l == 3 ? P_W4 : P_W5;
        const uint32_t rows = l == 4 ? 1 : WIDTH, fan = l == 0 ? inputs : WIDTH, cols = l == 0 ? IN : WIDTH;
        const double a = std::sqrt(6.0 / fan);
        for (uint32_t o = 0; o < rows; o++)
            for (uint32_t i = 0; i < fan; i++) p[at + (size_t)o * cols + i] = (float)((2.0 * next() - 1.0) * a);
    }
    if (pacuda_sg_set_params(n, p.data()) != ST_OK) {
        pacuda_sg_destroy(n);
        return nullptr;
    }
    return n;
}

extern "C" int pacuda_sg_set_params(pacuda_sg_net *n, const float *params) {
    g_last_launches = 0;
    if (!n || !params) return ST_INVALID;
    std::vector<float> p(params, params + P_COUNT);
    for (uint32_t o = 0; o < WIDTH; o++)
        for (uint32_t i = n->inputs; i < IN; i++) p[P_W1 + (size_t)o * IN + i] = 0.0f;
    if (failed(cudaMemcpy(n->params, p.data(), P_COUNT * 4, cudaMemcpyHostToDevice), "parameters") ||
        failed(cudaMemset(n->m1, 0, P_COUNT * 4), "moments") || failed(cudaMemset(n->m2, 0, P_COUNT * 4), "moments") ||
        failed(cudaMemset(n->error, 0, 16), "error flag") || failed(cudaMemset(n->wimg, 0, WIMG_BYTES), "images"))
        return ST_DEVICE;
    n->step = 0;
    if (refresh_images(n, 0) != ST_OK || failed(cudaDeviceSynchronize(), "images")) return ST_DEVICE;
    return ST_OK;
}

extern "C" int pacuda_sg_get_params(const pacuda_sg_net *n, float *params) {
    if (!n || !params) return ST_INVALID;
    return failed(cudaMemcpy(params, n->params, P_COUNT * 4, cudaMemcpyDeviceToHost), "parameters") ? ST_DEVICE : ST_OK;
}

namespace {

template <class F> bool allow_shared(F *kernel, uint32_t bytes, const char *what) {
    return !failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), what);
}

// launches `kernel` so that it may be set up while the stream's kernel before it ends (grid_wait)
template <class A>
bool launch_early(void (*kernel)(A), uint32_t blocks, uint32_t threads, uint32_t shared, cudaStream_t s, const A &args, const char *what) {
    cudaLaunchAttribute early;
    memset(&early, 0, sizeof early);
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c;
    memset(&c, 0, sizeof c);
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = shared;
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    g_last_launches++;
    return !failed(cudaLaunchKernelEx(&c, kernel, args), what);
}

// the forward and backward chain and the weight gradients' partials of one batch; `u` gets what the
// update reads of them
int products(pacuda_sg_net *n, const float *x, const float *y, uint32_t batch, UpdateArgs &u, cudaStream_t s) {
    if (!n || !x || !y || batch == 0 || batch % 128 || batch > n->max_batch) {
        fprintf(stderr, "%s: a batch of %u points (a multiple of 128, at most %u)\n", kTag, batch, n ? n->max_batch : 0);
        return ST_INVALID;
    }
    static bool configured = false;
    if (!configured) {
        if (!allow_shared(chain_kernel, CH_SMEM, "chain attributes") || !allow_shared(dw_kernel, DW_SMEM, "weight gradient attributes"))
            return ST_DEVICE;
        configured = true;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t tiles = batch / 128;
    ChainArgs c;
    DwArgs d;
    memset(&u, 0, sizeof u);
    c.wimg = n->wimg;
    c.wtimg = n->wtimg;
    c.params = n->params;
    c.x = x;
    c.y = y;
    c.inputs = n->inputs;
    c.tiles = d.tiles = u.tiles = tiles;
    c.inv_batch = 1.0f / (float)batch;
    c.x_img = n->x_img;
    d.x_img = n->x_img;
    for (int l = 0; l < 3; l++) {
        c.h_img[l] = n->h_img[l];
        d.h_img[l] = n->h_img[l];
        c.z[l] = n->z[l];
    }
    for (int l = 0; l < 4; l++) {
        c.dz_img[l] = n->dz_img[l];
        d.dz_img[l] = n->dz_img[l];
        c.db[l] = n->db_part[l];
        u.db[l] = n->db_part[l];
        d.partial[l] = n->dw_part[l];
        u.dw[l] = n->dw_part[l];
    }
    c.dw5 = n->dw5_part;
    u.dw5 = n->dw5_part;
    c.scalars = n->scal_part;
    u.scalars = n->scal_part;
    c.error = d.error = n->error;
    return launch_early(chain_kernel, std::min(tiles, (uint32_t)sms), CH_THREADS, CH_SMEM, s, c, "forward and backward") &&
                   launch_early(dw_kernel, 6 * dw_parts(1, tiles) + 2 * dw_parts(0, tiles), 256, DW_SMEM, s, d, "weight gradients")
               ? ST_OK
               : ST_DEVICE;
}

// the gradient of one batch into `grad` (UP_GRADIENT), the Adam step on it (UP_TRAIN), or on a given
// gradient (UP_APPLY)
template <int MODE> int update(pacuda_sg_net *n, UpdateArgs &u, float lr, cudaStream_t s) {
    u.params = n->params;
    u.m1 = n->m1;
    u.m2 = n->m2;
    u.wimg = n->wimg;
    u.wtimg = n->wtimg;
    u.inputs = n->inputs;
    if (MODE != UP_GRADIENT) {
        n->step++;
        u.lr = lr;
        u.c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)n->step)));
        u.c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)n->step)));
    }
    if (MODE != UP_APPLY) return launch_early(update_kernel<MODE>, UP_BLOCKS, 256, 0, s, u, "update") ? ST_OK : ST_DEVICE;
    // (a call of its own, after whatever the caller queued)
    update_kernel<MODE><<<UP_BLOCKS, 256, 0, s>>>(u);
    g_last_launches++;
    return failed(cudaGetLastError(), "update") ? ST_DEVICE : ST_OK;
}

}  // namespace

extern "C" int pacuda_sg_gradients(pacuda_sg_net *n, const float *x, const float *y, uint32_t batch, float *grad,
                                   float *loss, void *stream) {
    g_last_launches = 0;
    if (!grad) return ST_INVALID;
    UpdateArgs u;
    int st = products(n, x, y, batch, u, (cudaStream_t)stream);
    if (st != ST_OK) return st;
    u.grad = grad;
    u.loss = loss;
    return update<UP_GRADIENT>(n, u, 0.0f, (cudaStream_t)stream);
}

extern "C" int pacuda_sg_apply_gradients(pacuda_sg_net *n, const float *grad, float lr, void *stream) {
    g_last_launches = 0;
    if (!n || !grad) return ST_INVALID;
    UpdateArgs u;
    memset(&u, 0, sizeof u);
    u.grad = const_cast<float *>(grad);
    return update<UP_APPLY>(n, u, lr, (cudaStream_t)stream);
}

extern "C" int pacuda_sg_train_step(pacuda_sg_net *n, const float *x, const float *y, uint32_t batch, float lr,
                                    float *loss_sum, void *stream) {
    g_last_launches = 0;
    UpdateArgs u;
    int st = products(n, x, y, batch, u, (cudaStream_t)stream);
    if (st != ST_OK) return st;
    u.loss_sum = loss_sum;
    return update<UP_TRAIN>(n, u, lr, (cudaStream_t)stream);
}

extern "C" int pacuda_sg_forward(const pacuda_sg_net *n, const float *x, uint32_t count, float *out, void *stream) {
    g_last_launches = 0;
    if (!n || !x || !out || count == 0) return ST_INVALID;
    ForwardArgs g;
    memset(&g, 0, sizeof g);
    g.wimg = n->wimg;
    g.params = n->params;
    g.x = x;
    g.inputs = n->inputs;
    g.count = count;
    g.tiles = (count + 127) / 128;
    g.out = out;
    g.error = n->error;
    return launch_forward<FWD_FROM_X>(g, (cudaStream_t)stream) ? ST_OK : ST_DEVICE;
}

// the error flag of the network's kernels (0: none), for tests and callers that check after a run
extern "C" int pacuda_sg_error(const pacuda_sg_net *n) {
    int e = 0;
    if (!n || failed(cudaMemcpy(&e, n->error, sizeof e, cudaMemcpyDeviceToHost), "error flag")) return -1;
    return e;
}

// ---- two-stage unweighting ------------------------------------------------------------------------

namespace {

using pacuda::phase::Cuts;
using pacuda::phase::Map;
using pacuda::phase::Space;

// The candidates first .. first + count - 1 of one stream: the indices of those inside the cuts,
// appended (unordered) to index[] while below `capacity`; *count_out counts all of them. A block takes
// LIST_ROUNDS x 256 consecutive candidates (candidate k of the block in round k / 256 on thread
// k % 256): each thread gives its candidates the f32 first look (phase.cuh look32), which drops what
// surely fails and lists what surely passes; the rest are gathered in shared memory, and then the
// block's threads take those through the f64 map and cuts, which decide (gathering several rounds
// keeps the f64 pass's warps full). The block's list goes out in one piece: one counter atomic.
// What bounds it is arithmetic: the f32 look and the f64 map (FP64 and f64 functions) of the
// candidates that the look leaves open. 2^22 candidates of g g -> 3 g, 28 % of them inside the cuts:
// 216 us when the look only dropped and each candidate inside went through the f64 map, 128 now; of
// g g -> 4 g, 6 % inside: 218 -> 202. (Blocks of 256 threads: the kernels below are launched so.)
constexpr uint32_t LIST_ROUNDS = 16, LIST_BLOCK = 256 * LIST_ROUNDS;

// the positions of a warp's lanes with `set` in a list that *n (shared memory) counts
__device__ __forceinline__ uint32_t list_place(bool set, uint32_t *n) {
    const int lane = threadIdx.x & 31;
    const unsigned ballot = __ballot_sync(0xffffffffu, set);
    uint32_t base = 0;
    if (lane == 0 && ballot) base = atomicAdd(n, (uint32_t)__popc(ballot));
    return __shfl_sync(0xffffffffu, base, 0) + __popc(ballot & ((1u << lane) - 1u));
}

template <int N>
__device__ __forceinline__ void list_block(uint64_t seed, uint64_t first, uint32_t count, double sqrt_s,
                                           const Cuts &cuts, uint64_t *index, uint32_t capacity,
                                           unsigned long long *count_out, uint32_t block_first) {
    constexpr int F = N, L = Space<N>::LEGS;
    __shared__ uint16_t unsure[LIST_BLOCK], listed[LIST_BLOCK];  // (a block's candidates, by their place in it)
    __shared__ uint32_t n_unsure, n_listed;
    __shared__ unsigned long long out;
    if (threadIdx.x == 0) n_unsure = n_listed = 0;
    __syncthreads();
    for (uint32_t r = 0; r < LIST_ROUNDS; r++) {
        const uint32_t at = r * 256 + threadIdx.x;
        const uint64_t i = (uint64_t)block_first + at;
        pacuda::phase::Look look = pacuda::phase::LOOK_FAILS;
        if (i < count) {
            float u[Space<N>::NUMBERS], q[F][3];
            pacuda::phase::uniforms32(seed, first + i, u);
            pacuda::phase::final32(u, sqrt_s, q);
            look = pacuda::phase::look32(q, sqrt_s, cuts);
        }
        const uint32_t l = list_place(look == pacuda::phase::LOOK_PASSES, &n_listed);
        if (look == pacuda::phase::LOOK_PASSES) listed[l] = (uint16_t)at;
        const uint32_t m = list_place(look == pacuda::phase::LOOK_UNSURE, &n_unsure);
        if (look == pacuda::phase::LOOK_UNSURE) unsure[m] = (uint16_t)at;
    }
    __syncthreads();
    const uint32_t m = n_unsure;
    for (uint32_t k = threadIdx.x; k < ((m + 31u) & ~31u); k += 256) {  // (whole warps)
        bool pass = false;
        uint32_t at = 0;
        if (k < m) {
            at = unsure[k];
            double u[Space<N>::UNIFORMS], p[L][4];
            pacuda::phase::uniforms(seed, first + block_first + at, u);
            Map<N>::momenta(u, sqrt_s, p);
            pass = pacuda::phase::passes(p, cuts);
        }
        const uint32_t l = list_place(pass, &n_listed);
        if (pass) listed[l] = (uint16_t)at;
    }
    __syncthreads();
    const uint32_t n = n_listed;
    if (threadIdx.x == 0 && n) out = atomicAdd(count_out, (unsigned long long)n);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n; k += 256)
        if (out + k < capacity) index[out + k] = first + block_first + listed[k];
}

template <int N>
__global__ void __launch_bounds__(256) candidates_kernel(uint64_t seed, uint64_t first, uint32_t count, double sqrt_s,
                                                         Cuts cuts, uint64_t *index, uint32_t capacity,
                                                         unsigned long long *count_out) {
    list_block<N>(seed, first, count, sqrt_s, cuts, index, capacity, count_out, blockIdx.x * LIST_BLOCK);
}

// several subprocesses' candidates in one launch: block b lists segment k's candidates when
// block_first[k] <= b < block_first[k + 1]
struct CandidateSegments {
    pacuda_uw_candidate_segment seg[PACUDA_UW_MAX_SEGMENTS];
    uint32_t block_first[PACUDA_UW_MAX_SEGMENTS + 1];
    uint32_t segments;
};

template <int N>
__global__ void __launch_bounds__(256) candidate_segments_kernel(CandidateSegments c, double sqrt_s, Cuts cuts,
                                                                 uint32_t capacity) {
    uint32_t k = 0;
    while (k + 1 < c.segments && blockIdx.x >= c.block_first[k + 1]) k++;
    const pacuda_uw_candidate_segment &sg = c.seg[k];
    list_block<N>(sg.seed, sg.first, sg.count, sqrt_s, cuts, sg.index, capacity, sg.counter,
                  (blockIdx.x - c.block_first[k]) * LIST_BLOCK);
}

// the points of candidates index[0..n): source-major momenta [(leg * 4 + k) * n + i] for the
// runner, the network's inputs [i][inputs] (the phase-space numbers, then the family's one-hot)
// and the map's weight
template <int N>
__global__ void points_kernel(uint64_t seed, const uint64_t *index, uint32_t n, double sqrt_s, double *momenta,
                              float *inputs_out, uint32_t inputs, uint32_t family, double *jac) {
    constexpr int X = Space<N>::NUMBERS, L = Space<N>::LEGS;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double u[Space<N>::UNIFORMS], p[L][4];
    pacuda::phase::uniforms(seed, index[i], u);
    const double j = Map<N>::momenta(u, sqrt_s, p);
    if (momenta)
        for (int leg = 0; leg < L; leg++)
            for (int k = 0; k < 4; k++) momenta[(size_t)(leg * 4 + k) * n + i] = p[leg][k];
    if (inputs_out)
        for (uint32_t f = 0; f < inputs; f++)
            inputs_out[(size_t)i * inputs + f] = f < (uint32_t)X ? (float)u[f] : (f == X + family ? 1.0f : 0.0f);
    if (jac) jac[i] = j;
}

// |M|^2 = the sum of the runner's helicity outputs, w = |M|^2 J, and the accept/reject decision
// (u_a, u_b: the candidate's two decision uniforms, after its phase-space numbers):
// plain (s == null): kept when u_a w_max < w, weight max(1, w / w_max);
// second stage: r = w / s, kept when u_b r_max < r, weight max(1, s / s_max) max(1, r / r_max)
template <int N>
__global__ void decide_kernel(uint64_t seed, const uint64_t *index, uint32_t n, const double *outputs, uint32_t helicities,
                              const double *jac, const double *s, double w_max, double s_max, double r_max, uint8_t *keep,
                              double *weight, double *me) {
    constexpr int X = Space<N>::NUMBERS;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double m2 = 0.0;
    for (uint32_t h = 0; h < helicities; h++) m2 += outputs[(size_t)i * helicities + h];
    const double w = m2 * jac[i];
    double u[Space<N>::UNIFORMS];
    pacuda::phase::uniforms(seed, index[i], u);
    bool k;
    double wt;
    if (!s) {
        k = u[X] * w_max < w;
        wt = k ? fmax(1.0, w / w_max) : 0.0;
    } else {
        const double r = w / s[i];
        k = u[X + 1] * r_max < r;
        wt = k ? fmax(1.0, s[i] / s_max) * fmax(1.0, r / r_max) : 0.0;
    }
    if (keep) keep[i] = k;
    if (weight) weight[i] = wt;
    if (me) me[i] = m2;
}

bool final_state_valid(uint32_t n) { return n == 3 || n == 4; }

}  // namespace

extern "C" int pacuda_uw_candidates(uint64_t seed, uint64_t first, uint32_t count, uint32_t final_state, double sqrt_s,
                                    const pacuda_uw_cuts *cuts, uint64_t *index, uint32_t capacity,
                                    unsigned long long *counter, void *stream) {
    g_last_launches = 0;
    if (!cuts || !index || !counter || count == 0 || !(sqrt_s > 0) || !final_state_valid(final_state)) return ST_INVALID;
    Cuts c{cuts->pt_min, cuts->eta_max, cuts->dr_min};
    const dim3 grid((count + LIST_BLOCK - 1) / LIST_BLOCK);
    if (final_state == 4)
        candidates_kernel<4><<<grid, 256, 0, (cudaStream_t)stream>>>(seed, first, count, sqrt_s, c, index, capacity, counter);
    else
        candidates_kernel<3><<<grid, 256, 0, (cudaStream_t)stream>>>(seed, first, count, sqrt_s, c, index, capacity, counter);
    g_last_launches++;
    return failed(cudaGetLastError(), "candidates") ? ST_DEVICE : ST_OK;
}

extern "C" int pacuda_uw_candidates_segments(const pacuda_uw_candidate_segment *segs, uint32_t segments,
                                             uint32_t final_state, double sqrt_s, const pacuda_uw_cuts *cuts,
                                             uint32_t capacity, void *stream) {
    g_last_launches = 0;
    if (!segs || !cuts || segments == 0 || segments > PACUDA_UW_MAX_SEGMENTS || !(sqrt_s > 0) ||
        !final_state_valid(final_state))
        return ST_INVALID;
    CandidateSegments c;
    memset(&c, 0, sizeof c);
    uint32_t blocks = 0;
    for (uint32_t k = 0; k < segments; k++) {
        if ((segs[k].count && !segs[k].index) || !segs[k].counter) return ST_INVALID;
        c.seg[k] = segs[k];
        c.block_first[k] = blocks;
        blocks += (segs[k].count + LIST_BLOCK - 1) / LIST_BLOCK;
    }
    c.block_first[segments] = blocks;
    c.segments = segments;
    if (blocks == 0) return ST_OK;
    const Cuts cc{cuts->pt_min, cuts->eta_max, cuts->dr_min};
    if (final_state == 4)
        candidate_segments_kernel<4><<<blocks, 256, 0, (cudaStream_t)stream>>>(c, sqrt_s, cc, capacity);
    else
        candidate_segments_kernel<3><<<blocks, 256, 0, (cudaStream_t)stream>>>(c, sqrt_s, cc, capacity);
    g_last_launches++;
    return failed(cudaGetLastError(), "candidates") ? ST_DEVICE : ST_OK;
}

extern "C" int pacuda_uw_points(uint64_t seed, const uint64_t *index, uint32_t n, uint32_t final_state, double sqrt_s,
                                double *momenta, float *inputs, uint32_t input_count, uint32_t family, double *jac,
                                void *stream) {
    g_last_launches = 0;
    const uint32_t x = 3 * final_state - 4;
    if (!index || n == 0 || !(sqrt_s > 0) || !final_state_valid(final_state) ||
        (inputs && (input_count < x || input_count > IN || x + family >= input_count)))
        return ST_INVALID;
    const dim3 grid((n + 127) / 128);
    if (final_state == 4)
        points_kernel<4><<<grid, 128, 0, (cudaStream_t)stream>>>(seed, index, n, sqrt_s, momenta, inputs, input_count,
                                                                  family, jac);
    else
        points_kernel<3><<<grid, 128, 0, (cudaStream_t)stream>>>(seed, index, n, sqrt_s, momenta, inputs, input_count,
                                                                  family, jac);
    g_last_launches++;
    return failed(cudaGetLastError(), "points") ? ST_DEVICE : ST_OK;
}

extern "C" int pacuda_uw_decide(uint64_t seed, const uint64_t *index, uint32_t n, uint32_t final_state,
                                const double *outputs, uint32_t helicities, const double *jac, const double *s,
                                double w_max, double s_max, double r_max, uint8_t *keep, double *weight, double *me,
                                void *stream) {
    g_last_launches = 0;
    if (!index || !outputs || !jac || helicities == 0 || !final_state_valid(final_state)) return ST_INVALID;
    if (n == 0) return ST_OK;
    const dim3 grid((n + 127) / 128);
    if (final_state == 4)
        decide_kernel<4><<<grid, 128, 0, (cudaStream_t)stream>>>(seed, index, n, outputs, helicities, jac, s, w_max,
                                                                  s_max, r_max, keep, weight, me);
    else
        decide_kernel<3><<<grid, 128, 0, (cudaStream_t)stream>>>(seed, index, n, outputs, helicities, jac, s, w_max,
                                                                  s_max, r_max, keep, weight, me);
    g_last_launches++;
    return failed(cudaGetLastError(), "decide") ? ST_DEVICE : ST_OK;
}

extern "C" int pacuda_uw_stage1_segments(const pacuda_sg_net *n, const pacuda_uw_segment *segs, uint32_t segments,
                                         uint32_t final_state, double mu, double sigma, uint32_t capacity,
                                         void *stream) {
    g_last_launches = 0;
    if (!n || !segs || segments == 0 || segments > PACUDA_UW_MAX_SEGMENTS || !final_state_valid(final_state)) {
        fprintf(stderr, "%s: stage 1: 1 to %d segments of 3 or 4 final-state partons\n", kTag, PACUDA_UW_MAX_SEGMENTS);
        return ST_INVALID;
    }
    const uint32_t x = 3 * final_state - 4;
    ForwardArgs g;
    memset(&g, 0, sizeof g);
    uint32_t tiles = 0;
    for (uint32_t k = 0; k < segments; k++) {
        const pacuda_uw_segment &sg = segs[k];
        if ((sg.count && !sg.index) || !sg.kept_index || !sg.kept_s || !sg.kept_count || x + sg.family >= n->inputs) {
            fprintf(stderr, "%s: stage 1: segment %u: a missing array or a family beyond the inputs\n", kTag, k);
            return ST_INVALID;
        }
        g.seg[k] = sg;
        g.tile_first[k] = tiles;
        tiles += (sg.count + 127) / 128;
    }
    g.tile_first[segments] = tiles;
    if (tiles == 0) return ST_OK;
    g.segments = segments;
    g.wimg = n->wimg;
    g.params = n->params;
    g.inputs = n->inputs;
    g.tiles = tiles;
    g.error = n->error;
    g.mu = mu;
    g.sigma = sigma;
    g.capacity = capacity;
    g.numbers = x;
    return launch_forward<FWD_CANDIDATES>(g, (cudaStream_t)stream) ? ST_OK : ST_DEVICE;
}

extern "C" int pacuda_uw_stage1(const pacuda_sg_net *n, uint64_t seed, const uint64_t *index, uint32_t count,
                                uint32_t final_state, uint32_t family, double mu, double sigma, double s_max,
                                uint64_t *kept_index, double *kept_s, uint32_t capacity, unsigned long long *counter,
                                void *stream) {
    pacuda_uw_segment sg;
    sg.seed = seed;
    sg.index = index;
    sg.count = count;
    sg.family = family;
    sg.s_max = s_max;
    sg.kept_index = kept_index;
    sg.kept_s = kept_s;
    sg.kept_count = counter;
    if (!index) return ST_INVALID;
    return pacuda_uw_stage1_segments(n, &sg, 1, final_state, mu, sigma, capacity, stream);
}
