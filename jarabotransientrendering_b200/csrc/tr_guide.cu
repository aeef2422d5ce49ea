// tr_guide.cu - kernels of the learned directional proposal (no reference counterpart).
//
// The network is 64 -> 64 -> 64 -> 64 -> 40 (ReLU on the three hidden layers), BF16 operands,
// FP32 accumulation.  Forward and the hidden-layer backward run on the 5th-generation tensor
// cores: one CTA of 128 threads owns a 128-row tile; all four weight tiles stay resident in
// shared memory in the UMMA canonical K-major layout (8x16-byte core matrices, no swizzle);
// one elected thread issues tcgen05.mma (M=128, N=64, K=16, four per layer) into a 128x64 FP32
// accumulator in tensor memory; tcgen05.commit arrives on an mbarrier; every thread then reads
// its row back with tcgen05.ld, adds the bias, applies ReLU and writes the BF16 row as the next
// layer's A operand.  The weight gradients (a reduction over the batch, 2 GFLOP per 65,536-row
// step) run on the tensor cores too (k_dw_tc).  Every wait on an mbarrier is bounded (the
// guide's wait limit); on expiry the kernel records an error, waits (bounded) for its MMAs,
// frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <algorithm>

#include "tr_guide.cuh"
#include "tr_guide_math.cuh"
#include "tr_tcgen05.cuh"

namespace trg {


// ---------------------------------------------------------------------------------------------
// forward: out[m][0..40) = L4(relu(L3(relu(L2(relu(L1(x)))))))
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 4) k_mlp_fwd(GuideDev g, const uint4* __restrict__ x, uint32_t m,
                                                    float* __restrict__ out, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem + kSmemA;
    const float* sB = reinterpret_cast<const float*>(smem + kSmemBias);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kSmemBar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(smem + kSmemSlot);
    volatile int* s_ok = reinterpret_cast<volatile int*>(smem + kSmemOk);
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    stage_weights(smem, g.w_fwd, g.bias);
    if (tid == 0) { mbar_init(bar, 1); fence_mbar_init(); }
    if (warp == 0) { tmem_alloc(slot, 64); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *slot;
    const uint32_t lane_addr = taddr + ((32u * warp) << 16);
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t tile = blockIdx.x; tile * kTile < m && ok; tile += gridDim.x) {
        const uint32_t row = tile * kTile + tid;
        uint4 v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = row < m ? __ldg(&x[(size_t)row * 8 + c]) : make_uint4(0, 0, 0, 0);
        store_row_a(sA, tid, v);
        for (uint32_t l = 0; l < 4 && ok; ++l) {
            ok = layer_mma(taddr, smem_u32(sA), smem_u32(smem + kSmemW + l * 8192u), bar, phase, s_ok, g.spin);
            if (!ok) break;
            float acc[64];
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld16(lane_addr + 16u * j, acc + 16 * j);
            tmem_wait_ld();
            if (l < 3) {
                uint4 h[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float t[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) t[e] = acc[8 * c + e] + sB[l * 64 + 8 * c + e];
                    h[c] = make_uint4(pack2_relu(t[0], t[1]), pack2_relu(t[2], t[3]), pack2_relu(t[4], t[5]),
                                      pack2_relu(t[6], t[7]));
                }
                store_row_a(sA, tid, h);
            } else if (row < m) {
#pragma unroll
                for (int j = 0; j < kOut; ++j) out[(size_t)row * kOut + j] = acc[j] + sB[3 * 64 + j];
            }
        }
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    drain_and_free(taddr, bar, phase, ok);
}

// ---------------------------------------------------------------------------------------------
// One training tile of 128 rows: forward (H1..H3 kept for the weight gradients), the mixture loss and
// its gradient w.r.t. the outputs (dy), backward through the hidden layers with the transposed weights
// (dh[2] = dH3 = (dy W4^T) * 1[H3 > 0], dh[1] = dH2, dh[0] = dH1), all BF16.  A thread owns a row: its
// outputs and ReLU masks stay in registers between the passes.  The weight buffer holds the forward
// tiles first, then the backward ones, so four CTAs fit on an SM and a 65,536-row batch is one wave.
// Bound by the latency of its seven MMA chains: 41 us per 65,536 rows (three kernels that passed
// outputs, activations and gradients through memory took 88 us; with rows stored and masks re-read by
// their own threads 57 us).  loss_part[tile] = the tile's loss.
// ---------------------------------------------------------------------------------------------
constexpr int kSumBlocks = 64;
__device__ __forceinline__ void grad_row(const float* o, float dx, float dyy, float dz, float scale, float& loss, float* g) {
    Lobe L[kLobes];
    decode_mixture(o, L);
    float lg[kLobes], cs[kLobes];
    float lmax = -3.4e38f;
#pragma unroll
    for (int j = 0; j < kLobes; ++j) {
        cs[j] = L[j].mx * dx + L[j].my * dyy + L[j].mz * dz;
        lg[j] = logf(fmaxf(L[j].pi, 1e-30f)) + log_vmf(L[j].kappa, cs[j]);
        lmax = fmaxf(lmax, lg[j]);
    }
    float se = 0.0f;
#pragma unroll
    for (int j = 0; j < kLobes; ++j) se += expf(lg[j] - lmax);
    const float logq = lmax + logf(se);
    loss = -scale * logq;
#pragma unroll
    for (int j = 0; j < kLobes; ++j) {
        const float r = expf(lg[j] - logq);                 // responsibility
        const float kap = L[j].kappa;
        g[5 * j] = -scale * (r - L[j].pi);                  // d(-log q)/d logit
        const float c = r * kap / L[j].mnorm;
        g[5 * j + 1] = -scale * c * (dx - cs[j] * L[j].mx);
        g[5 * j + 2] = -scale * c * (dyy - cs[j] * L[j].my);
        g[5 * j + 3] = -scale * c * (dz - cs[j] * L[j].mz);
        const float e2 = expf(-2.0f * kap);
        const float dlogv = 1.0f / kap - 2.0f * e2 / (1.0f - e2) + (cs[j] - 1.0f);
        g[5 * j + 4] = -scale * r * dlogv * L[j].sig;
    }
}

// The calling warp's 32 rows of the A tile to rows [row0, row0 + 32) of a [m][64] bf16 array: 8 rows x 64
// bytes per store (a thread storing its own row touches a line per lane and store).
__device__ __forceinline__ void copy_rows(const uint8_t* sA, uint4* __restrict__ to, uint32_t row0, uint32_t m) {
    const uint32_t lane = threadIdx.x & 31u, r8 = lane & 7u, c4 = lane >> 3, w = threadIdx.x >> 5;
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t rg = i >> 1, c = (i & 1u) * 4u + c4, row = row0 + rg * 8u + r8;
        const uint4 v = *reinterpret_cast<const uint4*>(sA + (4u * w + rg) * 1024u + c * 128u + r8 * 16u);
        if (row < m) to[(size_t)row * 8 + c] = v;
    }
}

__global__ void __launch_bounds__(128, 4) k_train_tile(GuideDev g, const uint4* __restrict__ x, const float* __restrict__ dirs,
                                                       const float* __restrict__ w, const float* __restrict__ wsum_part,
                                                       uint32_t m, uint4* __restrict__ act, uint4* __restrict__ dy,
                                                       uint4* __restrict__ dh, float* __restrict__ loss_part, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem + kSmemA;
    const float* sB = reinterpret_cast<const float*>(smem + kSmemBias);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kSmemBar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(smem + kSmemSlot);
    volatile int* s_ok = reinterpret_cast<volatile int*>(smem + kSmemOk);
    __shared__ float s_wsum, s_loss[4];
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) { mbar_init(bar, 1); fence_mbar_init(); }
    if (warp == 0) {
        tmem_alloc(slot, 64);
        tmem_relinquish();
        // the batch's weight sum, from its blocks' sums in a fixed order
        float t = wsum_part[tid] + wsum_part[tid + 32u];
        for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        if (tid == 0) s_wsum = t;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *slot;
    const uint32_t lane_addr = taddr + ((32u * warp) << 16);
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t tile = blockIdx.x; tile * kTile < m && ok; tile += gridDim.x) {
        const uint32_t row = tile * kTile + tid, row0 = tile * kTile + 32u * warp;
        uint32_t alive[3][2];                // bit u: the row's unit u of H1..H3 is above zero
        stage_weights(smem, g.w_fwd, g.bias);
        {
            uint4 v[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = row < m ? __ldg(&x[(size_t)row * 8 + c]) : make_uint4(0, 0, 0, 0);
            store_row_a(sA, tid, v);
        }
#pragma unroll
        for (uint32_t l = 0; l < 3; ++l) {
            if (!ok) break;
            ok = layer_mma(taddr, smem_u32(sA), smem_u32(smem + kSmemW + l * 8192u), bar, phase, s_ok, g.spin);
            if (!ok) break;
            float acc[64];
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld16(lane_addr + 16u * j, acc + 16 * j);
            tmem_wait_ld();
            uint4 h[8];
            alive[l][0] = alive[l][1] = 0u;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                uint32_t hw[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = 8 * c + 2 * e;
                    hw[e] = pack2_relu(acc[k] + sB[l * 64 + k], acc[k + 1] + sB[l * 64 + k + 1]);
                    if (bf_lo(hw[e]) > 0.0f) alive[l][c >> 2] |= 1u << (k & 31);
                    if (bf_hi(hw[e]) > 0.0f) alive[l][c >> 2] |= 2u << (k & 31);
                }
                h[c] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
            }
            store_row_a(sA, tid, h);
            copy_rows(sA, act + (size_t)l * m * 8, row0, m);
        }
        if (ok) ok = layer_mma(taddr, smem_u32(sA), smem_u32(smem + kSmemW + 3u * 8192u), bar, phase, s_ok, g.spin);
        if (!ok) break;
        // the forward MMAs are done with the weight buffer
        {
            uint4* sw = reinterpret_cast<uint4*>(smem + kSmemW);
            for (uint32_t i = 512u + tid; i < 2048u; i += 128u) sw[i] = __ldg(&g.w_bwd[i]);
        }
        float gr[64];
        float loss = 0.0f;
#pragma unroll
        for (int k = 0; k < 64; ++k) gr[k] = 0.0f;
        {
            float o[48];
#pragma unroll
            for (int j = 0; j < 3; ++j) tmem_ld16(lane_addr + 16u * j, o + 16 * j);
            tmem_wait_ld();
            if (row < m) {
#pragma unroll
                for (int j = 0; j < kOut; ++j) o[j] += sB[3 * 64 + j];
                grad_row(o, dirs[3 * (size_t)row], dirs[3 * (size_t)row + 1], dirs[3 * (size_t)row + 2],
                         w[row] / fmaxf(s_wsum, 1e-30f), loss, gr);
            }
        }
        uint4 h[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            h[c] = make_uint4(pack2(gr[8 * c], gr[8 * c + 1]), pack2(gr[8 * c + 2], gr[8 * c + 3]),
                              pack2(gr[8 * c + 4], gr[8 * c + 5]), pack2(gr[8 * c + 6], gr[8 * c + 7]));
        }
        store_row_a(sA, tid, h);
        copy_rows(sA, dy, row0, m);
        for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
        if ((tid & 31u) == 0) s_loss[warp] = loss;
        // layer index of the weights used: 3 (W4), 2 (W3), 1 (W2); activation masks H3, H2, H1
#pragma unroll
        for (int l = 3; l >= 1; --l) {
            if (!ok) break;
            ok = layer_mma(taddr, smem_u32(sA), smem_u32(smem + kSmemW + (uint32_t)l * 8192u), bar, phase, s_ok, g.spin);
            if (!ok) break;
            float acc[64];
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld16(lane_addr + 16u * j, acc + 16 * j);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 64; ++k) acc[k] = (alive[l - 1][k >> 5] >> (k & 31)) & 1u ? acc[k] : 0.0f;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                h[c] = make_uint4(pack2(acc[8 * c], acc[8 * c + 1]), pack2(acc[8 * c + 2], acc[8 * c + 3]),
                                  pack2(acc[8 * c + 4], acc[8 * c + 5]), pack2(acc[8 * c + 6], acc[8 * c + 7]));
            store_row_a(sA, tid, h);
            copy_rows(sA, dh + (size_t)(l - 1) * m * 8, row0, m);
            if (l == 3 && tid == 0) loss_part[tile] = (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]);
        }
        __syncthreads();                  // the weight buffer and s_loss are taken again
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    drain_and_free(taddr, bar, phase, ok);
}

int resident_grid(int device, const void* kernel, int threads, size_t dyn_smem, int tmem_cols) {
    int sms = 1, smem_sm = 0, regs_sm = 0, warps_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, device);
    cudaDeviceGetAttribute(&warps_sm, cudaDevAttrMaxThreadsPerMultiProcessor, device);
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return sms > 0 ? sms : 1;
    const int per_cta_smem = (int)dyn_smem + (int)fa.sharedSizeBytes + 1024;     // 1 KB reserved per CTA
    const int regs = fa.numRegs > 0 ? ((fa.numRegs + 7) / 8) * 8 : 1;
    int per_sm = std::min(smem_sm / per_cta_smem, regs_sm / (regs * threads));
    per_sm = std::min(per_sm, warps_sm / threads);
    per_sm = std::min(per_sm, 512 / tmem_cols);                                   // TMEM columns each
    if (per_sm < 1) per_sm = 1;
    return (sms > 0 ? sms : 1) * per_sm;
}

int mlp_grid(int device) {
    static int grid = 0;
    if (!grid) grid = resident_grid(device, reinterpret_cast<const void*>(k_mlp_fwd), 128, kSmemBytes);
    return grid;
}

static int train_grid(int device) {
    static int grid = 0;
    if (!grid) grid = resident_grid(device, reinterpret_cast<const void*>(k_train_tile), 128, kSmemBytes);
    return grid;
}

cudaError_t mlp_forward(const GuideDev& g, const uint4* x, uint32_t m, float* out, int* err, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        attr = true;
    }
    if (m == 0) return cudaSuccess;
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t tiles = (m + kTile - 1) / kTile;
    const uint32_t grid = tiles < (uint32_t)mlp_grid(dev) ? tiles : (uint32_t)mlp_grid(dev);
    k_mlp_fwd<<<grid, 128, kSmemBytes, s>>>(g, x, m, out, err);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// parameters: master FP32 [4][64 in][64 out] weights + [4][64] biases; packed BF16 tiles
// ---------------------------------------------------------------------------------------------
__global__ void k_pack_weights(const float* __restrict__ params, uint8_t* __restrict__ w_fwd, uint8_t* __restrict__ w_bwd) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;          // one weight element
    if (i >= 4u * 4096u) return;
    const uint32_t l = i >> 12, in = (i >> 6) & 63u, o = i & 63u;
    const __nv_bfloat16 v = __float2bfloat16_rn(params[i]);
    // forward B tile: rows = output, K = input;  backward B tile: rows = input, K = output
    *reinterpret_cast<__nv_bfloat16*>(w_fwd + l * 8192u + canon_off(o, in)) = v;
    *reinterpret_cast<__nv_bfloat16*>(w_bwd + l * 8192u + canon_off(in, o)) = v;
}

// Sums of the batch weights, one per block of a fixed grid (the same order every time).
__global__ void __launch_bounds__(256) k_wsum(const float* __restrict__ w, uint32_t m, float* __restrict__ part) {
    __shared__ float s[8];
    float t = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) t += w[i];
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if ((threadIdx.x & 31u) == 0) s[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) part[blockIdx.x] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// Weight gradients of all four layers on the tensor cores (blockIdx.y = layer):
//   gw[l][in][out] = sum_rows prev[row][in] * grad[row][out],  gb[l][out] = sum_rows grad[row][out]
// with BF16 operands and FP32 accumulation in tensor memory.  One MMA chain per CTA computes
// D (128 x 64) += A (128 x K) * B (64 x K)^T over the CTA's rows, in K-tiles of 64 rows:
//   A rows 0..63 = prev^T (m = input unit, k = batch row); row 64 = 1 for every valid row, so
//   D row 64 is the bias gradient; rows 65..127 = 0;
//   B rows = grad^T (n = output unit, k = batch row).
// The batch rows are the K dimension, so both operands lie in shared memory as they do in global
// memory, units contiguous: the MN-major canonical layout (core matrices of 8 batch rows x 16 bytes of
// 8 units), written in 16-byte pieces without bank conflicts: 26 us per 65,536 rows, 48 us when they
// were transposed into the K-major layout by 2-byte stores.  Double-buffered: tile i + 1 is staged while
// the MMAs of tile i run (one mbarrier per stage, each wait bounded).  The CTA then writes D rows
// 0..64 to its place in `part`; k_update adds the CTAs' parts in a fixed order.
constexpr uint32_t kDwK = 64;                                  // batch rows per K-tile
constexpr uint32_t kDwA = 16384, kDwB = 8192;                  // bytes per stage
constexpr uint32_t kDwSmemA0 = 0, kDwSmemB0 = 2 * kDwA, kDwSmemBar = 2 * kDwA + 2 * kDwB,
                   kDwSmemSlot = kDwSmemBar + 16, kDwSmemOk = kDwSmemSlot + 4, kDwSmemBytes = kDwSmemOk + 12;
constexpr uint32_t kDwPart = 65 * 64;                          // floats per CTA and layer: weights, bias
// BF16 x BF16 -> FP32, M = 128, N = 64, A and B MN-major (transposed)
constexpr uint32_t kIdescMN = kIdesc | (1u << 15) | (1u << 16);
// MN-major descriptor, no swizzle: groups of 8 units 128 B apart, groups of 8 batch rows `rows8` apart
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr, uint32_t rows8) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(rows8 >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
}

__global__ void __launch_bounds__(128) k_dw_tc(DwLayers L, uint32_t m, uint32_t tiles_per_cta, uint32_t spin,
                                               int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kDwSmemBar);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kDwSmemSlot);
    volatile int* s_ok = reinterpret_cast<volatile int*>(smem + kDwSmemOk);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, l = blockIdx.y;
    // constant-index selects keep the parameter arrays out of local memory
    auto pick = [l](auto a0, auto a1, auto a2, auto a3) { return l == 0 ? a0 : l == 1 ? a1 : l == 2 ? a2 : a3; };
    const uint4* __restrict__ prev = pick(L.prev[0], L.prev[1], L.prev[2], L.prev[3]);
    const uint4* __restrict__ grad = pick(L.grad_bf[0], L.grad_bf[1], L.grad_bf[2], L.grad_bf[3]);
    const uint32_t ntiles = (m + kDwK - 1) / kDwK;
    const uint32_t t0 = blockIdx.x * tiles_per_cta;
    const uint32_t t1 = min(ntiles, t0 + tiles_per_cta);
    if (t0 >= t1) return;
    // zero both A stages (unit groups 9..15 stay zero; 0..8 are rewritten per tile)
    for (uint32_t i = tid; i < 2 * kDwA / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(smem + kDwSmemA0)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) { mbar_init(&bar[0], 1); mbar_init(&bar[1], 1); fence_mbar_init(); }
    if (warp == 0) { tmem_alloc(tslot, 64); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *tslot;
    uint32_t phases = 0u;              // bit s = parity of the next completion of stage s
    bool ok = true;
    // a warp's 32 lanes: 8 batch rows x 4 pieces of 8 units; four such blocks per tile and operand
    const uint32_t r8 = tid & 7u, c4 = (tid >> 3) & 3u;
    uint4 a[4], b[4];                    // the next tile's pieces, loaded while this one is staged
    auto load = [&](uint32_t t) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const uint32_t row = t * kDwK + (warp + 4u * (i >> 1)) * 8u + r8, c = (i & 1u) * 4u + c4;
            const bool valid = row < m;
            a[i] = valid ? __ldg(&prev[(size_t)row * 8 + c]) : make_uint4(0u, 0u, 0u, 0u);
            b[i] = valid ? __ldg(&grad[(size_t)row * 8 + c]) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    load(t0);
    for (uint32_t t = t0; t < t1 && ok; ++t) {
        const uint32_t st = (t - t0) & 1u;
        uint8_t* sA = smem + kDwSmemA0 + st * kDwA;
        uint8_t* sB = smem + kDwSmemB0 + st * kDwB;
        // the MMAs that last read this stage (two tiles ago) must have completed
        if (t - t0 >= 2u) {
            if (tid == 0) {
                bool done = false;
                for (uint32_t it = 0; it < spin && !done; ++it) done = mbar_try_wait(&bar[st], (phases >> st) & 1u);
                *s_ok = done ? 1 : 0;
            }
            __syncthreads();
            ok = *s_ok != 0;
            if (!ok) break;
            phases ^= 1u << st;
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const uint32_t rg = warp + 4u * (i >> 1), c = (i & 1u) * 4u + c4;
            *reinterpret_cast<uint4*>(sA + rg * 2048u + c * 128u + r8 * 16u) = a[i];
            *reinterpret_cast<uint4*>(sB + rg * 1024u + c * 128u + r8 * 16u) = b[i];
        }
        if (tid < kDwK)                                  // units 64..71: one, then zeros
            *reinterpret_cast<uint4*>(sA + (tid >> 3) * 2048u + 8u * 128u + (tid & 7u) * 16u) =
                make_uint4(t * kDwK + tid < m ? 0x3f80u : 0u, 0u, 0u, 0u);
        if (t + 1u < t1) load(t + 1u);
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)             // 16 batch rows each
                umma_bf16(taddr, smem_desc_mn(smem_u32(sA) + k * 4096u, 2048u), smem_desc_mn(smem_u32(sB) + k * 2048u, 1024u),
                          kIdescMN, (t > t0 || k > 0) ? 1u : 0u);
            umma_commit(&bar[st]);
        }
    }
    // the last one or two tiles' MMAs
    if (ok) {
        const uint32_t n = t1 - t0;
        if (tid == 0) {
            bool done = true;
            for (uint32_t back = (n >= 2u ? 2u : 1u); back >= 1u && done; --back) {
                const uint32_t st = (n - back) & 1u;
                done = false;
                for (uint32_t it = 0; it < spin && !done; ++it) done = mbar_try_wait(&bar[st], (phases >> st) & 1u);
                if (done) phases ^= 1u << st;
            }
            *s_ok = done ? 1 : 0;
        }
        __syncthreads();
        ok = *s_ok != 0;
    }
    tc_fence_after();
    if (ok) {
        if (warp < 3) {
            float v[64];
            const uint32_t lane_addr = taddr + ((32u * warp) << 16);
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld16(lane_addr + 16u * j, v + 16 * j);
            tmem_wait_ld();
            const uint32_t drow = 32u * warp + (tid & 31u);
            if (drow <= 64u) {
                float4* to = reinterpret_cast<float4*>(L.part + ((size_t)l * gridDim.x + blockIdx.x) * kDwPart + drow * 64u);
#pragma unroll
                for (int j = 0; j < 16; ++j) to[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
        }
    } else if (tid == 0) {
        atomicExch(err, 1);
    }
    // every MMA this CTA issued must have landed before its tensor memory is freed
    if (!ok && tid == 0) {
        for (uint32_t st = 0; st < 2; ++st) {
            uint32_t it = 0;
            while (!mbar_try_wait(&bar[st], (phases >> st) & 1u) && ++it < kSpin) {}
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, 64);
}

// The step's tail in one launch: every parameter's gradient as the sum of the CTAs' parts (four lanes
// per parameter, a fixed order), the batch loss, and with lr > 0 Adam (Kingma & Ba 2015) on the FP32
// master parameters and the repacked BF16 tiles.  After a wait that timed out (*err, written by this step's
// kernels before this one only, so every thread reads the same) the parts are not complete: parameters, moments
// and the count of steps stay.
__global__ void __launch_bounds__(256) k_update(UpdateArgs u) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, i = t >> 2, q = t & 3u;
    const bool bias = i >= 4u * 4096u;
    const uint32_t l = bias ? (i - 4u * 4096u) >> 6 : i >> 12, at = bias ? 4096u + (i & 63u) : i & 4095u;
    float g = 0.0f;
    if (i < (uint32_t)kParams) {
        const float* p = u.part + (size_t)l * u.nparts * kDwPart + at;
#pragma unroll 8
        for (uint32_t k = q; k < u.nparts; k += 4u) g += __ldg(p + (size_t)k * kDwPart);
    }
    g += __shfl_xor_sync(0xffffffffu, g, 1);
    g += __shfl_xor_sync(0xffffffffu, g, 2);
    if (i < (uint32_t)kParams && q == 0u) {
        u.grads[i] = g;
        if (u.lr > 0.0f && *u.err == 0) {
            const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
            const float a = b1 * u.m1[i] + (1.0f - b1) * g;
            const float b = b2 * u.m2[i] + (1.0f - b2) * g * g;
            u.m1[i] = a;
            u.m2[i] = b;
            const float p = u.params[i] - u.lr * (a / u.c1) / (sqrtf(b / u.c2) + eps);
            u.params[i] = p;
            if (!bias) {
                const uint32_t in = (i >> 6) & 63u, o = i & 63u;
                const __nv_bfloat16 v = __float2bfloat16_rn(p);
                *reinterpret_cast<__nv_bfloat16*>(u.w_fwd + l * 8192u + canon_off(o, in)) = v;
                *reinterpret_cast<__nv_bfloat16*>(u.w_bwd + l * 8192u + canon_off(in, o)) = v;
            }
        }
    }
    if (blockIdx.x == 0) {
        __shared__ float s[8];
        float loss = 0.0f;
        for (uint32_t k = threadIdx.x; k < u.ntiles; k += 256u) loss += u.loss_part[k];
        for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
        if ((threadIdx.x & 31u) == 0) s[threadIdx.x >> 5] = loss;
        __syncthreads();
        if (threadIdx.x == 0) {
            *u.loss = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
            if (u.lr > 0.0f && *u.err == 0) *u.steps += 1;
        }
    }
}

cudaError_t pack_weights(const float* params, uint8_t* w_fwd, uint8_t* w_bwd, cudaStream_t s) {
    k_pack_weights<<<(4 * 4096 + 255) / 256, 256, 0, s>>>(params, w_fwd, w_bwd);
    return cudaGetLastError();
}
// k_dw_tc: two CTAs per SM over the four layers; each CTA walks a contiguous run of K-tiles
static uint32_t dw_max_parts() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max<uint32_t>(1u, (uint32_t)sms / 2u);
}
static uint32_t dw_parts(uint32_t m) {
    const uint32_t ntiles = (m + kDwK - 1) / kDwK, most = dw_max_parts();
    const uint32_t tiles_per_cta = (ntiles + most - 1) / most;
    return (ntiles + tiles_per_cta - 1) / tiles_per_cta;
}
size_t train_scratch_floats(uint32_t m) {
    return kSumBlocks + (m + kTile - 1) / kTile + (size_t)4 * dw_max_parts() * kDwPart + 64;
}

cudaError_t train_step(const TrainArgs& a, uint32_t m, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(k_dw_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwSmemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    if (m == 0) return cudaSuccess;
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t tiles = (m + kTile - 1) / kTile, ktiles = (m + kDwK - 1) / kDwK, parts = dw_parts(m);
    float* wsum = a.scratch;                                   // [kSumBlocks]
    float* loss_part = wsum + kSumBlocks;                      // [tiles]
    float* part = a.scratch + ((kSumBlocks + tiles + 63u) & ~63u);   // [layer][parts][kDwPart]
    k_wsum<<<kSumBlocks, 256, 0, s>>>(a.w, m, wsum);
    k_train_tile<<<std::min(tiles, (uint32_t)train_grid(dev)), 128, kSmemBytes, s>>>(
        a.net, a.x, a.dirs, a.w, wsum, m, a.act, a.dy, a.dh, loss_part, a.err);
    const size_t mrow = (size_t)m * 8;
    DwLayers L{};
    L.prev[0] = a.x;                  L.grad_bf[0] = a.dh;
    L.prev[1] = a.act;                L.grad_bf[1] = a.dh + mrow;
    L.prev[2] = a.act + mrow;         L.grad_bf[2] = a.dh + 2 * mrow;
    L.prev[3] = a.act + 2 * mrow;     L.grad_bf[3] = a.dy;                // output layer
    L.part = part;
    k_dw_tc<<<dim3(parts, 4), 128, kDwSmemBytes, s>>>(L, m, (ktiles + parts - 1) / parts, a.net.spin, a.err);
    UpdateArgs u{};
    u.part = part; u.nparts = parts; u.loss_part = loss_part; u.ntiles = tiles; u.loss = a.loss;
    u.err = a.err; u.steps = a.steps;
    u.params = a.params; u.grads = a.grads; u.m1 = a.m1; u.m2 = a.m2; u.w_fwd = a.w_fwd; u.w_bwd = a.w_bwd;
    u.lr = a.lr;
    u.c1 = 1.0f - powf(0.9f, (float)a.step);
    u.c2 = 1.0f - powf(0.999f, (float)a.step);
    k_update<<<(4u * kParams + 255) / 256, 256, 0, s>>>(u);
    return cudaGetLastError();
}

}  // namespace trg
