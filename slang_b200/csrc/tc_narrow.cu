// learnGradient and forward for networks of widths up to 64, 16-bit operands: those that tc_chain.cu does not take (fp32
// storage, other activations than ReLU and leaky ReLU) and the smallest batches.  Times of larger batches below are this file's
// kernels' own.
//
// A warp carries 16 samples (training) or 32 (forward) through every layer in registers (tc_narrow.cuh) and never waits
// for another warp on the way down or back up.  What contracts over samples, the weight and bias gradients, is done
//   at padded width 32: in registers as well.  The layer inputs and the output gradients of the warp's samples are
//     transposed 8x8 blocks at a time (movmatrix) and multiplied with mma.sync into accumulators the warp keeps for
//     the whole launch (NL x 32 x 32 fp32 over 32 lanes); the warps' sums meet in shared memory once, at the end.
//   at padded width 64, where those accumulators do not fit a warp: on the tcgen05 tensor pipe.  Every warp stores
//     its samples' dZ_l and A_l rows into a slot of shared memory ([samples][64 features] tiles, 128-byte
//     swizzle), one warp issues dW_l | db_l [64 x 80] += dZ_l^T . [A_l | 1] (contraction over the slot's rows) into
//     tensor memory, and the slot is free again when that product has completed.  Slots belong to groups of one to
//     five warps: with one slot for all fifteen the warps ran in step, products against products and epilogues
//     against epilogues, and a 2^24-sample step took 5.3 ms instead of 3.9 (3.83 now).
// Either way each parameter receives one atomic add per CTA at the end.
//
// What the reference does instead: one thread per sample with per-element global atomics
// (examples/mlp-training/mlp_sw.slang:28-58) or CoopVec calls whose CPU/CUDA fallback is scalar loops
// (examples/mlp-training-coopvec/fflayer.slang:16-58, source/slang/hlsl.meta.slang:32835-32912).
#include <cuda.h>
#include <cuda_runtime.h>

#include <string>
#include <type_traits>

#include "launch_pdl.cuh"
#include "launchers.h"
#include "tc_host.h"
#include "tc_narrow.cuh"

namespace mlpb200 {

using namespace ptx;

namespace narrow {

enum : uint32_t { kStatusSlot = 0x2000u };

constexpr int kForwardWarps = 8;
// 16-sample blocks a training warp carries at a time: one (the fragment helpers shared with the forward kernel take more,
// what follows a layer's products here does not).
constexpr int kTrainBlocks = 1;

// Shared-memory map of the training kernel (bytes from a 1024-aligned base).  NG groups of GW warps carry samples.
template <int W, int NL, int NG, int GW>
struct TrainMap {
    static constexpr bool kSlots = W == 64;
    static constexpr int kWarps = NG * GW;                               // warps with samples; one more issues where there are slots
    static constexpr int kThreads = 32 * (kWarps + (kSlots ? 1 : 0));
    static constexpr int kUnit = GW * 16;                                // samples a group takes at a time
    static constexpr int kQ = W / 32, kT = W / 8;
    static constexpr uint32_t kPanel = kQ * kT * 512;                    // one weight matrix in fragment order
    static constexpr uint32_t kTile = GW * 16 * W * 2;                   // [samples of a group][W] operand tile
    static constexpr uint32_t kSlotBytes = 2 * kTile;                    // dZ, then A
    static constexpr int kNumSlots = kSlots ? 2 : 0;                     // per group
    static constexpr uint32_t kSlot0 = 0;
    static constexpr uint32_t kSums = 0;                                 // the outgoing gradients, over the slots and panels once they are done
    static constexpr uint32_t kOnes = kSlot0 + NG * kNumSlots * kSlotBytes;   // 16 rows whose first element is one
    static constexpr uint32_t kForward = kOnes + (kSlots ? 2048 : 0);
    static constexpr uint32_t kReverse = kForward + NL * kPanel;
    // [NL][W rows][W + 1]; one copy per warp where the warps keep their own sums
    static constexpr uint32_t kSumRow = W + 1, kSumFloats = NL * W * kSumRow;
    static constexpr uint32_t kSumBytes = kSumFloats * 4 * (kSlots ? 1 : kWarps);
    static constexpr uint32_t kPanelsEnd = kReverse + NL * kPanel;
    static constexpr uint32_t kBias = kPanelsEnd > kSumBytes ? kPanelsEnd : ((kSumBytes + 15) & ~15u);   // fp32 [NL][W / 2 pairs][twice]
    static constexpr uint32_t kLoss = kBias + NL * W * 8;                // fp32 [kWarps][2]
    static constexpr uint32_t kBars = kLoss + kWarps * 8;                // full and empty [group][slot], done
    static constexpr uint32_t kTmemPtr = kBars + (2 * NG * kNumSlots + 1) * 8;
    static constexpr uint32_t kAbort = kTmemPtr + 4;
    static constexpr uint32_t kNet = (kAbort + 4 + 15) & ~15u;           // MlpLayerPointers [NL], then where the weights are cut from
    static constexpr uint32_t kSmemBytes = kNet + NL * 40 + 1024;
    // the stored weights during set-up: where the slots, or the sums past the panels, will be
    static constexpr uint32_t kStored = kSlots ? kSlot0 : kPanelsEnd, kStoredEnd = kSlots ? kOnes : kBias;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
    // tensor memory: W + 16 columns per layer (dW_l, then db_l)
    static constexpr uint32_t kDwCols = W + 16;
    static_assert(!kSlots || NL * kDwCols <= 512, "tensor memory budget");
};

// W: padded width (32 or 64).  HACT: hidden activation, or -1 for any (one switch, run per element).  OT: 8-column
// tiles of the output layer.  NG, GW: groups of warps that share slots, and warps of a group.
template <int W, int NL, int FMT, int HACT, int OT, int NG, int GW>
__global__ void __launch_bounds__(32 * (NG * GW + (W == 64 ? 1 : 0)), 1) learn_gradient_narrow_kernel(const __grid_constant__ Params p)
{
    using M = TrainMap<W, NL, NG, GW>;
    using C = Cvt<FMT>;
    constexpr bool kSlots = M::kSlots;
    constexpr int NT = W / 8, KS = W / 16;
    constexpr int OK = (OT + 1) / 2;                       // K steps of the output layer's reverse product
    constexpr bool kKeepD = HACT != MLP_ACT_RELU && HACT != MLP_ACT_LEAKY_RELU;   // derivative kept, not recovered from the activation
    constexpr int kThreads = M::kThreads, NW = M::kWarps;
    constexpr int MT = kTrainBlocks;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const MlpConfig& cfg = p.cfg;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    uint64_t* slot_full = (uint64_t*)(smem + M::kBars);
    uint64_t* slot_empty = slot_full + NG * M::kNumSlots;
    uint64_t* all_done = slot_empty + NG * M::kNumSlots;
    volatile uint32_t* abort_flag = (volatile uint32_t*)(smem + M::kAbort);
    constexpr int okind = tile_kind(OT);
    const int ikind = input_kind(cfg.dims[0]);
    const int od = cfg.dims[NL];

    // ---- set-up ----
    if (threadIdx.x == 0) {
        for (int s = 0; s < NG * M::kNumSlots; ++s) { mbar_init(&slot_full[s], GW); mbar_init(&slot_empty[s], 1); }
        mbar_init(all_done, 1);
        *abort_flag = 0u;
        fence_mbar_init();
    }
    if constexpr (kSlots) {
        // 16 rows of 128 bytes, the first 16-bit element of each one; the swizzle moves the 16-byte chunk with the row
        for (int i = threadIdx.x; i < 512; i += kThreads) {
            const int row = i >> 5, word = i & 31;
            ((uint32_t*)(smem + M::kOnes))[i] = (word >> 2) == (row & 7) && (word & 3) == 0 ? (C::kOnes & 0xffffu) : 0u;
        }
    }
    if constexpr (!kSlots) grid_release();
    grid_wait();
    if constexpr (kSlots) {
        if (warp == NW) {
            tmem_alloc((uint32_t*)(smem + M::kTmemPtr), 512);
            tmem_relinquish();
            grid_release();
        }
    }
    const MlpLayerPointers* s_net = (const MlpLayerPointers*)(smem + M::kNet);
    if (threadIdx.x < NL * 4) ((uint64_t*)(smem + M::kNet))[threadIdx.x] = ((const uint64_t*)p.net)[threadIdx.x];
    __syncthreads();
    const void** s_from = (const void**)(smem + M::kNet + NL * 32);
    copy_weights<NL>(smem + M::kStored, M::kStoredEnd - M::kStored, cfg, s_net, s_from, threadIdx.x, kThreads);
    for (int i = threadIdx.x; i < NL * W; i += kThreads) {
        const int l = i / W, j = i % W;
        if (l == NL - 1 && j >= OT * 8) continue;
        // features past the real width: below zero for ReLU, so that no derivative there is the one at zero
        const int f = feature_of(l == NL - 1 ? okind : kEights, j >> 3, j & 7);
        float* b = (float*)(smem + M::kBias) + l * W * 2 + (j >> 1) * 4 + (j & 1);
        b[0] = b[2] = f < cfg.dims[l + 1] ? load_as_f32(cfg.dtype, (const void*)s_net[l].biases, f) : (HACT == MLP_ACT_RELU && l < NL - 1 ? -1.0f : 0.0f);
    }
    cp_async_wait_all();
    __syncthreads();
    // forward panels, then reverse panels from the last layer down (layer 0's only for the input gradients)
    cut_panels<FMT, M::kQ * NT * 32>(smem, cfg, p.input_grads ? 2 * NL : 2 * NL - 1, [&](int which, int* chunks) {
        const bool rev = which >= NL;
        const int l = rev ? 2 * NL - 1 - which : which;
        const bool last = l == NL - 1;
        Panel d;
        d.weights = s_from[l];
        d.in = cfg.dims[l]; d.out = cfg.dims[l + 1];
        d.in_kind = l == 0 ? ikind : kEights;
        d.out_kind = last ? okind : kEights;
        d.transposed = rev;
        d.tiles = !rev && last ? OT : NT;
        d.dst = (rev ? M::kReverse : M::kForward) + (uint32_t)l * M::kPanel;
        *chunks = (rev && last ? (OK + 1) / 2 : M::kQ) * d.tiles * 32;
        return d;
    }, threadIdx.x, kThreads);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = kSlots ? *(volatile uint32_t*)(smem + M::kTmemPtr) : 0u;

    // gradient sums a warp keeps itself (width 32): [layer][row block of 16 outputs][tile of 8 inputs], and the biases of
    // all layers in one block whose column is the layer
    float wsum[kSlots ? 1 : NL][2][4][4];
    float bsum[2][4];
    if constexpr (!kSlots) {
#pragma unroll
        for (int l = 0; l < NL; ++l)
#pragma unroll
            for (int i = 0; i < 32; ++i) wsum[l][i >> 4][(i >> 2) & 3][i & 3] = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) bsum[i >> 2][i & 3] = 0.0f;
    }
    float run_max = 0.0f, run_sum = 0.0f;
    bool ok = true;
    if (warp < NW) {
        const uint32_t fwd_panel = sbase + M::kForward + (uint32_t)lane * 16u;
        const uint32_t rev_panel = sbase + M::kReverse + (uint32_t)lane * 16u;
        const uint32_t s_bias = sbase + M::kBias + (uint32_t)c * 16u;
        const bool f32s = cfg.dtype == MLP_F32;   // fp32 storage: pre-activations and outputs are not rounded
        const float scale = cfg.loss == MLP_LOSS_MSE_MEAN ? 1.0f / (float)od : 1.0f;
        const float alpha = cfg.act_alpha, alpha_op = C::round(alpha);
        const int in_steps = cfg.dims[0] <= 16 ? 1 : cfg.dims[0] <= 32 ? 2 : KS;
        const bool tgt_f32 = cfg.target_dtype == MLP_F32, tgt_f16 = cfg.target_dtype == MLP_F16;
        auto target_value = [&](uint32_t bits) -> float {
            const float h = tgt_f16 ? __half2float(__ushort_as_half((uint16_t)bits)) : __uint_as_float(bits << 16);
            return tgt_f32 ? __uint_as_float(bits) : h;
        };
        uint32_t step = 0;                         // slots this warp has filled
        // Slot tiles hold vectors in (tile, column) order.  This lane's row of a fragment's blocks (rows 0-7 and 8-15 of the
        // even tile, then of the odd one), and its 16-byte chunk's swizzle: chunk 2 k + (block / 2), moved with the row.
        const uint32_t slot_row = sbase + M::kSlot0 + (uint32_t)((warp % GW) * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128u;
        const uint32_t slot_chunk = (uint32_t)(lane >> 4) ^ (uint32_t)(lane & 7);
        // unit u of the batch goes to CTA u % grid, group (u / grid) % NG: small batches spread over SMs first
        const uint32_t stride = gridDim.x * NG, in_unit = (uint32_t)((warp % GW) * 16 + g);
        uint32_t unit = blockIdx.x + gridDim.x * (uint32_t)(warp / GW);

        // dW_l | db_l of this warp's samples from dZ_l and A_l (operand fragments)
        auto gradients = [&](auto layer, const uint32_t (&dz)[kTrainBlocks][W / 16][4], const uint32_t (&a)[kTrainBlocks][W / 16][4]) {
            [[maybe_unused]] constexpr int l = decltype(layer)::value;
            if constexpr (kSlots) {
                const uint32_t slot = (uint32_t)(warp / GW) * M::kNumSlots + step % M::kNumSlots, use = step / M::kNumSlots;
                if (use > 0) ok = ok && mbar_wait(&slot_empty[slot], (use - 1) & 1u, abort_flag, p.status, kStatusSlot);
                if (!ok) return;
                const uint32_t rows = slot_row + slot * M::kSlotBytes;
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    store_fragment(rows + (((uint32_t)(2 * k) ^ slot_chunk) << 4), dz[0][k]);
                    store_fragment(rows + M::kTile + (((uint32_t)(2 * k) ^ slot_chunk) << 4), a[0][k]);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&slot_full[slot]);
                ++step;
            } else {
                constexpr int rows = l == NL - 1 ? OK : 2;   // 16-row blocks of outputs
                uint32_t tz[2 * rows][2];
#pragma unroll
                for (int t = 0; t < 2 * rows; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) tz[t][h] = (l == NL - 1 && t >= OT) ? 0u : transpose8x8(dz[0][t >> 1][(t & 1) * 2 + h]);
                const uint32_t one = g == l ? C::kOnes : 0u;   // B operand whose column l is ones
#pragma unroll
                for (int m = 0; m < rows; ++m) {
                    const uint32_t az[4] = {tz[2 * m][0], tz[2 * m + 1][0], tz[2 * m][1], tz[2 * m + 1][1]};
                    C::mma(bsum[m], az, one, one);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (l == 0 && t * 8 >= (cfg.dims[0] <= 16 ? cfg.dims[0] : 32)) break;   // tiles the input layer does not have
                    const uint32_t b0 = transpose8x8(a[0][t >> 1][(t & 1) * 2]), b1 = transpose8x8(a[0][t >> 1][(t & 1) * 2 + 1]);
#pragma unroll
                    for (int m = 0; m < rows; ++m) {
                        const uint32_t az[4] = {tz[2 * m][0], tz[2 * m + 1][0], tz[2 * m][1], tz[2 * m + 1][1]};
                        C::mma(wsum[l][m][t], az, b0, b1);
                    }
                }
            }
        };

        RawInputs<MT> raw;
        fetch_raw(raw, p, (uint64_t)unit * (uint64_t)M::kUnit + in_unit, 16u, c);
        for (; unit < p.n_tiles && ok; unit += stride) {
            // block m of this warp: samples base + 16 m + {0, 8}
            const uint64_t base = (uint64_t)unit * (uint64_t)M::kUnit + in_unit;
            uint32_t A[NL][MT][KS][4];                              // every layer's input
            uint32_t D[kKeepD ? NL - 1 : 1][MT][KS][4];             // derivatives of the hidden activations
            bool zero_seen = false;                                 // ReLU: whether any pre-activation was zero
            {
                // the next tile's input and target rows: start them on their way into L2
                const uint64_t ns = base + (uint64_t)stride * (uint64_t)M::kUnit + (uint64_t)((c & 1) * 8);
                if (ns < p.count && c < 2) {
                    if (!raw_inputs(cfg))
                        asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p.inputs + ns * (uint64_t)cfg.dims[0] * (cfg.input_dtype == MLP_F32 ? 4u : 2u)));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p.targets + ns * (uint64_t)od * (cfg.target_dtype == MLP_F32 ? 4u : 2u)));
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) load_inputs<FMT, KS>(A[0][m], p, raw.v[m], base + 16u * (uint64_t)m, c);
            fetch_raw(raw, p, base + (uint64_t)stride * (uint64_t)M::kUnit, 16u, c);
            // few targets per lane are fetched here, a forward pass ahead of their use (as stored: a conversion would wait)
            uint32_t tgt[MT][2][OT <= 2 ? OT * 2 : 1];
            if constexpr (OT <= 2) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
#pragma unroll
                    for (int i = 0; i < 4 * OT; ++i) {
                        const int h = i / (2 * OT), e = i % (2 * OT);
                        const uint64_t row = base + 16u * (uint64_t)m + 8u * (uint64_t)h;
                        const int f = feature_of(okind, e >> 1, 2 * c + (e & 1));
                        const bool real = row < p.count && f < od;
                        const uint64_t at = row * (uint64_t)od + (uint64_t)f;
                        uint32_t t = 0u;
                        if (real) t = tgt_f32 ? __ldg((const uint32_t*)p.targets + at) : (uint32_t)__ldg((const uint16_t*)p.targets + at);
                        tgt[m][h][e] = t;
                    }
                }
            }

            // ---- forward, hidden layers ----
#pragma unroll
            for (int l = 0; l < NL - 1; ++l) {
                float acc[MT][NT][4];
                const uint32_t start = s_bias + (uint32_t)(l * W) * 8u;
                if (l > 0 || in_steps == KS) layer_product<FMT, true, MT, NT, KS>(acc, A[l], fwd_panel + (uint32_t)l * M::kPanel, NT * 512u, start);
                else if (in_steps == 2) layer_product<FMT, true, MT, NT, 2>(acc, A[l], fwd_panel, NT * 512u, start);
                else layer_product<FMT, true, MT, NT, 1>(acc, A[l], fwd_panel, NT * 512u, start);
                if constexpr (HACT == MLP_ACT_RELU) {
                    // The backward pass recovers the derivative from the activation: one above zero, zero at +0, one half at
                    // the -0 that marks a zero pre-activation (one that rounds to a zero of either sign).  Few fragments
                    // hold one: the smallest magnitude is watched, one three-operand minimum for two values, and the marks
                    // are set only where it calls for them (2^24 texels: 3.80 ms a step; with the sign of every value
                    // settled in 16-bit arithmetic instead, 3.97 to 4.06).  Not rounded (fp32 storage), only a zero is
                    // zero, and what lies above it stays there.
                    if (f32s) {
#pragma unroll
                        for (int i = 0; i < MT * NT * 4; ++i) {
                            float& z = acc[i / (NT * 4)][i / 4 % NT][i & 3];
                            z = z > 0.0f ? fmaxf(z, C::kSmallest) : z;
                        }
                    }
                    const float tiny = f32s ? 0.0f : 0.5f * C::kSmallest;   // the largest magnitude that rounds to zero
                    float least = 1.0f;
#pragma unroll
                    for (int i = 0; i < MT * NT * 2; ++i) {
                        const int m = i / (NT * 2), t = (i >> 1) % NT, h = i & 1;
                        const float z0 = acc[m][t][2 * h], z1 = acc[m][t][2 * h + 1];
                        A[l + 1][m][t >> 1][(t & 1) * 2 + h] = C::relu2(C::pack2(z0, z1));
                        least = fminf(fminf(fabsf(z0), fabsf(z1)), least);
                    }
                    if (least <= tiny) {
                        zero_seen = true;
#pragma unroll
                        for (int i = 0; i < MT * NT * 2; ++i) {
                            const int m = i / (NT * 2), t = (i >> 1) % NT, h = i & 1;
                            uint32_t& a = A[l + 1][m][t >> 1][(t & 1) * 2 + h];
                            if (fabsf(acc[m][t][2 * h]) <= tiny) a |= 0x8000u;
                            if (fabsf(acc[m][t][2 * h + 1]) <= tiny) a |= 0x80000000u;
                        }
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                float z0 = acc[m][t][2 * h], z1 = acc[m][t][2 * h + 1];
                                uint32_t& a = A[l + 1][m][t >> 1][(t & 1) * 2 + h];
                                if constexpr (HACT == MLP_ACT_LEAKY_RELU) {
                                    // max(z, alpha z) with 0 < alpha < 1 (the launcher sees to it), from the rounded z where
                                    // z is rounded.  The sign bit is "z < 0": adding +0 to alpha z makes a zero z of either
                                    // sign a positive zero, while an alpha z that only rounds to zero keeps its sign.
                                    const uint32_t zp = C::pack2(z0, z1);
                                    if (!f32s) { z0 = C::lo(zp); z1 = C::hi(zp); }
                                    const float2 az = __ffma2_rn(make_float2(z0, z1), make_float2(alpha, alpha), make_float2(0.0f, 0.0f));
                                    a = C::max2(zp, C::pack2(az.x, az.y));
                                } else {
                                    if (!f32s) {
                                        const uint32_t zp = C::pack2(z0, z1);
                                        z0 = C::lo(zp);
                                        z1 = C::hi(zp);
                                    }
                                    if constexpr (HACT == MLP_ACT_GELU_TANH) {
                                        float v[2], d[2];
                                        gelu_pair(z0, v[0], d[0]);
                                        gelu_pair(z1, v[1], d[1]);
                                        a = C::pack2(v[0], v[1]);
                                        D[l][m][t >> 1][(t & 1) * 2 + h] = C::pack2(d[0], d[1]);
                                    } else {
                                        acc[m][t][2 * h] = z0;
                                        acc[m][t][2 * h + 1] = z1;
                                    }
                                }
                            }
                        }
                        if constexpr (HACT < 0) {
                            float v[NT * 4], d[NT * 4];
#pragma unroll
                            for (int i = 0; i < NT * 4; ++i) v[i] = acc[m][i >> 2][i & 3];
                            activate_any(cfg.hidden_act, alpha, v, d, true);
#pragma unroll
                            for (int i = 0; i < NT * 2; ++i) {
                                const int t = i >> 1, h = i & 1;
                                A[l + 1][m][t >> 1][(t & 1) * 2 + h] = C::pack2(v[t * 4 + 2 * h], v[t * 4 + 2 * h + 1]);
                                D[l][m][t >> 1][(t & 1) * 2 + h] = C::pack2(d[t * 4 + 2 * h], d[t * 4 + 2 * h + 1]);
                            }
                        }
                    }
                }
            }

            // ---- output layer, loss, dZ of the last layer ----
            uint32_t dz[MT][KS][4];
            {
                float acc[MT][OT][4];
                layer_product<FMT, true, MT, OT, KS>(acc, A[NL - 1], fwd_panel + (uint32_t)(NL - 1) * M::kPanel, OT * 512u, s_bias + (uint32_t)((NL - 1) * W) * 8u);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    float o[OT * 4], d[OT * 4];
#pragma unroll
                    for (int i = 0; i < OT * 4; ++i) {
                        const float z = acc[m][i >> 2][i & 3];
                        o[i] = f32s ? z : C::round(z);
                    }
                    activate_outputs(cfg.output_act, alpha, o, d, true);
                    float loss[2] = {0.0f, 0.0f};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint64_t row = base + 16u * (uint64_t)m + 8u * (uint64_t)h;
                        const bool valid = row < p.count;
                        float dzv[OT * 2];
                        if constexpr (OT <= 2) {
#pragma unroll
                            for (int i = 0; i < OT * 2; ++i) {
                                const int e = (i >> 1) * 4 + 2 * h + (i & 1);
                                const bool real = valid && feature_of(okind, i >> 1, 2 * c + (i & 1)) < od;
                                const float diff = real ? o[e] - target_value(tgt[m][h][i]) : 0.0f;
                                loss[h] = fmaf(diff * scale, diff, loss[h]);
                                dzv[i] = real ? ((2.0f * scale) * diff) * d[e] : 0.0f;
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < OT / 4; ++q) {
                                float tv[8];
                                const int f0 = 32 * q + 8 * c;
                                if (valid) load_values<8>(tv, cfg.target_dtype, p.targets, row, od, f0, p.vec_tgt != 0);
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    const int e = (4 * q + (i >> 1)) * 4 + 2 * h + (i & 1);
                                    const bool real = valid && f0 + i < od;
                                    const float diff = real ? o[e] - tv[i] : 0.0f;
                                    loss[h] = fmaf(diff * scale, diff, loss[h]);
                                    dzv[8 * q + i] = real ? ((2.0f * scale) * diff) * d[e] : 0.0f;
                                }
                            }
                        }
#pragma unroll
                        for (int t = 0; t < NT; ++t) dz[m][t >> 1][(t & 1) * 2 + h] = t < OT ? C::pack2(dzv[2 * t], dzv[2 * t + 1]) : 0u;
                        float total = loss[h];
                        total += __shfl_xor_sync(0xffffffffu, total, 1);
                        total += __shfl_xor_sync(0xffffffffu, total, 2);
                        run_max = fmaxf(run_max, total);
                        run_sum += c == 0 ? total : 0.0f;
                    }
                }
            }

            // ---- backward ----
            gradients(std::integral_constant<int, NL - 1>{}, dz, A[NL - 1]);
#pragma unroll
            for (int l = NL - 1; l >= 1; --l) {
                float acc[MT][NT][4];
                if (l == NL - 1) layer_product<FMT, false, MT, NT, OK>(acc, dz, rev_panel + (uint32_t)l * M::kPanel, NT * 512u, 0u);
                else layer_product<FMT, false, MT, NT, KS>(acc, dz, rev_panel + (uint32_t)l * M::kPanel, NT * 512u, 0u);
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < NT; ++t)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float g0 = acc[m][t][2 * h], g1 = acc[m][t][2 * h + 1];
                            const uint32_t a = A[l][m][t >> 1][(t & 1) * 2 + h];
                            uint32_t& z = dz[m][t >> 1][(t & 1) * 2 + h];
                            if constexpr (HACT == MLP_ACT_RELU) {
                                z = C::pack2(g0, g1) & C::positive_mask(a);
                            } else if constexpr (HACT == MLP_ACT_LEAKY_RELU) {
                                const uint32_t neg = sign_mask(a);
                                const float2 ag = __fmul2_rn(make_float2(g0, g1), make_float2(alpha_op, alpha_op));
                                z = (C::pack2(ag.x, ag.y) & neg) | (C::pack2(g0, g1) & ~neg);
                            } else {
                                const uint32_t d = D[l - 1][m][t >> 1][(t & 1) * 2 + h];
                                z = C::pack2(g0 * C::lo(d), g1 * C::hi(d));
                            }
                        }
                if constexpr (HACT == MLP_ACT_RELU) {
                    if (zero_seen) {   // some pre-activation was zero: half of the gradient passes there
#pragma unroll
                        for (int m = 0; m < MT; ++m)
#pragma unroll
                            for (int i = 0; i < NT * 2; ++i) {
                                const int t = i >> 1, h = i & 1;
                                const uint32_t a = A[l][m][t >> 1][(t & 1) * 2 + h];
                                const uint32_t zero = sign_mask(a);
                                dz[m][t >> 1][(t & 1) * 2 + h] |= C::pack2(0.5f * acc[m][t][2 * h], 0.5f * acc[m][t][2 * h + 1]) & zero;
                            }
                    }
                }
                if (l == 4) gradients(std::integral_constant<int, 3 < NL ? 3 : 0>{}, dz, A[l - 1]);
                if (l == 3) gradients(std::integral_constant<int, 2 < NL ? 2 : 0>{}, dz, A[l - 1]);
                if (l == 2) gradients(std::integral_constant<int, 1>{}, dz, A[l - 1]);
                if (l == 1) gradients(std::integral_constant<int, 0>{}, dz, A[l - 1]);
            }

            // ---- optional: the input gradients dZ_0 . W_0, rounded to the storage type ----
            if (p.input_grads) {
                const int in = cfg.dims[0];
                float acc[MT][NT][4];
                layer_product<FMT, false, MT, NT, KS>(acc, dz, rev_panel, NT * 512u, 0u);
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint64_t row = base + 16u * (uint64_t)m + 8u * (uint64_t)h;
                        if (row >= p.count) continue;
                        float* dst = p.input_grads + row * (uint64_t)in;
#pragma unroll
                        for (int t = 0; t < NT; t += 2) {
                            float v[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float x = acc[m][t + (i >> 1)][2 * h + (i & 1)];
                                v[i] = f32s ? x : C::round(x);
                            }
                            // kEights and kFours put the pairs of tiles t, t + 1 side by side; natural order does not
                            const int f0 = feature_of(ikind, t, 2 * c), f1 = feature_of(ikind, t + 1, 2 * c);
                            if (f0 >= in) continue;
                            if (p.vec_dx && ikind != kNatural) {
                                *(float4*)(dst + f0) = make_float4(v[0], v[1], v[2], v[3]);
                            } else {
                                dst[f0] = v[0];
                                if (f0 + 1 < in) dst[f0 + 1] = v[1];
                                if (f1 < in) dst[f1] = v[2];
                                if (f1 + 1 < in) dst[f1 + 1] = v[3];
                            }
                        }
                    }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            run_max = fmaxf(run_max, __shfl_xor_sync(0xffffffffu, run_max, o));
            run_sum += __shfl_xor_sync(0xffffffffu, run_sum, o);
        }
        if (lane == 0) {
            ((float*)(smem + M::kLoss))[warp * 2] = run_max;
            ((float*)(smem + M::kLoss))[warp * 2 + 1] = run_sum;
        }
    } else if constexpr (kSlots) {
        // =================================== issuing warp ==========================================
        // Every group fills its slots in the same order (tile by tile, last layer first) at its own pace; this warp
        // serves whichever group has a slot ready.  One thread issues every product, so those into one accumulator
        // are in order.
        const bool leader = elect_one();
        constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29);              // 8-row groups 1024 bytes apart, 128-byte swizzle
        constexpr uint32_t kIdesc = umma_idesc(C::kUmmaFmt, 1, 1, 64, W + 16);        // dZ^T (MN, 64 rows) x [A | ones] (MN)
        const uint32_t lo = (sbase & 0x3FFFFu) >> 4;
        const uint32_t stride = gridDim.x * NG;
        uint32_t done[NG], fills[NG];
        uint32_t left = 0, idle = 0;
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            const uint32_t first = blockIdx.x + gridDim.x * (uint32_t)j;
            done[j] = 0;
            fills[j] = first < p.n_tiles ? ((p.n_tiles - first + stride - 1) / stride) * NL : 0u;
            left += fills[j];
        }
        uint32_t started = 0;    // layers whose accumulator has been written
        while (left > 0 && ok) {
            bool any = false;
#pragma unroll
            for (int j = 0; j < NG; ++j) {
                const uint32_t slot = (uint32_t)j * M::kNumSlots + done[j] % M::kNumSlots;
                if (done[j] < fills[j] && mbar_test_wait(&slot_full[slot], (done[j] / M::kNumSlots) & 1u)) {
                    tc_fence_after();
                    const uint32_t l = NL - 1 - done[j] % NL;
                    if (leader) {
                        const uint32_t zbuf = M::kSlot0 + slot * M::kSlotBytes;
#pragma unroll
                        for (int k = 0; k < GW; ++k) {
                            // a K step is 16 rows of 128 bytes; the B operand's second block is the 16 rows of ones
                            const uint32_t za = zbuf + (uint32_t)k * 2048u, aa = za + M::kTile;
                            const uint64_t da = ((uint64_t)kHi << 32) | (lo + (za >> 4) + (1u << 16));
                            const uint64_t db = ((uint64_t)kHi << 32) | (lo + (aa >> 4) + (((M::kOnes - aa) >> 4) << 16));
                            umma_f16(tmem_base + l * M::kDwCols, da, db, kIdesc, k > 0 ? 1u : (started >> l) & 1u);
                        }
                        umma_commit(&slot_empty[slot]);
                    }
                    __syncwarp();
                    started |= 1u << l;
                    ++done[j];
                    --left;
                    any = true;
                }
            }
            if (any) idle = 0;
            else if (++idle > kMaxPolls || ((idle & 63u) == 63u && *abort_flag)) {
                *abort_flag = 1u;
                atomicOr(p.status, kStatusSlot);
                ok = false;
            }
        }
        if (leader && ok) umma_commit(all_done);
        __syncwarp();
    }

    // ---- one add per parameter per CTA ----
    if constexpr (kSlots) {
        ok = ok && mbar_wait(all_done, 0u, abort_flag, p.status, kStatusSlot);
        tc_fence_after();
        __syncthreads();
        if (!*abort_flag && warp < (NW + 1) / 4 * 4) {
            // Row r of a 64-row accumulator sits on lane 32 (r / 16) + r % 16: the first 16 lanes of this warp's quarter
            // hold rows 16 quarter + lane; the warps of a quarter take the 16-column pieces in turn.
            const int quarter = warp & 3, r = quarter * 16 + lane;
            float* sums = (float*)(smem + M::kSums);
#pragma unroll 1
            for (int l = 0; l < NL; ++l)
#pragma unroll 1
                for (int piece = warp >> 2; piece < (W + 16) / 16; piece += (NW + 1) / 4) {
                    uint32_t v[16];
                    tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)l * M::kDwCols + (uint32_t)piece * 16u, v);
                    tmem_ld_wait();
                    if (lane < 16) {
                        float* row = sums + (l * W + r) * (W + 1) + piece * 16;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (piece * 16 + i < W + 1) row[i] = __uint_as_float(v[i]);
                    }
                }
        }
        tc_fence_before();
    } else {
        __syncthreads();   // the sums overwrite the panels
        float* sums = (float*)(smem + M::kSums) + warp * M::kSumFloats;
#pragma unroll
        for (int l = 0; l < NL; ++l)
#pragma unroll
            for (int m = 0; m < (l == NL - 1 ? OK : 2); ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // rows and columns in (tile, column) order
                    float* row = sums + (l * W + 8 * (2 * m + i) + g) * (W + 1);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        row[8 * t + 2 * c] = wsum[l][m][t][2 * i];
                        row[8 * t + 2 * c + 1] = wsum[l][m][t][2 * i + 1];
                    }
                    if (c == l / 2) row[W] = bsum[m][2 * i + l % 2];
                }
    }
    __syncthreads();
    if (!*abort_flag) {
        // Real parameters in the order they are stored, the layers one after the other over the threads; four to a reduction
        // where rows are whole 16-byte pieces.  (Walking the padded matrices instead, one parameter to a reduction, took
        // 7 us.)
        constexpr int kCopies = kSlots ? 1 : NW;
        const float* sums = (const float*)(smem + M::kSums);
        int i = threadIdx.x;
#pragma unroll 1
        for (int l = 0; l < NL; ++l) {
            const int in = cfg.dims[l], out = cfg.dims[l + 1];
            const int ki = l == 0 ? ikind : kEights, ko = l == NL - 1 ? okind : kEights;
            float* dW = (float*)s_net[l].weightsGrad;
            float* dB = (float*)s_net[l].biasesGrad;
            auto total = [&](int o, int column) {
                const float* at = sums + (l * W + position_of(ko, o)) * M::kSumRow + column;
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < kCopies; ++w) v += at[w * M::kSumFloats];
                return v;
            };
            const bool fours = (in & 3) == 0 && cfg.param_layout == MLP_PARAMS_ROW_MAJOR && ((uint64_t)dW & 15u) == 0;
            const int per_row = fours ? in >> 2 : in;
            for (; i < out * per_row; i += kThreads) {
                const int o = i / per_row, k = i - o * per_row;
                if (fours)
                    atomicAdd((float4*)dW + i, make_float4(total(o, position_of(ki, 4 * k)), total(o, position_of(ki, 4 * k + 1)),
                                                           total(o, position_of(ki, 4 * k + 2)), total(o, position_of(ki, 4 * k + 3))));
                else atomicAdd(dW + weight_index(cfg.param_layout, in, out, o, k), total(o, position_of(ki, k)));
            }
            i -= out * per_row;
            for (; i < out; i += kThreads) atomicAdd(dB + i, total(i, W));
            i -= out;
        }
        if (threadIdx.x == 0) {
            const float* part = (const float*)(smem + M::kLoss);
            float mx = part[0], sm = part[1];
#pragma unroll
            for (int w = 1; w < NW; ++w) { mx = fmaxf(mx, part[2 * w]); sm += part[2 * w + 1]; }
            atomicMax(p.loss_words, __float_as_uint(mx));
            atomicAdd((float*)(p.loss_words + 1), sm);
        }
    }
    if constexpr (kSlots) {
        tc_fence_after();
        if (warp == NW) tmem_dealloc(tmem_base, 512);
    }
}

// The forward pass alone: no gradients, nothing kept between layers.  W may also be 16.
template <int W, int FMT, int HACT, int OT, int MT>
__global__ void __launch_bounds__(32 * kForwardWarps, 2) forward_narrow_kernel(const __grid_constant__ Params p)
{
    using C = Cvt<FMT>;
    constexpr int NT = W / 8, KS = W / 16, kQ = (W + 31) / 32;
    constexpr int HK = tile_kind(NT);                    // how hidden vectors are dealt to the lanes
    constexpr uint32_t kPanel = kQ * NT * 512;
    extern __shared__ __align__(128) uint8_t smem[];     // [n_layers] panels, then fp32 biases [n_layers][W / 2 pairs][twice], addresses, stored weights
    const uint32_t sbase = smem_u32(smem);
    const MlpConfig& cfg = p.cfg;
    const int nl = cfg.n_layers, od = cfg.dims[nl];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const int ikind = input_kind(cfg.dims[0]);
    constexpr int okind = tile_kind(OT);
    float* s_bias_w = (float*)(smem + (uint32_t)nl * kPanel);
    MlpLayerPointers* s_net = (MlpLayerPointers*)(s_bias_w + nl * W * 2);
    grid_release();
    grid_wait();
    if (threadIdx.x < nl * 4) ((uint64_t*)s_net)[threadIdx.x] = ((const uint64_t*)p.net)[threadIdx.x];
    __syncthreads();
    const void** s_from = (const void**)(s_net + nl);
    copy_weights<5>((uint8_t*)(s_from + 6), (uint32_t)p.raw_bytes, cfg, s_net, s_from, threadIdx.x, 32 * kForwardWarps);
    for (int i = threadIdx.x; i < nl * W; i += 32 * kForwardWarps) {
        const int l = i / W, j = i % W;
        if (l == nl - 1 && j >= OT * 8) continue;
        const int f = feature_of(l == nl - 1 ? okind : HK, j >> 3, j & 7);
        float* b = s_bias_w + l * W * 2 + (j >> 1) * 4 + (j & 1);
        b[0] = b[2] = f < cfg.dims[l + 1] ? load_as_f32(cfg.dtype, (const void*)s_net[l].biases, f) : 0.0f;
    }
    cp_async_wait_all();
    __syncthreads();
    cut_panels<FMT, kQ * NT * 32>(smem, cfg, nl, [&](int l, int* chunks) {
        Panel d;
        d.weights = s_from[l];
        d.in = cfg.dims[l]; d.out = cfg.dims[l + 1];
        d.in_kind = l == 0 ? ikind : HK;
        d.out_kind = l == nl - 1 ? okind : HK;
        d.transposed = false;
        d.tiles = l == nl - 1 ? OT : NT;
        d.dst = (uint32_t)l * kPanel;
        *chunks = kQ * d.tiles * 32;
        return d;
    }, threadIdx.x, 32 * kForwardWarps);
    __syncthreads();
    const uint32_t panel0 = sbase + (uint32_t)lane * 16u;
    const uint32_t s_bias = sbase + (uint32_t)nl * kPanel + (uint32_t)c * 16u;
    const bool f32s = cfg.dtype == MLP_F32;
    const float alpha = cfg.act_alpha;
    const int in_steps = cfg.dims[0] <= 16 ? 1 : cfg.dims[0] <= 32 ? 2 : KS;

    RawInputs<MT> raw;
    fetch_raw(raw, p, (uint64_t)blockIdx.x * (uint64_t)(kForwardWarps * 16 * MT) + (uint64_t)(warp * 16 * MT + g), 16u, c);
    for (uint32_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
        const uint64_t base = (uint64_t)tile * (uint64_t)(kForwardWarps * 16 * MT) + (uint64_t)(warp * 16 * MT + g);
        uint32_t A[MT][KS][4];
#pragma unroll
        for (int m = 0; m < MT; ++m) load_inputs<FMT, KS>(A[m], p, raw.v[m], base + 16u * (uint64_t)m, c);
        fetch_raw(raw, p, base + (uint64_t)gridDim.x * (uint64_t)(kForwardWarps * 16 * MT), 16u, c);
#pragma unroll 1
        for (int l = 0; l < nl - 1; ++l) {
            float acc[MT][NT][4];
            const uint32_t panel = panel0 + (uint32_t)l * kPanel;
            const uint32_t start = s_bias + (uint32_t)(l * W) * 8u;
            if (l > 0 || in_steps == KS) layer_product<FMT, true, MT, NT, KS>(acc, A, panel, NT * 512u, start);
            else if (in_steps == 2) layer_product<FMT, true, MT, NT, KS < 2 ? KS : 2>(acc, A, panel, NT * 512u, start);
            else layer_product<FMT, true, MT, NT, 1>(acc, A, panel, NT * 512u, start);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
#pragma unroll
                for (int i = 0; i < NT * 2; ++i) {
                    const int t = i >> 1, h = i & 1;
                    float z0 = acc[m][t][2 * h], z1 = acc[m][t][2 * h + 1];
                    uint32_t& a = A[m][t >> 1][(t & 1) * 2 + h];
                    const uint32_t zp = C::pack2(z0, z1);
                    if constexpr (HACT == MLP_ACT_RELU) {
                        a = C::relu2(zp);
                    } else {
                        if (!f32s) { z0 = C::lo(zp); z1 = C::hi(zp); }
                        if constexpr (HACT == MLP_ACT_LEAKY_RELU) {
                            const float2 az = __fmul2_rn(make_float2(z0, z1), make_float2(alpha, alpha));
                            a = C::max2(zp, C::pack2(az.x, az.y));
                            continue;
                        }
                        if constexpr (HACT == MLP_ACT_GELU_TANH) {
                            a = C::pack2(act_value(MLP_ACT_GELU_TANH, alpha, z0), act_value(MLP_ACT_GELU_TANH, alpha, z1));
                        } else {
                            acc[m][t][2 * h] = z0;
                            acc[m][t][2 * h + 1] = z1;
                        }
                    }
                }
                if constexpr (HACT < 0) {
                    float v[NT * 4], d[NT * 4];
#pragma unroll
                    for (int i = 0; i < NT * 4; ++i) v[i] = acc[m][i >> 2][i & 3];
                    activate_any(cfg.hidden_act, alpha, v, d, false);
#pragma unroll
                    for (int i = 0; i < NT * 2; ++i)
                        A[m][i >> 2][((i >> 1) & 1) * 2 + (i & 1)] = C::pack2(v[(i >> 1) * 4 + 2 * (i & 1)], v[(i >> 1) * 4 + 2 * (i & 1) + 1]);
                }
            }
        }
        float acc[MT][OT][4];
        layer_product<FMT, true, MT, OT, KS>(acc, A, panel0 + (uint32_t)(nl - 1) * kPanel, OT * 512u, s_bias + (uint32_t)((nl - 1) * W) * 8u);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float o[OT * 4], d[OT * 4];
#pragma unroll
            for (int i = 0; i < OT * 4; ++i) o[i] = f32s ? acc[m][i >> 2][i & 3] : C::round(acc[m][i >> 2][i & 3]);
            if (OT == 1 && od <= 4) {
                // half of the tile's columns are padding: the lanes that hold them take the second row of those that do not
                // (1920 x 1080 view with three outputs: 146.5 -> 142.1 us)
                const float z0 = __shfl_xor_sync(0xffffffffu, o[2], 2), z1 = __shfl_xor_sync(0xffffffffu, o[3], 2);
                float v[2] = {c < 2 ? o[0] : z0, c < 2 ? o[1] : z1}, dv[2];
                activate_outputs(cfg.output_act, alpha, v, dv, false);
                const uint64_t row = base + 16u * (uint64_t)m + 8u * (uint64_t)(c >> 1);
                const int f = 2 * (c & 1);
                if (row < p.count) {
                    float* dst = p.outputs + row * (uint64_t)od;
                    if (f < od) dst[f] = v[0];
                    if (f + 1 < od) dst[f + 1] = v[1];
                }
                continue;
            }
            activate_outputs(cfg.output_act, alpha, o, d, false);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint64_t row = base + 16u * (uint64_t)m + 8u * (uint64_t)h;
                if (row >= p.count) continue;
                float* dst = p.outputs + row * (uint64_t)od;
                if constexpr (OT == 1) {
                    if (2 * c < od) dst[2 * c] = o[2 * h];
                    if (2 * c + 1 < od) dst[2 * c + 1] = o[2 * h + 1];
                } else {
                    // the pairs of tiles t and t + 1 are four consecutive features
#pragma unroll
                    for (int t = 0; t < OT; t += 2) {
                        const int f = feature_of(okind, t, 2 * c);
                        if (f >= od) continue;
                        const float v[4] = {o[t * 4 + 2 * h], o[t * 4 + 2 * h + 1], o[t * 4 + 4 + 2 * h], o[t * 4 + 4 + 2 * h + 1]};
                        if (p.vec_out) {
                            *(float4*)(dst + f) = make_float4(v[0], v[1], v[2], v[3]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (f + i < od) dst[f + i] = v[i];
                        }
                    }
                }
            }
        }
    }
}

}  // namespace narrow

// ------------------------------------------------------------------------------------------------
// Host side.  The kernels are built for every layer count, format, activation class and output width; this file is
// compiled once per MLPB200_NARROW_PART (0..9) so that the builds run side by side: part 0 holds the entry points, part
// 1 + 4 w + (layers - 2) the training builds of padded width 32 (w = 0) or 64 (w = 1), part 9 the forward builds.
// ------------------------------------------------------------------------------------------------
#ifndef MLPB200_NARROW_PART
#error "compile with -DMLPB200_NARROW_PART=0..9 (slang_b200/build.py does)"
#endif

template <int W, int NL>
cudaError_t launch_narrow_train(cudaStream_t st, TcWorkspace* ws, int op, narrow::Params& p);
cudaError_t launch_narrow_forward(cudaStream_t st, TcWorkspace* ws, int op, narrow::Params& p);

#if MLPB200_NARROW_PART >= 1 && MLPB200_NARROW_PART <= 8
template <int W, int NL, int FMT, int HACT, int OT>
static cudaError_t launch_train(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    // Width 32: eight warps of 255 registers.  Width 64: as many warps as the state of a sample block leaves registers
    // for (16 with 128 each, 11 with 168, 8 with 255), one of them issuing.  Groups, fp16 learnGradient of 2^20 and of 20000
    // samples: 5 x 2 warps 415 / 25.1 us against 10 x 1 421 / 27.3 (32-64-64-3, GELU) and 624 / 33.3 against 710 / 35.8
    // (64 x 6, ReLU); 7 x 1 984 / 47.7 against 1 x 7 873 / 47.7 (64 x 5, GELU) and 1210 / 60.0 against 1146 / 62.4 (64 x 6,
    // GELU), where the one group would be the better one for large batches.
    constexpr bool kept = HACT != MLP_ACT_RELU && HACT != MLP_ACT_LEAKY_RELU;
    constexpr int state = NL + (kept ? NL - 1 : 0);
    constexpr int NG = W == 32 ? 8 : state <= 4 ? 3 : state <= 5 ? 5 : 7, GW = W == 32 ? 1 : state <= 4 ? 5 : state <= 5 ? 2 : 1;
    using M = narrow::TrainMap<W, NL, NG, GW>;
    auto kern = narrow::learn_gradient_narrow_kernel<W, NL, FMT, HACT, OT, NG, GW>;
    static SmemLimit limit;
    const cudaError_t e = limit.raise((const void*)kern, ws->ordinal, M::kSmemBytes);
    if (e != cudaSuccess) return e;
    p.n_tiles = (uint32_t)(((uint64_t)p.count + M::kUnit - 1) / M::kUnit);
    const uint32_t grid = p.n_tiles < (uint32_t)ws->sm_count ? p.n_tiles : (uint32_t)ws->sm_count;
    return launch_after(st, kern, grid, M::kThreads, M::kSmemBytes, p);
}

template <int W, int NL, int FMT, int OT>
static cudaError_t launch_train_act(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    switch (narrow::built_activation(p.cfg)) {
    case MLP_ACT_RELU: return launch_train<W, NL, FMT, MLP_ACT_RELU, OT>(st, ws, p);
    case MLP_ACT_LEAKY_RELU: return launch_train<W, NL, FMT, MLP_ACT_LEAKY_RELU, OT>(st, ws, p);
    case MLP_ACT_GELU_TANH: return launch_train<W, NL, FMT, MLP_ACT_GELU_TANH, OT>(st, ws, p);
    default: return launch_train<W, NL, FMT, -1, OT>(st, ws, p);
    }
}

template <int W, int NL>
cudaError_t launch_narrow_train(cudaStream_t st, TcWorkspace* ws, int op, narrow::Params& p)
{
    constexpr int OTX = W == 32 ? 2 : 8;
    const bool few = p.cfg.dims[NL] <= 8;
    if (op == MLP_BF16) return few ? launch_train_act<W, NL, MLP_BF16, 1>(st, ws, p) : launch_train_act<W, NL, MLP_BF16, OTX>(st, ws, p);
    return few ? launch_train_act<W, NL, MLP_F16, 1>(st, ws, p) : launch_train_act<W, NL, MLP_F16, OTX>(st, ws, p);
}
template cudaError_t launch_narrow_train<(MLPB200_NARROW_PART - 1) / 4 ? 64 : 32, 2 + (MLPB200_NARROW_PART - 1) % 4>(cudaStream_t, TcWorkspace*, int, narrow::Params&);
#endif

#if MLPB200_NARROW_PART == 9
template <int W, int FMT, int HACT, int OT>
static cudaError_t launch_forward(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    constexpr int MT = 2;
    auto kern = narrow::forward_narrow_kernel<W, FMT, HACT, OT, MT>;
    p.raw_bytes = 0;
    for (int l = 0; l < p.cfg.n_layers; ++l) p.raw_bytes += (int)((narrow::stored_weight_bytes(p.cfg, l) + 15u) & ~15u);
    const size_t smem = (size_t)p.cfg.n_layers * ((W + 31) / 32 * (W / 8) * 512 + W * 8 + 32) + 48 + (size_t)p.raw_bytes;
    static SmemLimit limit;   // (of the largest network, whatever this one needs)
    const cudaError_t e = limit.raise((const void*)kern, ws->ordinal, 5 * ((W + 31) / 32 * (W / 8) * 512 + W * 8 + 32) + 48 + 5 * W * W * 4);
    if (e != cudaSuccess) return e;
    constexpr uint32_t per_tile = narrow::kForwardWarps * 16 * MT;
    p.n_tiles = (uint32_t)(((uint64_t)p.count + per_tile - 1) / per_tile);
    const uint32_t slots = 2u * (uint32_t)ws->sm_count;
    return launch_after(st, kern, p.n_tiles < slots ? p.n_tiles : slots, 32 * narrow::kForwardWarps, smem, p);
}

template <int W, int FMT, int OT>
static cudaError_t launch_forward_act(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    switch (narrow::built_activation(p.cfg)) {
    case MLP_ACT_RELU: return launch_forward<W, FMT, MLP_ACT_RELU, OT>(st, ws, p);
    case MLP_ACT_LEAKY_RELU: return launch_forward<W, FMT, MLP_ACT_LEAKY_RELU, OT>(st, ws, p);
    case MLP_ACT_GELU_TANH: return launch_forward<W, FMT, MLP_ACT_GELU_TANH, OT>(st, ws, p);
    default: return launch_forward<W, FMT, -1, OT>(st, ws, p);
    }
}

template <int W, int FMT>
static cudaError_t launch_forward_out(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    const int od = p.cfg.dims[p.cfg.n_layers];
    if (od <= 8) return launch_forward_act<W, FMT, 1>(st, ws, p);
    return launch_forward_act<W, FMT, W / 8>(st, ws, p);
}

cudaError_t launch_narrow_forward(cudaStream_t st, TcWorkspace* ws, int op, narrow::Params& p)
{
    int widest = 0;
    for (int l = 0; l <= p.cfg.n_layers; ++l) widest = p.cfg.dims[l] > widest ? p.cfg.dims[l] : widest;
    if (op == MLP_BF16)
        return widest <= 16 ? launch_forward_out<16, MLP_BF16>(st, ws, p) : widest <= 32 ? launch_forward_out<32, MLP_BF16>(st, ws, p)
                                                                                        : launch_forward_out<64, MLP_BF16>(st, ws, p);
    return widest <= 16 ? launch_forward_out<16, MLP_F16>(st, ws, p) : widest <= 32 ? launch_forward_out<32, MLP_F16>(st, ws, p)
                                                                                   : launch_forward_out<64, MLP_F16>(st, ws, p);
}
#endif

#if MLPB200_NARROW_PART == 0
bool tc_train_narrow_supported(const MlpConfig& c)
{
    if (c.n_layers < 2 || c.n_layers > 5) return false;
    const int op = c.operand_dtype ? c.operand_dtype : c.dtype;  // fp32 storage runs here with 16-bit operands
    if (op != MLP_BF16 && op != MLP_F16) return false;
    for (int l = 0; l <= c.n_layers; ++l)
        if (c.dims[l] > 64) return false;
    if (c.encoding == MLP_ENC_FREQ2D && c.dims[0] != 32) return false;
    return true;
}

// Whether rows of `width` values may be read in whole pieces of four (fp32) or eight (16-bit) values from every
// feature that is a multiple of `step`.
static int whole_pieces(uint64_t address, int width, int dtype, int step)
{
    const int need = dtype == MLP_F32 ? 4 : 8;
    return (address & 15u) == 0 && width % (need > step ? need : step) == 0;
}

static narrow::Params narrow_params(TcWorkspace* ws, const MlpConfig& c, uint64_t network, uint64_t inputs, uint32_t count)
{
    narrow::Params p;
    p.cfg = c;
    p.net = (const MlpLayerPointers*)network;
    p.loss_words = nullptr;
    p.status = ws->status;
    p.inputs = (const void*)inputs;
    p.targets = nullptr;
    p.input_grads = nullptr;
    p.outputs = nullptr;
    p.count = count;
    p.n_tiles = 0;
    p.vec_in = whole_pieces(inputs, c.dims[0], c.input_dtype, c.dims[0] <= 16 ? 4 : 8);
    p.vec_tgt = p.vec_out = p.vec_dx = 0;
    return p;
}

cudaError_t launch_forward_narrow(cudaStream_t st, TcWorkspace* ws, const MlpConfig& c, const MlpForwardParams& a,
                                  int* launches, std::string* err)
{
    if (!tc_train_narrow_supported(c)) { if (err) *err = "shape not built for the narrow tensor-core path"; return cudaErrorInvalidValue; }
    if (a.count == 0) return cudaSuccess;
    if (chain_forward_suits(c, a.count)) return launch_forward_chain(st, ws, c, a, launches, err);
    narrow::Params p = narrow_params(ws, c, a.networkBuffer, a.inputs, a.count);
    p.outputs = (float*)a.outputs;
    p.vec_out = whole_pieces(a.outputs, c.dims[c.n_layers], MLP_F32, 4);
    *launches += 1;
    return launch_narrow_forward(st, ws, c.operand_dtype ? c.operand_dtype : c.dtype, p);
}

cudaError_t launch_learn_gradient_narrow(cudaStream_t st, TcWorkspace* ws, const MlpConfig& c, const MlpLearnGradParamsEx& a,
                                         int* launches, std::string* err, float* input_grads)
{
    if (!tc_train_narrow_supported(c)) { if (err) *err = "shape not built for the narrow tensor-core path"; return cudaErrorInvalidValue; }
    if (a.count == 0) return cudaSuccess;
    if (chain_train_suits(c, a.count)) return launch_learn_gradient_chain(st, ws, c, a, launches, err, input_grads);
    narrow::Params p = narrow_params(ws, c, a.networkBuffer, a.inputs, a.count);
    p.loss_words = (uint32_t*)a.lossBuffer;
    p.targets = (const void*)a.targets;
    p.input_grads = input_grads;
    p.vec_tgt = whole_pieces(a.targets, c.dims[c.n_layers], c.target_dtype, 8);
    p.vec_dx = whole_pieces((uint64_t)input_grads, c.dims[0], MLP_F32, 4);
    *launches += 1;
    const int op = c.operand_dtype ? c.operand_dtype : c.dtype;
    // Padded width 32 where every width fits it and the outputs fit one 16-row block of its gradient accumulators.
    bool fits32 = c.dims[c.n_layers] <= 16;
    for (int l = 0; l <= c.n_layers; ++l) fits32 = fits32 && c.dims[l] <= 32;
    switch (c.n_layers) {
    case 2: return fits32 ? launch_narrow_train<32, 2>(st, ws, op, p) : launch_narrow_train<64, 2>(st, ws, op, p);
    case 3: return fits32 ? launch_narrow_train<32, 3>(st, ws, op, p) : launch_narrow_train<64, 3>(st, ws, op, p);
    case 4: return fits32 ? launch_narrow_train<32, 4>(st, ws, op, p) : launch_narrow_train<64, 4>(st, ws, op, p);
    case 5: return fits32 ? launch_narrow_train<32, 5>(st, ws, op, p) : launch_narrow_train<64, 5>(st, ws, op, p);
    }
    return cudaErrorInvalidValue;
}
#endif

}  // namespace mlpb200
