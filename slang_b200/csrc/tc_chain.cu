// learnGradient for networks of widths up to 128 and forward for widths up to 64, 16-bit storage, ReLU or leaky ReLU hidden layers: tcgen05
// products over whole tiles of 128 samples, up to six tiles in flight per SM (tc_chain.cuh).  tc_narrow.cu and tc_kernels.cu have the other
// networks, the smallest batches and what the rules below leave them.
//
//   forward   Z_l [128 x H]    = 1 . b_l^T + A_l [128 x W] . W_l^T   A: A_l, K-major      B: W_l [out][in], K-major
//   input     dA_l [128 x H]   = dZ_l [128 x H] . W_l                A: dZ_l, K-major     B: W_l, MN-major
//   weights   dW_l | db_l [64 x (W + 8)] += dZ_l^T . [A_l | 1]       A: dZ_l, MN-major    B: A_l, then a tile whose first column is ones
//
// Bound by instruction issue and by the hand-offs between a chain's four warps and the tensor pipe; the chains' tiles fill
// shared memory, so there are no more of them.  Against the register-chained kernels of tc_narrow.cu, us: texture network
// (32-64-64-64-3) 2^24 samples a step 3830 -> 2110, width 32 (4-32-32-32-32-4, leaky ReLU) 2^20 samples 160 -> 130, 1920 x 1080 view of the
// texture network 142 -> 94.  Counters of 2^20 samples of the texture network: issue slots 44 %, tensor pipe 37 %, LSU wavefronts 40 %.
//
// What the reference does instead: one thread per sample with per-element global atomics
// (examples/mlp-training/mlp_sw.slang:28-58) or CoopVec calls whose CPU/CUDA fallback is scalar loops
// (examples/mlp-training-coopvec/fflayer.slang:16-58, source/slang/hlsl.meta.slang:32835-32912).
#include <cuda.h>
#include <cuda_runtime.h>

#include <string>

#include "launch_pdl.cuh"
#include "launchers.h"
#include "tc_chain.cuh"
#include "tc_host.h"

namespace mlpb200 {

using namespace ptx;

namespace chain {

enum : uint32_t { kStatusIssue = 0x20000u, kStatusRow = 0x40000u, kStatusGrad = 0x80000u };

// Warps that issue gradient products: two (even and odd layers) beside four chains; with three, sixteen warps in all leave
// each thread 128 registers and seventeen 96.
__host__ __device__ constexpr int grad_warps(int chains) { return chains == 3 ? 1 : 2; }
// Width 32: warps that take the windows' sums, one for each quarter of the lanes that has rows (registers are dealt four warps at a time, so they cost none).
__host__ __device__ constexpr int sum_warps(int h) { return h == 32 ? 2 : 0; }

// Shared-memory map of the training kernel (bytes from a 1024-aligned base).  H: padded hidden width; IW: padded input
// width; OW: padded output width; NCH: chains.
template <int H, int NL, int IW, int OW, int NCH>
struct TrainMap {
    static constexpr int kWarps = 4 * NCH;                // with samples; one more per chain issues its layer products, one or two the gradient products
    static constexpr int kGradWarps = grad_warps(NCH);
    static constexpr bool kWide = H == 128;
    // An accumulator in tensor memory is not rounded but cut off: every addition loses up to a unit in the last place, always toward zero.  Where all samples pull
    // one way, a gradient summed there over all of a CTA's tiles is 1e-7 short for every 16 samples: 4.5e-5 at 2^20 samples, 7e-4 at 2^24.  So what the kernels
    // of tc_narrow.cu and tc_kernels.cu sum in registers (all of width 32; dW_0 and the biases of width 128) is summed there over windows of a few tiles, and the windows
    // in fp32.  (What they sum in tensor memory too, all of width 64 and the hidden layers' dW at 128, is summed there over all tiles.)
    static constexpr bool kWindows = H != 64;
    // Width 32: windows of four tiles, one for each chain, are 2.9e-6 short at any batch (the register sums 5.3e-6 at 2^20, 9e-5 at 2^24).  Warps of their own take
    // them: a step of 2^20 samples of 4-32-32-32-32-4 takes 129.9 us, 141.6 with the tiles' warps taking them between two layers, 124.2
    // without windows; windows of eight tiles 129.1.
    static constexpr uint32_t kWindow = 4;
    // Width 128: dW_0 and db_0 are taken with every tile (1.3e-6, the register sums 1.0e-6), the other biases with some 32 (sums of 16-bit values are
    // exact for about as long), by the chain's warps: 2^20 samples of 32-128-128-3 231.8 -> 233.9 us, of 32-128-128-128-3 437.7 -> 452.
    // Whether tile `turn` of chain c (of its own count, at least modulo 16) ends a window of layer l.
    __host__ __device__ static constexpr bool ends_window(int l, uint32_t c, uint32_t turn) { return kWide && (l == 0 || (c == 0u && (turn & 15u) == 15u)); }
    static constexpr int kSumWarps = sum_warps(H);
    static_assert(kSumWarps == 0 || (kWarps + NCH) % 4 == 0, "the sums' warps reach the quarters 0 and 1");
    static constexpr int kThreads = 32 * (kWarps + NCH + kSumWarps + kGradWarps);
    static constexpr int kDzW = OW == 16 ? 32 : OW;            // row width of the last layer's dZ
    __host__ __device__ static constexpr int in_w(int l) { return l == 0 ? IW : H; }
    __host__ __device__ static constexpr int out_w(int l) { return l == NL - 1 ? OW : H; }
    static constexpr uint32_t kRowsIn = kTile * IW * 2, kRows = kTile * H * 2, kPanel = kTile * 128;   // (of 64 features)
    // A chain's tiles: A_0, A_1 .. A_{NL-1} (dZ_{l-1} replaces A_l), dZ_{NL-1}.  The first and the last change places with every
    // tile, so that a tile's inputs need not wait for the gradient product that still reads the last one's.
    static_assert(IW == kDzW, "inputs and the last layer's dZ share their layout");
    __host__ __device__ static constexpr uint32_t a_off(int l) { return l == 0 ? 0u : kRowsIn + (uint32_t)(l - 1) * kRows; }
    static constexpr uint32_t kDz = a_off(NL);
    static constexpr uint32_t kChainBytes = kDz + kTile * kDzW * 2;
    __host__ __device__ static constexpr uint32_t w_off(int l) { return l == 0 ? 0u : (uint32_t)H * IW * 2 + (uint32_t)(l - 1) * H * H * 2; }
    static constexpr uint32_t kWeights = 0;
    static constexpr uint32_t kChains = (w_off(NL - 1) + (uint32_t)OW * H * 2 + 1023) & ~1023u;
    static constexpr uint32_t kOnesIn = kChains + NCH * kChainBytes;   // 16 rows whose first element is one, in the layout of A_0
    static constexpr int kOnesW = H == 32 ? 32 : 64;
    static constexpr uint32_t kOnes = kOnesIn + (IW == kOnesW ? 0 : 16 * IW * 2);
    static constexpr uint32_t kUnit = kOnes + 16 * kOnesW * 2;
    static constexpr uint32_t kHiddenBias = kUnit + kUnitBytes;        // [NL - 1][H rows][16]
    static constexpr uint32_t kBias = kHiddenBias + (NL - 1) * H * 32; // the output layer's, fp32 [OW]
    static constexpr uint32_t kLoss = kBias + OW * 4;              // fp32 [kWarps][2]
    static constexpr uint32_t kBars = kLoss + kWarps * 8;              // per chain: ready, acc_full, and for each gradient warp dz_ready, dw_done
    static constexpr uint32_t kTaken = kBars + (2 + 2 * kGradWarps) * NCH * 8;   // more barriers, one a layer: a window's sums are taken
    static constexpr uint32_t kEnded = kTaken + (kWindows ? NL * 8 : 0);         // width 32, one a layer: a window's last product has completed
    static constexpr uint32_t kTmemPtr = kEnded + (kSumWarps ? NL * 8 : 0);
    static constexpr uint32_t kAbort = kTmemPtr + 4;
    static constexpr uint32_t kOpen = kAbort + 4;                      // bit l: layer l has products in tensor memory that no window took
    static constexpr uint32_t kNet = (kOpen + 4 + 15) & ~15u;
    // Sums of whole windows, fp32: biases [layer][H], then weights [layer][rows][32] with 16-byte chunks ^ (row % 8).  (Of width 128 only dW_0,
    // and only where tensor memory has no room for it.)
    static constexpr uint32_t kBiasSums = (kNet + NL * 32 + 15) & ~15u;
    static constexpr uint32_t kSums = (kBiasSums + (kWindows ? NL * H * 4 : 0) + 127) & ~127u;
    static constexpr bool kSumsInTmem = kWide && NL < 4;
    static constexpr uint32_t kSumsBytes = !kWindows || kSumsInTmem ? 0 : kWide ? H * 128 : ((NL - 1) * H + OW) * 128;
    static constexpr uint32_t kSmemBytes = kSums + kSumsBytes + 1024;
    // the outgoing gradients: fp32 [layers at a time][H][H + 1], over the chains' tiles
    static constexpr uint32_t kSumRow = H + 1;
    static constexpr int kSumLayers = kWide ? 1 : NL;
    static_assert(kSumLayers * H * kSumRow * 4 <= kOnesIn, "room for the sums");
    static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
    // Tensor memory: an accumulator per chain, then the gradients, which the chains share.  Up to width 64 dW_l | db_l is one
    // product of 64 rows; at 128 dW_l has 128 rows (and the last layer's lies the other way round, in features by outputs)
    // and db_l is a product of its own.
    __host__ __device__ static constexpr uint32_t dw_cols(int l) { return (uint32_t)in_w(l) + 16; }
    __host__ __device__ static constexpr uint32_t dw_col(int l)
    {
        if (kWide) return NCH * (uint32_t)H + (l == 0 ? (NL - 2) * 128u : l < NL - 1 ? (l - 1) * 128u : (NL - 2) * 128u + IW);
        return NCH * (uint32_t)H + (l == 0 ? 0u : dw_cols(0) + (uint32_t)(l - 1) * (H + 16));
    }
    __host__ __device__ static constexpr uint32_t db_col(int l) { return NCH * (uint32_t)H + (NL - 2) * 128u + IW + OW + 16u * (uint32_t)l; }
    __host__ __device__ static constexpr uint32_t sum_col() { return db_col(NL); }   // kSumsInTmem
    static_assert((kWide ? db_col(NL) + (kSumsInTmem ? IW : 0) : dw_col(NL)) <= 512, "tensor memory budget");
};

// Adds what layer l's products have summed in tensor memory since its last window to the sums of windows: dW and db, of width 128 only dW_0 and
// db.  By one warp for each lane quarter with rows (width 32: 0 and 1); `lanes` is the tensor-memory address of the warp's.
template <class M, int H, int NL, int IW>
static __device__ __noinline__ void take_window(uint32_t lanes, uint32_t sbase, int l)
{
    const int lane = threadIdx.x & 31, quarter = (int)(threadIdx.x >> 5) & 3;
    const bool half = !M::kWide || l == NL - 1;   // 64 rows: on lanes 0 to 15 of each quarter
    const int row = half ? quarter * 16 + lane : quarter * 32 + lane;
    const bool real = (!half || lane < 16) && row < (l == NL - 1 ? M::out_w(NL - 1) : H);
    const uint32_t bias = sbase + M::kBiasSums + 4u * (uint32_t)(l * H + row);
    tc_fence_after();
    uint32_t b;
    if constexpr (M::kWide) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(b) : "r"(lanes + M::db_col(0) + 16u * (uint32_t)l) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(b)::"memory");
        if (l == 0) {
            const uint32_t at = sbase + M::kSums + (uint32_t)row * 128u;
#pragma unroll 1
            for (int c = 0; c < IW; c += 16) {
                uint32_t v[16], s[16];
                tmem_ld_32x16(lanes + M::dw_col(0) + (uint32_t)c, v);
                if constexpr (M::kSumsInTmem) {
                    tmem_ld_32x16(lanes + M::sum_col() + (uint32_t)c, s);
                    wait_ld(v);
                    wait_ld(s);
#pragma unroll
                    for (int i = 0; i < 16; ++i) s[i] = __float_as_uint(__uint_as_float(s[i]) + __uint_as_float(v[i]));
                    tmem_st_32x16(lanes + M::sum_col() + (uint32_t)c, s);
                } else {
                    wait_ld(v);
                    add_chunks<4>(at, row, c / 4, v);
                }
            }
            if constexpr (M::kSumsInTmem) tmem_st_wait();
        }
    } else {
        const uint32_t col = lanes + (l == 0 ? M::dw_col(0) : M::dw_col(1) + (uint32_t)(l - 1) * (H + 16));
        uint32_t v[32];
        tmem_ld_32x32(col, v);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(b) : "r"(col + (uint32_t)H) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(b)::"memory");
        wait_ld(v);
        if (real) add_chunks<8>(sbase + M::kSums + (uint32_t)(l * H + row) * 128u, row, 0, v);
    }
    if (real) {
        float x;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(bias) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(bias), "f"(x + __uint_as_float(b)) : "memory");
    }
    tc_fence_before();
    __syncwarp();
}

template <int H, int NL, int IW, int OW, int NCH, int FMT, int HACT>
__global__ void __launch_bounds__(32 * (5 * NCH + sum_warps(H) + grad_warps(NCH)), 1) learn_gradient_chain_kernel(const __grid_constant__ Params p)
{
    using M = TrainMap<H, NL, IW, OW, NCH>;
    using C = Cvt<FMT>;
    constexpr int kThreads = M::kThreads, NW = M::kWarps, G = M::kGradWarps;
    constexpr bool kOverflow = M::kWide && HACT == MLP_ACT_RELU;   // reverse_whole_row() where a dA is not finite
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const MlpConfig& cfg = p.cfg;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    uint64_t* ready = (uint64_t*)(smem + M::kBars);   // the chain's operand rows are written and its accumulator is drained
    uint64_t* acc_full = ready + NCH;                 // a layer product has completed
    uint64_t* dz_ready = acc_full + NCH;              // [chain][layer % G]: a dZ is written
    uint64_t* dw_done = dz_ready + G * NCH;           // [chain][layer % G]: a gradient product has completed
    uint64_t* taken = (uint64_t*)(smem + M::kTaken);  // [layer]: a window's sums have left tensor memory
    uint64_t* ended = (uint64_t*)(smem + M::kEnded);  // [layer], width 32: a window's last product has completed
    volatile uint32_t* abort_flag = (volatile uint32_t*)(smem + M::kAbort);
    const int od = cfg.dims[NL];

    // ---- set-up ----
    if (threadIdx.x == 0) {
        for (int c = 0; c < NCH; ++c) {
            mbar_init(&ready[c], 4);
            mbar_init(&acc_full[c], 1);
            for (int g = 0; g < G; ++g) {
                mbar_init(&dz_ready[G * c + g], 4);
                mbar_init(&dw_done[G * c + g], 1);
            }
        }
        if constexpr (M::kWindows) {
            for (int l = 0; l < NL; ++l) {
                mbar_init(&taken[l], M::kWide ? 4 : 2);
                if (M::kSumWarps) mbar_init(&ended[l], 1);
            }
            *(uint32_t*)(smem + M::kOpen) = 0u;
        }
        *abort_flag = 0u;
        fence_mbar_init();
    }
    if constexpr (M::kWindows) {
        for (uint32_t i = M::kBiasSums + 16u * threadIdx.x; i < M::kSums + M::kSumsBytes; i += 16u * kThreads) *(uint4*)(smem + i) = make_uint4(0u, 0u, 0u, 0u);
    }
    constexpr int OH = M::kOnesW;
    for (int i = threadIdx.x; i < 16 * OH / 2; i += kThreads) {
        const int row = i / (OH / 2), word = i % (OH / 2);
        ((uint32_t*)(smem + M::kOnes))[i] = (uint32_t)(word * 4) == row_at<OH>(row) - (uint32_t)row * OH * 2 ? (C::kOnes & 0xffffu) : 0u;
    }
    if constexpr (IW != OH) {
        for (int i = threadIdx.x; i < 16 * IW / 2; i += kThreads) {
            const int row = i / (IW / 2), word = i % (IW / 2);
            ((uint32_t*)(smem + M::kOnesIn))[i] = (uint32_t)(word * 4) == row_at<IW>(row) - (uint32_t)row * IW * 2 ? (C::kOnes & 0xffffu) : 0u;
        }
    }
    grid_wait();
    if (warp == NW + NCH) {
        tmem_alloc((uint32_t*)(smem + M::kTmemPtr), 512);
        tmem_relinquish();
        grid_release();
    }
    const MlpLayerPointers* s_net = (const MlpLayerPointers*)(smem + M::kNet);
    if (threadIdx.x < NL * 4) ((uint64_t*)(smem + M::kNet))[threadIdx.x] = ((const uint64_t*)p.net)[threadIdx.x];
    __syncthreads();
    if constexpr (M::kSumsInTmem) {
        if (warp < 4) {
            const uint32_t zero[16] = {};
            const uint32_t at = *(volatile uint32_t*)(smem + M::kTmemPtr) + ((uint32_t)(warp * 32) << 16) + M::sum_col();
#pragma unroll
            for (int c = 0; c < IW; c += 16) tmem_st_32x16(at + (uint32_t)c, zero);
            tmem_st_wait();
        }
    }
    stage_weights<IW>(smem + M::kWeights, cfg, (const void*)s_net[0].weights, H, cfg.dims[0], cfg.dims[1], threadIdx.x, kThreads);
#pragma unroll 1
    for (int l = 1; l < NL; ++l)
        stage_weights<H>(smem + M::kWeights + M::w_off(1) + (uint32_t)(l - 1) * (H * H * 2), cfg, (const void*)s_net[l].weights, l == NL - 1 ? OW : H,
                         cfg.dims[l], cfg.dims[l + 1], threadIdx.x, kThreads);
    // hidden features past the real width: below zero for ReLU, so that no derivative there is the one at zero
    first_column(smem + M::kUnit, 8, threadIdx.x, kThreads, [](int) { return C::kOnes; });
    first_column(smem + M::kHiddenBias, (NL - 1) * H, threadIdx.x, kThreads, [&](int row) -> uint32_t {
        const int l = row / H, f = row % H;
        return f < cfg.dims[l + 1] ? ((const uint16_t*)s_net[l].biases)[f] : HACT == MLP_ACT_RELU ? C::kOnes | 0x8000u : 0u;
    });
    for (int i = threadIdx.x; i < OW; i += kThreads)
        ((float*)(smem + M::kBias))[i] = i < od ? load_as_f32(cfg.dtype, (const void*)s_net[NL - 1].biases, i) : 0.0f;
    cp_async_wait_all();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *(volatile uint32_t*)(smem + M::kTmemPtr);
    const uint32_t stride = gridDim.x * NCH;
    bool ok = true;
    auto tiles_here = [&]() {   // the CTA's
        uint32_t n = 0;
        for (int c = 0; c < NCH; ++c) {
            const uint32_t first = blockIdx.x + gridDim.x * (uint32_t)c;
            n += first < p.n_tiles ? (p.n_tiles - first + stride - 1) / stride : 0u;
        }
        return n;
    };

    if (warp < NW) {
        // =================================== samples ===============================================
        const int ch = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t t_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ch * H);
        const uint32_t cb = sbase + M::kChains + (uint32_t)ch * M::kChainBytes;
        uint32_t in_row = cb + row_at<IW>(r), dz_row = cb + M::kDz + row_at<M::kDzW>(r);   // change places with every tile
        const uint32_t own_row = cb + M::kRowsIn + row_at<H>(r);
        const uint32_t s_bias = sbase + M::kBias;
        const float scale = cfg.loss == MLP_LOSS_MSE_MEAN ? 1.0f / (float)od : 1.0f;
        const float alpha = cfg.act_alpha, alpha_op = C::round(alpha);
        float run_max = 0.0f, run_sum = 0.0f;
        uint32_t full = 0, done = 0;                   // phases seen of acc_full; bit g: parity of dw_done's g, from bit 2 on the chain's tiles so far
        auto wait_full = [&]() {
            ok = ok && wait_for(&acc_full[ch], full & 1u, abort_flag, p.status, kStatusRow);
            ++full;
            tc_fence_after();
        };
        auto wait_done = [&](int l) {
            ok = ok && wait_for(&dw_done[G * ch + l % G], (done >> (l % G)) & 1u, abort_flag, p.status, kStatusRow);
            done ^= 1u << (l % G);
        };
        // hands A_l over (gradient < 0), or dZ of layer `gradient`
        auto release = [&](bool product, int gradient) {
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (product) mbar_arrive(&ready[ch]);
                if (gradient >= 0) mbar_arrive(&dz_ready[G * ch + gradient % G]);
            }
        };
        // width 128: takes layer l's sums if this chain's tile `of`, whose product has completed, ends a window
        auto take = [&](int l, uint32_t of) {
            if constexpr (M::kWide) {
                if (!M::ends_window(l, (uint32_t)ch, of)) return;
                take_window<M, H, NL, IW>(t_acc - (uint32_t)(ch * H), sbase, l);
                if (lane == 0) mbar_arrive(&taken[l]);
            }
        };
        RawRow raw;
        uint32_t tile = blockIdx.x + gridDim.x * (uint32_t)ch;
        uint64_t sample = (uint64_t)tile * kTile + (uint64_t)r;
        Rows in(p.inputs, stored_inputs(cfg), cfg.input_dtype, sample, stride * kTile), tgt(p.targets, od, cfg.target_dtype, sample, stride * kTile);
        const bool wide_target = cfg.target_dtype == MLP_F32;
        fetch_row(raw, p, in.at, sample < p.count);
        for (; tile < p.n_tiles && ok; tile += stride) {
            const bool valid = sample < p.count;
            bool zero_seen = false;
            // ---- input row ----
            write_row<FMT, IW>(in_row, p, raw, in.at, valid);
            release(true, -1);
            // few targets are fetched a forward pass ahead of their use; the next tile's rows are started on their way
            uint32_t t4[4];
            if (od <= 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) t4[i] = load_bits(tgt.at, wide_target, i, valid && i < od);
            }
            const char* targets = tgt.at;
            const uint64_t current = sample;
            sample += (uint64_t)stride * kTile;
            in.at += in.step;
            tgt.at += tgt.step;
            fetch_row(raw, p, in.at, sample < p.count);
            if (sample < p.count) {
                if (!short_row(cfg)) prefetch_row(in.at);
                prefetch_row(tgt.at);
            }
            // ---- forward, hidden layers ----
#pragma unroll 1
            for (int l = 0; l < NL - 1; ++l) {
                wait_full();
                if (l == 0) {   // the last tile's dZ_0 lies where A_1 goes, its A_0 where dZ_{NL-1} will
                    if (done > 3u) wait_done(0);
                }
                if (!ok) break;
                const uint32_t dst = own_row + (uint32_t)l * M::kRows;   // A_{l + 1}
                float least = 1.0f;
                uint32_t v[H == 32 ? 1 : 2][32];
                tmem_ld_32x32(t_acc, v[0]);
#pragma unroll
                for (int b = 0; b < H / 32; ++b) {   // the next block's read runs under this one's arithmetic
                    wait_ld(v[b & 1]);
                    if (b + 1 < H / 32) tmem_ld_32x32(t_acc + (uint32_t)(32 * b + 32), v[(b + 1) & (H == 32 ? 0 : 1)]);
                    hidden_columns<FMT, HACT>(v[b & 1], block_at<H>(dst, b), alpha, least);
                }
                if (HACT == MLP_ACT_RELU && __any_sync(0xffffffffu, least <= 0.5f * C::kSmallest)) {   // one that rounds to zero
                    zero_seen = true;
                    marked_columns<FMT, H>(t_acc, dst);
                }
                release(true, -1);
                if (l == 0 && done > 3u) take(0, (done >> 2) - 1u);
            }
            // ---- output layer, loss, dZ of the last layer ----
            wait_full();
            if (!ok) break;
            float loss = 0.0f;
#pragma unroll 1
            for (int f = 0; f < od; f += 4) {
                float o[4], d[4], t[4] = {0.0f, 0.0f, 0.0f, 0.0f}, g[4];
                output_columns<FMT>(o, t_acc, s_bias, f);
                if (od <= 4) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) t[i] = bits_value(cfg.target_dtype, t4[i]);
                } else if (valid) {
                    load_targets(t, p, targets, od, f);
                }
                activate_outputs(cfg.output_act, alpha, o, d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool real = valid && f + i < od;
                    const float diff = real ? o[i] - t[i] : 0.0f;
                    loss = fmaf(diff * scale, diff, loss);
                    g[i] = real ? ((2.0f * scale) * diff) * d[i] : 0.0f;
                }
                sts64((dz_row ^ (uint32_t)(16 * (f >> 3))) + (uint32_t)(2 * (f & 4)), C::pack2(g[0], g[1]), C::pack2(g[2], g[3]));
            }
#pragma unroll 1
            for (int f = (od + 3) & ~3; f < ((od + 15) & ~15); f += 4)   // the rest of the K step
                sts64((dz_row ^ (uint32_t)(16 * (f >> 3))) + (uint32_t)(2 * (f & 4)), 0u, 0u);
            run_max = fmaxf(run_max, loss);
            run_sum += loss;
            release(true, NL - 1);
            // ---- backward: dA_l times the derivative is dZ_{l-1}, written over A_l once the gradient product has read it ----
#pragma unroll 1
            for (int l = NL - 1; l >= 1; --l) {
                wait_full();
                if (!ok) break;
                const uint32_t at = own_row + (uint32_t)(l - 1) * M::kRows;   // A_l
                uint32_t v[H == 32 ? 1 : 2][32];
                bool whole = HACT == MLP_ACT_RELU && zero_seen;
                tmem_ld_32x32(t_acc, v[0]);
                wait_ld(v[0]);
                if constexpr (kOverflow && FMT == MLP_F16) whole = whole || __any_sync(0xffffffffu, not_finite<FMT>(v[0]));
                if (whole) {
                    wait_done(l);
                    if (!ok) break;
                    reverse_whole_row<FMT, H>(t_acc, at);
                } else {
                    uint32_t z[H / 32][16];
                    bool odd = false;
#pragma unroll
                    for (int b = 0; b < H / 32; ++b) {
                        if (b > 0) wait_ld(v[b & 1]);
                        if (b + 1 < H / 32) tmem_ld_32x32(t_acc + (uint32_t)(32 * b + 32), v[(b + 1) & (H == 32 ? 0 : 1)]);
                        reverse_columns<FMT, HACT>(z[b], v[b & 1], block_at<H>(at, b), alpha_op);
                        if constexpr (kOverflow && FMT == MLP_BF16) odd = odd || not_finite<FMT>(v[b & 1]);
                    }
                    if constexpr (kOverflow && FMT == MLP_BF16) odd = __any_sync(0xffffffffu, odd);
                    wait_done(l);
                    if (!ok) break;
                    if (odd) {
                        reverse_whole_row<FMT, H>(t_acc, at);
                    } else {
#pragma unroll
                        for (int j = 0; j < H / 8; ++j) {
                            const uint32_t* w = &z[j >> 2][4 * (j & 3)];
                            sts128(block_at<H>(at, j >> 2) ^ (uint32_t)(16 * (j & 3)), w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                release(l > 1 || p.input_grads, l - 1);
                take(l, done >> 2);
            }
            done += 4u;
            // ---- optional: the input gradients dZ_0 . W_0, rounded to the storage type ----
            if (p.input_grads) {
                wait_full();
                if (!ok) break;
                const int in = cfg.dims[0];
                float* row = p.input_grads + current * (uint64_t)in;
#pragma unroll 1
                for (int f = 0; f < in; f += 8) {
                    uint32_t v[8];
                    tmem_ld_32x8(t_acc + (uint32_t)f, v);
                    tmem_ld_wait();
                    float x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = C::round(__uint_as_float(v[i]));
                    if (!valid) continue;
                    if (p.vec_dx) {
                        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row + f), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]),
                                     "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
                                     : "memory");
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (f + i < in) row[f + i] = x[i];
                    }
                }
                tc_fence_before();
            }
            const uint32_t swap = in_row;
            in_row = dz_row;
            dz_row = swap;
        }
        if (done > 3u) {
            wait_done(0);
            if (ok) take(0, (done >> 2) - 1u);
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
    } else if (warp < NW + NCH) {
        // =================================== layer products of one chain ===========================
        const int ch = warp - NW;
        const uint32_t lo = (sbase & 0x3FFFFu) >> 4;
        const uint32_t cb = M::kChains + (uint32_t)ch * M::kChainBytes;
        const uint32_t acc = tmem_base + (uint32_t)(ch * H);
        const int in_steps = (cfg.dims[0] + 15) / 16, out_steps = (od + 15) / 16;
        constexpr uint32_t F = C::kUmmaFmt;
        // A copy of the code per layer up to width 64 (width 32, 2^20 samples: 123.5 us, 128.5 with one for all layers), one at 128 (229
        // us for 2^20 samples of 32-128-128-3, 237 with a copy each).
        uint32_t seen = 0, x = cb, y = cb + M::kDz;   // A_0 and the last dZ
        auto wait_ready = [&]() {
            ok = ok && wait_for(&ready[ch], seen & 1u, abort_flag, p.status, kStatusIssue);
            ok = __all_sync(0xffffffffu, ok);
            ++seen;
            tc_fence_after();
        };
        for (uint32_t tile = blockIdx.x + gridDim.x * (uint32_t)ch; tile < p.n_tiles && ok; tile += stride) {
            if constexpr (M::kWide) {
#pragma unroll 1
                for (int l = 0; l < NL; ++l) {
                    wait_ready();
                    if (ok && elect_one()) {
                        if (l < NL - 1) umma_f16(acc, desc_unit(lo, M::kUnit), desc_k<16>(lo, M::kHiddenBias + (uint32_t)l * (H * 32), 0), umma_idesc(F, 0, 0, 128, H), 0u);
                        if (l == 0) {
#pragma unroll
                            for (int k = 0; k < IW / 16; ++k)
                                if (k < in_steps) umma_f16(acc, desc_k<IW>(lo, x, k), desc_k<IW>(lo, M::kWeights, k), umma_idesc(F, 0, 0, 128, H), 1u);
                        } else {
                            const uint32_t a = cb + M::kRowsIn + (uint32_t)(l - 1) * M::kRows, w = M::kWeights + M::w_off(1) + (uint32_t)(l - 1) * (H * H * 2);
                            const uint32_t id = l < NL - 1 ? umma_idesc(F, 0, 0, 128, H) : umma_idesc(F, 0, 0, 128, OW), panel = l < NL - 1 ? H * 128u : OW * 128u;
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, a, k, M::kPanel), desc_k<H>(lo, w, k, panel), id, l < NL - 1 || k > 0);
                        }
                        umma_commit(&acc_full[ch]);
                    }
                    __syncwarp();
                }
#pragma unroll 1
                for (int l = NL - 1; l >= (p.input_grads ? 0 : 1); --l) {
                    wait_ready();
                    if (ok && elect_one()) {
                        const uint32_t w = M::kWeights + M::w_off(1) + (uint32_t)(l - 1) * (H * H * 2), z = cb + M::kRowsIn + (uint32_t)l * M::kRows;
                        if (l == NL - 1) {
#pragma unroll
                            for (int k = 0; k < OW / 16; ++k)
                                if (k < out_steps)
                                    umma_f16(acc, desc_k<M::kDzW>(lo, y, k), desc_mn<H>(lo, w, k, (uint32_t)OW * 128u), umma_idesc(F, 0, 1, 128, H), k > 0);
                        } else if (l > 0) {
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, z, k, M::kPanel), desc_mn<H>(lo, w, k, (uint32_t)H * 128u), umma_idesc(F, 0, 1, 128, H), k > 0);
                        } else {
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, z, k, M::kPanel), desc_mn<IW>(lo, M::kWeights, k), umma_idesc(F, 0, 1, 128, IW), k > 0);
                        }
                        umma_commit(&acc_full[ch]);
                    }
                    __syncwarp();
                }
            } else {
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    wait_ready();
                    if (ok && elect_one()) {
                        if (l < NL - 1) umma_f16(acc, desc_unit(lo, M::kUnit), desc_k<16>(lo, M::kHiddenBias + (uint32_t)l * H * 32, 0), umma_idesc(F, 0, 0, 128, H), 0u);
                        if (l == 0) {
#pragma unroll
                            for (int k = 0; k < IW / 16; ++k)
                                if (k < in_steps) umma_f16(acc, desc_k<IW>(lo, x, k), desc_k<IW>(lo, M::kWeights, k), umma_idesc(F, 0, 0, 128, H), 1u);
                        } else {
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, cb + M::a_off(l), k, M::kPanel), desc_k<H>(lo, M::kWeights + M::w_off(l), k, (uint32_t)M::out_w(l) * 128u), umma_idesc(F, 0, 0, 128, M::out_w(l)),
                                         l < NL - 1 || k > 0);
                        }
                        umma_commit(&acc_full[ch]);
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int l = NL - 1; l >= 0; --l) {
                    if (l == 0 && !p.input_grads) break;
                    wait_ready();
                    if (ok && elect_one()) {
                        if (l == NL - 1) {
#pragma unroll
                            for (int k = 0; k < OW / 16; ++k)
                                if (k < out_steps)
                                    umma_f16(acc, desc_k<M::kDzW>(lo, y, k), desc_mn<H>(lo, M::kWeights + M::w_off(l), k, (uint32_t)OW * 128u), umma_idesc(F, 0, 1, 128, H), k > 0);
                        } else if (l > 0) {
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, cb + M::a_off(l + 1), k, M::kPanel), desc_mn<H>(lo, M::kWeights + M::w_off(l), k, (uint32_t)H * 128u), umma_idesc(F, 0, 1, 128, H), k > 0);
                        } else {
#pragma unroll
                            for (int k = 0; k < H / 16; ++k)
                                umma_f16(acc, desc_k<H>(lo, cb + M::a_off(1), k, M::kPanel), desc_mn<IW>(lo, M::kWeights, k), umma_idesc(F, 0, 1, 128, IW), k > 0);
                        }
                        umma_commit(&acc_full[ch]);
                    }
                    __syncwarp();
                }
            }
            const uint32_t swap = x;
            x = y;
            y = swap;
        }
    } else if (warp < NW + NCH + M::kSumWarps) {
        // =================================== the windows' sums =====================================
        // The n-th product of a layer comes before the n-th of the layer before it, so windows end in this order.
        if constexpr (M::kSumWarps > 0) {
            const uint32_t windows = tiles_here() / M::kWindow;
#pragma unroll 1
            for (uint32_t n = 0; n < windows && ok; ++n) {
#pragma unroll 1
                for (int l = NL - 1; l >= 0; --l) {
                    ok = ok && wait_for(&ended[l], n & 1u, abort_flag, p.status, kStatusGrad);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    take_window<M, H, NL, IW>(tmem_base + ((uint32_t)((warp & 3) * 32) << 16), sbase, l);
                    if (lane == 0) mbar_arrive(&taken[l]);
                }
            }
        }
    } else {
        // =================================== gradient products of all chains =======================
        // Warp g takes the layers g, g + G, .. of whichever chain has a dZ ready; one thread issues all
        // products into one accumulator, so those are in order.  (The loop is kept small: with a copy of the code per chain and
        // layer, its instructions were fetched anew each time.)
        const int g = warp - NW - NCH - M::kSumWarps;
        const uint32_t lo = (sbase & 0x3FFFFu) >> 4;
        constexpr uint32_t F = C::kUmmaFmt;
        const uint32_t top = (uint32_t)(NL - 1 - (NL - 1 - g) % G);        // this warp's last layer; its first is g
        uint32_t total = tiles_here() * (top / G + 1), idle = 0;   // hand-overs to come
        uint32_t started = 0, phase = 0, layers = 0;               // layers begun; four bits a chain: its layer
        uint32_t turns = 0;                                        // eight bits a chain: its tiles so far, modulo 16
        uint32_t over = 0, parity = 0;                             // layers whose window has ended and may not be taken yet; their parities of `taken`
        uint32_t summed = 0, filled = 0;                           // width 128: layers whose db's window has begun; width 32, four bits a layer: tiles in its window
        for (int c = 0; c < NCH; ++c) layers |= top << (4 * c);
        uint32_t c = 0;
#pragma unroll 1
        while (total > 0 && ok) {
            const uint32_t l = (layers >> (4 * c)) & 15u;
            bool go = __all_sync(0xffffffffu, mbar_test_wait(&dz_ready[G * c + g], (phase >> c) & 1u));
            if (M::kWindows && go && (over >> l) & 1u) go = __all_sync(0xffffffffu, mbar_test_wait(&taken[l], (parity >> l) & 1u));
            if (go) {
                tc_fence_after();
                const uint32_t cb = M::kChains + c * M::kChainBytes;
                const uint32_t turn = turns >> (8 * c);
                const bool flipped = turn & 1u;   // A_0 and the last dZ change places with every tile
                if (M::kWindows && (over >> l) & 1u) {
                    parity ^= 1u << l;
                    over ^= 1u << l;
                    if (M::kWide) summed ^= 1u << l;
                    if (!M::kWide || l == 0) started ^= 1u << l;
                }
                const uint32_t a = l == 0 ? cb + (flipped ? M::kDz : 0u) : cb + M::kRowsIn + (l - 1) * M::kRows;           // A_l
                const uint32_t z = l == NL - 1 ? cb + (flipped ? 0u : M::kDz) : cb + M::kRowsIn + l * M::kRows;   // dZ_l
                const uint32_t begun = (started >> l) & 1u;
                if constexpr (M::kWide) {
                    const uint32_t db = tmem_base + M::db_col(0) + 16u * l, window = (summed >> l) & 1u;
                    if (elect_one()) {
                        if (l == NL - 1) {
                            // A^T . dZ, and dZ^T . 1 of 64 rows (those past the outputs are never read)
#pragma unroll 2
                            for (int k = 0; k < kTile / 16; ++k)
                                umma_f16(tmem_base + M::dw_col(NL - 1), desc_mn<H>(lo, a, k, M::kPanel), desc_mn<M::kDzW>(lo, z, k), umma_idesc(F, 1, 1, 128, OW), k > 0 ? 1u : begun);
#pragma unroll 2
                            for (int k = 0; k < kTile / 16; ++k)
                                umma_f16(db, desc_mn<M::kDzW>(lo, z, k), desc_mn<M::kOnesW>(lo, M::kOnes, 0), umma_idesc(F, 1, 1, 64, 8), k > 0 ? 1u : window);
                        } else {
                            const uint32_t d = tmem_base + (l == 0 ? M::dw_col(0) : M::dw_col(1) + (l - 1) * 128u);
                            if (l == 0) {
#pragma unroll 2
                                for (int k = 0; k < kTile / 16; ++k)
                                    umma_f16(d, desc_mn<H>(lo, z, k, M::kPanel), desc_mn<IW>(lo, a, k), umma_idesc(F, 1, 1, 128, IW), k > 0 ? 1u : begun);
                            } else {
#pragma unroll 2
                                for (int k = 0; k < kTile / 16; ++k)
                                    umma_f16(d, desc_mn<H>(lo, z, k, M::kPanel), desc_mn<H>(lo, a, k, M::kPanel), umma_idesc(F, 1, 1, 128, 128), k > 0 ? 1u : begun);
                            }
#pragma unroll 2
                            for (int k = 0; k < kTile / 16; ++k)
                                umma_f16(db, desc_mn<H>(lo, z, k, M::kPanel), desc_mn<M::kOnesW>(lo, M::kOnes, 0), umma_idesc(F, 1, 1, 128, 16), k > 0 ? 1u : window);
                        }
                        umma_commit(&dw_done[G * c + g]);
                    }
                } else {
                    const uint32_t d = tmem_base + (l == 0 ? M::dw_col(0) : M::dw_col(1) + (l - 1) * (H + 16));
                    const bool ends = M::kWindows && ((filled >> (4 * l)) & (M::kWindow - 1u)) == M::kWindow - 1u;
                    auto gradient = [&](auto z_width, auto a_width, uint32_t ones) {
                        constexpr int ZW = decltype(z_width)::value, AW = decltype(a_width)::value;
#pragma unroll 2
                        for (int k = 0; k < kTile / 16; ++k)
                            umma_f16(d, desc_mn<ZW>(lo, z, k), desc_mn<AW>(lo, a, k, ones - a - (uint32_t)k * 16u * (uint32_t)layout::row_bytes(AW)),
                                     umma_idesc(F, 1, 1, 64, AW + 8), k > 0 ? 1u : begun);
                    };
                    using WideT = std::integral_constant<int, H>;
                    if (elect_one()) {
                        if (l == 0 && IW != H) gradient(WideT{}, std::integral_constant<int, IW>{}, M::kOnesIn);
                        else if (l == NL - 1 && M::kDzW != H) gradient(std::integral_constant<int, M::kDzW>{}, WideT{}, M::kOnes);
                        else gradient(WideT{}, WideT{}, M::kOnes);
                        umma_commit(&dw_done[G * c + g]);
                        if (ends) umma_commit(&ended[l]);
                    }
                    if (M::kWindows) filled = (filled + (1u << (4 * l))) & (0x11111u * (M::kWindow - 1u));
                    if (ends) over |= 1u << l;
                }
                __syncwarp();
                started |= 1u << l;
                if constexpr (M::kWide) {
                    summed |= 1u << l;
                    if (M::ends_window((int)l, c, turn)) over |= 1u << l;
                }
                layers += (l < G ? top - l : 0u - G) << (4 * c);
                if (l < G) turns = (turns + (1u << (8 * c))) & 0x0f0f0f0fu;
                phase ^= 1u << c;
                --total;
                idle = 0;
            } else if (++idle > kMaxPolls || ((idle & 255u) == 255u && __any_sync(0xffffffffu, *abort_flag != 0u))) {
                *abort_flag = 1u;
                atomicOr(p.status, kStatusGrad);
                ok = false;
            }
            c = c + 1 == NCH ? 0u : c + 1;
        }
        if (M::kWindows && lane == 0) atomicOr((uint32_t*)(smem + M::kOpen), (M::kWide ? summed : started) & ~over);
    }

    // ---- one add per parameter per CTA ----
    tc_fence_before();
    __syncthreads();   // every chain has seen its last gradient product completed (or the CTA is aborting)
    tc_fence_after();
    const bool good = !*abort_flag;
    if constexpr (M::kWindows) {   // the windows that are open, a chain's warps each
        if (good && warp < NW && (M::kWide || (warp & 3) < 2)) {
            const uint32_t open = *(const volatile uint32_t*)(smem + M::kOpen);
#pragma unroll 1
            for (int l = warp >> 2; l < NL; l += NCH)
                if ((open >> l) & 1u) take_window<M, H, NL, IW>(tmem_base + ((uint32_t)((warp & 3) * 32) << 16), sbase, l);
        }
        __syncthreads();
        tc_fence_after();
    }
    float* sums = (float*)smem;
    constexpr bool kStaged = H != 32;   // through shared memory, from tensor memory; width 32 has its sums there
#pragma unroll 1
    for (int l0 = 0; l0 < NL; l0 += M::kSumLayers) {
        if (l0 > 0) __syncthreads();
        if (kStaged && good && warp < NW) {
            // Row r of a 64-row accumulator sits on lane 32 (r / 16) + r % 16, of one of 128 rows on lane r.  The warps of a lane
            // quarter take the 16-column pieces in turn.
            const int quarter = warp & 3;
            const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int l = l0; l < l0 + M::kSumLayers; ++l) {
                if (M::kWide && l == 0 && !M::kSumsInTmem) break;
                const int w = M::kWide && l == NL - 1 ? OW : l == 0 ? IW : H;
                float* layer = sums + (l - l0) * H * (int)M::kSumRow;
#pragma unroll 1
                for (int piece = warp >> 2; piece < w / 16 + (M::kWide ? 0 : 1); piece += NCH) {
                    const bool bias = piece == w / 16;
                    uint32_t col;
                    if constexpr (M::kWide) col = (l == 0 ? M::sum_col() : l < NL - 1 ? M::dw_col(1) + (l - 1) * 128u : M::dw_col(NL - 1)) + piece * 16u;
                    else col = (l == 0 ? M::dw_col(0) : M::dw_col(1) + (l - 1) * (H + 16)) + piece * 16u;
                    uint32_t v[16];
                    tmem_ld_32x16(lanes + col, v);
                    wait_ld(v);
                    const int row = M::kWide ? quarter * 32 + lane : quarter * 16 + lane;
                    if (M::kWide || (lane < 16 && row < H)) {
                        // the last layer of width 128 lies in features by outputs
                        const bool across = M::kWide && l == NL - 1;
                        float* at = bias ? layer + row * (int)M::kSumRow + H : across ? layer + piece * 16 * (int)M::kSumRow + row : layer + row * (int)M::kSumRow + piece * 16;
                        const int step = across ? (int)M::kSumRow : 1;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (i == 0 || !bias) at[i * step] = __uint_as_float(v[i]);
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
        }
        if (kStaged) __syncthreads();
        if (!good) continue;
        // real parameters in the order they are stored, four to a reduction where rows are whole 16-byte pieces
        int i = threadIdx.x;
#pragma unroll 1
        for (int l = l0; l < l0 + M::kSumLayers; ++l) {
            const int in = cfg.dims[l], out = cfg.dims[l + 1];
            float* dW = (float*)s_net[l].weightsGrad;
            float* dB = (float*)s_net[l].biasesGrad;
            const bool swizzled = !kStaged || (M::kWide && l == 0 && !M::kSumsInTmem);   // rows of the windows' sums
            const float* s = swizzled ? (const float*)(smem + M::kSums) + (kStaged ? 0 : l * H * 32) : sums + (l - l0) * H * (int)M::kSumRow;
            const float* b = M::kWindows ? (const float*)(smem + M::kBiasSums) + l * H : s + H;
            const bool fours = (in & 3) == 0 && cfg.param_layout == MLP_PARAMS_ROW_MAJOR && ((uint64_t)dW & 15u) == 0;
            const int per_row = fours ? in >> 2 : in;
            for (; i < out * per_row; i += kThreads) {
                const int o = i / per_row, k = i - o * per_row;
                if (swizzled) {
                    const float* at = s + o * 32;
                    if (fours) atomicAdd((float4*)dW + i, *(const float4*)(at + 4 * (k ^ (o & 7))));
                    else atomicAdd(dW + weight_index(cfg.param_layout, in, out, o, k), at[(k ^ (4 * (o & 7)))]);
                    continue;
                }
                const float* at = s + o * (int)M::kSumRow;
                if (fours) atomicAdd((float4*)dW + i, make_float4(at[4 * k], at[4 * k + 1], at[4 * k + 2], at[4 * k + 3]));
                else atomicAdd(dW + weight_index(cfg.param_layout, in, out, o, k), at[k]);
            }
            i -= out * per_row;
            for (; i < out; i += kThreads) atomicAdd(dB + i, b[M::kWindows ? i : i * (int)M::kSumRow]);
            i -= out;
        }
    }
    if (good) {
        if (threadIdx.x == 0) {
            const float* part = (const float*)(smem + M::kLoss);
            float mx = part[0], sm = part[1];
#pragma unroll
            for (int w = 1; w < NW; ++w) { mx = fmaxf(mx, part[2 * w]); sm += part[2 * w + 1]; }
            atomicMax(p.loss_words, __float_as_uint(mx));
            atomicAdd((float*)(p.loss_words + 1), sm);
        }
    }
    tc_fence_after();
    if (warp == NW + NCH) tmem_dealloc(tmem_base, 512);
}

// Shared-memory map of the forward kernel.
template <int H, int IW, int OW, int NCH>
struct ForwardMap {
    static constexpr int kThreads = 32 * 5 * NCH;
    static constexpr int kMaxLayers = 5;
    static constexpr uint32_t kChainBytes = kTile * (IW > H ? IW : H) * 2;   // the current layer's input rows
    __host__ __device__ static constexpr uint32_t w_off(int l) { return l == 0 ? 0u : (uint32_t)H * IW * 2 + (uint32_t)(l - 1) * H * H * 2; }
    static constexpr uint32_t kChains = (w_off(kMaxLayers - 1) + (uint32_t)H * H * 2 + 1023) & ~1023u;
    static constexpr uint32_t kStageFloats = 32 * (OW + 1);                  // outputs of a warp's rows on their way out
    static constexpr uint32_t kStage = kChains + NCH * kChainBytes;
    static constexpr uint32_t kUnit = (kStage + 4 * NCH * kStageFloats * 4 + 255) & ~255u;
    static constexpr uint32_t kHiddenBias = kUnit + kUnitBytes;              // [4][H rows][16]
    static constexpr uint32_t kBias = kHiddenBias + (kMaxLayers - 1) * H * 32;   // the output layer's, fp32 [OW]
    static constexpr uint32_t kBars = kBias + OW * 4;                        // per chain: ready, acc_full
    static constexpr uint32_t kTmemPtr = kBars + 2 * NCH * 8;
    static constexpr uint32_t kAbort = kTmemPtr + 4;
    static constexpr uint32_t kNet = (kAbort + 4 + 15) & ~15u;
    static constexpr uint32_t kSmemBytes = kNet + kMaxLayers * 32 + 1024;
    static constexpr uint32_t kTmemCols = layout::pow2_at_least_32(NCH * H);
    static_assert(kSmemBytes <= 227 * 1024 && kTmemCols <= 512, "shared and tensor memory budget");
};

template <int H, int IW, int OW, int NCH, int FMT, int HACT>
__global__ void __launch_bounds__(32 * 5 * NCH, 1) forward_chain_kernel(const __grid_constant__ Params p)
{
    using M = ForwardMap<H, IW, OW, NCH>;
    using C = Cvt<FMT>;
    constexpr int kThreads = M::kThreads;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const MlpConfig& cfg = p.cfg;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int nl = cfg.n_layers, od = cfg.dims[nl];
    uint64_t* ready = (uint64_t*)(smem + M::kBars);
    uint64_t* acc_full = ready + NCH;
    volatile uint32_t* abort_flag = (volatile uint32_t*)(smem + M::kAbort);
    if (threadIdx.x == 0) {
        for (int c = 0; c < NCH; ++c) {
            mbar_init(&ready[c], 4);
            mbar_init(&acc_full[c], 1);
        }
        *abort_flag = 0u;
        fence_mbar_init();
    }
    grid_wait();
    if (warp == 4 * NCH) {
        tmem_alloc((uint32_t*)(smem + M::kTmemPtr), M::kTmemCols);
        tmem_relinquish();
        grid_release();
    }
    const MlpLayerPointers* s_net = (const MlpLayerPointers*)(smem + M::kNet);
    if (threadIdx.x < nl * 4) ((uint64_t*)(smem + M::kNet))[threadIdx.x] = ((const uint64_t*)p.net)[threadIdx.x];
    __syncthreads();
    stage_weights<IW>(smem, cfg, (const void*)s_net[0].weights, H, cfg.dims[0], cfg.dims[1], threadIdx.x, kThreads);
#pragma unroll 1
    for (int l = 1; l < nl; ++l)
        stage_weights<H>(smem + M::w_off(1) + (uint32_t)(l - 1) * (H * H * 2), cfg, (const void*)s_net[l].weights, l == nl - 1 ? OW : H, cfg.dims[l],
                         cfg.dims[l + 1], threadIdx.x, kThreads);
    first_column(smem + M::kUnit, 8, threadIdx.x, kThreads, [](int) { return C::kOnes; });
    first_column(smem + M::kHiddenBias, (nl - 1) * H, threadIdx.x, kThreads, [&](int row) -> uint32_t {
        const int l = row / H, f = row % H;
        return f < cfg.dims[l + 1] ? ((const uint16_t*)s_net[l].biases)[f] : 0u;
    });
    for (int i = threadIdx.x; i < OW; i += kThreads)
        ((float*)(smem + M::kBias))[i] = i < od ? load_as_f32(cfg.dtype, (const void*)s_net[nl - 1].biases, i) : 0.0f;
    cp_async_wait_all();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *(volatile uint32_t*)(smem + M::kTmemPtr);
    const uint32_t stride = gridDim.x * NCH;
    bool ok = true;
    if (warp < 4 * NCH) {
        const int ch = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t t_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ch * H);
        const uint32_t cb = sbase + M::kChains + (uint32_t)ch * M::kChainBytes;
        const uint32_t in_row = cb + row_at<IW>(r), own_row = cb + row_at<H>(r);
        const uint32_t s_bias = sbase + M::kBias;
        const float alpha = cfg.act_alpha;
        uint32_t full = 0;
        auto wait_full = [&]() {
            ok = ok && wait_for(&acc_full[ch], full & 1u, abort_flag, p.status, kStatusRow);
            ++full;
            tc_fence_after();
        };
        auto release = [&]() {
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[ch]);
        };
        RawRow raw;
        uint32_t tile = blockIdx.x + gridDim.x * (uint32_t)ch;
        uint64_t sample = (uint64_t)tile * kTile + (uint64_t)r;
        Rows in(p.inputs, stored_inputs(cfg), cfg.input_dtype, sample, stride * kTile), out(p.outputs, od, MLP_F32, sample, stride * kTile);
        // Rows of more than four outputs leave through shared memory, a warp's 32 rows as one run (row by row from the threads that
        // own them, 50 outputs of 2^20 samples took 353 us, 134 now).
        const bool staged = od > 4;
        const int od_odd = od | 1;
        float* stage = (float*)(smem + M::kStage) + warp * M::kStageFloats;
        const uint32_t od_inverse = ((1u << 20) + (uint32_t)od - 1u) / (uint32_t)od;   // (i * od_inverse) >> 20 is i / od for i < 32 od <= 2048
        fetch_row(raw, p, in.at, sample < p.count);
        for (; tile < p.n_tiles && ok; tile += stride) {
            const bool valid = sample < p.count;
            float* dst = (float*)out.at;
            write_row<FMT, IW>(in_row, p, raw, in.at, valid);
            release();
            sample += (uint64_t)stride * kTile;
            in.at += in.step;
            out.at += out.step;
            fetch_row(raw, p, in.at, sample < p.count);
            if (sample < p.count && !short_row(cfg)) prefetch_row(in.at);
#pragma unroll 1
            for (int l = 0; l < nl - 1; ++l) {
                wait_full();
                if (!ok) break;
                float least = 0.0f;
                uint32_t v[H / 32][32];
                tmem_ld_32x32(t_acc, v[0]);
                wait_ld(v[0]);
                if constexpr (H == 64) tmem_ld_32x32(t_acc + 32u, v[H / 32 - 1]);
                hidden_columns<FMT, HACT>(v[0], own_row, alpha, least);
                if constexpr (H == 64) {
                    wait_ld(v[H / 32 - 1]);
                    hidden_columns<FMT, HACT>(v[H / 32 - 1], own_row ^ 64u, alpha, least);
                }
                release();
            }
            wait_full();
            if (!ok) break;
#pragma unroll 1
            for (int f = 0; f < od; f += 4) {
                float o[4], d[4];
                output_columns<FMT>(o, t_acc, s_bias, f);
                activate_outputs(cfg.output_act, alpha, o, d);
                if (staged) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (f + i < od) stage[lane * od_odd + f + i] = o[i];
                } else if (valid) {
                    if (p.vec_out) {
                        *(float4*)dst = make_float4(o[0], o[1], o[2], o[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (i < od) dst[i] = o[i];
                    }
                }
            }
            if (staged) {
                __syncwarp();
                float* rows = dst - lane * od;
                const uint64_t first = (uint64_t)tile * kTile + (uint64_t)(quarter * 32);
                const uint32_t n = first >= p.count ? 0u : (p.count - first < 32u ? (uint32_t)(p.count - first) : 32u) * (uint32_t)od;
#pragma unroll 4
                for (uint32_t i = lane; i < n; i += 32) rows[i] = stage[i + ((i * od_inverse) >> 20) * (uint32_t)(od_odd - od)];
                __syncwarp();
            }
            tc_fence_before();
        }
    } else {
        const int ch = warp - 4 * NCH;
        const uint32_t lo = (sbase & 0x3FFFFu) >> 4;
        const uint32_t cb = M::kChains + (uint32_t)ch * M::kChainBytes, acc = tmem_base + (uint32_t)(ch * H);
        const int in_steps = (cfg.dims[0] + 15) / 16;
        constexpr uint32_t F = C::kUmmaFmt;
        uint32_t seen = 0;
        for (uint32_t tile = blockIdx.x + gridDim.x * (uint32_t)ch; tile < p.n_tiles && ok; tile += stride) {
#pragma unroll 1
            for (int l = 0; l < nl; ++l) {
                ok = ok && wait_for(&ready[ch], seen & 1u, abort_flag, p.status, kStatusIssue);
                ok = __all_sync(0xffffffffu, ok);
                ++seen;
                tc_fence_after();
                if (ok && elect_one()) {
                    if (l < nl - 1) umma_f16(acc, desc_unit(lo, M::kUnit), desc_k<16>(lo, M::kHiddenBias + (uint32_t)l * (H * 32), 0), umma_idesc(F, 0, 0, 128, H), 0u);
                    if (l == 0) {
#pragma unroll
                        for (int k = 0; k < IW / 16; ++k)
                            if (k < in_steps) umma_f16(acc, desc_k<IW>(lo, cb, k), desc_k<IW>(lo, 0u, k), umma_idesc(F, 0, 0, 128, H), 1u);
                    } else {
                        const uint32_t id = l == nl - 1 ? umma_idesc(F, 0, 0, 128, OW) : umma_idesc(F, 0, 0, 128, H);
                        const uint32_t w = (uint32_t)H * IW * 2 + (uint32_t)(l - 1) * (H * H * 2);
#pragma unroll
                        for (int k = 0; k < H / 16; ++k) umma_f16(acc, desc_k<H>(lo, cb, k), desc_k<H>(lo, w, k), id, l < nl - 1 || k > 0);
                    }
                    umma_commit(&acc_full[ch]);
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 4 * NCH) tmem_dealloc(tmem_base, M::kTmemCols);
}

}  // namespace chain

// ------------------------------------------------------------------------------------------------
// Host side.  Compiled once per MLPB200_CHAIN_PART: 0 the entry points, 1 .. 4 the training builds of 2 .. 5 layers, 5 the
// forward builds, 6 the training builds of widths up to 128.
// ------------------------------------------------------------------------------------------------
#ifndef MLPB200_CHAIN_PART
#error "compile with -DMLPB200_CHAIN_PART=0..6 (slang_b200/build.py does)"
#endif

template <int NL> cudaError_t launch_chain_train(cudaStream_t st, TcWorkspace* ws, narrow::Params& p);
cudaError_t launch_chain_forward(cudaStream_t st, TcWorkspace* ws, narrow::Params& p);

cudaError_t launch_chain_train_wide(cudaStream_t st, TcWorkspace* ws, narrow::Params& p);

#if (MLPB200_CHAIN_PART >= 1 && MLPB200_CHAIN_PART <= 4) || MLPB200_CHAIN_PART == 6
template <int H, int NL, int IW, int OW, int NCH, int FMT, int HACT>
static cudaError_t launch_train(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    using M = chain::TrainMap<H, NL, IW, OW, NCH>;
    auto kern = chain::learn_gradient_chain_kernel<H, NL, IW, OW, NCH, FMT, HACT>;
    static SmemLimit limit;
    const cudaError_t e = limit.raise((const void*)kern, ws->ordinal, M::kSmemBytes);
    if (e != cudaSuccess) return e;
    // A CTA per tile as far as the SMs go; beyond, as few CTAs as finish in the same number of tiles a chain: each brings a set of
    // gradients to add (20011 samples, 157 tiles, one CTA per SM against 79: 32-128-128-3 26.1 / 23.2 us a step, texture network 21.4 /
    // 20.6; 16384 samples, 128 tiles, packed 23.4 against 22.3 and 20.5 against 17.9).
    const uint32_t sms = (uint32_t)ws->sm_count, rounds = (p.n_tiles + sms * NCH - 1) / (sms * NCH);
    const uint32_t grid = p.n_tiles <= sms ? p.n_tiles : (p.n_tiles + rounds * NCH - 1) / (rounds * NCH);
    return launch_after(st, kern, grid, M::kThreads, M::kSmemBytes, p);
}

template <int H, int NL, int IW, int OW, int NCH>
static cudaError_t launch_shape(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    const bool relu = p.cfg.hidden_act == MLP_ACT_RELU;
    if (p.cfg.dtype == MLP_BF16) return relu ? launch_train<H, NL, IW, OW, NCH, MLP_BF16, MLP_ACT_RELU>(st, ws, p) : launch_train<H, NL, IW, OW, NCH, MLP_BF16, MLP_ACT_LEAKY_RELU>(st, ws, p);
    return relu ? launch_train<H, NL, IW, OW, NCH, MLP_F16, MLP_ACT_RELU>(st, ws, p) : launch_train<H, NL, IW, OW, NCH, MLP_F16, MLP_ACT_LEAKY_RELU>(st, ws, p);
}

#if MLPB200_CHAIN_PART <= 4
template <int NL>
cudaError_t launch_chain_train(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    bool fits32 = p.cfg.dims[NL] <= 16;
    for (int l = 0; l <= NL; ++l) fits32 = fits32 && p.cfg.dims[l] <= 32;
    if (fits32) return launch_shape<32, NL, 32, 16, 4>(st, ws, p);
    // as many chains as shared and tensor memory hold, up to three
    if (p.cfg.dims[0] <= 32 && p.cfg.dims[NL] <= 16) return launch_shape<64, NL, 32, 16, NL == 5 ? 2 : 3>(st, ws, p);
    if constexpr (NL <= 4) return launch_shape<64, NL, 64, 64, NL == 4 ? 2 : 3>(st, ws, p);
    return cudaErrorInvalidValue;
}
template cudaError_t launch_chain_train<1 + MLPB200_CHAIN_PART>(cudaStream_t, TcWorkspace*, narrow::Params&);
#else
// Two chains where shared memory (the tiles and all weights) and tensor memory hold them.
cudaError_t launch_chain_train_wide(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    const bool few_in = p.cfg.dims[0] <= 32, few_out = p.cfg.dims[p.cfg.n_layers] <= 16;
    switch (p.cfg.n_layers) {
    case 2:
        if (few_in && few_out) return launch_shape<128, 2, 32, 16, 2>(st, ws, p);
        return launch_shape<128, 2, 64, 64, 2>(st, ws, p);
    case 3:
        if (few_in && few_out) return launch_shape<128, 3, 32, 16, 2>(st, ws, p);
        return launch_shape<128, 3, 64, 64, 1>(st, ws, p);
    case 4:
        if (few_in && few_out) return launch_shape<128, 4, 32, 16, 1>(st, ws, p);
        break;
    }
    return cudaErrorInvalidValue;
}
#endif
#endif

#if MLPB200_CHAIN_PART == 5
template <int H, int IW, int OW, int NCH, int FMT, int HACT>
static cudaError_t launch_forward(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    using M = chain::ForwardMap<H, IW, OW, NCH>;
    auto kern = chain::forward_chain_kernel<H, IW, OW, NCH, FMT, HACT>;
    static SmemLimit limit;
    const cudaError_t e = limit.raise((const void*)kern, ws->ordinal, M::kSmemBytes);
    if (e != cudaSuccess) return e;
    const uint32_t grid = p.n_tiles < (uint32_t)ws->sm_count ? p.n_tiles : (uint32_t)ws->sm_count;
    return launch_after(st, kern, grid, M::kThreads, M::kSmemBytes, p);
}

template <int H, int IW, int OW, int NCH>
static cudaError_t launch_shape(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    const bool relu = p.cfg.hidden_act == MLP_ACT_RELU;
    if (p.cfg.dtype == MLP_BF16) return relu ? launch_forward<H, IW, OW, NCH, MLP_BF16, MLP_ACT_RELU>(st, ws, p) : launch_forward<H, IW, OW, NCH, MLP_BF16, MLP_ACT_LEAKY_RELU>(st, ws, p);
    return relu ? launch_forward<H, IW, OW, NCH, MLP_F16, MLP_ACT_RELU>(st, ws, p) : launch_forward<H, IW, OW, NCH, MLP_F16, MLP_ACT_LEAKY_RELU>(st, ws, p);
}

cudaError_t launch_chain_forward(cudaStream_t st, TcWorkspace* ws, narrow::Params& p)
{
    const int nl = p.cfg.n_layers;
    int widest = 0;
    for (int l = 0; l <= nl; ++l) widest = p.cfg.dims[l] > widest ? p.cfg.dims[l] : widest;
    const bool few = p.cfg.dims[nl] <= 16;
    if (widest <= 32) return few ? launch_shape<32, 32, 16, 6>(st, ws, p) : launch_shape<32, 32, 32, 6>(st, ws, p);
    if (p.cfg.dims[0] <= 32 && few) return launch_shape<64, 32, 16, 6>(st, ws, p);
    return launch_shape<64, 64, 64, 3>(st, ws, p);
}
#endif

#if MLPB200_CHAIN_PART == 0
// Rows of `width` values of `bytes` each from an address on whole pieces of `piece` bytes.
static int pieces(uint64_t address, int width, int bytes, int piece) { return address % (uint64_t)piece == 0 && (width * bytes) % piece == 0; }

static narrow::Params chain_params(TcWorkspace* ws, const MlpConfig& c, uint64_t network, uint64_t inputs, uint32_t count)
{
    narrow::Params p = {};
    p.cfg = c;
    p.net = (const MlpLayerPointers*)network;
    p.status = ws->status;
    p.inputs = (const void*)inputs;
    p.count = count;
    p.n_tiles = (uint32_t)(((uint64_t)count + chain::kTile - 1) / chain::kTile);
    p.vec_in = pieces(inputs, c.dims[0], c.input_dtype == MLP_F32 ? 4 : 2, 16);
    return p;
}

static bool chain_network(const MlpConfig& c)
{
    if (c.n_layers < 2 || c.n_layers > 5) return false;
    if ((c.dtype != MLP_BF16 && c.dtype != MLP_F16) || (c.operand_dtype && c.operand_dtype != c.dtype)) return false;
    const int act = narrow::built_activation(c);
    if (act != MLP_ACT_RELU && act != MLP_ACT_LEAKY_RELU) return false;
    for (int l = 0; l <= c.n_layers; ++l)
        if (c.dims[l] > 64) return false;
    return c.encoding != MLP_ENC_FREQ2D || c.dims[0] == 32;
}

// Batches from which the tiles are the better way, us against the kernels of tc_narrow.cu (which deal 16 samples at a time):
// learnGradient and adjustParameters of the texture network, 600 samples 22.5 / 20.5, 16384: 26.7 / 20.6, 2^20: 267 / 174; width
// 32, 16 samples 17.5 / 18.4, 600: 18.5 / 18.4, 2^20: 160 / 130; 16-32-3, 600: 12.9 / 12.6, 2^20: 113 / 54.
constexpr uint32_t kTrainFrom = 1024;
// forward, 20-48-48-3: 100 samples 6.5 / 9.3, 8192: 7.2 / 6.6, 2^20: 73.6 / 42.5; 4-32-32-32-32-4, 2000 samples 6.5 / 6.7, 16384: 9.3 /
// 6.8, 2^20: 45.6 / 41.6; 64-64-64-50, 2^20: 214 / 134.
constexpr uint32_t kForwardFrom = 4096;

static bool chain_train_network(const MlpConfig& c)
{
    if (!chain_network(c)) return false;
    if (c.n_layers < 5) return true;
    // five layers of width 64 with wide inputs or outputs leave room for one chain only
    return c.dims[0] <= 32 && c.dims[c.n_layers] <= 16;
}

// Rows that the chains read or write less well than the register kernels, which deal 16 or 32 samples to a warp and their columns to its lanes.
// Targets of no whole pieces of four: a thread reads its own row value by value.
static bool ragged_targets(const MlpConfig& c) { return c.dims[c.n_layers] > 40 && (c.dims[c.n_layers] & 3) != 0; }
// Odd input rows go to shared memory value by value (scatter_rows()).
static bool odd_inputs(const MlpConfig& c) { return c.encoding != MLP_ENC_FREQ2D && c.dims[0] > 32 && (c.dims[0] & 1) != 0; }
// Samples that a B200's 148 SMs have in flight at once, a tile in each of so many chains.  Just above it few SMs have a second round.
static constexpr uint32_t one_round(uint32_t chains) { return 148u * chains * (uint32_t)chain::kTile; }
static int widest_of(const MlpConfig& c)
{
    int w = 0;
    for (int l = 0; l <= c.n_layers; ++l) w = c.dims[l] > w ? c.dims[l] : w;
    return w;
}

// Networks of widths up to 128 (those that launch_learn_gradient_tc takes).
static bool chain_wide_network(const MlpConfig& c)
{
    if (c.n_layers < 2 || c.n_layers > 4 || (c.dtype != MLP_BF16 && c.dtype != MLP_F16) || (c.operand_dtype && c.operand_dtype != c.dtype)) return false;
    const int act = narrow::built_activation(c);
    if ((act != MLP_ACT_RELU && act != MLP_ACT_LEAKY_RELU) || c.encoding != MLP_ENC_NONE) return false;
    if (c.dims[0] > 64 || c.dims[c.n_layers] > 64) return false;
    for (int l = 1; l < c.n_layers; ++l)
        if (c.dims[l] > 128) return false;
    return c.n_layers < 4 || (c.dims[0] <= 32 && c.dims[c.n_layers] <= 16);
}
// Against the kernels of tc_kernels.cu, us a step.  Two chains: 32-128-128-3, 1024 samples 20.5 / 19.3, 2^20: 581 / 234; 16-128-3 14.3 /
// 12.0, 379 / 122; 64-128-64 16.4 / 19.9, 65536 samples 36.9 / 36.9, 2^20: 369 / 321.  One chain: 32-128-128-128-3 25.1 / 27.0, 65536
// samples 67.6 / 53.1, 2^20: 772 / 457; 56-103-103-3, 25505 samples (two tiles one after the other) 32.8 / 35.6, 65536: 53.0 / 47.2, 2^20: 597 /
// 336; 64-128-128-64 51 / 61, 567 / 606.  Leaky ReLU has no build of its own there below five layers: 64-96-96-40 33 / 25, 1433 / 578;
// 64-128-64, 1024 samples 19.3 / 19.9, 16384: 26.6 / 21.2.
bool chain_train_wide_suits(const MlpConfig& c, uint32_t count)
{
    if (!chain_wide_network(c)) return false;
    // Weight rows of hidden layers in no whole 16-byte pieces are staged value by value: 32-70-70-3, 4096 samples 18.7 / 20.7, 10000: 23.2 / 20.5; 8-109-109-15: 22.6 /
    // 25.9, 9000: 24.7 / 26.4, 20000: 32.9 / 29.7.  (Two layers, 16-100-3: 14.4 / 12.4 at 2048; leaky ReLU, 32-127-127-16: 35.0 / 27.7; but 24-99-99-62 34.9 / 42.4,
    // 20000: 64.6 / 59.2, whose targets are read so too.)
    bool pieces = c.param_layout == MLP_PARAMS_ROW_MAJOR;
    for (int l = 1; l < c.n_layers; ++l) pieces = pieces && (c.dims[l] & 7) == 0;
    // Rows that the other kernel would convert first (fp32) stay here: no launch in front, nothing allocated.
    if (count < 12288u && c.n_layers > 2 && !pieces && c.input_dtype == c.dtype && (c.hidden_act == MLP_ACT_RELU || ragged_targets(c))) return false;
    const bool few_out = c.dims[c.n_layers] <= 16, few = c.dims[0] <= 32 && few_out;
    if (c.hidden_act == MLP_ACT_LEAKY_RELU) return count >= (few || c.n_layers > 2 ? kTrainFrom : 4u * kTrainFrom);
    if (c.n_layers == 4 || (c.n_layers == 3 && !few)) return few_out && count >= 65536u;   // one chain
    return count >= (few ? kTrainFrom : 131072u);
}

bool chain_train_suits(const MlpConfig& c, uint32_t count)
{
    if (count < kTrainFrom || !chain_train_network(c)) return false;
    // us against tc_narrow.cu: 38-36-55, 4096 samples 18.5 / 22.3, 20000: 22.7 / 26.0, 50000: 31.2 / 26.5, 65536: 34.8 / 42.3, 600000: 175 / 266; 13-24-47: 18.5 /
    // 20.2, 20.7 / 23.3, 28.9 / 23.8, 31.3 / 37.2, 156 / 208; 50-44-44-44-61 (two chains): 28.3 / 30.9, 32.9 / 36.8, 48.2 / 60.6, 288 / 406.
    if (ragged_targets(c)) return count >= 32768u && count <= one_round(c.n_layers == 4 ? 2 : 3);
    // 37-54-6 of fp32 rows, 131072 samples 32.4 / 30.3, 600000: 90.8 / 107
    if (odd_inputs(c) && c.input_dtype == MLP_F32 && c.n_layers == 2) return count <= 262144u;
    return true;
}

bool chain_forward_suits(const MlpConfig& c, uint32_t count)
{
    if (count < kForwardFrom || !chain_network(c)) return false;
    const int nl = c.n_layers, in = c.dims[0], out = c.dims[nl], widest = widest_of(c);
    if (widest <= 32) {
        // Networks of a few products of 16 x 8 with fp32 rows, or with rows of nine to sixteen values in no whole pieces: 3-8-8-8-1, 131072 samples 8.1 / 9.3, 600000:
        // 19.3 / 22.0; 5-32-7: 7.5 / 8.3, 17.6 / 19.4; 10-8-8 of halves: 8.5 / 9.9, 22.9 / 24.2.  (2-16-16-2: 600000 within 3 %; 4-16-4 of halves: 8.4 / 6.8, 21.9 / 14.4.)
        int products = 0;
        for (int l = 0; l < nl; ++l) products += (c.dims[l] + 15) / 16 * ((c.dims[l + 1] + 7) / 8);
        const bool by_value = c.input_dtype == MLP_F32 ? in <= 8 : in > 8 && in < 16;
        if (by_value && c.encoding != MLP_ENC_FREQ2D && products <= (nl == 2 ? 6 : 4)) return false;
        // odd fp32 rows, which scatter_rows() takes value by value: 21-31-3, 65536 samples 6.5 / 7.6, 600000: 25.0 / 28.6; 21-28-28-28-28-3: 8.9 / 10.7, 32.8 / 38.8
        if (c.input_dtype == MLP_F32 && in > 16 && (in & 1) != 0) return false;
        return count >= 16384u || out <= 16;   // 10-32-32-20, 9000 samples 6.6 / 7.2, 50000: 9.5 / 8.1
    }
    if (in <= 32 && out <= 16) return true;    // six chains; three below
    // 37-54-6, 50000 samples 9.8 / 8.8, 65536: 9.8 / 12.5, 600000: 51.1 / 78.2; 53-41-41-41-41-54: 28.7 / 19.6, 30.6 / 31.2, 141 / 206
    if (odd_inputs(c)) return count <= one_round(3);
    // 64-64-64-64, 56832 samples 16.5 / 12.4, 65536: 16.8 / 18.0, 75000: 17.0 / 17.9, 80000: 21.6 / 18.7; 64-48-3: 8.7 / 7.6, 8.7 / 9.5, 8.8 / 9.2, 12.4 / 9.9.
    // (Narrower inputs or outputs of more layers, and outputs in no whole pieces, are faster here in between too.)  56-20-40, 131072: 22.7 / 23.5, 600000: 80.4 / 103.
    const bool whole = (out & 3) == 0 && out >= 40;
    if (whole && nl == 2 && c.dims[1] <= 32) return count <= one_round(3);
    if ((whole && nl > 2 && in > 32) || (out <= 4 && nl == 2)) return count <= one_round(3) || count > one_round(4);
    return true;
}

cudaError_t launch_learn_gradient_chain(cudaStream_t st, TcWorkspace* ws, const MlpConfig& c, const MlpLearnGradParamsEx& a,
                                        int* launches, std::string* err, float* input_grads)
{
    const bool wide = !chain_train_network(c);
    if (wide && !chain_wide_network(c)) { if (err) *err = "shape not built for tiles of samples"; return cudaErrorInvalidValue; }
    narrow::Params p = chain_params(ws, c, a.networkBuffer, a.inputs, a.count);
    p.loss_words = (uint32_t*)a.lossBuffer;
    p.targets = (const void*)a.targets;
    p.input_grads = input_grads;
    const int tgt = c.target_dtype == MLP_F32 ? 4 : 2;
    p.vec_tgt = pieces(a.targets, c.dims[c.n_layers], tgt, 4 * tgt);
    p.vec_dx = pieces((uint64_t)input_grads, c.dims[0], 4, 32);
    *launches += 1;
    if (wide) return launch_chain_train_wide(st, ws, p);
    switch (c.n_layers) {
    case 2: return launch_chain_train<2>(st, ws, p);
    case 3: return launch_chain_train<3>(st, ws, p);
    case 4: return launch_chain_train<4>(st, ws, p);
    case 5: return launch_chain_train<5>(st, ws, p);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_forward_chain(cudaStream_t st, TcWorkspace* ws, const MlpConfig& c, const MlpForwardParams& a,
                                 int* launches, std::string* err)
{
    if (!chain_network(c)) { if (err) *err = "shape not built for tiles of samples"; return cudaErrorInvalidValue; }
    narrow::Params p = chain_params(ws, c, a.networkBuffer, a.inputs, a.count);
    p.outputs = (float*)a.outputs;
    p.vec_out = pieces(a.outputs, c.dims[c.n_layers], 4, 16);
    *launches += 1;
    return launch_chain_forward(st, ws, p);
}
#endif

}  // namespace mlpb200
