// General kernels without tensor cores: the literal example entry points and the shape-generic path.
//
// The callers keep the reference's dispatch contract: [numthreads(256,1,1)], grid = ceil(count / 256)
// (examples/mlp-training/kernels.slang:8-41, examples/mlp-training/mlp-training.cpp:181-204).  The example kernels
// and the forward pass run a thread per sample, learnGradient a CTA per tiles of 32 samples.
// They serve every shape and number format; the tensor-core kernels take over for the shapes they
// are built for.  This file is compiled with -fmad=false: every multiply and add is separately
// rounded unless fmaf is written out, so fp32 results match a sequential CPU bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <string>

#include "mlp_common.cuh"
#include "launch_pdl.cuh"
#include "launchers.h"

#include "example_kernels.cuh"

namespace mlpb200 {

// ------------------------------------------------------------------------------------------------
// Shape-generic path: any MlpConfig whose layer widths sum to at most kMaxActFloats.
// ------------------------------------------------------------------------------------------------
constexpr int kMaxActFloats = 768;  // sum of all layer widths (a forward thread's arrays, a tile's shared memory)

struct SimtNet {
    MlpConfig cfg;
    int a_off[MLP_MAX_LAYERS + 2];  // offset of the vector entering layer l in the per-thread arrays
};

// The type products read their operands in: the storage type, or MlpConfig.operand_dtype (fp32 storage whose
// weights and inter-layer vectors are converted to a 16-bit type where a product reads them).
__device__ __forceinline__ int operand_type(const MlpConfig& c) { return c.operand_dtype ? c.operand_dtype : c.dtype; }
__device__ __forceinline__ float load_weight(const MlpConfig& c, const void* W, int64_t idx)
{
    const float w = load_as_f32(c.dtype, W, idx);
    return c.operand_dtype ? round_to(c.operand_dtype, w) : w;
}

__device__ __forceinline__ void encode_input(const MlpConfig& c, const void* inputs, int64_t s, float* a0)
{
    const int opd = operand_type(c);
    if (c.encoding == MLP_ENC_FREQ2D) {
        for (int u = 0; u < 2; ++u) {
            const float v = load_as_f32(c.input_dtype, inputs, s * 2 + u);
            for (int k = 0; k < 8; ++k) {
                const float arg = ldexpf(3.14159265358979323846f, k) * v;
                a0[u * 16 + k * 2 + 0] = round_to(opd, sinf(arg));
                a0[u * 16 + k * 2 + 1] = round_to(opd, cosf(arg));
            }
        }
    } else {
        for (int i = 0; i < c.dims[0]; ++i)
            a0[i] = round_to(opd, load_as_f32(c.input_dtype, inputs, s * c.dims[0] + i));
    }
}

// Activations with one copy of the switch behind a call: inlined at every use it made the tile kernel 11.9 k instructions long, most
// of whose time at small batches went into fetching them.
static __device__ __noinline__ float other_act_value(int act, float alpha, float x) { return act_value(act, alpha, x); }
static __device__ __noinline__ float other_act_deriv(int act, float alpha, float x) { return act_deriv(act, alpha, x); }
__device__ __forceinline__ float tile_act_value(int act, float alpha, float x)
{
    if (act == MLP_ACT_RELU) return act_value(MLP_ACT_RELU, alpha, x);
    if (act == MLP_ACT_IDENTITY) return x;
    return other_act_value(act, alpha, x);
}
__device__ __forceinline__ float tile_act_deriv(int act, float alpha, float x)
{
    if (act == MLP_ACT_RELU) return act_deriv(MLP_ACT_RELU, alpha, x);
    if (act == MLP_ACT_IDENTITY) return 1.0f;
    return other_act_deriv(act, alpha, x);
}

// One term of a scalar sum in the order MlpConfig.sum_order names: a fused multiply-add, or a rounded
// product followed by a rounded add (this file is compiled with -fmad=false, so `acc + a * b` is two
// roundings).
__device__ __forceinline__ float mac(float a, float b, float acc, bool fused)
{
    return fused ? fmaf(a, b, acc) : acc + __fmul_rn(a, b);
}

// Forward of one sample; a holds every layer's input vector, z every pre-activation (both rounded to
// the storage type); the last slot of a holds the fp32 outputs.
__device__ void simt_forward(const SimtNet& net, const MlpLayerPointers* __restrict__ lp, const void* inputs, int64_t s,
                             float* a, float* z)
{
    const MlpConfig& c = net.cfg;
    const bool fused = c.sum_order == MLP_SUM_BIAS_FIRST_FUSED;
    encode_input(c, inputs, s, a);
    for (int l = 0; l < c.n_layers; ++l) {
        const int in = c.dims[l], out = c.dims[l + 1];
        const bool last = (l == c.n_layers - 1);
        const float* ain = a + net.a_off[l];
        float* aout = a + net.a_off[l + 1];
        float* zl = z + net.a_off[l + 1] - net.a_off[1];
        const void* W = (const void*)lp[l].weights;
        const void* B = (const void*)lp[l].biases;
        for (int j = 0; j < out; ++j) {
            const float bias = load_as_f32(c.dtype, B, j);
            float r;
            if (fused) {
                r = bias;
                for (int i = 0; i < in; ++i) r = fmaf(load_weight(c, W, weight_index(c.param_layout, in, out, j, i)), ain[i], r);
            } else {
                r = 0.0f;
                for (int i = 0; i < in; ++i) r = mac(load_weight(c, W, weight_index(c.param_layout, in, out, j, i)), ain[i], r, false);
                r = r + bias;
            }
            const float zs = round_to(c.dtype, r);
            zl[j] = zs;
            aout[j] = last ? act_value(c.output_act, c.act_alpha, zs)
                           : round_to(operand_type(c), act_value(c.hidden_act, c.act_alpha, zs));
        }
    }
}

__global__ void __launch_bounds__(256)
forward_simt_kernel(SimtNet net, const MlpLayerPointers* __restrict__ lp, const void* __restrict__ inputs,
                    float* __restrict__ outputs, uint32_t count)
{
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= count) return;
    float a[kMaxActFloats], z[kMaxActFloats];
    simt_forward(net, lp, inputs, tid, a, z);
    const int od = net.cfg.dims[net.cfg.n_layers];
    const float* o = a + net.a_off[net.cfg.n_layers];
    for (int j = 0; j < od; ++j) outputs[int64_t(tid) * od + j] = o[j];
}

// learnGradient, generic.  A CTA walks tiles of 32 samples with the LANES on the samples and the warps on the
// output features: every vector of a tile (layer inputs, pre-activations, output gradients) is a shared-memory row
// of 32 floats per feature, a weight is one broadcast read shared by the 32 samples, and each sum runs over its
// terms in ascending order exactly as simt_forward does.  Parameters are summed over the tile in ascending sample
// order, over the CTA's tiles in shared memory where it has room, and leave through one atomic add per parameter
// per CTA; where it has none (fp32 64-128-128-128-128-64), per tile, with weights it has no room for read from global
// memory (65536 samples of that network: 12.2 ms; a thread per sample with its vectors in local memory: 29.2).  With MLP_FLAG_SEQUENTIAL_SUM the per-sample vectors go to a global scratch area instead and a second
// kernel adds them one sample at a time.
//
// Bound: the latency of the layer chain at small batches (a tile is 2 NL + 2 barriers), fp32 issue at large ones.
// One thread per sample with its vectors in local memory, which this replaces, put 4096 samples on 16 of the 148
// SMs and walked every sum behind local-memory loads.
constexpr int kTile = 32;                   // samples per tile, one per lane
constexpr int kRow = kTile + 4;             // floats per feature row: 16-byte reads of eight consecutive rows hit distinct banks
constexpr int kSimtThreads = 512;
constexpr int kSimtWarps = kSimtThreads / 32;
constexpr size_t kSimtSmemMax = 226 * 1024;   // (beside the layer addresses)

// Shared-memory map of a network, in floats: feature rows of a_0 .. a_{nl-1} and the outputs (a_off[l] * kRow), then
// of z_1 .. z_nl, then biases, and where there is room the weights (rows padded to multiples of four) and the
// gradient sums of the CTA's tiles.
struct SimtSmem {
    int z, bias, total;
    int w;                                  // -1: weights are read from global memory
    int grads;                              // -1: sums leave after every tile
    int w_off[MLP_MAX_LAYERS], b_off[MLP_MAX_LAYERS], g_off[MLP_MAX_LAYERS];   // inside their regions
};

// Four consecutive weights of output j, from shared memory (staged) or from the parameters.
template <bool STAGED>
struct WeightRows {
    const MlpConfig& c;
    const void* W;
    const float* s_w;
    int in, out, stride;
    __device__ __forceinline__ float one(int j, int i) const
    {
        return STAGED ? s_w[j * stride + i] : load_weight(c, W, weight_index(c.param_layout, in, out, j, i));
    }
    __device__ __forceinline__ float4 four(int j, int i) const
    {
        if constexpr (STAGED) return *reinterpret_cast<const float4*>(s_w + j * stride + i);
        return make_float4(one(j, i), i + 1 < in ? one(j, i + 1) : 0.0f, i + 2 < in ? one(j, i + 2) : 0.0f, i + 3 < in ? one(j, i + 3) : 0.0f);
    }
};

// z and a of J outputs from j0 on for this lane's sample.
template <int J, bool STAGED>
__device__ __forceinline__ void tile_layer_forward(const MlpConfig& c, const WeightRows<STAGED>& w, const float* s_bias, const float* ain,
                                                   float* z, float* aout, int j0, int act, bool round_act, bool fused)
{
    float r[J];
    int jr[J];
#pragma unroll
    for (int u = 0; u < J; ++u) {
        jr[u] = min(j0 + u, w.out - 1);
        r[u] = fused ? s_bias[jr[u]] : 0.0f;
    }
    int i = 0;
    for (; i + 4 <= w.in; i += 4) {
        const float a0 = ain[i * kRow], a1 = ain[(i + 1) * kRow], a2 = ain[(i + 2) * kRow], a3 = ain[(i + 3) * kRow];
#pragma unroll
        for (int u = 0; u < J; ++u) {
            const float4 v = w.four(jr[u], i);
            r[u] = mac(v.w, a3, mac(v.z, a2, mac(v.y, a1, mac(v.x, a0, r[u], fused), fused), fused), fused);
        }
    }
    for (; i < w.in; ++i) {
        const float a0 = ain[i * kRow];
#pragma unroll
        for (int u = 0; u < J; ++u) r[u] = mac(w.one(jr[u], i), a0, r[u], fused);
    }
#pragma unroll
    for (int u = 0; u < J; ++u) {
        if (j0 + u >= w.out) break;
        const float zs = round_to(c.dtype, fused ? r[u] : r[u] + s_bias[j0 + u]);
        const float v = tile_act_value(act, c.act_alpha, zs);
        z[(j0 + u) * kRow] = zs;
        aout[(j0 + u) * kRow] = round_act ? round_to(operand_type(c), v) : v;
    }
}

// r[u] = sum over j of W[j][i0 + u] dz[j], four inputs at a time (i0 a multiple of four).
template <bool STAGED>
__device__ __forceinline__ void tile_layer_backward(const WeightRows<STAGED>& w, const float* dz, int i0, float (&r)[4], bool fused)
{
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = 0.0f;
    for (int j = 0; j < w.out; ++j) {
        const float d = dz[j * kRow];
        const float4 v = w.four(j, i0);
        r[0] = mac(v.x, d, r[0], fused);
        r[1] = mac(v.y, d, r[1], fused);
        r[2] = mac(v.z, d, r[2], fused);
        r[3] = mac(v.w, d, r[3], fused);
    }
}

template <bool STAGED>
__global__ void __launch_bounds__(kSimtThreads)
learn_gradient_simt_kernel(const __grid_constant__ SimtNet net, const __grid_constant__ SimtSmem map, const MlpLayerPointers* __restrict__ lp,
                           uint32_t* lossBuffer, const void* __restrict__ inputs, const void* __restrict__ targets, uint32_t count,
                           uint32_t n_tiles, float* __restrict__ seq_scratch, float* __restrict__ input_grads)
{
    extern __shared__ __align__(16) float smem[];
    const MlpConfig& c = net.cfg;
    const int nl = c.n_layers;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int od = c.dims[nl];
    const bool fused = c.sum_order == MLP_SUM_BIAS_FIRST_FUSED;
    const int opd = operand_type(c);
    grid_release();
    grid_wait();
    const bool once = gridDim.x == n_tiles;       // one tile per CTA: its sums leave directly
    float* const s_z = smem + map.z;              // z rows, later dz: layer l's outputs from row a_off[l + 1] - a_off[1]
    auto z_rows = [&](int l) { return s_z + (net.a_off[l] - net.a_off[1]) * kRow; };   // of the vector leaving layer l - 1

    // Addresses first, then every layer's parameters without waiting in between.
    __shared__ MlpLayerPointers s_net[MLP_MAX_LAYERS];
    if (threadIdx.x < nl * 4) reinterpret_cast<uint64_t*>(s_net)[threadIdx.x] = reinterpret_cast<const uint64_t*>(lp)[threadIdx.x];
    __syncthreads();
    {
        int i = threadIdx.x;
        for (int l = 0; l < nl; ++l) {
            const int out = c.dims[l + 1];
            for (; i < out; i += kSimtThreads) smem[map.bias + map.b_off[l] + i] = load_as_f32(c.dtype, (const void*)s_net[l].biases, i);
            i -= out;
        }
        if constexpr (STAGED) {
            for (int l = 0; l < nl; ++l) {
                const int in = c.dims[l], out = c.dims[l + 1], stride = (in + 3) & ~3;
#pragma unroll 4
                for (; i < out * stride; i += kSimtThreads) {
                    const int j = i / stride, k = i - j * stride;
                    smem[map.w + map.w_off[l] + i] =
                        k < in ? load_weight(c, (const void*)s_net[l].weights, weight_index(c.param_layout, in, out, j, k)) : 0.0f;
                }
                i -= out * stride;
            }
        }
    }
    auto weights = [&](int l) {
        return WeightRows<STAGED>{c, STAGED ? nullptr : (const void*)s_net[l].weights, STAGED ? smem + map.w + map.w_off[l] : nullptr,
                                  c.dims[l], c.dims[l + 1], (c.dims[l] + 3) & ~3};
    };

    float run_max = 0.0f, run_sum = 0.0f;         // warp 0: this lane's samples
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t s0 = tile * kTile;
        const int n_here = (int)min((uint32_t)kTile, count - s0);
        const bool valid = lane < n_here;
        // ---- inputs; rows past the batch are zero ----
        for (int idx = threadIdx.x; idx < kTile * c.dims[0]; idx += kSimtThreads) {
            const int s = idx / c.dims[0], i = idx - s * c.dims[0];
            float v = 0.0f;
            if (s < n_here) {
                if (c.encoding == MLP_ENC_FREQ2D) {
                    const float x = load_as_f32(c.input_dtype, inputs, int64_t(s0 + s) * 2 + (i >> 4));
                    const float arg = ldexpf(3.14159265358979323846f, (i & 15) >> 1) * x;
                    v = (i & 1) ? cosf(arg) : sinf(arg);
                } else {
                    v = load_as_f32(c.input_dtype, inputs, int64_t(s0) * c.dims[0] + idx);
                }
                v = round_to(opd, v);
            }
            smem[i * kRow + s] = v;
        }
        // up to sixteen targets of a sample, a warp each, are fetched a forward pass ahead of their use
        float target = 0.0f;
        if (warp < od && valid) target = load_as_f32(c.target_dtype, targets, int64_t(s0 + lane) * od + warp);
        __syncthreads();
        // ---- forward ----
        for (int l = 0; l < nl; ++l) {
            const WeightRows<STAGED> w = weights(l);
            const bool last = l == nl - 1;
            const float* ain = smem + net.a_off[l] * kRow + lane;
            float* aout = smem + net.a_off[l + 1] * kRow + lane;
            float* z = z_rows(l + 1) + lane;
            const float* s_bias = smem + map.bias + map.b_off[l];
            const int act = last ? c.output_act : c.hidden_act;
            if (w.out <= kSimtWarps) {
                if (warp < w.out) tile_layer_forward<1, STAGED>(c, w, s_bias, ain, z, aout, warp, act, !last, fused);
            } else if (w.out <= 2 * kSimtWarps) {
                if (2 * warp < w.out) tile_layer_forward<2, STAGED>(c, w, s_bias, ain, z, aout, 2 * warp, act, !last, fused);
            } else {
                for (int j0 = 4 * warp; j0 < w.out; j0 += 4 * kSimtWarps)
                    tile_layer_forward<4, STAGED>(c, w, s_bias, ain, z, aout, j0, act, !last, fused);
            }
            __syncthreads();
        }
        // ---- loss (warp 0, a sample per lane, outputs in ascending order) and dz of the last layer (every warp) ----
        {
            const float scale = (c.loss == MLP_LOSS_MSE_MEAN) ? 1.0f / float(od) : 1.0f;
            const float* o = smem + net.a_off[nl] * kRow + lane;
            float* dz = z_rows(nl) + lane;
            for (int j = warp; j < od; j += kSimtWarps) {
                float g = 0.0f;
                if (valid) {
                    const float diff = o[j * kRow] - (j == warp ? target : load_as_f32(c.target_dtype, targets, int64_t(s0 + lane) * od + j));
                    g = round_to(opd, ((2.0f * scale) * diff) * tile_act_deriv(c.output_act, c.act_alpha, dz[j * kRow]));
                }
                dz[j * kRow] = g;
            }
            if (warp == 0 && valid) {
                float loss = 0.0f;
                for (int j = 0; j < od; ++j) {
                    const float diff = o[j * kRow] - (j == 0 ? target : load_as_f32(c.target_dtype, targets, int64_t(s0 + lane) * od + j));
                    loss = fmaf(diff * scale, diff, loss);
                }
                run_max = fmaxf(run_max, loss);
                run_sum += loss;
            }
        }
        __syncthreads();
        // ---- backward: dz of the layer before replaces its z; rows past the batch stay zero because dz is zero ----
        for (int l = nl - 1; l >= 1; --l) {
            const WeightRows<STAGED> w = weights(l);
            const float* dz = z_rows(l + 1) + lane;
            float* zprev = z_rows(l) + lane;
            for (int i0 = 4 * warp; i0 < w.in; i0 += 4 * kSimtWarps) {
                float r[4];
                tile_layer_backward<STAGED>(w, dz, i0, r, fused);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (i0 + u >= w.in) break;
                    const float d = round_to(opd, tile_act_deriv(c.hidden_act, c.act_alpha, zprev[(i0 + u) * kRow]));
                    zprev[(i0 + u) * kRow] = valid ? round_to(opd, r[u] * d) : 0.0f;
                }
            }
            __syncthreads();
        }
        if (input_grads) {
            // dx = W_0^T dz_0: dead in the example (its inputs are no_diff), wanted by an encoder in front
            const WeightRows<STAGED> w = weights(0);
            for (int i0 = 4 * warp; i0 < w.in; i0 += 4 * kSimtWarps) {
                float r[4];
                tile_layer_backward<STAGED>(w, z_rows(1) + lane, i0, r, fused);
                for (int u = 0; u < 4 && i0 + u < w.in; ++u)
                    if (valid) input_grads[int64_t(s0 + lane) * w.in + i0 + u] = round_to(c.dtype, r[u]);
            }
        }
        if (seq_scratch) {
            // Per sample: [a of all layers (a_off[nl] floats)][dz of all layers (a_off[nl + 1] - a_off[1] floats)].
            const int na = net.a_off[nl], n = na + net.a_off[nl + 1] - net.a_off[1];
            for (int idx = threadIdx.x; idx < n_here * n; idx += kSimtThreads) {
                const int s = idx / n, k = idx - s * n;
                seq_scratch[int64_t(s0 + s) * n + k] = k < na ? smem[k * kRow + s] : s_z[(k - na) * kRow + s];
            }
            __syncthreads();
            continue;
        }
        // ---- parameter sums of the tile: a thread takes one output and up to four inputs (the bias rides as one more) ----
        for (int l = 0; l < nl; ++l) {
            const int in = c.dims[l], out = c.dims[l + 1];
            const float* al = smem + net.a_off[l] * kRow;
            const float* dz = z_rows(l + 1);
            const int blocks = in / 4 + (in & 3) + 1;   // fours, then the remaining inputs one by one, then the bias
            for (int item = threadIdx.x; item < out * blocks; item += kSimtThreads) {
                const int j = item / blocks, b = item - j * blocks;
                const float* dzj = dz + j * kRow;
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                int i0, n;
                if (b == blocks - 1) {
                    i0 = in; n = 1;
                    for (int s = 0; s < n_here; ++s) acc[0] += dzj[s];
                } else if (b < in / 4) {
                    i0 = b * 4; n = 4;
                    // rows past the batch: dz is zero there, a_l need not be finite
                    if (n_here < kTile) {
                        for (int s = 0; s < n_here; ++s)
                            for (int u = 0; u < 4; ++u) acc[u] = mac(dzj[s], al[(i0 + u) * kRow + s], acc[u], fused);
                    } else
#pragma unroll
                    for (int s = 0; s < kTile; s += 4) {
                        const float4 d = *reinterpret_cast<const float4*>(dzj + s);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float4 v = *reinterpret_cast<const float4*>(al + (i0 + u) * kRow + s);
                            acc[u] = mac(d.w, v.w, mac(d.z, v.z, mac(d.y, v.y, mac(d.x, v.x, acc[u], fused), fused), fused), fused);
                        }
                    }
                } else {
                    i0 = in / 4 * 4 + (b - in / 4); n = 1;
                    for (int s = 0; s < n_here; ++s) acc[0] = mac(dzj[s], al[i0 * kRow + s], acc[0], fused);
                }
                if (!once && map.grads >= 0) {
                    float* g = smem + map.grads + map.g_off[l] + j * (in + 1) + i0;
                    for (int u = 0; u < n; ++u) g[u] = tile == blockIdx.x ? acc[u] : g[u] + acc[u];
                } else if (i0 == in) {
                    atomicAdd((float*)s_net[l].biasesGrad + j, acc[0]);
                } else {
                    for (int u = 0; u < n; ++u) atomicAdd((float*)s_net[l].weightsGrad + weight_index(c.param_layout, in, out, j, i0 + u), acc[u]);
                }
            }
        }
        __syncthreads();   // the next tile overwrites the rows
    }
    if (!seq_scratch && !once && map.grads >= 0) {
        for (int l = 0; l < nl; ++l) {
            const int in = c.dims[l], out = c.dims[l + 1];
            float* dW = (float*)s_net[l].weightsGrad;
            float* dB = (float*)s_net[l].biasesGrad;
            for (int item = threadIdx.x; item < out * (in + 1); item += kSimtThreads) {
                const int j = item / (in + 1), i = item - j * (in + 1);
                const float g = smem[map.grads + map.g_off[l] + item];
                if (i == in) atomicAdd(dB + j, g);
                else atomicAdd(dW + weight_index(c.param_layout, in, out, j, i), g);
            }
        }
    }
    // Loss words: the largest per-sample loss, and the sum added once per CTA.
    if (warp == 0) {
        for (int o = 16; o > 0; o >>= 1) {
            run_max = fmaxf(run_max, __shfl_xor_sync(0xffffffffu, run_max, o));
            run_sum += __shfl_xor_sync(0xffffffffu, run_sum, o);
        }
        if (lane == 0) {
            atomicMax(lossBuffer, __float_as_uint(run_max));
            atomicAdd((float*)(lossBuffer + 1), run_sum);
        }
    }
}

// learnGradient of small plain fp32 networks: ReLU, linear outputs, fp32 rows, widths up to 32.  The same tiles, rows and sums
// as the general kernel's, a layer's outputs two to a warp, without its choices: some 850 instructions instead of twelve thousand.  A
// step of 4096 samples runs every instruction once or twice, so fetching them was what it waited for (2-16-16-16-1: 14.3 us a
// step, 22.5 with the general kernel; 2^20 samples 684 and 1306).
constexpr int kSmallWidth = 32;

struct SmallNet {
    int nl, od;
    int dims[MLP_MAX_LAYERS + 1];
    int a_row[MLP_MAX_LAYERS + 1];          // first row of the vector entering layer l (the last: the outputs)
    int z_row[MLP_MAX_LAYERS + 1];          // first row of z_l, later dz_l (l from 1)
    int w_at[MLP_MAX_LAYERS], b_at[MLP_MAX_LAYERS], g_at[MLP_MAX_LAYERS];   // floats: weights (rows of a multiple of four), biases, gradient sums
    uint32_t per_row[MLP_MAX_LAYERS];       // 65536 / (in + 1), rounded up: (i * per_row) >> 16 is i / (in + 1) below 33 * 32
    uint32_t per_input;                     // the same of the input width
    float scale;
};

__device__ __forceinline__ void copy_float(float* dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <bool FUSED>
__global__ void __launch_bounds__(kSimtThreads)
learn_gradient_small_kernel(const __grid_constant__ SmallNet net, const MlpLayerPointers* __restrict__ lp, uint32_t* lossBuffer,
                            const float* __restrict__ inputs, const float* __restrict__ targets, uint32_t count, uint32_t n_tiles)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ MlpLayerPointers s_net[MLP_MAX_LAYERS];
    const int nl = net.nl, od = net.od, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    grid_release();
    grid_wait();
    if (tid < nl * 4) reinterpret_cast<uint64_t*>(s_net)[tid] = reinterpret_cast<const uint64_t*>(lp)[tid];
    const bool once = gridDim.x == n_tiles;
    float run_max = 0.0f, run_sum = 0.0f;
    bool staged = false;
#pragma unroll 1
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t s0 = tile * kTile;
        const uint32_t n_here = min((uint32_t)kTile, count - s0);
        const bool valid = lane < n_here;
        {
            const int in = net.dims[0];
            const float* x = inputs + uint64_t(s0) * in;
#pragma unroll 1
            for (int i = tid; i < kTile * in; i += kSimtThreads) {
                const int s = (int)(((uint32_t)i * net.per_input) >> 16);
                float* dst = smem + (i - s * in) * kRow + s;
                if (s < n_here) copy_float(dst, x + i);
                else *dst = 0.0f;
            }
        }
        float target = 0.0f;
        if (warp < od && valid) target = __ldg(targets + uint64_t(s0 + lane) * od + warp);
        if (!staged) {
            staged = true;
            __syncthreads();
#pragma unroll 1
            for (int l = 0; l < nl; ++l) {
                const int in = net.dims[l], out = net.dims[l + 1], stride = (in + 3) & ~3;
                const float* w = (const float*)s_net[l].weights;
#pragma unroll 1
                for (int j = warp; j < out; j += kSimtWarps) {
                    if (lane < in) copy_float(smem + net.w_at[l] + j * stride + lane, w + j * in + lane);
                    else if (lane < stride) smem[net.w_at[l] + j * stride + lane] = 0.0f;
                }
                if (tid < out) copy_float(smem + net.b_at[l] + tid, (const float*)s_net[l].biases + tid);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // ---- forward ----
#pragma unroll 1
        for (int l = 0; l < nl; ++l) {
            const int in = net.dims[l], out = net.dims[l + 1], stride = (in + 3) & ~3;
            if (2 * warp < out) {
                const int j0 = 2 * warp, j1 = min(j0 + 1, out - 1);
                const float* a = smem + net.a_row[l] * kRow + lane;
                const float* w0 = smem + net.w_at[l] + j0 * stride;
                const float* w1 = smem + net.w_at[l] + j1 * stride;
                const float b0 = smem[net.b_at[l] + j0], b1 = smem[net.b_at[l] + j1];
                float r0 = FUSED ? b0 : 0.0f, r1 = FUSED ? b1 : 0.0f;
                int i = 0;
#pragma unroll 1
                for (; i + 4 <= in; i += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(w0 + i), v = *reinterpret_cast<const float4*>(w1 + i);
                    const float a0 = a[i * kRow], a1 = a[(i + 1) * kRow], a2 = a[(i + 2) * kRow], a3 = a[(i + 3) * kRow];
                    r0 = mac(u.w, a3, mac(u.z, a2, mac(u.y, a1, mac(u.x, a0, r0, FUSED), FUSED), FUSED), FUSED);
                    r1 = mac(v.w, a3, mac(v.z, a2, mac(v.y, a1, mac(v.x, a0, r1, FUSED), FUSED), FUSED), FUSED);
                }
#pragma unroll 1
                for (; i < in; ++i) {
                    r0 = mac(w0[i], a[i * kRow], r0, FUSED);
                    r1 = mac(w1[i], a[i * kRow], r1, FUSED);
                }
                if (!FUSED) { r0 += b0; r1 += b1; }
                const bool hidden = l < nl - 1;
                float* z = smem + net.z_row[l + 1] * kRow + lane;
                float* o = smem + net.a_row[l + 1] * kRow + lane;
                // rows past the batch are zero throughout, whatever the biases are
                const float v0 = hidden && !(r0 > 0.0f) ? 0.0f : r0, v1 = hidden && !(r1 > 0.0f) ? 0.0f : r1;
                z[j0 * kRow] = r0;
                o[j0 * kRow] = valid ? v0 : 0.0f;
                if (j1 != j0) {
                    z[j1 * kRow] = r1;
                    o[j1 * kRow] = valid ? v1 : 0.0f;
                }
            }
            __syncthreads();
        }
        // ---- loss (warp 0, a sample per lane, outputs in ascending order) and dz of the last layer (every warp) ----
        {
            const float* o = smem + net.a_row[nl] * kRow + lane;
            const float* t = targets + uint64_t(s0 + lane) * od;
            float* dz = smem + net.z_row[nl] * kRow + lane;
#pragma unroll 1
            for (int j = warp; j < od; j += kSimtWarps)
                dz[j * kRow] = valid ? (2.0f * net.scale) * (o[j * kRow] - (j == warp ? target : __ldg(t + j))) : 0.0f;
            if (warp == 0 && valid) {
                float loss = 0.0f;
#pragma unroll 1
                for (int j = 0; j < od; ++j) {
                    const float diff = o[j * kRow] - (j == 0 ? target : __ldg(t + j));
                    loss = fmaf(diff * net.scale, diff, loss);
                }
                run_max = fmaxf(run_max, loss);
                run_sum += loss;
            }
        }
        __syncthreads();
        // ---- backward: dz of the layer before replaces its z ----
#pragma unroll 1
        for (int l = nl - 1; l >= 1; --l) {
            const int in = net.dims[l], out = net.dims[l + 1], stride = (in + 3) & ~3, i0 = 2 * warp;
            if (i0 < in) {
                const float* dz = smem + net.z_row[l + 1] * kRow + lane;
                const float* w = smem + net.w_at[l] + i0;
                float r0 = 0.0f, r1 = 0.0f;
#pragma unroll 4
                for (int j = 0; j < out; ++j) {
                    const float d = dz[j * kRow];
                    const float2 u = *reinterpret_cast<const float2*>(w + j * stride);
                    r0 = mac(u.x, d, r0, FUSED);
                    r1 = mac(u.y, d, r1, FUSED);
                }
                float* z = smem + (net.z_row[l] + i0) * kRow + lane;
                z[0] = valid ? r0 * act_deriv(MLP_ACT_RELU, 0.0f, z[0]) : 0.0f;
                if (i0 + 1 < in) z[kRow] = valid ? r1 * act_deriv(MLP_ACT_RELU, 0.0f, z[kRow]) : 0.0f;
            }
            __syncthreads();
        }
        // ---- parameter sums of the tile, a parameter at a time (the bias is a row's last), in ascending sample order ----
#pragma unroll 1
        for (int l = 0; l < nl; ++l) {
            const int in = net.dims[l], out = net.dims[l + 1];
            float* dW = (float*)s_net[l].weightsGrad;
            float* dB = (float*)s_net[l].biasesGrad;
#pragma unroll 1
            for (int item = tid; item < out * (in + 1); item += kSimtThreads) {
                const int j = (int)(((uint32_t)item * net.per_row[l]) >> 16), i = item - j * (in + 1);
                const float* d = smem + (net.z_row[l + 1] + j) * kRow;
                const float* a = smem + (net.a_row[l] + min(i, in - 1)) * kRow;
                float acc = 0.0f;
#pragma unroll 2
                for (int s = 0; s < kTile; s += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(d + s);
                    float4 v = *reinterpret_cast<const float4*>(a + s);
                    if (i == in) v = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                    acc = mac(u.w, v.w, mac(u.z, v.z, mac(u.y, v.y, mac(u.x, v.x, acc, FUSED), FUSED), FUSED), FUSED);
                }
                float* g = smem + net.g_at[l] + item;
                if (once) atomicAdd(i == in ? dB + j : dW + j * in + i, acc);
                else *g = tile == blockIdx.x ? acc : *g + acc;
            }
        }
        __syncthreads();   // the next tile overwrites the rows
    }
    if (!once) {
#pragma unroll 1
        for (int l = 0; l < nl; ++l) {
            const int in = net.dims[l], out = net.dims[l + 1];
#pragma unroll 1
            for (int item = tid; item < out * (in + 1); item += kSimtThreads) {
                const int j = (int)(((uint32_t)item * net.per_row[l]) >> 16), i = item - j * (in + 1);
                atomicAdd(i == in ? (float*)s_net[l].biasesGrad + j : (float*)s_net[l].weightsGrad + j * in + i, smem[net.g_at[l] + item]);
            }
        }
    }
    if (warp == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            run_max = fmaxf(run_max, __shfl_xor_sync(0xffffffffu, run_max, o));
            run_sum += __shfl_xor_sync(0xffffffffu, run_sum, o);
        }
        if (lane == 0) {
            atomicMax(lossBuffer, __float_as_uint(run_max));
            atomicAdd((float*)(lossBuffer + 1), run_sum);
        }
    }
}

// Second pass of the sequential mode: one thread per parameter walks the samples in ascending order,
// exactly the adds a sequential machine performs (load, fused multiply-add, store).
__global__ void __launch_bounds__(256)
sequential_sum_kernel(SimtNet net, const MlpLayerPointers* __restrict__ lp, const float* __restrict__ scratch,
                      uint32_t count, int layer)
{
    const MlpConfig& c = net.cfg;
    const bool fused = c.sum_order == MLP_SUM_BIAS_FIRST_FUSED;
    const int in = c.dims[layer], out = c.dims[layer + 1];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= in * out + out) return;
    const int nl = c.n_layers;
    const int na = net.a_off[nl], nz = net.a_off[nl + 1] - net.a_off[1];
    const int64_t stride = na + nz;
    const float* abase = scratch + net.a_off[layer];
    const float* zbase = scratch + na + net.a_off[layer + 1] - net.a_off[1];
    if (p < in * out) {
        const int j = p / in, i = p % in;
        float* dst = (float*)lp[layer].weightsGrad + weight_index(c.param_layout, in, out, j, i);
        float acc = *dst;
        for (uint32_t s = 0; s < count; ++s) acc = mac(zbase[s * stride + j], abase[s * stride + i], acc, fused);
        *dst = acc;
    } else {
        const int j = p - in * out;
        float* dst = (float*)lp[layer].biasesGrad + j;
        float acc = *dst;
        for (uint32_t s = 0; s < count; ++s) acc += zbase[s * stride + j];
        *dst = acc;
    }
}

// adjustParameters, fp32 state (examples/mlp-training/adam.slang:21-37 widened to float):
// NaN gradient -> zero it and skip; +-inf -> +-10000; eps inside the square root; gradient zeroed.
// A thread takes E elements a block apart, their loads issued together, and takes the bias corrections, two powers by
// squaring, once for elements of the same iteration (nearly always all of them).  A parameter that no gradient has
// reached yet (zero gradient, zero moments: the unused slots of a hash table) keeps its value exactly, so only its
// iteration count moves; three divisions and a root per element are what the kernel issues otherwise.  PLAIN: fp32
// parameters without a master copy.  Bound: HBM and instruction issue at E = 4.
template <int E, bool PLAIN>
__global__ void __launch_bounds__(256)
adjust_parameters_kernel(const __grid_constant__ MlpConfig c, MlpAdamState* __restrict__ states, void* __restrict__ params,
                         float* __restrict__ grads, uint32_t count)
{
    const uint32_t first = blockIdx.x * (256u * E) + threadIdx.x;
    grid_release();
    grid_wait();
    float g[E], p[E];
    float4 raw[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const uint32_t i = first + 256u * k;
        g[k] = __int_as_float(0x7fffffff);
        if (i < count) {
            g[k] = grads[i];
            raw[k] = __ldcs(reinterpret_cast<const float4*>(states) + i);
            if constexpr (PLAIN) p[k] = static_cast<const float*>(params)[i];
            else p[k] = c.adam_master ? raw[k].w : load_as_f32(c.dtype, params, i);
        }
    }
    int32_t known = -1;
    float c1 = 0.0f, c2 = 0.0f;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const uint32_t i = first + 256u * k;
        if (i >= count) break;
        float gk = g[k];
        const int32_t it = __float_as_int(raw[k].z) + 1;
        if (gk == 0.0f && (__float_as_uint(raw[k].x) | __float_as_uint(raw[k].y)) == 0u && c.eps > 0.0f) {
            __stcs(reinterpret_cast<float4*>(states) + i, make_float4(0.0f, 0.0f, __int_as_float(it), p[k]));
            if (!PLAIN && c.adam_master) store_from_f32(c.dtype, params, i, p[k]);
            continue;
        }
        grads[i] = 0.0f;
        if (isnan(gk)) continue;
        float mean = raw[k].x, var = raw[k].y;
        if (isinf(gk)) gk = gk > 0.0f ? 10000.0f : -10000.0f;
        mean = c.beta1 * mean + (1.0f - c.beta1) * gk;
        var = c.beta2 * var + ((1.0f - c.beta2) * gk) * gk;
        if (it != known) {
            known = it;
            c1 = 1.0f - pow_int(c.beta1, it);
            c2 = 1.0f - pow_int(c.beta2, it);
        }
        const float mean_hat = __fdiv_rn(mean, c1);
        const float var_hat = __fdiv_rn(var, c2);
        const float denom = __fsqrt_rn(fmaxf(0.0f, var_hat) + c.eps);
        const float v = p[k] - __fdiv_rn(c.lr * mean_hat, denom);
        __stcs(reinterpret_cast<float4*>(states) + i, make_float4(mean, var, __int_as_float(it), v));
        if constexpr (PLAIN) static_cast<float*>(params)[i] = v;
        else store_from_f32(c.dtype, params, i, v);
    }
}

// ------------------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------------------
static bool make_simt_net(const MlpConfig& c, SimtNet* net, std::string* err)
{
    net->cfg = c;
    int off = 0;
    for (int l = 0; l <= c.n_layers; ++l) { net->a_off[l] = off; off += c.dims[l]; }
    net->a_off[c.n_layers + 1] = off;
    if (off > kMaxActFloats) {
        if (err) *err = "sum of layer widths exceeds the limit of the general kernels";
        return false;
    }
    return true;
}

cudaError_t launch_example_learn_gradient(cudaStream_t st, const MlpLearnGradParams& a, uint32_t grid)
{
    return launch_after(st, learnGradient, grid, 256, 0, (const MlpLayerPointers*)a.networkBuffer, (uint32_t*)a.lossBuffer, (const float2*)a.inputs, a.count);
}

cudaError_t launch_example_learn_gradient_coopvec(cudaStream_t st, const MlpLearnGradParams& a, uint32_t grid)
{
    return launch_after(st, learnGradient_coopvec, grid, 256, 0, (const MlpLayerPointers*)a.networkBuffer, (uint32_t*)a.lossBuffer, (const float2*)a.inputs, a.count);
}

cudaError_t launch_example_adjust_parameters(cudaStream_t st, const MlpAdjustParamsParams& a, uint32_t grid)
{
    return launch_after(st, adjustParameters, grid, 256, 0, (MlpExampleAdamState*)a.adamStates, (__half*)a.params, (__half*)a.gradients, a.count);
}

cudaError_t launch_forward_simt(cudaStream_t st, const MlpConfig& c, const MlpForwardParams& a, int* launches,
                                std::string* err)
{
    SimtNet net;
    if (!make_simt_net(c, &net, err)) return cudaErrorInvalidValue;
    if (a.count == 0) return cudaSuccess;
    const uint32_t grid = (a.count + 255) / 256;
    forward_simt_kernel<<<grid, 256, 0, st>>>(net, (const MlpLayerPointers*)a.networkBuffer, (const void*)a.inputs,
                                              (float*)a.outputs, a.count);
    *launches += 1;
    return cudaGetLastError();
}

static bool small_network(const MlpConfig& c)
{
    if (c.dtype != MLP_F32 || (c.operand_dtype && c.operand_dtype != MLP_F32) || c.input_dtype != MLP_F32 || c.target_dtype != MLP_F32) return false;
    if (c.encoding != MLP_ENC_NONE || c.param_layout != MLP_PARAMS_ROW_MAJOR || c.hidden_act != MLP_ACT_RELU || c.output_act != MLP_ACT_IDENTITY) return false;
    for (int l = 0; l <= c.n_layers; ++l)
        if (c.dims[l] > kSmallWidth) return false;
    return true;
}

static cudaError_t launch_learn_gradient_small(cudaStream_t st, const MlpConfig& c, const MlpLearnGradParamsEx& a, int* launches)
{
    SmallNet net = {};
    net.nl = c.n_layers;
    net.od = c.dims[c.n_layers];
    net.scale = c.loss == MLP_LOSS_MSE_MEAN ? 1.0f / float(net.od) : 1.0f;
    net.per_input = (65536u + (uint32_t)c.dims[0] - 1u) / (uint32_t)c.dims[0];
    int rows = 0;
    for (int l = 0; l <= c.n_layers; ++l) { net.dims[l] = c.dims[l]; net.a_row[l] = rows; rows += c.dims[l]; }
    for (int l = 1; l <= c.n_layers; ++l) { net.z_row[l] = rows; rows += c.dims[l]; }
    int floats = rows * kRow;
    for (int l = 0; l < c.n_layers; ++l) {
        net.w_at[l] = floats; floats += c.dims[l + 1] * ((c.dims[l] + 3) & ~3);
        net.per_row[l] = (65536u + (uint32_t)c.dims[l]) / ((uint32_t)c.dims[l] + 1u);
    }
    for (int l = 0; l < c.n_layers; ++l) { net.b_at[l] = floats; floats += c.dims[l + 1]; }
    for (int l = 0; l < c.n_layers; ++l) { net.g_at[l] = floats; floats += c.dims[l + 1] * (c.dims[l] + 1); }
    const size_t smem = size_t(floats) * 4;
    constexpr size_t kLargest = ((2 * MLP_MAX_LAYERS + 1) * kSmallWidth * kRow + MLP_MAX_LAYERS * kSmallWidth * (2 * kSmallWidth + 2)) * 4;
    static_assert(kLargest <= kSimtSmemMax, "the largest small network fits");
    const bool fused = c.sum_order == MLP_SUM_BIAS_FIRST_FUSED;
    auto kern = fused ? learn_gradient_small_kernel<true> : learn_gradient_small_kernel<false>;
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    static SmemLimit limit[2];   // one per build
    if (e == cudaSuccess) e = limit[fused].raise((const void*)kern, device, kLargest);
    if (e != cudaSuccess) return e;
    const uint32_t tiles = (uint32_t)((uint64_t(a.count) + kTile - 1) / kTile);
    const uint32_t per_sm = uint32_t(std::max<size_t>(1, std::min<size_t>(4, kSimtSmemMax / (smem + 2048))));
    *launches += 1;
    return launch_after(st, kern, std::min(tiles, per_sm * uint32_t(sms)), kSimtThreads, smem, net, (const MlpLayerPointers*)a.networkBuffer,
                        (uint32_t*)a.lossBuffer, (const float*)a.inputs, (const float*)a.targets, a.count, tiles);
}

cudaError_t launch_learn_gradient_simt(cudaStream_t st, const MlpConfig& c, const MlpLearnGradParamsEx& a,
                                       float* seq_scratch, int* launches, std::string* err, float* input_grads)
{
    SimtNet net;
    if (!make_simt_net(c, &net, err)) return cudaErrorInvalidValue;
    if (a.count == 0) return cudaSuccess;
    const bool seq = (a.flags & MLP_FLAG_SEQUENTIAL_SUM) != 0;
    if (!seq && !input_grads && small_network(c)) return launch_learn_gradient_small(st, c, a, launches);
    SimtSmem map{};
    int floats = net.a_off[c.n_layers + 1] * kRow;
    map.z = floats;
    floats += (net.a_off[c.n_layers + 1] - net.a_off[1]) * kRow;
    map.bias = floats;
    int nb = 0, nw = 0, ng = 0;
    for (int l = 0; l < c.n_layers; ++l) {
        map.b_off[l] = nb; nb += c.dims[l + 1];
        map.w_off[l] = nw; nw += c.dims[l + 1] * ((c.dims[l] + 3) & ~3);
        map.g_off[l] = ng; ng += c.dims[l + 1] * (c.dims[l] + 1);
    }
    floats += (nb + 3) & ~3;
    // Weights first (every tile reads them twice), then the gradient sums.
    const int room = int(kSimtSmemMax / 4);
    map.w = map.grads = -1;
    if (floats + nw <= room) { map.w = floats; floats += nw; }
    if (!seq && floats + ng <= room) { map.grads = floats; floats += ng; }
    map.total = floats;
    const size_t smem = size_t(floats) * 4;
    static_assert((2 * kMaxActFloats * kRow + kMaxActFloats + 3) * 4 <= kSimtSmemMax, "the vectors of every accepted network fit");
    auto kern = map.w >= 0 ? learn_gradient_simt_kernel<true> : learn_gradient_simt_kernel<false>;
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    static SmemLimit limit[2];   // one per build
    if (e == cudaSuccess) e = limit[map.w >= 0].raise((const void*)kern, device, kSimtSmemMax);
    if (e != cudaSuccess) return e;
    // As many CTAs as are resident at once (512 threads each), each walking its share of the tiles.
    const uint32_t tiles = (uint32_t)((uint64_t(a.count) + kTile - 1) / kTile);
    const uint32_t per_sm = uint32_t(std::max<size_t>(1, std::min<size_t>(2, kSimtSmemMax / (smem + 1024))));
    const uint32_t grid = std::min(tiles, per_sm * uint32_t(sms));
    e = launch_after(st, kern, grid, kSimtThreads, smem, net, map, (const MlpLayerPointers*)a.networkBuffer, (uint32_t*)a.lossBuffer,
                     (const void*)a.inputs, (const void*)a.targets, a.count, tiles, seq ? seq_scratch : nullptr, input_grads);
    *launches += 1;
    if (e != cudaSuccess || !seq) return e;
    for (int l = 0; l < c.n_layers; ++l) {
        const int np = c.dims[l] * c.dims[l + 1] + c.dims[l + 1];
        sequential_sum_kernel<<<(np + 255) / 256, 256, 0, st>>>(net, (const MlpLayerPointers*)a.networkBuffer,
                                                                seq_scratch, a.count, l);
        *launches += 1;
    }
    return cudaGetLastError();
}

size_t sequential_scratch_floats_per_sample(const MlpConfig& c)
{
    size_t n = 0;
    for (int l = 0; l < c.n_layers; ++l) n += size_t(c.dims[l]) + size_t(c.dims[l + 1]);
    return n;
}

cudaError_t launch_adjust_parameters(cudaStream_t st, const MlpConfig& c, const MlpAdjustParamsParams& a, int* launches)
{
    if (a.count == 0) return cudaSuccess;
    // Four elements a thread once that still leaves every one of a B200's 148 SMs eight blocks of 256 (an encoder's table);
    // one below, where the launch is all there is (a network's parameters).  fp32, one against four: 2^18 4.2 / 4.4 us,
    // 2^19 5.3 / 5.1, 2^20 9.3 / 6.7, 1.5 M 12.9 / 8.8, 2^23 70.5 / 55.7.  One also for the
    // last counts, whose indices four apart would not fit 32 bits.
    constexpr uint32_t kMany = 148u * 8u * 1024u;
    MlpAdamState* states = (MlpAdamState*)a.adamStates;
    const auto many = c.dtype == MLP_F32 && !c.adam_master ? adjust_parameters_kernel<4, true> : adjust_parameters_kernel<4, false>;
    const cudaError_t e = a.count >= kMany && a.count <= 0xffffffffu - 1023u
        ? launch_after(st, many, (a.count + 1023) / 1024, 256, 0, c, states, (void*)a.params, (float*)a.gradients, a.count)
        : launch_after(st, adjust_parameters_kernel<1, false>, (a.count + 255) / 256, 256, 0, c, states, (void*)a.params, (float*)a.gradients, a.count);
    *launches += 1;
    return e;
}

// ------------------------------------------------------------------------------------------------
// learnGradient with ordered sums and no allocation
// ------------------------------------------------------------------------------------------------
// The ordered-sum mode parks every sample's layer inputs and output gradients in global memory
// between its two passes.  The variant below keeps that parking area inside the library image
// instead of asking the CUDA allocator for it: 4 MiB per GPU that has loaded the library, resident
// until the process exits.
constexpr size_t kStaticScratchFloats = size_t(1) << 20;
static __device__ __align__(256) float g_static_scratch[kStaticScratchFloats];

// In host code `g_static_scratch` is only a handle for the symbol; the address a kernel may
// dereference differs per device and comes from cudaGetSymbolAddress with that device current.
constexpr int kMaxDevices = 64;
static float* g_static_scratch_addr[kMaxDevices] = {};

void set_last_error(const char* text);                    // abi.cu
bool config_ok(const MlpConfig* c, std::string* why);     // abi.cu

}  // namespace mlpb200

using namespace mlpb200;

extern "C" int32_t mlp_learn_gradient_ordered_noalloc(int32_t device_ordinal, void* cuda_stream, const MlpConfig* config,
                                                      const MlpLearnGradParamsEx* args)
{
    // Everything that can be refused is refused here, before the first CUDA call.
    if (!config || !args) { set_last_error("null argument"); return MLP_E_INVALID_ARG; }
    if (device_ordinal < 0 || device_ordinal >= kMaxDevices) { set_last_error("device ordinal out of range"); return MLP_E_INVALID_ARG; }
    {
        std::string why;
        if (!config_ok(config, &why)) { set_last_error(("bad config: " + why).c_str()); return MLP_E_INVALID_ARG; }
    }
    const MlpConfig& c = *config;
    if (c.param_layout != MLP_PARAMS_ROW_MAJOR) { set_last_error("learnGradient takes row-major parameters"); return MLP_E_NOT_AVAILABLE; }
    if (args->flags & MLP_FLAG_INPUT_GRADIENT) {
        set_last_error("this entry point takes MlpLearnGradParamsEx, which has no input-gradient address: MLP_FLAG_INPUT_GRADIENT is not available here");
        return MLP_E_NOT_AVAILABLE;
    }
    if (args->flags & ~MLP_FLAG_SEQUENTIAL_SUM) { set_last_error("unknown flag bits"); return MLP_E_INVALID_ARG; }
    if (!args->networkBuffer || !args->lossBuffer || (args->count && (!args->inputs || !args->targets))) {
        set_last_error("null device address in the argument struct");
        return MLP_E_INVALID_ARG;
    }
    const size_t need = sequential_scratch_floats_per_sample(c) * size_t(args->count);
    if (need > kStaticScratchFloats) {
        char buf[256];
        snprintf(buf, sizeof buf,
                 "%u samples need %zu scratch floats; the built-in scratch area holds %zu (at most %zu samples of this network)",
                 args->count, need, (size_t)kStaticScratchFloats,
                 (size_t)kStaticScratchFloats / sequential_scratch_floats_per_sample(c));
        set_last_error(buf);
        return MLP_E_INVALID_ARG;
    }
    // The work runs with device_ordinal current; the caller's current device is put back on return.
    int prev_device = -1;
    cudaError_t e = cudaGetDevice(&prev_device);
    if (e == cudaSuccess && prev_device != device_ordinal) e = cudaSetDevice(device_ordinal);
    if (e == cudaSuccess && !g_static_scratch_addr[device_ordinal]) {
        // First call on this device: look the array's device address up once and keep it.
        float* addr = nullptr;
        e = cudaGetSymbolAddress((void**)&addr, g_static_scratch);
        if (e == cudaSuccess) g_static_scratch_addr[device_ordinal] = addr;
    }
    int32_t rc = MLP_OK;
    if (e != cudaSuccess) {
        std::string msg = std::string("CUDA set-up for the built-in scratch area failed: ") + cudaGetErrorString(e);
        set_last_error(msg.c_str());
        rc = MLP_E_CUDA;
    } else if (args->count != 0) {
        MlpLearnGradParamsEx a = *args;
        a.flags |= MLP_FLAG_SEQUENTIAL_SUM;
        int launches = 0;
        std::string err;
        e = launch_learn_gradient_simt((cudaStream_t)cuda_stream, c, a, g_static_scratch_addr[device_ordinal], &launches, &err);
        if (e != cudaSuccess) {
            if (err.empty()) err = std::string("kernel launch failed: ") + cudaGetErrorString(e);
            set_last_error(err.c_str());
            rc = e == cudaErrorInvalidValue ? MLP_E_NOT_AVAILABLE : MLP_E_CUDA;
        }
    }
    if (prev_device >= 0 && prev_device != device_ordinal) cudaSetDevice(prev_device);
    return rc;
}
