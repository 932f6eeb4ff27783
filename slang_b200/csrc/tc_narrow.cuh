// Register-chained networks of widths up to 64: what the training and the forward kernel of tc_narrow.cu share.
//
// A warp owns 16 samples (or 32, as two blocks of 16) and carries them through every layer in registers with
// mma.sync.m16n8k16: the accumulator fragment of one layer, rounded to 16 bits, IS the operand fragment of the next,
// so a layer is products, bias, rounding and activation with no shared-memory round trip, no barrier and no other
// warp to wait for.  At widths of 16 to 64 the tcgen05 products are bound by the shared-memory reads of their 128-row
// operand (40 to 48 cycles per 16 columns of K whatever N is, measured) and by the hand-offs around them; mma.sync
// runs at a quarter of the tensor rate (2 cycles per m16n8k16 per SM, measured) but only the weights, 16 bytes per
// lane for two products, come from shared memory.
//
// Fragments and features.  mma.sync leaves a lane (g = lane / 4, c = lane % 4) the columns 2c, 2c + 1 of every
// 8-column tile for the rows g and g + 8, and wants the same pairs of K as the next operand.  Which feature sits at
// which (tile, column) is free as long as both sides agree, so vectors wider than 16 give lane c eight CONSECUTIVE
// features of every 32 (tile t, column j: feature 32 (t / 4) + 8 (j / 2) + 2 (t % 4) + j % 2): input rows are read and
// output rows written as 16- or 32-byte pieces, and a weight fragment for two K steps is one 16-byte read.  Weights
// are laid out once per CTA in exactly the order the lanes read them: panel[q][t][lane] of 16 bytes holds, for the
// output feature of (t, column g), the eight K slots of lane c in the 32-wide group q.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "mlp_common.cuh"
#include "tc_layout.cuh"
#include "tc_ptx.cuh"

namespace mlpb200 {
namespace narrow {

// How a vector's features are dealt to (tile, column).
enum VectorKind : int { kNatural = 0, kFours = 1, kEights = 2 };

// Natural order up to 8 features (one tile), four consecutive per lane up to 16 (two tiles), eight beyond.
__host__ __device__ constexpr int input_kind(int width) { return width <= 8 ? kNatural : width <= 16 ? kFours : kEights; }
// The same by the number of 8-column tiles, for hidden vectors and outputs.
__host__ __device__ constexpr int tile_kind(int tiles) { return tiles == 1 ? kNatural : tiles == 2 ? kFours : kEights; }

__host__ __device__ constexpr int feature_of(int kind, int t, int j)
{
    return kind == kEights ? 32 * (t >> 2) + 8 * (j >> 1) + 2 * (t & 3) + (j & 1)
         : kind == kFours  ? (t < 2 ? 4 * (j >> 1) + 2 * t + (j & 1) : 1 << 20)
                           : 8 * t + j;
}

struct Params {
    MlpConfig cfg;
    const MlpLayerPointers* net;
    uint32_t* loss_words;
    uint32_t* status;
    const void* inputs;
    const void* targets;
    float* input_grads;   // training, optional: [count][dims[0]] gradient with respect to the (unencoded) inputs
    float* outputs;       // forward: fp32 [count][dims[n_layers]]
    uint32_t count;
    uint32_t n_tiles;     // units of work
    int raw_bytes;        // forward: shared memory for the stored weights
    int vec_in, vec_tgt, vec_out, vec_dx;   // rows may be read / written as whole 16-byte pieces (widths and addresses allow it)
};

template <int FMT> struct Cvt;
template <> struct Cvt<MLP_BF16> {
    static constexpr uint32_t kUmmaFmt = 1;
    static constexpr uint32_t kOnes = 0x3F803F80u;
    static constexpr float kSmallest = 0x1p-133f;   // the smallest number above zero
    __device__ static __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
    __device__ static __forceinline__ uint32_t pack2(float lo, float hi)
    {
        __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&t);
    }
    __device__ static __forceinline__ float lo(uint32_t p) { return __uint_as_float(p << 16); }
    __device__ static __forceinline__ float hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
    __device__ static __forceinline__ uint32_t relu2(uint32_t z2)
    {
        const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&z2), __floats2bfloat162_rn(0.0f, 0.0f));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    __device__ static __forceinline__ uint32_t max2(uint32_t a, uint32_t b)
    {
        const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    // 0xffff in the halves that are above zero
    __device__ static __forceinline__ uint32_t positive_mask(uint32_t a2) { return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&a2), __floats2bfloat162_rn(0.0f, 0.0f)); }
    __device__ static __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
    {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    // the same with the accumulator starting from c
    __device__ static __forceinline__ void mma_from(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float4 c)
    {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
    }
};
template <> struct Cvt<MLP_F16> {
    static constexpr uint32_t kUmmaFmt = 0;
    static constexpr uint32_t kOnes = 0x3C003C00u;
    static constexpr float kSmallest = 0x1p-24f;
    __device__ static __forceinline__ float round(float v) { return __half2float(__float2half_rn(v)); }
    __device__ static __forceinline__ uint32_t pack2(float lo, float hi)
    {
        __half2 t = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&t);
    }
    __device__ static __forceinline__ float lo(uint32_t p) { return __half2float(__ushort_as_half((uint16_t)(p & 0xffffu))); }
    __device__ static __forceinline__ float hi(uint32_t p) { return __half2float(__ushort_as_half((uint16_t)(p >> 16))); }
    __device__ static __forceinline__ uint32_t relu2(uint32_t z2)
    {
        const __half2 r = __hmax2(*reinterpret_cast<const __half2*>(&z2), __floats2half2_rn(0.0f, 0.0f));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    __device__ static __forceinline__ uint32_t max2(uint32_t a, uint32_t b)
    {
        const __half2 r = __hmax2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    __device__ static __forceinline__ uint32_t positive_mask(uint32_t a2) { return __hgt2_mask(*reinterpret_cast<const __half2*>(&a2), __floats2half2_rn(0.0f, 0.0f)); }
    __device__ static __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
    {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    // the same with the accumulator starting from c
    __device__ static __forceinline__ void mma_from(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float4 c)
    {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
    }
};

// Transposes an 8x8 block of 16-bit values held one row pair per lane.
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v)
{
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ float4 lds_float4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
// Four 8x8 blocks of 16-bit values from an operand fragment; lane i gives the address of row i % 8 of block i / 8.
__device__ __forceinline__ void store_fragment(uint32_t addr, const uint32_t (&a)[4])
{
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
}

// Where the 16-byte chunk `chunk` of row `row` of a [rows][W] operand tile lies inside its row (W 32 or 64).
template <int W>
__device__ __forceinline__ int swizzled_chunk(int row, int chunk) { return chunk ^ ((row >> layout::swz_shift(W)) & layout::swz_mask(W)); }

// Where feature f of a vector lies: 8 * tile + column.
__host__ __device__ constexpr int position_of(int kind, int f)
{
    return kind == kEights ? 32 * (f >> 5) + 8 * ((f & 7) >> 1) + 2 * ((f >> 3) & 3) + (f & 1)
         : kind == kFours  ? 8 * ((f >> 1) & 1) + 2 * (f >> 2) + (f & 1)
                           : f;
}

// One weight panel: groups of 32 K slots x `tiles` tiles x 32 lanes x 16 bytes.  `transposed`: the columns are the layer's
// inputs and K its outputs (the reverse products), else columns are outputs and K inputs.
struct Panel {
    const void* weights;   // the parameters, or their copy in shared memory
    uint32_t dst;          // byte offset
    int in, out, in_kind, out_kind, tiles;
    bool transposed;
};

// Chunk `idx` (16 bytes: lane idx % 32 of a tile) of a panel.
template <int FMT>
__device__ __forceinline__ uint4 panel_chunk(const MlpConfig& c, const Panel& p, int idx)
{
    using C = Cvt<FMT>;
    const uint16_t* w16 = (const uint16_t*)p.weights;
    const float* w32 = (const float*)p.weights;
    const int lane = idx & 31, tt = idx >> 5, q = tt / p.tiles, t = tt - q * p.tiles;
    const int g = lane >> 2, cc = lane & 3;
    const int n = feature_of(p.transposed ? p.in_kind : p.out_kind, t, g);
    uint16_t h[8];
    if ((p.transposed ? p.out_kind : p.in_kind) == kEights && c.param_layout == MLP_PARAMS_ROW_MAJOR && c.dtype != MLP_F32) {
        // the usual case: eight consecutive K features, along a stored row or down a stored column
        const int k0 = 32 * q + 8 * cc, limit = n < (p.transposed ? p.in : p.out) ? (p.transposed ? p.out : p.in) - k0 : 0;
        if (!p.transposed && (p.in & 7) == 0 && ((uint64_t)w16 & 15u) == 0) return limit > 0 ? *(const uint4*)(w16 + n * p.in + k0) : make_uint4(0u, 0u, 0u, 0u);
        const uint16_t* w = p.transposed ? w16 + k0 * p.in + n : w16 + n * p.in + k0;
        const int step = p.transposed ? p.in : 1;
#pragma unroll
        for (int r = 0; r < 8; ++r) h[r] = r < limit ? w[r * step] : (uint16_t)0;
        return make_uint4(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16), h[4] | ((uint32_t)h[5] << 16), h[6] | ((uint32_t)h[7] << 16));
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int k = feature_of(p.transposed ? p.out_kind : p.in_kind, 4 * q + (r >> 1), 2 * cc + (r & 1));
        const int o = p.transposed ? k : n, i = p.transposed ? n : k;
        h[r] = 0;
        if (o < p.out && i < p.in) {
            const int wi = (int)weight_index(c.param_layout, p.in, p.out, o, i);
            h[r] = c.dtype == MLP_F32 ? (uint16_t)(C::pack2(w32[wi], 0.0f) & 0xffffu) : w16[wi];
        }
    }
    return make_uint4(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16), h[4] | ((uint32_t)h[5] << 16), h[6] | ((uint32_t)h[7] << 16));
}

// Bytes of a layer's weights as they are stored.
__host__ __device__ inline uint32_t stored_weight_bytes(const MlpConfig& c, int l)
{
    uint32_t in = (uint32_t)c.dims[l], out = (uint32_t)c.dims[l + 1];
    if (c.param_layout == MLP_PARAMS_OPTIMAL) { in = (in + 15u) & ~15u; out = (out + 15u) & ~15u; }
    return in * out * (c.dtype == MLP_F32 ? 4u : 2u);
}

// Copies the stored weights of all layers to shared memory, all copies in flight together; copied[l] is where layer l's
// lie, or its own address where they do not fit `room` bytes or do not start on a 16-byte boundary.  Each panel is then
// cut from there.  Cut straight from global memory, value by value, the panels took 4 of the 20 us of a step of 128
// samples.  cp_async_wait_all() and a barrier are still to come.
template <int NLMAX>
__device__ __forceinline__ void copy_weights(uint8_t* raw, uint32_t room, const MlpConfig& c, const MlpLayerPointers* net, const void** copied, int tid, int nthreads)
{
    uint32_t at = 0;
#pragma unroll
    for (int l = 0; l < NLMAX; ++l) {
        if (l >= c.n_layers) break;
        const uint32_t bytes = stored_weight_bytes(c, l), whole = bytes & ~15u;
        const uint8_t* src = (const uint8_t*)net[l].weights;
        const bool fits = at + bytes <= room && ((uint64_t)src & 15u) == 0;
        if (fits) {
            const uint32_t dst = ptx::smem_u32(raw + at);
            for (uint32_t i = (uint32_t)tid * 16u; i < whole; i += (uint32_t)nthreads * 16u) ptx::cp_async_16(dst + i, src + i);
            if ((uint32_t)tid < (bytes - whole) / 2u) ((uint16_t*)(raw + at + whole))[tid] = ((const uint16_t*)(src + whole))[tid];
        }
        if (tid == 0) copied[l] = fits ? (const void*)(raw + at) : (const void*)src;
        at += (bytes + 15u) & ~15u;
    }
}

// Cuts every panel of a network: `panel(i)` describes panel i, whose chunks number at most PC.
template <int FMT, int PC, class F>
__device__ __forceinline__ void cut_panels(uint8_t* smem, const MlpConfig& c, int n_panels, F panel, int tid, int nthreads)
{
#pragma unroll 2
    for (int i = tid; i < n_panels * PC; i += nthreads) {
        int chunks;
        const Panel p = panel(i / PC, &chunks);
        if (i % PC < chunks) *(uint4*)(smem + p.dst + (uint32_t)(i % PC) * 16u) = panel_chunk<FMT>(c, p, i % PC);
    }
}

// acc[m][t] = start + A[m] (KS steps of 16) x panel; `panel` is this lane's address of (q 0, tile 0), `qstride` the bytes
// from one 32-wide K group to the next.  The start is zero, or (BIAS) the layer's biases, which lie in shared memory in
// (tile, column) order, every pair twice (both rows of the fragment), at `start` (this lane's address); either enters as the first product's third operand.
template <int FMT, bool BIAS, int MT, int NT, int KS, int NA, int KA>
__device__ __forceinline__ void layer_product(float (&acc)[MT][NA][4], const uint32_t (&A)[MT][KA][4], uint32_t panel, uint32_t qstride, uint32_t start)
{
#pragma unroll
    for (int q = 0; q < (KS + 1) / 2; ++q) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const uint4 b = lds128(panel + (uint32_t)q * qstride + (uint32_t)t * 512u);
            if (q == 0) {
                float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (BIAS) c = lds_float4(start + (uint32_t)t * 64u);
#pragma unroll
                for (int m = 0; m < MT; ++m) Cvt<FMT>::mma_from(acc[m][t], A[m][0], b.x, b.y, c);
            } else {
#pragma unroll
                for (int m = 0; m < MT; ++m) Cvt<FMT>::mma(acc[m][t], A[m][2 * q], b.x, b.y);
            }
            if (2 * q + 1 < KS) {
#pragma unroll
                for (int m = 0; m < MT; ++m) Cvt<FMT>::mma(acc[m][t], A[m][2 * q + 1], b.z, b.w);
            }
        }
    }
}

// N consecutive values of one row from feature f0 on, as floats; zero past the row's width.
template <int N>
__device__ __forceinline__ void load_values(float (&v)[N], int dtype, const void* base, uint64_t row, int width, int f0, bool vec)
{
    const uint64_t at = row * (uint64_t)width + (uint64_t)f0;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = 0.0f;
    if (f0 >= width) return;
    if (dtype == MLP_F32) {
        const float* p = (const float*)base + at;
        if (vec && N >= 4) {
#pragma unroll
            for (int i = 0; i + 4 <= N; i += 4) {
                const float4 x = __ldg((const float4*)(p + i));
                v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (f0 + i < width) v[i] = __ldg(p + i);
        }
    } else {
        const uint16_t* p = (const uint16_t*)base + at;
        uint16_t h[N];
        if (vec && N == 8) {
            const uint4 x = __ldg((const uint4*)p);
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int i = 0; i < N; ++i) h[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i) h[i] = f0 + i < width ? __ldg(p + i) : (uint16_t)0;
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            v[i] = dtype == MLP_F16 ? __half2float(__ushort_as_half(h[i])) : __uint_as_float((uint32_t)h[i] << 16);
    }
}

// Coordinates far outside the unit square: the library's own argument reduction.
static __device__ __noinline__ float2 sincos_far(float arg)
{
    float2 r;
    sincosf(arg, &r.x, &r.y);
    return r;
}

// Four octaves of the frequency encoding from octave k0 (0 or 4) on, of two coordinates at once: sin and cos of 2^k times
// the rounded product pi v.  (pi v) / pi is taken once, as an unevaluated sum of two floats; scaling by 2^k and removing
// whole turns of its leading part are exact.  What is left, an angle of at most pi, is quartered, put through the Taylor
// series (to x^9 and x^8: below 6e-8 on [0, pi / 4]) and doubled back twice; the odd octaves are one more doubling.  Sine
// and cosine carry an error of about 6e-7, against an operand rounding of 2e-4 (half) or 2e-3 (bfloat16), for a fifth of
// the instructions of eight sincosf calls (which took 0.4 of the forward kernel's).
__device__ __forceinline__ void encode_octaves(float v0, float v1, int k0, float2 (&x)[8])
{
    const auto both = [](float f) { return make_float2(f, f); };
    constexpr float kInvPi = 0.318309886183790671538f;                                // 1 / pi rounded to a float,
    constexpr float kInvPiLow = (float)(0.318309886183790671538 - (double)kInvPi);    // and what the rounding left
    const float2 y = __fmul2_rn(__fmul2_rn(make_float2(v0, v1), both(3.14159265358979323846f)), both(k0 ? 16.0f : 1.0f));
    if (fmaxf(fabsf(v0), fabsf(v1)) > 4096.0f) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 a = sincos_far(y.x * (float)(1 << k)), b = sincos_far(y.y * (float)(1 << k));
            x[2 * k] = make_float2(a.x, b.x);
            x[2 * k + 1] = make_float2(a.y, b.y);
        }
        return;
    }
    const float2 hi = __fmul2_rn(y, both(kInvPi));
    const float2 lo = __ffma2_rn(y, both(kInvPiLow), __ffma2_rn(y, both(kInvPi), make_float2(-hi.x, -hi.y)));
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const float2 h = __fmul2_rn(hi, both((float)(1 << k)));
        // nearest even multiple: half of h rounded to an integer by the 1.5 * 2^23 trick
        const float2 n = __fadd2_rn(__ffma2_rn(h, both(0.5f), both(12582912.0f)), both(-12582912.0f));
        const float2 r = __ffma2_rn(lo, both((float)(1 << k)), __ffma2_rn(n, both(-2.0f), h));
        const float2 q = __fmul2_rn(r, both(0.78539816339744830962f)), q2 = __fmul2_rn(q, q);
        float2 s = __ffma2_rn(q2, both(1.0f / 362880.0f), both(-1.0f / 5040.0f));
        s = __ffma2_rn(q2, s, both(1.0f / 120.0f));
        s = __ffma2_rn(q2, s, both(-1.0f / 6.0f));
        s = __ffma2_rn(__fmul2_rn(q, q2), s, q);
        float2 c = __ffma2_rn(q2, both(1.0f / 40320.0f), both(-1.0f / 720.0f));
        c = __ffma2_rn(q2, c, both(1.0f / 24.0f));
        c = __ffma2_rn(q2, c, both(-0.5f));
        c = __ffma2_rn(q2, c, both(1.0f));
#pragma unroll
        for (int d = 0; d < 3; ++d) {   // sin 2a = 2 sin a cos a, cos 2a = 1 - 2 sin^2 a
            const float2 s2 = __fadd2_rn(s, s);
            const float2 cd = __ffma2_rn(make_float2(-s2.x, -s2.y), s, both(1.0f));
            s = __fmul2_rn(s2, c);
            c = cd;
            if (d >= 1) { x[2 * (k + d - 1)] = s; x[2 * (k + d - 1) + 1] = c; }
        }
    }
}

// 0xffff in the halves whose sign bit is set.
__device__ __forceinline__ uint32_t sign_mask(uint32_t v)
{
    uint32_t m;
    asm("prmt.b32 %0, %1, %1, 0xbb99;" : "=r"(m) : "r"(v));
    return m;
}

// Up to two values per row that a lane reads itself (small inputs, coordinates of the frequency encoding), fetched a
// tile ahead of their use.
template <int MT> struct RawInputs { float v[MT][2][2]; };

__device__ __forceinline__ bool raw_inputs(const MlpConfig& cfg) { return cfg.encoding == MLP_ENC_FREQ2D || cfg.dims[0] <= 8; }

template <int MT>
__device__ __forceinline__ void fetch_raw(RawInputs<MT>& raw, const Params& p, uint64_t row0, uint64_t block_rows, int c)
{
    const MlpConfig& cfg = p.cfg;
    if (!raw_inputs(cfg)) return;
    const bool freq = cfg.encoding == MLP_ENC_FREQ2D;
    const int width = freq ? 2 : cfg.dims[0], f0 = freq ? c >> 1 : 2 * c;
    const bool two = !freq && f0 + 1 < width;
#pragma unroll
    for (int i = 0; i < MT * 2; ++i) {
        const uint64_t row = row0 + block_rows * (uint64_t)(i >> 1) + 8u * (uint64_t)(i & 1);
        float v0 = 0.0f, v1 = 0.0f;
        if (row < p.count && f0 < width) {
            const uint64_t at = row * (uint64_t)width + (uint64_t)f0;
            if (cfg.input_dtype == MLP_F32) {
                v0 = __ldg((const float*)p.inputs + at);
                if (two) v1 = __ldg((const float*)p.inputs + at + 1);
            } else {
                v0 = load_as_f32(cfg.input_dtype, p.inputs, (int64_t)at);
                if (two) v1 = load_as_f32(cfg.input_dtype, p.inputs, (int64_t)at + 1);
            }
        }
        raw.v[i >> 1][i & 1][0] = v0;
        raw.v[i >> 1][i & 1][1] = v1;
    }
}

// The operand fragments of the input rows `row0` (lane row g) and `row0 + 8` of one 16-sample block.
template <int FMT, int KA>
__device__ __forceinline__ void load_inputs(uint32_t (&A)[KA][4], const Params& p, const float (&raw)[2][2], uint64_t row0, int c)
{
    using C = Cvt<FMT>;
    const MlpConfig& cfg = p.cfg;
    const int in = cfg.dims[0];
#pragma unroll
    for (int k = 0; k < KA; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) A[k][i] = 0u;
    if (cfg.encoding == MLP_ENC_FREQ2D) {
        if constexpr (KA >= 2) {
            float2 x[8];
            encode_octaves(raw[0][0], raw[1][0], (c & 1) * 4, x);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                A[i >> 1][(i & 1) * 2] = C::pack2(x[2 * i].x, x[2 * i + 1].x);
                A[i >> 1][(i & 1) * 2 + 1] = C::pack2(x[2 * i].y, x[2 * i + 1].y);
            }
        }
    } else if (in <= 8) {
#pragma unroll
        for (int h = 0; h < 2; ++h) A[0][h] = C::pack2(raw[h][0], raw[h][1]);
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint64_t row = row0 + 8u * (uint64_t)h;
            if (row >= p.count) continue;
            if (in <= 16) {
                float x[4];
                load_values<4>(x, cfg.input_dtype, p.inputs, row, in, 4 * c, p.vec_in != 0);
#pragma unroll
                for (int i = 0; i < 2; ++i) A[0][i * 2 + h] = C::pack2(x[2 * i], x[2 * i + 1]);
            } else {
#pragma unroll
                for (int q = 0; q < KA / 2; ++q) {
                    if (32 * q >= in) break;
                    float x[8];
                    load_values<8>(x, cfg.input_dtype, p.inputs, row, in, 32 * q + 8 * c, p.vec_in != 0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) A[2 * q + (i >> 1)][(i & 1) * 2 + h] = C::pack2(x[2 * i], x[2 * i + 1]);
                }
            }
        }
    }
}

// Activations without a build of their own: one copy of the switch, run per element of a local array.
template <int N>
__device__ __forceinline__ void activate_any(int act, float alpha, float (&v)[N], float (&d)[N], bool with_derivative)
{
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
        const float z = v[i];
        v[i] = act_value(act, alpha, z);
        if (with_derivative) d[i] = act_deriv(act, alpha, z);
    }
}

// The hidden activation a network's build is chosen by: leaky ReLU as max(z, alpha z) needs 0 < alpha < 1 (at zero, an
// infinite z would not give the NaN that alpha z is).
inline int built_activation(const MlpConfig& c)
{
    if (c.hidden_act == MLP_ACT_LEAKY_RELU && !(c.act_alpha > 0.0f && c.act_alpha < 1.0f)) return -1;
    return c.hidden_act;
}

// n / d for 0 <= n <= 1 <= d <= 2: the hardware's reciprocal and one correction by the exact remainder (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990), which leaves half a unit in the last
// place and 2^-20 of one, without the range checks of a general division (1920 x 1080 view with a sigmoid on every column of
// the output tile: 146.5 us, with __fdiv_rn 151.7, with the two units of __fdividef 143.5).
__device__ __forceinline__ float divide_by_1_to_2(float n, float d)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = n * r;
    return fmaf(fmaf(-d, q, n), r, q);
}

// The output activation of N values and its derivative.
template <int N>
__device__ __forceinline__ void activate_outputs(int act, float alpha, float (&v)[N], float (&d)[N], bool with_derivative)
{
    if (act == MLP_ACT_IDENTITY) {
#pragma unroll
        for (int i = 0; i < N; ++i) d[i] = 1.0f;
    } else if (N <= 8 && act == MLP_ACT_SIGMOID) {   // few outputs: the usual image-fit head, without the switch
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float ex = expf(-fabsf(v[i]));
            v[i] = divide_by_1_to_2(v[i] >= 0.0f ? 1.0f : ex, 1.0f + ex);
            d[i] = v[i] * (1.0f - v[i]);
        }
    } else {
        activate_any(act, alpha, v, d, with_derivative);
    }
}

// GELU (tanh form) with one tanh for value and derivative: the expressions of act_value and act_deriv.
__device__ __forceinline__ void gelu_pair(float z, float& a, float& d)
{
    const float z2 = z * z;
    const float t = tanhf(MLPB200_SQRT_2_OVER_PI * (z + MLPB200_GELU_C * z * z2));
    const float du = MLPB200_SQRT_2_OVER_PI * (1.0f + 3.0f * MLPB200_GELU_C * z2);
    a = 0.5f * z * (1.0f + t);
    d = 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * du;
}

}  // namespace narrow
}  // namespace mlpb200
