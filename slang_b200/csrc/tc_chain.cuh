// Networks of widths up to 128 on tcgen05 with whole tiles of 128 samples: what the kernels of tc_chain.cu share.
//
// A "chain" is four warps that carry one tile through the network: a thread owns one sample (one tensor-memory lane).  The
// layer inputs A_l lie in shared memory as [128 samples][features] tiles, 16-bit, swizzled, so that one copy is the K-major
// operand of the next layer's product and the MN-major operand of the weight-gradient product, and dZ_l replaces A_{l+1} where
// it lay.  A fifth warp per chain issues its layer products and one or two warps the gradient products of all chains, so nothing
// waits for another chain, and a chain's hand-offs (some 500 cycles each) are covered by the others' work.
// The kernels are bound by instruction issue and by instruction fetches: what a tile runs through is some 2300 instructions,
// about as much as the instruction cache holds, so what runs once per tile or rarely is kept small or behind a call (texture
// network, 2^24 texels: 2.64 ms a step with a copy of the gradient products' code per layer and chain, 2.51 with one; later 2.42
// with the waits' polling loops and the marked zeros' code in line, 2.16 without; 2.11 with the least polling between gradient products).
#pragma once

#include "tc_layout.cuh"
#include "tc_narrow.cuh"

namespace mlpb200 {
namespace chain {

using narrow::Cvt;
using namespace ptx;
using narrow::Params;

constexpr int kTile = 128;   // samples of a tile

// tcgen05.wait::ld that the loaded registers depend on
__device__ __forceinline__ void wait_ld(uint32_t (&r)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 ::"memory");
}
__device__ __forceinline__ void wait_ld(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 ::"memory");
}

// mbar_wait() with all but the first poll behind a call.
static __device__ __noinline__ bool wait_on(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status, uint32_t code)
{
    return mbar_wait(bar, parity, abort_flag, status, code);
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status, uint32_t code)
{
    return mbar_try_wait(bar, parity) || wait_on(bar, parity, abort_flag, status, code);
}

__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b)
{
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Byte offset of the first 16-byte chunk of row r of a [rows][W] operand tile (W 16, 32, 64 or 128); chunk j is there ^ (16 j), as
// tiles start on 1024-byte boundaries.  128 features are two panels of 64, one after the other: chunk 8 + j is a panel further.
template <int W>
__device__ __forceinline__ uint32_t row_at(int r)
{
    return (uint32_t)r * (uint32_t)layout::row_bytes(W) + (uint32_t)(((r >> layout::swz_shift(W)) & layout::swz_mask(W)) << 4);
}

// Operand descriptors of a [rows][W] tile at byte offset `at` (lo: the base's address field).  K-major: step k is 16
// features, 32 bytes inside the row (of panel k / 4; `panel`: bytes of one).  MN-major: step k is 16 rows; `lbo` bytes lead
// from one row-wide block of the other dimension to the next.
template <int W>
__device__ __forceinline__ uint64_t desc_k(uint32_t lo, uint32_t at, int k, uint32_t panel = 0u)
{
    constexpr uint32_t hi = ((8u * (uint32_t)layout::row_bytes(W)) >> 4) | (1u << 14) | (layout::layout_type(W) << 29);
    return ((uint64_t)hi << 32) | (lo + ((at + (uint32_t)(k >> 2) * panel + (uint32_t)(W > 64 ? k & 3 : k) * 32u) >> 4) + (1u << 16));
}
template <int W>
__device__ __forceinline__ uint64_t desc_mn(uint32_t lo, uint32_t at, int k, uint32_t lbo = 16u)
{
    constexpr uint32_t hi = ((8u * (uint32_t)layout::row_bytes(W)) >> 4) | (1u << 14) | (layout::layout_type(W) << 29);
    return ((uint64_t)hi << 32) | (lo + ((at + (uint32_t)k * 16u * (uint32_t)layout::row_bytes(W)) >> 4) + ((lbo >> 4) << 16));
}
// Where the block of 32 features b of a row lies (row: row_at() of it).
template <int W>
__device__ __forceinline__ uint32_t block_at(uint32_t row, int b)
{
    return W == 128 ? (row ^ (uint32_t)(64 * (b & 1))) + (uint32_t)(b >> 1) * (kTile * 128u) : row ^ (uint32_t)(64 * b);
}

// The biases of hidden layers enter as one more K step of the layer product, the first: a tile of rows (1, 0, .. 0) times rows
// (bias, 0, .. 0), 16 wide.  The accumulator is then the pre-activation (one addition and half a shared-memory read per
// pair of values less: 1920 x 1080 view 106 -> 95 us, texture step of 2^24 texels 2.52 -> 2.39 ms).  All groups of eight rows of the first are one.
constexpr uint32_t kUnitBytes = 8 * 32;
__device__ __forceinline__ uint64_t desc_unit(uint32_t lo, uint32_t at)
{
    constexpr uint32_t hi = (1u << 14) | (layout::layout_type(16) << 29);
    return ((uint64_t)hi << 32) | (lo + (at >> 4) + (1u << 16));
}
// Rows whose first value is `value(row)` and the rest zero.
template <class F>
__device__ __forceinline__ void first_column(uint8_t* dst, int rows, int tid, int nthreads, F value)
{
    for (int row = tid; row < rows; row += nthreads) {
        uint8_t* at = dst + row_at<16>(row);
        *(uint4*)at = make_uint4(value(row) & 0xffffu, 0u, 0u, 0u);
        *(uint4*)(dst + (row_at<16>(row) ^ 16u)) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// A layer's weights as a zero-padded [rows][W] tile (rows: outputs), 16-bit storage.  cp_async_wait_all() is still to come.
template <int W>
__device__ __forceinline__ void stage_weights(uint8_t* dst, const MlpConfig& c, const void* weights, int rows, int in, int out, int tid, int nthreads)
{
    const uint16_t* w = (const uint16_t*)weights;
    const bool whole = c.param_layout == MLP_PARAMS_ROW_MAJOR && (in & 7) == 0 && ((uint64_t)w & 15u) == 0;
#pragma unroll 1
    for (int i = tid; i < rows * (W / 8); i += nthreads) {
        const int o = i / (W / 8), j = i % (W / 8);
        uint8_t* at = dst + (row_at<W>(o) ^ (uint32_t)(16 * (j & 7))) + (uint32_t)(j >> 3) * (uint32_t)rows * 128u;
        if (whole && o < out && 8 * j < in) {   // all copies of all layers in flight together
            cp_async_16(smem_u32(at), w + o * in + 8 * j);
            continue;
        }
        uint16_t h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) h[e] = o < out && 8 * j + e < in ? w[weight_index(c.param_layout, in, out, o, 8 * j + e)] : (uint16_t)0;
        *(uint4*)at = make_uint4(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16), h[4] | ((uint32_t)h[5] << 16), h[6] | ((uint32_t)h[7] << 16));
    }
}

// Value i of a row of fp32 or 16-bit values where `real`, else zero, without a branch; what is loaded is first touched by its use.
__device__ __forceinline__ uint32_t load_bits(const char* row, bool wide, int i, bool real)
{
    uint32_t v;
    if (wide)
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.b32 %0, [%1];\n\t}" : "=r"(v) : "l"(row + 4 * i), "r"((int)real));
    else
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.u16 %0, [%1];\n\t}" : "=r"(v) : "l"(row + 2 * i), "r"((int)real));
    return v;
}
__device__ __forceinline__ float bits_value(int dtype, uint32_t b)
{
    return dtype == MLP_F32 ? __uint_as_float(b) : dtype == MLP_F16 ? __half2float(__ushort_as_half((uint16_t)b)) : __uint_as_float(b << 16);
}

// What a thread needs of its next sample's input before it can build the row: the two coordinates of the frequency
// encoding, or the whole of a short row, as stored.
struct RawRow { uint32_t v[8]; };

__device__ __forceinline__ bool short_row(const MlpConfig& c) { return c.encoding == MLP_ENC_FREQ2D || c.dims[0] <= 8; }

// Where a thread's input or target rows lie: one tile's to the next's.
struct Rows {
    const char* at;
    uint64_t step;
    __device__ __forceinline__ Rows(const void* base, int width, int dtype, uint64_t sample, uint32_t samples)
        : at((const char*)base + sample * (uint64_t)(width * (dtype == MLP_F32 ? 4 : 2))), step((uint64_t)samples * (uint64_t)(width * (dtype == MLP_F32 ? 4 : 2))) {}
};
__device__ __forceinline__ int stored_inputs(const MlpConfig& c) { return c.encoding == MLP_ENC_FREQ2D ? 2 : c.dims[0]; }

// 16 bytes where `real`, else zero, as load_bits().
__device__ __forceinline__ void load_four(uint32_t* v, const char* at, bool real)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                 "@q ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(at), "r"((int)real));
}

__device__ __forceinline__ void fetch_row(RawRow& raw, const Params& p, const char* row, bool real)
{
    const MlpConfig& c = p.cfg;
    if (!short_row(c)) return;
    const int width = stored_inputs(c);
    const bool wide = c.input_dtype == MLP_F32;
    if (wide && p.vec_in && c.encoding != MLP_ENC_FREQ2D) {   // four or eight values
        load_four(raw.v, row, real);
        if (width > 4) load_four(raw.v + 4, row + 16, real);
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i == 2 && width <= 2) break;
        if (i == 4 && width <= 4) break;
        raw.v[i] = load_bits(row, wide, i, real && i < width);
    }
}

// Rows of nine to sixteen values that are not whole 16-byte pieces of fp32 or operand-type values.
template <int FMT>
static __device__ __forceinline__ void convert_row(uint32_t at, int dtype, const char* row, int width, bool real)
{
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = real && 8 * j + i < width ? load_as_f32(dtype, row, 8 * j + i) : 0.0f;
        using C = Cvt<FMT>;
        sts128(at ^ (uint32_t)(16 * j), C::pack2(x[0], x[1]), C::pack2(x[2], x[3]), C::pack2(x[4], x[5]), C::pack2(x[6], x[7]));
    }
}

// Wider ones: the warp reads its rows as the one run of memory they are, values or pairs of them side by side, and puts each where
// it belongs.  (A row a thread, value by value, every load touched 32 rows: forward of 600000 samples of 59-62-62-62-27, fp32 rows, 382 us, 123 so; a step of
// 33-63-63-63-9, halves, 217 and 161.)  `tile`: the tile's address; `rows`: how many of the warp's are real.
template <int FMT, int IW>
static __device__ __forceinline__ void scatter_rows(uint32_t tile, int dtype, const char* src, int width, int rows)
{
    using C = Cvt<FMT>;
    const int lane = threadIdx.x & 31, r0 = (int)(threadIdx.x & 96u), n = rows * width;
    const uint32_t inverse = ((1u << 20) + (uint32_t)width - 1u) / (uint32_t)width;   // (i * inverse) >> 20 is i / width for i < 32 width <= 2048
    const auto place = [&](int i) {
        const int r = (int)(((uint32_t)i * inverse) >> 20), f = i - r * width;
        return (tile + row_at<IW>(r0 + r)) ^ (uint32_t)(2 * f);   // (inside its row of 64 or 128 bytes a row's address has only the swizzle's bits)
    };
    // the rest of the last K step, and rows past the batch
    for (int f = rows > lane ? width & ~15 : 0; f < ((width + 15) & ~15); f += 8) sts128((tile + row_at<IW>(r0 + lane)) ^ (uint32_t)(2 * f), 0u, 0u, 0u, 0u);
    __syncwarp();
    if (dtype == FMT && ((width & 1) | (int)((uint64_t)src & 3u)) == 0) {
#pragma unroll 8
        for (int i = 2 * lane; i < n; i += 64) {
            const uint32_t v = __ldg((const uint32_t*)src + i / 2);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(place(i)), "r"(v) : "memory");
        }
    } else if (dtype == MLP_F32 && ((width & 1) | (int)((uint64_t)src & 7u)) == 0) {
#pragma unroll 8
        for (int i = 2 * lane; i < n; i += 64) {
            const float2 v = __ldg((const float2*)src + i / 2);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(place(i)), "r"(C::pack2(v.x, v.y)) : "memory");
        }
    } else if (dtype == MLP_F32) {
#pragma unroll 8
        for (int i = lane; i < n; i += 32) {
            const float v = __ldg((const float*)src + i);
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(place(i)), "h"((uint16_t)C::pack2(v, 0.0f)) : "memory");
        }
    } else {
#pragma unroll 8
        for (int i = lane; i < n; i += 32) {
            const uint32_t v = __ldg((const unsigned short*)src + i);
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(place(i)), "h"((uint16_t)(dtype == FMT ? v : C::pack2(bits_value(dtype, v), 0.0f))) : "memory");
        }
    }
    __syncwarp();
}

// Either, behind one call with the arguments that are at hand, so that the other kinds of rows do not fetch it.
template <int FMT, int IW>
static __device__ __noinline__ void ragged_row(uint32_t at, int dtype, const char* row, int width, bool real)
{
    if (width <= 16) {
        convert_row<FMT>(at, dtype, row, width, real);
    } else {
        const char* first = row - (size_t)(threadIdx.x & 31u) * (size_t)(width * (dtype == MLP_F32 ? 4 : 2));
        scatter_rows<FMT, IW>(at - row_at<IW>((int)(threadIdx.x & 127u)), dtype, first, width, __popc(__ballot_sync(0xffffffffu, real)));
    }
}

// A thread's input row in operand format, up to the end of its last K step.
template <int FMT, int IW>
__device__ __forceinline__ void write_row(uint32_t at, const Params& p, const RawRow& raw, const char* src_row, bool real)
{
    using C = Cvt<FMT>;
    const MlpConfig& c = p.cfg;
    const int width = c.dims[0], type = c.input_dtype;
    if (c.encoding == MLP_ENC_FREQ2D) {
        // chunks 0, 1: the first coordinate's octaves 0 to 3 and 4 to 7; chunks 2, 3: the second's
        const float u = bits_value(type, raw.v[0]), v = bits_value(type, raw.v[1]);
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            float2 x[8];
            narrow::encode_octaves(u, v, 4 * k, x);
            sts128(at ^ (uint32_t)(16 * k), C::pack2(x[0].x, x[1].x), C::pack2(x[2].x, x[3].x), C::pack2(x[4].x, x[5].x), C::pack2(x[6].x, x[7].x));
            sts128(at ^ (uint32_t)(32 + 16 * k), C::pack2(x[0].y, x[1].y), C::pack2(x[2].y, x[3].y), C::pack2(x[4].y, x[5].y), C::pack2(x[6].y, x[7].y));
        }
    } else if (width <= 8) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = i < width ? bits_value(type, raw.v[i]) : 0.0f;
        sts128(at, C::pack2(x[0], x[1]), C::pack2(x[2], x[3]), C::pack2(x[4], x[5]), C::pack2(x[6], x[7]));
        sts128(at ^ 16u, 0u, 0u, 0u, 0u);
    } else if (p.vec_in && type == MLP_F32) {
#pragma unroll 1
        for (int h = 0; h < IW; h += 32) {
            if (h >= width) break;
            const float4* src = (const float4*)src_row + h / 4;
            float4 x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = real && h + 4 * j < width ? __ldg(src + j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                sts128(at ^ (uint32_t)(2 * h + 16 * j), C::pack2(x[2 * j].x, x[2 * j].y), C::pack2(x[2 * j].z, x[2 * j].w), C::pack2(x[2 * j + 1].x, x[2 * j + 1].y),
                       C::pack2(x[2 * j + 1].z, x[2 * j + 1].w));
        }
    } else if (p.vec_in && type == FMT) {
        const uint4* src = (const uint4*)src_row;
        uint4 x[IW / 8];
#pragma unroll
        for (int j = 0; j < IW / 8; ++j) x[j] = real && 8 * j < width ? __ldg(src + j) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int j = 0; j < IW / 8; ++j) sts128(at ^ (uint32_t)(16 * j), x[j].x, x[j].y, x[j].z, x[j].w);
    } else {
        ragged_row<FMT, IW>(at, type, src_row, width, real);
    }
}

// Starts a row on its way into L2.
__device__ __forceinline__ void prefetch_row(const char* row) { asm volatile("prefetch.global.L2 [%0];" ::"l"(row)); }

// Four values of a sample's target row from feature f on (f a multiple of four); zero past its width.
__device__ __forceinline__ void load_targets(float (&t)[4], const Params& p, const char* row, int od, int f)
{
    const int dtype = p.cfg.target_dtype;
    if (p.vec_tgt) {   // rows are whole pieces of four values
        if (dtype == MLP_F32) {
            const float4 x = __ldg((const float4*)((const float*)row + f));
            t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
        } else {
            const uint2 x = __ldg((const uint2*)((const uint16_t*)row + f));
            t[0] = bits_value(dtype, x.x & 0xffffu);
            t[1] = bits_value(dtype, x.x >> 16);
            t[2] = bits_value(dtype, x.y & 0xffffu);
            t[3] = bits_value(dtype, x.y >> 16);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = bits_value(dtype, load_bits(row, dtype == MLP_F32, f + i, f + i < od));
    }
}

static __device__ __noinline__ float2 value_and_derivative(int act, float alpha, float z) { return make_float2(act_value(act, alpha, z), act_deriv(act, alpha, z)); }

// The output activation of four values and its derivative.
__device__ __forceinline__ void activate_outputs(int act, float alpha, float (&v)[4], float (&d)[4])
{
    if (act == MLP_ACT_IDENTITY) {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = 1.0f;
    } else if (act == MLP_ACT_SIGMOID) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float ex = expf(-fabsf(v[i]));
            v[i] = narrow::divide_by_1_to_2(v[i] >= 0.0f ? 1.0f : ex, 1.0f + ex);
            d[i] = v[i] * (1.0f - v[i]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 r = value_and_derivative(act, alpha, v[i]);
            v[i] = r.x;
            d[i] = r.y;
        }
    }
}

// Four output columns' accumulators plus bias, rounded, from output f on.
template <int FMT>
__device__ __forceinline__ void output_columns(float (&o)[4], uint32_t t_acc, uint32_t bias, int f)
{
    using C = Cvt<FMT>;
    uint32_t v[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(t_acc + (uint32_t)f) : "memory");
    const float4 b = narrow::lds_float4(bias + 4u * (uint32_t)f);
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3])::"memory");
    o[0] = C::round(__uint_as_float(v[0]) + b.x);
    o[1] = C::round(__uint_as_float(v[1]) + b.y);
    o[2] = C::round(__uint_as_float(v[2]) + b.z);
    o[3] = C::round(__uint_as_float(v[3]) + b.w);
}

// A row's hidden activations: 32 pre-activations rounded and activated, into the four chunks from `at` on (at: the first one's
// address, a multiple of four chunks in the row).  ReLU: the smallest magnitude seen goes to `least`.
template <int FMT, int HACT>
__device__ __forceinline__ void hidden_columns(const uint32_t (&v)[32], uint32_t at, float alpha, float& least)
{
    using C = Cvt<FMT>;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float z0 = __uint_as_float(v[8 * j + 2 * i]), z1 = __uint_as_float(v[8 * j + 2 * i + 1]);
            const uint32_t zp = C::pack2(z0, z1);
            if constexpr (HACT == MLP_ACT_RELU) {
                a[i] = C::relu2(zp);
                least = fminf(fminf(fabsf(z0), fabsf(z1)), least);
            } else {
                const float2 az = __ffma2_rn(make_float2(C::lo(zp), C::hi(zp)), make_float2(alpha, alpha), make_float2(0.0f, 0.0f));
                a[i] = C::max2(zp, C::pack2(az.x, az.y));
            }
        }
        sts128(at ^ (uint32_t)(16 * j), a[0], a[1], a[2], a[3]);
    }
}

// ReLU activations of a row in which a pre-activation rounds to zero, once more from the accumulator: those zeros are marked
// by the sign.  Rare, so kept small.
template <int FMT, int H>
__device__ __noinline__ void marked_columns(uint32_t t_acc, uint32_t row)
{
    using C = Cvt<FMT>;
    constexpr float kTiny = 0.5f * C::kSmallest;   // the largest magnitude that rounds to zero
#pragma unroll 1
    for (int j = 0; j < H / 8; ++j) {
        uint32_t v[8], a[4];
        tmem_ld_32x8(t_acc + (uint32_t)(8 * j), v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float z0 = __uint_as_float(v[2 * i]), z1 = __uint_as_float(v[2 * i + 1]);
            a[i] = C::relu2(C::pack2(z0, z1)) | (fabsf(z0) <= kTiny ? 0x8000u : 0u) | (fabsf(z1) <= kTiny ? 0x80000000u : 0u);
        }
        sts128(block_at<H>(row, j >> 2) ^ (uint32_t)(16 * (j & 3)), a[0], a[1], a[2], a[3]);
    }
}

// dZ = dA times the derivative, of the activations in the four chunks from `at` on.
template <int FMT, int HACT>
__device__ __forceinline__ void reverse_columns(uint32_t (&z)[16], const uint32_t (&v)[32], uint32_t at, float alpha_op)
{
    using C = Cvt<FMT>;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 act = narrow::lds128(at ^ (uint32_t)(16 * j));
        const uint32_t a[4] = {act.x, act.y, act.z, act.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float g0 = __uint_as_float(v[8 * j + 2 * i]), g1 = __uint_as_float(v[8 * j + 2 * i + 1]);
            if constexpr (HACT == MLP_ACT_RELU) {
                z[4 * j + i] = C::pack2(g0, g1) & C::positive_mask(a[i]);
            } else {
                const uint32_t neg = narrow::sign_mask(a[i]);
                const float2 ag = __fmul2_rn(make_float2(g0, g1), make_float2(alpha_op, alpha_op));
                z[4 * j + i] = (C::pack2(ag.x, ag.y) & neg) | (C::pack2(g0, g1) & ~neg);
            }
        }
    }
}

// Whether a row's dA holds an infinity or a NaN, from the first 32 features (halves) or of 32 features (bfloat16s).  An infinite or NaN
// dZ of the layer behind makes every feature so (times any weight, zero included, it is not finite), so the first one tells;
// from finite halves a sum of 128 products stays finite, of bfloat16s it can overflow, feature by feature.
template <int FMT>
__device__ __forceinline__ bool not_finite(const uint32_t (&v)[32])
{
    if constexpr (FMT == MLP_F16) {
        return (v[0] & 0x7f800000u) == 0x7f800000u;
    } else {
        float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 32; i += 2) s = __ffma2_rn(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), make_float2(0.0f, 0.0f), s);
        return !(s.x + s.y == 0.0f);
    }
}

// The same over a whole row, in place, where half of the gradient passes at marked zeros.  Width 128: as a product with the derivative, like the kernels
// of tc_kernels.cu, so that a dA that is not finite is NaN past a ReLU that is off; below that a ReLU that is off gives zero
// whatever comes, like the kernels of tc_narrow.cu.
template <int FMT, int H>
__device__ __noinline__ void reverse_whole_row(uint32_t t_acc, uint32_t row)
{
    using C = Cvt<FMT>;
#pragma unroll 1
    for (int j = 0; j < H / 8; ++j) {
        uint32_t v[8], z[4];
        tmem_ld_32x8(t_acc + (uint32_t)(8 * j), v);
        const uint32_t at = block_at<H>(row, j >> 2) ^ (uint32_t)(16 * (j & 3));
        const uint4 act = narrow::lds128(at);
        const uint32_t a[4] = {act.x, act.y, act.z, act.w};
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float g0 = __uint_as_float(v[2 * i]), g1 = __uint_as_float(v[2 * i + 1]);
            const uint32_t on = C::positive_mask(a[i]), zero = narrow::sign_mask(a[i]);
            if constexpr (H == 128) {
                const float d0 = (on & 1u) ? 1.0f : (zero & 1u) ? 0.5f : 0.0f, d1 = (on >> 31) ? 1.0f : (zero >> 31) ? 0.5f : 0.0f;
                z[i] = C::pack2(g0 * d0, g1 * d1);
            } else {
                z[i] = (C::pack2(g0, g1) & on) | (C::pack2(0.5f * g0, 0.5f * g1) & zero);
            }
        }
        sts128(at, z[0], z[1], z[2], z[3]);
    }
}

// Adds 4 N values to chunks first .. first + N - 1 of a row of fp32 sums at `at`, whose 16-byte chunks lie ^ (row % 8).
template <int N>
__device__ __forceinline__ void add_chunks(uint32_t at, int row, int first, const uint32_t* v)
{
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t chunk = at + (uint32_t)(16 * ((first + j) ^ (row & 7)));
        const float4 x = narrow::lds_float4(chunk);
        sts128(chunk, __float_as_uint(x.x + __uint_as_float(v[4 * j])), __float_as_uint(x.y + __uint_as_float(v[4 * j + 1])),
               __float_as_uint(x.z + __uint_as_float(v[4 * j + 2])), __float_as_uint(x.w + __uint_as_float(v[4 * j + 3])));
    }
}

}  // namespace chain
}  // namespace mlpb200
