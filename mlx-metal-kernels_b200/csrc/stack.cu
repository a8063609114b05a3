// Decode-layer glue between the matvec and attention kernels: split the fused QKV row, apply the
// interleaved-pair rotary embedding to q and k, and append the new token's k / v - quantised with
// the cache's own rule - to its page.
//
//   q_out[b, h, :]  = rope(qkv[b, h*D : (h+1)*D], pos[b])                          h < Hq
//   k = rope(qkv[b, (Hq + h)*D ...], pos[b]) ; v = qkv[b, (Hq + Hkv + h)*D ...]    h < Hkv
//   page = block_table[b, pos[b] / P], slot = pos[b] % P
//   per group of G along D: scale = max(max|v|, 1e-8) / (127 | 7) (fp32, stored fp16),
//                           code = clip(rint(v / scale), -127|-7, 127|7) + (128 | 8)
//
// RoPE follows the reference (ops/rope_ops.py:61-75): pairs (2i, 2i+1), cos/sin tables [S, D/2]
// in fp32, y_even = x_even*cos - x_odd*sin, y_odd = x_even*sin + x_odd*cos, rounded to fp16.
// The quantisation rule is _quantize_group_symmetric_8 / _4 of the reference cache
// (ops/paged_quantized_kv_ops.py:146-175); the reference itself has no append kernel (its update
// kernels copy the whole cache per token).
//
// One warp per (sequence, head); head_dim <= 128 and even; lanes own 4 consecutive elements.
#include "common.cuh"

#include <algorithm>

namespace b200q {

B200Q_DEFINE_STATUS_WORD(stack_read_status)

namespace {

struct RopeAppendParams {
    const __half* qkv;          // [B, (Hq + 2 Hkv) * D]
    const float* cos_table;     // [S, D/2]
    const float* sin_table;
    const int32_t* positions;   // [B]
    const int32_t* block_table; // [B, max_blocks]
    __half* q_out;              // [B, Hq, D]
    uint8_t* k_codes; uint8_t* v_codes;   // [num_pages, P, Hkv, D or D/2]
    __half* k_scales; __half* v_scales;   // [num_pages, P, Hkv, Gd]
    int B, Hq, Hkv, D, P, max_blocks, G, Gd, bits, table_len;
    int64_t num_pages;
};

__global__ void __launch_bounds__(128) rope_kv_append_kernel(const __grid_constant__ RopeAppendParams p) {
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int heads = p.Hq + 2 * p.Hkv;
    pdl_launch_dependents();
    pdl_wait();
    if (item >= p.B * heads) return;
    const int b = item / heads;
    const int hh = item - b * heads;
    const int pos = p.positions[b];
    const int d0 = lane * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    const bool live = d0 < p.D;
    if (live) {
        const uint2 u = *reinterpret_cast<const uint2*>(p.qkv + ((size_t)b * heads + hh) * p.D + d0);
        const __half2 h0 = *reinterpret_cast<const __half2*>(&u.x), h1 = *reinterpret_cast<const __half2*>(&u.y);
        v[0] = __low2float(h0); v[1] = __high2float(h0); v[2] = __low2float(h1); v[3] = __high2float(h1);
    }
    const bool is_v = hh >= p.Hq + p.Hkv;
    // a position outside the rotary table: the row passes through unrotated and the event is recorded
    if (!is_v && lane == 0 && (pos < 0 || pos >= p.table_len)) atomicMax(&g_device_status, (int)EV_ROPE_POSITION);
    if (!is_v && live && pos >= 0 && pos < p.table_len) {
        const int half_d = p.D / 2;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float c = p.cos_table[(size_t)pos * half_d + d0 / 2 + i];
            const float s = p.sin_table[(size_t)pos * half_d + d0 / 2 + i];
            const float xe = v[2 * i], xo = v[2 * i + 1];
            // two separately rounded products and one sum, as the reference's elementwise expression
            v[2 * i] = __fsub_rn(__fmul_rn(xe, c), __fmul_rn(xo, s));
            v[2 * i + 1] = __fadd_rn(__fmul_rn(xe, s), __fmul_rn(xo, c));
        }
    }
    // values as the cache / attention see them: rounded to fp16
    __half hv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { hv[i] = __float2half_rn(v[i]); v[i] = __half2float(hv[i]); }

    if (hh < p.Hq) {
        if (live) {
            uint2 o;
            o.x = (uint32_t)__half_as_ushort(hv[0]) | ((uint32_t)__half_as_ushort(hv[1]) << 16);
            o.y = (uint32_t)__half_as_ushort(hv[2]) | ((uint32_t)__half_as_ushort(hv[3]) << 16);
            *reinterpret_cast<uint2*>(p.q_out + ((size_t)b * p.Hq + hh) * p.D + d0) = o;
        }
        return;
    }
    // ---- k or v: quantise this head's row into its page slot ----
    const int hkv = is_v ? hh - p.Hq - p.Hkv : hh - p.Hq;
    const int blk = pos / p.P;
    int page = (pos >= 0 && blk < p.max_blocks) ? p.block_table[(size_t)b * p.max_blocks + blk] : -1;
    if (page < 0 || page >= p.num_pages) {                // unassigned page: nothing is written, the event is recorded
        if (lane == 0) atomicMax(&g_device_status, (int)EV_KV_PAGE_UNASSIGNED);
        return;
    }
    const int slot = pos % p.P;
    // group max over G elements = G/4 consecutive lanes (G a multiple of 4, power of two <= 128)
    float mx = live ? fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))) : 0.0f;
    const int lanes_per_group = p.G / 4;
    for (int o = 1; o < lanes_per_group; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float limit = p.bits == 8 ? 127.0f : 7.0f;
    const float offset = p.bits == 8 ? 128.0f : 8.0f;
    const float scale = __fdiv_rn(fmaxf(mx, 1e-8f), limit);
    uint32_t codes[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float qv = fminf(fmaxf(rintf(__fdiv_rn(v[i], scale)), -limit), limit) + offset;
        codes[i] = (uint32_t)(int)qv;
    }
    const size_t tok = ((size_t)page * p.P + slot) * p.Hkv + hkv;
    uint8_t* cdst = is_v ? p.v_codes : p.k_codes;
    __half* sdst = is_v ? p.v_scales : p.k_scales;
    if (live) {
        if (p.bits == 8) {
            const uint32_t w = codes[0] | (codes[1] << 8) | (codes[2] << 16) | (codes[3] << 24);
            *reinterpret_cast<uint32_t*>(cdst + tok * p.D + d0) = w;
        } else {
            const uint16_t w = (uint16_t)(codes[0] | (codes[1] << 4) | (codes[2] << 8) | (codes[3] << 12));
            *reinterpret_cast<uint16_t*>(cdst + tok * (p.D / 2) + d0 / 2) = w;
        }
        if ((lane % lanes_per_group) == 0) sdst[tok * p.Gd + d0 / p.G] = __float2half_rn(scale);
    }
}

// Symmetric group-wise quantisation of [rows, D] values with the cache rule above, for every row and group size the
// 16-byte kernel below does not take: one thread per (row, group) (per row when the group size is odd, so that a packed byte never straddles two threads).
template <typename T>
__global__ void __launch_bounds__(256) quantize_kv_kernel(const T* __restrict__ values, uint8_t* __restrict__ codes,
                                                          __half* __restrict__ scales, int64_t rows, int D, int G, int Gd,
                                                          int bits, bool per_row) {
    const int64_t items = per_row ? rows : rows * Gd;
    const float limit = bits == 8 ? 127.0f : 7.0f;
    const float offset = bits == 8 ? 128.0f : 8.0f;
    const int dp = bits == 4 ? (D + 1) / 2 : D;
    for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < items; it += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = per_row ? it : it / Gd;
        const int g_lo = per_row ? 0 : (int)(it - row * Gd);
        const int g_hi = per_row ? Gd : g_lo + 1;
        const T* src = values + row * D;
        uint8_t* dst = codes + row * dp;
        for (int g = g_lo; g < g_hi; ++g) {
            const int d_lo = g * G, d_hi = min(D, d_lo + G);
            float mx = 0.0f;
            for (int d = d_lo; d < d_hi; ++d) mx = fmaxf(mx, fabsf(to_f32(src[d])));
            const float scale = __fdiv_rn(fmaxf(mx, 1e-8f), limit);
            scales[row * Gd + g] = __float2half_rn(scale);
            for (int d = d_lo; d < d_hi; ++d) {
                const float qv = fminf(fmaxf(rintf(__fdiv_rn(to_f32(src[d]), scale)), -limit), limit) + offset;
                const uint32_t c = (uint32_t)(int)qv;
                if (bits == 8) {
                    dst[d] = (uint8_t)c;
                } else if (d & 1) {
                    dst[d >> 1] = (uint8_t)(dst[d >> 1] | (c << 4));     // the low nibble was written just before by this thread
                } else {
                    dst[d >> 1] = (uint8_t)c;                            // high nibble zero (stays zero for an odd D)
                }
            }
        }
    }
}

// The same rule on whole 16-byte pieces, and its inverse.  Rows whose groups are whole (D a multiple of G) are one flat
// run of groups, so a thread takes 8 consecutive values wherever they lie: one 16-byte load, the group's maximum over the
// G/8 neighbouring lanes, one 8-byte (q8) or 4-byte (q4) store.  The kernel is bound by HBM (2 bytes in, 1 or 1/2 out per
// value); four pieces per thread are in flight.  K and V go in one launch (blockIdx.y).  Against one thread per group of
// strided 2-byte loads and byte stores, quantising 2 x 33.5 M fp16 values to q8 groups of 32 and reading them back: 646 -> 71 us
// (the copies and the general dequantiser on the way back included).
constexpr int kVecPerThread = 4;
struct KvPair {
    const void* in[2];
    void* out[2];
    void* scales[2];      // written by the quantiser, read by the dequantiser
};

// largest magnitude of 8 packed values; a NaN among them is passed on
template <typename T> __device__ __forceinline__ float max_abs8(const uint4& u);
template <> __device__ __forceinline__ float max_abs8<__half>(const uint4& u) {
    const __half2* h = reinterpret_cast<const __half2*>(&u);
    const __half2 m = __hmax2_nan(__hmax2_nan(__habs2(h[0]), __habs2(h[1])), __hmax2_nan(__habs2(h[2]), __habs2(h[3])));
    return __half2float(__hmax_nan(__low2half(m), __high2half(m)));
}
template <> __device__ __forceinline__ float max_abs8<__nv_bfloat16>(const uint4& u) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    const __nv_bfloat162 m = __hmax2_nan(__hmax2_nan(__habs2(h[0]), __habs2(h[1])), __hmax2_nan(__habs2(h[2]), __habs2(h[3])));
    return __bfloat162float(__hmax_nan(__low2bfloat16(m), __high2bfloat16(m)));
}

// What bounds the quantiser is instructions (issue slots 81 % busy at 12 per value, 51.6 us for 67 M values; HBM would take 32): hence
// the maximum on packed pairs, one reciprocal per piece, two fused multiply-adds per value for code and distance to a tie,
// and byte permutes for the packing.
template <typename T, int BITS>
__global__ void __launch_bounds__(256) quantize_kv_vec_kernel(const __grid_constant__ KvPair p, int64_t pieces, int log_lanes) {
    const T* in = reinterpret_cast<const T*>(p.in[blockIdx.y]);
    __half* scales = reinterpret_cast<__half*>(p.scales[blockIdx.y]);
    const int64_t first = (int64_t)blockIdx.x * (256 * kVecPerThread) + threadIdx.x;
    uint4 u[kVecPerThread];
#pragma unroll
    for (int j = 0; j < kVecPerThread; ++j) {
        const int64_t i = first + j * 256;
        u[j] = i < pieces ? __ldcs(reinterpret_cast<const uint4*>(in) + i) : make_uint4(0u, 0u, 0u, 0u);
    }
    constexpr float limit = BITS == 8 ? 127.0f : 7.0f;
    constexpr float offset = BITS == 8 ? 128.0f : 8.0f;
    constexpr float magic = 12582912.0f + offset;          // 1.5 2^23: adding it rounds to nearest even and leaves the code in the low byte
#pragma unroll
    for (int j = 0; j < kVecPerThread; ++j) {
        const int64_t i = first + j * 256;
        const T* e = reinterpret_cast<const T*>(&u[j]);
        float v[8], mx = max_abs8<T>(u[j]);                // NaN when a value is
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = to_f32(e[k]);
        const bool plain = __all_sync(0xffffffffu, mx < 3e38f);
        if (!plain) {                                      // the maximum of what is a number, as the rule has it
            mx = 0.0f;
            for (int k = 0; k < 8; ++k) mx = fmaxf(mx, fabsf(v[k]));
        }
        for (int o = 1; o < (1 << log_lanes); o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float scale = __fdiv_rn(fmaxf(mx, 1e-8f), limit);
        // rint(v / scale) through the reciprocal: v * inv differs from the correctly rounded quotient by less than 2^-14 (|quotients|
        // stay below 128), so it rounds to the same integer unless it lies that close to a tie.  Pieces with a value near a tie,
        // and warps with one that is not finite, are done by division.
        const float inv = __fdividef(1.0f, scale);
        uint32_t c[8];
        float far = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float r = fmaf(v[k], inv, magic);
            far = fmaxf(far, fabsf(fmaf(v[k], inv, magic - r)));
            c[k] = __float_as_uint(r);
        }
        if (!plain || far > 0.4999f) {
#pragma unroll
            for (int k = 0; k < 8; ++k) c[k] = (uint32_t)(int)(fminf(fmaxf(rintf(__fdiv_rn(v[k], scale)), -limit), limit) + offset);
        }
        if (i >= pieces) continue;
        auto bytes = [](uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) { return prmt(prmt(c0, c1, 0x0040u), prmt(c2, c3, 0x0040u), 0x5410u); };
        if (BITS == 8) {
            reinterpret_cast<uint2*>(p.out[blockIdx.y])[i] = make_uint2(bytes(c[0], c[1], c[2], c[3]), bytes(c[4], c[5], c[6], c[7]));
        } else {
            reinterpret_cast<uint32_t*>(p.out[blockIdx.y])[i] = bytes(c[0], c[2], c[4], c[6]) | bytes(c[1], c[3], c[5], c[7]) << 4;
        }
        if ((i & ((1 << log_lanes) - 1)) == 0) scales[i >> log_lanes] = __float2half_rn(scale);
    }
}

// out = fp16((code - offset) * |scale|): code - offset is exact in fp16 and the product is rounded once, which is what
// the two fp32 operations and the cast of the reference give.
template <int BITS>
__global__ void __launch_bounds__(256) dequantize_kv_vec_kernel(const __grid_constant__ KvPair p, int64_t pieces, int log_lanes) {
    const __half* scales = reinterpret_cast<const __half*>(p.scales[blockIdx.y]);
    const int64_t first = (int64_t)blockIdx.x * (256 * kVecPerThread) + threadIdx.x;
    uint2 u[kVecPerThread];
    uint32_t s2[kVecPerThread];
#pragma unroll
    for (int j = 0; j < kVecPerThread; ++j) {
        const int64_t i = first + j * 256;
        u[j] = make_uint2(0u, 0u);
        s2[j] = 0u;
        if (i >= pieces) continue;
        if (BITS == 8) u[j] = __ldcs(reinterpret_cast<const uint2*>(p.in[blockIdx.y]) + i);
        else u[j].x = __ldcs(reinterpret_cast<const uint32_t*>(p.in[blockIdx.y]) + i);
        s2[j] = half_dup(__habs(scales[i >> log_lanes]));
    }
#pragma unroll
    for (int j = 0; j < kVecPerThread; ++j) {
        const int64_t i = first + j * 256;
        if (i >= pieces) continue;
        uint32_t h[4];
        if (BITS == 8) {
            h[0] = hmul2_u32(hsub2_u32(prmt(u[j].x, 0x64646464u, 0x4140u), 0x64806480u), s2[j]);
            h[1] = hmul2_u32(hsub2_u32(prmt(u[j].x, 0x64646464u, 0x4342u), 0x64806480u), s2[j]);
            h[2] = hmul2_u32(hsub2_u32(prmt(u[j].y, 0x64646464u, 0x4140u), 0x64806480u), s2[j]);
            h[3] = hmul2_u32(hsub2_u32(prmt(u[j].y, 0x64646464u, 0x4342u), 0x64806480u), s2[j]);
        } else {
            // nibbles (0,4) (1,5) (2,6) (3,7) as halves, then back into order
            uint32_t q[4];
            const uint32_t w = u[j].x, w2 = w >> 8;
            q[0] = hmul2_u32(hsub2_u32(lop3_and_or(w, 0x000F000Fu, 0x64006400u), 0x64086408u), s2[j]);
            q[1] = hmul2_u32(hsub2_u32(lop3_and_or(w, 0x00F000F0u, 0x54005400u), 0x54805480u), s2[j]);
            q[2] = hmul2_u32(hsub2_u32(lop3_and_or(w2, 0x000F000Fu, 0x64006400u), 0x64086408u), s2[j]);
            q[3] = hmul2_u32(hsub2_u32(lop3_and_or(w2, 0x00F000F0u, 0x54005400u), 0x54805480u), s2[j]);
            h[0] = prmt(q[0], q[1], 0x5410);
            h[1] = prmt(q[2], q[3], 0x5410);
            h[2] = prmt(q[0], q[1], 0x7632);
            h[3] = prmt(q[2], q[3], 0x7632);
        }
        __stcs(reinterpret_cast<uint4*>(p.out[blockIdx.y]) + i, make_uint4(h[0], h[1], h[2], h[3]));
    }
}

}  // namespace

// log2 of the lanes that share a group when the 16-byte kernels above apply: whole groups of 8, 16, ... 256 values, aligned
// buffers; else -1.
static int vec_group_lanes(int D, int G, int bits, const KvPair& p, bool quantize) {
    if (D % G != 0 || G < 8 || G > 256 || (G & (G - 1)) != 0) return -1;
    const uintptr_t coded = bits == 8 ? 7u : 3u;
    for (int i = 0; i < 2; ++i) {
        if (p.in[i] == nullptr) continue;
        const uintptr_t values = (uintptr_t)(quantize ? p.in[i] : p.out[i]), codes = (uintptr_t)(quantize ? p.out[i] : p.in[i]);
        if ((values & 15u) != 0 || (codes & coded) != 0) return -1;
    }
    int lanes = 0;
    while ((8 << lanes) < G) ++lanes;
    return lanes;
}

int quantize_kv_impl(int bits, const void* values, uint8_t* codes, void* scales, int64_t rows, int D, int group_size,
                     int in_dtype, cudaStream_t stream);

// K and V of the same shape in one launch (v may be null).
int quantize_kv_pair_impl(int bits, const void* k, const void* v, uint8_t* k_codes, uint8_t* v_codes, void* k_scales, void* v_scales,
                          int64_t rows, int D, int group_size, int in_dtype, cudaStream_t stream) {
    if ((bits != 4 && bits != 8) || k == nullptr || k_codes == nullptr || k_scales == nullptr ||
        (v != nullptr && (v_codes == nullptr || v_scales == nullptr)))
        return B200Q_ERR_BAD_ARG;
    if (rows <= 0 || D <= 0 || group_size <= 0 || !is_act_dtype(in_dtype)) return B200Q_ERR_BAD_ARG;
    const KvPair p = {{k, v}, {k_codes, v_codes}, {k_scales, v_scales}};
    const int lanes = vec_group_lanes(D, group_size, bits, p, true);
    if (lanes < 0) {
        const int rc = quantize_kv_impl(bits, k, k_codes, k_scales, rows, D, group_size, in_dtype, stream);
        if (rc != B200Q_OK || v == nullptr) return rc;
        return quantize_kv_impl(bits, v, v_codes, v_scales, rows, D, group_size, in_dtype, stream);
    }
    const int64_t pieces = rows * D / 8, blocks = (pieces + 256 * kVecPerThread - 1) / (256 * kVecPerThread);
    if (blocks > INT32_MAX) return B200Q_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)blocks, v == nullptr ? 1 : 2);
    if (in_dtype == B200Q_F16) {
        if (bits == 8) quantize_kv_vec_kernel<__half, 8><<<grid, 256, 0, stream>>>(p, pieces, lanes);
        else quantize_kv_vec_kernel<__half, 4><<<grid, 256, 0, stream>>>(p, pieces, lanes);
    } else {
        if (bits == 8) quantize_kv_vec_kernel<__nv_bfloat16, 8><<<grid, 256, 0, stream>>>(p, pieces, lanes);
        else quantize_kv_vec_kernel<__nv_bfloat16, 4><<<grid, 256, 0, stream>>>(p, pieces, lanes);
    }
    return finish_launch();
}

// The inverse, fp16 out and fp16 scales; B200Q_ERR_UNSUPPORTED for groups the 16-byte kernel does not take (callers then
// use b200q_dequant with the offset as zero points).
int dequantize_kv_pair_impl(int bits, const uint8_t* k_codes, const uint8_t* v_codes, const void* k_scales, const void* v_scales, void* k,
                            void* v, int64_t rows, int D, int group_size, cudaStream_t stream) {
    if ((bits != 4 && bits != 8) || k == nullptr || k_codes == nullptr || k_scales == nullptr ||
        (v_codes != nullptr && (v == nullptr || v_scales == nullptr)))
        return B200Q_ERR_BAD_ARG;
    if (rows <= 0 || D <= 0 || group_size <= 0) return B200Q_ERR_BAD_ARG;
    const KvPair p = {{k_codes, v_codes}, {k, v}, {const_cast<void*>(k_scales), const_cast<void*>(v_scales)}};
    const int lanes = vec_group_lanes(D, group_size, bits, p, false);
    if (lanes < 0) return B200Q_ERR_UNSUPPORTED;
    const int64_t pieces = rows * D / 8, blocks = (pieces + 256 * kVecPerThread - 1) / (256 * kVecPerThread);
    if (blocks > INT32_MAX) return B200Q_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)blocks, v_codes == nullptr ? 1 : 2);
    if (bits == 8) dequantize_kv_vec_kernel<8><<<grid, 256, 0, stream>>>(p, pieces, lanes);
    else dequantize_kv_vec_kernel<4><<<grid, 256, 0, stream>>>(p, pieces, lanes);
    return finish_launch();
}

int quantize_kv_impl(int bits, const void* values, uint8_t* codes, void* scales, int64_t rows, int D, int group_size,
                     int in_dtype, cudaStream_t stream) {
    if ((bits != 4 && bits != 8) || values == nullptr || codes == nullptr || scales == nullptr) return B200Q_ERR_BAD_ARG;
    if (rows <= 0 || D <= 0 || group_size <= 0 || !is_act_dtype(in_dtype)) return B200Q_ERR_BAD_ARG;
    const int Gd = (D + group_size - 1) / group_size;
    const bool per_row = bits == 4 && (group_size & 1);
    const int64_t items = per_row ? rows : rows * Gd;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, (int64_t)sm_count() * 16));
    if (in_dtype == B200Q_F16)
        quantize_kv_kernel<__half><<<grid, 256, 0, stream>>>((const __half*)values, codes, (__half*)scales, rows, D, group_size,
                                                            Gd, bits, per_row);
    else
        quantize_kv_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)values, codes, (__half*)scales, rows,
                                                                   D, group_size, Gd, bits, per_row);
    return finish_launch();
}

int rope_kv_append_impl(const void* qkv, const float* cos_table, const float* sin_table, const int32_t* positions,
                        const int32_t* block_table, void* q_out, uint8_t* k_codes, uint8_t* v_codes, void* k_scales,
                        void* v_scales, int bits, int B, int Hq, int Hkv, int D, int page_size, int64_t num_pages,
                        int max_blocks, int group_size, int table_len, cudaStream_t stream) {
    if (qkv == nullptr || cos_table == nullptr || sin_table == nullptr || positions == nullptr || block_table == nullptr ||
        q_out == nullptr || k_codes == nullptr || v_codes == nullptr || k_scales == nullptr || v_scales == nullptr)
        return B200Q_ERR_BAD_ARG;
    if ((bits != 4 && bits != 8) || B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || page_size <= 0 || num_pages <= 0 ||
        max_blocks <= 0 || group_size <= 0 || table_len <= 0)
        return B200Q_ERR_BAD_ARG;
    if (D > 128 || D % 4 != 0 || group_size % 4 != 0 || (group_size & (group_size - 1)) != 0 || group_size > 128 ||
        D % group_size != 0)
        return B200Q_ERR_UNSUPPORTED;
    RopeAppendParams p = {};
    p.qkv = (const __half*)qkv; p.cos_table = cos_table; p.sin_table = sin_table; p.positions = positions;
    p.block_table = block_table; p.q_out = (__half*)q_out; p.k_codes = k_codes; p.v_codes = v_codes;
    p.k_scales = (__half*)k_scales; p.v_scales = (__half*)v_scales;
    p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.P = page_size; p.max_blocks = max_blocks; p.G = group_size;
    p.Gd = D / group_size; p.bits = bits; p.table_len = table_len; p.num_pages = num_pages;
    const int warps = 4;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((B * (Hq + 2 * Hkv) + warps - 1) / warps);
    cfg.blockDim = dim3(warps * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning_get("no_pdl") ? 0 : 1;
    if (cudaLaunchKernelEx(&cfg, rope_kv_append_kernel, p) != cudaSuccess) return B200Q_ERR_LAUNCH;
    return finish_launch();
}

}  // namespace b200q
