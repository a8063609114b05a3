// One warp, one kv head, one page of 16 tokens of head_dim 128: the building blocks of the paged decode attention kernels, for
// quantised pages (q4 / q8 codes, symmetric fp16 scales per token and group) and for plain fp16 / bf16 pages.
//
// A page of q4 codes is 2.3 KB per kv head and an SM receives one every 100 clocks at the HBM rate, so the instructions per page
// decide.  (The form before this one dequantised K and V to fp16 with three operations per pair and took 591 warp
// instructions per page and kv head; it ran at 58 % issue and 0.27 of the DRAM rate.)
//   * copies: tensor copies put a page down token-major and swizzled, so that ldmatrix meets no bank conflicts.
//   * S = K Q^T: ldmatrix hands every lane the word of its token row; code - offset as exact fp16 integers takes two operations per
//     pair, the queries enter as they are, and the scale is applied once per token and group in fp32.  So neither side is rounded.
//     (The form before multiplied raw codes in u8 x s8 with queries in two signed bytes.  It saved these operations but rounded every
//     query at 2^-16 of its head's largest: with one channel 100 times the rest and K zero there the result's relative error was
//     9.2e-4 instead of 2.8e-4.  One column per head instead of two and no accumulator start values make up for the operations:
//     16 x 8192 tokens, 8 kv heads, groups of 8: q4 77.8 -> 51.3 us, q8 77.4 -> 59.9; groups of 4: q4 42.3 -> 44.0, 32 x 4096
//     q8 54.7 -> 54.4.)
//   * softmax: a lane holds one head (two when there are more than four query heads per kv head) of tokens g and g + 8.  The
//     reference maximum only moves when a score exceeds it by 2^8, decided by one vote per page; no shuffles otherwise.
//   * O^T += V^T P: ldmatrix.trans delivers the codes of two tokens side by side, exact fp16 code - offset takes two operations per
//     pair, and the scales are folded into the probabilities, (p * scale) rounded once to fp16 as an operand column
//     per scale group.  Plain pages need no arithmetic; there the spare columns carry the rounding remainder of p.
#pragma once

#include "common.cuh"

namespace b200q {
namespace attn {

constexpr int kHeadDim = 128;
constexpr float kLog2e = 1.4426950408889634f;

// BITS: 4, 8 (codes) or 16 (plain).  LOGG: log2 of the scale group, 5 or 6; for plain pages 0 = fp16, 1 = bf16.
template <int BITS> struct PageShape {
    static constexpr int ROW = kHeadDim * BITS / 8;        // bytes of one token row of one kv head
    static constexpr int TILE = 16 * ROW;                  // K (or V) bytes of a page
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ void lds64(uint32_t (&r)[2], uint32_t a) {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <bool BF>
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    } else {
        mma_m16n8k16(d, a0, a1, a2, a3, b0, b1);
    }
}
__device__ __forceinline__ float half_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
__device__ __forceinline__ float half_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// code - offset as exact halves: the nibbles (0, 4) (1, 5) (2, 6) (3, 7) of a q4 word; two bytes of a q8 word
__device__ __forceinline__ void q4_values(uint32_t w, uint32_t (&v)[4]) {
    const uint32_t w8 = w >> 8;
    v[0] = hsub2_u32(lop3_and_or(w, 0x000F000Fu, 0x64006400u), 0x64086408u);
    v[1] = hsub2_u32(lop3_and_or(w, 0x00F000F0u, 0x54005400u), 0x54805480u);
    v[2] = hsub2_u32(lop3_and_or(w8, 0x000F000Fu, 0x64006400u), 0x64086408u);
    v[3] = hsub2_u32(lop3_and_or(w8, 0x00F000F0u, 0x54005400u), 0x54805480u);
}
__device__ __forceinline__ uint32_t q8_values(uint32_t w, uint32_t sel) { return hsub2_u32(prmt(w, 0x64646464u, sel), 0x64806480u); }

// WIDE: five to eight query heads per kv head.  ST: heads ("streams") a lane holds: head t, and head 4 + t when WIDE.
template <int BITS, bool WIDE> struct WarpState {
    static constexpr int ST = WIDE ? 2 : 1;
    uint32_t qb[8][2];          // queries as B operand, per mma
    float qs[ST];               // factor of the scores: softmax scale * log2(e) (bf16 queries of codes: and their power of two)
    float m[ST], l[ST];         // reference maximum (log2 units), this lane's share of the sum
    float vk;                   // power of two on the V scales inside the probabilities
    float o[8][4];              // O^T tiles; see out_value()
};
template <int BITS, bool WIDE>
__device__ __forceinline__ void state_reset(WarpState<BITS, WIDE>& a) {
#pragma unroll
    for (int s = 0; s < WarpState<BITS, WIDE>::ST; ++s) { a.m[s] = -INFINITY; a.l[s] = 0.0f; }
    a.vk = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) a.o[i][e] = 0.0f;
}

// Queries of one kv head's group: row r of `rows` (128 values apart) is query head r (r < group <= 8).  Shared or global memory.
template <int BITS, int LOGG, bool WIDE>
__device__ __forceinline__ void load_queries(WarpState<BITS, WIDE>& a, const void* rows, int group, int dtype, float sm_scale, int lane) {
    constexpr int ST = WarpState<BITS, WIDE>::ST;
    const int g = lane >> 2, t = lane & 3;
    const uint16_t* q = reinterpret_cast<const uint16_t*>(rows);
    // column 2h is head h, column 2h + 1 head 4 + h (when WIDE): this lane feeds column g
    const int head = (g >> 1) + ((g & 1) ? 4 : 0);
    const bool live = ((g & 1) == 0 || WIDE) && head < group;
    const uint16_t* row = q + (size_t)head * kHeadDim;
#pragma unroll
    for (int s = 0; s < ST; ++s) a.qs[s] = sm_scale * kLog2e;
    if constexpr (BITS == 16) {
#pragma unroll
        for (int s = 0; s < 8; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) a.qb[s][h] = live ? *reinterpret_cast<const uint32_t*>(row + 16 * s + 8 * h + 2 * t) : 0u;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {                      // 32 dims, two mma
            if constexpr (BITS == 4) {
                // d = 8t .. 8t + 7 of the 32, in the order in which the masks take the nibbles of a word: (0, 4) (1, 5) (2, 6) (3, 7)
                const uint4 u = live ? *reinterpret_cast<const uint4*>(row + 32 * i + 8 * t) : make_uint4(0u, 0u, 0u, 0u);
                a.qb[2 * i][0] = prmt(u.x, u.z, 0x5410);
                a.qb[2 * i][1] = prmt(u.x, u.z, 0x7632);
                a.qb[2 * i + 1][0] = prmt(u.y, u.w, 0x5410);
                a.qb[2 * i + 1][1] = prmt(u.y, u.w, 0x7632);
            } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {              // d = 4t .. 4t + 3 of 16
                    const uint2 u = live ? *reinterpret_cast<const uint2*>(row + 32 * i + 16 * c + 4 * t) : make_uint2(0u, 0u);
                    a.qb[2 * i + c][0] = u.x;
                    a.qb[2 * i + c][1] = u.y;
                }
            }
        }
        if (dtype != B200Q_F16) {
            // bf16 queries in fp16: a power of two brings the head's largest element to [2^13, 2^14); bf16 has 8 significant bits, so all
            // within 2^-30 of the largest are exact
            uint32_t mx = 0u;
#pragma unroll
            for (int s = 0; s < 8; ++s)
#pragma unroll
                for (int h = 0; h < 2; ++h) mx = max(mx, max(a.qb[s][h] & 0x7FFFu, (a.qb[s][h] >> 16) & 0x7FFFu));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const uint32_t e = max(mx >> 7, 14u);
            const float up = __uint_as_float((267u - e) << 23), down = __uint_as_float((e - 13u) << 23);      // 2^(140 - e) and its inverse
#pragma unroll
            for (int s = 0; s < 8; ++s)
#pragma unroll
                for (int h = 0; h < 2; ++h) a.qb[s][h] = pack_h2(__uint_as_float(a.qb[s][h] << 16) * up, __uint_as_float(a.qb[s][h] & 0xFFFF0000u) * up);
            // as accumulator owner this lane holds columns 2t, 2t + 1
#pragma unroll
            for (int s = 0; s < ST; ++s) a.qs[s] *= __shfl_sync(0xffffffffu, down, 8 * t + 4 * s);
        }
    }
}

// Where process_page finds a page: tiles [16 tokens][row] that a tensor copy put down (rows of 64 or 128 bytes swizzled by the copy,
// plain rows as two halves of 128 bytes) and scales [16 tokens][heads] of K, then of V.
struct PageRead {
    uint32_t rd;                      // ldmatrix row address inside a tile, first pair of chunks
    uint32_t sc, sc8, scv;            // scales of token g; distances to token g + 8 and to V's
};
template <int BITS>
__device__ __forceinline__ PageRead box_read(int lane, int head, int heads, int Gd) {
    const int up = lane >> 4, row = (lane & 7) + ((lane >> 3) & 1) * 8;
    PageRead R;
    R.rd = BITS == 4 ? (uint32_t)row * 64 + (uint32_t)((up ^ ((row >> 1) & 3)) << 4) : (uint32_t)row * 128 + (uint32_t)((up ^ (row & 7)) << 4);
    R.sc = (uint32_t)(((lane >> 2) * heads + head) * Gd * 2);
    R.sc8 = (uint32_t)(8 * heads * Gd * 2);
    R.scv = 2 * R.sc8;
    return R;
}
// ldmatrix address of chunks 2c, 2c + 1
template <int BITS>
__device__ __forceinline__ uint32_t chunk_pair(uint32_t rd, int c) {
    return (rd ^ (uint32_t)(((2 * c) & 7) << 4)) + (BITS == 16 ? (uint32_t)(c >> 2) * 2048 : 0u);
}

// One page: its K and V tile and its scales in shared memory; `attended` = bit mask of the token slots that take part (at least one).
template <int BITS, int LOGG, bool WIDE>
__device__ __forceinline__ void process_page(WarpState<BITS, WIDE>& a, uint32_t k_tile, uint32_t v_tile, uint32_t scales, const PageRead& R, uint32_t attended, int lane) {
    constexpr int ST = WarpState<BITS, WIDE>::ST;
    constexpr bool BF = BITS == 16 && LOGG == 1;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t kr = k_tile + R.rd, vr = v_tile + R.rd;
    const bool in0 = (attended >> g) & 1u, in1 = (attended >> (g + 8)) & 1u;

    // ---------------- scores of tokens g, g + 8 ----------------
    float s[ST][2];
    float vs[2][4];                                        // V scales of the two tokens, per 32 dims
    if constexpr (BITS == 16) {
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t r[4];
            ldsm4(r, chunk_pair<BITS>(kr, i));
            mma_f16<BF>(c, r[0], r[1], r[2], r[3], a.qb[i][0], a.qb[i][1]);
        }
        s[0][0] = c[0] * a.qs[0];
        s[0][1] = c[2] * a.qs[0];
        if constexpr (WIDE) { s[ST - 1][0] = c[1] * a.qs[0]; s[ST - 1][1] = c[3] * a.qs[0]; }
    } else {
        uint32_t ks0[2], ks1[2], vs0[2], vs1[2];
        const uint32_t sc = scales + R.sc;
        if (LOGG == 6) {                            // two scales per token and head
            ks0[0] = lds32(sc); ks1[0] = lds32(sc + R.sc8); vs0[0] = lds32(sc + R.scv); vs1[0] = lds32(sc + R.scv + R.sc8);
            ks0[1] = ks1[1] = vs0[1] = vs1[1] = 0u;
        } else {
            lds64(ks0, sc); lds64(ks1, sc + R.sc8); lds64(vs0, sc + R.scv); lds64(vs1, sc + R.scv + R.sc8);
        }
        float acc[ST][2];
#pragma unroll
        for (int x = 0; x < ST; ++x) acc[x][0] = acc[x][1] = 0.0f;
        float c[4];
        uint32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (LOGG == 5 || i % 2 == 0) c[0] = c[1] = c[2] = c[3] = 0.0f;
            if constexpr (BITS == 4) {
                if (i % 2 == 0) ldsm4(r, chunk_pair<BITS>(kr, i / 2));
                uint32_t x[4], y[4];
                q4_values(r[(i & 1) * 2], x);
                q4_values(r[(i & 1) * 2 + 1], y);
                mma_m16n8k16(c, x[0], y[0], x[1], y[1], a.qb[2 * i][0], a.qb[2 * i][1]);
                mma_m16n8k16(c, x[2], y[2], x[3], y[3], a.qb[2 * i + 1][0], a.qb[2 * i + 1][1]);
            } else {
                ldsm4(r, chunk_pair<BITS>(kr, i));
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t x = r[2 * h], y = r[2 * h + 1];
                    mma_m16n8k16(c, q8_values(x, 0x4140u), q8_values(y, 0x4140u), q8_values(x, 0x4342u), q8_values(y, 0x4342u), a.qb[2 * i + h][0], a.qb[2 * i + h][1]);
                }
            }
            if (LOGG == 5 || i % 2 == 1) {
                const int gi = LOGG == 5 ? i : i / 2;
                const uint32_t k0 = ks0[gi / 2] & 0x7FFF7FFFu, k1 = ks1[gi / 2] & 0x7FFF7FFFu;
                const float f0 = (gi & 1) ? half_hi(k0) : half_lo(k0), f1 = (gi & 1) ? half_hi(k1) : half_lo(k1);
#pragma unroll
                for (int x = 0; x < ST; ++x) {
                    acc[x][0] = fmaf(f0, c[x], acc[x][0]);
                    acc[x][1] = fmaf(f1, c[2 + x], acc[x][1]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < ST; ++x) { s[x][0] = acc[x][0] * a.qs[x]; s[x][1] = acc[x][1] * a.qs[x]; }
        if (attended != 0xFFFFu) {                         // masked slots may hold anything
            if (!in0) vs0[0] = vs0[1] = 0u;
            if (!in1) vs1[0] = vs1[1] = 0u;
        }
#pragma unroll
        for (int w = 0; w < (LOGG == 5 ? 2 : 1); ++w) {
            vs0[w] &= 0x7FFF7FFFu; vs1[w] &= 0x7FFF7FFFu;
            constexpr int R = LOGG == 5 ? 1 : 2;           // 32-dim blocks per scale
#pragma unroll
            for (int q = 0; q < R; ++q) {
                vs[0][2 * w * R + q] = half_lo(vs0[w]); vs[0][(2 * w + 1) * R + q] = half_hi(vs0[w]);
                vs[1][2 * w * R + q] = half_lo(vs1[w]); vs[1][(2 * w + 1) * R + q] = half_hi(vs1[w]);
            }
        }
    }
    if (attended != 0xFFFFu) {
#pragma unroll
        for (int x = 0; x < ST; ++x) {
            s[x][0] = in0 ? s[x][0] : -INFINITY;
            s[x][1] = in1 ? s[x][1] : -INFINITY;
        }
    }
    // ---------------- reference maximum: moves only when a score passes it by 2^8 (or a V scale its range) ----------------
    bool move = false;
#pragma unroll
    for (int x = 0; x < ST; ++x) move = move || fmaxf(s[x][0], s[x][1]) > a.m[x] + 8.0f;
    float vmax = 0.0f;
    if constexpr (BITS != 16) {
        vmax = fmaxf(fmaxf(fmaxf(vs[0][0], vs[0][1]), fmaxf(vs[0][2], vs[0][3])), fmaxf(fmaxf(vs[1][0], vs[1][1]), fmaxf(vs[1][2], vs[1][3])));
        move = move || vmax * a.vk > 128.0f;
    }
    if (__any_sync(0xffffffffu, move)) {
        float f[ST];
#pragma unroll
        for (int x = 0; x < ST; ++x) {
            float mx = fmaxf(s[x][0], s[x][1]);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float mn = fmaxf(a.m[x], mx);
            f[x] = ex2(a.m[x] - mn);                       // 0 on the first page
            a.l[x] *= f[x];
            a.m[x] = mn;
        }
        if constexpr (BITS != 16) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
            // the page's largest scale to [16, 32): the products p * scale (p <= 2^8) stay inside fp16, small ones stay normal
            const float vk = fminf(a.vk == 0.0f ? INFINITY : a.vk, __uint_as_float((uint32_t)(258 - max(32, (int)(__float_as_uint(vmax) >> 23))) << 23));
            const float fv = a.vk == 0.0f ? 0.0f : vk / a.vk;
            a.vk = vk;
#pragma unroll
            for (int x = 0; x < ST; ++x) f[x] *= fv;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            a.o[i][0] *= f[0]; a.o[i][2] *= f[0];
            a.o[i][1] *= f[ST - 1]; a.o[i][3] *= f[ST - 1];
        }
    }
    float p[ST][2];
#pragma unroll
    for (int x = 0; x < ST; ++x) {
        p[x][0] = ex2(s[x][0] - a.m[x]);
        p[x][1] = ex2(s[x][1] - a.m[x]);
        a.l[x] += p[x][0] + p[x][1];
    }
    // ---------------- O^T += V^T P ----------------
    if constexpr (BITS == 16) {
        // columns 2t, 2t + 1: p rounded and its remainder (one head per lane), or two heads and a second pass with the remainders
        auto split = [&](float x, float& hi, float& lo) {
            hi = BF ? __bfloat162float(__float2bfloat16_rn(x)) : __half2float(__float2half_rn(x));
            lo = x - hi;
        };
        auto pack = [&](float x, float y) -> uint32_t {
            if constexpr (BF) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
                return *reinterpret_cast<const uint32_t*>(&h);
            } else {
                return pack_h2(x, y);
            }
        };
        float hi[ST][2], lo[ST][2];
#pragma unroll
        for (int x = 0; x < ST; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) split(p[x][e], hi[x][e], lo[x][e]);
        uint32_t b[2][2];
        if constexpr (WIDE) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                b[0][e] = movmatrix_trans(pack(hi[0][e], hi[ST - 1][e]));
                b[1][e] = movmatrix_trans(pack(lo[0][e], lo[ST - 1][e]));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) b[0][e] = movmatrix_trans(pack(hi[0][e], lo[0][e]));
        }
        const uint32_t two = attended >> (2 * t);
        const uint32_t mask0 = ((two & 1u) ? 0xFFFFu : 0u) | ((two & 2u) ? 0xFFFF0000u : 0u);            // tokens 2t, 2t + 1
        const uint32_t mask1 = ((two & 0x100u) ? 0xFFFFu : 0u) | ((two & 0x200u) ? 0xFFFF0000u : 0u);    // tokens 2t + 8, 2t + 9
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t r[4];
            ldsm4_trans(r, chunk_pair<BITS>(vr, i));
            if (attended != 0xFFFFu) { r[0] &= mask0; r[2] &= mask0; r[1] &= mask1; r[3] &= mask1; }
            mma_f16<BF>(a.o[i], r[0], r[2], r[1], r[3], b[0][0], b[0][1]);
            if constexpr (WIDE) mma_f16<BF>(a.o[i], r[0], r[2], r[1], r[3], b[1][0], b[1][1]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int q = 0; q < 4; ++q) vs[e][q] *= a.vk;
        // operand columns 2t, 2t + 1: one head with the scales of 32-dim blocks 2c and 2c + 1, or (WIDE) two heads with one block's
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) {                   // 64 dims
            uint32_t b[2][2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if constexpr (WIDE) {
                    b[0][e] = movmatrix_trans(pack_h2(p[0][e] * vs[e][2 * cp], p[ST - 1][e] * vs[e][2 * cp]));
                    b[1][e] = LOGG == 6 ? b[0][e] : movmatrix_trans(pack_h2(p[0][e] * vs[e][2 * cp + 1], p[ST - 1][e] * vs[e][2 * cp + 1]));
                } else {
                    b[0][e] = movmatrix_trans(pack_h2(p[0][e] * vs[e][2 * cp], p[0][e] * vs[e][2 * cp + 1]));
                    b[1][e] = b[0][e];
                }
            }
            if constexpr (BITS == 4) {
                uint32_t r[4];
                ldsm4_trans(r, chunk_pair<BITS>(vr, cp));
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {           // 32 dims: this lane's 4 codes of two token pairs
                    uint32_t x[4], y[4];
                    q4_values(r[2 * cc], x);
                    q4_values(r[2 * cc + 1], y);
                    mma_m16n8k16(a.o[4 * cp + 2 * cc], x[0], x[1], y[0], y[1], b[cc][0], b[cc][1]);
                    mma_m16n8k16(a.o[4 * cp + 2 * cc + 1], x[2], x[3], y[2], y[3], b[cc][0], b[cc][1]);
                }
            } else {
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {           // 32 dims = chunks 4cp + 2cc and the next
                    uint32_t r[4];
                    ldsm4_trans(r, chunk_pair<BITS>(vr, 2 * cp + cc));
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint32_t x = r[2 * q], y = r[2 * q + 1];
                        mma_m16n8k16(a.o[4 * cp + 2 * cc + q], q8_values(x, 0x4240u), q8_values(x, 0x4341u), q8_values(y, 0x4240u), q8_values(y, 0x4341u), b[cc][0], b[cc][1]);
                    }
                }
            }
        }
    }
}

// The warp's result: for every (head of the group, dim) this lane owns, put(head, dim, weighted sum); then the statistics
// of the heads lane g == 0 owns, stat(head, max in log2 units, sum).
template <int BITS, bool WIDE, typename Put, typename Stat>
__device__ __forceinline__ void emit(WarpState<BITS, WIDE>& a, int group, int lane, Put put, Stat stat) {
    constexpr int ST = WarpState<BITS, WIDE>::ST;
    const int g = lane >> 2, t = lane & 3;
    const float inv = BITS == 16 ? 1.0f : (a.vk > 0.0f ? 1.0f / a.vk : 0.0f);
#pragma unroll
    for (int x = 0; x < ST; ++x) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) a.l[x] += __shfl_xor_sync(0xffffffffu, a.l[x], o);
        const int head = t + 4 * x;
        if (head >= group) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int d = BITS == 4 ? 32 * (i >> 1) + 4 * g + 2 * (i & 1) + e : BITS == 8 ? 16 * i + 2 * g + e : 16 * i + 8 * e + g;
                float v;
                if (WIDE) v = a.o[i][2 * e + x];
                else if (BITS == 16) v = a.o[i][2 * e] + a.o[i][2 * e + 1];
                else v = a.o[i][2 * e + ((i >> 1) & 1)];      // column of the block's own scales
                put(head, d, v * inv);
            }
        if (g == 0) stat(head, a.m[x], a.l[x]);
    }
}

}  // namespace attn
}  // namespace b200q
