// Weight-streaming quantized matvec for one to four batch rows (sm_100a): integer tensor-core products of raw codes.
//
//   y[b, n] = sum_k x[b, k] * (code[n, k] - zero[n, k/G]) * scale[n, k/G]
//
// What bounds it: HBM.  At 6.5 TB/s an SM receives 23 bytes, i.e. 46 q4 codes, per clock, so the code path has to stay
// well below 4 issue slots per 46 codes.  The kernel it replaces for these batches (gemv_fast.cuh) turns every code pair into
// fp16 (5 logic instructions and 2 mma.sync per 512 codes and row half) and needed 2.2 slots per clock at 0.49 of the
// copy rate (2 x 14336 x 4096 q4, one row: 20.7 us; here 12.2 us, 0.84).
// Beside HBM it is loads from shared memory: with 13 of them per 1 KB of codes and warp "MIO throttle" was the first stall.  Hence digits in
// the order of the mma, two mma per 16-byte load, scales eight groups per load, constants two steps per load, 6.5 loads in all, and no
// conversions in the affine step.  Cold weights, passes back to back, 13 loads -> now: q4 2 x 14336 x 4096 one row 14.3 -> 12.2 us, four rows
// 24.6 -> 20.0; 4096 x 4096 one row 5.1 -> 4.8; q8 8192 x 3008 groups of 32 one row 8.9 -> 8.5.
//   * mma.sync.m16n8k32 u8 x s8: a q4 word gives its even codes with one mask and its odd ones with a shift and a mask, a
//     q8 word is the operand as it lies.  512 codes per instruction, exact in int32.
//   * the activations become integers.  Per quantisation group they are scaled by a power of two to 22-bit fixed point
//     (an element below 2^-11 of its group's largest is rounded, by at most 2^-22 of that, the size of an fp32 sum's own rounding;
//     all others are exact) and cut into three signed bytes.  The three digits of a row are three columns of the 8-wide B
//     operand, which a matvec leaves empty anyway; digit sums meet in int32 and fp32.
//   * per group, in fp32: y += scale * ((c2 2^16 + c1 2^8 + c0) 2^-e - zero * X), X = sum of the group's activations.  With
//     one batch row two neighbouring groups sit side by side in the 8 columns and share this step (and the operand: the codes of
//     both meet the digits of both, each lane takes the sums of its own).
// The weights are not rounded at all.
//
// Work: rows are dealt evenly to the CTAs (one per SM), cut into tiles of at most 16 rows; a unit is a tile x 256 bytes of every
// row (512 q4 or 256 q8 codes), units are dealt to the 16 warps in order.  A warp is on its own: every lane copies 16-byte pieces
// with cp.async into a private ring (4 KB of codes per warp in flight, 64 KB per SM, started before griddepcontrol.wait since
// weights do not depend on the previous kernel): no producer warps and no barriers in the stream.  While piece c of a unit is
// consumed, piece c of the warp's next unit takes its place, so all shared-memory addresses are constants.  (Twice the
// ring in flight gained nothing: 2 x 14336 x 4096 13.8 against 12.5 us.)
// One CTA per SM, by its shared memory: with room for two, the CTAs of the next kernel of a dependent chain start beside this
// one's, and later ones then share an SM while another SM has none (gate/up and down of one row in turn: 36 us against 26.8).
// The units' sums meet in shared memory and are added in k order: the order does not depend on the CTA, the tile or the
// number of rows, so a tensor-parallel shard reproduces the unsharded rows bit for bit.
//
// Long rows (several rounds of 512 threads into fixed point, or more digits than fit into an SM's shared memory): a pair of CTAs owns twice
// the rows and each of them half of every row (KS = 2), so each prepares half of the digits.  The second CTA's sums go straight into the
// first one's shared memory, unit by unit, and are added there in the same order: the same bits.  One CTA -> a pair: q4 4096 x 14336 one row
// 10.0 -> 9.5 us, two 13.1 -> 11.5, four 22.5 -> 15.4 (whose digits do not fit one CTA: the older kernel); 4096 x 11008 three rows
// 14.7 -> 12.9, four 24.9 -> 13.7; q8 4096 x 14336 four rows 26.5 -> 20.2; 4096 x 4096 four rows 7.6 -> 7.1, but one row 4.8 -> 5.2: not split.
//
// Compiled into one translation unit per code width.
#pragma once

#include "gemv_params.cuh"

#include <algorithm>
#include <climits>
#include <cmath>

namespace b200q {
namespace {

constexpr int kI8Warps = 16;
constexpr int kI8Threads = kI8Warps * 32;
constexpr int kI8UnitBytes = 256;             // bytes of a unit in one row: four 64-byte pieces
constexpr uint32_t kI8OnePerSm = 116 * 1024;  // shared memory that keeps a second CTA off the SM
constexpr int kI8MaxRes = 1024;               // residual values kept in shared memory
// A group's digit sum S, at most 255 * 128 * 128 < 2^22 in magnitude, is added to these bits: as a float they are then kI8Magic + S, exactly,
// and no conversion is needed.
constexpr uint32_t kI8MagicBits = 0x4B400000u;
constexpr float kI8Magic = 12582912.0f;       // 1.5 * 2^23
// Sums are taken times 2^-kI8Shift until the end of a unit: codes times values of up to 2^123, whose sums per group are still finite, stay below
// 2^138.  More would cost the smallest results: the sums' steps are 2^(kI8Shift - 149), and bf16 results have steps of 2^-133.
constexpr int kI8Shift = 10;

struct I8Params {
    const void* x;          // [B, K]
    const void* res_in;     // norm prologue: rows = rmsnorm(x + res_in); may be null
    const void* norm_w;     // [K]; null = no prologue
    void* z_out;            // [B, K] or null
    void* normed_out;       // [B, K] or null
    const uint8_t* w[2];
    const __half* s[2];
    const __half* z[2];
    const void* residual;
    void* y;
    void* gate_out;
    void* up_out;
    void* act_out;
    float eps;
    int B, N, K, Gn, mats;
    int act_dtype, norm_w_dtype, row_bytes;
    int rows_lo, rem;       // CTA c owns rows_lo (+1 if c < rem) rows
    int units;              // units per (tile, matrix)
    int batch;              // tiles whose sums fit into shared memory at once
    TpOut tp_out;
    TpIn tp_in;
    uint32_t off_zero, off_xd, off_cst, off_res, off_part, off_meta, off_ring;
    uint32_t xstride, cstride, meta_slot;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16_part(uint32_t dst, const void* src, uint32_t bytes) {      // the rest is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_piece(uint32_t dst, const void* src, bool live) {      // 4, 8 or 16 bytes, or as many zeros
    if constexpr (BYTES == 16) cp16_part(dst, src, live ? 16u : 0u);
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(live ? BYTES : 0) : "memory");
}
__device__ __forceinline__ float i8_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float i8_round_act(float v, int dtype) {
    return dtype == B200Q_F16 ? __half2float(__float2half_rn(v)) : __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ void i8_words_to_f32(const uint32_t (&w)[4], int dtype, float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (dtype == B200Q_F16) {
            const __half2 h = *reinterpret_cast<const __half2*>(&w[i]);
            v[2 * i] = __low2float(h);
            v[2 * i + 1] = __high2float(h);
        } else {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
    }
}
__device__ __forceinline__ void i8_pack(uint32_t (&w)[4], int dtype, const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (dtype == B200Q_F16) {
            const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
    }
}
__device__ __forceinline__ void i8_ldg(uint32_t (&w)[4], const void* base, int64_t idx) {
    const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + idx);
    w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
}
__device__ __forceinline__ void i8_stg(void* base, int64_t idx, const uint32_t (&w)[4]) {
    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(base) + idx) = make_uint4(w[0], w[1], w[2], w[3]);
}
// Eight values of an input row, packed: x, or cast(x + res).  Plain rows, or packets of a tensor-parallel exchange, polled
// until they carry the expected sequence number (a template parameter: kernels that read plain rows are compiled without it).
struct I8Source { uint32_t seq16, limit; };
template <bool PACKETS>
__device__ __forceinline__ void i8_load_z(const I8Params& p, int64_t idx, I8Source& xs, uint32_t (&w)[4]) {
    if constexpr (!PACKETS) {
        i8_ldg(w, p.x, idx);
    } else if (!tp_load8_packets(p.x, idx, xs.seq16, xs.limit, w)) {
        atomicMax(&g_device_status, (int)EV_PEER_WAIT);
        xs.limit = 64u;
    }
    if (p.res_in != nullptr) {
        uint32_t rw[4];
        float v[8], r[8];
        i8_ldg(rw, p.res_in, idx);
        i8_words_to_f32(w, p.act_dtype, v);
        i8_words_to_f32(rw, p.act_dtype, r);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += r[i];
        i8_pack(w, p.act_dtype, v);
    }
}

__device__ __forceinline__ uint32_t s_ld32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void s_ld64(uint32_t a, uint32_t& x, uint32_t& y) {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x), "=r"(y) : "r"(a));
}
__device__ __forceinline__ uint32_t s_ldu16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
template <int NW>
__device__ __forceinline__ void s_ldw(uint32_t a, uint32_t (&w)[NW]) {
    if constexpr (NW == 1) {
        w[0] = s_ld32(a);
    } else if constexpr (NW == 2) {
        s_ld64(a, w[0], w[1]);
    } else {
        static_assert(NW == 4, "one 16-byte piece at most");
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(a));
    }
}
// D(16x8, s32) (+)= A(16x32, u8, row) * B(32x8, s8, col).  FIRST: the sums start from the bits of kI8Magic.
template <bool FIRST>
__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (FIRST) {
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kI8MagicBits));
    } else {
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
}

// All threads of the KS CTAs of a cluster.
template <int KS> __device__ __forceinline__ void i8_sync() {
    if constexpr (KS == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_first_cta(uint32_t addr, float v) {      // the same place in the cluster's first CTA
    asm volatile("{ .reg .b32 a; mapa.shared::cluster.u32 a, %0, 0; st.shared::cluster.f32 [a], %1; }" ::"r"(addr), "f"(v) : "memory");
}

// This lane's A operands of one group of 16 rows, rows g and g + 8 at `a_addr` (+ 512): mma i of the group.
template <int BITS, int LOGG> struct I8Words {
    static constexpr int GB = (1 << LOGG) * BITS / 8;
    static constexpr int H = GB == 128 ? 2 : 1;              // 64-byte pieces
    static constexpr int NW = (GB / 4 > 16 ? 16 : GB / 4) / 4;
    static constexpr int MI = BITS == 4 ? NW : NW / 2;       // mma per piece
    uint32_t a[H][NW], b[H][NW];
    __device__ __forceinline__ void load(uint32_t a_addr) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
            s_ldw<NW>(a_addr + h * 1024, a[h]);
            s_ldw<NW>(a_addr + h * 1024 + 512, b[h]);
        }
    }
    __device__ __forceinline__ void operands(int i, uint32_t (&r)[4]) const {
        const int h = i / MI, j = i % MI;
        if constexpr (BITS == 4) {
            r[0] = a[h][j] & 0x0F0F0F0Fu; r[1] = b[h][j] & 0x0F0F0F0Fu;
            r[2] = (a[h][j] >> 4) & 0x0F0F0F0Fu; r[3] = (b[h][j] >> 4) & 0x0F0F0F0Fu;
        } else {
            r[0] = a[h][2 * j]; r[1] = b[h][2 * j]; r[2] = a[h][2 * j + 1]; r[3] = b[h][2 * j + 1];
        }
    }
};

struct I8Pos { int tile, m, i; };             // a unit: tile, matrix, position in the row
__device__ __forceinline__ void i8_advance(I8Pos& u, int by, int U, int mats) {
    u.i += by;
    while (u.i >= U) {
        u.i -= U;
        if (++u.m == mats) { u.m = 0; ++u.tile; }
    }
}

// BITS: code width.  LOGG: log2(group size), 5..7.  NB: batch columns, 1, 2 or 4.
template <int BITS, int LOGG> struct I8Shape {
    static constexpr int G = 1 << LOGG;
    static constexpr int GB = G * BITS / 8;                  // bytes of a group in one row: 16 .. 128
    static constexpr int NM = G / 32;                        // mma per group
    static constexpr int GU = kI8UnitBytes / GB;             // groups per unit: 16 .. 2
    static constexpr int CP = GB > 64 ? GB / 64 : 1;         // 64-byte pieces per chunk (a chunk holds whole groups)
    static constexpr int CH = 4 / CP;                        // chunks per unit
    static constexpr int CG = CP * 64 / GB;                  // groups per chunk: 4, 2 or 1
    static constexpr int MB = GU * 2;                        // bytes of a unit's scales in one row: 32 .. 4
    static constexpr int WIN = MB > 16 ? 3 : 2;              // 16-byte pieces of an aligned window around them
    static constexpr int XU = GU * 96 * NM;                  // digit bytes of a unit: 1536 (q4) or 768 (q8)
};

// PB: bytes of a piece of scales, 16, 8 or 4, where rows of scales (and the units in them) start at multiples of it: pieces then lie in
// shared memory as the affine step wants them, eight groups to a load.  0: rows that start anywhere; an aligned window is copied and read
// one value at a time.  KS: CTAs per row, 1 or 2.  (PB at run time: 3 % slower.)
template <int BITS, int LOGG, int NB, bool PACKETS, int PB, int KS>
__global__ void __launch_bounds__(kI8Threads, 1) qgemv_i8_kernel(const __grid_constant__ I8Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    using S = I8Shape<BITS, LOGG>;
    constexpr int G = S::G, GB = S::GB, NM = S::NM, GU = S::GU, CP = S::CP, CH = S::CH, CG = S::CG, MB = S::MB, WIN = S::WIN;
    constexpr bool VEC = PB != 0;
    constexpr int NT = NB <= 2 ? 1 : NB / 2;          // 8-column tiles: one batch row takes 4 columns (3 digits)

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2;
    const int t = lane & 3;
    const uint32_t smem0 = smem_u32(smem);
    float* red = reinterpret_cast<float*>(smem);                   // sums of squares of the norm prologue, one per 32 pieces
    float* part = reinterpret_cast<float*>(smem + p.off_part);     // [tiles of a batch][mats][units][16 rows][NB]
    uint16_t* resid = reinterpret_cast<uint16_t*>(smem + p.off_res);

    const int rank = KS == 1 ? 0 : blockIdx.x % KS;
    const int cta = blockIdx.x / KS;
    const int r_lo = cta * p.rows_lo + min(cta, p.rem);
    const int r_cnt = p.rows_lo + (cta < p.rem ? 1 : 0);
    const int n_tiles = (r_cnt + 15) >> 4;
    const int tile_rows = (r_cnt + n_tiles - 1) / n_tiles;
    const int u_lo = KS == 1 ? 0 : rank * ((p.units + 1) / 2);                        // this CTA's units of a row
    const int U = KS == 1 ? p.units : rank == 0 ? (p.units + 1) / 2 : p.units / 2;
    const int mats = p.mats, B = p.B, Gn = p.Gn;
    if (KS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (waited for before the first access to the other's memory)

    if (threadIdx.x < (S::XU + 128) / 16) *reinterpret_cast<uint4*>(smem + p.off_zero + threadIdx.x * 16) = make_uint4(0u, 0u, 0u, 0u);
    pdl_launch_dependents();

    // ---------------- the warp's stream: the chunks of its units, in order ----------------
    const uint32_t ring = smem0 + p.off_ring + (uint32_t)warp * 4096u;
    const uint32_t meta0 = smem0 + p.off_meta + (uint32_t)warp * (2u * p.meta_slot);
    const uint32_t sw = (uint32_t)(((g >> 1) & 1) << 1 | ((g >> 2) & 1)) << 4;      // 16-byte pieces of a row are XORed with this: no bank conflicts
    const uint32_t dst_lane = ring + (uint32_t)g * 64 + ((uint32_t)(t << 4) ^ sw);
    I8Pos nu = {0, 0, 0};                              // the unit being copied
    i8_advance(nu, warp, U, mats);
    const uint8_t *srcA = nullptr, *srcM = nullptr;    // this lane's first 16 bytes of row g of that unit; its scales / zero points
    int leftA = 0, leftB = 0;                          // bytes from there to the end of row g, of row g + 8 (0: no such row)
    int leftM = 0;                                     // bytes of scales to copy (-1: there are no zero points)
    const int row8 = 8 * p.row_bytes;
    const int lane_w = g * p.row_bytes + t * 16;
    const int m_row = g + 8 * (t & 1);                 // lanes t = 0, 1 copy scales of rows g, g + 8, lanes t = 2, 3 zero points
    auto locate = [&]() {
        leftA = leftB = leftM = 0;
        if (nu.tile < n_tiles) {
            const int row0 = r_lo + nu.tile * tile_rows;
            const int rows = min(tile_rows, r_lo + r_cnt - row0);
            const int u = nu.i + u_lo;
            const int left = p.row_bytes - u * kI8UnitBytes - t * 16;
            srcA = p.w[nu.m] + ((int64_t)row0 * p.row_bytes + (u * kI8UnitBytes + lane_w));
            leftA = g < rows ? left : 0;
            leftB = g + 8 < rows ? left : 0;
            const __half* mb = t < 2 ? p.s[nu.m] : p.z[nu.m];
            if (m_row < rows) {
                const int64_t first = (int64_t)(row0 + m_row) * Gn;
                const int64_t at = (first + u * GU) * 2;
                if (VEC) leftM = (Gn - u * GU) * 2;
                else leftM = (int)min((int64_t)(WIN * 16), (first + Gn) * 2 - (at & ~(int64_t)15));
                srcM = reinterpret_cast<const uint8_t*>(mb) + (VEC ? at : at & ~(int64_t)15);
                if (mb == nullptr) leftM = -1;
            }
        }
    };
    auto issue = [&](int c, uint32_t meta) {           // chunk c of that unit; its scales ride on the first
        if (c == 0 && leftM > 0) {
            if (VEC) {
                const uint32_t dst = meta + (uint32_t)(t * 8 + g) * MB;
                constexpr int SP = VEC ? PB : 16;
#pragma unroll
                for (int q = 0; q < MB / SP; ++q) cp_piece<SP>(dst + q * SP, srcM + (leftM > q * SP ? q * SP : 0), leftM > q * SP);
            } else {
                // the aligned window that holds the row's values, zeros past the end of the row
                const uint32_t dst = meta + (uint32_t)(t * 8 + g) * (WIN * 16);
#pragma unroll
                for (int q = 0; q < WIN; ++q) cp16_part(dst + q * 16, srcM + (leftM > q * 16 ? q * 16 : 0), (uint32_t)max(0, min(16, leftM - q * 16)));
            }
        } else if (c == 0 && leftM < 0) {
            const uint32_t stride = VEC ? MB : WIN * 16;
            for (uint32_t q = 0; q < stride; q += 4) asm volatile("st.shared.u32 [%0], %1;" ::"r"(meta + (uint32_t)(t * 8 + g) * stride + q), "r"(0) : "memory");
        }
#pragma unroll
        for (int q = 0; q < CP; ++q) {
            const int off = (c * CP + q) * 64;
            if (leftA > off) cp16(dst_lane + (c * CP + q) * 1024, srcA + off);
            if (leftB > off) cp16(dst_lane + (c * CP + q) * 1024 + 512, srcA + row8 + off);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    locate();
#pragma unroll
    for (int c = 0; c < CH; ++c) issue(c, meta0);

    // ---------------- activations: everything from here on depends on the previous kernel ----------------
    pdl_wait();
    I8Source xsrc = {0u, p.tp_in.spin_limit ? p.tp_in.spin_limit : kTpSpinLimit};
    if (PACKETS) {
        xsrc.seq16 = tp_seq16(*reinterpret_cast<const volatile uint32_t*>(p.tp_in.epoch));
    } else if (p.tp_in.world > 0) {
        if ((int)threadIdx.x < p.tp_in.world && !tp_wait_source(p.tp_in, threadIdx.x)) atomicMax(&g_device_status, (int)EV_PEER_WAIT);
        __syncthreads();
    }
    const bool res_smem = p.residual != nullptr && r_cnt * B <= kI8MaxRes;
    if (res_smem)
        for (int i = threadIdx.x; i < r_cnt * B; i += kI8Threads) {
            const int b = i / r_cnt;
            resid[i] = reinterpret_cast<const uint16_t*>(p.residual)[(size_t)b * p.N + r_lo + (i - b * r_cnt)];
        }
    // Items: 8-value pieces of the padded rows.  A warp's 32 pieces lie in one row (a padded row is a multiple of 32 pieces).
    // The loop stays small on purpose: hoisting four loads per thread made every launch 0.4 us longer (instruction fetch)
    // and gained nothing on rows of 14336.
    const int pieces = U * GU * (G / 8);
    const int total = B * pieces;
    auto row_of = [&](int it) { return NB == 1 ? 0 : it / pieces; };
    auto load_item = [&](int it, uint32_t (&w)[4]) -> bool {
        const int b = row_of(it), k = (it - b * pieces) * 8 + u_lo * (GU * G);
        w[0] = w[1] = w[2] = w[3] = 0u;
        if (k < p.K) i8_load_z<PACKETS>(p, (int64_t)b * p.K + k, xsrc, w);
        return k < p.K;
    };
    if (p.norm_w != nullptr) {
        // sums of squares per 32 pieces, added per row in order: the same bits whatever the rows and the CTAs
#pragma unroll 1
        for (int it = threadIdx.x; it < total; it += kI8Threads) {
            uint32_t w[4];
            float v[8], ss = 0.0f;
            load_item(it, w);
            i8_words_to_f32(w, p.act_dtype, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
            ss = i8_warp_sum(ss);
            if (lane == 0) red[it / 32] = ss;
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int it = threadIdx.x; it < total; it += kI8Threads) {      // whole warps (shuffles below)
        const int b = row_of(it), pc = it - b * pieces;
        const int k = pc * 8 + u_lo * (GU * G);
        const int64_t idx = (int64_t)b * p.K + k;
        uint32_t w[4];
        const bool live = load_item(it, w);
        float v[8];
        i8_words_to_f32(w, p.act_dtype, v);
        if (p.norm_w != nullptr && live) {
            float tot = 0.0f;
            for (int q = 0; q < pieces / 32; ++q) tot += red[b * (pieces / 32) + q];
            const float inv = rsqrtf(tot / (float)p.K + p.eps);
            if (cta == 0 && p.z_out != nullptr) i8_stg(p.z_out, idx, w);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] *= inv * load_as_f32(p.norm_w, p.norm_w_dtype, k + i);
            i8_pack(w, p.act_dtype, v);
            i8_words_to_f32(w, p.act_dtype, v);
            if (cta == 0 && p.normed_out != nullptr) i8_stg(p.normed_out, idx, w);
        }
        float mx = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(v[i]));
        float X = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
#pragma unroll
        for (int o = 1; o < G / 8; o <<= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            X += __shfl_xor_sync(0xffffffffu, X, o);
        }
        // 2^e brings the group's largest magnitude to [2^21, 2^22)
        const int e = min(120, 148 - (int)(__float_as_uint(mx) >> 23));
        const float up = __uint_as_float((uint32_t)(e + 127) << 23);
        uint32_t u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = __float_as_uint(fmaf(v[i], up, kI8Magic)) + (0x808080u - kI8MagicBits);      // three digits, each + 128
        const int in = pc & (G / 8 - 1), grp = pc / (G / 8);
        int tt, ii;                                    // lane and mma that meet these 8 values
        if (GB == 128) { tt = (in & 7) >> 1; ii = ((in >> 3) << 1) | (in & 1); }      // two 16-byte pieces per lane
        else { tt = in / NM; ii = in & (NM - 1); }
        // digits lie in the order of the mma they enter, two mma to a 16-byte piece: [mma pair][digit][lane tt]; one batch row: even groups
        // of the unit, then odd ones
        const int unit = grp / GU, gl = grp & (GU - 1), m = (NB == 1 ? gl >> 1 : gl) * NM + ii;
        uint8_t* dst = smem + p.off_xd + (size_t)b * p.xstride + (uint32_t)unit * S::XU + (NB == 1 ? (gl & 1) * (S::XU / 2) : 0) + (m >> 1) * 192 + tt * 16 + (m & 1) * 8;
        uint32_t d[3][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // q4: even codes of the word, then odd ones; q8: its first four bytes, then the next
            const uint32_t a = u[BITS == 4 ? h : 4 * h], b2 = u[BITS == 4 ? 2 + h : 4 * h + 1];
            const uint32_t c = u[BITS == 4 ? 4 + h : 4 * h + 2], d2 = u[BITS == 4 ? 6 + h : 4 * h + 3];
            const uint32_t lo0 = prmt(a, b2, 0x5140), lo1 = prmt(c, d2, 0x5140);
            d[2][h] = prmt(lo0, lo1, 0x5410) ^ 0x80808080u;
            d[1][h] = prmt(lo0, lo1, 0x7632) ^ 0x80808080u;
            d[0][h] = prmt(prmt(a, b2, 0x0062), prmt(c, d2, 0x0062), 0x5410) ^ 0x80808080u;
        }
#pragma unroll
        for (int s = 0; s < 3; ++s) *reinterpret_cast<uint2*>(dst + s * 64) = make_uint2(d[s][0], d[s][1]);
        if (in == 0) {
            // 2^(16 - e - shift), the weight of the high digit (e is at most 120, so all three weights are exact).  Even lanes own the two high
            // digits, odd lanes the low one and the zero-point term: [lane t & 1, one batch row: and parity of the group][step]
            const float high = mx < INFINITY ? __uint_as_float((uint32_t)(127 + 16 - kI8Shift - e) << 23) : NAN;
            float2* cst = reinterpret_cast<float2*>(smem + p.off_cst + (size_t)b * p.cstride) + unit * (2 * GU) + (NB == 1 ? (gl & 1) * GU + (gl >> 1) : gl);
            cst[0] = make_float2(high, 0.0f);
            cst[NB == 1 ? GU / 2 : GU] = make_float2(high * 0x1p-16f, X * __uint_as_float((uint32_t)(127 - kI8Shift) << 23));
        }
    }
    __syncthreads();
    if (KS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

    // ---------------- per-lane constants of the consumer ----------------
    const int col_b = g >> 2;                          // batch row of this lane's B column inside a tile; one batch row: parity of the group
    const bool digit = (g & 3) < 3;
    const uint32_t zaddr = smem0 + p.off_zero + 64 + t * 16;             // + 64: other banks than the third digit, which is read together with it
    const uint32_t xlane = smem0 + p.off_xd + (uint32_t)(g & 3) * 64 + t * 16;
    constexpr int FL = NB == 1 ? GU / 2 : GU;          // affine steps of a unit: a group, or with one batch row two neighbouring ones
    constexpr int CV = FL < 2 || NB == 4 ? 1 : 2;      // steps whose constants are read at once (four rows: no registers to spare)
    const uint32_t cbase = smem0 + p.off_cst + (uint32_t)(NB == 1 ? (t >> 1) * 2 + (t & 1) : t & 1) * (FL * 8);
    const float k_mid = (t & 1) ? 0.0f : 0x1p-8f;                        // weight of the second column by that of the first
    const float k_off = (t & 1) ? -kI8Magic : -kI8Magic * 1.00390625f;   // what the magic number adds to both, negative
    const uint32_t sel_par = t >> 1 ? 0x4432u : 0x4410u;                 // one batch row: the half of a pair of scales that is this lane's
    constexpr int LPP = GB >= 64 ? 16 : GB / 4;        // lane pitch in a row
    const uint32_t a_lane = (((uint32_t)(t * LPP) & ~15u) ^ sw) + ((uint32_t)(t * LPP) & 15u);
    uint32_t a_grp[CG];                                // this lane's bytes of the chunk's groups (first chunk)
#pragma unroll
    for (int q = 0; q < CG; ++q) a_grp[q] = ring + (uint32_t)g * 64 + (a_lane ^ (uint32_t)(q * GB));
    const uint32_t m_stride = VEC ? MB : WIN * 16;
    const uint32_t m_lane = (uint32_t)g * m_stride;

    I8Pos cu = nu;
    uint32_t cmeta = 0;                                // scale buffer of the unit being consumed
#pragma unroll 1
    for (int t0 = 0; t0 < n_tiles; t0 += p.batch) {
        const int t1 = min(n_tiles, t0 + p.batch);
#pragma unroll 1
        while (cu.tile < t1) {
            uint32_t m_s0 = meta0 + cmeta + m_lane, m_s1 = m_s0 + 8 * m_stride;
            if (!VEC) {
                const uint32_t e = (uint32_t)(r_lo + cu.tile * tile_rows + g) * (uint32_t)Gn + (cu.i + u_lo) * GU;      // low bits are enough
                m_s0 += (e * 2) & 15u;
                m_s1 += ((e + 8u * Gn) * 2) & 15u;
            }
            const uint32_t m_z0 = m_s0 + 16 * m_stride, m_z1 = m_s1 + 16 * m_stride;
            float y[NT][2];
            // B operand addresses: a lane without a digit reads zeros
            uint32_t xb[NT], cc[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                y[nt][0] = y[nt][1] = 0.0f;
                const int b = NB == 1 ? 0 : 2 * nt + col_b;
                const uint32_t a = xlane + (uint32_t)b * p.xstride + (uint32_t)cu.i * S::XU + (NB == 1 ? (uint32_t)col_b * (S::XU / 2) : 0u);
                xb[nt] = digit && b < B ? a : zaddr;
                const int cb = NB == 1 ? 0 : min(2 * nt + (t >> 1), B - 1);
                cc[nt] = cbase + (uint32_t)cb * p.cstride + (uint32_t)cu.i * (GU * 16);
            }

            i8_advance(nu, kI8Warps, U, mats);
            locate();
            // scales (and zero points) of rows g and g + 8, eight groups at a time, two to a register
            constexpr int SG = GU < 8 ? GU : 8;
            uint32_t sw0[SG / 2], sw1[SG / 2], zw0[SG / 2], zw1[SG / 2];
            auto scales = [&](int gl) {
                if (!VEC) return;
                s_ldw<SG / 2>(m_s0 + gl * 2, sw0);
                s_ldw<SG / 2>(m_s1 + gl * 2, sw1);
                s_ldw<SG / 2>(m_z0 + gl * 2, zw0);
                s_ldw<SG / 2>(m_z1 + gl * 2, zw1);
            };
            auto scale_of = [&](const uint32_t (&w)[SG / 2], uint32_t row, int f) -> float {      // of affine step f
                if (!VEC) {                     // rows of scales that start anywhere: one at a time
                    const uint32_t h = s_ldu16(row + (NB == 1 ? f * 4 + (t >> 1) * 2 : f * 2));
                    return __low2float(*reinterpret_cast<const __half2*>(&h));
                }
                if constexpr (NB == 1) {
                    const uint32_t h = prmt(w[f % (SG / 2)], 0u, sel_par);
                    return __low2float(*reinterpret_cast<const __half2*>(&h));
                } else {
                    const __half2 h = *reinterpret_cast<const __half2*>(&w[f % SG / 2]);
                    return f & 1 ? __high2float(h) : __low2float(h);
                }
            };
            constexpr int AC = NB == 1 ? 2 : NT;               // one batch row: sums of the even and of the odd group
            int acc[AC][4];
            uint32_t cw[NT][2 * CV];
            // affine step f:  y += s * (digits - zero * X)
            auto flush = [&](int f) {
                const float s0 = scale_of(sw0, m_s0, f), s1 = scale_of(sw1, m_s1, f), z0 = scale_of(zw0, m_z0, f), z1 = scale_of(zw1, m_z1, f);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    if (NB != 4 && f % CV == 0) s_ldw<2 * CV>(cc[nt] + f * 8, cw[nt]);
                    float c[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) c[e] = __int_as_float(NB == 1 ? (t >> 1 ? acc[AC - 1][e] : acc[0][e]) : acc[nt % AC][e]);
                    // the magic number goes first: times the weight of a large row it would not be finite
                    const float f0 = fmaf(c[1], k_mid, c[0] + k_off), f1 = fmaf(c[3], k_mid, c[2] + k_off);
                    if (NB == 4 && f % CV == 0) s_ldw<2 * CV>(cc[nt] + f * 8, cw[nt]);
                    const float w0 = __uint_as_float(cw[nt][f % CV * 2]), xf = __uint_as_float(cw[nt][f % CV * 2 + 1]);
                    y[nt][0] = fmaf(s0, fmaf(-z0, xf, f0 * w0), y[nt][0]);
                    y[nt][1] = fmaf(s1, fmaf(-z1, xf, f1 * w0), y[nt][1]);
                }
            };
            // Digits of two mma per load.  One batch row: the lanes of columns 0-3 hold the even group's, those of columns 4-7 the odd group's,
            // and both groups' codes meet the same operand; each lane then takes the sums that are its own.
            constexpr int BP = NM < 2 ? 1 : NM / 2;            // 16-byte pieces of a group's digits
            uint32_t bq[NT][BP][4];
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                asm volatile("cp.async.wait_group %0;" ::"n"(CH - 1) : "memory");
                __syncwarp();
                // groups past the end of the row have zero digits: whatever their codes are, they add nothing
#pragma unroll
                for (int q = 0; q < CG; ++q) {
                    const int gl = c * CG + q, f = NB == 1 ? gl >> 1 : gl;
                    if (gl % SG == 0) scales(gl);
                    if ((NB != 1 || gl % 2 == 0) && (f * NM) % 2 == 0) {
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                            for (int i = 0; i < BP; ++i) s_ldw<4>(xb[nt] + (f * NM / 2 + i) * 192, bq[nt][i]);
                    }
                    I8Words<BITS, LOGG> words;
                    words.load(a_grp[q] + c * CP * 1024);
#pragma unroll
                    for (int i = 0; i < NM; ++i) {
                        uint32_t r[4];
                        words.operands(i, r);
                        const int piece = i / 2, h = (f * NM + i) % 2 * 2;
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            int (&d)[4] = acc[NB == 1 ? gl % 2 : nt % AC];
                            if (i == 0) mma_u8s8<true>(d, r[0], r[1], r[2], r[3], bq[nt][piece][h], bq[nt][piece][h + 1]);
                            else mma_u8s8<false>(d, r[0], r[1], r[2], r[3], bq[nt][piece][h], bq[nt][piece][h + 1]);
                        }
                    }
                    if (NB != 1 || gl % 2 == 1) flush(f);
                }
                __syncwarp();
                issue(c, meta0 + (cmeta ^ p.meta_slot));
            }
            // ---- the unit's sums into their place ----
            float* dst = part + ((size_t)((cu.tile - t0) * mats + cu.m) * p.units + cu.i + u_lo) * (16 * NB);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v = y[nt][h] * (float)(1 << kI8Shift);
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    if (NB == 1) v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if ((NB == 1 ? t == 0 : (t & 1) == 0)) {
                        float* at = dst + (g + 8 * h) * NB + (NB == 1 ? 0 : 2 * nt + (t >> 1));
                        if constexpr (KS == 1) *at = v;
                        else st_first_cta(smem_u32(at), v);
                    }
                }
            cu = nu;
            cmeta ^= p.meta_slot;
        }
        i8_sync<KS>();
        // ---- rows of these tiles: units added in k order, clamp, round, residual add or SwiGLU, store ----
        const float fmax_act = p.act_dtype == B200Q_F16 ? 65504.0f : 3.3895313892515355e38f;
        const int rb0 = t0 * tile_rows, n_rows = min(r_cnt, t1 * tile_rows) - rb0;
        for (int it = threadIdx.x; it < (rank == 0 ? n_rows * B : 0); it += kI8Threads) {
            const int b = NB == 1 ? 0 : it / n_rows, rr = it - b * n_rows;
            const int tl = rr / tile_rows, r = rr - tl * tile_rows;
            const float* src = part + (size_t)tl * mats * p.units * (16 * NB) + r * NB + b;
            float val[2] = {0.0f, 0.0f};
            for (int m = 0; m < mats; ++m) {
                float sum = 0.0f;
#pragma unroll 8
                for (int i = 0; i < p.units; ++i) sum += src[(m * p.units + i) * (16 * NB)];
                val[m] = i8_round_act(fminf(fmaxf(sum, -fmax_act), fmax_act), p.act_dtype);
            }
            const int row = r_lo + rb0 + rr;
            const int64_t o = (int64_t)b * p.N + row;
            auto bits_of = [&](float v) {
                return p.act_dtype == B200Q_F16 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
            };
            float v = val[0];
            if (mats == 2) {
                if (p.gate_out != nullptr) reinterpret_cast<unsigned short*>(p.gate_out)[o] = bits_of(val[0]);
                if (p.up_out != nullptr) reinterpret_cast<unsigned short*>(p.up_out)[o] = bits_of(val[1]);
                v = (val[0] / (1.0f + expf(-val[0]))) * val[1];
                if (p.act_out != nullptr) reinterpret_cast<unsigned short*>(p.act_out)[o] = bits_of(v);
            } else {
                if (p.residual != nullptr) {
                    const uint16_t rb = res_smem ? resid[b * r_cnt + rb0 + rr] : reinterpret_cast<const uint16_t*>(p.residual)[o];
                    v = load_as_f32(&rb, p.act_dtype, 0) + v;
                }
                if (p.y != nullptr) reinterpret_cast<unsigned short*>(p.y)[o] = bits_of(v);
            }
            if (p.tp_out.world > 0) {
                // tensor-parallel exchange: the value goes to column block `rank` of every rank's full rows
                const int64_t of = (int64_t)b * p.N * p.tp_out.world + (int64_t)p.tp_out.rank * p.N + row;
                const unsigned short bits16 = bits_of(v);
                const uint32_t pk = p.tp_out.packets ? tp_packet(bits16, tp_seq16(tp_writer_seq(p.tp_out))) : 0u;
#pragma unroll 1
                for (int peer = 0; peer < p.tp_out.world; ++peer) {
                    if (p.tp_out.packets) st_volatile_u32(reinterpret_cast<uint32_t*>(p.tp_out.full[peer]) + of, pk);
                    else reinterpret_cast<unsigned short*>(p.tp_out.full[peer])[of] = bits16;
                }
            }
        }
        if (t1 < n_tiles || p.tp_out.world > 0) i8_sync<KS>();      // the sums have been read / all peer stores are issued
    }
    if (p.tp_out.world > 0 && warp == 0) {
        if (p.tp_out.packets) tp_finish_writer_packets(p.tp_out, lane);
        else tp_finish_writer(p.tp_out, lane);
    }
}

inline bool i8_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline uint32_t i8_align(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

template <int BITS, int LOGG, int NB>
int launch_i8(const GemvParams& q, bool gate_up, cudaStream_t stream) {
    using S = I8Shape<BITS, LOGG>;
    I8Params p = {};
    p.x = q.x; p.res_in = q.res_in; p.norm_w = q.norm_w; p.z_out = q.z_out; p.normed_out = q.normed_out;
    p.mats = gate_up ? 2 : 1;
    for (int m = 0; m < p.mats; ++m) {
        p.w[m] = q.w[m];
        p.s[m] = (const __half*)q.s[m];
        p.z[m] = (const __half*)q.z[m];
    }
    p.residual = q.residual; p.y = q.y; p.gate_out = q.gate_out; p.up_out = q.up_out; p.act_out = q.act_out;
    p.eps = q.eps; p.B = q.B; p.N = q.N; p.K = q.K; p.Gn = q.Gn; p.act_dtype = q.act_dtype; p.norm_w_dtype = q.norm_w_dtype;
    p.row_bytes = q.row_bytes; p.tp_out = q.tp_out; p.tp_in = q.tp_in;
    p.units = (p.row_bytes + kI8UnitBytes - 1) / kI8UnitBytes;
    // The largest piece of scales that rows and units are multiples of.  Window -> pieces, gate and up, one and four rows: q4 11008 x 2816
    // groups of 128, two pieces of 4 bytes, 9.5 -> 8.0 us and 13.4 -> 11.9; 9000 x 2816 groups of 64, two of 8, 8.9 -> 7.9 and 12.6 -> 11.4;
    // 6000 x 2688 groups of 32, four of 8, 8.4 -> 8.2 and 12.8 -> 12.1.  More pieces cost more than the window: one row of q8 8192 x 3008 groups
    // of 32, four of 4, 12.74 -> 12.78; q4 5003 x 2624 groups of 32, eight of 4, 8.2 -> 8.6.
    constexpr int P4 = S::MB <= (NB == 1 ? 8 : 16) ? 4 : 0, P8 = S::MB >= 8 ? 8 : P4, P16 = S::MB >= 16 ? 16 : P8;
    int pb = P16;
    while (pb > 0 && p.Gn * 2 % pb != 0) pb = pb == 16 ? P8 : pb == 8 ? P4 : 0;
    const int form = pb == 16 ? 3 : pb == 8 ? 2 : pb == 4 ? 1 : 0;
    p.meta_slot = 32u * (form ? S::MB : S::WIN * 16);
    const bool packets = p.tp_in.world > 0 && p.tp_in.packets;
    int ks = 1;
    const int tile_bytes = p.mats * p.units * 16 * NB * 4;
    int grid = 1;
    auto plan = [&]() -> uint32_t {
        // a CTA (or half a pair) per SM, fewer only when it would own less than four rows
        grid = std::max(1, std::min(sm_count() / ks, (p.N + 3) / 4));
        p.rows_lo = p.N / grid;
        p.rem = p.N % grid;
        const int r_max = p.rows_lo + (p.rem ? 1 : 0), units = (p.units + ks - 1) / ks;
        p.batch = std::min({(r_max + 15) / 16, std::max(1, (ks == 1 ? 24 : 64) * 1024 / tile_bytes), p.batch});
        p.xstride = (uint32_t)units * S::XU;
        p.cstride = (uint32_t)units * S::GU * 16 + (q.B > 1 ? 32 : 0);      // + 32: two batch rows are read together, from different banks
        uint32_t off = i8_align((uint32_t)q.B * p.units * S::GU * (S::G / 8) / 32 * 4, 128);
        p.off_zero = off;  off += S::XU + 128;
        p.off_xd = off;    off += i8_align((uint32_t)q.B * p.xstride, 128);
        p.off_cst = off;   off += (uint32_t)q.B * p.cstride;
        p.off_res = off;   off += p.residual != nullptr ? i8_align((uint32_t)std::min(r_max * q.B, kI8MaxRes) * 2, 128) : 0;
        off = i8_align(off, 128);
        p.off_part = off;  off += i8_align((uint32_t)(p.batch * tile_bytes), 128);
        p.off_meta = off;  off += kI8Warps * 2 * p.meta_slot;
        off = i8_align(off, 1024);
        p.off_ring = off;
        return std::max<uint32_t>(off + kI8Warps * 4096, kI8OnePerSm);
    };
    auto fit = [&](int parts) -> uint32_t {
        ks = parts;
        p.batch = INT_MAX;
        uint32_t off = plan();
        while (off > (uint32_t)max_smem_optin() && p.batch > 1) {      // long rows: fewer tiles whose sums lie in shared memory together
            --p.batch;
            off = plan();
        }
        return off;
    };
    // Rounds of the three phases in a CTA: rows into fixed point, units, results.  A pair costs a launch 0.4 us (4096 x 4096 one row, which it
    // saves nothing, 4.8 -> 5.2), a round of the first phase 0.6 us by the SM's clock, so two rounds less, of whichever phase, are asked
    // for.  (A fused norm needs the whole row in each CTA.)
    auto rounds = [&]() -> int {
        const int units = (p.units + ks - 1) / ks, r_max = p.rows_lo + (p.rem ? 1 : 0), tiles = (r_max + 15) / 16;
        auto per = [](int n, int by) { return (n + by - 1) / by; };
        return per(q.B * units * S::GU * (S::G / 8), kI8Threads) + per(tiles * p.mats * units, kI8Warps) + per(r_max * q.B, kI8Threads);
    };
    uint32_t off = fit(1);
    if (p.norm_w == nullptr && p.units >= 4) {
        const bool fits = off <= (uint32_t)max_smem_optin();
        const int one = rounds();
        const uint32_t off2 = fit(2);
        if (off2 <= (uint32_t)max_smem_optin() && (!fits || one - rounds() >= 2)) off = off2;
        else off = fit(1);
    }
    if (off > (uint32_t)max_smem_optin()) return B200Q_ERR_UNSUPPORTED;

    using KernelFn = void (*)(I8Params);
    static const KernelFn kernels[4][4] = {
        {qgemv_i8_kernel<BITS, LOGG, NB, false, 0, 1>, qgemv_i8_kernel<BITS, LOGG, NB, false, P4, 1>,
         qgemv_i8_kernel<BITS, LOGG, NB, false, P8, 1>, qgemv_i8_kernel<BITS, LOGG, NB, false, P16, 1>},
        {qgemv_i8_kernel<BITS, LOGG, NB, true, 0, 1>, qgemv_i8_kernel<BITS, LOGG, NB, true, P4, 1>,
         qgemv_i8_kernel<BITS, LOGG, NB, true, P8, 1>, qgemv_i8_kernel<BITS, LOGG, NB, true, P16, 1>},
        {qgemv_i8_kernel<BITS, LOGG, NB, false, 0, 2>, qgemv_i8_kernel<BITS, LOGG, NB, false, P4, 2>,
         qgemv_i8_kernel<BITS, LOGG, NB, false, P8, 2>, qgemv_i8_kernel<BITS, LOGG, NB, false, P16, 2>},
        {qgemv_i8_kernel<BITS, LOGG, NB, true, 0, 2>, qgemv_i8_kernel<BITS, LOGG, NB, true, P4, 2>,
         qgemv_i8_kernel<BITS, LOGG, NB, true, P8, 2>, qgemv_i8_kernel<BITS, LOGG, NB, true, P16, 2>}};
    const int kind = (ks - 1) * 2 + packets;
    KernelFn kernel = kernels[kind][form];
    static bool configured[16][64] = {};   // per instantiation and device; a race only repeats the call
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[kind * 4 + form][dev & 63]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem_optin()) != cudaSuccess)
            return B200Q_ERR_LAUNCH;
        configured[kind * 4 + form][dev & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid * ks);
    cfg.blockDim = dim3(kI8Threads);
    cfg.dynamicSmemBytes = off;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ks > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim = {(unsigned)ks, 1, 1};
        ++na;
    }
    if (!tuning_get("no_pdl")) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    if (cudaLaunchKernelEx(&cfg, kernel, p) != cudaSuccess) return B200Q_ERR_LAUNCH;
    return finish_launch();
}

template <int BITS, int LOGG>
int dispatch_i8_cols(const GemvParams& p, bool gate_up, cudaStream_t stream) {
    if (p.B <= 1) return launch_i8<BITS, LOGG, 1>(p, gate_up, stream);
    if (p.B <= 2) return launch_i8<BITS, LOGG, 2>(p, gate_up, stream);
    return launch_i8<BITS, LOGG, 4>(p, gate_up, stream);
}

template <int BITS>
int dispatch_i8(const GemvParams& p, bool gate_up, cudaStream_t stream) {
    if (p.B > 4 || p.scale_dtype != B200Q_F16) return B200Q_ERR_UNSUPPORTED;
    for (int m = 0; m < (gate_up ? 2 : 1); ++m)
        if (!i8_aligned16(p.s[m]) || !i8_aligned16(p.z[m])) return B200Q_ERR_UNSUPPORTED;
    if (p.G == 32) return dispatch_i8_cols<BITS, 5>(p, gate_up, stream);
    if (p.G == 64) return dispatch_i8_cols<BITS, 6>(p, gate_up, stream);
    return dispatch_i8_cols<BITS, 7>(p, gate_up, stream);
}

}  // namespace
}  // namespace b200q
