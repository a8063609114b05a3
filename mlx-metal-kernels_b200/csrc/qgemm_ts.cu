// Quantized GEMM for batches of rows on the 5th-generation tensor cores (tcgen05, sm_100a):
//
//   y[b, n] = sum_k x[b, k] * (code[n, k] - zero[n, k/G]) * scale[n, k/G]
//
// The weights are the A operand and live in TENSOR MEMORY, the activations are the B operand in
// shared memory, the accumulator D[128 weight rows, up to 128 batch columns] stays in tensor memory:
//
//   weight producer (one lane)    2-D TMA, 128-byte swizzle: 128 rows x 128 bytes of codes per stage and matrix; scales / zero
//                                 points 16 groups at a time where their rows allow it
//   row producer (one lane)       2-D TMA of the activations: 128 k x the block's columns straight into the operand layout (the
//                                 128-byte swizzle of the copy is the K-major layout of the MMA); rows past the batch are zero-filled
//   dequantise warps (16)         thread = weight row, four groups of four warps take the chunks (128 k) in turn.  Codes come out of
//                                 shared memory 16 bytes at a time (conflict-free through the swizzle), become fp16 weights in
//                                     w = ((base+q) - (base+rint(z))) * s + (rint(z) - z) * s
//                                 (exact subtraction, then one fused multiply-add) and go to tensor memory with tcgen05.st
//   MMA (two warps, one elected   tcgen05.mma.kind::f16, M = 128, N = block columns, K = 16, A from tensor memory; tcgen05.commit
//        lane of each issues)     releases the chunk / the operand slot / the accumulator.  Each warp has an accumulator of its own - gate
//                                 and up, or the even and the odd chunks of one matrix: one warp's waits, ring arithmetic and
//                                 commits cost it more than the 8 MMAs of a chunk
//   epilogue (dequantise warps)   tcgen05.ld of D, clamp, round, residual add or SwiGLU, store
//
// What bounds it: a chunk (128 x 128 weights) costs the dequantisation 4 x 260 warp instructions, i.e. about 340 clocks on the SM's four
// schedulers, and the tensor pipe 8 x 22 clocks up to 32 columns, 8 x 65 at 128; a chunk takes about 480, since stores into tensor
// memory and MMAs hold each other up and every barrier costs a waiting warp some time beside the others.  Fewer, longer pieces per wait are
// therefore better: eight warps per chunk instead of four were 12 % slower on an MLP block of 32 rows.  One block of up to 128 columns
// shares each dequantised weight.  q4 MLP blocks: 4096 -> 14336 -> 4096, 32 rows 45.9 us; 4096 -> 11008 -> 4096, 256 rows 104 us.
// Codes are unpacked in k order (one byte permute per pair): the activations need no rearrangement, and nothing but TMA touches
// them.  (The form before this one permuted the rows in shared memory with four warps, recomputed the group constants per 32 k and
// kept 32 columns per launch: 1800 warp instructions per chunk; a 256-row prompt chunk re-streamed its weights eight times.)
//
// Work items are (row tile, column block) pairs.  When there are fewer than SMs, the K range of an item is split over the CTAs of a
// thread-block cluster; the partial accumulators are summed in rank order through distributed shared memory by the cluster's first
// CTA (deterministic, no global scratch).
// Every wait is bounded; a wait that runs out records an event in the status word and the kernel
// carries on without the data so that it always terminates and frees its tensor memory.
#include "gemv_params.cuh"

#include "ring.h"
#include "tensor_map.cuh"

#include <algorithm>
#include <functional>
#include <mutex>
#include <unordered_map>

namespace b200q {

B200Q_DEFINE_STATUS_WORD(qgemm_ts_read_status)

namespace {

constexpr int kRows = 128;                     // weight rows per tile = lanes of tensor memory
constexpr int kChunkCols = 64;                 // tensor-memory columns of a chunk of A (2 halves each): 128 k, or 64 k in two terms
constexpr int chunk_k(bool split) { return split ? 64 : 128; }
constexpr int kRowBytes = 128;                 // bytes of one weight row per stage = the swizzle span
constexpr int kWTile = kRows * kRowBytes;      // 16 KB of codes per stage and matrix
constexpr int kMetaGroups = 16;                // groups per scale tile: 32 bytes of a row (one sector), several stages' worth
constexpr int kMetaTile = kRows * kMetaGroups * 2;   // 4 KB of scales (or zero points)
constexpr int kMaxMetaBufs = 4;
constexpr int kMaxStages = 8;
constexpr int kMaxASlots = 8;
constexpr int kMaxXSlots = 8;
constexpr int kMaxCols = 128;                  // batch columns per item
constexpr uint32_t kTsWaitLimit = 1u << 20;
constexpr int kDeqWarps = 16;
constexpr int kGroups = kDeqWarps / 4;         // a group = four warps = one per 32-lane quarter of tensor memory
constexpr int kMmaWarps = 2;                   // one accumulator each
constexpr int kTmaWarp = kDeqWarps, kRowWarp = kDeqWarps + 1, kMmaWarp0 = kDeqWarps + 2;
constexpr int kTsThreads = (kDeqWarps + 2 + kMmaWarps) * 32;

struct alignas(64) TsParams {
    CUtensorMap wmap[2];        // codes [N, row_bytes] u8, box 128 B x 128 rows, 128-byte swizzle
    CUtensorMap smap[2];        // scales [N, Gn] fp16 as bytes, box 32 B x 128 rows, 32-byte swizzle
    CUtensorMap zmap[2];        // zero points, same
    CUtensorMap xmap;           // activations [B, K] fp16 as bytes, box 128 B (64 k) x block columns, 128-byte swizzle
    const void* x;              // activations (host side: the map depends on the block's columns)
    const uint16_t* s[2];       // scales / zero points where a row is no multiple of 16 bytes: read by the dequantise warps
    const uint16_t* z[2];
    const float* col_scale;     // [B] factor of the result columns (rows that were scaled into fp16), or null
    const uint16_t* residual;   // plain: out = cast(residual + cast(y)); may be null
    uint16_t* y;
    uint16_t* gate_out;
    uint16_t* up_out;
    uint16_t* act_out;
    int B, N, Gn;
    int has_z;
    int bf16;                   // outputs and residual are bf16
    int ncols;                  // columns of a block: MMA N, a multiple of 16
    int nblk;                   // column blocks
    int items;                  // row tiles x column blocks
    int split;                  // CTAs per cluster = parts of the K range
    int n_stage_total;          // stages over the whole K (the last may be short: TMA fills zeros)
    int stages;                 // depth of the ring of weight stages
    int a_slots;                // chunks of A in tensor memory
    int a_col0;                 // first column of the A ring (the accumulators sit below it)
    int x_slots;                // depth of the ring of activation chunks
    int meta_bufs;              // depth of the ring of scale tiles
    uint32_t stage_bytes;       // one weight stage: codes x MATS
    uint32_t off_meta;          // ring of scale tiles, each [scales, zeros] x MATS
    uint32_t off_x, x_bytes;    // ring of activation chunks [2 x 64 k][columns], K-major, 128-byte swizzle
    uint32_t off_red;           // dedicated buffer for the cluster's partial sums (0: the rings are reused instead)
};

// ---- PTX wrappers specific to this kernel ---------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Both are executed by the whole (converged) MMA warp; one elected lane issues.  Keeping the warp converged lets the
// compiler hold addresses and descriptors in uniform registers instead of moving them there before every instruction.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile(
        "{\n"
        ".reg .pred pe;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
        "}\n" ::"r"(smem_u32(bar))
        : "memory");
}
// D[128, N] (+)= A[128, 16] (tensor memory) * B[16, N] (shared memory, K-major)
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, pe;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld4(uint32_t taddr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_cluster_f32(uint32_t local_addr, uint32_t rank, float v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}
__device__ __forceinline__ void arrive_remote(uint32_t local_bar_addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_bar_addr), "r"(rank));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// bounded wait with cluster-scope acquire (the data guarded by the barrier was written by other CTAs of the cluster)
__device__ __forceinline__ bool wait_bar_cluster(uint64_t* bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.b32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    atomicMax(&g_device_status, (int)EV_GEMV_FULL_WAIT);
    return false;
}
__device__ __forceinline__ uint32_t hadd2_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hfms2_u32(uint32_t a, uint32_t b, uint32_t c) {      // a * b - c; the negation is part of the instruction
    uint32_t r;
    asm("{\n.reg .b32 n;\nneg.f16x2 n, %3;\nfma.rn.f16x2 %0, %1, %2, n;\n}" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// A probe that suspends the warp for up to a microsecond.  The first probe of a wait is a plain one, all others are this: plain ones come back
// at once, and repeated by the waiting warps they took a third of a busy SM's issue slots from the dequantising ones (537 instructions
// per chunk and scheduler, 340 of them the dequantisation's).  Without -> with: 6144 x 4096 q4 for 32 rows 11.2 -> 10.4 us.
__device__ __forceinline__ bool probe_bar(uint32_t addr, uint32_t parity) {
    uint32_t got;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.b32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(got)
        : "r"(addr), "r"(parity), "r"(1000u)
        : "memory");
    return got != 0;
}
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, int event, bool& ok) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_try_wait(bar, parity)) return true;      // mostly it is there
    const uint32_t limit = ok ? kTsWaitLimit : 64u;
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i)
        if (probe_bar(addr, parity)) return true;
    atomicMax(&g_device_status, event);
    ok = false;
    return false;
}

// One wait of a warp for several barriers: lane i polls its own (address and parity per lane; lanes without one pass `need` false).
// For the operands of two chunks at once (gate and up, few columns): in turn is 1 % slower there, and so is suspending (14336 x 4096 q4, 32 rows).
// The two barriers of a single chunk are waited for in turn: together is 6 % slower, and one loop for both cases 7 % (gate and up of
// 11008 x 4096, 256 rows, 57 us).
__device__ __forceinline__ void wait_bars(uint32_t addr, uint32_t parity, bool need, int event, bool& ok) {
    const uint32_t limit = ok ? kTsWaitLimit : 64u;
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t got = 1;
        if (need)
            asm volatile(
                "{\n"
                ".reg .pred p;\n"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                "selp.b32 %0, 1, 0, p;\n"
                "}\n"
                : "=r"(got)
                : "r"(addr), "r"(parity)
                : "memory");
        if (__all_sync(0xffffffffu, got != 0)) return;
    }
    atomicMax(&g_device_status, event);
    ok = false;
}

// Per-group constants of the dequantisation, each duplicated into both halves of a register:
//   w = ((base + q) + c) * s + r,   c = -(base + zi),  zi = rint(z),  r = (zi - z) * s
// base: 1024 in both halves (q8), or 1024 / 64 for the low / high nibble of a byte (q4).
struct GroupConst { uint32_t s2, r2, c; };
template <int BITS>
__device__ __forceinline__ GroupConst group_const(uint32_t s_bits, uint32_t z_bits) {
    GroupConst c;
    c.s2 = prmt(s_bits, s_bits, 0x1010);
    const uint32_t z2 = prmt(z_bits, z_bits, 0x1010);
    // z rounded to an integer by adding and taking away 1536 with its sign (an even integer from 512 on: all that matters is that codes less zi
    // are exact, r holds the rest).  h2rint takes 16 clocks of a scheduler, this 4: gate and up of 14336 x 4096 q4 26.2 -> 25.1 us
    const uint32_t magic = (z2 & 0x80008000u) | 0x66006600u;
    const uint32_t zi2 = hsub2_u32(hadd2_u32(z2, magic), magic);
    c.r2 = hmul2_u32(hsub2_u32(zi2, z2), c.s2);
    c.c = hsub2_u32(BITS == 4 ? 0xD400E400u : 0xE400E400u, zi2);        // exact: integers below 2048
    return c;
}

// bf: the outputs are bf16 (a constant for weights in one term, which only fp16 calls have)
__device__ __forceinline__ float ts_round(bool bf, float v) {
    return bf ? __bfloat162float(__float2bfloat16_rn(v)) : __half2float(__float2half_rn(v));
}
__device__ __forceinline__ uint16_t ts_bits(bool bf, float v) {
    return bf ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}
__device__ __forceinline__ float ts_float(bool bf, uint16_t u) {
    return bf ? __uint_as_float((uint32_t)u << 16) : __half2float(__ushort_as_half(u));
}
// The residual values of output row n for 4 columns, fetched ahead of the accumulators and before the first store (y may
// alias the residual rows as far as the compiler knows).
template <int MATS>
__device__ __forceinline__ void ts_load_residual(const TsParams& p, int n, int b0, int nb, uint16_t (&res)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        res[j] = 0;
        if (MATS == 1 && p.residual != nullptr && n < p.N && j < nb) res[j] = p.residual[(size_t)(b0 + j) * p.N + n];
    }
}
// The epilogue of 4 columns (b0 .. b0 + nb of the batch): clamp, round, residual add or SwiGLU, store.
template <int MATS, bool SPLIT>
__device__ __forceinline__ void ts_store_cols(const TsParams& p, const float (&acc)[2][4], int n, int b0, int nb, const uint16_t (&res)[4]) {
    const bool bf = SPLIT && p.bf16;
    const float fmax_act = bf ? 3.3895313892515355e38f : 65504.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= nb) break;
        const int b = b0 + j;
        const size_t o = (size_t)b * p.N + n;
        const float cs = SPLIT && p.col_scale != nullptr ? p.col_scale[b] : 1.0f;
        if (MATS == 1) {
            float v = ts_round(bf, fminf(fmaxf((acc[0][j] + acc[1][j]) * cs, -fmax_act), fmax_act));
            if (p.residual != nullptr) v = ts_float(bf, res[j]) + v;
            p.y[o] = ts_bits(bf, v);
        } else {
            const float v0 = ts_round(bf, fminf(fmaxf(acc[0][j] * cs, -fmax_act), fmax_act));
            const float v1 = ts_round(bf, fminf(fmaxf(acc[1][j] * cs, -fmax_act), fmax_act));
            if (p.gate_out != nullptr) p.gate_out[o] = ts_bits(bf, v0);
            if (p.up_out != nullptr) p.up_out[o] = ts_bits(bf, v1);
            if (p.act_out != nullptr) p.act_out[o] = ts_bits(bf, (v0 / (1.0f + expf(-v0))) * v1);
        }
    }
}

// META: scales arrive by TMA (their rows are a multiple of 16 bytes), else the dequantise warps read them from global memory.
// SPLIT: weights in two fp16 terms, w = hi + lo with hi = (q - rint(z)) * s rounded and lo = what the rounding left out + (rint(z) - z) * s (see
// qgemm_ts for whom).  A chunk then holds 64 k: hi in its first 32 columns, lo in the others, both multiplied with the same
// activations.  14336 x 4096 q4, 32 bf16 rows: 26.4 us against 18.2 with one term and 93.8 of the mma.sync kernel.
template <int BITS, int LOGG, int MATS, bool META, bool SPLIT>
__global__ void __launch_bounds__(kTsThreads, 1) qgemm_ts_kernel(const __grid_constant__ TsParams p) {
    constexpr int KS = kRowBytes * 8 / BITS;           // k per stage: 256 (q4) or 128 (q8)
    constexpr int CK = chunk_k(SPLIT);                 // k per chunk
    constexpr int SC = KS / CK;                        // k-chunks per stage
    constexpr int APS = SC * MATS;                     // chunks of A per stage: 1, 2, 4 or 8
    constexpr int NG = kGroups;                        // chunk a (counted over the kernel) belongs to group a % NG
    constexpr int MS = (kMetaGroups << LOGG) / KS;     // stages per scale tile
    constexpr uint32_t kMetaBuf = MATS * 2 * kMetaTile;
    constexpr int CGR = CK >> LOGG > 1 ? CK >> LOGG : 1;      // scale groups of a chunk: 4, 2 or 1
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* const sbase = smem_raw + (base - smem_u32(smem_raw));

    uint64_t* bars = reinterpret_cast<uint64_t*>(sbase);
    uint64_t* full_w = bars;                            // [stages] codes of the stage have landed
    uint64_t* empty_w = full_w + kMaxStages;            // [stages] the dequantise warps are done with them
    uint64_t* full_x = empty_w + kMaxStages;            // [x_slots] a chunk of activations has landed
    uint64_t* empty_x = full_x + kMaxXSlots;            // [x_slots] the MMAs reading it are done
    uint64_t* a_full = empty_x + kMaxXSlots;            // [a_slots] a chunk of A is in tensor memory
    uint64_t* a_free = a_full + kMaxASlots;             // [a_slots] the MMAs reading it are done
    uint64_t* full_m = a_free + kMaxASlots;             // [meta_bufs] scales / zero points of kMetaGroups groups have landed
    uint64_t* empty_m = full_m + kMaxMetaBufs;          // [meta_bufs] every dequantise warp is done with them
    uint64_t* d_full = empty_m + kMaxMetaBufs;          // the item's accumulator is complete
    uint64_t* d_free = d_full + 1;                      // the epilogue has read the accumulator
    uint64_t* red_bar = d_free + 1;                     // first CTA of a cluster: the other CTAs' partial sums have arrived
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sbase + 768);
    const uint32_t stage0 = base + 1024;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = p.split > 1 ? cluster_rank() : 0u;
    const int first_item = (int)blockIdx.x / p.split;
    const int item_step = (int)gridDim.x / p.split;
    const int st_lo = (int)((int64_t)p.n_stage_total * rank / p.split);
    const int st_hi = (int)((int64_t)p.n_stage_total * (rank + 1) / p.split);
    const int n_st = st_hi - st_lo;
    const int my_items = first_item < p.items ? (p.items - first_item + item_step - 1) / item_step : 0;
    const int NS = p.stages;
    const int NA = p.a_slots;
    const int XS = p.x_slots;
    const int ncols = p.ncols;
    auto row_of = [&](int it) { return (first_item + it * item_step) / p.nblk * kRows; };        // column blocks of a tile run side by side
    auto col_of = [&](int it) { return (first_item + it * item_step) % p.nblk * ncols; };

    if (warp == kMmaWarp0) {
        if (lane < NS) { mbar_init(&full_w[lane], 1); mbar_init(&empty_w[lane], APS * 4); }
        if (lane < XS) { mbar_init(&full_x[lane], 1); mbar_init(&empty_x[lane], MATS); }
        if (lane < NA) { mbar_init(&a_full[lane], 4); mbar_init(&a_free[lane], 1); }
        if (META && lane < p.meta_bufs) { mbar_init(&full_m[lane], 1); mbar_init(&empty_m[lane], kDeqWarps); }
        if (lane == 0) {
            mbar_init(d_full, kMmaWarps);
            mbar_init(d_free, kDeqWarps);
            mbar_init(red_bar, p.split > 1 ? (uint32_t)(p.split - 1) * kDeqWarps * 32u : 1u);
        }
        mbar_fence_init();
    }
    if (warp == kTmaWarp) tmem_alloc(tmem_slot, 512u);
    tc_fence_before();
    __syncthreads();
    if (p.split > 1) cluster_sync_all();      // every CTA's barriers exist before a neighbour arrives on one
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_launch_dependents();

    // ================================ weight producer =============================================
    if (warp == kTmaWarp) {
        if (lane == 0) {
            bool ok = true;
            int slot = 0, mslot = 0;
            uint32_t par = 0, mpar = 0;
            const uint32_t meta_tx = MATS * kMetaTile * (p.has_z ? 2 : 1);
            for (int it = 0; it < my_items; ++it) {
                const int n0 = row_of(it);
                for (int s = st_lo; s < st_hi; ++s) {
                    if (META && (s == st_lo || s % MS == 0)) {      // scales / zero points of the next MS stages
                        wait_bar(&empty_m[mslot], mpar ^ 1u, EV_GEMV_EMPTY_WAIT, ok);
                        uint8_t* mb = sbase + p.off_meta + (size_t)mslot * kMetaBuf;
                        mbar_arrive_expect_tx(&full_m[mslot], meta_tx);
                        const int gx = s / MS * (kMetaGroups * 2);
#pragma unroll
                        for (int m = 0; m < MATS; ++m) {
                            tma_load_2d(mb + m * 2 * kMetaTile, &p.smap[m], gx, n0, &full_m[mslot]);
                            if (p.has_z) tma_load_2d(mb + m * 2 * kMetaTile + kMetaTile, &p.zmap[m], gx, n0, &full_m[mslot]);
                        }
                        if (++mslot == p.meta_bufs) { mslot = 0; mpar ^= 1u; }
                    }
                    wait_bar(&empty_w[slot], par ^ 1u, EV_GEMV_EMPTY_WAIT, ok);
                    uint8_t* st = sbase + 1024 + (size_t)slot * p.stage_bytes;
                    mbar_arrive_expect_tx(&full_w[slot], MATS * kWTile);
#pragma unroll
                    for (int m = 0; m < MATS; ++m) tma_load_2d(st + m * kWTile, &p.wmap[m], s * kRowBytes, n0, &full_w[slot]);
                    if (++slot == NS) { slot = 0; par ^= 1u; }
                }
            }
        }
    }
    // ================================ row producer ================================================
    else if (warp == kRowWarp) {
        pdl_wait();                           // the activations belong to the previous kernel until here
        if (lane == 0) {
            bool ok = true;
            int slot = 0;
            uint32_t par = 0;
            for (int it = 0; it < my_items; ++it) {
                const int c0 = col_of(it);
                for (int ch = st_lo * SC; ch < st_hi * SC; ++ch) {
                    wait_bar(&empty_x[slot], par ^ 1u, EV_GEMV_EMPTY_WAIT, ok);
                    uint8_t* dst = sbase + p.off_x + (size_t)slot * p.x_bytes;
                    mbar_arrive_expect_tx(&full_x[slot], p.x_bytes);
                    tma_load_2d(dst, &p.xmap, ch * CK * 2, c0, &full_x[slot]);                            // byte coordinates
                    if (!SPLIT) tma_load_2d(dst + (p.x_bytes >> 1), &p.xmap, ch * CK * 2 + 128, c0, &full_x[slot]);
                    if (++slot == XS) { slot = 0; par ^= 1u; }
                }
            }
        }
    }
    // ================================ MMA issuers =================================================
    else if (warp >= kMmaWarp0) {
        // warp j: matrix j of every chunk of k (two matrices), or the chunks of k with number = j modulo 2 (one matrix).  Two matrices and
        // few columns: two chunks per round of waits, where the rings are deep enough to hold one round and refill another
        // (gate and up, 14336 x 4096 q4: 27.6 -> 25.9 us for 8 rows; one matrix and more than 64 columns lose by it: 64 -> 71 us for 256)
        const int j = warp - kMmaWarp0;
        bool ok = true;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(ncols >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
        // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart, descriptor version 1
        const uint64_t desc_hi = ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61) | (1ull << 16);
        const uint32_t a_base = tmem + (uint32_t)p.a_col0;
        const uint32_t d_t = tmem + (uint32_t)(j * ncols);
        const uint32_t x0 = base + p.off_x;
        const uint32_t atom16 = (p.x_bytes >> 1) >> 4;                 // distance of the two 64-k atoms of a chunk, in 16-byte units
        const int n_ch = n_st * SC;
        const int per = MATS == 2 && ncols <= 64 && XS >= 4 && NA >= 5 ? 2 : 1;      // chunks per round
        const int first = ChunkWalk<MATS>::first(j);
        ChunkWalk<MATS> at(j);                                         // (NA >= 2)
        auto chunk = [&](int xs, int as, bool start) {
            const uint64_t desc0 = desc_hi | (uint64_t)(((x0 + (uint32_t)xs * p.x_bytes) & 0x3FFFFu) >> 4);
            const uint32_t a_t = a_base + (uint32_t)as * kChunkCols;
            tc_mma_ts(d_t, a_t, desc0, idesc, start ? 0u : 1u);
#pragma unroll
            for (int i = 1; i < 8; ++i)
                tc_mma_ts(d_t, a_t + i * 8, desc0 + (uint64_t)((SPLIT ? 0 : (i >> 2) * atom16) + (i & 3) * 2), idesc, 1u);
            tc_commit(&a_free[as]);
            tc_commit(&empty_x[xs]);
        };
        for (int it = 0; it < my_items; ++it) {
            if (it > 0) wait_bar(d_free, (uint32_t)(it - 1) & 1u, EV_GEMV_EMPTY_WAIT, ok);
            tc_fence_after();
            if (MATS == 2 && per == 2) {
#pragma unroll 1
                for (int ch = 0; ch < n_ch; ch += 2) {
                    at.to(it * n_ch + ch, XS, NA);
                    const RingPos x = at.x, a = at.a;
                    const bool two = ch + 1 < n_ch;
                    if (two) at.to(it * n_ch + ch + 1, XS, NA);
                    // lanes 0, 1: the first chunk's operands; lanes 2, 3: the second's
                    const uint32_t bar = lane == 0   ? smem_u32(&full_x[x.slot])
                                         : lane == 1 ? smem_u32(&a_full[a.slot])
                                         : lane == 2 ? smem_u32(&full_x[at.x.slot])
                                                     : smem_u32(&a_full[at.a.slot]);
                    const uint32_t par = lane == 0 ? x.par : lane == 1 ? a.par : lane == 2 ? at.x.par : at.a.par;
                    wait_bars(bar, par, lane < (two ? 4 : 2), EV_GEMV_FULL_WAIT, ok);
                    tc_fence_after();
                    chunk(x.slot, a.slot, ch == 0);
                    if (two) chunk(at.x.slot, at.a.slot, false);
                }
            } else {
#pragma unroll 1
                for (int ch = first; ch < n_ch; ch += 1 + ChunkWalk<MATS>::kSkip) {
                    at.to(it * n_ch + ch, XS, NA);
                    wait_bar(&full_x[at.x.slot], at.x.par, EV_GEMV_FULL_WAIT, ok);
                    wait_bar(&a_full[at.a.slot], at.a.par, EV_GEMV_FULL_WAIT, ok);
                    tc_fence_after();
                    chunk(at.x.slot, at.a.slot, ch == first);
                }
            }
            tc_commit(d_full);
        }
    }
    // ================================ dequantise warps + epilogue =================================
    else {
        const int grp = warp >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;                     // weight row inside the tile = lane of tensor memory
        const uint32_t sw = (uint32_t)(r & 7);
        const uint32_t msw = (uint32_t)((r >> 2) & 1) << 4;    // 32-byte swizzle of the scale tiles
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t row_u = stage0 + (uint32_t)r * kRowBytes;
        const bool second = n_st * SC > 1;                     // one matrix: the second accumulator is in use
        bool ok = true;
        int t = grp % NA;                                      // A slot of this group's next chunk
        uint32_t a_par = (uint32_t)(grp / NA) & 1u;
        int slot = 0;                                          // weight slot of stage `sl_at`
        uint32_t par = 0;
        int mslot = 0;
        uint32_t mpar = 0;
        const int n_ch = n_st * APS;                           // chunks of an item
        for (int it = 0; it < my_items; ++it) {
            const int n0 = row_of(it);
            int sl_at = 0;                                     // stage of the item that `slot` stands for
            int mt_at = 0;                                     // scale tile of the item that `mslot` stands for
            bool m_waited = false;
            const int mt0 = st_lo / MS;
            // scales and zero points of a chunk, read directly (META == false): one chunk ahead of their use
            uint32_t ns[2] = {0u, 0u}, nz[2] = {0u, 0u};
            auto fetch_meta = [&](int q) {
                const int s = st_lo + q / APS, u = q % APS, c = u / MATS, m = u % MATS;
                const int gi = (s * KS + c * CK) >> LOGG;
                ns[0] = ns[1] = nz[0] = nz[1] = 0u;
                if (n0 + r < p.N) {
                    const size_t at = (size_t)(n0 + r) * p.Gn + gi;
#pragma unroll
                    for (int j = 0; j < CGR; ++j)
                        if (gi + j < p.Gn) {
                            ns[j >> 1] |= (uint32_t)__ldg(p.s[m] + at + j) << (16 * (j & 1));
                            if (p.has_z) nz[j >> 1] |= (uint32_t)__ldg(p.z[m] + at + j) << (16 * (j & 1));
                        }
                }
            };
            const int a0 = (int)((uint32_t)it * (uint32_t)n_ch & (uint32_t)(NG - 1));      // chunk number of the item's first, modulo NG
            const int q0 = (grp - a0 + NG) & (NG - 1);
            if (!META && q0 < n_ch) fetch_meta(q0);
            // Up to four chunks a stage, a group always takes the same ones: their place in a stage is worked out once
            constexpr bool kSame = NG % APS == 0;
            constexpr int kPieces = CK * BITS / 128;           // 16-byte pieces of a chunk in one weight row
            uint32_t piece[kPieces];
            auto place = [&](int u) {
#pragma unroll
                for (int i = 0; i < kPieces; ++i) piece[i] = row_u + (uint32_t)((u % MATS) * kWTile) + ((((uint32_t)(u / MATS * kPieces + i)) ^ sw) << 4);
            };
            if (kSame) place(q0 % APS);
            const int u_same = q0 % APS;
#pragma unroll 1
            for (int q = q0; q < n_ch; q += NG) {
                const int sl = q / APS, u = kSame ? u_same : q % APS;
                const int s = st_lo + sl;
                const int c = u / MATS, m = u % MATS;
                slot += sl - sl_at;                            // at most NG / APS stages on
                sl_at = sl;
                if (slot >= NS) { slot -= NS; par ^= 1u; }     // a ring holds more stages than a group steps over
                if (!kSame) place(u);
                uint32_t sreg[2], zreg[2];
                if (META) {
                    const int mt = s / MS - mt0;
                    while (mt_at < mt) {                       // done with the scale tiles before (also one without a chunk of this group)
                        if (!m_waited) wait_bar(&full_m[mslot], mpar, EV_GEMV_FULL_WAIT, ok);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&empty_m[mslot]);
                        if (++mslot == p.meta_bufs) { mslot = 0; mpar ^= 1u; }
                        ++mt_at;
                        m_waited = false;
                    }
                }
                if (META && !m_waited) wait_bar(&full_m[mslot], mpar, EV_GEMV_FULL_WAIT, ok);
                wait_bar(&full_w[slot], par, EV_GEMV_FULL_WAIT, ok);
                if (META) {
                    m_waited = true;
                    const int g0 = ((s * KS + c * CK) >> LOGG) & (kMetaGroups - 1);      // first group of the chunk inside the scale tile
                    const uint32_t mrow = base + p.off_meta + (uint32_t)mslot * kMetaBuf + (uint32_t)(m * 2 * kMetaTile) +
                                          (uint32_t)r * (kMetaGroups * 2) + (((uint32_t)g0 * 2 & ~3u) ^ msw);
                    sreg[0] = lds32(mrow);
                    sreg[1] = CGR == 4 ? lds32(mrow + 4) : 0u;
                    zreg[0] = zreg[1] = 0u;
                    if (p.has_z) {
                        zreg[0] = lds32(mrow + kMetaTile);
                        if (CGR == 4) zreg[1] = lds32(mrow + kMetaTile + 4);
                    }
                    if (CGR == 1 && (g0 & 1)) { sreg[0] >>= 16; zreg[0] >>= 16; }
                } else {
                    sreg[0] = ns[0]; sreg[1] = ns[1]; zreg[0] = nz[0]; zreg[1] = nz[1];
                    if (q + NG < n_ch) fetch_meta(q + NG);
                }
                const uint32_t wslot = (uint32_t)slot * p.stage_bytes;
                const uint32_t a_t = lane_addr + (uint32_t)(p.a_col0 + t * kChunkCols);
                wait_bar(&a_free[t], a_par ^ 1u, EV_GEMV_EMPTY_WAIT, ok);
                tc_fence_after();
                // exact integers q - rint(z) of 32 k, in k order, two per register
                auto integers = [&](int k32, const GroupConst& gc, uint32_t* d) {
                    if (BITS == 4) {
                        const uint4 v = lds128(wslot + piece[k32]);
                        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            // byte j of the word holds k = 2j (low nibble) and 2j + 1: [byte, 0x64, byte, 0x54], nibbles masked
                            d[4 * w + 0] = hadd2_u32(prmt(w4[w], 0x00005464u, 0x5040) & 0xFFF0FF0Fu, gc.c);
                            d[4 * w + 1] = hadd2_u32(prmt(w4[w], 0x00005464u, 0x5141) & 0xFFF0FF0Fu, gc.c);
                            d[4 * w + 2] = hadd2_u32(prmt(w4[w], 0x00005464u, 0x5242) & 0xFFF0FF0Fu, gc.c);
                            d[4 * w + 3] = hadd2_u32(prmt(w4[w], 0x00005464u, 0x5343) & 0xFFF0FF0Fu, gc.c);
                        }
                    } else {
#pragma unroll
                        for (int q16 = 0; q16 < 2; ++q16) {
                            const uint4 v = lds128(wslot + piece[k32 * 2 + q16]);
                            const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int w = 0; w < 4; ++w) {
                                d[q16 * 8 + 2 * w] = hadd2_u32(prmt(w4[w], 0x64646464u, 0x4140u), gc.c);
                                d[q16 * 8 + 2 * w + 1] = hadd2_u32(prmt(w4[w], 0x64646464u, 0x4342u), gc.c);
                            }
                        }
                    }
                };
                auto constants = [&](int k32) {                // of the 32-k block's group
                    const int gi = (k32 * 32) >> LOGG;
                    return group_const<BITS>((gi & 1) ? sreg[gi >> 1] >> 16 : sreg[gi >> 1], (gi & 1) ? zreg[gi >> 1] >> 16 : zreg[gi >> 1]);
                };
                if constexpr (!SPLIT) {
#pragma unroll
                    for (int hb = 0; hb < 2; ++hb) {           // halves of the chunk: 64 k -> 32 columns
                        uint32_t out[32];
                        GroupConst gc;
#pragma unroll
                        for (int sb = 0; sb < 2; ++sb) {       // 32 k -> 16 columns
                            if (sb == 0 || LOGG == 5) gc = constants(hb * 2 + sb);
                            integers(hb * 2 + sb, gc, out + sb * 16);
#pragma unroll
                            for (int i = 0; i < 16; ++i) out[sb * 16 + i] = hfma2_u32(out[sb * 16 + i], gc.s2, gc.r2);
                        }
                        tc_st32(a_t + hb * 32, out);
                    }
                } else {
                    GroupConst gc;
#pragma unroll
                    for (int k32 = 0; k32 < 2; ++k32) {        // 32 k -> 16 columns of each term
                        if (k32 == 0 || LOGG == 5) gc = constants(k32);
                        uint32_t d[16], hi[16];
                        integers(k32, gc, d);
#pragma unroll
                        for (int i = 0; i < 16; ++i) hi[i] = hmul2_u32(d[i], gc.s2);
                        tc_st16(a_t + k32 * 16, hi);
#pragma unroll
                        for (int i = 0; i < 16; ++i) d[i] = hadd2_u32(hfms2_u32(d[i], gc.s2, hi[i]), gc.r2);
                        tc_st16(a_t + 32 + k32 * 16, d);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty_w[slot]);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[t]);
                t += NG;
                if (t >= NA) { t -= NA; a_par ^= 1u; }
            }
            // step over the rest of the item's stages and scale tiles
            slot += n_st - sl_at;
            while (slot >= NS) { slot -= NS; par ^= 1u; }
            if (META && n_st > 0) {
                const int mt_end = (st_hi - 1) / MS - mt0 + 1;
                while (mt_at < mt_end) {
                    if (!m_waited) wait_bar(&full_m[mslot], mpar, EV_GEMV_FULL_WAIT, ok);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty_m[mslot]);
                    if (++mslot == p.meta_bufs) { mslot = 0; mpar ^= 1u; }
                    ++mt_at;
                    m_waited = false;
                }
            }
            // ---- epilogue of the item (split == 1; with a split K range it follows the cluster exchange below): each group of warps takes
            //      4 columns of every 16 ----
            if (p.split == 1) {
                if (it == 0) pdl_wait();
                const int n = n0 + r, c0 = col_of(it) + grp * 4;
                uint16_t res[4];
                ts_load_residual<MATS>(p, n, c0, p.B - c0, res);
                wait_bar(d_full, (uint32_t)it & 1u, EV_GEMV_FULL_WAIT, ok);
                tc_fence_after();
#pragma unroll 1
                for (int cs = 0; cs < ncols; cs += 16) {
                    const int nb = p.B - c0 - cs;              // may be more than 4
                    if (nb <= 0) break;
                    uint16_t next[4];
                    ts_load_residual<MATS>(p, n, c0 + cs + 16, cs + 16 < ncols ? nb - 16 : 0, next);
                    float acc[2][4] = {};
                    tc_ld4(lane_addr + (uint32_t)(cs + grp * 4), acc[0]);
                    if (MATS == 2 || second) tc_ld4(lane_addr + (uint32_t)(ncols + cs + grp * 4), acc[1]);
                    if (n < p.N) ts_store_cols<MATS, SPLIT>(p, acc, n, c0 + cs, nb, res);
#pragma unroll
                    for (int j = 0; j < 4; ++j) res[j] = next[j];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_free);
            }
        }
    }

    // ---- split K range (one item per cluster): the partial accumulators are summed in rank order by the cluster's first CTA.  Small
    //      batches send only their real columns into a dedicated buffer and signal a barrier of the first CTA; otherwise the first
    //      CTA's rings are reused between two cluster-wide barriers. ----
    if (p.split > 1) {
        __syncwarp();
        const int grp = warp >> 2;
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const bool fast = p.off_red != 0;
        const int c0 = col_of(0);
        const int bcols = min(ncols, p.B - c0);               // real columns of the block
        const int rcols = fast ? min(ncols, p.B) : ncols;     // columns per matrix and part in the buffer
        const uint32_t red_base = fast ? base + p.off_red : stage0;
        const bool epi = warp < kDeqWarps && my_items > 0;
        bool ok = true;
        if (epi) {
            wait_bar(d_full, 0u, EV_GEMV_FULL_WAIT, ok);
            tc_fence_after();
        }
        if (!fast) cluster_sync_all();      // every CTA of the cluster is done with its rings: the first CTA's are free
        const bool second = n_st * SC > 1;                    // one matrix: the second accumulator is in use
        if (epi && rank != 0) {
#pragma unroll 1
            for (int cs = grp * 4; cs < bcols; cs += 16) {
                float acc[2][4] = {};
                tc_ld4(lane_addr + (uint32_t)cs, acc[0]);
                if (MATS == 2 || second) tc_ld4(lane_addr + (uint32_t)(ncols + cs), acc[1]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (cs + j >= bcols) break;
#pragma unroll
                    for (int m = 0; m < MATS; ++m)
                        st_cluster_f32(red_base + (uint32_t)(((((int)rank - 1) * MATS + m) * rcols + cs + j) * kRows + r) * 4u, 0u,
                                       MATS == 1 ? acc[0][j] + acc[1][j] : acc[m][j]);
                }
            }
            if (fast) arrive_remote(smem_u32(red_bar), 0u);
        }
        if (!fast) cluster_sync_all();      // the partial sums are in the first CTA's shared memory
        if (epi && rank == 0) {
            pdl_wait();
            const int n = row_of(0) + r;
            const float* red = reinterpret_cast<const float*>(sbase + (red_base - base));
            uint16_t res[4];
            ts_load_residual<MATS>(p, n, c0 + grp * 4, bcols - grp * 4, res);
            if (fast) wait_bar_cluster(red_bar, 0u, ok ? kTsWaitLimit : 64u);
#pragma unroll 1
            for (int cs = grp * 4; cs < bcols; cs += 16) {
                uint16_t next[4];
                ts_load_residual<MATS>(p, n, c0 + cs + 16, bcols - cs - 16, next);
                float acc[2][4] = {};
                tc_ld4(lane_addr + (uint32_t)cs, acc[0]);
                if (MATS == 2 || second) tc_ld4(lane_addr + (uint32_t)(ncols + cs), acc[1]);
                if (MATS == 1) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { acc[0][j] += acc[1][j]; acc[1][j] = 0.0f; }
                }
                for (int q = 1; q < p.split; ++q)
#pragma unroll
                    for (int m = 0; m < MATS; ++m)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (cs + j < bcols) acc[m][j] += red[((((q - 1) * MATS + m) * rcols + cs + j) * kRows + r)];
                if (n < p.N) ts_store_cols<MATS, SPLIT>(p, acc, n, c0 + cs, bcols - cs, res);
#pragma unroll
                for (int j = 0; j < 4; ++j) res[j] = next[j];
            }
        }
        // the first CTA must not leave while its neighbours still store into it
        if (fast && rank == 0 && epi) wait_bar_cluster(red_bar, 0u, ok ? kTsWaitLimit : 64u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kTmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem, 512u);
    }
}

// ---- host side ---------------------------------------------------------------------------------------------------
struct MapKey {
    const void* ptr; uint64_t d0, d1; uint32_t b0, b1, swz;
    bool operator==(const MapKey& o) const { return ptr == o.ptr && d0 == o.d0 && d1 == o.d1 && b0 == o.b0 && b1 == o.b1 && swz == o.swz; }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        size_t h = std::hash<const void*>()(k.ptr);
        h = h * 1000003u ^ std::hash<uint64_t>()(k.d0 * 31 + k.d1);
        h = h * 1000003u ^ std::hash<uint64_t>()(((uint64_t)k.b0 << 32) | (k.b1 * 4 + k.swz));
        return h;
    }
};
std::mutex g_map_mu;
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;

// 2-D byte tensor [d1 rows, d0 bytes] (rows d0 bytes apart), box b0 x b1.
bool tensor_map_2d(const void* ptr, uint64_t d0, uint64_t d1, uint32_t b0, uint32_t b1, CUtensorMapSwizzle swizzle, CUtensorMap* out) {
    const MapKey key = {ptr, d0, d1, b0, b1, (uint32_t)swizzle};
    std::lock_guard<std::mutex> lock(g_map_mu);
    auto it = g_maps.find(key);
    if (it != g_maps.end()) { *out = it->second; return true; }
    const PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {d0, d1};
    const cuuint64_t strides[1] = {d0};
    const cuuint32_t box[2] = {b0, b1};
    const cuuint32_t estr[2] = {1, 1};
    CUtensorMap m;
    const CUresult rc = encode(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return false;
    if (g_maps.size() > 4096) g_maps.clear();
    g_maps.emplace(key, m);
    *out = m;
    return true;
}

inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Clusters of `size` CTAs of one SM each that can be resident together: GPCs are not a multiple of every size.
template <typename Kernel>
int max_clusters(Kernel kernel, int size, uint32_t smem) {
    static int cached[64][9] = {};      // per device; a race only repeats the query (all instantiations have one CTA per SM)
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = cached[dev & 63][size];
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(size);
        cfg.blockDim = dim3(kTsThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int got = 0;
        if (cudaOccupancyMaxActiveClusters(&got, kernel, &cfg) != cudaSuccess || got <= 0) {
            cudaGetLastError();
            got = std::max(1, sm_count() / size);
        }
        n = got;
    }
    return n;
}

template <int BITS, int LOGG, int MATS, bool META, bool SPLIT>
int launch_ts(TsParams& p, int K, cudaStream_t stream) {
    constexpr int KS = kRowBytes * 8 / BITS;
    constexpr int CK = chunk_k(SPLIT), SC = KS / CK;
    constexpr int MS = (kMetaGroups << LOGG) / KS;         // stages per scale tile
    constexpr uint32_t kMetaBuf = META ? MATS * 2 * kMetaTile : 0;
    const int sms = sm_count();
    const int tiles = (p.N + kRows - 1) / kRows;
    p.n_stage_total = (K + KS - 1) / KS;
    p.stage_bytes = MATS * kWTile;
    auto kernel = qgemm_ts_kernel<BITS, LOGG, MATS, META, SPLIT>;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t cap = (uint32_t)max_smem_optin();
    if (!configured[dev & 63]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) != cudaSuccess)
            return B200Q_ERR_LAUNCH;
        configured[dev & 63] = true;
    }
    // Column blocks and K split by estimated time, in clocks: rounds of items over the SMs, each a chain of chunks whose cost is the
    // dequantisation's (450; 64 k in two terms 540) or the tensor pipe's: 22 clocks per MMA up to 32 columns, then half a clock per column,
    // and 260 a chunk in which the next chunk's way into tensor memory keeps it waiting (no arithmetic at all: 530 clocks at 64
    // columns, 650 at 96).  The first CTA of a cluster takes about 35 clocks per column and part for the partial sums.  The choice
    // must not depend on how many rows THIS launch holds: a tensor-parallel shard of the rows has to reproduce the unsharded result
    // bit for bit, so the tile count of the unsharded matrix decides ("ts.tp_world" = number of equal row shards).
    const int tiles_full = tiles * std::max(1, tuning_get("ts.tp_world"));
    const int forced = tuning_get("ts.split");
    // bytes of partial sums: in a dedicated buffer (4096 x 14336 q4: 72 KB, 48 rows, 17.0 us, through the rings 17.7; 96 KB, 64 rows, which leave
    // the rings too little, 19.8 and 18.7), and at all (not beyond 48 KB, and so fewer parts: 24.3 and 24.6)
    constexpr uint32_t kRedCap = 80u * 1024u, kRedMax = 128u * 1024u;
    double best = 0.0;
    int cols = 0, split = 1;
    const int nb0 = (p.B + kMaxCols - 1) / kMaxCols;
    for (int nb = nb0; nb <= (p.B + 15) / 16 && nb <= 4 * nb0; ++nb) {
        const int c = ((p.B + nb - 1) / nb + 15) / 16 * 16;
        const int blocks = (p.B + c - 1) / c;
        if (blocks != nb) continue;                        // the same blocks as a smaller nb
        const double chunk = std::max(SPLIT ? 540.0 : 450.0, 8.0 * std::max(22.2, c * 0.5 + 0.8) + 260.0);
        for (int sp = 1; sp <= 8; sp *= 2) {
            if (forced > 0 ? sp != std::min(forced, std::max(1, p.n_stage_total)) : sp > 1 && sp > p.n_stage_total / 2) continue;
            if (forced <= 0 && sp > 1 && (uint32_t)(sp - 1) * MATS * c * kRows * 4 > kRedMax) continue;
            const int64_t items = (int64_t)tiles_full * blocks;
            const int slots = sp == 1 ? sms : max_clusters(kernel, sp, cap - 2048u);
            if (forced <= 0 && sp > 1 && items > slots) continue;
            const double rounds = (double)((items + slots - 1) / slots);
            const double item = (double)((p.n_stage_total + sp - 1) / sp * SC * MATS) * chunk + 1500.0 + c * MATS * 10.0;
            const double t = rounds * item + (sp > 1 ? 1500.0 + 35.0 * (sp - 1) * MATS * std::min(c, p.B) : 0.0);
            if (cols == 0 || t < best) { best = t; cols = c; split = sp; }
        }
    }
    if (cols == 0) return B200Q_ERR_UNSUPPORTED;
    p.ncols = cols;
    p.nblk = (p.B + cols - 1) / cols;
    p.items = tiles * p.nblk;
    p.split = split;
    // tensor memory: accumulators below, ring of A chunks above
    const int dcols = 2 * cols;
    p.a_col0 = std::max(32, (dcols + 31) / 32 * 32);
    // A barrier is waited for by its parity, so whoever waits on a slot has to know that the slot's phase before has ended.  Ring depths
    // see to that: an even number of A slots (and, one matrix, of activation slots) gives every slot to the same MMA warp each time
    // round within an item, and a stage slot serves the same groups of warps each time (chunk n goes to group n modulo kGroups).
    // From one item to the next the MMA warps of one matrix change places when an item has an odd number of chunks; their wait for d_free
    // in between covers it, since the accumulators are read only after every chunk of the item has been consumed.  Four A slots or
    // more cover the groups' waits for a free one: the chunk a group wrote before lies at most one round of the ring back.
    p.a_slots = std::min(kMaxASlots, (512 - p.a_col0) / kChunkCols) & ~1;
    constexpr int kXStep = MATS == 2 ? 1 : 2;
    constexpr int kStageStep = std::max(1, kGroups / (SC * MATS));
    // partial sums of a K split: a dedicated buffer signalled by a barrier, else the first CTA's rings between two cluster-wide
    // barriers; both add them in rank order
    const uint32_t red_bytes = (uint32_t)(split - 1) * MATS * std::min(cols, p.B) * kRows * 4;
    const bool fast_red = split > 1 && red_bytes <= kRedCap && !tuning_get("ts.slow_reduce");
    const uint32_t red_alloc = fast_red ? (red_bytes + 1023u) / 1024u * 1024u : 0u;
    // rings: scale tiles so deep that the producer never waits for one before it waits for a weight stage, then activation chunks
    // and weight stages share what is left
    auto meta_bufs_for = [](int stages) { return META ? std::min(kMaxMetaBufs, (stages + MS - 1) / MS + 1) : 0; };
    p.x_bytes = (uint32_t)cols * CK * 2;
    const uint32_t budget = cap - 2048u - red_alloc;       // 1 KB of barriers, up to 1 KB of alignment
    auto need = [&](int xs, int stages) {
        return (uint32_t)xs * p.x_bytes + (uint32_t)stages * p.stage_bytes + (uint32_t)meta_bufs_for(stages) * kMetaBuf;
    };
    const int want = tuning_get("ts.stages");
    int xs = std::min(kMaxXSlots, std::max(2, (int)(64u * 1024u / p.x_bytes))) / kXStep * kXStep;
    constexpr int kMinStages = std::max(2, kStageStep);
    int stages = (want > 0 ? std::max(kMinStages, std::min(kMaxStages, want)) : kMaxStages) / kStageStep * kStageStep;
    while (stages > kMinStages + kStageStep && need(xs, stages) > budget) stages -= kStageStep;
    while (xs > 2 && need(xs, stages) > budget) xs -= kXStep;
    while (stages > kMinStages && need(xs, stages) > budget) stages -= kStageStep;
    if (need(xs, stages) > budget) return B200Q_ERR_UNSUPPORTED;
    p.stages = stages;
    p.x_slots = xs;
    p.meta_bufs = meta_bufs_for(stages);
    p.off_x = 1024u + (uint32_t)stages * p.stage_bytes;
    p.off_meta = p.off_x + (uint32_t)xs * p.x_bytes;
    const uint32_t rings_end = p.off_meta + (uint32_t)p.meta_bufs * kMetaBuf;
    p.off_red = fast_red ? rings_end : 0u;
    // only with a split or few stages by request ("ts.split", "ts.stages")
    if (split > 1 && !fast_red && (uint64_t)(split - 1) * MATS * cols * kRows * 4 > (uint64_t)rings_end - 1024u) return B200Q_ERR_UNSUPPORTED;

    if (!tensor_map_2d(p.x, (uint64_t)K * 2, (uint64_t)p.B, 128, (uint32_t)cols, CU_TENSOR_MAP_SWIZZLE_128B, &p.xmap)) return B200Q_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(split > 1 ? p.items * split : std::min(p.items, sms));
    cfg.blockDim = dim3(kTsThreads);
    cfg.dynamicSmemBytes = std::max(1024u + rings_end + red_alloc, cap / 2 + 2048u);      // one CTA per SM (it takes all of the tensor memory)
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (!tuning_get("no_pdl")) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (split > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = split;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    if (cudaLaunchKernelEx(&cfg, kernel, p) != cudaSuccess) return B200Q_ERR_LAUNCH;
    return finish_launch();
}

template <int BITS, int LOGG, int MATS>
int dispatch_ts_form(TsParams& p, int K, bool meta, bool split, cudaStream_t stream) {
    if (!meta) return launch_ts<BITS, LOGG, MATS, false, true>(p, K, stream);
    return split ? launch_ts<BITS, LOGG, MATS, true, true>(p, K, stream) : launch_ts<BITS, LOGG, MATS, true, false>(p, K, stream);
}
template <int BITS, int LOGG>
int dispatch_ts_mats(TsParams& p, int K, bool gate_up, bool meta, bool split, cudaStream_t stream) {
    return gate_up ? dispatch_ts_form<BITS, LOGG, 2>(p, K, meta, split, stream) : dispatch_ts_form<BITS, LOGG, 1>(p, K, meta, split, stream);
}
template <int BITS>
int dispatch_ts(TsParams& p, int K, int G, bool gate_up, bool meta, bool split, cudaStream_t stream) {
    if (G == 32) return dispatch_ts_mats<BITS, 5>(p, K, gate_up, meta, split, stream);
    if (G == 64) return dispatch_ts_mats<BITS, 6>(p, K, gate_up, meta, split, stream);
    return dispatch_ts_mats<BITS, 7>(p, K, gate_up, meta, split, stream);
}

}  // namespace

// Whether this kernel takes a problem (without looking at the norm prologue, which callers run as a launch of its own).  bf16 rows
// need `col_scale`: the caller has put them into fp16 with a power of two per row.
bool qgemm_ts_applies(const GemvParams& g, bool gate_up) {
    if (g.scale_dtype != B200Q_F16 || (g.act_dtype != B200Q_F16 && g.col_scale == nullptr)) return false;
    if (g.G != 32 && g.G != 64 && g.G != 128) return false;
    if (g.K % g.G != 0 || g.K % 8 != 0 || g.row_bytes % 16 != 0 || g.tp_in.world > 0 || g.tp_out.world > 0) return false;
    for (int m = 0; m < (gate_up ? 2 : 1); ++m)
        if (!al16(g.w[m])) return false;
    if (gate_up && ((g.z[0] == nullptr) != (g.z[1] == nullptr))) return false;
    return al16(g.x);
}

// Returns B200Q_ERR_UNSUPPORTED when the problem is outside this kernel (the caller then uses the other kernels).
int qgemm_ts(int bits, const GemvParams& g, bool gate_up, cudaStream_t stream) {
    if (!qgemm_ts_applies(g, gate_up) || g.norm_w != nullptr) return B200Q_ERR_UNSUPPORTED;
    const int mats = gate_up ? 2 : 1;
    bool meta = g.Gn % 8 == 0;
    for (int m = 0; m < mats; ++m) meta = meta && al16(g.s[m]) && al16(g.z[m]);
    TsParams p = {};
    p.B = g.B; p.N = g.N; p.Gn = g.Gn; p.has_z = g.z[0] != nullptr ? 1 : 0;
    p.bf16 = g.act_dtype == B200Q_BF16;
    p.col_scale = g.col_scale;
    for (int m = 0; m < mats; ++m) {
        p.s[m] = (const uint16_t*)g.s[m];
        p.z[m] = (const uint16_t*)g.z[m];
        if (!tensor_map_2d(g.w[m], (uint64_t)g.row_bytes, (uint64_t)g.N, kRowBytes, kRows, CU_TENSOR_MAP_SWIZZLE_128B, &p.wmap[m])) return B200Q_ERR_UNSUPPORTED;
        if (!meta) continue;
        if (!tensor_map_2d(g.s[m], (uint64_t)g.Gn * 2, (uint64_t)g.N, kMetaGroups * 2, kRows, CU_TENSOR_MAP_SWIZZLE_32B, &p.smap[m])) return B200Q_ERR_UNSUPPORTED;
        if (g.z[m] != nullptr &&
            !tensor_map_2d(g.z[m], (uint64_t)g.Gn * 2, (uint64_t)g.N, kMetaGroups * 2, kRows, CU_TENSOR_MAP_SWIZZLE_32B, &p.zmap[m]))
            return B200Q_ERR_UNSUPPORTED;
    }
    p.residual = (const uint16_t*)g.residual; p.y = (uint16_t*)g.y; p.gate_out = (uint16_t*)g.gate_out; p.up_out = (uint16_t*)g.up_out;
    p.act_out = (uint16_t*)g.act_out;
    p.x = g.x;
    // Weights in two terms where the kernel that these calls had before, fp16 mma.sync with up to 16 rows a launch, takes codes and scales
    // unrounded: bf16 rows, and scale rows that no tensor copy can fetch.  Relative error against fp64, 12 x 4561 x 1280 q4 groups
    // of 128: 2.93e-4 with one term, 2.07e-4 with two (the result's own rounding).
    const bool split = p.bf16 || !meta;
    return bits == 4 ? dispatch_ts<4>(p, g.K, g.G, gate_up, meta, split, stream) : dispatch_ts<8>(p, g.K, g.G, gate_up, meta, split, stream);
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess) fn = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    return encode;
}

}  // namespace b200q
