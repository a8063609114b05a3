// Paged quantized-KV GQA decode attention (q4 / q8 symmetric, fp16 scales) for sm_100a.
//
//   out[b, hq] = softmax_j( scale * q[b, hq] . Khat[j, hkv] ) . Vhat[j, hkv],  hkv = hq / (Hq/Hkv)
//   Khat = fp16((code - 8|128) * |k_scale|)   over the valid tokens j of sequence b.
//
// Fast kernels (head_dim 128, page size 16, q in fp16 or bf16, at most 8 query heads per kv head; quantised pages with fp16 scales in
// groups of 32 or 64, or plain pages in the dtype of q):
//   * the (sequence, page) pairs of the whole batch form one flattened list that is cut into
//     equal contiguous ranges, one per CTA ("stream-K" over ragged lengths: every CTA streams the
//     same number of pages whatever the length distribution).  A CTA writes one partial
//     (max, sum, accumulator) per sequence it touches; a second small kernel merges them.
//   * warp w of a CTA owns kv head w % Hkv (and, when there are fewer than 8 kv heads, every
//     (8/Hkv)-th page of the range; more than 8 kv heads are cut into chunks of 8, grid.y).  A ninth warp looks up the page ids and
//     fetches every page for all the CTA's heads with tensor copies into a ring in shared memory, several pages ahead.
//   * what a warp does with a page is in paged_attn_page.cuh.
//
// Everything else (other head dims, other group sizes) runs the simple kernel: one
// warp per (sequence, query head), the reference's streaming-softmax loop.
#include "attn_route.h"
#include "paged_attn_page.cuh"
#include "tensor_map.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace b200q {

B200Q_DEFINE_STATUS_WORD(attn_read_status)

namespace {

constexpr int kAttnWarps = 8;
constexpr int kAttnThreads = kAttnWarps * 32;
#ifndef B200Q_ATTN_CTAS
#define B200Q_ATTN_CTAS 2                    // resident CTAs per SM of the fast kernel's dense shape
#endif
constexpr int kMaxGrid = 152 * B200Q_ATTN_CTAS;   // upper bound on CTAs of the fast kernel (sizes the workspace)
constexpr int kMaxRanges = 4 * kMaxGrid;  // upper bound on page ranges: a CTA holds several when there are fewer than 8 kv heads
constexpr int kMaxBatchFast = 2048;       // prefix sums of page counts live in shared memory
using namespace attn;

struct AttnParams {
    const void* q;              // [B, Hq, D]
    const uint8_t* k_codes;
    const uint8_t* v_codes;
    const __half* k_scales;
    const __half* v_scales;
    const int32_t* block_table; // [B, max_blocks]
    const int32_t* lengths;     // [B]
    float* partial;             // [grid + B][Hq][D + 2]  (acc[D], max, sum); slot = range + sequence
    void* out;                  // [B, Hq, D]
    int B, Hq, Hkv, D, P, max_blocks, G, Gd, group;
    int64_t num_pages;
    float scale;
    int q_dtype;
    int bits;
    int stages;                 // pages in flight per range
    int subs;                   // ranges per CTA (8 / hc)
    int hc;                     // kv heads per CTA: Hkv, at most 8
    int row_bytes;              // bytes of one token row of codes, all kv heads
    int scale_row_halves;       // halves of one token row of scales, all kv heads
    int scales8;                // the scales are aligned to 8 bytes only: no bulk copies of them
    uint32_t off_bars, off_desc, off_prefix, slot_bytes;      // the ring comes first
    int grid;
    int sink, window;           // window > 0: only positions < sink or >= length - window are attended
    TpOut tp_out;               // tensor-parallel exchange of the merged rows (world == 0: off)
    int32_t* verdict;           // host-visible word: 1 or 2 once the lengths are read, all in range or not (null: off)
};

__device__ __forceinline__ int clamp_len(int len, int cap) { return max(0, min(len, cap)); }

// Pages of one sequence that hold at least one attended position.  Dense: all of them.  With a window: the
// pages of the sink tokens that lie below the window, then the pages from the window's first position on.
struct SeqPages { int n, sink_pages, first_recent, L; };
__device__ __forceinline__ SeqPages seq_pages(int len, int cap, int P, int sink, int window) {
    const int L = clamp_len(len, cap);
    const int n_all = (L + P - 1) / P;
    if (window <= 0 || L <= 0) return {n_all, n_all, n_all, L};
    const int lo = max(0, L - window);
    const int sink_pages = (min(sink, lo) + P - 1) / P;
    const int first_recent = max(sink_pages, lo / P);
    return {sink_pages + n_all - first_recent, sink_pages, first_recent, L};
}
// bit t set: slot t of page pg (16 slots) is an attended position of a sequence of L tokens
__device__ __forceinline__ uint32_t page_mask16(int pg, int L, int sink, int window) {
    const int valid = min(16, L - pg * 16);
    uint32_t m = valid >= 16 ? 0xFFFFu : ((1u << max(valid, 0)) - 1u);
    if (window > 0) {
        const int lo_t = max(0, L - window) - pg * 16;      // first slot of the window in this page
        const int sink_t = sink - pg * 16;                    // slots below this are sink tokens
        const uint32_t recent = lo_t <= 0 ? 0xFFFFu : (lo_t >= 16 ? 0u : (0xFFFFu << lo_t) & 0xFFFFu);
        const uint32_t sinks = sink_t <= 0 ? 0u : (sink_t >= 16 ? 0xFFFFu : (1u << sink_t) - 1u);
        m &= recent | sinks;
    }
    return m;
}

// Prefix sums of per-sequence page counts into shared memory; returns the total.
__device__ int build_prefix(const AttnParams& p, int* prefix) {
    // executed by every thread of the CTA up to the final __syncthreads
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int running = 0;
        for (int b0 = 0; b0 < p.B; b0 += 32) {
            const int b = b0 + lane;
            int n = 0;
            if (b < p.B) n = seq_pages(p.lengths[b], p.max_blocks * p.P, p.P, p.sink, p.window).n;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (b < p.B) prefix[b] = running + incl - n;
            running += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) prefix[p.B] = running;
    }
    __syncthreads();
    return prefix[p.B];
}

// largest b with prefix[b] <= f (f < prefix[B])
__device__ __forceinline__ int find_sequence(const int* prefix, int B, int f) {
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= f) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The split-KV kernel: eight consumer warps (process_page) and one producer warp.
// Bound by HBM (a page of q8 codes and scales is 4.3 KB per kv head: 181 clocks of an SM's share).  What held it back before was the
// path into shared memory: every warp copied its own head's pages with 16-byte cp.async pieces and 8-byte pieces of scales - 9 (q8) or
// 17 (plain) such instructions per page and head, 64 L2 requests - and the warps' ldmatrix, shuffles and conversions queued behind
// them (5 of 12.5 clocks per instruction on short scoreboards, issue 31 %): 303 clocks per page and head, 81 us for 32 x 4097 q8
// tokens of 8 kv heads (0.55 of the copy rate).  Now one elected lane fetches a page for ALL heads of the block: two
// 3-D tensor copies (row, token, head) whose swizzle is what ldmatrix wants, and two copies of the scales.
// The producer also looks up the page descriptors, 32 at a time, and leaves them in shared memory.
// TWO: two CTAs per SM, 16 consumer warps; otherwise (grids that do not fill the SMs twice, plain pages of 64 KB) one with a deeper ring.
constexpr int kSplitThreads = kAttnThreads + 32;
constexpr int kMaxRing = 16;                  // pages in flight per range
constexpr uint32_t kAttnWaitLimit = 1u << 20;
constexpr int kDescSlots = 64;                // descriptors per range: the window being issued and the one before (a ring is shorter than 32)

struct alignas(64) SplitParams {
    CUtensorMap kmap, vmap;     // codes (or values) as bytes [heads (x 2)][tokens][64 or 128], box hc (x 2) x 16 x row
    CUtensorMap ksmap, vsmap;   // scales as bytes [tokens][row], box 16 x (hc heads); used with more than 8 kv heads only
    AttnParams a;
};
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }
// A hint: bring a box into L2.
__device__ __forceinline__ void prefetch_box_3d(const CUtensorMap* map, int x, int y, int z) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// bytes of one range's ring slot: K tiles, V tiles, scales of K, scales of V; a multiple of the swizzle's repeat
__host__ __device__ constexpr uint32_t split_scale_bytes(int hc, int Gd) { return (uint32_t)(16 * hc * Gd * 2); }
__host__ __device__ constexpr uint32_t split_slot_bytes(int bits, int hc, int Gd) {
    const uint32_t tiles = (uint32_t)(2 * hc * 16 * kHeadDim * bits / 8), sc = bits == 16 ? 0u : 2 * split_scale_bytes(hc, Gd);
    return (tiles + sc + 1023u) & ~1023u;
}

// Scales that are aligned to 8 bytes only (a view that starts inside a tensor): copied by a whole warp in 8-byte pieces, `rows` rows of
// `row8` pieces that lie `pitch` bytes apart, into the same place and order as the bulk copies.  Every lane then arrives on the
// slot's barrier (whose count includes the 32 lanes) when its pieces are there.  16 x 4096 tokens of q4, 8 kv heads: 40 us against
// 38 us aligned, one cold call by events; the kernel for every shape, one warp per head, took 7675 us.
__device__ __forceinline__ void copy_scales8(uint32_t dst, const void* src, int rows, int row8, int64_t pitch, int lane) {
    for (int i = lane; i < rows * row8; i += 32) {
        const int r = i / row8;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + (uint32_t)i * 8),
                     "l"(static_cast<const uint8_t*>(src) + r * pitch + (i - r * row8) * 8) : "memory");
    }
}
__device__ __forceinline__ void arrive_on_copies(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int BITS, int LOGG, bool TWO, bool WIDE>
__global__ void __launch_bounds__(kSplitThreads, TWO ? B200Q_ATTN_CTAS : 1) paged_attn_kernel(const __grid_constant__ SplitParams sp) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const AttnParams& p = sp.a;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int D = kHeadDim;
    constexpr int TILE = PageShape<BITS>::TILE;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int NS = p.stages, subs = p.subs, hc = p.hc;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.off_bars);        // [subs][NS]
    uint64_t* empty = full + subs * NS;
    uint2* desc = reinterpret_cast<uint2*>(smem + p.off_desc);              // [subs][kDescSlots]: page, sequence << 16 | attended slots
    int* prefix = reinterpret_cast<int*>(smem + p.off_prefix);              // [B + 1]
    const uint32_t ring = smem_u32(smem);                                   // [subs][NS] slots

    if (threadIdx.x == kAttnThreads) {
        prefetch_map(&sp.kmap);
        prefetch_map(&sp.vmap);
    }
    if (threadIdx.x < subs * NS) {
        mbar_init(&full[threadIdx.x], BITS != 16 && p.scales8 ? 33 : 1);
        mbar_init(&empty[threadIdx.x], hc);
    }
    mbar_fence_init();
    __syncthreads();

    // The flattened page list is cut into p.grid equal ranges.  A CTA has 8 consumer warps = 8 (range, kv head) pairs:
    // with 8 kv heads one range, with fewer heads several consecutive ranges (subs of them).  Up to 32 sequences, every warp
    // keeps their lengths and page counts in its lanes: one load and a scan, no shared memory and no barrier.
    const bool small = p.B <= 32;
    const int cap = p.max_blocks * p.P;
    int len_l = 0, pre_l = 0, total = 0, ppc = 0;                // lane b: length of sequence b, pages before it; pages in all and per range
    auto scan = [&](int len) {
        len_l = len;
        const int n = lane < p.B ? seq_pages(len, cap, p.P, p.sink, p.window).n : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        pre_l = incl - n;
        total = __shfl_sync(0xffffffffu, incl, 31);
        ppc = (total + p.grid - 1) / p.grid;
    };
    auto range = [&](int sub, int& lo, int& hi) {
        const int vc = (int)blockIdx.x * subs + sub;
        lo = vc < p.grid ? min(total, vc * ppc) : total;
        hi = min(total, lo + ppc);
    };
    // largest b with pages before it <= f (executed by whole warps)
    auto sequence_of = [&](int f, int& len, int& before) -> int {
        int b = 0;
        if (small) {
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int v = __shfl_sync(0xffffffffu, pre_l, b + step);
                if (b + step < p.B && v <= f) b += step;
            }
            len = __shfl_sync(0xffffffffu, len_l, b);
            before = __shfl_sync(0xffffffffu, pre_l, b);
        } else {
            b = find_sequence(prefix, p.B, f);
            len = p.lengths[b];
            before = prefix[b];
        }
        return b;
    };
    auto page_index = [&](int f, int len, int before, SeqPages& sq) -> int {      // page of sequence `b` that item f of the list is
        sq = seq_pages(len, cap, p.P, p.sink, p.window);
        const int idx = f - before;
        return idx < sq.sink_pages ? idx : sq.first_recent + (idx - sq.sink_pages);
    };
    const int h0 = blockIdx.y * hc;                              // first kv head of the CTA

    // Lengths and block table may still change until the wait below, so what is read here is a hint (past L1, which must not keep it):
    // it brings the table's lines and the first pages of the CTA's ranges into L2 while the kernel before ends (16 ragged sequences
    // of bf16 pages: 35.6 -> 33.7 us; the decode stack's q8 attention 1 us).  Not for q4: no gain (16 x 4096 tokens: 27.6 against 28.0 us).
    if (BITS != 4 && small && warp == kAttnWarps) {
        scan(lane < p.B ? __ldcg(p.lengths + lane) : 0);
        for (int sub = 0; sub < subs; ++sub) {
            int lo, hi;
            range(sub, lo, hi);
            if (lo >= hi) continue;
            const int f = min(lo + lane, hi - 1);
            int len, before;
            SeqPages sq;
            const int b = sequence_of(f, len, before);
            const int page = __ldcg(p.block_table + (int64_t)b * p.max_blocks + page_index(f, len, before, sq));
            if (lane < NS && lo + lane < hi && page >= 0 && page < p.num_pages) {
                prefetch_box_3d(&sp.kmap, 0, page * 16, BITS == 16 ? 2 * h0 : h0);
                prefetch_box_3d(&sp.vmap, 0, page * 16, BITS == 16 ? 2 * h0 : h0);
            }
        }
    }
    pdl_wait();   // lengths / block table / q / the cache itself may be produced by the previous kernel
    pdl_launch_dependents();      // after the wait: the merge kernel may read the lengths before this kernel ends
    if (small) scan(lane < p.B ? p.lengths[lane] : 0);
    else {
        total = build_prefix(p, prefix);
        ppc = (total + p.grid - 1) / p.grid;
    }
    if (p.verdict != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && warp == kAttnWarps) {
        bool good = true;
        for (int b = lane; b < p.B; b += 32) {
            const int len = small ? len_l : p.lengths[b];
            good = good && len >= 0 && len <= cap;
        }
        good = __all_sync(0xffffffffu, good);
        if (lane == 0) *reinterpret_cast<volatile int32_t*>(p.verdict) = good ? 1 : 2;
    }
    const uint32_t limit = kAttnWaitLimit;

    // ================================ producer ================================
    if (warp == kAttnWarps) {
        const uint32_t sc_bytes = BITS == 16 ? 0u : split_scale_bytes(hc, p.Gd);
        const bool scales8 = BITS != 16 && p.scales8;
        const uint32_t tx = (uint32_t)(2 * hc * TILE) + (scales8 ? 0u : 2 * sc_bytes);
        bool ok = true;
        int slot = 0;
        uint32_t par = 1u;                                       // a fresh barrier's previous phase counts as done
        for (int j = 0; j < ppc; ++j) {
            for (int sub = 0; sub < subs; ++sub) {
                int lo, hi;
                range(sub, lo, hi);
                if (lo + j >= hi) continue;
                uint2* dsub = desc + sub * kDescSlots;
                if ((j & 31) == 0) {                             // descriptors of this range's next 32 pages, one per lane
                    const int f = min(lo + j + lane, hi - 1);
                    int len, before;
                    const int b = sequence_of(f, len, before);
                    SeqPages sq;
                    const int pg = page_index(f, len, before, sq);
                    const int page = p.block_table[(int64_t)b * p.max_blocks + pg];
                    dsub[(j + lane) & (kDescSlots - 1)] = make_uint2((uint32_t)(page < 0 || page >= p.num_pages ? -1 : page),
                                                                     ((uint32_t)b << 16) | page_mask16(pg, sq.L, p.sink, p.window));
                    __syncwarp();
                }
                const int bar = sub * NS + slot;
                ok = mbar_wait_bounded(&empty[bar], par, &g_device_status, EV_ATTN_EMPTY_WAIT, ok ? limit : 64u) && ok;
                __syncwarp();
                const int page = (int)dsub[j & (kDescSlots - 1)].x;
                if (scales8) {
                    if (page >= 0) {
                        const uint32_t sdst = ring + (uint32_t)bar * p.slot_bytes + 2 * hc * TILE;
                        const bool whole = p.Hkv == hc;          // the page's scales are contiguous
                        const int rows = whole ? 1 : 16, row8 = (int)(sc_bytes / 8) / rows;
                        const size_t at = (size_t)page * 16 * p.scale_row_halves + (whole ? 0 : h0 * p.Gd);
                        copy_scales8(sdst, p.k_scales + at, rows, row8, (int64_t)p.scale_row_halves * 2, lane);
                        copy_scales8(sdst + sc_bytes, p.v_scales + at, rows, row8, (int64_t)p.scale_row_halves * 2, lane);
                    }
                    arrive_on_copies(&full[bar]);
                }
                if (lane == 0) {
                    if (page < 0) {
                        mbar_arrive(&full[bar]);                 // a missing page: nothing to copy, the consumers skip it
                    } else {
                        const uint32_t dst = ring + (uint32_t)bar * p.slot_bytes;
                        mbar_arrive_expect_tx(&full[bar], tx);
                        tma_load_3d(dst, &sp.kmap, 0, page * 16, BITS == 16 ? 2 * h0 : h0, &full[bar]);
                        tma_load_3d(dst + hc * TILE, &sp.vmap, 0, page * 16, BITS == 16 ? 2 * h0 : h0, &full[bar]);
                        if (BITS != 16 && !scales8) {
                            const uint32_t sdst = dst + 2 * hc * TILE;
                            if (p.Hkv == hc) {                   // the page's scales are contiguous
                                const size_t at = (size_t)page * 16 * p.scale_row_halves;
                                bulk_g2s(smem + (sdst - ring), p.k_scales + at, sc_bytes, &full[bar]);
                                bulk_g2s(smem + (sdst + sc_bytes - ring), p.v_scales + at, sc_bytes, &full[bar]);
                            } else {
                                tma_load_2d(sdst, &sp.ksmap, h0 * p.Gd * 2, page * 16, &full[bar]);
                                tma_load_2d(sdst + sc_bytes, &sp.vsmap, h0 * p.Gd * 2, page * 16, &full[bar]);
                            }
                        }
                    }
                }
            }
            if (++slot == NS) { slot = 0; par ^= 1u; }
        }
        if (scales8) asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    // ================================ consumers ================================
    const int hl = warp % hc, h = h0 + hl;                       // kv head of this warp
    const int sub = warp / hc;
    if (sub >= subs) return;
    const int vc = (int)blockIdx.x * subs + sub;                 // range of this warp
    int lo, hi;
    range(sub, lo, hi);
    if (lo >= hi) return;
    const int group = p.group;
    const int n_my = hi - lo;                                    // pages this warp walks: f = lo + j

    WarpState<BITS, WIDE> acc;
    state_reset(acc);
    auto flush = [&](int b) {
        float* dst = p.partial + ((size_t)(vc + b) * p.Hq + h * group) * (D + 2);
        emit(acc, group, lane, [&](int head, int d, float v) { dst[head * (D + 2) + d] = v; },
             [&](int head, float m, float l) { dst[head * (D + 2) + D] = m; dst[head * (D + 2) + D + 1] = l; });
    };
    auto queries = [&](int b) {
        load_queries<BITS, LOGG>(acc, reinterpret_cast<const uint16_t*>(p.q) + ((size_t)b * p.Hq + h * group) * D, group, p.q_dtype, p.scale, lane);
    };
    int cur_b;
    {
        int len, before;
        cur_b = sequence_of(lo, len, before);
    }
    queries(cur_b);                                              // the first sequence's, while the copies are in flight
    const PageRead R = box_read<BITS>(lane, hl, hc, p.Gd);
    const uint2* dsub = desc + sub * kDescSlots;
    bool ok = true;
    int slot = 0;
    uint32_t par = 0;
    for (int j = 0; j < n_my; ++j) {
        const int bar = sub * NS + slot;
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[bar], par, &g_device_status, EV_ATTN_FULL_WAIT, ok ? limit : 64u)) && ok;
        const uint2 d = dsub[j & (kDescSlots - 1)];
        const int b = (int)(d.y >> 16);
        if (b != cur_b && ok) {
            flush(cur_b);
            cur_b = b;
            state_reset(acc);
            queries(b);
        }
        if ((int)d.x >= 0 && ok) {
            const uint32_t sl = ring + (uint32_t)bar * p.slot_bytes;
            process_page<BITS, LOGG>(acc, sl + hl * TILE, sl + (hc + hl) * TILE, sl + 2 * hc * TILE, R, d.y & 0xFFFFu, lane);
        }
        __syncwarp();   // every lane is done with this slot before it is refilled
        if (lane == 0) mbar_arrive(&empty[bar]);
        if (++slot == NS) { slot = 0; par ^= 1u; }
    }
    flush(cur_b);
}

// ------------------------------------------------------------------------------------------------
// Cluster kernel for small batches and short walks: one thread-block cluster per (sequence, kv head), no partials in global memory
// and no merge launch.  The CTAs of the cluster cut the sequence's pages into equal ranges, the 8 or 16 warps of a CTA cut
// their range again; a warp walks its pages exactly as in the split-KV kernel.  The warps' partial (max, sum,
// accumulator) triples are merged in shared memory, the CTAs' through distributed shared memory by the cluster's
// first CTA, always in the same order (bitwise repeatable, and independent of how many kv heads a tensor-parallel
// shard holds).  Optionally the kernel also does what precedes attention in a decode layer - split the fused QKV
// row, rotate q and k, quantise and append the new token's k / v to its page: the CTA that walks the page of the
// new position appends kv head h itself before it reads that page, every CTA rotates its own copy of q.
// ------------------------------------------------------------------------------------------------
struct ClusterAttnParams {
    const void* q;              // [B, Hq, D] rotated queries (fused == 0)
    const __half* qkv;          // fused: [B, (Hq + 2 Hkv) * D]
    const float* cos_table;     // fused: [table_len, D/2]
    const float* sin_table;
    const int32_t* positions;   // fused: [B]
    uint8_t* k_codes;
    uint8_t* v_codes;
    __half* k_scales;
    __half* v_scales;
    const int32_t* block_table;
    const int32_t* lengths;
    void* out;                  // [B, Hq, D]
    int B, Hq, Hkv, P, max_blocks, G, Gd, group, bits, q_dtype, table_len, fused, S;
    int64_t num_pages;
    float scale;
    int row_bytes, scale_row_halves;
    int hs;                     // kv heads whose scales one copy brings: Hkv, at most 8
    int stages;                 // pages in flight per warp
    uint32_t slot_bytes;        // K tile, V tile, scales of K, scales of V
    uint32_t off_bars, off_q, off_cpart;      // the warps' rings come first
    int sink, window;           // as in AttnParams (window > 0 only without the append)
    int walk_pages;             // pages that a sequence can have to visit (host side)
    int32_t* verdict;           // as in AttnParams
    TpOut tp_out;
};
struct alignas(64) ClusterParams {
    CUtensorMap kmap, vmap;     // as in SplitParams, box of one head
    CUtensorMap ksmap, vsmap;   // used with more than 8 kv heads only
    ClusterAttnParams a;
};
constexpr int kMaxClusterRing = 8;
constexpr int kClusterWarps = 16;

__device__ __forceinline__ uint32_t cluster_rank_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Bound by latency: one launch of a few microseconds whose chain is lengths -> page ids -> pages -> merge of the warps -> merge of the
// CTAs.  A warp's pages come by tensor copies that one lane issues as soon as the page ids are there, before the queries are
// rotated (16-byte cp.async pieces kept the CTA's memory path busy for 9100 of the kernel's 20000 clocks at one sequence of 4096 q8
// tokens); the scales come whole, all heads of the page, which costs less than sixteen pieces of 8 bytes.  Only the page that the new
// token goes to waits for its append.
// SC8: scales aligned to 8 bytes only (a template parameter: asked at run time it cost the aligned form 0.3 of 9.9 us).
// NW: warps of a CTA (with the number at run time the merge and the cut of the pages cost the shortest calls 0.5 of 5.3 us).  WIN: with a window.
template <int BITS, int LOGG, bool WIDE, bool SC8, int NW, bool WIN>
__global__ void __launch_bounds__(NW * 32, 1) paged_attn_cluster_kernel(const __grid_constant__ ClusterParams cp) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const ClusterAttnParams& p = cp.a;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int D = kHeadDim;
    constexpr int TILE = PageShape<BITS>::TILE;
    const int NS = p.stages;
    constexpr int PW = D + 2;                                     // floats of one partial: accumulator, max, sum
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank_x();
    const int h = blockIdx.y;
    const int b = blockIdx.z;
    const int group = p.group;
    const int S = p.S;
    __half* qs = reinterpret_cast<__half*>(smem + p.off_q);              // [group][D] rotated query rows
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.off_bars) + warp * NS;      // this warp's ring
    uint8_t* my_ring = smem + (size_t)warp * NS * p.slot_bytes;
    const int wstride = NS * (int)p.slot_bytes / 4;                      // a warp's partial [group][PW] takes the place of its pages
    const float* wpart = reinterpret_cast<const float*>(smem);
    float* cpart = reinterpret_cast<float*>(smem + p.off_cpart);         // [S][group][PW] (used in the first CTA)

    if (threadIdx.x == 0) {
        prefetch_map(&cp.kmap);
        prefetch_map(&cp.vmap);
    }
    if (lane < NS) mbar_init(&full[lane], SC8 ? 33 : 1);
    mbar_fence_init();
    __syncwarp();
    pdl_launch_dependents();
    pdl_wait();

    const SeqPages sq = seq_pages(p.lengths[b], p.max_blocks * p.P, p.P, WIN ? p.sink : 0, WIN ? p.window : 0);
    const int L = sq.L, n_pages = sq.n;
    if (BITS == 16 && p.verdict != nullptr && (blockIdx.x | blockIdx.y | blockIdx.z) == 0 && warp == 0) {
        bool good = true;
        for (int i = lane; i < p.B; i += 32) good = good && p.lengths[i] >= 0 && p.lengths[i] <= p.max_blocks * p.P;
        good = __all_sync(0xffffffffu, good);
        if (lane == 0) *reinterpret_cast<volatile int32_t*>(p.verdict) = good ? 1 : 2;
    }
    const int ppc = (n_pages + S - 1) / S;                               // pages per CTA
    const int c_lo = min(n_pages, (int)rank * ppc), c_hi = min(n_pages, c_lo + ppc);
    const int ppw = (c_hi - c_lo + NW - 1) / NW;         // pages per warp
    const int lo = min(c_hi, c_lo + warp * ppw), hi = min(c_hi, lo + ppw);

    const int n_my = hi - lo;
    auto page_at = [&](int i) { return !WIN || i < sq.sink_pages ? i : sq.first_recent + (i - sq.sink_pages); };      // of the sequence's visited pages
    auto page_ids = [&](int base) -> int {
        const int j = base + lane;
        const int page = j < n_my ? p.block_table[(size_t)b * p.max_blocks + page_at(lo + j)] : -1;
        return page >= p.num_pages ? -1 : page;
    };
    int ids_c = page_ids(0), ids_i = ids_c;                              // page ids of 32 consecutive pages, one per lane: consumed / issued window
    const uint32_t sc_bytes = split_scale_bytes(p.hs, p.Gd);
    auto issue = [&](int j) {                                            // copies of page j into its slot
        if (j > 0 && (j & 31) == 0) ids_i = page_ids(j);
        const int page = __shfl_sync(0xffffffffu, ids_i, j & 31);
        if constexpr (SC8) {
            if (page >= 0) {
                const uint32_t sdst = smem_u32(my_ring + (size_t)(j % NS) * p.slot_bytes + 2 * TILE);
                const bool whole = p.Hkv == p.hs;
                const int rows = whole ? 1 : 16, row8 = (int)(sc_bytes / 8) / rows;
                const size_t at = (size_t)page * 16 * p.scale_row_halves + (whole ? 0 : (h & ~7) * p.Gd);
                copy_scales8(sdst, p.k_scales + at, rows, row8, (int64_t)p.scale_row_halves * 2, lane);
                copy_scales8(sdst + sc_bytes, p.v_scales + at, rows, row8, (int64_t)p.scale_row_halves * 2, lane);
            }
            arrive_on_copies(&full[j % NS]);
        }
        if (lane == 0) {
            uint64_t* bar = &full[j % NS];
            if (page < 0) {
                mbar_arrive(bar);                                        // a missing page: nothing to copy, skipped where it is used
            } else {
                uint8_t* dst = my_ring + (size_t)(j % NS) * p.slot_bytes;
                const int z = BITS == 16 ? 2 * h : h;                    // a plain row is two tiles of 128 bytes
                mbar_arrive_expect_tx(bar, 2 * TILE + (SC8 || BITS == 16 ? 0u : 2 * sc_bytes));
                tma_load_3d(smem_u32(dst), &cp.kmap, 0, page * 16, z, bar);
                tma_load_3d(smem_u32(dst + TILE), &cp.vmap, 0, page * 16, z, bar);
                if (SC8 || BITS == 16) {
                } else if (p.Hkv == p.hs) {
                    const size_t at = (size_t)page * 16 * p.scale_row_halves;
                    bulk_g2s(dst + 2 * TILE, p.k_scales + at, sc_bytes, bar);
                    bulk_g2s(dst + 2 * TILE + sc_bytes, p.v_scales + at, sc_bytes, bar);
                } else {
                    const int x = (h & ~7) * p.Gd * 2;
                    tma_load_2d(smem_u32(dst + 2 * TILE), &cp.ksmap, x, page * 16, bar);
                    tma_load_2d(smem_u32(dst + 2 * TILE + sc_bytes), &cp.vsmap, x, page * 16, bar);
                }
            }
        }
    };
    // the page of the new token is copied after its append
    const int j_app = p.fused && p.positions[b] >= 0 ? p.positions[b] / p.P - lo : -1;
    for (int j = 0; j < min(NS, n_my); ++j)
        if (j != j_app) issue(j);

    if constexpr (BITS != 16) if (p.fused) {
        const int heads = p.Hq + 2 * p.Hkv;
        const int pos = p.positions[b];
        const bool pos_ok = pos >= 0 && pos < p.table_len;
        const int d0 = lane * 4;
        const __half* row = p.qkv + (size_t)b * heads * D;
        auto load4 = [&](int head, float (&v)[4]) {
            const uint2 u = *reinterpret_cast<const uint2*>(row + (size_t)head * D + d0);
            const __half2 h0 = *reinterpret_cast<const __half2*>(&u.x), h1 = *reinterpret_cast<const __half2*>(&u.y);
            v[0] = __low2float(h0); v[1] = __high2float(h0); v[2] = __low2float(h1); v[3] = __high2float(h1);
        };
        auto rope4 = [&](float (&v)[4]) {
            if (!pos_ok) return;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float c = p.cos_table[(size_t)pos * (D / 2) + d0 / 2 + i];
                const float sn = p.sin_table[(size_t)pos * (D / 2) + d0 / 2 + i];
                const float xe = v[2 * i], xo = v[2 * i + 1];
                // two separately rounded products and one sum, as the reference's elementwise expression
                v[2 * i] = __fsub_rn(__fmul_rn(xe, c), __fmul_rn(xo, sn));
                v[2 * i + 1] = __fadd_rn(__fmul_rn(xe, sn), __fmul_rn(xo, c));
            }
        };
        if (!pos_ok && threadIdx.x == 0) atomicMax(&g_device_status, (int)EV_ROPE_POSITION);
        // rotated query rows of this kv head's group, one warp per query head
        if (warp < group) {
            float v[4];
            load4(h * group + warp, v);
            rope4(v);
            const __half2 a0 = __floats2half2_rn(v[0], v[1]), a1 = __floats2half2_rn(v[2], v[3]);
            uint2 o2;
            o2.x = *reinterpret_cast<const uint32_t*>(&a0);
            o2.y = *reinterpret_cast<const uint32_t*>(&a1);
            *reinterpret_cast<uint2*>(qs + (size_t)warp * D + d0) = o2;
        }
        // append k (rotated) and v of kv head h to the page of `pos`: the CTA whose range holds that page
        const int blk = pos >= 0 ? pos / p.P : -1;
        const int owner = (ppc > 0 && blk >= 0) ? min(S - 1, blk / ppc) : 0;
        if ((int)rank == owner && append_role(warp, NW) != kAppendNothing) {
            const bool is_v = append_role(warp, NW) == kAppendV;
            int page = (blk >= 0 && blk < p.max_blocks) ? p.block_table[(size_t)b * p.max_blocks + blk] : -1;
            if (page < 0 || page >= p.num_pages) {
                if (lane == 0) atomicMax(&g_device_status, (int)EV_KV_PAGE_UNASSIGNED);
            } else {
                float v[4];
                load4(p.Hq + (is_v ? p.Hkv : 0) + h, v);
                if (!is_v) rope4(v);
                __half hv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { hv[i] = __float2half_rn(v[i]); v[i] = __half2float(hv[i]); }
                float mx = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
                const int lanes_per_group = p.G / 4;
                for (int o2 = 1; o2 < lanes_per_group; o2 <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o2));
                const float limit = BITS == 8 ? 127.0f : 7.0f;
                const float offset = BITS == 8 ? 128.0f : 8.0f;
                const float sc = __fdiv_rn(fmaxf(mx, 1e-8f), limit);
                uint32_t codes[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    codes[i] = (uint32_t)(int)(fminf(fmaxf(rintf(__fdiv_rn(v[i], sc)), -limit), limit) + offset);
                const size_t tok = ((size_t)page * p.P + (pos % p.P)) * p.Hkv + h;
                uint8_t* cdst = is_v ? p.v_codes : p.k_codes;
                __half* sdst = is_v ? p.v_scales : p.k_scales;
                if (BITS == 8)
                    *reinterpret_cast<uint32_t*>(cdst + tok * D + d0) = codes[0] | (codes[1] << 8) | (codes[2] << 16) | (codes[3] << 24);
                else
                    *reinterpret_cast<uint16_t*>(cdst + tok * (D / 2) + d0 / 2) =
                        (uint16_t)(codes[0] | (codes[1] << 4) | (codes[2] << 8) | (codes[3] << 12));
                if ((lane % lanes_per_group) == 0) sdst[tok * p.Gd + d0 / p.G] = __float2half_rn(sc);
            }
            // the appended bytes are in global memory, also for the copy engine, before this CTA's copies read the page
            __threadfence();
            fence_async_proxy();
        }
        __syncthreads();
        fence_async_proxy();
        if (j_app >= 0 && j_app < min(NS, n_my)) issue(j_app);
    }

    // ---- this warp's pages ----
    WarpState<BITS, WIDE> acc;
    state_reset(acc);
    if (n_my > 0) {
        const void* qrows = p.fused ? (const void*)qs : (const void*)(reinterpret_cast<const uint16_t*>(p.q) + ((size_t)b * p.Hq + h * group) * D);
        const PageRead R = box_read<BITS>(lane, h % p.hs, p.hs, p.Gd);
        load_queries<BITS, LOGG>(acc, qrows, group, p.fused ? B200Q_F16 : p.q_dtype, p.scale, lane);
        bool ok = true;
        int slot = 0;
        uint32_t par = 0;
        for (int j = 0; j < n_my; ++j) {
            if (j > 0 && (j & 31) == 0) ids_c = page_ids(j);
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[slot], par, &g_device_status, EV_ATTN_FULL_WAIT, ok ? kAttnWaitLimit : 64u)) && ok;
            const uint32_t attended = page_mask16(page_at(lo + j), L, WIN ? p.sink : 0, WIN ? p.window : 0);
            if (__shfl_sync(0xffffffffu, ids_c, j & 31) >= 0 && ok) {
                const uint32_t k_tile = smem_u32(my_ring) + (uint32_t)slot * p.slot_bytes;
                process_page<BITS, LOGG>(acc, k_tile, k_tile + TILE, k_tile + 2 * TILE, R, attended, lane);
            }
            __syncwarp();                                                // every lane is done with this slot before it is refilled
            if (j + NS < n_my) issue(j + NS);
            if (++slot == NS) { slot = 0; par ^= 1u; }
        }
    }
    {
        float* dst = reinterpret_cast<float*>(my_ring);
        emit(acc, group, lane, [&](int head, int d, float v) { dst[head * PW + d] = v; },
             [&](int head, float m, float l) { dst[head * PW + D] = m; dst[head * PW + D + 1] = l; });
    }
    __syncthreads();
    // ---- merge the warps (fixed order) into this CTA's partial; thread -> (head, d) ----
    auto merge = [&](const float* src, int n, int stride, int head, int d, float& m_tot, float& l_tot) -> float {
        src += head * PW;
        m_tot = -INFINITY;
#pragma unroll 8
        for (int i = 0; i < n; ++i) m_tot = fmaxf(m_tot, src[i * stride + D]);
        float accv = 0.0f;
        l_tot = 0.0f;
#pragma unroll 8
        for (int i = 0; i < n; ++i) {
            const float* ps = src + i * stride;
            const float m = ps[D];
            const float w = m == -INFINITY ? 0.0f : exp2f(m - m_tot);      // the maxima are in log2 units
            accv = fmaf(w, ps[d], accv);
            l_tot = fmaf(w, ps[D + 1], l_tot);
        }
        return accv;
    };
    const uint32_t cpart_u = smem_u32(cpart);
    for (int idx = threadIdx.x; idx < group * D; idx += (NW * 32)) {
        const int head = idx / D, d = idx - head * D;
        float m_tot, l_tot;
        const float v = merge(wpart, NW, wstride, head, d, m_tot, l_tot);
        // slot `rank` of the first CTA's table (its own slot for the first CTA itself)
        const uint32_t base = cpart_u + (uint32_t)((rank * group + head) * PW) * 4u;
        auto put = [&](uint32_t off, float val) {
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(base + off * 4u), "r"(0));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(val) : "memory");
        };
        put((uint32_t)d, v);
        if (d == 0) { put((uint32_t)D, m_tot); put((uint32_t)D + 1, l_tot); }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 0) {
        for (int idx = threadIdx.x; idx < group * D; idx += (NW * 32)) {
            const int head = idx / D, d = idx - head * D;
            float m_tot, l_tot;
            const float v = merge(cpart, S, group * PW, head, d, m_tot, l_tot);
            const float inv = l_tot > 0.0f ? 1.0f / l_tot : 0.0f;
            const unsigned short bits16 = p.fused || p.q_dtype == B200Q_F16 ? __half_as_ushort(__float2half_rn(v * inv))
                                                                            : __bfloat16_as_ushort(__float2bfloat16_rn(v * inv));
            const int hq = h * group + head;
            if (p.out != nullptr) reinterpret_cast<unsigned short*>(p.out)[((size_t)b * p.Hq + hq) * D + d] = bits16;
            if (p.tp_out.world > 0) {
                const size_t of = ((size_t)b * p.tp_out.world + p.tp_out.rank) * p.Hq * D + (size_t)hq * D + d;
                if (p.tp_out.packets) {
                    const uint32_t pk = tp_packet(bits16, tp_seq16(tp_writer_seq(p.tp_out)));
#pragma unroll 1
                    for (int peer = 0; peer < p.tp_out.world; ++peer)
                        st_volatile_u32(reinterpret_cast<uint32_t*>(p.tp_out.full[peer]) + of, pk);
                } else {
#pragma unroll 1
                    for (int peer = 0; peer < p.tp_out.world; ++peer)
                        reinterpret_cast<unsigned short*>(p.tp_out.full[peer])[of] = bits16;
                }
            }
        }
    }
    if (p.tp_out.world > 0) {
        __syncthreads();                         // all of this CTA's peer stores are issued
        if (warp == 0) {
            if (p.tp_out.packets) tp_finish_writer_packets(p.tp_out, lane, gridDim.x * gridDim.y * gridDim.z);
            else tp_finish_writer(p.tp_out, lane, gridDim.x * gridDim.y * gridDim.z);
        }
    }
}

// Merges the partials of every (sequence, query head): one warp each, lanes over d.

// One CTA per (sequence, query head).  The partials of a sequence may sit in every range of the
// main kernel (a single long sequence is cut over the whole grid), so the ranges are spread over the
// CTA's warps; lanes cover the head dimension.  The lengths are known before the main kernel ends, so everything but the
// partials themselves is worked out ahead of griddepcontrol.wait; a warp then loads maximum, sum and row of its ranges
// at once and rescales as it goes (16 ragged sequences of 32 heads: 7 -> 4.9 us after the main kernel's end).
// kMergeWarps: 32 for short batches (few CTAs, up to ~300 ranges each), 8 for long batches (many CTAs with a dozen each).
template <int kMergeWarps>
__global__ void __launch_bounds__(kMergeWarps * 32) paged_attn_merge_kernel(const __grid_constant__ AttnParams p) {
    __shared__ float red[kMergeWarps][128];
    __shared__ float red_s[2][kMergeWarps];
    pdl_launch_dependents();      // what follows waits for this kernel's end; until then it may set itself up or fetch its weights
    const int D = p.D;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int b = blockIdx.x / p.Hq;
    const int hq = blockIdx.x - b * p.Hq;

    // pages before sequence b and in total (the flattened page list of the main kernel); every warp for itself
    const int cap = p.max_blocks * p.P;
    int below = 0, all = 0, mine = 0;
    for (int i = lane; i < p.B; i += 32) {
        const int n = seq_pages(__ldcg(p.lengths + i), cap, p.P, p.sink, p.window).n;
        all += n;
        if (i < b) below += n;
        if (i == b) mine = n;
    }
    below = __reduce_add_sync(0xffffffffu, below);
    all = __reduce_add_sync(0xffffffffu, all);
    mine = __reduce_add_sync(0xffffffffu, mine);
    const int ppc = (all + p.grid - 1) / p.grid;
    pdl_wait();

    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    float l_part = 0.0f, m_run = -INFINITY;
    if (mine > 0) {
        // every range c_first..c_last holds at least one page of b, i.e. wrote a partial into slot c + b
        const int c_first = below / ppc, c_last = (below + mine - 1) / ppc;
#pragma unroll 4
        for (int c = c_first + warp; c <= c_last; c += kMergeWarps) {
            const float* src = p.partial + ((size_t)(c + b) * p.Hq + hq) * (D + 2);
            const float m = src[D], l = src[D + 1];
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = lane + 32 * j < D ? src[lane + 32 * j] : 0.0f;
            if (m == -INFINITY) continue;
            const float mn = fmaxf(m_run, m);                    // the maxima are in log2 units
            const float f = exp2f(m_run - mn), w = exp2f(m - mn);
            m_run = mn;
            l_part = fmaf(w, l, l_part * f);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = fmaf(w, v[j], acc[j] * f);
        }
    }
    if (lane == 0) { red_s[0][warp] = m_run; red_s[1][warp] = l_part; }
#pragma unroll
    for (int j = 0; j < 4; ++j) red[warp][lane + 32 * j] = acc[j];
    __syncthreads();
    if (threadIdx.x < D) {
        float m_tot = -INFINITY, sum = 0.0f, l_tot = 0.0f;
#pragma unroll
        for (int w = 0; w < kMergeWarps; ++w) m_tot = fmaxf(m_tot, red_s[0][w]);
#pragma unroll
        for (int w = 0; w < kMergeWarps; ++w) {
            const float f = red_s[0][w] == -INFINITY ? 0.0f : exp2f(red_s[0][w] - m_tot);
            sum = fmaf(f, red[w][threadIdx.x], sum);
            l_tot = fmaf(f, red_s[1][w], l_tot);
        }
        const float inv = l_tot > 0.0f ? 1.0f / l_tot : 0.0f;
        const size_t o = ((size_t)b * p.Hq + hq) * D + threadIdx.x;
        const unsigned short bits16 = p.q_dtype == B200Q_F16 ? __half_as_ushort(__float2half_rn(sum * inv))
                                                             : __bfloat16_as_ushort(__float2bfloat16_rn(sum * inv));
        if (p.out != nullptr) reinterpret_cast<unsigned short*>(p.out)[o] = bits16;
        if (p.tp_out.world > 0) {
            // tensor-parallel exchange: this head's row goes to column block `rank` of every rank's full rows
            const size_t of = ((size_t)b * p.tp_out.world + p.tp_out.rank) * p.Hq * D + (size_t)hq * D + threadIdx.x;
            if (p.tp_out.packets) {
                const uint32_t pk = tp_packet(bits16, tp_seq16(tp_writer_seq(p.tp_out)));
#pragma unroll 1
                for (int peer = 0; peer < p.tp_out.world; ++peer)
                    st_volatile_u32(reinterpret_cast<uint32_t*>(p.tp_out.full[peer]) + of, pk);
            } else {
#pragma unroll 1
                for (int peer = 0; peer < p.tp_out.world; ++peer)
                    reinterpret_cast<unsigned short*>(p.tp_out.full[peer])[of] = bits16;
            }
        }
    }
    if (p.tp_out.world > 0) {
        __syncthreads();                         // all of this CTA's peer stores are issued
        if (warp == 0) {
            if (p.tp_out.packets) tp_finish_writer_packets(p.tp_out, lane);
            else tp_finish_writer(p.tp_out, lane);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Simple kernel: one warp per (b, hq); any D <= 128, any group size, fp16/bf16 q, any scale dtype.
// ------------------------------------------------------------------------------------------------
struct SimpleParams {
    const void* q; const uint8_t* k_codes; const uint8_t* v_codes; const void* k_scales; const void* v_scales;
    const int32_t* block_table; const int32_t* lengths; void* out;
    int B, Hq, Hkv, D, P, max_blocks, G, Gd, bits, q_dtype, scale_dtype;
    int64_t num_pages;
    float scale;
    int sink, window;
    const uint8_t* block_mask;      // block-sparse decode: [n_qblocks, n_kblocks] bytes, or null
    int block_size, n_qblocks, n_kblocks;
};

__global__ void __launch_bounds__(128) paged_attn_simple_kernel(const __grid_constant__ SimpleParams p) {
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= p.B * p.Hq) return;
    const int b = item / p.Hq;
    const int hq = item - b * p.Hq;
    const int hkv = hq / (p.Hq / p.Hkv);
    const int DPk = p.bits == 4 ? (p.D + 1) / 2 : p.D;
    const int L = clamp_len(p.lengths[b], p.max_blocks * p.P);
    float qv[4], acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int d = lane + 32 * j;
        qv[j] = d < p.D ? load_as_f32(p.q, p.q_dtype, ((int64_t)b * p.Hq + hq) * p.D + d) : 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    const float off = p.bits == 4 ? 8.0f : 128.0f;
    // block-sparse: the query sits at position L - 1, i.e. in row (L - 1) / block_size of the mask
    const int qb = (p.block_mask != nullptr && L > 0) ? (L - 1) / p.block_size : 0;
    const uint8_t* mask_row = (p.block_mask != nullptr && qb < p.n_qblocks) ? p.block_mask + (size_t)qb * p.n_kblocks : nullptr;
    for (int j = 0; j < L; ++j) {
        if (p.window > 0 && j >= p.sink && j < L - p.window) continue;     // outside sink and window
        if (p.block_mask != nullptr) {
            const int kb = j / p.block_size;
            if (mask_row == nullptr || kb >= p.n_kblocks || mask_row[kb] == 0) continue;
        }
        const int page = p.block_table[(int64_t)b * p.max_blocks + j / p.P];
        if (page < 0 || page >= p.num_pages) continue;
        const int64_t tok = ((int64_t)page * p.P + (j % p.P)) * p.Hkv + hkv;
        float kd[4], vd[4], dot = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int d = lane + 32 * i;
            kd[i] = vd[i] = 0.0f;
            if (d < p.D) {
                uint32_t kc, vc;
                if (p.bits == 4) {
                    const uint8_t kb = p.k_codes[tok * DPk + (d >> 1)], vb = p.v_codes[tok * DPk + (d >> 1)];
                    kc = (d & 1) ? (kb >> 4) : (kb & 0xF);
                    vc = (d & 1) ? (vb >> 4) : (vb & 0xF);
                } else {
                    kc = p.k_codes[tok * DPk + d];
                    vc = p.v_codes[tok * DPk + d];
                }
                const float ks = fabsf(load_as_f32(p.k_scales, p.scale_dtype, tok * p.Gd + d / p.G));
                const float vs = fabsf(load_as_f32(p.v_scales, p.scale_dtype, tok * p.Gd + d / p.G));
                kd[i] = __half2float(__float2half_rn(__fmul_rn((float)kc - off, ks)));
                vd[i] = __half2float(__float2half_rn(__fmul_rn((float)vc - off, vs)));
                dot = fmaf(qv[i], kd[i], dot);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float sc = dot * p.scale;
        const float m_new = fmaxf(m, sc);
        const float alpha = (m == -INFINITY) ? 0.0f : expf(m - m_new);
        const float beta = expf(sc - m_new);
        l = l * alpha + beta;
        m = m_new;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = acc[i] * alpha + beta * vd[i];
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int d = lane + 32 * i;
        if (d < p.D) {
            const int64_t o = ((int64_t)b * p.Hq + hq) * p.D + d;
            if (p.q_dtype == B200Q_F16) reinterpret_cast<__half*>(p.out)[o] = __float2half_rn(acc[i] * inv);
            else reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(acc[i] * inv);
        }
    }
}

inline uint32_t align_up_u32(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }
inline int subs_for(int hc) { return kAttnWarps % hc == 0 ? kAttnWarps / hc : 1; }

inline bool heads_ok(int Hkv) { return Hkv <= kAttnWarps || Hkv % kAttnWarps == 0; }

// ---- cluster kernel: host side ----
ClusterChoice choose_cluster(int B, int Hkv, int group, int max_blocks, AttnUse use, bool split) {
    ClusterQuery c = {};
    c.B = B; c.Hkv = Hkv; c.group = group; c.walk_pages = max_blocks; c.use = use; c.split = split;
    c.tp_world = std::max(1, tuning_get("ts.tp_world"));
    c.mode = tuning_get("attn.cluster");
    c.forced_size = tuning_get("attn.cluster_size");
    c.sms = sm_count();
    return cluster_choice(c);
}

// Byte tensor [heads][tokens][row] of a page pool whose token rows are `pitch` bytes apart; box = heads of a CTA x 16 tokens x row.
bool page_map(const void* ptr, uint32_t row, int64_t tokens, int heads, int pitch, int box_heads, CUtensorMap* out) {
    const PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[3] = {row, (cuuint64_t)tokens, (cuuint64_t)heads};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch, row};
    const cuuint32_t box[3] = {row, 16, (cuuint32_t)box_heads};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  row == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool scale_map(const void* ptr, int pitch, int64_t tokens, int box_bytes, CUtensorMap* out) {
    const PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)tokens};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_bytes, 16};
    const cuuint32_t estr[2] = {1, 1};
    return encode(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int launch_cluster_attention(ClusterAttnParams& p, cudaStream_t stream) {
    const bool plain = p.bits == 16, bf = p.q_dtype == B200Q_BF16, g32 = p.G == 32, wide = p.group > 4;
    const bool sc8 = !plain && ((uintptr_t)p.k_scales | (uintptr_t)p.v_scales) % 16 != 0;
    // Sixteen warps where eight would have more than a page each: a page costs a warp about a microsecond, the merge of eight more partial
    // results 0.2 (one sequence, one page a warp: q8 5.4 us with eight, 5.7 with sixteen; two sequences of 2048 tokens 9.2 and 8.5).
    // Whether their rings fit is asked of the UNSHARDED cache's scales, like the choice of the kernel: the number of warps is part of the
    // summation order, and a shard's narrower scale rows would let it have sixteen where the unsharded call has eight.
    int warps = !plain && (p.walk_pages > p.S * 8 || p.window > 0) ? kClusterWarps : 8;
    auto slot_for = [&](int hs) {
        return split_slot_bytes(p.bits, 1, 0) + (plain ? 0u : align_up_u32(2 * split_scale_bytes(hs, p.Gd), p.bits == 4 ? 512 : 1024));
    };
    p.hs = std::min(p.Hkv, kAttnWarps);
    p.slot_bytes = slot_for(p.hs);
    const uint32_t slot_full = slot_for((int)std::min<int64_t>((int64_t)p.Hkv * std::max(1, tuning_get("ts.tp_world")), kAttnWarps));
    // shared memory: [1 KB alignment] rings, barriers, query rows, the CTAs' partials
    const uint32_t q_bytes = align_up_u32((uint32_t)p.group * 128 * 2, 128), c_bytes = align_up_u32((uint32_t)p.S * p.group * 130 * 4, 128);
    const uint32_t cap = (uint32_t)max_smem_optin(), fixed = 1024 + 128 * 8 + q_bytes + c_bytes;
    auto depth = [&](uint32_t slot_bytes) { return (int)std::min<uint32_t>(kMaxClusterRing, (cap - std::min(cap, fixed)) / (warps * slot_bytes)); };
    if (depth(slot_full) < 2 && p.window == 0) warps = 8;
    if (depth(slot_full) < 2) return B200Q_ERR_UNSUPPORTED;
    p.stages = depth(p.slot_bytes);
    p.off_bars = warps * p.stages * p.slot_bytes;
    p.off_q = p.off_bars + 128 * 8;
    p.off_cpart = p.off_q + q_bytes;
    const uint32_t off = 1024 + p.off_cpart + c_bytes;
    ClusterParams cp = {};
    cp.a = p;
    const uint32_t row = p.bits == 4 ? 64 : 128, tiles = plain ? 2 : 1;
    if (!page_map(p.k_codes, row, p.num_pages * 16, p.Hkv * tiles, p.row_bytes, tiles, &cp.kmap) ||
        !page_map(p.v_codes, row, p.num_pages * 16, p.Hkv * tiles, p.row_bytes, tiles, &cp.vmap))
        return B200Q_ERR_LAUNCH;
    if (!plain && p.Hkv > p.hs && !sc8 && (!scale_map(p.k_scales, p.scale_row_halves * 2, p.num_pages * 16, p.hs * p.Gd * 2, &cp.ksmap) ||
                         !scale_map(p.v_scales, p.scale_row_halves * 2, p.num_pages * 16, p.hs * p.Gd * 2, &cp.vsmap)))
        return B200Q_ERR_LAUNCH;
    using KernelFn = void (*)(ClusterParams);
    // [form]: eight warps, dense, scales aligned to 16 bytes or to 8; sixteen warps, dense; sixteen warps, any call, aligned or not
#define B200Q_CLUSTER_FORMS(BITS, LOGG, WIDE)                                                                                         \
    {paged_attn_cluster_kernel<BITS, LOGG, WIDE, false, 8, false>, paged_attn_cluster_kernel<BITS, LOGG, WIDE, true, 8, false>,         \
     paged_attn_cluster_kernel<BITS, LOGG, WIDE, false, 16, false>, paged_attn_cluster_kernel<BITS, LOGG, WIDE, false, 16, true>,       \
     paged_attn_cluster_kernel<BITS, LOGG, WIDE, true, 16, true>}
    static const KernelFn kernels[2][2][2][5] = {{{B200Q_CLUSTER_FORMS(8, 6, false), B200Q_CLUSTER_FORMS(8, 6, true)},      // [q4][group 32][wide][form]
                                                  {B200Q_CLUSTER_FORMS(8, 5, false), B200Q_CLUSTER_FORMS(8, 5, true)}},
                                                 {{B200Q_CLUSTER_FORMS(4, 6, false), B200Q_CLUSTER_FORMS(4, 6, true)},
                                                  {B200Q_CLUSTER_FORMS(4, 5, false), B200Q_CLUSTER_FORMS(4, 5, true)}}};
#undef B200Q_CLUSTER_FORMS
    static const KernelFn plain_kernels[2][2] = {      // [bf16][wide]
        {paged_attn_cluster_kernel<16, 0, false, false, 8, false>, paged_attn_cluster_kernel<16, 0, true, false, 8, false>},
        {paged_attn_cluster_kernel<16, 1, false, false, 8, false>, paged_attn_cluster_kernel<16, 1, true, false, 8, false>}};
    const int form = warps == 8 ? (sc8 ? 1 : 0) : sc8 ? 4 : p.window > 0 ? 3 : 2;
    KernelFn kernel = plain ? plain_kernels[bf][wide] : kernels[p.bits == 4][g32][wide][form];
    static bool configured[44][64] = {};
    const int slot = plain ? 40 + bf * 2 + wide : ((p.bits == 4) * 4 + g32 * 2 + wide) * 5 + form;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[slot][dev & 63]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) != cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return B200Q_ERR_LAUNCH;
        configured[slot][dev & 63] = true;
    }
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (!tuning_get("no_pdl")) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.S;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.S, p.Hkv, p.B);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = off;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = na;
    if (cudaLaunchKernelEx(&cfg, kernel, cp) != cudaSuccess) return B200Q_ERR_LAUNCH;
    return finish_launch();
}

// max_ranges: what the workspace has room for.
int launch_split_attention(AttnParams& p, int max_ranges, cudaStream_t stream) {
    const int bits = p.bits;
    p.hc = std::min(p.Hkv, kAttnWarps);
    p.subs = subs_for(p.hc);
    const int chunks = p.Hkv / p.hc;
    p.slot_bytes = split_slot_bytes(bits, p.hc, p.Gd);
    p.scales8 = bits != 16 && ((uintptr_t)p.k_scales | (uintptr_t)p.v_scales) % 16 != 0;
    int ctas_per_sm = tuning_get("attn.ctas_per_sm");
    if (ctas_per_sm <= 0) ctas_per_sm = bits == 16 ? 1 : B200Q_ATTN_CTAS;
    // At least three pages per range (by the block table's capacity; the lengths live on the device): short
    // batches otherwise pay for partial results and their merge more than for the KV bytes (measured on the
    // 32-layer stack at batch 1, context 4096: 2 -> 2.32-2.35, 3 -> 2.26, 4 -> 2.30, 8 -> 2.46 ms per step).
    const int64_t pages_cap = (int64_t)p.B * p.max_blocks;
    int min_pages = tuning_get("attn.min_pages");
    if (min_pages <= 0) min_pages = 3;
    // Ranges for every warp of the resident CTAs.  The cut follows the kv heads of the UNSHARDED cache ("ts.tp_world" equal head
    // shards), so that a head's partial results do not depend on the sharding.
    const int full_subs = subs_for(std::min(p.Hkv * std::max(1, tuning_get("ts.tp_world")), kAttnWarps));
    const int want = std::max(1, sm_count() * ctas_per_sm / chunks) * full_subs;
    p.grid = (int)std::max<int64_t>(1, std::min<int64_t>(std::min({max_ranges, kMaxRanges, kMaxGrid * full_subs, want}), (pages_cap + min_pages - 1) / min_pages));
    const int launch_grid = (p.grid + p.subs - 1) / p.subs;   // CTAs: each covers `subs` ranges
    const bool two = bits != 16 && launch_grid * chunks > sm_count();
    // shared memory: [1 KB alignment] ring, barriers, descriptors, prefix sums
    const uint32_t cap = (uint32_t)max_smem_optin();
    const uint32_t fixed = 1024 + align_up_u32(2 * p.subs * kMaxRing * 8, 128) + p.subs * kDescSlots * 8 + align_up_u32((p.B + 1) * sizeof(int), 128);
    const uint32_t budget = two ? (cap + 1024) / 2 - 1024 : cap;       // an SM keeps 1 KB per resident CTA
    p.stages = (int)std::min<uint32_t>(kMaxRing, (budget - std::min(budget, fixed)) / (p.subs * p.slot_bytes));
    if (p.stages < 2) return B200Q_ERR_UNSUPPORTED;
    p.off_bars = p.subs * p.stages * p.slot_bytes;
    p.off_desc = p.off_bars + align_up_u32(2 * p.subs * p.stages * 8, 128);
    p.off_prefix = p.off_desc + p.subs * kDescSlots * 8;
    const uint32_t total_smem = 1024 + p.off_prefix + align_up_u32((p.B + 1) * sizeof(int), 128);
    SplitParams sp = {};
    sp.a = p;
    const uint32_t row = bits == 4 ? 64 : 128, tiles = bits == 16 ? 2 : 1;       // a plain row is two tiles of 128 bytes
    if (!page_map(p.k_codes, row, p.num_pages * 16, p.Hkv * tiles, p.row_bytes, p.hc * tiles, &sp.kmap) ||
        !page_map(p.v_codes, row, p.num_pages * 16, p.Hkv * tiles, p.row_bytes, p.hc * tiles, &sp.vmap))
        return B200Q_ERR_LAUNCH;
    if (bits != 16 && chunks > 1 && !p.scales8 &&
        (!scale_map(p.k_scales, p.scale_row_halves * 2, p.num_pages * 16, p.hc * p.Gd * 2, &sp.ksmap) ||
         !scale_map(p.v_scales, p.scale_row_halves * 2, p.num_pages * 16, p.hc * p.Gd * 2, &sp.vsmap)))
        return B200Q_ERR_LAUNCH;

    const bool g32 = p.G == 32, wide_group = p.group > 4, bf = p.q_dtype == B200Q_BF16;
    using KernelFn = void (*)(SplitParams);
#define B200Q_ATTN_PAIR(BITS, LOGG, TWO) {paged_attn_kernel<BITS, LOGG, TWO, false>, paged_attn_kernel<BITS, LOGG, TWO, true>}
    static const KernelFn quantised[2][2][2][2] = {      // [q4][group 32][two][wide]
        {{B200Q_ATTN_PAIR(8, 6, false), B200Q_ATTN_PAIR(8, 6, true)}, {B200Q_ATTN_PAIR(8, 5, false), B200Q_ATTN_PAIR(8, 5, true)}},
        {{B200Q_ATTN_PAIR(4, 6, false), B200Q_ATTN_PAIR(4, 6, true)}, {B200Q_ATTN_PAIR(4, 5, false), B200Q_ATTN_PAIR(4, 5, true)}}};
    static const KernelFn plain[2][2] = {B200Q_ATTN_PAIR(16, 0, false), B200Q_ATTN_PAIR(16, 1, false)};
#undef B200Q_ATTN_PAIR
    KernelFn kernel = bits == 16 ? plain[bf][wide_group] : quantised[bits == 4][g32][two][wide_group];
    static bool configured[32][64] = {};
    const int slot = bits == 16 ? 16 + bf * 2 + wide_group : (bits == 4) * 8 + g32 * 4 + two * 2 + wide_group;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[slot][dev & 63]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) != cudaSuccess)
            return B200Q_ERR_LAUNCH;
        configured[slot][dev & 63] = true;
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(launch_grid, chunks);
        cfg.blockDim = dim3(kSplitThreads);
        cfg.dynamicSmemBytes = total_smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = tuning_get("no_pdl") ? 0 : 1;
        if (cudaLaunchKernelEx(&cfg, kernel, sp) != cudaSuccess) return B200Q_ERR_LAUNCH;
    }
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(p.B * p.Hq);
        const bool wide = p.B * p.Hq < 2 * sm_count();
        cfg.blockDim = dim3((wide ? 32 : 8) * 32);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = tuning_get("no_pdl") ? 0 : 1;
        if (cudaLaunchKernelEx(&cfg, wide ? paged_attn_merge_kernel<32> : paged_attn_merge_kernel<8>, p) != cudaSuccess)
            return B200Q_ERR_LAUNCH;
    }
    return finish_launch();
}

}  // namespace

int attention_stage_launches_impl(int B, int Hkv, int max_blocks, int with_append) {
    if (B <= 0 || Hkv <= 0) return 0;
    if (B <= 65535 && choose_cluster(B, Hkv, 1, max_blocks, with_append != 0 ? AttnUse::kAppend : AttnUse::kDense, true).preferred) return 1;
    return 2 + (with_append ? 1 : 0);
}

size_t paged_gqa_workspace_bytes_impl(int B, int Hq, int Hkv, int D) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0) return 0;
    const int ranges = std::min(kMaxRanges, kMaxGrid * subs_for(std::min(Hkv, kAttnWarps)));
    return (size_t)(ranges + B) * Hq * (D + 2) * sizeof(float);
}

// Calls that the kernel without scratch served before the split-KV kernels took them on: a workspace that is missing or too small
// sends them back to it and is no error.
static bool scratch_optional(int Hkv, int q_dtype) { return q_dtype != B200Q_F16 || Hkv > kAttnWarps; }
// Page ranges that a workspace has room for (range r and sequence b meet in slot r + b); 0: too few, or no workspace.  kMaxGrid ranges
// fill every SM twice; more only serve the warps that fewer than 8 kv heads leave over, so a workspace without room for them is cut to,
// not refused.  Where scratch is optional, one range per SM is enough to be faster than one warp per head.
static int split_ranges(const void* workspace, size_t bytes, int B, int Hq, int Hkv, int D, int q_dtype) {
    if (workspace == nullptr) return 0;
    const int64_t ranges = (int64_t)(bytes / ((size_t)Hq * (D + 2) * sizeof(float))) - B;
    const int chunks = std::max(1, Hkv / kAttnWarps), at_least = scratch_optional(Hkv, q_dtype) ? (sm_count() + chunks - 1) / chunks : kMaxGrid;
    return ranges >= at_least ? (int)std::min<int64_t>(ranges, kMaxRanges) : 0;
}

int paged_gqa_decode_impl(int bits, const void* q, const uint8_t* k_codes, const uint8_t* v_codes, const void* k_scales,
                          const void* v_scales, const int32_t* block_table, const int32_t* lengths, void* out,
                          void* workspace, size_t workspace_bytes, int B, int Hq, int Hkv, int D, int page_size,
                          int64_t num_pages, int max_blocks, int group_size, float scale, int q_dtype,
                          int scale_dtype, int sink_tokens, int window_size, cudaStream_t stream) {
    int tp_in_slot = -1, tp_out_slot = -1;
    tp_take(&tp_in_slot, &tp_out_slot);
    if ((bits != 4 && bits != 8) || q == nullptr || k_codes == nullptr || v_codes == nullptr || k_scales == nullptr ||
        v_scales == nullptr || block_table == nullptr || lengths == nullptr || (out == nullptr && tp_out_slot < 0))
        return B200Q_ERR_BAD_ARG;
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || page_size <= 0 || num_pages <= 0 || max_blocks <= 0 ||
        group_size <= 0 || Hq % Hkv != 0 || !is_act_dtype(q_dtype) || !is_scale_dtype(scale_dtype) ||
        sink_tokens < 0 || window_size < 0)
        return B200Q_ERR_BAD_ARG;
    if (D > 128) return B200Q_ERR_UNSUPPORTED;
    const int Gd = (D + group_size - 1) / group_size;
    const int group = Hq / Hkv;
    const int dp = bits == 4 ? D / 2 : D;

    const bool fast_ok = tuning_get("attn.force_simple") == 0 && D == kHeadDim &&
                         scale_dtype == B200Q_F16 && (group_size == 32 || group_size == 64) && group <= 8 &&
                         heads_ok(Hkv) && page_size == 16 && B <= kMaxBatchFast &&
                         ((uintptr_t)q % 16 == 0) && ((uintptr_t)k_codes % 16 == 0) && ((uintptr_t)v_codes % 16 == 0) &&
                         ((uintptr_t)k_scales % 8 == 0) && ((uintptr_t)v_scales % 8 == 0);
    if (!fast_ok && tp_out_slot >= 0) return B200Q_ERR_UNSUPPORTED;   // the exchange exists only in the split-KV kernels
    auto simple = [&]() -> int {
        SimpleParams sp = {q, k_codes, v_codes, k_scales, v_scales, block_table, lengths, out,
                           B, Hq, Hkv, D, page_size, max_blocks, group_size, Gd, bits, q_dtype, scale_dtype,
                           num_pages, scale, sink_tokens, window_size, nullptr, 0, 0, 0};
        const int warps = 4;
        paged_attn_simple_kernel<<<(B * Hq + warps - 1) / warps, warps * 32, 0, stream>>>(sp);
        return finish_launch();
    };
    if (!fast_ok) return simple();
    // small batches: one cluster per (sequence, kv head), merged on chip - no workspace, no second launch
    const int ranges = split_ranges(workspace, workspace_bytes, B, Hq, Hkv, D, q_dtype);
    // A window bounds the walk whatever the length of the sequence.  Windows as long as the table stay with the split-KV kernels, whose dense result they
    // reproduce bit for bit; without a workspace only dense calls are served.
    const int64_t visited = ((int64_t)window_size + 15) / 16 + 1 + ((int64_t)sink_tokens + 15) / 16;
    const int walk_pages = window_size > 0 ? (int)std::min<int64_t>(max_blocks, visited) : max_blocks;
    const bool may = window_size == 0 || (ranges > 0 && window_size < (int64_t)max_blocks * page_size);
    const AttnUse use = window_size > 0 ? AttnUse::kWindow : AttnUse::kDense;
    const ClusterChoice choice = may && B <= 65535 && Hkv <= 65535 ? choose_cluster(B, Hkv, group, walk_pages, use, ranges > 0) : ClusterChoice{0, false};
    const int cluster = choice.preferred || ranges == 0 ? choice.size : 0;
    if (cluster > 0) {
        ClusterAttnParams c = {};
        if (tp_out_slot >= 0) c.tp_out = tp_slot(tp_out_slot)->out;
        c.q = q; c.q_dtype = q_dtype;
        c.k_codes = const_cast<uint8_t*>(k_codes); c.v_codes = const_cast<uint8_t*>(v_codes);
        c.k_scales = (__half*)const_cast<void*>(k_scales); c.v_scales = (__half*)const_cast<void*>(v_scales);
        c.block_table = block_table; c.lengths = lengths; c.out = out;
        c.B = B; c.Hq = Hq; c.Hkv = Hkv; c.P = page_size; c.max_blocks = max_blocks; c.G = group_size; c.Gd = Gd;
        c.group = group; c.bits = bits; c.S = cluster; c.num_pages = num_pages; c.scale = scale;
        c.row_bytes = Hkv * dp; c.scale_row_halves = Hkv * Gd;
        c.sink = sink_tokens; c.window = window_size; c.walk_pages = walk_pages;
        const int rc = launch_cluster_attention(c, stream);
        if (rc != B200Q_ERR_UNSUPPORTED) return rc;
    }
    if (ranges == 0) return scratch_optional(Hkv, q_dtype) && tp_out_slot < 0 ? simple() : (int)B200Q_ERR_WORKSPACE;

    AttnParams p = {};
    if (tp_out_slot >= 0) p.tp_out = tp_slot(tp_out_slot)->out;
    p.q = q; p.k_codes = k_codes; p.v_codes = v_codes;
    p.k_scales = (const __half*)k_scales; p.v_scales = (const __half*)v_scales;
    p.block_table = block_table; p.lengths = lengths; p.partial = (float*)workspace; p.out = out;
    p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.P = page_size; p.max_blocks = max_blocks; p.G = group_size; p.Gd = Gd;
    p.group = group; p.num_pages = num_pages; p.scale = scale; p.q_dtype = q_dtype; p.bits = bits;
    p.sink = sink_tokens;
    p.window = window_size;
    p.row_bytes = Hkv * dp;
    p.scale_row_halves = Hkv * Gd;
    const int rc = launch_split_attention(p, ranges, stream);
    return rc == B200Q_ERR_UNSUPPORTED && tp_out_slot < 0 ? simple() : rc;      // scales of very many kv heads do not fit a ring
}

// Plain fp16 / bf16 pages on the cluster and the split-KV kernels (bf16, 8 kv heads, split-KV / cluster, us: 8 sequences of 128 tokens 12.0 / 5.1,
// of 1024 14.8 / 11.3; 2 kv heads, 32 of 512 17.4 / 8.1); B200Q_ERR_UNSUPPORTED outside their shapes.  `verdict`: see AttnParams.
int paged_plain_attention_impl(const void* q, const void* k_pages, const void* v_pages, const int32_t* block_table, const int32_t* lengths,
                               void* out, void* workspace, size_t workspace_bytes, int B, int Hq, int Hkv, int D, int page_size,
                               int64_t num_pages, int max_blocks, float scale, int dtype, int32_t* verdict, cudaStream_t stream) {
    if (tuning_get("attn.force_simple") || D != kHeadDim || page_size != 16 || Hq / Hkv > 8 || !heads_ok(Hkv) || B > kMaxBatchFast ||
        ((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) % 16 != 0)
        return B200Q_ERR_UNSUPPORTED;
    if (workspace == nullptr || workspace_bytes < paged_gqa_workspace_bytes_impl(B, Hq, Hkv, D)) return B200Q_ERR_WORKSPACE;
    AttnParams p = {};
    p.q = q; p.k_codes = (const uint8_t*)k_pages; p.v_codes = (const uint8_t*)v_pages;
    p.block_table = block_table; p.lengths = lengths; p.partial = (float*)workspace; p.out = out;
    p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.D = D; p.P = page_size; p.max_blocks = max_blocks;
    p.group = Hq / Hkv; p.num_pages = num_pages; p.scale = scale; p.q_dtype = dtype; p.bits = 16;
    p.row_bytes = Hkv * kHeadDim * 2;
    p.verdict = verdict;
    const ClusterChoice choice =
        B <= 65535 && Hkv <= 65535 ? choose_cluster(B, Hkv, Hq / Hkv, max_blocks, AttnUse::kPlain, true) : ClusterChoice{0, false};
    if (choice.preferred && choice.size > 0) {
        ClusterAttnParams c = {};
        c.q = q; c.q_dtype = dtype;
        c.k_codes = const_cast<uint8_t*>(p.k_codes); c.v_codes = const_cast<uint8_t*>(p.v_codes);
        c.block_table = block_table; c.lengths = lengths; c.out = out;
        c.B = B; c.Hq = Hq; c.Hkv = Hkv; c.P = page_size; c.max_blocks = c.walk_pages = max_blocks;
        c.group = p.group; c.bits = 16; c.S = choice.size; c.num_pages = num_pages; c.scale = scale;
        c.row_bytes = p.row_bytes; c.verdict = verdict;
        const int rc = launch_cluster_attention(c, stream);
        if (rc != B200Q_ERR_UNSUPPORTED) return rc;
    }
    return launch_split_attention(p, kMaxRanges, stream);
}

// Decode-layer attention in one call: split + rotate + append (as rope_kv_append_impl) followed by the attention over
// the cache including the new token.  Small batches run it as ONE launch of the cluster kernel; otherwise the two
// stages are launched one after the other (q_scratch [B, Hq, D] then holds the rotated queries).
int rope_kv_append_impl(const void* qkv, const float* cos_table, const float* sin_table, const int32_t* positions,
                        const int32_t* block_table, void* q_out, uint8_t* k_codes, uint8_t* v_codes, void* k_scales,
                        void* v_scales, int bits, int B, int Hq, int Hkv, int D, int page_size, int64_t num_pages,
                        int max_blocks, int group_size, int table_len, cudaStream_t stream);

int rope_append_attention_impl(const void* qkv, const float* cos_table, const float* sin_table, const int32_t* positions,
                               int table_len, int bits, uint8_t* k_codes, uint8_t* v_codes, void* k_scales, void* v_scales,
                               const int32_t* block_table, const int32_t* lengths, void* out, void* q_scratch, void* workspace,
                               size_t workspace_bytes, int B, int Hq, int Hkv, int D, int page_size, int64_t num_pages,
                               int max_blocks, int group_size, float scale, cudaStream_t stream) {
    if (qkv == nullptr || cos_table == nullptr || sin_table == nullptr || positions == nullptr || k_codes == nullptr ||
        v_codes == nullptr || k_scales == nullptr || v_scales == nullptr || block_table == nullptr || lengths == nullptr) {
        tp_discard();
        return B200Q_ERR_BAD_ARG;
    }
    if ((bits != 4 && bits != 8) || B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || page_size <= 0 || num_pages <= 0 ||
        max_blocks <= 0 || group_size <= 0 || table_len <= 0 || Hq % Hkv != 0) {
        tp_discard();
        return B200Q_ERR_BAD_ARG;
    }
    const int group = Hq / Hkv;
    const int Gd = (D + group_size - 1) / group_size;
    const int dp = bits == 4 ? D / 2 : D;
    const bool fast_ok = tuning_get("attn.force_simple") == 0 && D == 128 && (group_size == 32 || group_size == 64) &&
                         group <= 8 && heads_ok(Hkv) && page_size == 16 && B <= 65535 && ((uintptr_t)qkv % 16 == 0) &&
                         ((uintptr_t)k_codes % 16 == 0) && ((uintptr_t)v_codes % 16 == 0) && ((uintptr_t)k_scales % 8 == 0) &&
                         ((uintptr_t)v_scales % 8 == 0);
    const bool two_stages = q_scratch != nullptr && split_ranges(workspace, workspace_bytes, B, Hq, Hkv, D, B200Q_F16) > 0;
    const ClusterChoice choice = fast_ok ? choose_cluster(B, Hkv, group, max_blocks, AttnUse::kAppend, two_stages) : ClusterChoice{0, false};
    const int cluster = choice.preferred || !two_stages ? choice.size : 0;
    if (cluster > 0) {
        int tp_in_slot = -1, tp_out_slot = -1;
        tp_take(&tp_in_slot, &tp_out_slot);
        if (out == nullptr && tp_out_slot < 0) return B200Q_ERR_BAD_ARG;
        ClusterAttnParams c = {};
        if (tp_out_slot >= 0) c.tp_out = tp_slot(tp_out_slot)->out;
        c.qkv = (const __half*)qkv; c.cos_table = cos_table; c.sin_table = sin_table; c.positions = positions;
        c.table_len = table_len; c.fused = 1;
        c.k_codes = k_codes; c.v_codes = v_codes; c.k_scales = (__half*)k_scales; c.v_scales = (__half*)v_scales;
        c.block_table = block_table; c.lengths = lengths; c.out = out;
        c.B = B; c.Hq = Hq; c.Hkv = Hkv; c.P = page_size; c.max_blocks = max_blocks; c.G = group_size; c.Gd = Gd;
        c.group = group; c.bits = bits; c.S = cluster; c.num_pages = num_pages; c.scale = scale;
        c.row_bytes = Hkv * dp; c.scale_row_halves = Hkv * Gd;
        c.walk_pages = max_blocks;
        const int rc = launch_cluster_attention(c, stream);
        if (rc != B200Q_ERR_UNSUPPORTED) return rc;
        if (q_scratch == nullptr) return B200Q_ERR_WORKSPACE;
        // fall through to the two-stage route with the exchange slots restored for the attention stage
        int rc2 = rope_kv_append_impl(qkv, cos_table, sin_table, positions, block_table, q_scratch, k_codes, v_codes, k_scales,
                                      v_scales, bits, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size, table_len, stream);
        if (rc2 != B200Q_OK) return rc2;
        if (tp_out_slot >= 0) return B200Q_ERR_UNSUPPORTED;
        return paged_gqa_decode_impl(bits, q_scratch, k_codes, v_codes, k_scales, v_scales, block_table, lengths, out, workspace,
                                     workspace_bytes, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size, scale,
                                     B200Q_F16, B200Q_F16, 0, 0, stream);
    }
    if (q_scratch == nullptr) {
        tp_discard();
        return B200Q_ERR_WORKSPACE;
    }
    const int rc = rope_kv_append_impl(qkv, cos_table, sin_table, positions, block_table, q_scratch, k_codes, v_codes, k_scales,
                                       v_scales, bits, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size, table_len, stream);
    if (rc != B200Q_OK) {
        tp_discard();
        return rc;
    }
    return paged_gqa_decode_impl(bits, q_scratch, k_codes, v_codes, k_scales, v_scales, block_table, lengths, out, workspace,
                                 workspace_bytes, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size, scale, B200Q_F16,
                                 B200Q_F16, 0, 0, stream);
}

// ------------------------------------------------------------------------------------------------
// Variant without a caller-supplied workspace: the split-KV partials live in a fixed array in
// device memory that belongs to the library image.
// ------------------------------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = 8u << 20;     // 8 MiB, held by every GPU that loads the library
static __device__ __align__(256) unsigned char g_attn_static_scratch[kStaticScratchBytes];

size_t paged_gqa_static_scratch_bytes_impl() { return kStaticScratchBytes; }

int paged_gqa_decode_static_impl(int bits, const void* q, const uint8_t* k_codes, const uint8_t* v_codes,
                                 const void* k_scales, const void* v_scales, const int32_t* block_table,
                                 const int32_t* lengths, void* out, int B, int Hq, int Hkv, int D, int page_size,
                                 int64_t num_pages, int max_blocks, int group_size, float scale, int q_dtype,
                                 int scale_dtype, cudaStream_t stream) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0) {
        tp_discard();
        return B200Q_ERR_BAD_ARG;
    }
    // In host code the array's name is only a handle; the device address has to be asked for, once per
    // device, with that device current.
    static void* scratch_ptr[64] = {};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        tp_discard();
        return B200Q_ERR_LAUNCH;
    }
    void* ptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (scratch_ptr[dev] == nullptr) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_attn_static_scratch) != cudaSuccess || p == nullptr) {
                tp_discard();
                return B200Q_ERR_LAUNCH;
            }
            scratch_ptr[dev] = p;
        }
        ptr = scratch_ptr[dev];
    }
    // Only the split-KV kernels use the scratch: the size check is theirs (problems that take the one-warp-per-head
    // kernel need none), reported here under this entry point's own code.
    const int rc = paged_gqa_decode_impl(bits, q, k_codes, v_codes, k_scales, v_scales, block_table, lengths, out, ptr,
                                         kStaticScratchBytes, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size,
                                         scale, q_dtype, scale_dtype, 0, 0, stream);
    return rc == B200Q_ERR_WORKSPACE ? B200Q_ERR_STATIC_SCRATCH : rc;
}

// ------------------------------------------------------------------------------------------------
// Block-sparse decode: key j of a sequence of L tokens is attended iff block_mask[(L-1)/bs][j/bs] != 0 (the decode
// row of the reference's block_sparse mask; the causal bound j <= L-1 holds for every cached token).
// When bs is a multiple of the page size the attended keys are whole pages (and possibly the partly filled last
// one), and softmax attention does not depend on the order of its keys: one warp per sequence compacts the
// attended pages into a private block table with the matching length, and the dense kernels run on that.
// ------------------------------------------------------------------------------------------------
namespace {
__global__ void __launch_bounds__(128) block_sparse_pages_kernel(const int32_t* block_table, const int32_t* lengths,
                                                                 const uint8_t* block_mask, int n_qblocks, int n_kblocks,
                                                                 int pages_per_block, int P, int max_blocks, int B,
                                                                 int32_t* table_out, int32_t* lengths_out) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= B) return;
    const int L = clamp_len(lengths[b], max_blocks * P);
    const int npages = (L + P - 1) / P;
    const int bs = pages_per_block * P;
    const int qb = L > 0 ? (L - 1) / bs : 0;
    const uint8_t* row = (L > 0 && qb < n_qblocks) ? block_mask + (size_t)qb * n_kblocks : nullptr;
    const int32_t* src = block_table + (size_t)b * max_blocks;
    int32_t* dst = table_out + (size_t)b * max_blocks;
    int count = 0, tokens = 0;
    for (int p0 = 0; p0 < npages; p0 += 32) {
        const int pg = p0 + lane;
        bool vis = false;
        if (pg < npages && row != nullptr) {
            const int kb = pg / pages_per_block;
            vis = kb < n_kblocks && row[kb] != 0;
        }
        const uint32_t ballot = __ballot_sync(0xffffffffu, vis);
        if (vis) dst[count + __popc(ballot & ((1u << lane) - 1u))] = src[pg];
        count += __popc(ballot);
        // every attended page is full except the sequence's last page
        tokens += __popc(ballot) * P;
        if (npages - 1 >= p0 && npages - 1 < p0 + 32 && ((ballot >> (npages - 1 - p0)) & 1u)) tokens -= npages * P - L;
    }
    for (int i = count + lane; i < max_blocks; i += 32) dst[i] = -1;
    if (lane == 0) lengths_out[b] = tokens;
}
}  // namespace

int paged_gqa_decode_block_sparse_impl(int bits, const void* q, const uint8_t* k_codes, const uint8_t* v_codes,
                                       const void* k_scales, const void* v_scales, const int32_t* block_table,
                                       const int32_t* lengths, void* out, void* workspace, size_t workspace_bytes,
                                       const uint8_t* block_mask, int n_qblocks, int n_kblocks, int block_size,
                                       int32_t* page_scratch, int B, int Hq, int Hkv, int D, int page_size,
                                       int64_t num_pages, int max_blocks, int group_size, float scale, int q_dtype,
                                       int scale_dtype, cudaStream_t stream) {
    if (block_mask == nullptr || n_qblocks <= 0 || n_kblocks <= 0 || block_size <= 0) {
        tp_discard();
        return B200Q_ERR_BAD_ARG;
    }
    if (page_scratch != nullptr && page_size > 0 && block_size % page_size == 0 && B > 0 && max_blocks > 0 &&
        block_table != nullptr && lengths != nullptr) {
        int32_t* table2 = page_scratch;
        int32_t* lengths2 = page_scratch + (size_t)B * max_blocks;
        block_sparse_pages_kernel<<<(B + 3) / 4, 128, 0, stream>>>(block_table, lengths, block_mask, n_qblocks, n_kblocks,
                                                                  block_size / page_size, page_size, max_blocks, B, table2,
                                                                  lengths2);
        const int rc = finish_launch();
        if (rc != B200Q_OK) {
            tp_discard();
            return rc;
        }
        return paged_gqa_decode_impl(bits, q, k_codes, v_codes, k_scales, v_scales, table2, lengths2, out, workspace,
                                     workspace_bytes, B, Hq, Hkv, D, page_size, num_pages, max_blocks, group_size, scale,
                                     q_dtype, scale_dtype, 0, 0, stream);
    }
    // any block size: the one-warp-per-head kernel with a per-token test
    tp_discard();
    if ((bits != 4 && bits != 8) || q == nullptr || k_codes == nullptr || v_codes == nullptr || k_scales == nullptr ||
        v_scales == nullptr || block_table == nullptr || lengths == nullptr || out == nullptr)
        return B200Q_ERR_BAD_ARG;
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || page_size <= 0 || num_pages <= 0 || max_blocks <= 0 ||
        group_size <= 0 || Hq % Hkv != 0 || !is_act_dtype(q_dtype) || !is_scale_dtype(scale_dtype))
        return B200Q_ERR_BAD_ARG;
    if (D > 128) return B200Q_ERR_UNSUPPORTED;
    SimpleParams sp = {q, k_codes, v_codes, k_scales, v_scales, block_table, lengths, out,
                       B, Hq, Hkv, D, page_size, max_blocks, group_size, (D + group_size - 1) / group_size, bits, q_dtype,
                       scale_dtype, num_pages, scale, 0, 0, block_mask, block_size, n_qblocks, n_kblocks};
    const int warps = 4;
    paged_attn_simple_kernel<<<(B * Hq + warps - 1) / warps, warps * 32, 0, stream>>>(sp);
    return finish_launch();
}

}  // namespace b200q
