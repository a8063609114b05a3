// Choices of the decode attention, plain C++ so that they can be checked without a GPU.
#pragma once

#include <algorithm>
#include <stdint.h>

#include "ring.h"

namespace b200q {

// What a warp of a cluster CTA appends of the new token: the last warp its V row, the one before it its K row, so that every byte has
// one writer.  With sixteen warps neither has a query row to rotate.
enum AppendRole { kAppendNothing, kAppendK, kAppendV };
B200Q_HD AppendRole append_role(int warp, int warps) { return warp == warps - 1 ? kAppendV : warp == warps - 2 ? kAppendK : kAppendNothing; }

enum class AttnUse {
    kDense,       // quantised pages, every token
    kAppend,      // the same with the new token's append in the launch (three launches against one)
    kWindow,      // quantised pages, sliding window and sinks
    kPlain        // fp16 / bf16 pages
};
struct ClusterQuery {
    int B, Hkv, group;          // sequences, kv heads of this process, query heads per kv head
    int walk_pages;             // pages that a sequence can have to visit: the block table's capacity or the window's (lengths live on the device)
    AttnUse use;
    bool split;                 // the split-KV kernels could take the call; without them (no workspace) the rule is the one for tables of any
                                // length, so a call is not refused or served by its length
    int tp_world;               // "ts.tp_world": the choice follows the kv heads of the UNSHARDED cache, so that a tensor-parallel rank runs the same
                                // kernel, and the same summation order, as the unsharded call
    int mode, forced_size;      // "attn.cluster": 1 whenever possible, -1 never, 0 by the rule; "attn.cluster_size"
    int sms;
};
struct ClusterChoice { int size; bool preferred; };      // CTAs per cluster (0: not possible), and whether split-KV would be slower

inline ClusterChoice cluster_choice(const ClusterQuery& c) {
    if (c.mode < 0 || (c.mode > 0 && (int64_t)c.B * c.Hkv > 65535)) return {0, false};
    const int kv = c.Hkv * c.tp_world;
    const int64_t heads = (int64_t)c.B * kv;
    const int forced = c.forced_size;
    if (forced == 1 || forced == 2 || forced == 4 || forced == 8 || forced == 16)
        return {c.mode == 0 && heads * forced > 2 * c.sms ? 0 : forced, c.mode > 0 || heads * forced * 4 <= 3 * c.sms};
    if (c.mode > 0) return {8, true};
    // Eight CTAs per cluster while the clusters fill at most three quarters of the SMs (the opt-in size 16 is slower at every length: one
    // sequence of q8, 8 kv heads, sizes 4 / 8 / 16: 1024 tokens 14.3 / 12.3 / 18.4 us, 8192 26.6 / 20.5 / 24.6).
    if (heads * 8 * 4 <= 3 * c.sms) {
        // Plain pages and windows only up to the walk at which the split-KV kernels, which use all SMs, become the faster ones: the cluster
        // takes 0.85 us per 1024 tokens whatever the heads, split-KV 0.3 to 0.6 per sequence but starts 2 to 11 us later.
        // Split-KV / cluster, us, plain pages of 8192, 16384 and 65536 tokens: one sequence of 8 kv heads 12.6 / 12.4, 18.2 / 19.3, 46.4 / 56.7,
        // of 4 heads 11.4 / 11.2, 13.4 / 18.2, 30.0 / 55.8, of one 18.5 / 10.8, 20.2 / 17.0, 31.8 / 55.4; four sequences of 2 heads
        // 17.4 / 12.9, 22.7 / 19.1, 53.4 / 57.8; eight of one head 28.2 / 15.3, 37.4 / 23.5, 95.5 / 69.5.  q8 windows of 8192 and 16384, one
        // sequence: 8 heads 14.0 / 13.5 and 17.4 / 20.5, 4 heads 12.3 / 13.1 and 17.0 / 19.8, one head 20.1 / 12.8 and 22.7 / 19.1.  More than
        // four query heads per kv head cost the cluster a quarter more per page; with a number of kv heads that does not divide 8
        // split-KV starts sooner.  (Dense quantised calls and the append have this form at any length.)
        const bool bounded = c.split && (c.use == AttnUse::kPlain || c.use == AttnUse::kWindow) && c.B < 6;
        if (!bounded) return {8, true};
        const int64_t one = kv >= 8 ? 544 : 8 % kv != 0 ? 288 : std::max(416, 1408 / kv);      // pages, for one sequence
        const int64_t longest = one * (c.B * c.B + 7) / 8 * (c.group > 4 ? 3 : 4) / 4;
        return {8, c.walk_pages <= longest};
    }
    // More heads: as many CTAs per cluster as leave all clusters resident at once, if a warp's walk is short.  A page costs a warp about
    // one microsecond (it walks alone), the launch 5 us; the split-KV kernel balances ragged batches over all SMs, but with its partial
    // results and the merge launch takes 9 to 17 us for the shortest ones.  Split-KV / cluster, us, q4, 8 kv heads, equal lengths and
    // ragged ones down to an eighth: 2 sequences of 2048
    // tokens 11.1 / 8.2 and 9.1 / 8.1 (of 4096 in q8 13.0 / 12.1 and 11.1 / 11.5: not taken); 7 of 1024 15.7 / 8.2 and 14.4 / 8.0, of 3072
    // 20.2 / 15.6 and 16.5 / 14.6; 16 of 128 10.5 / 5.8, of 1024 15.1 / 12.6 and 13.4 / 11.1.  Fewer than 8 kv heads cost the split-KV
    // kernel more: 2 heads, 16 sequences of 4096 tokens 18.7 / 13.1 and 14.5 / 11.4 (of 8192, 7 sequences, 19.3 / 17.8 and 15.4 / 16.8).  With
    // the append in the same launch the cluster wins 1 to 3 us more (a layer of 2 sequences of 4000 tokens 65.2 / 63.8, 8 of 3000
    // 91.4 / 86.8, 16 of 1000 89.5 / 87.9).
    for (int size = 4; c.split && size >= 1; size /= 2) {
        if (heads * size * 8 > 7 * (int64_t)c.sms) continue;
        const int warps = size * (c.use == AttnUse::kPlain ? 8 : 16);      // plain pages: no room for more rings
        const int64_t walk = ((int64_t)c.walk_pages + warps - 1) / warps;
        int longest = 4;
        if (size == 4 && heads < 24) longest = kv >= 8 ? 2 : 3;
        if (size == 4 && kv < 4) longest = 5;
        if (size == 2) longest = (int)heads / 10;
        if (walk <= longest + (c.use == AttnUse::kAppend ? 2 : 0)) return {size, true};
        break;
    }
    // up to two waves of clusters stay possible for callers without a workspace
    return {heads * 8 <= 2 * c.sms ? 8 : 0, false};
}

}  // namespace b200q
