// Positions in rings of shared- or tensor-memory slots, plain C++ so that the arithmetic can be checked without a GPU.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define B200Q_HD __host__ __device__ __forceinline__
#else
#define B200Q_HD inline
#endif

namespace b200q {

// Slot of an item and the parity of that slot's phase: item i of a ring of n slots has slot i % n and parity (i / n) & 1.
struct RingPos {
    int slot = 0;
    uint32_t par = 0;
    B200Q_HD void advance(int by, int n) {      // by >= 0
        slot += by;
        while (slot >= n) { slot -= n; par ^= 1u; }
    }
};

// An MMA warp's place in the rings of activation chunks and of A chunks.  Chunks of k are numbered over all items of the CTA; a
// chunk of k has MATS chunks of A.  With two matrices warp j takes A chunk j of every chunk of k, with one every other chunk.
template <int MATS>
struct ChunkWalk {
    static constexpr int kSkip = MATS == 2 ? 0 : 1;      // chunks of the other warp between two of this one's
    RingPos x, a;
    int at = 0;                                          // the chunk of k that x and a stand for
    B200Q_HD explicit ChunkWalk(int j) { if (MATS == 2) a.slot = j; }
    B200Q_HD static int first(int j) { return MATS == 2 ? 0 : j; }
    // On to a chunk that is issued now.  Never past it: with an odd number of chunks per item and one matrix, the next item's first chunk
    // can be the one right after this warp's last.
    B200Q_HD void to(int chunk, int x_slots, int a_slots) {
        x.advance(chunk - at, x_slots);
        a.advance(MATS * (chunk - at), a_slots);
        at = chunk;
    }
};

}  // namespace b200q
