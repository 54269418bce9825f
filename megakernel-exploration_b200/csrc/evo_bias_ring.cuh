// Ring of bias half tiles of the D = 96 / 128 forward (evo_fwd_wide.cuh).  Four half tiles make a round, in
// the order stream 0 left, right, stream 1 left, right; half tile i of round n is load 4 n + i and lies in
// slot (4 n + i) % 3.  A stream reads its own two of a round and never looks at the other's.
//
// A slot is handed back ("empty") by whichever stream read it, to the one warp that fills all of them.  "Full" barriers
// belong to a half tile's place in the round, not to its slot: a parity wait tells phases apart only for a waiter that has
// seen the one before, and bulk loads land in any order.  With a barrier per slot a stream would meet phases
// made by the other's loads: stream 1's first wait on slot 0 (load 3, the slot's second phase) would pass before
// load 0 has landed there, read what the slot held before and hand it back early.  By place in the round each barrier
// has one waiter, which sees every phase; it is armed again only when that waiter is past the last one, because load
// k + 4 is issued after load k + 3, which waits for the release of load k.
//
// Plain host code as well, so that a model of the protocol can be run without a GPU.
#pragma once

#ifdef __CUDACC__
#define EVO_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define EVO_HOST_DEVICE inline
#endif

namespace evo {

struct WideBiasRing {
    static constexpr int SLOTS = 3;          // buffers, and their "empty" barriers
    static constexpr int PER_ROUND = 4;      // half tiles of a round, and "full" barriers
    int slot;                                // of the half tile in hand
    unsigned use;                            // how often the ring has come round to it
    EVO_HOST_DEVICE static WideBiasRing at(int load) { return WideBiasRing{load % SLOTS, static_cast<unsigned>(load / SLOTS)}; }
    EVO_HOST_DEVICE void advance(int loads) {                  // by up to SLOTS
        slot += loads;
        if (slot >= SLOTS) { slot -= SLOTS; ++use; }
    }
    // parity of the release that frees the slot for this use (use > 0)
    EVO_HOST_DEVICE unsigned empty_parity() const { return (use - 1) & 1u; }
    // barrier and parity of half tile `half` of stream s in round n
    EVO_HOST_DEVICE static int full_bar(int s, int half) { return 2 * s + half; }
    EVO_HOST_DEVICE static unsigned full_parity(int n) { return static_cast<unsigned>(n) & 1u; }
};

}  // namespace evo
