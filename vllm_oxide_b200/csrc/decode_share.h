// How a decode step's attention blocks are dealt out to requests of very different lengths: the kernel (attention_mma.cu,
// "Requests of very different lengths") and the host, which decides whether a step is worth it, run the same search.
#pragma once
#ifdef __CUDACC__
#define VOB_BOTH __host__ __device__ __forceinline__
#else
#define VOB_BOTH inline
#endif

constexpr int DEC_TILE_KEYS = 64;          // keys of a tile
constexpr int DEC_MIN_TILES = 3;           // fewest tiles a block is started for; measured on whole decode steps at batch 1: 8,192 keys
                                           // 0.808 ms with 3, 0.838 with 2, 0.812 with 4

// The smallest number of tiles a block (at least DEC_MIN_TILES, and an even share of `total` tiles over `want` blocks) at which
// the requests need no more than `blocks` blocks. need(share): the sum over the requests of max(1, ceil(tiles / share)). Twice the
// even share always suffices where blocks >= want / 2 + requests: want / 2 blocks hold the whole shares, every request has one rest.
template <typename Need> VOB_BOTH int balance_share(int total, int want, int blocks, Need need) {
    int lo = (total + want - 1) / want;
    if (lo < DEC_MIN_TILES) lo = DEC_MIN_TILES;
    // upwards in steps that double until a share suffices (mostly the first or the second does), then by halving. `need` stands here
    // once: the kernel comes by with cold instruction caches.
    int hi = 2 * lo, at = lo, step = 1;
    bool found = false;
    while (lo < hi) {
        if (need(at) <= blocks) {
            hi = at;
            found = true;
        } else {
            lo = at + 1;
        }
        at = (lo + hi) / 2;
        if (!found) {
            at = lo + step - 1 < hi ? lo + step - 1 : hi - 1;
            step *= 2;
        }
    }
    return lo;
}

// Blocks of a balanced launch a kv head: those that are to be filled, and enough for a rest of every request.
VOB_BOTH int balance_blocks(int want, int requests) { return want / 2 + requests > want ? want / 2 + requests : want; }
