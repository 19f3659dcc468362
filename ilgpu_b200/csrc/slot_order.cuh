// The order of a tile's slots: the check that ranks taken with atomics came out in order, and what puts
// a tile in order when they did not (see the top of digit_pass.cuh).  The device code and a host-side
// test share it: no hardware was seen to serve a warp's atomics in another order than the lanes'.
#pragma once

#if defined(__CUDACC__)
#define B200ALG_HD __host__ __device__
#else
#define B200ALG_HD
#endif

namespace b200alg {

// Whether of two neighbouring slots the first has to come after the second (and must not).
template <typename K, bool VALUES, typename XF>
B200ALG_HD inline bool out_of_order(K first, K second, unsigned int first_place, unsigned int second_place, XF xf, int shift) {
    if constexpr (!VALUES) {
        const K sorted = (K)((K)~(K)0 >> (8 * (int)sizeof(K) - 8 - shift));  // this digit and the ones below it
        return (K)(xf(first) & sorted) > (K)(xf(second) & sorted);
    } else {
        return (((xf(first) ^ xf(second)) >> shift) & 0xFFu) == 0 && first_place > second_place;
    }
}

// Neighbours that are the wrong way round change places until none are (every thread of the block calls
// this).  `meet` is the block's barrier: meet(p) returns whether p is true for any thread.
template <typename K, bool VALUES, typename XF, typename Meet>
B200ALG_HD inline void put_in_order(K *slots, unsigned short *place, int tile, int tid, int threads, XF xf, int shift, Meet meet) {
    bool again = true;
    for (int round = 0; again && round < tile; ++round) {
        bool moved = false;
        for (int odd = 0; odd < 2; ++odd) {
            for (int p = 2 * tid + odd; p + 1 < tile; p += 2 * threads) {
                if (!out_of_order<K, VALUES>(slots[p], slots[p + 1], VALUES ? place[p] : 0u, VALUES ? place[p + 1] : 0u, xf, shift)) continue;
                const K k = slots[p];
                slots[p] = slots[p + 1];
                slots[p + 1] = k;
                if (VALUES) {
                    const unsigned short s = place[p];
                    place[p] = place[p + 1];
                    place[p + 1] = s;
                }
                moved = true;
            }
            again = meet(moved);  // (of the second half: of either)
        }
    }
}

}  // namespace b200alg
