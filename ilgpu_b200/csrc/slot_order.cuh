// The order of a tile's slots, or of a block's words: the check that ranks taken with atomics came out in order, and
// what puts them in order when they did not (see the top of digit_pass.cuh).  The device code and a host-side
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
// this).  wrong(p): whether those at p and p + 1 are; swap(p) exchanges them.  `meet` is the block's barrier: meet(q)
// returns whether q is true for any thread.
template <typename Wrong, typename Swap, typename Meet>
B200ALG_HD inline void exchange_neighbours(int count, int tid, int threads, Wrong wrong, Swap swap, Meet meet) {
    bool again = true;
    for (int round = 0; again && round < count; ++round) {
        bool moved = false;
        for (int odd = 0; odd < 2; ++odd) {
            for (int p = 2 * tid + odd; p + 1 < count; p += 2 * threads) {
                if (!wrong(p)) continue;
                swap(p);
                moved = true;
            }
            again = meet(moved);  // (of the second half: of either)
        }
    }
}

template <typename K, bool VALUES, typename XF, typename Meet>
B200ALG_HD inline void put_in_order(K *slots, unsigned short *place, int tile, int tid, int threads, XF xf, int shift, Meet meet) {
    exchange_neighbours(
        tile, tid, threads,
        [=](int p) { return out_of_order<K, VALUES>(slots[p], slots[p + 1], VALUES ? place[p] : 0u, VALUES ? place[p + 1] : 0u, xf, shift); },
        [=](int p) {
            const K k = slots[p];
            slots[p] = slots[p + 1];
            slots[p + 1] = k;
            if (VALUES) {
                const unsigned short s = place[p];
                place[p] = place[p + 1];
                place[p + 1] = s;
            }
        },
        meet);
}

// ---- the words of the sort in one block (local_sort.cuh) -----------------------------------
// A word stands for an element: by place, its place in the block is in the lowest kPlaceBits and its key is looked
// up there; else it is the key, less the smallest one.  Words of places past the last element sort behind all others.
constexpr int kPlaceBits = 14;
B200ALG_HD inline unsigned int place_of(unsigned int word) { return word & ((1u << kPlaceBits) - 1u); }

template <typename K, bool PLACE> B200ALG_HD inline K word_key(unsigned int word, const K *keys, K low) {
    if constexpr (PLACE) return keys[place_of(word)];
    else return (K)(low + (K)word);
}
// (two neighbours of the sorted order)
template <typename K, bool PLACE> B200ALG_HD inline bool words_out_of_order(K key_a, unsigned int a, K key_b, unsigned int b) {
    if constexpr (PLACE) return key_a > key_b || (key_a == key_b && place_of(a) > place_of(b));
    else return a > b;
}
// Whether a word that came out behind the last place of an element stands for one all the same.
template <bool PLACE> B200ALG_HD inline bool is_stray(unsigned int word, int count) {
    if constexpr (PLACE) return place_of(word) < (unsigned int)count;
    else return word != ~0u;
}
// `all` words, of which `count` are elements.
template <typename K, bool PLACE, typename Meet>
B200ALG_HD inline void put_words_in_order(unsigned int *words, const K *keys, K low, int count, int all, int tid, int threads, Meet meet) {
    auto key = [=](unsigned int word) { return PLACE && place_of(word) >= (unsigned int)count ? (K)~(K)0 : word_key<K, PLACE>(word, keys, low); };
    exchange_neighbours(
        all, tid, threads, [=](int p) { return words_out_of_order<K, PLACE>(key(words[p]), words[p], key(words[p + 1]), words[p + 1]); },
        [=](int p) {
            const unsigned int w = words[p];
            words[p] = words[p + 1];
            words[p + 1] = w;
        },
        meet);
}

}  // namespace b200alg
