// The sort of up to kLocalMost elements by one block, in shared memory.
//
// What bounds it is the chain of steps of a pass and, from some 4000 elements on, the trips to random
// words of shared memory (a returning atomic, a look-up and a store per element and pass: 3.5 cycles of
// the pipe each for 32 lanes).  So there are few passes, and a pass moves 4 bytes per element whatever the
// keys and values are:
//
//   - Keys are taken as their distance from the smallest one.  Digits of up to nine bits cover the upper
//     27 bits of the range in three passes.  Few keys agree in all of these unless the range has outliers;
//     the writer compares neighbours by their whole keys, and where some are out of order it puts the groups
//     that agree in the upper bits in order.  Where there are too many, the passes run again over all bits.
//   - Where the range has more bits, those below the lowest one that a key of each thread has (in its distance) are left
//     out as well: whole numbers kept as floating-point end in zeros, and are few bits without these.
//   - With values or 8-byte keys an element travels as a word: its place in the block (14 bits) below the
//     digits that are still to come (18 bits after the first pass).  Keys and values stay where they were
//     loaded and are fetched by place in the end.  Keys of up to four bytes alone travel as themselves.
//   - The counts of two digits share a word (a block holds fewer than 2^14 elements), which halves what turning
//     counts into places reads and writes.  The atomic that returns costs the same: 3.53 against 3.57 cycles on
//     random digits.
//
// Order.  As in the digit pass, lanes that meet in one word are not promised any order; the comparison of
// whole keys (and of places, where they are equal) sees to that as well.
#pragma once

#include "sort_common.cuh"

namespace b200alg {

constexpr int kLocalMost = 12288;            // elements: 24 for each of 512 threads
static_assert(kLocalMost <= 1 << kPlaceBits, "a place fits its bits, a count its half of a word");
constexpr int kLocalDigitBits = 9;
constexpr int kLocalWords = 1 << (kLocalDigitBits - 1);  // counter words of a warp
constexpr int kLocalPrefixBits = 3 * kLocalDigitBits;
static_assert(kLocalPrefixBits - kLocalDigitBits + kPlaceBits <= 32, "the digits to come fit above the place");
constexpr int kLocalRows = 8;                // warps whose counts a thread adds up

// Shared memory besides the elements: counter tables, what the parts of the warps add up to, small words.
struct LocalShared {
    unsigned int *table;  // [warps][kLocalWords]: digit d in word d % 256, upper half from 256 on
    unsigned int *part;   // [threads / 256][kLocalWords]
    unsigned int *warp_sum;          // [8]
    unsigned int *found;             // neighbours out of order
    unsigned int *seen;              // [2]: bits of some keys' distances
    unsigned long long *low, *high;  // [32]
};
__host__ __device__ constexpr int local_fixed_bytes(int threads) { return threads / 32 * kLocalWords * 4 + threads / 256 * kLocalWords * 4 + 2 * 32 * 8 + 64; }
__device__ __forceinline__ LocalShared local_shared(unsigned char *smem) {
    const int threads = (int)blockDim.x;
    LocalShared s;
    s.table = reinterpret_cast<unsigned int *>(smem);
    s.part = s.table + threads / 32 * kLocalWords;
    s.low = reinterpret_cast<unsigned long long *>(s.part + threads / 256 * kLocalWords);
    s.high = s.low + 32;
    s.warp_sum = reinterpret_cast<unsigned int *>(s.high + 32);
    s.found = s.warp_sum + 8;
    s.seen = s.found + 1;
    return s;
}

__device__ __forceinline__ void local_clear(const LocalShared &s) {  // this warp's counters
    uint4 *mine = reinterpret_cast<uint4 *>(s.table + (threadIdx.x >> 5) * kLocalWords);
#pragma unroll
    for (int i = 0; i < kLocalWords / 4 / 32; ++i) mine[i * 32 + (threadIdx.x & 31)] = make_uint4(0u, 0u, 0u, 0u);
}

// Counts `digit` on the warp's table; how many of that digit the warp has counted before.
__device__ __forceinline__ unsigned int local_rank(unsigned int *mine, unsigned int digit) {
    const unsigned int half = digit >> (kLocalDigitBits - 1) << 4;
    return (atomicAdd(mine + (digit & (kLocalWords - 1)), 1u << half) >> half) & 0xFFFFu;
}
// Where the warp's elements of the digit begin, once local_places has run.
__device__ __forceinline__ unsigned int local_place(const unsigned int *mine, unsigned int digit) {
    return (mine[digit & (kLocalWords - 1)] >> (digit >> (kLocalDigitBits - 1) << 4)) & 0xFFFFu;
}

// Turns the warps' counts (complete behind a barrier) into the places where each warp's elements of a
// digit begin.  Threads whose index agrees modulo 256 share a word, each adds up kLocalRows warps.  Returns,
// for word threadIdx.x % 256, the block's count and first place (two digits each).  Ends with a barrier.
__device__ __forceinline__ uint2 local_places(const LocalShared &s) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = tid & (kLocalWords - 1), part = tid / kLocalWords, parts = (int)blockDim.x / kLocalWords;
    unsigned int *column = s.table + part * (kLocalRows * kLocalWords) + c;
    unsigned int before[kLocalRows], sum = 0u;
#pragma unroll
    for (int r = 0; r < kLocalRows; ++r) {
        const unsigned int v = column[r * kLocalWords];
        before[r] = sum;
        sum += v;
    }
    s.part[part * kLocalWords + c] = sum;
    __syncthreads();
    unsigned int total = 0u, ahead = 0u;
    for (int q = 0; q < parts; ++q) {
        const unsigned int v = s.part[q * kLocalWords + c];
        ahead += q < part ? v : 0u;
        total += v;
    }
    unsigned int incl = total;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
        if (lane >= k) incl += up;
    }
    if (part == 0 && lane == 31) s.warp_sum[warp] = incl;
    __syncthreads();
    const unsigned int sums = lane < kLocalWords / 32 ? s.warp_sum[lane] : 0u;
    const unsigned int all = __reduce_add_sync(0xffffffffu, sums);
    // digits of the lower halves come first
    const unsigned int first = __reduce_add_sync(0xffffffffu, lane < (warp & (kLocalWords / 32 - 1)) ? sums : 0u) + incl - total + (all << 16);
#pragma unroll
    for (int r = 0; r < kLocalRows; ++r) column[r * kLocalWords] = first + ahead + before[r];
    __syncthreads();
    return make_uint2(total, first);
}

// The smallest and the largest of the block's keys (one barrier; low / high may be written again behind the next).
// Clears seen.
template <typename K> __device__ __forceinline__ void local_range(const LocalShared &s, K &low, K &high) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)blockDim.x >> 5;
    auto least = [](K v) {
        if constexpr (sizeof(K) == 8) {
            const unsigned int hi = __reduce_min_sync(0xffffffffu, (unsigned int)(v >> 32));
            const unsigned int lo = __reduce_min_sync(0xffffffffu, (unsigned int)(v >> 32) == hi ? (unsigned int)v : ~0u);
            return (K)hi << 32 | lo;
        } else {
            return (K)__reduce_min_sync(0xffffffffu, (unsigned int)v);
        }
    };
    const K warp_low = least(low), warp_high = (K)~least((K)~high);
    if (threadIdx.x < 2) s.seen[threadIdx.x] = 0u;
    if (lane == 0) {
        s.low[warp] = (unsigned long long)warp_low;
        s.high[warp] = (unsigned long long)warp_high;
    }
    __syncthreads();
    low = least(lane < warps ? (K)s.low[lane] : (K)~(K)0);
    high = (K)~least((K)~(lane < warps ? (K)s.high[lane] : (K)0));
}

// Values of a thread's elements of a block (element own + i * 32) to shared memory, eight under way at a time.
template <typename V>
__device__ __forceinline__ void load_values(V *values, const V *from, int value_seq, int64_t base, int own, int count, int items) {
    constexpr int AHEAD = sizeof(V) <= 8 ? 8 : 4;
#pragma unroll 1
    for (int first = 0; first < items; first += AHEAD) {
        V v[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int at = own + (first + i) * 32;
            if (first + i < items && at < count) {
                if constexpr (sizeof(V) <= 8) v[i] = value_seq != kSeqNone ? sequence_value<V>(value_seq, base + at) : from[base + at];
                else v[i] = from[base + at];
            }
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int at = own + (first + i) * 32;
            if (first + i < items && at < count) values[at] = v[i];
        }
    }
}

// Bytes of shared memory of an element.
constexpr int local_bytes(int key_bytes, int value_bytes) { return 4 + value_bytes + (value_bytes || key_bytes == 8 ? key_bytes : 0); }

// Whether elements of a key / value size travel as places.
template <typename K> __host__ __device__ constexpr bool by_place(bool values) { return values || sizeof(K) == 8; }

// Sorts `count` elements.  By place: keys (in shared memory, transformed) stay, words receive the places
// in order; key is not read.  Else: key[] holds this thread's transformed keys (element warp * 32 * items + i * 32 + lane), words
// receive the keys less `low`.  store(p, key, word) is called for the p-th in order, possibly again.
template <typename K, bool PLACE, int ITEMS> struct LocalSort {
    LocalShared s;
    unsigned int *words;
    const K *keys;
    int count, items;
    K low, high;

    __device__ __forceinline__ K key_at(unsigned int word) const { return word_key<K, PLACE>(word, keys, low); }
    static __device__ __forceinline__ unsigned int place_of(unsigned int word) { return b200alg::place_of(word); }
    static __device__ __forceinline__ bool wrong(K key_a, unsigned int a, K key_b, unsigned int b) {
        return words_out_of_order<K, PLACE>(key_a, a, key_b, b);
    }
    // Whether an element came out behind a place that holds none: in a tie of the last digits a warp's lanes past
    // the last element, served before the others, would push it out of what emit looks at.  (Not taking part would
    // be a test per element and pass: 9000 keys 18.5 against 16.5 us.)
    __device__ __forceinline__ bool strays() const {
        bool any = false;
        for (int p = count + (int)threadIdx.x; p < items * (int)blockDim.x; p += (int)blockDim.x)
            any |= is_stray<PLACE>(words[p], count);
        if (any) atomicAdd(s.found, blockDim.x + 1u);  // more than settle takes
        return any;
    }

    // counted(c): c.x and c.y are the block's count and first place of digits threadIdx.x % 256 (lower half) and
    // 256 + threadIdx.x % 256 (upper half).
    template <typename Digit, typename Next, typename Counted>
    __device__ __forceinline__ void pass(unsigned int (&w)[ITEMS], Digit digit, Next next, Counted counted) const {
        unsigned int *mine = s.table + (threadIdx.x >> 5) * kLocalWords;
        unsigned int rank[(ITEMS + 1) / 2];  // two to a word
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            const unsigned int r = local_rank(mine, digit(w[i]));
            if (i & 1) rank[i / 2] |= r << 16; else rank[i / 2] = r;
        }
        __syncthreads();
        counted(local_places(s));
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            words[(i & 1 ? rank[i / 2] >> 16 : rank[i / 2] & 0xFFFFu) + local_place(mine, digit(w[i]))] = next(w[i], i);
        }
        __syncwarp();
        local_clear(s);
        __syncthreads();
    }

    // What is rarely needed stays out of line and takes copies: the address of this object, or of what `store`
    // holds, in the hands of a function would keep them all in memory (pairs of 5000: 28600 cycles instead of 18000).

    // Puts the words in order that the passes did not (those past the last element included).
    static __device__ __noinline__ void repair(LocalSort me) {
        put_words_in_order<K, PLACE>(me.words, me.keys, me.low, me.count, me.items * (int)blockDim.x, (int)threadIdx.x, (int)blockDim.x,
                                     [](bool moved) { return __syncthreads_or(moved) != 0; });
    }

    // The pairs that emit found (s.part, *s.found of them) lie in groups that agree in all bits but the lowest `below`:
    // a thread per pair puts its group in order and stores it again.  True: too many pairs, too large a group, or a
    // pair that differs above.
    template <typename Store> static __device__ __noinline__ bool settle(LocalSort me, int below, Store store) {
        constexpr int MOST = 16;
        unsigned int *const words = me.words;
        auto upper = [&](unsigned int word) {
            if constexpr (PLACE) return (K)((K)(me.key_at(word) - me.low) >> below);
            else return word >> below;
        };
        const unsigned int found = *me.s.found;
        bool unsettled = found > blockDim.x, mine = false;
        int first = 0, end = 0;
        if (threadIdx.x < found && !unsettled) {
            const int p = (int)me.s.part[threadIdx.x];
            const auto group = upper(words[p]);
            unsettled = upper(words[p + 1]) != group;
            // the group's first pair of this kind takes care of it
            mine = !unsettled;
            for (first = p; mine && first > 0 && upper(words[first - 1]) == group; --first) {
                mine = !wrong(me.key_at(words[first - 1]), words[first - 1], me.key_at(words[first]), words[first]);
                unsettled |= p - first == MOST;
                mine &= !unsettled;
            }
            end = p + 2;
            while (mine && end < me.count && end - first < MOST && upper(words[end]) == group) ++end;
            unsettled |= mine && end - first >= MOST;
        }
        if (__syncthreads_or(unsettled)) return true;
        if (mine) {
            for (int i = first + 1; i < end; ++i) {
                const unsigned int w = words[i];
                const K k = me.key_at(w);
                int j = i;
                for (; j > first && wrong(me.key_at(words[j - 1]), words[j - 1], k, w); --j) words[j] = words[j - 1];
                words[j] = w;
            }
            for (int i = first; i < end; ++i) store(i, me.key_at(words[i]), words[i]);
        }
        return false;
    }

    // Calls store(p, key, word) for the sorted order; whether neighbours are out of order (and which: s.part).
    template <typename Store> __device__ __forceinline__ bool emit(Store store) const {
        const int threads = (int)blockDim.x, lane = threadIdx.x & 31;
        bool bad = false;
#pragma unroll 1
        for (int first = 0; first < items; first += 4) {
            unsigned int word[4];
            K key[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int p = (int)threadIdx.x + (first + i) * threads;
                word[i] = words[p < count ? p : 0];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) key[i] = key_at(word[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int p = (int)threadIdx.x + (first + i) * threads;
                unsigned int next = __shfl_down_sync(0xffffffffu, word[i], 1);
                K next_key;
                if constexpr (sizeof(K) == 8) next_key = __shfl_down_sync(0xffffffffu, key[i], 1);
                else next_key = (K)__shfl_down_sync(0xffffffffu, (unsigned int)key[i], 1);
                if (p + 1 < count) {
                    if (lane == 31) {
                        next = words[p + 1];
                        next_key = key_at(next);
                    }
                    if (wrong(key[i], word[i], next_key, next)) {
                        const unsigned int at = atomicAdd(s.found, 1u);
                        if (at < (unsigned int)threads) s.part[at] = (unsigned int)p;
                        bad = true;
                    }
                }
                if (p < count) store(p, key[i], word[i]);
            }
        }
        return bad;
    }

    // The lowest bit to sort by, of more bits than the digits cover; `below` are left over.  One key of every thread is
    // looked at.  Where two neighbours of a few agree in all bits but the lowest `below` and differ in those, many of the
    // block's do; and what none has below its lowest bit hardly any has (else the writer finds it).
    __device__ __forceinline__ int lowest_bit(const K *key, int own, int below) const {
        const int lane = threadIdx.x & 31;
        K mine = 0;
        if (own < count) mine = PLACE ? (K)(keys[own] - low) : (K)(key[0] - low);
        bool tie = false;
#pragma unroll
        for (int k = 1; k <= 8; k *= 2) {
            K other;
            if constexpr (sizeof(K) == 8) other = __shfl_down_sync(0xffffffffu, mine, k);
            else other = (K)__shfl_down_sync(0xffffffffu, (unsigned int)mine, k);
            tie |= lane + k < 32 && own + k < count && other != mine && other >> below == mine >> below;
        }
        const unsigned int lower = __reduce_or_sync(0xffffffffu, (unsigned int)mine);
        if (lane == 0) atomicOr(s.seen, lower);
        if constexpr (sizeof(K) == 8) {
            const unsigned int upper = __reduce_or_sync(0xffffffffu, (unsigned int)(mine >> 32));
            if (lane == 0) atomicOr(s.seen + 1, upper);
        }
        tie = __syncthreads_or(tie) != 0;
        const unsigned int first = s.seen[0];
        int lowest = __ffs((int)first) - 1;
        if constexpr (sizeof(K) == 8) {
            if (first == 0u) lowest = __ffs((int)s.seen[1]) - 1 + (s.seen[1] ? 32 : 0);
        }
        return lowest > below || (tie && lowest >= 0) ? lowest : below;
    }

    // The tables are clear, keys (by place) are in shared memory behind a barrier, low and high are known.
    template <typename Store> __device__ __forceinline__ void run(const K *key, Store store) const {
        const int own = (int)(threadIdx.x >> 5) * 32 * items + (int)(threadIdx.x & 31);
        const K range = (K)(high - low);
        const int bits = sizeof(K) == 8 ? 64 - __clzll((long long)range) : 32 - __clz((int)(unsigned int)range);
        if (threadIdx.x == 0) *s.found = 0u;
        int from = 0;  // the lowest bit that is sorted by
        if (bits > kLocalPrefixBits) from = lowest_bit(key, own, bits - kLocalPrefixBits);
        unsigned int w[ITEMS];
        bool fresh = true;  // words hold nothing yet
        for (;;) {
            // By place, bits go in turns of up to 27; in the first pass of a turn the keys are looked up, later ones
            // find their digits above the place.  Elements past the last one sort behind all others: largest digits,
            // and last in every tie.
            if (bits == 0) {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    if (i >= items) break;
                    words[own + i * 32] = PLACE ? (unsigned int)(own + i * 32) : own + i * 32 < count ? 0u : ~0u;
                }
                __syncthreads();
            }
            if (PLACE) fresh = true;
            for (int turn = from; turn < bits;) {
                const int left = bits - turn, length = !PLACE ? left : left % kLocalPrefixBits ? left % kLocalPrefixBits : kLocalPrefixBits;
                const int passes = (length + kLocalDigitBits - 1) / kLocalDigitBits, width = (length + passes - 1) / passes;
                const unsigned int mask = (1u << width) - 1u;
                for (int p = 0; p < passes; ++p) {
                    const bool look_up = PLACE && p == 0;
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i) {
                        if (i >= items) break;
                        const int at = own + i * 32;
                        if constexpr (PLACE) w[i] = fresh ? (unsigned int)at : words[at];
                        else w[i] = !fresh ? words[at] : at < count ? (unsigned int)(K)(key[i] - low) : ~0u;
                    }
                    if (look_up) {
                        unsigned int place[(ITEMS + 1) / 2];  // two to a word
#pragma unroll
                        for (int i = 0; i < ITEMS; ++i) {
                            if (i >= items) break;
                            const unsigned int at = place_of(w[i]);
                            if (i & 1) place[i / 2] |= at << 16; else place[i / 2] = at;
                            w[i] = (at < (unsigned int)count ? (unsigned int)((K)(keys[at] - low) >> turn) : ~0u) & (unsigned int)((1ull << length) - 1ull);
                        }
                        pass(w, [=](unsigned int v) { return v & mask; },
                             [&](unsigned int v, int i) { return v >> width << kPlaceBits | (i & 1 ? place[i / 2] >> 16 : place[i / 2] & 0xFFFFu); }, [](uint2) {});
                    } else {
                        const int shift = PLACE ? kPlaceBits + (p - 1) * width : turn + p * width;
                        pass(w, [=](unsigned int v) { return v >> shift & mask; }, [](unsigned int v, int) { return v; }, [](uint2) {});
                    }
                    fresh = false;
                }
                turn += length;
            }
            const bool stray = strays();
            if (!__syncthreads_or(emit(store) || stray)) return;
            if (from == 0) break;
            if (!settle(*this, from, store)) return;
            from = 0;
        }
        repair(*this);
        emit(store);
    }
};

}  // namespace b200alg
