// Radix sort of views of some ten thousand to one and a half million elements: one partition into buckets that a
// block can sort alone (local_sort.cuh), in one launch; where keys differ in a few bytes only, a partition by each
// of these instead.
//
// What such a sort costs with a pass per key byte is the exchange between the blocks that ends each of them
// (10^6 keys: 12 us a pass, 3 of them for the keys' trips through shared memory).  Here keys move between
// blocks once:
//
//   sample     every block looks at kSampled keys of its share, orders them and publishes every other; every
//              block ranks its published ones among all, and those of rank j * samples / buckets are the
//              splitters.  In the order (key, position), so that equal keys are spread like all others and any
//              distribution gives even buckets.
//   partition  a block's elements go to their buckets' places in shared memory (bucket by a search in the
//              splitters, place by local_sort.cuh's counting), the blocks add up one another's counts, and the
//              elements go to the buckets in the alternate buffer, in order.
//   sort       every block sorts its buckets and stores them in the output view.
//
// The blocks meet four times, which is 5 us; 10^6 uint64 keys spend 9 us on the splitters, 13 on the partition and
// 14 on the sort (512 threads a block; 1024 were slower below 10^6 elements, 35 against 29 us for 13000: code that
// runs once is fetched once per launch, and more warps do not fetch it faster).  A bucket that came out larger than
// a block holds (the sample misled: keys made for it, no distribution) is known to all blocks before anything has
// been written; then they sort by digits of eight bits instead, with the same partition.
//
// Labels, small counters and whole numbers kept as floating-point differ in so few bytes that a partition by each
// of them, lowest first, takes less time than the splitters and the sort of the buckets do, up to kFewDigits of them
// (400000 uint32 keys with 4-byte values, us with the copies that bring them: 24.1, 33.4 and 42.6 by one, two and three
// bytes, 50.7 by four; 45.4 by buckets whatever the keys are).  Whether they are such keys every block guesses from the
// same kLooks keys of the view, so that all guess alike; when the blocks first meet they learn in which bytes keys
// differ and, where the guess was wrong, start again before anything has been written.
//
// The blocks are a cooperative grid, or up to kClusterSort elements one cluster, whose blocks meet sooner and which
// starts while the kernel before it drains: 20000 doubles 24.9 instead of 32.0 us, of two bytes 16.7 instead of 21.1 (and 40000 28.9 instead of 31.4, 50000
// 31.0 and 31.9, with 4-byte values 36.2 and 35.1).
#include "local_sort.cuh"
#include "../../include/b200alg_testing.h"

#include <cooperative_groups.h>

namespace b200alg {

namespace cg = cooperative_groups;

constexpr int kSampleThreads = 512, kSampleItems = kLocalMost / kSampleThreads;
constexpr int kSampled = 128, kPublished = 64;  // keys of a block
constexpr int kLooks = 64;                      // keys of the view, by one warp (384 by twelve: 0.5 us more)
constexpr int kFewDigits = 3;
constexpr int kMaxBuckets = 480;                // the last digit (511) is what fills a share up
constexpr int kPartitionDigits = 1 << kLocalDigitBits;
constexpr int kSampleSmem = 227 * 1024;
constexpr int kCtlDigitMoves = B200ALG_TESTING_SORT_MOVES_WORD - 1;  // (behind wait_limit_hit)

// The small arrays of a block.
template <typename K> struct SampleShared {
    K tree[kPartitionDigits];                  // splitters as a search tree (node 1 the root); before: the sample in order
    K splitter[kPartitionDigits];              // in order; before: the sample
    unsigned int index[kPartitionDigits];      // of the splitters; before: of the sample
    unsigned int first[kPartitionDigits];      // a bucket's first place in the block; then its global index less that
    unsigned int count[kPartitionDigits];      // and its elements of the block
    unsigned int total[kPartitionDigits];      // its elements of all blocks
    unsigned int before[kPartitionDigits];     // of those in front of this one
    unsigned int start[kPartitionDigits + 8];  // where a bucket starts
    unsigned int warp_sum[kSampleThreads / 32];
};
template <typename K> __host__ __device__ constexpr int sample_items(int value_bytes) {
    const int fit = (kSampleSmem - local_fixed_bytes(kSampleThreads) - (int)sizeof(SampleShared<K>)) / (kSampleThreads * (4 + value_bytes + (int)sizeof(K)));
    return fit < kSampleItems ? fit : kSampleItems;
}

template <typename K, typename V> struct SampleSort {
    SortBuffers<K, V> io;
    KeyXform<K> xf;
    TempHeader *hdr;
    K *sample_keys;              // [blocks][kPublished]
    unsigned int *sample_index;
    K *splitter_keys;            // [buckets - 1]; before: the bits in which a block's keys differ from the view's first
    unsigned int *splitter_index;
    unsigned short *counts;      // [blocks][padded buckets]
    int buckets, value_seq;
    int in_cluster;              // the grid is one cluster
};

// An element, asynchronously, from global to shared memory.
template <typename T> __device__ __forceinline__ void copy_element(T *to, const T *from) {
    if constexpr (sizeof(T) >= 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(to)), "l"(from), "n"((int)sizeof(T)) : "memory");
    else
        *to = *from;
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// What a block works with.
template <typename K, typename V> struct SampleBlock {
    static constexpr int VB = ValueBytes<V>::value;
    static constexpr int ITEMS = sample_items<K>(VB), MOST = ITEMS * kSampleThreads;
    LocalShared shared;
    unsigned int *words;
    V *values;
    K *keys;
    unsigned int n, lo;  // elements of the view; this block's begin at lo

    // Elements [base, base + count) on their way to keys and values (this thread's places, as in LocalSort).
    __device__ __forceinline__ void fetch(const K *from, int64_t stride, const V *vfrom, int value_seq, unsigned int base, int count, int items) const {
        const int own = (int)(threadIdx.x >> 5) * 32 * items + (int)(threadIdx.x & 31);
#pragma unroll 4
        for (int i = 0; i < items; ++i) {
            const int at = own + i * 32;
            if (at < count) {
                copy_element(keys + at, from + (int64_t)(base + at) * stride);
                if constexpr (VB != 0 && VB <= 8) {
                    if (value_seq != kSeqNone) values[at] = sequence_value<V>(value_seq, (int64_t)base + at);
                    else copy_element(values + at, vfrom + base + at);
                } else if constexpr (VB != 0) {
                    copy_element(values + at, vfrom + base + at);
                }
            }
        }
    }

};

// The bits that some lane of the warp has.
template <typename K> __device__ __forceinline__ K warp_or(K v) {
    if constexpr (sizeof(K) == 8)
        return (K)__reduce_or_sync(0xffffffffu, (unsigned int)(v >> 32)) << 32 | __reduce_or_sync(0xffffffffu, (unsigned int)v);
    else
        return (K)__reduce_or_sync(0xffffffffu, (unsigned int)v);
}
// How many bytes of a key hold one of the bits.
template <typename K> __device__ __forceinline__ int bytes_with(K bits) {
    constexpr K LOW = (K)0x7F7F7F7F7F7F7F7Full;
    const K top = (K)(((bits & LOW) + LOW) | bits) & (K)~LOW;
    if constexpr (sizeof(K) == 8) return __popcll(top);
    else return __popc(top);
}
template <typename K> __device__ __forceinline__ int lowest_byte(K bits) {  // where it begins (no bits: 0)
    if constexpr (sizeof(K) == 8) return bits ? (__ffsll((long long)bits) - 1) & ~7 : 0;
    else return bits ? (__ffs((int)bits) - 1) & ~7 : 0;
}

// One partition: where its elements come from and go to, and what their buckets are.
struct Partition {
    bool moved;   // elements come from the alternate buffer, transformed; else from the input, as the caller has them
    bool last;    // and go to the output; else to the alternate buffer, transformed
    bool raw;     // keys of the share are as the caller has them
    int shift;    // of the digit (eight bits), or
    int height;   // of the tree of splitters (shift < 0)
    int buckets;
};

template <typename K, typename V>
__global__ void __launch_bounds__(kSampleThreads, 1)
sample_sort_kernel(SampleSort<K, V> a) {
    using B = SampleBlock<K, V>;
    constexpr int VB = B::VB;
    static_assert(by_place<K>(VB != 0), "keys stay in shared memory and are looked up there");
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blocks = (int)gridDim.x;
    SampleShared<K> *const m = reinterpret_cast<SampleShared<K> *>(smem + local_fixed_bytes(kSampleThreads));
    auto meet = [&]() {
        if (a.in_cluster) cg::this_cluster().sync();
        else cg::this_grid().sync();
    };
    B b;
    b.shared = local_shared(smem);
    local_clear(b.shared);
    grid_dependency_wait();
    b.n = (unsigned int)effective_n(a.io);
    const unsigned int share = (b.n + blocks - 1) / blocks;
    b.lo = blockIdx.x * share < b.n ? blockIdx.x * share : b.n;
    const int len = (int)(b.n - b.lo < share ? b.n - b.lo : share);  // of this block
    const int items = ((int)share + kSampleThreads - 1) / kSampleThreads, own = warp * 32 * items + lane;
    b.words = reinterpret_cast<unsigned int *>(m + 1);
    b.values = reinterpret_cast<V *>(b.words + B::MOST);
    b.keys = reinterpret_cast<K *>(reinterpret_cast<unsigned char *>(b.values) + (size_t)B::MOST * VB);

    Partition part{false, false, true, -1, 0, a.buckets};
    auto fetch_share = [&]() {
        if (part.moved) b.fetch(a.io.alt, 1, a.io.valt, kSeqNone, b.lo, len, items);
        else b.fetch(a.io.in, a.io.stride, a.io.vin, a.value_seq, b.lo, len, items);
    };
    if (blockIdx.x == 0 && tid == 0) a.hdr->wait_limit_hit = a.hdr->reserved[kCtlDigitMoves] = 0u;

    // ---- which way, and the block's sample ----
    K own_key = (K)~(K)0;
    unsigned int own_index = b.n;
    if (tid < kSampled) {
        if (len > 0) {
            const unsigned int stratum = len / kSampled;
            const unsigned int shift = stratum ? ((blockIdx.x * kSampled + tid) * 2654435761u >> 8) % stratum : 0u;
            own_index = b.lo + (unsigned int)((unsigned long long)tid * len / kSampled) + shift;
            own_key = a.io.in[(int64_t)own_index * a.io.stride];
        }
    }
    const bool looks = warp == kSampled / 32;  // at keys of the whole view: the same in every block
    K look[kLooks / 32];
    if (looks) {
#pragma unroll
        for (int i = 0; i < kLooks / 32; ++i) {
            const unsigned int j = i * 32 + lane;
            const unsigned int at = (unsigned int)((unsigned long long)j * b.n / kLooks) + __umulhi(b.n / kLooks, j * 2654435761u);
            if (at < b.n) look[i] = a.io.in[(int64_t)at * a.io.stride];
            else look[i] = 0;
        }
    }
    fetch_share();  // comes while it is found out where the elements go
    if (own_index < b.n) own_key = a.xf(own_key);
    if (tid < kSampled) {
        m->splitter[tid] = own_key;
        m->count[tid] = 0u;
    }
    if (looks) {
        K bits = 0, first = 0;
#pragma unroll
        for (int i = 0; i < kLooks / 32; ++i) {
            const K k = a.xf(look[i]);
            if (i == 0) first = __shfl_sync(0xffffffffu, k, 0);
            bits |= k ^ first;
        }
        bits = warp_or(bits);
        if (lane == 0) {
            b.shared.low[0] = bits;
            b.shared.low[1] = first;
            b.shared.low[2] = bytes_with(bits) <= kFewDigits;
        }
    }
    __syncthreads();
    {   // a few threads per key count the smaller ones of a part of the sample each
        constexpr int PART = kSampled * kSampled / kSampleThreads;
        const int j = tid % kSampled, from = tid / kSampled * PART;
        const K mine = m->splitter[j];
        unsigned int rank = 0u;
#pragma unroll 8
        for (int i = from; i < from + PART; ++i) {
            const K other = m->splitter[i];
            rank += other < mine || (other == mine && i < j);
        }
        atomicAdd(&m->count[j], rank);
    }
    __syncthreads();
    const unsigned int own_rank = tid < kSampled ? m->count[tid] : 0u;
    // The bits in which keys differ from the first one, as far as is known: where a few bytes hold them all, keys go by
    // digits.
    K differ = (K)b.shared.low[0];
    const K first_key = (K)b.shared.low[1];
    bool looking = b.shared.low[2] != 0;  // what differs is a guess yet
    // what the warps have put there, behind a barrier
    auto known = [&]() { return warp_or(lane < kSampleThreads / 32 ? (K)b.shared.high[lane] : (K)0); };
    auto by_digit = [&](int shift) {
        part.shift = shift;
        part.last = (K)(differ >> shift) >> 8 == 0;
        part.buckets = kRadix;
    };
    if (looking) by_digit(lowest_byte(differ));

    auto find_splitters = [&]() {
        static_assert(kSampleThreads == kPartitionDigits, "a thread clears a total");
        m->total[tid] = 0u;
        constexpr int EVERY = kSampled / kPublished;
        static_assert(EVERY == 2, "of a pair, neighbouring blocks publish one the lower and one the upper: the ranks stay unbiased");
        if (tid < kSampled && own_rank % EVERY == (blockIdx.x & 1)) {
            const int e = (int)(own_rank / EVERY);
            m->tree[e] = own_key;
            m->index[e] = own_index;
            a.sample_keys[blockIdx.x * kPublished + e] = own_key;
            a.sample_index[blockIdx.x * kPublished + e] = own_index;
        }
        meet();
        const unsigned int samples = (unsigned int)blocks * kPublished;
        // how many of this block's published keys are in front of each of the others'
        constexpr int TOGETHER = 10;
#pragma unroll 1
        for (unsigned int first = tid; first < samples; first += TOGETHER * kSampleThreads) {
            K key[TOGETHER];  // those below key[i] are in front: the next larger key for blocks behind this one
            int pos[TOGETHER];
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) {
                const unsigned int q = first + i * kSampleThreads;
                key[i] = q < samples ? __ldcg(a.sample_keys + q) : (K)0;
                pos[i] = 0;
            }
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) {
                if ((first + i * kSampleThreads) / kPublished <= blockIdx.x) continue;
                if (key[i] == (K)~(K)0) pos[i] = kPublished;
                else ++key[i];
            }
#pragma unroll 1
            for (int step = kPublished / 2; step > 0; step >>= 1)
#pragma unroll
                for (int i = 0; i < TOGETHER; ++i)
                    if (m->tree[(pos[i] + step - 1) & (2 * kPublished - 1)] < key[i]) pos[i] += step;
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) {
                const unsigned int q = first + i * kSampleThreads;
                if (pos[i] < kPublished && m->tree[pos[i]] < key[i]) ++pos[i];
                if (q < samples && q / kPublished != blockIdx.x) atomicAdd(&m->total[pos[i] < kPublished ? pos[i] : kPublished], 1u);
            }
        }
        __syncthreads();
        if (warp == 0) {
            const unsigned int one = m->total[2 * lane], two = m->total[2 * lane + 1];
            unsigned int incl = one + two;
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += up;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = 2 * lane + h;
                const unsigned int rank = e + (h ? incl : incl - two);
                const unsigned int j = (rank * a.buckets + samples - 1) / samples;
                if (j >= 1 && j < (unsigned int)a.buckets && j * samples / a.buckets == rank) {
                    a.splitter_keys[j - 1] = m->tree[e];
                    a.splitter_index[j - 1] = m->index[e];
                }
            }
        }
        meet();
        while (1 << part.height < a.buckets) ++part.height;
        // (all loads ahead of the stores)
        const bool node = tid > 0 && tid < 1 << part.height, splits = tid < a.buckets - 1;
        const int level = 31 - __clz(tid | 1), at = ((2 * (tid - (1 << level)) + 1) << (part.height - 1 - level)) - 1;
        K node_key = (K)~(K)0, key = 0;
        unsigned int index = 0u;
        if (node && at < a.buckets - 1) node_key = __ldcg(a.splitter_keys + at);
        if (splits) {
            key = __ldcg(a.splitter_keys + tid);
            index = __ldcg(a.splitter_index + tid);
        }
        if (node) m->tree[tid] = node_key;
        if (splits) {
            m->splitter[tid] = key;
            m->index[tid] = index;
        }
    };
    if (!looking) find_splitters();
    const bool bucket_thread = tid < kPartitionDigits;
    int moves = 0;
    for (;;) {  // (once, where keys go by buckets and none is too large)
        // ---- partition ----
        const int splitters = a.buckets - 1;
        const LocalSort<K, true, kSampleItems> local{b.shared, b.words, b.keys, 0, items, (K)0, (K)0};
        const int padded = (part.buckets + 7) / 8 * 8;
        if (bucket_thread) {
            m->total[tid] = 0u;
            m->before[tid] = 0u;
        }
        __syncthreads();
        copies_wait();
        // the share's words: bucket and place.  (Fillers go by a digit of their own; what is computed for them, and
        // for elements of other threads that are read in their place, is not used.)
        constexpr int AHEAD = 6;
        K other = 0;  // bits that the first key of the view does not have
#pragma unroll 1
        for (int first = 0; first < items; first += AHEAD) {
            const int mine = own + first * 32;
            K bits[AHEAD];
            unsigned int bucket[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int at = mine + i * 32;
                bits[i] = b.keys[at < len ? at : 0];
                if (part.raw) bits[i] = a.xf(bits[i]);
                bucket[i] = 1u;
            }
            if (part.shift >= 0) {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    bucket[i] = (unsigned int)(bits[i] >> part.shift) & (kRadix - 1u);
                    if (first + i < items && mine + i * 32 < len) other |= bits[i] ^ first_key;
                }
            } else {
#pragma unroll 1
                for (int level = 0; level < part.height; ++level)
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i) bucket[i] = 2 * bucket[i] + (m->tree[bucket[i]] < bits[i]);
                bool tie = false;
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    bucket[i] -= 1u << part.height;  // splitters below the key
                    tie |= bucket[i] < (unsigned int)splitters && m->splitter[bucket[i]] == bits[i];
                }
                if (tie) {  // equal keys go by position
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i) {
                        const unsigned int index = b.lo + mine + i * 32;
                        unsigned int low = bucket[i], high = (unsigned int)splitters;
                        while (low < high) {
                            const unsigned int mid = (low + high) / 2;
                            if (m->splitter[mid] == bits[i] && m->index[mid] <= index) low = mid + 1;
                            else high = mid;
                        }
                        bucket[i] = low;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int at = mine + i * 32;
                if (first + i >= items) break;
                if (at < len) b.keys[at] = bits[i];
                b.words[at] = (at < len ? bucket[i] : kPartitionDigits - 1u) << kPlaceBits | (unsigned int)at;
            }
        }
        auto collect = [&]() {  // for known()
            other = warp_or(other);
            if (lane == 0) b.shared.high[warp] = other;
        };
        if (looking) collect();
        {   // in bucket order; first and count of the buckets
            unsigned int w[kSampleItems];
#pragma unroll
            for (int i = 0; i < kSampleItems; ++i) {
                if (i >= items) break;
                w[i] = b.words[own + i * 32];
            }
            local.pass(w, [](unsigned int v) { return v >> kPlaceBits; }, [](unsigned int v, int) { return v; },
                       [&](uint2 c) {
                           if (tid < kLocalWords) {
                               m->count[tid] = c.x & 0xFFFFu;
                               m->first[tid] = c.y & 0xFFFFu;
                               m->count[kLocalWords + tid] = c.x >> 16;
                               m->first[kLocalWords + tid] = c.y >> 16;
                           }
                       });
        }
        // the buckets' sizes, and what the blocks ahead have of them
        if (tid < padded) a.counts[(size_t)blockIdx.x * padded + tid] = (unsigned short)(tid < part.buckets ? m->count[tid] : 0u);
        if (looking && warp == 0) {
            other = known();
            if (lane == 0) a.splitter_keys[blockIdx.x] = other;
        }
        meet();
        if (looking) {
            other = tid < blocks ? __ldcg(a.splitter_keys + tid) : (K)0;
            collect();
        }
        // eight buckets of a row per thread, ROWS rows under way (four: 0.3 us more; ten: 1)
        constexpr int ROWS = 6;
        const int chunks = padded / 8, groups = kSampleThreads / chunks, chunk = tid % chunks, group = tid / chunks;
        unsigned int all_of[8] = {0, 0, 0, 0, 0, 0, 0, 0}, ahead[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (group < groups) {
#pragma unroll 1
            for (int r = group; r < blocks; r += ROWS * groups) {
                uint4 c[ROWS];
#pragma unroll
                for (int j = 0; j < ROWS; ++j)
                    c[j] = r + j * groups < blocks ? __ldcg(reinterpret_cast<const uint4 *>(a.counts + (size_t)(r + j * groups) * padded) + chunk)
                                                   : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int j = 0; j < ROWS; ++j) {
                    const unsigned int v[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
                    const bool mine = r + j * groups < (int)blockIdx.x;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        all_of[2 * q] += v[q] & 0xFFFFu;
                        all_of[2 * q + 1] += v[q] >> 16;
                        ahead[2 * q] += mine ? v[q] & 0xFFFFu : 0u;
                        ahead[2 * q + 1] += mine ? v[q] >> 16 : 0u;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {  // (neighbouring lanes, neighbouring banks)
                atomicAdd(&m->total[q * (kPartitionDigits / 8) + chunk], all_of[q]);
                atomicAdd(&m->before[q * (kPartitionDigits / 8) + chunk], ahead[q]);
            }
        }
        __syncthreads();
        if (looking) {
            // Nothing has been stored yet: where the guess was wrong, once more (the share is transformed by now).  But the
            // first digit has been paid for, so that two more may follow than if the keys were known to need them.
            looking = false;
            differ = known();
            const bool right = lowest_byte(differ) == part.shift, few = bytes_with(differ) <= kFewDigits + (right ? 2 : 0);
            if (!right || !few) part = Partition{false, false, false, -1, 0, a.buckets};
            if (few) by_digit(lowest_byte(differ));
            else find_splitters();
            if (!right || !few) continue;
        }
        const int from = tid % 8 * (kPartitionDigits / 8) + tid / 8;
        const unsigned int size = bucket_thread ? m->total[from] : 0u;  // of bucket tid (nothing is in those past the last)
        unsigned int incl = size;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
            if (lane >= k) incl += up;
        }
        if (lane == 31) m->warp_sum[warp] = incl;
        const bool too_large = __syncthreads_or(size > (unsigned int)B::MOST) != 0 && part.shift < 0;
        const unsigned int start = __reduce_add_sync(0xffffffffu, lane < warp ? m->warp_sum[lane] : 0u) + incl - size;
        if (bucket_thread) {
            m->start[tid] = start;
            m->first[tid] = start + m->before[from] - m->first[tid];
        }
        if (tid == 0) m->start[kPartitionDigits] = b.n;
        __syncthreads();
        if (!too_large) {
            // (where keys alone go to buckets of the sample, any order will do: the buckets are sorted)
            const bool in_order = VB != 0 || part.shift >= 0;
            auto store = [&](auto put) {
                bool bad = false;
#pragma unroll 4
                for (int p = tid; p < len; p += kSampleThreads) {
                    const unsigned int word = b.words[p], place = word & ((1u << kPlaceBits) - 1u);
                    if (in_order) bad |= p + 1 < len && b.words[p + 1] < word;
                    put(m->first[word >> kPlaceBits] + p, place, b.keys[place]);
                }
                return bad;
            };
            for (;;) {
                const bool bad = part.last ? store([&](unsigned int at, unsigned int place, K bits) {
                    a.io.out[(int64_t)at * a.io.stride] = a.xf.raw(bits);
                    if constexpr (VB != 0) a.io.vout[at] = b.values[place];
                })
                                           : store([&](unsigned int at, unsigned int place, K bits) {
                    a.io.alt[at] = bits;
                    if constexpr (VB != 0) a.io.valt[at] = b.values[place];
                });
                // Lanes that met in one counter were served in another order than theirs: what is in which bucket is
                // right, the order inside is put right and the elements are stored again.
                if (!__syncthreads_or(bad)) break;
                using Words = LocalSort<unsigned int, false, kSampleItems>;
                Words::repair(Words{b.shared, b.words, nullptr, len, items, 0u, 0u});
            }
        }
        if (part.shift >= 0) ++moves;
        if (part.last) {
            if (blockIdx.x == 0 && tid == 0) a.hdr->reserved[kCtlDigitMoves] = (unsigned int)moves;
            return;
        }
        meet();  // the elements have been stored, and all blocks have read the counts
        if (!too_large && part.shift < 0) break;
        // The next digit in which keys differ, lowest first; all of them where a sample misled.  (A block holds its share
        // before it meets the others, so that a pass may store where it has read.)
        if (too_large) {
            differ = (K)~(K)0;
            part.raw = true;
            by_digit(0);
        } else {
            part.moved = true;
            part.raw = false;
            const int done = part.shift + 8;
            by_digit(done + lowest_byte((K)(differ >> done)));
        }
        fetch_share();
    }

    // ---- sort ----
    K *const out = a.io.out;
    V *const vout = a.io.vout;
    const V *const values = b.values;
    const int64_t stride = a.io.stride;
    const KeyXform<K> xf = a.xf;
    for (int bucket = (int)blockIdx.x; bucket < a.buckets; bucket += blocks) {
        const unsigned int start = m->start[bucket];
        const int count = (int)(m->start[bucket + 1] - start), items = (count + kSampleThreads - 1) / kSampleThreads;
        const int own = warp * 32 * items + lane;
        K low = (K)~(K)0, high = 0;
        b.fetch(a.io.alt, 1, a.io.valt, kSeqNone, start, count, items);
        copies_wait();
#pragma unroll
        for (int i = 0; i < kSampleItems; ++i) {
            if (i >= items) break;
            if (own + i * 32 < count) {
                const K k = b.keys[own + i * 32];
                low = k < low ? k : low;
                high = k > high ? k : high;
            }
        }
        local_range(b.shared, low, high);
        const LocalSort<K, true, kSampleItems> sort{b.shared, b.words, b.keys, count, items, low, high};
        sort.run(nullptr, [=](int p, K k, unsigned int word) {
            out[(int64_t)(start + p) * stride] = xf.raw(k);
            if constexpr (VB != 0) vout[start + p] = values[place_of(word)];
        });
        __syncthreads();
    }
}

// ---- host side ---------------------------------------------------------------------------
// Which sorts: 8-byte keys, and 4-byte keys with values, as long as a share fits a block with some room to spare; a
// bucket is meant to be 60 % of what fits (the largest is 1.2 to 1.4 times that).  4-byte keys alone gain nothing
// (300000: 37.3 against 38.0 us, 10^6: 62.9 against 63.5).  This way (the first figure) and a pass per key byte with
// the bytes skipped in which keys agree, us with the copy that brings the data, by key bytes / value bytes:
//              20000        50000        100000       200000       400000       800000       1100000      1500000
//   8 / 0    25.0  44.4   30.1  53.8   33.0  65.9   38.8  68.6   43.2  90.2   53.4 102.6   67.7 116.3   76.4 129.9
//            22.9  21.7   27.8  23.8   28.9  28.9   33.6  31.4   37.1  39.1   43.2  57.5   47.8  65.2   54.1  70.8  below 2^20
//            12.5  12.0   14.5  11.5   15.5  14.5   18.0  16.1   18.9  18.6   20.8  40.7   22.7  43.6   24.8  46.8  below 2^8
//   8 / 4    27.9  55.4   33.9  65.7   36.0  79.4   43.1  90.8   51.0 110.9   61.7 126.5   77.8 138.3   does not fit
//            25.9  26.6   32.0  30.2   33.8  36.1   38.3  42.4   45.4  51.4   52.6  74.2   58.7  79.3                below 2^20
//            13.7  16.4   17.7  15.7   18.7  19.4   22.7  24.0   26.8  28.1   28.9  51.7   31.0  53.5                below 2^8
//   4 / 4    25.6  30.5   32.0  36.1   33.7  41.5   38.1  47.3   45.4  59.0   54.3  68.9   67.8  76.4   76.0  80.1
//            24.1  24.5   30.9  29.0   30.9  33.1   35.0  37.6   42.6  49.3   49.4  63.6   53.8  70.5   61.3  73.6  below 2^20
//            13.3  14.4   16.6  15.5   16.6  16.6   20.0  20.5   24.1  26.3   26.9  44.2   28.9  46.7   31.0  48.4  below 2^8
// (The passes' clearing has since come to start early, 3 us less for them.)  Integers go this way from where those
// below 2^20 lost nothing when they went by buckets too (now shorter ones of 8 bytes would gain); floating-point keys
// wherever one block is not faster (alone_most in small_sort.cu; float keys with 4-byte values 12288: 25.3 against 26.2
// by a cluster with a pass per byte, of whole numbers below 2^8 18.6 against 21.5; but with 2-byte values 14000: 26.6
// against 24.5, 19000: 26.6 and 27.1).  Whole numbers
// kept as double below 2^8 differ in three bytes: 20000 of them 22.8 against 23.8 us by passes, 400000 39.2 and 49.0.
// A wrong guess costs 4 to 7 us: 400000 uint64 + 4 bytes below 2^16 but for one key that differs in five bytes 55.6 us
// (by passes 63.9), in six, which then go by buckets, 65.9 (75.4).
// Shares of 1024, 1536, 2048 and 3072 elements: 100000 uint32 pairs 33.3, 32.5, 32.9, 34.8; 30000 30.7, 30.9, 32.8, 34.7.
constexpr int kSampleShare = 1536;
constexpr int kSampleCluster = 16;
constexpr int64_t kClusterSort = 40960;
constexpr int64_t sample_least(int key_bytes, int value_bytes, bool floating) {
    return floating ? (key_bytes == 4 && value_bytes < 4 ? 20000 : 1) : value_bytes ? 100000 : 700000;
}

struct SampleLimits {
    int grid;      // most blocks of a cooperative launch
    bool cluster;  // whether a cluster of kSampleCluster blocks fits
};
// A cooperative launch, or one cluster, which starts while the kernel before it drains.
struct SampleLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2] = {};
    SampleLaunch(cudaStream_t s, int blocks, bool in_cluster) {
        if (in_cluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = blocks;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
        } else {
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(kSampleThreads);
        cfg.dynamicSmemBytes = kSampleSmem;
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = in_cluster ? 2 : 1;
    }
    SampleLaunch(const SampleLaunch &) = delete;
};

template <typename K, typename V>
static int run_sample_sort(cudaStream_t s, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, const SortScratch &scratch, bool *taken) {
    using B = SampleBlock<K, V>;
    constexpr int VB = B::VB;
    *taken = false;
    auto kernel = sample_sort_kernel<K, V>;
    static ContextCache<SampleLimits> cache;
    SampleLimits lim;
    if (!cache.find(&lim)) {
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmem));
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        int per_sm = 0, clusters = 0;
        B200ALG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSampleThreads, kSampleSmem));
        lim.grid = per_sm * sm_count();
        SampleLaunch launch(nullptr, kSampleCluster, true);
        lim.cluster = cudaOccupancyMaxActiveClusters(&clusters, kernel, &launch.cfg) == cudaSuccess && clusters > 0;
        (void)cudaGetLastError();
        cache.store(lim);
    }
    const int64_t n = call.n;
    if (n < sample_least(sizeof(K), VB, xn != xp)) return B200ALG_OK;  // (integers' transforms have one constant)
    const bool in_cluster = lim.cluster && n <= kClusterSort;
    int64_t blocks = in_cluster ? kSampleCluster : ceil_div(n, kSampleShare);
    blocks = blocks < lim.grid ? blocks : lim.grid;
    const int64_t share = ceil_div(n, blocks), buckets = blocks * ceil_div(share * 5, B::MOST * 3);
    if (blocks < 2 || buckets > kMaxBuckets || share * 20 > B::MOST * 17) return B200ALG_OK;
    // the small arrays lie where the passes over tiles have their counts
    char *at = (char *)temp + sizeof(TempHeader);
    auto take = [&](int64_t bytes) {
        char *p = at;
        at += round_up(bytes, 256);
        return p;
    };
    SampleSort<K, V> a;
    a.splitter_keys = (K *)take(buckets * sizeof(K));
    a.splitter_index = (unsigned int *)take(buckets * 4);
    char *const over = at;  // the counts go over the sample: no block counts before all have ranked
    a.sample_keys = (K *)take(blocks * kPublished * sizeof(K));
    a.sample_index = (unsigned int *)take(blocks * kPublished * 4);
    if (at - (char *)temp > scratch.control_bytes) return B200ALG_OK;
    at = over;
    a.counts = (unsigned short *)take(blocks * (buckets > kRadix ? round_up(buckets, 8) : kRadix) * 2);
    if (at - (char *)temp > scratch.control_bytes) return B200ALG_OK;
    a.io = SortBuffers<K, V>{(const K *)call.in_keys, (K *)call.out_keys, (K *)scratch.alt_keys, (const V *)call.in_values, (V *)call.out_values,
                             (V *)scratch.alt_values, call.stride, n, call.n_device};
    a.xf = KeyXform<K>{(K)xn, (K)xp};
    a.hdr = (TempHeader *)temp;
    a.buckets = (int)buckets;
    a.value_seq = call.value_seq;
    a.in_cluster = in_cluster;
    const SampleLaunch launch(s, (int)blocks, in_cluster);
    const cudaError_t e = cudaLaunchKernelEx(&launch.cfg, kernel, a);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {  // not resident as a whole: other ways need no such thing
        (void)cudaGetLastError();
        return B200ALG_OK;
    }
    B200ALG_CUDA_TRY(e);
    *taken = true;
    return B200ALG_OK;
}

template <typename K>
static int sample_sort_key(cudaStream_t s, const SortCall &call, int value_bytes, uint64_t xn, uint64_t xp, void *temp, const SortScratch &scratch, bool *taken) {
    switch (value_bytes) {
    case 0:
        if constexpr (sizeof(K) == 8) return run_sample_sort<K, NoValue>(s, call, xn, xp, temp, scratch, taken);
        break;
    case 1: return run_sample_sort<K, uint8_t>(s, call, xn, xp, temp, scratch, taken);
    case 2: return run_sample_sort<K, uint16_t>(s, call, xn, xp, temp, scratch, taken);
    case 4: return run_sample_sort<K, uint32_t>(s, call, xn, xp, temp, scratch, taken);
    case 8: return run_sample_sort<K, uint64_t>(s, call, xn, xp, temp, scratch, taken);
    case 16: return run_sample_sort<K, uint4>(s, call, xn, xp, temp, scratch, taken);
    }
    return B200ALG_UNSUPPORTED;
}

int sample_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xn, uint64_t xp, void *temp,
                const SortScratch &scratch, bool *taken) {
    *taken = false;
    if (key_bytes == 4 && value_bytes) return sample_sort_key<uint32_t>(s, call, value_bytes, xn, xp, temp, scratch, taken);
    if (key_bytes == 8) return sample_sort_key<uint64_t>(s, call, value_bytes, xn, xp, temp, scratch, taken);
    return B200ALG_OK;
}

}  // namespace b200alg
