// Radix sort of views of some ten thousand to a few million elements: one partition into buckets that a block
// can sort alone (local_sort.cuh), in one cooperative launch.
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
#include "local_sort.cuh"

#include <cooperative_groups.h>

namespace b200alg {

namespace cg = cooperative_groups;

constexpr int kSampleThreads = 512, kSampleItems = kLocalMost / kSampleThreads;
constexpr int kSampled = 128, kPublished = 64;  // keys of a block
constexpr int kMaxBuckets = 480;                // the last digit (511) is what fills a share up
constexpr int kPartitionDigits = 1 << kLocalDigitBits;
constexpr int kSampleSmem = 227 * 1024;

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
    K *splitter_keys;            // [buckets - 1]
    unsigned int *splitter_index;
    unsigned short *counts;      // [blocks][padded buckets]
    int buckets, value_seq;
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
    SampleShared<K> *m;
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

// One partition: where its elements come from and go to, and what their buckets are.
template <typename K, typename V> struct Partition {
    const K *from;
    K *to;
    const V *vfrom;
    V *vto;
    int64_t from_stride, to_stride;
    bool raw_in, raw_out;  // keys as the caller has them, else transformed
    int value_seq;
    int shift;    // of the digit (eight bits), or
    int height;   // of the tree of splitters (shift < 0)
    int buckets;
};

template <typename K, typename V>
__global__ void __launch_bounds__(kSampleThreads, 1)
sample_sort_kernel(SampleSort<K, V> a) {
    using B = SampleBlock<K, V>;
    constexpr int VB = B::VB;
    constexpr bool PLACE = by_place<K>(VB != 0);
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blocks = (int)gridDim.x;
    SampleShared<K> *const m = reinterpret_cast<SampleShared<K> *>(smem + local_fixed_bytes(kSampleThreads));
    const int64_t n64 = effective_n(a.io);
    B b;
    b.shared = local_shared(smem);
    b.m = m;
    b.n = (unsigned int)n64;
    const unsigned int share = (b.n + blocks - 1) / blocks;
    b.lo = blockIdx.x * share < b.n ? blockIdx.x * share : b.n;
    const int len = (int)(b.n - b.lo < share ? b.n - b.lo : share);  // of this block
    const int items = ((int)share + kSampleThreads - 1) / kSampleThreads, own = warp * 32 * items + lane;
    b.words = reinterpret_cast<unsigned int *>(m + 1);
    b.values = reinterpret_cast<V *>(b.words + B::MOST);
    b.keys = reinterpret_cast<K *>(reinterpret_cast<unsigned char *>(b.values) + (size_t)B::MOST * VB);

    Partition<K, V> part{a.io.in, a.io.alt, a.io.vin, a.io.valt, a.io.stride, 1, true, false, a.value_seq, -1, 0, a.buckets};
    auto fetch_share = [&]() { b.fetch(part.from, part.from_stride, part.vfrom, part.value_seq, b.lo, len, items); };
    if (blockIdx.x == 0 && tid == 0) a.hdr->wait_limit_hit = 0u;
    local_clear(b.shared);

    // ---- sample ----
    K own_key = (K)~(K)0;
    unsigned int own_index = b.n;
    if (tid < kSampled && len > 0) {
        const unsigned int stratum = len / kSampled;
        const unsigned int shift = stratum ? ((blockIdx.x * kSampled + tid) * 2654435761u >> 8) % stratum : 0u;
        own_index = b.lo + (unsigned int)((unsigned long long)tid * len / kSampled) + shift;
        own_key = a.io.in[(int64_t)own_index * a.io.stride];
    }
    fetch_share();  // comes while the splitters are found
    if (tid < kPartitionDigits) m->total[tid] = 0u;
    if (tid < kSampled) {
        if (len > 0) own_key = a.xf(own_key);
        m->splitter[tid] = own_key;
        m->count[tid] = 0u;
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
    constexpr int EVERY = kSampled / kPublished;
    static_assert(EVERY == 2, "of a pair, neighbouring blocks publish one the lower and one the upper: the ranks stay unbiased");
    if (tid < kSampled && m->count[tid] % EVERY == (blockIdx.x & 1)) {
        const int e = (int)(m->count[tid] / EVERY);
        m->tree[e] = own_key;
        m->index[e] = own_index;
        a.sample_keys[blockIdx.x * kPublished + e] = own_key;
        a.sample_index[blockIdx.x * kPublished + e] = own_index;
    }
    cg::this_grid().sync();
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
    cg::this_grid().sync();

    // ---- partition ----
    const int splitters = a.buckets - 1;
    while (1 << part.height < a.buckets) ++part.height;
    if (tid > 0 && tid < 1 << part.height) {
        const int level = 31 - __clz(tid), at = ((2 * (tid - (1 << level)) + 1) << (part.height - 1 - level)) - 1;
        m->tree[tid] = at < splitters ? __ldcg(a.splitter_keys + at) : (K)~(K)0;
    }
    if (tid < splitters) {
        m->splitter[tid] = __ldcg(a.splitter_keys + tid);
        m->index[tid] = __ldcg(a.splitter_index + tid);
    }
    const bool bucket_thread = tid < kPartitionDigits;
    for (;;) {  // (once, if no bucket is too large)
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
#pragma unroll 1
        for (int first = 0; first < items; first += AHEAD) {
            const int mine = own + first * 32;
            K bits[AHEAD];
            unsigned int bucket[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int at = mine + i * 32;
                bits[i] = b.keys[at < len ? at : 0];
                if (part.raw_in) bits[i] = a.xf(bits[i]);
                bucket[i] = 1u;
            }
            if (part.shift >= 0) {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) bucket[i] = (unsigned int)(bits[i] >> part.shift) & (kRadix - 1u);
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
        cg::this_grid().sync();
        // eight buckets of a row per thread and turn
        const int chunks = padded / 8, groups = kSampleThreads / chunks, chunk = tid % chunks, group = tid / chunks;
        unsigned int all[8] = {0, 0, 0, 0, 0, 0, 0, 0}, ahead[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (group < groups) {
#pragma unroll 1
            for (int r = group; r < blocks; r += 4 * groups) {
                uint4 c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    c[j] = r + j * groups < blocks ? __ldcg(reinterpret_cast<const uint4 *>(a.counts + (size_t)(r + j * groups) * padded) + chunk)
                                                   : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned int v[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
                    const bool mine = r + j * groups < (int)blockIdx.x;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        all[2 * q] += v[q] & 0xFFFFu;
                        all[2 * q + 1] += v[q] >> 16;
                        ahead[2 * q] += mine ? v[q] & 0xFFFFu : 0u;
                        ahead[2 * q + 1] += mine ? v[q] >> 16 : 0u;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {  // (neighbouring lanes, neighbouring banks)
                atomicAdd(&m->total[q * (kPartitionDigits / 8) + chunk], all[q]);
                atomicAdd(&m->before[q * (kPartitionDigits / 8) + chunk], ahead[q]);
            }
        }
        __syncthreads();
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
            for (;;) {
                bool bad = false;
#pragma unroll 4
                for (int p = tid; p < len; p += kSampleThreads) {
                    const unsigned int word = b.words[p], place = word & ((1u << kPlaceBits) - 1u);
                    const unsigned int at = m->first[word >> kPlaceBits] + p;
                    const K bits = b.keys[place];
                    if (in_order) bad |= p + 1 < len && b.words[p + 1] < word;
                    part.to[(int64_t)at * part.to_stride] = part.raw_out ? a.xf.raw(bits) : bits;
                    if constexpr (VB != 0) part.vto[at] = b.values[place];
                }
                // Lanes that met in one counter were served in another order than theirs: what is in which bucket is
                // right, the order inside is put right and the elements are stored again.
                if (!__syncthreads_or(bad)) break;
                using Words = LocalSort<unsigned int, false, kSampleItems>;
                Words::repair(Words{b.shared, b.words, nullptr, len, items, 0u, 0u});
            }
        }
        cg::this_grid().sync();  // the elements have been stored, and all blocks have read the counts
        if (!too_large && part.shift < 0) break;
        // All digits of eight bits, lowest first: from the input to the alternate buffer, to the output, and so on.
        static_assert(sizeof(K) % 2 == 0, "the last pass writes the output view");
        const int pass = part.shift < 0 ? 0 : part.shift / 8 + 1;
        if (pass == (int)sizeof(K)) return;
        const bool home = (pass & 1) != 0;
        part = Partition<K, V>{pass == 0 ? a.io.in : home ? a.io.alt : a.io.out, home ? a.io.out : a.io.alt,
                               pass == 0 ? a.io.vin : home ? a.io.valt : a.io.vout, home ? a.io.vout : a.io.valt,
                               home ? 1 : a.io.stride, home ? a.io.stride : 1, pass == 0, pass + 1 == (int)sizeof(K),
                               pass == 0 ? a.value_seq : kSeqNone, pass * 8, 0, kRadix};
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
        K key[kSampleItems];
        K low = (K)~(K)0, high = 0;
        if constexpr (PLACE) {
            b.fetch(a.io.alt, 1, a.io.valt, kSeqNone, start, count, items);
            copies_wait();
        }
#pragma unroll
        for (int i = 0; i < kSampleItems; ++i) {
            if (i >= items) break;
            const int at = own + i * 32;
            if (at < count) {
                if constexpr (PLACE) {
                    const K k = b.keys[at];
                    low = k < low ? k : low;
                    high = k > high ? k : high;
                } else {
                    key[i] = __ldcg(a.io.alt + start + at);
                }
            }
        }
        if constexpr (!PLACE) {
#pragma unroll
            for (int i = 0; i < kSampleItems; ++i) {
                if (i >= items) break;
                if (own + i * 32 < count) {
                    low = key[i] < low ? key[i] : low;
                    high = key[i] > high ? key[i] : high;
                }
            }
        }
        local_range(b.shared, low, high);
        const LocalSort<K, PLACE, kSampleItems> sort{b.shared, b.words, b.keys, count, items, low, high};
        sort.run(key, [=](int p, K k, unsigned int word) {
            out[(int64_t)(start + p) * stride] = xf.raw(k);
            if constexpr (VB != 0) vout[start + p] = values[LocalSort<K, PLACE, kSampleItems>::place_of(word)];
        });
        __syncthreads();
    }
}

// ---- host side ---------------------------------------------------------------------------
// Which sorts: 8-byte keys, and 4-byte keys with values, as long as a share fits a block with some room to spare; a
// bucket is meant to be 60 % of what fits (the largest is 1.2 to 1.4 times that).  4-byte keys alone gain nothing
// (300000: 37.3 against 38.0 us, 10^6: 62.9 against 63.5).  Against a pass per key byte, us with the copy that brings
// the data, by key bytes / value bytes:
//              20000         50000         100000        200000        400000        800000        1100000       1500000
//   8 / 0    29.3          29.7          31.7  65.6    38.2  67.4    42.0  88.0    51.7          66.3          76.6  131.4
//            27.7  20.9    27.7  23.6    30.4  28.7    36.2  30.9    40.0  39.3    49.2  57.0    63.1  64.7    73.2   72.3  below 2^20
//   8 / 4    32.4          32.9          35.5  76.4    42.7  84.5    49.1  104.2   60.9          78.4            does not fit
//            30.6  26.1    31.5  30.2    33.8  35.8    40.0  40.8    47.0  51.2    57.6  74.7    75.6  83.0       below 2^20
//   4 / 4    30.4          30.9          32.0  40.7    37.1  46.4    44.5  59.6    54.6          68.4          77.4   81.4
//            29.5  23.5    30.1  28.7    30.7  33.0    36.0  37.6    42.0  46.8    52.4  62.4    65.2  69.9    75.2   76.4  below 2^20
// (The passes' clearing has since come to start early, 3 us less for them: at the end of the range, uint32 pairs 67.7 us
// by buckets against 68.7 just past it, below 2^20 65.8 against 65.8; uint64 keys 79.6 against 127.2, 71.9 against 67.9.)
// so integers go this way from where those below 2^20 (three passes) lose nothing, floating-point keys, which differ
// in all bytes, from where one block does not hold them (8 bytes) or a cluster is not faster (4).
// Shares of 1024, 1536, 2048 and 3072 elements: 100000 uint32 pairs 33.3, 32.5, 32.9, 34.8; 30000 30.7, 30.9, 32.8, 34.7.
constexpr int kSampleShare = 1536;
constexpr int64_t sample_least(int key_bytes, int value_bytes, bool floating) {
    return floating ? (key_bytes == 8 ? 1 : 20000) : value_bytes ? 100000 : 700000;
}

template <typename K, typename V>
static int run_sample_sort(cudaStream_t s, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, const SortScratch &scratch, bool *taken) {
    using B = SampleBlock<K, V>;
    constexpr int VB = B::VB;
    *taken = false;
    auto kernel = sample_sort_kernel<K, V>;
    static ContextCache<int> cache;
    int resident = 0;
    if (!cache.find(&resident)) {
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmem));
        int per_sm = 0;
        B200ALG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSampleThreads, kSampleSmem));
        resident = per_sm * sm_count();
        cache.store(resident);
    }
    const int64_t n = call.n;
    if (n < sample_least(sizeof(K), VB, xn != xp)) return B200ALG_OK;  // (integers' transforms have one constant)
    int64_t blocks = ceil_div(n, kSampleShare);
    blocks = blocks < resident ? blocks : resident;
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
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kSampleThreads);
    cfg.dynamicSmemBytes = kSampleSmem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
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
