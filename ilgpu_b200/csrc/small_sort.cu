// Radix sort of views that fit on the SMs as a whole: one launch.
//
// What a short sort costs is not moving keys but the chain of steps: with one kernel per step (clear,
// histogram, offsets, one per digit, copy home) 5000 keys took 50 us, 25 of them inside kernels that
// wait for memory or for one another.
//
// What one block can hold it sorts alone (block_sort_kernel, local_sort.cuh).  Several blocks keep their
// shares of the keys in registers and shared memory (resident_sort_kernel); a pass is
//
//   rank      one shared-memory atomic per key on the warp's count of its digit
//   count     the warps' counts become slots of the block's tile
//   reorder   keys to their slots in shared memory, and a check of their order (see digit_pass.cuh)
//   exchange  blocks publish their counts, meet, add up the counts of all blocks, move their slots to
//             where they go, and meet again
//
// The up to sixteen blocks of a cluster read one another's counts and move keys through distributed
// shared memory; only the first and the last step touch global memory.  More blocks than that exchange
// through global memory, in place (everybody has read its share when they meet), and meet in the grid
// barrier of a cooperative launch.  Digits that all keys share are skipped.
#include "local_sort.cuh"

#include <cooperative_groups.h>

namespace b200alg {

namespace cg = cooperative_groups;

constexpr int kResidentThreads = 512;
constexpr int kResidentWarps = kResidentThreads / 32;
constexpr int kResidentSmem = 227 * 1024;
constexpr int kResidentFixed = kResidentWarps * kRadix * 4 + 2 * kRadix * 4 + kRadix * 2 + 1024;
constexpr int kColumnThreads = kResidentThreads / kRadix;     // threads that share a digit when counts become slots
constexpr int kColumnRows = kResidentWarps / kColumnThreads;  // and warps each of them adds up
constexpr int kMaxCluster = 16;
enum : int { kInCluster = 0, kInGrid = 1 };

// Shared memory of a key and its value: slots and the value's place; in a cluster, where the next pass
// comes in as well.
__host__ __device__ constexpr int resident_bytes(int key_bytes, int value_bytes, bool cluster) {
    return (cluster ? 2 : 1) * (key_bytes + value_bytes) + (value_bytes ? 2 : 0);
}
__host__ __device__ constexpr int resident_items(int key_bytes, int value_bytes, bool cluster) {
    const int fit = (kResidentSmem - kResidentFixed) / (kResidentThreads * resident_bytes(key_bytes, value_bytes, cluster));
    return fit < 16 ? fit : 16;
}
static size_t resident_smem(int key_bytes, int value_bytes, bool cluster, int items) {
    return (size_t)kResidentThreads * items * resident_bytes(key_bytes, value_bytes, cluster) + kResidentFixed;
}

struct ResidentWords {  // the small shared words of a block
    unsigned int warp_sum[kResidentWarps];
    unsigned long long warp_any[kResidentWarps], warp_all[kResidentWarps];
    unsigned long long any, all;  // bits set in some key, bits set in every key of the block
    unsigned long long differ;    // bits in which keys of the view differ
};

template <typename K, typename V>
__global__ void __launch_bounds__(kResidentThreads, 1)
resident_sort_kernel(SortBuffers<K, V> io, KeyXform<K> xf, TempHeader *hdr, unsigned long long *masks, unsigned short *all_counts, int items,
                     int meeting, int value_seq) {
    constexpr int VB = ValueBytes<V>::value;
    constexpr int ITEMS = resident_items(sizeof(K), VB, false);
    constexpr bool VALUES = VB != 0;
    constexpr int PASSES = sizeof(K);
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned int tile = kResidentThreads * items;
    unsigned int *table = reinterpret_cast<unsigned int *>(smem);        // counts per warp and digit
    unsigned int *excl = table + kResidentWarps * kRadix;                // a digit's first slot
    unsigned int *goff = excl + kRadix;                                  // global index of a slot minus the slot
    unsigned short *counts = reinterpret_cast<unsigned short *>(goff + kRadix);  // the block's keys of a digit
    ResidentWords &m = *reinterpret_cast<ResidentWords *>(counts + kRadix);
    V *values = reinterpret_cast<V *>(smem + kResidentFixed);            // in input order
    V *next_values = values + (meeting == kInCluster && VALUES ? tile : 0);
    K *slots = reinterpret_cast<K *>(smem + kResidentFixed + (size_t)tile * VB * (meeting == kInCluster ? 2 : 1));  // keys in slot order
    K *next_keys = slots + tile;                                         // (cluster) keys of the next pass
    unsigned short *place = reinterpret_cast<unsigned short *>(slots + (meeting == kInCluster ? 2 * tile : tile));  // slot's place in the input
    static_assert(sizeof(ResidentWords) <= 1024, "room for the small words");

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_dependency_wait();
    const int64_t n = effective_n(io);
    const int64_t base = (int64_t)blockIdx.x * tile;
    const int valid = (int)(n - base < 0 ? 0 : (n - base < tile ? n - base : tile));
    const int own = warp * 32 * items + lane;  // this lane's first key; the others follow 32 apart
    const int blocks = (int)gridDim.x;
    cg::cluster_group cluster = cg::this_cluster();
    auto meet = [&]() {
        if (meeting == kInCluster) cluster.sync();
        else cg::this_grid().sync();
    };
    if (blockIdx.x == 0 && tid == 0) hdr->wait_limit_hit = 0u;
    unsigned int *mine = table + warp * kRadix;
    const unsigned int swizzle = (unsigned int)(warp / kColumnRows * (32 / kColumnThreads));  // the threads of a digit read different banks
    auto clear_mine = [&]() {
#pragma unroll
        for (int i = 0; i < kRadix / 4 / 32; ++i) reinterpret_cast<uint4 *>(mine)[i * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
    };
    clear_mine();

    // (The loops over a thread's keys end with a jump out of the unrolled code: testing every step costs
    // as much as the step.)
    K key[ITEMS];
    // the block's share of a global view (past L1: other blocks have written it)
    auto load = [&](const K *from, const V *vfrom, bool sequence) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            const int at = own + i * 32;
            key[i] = at < valid ? __ldcg(from + (base + at) * io.stride) : padding_key<K>(xf);
        }
        if constexpr (VALUES) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                if (i >= items) break;
                const int at = own + i * 32;
                if (at < valid) {
                    if constexpr (VB <= 8) values[at] = sequence ? sequence_value<V>(value_seq, base + at) : __ldcg(vfrom + base + at);
                    else values[at] = __ldcg(vfrom + base + at);
                }
            }
        }
    };
    load(io.in, io.vin, value_seq != kSeqNone);
    {   // which bits differ between keys
        unsigned long long any = 0ull, all = ~0ull;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            if (own + i * 32 < valid) {
                any |= (unsigned long long)xf(key[i]);
                all &= (unsigned long long)xf(key[i]);
            }
        }
        unsigned int any_hi = 0u, all_hi = ~0u;
        if (sizeof(K) == 8) {
            any_hi = __reduce_or_sync(0xffffffffu, (unsigned int)(any >> 32));
            all_hi = __reduce_and_sync(0xffffffffu, (unsigned int)(all >> 32));
        }
        any = (unsigned long long)any_hi << 32 | __reduce_or_sync(0xffffffffu, (unsigned int)any);
        all = (unsigned long long)all_hi << 32 | __reduce_and_sync(0xffffffffu, (unsigned int)all);
        if (lane == 0) {
            m.warp_any[warp] = any;
            m.warp_all[warp] = all;
        }
        __syncthreads();
        if (warp == 0) {
            any = m.warp_any[lane % kResidentWarps];
            all = m.warp_all[lane % kResidentWarps];
#pragma unroll
            for (int k = 1; k < kResidentWarps; k <<= 1) {
                any |= __shfl_xor_sync(0xffffffffu, any, k);
                all &= __shfl_xor_sync(0xffffffffu, all, k);
            }
            if (lane == 0) {
                m.any = any;
                m.all = all;
                m.differ = any & ~all;
                if (meeting == kInGrid) {
                    masks[2 * blockIdx.x] = any;
                    masks[2 * blockIdx.x + 1] = all;
                }
            }
        }
    }
    auto next_pass = [&](int p) {  // the first digit from p on in which keys differ
        const unsigned long long differ = m.differ;
        while (p < PASSES && !(differ >> (8 * p) & 0xFFull)) ++p;
        return p;
    };
    bool first = true;
    // (what differs is known only when the blocks have met, so the first pass always runs)
    int pass = 0;
    while (pass < PASSES) {
        const int shift = pass * 8;
        if (!first) {
            if (meeting == kInGrid) {
                load(io.out, io.vout, false);
            } else {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    if (i >= items) break;
                    key[i] = next_keys[own + i * 32];
                }
            }
        }
        unsigned int rank[ITEMS];  // keys of the digit the warp has counted before
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            rank[i] = atomicAdd(mine + (((unsigned int)(xf(key[i]) >> shift) & 0xFFu) ^ swizzle), 1u);
        }
        __syncthreads();
        {   // kColumnThreads neighbouring threads share a digit, each adds up the counts of kColumnRows warps
            const int d = tid / kColumnThreads, part = tid % kColumnThreads;
            unsigned int *column = table + part * (kColumnRows * kRadix) + (d ^ (part * (32 / kColumnThreads)));
            unsigned int ahead[kColumnRows], part_total = 0;
#pragma unroll
            for (int w = 0; w < kColumnRows; ++w) {
                const unsigned int a = column[w * kRadix];
                ahead[w] = part_total;
                part_total += a;
            }
            unsigned int total = part_total;  // of the parts up to mine, then of all
#pragma unroll
            for (int k = 1; k < kColumnThreads; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, total, k);
                if (part >= k) total += up;
            }
            const unsigned int parts_ahead = total - part_total;
            total = __shfl_sync(0xffffffffu, total, lane | (kColumnThreads - 1));
            if (part == 0) {
                if (meeting == kInCluster) counts[d] = (unsigned short)total;
                else all_counts[(size_t)blockIdx.x * kRadix + d] = (unsigned short)total;
            }
            // exclusive scan of the digits' counts, over the warp and then over the warps
            unsigned int incl = total;
#pragma unroll
            for (int k = kColumnThreads; k < 32; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += up;
            }
            if (lane == 31) m.warp_sum[warp] = incl;
            __syncthreads();
            const unsigned int start = __reduce_add_sync(0xffffffffu, lane < warp ? m.warp_sum[lane] : 0u) + incl - total;
            if (part == 0) excl[d] = start;
#pragma unroll
            for (int w = 0; w < kColumnRows; ++w) column[w * kRadix] = start + parts_ahead + ahead[w];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            const unsigned int slot = rank[i] + mine[((unsigned int)(xf(key[i]) >> shift) & 0xFFu) ^ swizzle];
            slots[slot] = key[i];
            if (VALUES) place[slot] = (unsigned short)(own + i * 32);
        }
        __syncthreads();
        auto wrong = [&](unsigned int p) {
            return out_of_order<K, VALUES>(slots[p], slots[p + 1], VALUES ? place[p] : 0u, VALUES ? place[p + 1] : 0u, xf, shift);
        };
        bool bad = false;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= items) break;
            const unsigned int p = tid + i * kResidentThreads;
            if (p + 1 < tile) bad |= wrong(p);
        }
        if (__syncthreads_or(bad))  // (the atomics of a warp were not served in lane order: not observed)
            put_in_order<K, VALUES>(slots, place, (int)tile, tid, kResidentThreads, xf, shift, [](bool moved) { return __syncthreads_or(moved) != 0; });

        meet();  // counts (and, the first time, masks) of all blocks are there; every block holds its share
        // the counts of all blocks, one row per warp and turn, summed in the ranking tables' place
        unsigned int *part_all = table, *part_before = table + kResidentWarps / 2 * kRadix;
        constexpr int kSumWarps = kResidentWarps / 2;
        if (warp < kSumWarps && warp < blocks) {
            unsigned int all[8] = {0, 0, 0, 0, 0, 0, 0, 0}, before[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            auto add = [&](int r, const uint4 c) {
                const unsigned int w[4] = {c.x, c.y, c.z, c.w};
                const bool ahead = r < (int)blockIdx.x;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    all[2 * q] += w[q] & 0xFFFFu;
                    all[2 * q + 1] += w[q] >> 16;
                    before[2 * q] += ahead ? w[q] & 0xFFFFu : 0u;
                    before[2 * q + 1] += ahead ? w[q] >> 16 : 0u;
                }
            };
            if (meeting == kInCluster) {
                for (int r = warp; r < blocks; r += kSumWarps) add(r, reinterpret_cast<const uint4 *>(cluster.map_shared_rank(counts, r))[lane]);
            } else {
                constexpr int AHEAD = 10; // rows in flight
                for (int r = warp; r < blocks; r += AHEAD * kSumWarps) {
                    uint4 c[AHEAD];
#pragma unroll
                    for (int j = 0; j < AHEAD; ++j)
                        c[j] = r + j * kSumWarps < blocks ? __ldcg(reinterpret_cast<const uint4 *>(all_counts + (size_t)(r + j * kSumWarps) * kRadix) + lane)
                                                          : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                    for (int j = 0; j < AHEAD; ++j) add(r + j * kSumWarps, c[j]);
                }
            }
            uint4 *to = reinterpret_cast<uint4 *>(part_all + warp * kRadix) + lane * 2;
            to[0] = make_uint4(all[0], all[1], all[2], all[3]);
            to[1] = make_uint4(all[4], all[5], all[6], all[7]);
            to = reinterpret_cast<uint4 *>(part_before + warp * kRadix) + lane * 2;
            to[0] = make_uint4(before[0], before[1], before[2], before[3]);
            to[1] = make_uint4(before[4], before[5], before[6], before[7]);
        } else if (first && warp == kResidentWarps - 1) {
            unsigned long long any = 0ull, all = ~0ull;
            for (int r = lane; r < blocks; r += 32) {
                if (meeting == kInCluster) {
                    const ResidentWords *other = cluster.map_shared_rank(&m, r);
                    any |= other->any;
                    all &= other->all;
                } else {
                    any |= __ldcg(masks + 2 * r);
                    all &= __ldcg(masks + 2 * r + 1);
                }
            }
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                any |= __shfl_xor_sync(0xffffffffu, any, k);
                all &= __shfl_xor_sync(0xffffffffu, all, k);
            }
            if (lane == 0) m.differ = any & ~all;
        }
        __syncthreads();
        unsigned int at_digit = 0u;
        if (tid < kRadix) {
            unsigned int all = 0u, before = 0u;
            const int rows = blocks < kSumWarps ? blocks : kSumWarps;
#pragma unroll
            for (int w = 0; w < kSumWarps; ++w)
                if (w < rows) {
                    all += part_all[w * kRadix + tid];
                    before += part_before[w * kRadix + tid];
                }
            unsigned int incl = all;
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += up;
            }
            if (lane == 31) m.warp_sum[warp] = incl;
            at_digit = incl - all + before - excl[tid];
        }
        __syncthreads();
        if (tid < kRadix) goff[tid] = at_digit + __reduce_add_sync(0xffffffffu, lane < warp ? m.warp_sum[lane] : 0u);
        clear_mine();
        __syncthreads();
        first = false;
        const int after = next_pass(pass + 1);
        if (meeting == kInCluster && after < PASSES) {
            const unsigned int inverse = 0xFFFFFFFFu / tile + 1u;  // at / tile for at below 2^17
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                if (i >= items) break;
                const unsigned int p = tid + i * kResidentThreads;
                const K k = slots[p];
                const unsigned int at = goff[(unsigned int)(xf(k) >> shift) & 0xFFu] + p;
                const unsigned int to = __umulhi(at, inverse);
                if (at < (unsigned int)blocks * tile) {
                    cluster.map_shared_rank(next_keys, to)[at - to * tile] = k;
                    if constexpr (VALUES) cluster.map_shared_rank(next_values, to)[at - to * tile] = values[place[p]];
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                if (i >= items) break;
                const int p = tid + i * kResidentThreads;
                if (p < valid) {
                    const K k = slots[p];
                    const unsigned int at = goff[(unsigned int)(xf(k) >> shift) & 0xFFu] + (unsigned int)p;
                    io.out[(int64_t)at * io.stride] = k;
                    if constexpr (VALUES) io.vout[at] = values[place[p]];
                }
            }
        }
        pass = after;
        // everything has arrived (or, at the end, nobody reads this block's shared memory any more)
        if (pass < PASSES || meeting == kInCluster) meet();
        if (VALUES && meeting == kInCluster) {
            V *v = values;
            values = next_values;
            next_values = v;
        }
    }
}

// ---- one block ---------------------------------------------------------------------------
// 1024 threads of half as many elements: 5000 uint32 keys 14.3 instead of 12.3 us (turning counts into places takes 1800
// instead of 930 cycles a pass).
constexpr int kAloneThreads = 512, kAloneItems = kLocalMost / kAloneThreads;
template <typename K, typename V>
__global__ void __launch_bounds__(kAloneThreads, 1)
block_sort_kernel(SortBuffers<K, V> io, KeyXform<K> xf, TempHeader *hdr, int items, int value_seq) {
    constexpr int VB = ValueBytes<V>::value;
    constexpr bool PLACE = by_place<K>(VB != 0);
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, threads = (int)blockDim.x, most = threads * items;
    unsigned int *words = reinterpret_cast<unsigned int *>(smem + local_fixed_bytes(threads));
    V *values = reinterpret_cast<V *>(words + most);
    K *keys = reinterpret_cast<K *>(reinterpret_cast<unsigned char *>(values) + (size_t)most * VB);
    const int own = (tid >> 5) * 32 * items + (tid & 31);
    const LocalShared shared = local_shared(smem);
    local_clear(shared);
    grid_dependency_wait();
    const int count = (int)effective_n(io);
    if (tid == 0) hdr->wait_limit_hit = 0u;

    K key[kAloneItems];
    K low = (K)~(K)0, high = 0;
#pragma unroll
    for (int i = 0; i < kAloneItems; ++i) {
        if (i >= items) break;
        const int at = own + i * 32;
        if (at < count) key[i] = io.in[(int64_t)at * io.stride];
    }
    if constexpr (VB != 0) load_values<V>(values, io.vin, value_seq, 0, own, count, items);
#pragma unroll
    for (int i = 0; i < kAloneItems; ++i) {
        if (i >= items) break;
        const int at = own + i * 32;
        if (at < count) {
            const K b = xf(key[i]);
            key[i] = b;
            low = b < low ? b : low;
            high = b > high ? b : high;
            if constexpr (PLACE) keys[at] = b;
        }
    }
    local_range(shared, low, high);
    const LocalSort<K, PLACE, kAloneItems> sort{shared, words, keys, count, items, low, high};
    K *const out = io.out;
    V *const vout = io.vout;
    const int64_t stride = io.stride;
    sort.run(key, [=](int p, K k, unsigned int word) {
        out[p * stride] = xf.raw(k);
        if constexpr (VB != 0) vout[p] = values[LocalSort<K, PLACE, kAloneItems>::place_of(word)];
    });
}

// ---- host side ---------------------------------------------------------------------------
// Which blocks (times on the GPU, us, with the launch and the copy that brings the data):
//   one       block_sort_kernel, against a cluster, by key bytes / value bytes.  What a cluster takes depends on the
//             bytes in which keys differ; the line for integers is where identifiers below 2^20 (three bytes) cost the
//             same either way.
//                          4500          6200          7500          9000         12000
//                1 / 0    8.4   8.3    8.2   8.4   10.2   8.6   10.3   8.2   12.3   8.8
//                2 / 0   10.2  12.3   10.3  12.3   12.3  12.3   14.3  12.5   16.4  13.1
//                1 / 4   12.5  13.2   12.3  13.2   14.4  13.2   16.7  13.3   21.3  24.7
//                2 / 8   14.7  17.3   15.9  17.6   16.9  17.4   19.1  17.6   22.6  17.4
//                4 / 0   11.3  16.6   12.3  18.4   14.3  18.5   16.4  20.8   19.1  20.8
//                        12.1  14.3   14.3  16.4   14.4  16.2   16.4  16.4   19.2  16.4   below 2^20
//                4 / 4   15.1  23.6   16.6  24.8   19.5  24.3   21.9  25.5   25.7  27.8
//                        16.3  19.9   18.5  20.3   19.9  20.1   22.5  21.3   26.3  21.3   below 2^20
//                8 / 0   12.3  29.0   14.4  35.2   16.4  34.7   18.4  37.5   22.5  39.9
//                        13.3  15.4   16.4  16.4   18.3  16.4   20.5  19.1   24.6  18.6   below 2^20
//                8 / 4   17.0  42.2   19.1  42.5   21.3  42.3   23.5  46.7   27.7  46.8
//                        16.4  21.3   20.5  21.3   20.5  21.3   24.5  22.7   29.1  23.4   below 2^20
//                8 / 8   18.7  41.9   21.2  43.3   25.3  42.4   28.3  46.9    does not fit
//             Longer floating-point keys go by buckets in a cluster (4 / 0: by bytes).  One block against these:
//                          5000          6600          8100          9000         12288
//                4 / 0   13.8  18.4   14.4  18.4   16.4  18.2   18.4  18.5   20.5  18.5
//                        12.3  14.4   14.4  14.4   16.4  14.4   16.4  15.3   20.5  15.4   whole numbers below 2^8
//                4 / 4   18.5  24.6   21.2  23.3   23.4  25.1   24.6  25.4   28.6  25.4
//                        16.9  16.4   18.6  16.7   21.2  16.4   22.7  18.7   27.2  17.7   whole numbers below 2^8
//                8 / 0   18.4  22.6   20.5  22.5   22.6  24.6   26.6  24.2   30.8  24.6
//                        14.4  20.5   17.4  20.5   19.5  20.5   21.6  21.6   26.6  21.5   whole numbers below 2^8
//                8 / 4   20.6  27.5   25.6  25.3   27.5  27.5   29.3  27.5   35.9  27.6
//                        19.4  23.5   21.5  23.3   23.5  23.2   25.6  25.5   30.5  24.6   whole numbers below 2^8
//             What one block does not do well is keys that need one pass: 8100 int64 below 2^8 with 4 bytes 17.3, by a
//             block of 1024 threads with a pass per byte 13.7 (but of the full range 23.5 and 42.7).
//   cluster   up to 40960 elements (uint32 keys / pairs: 40000: 27 / 33 us against 29 / 32 us with a
//             grid; 60000: 35 / 43 us against 29 / 33 us);
//   grid      about 64 blocks until they have 4 keys per thread, then more, up to about the length from
//             which the passes over tiles are as fast (against those: 2^20 uint32 keys 61.4 us against 62.1, keys
//             below 2^20 47.2 against 54.1; 786432 uint16 keys with 1, 4 and 8 bytes 37.8, 38.5 and 39.8 against 51.9,
//             50.9 and 43.0).
// Keys of 8 bytes, and of 4 with values, go by buckets from where that is faster (sample_least in sample_sort.cu, asked
// before these two are).
constexpr int64_t alone_most(int key_bytes, int value_bytes, bool floating) {
    if (key_bytes < 4) return key_bytes == 1 ? 6144 : 7680;
    if (key_bytes == 4) return floating || value_bytes == 0 ? 9216 : 7168;
    return floating ? (value_bytes ? 7168 : 8704) : (value_bytes ? 8192 : 6656);
}
constexpr int64_t kClusterMost = 5 * kMaxCluster * kResidentThreads;
constexpr int64_t kGridMostNarrow = 1 << 20, kGridMost = 3 << 18;

template <typename K, typename V>
static int run_block_sort(cudaStream_t s, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, bool *taken) {
    constexpr int VB = ValueBytes<V>::value;
    const int64_t n = call.n;
    if (n > alone_most(sizeof(K), VB, xn != xp)) return B200ALG_OK;  // (integers' transforms have one constant)
    const int threads = n <= kAloneThreads * 2 ? kAloneThreads / 2 : kAloneThreads;  // (1000 keys: 7.2 against 8.1 us)
    const int items = (int)ceil_div(n, threads);
    const size_t smem = local_fixed_bytes(threads) + (size_t)threads * items * local_bytes(sizeof(K), VB);
    if (items > kAloneItems || smem > kResidentSmem) return B200ALG_OK;
    auto kernel = block_sort_kernel<K, V>;
    static ContextCache<int> opted_in;
    int done = 0;
    if (!opted_in.find(&done)) {
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem));
        opted_in.store(1);
    }
    SortBuffers<K, V> io{(const K *)call.in_keys, (K *)call.out_keys, nullptr, (const V *)call.in_values, (V *)call.out_values, nullptr,
                         call.stride, n, call.n_device};
    B200ALG_CUDA_TRY(launch_dependent(kernel, dim3(1), dim3(threads), smem, s, io, KeyXform<K>{(K)xn, (K)xp}, (TempHeader *)temp, items, call.value_seq));
    *taken = true;
    return B200ALG_OK;
}

struct ResidentLimits {
    int cluster;  // most blocks of one cluster
    int grid;     // most blocks of a cooperative launch
};

template <typename K, typename V>
static int run_resident(cudaStream_t s, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, int64_t temp_bytes, bool *taken) {
    constexpr int VB = ValueBytes<V>::value, ITEMS = resident_items(sizeof(K), VB, false), CLUSTER_ITEMS = resident_items(sizeof(K), VB, true);
    auto kernel = resident_sort_kernel<K, V>;
    static ContextCache<ResidentLimits> cache;
    ResidentLimits lim;
    if (!cache.find(&lim)) {
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem));
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        lim.cluster = 1;
        for (int size = kMaxCluster; size > 1; size /= 2) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = size;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(size);
            cfg.blockDim = dim3(kResidentThreads);
            cfg.dynamicSmemBytes = resident_smem(sizeof(K), VB, true, CLUSTER_ITEMS);
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) {
                lim.cluster = size;
                break;
            }
            (void)cudaGetLastError();
        }
        int per_sm = 0;
        B200ALG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kResidentThreads, resident_smem(sizeof(K), VB, false, ITEMS)));
        lim.grid = per_sm * sm_count();
        cache.store(lim);
    }
    const int64_t n = call.n;
    int meeting, blocks;
    if (n <= kClusterMost && n <= (int64_t)lim.cluster * kResidentThreads * CLUSTER_ITEMS) {
        meeting = kInCluster;
        blocks = 2;
        while (blocks < lim.cluster && blocks * kResidentThreads * 2 < n) blocks *= 2;
    } else if (n <= (sizeof(K) <= 4 && VB == 0 ? kGridMostNarrow : kGridMost) && n <= (int64_t)lim.grid * kResidentThreads * ITEMS) {
        meeting = kInGrid;
        const int64_t some = ceil_div(n, kResidentThreads * 2), more = ceil_div(n, kResidentThreads * 4);
        const int64_t want = more > 64 ? more : (some < 64 ? some : 64);
        blocks = (int)(want < lim.grid ? want : lim.grid);
    } else {
        return B200ALG_OK;
    }
    const int items = (int)ceil_div(ceil_div(n, blocks), kResidentThreads);
    unsigned long long *masks = (unsigned long long *)((char *)temp + sizeof(TempHeader));
    unsigned short *counts = (unsigned short *)(masks + 2 * (int64_t)round_up(blocks, 16));
    if ((char *)(counts + (int64_t)blocks * kRadix) - (char *)temp > temp_bytes) return B200ALG_OK;
    SortBuffers<K, V> io{(const K *)call.in_keys, (K *)call.out_keys, nullptr, (const V *)call.in_values, (V *)call.out_values, nullptr,
                         call.stride, n, call.n_device};
    KeyXform<K> xf{(K)xn, (K)xp};
    TempHeader *hdr = (TempHeader *)temp;
    const size_t smem = resident_smem(sizeof(K), VB, meeting == kInCluster, items);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kResidentThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = meeting == kInCluster ? 2 : 1;
    if (meeting == kInCluster) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = blocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, io, xf, hdr, masks, counts, items, meeting, call.value_seq);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {  // not resident as a whole: the passes that need no such thing
        (void)cudaGetLastError();
        return B200ALG_OK;
    }
    B200ALG_CUDA_TRY(e);
    *taken = true;
    return B200ALG_OK;
}

template <typename V>
static int block_sort_key(cudaStream_t s, int key_bytes, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, bool *taken) {
    switch (key_bytes) {
    case 1: return run_block_sort<uint8_t, V>(s, call, xn, xp, temp, taken);
    case 2: return run_block_sort<uint16_t, V>(s, call, xn, xp, temp, taken);
    case 4: return run_block_sort<uint32_t, V>(s, call, xn, xp, temp, taken);
    case 8: return run_block_sort<uint64_t, V>(s, call, xn, xp, temp, taken);
    }
    return B200ALG_UNSUPPORTED;
}

int block_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xn, uint64_t xp, void *temp, bool *taken) {
    *taken = false;
    switch (value_bytes) {
    case 0: return block_sort_key<NoValue>(s, key_bytes, call, xn, xp, temp, taken);
    case 1: return block_sort_key<uint8_t>(s, key_bytes, call, xn, xp, temp, taken);
    case 2: return block_sort_key<uint16_t>(s, key_bytes, call, xn, xp, temp, taken);
    case 4: return block_sort_key<uint32_t>(s, key_bytes, call, xn, xp, temp, taken);
    case 8: return block_sort_key<uint64_t>(s, key_bytes, call, xn, xp, temp, taken);
    case 16: return block_sort_key<uint4>(s, key_bytes, call, xn, xp, temp, taken);
    }
    return B200ALG_UNSUPPORTED;
}

template <typename V>
static int resident_key(cudaStream_t s, int key_bytes, const SortCall &call, uint64_t xn, uint64_t xp, void *temp, int64_t temp_bytes, bool *taken) {
    switch (key_bytes) {
    case 1: return run_resident<uint8_t, V>(s, call, xn, xp, temp, temp_bytes, taken);
    case 2: return run_resident<uint16_t, V>(s, call, xn, xp, temp, temp_bytes, taken);
    case 4: return run_resident<uint32_t, V>(s, call, xn, xp, temp, temp_bytes, taken);
    case 8: return run_resident<uint64_t, V>(s, call, xn, xp, temp, temp_bytes, taken);
    }
    return B200ALG_UNSUPPORTED;
}

int resident_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xn, uint64_t xp, void *temp,
                  int64_t temp_bytes, bool *taken) {
    *taken = false;
    switch (value_bytes) {
    case 0: return resident_key<NoValue>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    case 1: return resident_key<uint8_t>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    case 2: return resident_key<uint16_t>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    case 4: return resident_key<uint32_t>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    case 8: return resident_key<uint64_t>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    case 16: return resident_key<uint4>(s, key_bytes, call, xn, xp, temp, temp_bytes, taken);
    }
    return B200ALG_UNSUPPORTED;
}

}  // namespace b200alg
