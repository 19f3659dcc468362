// Unique: removes consecutive duplicates in place and reports how many elements are left.
// Replaces UniqueKernel / CreateUnique (UniqueExtensions.cs:59-195), whose groups run one after
// the other (SequentialGroupExecutor) and whose first thread compacts a whole tile alone.
// Here every tile flags the elements that differ from their left neighbour, learns how many survive
// before it, and writes its survivors where they belong, in place.  Equality follows Comparison{T} = first.CompareTo(second)
// (ComparisonOperations.tt): integers compare by value; floating-point values compare equal when
// they are numerically equal or both NaN.
#include "common.cuh"
#include "lookback.cuh"

#include <type_traits>

namespace b200alg {

constexpr int kUniqueThreads = 512;
constexpr int kUniqueVecs = 4;                                        // 16-byte vectors per thread
constexpr int kUniqueTileBytes = kUniqueThreads * kUniqueVecs * 16;

template <typename T> struct SameValue {
    static __device__ __forceinline__ bool eq(T a, T b) { return a == b; }
};
template <> struct SameValue<float> {
    static __device__ __forceinline__ bool eq(float a, float b) { return a == b || (a != a && b != b); }
};
template <> struct SameValue<double> {
    static __device__ __forceinline__ bool eq(double a, double b) { return a == b || (a != a && b != b); }
};
template <> struct SameValue<__half> {
    static __device__ __forceinline__ bool eq(__half a, __half b) {
        const float x = __half2float(a), y = __half2float(b);
        return x == y || (x != x && y != y);
    }
};

// The 1- and 2-byte integers travel through the 32-bit shuffles.
template <typename T> __device__ __forceinline__ T shfl_value_up(T v) {
    if constexpr (sizeof(T) <= 2 && !std::is_same<T, __half>::value) return (T)__shfl_up_sync(0xffffffffu, (unsigned int)v, 1);
    else return shfl_up(v, 1);
}
template <typename T> __device__ __forceinline__ T shfl_value(T v, int from) {
    if constexpr (sizeof(T) <= 2 && !std::is_same<T, __half>::value) return (T)__shfl_sync(0xffffffffu, (unsigned int)v, from);
    else return shfl_idx(v, from);
}

// ---- run-length encoding ------------------------------------------------------------------
// Bound: HBM.  A tile is 32 KB: 16-byte loads, four in flight per thread, in warp-striped order (vector
// j of lane l holds elements (warp * 4 * 32 + j * 32 + l) * VEC ... of the tile), so a warp reads whole
// lines; survivors meet in shared memory and leave in consecutive stores.  Tiles are chained with
// decoupled look-back.  (The places of the survivors are stored too, once the prefix is known: the tile
// stays in registers until then.)
template <typename T>
__global__ void __launch_bounds__(kUniqueThreads, 4)
unique_select_kernel(const T *in, int64_t n, T *kept, long long *__restrict__ starts, long long *out_count, TempHeader *hdr,
                     void *state_base, int num_tiles) {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int NV = kUniqueVecs;
    constexpr int TILE = VEC * NV * kUniqueThreads;
    constexpr int WARPS = kUniqueThreads / 32;
    union Vec { uint4 u; T t[VEC]; __device__ Vec() {} };

    __shared__ __align__(16) unsigned char survivors_raw[TILE * sizeof(T)];
    __shared__ unsigned int warp_total[WARPS];
    __shared__ unsigned int s_prefix;
    __shared__ int s_tile;
    T *survivors = reinterpret_cast<T *>(survivors_raw);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = (int)atomicAdd(&hdr->reserved[0], 1u);  // tiles are handed out in order
    __syncthreads();
    const int tile = s_tile;
    const int64_t base = (int64_t)tile * TILE;
    const int64_t remaining = n - base;
    const int warp_first = warp * (NV * 32 * VEC);  // the warp's first element inside the tile

    Vec v[NV];
    if (remaining >= TILE && ((uintptr_t)in & 15u) == 0) {
        const uint4 *src = reinterpret_cast<const uint4 *>(in + base + warp_first) + lane;
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j].u = src[j * 32];
    } else {
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                const int at = warp_first + (j * 32 + lane) * VEC + e;
                if (at < remaining) v[j].t[e] = in[base + at];
            }
    }
    // the element in front of the warp's chunk
    const bool has_left = base + warp_first > 0 && warp_first < remaining;
    T left = v[0].t[0];
    if (has_left) left = in[base + warp_first - 1];

    // keep bit e of vector j: element starts a new run.  The counts of two vectors share a word
    // (16 bits each: a warp holds at most 512 elements of one j).
    unsigned int keep[NV], packed[NV / 2];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        T before = shfl_value_up(v[j].t[VEC - 1]);
        if (lane == 0) before = left;
        left = shfl_value(v[j].t[VEC - 1], 31);
        unsigned int m = 0u;
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            const int at = warp_first + (j * 32 + lane) * VEC + e;
            const bool first = base == 0 && at == 0;
            if (at < remaining && (first || !SameValue<T>::eq(v[j].t[e], e == 0 ? before : v[j].t[e == 0 ? 0 : e - 1]))) m |= 1u << e;
        }
        keep[j] = m;
        if (j & 1) packed[j / 2] |= (unsigned int)__popc(m) << 16;
        else packed[j / 2] = (unsigned int)__popc(m);
    }
    unsigned int incl[NV / 2];
#pragma unroll
    for (int q = 0; q < NV / 2; ++q) incl[q] = packed[q];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
        for (int q = 0; q < NV / 2; ++q) {
            const unsigned int up = __shfl_up_sync(0xffffffffu, incl[q], d);
            if (lane >= d) incl[q] += up;
        }
    unsigned int local[NV];  // survivors of the warp in front of this lane's vector j
    unsigned int chunk = 0u;
#pragma unroll
    for (int q = 0; q < NV / 2; ++q) {
        const unsigned int total = __shfl_sync(0xffffffffu, incl[q], 31);
        const unsigned int excl = incl[q] - packed[q];
        local[2 * q] = chunk + (excl & 0xffffu);
        chunk += total & 0xffffu;
        local[2 * q + 1] = chunk + (excl >> 16);
        chunk += total >> 16;
    }
    if (lane == 31) warp_total[warp] = chunk;
    __syncthreads();
    const unsigned int wt = lane < WARPS ? warp_total[lane] : 0u;
    const unsigned int first_slot = __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
    const unsigned int aggregate = __reduce_add_sync(0xffffffffu, wt);
    // Survivors gather while the first warp, once it has told the tiles behind this one its count,
    // looks for its prefix.
    TileState<unsigned int> state(state_base, num_tiles);
    if (tid == 0) state.publish(tile, tile == 0 ? kInclusive : kAggregate, aggregate);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        unsigned int slot = first_slot + local[j];
#pragma unroll
        for (int e = 0; e < VEC; ++e)
            if ((keep[j] >> e) & 1u) survivors[slot++] = v[j].t[e];
    }
    if (warp == 0) {
        unsigned int prefix = 0u;
        if (tile > 0) {
            int look = tile - 1 - lane;  // 32 predecessors per round, nearest first
            bool gave_up = false;
            while (true) {
                unsigned int v = 0u;
                unsigned int flag = kInclusive;
                if (look >= 0) {
                    unsigned int spins = 0;
                    flag = state.poll(look, v);
                    while (flag == kInvalid) {
                        if (++spins > kMaxSpin) { gave_up = true; flag = kInclusive; v = 0u; break; }
                        __nanosleep(20);
                        flag = state.poll(look, v);
                    }
                }
                const unsigned int incl_mask = __ballot_sync(0xffffffffu, flag == kInclusive);
                const int nearest = incl_mask ? (__ffs(incl_mask) - 1) : 31;
                unsigned int contrib = lane <= nearest ? v : 0u;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) contrib += __shfl_down_sync(0xffffffffu, contrib, d);
                prefix += __shfl_sync(0xffffffffu, contrib, 0);
                if (incl_mask) break;
                look -= 32;
            }
            if (__any_sync(0xffffffffu, gave_up) && lane == 0) atomicExch(&hdr->wait_limit_hit, 1u);
            if (lane == 0) state.publish(tile, kInclusive, prefix + aggregate);
        }
        if (lane == 0) {
            s_prefix = prefix;
            if (tile == num_tiles - 1) *out_count = (long long)prefix + aggregate;
        }
    }
    __syncthreads();

    // where the runs begin
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        unsigned int slot = first_slot + local[j];
#pragma unroll
        for (int e = 0; e < VEC; ++e)
            if ((keep[j] >> e) & 1u) starts[(int64_t)s_prefix + slot++] = base + warp_first + (j * 32 + lane) * VEC + e;
    }
    T *to = kept + s_prefix;
    for (unsigned int i = tid; i < aggregate; i += kUniqueThreads) to[i] = survivors[i];
}

// ---- in place -------------------------------------------------------------------------------
// The words the tiles and the scanner exchange.
constexpr unsigned int kCounted = 0x80000000u;  // beside a tile's count of survivors
constexpr unsigned int kRead = 0x40000000u;     // likewise, set with release: the tile may be overwritten
static __host__ __device__ int64_t padded_tiles(int64_t tiles) { return (tiles + 3) / 4 * 4; }
static int64_t unique_word_bytes(int64_t tiles) { return padded_tiles(tiles) * (4 + 8); }

// A wait ran out: noted in the control block and, for a caller that reads the result from host memory,
// beside it.
__device__ __forceinline__ void report_wait_limit(TempHeader *hdr, long long *host_status) {
    atomicExch(&hdr->wait_limit_hit, 1u);
    if (host_status) *host_status = B200ALG_WAIT_LIMIT;
}

// One warp turns the tiles' counts into their prefixes (published as 2 * prefix + 1), four neighbouring
// tiles per lane.
__device__ __forceinline__ void scan_tile_counts(const unsigned int *counts, unsigned long long *prefixes, int num_tiles, TempHeader *hdr,
                                                 long long *host_status) {
    const int lane = threadIdx.x & 31;
    unsigned long long carry = 0ull;  // of the tiles before pos
    ScannerPolls limit;
    int pos = 0, done = 0;            // tiles before done have their prefixes
    while (done < num_tiles) {
        const int t = pos + 4 * lane;
        unsigned int c[4] = {kCounted, kCounted, kCounted, kCounted};
        if (t < num_tiles) {
            asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "l"(counts + t) : "memory");
#pragma unroll
            for (int q = 1; q < 4; ++q)
                if (t + q >= num_tiles) c[q] = kCounted;
        }
        int known = 0;  // of this lane's tiles, from the first one on
#pragma unroll
        for (int q = 0; q < 4; ++q) known += known == q && c[q] >= kCounted;
        const unsigned int partial = __ballot_sync(0xffffffffu, known < 4);
        const int first = partial ? __ffs((int)partial) - 1 : 32;  // the first lane that misses one
        const int upto = pos + 4 * first + (partial ? __shfl_sync(0xffffffffu, known, first) : 0);
        if (upto <= done) {
            if (!limit.again(done > 0, [](unsigned int ns) { __nanosleep(ns); })) {
                if (lane == 0) report_wait_limit(hdr, host_status);
                return;
            }
            continue;
        }
        limit.progress();
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] &= kRead - 1u;
        const unsigned int own = lane < first ? c[0] + c[1] + c[2] + c[3] : 0u;
        unsigned int incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned int up = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += up;
        }
        unsigned long long word = (carry + (incl - own)) * 2 + 1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (t + q < upto && t + q < num_tiles && t + q >= done) st_relaxed_u64(prefixes + t + q, word);
            word += 2ull * c[q];
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
        pos += 4 * first;
        done = upto;
    }
}

// Bound: HBM (every element read once, every survivor written once).  As in the pipelined scan, blocks
// hand their tiles' counts to a scanner warp (the first block to start) and do the next tile until
// the prefix has come; a tile waits in a ring in shared memory, where its survivors gather in the
// place its elements came to.  Tiles of 32 KB, three to a block, two blocks per SM: 5 * 10^7 uint32 of
// which a quarter is kept take 65 us (look-back in every block, one tile per block: 74 us); 2^27 of
// which one in fifty is kept 136 (157) us.
//
// The result goes over the input: a tile's survivors are stored at or below its own elements' places,
// over elements of at most two earlier tiles.  Those have been counted, hence read, long before the
// prefix is known, but that chain of relaxed words orders nothing.  So a block says of each of its
// tiles that it has been read (kRead beside the count, with release, after the barrier behind the
// reads), and two lanes of the warp that fetches a prefix look for that word of the two tiles (with
// acquire) before the block stores.  That is a trip to L2 more per tile; without it the two sizes above
// take 62.5 and 130 us.  (Release by the counting thread and fences in the scanner: 85 and 194 us;
// release by the counting thread and acquire by the fetching lanes: 77 and 167 us; looking for the words
// while the prefix is on its way, in 128 tiles at a time: 66 and 139 us.)
//
// The one element a tile reads outside its own range is the last one of the tile before.  A tile of
// which nothing moves is not stored at all, so that element is written only by tiles that have waited
// for its second reader, too: the second of the two tiles above.
constexpr int kRingStages = 3;
constexpr int kRingWorkers = 256, kRingVecs = 8;  // 512 threads of four vectors: 71 us
static_assert(kRingWorkers * kRingVecs * 16 == kUniqueTileBytes, "one size of tile");
constexpr int kRingStageBytes = kUniqueTileBytes + 128;  // the last 16 of the first 128 hold what precedes the tile
constexpr int kRingThreads = kRingWorkers + 64;
constexpr int kRingBlocks = 2;  // per SM
static __device__ __forceinline__ bool unique_block_any(bool p) {  // of the kRingWorkers threads that sort out the tiles
    unsigned int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"((unsigned int)p), "n"(kRingWorkers) : "memory");
    return any != 0u;
}

// Stores v at the shared address and moves it on when the bit is set; without a branch, which the
// compiler makes of it (three instructions instead of five).
template <typename T> __device__ __forceinline__ void put_if(unsigned int keep, unsigned int bit, unsigned int &at, T v) {
    if constexpr (sizeof(T) == 8) {
        unsigned long long bits;
        memcpy(&bits, &v, 8);
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.u32 p, t, 0;\n\t"
                     "@p st.shared.b64 [%0], %3;\n\t@p add.u32 %0, %0, 8;\n\t}" : "+r"(at) : "r"(keep), "r"(bit), "l"(bits) : "memory");
    } else if constexpr (sizeof(T) == 4) {
        unsigned int bits;
        memcpy(&bits, &v, 4);
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.u32 p, t, 0;\n\t"
                     "@p st.shared.b32 [%0], %3;\n\t@p add.u32 %0, %0, 4;\n\t}" : "+r"(at) : "r"(keep), "r"(bit), "r"(bits) : "memory");
    } else {
        unsigned short bits = 0;
        memcpy(&bits, &v, sizeof(T));
        if constexpr (sizeof(T) == 2)
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.u32 p, t, 0;\n\t"
                         "@p st.shared.b16 [%0], %3;\n\t@p add.u32 %0, %0, 2;\n\t}" : "+r"(at) : "r"(keep), "r"(bit), "h"(bits) : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.u32 p, t, 0;\n\t"
                         "@p st.shared.u8 [%0], %3;\n\t@p add.u32 %0, %0, 1;\n\t}" : "+r"(at) : "r"(keep), "r"(bit), "h"(bits) : "memory");
    }
}

template <typename T>
__global__ void __launch_bounds__(kRingThreads, kRingBlocks)
unique_in_place_kernel(T *data, int64_t n, long long *out_count, long long *host_status, TempHeader *hdr, unsigned int *counts, int num_tiles) {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int NV = kRingVecs;
    constexpr int TILE = VEC * NV * kRingWorkers;
    constexpr int WARPS = kRingWorkers / 32;
    constexpr int PER = VEC <= 4 ? 4 : 2, BITS = 32 / PER;
    static_assert(32 * VEC < 1 << BITS && NV % PER == 0, "a warp's count of one vector fits its bits");
    union Vec { uint4 u; T t[VEC]; __device__ Vec() {} };

    extern __shared__ __align__(128) unsigned char ring[];  // kRingStages x kRingStageBytes
    __shared__ __align__(8) unsigned long long full_bar[kRingStages];  // the tile's number is known, its elements have arrived
    __shared__ __align__(8) unsigned long long read_bar[kRingStages];  // the tile is in registers, its count is on its way
    __shared__ __align__(8) unsigned long long free_bar[kRingStages];  // every warp has stored its part of the survivors
    __shared__ __align__(8) unsigned long long base_bar[2];            // the tile's prefix is known
    __shared__ unsigned long long s_prefix[2];
    __shared__ unsigned int warp_total[2][WARPS];
    __shared__ int tile_of[kRingStages];
    __shared__ int s_role, s_failed;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long *prefixes = reinterpret_cast<unsigned long long *>(counts + padded_tiles(num_tiles));
    // Views off 16 bytes are loaded element by element when their turn comes: 81 instead of 65 us (5 * 10^7
    // uint32, a quarter kept), 165 instead of 85 for 10^8 bytes.
    auto bulk = [&](int tile) { return (int64_t)(tile + 1) * TILE <= n && ((uintptr_t)data & 15u) == 0; };
    auto stage_of = [&](int k) { return ring + k % kRingStages * kRingStageBytes + 128; };
    auto take_tile = [&](int k) {  // tiles are handed out in order
        const int st = k % kRingStages, tile = (int)atomicAdd(&hdr->reserved[0], 1u);
        tile_of[st] = tile;
        if (tile < num_tiles && bulk(tile)) {
            const int ahead = tile > 0 ? 16 : 0;
            mbar_expect_tx(&full_bar[st], kUniqueTileBytes + ahead);
            bulk_load(stage_of(k) - ahead, reinterpret_cast<const unsigned char *>(data + (int64_t)tile * TILE) - ahead, kUniqueTileBytes + ahead, &full_bar[st]);
        } else {
            mbar_arrive(&full_bar[st]);
        }
        return tile < num_tiles;
    };
    bool more = true;
    // Few tiles: one at the start, the next when it has arrived, so that every block gets some.
    const int share = num_tiles / (int)(gridDim.x - 1), at_once = share < 1 ? 1 : share < kRingStages ? share : kRingStages;
    if (tid == kRingWorkers) {
        s_failed = 0;
        s_role = (int)atomicAdd(&hdr->reserved[1], 1u);
        for (int st = 0; st < kRingStages; ++st) {
            mbar_init(&full_bar[st], 1u);
            mbar_init(&read_bar[st], 1u);
            mbar_init(&free_bar[st], WARPS);
        }
        for (int h = 0; h < 2; ++h) mbar_init(&base_bar[h], 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (s_role != 0)
            for (int k = 0; k < at_once && more; ++k) more = take_tile(k);
    }
    __syncthreads();
    if (s_role == 0) {
        if (warp == 0) scan_tile_counts(counts, prefixes, num_tiles, hdr, host_status);
        return;
    }
    unsigned int max_polls = kMaxBarrierPolls;  // a thread whose wait ran out does not wait as long again
    auto wait = [&](unsigned long long *bar, unsigned int parity) {
        if (mbar_wait(bar, parity, max_polls)) return true;
        max_polls = 1u;
        s_failed = 1;
        return false;
    };

    if (warp == WARPS) {  // keeps tiles coming, and tells the other blocks when they have been read
        if (lane == 0) {
            bool well = true;
            for (int k = at_once; k < kRingStages && more && well; ++k)
                if ((well = wait(&full_bar[0], 0u))) more = take_tile(k);
            for (int k = 0; well && tile_of[k % kRingStages] < num_tiles; ++k) {
                if (!wait(&read_bar[k % kRingStages], (unsigned int)(k / kRingStages) & 1u)) break;
                or_release_u32(counts + tile_of[k % kRingStages], kRead);
                if (k > 0 && more) {  // the tile before is stored next
                    if (!wait(&free_bar[(k - 1) % kRingStages], (unsigned int)((k - 1) / kRingStages) & 1u)) break;
                    more = take_tile(k - 1 + kRingStages);
                }
            }
        }
        __syncwarp();
    } else if (warp > WARPS) {  // fetches their prefixes
        if (lane < 2) {
            unsigned int max_spins = kMaxSpin;
            for (int k = 0;; ++k) {
                const bool arrived = wait(&full_bar[k % kRingStages], (unsigned int)(k / kRingStages) & 1u);
                if (__any_sync(3u, !arrived)) break;
                const int tile = tile_of[k % kRingStages];
                if (tile >= num_tiles) break;
                unsigned long long word = 1ull;
                unsigned int spins = 0;
                auto again = [&]() {
                    if (++spins <= max_spins) return true;
                    s_failed = 1;
                    max_spins = 1u;
                    return false;
                };
                while (tile > 0 && ((word = ld_relaxed_u64(prefixes + tile)) & 1ull) == 0 && again()) {}
                // the first of the tiles that the survivors go over, and the one behind it, have been read
                const int64_t over = (int64_t)(word >> 1) / TILE + lane;
                while (over < tile && (ld_acquire_u32(counts + over) & kRead) == 0 && again()) {}
                __syncwarp(3u);
                if (lane == 0) {
                    s_prefix[k & 1] = word >> 1;
                    mbar_arrive(&base_bar[k & 1]);
                }
            }
        }
        __syncwarp();
    } else {
        const int warp_first = warp * (NV * 32 * VEC);  // the warp's first element inside a tile
        unsigned int before_count = 0u;                 // survivors of the tile before
        int before = -1;                                // and its number
        for (int k = 0;; ++k) {
            const int st = k % kRingStages;
            const bool arrived = wait(&full_bar[st], (unsigned int)(k / kRingStages) & 1u);
            const int tile = arrived ? tile_of[st] : num_tiles;
            const bool work = tile < num_tiles;
            const int64_t base = (int64_t)tile * TILE;
            const int valid = n - base < TILE ? (int)(n - base) : TILE;
            T *stage = reinterpret_cast<T *>(stage_of(k));
            Vec v[NV];
            unsigned int keep[NV], local[NV];  // local: survivors of the warp in front of this lane's vector j
            if (work) {
                T left;  // the element in front of the warp's part
                if (bulk(tile)) {
                    const uint4 *src = reinterpret_cast<const uint4 *>(stage + warp_first) + lane;
#pragma unroll
                    for (int j = 0; j < NV; ++j) v[j].u = src[j * 32];
                    left = base + warp_first > 0 ? stage[warp_first - 1] : v[0].t[0];
                } else {
#pragma unroll
                    for (int j = 0; j < NV; ++j)
#pragma unroll
                        for (int e = 0; e < VEC; ++e) {
                            const int at = warp_first + (j * 32 + lane) * VEC + e;
                            if (at < valid) v[j].t[e] = data[base + at];
                        }
                    left = base + warp_first > 0 && warp_first < valid ? data[base + warp_first - 1] : v[0].t[0];
                }
                // keep bit e of vector j: element starts a new run.  The counts of several vectors share a
                // word: a warp holds 32 * VEC elements of one j.
                unsigned int packed[NV / PER], incl[NV / PER];
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    const T around = shfl_value(v[j].t[VEC - 1], (lane + 31) & 31);  // (lane 0: what precedes it in j + 1)
                    const T in_front = lane == 0 ? left : around;
                    left = around;
                    unsigned int m = 0u;
#pragma unroll
                    for (int e = 0; e < VEC; ++e)
                        if (!SameValue<T>::eq(v[j].t[e], e == 0 ? in_front : v[j].t[e == 0 ? 0 : e - 1])) m |= 1u << e;
                    if (j == 0 && base == 0 && tid == 0) m |= 1u;  // the very first element
                    if (valid < TILE) {
                        const int there = valid - (warp_first + (j * 32 + lane) * VEC);  // of this vector
                        m &= there <= 0 ? 0u : there < VEC ? (1u << there) - 1u : ~0u;
                    }
                    keep[j] = m;
                    if (j % PER) packed[j / PER] |= (unsigned int)__popc(m) << BITS * (j % PER);
                    else packed[j / PER] = (unsigned int)__popc(m);
                }
#pragma unroll
                for (int q = 0; q < NV / PER; ++q) incl[q] = packed[q];
#pragma unroll
                for (int d = 1; d < 32; d <<= 1)
#pragma unroll
                    for (int q = 0; q < NV / PER; ++q) {
                        const unsigned int up = __shfl_up_sync(0xffffffffu, incl[q], d);
                        if (lane >= d) incl[q] += up;
                    }
                unsigned int chunk = 0u;
#pragma unroll
                for (int q = 0; q < NV / PER; ++q) {
                    const unsigned int total = __shfl_sync(0xffffffffu, incl[q], 31);
                    const unsigned int excl = incl[q] - packed[q];
#pragma unroll
                    for (int r = 0; r < PER; ++r) {
                        local[q * PER + r] = chunk + (excl >> BITS * r & ((1u << BITS) - 1u));
                        chunk += total >> BITS * r & ((1u << BITS) - 1u);
                    }
                }
                if (lane == 31) warp_total[k & 1][warp] = chunk;
            }
            // the warps' counts are there, the tile is in registers, the tile before has its survivors together
            if (unique_block_any(!arrived)) break;
            unsigned int count = 0u;
            if (work) {
                const unsigned int wt = lane < WARPS ? warp_total[k & 1][lane] : 0u;
                const unsigned int first_slot = __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
                count = __reduce_add_sync(0xffffffffu, wt);
                if (tid == 0) {
                    st_relaxed_u32(counts + tile, count | kCounted);
                    mbar_arrive(&read_bar[st]);
                }
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    unsigned int at = smem_addr(stage) + (first_slot + local[j]) * (unsigned int)sizeof(T);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) put_if<T>(keep[j], 1u << e, at, v[j].t[e]);
                }
            }
            if (before >= 0) {
                const int q = k - 1;
                if (wait(&base_bar[q & 1], (unsigned int)(q >> 1) & 1u)) {
                    const int64_t prefix = (int64_t)s_prefix[q & 1];
                    if (before == num_tiles - 1 && tid == 0) *out_count = prefix + before_count;
                    const T *survivors = reinterpret_cast<const T *>(stage_of(q));
                    T *to = data + prefix;
                    const unsigned int stored = prefix + before_count == (int64_t)(before + 1) * TILE ? 0u : before_count;  // 0: nothing has moved
#pragma unroll 4
                    for (unsigned int i = tid; i < stored; i += kRingWorkers) to[i] = survivors[i];
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // a copy may come into these places next
                __syncwarp();
                if (lane == 0) mbar_arrive(&free_bar[q % kRingStages]);
            }
            if (!work) break;
            before = tile;
            before_count = count;
        }
    }

    // A wait that ran out is reported; copies that may still be in flight are given one more bounded
    // wait so that the block does not retire underneath them.
    __syncthreads();
    if (s_failed && tid == kRingWorkers) {
        report_wait_limit(hdr, host_status);
        for (int st = 0; st < kRingStages; ++st) {
            mbar_wait(&full_bar[st], 0u);
            mbar_wait(&full_bar[st], 1u);
        }
    }
}

// lengths[r] = distance from the start of run r to the start of the next run (or to n).
__global__ void __launch_bounds__(256)
run_lengths_kernel(const long long *starts, const long long *count, long long n, long long *lengths) {
    const long long m = *count;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += step)
        lengths[r] = (r + 1 < m ? starts[r + 1] : n) - starts[r];
}

struct UniqueLayout {
    int64_t tiles, off_state, total;
};

static UniqueLayout unique_layout(int elem_bytes, int64_t n) {
    UniqueLayout L;
    L.tiles = ceil_div((n < 1 ? 1 : n) * elem_bytes, kUniqueTileBytes);
    L.off_state = sizeof(TempHeader);
    L.total = L.off_state + round_up(L.tiles * kDescStride, 256);
    return L;
}

template <typename T>
static int run_unique(cudaStream_t s, void *data, int64_t n, void *out_count, long long *host_status, void *temp, const UniqueLayout &L) {
    char *t = (char *)temp;
    auto kernel = unique_in_place_kernel<T>;
    constexpr int ring_bytes = kRingStages * kRingStageBytes;
    static ContextCache<int> cache;  // per kernel instantiation and CUDA context
    int set = 0;
    if (!cache.find(&set)) {
        B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ring_bytes));
        cache.store(1);
    }
    const int64_t most = (int64_t)kRingBlocks * sm_count();
    const int blocks = (int)(L.tiles < most ? L.tiles + 1 : most);  // one of them the scanner
    B200ALG_CUDA_TRY(cudaMemsetAsync(temp, 0, (size_t)(L.off_state + unique_word_bytes(L.tiles)), s));
    kernel<<<blocks, kRingThreads, ring_bytes, s>>>((T *)data, n, (long long *)out_count, host_status, (TempHeader *)temp, (unsigned int *)(t + L.off_state),
                                                (int)L.tiles);
    B200ALG_LAUNCH_CHECK();
    return B200ALG_OK;
}

// Run-length encoding: the same selection, with the survivors written to the caller's array
// and the run starts to scratch, from which the lengths follow.
struct RunLengthLayout {
    int64_t tiles, off_state, off_starts, total;
};
static RunLengthLayout run_length_layout(int elem_bytes, int64_t n) {
    RunLengthLayout L;
    L.tiles = ceil_div((n < 1 ? 1 : n) * elem_bytes, kUniqueTileBytes);
    L.off_state = sizeof(TempHeader);
    L.off_starts = L.off_state + round_up(L.tiles * kDescStride, 256);
    L.total = L.off_starts + round_up((n < 1 ? 1 : n) * 8, 256);
    return L;
}

template <typename T>
static int run_rle(cudaStream_t s, const void *data, int64_t n, void *values, void *lengths, void *num_runs, void *temp,
                   const RunLengthLayout &L) {
    char *t = (char *)temp;
    B200ALG_CUDA_TRY(cudaMemsetAsync(temp, 0, (size_t)L.off_starts, s));
    unique_select_kernel<T><<<(int)L.tiles, kUniqueThreads, 0, s>>>((const T *)data, n, (T *)values, (long long *)(t + L.off_starts),
                                                                  (long long *)num_runs, (TempHeader *)temp, t + L.off_state,
                                                                  (int)L.tiles);
    B200ALG_LAUNCH_CHECK();
    int64_t want = ceil_div(n, 256 * 8);
    const int64_t cap = (int64_t)sm_count() * 8;
    const int blocks = (int)(want < 1 ? 1 : (want > cap ? cap : want));
    run_lengths_kernel<<<blocks, 256, 0, s>>>((const long long *)(t + L.off_starts), (const long long *)num_runs, (long long)n,
                                              (long long *)lengths);
    B200ALG_LAUNCH_CHECK();
    return B200ALG_OK;
}

}  // namespace b200alg

using namespace b200alg;

extern "C" int b200alg_run_length_encode_temp_bytes(int dtype, int64_t n, int64_t *out_bytes) {
    if (!out_bytes || n < 0) return B200ALG_INVALID_ARGUMENT;
    if (dtype_bytes(dtype) == 0) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    *out_bytes = run_length_layout(dtype_bytes(dtype), n).total;
    return B200ALG_OK;
}

extern "C" int b200alg_run_length_encode(void *stream, const void *data, int64_t n, int dtype, void *values, int64_t *lengths,
                                         int64_t *num_runs, void *temp, int64_t temp_bytes) {
    if (!num_runs || n < 0) return B200ALG_INVALID_ARGUMENT;
    if ((uintptr_t)num_runs % 8) return B200ALG_MISALIGNED;
    if (n == 0) {
        B200ALG_CUDA_TRY(cudaMemsetAsync(num_runs, 0, 8, (cudaStream_t)stream));
        return B200ALG_OK;
    }
    if (!data || !values || !lengths || !temp) return B200ALG_INVALID_ARGUMENT;
    const int es = dtype_bytes(dtype);
    if (es == 0) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    if (((uintptr_t)data % es) || ((uintptr_t)values % es) || ((uintptr_t)lengths % 8) || ((uintptr_t)temp % 256)) return B200ALG_MISALIGNED;
    const RunLengthLayout L = run_length_layout(dtype_bytes(dtype), n);
    if (temp_bytes < L.total) return B200ALG_TEMP_TOO_SMALL;
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
    case B200ALG_I8: case B200ALG_U8: return run_rle<uint8_t>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_I16: case B200ALG_U16: return run_rle<uint16_t>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_I32: case B200ALG_U32: return run_rle<uint32_t>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_I64: case B200ALG_U64: return run_rle<uint64_t>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_F16: return run_rle<__half>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_F32: return run_rle<float>(s, data, n, values, lengths, num_runs, temp, L);
    case B200ALG_F64: return run_rle<double>(s, data, n, values, lengths, num_runs, temp, L);
    }
    return B200ALG_UNSUPPORTED;
}

extern "C" int b200alg_unique_temp_bytes(int dtype, int64_t n, int64_t *out_bytes) {
    if (!out_bytes || n < 0) return B200ALG_INVALID_ARGUMENT;
    const int es = dtype_bytes(dtype);
    if (es == 0) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    *out_bytes = unique_layout(es, n).total;
    return B200ALG_OK;
}

static int unique(void *stream, void *data, int64_t n, int dtype, void *out_count, long long *host_status, void *temp, int64_t temp_bytes) {
    // Argument checks mirror CreateUnique's (UniqueExtensions.cs:150-172).
    if (!out_count || n < 0) return B200ALG_INVALID_ARGUMENT;
    if ((uintptr_t)out_count % 8) return B200ALG_MISALIGNED;
    if (n == 0) {  // an empty view has no address
        B200ALG_CUDA_TRY(cudaMemsetAsync(out_count, 0, 8, (cudaStream_t)stream));
        return B200ALG_OK;
    }
    if (!data || !temp) return B200ALG_INVALID_ARGUMENT;
    const int es = dtype_bytes(dtype);
    if (es == 0) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    if (((uintptr_t)data % es) || ((uintptr_t)out_count % 8) || ((uintptr_t)temp % 256)) return B200ALG_MISALIGNED;
    const UniqueLayout L = unique_layout(es, n);
    if (temp_bytes < L.total) return B200ALG_TEMP_TOO_SMALL;
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
    case B200ALG_I8: case B200ALG_U8: return run_unique<uint8_t>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_I16: case B200ALG_U16: return run_unique<uint16_t>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_I32: case B200ALG_U32: return run_unique<uint32_t>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_I64: case B200ALG_U64: return run_unique<uint64_t>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_F16: return run_unique<__half>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_F32: return run_unique<float>(s, data, n, out_count, host_status, temp, L);
    case B200ALG_F64: return run_unique<double>(s, data, n, out_count, host_status, temp, L);
    }
    return B200ALG_UNSUPPORTED;
}

extern "C" int b200alg_unique(void *stream, void *data, int64_t n, int dtype, void *out_count, void *temp, int64_t temp_bytes) {
    return unique(stream, data, n, dtype, out_count, nullptr, temp, temp_bytes);
}

extern "C" int b200alg_unique_to_host(void *stream, void *data, int64_t n, int dtype, int64_t *host_out, void *temp, int64_t temp_bytes) {
    return unique(stream, data, n, dtype, host_out, host_out ? (long long *)host_out + 1 : nullptr, temp, temp_bytes);
}
