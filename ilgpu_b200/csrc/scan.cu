// Scan: every tile is read once and written once; the tiles' prefixes come from a scanner warp that
// follows their totals (dense views) or from decoupled look-back (all others).
// Replaces SinglePassScanKernel + its tile helpers (ScanExtensions.cs:284-388, :530-706),
// whose groups hand one running value down a strictly serial chain
// (SequentialGroupExecutor.cs:58-77) and read the input twice.  Here every tile is read
// once and written once (8 B / element for 4-byte types).
#include "common.cuh"
#include "lookback.cuh"

#include <cooperative_groups.h>

namespace b200alg {

namespace cg = cooperative_groups;

constexpr int kScanThreads = 256;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanVecPerThread = 8;  // 8 x 16 bytes per thread -> 32 KB per tile

constexpr int kScanMinTileElems = 2 * kScanVecPerThread * kScanThreads;  // tile of an 8-byte type

// General variant (strided or unaligned views): one tile per block, handed out by an atomic
// ticket.  Thread t scans ITEMS consecutive elements of the tile, but global memory is touched
// warp-striped (consecutive lanes, consecutive elements: for a strided view, addresses one
// stride apart instead of ITEMS strides apart) and the warp transposes its chunk through
// shared memory, padded by one slot per 32 so that both access patterns are conflict-free.
template <typename T, int OP, bool INCLUSIVE>
__global__ void __launch_bounds__(kScanThreads)
scan_kernel(const T *in, int64_t in_stride, T *out, int64_t out_stride, int64_t n, const T *carry_in,
            TempHeader *hdr, void *state_base, int num_tiles) {
    using O = Op<T, OP>;
    constexpr int VEC = 16 / sizeof(T);
    constexpr int ITEMS = VEC * kScanVecPerThread;
    constexpr int TILE = ITEMS * kScanThreads;
    struct Items { T t[ITEMS]; };

    __shared__ T exchange[kScanWarps][32 * ITEMS + ITEMS];
    __shared__ T warp_total[kScanWarps];
    __shared__ T warp_excl[kScanWarps];
    __shared__ T s_prefix;
    __shared__ int s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto slot = [](int e) { return e + (e >> 5); };
    grid_dependency_wait();  // the descriptors and the ticket counter have been cleared
    if (tid == 0) s_tile = (int)atomicAdd(&hdr->reserved[0], 1u);
    __syncthreads();
    const int tile = s_tile;
    const int64_t base = (int64_t)tile * TILE;
    const int64_t remaining = n - base;

    Items it;
    const int64_t warp_first = (int64_t)warp * (32 * ITEMS);  // first element of the warp's chunk inside the tile
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int e = j * 32 + lane;
        const int64_t idx = warp_first + e;
        exchange[warp][slot(e)] = idx < remaining ? in[(base + idx) * in_stride] : O::identity();
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) it.t[k] = exchange[warp][slot(lane * ITEMS + k)];

    // Thread total -> warp scan -> block scan.
    T tsum = it.t[0];
#pragma unroll
    for (int k = 1; k < ITEMS; ++k) tsum = O::apply(tsum, it.t[k]);
    T wincl = tsum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T up = shfl_up(wincl, d);
        if (lane >= d) wincl = O::apply(up, wincl);
    }
    T lane_excl = shfl_up(wincl, 1);
    if (lane == 0) lane_excl = O::identity();
    if (lane == 31) warp_total[warp] = wincl;
    __syncthreads();

    if (warp == 0) {
        T wt = lane < kScanWarps ? warp_total[lane] : O::identity();
        T wi = wt;
#pragma unroll
        for (int d = 1; d < kScanWarps; d <<= 1) {
            T up = shfl_up(wi, d);
            if (lane >= d) wi = O::apply(up, wi);
        }
        T we = shfl_up(wi, 1);
        if (lane == 0) we = O::identity();
        if (lane < kScanWarps) warp_excl[lane] = we;
        const T aggregate = shfl_idx(wi, kScanWarps - 1);

        TileState<T> state(state_base, num_tiles);
        T prefix;
        if (tile == 0) {
            prefix = carry_in ? *carry_in : O::identity();
            if (lane == 0) state.publish(0, kInclusive, O::apply(prefix, aggregate));
        } else {
            if (lane == 0) state.publish(tile, kAggregate, aggregate);
            // Decoupled look-back: 32 predecessors per round, nearest first.
            prefix = O::identity();
            int look = tile - 1 - lane;
            bool gave_up = false;
            while (true) {
                T v = O::identity();
                unsigned int flag = kInclusive;  // tiles before tile 0 act as "inclusive identity"
                if (look >= 0) {
                    unsigned int spins = 0;
                    flag = state.poll(look, v);
                    while (flag == kInvalid) {
                        if (++spins > kMaxSpin) { gave_up = true; flag = kInclusive; v = O::identity(); break; }
                        __nanosleep(20);
                        flag = state.poll(look, v);
                    }
                }
                const unsigned int incl_mask = __ballot_sync(0xffffffffu, flag == kInclusive);
                // Lanes beyond the nearest tile with an inclusive prefix do not contribute.
                const int first = incl_mask ? (__ffs(incl_mask) - 1) : 31;
                T contrib = lane <= first ? v : O::identity();
                // In-order fold: lane 0 is the nearest predecessor, so fold from far to near.
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    T dn = shfl_down(contrib, d);
                    if (lane + d < 32) contrib = O::apply(dn, contrib);
                }
                const T window = shfl_idx(contrib, 0);
                prefix = O::apply(window, prefix);
                if (incl_mask) break;
                look -= 32;
            }
            if (__any_sync(0xffffffffu, gave_up) && lane == 0) atomicExch(&hdr->wait_limit_hit, 1u);
            if (lane == 0) state.publish(tile, kInclusive, O::apply(prefix, aggregate));
        }
        if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();

    T running = O::apply(s_prefix, O::apply(warp_excl[warp], lane_excl));
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const T x = it.t[k];
        if (INCLUSIVE) {
            running = O::apply(running, x);
            it.t[k] = running;
        } else {
            it.t[k] = running;
            running = O::apply(running, x);
        }
    }

    __syncwarp();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) exchange[warp][slot(lane * ITEMS + k)] = it.t[k];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int e = j * 32 + lane;
        const int64_t idx = warp_first + e;
        if (idx < remaining) out[(base + idx) * out_stride] = exchange[warp][slot(e)];
    }
}

// Clears the control block and the tile descriptors a scan is about to use.  The scan kernel
// is launched as a programmatic dependent of this one, so its blocks are already resident
// (barriers initialised) when the last descriptor has been cleared.
__global__ void __launch_bounds__(256) scan_clear_kernel(uint4 *words, int64_t count) {
    grid_dependency_release();
    const int64_t step = (int64_t)gridDim.x * 256;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < count; i += step) words[i] = make_uint4(0u, 0u, 0u, 0u);
}

// ---- pipelined variant for dense views that are aligned alike ---------------------------
// Persistent blocks take tiles round-robin (tile = blockIdx.x + k * (gridDim.x - 1)); the last block is
// the scanner, one warp that reads the tiles' totals as they appear and publishes the tiles' prefixes.
// Blocks wait for one another, so every block of the grid has to be resident at the same time: the
// kernel is launched cooperatively, which makes the driver guarantee exactly that (or refuse the
// launch, in which case the ticketed kernel above runs instead).  Handing the tiles out by an atomic
// ticket, as the general kernel does, needs no such guarantee but measured 2.5 to 3 times slower on
// long inputs, whatever the prefetch distance.
//
// A prefix takes several trips through an L2 that is busy with the tiles themselves, some 5000 cycles.
// They pass while the block works on the tile before and the tile after: a tile is looked at twice,
// first for its total, which is handed to the scanner, and one tile later, when its prefix has come,
// to be scanned and stored.  In between it stays in a ring of kPipeStages tiles in shared memory, into
// which bulk copies (TMA) bring the tiles ahead.  Eight warps do that; one more hands out the totals
// and issues the copies, one fetches the prefixes; they meet only in mbarriers.
//
// Bound by DRAM: 2^30 floats take 1304 us (6590 GB/s) where look-back in every block, with the tile held
// in registers meanwhile, took 1490; 2^28 int64 672 instead of 900 us, 2^24 int32 29.7 instead of
// 33.4 us.  Tiles of 32 KB and two blocks per SM: the scanner manages a tile every 18 cycles or so,
// which tiles of 24 KB (1357 us) and 16 KB (1791 us) outrun; one block of 512 threads with 64 KB tiles
// 1330 us, a fourth stage of 24 KB 1399 us.
//
// in and out start on 16 bytes; a view that does not begins with `lead` elements that belong to
// whatever is in front of it, read as Identity and not stored.
constexpr int kPipeStages = 3;
constexpr int kPipeVecs = 8;
constexpr int kPipeTileBytes = kScanThreads * kPipeVecs * 16;
constexpr int kPipeThreads = kScanThreads + 64;
constexpr int kPrefixRows = 4;  // rows of 32 tiles a scanner round looks at (2 and 8: 6 and 10 % slower)

// The words the tiles of the pipelined scan and its scanner exchange: two dense arrays, the tiles' totals
// and the tiles' prefixes.
template <typename T> struct TileWords {
    static constexpr int kBytes = 2 * sizeof(T);
    static_assert(2 * kBytes <= kDescStride, "fits where the general kernel has its records");
    TileState<T> totals, prefixes;
    __device__ TileWords(void *base, int tiles)
        : totals(base, tiles, kBytes), prefixes((unsigned char *)base + (size_t)(tiles + 1) / 2 * 2 * kBytes, tiles, kBytes) {}
    static __host__ __device__ int64_t vectors(int tiles) { return (int64_t)((tiles + 1) / 2) * 2 * 2 * kBytes / 16; }
};

// One warp turns the tiles' totals into their prefixes, kPrefixRows * 32 tiles at a time.
template <typename T, int OP>
__device__ __forceinline__ void scan_totals(TileWords<T> words, const T *carry_in, int num_tiles, TempHeader *hdr) {
    using O = Op<T, OP>;
    const int lane = threadIdx.x & 31;
    T carry = carry_in ? *carry_in : O::identity();
    unsigned int spins = 0;
    for (int pos = 0; pos < num_tiles;) {
        T own[kPrefixRows];
        unsigned int flag[kPrefixRows];
#pragma unroll
        for (int m = 0; m < kPrefixRows; ++m) {
            const int t = pos + m * 32 + lane;
            flag[m] = kInvalid;
            own[m] = O::identity();
            if (t < num_tiles) flag[m] = words.totals.poll(t, own[m]);
        }
        int ready = 0;  // totals that are there, from the first one on
#pragma unroll
        for (int m = 0; m < kPrefixRows; ++m) {
            const unsigned int missing = __ballot_sync(0xffffffffu, flag[m] == kInvalid);
            if (ready == m * 32) ready += missing ? __ffs((int)missing) - 1 : 32;
        }
        if (ready == 0) {
            if (++spins > kMaxSpin) {
                if (lane == 0) atomicExch(&hdr->wait_limit_hit, 1u);
                return;
            }
            continue;
        }
        spins = 0;
        T incl[kPrefixRows];
#pragma unroll
        for (int m = 0; m < kPrefixRows; ++m) incl[m] = m * 32 + lane < ready ? own[m] : O::identity();
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
            for (int m = 0; m < kPrefixRows; ++m) {
                const T up = shfl_up(incl[m], d);
                if (lane >= d) incl[m] = O::apply(up, incl[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < kPrefixRows; ++m) {
            T ex = shfl_up(incl[m], 1);
            if (lane == 0) ex = O::identity();
            if (m * 32 + lane < ready) words.prefixes.publish(pos + m * 32 + lane, kInclusive, O::apply(carry, ex));
            carry = O::apply(carry, shfl_idx(incl[m], 31));
        }
        pos += ready;
    }
}

template <typename T, int OP, bool INCLUSIVE, bool LEAD>
__global__ void __launch_bounds__(kPipeThreads, 2)
scan_pipeline_kernel(const T *in, T *out, int64_t n, int lead_arg, const T *carry_in, TempHeader *hdr, void *state_base, int num_tiles) {
    using O = Op<T, OP>;
    constexpr int VEC = 16 / sizeof(T);
    constexpr int NV = kPipeVecs;
    constexpr int TILE = VEC * NV * kScanThreads;
    union Vec { uint4 u; T t[VEC]; };

    extern __shared__ __align__(128) unsigned char ring[];  // kPipeStages x kPipeTileBytes
    __shared__ __align__(8) unsigned long long full_bar[kPipeStages];  // the copy of a tile has arrived
    __shared__ __align__(8) unsigned long long free_bar[kPipeStages];  // every warp has taken its part of a tile
    __shared__ __align__(8) unsigned long long totals_bar[2];          // every warp has its total of a tile
    __shared__ __align__(8) unsigned long long base_bar[2];            // what precedes each warp's part is known
    __shared__ T totals[2][kScanWarps];
    __shared__ T bases[2][kScanWarps];
    __shared__ int s_failed;  // a wait ran out

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (LEAD is a template parameter because the extra register costs aligned views 5 %)
    const int lead = LEAD ? lead_arg : 0;
    const int full_tiles = (int)(n / TILE);          // tiles below this index are complete,
    constexpr int first_full = LEAD ? 1 : 0;         // from this one on
    const int G = (int)gridDim.x - 1;                // the last block is the scanner
    const bool scanner = (int)blockIdx.x == G;
    const int my_tiles = scanner ? 0 : (num_tiles - (int)blockIdx.x + G - 1) / G;
    auto tile_of = [&](int k) { return (int)blockIdx.x + k * G; };
    auto is_full = [&](int tile) { return tile >= first_full && tile < full_tiles; };
    auto stage_in = [&](int k) {
        const int st = k % kPipeStages;
        mbar_expect_tx(&full_bar[st], kPipeTileBytes);
        bulk_load(ring + st * kPipeTileBytes, in + (int64_t)tile_of(k) * TILE, kPipeTileBytes, &full_bar[st]);
    };
    if (tid == kScanThreads) {
        s_failed = 0;
        for (int st = 0; st < kPipeStages; ++st) {
            mbar_init(&full_bar[st], 1u);
            mbar_init(&free_bar[st], kScanWarps);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(&totals_bar[h], kScanWarps);
            mbar_init(&base_bar[h], 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int k = 0; k < kPipeStages && k < my_tiles; ++k)
            if (is_full(tile_of(k))) stage_in(k);
    }
    // The words have to be cleared before anybody publishes (while the first tiles are on their way).
    if (blockIdx.x == 0 && tid == 0) hdr->wait_limit_hit = 0u;
    for (int64_t i = (int64_t)blockIdx.x * kPipeThreads + tid; i < TileWords<T>::vectors(num_tiles); i += (int64_t)gridDim.x * kPipeThreads)
        reinterpret_cast<uint4 *>(state_base)[i] = make_uint4(0u, 0u, 0u, 0u);
    cg::this_grid().sync();
    TileWords<T> words(state_base, num_tiles);
    if (scanner) {
        if (warp == 0) scan_totals<T, OP>(words, carry_in, num_tiles, hdr);
        return;
    }
    unsigned int max_polls = kMaxBarrierPolls;  // a thread whose wait ran out does not wait as long again
    auto wait = [&](unsigned long long *bar, unsigned int parity) {
        if (mbar_wait(bar, parity, max_polls)) return true;
        max_polls = 1u;
        s_failed = 1;
        return false;
    };

    if (warp == kScanWarps) {  // hands the tiles' totals to the scanner and keeps copies coming
        for (int k = 0; k < my_tiles; ++k) {
            wait(&totals_bar[k & 1], (unsigned int)(k >> 1) & 1u);
            T total = lane < kScanWarps ? totals[k & 1][lane] : O::identity();
#pragma unroll
            for (int d = kScanWarps / 2; d > 0; d >>= 1) total = O::apply(total, shfl_down(total, d));
            if (lane == 0) {
                words.totals.publish(tile_of(k), kAggregate, total);
                const int next = k + kPipeStages - 1;
                if (k >= 1 && next < my_tiles && is_full(tile_of(next))) {
                    wait(&free_bar[(k - 1) % kPipeStages], (unsigned int)((k - 1) / kPipeStages) & 1u);
                    stage_in(next);
                }
            }
            __syncwarp();
        }
    } else if (warp > kScanWarps) {  // fetches the tiles' prefixes
        unsigned int max_spins = kMaxSpin;
        for (int k = 0; k < my_tiles; ++k) {
            wait(&totals_bar[k & 1], (unsigned int)(k >> 1) & 1u);
            T sum = lane < kScanWarps ? totals[k & 1][lane] : O::identity();
#pragma unroll
            for (int d = 1; d < kScanWarps; d <<= 1) {
                const T up = shfl_up(sum, d);
                if (lane >= d) sum = O::apply(up, sum);
            }
            T ahead = shfl_up(sum, 1);
            if (lane == 0) ahead = O::identity();
            T prefix = O::identity();
            if (lane == 0) {
                unsigned int spins = 0;
                while (words.prefixes.poll(tile_of(k), prefix) == kInvalid) {
                    if (++spins > max_spins) {
                        atomicExch(&hdr->wait_limit_hit, 1u);
                        max_spins = 1u;
                        prefix = O::identity();
                        break;
                    }
                }
            }
            prefix = shfl_idx(prefix, 0);
            if (lane < kScanWarps) bases[k & 1][lane] = O::apply(prefix, ahead);
            __syncwarp();
            if (lane == 0) mbar_arrive(&base_bar[k & 1]);
        }
    } else {
        // Vector j of lane l covers elements (warp*32*NV + j*32 + l) * VEC ... + VEC of the tile.
        unsigned int phase = 0u;  // bit st = parity of the next completion of stage st's copy
        for (int k = 0; k <= my_tiles; ++k) {
            if (k < my_tiles) {  // this warp's total of tile k
                const int st = k % kPipeStages;
                const int64_t base = (int64_t)tile_of(k) * TILE;
                uint4 *slot = reinterpret_cast<uint4 *>(ring + st * kPipeTileBytes) + warp * (32 * NV) + lane;
                bool staged = is_full(tile_of(k));
                if (staged) {
                    staged = wait(&full_bar[st], (phase >> st) & 1u);
                    phase ^= 1u << st;
                }
                T total = O::identity();
                if (staged) {
                    Vec v[NV];
#pragma unroll
                    for (int j = 0; j < NV; ++j) v[j].u = slot[j * 32];
#pragma unroll
                    for (int j = 0; j < NV; ++j)
#pragma unroll
                        for (int e = 0; e < VEC; ++e) total = O::apply(total, v[j].t[e]);
                } else {
                    for (int j = 0; j < NV; ++j) {
                        Vec v;
#pragma unroll
                        for (int e = 0; e < VEC; ++e) {
                            const int64_t idx = base + (int64_t)(warp * (32 * NV) + j * 32 + lane) * VEC + e;
                            v.t[e] = idx >= lead && idx < n ? in[idx] : O::identity();
                            total = O::apply(total, v.t[e]);
                        }
                        slot[j * 32] = v.u;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (a copy may come into these slots next)
                }
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) total = O::apply(total, shfl_down(total, d));
                if (lane == 0) {
                    totals[k & 1][warp] = total;
                    mbar_arrive(&totals_bar[k & 1]);
                }
            }
            if (k == 0) continue;

            // tile k - 1: scan and store
            const int q = k - 1, st = q % kPipeStages;
            const int64_t base = (int64_t)tile_of(q) * TILE;
            const uint4 *slot = reinterpret_cast<const uint4 *>(ring + st * kPipeTileBytes) + warp * (32 * NV) + lane;
            Vec v[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) v[j].u = slot[j * 32];
            // inclusive scan inside each vector, then NV interleaved warp scans of the vector totals
            T w[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) {
#pragma unroll
                for (int e = 1; e < VEC; ++e) v[j].t[e] = O::apply(v[j].t[e - 1], v[j].t[e]);
                w[j] = v[j].t[VEC - 1];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&free_bar[st]);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    const T up = shfl_up(w[j], d);
                    if (lane >= d) w[j] = O::apply(up, w[j]);
                }
            }
            T before[NV];  // fold of everything in the warp's part that precedes vector j of this lane
            T chunk = O::identity();
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                T ex = shfl_up(w[j], 1);
                if (lane == 0) ex = O::identity();
                before[j] = O::apply(chunk, ex);
                chunk = O::apply(chunk, shfl_idx(w[j], 31));
            }
            wait(&base_bar[q & 1], (unsigned int)(q >> 1) & 1u);
            const T warp_base = bases[q & 1][warp];
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const T p = O::apply(warp_base, before[j]);
                if (INCLUSIVE) {
#pragma unroll
                    for (int e = 0; e < VEC; ++e) v[j].t[e] = O::apply(p, v[j].t[e]);
                } else {
#pragma unroll
                    for (int e = VEC - 1; e > 0; --e) v[j].t[e] = O::apply(p, v[j].t[e - 1]);
                    v[j].t[0] = p;
                }
            }
            if (is_full(tile_of(q))) {
                uint4 *dst = reinterpret_cast<uint4 *>(out + base) + warp * (32 * NV) + lane;
#pragma unroll
                for (int j = 0; j < NV; ++j) __stcs(dst + j * 32, v[j].u);
            } else {
#pragma unroll
                for (int j = 0; j < NV; ++j)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) {
                        const int64_t idx = base + (int64_t)(warp * (32 * NV) + j * 32 + lane) * VEC + e;
                        if (idx >= lead && idx < n) out[idx] = v[j].t[e];
                    }
            }
        }
    }

    // A wait that ran out is reported; copies that may still be in flight are given one more bounded
    // wait so that the block does not retire underneath them.
    __syncthreads();
    if (s_failed && tid == kScanThreads) {
        atomicExch(&hdr->wait_limit_hit, 1u);
        for (int st = 0; st < kPipeStages; ++st) {
            mbar_wait(&full_bar[st], 0u);
            mbar_wait(&full_bar[st], 1u);
        }
    }
}

// ---- short inputs: one block or one cluster ----------------------------------------------
// Every thread scans kShortItems neighbouring elements; the blocks of a cluster hand their totals on
// through distributed shared memory.  One launch, no descriptors to clear.  (As for the pipelined
// variant, a view that does not start on 16 bytes is scanned from the boundary in front of it.)
constexpr int kShortThreads = 1024, kShortItems = 8, kShortCluster = 8;
constexpr int kShortTile = kShortThreads * kShortItems;
template <typename T, int OP, bool INCLUSIVE>
__global__ void __launch_bounds__(kShortThreads)
scan_short_kernel(const T *in, int64_t in_stride, T *out, int64_t out_stride, int n, int lead, bool vectors, const T *carry_in, TempHeader *hdr) {
    using O = Op<T, OP>;
    constexpr int WARPS = kShortThreads / 32, VEC = 16 / sizeof(T), NV = kShortItems / VEC;
    union Vec { uint4 u; T t[VEC]; };
    __shared__ T warp_total[WARPS];
    __shared__ T block_total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = (int)blockIdx.x * kShortTile + tid * kShortItems;
    grid_dependency_wait();
    if (blockIdx.x == 0 && tid == 0) hdr->wait_limit_hit = 0u;
    T v[kShortItems];
    const bool whole = vectors && first >= lead && first + kShortItems <= n;
    if (whole) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            Vec a;
            a.u = reinterpret_cast<const uint4 *>(in + first)[q];
#pragma unroll
            for (int e = 0; e < VEC; ++e) v[q * VEC + e] = a.t[e];
        }
    } else {
#pragma unroll
        for (int k = 0; k < kShortItems; ++k) v[k] = first + k >= lead && first + k < n ? in[(first + k) * in_stride] : O::identity();
    }
    T sum = v[0];
#pragma unroll
    for (int k = 1; k < kShortItems; ++k) sum = O::apply(sum, v[k]);
    T incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T up = shfl_up(incl, d);
        if (lane >= d) incl = O::apply(up, incl);
    }
    T running = shfl_up(incl, 1);
    if (lane == 0) running = O::identity();
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    T warps = warp_total[lane];  // every warp scans the totals of all
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T up = shfl_up(warps, d);
        if (lane >= d) warps = O::apply(up, warps);
    }
    const T ahead = shfl_idx(warps, warp > 0 ? warp - 1 : 0);
    if (warp > 0) running = O::apply(ahead, running);
    T base = carry_in ? *carry_in : O::identity();
    if (gridDim.x > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        if (tid == kShortThreads - 1) block_total = warps;
        cluster.sync();
        T before = lane < (int)blockIdx.x ? *cluster.map_shared_rank(&block_total, lane) : O::identity();
#pragma unroll
        for (int d = 1; d < kShortCluster; d <<= 1) before = O::apply(before, shfl_down(before, d));
        base = O::apply(base, shfl_idx(before, 0));
        cluster.sync();  // nobody leaves while its total is being read
    }
    running = O::apply(base, running);
#pragma unroll
    for (int k = 0; k < kShortItems; ++k) {
        const T next = O::apply(running, v[k]);
        v[k] = INCLUSIVE ? next : running;
        running = next;
    }
    if (whole) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            Vec a;
#pragma unroll
            for (int e = 0; e < VEC; ++e) a.t[e] = v[q * VEC + e];
            reinterpret_cast<uint4 *>(out + first)[q] = a.u;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kShortItems; ++k)
            if (first + k >= lead && first + k < n) out[(first + k) * out_stride] = v[k];
    }
}

template <typename T> constexpr int scan_tile_elems() { return (16 / (int)sizeof(T)) * kScanVecPerThread * kScanThreads; }

static int64_t scan_temp_bytes_for(int dtype, int64_t n) {
    // Sized for the smaller tile (8-byte types) so that one formula covers every type.
    const int64_t tiles = ceil_div((n < 1 ? 1 : n) + 3, kScanMinTileElems);  // (a view may start up to 3 elements off)
    (void)dtype;
    return (int64_t)sizeof(TempHeader) + round_up(tiles * kDescStride, 256);
}

template <typename T, int OP, bool INCLUSIVE>
static int launch_scan(cudaStream_t s, const void *in, int64_t in_stride, void *out, int64_t out_stride, int64_t n,
                       const void *carry_in, void *temp) {
    constexpr int TILE = scan_tile_elems<T>();
    TempHeader *hdr = (TempHeader *)temp;
    void *state = (char *)temp + sizeof(TempHeader);
    // A view that does not start on 16 bytes is scanned from the 16-byte boundary in front of it, when
    // input and output are off by as much.
    const bool alike = in_stride == 1 && out_stride == 1 && ((uintptr_t)in % 16 == (uintptr_t)out % 16);
    const int lead = alike ? (int)((uintptr_t)in % 16 / sizeof(T)) : 0;
    const T *in_t = (const T *)in - lead;
    T *out_t = (T *)out - lead;
    const T *carry_t = (const T *)carry_in;
    int64_t n_arg = n + lead;
    if (n_arg <= kShortCluster * kShortTile) {
        int blocks = 1;
        while (blocks * kShortTile < n_arg) blocks *= 2;
        B200ALG_CUDA_TRY(launch_dependent_cluster(scan_short_kernel<T, OP, INCLUSIVE>, dim3(blocks), dim3(kShortThreads), 0, s, (unsigned int)blocks, in_t,
                                                  in_stride, out_t, out_stride, (int)n_arg, lead, alike, carry_t, hdr));
        return B200ALG_OK;
    }
    bool launched = false;
    if (alike) {
        const int tiles = (int)ceil_div(n_arg, kPipeTileBytes / (int)sizeof(T));
        auto kernel = lead ? scan_pipeline_kernel<T, OP, INCLUSIVE, true> : scan_pipeline_kernel<T, OP, INCLUSIVE, false>;
        constexpr size_t ring_bytes = (size_t)kPipeStages * kPipeTileBytes;
        static ContextCache<int> caches[2];  // per kernel instantiation and CUDA context
        ContextCache<int> &cache = caches[lead != 0];
        int blocks_per_sm = 0;
        if (!cache.find(&blocks_per_sm)) {
            B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring_bytes));
            B200ALG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, kernel, kPipeThreads, ring_bytes));
            if (blocks_per_sm < 1) return B200ALG_UNSUPPORTED;
            cache.store(blocks_per_sm);
        }
        // One wave of persistent blocks, launched cooperatively: the driver either makes all of
        // them resident at once (tiles are taken round-robin and wait for one another) or
        // refuses the launch.
        const int resident = sm_count() * blocks_per_sm;  // (two at least, as there are two SMs at least)
        const int blocks = tiles < resident ? tiles + 1 : resident;  // one of them the scanner
        int lead_arg = lead, tiles_arg = tiles;
        void *args[] = {&in_t, &out_t, &n_arg, &lead_arg, &carry_t, &hdr, &state, &tiles_arg};
        const cudaError_t e = cudaLaunchCooperativeKernel((const void *)kernel, dim3(blocks), dim3(kPipeThreads), args, ring_bytes, s);
        if (e == cudaSuccess) launched = true;
        else if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) (void)cudaGetLastError();
        else return cuda_fail(e);
    }
    if (!launched) {
        const int general_tiles = (int)ceil_div(n, TILE);
        {
            const int64_t words = (int64_t)((sizeof(TempHeader) + (size_t)general_tiles * kDescStride) / 16);
            const int64_t want = ceil_div(words, 256 * 4);
            const int64_t cap = (int64_t)sm_count() * 4;
            scan_clear_kernel<<<(int)(want < 1 ? 1 : (want > cap ? cap : want)), 256, 0, s>>>((uint4 *)temp, words);
            B200ALG_LAUNCH_CHECK();
        }
        B200ALG_CUDA_TRY(launch_dependent(scan_kernel<T, OP, INCLUSIVE>, dim3(general_tiles), dim3(kScanThreads), 0, s, (const T *)in, in_stride,
                                          (T *)out, out_stride, n, carry_t, hdr, state, general_tiles));
    }
    return B200ALG_OK;
}

template <typename T, int OP>
static int dispatch_kind(cudaStream_t s, const void *in, int64_t is, void *out, int64_t os, int64_t n, int inclusive,
                         const void *carry, void *temp) {
    return inclusive ? launch_scan<T, OP, true>(s, in, is, out, os, n, carry, temp)
                     : launch_scan<T, OP, false>(s, in, is, out, os, n, carry, temp);
}

template <typename T>
static int dispatch_scan_op(cudaStream_t s, const void *in, int64_t is, void *out, int64_t os, int64_t n, int op,
                            int inclusive, const void *carry, void *temp) {
    switch (op) {
    case B200ALG_ADD: return dispatch_kind<T, B200ALG_ADD>(s, in, is, out, os, n, inclusive, carry, temp);
    case B200ALG_MAX: return dispatch_kind<T, B200ALG_MAX>(s, in, is, out, os, n, inclusive, carry, temp);
    case B200ALG_MIN: return dispatch_kind<T, B200ALG_MIN>(s, in, is, out, os, n, inclusive, carry, temp);
    }
    return B200ALG_UNSUPPORTED;
}

}  // namespace b200alg

using namespace b200alg;

extern "C" int b200alg_scan_temp_bytes(int dtype, int64_t n, int64_t *out_bytes) {
    if (!out_bytes || n < 0) return B200ALG_INVALID_ARGUMENT;
    if (!is_atomic_numeric(dtype)) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    *out_bytes = scan_temp_bytes_for(dtype, n);
    return B200ALG_OK;
}

extern "C" int b200alg_scan_carry(void *stream, const void *in, int64_t in_stride, void *out, int64_t out_stride,
                                  int64_t n, int dtype, int op, int inclusive, const void *carry_in, void *temp,
                                  int64_t temp_bytes) {
    // Argument checks mirror CreateSinglePassScan's (ScanExtensions.cs:675-689).
    if (!in || !out || !temp) return B200ALG_INVALID_ARGUMENT;
    if (n < 0 || in_stride < 1 || out_stride < 1) return B200ALG_INVALID_ARGUMENT;
    if (!is_atomic_numeric(dtype)) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements) return B200ALG_TOO_LARGE;
    const int es = dtype_bytes(dtype);
    if (((uintptr_t)in % es) || ((uintptr_t)out % es) || (carry_in && ((uintptr_t)carry_in % es))) return B200ALG_MISALIGNED;
    if ((uintptr_t)temp % 256) return B200ALG_MISALIGNED;
    if (temp_bytes < scan_temp_bytes_for(dtype, n)) return B200ALG_TEMP_TOO_SMALL;
    if (n == 0) return B200ALG_OK;
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
    case B200ALG_I32: return dispatch_scan_op<int32_t>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    case B200ALG_U32: return dispatch_scan_op<uint32_t>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    case B200ALG_I64: return dispatch_scan_op<int64_t>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    case B200ALG_U64: return dispatch_scan_op<uint64_t>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    case B200ALG_F32: return dispatch_scan_op<float>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    case B200ALG_F64: return dispatch_scan_op<double>(s, in, in_stride, out, out_stride, n, op, inclusive, carry_in, temp);
    }
    return B200ALG_UNSUPPORTED;
}

extern "C" int b200alg_scan(void *stream, const void *in, int64_t in_stride, void *out, int64_t out_stride, int64_t n,
                            int dtype, int op, int inclusive, void *temp, int64_t temp_bytes) {
    return b200alg_scan_carry(stream, in, in_stride, out, out_stride, n, dtype, op, inclusive, nullptr, temp, temp_bytes);
}

// ---- scan without caller-provided scratch ------------------------------------------------
// Some callers can neither size nor allocate a temp view: code that runs where device
// allocation is off the table (a host callback on a stream, a real-time loop that may not
// take the allocator's lock, a plug-in that is handed input and output views and nothing
// else).  For them the tile descriptors of the chained scan live in this fixed array,
// which every GPU that loads the library carries until the process exits.
constexpr int64_t kStaticScanMaxElements = 1ll << 26;
constexpr size_t kStaticScanScratchBytes = sizeof(TempHeader) + (size_t)(kStaticScanMaxElements / kScanMinTileElems + 2) * kDescStride;
static __device__ __align__(256) unsigned char g_static_scan_scratch[kStaticScanScratchBytes];

namespace b200alg {
// Device address of the array in the current CUDA context.  The array's name is only a handle
// on the host side, so the address is asked for once per context, with that context current.
int static_scan_scratch(void **out) {
    static ContextCache<void *> cache;
    void *p = nullptr;
    if (!cache.find(&p)) {
        B200ALG_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scan_scratch));
        cache.store(p);
    }
    *out = p;
    return B200ALG_OK;
}
}  // namespace b200alg

extern "C" int b200alg_scan_static(void *stream, const void *in, int64_t in_stride, void *out, int64_t out_stride,
                                   int64_t n, int dtype, int op, int inclusive) {
    if (n > kStaticScanMaxElements) return B200ALG_STATIC_LIMIT;
    void *scratch = nullptr;
    const int rc = static_scan_scratch(&scratch);
    if (rc != B200ALG_OK) return rc;
    // Same launch sequence as b200alg_scan: it clears the descriptors it is about to use, so
    // whatever the previous call left in the array does not matter.
    return b200alg_scan_carry(stream, in, in_stride, out, out_stride, n, dtype, op, inclusive, nullptr, scratch,
                              (int64_t)kStaticScanScratchBytes);
}
