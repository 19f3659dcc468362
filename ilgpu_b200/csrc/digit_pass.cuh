// The digit pass of the radix sort (included by radix_sort.cu, which defines the key transforms, the
// look-back words and the buffer schedule).
//
// Persistent blocks, two per SM.  Most of them move keys; a tile goes through
//
//   load      its keys, out of the staging buffer (one bulk copy, issued a tile ahead) into registers
//   rank      one shared-memory atomic per key on the warp's count of its digit
//   count     the warps' counts become slots of the tile; the tile's counts are published
//   reorder   keys (and, with values, their places in the tile) to their slots in shared memory
//   write     slots out to global memory, runs of one digit in a row
//
// kScanners blocks (the first to arrive) move no keys: each adds up the published counts of its share
// of the digits, tile after tile, and publishes where every tile's keys go.  The tile before is written
// between count and reorder, which leaves the scanners the steps of a whole tile to answer.  (With
// decoupled look-back in every block instead, the waiting was half of a tile's time, 8700 of 18300
// cycles: some 25 rows of 1 KB read per tile, each behind the shared-memory instructions that fill
// the SM's load/store queue; wider look-back windows and separate look-back warps were no faster.)
//
// Order.  The atomic returns how many keys of the digit the warp has counted before.  Lanes that meet
// in one word are not promised any order, and the sort needs theirs: keys of one digit stay in lane
// order.  The hardware does serve them in lane order (none of 1.6e7 collisions differed), and nothing
// relies on it: the write step checks every slot against the one before it - by what this and the
// earlier passes have sorted, for keys alone; by the places in the tile when there are values - and a
// tile that fails is put in order in shared memory and written again.  (Finding a digit's lanes
// through masks in shared memory is ordered by construction, but takes three more trips to random
// words per key: 10 of 30 shared-memory cycles per 32 keys.)
//
// Few words for many lanes cost what serving them takes, which is little when all meet in one.  2^26
// uint32, one pass: random keys 172 us; keys that arrive in order 163 to 172; a running number's
// highest byte, one word for nearly every warp, 188.  Two words in random alternation are the worst
// case: a sort of two values mixed takes 1350 us, of random keys 749.
#pragma once

namespace b200alg {

constexpr int kPassThreads = 512;
constexpr int kPassWarps = kPassThreads / 32;
constexpr int kPassBlocksPerSm = 2;
constexpr int kPassSmem = 113 * 1024;                  // what a block may use so that two fit on an SM
constexpr int kDigitThreads = kPassThreads / kRadix;   // threads that share a digit when counts become slots
constexpr int kDigitRows = kPassWarps / kDigitThreads; // and warps each of them adds up
constexpr int kSwizzle = 32 / kDigitThreads;
constexpr int kScanners = 4;
constexpr int kScanDigits = kRadix / kScanners;
constexpr int kPassFixedSmem = kPassWarps * kRadix * 4 + 2 * kRadix * (4 + 8) + 2 * 1024;
constexpr int kPassMaxItems = 20;

// Keys per thread: as many as fit, up to twenty (registers; a tile's fixed costs, some 2500 cycles of
// counting, weigh less the longer it is: 2^26 keys 812 us with 16, 765 us with 20, 787 us with 21).
constexpr int pass_items(int key_bytes, int value_bytes) {
    const int per_item = kPassThreads * (2 * key_bytes + (value_bytes ? value_bytes + 2 : 0));
    const int fit = (kPassSmem - kPassFixedSmem) / per_item;
    return fit < kPassMaxItems ? fit : kPassMaxItems;
}
constexpr int pass_tile(int key_bytes, int value_bytes) { return kPassThreads * pass_items(key_bytes, value_bytes); }
static_assert(3 * 2 * pass_tile(1, 0) < 65536, "three rows of two tiles are summed in 16 bits");

template <typename K, typename V, typename Idx> struct PassSmem {
    static constexpr int VB = ValueBytes<V>::value;
    static constexpr int ITEMS = pass_items(sizeof(K), VB);
    static constexpr int TILE = kPassThreads * ITEMS;
    static constexpr size_t up(size_t v) { return (v + 127) / 128 * 128; }
    static constexpr size_t off_stage = 0;                                          // keys of the next tile
    static constexpr size_t off_values = up(off_stage + (size_t)TILE * sizeof(K));  // values of a tile, in input order
    static constexpr size_t off_keys = up(off_values + (size_t)TILE * VB);          // keys in slot order
    static constexpr size_t off_place = up(off_keys + (size_t)TILE * sizeof(K));    // where in the tile a slot's key came from
    static constexpr size_t off_table = up(off_place + (VB ? (size_t)TILE * 2 : 0));
    // a digit's first slot, for this tile and the one before; global index of a slot minus the slot
    static constexpr size_t off_excl = off_table + (size_t)kPassWarps * kRadix * 4;
    static constexpr size_t off_goff = off_excl + 2 * kRadix * 4;
    static constexpr size_t off_misc = off_goff + kRadix * sizeof(Idx);
    static constexpr size_t bytes = off_misc + 512;
    static_assert(bytes <= kPassSmem, "two blocks per SM");
};

// Everything a block needs to know about its pass.
template <typename K, typename V, typename SW> struct Pass {
    const K *src;
    K *dst;
    int64_t src_stride, dst_stride;
    const V *vsrc;
    V *vdst;
    int64_t n;
    int num_tiles;
    int value_seq;  // not kSeqNone: this pass makes the values from the element index
    bool dense;     // source and destination are contiguous
    // the keys of a full tile come by bulk copy (dense, 16-byte aligned source; the first pass of a sort
    // whose view starts elsewhere does without, and the last one stores off the boundary: 2^26 uint32
    // 828 instead of 749 us)
    bool bulk;
    bool vbulk;     // likewise its values
    TempHeader *hdr;
    unsigned int *ticket;
    const unsigned long long *gbase;
    unsigned short *counts, *counts_next;  // per tile and digit: keys | kCounted
    SW *places, *places_next;              // per two tiles and digit: where their keys go | StatusWord::kIncl
};
constexpr unsigned int kCounted = 0x8000u;
// The small shared words of a block.
template <typename K, typename V, typename SW> struct PassMisc {
    unsigned long long key_bar, value_bar;  // bulk copies
    unsigned int warp_sum[kPassWarps];
    int next_tile;
    int role;  // below kScanners: this block is a scanner
    Pass<K, V, SW> pass;
};

__device__ __forceinline__ bool block_any(bool p) { return __syncthreads_or(p) != 0; }

// The published words of four neighbouring digits.
template <typename SW> struct Words4 { SW w[4]; };
__device__ __forceinline__ void load_words(Words4<unsigned int> &v, const unsigned int *p) {
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void load_words(Words4<unsigned long long> &v, const unsigned long long *p) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.w[0]), "=l"(v.w[1]) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.w[2]), "=l"(v.w[3]) : "l"(p + 2) : "memory");
}

__device__ __forceinline__ void store_words(unsigned int *p, const Words4<unsigned int> &v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]) : "memory");
}
__device__ __forceinline__ void store_words(unsigned long long *p, const Words4<unsigned long long> &v) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(v.w[0]), "l"(v.w[1]) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1,%2};" ::"l"(p + 2), "l"(v.w[2]), "l"(v.w[3]) : "memory");
}

// A scanner block: goes over the published counts, two tiles to a row, 64 rows and kScanDigits digits
// at a time, and stores the running sums (which start from the digits' global offsets).
template <typename K, typename V, typename SW>
__device__ __noinline__ void scan_counts(unsigned char *smem, const Pass<K, V, SW> &c, int scanner) {
    using S = StatusWord<SW>;
    using Idx = typename IndexOf<SW>::type;
    constexpr int LANES = kScanDigits / 8;      // threads per row, eight digits each
    constexpr int WARP_ROWS = 32 / LANES;
    static_assert(WARP_ROWS == 4, "four rows per warp, three of which are summed in 16 bits");
    unsigned int *warp_rows = reinterpret_cast<unsigned int *>(smem);                        // [2][warps]: which rows of the warp are complete
    uint4 *warp_total = reinterpret_cast<uint4 *>(smem + 256);                               // [2][warps][digits], 16 bits: three rows, the fourth
    Idx *warp_base = reinterpret_cast<Idx *>(smem + 256 + 2 * kPassWarps * kScanDigits * 2); // [warps][digits]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = warp * WARP_ROWS + lane / LANES, octet = lane % LANES, d0 = scanner * kScanDigits + octet * 8;
    const int pairs = (c.num_tiles + 1) / 2;
    Idx carry = tid < kScanDigits ? (Idx)c.gbase[scanner * kScanDigits + tid] : 0;
    ScannerPolls limit;
    for (int pos = 0, turn = 0; pos < pairs; turn ^= 1) {
        const int t = pos + row;
        Words4<unsigned int> a, b;
#pragma unroll
        for (int q = 0; q < 4; ++q) a.w[q] = 0u, b.w[q] = 0x80008000u;
        if (t < pairs) {
            const unsigned short *from = c.counts + (size_t)(2 * t) * kRadix + d0;
            load_words(a, reinterpret_cast<const unsigned int *>(from));
            if (2 * t + 1 < c.num_tiles) load_words(b, reinterpret_cast<const unsigned int *>(from + kRadix));
        }
        const bool here = (a.w[0] & a.w[1] & a.w[2] & a.w[3] & b.w[0] & b.w[1] & b.w[2] & b.w[3] & 0x80008000u) == 0x80008000u;
        const unsigned int complete = __ballot_sync(0xffffffffu, here);
        if (lane == 0) {
            unsigned int rows = 0u;
#pragma unroll
            for (int r = 0; r < WARP_ROWS; ++r) rows |= (complete >> (LANES * r) & ((1u << LANES) - 1u)) == (1u << LANES) - 1u ? 1u << r : 0u;
            warp_rows[turn * kPassWarps + warp] = rows;
        }
        __syncthreads();
        // rows complete from the first on
        const unsigned int rows = lane < kPassWarps ? warp_rows[turn * kPassWarps + lane] : 0u;
        const int whole = __ffs((int)~__ballot_sync(0xffffffffu, rows == 15u)) - 1;  // warps (of sixteen)
        const int ready = whole * WARP_ROWS + __ffs((int)~__shfl_sync(0xffffffffu, rows, whole)) - 1;
        if (ready == 0) {
            if (!limit.again(pos > 0, [](unsigned int ns) { __nanosleep(ns); })) {
                if (tid == 0) atomicExch(&c.hdr->wait_limit_hit, 1u);
                return;
            }
            continue;
        }
        limit.progress();
        const bool mine = row < ready, last = lane >= 32 - LANES;
        unsigned int own[4], incl[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            own[q] = mine ? (a.w[q] & 0x7FFF7FFFu) + (b.w[q] & 0x7FFF7FFFu) : 0u;
            incl[q] = last ? 0u : own[q];  // with the fourth row the sums might need a 17th bit
        }
#pragma unroll
        for (int k = LANES; k < 32; k <<= 1)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, incl[q], k);
                if (lane >= k) incl[q] += up;
            }
        if (last) {
            warp_total[warp * LANES + octet] = make_uint4(incl[0], incl[1], incl[2], incl[3]);
            warp_total[(kPassWarps + warp) * LANES + octet] = make_uint4(own[0], own[1], own[2], own[3]);
        }
        __syncthreads();
        if (tid < kScanDigits) {
            const unsigned short *total = reinterpret_cast<const unsigned short *>(warp_total);
            unsigned int v[kPassWarps];
#pragma unroll
            for (int k = 0; k < kPassWarps; ++k) v[k] = (unsigned int)total[k * kScanDigits + tid] + total[(kPassWarps + k) * kScanDigits + tid];
#pragma unroll
            for (int k = 0; k < kPassWarps; ++k) {
                warp_base[k * kScanDigits + tid] = carry;
                carry += v[k];
            }
        }
        __syncthreads();
        if (mine) {
            const Idx *base = warp_base + warp * kScanDigits + octet * 8;
            SW *out = c.places + (size_t)t * kRadix + d0;
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                const unsigned int a0 = incl[q] - (last ? 0u : own[q]), a1 = incl[q + 1] - (last ? 0u : own[q + 1]);
                Words4<SW> v;
                v.w[0] = (SW)S::kIncl | (SW)(base[2 * q] + (a0 & 0xFFFFu));
                v.w[1] = (SW)S::kIncl | (SW)(base[2 * q + 1] + (a0 >> 16));
                v.w[2] = (SW)S::kIncl | (SW)(base[2 * q + 2] + (a1 & 0xFFFFu));
                v.w[3] = (SW)S::kIncl | (SW)(base[2 * q + 3] + (a1 >> 16));
                store_words(out + 2 * q, v);
            }
        }
        pos += ready;
    }
}

// Takes the block's next tile; the keys of a full one start on their way to the staging buffer.
template <typename K, typename V, typename SW, typename L>
__device__ __forceinline__ void take_tile(PassMisc<K, V, SW> &m, unsigned char *smem) {
    const Pass<K, V, SW> &c = m.pass;
    const int next = (int)atomicAdd(c.ticket, 1u);
    m.next_tile = next;
    if (c.bulk && (int64_t)(next + 1) * L::TILE <= c.n) {
        mbar_expect_tx(&m.key_bar, (unsigned int)(L::TILE * sizeof(K)));
        bulk_load(smem + L::off_stage, c.src + (int64_t)next * L::TILE, (unsigned int)(L::TILE * sizeof(K)), &m.key_bar);
    }
}

// Puts the slots of a tile in order.  Reached only when the atomics of a warp were not served in lane
// order.
template <typename K, typename V, typename XF, typename L>
__device__ __noinline__ void repair_order(unsigned char *smem, XF xf, int shift) {
    put_in_order<K, L::VB != 0>(reinterpret_cast<K *>(smem + L::off_keys), reinterpret_cast<unsigned short *>(smem + L::off_place), L::TILE,
                                (int)threadIdx.x, kPassThreads, xf, shift, [](bool moved) { return block_any(moved); });
}

// Writes the tile in the slots to global memory; true when a slot is out of order.
template <typename K, typename V, typename SW, typename XF, typename L, bool FAST>
__device__ __forceinline__ bool write_tile(unsigned char *smem, const Pass<K, V, SW> &c, int tile, XF xf, int shift) {
    using Idx = typename IndexOf<SW>::type;
    const K *keys = reinterpret_cast<const K *>(smem + L::off_keys);
    const V *values = reinterpret_cast<const V *>(smem + L::off_values);
    const unsigned short *place = reinterpret_cast<const unsigned short *>(smem + L::off_place);
    const Idx *goff = reinterpret_cast<const Idx *>(smem + L::off_goff);
    const int64_t base = (int64_t)tile * L::TILE;
    const int valid = FAST ? L::TILE : (int)(c.n - base < L::TILE ? c.n - base : L::TILE);
    K *const dst = c.dst;
    const int64_t stride = c.dst_stride;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < L::ITEMS; ++i) {
        const int p = (int)threadIdx.x + i * kPassThreads, ahead = p > 0 ? p - 1 : 0;
        const K k = keys[p], k_ahead = keys[ahead];
        unsigned int from = 0u, from_ahead = 0u;
        if constexpr (L::VB != 0) {
            from = place[p];
            from_ahead = place[ahead];
        }
        bad |= out_of_order<K, L::VB != 0>(k_ahead, k, from_ahead, from, xf, shift);
        if (FAST || p < valid) {
            const Idx at = goff[(unsigned int)(xf(k) >> shift) & 0xFFu] + (Idx)p;
            if (FAST) dst[at] = k; else dst[(int64_t)at * stride] = k;
            if constexpr (L::VB != 0) {
                if constexpr (L::VB <= 8) c.vdst[at] = c.value_seq != kSeqNone ? sequence_value<V>(c.value_seq, base + from) : values[from];
                else c.vdst[at] = values[from];
            }
        }
    }
    return bad;
}

template <typename K, typename V, typename SW, typename XF>
__global__ void __launch_bounds__(kPassThreads, kPassBlocksPerSm)
digit_pass_kernel(SortBuffers<K, V> io, int pass, XF xf, TempHeader *hdr, const unsigned long long *gbase_all, void *published,
                  int max_tiles, int value_seq) {
    using S = StatusWord<SW>;
    using Idx = typename IndexOf<SW>::type;
    using L = PassSmem<K, V, Idx>;
    constexpr int ITEMS = L::ITEMS, TILE = L::TILE;
    extern __shared__ __align__(128) unsigned char smem[];
    static_assert(sizeof(PassMisc<K, V, SW>) <= 512, "room for the small words");
    PassMisc<K, V, SW> &m = *reinterpret_cast<PassMisc<K, V, SW> *>(smem + L::off_misc);
    const Pass<K, V, SW> &c = m.pass;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int shift = pass * 8;

    grid_dependency_release();  // the next kernel of the call may take the SMs this one leaves
    grid_dependency_wait();     // everything the kernels before this one wrote is visible from here on
    if (hdr->reserved[kCtlSkip + pass]) return;
    if (tid == kPassThreads - 1) {
        Pass<K, V, SW> &w = m.pass;
        const unsigned int src = hdr->reserved[kCtlSrc + pass], dst = hdr->reserved[kCtlDst + pass];
        w.src = src == kBufIn ? io.in : (src == kBufOut ? io.out : io.alt);
        w.dst = dst == kBufOut ? io.out : io.alt;
        w.src_stride = src == kBufAlt ? 1 : io.stride;
        w.dst_stride = dst == kBufAlt ? 1 : io.stride;
        w.vsrc = src == kBufIn ? io.vin : (src == kBufOut ? io.vout : io.valt);
        w.vdst = dst == kBufOut ? io.vout : io.valt;
        w.n = effective_n(io);
        w.num_tiles = (int)((w.n + TILE - 1) / TILE);
        w.value_seq = hdr->reserved[kCtlFirstPass] == (unsigned int)pass ? value_seq : kSeqNone;
        w.dense = io.stride == 1;
        w.bulk = w.dense && ((uintptr_t)w.src % 16 == 0);
        w.vbulk = L::VB != 0 && w.value_seq == kSeqNone && ((uintptr_t)w.vsrc % 16 == 0);
        w.hdr = hdr;
        w.ticket = &hdr->reserved[kCtlTicket + pass];
        w.gbase = gbase_all + pass * kRadix;
        // two sets of published words alternate between the passes that run; this pass clears the ones
        // the next will use (the previous pass, their last user, has completed)
        const bool upper = hdr->reserved[kCtlStatusHalf + pass] != 0;
        const size_t pairs = (size_t)(max_tiles + 1) / 2;
        SW *half[2] = {(SW *)published, (SW *)((unsigned char *)published + pairs * kRadix * (sizeof(SW) + 4))};
        w.places = half[upper];
        w.places_next = half[!upper];
        w.counts = (unsigned short *)(w.places + pairs * kRadix);
        w.counts_next = (unsigned short *)(w.places_next + pairs * kRadix);
        m.role = (int)atomicAdd(&hdr->reserved[kCtlRole + pass], 1u);
        mbar_init(&m.key_bar, 1u);
        mbar_init(&m.value_bar, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (m.role >= kScanners) take_tile<K, V, SW, L>(m, smem);
    }
    // counts of this warp's keys per digit; swizzled, so that the threads that share a digit read their
    // rows of it without meeting in a bank
    unsigned int *table = reinterpret_cast<unsigned int *>(smem + L::off_table);
    unsigned int *mine = table + warp * kRadix;
    const unsigned int swizzle = (unsigned int)(warp / kDigitRows * kSwizzle);
    auto clear_mine = [&]() {
#pragma unroll
        for (int i = 0; i < kRadix / 4 / 32; ++i) reinterpret_cast<uint4 *>(mine)[i * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
    };
    clear_mine();
    __syncthreads();
    if (m.role < kScanners) {
        scan_counts<K, V, SW>(smem, c, m.role);
        return;
    }

    K *stage = reinterpret_cast<K *>(smem + L::off_stage);
    K *slots = reinterpret_cast<K *>(smem + L::off_keys);
    unsigned short *place = reinterpret_cast<unsigned short *>(smem + L::off_place);
    const int own = warp * 32 * ITEMS + lane;  // this lane's first key; the others follow 32 apart
    unsigned int key_phase = 0u, value_phase = 0u;
    int tile = m.next_tile, before = -1;
    bool before_bulk_values = false;
    for (int turn = 0;; turn ^= 1) {
        const bool work = tile < c.num_tiles;
        K key[ITEMS];
        unsigned int rank[(ITEMS + 1) / 2];  // two to a word: keys of the digit the warp has counted before
        if (work) {
            const int64_t base = (int64_t)tile * TILE;
            if (c.bulk && base + TILE <= c.n) {
                if (!mbar_wait(&m.key_bar, key_phase) && lane == 0) atomicExch(&c.hdr->wait_limit_hit, 1u);
                key_phase ^= 1u;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) key[i] = stage[own + i * 32];
            } else {
                const K *from = c.src;
                const int64_t stride = c.src_stride, left = c.n - base;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) key[i] = own + i * 32 < left ? from[(base + own + i * 32) * stride] : padding_key<K>(xf);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const unsigned int d = (unsigned int)(xf(key[i]) >> shift) & 0xFFu;
                const unsigned int r = atomicAdd(mine + (d ^ swizzle), 1u);
                if (i & 1) rank[i / 2] |= r << 16; else rank[i / 2] = r;
            }
        }
        __syncthreads();  // the tables are complete, the staging buffer is free, the tile before is in its slots
        // where the keys of the tile before go: four digits each for the first threads.  The second tile
        // of a pair goes behind the first one's keys.
        Words4<SW> target;
        unsigned int first_of_pair[2];
        auto load_target = [&](int of) {
            load_words(target, c.places + (size_t)(of / 2) * kRadix + tid * 4);
            first_of_pair[0] = first_of_pair[1] = kCounted | kCounted << 16;
            if (of & 1)
                asm volatile("ld.relaxed.gpu.global.v2.u32 {%0,%1}, [%2];" : "=r"(first_of_pair[0]), "=r"(first_of_pair[1])
                             : "l"(c.counts + (size_t)(of - 1) * kRadix + tid * 4) : "memory");
            return (target.w[0] & target.w[1] & target.w[2] & target.w[3] & S::kIncl) != 0 &&
                   (first_of_pair[0] & first_of_pair[1] & (kCounted | kCounted << 16)) == (kCounted | kCounted << 16);
        };
        bool known = true;
        if (before >= 0 && tid < kRadix / 4) known = load_target(before);
        if (work) {
            if (tid == kPassThreads - 1) take_tile<K, V, SW, L>(m, smem);
            // kDigitThreads neighbouring threads share a digit, each adds up the counts of kDigitRows warps.
            const int d = tid / kDigitThreads, part = tid % kDigitThreads;
            unsigned int *column = table + part * (kDigitRows * kRadix) + (d ^ (part * kSwizzle));
            unsigned int first[kDigitRows / 2];  // d-keys of my warps before each of them, two to a word
            unsigned int part_total = 0;
#pragma unroll
            for (int w = 0; w < kDigitRows; w += 2) {
                const unsigned int a = column[w * kRadix], b = column[(w + 1) * kRadix];
                first[w / 2] = part_total | (part_total + a) << 16;
                part_total += a + b;
            }
            unsigned int total = part_total;  // of the parts up to mine, then of all
#pragma unroll
            for (int k = 1; k < kDigitThreads; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, total, k);
                if (part >= k) total += up;
            }
            const unsigned int ahead = total - part_total;
            total = __shfl_sync(0xffffffffu, total, lane | (kDigitThreads - 1));
            if (part == 0) {
                asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(c.counts + (size_t)tile * kRadix + d), "h"((unsigned short)(total | kCounted)) : "memory");
                c.counts_next[(size_t)tile * kRadix + d] = 0;
                if (!(tile & 1)) c.places_next[(size_t)(tile / 2) * kRadix + d] = 0;
            }
            // exclusive scan of the digits' counts: sixteen digits per warp, then over the warps
            unsigned int incl = total;
#pragma unroll
            for (int k = kDigitThreads; k < 32; k <<= 1) {
                const unsigned int up = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += up;
            }
            if (lane == 31) m.warp_sum[warp] = incl;
            __syncthreads();
            const unsigned int excl = incl - total + __reduce_add_sync(0xffffffffu, lane < warp ? m.warp_sum[lane] : 0u);
            if (part == 0) reinterpret_cast<unsigned int *>(smem + L::off_excl)[turn * kRadix + d] = excl;
#pragma unroll
            for (int w = 0; w < kDigitRows; w += 2) {
                column[w * kRadix] = excl + ahead + (first[w / 2] & 0xFFFFu);
                column[(w + 1) * kRadix] = excl + ahead + (first[w / 2] >> 16);
            }
        }
        bool bad = false;
        const bool before_fast = c.dense && (int64_t)(before + 1) * TILE <= c.n;
        auto write_before = [&]() {
            return before_fast ? write_tile<K, V, SW, XF, L, true>(smem, c, before, xf, shift)
                               : write_tile<K, V, SW, XF, L, false>(smem, c, before, xf, shift);
        };
        if (before >= 0) {
            if (tid < kRadix / 4) {
                const unsigned int *excl = reinterpret_cast<const unsigned int *>(smem + L::off_excl) + (turn ^ 1) * kRadix + tid * 4;
                Idx *goff = reinterpret_cast<Idx *>(smem + L::off_goff) + tid * 4;
                unsigned int spins = 0;
                while (!known) {
                    if (++spins > kMaxSpin) {
                        atomicExch(&c.hdr->wait_limit_hit, 1u);
                        break;
                    }
                    __nanosleep(20);
                    known = load_target(before);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const unsigned int ahead = (first_of_pair[q / 2] >> (q & 1) * 16) & (kCounted - 1u);
                    goff[q] = (Idx)(target.w[q] & S::kMask) + ahead - (Idx)excl[q];
                }
            }
            __syncthreads();
            if (L::VB != 0 && before_bulk_values) {
                if (!mbar_wait(&m.value_bar, value_phase) && lane == 0) atomicExch(&c.hdr->wait_limit_hit, 1u);
                value_phase ^= 1u;
            }
            bad = write_before();
        }
        if (block_any(bad)) {  // (also: the slots are free, every slot of this tile is known)
            repair_order<K, V, XF, L>(smem, xf, shift);
            write_before();
            __syncthreads();
        }
        if (!work) break;

        if constexpr (L::VB != 0) {
            if (c.value_seq == kSeqNone) {  // values are fetched by place when the tile is written
                const int64_t base = (int64_t)tile * TILE;
                before_bulk_values = c.vbulk && base + TILE <= c.n;
                V *values = reinterpret_cast<V *>(smem + L::off_values);
                if (before_bulk_values) {
                    if (tid == kPassThreads - 1) {
                        mbar_expect_tx(&m.value_bar, (unsigned int)(TILE * sizeof(V)));
                        bulk_load(values, c.vsrc + base, (unsigned int)(TILE * sizeof(V)), &m.value_bar);
                    }
                } else {
                    for (int j = tid; j < TILE && base + j < c.n; j += kPassThreads) values[j] = c.vsrc[base + j];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const unsigned int d = (unsigned int)(xf(key[i]) >> shift) & 0xFFu;
            const unsigned int slot = (i & 1 ? rank[i / 2] >> 16 : rank[i / 2] & 0xFFFFu) + mine[d ^ swizzle];
            slots[slot] = key[i];
            if constexpr (L::VB != 0) place[slot] = (unsigned short)(own + i * 32);
        }
        __syncwarp();
        clear_mine();
        before = tile;
        tile = m.next_tile;
    }
}

}  // namespace b200alg
