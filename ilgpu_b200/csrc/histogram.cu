// Histogram: per-block privatised bins in shared memory, replicated per lane so that the
// shared-memory atomics of a warp fall into distinct banks, flushed with one global atomic
// per non-empty bin.
// Replaces HistogramWorkKernel (HistogramExtensions.cs:237-277), which issues one global
// atomic per element, and the overflow reporting of HistogramKernel (:176-198) with
// HistogramIncrement* (HistogramOperations.tt:30-41).
#include "common.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace b200alg {

namespace cg = cooperative_groups;

constexpr int kHistThreads = 512;
constexpr int64_t kHistSmemBytes = 48 * 1024;  // static limit, no opt-in needed

struct LocParams {
    double lo_d, scale_d, bins_d;  // bins_* = num_bins as a floating-point value
    float lo_f, scale_f, bins_f;
    long long num_bins;
    int last;  // num_bins - 1
    unsigned int inverse32;        // floor(2^32 / num_bins), all ones for one bin
    unsigned long long inverse64;  // floor(2^64 / num_bins), likewise
};

// ---- bin locators ---------------------------------------------------------------------
// run() returns the bin as an int (the bin count is below 2^31); kInRange = the result needs
// no bounds check.
template <typename T, int LOCATOR> struct Locate;

template <> struct Locate<float, B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(float x, const LocParams &p) {
        // floor, then clamp == clamp, then truncate; fmaxf(NaN, 0) = 0 sends NaN to bin 0
        const float t = fminf(fmaxf((x - p.lo_f) * p.scale_f, 0.0f), p.bins_f);
        return min(__float2int_rz(t), p.last);
    }
};
template <typename T> struct Locate<T, B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(T x, const LocParams &p) {
        const double t = ((double)x - p.lo_d) * p.scale_d;
        // Integers give no NaN, the conversion saturates, and what lies below 0 truncates to 0 or less: clamped as an
        // integer it saves a minimum and a maximum of doubles, which are several instructions each (2 * 10^8 int32,
        // 256 bins: 131 instead of 180 us).  Doubles are at the memory's rate either way (249 us against 256).
        if constexpr (std::is_integral<T>::value) return min(max(__double2int_rz(t), 0), p.last);
        else return min(__double2int_rz(fmin(fmax(t, 0.0), p.bins_d)), p.last);
    }
};
// x mod d by the rounded-down inverse of d: x * floor(2^k / d) / 2^k is less than one below x / d for x below 2^k, so
// the quotient is right or one too small, and the remainder or the remainder less d is the smaller one (2 * 10^8
// int32, 256 bins: 123 instead of 137 us with the division of the compiler).
__device__ __forceinline__ int remainder_of(unsigned int x, const LocParams &p) {
    const unsigned int d = (unsigned int)p.num_bins, r = x - __umulhi(x, p.inverse32) * d;
    return (int)min(r, r - d);
}
__device__ __forceinline__ int remainder_of(unsigned long long x, const LocParams &p) {
    const unsigned long long d = (unsigned long long)p.num_bins;
    const unsigned int r = (unsigned int)(x - __umul64hi(x, p.inverse64) * d);  // below 2 d, hence below 2^32
    return (int)min(r, r - (unsigned int)d);
}
template <> struct Locate<int32_t, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(int32_t x, const LocParams &p) { return remainder_of(x < 0 ? 0u - (unsigned int)x : (unsigned int)x, p); }
};
template <> struct Locate<int64_t, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(int64_t x, const LocParams &p) {
        return remainder_of(x < 0 ? 0ull - (unsigned long long)x : (unsigned long long)x, p);
    }
};
template <> struct Locate<uint32_t, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(uint32_t x, const LocParams &p) { return remainder_of((unsigned int)x, p); }
};
template <> struct Locate<uint64_t, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = true;
    static __device__ __forceinline__ int run(uint64_t x, const LocParams &p) { return remainder_of((unsigned long long)x, p); }
};
template <> struct Locate<float, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = false;
    static __device__ __forceinline__ int run(float x, const LocParams &p) {
        return (int)fabsf(fmodf(x, (float)p.num_bins));
    }
};
template <> struct Locate<double, B200ALG_LOCATOR_MODULO> {
    static constexpr bool kInRange = false;
    static __device__ __forceinline__ int run(double x, const LocParams &p) {
        return (int)fabs(fmod(x, (double)p.num_bins));
    }
};

// ---- adding a block's count to a global bin --------------------------------------------
// The reference raises the overflow flag when some single increment starts from
// MaxValue.  Adding c at once starts from old, old+1, ..., old+c-1 (wrapping), so the flag
// is raised iff the distance from old up to MaxValue is below c.
__device__ __forceinline__ bool add_to_bin(void *bins, long long b, unsigned long long c, int bin_dtype) {
    switch (bin_dtype) {
    case B200ALG_I32: {
        unsigned int old = atomicAdd((unsigned int *)bins + b, (unsigned int)c);
        return (unsigned long long)(unsigned int)(0x7FFFFFFFu - old) < c;
    }
    case B200ALG_U32: {
        unsigned int old = atomicAdd((unsigned int *)bins + b, (unsigned int)c);
        return (unsigned long long)(unsigned int)(0xFFFFFFFFu - old) < c;
    }
    case B200ALG_I64: {
        unsigned long long old = atomicAdd((unsigned long long *)bins + b, c);
        return (0x7FFFFFFFFFFFFFFFull - old) < c;
    }
    case B200ALG_U64: {
        unsigned long long old = atomicAdd((unsigned long long *)bins + b, c);
        return (0xFFFFFFFFFFFFFFFFull - old) < c;
    }
    case B200ALG_F32: {
        float old = atomicAdd((float *)bins + b, (float)c);
        return old == FLT_MAX;
    }
    default: {
        double old = atomicAdd((double *)bins + b, (double)c);
        return old == DBL_MAX;
    }
    }
}

// ---- shared-memory privatised kernel ---------------------------------------------------
template <typename T, int LOCATOR, bool VECTOR>
__global__ void __launch_bounds__(kHistThreads)
histogram_smem_kernel(const T *__restrict__ in, int64_t stride, int64_t n, LocParams p, void *bins, int bin_dtype,
                      int *overflow, int replicas) {
    // Bin b has `replicas` (a power of two, up to 32) counters at sh[b * replicas + r]; lane l
    // uses r = l % replicas.  With 32 replicas every lane of a warp has a bank of its own, so
    // an atomic instruction is one wavefront whatever the distribution of the data.
    extern __shared__ unsigned int sh[];
    const int nb = (int)p.num_bins;
    for (int i = threadIdx.x; i < nb * replicas; i += kHistThreads) sh[i] = 0u;
    grid_dependency_wait();
    __syncthreads();

    unsigned int *mine = sh + (threadIdx.x & (replicas - 1));
    const int rshift = 31 - __clz(replicas);
    const int64_t step = (int64_t)gridDim.x * kHistThreads;
    const int64_t gtid = (int64_t)blockIdx.x * kHistThreads + threadIdx.x;

    if (VECTOR) {
        constexpr int VEC = 16 / sizeof(T);
        union V { uint4 u; T t[VEC]; };
        int64_t head = (int64_t)(((16u - (unsigned)((uintptr_t)in & 15u)) & 15u) / sizeof(T));
        if (head > n) head = n;
        const uint4 *vin = reinterpret_cast<const uint4 *>(in + head);
        const int64_t nvec = (n - head) / VEC;
        const int64_t tail = head + nvec * VEC;
        int64_t i = gtid;
        for (; i + step < nvec; i += 2 * step) {
            V a, b;
            a.u = __ldcs(vin + i);
            b.u = __ldcs(vin + i + step);
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                const int ba = Locate<T, LOCATOR>::run(a.t[k], p);
                if (Locate<T, LOCATOR>::kInRange || (unsigned int)ba < (unsigned int)nb) atomicAdd(mine + (ba << rshift), 1u);
            }
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                const int bb = Locate<T, LOCATOR>::run(b.t[k], p);
                if (Locate<T, LOCATOR>::kInRange || (unsigned int)bb < (unsigned int)nb) atomicAdd(mine + (bb << rshift), 1u);
            }
        }
        for (; i < nvec; i += step) {
            V a;
            a.u = __ldcs(vin + i);
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                const int ba = Locate<T, LOCATOR>::run(a.t[k], p);
                if (Locate<T, LOCATOR>::kInRange || (unsigned int)ba < (unsigned int)nb) atomicAdd(mine + (ba << rshift), 1u);
            }
        }
        if (blockIdx.x == 0) {
            for (int64_t j = threadIdx.x; j < head; j += kHistThreads) {
                const int b = Locate<T, LOCATOR>::run(in[j], p);
                if (Locate<T, LOCATOR>::kInRange || (unsigned int)b < (unsigned int)nb) atomicAdd(mine + (b << rshift), 1u);
            }
            for (int64_t j = tail + threadIdx.x; j < n; j += kHistThreads) {
                const int b = Locate<T, LOCATOR>::run(in[j], p);
                if (Locate<T, LOCATOR>::kInRange || (unsigned int)b < (unsigned int)nb) atomicAdd(mine + (b << rshift), 1u);
            }
        }
    } else {
        for (int64_t i = gtid; i < n; i += step) {
            const int b = Locate<T, LOCATOR>::run(in[i * stride], p);
            if (Locate<T, LOCATOR>::kInRange || (unsigned int)b < (unsigned int)nb) atomicAdd(mine + (b << rshift), 1u);
        }
    }
    __syncthreads();

    bool of = false;
    for (int b = threadIdx.x; b < nb; b += kHistThreads) {
        unsigned long long c = 0;
        for (int r = 0; r < replicas; ++r) c += sh[b * replicas + ((r + threadIdx.x) & (replicas - 1))];
        if (c) of |= add_to_bin(bins, b, c, bin_dtype);
    }
    if (overflow && __syncthreads_or(of) && threadIdx.x == 0) atomicOr(overflow, 1);
}

// ---- one table per SM, for more bins than the kernel above holds ------------------------
// One 1024-thread block per SM keeps a table of all bins in most of the SM's shared memory:
// 32-bit counters, or, when those do not fit, 16-bit counters two to a word.  The blocks of a
// cluster add their tables up through distributed shared memory before they are flushed with one
// atomic per non-empty bin and cluster.  Bound: HBM for long inputs, the flush for short ones.
//
// 16-bit counters are below 2^14 at the start of a chunk of 3 * 2^14 elements, so they cannot
// wrap inside it; a sweep over the table after every chunk moves what a counter holds above that
// to the global bin.  (Counting with an atomic that returns the old value finds those counters
// without a sweep, but took twice as long per element.)
constexpr int kTableThreads = 1024;
constexpr int kTableBytes = 224 * 1024;
constexpr int kTableChunk = 3 << 14;   // elements of a block between two sweeps
constexpr int kTableMaxCluster = 4;

// Which kernel: the table where bins are many and the elements enough to pay for the flush.  Below
// 16 elements per bin one global atomic per element is as fast (int32 modulo 65536 bins, this kernel
// and the others: 19 against 9 us at 2^18 elements, 20.5 both at 2^20, 22 against 59 at 2^22, 49 against
// 391 at 3 * 10^7); up to 1024 bins the kernel above, whose smaller blocks are cleared and flushed
// sooner, unless the input does not fit in L2 and its locator does more than a few float operations
// per element (2^26 doubles, 256 bins: 84 us against 96 us; floats are at the HBM rate either way).
constexpr int64_t kTableLongInput = 1ll << 27;  // bytes
template <typename T, int LOCATOR> bool use_table(int64_t nb, int64_t n, bool dense) {
    if (nb * 2 > kTableBytes || n < 16 * nb) return false;
    if (!dense) return nb * 4 > kHistSmemBytes;  // few loads in flight here
    const bool costly = !(std::is_same<T, float>::value && LOCATOR == B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP);
    return (nb > 1024 && n >= (1 << 17)) || (costly && n * (int64_t)sizeof(T) >= kTableLongInput);
}

template <typename T, int LOCATOR, bool HALVES>
__global__ void __launch_bounds__(kTableThreads, 1)
histogram_table_kernel(const T *__restrict__ in, int64_t stride, int64_t n, LocParams p, void *bins, int bin_dtype, int *overflow) {
    extern __shared__ __align__(16) unsigned int table[];
    const int nb = (int)p.num_bins;
    const int quads = ((HALVES ? (nb + 1) / 2 : nb) + 3) / 4;  // 16-byte pieces of the table
    uint4 *table4 = reinterpret_cast<uint4 *>(table);
    for (int i = threadIdx.x; i < quads; i += kTableThreads) table4[i] = make_uint4(0u, 0u, 0u, 0u);
    grid_dependency_wait();
    __syncthreads();
    bool of = false;
    auto count = [&](T x) {
        const int b = Locate<T, LOCATOR>::run(x, p);
        if (!Locate<T, LOCATOR>::kInRange && (unsigned int)b >= (unsigned int)nb) return;
        if (HALVES) atomicAdd(table + (b >> 1), (b & 1) ? 0x10000u : 1u);
        else atomicAdd(table + b, 1u);  // lanes that meet in one bin cost little: they all add one
    };
    auto sweep = [&]() {
        __syncthreads();
        for (int i = threadIdx.x; i < quads; i += kTableThreads) {
            const uint4 q = table4[i];
            if ((q.x | q.y | q.z | q.w) & 0xC000C000u) {
                const unsigned int w[4] = {q.x & 0xC000C000u, q.y & 0xC000C000u, q.z & 0xC000C000u, q.w & 0xC000C000u};
#pragma unroll 1
                for (int k = 0; k < 8; ++k) {
                    const unsigned int c = (w[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu;
                    if (c) of |= add_to_bin(bins, i * 8 + k, c, bin_dtype);
                }
                table4[i] = make_uint4(q.x & 0x3FFF3FFFu, q.y & 0x3FFF3FFFu, q.z & 0x3FFF3FFFu, q.w & 0x3FFF3FFFu);
            }
        }
        __syncthreads();
    };
    if (stride == 1) {
        constexpr int VEC = 16 / sizeof(T);
        union V { uint4 u; T t[VEC]; };
        int64_t head = (int64_t)(((16u - (unsigned)((uintptr_t)in & 15u)) & 15u) / sizeof(T));
        if (head > n) head = n;
        const uint4 *vin = reinterpret_cast<const uint4 *>(in + head);
        const int64_t nvec = (n - head) / VEC;
        const int64_t tail = head + nvec * VEC;
        constexpr int NV = 4;  // 16-byte loads in flight per thread
        constexpr int ROUND = kTableThreads * NV * VEC;  // elements of a block per round
        static_assert(kTableChunk >= ROUND, "a chunk is whole rounds");
        const int64_t step = (int64_t)gridDim.x * kTableThreads;
        int pending = 0;
        auto whole = [&](int64_t first) { return first + (NV - 1) * step + kTableThreads <= nvec; };
        const int64_t begin = (int64_t)blockIdx.x * kTableThreads;
        // The next round is on its way while one is counted, unless counting is little (floats, 32-bit counters: 20000
        // bins 138 us with it, 134 without; 2 * 10^8 int32 into 65536 equal bins 197 with, 228 without).
        constexpr bool AHEAD = HALVES || !(std::is_same<T, float>::value && LOCATOR == B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP);
        V v[NV];
        if (AHEAD && whole(begin)) {
#pragma unroll
            for (int k = 0; k < NV; ++k) v[k].u = __ldcs(vin + begin + threadIdx.x + k * step);
        }
        for (int64_t first = begin; first < nvec; first += NV * step) {
            if (whole(first)) {  // bounds checks cost as much as the counting
                const bool more = AHEAD && whole(first + NV * step);
                const uint4 *ahead = vin + first + NV * step + threadIdx.x;
                if (!AHEAD) {
#pragma unroll
                    for (int k = 0; k < NV; ++k) v[k].u = __ldcs(vin + first + threadIdx.x + k * step);
                }
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    const V now = v[k];
                    if (more) v[k].u = __ldcs(ahead + k * step);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) count(now.t[e]);
                }
            } else {
                const uint4 *from = vin + first + threadIdx.x;
#pragma unroll 1
                for (int k = 0; k < NV; ++k)
                    if (first + threadIdx.x + k * step < nvec) {
                        V w;
                        w.u = __ldcs(from + k * step);
#pragma unroll
                        for (int e = 0; e < VEC; ++e) count(w.t[e]);
                    }
            }
            if (HALVES) {
                pending += ROUND;
                if (pending > kTableChunk - ROUND) {
                    sweep();
                    pending = 0;
                }
            }
        }
        if (blockIdx.x == 0) {  // the unaligned ends: fewer than 16 bytes each
            if (HALVES) sweep();
            if (threadIdx.x < head) count(in[threadIdx.x]);
            if (tail + threadIdx.x < n) count(in[tail + threadIdx.x]);
        }
    } else {
        int pending = 0;
        for (int64_t first = (int64_t)blockIdx.x * kTableThreads; first < n; first += (int64_t)gridDim.x * kTableThreads) {
            if (first + threadIdx.x < n) count(in[(first + threadIdx.x) * stride]);
            if (HALVES && (pending += kTableThreads) == kTableChunk) {
                sweep();
                pending = 0;
            }
        }
    }
    // every block of the cluster flushes its share of the bins
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int blocks = (int)cluster.num_blocks();
    const int share = ((nb + blocks - 1) / blocks + 1) / 2 * 2;
    const int lo = (int)cluster.block_rank() * share;
    const int hi = lo + share < nb ? lo + share : nb;
    const unsigned int *peer[kTableMaxCluster];
#pragma unroll
    for (int r = 0; r < kTableMaxCluster; ++r) peer[r] = cluster.map_shared_rank(table, r < blocks ? r : 0);
#pragma unroll 2
    for (int b = lo + threadIdx.x; b < hi; b += kTableThreads) {
        unsigned long long c = 0ull;
#pragma unroll
        for (int r = 0; r < kTableMaxCluster; ++r)
            if (r < blocks) c += HALVES ? (peer[r][b >> 1] >> ((b & 1) * 16)) & 0xFFFFu : peer[r][b];
        if (c) of |= add_to_bin(bins, b, c, bin_dtype);
    }
    cluster.sync();  // nobody leaves while its table is being read
    if (overflow && __syncthreads_or(of) && threadIdx.x == 0) atomicOr(overflow, 1);
}

// ---- fallback for bin counts that do not fit in shared memory ---------------------------
template <typename T, int LOCATOR>
__global__ void __launch_bounds__(256)
histogram_global_kernel(const T *__restrict__ in, int64_t stride, int64_t n, LocParams p, void *bins, int bin_dtype,
                        int *overflow) {
    grid_dependency_wait();
    bool of = false;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const int b = Locate<T, LOCATOR>::run(in[i * stride], p);
        if (Locate<T, LOCATOR>::kInRange || (unsigned int)b < (unsigned int)p.num_bins) of |= add_to_bin(bins, b, 1ull, bin_dtype);
    }
    if (overflow && __syncthreads_or(of) && threadIdx.x == 0) atomicOr(overflow, 1);
}

template <typename T, int LOCATOR>
static int launch_histogram(cudaStream_t s, const void *in, int64_t stride, int64_t n, const LocParams &p, void *bins,
                            int bin_dtype, void *overflow) {
    const int64_t nb = p.num_bins;
    const bool table = use_table<T, LOCATOR>(nb, n, stride == 1);
    if (nb * 4 <= kHistSmemBytes && !table) {
        int replicas = 1;
        while (replicas < 32 && (int64_t)replicas * 2 * nb * 4 <= kHistSmemBytes) replicas *= 2;
        const size_t smem = (size_t)replicas * nb * 4;
        constexpr int VEC = 16 / sizeof(T);
        const int64_t per_block = (int64_t)kHistThreads * (stride == 1 ? VEC * 2 : 2);
        int64_t want = ceil_div(n, per_block);
        const int64_t cap = (int64_t)sm_count() * (2048 / kHistThreads);
        const int blocks = (int)(want < 1 ? 1 : (want > cap ? cap : want));
        if (stride == 1)
            B200ALG_CUDA_TRY(launch_dependent(histogram_smem_kernel<T, LOCATOR, true>, dim3(blocks), dim3(kHistThreads), smem, s, (const T *)in, 1, n, p, bins, bin_dtype, (int *)overflow, replicas));
        else
            B200ALG_CUDA_TRY(launch_dependent(histogram_smem_kernel<T, LOCATOR, false>, dim3(blocks), dim3(kHistThreads), smem, s, (const T *)in, stride, n, p, bins, bin_dtype, (int *)overflow, replicas));
    } else if (table) {
        const bool halves = nb * 4 > kTableBytes;
        const size_t smem = (size_t)round_up(halves ? (nb + 1) / 2 * 4 : nb * 4, 16);
        auto kernel = halves ? histogram_table_kernel<T, LOCATOR, true> : histogram_table_kernel<T, LOCATOR, false>;
        // Clusters of four leave some SMs without one (their GPC holds no multiple of four) but
        // quarter the flush; long inputs would rather have every SM.
        const bool big = n * (int64_t)sizeof(T) >= kTableLongInput;
        const unsigned int cluster = big ? 2 : kTableMaxCluster;
        static ContextCache<int> resident[4];
        int blocks = 0;
        if (!resident[halves * 2 + big].find(&blocks)) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = cluster;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.blockDim = dim3(kTableThreads);
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            B200ALG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes));
            cfg.gridDim = dim3(cluster);
            cfg.dynamicSmemBytes = kTableBytes;
            int clusters = 0;
            B200ALG_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
            if (clusters < 1) return B200ALG_UNSUPPORTED;
            blocks = clusters * (int)cluster;
            resident[halves * 2 + big].store(blocks);
        }
        B200ALG_CUDA_TRY(launch_dependent_cluster(kernel, dim3(blocks), dim3(kTableThreads), smem, s, cluster, (const T *)in, stride, n, p, bins, bin_dtype, (int *)overflow));
    } else {
        int64_t want = ceil_div(n, 256 * 4);
        const int64_t cap = (int64_t)sm_count() * 8;
        const int blocks = (int)(want < 1 ? 1 : (want > cap ? cap : want));
        B200ALG_CUDA_TRY(launch_dependent(histogram_global_kernel<T, LOCATOR>, dim3(blocks), dim3(256), 0, s, (const T *)in, stride, n, p, bins, bin_dtype, (int *)overflow));
    }
    B200ALG_LAUNCH_CHECK();
    return B200ALG_OK;
}

template <typename T>
static int dispatch_locator(cudaStream_t s, const void *in, int64_t stride, int64_t n, int locator, const LocParams &p,
                            void *bins, int bin_dtype, void *overflow) {
    switch (locator) {
    case B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP:
        return launch_histogram<T, B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP>(s, in, stride, n, p, bins, bin_dtype, overflow);
    case B200ALG_LOCATOR_MODULO:
        return launch_histogram<T, B200ALG_LOCATOR_MODULO>(s, in, stride, n, p, bins, bin_dtype, overflow);
    }
    return B200ALG_UNSUPPORTED;
}

}  // namespace b200alg

using namespace b200alg;

extern "C" int b200alg_histogram(void *stream, const void *in, int64_t stride, int64_t n, int in_dtype, int locator,
                                 double lo, double hi, void *bins, int64_t num_bins, int bin_dtype, void *overflow) {
    // Argument checks mirror CreateHistogram's (HistogramExtensions.cs:322-338).
    if (!in || !bins) return B200ALG_INVALID_ARGUMENT;
    if (n < 0 || stride < 1 || num_bins < 1) return B200ALG_INVALID_ARGUMENT;
    if (!is_atomic_numeric(in_dtype) || !is_atomic_numeric(bin_dtype)) return B200ALG_UNSUPPORTED;
    if (n > kMaxElements || num_bins > INT32_MAX) return B200ALG_TOO_LARGE;
    if (locator == B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP && !(hi > lo)) return B200ALG_INVALID_ARGUMENT;
    if (((uintptr_t)in % dtype_bytes(in_dtype)) || ((uintptr_t)bins % dtype_bytes(bin_dtype)) ||
        (overflow && ((uintptr_t)overflow % 4)))
        return B200ALG_MISALIGNED;
    if (n == 0) return B200ALG_OK;
    LocParams p;
    p.num_bins = num_bins;
    p.lo_d = lo;
    p.scale_d = (double)num_bins / (hi - lo);
    p.lo_f = (float)lo;
    p.scale_f = (float)num_bins / ((float)hi - (float)lo);
    p.bins_d = (double)num_bins;
    p.bins_f = (float)num_bins;
    p.last = (int)(num_bins - 1);
    p.inverse32 = num_bins == 1 ? ~0u : (unsigned int)((1ull << 32) / (unsigned long long)num_bins);
    // (2^64 - 1) / d is 2^64 / d for every d that does not divide 2^64, and one less for those that do
    p.inverse64 = ~0ull / (unsigned long long)num_bins + (num_bins > 1 && (num_bins & (num_bins - 1)) == 0 ? 1 : 0);
    // float input computes in float: a range that collapses or overflows there would put every
    // element into an edge bin without a word
    if (locator == B200ALG_LOCATOR_EQUAL_WIDTH_CLAMP && in_dtype == B200ALG_F32 &&
        (!isfinite((float)lo) || !isfinite((float)hi) || !((float)hi > (float)lo) || !isfinite(p.scale_f) || !(p.scale_f > 0.0f)))
        return B200ALG_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    switch (in_dtype) {
    case B200ALG_I32: return dispatch_locator<int32_t>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    case B200ALG_U32: return dispatch_locator<uint32_t>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    case B200ALG_I64: return dispatch_locator<int64_t>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    case B200ALG_U64: return dispatch_locator<uint64_t>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    case B200ALG_F32: return dispatch_locator<float>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    case B200ALG_F64: return dispatch_locator<double>(s, in, stride, n, locator, p, bins, bin_dtype, overflow);
    }
    return B200ALG_UNSUPPORTED;
}
