// Unique: removes consecutive duplicates in place and reports how many elements are left.
// Replaces UniqueKernel / CreateUnique (UniqueExtensions.cs:59-195), whose groups run one after
// the other (SequentialGroupExecutor) and whose first thread compacts a whole tile alone.
// Here every tile flags the elements that differ from their left neighbour, chains its count
// to the previous tiles with decoupled look-back, and writes its survivors where they belong,
// in place.  Equality follows Comparison{T} = first.CompareTo(second)
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
template <typename T> __device__ __forceinline__ T shfl_value_last(T v) {
    if constexpr (sizeof(T) <= 2 && !std::is_same<T, __half>::value) return (T)__shfl_sync(0xffffffffu, (unsigned int)v, 31);
    else return shfl_idx(v, 31);
}

// Bound: HBM (every element read once, every survivor written once).  A tile is 32 KB: 16-byte
// loads, four in flight per thread, in warp-striped order (vector j of lane l holds elements
// (warp * 4 * 32 + j * 32 + l) * VEC ... of the tile), so a warp reads whole lines; survivors meet
// in shared memory and leave in consecutive stores.  (Scalar loads of 16 consecutive elements per thread, with
// the survivors written to scratch and copied back by a second kernel, took 153 + 26 us for 5 * 10^7
// uint32 of which a quarter is kept; this 73 us, 81 us with three blocks per SM.)
//
// `kept` may be `in` itself (the in-place unique): a tile stores only once it knows its prefix,
// hence after every earlier tile has published its count and so has read its elements, and it
// stores at or below its own elements' places.  The one element a tile reads outside its own
// range is the last one of the tile before; only that element itself (unmoved) is stored there
// before this tile has published.
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
        left = shfl_value_last(v[j].t[VEC - 1]);
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

    if (starts) {  // where the runs begin (run-length encoding)
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            unsigned int slot = first_slot + local[j];
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if ((keep[j] >> e) & 1u) starts[(int64_t)s_prefix + slot++] = base + warp_first + (j * 32 + lane) * VEC + e;
        }
    }
    T *to = kept + s_prefix;
    for (unsigned int i = tid; i < aggregate; i += kUniqueThreads) to[i] = survivors[i];
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
static int run_unique(cudaStream_t s, void *data, int64_t n, void *out_count, void *temp, const UniqueLayout &L) {
    char *t = (char *)temp;
    B200ALG_CUDA_TRY(cudaMemsetAsync(temp, 0, (size_t)L.total, s));
    unique_select_kernel<T><<<(int)L.tiles, kUniqueThreads, 0, s>>>((const T *)data, n, (T *)data, nullptr, (long long *)out_count,
                                                                  (TempHeader *)temp, t + L.off_state, (int)L.tiles);
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

extern "C" int b200alg_unique(void *stream, void *data, int64_t n, int dtype, void *out_count, void *temp, int64_t temp_bytes) {
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
    case B200ALG_I8: case B200ALG_U8: return run_unique<uint8_t>(s, data, n, out_count, temp, L);
    case B200ALG_I16: case B200ALG_U16: return run_unique<uint16_t>(s, data, n, out_count, temp, L);
    case B200ALG_I32: case B200ALG_U32: return run_unique<uint32_t>(s, data, n, out_count, temp, L);
    case B200ALG_I64: case B200ALG_U64: return run_unique<uint64_t>(s, data, n, out_count, temp, L);
    case B200ALG_F16: return run_unique<__half>(s, data, n, out_count, temp, L);
    case B200ALG_F32: return run_unique<float>(s, data, n, out_count, temp, L);
    case B200ALG_F64: return run_unique<double>(s, data, n, out_count, temp, L);
    }
    return B200ALG_UNSUPPORTED;
}
