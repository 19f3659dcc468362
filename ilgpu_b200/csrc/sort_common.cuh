// What the kernels of the radix sort share: key transforms, sequenced values, and (slot_order.cuh) the
// check that ranks taken with atomics came out in order.
#pragma once

#include "common.cuh"
#include "slot_order.cuh"

namespace b200alg {

constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;

// Views of one sort call.  An in-place sort has in == out (possibly strided); an out-of-place
// sort leaves `in` untouched.  The alternate buffer is dense scratch of n elements.
template <typename K, typename V> struct SortBuffers {
    const K *in;
    K *out, *alt;
    const V *vin;
    V *vout, *valt;
    int64_t stride;             // of the input / output view
    int64_t n;                  // element count, or its upper bound when n_device is set
    const long long *n_device;  // element count in device memory (NULL: n is exact)
};
template <typename K, typename V> __device__ __forceinline__ int64_t effective_n(const SortBuffers<K, V> &io) {
    if (!io.n_device) return io.n;
    const long long v = *io.n_device;
    return v < 0 ? 0 : (v > io.n ? io.n : (int64_t)v);
}

// Values that are a function of the element's index (the reference's sequencers:
// IndexSequencer and the integer / Half / Float / Double sequencers, Sequencer.cs:37-72,
// Sequencers.tt:26-38): the pairs sort can produce them in its first pass instead of reading
// a value view.
enum : int { kSeqNone = 0, kSeqInteger = 1, kSeqFloating = 2 };
template <typename V> __device__ __forceinline__ V sequence_value(int kind, int64_t i) {
    if constexpr (sizeof(V) == 2) {
        if (kind == kSeqFloating) return (V)__half_as_ushort(__float2half_rn((float)i));
        return (V)i;
    } else if constexpr (sizeof(V) == 4) {
        if (kind == kSeqFloating) return (V)__float_as_uint((float)i);
        return (V)i;
    } else if constexpr (sizeof(V) == 8) {
        if (kind == kSeqFloating) return (V)__double_as_longlong((double)i);
        return (V)i;
    } else if constexpr (sizeof(V) == 1) {
        return (V)i;
    } else {
        return V{};
    }
}

// Key transform: bits = raw ^ (sign(raw) ? xor_neg : xor_pos) covers every key type of
// RadixSortOperations.tt:77-93 and the descending complement of :122-123.
template <typename K> struct KeyXform {
    K xor_neg, xor_pos;
    __host__ __device__ __forceinline__ K operator()(K raw) const {
        return raw ^ ((raw >> (sizeof(K) * 8 - 1)) ? xor_neg : xor_pos);
    }
    // The key of the transformed bits.  (No transform has constants that differ in their sign bit, so the sign
    // of bits ^ xor_pos is the key's.)
    __host__ __device__ __forceinline__ K raw(K bits) const {
        const K r = (K)(bits ^ xor_pos);
        return (r >> (sizeof(K) * 8 - 1)) ? (K)(bits ^ xor_neg) : r;
    }
};
// Ascending unsigned keys need no transform at all.
template <typename K> struct KeyIdentity {
    __host__ __device__ __forceinline__ K operator()(K raw) const { return raw; }
};

struct NoValue {};
template <typename V> struct ValueBytes { static constexpr int value = sizeof(V); };
template <> struct ValueBytes<NoValue> { static constexpr int value = 0; };

// The raw key whose transform is all ones: it fills a ragged tile up and sorts behind every real key.
template <typename K> __device__ __forceinline__ K padding_key(const KeyXform<K> &xf) {
    return xf.raw((K)~(K)0);
}
template <typename K> __device__ __forceinline__ K padding_key(const KeyIdentity<K> &) { return (K)~(K)0; }

// What a sort call works on, untyped (the entry points fill this in).
struct SortCall {
    const void *in_keys;
    void *out_keys;
    const void *in_values;
    void *out_values;
    int64_t stride;
    int64_t n;                  // element count, or its upper bound when n_device is set
    const long long *n_device;
    int value_seq;
    bool out_of_place;
};

// Parts of a sort's temp: the alternate buffers (dense, n elements), and how much lies in front of them.
struct SortScratch {
    void *alt_keys, *alt_values;
    int64_t control_bytes;
};

// A sort is made by the first of these that takes it (*taken), each in one launch, and else by passes over tiles:
// one block's (small_sort.cu);
int block_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xor_neg, uint64_t xor_pos, void *temp, bool *taken);

// by one partition into buckets that a block holds, 8-byte keys and 4-byte keys with values (sample_sort.cu);
int sample_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xor_neg, uint64_t xor_pos, void *temp,
                const SortScratch &scratch, bool *taken);

// by passes of a cluster or a grid that holds the view as a whole, keys of any size (small_sort.cu).
int resident_sort(cudaStream_t s, const SortCall &call, int key_bytes, int value_bytes, uint64_t xor_neg, uint64_t xor_pos, void *temp,
                  int64_t temp_bytes, bool *taken);

}  // namespace b200alg
