// Tile descriptors of the chained (decoupled look-back) kernels: scan and unique.
#pragma once

#include "common.cuh"

namespace b200alg {

enum : unsigned int { kInvalid = 0u, kAggregate = 1u, kInclusive = 2u };

// Tile descriptors, one record of kDescStride bytes per tile.  Records are spread out so that
// the polls of many successor tiles do not all land on one L2 line.  {flag, value} is one word of
// 64 bits (4-byte types) or 128 bits (8-byte types) that is read and written with single relaxed
// accesses.  (With flag and value in words of their own, ordered by release and acquire, the scan of
// 2^29 int64 took 2.9 ms, at half the rate of 4-byte types.)
constexpr int kDescStride = 128;
static_assert(kDescStride % 16 == 0, "a record holds one 128-bit word");

template <typename T, int BYTES = sizeof(T)> struct TileState;

template <typename T> struct TileState<T, 4> {
    unsigned char *base;
    int stride;
    __host__ __device__ TileState(void *b, int, int stride_ = kDescStride) : base((unsigned char *)b), stride(stride_) {}
    __device__ __forceinline__ unsigned long long *word(int tile) const {
        return (unsigned long long *)(base + (size_t)tile * stride);
    }
    __device__ __forceinline__ void publish(int tile, unsigned int flag, T v) {
        unsigned int bits;
        memcpy(&bits, &v, 4);
        st_relaxed_u64(word(tile), ((unsigned long long)flag << 32) | bits);
    }
    __device__ __forceinline__ unsigned int poll(int tile, T &v) {
        unsigned long long w = ld_relaxed_u64(word(tile));
        unsigned int bits = (unsigned int)w;
        memcpy(&v, &bits, 4);
        return (unsigned int)(w >> 32);
    }
};

template <typename T> struct TileState<T, 8> {
    unsigned char *base;
    int stride;
    __host__ __device__ TileState(void *b, int, int stride_ = kDescStride) : base((unsigned char *)b), stride(stride_) {}
    __device__ __forceinline__ void publish(int tile, unsigned int flag, T v) {
        unsigned long long bits;
        memcpy(&bits, &v, 8);
        asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}"
                     ::"l"(base + (size_t)tile * stride), "l"(bits), "l"((unsigned long long)flag) : "memory");
    }
    __device__ __forceinline__ unsigned int poll(int tile, T &v) {
        unsigned long long bits, flag;
        asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                     : "=l"(bits), "=l"(flag) : "l"(base + (size_t)tile * stride) : "memory");
        memcpy(&v, &bits, 8);
        return (unsigned int)flag;
    }
};

}  // namespace b200alg
