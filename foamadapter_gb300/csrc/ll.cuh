// Data that crosses blocks of one running kernel with its epoch beside it: a value
// travels as two 8-byte words, each half the value and the 32-bit epoch, so a
// reader polls the data itself and needs no fence, counter or second read (a fence
// behind a block's vector stores costs 930 clocks; one such hop takes 720 clocks
// on a die and 1,060 across).  The memory is zero before the kernel starts and
// epochs count from 1.
#pragma once
#include <cuda_runtime.h>

struct GridBar {
    unsigned long long count;  // arrivals since the launch (never reset inside it)
    int abort, pad;
};

struct alignas(16) LLWord {  // one published value
    unsigned long long w0, w1;  // epoch << 32 | low half, epoch << 32 | high half
};
__device__ __forceinline__ void ll_store(LLWord* p, double v, unsigned epoch) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(e | (u & 0xffffffffull)),
                 "l"(e | (u >> 32))
                 : "memory");
}
__device__ __forceinline__ bool ll_load(const LLWord* p, unsigned epoch, double* v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    *v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (unsigned)(a >> 32) == epoch && (unsigned)(b >> 32) == epoch;
}

// a float travels as one word
__device__ __forceinline__ void ll_store(unsigned long long* p, float v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"(((unsigned long long)epoch << 32) | __float_as_uint(v))
                 : "memory");
}
__device__ __forceinline__ bool ll_load(const unsigned long long* p, unsigned epoch, float* v) {
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    *v = __uint_as_float((unsigned)a);
    return (unsigned)(a >> 32) == epoch;
}

// Bound of every wait: true when it has run out, here or in another block.
__device__ __forceinline__ bool ll_give_up(GridBar* gb, unsigned spins) {
    if ((spins & 63u) != 63u) return false;
    int ab;
    asm volatile("ld.relaxed.gpu.s32 %0, [%1];" : "=r"(ab) : "l"(&gb->abort) : "memory");
    if (ab) return true;
    if (spins < (1u << 23)) return false;  // seconds
    atomicExch(&gb->abort, 1);
    return true;
}


// A poll in two halves, for work during its round trip.
__device__ __forceinline__ void ll_issue(const LLWord* p, unsigned long long* a, unsigned long long* b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(*a), "=l"(*b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool ll_take(unsigned long long a, unsigned long long b, unsigned epoch, double* v) {
    if ((unsigned)(a >> 32) != epoch || (unsigned)(b >> 32) != epoch) return false;
    *v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return true;
}
