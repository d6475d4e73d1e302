// march_words.cuh -- the words that cross tiles of the marching sweeps through L2: 64 bits, 32 of
// payload and the tag of the sweep.  A 64-bit access is single, so a word with the right tag has its
// payload; stale words carry another sweep's tag.
#pragma once
#include <cuda_runtime.h>

namespace tg {

__device__ __forceinline__ ulonglong2 march_ld(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void march_st(ulonglong2* p, float x, float y, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(x)), "l"(t | __float_as_uint(y)));
}
// a double handed on as its two halves
__device__ __forceinline__ double march_double(const ulonglong2& w) { return __hiloint2double((int)(unsigned)w.y, (int)(unsigned)w.x); }

}  // namespace tg
