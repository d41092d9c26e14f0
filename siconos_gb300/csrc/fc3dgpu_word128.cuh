// 128-bit global words stored and loaded as one access (relaxed, device
// scope): a value and the stamp that says which sweep wrote it arrive
// together, so a reader needs no fence between them.
#pragma once
#include <cuda_runtime.h>

namespace fc3dgpu {

__device__ __forceinline__ void st_word128(void* p, unsigned long long lo, unsigned long long hi) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}
__device__ __forceinline__ void ld_word128(const void* p, unsigned long long& lo, unsigned long long& hi) {
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
}

// The same where `yes`, else lo and hi as they are: a predicated load, so that
// several of them are in flight together.
__device__ __forceinline__ void ld_word128_if(bool yes, const void* p, unsigned long long& lo, unsigned long long& hi) {
  asm volatile(
      "{\n .reg .pred q;\n .reg .b128 t;\n setp.ne.u32 q, %3, 0;\n mov.b128 t, {%0, %1};\n"
      " @q ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
      : "+l"(lo), "+l"(hi)
      : "l"(p), "r"((unsigned)yes)
      : "memory");
}

}  // namespace fc3dgpu
