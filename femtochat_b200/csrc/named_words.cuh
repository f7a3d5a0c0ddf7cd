// Words that carry a name beside their data, 16 bytes wide, and counts without order: what blocks of one resident kernel hand to each other
// through L2.
#pragma once
#include <stdint.h>

// 12 bytes of data and the name, ONE 128-bit scalar, which the memory model never tears.
__device__ __forceinline__ uint4 named_load(const uint4* p) {
  uint4 v;
  asm volatile("{\n\t.reg .b128 a;\n\t.reg .b64 x, y;\n\tld.relaxed.gpu.global.b128 a, [%4];\n\tmov.b128 {x, y}, a;\n\tmov.b64 {%0, %1}, x;\n\tmov.b64 {%2, %3}, y;\n\t}"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void named_store(uint4* p, uint32_t a, uint32_t b, uint32_t c, uint32_t name) {
  asm volatile("{\n\t.reg .b128 a;\n\t.reg .b64 x, y;\n\tmov.b64 x, {%1, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b128 a, {x, y};\n\tst.relaxed.gpu.global.b128 [%0], a;\n\t}"
               ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(name) : "memory");
}
// A count of finished items.  It orders nothing: who reads it high enough knows that the items' words are on their way.
__device__ __forceinline__ void count_one(unsigned int* p) { asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }
__device__ __forceinline__ uint32_t counted_so_far(const unsigned int* p) {
  uint32_t n;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(p) : "memory");
  return n;
}
