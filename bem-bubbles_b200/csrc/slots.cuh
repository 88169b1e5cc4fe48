// Exchange slots in global memory: a value and a sequence number, written and read as one 128-bit access, so
// that a reader that sees the number it waits for has the value with it: no fence, flag or barrier.
#pragma once

namespace bemb {

__device__ __forceinline__ void slot_store(ulonglong2* p, double v, unsigned long long seq) {
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(seq)
                 : "memory");
}
__device__ __forceinline__ void slot_load(const ulonglong2* p, unsigned long long& v, unsigned long long& seq) {
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(v), "=l"(seq)
                 : "l"(p)
                 : "memory");
}

}  // namespace bemb
