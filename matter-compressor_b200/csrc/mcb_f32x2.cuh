// mcb_f32x2.cuh -- packed single-precision adds and multiplies.
#pragma once
#include <cuda_runtime.h>

namespace mcb {

// Packed pairs: sm_100 executes two IEEE single-precision round-to-nearest
// adds or multiplies per instruction (add/sub/mul.rn.f32x2), each lane of the
// pair rounding exactly like its scalar __fadd_rn / __fmul_rn. One caution,
// measured with ptxas 12.9 on sm_100a: a packed multiply whose result feeds a
// packed add is contracted into a single-rounding packed FMA despite the .rn
// qualifiers (even inside one asm statement, and also when the product is
// written as fma with a -0 addend). Where a product is added in its own basic
// block (madd2 in mcb_decode.cu) the multiply is packed and the adds are scalar
// __fadd_rn, a combination that keeps both roundings; packed adds take sums, and
// products that arrive through a loop's back edge (lines4p and pass3 there,
// dct_lines and idct_lines in mcb_encode.cu). tests/test_transform_rounding.py holds
// inputs that a contraction anywhere in them changes.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

}  // namespace mcb
