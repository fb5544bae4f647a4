// FP64 products on the integer pipes.
//
// GB300 executes one FP64 warp instruction per sub-partition every 64 cycles,
// while its integer and FP32 pipes take one every cycle or two, so a kernel bound by
// FP64 work leaves them idle (the FP64 advection: FP64 pipe 86 %, ALU 10 %).
// mul64i forms the IEEE 754 product, rounded to nearest with ties to even, from
// 32 x 32 -> 64 bit multiplications of the significands in about 40
// instructions: straight from the format (a normal binary64 is (-1)^s m 2^(e -
// 1075) with a 53-bit significand m), m_a m_b has 105 or 106 bits, the top 53
// are kept and the rest rounds.  Operands outside [2^-383, 2^129) in magnitude
// other than zeros (subnormals, infinities and NaNs among them) take the hardware
// product, so every result is the hardware's.  Alone it takes some 70 cycles of a
// sub-partition, beside FP64 instructions none of theirs: it pays where products
// are a good part of a kernel that the FP64 pipe bounds.
//
// Plain C++ so that the host can run it too.
#pragma once
#include <stdint.h>
#ifndef __CUDACC__
#include <string.h>
#endif

namespace cf {

#ifdef __CUDACC__
#define CF_HD __host__ __device__ __forceinline__
#else
#define CF_HD inline
#endif

CF_HD void split64(double d, uint32_t& hi, uint32_t& lo) {
#ifdef __CUDA_ARCH__
    hi = (uint32_t)__double2hiint(d);
    lo = (uint32_t)__double2loint(d);
#else
    uint64_t u;
    memcpy(&u, &d, 8);
    hi = (uint32_t)(u >> 32);
    lo = (uint32_t)u;
#endif
}
CF_HD double join64(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double d;
    memcpy(&d, &u, 8);
    return d;
#endif
}
// (hi : lo) << s, upper word, 0 <= s < 32
CF_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

CF_HD double mul64i(double a, double b) {
    uint32_t ah, al, bh, bl;
    split64(a, ah, al);
    split64(b, bh, bl);
    const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
    if (((ea - 0x28000000u) | (eb - 0x28000000u)) >= 0x20000000u) {
        // zero times a finite number is the usual case here
        if ((((ah << 1 | al) == 0u) & (eb != 0x7ff00000u)) | (((bh << 1 | bl) == 0u) & (ea != 0x7ff00000u)))
            return join64((ah ^ bh) & 0x80000000u, 0u);
        return a * b;
    }
    const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
    // A = m_a 2^11 in [2^63, 2^64), B = m_b in [2^52, 2^53): the product's upper
    // 64 bits are in [2^51, 2^53)
    const uint32_t Ah = shl_hi(al, ma, 11), Al = al << 11;
    const uint64_t w0 = (uint64_t)Al * bl;
    const uint64_t w1 = (uint64_t)Ah * bl + (w0 >> 32);
    const uint64_t w2 = (uint64_t)Al * mb + (uint32_t)w1;
    const uint64_t w3 = (uint64_t)Ah * mb + (w1 >> 32) + (w2 >> 32);
    const uint32_t th = (uint32_t)(w3 >> 32), tl = (uint32_t)w3, rh = (uint32_t)w2, rl = (uint32_t)w0;
    const uint32_t c = th >> 20, s = 1u - c;  // c: the product of the significands is 2 or more
    const uint32_t mh = shl_hi(tl, th, s), ml = shl_hi(rh, tl, s);
    // what follows the 53 bits: its upper word, with the lowest bit set for
    // anything below
    const uint32_t r = shl_hi(rl, rh, s) | ((rl << s) != 0u ? 1u : 0u);
    const uint64_t m = (((uint64_t)mh << 32) | ml) + (r > 0x80000000u - (ml & 1u) ? 1u : 0u);
    const uint32_t e = ea + eb + (c << 20) - 0x40000000u;  // m carries the hidden bit
    return join64((((uint32_t)(m >> 32) + e) | ((ah ^ bh) & 0x80000000u)), (uint32_t)m);
}

}  // namespace cf
