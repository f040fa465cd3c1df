// llg_gateblock.cuh -- device code shared by the kernels that multiply in exact 8-bit digits on the
// tensor cores (llg_gateblock.cu, llg_adjblock.cu): barriers with bounded waits, shared-memory
// descriptors, digits of FP64 numbers.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "llg_common.cuh"
#include "llg_internal.h"

namespace llg {

namespace {

constexpr int kGroups = 128;     // groups per tile (the MMA's M)
constexpr int kAmps = 32;        // amplitudes per group
constexpr int kChunks = 4;       // K steps of 16 reals (8 amplitudes) per tile
constexpr int kRing = 5;         // chunk buffers
constexpr int kSlicerWarps = 8;
constexpr int kSliceBytes = kGroups * 16 * 2;  // one digit of one chunk
constexpr int kTmemCols = 512;                 // two accumulator sets
constexpr long kWaitLimit = 1L << 22;          // mbarrier polls before the kernel reports a timeout

// setmaxnreg to kTo registers from kFrom (an increase must not name fewer than there are)
template <int kFrom, int kTo>
__device__ __forceinline__ void set_registers() {
    if constexpr (kTo > kFrom) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTo));
    else if constexpr (kTo < kFrom) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTo));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// tcgen05 shared-memory descriptor, no swizzle (start, leading and stride byte offsets, version 1)
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 | (uint64_t)((sbo >> 4) & 0x3FFF) << 32 |
           (uint64_t)1 << 46;
}

// byte offset of element (row, c) of a rows x kreals fp16 operand: 8x8 cores of 128 bytes,
// K-direction cores adjacent, 8-row groups kreals / 8 cores apart
__device__ __forceinline__ uint32_t core_off(int row, int c, int kreals) {
    return (uint32_t)((row >> 3) * (kreals / 8) * 128 + (c >> 3) * 128 + (row & 7) * 16 + (c & 7) * 2);
}

// Column (K index) of part p (0 real, 1 imaginary) of amplitude j: 16 (j >> 3) + 8 (j & 1) + 2 ((j >> 1) & 3) + p,
// so that a slicer thread's four amplitudes of a chunk (j bit 0 fixed) fill one 8-wide core row.

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for the completion of phase `ph`; false when the limit ran out here or in another
// role (then *abort_s is set).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t ph, volatile int* abort_s) {
    for (long it = 0; it < kWaitLimit; ++it) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(bar), "r"(ph)
                     : "memory");
        if (done) return true;
        if ((it & 255) == 255 && *abort_s) return false;
    }
    *abort_s = 1;
    return false;
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t ph, volatile int* abort_s) {
    return __all_sync(0xffffffffu, mbar_wait(bar, ph, abort_s));
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// X = the 62-bit fixed-point integer of |x| against the group exponent eg (eg20 = eg 2^20 + 2^20 - 1;
// a shift by 64 or more gives zero), plus the digit bias.  eg > 64: zeros and subnormals need no
// care, their X is zero.
__device__ __forceinline__ uint64_t fixed_f64(double x, uint32_t eg20) {
    const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
    const uint32_t s = (eg20 - (h & 0x7FFFFFFFu)) >> 20;
    const uint32_t mh = (__funnelshift_l(l, h, 9) & 0x1FFFFFFFu) | 0x20000000u;
    uint64_t X = ((uint64_t)mh << 32) | (l << 9);
    asm("shr.u64 %0, %0, %1;" : "+l"(X) : "r"(s));
    return X + 0x8080808080808080ULL;
}
// the same for any group exponent: a zero or subnormal has no hidden bit and exponent 1
__device__ __noinline__ uint64_t fixed_f64_any(double x, int eg) {
    const uint64_t b = (uint64_t)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFULL;
    const int ex = (int)(b >> 52);
    const uint64_t m = (b & 0xFFFFFFFFFFFFFULL) | (ex ? 1ULL << 52 : 0ULL);
    return ((m << 9) >> min(eg - max(ex, 1), 63)) + 0x8080808080808080ULL;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) {
    uint32_t b;
    memcpy(&b, &v, 4);
    return b;
}
__device__ __forceinline__ __half2 h2_of(uint32_t b) {
    __half2 v;
    memcpy(&v, &b, 4);
    return v;
}

// The first kCount of four digits (bytes 3 .. 0 of the biased words) of eight reals as fp16, one
// 16-byte core row each, kStride bytes apart; sgn: +-1 of each pair of reals, bias: -1152 sgn
template <int kCount, int kStride = kSliceBytes>
__device__ __forceinline__ void digits4(const uint32_t (&w)[8], const __half2 (&sgn)[4], const __half2 (&bias)[4],
                                        unsigned char* dst) {
    uint32_t v[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const uint32_t t = __byte_perm(w[2 * p], w[2 * p + 1], 0x6273);
        const uint32_t u = __byte_perm(w[2 * p], w[2 * p + 1], 0x4051);
        v[0][p] = h2_bits(__hfma2(h2_of(__byte_perm(t, 0x64646464u, 0x4140)), sgn[p], bias[p]));
        v[1][p] = h2_bits(__hfma2(h2_of(__byte_perm(t, 0x64646464u, 0x4342)), sgn[p], bias[p]));
        v[2][p] = h2_bits(__hfma2(h2_of(__byte_perm(u, 0x64646464u, 0x4140)), sgn[p], bias[p]));
        v[3][p] = h2_bits(__hfma2(h2_of(__byte_perm(u, 0x64646464u, 0x4342)), sgn[p], bias[p]));
    }
#pragma unroll
    for (int k = 0; k < kCount; ++k)
        *reinterpret_cast<uint4*>(dst + k * kStride) = make_uint4(v[k][0], v[k][1], v[k][2], v[k][3]);
}

struct Fixed2 {  // a complex fixed-point number
    int64_t x, y;
};
// p a + q b with p, q in units of 2^-62, rounded once
__device__ __forceinline__ Fixed2 mix(Fixed2 p, Fixed2 a, Fixed2 q, Fixed2 b) {
    const __int128 half = (__int128)1 << 61;
    const __int128 re = (__int128)p.x * a.x - (__int128)p.y * a.y + (__int128)q.x * b.x - (__int128)q.y * b.y;
    const __int128 im = (__int128)p.x * a.y + (__int128)p.y * a.x + (__int128)q.x * b.y + (__int128)q.y * b.x;
    return {(int64_t)((re + half) >> 62), (int64_t)((im + half) >> 62)};
}

// Entry e (row-major) of a block's 2x2 gate in units of 2^-62, or of its inverse; cs: (cos, sin) of half
// the angle (kind 3).
__device__ __forceinline__ Fixed2 gate_entry(const BlockGate& o, int e, double2 cs, bool inverse) {
    double re = 0.0, im = 0.0;
    if (o.kind == 0) {
        const int from = inverse ? (e == 1 ? 2 : (e == 2 ? 1 : e)) : e;  // conjugate transpose
        re = o.m[2 * from];
        im = inverse ? -o.m[2 * from + 1] : o.m[2 * from + 1];
    } else if (o.kind == 3) {
        const double s = inverse ? -cs.y : cs.y;
        const bool off = e == 1 || e == 2;
        if (o.pad == 2) {  // diag(c - i s, c + i s)
            if (!off) re = cs.x, im = e == 0 ? -s : s;
        } else if (!off) {
            re = cs.x;
        } else if (o.pad == 1) {  // [c, -s; s, c]
            re = e == 1 ? -s : s;
        } else {  // [c, -i s; -i s, c]
            im = -s;
        }
    }
    return {__double2ll_rn(re * 0x1p62), __double2ll_rn(im * 0x1p62)};
}

}  // namespace

}  // namespace llg
