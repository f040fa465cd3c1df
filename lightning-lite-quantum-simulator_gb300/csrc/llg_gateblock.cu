// llg_gateblock.cu -- dense 5-qubit blocks of 16-byte states (IEEE complex128, double-float) on the
// fifth-generation tensor cores, as a warp-specialised pipeline.
//
// A block maps every group of 32 amplitudes that differ only in its five target qubits through a
// 32 x 32 complex matrix.  Over reals, a tile of 128 groups is one product D[g][r] = sum_c X[g][c]
// W[r][c] with W the 64 x 64 real form.  Both operands are cut into S balanced 8-bit digits (the
// Ozaki scheme: Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 2012), exact in fp16:
//     x = 2^(e_g - 1084) sum_i x_i 2^(56 - 8 i),   w = 2^(e_r - 6) sum_j w_j 2^(-8 j),
// where e_g is the group's largest biased exponent (the digits are the bytes of the 62-bit integer
// X = m 2^(9 - e_g + e) plus a bias), |x_0|, |w_0| <= 64 and the other digits at most 128 in size.
// The products with i + j <= S - 1 are accumulated by diagonal d = i + j in fp32: a diagonal is a
// sum of at most 64 (d + 1) products of integers, below 2^24, so every diagonal is exact.  The
// epilogue adds the diagonals in a 64-bit integer (D_0 .. D_4 exactly, the rest rounded at 2^-57 of
// the full scale) and converts once.  The error against the group's largest amplitude is that one
// rounding plus dropped products near 2^-58 (S = 8) or 2^-50 (S = 7, for double-float states, whose
// own significand has about 48 bits).
//
// What bounds it: 32 bytes of HBM per amplitude (5.1 ms per 2^30) against 36 slice products of
// M128 N64 K64 per tile (4608 clocks of the tensor pipe, 4.2 ms per 2^30).  Both need every phase to
// run at the same time, so the CTA (one per SM, persistent) has three roles:
//   * 8 slicer warps: load the tile into registers, agree on e_g, cut the amplitudes into digits and
//     write them in the no-swizzle K-major core-matrix layout.  A tile is 4 chunks of 8 amplitudes
//     per group (K = 16); a ring of 5 chunks lets the slicing run ahead of the products.  The next
//     tile's loads reuse a chunk's registers as soon as it is sliced.
//   * one MMA warp: D is computed in two halves of 16 output amplitudes, each with its own
//     accumulator set, so one half is recombined while the other is computed.  The gate's S slices
//     are stacked along N: X_i times [W_0 .. W_(S-1-i)] is one instruction whose columns are the
//     diagonals i .. S-1, so a state slice is read once per K step instead of S - i times (N = 64
//     products were bound by shared-memory reads, 48 clocks for 32 of tensor work).
//   * 16 (FP64) or 8 epilogue warps: tcgen05.ld, recombination, stores.
//   * one warp that prefetches into L2.
// Measured at 26 qubits, ms per 2^30 amplitudes, targets (5, 9, 13, 17, 25) / (0, 1, 2, 3, 4): FP64 8.5 /
// 12.6 (9.0k clocks per tile: the MMAs take 6.7k of them, sharing shared memory with the slicers'
// stores; FP64 pipe 43 % busy with the conversions), double-float 10.5 / 12.3 (bound by slicing); with the guards
// of partly filled tiles 8.7 / 12.7 and 10.7 / 12.3.
// With the lowest five qubits a warp's 32 accesses go to 32 lines.  The serial form that this replaced
// (one set of accumulators, load - slice - multiply - recombine one after the other on 16 warps)
// took 25k clocks per tile, 22 / 26 and 14 / 19 ms.
//
// Digits without integer work: the bytes u of |X| + 0x8080..80 are d + 128, and the fp16 with bits
// 0x6400 | u is 1024 + u, so a byte permute and one packed multiply-add (by the sign, minus 1152) make
// two digits.
// fp32 to integer without conversions (16 per clock and SM): diagonals 0 .. 4 are at most 2^22 in
// size, so adding 1.5 2^23 leaves the integer in the low bits of the float.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "llg_common.cuh"
#include "llg_gateblock.cuh"
#include "llg_internal.h"
#include "llg_launch.h"

namespace llg {

namespace {

template <int P>
struct Shape {
    static constexpr int S = P == LLG_F64 ? 8 : 7;             // digits per operand
    static constexpr int kChunkBytes = S * kSliceBytes;
    static constexpr int kWHalfBytes = S * 32 * 64 * 2;        // 32 S rows (digit, output) of 64 columns
    static constexpr int kSetStride = 256;                     // columns between the accumulator sets (32 S used)
    static constexpr size_t kSmem = (size_t)kRing * kChunkBytes + 2 * kWHalfBytes;
    // FP64: the conversion of the 64-bit sums (2 a clock and SM) leaves its warps waiting, so twice as
    // many with half the registers (8.54 -> 8.30 ms per 2^30; double-float loses 4 %)
    static constexpr int kEpiWarps = P == LLG_F64 ? 16 : 8;
    static constexpr int kStep = P == LLG_F64 ? 4 : 8;         // reals that an epilogue thread recombines at a time
    // the MMA warp, the prefetching warp and two more fill the last warpgroup
    static constexpr int kMmaWarp = kSlicerWarps + kEpiWarps;
    static constexpr int kThreads = (kMmaWarp + 4) * 32;
    // registers a thread at launch and by role (setmaxnreg): the roles' sum over the warps of a
    // scheduler is at most the launch's
    static constexpr int kLaunchRegs = P == LLG_F64 ? 72 : 96;
    static constexpr int kSlicerRegs = 112, kEpiRegs = P == LLG_F64 ? 64 : 104, kMmaRegs = P == LLG_F64 ? 24 : 40;
    static_assert(kSlicerWarps / 4 * kSlicerRegs + kEpiWarps / 4 * kEpiRegs + kMmaRegs <= kThreads / 128 * kLaunchRegs,
                  "the roles' registers come out of the launch's");
    static_assert(kThreads / 128 * kLaunchRegs * 128 <= 65536, "one CTA's registers");
};

// 2^e as a float for e in [-126, 127]
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// r 2^e for a result outside the range of the exponent-field addition
__device__ __noinline__ double scale_slow(double r, int e) { return ldexp(r, e); }

// element offset of every amplitude of a group (a kernel parameter: constant-bank operands)
struct TargetOffsets {
    uint64_t o[kAmps];
};

template <int P>
struct Elem;
template <>
struct Elem<LLG_F64> {
    using S = double2;
};
template <>
struct Elem<LLG_DF64> {
    using S = float4;
};

// `mirror` (nullptr: none): the device address of a mapped host buffer that also receives the
// output as FP64.
// A batch of states: row y of the grid is set y mod `sets`, whose state is 2^n elements from the
// first one's (the next `sets` rows: from `second`) and whose weights are `wstride` 16-byte words from
// the first set's.  max_exp (nullptr: none): per row, raised to the largest biased exponent stored (FP64).
// mixed (nullptr: none): blocks of different states in one launch, each CTA's given by its entry.
template <int P>
struct BlockBatch {
    typename Elem<P>::S* second;
    int sets;
    uint64_t wstride;
    uint32_t* max_exp;
    const MixedCta* mixed;
};

// kRows: the gate's rows have exponents of their own (any matrix); else all have exponent 0 (a product
// of unitary gates, entries at most 1).
// kMixed: the state, its block and the CTA's tiles come from batch.mixed, and the targets' offsets from shared
// memory instead of the parameters.
// kSplit: a cluster of two CTAs takes one tile, each slices it and computes half of the output amplitudes.
// A launch of few tiles is a chain of latencies, in which the products and the recombination are
// halved: 9.3 -> 7.6 us on 12 qubits, 1000 H and CNOT there 1159 -> 978 us, 20 layers of rotations and
// CNOTs on 17 qubits 430 -> 397 us.  Neither CTA stores before both have loaded.
template <int P, bool kRows, bool kMixed, bool kSplit>
__global__ void __launch_bounds__(Shape<P>::kThreads, 1)
    k_gate_block(typename Elem<P>::S* __restrict__ psi, int n, const __grid_constant__ TargetOffsets to, uint64_t tmask,
                 const uint4* __restrict__ weights, bool weights_ready, int* __restrict__ err_flag, double2* __restrict__ mirror,
                 BlockBatch<P> batch) {
    using T = Shape<P>;
    constexpr int S = T::S;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;                            // kRing chunks of S digits
    unsigned char* sW = smem + kRing * T::kChunkBytes;   // two halves of the gate's digits
    __shared__ uint64_t toff[kAmps];
    __shared__ int32_t eg_s[3][kGroups];  // group exponents, three tiles in turn
    __shared__ __align__(16) int32_t er_s[64];
    __shared__ __align__(8) uint64_t bars[2 * kRing + 8];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_flag, progress;
    volatile int* abort_s = &abort_flag;
    volatile int* progress_s = &progress;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kRing]);
    const uint32_t accfull0 = smem_u32(&bars[2 * kRing]), accempty0 = smem_u32(&bars[2 * kRing + 2]);
    const uint32_t egfull0 = smem_u32(&bars[2 * kRing + 4]), drain = smem_u32(&bars[2 * kRing + 7]);

    const int row_y = blockIdx.y;
    uint64_t tile0 = blockIdx.x, step = gridDim.x;  // this CTA's tiles
    if constexpr (kMixed) {
        const MixedCta& m = batch.mixed[blockIdx.x];
        psi += m.offset;
        weights += m.weights * batch.wstride;
        n = m.n;
        tmask = m.tmask;
        tile0 = m.first;
        step = m.step;
        if (tid < kAmps) {
            uint64_t o = 0;
            for (int b = 0; b < 5; ++b)
                if ((tid >> b) & 1) o |= 1ULL << m.q[b];
            toff[tid] = o;
        }
    } else {
        const int set_y = row_y % batch.sets;
        psi = (row_y < batch.sets ? psi : batch.second) + ((uint64_t)set_y << n);
        weights += set_y * batch.wstride;
        if (tid < kAmps) toff[tid] = to.o[tid];
    }
    const int half0 = kSplit ? (int)(blockIdx.x & 1) : 0, half1 = kSplit ? half0 + 1 : 2;
    if constexpr (kSplit) {
        tile0 = blockIdx.x >> 1;
        step = gridDim.x;  // one tile a cluster
    }
    bool met = !kSplit;  // the cluster's barrier is behind this thread
    auto loaded = [&]() {
        if constexpr (kSplit) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    };
    auto meet = [&]() {
        if (!met) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        met = true;
    };
    auto off = [&](int j) {
        if constexpr (kMixed) return toff[j];
        else return to.o[j];
    };
    // Launched while the previous kernel of the stream runs: everything up to the wait below touches
    // nothing that it writes (the weights only if they were ready before it began).
    if (!weights_ready) asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        uint4* dst = reinterpret_cast<uint4*>(sW);
        for (int i = half0 * T::kWHalfBytes / 16 + tid; i < half1 * T::kWHalfBytes / 16; i += T::kThreads) dst[i] = weights[i];
        if (tid < 16) reinterpret_cast<uint4*>(er_s)[tid] = weights[2 * T::kWHalfBytes / 16 + tid];
    }
    if (tid == 0) {
        abort_flag = 0;
        progress = 0;
        for (int i = 0; i < kRing; ++i) {
            mbar_init(full0 + 8 * i, kSlicerWarps);
            mbar_init(empty0 + 8 * i, 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(accfull0 + 8 * h, 1);
            mbar_init(accempty0 + 8 * h, T::kEpiWarps);
        }
        for (int i = 0; i < 3; ++i) mbar_init(egfull0 + 8 * i, kSlicerWarps);
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == T::kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the gate's digits are read by the MMAs
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_s;
    // registers of fewer than 12 qubits fill a part of their one tile: the other groups are zeros that nobody stores
    constexpr bool kPart = kSplit || kMixed;  // the forms that such registers take
    const int present = n >= 12 ? kGroups : 1 << (n - 5), groups = kPart ? present : kGroups;
    // (double-float's first loads ask in every form: as the compiler orders them without, targets 0 .. 4 take 13.1 ms per 2^30
    // amplitudes instead of 12.3)
    constexpr bool kAsk = kPart || P == LLG_DF64;
    const uint64_t ntiles = !kPart || n >= 12 ? (1ULL << (n - 5)) / kGroups : 1;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp < kSlicerWarps) {
        set_registers<T::kLaunchRegs, T::kSlicerRegs>();
        // ---- slicers: group g = 16 warp + (lane & 15), amplitudes j = 8 ks + 2 i + h with h = lane / 16:
        // a warp reads whole 32-byte sectors when the lowest target is qubit 0 (j and j + 1 adjacent),
        // and eight neighbouring lanes store one 128-byte core ----
        const int g = 16 * warp + (lane & 15), h = lane >> 4;
        int seen = 0;  // tiles begun, for the prefetching warp
        typename Elem<P>::S a[16];
        uint64_t tile = tile0;
        if (tile < ntiles) {
            const auto* pb = psi + (insert0_mask(tile * kGroups + (uint64_t)g, tmask) | (h ? off(1) : 0));
#pragma unroll
            for (int k = 0; k < 16; ++k) a[k] = !kAsk || g < present ? __ldcg(pb + off(2 * k)) : typename Elem<P>::S{};
        }
        int slot = 0, egb = 0;
        uint32_t phase = 1;  // of the slot's previous release: the first round needs no wait
        bool first = true, ok = true;
        for (; tile < ntiles && ok; tile += step, egb = egb == 2 ? 0 : egb + 1) {
            int eg;
            if constexpr (P == LLG_F64) {
                uint32_t mx = 0;
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    mx = max(mx, max((uint32_t)__double2hiint(a[k].x) & 0x7FFFFFFFu, (uint32_t)__double2hiint(a[k].y) & 0x7FFFFFFFu));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                eg = (int)(mx >> 20);
                if (eg == 0) {  // zeros (any scale gives zero) or subnormals
                    uint32_t any = 0;
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        any |= (uint32_t)__double2hiint(a[k].x) << 1 | (uint32_t)__double2loint(a[k].x) |
                               (uint32_t)__double2hiint(a[k].y) << 1 | (uint32_t)__double2loint(a[k].y);
                    eg = any ? 1 : 1023;
                }
                eg = min(eg, __shfl_xor_sync(0xffffffffu, eg, 16));  // one half zero, the other subnormal
            } else {
                // stored pairs may be unnormalised: TwoSum makes the high part the leading one
                float mx = 0.0f;
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const df re = two_sum(a[k].x, a[k].z), im = two_sum(a[k].y, a[k].w);
                    a[k] = make_float4(re.hi, im.hi, re.lo, im.lo);
                    mx = fmaxf(mx, fmaxf(fabsf(re.hi), fabsf(im.hi)));
                }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                // clamped so that the scale factor 2^(132 - e) below stays a normal float
                eg = max((int)(__float_as_uint(mx) >> 23), 8);
            }
            loaded();
            const uint64_t next = tile + step;
            if (tid == 0) *progress_s = ++seen;
            const auto* pb = psi + ((next < ntiles ? insert0_mask(next * kGroups + (uint64_t)g, tmask) : 0) | (h ? off(1) : 0));
#pragma unroll
            for (int ks = 0; ks < kChunks; ++ks) {
                if (!first && !warp_wait(empty0 + 8 * slot, phase, abort_s)) {
                    ok = false;
                    break;
                }
                if (ks == 0) {
                    // the slot's last reader, the epilogue three tiles back, ended before the products
                    // that freed this chunk were issued
                    if (h == 0) eg_s[egb][g] = eg;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(egfull0 + 8 * egb);
                }
                unsigned char* dst = sA + slot * T::kChunkBytes + core_off(g, 8 * h, 16);
                if constexpr (P == LLG_F64) {
                    uint32_t wh[8], wl[8];
                    __half2 sgn[4], bias[4];
                    const uint32_t eg20 = ((uint32_t)eg << 20) | 0xFFFFFu;
                    const bool small = __any_sync(0xffffffffu, eg <= 64);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const double2 v = a[4 * ks + i];
                        const uint64_t xr = small ? fixed_f64_any(v.x, eg) : fixed_f64(v.x, eg20);
                        const uint64_t xi = small ? fixed_f64_any(v.y, eg) : fixed_f64(v.y, eg20);
                        wh[2 * i] = (uint32_t)(xr >> 32);
                        wl[2 * i] = (uint32_t)xr;
                        wh[2 * i + 1] = (uint32_t)(xi >> 32);
                        wl[2 * i + 1] = (uint32_t)xi;
                        const uint32_t sg = __byte_perm((uint32_t)__double2hiint(v.x), (uint32_t)__double2hiint(v.y), 0x7733);
                        sgn[i] = h2_of((sg & 0x80008000u) | 0x3C003C00u);
                        bias[i] = __hmul2(sgn[i], __half2half2(__ushort_as_half(0xE480)));  // -1152
                    }
                    digits4<4>(wh, sgn, bias, dst);
                    digits4<4>(wl, sgn, bias, dst + 4 * kSliceBytes);
                } else {
                    // nearest-integer digits by the magic addition, from the high part and (from the
                    // fourth digit on) the low part added to what is left of it
                    const float sc = pow2f(132 - eg);  // the largest high part becomes 2^5 .. 2^6
#pragma unroll
                    for (int hv2 = 0; hv2 < 2; ++hv2) {  // four reals at a time: half a core row
                        float dg[S][4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float4 v = a[4 * ks + 2 * hv2 + (q >> 1)];
                            float r = ((q & 1) ? v.y : v.x) * sc, rest = 0.0f;
                            const float lo = ((q & 1) ? v.w : v.z) * sc * 16777216.0f;
#pragma unroll
                            for (int s = 0; s < S; ++s) {
                                if (s == 3) {
                                    const df t = two_sum(r, lo);
                                    r = t.hi;
                                    rest = t.lo;
                                }
                                if (s == 6) r = fmaf(rest, 16777216.0f, r);
                                dg[s][q] = __fsub_rn(__fadd_rn(r, 12582912.0f), 12582912.0f);
                                r = __fsub_rn(r, dg[s][q]) * 256.0f;
                            }
                        }
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const __half2 h0 = __floats2half2_rn(dg[s][0], dg[s][1]), h1 = __floats2half2_rn(dg[s][2], dg[s][3]);
                            uint2 o;
                            memcpy(&o.x, &h0, 4);
                            memcpy(&o.y, &h1, 4);
                            *reinterpret_cast<uint2*>(dst + s * kSliceBytes + 8 * hv2) = o;
                        }
                    }
                }
                if (next < ntiles) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[4 * ks + i] = __ldcg(pb + off(2 * (4 * ks + i)));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * slot);
                if (++slot == kRing) {
                    slot = 0;
                    phase ^= 1;
                    first = false;
                }
            }
        }
    } else if (warp < T::kMmaWarp) {
        set_registers<T::kLaunchRegs, T::kEpiRegs>();
        loaded();
        // ---- epilogue: tensor-memory lanes 32 (warp & 3) .. +31 (the groups), amplitudes
        // kStep / 2 of the half's 16 at a time ----
        const int row = 32 * (warp & 3) + lane, e = (warp - kSlicerWarps) >> 2;
        const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        const bool pair32 = off(1) == 1;  // amplitudes j and j + 1 (j even) are adjacent
        int erm = 1;
        if (kRows)
            for (int r = 0; r < 64; ++r) erm = max(erm, abs(er_s[r]));
        int egb = 0;
        uint32_t phase = 0, egphase = 0, largest = 0;
        bool ok = true;
        for (uint64_t tile = tile0; tile < ntiles && ok; tile += step, phase ^= 1) {
            const uint64_t base = insert0_mask(tile * kGroups + (uint64_t)row, tmask) | toff[T::kStep * e];
            if (!warp_wait(egfull0 + 8 * egb, egphase, abort_s)) break;
            const int eg = eg_s[egb][row];
            if (++egb == 3) {
                egb = 0;
                egphase ^= 1;
            }
            // the exponent-field addition is safe (results normal or zero)
            const bool all_fast = __all_sync(0xffffffffu, erm <= 32 && eg >= 128 && eg <= 1984);
#pragma unroll 1
            for (int half = half0; half < half1; ++half) {
                if (!warp_wait(accfull0 + 8 * half, phase, abort_s)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int p = 0; p < 2; ++p) {
                    const int col = T::kStep * (2 * e + p);  // within each diagonal's 32 columns
                    uint32_t v[S][T::kStep];
#pragma unroll
                    for (int d = 0; d < S; ++d) {
                        const uint32_t taddr = tlane + (uint32_t)(half * T::kSetStride + 32 * d + col);
                        if constexpr (T::kStep == 4)
                            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                                         : "=r"(v[d][0]), "=r"(v[d][1]), "=r"(v[d][2]), "=r"(v[d][3])
                                         : "r"(taddr));
                        else
                            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                         : "=r"(v[d][0]), "=r"(v[d][1]), "=r"(v[d][2]), "=r"(v[d][3]), "=r"(v[d][4]),
                                           "=r"(v[d][5]), "=r"(v[d][6]), "=r"(v[d][7])
                                         : "r"(taddr));
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (p == 1) {  // this warp has read the set
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(accempty0 + 8 * half);
                    }
                    const uint64_t pos = base | toff[16 * half + T::kStep / 2 * p];
                    typename Elem<P>::S out[T::kStep / 2];
#pragma unroll
                    for (int c = 0; c < T::kStep; ++c) {
                        const int er = kRows ? er_s[32 * half + col + c] : 0;
                        if constexpr (P == LLG_F64) {
                            // 2^44 sum_d 2^(-8 d) D_d: D_0 .. D_4 exact, D_5 .. D_7 rounded to an integer
                            const float magic = 12582912.0f;
                            const uint32_t b0 = __float_as_uint(__fadd_rn(__uint_as_float(v[0][c]), magic));
                            const uint32_t b1 = __float_as_uint(__fadd_rn(__uint_as_float(v[1][c]), magic));
                            const uint32_t b2 = __float_as_uint(__fadd_rn(__uint_as_float(v[2][c]), magic));
                            const uint32_t b3 = __float_as_uint(__fadd_rn(__uint_as_float(v[3][c]), magic));
                            const uint32_t b4 = __float_as_uint(__fadd_rn(__uint_as_float(v[4][c]), magic));
                            const float low = fmaf(__uint_as_float(v[7][c]), 0x1p-12f,
                                                   fmaf(__uint_as_float(v[6][c]), 0x1p-4f, __uint_as_float(v[5][c]) * 16.0f));
                            constexpr uint64_t kM = 0x4B400000ULL;
                            constexpr uint64_t kC = kM * ((1ULL << 28) + (1ULL << 20) + (1ULL << 12)) +
                                                    (kM * ((1ULL << 12) + (1ULL << 4)) << 32);
                            uint64_t acc = (uint64_t)(int64_t)__float2int_rn(low) - kC;
                            asm("mad.wide.u32 %0, %1, 4096, %0;" : "+l"(acc) : "r"(b4));
                            asm("mad.wide.u32 %0, %1, 1048576, %0;" : "+l"(acc) : "r"(b3));
                            asm("mad.wide.u32 %0, %1, 268435456, %0;" : "+l"(acc) : "r"(b2));
                            acc += (uint64_t)((b0 << 12) + (b1 << 4)) << 32;
                            double r = __ll2double_rn((long long)acc);
                            const int et = eg + er - 1078;
                            if (all_fast) {
                                const int hi = __double2hiint(r);
                                r = __hiloint2double(hi ? hi + (et << 20) : hi, __double2loint(r));
                            } else {
                                if (eg == 2047) r = __longlong_as_double(0x7FF8000000000000LL);  // an Inf or a NaN in the group
                                else r = scale_slow(r, et);
                                __syncwarp();  // the lanes parted
                            }
                            if (batch.max_exp) largest = max(largest, (uint32_t)__double2hiint(r) & 0x7FFFFFFFu);
                            if (c & 1) out[c >> 1].y = r;
                            else out[c >> 1].x = r;
                        } else {
                            // D_0 + 2^-8 D_1 + 2^-16 D_2 exactly, then 2^-24 (D_3 + ..) rounded
                            const float d0 = __uint_as_float(v[0][c]), d1 = __uint_as_float(v[1][c]) * 0x1p-8f;
                            const float d2 = __uint_as_float(v[2][c]) * 0x1p-16f, d3 = __uint_as_float(v[3][c]) * 0x1p-24f;
                            const float t = fmaf(__uint_as_float(v[6][c]), 0x1p-16f,
                                                 fmaf(__uint_as_float(v[5][c]), 0x1p-8f, __uint_as_float(v[4][c]))) * 0x1p-32f;
                            const df s1 = two_sum(d0, d1), s2 = two_sum(s1.hi, d2);
                            const df s3 = two_sum(__fadd_rn(s1.lo, s2.lo), d3);
                            const df s4 = two_sum(s2.hi, s3.hi);
                            const df acc = fast_two_sum(s4.hi, __fadd_rn(s4.lo, __fadd_rn(s3.lo, t)));
                            const int et = eg + er - 138;  // x = 2^(e_g - 132) .., w = 2^(e_r - 6) ..
                            const int e1 = max(min(et, 100), -100), e2 = max(min(et - e1, 100), -126);
                            const float f1 = pow2f(e1), f2 = pow2f(e2);
                            const float oh = acc.hi * f1 * f2, ol = acc.lo * f1 * f2;
                            if (c & 1) {
                                out[c >> 1].y = oh;
                                out[c >> 1].w = ol;
                            } else {
                                out[c >> 1].x = oh;
                                out[c >> 1].z = ol;
                            }
                        }
                    }
                    meet();
                    if (!kPart || row < groups) {
                        if (pair32) {
#pragma unroll
                            for (int c = 0; c < T::kStep / 2; c += 2) {
                                uint64_t w[4];
                                memcpy(w, &out[c], 32);
                                asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(psi + pos + off(c)), "l"(w[0]),
                                             "l"(w[1]), "l"(w[2]), "l"(w[3])
                                             : "memory");
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < T::kStep / 2; ++c) psi[pos + off(c)] = out[c];
                        }
                        if (mirror) {
#pragma unroll
                            for (int c = 0; c < T::kStep / 2; ++c) {
                                if constexpr (P == LLG_F64) mirror[pos + off(c)] = out[c];
                                else
                                    mirror[pos + off(c)] = make_double2((double)out[c].x + (double)out[c].z,
                                                                        (double)out[c].y + (double)out[c].w);
                            }
                        }
                    }
                    // the next tensor-memory loads are of the whole warp
                    if (kPart && groups < kGroups) __syncwarp();
                }
            }
        }
        if (batch.max_exp) {
            largest = __reduce_max_sync(0xffffffffu, largest);
            if (lane == 0) atomicMax(batch.max_exp + row_y, largest >> 20);
        }
    } else {
        set_registers<T::kLaunchRegs, T::kMmaRegs>();
        loaded();
        if (warp == T::kMmaWarp) {
            // ---- the MMA warp: the whole warp walks the loop (so that the descriptors are uniform), one
            // elected thread issues ----
            constexpr uint32_t idesc0 = (1u << 4) | ((uint32_t)(kGroups >> 4) << 24);  // fp32 from fp16, M = 128
            const uint64_t dA = tc_desc(smem_u32(sA), 128, 256), dW = tc_desc(smem_u32(sW), 128, 1024);
            uint32_t leader;
            asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(leader));
            int slot0 = 0;  // ring slot of the tile's first chunk
            uint32_t fphase = 0, aphase = 1;
            bool ok = true, any = false;
            for (uint64_t tile = tile0; tile < ntiles && ok; tile += step, aphase ^= 1) {
#pragma unroll 1
                for (int half = half0; half < half1 && ok; ++half) {
                    if (any && !warp_wait(accempty0 + 8 * half, aphase, abort_s)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    int slot = slot0;
                    uint32_t fp = fphase;
#pragma unroll 1
                    for (int ks = 0; ks < kChunks; ++ks) {
                        if (half == half0) {
                            if (!warp_wait(full0 + 8 * slot, fp, abort_s)) {
                                ok = false;
                                break;
                            }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        const uint64_t da = dA + (uint64_t)((uint32_t)(slot * T::kChunkBytes) >> 4);
                        const uint64_t dw = dW + (uint64_t)((uint32_t)(half * T::kWHalfBytes + ks * 256) >> 4);
                        const uint32_t dcol = tmem + (uint32_t)(half * T::kSetStride);
                        if (leader) {
#pragma unroll
                            for (int i = 0; i < S; ++i) {
                                const uint32_t acc = (ks > 0 || i > 0) ? 1u : 0u;
                                asm volatile(
                                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, "
                                    "p;\n}" ::"r"(dcol + (uint32_t)(32 * i)),
                                    "l"(da + (uint64_t)(i * (kSliceBytes >> 4))), "l"(dw),
                                    "r"(idesc0 | ((uint32_t)(32 * (S - i) >> 3) << 17)), "r"(acc)
                                    : "memory");
                            }
                            if (half == half1 - 1) tc_commit(empty0 + 8 * slot);
                            if (ks == kChunks - 1) tc_commit(accfull0 + 8 * half);
                        }
                        __syncwarp();
                        if (++slot == kRing) {
                            slot = 0;
                            fp ^= 1;
                        }
                    }
                    if (half == half1 - 1) {
                        slot0 = slot;
                        fphase = fp;
                    }
                }
                any = true;
            }
            // every product has ended before the columns are freed, after a timeout too
            if (leader) tc_commit(drain);
            for (long it = 0; it < kWaitLimit; ++it) {
                uint32_t done;
                asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                             : "=r"(done)
                             : "r"(drain), "r"(0u)
                             : "memory");
                if (done) break;
            }
        } else if (warp == T::kMmaWarp + 1) {
            // ---- a tile is runs of 2^cl contiguous amplitudes (at least 2 KB); lane j asks for the run that
            // starts at target offset j, two tiles ahead of the slicers, so that their loads come from L2
            // (issued by a slicer warp, the same instructions held it up for 3000 clocks a tile) ----
            const uint64_t in_tile = insert0_mask(kGroups - 1, tmask) | tmask;
            const int cl = __ffsll((long long)~in_tile) - 1;
            const bool run_start = (toff[lane] & ((1ULL << cl) - 1)) == 0;
            int begun = 0;
            for (uint64_t t = tile0 + step; t < ntiles && !*abort_s; t += step, ++begun) {
                for (int it = 0; it < 100000 && *progress_s < begun && !*abort_s; ++it) __nanosleep(200);
                if (run_start)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(psi + (insert0_mask(t * kGroups, tmask) | toff[lane])),
                                 "r"((uint32_t)sizeof(typename Elem<P>::S) << cl)
                                 : "memory");
            }
        }
    }
    __syncwarp();
    meet();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0 && abort_flag) atomicExch(err_flag, 1);
    if (warp == T::kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// ---- the gate's digits -------------------------------------------------------------------------
// Device layout of a block's weights: two halves (outputs 0-15 and 16-31) of 32 S rows (digit-major)
// by 64 columns in core-matrix order, then 64 row exponents.

// A CTA cuts the eight input amplitudes (16 columns) of one K chunk, blockIdx.y, of one block,
// blockIdx.x.  k_weights_matrix: the matrix m (row-major, in the order of the sorted targets), any finite
// entries.  k_weights_gates: the product of the block's gates, run on the identity's columns in shared
// memory in 64-bit fixed point (units of 2^-62, every 2x2 product rounded once from 128 bits): ten bits
// closer than FP64 where an error would repeat in every group, and faster here than FP64's two
// multiply-adds a clock and SM.  Gates of kind 3 take (cos, sin) of their half angle from `angles`, nocc
// entries a set, blockIdx.z the set; inverse: the inverse product (the gates' inverses, last first).

// Thread tid's core row: real output row tid / 2 (2 jo + po), inputs j = 8 ks + 2 i + h with h = tid & 1.
// x: the biased fixed-point magnitudes of its eight reals, neg: their signs in bit 31
template <int S>
__device__ __forceinline__ void put_core_row(unsigned char* wt, int ks, const uint64_t (&x)[8], const uint32_t (&neg)[8], int er) {
    const int row = threadIdx.x >> 1, h = threadIdx.x & 1;
    uint32_t wh[8], wl[8];
    __half2 sgn[4], bias[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        wh[i] = (uint32_t)(x[i] >> 32);
        wl[i] = (uint32_t)x[i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t sg = __byte_perm(neg[2 * i], neg[2 * i + 1], 0x7733);
        sgn[i] = h2_of((sg & 0x80008000u) | 0x3C003C00u);
        bias[i] = __hmul2(sgn[i], __half2half2(__ushort_as_half(0xE480)));
    }
    unsigned char* dst = wt + (row >> 5) * (S * 32 * 64 * 2) + core_off(row & 31, 16 * ks + 8 * h, 64);
    static_assert(kSliceBytes == 32 * 64 * 2, "a digit's 32 rows are kSliceBytes apart");
    digits4<4>(wh, sgn, bias, dst);
    digits4<S - 4>(wl, sgn, bias, dst + 4 * kSliceBytes);
    if (ks == 0 && h == 0) reinterpret_cast<int32_t*>(wt + 2 * (S * 32 * 64 * 2))[row] = er;
}

template <int S>
__global__ void __launch_bounds__(128) k_weights_matrix(const double2* __restrict__ m, unsigned char* __restrict__ wt) {
    __shared__ int eg_s[kAmps];
    const int tid = threadIdx.x, ks = blockIdx.y;
    if (tid < kAmps) {
        // both real rows of an output hold the same magnitudes
        uint32_t mx = 0;
        for (int j = 0; j < kAmps; ++j) {
            const double2 v = m[tid * kAmps + j];
            mx = max(mx, max((uint32_t)__double2hiint(v.x) & 0x7FFFFFFFu, (uint32_t)__double2hiint(v.y) & 0x7FFFFFFFu));
        }
        eg_s[tid] = max((int)(mx >> 20), 1);
    }
    __syncthreads();
    const int row = tid >> 1, h = tid & 1, jo = row >> 1, po = row & 1, eg = eg_s[jo];
    uint64_t x[8];
    uint32_t neg[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 v = m[jo * kAmps + 8 * ks + 2 * i + h];
        const double w[2] = {po ? v.y : v.x, po ? v.x : -v.y};  // real part in, imaginary part in
#pragma unroll
        for (int pi = 0; pi < 2; ++pi) {
            x[2 * i + pi] = fixed_f64_any(w[pi], eg);
            neg[2 * i + pi] = (uint32_t)__double2hiint(w[pi]);
        }
    }
    put_core_row<S>(wt, ks, x, neg, eg - 1022);
}

template <int S>
__global__ void __launch_bounds__(128)
    k_weights_gates(const BlockGate* __restrict__ gates, const BlockStep* __restrict__ steps,
                    const double2* __restrict__ matrices, const double2* __restrict__ angles, int nocc, bool inverse, unsigned char* __restrict__ wt, size_t stride) {
    constexpr int kStage = 32;  // gates whose coefficients are in shared memory
    __shared__ Fixed2 M[kAmps][9];
    __shared__ Fixed2 coef[kStage][4];  // 2x2 matrices, row-major
    __shared__ int4 what[kStage];       // kind, q0, q1, mask (kind 4: the matrix's first entry)
    __shared__ Fixed2 dense[256];       // a gate of kind 4
    const int tid = threadIdx.x, ks = blockIdx.y, c = tid & 7, p = tid >> 3;
    wt += ((size_t)blockIdx.x * gridDim.z + blockIdx.z) * stride;
    constexpr int64_t one = (int64_t)1 << 62;
    for (int r = p; r < kAmps; r += 16) M[r][c] = {r == 8 * ks + c ? one : 0, 0};
    const BlockStep st = steps[blockIdx.x];
    for (int k0 = 0; k0 < st.ngates; k0 += kStage) {
        const int cnt = min(kStage, st.ngates - k0);
        __syncthreads();
        // thread: entry (tid & 3) of gate tid / 4
        if (tid / 4 < cnt) {
            const int k = k0 + tid / 4, e = tid & 3;
            const BlockGate& o = gates[st.gate_begin + (inverse ? st.ngates - 1 - k : k)];
            coef[tid / 4][e] = gate_entry(o, e, o.kind == 3 ? angles[(size_t)blockIdx.z * nocc + o.q1] : make_double2(0.0, 0.0), inverse);
            if (e == 0) what[tid / 4] = make_int4(o.kind, o.q0, o.q1, o.kind == 4 ? o.pad : (int)o.mask);
        }
        __syncthreads();
        for (int k = 0; k < cnt; ++k) {
            const int4 o = what[k];
            if (o.x == 0 || o.x == 3) {
                const int b = o.y, r0 = ((p >> b) << (b + 1)) | (p & ((1 << b) - 1)), r1 = r0 | 1 << b;
                const Fixed2 x = M[r0][c], y = M[r1][c];
                M[r0][c] = mix(coef[k][0], x, coef[k][1], y);
                M[r1][c] = mix(coef[k][2], x, coef[k][3], y);
            } else if (o.x == 1) {
                if (p < 8) {
                    const int r = (int)insert0_mask((uint64_t)p, 1ULL << o.y | 1ULL << o.z) | 1 << o.y, r1 = r | 1 << o.z;
                    const Fixed2 x = M[r][c];
                    M[r][c] = M[r1][c];
                    M[r1][c] = x;
                }
            } else if (o.x == 4) {
                const int dim = 1 << o.z;
                for (int e = tid; e < dim * dim; e += 128) {
                    const double2 v = matrices[o.w + e];
                    dense[e] = {__double2ll_rn(v.x * 0x1p62), __double2ll_rn(v.y * 0x1p62)};
                }
                __syncthreads();
                // rows p and p + 16 of column c: the matrix's row picked by the row's bits, over the rows
                // that differ in them
                Fixed2 out[2];
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int r = p + 16 * w;
                    int mine = 0, rest = r;
                    for (int j = 0; j < o.z; ++j) {
                        const int b = (o.y >> (4 * j)) & 15;
                        mine |= ((r >> b) & 1) << j;
                        rest &= ~(1 << b);
                    }
                    __int128 re = (__int128)1 << 61, im = re;
                    for (int l = 0; l < dim; ++l) {
                        const Fixed2 d = dense[mine * dim + l];
                        if (d.x == 0 && d.y == 0) continue;
                        int from = rest;
                        for (int j = 0; j < o.z; ++j) from |= ((l >> j) & 1) << ((o.y >> (4 * j)) & 15);
                        const Fixed2 x = M[from][c];
                        re += (__int128)d.x * x.x - (__int128)d.y * x.y;
                        im += (__int128)d.x * x.y + (__int128)d.y * x.x;
                    }
                    out[w] = {(int64_t)(re >> 62), (int64_t)(im >> 62)};
                }
                __syncthreads();
                M[p][c] = out[0];
                M[p + 16][c] = out[1];
            } else {
                for (int r = p; r < kAmps; r += 16)
                    if ((r & o.w) == o.w) M[r][c] = {-M[r][c].x, -M[r][c].y};
            }
            __syncthreads();
        }
    }
    __syncthreads();
    const int row = tid >> 1, h = tid & 1, jo = row >> 1, po = row & 1;
    uint64_t x[8];
    uint32_t neg[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const Fixed2 v = M[jo][2 * i + h];
        const int64_t w[2] = {po ? v.y : v.x, po ? v.x : -v.y};  // real part in, imaginary part in
#pragma unroll
        for (int pi = 0; pi < 2; ++pi) {
            x[2 * i + pi] = (uint64_t)(w[pi] < 0 ? -w[pi] : w[pi]) + 0x8080808080808080ULL;
            neg[2 * i + pi] = (uint32_t)((uint64_t)w[pi] >> 32);
        }
    }
    put_core_row<S>(wt, ks, x, neg, 0);
}

int sm_count() {
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

std::atomic<int64_t> g_block_launches{0};

// ctas: CTAs a state (0: one per SM); sets states from psi and, unless nullptr, as many from `second`
template <int P, bool kRows, bool kMixed = false, bool kSplit = false>
cudaError_t launch(void* psi, int n, const BlockDesc& bd, const void* w, bool ready, int* err, cudaStream_t s, double* mirror,
                   int ctas, void* second, int sets, uint32_t* max_exp, const MixedCta* mixed = nullptr) {
    using T = Shape<P>;
    if (!kSplit && !kMixed && n < 12) return cudaErrorInvalidValue;  // whole tiles only
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_gate_block<P, kRows, kMixed, kSplit>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem);
    if (attr != cudaSuccess) return attr;
    TargetOffsets to;
    for (int j = 0; j < kAmps; ++j) {
        to.o[j] = 0;
        for (int b = 0; b < 5; ++b)
            if ((j >> b) & 1) to.o[j] |= 1ULL << bd.q[b];
    }
    const uint64_t most = ctas > 0 ? (uint64_t)ctas : (uint64_t)sm_count();
    const uint64_t ntiles = kMixed ? most : n >= 12 ? (1ULL << (n - 5)) / kGroups : 1;
    // programmatic dependent launch: the CTA's set-up (barriers, tensor memory, the gate's digits)
    // runs under the end of the stream's previous kernel
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 2;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(kSplit ? 2 * ntiles : ntiles < most ? ntiles : most), (unsigned)(second ? 2 * sets : sets));
    cfg.blockDim = dim3(T::kThreads);
    cfg.dynamicSmemBytes = T::kSmem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = kSplit ? 2 : 1;
    ++g_block_launches;
    return cudaLaunchKernelEx(&cfg, k_gate_block<P, kRows, kMixed, kSplit>, static_cast<typename Elem<P>::S*>(psi), n, to, bd.tmask,
                              static_cast<const uint4*>(w), ready, err, reinterpret_cast<double2*>(mirror),
                              BlockBatch<P>{static_cast<typename Elem<P>::S*>(second), sets, gate_block_weight_bytes(P) / 16, max_exp, mixed});
}

}  // namespace

int64_t gate_block_launches() { return g_block_launches.load(); }

bool gate_block_eligible(int P, int n) { return (P == LLG_F64 || P == LLG_DF64) && n >= kBlockMinQubits; }

namespace {
// f with the precision as a compile-time constant
template <class F>
auto by_precision(int P, F&& f) {
    if (P == LLG_F64) return f(std::integral_constant<int, LLG_F64>());
    return f(std::integral_constant<int, LLG_DF64>());
}
}  // namespace

size_t gate_block_weight_bytes(int P) {
    return by_precision(P, [](auto p) { return (size_t)2 * Shape<decltype(p)::value>::kWHalfBytes + 64 * sizeof(int32_t); });
}

cudaError_t launch_gate_block_matrix(int P, const double* d_matrix, void* d_weights, cudaStream_t s) {
    return by_precision(P, [&](auto p) {
        k_weights_matrix<Shape<decltype(p)::value>::S><<<dim3(1, kChunks), 128, 0, s>>>(
            reinterpret_cast<const double2*>(d_matrix), static_cast<unsigned char*>(d_weights));
        return cudaGetLastError();
    });
}

cudaError_t launch_gate_block_weights(int P, const BlockGate* d_gates, const BlockStep* d_steps, int nblocks, void* d_weights,
                                      cudaStream_t s, const double2* d_matrices, const double2* d_angles, int nocc, int sets,
                                      bool inverse) {
    return by_precision(P, [&](auto p) {
        k_weights_gates<Shape<decltype(p)::value>::S><<<dim3((unsigned)nblocks, kChunks, (unsigned)sets), 128, 0, s>>>(
            d_gates, d_steps, d_matrices, d_angles, nocc, inverse, static_cast<unsigned char*>(d_weights), gate_block_weight_bytes(P));
        return cudaGetLastError();
    });
}

cudaError_t launch_gate_block(int P, void* psi, int n, const BlockDesc& bd, const void* d_weights, bool rows, bool ready,
                              int* err_flag, cudaStream_t s, double* mirror) {
    return by_precision(P, [&](auto p) {
        constexpr int PP = decltype(p)::value;
        // two CTAs a tile as long as that leaves SMs over
        if (!rows && (n <= 12 || 2ULL << (n - 12) <= (uint64_t)sm_count()))
            return launch<PP, false, false, true>(psi, n, bd, d_weights, ready, err_flag, s, mirror, 0, nullptr, 1, nullptr);
        return rows ? launch<PP, true>(psi, n, bd, d_weights, ready, err_flag, s, mirror, 0, nullptr, 1, nullptr)
                    : launch<PP, false>(psi, n, bd, d_weights, ready, err_flag, s, mirror, 0, nullptr, 1, nullptr);
    });
}

cudaError_t launch_gate_block_batch(void* psi, void* second, int sets, int ctas, int n, const BlockDesc& bd,
                                    const void* d_weights, bool ready, uint32_t* max_exp, int* err_flag, cudaStream_t s) {
    return launch<LLG_F64, false>(psi, n, bd, d_weights, ready, err_flag, s, nullptr, ctas, second, sets, max_exp);
}

cudaError_t launch_gate_block_mixed(void* arena, int ctas, const MixedCta* d_ctas, const void* d_weights, int* err_flag,
                                    cudaStream_t s) {
    const BlockDesc none = {};
    return launch<LLG_F64, false, true>(arena, 12, none, d_weights, true, err_flag, s, nullptr, ctas, nullptr, 1, nullptr, d_ctas);
}

}  // namespace llg
