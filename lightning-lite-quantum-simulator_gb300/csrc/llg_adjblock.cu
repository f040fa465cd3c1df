// llg_adjblock.cu -- gradients of a whole 5-qubit block at once, for the adjoint method on IEEE
// complex128 states (llg_adjoint.cu).
//
// With U = G_m .. G_1 the block, psi and lambda the two vectors after it, and g running over the groups
// of 32 amplitudes that differ only in the block's targets,
//     R[a][b] = sum_g psi_g[a] conj(lambda_g[b])        (32 x 32)
// holds every inner product that the block's gradients need: after gate k the matrix is
// G_(k+1)^+ .. G_m^+ R G_m .. G_(k+1), and Im <lambda|P|psi> = Im tr(P R).  So the vectors are swept once a
// block (R, then U^+ applied by llg_gateblock.cu) instead of once a gate, and the per-gate work is on a
// 32 x 32 matrix (k_block_grads).
//
// R is a contraction over groups, on the tensor cores in the digits of llg_gateblock.cu: over reals
// D = X^T Y, X and Y the 64 real columns of the groups' psi and lambda.  A digit's 8 x 8 core (8 groups
// by 8 columns) is a K-major core of X and at the same time an MN-major core of X^T, so both operands
// are written as the slicers of the gate blocks write theirs.  The scale is one exponent a vector
// (FP64's block kernel raises it as it stores), so the digit products are sums over all groups alike:
// two of X's digits fill the MMA's M = 128 (rows 0-63 digit 2 p, rows 64-127 digit 2 p + 1), up to four of
// Y's its N = 256, and the columns 64 e of the accumulators collect the pairs with 2 p + j = e: diagonal
// e in the low rows, e + 1 in the high ones.  128 groups give integers below 2^24, exact in fp32; the
// epilogue adds them to 64-bit integers, each tile's sum rounded to what keeps the total from overflowing:
// 2^-62 of a bound on |psi| |lambda| (by Cauchy and Schwarz no part of a sum is larger; this serves states
// that sit in a few amplitudes) or 2^-62 of the CTA's groups at full scale, whichever is finer.  The CTAs' sums are added in 128 bits, and R is a
// pair of doubles.  In FP64 the sum would take 128 multiply-adds per amplitude, 0.2 ms per 2^20.
//
// What bounds k_cross: 32 bytes per amplitude pair against 20 digit products of M128 N64 K128 per 128
// groups (5120 clocks of the tensor pipe) and 65536 accumulators read back for each.  The accumulators
// fill tensor memory (512 columns), so products and epilogue of one CTA alternate.  Cutting both vectors into
// digits takes most instructions: two teams of eight warps take the chunks in turn, since two warps a
// scheduler issued on half of its cycles only (8 sets of 20 qubits: 173 us a block, with the two teams 115).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <type_traits>

#include "llg_adjblock.h"
#include "llg_common.cuh"
#include "llg_gateblock.cuh"
#include "llg_internal.h"
#include "llg_launch.h"

namespace llg {

namespace {

constexpr int kRRing = 6;                 // chunks in flight
constexpr int kRGroups = 16;              // groups per chunk (the MMA's K)
constexpr int kDigits = 8;
constexpr int kDigitBytes = kRGroups * 64 * 2;             // one digit of one vector's chunk
constexpr int kVecBytes = kDigits * kDigitBytes;           // 16 KB
constexpr int kRChunkBytes = 2 * kVecBytes;                // psi, lambda
constexpr int kTileChunks = kGroups / kRGroups;            // 8 chunks per drain of the accumulators
constexpr int kTeams = 2;                                  // of kSlicerWarps warps, which take the chunks in turn
constexpr int kRSlicers = kTeams * kSlicerWarps;
constexpr int kREpiWarps = 8;
constexpr int kRMmaWarp = kRSlicers + kREpiWarps;
constexpr int kRThreads = (kRMmaWarp + 4) * 32;
constexpr size_t kRSmem = (size_t)kRRing * kRChunkBytes;
constexpr int kRLaunchRegs = 72, kRSlicerRegs = 64, kREpiRegs = 104, kRMmaRegs = 40;
static_assert(4 * kRSlicerRegs + 2 * kREpiRegs + kRMmaRegs <= 7 * kRLaunchRegs, "the roles' registers come out of the launch's");
static_assert(kRRing % kTeams == 0, "a team keeps its slots");
static_assert(kRSmem >= 128 * 64 * sizeof(double), "the sums pass through the ring at the end");

struct CrossOffsets {
    uint64_t o[kAmps];
};

// the biased exponent that a vector's digits are cut against, from its largest one (zero vector: any scale)
__device__ __forceinline__ uint32_t cut_exponent(uint32_t e) { return e == 0 ? 1023u : max(e, 128u); }
// right shift of the tiles' sums (units of 2^-56 of the two scales' product), see above; `tiles` per CTA
__device__ __forceinline__ int cross_shift(int log2_bound, int tiles, uint32_t e0, uint32_t e1) {
    return max(min(log2_bound - 6 + 2044 - (int)e0 - (int)e1, 33 - __clz(tiles)), 0);
}

// exps: per set the largest biased exponents of psi and (sets further on) lambda.  partial: per set and
// CTA 32 x 32 complex sums in units of 2^(e_psi + e_lambda - 2100 + cross_shift).  log2_bound: of |psi| |lambda|;
// tiles: at most this many for a CTA.
__global__ void __launch_bounds__(kRThreads, 1)
    k_cross(const double2* __restrict__ psi, const double2* __restrict__ lam, int n, const __grid_constant__ CrossOffsets to,
            uint64_t tmask, int log2_bound, int tiles, const uint32_t* __restrict__ exps, Fixed2* __restrict__ partial, int* __restrict__ err_flag) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t coff[kTileChunks];  // element offset of a tile's chunks
    __shared__ __align__(8) uint64_t bars[2 * kRRing + 3];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_flag;
    volatile int* abort_s = &abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, set = blockIdx.y;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kRRing]);
    const uint32_t accfull = smem_u32(&bars[2 * kRRing]), accempty = smem_u32(&bars[2 * kRRing + 1]);
    const uint32_t drain = smem_u32(&bars[2 * kRRing + 2]);
    if (tid < kTileChunks) coff[tid] = insert0_mask((uint64_t)tid * kRGroups, tmask);
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < kRRing; ++i) {
            mbar_init(full0 + 8 * i, kSlicerWarps);
            mbar_init(empty0 + 8 * i, 1);
        }
        mbar_init(accfull, 1);
        mbar_init(accempty, kREpiWarps);
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kRMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_s;
    const uint64_t ntiles = (1ULL << (n - 5)) / kGroups;
    const int mine = (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);  // tiles of this CTA, at least 1
    const int chunks = mine * kTileChunks;

    if (warp < kRSlicers) {
        set_registers<kRLaunchRegs, kRSlicerRegs>();
        // ---- slicers: of a team, warps 0-3 psi, 4-7 lambda; group g of the chunk, amplitudes j = h + 2 i + 8 u ----
        const int team = warp / kSlicerWarps, vec = (warp >> 2) & 1, u = warp & 3, g = lane & 15, h = lane >> 4;
        const uint32_t eg = cut_exponent(exps[vec * gridDim.y + set]);
        const uint32_t eg20 = (eg << 20) | 0xFFFFFu;
        const double2* src = (vec ? lam : psi) + ((uint64_t)set << n) +
                             (insert0_mask((uint64_t)g, tmask) | (h ? to.o[1] : 0) | (u & 1 ? to.o[8] : 0) | (u & 2 ? to.o[16] : 0));
        const uint32_t at = (uint32_t)(vec * kVecBytes + (h + 2 * u) * 256 + (g >> 3) * 128 + (g & 7) * 16);
        double2 a[4];
        auto load = [&](int q) {
            const uint64_t tile = blockIdx.x + (uint64_t)(q >> 3) * gridDim.x;
            const double2* p = src + (insert0_mask(tile * kGroups, tmask) | coff[q & 7]);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = __ldcg(p + to.o[2 * i]);
        };
        load(team);  // chunks is a multiple of 8
        int slot = team;
        uint32_t phase = 1;
        bool first = true;
#pragma unroll 1
        for (int q = team; q < chunks; q += kTeams) {
            uint32_t wh[8], wl[8];
            __half2 sgn[4], bias[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 v = a[i];
                const uint64_t xr = fixed_f64(v.x, eg20), xi = fixed_f64(v.y, eg20);
                wh[2 * i] = (uint32_t)(xr >> 32);
                wl[2 * i] = (uint32_t)xr;
                wh[2 * i + 1] = (uint32_t)(xi >> 32);
                wl[2 * i + 1] = (uint32_t)xi;
                const uint32_t sg = __byte_perm((uint32_t)__double2hiint(v.x), (uint32_t)__double2hiint(v.y), 0x7733);
                sgn[i] = h2_of((sg & 0x80008000u) | 0x3C003C00u);
                bias[i] = __hmul2(sgn[i], __half2half2(__ushort_as_half(0xE480)));  // -1152
            }
            if (q + kTeams < chunks) load(q + kTeams);  // under the digits and the wait for a slot
            if (!first && !warp_wait(empty0 + 8 * slot, phase, abort_s)) break;
            unsigned char* dst = smem + slot * kRChunkBytes + at;
            digits4<4, kDigitBytes>(wh, sgn, bias, dst);
            digits4<4, kDigitBytes>(wl, sgn, bias, dst + 4 * kDigitBytes);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * slot);
            slot += kTeams;
            if (slot >= kRRing) {
                slot = team;
                phase ^= 1;
                first = false;
            }
        }
    } else if (warp < kRMmaWarp) {
        set_registers<kRLaunchRegs, kREpiRegs>();
        // ---- epilogue: rows 32 (warp & 3) + lane, columns 32 e .. +31 ----
        const int row = 32 * (warp & 3) + lane, e = (warp - kRSlicers) >> 2;
        const uint32_t tbase = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * e);
        const int shift = cross_shift(log2_bound, tiles, cut_exponent(exps[set]), cut_exponent(exps[gridDim.y + set]));
        const int64_t half = shift ? (int64_t)1 << (shift - 1) : 0;
        int64_t acc[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = 0;
        // a tile's sums in units of 2^-56: sum_e 2^(44 - 8 e) P_e in the low rows, 2^(36 - 8 e) in the high
        // ones (odd digits), whose lowest terms are rounded at once.  |P_0 .. P_3| <= 2^22: the integer is in
        // the low bits of the float plus 1.5 2^23
        auto add_tile = [&](auto odd) {
            constexpr bool kOdd = decltype(odd)::value;
            constexpr uint64_t kM = 0x4B400000ULL;
            constexpr uint64_t kC = kOdd ? kM * ((1ULL << 28) + (1ULL << 20) + (1ULL << 12)) + (kM << 36)
                                         : kM * ((1ULL << 28) + (1ULL << 20)) + (kM * ((1ULL << 12) + (1ULL << 4)) << 32);
#pragma unroll
            for (int cg = 0; cg < 8; ++cg) {
                uint32_t v[kDigits][4];
#pragma unroll
                for (int d = 0; d < kDigits; ++d)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(v[d][0]), "=r"(v[d][1]), "=r"(v[d][2]), "=r"(v[d][3])
                                 : "r"(tbase + (uint32_t)(64 * d + 4 * cg)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (cg == 7) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float magic = 12582912.0f;
                    const uint32_t b0 = __float_as_uint(__fadd_rn(__uint_as_float(v[0][c]), magic));
                    const uint32_t b1 = __float_as_uint(__fadd_rn(__uint_as_float(v[1][c]), magic));
                    const uint32_t b2 = __float_as_uint(__fadd_rn(__uint_as_float(v[2][c]), magic));
                    const uint32_t b3 = __float_as_uint(__fadd_rn(__uint_as_float(v[3][c]), magic));
                    const int b4 = __float2int_rn(__uint_as_float(v[4][c]));
                    const int low = __float2int_rn(fmaf(__uint_as_float(v[7][c]), kOdd ? 0x1p-20f : 0x1p-12f,
                                                        fmaf(__uint_as_float(v[6][c]), kOdd ? 0x1p-12f : 0x1p-4f,
                                                             __uint_as_float(v[5][c]) * (kOdd ? 0x1p-4f : 0x1p4f))));
                    uint64_t s = (uint64_t)(int64_t)low - kC;
                    if constexpr (kOdd) {
                        asm("mad.wide.s32 %0, %1, 16, %0;" : "+l"(s) : "r"(b4));
                        asm("mad.wide.u32 %0, %1, 4096, %0;" : "+l"(s) : "r"(b3));
                        asm("mad.wide.u32 %0, %1, 1048576, %0;" : "+l"(s) : "r"(b2));
                        asm("mad.wide.u32 %0, %1, 268435456, %0;" : "+l"(s) : "r"(b1));
                        s += (uint64_t)(b0 << 4) << 32;
                    } else {
                        asm("mad.wide.s32 %0, %1, 4096, %0;" : "+l"(s) : "r"(b4));
                        asm("mad.wide.u32 %0, %1, 1048576, %0;" : "+l"(s) : "r"(b3));
                        asm("mad.wide.u32 %0, %1, 268435456, %0;" : "+l"(s) : "r"(b2));
                        s += (uint64_t)((b0 << 12) + (b1 << 4)) << 32;
                    }
                    // the rounding bit apart: s alone may be near 2^63
                    acc[4 * cg + c] += ((int64_t)s >> shift) + (int64_t)(((int64_t)s & half) != 0);
                }
            }
        };
        uint32_t phase = 0;
        bool ok = true;
        for (int t = 0; t < mine; ++t, phase ^= 1) {
            if (!warp_wait(accfull, phase, abort_s)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (warp & 2) add_tile(std::true_type());
            else add_tile(std::false_type());
        }
        // ---- the CTA's 32 x 32 sums, through the ring (every product has been read) ----
        int64_t* D = reinterpret_cast<int64_t*>(smem);  // [row][64]
        if (ok) {
#pragma unroll
            for (int c = 0; c < 32; ++c) D[row * 64 + 32 * e + c] = acc[c];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kREpiWarps * 32) : "memory");
        if (ok) {
            Fixed2* out = partial + ((size_t)set * gridDim.x + blockIdx.x) * kAmps * kAmps;
            auto real = [&](int r, int c) { return D[r * 64 + c] + D[(r + 64) * 64 + c]; };
            for (int k = tid - kRSlicers * 32; k < kAmps * kAmps; k += kREpiWarps * 32) {
                const int ja = k >> 5, jb = k & 31;
                const int ra = 16 * (ja >> 3) + 8 * (ja & 1) + 2 * ((ja >> 1) & 3);
                const int cb = 16 * (jb >> 3) + 8 * (jb & 1) + 2 * ((jb >> 1) & 3);
                out[k] = {real(ra, cb) + real(ra + 1, cb + 1), real(ra + 1, cb) - real(ra, cb + 1)};
            }
        }
    } else {
        set_registers<kRLaunchRegs, kRMmaRegs>();
        if (warp == kRMmaWarp) {
            // ---- the MMA warp: fp32 from fp16, both operands MN-major, M = 128 ----
            constexpr uint32_t idesc0 = (1u << 4) | (1u << 15) | (1u << 16) | (8u << 24);
            const uint64_t d0 = tc_desc(smem_u32(smem), 128, 256);
            uint32_t leader;
            asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(leader));
            int slot = 0;
            uint32_t fphase = 0, aphase = 1;
            bool ok = true;
#pragma unroll 1
            for (int q = 0; q < chunks && ok; ++q) {
                if ((q & 7) == 0) {
                    if (q > 0 && !warp_wait(accempty, aphase, abort_s)) {
                        ok = false;
                        break;
                    }
                    aphase ^= 1;
                }
                if (!warp_wait(full0 + 8 * slot, fphase, abort_s)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = d0 + (uint64_t)((uint32_t)(slot * kRChunkBytes) >> 4);
                const uint64_t db = da + (uint64_t)(kVecBytes >> 4);
                if (leader) {
#pragma unroll
                    for (int p = 0; p < 4; ++p)
#pragma unroll
                        for (int j0 = 0; j0 < 8 - 2 * p; j0 += 4) {
                            const int nd = 8 - 2 * p - j0 < 4 ? 8 - 2 * p - j0 : 4;  // of lambda's digits
                            const uint32_t acc = (p > 0 || (q & 7) > 0) ? 1u : 0u;
                            asm volatile(
                                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, "
                                "p;\n}" ::"r"(tmem + (uint32_t)(64 * (2 * p + j0))),
                                "l"(da + (uint64_t)(2 * p * kDigitBytes >> 4)), "l"(db + (uint64_t)(j0 * kDigitBytes >> 4)),
                                "r"(idesc0 | ((uint32_t)(64 * nd >> 3) << 17)), "r"(acc)
                                : "memory");
                        }
                    tc_commit(empty0 + 8 * slot);
                    if ((q & 7) == 7) tc_commit(accfull);
                }
                __syncwarp();
                if (++slot == kRRing) {
                    slot = 0;
                    fphase ^= 1;
                }
            }
            if (leader) tc_commit(drain);
            for (long it = 0; it < kWaitLimit; ++it) {
                uint32_t done;
                asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                             : "=r"(done)
                             : "r"(drain), "r"(0u)
                             : "memory");
                if (done) break;
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0 && abort_flag) atomicExch(err_flag, 1);
    if (warp == kRMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// s 2^e as a double and what is left of it, as a double
__device__ __forceinline__ double2 pair_of(__int128 s, int e) {
    const double hi = (double)s;
    return make_double2(ldexp(hi, e), ldexp((double)(int64_t)(s - (__int128)hi), e));
}

// The CTAs' sums added exactly and scaled: R of set blockIdx.y, the high parts of its 32 x 32 entries, then
// the low ones.  NaN where a vector held one or an infinity.
__global__ void __launch_bounds__(128)
    k_cross_sum(const Fixed2* __restrict__ partial, int ctas, int log2_bound, int tiles, const uint32_t* __restrict__ exps,
                double2* __restrict__ R) {
    const int set = blockIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
    const longlong2* p = reinterpret_cast<const longlong2*>(partial) + (size_t)set * ctas * kAmps * kAmps + k;
    __int128 re = 0, im = 0;
#pragma unroll 4
    for (int c = 0; c < ctas; ++c) {
        const longlong2 v = __ldcg(p + (size_t)c * kAmps * kAmps);
        re += v.x;
        im += v.y;
    }
    const uint32_t e0 = exps[set], e1 = exps[gridDim.y + set];
    const uint32_t c0 = cut_exponent(e0), c1 = cut_exponent(e1);
    const int e = (int)(c0 + c1) - 2100 + cross_shift(log2_bound, tiles, c0, c1);
    double2 a = pair_of(re, e), b = pair_of(im, e);
    if (e0 == 2047 || e1 == 2047) a.x = b.x = __longlong_as_double(0x7FF8000000000000LL);
    double2* out = R + (size_t)set * 2 * kAmps * kAmps + k;
    out[0] = make_double2(a.x, b.x);
    out[kAmps * kAmps] = make_double2(a.y, b.y);
}

// largest biased exponent of the 2^n amplitudes of each set, psi then lambda
__global__ void __launch_bounds__(256)
    k_max_exponent(const double2* __restrict__ psi, const double2* __restrict__ lam, int n, int sets, uint32_t* __restrict__ exps) {
    const int y = blockIdx.y;
    const double2* v = (y < sets ? psi : lam) + ((uint64_t)(y % sets) << n);
    uint32_t mx = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < 1ULL << n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = v[i];
        mx = max(mx, max((uint32_t)__double2hiint(a.x) & 0x7FFFFFFFu, (uint32_t)__double2hiint(a.y) & 0x7FFFFFFFu));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(exps + y, mx >> 20);
}

// (cos, sin) of half of every parametrised gate's angle
__global__ void k_angles(const double* __restrict__ params, int nparams, const int* __restrict__ occ_code, int nocc, int sets,
                         double2* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sets * nocc) return;
    double s, c;
    sincos(0.5 * params[(size_t)(i / nocc) * nparams + occ_code[i % nocc] / 2], &s, &c);
    out[i] = make_double2(c, s);
}

// |0..0> in set blockIdx.x (its amplitudes were zeroed).  A set with an angle that is not finite starts from NaN, which
// the blocks carry to its energy and gradients: in the integers of its weights the angle would look like any other.
__global__ void __launch_bounds__(128)
    k_block_init(double2* __restrict__ psi, int n, const double2* __restrict__ angles, int nocc) {
    const int set = blockIdx.x;
    bool bad = false;
    for (int k = threadIdx.x; k < nocc; k += 128) bad = bad || !isfinite(angles[(size_t)set * nocc + k].x);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) psi[(uint64_t)set << n] = make_double2(bad ? __longlong_as_double(0x7FF8000000000000LL) : 1.0, 0.0);
}

// Gradients of block blockIdx.x's parametrised gates for set blockIdx.y, from R after the block: per gate,
// last to first, Im tr(P R), then R <- G^+ R G.  In fixed point against the Frobenius norm (60 bits; the
// norm is kept, so entries stay below 2^60 and traces below 2^63), every product rounded once: a gradient
// is a small difference of large traces, and the roundings of some 25 gates on one matrix do not
// average out as those of 2^n amplitudes do (in FP64 they cost 1.5e-15 of the gradients on 12 qubits).
__global__ void __launch_bounds__(128)
    k_block_grads(const double2* __restrict__ R, const BlockStep* __restrict__ steps, const BlockGate* __restrict__ gates,
                  const double2* __restrict__ angles, int nocc, double* __restrict__ grads) {
    __shared__ Fixed2 M[kAmps][kAmps + 1];
    __shared__ Fixed2 u[2][4];  // this gate's matrix and its inverse's
    __shared__ double sq_s[4];
    const int step = blockIdx.x, set = blockIdx.y, sets = gridDim.y, tid = threadIdx.x;
    const BlockStep st = steps[step];
    int first = st.ngates;  // the earliest parametrised gate: nothing before it is needed
    for (int k = st.ngates - 1; k >= 0; --k)
        if (gates[st.gate_begin + k].kind == 3) first = k;
    if (first == st.ngates) return;
    const double2* src = R + ((size_t)step * sets + set) * 2 * kAmps * kAmps;
    double sq = 0.0;
    for (int k = tid; k < kAmps * kAmps; k += 128) sq = fma(src[k].x, src[k].x, fma(src[k].y, src[k].y, sq));
    for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
    if ((tid & 31) == 0) sq_s[tid >> 5] = sq;
    __syncthreads();
    const double norm = sqrt(sq_s[0] + sq_s[1] + sq_s[2] + sq_s[3]);
    int ex = 0;
    if (norm > 0.0 && norm < 1e300) frexp(norm, &ex);  // norm < 2^ex
    for (int k = tid; k < kAmps * kAmps; k += 128) {
        const double2 h = src[k], l = src[kAmps * kAmps + k];
        M[k >> 5][k & 31] = {__double2ll_rn(ldexp(h.x, 60 - ex)) + __double2ll_rn(ldexp(l.x, 60 - ex)),
                             __double2ll_rn(ldexp(h.y, 60 - ex)) + __double2ll_rn(ldexp(l.y, 60 - ex))};
    }
    __syncthreads();
    for (int k = st.ngates - 1; k >= first; --k) {
        const BlockGate& o = gates[st.gate_begin + k];
        if (o.kind == 3 && tid < 32) {
            const int a = tid, m = 1 << o.q0;
            int64_t v;
            if (o.pad == 2) v = a & m ? -M[a][a].y : M[a][a].y;
            else if (o.pad == 0) v = M[a][a ^ m].y;
            else v = a & m ? -M[a][a ^ m].x : M[a][a ^ m].x;
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (tid == 0)
                grads[(size_t)set * nocc + o.q1] =
                    norm < 1e300 ? ldexp((double)v, ex - 60) : __longlong_as_double(0x7FF8000000000000LL);
        }
        if (k == first) break;
        if ((o.kind == 0 || o.kind == 3) && tid >= 32 && tid < 40)
            u[(tid - 32) >> 2][tid & 3] =
                gate_entry(o, tid & 3, o.kind == 3 ? angles[(size_t)set * nocc + o.q1] : make_double2(0.0, 0.0), tid >= 36);
        __syncthreads();
        if (o.kind == 0 || o.kind == 3) {
            const int b = o.q0;
            for (int w = tid; w < 512; w += 128) {  // rows: G^+
                const int r = w >> 5, c = w & 31, r0 = ((r >> b) << (b + 1)) | (r & ((1 << b) - 1)), r1 = r0 | 1 << b;
                const Fixed2 x = M[r0][c], y = M[r1][c];
                M[r0][c] = mix(u[1][0], x, u[1][1], y);
                M[r1][c] = mix(u[1][2], x, u[1][3], y);
            }
            __syncthreads();
            for (int w = tid; w < 512; w += 128) {  // columns: G
                const int c = w >> 5, r = w & 31, c0 = ((c >> b) << (b + 1)) | (c & ((1 << b) - 1)), c1 = c0 | 1 << b;
                const Fixed2 x = M[r][c0], y = M[r][c1];
                M[r][c0] = mix(u[0][0], x, u[0][2], y);
                M[r][c1] = mix(u[0][1], x, u[0][3], y);
            }
        } else if (o.kind == 1) {
            const uint64_t both = 1ULL << o.q0 | 1ULL << o.q1;
            for (int w = tid; w < 8 * kAmps; w += 128) {
                const int c = w & 31, r0 = (int)insert0_mask((uint64_t)(w >> 5), both) | 1 << o.q0, r1 = r0 | 1 << o.q1;
                const Fixed2 x = M[r0][c];
                M[r0][c] = M[r1][c];
                M[r1][c] = x;
            }
            __syncthreads();
            for (int w = tid; w < 8 * kAmps; w += 128) {
                const int r = w & 31, c0 = (int)insert0_mask((uint64_t)(w >> 5), both) | 1 << o.q0, c1 = c0 | 1 << o.q1;
                const Fixed2 x = M[r][c0];
                M[r][c0] = M[r][c1];
                M[r][c1] = x;
            }
        } else {
            const int m = (int)o.mask;
            for (int w = tid; w < kAmps * kAmps; w += 128) {
                const int r = w >> 5, c = w & 31;
                if (((r & m) == m) != ((c & m) == m)) M[r][c] = {-M[r][c].x, -M[r][c].y};
            }
        }
        __syncthreads();
    }
}

}  // namespace

int cross_ctas(int n, int sets, int sms) {
    const uint64_t tiles = (1ULL << (n - 5)) / kGroups;
    return block_ctas(tiles, sets, sms);
}

int block_ctas(uint64_t tiles, int sets, int sms) {
    // a CTA costs about one tile to start; the CTAs beyond one per SM run in turn
    int best = 1;
    double cost = 1e300;
    for (uint64_t k = 1; k <= tiles && k <= (uint64_t)(4 * sms); ++k) {
        const double rounds = std::ceil((double)(k * sets) / sms), per = std::ceil((double)tiles / (double)k) + 1.0;
        if (rounds * per < cost) {
            cost = rounds * per;
            best = (int)k;
        }
    }
    return best;
}

cudaError_t launch_cross(const void* psi, const void* lam, int n, int sets, int ctas, const BlockDesc& bd, int log2_bound,
                         const uint32_t* exps, void* partial, double2* R, int* err_flag, cudaStream_t s) {
    static const cudaError_t attr = cudaFuncSetAttribute(k_cross, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRSmem);
    if (attr != cudaSuccess) return attr;
    CrossOffsets to;
    for (int j = 0; j < kAmps; ++j) {
        to.o[j] = 0;
        for (int b = 0; b < 5; ++b)
            if ((j >> b) & 1) to.o[j] |= 1ULL << bd.q[b];
    }
    const int tiles = (int)(((1ULL << (n - 5)) / kGroups + ctas - 1) / ctas);
    k_cross<<<dim3((unsigned)ctas, (unsigned)sets), kRThreads, kRSmem, s>>>(
        static_cast<const double2*>(psi), static_cast<const double2*>(lam), n, to, bd.tmask, log2_bound, tiles, exps,
        static_cast<Fixed2*>(partial), err_flag);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_cross_sum<<<dim3(kAmps * kAmps / 128, (unsigned)sets), 128, 0, s>>>(static_cast<const Fixed2*>(partial), ctas, log2_bound, tiles, exps, R);
    return cudaGetLastError();
}

cudaError_t launch_max_exponent(const void* psi, const void* lam, int n, int sets, uint32_t* exps, cudaStream_t s) {
    const uint64_t blocks = std::min<uint64_t>(64, std::max<uint64_t>(1, (1ULL << n) >> 10));
    k_max_exponent<<<dim3((unsigned)blocks, (unsigned)(2 * sets)), 256, 0, s>>>(
        static_cast<const double2*>(psi), static_cast<const double2*>(lam), n, sets, exps);
    return cudaGetLastError();
}

cudaError_t launch_angles(const double* params, int nparams, const int* occ_code, int nocc, int sets, double2* out, cudaStream_t s) {
    k_angles<<<(sets * nocc + 255) / 256, 256, 0, s>>>(params, nparams, occ_code, nocc, sets, out);
    return cudaGetLastError();
}

cudaError_t launch_block_init(double2* psi, int n, const double2* angles, int nocc, int sets, cudaStream_t s) {
    k_block_init<<<sets, 128, 0, s>>>(psi, n, angles, nocc);
    return cudaGetLastError();
}

cudaError_t launch_block_grads(const double2* R, const BlockStep* steps, int nsteps, const BlockGate* gates, const double2* angles,
                               int nocc, int sets, double* grads, cudaStream_t s) {
    k_block_grads<<<dim3((unsigned)nsteps, (unsigned)sets), 128, 0, s>>>(R, steps, gates, angles, nocc, grads);
    return cudaGetLastError();
}

}  // namespace llg
