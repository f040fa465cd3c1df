// llg_traj_f64.cuh -- weak-noise Kraus trajectories of IEEE complex128 states with one pass and one
// barrier per gate (included by llg_traj.cu).
//
// The general kernel runs a gate, a P(1) reduction, one thread's FP64 decision and a Kraus pass one after
// the other, each behind a barrier, and its FP64 pipe (2 multiply-adds a clock and SM) idled half of the
// time.  Without a jump everything but P(1) is known beforehand:
//   * A site pair's operator is diag(1, g) times a scalar, g = sqrt(1 - gamma) sqrt(1 - lambda) a constant.
//     Nobody applies it: qubit q's |1> amplitudes are held short of a pending factor p_q, which the host
//     follows through the circuit.  A rotation takes its qubit's into its two coefficients, a CNOT leaves
//     its control's and moves its target's by one product of a quarter of the amplitudes.
//   * P(1) is summed by the pass that writes the amplitudes, |a|^2 weighed by the product of the other
//     qubits' p^2: one multiply-add per amplitude with the (loop, warp) part and one multiply per thread
//     with the lane's, from tables of the host.  A CNOT's pass sums what both of its sites need.
//   * The sums are reduced as 64-bit fixed point (exact, so both CTAs and every warp get the same bits
//     without a broadcast), and a site jumps neither way exactly when P(1) is below a threshold of its two
//     uniforms, drawn ahead: an integer comparison that every warp makes for itself.
//   * The carried norm, the margins and the log are one extra warp's work, during the next pass, all in 64-bit
//     integers: one of its FP64 instructions would hold the sub-core's FP64 pipe for 64 clocks.  The same warp
//     brings the next step's record and tables into shared memory.
//   * A gate on a cluster's top qubit is preceded by an exchange of that qubit with the local one whose next
//     gate is farthest off.
// Within 2^-44 of the threshold, or above it, the pending factors are applied and the general code decides
// the gate's sites (amplitudes, P(1) and uniforms are the same, so are the jumps).
#pragma once

enum : int32_t { FS_SLOW = 0, FS_RT, FS_RC, FS_RXT, FS_RXC, FS_PHASE, FS_CNOT, FS_CZ, FS_SCALE, FS_SWAP };

// m 2^(e - 62), m in [2^62, 2^63)
struct Fix62 {
    uint64_t m;
    int64_t e;
};

// One step, in positions (bit positions of the held state).
struct alignas(16) FastStep {
    int32_t kind;
    int32_t q;       // target; CNOT / CZ: control; FS_SWAP: the local position
    int32_t t;       // CNOT / CZ: target
    int32_t gate;    // FS_SLOW: its gate
    int32_t tab;     // offset of the weights: by lane for rank 0, by lane for rank 1, by (index >> 5)
    int32_t ntab;    // doubles there
    int32_t pend;    // offset of the pending factors of all positions after the gate, before its sites, followed by
                     // the reciprocals of those after its sites without a jump; FS_SCALE: of the factors to apply
    int32_t flat;    // the weights do not depend on the loop index
    double c0, c1;   // rotation coefficients; phase (cos, sin); CNOT: c0 the factor of the (1, 1) amplitudes
    double k0, k1;   // CNOT / CZ: weights of the (1, 1) part in the first and in the second sum
    Fix62 f;         // real factor that the step leaves out, squared
    Fix62 f0, f1;    // f times p^2 of the target / control, of the second qubit
};

constexpr int kFastWorkers = 512;
constexpr int kFastThreads = kFastWorkers + 32;
constexpr int kFastPairs = kUChunk / 2;
constexpr int kTabLanes = 32;
// 13 local qubits: 12 index bits of a pass, or 8 loop bits of 32 threads in an FS_SCALE
constexpr int kTabMax = 256;
static_assert(kTabMax >= 2 * kTabLanes + 128 && kTabMax >= (1 << 13) / 32, "a step's table");
constexpr size_t kFastTabWords = (size_t)4 << 20;  // 32 MB of tables at most
constexpr double kFastKappa = 0.125;
constexpr int kFastMinQubits = 3;

struct FastNow {     // the extra warp's words for a step: (sig fs)^2 p^2 = m 2^(e - 62)
    uint64_t m0, m1;
    int32_t e0, e1;
    int32_t far;     // the held factor is to be applied after the step
};

struct FastShared {
    uint64_t part[2][2][kFastWorkers / 32][2];  // [parity][CTA][warp][sum]
    FastNow now[2];
    FastStep step[2];
    double tab[2][kTabMax];
    Fix62 sig2;                                 // the held state's factor, squared
    uint64_t thr[kFastPairs];                   // per site pair: no jump while P(1) 2^62 is below this
    uint64_t comp[kUChunk];                     // (1 - u) 2^62
};

// x 2^e as an integer, rounded to nearest; x >= 0
__device__ __forceinline__ uint64_t fixed_of(double x, int e) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7FF);
    if (ex == 0) return 0;
    const uint64_t m = (b & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);
    const int s = ex - 1075 + e;  // x 2^e = m 2^s
    if (s >= 0) return s > 10 ? ~0ULL >> 1 : m << s;
    if (s < -54) return 0;
    return ((m >> (-s - 1)) + 1) >> 1;
}
// sum over the warp of integers whose sum is below 2^63
__device__ __forceinline__ uint64_t warp_sum_u63(uint64_t x) {
    const uint32_t a = __reduce_add_sync(0xffffffffu, (uint32_t)x & 0x1FFFFFu);
    const uint32_t b = __reduce_add_sync(0xffffffffu, (uint32_t)(x >> 21) & 0x1FFFFFu);
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)(x >> 42));
    return (uint64_t)a + ((uint64_t)b << 21) + ((uint64_t)c << 42);
}
// a b 2^-s for 0 < s < 128
__device__ __forceinline__ uint64_t mul_shift(uint64_t a, uint64_t b, int s) {
    return (uint64_t)(((unsigned __int128)a * b) >> s);
}
__device__ __forceinline__ uint64_t mul62(uint64_t a, uint64_t b) { return mul_shift(a, b, 62); }
// a b for b in [2^62, 2^63) with exponent eb
__device__ __forceinline__ Fix62 fix_mul(const Fix62& a, uint64_t b, int64_t eb) {
    const uint64_t m = mul62(a.m, b);
    const int up = (int)(m >> 63);
    return {m >> up, a.e + eb + up};
}
__device__ __forceinline__ Fix62 fix_of(double x) {  // x > 0, normal
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return {((b & 0xFFFFFFFFFFFFFULL) | (1ULL << 52)) << 10, (int64_t)((b >> 52) & 0x7FF) - 1023};
}
__device__ __forceinline__ double fix_value(const Fix62& a) { return scalbn((double)a.m, (int)a.e - 62); }

struct FastTraj {
    double2* s;
    uint32_t NL;
    uint32_t tid, workers;
    int rank;

    __device__ static double norm(double2 a) { return fma(a.x, a.x, a.y * a.y); }
    __device__ static double norm(double2 a, double acc) { return fma(a.x, a.x, fma(a.y, a.y, acc)); }

    template <int KIND>
    __device__ static void rotate(double2& a, double2& b, double c0, double c1) {
        const double2 x = a, y = b;
        if constexpr (KIND == FS_RT) {
            a = make_double2(fma(-c0, y.x, x.x), fma(-c0, y.y, x.y));
            b = make_double2(fma(c1, x.x, y.x), fma(c1, x.y, y.y));
        } else if constexpr (KIND == FS_RC) {
            a = make_double2(fma(c0, x.x, -y.x), fma(c0, x.y, -y.y));
            b = make_double2(fma(c1, y.x, x.x), fma(c1, y.y, x.y));
        } else if constexpr (KIND == FS_RXT) {
            a = make_double2(fma(c0, y.y, x.x), fma(-c0, y.x, x.y));
            b = make_double2(fma(c1, x.y, y.x), fma(-c1, x.x, y.y));
        } else if constexpr (KIND == FS_RXC) {
            a = make_double2(fma(c0, x.x, y.y), fma(c0, x.y, -y.x));
            b = make_double2(fma(c1, y.x, x.y), fma(c1, y.y, -x.x));
        } else {  // FS_PHASE
            b = make_double2(fma(c0, y.x, -c1 * y.y), fma(c0, y.y, c1 * y.x));
        }
    }

    // one-qubit gate on st.q; returns this thread's weighed sum of |a_1|^2
    template <int KIND>
    __device__ double single(const FastStep& st, const double* tab) const {
        const double wl = tab[kTabLanes * rank + (tid & 31)];
        const double* wt = tab + 2 * kTabLanes;
        const double c0 = st.c0, c1 = st.c1;
        const uint32_t qb = 1u << st.q;
        double acc = 0.0;
        auto move = [&](uint32_t r) {
            const uint32_t j = ins0(r, qb);
            double2 a, b = s[j | qb];
            if constexpr (KIND != FS_PHASE) a = s[j];
            rotate<KIND>(a, b, c0, c1);
            if constexpr (KIND != FS_PHASE) s[j] = a;
            s[j | qb] = b;
            return b;
        };
        if (st.flat) {
#pragma unroll 4
            for (uint32_t r = tid; r < NL >> 1; r += workers) acc = norm(move(r), acc);
            return acc * (wl * wt[(tid & (NL / 2 - 1)) >> 5]);
        }
#pragma unroll 4
        for (uint32_t r = tid; r < NL >> 1; r += workers) {
            const double w = wt[r >> 5];
            acc = fma(w, norm(move(r)), acc);
        }
        return acc * wl;
    }

    // CNOT or CZ; s0: the control's sum, s1: the target's
    template <int KIND>
    __device__ void pair(const FastStep& st, const double* tab, double& s0, double& s1) const {
        double wl = tab[kTabLanes * rank + (tid & 31)];
        const double* wt = tab + 2 * kTabLanes;
        const uint32_t cb = 1u << st.q, tb = 1u << st.t, lo = min(cb, tb), hi = max(cb, tb);
        const double f = st.c0;
        double n10 = 0.0, n01 = 0.0, n11 = 0.0;
        auto move = [&](uint32_t r, double2& b, double2& c, double2& d) {
            const uint32_t j = ins0(ins0(r, lo), hi);
            b = s[j | tb];
            c = s[j | cb];
            d = s[j | cb | tb];
            if constexpr (KIND == FS_CNOT) {
                const double2 x = c;
                c = d;
                d = make_double2(f * x.x, f * x.y);
                s[j | cb] = c;
            } else {
                d = make_double2(PolF64::neg(d.x), PolF64::neg(d.y));  // not on the FP64 pipe
            }
            s[j | cb | tb] = d;
        };
        if (st.flat) {
#pragma unroll 4
            for (uint32_t r = tid; r < NL >> 2; r += workers) {
                double2 b, c, d;
                move(r, b, c, d);
                n01 = norm(b, n01);
                n10 = norm(c, n10);
                n11 = norm(d, n11);
            }
            wl *= wt[(tid & (NL / 4 - 1)) >> 5];
        } else {
#pragma unroll 2
            for (uint32_t r = tid; r < NL >> 2; r += workers) {
                const double w = wt[r >> 5];
                double2 b, c, d;
                move(r, b, c, d);
                n01 = fma(w, norm(b), n01);
                n10 = fma(w, norm(c), n10);
                n11 = fma(w, norm(d), n11);
            }
        }
        s0 = fma(st.k0, n11, n10) * wl;
        s1 = fma(st.k1, n11, n01) * wl;
    }

    // every amplitude times w[loop index] (the workers)
    __device__ void scale_loop(const double* w) const {
        uint32_t i = 1;
        for (uint32_t l = tid + workers; l < NL; l += workers, ++i) {
            const double f = w[i];
            if (f != 1.0) {
                const double2 a = s[l];
                s[l] = make_double2(a.x * f, a.y * f);
            }
        }
    }

    // every amplitude times the product of f[q] over its bits q; nl local positions (the workers)
    __device__ void scale_all(const double* __restrict__ f, int nl) const {
        const int lw = 31 - __clz(workers);  // workers = 2^lw
        double base = rank ? f[nl] : 1.0;
        for (int q = 0; q < min(lw, nl); ++q)
            if ((tid >> q) & 1) base *= f[q];
        for (uint32_t l = tid; l < NL; l += workers) {
            double w = base;
            for (int q = lw; q < nl; ++q)
                if ((l >> q) & 1) w *= f[q];
            const double2 a = s[l];
            s[l] = make_double2(a.x * w, a.y * w);
        }
    }
};

template <int CL>
__device__ void traj_fast_body(int n, const TrajGate* __restrict__ gates, const FastStep* __restrict__ steps, int nsteps,
                               const double* __restrict__ tabs, int zpos, KrausParams kp, uint64_t traj_begin, uint64_t n_traj,
                               double* __restrict__ z0_out, uint32_t* __restrict__ jumps_out, uint8_t* __restrict__ jump_log,
                               int64_t log_stride, double* __restrict__ margin_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double part2[2 * kPartWarps];
    __shared__ Decision dec;
    __shared__ double uni[kUChunk];
    __shared__ FastShared sh;
    Traj<PolF64, CL> T;
    T.nl = (CL == 2) ? n - 1 : n;
    T.NL = 1u << T.nl;
    T.s = reinterpret_cast<double2*>(smem_raw);
    T.rank = 0;
    T.remote = nullptr;
    uint64_t* other_part = nullptr;  // the partner's slots
    if (CL == 2) {
        cg::cluster_group cl = cg::this_cluster();
        T.rank = (int)cl.block_rank();
        T.remote = cl.map_shared_rank(T.s, T.rank ^ 1);
        other_part = cl.map_shared_rank(&sh.part[0][0][0][0], T.rank ^ 1);
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    FastTraj F;
    F.s = T.s;
    F.NL = T.NL;
    F.tid = tid;
    F.workers = blockDim.x - 32;
    F.rank = T.rank;
    const bool worker = tid < (int)F.workers;
    const int nw = (int)F.workers >> 5;
    const int npos = T.nl + (CL == 2);
    const double kappa = kp.gamma + kp.lambda - kp.gamma * kp.lambda;
    const uint64_t kfix = fixed_of(kappa, 62), gfix = fixed_of(kp.gamma, 62), lfix = fixed_of(kp.lambda * (1.0 - kp.gamma), 62);
    const uint64_t group = blockIdx.x / CL, ngroups = gridDim.x / CL;
    double min_margin = 1.0;
    uint64_t min_fix = 1ULL << 62;  // the extra warp's, as a fixed-point number
    // the record and the weights of step k, by the extra warp; visible after the next barrier
    auto fetch = [&](int k) {
        if (k >= nsteps) return;
        constexpr int kWords = sizeof(FastStep) / 16;
        static_assert(kWords <= 32 && sizeof(FastStep) % 16 == 0, "one 16-byte word a lane");
        if (lane < kWords)
            reinterpret_cast<uint4*>(&sh.step[k & 1])[lane] = __ldg(reinterpret_cast<const uint4*>(&steps[k]) + lane);
        __syncwarp();
        const int at = sh.step[k & 1].tab, count = sh.step[k & 1].ntab;
        for (int i = lane; i < count; i += 32) sh.tab[k & 1][i] = __ldg(tabs + at + i);
    };
    for (uint64_t tt = group; tt < n_traj; tt += ngroups) {
        const uint64_t traj = traj_begin + tt;
        for (uint32_t l = tid; l < T.NL; l += blockDim.x) T.s[l] = make_double2(l == 0 && T.rank == 0 ? 1.0 : 0.0, 0.0);
        if (tid == 0) sh.sig2 = fix_of(1.0);
        if (!worker) fetch(0);
        group_sync<CL>();
        uint64_t site = 0, u_begin = 0, u_end = 0;
        uint32_t jumps = 0;
        int par = 0;
        auto draw = [&](uint64_t first) {  // every thread, at the same site; first is even
            __syncthreads();
            for (int i = tid; i < kUChunk; i += blockDim.x) uni[i] = philox_u1(kp.seed, traj, first + i);
            __syncthreads();
            for (int i = tid; i < kUChunk; i += blockDim.x) sh.comp[i] = fixed_of(1.0 - uni[i], 62);
            for (int i = tid; i < kFastPairs; i += blockDim.x) {
                // no jump while u1 < 1 - gamma P and u2 < 1 - lambda p, p = (1 - gamma) P / (1 - gamma P)
                const double a = kp.gamma > 0.0 ? (1.0 - uni[2 * i]) / kp.gamma : 4.0;
                const double t = kp.lambda > 0.0 ? (1.0 - uni[2 * i + 1]) / kp.lambda : 4.0;
                const double b = t >= 1.0 ? 4.0 : t / ((1.0 - kp.gamma) + kp.gamma * t);
                const double m = fmin(fmin(a, b), 1.5) - 0x1p-44;
                sh.thr[i] = m > 0.0 ? fixed_of(m, 62) : 0;
            }
            u_begin = first;
            u_end = first + kUChunk;
            __syncthreads();
        };
        auto site_of = [&](int q, double sig) {  // the general code: a site whose amplitudes are true up to sig
            if (site + 1 >= u_end) draw(site);
            const double P1 = T.reduce(q, false, part2);
            if (tid == 0) decide<PolF64>(P1, sig, kp, uni[site - u_begin], uni[site + 1 - u_begin], &dec, &min_margin);
            __syncthreads();
            sig = dec.sig_next;
            const int code = dec.ad_jump | (dec.pd_jump << 1);
            T.kraus_apply(q, &dec);
            if (tid == 0 && T.rank == 0 && jump_log) jump_log[(int64_t)tt * log_stride + (int64_t)(site >> 1)] = (uint8_t)code;
            jumps += (code & 1) + (code >> 1);
            site += 2;
            return sig;
        };
        auto set_sig = [&](double sig) {  // every thread
            if (outside_carry_range<PolF64>(sig)) {
                T.rescale(sig);
                sig = 1.0;
            }
            __syncthreads();
            if (tid == 0) sh.sig2 = fix_of(sig * sig);
            group_sync<CL>();
        };
        for (int k = 0; k < nsteps; ++k) {
            const FastStep& st = sh.step[k & 1];  // its words were written before the last barrier
            const int kind = st.kind;
            if (kind == FS_SLOW || kind == FS_SCALE || kind == FS_SWAP) {
                if (!worker) fetch(k + 1);
                if (kind == FS_SCALE) {
                    if (worker && st.flat) F.scale_loop(sh.tab[k & 1]);
                    else if (worker) F.scale_all(tabs + st.pend, T.nl);
                } else if (kind == FS_SWAP) {
                    if (CL == 2) {  // (0, q = 1) and (1, q = 0) change places
                        const uint32_t qb = 1u << st.q, mine = T.rank ? 0u : qb;
                        double2 out[kMaxPerThread / 2];
                        group_sync<CL>();  // the partner's writes are complete
#pragma unroll
                        for (int i = 0; i < kMaxPerThread / 2; ++i) {
                            const uint32_t r = tid + i * blockDim.x;
                            if (r < T.NL >> 1) out[i] = T.remote[ins0(r, qb) | (qb ^ mine)];
                        }
                        group_sync<CL>();  // the partner has read this CTA's half
#pragma unroll
                        for (int i = 0; i < kMaxPerThread / 2; ++i) {
                            const uint32_t r = tid + i * blockDim.x;
                            if (r < T.NL >> 1) T.s[ins0(r, qb) | mine] = out[i];
                        }
                    }
                } else {
                    const TrajGate& G = gates[st.gate];
                    __syncthreads();  // the factor of the step before
                    double sig = sqrt(fix_value(sh.sig2)) * G.f;
                    T.gate(G.op);
                    for (int i = 0; i < G.nt; ++i) sig = site_of(G.q[i], sig);
                    set_sig(sig);
                }
                __syncthreads();
                continue;
            }
            const bool two = kind >= FS_CNOT;
            if (site + (two ? 3 : 1) >= u_end) draw(site);
            if (worker) {
                const double* tab = sh.tab[k & 1];
                double s0, s1 = 0.0;
                switch (kind) {
                    case FS_RT: s0 = F.single<FS_RT>(st, tab); break;
                    case FS_RC: s0 = F.single<FS_RC>(st, tab); break;
                    case FS_RXT: s0 = F.single<FS_RXT>(st, tab); break;
                    case FS_RXC: s0 = F.single<FS_RXC>(st, tab); break;
                    case FS_PHASE: s0 = F.single<FS_PHASE>(st, tab); break;
                    case FS_CZ: F.pair<FS_CZ>(st, tab, s0, s1); break;
                    default: F.pair<FS_CNOT>(st, tab, s0, s1); break;
                }
                __syncwarp();
                asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x) : "memory");  // the extra warp's words are there
                // S sig^2 fs^2 p^2 <= 1 and sig^2 fs^2 p^2 >= 2^e: x = S 2^(60 + e) <= 2^60
                const uint64_t x0 = warp_sum_u63(fixed_of(s0, 60 + sh.now[par].e0));
                const uint64_t x1 = two ? warp_sum_u63(fixed_of(s1, 60 + sh.now[par].e1)) : 0;
                if (lane == 0) {
                    sh.part[par][0][warp][0] = x0;
                    sh.part[par][0][warp][1] = x1;
                    if (CL == 2) {
                        uint64_t* o = other_part + ((par * 2 + 1) * (kFastWorkers / 32) + warp) * 2;
                        o[0] = x0;
                        o[1] = x1;
                    }
                }
            } else {
                if (lane == 0) {
                    FastNow& nx = sh.now[par];
                    const Fix62 sig2 = sh.sig2, a = fix_mul(sig2, st.f0.m, st.f0.e), b = fix_mul(sig2, st.f1.m, st.f1.e);
                    nx.m0 = a.m;
                    nx.e0 = (int32_t)a.e;
                    nx.m1 = b.m;
                    nx.e1 = (int32_t)b.e;
                    nx.far = sig2.e < -600 || sig2.e >= 600;
                }
                __syncwarp();
                asm volatile("bar.arrive 1, %0;" ::"r"(blockDim.x) : "memory");
                fetch(k + 1);
            }
            group_sync<CL>();
            // P(1) 2^62 of the first qubit, and of the second one times (1 - kappa P of the first)
            uint64_t P0, P1 = 0, left = 1ULL << 62;
            bool calm;
            {
                const int cta = lane >> 4, i = lane & 15;
                const bool in = i < nw && cta < CL;
                const uint64_t x0 = warp_sum_u63(in ? sh.part[par][cta][i][0] : 0);
                P0 = mul_shift(x0, sh.now[par].m0, 60);
                const uint64_t* thr = &sh.thr[(site - u_begin) >> 1];
                calm = P0 < thr[0];
                if (two) {
                    const uint64_t x1 = warp_sum_u63(in ? sh.part[par][cta][i][1] : 0);
                    P1 = mul_shift(x1, sh.now[par].m1, 60);
                    left -= mul62(P0, kfix);
                    calm = calm && P1 + (1ULL << 18) < mul62(thr[1], left);
                }
            }
            if (calm) {
                const bool far = sh.now[par].far;
                if (tid == (int)F.workers) {
                    // sig^2 fs^2 / (1 - x), x = kappa (P0 + P1) <= 1/4
                    uint64_t x = mul62(P0 + P1, kfix), r = (1ULL << 62) + x;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        x = mul62(x, x);
                        r += mul62(r, x);
                    }
                    sh.sig2 = fix_mul(fix_mul(sh.sig2, st.f.m, st.f.e), r, 0);
                    uint64_t P = P0, l = 1ULL << 62;
                    for (int i = 0; i < (two ? 2 : 1); ++i) {
                        // margins |u1 - 1 + gamma P / l| and |u2 - 1 + lambda (1 - gamma) P / (l - gamma P)|, times the
                        // denominators; the quotients only where they may be a new minimum
                        const int u = (int)(site - u_begin) + 2 * i;
                        const uint64_t gp = mul62(gfix, P);
                        const int64_t a = (int64_t)(mul62(sh.comp[u], l) - gp), b = (int64_t)(mul62(sh.comp[u + 1], l - gp) - mul62(lfix, P));
                        const uint64_t m = min((uint64_t)llabs(a), (uint64_t)llabs(b));
                        if (m < min_fix) {
                            const double pd = (double)P / (double)l;
                            const double s_ad = 1.0 - kp.gamma * pd, s_pd = 1.0 - kp.lambda * ((1.0 - kp.gamma) * pd / s_ad);
                            min_margin = fmin(min_margin, fmin(fabs(uni[u] - s_ad), fabs(uni[u + 1] - s_pd)));
                            min_fix = fixed_of(min_margin, 62);
                        }
                        if (T.rank == 0 && jump_log) jump_log[(int64_t)tt * log_stride + (int64_t)(site >> 1) + i] = 0;
                        P = P1;
                        l = left;
                    }
                }
                __syncwarp();
                site += two ? 4 : 2;
                par ^= 1;
                if (far) {
                    __syncthreads();
                    const double sig = sqrt(fix_value(sh.sig2));
                    set_sig(sig);
                }
                continue;
            }
            // a jump, or too near to tell: true amplitudes, the general decisions, the pending factors again
            const int q = st.q, t = st.t;
            const double* pend = tabs + st.pend;
            if (worker) F.scale_all(pend, T.nl);
            __syncthreads();
            double sig = sqrt(fix_value(sh.sig2) * fix_value(st.f));
            sig = site_of(q, sig);
            if (two) sig = site_of(t, sig);
            if (worker) F.scale_all(pend + npos, T.nl);
            __syncthreads();
            set_sig(sig);
        }
        __syncthreads();
        // <Z> of the position of qubit 0
        double acc = 0.0;
        for (uint32_t l = tid; l < T.NL; l += blockDim.x) {
            const double2 a = T.s[l];
            const double w = FastTraj::norm(a);
            acc += ((zpos == T.nl ? (uint32_t)T.rank : l >> zpos) & 1) ? -w : w;
        }
        const double z = T.group_total(acc, part2) * fix_value(sh.sig2);
        if (tid == 0 && T.rank == 0) {
            z0_out[tt] = z;
            if (jumps_out) jumps_out[tt] = jumps;
        }
        group_sync<CL>();
    }
    // the margins of thread 0 (general decisions) and of the extra warp
    __syncthreads();
    if (tid == (int)F.workers) part2[0] = min_margin;
    __syncthreads();
    if (tid == 0 && margin_out) margin_out[blockIdx.x] = fmin(min_margin, part2[0]);
}

__global__ void __launch_bounds__(kFastThreads)
    k_traj_fast1(int n, const TrajGate* gates, const FastStep* steps, int nsteps, const double* tabs, int zpos, KrausParams kp,
                 uint64_t traj_begin, uint64_t n_traj, double* z0, uint32_t* jumps, uint8_t* log, int64_t log_stride,
                 double* margins) {
    traj_fast_body<1>(n, gates, steps, nsteps, tabs, zpos, kp, traj_begin, n_traj, z0, jumps, log, log_stride, margins);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFastThreads)
    k_traj_fast2(int n, const TrajGate* gates, const FastStep* steps, int nsteps, const double* tabs, int zpos, KrausParams kp,
                 uint64_t traj_begin, uint64_t n_traj, double* z0, uint32_t* jumps, uint8_t* log, int64_t log_stride,
                 double* margins) {
    traj_fast_body<2>(n, gates, steps, nsteps, tabs, zpos, kp, traj_begin, n_traj, z0, jumps, log, log_stride, margins);
}
