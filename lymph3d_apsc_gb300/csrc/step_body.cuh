// step_body.cuh -- the per-polyhedron body of the time step, shared by the
// single-problem kernel (step.cu) and the multi-problem persistent kernel
// (batch.cu).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace stepk {

// ---- FP64 products on the integer pipe ----
//
// The GB300 retires 2 FP64 multiply-adds per clock and SM, which holds a product
// with FP64 blocks at two thirds of the copy bandwidth, while its integer pipe idles.
// At p = 3 and 4, and at p = 2 where it pays (lymph_dev_int_columns), 60 % of each row's
// columns (the last ones, c >= C0) are therefore multiplied there: a block entry and a
// coefficient are doubles as before, their mantissas multiply to the product's top 64
// bits (three dropped parts of less than a unit each of at least 2^62: truncated towards
// zero by less than 3 2^-62 of it, where an FP64 product rounds by 2^-53), and the
// product, shifted by the exponents, adds up exactly in a 128-bit accumulator whose top
// stands at the largest product any block of the row could have.  A term loses bits only
// below 2^-117 of that.  The sum is converted to FP64 once per 16 blocks (acc_value: its
// two words and their sum are rounded), so the row's error falls (K u of random, graded
// and near-constant states: by 40 % in the mean).
// 16 steps of 46,767 polyhedra at p = 3: 56.0 -> 38.0 ms (61 -> 90 % of the copy
// bandwidth); 24 steps of a mesh of 17^3 cubes at p = 4: 18.8 -> 13.2 ms.
constexpr bool int_columns(int p, size_t elem) { return p >= 3 && elem == 8; }
constexpr int INT_HEAD = 10;         // bits of headroom: at most 2^9 terms of a thread
constexpr int EXP_NONE = -(1 << 20);
constexpr int EXP_NONFINITE = 1 << 20;

// |x| = m 2^(e - 1086), m with its top bit set (m = 0, e = EXP_NONE for zero).
__device__ __forceinline__ unsigned long long split_mantissa(double x, int* e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    const int ef = (int)(b >> 52);
    if (ef == 0x7ff) { *e = EXP_NONFINITE; return 0; }
    if (ef > 0) { *e = ef; return 1ull << 63 | b << 11; }
    if (b == 0) { *e = EXP_NONE; return 0; }
    const int lz = __clzll((long long)b);
    *e = 12 - lz;
    return b << lz;
}

struct Acc128 {
    unsigned long long lo;
    long long hi;
};
// acc += K u; u: the mantissa's words, the shift before K's exponent, the sign in bit 31.
__device__ __forceinline__ void int_fma(Acc128& acc, double K, const uint4 u) {
    const unsigned kh = (unsigned)__double2hiint(K), kl = (unsigned)__double2loint(K);
    // K's mantissa with its top bit set; a zero or denormal entry's exponent 0
    // shifts it out of the accumulator
    const unsigned mh = __funnelshift_l(kl, kh, 11) | 0x80000000u, ml = kl << 11;
    const unsigned long long p =
        (unsigned long long)mh * u.x + __umulhi(mh, u.y) + (unsigned long long)__umulhi(ml, u.x);
    const unsigned s = u.z - (kh >> 20 & 0x7ff);
    unsigned long long vh, v1, v2;   // (p 2^64) >> s in two words; PTX shifts by 64 and more give 0
    asm("shr.u64 %0, %1, %2;" : "=l"(vh) : "l"(p), "r"(s));
    asm("shl.b64 %0, %1, %2;" : "=l"(v1) : "l"(p), "r"(64u - s));
    asm("shr.u64 %0, %1, %2;" : "=l"(v2) : "l"(p), "r"(s - 64u));
    const unsigned m32 = (unsigned)((int)(kh ^ u.w) >> 31);   // all ones: a negative product
    const unsigned long long m = (unsigned long long)m32 << 32 | m32;
    const unsigned long long a = (v1 | v2) ^ m, b = vh ^ m;
    asm("{\n\t.reg .u32 t;\n\t"
        "add.cc.u32 t, %2, 1;\n\t"     // carry: + 1 for a negated term
        "addc.cc.u64 %0, %0, %3;\n\t"
        "addc.u64 %1, %1, %4;\n\t}"
        : "+l"(acc.lo), "+l"(acc.hi)
        : "r"(m32), "l"(a), "l"(b));
}
// The accumulator's value: acc 2^(R - 2162), R the exponent its top stands at.
__device__ __forceinline__ double acc_value(Acc128 acc, int R) {
    if (R == EXP_NONE) return 0.0;
    if (R >= EXP_NONFINITE / 2) return __longlong_as_double(0x7ff8000000000000ll);
    const bool neg = acc.hi < 0;
    if (neg) {
        acc.lo = ~acc.lo + 1;
        acc.hi = ~acc.hi + (acc.lo == 0);
    }
    const double d = fma((double)acc.lo, 5.42101086242752217e-20 /* 2^-64 */, (double)(unsigned long long)acc.hi);
    const double v = ldexp(d, R - 2098);
    return neg ? -v : v;
}

template <int P> struct Deg {
    static constexpr int NP = (P + 1) * (P + 2) * (P + 3) / 6;
    static constexpr int ND = 3 * NP;
};

// Thread shape per degree: S column slices x ND rows (ND*S fills whole warps
// but for a few lanes), and the CTAs per SM the launch bounds ask for.
template <int P> struct Shape {
    static constexpr int ND = Deg<P>::ND;
    static constexpr int S = P == 1 ? 8 : (P == 2 ? 8 : (P == 3 ? 4 : 3));
    static constexpr int T = ((ND * S + 31) / 32) * 32;       // 96, 256, 256, 320
    static constexpr int MINB = P == 1 ? 16 : (P == 4 ? 3 : 6);
};

// Bytes of a row's blocks prefetched before its state is ready, while a step's
// blocks have at most 512 MB: then the prefetch is worth 1 to 10 % (48 FP32 steps
// of 2,744 polyhedra at p = 3: 2.00 against 2.21 ms), with more it displaces what the
// 129 MB L2 keeps from step to step (4,096 at p = 4: 9.62 against 8.92 ms; of 10,648
// at p = 3: 8.37 against 7.66 ms).
constexpr int STEP_PREFETCH = 32 * 1024;
constexpr int64_t STEP_PREFETCH_MAX = 512ll << 20;

constexpr int NBB = 16;   // neighbour blocks staged in shared memory at once

// Doubles of scratch finish_poly needs behind the right-hand side for polyhedra
// with absorbing faces: a vector of ND, and two partial sums per row where the CTA
// has the threads to form them side by side.
constexpr int MAX_STEP_THREADS = 320;
constexpr int finish_scratch(int nd, int threads) { return nd + (threads >= 2 * nd ? 2 * nd : 0); }

// MODE_APPLY: out = M^-1 K u (power iteration for the CFL bound)
// MODE_BILIN: partial[P] = un_P . (K u0)_P (the bilinear form of the leapfrog energy)
// MODE_KU:    out = K u (the operator apply alone, before M^-1)
enum { MODE_STEP = 0, MODE_FIRST = 1, MODE_APPLY = 3, MODE_BILIN = 4, MODE_KU = 5 };

struct StepArgs {
    const int32_t* row_ptr;
    const int32_t* col;
    const void* K;             // [n_blocks][ND][ND] column-major (double or float)
    const int32_t* Kex;        // with integer columns: largest biased exponent of each block's entries
    const double* Minv;        // [n_poly][NP][NP] column-major inverse of M_loc
    const double* rhs_stat;
    const double* rhs_dyn;
    const double* gvals;       // time-function values (null: the one value g)
    const int64_t* step_idx;   // index into gvals: the device counter (steps of earlier graph launches) ...
    int step_off;              // ... plus this step's place in the graph
    double g;
    float* u32_out;            // FP32 copy of u^{n+1} for the next matrix-free step, [n_poly][NP] x 4 (may be null)
    const double* u0;          // u^{n-1} (MODE_STEP), u^0 (MODE_FIRST)
    const double* un;          // u^n (MODE_STEP, MODE_APPLY), v^0 (MODE_FIRST)
    double* out;               // u^{n+1} (MODE_STEP: may alias u0), u^1 (MODE_FIRST), M^-1 K u (MODE_APPLY),
                               // K u (MODE_KU)
    double* partial;           // MODE_BILIN: per-polyhedron sums
    const int32_t* abs_idx;    // per polyhedron its index among those with absorbing faces, -1 for the
                               // others; null when the mesh has no absorbing face
    const double* Dabs;        // [n_abs][ND][ND] damping blocks (symmetric)
    const double* Winv;        // [n_abs][ND][ND] column-major inverse of M (x) I + dt/2 D
    double dt, dt2;            // and dt^2, formed once: 65 matrix-free steps of 46,767 polyhedra 56.7 -> 56.1 ms
                               // with it and finite64
    int* status;
    int n_poly;
    int prefetch;              // whether a step prefetches its rows' heads
    int early;                 // whether it lets the next step's CTAs be placed before it sums (trigger_early)
};

// Programmatic dependent launch: a step kernel starts while the one before it
// finishes, reads what no step writes, and waits for that kernel and its writes
// before it touches a state.  No-ops on a plain launch.  The next step's CTAs may
// be placed once every CTA of this one has triggered or ended.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// With stored blocks a grid of at most one CTA per SM (8 at p = 1) triggers as soon
// as it may touch the state, a larger one when a CTA has summed its row: CTAs that
// are placed early fill the slots of the SMs that are done first and leave the
// others idle (48 steps of 512 polyhedra in FP64: p = 3 1.70 against 1.26 ms, p = 4
// 6.0 against 4.3 ms with FP64 products alone; of 125 polyhedra at p = 4: 1.17
// against 1.34 ms, of 1,000 at p = 1 374 against 433 us).
inline bool trigger_early(int p, int n_poly, int sms) { return n_poly <= (p == 1 ? 8 : 1) * sms; }

// Launches a step kernel that may start before the stream's previous kernel ends.
template <typename K, typename A>
inline cudaError_t launch_pdl(K kernel, unsigned grid, unsigned block, cudaStream_t st, const A& arg, size_t smem = 0) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, arg);
}

// One bulk prefetch into L2 of the whole 16-byte words inside [p, p + bytes).
__device__ __forceinline__ void prefetch_inside(const void* p, int64_t bytes) {
    const uintptr_t s = ((uintptr_t)p + 15) & ~(uintptr_t)15, e = ((uintptr_t)p + (uintptr_t)bytes) & ~(uintptr_t)15;
    if (e > s) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s), "r"((uint32_t)(e - s)) : "memory");
}

__device__ __forceinline__ double ld_stream(const double* p) { return __ldcs(p); }
__device__ __forceinline__ float ld_stream(const float* p) { return __ldcs(p); }

// Shared-memory layout of one polyhedron's step: the gathered coefficients
// and the row partial sums in the accumulation type, then the FP64 right-hand
// side at an offset rounded up to 16 bytes (with FP32 blocks and odd ND the
// raw offset is not 8-byte aligned).
template <int PD, typename KT, int S_ = Shape<PD>::S, bool INT = int_columns(PD, sizeof(KT))> struct SmemSize {
    static constexpr int ND = Deg<PD>::ND, S = S_;
    static constexpr size_t b_offset = ((sizeof(KT) * (size_t)(NBB * ND + S * ND)) + 15) & ~(size_t)15;
    // the columns of the integer pipe: a thread's last NI of CPT, c >= C0 (12 of 35:
    // 14.1 and 44.0 ms for the runs above, 16 of 35: 13.5 and 41.0, 19 of 35: 13.4 and
    // 38.1, 24 of 35: 13.2 and 38.9)
    static constexpr int CPT = (ND + S - 1) / S, NI = INT ? CPT * 21 / 35 : 0;
    static constexpr int C0 = (CPT - NI) * S < ND ? (CPT - NI) * S : ND, NC = ND - C0;
    static_assert(NI * NBB < 1 << (INT_HEAD - 1), "the accumulator's headroom");
    static constexpr size_t m_offset =
        (b_offset + sizeof(double) * (ND + finish_scratch(ND, MAX_STEP_THREADS)) + 15) & ~(size_t)15;
    static constexpr size_t r_offset = m_offset + sizeof(uint4) * NBB * NC;
    static constexpr size_t bytes = r_offset + (NI ? sizeof(int) : 0);
};

// isfinite on the integer pipe: the FP64 pipe takes 64 cycles for a warp's comparison.
__device__ __forceinline__ bool finite64(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// Component i of the FP32 record (u_0, u_1, u_2, u_2) of basis function q.
__device__ __forceinline__ void store_u32(float* u32, int64_t q, int i, double v) {
    u32[q * 4 + i] = (float)v;
    if (i == 2) u32[q * 4 + 3] = (float)v;
}

// Columns c0, c0 + step, ... of row r of a column-major ND x ND matrix in device
// memory times w in shared memory, one chain in increasing c (the FP32 operators'
// steps carry a change of rounding here back through their inputs: on tetrahedra at
// p = 4 sums in slices ended 4e-5 apart after 74 steps).  Sixteen loads are in flight
// at once (80 matrix-free steps of 1,273 polyhedra at p = 2: 1.24 ms, 1.92 with rolled
// chains and without the overlapping launches, 1.18 with sums in slices).
template <int ND, int UNROLL>
__device__ __forceinline__ double row_chain(const double* __restrict__ A, const double* w, int r, int c0, int step) {
    double a = 0.0;
#pragma unroll UNROLL
    for (int c = c0; c < ND; c += step) a = fma(__ldg(A + c * ND + r), w[c], a);
    return a;
}

// The end of one polyhedron's step once thread tid < ND holds y = (K u)_tid
// of row tid in FP64: the right-hand side, the mass-matrix inverse and the
// leapfrog update (or the bilinear partial sum).  The mass-matrix inverse is
// applied in FP64 as a dense Np x Np product per component (precomputed from
// the Cholesky factor), which replaces the reference's two triangular solves
// per component with a parallel product of the same value.  s_b holds ND
// doubles, 16-byte aligned, then finish_scratch(ND, threads) more.  Every
// thread of the CTA must call this (it synchronises).
// U32: also leave the FP32 copy of u^{n+1} (A.u32_out) for the next
// matrix-free step.
// ABS: with the code of polyhedra with absorbing faces; CHAIN: the loads of a damping
// chain in flight.
template <int PD, int MODE, bool U32 = false, bool ABS = true, int CHAIN = 16>
__device__ __forceinline__ void finish_poly(const StepArgs& A, int P, double y, double* s_b) {
    constexpr int NP = Deg<PD>::NP, ND = Deg<PD>::ND;
    const int tid = threadIdx.x;
    if (MODE == MODE_BILIN) {
        if (tid < ND) s_b[tid] = y;
        __syncthreads();
        if (tid == 0) {
            double e = 0.0;
            for (int rr = 0; rr < ND; ++rr) {
                const int64_t q = (int64_t)P * ND + rr;
                e = e + A.un[q] * s_b[rr];
            }
            A.partial[P] = e;
        }
        return;
    }
    if (MODE == MODE_KU) {
        if (tid < ND) {
            if (!finite64(y)) atomicOr(A.status, ST_NONFINITE);
            A.out[(int64_t)P * ND + tid] = y;
        }
        return;
    }
    if (tid < ND) {
        const int64_t q = (int64_t)P * ND + tid;
        if (MODE == MODE_APPLY) {
            s_b[tid] = y;
        } else {
            const double g = A.gvals ? A.gvals[*A.step_idx + A.step_off] : A.g;
            s_b[tid] = -y + A.rhs_stat[q] + A.rhs_dyn[q] * g;
        }
    }
    __syncthreads();
    // polyhedra with absorbing faces (the index is the same for the whole CTA)
    const int ai = ABS && (MODE == MODE_STEP || MODE == MODE_FIRST) && A.abs_idx ? A.abs_idx[P] : -1;
    if (ai >= 0) {
        const int64_t base = (int64_t)P * ND;
        double *s_w = s_b + ND, *s_p = s_w + ND;
        // MODE_STEP: D (u^n - u^{n-1}); MODE_FIRST: D v^0 (v^0 is in un)
        if (tid < ND) s_w[tid] = (MODE == MODE_STEP) ? A.un[base + tid] - A.u0[base + tid] : A.un[base + tid];
        __syncthreads();
        const double dv = tid < ND ? row_chain<ND, CHAIN>(A.Dabs + (int64_t)ai * ND * ND, s_w, tid, 0, 1) : 0.0;
        if (tid < ND) s_b[tid] = (MODE == MODE_STEP) ? A.dt * A.dt * s_b[tid] - A.dt * dv : s_b[tid] - dv;
        __syncthreads();
        if (MODE == MODE_STEP) {
            // u^{n+1} = 2 u^n - u^{n-1} + W^-1 (dt^2 (F - K u^n) - dt D (u^n - u^{n-1}))
            // the even and the odd columns, side by side where the CTA has the threads
            const double* W = A.Winv + (int64_t)ai * ND * ND;
            double x = 0.0;
            if (blockDim.x >= 2 * ND) {
                if (tid < 2 * ND) s_p[tid] = row_chain<ND, CHAIN>(W, s_b, tid % ND, tid / ND, 2);
                __syncthreads();
                if (tid < ND) x = s_p[tid] + s_p[ND + tid];
            } else if (tid < ND) {
                x = row_chain<ND, CHAIN>(W, s_b, tid, 0, 2) + row_chain<ND, CHAIN>(W, s_b, tid, 1, 2);
            }
            if (tid < ND) {
                const int64_t q = base + tid;
                const double v = x + 2.0 * A.un[q] - A.u0[q];
                if (!finite64(v)) atomicOr(A.status, ST_NONFINITE);
                A.out[q] = v;
                if (U32 && A.u32_out) store_u32(A.u32_out, (int64_t)P * NP + tid % NP, tid / NP, v);
            }
            return;
        }
        // MODE_FIRST continues with M^-1 (F - K u^0 - D v^0) below
    }
    if (tid < ND) {
        const int i = tid / NP, m = tid % NP;
        const double* Mi = A.Minv + (int64_t)P * NP * NP + m;
        const double* bi = s_b + i * NP;
        double x0 = 0.0, x1 = 0.0;
#pragma unroll
        for (int c = 0; c < NP; c += 2) {
            x0 += Mi[c * NP] * bi[c];
            if (c + 1 < NP) x1 += Mi[(c + 1) * NP] * bi[c + 1];
        }
        const double x = x0 + x1;
        const int64_t q = (int64_t)P * ND + tid;
        double v;
        if (MODE == MODE_STEP) {
            const double dt2 = A.dt2;
            v = dt2 * x + 2.0 * A.un[q] - A.u0[q];
        } else if (MODE == MODE_FIRST) {
            const double half_dt2 = 0.5 * (A.dt * A.dt);
            v = half_dt2 * x + A.u0[q] + A.dt * A.un[q];
        } else {
            v = x;
        }
        if (!finite64(v)) atomicOr(A.status, ST_NONFINITE);
        A.out[q] = v;
        if (U32 && MODE == MODE_STEP && A.u32_out) store_u32(A.u32_out, (int64_t)P * NP + m, i, v);
    }
}

// ---- meshes of at most one polyhedron per SM ----
//
// A step is then a chain of latencies, and the next step's CTA already sits beside
// this one's while it runs: it copies the head of its block row, M^-1, the column
// indices and the blocks' exponents into its shared memory before it waits for the
// state, and reads right-hand side and own coefficients with the gather instead of
// one after another at the end.  Two CTAs share an SM's 227 KB.
// 48 steps of 125 hexahedra: p = 1 in FP64 267 -> 240 us, p = 2 346 -> 335 (FP64-pipe
// bound), p = 3 627 -> 591, in FP32 263 -> 239, 285 -> 265, 371 -> 337; 100 FP64 steps
// of 90 polyhedra (10 blocks a row): 605 -> 503, 852 -> 803, 1,856 -> 1,615 us.
constexpr int SMALL_STAGE = 88 * 1024;   // bytes of staged blocks per CTA
template <int PD, typename KT> struct SmallSmem {
    static constexpr int ND = Deg<PD>::ND, NP = Deg<PD>::NP;
    static constexpr int FIT = SMALL_STAGE / (ND * ND * (int)sizeof(KT)), STAGE = FIT < NBB ? FIT : NBB;
    static constexpr size_t minv_offset = (size_t)STAGE * ND * ND * sizeof(KT);   // 16-byte multiples for p <= 3
    static constexpr size_t col_offset = minv_offset + sizeof(double) * NP * NP;
    static constexpr size_t bytes = col_offset + 2 * sizeof(int) * NBB;
};
__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// What finish_poly reads of polyhedron P's own, row tid.
struct Own { double rs, rd, g, un, u0; };

// finish_poly for MODE_STEP without absorbing faces, its inputs already read.
template <int PD>
__device__ __forceinline__ void finish_small(const StepArgs& A, int P, double y, double* s_b, const Own& o, const double* s_Mi) {
    constexpr int NP = Deg<PD>::NP, ND = Deg<PD>::ND;
    const int tid = threadIdx.x;
    if (tid < ND) s_b[tid] = -y + o.rs + o.rd * o.g;
    __syncthreads();
    if (tid < ND) {
        const int i = tid / NP, m = tid % NP;
        const double* Mi = s_Mi + m;
        const double* bi = s_b + i * NP;
        double x0 = 0.0, x1 = 0.0;
#pragma unroll
        for (int c = 0; c < NP; c += 2) {
            x0 += Mi[c * NP] * bi[c];
            if (c + 1 < NP) x1 += Mi[(c + 1) * NP] * bi[c + 1];
        }
        const double x = x0 + x1, dt2 = A.dt2;
        const double v = dt2 * x + 2.0 * o.un - o.u0;
        if (!finite64(v)) atomicOr(A.status, ST_NONFINITE);
        A.out[(int64_t)P * ND + tid] = v;
    }
}

// The block row of polyhedron P is one contiguous column-major
// [ND x nb*ND] matrix (its blocks are adjacent in memory), multiplied by the
// gathered coefficients of the column polyhedra, then finish_poly.  S_ is
// the number of column slices (the tile shape; the CTA needs ND * S_ threads).
// Every thread of the CTA must call this (it synchronises); threads beyond the
// degree's shape only help with the gather.
// SMALL: dyn is the shared memory of SmallSmem.  BLOCKS: blocks loaded at once, 0: the compiler's choice.
template <int PD, typename KT, int MODE, int S_ = Shape<PD>::S, bool INT = int_columns(PD, sizeof(KT)), bool SMALL = false,
          bool ABS = true, int CHAIN = 16, int BLOCKS = 0>
__device__ __forceinline__ void step_poly(const StepArgs& A, int P, char* smem, char* dyn = nullptr) {
    constexpr int ND = Deg<PD>::ND, S = S_;
    constexpr int CPT = (ND + S - 1) / S;
    using AT = KT;  // FP64 blocks accumulate in FP64, FP32 blocks in FP32
    AT* s_u = (AT*)smem;
    AT* s_red = s_u + NBB * ND;
    using SZ = SmemSize<PD, KT, S, INT>;
    double* s_b = (double*)(smem + SZ::b_offset);
    static_assert(SZ::b_offset % 16 == 0, "FP64 rhs must be 16-byte aligned");
    const int nthr = blockDim.x;
    const int tid = threadIdx.x;
    const int r = tid % ND, s = tid / ND;
    const bool act = tid < ND * S;
    const int rb = A.row_ptr[P], re = A.row_ptr[P + 1];
    const KT* Kbase = (const KT*)A.K;
    using SS = SmallSmem<PD, KT>;
    int* s_col = (int*)(dyn + SS::col_offset);
    Own own = {0.0, 0.0, 0.0, 0.0, 0.0};
    const int nst = SMALL ? (re - rb < SS::STAGE ? re - rb : SS::STAGE) : 0;
    if constexpr (SMALL) {
        const int n16 = nst * (int)(ND * ND * sizeof(KT) / 16), m16 = Deg<PD>::NP * Deg<PD>::NP / 2;
        const char* src = (const char*)(Kbase + (int64_t)rb * ND * ND);
        for (int i = tid; i < n16; i += nthr) cp16(dyn + 16 * i, src + 16 * i);
        const char* mi = (const char*)(A.Minv + (int64_t)P * Deg<PD>::NP * Deg<PD>::NP);
        for (int i = tid; i < m16; i += nthr) cp16(dyn + SS::minv_offset + 16 * i, mi + 16 * i);
        if (tid < NBB && tid < re - rb) {
            s_col[tid] = A.col[rb + tid];
            if (INT) s_col[NBB + tid] = A.Kex[rb + tid];
        }
        pdl_wait();
        pdl_trigger();
        if (tid < ND) {
            const int64_t q = (int64_t)P * ND + tid;
            own.g = A.gvals ? A.gvals[*A.step_idx + A.step_off] : A.g;
            own.rs = A.rhs_stat[q];
            own.rd = A.rhs_dyn[q];
            own.un = A.un[q];
            own.u0 = A.u0[q];
        }
    } else if (MODE == MODE_STEP) {
        if (A.prefetch && tid == 0) {   // the head of the row's blocks and M^-1, while the previous step ends
            const int64_t row = (int64_t)(re - rb) * ND * ND * (int64_t)sizeof(KT);
            prefetch_inside(Kbase + (int64_t)rb * ND * ND, row < STEP_PREFETCH ? row : STEP_PREFETCH);
            prefetch_inside(A.Minv + (int64_t)P * Deg<PD>::NP * Deg<PD>::NP, (int64_t)Deg<PD>::NP * Deg<PD>::NP * 8);
        }
        pdl_wait();
        if (A.early) pdl_trigger();
    }

    constexpr int NI = SZ::NI, C0 = SZ::C0, NC = SZ::NC, JF = CPT - NI;
    uint4* s_m = (uint4*)(smem + SZ::m_offset);   // the integer columns' coefficients
    int* s_R = (int*)(smem + SZ::r_offset);       // the accumulators' exponent

    AT acc0 = 0, acc1 = 0;
    for (int b0 = rb; b0 < re; b0 += NBB) {
        const int nb = (re - b0) < NBB ? (re - b0) : NBB;
        if (NI && tid == 0) *s_R = EXP_NONE;
        __syncthreads();
        const bool staged = SMALL && b0 == rb;
        for (int i = tid; i < nb * ND; i += nthr) {
            const int bb = i / ND, c = i % ND;
            const int64_t q = (int64_t)(staged ? s_col[bb] : A.col[b0 + bb]) * ND + c;
            s_u[i] = (AT)((MODE == MODE_FIRST || MODE == MODE_BILIN) ? A.u0[q] : A.un[q]);
        }
        Acc128 iacc = {0, 0};
        int R = EXP_NONE;
        if constexpr (NI > 0) {
            __syncthreads();
            // mantissas and exponents of the integer columns, then the largest
            // exponent a product of the row can have
            int mx = EXP_NONE;
            for (int i = tid; i < nb * NC; i += nthr) {
                const int bb = i / NC, kx = staged ? s_col[NBB + bb] : A.Kex[b0 + bb];
                const double u = s_u[bb * ND + C0 + i - bb * NC];
                int e;
                const unsigned long long m = split_mantissa(u, &e);
                s_m[i] = make_uint4((unsigned)(m >> 32), (unsigned)m, (unsigned)e, u < 0.0 ? 0x80000000u : 0u);
                if (e > EXP_NONE) mx = max(mx, e + kx);
                else if (kx == EXP_NONFINITE) mx = kx;
            }
            mx = __reduce_max_sync(0xffffffffu, mx);
            if ((tid & 31) == 0 && mx > EXP_NONE) atomicMax(s_R, mx);
            __syncthreads();
            R = *s_R;
            for (int i = tid; i < nb * NC; i += nthr) {   // each thread's own entries
                const int e = (int)s_m[i].z;
                s_m[i].z = e > EXP_NONE && R < EXP_NONFINITE / 2 ? (unsigned)(INT_HEAD + R - e) : 1u << 16;
            }
        }
        if (SMALL && b0 == rb) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (act) {
            const auto products = [&](int bb, const KT(&kv)[CPT]) {
                const AT* ub = s_u + bb * ND;
#pragma unroll
                for (int j = 0; j < CPT; ++j) {
                    const int c = s + j * S;
                    if (c < ND) {
                        if constexpr (NI > 0) {
                            if (j >= JF) {
                                int_fma(iacc, kv[j], s_m[bb * NC + c - C0]);
                                continue;
                            }
                        }
                        if (j & 1) acc1 += (AT)kv[j] * ub[c];
                        else acc0 += (AT)kv[j] * ub[c];
                    }
                }
            };
            int bb = 0;
            if constexpr (SMALL) {
                if (b0 == rb) {
#pragma unroll 2
                    for (; bb < nst; ++bb) {
                        const KT* Kb = (const KT*)dyn + bb * ND * ND + r;
                        KT kv[CPT];
#pragma unroll
                        for (int j = 0; j < CPT; ++j) kv[j] = s + j * S < ND ? Kb[(s + j * S) * ND] : (KT)0;
                        products(bb, kv);
                    }
                }
            }
            const auto block = [&](int k) {
                const KT* Kb = Kbase + (int64_t)(b0 + k) * ND * ND + r;
                KT kv[CPT];
#pragma unroll
                for (int j = 0; j < CPT; ++j) {
                    const int c = s + j * S;
                    kv[j] = (c < ND) ? ld_stream(Kb + (int64_t)c * ND) : (KT)0;
                }
                products(k, kv);
            };
            if constexpr (BLOCKS > 0) {
#pragma unroll BLOCKS
                for (; bb < nb; ++bb) block(bb);
            } else {
                for (; bb < nb; ++bb) block(bb);
            }
            if constexpr (NI > 0) acc1 += acc_value(iacc, R);
        }
    }
    if (MODE == MODE_STEP && !SMALL) pdl_trigger();
    if (act) s_red[s * ND + r] = acc0 + acc1;
    __syncthreads();
    double y = 0.0;
    if (tid < ND)
        for (int ss = 0; ss < S; ++ss) y += (double)s_red[ss * ND + tid];
    if constexpr (SMALL) finish_small<PD>(A, P, y, s_b, own, (const double*)(dyn + SS::minv_offset));
    else finish_poly<PD, MODE, false, ABS, CHAIN>(A, P, y, s_b);
}

}  // namespace stepk
