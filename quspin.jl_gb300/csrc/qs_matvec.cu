// qs_matvec.cu -- the fused matrix-free Hamiltonian action y = alpha*op(A)x + beta*y.
//
// Replaces the reference's serial scatter (_apply_spin_term!, src/operators.jl:
// 2554-2589) and its symmetric lift -> parent apply -> project path
// (_apply_spin_terms!, 2591-2636) with a row-wise pull form in representative
// space.  One thread owns one output row r (its representative s_r):
//
//   y[r] = beta*y[r] + alpha*( d[r] x[r] +
//          sum_progs  A[s_r, t] * chi(h_t) * sqrt(stab(m_t) / stab(s_r)) * x[rank(m_t)] )
//
// where t runs over the states reached from s_r by the transposed term chain
// (A[s,t] = <t|A^T|s>), m_t = h_t(t) is the orbit minimum of t, chi the sector
// character and stab the stabiliser order.  This equals (P'AP)[r, :] x for the
// reference's projector P (columns P_chi|s_min>/norm) when A commutes with the
// group.  No scatter, no atomics: every row is written once, and the summation
// order per row is fixed, so repeated calls are bit-identical.
//
// The transitions of a row (which programs are alive, orbit minimum, rank) are
// walked by qs_rows.cuh, shared with the assembly.  Bound: integer issue in the
// orbit search; FP64 is one multiply-add per transition (amplitude times
// character from a table, the rare sqrt(stab) != 1 and the row's 1/sqrt(stab)
// apart), which GB300's FP64 pipe takes 16 cycles a warp for.  The eigensolvers,
// which run on this product below 4,096 rows, have every term rounded on its own
// (MatvecCall::solver): the last bits of their projected matrix decide an
// eigenvector's sign.
//
// Rank lookups: full 2^L space -> the state itself; fixed-weight sector
// without spatial symmetry -> combinadic rank (src/discrete_basis.jl:1879-1906);
// symmetric sector -> search of the sorted representatives with a
// shared-memory splitter stage.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

#include <algorithm>
#include <atomic>
#include <map>
#include <vector>

#include "qs_device.cuh"
#include "qs_df.cuh"
#include "qs_internal.h"
#include "qs_rows.cuh"

namespace qs {

namespace {

constexpr int kMvThreads = kRowThreads;
constexpr int kMaxSplit = 2048;

template <typename T> struct V2;
template <> struct V2<double> { using t = double2; };
template <> struct V2<float> { using t = float2; };

struct MvArgs {
    const void* reps;
    const uint16_t* stab;
    const void* split;
    int64_t n, nsplit, stride;
    const GroupDesc* group;
    const uint64_t* binom;
    int L, nup, pauli;
    const TermProg* progs;
    int nprog;
    RowArgs row;             // the transitions (matvec_kernel, matvec_warp_rank_kernel)
    const double* chi_re;    // character of element code e at [e * chi_stride]
    const double* chi_im;
    int chi_stride, nelem;   // nelem 1: every character is 1
    const double2* amp;      // amplitude per program class
    int nclass;
    int table;               // amplitude x character staged per (class, element)
    int any_chars;
    const double* sq;        // sqrt(i), then 1/sqrt(i), i = 0 .. kMaxGroup
    int solver;              // MatvecCall::solver (the general kernels alone)
    int full_diag;           // real operator, complex vectors: the complex diagonal as it stands
    const void* diag;        // complex, precision of the call
    const void* diag_re;     // its real part (real operators)
    int conj_amp, conj_chi;
    double ar, ai, br, bi;
    int beta_zero;
    const void* x;
    void* y;
};

// Applies one transition program to s (operator characters as in
// src/operators.jl:343-379).  Returns false when an operator annihilates the
// state.  Distinct-site programs use their compiled masks; programs that touch
// a site twice run the character interpreter.
template <typename U, typename T>
__device__ __forceinline__ bool run_prog(const TermProg& p, int pauli, U s, U& t, T& ar, T& ai) {
    if (p.distinct) {
        if ((s & (U)p.need1) != (U)p.need1 || (s & (U)p.need0) != (U)0) return false;
        t = s ^ (U)p.flip;
        int par = __popcll((unsigned long long)(~s & (U)p.zmask)) + __popcll((unsigned long long)(s & (U)p.ymask));
        T re = (T)p.amp0_re, im = (T)p.amp0_im;
        if (par & 1) {
            re = -re;
            im = -im;
        }
        ar = re;
        ai = im;
        return true;
    }
    double re = p.coef_re, im = p.coef_im;
    const double zs = pauli ? 1.0 : 0.5;
    const double pm = pauli ? 2.0 : 1.0;
    t = s;
    for (int i = 0; i < p.nops; ++i) {
        const U bit = (U)1 << p.sites[i];
        const bool occ = (t & bit) != 0;
        switch (p.ops[i]) {
            case 'I':
                break;
            case 'z':
                re *= occ ? zs : -zs;
                im *= occ ? zs : -zs;
                break;
            case '+':
                if (occ) return false;
                t |= bit;
                re *= pm;
                im *= pm;
                break;
            case '-':
                if (!occ) return false;
                t &= ~bit;
                re *= pm;
                im *= pm;
                break;
            case 'x':
                t ^= bit;
                re *= zs;
                im *= zs;
                break;
            case 'y': {
                // occupied -> -i*scale, empty -> +i*scale
                t ^= bit;
                double f = occ ? -zs : zs;
                double nre = -im * f, nim = re * f;
                re = nre;
                im = nim;
                break;
            }
            default:
                return false;
        }
    }
    ar = (T)re;
    ai = (T)im;
    return true;
}

template <typename U>
__device__ __forceinline__ U row_state(const MvArgs& a, int mode, int64_t r) {
    if (mode == 2) return ((const U*)a.reps)[r];
    if (mode == 0) return (U)r;
    // unrank a fixed-weight state (inverse of the combinadic rank)
    U s = 0;
    int b = a.L - 1;
    int64_t rem = r;
    for (int p = a.nup; p >= 1; --p) {
        while ((int64_t)__ldg(a.binom + b * 65 + p) > rem) --b;
        s |= (U)1 << b;
        rem -= (int64_t)__ldg(a.binom + b * 65 + p);
        --b;
    }
    return s;
}

// The fixed-weight state of combinadic rank r (inverse of combinadic_rank),
// with the C(bit, p) table in shared memory.
__device__ __forceinline__ uint32_t unrank32(int64_t r, const uint32_t* binom32, int L, int nup) {
    uint32_t s = 0, rem = (uint32_t)r;
    int b = L - 1;
    for (int p = nup; p >= 1; --p) {
        while (binom32[b * 33 + p] > rem) --b;
        s |= 1u << b;
        rem -= binom32[b * 33 + p];
        --b;
    }
    return s;
}

template <typename T, bool kCV>
__device__ __forceinline__ void load_x(const MvArgs& a, int64_t i, T& xr, T& xi) {
    if (kCV) {
        typename V2<T>::t v = ((const typename V2<T>::t*)a.x)[i];
        xr = v.x;
        xi = v.y;
    } else {
        xr = ((const T*)a.x)[i];
        xi = 0;
    }
}

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_r(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// (wr, wi) times the character of element code ec
template <bool kCM, typename T>
__device__ __forceinline__ void times_chi(const MvArgs& a, int ec, T& wr, T& wi) {
    if (a.nelem == 1) return;
    const T cr = (T)__ldg(a.chi_re + (size_t)ec * a.chi_stride);
    if (kCM) {
        T ci = (T)__ldg(a.chi_im + (size_t)ec * a.chi_stride);
        if (a.conj_chi) ci = -ci;
        const T nr = wr * cr - wi * ci, ni = wr * ci + wi * cr;
        wr = nr;
        wi = ni;
    } else {
        wr = mul_rn(wr, cr);
    }
}

// amplitude of a program class, conjugated with the operator
template <typename T>
__device__ __forceinline__ void class_amp(const MvArgs& a, uint32_t cls, T& wr, T& wi) {
    const double2 v = __ldg(a.amp + cls);
    wr = (T)v.x;
    wi = a.conj_amp ? -(T)v.y : (T)v.y;
}

// amplitude x character of every (class, element) pair, when they are few
template <bool kCM, typename T>
__device__ __forceinline__ void stage_values(const MvArgs& a, void* tab) {
    if (!a.table) return;
    for (int i = threadIdx.x; i < a.nclass * a.nelem; i += blockDim.x) {
        T wr, wi;
        class_amp<T>(a, i / a.nelem, wr, wi);
        times_chi<kCM, T>(a, i % a.nelem, wr, wi);
        if (kCM) {
            typename V2<T>::t v;
            v.x = wr;
            v.y = wi;
            ((typename V2<T>::t*)tab)[i] = v;
        } else {
            ((T*)tab)[i] = wr;
        }
    }
}

// Program k on s by its characters (a site acted on twice): false when it
// annihilates the state.
template <typename U>
__device__ __noinline__ bool run_chars(const MvArgs& a, int k, U s, U& t, double& wr, double& wi) {
    if (!run_prog<U, double>(a.progs[k], a.pauli, s, t, wr, wi)) return false;
    if (a.conj_amp) wi = -wi;
    return true;
}

// 1/sqrt(st) in the arithmetic of the call
template <typename T> __device__ __forceinline__ T inv_root(const MvArgs& a, int st);
template <> __device__ __forceinline__ double inv_root<double>(const MvArgs& a, int st) {
    return __ldg(a.sq + kMaxGroup + 1 + st);
}
template <> __device__ __forceinline__ float inv_root<float>(const MvArgs& a, int st) {
    return 1.f / (float)__ldg(a.sq + st);
}

// acc += w x with the character, sqrt(stab) of the column and the sign of a
// transition of class cls (a program run by its characters brings its own w).
// Solver calls: sqrt(stab) of the column times 1/sqrt(stab) of the row (st_r) as
// one factor of w, and w x of a complex operator rounded before it is added
// (six FP64 instructions against four).
template <bool kSym, bool kCM, bool kCV, typename T, bool kPlain>
__device__ __forceinline__ void add_transition(const MvArgs& a, const void* tab, uint32_t cls, int ec, int st, int st_r,
                                               int sign, T wr, T wi, int64_t idx, T& acc_r, T& acc_i) {
    if (!kPlain && cls == kCharsClass) {
        times_chi<kCM, T>(a, ec, wr, wi);
    } else if (kPlain || a.table) {
        const int i = (int)cls * a.nelem + (a.nelem == 1 ? 0 : ec);
        if (kCM) {
            const typename V2<T>::t v = ((const typename V2<T>::t*)tab)[i];
            wr = v.x;
            wi = v.y;
        } else {
            wr = ((const T*)tab)[i];
        }
    } else {
        class_amp<T>(a, cls, wr, wi);
        times_chi<kCM, T>(a, ec, wr, wi);
    }
    if (!kPlain && sign) {
        wr = -wr;
        wi = -wi;
    }
    if (st != 1 || (!kPlain && st_r != 1)) {
        T f = (T)__ldg(a.sq + st);
        if (!kPlain && st_r != 1) f = mul_rn(f, inv_root<T>(a, st_r));
        wr = mul_rn(wr, f);
        if (kCM) wi = mul_rn(wi, f);
    }
    T xr, xi;
    load_x<T, kCV>(a, idx, xr, xi);
    if (kCM && !kPlain && a.solver) {
        acc_r = add_rn(acc_r, fma_r(wr, xr, -mul_rn(wi, xi)));
        acc_i = add_rn(acc_i, kSym ? fma_r(wr, xi, mul_rn(wi, xr)) : fma_r(wi, xr, mul_rn(wr, xi)));
        return;
    }
    acc_r = fma_r(wr, xr, acc_r);
    if (kCM) {
        acc_r = fma_r(-wi, xi, acc_r);
        acc_i = fma_r(wr, xi, acc_i);
        acc_i = fma_r(wi, xr, acc_i);
    } else if (kCV) {
        acc_i = fma_r(wr, xi, acc_i);
    }
}

// y[r] = beta y[r] + alpha (d[r] x[r] + acc / sqrt(stab_r)); solver calls have
// the root in their terms
template <bool kSym, bool kCM, bool kCV, typename T, bool kPlain>
__device__ __forceinline__ void store_row(const MvArgs& a, int64_t r, T acc_r, T acc_i) {
    if (kSym && (kPlain || !a.solver)) {
        const int st = a.stab[r];
        if (st != 1) {
            const T f = (T)__ldg(a.sq + kMaxGroup + 1 + st);
            acc_r *= f;
            acc_i *= f;
        }
    }
    // diagonal (user + extracted), conjugated with the operator
    T xr, xi;
    load_x<T, kCV>(a, r, xr, xi);
    if (kCM || (kCV && a.full_diag)) {
        const typename V2<T>::t d = ((const typename V2<T>::t*)a.diag)[r];
        const T dr = d.x, di = a.conj_amp ? -d.y : d.y;
        acc_r += dr * xr - di * xi;
        acc_i += dr * xi + di * xr;
    } else {
        const T dr = ((const T*)a.diag_re)[r];
        acc_r += dr * xr;
        if (kCV) acc_i += dr * xi;
    }
    if (kCV) {
        typename V2<T>::t* y = (typename V2<T>::t*)a.y;
        T yr = 0, yi = 0;
        if (!a.beta_zero) {
            const typename V2<T>::t yo = y[r];
            yr = (T)a.br * yo.x - (T)a.bi * yo.y;
            yi = (T)a.br * yo.y + (T)a.bi * yo.x;
        }
        typename V2<T>::t out;
        out.x = yr + (T)a.ar * acc_r - (T)a.ai * acc_i;
        out.y = yi + (T)a.ar * acc_i + (T)a.ai * acc_r;
        y[r] = out;
    } else {
        T* y = (T*)a.y;
        const T yr = a.beta_zero ? (T)0 : (T)a.br * y[r];
        y[r] = yr + (T)a.ar * acc_r;
    }
}

// dynamic shared memory: the staged values, then the split rank tables
QS_HD size_t mv_table_bytes(int entries, bool cm, size_t real) {
    return ((size_t)entries * real * (cm ? 2 : 1) + 15) / 16 * 16;
}

// kPlain: every program by its masks with a state-independent sign, the values
// staged and the particle number kept: what exchange couplings and transverse
// fields need, without the flags' tests on every transition.
template <typename U, int kMode, bool kCM, bool kCV, typename T, bool kPlain>
__global__ void __launch_bounds__(kMvThreads) matvec_kernel(MvArgs a) {
    constexpr bool kSym = kMode >= 2;
    constexpr bool k32 = sizeof(U) == 4;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ RowSmem<U> sm;
    __shared__ GroupSmem g;
    __shared__ U spl[kMode == 2 ? kMaxSplit : 1];
    __shared__ uint32_t binom32[kMode == 1 && k32 ? 32 * 33 : 1];
    const RowArgs& R = a.row;
    uint32_t* rtab = (uint32_t*)(dyn + (a.table ? mv_table_bytes(a.nclass * a.nelem, kCM, sizeof(T)) : 0));
    if (kSym && !R.fast.enabled) load_group_smem(g, R.group);
    if (kMode == 2)
        for (int i = threadIdx.x; i < R.nsplit; i += blockDim.x) spl[i] = ((const U*)R.split)[i];
    if (k32 && (kMode == 1 || kMode == 3))
        for (int i = threadIdx.x; i < R.rank.size; i += blockDim.x) rtab[i] = R.rank_tab[i];
    // C(bit, p) for bit < 32, p <= 32: all below 2^32
    if (kMode == 1 && k32)
        for (int i = threadIdx.x; i < 32 * 33; i += blockDim.x)
            binom32[i] = (uint32_t)a.binom[(i / 33) * 65 + (i % 33)];
    stage_values<kCM, T>(a, dyn);
    load_row_progs(sm, R, 0);
    __syncthreads();

    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < a.n; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = base + threadIdx.x;
        const bool valid = r < a.n;
        U s = 0;
        if (valid) s = (k32 && kMode == 1) ? (U)unrank32(r, binom32, a.L, a.nup) : row_state<U>(a, kSym ? 2 : kMode, r);
        const int st_r = kSym && !kPlain && a.solver && valid ? a.stab[r] : 1;
        T acc_r = 0, acc_i = 0;
        for (int c0 = 0; c0 < R.nprog; c0 += kRowChunk) {
            if (R.nprog > kRowChunk) {
                __syncthreads();
                load_row_progs(sm, R, c0);
                __syncthreads();
            }
            row_hops<U, !kPlain>(sm, R, min(kRowChunk, R.nprog - c0), valid, s, [&](int i, U t, int sign) {
                const uint32_t cls = sm.cls[i];
                T wr = 0, wi = 0;
                if (!kPlain && a.any_chars && cls == kCharsClass) {
                    U tc;
                    double dr, di;
                    if (!run_chars<U>(a, c0 + i, s, tc, dr, di)) return;
                    t = tc;
                    wr = (T)dr;
                    wi = (T)di;
                }
                if (!kPlain && kMode != 0 && R.check_weight && __popcll((unsigned long long)t) != a.nup) return;
                U m = t;
                int ec = 0, st = 1;
                if (kSym) row_orbit<U>(R, g, t, m, ec, st);
                const int64_t idx = row_column<U, kMode>(R, spl, rtab, m);
                if (kSym && idx < 0) return;
                add_transition<kSym, kCM, kCV, T, kPlain>(a, dyn, cls, ec, st, st_r, sign, wr, wi, idx,
                                                       acc_r, acc_i);
            });
        }
        if (valid) store_row<kSym, kCM, kCV, T, kPlain>(a, r, acc_r, acc_i);
    }
}


// ----------------------------------------------------- warp-cooperative rank
// First index in [a, b) whose value is >= q (b when none), with all 32 lanes
// of the warp probing together: each round reads 32 evenly spaced entries and
// a ballot keeps the one stride that holds the bound, so a range shrinks
// 32-fold per round.  q and the range are the same in every lane.
template <typename U, class Get>
__device__ __forceinline__ int64_t warp_lower_bound(int64_t a, int64_t b, U q, Get get) {
    const int lane = threadIdx.x & 31;
    while (b - a > 32) {
        const int64_t step = (b - a + 31) / 32;
        const int64_t idx = a + (int64_t)lane * step;
        const unsigned below = __ballot_sync(0xffffffffu, idx < b && get(idx) < q);
        const int c = __popc(below);   // probes are ascending, so the ones below q are a prefix
        if (c == 0) return a;
        const int64_t nb = a + (int64_t)c * step;
        a = a + (int64_t)(c - 1) * step + 1;
        b = nb < b ? nb : b;
    }
    const int64_t idx = a + lane;
    return a + __popc(__ballot_sync(0xffffffffu, idx < b && get(idx) < q));
}

// Column of the representative `key` of every lane that wants one (-1: not a
// representative), resolved for one lane after another by the whole warp: two
// rounds over the shared-memory splitters (splitter i = reps[i * stride]),
// then rounds over the splitter's segment of the sorted representatives in
// global memory.  Every lane of the warp must call it.
template <typename U>
__device__ __forceinline__ int64_t rank_warp(const U* __restrict__ reps, int64_t n, const U* spl, int nsplit,
                                             int64_t stride, U key, bool want) {
    const int lane = threadIdx.x & 31;
    int64_t out = -1;
    unsigned pend = __ballot_sync(0xffffffffu, want);
    while (pend) {
        const int j = __ffs(pend) - 1;
        pend &= pend - 1;
        const U q = __shfl_sync(0xffffffffu, key, j);
        const int64_t ls = warp_lower_bound<U>(0, nsplit, q, [&](int64_t i) { return spl[i]; });
        int64_t idx = -1;
        if (ls < nsplit && spl[ls] == q) {
            idx = ls * stride;
        } else if (ls > 0) {
            const int64_t sa = (ls - 1) * stride, sb = sa + stride < n ? sa + stride : n;
            const int64_t lb = warp_lower_bound<U>(sa, sb, q, [&](int64_t i) { return __ldg(reps + i); });
            if (lb < sb && __ldg(reps + lb) == q) idx = lb;
        }
        if (lane == j) out = idx;
    }
    return out;
}

// The symmetric-sector product of matvec_kernel with the rank of every
// generated state found by rank_warp (QS_RANK_MODE=warp): rows are taken a
// warp at a time and programs in step, so that all 32 lanes reach every lookup
// together.
template <typename U, bool kCM, bool kCV, typename T>
__global__ void __launch_bounds__(kMvThreads) matvec_warp_rank_kernel(MvArgs a) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ GroupSmem g;
    __shared__ U spl[kMaxSplit];
    const RowArgs& R = a.row;
    load_group_smem(g, R.group);
    for (int i = threadIdx.x; i < R.nsplit; i += blockDim.x) spl[i] = ((const U*)R.split)[i];
    stage_values<kCM, T>(a, dyn);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base < a.n; base += nthreads) {
        const int64_t r = base + lane;
        const bool rv = r < a.n;
        const U s = rv ? ((const U*)a.reps)[r] : (U)0;
        const int st_r = a.solver && rv ? a.stab[r] : 1;
        T acc_r = 0, acc_i = 0;
        for (int k = 0; k < R.nprog; ++k) {
            const RowProg p = R.progs[k];
            U t = s ^ (U)p.flip, m = 0;
            T wr = 0, wi = 0;
            int ec = 0, st = 1;
            bool alive = rv && (s & (U)p.care) == (U)p.value;
            if (alive && p.cls == kCharsClass) {
                U tc;
                double dr, di;
                alive = run_chars<U>(a, k, s, tc, dr, di);
                t = tc;
                wr = (T)dr;
                wi = (T)di;
            }
            if (R.check_weight && __popcll((unsigned long long)t) != a.nup) alive = false;
            if (alive) row_orbit<U>(R, g, t, m, ec, st);
            const int64_t idx = rank_warp<U>((const U*)R.reps, a.n, spl, (int)R.nsplit, R.stride, m, alive);
            if (!alive || idx < 0) continue;
            const int sign = __popcll((unsigned long long)(s & (U)p.zy)) & 1;
            add_transition<true, kCM, kCV, T, false>(a, dyn, p.cls, ec, st, st_r, sign, wr, wi, idx, acc_r, acc_i);
        }
        if (rv) store_row<true, kCM, kCV, T, false>(a, r, acc_r, acc_i);
    }
}

// General path for operators that do not commute with the group (reference:
// check_symm=false on a symmetric basis, src/operators.jl:2500-2506): the full
// P' A P with both projector sides expanded over the group,
//   y[r] = (1/stab_r) sum_e chi'(g_e)/sqrt|orb r| sum_t A[g_e s_r, t] chi'(h_t)/sqrt|orb m_t| x[m_t]
template <typename U, bool kCV>
__global__ void __launch_bounds__(kMvThreads) matvec_general_kernel(MvArgs a) {
    __shared__ GroupSmem g;
    __shared__ U spl[kMaxSplit];
    load_group_smem(g, a.group);
    for (int i = threadIdx.x; i < a.nsplit; i += blockDim.x) spl[i] = ((const U*)a.split)[i];
    __syncthreads();
    const GroupDesc* G = a.group;
    const int L = g.L;
    const U lm = (U)g.lmask;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < a.n; r += (int64_t)gridDim.x * blockDim.x) {
        const U s = ((const U*)a.reps)[r];
        const int stab_r = a.stab[r];
        const double orb_r = (double)g.ng / (double)stab_r;
        double acc_r = 0, acc_i = 0;
        U base[2] = {s, brev_bits(s, L)};
        for (int p = 0; p < g.nperm; ++p) {
            U rot = g.general ? (U)gperm_apply(g.gtab, p, g.nbytes, (uint64_t)s)
                              : rotl_bits<U>(base[g.refl[p]], g.shift[p], L, lm);
            for (int e = g.begin[p]; e < g.begin[p + 1]; ++e) {
                const U tp = rot ^ (U)g.mask[e];
                double er = G->chi_re[e], ei = a.conj_chi ? -G->chi_im[e] : G->chi_im[e];
                for (int k = 0; k < a.nprog; ++k) {
                    U t;
                    double are, aim;
                    if (!run_prog<U, double>(a.progs[k], a.pauli, tp, t, are, aim)) continue;
                    if (a.conj_amp) aim = -aim;
                    U m;
                    int bi, st;
                    orbit_min<U>(g, t, m, bi, st);
                    int64_t idx = rank_search<U>((const U*)a.reps, a.n, spl, (int)a.nsplit, a.stride, m);
                    if (idx < 0) continue;
                    double hr = G->chi_re[bi], hi = a.conj_chi ? -G->chi_im[bi] : G->chi_im[bi];
                    double orb_m = (double)g.ng / (double)st;
                    double f = 1.0 / ((double)stab_r * sqrt(orb_r * orb_m));
                    // w = chi(g_e) * A * chi(h) * f
                    double t1r = er * are - ei * aim, t1i = er * aim + ei * are;
                    double wr = (t1r * hr - t1i * hi) * f, wi = (t1r * hi + t1i * hr) * f;
                    double xr, xi;
                    if (kCV) {
                        double2 v = ((const double2*)a.x)[idx];
                        xr = v.x;
                        xi = v.y;
                    } else {
                        xr = ((const double*)a.x)[idx];
                        xi = 0;
                    }
                    acc_r += wr * xr - wi * xi;
                    acc_i += wr * xi + wi * xr;
                }
            }
        }
        double2 d = ((const double2*)a.diag)[r];
        double dr = d.x, di = a.conj_amp ? -d.y : d.y;
        double xr, xi;
        if (kCV) {
            double2 v = ((const double2*)a.x)[r];
            xr = v.x;
            xi = v.y;
        } else {
            xr = ((const double*)a.x)[r];
            xi = 0;
        }
        acc_r += dr * xr - di * xi;
        acc_i += dr * xi + di * xr;
        if (kCV) {
            double2* y = (double2*)a.y;
            double yr = 0, yi = 0;
            if (!a.beta_zero) {
                double2 yo = y[r];
                yr = a.br * yo.x - a.bi * yo.y;
                yi = a.br * yo.y + a.bi * yo.x;
            }
            y[r] = make_double2(yr + a.ar * acc_r - a.ai * acc_i, yi + a.ar * acc_i + a.ai * acc_r);
        } else {
            double* y = (double*)a.y;
            double yr = a.beta_zero ? 0.0 : a.br * y[r];
            y[r] = yr + a.ar * acc_r;
        }
    }
}

// The operator's diagonal in the forms that the products read: complex, real
// part, single precision, float pairs.
struct DiagOut {
    const double* user;   // null: no user diagonal
    double *d64, *re64;
    float *d32, *re32;
    float4* df;
};

// Diagonal of the structurally diagonal programs on each row's representative,
// and its copies.  Nearly every program is alive on every row, so the row's sum
// is bound by its FP64 additions: one per program where all amplitudes are real
// (kIm false), the sign put on by an integer XOR, the programs' masks from
// shared memory.  60 programs on 1.3 M rows: 0.36 ms, against 1.22 ms with the
// programs read from global memory and two additions and two negations each,
// and the four conversions another 0.06 ms in kernels of their own.
constexpr int kDiagChunk = 256;

template <typename U>
struct DiagSmem {
    RowTest<U> test[kDiagChunk];
    U zy[kDiagChunk];
    double2 amp[kDiagChunk];
    int8_t chars[kDiagChunk];
};

template <typename U, bool kIm>
__global__ void __launch_bounds__(kMvThreads) diag_kernel(MvArgs a, DiagOut o) {
    __shared__ DiagSmem<U> sm;
    const int mode = a.reps ? 2 : (a.nup >= 0 ? 1 : 0);
    const bool one = a.nprog <= kDiagChunk;   // staged once
    for (int64_t r0 = blockIdx.x * (int64_t)blockDim.x; r0 < a.n; r0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = r0 + threadIdx.x;
        const U s = r < a.n ? row_state<U>(a, mode, r) : 0;
        // extracted diagonal summed from zero in term order, then added to the
        // user diagonal (diagonal + extracted_diagonal, src/operators.jl:3103-3106)
        double dr = 0.0, di = 0.0;
        for (int c0 = 0; c0 < a.nprog; c0 += kDiagChunk) {
            const int nc = min(kDiagChunk, a.nprog - c0);
            if (!one || r0 == blockIdx.x * (int64_t)blockDim.x) {
                __syncthreads();
                for (int i = threadIdx.x; i < nc; i += blockDim.x) {
                    const TermProg& p = a.progs[c0 + i];
                    sm.test[i] = RowTest<U>{(U)(p.need0 | p.need1), (U)p.need1};
                    sm.zy[i] = (U)(p.zmask ^ p.ymask);
                    // popc(~s & z) = popc(z) - popc(s & z)
                    const bool neg = __popcll(p.zmask) & 1;
                    sm.amp[i] = neg ? make_double2(-p.amp0_re, -p.amp0_im) : make_double2(p.amp0_re, p.amp0_im);
                    sm.chars[i] = !p.distinct;
                }
                __syncthreads();
            }
            for (int i = 0; i < nc; ++i) {
                if (sm.chars[i]) {
                    U t;
                    double are, aim;
                    if (!run_prog<U, double>(a.progs[c0 + i], a.pauli, s, t, are, aim)) continue;
                    dr += are;
                    if (kIm) di += aim;
                    continue;
                }
                const RowTest<U> q = sm.test[i];
                if ((s & q.care) != q.value) continue;
                const long long sign = (long long)__popcll((unsigned long long)(s & sm.zy[i])) << 63;
                const double2 v = sm.amp[i];
                dr += __longlong_as_double(__double_as_longlong(v.x) ^ sign);
                if (kIm) di += __longlong_as_double(__double_as_longlong(v.y) ^ sign);
            }
        }
        if (r >= a.n) continue;
        const double re = (o.user ? o.user[2 * r] : 0.0) + dr, im = (o.user ? o.user[2 * r + 1] : 0.0) + di;
        ((double2*)o.d64)[r] = make_double2(re, im);
        o.re64[r] = re;
        ((float2*)o.d32)[r] = make_float2((float)re, (float)im);
        o.re32[r] = (float)re;
        const DF h = df_from_double(re), l = df_from_double(im);
        o.df[r] = make_float4(h.h, h.l, l.h, l.l);
    }
}

int mv_grid(int64_t n, int threads = kMvThreads) {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t blocks = (n + threads - 1) / threads;
    int64_t cap = (int64_t)sms * 8;
    return (int)std::max<int64_t>(1, std::min(blocks, cap));
}

MvArgs base_args(const Op& op) {
    const Basis& b = *op.basis;
    MvArgs a{};
    a.reps = b.symmetric ? b.d_reps.p : nullptr;
    a.stab = b.d_stab.as<uint16_t>();
    a.split = b.d_split.p;
    a.n = b.n;
    a.nsplit = b.nsplit;
    a.stride = b.split_stride;
    a.group = b.d_group.as<GroupDesc>();
    a.binom = b.d_binom.as<uint64_t>();
    a.L = b.L;
    a.nup = b.nup;
    a.pauli = b.spec.pauli;
    return a;
}

// What matvec_kernel and matvec_warp_rank_kernel take besides: the row walk and
// the values.  `bwd`: the second half of the programs (the chain of A itself).
void row_args(const Op& op, bool bwd, MvArgs& a) {
    const Basis& b = *op.basis;
    const size_t half = op.progs.size() / 2;
    a.progs = op.d_progs.as<TermProg>() + (bwd ? half : 0);
    a.nprog = (int)half;
    a.row = op_row_args(op, bwd);
    if (b.symmetric && b.fast.enabled) {
        a.chi_re = b.d_fast_chi.as<double>();
        a.chi_im = a.chi_re + 1;
        a.chi_stride = 2;
        a.nelem = 4 * b.fast.nT;
    } else if (b.symmetric) {
        a.chi_re = b.d_group.as<GroupDesc>()->chi_re;
        a.chi_im = b.d_group.as<GroupDesc>()->chi_im;
        a.chi_stride = 1;
        a.nelem = b.group.ng;
    }
    bool ones = true;
    for (int e = 0; b.symmetric && e < b.group.ng; ++e)
        ones = ones && b.group.chi_re[e] == 1.0 && b.group.chi_im[e] == 0.0;
    if (ones) a.nelem = 1;
    a.amp = op.d_amp.as<double2>();
    a.nclass = op.nclass;
    a.table = (int64_t)op.nclass * a.nelem <= kRowValues;
    a.any_chars = op.any_chars;
    a.sq = b.d_sqrt.as<double>();
}

// Launches a row kernel with `dyn` bytes of dynamic shared memory.
template <class K>
void launch_rows(K kernel, int grid, int threads, size_t dyn, cudaStream_t s, const MvArgs& a) {
    allow_row_smem(kernel, dyn);
    kernel<<<grid, threads, dyn, s>>>(a);
}

// Threads per block: at least four blocks per SM where the rows allow (one
// product of 12,870 rows: 51 blocks of 256 threads left two SMs of three idle)
int mv_threads(int64_t n) {
    int t = kMvThreads;
    while (t > 64 && n < (int64_t)t * 152 * 4) t /= 2;
    return t;
}

template <typename U, int kMode, typename T>
void launch_mode(const MvArgs& a, bool cm, bool cv, cudaStream_t s) {
    const int threads = mv_threads(a.n);
    const int grid = mv_grid(a.n, threads);
    const bool ranks = sizeof(U) == 4 && (kMode == 1 || kMode == 3);
    const size_t dyn = (a.table ? mv_table_bytes(a.nclass * a.nelem, cm, sizeof(T)) : 0) +
                       (ranks ? (size_t)a.row.rank.size * sizeof(uint32_t) : 0);
#define QS_ROWS(P_)                                                                                       \
    do {                                                                                                   \
        if (cm) launch_rows(matvec_kernel<U, kMode, true, true, T, P_>, grid, threads, dyn, s, a);         \
        else if (cv) launch_rows(matvec_kernel<U, kMode, false, true, T, P_>, grid, threads, dyn, s, a);   \
        else launch_rows(matvec_kernel<U, kMode, false, false, T, P_>, grid, threads, dyn, s, a);          \
    } while (0)
    if constexpr (sizeof(U) == 4 && (kMode == 1 || kMode == 3)) {
        if (a.table && !a.any_chars && !a.row.any_zy && !a.row.check_weight && !a.solver) {
            QS_ROWS(true);
            return;
        }
    }
    QS_ROWS(false);
#undef QS_ROWS
}

// QS_RANK_MODE picks the rank lookup of a symmetric sector's generated states
// (read on every product): "direct" (the rank -> column table, when built),
// "search" (per-thread binary search behind shared-memory splitters) or
// "warp" (the warp-cooperative search); default: direct when built, else search.
int rank_mode_env() {
    const char* e = std::getenv("QS_RANK_MODE");
    if (!e || !e[0]) return -1;
    if (!std::strcmp(e, "direct")) return 3;
    if (!std::strcmp(e, "search")) return 2;
    if (!std::strcmp(e, "warp")) return 4;
    return -1;
}

template <typename T>
void launch_matvec(const Basis& b, const MvArgs& a, bool cm, bool cv, cudaStream_t s) {
    const int rm = b.symmetric ? rank_mode_env() : -1;
    if (rm == 4) {
        const int grid = mv_grid(a.n);
        const size_t dyn = a.table ? mv_table_bytes(a.nclass * a.nelem, cm, sizeof(T)) : 0;
#define QS_WARP(U_)                                                                                                 \
        do {                                                                                                        \
            if (cm) launch_rows(matvec_warp_rank_kernel<U_, true, true, T>, grid, kMvThreads, dyn, s, a);           \
            else if (cv) launch_rows(matvec_warp_rank_kernel<U_, false, true, T>, grid, kMvThreads, dyn, s, a);     \
            else launch_rows(matvec_warp_rank_kernel<U_, false, false, T>, grid, kMvThreads, dyn, s, a);            \
        } while (0)
        if (b.wide) QS_WARP(uint64_t);
        else QS_WARP(uint32_t);
#undef QS_WARP
        return;
    }
    if (b.symmetric && rm == 2) {
        if (b.wide) launch_mode<uint64_t, 2, T>(a, cm, cv, s);
        else launch_mode<uint32_t, 2, T>(a, cm, cv, s);
        return;
    }
    if (b.symmetric && b.has_index) {
        if (b.wide) launch_mode<uint64_t, 3, T>(a, cm, cv, s);
        else launch_mode<uint32_t, 3, T>(a, cm, cv, s);
    } else if (b.symmetric) {
        if (b.wide) launch_mode<uint64_t, 2, T>(a, cm, cv, s);
        else launch_mode<uint32_t, 2, T>(a, cm, cv, s);
    } else if (b.nup >= 0) {
        // up to 32 sites: 32-bit states and the split rank tables
        if (b.wide) launch_mode<uint64_t, 1, T>(a, cm, cv, s);
        else launch_mode<uint32_t, 1, T>(a, cm, cv, s);
    } else {
        launch_mode<uint64_t, 0, T>(a, cm, cv, s);
    }
}

}  // namespace

namespace {
std::atomic<int64_t> g_launches{0};
std::atomic<int64_t> g_device_allocs{0};
}
void note_launches(int64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
int64_t launches() { return g_launches.load(std::memory_order_relaxed); }
void note_device_alloc() { g_device_allocs.fetch_add(1, std::memory_order_relaxed); }
int64_t device_allocs() { return g_device_allocs.load(std::memory_order_relaxed); }

Op::~Op() {
    if (copy_stream) {
        cudaStreamSynchronize(copy_stream);
        cudaStreamDestroy(copy_stream);
        for (cudaEvent_t e : range_done)
            if (e) cudaEventDestroy(e);
    }
    if (own_stream) cudaStreamDestroy(own_stream);
}

namespace {

// The programs as the row kernels read them (RowProg) and their amplitude
// classes.
void prepare_row_programs(Op& op, std::vector<RowProg>& rows, std::vector<double>& amp) {
    const Basis& b = *op.basis;
    rows.assign(op.progs.size(), RowProg{});
    // by the values' bits: a coupling that is not a number is a class of its own
    std::map<std::pair<uint64_t, uint64_t>, uint32_t> seen;
    auto bits = [](double v) {
        uint64_t u;
        std::memcpy(&u, &v, sizeof(u));
        return u;
    };
    op.any_zy = op.check_weight = op.any_chars = false;
    for (size_t k = 0; k < op.progs.size(); ++k) {
        const TermProg& p = op.progs[k];
        RowProg& r = rows[k];
        if (!p.distinct) {
            // care = value = 0: alive on every state until its characters say otherwise
            r.cls = kCharsClass;
            op.any_chars = true;
            op.check_weight = b.nup >= 0;
            continue;
        }
        r.care = p.need0 | p.need1;
        r.value = p.need1;
        r.flip = p.flip;
        r.zy = p.zmask ^ p.ymask;
        // popc(~s & z) = popc(z) - popc(s & z): the constant part joins the amplitude
        const double sg = (__builtin_popcountll(p.zmask) & 1) ? -1.0 : 1.0;
        const double re = sg * p.amp0_re, im = sg * p.amp0_im;
        const std::pair<uint64_t, uint64_t> v{bits(re), bits(im)};
        auto it = seen.find(v);
        if (it == seen.end()) {
            it = seen.emplace(v, (uint32_t)(amp.size() / 2)).first;
            amp.push_back(re);
            amp.push_back(im);
        }
        r.cls = it->second;
        if (r.zy) op.any_zy = true;
        // the particle number: every flipped site raised or lowered, as many up as down
        if ((p.flip & ~(p.need0 | p.need1)) != 0 ||
            __builtin_popcountll(p.flip & p.need0) != __builtin_popcountll(p.flip & p.need1))
            op.check_weight = op.check_weight || b.nup >= 0;
    }
    op.nclass = (int)(amp.size() / 2);
    op.prog_class.resize(rows.size());
    for (size_t k = 0; k < rows.size(); ++k) op.prog_class[k] = rows[k].cls;
    if (amp.empty()) amp.assign(2, 0.0);
}

}  // namespace

RowArgs op_row_args(const Op& op, bool bwd) {
    const Basis& b = *op.basis;
    RowArgs R{};
    R.reps = b.symmetric ? b.d_reps.p : nullptr;
    R.stab = b.d_stab.as<uint16_t>();
    R.split = b.d_split.p;
    R.n = b.n;
    R.nsplit = b.nsplit;
    R.stride = b.split_stride;
    R.group = b.d_group.as<GroupDesc>();
    R.binom = b.d_binom.as<uint64_t>();
    R.index = b.has_index ? b.d_index.as<int32_t>() : nullptr;
    R.L = b.L;
    R.nup = b.nup;
    R.nprog = (int)(op.progs.size() / 2);
    R.progs = op.d_rowprogs.as<RowProg>() + (bwd ? R.nprog : 0);
    R.any_zy = op.any_zy;
    R.check_weight = op.check_weight;
    R.fast = b.fast;
    R.rank = b.rank;
    R.rank_tab = b.d_rank.as<uint32_t>();
    return R;
}

void op_prepare_device(Op& op) {
    Basis& b = *op.basis;
    if (!op.own_stream) {
        QS_CUDA(cudaStreamCreateWithFlags(&op.own_stream, cudaStreamNonBlocking));
        op.stream = op.own_stream;
    }
    std::vector<RowProg> rows;
    std::vector<double> amp;
    prepare_row_programs(op, rows, amp);
    if (rows.empty()) rows.resize(1);
    const size_t np = std::max<size_t>(1, op.progs.size()), nd = std::max<size_t>(1, op.diag_progs.size());
    DevBuf dprogs;
    BufPack tables;
    tables.add(op.d_progs, np * sizeof(TermProg), op.progs.empty() ? nullptr : op.progs.data());
    tables.add(op.d_rowprogs, rows.size() * sizeof(RowProg), rows.data());
    tables.add(op.d_amp, amp.size() * sizeof(double), amp.data());
    tables.add(dprogs, nd * sizeof(TermProg), op.diag_progs.empty() ? nullptr : op.diag_progs.data());
    tables.place(op.d_tables, op.stream);
    // diagonal: user diagonal plus, when extracted, the diagonal programs
    PoolBuf user;
    if (!op.user_diag.empty()) {
        user.alloc(2 * b.n * sizeof(double), op.stream);
        QS_CUDA(cudaMemcpyAsync(user.p, op.user_diag.data(), user.bytes, cudaMemcpyHostToDevice, op.stream));
    }
    op.diag_im = false;
    for (const std::complex<double>& v : op.user_diag) op.diag_im = op.diag_im || v.imag() != 0.0;
    BufPack diags;
    diags.add(op.d_diag, 2 * b.n * sizeof(double));
    diags.add(op.d_diag32, 2 * b.n * sizeof(float));
    diags.add(op.d_diag_df, b.n * 4 * sizeof(float));
    diags.add(op.d_diag_re, b.n * sizeof(double));
    diags.add(op.d_diag32_re, b.n * sizeof(float));
    diags.place(op.d_diags, op.stream);
    MvArgs a = base_args(op);
    a.progs = dprogs.as<TermProg>();
    a.nprog = (int)op.diag_progs.size();
    const DiagOut o{user.as<double>(),           op.d_diag.as<double>(),   op.d_diag_re.as<double>(),
                    op.d_diag32.as<float>(),     op.d_diag32_re.as<float>(), op.d_diag_df.as<float4>()};
    bool im = false;
    for (const TermProg& p : op.diag_progs) im = im || !p.distinct || p.amp0_im != 0.0;
    const int grid = mv_grid(b.n);
    if (b.symmetric && !b.wide) {
        if (im) diag_kernel<uint32_t, true><<<grid, kMvThreads, 0, op.stream>>>(a, o);
        else diag_kernel<uint32_t, false><<<grid, kMvThreads, 0, op.stream>>>(a, o);
    } else {
        if (im) diag_kernel<uint64_t, true><<<grid, kMvThreads, 0, op.stream>>>(a, o);
        else diag_kernel<uint64_t, false><<<grid, kMvThreads, 0, op.stream>>>(a, o);
    }
    QS_CUDA(cudaGetLastError());
    QS_CUDA(cudaStreamSynchronize(op.stream));
}

void op_matvec_device(Op& op, const MatvecCall& c, cudaStream_t s) {
    if (op.dense) {
        op_matvec_dense(op, c, s);
        return;
    }
    const Basis& b = *op.basis;
    MvArgs a = base_args(op);
    a.progs = op.d_progs.as<TermProg>();
    a.nprog = (int)op.progs.size();
    const bool T = (c.flags & QS_TRANSPOSE) != 0, C = (c.flags & QS_CONJUGATE) != 0;
    a.conj_amp = C;
    a.conj_chi = T != C;
    a.ar = c.alpha.re;
    a.ai = c.alpha.im;
    a.br = c.beta.re;
    a.bi = c.beta.im;
    a.beta_zero = (c.beta.re == 0.0 && c.beta.im == 0.0);
    a.solver = c.solver;
    a.full_diag = c.solver || op.diag_im;
    a.x = c.x;
    a.y = c.y;
    // the pull form of op(A) runs the chain of op(A)^T; a transposed call runs
    // A's own chain (programs are stored for both)
    row_args(op, T, a);
    const bool cm = op.complex_mat;
    const bool cv = c.y_complex;
    if (c.x_complex && !c.y_complex) throw Error(QS_ERR_ARGUMENT, "a complex input needs a complex output");
    if (cm && !cv) throw Error(QS_ERR_ARGUMENT, "a complex operator needs a complex output");
    if (!cv && c.x_complex) throw Error(QS_ERR_ARGUMENT, "a complex input needs a complex output");
    if (c.x_complex != cv) throw Error(QS_ERR_UNSUPPORTED, "input and output must share a dtype at the device boundary");
    if (!op.commuting) {
        if (c.single) throw Error(QS_ERR_UNSUPPORTED, "the single-precision form needs a symmetry-commuting operator");
        a.diag = op.d_diag.p;
        int grid = mv_grid(b.n);
        if (b.wide) {
            if (cv) matvec_general_kernel<uint64_t, true><<<grid, kMvThreads, 0, s>>>(a);
            else matvec_general_kernel<uint64_t, false><<<grid, kMvThreads, 0, s>>>(a);
        } else {
            if (cv) matvec_general_kernel<uint32_t, true><<<grid, kMvThreads, 0, s>>>(a);
            else matvec_general_kernel<uint32_t, false><<<grid, kMvThreads, 0, s>>>(a);
        }
        QS_CUDA(cudaGetLastError());
        note_launches(1);
        return;
    }
    if (op.assembled && (!T || op.hermitian)) {
        op_spmv_device(op, c, s);
        return;
    }
    if (c.df_io) throw Error(QS_ERR_UNSUPPORTED, "double-float vectors need an assembled operator");
    if (c.single) {
        a.diag = op.d_diag32.p;
        a.diag_re = op.d_diag32_re.p;
        launch_matvec<float>(b, a, cm, cv, s);
    } else {
        a.diag = op.d_diag.p;
        a.diag_re = op.d_diag_re.p;
        launch_matvec<double>(b, a, cm, cv, s);
    }
    QS_CUDA(cudaGetLastError());
    note_launches(1);
}

}  // namespace qs
