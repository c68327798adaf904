// qs_rows.cuh -- the transitions of one row: shared by the matrix-free product
// (qs_matvec.cu) and the assembly (qs_assembled.cu).
//
// Only some of the programs are alive on a row (a "+-" exchange on a quarter of
// the rows, 33 of 128 programs on the J1-J2 L=32 sector), and different ones in
// every lane.  Walking the programs in step leaves three lanes of four idle
// through the orbit search (16.6 active lanes of 32 measured, the idle ones
// included in 745 issued instructions a program).  So each lane first tests the
// programs of a chunk in uniform order (three instructions each) into a bit
// mask, then walks its own set bits: a warp runs as many orbit searches as its
// fullest lane has live programs (about 41 instead of 128), all lanes busy.
// Every lane still takes its programs in ascending order, so a row's sum adds
// in the same order as before.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "qs_device.cuh"
#include "qs_internal.h"

namespace qs {

constexpr int kRowThreads = 256;   // threads of a row kernel, at most
constexpr int kRowChunk = 128;     // programs held in shared memory at once

constexpr int kRowValues = 1024;   // (class, element) values staged in shared memory, at most

// Dynamic shared memory of a row kernel past the 16 KB that fit beside its
// static arrays: the limit belongs to the kernel, not to a call, and a launch
// above it fails, so every call allows the same, the most a sector can need
// (complex FP64 values, and the rank tables of 16 particles on 32 sites: 36 rows
// of 256 entries); calls from several threads meet the same limit.
constexpr size_t kRowDyn = (size_t)kRowValues * 16 + 36 * 256 * sizeof(uint32_t);
template <class K>
void allow_row_smem(K kernel, size_t dyn) {
    if (dyn > kRowDyn) throw Error(QS_ERR_UNSUPPORTED, "row kernel tables exceed their shared memory");
    if (dyn > 16 * 1024)
        QS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowDyn));
}

// What the row kernels need to know about the basis and the programs.
struct RowArgs {
    const void* reps;
    const uint16_t* stab;
    const void* split;
    int64_t n, nsplit, stride;
    const GroupDesc* group;
    const uint64_t* binom;
    const int32_t* index;        // direct rank -> column table
    int L, nup;
    const RowProg* progs;
    int nprog;
    int any_zy;                  // some program's sign depends on the state
    int check_weight;            // nup is given and some program changes the particle number
    FastGroup fast;
    RankSplit rank;
    const uint32_t* rank_tab;    // rank.size entries, staged in shared memory
};

// The arguments for an operator's forward (A^T's chain) or backward programs
// (qs_matvec.cu).
RowArgs op_row_args(const Op& op, bool bwd);

template <typename U>
struct RowTest {
    U care, value;
};
template <typename U>
struct RowSmem {
    RowTest<U> test[kRowChunk];   // one 8- or 16-byte read per test
    U flip[kRowChunk], zy[kRowChunk];
    uint32_t cls[kRowChunk];
    uint32_t live[kRowChunk / 32][kRowThreads];
};

// Programs c0 .. of the chunk into shared memory (every thread of the block).
template <typename U>
__device__ __forceinline__ void load_row_progs(RowSmem<U>& sm, const RowArgs& a, int c0) {
    const int nc = min(kRowChunk, a.nprog - c0);
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
        const RowProg p = a.progs[c0 + i];
        sm.test[i] = RowTest<U>{(U)p.care, (U)p.value};
        sm.flip[i] = (U)p.flip;
        sm.zy[i] = (U)p.zy;
        sm.cls[i] = p.cls;
    }
}

// ------------------------------------------------------------ orbit minimum
// Orbit minimum over one-site translations (and parity, and the full flip) of
// a state of at most 32 sites, all rotations compared.  The state's bits,
// repeated periodically over 64 bits from the top, hold rotation j as the
// 32-bit window at offset j; windows compare as the rotations do (their bits
// past L repeat the first ones), so one funnel shift and half a three-input
// minimum serve a rotation, and the maximum over the same windows gives the
// flipped states' minimum.  About 130 instructions for 2 x 32 rotations and both
// flips with no divergence, where the zero-run search took about 500 with its
// lane-dependent loops; windows beyond L - 1 repeat earlier ones.
struct WinBase {
    uint32_t hi, lo;
    uint32_t mn, mx;
    int gmn, gmx;   // groups of eight windows that hold them first (kJ)
};

// t's L bits repeated from the top of hi, through lo
__device__ __forceinline__ void win_periodic(uint32_t t, int L, uint32_t& hi, uint32_t& lo) {
    hi = t << (32 - L);
    for (int w = L; w < 32; w <<= 1) hi |= hi >> w;
    // the string's bit 32 + i is its bit 32 - L + i
    lo = hi << (32 - L);
    for (int w = L; w < 32; w <<= 1) lo |= lo >> w;
}

template <bool kFlip, bool kJ>
__device__ __forceinline__ void win_scan(WinBase& b, int L) {
    b.mn = 0xffffffffu;
    b.mx = 0u;
    b.gmn = b.gmx = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (8 * g >= L) break;
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = __funnelshift_l(b.lo, b.hi, 8 * g + i);
        if (kJ) {
            const uint32_t m =
                __vimin3_u32(__vimin3_u32(w[0], w[1], w[2]), __vimin3_u32(w[3], w[4], w[5]), min(w[6], w[7]));
            if (m < b.mn) b.gmn = g;
            b.mn = min(b.mn, m);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i += 2) b.mn = __vimin3_u32(b.mn, w[i], w[i + 1]);
        }
        if (kFlip && kJ) {
            const uint32_t x =
                __vimax3_u32(__vimax3_u32(w[0], w[1], w[2]), __vimax3_u32(w[3], w[4], w[5]), max(w[6], w[7]));
            if (x > b.mx) b.gmx = g;
            b.mx = max(b.mx, x);
        } else if (kFlip) {
#pragma unroll
            for (int i = 0; i < 8; i += 2) b.mx = __vimax3_u32(b.mx, w[i], w[i + 1]);
        }
    }
}

// elem = (r * 2 + f) * nT + j as orbit_min_fast numbers the elements (j = 0
// without kJ: the characters do not depend on it), the first in that order
// among the elements that reach the minimum; stab = their number.
template <bool kFlip, bool kJ>
__device__ __forceinline__ void orbit_min_bases(const FastGroup& G, uint32_t t, uint32_t& best, int& elem, int& stab) {
    const int L = G.L;
    WinBase b[2];
    win_periodic(t, L, b[0].hi, b[0].lo);
    win_scan<kFlip, kJ>(b[0], L);
    uint32_t w = b[0].mn;
    int q = 0, g = b[0].gmn, n = 1;
    auto take = [&](uint32_t c, int code, int grp) {
        if (c == w) ++n;
        if (c < w) {
            w = c;
            q = code;
            if (kJ) g = grp;
            n = 1;
        }
    };
    if (kFlip) take(~b[0].mx, 1, b[0].gmx);
    if (G.has_refl) {
        win_periodic(__brev(t) >> (32 - L), L, b[1].hi, b[1].lo);
        win_scan<kFlip, kJ>(b[1], L);
        take(b[1].mn, 2, b[1].gmn);
        if (kFlip) take(~b[1].mx, 3, b[1].gmx);
    }
    best = w >> (32 - L);
    // rotations that fix the state (the same number from every base)
    bool sym = false;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (i < G.nper) sym |= __funnelshift_l(b[0].lo, b[0].hi, G.per[i]) == b[0].hi;
    if (sym) {
        int c = 1;
        for (int j = 1; j < L; ++j) c += __funnelshift_l(b[0].lo, b[0].hi, j) == b[0].hi;
        n *= c;
    }
    stab = n;
    elem = q * G.nT;
    if (kJ) {
        const uint32_t hi = (q & 2) ? b[1].hi : b[0].hi, lo = (q & 2) ? b[1].lo : b[0].lo;
        const uint32_t target = (q & 1) ? ~w : w;
        int j = 0;
#pragma unroll
        for (int i = 7; i >= 0; --i)
            if (__funnelshift_l(lo, hi, 8 * g + i) == target) j = i;
        elem += 8 * g + j;
    }
}

__device__ __forceinline__ void orbit_min_win(const FastGroup& G, uint32_t t, uint32_t& best, int& elem, int& stab) {
    if (G.win == 2) {   // no translations
        const uint32_t lm = (uint32_t)G.lmask;
        const uint32_t tr = __brev(t) >> (32 - G.L);
        const uint32_t c[4] = {t, ~t & lm, tr, ~tr & lm};
        best = t;
        elem = 0;
        stab = 1;
#pragma unroll
        for (int q = 1; q < 4; ++q) {
            if (((q & 1) && !G.has_flip) || ((q & 2) && !G.has_refl)) continue;
            if (c[q] < best) {
                best = c[q];
                elem = q;
                stab = 1;
            } else if (c[q] == best) {
                ++stab;
            }
        }
        return;
    }
    if (G.need_j) {
        if (G.has_flip) orbit_min_bases<true, true>(G, t, best, elem, stab);
        else orbit_min_bases<false, true>(G, t, best, elem, stab);
    } else {
        if (G.has_flip) orbit_min_bases<true, false>(G, t, best, elem, stab);
        else orbit_min_bases<false, false>(G, t, best, elem, stab);
    }
}

// Minimum, element and stabiliser order by the cheapest search the group allows.
template <typename U>
__device__ __forceinline__ void row_orbit(const RowArgs& a, const GroupSmem& g, U t, U& m, int& ec, int& st) {
    if (sizeof(U) == 4 && a.fast.win) {
        uint32_t m32;
        orbit_min_win(a.fast, (uint32_t)t, m32, ec, st);
        m = (U)m32;
    } else if (a.fast.enabled) {
        orbit_min_fast<U>(a.fast, t, m, ec, st);
    } else {
        orbit_min<U>(g, t, m, ec, st);
    }
}

// ------------------------------------------------------------ ranks
// Combinadic rank of a fixed-weight state of at most 32 sites from four table
// reads: piece k holds the terms C(bit, particle) of the bits k w .. k w + w - 1
// summed for every pattern of those bits and every number of particles below
// (36 KB at L = 32, nup = 16; the loop over the set bits took 16 dependent reads).
__device__ __forceinline__ uint32_t rank_split(const RankSplit& R, const uint32_t* tab, uint32_t s) {
    const int w = R.w;
    const uint32_t pm = (1u << w) - 1u;
    uint32_t below = s & pm;
    uint32_t r = tab[below];
    int p = __popc(below);
#pragma unroll
    for (int k = 1; k < 4; ++k) {
        const uint32_t bits = (s >> (k * w)) & pm;
        r += tab[R.off[k] + (p << w) + (int)bits];
        if (k < 3) p += __popc(bits);
    }
    return r;
}

// kMode: 0 full space, 1 fixed weight without symmetry, 2 representatives found
// by search, 3 by the direct table
template <typename U, int kMode>
__device__ __forceinline__ int64_t row_column(const RowArgs& a, const U* spl, const uint32_t* rtab, U m) {
    if (kMode == 0) return (int64_t)m;
    if (kMode == 2) return rank_search<U>((const U*)a.reps, a.n, spl, (int)a.nsplit, a.stride, m);
    int64_t rk;
    if (kMode == 3 && a.nup < 0) rk = (int64_t)m;
    else if (sizeof(U) == 4) rk = (int64_t)rank_split(a.rank, rtab, (uint32_t)m);
    else rk = combinadic_rank<U>(m, a.binom, 65);
    return kMode == 3 ? (int64_t)__ldg(a.index + rk) : rk;
}

// Walks the live programs of the chunk [c0, c0 + nc) on state s: one call of
// hop(i, t, sign) per live program i of the chunk, ascending.  kSign: some sign
// depends on the state.
template <typename U, bool kSign, class Hop>
__device__ __forceinline__ void row_hops(RowSmem<U>& sm, const RowArgs& a, int nc, bool valid, U s, Hop hop) {
    const int nw = (nc + 31) >> 5;
    for (int w = 0; w < nw; ++w) {
        uint32_t bits = 0;
        const int k1 = min(32, nc - 32 * w);
        if (k1 == 32) {
#pragma unroll 8
            for (int i = 0; i < 32; ++i) {
                const RowTest<U> q = sm.test[32 * w + i];
                if ((s & q.care) == q.value) bits |= 1u << i;
            }
        } else {
            for (int i = 0; i < k1; ++i) {
                const RowTest<U> q = sm.test[32 * w + i];
                if ((s & q.care) == q.value) bits |= 1u << i;
            }
        }
        sm.live[w][threadIdx.x] = valid ? bits : 0u;
    }
    int w = 0;
    uint32_t cur = sm.live[0][threadIdx.x];
    while (true) {
        while (cur == 0u && ++w < nw) cur = sm.live[w][threadIdx.x];
        if (cur == 0u) break;
        const int i = 32 * w + __ffs((int)cur) - 1;
        cur &= cur - 1u;
        int sign = 0;
        if (kSign && a.any_zy)
            sign = (sizeof(U) == 8 ? __popcll((unsigned long long)(s & sm.zy[i])) : __popc((unsigned)(s & sm.zy[i]))) & 1;
        hop(i, (U)(s ^ sm.flip[i]), sign);
    }
}

}  // namespace qs
